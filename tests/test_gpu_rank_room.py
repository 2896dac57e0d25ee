"""The rank stage's bitmap (118 MB a workspace) is optional: where the device
has no room for it a reservation succeeds all the same and the streams are the
same."""
import pytest

import synth

pytestmark = pytest.mark.gpu

BITMAP = 100 << 20      # less than the allocation


@pytest.fixture(scope="module")
def T():
    import torch
    import toposzp_b200
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    toposzp_b200.lib()
    return toposzp_b200


def _field(dims, kind="noise"):
    import torch
    return torch.from_numpy(synth.small_field(dims, seed=3, kind=kind).reshape(-1).copy()).cuda()


def _buffers(T, n):
    import torch
    L = T.lib()
    return (torch.empty(L.szp_b200_topo_bound(n, 64), dtype=torch.uint8, device="cuda"),
            torch.empty(L.szp_b200_sort_bound(n, 64), dtype=torch.uint8, device="cuda"))


def _streams(topo, sort, sz):
    return topo[:sz.topo_bytes].cpu().numpy().tobytes(), sort[:sz.sort_bytes].cpu().numpy().tobytes()


def _hog(leave):
    import torch
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free, _ = torch.cuda.mem_get_info()
    return torch.empty(max(free - leave, 1), dtype=torch.uint8, device="cuda")


@pytest.mark.parametrize("dims", [(300, 300), (700, 601)])     # the bits set from pairs, and by the encoder
def test_compression_without_room(T, dims):
    import ctypes
    import torch
    x = _field(dims)
    n = x.numel()
    ref, bufs = T.Context(), _buffers(T, n)
    t, s, _, sz = ref.compress(x, dims, 1e-3, 64, index=False)
    want = _streams(t, s, sz)
    ref.close()
    ctx = T.Context()
    hog = _hog(BITMAP)
    for k in range(3):
        if k == 2:                      # room again
            del hog
            torch.cuda.empty_cache()
        got = T.Sizes()
        rc = T.lib().szp_b200_topo_compress_dev(ctx.ptr, x.data_ptr(), T.geom_of(dims), 1e-3, 64, bufs[0].data_ptr(),
                                                bufs[1].data_ptr(), None, ctypes.byref(got))
        assert rc == 0, T.last_error()
        assert _streams(*bufs, got) == want
    ctx.close()


def test_server_reservation_without_room(T):
    import torch
    dims = (160, 128, 128)
    x = _field(dims, "band")
    n = x.numel()
    ref, bufs = T.Context(), _buffers(T, n)
    t, s, _, sz = ref.compress(x, dims, 1e-4, 64, index=False)
    want = _streams(t, s, sz)
    ref.close()
    torch.cuda.empty_cache()
    torch.cuda.synchronize()
    before, _ = torch.cuda.mem_get_info()
    srv = T.Server(slots=1, max_batch=4)
    srv.reserve(n)
    torch.cuda.synchronize()
    need = before - torch.cuda.mem_get_info()[0]
    srv.close()
    srv = T.Server(slots=1, max_batch=4)
    hog = _hog(need - BITMAP // 2)      # all that a reservation takes, less half of the bitmap
    srv.reserve(n)
    arr = (T.Request * 1)()
    arr[0] = srv.compress_request(x, dims, 1e-4, False, *bufs)
    srv.run_trace(arr)
    assert arr[0].status == 0, arr[0].message
    assert _streams(*bufs, arr[0].sizes) == want
    srv.close()
    del hog
    torch.cuda.empty_cache()
