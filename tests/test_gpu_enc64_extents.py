"""The blockSize-64 topology encoder on fields with an extent of 1 or 2, which
have no interior point, and of 3, larger than a tile (2048 elements) and with
rows that an octet crosses: one call, a batch, and the slab encoder, against
the oracle."""
import numpy as np
import pytest


pytestmark = pytest.mark.gpu

DIMS = [(512, 1, 12), (70, 1, 100), (300, 1, 37), (2048, 1, 100), (400, 2, 9), (64, 2, 75), (1, 300, 13), (2, 300, 13),
        (3, 300, 13), (300, 3, 13), (300, 13, 1), (300, 13, 2), (300, 13, 3), (1, 2100), (2100, 1), (2, 1100), (3, 1100)]
EB = 1e-2


@pytest.fixture(scope="module")
def T():
    import torch
    import toposzp_b200
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    toposzp_b200.lib()
    return toposzp_b200


def _field(dims):
    return np.random.default_rng(sum(dims)).standard_normal(dims).astype(np.float32)


def _expect(ora, d):
    cp = ora.sort_cp(ora.find_cp(d, EB), d)
    sp = ora.extract_sp(cp)
    return ora.encode_topo(d, EB, 64, ora.mark_types(cp, d.shape)), ora.encode_ints(sp, 64) if len(sp) else b"", len(cp)


def _bytes(t, n):
    return t[:n].cpu().numpy().tobytes()


@pytest.mark.parametrize("dims", DIMS, ids=lambda d: "x".join(map(str, d)))
def test_call_and_slabs(T, ora, dims):
    import torch
    import shard
    d = _field(dims)
    topo, sort, K = _expect(ora, d)
    x = torch.from_numpy(d.reshape(-1).copy()).cuda()
    ctx = T.Context()
    t, s, _, sz = ctx.compress(x, dims, EB, 64)
    assert sz.cp_count == K
    assert _bytes(t, sz.topo_bytes) == topo
    assert sz.sort_bytes == len(sort) and _bytes(s, sz.sort_bytes) == sort
    # the payload of two slabs in turn is the stream's
    parts, cps = topo[:8], 0
    bounds = shard.slab_bounds(d.size, 2)
    for begin, end in zip(bounds[:-1], bounds[1:]):
        lo, hi = shard.halo_of(dims, begin, end, d.size)
        payload, pairs, _ = shard.CudaBackend(T, ctx).encode_slab(x[begin - lo:end + hi].clone(), lo, dims, EB, begin,
                                                                  end)
        parts += payload.cpu().numpy().tobytes()
        cps += pairs.shape[0]
    assert cps == K and parts == topo
    ctx.close()


def test_batch(T, ora):
    import torch
    b = T.Batch(64)
    fields = [_field(dims) for dims in DIMS]
    items = [(torch.from_numpy(d.reshape(-1).copy()).cuda(), d.shape, EB, False) for d in fields]
    for d, (t, s, sz, _) in zip(fields, b.compress(items)):
        topo, sort, K = _expect(ora, d)
        assert sz.cp_count == K, d.shape
        assert _bytes(t, sz.topo_bytes) == topo, d.shape
        assert sz.sort_bytes == len(sort) and _bytes(s, sz.sort_bytes) == sort, d.shape
    b.close()
