"""Short lists and fields around the sizes at which the rank stage changes its
way: pairs around 2^16, buckets around the sizes that one CTA sorts with 2, 4,
8 and 16 keys a thread and beyond, and fields around 2^14 values."""
import ctypes

import numpy as np
import pytest

from test_gpu_rank import _codes, _expect

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def T():
    import torch
    import toposzp_b200
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    toposzp_b200.lib()
    return toposzp_b200


def _rank(T, v, eb, rng):
    import torch
    n = v.size
    ext = rng.random(n) < 0.7
    ext[0] = True
    idx = np.where(ext, np.cumsum(ext) - 1, 0xffffffff).astype(np.uint32)
    pairs = torch.from_numpy(np.stack([_codes(v), idx], 1).astype(np.uint32).view(np.int32)).cuda()
    sp = torch.full((int(ext.sum()),), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    ctx = T.Context()
    rc = T.lib().szp_b200_rank_pairs_dev(ctx.ptr, ctypes.c_void_p(pairs.data_ptr()), n, sp.numel(), ctypes.c_float(eb),
                                         ctypes.c_void_p(sp.data_ptr()))
    assert rc == 0, T.last_error()
    assert (sp.cpu().numpy() == _expect(v, eb)[ext]).all()
    ctx.close()


@pytest.mark.parametrize("n", [65535, 65536, 65537])
@pytest.mark.parametrize("eb", [1e-4, 0.3, 1e3])
def test_pairs_around_the_line(T, n, eb):
    rng = np.random.default_rng(n)
    _rank(T, rng.standard_normal(n).astype(np.float32), eb, rng)


@pytest.mark.parametrize("m", [1, 2047, 2048, 2049, 4095, 4096, 4097, 8191, 8192, 8193, 16383, 16384, 16385, 40000])
@pytest.mark.parametrize("ties", [False, True])
def test_one_wide_bin(T, m, ties):
    """m values over all magnitudes below eb, in one bin, and 2500 in others."""
    rng = np.random.default_rng(m)
    eb = 0.5
    v = 10.0 ** rng.uniform(-30, np.log10(0.49), m)
    if ties:
        v = rng.choice(v[:max(m // 3, 1)], m)
    v = np.r_[v, rng.uniform(1, 400, 2500)].astype(np.float32)
    _rank(T, rng.permutation(v), eb, rng)


@pytest.mark.parametrize("dims", [(127, 129), (128, 128), (113, 145), (24, 26, 27), (16, 32, 32)])
@pytest.mark.parametrize("eb", [1e-3, 0.3, 1e3])
def test_fields_around_the_line(T, ora, dims, eb):
    import torch
    d = np.random.default_rng(sum(dims)).standard_normal(dims).astype(np.float32)
    cp = ora.sort_cp(ora.find_cp(d, eb), d)
    ctx = T.Context()
    x = torch.from_numpy(d.reshape(-1).copy()).cuda()
    for _ in range(2):
        t, s, _, sz = ctx.compress(x, dims, eb, 64)
        assert t[:sz.topo_bytes].cpu().numpy().tobytes() == ora.encode_topo(d, eb, 64, ora.mark_types(cp, dims))
        assert s[:sz.sort_bytes].cpu().numpy().tobytes() == ora.encode_ints(ora.extract_sp(cp), 64)
    ctx.close()
