"""Sort positions: the bitmap over the values, the one-CTA sort of short
lists, and their hand-over to the bucket ranking, against dense ranks in numpy
(szp_b200_rank_pairs_dev) and against the oracle's sort stream (compression)."""
import ctypes

import numpy as np
import pytest

import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def T():
    import torch
    import toposzp_b200
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    toposzp_b200.lib()
    return toposzp_b200


def _codes(v):
    b = np.where(v == 0, np.float32(0), v).astype(np.float32).view(np.uint32)
    return np.where(b >> 31, ~b, b | np.uint32(0x80000000)).astype(np.uint32)


def _bins(v, eb):
    with np.errstate(all="ignore"):
        s = (v + np.float32(eb)).astype(np.float32).astype(np.float64) * (1.0 / np.float64(np.float32(eb)))
    return np.clip(np.trunc(s), -2.0 ** 31, 2.0 ** 31 - 1).astype(np.int64)


def _expect(v, eb):
    """Dense rank of each value among the distinct values of its bin."""
    c, bins = _codes(v), _bins(np.where(v == 0, np.float32(0), v), eb)
    u, inv = np.unique(c, return_inverse=True)
    ub = np.zeros(u.size, np.int64)
    ub[inv] = bins
    head = np.r_[True, ub[1:] != ub[:-1]]
    first = np.maximum.accumulate(np.where(head, np.arange(u.size), 0))
    return (np.arange(u.size) - first)[inv]


def _values(kind, n, eb, rng):
    if kind == "uniform":
        return rng.uniform(-3, 3, n)
    if kind == "positive":
        return rng.uniform(0.2, 1.0, n)
    if kind == "few":                      # many ties
        return rng.integers(-50, 50, n) * 0.37 * eb
    if kind == "near_zero":                # some values below 2^-6 eb, zeros of both signs
        v = rng.uniform(-4, 4, n) * eb
        v[::97] *= 1e-4
        v[5::311] = 0.0
        v[7::311] = -0.0
        v[9::311] = 1e-42
        return v
    if kind == "aside":                    # more of them than are kept aside
        return rng.uniform(-1, 1, n) * eb * 2.0 ** -8
    if kind == "edges":                    # around bin edges and the smallest magnitude with a bit
        k = rng.integers(-40, 40, n)
        v = (k * np.float32(eb)).astype(np.float32)
        v = np.nextafter(v, np.where(rng.random(n) < 0.5, -np.inf, np.inf).astype(np.float32))
        m = 2.0 ** (np.floor(np.log2(eb)) - 6)
        v[::13] = np.nextafter(np.float32(m), np.float32(0))
        v[1::13] = m
        v[2::13] = -m
        return v
    if kind == "huge":                     # beyond 2^30 eb
        return np.r_[rng.uniform(-1, 1, n - 2) * 1e3, 1e30, -np.inf]
    if kind == "many_bins":                # more than 2^22 bins
        return rng.uniform(0, 1, n) * eb * 2.0 ** 24
    raise ValueError(kind)


@pytest.mark.parametrize("n", [1, 2, 33, 2047, 2048, 2049, 70001])
@pytest.mark.parametrize("kind", ["uniform", "positive", "few", "near_zero", "aside", "edges", "huge", "many_bins"])
@pytest.mark.parametrize("eb", [1e-3, 2.0 ** -10, 7.7])
def test_positions(T, kind, n, eb):
    import torch
    rng = np.random.default_rng(n + 7)
    v = _values(kind, max(n, 4), eb, rng)[:n].astype(np.float32)
    ext = rng.random(n) < 0.7
    ext[0] = True
    idx = np.where(ext, np.cumsum(ext) - 1, 0xffffffff).astype(np.uint32)
    pairs = torch.from_numpy(np.stack([_codes(v), idx], 1).astype(np.uint32).view(np.int32)).cuda()
    sp = torch.full((int(ext.sum()),), -1, dtype=torch.int32, device="cuda")
    ctx = T.Context()
    for _ in range(2):                     # the second call finds the bits cleared
        sp.fill_(-1)
        torch.cuda.synchronize()
        rc = T.lib().szp_b200_rank_pairs_dev(ctx.ptr, ctypes.c_void_p(pairs.data_ptr()), n, sp.numel(),
                                             ctypes.c_float(eb), ctypes.c_void_p(sp.data_ptr()))
        assert rc == 0, T.last_error()
        assert (sp.cpu().numpy() == _expect(v, eb)[ext]).all()
    ctx.close()


@pytest.mark.parametrize("dims", [(511, 512), (512, 513), (64, 65, 66), (700, 601)])
@pytest.mark.parametrize("kind,eb", [("noise", 1e-2), ("noise", 1e-4), ("bumps", 1e-3), ("zero", 1e-2),
                                     ("huge", 1e-3), ("aside", 10.0)])
def test_sort_stream(T, ora, kind, eb, dims):
    """Fields on either side of the size from which the encoder sets the bits."""
    import torch
    d = synth.small_field(dims, seed=2, kind="bumps" if kind == "bumps" else "noise")
    if kind == "zero":
        d[::2] *= np.float32(1e-4)
    if kind == "huge":
        d.reshape(-1)[1000] = np.float32(1e9)
        d.reshape(-1)[70000] = -np.float32(1e9)
    if kind == "aside":
        d *= np.float32(0.01)
    ctx = T.Context()
    x = torch.from_numpy(d.reshape(-1).copy()).cuda()
    cp = ora.sort_cp(ora.find_cp(d, eb), d)
    want_t = ora.encode_topo(d, eb, 64, ora.mark_types(cp, dims))
    want_s = ora.encode_ints(ora.extract_sp(cp), 64)
    for _ in range(2):
        topo, sort, _, sz = ctx.compress(x, dims, eb, 64)
        assert topo[:sz.topo_bytes].cpu().numpy().tobytes() == want_t
        assert sort[:sz.sort_bytes].cpu().numpy().tobytes() == want_s
    # the host-buffer form, whose field arrives in parts from 2^24 values on
    ht, hs = np.zeros(topo.numel(), np.uint8), np.zeros(sort.numel(), np.uint8)
    sz = ctx.compress_host(d, eb, 64, ht, hs)
    assert ht[:sz.topo_bytes].tobytes() == want_t and hs[:sz.sort_bytes].tobytes() == want_s
    ctx.close()
