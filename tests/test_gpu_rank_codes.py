"""Sort positions of fields whose values the bitmap does not cover, ranked in
buckets from the encoder's codes: around the number of values that are kept
aside, values beyond 2^30 eb, more bins than the table has, and fields that lie
near zero altogether, against the oracle; and the host-buffer form, whose field
arrives in parts, against the device form."""
import numpy as np
import pytest

import synth

pytestmark = pytest.mark.gpu

DIMS = [(700, 601), (61, 70, 99)]      # from 2^18 values on the encoder sets the bits


@pytest.fixture(scope="module")
def T():
    import torch
    import toposzp_b200
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    toposzp_b200.lib()
    return toposzp_b200


def _aside(dims, m, eb, rng):
    """Noise in [1, 2] with m isolated minima whose magnitudes are below eb / 64:
    both signs, zeros of both signs, ties."""
    d = rng.uniform(1, 2, dims).astype(np.float32)
    inner = tuple(slice(1, -1, 2) for _ in dims)
    v = d[inner].copy()
    at = rng.permutation(v.size)[:m]
    t = (rng.uniform(-1, 1, m) * eb / 128).astype(np.float32)
    t[::5] = t[0]
    t[1::7], t[2::7] = 0.0, -0.0
    v.reshape(-1)[at] = t
    d[inner] = v
    return d


def _check(T, ora, d, eb):
    import torch
    cp = ora.sort_cp(ora.find_cp(d, eb), d)
    topo = ora.encode_topo(d, eb, 64, ora.mark_types(cp, d.shape))
    sort = ora.encode_ints(ora.extract_sp(cp), 64)
    ctx = T.Context()
    x = torch.from_numpy(d.reshape(-1).copy()).cuda()
    for _ in range(2):                 # the second call finds the bits cleared
        t, s, _, sz = ctx.compress(x, d.shape, eb, 64)
        assert sz.cp_count == len(cp)
        assert t[:sz.topo_bytes].cpu().numpy().tobytes() == topo
        assert s[:sz.sort_bytes].cpu().numpy().tobytes() == sort
    # and the next field, whose values have bits
    y = synth.small_field((600, 500), seed=9, kind="noise")
    cp = ora.sort_cp(ora.find_cp(y, 1e-3), y)
    _, s, _, sz = ctx.compress(torch.from_numpy(y.reshape(-1).copy()).cuda(), y.shape, 1e-3, 64)
    assert s[:sz.sort_bytes].cpu().numpy().tobytes() == ora.encode_ints(ora.extract_sp(cp), 64)
    ctx.close()


@pytest.mark.parametrize("dims", DIMS, ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("m", [1, 4095, 4096, 4097, 12000])
def test_values_aside(T, ora, dims, m):
    eb = 1e-2
    _check(T, ora, _aside(dims, m, eb, np.random.default_rng(m)), eb)


@pytest.mark.parametrize("dims", DIMS, ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("kind", ["near zero", "beyond", "one beyond", "bins", "zeros"])
def test_values_without_bits(T, ora, dims, kind):
    rng = np.random.default_rng(3)
    d = rng.standard_normal(dims).astype(np.float32)
    eb = 1e-2
    if kind == "near zero":
        d *= np.float32(1e-6)
    elif kind == "beyond":
        d *= np.float32(1e9)
    elif kind == "one beyond":
        d.reshape(-1)[d.size // 2 + 3] = np.float32(3e7)
        d.reshape(-1)[d.size // 3 + 3] = np.float32(-3e7)
    elif kind == "bins":
        eb = 1e-6
    else:
        d = rng.choice(np.array([0.0, -0.0, 1e-40, -1e-40], np.float32), dims)
    _check(T, ora, d, eb)


def test_host_form_in_parts(T):
    """2^24 values and more: the field is encoded part by part as it arrives."""
    import torch
    dims, eb = (4100, 4100), 10.0
    d = (synth.small_field((410, 410), seed=1, kind="noise").repeat(10, 0).repeat(10, 1) +
         np.random.default_rng(1).standard_normal(dims) * 1e-3).astype(np.float32)
    ctx = T.Context()
    t, s, _, sz = ctx.compress(torch.from_numpy(d.reshape(-1).copy()).cuda(), dims, eb, 64)
    assert sz.extrema_count > 4096
    ht, hs = np.zeros(t.numel(), np.uint8), np.zeros(s.numel(), np.uint8)
    hz = ctx.compress_host(d, eb, 64, ht, hs)
    assert (hz.topo_bytes, hz.sort_bytes, hz.cp_count) == (sz.topo_bytes, sz.sort_bytes, sz.cp_count)
    assert ht[:sz.topo_bytes].tobytes() == t[:sz.topo_bytes].cpu().numpy().tobytes()
    assert hs[:sz.sort_bytes].tobytes() == s[:sz.sort_bytes].cpu().numpy().tobytes()
    ctx.close()
