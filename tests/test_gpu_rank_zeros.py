"""Sort positions of exact zeros (masked, sparse and integer fields): many of
them, as extrema, saddles or both, with and without other values next to zero,
and with bounds for which eb * (1 / eb) is 1 and just below it, so that a zero
lies in bin 1 or in bin 0."""
import ctypes

import numpy as np
import pytest

from test_gpu_rank import _codes, _expect

pytestmark = pytest.mark.gpu

EBS = [1e-2, 49.0 / 4096, 0.3, 49.0]


@pytest.fixture(scope="module")
def T():
    import torch
    import toposzp_b200
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    toposzp_b200.lib()
    return toposzp_b200


def test_bounds_are_of_both_kinds():
    one = [float(np.float32(e)) * (1.0 / float(np.float32(e))) for e in EBS]
    assert any(v == 1.0 for v in one) and any(v < 1.0 for v in one)


def _field(kind, dims, rng):
    if kind == "integers":
        d = np.floor(rng.standard_normal(dims) * 3)
    elif kind == "sparse":
        d = np.where(rng.random(dims) < 0.2, rng.standard_normal(dims), 0.0)
    else:
        # isolated zeros, and with "aside" values below eb / 64, on either side of their neighbours
        d = rng.uniform(1, 2, dims) * rng.choice([-1.0, 1.0], (dims[0],) + (1,) * (len(dims) - 1))
        inner = tuple(slice(1, -1, 2) for _ in dims)
        v = np.where(rng.random(d[inner].shape) < 0.3, 0.0, d[inner])
        if kind == "aside":
            v = np.where(rng.random(v.shape) < 0.01, rng.uniform(-1e-5, 1e-5, v.shape), v)
        d[inner] = v * rng.choice([-1.0, 1.0], v.shape)     # zeros of both signs
    return d.astype(np.float32)


@pytest.mark.parametrize("dims", [(300, 400), (40, 50, 61)], ids=lambda d: "x".join(map(str, d)))
@pytest.mark.parametrize("kind", ["integers", "sparse", "isolated", "aside"])
@pytest.mark.parametrize("eb", EBS)
def test_fields(T, ora, kind, dims, eb):
    import torch
    d = _field(kind, dims, np.random.default_rng(len(kind)))
    eb = float(np.float32(eb))
    cp = ora.sort_cp(ora.find_cp(d, eb), d)
    want_t = ora.encode_topo(d, eb, 64, ora.mark_types(cp, dims))
    want_s = ora.encode_ints(ora.extract_sp(cp), 64)
    ctx = T.Context()
    x = torch.from_numpy(d.reshape(-1).copy()).cuda()
    for _ in range(2):
        t, s, _, sz = ctx.compress(x, dims, eb, 64)
        assert t[:sz.topo_bytes].cpu().numpy().tobytes() == want_t
        assert s[:sz.sort_bytes].cpu().numpy().tobytes() == want_s
    ctx.close()


@pytest.mark.parametrize("eb", EBS)
@pytest.mark.parametrize("share,aside", [(0.5, 0), (0.001, 0), (0.5, 3000), (0.5, 4095), (0.5, 4096)])
def test_pairs(T, eb, share, aside):
    import torch
    rng = np.random.default_rng(aside + 1)
    n = 70001
    v = rng.uniform(-4, 4, n) * eb
    v[rng.random(n) < share] = 0.0
    at = rng.permutation(n)[:aside]
    v[at] = rng.uniform(-1, 1, aside) * eb * 2.0 ** -9
    v = v.astype(np.float32)
    ext = rng.random(n) < 0.7
    ext[0] = True
    idx = np.where(ext, np.cumsum(ext) - 1, 0xffffffff).astype(np.uint32)
    pairs = torch.from_numpy(np.stack([_codes(v), idx], 1).astype(np.uint32).view(np.int32)).cuda()
    ctx = T.Context()
    for _ in range(2):
        sp = torch.full((int(ext.sum()),), -1, dtype=torch.int32, device="cuda")
        torch.cuda.synchronize()
        rc = T.lib().szp_b200_rank_pairs_dev(ctx.ptr, ctypes.c_void_p(pairs.data_ptr()), n, sp.numel(),
                                             ctypes.c_float(eb), ctypes.c_void_p(sp.data_ptr()))
        assert rc == 0, T.last_error()
        assert (sp.cpu().numpy() == _expect(v, eb)[ext]).all()
    ctx.close()
