"""The blockSize-64 topology encoder at the edges of its tiles (2048 elements),
octets and rows, on values whose comparisons go wrong when a sign of zero, a
NaN, an infinity or a denormal difference is mistaken, against the oracle."""
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


def _field(kind, dims, rng):
    n = int(np.prod(dims))
    tiny = np.float32(1e-45)
    if kind == "zeros":
        v = rng.choice(np.array([0.0, -0.0, 1.0, -1.0], np.float32), n)
    elif kind == "denormal":
        v = (rng.integers(-3, 4, n) * tiny).astype(np.float32)
    elif kind == "special":
        v = rng.choice(np.array([0.0, -0.0, 1.0, -1.0, np.inf, -np.inf, np.nan, tiny, -tiny, 3e38, -3e38],
                                np.float32), n)
    elif kind == "steps":      # wide deltas: more than one full byte, bit counts to 31
        v = (rng.standard_normal(n) * 10.0 ** rng.integers(-3, 7, n)).astype(np.float32)
    else:
        v = synth.small_field(dims, seed=4, kind="noise").reshape(-1)
    return v.astype(np.float32).reshape(dims)


@pytest.mark.parametrize("kind", ["zeros", "denormal", "special", "steps", "noise"])
@pytest.mark.parametrize("dims", [(3, 3), (32, 64), (31, 66), (33, 62), (64, 65), (2, 1024), (16, 256), (5, 2047),
                                  (4, 8, 64), (5, 9, 47), (3, 3, 2048), (6, 7, 9), (3, 4, 8), (9, 16, 100)])
def test_topology_stream(T, ora, kind, dims):
    import torch
    d = _field(kind, dims, np.random.default_rng(sum(dims)))
    eb = 1e-2
    x = torch.from_numpy(d.reshape(-1).copy()).cuda()
    ctx = T.Context()
    topo, _, idx, sz = ctx.compress(x, dims, eb, 64)
    cp = ora.find_cp(d, eb)
    want = ora.encode_topo(d, eb, 64, ora.mark_types(cp, dims))
    assert sz.cp_count == len(cp)
    assert topo[:sz.topo_bytes].cpu().numpy().tobytes() == want
    nb = -(-d.size // 64)
    out = torch.empty(d.size, dtype=torch.float32, device="cuda")
    ref = ctx.decompress(topo, sz.topo_bytes, None, 0, None, dims, eb, 64, postprocess=0)
    ctx.decompress(topo, sz.topo_bytes, None, 0, idx, dims, eb, 64, postprocess=0, out=out)
    assert idx.numel() == 2 * nb and torch.equal(out.view(torch.int32), ref.view(torch.int32))
    ctx.close()
