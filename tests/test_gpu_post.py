"""Post-processing at the edges of its bitmap words (rows around 32 and 64
points), on both sides of the size up to which a pass is one launch, with the
types from the block decoder and from the caller, and with an original field of
its own, against the oracle (equal bits)."""
import numpy as np
import pytest

import synth

pytestmark = pytest.mark.gpu

SHAPES = [(3, 31), (5, 32), (9, 33), (64, 34), (40, 63), (33, 64), (31, 65), (17, 97),
          (3, 3, 31), (4, 5, 32), (5, 9, 33), (6, 11, 34), (9, 7, 63), (8, 8, 64), (7, 5, 65),
          # more extrema than one cooperative launch holds
          (700, 901), (37, 130, 131)]


@pytest.fixture(scope="module")
def T():
    import torch
    import toposzp_b200
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    toposzp_b200.lib()
    return toposzp_b200


def _same(a, b):
    return np.array_equal(np.asarray(a, np.float32).reshape(-1).view(np.int32),
                          np.asarray(b, np.float32).reshape(-1).view(np.int32))


@pytest.mark.parametrize("B", [64, 32])
@pytest.mark.parametrize("dims", SHAPES, ids=lambda d: "x".join(map(str, d)))
def test_passes(T, ora, dims, B):
    import torch
    eb = 0.02
    d = synth.small_field(dims, seed=sum(dims), kind="noise").astype(np.float32)
    cp = ora.sort_cp(ora.find_cp(d, eb), d)
    raw, fn, _ = ora.decode_topo(ora.encode_topo(d, eb, B, ora.mark_types(cp, dims)), d.size, eb, B)
    sp = ora.extract_sp(cp)
    x = torch.from_numpy(d.reshape(-1).copy()).cuda()
    ctx = T.Context()
    topo, sort, idx, sz = ctx.compress(x, dims, eb, B)
    # an original that differs from the decoded field by a bound or less
    noise = np.random.default_rng(7).uniform(-eb, eb, d.size).astype(np.float32)
    other = (raw.reshape(-1) + noise).astype(np.float32)
    for mode in range(len(dims)):
        got = ctx.decompress(topo, sz.topo_bytes, sort, sz.sort_bytes, idx, dims, eb, B, postprocess=mode)
        ref = raw
        if mode:
            ref, _ = ora.post(raw.reshape(dims), raw.reshape(dims), fn.reshape(dims), sp, eb, axis_stencil=mode == 2)
        assert _same(got.cpu().numpy(), ref), mode
        if mode:
            f = torch.from_numpy(raw.reshape(-1).copy()).cuda()
            o = torch.from_numpy(other.copy()).cuda()
            t = torch.from_numpy(fn.reshape(-1).copy()).cuda()
            s = torch.from_numpy(sp.copy()).cuda() if len(sp) else None
            ctx.postprocess(f, o, t, s, dims, eb, axis_stencil=mode == 2)
            ref, _ = ora.post(raw.reshape(dims), other.reshape(dims), fn.reshape(dims), sp, eb,
                              axis_stencil=mode == 2)
            assert _same(f.cpu().numpy(), ref), ("original", mode)
    ctx.close()
