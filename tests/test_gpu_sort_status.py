"""A sort-position stream that its decoder cannot read (a bit count above 32, or
cut off), with the caller's block index, under post-processing: the call
reports it, whatever lies in the workspace, and the next call is unaffected."""
import numpy as np
import pytest

import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("B", [64, 32])
@pytest.mark.parametrize("dims,post", [((64, 70), 1), ((20, 24, 28), 1), ((20, 24, 28), 2), ((300, 300), 1)])
@pytest.mark.parametrize("what", ["bit count", "cut"])
def test_malformed_sort_positions(B, dims, post, what):
    import torch
    import toposzp_b200 as T
    eb = 1e-2
    d = synth.small_field(dims, seed=5, kind="noise")
    ctx = T.Context()
    x = torch.from_numpy(d.reshape(-1).copy()).cuda()
    topo, sort, idx, sz = ctx.compress(x, dims, eb, B)
    want = ctx.decompress(topo, sz.topo_bytes, sort, sz.sort_bytes, idx, dims, eb, B, postprocess=post)
    nb, nbs = -(-d.size // B), -(-sz.extrema_count // B)
    assert nbs > 2
    bad, size = sort.clone(), sz.sort_bytes
    if what == "cut":
        size = 8 + int(idx[nb + nbs - 1]) + 3
    else:
        bad[8 + int(idx[nb + nbs // 2]) + 4] = 33
    with pytest.raises(T.ToposzpError, match="malformed sort-position stream"):
        ctx.decompress(topo, sz.topo_bytes, bad, size, idx, dims, eb, B, postprocess=post)
    got = ctx.decompress(topo, sz.topo_bytes, sort, sz.sort_bytes, idx, dims, eb, B, postprocess=post)
    assert np.array_equal(got.cpu().numpy().view(np.int32), want.cpu().numpy().view(np.int32))
    ctx.close()
