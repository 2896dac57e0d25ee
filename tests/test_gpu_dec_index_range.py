"""A block index with offsets at the top of the 64-bit range, where offset + 4
is small again: every decoder reports it.  (The kernels compare without that
sum, so nothing is read for such a block.)"""
import numpy as np
import pytest

import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("low", [1, 2, 3, 4])
@pytest.mark.parametrize("first,count", [(8, None), (8, 1), (4, 2), (0, None)])   # a share of the blocks before; blocks
@pytest.mark.parametrize("B", [64, 32, 16, 257])
def test_offsets_near_the_end_of_the_range(B, first, count, low):
    import torch
    import toposzp_b200 as T
    dims, eb = (64, 64), 1e-2
    d = synth.small_field(dims, seed=5, kind="noise")
    ctx = T.Context()
    x = torch.from_numpy(d.reshape(-1).copy()).cuda()
    topo, _, idx, sz = ctx.compress(x, dims, eb, B)
    want = ctx.decompress(topo, sz.topo_bytes, None, 0, idx, dims, eb, B, postprocess=0)
    # from inside the first tile on, whose end is then at the top of the range too
    nb = -(-d.size // B)
    at = nb // first if first else 0
    bad = idx.clone()
    bad[at:nb if count is None else at + count] = -low      # 2^64 - low
    with pytest.raises(T.ToposzpError, match="malformed"):
        ctx.decompress(topo, sz.topo_bytes, None, 0, bad, dims, eb, B, postprocess=0)
    got = ctx.decompress(topo, sz.topo_bytes, None, 0, idx, dims, eb, B, postprocess=0)
    assert np.array_equal(got.cpu().numpy().view(np.int32), want.cpu().numpy().view(np.int32))
    ctx.close()
