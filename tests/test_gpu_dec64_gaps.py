"""Streams read with the caller's block index whose blocks do not follow one
another directly: bytes that belong to no block between two of them, within
what a tile of 32 blocks of the largest length can hold.  Reads as the stream
without them; a gap beyond that is reported."""
import numpy as np
import pytest

import synth

pytestmark = pytest.mark.gpu

ROOM = 32 * 289 + 64 - 48      # bytes of a tile with type tags (blockSize 64)


@pytest.fixture(scope="module")
def T():
    import torch
    import toposzp_b200
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    toposzp_b200.lib()
    return toposzp_b200


def _spread(payload, offs, at, gap):
    """The payload with gap bytes of 0xff before block `at`, and its offsets."""
    o = offs.copy()
    cut = int(o[at])
    o[at:] += gap
    return np.concatenate([payload[:cut], np.full(gap, 0xff, np.uint8), payload[cut:]]), o


def _case(T, dims, eb, at, gap, sort_at, sort_gap):
    import torch
    d = synth.small_field(dims, seed=5, kind="noise")
    ctx = T.Context()
    x = torch.from_numpy(d.reshape(-1).copy()).cuda()
    topo, sort, idx, sz = ctx.compress(x, dims, eb, 64)
    want = ctx.decompress(topo, sz.topo_bytes, sort, sz.sort_bytes, idx, dims, eb, 64, postprocess=1)
    nb, nbs = -(-d.size // 64), -(-sz.extrema_count // 64)
    offs = idx.cpu().numpy()
    t, ot = _spread(topo[8:sz.topo_bytes].cpu().numpy(), offs[:nb], at, gap)
    s, os_ = _spread(sort[8:sz.sort_bytes].cpu().numpy(), offs[nb:nb + nbs], sort_at, sort_gap)
    pad = np.zeros(8, np.uint8)
    tt, ss = (torch.from_numpy(np.concatenate([pad, v])).cuda() for v in (t, s))
    ii = torch.from_numpy(np.concatenate([ot, os_])).cuda()
    try:
        got = ctx.decompress(tt, tt.numel(), ss, ss.numel(), ii, dims, eb, 64, postprocess=1)
        return torch.equal(got.view(torch.int32), want.view(torch.int32))
    finally:
        ctx.close()


@pytest.mark.parametrize("at,gap", [(1, 3), (8, 2000), (8, 4700), (15, 6000), (17, 6000), (40, 6000), (63, 6001)])
def test_gap_between_blocks(T, at, gap):
    # a block of this field takes at most 100 bytes
    assert gap + 32 * 100 <= ROOM
    assert _case(T, (64, 64), 1e-2, at, gap, 1, gap % 1000)


def test_gap_beyond_a_tile(T):
    with pytest.raises(T.ToposzpError, match="malformed"):
        _case(T, (64, 64), 1e-2, 8, ROOM + 1, 1, 0)
