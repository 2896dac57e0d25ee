"""An .SZp container whose streams are one chunk each that starts above payload
offset 0: the table entry says where, and the bytes before it belong to no
block.  Reads as the container without them."""
import struct

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


def _u64(v):
    return struct.pack("<Q", v)


@pytest.mark.parametrize("skip_topo,skip_sort", [(0, 0), (1, 0), (0, 3), (5, 16), (40, 7)])
@pytest.mark.parametrize("B", [64, 16])
def test_one_chunk_behind_an_offset(T, B, skip_topo, skip_sort):
    import torch
    dims, eb = (60, 90), 1e-2
    d = synth.small_field(dims, seed=11, kind="noise")
    ctx = T.Context()
    x = torch.from_numpy(d.reshape(-1).copy()).cuda()
    topo, sort, _, sz = ctx.compress(x, dims, eb, B, index=False)
    cont = ctx.to_container(topo, sz.topo_bytes, sort, sz.sort_bytes, dims, B, sz.extrema_count, threads=1)
    blob = cont.cpu().numpy().tobytes()
    ts, ss = struct.unpack("<QQ", blob[-16:])
    # topology: offset, payload; sort positions: extrema, offset, payload
    t, s = blob[:ts], blob[ts:ts + ss]
    new_t = _u64(skip_topo) + b"\xff" * skip_topo + t[8:]
    new_s = s[:8] + _u64(skip_sort) + b"\xff" * skip_sort + s[16:]
    moved = np.frombuffer(new_t + new_s + _u64(len(new_t)) + _u64(len(new_s)), dtype=np.uint8)
    want = ctx.decompress_container(cont, dims, eb, B, postprocess=1)
    got = ctx.decompress_container(torch.from_numpy(moved.copy()).cuda(), dims, eb, B, postprocess=1)
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    ctx.close()
