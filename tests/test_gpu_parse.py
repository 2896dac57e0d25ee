"""Block offsets parsed on the device from the stream bytes alone.

A parsed decode must equal the decode with the block index that the compressor
wrote.  Sizes put the stream's end on either side of the parser's 8 KB
segments, its 32-segment groups (256 KB) and its second group level (8 MB);
blockSizes reach every group size and both composition paths; the constant
field has blocks of 21 bytes whose bit count bytes are all zero, so that walks
from wrong entries survive and every entry's function is needed."""
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


def _field(kind, dims, seed):
    if kind == "constant":
        return np.full(dims, 0.25, dtype=np.float32)
    if kind == "steps":
        # constant rows, a jump between rows: blocks of two lengths
        return np.repeat(np.arange(dims[0], dtype=np.float32) % 3, dims[1]).reshape(dims)
    return synth.small_field(dims, seed=seed, kind="noise")


def _bits(t):
    import torch
    return t.view(torch.int32)


@pytest.mark.parametrize("kind", ["noise", "constant", "steps"])
@pytest.mark.parametrize("dims,B", [((1, 5), 2), ((3, 3), 1), ((40, 41), 1), ((64, 65), 2), ((300, 301), 7),
                                    ((75, 64), 64), ((77, 65), 64), ((450, 449), 64), ((460, 471), 64),
                                    ((2300, 2200), 64), ((500, 333), 128), ((900, 1011), 256), ((900, 1011), 257)])
def test_parsed_decode_equals_indexed_decode(T, kind, dims, B):
    import torch
    d = _field(kind, dims, 7)
    x = torch.from_numpy(d.reshape(-1).copy()).cuda()
    ctx = T.Context()
    topo, sort, idx, sz = ctx.compress(x, dims, 1e-2, B)
    t1 = torch.empty(d.size, dtype=torch.uint8, device="cuda")
    t2 = torch.empty_like(t1)
    a = ctx.decompress(topo, sz.topo_bytes, sort, sz.sort_bytes, idx, dims, 1e-2, B, postprocess=1, types=t1)
    # the parsed copy starts at an odd address; 4-byte aligned above blockSize 256
    shift = 4 if B > 256 else 3
    tp = torch.zeros(sz.topo_bytes + shift, dtype=torch.uint8, device="cuda")
    tp[shift:] = topo[:sz.topo_bytes]
    b = ctx.decompress(tp[shift:], sz.topo_bytes, sort, sz.sort_bytes, None, dims, 1e-2, B, postprocess=1, types=t2)
    assert torch.equal(_bits(a), _bits(b)) and torch.equal(t1, t2)
    # one byte short, and a bit count byte above 32, are errors
    with pytest.raises(T.ToposzpError):
        ctx.decompress(topo, sz.topo_bytes - 1, sort, sz.sort_bytes, None, dims, 1e-2, B, postprocess=0)
    if B > 1:
        nb = idx.numel() // 2
        for k in (0, (nb - 1) // 2):
            bad = topo.clone()
            bad[8 + int(idx[k]) + 4] = 33
            with pytest.raises(T.ToposzpError):
                ctx.decompress(bad, sz.topo_bytes, sort, sz.sort_bytes, None, dims, 1e-2, B, postprocess=0)
    ctx.close()


@pytest.mark.parametrize("n,B", [(1, 64), (65, 64), (70001, 64), (3000017, 64), (400009, 1025), (33000, 2)])
def test_plain_parse(T, n, B):
    import torch
    x = synth.plain_field(n, seed=5, kind="wave")
    d = torch.from_numpy(x).cuda()
    ctx = T.Context()
    s = torch.zeros(T.lib().szp_b200_plain_bound(n, B, 0, 0), dtype=torch.uint8, device="cuda")
    out = torch.empty_like(d)
    k = ctx.plain_compress(d, 1e-3, B, s)
    ctx.plain_decompress(s, k, n, 1e-3, B, out)
    eb = np.float32(1e-3)
    q = (x.astype(np.float64) * (1.0 / np.float64(eb))).astype(np.int32)
    host = T.plain_decompress(s[:k].cpu().numpy().tobytes(), n, 1e-3, B)   # walked on the host
    assert (out.cpu().numpy().view(np.int32) == host.view(np.int32)).all()
    assert np.abs(host.astype(np.float64) - q * np.float64(eb)).max() <= np.abs(q).max() * float(eb) * 2.0 ** -23
    ctx.close()


@pytest.mark.parametrize("dims,B", [((70, 90), 16), ((300, 500), 64), ((50, 60), 7)])
def test_container_chunks(T, dims, B):
    """Chunk tables confirmed by the whole parse, and one whose second chunk
    starts ten bytes late, which is walked chunk by chunk.  (The reference's
    rule takes the first thread count that walks, which on some streams is a
    smaller one than the writer's; it is not on these.)"""
    import torch
    d = synth.small_field(dims, seed=4, kind="noise")
    ctx = T.Context()
    x = torch.from_numpy(d.reshape(-1).copy()).cuda()
    topo, sort, _, sz = ctx.compress(x, dims, 1e-2, B, index=False)
    ref = ctx.decompress(topo, sz.topo_bytes, sort, sz.sort_bytes, None, dims, 1e-2, B, postprocess=1)
    for threads in (1, 2, 5, 8, 128):
        cont = ctx.to_container(topo, sz.topo_bytes, sort, sz.sort_bytes, dims, B, sz.extrema_count, threads=threads)
        out = ctx.decompress_container(cont, dims, 1e-2, B, postprocess=1)
        assert torch.equal(_bits(out), _bits(ref)), threads
    c = ctx.to_container(topo, sz.topo_bytes, sort, sz.sort_bytes, dims, B, sz.extrema_count,
                         threads=2).cpu().numpy().tobytes()
    ts = int(np.frombuffer(c[-16:-8], dtype=np.uint64)[0])
    cut = int(np.frombuffer(c[8:16], dtype=np.uint64)[0])
    late = (c[:8] + np.uint64(cut + 10).tobytes() + c[16:16 + cut] + b"\xff" * 10 + c[16 + cut:-16] +
            np.uint64(ts + 10).tobytes() + c[-8:])
    out = ctx.decompress_container(torch.from_numpy(np.frombuffer(late, dtype=np.uint8).copy()).cuda(), dims, 1e-2, B,
                                   postprocess=1)
    assert torch.equal(_bits(out), _bits(ref))
    ctx.close()
