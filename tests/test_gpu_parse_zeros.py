"""Streams whose every byte is a valid bit count (blocks of one value, most of
all zeros): the walks of the parser's guess never meet, and are given up for
large blocks.  Whole fields of one value, with a stretch of noise, and noise
with stretches of zeros; plain and topology streams without an index."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def T():
    import torch
    import toposzp_b200
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    toposzp_b200.lib()
    return toposzp_b200


def _values(kind, n, rng):
    if kind == "zeros":
        return np.zeros(n, np.float32)
    if kind == "value":
        return np.full(n, 7.25, np.float32)
    v = rng.standard_normal(n).astype(np.float32)
    keep = np.zeros(n, bool)
    if kind == "one stretch":
        keep[n // 3:n // 3 + 5000] = True
    else:
        for s in range(0, n, 40000):
            keep[s:s + 20000] = True
    return np.where(keep, v, np.float32(0))


KINDS = ["zeros", "value", "one stretch", "stretches"]


@pytest.mark.parametrize("B", [2, 16, 64, 128, 200, 256, 257, 600])
@pytest.mark.parametrize("kind", KINDS)
def test_plain(T, kind, B):
    import torch
    n = 900001 if B > 16 else 120001
    x = _values(kind, n, np.random.default_rng(B))
    ctx = T.Context()
    d = torch.from_numpy(x).cuda()
    s = torch.zeros(T.lib().szp_b200_plain_bound(n, B, 0, 0), dtype=torch.uint8, device="cuda")
    out = torch.empty_like(d)
    k = ctx.plain_compress(d, 1e-3, B, s)
    ctx.plain_decompress(s, k, n, 1e-3, B, out)
    host = T.plain_decompress(s[:k].cpu().numpy().tobytes(), n, 1e-3, B)   # walked on the host
    assert (out.cpu().numpy().view(np.int32) == host.view(np.int32)).all()
    ctx.close()


@pytest.mark.parametrize("B", [16, 64, 128, 256])
@pytest.mark.parametrize("kind", KINDS)
def test_topology(T, kind, B):
    import torch
    dims = (900, 1000)
    x = _values(kind, 900000, np.random.default_rng(B)).reshape(dims)
    ctx = T.Context()
    topo, sort, idx, sz = ctx.compress(torch.from_numpy(x.reshape(-1)).cuda(), dims, 1e-2, B)
    want = ctx.decompress(topo, sz.topo_bytes, sort, sz.sort_bytes, idx, dims, 1e-2, B, postprocess=1)
    got = ctx.decompress(topo, sz.topo_bytes, sort, sz.sort_bytes, None, dims, 1e-2, B, postprocess=1)
    assert torch.equal(got.view(torch.int32), want.view(torch.int32))
    ctx.close()
