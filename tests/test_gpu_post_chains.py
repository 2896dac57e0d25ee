"""Post-processing of a checkerboard, nearly every point of which is an extremum
that waits for its neighbours: worklists of many times the points that are in
flight at once, and of about as many, against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(60, 70), (300, 320), (860, 880), (20, 60, 70)])
def test_checkerboard(ora, dims):
    import torch
    import toposzp_b200 as T
    eb, B = 1e-2, 64
    rng = np.random.default_rng(sum(dims))
    d = ((np.indices(dims).sum(0) % 2) * 2.0 - 1.0 + 0.05 * rng.standard_normal(dims)).astype(np.float32)
    ctx = T.Context()
    topo, sort, _, sz = ctx.compress(torch.from_numpy(d.reshape(-1)).cuda(), dims, eb, B, index=False)
    got = ctx.decompress(topo, sz.topo_bytes, sort, sz.sort_bytes, None, dims, eb, B, postprocess=1).cpu().numpy()
    cp = ora.sort_cp(ora.find_cp(d, eb), d)
    raw, fn, _ = ora.decode_topo(topo[:sz.topo_bytes].cpu().numpy().tobytes(), d.size, eb, B)
    want, _ = ora.post(raw.reshape(dims), raw.reshape(dims), fn.reshape(dims), ora.extract_sp(cp), eb)
    assert (got.view(np.int32) == want.reshape(-1).view(np.int32)).all()
    ctx.close()
