"""The blockSize-64 encoder of quantized fields, integers and integers with
types, at the edges of its tiles (2048 elements) and blocks, from aligned and
unaligned inputs, against the oracle (equal bytes)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 2, 63, 64, 65, 2047, 2048, 2049, 2111, 2112, 4096, 4097, 65 * 2048 - 63]


@pytest.fixture(scope="module")
def T(ora):
    import torch
    import toposzp_b200
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    toposzp_b200.lib()
    return toposzp_b200


def _floats(kind, n, rng):
    if kind == "smooth":
        return np.cumsum(rng.standard_normal(n) * 0.02).astype(np.float32)
    if kind == "steps":        # bit counts to 31
        return (rng.standard_normal(n) * 10.0 ** rng.integers(-3, 7, n)).astype(np.float32)
    return rng.choice(np.array([0.0, -0.0, 1.0, np.inf, -np.inf, np.nan, 1e-45, -3e38], np.float32), n)


@pytest.mark.parametrize("kind", ["smooth", "steps", "special"])
@pytest.mark.parametrize("n", SIZES)
def test_plain_stream(T, ora, n, kind):
    import torch
    eb = 1e-2
    x = _floats(kind, n, np.random.default_rng(n))
    want = ora.plain_compress(x, eb, 64)
    ctx = T.Context()
    for off in (0, 1):
        d = torch.zeros(n + off, dtype=torch.float32, device="cuda")
        d[off:] = torch.from_numpy(x).cuda()
        out = torch.full((len(want) + 4096 + 6 * n,), 0xAB, dtype=torch.uint8, device="cuda")
        ln = ctx.plain_compress(d[off:], eb, 64, out)
        assert ln == len(want) and out[:ln].cpu().numpy().tobytes() == want, off
    ctx.close()


@pytest.mark.parametrize("span", [3, 1 << 12, 1 << 30])
@pytest.mark.parametrize("n", SIZES)
def test_sort_position_stream(T, ora, n, span):
    rng = np.random.default_rng(n + span)
    v = rng.integers(-span, span, n).astype(np.int32)
    cps = np.zeros(n, dtype=T.CP2_DT)
    cps["type"] = rng.integers(1, 3, n)
    cps["sort_position"] = v
    assert T.compress_sort_positions(cps, 64).endswith(ora.encode_ints(v, 64))


@pytest.mark.parametrize("dims", [(8, 16, 16), (3, 3, 228), (7, 17, 17), (9, 15, 31), (4, 32, 32), (3, 5, 137)],
                         ids=lambda d: "x".join(map(str, d)))
def test_integers_with_types(T, ora, dims):
    import synth
    d = synth.small_field(dims, seed=sum(dims), kind="noise").astype(np.float64)
    eb = 1e-3
    cps = ora.find_cp(d.astype(np.float32), eb)
    want = ora.double_compress_topo_3d(d, eb, 64, ora.mark_types(cps, dims), dims)
    assert T.double_compress_topology_3d(d, eb, 64, cps.view(T.CP3_DT).reshape(-1)) == want
