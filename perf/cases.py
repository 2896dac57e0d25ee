"""The calls that the library's users make, as timed and compared cases.

Every case is one call (or a write-and-read pair) through the public Python
binding and C ABI of libtoposzp_b200.so, on inputs made on the GPU from a seed.
Streams are returned in the caller's whole, once zeroed buffers, with their
lengths beside them:

  compress     szp_b200_topo_compress_dev: a device field into its topology
               and sort-position streams, in buffers that the caller keeps
  decompress   Context.decompress: device streams back into a field, with the
               post-processing the case asks for
  container    Context.decompress_container: an .SZp file's bytes, read as the
               CPU writer of T threads laid them out
  batch        Batch.compress: many fields of mixed sizes and bounds, one call
  plain        Context.plain_compress + plain_decompress: the codec without
               topology, float32 or float64
  f64          Context.compress_f64: the float64 3D compressor with its
               saddle-repair passes
  host         Context.compress_host + decompress_host on pinned host buffers

Fields are the two families that the repository's own workloads use: sums of
Gaussian bumps with a low-frequency term and white noise, and band-limited
noise with power spectrum k^-3.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "toposzp-cuda_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import toposzp_b200 as T  # noqa: E402


def listed():
    return [
        # a small 2D tile compressed on its own: launches and waits are what counts
        {"name": "compress_2d_60x90", "op": "compress", "dims": "60x90", "field": "bumps", "mode": "abs", "eb": 1e-3,
         "B": 64, "index": True},
        # the same tile read back from its stored bytes (no block index)
        {"name": "decompress_2d_60x90", "op": "decompress", "dims": "60x90", "field": "bumps", "mode": "abs",
         "eb": 1e-3, "B": 64, "index": False, "post": 1},
        # a climate-model surface field (1800 x 3600)
        {"name": "compress_2d_1800x3600", "op": "compress", "dims": "1800x3600", "field": "bumps", "mode": "abs",
         "eb": 1e-3, "B": 64, "index": False},
        {"name": "decompress_2d_1800x3600", "op": "decompress", "dims": "1800x3600", "field": "bumps", "mode": "abs",
         "eb": 1e-3, "B": 64, "index": False, "post": 1},
        # a hurricane-like volume (100 x 500 x 500) with a value-range bound,
        # compressed, and read back from an .SZp file of an 8-thread CPU writer
        {"name": "compress_3d_100x500x500", "op": "compress", "dims": "100x500x500", "field": "bumps", "mode": "rel",
         "eb": 1e-4, "B": 64, "index": True},
        {"name": "container_3d_100x500x500", "op": "container", "dims": "100x500x500", "field": "bumps", "mode": "rel",
         "eb": 1e-4, "B": 64, "threads": 8, "post": 1},
        # a turbulence snapshot (512^3), the largest field; read back with the
        # index its writer kept
        {"name": "compress_3d_512", "op": "compress", "dims": "512x512x512", "field": "band", "mode": "abs",
         "eb": 1e-4, "B": 64, "index": True},
        {"name": "decompress_3d_512", "op": "decompress", "dims": "512x512x512", "field": "band", "mode": "abs",
         "eb": 1e-4, "B": 64, "index": True, "post": 1},
        # 256 fields of mixed 2D and 3D sizes and bounds in one call
        {"name": "batch_256", "op": "batch", "count": 256, "B": 64, "spec_seed": 3},
        # the codec without topology on a long array of odd length
        {"name": "plain_f32_60000007", "op": "plain", "n": 60000007, "dtype": "f32", "eb": 1e-3, "B": 64},
        # float64 compression of a 3D field with critical points given
        {"name": "f64_3d_256", "op": "f64", "dims": "256x256x256", "eb": 1e-5, "B": 64},
        # compression and decompression of a surface field that lives on the host
        {"name": "host_2d_1800x3600", "op": "host", "dims": "1800x3600", "field": "bumps", "mode": "abs", "eb": 1e-3,
         "B": 64, "post": 1},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """A case of the listed ranges: 2D fields from a few thousand points to
    about 8 M, 3D fields from 16^3 to 400^3, the operations, bounds and block
    sizes in the proportions of the list."""
    op = rng.choice(["compress"] * 4 + ["decompress"] * 4 + ["container", "batch", "plain", "f64", "host"])
    B = rng.choice([64, 64, 64, 64, 32, 128])
    if op == "batch":
        return {"op": op, "count": _log_int(rng, 2, 96), "B": 64, "spec_seed": rng.randrange(1 << 20)}
    if op == "plain":
        return {"op": op, "n": _log_int(rng, 20000, 60000000), "dtype": rng.choice(["f32", "f32", "f64"]),
                "eb": 10 ** rng.uniform(-4, -1), "B": B}
    if op == "f64":
        dims = [_log_int(rng, 16, 256) for _ in range(3)]
        return {"op": op, "dims": "x".join(map(str, dims)), "eb": 10 ** rng.uniform(-5, -2), "B": B}
    if rng.random() < 0.5:
        dims = [_log_int(rng, 50, 2800) for _ in range(2)]
    else:
        dims = [_log_int(rng, 16, 400) for _ in range(3)]
    case = {"op": op, "dims": "x".join(map(str, dims)), "field": rng.choice(["bumps", "bumps", "band"]),
            "mode": rng.choice(["abs", "rel"]), "eb": 10 ** rng.uniform(-4.5, -2.5), "B": B}
    if op in ("compress", "decompress"):
        case["index"] = rng.random() < 0.5
    if op == "container":
        case["threads"] = rng.choice([1, 3, 8, 16])
    if op != "compress":
        case["post"] = rng.choice([0, 1, 1, 1, 2]) if len(dims) == 3 else rng.choice([0, 1, 1, 1])
    return case


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------

def _dims(case):
    return tuple(int(v) for v in case["dims"].split("x"))


def _bumps(dims, count, sigma_lo, sigma_hi, noise, gen):
    """Separable Gaussian bumps, 0.3 sin cos (cos) and N(0, noise), float32."""
    dev, f64 = "cuda", torch.float64
    g = []
    for s in dims:
        c = torch.rand(count, 1, generator=gen, device=dev, dtype=f64) * s
        g.append([torch.arange(s, device=dev, dtype=f64)[None, :] - c])
    sigma = sigma_lo + (sigma_hi - sigma_lo) * torch.rand(count, 1, generator=gen, device=dev, dtype=f64)
    amp = torch.randn(count, 1, generator=gen, device=dev, dtype=f64)
    g = [torch.exp(-(d[0] ** 2) / (2 * sigma ** 2)) for d in g]
    trig = [torch.cos(2 * math.pi * torch.arange(s, device=dev, dtype=f64) / s) for s in dims]
    trig[-1] = torch.sin(2 * math.pi * torch.arange(dims[-1], device=dev, dtype=f64) / dims[-1])
    if len(dims) == 2:
        out = (g[0] * amp).T @ g[1] + 0.3 * trig[0][:, None] * trig[1][None, :]
    else:
        rest = (g[1][:, :, None] * g[2][:, None, :]).reshape(count, -1)
        out = ((g[0] * amp).T @ rest).reshape(dims)
        out += 0.3 * trig[0][:, None, None] * trig[1][None, :, None] * trig[2][None, None, :]
    out = out.to(torch.float32)
    out += noise * torch.randn(dims, generator=gen, device=dev, dtype=torch.float32)
    return out.reshape(-1)


def _band(dims, gen):
    """White noise filtered to a k^-3 power spectrum, scaled to [0, 1]."""
    spec = torch.fft.rfftn(torch.randn(dims, generator=gen, device="cuda", dtype=torch.float64))
    k2 = torch.zeros((), device="cuda", dtype=torch.float64)
    for a, s in enumerate(dims):
        f = (torch.fft.rfftfreq if a == len(dims) - 1 else torch.fft.fftfreq)(s, device="cuda", dtype=torch.float64) * s
        shape = [1] * len(dims)
        shape[a] = f.numel()
        k2 = k2 + (f * f).reshape(shape)
    k2.view(-1)[0] = 1.0
    amp = k2.pow_(-0.75)
    amp.view(-1)[0] = 0.0
    spec *= amp
    out = torch.fft.irfftn(spec, s=dims)
    lo, hi = out.min(), out.max()
    return ((out - lo) / (hi - lo)).to(torch.float32).reshape(-1).contiguous()


def _noise(dims):
    """Noise of the bump fields: a smooth 3D volume carries less of it."""
    return 1e-3 if len(dims) == 2 else 1e-4


def _field(case, gen):
    dims = _dims(case)
    if case["field"] == "band":
        return _band(dims, gen)
    side = min(dims)
    lo, hi = (0.01, 0.12) if len(dims) == 2 else (0.05, 0.6)
    return _bumps(dims, 40 if len(dims) == 2 else 200, max(1.0, lo * side), max(2.0, hi * side), _noise(dims), gen)


def _abs_eb(x, mode, eb):
    """The bound as the reference's parser gives it: float arithmetic."""
    if mode == "abs":
        return float(np.float32(eb))
    span = np.float32(x.max().item()) - np.float32(x.min().item())
    return float(np.float32(np.float32(eb) * span))


def _batch_specs(case):
    """Shapes and bounds of a batch: half 2D (sides 64..2048), half 3D (32..256)."""
    rng = np.random.default_rng(case["spec_seed"])
    specs = []
    for i in range(case["count"]):
        nd, lo, hi = (2, 64, 2048) if i < (case["count"] + 1) // 2 else (3, 32, 256)
        dims = tuple(int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) for _ in range(nd))
        specs.append((dims, float(math.exp(rng.uniform(math.log(1e-5), math.log(1e-2)))), i % 2 == 1))
    return specs


def _plain_input(case, gen):
    """Two incommensurate waves and a random walk of step 0.03."""
    n = case["n"]
    i = torch.arange(n, device="cuda", dtype=torch.float64)
    x = 80.0 * torch.sin(i * 0.0123 + 0.4) + 20.0 * torch.sin(i * 0.00071 + 1.3)
    x += torch.cumsum(0.03 * torch.randn(n, generator=gen, device="cuda", dtype=torch.float64), 0)
    return x.to(torch.float64 if case["dtype"] == "f64" else torch.float32)


def _f64_input(dims, gen):
    """Eight separable cosine products and N(0, 1e-4), with the records of its
    strict 6-neighbour critical points (x, y, z, type, 0, 0)."""
    dev, f64 = "cuda", torch.float64
    facs = []
    for s in dims:
        f = 0.5 + 3.5 * torch.rand(8, 1, generator=gen, device=dev, dtype=f64)
        p = 2 * math.pi * torch.rand(8, 1, generator=gen, device=dev, dtype=f64)
        facs.append(torch.cos(2 * math.pi * f * torch.arange(s, device=dev, dtype=f64)[None, :] / s + p))
    amp = torch.randn(8, 1, generator=gen, device=dev, dtype=f64)
    rest = (facs[1][:, :, None] * facs[2][:, None, :]).reshape(8, -1)
    d = ((facs[0] * amp).T @ rest).reshape(dims)
    d += 1e-4 * torch.randn(dims, generator=gen, device=dev, dtype=f64)
    c = d[1:-1, 1:-1, 1:-1]
    hi, lo = [], []
    for a in range(3):
        m = d[tuple(slice(0, -2) if b == a else slice(1, -1) for b in range(3))]
        p = d[tuple(slice(2, None) if b == a else slice(1, -1) for b in range(3))]
        hi.append((c > m) & (c > p))
        lo.append((c < m) & (c < p))
    mx, mn = hi[0] & hi[1] & hi[2], lo[0] & lo[1] & lo[2]
    sd = (hi[0] | hi[1] | hi[2]) & (lo[0] | lo[1] | lo[2])
    t = torch.zeros(c.shape, device=dev, dtype=torch.int32)
    t[sd], t[mn], t[mx] = 3, 2, 1
    at = t.nonzero()
    rec = torch.zeros((at.shape[0], 6), device=dev, dtype=torch.int32)
    rec[:, :3] = at + 1
    rec[:, 3] = t[t != 0]
    return d.reshape(-1).contiguous(), rec


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------

_kept = {}


def _workspace():
    """The one stream and workspace that a program keeps for all its fields."""
    if "ctx" not in _kept:
        _kept["stream"] = torch.cuda.Stream()
        _kept["ctx"] = T.Context(_kept["stream"].cuda_stream)
    return _kept["stream"], _kept["ctx"]


def _batcher(B):
    if B not in _kept:
        stream, _ = _workspace()
        _kept[B] = T.Batch(B, stream.cuda_stream)
    return _kept[B]


def prepare(case, seed):
    stream, ctx = _workspace()
    with torch.cuda.stream(stream):
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        op, st = case["op"], {"case": case}
        if op == "batch":
            specs = _batch_specs(case)
            items, nt, ns = [], 0, 0
            for dims, eb, rel in specs:
                side, nd = min(dims), len(dims)
                lo, hi = (0.02, 0.2) if nd == 2 else (0.05, 0.3)
                x = _bumps(dims, 20 * (nd - 1), max(1.0, lo * side), max(2.0, hi * side), 1e-3, gen)
                items.append((x, dims, eb, rel))
            # the streams of all fields go into two buffers, each field's
            # share of the size that its bound asks for
            L = T.lib()
            tb = [(L.szp_b200_topo_bound(t.numel(), case["B"]) + 255) // 256 * 256 for t, _, _, _ in items]
            sb = [(L.szp_b200_sort_bound(t.numel(), case["B"]) + 255) // 256 * 256 for t, _, _, _ in items]
            st["topo"] = torch.zeros(sum(tb), dtype=torch.uint8, device="cuda")
            st["sort"] = torch.zeros(sum(sb), dtype=torch.uint8, device="cuda")
            bufs = []
            for a, b in zip(tb, sb):
                bufs.append((st["topo"][nt:nt + a], st["sort"][ns:ns + b]))
                nt, ns = nt + a, ns + b
            st.update(items=items, bufs=bufs, batch=_batcher(case["B"]))
        elif op == "plain":
            st["x"] = _plain_input(case, gen)
            dbl = int(case["dtype"] == "f64")
            st["stream"] = torch.zeros(T.lib().szp_b200_plain_bound(case["n"], case["B"], dbl, 0), dtype=torch.uint8,
                                       device="cuda")
            st["out"] = torch.empty_like(st["x"])
        elif op == "f64":
            dims = _dims(case)
            st["x"], st["cps"] = _f64_input(dims, gen)
            st["stream"] = torch.zeros(T.lib().szp_b200_topo_bound(st["x"].numel(), case["B"]), dtype=torch.uint8,
                                       device="cuda")
            st["q"] = torch.empty(st["x"].numel(), dtype=torch.int32, device="cuda")
        else:
            dims, B = _dims(case), case["B"]
            x = _field(case, gen)
            eb = _abs_eb(x, case["mode"], case["eb"])
            st["eb"] = eb
            if op == "compress":
                n, L = x.numel(), T.lib()
                st["x"] = x
                st["topo"] = torch.zeros(L.szp_b200_topo_bound(n, B), dtype=torch.uint8, device="cuda")
                st["sort"] = torch.zeros(L.szp_b200_sort_bound(n, B), dtype=torch.uint8, device="cuda")
                st["idx"] = torch.zeros(2 * (-(-n // B)), dtype=torch.int64, device="cuda") if case["index"] else None
            elif op == "host":
                n, L = x.numel(), T.lib()
                st["x"] = x.cpu().pin_memory().numpy().reshape(dims)
                st["topo"] = torch.zeros(L.szp_b200_topo_bound(n, B), dtype=torch.uint8).pin_memory().numpy()
                st["sort"] = torch.zeros(L.szp_b200_sort_bound(n, B), dtype=torch.uint8).pin_memory().numpy()
                st["out"] = torch.zeros(n, dtype=torch.float32).pin_memory().numpy()
            else:
                topo, sort, idx, sz = ctx.compress(x, dims, eb, B, index=bool(case.get("index")))
                if op == "container":
                    st["cont"] = ctx.to_container(topo, sz.topo_bytes, sort, sz.sort_bytes, dims, B, sz.extrema_count,
                                                  threads=case["threads"]).clone()
                else:
                    st["topo"], st["sort"], st["idx"] = topo[:sz.topo_bytes].clone(), sort[:sz.sort_bytes].clone(), idx
    return st


def run(st):
    case = st["case"]
    op = case["op"]
    stream, ctx = _workspace()
    with torch.cuda.stream(stream):
        if op == "compress":
            sz = T.Sizes()
            rc = T.lib().szp_b200_topo_compress_dev(
                ctx.ptr, st["x"].data_ptr(), T.geom_of(_dims(case)), st["eb"], case["B"], st["topo"].data_ptr(),
                st["sort"].data_ptr(), st["idx"].data_ptr() if case["index"] else None, ctypes.byref(sz))
            if rc:
                raise T.ToposzpError(T.last_error())
            return {"topo": st["topo"], "sort": st["sort"], "index": st["idx"],
                    "sizes": [sz.topo_bytes, sz.sort_bytes, sz.cp_count, sz.extrema_count]}
        if op == "decompress":
            return ctx.decompress(st["topo"], st["topo"].numel(), st["sort"], st["sort"].numel(), st["idx"],
                                  _dims(case), st["eb"], case["B"], postprocess=case["post"])
        if op == "container":
            return ctx.decompress_container(st["cont"], _dims(case), st["eb"], case["B"], postprocess=case["post"])
        if op == "batch":
            got = st["batch"].compress(st["items"], st["bufs"])
            sizes = np.array([[s.topo_bytes, s.sort_bytes, s.cp_count, s.extrema_count] for _, _, s, _ in got],
                             dtype=np.int64)
            return {"topo": st["topo"], "sort": st["sort"], "sizes": sizes,
                    "eb": np.array([e for _, _, _, e in got], dtype=np.float32)}
        if op == "plain":
            k = ctx.plain_compress(st["x"], case["eb"], case["B"], st["stream"])
            ctx.plain_decompress(st["stream"], k, case["n"], case["eb"], case["B"], st["out"])
            return {"stream": st["stream"], "bytes": k, "out": st["out"]}
        if op == "f64":
            k = ctx.compress_f64(st["x"], _dims(case), case["eb"], case["B"], st["cps"], st["cps"].shape[0],
                                 st["stream"], d_q=st["q"])
            return {"stream": st["stream"], "bytes": k, "q": st["q"]}
        sz = ctx.compress_host(st["x"], st["eb"], case["B"], st["topo"], st["sort"])
        out = ctx.decompress_host(st["topo"], sz.topo_bytes, st["sort"], sz.sort_bytes, _dims(case), st["eb"],
                                  case["B"], st["out"], postprocess=case["post"])
        return {"topo": st["topo"], "sort": st["sort"], "sizes": [sz.topo_bytes, sz.sort_bytes], "out": out}


def exact(case, seed):
    """The decoded values of quantized fields in 64 bits.  The streams are
    whole numbers and the post-processed fields come from a serial raster
    pass over the field, which has no form of its own in 64 bits."""
    if case["op"] == "plain":
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        x = _plain_input(case, gen).double()
        eb = float(np.float32(case["eb"])) if case["dtype"] == "f32" else case["eb"]
        return {"stream": None, "bytes": None, "out": torch.trunc(x * (1.0 / eb)) * eb}
    if case["op"] in ("decompress", "container", "host") and case["post"] == 0:
        gen = torch.Generator(device="cuda")
        gen.manual_seed(seed)
        x = _field(case, gen)
        eb = _abs_eb(x, case["mode"], case["eb"])
        out = torch.trunc(x.double() * (1.0 / eb)) * eb
        if case["op"] == "host":
            return {"topo": None, "sort": None, "sizes": None, "out": out}
        return out
    return None


# ---------------------------------------------------------------------------
# bytes that a call cannot do without
# ---------------------------------------------------------------------------

def _block_stream(n, B, delta, tags):
    """Stream bytes of n values whose largest step in a block is delta."""
    bits = math.floor(math.log2(max(delta, 1.0))) + 1
    return math.ceil(n / B) * 5 + n * (1 + bits + (2 if tags else 0)) / 8


def _topo_bytes(dims, field, noise, eb):
    """Topology and sort-position streams of a field, about: the field's own
    steps and about 3.4 standard deviations of the noise's differences (the
    largest of a block of 64) set the bits; the noise sets the share of
    extrema where it is above the field's slope (in 2D)."""
    n, nd = math.prod(dims), len(dims)
    if field == "band":
        step, share = (0.12, 0.14) if nd == 3 else (0.02, 0.1)
    else:
        step = 5.0 / min(dims) + 4.8 * noise if nd == 3 else 4.8 * noise
        share = 1e-4 if nd == 3 else 0.2
    ext = n * share
    return _block_stream(n, 64, step / eb, True) + _block_stream(ext, 64, max(2.0, ext * eb), False)


def work(case):
    op = case["op"]
    if op == "batch":
        total = 0.0
        for dims, eb, rel in _batch_specs(case):
            total += 4 * math.prod(dims) + _topo_bytes(dims, "bumps", 1e-3, eb * (4.0 if rel else 1.0))
        return {"bytes": total, "flops": 0.0}
    if op == "plain":
        n, es = case["n"], 8 if case["dtype"] == "f64" else 4
        return {"bytes": 2.0 * (es * n + _block_stream(n, case["B"], 1.0 / case["eb"], False)), "flops": 0.0}
    dims = _dims(case)
    n = math.prod(dims)
    if op == "f64":
        return {"bytes": 12.0 * n + _block_stream(n, case["B"], 0.06 / case["eb"], True), "flops": 0.0}
    streams = _topo_bytes(dims, case["field"], _noise(dims), case["eb"] * (4.0 if case["mode"] == "rel" and
                                                                        case["field"] == "bumps" else 1.0))
    if op == "compress" and case["index"]:
        streams += 8.0 * (n // case["B"] + 1)
    if op == "host":
        return {"bytes": 2 * (4.0 * n + streams), "flops": 0.0}
    return {"bytes": 4.0 * n + streams, "flops": 0.0}
