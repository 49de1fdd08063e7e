"""The work whose speed is watched: the passes a user of the codec makes, over
the range of snapshots it meets.

A case is one pass through the package's public entry points on device-resident
data: compressing a snapshot (the bound given, or converted from a relative one
first), decompressing a stream, the round trip, a batch of mixed snapshots in
one launch, or the per-point check of a reconstruction.  Snapshots come in four
layouts: clustered (dark-matter-like halos over a uniform background, shuffled),
lattice (jittered FCC in 3D, square in 2D, shuffled), uniform, and ordered
(clustered points in the order of a space-filling curve, as domain-decomposed
codes write them).
"""
import math

import numpy as np
import torch

import gpz_b200 as gz
from gpz_b200.batch import Batch, Snapshot

CHUNK = 1024


def listed():
    c = dict(op="compress", layout="clustered", n=0, dim=3, bits=32, mode="rel", bound=1e-4, seg=0)
    return [
        # one rank's particles of a small run, or one halo cut out of a snapshot:
        # the call's own latency is what counts
        dict(c, name="halo_compress", n=5_003, bound=1e-3),
        dict(c, name="halo_decompress", op="decompress", n=5_003, bound=1e-3),
        # one time step of a domain-decomposed code, written in the order of its
        # space-filling curve: few blocks per chunk, many points per block
        dict(c, name="step_compress", layout="ordered", n=2_000_003),
        dict(c, name="step_decompress", op="decompress", layout="ordered", n=2_000_003),
        # the headline snapshot of bench.py
        dict(c, name="snapshot_compress", n=143_735_721),
        dict(c, name="snapshot_decompress", op="decompress", n=143_735_721),
        # analysis-quality storage: a tight absolute bound, wide positions inside
        # large blocks (bench.py's clustered-abs on a smaller snapshot)
        dict(c, name="tight_compress", n=24_000_001, mode="abs", bound=1e-3, seg=32),
        # molecular dynamics in double precision: bench.py's FCC crystal
        dict(c, name="crystal_compress", layout="lattice", n=50_000_003, bits=64, bound=1e-5),
        dict(c, name="crystal_decompress", op="decompress", layout="lattice", n=50_000_003, bits=64, bound=1e-5),
        # a 2D double-precision sheet stored and read back
        dict(c, name="sheet_roundtrip", op="roundtrip", layout="lattice", n=25_000_001, dim=2, bits=64, bound=1e-5),
        # many snapshots of mixed sizes and types in one launch of a kept plan
        dict(c, name="mixed_batch", op="batch", count=48, n=300_007),
        # a user who checks every point of what was stored
        dict(c, name="step_verify", op="verify", n=4_000_037),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    op = rng.choice(["compress", "compress", "decompress", "decompress", "roundtrip", "batch", "verify"])
    if op == "batch":
        return dict(op=op, layout="clustered", n=log_int(20_000, 400_000), dim=3, bits=32, mode="rel", bound=1e-4,
                    seg=0, count=rng.randint(8, 48))
    bits = rng.choice([32, 32, 64])
    dim = rng.choice([3, 3, 2])
    n = log_int(1_000, 4_000_000 if op == "verify" else 40_000_000 if bits == 32 else 20_000_000)
    layout = rng.choice(["clustered", "lattice", "uniform", "ordered"])
    if rng.random() < 0.7:
        mode, bound, seg = "rel", rng.choice([1e-2, 1e-3, 3e-4, 1e-4, 1e-5]), 0
    else:
        mode, bound, seg = "abs", 10.0 ** rng.uniform(-3.0, 0.0), rng.choice([1, 2, 4, 8, 16, 32, 64])
    return dict(op=op, layout=layout, n=n, dim=dim, bits=bits, mode=mode, bound=bound, seg=seg)


# ---------------------------------------------------------------------------
# snapshots
# ---------------------------------------------------------------------------
def _device():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _generator(seed):
    g = torch.Generator(device=_device())
    g.manual_seed(seed)
    return g


def _clustered(n, dim, dt, g):
    """70 % of the points in Gaussian clusters of Pareto(1.5) populations, 30 %
    uniform, box [0, 1000): bench.py's generator for any size."""
    dev = _device()
    k = max(1, min(20_000, n // 200))
    cen = torch.rand(dim, k, generator=g, device=dev) * 1000
    sig = 0.5 * 20 ** torch.rand(k, generator=g, device=dev)
    cdf = torch.cumsum(((1 - torch.rand(k, generator=g, device=dev)) ** (-1 / 1.5)).double(), 0)
    idx = torch.searchsorted(cdf, torch.rand(n, generator=g, device=dev, dtype=torch.float64) * cdf[-1])
    idx.clamp_(max=k - 1)
    halo = torch.rand(n, generator=g, device=dev) < 0.7  # the points come out shuffled
    out = []
    for d in range(dim):
        p = cen[d][idx].to(dt) + sig[idx].to(dt) * torch.randn(n, generator=g, device=dev, dtype=dt)
        u = torch.rand(n, generator=g, device=dev, dtype=dt) * 1000
        out.append(torch.where(halo, p.clamp_(0, 999.999), u))
    return out


def _lattice(n, dim, dt, g):
    """Jittered FCC (3D) or square (2D) lattice of spacing 1, shuffled."""
    dev = _device()
    i = torch.randperm(n, generator=g, device=dev)
    if dim == 3:
        cells = max(1, round((n / 4) ** (1 / 3)))
        cell, b = i // 4, i % 4
        basis = torch.tensor([[0.0, 0.5, 0.5, 0.0], [0.0, 0.5, 0.0, 0.5], [0.0, 0.0, 0.5, 0.5]], dtype=dt, device=dev)
        out = [(c.to(dt) + basis[d][b]) for d, c in enumerate((cell % cells, (cell // cells) % cells,
                                                               cell // (cells * cells)))]
    else:
        side = max(1, math.isqrt(n))
        out = [(i % side).to(dt), (i // side).to(dt)]
    return [a + 0.05 * torch.randn(n, generator=g, device=dev, dtype=dt) for a in out]


def _snapshot(layout, n, dim, bits, seed):
    dt = torch.float32 if bits == 32 else torch.float64
    g = _generator(seed)
    if layout == "lattice":
        return _lattice(n, dim, dt, g)
    if layout == "uniform":
        return [torch.rand(n, generator=g, device=_device(), dtype=dt) * 1000 for _ in range(dim)]
    axes = _clustered(n, dim, dt, g)
    if layout == "ordered":  # Morton order on a 1024-cell grid per axis
        code = torch.zeros(n, dtype=torch.int64, device=axes[0].device)
        for d, a in enumerate(axes):
            q = (a * 1.024).to(torch.int64).clamp_(0, 1023)
            for b in range(10):
                code |= ((q >> b) & 1) << (dim * b + d)
        order = torch.argsort(code, stable=True)
        axes = [a[order].contiguous() for a in axes]
    return axes


def _typed(bits, v):
    return float(np.float32(v)) if bits == 32 else float(v)


def _xyz(axes):
    return axes[0], axes[1], axes[2] if len(axes) == 3 else None


def _bound_args(case):
    b = _typed(case["bits"], case["bound"])
    return dict(rel=b) if case["mode"] == "rel" else dict(eb=b, seg=case["seg"])


def _buffers(case):
    """The stream buffer and scratch a program keeps for its snapshots."""
    n = case["n"]
    return (torch.zeros(gz.stream_bound(n, case["dim"], case["bits"]), dtype=torch.uint8, device=_device()),
            torch.empty(gz.compress_scratch_bytes(n), dtype=torch.uint8, device=_device()))


def _compress(axes, args, bits, out, scratch):
    """What a user does with a snapshot: a relative bound is converted first."""
    x, y, z = _xyz(axes)
    n, dim = x.numel(), len(axes)
    if "rel" in args:
        eb, _ = gz.rel_to_abs(x, y, z, args["rel"])
        p = gz.make_params(n, dim, bits, eb, rel_mode=True, rel_eb=args["rel"])
    else:
        p = gz.make_params(n, dim, bits, args["eb"], seg_size=args["seg"])
    return gz.compress_into(p, x, y, z if dim == 3 else x, out, scratch)


def _batch_members(case, seed):
    """Sizes from n / 32 to 4 n, both precisions and dimensions, bounds relative
    (converted on the device) or given."""
    out = []
    for i in range(case["count"]):
        bits, dim = (32, 32, 64)[i % 3], (3, 3, 3, 2)[i % 4]
        n = max(1, int(case["n"] * 2.0 ** ((i * 7) % 8 - 5)) + 13 * i)
        out.append((("clustered", "uniform", "lattice", "ordered")[(i // 2) % 4], n, dim, bits, seed * 1009 + i))
    return out


def prepare(case, seed):
    op = case["op"]
    if op == "batch":
        snaps = []  # streams go to buffers the program keeps
        for i, m in enumerate(_batch_members(case, seed)):
            x, y, z = _xyz(_snapshot(*m))
            out = torch.zeros(gz.stream_bound(m[1], m[2], m[3]), dtype=torch.uint8, device=_device())
            if i % 4 == 1:
                snaps.append(Snapshot(x, y, z, eb=_typed(m[3], 0.05), seg_size=8, out=out))
            else:
                snaps.append(Snapshot(x, y, z, rel_eb=_typed(m[3], (1e-4, 1e-3)[i % 2]), out=out))
        return dict(op=op, plan=Batch(snaps))
    axes = _snapshot(case["layout"], case["n"], case["dim"], case["bits"], seed)
    args = _bound_args(case)
    out, scratch = _buffers(case)
    state = dict(op=op, bits=case["bits"], axes=axes, args=args)
    if op in ("compress", "roundtrip"):
        state.update(out=out, scratch=scratch)
    else:
        r = _compress(axes, args, case["bits"], out, scratch)
        state["stream"] = out[: r.stream_bytes].clone()
    if op == "verify":
        state["header"] = gz.parse_header(state["stream"][:32].cpu().numpy().tobytes())
        state["back"] = gz.decompress(state["stream"])
    return state


def run(state):
    op = state["op"]
    if op in ("compress", "roundtrip"):
        r = _compress(state["axes"], state["args"], state["bits"], state["out"], state["scratch"])
        res = {"stream": state["out"], "bytes": int(r.stream_bytes), "segment": int(r.seg_size)}
        if op == "roundtrip":
            res["points"] = [t for t in gz.decompress(state["out"][: r.stream_bytes]) if t is not None]
        return res
    if op == "decompress":
        return [t for t in gz.decompress(state["stream"]) if t is not None]
    if op == "batch":
        state["plan"].launch()
        sizes = np.array([r.stream_bytes for r, _ in state["plan"].results()])
        return [sizes] + [s.out for s in state["plan"].snapshots]
    x, y, z = _xyz(state["axes"])
    h = state["header"]
    v = gz.verify(x, y, z, *state["back"], h["eb"], h["seg"])
    d = len(state["axes"])
    return {"points": int(v.points), "over_bound_tol": int(v.over_bound_tol), "over_bound": int(v.over_bound),
            "max_abs_err": np.array(v.max_abs_err[:d]), "mse": np.array(v.mse[:d]), "psnr": np.array(v.psnr[:d])}


# stream bytes per point, measured for the listed cases; drawn ones use the
# layout's estimate below
_STREAM_BYTES = {"halo": 2.54, "step": 2.69, "snapshot": 4.17, "tight": 6.55, "crystal": 5.17, "sheet": 3.28}


def _stream_bytes(layout, n, dim, bits, mode, bound):
    """Coarse: the information in n sorted points at this bound, per point, over
    a chunk's extent."""
    cells = math.log2(1 / (2 * bound)) if mode == "rel" else math.log2(1000 / (2 * bound))
    per = dim * max(cells, 1.0) - (8.0 if layout != "ordered" else 18.0)
    return n * max(per, 4.0) / 8.0 + (n / CHUNK + 1) * (44 if bits == 32 else 72)


def work(case):
    op = case["op"]
    if op == "batch":
        moved = ops = 0.0
        for m in _batch_members(case, 1):
            raw = m[1] * m[2] * m[3] // 8
            moved += raw + _stream_bytes(m[0], m[1], m[2], m[3], "rel", 3e-4)
            ops += 6.0 * m[1] * m[2]
        return {"bytes": moved, "flops": ops}
    n, dim, bits = case["n"], case["dim"], case["bits"]
    raw = float(n * dim * bits // 8)
    key = case.get("name", "").split("_")[0]
    sb = n * _STREAM_BYTES[key] if key in _STREAM_BYTES else \
        _stream_bytes(case["layout"], n, dim, bits, case["mode"], case["bound"])
    if op == "verify":
        return {"bytes": 2 * raw, "flops": 8.0 * n * dim}
    # one multiply-add and one conversion per coordinate each way, the block id,
    # the position in it
    return {"bytes": (raw + sb) * (2 if op == "roundtrip" else 1), "flops": 6.0 * n * dim * (2 if op == "roundtrip" else 1)}


# ---------------------------------------------------------------------------
# the same results in plain torch, 64 bits
# ---------------------------------------------------------------------------
def _fma(a, b, c, bits):
    """a * b + c rounded once to the codec's float type, in float64 tensors.
    float32 operands: the product is exact in float64.  float64: the product's
    error term by Veltkamp splitting, the sum's by two-sum."""
    p = a * b
    if bits == 32:
        return (p + c).float().double()
    k = 134217729.0
    ah, bh = a * k - (a * k - a), b * k - (b * k - b)
    al, bl = a - ah, b - bh
    e = ((ah * bh - p) + ah * bl + al * bh) + al * bl
    s = p + c
    t = s - p
    return s + (((p - (s - t)) + (c - t)) + e)


def _round(v, bits):
    return v.float().double() if bits == 32 else v


def _segment(axes, dim, bits, case, eb):
    """The automatic segment size: the spread of the axes' sampled ranges picks
    it, the 32-bit limit on block ids doubles it (float32)."""
    n = axes[0].numel()
    if case["mode"] == "rel":
        stride = max((n - 256) // 1024, 1) if n >= 256 else 1
        starts = torch.arange(1024, device=axes[0].device) * stride
        live = starts + 256 <= n
        pick = (starts[live][:, None] + torch.arange(256, device=axes[0].device)).reshape(-1)
        rng = []
        for d in range(3):
            v = axes[d][pick] if d < dim else torch.zeros(1, dtype=axes[0].dtype, device=axes[0].device)
            lo, hi = (v.min().item(), v.max().item()) if v.numel() else (math.inf, -math.inf)
            if d < dim and not bool(live.all()):
                lo, hi = min(lo, 0.0), max(hi, 0.0)
            rng.append(hi - lo)
        mean = sum(rng) / 3
        var = sum((r - mean) ** 2 for r in rng) / (2 if bits == 32 and dim == 2 else 3)
        tight = case["bound"] <= 1e-4 * (1 + 1e-7)
        seg = (32 if tight else 2) if math.sqrt(var) / mean < 0.1 else (4 if tight else 1)
    else:
        seg = case["seg"]
        rng = [(a.max() - a.min()).item() for a in axes]
    if bits == 32:
        while (math.ceil(max(rng) / (2 * seg * eb)) + 1) ** dim > 0xFFFFFFFF:
            seg *= 2
    return seg


def _reconstruct(axes, case):
    """Reconstruction of every point in stream order (float64), and the
    originals in the same order."""
    dim, bits, n = case["dim"], case["bits"], case["n"]
    if case["mode"] == "rel":
        span = [_round((a.max().double() - a.min().double()), bits).item() for a in axes]
        eb = _typed(bits, max(span + ([0.0] if dim == 2 else [])) * _typed(bits, case["bound"]))
    else:
        eb = _typed(bits, case["bound"])
    seg = _segment(axes, dim, bits, case, eb)
    inv = _typed(bits, 1.0 / (2.0 * eb))
    sh = seg.bit_length() - 1
    outs, origs = [[] for _ in range(dim)], [[] for _ in range(dim)]
    step = CHUNK * 16_384
    rank = torch.arange(CHUNK, device=axes[0].device)
    rank = (rank % 32) * 32 + rank // 32
    for lo in range(0, n, step):
        hi = min(n, lo + step)
        rows = -(-(hi - lo) // CHUNK)
        pad = rows * CHUNK - (hi - lo)
        key = rel = None
        mul = 1
        mins, counts, vals = [], [], []
        for d in range(dim):
            v = axes[d][lo:hi].double()
            if pad:  # a short last chunk repeats its first point
                v = torch.cat([v, v[(rows - 1) * CHUNK].expand(pad)])
            v = v.reshape(rows, CHUNK)
            mn, mx = v.min(1, keepdim=True).values, v.max(1, keepdim=True).values
            nmn = _round(-mn * inv, bits)
            q = _fma(v, torch.full_like(v, inv), nmn.expand_as(v), bits).trunc().clamp_(min=0).to(torch.int64)
            den = _round(torch.tensor(2.0 * seg * eb, dtype=torch.float64), bits).item()
            bn = torch.ceil(_round(_round(mx - mn, bits) / den, bits)).to(torch.int64) + 1
            m = torch.ones_like(bn) if d == 0 else mul
            key = (q >> sh) * m if key is None else key + (q >> sh) * m
            rel = (q & (seg - 1)) if rel is None else rel | ((q & (seg - 1)) << (sh * d))
            mul = m * bn
            mins.append(mn)
            counts.append(bn)
            vals.append(v)
        key &= 0x7FFFFFFF
        order_key = (key << 10) | rank
        if pad:
            order_key[-1, CHUNK - pad:] |= 1 << 62  # the padding goes last
        order = torch.argsort(order_key, 1)
        key, rel = torch.gather(key, 1, order), torch.gather(rel, 1, order)
        bx, by = counts[0], counts[1]
        block = [key % bx, (key // bx) % by, key // (bx * by)] if dim == 3 else [key % bx, (key // bx) % by]
        for d in range(dim):
            q = block[d] * seg + ((rel >> (sh * d)) & (seg - 1))
            outs[d].append(((2 * q + 1).double() * eb + mins[d]).reshape(-1)[: hi - lo])
            origs[d].append(torch.gather(vals[d], 1, order).reshape(-1)[: hi - lo])
    return [torch.cat(o) for o in outs], [torch.cat(o) for o in origs]


def exact(case, seed):
    op = case["op"]
    if op in ("compress", "batch"):
        return None  # bytes
    axes = _snapshot(case["layout"], case["n"], case["dim"], case["bits"], seed)
    back, orig = _reconstruct(axes, case)
    if op == "decompress":
        return back
    if op == "roundtrip":
        return {"stream": None, "bytes": None, "segment": None, "points": back}
    err = [(o - _round(b, case["bits"])).abs() for o, b in zip(orig, back)]
    mse = np.array([(e * e).mean().item() for e in err])
    span = np.array([(o.max() - o.min()).item() for o in orig])
    return {"points": None, "over_bound_tol": None, "over_bound": None,
            "max_abs_err": np.array([e.max().item() for e in err]), "mse": mse,
            "psnr": 20 * np.log10(span) - 10 * np.log10(mse)}
