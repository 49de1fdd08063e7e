"""Infinities and NaNs through compress, decompress and verify: the stream is the
oracle's byte for byte, the reconstruction the oracle's values, and verify pairs
and counts such points as the block order says.  The chunks around are finite.

The reconstruction of a double chunk with an infinity is not compared: its block
count wraps to 0 in the format's decoder, which then divides 64-bit ids by zero."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import gpz_b200 as gz  # noqa: E402
from oracle import pyoracle as po  # noqa: E402

VALUES = {"+inf": [np.inf], "-inf": [-np.inf], "both": [np.inf, -np.inf], "nan": [np.nan],
          "all": [np.inf, -np.inf, np.nan]}


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    gz.lib()


def _axes(bits, dim, what, share, n=7 * 1024 + 77):
    """Integer coordinates; every second chunk and the short last one have `share` of their
    points non-finite on one axis or another."""
    dt = np.float32 if bits == 32 else np.float64
    rng = np.random.default_rng(dim * 100 + int(share * 10) + len(what))
    axes = [rng.integers(0, 200, n).astype(dt) for _ in range(dim)]
    for c in range(0, n, 1024):
        m = min(1024, n - c)
        if (c // 1024) % 2 and m == 1024:
            continue
        at = c + rng.permutation(m)[:max(1, int(m * share))]
        axis = rng.integers(0, dim, at.size)
        put = rng.choice(VALUES[what], at.size)
        for d in range(dim):
            axes[d][at[axis == d]] = put[axis == d]
    return axes


def _block_order(axes, lo, m, bits, sh=3):
    """Order of points lo .. lo + m (one chunk) by block id and rank, blocks of size 1
    (eb 1/16, segment 8): quantized values are exact multiples of 8 and saturate."""
    top = 0xFFFFFFFF if bits == 32 else (1 << 64) - 1
    big = np.finfo(np.float32 if bits == 32 else np.float64).max
    key, mul = [0] * m, 1
    for a in axes:
        v = a[lo:lo + m].astype(np.float64)
        num = v[~np.isnan(v)]
        mn, mx = min([big] + list(num)), max([-big] + list(num))
        with np.errstate(all="ignore"):
            nm = np.array(-mn * 8.0) if bits == 64 else np.float64(np.float32(-mn) * np.float32(8.0))
            q = v * 8.0 + nm
            rng = np.float64(np.float32(mx) - np.float32(mn)) if bits == 32 else np.float64(mx) - np.float64(mn)
        q = [0 if not x > 0 else top if x >= top else int(x) for x in q]
        key = [k + (x >> sh) * mul for k, x in zip(key, q)]
        n = 0 if not rng > 0 else 0xFFFFFFFF if rng >= 2.0 ** 32 else int(np.ceil(rng))
        if len(axes) == 2 and bits == 64 and a is axes[0]:
            n = 0 if not rng > 0 else top if rng >= 2.0 ** 64 else int(np.ceil(rng))
            mul = (mul * ((n + 1) & top)) & top
        else:
            mul = (mul * ((n + 1) & 0xFFFFFFFF)) & top
    p = np.arange(m)
    return np.lexsort(((p % 32) * 32 + p // 32, np.array([k & 0x7FFFFFFF for k in key])))


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("what", list(VALUES))
@pytest.mark.parametrize("share", [0.001, 0.3, 1.0])
def test_nonfinite_points(bits, dim, what, share):
    axes = _axes(bits, dim, what, share)
    n = axes[0].size
    z = axes[2] if dim == 3 else np.zeros_like(axes[0])
    with np.errstate(all="ignore"):
        want = po.compress(axes[0], axes[1], z, dim, 0.0625, 8)
        back = po.decompress(want)[:dim]
    dev = [torch.from_numpy(a).cuda() for a in axes]
    p = gz.make_params(n, dim, bits, 0.0625, 8)
    p.flags |= gz.GPZ_FLAG_SEG_FIXED
    out = torch.zeros(gz.stream_bound(n, dim, bits), dtype=torch.uint8, device="cuda")
    scratch = torch.empty(gz.compress_scratch_bytes(n), dtype=torch.uint8, device="cuda")
    r = gz.compress_into(p, dev[0], dev[1], dev[2] if dim == 3 else dev[0], out, scratch)
    assert r.status == 0 and out[: r.stream_bytes].cpu().numpy().tobytes() == want
    got = gz.decompress(out[: r.stream_bytes])[:dim]
    inf = np.any([np.isinf(a) for a in axes], 0)
    defined = np.concatenate([np.full(min(1024, n - lo), bits == 32 or not inf[lo:lo + 1024].any())
                              for lo in range(0, n, 1024)])
    for a, b in zip(got, back):
        assert np.array_equal(a.cpu().numpy()[defined], b[defined], equal_nan=True)
    # verify: every point meets itself plus an error, infinities meet 0
    rng = np.random.default_rng(n)
    err = rng.choice([0.0, 0.03125, 0.0625, 0.0703125], size=(dim, n)).astype(axes[0].dtype)
    rec = [np.empty_like(a) for a in axes]
    off = [np.empty(n) for _ in axes]
    for lo in range(0, n, 1024):
        m = min(1024, n - lo)
        order = _block_order(axes, lo, m, bits)
        for d in range(dim):
            o = axes[d][lo:lo + m][order]
            rec[d][lo:lo + m] = np.where(np.isfinite(o), o + err[d][lo:lo + m], 0)
            off[d][lo:lo + m] = np.abs(o - rec[d][lo:lo + m])
    put = [torch.from_numpy(a).cuda() for a in rec]
    v = gz.verify(dev[0], dev[1], dev[2] if dim == 3 else None, put[0], put[1], put[2] if dim == 3 else None, 0.0625, 8)
    assert v.over_bound == int((~(np.array(off) <= 0.0625)).any(0).sum())
    for d in range(dim):
        assert v.max_abs_err[d] == max([0.0] + list(off[d][~np.isnan(off[d])]))
