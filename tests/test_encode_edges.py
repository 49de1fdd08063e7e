"""The compress kernel at the edges of its rules, byte for byte against the
oracle: chunk counts around the look-back's records (16 chunks) and windows
(512), id ranges where the ranking changes (2^11, 2^22, beyond), buckets at the
size that declines a chunk, few distinct ids (one to four radix passes),
misaligned axes, short last chunks."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import gpz_b200 as gz  # noqa: E402
from oracle import pyoracle as po  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    gz.lib()


def check(axes, eb, seg, shift=0):
    """Stream of the axes (as views starting `shift` elements into their buffers) equals the oracle's, three times."""
    dim = len(axes)
    z = axes[2] if dim == 3 else np.zeros_like(axes[0])
    ebT = float(axes[0].dtype.type(eb))
    want = po.compress(axes[0], axes[1], z, dim, ebT, seg)
    dev = []
    for a in axes:
        buf = torch.zeros(a.size + shift, dtype=torch.from_numpy(a).dtype, device="cuda")
        buf[shift:] = torch.from_numpy(a).cuda()
        dev.append(buf[shift:])
    for _ in range(3):
        s, r = gz.compress(dev[0], dev[1], dev[2] if dim == 3 else None, eb=ebT, seg_size=seg)
        assert r.status == 0 and r.seg_size == seg
        assert s.cpu().numpy().tobytes() == want


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("chunks", [1, 2, 3, 4, 15, 16, 17, 31, 33, 511, 512, 513, 529, 1800])
def test_chunk_counts(bits, chunks):
    dt = np.float32 if bits == 32 else np.float64
    rng = np.random.default_rng(chunks)
    n = chunks * 1024 - (0 if chunks % 2 else 1000)
    check([(rng.random(n) * 100).astype(dt) for _ in range(3)], 0.05, 4)


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("bx,by", [(1, 1), (2, 1), (16, 16), (89, 23), (64, 32), (2049, 1), (512, 512), (513, 2048),
                                   (2048, 2048), (2048, 2049), (40000, 50000)])
@pytest.mark.parametrize("crowd", [0, 14, 15, 16, 17, 250, 300])
def test_id_ranges_and_crowded_buckets(bits, bx, by, crowd):
    """2D grids of bx * by blocks (both corners present), `crowd` points of every other chunk in one block."""
    dt = np.float32 if bits == 32 else np.float64
    rng = np.random.default_rng(bx * 7 + by + crowd)
    n = 6 * 1024 + 17
    x = rng.integers(0, bx, n).astype(dt)
    y = rng.integers(0, by, n).astype(dt)
    for c in range(0, n, 1024):
        x[c], y[c], x[c + 1], y[c + 1] = 0, 0, bx - 1, by - 1
        if crowd and (c // 1024) % 2:
            at = c + 2 + rng.permutation(1022)[:crowd]
            at = at[at < n]
            x[at], y[at] = bx // 3, by // 2
    x += (rng.random(n) * 0.25).astype(dt) * (x < bx - 1) * (x > 0)
    check([x, y], 0.5, 1)


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("shift", [1, 2, 3])
def test_misaligned_axes(bits, shift):
    dt = np.float32 if bits == 32 else np.float64
    rng = np.random.default_rng(shift)
    check([(rng.random(40 * 1024 + 5) * 100).astype(dt) for _ in range(3)], 0.05, 4, shift)


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n", [1, 255, 256, 257, 1279, 1280, 1281, 2303, 2304, 5003, 16383, 16384, 16385])
@pytest.mark.parametrize("rel", [1e-2, 1e-4])
def test_automatic_segment_size_of_small_snapshots(bits, dim, n, rel):
    """The one-block sampling (up to 16,384 points, scratch not cleared) against the oracle's windows."""
    dt = np.float32 if bits == 32 else np.float64
    rng = np.random.default_rng(n + dim)
    axes = [(5.0 + 10.0 ** d * rng.random(n)).astype(dt) for d in range(dim)]
    axes[0][-1] = 400.0  # outside the last window of many sizes
    z = axes[2] if dim == 3 else np.zeros_like(axes[0])
    relT = float(dt(rel))
    eb = po.rel_to_abs(axes[0], axes[1], z if dim == 3 else None, relT)
    dev = [torch.from_numpy(a).cuda() for a in axes]
    got_eb, _ = gz.rel_to_abs(dev[0], dev[1], dev[2] if dim == 3 else None, relT)
    assert got_eb == eb
    if eb == 0.0:  # one point in 3D: no range, no bound to compress with
        return
    seg, _ = po.seg_size(axes[0], axes[1], z, dim, 0, True, relT, eb)
    want = po.compress(axes[0], axes[1], z, dim, eb, seg)
    out = torch.zeros(gz.stream_bound(n, dim, bits), dtype=torch.uint8, device="cuda")
    scratch = torch.full((gz.compress_scratch_bytes(n),), 255, dtype=torch.uint8, device="cuda")
    p = gz.make_params(n, dim, bits, eb, rel_mode=True, rel_eb=relT)
    for _ in range(2):
        r = gz.compress_into(p, dev[0], dev[1], dev[2] if dim == 3 else dev[0], out, scratch)
        assert (r.status, r.seg_size) == (0, seg)
        assert out[: r.stream_bytes].cpu().numpy().tobytes() == want
