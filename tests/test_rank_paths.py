"""Where the encoder's ranking changes form, byte for byte against the oracle:
id counts on both sides of one radix pass (512), of the bucket count (1024) and
of 32-bit composites (2^22), chunks without a crowd, with one that a bucket
still takes, and with ones that it does not (one place, many places)."""
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


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("bx,by", [(511, 1), (512, 1), (513, 1), (514, 1), (27, 19), (1022, 1), (1023, 1), (1024, 1),
                                   (1025, 1), (2047, 1), (600, 600), (2047, 2049), (2048, 2048), (65, 65000), (2, 2097153)])
@pytest.mark.parametrize("crowd,places", [(0, 1), (200, 1), (257, 1), (600, 1), (600, 30), (1000, 3), (1020, 60)])
def test_ranking_forms(bits, bx, by, crowd, places):
    """2D grids of bx * by blocks of size 1 (both corners in every chunk); `crowd` points
    of most chunks in `places` blocks, several chunks in a row and single ones."""
    dt = np.float32 if bits == 32 else np.float64
    rng = np.random.default_rng(bx * 31 + by + crowd + places)
    n = 24 * 1024 + 5
    x = rng.integers(0, bx, n).astype(dt)
    y = rng.integers(0, by, n).astype(dt)
    for c in range(0, n, 1024):
        m = min(1024, n - c)
        x[c], y[c], x[c + m - 1], y[c + m - 1] = 0, 0, bx - 1, by - 1
        if crowd and (c // 1024) % 5 != 2 and m == 1024:
            at = c + 1 + rng.permutation(1022)[:crowd]
            px, py = rng.integers(0, bx, places).astype(dt), rng.integers(0, by, places).astype(dt)
            k = rng.integers(0, places, at.size)
            x[at], y[at] = px[k], py[k]
    dx, dy = torch.from_numpy(x).cuda(), torch.from_numpy(y).cuda()
    z = np.zeros_like(x)
    seg, _ = po.seg_size(x, y, z, 2, 1, False, 0.0, 0.5)  # float32: doubled until block ids fit 32 bits
    want = po.compress(x, y, z, 2, 0.5, seg)
    for _ in range(2):
        s, r = gz.compress(dx, dy, None, eb=0.5, seg_size=1)
        assert (r.status, r.seg_size) == (0, seg) and s.cpu().numpy().tobytes() == want
    rx, ry, _ = gz.decompress(s)
    # a point paired with another block's reconstruction is off by 1 at least
    v = gz.verify(dx, dy, None, rx, ry, None, 0.5, seg)
    assert max(v.max_abs_err[:2]) <= 0.75 and v.points == n
