"""Decoder sections at their edges: run counts around the lengths where a
plane's last word comes from the plane behind (992..1024 runs, every alignment),
delta and relative-position widths on both sides of 8, 16 and 32 planes.  The
streams are the oracle's; the reconstruction must be the oracle's bits."""
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
@pytest.mark.parametrize("span", [2_000, 200_000, 20_000_000, 2_000_000_000])
@pytest.mark.parametrize("runs", [1, 31, 33, 500, 991, 992, 993, 997, 1002, 1007, 1016, 1017, 1023, 1024])
def test_run_counts_and_delta_widths(bits, span, runs):
    """2D chunks of `runs` distinct blocks spread over `span` block ids."""
    dt = np.float32 if bits == 32 else np.float64
    rng = np.random.default_rng(runs * 11 + span % 97)
    n = 3 * 1024 + 77
    side = int(np.sqrt(span))
    x, y = np.empty(n, dt), np.empty(n, dt)
    for c in range(0, n, 1024):
        m = min(1024, n - c)
        k = min(runs, m)
        ids = rng.choice(side * side, size=k, replace=False)
        pick = np.concatenate([np.arange(k), rng.integers(0, k, m - k)])
        rng.shuffle(pick)
        x[c:c + m], y[c:c + m] = ids[pick] % side, ids[pick] // side
    s = po.compress(x, y, np.zeros_like(x), 2, 0.5, 1)
    ox, oy, _ = po.decompress(s)
    dx, dy, _ = gz.decompress(torch.from_numpy(np.frombuffer(s, np.uint8).copy()).cuda())
    assert np.array_equal(dx.cpu().numpy(), ox) and np.array_equal(dy.cpu().numpy(), oy)


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("seg", [1, 4, 8, 32, 64, 512, 1024])
def test_relative_position_widths(bits, seg):
    dt = np.float32 if bits == 32 else np.float64
    rng = np.random.default_rng(seg)
    axes = [(rng.random(5 * 1024 + 3) * 30_000).astype(dt) for _ in range(3)]
    s = po.compress(*axes, 3, 0.5 if seg > 64 else 50.0, seg)
    want = po.decompress(s)
    got = gz.decompress(torch.from_numpy(np.frombuffer(s, np.uint8).copy()).cuda())
    for a, b in zip(got, want):
        assert np.array_equal(a.cpu().numpy(), b)


@pytest.mark.parametrize("scale", [1.0, 1e3, 1e6])
@pytest.mark.parametrize("flat", [0, 1])
def test_double_quantized_values_around_2_to_the_31(scale, flat):
    """Double 2D chunks whose quantized values pass 2^31 on one axis while the block counts' product stays in 32 bits."""
    rng = np.random.default_rng(int(scale) + flat)
    n = 2 * 1024 + 5
    long = rng.random(n) * 1500.0 * scale
    short = rng.random(n) * 1e-3
    x, y = (short, long) if flat else (long, short)
    s = po.compress(x, y, np.zeros_like(x), 2, 2.5e-4, 64)
    ox, oy, _ = po.decompress(s)
    dx, dy, _ = gz.decompress(torch.from_numpy(np.frombuffer(s, np.uint8).copy()).cuda())
    assert np.array_equal(dx.cpu().numpy(), ox) and np.array_equal(dy.cpu().numpy(), oy)
