"""The grid-wide min / max behind gpz_rel_to_abs (16-byte loads with ragged and
misaligned ends) against numpy, exactly: NaNs ignored, -0.0 below +0.0."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import gpz_b200 as gz  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    gz.lib()


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("n", [1, 3, 4, 5, 1023, 4095, 4097, 70_001, 4_000_003])
@pytest.mark.parametrize("shift", [0, 1, 3])
def test_minmax_matches_numpy(bits, n, shift):
    dt = np.float32 if bits == 32 else np.float64
    rng = np.random.default_rng(n * 8 + shift)
    axes = [(rng.standard_normal(n + shift) * 10 ** k).astype(dt) for k in range(3)]
    if n >= 5:
        axes[0][shift + n - 1] = 1e9     # extremes in the ragged ends
        axes[0][shift] = -1e9
        axes[1][shift + 1] = np.nan
        axes[2][shift:] = 0.0
        axes[2][shift + n // 2] = -0.0
    dev = [torch.from_numpy(a).cuda()[shift:] for a in axes]
    for dim in (3, 2):
        eb, mm = gz.rel_to_abs(dev[0], dev[1], dev[2] if dim == 3 else None, 1e-3)
        want_min = [np.nanmin(a[shift:]) for a in axes[:dim]] + [dt(0)] * (3 - dim)
        want_max = [np.nanmax(a[shift:]) for a in axes[:dim]] + [dt(0)] * (3 - dim)
        assert mm == [float(v) for v in want_min + want_max]
        if dim == 3 and n >= 5:
            assert np.signbit(mm[2]) and not np.signbit(mm[5])
        spans = [hi - lo for lo, hi in zip(want_min, want_max)]
        assert eb == float(dt(max(spans)) * dt(1e-3))


@pytest.mark.parametrize("bits", [32, 64])
def test_axis_without_numbers(bits):
    dt = torch.float32 if bits == 32 else torch.float64
    x = torch.full((5000,), float("nan"), dtype=dt, device="cuda")
    y = torch.full((5000,), float("inf"), dtype=dt, device="cuda")
    z = torch.full((5000,), float("-inf"), dtype=dt, device="cuda")
    _, mm = gz.rel_to_abs(x, y, z, 1e-3)
    big = float(np.finfo(np.float32).max)
    # the reference's scan starts from the float limits
    assert mm == [big, big, float("-inf"), -big, float("inf"), -big]
