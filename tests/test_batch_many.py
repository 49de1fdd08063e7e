"""Batches of more snapshots than one and two steps of the search over a class's
work list find (32, 1024), and failed snapshots between good ones: each good
snapshot's stream equals a single call's."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import gpz_b200 as gz  # noqa: E402
from gpz_b200.batch import Batch, Snapshot  # noqa: E402


@pytest.fixture(scope="module", autouse=True)
def _cuda():
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    gz.lib()


def _single(axes, eb, seg):
    s, r = gz.compress(axes[0], axes[1], axes[2] if len(axes) == 3 else None, eb=eb, seg_size=seg)
    assert r.status == 0
    return s.cpu().numpy().tobytes()


def _axes(rng, n, dim, bits):
    return [torch.from_numpy((rng.random(n) * 50).astype(np.float32 if bits == 32 else np.float64)).cuda()
            for _ in range(dim)]


@pytest.mark.parametrize("count", [31, 32, 33, 1023, 1024, 1025, 1100])
def test_many_snapshots_of_one_class(count):
    rng = np.random.default_rng(count)
    data = [_axes(rng, int(rng.choice([1, 700, 1024, 1025, 2100, 5000])), 3, 32) for _ in range(count)]
    b = Batch([Snapshot(*a, eb=0.0625, rel_mode=False, seg_size=8) for a in data])
    try:
        b.launch()
        for a, s in zip(data, b.streams()):
            assert s.cpu().numpy().tobytes() == _single(a, 0.0625, 8)
    finally:
        b.close()


@pytest.mark.parametrize("bits", [32, 64])
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("bad_points", [900, 70_000, 1_500_000])
def test_failed_snapshots_between_good_ones(bits, dim, bad_points):
    """The failed ones (no segment size in absolute mode) are skipped by CTAs that hold parked payloads
    of the good ones on either side; several launches."""
    rng = np.random.default_rng(bad_points + dim + bits)
    sizes = [3_000, bad_points, 250_000, bad_points, 1_200_000, 1, bad_points, 40_001]
    data = [_axes(rng, n, dim, bits) for n in sizes]
    snaps = [Snapshot(a[0], a[1], a[2] if dim == 3 else None, eb=0.0625, rel_mode=False, seg_size=0 if n == bad_points else 8)
             for a, n in zip(data, sizes)]
    want = [None if n == bad_points else _single(a, 0.0625, 8) for a, n in zip(data, sizes)]
    b = Batch(snaps)
    try:
        for _ in range(3):
            b.launch()
            for (r, _), s, w in zip(b.results(), snaps, want):
                if w is None:
                    assert r.status != 0
                else:
                    assert r.status == 0 and s.out[: r.stream_bytes].cpu().numpy().tobytes() == w
    finally:
        b.close()
