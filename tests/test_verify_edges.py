"""gpz_verify over the forms its ranking takes (narrow, wide, radix, crowded,
short last chunk, misaligned axes) against a host computation over the oracle's
block order."""
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
@pytest.mark.parametrize("dim", [2, 3])
@pytest.mark.parametrize("n,blocks,crowd,shift", [(1, 4, 0, 0), (1000, 4, 0, 0), (1025, 300, 0, 1), (40_000, 40, 0, 0),
                                                  (40_000, 120, 20, 0), (40_000, 1500, 0, 0), (9_216, 120, 300, 2)])
def test_pairs_points_with_their_reconstruction(bits, dim, n, blocks, crowd, shift):
    """Blocks of size 1 (eb 1/16, seg 8) and integer coordinates: the chunk's block ids are
    x + y bnx + z bnx bny of the offsets from its minimum (31 bits kept, as the stream
    does), and equal ids keep the order of the ranks."""
    dt = np.float32 if bits == 32 else np.float64
    rng = np.random.default_rng(n + blocks + dim)
    axes = [rng.integers(0, blocks, n).astype(dt) for _ in range(dim)]
    if crowd:
        for c in range(0, n, 1024):
            at = c + rng.permutation(min(1024, n - c))[:crowd]
            for a in axes:
                a[at] = blocks // 2
    err = rng.choice([0.0, 0.03125, 0.0625, 0.0703125, 0.125], size=(dim, n)).astype(dt)  # exact in both types
    rec = []
    for c in range(0, n, 1024):
        sl = [a[c:c + 1024] for a in axes]
        ids, mul = np.zeros(sl[0].size, np.uint64), 1
        for s in sl:
            ids += (s - s.min()).astype(np.uint64) * np.uint64(mul)
            mul *= int(s.max() - s.min()) + 1
        p = np.arange(sl[0].size)
        order = np.lexsort(((p % 32) * 32 + p // 32, ids & np.uint64(0x7FFFFFFF)))
        rec.append([s[order] for s in sl])
    back = [np.concatenate([r[d] for r in rec]) for d in range(dim)]
    want_max = [float(np.abs(err[d]).max()) for d in range(dim)]
    got = [(b + e).astype(dt) for b, e in zip(back, err)]
    put = []
    for a in axes + got:
        buf = torch.zeros(n + shift, dtype=torch.float32 if bits == 32 else torch.float64, device="cuda")
        buf[shift:] = torch.from_numpy(a).cuda()
        put.append(buf[shift:])
    x, y, z = put[0], put[1], put[2] if dim == 3 else None
    rx, ry, rz = put[dim], put[dim + 1], put[dim + 2] if dim == 3 else None
    v = gz.verify(x, y, z, rx, ry, rz, 0.0625, 8)
    assert v.points == n
    assert list(v.max_abs_err[:dim]) == want_max
    assert v.over_bound == int((np.abs(err) > 0.0625).any(0).sum())
    assert v.over_bound_tol == int((np.abs(err) > dt(np.float32(1.01)) * dt(0.0625)).any(0).sum())
    for d in range(dim):
        # squares of multiples of 1/128 sum exactly in double
        assert v.mse[d] == float((err[d].astype(np.float64) ** 2).sum()) / n
        assert v.value_range[d] == float(axes[d].max() - axes[d].min())
