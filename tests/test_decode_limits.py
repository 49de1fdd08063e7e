"""Double chunks whose quantized values lie on both sides of the decoder's 32-bit
form (2.0e9 on z, 2^31 on x and y), on every axis, bit for bit against the oracle."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

import gpz_b200 as gz  # noqa: E402
from oracle import pyoracle as po  # noqa: E402


@pytest.mark.parametrize("top", [1.9e9, 2.0e9 - 200, 2.0e9 + 200, 2.1e9, 2.0 ** 31 - 3, 2.0 ** 31 + 3, 2.2e9, 4.0e9, 5.0e9])
@pytest.mark.parametrize("dim,axis", [(2, 0), (2, 1), (3, 0), (3, 1), (3, 2)])
@pytest.mark.parametrize("seg", [1, 4, 64])
def test_tall_axis(top, dim, axis, seg):
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    if axis < dim - 1 and top / seg >= 2.0 ** 32:
        pytest.skip("the block count wraps to 0 in the format's decoder: 64-bit division by zero")
    rng = np.random.default_rng(int(top % 1e6) + axis + seg)
    n = 3 * 1024 + 5
    eb = 0.0625  # exact: quantized value = 8 x
    axes = [rng.random(n) * 2.0 for _ in range(dim)]
    axes[axis] = rng.random(n) * (top / 8.0)
    for c in range(0, n, 1024):  # the whole range in every chunk
        axes[axis][c], axes[axis][min(c + 1, n - 1)] = 0.0, top / 8.0
    z = axes[2] if dim == 3 else np.zeros(n)
    s = po.compress(axes[0], axes[1], z, dim, eb, seg)
    want = po.decompress(s)
    got = gz.decompress(torch.from_numpy(np.frombuffer(s, np.uint8).copy()).cuda())
    for a, b in zip(got[:dim], want[:dim]):
        assert np.array_equal(a.cpu().numpy(), b)
    if seg == 64:
        dev = [torch.from_numpy(a).cuda() for a in axes]
        t, r = gz.compress(dev[0], dev[1], dev[2] if dim == 3 else None, eb=eb, seg_size=seg)
        assert r.status == 0 and t.cpu().numpy().tobytes() == s
