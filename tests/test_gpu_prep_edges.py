"""Weight preparation at the sizes where its 32 x 32 tile pairs and groups of four
end, against the definition in numpy: classification counts, the maximum, the
upper sum, the padded copies and the digit planes, scaled where float32 cannot
hold 2^S too."""

import numpy as np
import pytest

from pyqrackising_b200 import device as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 31, 32, 33, 63, 65, 126, 129, 1027])
@pytest.mark.parametrize("kind,scale", [("int", 1.0), ("float", 1.0), ("float", 2.0**-120), ("float", 2.0**100)])
def test_prepared_copies(kind, scale, n):
    rng = np.random.default_rng(n)
    U = rng.integers(-5, 6, (n, n)) if kind == "int" else rng.standard_normal((n, n))
    U = np.triu(U * scale, 1).astype(np.float32)
    W = U + U.T
    dg = D.DeviceGraph(W)
    ld = dg.w.ld
    up = W[np.triu_indices(n, 1)].astype(np.float64)
    # (a sum of k float64 terms: k roundings of the sum of magnitudes at most)
    assert abs(dg.w.upper_sum - up.sum()) <= len(up) * 2.0**-52 * np.abs(up).sum()
    assert dg.stats.nonint == np.count_nonzero(W != np.rint(W))
    assert dg.stats.maxabs == (np.abs(W).max() if n else 0.0)
    pad = np.zeros((n, ld), np.float32)
    pad[:, :n] = W
    np.testing.assert_array_equal(dg.W_f32z.cpu().numpy().reshape(n, ld), pad)
    if dg.W_i8 is not None:
        np.testing.assert_array_equal(dg.W_i8.cpu().numpy().reshape(n, ld), pad.astype(np.int8))
    if getattr(dg, "W_d", None) is not None:
        v = np.rint(pad.astype(np.float64) / dg.w.wscale).astype(np.int64)
        planes = dg.W_d.cpu().numpy().reshape(4, n, ld).astype(np.int64)
        np.testing.assert_array_equal(((planes[0] * 256 + planes[1]) * 256 + planes[2]) * 256 + planes[3], v)
