"""The Gray walk by positive-gain words against the oracle's position-by-position
walk, bit for bit on integer weights: sizes around the 64-node blocks and the
32-iteration steps, from random states (many flips) and from local optima."""

import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [3, 24, 63, 64, 65, 96, 127, 129, 500, 1000, 2113])
@pytest.mark.parametrize("descend", [False, True])
def test_gray_walk_matches_oracle(n, descend):
    from pyqrackising_b200 import device as D

    rng = np.random.default_rng(n)
    U = np.triu(rng.integers(-3, 4, (n, n)), 1).astype(np.float32)
    W = U + U.T
    dg = D.DeviceGraph(W)
    words = dg.pack(rng.random(n) < 0.5)
    _, g64 = dg.gains(words)
    if descend:
        dg.single_descent(words, g64, True, *D.geometry(min(D.WORK_GROUP_MULTIPLE, n), n, 148), 4 * n)
    th = dg.unpack(words)[0]
    for S, T in ((1, 70), (3, 100), (148, 148 * 5 + 3 if n < 2000 else 300)):
        tout, eout = dg.gray(words, g64, True, T, S)
        rt, rE = O.gray(W, O.pack64(th), 1, T, S)[:2]
        assert np.array_equal(tout.cpu().numpy().view(np.uint64).reshape(S, -1), rt)
        assert np.array_equal(eout.cpu().numpy(), rE)
