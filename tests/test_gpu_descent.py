"""The device-resident descent against a step-for-step restatement on the host
(float64 gains updated in the same order, the reference's selection), bit for
bit: one warp, one CTA and cluster launches, at the sizes where the split
changes or leaves a remainder, both weight kinds, cut short and run out."""

import numpy as np
import pytest
import torch

from oracle import oracle as O

pytestmark = pytest.mark.gpu


def _descend(W, bits, g, spin, G, L, limit):
    bits, g, trace, total, rc = bits.copy(), g.copy(), [], 0.0, 0
    while True:
        v = g.astype(np.float32) * np.float32(2.0 if spin else 1.0)
        val, k = O.select(v, G, L)
        if not val > 0:
            break
        if len(trace) >= limit:
            rc = 3
            break
        total += float(val)
        trace.append(int(k))
        w2 = 2.0 * W[k].astype(np.float64)
        gk = -g[k]
        g += np.where(bits == bits[k], -w2, w2)
        g[k] = gk
        bits[k] = not bits[k]
    return bits, g, trace, total, rc


@pytest.mark.parametrize("kind", ["int", "float"])
@pytest.mark.parametrize("n", [3, 31, 33, 127, 128, 129, 511, 1000, 2047, 2048, 2049, 4101, 8191, 8193, 16500])
def test_descent_follows_the_reference_steps(kind, n):
    from pyqrackising_b200 import device as D

    rng = np.random.default_rng(n)
    U = (rng.random((n, n), dtype=np.float32) < 0.5).astype(np.float32) if kind == "int" else rng.standard_normal((n, n), dtype=np.float32)
    U = np.triu(U, 1)
    W = U + U.T
    del U
    dg = D.DeviceGraph(W)
    bits = rng.random(n) < 0.5
    G, L = D.geometry(min(D.WORK_GROUP_MULTIPLE, n), n, 148)
    for spin, limit in ((True, 40), (False, 4 * n if n <= 600 else 7)):
        words = dg.pack(bits)
        _, g64 = dg.gains(words)
        want = _descend(W, bits, g64.cpu().numpy(), spin, G, L, limit)
        trace = torch.full((limit,), -1, dtype=torch.int32, device=dg.device)
        esum, flips, rc = dg.single_descent(words, g64, spin, G, L, limit, trace)
        nf = int(flips.item())
        assert rc == want[4]
        assert trace[:nf].tolist() == want[2]
        assert float(esum.item()) == want[3]
        assert np.array_equal(dg.unpack(words)[0], want[0])
        assert np.array_equal(g64.cpu().numpy(), want[1])
