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


class _Rows:
    """Symmetric weights by formula, one row at a time."""

    def __init__(self, kind, n):
        self.kind, self.n = kind, n

    def __getitem__(self, k):
        h = ((np.arange(self.n, dtype=np.uint64) ^ np.uint64(k)) * np.uint64(0x9E3779B97F4A7C15)) >> np.uint64(40)
        w = (h % np.uint64(7)).astype(np.float32) - 3.0 if self.kind == "int" else h.astype(np.float32) / 2.0**23 - 1.0
        w[k] = 0.0
        return w


@pytest.mark.parametrize("kind,n", [("int", 33001), ("float", 33001), ("int", 66001), ("float", 66001),
                                    ("int", 131075), ("int", 262148)])
def test_descent_on_the_largest_graphs(kind, n):
    """Two to sixteen groups of nodes per thread (past 32768, 65536, 131072 and 262144
    nodes on clusters of sixteen), a few flips from gains as given. Only the rows of the
    flipped nodes are read, so only they are filled in (the last matrix has 69 GB)."""
    import ctypes

    from pyqrackising_b200 import _lib
    from pyqrackising_b200 import device as D

    rng = np.random.default_rng(n)
    W, limit, spin = _Rows(kind, n), 12, True
    bits = rng.random(n) < 0.5
    g = rng.integers(-40, 40, n).astype(np.float64) if kind == "int" else rng.standard_normal(n)
    G, L = D.geometry(min(D.WORK_GROUP_MULTIPLE, n), n, 148)
    want = _descend(W, bits, g, spin, G, L, limit)
    assert len(want[2]) == limit
    torch.cuda.empty_cache()
    ld = int(_lib.load().pqi_padded_ld(n))
    M = torch.empty((n, ld), dtype=torch.int8 if kind == "int" else torch.float32, device="cuda")
    for k in set(want[2]):
        M[k].zero_()
        M[k, :n] = torch.from_numpy(W[k]).cuda().to(M.dtype)
    w = _lib.PqiWeights()
    w.n, w.ld = n, ld
    if kind == "int":
        w.kind, w.W_i8 = 1, M.data_ptr()
    else:
        w.kind, w.W_f32z = 0, M.data_ptr()
    words = torch.from_numpy(O.pack32(bits).reshape(-1).view(np.int32)).cuda()
    g64 = torch.from_numpy(g).cuda()
    esum = torch.zeros(1, dtype=torch.float64, device="cuda")
    flips = torch.zeros(1, dtype=torch.int32, device="cuda")
    trace = torch.full((limit,), -1, dtype=torch.int32, device="cuda")
    ws = torch.empty(4096, dtype=torch.uint8, device="cuda")
    rc = _lib.status("pqi_single_descent", ctypes.byref(w), D._ptr(words), D._ptr(g64), int(spin), G, L, limit, D._ptr(esum),
                     D._ptr(flips), D._ptr(trace), D._ptr(ws), ctypes.c_size_t(ws.numel()), D.stream_ptr())
    got = words.cpu().numpy().view(np.uint32), g64.cpu().numpy()
    del M
    torch.cuda.empty_cache()
    assert rc == want[4] == 3
    assert trace.tolist() == want[2] and int(flips.item()) == limit
    assert float(esum.item()) == want[3]
    assert np.array_equal(got[0], O.pack32(want[0]).reshape(-1))
    assert np.array_equal(got[1], want[1])
