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


def _row(kind, n, k):
    """Row k of symmetric weights given by a formula."""
    h = ((np.arange(n, dtype=np.uint64) ^ np.uint64(k)) * np.uint64(0x9E3779B97F4A7C15)) >> np.uint64(40)
    w = (h % np.uint64(7)).astype(np.float32) - 3.0 if kind == "int" else h.astype(np.float32) / 2.0**23 - 1.0
    w[k] = 0.0
    return w


def _walk(kind, n, bits, gains, spin, T, S):
    """The search step by step, with float64 gains updated flip by flip."""
    out, energies, flipped = [], [], set()
    th = O.pack64(bits).reshape(-1)
    for s in range(S):
        x, g, words, E = bits.copy(), gains.copy(), O.gray_seed(th, n, s), 0.0

        def flip(k):
            nonlocal E
            E += g[k]
            w2 = 2.0 * _row(kind, n, k).astype(np.float64)
            gk = -g[k]
            g[:] += np.where(x == x[k], -w2, w2)
            g[k] = gk
            x[k] = not x[k]
            flipped.add(k)

        for k in np.nonzero(O.unpack64(words, n) != bits)[0]:
            flip(int(k))
        pad = words ^ O.pack64(x).reshape(-1)  # seed bits past the last node
        for i in range(s, T, S):
            c = (i + 1 & -(i + 1)).bit_length() - 1
            for k in range(c, n, 64):
                if g[k] > 0:
                    flip(k)
        out.append(O.pack64(x).reshape(-1) ^ pad)
        energies.append(np.float32(E if spin else E / 2.0))
    return np.stack(out), np.array(energies, dtype=np.float32), flipped


@pytest.mark.parametrize("kind,n", [("float", 26501), ("int", 51003)])
@pytest.mark.parametrize("ctas", [1, 2])
def test_gains_in_global_memory(kind, n, ctas):
    """Graphs whose gains do not fit in shared memory; a workspace for fewer CTAs than
    seeds, so that a CTA's gains serve several seeds. Only flipped rows are filled in."""
    import ctypes

    import torch

    from pyqrackising_b200 import _lib
    from pyqrackising_b200 import device as D

    rng = np.random.default_rng(n)
    bits = rng.random(n) < 0.5
    # mostly below zero, so that the walk passes over whole iterations too
    gains = rng.integers(-3000, 40, n).astype(np.float64) if kind == "int" else rng.standard_normal(n) * 50.0 - 120.0
    S, T, spin = 5, 23, kind == "int"
    want = _walk(kind, n, bits, gains, spin, T, S)
    assert len(want[2]) > 20
    torch.cuda.empty_cache()
    ld = int(_lib.load().pqi_padded_ld(n))
    M = torch.empty((n, ld), dtype=torch.int8 if kind == "int" else torch.float32, device="cuda")
    for k in want[2]:
        M[k].zero_()
        M[k, :n] = torch.from_numpy(_row(kind, n, k)).cuda().to(M.dtype)
    w = _lib.PqiWeights()
    w.n, w.ld = n, ld
    if kind == "int":
        w.kind, w.W_i8 = 1, M.data_ptr()
    else:
        w.kind, w.W_f32z = 0, M.data_ptr()
    theta = torch.from_numpy(O.pack64(bits).reshape(-1).view(np.int64)).cuda()
    g64 = torch.from_numpy(gains).cuda()
    tout = torch.zeros((S, theta.numel()), dtype=torch.int64, device="cuda")
    eout = torch.zeros(S, dtype=torch.float32, device="cuda")
    ws = torch.empty(ctas * n * (4 if kind == "int" else 8) + 512, dtype=torch.uint8, device="cuda")
    _lib.call("pqi_gray", ctypes.byref(w), D._ptr(theta), D._ptr(g64), int(spin), T, S, D._ptr(tout), D._ptr(eout),
              D._ptr(ws), ctypes.c_size_t(ws.numel()), D.stream_ptr())
    got = tout.cpu().numpy().view(np.uint64), eout.cpu().numpy()
    del M
    torch.cuda.empty_cache()
    assert np.array_equal(got[0], want[0])
    assert np.array_equal(got[1], want[1])
