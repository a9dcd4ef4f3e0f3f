"""The sampler's pick at the end of the running sums. The warp's prefixes are summed
in different orders, so for a draw next to 1 a lane without nodes can be above the
point drawn by a rounding, or the remainder in the last lane can pass its last node.
Weights for which that happens are found with a host restatement of the sums, and
the seed that makes the draw by inverting its hash; every form then takes node 0, as
where no prefix is above the point, and goes on with node 0's row."""

import ctypes

import numpy as np
import pytest
import torch

from pyqrackising_b200 import _lib
from pyqrackising_b200 import device as D

M64 = (1 << 64) - 1
SHOT, ROUND = 1, 2  # shot 1 starts at node 1


def _mix(z):
    z = (z + 0x9E3779B97F4A7C15) & M64
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & M64
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & M64
    return z ^ (z >> 31)


def _unshift(z, k):
    x = z
    for _ in range(64 // k + 1):
        x = z ^ (x >> k)
    return x


def _unmix(z):
    z = _unshift(z, 31)
    z = _unshift((z * pow(0x94D049BB133111EB, -1, 1 << 64)) & M64, 27)
    z = _unshift((z * pow(0xBF58476D1CE4E5B9, -1, 1 << 64)) & M64, 30)
    return (z - 0x9E3779B97F4A7C15) & M64


_SHOT_KEY = _mix((ROUND * 0x632BE59BD9B4E019 + SHOT) & M64)


def _draw(seed, d):
    return (_mix(_mix(seed ^ _SHOT_KEY) ^ ((d * 0xD1B54A32D192ED03) & M64)) >> 11) / 2.0**53


def _seed_for(low):
    """The seed whose first pick's draw is 1 - 2^-53, varied by the hash's low bits."""
    return _unmix(_unmix(M64 ^ low) ^ 0xD1B54A32D192ED03) ^ _SHOT_KEY


def _tree(x):
    return x[0] if len(x) == 1 else _tree(x[: (len(x) + 1) // 2]) + _tree(x[(len(x) + 1) // 2:])


def _lane_sums(form, w, n):
    """(nodes per lane, the 32 lanes' sums in the form's order of additions)"""
    if form == "shared":
        C = (n + 31) // 32
        x = np.zeros(32 * C)
        x[:n] = w
        x = x.reshape(32, C)
        a = np.zeros((4, 32))
        for i in range(C):
            a[i & 3 if i < C // 4 * 4 else 0] += x[:, i]
        return C, (a[0] + a[1]) + (a[2] + a[3])
    if form in ("bits", "table"):
        C = ((n + 31) // 32 + 7) // 8 * 8
        x = np.zeros(32 * C)
        x[:n] = w
        g = x.reshape(32, C // 8, 8)
        g = ((g[..., 0] + g[..., 1]) + (g[..., 2] + g[..., 3])) + ((g[..., 4] + g[..., 5]) + (g[..., 6] + g[..., 7]))
        return C, _tree([g[:, i] for i in range(C // 8)])
    GP = 1 if n <= 1024 else 2
    x = np.zeros(1024 * GP)
    x[:n] = w
    g = x.reshape(32 * GP, 32)
    if form == "codes":
        g = g.reshape(-1, 8, 4)
        y = (g[..., 0] + g[..., 1]) + (g[..., 2] + g[..., 3])
    else:
        g = g.reshape(-1, 4, 8)
        y = (g[:, 0] + g[:, 1]) + (g[:, 2] + g[:, 3])
    for o in (1, 2, 4):
        y = y + y[:, np.arange(8) ^ o]
    return 32 * GP, _tree([y[:, 0].reshape(32, GP)[:, i] for i in range(GP)])


def _unguarded_pick(form, w, n):
    """Where the sums alone lead for the draw 1 - 2^-53 (None: to a node)."""
    per, loc = _lane_sums(form, w, n)
    incl = loc.copy()
    for o in (1, 2, 4, 8, 16):
        incl[o:] = incl[o:] + incl[:-o]
    p = incl[31] * (1.0 - 2.0**-53)
    owner = int(np.argmax(p < incl))
    if not p < incl[owner]:
        return None
    if per * owner >= n:
        return per * owner
    if n < 8 and form in ("bits", "table"):  # one lane holds all: the halving of its eight slots
        x = np.zeros(8)
        x[:n] = w
        lo, N, q = 0, 8, p
        while N > 1:
            m = _tree(list(x[lo:lo + N // 2]))
            if not q < m:
                q, lo = q - m, lo + N // 2
            N //= 2
        if lo >= n:
            return lo
    return None


def _weights(form, n, rng):
    """Symmetric weights that the form takes."""
    U = np.zeros((n, n), dtype=np.float32)
    if form in ("codes", "lists"):
        for k in (1, 7, 12):
            i = np.arange(n)
            U[i, (i + k) % n] = rng.choice([-1.0, 1.0], n) if form == "codes" else rng.standard_normal(n)
    elif form == "bits":
        U = (rng.random((n, n)) < 0.5).astype(np.float32)
    else:
        U = rng.standard_normal((n, n)).astype(np.float32)
    U = np.triu(U, 1) + np.tril(U, -1).T
    U = np.triu(U, 1)
    return (U + U.T).astype(np.float32)


def _numpy_factors(row, base):
    return np.where(row == 0, 1.0, np.exp(-np.log(base) * row.astype(np.float64)))


def _find(form, n, factors):
    """Weights and a base for which shot 1's first pick is led past the last node."""
    rng = np.random.default_rng(n)
    for _ in range(400):
        W = _weights(form, n, rng)
        for base in 1.5 + 4.0 * rng.random(8):
            w = np.ones(n)
            w[SHOT] = 0.0
            w = w * factors(W[SHOT], base)
            led = _unguarded_pick(form, w, n)
            if led is not None:
                return W, base, w, led
    raise AssertionError("no case found")


FORMS = [("bits", 100), ("table", 100), ("table", 7), ("codes", 300), ("codes", 1100), ("lists", 1100), ("shared", 100)]


@pytest.mark.parametrize("form,n", FORMS)
def test_sums_can_lead_past_the_last_node(form, n):
    W, base, w, led = _find(form, n, _numpy_factors)
    assert led >= n
    for low in range(8):
        assert _draw(_seed_for(low), 1) == 1.0 - 2.0**-53


@pytest.mark.gpu
@pytest.mark.parametrize("form,n", FORMS)
def test_pick_stays_within_the_nodes(form, n):
    def factors(row, base):  # as the device computes them
        r = torch.from_numpy(row).cuda().double()
        lnb = torch.log(torch.tensor(base, dtype=torch.float64, device="cuda"))
        f = torch.where(r == 0, torch.ones_like(r), torch.exp(-lnb * r))
        return f.cpu().numpy()

    W, base, w, led = _find(form, n, factors)
    assert led >= n
    # node 0 next, then a second pick by an ordinary draw, well inside a node's share
    w = w.copy()
    w[0] = 0.0
    w = w * factors(W[0], base)
    cum = np.cumsum(w)
    for low in range(2048):
        seed = _seed_for(low)
        p = cum[-1] * _draw(seed, 2)
        pick = int(np.argmax(p < cum))
        if min(cum[pick] - p, p - (cum[pick] - w[pick])) > 0.1 * w[pick]:
            break
    else:
        raise AssertionError("no second draw found")
    words = np.zeros((n + 31) // 32, dtype=np.uint32)
    for v in (SHOT, 0, pick):
        words[v >> 5] |= np.uint32(1 << (v & 31))
    dist = np.where(np.arange(n - 1) < 3, 0.0, 1.0)  # Hamming-weight index 3: two picks
    dW = torch.from_numpy(W).cuda()
    dcum = torch.from_numpy(dist).cuda()
    out = torch.zeros(2 * len(words), dtype=torch.int32, device="cuda")
    size = 1024 if form == "shared" else _lib.load().pqi_tfim_sample_workspace_bytes(n)
    ws = torch.empty(size, dtype=torch.uint8, device="cuda")
    _lib.call("pqi_tfim_sample", D._ptr(dW), n, D._ptr(dcum), float(base), ctypes.c_uint64(seed), ctypes.c_uint64(ROUND), 2,
              D._ptr(out), D._ptr(ws), ctypes.c_size_t(ws.numel()), D.stream_ptr())
    assert np.array_equal(out.cpu().numpy().view(np.uint32)[len(words):], words)
