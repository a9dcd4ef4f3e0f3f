"""The sampler's register and sparse forms draw the same candidates as the
shared-memory form (reached by a workspace too small for their tables), bit for
bit: sizes at the edges of the lanes' chunks and of the packed words, weights of
each kind, with and without repulsion, row degrees around the sparse limits."""

import ctypes
import importlib

import numpy as np
import pytest
import torch

from pyqrackising_b200 import _lib
from pyqrackising_b200 import device as D

pytestmark = pytest.mark.gpu

MT = importlib.import_module("pyqrackising_b200.maxcut_tfim")


def _weights(kind, n, rng):
    if kind == "unit":
        U = (rng.random((n, n)) < 0.5).astype(np.float32)
    elif kind == "pm1":
        U = rng.choice(np.array([-1.0, 0.0, 1.0], dtype=np.float32), (n, n))
    elif kind == "float":
        U = rng.standard_normal((n, n)).astype(np.float32)
    elif kind == "tenth":
        U = np.where(rng.random((n, n)) < 0.1, rng.random((n, n)), 0.0).astype(np.float32)
    else:  # rings of degree 2 d: +-1 ("ringD"), or +-1 with some other weights ("mixD")
        d = int(kind[4:] if kind.startswith("ring") else kind[3:])
        U = np.zeros((n, n), dtype=np.float32)
        for k in range(1, d + 1):
            i = np.arange(n)
            U[i, (i + k) % n] = rng.choice(np.array([-1.0, 1.0], dtype=np.float32), n)
            if kind.startswith("mix"):
                U[i[::5], (i[::5] + k) % n] = 0.5
        U = np.triu(U, 1) + np.tril(U, -1).T
    U = np.triu(U, 1)
    return (U + U.T).astype(np.float32)


def _draw(dg, cum, shots, base, seed, ws):
    out = torch.zeros(shots * dg.n32 + 1, dtype=torch.int32, device=dg.device)
    _lib.call("pqi_tfim_sample", D._ptr(dg.W), dg.n, D._ptr(cum), float(base), ctypes.c_uint64(seed),
              ctypes.c_uint64(2), shots, D._ptr(out), D._ptr(ws), ctypes.c_size_t(ws.numel()), dg.sp())
    return out


@pytest.mark.parametrize("kind,n", [
    ("unit", 24), ("unit", 255), ("unit", 257), ("unit", 513), ("unit", 1024), ("unit", 1025), ("unit", 1537),
    ("unit", 2048), ("pm1", 31), ("pm1", 300), ("pm1", 777), ("pm1", 1793), ("float", 33), ("float", 256),
    ("float", 769), ("float", 1281), ("float", 2047), ("tenth", 1500), ("tenth", 100),
    ("ring1", 64), ("ring1", 258), ("ring3", 1024), ("ring3", 1025), ("ring3", 2048), ("ring4", 1100), ("ring4", 400),
    ("mix3", 2001), ("mix7", 1500), ("mix8", 1500), ("mix3", 600)])
def test_forms_draw_the_same_candidates(kind, n):
    dg = D.DeviceGraph(_weights(kind, n, np.random.default_rng(n)))
    _, _, cum = MT.hamming_cdf(dg, 2, 8.0, 8.0)
    full = torch.empty(_lib.load().pqi_tfim_sample_workspace_bytes(n), dtype=torch.uint8, device=dg.device)
    small = torch.empty(1024, dtype=torch.uint8, device=dg.device)
    for shots, base in ((3, 5.0), (257, 5.0), (130, 1.0), (64, 0.25)):
        a = _draw(dg, cum, shots, base, 11, full)
        b = _draw(dg, cum, shots, base, 11, small)
        assert torch.equal(a, b), (shots, base)


@pytest.mark.parametrize("n,kind", [(300, "column"), (1500, "column"), (300, "ring"), (1100, "ring")])
def test_weights_need_not_be_symmetric(n, kind):
    """A bare W: every row has at most three +-1 entries, one column has one in
    every row ("column"), or the entries of a ring run one way ("ring")."""
    rng = np.random.default_rng(n)
    i = np.arange(n)
    W = np.zeros((n, n), dtype=np.float32)
    for k in (1, 5):
        W[i, (i + k) % n] = rng.choice(np.array([-1.0, 1.0], dtype=np.float32), n)
    if kind == "column":
        W[:, 7] = 1.0
    np.fill_diagonal(W, 0.0)
    sym = D.DeviceGraph(_weights("ring1", n, rng))
    _, _, cum = MT.hamming_cdf(sym, 2, 8.0, 8.0)
    full = torch.empty(_lib.load().pqi_tfim_sample_workspace_bytes(n), dtype=torch.uint8, device=sym.device)
    small = torch.empty(1024, dtype=torch.uint8, device=sym.device)
    sym.W = torch.from_numpy(W).to(sym.device)
    for base in (5.0, 0.5):
        a = _draw(sym, cum, 512, base, 11, full)
        b = _draw(sym, cum, 512, base, 11, small)
        assert torch.equal(a, b), base


@pytest.mark.parametrize("n", [300, 1100, 2048])
def test_diagonal_with_an_infinite_factor(n):
    """base^(-w) overflows for a diagonal weight of -500: the picked node's weight,
    zero until then, is NaN from there on in every form."""
    rng = np.random.default_rng(n)
    W = _weights("mix3", n, rng)
    i = rng.choice(n, n // 8, replace=False)
    W[i, i] = -500.0
    sym = D.DeviceGraph(_weights("ring1", n, rng))
    _, _, cum = MT.hamming_cdf(sym, 2, 8.0, 8.0)
    full = torch.empty(_lib.load().pqi_tfim_sample_workspace_bytes(n), dtype=torch.uint8, device=sym.device)
    small = torch.empty(1024, dtype=torch.uint8, device=sym.device)
    sym.W = torch.from_numpy(W).to(sym.device)
    for base in (5.0, 0.2):
        a = _draw(sym, cum, 256, base, 11, full)
        b = _draw(sym, cum, 256, base, 11, small)
        assert torch.equal(a, b), base
