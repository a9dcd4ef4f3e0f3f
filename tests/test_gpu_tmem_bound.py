"""The tensor-memory form skips gains below its references' bound; the selection
must not change where many gains tie as floats, weights vanish or are denormal,
kicks flip nodes that are no selection, and graphs of different size share a
launch: the same searches as with fields in shared memory, bit for bit."""

import numpy as np
import pytest
import torch

from pyqrackising_b200 import _lib
from pyqrackising_b200 import device as D
from pyqrackising_b200.batch import BatchedSearch

pytestmark = pytest.mark.gpu


def _matrix(kind, n, seed):
    rng = np.random.default_rng(seed)
    if kind == "ties":  # few distinct values, none an integer
        U = rng.choice(np.array([-0.5, 0.0, 0.5], dtype=np.float32), (n, n))
    elif kind == "tiny":  # denormal weights among normal ones
        U = np.where(rng.random((n, n)) < 0.5, 1e-41, rng.standard_normal((n, n)) * 1e-38).astype(np.float32)
    elif kind == "wide":  # a few weights far above the rest
        U = rng.standard_normal((n, n)).astype(np.float32) * np.where(rng.random((n, n)) < 1e-4, 1e4, 1e-3).astype(np.float32)
    else:
        U = np.where(rng.random((n, n)) < 0.002, rng.standard_normal((n, n)), 0.0).astype(np.float32)
    U = np.triu(U, 1)
    return (U + U.T).astype(np.float32)


@pytest.mark.parametrize("kind", ["ties", "tiny", "wide", "sparse"])
@pytest.mark.parametrize("sizes", [(4097,), (6143, 4500, 5999), (8200, 2047)])
def test_bound_keeps_the_selection(kind, sizes):
    bs = BatchedSearch([D.DeviceGraph(_matrix(kind, n, n)) for n in sizes], row_lists=False)
    tg = np.arange(6, dtype=np.int32) % len(sizes)
    words = bs.random_states(tg, 5)
    args = dict(rounds=2, kick=9, seed=11, flip_budget=400)
    got = bs.run(tg, words, True, **args)
    _lib.call("pqi_batch_set_tmem_fields", 0)
    try:
        want = bs.run(tg, words, True, **args)
    finally:
        _lib.call("pqi_batch_set_tmem_fields", 1)
    assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
    # (the starting value sums x_v y_v in another order; the gains added are equal)
    assert torch.all((got[0] - want[0]).abs() <= 1e-10 * (want[0].abs() + max(sizes) * 1e-38))


def test_tasks_that_follow_one_another_in_the_same_columns():
    """Several tasks per CTA, of two sizes: each starts from its own fields, whatever
    the one before still had on the way."""
    sizes = (4097, 6000)
    bs = BatchedSearch([D.DeviceGraph(_matrix("wide", n, n)) for n in sizes], row_lists=False)
    tg = (np.arange(1500, dtype=np.int32) // 2) % 2
    words = bs.random_states(tg, 6)
    args = dict(rounds=1, kick=3, seed=12, flip_budget=25)
    got = bs.run(tg, words, True, **args)
    _lib.call("pqi_batch_set_tmem_fields", 0)
    try:
        want = bs.run(tg, words, True, **args)
    finally:
        _lib.call("pqi_batch_set_tmem_fields", 1)
    assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
    assert torch.all((got[0] - want[0]).abs() <= 1e-10 * (want[0].abs() + 1.0))
