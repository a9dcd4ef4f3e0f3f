"""The shared pass of starting fields gives the search kernels' own column-order
sums: the same searches bit for bit with and without it (dense graphs of 2048
nodes or more, whose kernels sum in column order), at the task counts where the
tiles change, for one graph and for tiles that mix graphs."""

import numpy as np
import pytest
import torch

from pyqrackising_b200 import _lib
from pyqrackising_b200 import device as D
from pyqrackising_b200.batch import BatchedSearch

pytestmark = pytest.mark.gpu


def _graph(kind, n, seed):
    rng = np.random.default_rng(seed)
    U = rng.standard_normal((n, n), dtype=np.float32) if kind == "float" else rng.integers(-3, 4, (n, n)).astype(np.float32)
    U = np.triu(U, 1)
    return D.DeviceGraph(U + U.T)


@pytest.mark.parametrize("kind", ["float", "int"])
@pytest.mark.parametrize("sizes,tasks", [((2048,), 1), ((2051,), 16), ((2080,), 17), ((2048,), 33), ((2111, 2048, 2300), 65)])
def test_start_pass_gives_the_same_search(kind, sizes, tasks):
    bs = BatchedSearch([_graph(kind, n, n) for n in sizes])
    tg = np.arange(tasks, dtype=np.int32) % len(sizes)
    words = bs.random_states(tg, 3)
    got = bs.run(tg, words, True, flip_budget=30)
    _lib.call("pqi_batch_set_start_pass", 0)
    try:
        want = bs.run(tg, words, True, flip_budget=30)
    finally:
        _lib.call("pqi_batch_set_start_pass", 1)
    assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
    # (the starting value sums x_v y_v in another order: n roundings of it at most)
    scale = want[0].abs() + 1.0
    assert torch.all((got[0] - want[0]).abs() <= max(sizes) * 2.0 ** -52 * scale * (0.0 if kind == "int" else 100.0))
