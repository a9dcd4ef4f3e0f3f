"""The cluster ascent follows the CTA search flip for flip on both of its register
budgets (few tasks; more tasks than the larger budget keeps resident), with one
and two groups of nodes per thread and ragged last slices."""

import numpy as np
import pytest
import torch

from pyqrackising_b200 import device as D
from pyqrackising_b200.batch import BatchedSearch

pytestmark = pytest.mark.gpu


def _graph(kind, n, seed):
    rng = np.random.default_rng(seed)
    U = rng.standard_normal((n, n), dtype=np.float32) if kind == "float" else rng.integers(-3, 4, (n, n)).astype(np.float32)
    U = np.triu(U, 1)
    return D.DeviceGraph(U + U.T)


@pytest.mark.parametrize("kind", ["float", "int"])
@pytest.mark.parametrize("n,tasks,csize", [(33, 3, 2), (1000, 3, 16), (2050, 4, 2), (2305, 2, 2), (2050, 160, 16),
                                           (1029, 400, 8), (2100, 250, 2)])
def test_cluster_ascent_follows_the_cta_search(kind, n, tasks, csize):
    bs = BatchedSearch([_graph(kind, n, n)])
    tg = np.zeros(tasks, np.int32)
    words = bs.random_states(tg, 5)
    got = bs.cluster_ascent(tg, words, True, cluster_size=csize)
    want = bs.run(tg, words, True, rounds=0, fields="f64")
    assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
    # (values: x^T W x, n^2 terms, summed in another order)
    tol = 0.0 if kind == "int" else n ** 2 * 2.0 ** -52 * (want[0].abs() + 1.0)
    assert torch.all((got[0] - want[0]).abs() <= tol)
