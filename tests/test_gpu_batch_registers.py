"""The register form of the CTA search follows the shared-memory form (used when
the start pass is off) flip for flip, at the graph sizes where a thread's groups
and the idle warps change, with more tasks than resident CTAs (a queue, largest
graphs first) and with fewer."""

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
@pytest.mark.parametrize("variant", ["cta", "cta128", "cta64"])
@pytest.mark.parametrize("sizes,tasks", [((64, 65, 127, 128, 129), 3000), ((255, 256, 257, 2, 3), 40),
                                         ((511, 512, 513, 1023, 1024), 25), ((1025, 33, 2047, 2048), 12),
                                         ((2049, 4095, 4096), 6)])
def test_register_form_follows_the_shared_form(kind, variant, sizes, tasks):
    bs = BatchedSearch([_graph(kind, n, n) for n in sizes])
    tg = np.arange(tasks, dtype=np.int32) % len(sizes)
    words = bs.random_states(tg, 3)
    run = lambda: bs.run(tg, words, False, rounds=2, kick=3, seed=5, variant=variant, fields="f64")
    got = run()
    _lib.call("pqi_batch_set_start_pass", 0)
    try:
        want = run()
    finally:
        _lib.call("pqi_batch_set_start_pass", 1)
    assert torch.equal(got[1], want[1]) and torch.equal(got[2], want[2])
    # (values: the starting fields' sums, n^2 terms, in another order)
    tol = 0.0 if kind == "int" else max(sizes) ** 2 * 2.0 ** -52 * (want[0].abs() + 1.0)
    assert torch.all((got[0] - want[0]).abs() <= tol)
