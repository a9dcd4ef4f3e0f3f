"""The default scoring form - the candidates expanded in 16-byte pieces, the
triangular half of the node tiles - gives the full form's scores bit for bit (path
5: every tile, candidates expanded in the kernel; both sum whole numbers exactly),
at the sizes where tiles, words and candidate blocks end."""

import numpy as np
import pytest
import torch

from pyqrackising_b200 import _lib
from pyqrackising_b200 import device as D

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("kind", ["float", "int"])
@pytest.mark.parametrize("n", [31, 256, 257, 385, 512, 513, 1023])
@pytest.mark.parametrize("shots", [1, 128, 129, 300])
def test_triangular_form_gives_the_full_scores(kind, n, shots):
    rng = np.random.default_rng(n + shots)
    U = rng.standard_normal((n, n), dtype=np.float32) if kind == "float" else rng.integers(-9, 10, (n, n)).astype(np.float32)
    U = np.triu(U, 1)
    dg = D.DeviceGraph(U + U.T)
    words = dg.pack(rng.integers(0, 2, (shots, n), dtype=np.uint8))
    geo = D.geometry(shots, shots, 148)
    out = {}
    for path in (0, 5):
        _lib.call("pqi_score_set_path", path)
        try:
            out[path] = [torch.as_tensor(x).clone() for x in dg.calculate_cut(words, shots, True, *geo)]
        finally:
            _lib.call("pqi_score_set_path", 0)
    assert all(torch.equal(a, b) for a, b in zip(out[0], out[5]))
    assert torch.isfinite(out[0][0].float()).all()
