"""The local search ends where the Gray search brings nothing: a walk that comes back to
the state it began from (or flips a component of its own) changes no value, but its
float gains can sum to a rounding above 0. A graph whose kernels are stood in for on the
host. (On the device 200 of 35,700 searches of complete Gaussian graphs of 8192 nodes met
such a sum, at most 9e-16; the smallest change of value among 246 others was 1e-4.)"""

import importlib

import numpy as np
import pytest
import torch

S = importlib.import_module("pyqrackising_b200.spin_glass_solver")


class _Graph:
    """Two components {0, 1}, {2, .., n-1}; the Gray search answers with `states` in
    turn (the last one for good), each with energy 2^-52."""

    def __init__(self, n, states, is_integer=False):
        self.n, self.n32, self.n64, self.device = n, (n + 31) >> 5, (n + 63) >> 6, torch.device("cpu")
        self.is_integer, self.states, self.grays = is_integer, list(states), 0
        rng = np.random.default_rng(n)
        W = np.triu(rng.standard_normal((n, n)), 1)
        W[:2, 2:] = 0.0
        self.W = W + W.T

    def pack(self, bits):
        w = np.zeros(self.n32 + 1, dtype=np.uint32)  # (a spare word)
        for v in np.nonzero(bits)[0]:
            w[v >> 5] |= np.uint32(1 << (v & 31))
        return torch.from_numpy(w.view(np.int32))

    def bits(self, words):
        w = words.numpy().view(np.uint32)
        return np.array([(w[v >> 5] >> (v & 31)) & 1 for v in range(self.n)], dtype=bool)

    def gains(self, words):
        return None, torch.zeros(self.n, dtype=torch.float64)

    def single_descent(self, words, g64, spin, G, L, budget, trace=None):
        return torch.zeros(1, dtype=torch.float64), torch.zeros(1, dtype=torch.int32), 0

    def double_bit_flips(self, words, g64, spin, G, L, improving=False):
        return torch.tensor([-1.0]), torch.tensor([0])

    def gray(self, words, g64, spin, iters, seeds):
        change = self.states[min(self.grays, len(self.states) - 1)]
        self.grays += 1
        row = self.pack(self.bits(words) ^ change)
        out = torch.zeros(2 * self.n64, dtype=torch.int32)
        out[: row.numel() - 1] = row[:-1]
        return out, torch.tensor([2.0**-52])

    def select(self, values, count, local):
        return values.max().reshape(1), values.argmax().reshape(1)

    def rescore(self, words, rows=1):
        x = 2.0 * self.bits(words) - 1.0
        cut = ((self.W * (x[:, None] != x[None, :])).sum() / 2.0).reshape(1)
        return torch.from_numpy(cut), torch.from_numpy(2.0 * cut - self.W.sum() / 2.0)


def _search(g, theta):
    stats = S.SearchStats()
    words, _ = S.local_search(g, theta, True, 100, 1, 148, 0.0, stats=stats, max_rounds=40)
    return g.bits(words), stats


@pytest.mark.parametrize("n", [33, 64, 70])
def test_a_walk_that_changes_nothing_is_no_improvement(n):
    theta = np.random.default_rng(1).random(n) < 0.5
    got, stats = _search(_Graph(n, [np.zeros(n, dtype=bool)]), theta)
    assert stats.rounds == 1 and stats.gray == 0 and np.array_equal(got, theta)


@pytest.mark.parametrize("n", [33, 64])
def test_a_flipped_component_is_no_improvement(n):
    theta = np.random.default_rng(2).random(n) < 0.5
    got, stats = _search(_Graph(n, [np.arange(n) < 2]), theta)
    assert stats.rounds == 1 and np.array_equal(got, theta)
    got, stats = _search(_Graph(n, [np.ones(n, dtype=bool)]), theta)
    assert stats.rounds == 1 and np.array_equal(got, theta)


@pytest.mark.parametrize("is_integer", [False, True])
def test_improvements_are_taken(is_integer):
    n = 40
    g = _Graph(n, [np.zeros(n, dtype=bool)], is_integer)
    theta = np.zeros(n, dtype=bool)
    gain = (g.W * np.where(theta[:, None] == theta[None, :], 1.0, -1.0)).sum(1)  # of each flip
    g.states = [np.arange(n) == int(gain.argmax()), np.zeros(n, dtype=bool)]
    got, stats = _search(g, theta)
    assert np.array_equal(got, theta ^ g.states[0])
    # (integer weights: the sum is exact, what the search says is taken)
    assert stats.rounds == (40 + 1 if is_integer else 2) and stats.gray == (40 if is_integer else 1)
