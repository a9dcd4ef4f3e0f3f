"""The Hamming-weight distribution's closed-form normalisers and ratio-stepped
bins against a plain float64 restatement that sums every bin: sizes around the
kernel's runs of 8 bins and blocks of 1024, both parities, time scales whose
envelopes are deltas, ordinary or growing towards an end."""

import importlib

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

MT = importlib.import_module("pyqrackising_b200.maxcut_tfim")
EPS = 1.1920928955078125e-07


def _cdf(J, z, n, quality, tot, h, start):
    steps = 1 << quality
    k = np.arange(n + 1.0)
    half = n / 2.0
    acc = start.copy()
    live = np.abs(J) >= EPS
    J, z = J[live], z[live]
    with np.errstate(all="ignore"):
        theta = np.arcsin(np.clip(h / (z * J), -1, 1))
        for step in range(1, steps):
            t, dt = step * (tot / steps), tot / steps
            ht = h * (tot - t)
            theta_c = np.arcsin(np.clip(ht / (z * J), -1, 1))
            for sign, tt in ((1.0, t), (-1.0, t - dt)):
                p = np.exp2(np.abs(J / ht) - 1.0) * (1.0 + np.sin(theta - theta_c) * np.cos(1.5 * np.pi * J * tt + theta) / (1.0 + np.sqrt(tt))) - 0.5
                env = np.exp2(-(p / (n + 1))[:, None] * (k + 1.0)) * np.exp(-np.abs(k - half) / max(tt, 1e-9))
                tot_env = env.sum(1, keepdims=True)
                delta = (k == n // 2).astype(float)
                acc += sign * np.where(tot_env > 0, env / tot_env, delta).sum(0)
    mid = acc[1:n]
    cum = np.cumsum(mid / mid.sum())
    cum[-1] = 1.0
    return cum


@pytest.mark.parametrize("n", [3, 4, 15, 16, 17, 127, 1023, 1024, 2045, 2049, 2050])
@pytest.mark.parametrize("quality,tot,scale", [(0, 8.0, 1.0), (1, 8.0, 1.0), (4, 8.0, 1.0), (3, 0.05, 1.0), (2, 40.0, 30.0), (2, 1e-4, 1.0)])
def test_cdf_matches_plain_sums(n, quality, tot, scale):
    rng = np.random.default_rng(n)
    W = np.triu(rng.random((n, n)) * (rng.random((n, n)) < 0.5) * scale, 1).astype(np.float32)
    from pyqrackising_b200.device import DeviceGraph

    dg = DeviceGraph(W + W.T)
    J, degrees, cum = MT.hamming_cdf(dg, quality, tot, 8.0)
    want = _cdf(J.cpu().numpy(), degrees.cpu().numpy().astype(np.float64), n, quality, tot, 8.0, MT.init_thresholds(n))
    # The bins' sum (the normaliser, about 1) is what is left of 2 (steps - 1) n unit
    # envelopes of either sign, each summing to 1 within a few roundings (4 for the
    # exponent and normaliser, 8 for the ratio steps) on either side: the error of both
    # is bounded by that many roundings of the envelopes' total, 2 (steps - 1) n.
    tol = 2 * 16 * 2.0 ** -53 * max(1.0, 2.0 * ((1 << quality) - 1) * n)
    got = cum.cpu().numpy()
    assert np.abs(got - want).max() <= tol * max(1.0, np.abs(want).max())


def test_thresholds_are_the_binomials():
    """Each weight is the coefficient over the sum of those kept, rounded once."""
    import math
    from fractions import Fraction

    for n in (3, 4, 24, 25, 300, 1101):
        kept = [math.comb(n, q) for q in range(n + 1)]
        kept[(n + 1) // 2] = 0  # never written by the reference (the upper middle one for odd n)
        want = [float(Fraction(c, sum(kept))) for c in kept]
        assert MT.init_thresholds(n).tolist() == want
