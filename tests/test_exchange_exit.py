"""How the warps of a cluster leave a loop of exchanges when a bounded wait runs out
in some of them only: the barriers of the flip loops of the cluster ascent
(pqi_cluster.cu) and the descent (pqi_gray.cu), restated as coroutines and run in
random orders. Every warp must reach every barrier, whichever waits fail, and the
whole cluster must come to one verdict. (The passes of the tensor-memory search,
pqi_batch.cu, alternate their flags for the reason of the last case.)"""

import random

import pytest


def _warp(cta, warp, flips, S, flags, report, uniform, rng, inside=None, flip=1):
    """One warp's barriers. uniform: the verdict is taken behind a CTA barrier;
    else a warp whose wait runs out leaves by itself. inside: a flip before which
    the cluster meets (a barrier inside the loop). flip: flags alternate between
    exchanges (0: one flag for all)."""
    f, failed = 0, 0
    while True:
        if f == inside:
            yield "cluster", "inside"
        yield "cta", 0
        yield "pause", 0  # (a slow warp reads the flag late)
        failed = flags[cta][(f & flip) ^ flip]
        if warp == 0:
            S[f].add(cta)
        if uniform and failed:
            break
        ok = yield "wait", f
        end = f == flips - 1  # every warp whose wait succeeded reads that no flip is left
        if not ok:
            flags[cta][f & flip] = 1
            end = rng.random() < 0.5  # (what the slots held)
        if not uniform:
            if end or not ok:
                failed = not ok
                break
        elif end:
            yield "cta", 0
            yield "pause", 0
            failed = flags[cta][f & flip]
            break
        f += 1
    if failed:
        report.add(cta)
    yield "cluster", "behind"
    return bool(report)


def _run(seed, uniform, ctas=3, warps=3, flips=3, chance=0.2, inside=None, flip=1):
    rng = random.Random(seed)
    S, report, flags = [set() for _ in range(flips + 2)], set(), [[0, 0] for _ in range(ctas)]
    gens = {(c, w): _warp(c, w, flips, S, flags, report, uniform, rng, inside, flip) for c in range(ctas) for w in range(warps)}
    at = {k: next(g) for k, g in gens.items()}  # what each warp stands at
    done = {}

    def go(k, value):
        try:
            at[k] = gens[k].send(value)
        except StopIteration as e:
            at[k] = None
            done[k] = e.value

    while len(done) < len(gens):
        ready = []
        for k, e in at.items():
            if e and e[0] in ("wait", "pause"):
                ready.append((k,))
        for c in range(ctas):
            mine = [(c, w) for w in range(warps)]
            if all(at[k] and at[k][0] == "cta" for k in mine):
                ready.append(tuple(mine))
        if all(e and e[0] == "cluster" for e in at.values()):
            ready.append(tuple(at))
        if not ready:
            return None  # some warps wait for others that never come
        group = rng.choice(ready)
        kind, f = at[group[0]]
        if any(at[k][1] != f for k in group if kind == "cluster"):
            return None  # two different barriers taken for one
        if kind == "wait":
            full = len(S[f]) == ctas
            if full or rng.random() < chance:  # (else it goes on waiting)
                go(group[0], full and rng.random() >= chance)
        else:
            for k in group:
                go(k, None)
    return set(done.values()), bool(report)


@pytest.mark.parametrize("chance", [0.02, 0.2, 0.7])
def test_every_warp_leaves_with_one_verdict(chance):
    seen = set()
    for seed in range(600):
        got = _run(seed, True, chance=chance)
        assert got is not None, seed
        assert got[0] == {got[1]}
        seen.add(got[1])
    assert True in seen


def test_warps_that_leave_by_themselves_would_hang():
    assert any(_run(seed, False) is None for seed in range(200))


def test_a_cluster_barrier_inside_the_loop_would_not_match():
    assert any(_run(seed, True, inside=2) is None for seed in range(200))


def test_one_flag_for_all_exchanges_would_be_read_too_late():
    assert any(_run(seed, True, flip=0) is None for seed in range(600))
