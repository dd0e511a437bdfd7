"""FP64 sums in the resident grid form, whose tiles keep their variables by falling list length
(one thread's network up to 32 entries, whole warps past that): lists on both sides of every
limit, against the oracle bit for bit."""
import numpy as np
import pytest

import dmm_b200 as dmm
from conftest import uniform_init
from test_gpu_cluster import check, random_formula

pytestmark = pytest.mark.gpu


def formula_of_lengths(n, lengths, seed):
    """3-literal clauses in which variable v occurs lengths[v mod len(lengths)] times."""
    rng = np.random.default_rng(seed)
    occ = np.repeat(np.arange(n), np.resize(lengths, n))
    occ = occ[: len(occ) // 3 * 3]
    rng.shuffle(occ)
    cl = occ.reshape(-1, 3)
    for _ in range(200):  # a clause with a variable twice swaps it with another clause's
        s = np.sort(cl, axis=1)
        bad = np.flatnonzero((s[:, 0] == s[:, 1]) | (s[:, 1] == s[:, 2]))
        if not len(bad):
            break
        for c in bad:
            i, o, k = rng.integers(3), rng.integers(len(cl)), rng.integers(3)
            cl[c, i], cl[o, k] = cl[o, k], cl[c, i]
    assert not len(bad)
    lits = (cl + 1) * rng.choice([-1, 1], size=cl.shape)
    return dmm.from_arrays(lits.astype(np.int32).ravel(), np.arange(len(cl) + 1) * 3, n)


@pytest.mark.parametrize("n,lengths", [
    (3300, [0, 1, 31, 32, 33, 2, 16, 17, 24, 25, 8]),      # around the network's length
    (3120, [0, 63, 64, 65, 1, 3, 5, 7]),                   # around the warp's ranking
    (4000, [6] * 97 + [254, 255, 256, 257, 700, 0, 0]),    # past the ordering's longest class
    (3001, [40]),                                          # every list summed by a warp
    (4736, [9]),                                           # every list alike
])
def test_lists_of_given_lengths(n, lengths):
    form = formula_of_lengths(n, lengths, n)
    check(form, uniform_init(form.n, form.m, 3), "fp64", 8, pieces=[3, 5])


def test_unit_clauses_follow_their_variables():
    form = random_formula(5003, 30011, 1, 9, seed=4)
    check(form, uniform_init(form.n, form.m, 6), "fp64", 8, pieces=[1, 7])


def formula_of_clause_lengths(n, lengths, m, seed):
    """m clauses over distinct variables, clause c of lengths[c mod len(lengths)] literals."""
    rng = np.random.default_rng(seed)
    lens = np.resize(lengths, m)
    rng.shuffle(lens)
    off = np.concatenate([[0], np.cumsum(lens)])
    lits = np.concatenate([rng.choice(n, k, replace=False) + 1 for k in lens])
    lits = lits * rng.choice([-1, 1], size=len(lits))
    return dmm.from_arrays(lits.astype(np.int32), off, n)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("n,m,lengths", [
    (4001, 12345, [2, 3, 4, 5, 8, 9]),           # both sides of whole groups of four literals
    (3000, 11111, [3] * 200 + [1, 14, 15, 16, 17, 25]),  # around the last class of the ordering
    (5000, 9001, [4]),                           # all alike, none of three
    (60000, 330001, [2, 3, 3, 5]),               # clause memories not resident
])
def test_clauses_of_given_lengths(prec, n, m, lengths):
    """Clause tiles are gone through by falling clause length."""
    form = formula_of_clause_lengths(n, lengths, m, n)
    check(form, uniform_init(form.n, form.m, 4), prec, 8, pieces=[3, 5])
