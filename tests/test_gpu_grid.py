"""The resident grid form (formulas on groups of blocks, exchanges through self-flagging
entries) where its tables, tilings and exchanges can go wrong: against the oracle bit for bit,
and against the tile forms in batches."""
import numpy as np
import pytest

import dmm_b200 as dmm
from conftest import uniform_init
from test_gpu_cluster import check, random_formula

pytestmark = pytest.mark.gpu


def skewed_formula(n, m, seed, power=2.5):
    """3-literal clauses whose variables follow a power law: occurrence lists from none to
    thousands of entries, so that tiles of equal size hold very different numbers of slots."""
    rng = np.random.default_rng(seed)
    v = (n * rng.random((2 * m, 3)) ** power).astype(np.int64)
    v = v[(v[:, 0] != v[:, 1]) & (v[:, 0] != v[:, 2]) & (v[:, 1] != v[:, 2])][:m]
    lits = (v + 1) * rng.choice([-1, 1], size=v.shape)
    return dmm.from_arrays(lits.astype(np.int32).ravel(), np.arange(len(v) + 1) * 3, n)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("n,m", [(4001, 32003), (5000, 21500), (12345, 98765), (30011, 129047)])
def test_three_literal_formulas(prec, n, m):
    form, _ = dmm.generate_planted(n, m, p0=0.08, p1=0.58, seed=n + m)
    check(form, uniform_init(n, m, n), prec, 12, pieces=[1, 2, 9])


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("n,m,kmin,kmax", [(3001, 16007, 1, 8), (2000, 9001, 2, 25)])
def test_general_clauses(prec, n, m, kmin, kmax):
    """Unit clauses among them; the initial state does not pin their variables, so that the
    first step moves them to their signs everywhere."""
    form = random_formula(n, m, kmin, kmax, seed=n)
    check(form, uniform_init(n, m, 3), prec, 12, pieces=[5, 7])


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_alpha_per_clause(prec):
    form, _ = dmm.generate_planted(4500, 36001, p0=0.08, p1=0.58, seed=6)
    alpha = np.random.default_rng(1).uniform(0.5, 4.0, form.m)
    check(form, uniform_init(4500, 36001, 2), prec, 10, alpha=alpha)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("power", [1.5, 4.0])
def test_skewed_occurrences(prec, power):
    """Long lists (past the networks and the warp's ranking) and uneven tiles, up to tilings
    that fit only with several tiles per block or not at all."""
    form = skewed_formula(6000, 30000, 3, power)
    check(form, uniform_init(form.n, form.m, 8), prec, 6)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("sizes", [(20000, 9000), (9000,) * 8, (30000, 300, 5000, 200, 100),
                                   (3000,) * 60])
def test_groups_of_blocks_equal_the_tile_form(prec, sizes):
    """Several formulas side by side, finishing at different steps, with one to many tiles
    per block."""
    forms = [dmm.generate_planted(n, 8 * n + k, 0.08, 0.46 if k % 2 else 0.58, seed=40 + k)[0]
             for k, n in enumerate(sizes)]
    x0s = [dmm.initial_state_uniform(f, 60 + k) for k, f in enumerate(forms)]
    caps = [35 + 7 * (k % 5) for k in range(len(forms))]
    got = []
    for mode in (0, 2):
        b = dmm.Batch.for_formulas(forms, precision=prec)
        try:
            b.set_tuning(launch_mode=mode)
            for f, x0, cap in zip(forms, x0s, caps):
                b.add(f, x0, max_steps=cap)
            b.run()
            b.set_state_at(0, x0s[0], 0.5, 3)  # a second run of one of them
            b.run()
            got.append([(b.result(k), b.state(k)) for k in range(len(forms))])
        finally:
            b.close()
    for (ra, sa), (rb, sb) in zip(*got):
        a, c = ra[0], rb[0]
        assert (a.status, a.steps, a.t, a.loc, a.best_loc, a.solved_step, a.solved_t) == (
            c.status, c.steps, c.t, c.loc, c.best_loc, c.solved_step, c.solved_t)
        assert np.array_equal(ra[1], rb[1])
        assert np.array_equal(sa[0], sb[0]) and sa[1] == sb[1]
        assert abs(a.energy - c.energy) <= 1e-12 * abs(c.energy)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_not_a_number_in_the_state(prec):
    """A NaN voltage spreads as in the tile forms; entries of the exchanges that hold NaN are
    still entries."""
    form, _ = dmm.generate_planted(5000, 21500, p0=0.08, p1=0.58, seed=2)
    x0 = dmm.initial_state_uniform(form, 3)
    x0[[17, 4000]] = np.nan
    out = []
    for mode in (0, 2):
        with dmm.Instance(form, precision=prec) as inst:
            inst.set_tuning(launch_mode=mode)
            inst.set_state(x0)
            r = inst.step(4)
            out.append((inst.get_state()[0], r.steps, r.t, r.loc))
    assert np.array_equal(out[0][0], out[1][0], equal_nan=True)
    assert out[0][1:] == out[1][1:]
    assert np.isnan(out[0][0]).sum() > 2
