"""The cluster form (one small formula per thread-block cluster) at the sizes where its split
over blocks, its tables and its sums can go wrong, against the oracle: states bit for bit, the
FP64 energy (whose last bits depend on the split) within 1e-12 relative."""
import numpy as np
import pytest

import dmm_b200 as dmm
from conftest import uniform_init
from oracle.oracle import Oracle

pytestmark = pytest.mark.gpu


def random_formula(n, m, kmin, kmax, seed):
    """Clauses of kmin..kmax distinct variables (fewer when n is smaller), random signs."""
    rng = np.random.default_rng(seed)
    lits, off = [], [0]
    for _ in range(m):
        k = min(int(rng.integers(kmin, kmax + 1)), n)
        v = rng.choice(n, size=k, replace=False) + 1
        lits += list(v * rng.choice([-1, 1], size=k))
        off.append(len(lits))
    return dmm.from_arrays(np.array(lits, dtype=np.int32), np.array(off, dtype=np.int64), n)


def check(form, x0, prec, steps, pieces=None, alpha=None):
    o = Oracle(form.n, form.m, form.lits, form.clause_off, precision=prec, alpha_cm=alpha)
    ref = o.run(x0, steps, dump_every=1)
    with dmm.Instance(form, precision=prec) as inst:
        if alpha is not None:
            inst.set_params(alpha_cm=alpha)
        inst.set_state(x0)
        for k in pieces or [steps]:
            r = inst.step(k)
        x, _ = inst.get_state()
        with dmm.Instance(form, precision=prec) as grid:  # the grid-wide form of the same step
            grid.set_tuning(launch_mode=2)
            if alpha is not None:
                grid.set_params(alpha_cm=alpha)
            grid.set_state(x0)
            g = grid.step(steps)
    assert r.steps == ref["steps"]
    assert np.array_equal(x, ref["dump"][ref["steps"]])
    assert (r.t, r.loc, r.best_loc, r.solved_step, r.status) == (g.t, g.loc, g.best_loc,
                                                                 g.solved_step, g.status)
    assert abs(r.energy - g.energy) <= 1e-12 * abs(g.energy)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("n,m", [
    (3, 5),        # fewer variables and clauses than blocks
    (17, 160),     # one variable tile of 4 per block, most blocks without clauses' owners
    (64, 270), (65, 513), (127, 1016),
    (300, 2400), (1021, 4391),
    (20, 2500),    # lists of about 375 entries (past the warp's ranking and networks)
    (120, 2700),   # lists of about 68: around the ranking's 64 entries
    (2003, 16001), (3200, 13760),  # near the capacity of a cluster
])
def test_three_literal_formulas(prec, n, m):
    form, _ = dmm.generate_planted(n, m, p0=0.08, p1=0.58, seed=n + m)
    check(form, uniform_init(n, m, n), prec, 40)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("n,m,kmin,kmax", [(5, 9, 1, 3), (150, 700, 1, 8), (33, 64, 2, 2),
                                           (700, 2500, 1, 25), (1500, 6000, 2, 5)])
def test_general_clauses(prec, n, m, kmin, kmax):
    form = random_formula(n, m, kmin, kmax, seed=n)
    x0 = dmm.initial_state_uniform(form, 3)
    check(form, x0, prec, 40)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_alpha_per_clause(prec):
    form, _ = dmm.generate_planted(250, 1999, p0=0.08, p1=0.58, seed=6)
    alpha = np.random.default_rng(1).uniform(0.5, 4.0, form.m)
    check(form, uniform_init(250, 1999, 2), prec, 40, alpha=alpha)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_launches_of_a_few_steps_equal_one(prec):
    form, _ = dmm.generate_planted(400, 3200, p0=0.08, p1=0.58, seed=9)
    check(form, uniform_init(400, 3200, 4), prec, 60, pieces=[1, 2, 7, 50])


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("count", [2, 7, 40, 120])
def test_batches_over_cluster_sizes(prec, count):
    """Formulas of both clause kinds and many sizes in one pack (cluster sizes 1 to 16, several
    launches side by side, some too large for a cluster) equal the grid-wide form."""
    rng = np.random.default_rng(count)
    forms, x0s = [], []
    for k in range(count):
        n = int(np.exp(rng.uniform(np.log(20), np.log(6000 if k % 10 == 0 else 1500))))
        m = int(n * rng.uniform(3, 8)) + 1
        f = random_formula(n, min(m, 400), 1, 6, seed=k) if k % 4 == 3 else \
            dmm.generate_planted(n, m, p0=0.08, p1=0.46, seed=k)[0]
        forms.append(f)
        x0s.append(dmm.initial_state_uniform(f, 50 + k))
    got = []
    for mode in (0, 2):
        b = dmm.Batch.for_formulas(forms, precision=prec)
        try:
            b.set_tuning(launch_mode=mode)
            for f, x0 in zip(forms, x0s):
                b.add(f, x0, max_steps=60)
            b.run()
            got.append([(b.result(k), b.state(k)) for k in range(count)])
        finally:
            b.close()
    for (ra, sa), (rb, sb) in zip(*got):
        a, c = ra[0], rb[0]
        assert (a.status, a.steps, a.t, a.loc, a.best_loc, a.solved_step, a.solved_t) == (
            c.status, c.steps, c.t, c.loc, c.best_loc, c.solved_step, c.solved_t)
        assert np.array_equal(ra[1], rb[1])
        assert np.array_equal(sa[0], sb[0]) and sa[1] == sb[1]
        assert abs(a.energy - c.energy) <= 1e-12 * abs(c.energy)
