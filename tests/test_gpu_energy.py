"""The FP64 energy of the forms that split a formula over blocks is the exact sum of the clauses' C_m,
rounded once: the same alone, in a batch and for any split."""
import math

import numpy as np
import pytest

import dmm_b200 as dmm
from oracle.oracle import Oracle
from test_gpu_cluster import random_formula

pytestmark = pytest.mark.gpu

STEPS = 40


def formula(kind, n):
    if kind == "mixed":
        return random_formula(n, 5 * n, 1, 6, seed=n)
    return dmm.generate_planted(n, 8 * n, 0.08, 0.58, seed=n)[0]


def exact_energy(f, v):
    """Sum of C_m at voltages v: every C_m is exact in the kernels' order of operations, fsum rounds
    their sum once.  The kernels carry the rounding errors of at most m additions along, which
    leaves a relative error of (m 2^-53)^2 < 1e-20 before their one rounding: the same double
    unless the sum lies that close to the middle between two."""
    lits = f.lits.astype(np.int64)
    a = 1.0 - np.sign(lits) * v[np.abs(lits) - 1]
    off = f.clause_off
    c = 0.5 * np.minimum.reduceat(a, off[:-1])
    c[np.diff(off) == 1] = 0.0
    return math.fsum(c)


@pytest.mark.parametrize("kind,n,kernel", [
    ("r8", 100, "cluster"), ("r8", 1000, "cluster"), ("mixed", 700, "cluster"),
    ("r8", 5000, "resident-grid"), ("r8", 6001, "resident-grid"), ("r8", 9000, "resident-grid"),
    ("mixed", 4001, "resident-grid"),
])
def test_energy_rounded_once(kind, n, kernel):
    f = formula(kind, n)
    x0 = dmm.initial_state_uniform(f, 5)
    ref = Oracle(f.n, f.m, f.lits, f.clause_off, precision="fp64").run(x0, STEPS, dump_every=1)
    want = exact_energy(f, ref["dump"][ref["steps"] - 1][:f.n])  # (the smallest is solved earlier)
    with dmm.Instance(f, precision="fp64") as inst:
        assert inst.step_kernel == kernel
        inst.set_state(x0)
        assert inst.step(STEPS).energy == want
    for copies in (2, 9):
        b = dmm.Batch.for_formulas([f] * copies, precision="fp64")
        for _ in range(copies):
            b.add(f, x0, max_steps=STEPS)
        b.run()
        assert [b.result(k)[0].energy for k in range(copies)] == [want] * copies
        b.close()
