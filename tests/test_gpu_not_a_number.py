"""NaN voltages in formulas of mixed clause lengths: the reference's minimum over a clause's literals
passes them over, and so does every form, the three-literal clauses among them included."""
import numpy as np
import pytest

import dmm_b200 as dmm
from oracle.oracle import Oracle
from test_gpu_cluster import random_formula

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("n,kernel", [(300, "cluster"), (5003, "resident-grid"), (30011, "resident-grid")])
def test_nan_voltages(n, kernel, prec):
    f = random_formula(n, 4 * n, 1, 6, seed=n)
    x0 = dmm.initial_state_uniform(f, 3)
    x0[[7, n // 2, n - 1]] = np.nan
    steps = 8
    ref = Oracle(f.n, f.m, f.lits, f.clause_off, precision=prec).run(x0, steps, dump_every=1)
    for mode in (0, 2):
        with dmm.Instance(f, precision=prec) as inst:
            inst.set_tuning(launch_mode=mode)
            assert mode == 2 or inst.step_kernel == kernel
            inst.set_state(x0)
            r = inst.step(steps)
            assert r.steps == ref["steps"] == steps
            assert np.array_equal(inst.get_state()[0], ref["dump"][steps], equal_nan=True)
