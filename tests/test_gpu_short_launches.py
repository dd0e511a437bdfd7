"""Launches of a few steps, which leave a formula of the cluster or resident grid form to the tile
forms: the same trajectory in any mixture of short and long launches, and no slower than those."""
import numpy as np
import pytest

import dmm_b200 as dmm
from test_gpu_cluster import random_formula

pytestmark = pytest.mark.gpu

LAUNCHES = [1, 3, 40, 2, 1, 33, 8, 64, 1]


def formula(kind, n):
    if kind == "mixed":
        return random_formula(n, 5 * n, 1, 6, seed=n)
    return dmm.generate_planted(n, int({"r4": 4.3, "r8": 8.0}[kind] * n), 0.08, 0.58, seed=n)[0]


CASES = [(k, n, p) for k, n in (("r8", 300), ("r8", 2000), ("r4", 4000), ("r8", 6007), ("r4", 30000),
                                ("mixed", 900), ("mixed", 5003)) for p in ("fp32", "fp64")]


@pytest.mark.parametrize("kind,n,prec", CASES)
def test_short_and_long_launches_mixed(kind, n, prec):
    f = formula(kind, n)
    x0 = dmm.initial_state_uniform(f, 11)
    with dmm.Instance(f, precision=prec) as a, dmm.Instance(f, precision=prec) as b:
        b.set_tuning(launch_mode=2)
        assert a.step_kernel in ("cluster", "resident-grid")
        for inst in (a, b):
            inst.set_state(x0)
        for k in LAUNCHES:
            ra, rb = a.step(k), b.step(k)
            assert (ra.status, ra.steps, ra.loc, ra.best_loc, ra.t) == \
                   (rb.status, rb.steps, rb.loc, rb.best_loc, rb.t)
            # at most m terms of at most 1, in any order
            assert abs(ra.energy - rb.energy) <= f.m * 2.0 ** -53 * abs(rb.energy)
            (xa, ta), (xb, tb) = a.get_state(), b.get_state()
            assert ta == tb and np.array_equal(xa, xb)


@pytest.mark.parametrize("n,prec", [(2000, "fp32"), (9000, "fp32"), (9000, "fp64")])
def test_solution_found_in_a_short_launch(n, prec):
    f = dmm.generate_planted(n, 8 * n, 0.08, 0.46, seed=n)[0]
    x0 = dmm.initial_state_uniform(f, 3)
    out = []
    for mode in (0, 2):
        with dmm.Instance(f, precision=prec) as inst:
            inst.set_tuning(launch_mode=mode)
            inst.set_state(x0)
            r = inst.step(1)
            while not r.solved and r.steps < 2000:
                r = inst.step(1)
            assert r.solved
            out.append((r.steps, r.solved_step, r.t, inst.assignment(), inst.get_state()[0]))
    assert out[0][:3] == out[1][:3]
    assert all(np.array_equal(p, q) for p, q in zip(out[0][3], out[1][3]))
    assert np.array_equal(out[0][4], out[1][4])


@pytest.mark.parametrize("kind,n,prec", [("r8", 50000, "fp32"), ("r4", 90000, "fp32"), ("r4", 50000, "fp64")])
def test_single_steps_not_slower_than_the_tile_forms(kind, n, prec):
    """Device time of launches of one step: it was 1.9 to 2.3 times that of the tile forms."""
    f = formula(kind, n)
    x0 = dmm.initial_state_uniform(f, 11)
    with dmm.Instance(f, precision=prec) as a, dmm.Instance(f, precision=prec) as b:
        b.set_tuning(launch_mode=2)
        ms = []
        for inst in (a, b):
            inst.set_state(x0)
            inst.step(1)
            ms.append(min(inst.time_steps(1) for _ in range(30)))
    assert ms[0] <= 1.25 * ms[1], ms
