"""Formulas admitted many at a time (laid aside by the host, unpacked by one launch): the same
results as one at a time, over list lengths, clause kinds and block limits."""
import numpy as np
import pytest

import dmm_b200 as dmm
from test_gpu_cluster import random_formula

pytestmark = pytest.mark.gpu


def formulas():
    fs = [dmm.generate_planted(n, m, 0.08, 0.46, seed=n + m)[0]
          for n, m in ((3, 1), (12, 256), (5, 600), (3, 1100),  # lists up to and past 1,024
                       (100, 430), (1024, 8192), (1025, 8193), (16384, 70000),
                       (16385, 70001),    # admitted by itself
                       (300, 90000))]     # too many literals for the shared launch
    fs += [random_formula(n, m, 1, 8, seed=n) for n, m in ((7, 11), (500, 1999), (3000, 9000))]
    return fs


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_states_and_results_equal_single_instances(prec):
    fs = formulas()
    x0s = [dmm.initial_state_uniform(f, 5 + k) for k, f in enumerate(fs)]
    b = dmm.Batch.for_formulas(fs, precision=prec)
    try:
        for k, (f, x0) in enumerate(zip(fs, x0s)):
            assert b.add(f, x0, max_steps=12) == k
            if k == 4:  # state read before the run: unpacks what was laid aside
                x, t = b.state(2)
                want = x0s[2] if prec == "fp64" else x0s[2].astype(np.float32).astype(np.float64)
                assert np.array_equal(x, want) and t == 0.0
        b.run()
        for k, (f, x0) in enumerate(zip(fs, x0s)):
            with dmm.Instance(f, precision=prec) as inst:
                inst.set_state(x0)
                r = inst.solve(max_steps=12)
                got, post = b.result(k)
                assert (got.steps, got.t, got.loc, got.status) == (r.steps, r.t, r.loc, r.status)
                assert np.array_equal(b.state(k)[0], inst.get_state()[0])
                assert np.array_equal(post, inst.assignment(pre=False)[1])
        # results follow later changes of the batch
        b.set_state_at(4, x0s[4], 0.0)
        assert b.result(4)[0].steps == 0
        assert np.array_equal(b.result(4)[1] > 0, x0s[4][:fs[4].n] > 0)
    finally:
        b.close()


def test_more_formulas_than_one_block_of_records():
    f, _ = dmm.generate_planted(60, 258, 0.08, 0.46, seed=1)
    x0 = dmm.initial_state_uniform(f, 2)
    count = 2100
    b = dmm.Batch.for_formulas([f] * count)
    try:
        for k in range(count):
            x = x0.copy()
            x[0] = -1 + 2 * k / count
            b.add(f, x, max_steps=3)
        b.run()
        for k in (0, 1023, 1024, 2047, 2048, count - 1):
            x = x0.copy()
            x[0] = -1 + 2 * k / count
            with dmm.Instance(f) as inst:
                inst.set_state(x)
                inst.solve(max_steps=3)
                assert np.array_equal(b.state(k)[0], inst.get_state()[0])
                assert np.array_equal(b.result(k)[1], inst.assignment(pre=False)[1])
    finally:
        b.close()


def test_bad_formulas_are_refused_and_leave_the_batch_usable():
    f, _ = dmm.generate_planted(60, 258, 0.08, 0.46, seed=1)
    x0 = dmm.initial_state_uniform(f, 2)
    b = dmm.Batch.for_formulas([f] * 3)
    try:
        b.add(f, x0, max_steps=5)
        bad = dmm.Formula(f.n, f.m, f.lits.copy(), f.clause_off)
        bad.lits[17] = f.n + 1
        with pytest.raises(dmm.DmmError) as e:
            b.add(bad, x0, max_steps=5)
        assert e.value.name == "DMM_ERR_LITERAL"
        assert b.add(f, x0, max_steps=5) == 1
        b.run()
        assert np.array_equal(b.state(0)[0], b.state(1)[0])
    finally:
        b.close()
