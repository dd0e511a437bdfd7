"""Which kernel runs a formula: `Instance.step_kernel` on both sides of every line of the dispatch, and
the kernels that the cluster, resident grid and streaming ones stand in for, which the default
tuning no longer takes at small sizes, against the oracle there."""
import numpy as np
import pytest

import dmm_b200 as dmm
from conftest import uniform_init
from oracle.oracle import Oracle
from test_gpu_cluster import random_formula

pytestmark = pytest.mark.gpu


def kernel_of(form, prec, **tuning):
    with dmm.Instance(form, precision=prec) as inst:
        inst.set_tuning(**tuning)
        return inst.step_kernel, inst.launch_form


def planted(n, m):
    return dmm.generate_planted(n, m, 0.08, 0.58, seed=n + m)[0]


@pytest.mark.parametrize("prec,n,m,kernel,form", [
    # 8 clauses per variable: cluster up to about 18,000 (FP32) and 13,000 clauses (FP64)
    ("fp32", 100, 800, "cluster", "staged"), ("fp32", 2000, 16000, "cluster", "staged"),
    ("fp32", 2700, 21600, "resident-grid", "staged"),
    ("fp64", 100, 800, "cluster", "cooperative-single"),
    ("fp64", 1450, 11600, "cluster", "cooperative-single"),
    ("fp64", 1900, 15200, "resident-grid", "cooperative-single"),
    # a block's share: 9,000 literals in FP32 (444,000 clauses on 148 SMs), one tile each in FP64
    ("fp32", 54000, 432000, "resident-grid", "staged"), ("fp32", 57000, 456000, "staged", "staged"),
    ("fp64", 50000, 400000, "resident-grid", "cooperative-single"),
    ("fp64", 100000, 800000, "cooperative-single", "cooperative-single"),
    # one staged tile per block, several, and from 9 million literals on the streaming form
    ("fp32", 100000, 800000, "staged", "staged"),
    ("fp32", 700000, 2999999, "staged-multi", "staged-multi"),
    ("fp32", 700000, 3000000, "streaming", "staged-multi"),
    ("fp64", 700000, 3000000, "cooperative-single", "cooperative-single"),
])
def test_three_literal_formulas(prec, n, m, kernel, form):
    f = planted(n, m)
    assert kernel_of(f, prec) == (kernel, form)
    # the form it stands in for, when the launch shape is not left open
    assert kernel_of(f, prec, launch_mode=2) == (form, form)
    assert kernel_of(f, prec, launch_mode=1) == ("two-kernel", "two-kernel")


@pytest.mark.parametrize("prec,n,m,kernel", [("fp32", 1400, 8000, "cluster"), ("fp32", 2400, 14000, "resident-grid"),
                                             ("fp64", 1200, 7500, "cluster"), ("fp64", 2200, 13000, "resident-grid")])
def test_general_formulas(prec, n, m, kernel):
    f = random_formula(n, m, 1, 6, seed=n)
    assert kernel_of(f, prec) == (kernel, "cooperative-single")
    assert kernel_of(f, prec, launch_mode=2) == ("cooperative-single",) * 2


@pytest.mark.parametrize("prec,layout,kernel", [("fp32", 0, "staged"), ("fp32", 1, "cooperative-single"),
                                                ("fp64", 0, "cooperative-single")])
@pytest.mark.parametrize("n,m", [(100, 800), (500, 4000), (1000, 4300), (6000, 48000)])
def test_forms_stood_in_for_equal_the_oracle(prec, layout, kernel, n, m):
    form = planted(n, m)
    x0 = uniform_init(n, m, n)
    ref = Oracle(n, m, form.lits, form.clause_off, precision=prec).run(x0, 30, dump_every=1)
    with dmm.Instance(form, precision=prec) as inst:
        inst.set_tuning(launch_mode=2, u_layout=layout)
        assert inst.step_kernel == kernel
        inst.set_state(x0)
        for k in (1, 12, 17):
            r = inst.step(k)
        x, _ = inst.get_state()
    assert r.steps == ref["steps"]
    assert np.array_equal(x, ref["dump"][ref["steps"]])


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_general_form_stood_in_for_equals_the_oracle(prec):
    form = random_formula(700, 2500, 1, 25, seed=9)
    x0 = uniform_init(form.n, form.m, 3)
    ref = Oracle(form.n, form.m, form.lits, form.clause_off, precision=prec).run(x0, 30, dump_every=1)
    with dmm.Instance(form, precision=prec) as inst:
        inst.set_tuning(launch_mode=2)
        assert inst.step_kernel == "cooperative-single"
        inst.set_state(x0)
        r = inst.step(30)
        assert r.steps == ref["steps"]
        assert np.array_equal(inst.get_state()[0], ref["dump"][ref["steps"]])
