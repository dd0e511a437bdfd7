"""Distinct handles are independent: threads that create, step and solve formulas of different
sizes at the same time get what each gets alone.  The kernels' attributes belong to the function
on the device and not to a handle, so a launch must not depend on what another thread set last."""
import threading

import numpy as np
import pytest

import dmm_b200 as dmm

pytestmark = pytest.mark.gpu


def outcome(inst, x0, steps):
    inst.set_state(x0)
    r = inst.step(steps)
    return r.status, r.steps, r.t, r.loc, inst.get_state()[0]


def same(a, b):
    return a[:4] == b[:4] and np.array_equal(a[4], b[4])


def together(works):
    errors = []
    start = threading.Barrier(len(works))

    def call(f):
        try:
            start.wait()
            f()
        except Exception as e:  # noqa: BLE001 - reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=call, args=(f,)) for f in works]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]


@pytest.mark.parametrize("prec,mode,sizes", [
    ("fp32", 0, [(200, 1600), (2000, 16000)]),          # one cluster each
    ("fp64", 0, [(200, 1600), (1500, 12000)]),
    ("fp32", 0, [(5000, 21500), (30000, 240000)]),      # resident on the whole grid
    ("fp64", 0, [(5000, 21500), (30000, 240000)]),
    ("fp32", 2, [(3000, 24000), (90000, 720000)]),      # staged
])
def test_launches_of_two_sizes(prec, mode, sizes):
    """Launches of one step each, back to back, from three threads per size: the time between a
    launch and the call that prepares it is short."""
    works = []
    for n, m in sizes:
        form, _ = dmm.generate_planted(n, m, 0.08, 0.58, seed=n)
        x0 = dmm.initial_state_uniform(form, 5)
        with dmm.Instance(form, precision=prec) as inst:
            inst.set_tuning(launch_mode=mode)
            alone = outcome(inst, x0, 200)

        def work(form=form, x0=x0, alone=alone):
            with dmm.Instance(form, precision=prec) as inst:
                inst.set_tuning(launch_mode=mode, steps_per_graph=1)
                for _ in range(4):
                    inst.set_state(x0)
                    for _ in range(100):
                        inst.step(1)
                    inst.step(100)
                    assert np.array_equal(inst.get_state()[0], alone[4])
                    assert same(outcome(inst, x0, 200), alone)

        works += [work] * 3
    together(works)


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
def test_creation_and_solves_of_several_sizes(prec):
    """The table builds and the plans of each size while others launch."""
    works = []
    for n, m in [(300, 2400), (4000, 32000), (20000, 86000), (45000, 360000), (100000, 430000)]:
        form, _ = dmm.generate_planted(n, m, 0.08, 0.58, seed=n + 1)
        x0 = dmm.initial_state_uniform(form, 6)
        with dmm.Instance(form, precision=prec) as inst:
            alone = outcome(inst, x0, 8)

        def work(form=form, x0=x0, alone=alone):
            for _ in range(12):
                with dmm.Instance(form, precision=prec) as inst:
                    assert same(outcome(inst, x0, 8), alone)

        works.append(work)
    together(works)
