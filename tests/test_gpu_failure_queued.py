"""A launch that was queued before the host saw that a wait of the launch before it gave up (a run
keeps one launch in flight) takes no step: the exchange buffers it would read belong to the
abandoned step.  The failure is made on the host, as in test_gpu_failure.py; nothing faults or
hangs."""
import numpy as np
import pytest

import dmm_b200 as dmm
from dmm_b200._lib import Report, check, lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec,n,m", [("fp32", 6_000, 25_800), ("fp64", 6_000, 25_800)])
def test_queued_launch_leaves_the_record_alone(prec, n, m):
    import ctypes

    form, _ = dmm.generate_planted(n, m, 0.08, 0.58, seed=31)
    x0 = dmm.initial_state_uniform(form, 32)
    with dmm.Instance(form, precision=prec) as inst:
        inst.set_state(x0)
        before = inst.step(3)
        v_before = inst.get_state()[0][:n]
        with pytest.raises(dmm.DmmError) as e:
            check(lib().dmm_instance_test_barrier_timeout(inst._h))
        assert e.value.name == "DMM_ERR_CUDA"
        r = Report()
        check(lib().dmm_instance_report(inst._h, ctypes.byref(r)))
        assert (r.status, r.steps, r.t, r.loc, r.best_loc) == (
            before.status, before.steps, before.t, before.loc, before.best_loc) == (
            0, 3, before.t, before.loc, before.best_loc)
        assert np.array_equal(inst.get_state()[0][:n], v_before)
        # reported once: from a new state the instance integrates as another one does
        inst.set_state(x0)
        got = inst.step(10)
        x = inst.get_state()[0]
    with dmm.Instance(form, precision=prec) as ref:
        ref.set_state(x0)
        want = ref.step(10)
        assert (got.status, got.steps, got.t, got.loc) == (want.status, want.steps, want.t, want.loc)
        assert np.array_equal(x, ref.get_state()[0])
