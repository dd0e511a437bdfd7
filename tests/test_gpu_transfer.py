"""State copies at the sizes where their route changes (the driver's copy, page-locked chunks of
1 MB, several chunks, page-locked callers) and from several threads at once."""
import threading

import numpy as np
import pytest

import dmm_b200 as dmm

pytestmark = pytest.mark.gpu


def round_trip(form, x0, prec):
    with dmm.Instance(form, precision=prec) as inst:
        inst.set_state(x0)
        x, t = inst.get_state()
        want = x0 if prec == "fp64" else x0.astype(np.float32).astype(np.float64)
        assert np.array_equal(x, want) and t == 0.0
        d, loc, _ = inst.generate_dxdt(x0)
        y = inst.dostep(x0, d, 0.0)
        inside = np.concatenate([np.clip(x0[:form.n], -1, 1), x0[form.n:]])
        assert np.array_equal(y, inside if prec == "fp64" else
                              inside.astype(np.float32).astype(np.float64))
        return d, loc


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("n,m", [(100, 4045), (100, 4046), (100, 4047), (1000, 65036), (1001, 65036),
                                 (4096, 129024), (4097, 260097), (30000, 700001)])
def test_round_trip(prec, n, m):
    form, _ = dmm.generate_planted(n, m, 0.08, 0.58, seed=m)
    x0 = dmm.initial_state_uniform(form, 1)
    x0[0] = 1.5  # clamped by the step only
    d, loc = round_trip(form, x0, prec)
    import torch

    pinned = torch.from_numpy(x0).pin_memory().numpy()
    d2, loc2 = round_trip(form, pinned, prec)
    assert np.array_equal(d, d2) and loc == loc2


def test_copies_from_several_threads():
    form, _ = dmm.generate_planted(20000, 160000, 0.08, 0.58, seed=3)
    errors = []

    def work(k):
        try:
            x0 = dmm.initial_state_uniform(form, k)
            for _ in range(5):
                round_trip(form, x0, "fp64" if k % 2 else "fp32")
        except Exception as e:  # noqa: BLE001 - reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors[0]
    dmm.lib().dmm_release_cached_memory()
    round_trip(form, dmm.initial_state_uniform(form, 9), "fp32")
