"""Device memory that the library takes beside a pack's own arrays: little for small packs, and none
that a formula cannot do without: where the device has no room for it the same results come from
the forms that need none."""
import contextlib

import numpy as np
import pytest

import dmm_b200 as dmm
from dmm_b200._lib import lib

pytestmark = pytest.mark.gpu

MB = 1 << 20


@contextlib.contextmanager
def device_filled(leave):
    """All but about `leave` bytes of the device's free memory held by this process."""
    import torch

    lib().dmm_release_cached_memory()
    torch.cuda.empty_cache()
    held = []
    try:
        while True:
            take = torch.cuda.mem_get_info()[0] - leave
            if take < 2 * MB:
                break
            held.append(torch.empty(take // (2 * MB) * 2 * MB, dtype=torch.uint8, device="cuda"))
        yield
    finally:
        held.clear()
        torch.cuda.empty_cache()


def make(prec, sizes):
    forms = [dmm.generate_planted(n, m, 0.08, 0.58, seed=n + k)[0] for k, (n, m) in enumerate(sizes)]
    return forms, dmm.Batch.for_formulas(forms, precision=prec)


def outcome(batch, forms):
    for k, f in enumerate(forms):
        batch.add(f, dmm.initial_state_uniform(f, 50 + k), max_steps=30)
    batch.run()
    return [(batch.result(k), batch.state(k)) for k in range(len(forms))]


def same(got, want):
    for ((ra, pa), (xa, ta)), ((rb, pb), (xb, tb)) in zip(got, want):
        assert (ra.status, ra.steps, ra.t, ra.loc, ra.best_loc) == (rb.status, rb.steps, rb.t, rb.loc,
                                                                    rb.best_loc)
        assert np.array_equal(pa, pb) and np.array_equal(xa, xb) and ta == tb
        assert abs(ra.energy - rb.energy) <= 1e-12 * abs(rb.energy)


def test_small_batch_takes_little_memory():
    import torch

    forms, b = make("fp32", [(100, 430), (120, 500)])
    outcome(b, forms)  # kernels loaded
    b.close()
    lib().dmm_release_cached_memory()
    torch.cuda.empty_cache()
    before = torch.cuda.mem_get_info()[0]
    forms, b = make("fp32", [(100, 430), (120, 500)])
    created = torch.cuda.mem_get_info()[0]
    for k, f in enumerate(forms):
        b.add(f, dmm.initial_state_uniform(f, k))
    added = torch.cuda.mem_get_info()[0]
    b.close()
    assert before - created <= 16 * MB
    assert created - added <= 4 * MB


def test_blocks_for_added_formulas_refused():
    """No room for the block that small formulas are laid aside in."""
    sizes = [(12000, 60000)] * 12
    forms, b = make("fp32", sizes)
    b.set_tuning(launch_mode=2)
    want = outcome(b, forms)
    b.close()
    forms, b = make("fp32", sizes)
    b.set_tuning(launch_mode=2)
    with device_filled(12 * MB):
        got = outcome(b, forms)
    b.close()
    same(got, want)


@pytest.mark.parametrize("prec,sizes", [("fp64", [(12000, 96000)] * 8), ("fp32", [(30000, 240000)] * 3)])
def test_tables_of_the_resident_form_refused(prec, sizes):
    forms, b = make(prec, sizes)
    want = outcome(b, forms)
    b.close()
    forms, b = make(prec, sizes)
    with device_filled(48 * MB):
        got = outcome(b, forms)
    # with memory again the next run builds the tables after all
    again = outcome_again(b, forms)
    b.close()
    same(got, want)
    same(again, want)


def outcome_again(batch, forms):
    batch.set_tuning(launch_mode=0)
    for k, f in enumerate(forms):
        batch.set_state_at(k, dmm.initial_state_uniform(f, 50 + k), 0.0)
    batch.run()
    return [(batch.result(k), batch.state(k)) for k in range(len(forms))]


def test_tables_of_the_streaming_form_refused():
    import torch

    form, _ = dmm.generate_planted(400_000, 3_200_000, 0.08, 0.58, seed=3)
    x0 = dmm.initial_state_uniform(form, 4)

    def run():
        with dmm.Instance(form, precision="fp32") as inst:
            inst.set_state(x0)
            r = inst.step(6)
            return r.steps, r.t, r.loc, inst.get_state()[0]

    want = run()
    # room for the formula and, beside it, for less than the streaming form's tables
    lib().dmm_release_cached_memory()
    before = torch.cuda.mem_get_info()[0]
    inst = dmm.Instance(form, precision="fp32")
    inst.set_state(x0)
    whole = before - torch.cuda.mem_get_info()[0]
    inst.close()
    with device_filled(whole - 100 * MB):
        got = run()
    assert got[:3] == want[:3] and np.array_equal(got[3], want[3])
