"""Results of a batch read one after another (one launch makes every formula's signs): sizes around a
block's and a formula's share of the launch, against the state's own signs, and no slower for a
few large formulas than reading each by itself."""
import time

import numpy as np
import pytest

import dmm_b200 as dmm

pytestmark = pytest.mark.gpu


def batch(prec, sizes):
    forms = [dmm.generate_planted(n, m, 0.08, 0.58, seed=n + k)[0] for k, (n, m) in enumerate(sizes)]
    b = dmm.Batch.for_formulas(forms, precision=prec)
    for k, f in enumerate(forms):
        b.add(f, dmm.initial_state_uniform(f, k), max_steps=3)
    b.run()
    return b


@pytest.mark.parametrize("prec", ["fp32", "fp64"])
@pytest.mark.parametrize("sizes", [[(3, 2), (100, 430), (255, 900), (257, 900)],
                                   [(1023, 3000), (1025, 3000), (5, 9)],
                                   [(65535, 70000), (65537, 70000), (200001, 210000), (100, 400)]])
def test_signs_of_every_variable(prec, sizes):
    b = batch(prec, sizes)
    for k in range(len(sizes)):
        r, post = b.result(k)
        v = b.state(k)[0][:sizes[k][0]]
        assert r.steps > 0 and np.array_equal(post, np.where(v > 0, 1, -1))
    b.close()


def test_a_few_large_formulas():
    sizes = [(400_000, 400_000)] * 2
    b = batch("fp32", sizes)
    best = {"first": 1e9, "second": 1e9}
    for _ in range(5):
        x0 = b.state(0)[0]
        b.set_state_at(0, x0, 0.0)
        b.run()
        for k, which in ((0, "first"), (1, "second")):  # alone, then with one launch for all
            t = time.perf_counter()
            b.result(k)
            best[which] = min(best[which], time.perf_counter() - t)
    b.close()
    # both copy the same bytes twice over at most; a formula of one block took 0.3 ms by itself
    assert best["second"] <= 2.0 * best["first"] + 60e-6
