"""The streaming form (one large formula, tiles passing through shared memory) against the tile
form: states bit for bit."""
import numpy as np
import pytest

import dmm_b200 as dmm

pytestmark = pytest.mark.gpu


def mixed_formula(n, m, seed):
    """Clauses of 1 to 6 literals, a variable at most once per clause."""
    rng = np.random.default_rng(seed)
    lens = rng.choice(np.arange(1, 7), size=m, p=[0.002, 0.148, 0.5, 0.2, 0.1, 0.05])
    off = np.zeros(m + 1, dtype=np.int64)
    np.cumsum(lens, out=off[1:])
    clause = np.repeat(np.arange(m), lens)
    var = rng.integers(0, n, size=int(off[-1]))
    while True:
        key = clause * n + var
        order = np.argsort(key, kind="stable")
        again = np.zeros(len(var), dtype=bool)
        again[order[1:]] = key[order[1:]] == key[order[:-1]]
        if not again.any():
            break
        var[again] = rng.integers(0, n, size=int(again.sum()))
    lits = ((var + 1) * rng.choice([-1, 1], size=len(var))).astype(np.int32)
    return dmm.from_arrays(lits, off, n)


def compare(form, x0, steps):
    out = []
    for mode in (0, 2):
        with dmm.Instance(form, precision="fp32") as inst:
            inst.set_tuning(launch_mode=mode)
            inst.set_state(x0)
            for k in steps:
                r = inst.step(k)
            out.append((inst.get_state()[0], r.steps, r.t, r.loc, r.best_loc, r.energy, r.status,
                        inst.assignment(pre=False)[1]))
    a, b = out
    assert np.array_equal(a[0], b[0]) and a[1:7] == b[1:7] and np.array_equal(a[7], b[7])


@pytest.mark.parametrize("n,m", [(700_003, 3_010_013), (375_001, 3_000_008)])
def test_three_literal_formulas(n, m):
    form, _ = dmm.generate_planted(n, m, 0.08, 0.46, seed=n)
    with dmm.Instance(form, precision="fp32") as inst:
        assert inst.launch_form == "staged-multi"
    compare(form, dmm.initial_state_uniform(form, 2), [1, 2, 4])


def test_general_clauses_with_units_not_pinned_at_first():
    form = mixed_formula(400_001, 2_800_003, 5)
    assert form.nlits >= 9_000_000
    rng = np.random.default_rng(1)
    x0 = np.concatenate([rng.uniform(-1, 1, form.n), rng.uniform(0, 1, form.m), np.ones(form.m)])
    compare(form, x0, [1, 3])
