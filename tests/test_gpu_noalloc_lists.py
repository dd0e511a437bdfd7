"""dmm_rhs3_f32_noalloc over its slot-list lengths and limits, against dmm_instance_rhs on an
FP32 instance (same arithmetic: bit-exact)."""
import ctypes

import numpy as np
import pytest

import dmm_b200 as dmm
from conftest import uniform_init
from dmm_b200 import _lib

pytestmark = pytest.mark.gpu


def call(lits, n, m, x, stream):
    import torch

    lits_d = torch.from_numpy(lits).to("cuda")
    x_d = torch.from_numpy(x.astype(np.float32)).to("cuda")
    out = torch.full((n + 2 * m,), float("nan"), dtype=torch.float32, device="cuda")
    loc = torch.full((1,), -1, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    _lib.check(_lib.lib().dmm_rhs3_f32_noalloc(
        ctypes.c_void_p(lits_d.data_ptr()), n, m, ctypes.c_void_p(x_d.data_ptr()), None,
        ctypes.c_void_p(out.data_ptr()), ctypes.c_void_p(loc.data_ptr()),
        ctypes.c_void_p(stream.cuda_stream)))
    stream.synchronize()
    return out.cpu().numpy().astype(np.float64), int(loc.item())


@pytest.mark.parametrize("n,m", [
    (3, 1), (3, 32), (3, 33),     # lists of one, 32 and 33 slots
    (12, 256), (5, 600), (3, 1024),  # up to the longest list
    (31, 700), (1000, 1), (8009, 64007),
    (32768, 65536),               # the limits
])
def test_slot_lists(n, m):
    import torch

    form, _ = dmm.generate_planted(n, m, p0=0.08, p1=0.58, seed=n + m)
    x = uniform_init(n, m, 5).astype(np.float32).astype(np.float64)
    with dmm.Instance(form, precision="fp32") as inst:
        want, want_loc, _ = inst.generate_dxdt(x)
    for _ in range(2):
        got, loc = call(form.lits, n, m, x, torch.cuda.Stream())
        assert np.array_equal(got, want) and loc == want_loc


def test_no_clauses():
    import torch

    got, loc = call(np.ones(3, dtype=np.int32), 700, 0, np.full(700, 0.5), torch.cuda.Stream())
    assert np.array_equal(got, np.zeros(700)) and loc == 0
