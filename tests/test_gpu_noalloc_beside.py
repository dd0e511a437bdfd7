"""The allocation-free right-hand side beside a kernel that holds some of the SMs for a long time, as
a caller's other streams may: it runs on the others and returns while that kernel still runs."""
import ctypes
import threading
import time

import numpy as np
import pytest

import dmm_b200 as dmm
from dmm_b200 import _lib

pytestmark = pytest.mark.gpu


def random_3sat(n, m, seed):
    """Clauses of three distinct variables with random signs (at 8 per variable: unsatisfiable)."""
    rng = np.random.default_rng(seed)
    v = rng.integers(0, n, size=(2 * m, 3))
    v = v[(v[:, 0] != v[:, 1]) & (v[:, 0] != v[:, 2]) & (v[:, 1] != v[:, 2])][:m]
    lits = (v + 1) * rng.choice([-1, 1], size=v.shape)
    return dmm.from_arrays(lits.astype(np.int32).ravel(), np.arange(m + 1) * 3, n)


def test_returns_while_another_kernel_holds_sms():
    import torch

    # one cluster of 16 blocks with some 110 KB of shared memory each, for about a second
    hold = random_3sat(1500, 12000, 1)
    steps = 100_000
    form, _ = dmm.generate_planted(8009, 64007, 0.08, 0.58, seed=2)
    x0 = dmm.initial_state_uniform(form, 3).astype(np.float32)
    lits_d, x_d = torch.from_numpy(form.lits).cuda(), torch.from_numpy(x0).cuda()
    out_d = torch.empty_like(x_d)
    loc_d = torch.empty(1, dtype=torch.int32, device="cuda")
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()

    def rhs():
        out_d.fill_(float("nan"))
        torch.cuda.current_stream().synchronize()
        _lib.check(_lib.lib().dmm_rhs3_f32_noalloc(
            ctypes.c_void_p(lits_d.data_ptr()), form.n, form.m, ctypes.c_void_p(x_d.data_ptr()),
            None, ctypes.c_void_p(out_d.data_ptr()), ctypes.c_void_p(loc_d.data_ptr()),
            ctypes.c_void_p(stream.cuda_stream)))
        return out_d.cpu().numpy(), int(loc_d.item())

    with torch.cuda.stream(stream), dmm.Instance(hold, precision="fp64") as inst:
        alone = rhs()
        inst.set_state(dmm.initial_state_uniform(hold, 4))
        inst.step(10)  # kernels loaded
        ended = threading.Event()
        got = []

        def run():
            got.append(inst.step(steps))
            ended.set()

        t = threading.Thread(target=run)
        t.start()
        time.sleep(0.1)
        beside = [rhs() for _ in range(3)]
        still_running = not ended.is_set()
        t.join()
        assert got[0].steps == steps + 10
        assert still_running
        for d, loc in beside:
            assert np.array_equal(d, alone[0]) and loc == alone[1]
