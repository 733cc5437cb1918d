"""The device memory that adjoint runs leave behind: at most 256 MB of idle
scratch over all contexts of the process, given back when the context is
destroyed and when another allocation of the library needs it."""
import gc

import pytest

from cubismup_2d_b200 import Simulation

pytestmark = pytest.mark.gpu

KEEP = 256 << 20
SLACK = 8 << 20        # the driver's own small allocations (events, modules)


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _sim(bpdx, bpdy):
    s = Simulation(f"-bpdx {bpdx} -bpdy {bpdy} -extent 1 -CFL 0.1 -nu 1e-3 -poissonType freespace -muteAll 1 "
                   "-shapes 'disk radius=0.06 xpos=0.4 ypos=0.25 bForced=1 bFixed=1 xvel=0.2'")
    s.init()
    return s


def _gradient(s, steps=4):
    return s.ctx.adjoint(steps, every=4, w_energy=0.0, w_force=(1.0, 0.0))


def _warm():
    import torch
    torch.zeros(1, device="cuda")
    s = _sim(8, 4)                     # the kernels are loaded on first use
    _gradient(s)
    s.ctx.close()
    gc.collect()


def test_a_large_run_keeps_nothing():
    _warm()
    s = _sim(64, 32)                   # 16 MB a plane: some 600 MB of scratch
    s.ctx.calc_dt()
    before = _free()
    _gradient(s)
    assert before - _free() <= SLACK
    s.ctx.close()


def test_small_runs_share_one_bound():
    _warm()
    sims = [_sim(24, 12) for _ in range(8)]   # 2.4 MB a plane: some 90 MB of scratch each
    before = _free()
    for s in sims:
        _gradient(s)
    kept = before - _free()
    assert kept <= KEEP + SLACK
    for s in sims:
        s.ctx.close()
    gc.collect()


def test_idle_scratch_is_given_back_on_a_full_device():
    import torch
    _warm()
    a, b = _sim(24, 12), _sim(24, 12)
    before = _free()
    J = _gradient(a)[0]
    kept = before - _free()
    assert kept > 0                    # small enough to stay for a's next run
    left = _free() - kept // 2         # b's run needs as much, and half of it stays free
    fill = torch.empty(left, dtype=torch.uint8, device="cuda")
    try:
        assert _gradient(b)[0] == J
    finally:
        del fill
        torch.cuda.empty_cache()
        a.ctx.close()
        b.ctx.close()
