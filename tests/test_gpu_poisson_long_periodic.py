"""The longest transforms of the periodic solver, which keep the whole input
and output (the free-space ones of 4096 points keep half): rows of 8192 cells
and columns of 4096, FP64 with 8 and 16 values per thread against numpy's
FFT, FP32 against FP64.

Tolerances: FP64, the relative 2-norm error of two transforms each way, a few
eps log2 N, as for the shorter ones; FP32, eps = 2^-24 a level, twice the sum
of the levels of the four transforms."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

GRIDS = [(256, 1), (256, 4), (1, 128), (4, 128)]


def solve(bpdx, bpdy, options):
    from cubismup_2d_b200 import Simulation
    from cubismup_2d_b200.synthetic import noise_field
    X, Y = bpdx / max(bpdx, bpdy), bpdy / max(bpdx, bpdy)
    sim = Simulation(f"-bpdx {bpdx} -bpdy {bpdy} -extent 1 -nu 1e-3 -poissonType periodic -muteAll 1 {options} "
                     f"-shapes 'disk radius={0.2 * min(X, Y)} xpos={X / 2} ypos={Y / 2}'")
    sim.init()
    ctx = sim.ctx
    ctx.set("tmp", noise_field(43, 0, ctx.ny, ctx.nx, amp=1.0))
    ctx.poisson_solve("tmp", "pres")
    out = ctx.get("pres"), ctx.get("tmp")
    ctx.close()
    return out


@pytest.mark.parametrize("bpdx,bpdy", GRIDS)
@pytest.mark.parametrize("tune", [0, 1])
def test_fp64(bpdx, bpdy, tune):
    from oracle import cup2d_oracle as oracle
    got, faded = solve(bpdx, bpdy, f"-autotune {tune}")
    want = oracle.poisson_periodic(faded)
    assert np.linalg.norm(got - want) <= 30 * np.finfo(float).eps * 25 * np.linalg.norm(want)


@pytest.mark.parametrize("bpdx,bpdy", GRIDS)
def test_fp32(bpdx, bpdy):
    p, faded = solve(bpdx, bpdy, "")
    p32, faded32 = solve(bpdx, bpdy, "-precision fp32")
    assert np.array_equal(faded32, faded)             # the fade is FP64 in both
    tol = 4 * 2.0 ** -24 * (np.log2(2 * 32 * bpdx) + np.log2(2 * 32 * bpdy) + 2)
    assert np.linalg.norm(p32 - p) <= tol * np.linalg.norm(p)
