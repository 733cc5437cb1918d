"""The FP32 Poisson passes against the FP64 ones over their transform lengths:
one to four columns a CTA, a last group of one column, rows that leave a CTA
part empty, and every number of radix passes.

Tolerance: a transform of n points in FP32 is off by at most about eps log2 n
in the 2-norm (eps = 2^-24, the rounding of each of its levels), and a solve
is one forward and one inverse transform in each direction; twice their sum."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bpdx,bpdy,solver", [
    (1, 1, "freespace"), (2, 1, "freespace"), (3, 5, "freespace"), (7, 9, "freespace"), (9, 18, "freespace"),
    (33, 17, "freespace"), (40, 35, "freespace"), (65, 33, "freespace"), (128, 64, "freespace"),
    (1, 2, "periodic"), (4, 16, "periodic"), (32, 32, "periodic"), (2, 64, "periodic"), (128, 4, "periodic")])
def test_fp32_lengths(bpdx, bpdy, solver):
    from cubismup_2d_b200 import Simulation
    from cubismup_2d_b200.synthetic import noise_field
    nx, ny = 32 * bpdx, 32 * bpdy
    f = noise_field(41, 0, ny, nx, amp=1.0)
    out = {}
    for prec in ("fp64", "fp32"):
        sim = Simulation(f"-bpdx {bpdx} -bpdy {bpdy} -extent 1 -nu 1e-3 -poissonType {solver} -muteAll 1 "
                         f"-precision {prec} -shapes 'disk radius=0.1 xpos=0.5 ypos=0.2'")
        sim.init()
        sim.ctx.set("tmp", f)
        sim.ctx.poisson_solve("tmp", "pres")
        out[prec] = sim.ctx.get("pres"), sim.ctx.get("tmp")
        sim.ctx.close()
    (p, faded), (p32, faded32) = out["fp64"], out["fp32"]
    assert np.array_equal(faded32, faded)             # the fade is FP64 in both
    tol = 4 * 2.0 ** -24 * (np.log2(2 * nx) + np.log2(2 * ny) + 2)
    assert np.linalg.norm(p32 - p) <= tol * np.linalg.norm(p)
