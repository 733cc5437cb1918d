"""The FP64 Poisson passes at every transform length of their range (16 to
4096 points: one to three radix passes, each remainder factor 2, 4, 8, each
number of rows and columns per CTA, staged and unstaged twiddle tables),
with 8 and 16 values per thread, grids padded in x, in y and in both, and
fade strips on both sides of the in-place limit of fadeCorr, against
numpy's FFT on the same padded grid."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def context(bpdx, bpdy, solver, tune):
    from cubismup_2d_b200 import Simulation
    X, Y = bpdx / max(bpdx, bpdy), bpdy / max(bpdx, bpdy)
    sim = Simulation(f"-bpdx {bpdx} -bpdy {bpdy} -extent 1 -nu 1e-3 -poissonType {solver} -muteAll 1 "
                     f"-autotune {tune} -shapes 'disk radius={0.2 * min(X, Y)} xpos={X / 2} ypos={Y / 2}'")
    sim.init()
    return sim.ctx


@pytest.mark.parametrize("bpdx,bpdy,solver", [
    (1, 1, "freespace"), (2, 1, "freespace"), (3, 2, "freespace"), (4, 5, "freespace"), (8, 16, "freespace"), (8, 20, "freespace"), (16, 10, "freespace"),
    (17, 9, "freespace"), (33, 31, "freespace"), (64, 33, "freespace"), (65, 40, "freespace"), (128, 64, "freespace"),
    (1, 1, "periodic"), (2, 4, "periodic"), (8, 2, "periodic"), (16, 64, "periodic"), (128, 16, "periodic"),
    (1, 1, "cosine"), (2, 8, "cosine"), (8, 2, "cosine"), (32, 4, "cosine"), (16, 32, "cosine"),
    (64, 64, "cosine"), (128, 16, "cosine")])
@pytest.mark.parametrize("tune", [0, 1])
def test_poisson_solve_lengths(bpdx, bpdy, solver, tune):
    from cubismup_2d_b200.synthetic import noise_field
    from oracle import cup2d_oracle as oracle
    ctx = context(bpdx, bpdy, solver, tune)
    b = noise_field(41, 0, ctx.ny, ctx.nx, amp=1.0)
    ctx.set("tmp", b)
    ctx.poisson_solve("tmp", "pres")
    faded = ctx.get("tmp")                            # the solver fades its right-hand side in place
    # (the oracle's fadeLen is a fraction of the extent, as the context's default)
    want = oracle.cub2rhs(b, oracle.Grid(bpdx, bpdy, 1.0))
    assert np.abs(faded - want).max() <= 1e-12 * np.abs(b).max()
    if solver == "freespace":
        want = oracle.poisson_freespace(faded, ctx.h, pad=0)
    elif solver == "periodic":
        want = oracle.poisson_periodic(faded)
    else:
        want = oracle.poisson_cosine(faded)
    got = ctx.get("pres")
    # rounding of two transforms each way of up to 2^13 x 2^12 points: the
    # relative 2-norm error of an FFT is at most a few eps log2 N
    err = np.linalg.norm(got - want) / np.linalg.norm(want)
    assert err <= 30 * np.finfo(float).eps * 25
    ctx.close()
