"""Whole steps on both sides of two launch rules: advDiff from the step's
start beside the placement of a swimmer (2048 blocks or more), and the row
passes' full number of rows a CTA at row transforms of 512 points or fewer
(grids of at least 74 full CTAs)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _swimmer(bpdx, bpdy):
    from cubismup_2d_b200 import Simulation
    from cubismup_2d_b200.synthetic import noise_field
    h = 1.0 / (32 * max(bpdx, bpdy))
    L = 150 * h
    s = Simulation(f"-bpdx {bpdx} -bpdy {bpdy} -extent 1 -CFL 0.1 -nu 1e-5 -poissonType freespace -muteAll 1 "
                   f"-shapes 'stefanfish L={L!r} T=1 xpos=0.5 ypos={16 * bpdy * h!r}'")
    s.init()
    c = s.ctx
    for k, f in enumerate("uv"):
        c.set(f, c.get(f) + noise_field(5, k, c.ny, c.nx, amp=1e-2))
    return s


# 2048 blocks: the first grid of the early start; 2046: below it
@pytest.mark.parametrize("bpdx,bpdy", [(64, 32), (62, 33)])
def test_advdiff_beside_the_placement(bpdx, bpdy):
    """advDiff beside the swimmer's placement reads and writes nothing that it
    does: the same bits from graph steps, from operator steps, and from
    operator steps whose advDiff runs after the placement (a field written in
    between takes it out of the overlap)."""
    out = []
    for how in ("graph", "operators", "after"):
        s = _swimmer(bpdx, bpdy)
        c = s.ctx
        if how == "graph":
            c.advance(3)
        else:
            for _ in range(3):
                dt = s.calcMaxTimestep()
                c.put_objects(dt)
                if how == "after":
                    c.set("pres", c.get("pres"))
                c.adv_diff(dt)
                c.pressure_single(dt)
                c.compute_forces(dt)
                c.end_step()
        out.append({**{f: c.get(f) for f in ("u", "v", "pres", "chi")}, "shape": c.shape(0), "sc": c.scalars()})
        c.close()
    for other in out[1:]:
        for f in ("u", "v", "pres", "chi"):
            assert np.array_equal(out[0][f], other[f]), f
        assert out[0]["shape"] == other["shape"]
        assert out[0]["sc"]["time"] == other["sc"]["time"]


# row transforms of 512, 256 and 128 points with four and eight rows a CTA
@pytest.mark.parametrize("bpdx,bpdy,solver", [(16, 10, "freespace"), (8, 19, "freespace"), (8, 32, "cosine"),
                                              (16, 32, "periodic")])
def test_disk_steps_with_full_row_ctas(bpdx, bpdy, solver):
    """Against the numpy restatement, with the tolerances of its own tests:
    1e-9 the velocity, 1e-8 the pressure."""
    from cubismup_2d_b200 import Simulation
    from cubismup_2d_b200.synthetic import noise_field
    from oracle import cup2d_oracle as oracle
    nx, ny = 32 * bpdx, 32 * bpdy
    h = 1.0 / max(nx, ny)
    R, x, y = 20 * h, 100 * h, 130 * h
    s = Simulation(f"-bpdx {bpdx} -bpdy {bpdy} -extent 1 -CFL 0.1 -nu 1e-3 -poissonType {solver} -muteAll 1 "
                   f"-shapes 'disk radius={R!r} xpos={x!r} ypos={y!r} xvel=0.2 yvel=0.05'")
    s.init()
    want = oracle.DiskSimulation(bpdx=bpdx, bpdy=bpdy, extent=1.0, nu=1e-3, CFL=0.1, center=(x, y), radius=R,
                                 xvel=0.2, yvel=0.05, poisson=solver)
    noise = [noise_field(17, c, ny, nx, amp=1e-3) for c in range(2)]
    want.u, want.v = want.u + noise[0], want.v + noise[1]
    for f, n in zip("uv", noise):
        s.ctx.set(f, s.ctx.get(f) + n)
    for _ in range(3):
        want.calc_dt()
        want.advance()
    s.ctx.advance(3)
    for f, w, tol in (("u", want.u, 1e-9), ("v", want.v, 1e-9), ("pres", want.p, 1e-8)):
        assert np.abs(s.ctx.get(f) - w).max() <= tol * np.abs(w).max(), f
    s.ctx.close()
