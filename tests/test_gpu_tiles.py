"""Whole steps of a disk, through graph steps and through the operators,
against the numpy restatement where the tile kernels and the grid kernels
change their split: one tile row, rows that end in half a warp's 64 columns,
the grids on both sides of the row passes' two-row and advDiff's early-start
rules, and a disk of more tiles than CTAs are launched for.

Tolerances (fp64): what tests/test_oracle_cpu.py derives for the restatement
itself (FFT and sum orders differ): 1e-12 the dt, 1e-9 the velocity, 1e-8 the
pressure, 1e-7 of the largest force component the forces."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# blocks, solver, the disk's radius and centre in cells
@pytest.mark.parametrize("bpdx,bpdy,solver,radius,xc,yc", [
    (3, 1, "freespace", 6.0, 40.0, 16.0), (5, 3, "freespace", 20.0, 61.0, 47.0), (7, 9, "freespace", 30.5, 96.0, 128.0),
    (8, 4, "cosine", 17.0, 127.0, 66.0), (16, 2, "periodic", 9.0, 256.0, 30.0),
    (21, 13, "freespace", 70.0, 250.0, 210.0), (40, 24, "freespace", 215.0, 500.0, 380.0)])
def test_disk_steps(bpdx, bpdy, solver, radius, xc, yc):
    from cubismup_2d_b200 import Simulation
    from cubismup_2d_b200.synthetic import noise_field
    from oracle import cup2d_oracle as oracle
    nx, ny, nsteps = 32 * bpdx, 32 * bpdy, 3
    h = 1.0 / max(nx, ny)
    R, x, y = radius * h, xc * h, yc * h
    args = (f"-bpdx {bpdx} -bpdy {bpdy} -extent 1 -CFL 0.1 -nu 1e-3 -poissonType {solver} -muteAll 1 "
            f"-shapes 'disk radius={R!r} xpos={x!r} ypos={y!r} xvel=0.2 yvel=0.05'")
    noise = [noise_field(17, c, ny, nx, amp=1e-3) for c in range(2)]
    want = oracle.DiskSimulation(bpdx=bpdx, bpdy=bpdy, extent=1.0, nu=1e-3, CFL=0.1, center=(x, y), radius=R,
                                 xvel=0.2, yvel=0.05, poisson=solver)
    want.u, want.v = want.u + noise[0], want.v + noise[1]
    for _ in range(nsteps):
        want.calc_dt()
        want.advance()

    def rel(a, b):
        return float(np.max(np.abs(a - b)) / max(np.max(np.abs(b)), 1e-300))

    for graph in (True, False):
        sim = Simulation(args)
        sim.init()
        for f, n in zip("uv", noise):
            sim.ctx.set(f, sim.ctx.get(f) + n)
        if graph:
            sim.ctx.advance(nsteps)
        else:
            for _ in range(nsteps):
                dt = sim.calcMaxTimestep()
                for op in sim.pipeline:
                    op(dt)
                sim.ctx.end_step()
        sh = sim.ctx.shape(0)
        assert abs(sim.ctx.scalars()["time"] - want.time) <= 1e-12 * want.time
        assert rel(sim.ctx.get("u"), want.u) < 1e-9 and rel(sim.ctx.get("v"), want.v) < 1e-9
        assert rel(sim.ctx.get("pres"), want.p) < 1e-8
        assert rel(sim.ctx.get("chi"), np.maximum(0.0, want.CHI)) < 1e-12
        for key, w in (("u", want.S.u), ("v", want.S.v), ("omega", want.S.omega)):
            assert abs(sh[key] - w) <= 1e-9 * max(abs(w), 1e-3), key
        F = max(abs(want.S.forces["forcex"]), abs(want.S.forces["forcey"]))
        for key in ("forcex", "forcey", "torque", "perimeter"):
            assert abs(sh[key] - want.S.forces[key]) <= 1e-7 * F, key
