"""Rounding of the cosine solver: against the same solve in long double it is
no further off than scipy's DCTs in double are, on vorticity-like right-hand
sides (the mean of 12; a mean's scatter is some 5%, so 10% are allowed)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def multiplier(nx, ny, tol=0.1):
    """FFTW_dirichlet.h:49-61 in long double, its cosines and sum in float."""
    ld, one, two = np.longdouble, np.float32(1), np.float32(2)
    c = [np.cos(np.pi / n * 2.0 * np.arange(n)).astype(np.float32) for n in (nx, ny)]
    fd = (one - c[0][None, :] / two - c[1][:, None] / two).astype(ld)
    pi = ld("3.14159265358979323846264338327950288")
    kx, ky = ((np.arange(n) + ld(0.5)) * (pi / n) for n in (nx, ny))
    M = -ld(0.25) / (nx * ny) / ((1 - ld(tol)) * fd + ld(tol) * ((kx * kx)[None, :] + (ky * ky)[:, None]))
    M[0, 0] = 0
    return M


def source(nx, ny, seed):
    """The curl of eight Gaussian vortices, by differences."""
    r = np.random.default_rng([seed, nx, ny])
    x, y = np.arange(nx) + 0.5, np.arange(ny) + 0.5
    b = np.zeros((ny, nx))
    for _ in range(8):
        s = min(nx, ny) * r.uniform(0.05, 0.15)
        dx, dy = x - nx * r.uniform(0.1, 0.9), y - ny * r.uniform(0.1, 0.9)
        psi = r.uniform(-0.1, 0.1) * np.outer(np.exp(-0.5 * (dy / s) ** 2), np.exp(-0.5 * (dx / s) ** 2))
        b += np.gradient(np.gradient(psi, axis=0), axis=0) + np.gradient(np.gradient(psi, axis=1), axis=1)
    return b


@pytest.mark.parametrize("bpdx,bpdy", [(2, 2), (8, 4), (16, 8), (16, 16)])
def test_solve(bpdx, bpdy):
    import scipy.fft
    from cubismup_2d_b200 import Simulation
    from oracle import cup2d_oracle as oracle
    s = Simulation(f"-bpdx {bpdx} -bpdy {bpdy} -extent 1 -nu 1e-3 -poissonType cosine -muteAll 1 "
                   f"-shapes 'disk radius=0.1 xpos=0.5 ypos={0.5 * bpdy / bpdx}'")
    s.init()
    c = s.ctx
    M, ours, plain = multiplier(c.nx, c.ny), [], []
    for seed in range(12):
        c.set("tmp", source(c.nx, c.ny, seed))
        c.poisson_solve("tmp", "pres")
        b = c.get("tmp")                              # faded in place
        want = scipy.fft.idctn(scipy.fft.dctn(b.astype(np.longdouble), type=2) * M, type=2) * (4 * c.nx * c.ny)
        for out, got in ((ours, c.get("pres")), (plain, oracle.poisson_cosine(b))):
            out.append(float(np.linalg.norm((got - want).astype(float)) / np.linalg.norm(want.astype(float))))
    assert np.mean(ours) <= 1.1 * np.mean(plain)
    c.close()
