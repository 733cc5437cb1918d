"""cup2d_adv_diff_noalloc against the numpy restatement of advDiff at the
edges of its two paths: one and two blocks, rows that end in half a warp's
64 columns, the longest boundary (1024 cells) of the single launch and the
shortest of the two launches, long thin grids, planes that are only 8-byte
aligned, and every sign of the lab velocity (the faded inflow edges)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bpdx,bpdy,uinf,shift", [
    (1, 1, (0.2, 0.01), 0), (2, 1, (-0.2, 0.1), 0), (5, 3, (0.1, -0.3), 1), (8, 8, (0.0, 0.0), 0),
    (9, 7, (-0.2, -0.1), 1), (8, 9, (0.2, 0.3), 0), (9, 8, (0.2, 0.3), 1), (3, 40, (0.3, -0.2), 0),
    (61, 2, (-0.3, 0.2), 0)])
def test_adv_diff_noalloc_sizes(bpdx, bpdy, uinf, shift):
    import torch
    from cubismup_2d_b200 import abi
    from cubismup_2d_b200.synthetic import noise_field
    from oracle import cup2d_oracle as oracle
    nx, ny = 32 * bpdx, 32 * bpdy
    h, nu, dt = 1.0 / max(nx, ny), 3e-4, 2e-3
    f = np.stack([noise_field(31, c, ny, nx, amp=1.0) for c in range(2)])
    n = nx * ny

    def plane(a):                                     # a plane starting `shift` doubles into its buffer
        buf = torch.full((n + 2,), float("nan"), dtype=torch.float64, device="cuda")
        view = buf[shift:shift + n]
        view.copy_(torch.from_numpy(np.ascontiguousarray(a)).reshape(-1))
        return buf, view

    (_, u), (_, v) = plane(f[0]), plane(f[1])
    outs = [plane(np.zeros((ny, nx))) for _ in range(2)]
    rc = abi.lib().cup2d_adv_diff_noalloc(u.data_ptr(), v.data_ptr(), outs[0][1].data_ptr(), outs[1][1].data_ptr(),
                                          bpdx, bpdy, h, nu, dt, *uinf, torch.cuda.current_stream().cuda_stream)
    assert rc == abi.OK
    torch.cuda.synchronize()
    want = oracle.adv_diff(f[0], f[1], uinf, dt, h, nu)
    # every cell but the boundary's is the same expression, bit for bit; the
    # mean outflow is a sum of 2 (nx + ny) values in another order
    tol = 2 * (nx + ny) * np.finfo(float).eps * max(np.abs(w).max() for w in want)
    for (buf, view), w in zip(outs, want):
        got = view.cpu().numpy().reshape(ny, nx)
        assert np.array_equal(got[1:-1, 1:-1], w[1:-1, 1:-1])
        assert np.abs(got - w).max() <= tol
        rest = torch.cat([buf[:shift], buf[shift + n:]])
        assert bool(torch.isnan(rest).all())          # nothing written outside the plane
