"""The swimmers' midline and raster without the reference: the Frenet
recurrence (a block scan on the device) against the serial recurrence, the
prescribed-amplitude fish's running sums, and the rastered signed distance and
deformation velocity (two threads a cell) against a walk over the points in
the reference's order (FishLibrary.cpp:419-638), ties included.

The device arrays are read from a checkpoint, whose last sections are the
body's tiles, its midline arrays and its segments."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(float).eps


def fish_points(L, h):
    """Number of midline points (FishLibrary.cpp:14-38)."""
    n_mid = int(np.ceil(L * 0.8 / (h / np.sqrt(2)) / 8)) * 8
    n_end = int(np.ceil(0.1 * L * 2 / (L * 0.8 / n_mid + 0.125 * h) / 4)) * 4
    return n_mid + 2 * n_end + 1


def placed(kind, bpdx, bpdy, cells, time, angle=0.0, y=None):
    """A body of `cells` cells placed at `time`; (context, its arrays)."""
    from cubismup_2d_b200 import Simulation
    h = 1.0 / (32 * max(bpdx, bpdy))
    L = cells * h
    y = 0.5 * bpdy * 32 * h if y is None else y
    s = Simulation(f"-bpdx {bpdx} -bpdy {bpdy} -extent 1 -CFL 0.1 -nu 1e-4 -poissonType freespace -muteAll 1 "
                   f"-shapes '{kind} L={L!r} T=1 phi=0.2 xpos=0.5 ypos={y!r} angle={angle}'")
    s.init()
    c = s.ctx
    c.set_scalars(time, 1e-3, 0, 0.0, 0.0)
    c.put_objects(1e-3)
    nm = fish_points(L, h)
    nseg = (nm - 1) // 8
    nblocks = bpdx * bpdy
    cap = min((int(np.ceil(2 * (1.2 * L + 8 * h) / (32 * h))) + 2) ** 2, nblocks)
    blob = c.checkpoint()
    end = blob.size

    def take(nbytes, dtype):
        nonlocal end
        end -= nbytes
        return blob[end:end + nbytes].view(dtype)

    A = {"seg": take(136 * nseg, np.uint8).reshape(nseg, 136)[:, :8].copy().view(np.int32)}
    pool = take(8 * (36 * nm + 16), np.float64)
    names = ["rS", "width", "p1f", "w3"] + [f"{m}_{a}" for m in ("mid0", "mid1", "frame")
                                           for a in ("rX", "rY", "vX", "vY", "norX", "norY", "vNorX", "vNorY")]
    for k, n in enumerate(names):
        A[n] = pool[k * nm:(k + 1) * nm].copy()
    for n in ("sdy", "sdx", "sD", "udy", "udx", "dist", "chi"):
        A[n] = take(8 * 1024 * cap, np.float64).reshape(cap, 32, 32).copy()
    slot = take(4 * nblocks, np.int32).copy()
    A["tiles"] = {int(slot[b]): b for b in range(nblocks) if slot[b] >= 0}
    A["L"], A["h"], A["nm"], A["bpdx"] = L, c.h, nm, bpdx
    assert A["rS"][0] == 0 and abs(A["rS"][-1] - L) <= 1e-12 * L      # the layout read is the one written
    return c, A


def serial_frenet(s, curv, curv_dt, dtype=float):
    """IF2D_Frenet2D::solve (FishUtilities.h:15-79), point by point."""
    n = len(s)
    s, curv, curv_dt = (a.astype(dtype) for a in (s, curv, curv_dt))
    r, v, nor, vnor = np.zeros((4, n, 2), dtype)
    ksi, nu = np.array([1.0, 0.0], dtype), np.array([0.0, 1.0], dtype)
    vksi, vnu = np.zeros((2, 2), dtype)
    nor[0] = nu
    for i in range(1, n):
        ds, k, kt = s[i] - s[i - 1], curv[i - 1], curv_dt[i - 1]
        r[i], v[i] = r[i - 1] + ds * ksi, v[i - 1] + ds * vksi
        dksi, dnu = k * nu, -k * ksi
        dvksi, dvnu = kt * nu + k * vnu, -kt * ksi - k * vksi
        nu, ksi = nu + ds * dnu, ksi + ds * dksi
        vnu, vksi = vnu + ds * dvnu, vksi + ds * dvksi
        ksi, nu = ksi / np.sqrt(ksi @ ksi), nu / np.sqrt(nu @ nu)
        nor[i], vnor[i] = nu, vnu
    return r, v, nor, vnor


def curvature(A, time, T=1.0):
    """StefanFish's curvature and its time derivative along the midline, from its control profile."""
    if time > T:
        rc, vc = A["p1f"], 0.0
    else:                                   # it ramps up as a cubic over the first period
        a, b = -2 * A["p1f"] / T ** 3, 3 * A["p1f"] / T ** 2
        rc, vc = a * time ** 3 + b * time ** 2, 3 * a * time ** 2 + 2 * b * time
    arg = 2 * np.pi * time / T + np.pi * 0.2 - 2 * np.pi * A["rS"] / A["L"]
    return rc * np.sin(arg), vc * np.sin(arg) + rc * np.cos(arg) * 2 * np.pi / T


# 81 to 697 midline points: up to one and up to two for each of the 512 threads
@pytest.mark.parametrize("bpdx,bpdy,cells", [(4, 2, 46), (8, 4, 90), (32, 16, 205), (32, 16, 330), (32, 16, 430)])
@pytest.mark.parametrize("time", [0.37, 1.71])
def test_frenet(bpdx, bpdy, cells, time):
    c, A = placed("stefanfish", bpdx, bpdy, cells, time)
    L = A["L"]
    r, v, nor, vnor = serial_frenet(A["rS"], *curvature(A, time))
    # every step rounds its turn and its sums a few times: 32 eps a point, of
    # the unit normal, the length, and the normal's speed times the length
    tol, speed = 32 * EPS * A["nm"], np.abs(vnor).max()
    for name, want, scale in (("nor", nor, 1.0), ("vNor", vnor, speed), ("r", r, L), ("v", v, speed * L)):
        for k, x in enumerate("XY"):
            got = A[f"mid0_{name}{x}"]
            if name in "rv":                # the device's midline is shifted to its centre of mass
                got = got - got[0]
            assert np.abs(got - want[:, k]).max() <= tol * scale, name + x
    c.close()


@pytest.mark.parametrize("bpdx,bpdy,cells", [(8, 4, 46), (8, 4, 90), (32, 16, 205), (32, 16, 330), (32, 16, 430)])
def test_frenet_rounding(bpdx, bpdy, cells):
    """Against the recurrence in long double the scan is no further off than
    the recurrence in double: the largest error over the points, the mean of
    six times; such a mean scatters by some 20% for the 81 points, so a quarter
    more is allowed."""
    off = np.zeros((2, 4))
    for time in (0.21, 0.37, 0.83, 1.3, 1.71, 2.2):
        c, A = placed("stefanfish", bpdx, bpdy, cells, time)
        exact, plain = (serial_frenet(A["rS"], *curvature(A, time), t) for t in (np.longdouble, float))
        for k, name in enumerate(("r", "v", "nor", "vNor")):
            got = np.stack([A[f"mid0_{name}{x}"] for x in "XY"], -1)
            if name in "rv":
                got = got - got[0]
            for q, a in enumerate((got, plain[k])):
                off[q, k] += float(np.abs(a - exact[k]).max() / np.abs(exact[k]).max()) / 6
        c.close()
    assert np.all(off[0] <= 1.25 * off[1]), off


@pytest.mark.parametrize("bpdx,bpdy,cells", [(8, 4, 46), (32, 16, 430)])
def test_running_sums(bpdx, bpdy, cells):
    time = 0.4
    c, A = placed("carlingfish", bpdx, bpdy, cells, time)
    s, L = A["rS"], A["L"]
    ramp, dramp = np.sin(0.5 * np.pi * time), 0.5 * np.pi * np.cos(0.5 * np.pi * time)
    arg = 2 * np.pi * (s / L - time + 0.2)
    pos = 4 / 33 * (s + 0.03125 * L) * np.sin(arg)
    vel = -4 / 33 * (s + 0.03125 * L) * 2 * np.pi * np.cos(arg)
    y, vy = ramp * pos, ramp * vel + dramp * pos
    ds, dy, dvy = np.diff(s), np.diff(y), np.diff(vy)
    dx = np.sqrt(ds * ds - dy * dy)
    x = np.concatenate([[0], np.cumsum(dx)])
    vx = np.concatenate([[0], np.cumsum(-dy / dx * dvy)])
    # differences of neighbouring points (1e-3 L apart or more) lose three
    # digits before they are summed
    tol = 32 * EPS * A["nm"] * 1e3
    for name, want, scale in (("rX", x, L), ("rY", y - y[0], L), ("vX", vx, np.abs(vy).max()),
                              ("vY", vy - vy[0], np.abs(vy).max())):
        got = A["mid0_" + name]
        assert np.abs(got - got[0] - want).max() <= tol * scale, name
    c.close()


def walk(A, center, angle, b):
    """constructSurface and constructInternl of block b, point by point in the
    order of the segments, s and side (or width offset)."""
    h, invh, bx, by = A["h"], 1.0 / A["h"], b % A["bpdx"], b // A["bpdx"]
    cell = np.arange(32) + 0.5
    X, Y = bx * 32 * h + h * cell, by * 32 * h + h * cell
    PX, PY = np.meshgrid(X, Y)
    rX, rY, nX, nY, W = (A[k] for k in ("frame_rX", "frame_rY", "frame_norX", "frame_norY", "width"))
    vX, vY, vnX, vnY = (A[k] for k in ("frame_vX", "frame_vY", "frame_vNorX", "frame_vNorY"))
    co, si = np.cos(angle), np.sin(angle)

    def at(x, y, nx, ny, o, shift):
        m0, m1 = x + o * nx, y + o * ny
        out = np.stack([co * m0 - si * m1, si * m0 + co * m1], -1)
        return out + center if shift else out

    side = {sg: (at(rX, rY, nX, nY, sg * W, True), at(vX, vY, vnX, vnY, sg * W, False)) for sg in (-1, 1)}
    best, win = np.ones((32, 32)), np.full((32, 32), -1)
    rec = []
    org = np.array([X[0], Y[0]])
    spans = [(max(a, 1), min(e, A["nm"] - 2)) for a, e in A["seg"]]
    for a, e in spans:
        for ss in range(a, e + 1):
            for sg in (-1, 1):
                P = side[sg][0]
                i0, j0 = np.floor((P[ss] - org) * invh).astype(int)
                x0, x1, y0, y1 = max(0, i0 - 1), min(32, i0 + 3), max(0, j0 - 1), min(32, j0 + 3)
                if x0 >= x1 or y0 >= y1:
                    continue
                w = (slice(y0, y1), slice(x0, x1))
                d = [(PX[w] - P[q, 0]) ** 2 + (PY[w] - P[q, 1]) ** 2 for q in (ss, ss + 1, ss - 1)]
                d1 = np.minimum(np.minimum(d[0], d[1]), d[2])
                less = best[w] > d1
                best[w] = np.where(less, d1, best[w])
                win[w] = np.where(less, len(rec), win[w])
                rec.append((ss, sg))
    dist, chi = np.full((32, 32), -1.0), np.zeros((32, 32))
    ud = np.zeros((2, 32, 32))
    for j, i in zip(*np.nonzero(win >= 0)):
        ss, sg = rec[win[j, i]]
        P, U = side[sg]
        dd = [(PX[j, i] - P[q, 0]) ** 2 + (PY[j, i] - P[q, 1]) ** 2 for q in (ss, ss + 1, ss - 1)]
        close, second = ss, ss + (1 if dd[1] < dd[2] else -1)
        d1, d2 = dd[0], min(dd[1], dd[2])
        if dd[1] < dd[0] or dd[2] < dd[0]:
            d1, close, second = d2, second, close
        q0, q1 = PX[j, i] - center[0], PY[j, i] - center[1]
        p = np.array([co * q0 + si * q1, -si * q0 + co * q1])
        dS = (rX[close] - rX[second]) ** 2 + (rY[close] - rY[second]) ** 2
        wc, wn = W[close] ** 2, W[second] ** 2
        g2 = (p[0] - rX[close]) ** 2 + (p[1] - rY[close]) ** 2
        if dS > (W[close] - W[second]) ** 2 or g2 > (max(W[close], W[second]) + 2 * h) ** 2:
            sign = -1 if g2 > wc else 1
        else:
            corr = 2 * np.sqrt(wc * wn)
            R = (wc + wn - corr + dS) * (wc + wn + corr + dS) / 4 / dS
            k1, k2 = (close, second) if wc > wn else (second, close)
            d = np.sqrt((R - max(wc, wn)) / dS)
            xc = np.array([rX[k1] + (rX[k1] - rX[k2]) * d, rY[k1] + (rY[k1] - rY[k2]) * d])
            sign = -1 if (p[0] - xc[0]) ** 2 + (p[1] - xc[1]) ** 2 > R else 1
        wgt = 1 - np.sqrt(d1) * (invh / 3)
        dist[j, i], chi[j, i] = sign * d1, wgt
        ud[:, j, i] = wgt * U[ss]
    inside = np.zeros((32, 32), dtype=bool)
    nw = np.floor(W / h).astype(int)
    for a, e in spans:
        for ss in range(a, e + 1):
            for iw in range(-nw[ss] + 1, nw[ss]):
                P = at(rX[ss], rY[ss], nX[ss], nY[ss], iw * h, True)
                U = at(vX[ss], vY[ss], vnX[ss], vnY[ss], iw * h, False)
                q = (P - org) * invh
                f = np.floor(q)
                for dj in (0, 1):
                    for di in (0, 1):
                        i, j = int(f[0]) + di, int(f[1]) + dj
                        if 0 <= i < 32 and 0 <= j < 32:
                            w = (1 - abs(q[1] - (f[1] + dj))) * (1 - abs(q[0] - (f[0] + di)))
                            ud[:, j, i] += w * U
                            chi[j, i] += w
                            inside[j, i] = True
    dist = np.where(inside & (np.abs(dist + 1) < EPS), 1.0, dist)
    ud /= np.where(chi > EPS, chi, 1)
    return np.where(dist >= 0, np.sqrt(np.abs(dist)), -np.sqrt(np.abs(dist))), ud


# straight at t = 0 and on a line of cell faces, or of cell centres: every cell
# beside the midline has ties; then bent, and turned
@pytest.mark.parametrize("kind,time,angle,off", [("stefanfish", 0.0, 0.0, 0.0), ("stefanfish", 0.0, 0.0, 0.5),
                                                 ("stefanfish", 1.71, 0.0, 0.3), ("carlingfish", 0.6, 25.0, 0.0)])
def test_raster(kind, time, angle, off):
    c, A = placed(kind, 8, 4, 60, time, angle, y=(64 + off) / 256)
    sh = c.shape(0)
    center, turn = np.array([sh["center_x"], sh["center_y"]]), sh["orientation"]
    top = max(np.abs(A[k]).max() for k in ("frame_vX", "frame_vY")) + 1e-300
    assert len(A["tiles"]) >= 2
    for slot, b in A["tiles"].items():
        dist, ud = walk(A, center, turn, b)
        # the same expressions on the same values: the distance to the bit
        # without a rotation, whose sine and cosine may differ in the last place
        assert np.abs(A["dist"][slot] - dist).max() <= (0 if angle == 0 else 1e-12)
        # up to some 100 products summed in another order, of speeds up to 2 top
        assert np.abs(A["udx"][slot] - ud[0]).max() <= 400 * EPS * top
        assert np.abs(A["udy"][slot] - ud[1]).max() <= 400 * EPS * top
    c.close()
