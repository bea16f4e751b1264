"""The wall nodes' part of the drag gradient against plain FP64 torch, on the handle's own trajectory.

The gradient by the body force of step n - 1 for the drag of step n alone passes through nothing but the wall
nodes' map (stencil moments, extrapolation, closure, collision, momentum exchange), so it needs one level of the
handle and the map written out here.  An FP32 handle's level, node tables, weights and relaxation are FP32
numbers; everything formed from them is FP64, and the gradient has to be that to FP64 rounding.

Bound: some hundred operations of 2^-53 each, times the closure's cancellation (L12 loses up to about three
digits): 1e-11 of the largest entry; 1e-10 is asked for.  One constant rounded to FP32 moves it by 1e-8 and more.
"""
import numpy as np
import pytest

from mrlbm_2d_b200.config import cylinder_case
from perf.cases import EX, EY, INCS, OUTS, W

pytestmark = pytest.mark.gpu

CLOSURES = {"strong": {}, "weak": dict(strong_mass_bc=0, weak_mass_bc=1), "rhoeq": dict(strong_mass_bc=0, eq_mass_bc=1)}


def wall_gradient(cfg, geo, omega, f, prec, closure):
    """d(drag)/d(f) for incoming populations f (nx, ny, 9): torch FP64, tables as a handle of `prec` holds them."""
    import torch

    def held(v):
        return torch.as_tensor(np.asarray(v, np.float64 if prec == 64 else np.float32).astype(np.float64))

    i, j = geo["bou_i"].astype(float), geo["bou_j"].astype(float)

    def rot(a, b):
        q = np.sqrt((a - cfg.x_c) ** 2 + (b - cfg.y_c) ** 2)
        c, s = (a - cfg.x_c) / q, (b - cfg.y_c) / q
        return c, s, 2.0 * s * c, c * c - s * s

    c, s, s2, c2 = rot(i, j)
    cc, ss, cth, sth, s2th, c2th = (held(v) for v in (c * c, s * s, c, s, s2, c2))
    d, dx = geo["delta_uk"], np.sqrt(2.0)
    t2, t3 = held(d * (d - 2.0 * dx) / (dx * dx)), held(d * (d - dx) / (2.0 * (dx * dx)))
    F = torch.as_tensor(f).requires_grad_(True)
    hx, hy = held([e * e - 1.0 / 3.0 for e in EX]), held([e * e - 1.0 / 3.0 for e in EY])
    hxy = [float(a * b) for a, b in zip(EX, EY)]
    w, om, om1 = held(W), held(omega), held(1.0 - omega)

    def moments(q):
        rho = q.sum(-1)
        ux, uy = ((q * torch.tensor(e, dtype=q.dtype)).sum(-1) / rho for e in (EX, EY))
        return rho, ux, uy, (q * hx).sum(-1) / rho, (q * hy).sum(-1) / rho, (q * torch.tensor(hxy, dtype=q.dtype)).sum(-1) / rho

    ext = []                                                  # (u, v, X, Y) extrapolated to the node
    for a in (0, 1):
        ref, st = geo["ref_xy"], geo["stencil"][:, 8 * a:8 * a + 8]
        xd, yd = (held(ref[:, 4 * q + 1 + a] - np.floor(ref[:, 4 * q + 1 + a])) for q in (0, 1))
        rows = []
        for m in range(4):
            si, sj = st[:, m], st[:, 4 + m]
            sc, sn, sn2, _ = rot(si.astype(float), sj.astype(float))
            c2m, s2m, x2m = held(sc * sc), held(sn * sn), held(sn2)
            _, u, v, xx, yy, xy = moments(F[si - 1, sj - 1])
            rows.append((u, v, xx * c2m + yy * s2m + xy * x2m, xx * s2m + yy * c2m - xy * x2m))
        ext.append([(1 - yd) * ((1 - xd) * p + xd * q) + yd * ((1 - xd) * r + xd * t) for p, q, r, t in zip(*rows)])
    u, v, X, Y = (t2 * p - t3 * q for p, q in zip(*ext))
    up, vp = u * cth + v * sth, v * cth - u * sth
    fw = F[geo["bou_i"] - 1, geo["bou_j"] - 1]
    bits = lambda t: torch.tensor([[float(ch == "1") for ch in t[q]] for q in geo["label_bc"]], dtype=torch.float64)  # noqa: E731
    I, O = bits(INCS), bits(OUTS)
    L = I if closure == "weak" else O
    lx, ly = np.array(EX) ** 2 - 1.0 / 3.0, np.array(EY) ** 2 - 1.0 / 3.0
    zero = torch.zeros_like(u)
    A, E, Ei, B11, B22, B12, rI, mI, D, F11, F22, F12 = [zero] * 12
    for k in range(9):
        cx, cy = held(EX[k] * c + EY[k] * s), held(-(EX[k] * s) + EY[k] * c)
        kxx, kyy = held(lx[k] * (c * c) + ly[k] * (s * s) + hxy[k] * s2), held(lx[k] * (s * s) + ly[k] * (c * c) - hxy[k] * s2)
        kxy = held((ly[k] - lx[k]) * 0.5 * s2 + hxy[k] * c2)
        a = w[k] * (1 + 3 * up * cx + 3 * vp * cy)
        e = a + w[k] * (4.5 * up * up * kxx + 4.5 * vp * vp * kyy + 9 * up * vp * kxy)
        b = 4.5 * w[k]
        A, E, Ei = A + L[:, k] * a, E + L[:, k] * e, Ei + I[:, k] * e
        B11, B22, B12 = B11 + L[:, k] * b * kxx, B22 + L[:, k] * b * kyy, B12 + L[:, k] * b * kxy
        rI, mI, D = rI + I[:, k] * fw[:, k], mI + I[:, k] * fw[:, k] * kxy, D + I[:, k] * a * kxy
        F11, F22, F12 = F11 + I[:, k] * b * kxx * kxy, F22 + I[:, k] * b * kyy * kxy, F12 + I[:, k] * b * kxy * kxy
    mI = mI / rI
    if closure == "rhoeq":
        Z, den = (Ei * mI - D - X * F11 - Y * F22) / (2 * F12), Ei
    else:
        beta = 1 - om if closure == "strong" else torch.ones_like(om)
        P = beta * A + om * E if closure == "strong" else A
        Z = (D - P * mI - X * (beta * B11 * mI - F11) - Y * (beta * B22 * mI - F22)) / (2 * (beta * B12 * mI - F12))
        den = P + beta * (X * B11 + Y * B22 + 2 * Z * B12)
    rho = rI / den
    xx = om1 * (X * cc + Y * ss - Z * s2th) + om * u * u
    yy = om1 * (X * ss + Y * cc + Z * s2th) + om * v * v
    xy = om1 * ((X - Y) * 0.5 * s2th + Z * c2th) + om * u * v
    drag = zero
    for k in range(9):
        fo = w[k] * rho * (1 + 3 * (EX[k] * u + EY[k] * v) + 4.5 * xx * hx[k] + 4.5 * yy * hy[k] + 9 * xy * hxy[k])
        drag = drag + EX[k] * (I[:, k] * fw[:, k] - O[:, k] * fo)
    drag.sum().backward()
    return F.grad.numpy(), w.numpy()


@pytest.mark.parametrize("prec", [64, 32])
@pytest.mark.parametrize("closure", sorted(CLOSURES))
def test_wall_gradient_is_fp64_arithmetic(mrlbm, prec, closure):
    cfg = cylinder_case(96, 32, 8, 24.0, 16.5, 100.0, 0.05, seed=11, noise=1e-2).replace(**CLOSURES[closure])
    s, t = mrlbm.Simulation(cfg, precision=prec), mrlbm.Simulation(cfg, precision=prec)
    body = 1e-5 * np.random.default_rng(2).standard_normal((2, cfg.nx, cfg.ny))
    for q in (s, t):
        q.set_body_force(body)
    s.step(20)
    t.step(21)
    _, gb, _ = s.adjoint_drag(2, 1, 5)                          # the drag of step 22, the body force of steps 21 and 22
    g, w = wall_gradient(cfg, s.boundary_nodes(), s.info.omega, t.get_state(), prec, closure)
    want = np.zeros_like(gb)
    for k in range(1, 9):                                       # population k of node x arrives at x + e_k
        lam = np.roll(g[:, :, k], (-EX[k], -EY[k]), (0, 1))
        want[0] += 3.0 * w[k] * EX[k] * lam
        want[1] += 3.0 * w[k] * EY[k] * lam
    want *= t.node_classes()["isbound"] == 0                    # no body force at curved-wall nodes
    assert np.abs(want).max() > 0.0
    assert np.abs(gb - want).max() <= 1e-10 * np.abs(want).max()
    s.close()
    t.close()
