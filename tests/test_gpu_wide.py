"""FP64 stage of orders 6 and 7 at both tile sizes (8 or 16 elements by problem size), with partial tiles,
both volume forms, against a numpy evaluation on the problem's own arrays.  Bound per value: the rounding of the sums
in either order, (terms) * 2^-52 times the sum of the terms' magnitudes."""
import numpy as np
import pytest

from dgkernel_b200.burgers import FACE, GEO, RK4B, BurgersProblem

pytestmark = pytest.mark.gpu


def _rhs_and_bound(P, u, conservative):
    el, K = P.el, P.K
    Np, NF = el.Np, 4 * el.Nfp
    u = u.reshape(K, Np)
    geo = [P.get(g).reshape(K, Np) for g in GEO]
    nx, ny, nz, fs = (P.get(f).reshape(K, NF) for f in FACE)
    w = 0.5 * u * u if conservative else u
    d = [w @ D.T for D in (el.Dr, el.Ds, el.Dt)]
    da = [np.abs(w) @ np.abs(D).T for D in (el.Dr, el.Ds, el.Dt)]
    g = sum(geo[3 * k + x] * d[k] for k in range(3) for x in range(3))
    ga = sum(np.abs(geo[3 * k + x]) * da[k] for k in range(3) for x in range(3))
    uM, uP = u[:, np.asarray(el.Fmask).reshape(-1)], u.reshape(-1)[P.vmapP].reshape(K, NF)
    ns = nx + ny + nz
    fM, fP = 0.5 * uM * uM * ns, 0.5 * uP * uP * ns
    lam = np.maximum(np.abs(uM * ns), np.abs(uP * ns))
    flux = fs * (fM - (0.5 * (fM + fP) + 0.5 * lam * (uM - uP)))
    fa = np.abs(fs) * (1.5 * np.abs(fM) + 0.5 * np.abs(fP) + 0.5 * lam * (np.abs(uM) + np.abs(uP)))
    rhs = (-g if conservative else -u * g) + flux @ el.LIFT.T
    mag = (ga if conservative else np.abs(u) * ga) + fa @ np.abs(el.LIFT).T
    return rhs, (Np + NF + 32) * 2.0 ** -52 * mag


@pytest.mark.parametrize("N", [6, 7])
@pytest.mark.parametrize("n,slabs,conservative", [(3, 1, 0), (4, 2, 1), (11, 11, 0), (13, 13, 1)])
def test_stage(N, n, slabs, conservative):
    P = BurgersProblem(N, n, slabs, np.float64, "modes", seed=3, conservative=conservative)
    u0 = P.get("u")
    rhs, tol = _rhs_and_bound(P, u0, conservative)
    dt = 0.5
    P.runner.ExecuteKernel("rhsStage", 0.0, RK4B[0], dt)
    resu, u = P.get("resu").reshape(rhs.shape), P.get("u").reshape(rhs.shape)
    assert np.all(np.abs(resu - dt * rhs) <= dt * tol)
    want = u0.reshape(rhs.shape) + RK4B[0] * resu
    assert np.all(np.abs(u - want) <= 2.0 ** -52 * (np.abs(want) + np.abs(resu)))
    P.free()
