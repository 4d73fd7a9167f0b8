"""Volume derivative and the reference's volume-only right-hand side at every order and both types, on partitions that
start on any value and end inside a tile, against numpy on the problem's own arrays.  Bound per value: FP64, the rounding
of the sums in either order, (Np + 16) * 2^-52 times the sum of the terms' magnitudes; FP32, whose products and sums run
in FP64, the rounding of three derivatives, nine metric terms and the product with u, 16 * 2^-24 of the same."""
import numpy as np
import pytest

from dgkernel_b200 import mesh as M
from dgkernel_b200._lib import check, lib
from dgkernel_b200.burgers import GEO, _TetBurgers, _pd, random_modes

pytestmark = pytest.mark.gpu


class _Parts(_TetBurgers):
    """A periodic n^3 x 6 problem with derivative outputs whose partitions are element ranges of the given sizes."""

    derivatives = True

    def __init__(self, N, n, sizes, dtype):
        VX, VY, VZ, EToV, EToVp, _ = M.kuhn_mesh(n, 1)
        EToE, EToF = M.ti_connect3d(EToVp)
        EToP = np.repeat(np.arange(len(sizes), dtype=np.int64), sizes)
        self._assemble(N, VX, VY, VZ, EToV, EToE, EToF, EToP, sizes, dtype, None)
        r, modes = self.runner, random_modes(7)
        check(lib().dgk_init_field(r._h, b"u", b"X", b"Y", b"Z", 2, 0.5, 0.0, len(modes), _pd(modes)), r._h)
        self._finish(0.3, 0)


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("N,n,sizes", [(1, 3, (33, 1, 128)), (2, 3, (17, 145)), (3, 3, (9, 16, 137)), (4, 3, (7, 155)),
                                       (4, 10, (1, 2998, 3001)), (5, 3, (3, 159)), (6, 3, (5, 157)), (7, 3, (8, 154)),
                                       (7, 10, (17, 5983))])
def test_derivative_and_rhs(N, n, sizes, dtype):
    P = _Parts(N, n, list(sizes), dtype)
    Np, K = P.el.Np, P.K
    u = P.get("u").astype(np.float64).reshape(K, Np)
    geo = [P.get(g).astype(np.float64).reshape(K, Np) for g in GEO]
    d = [u @ D.T for D in (P.el.Dr, P.el.Ds, P.el.Dt)]
    da = [np.abs(u) @ np.abs(D).T for D in (P.el.Dr, P.el.Ds, P.el.Dt)]
    gamma = (Np + 16) * 2.0 ** -52 if dtype == np.float64 else 16 * 2.0 ** -24
    P.differentiate()
    total, mag = 0.0, 0.0
    for x, name in enumerate(("DuDx", "DuDy", "DuDz")):
        want = sum(geo[3 * k + x] * d[k] for k in range(3))
        size = sum(np.abs(geo[3 * k + x]) * (da[k] if dtype == np.float64 else np.abs(d[k])) for k in range(3))
        if dtype == np.float32:  # and the FP64 sums themselves
            size = size + 2.0 ** -24 * sum(np.abs(geo[3 * k + x]) * da[k] for k in range(3))
        assert np.all(np.abs(P.get(name).astype(np.float64).reshape(K, Np) - want) <= gamma * size)
        total, mag = total + want, mag + size
    r, sn = P.runner, P.el.ShortName
    r.ConfigureKernel("computeRHS", r.Param("u"), *[r.Param(g) for g in GEO], r.Param("DuDx"),
                      *[r.Param(f"{m}_{sn}") for m in ("Dr", "Ds", "Dt")])
    r.BuildKernel("computeRHS(rhsu=DuDx)", "computeRHS")
    r.ExecuteKernel("computeRHS")
    rhs = P.get("DuDx").astype(np.float64).reshape(K, Np)
    assert np.all(np.abs(rhs + u * total) <= gamma * np.abs(u) * mag)
    P.free()
