"""Gather indices outside the state in the kernels that read the caller's map: reported at the next synchronisation, and the
point takes its own trace, so the result has the bits of a map that points it at itself."""
import numpy as np
import pytest

import dgkernel_b200 as d
from dgkernel_b200.burgers import BurgersProblem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,dtype,kw", [(2, np.float32, {}), (5, np.float64, {}), (6, np.float64, {}), (6, np.float32, {}),
                                        (7, np.float64, {}), (7, np.float32, {}),
                                        *[(N, np.float64, {"viscosity": "pp", "mode_sigma": 0.3, "cfl": 0.02})
                                          for N in (1, 2, 3, 4, 5)]])
def test_rejected_points_take_their_own_trace(N, dtype, kw):
    P = BurgersProblem(N, 3, 1, dtype, "modes", seed=5, **kw)
    Q = BurgersProblem(N, 3, 1, dtype, "modes", seed=5, **kw)
    own = P.gmap.copy()
    fmask = np.asarray(P.el.Fmask).reshape(-1)
    NF, n = len(fmask), P.K * P.el.Np
    bad = own.copy()
    for i, (e, m) in enumerate([(0, 1), (7, NF - 1), (8, 0), (P.K // 2, NF // 2), (P.K - 1, NF - 1)]):
        bad[e * NF + m] = (2 ** 30, -1, n, -2 ** 31, 2 ** 31 - 1)[i]
        own[e * NF + m] = e * P.el.Np + fmask[m]
    P.runner.CopyToDevice("gmap", bad)
    Q.runner.CopyToDevice("gmap", own)
    for p in (P, Q):
        p.run_stages(1)
    with pytest.raises(d.DGKError, match="gather index"):
        P.runner.Sync()
    Q.runner.Sync()
    assert np.array_equal(P.get("u"), Q.get("u")) and np.array_equal(P.get("resu"), Q.get("resu"))
    P.runner.CopyToDevice("gmap", P.gmap)  # the context stays usable
    P.run_stages(1)
    P.runner.Sync()
    for p in (P, Q):
        p.free()
