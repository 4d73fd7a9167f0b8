"""The sensor network's FP16 tensor products at every order (inputs 4, 10, 20 and 35: one to three k-steps of 16,
the last one padded), on a mesh whose last group of 8 elements is partial.

Bound: relative L2 against the FP64 oracle after 5 LSERK4 stages of 1.2e-7, the mixed form's 1e-7 plus the network's
share (FP32 sums over inputs carried to 2^-23 against the oracle's FP64 sums)."""
import numpy as np
import pytest

from dgkernel_b200 import sensor as SN
from dgkernel_b200.burgers import BurgersProblem, MIXED
from oracle import burgers_ref as b
from oracle import mlp_ref as MR
from oracle import oracle as O

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N", [1, 2, 3, 4])
def test_network_at_every_order(N):
    nin = (N + 1) * (N + 2) * (N + 3) // 6
    base = SN.init_params(nin, seed=5)
    p = (base * 3 + np.random.default_rng(4).normal(size=base.size) * 0.1).astype(np.float32)
    P = BurgersProblem(N, 3, 1, MIXED, "modes", mode_sigma=0.3, mma=True, learned="mlp")
    P.dt *= 0.05  # the diffusive limit of a coarse mesh at low order
    P.set_sensor("mlp", p)
    u0 = P.u0.copy()
    P.run_stages(5)
    u = np.ascontiguousarray(u0, dtype=np.float64).copy()
    resu = np.zeros_like(u)
    O.AVState(b.Problem(N, 3, 1, "sine")).run(u, resu, P.dt, 5, "mlp", mlp=MR.to_fp16(p))
    Q = BurgersProblem(N, 3, 1, MIXED, "modes", mode_sigma=0.3, mma=True)
    Q.dt = P.dt
    Q.build_stage()
    Q.run_stages(5)
    err, gap = rel_l2(P.get("u"), u), rel_l2(Q.get("u"), u)
    print(f"order {N}: relative L2 vs oracle {err:.3e}; without viscosity {gap:.3e}")
    assert err < 1.2e-7 and gap > 10 * err, (err, gap)
    P.free()
    Q.free()
