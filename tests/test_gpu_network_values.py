"""The sensor network where its value decides: with an empty low-confidence band every element takes it (inside the band
the Persson-Peraire activation stands, whatever the network gives).

Bounds: the network's output against the FP64 restatement with FP16 weights 2e-5 (FP32 features and sums: weights up to 3 and
56 inputs give 1e-5 at the first layer's worst, damped by the tanh and the sigmoid); the FP64 viscosity stage 1e-6 after 10
stages and the composite 1.2e-7 after 5, the bounds of their own tests.  Either must differ from the run with the
Persson-Peraire sensor by a hundred times its bound."""
import numpy as np
import pytest

from dgkernel_b200 import sensor as SN
from dgkernel_b200.burgers import BurgersProblem, MIXED
from oracle import burgers_ref as b
from oracle import mlp_ref as MR
from oracle import oracle as O

from conftest import rel_l2

pytestmark = pytest.mark.gpu
EMPTY = (0.5, 0.5)


def _params(nin):
    return (3 * SN.init_params(nin, seed=5)).astype(np.float32)


def _oracle(ref, u0, dt, stages, sensor, p):
    u = np.ascontiguousarray(u0, dtype=np.float64).copy()
    O.AVState(ref, conf=EMPTY).run(u, np.zeros_like(u), dt, stages, sensor, mlp=MR.to_fp16(p) if sensor == "mlp" else None)
    return u


@pytest.mark.parametrize("N,n", [(1, 4), (2, 3), (3, 3), (4, 3), (5, 3)])
def test_viscosity_stage(N, n):
    P = BurgersProblem(N, n, 1, u0="modes", seed=5, mode_sigma=0.3, viscosity="pp", cfl=0.02, conf=EMPTY)
    p, ref = _params(P.el.Np), b.Problem(N, n, 1, "sine")
    P.set_sensor("mlp", p)
    u0 = P.get("u")
    got = P.sensor_features("mlp")[2]
    want = MR.forward(MR.to_fp16(p), O.AVState(ref).sensor(u0)[2], P.el.Np)[0]
    assert want.max() - want.min() > 0.4
    assert np.max(np.abs(got - want)) < 2e-5
    P.run_stages(10)
    w = _oracle(ref, u0, P.dt, 10, "mlp", p)
    err, gap = rel_l2(P.get("u"), w), rel_l2(_oracle(ref, u0, P.dt, 10, "pp", p), w)
    print(f"order {N}: output {np.max(np.abs(got - want)):.1e}, stage {err:.1e}, PP instead {gap:.1e}")
    assert err < 1e-6 and gap > 1e-4
    P.free()


@pytest.mark.parametrize("N", [1, 2, 3, 4])
def test_composite(N):
    P = BurgersProblem(N, 3, 1, MIXED, "modes", mode_sigma=0.3, mma=True, learned="mlp", conf=EMPTY)
    P.dt *= 0.05  # the diffusive limit of a coarse mesh at low order
    p, ref = _params(P.el.Np), b.Problem(N, 3, 1, "sine")
    P.set_sensor("mlp", p)
    u0 = P.u0.copy()
    P.run_stages(5)
    w = _oracle(ref, u0, P.dt, 5, "mlp", p)
    err, gap = rel_l2(P.get("u"), w), rel_l2(_oracle(ref, u0, P.dt, 5, "pp", p), w)
    print(f"order {N}: composite {err:.1e}, PP instead {gap:.1e}")
    assert err < 1.2e-7 and gap > 1.2e-5
    P.free()
