"""Small inputs of the sensor network in the composite stage keep their bits.  The state is two large modes per element and
one of the highest degree of 1e-8 to 3e-8 of the whole; the network looks at that one alone, through a large weight, so
the viscosity follows its value.

Bound, relative to the viscous change of one stage against the FP64 oracle: 5e-6.  An input is good to 2.4e-7 (pair 1.2e-7,
FP32 feature 6e-8, modal transform 6e-8) and the gain from it to eps is below one; the network's FP32 sums, its two tanh
and the sigmoid add about 1e-6, the FP32 residual 1e-7.  Inputs good to 2.9e-11 absolute give 2e-4."""
import numpy as np
import pytest

from dgkernel_b200.burgers import BurgersProblem, MIXED
from oracle import burgers_ref as b
from oracle import mlp_ref as MR
from oracle import oracle as O

pytestmark = pytest.mark.gpu
H = 32


@pytest.mark.parametrize("N", [1, 2, 3, 4])
def test_small_inputs(N):
    eps0, conf = 50.0, (0.5, 0.5)  # an empty band: the network's value stands
    P = BurgersProblem(N, 3, 1, MIXED, "modes", mma=True, learned="mlp", eps0=eps0, conf=conf)
    P.dt = 1e-6
    nin = P.el.Np
    deg = O.mode_degrees(N)
    k = int(np.flatnonzero(deg == N)[-1])
    lin = int(np.flatnonzero(deg == 1)[0])
    assert k != lin and k % 16 != lin % 16
    rng = np.random.default_rng(6)
    c = np.zeros((P.K, nin))
    c[:, 0] = 1.0 + 0.1 * rng.normal(size=P.K)
    c[:, lin] = 0.2 * rng.normal(size=P.K)
    c[:, k] = rng.choice([-1.0, 1.0], P.K) * 10.0 ** rng.uniform(-8.0, -7.5, P.K)
    P.set("u", (c @ np.asarray(P.el.V).T).reshape(-1))
    p = np.zeros(H * nin + H + H * H + H + H + 1, dtype=np.float32)
    p[k] = 60000.0                   # W1[0][k]
    p[H * nin + H] = 256.0           # W2[0][0]
    p[H * nin + H + H * H + H] = 2.0  # w3[0]
    P.set_sensor("mlp", p)
    u0 = P.get("u")
    P.run_stages(1)

    def oracle(mode):
        u = u0.copy()
        O.AVState(b.Problem(N, 3, 1, "sine"), eps0=eps0, conf=conf).run(u, np.zeros_like(u), P.dt, 1, mode,
                                                                       mlp=MR.to_fp16(p) if mode == "mlp" else None)
        return u
    want, plain = oracle("mlp"), oracle("none")
    feat = O.AVState(b.Problem(N, 3, 1, "sine")).sensor(u0)[2]
    out = MR.forward(MR.to_fp16(p), feat, nin)[0]
    assert out.std() > 0.05 and np.abs(feat[:, k]).max() < 4e-8
    err = np.linalg.norm(P.get("u") - want) / np.linalg.norm(want - plain)
    print(f"order {N}: error {err:.2e} of the viscous change; outputs {out.min():.3f} .. {out.max():.3f}")
    assert err < 5e-6
    P.free()
