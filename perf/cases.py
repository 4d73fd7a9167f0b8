"""The work that a program using dgkernel_b200 has the GPU do, as cases that can be timed and compared.

Every case goes through the package's public entry points (`BurgersProblem`, `BurgersEnsemble`, `SensorNet`) and is
one unit of a time-stepping or training program: one LSERK4 step of a single-buffer state (five stages), two steps
of a mixed-precision state followed by the joined FP64 read-out, one volume derivative, one reference-form
right-hand side and update, one training step of the sensor network.

The time step is well below the CFL step, so that a state can be advanced thousands of times before the unlimited
scheme meets its shock; the stage kernels' work does not depend on it.  The result of a step is the state u (the
first stage of the next step multiplies the residual by zero); the FP64 forms of orders 1 to 5 return the residual
as well.  It is left out where a change in the order of a sum shows in it a thousand times larger than in u: in
the forms that keep it in FP32, and at orders 6 and 7, whose node set is ill-conditioned.  Initial states are seeded: eight
random cosine modes about 0.5 (the benchmark's field), or a steep front over the same modes where a shock sensor is
part of the work (about a tenth of the elements see it, as near the shock time of the viscosity configuration).
"""
import math

import numpy as np
import torch

from dgkernel_b200.burgers import (MIXED, RK4A, RK4B, BurgersEnsemble, BurgersProblem, ensemble_sizes,
                                   mlp_param_count)
from dgkernel_b200.sensor import SensorNet, init_params

GEO = ("Rx", "Ry", "Rz", "Sx", "Sy", "Sz", "Tx", "Ty", "Tz")
FACE = ("nx", "ny", "nz", "Fscale")
DT, DT32 = 2e-5, 2e-4  # time step (see above); FP32 states take a larger one, which their rounding does not hide


def np_of(N):
    return (N + 1) * (N + 2) * (N + 3) // 6


def nf_of(N):
    return 2 * (N + 1) * (N + 2)


def listed():
    return [
        # the reference's own parity configuration (order 2, 8^3 x 6, 4 partitions): launches and host calls count
        {"name": "step_fp64_small", "kind": "fp64", "N": 2, "n": 8, "slabs": 4, "conservative": 0},
        # a few small instances of the batch form, replayed as a captured graph of two steps
        {"name": "graph_ensemble_small", "kind": "ensemble", "N": 3, "count": 6, "lo": 4, "hi": 9, "graph": True,
         "conservative": 0},
        # the plain FP64 stage at the benchmark's order and partition count
        {"name": "step_fp64_n4", "kind": "fp64", "N": 4, "n": 32, "slabs": 16, "conservative": 0},
        # the plain FP32 stage on the same mesh
        {"name": "step_fp32_n4", "kind": "fp32", "N": 4, "n": 32, "slabs": 16, "conservative": 0},
        # the plain FP64 stage at the highest order (the precision configuration's reference run)
        {"name": "step_fp64_n7", "kind": "fp64", "N": 7, "n": 16, "slabs": 4, "conservative": 0},
        # the chosen form of the benchmark: mixed precision with tensor-core products
        {"name": "step_mma_n4", "kind": "mma", "N": 4, "n": 40, "slabs": 8, "conservative": 0},
        # the batch form: uneven independent instances of order 3 in one launch (default product form)
        {"name": "ensemble_n3", "kind": "ensemble", "N": 3, "count": 24, "lo": 6, "hi": 24, "graph": False,
         "conservative": 0},
        # the precision form (order 7, exact digit products)
        {"name": "step_precision_n7", "kind": "precision", "N": 7, "n": 16, "slabs": 1, "conservative": 0},
        # the FP64 artificial-viscosity stage with the Persson-Peraire sensor on a steep front
        {"name": "step_viscosity_n4", "kind": "viscosity", "N": 4, "n": 24, "slabs": 1, "sensor": "pp"},
        # the composite: tensor-core stage, sensor network over every element, sparse viscous term
        {"name": "step_learned_n4", "kind": "learned", "N": 4, "n": 32, "slabs": 1, "sensor": "mlp0"},
        # the volume derivative (the reference's bandwidth test) at the benchmark's order
        {"name": "derivative_n4", "kind": "derivative", "N": 4, "n": 32, "slabs": 16, "dtype": "float64",
         "reference": False},
        # one Adam step of the sensor network on a mini-batch of the trainer's default size
        {"name": "train_n4", "kind": "train", "N": 4, "batch": 8192},
    ]


# drawn cases: per kind the orders it is built for and the most degrees of freedom (of its listed case)
_RANGES = {"fp64": (1, 7, 2.9e6), "fp32": (1, 7, 6.8e6), "compact": (1, 5, 6.8e6), "mma": (1, 4, 1.3e7),
           "mixed": (1, 5, 6.8e6), "precision": (4, 7, 2.9e6), "viscosity": (1, 5, 2.9e6), "learned": (1, 4, 6.8e6),
           "derivative": (1, 7, 6.8e6)}


def draw(rng):
    kind = rng.choice(sorted(_RANGES) + ["ensemble", "train"])
    if kind == "train":
        return {"kind": kind, "N": rng.randint(1, 5), "batch": int(round(2 ** rng.uniform(8, 13)))}
    if kind == "ensemble":
        lo = rng.randint(4, 8)
        return {"kind": kind, "N": rng.randint(1, 4), "count": rng.randint(2, 16), "lo": lo,
                "hi": lo + rng.randint(2, 8), "graph": rng.random() < 0.5, "conservative": rng.randint(0, 1)}
    a, b, most = _RANGES[kind]
    N = rng.randint(a, b)
    dofs = math.exp(rng.uniform(math.log(2e4), math.log(most)))
    n = max(3, int((dofs / (6 * np_of(N))) ** (1.0 / 3.0)))
    slabs = rng.choice([s for s in range(1, min(n, 16) + 1) if n % s == 0])
    case = {"kind": kind, "N": N, "n": n, "slabs": slabs}
    if kind in ("viscosity", "learned"):
        case["sensor"] = rng.choice(["pp", "mlp"] if kind == "viscosity" else ["pp", "mlp0"])
    elif kind == "derivative":
        case["dtype"] = rng.choice(["float64", "float32"])
        case["reference"] = rng.random() < 0.5
    else:
        case["conservative"] = rng.randint(0, 1)
    return case


# ---- device views -------------------------------------------------------------------------------------------
class _Device:
    """Device memory of a runner, which lives as long as a view of it."""

    def __init__(self, runner, ptr, count, typestr):
        self.runner = runner
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (ptr, False), "version": 2}


_TYPES = {"float64": "<f8", "float32": "<f4", "int32": "<i4", "int64": "<i8"}


class _Views:
    """Torch views of a runner's arrays by device address (the ping-pong state alternates between two)."""

    def __init__(self, runner):
        self.runner, self.seen = runner, {}

    def flat(self, name, dtype):
        ptr = self.runner.DevicePtr(name)
        key = (ptr, dtype)
        if key not in self.seen:
            count = self.runner.GetOffsets(name)[-1]
            self.seen[key] = torch.as_tensor(_Device(self.runner, ptr, count, _TYPES[dtype]), device="cuda")
        return self.seen[key]


# ---- inputs -------------------------------------------------------------------------------------------------
def _front(problem, seed):
    """The seeded modes plus a steep front of about one element across a random axis direction."""
    rng = np.random.default_rng(seed)
    views = _Views(problem.runner)
    dt = "float64"
    X, Y, Z = (views.flat(c, dt) for c in "XYZ")
    k = [(1, 0, 0), (0, 1, 0), (0, 0, 1)][int(rng.integers(3))]
    phi = float(rng.uniform(-1.0, 1.0))
    s = torch.sin(math.pi * (k[0] * X + k[1] * Y + k[2] * Z - phi))
    front = 0.3 * torch.tanh(s * problem.n / 4.0)
    return torch.from_numpy(problem.u0).cuda().add_(front).cpu().numpy()


def _network(N, seed):
    """An untrained network whose outputs stay inside the low-confidence band: the sensor falls back to the
    Persson-Peraire activation, so the result does not hang on an output at a threshold."""
    return 0.5 * init_params(np_of(N), seed=1 + seed % 1000)


def prepare(case, seed):
    kind, N = case["kind"], case["N"]
    if kind == "train":
        return _prepare_train(case, seed)
    if kind == "ensemble":
        p = BurgersEnsemble(N, ensemble_sizes(case["count"], case["lo"], case["hi"]), seed=1 + seed,
                            conservative=case["conservative"])
        p.dt = min(p.dt, DT)
        state = {"p": p, "mixed": True}
        if case["graph"]:
            state["graph"] = p.capture_steps(2)
    else:
        kw = {"seed": 1 + seed, "u0": "modes"}
        if kind == "viscosity":
            kw.update(viscosity="pp", mode_sigma=0.05)
        elif kind == "learned":
            kw.update(dtype=MIXED, mma=True, learned="pp", mode_sigma=0.05)
        elif kind == "derivative":
            kw.update(dtype=np.dtype(case["dtype"]), derivatives=True)
        else:
            kw["conservative"] = case["conservative"]
            kw.update({"fp64": {"dtype": np.float64}, "fp32": {"dtype": np.float32},
                       "compact": {"dtype": np.float64, "compact": True}, "mma": {"dtype": MIXED, "mma": True},
                       "mixed": {"dtype": MIXED, "tensor": False}, "precision": {"dtype": MIXED, "tensor": True}}[kind])
        p = BurgersProblem(N, case["n"], case["slabs"], **kw)
        p.dt = min(p.dt, DT32 if kind == "fp32" else DT)
        state = {"p": p, "mixed": kind in ("mma", "mixed", "precision", "learned")}
        if kind in ("viscosity", "learned"):
            p.set("u", _front(p, seed))
            if case["sensor"] != "pp":
                p.set_sensor(case["sensor"], _network(N, seed))
        if kind == "derivative" and case["reference"]:
            r, sn = p.runner, p.el.ShortName
            r.ConfigureKernel("computeRHS", r.Param("u"), *[r.Param(g) for g in GEO], r.Param("DuDx"),
                              *[r.Param(f"{m}_{sn}") for m in ("Dr", "Ds", "Dt")])
            r.BuildKernel("computeRHS(rhsu=DuDx)", "computeRHS")
            r.ConfigureKernel("lserkUpdate", r.Param("u"), r.Param("resu"), r.Param("DuDx"), r.Param("a"),
                              r.Param("b"), r.Param("dt"))
            r.BuildKernel("lserkUpdate(rhs=DuDx)", "lserkUpdate")
    state.update(case=case, views=_Views(p.runner))
    return state


def _prepare_train(case, seed):
    """A mini-batch of unit-norm modal coefficients that fall off with the mode, their activations, and a network
    in the middle of its training (Adam moments of the size that gradients have)."""
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    nin, n = np_of(case["N"]), case["batch"]
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    X = rand(n, nin) * torch.exp(-4.0 * torch.rand(n, 1, generator=g, device="cuda") *
                                 torch.linspace(0.0, 1.0, nin, device="cuda"))
    X = X / X.norm(dim=1, keepdim=True)
    y = torch.clamp(2.0 * torch.rand(n, generator=g, device="cuda") - 0.8, 0.0, 1.0)
    net = SensorNet(nin, seed=1 + seed % 1000)
    net.m.copy_(1e-3 * rand(net.P))
    net.v.copy_(1e-6 + 1e-6 * rand(net.P) ** 2)
    net.t = 100
    return {"net": net, "X": X, "y": y, "case": case}


def _residual(case):
    return case["kind"] in ("fp64", "compact", "viscosity") and case["N"] <= 5


# ---- one pass -----------------------------------------------------------------------------------------------
def run(state):
    case = state["case"]
    if case["kind"] == "train":
        net = state["net"]
        loss = net.step(state["X"], state["y"])
        return {"loss": loss, "grad": net.g, "params": net.p, "m": net.m, "v": net.v}
    p, views = state["p"], state["views"]
    if case["kind"] == "derivative":
        dt = case["dtype"]
        if not case["reference"]:
            p.differentiate()
            return [views.flat(d, dt) for d in ("DuDx", "DuDy", "DuDz")]
        p.runner.ExecuteKernel("computeRHS")
        p.runner.ExecuteKernel("lserkUpdate", RK4A[1], RK4B[1], p.dt)
        return {"rhs": views.flat("DuDx", dt), "u": views.flat("u", dt), "resu": views.flat("resu", dt)}
    if not state["mixed"]:
        p.run_stages(5)
        dt = "float32" if case["kind"] == "fp32" else "float64"
        out = {"u": views.flat("u", dt)}
        if _residual(case):
            out["resu"] = views.flat("resu", dt)
        return out
    if "graph" in state:
        p.run_graph(state["graph"])
    else:
        p.run_stages(10)
    p.runner.ExecuteKernel("joinState")
    return {"u": views.flat("u", "float64")}


# ---- what a pass cannot do without --------------------------------------------------------------------------
def work(case):
    kind, N = case["kind"], case["N"]
    Np, NF = np_of(N), nf_of(N)
    if kind == "train":
        P, n = mlp_param_count(Np), case["batch"]
        return {"bytes": 4.0 * (n * (Np + 1) + 8 * P), "flops": 6.0 * n * (32 * Np + 32 * 32 + 32)}
    if kind == "ensemble":
        K = sum(6 * m ** 3 for m in ensemble_sizes(case["count"], case["lo"], case["hi"]))
    else:
        K = 6 * case["n"] ** 3
    dofs, r = float(K * Np), NF / Np
    if kind == "derivative":
        w = 8 if case["dtype"] == "float64" else 4
        if case["reference"]:  # u, 9 metrics, rhs; then u and resu read and written, rhs read
            return {"bytes": dofs * w * 16, "flops": dofs * (6 * Np + 30)}
        return {"bytes": dofs * w * 13, "flops": dofs * (6 * Np + 15)}
    # a stage: three derivative products and LIFT per node, and the point-wise terms
    flops = 6 * Np + 2 * NF + 40
    if kind in ("fp64", "fp32", "viscosity"):
        w = 4 if kind == "fp32" else 8
        per = 4 * w + 9 * w + r * (4 * w + 4)  # state, residual, metrics, face data, gather map
        if kind == "viscosity":  # the gradient and eps written and read; sensor, gradient and divergence products
            per += 2 * 4 * 8
            flops += 2 * Np + 6 * NF + 6 * Np + 60
        return {"bytes": 5 * dofs * per, "flops": 5 * dofs * flops}
    if kind == "compact":
        return {"bytes": 5 * dofs * (32 + (200 + 20) / Np), "flops": 5 * dofs * flops}
    per = 24 + 52 / Np  # the compensated pair and the residual, compact geometry and connectivity
    if kind == "learned":
        per += 8
        flops += 2 * Np + (2 * (32 * Np + 32 * 33) / Np if case["sensor"] != "pp" else 0)
    return {"bytes": dofs * (10 * per + 16), "flops": 10 * dofs * flops}


# ---- the same results in 64 bits ----------------------------------------------------------------------------
class _Stage64:
    """The strong-form Lax-Friedrichs right-hand side (with the BR1 viscosity where a sensor is given) and its
    LSERK4 stages in FP64 torch, on the arrays that the problem was given."""

    def __init__(self, state):
        p, case = state["p"], state["case"]
        v = _Views(p.runner)
        dt = case.get("dtype", "float32" if case["kind"] == "fp32" else "float64")
        K, Np, NF = p.K, p.el.Np, 4 * p.el.Nfp
        self.K, self.Np = K, Np
        self.geo = [v.flat(g, dt).double().view(K, Np) for g in GEO]
        self.face = [v.flat(f, dt).double().view(K, NF) for f in FACE]
        up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).cuda()  # noqa: E731
        self.D = [up(getattr(p.el, m)).double() for m in ("Dr", "Ds", "Dt")]
        self.LIFT, self.Vinv = up(p.el.LIFT).double(), up(p.el.Vinv).double()
        self.fmask = up(np.asarray(p.el.Fmask).reshape(-1)).long()
        self.vmapP = up(p.vmapP)
        self.conservative = case.get("conservative", 0)
        self.N, self.sensor = case["N"], case.get("sensor")
        if self.sensor:
            self.av = p.av
            top = [i + j + k == self.N for i in range(self.N + 1) for j in range(self.N + 1 - i)
                   for k in range(self.N + 1 - i - j)]
            self.top = torch.tensor(top, device="cuda")
            self.h_over_n = (2.0 / self.face[3].max(dim=1).values) / self.N

    def ddx(self, f):
        d = [f @ M.T for M in self.D]
        return [self.geo[x] * d[0] + self.geo[3 + x] * d[1] + self.geo[6 + x] * d[2] for x in range(3)]

    def traces(self, f):
        return f[:, self.fmask], f.reshape(-1)[self.vmapP].view(self.K, -1)

    def epsilon(self, u):
        uh = u @ self.Vinv.T
        tot = (uh ** 2).sum(dim=1)
        S = torch.log10((uh[:, self.top] ** 2).sum(dim=1) / tot)
        kappa = self.av["kappa"]
        s0 = -(self.av["c0"] + 4.0 * math.log10(self.N))
        sig = 0.5 * (1.0 + torch.sin(math.pi * (S - s0) / (2.0 * kappa)))
        sig = torch.where(S > s0 + kappa, torch.ones_like(sig), sig)
        sig = torch.where(S >= s0 - kappa, sig, torch.zeros_like(sig))
        # (the cases' networks stay inside the low-confidence band, where this activation stands)
        return (self.av["eps0"] * sig * self.h_over_n).unsqueeze(1)

    def rhs(self, u):
        nx, ny, nz, fs = self.face
        uM, uP = self.traces(u)
        ns = nx + ny + nz
        fM, fP = 0.5 * uM * uM * ns, 0.5 * uP * uP * ns
        lam = torch.maximum((uM * ns).abs(), (uP * ns).abs())
        flux = fs * (fM - (0.5 * (fM + fP) + 0.5 * lam * (uM - uP)))
        g = sum(self.ddx(0.5 * u * u if self.conservative else u))
        out = -g if self.conservative else -u * g
        if self.sensor:
            eps = self.epsilon(u)
            jump = 0.5 * fs * (uP - uM)
            eq = [eps * (q + (n * jump) @ self.LIFT.T) for q, n in zip(self.ddx(u), (nx, ny, nz))]
            for d, n in enumerate((nx, ny, nz)):
                M, P = self.traces(eq[d])
                flux = flux + 0.5 * fs * n * (P - M)
                out = out + self.ddx(eq[d])[d]
        return out + flux @ self.LIFT.T

    def steps(self, u, dt, stages):
        res = torch.zeros_like(u)
        for s in range(stages):
            res = RK4A[s % 5] * res + dt * self.rhs(u)
            u = u + RK4B[s % 5] * res
        return u, res


def exact(case, seed):
    state = prepare(case, seed)
    if case["kind"] == "train":
        return _exact_train(state)
    p = state["p"]
    S = _Stage64(state)
    u = torch.from_numpy(p.get("u")).cuda().double().view(S.K, S.Np)
    if case["kind"] == "derivative":
        g = S.ddx(u)
        if not case["reference"]:
            return [x.reshape(-1) for x in g]
        rhs = -u * sum(g)
        res = p.dt * rhs
        return {"rhs": rhs.reshape(-1), "u": (u + RK4B[1] * res).reshape(-1), "resu": res.reshape(-1)}
    u, res = S.steps(u, p.dt, 10 if state["mixed"] else 5)
    out = {"u": u.reshape(-1)}
    if _residual(case):
        out["resu"] = res.reshape(-1)
    return out


def _exact_train(state):
    net, X, y = state["net"], state["X"].double(), state["y"].double()
    p = net.p.double().requires_grad_(True)
    nin, h = net.nin, 32
    W1, b1, W2, b2, w3, b3 = torch.split(p, [h * nin, h, h * h, h, h, 1])
    z = torch.tanh(torch.tanh(X @ W1.view(h, nin).T + b1) @ W2.view(h, h).T + b2) @ w3 + b3
    loss = ((torch.sigmoid(z) - y) ** 2).mean()
    loss.backward()
    g, t, lr = p.grad, net.t + 1, 3e-3
    m = 0.9 * net.m.double() + 0.1 * g
    v = 0.999 * net.v.double() + 0.001 * g * g
    new = p.detach() - lr * (m / (1 - 0.9 ** t)) / ((v / (1 - 0.999 ** t)).sqrt() + 1e-8)
    return {"loss": loss.detach(), "grad": g, "params": new, "m": m, "v": v}
