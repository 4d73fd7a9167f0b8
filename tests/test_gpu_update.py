"""Elementwise updates (lserkUpdate, updateSolution) over runs of values: bits for any values per element and partition
sizes, and a cost per value that does not depend on the values per element (a value costs the same work in both: bound
1.4; a grid over tiles of 64 elements cost 2.0 at 4 values per element against 35, FP32)."""
import numpy as np
import pytest

from dgkernel_b200.runner import Config, Float32, Float64, Runner, Scalar, Temp

pytestmark = pytest.mark.gpu
NAMES = ("u", "resu", "rhs")


def _runner(K, npe, dtype, op, scalars, stream=None):
    r = Runner(Config(K=K), stream=stream)
    code = Float64 if dtype == np.float64 else Float32
    r.DefineBindings(*[Temp(n).Type(code).Size(sum(K) * npe) for n in NAMES], *[Scalar(s).Type(Float64) for s in scalars])
    r.AllocateDevice()
    r.ConfigureKernel("up", *[r.Param(n) for n in NAMES], *[r.Param(s) for s in scalars])
    r.BuildKernel(op, "up")
    return r


@pytest.mark.parametrize("dtype", [np.float64, np.float32])
@pytest.mark.parametrize("op,scalars", [("lserkUpdate", ("a", "b", "dt")), ("updateSolution(rhsu=rhs)", ("rka", "rkb"))])
@pytest.mark.parametrize("K,npe", [([1], 1), ([1023, 1, 1025], 1), ([256, 255, 257], 4), ([1024], 2), ([103, 1, 7], 10),
                                   ([300, 5], 35), ([9, 10], 120), ([1], 3000)])
def test_bits(K, npe, op, scalars, dtype):
    n = sum(K) * npe
    rng = np.random.default_rng(2)
    x = {k: (rng.integers(-64, 64, n) / 8).astype(dtype) for k in NAMES}  # exact under the scalars below
    r = _runner(K, npe, dtype, op, scalars)
    for k in NAMES:
        r.CopyToDevice(k, x[k])
    if len(scalars) == 3:
        r.ExecuteKernel("up", 0.5, 2.0, 0.25)
        res = 0.5 * x["resu"] + 0.25 * x["rhs"]
        u = x["u"] + 2.0 * res
    else:
        r.ExecuteKernel("up", 0.5, 0.25)
        res = 0.5 * x["resu"] + 0.25 * x["rhs"]
        u = x["u"] + res
    for k, want in (("u", u), ("resu", res), ("rhs", x["rhs"])):
        got = np.zeros(n, dtype)
        r.CopyFromDevice(k, got)
        assert np.array_equal(got, want), k
    r.Free()


def _time(npe):
    import torch
    st = torch.cuda.Stream()
    n = 4 * (4000000 // npe)
    r = _runner([n // 4] * 4, npe, np.float32, "lserkUpdate", ("a", "b", "dt"), st.cuda_stream)
    for k in NAMES:
        r.CopyToDevice(k, np.zeros(n * npe, np.float32))
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    best = float("inf")
    for _ in range(5):
        with torch.cuda.stream(st):
            e0.record(st)
            for _ in range(10):
                r.ExecuteKernel("up", 0.5, 2.0, 0.25)
            e1.record(st)
        e1.synchronize()
        best = min(best, e0.elapsed_time(e1) / 10)
    r.Free()
    return best / (n * npe)


def test_cost_per_value():
    assert _time(4) < 1.4 * _time(35)
