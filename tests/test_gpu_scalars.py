"""Scalars of ExecuteKernel by place: a scalar that a kernel lists twice takes its last place that was given a value, and
one that was given none is refused."""
import numpy as np
import pytest

import dgkernel_b200 as d
from dgkernel_b200.runner import Config, Float64, Runner, Scalar, Temp

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("listed,given,want", [
    (("a", "b", "dt"), (0.5, 2.0, 0.25), (0.5, 2.0, 0.25)),
    (("a", "b", "dt", "a"), (0.5, 2.0, 0.25), (0.5, 2.0, 0.25)),
    (("a", "b", "dt", "a"), (0.5, 2.0, 0.25, -0.5), (-0.5, 2.0, 0.25)),
    (("b", "a", "dt", "b", "dt"), (2.0, 0.5, 0.25, 3.0), (0.5, 3.0, 0.25)),
    (("a", "b", "dt"), (0.5, 2.0), None),
    (("a", "a", "b", "dt"), (0.5, 0.5), None),
])
def test_places(listed, given, want):
    r = Runner(Config(K=[5]))
    names = ("u", "resu", "rhs")
    r.DefineBindings(*[Temp(n).Type(Float64).Size(20) for n in names], *[Scalar(s).Type(Float64) for s in ("a", "b", "dt")])
    r.AllocateDevice()
    x = {n: np.arange(20.0) + i for i, n in enumerate(names)}
    for n in names:
        r.CopyToDevice(n, x[n])
    r.ConfigureKernel("up", *[r.Param(n) for n in names], *[r.Param(s) for s in listed])
    r.BuildKernel("lserkUpdate", "up")
    if want is None:
        with pytest.raises(d.DGKError, match="not provided"):
            r.ExecuteKernel("up", *given)
    else:
        r.ExecuteKernel("up", *given)
        got = np.zeros(20)
        r.CopyFromDevice("u", got)
        a, b, dt = want
        assert np.array_equal(got, x["u"] + b * (a * x["resu"] + dt * x["rhs"]))
    r.Free()
