"""splitState / joinState over partitions of very different sizes: the pair is u rounded to FP32 and the rounded rest,
and the join is their FP64 sum, bit for bit; and a large partition beside many small ones costs no more than a few times
the values in one partition (its work list has no empty blocks: measured about 1, bound 8; a grid of runs x partitions
took 35)."""
import numpy as np
import pytest

from dgkernel_b200.burgers import BurgersEnsemble

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("N,sizes", [(1, [7, 3, 20]), (2, [3] * 40), (3, [3, 12, 4]), (5, [9])])
def test_split_and_join_bits(N, sizes):
    E = BurgersEnsemble(N, sizes)
    rng = np.random.default_rng(3)
    u = rng.normal(size=E.K * E.el.Np)
    u[:4] = 0.0, -0.0, 1e-30, 1.0 + 2.0 ** -40
    E.set("u", u)
    hi = u.astype(np.float32)
    lo = (u - hi.astype(np.float64)).astype(np.float32)
    assert np.array_equal(E.get("uhi"), hi) and np.array_equal(E.get("ulo"), lo)
    E.set("u", u)
    E.runner.ExecuteKernel("joinState")
    out = np.zeros_like(u)
    E.runner.CopyFromDevice("u", out)
    assert np.array_equal(out, hi.astype(np.float64) + lo.astype(np.float64))
    E.free()


def _time(sizes, op):
    import torch
    st = torch.cuda.Stream()
    E = BurgersEnsemble(2, sizes, stream=st.cuda_stream)
    e0, e1 = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
    best = float("inf")
    for _ in range(5):
        with torch.cuda.stream(st):
            e0.record(st)
            for _ in range(10):
                E.runner.ExecuteKernel(op)
            e1.record(st)
        e1.synchronize()
        best = min(best, e0.elapsed_time(e1) / 10)
    n = E.dofs
    E.free()
    return best / n


@pytest.mark.parametrize("op", ["splitState", "joinState"])
def test_uneven_partitions_cost_their_values(op):
    assert _time([40] + [3] * 1000, op) < 8 * _time([45], op)
