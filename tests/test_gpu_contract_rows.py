"""The FP32 contraction of few rows does not take longer than that of more rows
(its own kernel is chosen only where it is the faster one)."""
import pytest
import torch

from pointint_gb300 import core
from pointint_gb300.kgrid import standard_kgrid

pytestmark = pytest.mark.gpu


def contraction_us(kg, n):
    """Microseconds a call, the least of ten groups of ten calls back to back."""
    J = torch.randn(n, kg.num_nodes, dtype=torch.complex64, device="cuda")
    out = torch.empty(n, n, dtype=torch.float64, device="cuda")
    times = []
    for _ in range(10):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        for _ in range(10):
            core.contract(kg, J, "fp32", out=out)
        b.record()
        torch.cuda.synchronize()
        times.append(a.elapsed_time(b) * 100)
    return min(times)


@pytest.mark.parametrize("order,radii", [(9, 64), (29, 32), (29, 64), (131, 128)])  # 2,432 to 743,680 nodes
def test_time_does_not_fall_with_the_rows(cuda, order, radii):
    kg = standard_kgrid(order, radii)
    t = {n: contraction_us(kg, n) for n in (2, 16, 24, 32, 36, 40, 48, 56, 57, 60, 64, 65)}
    print(f"\n{kg.num_nodes} nodes: " + ", ".join(f"{n}: {v:.1f}" for n, v in t.items()))
    slack = 2.0 + 0.05 * t[65]  # us: what two runs differ by
    assert all(v <= t[65] + slack for v in t.values())
