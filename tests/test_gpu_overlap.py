"""FP32-value products on a GPU that other work keeps busy: the main kernel
is launched while the rounding of x to FP32 may still run, and may gather
only after it.  Every product equals, bit for bit, the same plan's product
made alone."""
from __future__ import annotations

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", [0, 4, 16, 32])
def test_f32_products_beside_other_work(variant):
    import torch

    from int_spmv_b200 import device as D
    from int_spmv_b200 import formats as F
    from int_spmv_b200 import matrices as M
    row, col, val = M.powerlaw(400_000, seed=variant)
    plan = D.Plan(F.CSR(row, col, val), None, kernel="wide", variant=variant, val="f32")
    n = len(row) - 1
    xs = [torch.rand(n, dtype=torch.float64, device="cuda") for _ in range(3)]
    for x in xs:  # work areas, a texture over them
        plan.spmv(x)
    torch.cuda.synchronize()
    alone = []
    for x in xs:
        rounded = x.float().double()  # the rounding of x leaves this one as it is
        plan.spmv(rounded)
        torch.cuda.synchronize()
        alone.append(plan.spmv(rounded).clone())  # x rounded before: the same values twice
        torch.cuda.synchronize()
    a = torch.randn(2048, 2048, device="cuda")
    side, y = torch.cuda.Stream(), torch.empty_like(xs[0])
    wrong = 0
    for i in range(60):
        with torch.cuda.stream(side):
            for _ in range(3):
                a @ a
        y.fill_(0.0)
        plan.spmv(xs[i % 3], y)
        torch.cuda.current_stream().synchronize()
        wrong += not torch.equal(y, alone[i % 3])
    assert wrong == 0
