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


CHAINS = [("CSR", {}), ("CSR", dict(kernel="wide", variant=26)), ("CSR", dict(kernel="wide", variant=4)),
          ("CSR", dict(kernel="wide", variant=11)), ("CSR", dict(kernel="wide", variant=16)),
          ("CSR", dict(val="f32")), ("CSR", dict(val="f32", kernel="wide", variant=16)),
          ("CSR", dict(val="f32lo")), ("CSR", dict(col="d16", kernel="wide", variant=9)), ("STENCIL", dict(col="d16")),
          ("STENCIL", dict(val="f32", col="d16")), ("STENCIL", {}), ("K1", {}), ("K1P", {}), ("CSR", dict(kernel="ldg"))]


@pytest.mark.parametrize("fmt,kw", CHAINS)
@pytest.mark.parametrize("spmm", [0, 8, 11, 32])
def test_products_in_a_chain(fmt, kw, spmm):
    """Products whose x is the y of the product before (through one more
    kernel, or directly), enqueued without a wait on a GPU that other work
    keeps busy: each may start while the one before it finishes, and gives the
    bits it gives alone."""
    import numpy as np
    import torch

    from int_spmv_b200 import device as D
    from int_spmv_b200 import formats as F
    from int_spmv_b200 import matrices as M
    if spmm and (fmt.startswith("K1") or "d16" in kw.values() or kw.get("val") == "f32lo"):
        pytest.skip("SpMM needs a slot-stream plan with u32 columns")
    row, col, val = M.stencil27(30) if fmt == "STENCIL" else M.random_csr(40_000, 5, rl_max=24, empty_frac=0.05)
    if fmt != "STENCIL":
        col = col.copy()
    csr = F.CSR(row, col, val / np.abs(val).max() * 0.1)
    f = F.getFormatDataK1(8, csr, np.zeros(csr.n))[1] if fmt.startswith("K1") else None
    plan = D.Plan(csr, f, **({"reorder": fmt == "K1P"} if f is not None else {}), **kw)
    shape = (csr.n, spmm) if spmm else (csr.n,)
    g = torch.Generator(device="cuda").manual_seed(1)
    x0 = torch.rand(shape, dtype=torch.float64, device="cuda", generator=g)

    def chain(wait):
        a, b = x0.clone(), torch.ones_like(x0)
        for i in range(24):
            if spmm:
                plan.spmm(a, b)
            elif i % 8 == 7:
                plan.spmv_graph(a, b)
            else:
                plan.spmv(a, b, beta=i % 3 == 1)
            if wait:
                torch.cuda.synchronize()
            if i % 2:
                b.mul_(0.5).add_(a, alpha=0.25)
            a, b = b, a
            if wait:
                torch.cuda.synchronize()
        return a

    alone = chain(True).clone()
    torch.cuda.synchronize()
    m = torch.randn(2048, 2048, device="cuda")
    side = torch.cuda.Stream()
    for _ in range(6):
        with torch.cuda.stream(side):
            for _ in range(8):
                m @ m
        got = chain(False)
        torch.cuda.synchronize()
        assert torch.equal(got, alone)


@pytest.mark.parametrize("kw", [dict(kernel="wide", variant=26), dict(kernel="wide", variant=11), dict(val="f32"),
                                dict(col="d16"), dict(fmt="K1P"), dict(fmt="K1")])
@pytest.mark.parametrize("before", ["kernel", "memset", "copy", "join", "nothing"])
def test_products_in_a_captured_graph(kw, before):
    """Products captured into a caller's CUDA graph after a kernel, a memset, a
    copy, the join of another stream, or as its first node: replays give what
    the same calls give outside."""
    import numpy as np
    import torch

    from int_spmv_b200 import device as D
    from int_spmv_b200 import formats as F
    from int_spmv_b200 import matrices as M
    kw = dict(kw)
    fmt = kw.pop("fmt", "CSR")
    row, col, val = M.stencil27(24)
    csr = F.CSR(row, col, val / 60.0)
    f = F.getFormatDataK1(8, csr, np.zeros(csr.n))[1] if fmt != "CSR" else None
    plan = D.Plan(csr, f, **({"reorder": fmt == "K1P"} if f is not None else {}), **kw)
    src = torch.rand(csr.n, dtype=torch.float64, device="cuda")
    x, y, z = src.clone(), torch.zeros_like(src), torch.zeros_like(src)
    side = torch.cuda.Stream()

    def step():
        if before == "kernel":
            x.mul_(0.5).add_(1.0)
        elif before == "memset":
            y.zero_()
        elif before == "copy":
            x.copy_(src)
        elif before == "join":
            s = torch.cuda.current_stream()
            side.wait_stream(s)
            with torch.cuda.stream(side):
                x.mul_(0.75)
            s.wait_stream(side)
        plan.spmv(x, y)
        plan.spmv(y, z, beta=1)
        x.add_(z, alpha=0.125)

    def start():
        x.copy_(src), y.zero_(), z.zero_()

    start()
    torch.cuda.synchronize()
    for _ in range(5):
        step()
        torch.cuda.synchronize()
    want = [t.clone() for t in (x, y, z)]
    start()
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        step()
    start()
    torch.cuda.synchronize()
    for _ in range(5):
        graph.replay()
    torch.cuda.synchronize()
    for got, ref in zip((x, y, z), want):
        assert torch.equal(got, ref)


@pytest.mark.parametrize("kw", [dict(variant=16), dict(variant=16, val="f32"), dict(variant=16, col="d16"),
                                dict(variant=16, val="f32", col="d16")])
def test_texture_products_back_to_back(kw):
    """Texture gathers, product after product with no other kernel between
    and x, y swapped: every third product reads anew a buffer whose lines an
    SM may still hold from the product before last."""
    import numpy as np
    import torch

    from int_spmv_b200 import device as D
    from int_spmv_b200 import formats as F
    from int_spmv_b200 import matrices as M
    row, col, val = M.random_csr(40_000, 5, rl_max=24, empty_frac=0.05)
    csr = F.CSR(row, col, val / np.abs(val).max() * 0.1)
    plan = D.Plan(csr, None, kernel="wide", **kw)
    x0 = torch.rand(csr.n, dtype=torch.float64, device="cuda")

    def chain(wait):
        a, b = x0.clone(), torch.ones_like(x0)
        for _ in range(12):
            plan.spmv(a, b)
            if wait:
                torch.cuda.synchronize()
            a, b = b, a
        return a

    alone = chain(True).clone()
    torch.cuda.synchronize()
    assert "tex" in plan.kernel_name(), plan.kernel_name()
    m = torch.randn(2048, 2048, device="cuda")
    side = torch.cuda.Stream()
    for i in range(12):
        if i % 2:
            with torch.cuda.stream(side):
                for _ in range(8):
                    m @ m
        got = chain(False)
        torch.cuda.synchronize()
        assert torch.equal(got, alone)


@pytest.mark.parametrize("kind", ["slices", "slices_f32", "K1", "K1P", "rows", "axc_rows", "noc4_ldg", "auto", "f32lo"])
def test_product_on_another_stream_right_after_the_plan(kind):
    """A host-built plan's arrays are on the device when the builder returns:
    a product at once, on a stream the default stream does not order, on blocks
    that held another matrix's arrays."""
    import numpy as np
    import torch

    from int_spmv_b200 import device as D
    from int_spmv_b200 import formats as F
    from int_spmv_b200 import matrices as M
    from oracle import Oracle
    from paritylib import assert_parity
    orc = Oracle()
    mats = []
    for seed in (1, 2):  # two matrices of the same size
        row, col, val = M.stencil27(30 if kind.startswith("slices") else 12)
        val = np.random.default_rng(seed).standard_normal(len(val))
        x = M.uniform_x(len(row) - 1, seed)
        csr = F.CSR(row, col, val)
        z = np.zeros(csr.n)
        f = F.getFormatDataK1(8, csr, z)[1] if kind.startswith("K1") else \
            F.getFormatDataAXC(0, csr, z)[1] if kind == "axc_rows" else \
            F.getFormatDataAXT(0, 128, 8, 4, "NOC", csr, z)[1] if kind == "noc4_ldg" else None
        mats.append((csr, f, torch.from_numpy(x).cuda(), orc.cf_csr(row, col, val, x), orc.abs_csr(row, col, val, x)))
    kw = {"slices": dict(col="d16"), "slices_f32": dict(col="d16", val="f32"), "K1": dict(reorder=False),
          "rows": dict(kernel="rows"), "axc_rows": dict(kernel="rows"), "noc4_ldg": dict(kernel="ldg"),
          "f32lo": dict(val="f32lo")}.get(kind, {})
    side = torch.cuda.Stream()
    y = torch.empty_like(mats[0][2])
    torch.cuda.synchronize()
    for i in range(20):
        csr, f, x, ref, absax = mats[i % 2]
        plan = D.Plan(csr, f, **kw)
        plan.spmv(x, y, stream=side)
        side.synchronize()
        assert_parity(y.cpu().numpy(), ref, absax, 1e-6 if "f32" in kind else 1e-12, what=f"{kind} {i}")
        assert ("rows32" in plan.kernel_name()) == kind.startswith("slices")
        del plan
