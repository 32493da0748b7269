"""The work that users of int_spmv_b200 have it do, as cases for timing.

A case is a dict of plain values.  `op` is the call:

  spmv     Plan.spmv: y = A x (beta = 0) or y += A x (beta = 1), the inner
           step of a Krylov solver or a time stepper; `fmt` is the format the
           plan was built from, `val` and `col` the plan's value and column form
  graph    Plan.spmv_graph on a block-diagonal plan of many uneven matrices
  spmm     Plan.spmm: Y = A X for k right-hand sides (block solvers)
  rebuild  Plan.from_device_csr and one product: a matrix assembled anew on
           the GPU in every step of a nonlinear solve
  convert  DeviceAXT and one product with it: the reference's conversion for
           a new x (its AXT bakes x in), then its kernel

`matrix` is the generator: the matrix families of the repository's benchmark
(2D Poisson, 27-point stencil, power-law rows with 70% banded and 30%
uniform columns, FEM-like banded blocks), made here on the GPU from the seed.
"""
import math

import numpy as np
import torch

from int_spmv_b200 import batch as B
from int_spmv_b200 import device as D
from int_spmv_b200 import formats as F

DEV = "cuda"
PL_MU, PL_SIGMA, PL_MAX, PL_BAND = 2.2, 1.0, 5000, 1000
FEM_LO, FEM_HI = 7, 81


def _case(name, op, matrix, n, fmt="dev", val="f64", col="u32", beta=0, k=0, count=0):
    c = dict(op=op, matrix=matrix, n=n, fmt=fmt, val=val, col=col, beta=beta, k=k, count=count)
    return dict(c, name=name) if name else c


def listed():
    return [
        # a coarse multigrid level or a small subdomain: launch and latency bound
        _case("spmv_poisson_4k", "spmv", "poisson", 64 * 64, fmt="com128"),
        # the 512 x 512 Poisson problem on the uncompacted AXT of tile height 1
        _case("spmv_poisson_512_noc1", "spmv", "poisson", 512 * 512, fmt="noc1"),
        # the headline: a graph-like matrix of 4M rows, FP64, compacted AXT stream
        _case("spmv_powerlaw_4m", "spmv", "powerlaw", 4_000_000),
        # a tall-tile format on an odd row count, accumulating into y
        _case("spmv_powerlaw_1m_noc8_acc", "spmv", "powerlaw", 1_000_003, fmt="noc8", beta=1),
        # K1 with integrated reordering, the reference's sorted-row format
        _case("spmv_powerlaw_1m_k1p", "spmv", "powerlaw", 1_000_000, fmt="k1p"),
        # the large regular problem of an implicit PDE solver, FP64
        _case("spmv_stencil_160", "spmv", "stencil", 160 ** 3),
        # the reduced-byte form of a mixed-precision solver, odd grid
        _case("spmv_stencil_101_f32_d16", "spmv", "stencil", 101 ** 3, fmt="com128", val="f32", col="d16"),
        # block solvers: a narrow and a wide block of right-hand sides
        _case("spmm_powerlaw_1m_k8", "spmm", "powerlaw", 1_000_000, k=8),
        _case("spmm_powerlaw_1m_k32", "spmm", "powerlaw", 1_000_000, k=32),
        # many uneven FEM blocks in one graph launch
        _case("graph_fem_32", "graph", "fem", 50_000, fmt="com128", count=32),
        # a matrix reassembled on the GPU: plan and product
        _case("rebuild_powerlaw_1m", "rebuild", "powerlaw", 1_000_000),
        # the reference's conversion and its compacted kernel for a new x
        _case("convert_powerlaw_1m_com128", "convert", "powerlaw", 1_000_000, fmt="com128"),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One case of the ranges above: every format, value and column form the
    plans take in use, sizes over their logarithm."""
    op = rng.choices(["spmv", "spmm", "graph", "rebuild", "convert"], [12, 4, 1, 2, 2])[0]
    matrix = rng.choices(["powerlaw", "stencil", "poisson"], [5, 3, 2])[0]
    if op == "graph":
        return _case(None, op, "fem", _size(rng, 2_000, 50_000), fmt=rng.choice(["com128", "csr"]),
                     val=rng.choice(["f64", "f32"]), count=rng.randint(4, 32))
    fmt, val, col, beta, k = "dev", "f64", "u32", 0, 0
    if op == "spmv":
        fmt = rng.choices(["dev", "csr", "com128", "com512", "noc1", "noc4", "noc8", "noc16", "axc", "k1", "k1p"],
                          [6, 2, 2, 1, 1, 1, 1, 1, 1, 1, 1])[0]
        val = rng.choice(["f64", "f64", "f32"])
        beta = rng.choice([0, 0, 1])
        if fmt in ("csr", "com128", "com512") and rng.random() < 0.4:
            col = "d16"
        if fmt in ("csr", "com128", "com512") and rng.random() < 0.15:
            val = "f32lo"
    elif op == "spmm":
        val, k = rng.choice(["f64", "f64", "f32"]), rng.choice([8, 16, 32, 24, 11, 13, 10])
    elif op == "rebuild":
        val = rng.choice(["f64", "f32"])
    else:
        fmt = rng.choice(["com128", "com512", "noc1", "noc4", "noc8"])
    large = op == "spmv" and fmt == "dev"  # the other formats are built on the host: up to about 1M rows
    if matrix == "poisson":
        n = _size(rng, 48, 1000) ** 2
    elif matrix == "stencil":
        n = _size(rng, 16, 160 if large else 80) ** 3
    else:
        n = _size(rng, 4_000, 4_000_000 if large else 1_000_000)
    return _case(None, op, matrix, n, fmt, val, col, beta, k)


# --- matrices on the GPU -------------------------------------------------

def _stencil(n, dims, values):
    """CSR of a grid stencil: `values(offset, rows)` for every neighbour."""
    m = round(n ** (1.0 / dims))
    idx = torch.arange(n, device=DEV)
    xyz = [(idx // m ** d) % m for d in range(dims)]
    if dims == 2:
        offs = [(0, -1), (-1, 0), (0, 0), (1, 0), (0, 1)]
    else:
        offs = [(x, y, z) for z in (-1, 0, 1) for y in (-1, 0, 1) for x in (-1, 0, 1)]
    valid = torch.ones((len(offs), n), dtype=torch.bool, device=DEV)
    for k, o in enumerate(offs):
        for d, s in enumerate(o):
            if s:
                valid[k] &= (xyz[d] + s >= 0) & (xyz[d] + s < m)
    rl = valid.sum(0)
    row = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    row[1:] = rl.cumsum(0)
    nnz = int(row[-1])
    col = torch.empty(nnz, dtype=torch.int32, device=DEV)
    val = torch.empty(nnz, dtype=torch.float64, device=DEV)
    at = row[:-1].clone()
    for k, o in enumerate(offs):
        r = idx[valid[k]]
        q = at[r]
        col[q] = (r + sum(s * m ** d for d, s in enumerate(o))).to(torch.int32)
        val[q] = values(o, r.numel())
        at += valid[k]
    return row, col, val


def _rows_from_keys(n, key):
    key = torch.unique(key)  # sorted: rows ascending, columns ascending inside a row, duplicates once
    r = key // n
    col = (key - r * n).to(torch.int32)
    row = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    row[1:] = torch.bincount(r, minlength=n).cumsum(0)
    return row, col


def _powerlaw(n, g):
    rl = torch.exp(PL_MU + PL_SIGMA * torch.randn(n, device=DEV, generator=g, dtype=torch.float64))
    rl = rl.round().clamp(1, min(PL_MAX, n)).to(torch.int64)
    nb = (0.7 * rl).round().to(torch.int64)
    r = torch.repeat_interleave(torch.arange(n, device=DEV), nb)
    lo = (r - PL_BAND).clamp(min=0)
    w = (r + PL_BAND).clamp(max=n - 1) - lo + 1
    near = r * n + lo + (torch.rand(r.numel(), device=DEV, generator=g, dtype=torch.float64) * w).to(torch.int64)
    r = torch.repeat_interleave(torch.arange(n, device=DEV), rl - nb)
    far = r * n + torch.randint(0, n, (r.numel(),), device=DEV, generator=g)
    row, col = _rows_from_keys(n, torch.cat([near, far]))
    return row, col, torch.randn(col.numel(), device=DEV, generator=g, dtype=torch.float64)


def _fem_sizes(count, hi):
    """The blocks' row counts: log-uniform in [1000, hi], the same for every seed."""
    u = np.random.default_rng(4).uniform(0.0, 1.0, count)
    return np.exp(math.log(1e3) + u * (math.log(max(hi, 1001)) - math.log(1e3))).astype(np.int64)


def _fem(count, hi, g):
    """`count` banded blocks as one block-diagonal CSR and the blocks' first rows."""
    ns = torch.from_numpy(_fem_sizes(count, hi)).to(DEV)
    off = torch.zeros(count + 1, dtype=torch.int64, device=DEV)
    off[1:] = ns.cumsum(0)
    n = int(off[-1])
    first = torch.repeat_interleave(off[:-1], ns)
    last = torch.repeat_interleave(off[1:], ns) - 1
    idx = torch.arange(n, device=DEV)
    rl = torch.randint(FEM_LO, FEM_HI + 1, (n,), device=DEV, generator=g)
    r = torch.repeat_interleave(idx, rl - 1)
    lo = torch.maximum(r - 3 * rl[r], first[r])
    w = torch.minimum(r + 3 * rl[r], last[r]) - lo + 1
    c = lo + (torch.rand(r.numel(), device=DEV, generator=g, dtype=torch.float64) * w).to(torch.int64)
    row, col = _rows_from_keys(n, torch.cat([idx * n + idx, r * n + c]))
    val = torch.randn(col.numel(), device=DEV, generator=g, dtype=torch.float64)
    rr = torch.repeat_interleave(idx, row[1:] - row[:-1])
    diag = rr == col
    off_sum = torch.segment_reduce(val.masked_fill(diag, 0.0), "sum", lengths=row[1:] - row[:-1])
    val[diag] = off_sum.abs() + 1.0
    return row, col, val, off


def _inputs(case, seed):
    """(row int64, col int32, val f64, block offsets or None, x or X, y) on
    the GPU, from the seed alone."""
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    n, off = case["n"], None
    if case["matrix"] == "poisson":
        row, col, val = _stencil(n, 2, lambda o, c: 4.0 if o == (0, 0) else -1.0)
    elif case["matrix"] == "stencil":
        row, col, val = _stencil(n, 3, lambda o, c: 26.0 if o == (0, 0, 0) else
                                 -1.1 + 0.2 * torch.rand(c, device=DEV, generator=g, dtype=torch.float64))
    elif case["matrix"] == "powerlaw":
        row, col, val = _powerlaw(n, g)
    else:
        row, col, val, off = _fem(case["count"], n, g)
    n = row.numel() - 1
    shape = (n, case["k"]) if case["k"] else (n,)
    x = torch.rand(shape, device=DEV, generator=g, dtype=torch.float64) * 2 - 1
    y = torch.rand(shape, device=DEV, generator=g, dtype=torch.float64) if case["beta"] else torch.empty_like(x)
    return row, col, val, off, x, y


def _host_plan(case, row, col, val, off, x):
    """The plan of a host-built format, as a program that reads its matrix
    from a file makes it."""
    row, col, val, x = (t.cpu().numpy() for t in (row, col, val, x))
    if off is not None:  # the batched path: separate matrices joined by the library
        o = off.cpu().numpy()
        mats = [((row[a:b + 1] - row[a]).astype(np.uint32), (col[row[a]:row[b]] - a).astype(np.uint32),
                 val[row[a]:row[b]]) for a, b in zip(o[:-1], o[1:])]
        csr = B.blockdiag(mats)[0]
    else:
        csr = F.CSR(row.astype(np.uint32), col.view(np.uint32), val)
    fmt, kw = case["fmt"], {}
    if fmt == "csr":
        f = None
    elif fmt == "axc":
        f = F.getFormatDataAXC(0, csr, x)[1]
    elif fmt in ("k1", "k1p"):
        f, kw = F.getFormatDataK1(512, csr, x)[1], dict(reorder=fmt == "k1p")
    else:
        mode, p = fmt[:3].upper(), int(fmt[3:])
        f = F.getFormatDataAXT(0, p if mode == "COM" else 128, 8, p if mode == "NOC" else 1, mode, csr, x)[1]
    return D.Plan(csr, f, val=case["val"], col=case["col"], **kw)


def prepare(case, seed):
    row, col, val, off, x, y = _inputs(case, seed)
    s = dict(case=case, x=x, y=y)
    if case["op"] in ("rebuild", "convert"):
        s.update(row=row.to(torch.int32), col=col, val=val)
    elif case["fmt"] == "dev":
        s["plan"] = D.Plan.from_device_csr(row.to(torch.int32), col, val, val_kind=case["val"])
    else:
        s["plan"] = _host_plan(case, row, col, val, off, x)
    return s


def run(s):
    case, x, y = s["case"], s["x"], s["y"]
    op = case["op"]
    if op == "spmv":
        return s["plan"].spmv(x, y, case["beta"])
    if op == "graph":
        return s["plan"].spmv_graph(x, y)
    if op == "spmm":
        return s["plan"].spmm(x, y)
    if op == "rebuild":
        return D.Plan.from_device_csr(s["row"], s["col"], s["val"], val_kind=case["val"]).spmv(x, y)
    mode, p = case["fmt"][:3].upper(), int(case["fmt"][3:])
    axt = D.DeviceAXT(s["row"], s["col"], s["val"], x, bs=p if mode == "COM" else 128,
                      th=p if mode == "NOC" else 1, mode=mode)
    return axt.spmv(y.zero_())  # the reference's kernels accumulate


def exact(case, seed):
    row, col, val, _, x, y = _inputs(case, seed)
    rl = row[1:] - row[:-1]

    def product(v):
        return torch.segment_reduce(val * v[col], "sum", lengths=rl, initial=0.0)

    if case["k"]:
        for j in range(case["k"]):
            y[:, j] = product(x[:, j].contiguous())
        return y
    return product(x) + y if case["beta"] else product(x)


def work(case):
    n = case["n"]
    if case["matrix"] == "poisson":
        nnz = 5 * n - 4 * round(n ** 0.5)
    elif case["matrix"] == "stencil":
        nnz = (3 * round(n ** (1.0 / 3.0)) - 2) ** 3
    elif case["matrix"] == "powerlaw":
        nnz = int(14.85 * n)
    else:
        n = int(_fem_sizes(case["count"], n).sum())
        nnz = int((FEM_LO + FEM_HI) / 2 * n * 0.92)  # drawn columns that coincide are kept once
    k = max(1, case["k"])
    vectors = 8 * n * k * (3 if case["beta"] else 2)
    vb = 8 if case["val"] == "f64" or case["op"] == "rebuild" else 6 if case["val"] == "f32lo" else 4
    cb = 2 if case["col"] == "d16" else 4
    b = nnz * (vb + cb) + 4 * (n + 1) + vectors
    if case["op"] == "convert":  # the x-baked array written and read again, and the row descriptors
        b += 2 * (16 * nnz + 4 * nnz)
    if case["op"] == "rebuild":  # the plan's stream written and read again
        b += 2 * nnz * ((8 if case["val"] == "f64" else 4) + 4)
    return {"bytes": b, "flops": 2.0 * nnz * k}
