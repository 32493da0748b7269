"""The sizes at which a kernel's split of the work changes, against the
oracle's CSR product: |y - y_ref| <= tol (|A||x|), componentwise, the bounds of
every other plan test."""
from __future__ import annotations

import numpy as np
import pytest

from paritylib import TOL_F32, TOL_F64, assert_parity

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    import torch
    from int_spmv_b200 import device as D
    from int_spmv_b200 import formats as F
    from oracle import Oracle
    return torch, D, F, Oracle()


def rows_of(lengths, n, seed):
    """CSR of len(lengths) rows over n columns: distinct sorted columns, N(0,1)."""
    rng = np.random.default_rng(seed)
    row = np.zeros(len(lengths) + 1, np.uint32)
    row[1:] = np.cumsum(lengths)
    col = np.concatenate([np.sort(rng.permutation(n)[:k]) for k in lengths] + [np.zeros(0, int)]).astype(np.uint32)
    return row, col, rng.standard_normal(int(row[-1]))


def check(env, row, col, val, plan, val_kind, betas=(0, 1)):
    torch, _, _, orc = env
    n = len(row) - 1
    rng = np.random.default_rng(7)
    x, y0 = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
    for beta in betas:
        y = torch.from_numpy(y0.copy()).cuda()
        plan.spmv(torch.from_numpy(x).cuda(), y, beta=beta)
        ref = orc.cf_csr(row, col, val, x) + (y0 if beta else 0.0)
        absax = orc.abs_csr(row, col, val, x) + (np.abs(y0) * 1e-4 if beta else 0.0)
        assert_parity(y.cpu().numpy(), ref, absax, TOL_F64 if val_kind == "f64" else TOL_F32, what=f"beta {beta}")


@pytest.mark.parametrize("reorder", [True, False])
@pytest.mark.parametrize("val_kind", ["f64", "f32"])
@pytest.mark.parametrize("top", [0, 1, 2, 7, 8, 9, 63, 64, 65, 255, 256, 257, 263, 1299])
def test_k1_chunk_classes(env, reorder, val_kind, top):
    """K1 chunks of a group (< 64 columns), a warp (< 256) and a CTA, odd and
    even column counts, remainders of the unrolled loops, an unfilled last chunk."""
    _, D, F, _ = env
    n = 1301
    lengths = np.random.default_rng(top).integers(0, 12, n)
    lengths[5:5 + 61] = top
    lengths[700:711] = max(0, top - 1)
    row, col, val = rows_of(np.minimum(lengths, n), n, top)
    csr = F.CSR(row, col, val)
    plan = D.Plan(csr, F.getFormatDataK1(8, csr, np.zeros(n))[1], reorder=reorder, val=val_kind)
    check(env, row, col, val, plan, val_kind)


@pytest.mark.parametrize("fmt", ["CSR", "AXC", "NOC1", "NOC8", "NOC16"])
@pytest.mark.parametrize("nnz", [1, 511, 512, 513, 4097, 70_001, 2_300_001])
def test_segment_sizes(env, fmt, nnz):
    """The lengths of a warp's segment (512 slots up to the variant's), the
    stream's last partial segment, and formats whose row padding the plan drops."""
    _, D, F, _ = env
    n = max(40, nnz // 7)
    lengths = np.full(n, nnz // n)
    lengths[: nnz - int(lengths.sum())] += 1
    lengths[n // 2] += lengths[n // 3]  # an empty row and a longer one
    lengths[n // 3] = 0
    rng = np.random.default_rng(nnz)
    row = np.zeros(n + 1, np.uint32)
    row[1:] = np.cumsum(lengths)
    col = np.concatenate([(r + 3 * np.arange(k)) % n for r, k in enumerate(lengths)]).astype(np.uint32)
    val = rng.standard_normal(nnz)
    csr = F.CSR(row, col, val)
    z = np.zeros(n)
    f = None if fmt == "CSR" else F.getFormatDataAXC(0, csr, z)[1] if fmt == "AXC" else \
        F.getFormatDataAXT(0, 128, 8, int(fmt[3:]), "NOC", csr, z)[1]
    for val_kind in ("f64", "f32"):
        plan = D.Plan(csr, f, val=val_kind)
        check(env, row, col, val, plan, val_kind)
        if fmt != "CSR":
            assert plan.info["slots"] >= nnz  # the format's own slots, its padding included


def test_padding_reads_no_x(env):
    """A format's row padding contributes nothing, whatever x[0] is."""
    torch, D, F, orc = env
    row, col, val = rows_of(np.array([2, 3, 5, 1, 0, 4]), 6, 3)
    col = np.maximum(col, 1).astype(np.uint32)  # no element in column 0
    csr = F.CSR(row, col, val)
    x = np.random.default_rng(1).uniform(-1, 1, 6)
    ref, absax = orc.cf_csr(row, col, val, x), orc.abs_csr(row, col, val, x)
    x[0] = np.inf
    for f in (F.getFormatDataAXC(0, csr, x)[1], F.getFormatDataAXT(0, 128, 8, 1, "NOC", csr, x)[1],
              F.getFormatDataAXT(0, 128, 8, 4, "NOC", csr, x)[1]):
        assert_parity(D.Plan(csr, f).spmv(torch.from_numpy(x).cuda()).cpu().numpy(), ref, absax, TOL_F64)


@pytest.mark.parametrize("n", [3583, 3584, 3585, 3586, 8191, 9000, 70_001])
def test_windows_host_device(env, n):
    """Per-CTA x windows at sizes around the window's (3584): the device's
    choice is the host's, inside x, and the product is right; far columns at
    both ends of x, tiles past the last slot."""
    torch, D, F, _ = env
    rng = np.random.default_rng(n)
    lengths = rng.integers(1, 9, n)
    row, col, val = rows_of(np.zeros(n, int), n, n)
    row[1:] = np.cumsum(lengths)
    near = (np.repeat(np.arange(n), lengths) + rng.integers(-40, 41, int(row[-1]))) % n
    col = np.where(rng.random(len(near)) < 0.6, near, rng.integers(0, n, len(near))).astype(np.uint32)
    val = rng.standard_normal(len(col))
    host = D.Plan(F.CSR(row, col, val), None, kernel="wide", variant=26)
    dev = D.Plan.from_device_csr(D.to_device(row), D.to_device(col), D.to_device(val), kernel="wide", variant=26)
    a, b = host.export_stream(), dev.export_stream()
    for k in ("val", "col", "heads", "segh", "win_lo", "win_len"):
        assert np.array_equal(a[k], b[k]), k
    assert np.all(a["win_lo"] % 2 == 0) and np.all(a["win_lo"].astype(int) + a["win_len"] <= n)
    check(env, row, col, val, dev, "f64")


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("nnz", [1, 7, 8, 127, 128, 129, 511, 512, 513, 1025, 30_001])
def test_axt_kernels_steps(env, nnz, offset):
    """The tileH = 1 kernels (x-baked arrays) around a warp's step (128 slots)
    and range (512), 16-byte aligned arrays or not; the GPU's conversion of the
    same matrix at tile heights that fill tiles in ax order and in slot order."""
    torch, D, F, orc = env
    n = max(3, nnz // 3)
    rng = np.random.default_rng(nnz)
    cuts = np.sort(rng.integers(0, nnz + 1, n - 1))
    lengths = np.minimum(np.diff(np.concatenate([[0], cuts, [nnz]])), n)
    row, col, val = rows_of(lengths, n, nnz)
    x = rng.uniform(-1, 1, n)
    csr = F.CSR(row, col, val)
    ref, absax = orc.cf_csr(row, col, val, x), orc.abs_csr(row, col, val, x)

    def up(a):  # a device copy that starts `offset` elements into its buffer
        t = D.to_device(a)
        buf = torch.zeros(t.numel() + offset, dtype=t.dtype, device="cuda")
        buf[offset:] = t
        return buf[offset:]

    y = torch.zeros(n, dtype=torch.float64, device="cuda")
    noc = F.getFormatDataAXT(0, 128, 8, 1, "NOC", csr, x)[1]
    D.int_axt_noc_h1(noc.c.tileN, up(noc.ax), up(noc.sec), y)
    assert_parity(y.cpu().numpy(), ref, absax, TOL_F64, "NOC")
    for bs in (8, 512):
        com = F.getFormatDataAXT(0, bs, 8, 1, "COM", csr, x)[1]
        c = com.c
        y.zero_()
        D.int_axt_com_h1((c.lenSEC + bs - 1) // bs, bs, c.log, 8, c.tileN, c.lenAX, c.lenSEC, up(com.ax), up(com.sec), y)
        assert_parity(y.cpu().numpy(), ref, absax, TOL_F64, f"COM {bs}")
    dev = [D.to_device(a) for a in (row, col, val, x)]
    for mode, th in (("COM", 1), ("NOC", 1), ("NOC", 3), ("NOC", 64), ("NOC", 65)):
        got = D.DeviceAXT(*dev, th=th, mode=mode).to_host()
        want = F.getFormatDataAXT(0, 128, 8, th, mode, csr, x)[1]
        for k in ("con", "ax", "sec"):
            assert np.array_equal(got[k], getattr(want, k)), (mode, th, k)


@pytest.mark.parametrize("k", [8, 16, 32, 11])
@pytest.mark.parametrize("n,rl", [(40, 3), (64, 8), (3000, 1), (700, 37), (130, 129), (2, 1)])
def test_spmm_parts(env, k, n, rl):
    """SpMM parts of 64 slots and up: rows that start at part and CTA edges,
    rows of a slot, rows over many parts, of whole CTAs, and the last part."""
    torch, D, F, orc = env
    rng = np.random.default_rng(n + rl)
    lengths = np.full(n, rl)
    lengths[n // 2:] = rng.integers(0, min(n, 2 * rl) + 1, n - n // 2)
    if n == 3000:
        lengths[77] = 2999  # one row over several CTAs
    row, col, val = rows_of(lengths, n, n)
    X = rng.uniform(-1, 1, (n, k))
    for f, kw in ((None, {}), (None, dict(kernel="ldg")), (None, dict(kernel="wide", variant=0))):
        plan = D.Plan(F.CSR(row, col, val), f, **kw)
        Y = torch.full((n, k), 9.0, dtype=torch.float64, device="cuda")
        plan.spmm(torch.from_numpy(X).cuda(), Y)
        for j in range(k):
            xj = np.ascontiguousarray(X[:, j])
            assert_parity(Y[:, j].cpu().numpy(), orc.cf_csr(row, col, val, xj), orc.abs_csr(row, col, val, xj), TOL_F64)


@pytest.mark.parametrize("val_kind", ["f64", "f32"])
@pytest.mark.parametrize("n,w,span", [(1, 1, 0), (31, 3, 40), (32, 48, 60), (33, 9, 100), (4000, 10, 65_000), (70_000, 19, 65_535),
                                      (70_000, 19, 65_536), (5000, 49, 300)])
def test_slices_of_rows(env, val_kind, n, w, span):
    """16-bit-delta plans of 32 equally long rows side by side: unfilled last
    slices, remainders of the unrolled loop, shorter and empty rows, the widest
    rows (48) and columns (65535) they take and the first they do not, no read
    of x for padding."""
    torch, D, F, orc = env
    rng = np.random.default_rng(n + w)
    lengths = np.full(n, min(w, n))
    if n > 100:
        lengths[rng.integers(0, n, n // 300)] = 0
        lengths[rng.integers(0, n, n // 200)] = w - 1
    row = np.zeros(n + 1, np.uint32)
    row[1:] = np.cumsum(lengths)
    k = np.arange(int(row[-1])) - np.repeat(row[:-1], lengths)
    r = np.repeat(np.arange(n), lengths) // 32 * 32
    lo = np.minimum(r, max(0, n - 1 - span))
    col = np.minimum(lo + np.where(k == w - 1, span, k), n - 1).astype(np.uint32)
    val = rng.standard_normal(len(col))
    csr = F.CSR(row, col, val)
    for f in (None, F.getFormatDataAXT(0, 128, 8, 4, "NOC", csr, np.zeros(n))[1]):
        plan = D.Plan(csr, f, val=val_kind, col="d16")
        assert plan.info["col_kind"] == 1
        check(env, row, col, val, plan, val_kind)
        assert ("rows32" in plan.kernel_name()) == (w <= 48 and span <= 65_535)
        x = torch.rand(n, dtype=torch.float64, device="cuda")
        y = torch.empty_like(x)
        a = plan.spmv(x, y).clone()
        assert torch.equal(plan.spmv_graph(x, y), a)
    with pytest.raises(Exception):
        plan.spmm(torch.zeros((n, 8), dtype=torch.float64, device="cuda"))


@pytest.mark.parametrize("kw", [{}, dict(val="f32"), dict(kernel="wide", variant=0), dict(kernel="ldg")])
@pytest.mark.parametrize("segs", [1, 7, 8, 9, 16, 17, 60, 128, 129, 137])
def test_rows_over_many_segments(env, kw, segs):
    """Rows of more records than one thread adds up, next to short and empty
    rows and to one another: the records before and after the row are others',
    none, or a whole pass of the warp's."""
    _, D, F, _ = env
    n, k = 80_000, 512 * segs
    lengths = np.zeros(n, int)
    lengths[100:3000] = 3
    lengths[[0, 1, 50, 3000, 3002, n - 1]] = [k, k + 1, k - 1, k + 255, k, k]
    row = np.zeros(n + 1, np.uint32)
    row[1:] = np.cumsum(lengths)
    j = np.arange(int(row[-1])) - np.repeat(row[:-1], lengths)
    col = (np.repeat((np.arange(n) * 7) % (n - lengths.max()), lengths) + j).astype(np.uint32)
    val = np.random.default_rng(segs).standard_normal(len(col))
    check(env, row, col, val, D.Plan(F.CSR(row, col, val), None, **kw), kw.get("val", "f64"))


def test_one_very_long_row(env):
    """A matrix with one row of a million nonzeros takes a few times what as
    many in short rows take, not what adding its records one by one does."""
    torch, D, _, _ = env
    def us(lengths):
        n = len(lengths)
        row = torch.zeros(n + 1, dtype=torch.int32, device="cuda")
        row[1:] = torch.from_numpy(lengths).cuda().cumsum(0)
        nnz = int(row[-1])
        col = torch.randint(0, n, (nnz,), dtype=torch.int32, device="cuda")
        plan = D.Plan.from_device_csr(row, col, torch.rand(nnz, dtype=torch.float64, device="cuda"))
        x = torch.rand(n, dtype=torch.float64, device="cuda")
        y, best = torch.empty_like(x), 1e9
        for _ in range(6):
            a, b = (torch.cuda.Event(enable_timing=True) for _ in range(2))
            a.record()
            for _ in range(20):
                plan.spmv(x, y)
            b.record()
            torch.cuda.synchronize()
            best = min(best, a.elapsed_time(b) * 50)
        return best

    short = us(np.full(70_000, 15))
    one = us(np.concatenate([np.full(5_000, 5), [1_000_000], np.full(5_000, 5)]))
    assert one < 6 * short, (one, short)


@pytest.mark.parametrize("fmt", ["AXC", "NOC1", "NOC4"])
@pytest.mark.parametrize("last", [1, 2, 3, 4, 300])
def test_format_of_another_matrix(env, fmt, last):
    """A plan multiplies what its format holds, also where the CSR beside it
    has rows of other lengths (its last row shorter or longer here)."""
    torch, D, F, orc = env
    n = 300
    row, col, val = rows_of(np.full(n, 3), n, 1)
    made = F.CSR(row, col, val)
    lengths = np.full(n, 3)
    lengths[-1] = last
    given = F.CSR(*rows_of(lengths, n, 2))
    f = F.getFormatDataAXC(0, made, np.zeros(n))[1] if fmt == "AXC" else \
        F.getFormatDataAXT(0, 128, 8, int(fmt[3:]), "NOC", made, np.zeros(n))[1]
    x = np.random.default_rng(3).uniform(-1, 1, n)
    for kw in (dict(kernel="wide", variant=4), dict(kernel="wide", variant=4, col="d16"), dict(col="d16"), {}):
        y = D.Plan(given, f, **kw).spmv(torch.from_numpy(x).cuda()).cpu().numpy()
        assert_parity(y, orc.cf_csr(row, col, val, x), orc.abs_csr(row, col, val, x), TOL_F64, what=str(kw))


def test_slices_name_their_kernel(env):
    """kernel_name() is the kernel that a profiler shows."""
    torch, D, F, _ = env
    from int_spmv_b200 import matrices as M
    row, col, val = M.stencil27(30)
    plan = D.Plan(F.CSR(row, col, val), None, col="d16")
    plan.spmv(torch.rand(len(row) - 1, dtype=torch.float64, device="cuda"))
    assert plan.kernel_name().startswith("slice_rows<"), plan.kernel_name()


@pytest.mark.parametrize("empty", ["none", "first", "last", "some", "all but one"])
def test_padding_is_dropped(env, empty):
    """The lane-interleaved plans of padded formats hold the nonzeros alone,
    wherever the empty rows are; the 4-slots-per-lane ones of small matrices
    hold the format's slots."""
    _, D, F, _ = env
    n = 700
    lengths = np.random.default_rng(3).integers(1, 30, n)
    lengths[{"none": [], "first": [0, 1, 2], "last": [n - 1, n - 2], "some": [5, 6, 100, 690],
             "all but one": [r for r in range(n) if r != 400]}[empty]] = 0
    row, col, val = rows_of(lengths, n, 4)
    csr = F.CSR(row, col, val)
    z = np.zeros(n)
    for f in [F.getFormatDataAXC(0, csr, z)[1]] + [F.getFormatDataAXT(0, 128, 8, th, "NOC", csr, z)[1] for th in (1, 3, 4, 8, 16)]:
        p = D.Plan(csr, f)
        assert p.export_stream()["layout"]["slots"] == len(col)
        check(env, row, col, val, p, "f64")
    axc = F.getFormatDataAXC(0, csr, z)[1]
    for kernel in ("ldg", "tma"):
        p = D.Plan(csr, axc, kernel=kernel)
        assert p.export_stream()["layout"]["slots"] == p.info["slots"]
        check(env, row, col, val, p, "f64")
