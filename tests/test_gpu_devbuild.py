"""Format conversion on the GPU (ispmv_dev_build_axt, ispmv_dev_build_k1):
the AXT and K1 arrays built from device CSR arrays are bit-identical to the
host builders' (which the golden fixtures pin to the reference), for NOC at
tileHeight 1, 3, 4, 8, 16, 48, COM at bs 8, 128, 256, 512, and K1 with many
equal row lengths (the stable order); the reference's kernels on them match
the CSR oracle; and the multi-block prefix scan is exercised past one block
of block totals (> 4M rows)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import golden_names, load_golden
from paritylib import TOL_F64, assert_parity

pytestmark = pytest.mark.gpu

SHAPES = [("NOC", 1, 128), ("NOC", 3, 128), ("NOC", 4, 128), ("NOC", 8, 128), ("NOC", 16, 128), ("NOC", 48, 128),
          ("COM", 1, 8), ("COM", 1, 128), ("COM", 1, 256), ("COM", 1, 512)]


def _dev(a):
    from int_spmv_b200 import device as D
    return D.to_device(np.ascontiguousarray(a))


def check_build(row, col, val, x, mode, th, bs, run_kernel=True):
    import torch

    from int_spmv_b200 import device as D
    from int_spmv_b200 import formats as F
    from oracle import Oracle
    csr = F.CSR(row, col, val)
    fd_h, h = F.getFormatDataAXT(0, bs, 8, th, mode, csr, x)
    d = D.DeviceAXT(_dev(row), _dev(col if len(col) else np.zeros(1, np.uint32)), _dev(val if len(val) else np.zeros(1)),
                    _dev(x), bs=bs, th=th, mode=mode)
    for f in ("tileN", "lenAX", "lenSEC", "lenCON", "log", "logTH", "tileH", "tileHW"):
        assert getattr(d.c, f) == getattr(h.c, f), f
    arrs = d.to_host()
    assert np.array_equal(arrs["con"], h.con)
    assert np.array_equal(arrs["sec"], h.sec)
    assert np.array_equal(arrs["ax"].view(np.uint64), h.ax.view(np.uint64))  # bit for bit
    assert d.fd.name.decode() == fd_h.name
    assert d.fd.mfp == fd_h.mfp and d.fd.beta == fd_h.beta
    assert d.conversion_s > 0
    if run_kernel:
        # the reference kernels on the device-built arrays; the compacted one
        # is judged against the CSR oracle (the reference's own result drops
        # row-0 segments, README.md:33)
        y = torch.zeros(csr.n, dtype=torch.float64, device="cuda")
        d.spmv(y)
        orc = Oracle()
        assert_parity(y.cpu().numpy(), orc.cf_csr(row, col, val, x), orc.abs_csr(row, col, val, x), TOL_F64,
                      what=f"{mode}{th}/{bs}")
    return d


@pytest.mark.parametrize("name", golden_names())
@pytest.mark.parametrize("mode,th,bs", SHAPES)
def test_device_axt_matches_host_golden(name, mode, th, bs):
    g = load_golden(name)
    check_build(g["row"], g["col"], g["val"], g["x"], mode, th, bs)


@pytest.mark.parametrize("mode,th,bs", SHAPES)
def test_device_axt_random(mode, th, bs):
    from int_spmv_b200 import matrices as M
    row, col, val = M.random_csr(30011, 41, rl_max=300, empty_frac=0.1)
    check_build(row, col, val, M.uniform_x(30011, 41), mode, th, bs)


def test_device_axt_many_rows():
    """n + 1 > 1024 scan blocks of 4096 entries: the block totals take more
    than one pass of the totals scan."""
    rng = np.random.default_rng(7)
    n = 4_300_000
    rl = rng.integers(0, 3, n)
    row = np.concatenate([[0], np.cumsum(rl)]).astype(np.uint32)
    rows = np.repeat(np.arange(n), rl)
    col = ((rows + rng.integers(0, 50, len(rows))) % n).astype(np.uint32)
    # distinct ascending columns within each row
    key = rows.astype(np.int64) * n + col
    key = np.unique(key)
    rows, col = (key // n).astype(np.int64), (key % n).astype(np.uint32)
    rl = np.bincount(rows, minlength=n)
    row = np.concatenate([[0], np.cumsum(rl)]).astype(np.uint32)
    val = rng.standard_normal(len(col))
    x = rng.uniform(-1, 1, n)
    for mode, th, bs in (("COM", 1, 128), ("NOC", 1, 128), ("NOC", 4, 128)):
        check_build(row, col, val, x, mode, th, bs, run_kernel=False)


@pytest.mark.parametrize("mode,th,bs", SHAPES + [("NOC", 3, 128), ("NOC", 64, 128), ("NOC", 65, 128), ("NOC", 200, 128)])
@pytest.mark.parametrize("kind", ["long", "edges", "gaps", "none", "many"])
def test_device_axt_rows_and_chunks(mode, th, bs, kind):
    """Rows over many CTAs' slots, rows that end just before, at and after the
    end of a CTA's slots, long runs of empty rows inside them, no slots at all,
    and enough slots for the longer chunks."""
    rng = np.random.default_rng(len(kind))
    if kind == "long":
        rl = np.r_[[0, 9001, 5, 20000, 0, 0, 1], np.full(70, 300)]
    elif kind == "edges":
        rl = np.r_[[1024, 1023, 1, 1025, 2047, 1, 2048, 0, 2049, 1, 511, 512, 513], np.full(600, 5), [2048, 0]]
    elif kind == "gaps":
        rl = np.zeros(300_000, int)
        rl[[3, 4, 260, 70_000, 70_300, 299_999]] = [7, 600, 3, 40, 1, 12]
    elif kind == "none":
        rl = np.zeros(1000, int)
    else:
        rl = rng.integers(0, 24, 150_000)
        rl[1000] = 30_000
    n = len(rl) if len(rl) > 30_000 else 30_000
    rl = np.r_[rl, np.zeros(n - len(rl), int)]
    row = np.concatenate([[0], np.cumsum(rl)]).astype(np.uint32)
    j = np.arange(int(row[-1])) - np.repeat(row[:-1], rl)
    col = ((np.repeat(np.arange(n) * 13 % (n - rl.max()) if rl.max() < n else np.zeros(n, int), rl)) + j).astype(np.uint32)
    check_build(row, col, rng.standard_normal(len(col)), rng.uniform(-1, 1, n), mode, th, bs, run_kernel=False)


@pytest.mark.parametrize("mode,th", [("COM", 1), ("NOC", 1), ("NOC", 4)])
def test_device_axt_counts_from_the_row_pointer(mode, th):
    """The slots come from the row pointer: a smaller nnz argument (it only
    names itself in the result) changes no array."""
    import ctypes as C

    import torch

    from int_spmv_b200 import device as D
    from int_spmv_b200 import matrices as M
    row, col, val = M.random_csr(20_011, 3, rl_max=60, empty_frac=0.1)
    t = [_dev(a) for a in (row, col, val, M.uniform_x(20_011, 3))]
    a = D.DeviceAXT(*t, th=th, mode=mode)
    b = D.DeviceAXT.__new__(D.DeviceAXT)
    b.c, b.fd = D.abi.StrMatAXT(), D.abi.StrFormatData()
    p = [x.data_ptr() for x in t]
    assert D.load().ispmv_dev_build_axt(128, 8, th, mode.encode(), 20_011, 1, *p, C.byref(b.c), C.byref(b.fd), 0) == 0
    torch.cuda.synchronize()
    ha, hb = a.to_host(), b.to_host()
    assert all(np.array_equal(ha[k].view(np.uint32), hb[k].view(np.uint32)) for k in ha)


def test_device_axt_time_of_long_rows():
    """Ten million nonzeros in 2000 rows convert in about the time they take
    in a million rows."""
    import torch

    from int_spmv_b200 import device as D

    def us(n, k):
        row = torch.arange(0, n * k + 1, k, dtype=torch.int32, device="cuda")
        col = torch.randint(0, n, (n * k,), dtype=torch.int32, device="cuda")
        val = torch.rand(n * k, dtype=torch.float64, device="cuda")
        x = torch.rand(n, dtype=torch.float64, device="cuda")
        return [min(D.DeviceAXT(row, col, val, x, th=th, mode=m).conversion_s for _ in range(6))
                for m, th in (("COM", 1), ("NOC", 1), ("NOC", 8))]

    for long, short in zip(us(2_000, 5_000), us(1_000_000, 10)):
        assert long < 2 * short, (long, short)


def check_build_k1(row, col, val, x):
    import torch

    from int_spmv_b200 import device as D
    from int_spmv_b200 import formats as F
    from oracle import Oracle
    csr = F.CSR(row, col, val)
    fd_h, h = F.getFormatDataK1(8, csr, x)
    d = D.DeviceK1(_dev(row), _dev(col if len(col) else np.zeros(1, np.uint32)),
                   _dev(val if len(val) else np.zeros(1)))
    assert (d.c.chunkNum, d.c.lenVC, d.c.nrows, d.c.nnz) == (h.c.chunkNum, h.c.lenVC, h.c.nrows, h.c.nnz)
    a = d.to_host()
    assert np.array_equal(a["permi"], h.permi)
    assert np.array_equal(a["nmc"], h.nmc) and np.array_equal(a["chp"], h.chp)
    assert np.array_equal(a["col"], h.col)
    assert np.array_equal(a["val"].view(np.uint64), h.val.view(np.uint64))
    assert d.fd.name.decode() == fd_h.name and d.fd.mfp == fd_h.mfp and d.fd.beta == fd_h.beta
    xt = _dev(x)
    y = torch.zeros(csr.n + 8, dtype=torch.float64, device="cuda")
    d.spmv(xt, y)
    orc = Oracle()
    assert_parity(y[:csr.n].cpu().numpy(), orc.cf_csr(row, col, val, x), orc.abs_csr(row, col, val, x), TOL_F64,
                  what="K1 built on the GPU")


@pytest.mark.parametrize("name", golden_names())
def test_device_k1_matches_host_golden(name):
    g = load_golden(name)
    check_build_k1(g["row"], g["col"], g["val"], g["x"])


def test_device_k1_random_and_ties():
    from int_spmv_b200 import matrices as M
    for n, seed, rl_max in ((30011, 41, 300), (20000, 7, 3), (4099, 3, 64)):  # many equal lengths
        row, col, val = M.random_csr(n, seed, rl_max=rl_max, empty_frac=0.1)
        check_build_k1(row, col, val, M.uniform_x(n, seed))


@pytest.mark.parametrize("mode", ["NOC", "COM"])
@pytest.mark.parametrize("k", [1, 3, 65])
def test_axt_h1_arrays_with_nothing_around_them(mode, k):
    """The tileH = 1 kernels on arrays that are each an allocation of their own
    (multiples of 2 MiB, whole): they read nothing before an array or past it."""
    import ctypes as C

    import torch

    from int_spmv_b200 import device as D
    rt = C.CDLL("libcudart.so.12")
    size = 2 << 20  # bytes of sec: k * 2 MiB (NOC: a word per tile of 8 slots; COM: per slot)
    words = k * size // 4
    tiles = words if mode == "NOC" else words // 8
    n = 1000
    rng = np.random.default_rng(k)
    ax = rng.uniform(-1, 1, (tiles, 16))
    rows = np.sort(rng.integers(0, n, tiles)).astype(np.uint32)
    sec = rows if mode == "NOC" else np.zeros(words, np.uint32)
    if mode == "COM":  # one row per tile, and one per block start: (row << 7) | length - 1
        sec[::8] = (rows << 7) | 7
    want = np.bincount(rows, (ax[:, :8] * ax[:, 8:]).sum(1), n)
    bound = np.bincount(rows, np.abs(ax[:, :8] * ax[:, 8:]).sum(1), n)
    p = []
    for a in (ax, sec):
        q = C.c_void_p()
        assert rt.cudaMalloc(C.byref(q), C.c_size_t(a.nbytes)) == 0
        assert rt.cudaMemcpy(q, a.ctypes.data_as(C.c_void_p), C.c_size_t(a.nbytes), 1) == 0
        p.append(q)
    y = torch.zeros(n, dtype=torch.float64, device="cuda")
    lib = D.load()
    if mode == "NOC":
        assert lib.ispmv_dev_int_axt_noc_h1(tiles, p[0], p[1], y.data_ptr(), None) == 0
    else:
        bn = (words + 127) // 128
        assert lib.ispmv_dev_int_axt_com_h1(bn, 128, 7, 8, tiles, 16 * tiles, words, p[0], p[1], y.data_ptr(), None) == 0
    torch.cuda.synchronize()
    for q in p:
        assert rt.cudaFree(q) == 0
    assert np.all(np.abs(y.cpu().numpy() - want) <= 1e-12 * bound)
