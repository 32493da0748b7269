"""The library's memory pool: plans and GPU-built formats on recycled
blocks, dropped with work in flight, from several threads, and given back."""
from __future__ import annotations

import threading

import numpy as np
import pytest

from paritylib import assert_parity

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def env():
    import torch
    from int_spmv_b200 import device as D
    from int_spmv_b200 import matrices as M
    from oracle import Oracle
    return torch, D, M, Oracle()


def make(env, n, seed):
    torch, D, M, orc = env
    row, col, val = M.random_csr(n, seed, rl_max=30, empty_frac=0.1)
    x = M.uniform_x(n, seed)
    dev = [D.to_device(a) for a in (row, col, val, x)]
    return dev, orc.cf_csr(row, col, val, x), orc.abs_csr(row, col, val, x)


def test_recycled_blocks(env):
    """Plans and formats of nearly the same sizes, one after the other: each
    starts on memory that holds another's arrays."""
    torch, D, _, _ = env
    for i in range(6):
        (row, col, val, x), ref, absax = make(env, 20_000 + 37 * i, i)
        for kind in ("f64", "f32"):
            y = D.Plan.from_device_csr(row, col, val, val_kind=kind).spmv(x)
            assert_parity(y.cpu().numpy(), ref, absax, 1e-12 if kind == "f64" else 1e-6)
        for mode, th in (("COM", 1), ("NOC", 1), ("NOC", 4)):
            y = D.DeviceAXT(row, col, val, x, th=th, mode=mode).spmv(torch.zeros_like(x))
            assert_parity(y.cpu().numpy(), ref, absax)
        assert_parity(D.DeviceK1(row, col, val).spmv(x, torch.empty_like(x)).cpu().numpy(), ref, absax)
    assert 0 < D.trim_pool(1 << 40) <= 2 << 30
    assert D.trim_pool(0) == 0


def test_dropped_in_flight(env):
    """A plan dropped right after its product is launched on another stream:
    its blocks are not reused before the product is done."""
    torch, D, _, _ = env
    (row, col, val, x), ref, absax = make(env, 60_000, 3)
    (row2, col2, val2, x2), ref2, absax2 = make(env, 60_100, 4)
    side = torch.cuda.Stream()
    a = torch.randn(4096, 4096, device="cuda")
    for _ in range(5):
        plan, y = D.Plan.from_device_csr(row, col, val), torch.empty_like(x)
        torch.cuda.synchronize()
        with torch.cuda.stream(side):
            a @ a  # keeps the product waiting
            plan.spmv(x, y)
        del plan
        y2 = D.Plan.from_device_csr(row2, col2, val2).spmv(x2)
        torch.cuda.synchronize()
        assert_parity(y.cpu().numpy(), ref, absax)
        assert_parity(y2.cpu().numpy(), ref2, absax2)


def test_threads(env):
    """Four threads build, multiply and drop at once, each on its stream."""
    torch, D, _, _ = env
    mats = [make(env, 8_000 + 11 * t, t) for t in range(4)]
    torch.cuda.synchronize()
    wrong = []

    def work(t):
        (row, col, val, x), ref, absax = mats[t]
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for _ in range(20):
                y = D.Plan.from_device_csr(row, col, val).spmv(x)
                s.synchronize()
                if np.any(np.abs(y.cpu().numpy() - ref) > 1e-12 * absax):
                    wrong.append(t)

    ts = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not wrong


@pytest.mark.parametrize("mode", ["thread_local", "relaxed"])
def test_dropped_beside_a_capture(env, mode):
    """Plans and GPU-built formats dropped by one thread while another
    captures a graph: the capture goes on, and its graph runs."""
    torch, D, _, _ = env
    (row, col, val, x), ref, absax = make(env, 20_000, 5)
    plan, y = D.Plan.from_device_csr(row, col, val), torch.empty_like(x)
    for _ in range(2):  # also the memory the drops need, once
        drop = [D.Plan.from_device_csr(row, col, val), D.DeviceAXT(row, col, val, x), D.DeviceK1(row, col, val)]
        plan.spmv(x, y)
        torch.cuda.synchronize()
        s, graph = torch.cuda.Stream(), torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s, capture_error_mode=mode):
            plan.spmv(x, y)
            t = threading.Thread(target=drop.clear)
            t.start()
            t.join()
            y.mul_(2.0)
        y.zero_()
        graph.replay()
        torch.cuda.synchronize()
        assert_parity(0.5 * y.cpu().numpy(), ref, absax)


def test_graph_products_beside_drops(env):
    """spmv_graph captures anew for each pair of x and y while another thread
    builds and drops plans."""
    torch, D, _, _ = env
    (row, col, val, x), ref, absax = make(env, 20_000, 6)
    plan, ys = D.Plan.from_device_csr(row, col, val), [torch.empty_like(x) for _ in range(2)]
    torch.cuda.synchronize()
    stop, built = threading.Event(), []

    def churn():
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            while not stop.is_set():
                D.Plan.from_device_csr(row, col, val)
                built.append(1)

    t = threading.Thread(target=churn)
    t.start()
    try:
        for i in range(200):
            plan.spmv_graph(x, ys[i % 2])
    finally:
        stop.set()
        t.join()
    torch.cuda.synchronize()
    assert built
    for y in ys:
        assert_parity(y.cpu().numpy(), ref, absax)


@pytest.mark.parametrize("where", ["new_thread", "other_context"])
def test_trim_gives_memory_back(env, where):
    """ispmv_pool_trim frees what it no longer counts, from a thread that has
    no context yet and from one whose current context is another one of the
    device's."""
    import ctypes as C
    torch, D, _, _ = env
    D.trim_pool(0)
    n = 2_000_000
    row = torch.arange(0, 8 * n + 1, 8, dtype=torch.int32, device="cuda")
    col = torch.randint(0, n, (8 * n,), dtype=torch.int32, device="cuda")
    val = torch.rand(8 * n, dtype=torch.float64, device="cuda")
    D.Plan.from_device_csr(row, col, val)
    torch.cuda.synchronize()
    kept = D.trim_pool(1 << 40)
    assert kept > 100 << 20
    before = torch.cuda.mem_get_info()[0]
    left, cu = [], C.CDLL("libcuda.so.1")

    def trim():
        ctx = C.c_void_p()
        if where == "other_context":
            assert cu.cuCtxCreate_v2(C.byref(ctx), 0, 0) == 0
        left.append(D.trim_pool(0))
        if where == "other_context":
            assert cu.cuCtxDestroy_v2(ctx) == 0

    t = threading.Thread(target=trim)
    t.start()
    t.join()
    assert left == [0]
    assert torch.cuda.mem_get_info()[0] - before > 0.9 * kept


def test_large_plan_takes_its_bytes(env):
    """Blocks of gigabytes are not rounded up by a share of their size: a plan
    takes the device memory its info names (and work areas, and pages)."""
    torch, D, _, _ = env
    n = 37_800_000  # 302.4M nonzeros: 2.42 GB of values, 1.21 GB of columns, both just above a step of 1/8
    row = torch.arange(0, 8 * n + 1, 8, dtype=torch.int32, device="cuda")
    col = torch.randint(0, n, (8 * n,), dtype=torch.int32, device="cuda")
    val = torch.rand(8 * n, dtype=torch.float64, device="cuda")
    D.trim_pool(0)
    torch.cuda.synchronize()
    before = torch.cuda.mem_get_info()[0]
    plan = D.Plan.from_device_csr(row, col, val)
    D.trim_pool(0)
    used = before - torch.cuda.mem_get_info()[0]
    assert used <= 1.01 * plan.info["device_bytes"] + (64 << 20), (used, plan.info["device_bytes"])


def test_graph_products_in_threads(env):
    """Graph products of new plans captured by four threads at once, the plans
    dropped and others captured on the streams they left."""
    torch, D, _, _ = env
    mats = [make(env, 8_000 + 13 * t, 20 + t) for t in range(4)]
    torch.cuda.synchronize()
    wrong = []

    def work(t):
        (row, col, val, x), ref, absax = mats[t]
        s = torch.cuda.Stream()
        with torch.cuda.stream(s):
            for i in range(25):
                plan, y = D.Plan.from_device_csr(row, col, val, val_kind="f32" if i % 3 == 1 else "f64"), torch.empty_like(x)
                for _ in range(2):
                    plan.spmv_graph(x, y)
                s.synchronize()
                if np.any(np.abs(y.cpu().numpy() - ref) > (1e-6 if i % 3 == 1 else 1e-12) * absax):
                    wrong.append((t, i))

    ts = [threading.Thread(target=work, args=(t,)) for t in range(4)]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    assert not wrong
