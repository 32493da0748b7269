"""Synthetic workload generators (sizes and distributions the benchmark
configurations state) and the multi-process timing reduction bench.py uses
(max over ranks), run as world-size-2 gloo ranks on the CPU."""
from __future__ import annotations

import os

import numpy as np
import pytest

from int_spmv_b200 import matrices as M


def test_poisson_sizes():
    row, col, val = M.poisson2d(512)
    n = 512 * 512
    assert len(row) - 1 == n and len(col) == 5 * n - 4 * 512 == 1308672
    assert np.all(val[row[:-1][:3] + 0] <= 4.0)
    rl = np.diff(row.astype(np.int64))
    assert rl.min() == 3 and rl.max() == 5
    k = np.repeat(np.arange(n, dtype=np.int64), rl) * n + col
    assert np.all(np.diff(k) > 0)


def test_stencil27_small():
    m = 12
    row, col, val = M.stencil27(m, seed=2)
    n = m ** 3
    assert len(col) == (3 * m - 2) ** 3
    rl = np.diff(row.astype(np.int64))
    assert rl.min() == 8 and rl.max() == 27
    r = np.repeat(np.arange(n), rl)
    diag = r == col
    assert np.all(val[diag] == 26.0)
    assert np.all((val[~diag] >= -1.1) & (val[~diag] <= -0.9))
    assert np.array_equal(M.stencil27(m, seed=2)[2], val)  # seeded


def test_powerlaw_properties():
    n = 200_000
    row, col, val = M.powerlaw(n, seed=1)
    rl = np.diff(row.astype(np.int64))
    assert rl.min() >= 1 and rl.max() <= 5000
    assert 13.5 < rl.mean() < 16.5  # lognormal(2.2, 1): mean e^2.7 = 14.9
    r = np.repeat(np.arange(n, dtype=np.int64), rl)
    k = r * n + col
    assert np.all(np.diff(k) > 0)  # distinct, sorted in each row
    band = np.abs(r - col.astype(np.int64)) <= 1000
    assert 0.69 < band.mean() < 0.72
    assert abs(val.mean()) < 0.01 and abs(val.std() - 1) < 0.01
    row2, col2, val2 = M.powerlaw(n, seed=1)
    assert np.array_equal(col, col2) and np.array_equal(val, val2)


def test_fem_batch_small():
    mats = M.fem_batch(count=6, seed=4, n_lo=1000, n_hi=3000)
    assert len(mats) == 6
    for row, col, val in mats:
        n = len(row) - 1
        rl = np.diff(row.astype(np.int64))
        assert rl.min() >= 7 and rl.max() <= 81
        r = np.repeat(np.arange(n), rl)
        assert np.all(np.abs(r - col.astype(np.int64)) <= 3 * 81)
        d = val[r == col]
        off = np.abs(np.where(r == col, 0, val))
        assert np.all(d >= 1.0)


def _rank_main(rank, world, port, q):
    import torch.distributed as dist
    os.environ.update(MASTER_ADDR="127.0.0.1", MASTER_PORT=str(port))
    dist.init_process_group("gloo", rank=rank, world_size=world)
    import bench
    v = bench.max_over_ranks(1.0 + rank * 2.5, world, device="cpu")
    bench.barrier(world)
    q.put((rank, v))
    dist.destroy_process_group()


def test_max_over_ranks_gloo():
    import multiprocessing as mp
    import socket
    s = socket.socket()
    s.bind(("127.0.0.1", 0))
    port = s.getsockname()[1]
    s.close()
    ctx = mp.get_context("spawn")
    q = ctx.Queue()
    ps = [ctx.Process(target=_rank_main, args=(r, 2, port, q)) for r in range(2)]
    for p in ps:
        p.start()
    res = dict(q.get(timeout=120) for _ in ps)
    for p in ps:
        p.join(timeout=60)
    assert res == {0: 3.5, 1: 3.5}


def test_gen_banded_invariants():
    """The C generator of the batched workload: row lengths, band, distinct
    ascending columns with the diagonal, diagonal = |off-diagonal sum| + 1,
    N(0,1) off-diagonals, and determinism."""
    from int_spmv_b200 import matrices as M
    for n, seed in ((1, 3), (9, 4), (1000, 5), (20011, 6)):
        row, col, val = M.fem_banded_c(n, seed)
        rl = np.diff(row.astype(np.int64))
        assert np.all(rl >= min(7, n)) and np.all(rl <= min(81, n))
        rows = np.repeat(np.arange(n), rl)
        assert np.all(np.abs(col.astype(np.int64) - rows) <= 3 * rl[rows])
        # ascending, distinct within each row
        d = np.diff(col.astype(np.int64))
        inner = np.ones(len(col), bool)
        inner[row[1:-1].astype(np.int64)] = False
        assert np.all(d[inner[1:]] > 0)
        diag = col.astype(np.int64) == rows
        assert np.array_equal(np.bincount(rows[diag], minlength=n), np.ones(n, np.int64))
        offsum = np.bincount(rows[~diag], weights=val[~diag], minlength=n)
        assert np.allclose(val[diag], np.abs(offsum) + 1.0)
        r2, c2, v2 = M.fem_banded_c(n, seed)
        assert np.array_equal(row, r2) and np.array_equal(col, c2) and np.array_equal(val, v2)
    off = val[~diag]
    assert abs(off.mean()) < 0.01 and abs(off.std() - 1.0) < 0.01
    # uniform within the band: the mean offset is near 0 and |offset|/(3*rl) near 1/2
    offs = (col.astype(np.int64) - rows)[~diag] / (3.0 * rl[rows][~diag])
    interior = (rows[~diag] > 300) & (rows[~diag] < n - 300)
    assert abs(offs[interior].mean()) < 0.01 and abs(np.abs(offs[interior]).mean() - 0.5) < 0.01


def test_fem_batch_c_sizes_match_fem_batch():
    from int_spmv_b200 import matrices as M
    mats = M.fem_batch_c(count=6, seed=4, n_lo=1e3, n_hi=3e3)
    rng = np.random.default_rng(4)
    ns = np.exp(rng.uniform(np.log(1e3), np.log(3e3), 6)).astype(np.int64)
    assert [len(r) - 1 for r, _, _ in mats] == list(ns)


def test_bench_line_is_short():
    """bench.py's printed line keeps what a reader of the run needs (value,
    config, roofline, end to end, clocks, parity, each form's time) and stays
    below 4 KB, however many formats were timed."""
    import json

    import bench
    wl = dict(name="powerlaw_n4M_seed1", row=np.zeros(4_000_001, np.int8), col=np.zeros(59_395_000, np.int8))
    row = {"ms": 0.168212345678, "gflops": 700.123456789, "gbs": 4800.123456789, "frac": 0.7432123456789,
           "kernel_ms": 0.1581234567, "kernel_frac": 0.78123456789, "kernel": "stream_wide<8,stg,b4>",
           "max_componentwise_err": 6.123456789e-16, "normwise_err": 1.23456789e-16, "aErr": 1.0, "rErr": 2.0, "pos": 7}
    out = {"metric": bench.METRIC, "value": 701.123456789, "unit": bench.UNIT, "n_gpus": 1, "steps": 20, "warmup": 5,
           "ms_per_step": 0.169123456789, "higher_is_better": True, "scaling": "weak", "vs_baseline": None,
           "dtype": "f64", "data": "synthetic: " + "x" * 200,
           "config": bench.run_config(wl, bench.format_name("COM128"), "f64", "u32", 8.1e8),
           "kernel": {"family": "wide", "name": "stream_wide<8,stg,b4>", "replicas": 1}, "gb_per_s": 4700.123456,
           "roofline": {"bound": "hbm", "achieved": 5043.123456, "peak": 6463.0, "unit": "GB/s", "frac": 0.78,
                        "traffic": {"dram_bytes": 1, "source": "x" * 80}, "kernel": "stream_wide<8,stg,b4>",
                        "kernel_ms": 0.158123456, "kernel_ms_chunks": [0.158123456789] * 5, "note": "n" * 700},
           "cpu_baseline": {"value": 31.5, "unit": bench.UNIT, "cores": 64, "kind": "reference", "sample": "s" * 160},
           "e2e": {"value": 93.1, "unit": bench.UNIT, "h2d_bytes_per_step": 32_000_000, "d2h_bytes_per_step": 32_000_000},
           "gpu_launches": 40, "clocks": {"sm_mhz": 1965.0, "sm_max_mhz": 1965.0, "reasons": [], "samples": 9},
           "parity": {"max_componentwise": 6e-16, "bound": 1e-12, "pass": True, "normwise": 1e-16},
           "formats": {f"AXT_COM_H1_HW8_BS{i}/f32lo/d16/wide": dict(row) for i in range(40)},
           "precision": {"workload": "w", "n": 1, **{f"f{i}/u32/plain-loads": dict(row) for i in range(6)}},
           "spmm": {"workload": "w", **{f"f64/k{i}": dict(row) for i in range(6)}},
           "batched": {"results": {"graph_wide": dict(row), "graph_queue": dict(row), "separate": dict(row)}},
           "conversion": {"host_s": 0.1, "gpu_s": 0.001, "note": "n" * 90, "plan": {"host_s": 1.0, "gpu_s": 0.01, "note": "n"}}}
    line = bench.headline(out)
    assert len(json.dumps(line)) < 4096
    for k in ("metric", "value", "unit", "n_gpus", "steps", "warmup", "ms_per_step", "higher_is_better", "scaling",
              "vs_baseline", "dtype", "data", "config", "roofline", "e2e", "gpu_launches", "clocks", "parity"):
        assert k in line, k
    assert line["config"] == out["config"] and line["e2e"]["h2d_bytes_per_step"] == 32_000_000
    assert abs(line["value"] / out["value"] - 1) < 1e-5 and len(line["ms"]["formats"]) == 40
    # without the extra tables (another workload, several GPUs)
    assert "ms" in bench.headline(dict(out, formats={}, precision=None, spmm=None, batched=None, conversion=None))
    assert bench.headline(dict(out, precision={"unavailable": "x"}, batched={"unavailable": "x"},
                               conversion={"unavailable": "x"}))["value"]
