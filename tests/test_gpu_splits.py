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
