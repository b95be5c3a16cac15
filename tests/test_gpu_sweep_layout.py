"""The sliced layout of the swept ILU(0) factors: row counts around a slice (32) and a window (256),
rows longer than their slice's width (kept in the tail), empty triangles; double, float and
half-value sweeps against the oracle's on the same factor."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _system(n, dense, seed):
    """A diagonally dominant random band plus, in `dense` of the rows, entries all over the row."""
    rng = np.random.default_rng(seed)
    rows = [np.unique(np.clip(np.concatenate([[i], i + rng.integers(-6, 7, rng.integers(0, 9))]), 0, n - 1)) for i in range(n)]
    for i in rng.choice(n, min(dense, n), replace=False):
        rows[i] = np.unique(np.concatenate([[i], rng.integers(0, n, n // 2)]))
    rp = np.concatenate([[0], np.cumsum([r.size for r in rows])]).astype(np.int64)
    ci = np.concatenate(rows).astype(np.int32)
    va = rng.uniform(-1.0, 1.0, ci.size)
    own = np.repeat(np.arange(n), np.diff(rp))
    va /= np.diff(rp)[own]
    va[own == ci] = 2.0
    return rp, ci, va


def _rel(a, b):
    return np.max(np.abs(a - b)) / np.max(np.abs(b))


@pytest.mark.parametrize("n,dense", [(1, 0), (31, 0), (32, 1), (33, 0), (255, 3), (256, 0), (257, 1), (1000, 0), (1000, 2), (3001, 40)])
@pytest.mark.parametrize("order", [0, 1])
def test_sweeps_match_oracle(gpu_ctx, n, dense, order):
    import torch
    from vfvchem_vfvm3d_b200 import Pattern
    rp, ci, va = _system(n, dense, n + dense)
    p = Pattern.from_csr(gpu_ctx, rp.astype(np.int32), ci)
    p.set_values(va)
    perm = p.ilu0_ordering(0)[0] if order == 0 else np.arange(n, dtype=np.int32)
    ilu = oracle.Ilu0(rp, ci, va, perm)
    r = np.random.default_rng(1).standard_normal(n)
    rd = torch.tensor(r, device="cuda")
    zd = torch.empty_like(rd)
    p.ilu0_sweep_apply_device(rd.data_ptr(), zd.data_ptr(), 3, order)
    rf = rd.float()
    zf, zh = torch.empty_like(rf), torch.empty_like(rf)
    p.ilu0_sweep_apply_device(rf.data_ptr(), zf.data_ptr(), 3, order, f32=True)
    p.ilu0_sweep_apply_device(rf.data_ptr(), zh.data_ptr(), 3, order, half=True)
    gpu_ctx.synchronize()
    r32 = rf.cpu().numpy().astype(np.float64)
    # the bars of the other sweep tests: 1e-12 in double, 1e-5 in float
    assert _rel(zd.cpu().numpy(), ilu.sweep_apply(r, 3)) <= 1e-12
    assert _rel(zf.cpu().numpy().astype(np.float64), ilu.sweep_apply(r32, 3)) <= 1e-5
    assert _rel(zh.cpu().numpy().astype(np.float64), ilu.sweep_apply(r32, 3, half=True)) <= 1e-5
