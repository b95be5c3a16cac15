"""The dataflow factorisation with many blocks at work: matrices with hundreds of rows per level, so
that pivots are handed over between blocks and SMs, against level-by-level launches; and values that
are not finite, among them the very bits that mark an open entry."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _chains(levels, width, low, extra, seed):
    """`width` chains of `levels` rows, row l * width + c: coupled to `low` rows of the level before, and
    every 50th row to `extra` rows of the levels before that; symmetric structure, diagonally dominant."""
    rng = np.random.default_rng(seed)
    n = levels * width
    i = np.arange(width, n)
    prev = (i // width - 1) * width
    pairs = [np.stack([i, i - width])]
    for _ in range(low - 1):
        pairs.append(np.stack([i, prev + rng.integers(0, width, i.size)]))
    some = i[(i >= 3 * width) & (i % 50 == 7)]
    for _ in range(extra):
        pairs.append(np.stack([some, rng.integers(0, 2 * width, some.size)]))
    rc = np.concatenate(pairs, 1)
    key = np.unique(np.concatenate([rc[0] * np.int64(n) + rc[1], rc[1] * np.int64(n) + rc[0], np.arange(n, dtype=np.int64) * (n + 1)]))
    row, col = key // n, key % n
    va = -rng.uniform(0.1, 1.0, key.size)
    va[row == col] = 0.0
    off = np.bincount(row, -va, minlength=n)
    va[row == col] = off + 1.0
    return np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))]).astype(np.int32), col.astype(np.int32), va


def _apply(p, va, r):
    import torch
    p.set_values(va)
    z = torch.empty_like(r)
    p.ilu0_apply_device(r.data_ptr(), z.data_ptr(), 1)
    torch.cuda.synchronize()
    return z.cpu().numpy()


# rows within the staging (16 lower entries, 24 upper, 32 in all), rows beyond it
@pytest.mark.parametrize("levels,width,low,extra", [(40, 700, 3, 0), (33, 2900, 2, 0), (300, 331, 3, 0), (40, 700, 3, 24), (120, 331, 2, 40)])
def test_blocks_hand_rows_over(gpu_ctx, monkeypatch, levels, width, low, extra):
    import torch
    from vfvchem_vfvm3d_b200 import Pattern
    from vfvchem_vfvm3d_b200 import _lib as L
    rp, ci, va = _chains(levels, width, low, extra, levels + extra)
    n = levels * width
    r = torch.tensor(np.random.default_rng(4).standard_normal(n), device="cuda")
    values = [va, 3.0 * va, va + 0.01 * np.abs(va)]
    monkeypatch.delenv("VFV_ILU_FACTOR", raising=False)
    p = Pattern.from_csr(gpu_ctx, rp, ci)
    _, lev = p.ilu0_ordering(L.ILU_NATURAL)
    assert len(lev) - 1 == levels >= 32 and np.max(np.diff(lev)) < 32768  # the dataflow kernels serve it
    # rows of six levels in flight, 8 to a block: well over one block per SM
    assert 6 * n // levels // 8 > 148
    diag = ci == np.repeat(np.arange(n), np.diff(rp))
    low_len = np.add.reduceat((ci < np.repeat(np.arange(n), np.diff(rp))).astype(int), rp[:-1])
    short = np.diff(rp).max() <= 32 and low_len.max() <= 16 and (np.diff(rp) - low_len - 1).max() <= 24
    assert diag.sum() == n and short == (extra == 0)
    flow = [_apply(p, v, r) for v in values]
    monkeypatch.setenv("VFV_ILU_FACTOR", "levels")
    q = Pattern.from_csr(gpu_ctx, rp, ci)
    for got, v in zip(flow, values):
        assert np.array_equal(got, _apply(q, v, r))


@pytest.mark.parametrize("extra", [0, 24])
def test_values_that_are_not_finite(gpu_ctx, monkeypatch, extra):
    """The factorisation ends, and the entries that are not finite are those of the level launches."""
    import torch
    from vfvchem_vfvm3d_b200 import Pattern
    rp, ci, va = _chains(40, 350, 3, extra, 5)
    n = 40 * 350
    own = np.repeat(np.arange(n), np.diff(rp))
    open_bits = np.frombuffer(b"\xff" * 8, np.float64)[0]
    r = torch.ones(n, dtype=torch.float64, device="cuda")
    spots = {"open, diagonal": ((own == ci) & (own % 4001 == 90), open_bits), "open, lower": ((own > ci) & (own % 4001 == 900), open_bits),
             "open, upper": ((own < ci) & (own % 4001 == 1700), open_bits), "nan": ((own == ci) & (own == 777), np.nan),
             "inf": ((own == ci) & (own % 4001 == 500), np.inf), "-inf, upper": ((own < ci) & (own == 2500), -np.inf)}
    for name, (where, x) in spots.items():
        assert where.any(), name
        v = va.copy()
        v[where] = x
        out = []
        for mode in ("flow", "levels"):
            if mode == "levels":
                monkeypatch.setenv("VFV_ILU_FACTOR", "levels")
            else:
                monkeypatch.delenv("VFV_ILU_FACTOR", raising=False)
            out.append(_apply(Pattern.from_csr(gpu_ctx, rp, ci), v, r))
        assert np.array_equal(np.isnan(out[0]), np.isnan(out[1])), name
        assert np.array_equal(out[0], out[1], equal_nan=True), name
