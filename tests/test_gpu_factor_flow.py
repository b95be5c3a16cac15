"""The dataflow factorisation (pivot values as their own flags) against level-by-level launches, bit by
bit: rows up to the staging's limits (16 lower entries, 24 upper ones, 32 in all) and one beyond, few
and many rows in flight, repeated with new values, a zero pivot."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(n, low, up, seed):
    """Tridiagonal (one level per row in natural order) plus rows coupled to the `low` before them, and
    rows coupled to the `up` after them; symmetric structure, diagonally dominant."""
    rng = np.random.default_rng(seed)
    pairs = {(i, i - 1) for i in range(1, n)}
    for i in range(low, n, 61):
        pairs.update((i, j) for j in range(i - low, i))
    for i in range(30, n - up, 67):
        pairs.update((j, i) for j in range(i + 1, i + 1 + up))
    pairs |= {(j, i) for i, j in pairs} | {(i, i) for i in range(n)}
    rc = np.array(sorted(pairs))
    va = -rng.uniform(0.1, 1.0, len(rc))
    diag = rc[:, 0] == rc[:, 1]
    va[diag] = 0.0
    off = np.bincount(rc[:, 0], -va, minlength=n)
    va[diag] = off + 1.0
    return np.concatenate([[0], np.cumsum(np.bincount(rc[:, 0], minlength=n))]).astype(np.int32), rc[:, 1].astype(np.int32), va


def _applies(gpu_ctx, rp, ci, values, r):
    import torch
    from vfvchem_vfvm3d_b200 import Pattern
    p = Pattern.from_csr(gpu_ctx, rp, ci)
    out = []
    for va in values:
        p.set_values(va)
        z = torch.empty_like(r)
        p.ilu0_apply_device(r.data_ptr(), z.data_ptr(), 1)
        torch.cuda.synchronize()
        out.append(z)
    return out


@pytest.mark.parametrize("n,low,up", [(33, 1, 1), (257, 15, 3), (900, 16, 14), (900, 8, 23), (900, 8, 24), (900, 17, 4), (900, 4, 25), (1300, 16, 15)])
def test_values_as_flags_match_levels(gpu_ctx, monkeypatch, n, low, up):
    import torch
    rp, ci, va = _system(n, low, up, n + low)
    r = torch.tensor(np.random.default_rng(4).standard_normal(n), device="cuda")
    values = [va, 3.0 * va, va + 0.01 * np.abs(va), va]
    monkeypatch.delenv("VFV_ILU_FACTOR", raising=False)
    flow = _applies(gpu_ctx, rp, ci, values, r)
    monkeypatch.setenv("VFV_ILU_FACTOR", "levels")
    for a, b in zip(flow, _applies(gpu_ctx, rp, ci, values, r)):
        assert torch.equal(a, b)


def test_zero_pivot_is_reported(gpu_ctx, monkeypatch):
    """A zero pivot in the middle of the chain ends in the same error, and the next values factor."""
    import torch
    from vfvchem_vfvm3d_b200 import LinearGmresNonFinite, Pattern
    rp, ci, va = _system(400, 6, 6, 1)
    own = np.repeat(np.arange(400), np.diff(rp))
    bad = np.where((own != ci) & ((own == 200) | (ci == 200)), 0.0, va)
    bad[(own == 200) & (ci == 200)] = 0.0
    r = torch.ones(400, dtype=torch.float64, device="cuda")
    for levels in (False, True):
        if levels:
            monkeypatch.setenv("VFV_ILU_FACTOR", "levels")
        else:
            monkeypatch.delenv("VFV_ILU_FACTOR", raising=False)
        p = Pattern.from_csr(gpu_ctx, rp, ci)
        z = torch.empty_like(r)
        p.set_values(bad)
        with pytest.raises(LinearGmresNonFinite):
            p.ilu0_apply_device(r.data_ptr(), z.data_ptr(), 1)
        p.set_values(va)
        p.ilu0_apply_device(r.data_ptr(), z.data_ptr(), 1)
        torch.cuda.synchronize()
        assert torch.isfinite(z).all()
