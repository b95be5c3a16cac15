"""The solvers' SpMV from CSR rows and from sliced rows: the same bits for every order of sums that the
slices keep (2, 4 and 8 lanes), which of them a solver reads, and the engine that reads CSR alone on a
pattern that has slices."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS = 148 * 5 * 256


def _ragged(n, longest, seed):
    """Strictly diagonally dominant, 1 to 20 entries a row and `longest` in one."""
    rng = np.random.default_rng(seed)
    cnt = rng.integers(0, 20, n)
    cnt[n // 3] = longest
    own = np.repeat(np.arange(n), cnt)
    key = np.unique(np.concatenate([own * np.int64(n) + np.clip(own + rng.integers(-300, 301, own.size), 0, n - 1),
                                    np.arange(n, dtype=np.int64) * (n + 1)]))
    row, col = key // n, key % n
    rp = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))])
    va = rng.uniform(-1.0, 1.0, key.size) / np.diff(rp)[row]
    va[row == col] = rng.uniform(1.6, 2.4, n)
    return rp.astype(np.int32), col.astype(np.int32), va, rng.standard_normal(n)


@pytest.mark.parametrize("n,longest,sliced", [(ROWS - 1, 20, False), (ROWS, 20, True), (ROWS + 1, 26, True), (ROWS + 300, 250, False)])
@pytest.mark.parametrize("precision", [0, 1])
def test_layouts_give_the_same_bits(gpu_ctx, monkeypatch, n, longest, sliced, precision):
    from vfvchem_vfvm3d_b200 import GmresOptions, Pattern
    from vfvchem_vfvm3d_b200 import _lib as L
    rp, ci, va, b = _ragged(n, longest, n)

    def solves(lanes):
        p = Pattern.from_csr(gpu_ctx, rp, ci)
        p.set_values(va)
        p.set_spmv_lanes(lanes, lanes)
        out = []
        for precond, engine in ((L.PRECOND_NONE, 1), (L.PRECOND_JACOBI, 1), (L.PRECOND_ILU0, 2)):
            x, info = p.solve(b, None, GmresOptions(tol=1e-10, restart=20, max_outer=50, precision=precision, inner_rtol=1e-5,
                                                    precond=precond, engine=engine))
            out.append((x, info.iters))
        return out, p.solvers()[:2]

    for lanes in (2, 4, 8, 16):
        monkeypatch.delenv("VFV_SOLVER_ROWS", raising=False)
        got, kinds = solves(lanes)
        assert kinds == ((0, 3) if sliced and lanes <= 8 else (3, 0))
        if kinds == (3, 0):
            continue
        monkeypatch.setenv("VFV_SOLVER_ROWS", "csr")
        ref, kinds = solves(lanes)
        assert kinds == (3, 0)
        for (x, it), (y, jt) in zip(got, ref):
            assert it == jt and np.array_equal(x, y)


@pytest.mark.parametrize("precision", [0, 1])
def test_persistent_engine_beside_sliced_rows(gpu_ctx, precision):
    """The one-kernel engine reads CSR on a pattern whose other solvers read slices: the same result."""
    from vfvchem_vfvm3d_b200 import GmresOptions, Pattern
    rp, ci, va, b = _ragged(ROWS + 77, 20, 5)
    kw = dict(tol=1e-10, restart=20, max_outer=50, precision=precision, inner_rtol=1e-5, precond=1)
    out = []
    for slices_first in (False, True):
        p = Pattern.from_csr(gpu_ctx, rp, ci)
        p.set_values(va)
        if slices_first:
            p.solve(b, None, GmresOptions(engine=1, **kw))
            assert p.solvers()[:2] == (0, 1)
        out.append(p.solve(b, None, GmresOptions(engine=0, **kw)))
    assert out[0][1].iters == out[1][1].iters and np.array_equal(out[0][0], out[1][0])
