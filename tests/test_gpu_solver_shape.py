"""A solver keeps the SpMV shape that its pattern had when the solver was made: its cycle graphs, some of
them added after several solves, all sum a row in the same order."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _banded(n):
    """Nine entries a row: 2 to 32 lanes sum them in different orders."""
    rng = np.random.default_rng(n)
    cols = np.arange(n)[:, None] + np.arange(-4, 5)
    ok = (cols >= 0) & (cols < n)
    vals = rng.uniform(-1.0, 1.0, cols.shape)
    vals[:, 4] = rng.uniform(6.0, 8.0, n)
    rp = np.concatenate([[0], np.cumsum(ok.sum(1))]).astype(np.int32)
    return rp, cols[ok].astype(np.int32), vals[ok], rng.standard_normal(n)


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("lanes", [2, 8, 32])
def test_shape_set_after_the_first_solve_changes_no_result(gpu_ctx, precision, lanes):
    from vfvchem_vfvm3d_b200 import GmresOptions, Pattern
    rp, ci, va, b = _banded(5000)
    opts = GmresOptions(tol=1e-12, restart=20, max_outer=300, precond=1, precision=precision, inner_rtol=1e-6, engine=1)

    def passes(change):
        p = Pattern.from_csr(gpu_ctx, rp, ci)
        p.set_values(va)
        out = []
        for i in range(16):  # more than the six wishes after which a cycle graph is added
            if change and i == 1:
                p.set_spmv_lanes(lanes, lanes)
            x, info = p.solve(b, None, opts)
            out.append((x, info.iters))
        return out

    for (x, it), (y, jt) in zip(passes(True), passes(False)):
        assert it == jt and np.array_equal(x, y)
