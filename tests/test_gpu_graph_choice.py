"""Long and short solves in turn on one handle: a short one does not run the long one's steps as kernels
that do nothing."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

N = 5000


def _system():
    rng = np.random.default_rng(8)
    cols = np.arange(N)[:, None] + np.array([-1, 0, 1])
    ok = (cols >= 0) & (cols < N)
    rp = np.concatenate([[0], np.cumsum(ok.sum(1))]).astype(np.int32)
    vals = rng.uniform(-1.0, 1.0, cols.shape)
    vals[:, 1] = rng.uniform(2.2, 3.0, N)
    return rp, cols[ok].astype(np.int32), vals[ok], rng.standard_normal(N)


@pytest.mark.parametrize("precond", [0, 2])
def test_short_solves_between_long_ones(gpu_ctx, precond):
    from vfvchem_vfvm3d_b200 import GmresOptions, Pattern
    rp, ci, va, b = _system()

    def launches(p, tol):
        at = gpu_ctx.launch_count
        _, info = p.solve(b, None, GmresOptions(tol=tol, restart=60, max_outer=20, precond=precond, engine=1))
        assert info.status == 0
        return gpu_ctx.launch_count - at, info.iters

    p = Pattern.from_csr(gpu_ctx, rp, ci)
    p.set_values(va)
    launches(p, 0.1)
    first, short = launches(p, 0.1)  # the matrix is prepared and factored
    _, long = launches(p, 1e-12)
    assert long >= short + 8
    for _ in range(12):
        launches(p, 1e-12)
        again, its = launches(p, 0.1)
        assert its == short
        assert again <= first


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("precond,engine", [(1, 1), (2, 2)])
def test_added_graphs_are_built_and_change_nothing(gpu_ctx, monkeypatch, precond, engine, precision):
    """A steady number of steps: graphs beyond the first exist after some solves (so what is compared did
    run), and every solve has the bits of the straight graph's."""
    from vfvchem_vfvm3d_b200 import GmresOptions, Pattern
    rp, ci, va, b = _system()

    def passes():
        p = Pattern.from_csr(gpu_ctx, rp, ci)
        p.set_values(va)
        out = [p.solve(b, None, GmresOptions(tol=1e-11, restart=25, max_outer=50, precond=precond, precision=precision, inner_rtol=1e-5,
                                             engine=engine)) for _ in range(10)]
        return out, p.solvers()[2]

    monkeypatch.delenv("VFV_STRAIGHT_GRAPH", raising=False)
    got, graphs = passes()
    assert graphs > 1
    monkeypatch.setenv("VFV_STRAIGHT_GRAPH", "1")
    ref, straight = passes()
    assert straight == 1
    for (x, info), (y, other) in zip(got, ref):
        assert info.iters == other.iters and info.relres == other.relres and np.array_equal(x, y)
