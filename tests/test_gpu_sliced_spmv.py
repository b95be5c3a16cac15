"""The solvers' SpMV over sliced rows: row counts around the rule's 148 * 5 * 256, ragged slices and a
row that is too long for the layout, each engine's preconditioners that read it, against a known
solution; a batch that reads it against each mesh alone (CSR)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ROWS = 148 * 5 * 256


def _ragged(n, long, seed):
    """Strictly diagonally dominant (condition below 4), 1 to 12 entries per row; `long` entries in one."""
    rng = np.random.default_rng(seed)
    cnt = rng.integers(0, 12, n)
    cnt[rng.integers(0, n, 1)] = long
    own = np.repeat(np.arange(n), cnt)
    key = np.unique(np.concatenate([own * np.int64(n) + np.clip(own + rng.integers(-300, 301, own.size), 0, n - 1),
                                    np.arange(n, dtype=np.int64) * (n + 1)]))
    row, col = key // n, key % n
    rp = np.concatenate([[0], np.cumsum(np.bincount(row, minlength=n))])
    va = rng.uniform(-1.0, 1.0, key.size) / np.diff(rp)[row]
    va[row == col] = rng.uniform(1.6, 2.4, n)
    x = rng.standard_normal(n)
    b = np.bincount(row, va * x[col], minlength=n)
    return rp.astype(np.int32), col.astype(np.int32), va, x, b


@pytest.mark.parametrize("n,long", [(ROWS - 1, 12), (ROWS, 12), (ROWS + 1, 24), (ROWS + 255, 40), (ROWS + 257, 200), (300007, 12)])
@pytest.mark.parametrize("precision", [0, 1])
def test_solves_match_known_solution(gpu_ctx, n, long, precision):
    from vfvchem_vfvm3d_b200 import GmresOptions, Pattern
    from vfvchem_vfvm3d_b200 import _lib as L
    rp, ci, va, x, b = _ragged(n, long, n)
    p = Pattern.from_csr(gpu_ctx, rp, ci)
    for scale in (1.0, 2.0):  # the second pass: new values on the same solver
        p.set_values(scale * va)
        for precond, engine in ((L.PRECOND_JACOBI, 1), (L.PRECOND_ILU0, 1), (L.PRECOND_ILU0, 2)):
            got, info = p.solve(scale * b, None, GmresOptions(tol=1e-12, restart=30, max_outer=50, precision=precision, inner_rtol=1e-5,
                                                              precond=precond, engine=engine))
            assert info.status == 0
            # ||x - x*|| <= cond * tol * ||x||, cond < 12: row sums of |off-diagonal| below 1, diagonal above 1.6,
            # columns below 12 / 2 entries of at most 1 / 2
            assert np.linalg.norm(got - x) <= 1.2e-11 * np.linalg.norm(x)


@pytest.mark.parametrize("precision", [0, 1])
def test_batch_equals_alone(gpu_ctx, precision):
    """185,193 + 4,913 + 27 rows: sliced together, with meshes inside a window; CSR alone."""
    from vfvchem_vfvm3d_b200 import GmresOptions, Mesh, TransientTransportGpu
    from vfvchem_vfvm3d_b200 import _lib as L
    from vfvchem_vfvm3d_b200.problems import transport_fields
    meshes = [Mesh.jitter_cube(n, 50 + n) for n in (3, 57, 17)]
    vel, c0 = transport_fields(meshes)
    opts = GmresOptions(tol=1e-12, restart=20, max_outer=100, precond=L.PRECOND_ILU0, precision=precision, inner_rtol=1e-6,
                        ilu_order=L.ILU_NATURAL, ilu_sweeps=2)
    batch = TransientTransportGpu(meshes, 1e-2, ctx=gpu_ctx)
    batch.assemble(1e-3, vel)
    c, _ = batch.run(c0, 2, opts)
    at = np.concatenate([[0], np.cumsum([m.n_tot for m in meshes])])
    for i, m in enumerate(meshes):
        rows = slice(at[i], at[i + 1])
        one = TransientTransportGpu([m], 1e-2, ctx=gpu_ctx)
        one.assemble(1e-3, vel[:, rows])
        c1, _ = one.run(c0[rows], 2, opts)
        # both meet relres 1e-12 in two well-conditioned steps
        assert np.linalg.norm(c[rows] - c1) <= 1e-11 * np.linalg.norm(c1)
