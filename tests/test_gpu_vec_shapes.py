"""The multi-vector kernels' shapes (rows, dtypes, restart lengths at the edges of their tiles and of
the rules that choose them), through whole solves of banded systems with a known solution, and the
batched kernels on meshes that start off a 16-byte boundary against each mesh solved alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _banded(n, seed):
    """Pentadiagonal, strictly diagonally dominant (condition below 4): CSR, solution, right-hand side."""
    rng = np.random.default_rng(seed)
    offs = [o for o in (-2, -1, 0, 1, 2) if abs(o) < n]
    i = np.arange(n)[:, None]
    cols = i + np.array(offs)
    ok = (cols >= 0) & (cols < n)
    vals = rng.uniform(-0.25, 0.25, cols.shape)
    vals[:, offs.index(0)] = rng.uniform(1.6, 2.4, n)
    x = rng.standard_normal(n)
    b = np.where(ok, vals * x[np.clip(cols, 0, n - 1)], 0.0).sum(1)
    rp = np.concatenate([[0], np.cumsum(ok.sum(1))]).astype(np.int32)
    return rp, cols[ok].astype(np.int32), vals[ok], x, b


# 256 threads of 2 doubles or 4 floats a block: one row, ragged chunks, block edges, the small / mid
# rule at 150 blocks, the folded sums' limit of 128 blocks of a quarter's rows, the wide rule at 800
SIZES = [1, 2, 3, 5, 127, 513, 1025, 128 * 128, 128 * 128 + 1, 150 * 512 - 1, 150 * 512 + 1, 150 * 1024 - 512, 800 * 512 + 3, 800 * 1024 + 1]


@pytest.mark.parametrize("n", SIZES)
@pytest.mark.parametrize("precision", [0, 1])
def test_solves_at_the_edges_of_the_shapes(gpu_ctx, n, precision):
    from vfvchem_vfvm3d_b200 import GmresOptions, Pattern
    from vfvchem_vfvm3d_b200 import _lib as L
    rp, ci, va, x, b = _banded(n, n)
    p = Pattern.from_csr(gpu_ctx, rp, ci)
    p.set_values(va)
    for ortho in (L.ORTHO_CGS2, L.ORTHO_DGKS, L.ORTHO_CGS):
        got, info = p.solve(b, None, GmresOptions(tol=1e-12, restart=min(40, max(1, n)), max_outer=50, precision=precision, inner_rtol=1e-5,
                                                  ortho=ortho))
        assert info.status == 0
        # ||x - x*|| <= cond * tol * ||x||, cond < 4
        assert np.linalg.norm(got - x) <= 4e-12 * np.linalg.norm(x)


@pytest.mark.parametrize("restart", [1, 2, 31, 32, 33, 64, 127])
@pytest.mark.parametrize("precond", [0, 2])
def test_hessenberg_column_and_back_substitution(gpu_ctx, restart, precond):
    """Restart lengths around a warp's 32 unknowns per register; a matrix that takes many steps."""
    from vfvchem_vfvm3d_b200 import GmresOptions, Pattern
    n = 4000
    rp, ci, va, x, b = _banded(n, 3)
    rng = np.random.default_rng(1)
    scale = np.exp(rng.uniform(-1.0, 1.0, n))  # rows scaled: the same solution, slower convergence
    va, b = va * np.repeat(scale, np.diff(rp)), b * scale
    p = Pattern.from_csr(gpu_ctx, rp, ci)
    p.set_values(va)
    for engine in ((1,) if precond == 0 else (1, 2)):
        got, info = p.solve(b, None, GmresOptions(tol=1e-12, restart=restart, max_outer=2000, precond=precond, engine=engine))
        assert info.status == 0
        # condition of the scaled matrix below 4 e^2
        assert np.linalg.norm(got - x) <= 4 * np.e ** 2 * 1e-12 * np.linalg.norm(x) * np.e


@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("sweeps", [0, 2])
def test_batch_off_alignment_equals_alone(gpu_ctx, precision, sweeps):
    """27, 125, 64 and 2,197 rows: meshes that start at rows 27, 152 and 216."""
    from vfvchem_vfvm3d_b200 import GmresOptions, Mesh, TransientTransportGpu
    from vfvchem_vfvm3d_b200 import _lib as L
    from vfvchem_vfvm3d_b200.problems import transport_fields
    meshes = [Mesh.jitter_cube(n, 50 + n) for n in (3, 5, 4, 13)]
    vel, c0 = transport_fields(meshes)
    opts = GmresOptions(tol=1e-12, restart=20, max_outer=100, precond=L.PRECOND_ILU0, precision=precision, inner_rtol=1e-6,
                        ilu_order=L.ILU_NATURAL, ilu_sweeps=sweeps)
    batch = TransientTransportGpu(meshes, 1e-2, ctx=gpu_ctx)
    batch.assemble(1e-3, vel)
    c, _ = batch.run(c0, 3, opts)
    at = np.concatenate([[0], np.cumsum([m.n_tot for m in meshes])])
    for i, m in enumerate(meshes):
        rows = slice(at[i], at[i + 1])
        one = TransientTransportGpu([m], 1e-2, ctx=gpu_ctx)
        one.assemble(1e-3, vel[:, rows])
        c1, _ = one.run(c0[rows], 3, opts)
        # both meet relres 1e-12 in three well-conditioned steps
        assert np.linalg.norm(c[rows] - c1) <= 1e-11 * np.linalg.norm(c1)
