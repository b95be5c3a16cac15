"""Rows of the coupled flow system at the edges of the assembly kernels: vertices with more neighbours
than a warp has lanes, rows longer than the shared-memory buffer (1,152 entries), grad_coeff lists
of more than three entries per lane, 32-bit places; against the oracle's triplet sums."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _hub_problem(points, grid):
    """A cube whose surface is a jittered grid and whose interior is one vertex inside a shell of
    `points` others: the hub neighbours all of them, and every row reaches most of the mesh."""
    from vfvchem_vfvm3d_b200 import Mesh
    from vfvchem_vfvm3d_b200.problems import FlowProblem
    base = Mesh.jitter_cube(grid, 42, 0.25)
    pos, nb, _ = base.export()
    rng = np.random.default_rng(points)
    d = rng.standard_normal((points, 3))
    shell = 0.5 + 0.3 * d / np.linalg.norm(d, axis=1, keepdims=True)
    mesh = Mesh.from_vertices(np.concatenate([[[0.5, 0.5, 0.5]], shell, pos[base.n_pts:]]), points + 1, nb)
    n = mesh.n_tot
    node_bnd = np.full(n, -1, np.int32)
    node_bnd[mesh.n_pts:] = nb
    bc = np.zeros((3, n))
    bc[0, node_bnd == 5] = 1.0
    rho, mu = rng.uniform(0.8, 1.2, n), rng.uniform(0.01, 0.02, n)
    fce = 0.1 * rng.standard_normal((3, n))
    return FlowProblem(mesh, rho, mu, fce, bc, node_bnd, mesh.n_pts + 3, 0.25)


@pytest.mark.parametrize("points,grid,wide", [(3, 3, 0), (20, 4, 0), (40, 5, 0), (70, 9, 0), (130, 10, 0), (40, 5, 1), (130, 10, 1)])
def test_flow_rows_match_oracle(gpu_ctx, monkeypatch, points, grid, wide):
    from vfvchem_vfvm3d_b200 import SteadyFlowGpu
    monkeypatch.setenv("VFV_NS_WIDE", str(wide))
    prob = _hub_problem(points, grid)
    n = prob.n
    flow = SteadyFlowGpu(prob, ctx=gpu_ctx)
    rng = np.random.default_rng(5)
    x = rng.standard_normal(4 * n)
    geom = oracle.NsGeom(prob.mesh.dual(), prob.mesh.n_pts)
    r, c, v, b_o = geom.triplets(prob.node_bnd, prob.bnd_order, prob.bc_vel, prob.pref_vid, prob.pref, x[:3 * n].reshape(3, n), x[3 * n:],
                                 prob.rho, prob.mu, prob.fce)
    rp, ci, va = oracle.csr_from_triplets(4 * n, r, c, v)
    # |entry - oracle| <= eps * (triplets of the entry) * (largest triplet), below 1e-12 of it
    scale = np.max(np.abs(v))
    b = flow.assemble(x)
    grp, gci, gva = flow.pattern.export()
    assert np.array_equal(grp.astype(np.int64), rp) and np.array_equal(gci, ci)
    assert np.max(np.abs(gva - va)) <= 1e-12 * scale
    assert np.max(np.abs(b - b_o)) <= 1e-12 * max(np.max(np.abs(b_o)), scale)
    assert flow.ntrip == r.size
