"""A mesh in a batch iterates with the bits of the same mesh solved alone: batches whose size, largest
mesh or row offsets would choose other shapes of the vector kernels than the mesh alone."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def cubes(lib_built):
    from vfvchem_vfvm3d_b200 import Mesh
    return {n: Mesh.jitter_cube(n, 70 + n) for n in (3, 4, 5, 13, 17, 20, 28, 45)}


# edge lengths of the meshes: off every alignment; a mesh that folds its sums beside one that does not
# (45^3 rows: 178 blocks of 512, 89 of 1,024); enough rows for the middle and for the wide shape
BATCHES = [(3, 5, 4, 13), (5, 28, 17), (17, 45, 20), (3,) + (28, 17, 20) * 3, (5,) + (28, 17, 20, 28) * 8, (3,) + (28, 17, 20, 28) * 15]


@pytest.mark.parametrize("edges", BATCHES, ids=lambda e: f"{len(e)}x{max(e)}")
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("sweeps", [0, 3])
def test_bits_do_not_depend_on_the_batch(gpu_ctx, cubes, edges, precision, sweeps):
    from vfvchem_vfvm3d_b200 import GmresOptions, TransientTransportGpu
    from vfvchem_vfvm3d_b200 import _lib as L
    from vfvchem_vfvm3d_b200.problems import transport_fields
    meshes = [cubes[e] for e in edges]
    vel, c0 = transport_fields(meshes)
    opts = GmresOptions(tol=1e-10, restart=20, max_outer=100, precond=L.PRECOND_ILU0, precision=precision, inner_rtol=1e-6,
                        ilu_order=L.ILU_NATURAL if sweeps else L.ILU_MULTICOLOR, ilu_sweeps=sweeps)
    batch = TransientTransportGpu(meshes, 1e-2, ctx=gpu_ctx)
    batch.assemble(1e-3, vel)
    c, _ = batch.run(c0, 2, opts)
    at = np.concatenate([[0], np.cumsum([m.n_tot for m in meshes])])
    for i in sorted({0, 1, 2, 3, len(meshes) - 1} & set(range(len(meshes)))):
        rows = slice(at[i], at[i + 1])
        one = TransientTransportGpu([meshes[i]], 1e-2, ctx=gpu_ctx)
        one.assemble(1e-3, vel[:, rows])
        c1, _ = one.run(c0[rows], 2, opts)
        assert np.array_equal(c[rows], c1)
