"""The AMG-PCG solve against a direct solve on hierarchies of one level (the
dense inverse), two and three, operators in natural and random order, systems
of one block, of a cluster (up to 12,288 rows) and of a grid, row counts that are
no multiple of a slice."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spl

from puncpp_gb300 import _lib as L
from puncpp_gb300 import meshgen, punc

pytestmark = pytest.mark.gpu


def matrices(mesh):
    rp, ci = mesh.table(L.T_CSR_ROWPTR), mesh.table(L.T_CSR_COL)
    n = len(rp) - 1
    return tuple(sp.csr_matrix((mesh.table(t), ci, rp), shape=(n, n)) for t in (L.T_STIFFNESS, L.T_MASS))


def renumbered(ma, rng):
    perm = rng.permutation(ma.n_vertices)
    coords = np.empty_like(ma.coords)
    coords[perm] = ma.coords
    return meshgen.MeshArrays(coords=coords, cells=perm[ma.cells], bfacets=perm[ma.bfacets], btags=ma.btags.copy(),
                              vertex_to_dof=None, n_dofs=ma.n_dofs, Ld=ma.Ld, origin=ma.origin,
                              n_objects=ma.n_objects)


@pytest.mark.parametrize("order", ["natural", "random"])
@pytest.mark.parametrize("n", [3, 5, 7, 8, 13, 22])
def test_probe_solve(lib, n, order):
    """Dirichlet problem; the residual test is rtol 1e-12 and the smallest
    eigenvalue of the reduced matrix over its largest is above 1e-3 / n, so phi
    is within 1e-9."""
    rng = np.random.default_rng(n)
    ma = meshgen.probe_box(n, 2.0, 0.9)
    if order == "random":
        ma = renumbered(ma, rng)
    mesh = punc.Mesh(ma)
    K, M = matrices(mesh)
    kind = mesh.table(L.T_BC_KIND)
    pop = punc.Population(mesh, warm_start=0)
    rho = rng.normal(size=mesh.n_dofs)
    punc.Function(pop, "rho").set_local(rho)
    solver = punc.PoissonSolver(pop)
    phi = solver.solve(punc.Function(pop, "phi"), None, [punc.Object(2, potential=-1.5)])
    free = np.nonzero(kind < 0)[0]
    want = np.where(kind == 1, -1.5, 0.0)
    b = (M @ rho - K @ want)[free]
    want[free] = spl.spsolve(K[free][:, free].tocsc(), b)
    assert np.abs(phi - want).max() <= 1e-9 * np.abs(want).max()
    assert solver.last_info.residual <= 1e-12 * solver.last_info.rhs_norm * 1.0001
    again = solver.solve(punc.Function(pop, "phi"), None, [punc.Object(2, potential=-1.5)])
    assert np.array_equal(again, phi)
    pop.close()


@pytest.mark.parametrize("n,order", [(24, "natural"), (34, "natural"), (40, "random"), (42, "natural"),
                                     (54, "natural")])
def test_grid_solve(lib, n, order):
    """The grid's forms: two blocks per 512 rows (15k rows), one block per SM
    (42k; 69k in random order, whose columns span more than 16 bits), one per 512
    rows (79k), more rows than threads (166k), against
    a CG of the host at a residual of 1e-13, with the bound of test_probe_solve."""
    rng = np.random.default_rng(n)
    ma = meshgen.probe_box(n, 2.0, 0.9)
    if order == "random":
        ma = renumbered(ma, rng)
    mesh = punc.Mesh(ma)
    K, M = matrices(mesh)
    kind = mesh.table(L.T_BC_KIND)
    pop = punc.Population(mesh, warm_start=0)
    rho = rng.normal(size=mesh.n_dofs)
    punc.Function(pop, "rho").set_local(rho)
    solver = punc.PoissonSolver(pop)
    phi = solver.solve(punc.Function(pop, "phi"), None, [punc.Object(2, potential=-1.5)])
    free = np.nonzero(kind < 0)[0]
    want = np.where(kind == 1, -1.5, 0.0)
    b = (M @ rho - K @ want)[free]
    A = K[free][:, free]
    want[free], status = spl.cg(A, b, rtol=1e-13, atol=0.0, maxiter=5000, M=sp.diags(1.0 / A.diagonal()))
    assert status == 0
    assert np.abs(phi - want).max() <= 1e-9 * np.abs(want).max()
    assert solver.last_info.residual <= 1e-12 * solver.last_info.rhs_norm * 1.0001
    again = solver.solve(punc.Function(pop, "phi"), None, [punc.Object(2, potential=-1.5)])
    assert np.array_equal(again, phi)
    pop.close()


@pytest.mark.parametrize("n", [3, 6, 8, 11, 16, 23])
def test_periodic_solve(lib, n):
    """Pure Neumann problem on the torus, mean zero."""
    rng = np.random.default_rng(n)
    mesh = punc.Mesh(meshgen.langmuir_cube(n))
    K, M = matrices(mesh)
    pop = punc.Population(mesh, periodic=True, warm_start=0)
    rho = rng.normal(size=mesh.n_dofs)
    punc.Function(pop, "rho").set_local(rho)
    phi = punc.PoissonSolver(pop).solve(punc.Function(pop, "phi"), None, [])
    b = M @ rho
    b -= b.mean()
    want = np.zeros(mesh.n_dofs)
    want[1:] = spl.spsolve(K[1:, 1:].tocsc(), b[1:])
    want -= want.mean()
    assert np.abs(phi - want).max() <= 1e-9 * np.abs(want).max()
    pop.close()
