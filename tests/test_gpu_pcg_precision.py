"""The AMG-PCG solve's FP64 parts: the step lengths, and the residual that it
stops at on graded meshes and for sources of small and large units."""
import dataclasses

import numpy as np
import pytest
import scipy.sparse as sp

from puncpp_gb300 import _lib as L
from puncpp_gb300 import meshgen, punc

pytestmark = pytest.mark.gpu


def operators(mesh, potential):
    rp, ci = mesh.table(L.T_CSR_ROWPTR), mesh.table(L.T_CSR_COL)
    n = len(rp) - 1
    K, M = (sp.csr_matrix((mesh.table(t), ci, rp), shape=(n, n)) for t in (L.T_STIFFNESS, L.T_MASS))
    kind = mesh.table(L.T_BC_KIND)
    return K, M, np.nonzero(kind < 0)[0], np.where(kind == 1, potential, 0.0)


@pytest.mark.parametrize("n", [4, 8, 16, 27])   # one, two and three levels, a cluster and a grid
def test_step_length_is_fp64(lib, n):
    """After one step from zero x = alpha p with p of 24 bits: an alpha of 24
    bits gives products of at most 48, whose last five bits are zero."""
    mesh = punc.Mesh(meshgen.probe_box(n, 2.0, 0.9))
    _, _, free, _ = operators(mesh, 0.0)
    pop = punc.Population(mesh, warm_start=0, pcg_max_iter=1)
    punc.Function(pop, "rho").set_local(np.random.default_rng(n).normal(size=mesh.n_dofs))
    phi = punc.Function(pop, "phi")
    try:
        punc.PoissonSolver(pop).solve(phi, None, [punc.Object(2)])
    except L.PgError as e:
        assert e.code == 6
    x = phi.vector()[free]
    x = x[x != 0.0]
    assert len(x) > 0.9 * len(free)
    assert (x.view(np.uint64) & 31 != 0).mean() > 0.9   # 31 of 32 expected
    pop.close()


def graded(n, power):
    """A probe box whose cells shrink towards one corner."""
    ma = meshgen.probe_box(n, 2.0, 0.9)
    return dataclasses.replace(ma, coords=np.ascontiguousarray(4.0 * ((ma.coords + 2.0) / 4.0) ** power))


@pytest.mark.parametrize("n,power", [(6, 2.0), (12, 1.5), (12, 2.0), (20, 1.5), (27, 1.5), (42, 1.25)])
@pytest.mark.parametrize("units", [1e-4, 1.0, 1e10])
def test_residual_on_graded_meshes(lib, n, power, units):
    """||b - K phi|| <= 1e-12 ||b|| on the rows without a boundary value, with the
    host's rounding of K phi (at most 2^-50 of its terms)."""
    mesh = punc.Mesh(graded(n, power))
    K, M, free, g = operators(mesh, -1.5 * units)
    pop = punc.Population(mesh, warm_start=0, pcg_atol=1e-30)
    rho = units * np.random.default_rng(n).normal(size=mesh.n_dofs)
    punc.Function(pop, "rho").set_local(rho)
    solver = punc.PoissonSolver(pop)
    phi = solver.solve(punc.Function(pop, "phi"), None, [punc.Object(2, potential=-1.5 * units)])
    b = M @ rho - K @ g
    r = (M @ rho - K @ phi)[free]
    b[np.setdiff1d(np.arange(len(b)), free)] = g[np.setdiff1d(np.arange(len(b)), free)]
    rounding = 2.0 ** -50 * np.linalg.norm((abs(K) @ abs(phi) + abs(M) @ abs(rho))[free])
    assert np.linalg.norm(r) <= 1e-12 * np.linalg.norm(b) * (1 + 1e-9) + rounding
    assert solver.last_info.residual <= 1e-12 * solver.last_info.rhs_norm * (1 + 1e-9)
    assert abs(solver.last_info.rhs_norm - np.linalg.norm(b)) <= 1e-9 * np.linalg.norm(b)
    pop.close()
