"""The ESolver's Chebyshev iteration against conjugate gradients in 64 bits on
the same mass matrix: systems smaller than a warp, in registers and over both
block shapes of the other form, rows no multiple of a slice, rows of more entries
than are held, a second solve from the first one's solution."""
import numpy as np
import pytest
import scipy.sparse as sp
import scipy.sparse.linalg as spl

from puncpp_gb300 import _lib as L
from puncpp_gb300 import meshgen, punc

pytestmark = pytest.mark.gpu

# the condition number of D^-1 M is at most 5, so a relative residual t leaves
# a relative error of at most 5 t, and FP32 sums of the mixed form some 1e-6
BAR = {L.PG_FP64: 5e-12, L.PG_MIXED: 1e-5}


def reference(mesh, phi):
    rp, ci = mesh.table(L.T_CSR_ROWPTR), mesh.table(L.T_CSR_COL)
    n = len(rp) - 1
    M = sp.csr_matrix((mesh.table(L.T_MASS), ci, rp), shape=(n, n))
    dofs = mesh.table(L.T_CELL_DOFS).reshape(-1, 4)
    bary = mesh.table(L.T_BARYCENTRIC).reshape(-1, 3, 4)[:, :, 1:]
    grad = np.concatenate([bary, -bary.sum(1, keepdims=True)], axis=1)
    E = -np.einsum("ck,ckj->cj", phi[dofs], grad)
    w = 0.25 * mesh.table(L.T_VOLUME)
    out = np.zeros((n, 3))
    d = M.diagonal()
    for j in range(3):
        b = np.bincount(dofs.ravel(), np.repeat(w * E[:, j], 4), minlength=n)
        out[:, j], info = spl.cg(M, b, rtol=1e-14, atol=0.0, M=sp.diags(1.0 / d))
        assert info == 0
    return out


def fans(n):
    """A probe mesh with the cells around every 40th vertex split at their
    centroids: rows of up to 39 entries."""
    ma = meshgen.probe_box(n, 2.0, 0.9)
    split = np.isin(ma.cells, np.arange(7, ma.n_vertices, 40)).any(1)
    old = ma.cells[split]
    new = ma.n_vertices + np.arange(len(old))
    parts = []
    for k in range(4):
        part = old.copy()
        part[:, k] = new
        parts.append(part)
    coords = np.concatenate([ma.coords, ma.coords[old].mean(1)])
    return meshgen.MeshArrays(coords=coords, cells=np.concatenate([ma.cells[~split]] + parts), bfacets=ma.bfacets,
                              btags=ma.btags.copy(), vertex_to_dof=None, n_dofs=len(coords), Ld=ma.Ld,
                              origin=ma.origin, n_objects=ma.n_objects)


@pytest.mark.parametrize("prec", [L.PG_FP64, L.PG_MIXED])
@pytest.mark.parametrize("geom,n", [("periodic", 2), ("periodic", 3), ("probe", 5), ("fans", 9), ("periodic", 17),
                                    ("probe", 27), ("probe", 34), ("probe", 43)])
def test_esolver(lib, prec, geom, n):
    ma = fans(n) if geom == "fans" else meshgen.langmuir_cube(n) if geom == "periodic" else meshgen.probe_box(n, 2.0, 0.9)
    mesh = punc.Mesh(ma)
    if geom == "fans":
        assert np.diff(mesh.table(L.T_CSR_ROWPTR)).max() > 24
    pop = punc.Population(mesh, precision=prec, periodic=geom == "periodic")
    E = punc.Function(pop, "E_cg1")
    es = punc.ESolver(pop)
    rng = np.random.default_rng(n)
    phi = rng.normal(size=mesh.n_dofs)
    for scale in (1.0, 1.01, 3.0, 0.0):
        punc.Function(pop, "phi").set_local(scale * phi)
        got = es.solve(E, None)
        want = reference(mesh, scale * phi) if scale else np.zeros((mesh.n_dofs, 3))
        bar = BAR[prec] * np.linalg.norm(want) + 1e-12
        assert np.linalg.norm(got - want) <= bar
        assert es.last_info.iterations < 80
    pop.close()
