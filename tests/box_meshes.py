"""Meshes whose cells fill their bounding box, or all but a trace of it, though
walls stand inside: a plate of no thickness, an object of a billionth of the
volume, two boxes side by side; and a slender box."""
import numpy as np

from puncpp_gb300 import meshgen


def _arrays(coords, cells, tags_of, n_objects):
    bf = meshgen._boundary_facets(cells, len(coords))
    return meshgen.MeshArrays(coords=np.ascontiguousarray(coords), cells=np.ascontiguousarray(cells), bfacets=bf,
                              btags=tags_of(coords[bf]).astype(np.int32), n_dofs=len(coords),
                              Ld=tuple(np.ptp(coords, axis=0)), origin=tuple(coords.min(axis=0)),
                              n_objects=n_objects)


def _outer(fx, lo, hi):
    """Facets (coordinates [n][3][3]) in a plane of the box."""
    return np.any([np.all(fx[:, :, a] == w[a], axis=1) for a in range(3) for w in (lo, hi)], axis=0)


def plate(n=12):
    """Unit box with a plate at x = 1/2, y and z in [1/4, 3/4] (n a multiple of
    4): the vertices inside its rim are doubled, one set for the cells of
    either side, and the facets of both sides are object 2."""
    base = meshgen.kuhn_box(n, 0.0, 1.0)
    x = base.coords
    inner = (x[:, 0] == 0.5) & np.all((x[:, 1:] > 0.25) & (x[:, 1:] < 0.75), axis=1)
    twin = np.full(len(x), -1)
    twin[inner] = len(x) + np.arange(inner.sum())
    cells = base.cells.copy()
    right = x[cells].mean(axis=1)[:, 0] > 0.5
    cells[right] = np.where(twin[cells[right]] >= 0, twin[cells[right]], cells[right])
    coords = np.concatenate([x, x[inner]])
    return _arrays(coords, cells, lambda fx: np.where(_outer(fx, (0, 0, 0), (1, 1, 1)), 1, 2), 1)


def speck(n=4, size=0.005):
    """Unit box with a tetrahedral hole (object 2): one cell holds a copy of
    itself scaled by size about its centroid, and the shell between the two is
    cut into prisms over the facets, three tetrahedra each."""
    base = meshgen.kuhn_box(n, 0.0, 1.0)
    k = 6 * ((n // 2 * n + n // 2) * n + n // 2)
    outer = np.sort(base.cells[k])
    p = base.coords[outer]
    inner = len(base.coords) + np.arange(4)
    shell = []
    for f in range(4):
        a, b, c = np.delete(np.arange(4), f)
        shell += [(outer[a], outer[b], outer[c], inner[c]), (outer[a], outer[b], inner[b], inner[c]),
                  (outer[a], inner[a], inner[b], inner[c])]
    coords = np.concatenate([base.coords, p.mean(axis=0) + size * (p - p.mean(axis=0))])
    cells = np.concatenate([np.delete(base.cells, k, axis=0), np.array(shell, np.int64)])
    return _arrays(coords, cells, lambda fx: np.where(_outer(fx, (0, 0, 0), (1, 1, 1)), 1, 2), 1), p.mean(axis=0)


def side_by_side(n=6):
    """Two unit boxes that touch at x = 1 and share no vertex; all facets tag 1."""
    a, b = meshgen.kuhn_box(n, 0.0, 1.0), meshgen.kuhn_box(n, 0.0, 1.0)
    coords = np.concatenate([a.coords, b.coords + [1.0, 0.0, 0.0]])
    cells = np.concatenate([a.cells, b.cells + a.n_vertices])
    return _arrays(coords, cells, lambda fx: np.ones(len(fx)), 0), a.n_cells


def slender(n):
    """Box of 1 x 1 x n unit cubes."""
    corner = np.array([[i, j, k] for i in (0, 1) for j in (0, 1) for k in (0, 1)])
    cube = meshgen._kuhn_cells(1)
    ids = np.empty((n, 8), np.int64)
    for v, (i, j, k) in enumerate(corner):
        ids[:, v] = 4 * (np.arange(n) + k) + 2 * i + j
    z = np.repeat(np.arange(n + 1), 4)
    coords = np.stack([np.tile([0, 0, 1, 1], n + 1), np.tile([0, 1, 0, 1], n + 1), z], axis=1).astype(float)
    return _arrays(coords, ids[:, cube].reshape(-1, 4), lambda fx: np.ones(len(fx)), 0)
