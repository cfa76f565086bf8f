"""The walk of both particle forms for points up to 1e21 boxes away, where the
rounding of the FP64 tables themselves decides, against relocate_fast's FP64 plane
tests restated on the mesh's tables."""
import dataclasses

import numpy as np
import pytest

from helpers import sort_by_id
from puncpp_gb300 import _lib as L
from puncpp_gb300 import meshgen, punc

pytestmark = pytest.mark.gpu


def walk(mesh, x, cell):
    """relocate_fast (punc/include/punc/population.h:539-569) of all points."""
    P = mesh.table(L.T_PLANES).reshape(-1, 4, 4)
    nbr = mesh.table(L.T_NEIGHBOURS).reshape(-1, 4)
    cell = cell.copy()
    for _ in range(1000):
        on = np.nonzero(cell >= 0)[0]
        p = P[cell[on]]
        v = p[..., 0] + p[..., 1] * x[on, None, 0]
        v = v + p[..., 2] * x[on, None, 1]
        v = v + p[..., 3] * x[on, None, 2]
        out = (v > 0).any(axis=1)
        if not out.any():
            return cell
        cell[on[out]] = nbr[cell[on[out]], np.argmax(v[out] > 0, axis=1)]
    raise AssertionError("a walk does not end")


@pytest.mark.parametrize("prec", [L.PG_FP64, L.PG_MIXED])
@pytest.mark.parametrize("n,noise,shift", [(2, 1e-16, 0.0), (5, 1e-16, 0.37), (5, 1e-15, 1.3)])
def test_points_far_outside(lib, prec, n, noise, shift):
    rng = np.random.default_rng(3)
    base = meshgen.kuhn_box(n, 0.0, 1.0)
    # a tag for each side of the box: which one a walk leaves through is decided
    # by the facets on its way
    c = base.coords[base.bfacets].mean(axis=1)
    side = np.argmin(np.concatenate([c, 1.0 - c], axis=1), axis=1)
    ma = dataclasses.replace(base, coords=base.coords + shift + noise * rng.integers(-2, 3, base.coords.shape),
                             btags=(1 + side).astype(np.int32), n_objects=5)
    mesh = punc.Mesh(ma)
    k = np.repeat(np.arange(4, 22), 4000)
    cell = rng.integers(0, ma.n_cells, len(k))
    w = rng.dirichlet(np.ones(4), len(k))
    x = np.einsum("nk,nkj->nj", w, ma.coords[ma.cells[cell]])
    v = np.zeros_like(x)
    v[np.arange(len(k)), rng.integers(0, 3, len(k))] = 10.0 ** k * rng.choice([-1.0, 1.0], len(k)) * rng.random(len(k))
    pop = punc.Population(mesh, precision=prec)
    assert pop.add_particles(x, v, -1.0, 1.0) == len(x)
    before = sort_by_id(pop.particles())
    punc.move(pop, 1.0)
    moved = sort_by_id(pop.particles())
    want = walk(mesh, moved["x"], before["cell"])
    assert np.array_equal(pop.relocate(moved["x"], before["cell"]), want)
    pop.update([punc.Object(t) for t in range(2, 7)], 1.0)
    after = sort_by_id(pop.particles())
    assert np.array_equal(after["id"], before["id"][want >= 0])
    assert np.array_equal(after["cell"], want[want >= 0])
    counts, _, _ = punc.absorbed_counts(pop)
    assert np.array_equal(counts[1:, 0], np.bincount(-want[want < 0], minlength=7)[1:])
    pop.close()
