"""Walks of Population::update in meshes that fill their bounding box though
walls stand inside, against pg_relocate's walk through every cell between: no
particle may pass a wall.  And the step limit in a slender box."""
import numpy as np
import pytest

import box_meshes
from helpers import sort_by_id
from puncpp_gb300 import _lib as L
from puncpp_gb300 import punc

pytestmark = pytest.mark.gpu

FORMS = [L.PG_FP64, L.PG_MIXED]


def crossing(ma, prec, x, to, objects):
    """Move particles from x to the points and update; the ids kept, their
    cells, the counts per tag, and the cells or tags of pg_relocate."""
    pop = punc.Population(punc.Mesh(ma), precision=prec)
    assert pop.add_particles(x, to - x, -1.0, 1.0) == len(x)
    before = sort_by_id(pop.particles())
    punc.move(pop, 1.0)
    moved = sort_by_id(pop.particles())
    want = pop.relocate(moved["x"], before["cell"])
    pop.update(objects, 1.0)
    after = sort_by_id(pop.particles())
    counts, _, _ = punc.absorbed_counts(pop)
    assert np.array_equal(after["id"], before["id"][want >= 0])
    assert np.array_equal(after["cell"], want[want >= 0])
    for tag in range(1, 2 + ma.n_objects):
        assert counts[tag, 0] == (want == -tag).sum()
    pop.close()
    return want


@pytest.mark.parametrize("prec", FORMS)
def test_plate_of_no_thickness(lib, prec):
    rng = np.random.default_rng(3)
    x = np.array([0.03, 0.3, 0.3]) + np.array([0.1, 0.4, 0.4]) * rng.random((3000, 3))
    to = x + np.array([0.8, 0.0, 0.0])
    want = crossing(box_meshes.plate(), prec, x, to, [punc.Object(2)])
    assert (want == -2).sum() > 2000


@pytest.mark.parametrize("prec", FORMS)
def test_object_of_a_billionth_of_the_box(lib, prec):
    rng = np.random.default_rng(4)
    ma, centre = box_meshes.speck()
    x = centre + 0.004 * rng.normal(size=(20000, 3))
    x = x[np.abs(x - centre).max(axis=1) > 0.0015]
    u = rng.normal(size=x.shape)
    to = np.clip(x + 0.2 * u / np.linalg.norm(u, axis=1)[:, None], 0.01, 0.99)
    pop = punc.Population(punc.Mesh(ma))
    inside = pop.locate(x) >= 0
    pop.close()
    want = crossing(ma, prec, x[inside], to[inside], [punc.Object(2)])
    assert (want == -2).sum() > 100


@pytest.mark.parametrize("prec", FORMS)
def test_boxes_side_by_side(lib, prec):
    """A particle that leaves the one box is not in the other."""
    rng = np.random.default_rng(5)
    ma, n_first = box_meshes.side_by_side()
    x = 0.02 + np.array([0.1, 0.96, 0.96]) * rng.random((2000, 3))
    to = x + np.array([1.75, 0.0, 0.0])
    want = crossing(ma, prec, x, to, [])
    assert (want == -1).all()


@pytest.mark.parametrize("prec", FORMS)
def test_walk_limit_of_a_slender_box(lib, prec):
    """120,000 cells between the ends, 100,000 the default limit."""
    n = 40000
    pop = punc.Population(punc.Mesh(box_meshes.slender(n)), precision=prec, pcg_precond=1)
    x = np.array([[0.3, 0.6, 0.5], [0.3, 0.6, 0.5]])
    to = np.array([[0.4, 0.5, 20000.25], [0.4, 0.5, n - 0.25]])
    assert pop.add_particles(x[:1], to[:1] - x[:1], -1.0, 1.0) == 1
    punc.move(pop, 1.0)
    pop.update([], 1.0)
    assert pop.num_of_particles() == 1
    assert pop.add_particles(x[1:], to[1:] - x[1:], -1.0, 1.0) == 1
    punc.move(pop, 1.0)
    with pytest.raises(L.PgError) as e:
        pop.update([], 1.0)
    assert e.value.code == 5
    pop.close()
