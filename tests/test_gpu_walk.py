"""The screened walk of both particle forms against pg_relocate's FP64 walk from
the same start cells, and move_periodic against its formula: points inside
cells, on facets, edges and vertices of the mesh, one cell and a whole box
away."""
import numpy as np
import pytest

from helpers import sort_by_id
from puncpp_gb300 import _lib as L
from puncpp_gb300 import meshgen, punc

pytestmark = pytest.mark.gpu

FORMS = [L.PG_FP64, L.PG_MIXED]


def load(ma, prec, x, v, **kw):
    pop = punc.Population(punc.Mesh(ma), precision=prec, **kw)
    assert pop.add_particles(x, v, -1.0, 1.0) == len(x)
    return pop


def lattice_and_random(rng, lo, hi, n, count):
    """Random points, points on a lattice of half cells (facets, edges and
    vertices of Kuhn cells) and points a rounding away from it."""
    h = (hi - lo) / n
    x = lo + (hi - lo) * rng.random((count, 3))
    y = lo + h * (0.5 * rng.integers(1, 2 * n, (count, 3)))
    z = y * (1.0 + 1e-16 * rng.integers(-3, 4, (count, 3)))
    return np.concatenate([x, y, np.clip(z, lo + 1e-9, hi - 1e-9)])


@pytest.mark.parametrize("prec", FORMS)
@pytest.mark.parametrize("n", [1, 2, 5, 24])
def test_walk_across_a_periodic_box(lib, prec, n):
    rng = np.random.default_rng(n)
    ma = meshgen.langmuir_cube(n)
    x = lattice_and_random(rng, 0.0, 1.0, n, 4000)
    v = rng.normal(0.0, 0.6, x.shape)
    v[::3] = 0.5 / n * rng.integers(-2 * n, 2 * n + 1, v[::3].shape)
    pop = load(ma, prec, x, v, periodic=True)
    for _ in range(3):
        before = sort_by_id(pop.particles())
        punc.move_periodic(pop, 1.0, ma.Ld)
        moved = sort_by_id(pop.particles())
        if prec == L.PG_FP64:
            y = before["x"] + 1.0 * before["v"]
            assert np.array_equal(moved["x"], y - np.floor(y))
        want = pop.relocate(moved["x"], before["cell"])
        pop.update([], 1.0)
        after = sort_by_id(pop.particles())
        stay = want >= 0
        assert np.array_equal(after["id"], before["id"][stay])
        assert np.array_equal(after["cell"], want[stay])
    pop.close()


@pytest.mark.parametrize("prec", FORMS)
def test_walk_around_an_object(lib, prec):
    """Domain with a hole: no restart, absorbed where the FP64 walk is."""
    rng = np.random.default_rng(11)
    ma = meshgen.probe_box(9, 2.0, 0.7)
    x = lattice_and_random(rng, -2.0, 2.0, 9, 6000)
    pop = punc.Population(punc.Mesh(ma), precision=prec)
    pop.add_particles(x, rng.normal(0.0, 1.0, x.shape), -1.0, 1.0)
    before = sort_by_id(pop.particles())
    punc.move(pop, 1.0)
    moved = sort_by_id(pop.particles())
    want = pop.relocate(moved["x"], before["cell"])
    pop.update([punc.Object(2)], 1.0)
    after = sort_by_id(pop.particles())
    assert np.array_equal(after["id"], before["id"][want >= 0])
    assert np.array_equal(after["cell"], want[want >= 0])
    counts, _, _ = punc.absorbed_counts(pop)
    assert counts[1, 0] == (want == -1).sum() and counts[2, 0] == (want == -2).sum()
    pop.close()


@pytest.mark.parametrize("length", [1.0, 0.7, 3.0])
def test_move_periodic_bits(lib, length):
    """x - L floor(x / L) at and around the multiples of L, FP64."""
    edges = np.array([0.0, -0.0, 5e-324, -5e-324, 1e-310, -1e-310, -1e-201, -1e-199, 1e-18, -1e-18])
    around = [np.nextafter(k * length, s) for k in (-2, -1, 1, 2) for s in (-np.inf, np.inf)]
    targets = np.concatenate([edges, around, length * np.array([-2.5, -2.0, -1.0, -0.3, 0.4, 1.0, 1.7, 2.0, 7.3])])
    ma = meshgen.kuhn_box(2, 0.0, length, periodic=True)
    # x + 1.0 * v is rounded once: start next to the target's scale so that
    # the small ones are reached from a particle near 0
    x = np.full((len(targets), 3), 0.25 * length)
    x[:, 0] = np.where(np.abs(targets) < 1e-6, 2.0 ** -30, x[:, 0])
    v = np.zeros_like(x)
    v[:, 0] = targets - x[:, 0]
    pop = load(ma, L.PG_FP64, x, v, periodic=True)
    before = sort_by_id(pop.particles())
    punc.move_periodic(pop, 1.0, ma.Ld)
    y = before["x"] + 1.0 * before["v"]
    assert np.array_equal(sort_by_id(pop.particles())["x"], y - length * np.floor(y / length))
    pop.close()
