"""move_periodic for lengths that are no box: x - L floor(x / L) as it is
evaluated, also for negative, zero and infinite L and NaN."""
import numpy as np
import pytest

from helpers import sort_by_id
from puncpp_gb300 import _lib as L
from puncpp_gb300 import meshgen, punc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [L.PG_FP64, L.PG_MIXED])
@pytest.mark.parametrize("length", [-0.5, -2.0, 0.0, -0.0, np.inf, -np.inf, np.nan])
def test_move_periodic_of_any_length(lib, prec, length):
    """The values are multiples of 2^-10 and the lengths powers of two, so that
    no operation of either precision rounds."""
    rng = np.random.default_rng(1)
    x = rng.integers(1, 1024, (4000, 3)) / 1024.0
    v = rng.integers(-4096, 4096, (4000, 3)) / 1024.0
    pop = punc.Population(punc.Mesh(meshgen.kuhn_box(2, 0.0, 1.0)), precision=prec)
    assert pop.add_particles(x, v, -1.0, 1.0) == len(x)
    before = sort_by_id(pop.particles())
    punc.move_periodic(pop, 1.0, (length, 0.5, length))
    got = sort_by_id(pop.particles())["x"]
    y = before["x"] + before["v"]
    ld = np.array([length, 0.5, length])
    with np.errstate(all="ignore"):
        want = y - ld * np.floor(y / ld)
    assert np.array_equal(got, want, equal_nan=True)
    pop.close()
