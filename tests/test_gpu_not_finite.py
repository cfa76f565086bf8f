"""A potential that is not finite ends the ESolver as not converged, in each
of its forms, and leaves nothing behind for the next solve."""
import numpy as np
import pytest

from puncpp_gb300 import _lib as L
from puncpp_gb300 import meshgen, punc
from test_gpu_esolver import BAR, reference

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", [L.PG_FP64, L.PG_MIXED])
@pytest.mark.parametrize("n", [9, 43])   # rows in registers, and not (80k dofs)
@pytest.mark.parametrize("bad", [np.nan, np.inf, 1e300])
@pytest.mark.parametrize("warm", [False, True])
def test_esolver_of_a_bad_potential(lib, prec, n, bad, warm):
    mesh = punc.Mesh(meshgen.probe_box(n, 2.0, 0.9))
    pop = punc.Population(mesh, precision=prec)
    es = punc.ESolver(pop)
    E = punc.Function(pop, "E_cg1")
    phi = np.random.default_rng(n).normal(size=mesh.n_dofs)
    if warm:
        punc.Function(pop, "phi").set_local(phi)
        es.solve(E, None)
    worse = phi.copy()
    worse[mesh.n_dofs // 2] = bad
    punc.Function(pop, "phi").set_local(worse)
    for _ in range(2):
        with pytest.raises(L.PgError) as e:
            es.solve(E, None)
        assert e.value.code == 6
    punc.Function(pop, "phi").set_local(phi)
    want = reference(mesh, phi)
    assert np.linalg.norm(es.solve(E, None) - want) <= BAR[prec] * np.linalg.norm(want) + 1e-12
    pop.close()
