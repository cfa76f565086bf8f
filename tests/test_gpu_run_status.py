"""pg_run_steps reports an ESolver of its last step that did not converge."""
import pytest

from puncpp_gb300 import _lib as L
from puncpp_gb300 import meshgen, punc

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("graph", [False, True])
def test_run_reports_the_esolver(lib, graph):
    """The potential of an object, 1e60, is within the FP64 solver's range and
    beyond the FP32 field's."""
    pop = punc.Population(punc.Mesh(meshgen.probe_box(6, 2.0, 0.9)), precision=L.PG_MIXED, pcg_precond=1,
                          pcg_precision=1)
    punc.run_steps(pop, [punc.Object(2, potential=1.0)], 0.1, 3, efield_cg1=True, use_graph=graph)
    with pytest.raises(L.PgError) as e:
        punc.run_steps(pop, [punc.Object(2, potential=1e60)], 0.1, 3, efield_cg1=True, use_graph=graph)
    assert e.value.code == 6 and "ESolver" in str(e.value)
    punc.run_steps(pop, [punc.Object(2, potential=1.0)], 0.1, 3, efield_cg1=True, use_graph=graph)
    pop.close()
