"""Step bookkeeping with several objects in one engine: the device path of
pg_run_steps (image charges, circuit, object charges, result rows) against
pg_step's host path, bit for bit in the mixed form, for one object, a warp's
worth and more than a warp of them."""
import numpy as np
import pytest

from puncpp_gb300 import _lib as L
from puncpp_gb300 import batch, meshgen, punc

pytestmark = pytest.mark.gpu


def make(runs, sources):
    meshes = [meshgen.probe_box(5 + r % 3, 2.0, 0.7) for r in range(runs)]
    b = batch.Batch(meshes, precision=L.PG_MIXED)
    rng = np.random.default_rng(runs)
    for r in range(runs):
        x = 4.0 * rng.random((600, 3)) - 2.0
        b.add_particles(r, x, rng.normal(0.0, 1.0, x.shape), -0.01, 0.01)
        b.add_particles(r, x, rng.normal(0.0, 0.1, x.shape), 0.01, 1.0)
    b.create_flux([punc.Species(-0.01, 0.01, n=100.0, vth=1.0), punc.Species(0.01, 1.0, n=100.0, vth=0.1)],
                  seeds=[7 * r + 1 for r in range(runs)])
    objs = b.objects()
    punc.CircuitCM(b.pop, objs, sources(runs), [], 0.1)
    return b, objs


def ground(runs):
    return [(-1, r, 0.1 * r - 1.0) for r in range(runs)]


def mixed_circuit(runs):
    """Some objects grounded through a source, some joined in pairs (sharing
    charge), the rest floating."""
    out = [(-1, r, 0.5) for r in range(0, runs, 4)]
    return out + [(r, r + 1, 0.25) for r in range(1, runs - 1, 4)]


@pytest.mark.parametrize("sources", [ground, mixed_circuit])
@pytest.mark.parametrize("runs", [1, 5, 37])
def test_run_steps_equal_steps(lib, runs, sources):
    a, oa = make(runs, sources)
    c, oc = make(runs, sources)
    steps = 4
    rows = [punc.step(a.pop, oa, 0.1, first_step=(n == 0), inject=True, step_no=n) for n in range(steps)]
    got = punc.run_steps(c.pop, oc, 0.1, steps, first_step=True, inject=True)
    for r, g in zip(rows, got):
        assert (r.n_particles, r.n_absorbed, r.n_injected, r.KE) == (g.n_particles, g.n_absorbed, g.n_injected, g.KE)
    assert [(o.charge, o.current, o.potential) for o in oa] == [(o.charge, o.current, o.potential) for o in oc]
    assert np.array_equal(punc.Function(a.pop, "phi").vector(), punc.Function(c.pop, "phi").vector())
    assert any(o.current != 0.0 for o in oa)
    a.pop.close()
    c.pop.close()
