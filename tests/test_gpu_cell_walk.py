"""Repulsion by the queued walk over the cells, where the near rows do not serve:
a vertex has left its skin, or rows have overflowed, and every vertex is queued.
Queues within the first blocks' warps (one vertex each) and far past them, cells
of a few members and of more than a warp's lanes; double-word stencils against
the FP64 ones, whose walk is a kernel of its own.  Bit-equal on a second call."""
import numpy as np
import pytest

from helpers import workload_params
from trimem_gb300 import meshgen

pytestmark = pytest.mark.gpu


# cut-off in mean edges, exclusion, vertices moved out of their skin
@pytest.mark.parametrize("rep,excl,moved", [(0.8, 2, 1), (1.6, 1, 3), (2.2, 0, 0), (2.2, 2, 0), (6.0, 1, 1)])
@pytest.mark.parametrize("level", [2, 4, 5, 6])  # 162 .. 40,962 vertices
def test_every_vertex_queued(built, level, rep, excl, moved):
    from trimem_gb300 import capi

    if rep > 5 and level > 4:
        pytest.skip("hundreds of pairs a vertex")
    p, f = meshgen.icosphere(level)
    rng = np.random.default_rng(level)
    p = p + rng.normal(0.0, 0.02 * meshgen.mean_edge_length(p, f), p.shape)
    prm = workload_params(p, f, excl=excl, rep_scale=rep)
    mesh = capi.Mesh(p, f)
    en = capi.Energy(mesh, capi.params(**prm))
    if moved:
        mesh.points()[rng.integers(len(p), size=moved)] *= 1 + 0.6 * prm["rep_lc1"]
    e, g = en.gradient(mesh, with_energy=True)
    again = en.gradient(mesh, with_energy=True)
    assert e == again[0] and np.array_equal(g, again[1])
    en.set_stencil_precision(0)
    eref, gref = en.gradient(mesh, with_energy=True)
    assert abs(e - eref) <= 1e-10 * abs(eref)  # the parity bar of the double-word stencils
    assert np.linalg.norm(g - gref) <= 1e-10 * np.linalg.norm(gref)
