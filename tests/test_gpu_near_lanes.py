"""Near rows built by eight lanes a vertex and by one, on both sides of the limit
between them, and with the next kernel started early and late: after every
vertex has left its skin the rows are rebuilt, and the evaluation through them
is the one of a handle made at the new positions, bit for bit, and agrees with
the FP64 stencils."""
import numpy as np
import pytest

from helpers import workload_params
from trimem_gb300 import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("segments", [40, 105, 107, 295, 297])  # 960, 2,415 | 2,461, 44,840 | 45,144 vertices
@pytest.mark.parametrize("rep,excl", [(0.8, 2), (1.2, 1), (1.2, 0)])
def test_rows_follow_a_move(built, segments, rep, excl):
    from trimem_gb300 import capi

    p, f = meshgen.tube(length=min(5.0, 2.0 * np.pi / segments * (23 if segments < 200 else 152)), radius=1.0,
                        segments=segments)
    l = meshgen.mean_edge_length(p, f)
    rng = np.random.default_rng(segments)
    p = p + rng.normal(0.0, 0.02 * l, p.shape)
    prm = capi.params(**workload_params(p, f, bond_type=1, excl=excl, rep_scale=rep))
    moved = p * 1.02 + [2.0 * rep * l, 0.0, 0.0]
    mesh = capi.Mesh(p, f)
    en = capi.Energy(mesh, prm)
    mesh.points()[:] = moved
    en.update_repulsion(mesh)
    e, g = en.gradient(mesh, with_energy=True)
    fresh_mesh = capi.Mesh(moved, f)
    fresh = capi.Energy(fresh_mesh, prm)
    fresh.set_initial_props(en.initial_props())
    assert fresh.energy(fresh_mesh) == e
    assert np.array_equal(fresh.gradient(fresh_mesh), g)
    en.set_stencil_precision(0)
    eref, gref = en.gradient(mesh, with_energy=True)
    assert abs(e - eref) <= 1e-10 * abs(eref)
    assert np.linalg.norm(g - gref) <= 1e-10 * np.linalg.norm(gref)
