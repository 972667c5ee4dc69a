"""Candidate rows of a cell list whose box is so wide that the margin added to
its sides (1e-6) is lost in rounding: a vertex on the upper x face has a cell
coordinate past the side, and with one cell along x its id is that of the next
cell along y, which the row's scan visits at another place than the middle."""
import numpy as np
import pytest

from helpers import unit_params
from oracle import oracle as O
from trimem_gb300 import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("low", [True, False])
def test_vertex_on_the_upper_face_of_a_wide_box(built, low):
    from trimem_gb300 import capi

    p, f = meshgen.icosphere(1)  # 42 vertices: rows of up to 41 entries are kept
    p = p + np.random.default_rng(0).normal(0.0, 0.02, p.shape)
    p = p * [0.9e10, 2.0e10, 0.9e10]
    # one vertex ahead of all others in x, in the lower or the upper y half
    v = int(np.argmax(np.where(p[:, 1] < 0 if low else p[:, 1] > 0, p[:, 0], -np.inf)))
    p[v, 0] = p[:, 0].max() + 1e8
    assert np.argmax(p[:, 0]) == v and (p[:, 0].max() - p[:, 0].min()) + 1e-6 == p[:, 0].max() - p[:, 0].min()
    prm = unit_params(p, f, 1)
    for k in ("kappa_b", "kappa_a", "kappa_v", "kappa_c", "kappa_t"):
        prm[k] = 0.0
    # a list cut-off below the repulsion's: rows of candidates, no near rows
    prm.update(kappa_r=1e25, rep_lc1=2.5e10, rlist=1.75e10, exclusion_level=1)
    mo, mg = O.Mesh(p, f), capi.Mesh(p, f)
    eo, eg = O.Energy(mo, O.default_params(**prm)), capi.Energy(mg, capi.params(**prm))
    eg.set_stencil_precision(0)
    e, g = eg.gradient(mg, with_energy=True)
    eref, gref = eo.energy(mo), eo.gradient(mo)
    assert eref > 0 and np.abs(gref[v]).max() > 0
    # FP64 sums of up to 41 terms a vertex in the oracle's order
    assert abs(e - eref) <= 1e-12 * abs(eref)
    assert np.linalg.norm(g - gref) <= 1e-12 * np.linalg.norm(gref)
