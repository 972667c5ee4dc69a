"""FP64 evaluation where its blocks and lanes end: rings of every parity
shared by two lanes (double cones of n sides, apex valence n), blocks with no,
some and only short bonds, closed and open meshes, edge and area bonds;
energy and gradient against the oracle.

Both sides are FP64 with other orders of summation: 1e-11 relative covers
sums of 1e4 terms and rings of 31 slots with condition numbers of 1e3."""
import numpy as np
import pytest

from helpers import unit_params
from test_gpu_surrogate_rings import _cone
from trimem_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _mesh(kind, n):
    p, f = {"cone": lambda: _cone(n), "tube": lambda: meshgen.tube(length=5.0, radius=1.0, segments=n),
            "sphere": lambda: meshgen.icosphere(n)}[kind]()
    return p + np.random.default_rng(n).normal(0, 0.003, p.shape), f


@pytest.mark.parametrize("kind,n", [("cone", k) for k in (3, 4, 5, 6, 7, 8, 31)] + [("sphere", 2), ("sphere", 4)] +
                         [("tube", k) for k in (7, 24, 45)])
@pytest.mark.parametrize("bond,short", [(0, "none"), (0, "some"), (0, "all"), (1, "none")])
def test_energy_and_gradient(built, kind, n, bond, short):
    from oracle import oracle as O
    from trimem_gb300 import capi

    p, f = _mesh(kind, n)
    e = np.concatenate([f[:, [0, 1]], f[:, [1, 2]], f[:, [2, 0]]])
    l = np.linalg.norm(p[e[:, 0]] - p[e[:, 1]], axis=1)
    lc1 = {"none": 0.5 * l.min(), "some": np.median(l), "all": 1.5 * l.max()}[short]
    prm = dict(unit_params(p, f, bond), kappa_t=0.1, bond_lc1=lc1, bond_lc0=1.1 * max(lc1, np.median(l)), bond_r=3)
    mg, mo = capi.Mesh(p, f), O.Mesh(p, f)
    eg, eo = capi.Energy(mg, capi.params(**prm)), O.Energy(mo, O.default_params(**prm))
    eg.set_stencil_precision(0)
    en, g = eg.gradient(mg, with_energy=True)
    eref, gref = eo.energy(mo), eo.gradient(mo)
    assert abs(en - eref) <= 1e-11 * abs(eref), (en, eref)
    assert np.linalg.norm(g - gref) <= 1e-11 * np.linalg.norm(gref)
