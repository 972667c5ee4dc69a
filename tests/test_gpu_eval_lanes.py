"""Double-word evaluations on both sides of the sizes where the lanes per
vertex change (4,500 and 50,000 vertices), closed and open, against the
oracle (1e-10, the parity bar of the double-word stencils)."""
import numpy as np
import pytest

from helpers import workload_params
from trimem_gb300 import meshgen

pytestmark = pytest.mark.gpu


# tubes of 4,500, 4,636, 49,750 and 50,200 vertices (length 5, radius 1), spheres of 2,562, 10,242 and 163,842
@pytest.mark.parametrize("kind,n", [("tube", 75), ("tube", 76), ("tube", 250), ("tube", 251), ("sphere", 4),
                                    ("sphere", 5), ("sphere", 7)])
def test_evaluation_matches_the_oracle(built, kind, n):
    from oracle import oracle as O
    from trimem_gb300 import capi

    p, f = meshgen.tube(length=5.0, radius=1.0, segments=n) if kind == "tube" else meshgen.icosphere(n)
    l = meshgen.mean_edge_length(p, f)
    p = p + np.random.default_rng(n).normal(0, 0.02 * l, p.shape)
    prm = workload_params(p, f, bond_type=1 if kind == "tube" else 0)
    mg, mo = capi.Mesh(p, f), O.Mesh(p, f)
    eg, eo = capi.Energy(mg, capi.params(**prm)), O.Energy(mo, O.default_params(**prm))
    e, g = eg.gradient(mg, with_energy=True)
    eref, gref = eo.energy(mo), eo.gradient(mo)
    assert abs(e - eref) <= 1e-10 * abs(eref)
    assert np.linalg.norm(g - gref) <= 1e-10 * np.linalg.norm(gref)
    assert eg.energy(mg) == e
