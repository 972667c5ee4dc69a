"""FP32-stencil evaluation (single meshes and batches) on rings of every
parity, closed and open meshes, edge and area bonds, short bonds and pairs,
against the FP64 oracle.

FP32 terms carry 6e-8 each; a few tens of operations per term and conditioning
of the shapes up to 50 (flat cones, short bonds) give 1e-4 of the gradient's
norm, 2e-5 of the energy."""
import numpy as np
import pytest

from helpers import unit_params
from test_gpu_fp64_stages import _mesh

pytestmark = pytest.mark.gpu

MESHES = [("cone", k) for k in (3, 4, 5, 6, 7, 8, 31)] + [("sphere", 2), ("sphere", 4)] + [("tube", k) for k in (7, 24, 45)]


def _params(p, f, bond, short):
    e = np.concatenate([f[:, [0, 1]], f[:, [1, 2]], f[:, [2, 0]]])
    l = np.linalg.norm(p[e[:, 0]] - p[e[:, 1]], axis=1)
    lc1 = {"none": 0.5 * l.min(), "some": np.median(l)}[short]
    return dict(unit_params(p, f, bond), kappa_t=0.1, bond_lc1=lc1, bond_lc0=1.1 * max(lc1, np.median(l)), bond_r=2,
                kappa_r=0.01, rep_lc1=1.3 * l.mean(), rlist=1.3 * l.mean(), exclusion_level=1)


def _check(en, g, mo, eo):
    eref, gref = eo.energy(mo), eo.gradient(mo)
    assert abs(en - eref) <= 2e-5 * abs(eref), (en, eref)
    assert np.linalg.norm(g - gref) <= 1e-4 * np.linalg.norm(gref)


@pytest.mark.parametrize("kind,n", MESHES)
@pytest.mark.parametrize("bond,short", [(0, "none"), (0, "some"), (1, "none")])
def test_single_mesh(built, kind, n, bond, short):
    from oracle import oracle as O
    from trimem_gb300 import capi

    p, f = _mesh(kind, n)
    prm = _params(p, f, bond, short)
    mg, mo = capi.Mesh(p, f), O.Mesh(p, f)
    eg, eo = capi.Energy(mg, capi.params(**prm)), O.Energy(mo, O.default_params(**prm))
    eg.set_stencil_precision(1)
    en, g = eg.gradient(mg, with_energy=True)
    _check(en, g, mo, eo)


@pytest.mark.parametrize("kinds", [[("sphere", 2), ("cone", 7), ("cone", 8), ("sphere", 4)],
                                   [("tube", 7), ("sphere", 2), ("tube", 24)]])
def test_batch(built, kinds):
    from oracle import oracle as O
    from trimem_gb300 import capi

    reps = []
    for kind, n in kinds:
        p, f = _mesh(kind, n)
        reps.append((p, f, _params(p, f, 0, "some")))
    b = capi.Batch([(p, f) for p, f, _ in reps], [capi.params(**prm) for _, _, prm in reps])
    energies, grads = b.energy(with_grad=True)
    for (p, f, prm), en, g in zip(reps, energies, grads):
        mo = O.Mesh(p, f)
        _check(en, g, mo, O.Energy(mo, O.default_params(**prm)))
