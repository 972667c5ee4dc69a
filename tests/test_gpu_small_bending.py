"""Bending moduli at and below the smallest float in the double-word stencils:
a modulus that no float can hold bends nothing (the bits of a modulus of zero),
a small one that a float can hold keeps the gradient of the FP64 stencils."""
import numpy as np
import pytest

from helpers import workload_params
from trimem_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _gradient(kappa_b, stencil):
    from trimem_gb300 import capi

    p, f = meshgen.jittered_icosphere(2, seed=1)
    mesh = capi.Mesh(p, f)
    en = capi.Energy(mesh, capi.params(**dict(workload_params(p, f), kappa_b=kappa_b)))
    en.set_stencil_precision(stencil)
    return en.gradient(mesh)


@pytest.mark.parametrize("kappa_b", [1e-60, 1e-75, -1e-80, 1e-300])
def test_modulus_below_the_float_range(built, kappa_b):
    g = _gradient(kappa_b, 2)
    assert np.isfinite(g).all() and np.array_equal(g, _gradient(0.0, 2))


@pytest.mark.parametrize("kappa_b", [1e-44, 1e-30, 1e-3])
def test_small_modulus(built, kappa_b):
    g, ref = _gradient(kappa_b, 2), _gradient(kappa_b, 0)
    assert np.linalg.norm(g - ref) <= 1e-10 * np.linalg.norm(ref)
