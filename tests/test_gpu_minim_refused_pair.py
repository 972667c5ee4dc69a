"""Device L-BFGS with steps whose correction pair is refused (s.y <= 0, here
from a tether of negative weight) once the history is full: the pairs kept are
those of the accepted ones, the oldest included, as in the numpy recursion.

Both sides evaluate the same kernels; a relative difference of 1e-13 in the dot
products grows to about 1e-11 over these runs (the recursion on evaluations of
the CPU oracle agrees with itself to that), while a run that lost its oldest
pair ends a thirtieth of the displacement away or more: 1e-8."""
import numpy as np
import pytest

from helpers import workload_params
from test_gpu_minim_direction import _numpy_lbfgs
from trimem_gb300 import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("seed,noise,history,maxiter", [(3, 0.2, 1, 6), (3, 0.05, 2, 6), (1, 0.05, 2, 4)])
def test_refused_pair_leaves_the_oldest(built, seed, noise, history, maxiter):
    import torch

    from trimem_gb300 import capi
    from trimem_gb300.mc.minim import minimize_device

    p, f = meshgen.icosphere(2)
    p = p + np.random.default_rng(seed).normal(0, noise * meshgen.mean_edge_length(p, f), p.shape)
    mesh = capi.Mesh(p, f)
    prm = capi.params(**dict(workload_params(p, f, bond_type=1), kappa_t=-1000.0))
    x = torch.tensor(p, dtype=torch.float64, device="cuda")
    want, fw, nw = _numpy_lbfgs(capi.Energy(mesh, prm), mesh, x, maxiter, history)
    it, e = minimize_device(capi.Energy(mesh, prm), mesh, x, maxiter=maxiter, history=history)
    assert it == nw
    assert abs(e - fw) <= 1e-9 * abs(fw)
    assert np.linalg.norm(x.cpu().numpy() - want) <= 1e-8 * np.linalg.norm(want - p)
