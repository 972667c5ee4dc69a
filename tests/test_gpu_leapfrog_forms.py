"""Velocity Verlet inside the moves (the update runs in the evaluation's first
pass where the stencils allow it) against the same steps in numpy on the
library's own gradients, for each stencil and for a batch of replicas whose
sizes end below, at and past a 256-vertex block.

The momenta come from the one-step move: p = (x1 - x0) / dt + g dt / 2, exact to
2^-52 |x| / dt = 1e-13.  Over a few steps the positions then agree to 1e-12 dt
plus what the gradient's rounding adds: dt^2 |g| times 1e-13 (FP64 and
double-word stencils) or 1e-5 (FP32)."""
import ctypes

import numpy as np
import pytest

from helpers import workload_params
from trimem_gb300 import meshgen

pytestmark = pytest.mark.gpu
DT = 1e-4


def _verlet(x, p, grad, dt, n):
    g, gmax = grad(x), 0.0
    for _ in range(n):
        x = x + p * dt - 0.5 * g * dt * dt
        g1 = grad(x)
        p = p - 0.5 * (g + g1) * dt
        g, gmax = g1, max(gmax, np.abs(g1).max())
    return x, gmax


def _grad_of(capi, p, f, prm, stencil):
    import torch

    mesh, P = capi.Mesh(p, f), lambda t: ctypes.c_void_p(t.data_ptr())
    en = capi.Energy(mesh, capi.params(**prm))
    en.set_stencil_precision(stencil)

    def grad(x):
        d = torch.tensor(x, device="cuda")
        g = torch.empty_like(d)
        capi.check(capi.lib().tm_energy_eval_device(en.h, mesh.h, P(d), P(g), None, None))
        torch.cuda.synchronize()
        return g.cpu().numpy()

    grad.keep = mesh, en
    return grad


@pytest.mark.parametrize("stencil", [0, 1, 2])
@pytest.mark.parametrize("segments", [9, 24, 61])
def test_move_matches_numpy(built, stencil, segments):
    import torch

    from trimem_gb300 import capi

    p, f = meshgen.tube(length=5.0, radius=1.0, segments=segments)
    prm = workload_params(p, f, bond_type=1)
    p = p + np.random.default_rng(segments).normal(0, 1e-3, p.shape)
    grad = _grad_of(capi, p, f, prm, stencil)

    def move(n):
        mesh = capi.Mesh(p, f)
        en = capi.Energy(mesh, capi.params(**prm))
        en.set_stencil_precision(stencil)
        x = torch.tensor(p, device="cuda")
        out = (ctypes.c_double * 4)()
        capi.check(capi.lib().tm_hmc_step_device(en.h, mesh.h, ctypes.c_void_p(x.data_ptr()), 1.0, DT, n, 1.0, 7, 3,
                                                 0.0, out, None, None))
        assert out[0] == 1.0
        return x.cpu().numpy()

    assert np.array_equal(move(0), p)
    mom = (move(1) - p) / DT + 0.5 * grad(p) * DT
    for n in (2, 3, 6):
        want, gmax = _verlet(p, mom, grad, DT, n)
        tol = 1e-12 + n * n * DT * DT * gmax * (1e-5 if stencil == 1 else 1e-13)
        assert np.abs(move(n) - want).max() <= tol, n


@pytest.mark.parametrize("sizes", [(9,), (10, 24), (5, 9, 9, 40, 16)])
@pytest.mark.parametrize("graph", [False, True])
def test_batch_matches_numpy(built, sizes, graph):
    from trimem_gb300 import capi

    reps = []
    for k, s in enumerate(sizes):
        p, f = meshgen.tube(length=5.0, radius=1.0, segments=s)
        prm = workload_params(p, f, bond_type=1)
        reps.append((p + np.random.default_rng(k).normal(0, 1e-3, p.shape), f, prm))

    def move(n):
        b = capi.Batch([(p, f) for p, f, _ in reps], [capi.params(**prm) for _, _, prm in reps])
        acc = b.hmc(1, n, 1e-3 * DT, seed=5, use_graph=graph)
        assert (np.asarray(acc) == 1).all()  # the step is far below the Hamiltonian's error
        return b.positions()

    one = move(1)
    for n in (2, 3, 6):
        got = move(n)
        for (p, f, prm), x1, x in zip(reps, one, got):
            dt = 1e-3 * DT
            grad = _grad_of(capi, p, f, prm, 1)
            mom = (x1 - p) / dt + 0.5 * grad(p) * dt
            want, gmax = _verlet(p, mom, grad, dt, n)
            assert np.abs(x - want).max() <= 1e-14 * n + n * n * dt * dt * gmax * 1e-5, n
