"""Device L-BFGS against the same recursion in numpy on the library's own
energies and gradients, at each number of vector elements a thread holds
(sizes on both sides of one, two, four and eight elements per thread, and
past them), with the history shorter and longer than the run.

Both sides evaluate the same kernels; only dot products are summed in another
order: relative errors of sqrt(n) 2^-53 (1e-13 here), which the recursion's
conditioning (ratios of s.y along the run, up to 1e3) carries into the
displacement: 1e-8 of its norm leaves two digits."""
import ctypes

import numpy as np
import pytest

from helpers import workload_params
from trimem_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _numpy_lbfgs(energy, mesh, x, maxiter, history):
    import torch

    from trimem_gb300 import capi

    L = capi.lib()
    P = lambda t: ctypes.c_void_p(t.data_ptr())
    g, e = torch.empty_like(x), torch.empty(1, dtype=torch.float64, device="cuda")

    def ev(y):
        d = torch.tensor(y, device="cuda")
        capi.check(L.tm_energy_update_repulsion_device(energy.h, mesh.h, P(d), None))
        capi.check(L.tm_energy_eval_device(energy.h, mesh.h, P(d), P(g), P(e), None))
        torch.cuda.synchronize()
        return float(e.item()), g.cpu().numpy()

    y = x.cpu().numpy()
    f, gr = ev(y)
    pairs, gamma, n = [], 1.0, 0
    for n in range(maxiter):
        d, al = -gr, []
        for s, t in reversed(pairs):
            al.append((s * d).sum() / (s * t).sum())
            d = d - al[-1] * t
        d = gamma * d
        for (s, t), a in zip(pairs, reversed(al)):
            d = d + (a - (t * d).sum() / (s * t).sum()) * s
        gd = (gr * d).sum()
        assert gd < 0
        a = 1.0 if pairs else min(1.0, 1e-3 / np.abs(gr).max())
        for _ in range(40):
            z = y + a * d
            fz, gz = ev(z)
            if np.isfinite(fz) and fz <= f + 1e-4 * a * gd:
                break
            a *= 0.5
        else:
            break
        s, t = z - y, gz - gr
        fp, f, y, gr = f, fz, z, gz
        if (s * t).sum() > 1e-300:
            pairs = (pairs + [(s, t)])[-history:]
            gamma = (s * t).sum() / (t * t).sum()
        if fp - f <= 2.220446049250313e-09 * max(abs(fp), abs(f), 1.0):
            return y, f, n + 1
    else:
        n = maxiter
    return y, f, n


# vertices (three elements each) over 75,776 threads
@pytest.mark.parametrize("segments", [9, 24, 161, 170, 230, 340, 450, 520])
@pytest.mark.parametrize("history", [2, 10])
def test_iterates_match_numpy(built, segments, history):
    import torch

    from trimem_gb300 import capi
    from trimem_gb300.mc.minim import minimize_device

    p, f = meshgen.tube(length=5.0, radius=1.0, segments=segments)
    l = meshgen.mean_edge_length(p, f)
    p = p + np.random.default_rng(segments).normal(0, 0.02 * l, p.shape)
    mesh = capi.Mesh(p, f)
    prm = capi.params(**workload_params(p, f, bond_type=1))
    x = torch.tensor(p, dtype=torch.float64, device="cuda")
    want, fw, nw = _numpy_lbfgs(capi.Energy(mesh, prm), mesh, x, 6, history)
    it, e = minimize_device(capi.Energy(mesh, prm), mesh, x, maxiter=6, history=history)
    assert it == nw
    assert abs(e - fw) <= 1e-9 * abs(fw)
    assert np.linalg.norm(x.cpu().numpy() - want) <= 1e-8 * np.linalg.norm(want - p)
