"""The kernels of a double-word evaluation start before the ones before them
have ended.  What they read of each other's results is the finished data:
evaluations queued one after another at changing positions, whose stages
overlap, give the bits of evaluations whose stages are kept apart (with an
event between any two, as the timed call records them)."""
import ctypes

import numpy as np
import pytest

from helpers import workload_params
from trimem_gb300 import meshgen

pytestmark = pytest.mark.gpu


# one, a few and many blocks per stage, and every number of lanes per vertex
@pytest.mark.parametrize("name", ["sphere1", "sphere4", "sphere5", "sphere6", "tube61"])
def test_overlapped_stages_give_the_bits_of_separate_ones(built, name):
    import torch

    from trimem_gb300 import capi

    L = capi.lib()
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    tube = name.startswith("tube")
    p, f = meshgen.tube(length=5.0, radius=1.0, segments=int(name[4:])) if tube else meshgen.icosphere(int(name[6:]))
    l = meshgen.mean_edge_length(p, f)
    rng = np.random.default_rng(5)
    mesh = capi.Mesh(p, f)
    en = capi.Energy(mesh, capi.params(**workload_params(p, f, bond_type=1 if tube else 0)))
    xs = [torch.tensor(p + rng.normal(0.0, 0.03 * l, p.shape), device="cuda") for _ in range(3)]
    ms = (ctypes.c_float * 5)()
    want, got = [], []
    for x in xs:
        g = torch.empty_like(x)
        capi.check(L.tm_energy_eval_timed(en.h, mesh.h, ptr(x), ptr(g), ms, None))
        want.append(g)
    for k in range(60):
        g, e = torch.empty_like(xs[0]), torch.empty(1, dtype=torch.float64, device="cuda")
        got.append((g, e))
    torch.cuda.synchronize()
    for k, (g, e) in enumerate(got):
        capi.check(L.tm_energy_eval_device(en.h, mesh.h, ptr(xs[k % 3]), ptr(g), ptr(e), None))
    torch.cuda.synchronize()
    for k, (g, e) in enumerate(got):
        assert torch.equal(g, want[k % 3])
        assert torch.equal(e, got[k % 3][1])
