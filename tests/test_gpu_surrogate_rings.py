"""The learned force on rings that end at, before and past the eight slots
that eight lanes take at once, and on last tiles of every kind: a double cone
of n sides (apex valence n, four elsewhere) and open tubes, forward against
the torch restatement of the network and training gradients against the
float64 reference.  Tolerances are those of the network tests (bf16
activations through three rounds: 2e-2 norm-wise)."""
import ctypes

import numpy as np
import pytest

from helpers import workload_params
from test_gpu_surrogate import _random_blob
from test_gpu_surrogate_train import cpu_reference, groups
from trimem_gb300 import meshgen

pytestmark = pytest.mark.gpu


def _cone(n):
    a = 2 * np.pi * np.arange(n) / n
    p = np.concatenate([np.stack([np.cos(a), np.sin(a), 0.1 * np.cos(2 * a)], 1), [[0, 0, 0.9], [0, 0, -1.1]]])
    k = np.arange(n)
    f = np.concatenate([np.stack([k, (k + 1) % n, np.full(n, n)], 1), np.stack([(k + 1) % n, k, np.full(n, n + 1)], 1)])
    return p, f.astype(np.int32)


CASES = [("cone", n) for n in (5, 7, 8, 9, 16, 17, 31)] + [("tube", s) for s in (10, 24, 41)]


@pytest.mark.parametrize("kind,n", CASES)
def test_forward_and_gradient(built, kind, n):
    import torch

    from trimem_gb300 import capi
    from trimem_gb300 import surrogate as S

    p, f = _cone(n) if kind == "cone" else meshgen.tube(length=5.0, radius=1.0, segments=n)
    p = p + np.random.default_rng(n).normal(0, 0.01, p.shape)
    prm = dict(workload_params(p, f, bond_type=1), cont_lambda=0.0)
    mesh = capi.Mesh(p, f)
    en = capi.Energy(mesh, capi.params(**prm))
    net, blob = _random_blob(p, f, n)
    sg = capi.Surrogate(mesh, blob)
    x = torch.tensor(p, dtype=torch.float64, device="cuda").contiguous()
    inp = S.Inputs(sg, en, mesh, x, 32)
    g = torch.empty_like(x)
    P = lambda t: ctypes.c_void_p(t.data_ptr())
    capi.check(capi.lib().tm_surrogate_gradient_device(sg.h, en.h, mesh.h, P(x), P(g), None))
    torch.cuda.synchronize()
    F = (inp.gloc - g).float()
    with torch.no_grad():
        ref = net.cuda()(inp.u, inp.nrm, inp.nbr, inp.ef, inp.dirs, bf16=True)
    assert torch.linalg.norm(F - ref) < 2e-2 * torch.linalg.norm(ref)
    inp.target = torch.randn(F.shape, device="cuda", generator=torch.Generator(device="cuda").manual_seed(n))
    l_ref, F_ref, g_ref = cpu_reference(blob, inp, 1.0)
    loss, Ft, gt = S.DeviceTrainer(len(p), inp.D, blob).grad(inp, 1.0)
    assert abs(loss - l_ref) <= 2e-2 * abs(l_ref)
    assert np.linalg.norm(Ft.cpu().numpy() - F_ref) <= 2e-2 * np.linalg.norm(F_ref)
    gt = gt.cpu().numpy()
    # all parameters at once: a single one (b_o on a closed mesh) can cancel
    assert np.linalg.norm(gt - g_ref) <= 2e-2 * np.linalg.norm(g_ref)
    for name, a, b in groups():
        if b - a > 1:
            assert np.linalg.norm(gt[a:b] - g_ref[a:b]) <= 4e-2 * np.linalg.norm(g_ref[a:b]), name
