"""What an evaluation and an HMC move need is allocated with the handle: the
first evaluation in each stencil precision and the first move take no device
memory (163,842 vertices, where every array is a block of its own)."""
import ctypes

import pytest

from helpers import workload_params
from trimem_gb300 import meshgen

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stencil", [0, 1, 2])
def test_first_evaluation_allocates_nothing(built, stencil):
    import torch

    from trimem_gb300 import capi

    p, f = meshgen.icosphere(7)
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())
    x = torch.tensor(p, device="cuda")
    g, ms = torch.empty_like(x), (ctypes.c_float * 5)()

    def first():
        mesh = capi.Mesh(p, f)
        en = capi.Energy(mesh, capi.params(**workload_params(p, f)))
        en.set_stencil_precision(stencil)
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        capi.check(capi.lib().tm_energy_eval_timed(en.h, mesh.h, ptr(x), ptr(g), ms, None))
        torch.cuda.synchronize()
        return free - torch.cuda.mem_get_info()[0]

    first()  # kernels of this precision are loaded
    assert first() == 0


def test_first_move_allocates_nothing(built):
    import torch

    from trimem_gb300 import capi

    p, f = meshgen.icosphere(7)
    x, out4 = torch.tensor(p, device="cuda"), (ctypes.c_double * 4)()

    def first():
        mesh = capi.Mesh(p, f)
        en = capi.Energy(mesh, capi.params(**workload_params(p, f)))
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        capi.check(capi.lib().tm_hmc_step_device(en.h, mesh.h, ctypes.c_void_p(x.data_ptr()), 1.0, 1e-7, 2, 1.0, 3, 0,
                                                 0.5, out4, None, None))
        torch.cuda.synchronize()
        return free - torch.cuda.mem_get_info()[0]

    first()
    assert first() == 0
