"""What an evaluation needs is allocated with the handle: the first one in each
stencil precision takes no device memory (163,842 vertices, where every array
is a block of its own)."""
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
