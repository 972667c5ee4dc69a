"""Parameter gradients of the training kernels where a tile or a persistent
block ends: fewer vertices than a tile, a ragged last tile, and more vertices
than the resident blocks take at once.  k copies of one input side by side
have the loss, and every parameter gradient, of the single input (both are
means over the vertices), so the float64 reference of the single input serves
all sizes; tolerances are those of the gradient test (bf16 activations).

The sums over the copies are also compared with the single input's own
gradient: the same terms in another order, n fp32 additions of them, so each
group stays within 64 * 2^-24 * sqrt(n copies) of the sum of magnitudes; 1e-4
of the group's norm leaves room for the cancellation within a group."""
import numpy as np
import pytest

from test_gpu_surrogate_train import _state, cpu_reference, groups

pytestmark = pytest.mark.gpu


class _Copies:
    """k copies of exported training inputs as one input."""

    def __init__(self, inp, k):
        import torch

        n = inp.u.shape[0]
        self.D = inp.D
        self.u, self.nrm, self.target = (t.repeat(k, 1).contiguous() for t in (inp.u, inp.nrm, inp.target))
        off = (torch.arange(k, device=inp.nbr.device, dtype=inp.nbr.dtype) * n)[None, :, None]
        nbr = inp.nbr[:, None, :].expand(-1, k, -1)
        self.nbr = torch.where(nbr >= 0, nbr + off, nbr).reshape(inp.D, k * n).contiguous()
        self.ef, self.dirs = (t[:, None].expand(-1, k, -1, -1).reshape(inp.D, k * n, t.shape[-1]).contiguous()
                              for t in (inp.ef, inp.dirs))


@pytest.mark.parametrize("level,copies", [(1, 1), (1, 2), (4, 1), (4, 3), (4, 9), (3, 37)])
def test_gradient_at_tile_and_block_edges(built, level, copies):
    from trimem_gb300 import surrogate as S

    _, _, _, _, inp, blob = _state(seed=11, level=level)
    rms = float((inp.target ** 2).mean().sqrt())
    l_ref, F_ref, g_ref = cpu_reference(blob, inp, rms)
    one = S.DeviceTrainer(inp.u.shape[0], inp.D, blob).grad(inp, rms)[2].cpu().numpy()
    many = _Copies(inp, copies)
    loss, F, g = S.DeviceTrainer(many.u.shape[0], many.D, blob).grad(many, rms)
    F, g = F.cpu().numpy(), g.cpu().numpy()
    assert abs(loss - l_ref) <= 1e-3 * abs(l_ref), (loss, l_ref)
    assert np.linalg.norm(F - np.tile(F_ref, (copies, 1))) <= 2e-2 * np.linalg.norm(F)
    for name, a, b in groups():
        norm = max(np.linalg.norm(g_ref[a:b]), 1e-30)
        assert np.linalg.norm(g[a:b] - g_ref[a:b]) < 2e-2 * norm, name
        assert np.linalg.norm(g[a:b] - one[a:b]) < 1e-4 * max(np.linalg.norm(one[a:b]), 1e-30), name
