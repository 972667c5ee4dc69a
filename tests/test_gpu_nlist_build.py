"""Cell-list builds at the edges of the build's blocks and cells: the distance
matrix of the cell list
and of the Verlet list against the oracle, exactly, for vertex counts below,
at and past one 256-vertex block, coarse boxes (one cell that holds every
vertex, cells of many members), fine ones (empty cells between), points on
cell boundaries and coordinates that truncate next to an integer."""
import numpy as np
import pytest

from helpers import unit_params
from test_gpu_parity import _pairs

pytestmark = pytest.mark.gpu


def _strip(nv):
    """Open strip of nv vertices in a zig-zag on a 0.5 lattice (so that
    coordinates over the cell width truncate at and next to integers)."""
    i = np.arange(nv)
    p = np.stack([0.5 * (i // 2), 0.5 * (i % 2), 0.25 * ((i // 2) % 3)], 1).astype(np.float64)
    k = np.arange(nv - 2)
    f = np.where((k % 2 == 0)[:, None], np.stack([k, k + 1, k + 2], 1), np.stack([k + 1, k, k + 2], 1))
    return p, f.astype(np.int32)


@pytest.mark.parametrize("nv", [4, 31, 255, 256, 257, 511, 1500])
@pytest.mark.parametrize("rlist", [0.3, 0.5, 0.75, 1e3])
@pytest.mark.parametrize("search,excl", [(0, 0), (0, 1), (1, 0)])
def test_pairs_match_the_oracle(built, nv, rlist, search, excl):
    from oracle import oracle as O
    from trimem_gb300 import capi

    if rlist > 100 and nv > 600:
        pytest.skip("all pairs of the coarse box")
    p, f = _strip(nv)
    prm = dict(unit_params(p, f, 0), rlist=rlist, rep_lc1=0.25, n_search=search, exclusion_level=excl)
    rd = min(rlist, 0.9)
    mg, mo = capi.Mesh(p, f), O.Mesh(p, f)
    (pg, dg) = _pairs(*capi.NList(mg, capi.params(**prm)).distance_matrix(mg, rd))
    (po, do) = _pairs(*O.NList(mo, search, excl, rlist).distance_matrix(mo, rd))
    assert np.array_equal(pg, po) and np.array_equal(dg, do)


@pytest.mark.parametrize("nv", [31, 257, 1500])
@pytest.mark.parametrize("shift", [0.0, -7.3])
def test_near_rows_after_moves(built, nv, shift):
    """Energy and gradient through the near rows, built, kept over a small
    move and rebuilt after a large one, against the oracle (1e-9: terms good to
    about 1e-14, corners of the moved strip with condition numbers to 1e4)."""
    from oracle import oracle as O
    from trimem_gb300 import capi

    rng = np.random.default_rng(nv)
    p, f = _strip(nv)
    p = p + shift + rng.normal(0, 0.02, p.shape)
    prm = dict(unit_params(p, f, 0), rlist=0.6, rep_lc1=0.6, n_search=0, exclusion_level=1, kappa_r=10.0)
    mg, mo = capi.Mesh(p, f), O.Mesh(p, f)
    eg, eo = capi.Energy(mg, capi.params(**prm)), O.Energy(mo, O.default_params(**prm))
    for size in (0.0, 0.01, 0.25, 0.01):
        p = p + rng.normal(0, size, p.shape) if size else p
        mg.points()[:] = p
        mo.points()[:] = p
        eg.update_repulsion(mg)
        eo.update_repulsion(mo)
        e, g = eg.gradient(mg, with_energy=True)
        eref, gref = eo.energy(mo), eo.gradient(mo)
        assert abs(e - eref) <= 1e-9 * abs(eref), (size, e, eref)
        assert np.linalg.norm(g - gref) <= 1e-9 * np.linalg.norm(gref), size
