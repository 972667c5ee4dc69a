"""Cells of a box of millions of cells along x: the list bins by the quotient
(x - min) / width as the reference does (src/nlists/cell_list.h:71-78), also
where the product with the reciprocal width truncates to another integer.  The
points are chosen so that it does (the product is off by a unit in the last
place or two: 2e-9 to 6e-8 here); each has a partner 1.3 widths above, in the
next cell under one of the two roundings and two cells away under the other."""
import numpy as np
import pytest

from helpers import unit_params
from oracle import oracle as O
from test_gpu_nlist_build import _strip
from test_gpu_parity import _pairs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rlist,cells", [(0.9, 1e7), (0.9, 2e7), (0.7, 1e8), (0.9, 1e8), (0.9, 3e8)])
def test_points_beside_cell_boundaries(built, rlist, cells):
    from trimem_gb300 import capi

    nv = 400
    rng = np.random.default_rng(int(cells))
    top = cells * rlist
    dim = top + 1e-6
    width = dim / np.trunc(dim / rlist)
    x = rng.integers(2, int(cells) - 10, 400000) * width
    x = np.concatenate([x, np.nextafter(x, 0.0), np.nextafter(x, np.inf)])
    product = x * (1.0 / width)
    from_integer = np.abs(product - np.rint(product))
    x = x[(np.trunc(product) != np.trunc(x / width)) & (from_integer > 1e-9)][:nv // 2 - 1]
    assert len(x) == nv // 2 - 1
    p, f = _strip(nv)
    prm = dict(unit_params(p, f, 0), rlist=rlist, rep_lc1=0.25, n_search=0, exclusion_level=0)
    p[:, 0] = np.concatenate([x, x + 1.3 * width, [0.0, top]])
    p[:, 1:] = 0.1
    mg, mo = capi.Mesh(p, f), O.Mesh(p, f)
    (pg, dg) = _pairs(*capi.NList(mg, capi.params(**prm)).distance_matrix(mg, 1.5 * rlist))
    (po, do) = _pairs(*O.NList(mo, 0, 0, rlist).distance_matrix(mo, 1.5 * rlist))
    assert np.array_equal(pg, po) and np.array_equal(dg, do)
