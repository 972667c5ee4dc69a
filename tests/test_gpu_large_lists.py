"""Verlet lists and distance matrices on both sides of the size from which the
exclusion of a build's pairs is tested one vertex at a time, at every level,
against the oracle, exactly."""
import numpy as np
import pytest

from oracle import oracle as O
from trimem_gb300 import meshgen
from trimem_gb300.workloads import workload_params
from test_gpu_parity import _pairs

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("segments", [243, 245])  # 59,778 and 60,270 vertices
@pytest.mark.parametrize("search,excl", [(0, 0), (0, 1), (0, 2), (1, 0), (1, 2)])
def test_pairs_match_the_oracle(built, segments, search, excl):
    from trimem_gb300 import capi

    p, f = meshgen.tube(length=2.0 * np.pi / segments * 245.5, radius=1.0, segments=segments)
    l = meshgen.mean_edge_length(p, f)
    p = p + np.random.default_rng(segments).normal(0.0, 0.02 * l, p.shape)
    prm = dict(workload_params(p, f, bond_type=1, n_search=search, excl=excl), rlist=1.6 * l)
    mg, mo = capi.Mesh(p, f), O.Mesh(p, f)
    (pg, dg) = _pairs(*capi.NList(mg, capi.params(**prm)).distance_matrix(mg, 1.5 * l))
    (po, do) = _pairs(*O.NList(mo, search, excl, 1.6 * l).distance_matrix(mo, 1.5 * l))
    assert len(po) > 0 or excl == 2
    assert np.array_equal(pg, po) and np.array_equal(dg, do)
