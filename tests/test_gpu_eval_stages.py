"""Double-word evaluations at the edges of their kernels' ranges, against the
oracle: one and eight lanes per vertex (meshes on both sides of the limit),
rings longer than the lanes, open fans, Verlet rows walked by one and by
eight lanes, lists whose exclusions are older than the topology."""
import numpy as np
import pytest

from helpers import workload_params
from oracle import oracle as O
from trimem_gb300 import meshgen

pytestmark = pytest.mark.gpu

RTOL = 1e-10  # the parity bar of the double-word stencils


@pytest.fixture(scope="module")
def C(built):
    from trimem_gb300 import capi
    return capi


def bipyramid(n):
    """Closed mesh with two vertices of valence n and n of valence 4."""
    a = 2 * np.pi * np.arange(n) / n
    p = np.concatenate([np.stack([np.cos(a), np.sin(a), 0.05 * np.cos(3 * a)], 1), [[0, 0, 0.6], [0, 0, -0.5]]])
    i, j = np.arange(n), (np.arange(n) + 1) % n
    f = np.concatenate([np.stack([i, j, np.full(n, n)], 1), np.stack([j, i, np.full(n, n + 1)], 1)])
    return p, f.astype(np.int32)


def mesh(name):
    if name.startswith("bipyramid"):
        return bipyramid(int(name[9:]))
    if name.startswith("tube"):
        return meshgen.tube(length=3.0, radius=1.0, segments=int(name[4:]))
    return meshgen.icosphere(int(name[6:]))


CASES = [
    ("bipyramid3", {}), ("bipyramid9", {}), ("bipyramid17", {}), ("bipyramid32", {}),  # runs of 1, 2, 3 and 4 slots
    ("sphere0", {}), ("sphere2", {}), ("sphere5", {}),  # 12, 162 and 10,242 vertices
    ("tube9", dict(bond_type=1)), ("tube127", dict(bond_type=1)), ("tube140", dict(bond_type=1)),  # open: 45 .. 9,380
    ("sphere4", dict(n_search=1, excl=1, rep_scale=1.6)),  # rows of a few entries
    ("sphere4", dict(n_search=1)),  # nearly empty rows
    ("sphere5", dict(excl=0, rep_scale=1.1)),  # many pairs through the near rows
    ("tube40", dict(bond_type=1, n_search=1, excl=1, rep_scale=1.6)),
]


@pytest.mark.parametrize("name,kw", CASES, ids=["-".join([n] + [f"{k}{v}" for k, v in kw.items()]) for n, kw in CASES])
def test_evaluation_matches_the_oracle(C, name, kw):
    p, f = mesh(name)
    l = meshgen.mean_edge_length(p, f)
    rng = np.random.default_rng(3)
    p = p + rng.normal(0.0, 0.05 * l, size=p.shape)
    prm = workload_params(p, f, **kw)
    mo, mg = O.Mesh(p, f), C.Mesh(p, f)
    eo, eg = O.Energy(mo, O.default_params(**prm)), C.Energy(mg, C.params(**prm))
    d = rng.normal(0.0, 1e-3 * l, size=p.shape)
    mo.points()[:] += d
    mg.points()[:] += d
    e, g = eg.gradient(mg, with_energy=True)
    eref, gref = eo.energy(mo), eo.gradient(mo)
    assert abs(e - eref) <= RTOL * abs(eref)
    assert np.linalg.norm(g - gref) <= RTOL * np.linalg.norm(gref)
    assert eg.energy(mg) == e


@pytest.mark.parametrize("n_search", [0, 1])
def test_exclusions_follow_a_flipped_topology(C, n_search):
    """Pairs excluded when the lists were built are tested again once the
    connectivity has changed: the double-word path trusts a list's exclusions
    only for the topology it was built on, the FP64 path tests every pair of
    a Verlet row."""
    p, f = meshgen.jittered_icosphere(3, seed=2)
    prm = workload_params(p, f, n_search=n_search, excl=1, rep_scale=1.6)
    mg = C.Mesh(p, f)
    eg = C.Energy(mg, C.params(**prm))
    before = eg.energy(mg)
    assert C.flip(mg, eg, 0.5, 4, 1, 256) > 0
    e, g = eg.gradient(mg, with_energy=True)
    assert e != before
    if n_search == 0:
        mo = O.Mesh(p, f)
        eo = O.Energy(mo, O.default_params(**prm))
        assert O.flip_windowed(mo, eo, 0.5, 4, 1, 256) > 0  # the same flips on the oracle's mesh, lists of before
        eref, gref = eo.energy(mo), eo.gradient(mo)
    else:
        eg.set_stencil_precision(0)
        eref, gref = eg.gradient(mg, with_energy=True)
    assert abs(e - eref) <= RTOL * abs(e)
    assert np.linalg.norm(g - gref) <= RTOL * np.linalg.norm(gref)
