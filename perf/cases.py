"""Timed cases of the library: the calls its users make, with the inputs they
make them on, and the same results in plain 64-bit torch.

``listed()`` gives the fixed cases, ``draw(rng)`` one more of the same kinds
and ranges, ``prepare(case, seed)`` what a program holds before the call (mesh,
energy manager, device buffers), ``run(state)`` one call, ``work(case)`` the
bytes and operations the call cannot do without, and ``exact(case, seed)`` its
results from an independent evaluation in 64 bits (None where a flip sweep
makes the result a matter of discrete decisions).

Kinds:
  eval       energy + gradient on device positions (tm_energy_eval_device)
  hmc        one device HMC move (tm_hmc_step_device)
  minimise   a short L-BFGS minimisation on the device (minimize_device)
  chain      one step of a device chain: HMC move, flip sweep, list rebuild
  pflip      one parallel flip sweep through trimem_gb300.core
  host       energy() and gradient() through trimem_gb300.core, host positions
  surrogate  learned force (tm_surrogate_gradient_device)
  train      one Adam step of the learned force
  batch      HMC steps of a batch of replicas
"""
import ctypes
import functools
import math

import numpy as np
import torch

from trimem_gb300 import capi, load_core, meshgen, workloads
from trimem_gb300 import surrogate as S
from trimem_gb300.mc.device import DeviceChain
from trimem_gb300.mc.equilibrate import load_state
from trimem_gb300.mc.minim import minimize_device

JITTER = 0.01 / meshgen.L4_MEAN_EDGE  # vertex noise of the membranes, in mean edge lengths
MOVE = 0.01  # displacement since the neighbour list was built, in mean edge lengths
CALM = 0.01  # vertex noise of the membranes that are sampled: the tether's steep wall is out of reach
STEP = 1e-4  # time step of a move, in mean edge lengths: most moves are accepted


# ---- cases -------------------------------------------------------------------
def listed():
    return [
        # a small vesicle of the test-suite and the replica batch: latency and
        # launches only
        dict(name="eval_small", kind="eval", mesh="sphere", freq=8, stencil=2, bond=0, search=0, excl=2, rep=0.8),
        # an open tube with area bonds and a Verlet list: boundaries, odd
        # sizes, many active repulsion pairs
        dict(name="eval_open_verlet", kind="eval", mesh="tube", segments=97, stencil=2, bond=1, search=1, excl=1,
             rep=1.6),
        # the evaluation loop of the 163,842-vertex membrane
        dict(name="eval_large", kind="eval", mesh="sphere", freq=128, stencil=2, bond=0, search=0, excl=2, rep=0.8),
        # the same loop at 40,962 vertices with plain FP64 stencils
        dict(name="eval_fp64", kind="eval", mesh="sphere", freq=64, stencil=0, bond=0, search=0, excl=2, rep=0.8),
        # sampling a mid-sized membrane: 20 velocity-Verlet steps and the test
        dict(name="hmc_mid", kind="hmc", mesh="sphere", freq=32, stencil=2, bond=0, search=0, excl=2, rep=0.8,
             leapfrog=20),
        # start of a run: minimisation with the list rebuilt at every evaluation
        dict(name="minimise_mid", kind="minimise", mesh="sphere", freq=32, stencil=2, bond=0, search=0, excl=2,
             rep=0.8, maxiter=10),
        # the sampling step of the large membrane at equilibrium
        dict(name="chain_large", kind="chain", leapfrog=20, ratio=0.2),
        # flips of a small membrane from a Python driver of the reference
        dict(name="pflip_small", kind="pflip", mesh="sphere", freq=16, ratio=0.1),
        # the reference's Python drivers: host positions in, energy and
        # gradient out
        dict(name="host_mid", kind="host", mesh="sphere", freq=64),
        # the learned force of the large membrane
        dict(name="surrogate_large", kind="surrogate", mesh="sphere", freq=128),
        # fitting that force
        dict(name="train_mid", kind="train", mesh="sphere", freq=64),
        # a parameter study: membranes of four sizes side by side
        dict(name="batch_mixed", kind="batch", freqs="8,16,32,64", each=4, leapfrog=10, search=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["eval", "eval", "eval", "hmc", "minimise", "chain", "pflip", "host", "surrogate", "train",
                       "batch"])
    if kind == "eval":
        c = dict(kind=kind, stencil=rng.choice([2, 2, 0]), bond=rng.choice([0, 0, 1]), search=rng.choice([0, 0, 1]),
                 excl=rng.choice([1, 2]))
        c["rep"] = rng.choice([0.8, 1.6]) if c["excl"] == 1 else 0.8
        if rng.random() < 0.3:  # open mesh: bonds per face (the reference counts boundary edges one-sidedly)
            return dict(c, mesh="tube", segments=_log_int(rng, 24, 240), bond=1)
        return dict(c, mesh="sphere", freq=_log_int(rng, 4, 127))
    sphere = dict(kind=kind, mesh="sphere")
    if kind == "hmc":
        return dict(sphere, freq=_log_int(rng, 6, 100), stencil=rng.choice([2, 2, 0]), bond=rng.choice([0, 1]),
                    search=0, excl=2, rep=0.8, leapfrog=rng.randrange(5, 26))
    if kind == "minimise":
        return dict(sphere, freq=_log_int(rng, 6, 100), stencil=2, bond=0, search=rng.choice([0, 0, 1]), excl=2,
                    rep=0.8, maxiter=rng.randrange(4, 13))
    if kind == "chain":
        return dict(kind=kind, leapfrog=rng.randrange(5, 20), ratio=round(rng.uniform(0.02, 0.19), 3))
    if kind == "pflip":
        return dict(sphere, freq=_log_int(rng, 6, 64), ratio=round(rng.uniform(0.05, 0.5), 3))
    if kind == "host":
        return dict(sphere, freq=_log_int(rng, 4, 120))
    if kind == "surrogate":
        return dict(sphere, freq=_log_int(rng, 6, 127))
    if kind == "train":
        return dict(sphere, freq=_log_int(rng, 6, 100))
    freqs, each = sorted(_log_int(rng, 5, 60) for _ in range(rng.randrange(1, 5))), rng.randrange(1, 5)
    while each * sum(10 * q * q + 2 for q in freqs) > 200000:  # no larger than the listed batch
        each, freqs = (each - 1, freqs) if each > 1 else (each, freqs[:-1])
    return dict(kind=kind, freqs=",".join(map(str, freqs)), each=each, leapfrog=rng.randrange(4, 11),
                search=rng.choice([0, 0, 1]))


# ---- meshes ------------------------------------------------------------------
@functools.lru_cache(maxsize=None)
def _sphere(freq):
    """Geodesic sphere, every icosahedron edge cut into freq: 10 freq^2 + 2
    vertices (the package's icosphere where freq is a power of two)."""
    if freq & (freq - 1) == 0:
        return meshgen.icosphere(freq.bit_length() - 1)
    v, f = meshgen.icosahedron()
    a = np.arange(freq + 1)
    i, j = [t.ravel() for t in np.meshgrid(a, a, indexing="ij")]
    keep = i + j <= freq
    i, j = i[keep], j[keep]
    at = -np.ones((freq + 1, freq + 1), np.int64)
    at[i, j] = np.arange(len(i))
    up = (i + j) < freq
    tri = [np.stack([at[i[up], j[up]], at[i[up] + 1, j[up]], at[i[up], j[up] + 1]], 1)]
    dn = (i + j) < freq - 1
    tri.append(np.stack([at[i[dn] + 1, j[dn]], at[i[dn] + 1, j[dn] + 1], at[i[dn], j[dn] + 1]], 1))
    tri = np.concatenate(tri)
    pts, faces = [], []
    for k, (p, q, r) in enumerate(f):
        # sine weights keep the edges within 10% of their mean
        w = np.sin(np.stack([freq - i - j, i, j], 1) / freq * math.atan(2.0)) @ v[[p, q, r]]
        pts.append(w / np.linalg.norm(w, axis=1, keepdims=True))
        faces.append(tri + k * len(i))
    pts, faces = np.concatenate(pts), np.concatenate(faces)
    # points on shared edges and corners are one vertex
    _, first, back = np.unique(np.round(pts * 1e7).astype(np.int64), axis=0, return_index=True, return_inverse=True)
    order = np.argsort(np.argsort(first))  # vertices in order of first appearance
    pts = pts[np.sort(first)]
    assert len(pts) == 10 * freq * freq + 2
    return pts, order[back.ravel()][faces].astype(np.int32)


@functools.lru_cache(maxsize=None)
def _tube(segments):
    return meshgen.tube(length=5.0, radius=1.0, segments=segments)


@functools.lru_cache(maxsize=None)
def _mean_edge(kind, n):
    p, f = _sphere(n) if kind == "sphere" else _tube(n)
    return meshgen.mean_edge_length(p, f)


def _base(case):
    n = case["freq"] if case["mesh"] == "sphere" else case["segments"]
    p, f = _sphere(n) if case["mesh"] == "sphere" else _tube(n)
    return p, f, _mean_edge(case["mesh"], n)


def _membrane(case, seed):
    """(points the energy manager is made from, faces, parameters, displaced
    points)."""
    rng = np.random.default_rng(seed)
    p, f, l = _base(case)
    calm = case["kind"] == "hmc"
    p = p + rng.normal(0.0, (CALM if calm else JITTER) * l, size=p.shape)
    prm = workloads.workload_params(p, f, kappa_b=20.0, vfrac=0.8, bond_type=case.get("bond", 0),
                                    n_search=case.get("search", 0), excl=case.get("excl", 2),
                                    rep_scale=case.get("rep", 0.8))
    return p, f, prm, p + rng.normal(0.0, (0.1 * CALM if calm else MOVE) * l, size=p.shape)


def _time_step(case):
    freq = case["freq"] if "freq" in case else max(map(int, case["freqs"].split(",")))
    return STEP * _mean_edge("sphere", freq)


def _counts(case):
    if case["mesh"] == "sphere":
        v = 10 * case["freq"] ** 2 + 2
        return v, 3 * v - 6, 2 * v - 4
    s = case["segments"]
    rings = int(5.0 // (2.0 * math.pi / s)) + 1
    return s * rings, 3 * s * (rings - 1) + s, 2 * s * (rings - 1)


@functools.lru_cache(maxsize=None)
def _stream():
    return torch.cuda.Stream()


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


# ---- prepare -----------------------------------------------------------------
def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case, kind=kind, stream=_stream())
    if kind == "chain":
        p, f, prm = _large()
        eq = _equilibrated()
        rng = np.random.default_rng(seed)
        l = prm["bond_lc0"] / 1.15
        x = eq["x"] + rng.normal(0.0, 1e-3 * l, size=eq["x"].shape)
        st["mesh"] = capi.Mesh(x, eq["faces"])
        st["energy"] = capi.Energy(st["mesh"], capi.params(**prm))
        st["energy"].set_initial_props(eq["initial"])
        st["x"] = torch.tensor(x, dtype=torch.float64, device="cuda")
        st["chain"] = DeviceChain(st["mesh"], st["energy"], st["x"], dt=2e-6, n_leapfrog=case["leapfrog"],
                                  flip_ratio=case["ratio"], seed=seed % 100003, stream=st["stream"].cuda_stream)
        return st
    if kind == "batch":
        reps = _replicas(case, seed)
        st["batch"] = capi.Batch([(p, f) for p, f, _ in reps], [capi.params(**prm) for _, _, prm in reps])
        st["seed"] = seed % 100003
        return st
    p, f, prm, x = _membrane(case, seed)
    if kind in ("host", "pflip"):
        core = load_core()
        st["core"] = core
        st["mesh"] = core.TriMesh(p, f)
        st["energy"] = core.EnergyManager(st["mesh"], _core_params(core, prm))
        st["x"] = x
        st["sweep"] = 1000 * (seed % 100003)
        return st
    st["mesh"] = capi.Mesh(p, f)
    st["energy"] = capi.Energy(st["mesh"], capi.params(**prm))
    st["x"] = torch.tensor(x, dtype=torch.float64, device="cuda")
    if kind in ("eval", "hmc", "minimise"):
        st["energy"].set_stencil_precision(case["stencil"])
    if kind in ("eval", "surrogate"):
        st["grad"] = torch.empty_like(st["x"])
        st["e"] = torch.empty(1, dtype=torch.float64, device="cuda")
    if kind == "hmc":
        st["seed"], st["step"] = seed % 100003, 0
        st["u"] = float(np.random.default_rng(seed + 1).uniform())
    if kind == "minimise":
        st["x0"] = st["x"].clone()
    if kind in ("surrogate", "train"):
        st["blob"] = _weights(p, f, seed)
        st["net"] = capi.Surrogate(st["mesh"], st["blob"])
    if kind == "train":
        st["inputs"] = S.Inputs(st["net"], st["energy"], st["mesh"], st["x"], 16)
        gen = torch.Generator(device="cuda").manual_seed(seed)
        st["inputs"].target = torch.randn(len(p), 3, device="cuda", generator=gen)
        st["trainer"] = S.DeviceTrainer(len(p), 16, st["blob"])
        st["loss"] = torch.empty(1, device="cuda")
    return st


@functools.lru_cache(maxsize=None)
def _large():
    return workloads.very_large_mesh()


@functools.lru_cache(maxsize=None)
def _equilibrated():
    p, _, prm = _large()
    st = load_state(prm, len(p))
    assert st is not None
    return st


def _replicas(case, seed):
    rng = np.random.default_rng(seed)
    reps = []
    for freq in map(int, case["freqs"].split(",")):
        for _ in range(case["each"]):
            p, f = _sphere(freq)
            p = p + rng.normal(0.0, CALM * _mean_edge("sphere", freq), size=p.shape)
            reps.append((p, f, workloads.workload_params(p, f, kappa_b=float(rng.uniform(10, 50)),
                                                         vfrac=float(rng.uniform(0.6, 0.95)),
                                                         n_search=case["search"])))
    return reps


def _core_params(core, prm):
    bp, rp, cp = core.BondParams(), core.SurfaceRepulsionParams(), core.ContinuationParams()
    bp.lc0, bp.lc1, bp.a0, bp.r = prm["bond_lc0"], prm["bond_lc1"], prm["bond_a0"], prm["bond_r"]
    bp.type = core.BondType.Edge if prm["bond_type"] == 0 else core.BondType.Area
    rp.lc1, rp.r, rp.rlist, rp.exclusion_level = prm["rep_lc1"], prm["rep_r"], prm["rlist"], prm["exclusion_level"]
    rp.n_search = "cell-list" if prm["n_search"] == 0 else "verlet-list"
    cp.delta, cp.lam = prm["cont_delta"], prm["cont_lambda"]
    ep = core.EnergyParams()
    for k in ("kappa_b", "kappa_a", "kappa_v", "kappa_c", "kappa_t", "kappa_r", "area_frac", "volume_frac",
              "curvature_frac"):
        setattr(ep, k, prm[k])
    ep.bond_params, ep.repulse_params, ep.continuation_params = bp, rp, cp
    return ep


def _weights(p, f, seed):
    """Weight blob of an untrained network for this membrane."""
    torch.manual_seed(seed)
    net = S.make_net()
    lbar, abar = S.mesh_scales(p, f)
    with torch.no_grad():
        net.scales.copy_(torch.tensor([lbar, abar, 50.0]))
        net.wo.normal_(0, 0.3)
        net.wn.normal_(0, 0.3)
    return S.to_blob(net)


# ---- run ---------------------------------------------------------------------
def run(st):
    kind, L = st["kind"], capi.lib()
    stream = ctypes.c_void_p(st["stream"].cuda_stream)
    if kind == "eval":
        capi.check(L.tm_energy_eval_device(st["energy"].h, st["mesh"].h, _ptr(st["x"]), _ptr(st["grad"]),
                                           _ptr(st["e"]), stream))
        return {"energy": st["e"], "grad": st["grad"]}
    if kind == "hmc":
        out4, props = (ctypes.c_double * 4)(), (ctypes.c_double * 6)()
        capi.check(L.tm_hmc_step_device(st["energy"].h, st["mesh"].h, _ptr(st["x"]), 1.0,
                                        _time_step(st["case"]), st["case"]["leapfrog"], 1.0, st["seed"], st["step"], st["u"], out4, props,
                                        stream))
        st["step"] += 1
        return {"accepted": int(out4[0]), "hamiltonian": np.array(out4[1:3]), "energy": out4[3],
                "props": np.array(props[:]), "x": st["x"]}
    if kind == "minimise":
        with torch.cuda.stream(st["stream"]):
            st["x"].copy_(st["x0"])  # a run starts from the membrane it is given
        it, e = minimize_device(st["energy"], st["mesh"], st["x"], maxiter=st["case"]["maxiter"],
                                stream=st["stream"].cuda_stream)
        return {"iterations": it, "energy": e, "x": st["x"]}
    if kind == "chain":
        ch = st["chain"]
        before = ch.flips
        acc, props, e = ch.step()
        return {"accepted": int(acc), "flips": ch.flips - before, "props": props, "energy": e, "x": st["x"]}
    if kind == "pflip":
        st["sweep"] += 1
        n = st["core"].pflip(st["mesh"], st["energy"], st["case"]["ratio"], seed=st["sweep"])
        return {"flips": int(n), "faces": st["mesh"].fv_indices()}
    if kind == "host":
        st["mesh"].points()[:] = st["x"]
        return {"energy": st["energy"].energy(st["mesh"]), "grad": st["energy"].gradient(st["mesh"])}
    if kind == "surrogate":
        capi.check(L.tm_surrogate_gradient_device(st["net"].h, st["energy"].h, st["mesh"].h, _ptr(st["x"]),
                                                  _ptr(st["grad"]), stream))
        return {"grad": st["grad"]}
    if kind == "train":
        st["trainer"].step(st["inputs"], 1.0, lr=1e-3, loss_out=st["loss"], stream=st["stream"].cuda_stream)
        return {"loss": st["loss"], "weights": st["trainer"].weights()}
    assert kind == "batch"
    acc = st["batch"].hmc(2, st["case"]["leapfrog"], _time_step(st["case"]), seed=st["seed"])
    return {"accepted": acc, "x": np.concatenate(st["batch"].positions()), "energy": st["batch"].energy()}


# ---- work --------------------------------------------------------------------
# Operations per vertex of one energy + gradient evaluation: 2 faces of about
# 60, 3 edges of about 70, 6 ring slots of about 60, sums and penalties.
EVAL_FLOPS = 700
# forward pass of the learned force: embedding, three rounds of six messages
# and one 128 x 64 layer, output head
NET_FLOPS = 2 * (8 * 64 + 3 * (6 * 64 * 6 + 128 * 64) + 7 * 128)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        v = sum(10 * f * f + 2 for f in map(int, case["freqs"].split(","))) * case["each"]
        return {"bytes": v * (24 + 72 + 24) + 4 * case["each"], "flops": (2 * (case["leapfrog"] + 1) + 1) * EVAL_FLOPS * v}
    if kind == "chain":
        v = 163842
        # positions in and out, topology in and out, each proposal's quad
        # re-evaluated before and after the flip
        return {"bytes": v * (48 + 144), "flops": (case["leapfrog"] + 2) * EVAL_FLOPS * v +
                3 * v * case["ratio"] * 8 * EVAL_FLOPS}
    v, e, f = _counts(case)
    topo = 12 * f + 16 * e
    if kind == "eval":
        return {"bytes": 48 * v + topo + 8, "flops": EVAL_FLOPS * v}
    if kind == "hmc":
        return {"bytes": 48 * v + topo + 80, "flops": (case["leapfrog"] + 1) * EVAL_FLOPS * v}
    if kind == "minimise":
        it = case["maxiter"]
        return {"bytes": 48 * v + topo, "flops": (it + 1) * EVAL_FLOPS * v + it * 6 * it * 3 * v}
    if kind == "pflip":
        return {"bytes": 24 * v + 2 * topo + 12 * f, "flops": (EVAL_FLOPS + 3 * case["ratio"] * 8 * EVAL_FLOPS) * v}
    if kind == "host":
        return {"bytes": 48 * v + topo + 8, "flops": EVAL_FLOPS * v}
    if kind == "surrogate":
        return {"bytes": 48 * v + topo, "flops": (EVAL_FLOPS + NET_FLOPS) * v}
    # train: features, rings (six neighbours, edge features, directions), targets in
    return {"bytes": v * (32 + 16 + 6 * (4 + 16 + 12) + 12) + 8 * S.BLOB_SIZE, "flops": 3 * NET_FLOPS * v}


# ---- the same results in 64 bits -----------------------------------------------
class _Energy:
    """Membrane energy in float64 torch; gradients by autograd."""

    def __init__(self, p, f, prm, device="cuda"):
        self.prm, self.nv = prm, len(p)
        t = lambda a: torch.tensor(np.ascontiguousarray(a), device=device)
        f = f.astype(np.int64)
        self.f = t(f)
        # undirected edges with the corner opposite on either side
        d = np.concatenate([f[:, [0, 1]], f[:, [1, 2]], f[:, [2, 0]]])
        opp = np.concatenate([f[:, 2], f[:, 0], f[:, 1]])
        fwd = d[:, 0] < d[:, 1]
        key = np.where(fwd, d[:, 0] * len(p) + d[:, 1], d[:, 1] * len(p) + d[:, 0])
        uniq, inv = np.unique(key, return_inverse=True)
        ab = np.stack([uniq // len(p), uniq % len(p)], 1)
        left, right = -np.ones(len(uniq), np.int64), -np.ones(len(uniq), np.int64)
        left[inv[fwd]] = opp[fwd]
        right[inv[~fwd]] = opp[~fwd]
        self.edges = t(ab)
        inner = (left >= 0) & (right >= 0)
        self.ie, self.il, self.ir = t(ab[inner]), t(left[inner]), t(right[inner])
        # ring table for the exclusion test
        val = np.bincount(ab.ravel(), minlength=len(p))
        order = np.argsort(np.concatenate([ab[:, 0], ab[:, 1]]), kind="stable")
        flat = np.concatenate([ab[:, 1], ab[:, 0]])[order]
        ring = -np.ones((len(p), val.max()), np.int64)
        start = np.concatenate([[0], np.cumsum(val)[:-1]])
        rows = np.repeat(np.arange(len(p)), val)
        ring[rows, np.arange(len(flat)) - start[rows]] = flat
        self.ring = t(ring)
        self.ref = None
        q = self.props(t(p.astype(np.float64)))
        lam = prm["cont_lambda"]
        self.ref = [float(q[k]) * (1 - lam * (1 - prm[n]))
                    for k, n in enumerate(("area_frac", "volume_frac", "curvature_frac"))]

    def pairs(self, x):
        """Pairs i < j closer than the repulsion cut-off, not excluded."""
        lc1, out = self.prm["rep_lc1"], []
        if not lc1 > 0:
            return torch.zeros(0, 2, dtype=torch.int64, device=x.device)
        xs = x.detach()
        # only vertices in the same or a neighbouring slab along x can be close
        order = torch.argsort(xs[:, 0])
        xo = xs[order]
        first = xo[:, 0].contiguous()
        hi = torch.searchsorted(first, first + lc1, right=True)
        B = 1024
        for a in range(0, len(xo), B):
            b = int(hi[min(a + B, len(xo)) - 1])
            s = torch.cdist(xo[a:a + B].float(), xo[a:b].float(), compute_mode="donot_use_mm_for_euclid_dist")
            i, j = torch.nonzero(s < lc1 * (1 + 1e-4), as_tuple=True)
            k = j > i
            out.append(torch.stack([order[a + i[k]], order[a + j[k]]], 1))
        ij = torch.cat(out)
        ij = ij[(xs[ij[:, 0]] - xs[ij[:, 1]]).norm(dim=1) < lc1]
        excl = self.prm["exclusion_level"]
        if excl >= 1:
            r = self.ring[ij[:, 0]]
            bad = (r == ij[:, 1:]).any(1)
            if excl >= 2:
                rr = self.ring[r.clamp(min=0)].masked_fill((r < 0)[:, :, None], -1)
                bad |= (rr == ij[:, 1, None, None]).any(2).any(1)
            ij = ij[~bad]
        return ij

    def props(self, x):
        """The six global sums; also keeps curvature / area per vertex."""
        p, nv = self.prm, self.nv
        a, b, c = x[self.f[:, 0]], x[self.f[:, 1]], x[self.f[:, 2]]
        N = torch.linalg.cross(b - a, c - a)
        A = 0.5 * N.norm(dim=1)
        V = (torch.linalg.cross(a, b) * c).sum(1) / 6
        va = torch.zeros(nv, dtype=x.dtype, device=x.device)
        for k in range(3):
            va = va.index_add(0, self.f[:, k], A / 3)
        i, j = x[self.ie[:, 0]], x[self.ie[:, 1]]
        e = j - i
        l = e.norm(dim=1)
        # (i, j, left) and (j, i, right) are the faces of the edge
        n0 = torch.linalg.cross(e, x[self.il] - i)
        n1 = torch.linalg.cross(x[self.ir] - i, e)
        th = torch.atan2((torch.linalg.cross(n0, n1) * e).sum(1) / l, (n0 * n1).sum(1))
        vc = torch.zeros(nv, dtype=x.dtype, device=x.device)
        for k in range(2):
            vc = vc.index_add(0, self.ie[:, k], 0.25 * l * th)
        if p["bond_type"] == 0:
            le = (x[self.edges[:, 1]] - x[self.edges[:, 0]]).norm(dim=1)
            T = self._flat(le, p["bond_lc0"], p["bond_lc1"], p["bond_r"])
        else:
            T = ((A / p["bond_a0"] - 1) ** 2).sum()
        ij = self.pairs(x)
        d = (x[ij[:, 0]] - x[ij[:, 1]]).norm(dim=1)
        R = 2 * (torch.exp(d / (d - p["rep_lc1"])) / d ** p["rep_r"]).sum()
        self.th, self.l, self.rho, self.A, self.N, self.va = th, l, vc / va, A, N, va
        return torch.stack([A.sum(), V.sum(), vc.sum(), (2 * vc * vc / va).sum(), T, R])

    @staticmethod
    def _flat(l, lc0, lc1, r):
        long, short = l[l > lc0], l[l < lc1]
        return (r ** (r + 1) * (long - lc0) ** r).sum() + (torch.exp(short / (short - lc1)) / short ** r).sum()

    def energy(self, x, local=False):
        p, q = self.prm, self.props(x)
        e = sum(p[k] * (q[n] / self.ref[n] - 1) ** 2 for n, k in enumerate(("kappa_a", "kappa_v", "kappa_c")))
        e = e + p["kappa_t"] * q[4]
        return e if local else e + p["kappa_b"] * q[3] + p["kappa_r"] * q[5]

    def energy_grad(self, x, local=False):
        x = x.detach().clone().requires_grad_(True)
        e = self.energy(x, local)
        g, = torch.autograd.grad(e, x)
        return float(e.detach()), g


def _mix(z):
    with np.errstate(over="ignore"):
        z = np.uint64(z) + np.uint64(0x9E3779B97F4A7C15)
        z = (z ^ (z >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        z = (z ^ (z >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return z ^ (z >> np.uint64(31))


def _momenta(nv, seed, step):
    """The documented stream: SplitMix64 of (seed, step, pair), Box-Muller."""
    with np.errstate(over="ignore"):
        k = _mix(_mix(seed) ^ _mix(np.uint64(step) + np.uint64(0x632BE59BD9B4E019)))
    a = _mix(k ^ np.arange((3 * nv + 1) // 2, dtype=np.uint64))
    b = _mix(a)
    r = np.sqrt(-2 * np.log(((a >> np.uint64(11)).astype(np.float64) + 1) * 2.0 ** -53))
    t = 2 * np.pi * ((b >> np.uint64(11)).astype(np.float64) * 2.0 ** -53)
    return np.stack([r * np.cos(t), r * np.sin(t)], 1).ravel()[:3 * nv].reshape(nv, 3)


def _verlet(en, x, p, dt, n):
    """(H at the start, H at the end, energies, end positions)"""
    e0, g = en.energy_grad(x)
    h0, y = e0 + 0.5 * float((p * p).sum()), x
    e1 = e0
    for _ in range(n):
        y = y + p * dt - 0.5 * g * dt * dt
        e1, g1 = en.energy_grad(y)
        p = p - 0.5 * (g + g1) * dt
        g = g1
    return h0, e1 + 0.5 * float((p * p).sum()), e0, e1, y


def exact(case, seed):
    kind = case["kind"]
    if kind in ("chain", "pflip"):
        return None
    dev = lambda a: torch.tensor(a, dtype=torch.float64, device="cuda")
    if kind == "batch":
        return _exact_batch(case, seed)
    p, f, prm, x = _membrane(case, seed)
    en = _Energy(p, f, prm)
    x = dev(x)
    if kind in ("eval", "host"):
        e, g = en.energy_grad(x)
        return {"energy": e if kind == "host" else dev([e]), "grad": g if kind == "eval" else g.cpu().numpy()}
    if kind == "hmc":
        mom = dev(_momenta(len(p), seed % 100003, 0))
        h0, h1, e0, e1, y = _verlet(en, x, mom, _time_step(case), case["leapfrog"])
        u = float(np.random.default_rng(seed + 1).uniform())
        ok = u <= math.exp(min(0.0, -(h1 - h0)))
        y = y if ok else x
        return {"accepted": int(ok), "hamiltonian": np.array([h0, h1]), "energy": e1 if ok else e0,
                "props": en.props(y).cpu().numpy(), "x": y}
    if kind == "minimise":
        it, e, y = _lbfgs(en, x, case["maxiter"])
        return {"iterations": it, "energy": e, "x": y}
    blob = _weights(p, f, seed).astype(np.float64)
    net = _Net(blob, en, x)
    if kind == "surrogate":
        _, g = en.energy_grad(x, local=True)
        return {"grad": g - net.force(net.theta)}
    gen = torch.Generator(device="cuda").manual_seed(seed)
    target = torch.randn(len(p), 3, device="cuda", generator=gen).double()
    th = net.theta.clone().requires_grad_(True)
    loss = ((net.force(th) - target) ** 2).mean()
    g, = torch.autograd.grad(loss, th)
    w = net.theta - 1e-3 * g / (g.abs() + 1e-8)  # the first step of Adam
    return {"loss": loss.detach().reshape(1), "weights": np.concatenate([blob[:8], w.cpu().numpy()])}


def _exact_batch(case, seed):
    reps = _replicas(case, seed)
    off = np.concatenate([[0], np.cumsum([-(-len(p) // 256) * 256 for p, _, _ in reps])])
    mom = [_momenta(int(off[-1]), seed % 100003, k) for k in range(2)]
    xs, es, acc = [], [], []
    for r, (p, f, prm) in enumerate(reps):
        en = _Energy(p, f, prm)
        x, n, e = torch.tensor(p, device="cuda"), 0, 0.0
        for k in range(2):
            h0, h1, e0, e1, y = _verlet(en, x, torch.tensor(mom[k][off[r]:off[r] + len(p)], device="cuda"),
                                        _time_step(case), case["leapfrog"])
            with np.errstate(over="ignore"):
                z = _mix(_mix(np.uint64(seed % 100003) ^ np.uint64(0xA5A5A5A5)) ^ _mix(np.uint64(131 * k + r)))
            ok = float(z >> np.uint64(11)) * 2.0 ** -53 <= math.exp(min(0.0, -(h1 - h0)))
            x, e, n = (y, e1, n + 1) if ok else (x, e0, n)
        xs.append(x.cpu().numpy())
        es.append(e)
        acc.append(n)
    return {"accepted": np.array(acc, np.int32), "x": np.concatenate(xs), "energy": np.array(es)}


def _lbfgs(en, x, maxiter, history=10, gtol=1e-5, ftol=2.220446049250313e-09):
    """L-BFGS with Armijo backtracking, first step limited to a move of 1e-3."""
    f, g = en.energy_grad(x)
    pairs, gamma, k = [], 1.0, 0
    while k < maxiter and float(g.abs().max()) > gtol:
        d, alpha = -g, []
        for s, y in reversed(pairs):
            a = float((s * d).sum()) / float((s * y).sum())
            alpha.append(a)
            d = d - a * y
        d = gamma * d
        for (s, y), a in zip(pairs, reversed(alpha)):
            d = d + (a - float((y * d).sum()) / float((s * y).sum())) * s
        gd = float((g * d).sum())
        if not gd < 0:
            d, pairs, gamma = -g, [], 1.0
            gd = float((g * d).sum())
        a = 1.0 if pairs else min(1.0, 1e-3 / float(g.abs().max()))
        for _ in range(40):
            fn, gn = en.energy_grad(x + a * d)
            if math.isfinite(fn) and fn <= f + 1e-4 * a * gd:
                break
            a *= 0.5
        else:
            break
        s, y = (x + a * d) - x, gn - g
        x, g, fp, f = x + a * d, gn, f, fn
        if float((s * y).sum()) > 1e-300:
            gamma = float((s * y).sum()) / float((y * y).sum())
            pairs = (pairs + [(s, y)])[-history:]
        k += 1
        if fp - f <= ftol * max(abs(fp), abs(f), 1.0):
            break
    return k, f, x


class _Net:
    """The learned force in float64 torch, from the weight blob and the
    geometry."""

    def __init__(self, blob, en, x):
        self.lbar, self.abar, self.scale = blob[5:8]
        self.theta = torch.tensor(blob[8:], device=x.device)
        en.props(x)
        nv = en.nv
        i, j = en.ie[:, 0], en.ie[:, 1]
        self.src, self.dst = torch.cat([i, j]), torch.cat([j, i])  # both directions
        l, th, rho = torch.cat([en.l, en.l]), torch.cat([en.th, en.th]), en.rho
        d = x[self.dst] - x[self.src]
        self.dirs = d / d.norm(dim=1, keepdim=True)
        lr = l / self.lbar
        add = lambda v: torch.zeros(nv, dtype=x.dtype, device=x.device).index_add(0, self.src, v)
        deg = add(torch.ones_like(l))
        ls, l2, ths, th2 = add(lr) / deg, add(lr * lr) / deg, add(th) / deg, add(th * th) / deg
        rl = rho * self.lbar
        self.u = torch.stack([en.va / self.abar - 1, rl, rl * rl, (deg - 6) / 6, ths, th2.sqrt(), ls - 1,
                              (l2 - ls * ls).clamp(min=0).sqrt()], 1)
        self.e = torch.stack([lr - 1, th, (rho[self.dst] - rho[self.src]) * self.lbar,
                              0.5 * (rho[self.dst] + rho[self.src]) * self.lbar], 1)
        n = torch.zeros(nv, 3, dtype=x.dtype, device=x.device)
        for k in range(3):
            n = n.index_add(0, en.f[:, k], 0.5 * en.N)
        self.n = n / n.norm(dim=1, keepdim=True)

    def force(self, th):
        silu = torch.nn.functional.silu
        at = 0

        def take(*shape):
            nonlocal at
            v = th[at:at + math.prod(shape)].reshape(shape)
            at += math.prod(shape)
            return v

        win, bin_ = take(64, 8), take(64)
        h = silu(self.u @ win.t() + bin_)
        for _ in range(3):
            we, be, w, b = take(64, 4), take(64), take(64, 128), take(64)
            m = torch.zeros_like(h).index_add(0, self.src, (self.e @ we.t() + be) * h[self.dst])
            h = h + silu(torch.cat([h, m], 1) @ w.t() + b)
        wo, bo, wn, bn = take(64), take(1), take(64), take(1)
        c = (h[self.src] * h[self.dst]) @ wo + bo
        F = torch.zeros_like(self.n).index_add(0, self.src, c[:, None] * self.dirs)
        return self.scale * (F + (h @ wn + bn)[:, None] * self.n)
