"""Timed cases of the step and its analysis, through the package's public entry points.

A case is one of eight kinds of program:

* ``dropin``   a simulation loop that calls ``updates.SRK2_force_calc`` on host populations, as the
  reference's control loop does, one call per output interval;
* ``sweep``    a parameter sweep of independent 2D systems in one ``Batch`` (n_chains log-uniform in
  [50, 4000], chain length uniform in [5, 40], area fraction in [0.1, 0.4]);
* ``lj2d``     one large 2D box of attracting (LJ) chiral chains in a ``Batch``;
* ``lj3d``     one 3D box of attracting chains with rotationally diffusing propulsion;
* ``pops``     boxes of chains and passive beads, two coupled populations a box;
* ``motors``   boxes of passive chains pushed by motors;
* ``srk4``     the sweep's systems under the fourth-order update;
* ``analysis`` the observables of one stored 2D state: order parameters, chain frames, g(r), Cvv, Cnn.

Sizes are those of the benchmark workloads and the tests, from the 2000-bead single system to the
256-system sweep.  States are laid without overlaps, as a stored, relaxed run would have them:
chains in wavy lanes one contact distance apart, in random slots, so that neighbours in space are
not neighbours in memory; 2D LJ chains in bundles.  Every step follows the adaptive dt rule.

``exact`` restates the step in 64 bits with torch operations and nothing of the package.
"""
import math
from types import SimpleNamespace

import numpy as np
import torch

from gliding_collective_rotation_b200 import config, observables, updates
from gliding_collective_rotation_b200.batch import Batch
from gliding_collective_rotation_b200.engine import SystemParams
from gliding_collective_rotation_b200.workloads import SystemSpec

BOND = 0.5                       # bond rest length
LJ_CUT = 2.5 / 2 ** (1 / 6)      # 2.5 sigma in units of the repulsion diameter


# ---------------------------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------------------------
def listed():
    return [
        # the reference's own use: the 2000-bead system in FP64, 40 steps (one list interval) a call
        {"name": "dropin_2k_fp64", "kind": "dropin", "n_chains": 200, "clen": 10, "phi": 0.3056, "steps": 40,
         "precision": "fp64"},
        # one small mixed-precision system stepped on its own: launch latency is all of it
        {"name": "one_2k_mixed", "kind": "sweep", "n_systems": 1, "n_chains": 200, "clen": 10, "phi": 0.3056,
         "steps": 100, "precision": "mixed", "series": 0},
        # a handful of sweep points with the order-parameter series recorded, as a served request asks for it
        {"name": "sweep_9_series_mixed", "kind": "sweep", "n_systems": 9, "n_chains": 0, "clen": 0, "phi": 0.0,
         "steps": 60, "precision": "mixed", "series": 20},
        # the whole sweep: the throughput workload
        {"name": "sweep_256_mixed", "kind": "sweep", "n_systems": 256, "n_chains": 0, "clen": 0, "phi": 0.0,
         "steps": 40, "precision": "mixed", "series": 0},
        # part of the sweep in FP64, the precision that results are checked in
        {"name": "sweep_64_fp64", "kind": "sweep", "n_systems": 64, "n_chains": 0, "clen": 0, "phi": 0.0,
         "steps": 20, "precision": "fp64", "series": 0},
        # one large box of attracting chains: long neighbour lists
        {"name": "lj2d_500k_mixed", "kind": "lj2d", "n_chains": 20000, "clen": 25, "phi": 0.26, "steps": 40,
         "precision": "mixed", "pair_mode": 1},
        # a mid-size ragged box of the same kind in FP64
        {"name": "lj2d_37k_fp64", "kind": "lj2d", "n_chains": 1637, "clen": 23, "phi": 0.31, "steps": 40,
         "precision": "fp64", "pair_mode": 0},
        # the 3D box of a million beads
        {"name": "lj3d_1m_mixed", "kind": "lj3d", "n_chains": 40000, "clen": 25, "side": 200.0, "steps": 20,
         "precision": "mixed"},
        # chains and passive beads in one box: coupled populations
        {"name": "pops_128_mixed", "kind": "pops", "n_boxes": 128, "steps": 40, "precision": "mixed"},
        # chains pushed by motors
        {"name": "motors_16_mixed", "kind": "motors", "n_boxes": 16, "steps": 40, "precision": "mixed"},
        # the fourth-order update on sweep systems
        {"name": "srk4_16_mixed", "kind": "srk4", "n_systems": 16, "steps": 20, "precision": "mixed"},
        # the analysis of a stored state of the sweep's largest kind
        {"name": "analysis_4k_chains", "kind": "analysis", "n_chains": 4000, "clen": 13, "phi": 0.3, "binsize": 0.25,
         "precision": "mixed"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dropin", "one", "sweep", "sweep", "lj2d", "lj3d", "pops", "motors", "srk4", "analysis"])
    precision = rng.choice(["mixed", "mixed", "fp64"])
    if kind == "dropin":
        return {"kind": kind, "n_chains": _log(rng, 50, 4000), "clen": rng.randint(5, 40),
                "phi": round(rng.uniform(0.1, 0.4), 3), "steps": rng.randint(10, 60), "precision": precision}
    if kind == "one":
        return {"kind": "sweep", "n_systems": 1, "n_chains": _log(rng, 50, 4000), "clen": rng.randint(5, 40),
                "phi": round(rng.uniform(0.1, 0.4), 3), "steps": rng.randint(20, 100), "precision": precision,
                "series": rng.choice([0, 10])}
    if kind == "sweep":
        return {"kind": kind, "n_systems": _log(rng, 2, 200), "n_chains": 0, "clen": 0, "phi": 0.0,
                "steps": rng.randint(10, 50), "precision": precision, "series": rng.choice([0, 0, 10])}
    if kind == "lj2d":
        return {"kind": kind, "n_chains": _log(rng, 400, 20000), "clen": rng.randint(10, 40),
                "phi": round(rng.uniform(0.15, 0.35), 3), "steps": rng.randint(10, 30), "precision": precision,
                "pair_mode": rng.choice([0, 1])}
    if kind == "lj3d":
        n, clen = _log(rng, 600, 36000), rng.randint(10, 27)
        return {"kind": kind, "n_chains": n, "clen": clen,
                "side": round(max((n * clen / 0.125) ** (1 / 3), 2.2 * (BOND * (clen - 1) + 1.1)), 3),
                "steps": rng.randint(5, 15), "precision": precision}
    if kind == "pops":
        return {"kind": kind, "n_boxes": _log(rng, 1, 128), "steps": rng.randint(10, 40), "precision": precision}
    if kind == "motors":
        return {"kind": kind, "n_boxes": _log(rng, 1, 64), "steps": rng.randint(10, 40), "precision": precision}
    if kind == "srk4":
        return {"kind": kind, "n_systems": _log(rng, 1, 32), "steps": rng.randint(5, 25), "precision": precision}
    return {"kind": "analysis", "n_chains": _log(rng, 50, 12000), "clen": rng.randint(5, 40),
            "phi": round(rng.uniform(0.1, 0.4), 3), "binsize": rng.choice([0.125, 0.25, 0.5]), "precision": precision}


# ---------------------------------------------------------------------------------------------
# states
# ---------------------------------------------------------------------------------------------
def _fill(rng, n, lanes, slots, bundle):
    """n of the lanes x slots places of chains: at random, or bundles of neighbouring lanes together."""
    if lanes * slots < n:
        raise ValueError("the box does not hold the chains")
    key = rng.random((lanes, slots))
    if bundle > 1:
        key = 1e-3 * key + rng.random((lanes // bundle + 1, slots // 2 + 1))[np.arange(lanes)[:, None] // bundle,
                                                                              np.arange(slots)[None, :] // 2]
    order = np.argsort(key.ravel())
    pick = order[:n].copy()
    rng.shuffle(pick)
    return pick, order[n:]


def _lay2d(rng, n_chains, clen, L, bundle=1):
    """Chains in wavy lanes along x, 1.02 apart or more; the free places come too."""
    extent = BOND * (clen - 1) + 1.04
    lanes, slots = int(L / 1.02), int(L / extent)
    pick, free = _fill(rng, n_chains, lanes, slots, bundle)
    gap, pitch = L / lanes, L / slots
    amp = 0.02 * L / (2 * math.pi)
    phase = rng.uniform(0, 2 * math.pi)

    def place(u, v):  # along the lane, across the lanes
        return np.stack([u, v + amp * np.sin(2 * math.pi * u / L + phase)], axis=-1)

    j = np.arange(clen) - 0.5 * (clen - 1)
    way = np.where(rng.random(n_chains) < 0.5, 1.0, -1.0)
    shift = (pitch - extent) * (rng.random(n_chains) - 0.5)
    u = ((pick % slots) + 0.5) * pitch + shift
    u = u[:, None] - way[:, None] * BOND * j[None, :] + rng.normal(0, 0.006, (n_chains, clen))
    v = ((pick // slots) + 0.5)[:, None] * gap + rng.normal(0, 0.004, (n_chains, clen))
    v = v + 0.015 * np.sin(1.3 * j[None, :] + rng.uniform(0, 2 * math.pi, (n_chains, 1)))
    pos = np.mod(place(u, v), L).reshape(-1, 2)
    spot = place(((free % slots) + 0.5) * pitch, ((free // slots) + 0.5) * gap)
    tan = np.zeros((n_chains * clen, 2))
    tan[:, 0] = np.repeat(way, clen)
    return pos, tan, np.repeat(np.arange(n_chains), clen), np.mod(spot, L), extent


def _lay3d(rng, n_chains, clen, L):
    """Chains in lanes along x on a square lattice of lanes, in random slots; propulsion directions at random."""
    extent = BOND * (clen - 1) + 1.05
    m, slots = int(L / 1.04), int(L / extent)
    gap, pitch = L / m, L / slots
    pick, _ = _fill(rng, n_chains, m * m, slots, 1)
    a, b, s = pick // (m * slots), pick // slots % m, pick % slots
    way = np.where(rng.random(n_chains) < 0.5, 1.0, -1.0)
    j = np.arange(clen) - 0.5 * (clen - 1)
    u = (s + 0.5) * pitch + (pitch - extent) * (rng.random(n_chains) - 0.5)
    pos = np.empty((n_chains, clen, 3))
    pos[..., 0] = u[:, None] - way[:, None] * BOND * j + rng.normal(0, 0.006, (n_chains, clen))
    for axis, lane in ((1, a), (2, b)):
        wave = 0.012 * np.sin(1.1 * j[None, :] + rng.uniform(0, 2 * math.pi, (n_chains, 1)))
        pos[..., axis] = ((lane + 0.5) * gap)[:, None] + wave + rng.normal(0, 0.004, (n_chains, clen))
    t = rng.normal(size=(n_chains, 3))
    t = (t / np.linalg.norm(t, axis=1, keepdims=True)).astype(np.float32).astype(np.float64)
    return np.mod(pos.reshape(-1, 3), L), np.repeat(t, clen, axis=0), np.repeat(np.arange(n_chains), clen)


def _wca(radius, eps, cutoff):
    r6 = radius ** 6
    return np.array([12 * eps * r6, 12 * eps * r6 * r6, 0.0, cutoff * radius])


def _spec(name, dim, pos, tan, chain, L, noise_seed, *, kappa=20.0, eps=1.0, cutoff=1.0, v0=1.0, ang=0.0, T=0.01,
          Dr=None, locked=True, dt=1e-3, radius=1.0, skin=None, n_nearby=4, wca=None, springs=True, mdps=None):
    wca = _wca(radius, eps, cutoff) if wca is None else wca
    D = T / radius
    # the step limit that goes with lists of twice the interaction range checked every 40 steps
    mdps = 0.5 * max(2 * BOND, wca[3]) / 40 if mdps is None else mdps
    params = SystemParams(
        L=L, spring_params=np.array([100.0 if springs else 0.0, kappa if springs else 0.0, 0.0, 0.0,
                                     float(locked and springs), 0.1]),
        wca_params=wca, active_params=np.array([v0, 0.0, ang]), D=D,
        Dr=3 * D / (4 * radius * radius) if Dr is None else Dr, radius=radius, n_nearby=n_nearby,
        calc_springs=springs, calc_wca=True, self_propel=v0 != 0.0, dtmax=dt, max_dist_per_step=mdps,
        seed=noise_seed, skin=skin)
    n_chains = int(chain[-1]) + 1
    return SystemSpec(name, dim, pos, tan, chain, np.full(n_chains, BOND), params, dt, mdps)


def _sweep_points(n):
    """(n_chains, chain length, area fraction, chirality, bending) of the first n points of the sweep."""
    rng = np.random.default_rng(12345)
    nch = np.exp(rng.uniform(np.log(50), np.log(4000), size=256)).astype(int)
    clen = rng.integers(5, 41, size=256)
    phi, ang, kap = rng.uniform(0.1, 0.4, size=256), rng.uniform(-0.5, 0.5, size=256), rng.uniform(1, 50, size=256)
    return [(int(nch[i]), int(clen[i]), float(phi[i]), float(ang[i]), float(kap[i])) for i in range(n)]


def _side(n_chains, clen, phi):
    return math.sqrt(n_chains * (BOND * (clen - 1) + 1.0) / phi)


def _specs(case, seed):
    """The systems of a case: a list of SystemSpec, and the coupled groups and motors among them."""
    rng = np.random.default_rng([seed, 77])
    kind = case["kind"]
    groups, mots = [], []
    if kind in ("dropin", "analysis"):
        L = _side(case["n_chains"], case["clen"], case["phi"])
        pos, tan, chain, _, _ = _lay2d(rng, case["n_chains"], case["clen"], L)
        if kind == "analysis":
            a = np.repeat(rng.vonmises(0.3, 2.0, case["n_chains"]), case["clen"])
            tan = np.stack([np.cos(a), np.sin(a)], axis=1).astype(np.float32).astype(np.float64)
        return [_spec("box", 2, pos, tan, chain, L, seed)], groups, mots
    if kind in ("sweep", "srk4"):
        points = _sweep_points(case["n_systems"])
        if case.get("n_chains"):
            points = [(case["n_chains"], case["clen"], case["phi"], 0.0, 20.0)]
        out = []
        for i, (n, c, phi, ang, kap) in enumerate(points):
            L = _side(n, c, phi)
            pos, tan, chain, _, _ = _lay2d(rng, n, c, L)
            out.append(_spec("sweep%d" % i, 2, pos, tan, chain, L, 1000 * seed + i, ang=ang, kappa=kap))
        return out, groups, mots
    if kind == "lj2d":
        L = _side(case["n_chains"], case["clen"], case["phi"])
        pos, tan, chain, _, _ = _lay2d(rng, case["n_chains"], case["clen"], L, bundle=2)
        return [_spec("lj2d", 2, pos, tan, chain, L, seed, eps=0.5, cutoff=LJ_CUT, ang=0.2)], groups, mots
    if kind == "lj3d":
        L = case["side"]
        pos, tan, chain = _lay3d(rng, case["n_chains"], case["clen"], L)
        return [_spec("lj3d", 3, pos, tan, chain, L, seed, kappa=10.0, cutoff=LJ_CUT, T=0.05, Dr=0.1, locked=False,
                      dt=5e-4)], groups, mots
    out = []
    for i in range(case["n_boxes"]):
        motors = kind == "motors"
        n, L = (200, 60.0) if motors else (1000, 150.0)
        pos, tan, chain, free, extent = _lay2d(rng, n, 10, L)
        chains = _spec("box%d_chains" % i, 2, pos, tan, chain, L, 100000 * seed + 2 * i, v0=0.0 if motors else 1.0)
        cross = np.zeros((2, 2, 4))
        if motors:
            nm = int(round(L * L * 0.5))
            r_list = L / int(L / 2.0)  # one cell of the grid of twice the contact distance
            other = _spec("box%d_motors" % i, 2, rng.uniform(0, L, (nm, 2)), np.tile([1.0, 0.0], (nm, 1)),
                          np.arange(nm), L, 100000 * seed + 2 * i + 1, v0=0.0, T=0.1, Dr=0.0, springs=False,
                          wca=np.array([0.0, 0.0, 0.0, r_list]), n_nearby=0, mdps=chains.params.max_dist_per_step)
            cross[1, 0] = [0.0, 0.0, 0.0, r_list]
            mots.append((2 * i + 1, 2 * i, np.array([(BOND / 2) ** 2, 0.0, 1.0, 0.9, 0.2]), True))
        else:
            # five places a free slot, one contact distance apart
            spots = np.concatenate([np.mod(free + np.array([s, 0.0]), L) for s in np.arange(-2, 3) * 0.98])
            spots = spots[rng.permutation(len(spots))[:3000]] + rng.normal(0, 0.01, (3000, 2))
            a = rng.uniform(0, 2 * math.pi, 3000)
            t = np.stack([np.cos(a), np.sin(a)], axis=1).astype(np.float32).astype(np.float64)
            other = _spec("box%d_beads" % i, 2, np.mod(spots, L), t, np.arange(3000), L, 100000 * seed + 2 * i + 1,
                          v0=0.0, radius=0.7, springs=False, mdps=chains.params.max_dist_per_step)
            cross[0, 1] = cross[1, 0] = 0.5 * (chains.params.wca_params + other.params.wca_params)
        out += [chains, other]
        groups.append(([2 * i, 2 * i + 1], [False, False], cross))
    return out, groups, mots


# ---------------------------------------------------------------------------------------------
# programs
# ---------------------------------------------------------------------------------------------
def prepare(case, seed):
    specs, groups, mots = _specs(case, seed)
    kind = case["kind"]
    if kind == "dropin":
        s = specs[0]
        p = s.params
        config.dim, config.Lx, config.SRK_order = 2, p.L, 2
        config.n_steps_update_grid_list, config.max_dist_per_step, config.RK_cheat_factor = 40, s.relax_mdps, 1.0
        pop = SimpleNamespace(
            name="beads", fixed=False, total_pop=s.n, pos=s.pos, pos1=np.zeros_like(s.pos), tangent_list=s.tangent,
            forces=np.zeros_like(s.pos), chain_id=s.chain_id, rest_lengths=s.rest_lengths,
            longest_chain_length=case["clen"], rigid_rod_projection_factor=0.0, D=p.D, Dr=p.Dr, repel_d_max=p.radius,
            n_nearby_beads_dont_repel=p.n_nearby, b_init_growing=False, special_interactions={},
            self_interactions=lambda: [["springs", p.spring_params], ["WCA", p.wca_params],
                                       ["self-propulsion", p.active_params]])
        status = SimpleNamespace(dt=s.dt, dtmax=s.dt, dt_used=0.0, stepnum=0, t=0.0, next_output_step=0,
                                 next_save_time=0.0, update_grid_list_counter=0, max_forces_strength=0.0,
                                 b_calc_active_forces=True)
        sim = {"gpu_precision": case["precision"], "gpu_noise": "philox", "seed": seed, "save_state_every": -1.0}
        return SimpleNamespace(case=case, pop=pop, status=status, sim=sim, L=p.L, mdps=s.relax_mdps)
    order = 4 if kind == "srk4" else 2
    # lists deep enough for a dense bundle (attracting chains condense further while they run) and for
    # a motor's candidate beads
    depth = {"lj2d": 96, "lj3d": 768, "motors": 96}.get(kind)
    batch = Batch(specs, precision=case["precision"], list_depth=depth, srk_order=order,
                  pair_mode=case.get("pair_mode", 0))
    for g in groups:
        batch.couple(*g)
    for m in mots:
        batch.set_motors(*m)
    return SimpleNamespace(case=case, batch=batch, motors=bool(mots))


def run(state):
    case = state.case
    if case["kind"] == "dropin":
        config.Lx, config.max_dist_per_step = state.L, state.mdps
        state.status.next_output_step = state.status.stepnum + case["steps"]
        updates.SRK2_force_calc([state.pop], state.status, state.sim)
        p = state.pop
        return {"pos": p.pos, "pos1": p.pos1, "tangent": p.tangent_list, "forces": p.forces, "t": state.status.t}
    b = state.batch
    if case["kind"] == "analysis":
        eng, slot = b.engine, b.states[0].slot
        com, phi = observables.chain_frames(eng, slot)
        out = {"order": observables.order_parameters(eng, slot), "com": com, "phi": phi}
        for kind in ("g_of_r", "Cvv", "Cnn"):
            out[kind] = observables.pair_correlation(eng, slot, kind, case["binsize"])
        return out
    b.begin(case["steps"], series_every=case.get("series", 0))
    b.run(case["steps"])
    out = {k: b.big[k] for k in ("pos", "pos1", "tangent", "forces")}
    if case.get("series"):
        out["series"] = b.series_buf
    if case["kind"] == "srk4":
        out["forces_aux"] = b.big["forces_aux"]
    if state.motors:
        out["where_active"] = torch.cat([b.engine.where_active(st.slot) for st in b.states])
    return out


def work(case):
    """Bytes and operations of a pass.  A step of the whole path reads and writes 7 d position components and
    3 d force components a bead and 16 bytes of list; a state that fits the 126 MB cache need only come in and
    go out once a pass.  Operations: the two (four) force evaluations with their listed pairs, and the noise."""
    kind = case["kind"]
    F = 8 if case["precision"] == "fp64" else 4
    if kind == "analysis":
        n, c = case["n_chains"] * case["clen"], case["n_chains"]
        return {"bytes": n * (16 + 2 * F) + c * 32, "flops": 3 * 30.0 * c * (c - 1) / 2 + 40.0 * n}
    d = 3 if kind == "lj3d" else 2
    if kind in ("sweep", "srk4"):
        pts = _sweep_points(case["n_systems"])
        n = case["n_chains"] * case["clen"] if case.get("n_chains") else sum(a * b for a, b, *_ in pts)
    elif kind in ("pops", "motors"):
        n = case["n_boxes"] * (13000 if kind == "pops" else 3800)
    else:
        n = case["n_chains"] * case["clen"]
    pairs = {"lj2d": 13.0, "lj3d": 20.0, "motors": 3.0}.get(kind, 1.5)
    evals = 4 if kind == "srk4" else 2
    state = n * (2 * 8 * d + 2 * F * d + 4)
    step = n * (7 * d * 8 + 3 * d * F + 16) * (evals // 2)
    once = 2 * state
    return {"bytes": float(once if state <= 64e6 else case["steps"] * step),
            "flops": float(case["steps"]) * n * (evals * (60.0 + 25.0 * pairs) + 100.0)}


# ---------------------------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------------------------
M32 = 0xFFFFFFFF


def _philox(c0, c1, c2, c3, k0, k1):
    """Philox4x32-10 on int64 tensors holding 32-bit words."""
    for _ in range(10):
        p0, p1 = c0 * 0xD2511F53, c2 * 0xCD9E8D57
        c0, c1, c2, c3 = ((p1 >> 32) & M32) ^ c1 ^ k0, p1 & M32, ((p0 >> 32) & M32) ^ c3 ^ k1, p0 & M32
        k0, k1 = (k0 + 0x9E3779B9) & M32, (k1 + 0xBB67AE85) & M32
    return c0, c1, c2, c3


def _uniforms(words):
    m = (1 << 53) - 1
    a = ((words[0] << 21) ^ (words[1] >> 11)) & m
    b = ((words[2] << 21) ^ (words[3] >> 11)) & m
    return a, b


def _normals(idx, seed, step, stream, d):
    out = []
    for s in range(d - 1):
        o = torch.zeros_like(idx)
        a, b = _uniforms(_philox(idx, o + (step & M32), o + (step >> 32), o + (stream + s), seed & M32, seed >> 32))
        r = torch.sqrt(-2.0 * torch.log((a.double() + 1.0) * 2.0 ** -53))
        w = 2.0 * math.pi * b.double() * 2.0 ** -53
        out += [r * torch.cos(w), r * torch.sin(w)]
    return torch.stack(out[:d], dim=1)


class _Exact:
    """All systems of a case as one set of beads in separate boxes, stepped with torch operations in float64."""

    def __init__(self, specs, groups, mots, steps):
        self.dev = dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        self.d = specs[0].dim
        t = lambda a, ty=torch.float64: torch.as_tensor(np.ascontiguousarray(a), dtype=ty, device=dev)  # noqa: E731
        n = [s.n for s in specs]
        per = lambda f: t(np.repeat([float(f(s)) for s in specs], n))  # noqa: E731
        box = list(range(len(specs)))
        for members, _, _ in groups:
            for m in members:
                box[m] = members[0]
        box = list(np.unique(box, return_inverse=True)[1])
        self.nbox = max(box) + 1
        self.box = t(np.repeat(box, n), torch.int64)
        self.sys = t(np.repeat(np.arange(len(specs)), n), torch.int64)
        self.local = t(np.concatenate([np.arange(k) for k in n]), torch.int64)
        self.seed = t(np.repeat([s.params.seed for s in specs], n), torch.int64)
        off = np.cumsum([0] + [len(s.rest_lengths) for s in specs])
        self.chain = t(np.concatenate([s.chain_id + o for s, o in zip(specs, off)]), torch.int64)
        self.pos = t(np.concatenate([s.pos for s in specs]))
        self.pos1 = self.pos.clone()
        self.tan = t(np.concatenate([s.tangent for s in specs]))
        self.L = per(lambda s: s.params.L)[:, None]
        self.k, self.kappa = per(lambda s: s.params.spring_params[0]), per(lambda s: s.params.spring_params[1])
        self.locked = per(lambda s: s.params.spring_params[4]) > 0
        self.v0 = per(lambda s: s.params.active_params[0])[:, None]
        ang = per(lambda s: s.params.active_params[2])
        self.cs, self.sn = torch.cos(ang), torch.sin(ang)
        self.D, self.Dr, self.rad = (per(lambda s: s.params.D)[:, None], per(lambda s: s.params.Dr)[:, None],
                                     per(lambda s: s.params.radius)[:, None])
        self.nearby = per(lambda s: s.params.n_nearby)
        first = [box.index(b) for b in range(self.nbox)]
        self.dtmax = t([specs[i].params.dtmax for i in first])
        self.mdps = t([specs[i].params.max_dist_per_step for i in first])
        self.dt = self.dtmax.clone()
        self.elapsed = torch.zeros_like(self.dt)
        # pair parameters by (system, system): its own, and the coupled ones
        S = len(specs)
        self.other = np.arange(S)
        cross = np.zeros((S, 4))
        for (a, b), _, w in groups:
            self.other[a], self.other[b] = b, a
            cross[a], cross[b] = w[0, 1], w[1, 0]
        self.own_w, self.cross_w = t(np.stack([s.params.wca_params for s in specs])), t(cross)
        self.motor = np.zeros(S, dtype=bool)
        self.pushed = np.zeros(S)
        for m, c, prm, _ in mots:
            self.motor[m] = True
            self.pushed[c] = prm[2]
            self.mprm = prm
        self.has_motors = bool(mots)
        self.bmotor = t(self.motor, torch.bool)[self.sys]
        self.act = torch.full_like(self.local, -1)
        same = torch.zeros(len(self.pos) + 1, dtype=torch.bool, device=dev)
        same[1:-1] = (self.chain[1:] == self.chain[:-1]) & (self.k[1:] > 0)
        self.prev, self.next = same[:-1], same[1:]  # a bond to the bead before / after
        self.step0 = torch.tensor([s.params.step for s in specs])[0].item()
        reach = float(max(self.mdps)) * 2.2 * steps + 0.3
        self._pairs(specs, box, reach)

    def _pairs(self, specs, box, reach):
        rc = max(float(s.params.wca_params[3]) for s in specs) + reach
        nc, first, total = np.zeros(self.nbox, dtype=np.int64), np.zeros(self.nbox, dtype=np.int64), 0
        for s, b in zip(specs, box):
            nc[b] = max(3, int(s.params.L / rc))
        for b in range(self.nbox):
            first[b] = total
            total += nc[b] ** self.d
        t = lambda a: torch.as_tensor(a, device=self.dev)  # noqa: E731
        ncb, fb = t(nc)[self.box], t(first)[self.box]
        ci = torch.minimum((self.pos / self.L * ncb[:, None]).long(), ncb[:, None] - 1)

        def cell(c):
            out = torch.zeros_like(ncb)
            for i in reversed(range(self.d)):
                out = out * ncb + torch.remainder(c[:, i], ncb)
            return out + fb

        order = torch.argsort(cell(ci), stable=True)
        count = torch.bincount(cell(ci), minlength=total)
        start = torch.cumsum(count, 0) - count
        I, J = [], []
        for off in np.ndindex(*([3] * self.d)):
            q = cell(ci + torch.tensor(off, device=self.dev) - 1)
            for lo in range(0, len(q), 400000):
                m = count[q[lo:lo + 400000]]
                i = torch.repeat_interleave(torch.arange(lo, lo + len(m), device=self.dev), m)
                at = torch.arange(len(i), device=self.dev) - torch.repeat_interleave(torch.cumsum(m, 0) - m, m)
                j = order[start[q[i]] + at]
                ok = (((self.chain[i] != self.chain[j]) | ((i - j).abs().double() > self.nearby[i])) & (i != j))
                ok &= (self._sep(self.pos, i, j) ** 2).sum(1) <= rc * rc
                I.append(i[ok])
                J.append(j[ok])
        i, j = torch.cat(I), torch.cat(J)
        if self.has_motors:
            mot = self.bmotor[i] & ~self.bmotor[j]
            key = torch.argsort(i[mot] * len(self.pos) + j[mot])
            self.mi, self.mj = i[mot][key], j[mot][key]
            keep = ~self.bmotor[i] & ~self.bmotor[j]
            i, j = i[keep], j[keep]
        w = torch.where((self.sys[i] == self.sys[j])[:, None], self.own_w[self.sys[i]], self.cross_w[self.sys[i]])
        self.pi, self.pj, self.pw = i, j, w

    def _sep(self, X, i, j):
        s = X[j] - X[i]
        return s - self.L[i] * torch.round(s / self.L[i])

    def _motors(self, X, stage, step):
        """The motors' decisions at a stage: each goes through its candidates in ascending id."""
        if stage == 0:
            self.act[self.bmotor] = -1
        r_list = self.own_w[self.sys[self.mi], 3]
        ds = (self._sep(X, self.mi, self.mj) ** 2).sum(1)
        near = ds <= r_list * r_list
        mi, mj, ds = self.mi[near], self.mj[near], ds[near]
        count = torch.bincount(mi, minlength=len(X))
        rank = torch.arange(len(mi), device=self.dev) - (torch.cumsum(count, 0) - count)[mi]
        seed = self.seed[mi]
        a, b = _uniforms(_philox(self.local[mi], self.local[mj], torch.full_like(mi, step & M32),
                                 torch.full_like(mi, (step >> 32) & 0xFFFF | stage << 16),
                                 (seed & M32) ^ 0x6D6F746F, seed >> 32))
        uoff, uon = a.double() * 2.0 ** -53, b.double() * 2.0 ** -53
        delta, push = torch.zeros_like(self.act), torch.zeros_like(self.act)
        for r in range(int(rank.max()) + 1 if len(rank) else 0):
            s = rank == r
            m, j = mi[s], mj[s]
            on = self.act[m] >= 0
            off = on & (uoff[s] <= self.mprm[4])
            take = (~on | off) & (uon[s] < self.mprm[3]) & (ds[s] <= self.mprm[0])
            delta.index_add_(0, j, take.long() - off.long())
            push.index_add_(0, j, take.long())
            self.act[m] = torch.where(take, self.local[j], torch.where(off, torch.full_like(m, -1), self.act[m]))
        ch = ~self.bmotor
        self.act[ch] = (torch.full_like(self.act, -1) if stage == 0 else self.act)[ch] + delta[ch]
        return push.double()[:, None]

    def force(self, X, stage, step):
        push = self._motors(X, stage, step) if self.has_motors else None
        n = len(X)
        d = torch.zeros_like(X)
        d[:-1] = X[:-1] - X[1:]
        d = (d - self.L * torch.round(d / self.L)) * self.next[:, None]
        r = d.norm(dim=1)
        t = torch.where(self.next[:, None], d / torch.where(r > 0, r, 1.0)[:, None], 0.0)
        s = torch.where(self.next, self.k * (BOND / torch.where(r > 0, r, 1.0) - 1.0), 0.0)[:, None] * d
        back = lambda a: torch.cat([torch.zeros_like(a[:1]), a[:-1]])  # noqa: E731
        ahead = lambda a: torch.cat([a[1:], torch.zeros_like(a[:1])])  # noqa: E731
        inner = (self.prev & self.next)[:, None]
        tj = back(t)
        dv = tj - t
        omc = 0.5 * (dv * dv).sum(1, keepdim=True)  # 1 - cosine
        live = inner & (omc > 0) & (omc < 2)
        safe = torch.where(live, omc, 1.0)
        phi = 2.0 * torch.asin(torch.sqrt(0.5 * safe)) * self.kappa[:, None] / torch.sqrt(safe * (2.0 - safe))
        fw = torch.where(live, phi * (dv - omc * tj), 0.0)
        bw = torch.where(live, phi * (dv + omc * t), 0.0)
        F = s - back(s) + fw + bw - back(bw) - ahead(fw)
        one = torch.where(live, (t + tj) / torch.sqrt(2.0 * (2.0 - safe)), t)
        tg = torch.where(inner, one, torch.where(self.next[:, None], t, tj))
        lock = self.locked & (self.prev | self.next)
        self.tan = torch.where(lock[:, None], tg, self.tan)
        for lo in range(0, len(self.pi), 8_000_000):
            i, j, w = self.pi[lo:lo + 8_000_000], self.pj[lo:lo + 8_000_000], self.pw[lo:lo + 8_000_000]
            sep = self._sep(X, i, j)
            ds = (sep * sep).sum(1)
            on = (ds > 0) & (ds <= w[:, 3] ** 2)
            i, sep, ds, w = i[on], sep[on], ds[on], w[on]
            F.index_add_(0, i, sep * (ds ** -4 * (w[:, 0] - w[:, 1] * ds ** -3))[:, None])
        tan = self.tan
        if self.d == 2:
            tan = torch.stack([self.cs * tan[:, 0] - self.sn * tan[:, 1], self.sn * tan[:, 0] + self.cs * tan[:, 1]], 1)
        F = F + self.v0 * tan
        if push is not None:
            F = F + push * self.mprm[2] * self.tan
        return F

    def move(self, x0, F, xi, dt):
        b = dt[self.box][:, None]
        return torch.remainder(x0 + b / self.rad * F + torch.sqrt(2.0 * b.abs() * self.D) * xi, self.L)

    def _limit(self, G, pref):
        s = torch.sqrt(2.0 * self.D[:, 0]) + pref * G.norm(dim=1) / self.rad[:, 0]
        S = torch.zeros(self.nbox, dtype=torch.float64, device=self.dev)
        S.scatter_reduce_(0, self.box, s, "amax")
        return torch.minimum(self.dtmax, self.mdps / S)

    def step(self, step, order):
        xi = _normals(self.local, self.seed, step, 0, self.d)
        xi = torch.where(self.D > 0, xi, torch.zeros_like(xi))
        if order == 2:
            F = self.force(self.pos, 0, step)
            x1 = self.move(self.pos, F, xi, self.dt)
            if self.has_motors:
                x1 = torch.where((self.bmotor & (self.act >= 0))[:, None], self.pos1, x1)
            self.pos1 = x1
            F = F + self.force(self.pos1, 1, step)
            pref = 0.5
        else:
            F, x = 0.0, self.pos
            for k in range(4):
                self.faux = self.force(x, k, step)
                F = F + self.faux * (1 / 6, 1 / 3, 1 / 3, 1 / 6)[k]
                if k < 3:
                    # the noise term of a virtual update has the whole step's variance
                    b = self.dt[self.box][:, None]
                    x = torch.remainder(self.pos + b * (0.5, 0.5, 1.0)[k] / self.rad * self.faux +
                                        torch.sqrt(2.0 * b * self.D) * xi, self.L)
            self.pos1 = x
            pref = 1.0
        self.dt = dt = self._limit(F, pref)
        b = dt[self.box][:, None]
        new = torch.remainder(self.pos + b * pref / self.rad * F + torch.sqrt(2.0 * b * self.D) * xi, self.L)
        if self.has_motors:
            new = torch.where((self.bmotor & (self.act >= 0))[:, None], self.pos, new)
        self.pos = new
        self.elapsed = self.elapsed + dt
        turn = ((self.Dr[:, 0] > 0) & ~self.locked)[:, None]
        if bool(turn.any()):
            q = _normals(self.local, self.seed, step, 2, self.d)
            q = q - (q * self.tan).sum(1, keepdim=True) * self.tan
            v = self.tan + torch.sqrt(2.0 * b * self.Dr) * math.pi * q
            self.tan = torch.where(turn, v / v.norm(dim=1, keepdim=True), self.tan)
        self.forces = F

    def order(self):
        """P, S and the director angle of every system."""
        S = len(self.other)
        nch = int(self.chain[-1]) + 1
        s = torch.zeros(nch, 2, dtype=torch.float64, device=self.dev).index_add_(0, self.chain, self.tan[:, :2])
        a = torch.atan2(s[:, 1], s[:, 0])
        own = torch.zeros(nch, dtype=torch.int64, device=self.dev)
        own[self.chain] = self.sys
        v = torch.stack([torch.cos(a), torch.sin(a), torch.cos(2 * a), torch.sin(2 * a), torch.ones_like(a)], 1)
        m = torch.zeros(S, 5, dtype=torch.float64, device=self.dev).index_add_(0, own, v)
        q = torch.hypot(m[:, 2], m[:, 3])
        return torch.stack([torch.hypot(m[:, 0], m[:, 1]) / m[:, 4], q / m[:, 4],
                            torch.atan((q - m[:, 2]) / m[:, 3])], 1)


def _true_sep(a, b, L):
    return torch.remainder(b - a + 0.5 * L, L) - 0.5 * L


def _exact_analysis(case, e, spec):
    L, n, c = spec.params.L, spec.n, case["n_chains"]
    x, tan = e.pos.view(c, case["clen"], 2), e.tan.view(c, case["clen"], 2)
    head = x[:, :1]
    com = torch.remainder(head[:, 0] + _true_sep(x, head, L).sum(1), L)
    a = torch.atan2(tan[..., 1], tan[..., 0])
    phi = torch.stack([torch.atan2(tan[..., 1].sum(1), tan[..., 0].sum(1)),
                       torch.atan2(torch.sin(2 * a).sum(1), torch.cos(2 * a).sum(1)) / 2], 1)
    bins = math.ceil(int(L / 2) * math.sqrt(2) / case["binsize"])
    hist, cvv, cnn = (torch.zeros(bins, dtype=torch.float64, device=e.dev) for _ in range(3))
    for lo in range(0, c, 1000):
        i, j = torch.meshgrid(torch.arange(lo, min(c, lo + 1000), device=e.dev), torch.arange(c, device=e.dev),
                              indexing="ij")
        s = i > j
        i, j = i[s], j[s]
        sep = _true_sep(com[i], com[j], L)
        at = (torch.sqrt(sep[:, 0] * sep[:, 0] + sep[:, 1] * sep[:, 1]) / case["binsize"]).long()
        s = at < bins
        i, j, at = i[s], j[s], at[s]
        hist += 2.0 * torch.bincount(at, minlength=bins)
        cvv += 2.0 * torch.bincount(at, torch.cos(phi[i, 0] - phi[j, 0]), minlength=bins)
        cnn += 2.0 * torch.bincount(at, torch.cos(phi[i, 1] - phi[j, 1]).abs(), minlength=bins)
    r = torch.arange(bins, dtype=torch.float64, device=e.dev) * case["binsize"]
    keep = r < L / 2
    g = hist / (hist.sum() / (L * L) * 2.0 * math.pi * case["binsize"] * (r + case["binsize"] / 2))
    row = lambda v: torch.stack([r[keep], v[keep]], 1).cpu().numpy()  # noqa: E731
    one = hist.clamp(min=1.0)
    return {"order": e.order()[0].cpu().numpy(), "com": com.cpu().numpy(), "phi": phi.cpu().numpy(), "g_of_r": row(g),
            "Cvv": row(cvv / one), "Cnn": row(cnn / one)}


def exact(case, seed):
    specs, groups, mots = _specs(case, seed)
    kind = case["kind"]
    e = _Exact(specs, groups, mots, case.get("steps", 0))
    if kind == "analysis":
        return _exact_analysis(case, e, specs[0])
    every, rows = case.get("series", 0), []
    for k in range(case["steps"]):
        e.step(e.step0 + k, 4 if kind == "srk4" else 2)
        if every and (k + 1) % every == 0:
            o = e.order()
            rows.append(torch.cat([torch.full_like(o[:, :1], e.step0 + k + 1), e.elapsed[:, None], o], 1))
    out = {"pos": e.pos, "pos1": e.pos1, "tangent": e.tan, "forces": e.forces}
    if every:
        out["series"] = torch.stack(rows + [torch.zeros_like(rows[0])] * (case["steps"] // every + 1 - len(rows)), 1)
    if kind == "dropin":
        out = {k: v.cpu().numpy() for k, v in out.items()}
        out["t"] = float(e.elapsed[0])
    if kind == "srk4":
        out["forces_aux"] = e.faux
    if mots:
        out["where_active"] = None
    return out
