"""Workloads of the hot path, each through the entry points a program calls.

listed() names the cases, draw() gives more of the same ranges, prepare() makes
what a program holds before the call (inputs from the seed alone, engines and
output buffers), run() is one pass, work() the bytes and operations that pass
cannot do without, exact() the same outputs in 64-bit torch without the
library.  Sizes, densities and parameters are those of the benchmark, the tests
and the reference's scripts.
"""
import math
import os
import sys

import numpy as np
import torch
from torch.utils.checkpoint import checkpoint

_ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(_ROOT, "naivedynamics.jl_gb300"))

DEV = "cuda" if torch.cuda.is_available() else "cpu"
RHO = 0.83        # density of the Lennard-Jones boxes (4,096 atoms in a cube of side 17)
CUTOFF = 2.5
HALF_NEIGHBOURS = 0.5 * RHO * 4.0 / 3.0 * math.pi * CUTOFF ** 3  # pairs per atom in the bulk
PAIR_FLOPS = 40   # separation, r^2, 1/r^2, the Lennard-Jones term and the two force updates


def listed():
    return [
        # a script's pair list at the smallest size: launches and the round trip count
        {"name": "pairs_512", "kind": "pairs", "n": 512, "apl": 4, "order": 0, "box": "lj"},
        # gpubvh_neighborlist of the reference's position files: unit cube, r 0.1, the
        # list and the tree come back
        {"name": "neighborlist_20000", "kind": "neighborlist", "n": 20000, "apl": 4, "r": 0.1,
         "refresh": False},
        # device-resident list of a 262,144-atom box in the order of the traversal
        {"name": "pairs_dev_262144", "kind": "pairs_dev", "n": 262144, "apl": 4, "ordered": True,
         "box": "lj"},
        # the clustered stress set: unordered list into device memory
        {"name": "stress_4194304", "kind": "pairs_dev", "n": 4194304, "apl": 4, "ordered": False,
         "box": "clusters"},
        # a force evaluation of a reference-style step: pair list, both force calls, their sum
        {"name": "force_calls_4096", "kind": "force_calls", "n": 4096},
        # fused forces and energy of a configuration held on the host
        {"name": "forces_30004", "kind": "forces", "n": 30004, "coulomb": True},
        # plain Lennard-Jones steps of a small box
        {"name": "md_4096", "kind": "md", "n": 4096, "steps": 100, "coulomb": False,
         "mass": False, "skin": 0.3, "check": 1},
        # Lennard-Jones and Coulomb steps of the large box, with its tuned settings
        {"name": "md_coulomb_262144", "kind": "md", "n": 262144, "steps": 50, "coulomb": True,
         "mass": False, "skin": 0.4, "check": 3},
        # simulate! on host arrays, masses given
        {"name": "simulate_20004", "kind": "simulate", "n": 20004, "steps": 100, "coulomb": False,
         "log": 0, "damp": 0.0},
        # a batched ensemble of uneven systems
        {"name": "ensemble_64", "kind": "ensemble", "systems": 64, "nmin": 256, "nmax": 4096,
         "steps": 50},
        # one gradient of the histogram loss through 100 steps, by a program that takes many
        {"name": "adjoint_32768", "kind": "adjoint", "n": 32768, "steps": 100},
        # simulate! as the reference writes it, over the all-pairs list
        {"name": "compat_4096", "kind": "compat", "n": 4096, "steps": 20},
    ]


def _log_uniform(rng, lo, hi, multiple=1):
    n = math.exp(rng.uniform(math.log(lo), math.log(hi)))
    return max(int(lo), int(n)) // multiple * multiple


def draw(rng):
    kind = rng.choice(["pairs", "neighborlist", "pairs_dev", "stress", "force_calls", "forces",
                       "md", "md", "md", "simulate", "ensemble", "adjoint", "compat"])
    apl = rng.choice([2, 4, 4, 8])
    if kind == "pairs":
        return {"kind": kind, "n": _log_uniform(rng, 64, 30000, apl), "apl": apl,
                "order": rng.choice([0, 1]), "box": "lj"}
    if kind == "neighborlist":
        return {"kind": kind, "n": _log_uniform(rng, 100, 20000, apl), "apl": apl,
                "r": rng.choice([0.01, 0.03, 0.1]), "refresh": rng.choice([False, True])}
    if kind == "pairs_dev":
        return {"kind": kind, "n": _log_uniform(rng, 1000, 262144, apl), "apl": apl,
                "ordered": True, "box": "lj"}
    if kind == "stress":
        return {"kind": "pairs_dev", "n": _log_uniform(rng, 65536, 4194304, 4), "apl": 4,
                "ordered": False, "box": "clusters"}
    if kind == "force_calls":
        return {"kind": kind, "n": _log_uniform(rng, 256, 32768, 4)}
    if kind == "forces":
        return {"kind": kind, "n": _log_uniform(rng, 256, 131072, 4),
                "coulomb": rng.choice([False, True])}
    if kind == "md":
        return {"kind": kind, "n": _log_uniform(rng, 256, 262144, 4),
                "steps": rng.choice([10, 20, 35, 50]), "coulomb": rng.choice([False, True]),
                "mass": rng.choice([False, True]), "skin": rng.choice([0.3, 0.4]),
                "check": rng.choice([1, 3])}
    if kind == "simulate":
        log, damp = rng.choice([(0, 0.0), (0, 0.0), (10, 0.0), (20, 0.5)])
        return {"kind": kind, "n": _log_uniform(rng, 256, 65536, 4), "steps": rng.choice([40, 100]),
                "coulomb": rng.choice([False, True]), "log": log, "damp": damp}
    if kind == "ensemble":
        return {"kind": kind, "systems": rng.randint(8, 64), "nmin": 256,
                "nmax": rng.choice([1024, 4096]), "steps": rng.choice([20, 50])}
    if kind == "adjoint":
        return {"kind": kind, "n": _log_uniform(rng, 256, 32768, 4), "steps": rng.choice([50, 100])}
    return {"kind": kind, "n": _log_uniform(rng, 64, 4096), "steps": rng.choice([5, 10, 20])}


# ------------------------------------------------------------------ inputs


def _expand(start, count):
    """For each row k the integers start[k] .. start[k] + count[k] - 1: (rows, integers)."""
    rows = torch.repeat_interleave(torch.arange(len(count), device=count.device), count)
    first = torch.cumsum(count, 0) - count
    return rows, start[rows] + torch.arange(len(rows), device=count.device) - first[rows]


def _pairs_within(x, r):
    """Every pair (i, j) of rows of x (N x 3 FP64) closer than r, once: a cell list."""
    n = x.shape[0]
    cell = torch.floor((x - x.min(0).values) / r).long() + 1
    ny, nz = int(cell[:, 1].max()) + 2, int(cell[:, 2].max()) + 2
    key, perm = torch.sort((cell[:, 0] * ny + cell[:, 1]) * nz + cell[:, 2], stable=True)
    xs = x[perm]
    at = torch.arange(n, device=x.device)
    found = []
    for dx in (0, 1):
        for dy in (-1, 0, 1):
            if dx == 0 and dy < 0:
                continue
            # cells of increasing z are consecutive keys: one run of them at a time
            if dx == 0 and dy == 0:
                lo, hi = at + 1, torch.searchsorted(key, key + 1, right=True)
            else:
                t = key + dx * ny * nz + dy * nz
                lo = torch.searchsorted(key, t - 1)
                hi = torch.searchsorted(key, t + 1, right=True)
            i, j = _expand(lo, (hi - lo).clamp(min=0))
            d2 = ((xs[i] - xs[j]) ** 2).sum(1)
            keep = d2 < r * r
            found.append((i[keep], j[keep]))
    return perm[torch.cat([f[0] for f in found])], perm[torch.cat([f[1] for f in found])]


def _gen(seed, stream=0):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 64 + stream)
    return g


def _uniform(g, *shape):
    return torch.rand(*shape, generator=g, dtype=torch.float64, device=DEV)


def _fill_boxes(g, side, dmin, apart):
    """One position per row, uniform in its cube [0, side)^3; rows of the same cube (the
    same offset in `apart`) no closer than dmin: an atom closer than that to one already
    placed is drawn again."""
    n = len(side)
    x = _uniform(g, n, 3) * side[:, None]
    reach, span = float(dmin.max()), float((apart.max(0).values + side.max()).max())
    nc = int(span / reach) + 3
    open_ = torch.ones(n, dtype=torch.bool, device=DEV)
    for _ in range(2000):
        todo = open_.nonzero()[:, 0]
        if not len(todo):
            return x
        y = x + apart
        cell = torch.floor(y / reach).long() + 1
        key, perm = torch.sort((cell[:, 0] * nc + cell[:, 1]) * nc + cell[:, 2], stable=True)
        mine = (cell[todo, 0] * nc + cell[todo, 1]) * nc + cell[todo, 2]
        runs = torch.stack([mine + (dx * nc + dy) * nc for dx in (-1, 0, 1) for dy in (-1, 0, 1)])
        lo = torch.searchsorted(key, (runs - 1).view(-1))
        hi = torch.searchsorted(key, (runs + 1).view(-1), right=True)
        k, at = _expand(lo, hi - lo)
        i, j = todo[k % len(todo)], perm[at]
        close = ((y[i] - y[j]) ** 2).sum(1) < torch.maximum(dmin[i], dmin[j]) ** 2
        # a placed atom stays; of two new ones the first does
        close &= (i != j) & (~open_[j] | (j < i))
        bad = torch.zeros(n, dtype=torch.bool, device=DEV)
        bad[i[close]] = True
        open_ = bad
        again = bad.nonzero()[:, 0]
        x[again] = _uniform(g, len(again), 3) * side[again][:, None]
    raise RuntimeError("no configuration with that separation")


def _lj_box(case, seed):
    """x, v (N x 3), q, m (N or None) and the side of a box at density RHO, minimum
    separation 0.8, velocities N(0, 1)."""
    n = case["n"]
    side = (n / RHO) ** (1.0 / 3.0)
    g = _gen(seed)
    one = torch.ones(n, dtype=torch.float64, device=DEV)
    x = _fill_boxes(g, side * one, 0.8 * one, torch.zeros(n, 3, dtype=torch.float64, device=DEV))
    v = torch.randn(n, 3, generator=g, dtype=torch.float64, device=DEV)
    q = m = None
    if case.get("coulomb"):
        q = one.clone()
        q[torch.randperm(n, generator=g, device=DEV)[: n // 2]] = -1.0
    if case.get("mass"):
        m = 0.5 + 1.5 * _uniform(g, n)
    return x, v, q, m, side


def _points(case, seed):
    """Float32 points of a pair-list case (N x 3) and the radius."""
    n = case["n"]
    if case["box"] == "clusters":
        # 64 Gaussian clusters, centres uniform in a cube of side 400, widths U[2, 10]
        g = _gen(seed)
        centre, width = 400.0 * _uniform(g, 64, 3), 2.0 + 8.0 * _uniform(g, 64)
        k = torch.arange(n, device=DEV) % 64
        z = torch.randn(n, 3, generator=g, dtype=torch.float64, device=DEV)
        return (centre[k] + width[k][:, None] * z).float().contiguous(), CUTOFF
    # Float32 positions uniform in a cube at density RHO, as the search tests draw them
    return ((n / RHO) ** (1.0 / 3.0) * _uniform(_gen(seed), n, 3)).float().contiguous(), CUTOFF


def _systems(case, seed):
    """A batched ensemble: sizes evenly spread in their logarithm and shuffled, densities
    U[0.75, 0.9], sigma U[0.95, 1.05], epsilon U[0.8, 1.2] (fluids that stay as dense in
    a long run as they start); atoms concatenated."""
    rng = np.random.default_rng(int(seed))
    ns = case["systems"]
    size = np.exp(np.linspace(math.log(case["nmin"]), math.log(case["nmax"]), ns))
    size = rng.permutation((8 * np.round(size / 8)).astype(np.int64))
    side = (size / rng.uniform(0.75, 0.9, ns)) ** (1.0 / 3.0)
    sigma, eps = rng.uniform(0.95, 1.05, ns), rng.uniform(0.8, 1.2, ns)
    sid = torch.repeat_interleave(torch.arange(ns, device=DEV), torch.as_tensor(size, device=DEV))
    per = lambda a: torch.as_tensor(a, dtype=torch.float64, device=DEV)[sid]  # noqa: E731
    apart = torch.zeros(len(sid), 3, dtype=torch.float64, device=DEV)
    g = _gen(seed)
    pitch = float(side.max()) + 10.0
    for d, k in enumerate((sid % 8, sid // 8 % 8, sid // 64)):
        apart[:, d] = pitch * k
    x = _fill_boxes(g, per(side), 0.8 * per(sigma), apart)
    v = torch.randn(len(sid), 3, generator=g, dtype=torch.float64, device=DEV)
    return dict(size=size, side=side, sigma=sigma, eps=eps, x=x, v=v, apart=apart,
                atom_side=per(side), atom_sigma=per(sigma), atom_eps=per(eps))


def _collector(case, seed):
    """Inputs of simulate! as written, drawn like the reference's scripts: unit box,
    temperature 0.01, masses in [1, 5), charges within 1e-9 of zero."""
    n = case["n"]
    rng = np.random.default_rng(int(seed))
    m = rng.uniform(1.0, 5.0, n).astype(np.float32)
    q = rng.uniform(-1e-9, 1e-9, n).astype(np.float32)
    x = rng.uniform(0.0, 1.0, (n, 3)).astype(np.float32)
    v = np.repeat((np.float32(0.01) / np.float32(n) * np.float32(3 * n) / m)[:, None], 3, axis=1)
    return x, v, m, q


def _host(t):
    return None if t is None else t.cpu().numpy()


# --------------------------------------------------------------- one pass


def prepare(case, seed):
    import naivedynamics as nd

    s = dict(case, nd=nd)
    kind = case["kind"]
    if kind == "pairs":
        x, r = _points(case, seed)
        s.update(x=_host(x), spec=nd.SpheresBVHSpecs(r, case["n"], case["apl"]),
                 room=_room(case))
    elif kind == "neighborlist":
        x = _host(_uniform(_gen(seed), case["n"], 3).float())
        s.update(x=x, spec=nd.SpheresBVHSpecs(case["r"], case["n"], case["apl"]),
                 room=_room(case))
        if case["refresh"]:
            # the positions a short time later, searched through the kept tree
            step = 0.1 * case["r"] * np.random.default_rng(int(seed)).uniform(-1, 1, x.shape)
            s.update(moved=(x + step).astype(np.float32),
                     kept=nd.gpubvh_neighborlist(None, x, s["spec"]))
    elif kind == "pairs_dev":
        x, r = _points(case, seed)
        spec = nd.SpheresBVHSpecs(r, case["n"], case["apl"])
        mode = nd.ND_PAIRS_ORDERED if case["ordered"] else nd.ND_PAIRS_UNORDERED
        torch.cuda.synchronize()
        if case["ordered"]:
            cap = _room(case)
        else:  # clusters may overlap: the program asks for the count first
            _, count = nd.neighbor_pairs_dev(x, spec, None, None, None, 0, mode=mode)
            cap = count + count // 16 + 64
        s.update(x=x, spec=spec, mode=mode, cap=cap,
                 pi=torch.zeros(cap, dtype=torch.int32, device=DEV),
                 pj=torch.zeros(cap, dtype=torch.int32, device=DEV),
                 pd=torch.zeros(cap, dtype=torch.float32, device=DEV))
    elif kind == "force_calls":
        x, _, q, _, _ = _lj_box(dict(case, coulomb=True), seed)
        x = _host(x).astype(np.float32)  # the reference's Float32 positions
        s.update(x=x, q=_host(q), spec=nd.SpheresBVHSpecs(CUTOFF, case["n"], 4),
                 f=[np.zeros((case["n"], 3), np.float32) for _ in range(3)])
    elif kind == "forces":
        x, _, q, _, _ = _lj_box(case, seed)
        s.update(x=_host(x), q=_host(q), ff=nd.ForceField(1.0, 1.0, 1.0, CUTOFF))
    elif kind == "md":
        x, v, q, m, side = _lj_box(case, seed)
        torch.cuda.synchronize()
        s["engine"] = nd.MDEngine(_md_params(nd, case, side), x, v, q, m, device=True)
        _md_buffers(s, case["n"])
    elif kind == "simulate":
        x, v, q, m, side = _lj_box(dict(case, mass=True), seed)
        s.update(x=_host(x), v=_host(v), q=_host(q), m=_host(m),
                 spec=nd.SimSpec(duration=case["steps"], stepwidth=1e-3, vDamp=case["damp"]),
                 clct=nd.GenericRandomCollector(objectnumber=case["n"], minDim=(0.0,) * 3,
                                                maxDim=(side,) * 3, temperature=1.0))
    elif kind == "ensemble":
        e = _systems(case, seed)
        hi = np.repeat(e["side"][:, None], 3, axis=1)
        table = nd.systems_table(e["size"], e["sigma"], e["eps"], 0.0 * hi, hi)
        p = nd.md_params(cutoff=CUTOFF, skin=0.4, dt=1e-3, refit_check_every=3, atomsperleaf=8)
        torch.cuda.synchronize()
        s["engine"] = nd.Ensemble(p, table, e["x"], e["v"], device=True)
        _md_buffers(s, len(e["x"]))
    elif kind == "adjoint":
        x, v, _, _, side = _lj_box(case, seed)
        p = nd.md_params(cutoff=CUTOFF, skin=0.3, dt=1e-3, box_hi=(side,) * 3, resort_every=5)
        adj = nd.Adjoint(p, nd.adj_spec(case["steps"], checkpoint_every=50), _host(x), _host(v))
        adj.set_target(_adjoint_target())
        adj.forward()  # both passes are captured by their first call
        adj.backward()
        s["adjoint"] = adj
    elif kind == "compat":
        x, v, m, q = _collector(case, seed)
        s.update(x=x, v=v, m=m, q=q,
                 spec=nd.SimSpec(duration=case["steps"], stepwidth=1, vDamp=1.0),
                 clct=nd.GenericRandomCollector(objectnumber=case["n"], minDim=(0.0,) * 3,
                                                maxDim=(1.0,) * 3, temperature=0.01))
    else:
        raise ValueError(kind)
    return s


def _md_params(nd, case, side):
    return nd.md_params(coulomb_k=1.0 if case["coulomb"] else 0.0, cutoff=CUTOFF,
                        skin=case["skin"], dt=1e-3, box_hi=(side,) * 3,
                        refit_check_every=case["check"])


def _md_buffers(s, n):
    s.update(x=torch.empty(n, 3, dtype=torch.float64, device=DEV),
             v=torch.empty(n, 3, dtype=torch.float64, device=DEV),
             f=torch.empty(n, 3, dtype=torch.float32, device=DEV))


def _adjoint_target():
    """A pair-distance histogram of a fluid at this density: 64 bins on [0, 2.5]."""
    r = (np.arange(64) + 0.5) * CUTOFF / 64
    return RHO * 2.0 * math.pi * r ** 2 * (1.0 + 0.8 * np.exp(-((r - 1.1) / 0.15) ** 2)) \
        * (r > 0.85) * CUTOFF / 64 * math.sqrt(2.0 * math.pi)


def _tree_out(treedata):
    keys, pos, perm, _ = treedata
    return {"min": keys["min"], "max": keys["max"], "left": keys["left"], "skip": keys["skip"],
            "index": pos.index, "code": pos.morton_code, "position": pos.position, "perm": perm}


def _list_out(pairs, room):
    # the list keeps one length from step to step, as the reference's resized vector does:
    # zeros after the last pair
    count = len(pairs)
    pairs.resize(room, refcheck=False)
    return {"count": count, "i": pairs["i"], "j": pairs["j"], "d": pairs["d"]}


def _room(case):
    """Entries that hold the pair list of a case at any seed."""
    expect = case["n"] * _pairs_per_atom(case)
    return int(1.05 * expect + 12.0 * math.sqrt(expect)) + 64


def run(s):
    nd, kind = s["nd"], s["kind"]
    if kind == "pairs":
        return _list_out(nd.leafbuild_traverse_bvh(s["x"], s["spec"], order=s["order"]),
                         s["room"])
    if kind == "neighborlist":
        if s["refresh"]:
            pairs, tree = nd.gpubvh_neighborlist_(None, s["kept"].treedata, s["spec"], None,
                                                  position=s["moved"])
        else:
            pairs, tree = nd.gpubvh_neighborlist(None, s["x"], s["spec"])
        return {"pairs": _list_out(pairs, s["room"]), "tree": _tree_out(tree)}
    if kind == "pairs_dev":
        _, count = nd.neighbor_pairs_dev(s["x"], s["spec"], s["pi"], s["pj"], s["pd"], s["cap"],
                                         mode=s["mode"])
        if s["ordered"]:
            return {"count": count, "i": s["pi"], "j": s["pj"], "d": s["pd"]}
        # an unordered list has no order of its own, and one of this size is not copied or
        # sorted: a program that keeps or compares it takes its count and order-free hash
        h = nd.pair_hash_dev(s["pi"], s["pj"], s["pd"], count)
        return {"count": count, "hash": np.array(h, np.uint64).view(np.int32)}
    if kind == "force_calls":
        pairs = nd.leafbuild_traverse_bvh(s["x"], s["spec"])
        f, lj, coul = s["f"]
        e_lj = nd.force_lennardjones_(lj, pairs, s["x"], cutoff=CUTOFF)
        e_coul = nd.force_coulomb_(coul, pairs, s["q"], s["x"], cutoff=CUTOFF)
        return {"lj": lj, "coulomb": coul, "sum": nd.sum_forces_(f, lj, coul), "e_lj": e_lj,
                "e_coulomb": e_coul}
    if kind == "forces":
        f, e = nd.forces(s["x"], s["q"], s["ff"])
        return {"f": f, "energy": e}
    if kind in ("md", "ensemble"):
        s["engine"].run(s["steps"])
        s["engine"].get_dev(s["x"], s["v"], s["f"])
        return {"x": s["x"], "v": s["v"], "f": s["f"]}
    if kind == "simulate":
        sys_ = nd.GenericObjectCollection(s["x"], s["v"], mass=s["m"], charge=s["q"])
        out = nd.simulate_(sys_, s["spec"], s["clct"], log_every=s["log"] or None)
        res = {"x": sys_.position, "v": sys_.velocity, "f": sys_.force}
        if s["log"]:
            res["log"] = out
        return res
    if kind == "adjoint":
        loss, hist = s["adjoint"].forward()
        g = s["adjoint"].backward()
        return {"loss": loss, "hist": hist, **g}
    if kind == "compat":
        sys_ = nd.GenericObjectCollection(s["x"], s["v"], mass=s["m"], charge=s["q"])
        log = nd.simulate_compat_(sys_, s["spec"], s["clct"])
        return {"x": sys_.position, "v": sys_.velocity, "f": sys_.force, "log": log}
    raise ValueError(kind)


# ------------------------------------------------------- least work of a pass


def _pairs_per_atom(case):
    if case["kind"] == "neighborlist":
        return 0.5 * case["n"] * 4.0 / 3.0 * math.pi * case["r"] ** 3
    if case.get("box") == "clusters":
        # mean density seen by a point of a Gaussian cluster of width w: N_c / (2 sqrt(pi) w)^3
        w = np.linspace(2.0, 10.0, 64)
        rho = (case["n"] / 64) / (2.0 * math.sqrt(math.pi) * w) ** 3
        return float(np.mean(0.5 * rho * 4.0 / 3.0 * math.pi * CUTOFF ** 3))
    return HALF_NEIGHBOURS


def work(case):
    kind = case["kind"]
    if kind == "ensemble":
        n = case["systems"] * (case["nmax"] - case["nmin"]) / math.log(case["nmax"] / case["nmin"])
    else:
        n = case["n"]
    pairs = n * _pairs_per_atom(case)
    if kind in ("pairs", "pairs_dev"):
        return {"bytes": 12 * n + 12 * pairs, "flops": 9 * pairs}
    if kind == "neighborlist":
        return {"bytes": 12 * n + 12 * pairs + 32 * n + 24 * n, "flops": 9 * pairs}
    if kind == "force_calls":
        return {"bytes": (12 + 8 + 36) * n, "flops": (9 + PAIR_FLOPS + 20) * pairs}
    if kind == "forces":
        return {"bytes": (24 + 8 + 12) * n, "flops": (9 + PAIR_FLOPS) * pairs}
    if kind in ("md", "ensemble", "simulate"):
        logged = 24 * (case["steps"] // case["log"]) if case.get("log") else 0
        return {"bytes": (48 + 16 + 60 + logged) * n, "flops": case["steps"] * PAIR_FLOPS * pairs}
    if kind == "adjoint":
        # the steps, their recomputation and the Hessian-vector product of each
        return {"bytes": (48 + 48) * n, "flops": case["steps"] * (2 * PAIR_FLOPS + 60) * pairs}
    return {"bytes": (24 + 8 + 36 + 12 * case["steps"]) * n,
            "flops": case["steps"] * 40 * 0.5 * n * (n - 1)}


# ------------------------------------------------------- the same in 64 bits


def _pair_forces64(x, i, j, n, sigma, eps, q, kc, rc):
    """Forces (N x 3) and energy of the listed pairs within rc; sigma and eps per pair or
    numbers."""
    d = x[i] - x[j]
    r2 = (d * d).sum(1)
    inside = r2 < rc * rc
    ir2 = 1.0 / r2
    s6 = (sigma * sigma * ir2) ** 3
    mag = 24.0 * eps * ir2 * s6 * (2.0 * s6 - 1.0)
    u = 4.0 * eps * s6 * (s6 - 1.0)
    if q is not None and kc:
        c = kc * q[i] * q[j] * torch.sqrt(ir2)
        mag, u = mag + c * ir2, u + c
    t = torch.where(inside, mag, torch.zeros_like(mag))[:, None] * d
    f = torch.zeros(n, 3, dtype=torch.float64, device=x.device)
    f = f.index_add(0, i, t).index_add(0, j, -t)
    return f, torch.where(inside, u, torch.zeros_like(u)).sum()


class _Near:
    """Pairs within reach of rc while no atom moves more than half the margin."""

    def __init__(self, rc, apart=None, margin=0.6):
        self.rc, self.apart, self.margin, self.at = rc, apart, margin, None

    def __call__(self, x):
        x, far = x.detach(), (0.49 * self.margin) ** 2
        if self.at is None or float(((x - self.at) ** 2).sum(1).max()) > far:
            self.at = x.clone()
            y = self.at if self.apart is None else self.at + self.apart
            self.pairs = _pairs_within(y, self.rc + self.margin)
        return self.pairs


def _walls(x, u, hi):
    lo = torch.zeros_like(x)
    out = (x < lo) | (x > hi)
    return torch.where(x < lo, lo, torch.where(x > hi, hi, x)), torch.where(out, -u, u)


def _trajectory64(x, v, steps, force, hi, m=None, dt=1e-3, after=None):
    """Kick-drift-kick velocity Verlet with reflecting walls; after(k, x, v) may replace v."""
    im = 1.0 if m is None else (1.0 / m)[:, None]
    f = force(x)
    for k in range(1, steps + 1):
        u = v + 0.5 * dt * f * im
        x, u = _walls(x + dt * u, u, hi)
        f = force(x)
        v = u + 0.5 * dt * f * im
        if after is not None:
            v = after(k, x, v)
    return x, v, f


def exact(case, seed):
    kind = case["kind"]
    if kind == "force_calls":
        x, _, q, _, _ = _lj_box(dict(case, coulomb=True), seed)
        x = x.float()
        i, j = _pairs_within(x.double(), CUTOFF * 1.001)
        d = x[i] - x[j]  # the list's Float32 criterion
        keep = (d[:, 0] * d[:, 0] + d[:, 1] * d[:, 1]) + d[:, 2] * d[:, 2] < CUTOFF * CUTOFF
        i, j, x, n = i[keep], j[keep], x.double(), case["n"]
        lj, e_lj = _pair_forces64(x, i, j, n, 1.0, 1.0, None, 0.0, CUTOFF)
        co, e_co = _pair_forces64(x, i, j, n, 1.0, 0.0, q, 1.0, CUTOFF)
        return {"lj": lj, "coulomb": co, "sum": lj + co, "e_lj": float(e_lj),
                "e_coulomb": float(e_co)}
    if kind == "forces":
        x, _, q, _, _ = _lj_box(case, seed)
        f, e = _pair_forces64(x, *_pairs_within(x, CUTOFF), case["n"], 1.0, 1.0, q, 1.0, CUTOFF)
        return {"f": f, "energy": float(e)}
    if kind in ("md", "simulate"):
        x, v, q, m, side = _lj_box(dict(case, mass=case.get("mass", True)), seed)
        near = _Near(CUTOFF)
        force = lambda y: _pair_forces64(y, *near(y), len(y), 1.0, 1.0, q, 1.0, CUTOFF)[0]  # noqa: E731
        log, damp = case.get("log", 0), case.get("damp", 0.0)
        frames = [x]

        def after(k, y, w):
            if damp and k % 10 == 0:  # rescale_velocity! towards temperature 1
                ti = 2.0 / (3.0 * len(w)) * float((w.norm(dim=1) * m / 2.0).sum())
                w = w * math.sqrt(1.0 + damp * (1.0 / ti - 1.0))
            if log and k % log == 0:
                frames.append(y)
            return w

        hi = torch.full_like(x, side)
        x, v, f = _trajectory64(x, v, case["steps"], force, hi, m, after=after)
        out = {"x": x, "v": v, "f": f}
        if log:
            out["log"] = torch.stack(frames)
        return out
    if kind == "ensemble":
        e = _systems(case, seed)
        near, sg, ep = _Near(CUTOFF, e["apart"]), e["atom_sigma"], e["atom_eps"]

        def force(y):
            i, j = near(y)
            return _pair_forces64(y, i, j, len(y), sg[i], ep[i], None, 0.0, CUTOFF)[0]

        hi = e["atom_side"][:, None].expand(-1, 3)
        x, v, f = _trajectory64(e["x"], e["v"], case["steps"], force, hi)
        return {"x": x, "v": v, "f": f}
    if kind == "adjoint":
        return _adjoint64(case, seed)
    return None  # lists and trees are whole numbers; simulate! as written is rounded step by step


def _adjoint64(case, seed):
    x0, v0, _, _, side = _lj_box(case, seed)
    n, near = case["n"], _Near(CUTOFF)
    sigma = torch.ones((), dtype=torch.float64, device=DEV, requires_grad=True)
    eps = torch.ones((), dtype=torch.float64, device=DEV, requires_grad=True)
    x0.requires_grad_()
    v0.requires_grad_()
    hi = torch.full_like(x0, side).detach()

    def step(x, u, i, j, dt):
        u = u + dt * _pair_forces64(x, i, j, n, sigma, eps, None, 0.0, CUTOFF)[0]
        return _walls(x + 1e-3 * u, u, hi)

    x, u = x0, v0
    for k in range(case["steps"]):
        x, u = checkpoint(step, x, u, *near(x), 0.5e-3 if k == 0 else 1e-3, use_reentrant=False)
    i, j = near(x)
    r = ((x[i] - x[j]) ** 2).sum(1)
    r = torch.sqrt(r[r < CUTOFF * CUTOFF])
    t = ((r - (CUTOFF - 0.25)) / 0.25).clamp(min=0.0)
    weight = 1.0 - t ** 3 * (10.0 - 15.0 * t + 6.0 * t ** 2)
    width = CUTOFF / 64
    bins = [(weight * torch.exp(-((r - (b + 0.5) * width) ** 2) / (2.0 * width ** 2))).sum() / n
            for b in range(64)]
    hist = torch.stack(bins)
    target = torch.as_tensor(_adjoint_target(), dtype=torch.float64, device=DEV)
    loss = ((hist - target) ** 2).sum()
    gx, gv, gs, ge = torch.autograd.grad(loss, (x0, v0, sigma, eps))
    return {"loss": float(loss), "hist": hist.detach(), "x0": gx, "v0": gv, "sigma": float(gs),
            "epsilon": float(ge)}
