"""The framework's work, as cases that can be timed: what its users call, over the range they call it in.

Three kinds of work:

* ``impact``: one giant impact advanced on the device (main.cpp:92-173).  ``io`` "resident": the state goes
  up once, the prologue and ``steps`` steps run, the whole state comes back (a run between two snapshots).
  ``io`` "host": a host that keeps its particles sends a step's inputs and reads its outputs every step.
* ``sweep``: ``runs`` impacts of uneven size in one context, advanced together.
* ``walks``: a host that keeps FDPS hands the interaction functors over: every i-group of a state with its
  j-list through the MultiWalk callbacks (density, derivative, hydro, gravity), payload or index form.
* ``order``: the allocation-free Morton ordering of device arrays.

``exact`` restates the physics in plain 64-bit torch: all pairs instead of neighbour lists, cell sums over
particles instead of a bottom-up pass, the octree's opening rule applied level by level.
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from fdps_sph_gb300 import eos, ic, layouts, lib

FIELDS = lib.FIELDS
FIELD = lib.FIELD
THETA = 0.5
KINDS = ("dens", "drvt", "hydro", "grav")
MAX_EXACT = 60_000     # particles up to which the 64-bit restatement is quick


def listed():
    return [
        # one plain functor call per kind: a single i-group, where a call's latency is all there is
        {"name": "walks_one_group", "kind": "walks", "n": 180, "precision": "fp64", "form": "payload"},
        # an FDPS host with the default (reference) arithmetic
        {"name": "walks_30k_fp64", "kind": "walks", "n": 30_011, "precision": "fp64", "form": "payload"},
        # the same boundary in mixed precision, the pass's particles sent once
        {"name": "walks_100k_mixed", "kind": "walks", "n": 100_003, "precision": "mixed", "form": "index"},
        # a host under a fixed device-memory budget orders its particles
        {"name": "order_100k", "kind": "order", "n": 100_003},
        # the smallest impact people run (the reference's CPU size): analytic Tillotson, plain FP64
        {"name": "impact_10k_fp64", "kind": "impact", "n": 10_000, "precision": "fp64", "eos": "tillotson",
         "theta": 0.5, "contact": False, "io": "resident", "steps": 4},
        # the smallest run of a sweep, alone, with the bodies in contact (artificial viscosity active)
        {"name": "impact_5k_mixed", "kind": "impact", "n": 5_003, "precision": "mixed", "eos": "table2",
         "theta": 0.5, "contact": True, "io": "resident", "steps": 8},
        # plain FP64 at a production size with table EoS
        {"name": "impact_200k_fp64", "kind": "impact", "n": 200_003, "precision": "fp64", "eos": "table2",
         "theta": 0.5, "contact": True, "io": "resident", "steps": 2},
        # mode 2: entropies kept constant, energies looked up every step
        {"name": "impact_100k_mode2", "kind": "impact", "n": 100_000, "precision": "mixed", "eos": "mode2",
         "theta": 0.5, "contact": True, "io": "resident", "steps": 8},
        # the headline: 1M particles between two snapshots
        {"name": "impact_1m", "kind": "impact", "n": 1_000_000, "precision": "mixed", "eos": "table2",
         "theta": 0.5, "contact": False, "io": "resident", "steps": 8},
        # the same size driven step by step by a host that keeps its particles
        {"name": "impact_1m_host", "kind": "impact", "n": 1_000_000, "precision": "mixed", "eos": "table2",
         "theta": 0.5, "contact": False, "io": "host", "steps": 1},
        # the largest impact: three layers, the wider opening angle
        {"name": "impact_4m", "kind": "impact", "n": 4_000_000, "precision": "mixed", "eos": "table3",
         "theta": 0.7, "contact": True, "io": "resident", "steps": 4},
        # many impacts of 5k-200k particles advanced together
        {"name": "sweep_24", "kind": "sweep", "runs": 24, "n_lo": 5_000, "n_hi": 200_000, "steps": 16},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["impact"] * 5 + ["walks"] * 3 + ["sweep", "order"])
    if kind == "order":
        return {"kind": kind, "n": _log_int(rng, 1_000, lib.NOALLOC_MAX_N)}
    if kind == "walks":
        return {"kind": kind, "n": _log_int(rng, 150, 60_000), "precision": rng.choice(["fp64", "mixed"]),
                "form": rng.choice(["payload", "index"])}
    if kind == "sweep":
        return {"kind": kind, "runs": rng.randint(2, 24), "n_lo": 5_000, "n_hi": _log_int(rng, 20_000, 200_000),
                "steps": rng.choice([4, 8, 16])}
    precision = rng.choice(["mixed", "mixed", "fp64"])
    io = rng.choice(["resident", "resident", "host"])
    return {"kind": kind, "n": _log_int(rng, 2_000, 150_000 if precision == "fp64" else 1_500_000),
            "precision": precision, "eos": rng.choice(["tillotson", "table2", "table3"]),
            "theta": rng.choice([0.5, 0.5, 0.7]), "contact": rng.random() < 0.5, "io": io,
            "steps": 1 if io == "host" else rng.choice([1, 2, 4])}


# ---------------------------------------------------------------------------
# what a program has in hand

def _materials(kind):
    if kind == "tillotson":
        return [eos.Tillotson("iron", eos.TILLOTSON["iron"]), eos.Tillotson("granite", eos.TILLOTSON["granite"])]
    if kind == "mode2":   # tables down to 1e-3 kg/m^3, so that every density has a defined entropy lookup
        return [eos.synthetic_table(m, 120, 120, rho_range=(1e-3, 3e4)) for m in ("iron", "dunite")]
    names = ("iron", "dunite") if kind == "table2" else ("iron", "dunite", "granite")
    return [eos.synthetic_table(m, 200, 200) for m in names]


def _layers(kind):
    if kind == "tillotson":
        return [ic.Layer(0, 0.3, 7800.0), ic.Layer(1, 0.7, 2700.0)]
    if kind == "table3":
        return [ic.Layer(0, 0.3, 7800.0), ic.Layer(1, 0.65, 3320.0), ic.Layer(2, 0.05, 2700.0)]
    return [ic.Layer(0, 0.3, 7800.0), ic.Layer(1, 0.7, 3320.0)]


def _bodies(n, eos_kind, contact, seed):
    """0.89 and 0.11 Earth masses, spinning and stirred, 4 target radii apart or just in contact."""
    layers = _layers(eos_kind)
    mt, mi = 0.89 * ic.M_EARTH, 0.11 * ic.M_EARTH
    sep = ic.contact_separation(mt, mi, layers, 0.02) if contact else 4.0
    n_i = max(32, n // 10)
    F, ids, mats, _ = ic.make_impact(n - n_i, n_i, mt, mi, layers, layers, 30.0, 1.2, seed, sep_over_rt=sep)
    rng = np.random.default_rng(seed + 1)
    sx, sy, sz = 3.0e-5, -2.0e-5, 1.0e-4
    x, y, z = F[FIELD["x"]], F[FIELD["y"]], F[FIELD["z"]]
    F[FIELD["vx"]] += sy * z - sz * y + 30.0 * rng.standard_normal(n)
    F[FIELD["vy"]] += sz * x - sx * z + 30.0 * rng.standard_normal(n)
    F[FIELD["vz"]] += sx * y - sy * x + 30.0 * rng.standard_normal(n)
    return F, ids, mats


def _pinned(shape, dtype=torch.float64):
    return torch.empty(shape, dtype=dtype, pin_memory=True).numpy()


def _pinned_copy(a):
    out = _pinned(a.shape, {np.dtype("f8"): torch.float64, np.dtype("i8"): torch.int64,
                            np.dtype("i4"): torch.int32}[a.dtype])
    out[...] = a
    return out


def _context(materials, **kw):
    ctx = lib.Context(**kw)
    for k, m in enumerate(materials):
        ctx.set_material(k, m)
    return ctx


def _impact_block(case, seed):
    F, ids, mats = _bodies(case["n"], case["eos"], case["contact"], seed)
    dt = 0.0
    if case["io"] == "host":   # the last step's forces: gravity about as two point masses, dt about the CFL step
        rng = np.random.default_rng(seed + 2)
        pos = F[[FIELD[c] for c in "xyz"]]
        n_i = max(32, case["n"] // 10)
        for lo, hi in ((0, case["n"] - n_i), (case["n"] - n_i, case["n"])):
            d = pos[:, lo:hi] - pos[:, lo:hi].mean(1, keepdims=True)
            for k, c in enumerate("xyz"):
                F[FIELD["g" + c], lo:hi] = -1.5e-6 * d[k]
        for c in "xyz":
            F[FIELD["a" + c]] = 0.1 * rng.standard_normal(case["n"])
        F[FIELD["eng_dot"]] = 10.0 * rng.standard_normal(case["n"])
        dt = 0.3 * float(F[FIELD["smth"]].min()) / 2.0e4
    if case["eos"] == "mode2":
        F[FIELD["ent"]] = np.where(mats == 0, M2["mantle_entropy"], M2["core_entropy"])
    return F, ids, mats, dt


M2 = {"mantle_entropy": 3000.0, "core_entropy": 2500.0}


def _config(case):
    kw = dict(precision=case["precision"], theta=case["theta"])
    if case["eos"] == "mode2":
        kw |= dict(mode=2, **M2)
    return kw


def _sweep_blocks(case, seed):
    rng = np.random.default_rng(case["runs"])   # the runs' sizes and geometry belong to the case, their particles to the seed
    return [ic.sweep_impact(rng, case["n_lo"], case["n_hi"], seed * 1009 + k)[:3] for k in range(case["runs"])]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "impact":
        F, ids, mats, dt = _impact_block(case, seed)
        return {"case": case, "ctx": _context(_materials(case["eos"]), **_config(case)), "F": _pinned_copy(F),
                "ids": _pinned_copy(ids), "mats": _pinned_copy(mats), "dt": dt, "out": _pinned(F.shape)}
    if kind == "sweep":
        runs = [tuple(_pinned_copy(a) for a in r) for r in _sweep_blocks(case, seed)]
        return {"case": case, "ctx": _context(_materials("table2"), precision="mixed"), "runs": runs,
                "out": _pinned((len(FIELDS), sum(r[0].shape[1] for r in runs)))}
    if kind == "walks":
        return _prepare_walks(case, seed)
    pos = _order_positions(case, seed)
    return {"case": case, "pos": pos, "lib": lib.load(),
            "keys": torch.empty(case["n"], dtype=torch.int64, device="cuda"),
            "order": torch.empty(case["n"], dtype=torch.int32, device="cuda")}


def _order_positions(case, seed):
    F, _, _ = _bodies(max(200, case["n"]), "table2", False, seed)
    return torch.from_numpy(np.ascontiguousarray(F[:3, :case["n"]])).cuda()


# ---------------------------------------------------------------------------
# one pass

def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "impact":
        ctx, F, out = state["ctx"], state["F"], state["out"]
        if case["io"] == "host":
            ctx.upload(F, state["ids"], state["mats"], dt=state["dt"], forces_valid=True, inputs_only=True)
            ctx.step_download(out, lib.STEP_OUTPUT_FIELDS)
            res = {f: out[FIELD[f]] for f in lib.STEP_OUTPUT_FIELDS}
        else:
            ctx.upload(F, state["ids"], state["mats"])
            ctx.prologue()
            ctx.step(case["steps"])
            ctx.download_fields(out, FIELDS)
            res = {f: out[FIELD[f]] for f in FIELDS}
        res["next_dt"] = ctx.time()[1]
        return res
    if kind == "sweep":
        ctx, out = state["ctx"], state["out"]
        handles = [ctx.add_run(F, ids, mats) for F, ids, mats in state["runs"]]
        ctx.step(1 + case["steps"])   # a run's first step is its prologue
        ctx.download_fields(out, FIELDS)
        dts = [ctx.run_info(h)["dt"] for h in handles]
        for h in handles:
            ctx.remove_run(h)
        res = {f: out[FIELD[f]] for f in FIELDS}
        res["next_dt"] = np.array(dts)
        return res
    if kind == "walks":
        return _run_walks(state)
    x, y, z = state["pos"]
    stream = torch.cuda.current_stream().cuda_stream
    rc = state["lib"].sph_morton_order_noalloc(x.data_ptr(), y.data_ptr(), z.data_ptr(), case["n"],
                                               state["keys"].data_ptr(), state["order"].data_ptr(), stream)
    if rc != lib.SPH_OK:
        raise lib.SphError(rc, "sph_morton_order_noalloc")
    return {"keys": state["keys"], "order": state["order"]}


def work(case):
    """Bytes of each input and output once; operations of the interactions that count (pairs inside the
    support, the tree's interactions), by the formulas' own operations."""
    kind = case["kind"]
    if kind == "order":
        return {"bytes": case["n"] * (24 + 12), "flops": case["n"] * 6}
    near, far = 108, 2500
    per_step = 4 * near * 24 + near * 75 + near * 120 + far * 24
    if kind == "walks":
        n = case["n"]
        near, far = min(near, n), min(far, n)
        per = near * (24 + 75 + 120) + far * 24
        size = sum(layouts.SIZES[p + k] for k in KINDS for p in ("epi_", "epj_", "res_"))
        return {"bytes": n * size, "flops": n * per}
    if kind == "sweep":
        n = case["runs"] * (case["n_hi"] - case["n_lo"]) / math.log(case["n_hi"] / case["n_lo"])
        steps = case["steps"] + 1
        return {"bytes": n * 2 * 8 * len(FIELDS), "flops": n * per_step * steps}
    n = case["n"]
    if case["theta"] > 0.6:
        per_step -= 1200 * 24
    if case["io"] == "host":
        return {"bytes": n * 8 * (len(lib.STEP_INPUT_FIELDS) + len(lib.STEP_OUTPUT_FIELDS)), "flops": n * per_step}
    return {"bytes": n * 8 * 2 * len(FIELDS), "flops": n * per_step * (case["steps"] + 1)}


# ---------------------------------------------------------------------------
# the octree and its interaction lists in plain 64-bit torch

def _spread3(v):
    v = v & 0x1fffff
    for s, m in ((32, 0x1f00000000ffff), (16, 0x1f0000ff0000ff), (8, 0x100f00f00f00f00f),
                 (4, 0x10c30c30c30c30c3), (2, 0x1249249249249249)):
        v = (v | (v << s)) & m
    return v


def _order(pos):
    """Morton keys over the root cube, the stable order, and the cube's side (pos [3, n])."""
    lo, hi = pos.amin(1), pos.amax(1)
    side = float((hi - lo).max())
    half = (side if side > 0 else 1.0) * 0.50048828125
    base = (lo + hi) * 0.5 - half
    length = half + half
    q = torch.floor((pos - base[:, None]) * (2097152.0 / length)).clamp(0, 2097151).to(torch.int64)
    keys = (_spread3(q[0]) << 2) | (_spread3(q[1]) << 1) | _spread3(q[2])
    keys, perm = torch.sort(keys, stable=True)
    return keys, perm, length


def _seg_sum(v, seg, m):
    return torch.zeros(m, dtype=v.dtype, device=v.device).index_add_(0, seg, v)


def _lists(pos, mass, keys, length, theta, n_leaf=8, n_group=256):
    """i-groups (start, count) of the sorted particles, and per group its EPJ cells (start, count) and SPJ
    cells as flat (group, cell) pairs, in breadth-first order; cells as (start, count, level, com, mass)."""
    dev = pos.device
    n = pos.shape[1]
    start, count, level, parent = ([torch.zeros(1, dtype=torch.int64, device=dev)] for _ in range(4))
    count[0] += n
    parent[0] -= 1
    at, total = 0, 1
    for L in range(1, 22):
        ps, pc = start[-1], count[-1]
        big = pc > n_leaf
        if not bool(big.any()):
            break
        inside = torch.zeros(n + 1, dtype=torch.int64, device=dev)
        inside.index_add_(0, ps[big], torch.ones_like(ps[big])).index_add_(0, (ps + pc)[big], -torch.ones_like(ps[big]))
        idx = torch.nonzero(torch.cumsum(inside, 0)[:n] > 0).reshape(-1)
        pre = keys[idx] >> (63 - 3 * L)
        new = torch.ones(len(idx), dtype=torch.bool, device=dev)
        new[1:] = pre[1:] != pre[:-1]
        first = torch.nonzero(new).reshape(-1)
        s = idx[first]
        c = torch.diff(first, append=torch.tensor([len(idx)], device=dev))
        par = torch.searchsorted(ps, s, right=True) - 1 + at
        start.append(s), count.append(c), level.append(torch.full_like(s, L)), parent.append(par)
        at, total = total, total + len(s)
    start, count, level, parent = (torch.cat(v) for v in (start, count, level, parent))
    m = len(start)
    # moments of a cell: sums over its particles, level by level
    com = torch.zeros(4, m, dtype=pos.dtype, device=dev)
    for L in range(int(level.max()) + 1):
        c = torch.nonzero(level == L).reshape(-1)
        rep = torch.repeat_interleave(c, count[c])
        off = torch.cumsum(count[c], 0) - count[c]
        p = torch.arange(len(rep), device=dev) - torch.repeat_interleave(off, count[c]) + torch.repeat_interleave(start[c], count[c])
        for k in range(3):
            com[k].index_add_(0, rep, mass[p] * pos[k, p])
        com[3].index_add_(0, rep, mass[p])
    com[:3] /= com[3]
    nch = torch.zeros(m, dtype=torch.int64, device=dev).index_add_(0, parent[1:], torch.ones_like(parent[1:]))
    fch = torch.full((m,), m, dtype=torch.int64, device=dev).scatter_reduce_(0, parent[1:], torch.arange(1, m, device=dev), "amin")
    g = torch.nonzero((count <= n_group) & ((parent < 0) | (count[parent.clamp(min=0)] > n_group))).reshape(-1)
    gs, gc = start[g], count[g]
    rep = torch.repeat_interleave(torch.arange(len(g), device=dev), gc)
    off = torch.cumsum(gc, 0) - gc
    p = torch.arange(len(rep), device=dev) - off[rep] + gs[rep]
    inf = torch.full((3, len(g)), math.inf, dtype=pos.dtype, device=dev)
    lo = torch.stack([inf[k].scatter_reduce(0, rep, pos[k, p], "amin") for k in range(3)])
    hi = torch.stack([(-inf[k]).scatter_reduce(0, rep, pos[k, p], "amax") for k in range(3)])
    rc2 = length * length / (theta * theta) * 0.25 ** torch.arange(23, dtype=pos.dtype, device=dev)
    G, C = torch.arange(len(g), device=dev), torch.zeros(len(g), dtype=torch.int64, device=dev)
    eg, ec, sg, sc = [], [], [], []
    while len(G):
        leaf = nch[C] == 0
        eg.append(G[leaf]), ec.append(C[leaf])
        G, C = G[~leaf], C[~leaf]
        k = nch[C]
        off = torch.cumsum(k, 0) - k
        ch = torch.arange(int(k.sum()), device=dev) - torch.repeat_interleave(off, k) + torch.repeat_interleave(fch[C], k)
        G = torch.repeat_interleave(G, k)
        d = torch.clamp(torch.maximum(lo[:, G] - com[:3, ch], com[:3, ch] - hi[:, G]), min=0)
        near = (d[0] * d[0] + d[1] * d[1]) + d[2] * d[2] <= rc2[level[ch]]
        sg.append(G[~near]), sc.append(ch[~near])
        G, C = G[near], ch[near]
    out = []
    for a, b in ((eg, ec), (sg, sc)):
        a, b = torch.cat(a), torch.cat(b)
        o = torch.sort(a, stable=True)[1]
        out.append((a[o], b[o]))
    return {"gs": gs, "gc": gc, "lo": lo, "hi": hi, "start": start, "count": count, "com": com, "epj": out[0],
            "spj": out[1]}


def _expand(first, num):
    """[first[0], first[0]+1, ... num[0] values, first[1], ...] and the segment of each."""
    seg = torch.repeat_interleave(torch.arange(len(num), device=num.device), num)
    off = torch.cumsum(num, 0) - num
    return torch.arange(len(seg), device=num.device) - off[seg] + first[seg], seg


def _chunks(cost, most=40_000_000):
    """ranges of items whose costs add up to about `most`"""
    c = torch.cumsum(cost, 0).cpu().numpy()
    a = 0
    while a < len(c):
        base = c[a - 1] if a else 0
        b = max(a + 1, int(np.searchsorted(c, base + most, side="right")))
        yield a, b
        a = b


# ---------------------------------------------------------------------------
# walks

def _walk_state(case, seed):
    """a sorted particle state with the fields the functors read, as an impact under way has them"""
    F, ids, mats = _bodies(case["n"], "table2", True, seed)
    rng = np.random.default_rng(seed + 3)
    n = case["n"]
    S = torch.from_numpy(F).cuda()
    keys, perm, length = _order(S[:3])
    S = S[:, perm].contiguous()
    S[FIELD["dens"]] *= torch.from_numpy(1.0 + 0.05 * rng.standard_normal(n)).cuda()
    rho0 = torch.where(S[FIELD["dens"]] > 5500.0, 7800.0, 3320.0)
    S[FIELD["smth"]] = 1.2 * (S[FIELD["mass"]] / S[FIELD["dens"]]) ** (1.0 / 3.0)
    S[FIELD["pres"]] = 1.0e11 * (S[FIELD["dens"]] / rho0 - 1.0) + 0.4 * S[FIELD["dens"]] * S[FIELD["eng"]]
    S[FIELD["snds"]] = torch.from_numpy(rng.uniform(3.0e3, 9.0e3, n)).cuda()
    S[FIELD["grad_smth"]] = torch.from_numpy(rng.uniform(0.9, 1.1, n)).cuda()
    S[FIELD["bal"]] = torch.from_numpy(rng.uniform(0.0, 1.0, n)).cuda()
    return S, torch.from_numpy(ids).cuda()[perm], keys, length


def _walk_lists(S, keys, length):
    """gravity lists, and per group the gather and symmetric supersets of FDPS (flat j, offsets)"""
    T = _lists(S[:3], S[FIELD["mass"]], keys, length, THETA)
    h = S[FIELD["smth"]]
    ng = len(T["gs"])
    i, seg = _expand(T["gs"], T["gc"])
    hg = torch.zeros(ng, dtype=h.dtype, device=h.device).scatter_reduce(0, seg, h[i], "amax") * 2.5
    lists = {"gather": [], "sym": []}
    for a in range(0, ng, 256):
        b = min(ng, a + 256)
        d2 = sum(torch.clamp(torch.maximum(T["lo"][k, a:b, None] - S[k], S[k] - T["hi"][k, a:b, None]), min=0) ** 2
                 for k in range(3))
        for name, reach in (("gather", hg[a:b, None].expand(-1, len(h))), ("sym", torch.maximum(hg[a:b, None], 2.5 * h))):
            m = torch.nonzero(d2 < reach * reach)
            lists[name].append((m[:, 0] + a, m[:, 1]))
    for name in lists:
        g, j = (torch.cat(v) for v in zip(*lists[name]))
        lists[name] = (j, torch.bincount(g, minlength=ng))
    j, seg = _expand(T["start"][T["epj"][1]], T["count"][T["epj"][1]])
    lists["epj"] = (j, torch.bincount(T["epj"][0][seg], minlength=ng))
    lists["spj"] = (T["spj"][1], torch.bincount(T["spj"][0], minlength=ng))
    return T, lists


def _payloads(S, ids):
    f = lambda *k: np.stack([S[FIELD[c]].cpu().numpy() for c in k], 1) if len(k) > 1 else S[FIELD[k[0]]].cpu().numpy()  # noqa: E731
    n = S.shape[1]
    epi = {k: np.zeros(n, lib._KINDS[k][0]) for k in KINDS}
    epj = {k: np.zeros(n, lib._KINDS[k][1]) for k in KINDS}
    pos, vel, ids = f("x", "y", "z"), f("vx", "vy", "vz"), ids.cpu().numpy()
    for k in KINDS:
        epi[k]["pos"] = epj[k]["pos"] = pos
        epj[k]["mass"] = f("mass")
        if k in ("drvt", "hydro"):
            epi[k]["vel"] = epj[k]["vel"] = vel
        if k != "grav":
            epi[k]["smth"] = epj[k]["smth"] = f("smth")
        if k != "drvt":
            epi[k]["id"] = ids
    epi["dens"]["mass"], epi["drvt"]["dens"], epi["grav"]["eps2"] = f("mass"), f("dens"), f("smth") ** 2
    epj["grav"]["id"] = epj["hydro"]["id"] = ids
    for a in (epi["hydro"], epj["hydro"]):
        for k, c in (("dens",) * 2, ("pres",) * 2, ("snds",) * 2, ("grad_smth",) * 2, ("Bal", "bal"), ("AVa", "ava")):
            a[k] = f(c)
    return epi, epj


JLIST = {"dens": "gather", "drvt": "gather", "hydro": "sym", "grav": "epj"}


def _prepare_walks(case, seed, limit=256):
    """every walk's payload (or index) arrays and the callbacks' argument arrays, as FDPS keeps them"""
    S, ids, keys, length = _walk_state(case, seed)
    T, lists = _walk_lists(S, keys, length)
    epi, epj = _payloads(S, ids)
    com = T["com"].cpu().numpy()
    spj = np.zeros(com.shape[1], layouts.SPJ_MONO)
    spj["pos"], spj["mass"] = com[:3].T, com[3]
    index = case["form"] == "index"
    gs, gc = T["gs"].cpu().numpy(), T["gc"].cpu().numpy()
    ng = len(gs)
    keep = {"epi": epi, "epj": epj, "spj": spj}
    res = {k: np.zeros(case["n"], lib._KINDS[k][2]) for k in KINDS}
    flat = {k: (v[0].cpu().numpy().astype(np.int32), np.concatenate([[0], np.cumsum(v[1].cpu().numpy())])) for k, v in lists.items()}

    def pointers(a, off, w0, w1):
        return (ctypes.c_void_p * (w1 - w0))(*[a.ctypes.data + int(o) * a.itemsize for o in off[w0:w1]])

    calls = {}
    for k in KINDS:
        j, jo = flat[JLIST[k]]
        ja = j if index else epj[k][j]
        sj, so = flat["spj"]
        sa = sj if index else spj[sj]
        keep[k] = (ja, sa)
        calls[k] = []
        for w0 in range(0, ng, limit):
            w1 = min(ng, w0 + limit)
            nw = w1 - w0
            ints = lambda v: (ctypes.c_int * nw)(*[int(t) for t in v])  # noqa: E731
            args = [nw, pointers(epi[k], gs, w0, w1), ints(gc[w0:w1]), pointers(ja, jo, w0, w1), ints(np.diff(jo[w0:w1 + 1]))]
            if k == "grav":
                args += [pointers(sa, so, w0, w1), ints(np.diff(so[w0:w1 + 1]))]
            if index:
                args += [epj[k].ctypes.data, len(epj[k])] + ([spj.ctypes.data, len(spj)] if k == "grav" else [])
            calls[k].append((args, pointers(res[k], gs, w0, w1)))
    return {"case": case, "calls": calls, "res": res, "keep": keep, "lib": lib.load()}


def _run_walks(state):
    """the functors of a step over every walk: batches on four tags, a batch's results fetched before its tag
    is used again, as calcForceAllAndWriteBackMultiWalk does"""
    case, L = state["case"], state["lib"]
    lib.batch_precision(case["precision"])

    def ok(rc):
        if rc != lib.SPH_OK:
            raise lib.SphError(rc, L.sph_batch_last_error().decode())

    index = case["form"] == "index"
    for k in KINDS:
        put = getattr(L, f"sph_dispatch_index_{k}" if index else f"sph_dispatch_{k}")
        get = getattr(L, f"sph_retrieve_{k}")
        if index:   # the pass's particles, once
            a = state["calls"][k][0][0]
            none = [0] + [None] * (6 if k == "grav" else 4)
            ok(put(0, *none, *a[len(none):], 1))
        pending = {}
        for b, (args, out) in enumerate(state["calls"][k]):
            tag = b % 4
            if tag in pending:
                ok(get(tag, *pending.pop(tag)))
            ok(put(tag, *args, *([0] if index else [])))
            pending[tag] = (args[0], args[2], out)
        for tag, p in pending.items():
            ok(get(tag, *p))
    return {k: {name: state["res"][k][name] for name in state["res"][k].dtype.names} for k in KINDS}


# ---------------------------------------------------------------------------
# 64-bit restatement of the physics on pairs

def _wendland(r, H):
    s = r / H
    p = torch.clamp(1.0 - s, min=0.0)
    norm = (1365.0 / 64.0) / (H * H * H * math.pi)
    w = norm * (1.0 + s * (8.0 + s * (25.0 + s * 32.0))) * p ** 8
    g = norm * (-22.0) * s * (1.0 + s * (7.0 + s * 16.0)) * p ** 7
    return w, g / (r * H + 1.0e-6 * H / 2.5)


def _sph_pass(kind, P, i, j, out):
    """adds the pairs' terms of one functor to the per-i sums"""
    f = lambda k, a: P[k][a]  # noqa: E731
    d = [f(c, i) - f(c, j) for c in "xyz"]
    r2 = d[0] * d[0] + d[1] * d[1] + d[2] * d[2]
    r = torch.sqrt(r2)
    hi, m = f("smth", i), f("mass", j)
    w, gf = _wendland(r, 2.5 * hi)
    add = lambda k, v: out[k].index_add_(0, i, v)  # noqa: E731
    if kind == "dens":
        add("sum", m * w)
        return
    v = [f("v" + c, i) - f("v" + c, j) for c in "xyz"]
    dvdr = v[0] * d[0] + v[1] * d[1] + v[2] * d[2]
    if kind == "drvt":
        mg = -m * gf
        add("div", mg * dvdr)
        for k in range(3):
            a, b = (k + 1) % 3, (k + 2) % 3
            add("rot%d" % k, mg * (v[a] * d[b] - v[b] * d[a]))
        add("grad", -m / hi * (3.0 * w + gf * r2))
        return
    wr = torch.where(dvdr < 0, dvdr / r, torch.zeros_like(r))
    vs = f("snds", i) + f("snds", j) - 3.0 * wr
    out["vmax"].scatter_reduce_(0, i, vs, "amax")
    av = -0.5 * vs * wr / (0.5 * (f("dens", i) + f("dens", j))) * 0.5 * (f("bal", i) + f("bal", j))
    _, gj = _wendland(r, 2.5 * f("smth", j))
    gw = 0.5 * (gf * f("grad_smth", i) + gj * f("grad_smth", j))
    pi, pj = (f("grad_smth", a) * f("pres", a) / f("dens", a) ** 2 for a in (i, j))
    c = m * (pi * gf + pj * gj + av * gw)
    for k in range(3):
        add("a%d" % k, -c * d[k])
    add("e", m * (pi + 0.5 * av) * gw * dvdr)


SUMS = {"dens": ("sum",), "drvt": ("div", "rot0", "rot1", "rot2", "grad"), "hydro": ("a0", "a1", "a2", "e", "vmax")}


def _sph_sums(kind, P, pairs):
    n = len(P["x"])
    out = {k: torch.zeros(n, dtype=torch.float64, device="cuda") for k in SUMS[kind]}
    for i, j in pairs():
        _sph_pass(kind, P, i, j, out)
    return out


def _density(P, pairs):
    d = torch.clamp(_sph_sums("dens", P, pairs)["sum"], min=5.0)
    return d, 1.2 * (P["mass"] / d) ** (1.0 / 3.0)


def _derivative(P, pairs):
    s = _sph_sums("drvt", P, pairs)
    return (s["div"] / P["dens"], [s["rot%d" % k] / P["dens"] for k in range(3)],
            1.0 / (1.0 + P["smth"] * s["grad"] / (3.0 * P["dens"])))


def _hydro(P, pairs):
    s = _sph_sums("hydro", P, pairs)
    return [s["a%d" % k] for k in range(3)], s["e"], 0.6 * P["smth"] / s["vmax"]


def _gravity(P, eps2, T):
    """EPJ and SPJ sums of every group's particles, from cell lists"""
    n = len(P["x"])
    acc = torch.zeros(4, n, dtype=torch.float64, device="cuda")
    cx = [P["x"], P["y"], P["z"]]

    def add(i, dx, gm):
        dri = 1.0 / torch.sqrt(dx[0] * dx[0] + dx[1] * dx[1] + dx[2] * dx[2] + eps2[i])
        for k in range(3):
            acc[k].index_add_(0, i, -gm * dri ** 3 * dx[k])
        acc[3].index_add_(0, i, -gm * dri)

    g, c = T["spj"]
    for a, b in _chunks(T["gc"][g]):
        i, s = _expand(T["gs"][g[a:b]], T["gc"][g[a:b]])
        q = T["com"][:, c[a:b][s]]
        add(i, [cx[k][i] - q[k] for k in range(3)], ic.G * q[3])
    g, c = T["epj"]
    j, s = _expand(T["start"][c], T["count"][c])
    g = g[s]
    for a, b in _chunks(T["gc"][g]):
        i, s = _expand(T["gs"][g[a:b]], T["gc"][g[a:b]])
        jj = j[a:b][s]
        add(i, [cx[k][i] - cx[k][jj] for k in range(3)], ic.G * P["mass"][jj])
    return acc


def _eos(mats_list, kind, mats, rho, u):
    P, cs = torch.zeros_like(rho), torch.zeros_like(rho)
    for k, m in enumerate(mats_list):
        d = m.as_material()
        a = torch.nonzero(mats == k).reshape(-1)
        r, e = rho[a], u[a]
        if d["kind"] == "table":
            ax, au = (torch.from_numpy(np.ascontiguousarray(d[c])).cuda() for c in ("rho", "u"))
            li = torch.searchsorted(ax, r).clamp(max=len(ax) - 1)
            ci = torch.searchsorted(au, e).clamp(max=len(au) - 1)
            inner = (li < len(ax) - 1) & (ci < len(au) - 1) & (li > 0) & (ci > 0)
            l0, c0 = (li - 1).clamp(min=0), (ci - 1).clamp(min=0)
            xi, et = (r - ax[l0]) / (ax[li] - ax[l0]), (e - au[c0]) / (au[ci] - au[c0])
            for name, out in (("pres", P), ("snds", cs)):
                t = torch.from_numpy(np.ascontiguousarray(d[name])).cuda().reshape(len(ax), len(au))
                v = ((1 - xi) * (1 - et) * t[l0, c0] + xi * (1 - et) * t[li, c0] + (1 - xi) * et * t[l0, ci]
                     + xi * et * t[li, ci])
                out[a] = torch.where(inner, v, t[li, ci])
            continue
        rho0, u0, uiv, ucv, A, B, ca, cb, alpha, beta = (float(v) for v in d["par"])
        eta = r / rho0
        mu, om = eta - 1.0, e / u0 / eta / eta + 1.0
        pc = (ca + cb / om) * r * e + A * mu + B * mu * mu
        pc_r = (ca + cb / om) * e + 2.0 * cb * e * (om - 1.0) / (om * om) + (A + 2.0 * B * mu) / rho0
        pc_u = (ca + cb / om) * r - r * cb * (om - 1.0) / (om * om)
        z = 1.0 / eta - 1.0
        e1, e2 = torch.exp(-alpha * z), torch.exp(-beta * z * z)
        q = cb * r * e / om + A * mu * e1
        q_r = cb * e / om + 2.0 * cb * e * (om - 1.0) / (om * om) + A / rho0 * e1 + A * mu * alpha * e1 * (z + 1.0) / r
        pe = ca * r * e + q * e2
        pe_r = ca * e + q_r * e2 + q * 2.0 * beta * z * (z + 1.0) * e2 / r
        pe_u = ca * r + e2 * (cb * r / om - cb * r * (om - 1.0) / (om * om))
        f = torch.where((r >= rho0) | (e <= uiv), torch.zeros_like(e), ((e - uiv) / (ucv - uiv)).clamp(max=1.0))
        mid = (f > 0) & (f < 1)
        pv = f * pe + (1 - f) * pc
        p_r = f * pe_r + (1 - f) * pc_r
        p_u = f * pe_u + (1 - f) * pc_u + torch.where(mid, (pe - pc) / (ucv - uiv), torch.zeros_like(e))
        c2 = torch.clamp(p_r + pv / (r * r) * p_u, min=1.0e-2 * A / rho0)
        P[a], cs[a] = pv, torch.sqrt(c2)
    return P, cs


def _all_pairs(P, grow):
    """every (i, j) closer than 2.5 grow max(h_i, h_j), in pieces"""
    x = torch.stack([P["x"], P["y"], P["z"]])
    R = 2.5 * grow * P["smth"]
    n = x.shape[1]
    rows = max(1, 100_000_000 // n)
    found = []
    for a in range(0, n, rows):
        b = min(n, a + rows)
        d2 = sum((x[k, a:b, None] - x[k]) ** 2 for k in range(3))
        m = torch.nonzero(d2 < torch.maximum(R[a:b, None], R) ** 2)
        found.append((m[:, 0] + a, m[:, 1]))
    return lambda: found


def _exact_forces(P, mats, mats_list, eos_kind, theta):
    """density x 4, EoS, derivative, hydro, gravity of the state P (a dict of fields), in place"""
    keys, perm, length = _order(torch.stack([P["x"], P["y"], P["z"]]))
    inv = torch.argsort(perm)
    pairs = _all_pairs(P, 1.7)
    for _ in range(4):
        P["dens"], P["smth"] = _density(P, pairs)
    P["pres"], P["snds"] = _eos(mats_list, eos_kind, mats, P["dens"], P["eng"])
    P["div_v"], rot, P["grad_smth"] = _derivative(P, pairs)
    P["rot_x"], P["rot_y"], P["rot_z"] = rot
    dv = P["div_v"].abs()
    P["bal"] = dv / (dv + torch.sqrt(sum(r * r for r in rot)) + 1.0e-4 * P["snds"] / P["smth"])
    # v_sig is over the symmetric set only
    x = [P[c] for c in "xyz"]

    def inside():
        for i, j in pairs():
            d2 = sum((v[i] - v[j]) ** 2 for v in x)
            k = d2 < (2.5 * torch.maximum(P["smth"][i], P["smth"][j])) ** 2
            yield i[k], j[k]

    (P["ax"], P["ay"], P["az"]), P["eng_dot"], P["dt"] = _hydro(P, inside)
    Q = {k: P[k][perm] for k in ("x", "y", "z", "mass")}
    T = _lists(torch.stack([Q["x"], Q["y"], Q["z"]]), Q["mass"], keys, length, theta)
    g = _gravity(Q, (P["smth"] * P["smth"])[perm], T)[:, inv]
    P["gx"], P["gy"], P["gz"], P["pot"] = g
    return float(P["dt"].min())


def _exact_step(P, dt, *how):
    a = {c: P["a" + c] + P["g" + c] for c in "xyz"}
    for c in "xyz":
        P["vh" + c] = P["v" + c] + 0.5 * dt * a[c]
        P[c] = P[c] + dt * P["vh" + c]
        P["v" + c] = P["v" + c] + dt * a[c]
    P["eng_half"] = P["eng"] + 0.5 * dt * P["eng_dot"]
    P["eng"] = P["eng"] + dt * P["eng_dot"]
    new = _exact_forces(P, *how)
    for c in "xyz":
        P["v" + c] = P["vh" + c] + 0.5 * dt * (P["a" + c] + P["g" + c])
    P["eng"] = P["eng_half"] + 0.5 * dt * P["eng_dot"]
    return new


def _exact_walks(case, seed):
    S, _, keys, length = _walk_state(case, seed)
    T, lists = _walk_lists(S, keys, length)
    P = {f: S[k] for k, f in enumerate(FIELDS)}

    def pairs(name):
        j, nj = lists[name]
        first = torch.cumsum(nj, 0) - nj
        for a, b in _chunks(T["gc"] * nj):
            # all i of a group against all of its j
            i, seg = _expand(T["gs"][a:b], T["gc"][a:b])
            jj, s2 = _expand(first[a:b][seg], nj[a:b][seg])
            yield i[s2], j[jj]

    dens, smth = _density(P, lambda: pairs("gather"))
    div, rot, grad = _derivative(P, lambda: pairs("gather"))
    acc, edot, dt = _hydro(P, lambda: pairs("sym"))
    grav = _gravity(P, P["smth"] ** 2, T)
    return {"dens": {"dens": dens, "smth": smth},
            "drvt": {"div_v": div, "rot_v": torch.stack(rot, 1), "grad_smth": grad},
            "hydro": {"acc": torch.stack(acc, 1), "eng_dot": edot, "dt": dt},
            "grav": {"acc": grav[:3].T.contiguous(), "pot": grav[3], "dt": None}}


def exact(case, seed):
    kind = case["kind"]
    if kind == "walks":
        return _exact_walks(case, seed) if case["n"] <= 120_000 else None
    if kind == "order":
        pos = _order_positions(case, seed)
        keys, perm, _ = _order(pos)
        return {"keys": keys, "order": perm.to(torch.int32)}
    if kind != "impact" or case["eos"] == "mode2" or case["n"] > MAX_EXACT:
        return None
    F, _, mats, dt = _impact_block(case, seed)
    mats = torch.from_numpy(mats).cuda()
    P = {f: torch.from_numpy(F[k].copy()).cuda() for k, f in enumerate(FIELDS)}
    how = (mats, _materials(case["eos"]), case["eos"], case["theta"])
    if case["io"] == "host":
        new = _exact_step(P, dt, *how)
        out = {f: P[f] for f in lib.STEP_OUTPUT_FIELDS}
    else:
        new = _exact_forces(P, *how)
        for _ in range(case["steps"]):
            new = _exact_step(P, new, *how)
        out = {f: P[f] for f in FIELDS}
    return out | {"next_dt": new}
