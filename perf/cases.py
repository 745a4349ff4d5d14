"""The work that users of this framework have it do, as cases that can be timed.

Particle step (sdem_gb300.capi): a host program uploads a bed once, advances
it by some steps between two outputs and takes the state into page-locked
arrays that it reuses; or it uploads, steps and downloads each time (the
plain path as judge of another model does that); or it advances many small
beds together.  Learned surrogate (sdem_gb300.surrogate): a neighbour graph,
a forward pass, a training step, and one edge layer in both directions.

listed()   the cases, with a size each
draw(rng)  another case of the same ranges
prepare    what a program has in hand before the call
run        one pass through the public entry points
work       bytes and operations that the pass cannot do without
exact      the results in 64 bits, from plain torch
"""
from __future__ import annotations

import ctypes
import math

import numpy as np
import torch

from sdem_gb300 import beds, props
from sdem_gb300 import surrogate as sg
from sdem_gb300.capi import DEMBatch, DEMSystem

DEV = "cuda"
LATENT = 128
DMAX = 1.2e-3          # largest diameter of the polydisperse material
VSCALE = 0.05          # velocity scale of the surrogate's features
EDGES_PER_SPHERE = 19  # neighbours within 1.5 d_max in a packed bed
BATCH_MEMBERS = 16


def listed():
    return [
        # the smallest bed of the sandbox workload: one simulation of a few
        # thousand spheres, watched every 20 steps; launches and latency
        {"name": "step_lsd_2k", "kind": "step", "bed": "sandbox", "model": "lsd", "n": 2000, "steps": 20},
        # a laboratory-size bed of 20k LSD spheres in contact, AB2, odd count
        {"name": "step_lsd_20k", "kind": "step", "bed": "sandbox", "model": "lsd", "n": 20011, "steps": 20},
        # the 1M polydisperse Hertz configuration (41 types, five walls)
        # resting on itself, 20 steps between outputs
        {"name": "step_hertz_1m", "kind": "step", "bed": "column", "model": "hertz", "n": 1000000, "steps": 20},
        # bidisperse 1:3 hopper of finite quads discharging through its
        # outlet, hierarchical search
        {"name": "step_hopper_400k", "kind": "step", "bed": "hopper", "model": "hertz", "n": 400009, "steps": 20},
        # a shear cell without side walls: periodic in x and z, a floor,
        # Adams-Bashforth 3, speed-scaled rolling resistance
        {"name": "step_periodic_60k", "kind": "step", "bed": "periodic", "model": "hertz", "n": 60000, "steps": 20},
        # a host program that keeps the state itself: upload, 20 steps,
        # download, each time (judged strides, coupled solvers)
        {"name": "cycle_hertz_200k", "kind": "cycle", "bed": "column", "model": "hertz", "n": 200003, "steps": 20},
        # a parameter sweep: independent sandboxes of 2,000 to 50,000 spheres
        # advanced together by one batch
        {"name": "batch_sandboxes", "kind": "batch", "n_lo": 2000, "n_hi": 50000, "steps": 10},
        # surrogate rollout: the neighbour graph is built anew every stride
        {"name": "graph_200k", "kind": "graph", "n": 200003},
        # surrogate rollout: the forward pass on a bed of sandbox size
        {"name": "forward_50k", "kind": "forward", "n": 50000},
        # surrogate training: one optimiser step on one sandbox frame
        {"name": "train_16k", "kind": "train", "n": 16011},
        # the network's largest layer alone (first edge layer): forward with
        # gathered inputs, input gradient, weight gradient
        {"name": "edge_layer_600k", "kind": "layer", "n": 31579, "edges": 600005},
    ]


def draw(rng):
    def size(lo, hi):
        n = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
        return n | 1 if rng.random() < 0.5 else n

    kind = rng.choice(["step", "step", "step", "step", "cycle", "batch", "graph", "forward", "train", "layer"])
    if kind == "step":
        bed = rng.choice(["sandbox", "sandbox", "column", "hopper", "periodic"])
        lo, hi = {"sandbox": (2000, 50000), "column": (20000, 900000), "hopper": (20000, 400000),
                  "periodic": (4000, 60000)}[bed]
        model = rng.choice(["lsd", "hertz"]) if bed == "sandbox" else "hertz"
        return {"kind": kind, "bed": bed, "model": model, "n": size(lo, hi), "steps": rng.choice([6, 10, 13, 20])}
    if kind == "cycle":
        return {"kind": kind, "bed": "column", "model": "hertz", "n": size(20000, 400000),
                "steps": rng.choice([6, 10, 20])}
    if kind == "batch":
        hi = size(8000, 50000)
        return {"kind": kind, "n_lo": 2000, "n_hi": hi, "steps": rng.choice([6, 10])}
    if kind == "graph":
        return {"kind": kind, "n": size(4000, 400000)}
    if kind == "forward":
        return {"kind": kind, "n": size(2000, 50000)}
    if kind == "train":
        return {"kind": kind, "n": size(1000, 16000)}
    e = size(20000, 600000)
    return {"kind": kind, "n": max(e // EDGES_PER_SPHERE, 64), "edges": e}


# ------------------------------------------------------------------ inputs

def _column(n, seed):
    """n spheres of the 1M configuration's material (41 types, Hertz, five
    walls, as wide as high) at a settled bed's solid fraction, in contact: a
    jittered face-centred lattice, neighbours pushed apart until they overlap
    by no more than resting contacts do, stored in random order."""
    rng = np.random.default_rng(seed)
    diam, tables = beds.hertz_poly_tables(41)
    a = (4.0 * math.pi / 6.0 * float((diam ** 3).mean()) / 0.59) ** (1.0 / 3.0)
    m = max(2, int(round((n / 4.0) ** (1.0 / 3.0))))
    k = -(-n // (4 * m * m))
    side = m * a
    opts, walls = beds.hertz_poly_setup((side, 2.0 * k * a, side))
    cells = np.stack(np.meshgrid(np.arange(k), np.arange(m), np.arange(m), indexing="ij"), -1).reshape(-1, 1, 3)
    basis = np.array([[0.25, 0.25, 0.25], [0.25, 0.75, 0.75], [0.75, 0.25, 0.75], [0.75, 0.75, 0.25]])
    pos = ((cells + basis).reshape(-1, 3) * a)[:n, [1, 0, 2]]     # from the floor up
    pos = (pos + rng.uniform(-0.05, 0.05, size=pos.shape) * a)[rng.permutation(n)]
    ptype = rng.integers(1, len(diam) + 1, size=n).astype(np.int32)
    pos = _relaxed(pos, tables.radius[ptype - 1], opts.maxpoint)
    p = beds.new_particles(pos, ptype, tables.radius, rng.uniform(-0.01, 0.01, size=(n, 3)), opts.tsize, opts.rsize)
    p.rotVel[:] = rng.uniform(-5.0, 5.0, size=(n, 1, 3))
    return beds.Case(f"column_{n}_{seed}", opts, tables, walls, p)


def _relaxed(pos, radius, box):
    """Centres moved until neighbours (and walls) overlap by about a micron."""
    x = torch.from_numpy(np.ascontiguousarray(pos)).to(DEV)
    r = torch.from_numpy(np.ascontiguousarray(radius)).to(DEV)
    lo = torch.stack([r, r, r], 1) - 1.0e-6
    hi = torch.tensor(box, dtype=torch.float64, device=DEV) - lo
    for _ in range(4):
        i, j = _near_pairs(x, r, 1.0e-4)
        a, b = torch.cat([i, j]), torch.cat([j, i])
        order = torch.argsort(a, stable=True)
        a, b = a[order], b[order]
        count = torch.bincount(a, minlength=len(x))
        rank = torch.arange(len(a), device=DEV) - (torch.cumsum(count, 0) - count)[a]
        table = torch.arange(len(x), device=DEV)[:, None].repeat(1, int(count.max()))   # padded with itself
        table[a, rank] = b
        rs = torch.where(table == torch.arange(len(x), device=DEV)[:, None], 0.0, r[:, None] + r[table] - 1.0e-6)
        for _ in range(60):
            d = x[:, None, :] - x[table]
            dist = d.norm(dim=2).clamp_min(1.0e-9)
            push = (rs - dist).clamp_min(0.0) / dist
            x = torch.minimum(torch.maximum(x + 0.3 * (d * push[:, :, None]).sum(1), lo), hi)
    return x.cpu().numpy()


def _sandbox(n, seed, cf):
    """A sandbox bed already in contact (overlaps of about a micron) and
    still moving, as one that settles."""
    c = beds.sandbox_case(np.random.default_rng(seed), 0, n_lo=n, n_hi=n, layout="deposited", cf_type=cf)
    rng = np.random.default_rng(seed + 1)
    c.particles.posR[:, 1] *= 0.999
    c.particles.linVel[:] = rng.uniform(-0.05, 0.05, size=(n, 1, 3))
    c.particles.rotVel[:] = rng.uniform(-5.0, 5.0, size=(n, 1, 3))
    return c


def _bed(case, seed):
    """The beds.Case of a step or cycle case."""
    n, bed = case["n"], case["bed"]
    if bed == "sandbox":
        return _sandbox(n, seed, props.CFT_LSD if case["model"] == "lsd" else props.CFT_NLIN)
    if bed == "column":
        return _column(n, seed)
    if bed == "hopper":
        width = 0.27 * (n / 4.0e6) ** (1.0 / 3.0) + 4.0e-3
        c = beds.hopper_case(n, seed, width=width, outlet=min(10.0e-3, 0.3 * width))
        return beds.scaled(c, cs_method=2)
    c = beds.periodic_lattice_case(n, seed, periodic=(1, 0, 1), nn=1.15e-3, pi=3, pri=3, vmax=0.1)
    return beds.scaled(c, ct_model=2)


def _members(case):
    """(spheres, contact model) of each bed of a batch, spread over its range."""
    step = (case["n_hi"] - case["n_lo"]) / (BATCH_MEMBERS - 1)
    return [(int(case["n_lo"] + k * step), (props.CFT_LSD, props.CFT_NLIN)[k % 2]) for k in range(BATCH_MEMBERS)]


def _pinned(rows, opts):
    """Page-locked state arrays of `rows` rows, as a program reuses them."""
    def f64(*shape):
        return torch.zeros(shape, dtype=torch.float64, pin_memory=True).numpy()

    def i32():
        return torch.zeros(rows, dtype=torch.int32, pin_memory=True).numpy()

    return beds.Particles(i32(), i32(), i32(), f64(rows, 4), f64(rows, opts.tsize, 3), f64(rows, opts.tsize, 3),
                          f64(rows, 3), f64(rows, opts.rsize, 3), f64(rows, opts.rsize, 3))


def _copy_into(dst, src):
    for f in ("id", "ptype", "usrmark", "posR", "linVel", "linAcc", "theta", "rotVel", "rotAcc"):
        getattr(dst, f)[...] = getattr(src, f)
    return dst


def _packed(n, seed):
    """A packed bed and the surrogate's view of it on the GPU."""
    c = _column(n, n)
    # one bed of this size, its spheres stored in the seed's order
    posR = torch.from_numpy(c.particles.posR[np.random.default_rng(seed).permutation(n)]).to(DEV)
    return c, posR, sg.make_grid(c.opts.minpoint, c.opts.maxpoint, DMAX)


def _sample(n, seed, sender_order):
    c, posR, grid = _packed(n, seed)
    g = torch.Generator(device=DEV).manual_seed(seed)
    vel = torch.randn((3, n, 3), dtype=torch.float64, device=DEV, generator=g) * VSCALE
    omega = torch.randn((n, 3), dtype=torch.float64, device=DEV, generator=g) * 30.0
    planes = torch.from_numpy(sg.planes_of(c.walls)).to(DEV)
    graph = sg.build_graph(posR, grid, sender_order=sender_order)
    xn = sg.node_features(posR, vel, omega, planes, DMAX, VSCALE)
    target = torch.randn((n, sg.OUT_USED), dtype=torch.float32, device=DEV, generator=g)
    return graph, xn, target


def _layer_inputs(case, seed):
    n, e = case["n"], case["edges"]
    g = torch.Generator(device=DEV).manual_seed(seed)

    def normal(*shape, scale):
        return (torch.randn(shape, device=DEV, generator=g) * scale).to(torch.bfloat16)

    dst = torch.sort(torch.randint(0, n, (e,), device=DEV, generator=g, dtype=torch.int32)).values
    src = torch.randint(0, n, (e,), device=DEV, generator=g, dtype=torch.int32)
    return {"h": normal(n, LATENT, scale=0.5), "e": normal(e, LATENT, scale=0.5), "dst": dst, "src": src,
            "w": normal(LATENT, 3 * LATENT, scale=0.07), "b": torch.randn(LATENT, device=DEV, generator=g) * 0.05,
            "dz": normal(e, LATENT, scale=1.0e-3)}


def _operand(trans, *segs):
    """sdem_sg_operand over (tensor, row indices or None) segments."""
    o = sg.SgOperand()
    o.trans, o.nseg = trans, len(segs)
    for k, (t, idx) in enumerate(segs):
        o.ptr[k] = t.data_ptr()
        o.idx[k] = idx.data_ptr() if idx is not None else None
        o.ld[k] = o.width[k] = t.shape[1]
    return o


def _epilogue(**kw):
    e = sg.SgEpilogue()
    for k, v in kw.items():
        setattr(e, k, v.data_ptr() if isinstance(v, torch.Tensor) else v)
    return e


def prepare(case, seed):
    kind = case["kind"]
    if kind == "step":
        bed = _bed(case, seed)
        s = DEMSystem(bed)
        s.step(2)
        return {"case": case, "sys": s, "out": _pinned(s.cfg.n_capacity, bed.opts)}
    if kind == "cycle":
        bed = _bed(case, seed)
        s = DEMSystem(bed)
        s.step(2)
        rows = s.cfg.n_capacity
        start = _copy_into(_pinned(rows, bed.opts), bed.particles)
        return {"case": case, "sys": s, "start": start, "out": _pinned(rows, bed.opts)}
    if kind == "batch":
        members = [DEMSystem(_sandbox(n, BATCH_MEMBERS * seed + k, cf)) for k, (n, cf) in enumerate(_members(case))]
        batch = DEMBatch(members)
        batch.step(2)
        return {"case": case, "members": members, "batch": batch,
                "out": [_pinned(m.cfg.n_capacity, m.case.opts) for m in members]}
    if kind == "graph":
        _, posR, grid = _packed(case["n"], seed)
        return {"case": case, "posR": posR, "grid": grid}
    if kind == "forward":
        graph, xn, _ = _sample(case["n"], seed, False)
        return {"case": case, "net": sg.Network(seed=seed), "graph": graph, "xn": xn}
    if kind == "train":
        graph, xn, target = _sample(case["n"], seed, True)
        return {"case": case, "net": sg.Network(seed=seed), "graph": graph, "xn": xn, "target": target}
    s = _layer_inputs(case, seed)
    e, wide = case["edges"], 3 * LATENT
    s["z"] = torch.empty((e, LATENT), dtype=torch.bfloat16, device=DEV)
    s["dx"] = torch.empty((e, wide), dtype=torch.float32, device=DEV)
    s["dw"] = torch.empty((LATENT, wide), dtype=torch.float32, device=DEV)
    # the split of the reduction that the network's own backward pass asks for
    s["splits"] = max(1, min(e // 256, 608 // (6 * 2)))
    s["partial"] = torch.empty(s["splits"] * LATENT * wide, dtype=torch.float32, device=DEV)
    s["case"], s["lib"] = case, sg.load()
    return s


# -------------------------------------------------------------------- pass

def _state(p):
    return {"id": p.id, "posR": p.posR, "linVel": p.linVel, "linAcc": p.linAcc, "theta": p.theta,
            "rotVel": p.rotVel, "rotAcc": p.rotAcc}


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind in ("step", "cycle"):
        s = state["sys"]
        if kind == "cycle":
            s.upload(state["start"])
        s.step(case["steps"])
        s.state(out=state["out"])
        out = _state(state["out"])
        c = s.counters()
        out["counters"] = np.array([c[k] for k in ("pp", "ppg", "pw", "cnsv", "nlocal", "cnsv_cross")], np.int64)
        return out
    if kind == "batch":
        state["batch"].step(case["steps"])
        outs = []
        for m, buf in zip(state["members"], state["out"]):
            m.state(out=buf)
            outs.append({"posR": buf.posR, "linVel": buf.linVel, "rotVel": buf.rotVel})
        return outs
    if kind == "graph":
        g = sg.build_graph(state["posR"], state["grid"], sender_order=False)
        return {"row_off": g.row_off, "dst": g.dst, "src": g.src, "efeat": g.efeat}
    if kind == "forward":
        return state["net"].forward(state["graph"], state["xn"], keep=False)
    if kind == "train":
        net = state["net"]
        loss = net.train_step(state["graph"], state["xn"], state["target"], lr=1.0e-3)
        return {"loss": loss, "grad": net.grad, "weights": net.p}
    lib, n_e, wide = state["lib"], case["edges"], 3 * LATENT
    stream = torch.cuda.current_stream().cuda_stream

    def gemm(i, j, r, a, b, ep, splits, partial):
        rc = lib.sdem_sg_gemm(i, j, r, ctypes.byref(a), ctypes.byref(b), ctypes.byref(ep), splits, partial, stream)
        if rc:
            raise RuntimeError(f"sdem_sg_gemm: code {rc}")

    x = ((state["h"], state["dst"]), (state["h"], state["src"]), (state["e"], None))
    gemm(n_e, LATENT, wide, _operand(0, *x), _operand(0, (state["w"], None)),
         _epilogue(bias=state["b"], relu=1, out_bf=state["z"], ld_out_bf=LATENT), 1, None)
    gemm(n_e, wide, LATENT, _operand(0, (state["dz"], None)), _operand(1, (state["w"], None)),
         _epilogue(out=state["dx"], ld_out=wide), 1, None)
    gemm(LATENT, wide, n_e, _operand(1, (state["dz"], None)), _operand(1, *x),
         _epilogue(out=state["dw"], ld_out=wide), state["splits"], state["partial"].data_ptr())
    return {"z": state["z"], "dx": state["dx"], "dw": state["dw"]}


# -------------------------------------------------------------------- work

def _step_work(n, contacts, levels):
    """One step: per sphere the state read and written (position, radius,
    velocities, accelerations, rotations and their history) and per contact
    its key and spring read and written; operations of the force law and of
    the update."""
    per = 2 * (4 + 3 + 6 * levels + 6 * levels) * 8
    return per * n + 80.0 * contacts, 136.0 * contacts + 60.0 * n


def _network_flops(n, e):
    edge = 2 * (16 * LATENT + LATENT * LATENT) + sg.LAYERS * 2 * (4 * LATENT * LATENT)
    node = 2 * (32 * LATENT + LATENT * LATENT) + sg.LAYERS * 2 * (3 * LATENT * LATENT) + 2 * (LATENT * LATENT
                                                                                              + LATENT * 16)
    return float(e) * edge + float(n) * node


def work(case):
    kind = case["kind"]
    if kind in ("step", "cycle"):
        n, steps = case["n"], case["steps"]
        levels = 3 if case["bed"] == "periodic" else 2
        contacts = {"sandbox": 0.5, "column": 1.55, "hopper": 0.05, "periodic": 0.3}[case["bed"]] * n
        b, f = _step_work(n, contacts, levels)
        state = n * (12 + 8 * (4 + 3 + 12 * levels))
        return {"bytes": steps * b + state * (2 if kind == "cycle" else 1), "flops": steps * f}
    if kind == "batch":
        n = sum(m for m, _ in _members(case))
        b, f = _step_work(n, 0.4 * n, 2)
        return {"bytes": case["steps"] * b + n * 8 * 16, "flops": case["steps"] * f}
    if kind == "graph":
        e = EDGES_PER_SPHERE * case["n"]
        return {"bytes": 36.0 * case["n"] + 40.0 * e, "flops": 8.0 * 4 * e}
    if kind in ("forward", "train"):
        n = case["n"]
        e = EDGES_PER_SPHERE * n
        params = 4 * sg.param_count()
        if kind == "forward":
            return {"bytes": float(n * (64 + 64) + e * 40 + params), "flops": _network_flops(n, e)}
        return {"bytes": float(n * (64 + 24) + e * 48 + 8 * params), "flops": 3.0 * _network_flops(n, e)}
    n, e, wide = case["n"], case["edges"], 3 * LATENT
    return {"bytes": float(2 * n * LATENT + e * (2 * LATENT + 8 + 2 * LATENT + 2 * LATENT + 4 * wide)
                           + 6 * LATENT * wide), "flops": 3 * 2.0 * e * LATENT * wide}


# ------------------------------------------------- the results in 64 bits

def _near_pairs(x, r, skin):
    """Index pairs i < j whose gap is below `skin`, by cells."""
    cell = float(2.0 * r.max()) + skin
    c = torch.floor((x - x.min(0).values) / cell).long() + 1
    dim = c.max(0).values + 2
    key = (c[:, 0] * dim[1] + c[:, 1]) * dim[2] + c[:, 2]
    order = torch.argsort(key, stable=True)
    skey = key[order]
    most = int(torch.unique_consecutive(skey, return_counts=True)[1].max())
    me = torch.arange(len(x), device=x.device)
    found = []
    for dx in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dz in (-1, 0, 1):
                k = key + (dx * dim[1] + dy) * dim[2] + dz
                lo, hi = torch.searchsorted(skey, k), torch.searchsorted(skey, k, right=True)
                for m in range(most):
                    at = lo + m
                    i = me[at < hi]
                    j = order[at[at < hi]]
                    i, j = i[j > i], j[j > i]
                    on = (x[i] - x[j]).norm(dim=1) < r[i] + r[j] + skin
                    found.append(torch.stack([i[on], j[on]]))
    return torch.cat(found, 1)


def _force_law(model, dt, P, vi, vj, wi, wj, ri, rj, nv, ov, tan, vrel):
    """Spring-dashpot or Hertz-Mindlin contact: (S, M, Mr, tan, vrel)."""
    dot = lambda a, b: (a * b).sum(1, keepdim=True)
    cross = lambda a, b: torch.linalg.cross(a, b)
    V = vi - vj + cross(wi * ri + wj * rj, nv)
    vrn = dot(V, nv)
    vrel = torch.where(vrel < -1.0, vrn.abs(), vrel)
    vt = V - nv * vrn
    n1 = tan.norm(dim=1, keepdim=True)
    tan = tan - nv * dot(tan, nv)
    n2 = tan.norm(dim=1, keepdim=True)
    tan = torch.where(n2 > 1e-10, tan * (n1 / n2.clamp_min(1e-300)), torch.zeros_like(tan)) + vt * dt
    kn, kt, cn, mus, muk, mur, reff = (P[:, k:k + 1] for k in (2, 3, 4, 8, 9, 10, 0))
    if model == props.CFT_LSD:
        vin = vrel.clamp_min(0.01)
        fn = -kn * vin ** 0.4 * ov - cn * vin ** 0.2 * vrn
        k_t = -kt * vin ** 0.4
    else:
        fn = -kn * ov ** 1.5 - cn * ov ** 0.25 * vrn
        k_t = -kt * ov ** 0.5
    ft = tan * k_t
    size = ft.norm(dim=1, keepdim=True)
    slide = size > mus * fn.abs()
    ft = torch.where(slide, ft * (muk * fn.abs() / size.clamp_min(1e-300)), ft)
    tan = torch.where(slide, ft / k_t, tan)
    w = wi - wj
    wn = w.norm(dim=1, keepdim=True)
    w = torch.where(wn > 1e-10, w / wn.clamp_min(1e-300), torch.zeros_like(w))
    return nv * fn + ft, cross(nv, ft), w * (-mur * fn.abs() * reff), tan, vrel


def _exact_steps(case, seed):
    """The state after prepare()'s two steps and one pass, for beds in boxes
    of infinite walls under Adams-Bashforth 2.  Images at periodic faces and
    the finite quads of a hopper have no short plain statement: None."""
    if case["bed"] not in ("sandbox", "column"):
        return None
    bed = _bed(case, seed)
    o, t = bed.opts, bed.tables
    nT = t.n_types
    gpu = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(DEV)
    p = bed.particles
    typ = gpu(p.ptype).long() - 1
    x, r = gpu(p.posR[:, :3]), gpu(p.posR[:, 3:4])
    v, v2 = gpu(p.linVel[:, 0]), gpu(p.linVel[:, 1])
    a, a2 = gpu(p.linAcc[:, 0]), gpu(p.linAcc[:, 1])
    w, w2 = gpu(p.rotVel[:, 0]), gpu(p.rotVel[:, 1])
    al, al2 = gpu(p.rotAcc[:, 0]), gpu(p.rotAcc[:, 1])
    th = gpu(p.theta)
    bpp, bpw = gpu(t.bpp).view(nT * nT, 11), gpu(t.bpw).view(-1, nT, 11)
    mass, inertia = gpu(t.mass)[typ][:, None], gpu(t.inertia)[typ][:, None]
    grav = torch.tensor(o.gravity, dtype=torch.float64, device=DEV)
    i, j = _near_pairs(x, r[:, 0], 1.0e-4)
    P = bpp[typ[j] * nT + typ[i]]
    zero = lambda m: torch.zeros((m, 3), dtype=torch.float64, device=DEV)
    fresh = lambda m: torch.full((m, 1), -2.0, dtype=torch.float64, device=DEV)
    tan, vrel = zero(len(i)), fresh(len(i))
    walls = [gpu(q) for q in bed.walls.walls]
    wtan, wvrel = [zero(len(x)) for _ in walls], [fresh(len(x)) for _ in walls]
    for _ in range(case["steps"] + (2 if case["kind"] == "step" else 0)):
        F, T = zero(len(x)), zero(len(x))
        d = x[j] - x[i]
        on = torch.nonzero(((d * d).sum(1, keepdim=True) <= (r[i] + r[j]) ** 2)[:, 0])[:, 0]
        ia, ja = i[on], j[on]
        dist = d[on].norm(dim=1, keepdim=True)
        S, M, Mr, tn, vr = _force_law(o.cf_type, o.dt, P[on], v[ia], v[ja], w[ia], w[ja], r[ia], r[ja], d[on] / dist,
                                      r[ia] + r[ja] - dist, tan[on], vrel[on])
        tan, vrel = zero(len(i)), fresh(len(i))
        tan[on], vrel[on] = tn, vr
        F.index_add_(0, ia, S).index_add_(0, ja, -S)
        T.index_add_(0, ia, r[ia] * M + Mr).index_add_(0, ja, r[ja] * M - Mr)
        for k, q in enumerate(walls):
            s = (x @ q[12:15] + q[15])[:, None]
            on = torch.nonzero(((s >= 0) & (r - s >= 0))[:, 0])[:, 0]
            rest = zero(len(on))
            S, M, Mr, tn, vr = _force_law(o.cf_type, o.dt, bpw[0][typ[on]], v[on], rest, w[on], rest, r[on], r[on],
                                          (-q[12:15]).expand(len(on), 3), (r - s)[on], wtan[k][on], wvrel[k][on])
            wtan[k], wvrel[k] = zero(len(x)), fresh(len(x))
            wtan[k][on], wvrel[k][on] = tn, vr
            F.index_add_(0, on, S)
            T.index_add_(0, on, r[on] * M + Mr)
        a, al = F / mass + grav, T / inertia
        x = x + o.dt * (1.5 * v - 0.5 * v2)
        v, v2, a2 = v + o.dt * (1.5 * a - 0.5 * a2), v, a
        wa = v if o.quirk_ab2_rot else w          # the update the reference makes
        th = th + o.dt * (1.5 * wa - 0.5 * w2)
        w, w2, al2 = wa + o.dt * (1.5 * al - 0.5 * al2), wa, al
    st = lambda *q: torch.stack(q, 1)
    return {"id": None, "posR": torch.cat([x, r], 1), "linVel": st(v, v2), "linAcc": st(a, a2), "theta": th,
            "rotVel": st(w, w2), "rotAcc": st(al, al2), "counters": None}


def _exact_graph(case, seed):
    """Edges in the order neighbour cell, sphere index; features in 64 bits."""
    _, posR, grid = _packed(case["n"], seed)
    lo = torch.tensor(list(grid.lo), dtype=torch.float64, device=DEV)
    dim = list(grid.dim)
    c = torch.floor((posR[:, :3] - lo) / grid.cell).long()
    key = (c[:, 2] * dim[1] + c[:, 1]) * dim[0] + c[:, 0]
    order = torch.argsort(key, stable=True)
    skey = key[order]
    most = int(torch.unique_consecutive(skey, return_counts=True)[1].max())
    rows = []
    for dz in (-1, 0, 1):
        for dy in (-1, 0, 1):
            for dx in (-1, 0, 1):
                k = key + (dz * dim[1] + dy) * dim[0] + dx
                s, e = torch.searchsorted(skey, k), torch.searchsorted(skey, k, right=True)
                for m in range(most):
                    at = s + m
                    j = order[at.clamp_max(len(order) - 1)]
                    near = ((posR[j, :3] - posR[:, :3]) ** 2).sum(1) < grid.cutoff ** 2
                    me = torch.arange(len(j), device=DEV)
                    rows.append(torch.where((at < e) & near & (j != me), j, torch.full_like(j, -1)))
    table = torch.stack(rows, 1)
    i, col = torch.nonzero(table >= 0, as_tuple=True)
    j = table[i, col]
    d = posR[j, :3] - posR[i, :3]
    dist = d.norm(dim=1)
    ov = (posR[i, 3] + posR[j, 3] - dist).clamp_min(0.0)
    feat = torch.zeros((len(i), sg.EDGE_IN), dtype=torch.float64, device=DEV)
    feat[:, :3], feat[:, 3], feat[:, 4] = d / grid.scale, dist / grid.scale, 100.0 * ov / grid.scale
    return {"row_off": None, "dst": None, "src": None, "efeat": feat}


def _exact_network(params, layout, graph, xn):
    """The network's output for 64-bit parameters (a dict by name)."""
    q = params
    mlp = lambda name, u: torch.relu(u @ q[name + ".w1"].T + q[name + ".b1"]) @ q[name + ".w2"].T + q[name + ".b2"]
    dst, src = graph.dst.long(), graph.src.long()
    h, e = mlp("enc_n", xn), mlp("enc_e", graph.efeat.double())
    for k in range(sg.LAYERS):
        m = mlp(f"edge{k}", torch.cat([h[dst], h[src], e], 1))
        e = e + m
        agg = torch.zeros_like(h).index_add(0, dst, m)
        h = h + mlp(f"node{k}", torch.cat([h, agg], 1))
    return mlp("dec", h)


def _named(flat, layout):
    return {name: flat[off:off + int(np.prod(shape))].view(shape) for name, shape, off in layout}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("step", "cycle"):
        return _exact_steps(case, seed)
    if kind == "batch":
        return None   # each member is a step case of its own
    if kind == "graph":
        return _exact_graph(case, seed)
    layout = sg.param_layout()
    if kind in ("forward", "train"):
        graph, xn, target = _sample(case["n"], seed, False)
        master = torch.from_numpy(sg.init_params(seed)).to(DEV)
        flat = master.double()
        for name, shape, off in layout:   # weights are bf16 operands, biases stay fp32
            if ".w" in name:
                m = int(np.prod(shape))
                flat[off:off + m] = master[off:off + m].bfloat16().double()
        if kind == "forward":
            with torch.no_grad():
                return _exact_network(_named(flat, layout), layout, graph, xn.double())
        flat.requires_grad_(True)
        y = _exact_network(_named(flat, layout), layout, graph, xn.double())
        loss = ((y[:, :sg.OUT_USED] - target.double()) ** 2).mean()
        loss.backward()
        g = flat.grad
        # the first Adam step from zero moments: both bias corrections cancel
        return {"loss": loss.detach(), "grad": g, "weights": master.double() - 1.0e-3 * g / (g.abs() + 1.0e-8)}
    s = _layer_inputs(case, seed)
    x = torch.cat([s["h"][s["dst"].long()], s["h"][s["src"].long()], s["e"]], 1).double()
    w, dz = s["w"].double(), s["dz"].double()
    return {"z": torch.relu(x @ w.T + s["b"].double()), "dx": dz @ w, "dw": dz.T @ x}
