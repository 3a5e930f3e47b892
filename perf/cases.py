"""What is timed: the work that a program built on this engine has it do.

Every case is one call (or one loop of calls) of the public API on inputs made
from a seed: whole forward solves of flat-shell plates in both precisions and
on every mesh kind, batches of plates, the 3D solid, the misfit gradient, the
wavefield images and the allocation-free internal force.  The sizes are those
of the engine's reference configurations with the number of time steps cut to
what a pass of a fraction of a second allows; ``draw`` spreads them over the
same ranges.

A plan of precision 32 computes FP32 numbers, which the C ABI hands over in
FP64 arrays; the programs here keep them as FP32.
"""
from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

import __graft_entry__ as _entry

pkg = _entry.package()
from mashm_gb300 import element as EL  # noqa: E402  (registered by package())
from mashm_gb300 import materials as M  # noqa: E402
from mashm_gb300 import mesh as MS  # noqa: E402
from mashm_gb300 import mesher as MR  # noqa: E402
from mashm_gb300 import workloads as W  # noqa: E402

CARRIERS = (50e3, 75e3, 100e3)


def listed():
    return [
        # the smallest call: the internal force of a small mesh inside a
        # caller's own loop on its own device memory (monitoring, MEX gateway)
        dict(name="static force 11x9 f64", kind="static", nex=11, ney=9),
        # the reference's solver as it is called by default: FP64, one plate
        # under a point force (0.5 m square, 20x20 elements, 50 kHz)
        dict(name="plate 20x20 f64", kind="plate", n=1, nex=20, ney=20, edge_mm=25.0, precision=64, steps=200, graph=0),
        # the same plate in FP32, in graph chunks: a parameter study of small plates
        dict(name="plate 20x20 f32", kind="plate", n=1, nex=20, ney=20, edge_mm=25.0, precision=32, steps=200, graph=50),
        # a large plate with a PZT disc, sensor voltage and wavefield frames
        # (1 m square, 200x200 elements, 5 M DOF)
        dict(name="pzt plate 200 f32 frames", kind="pzt", nex=200, discs=1, precision=32, steps=400, frames=100, graph=50),
        # the multi-PZT entry point: every disc bonded and sensing, all five
        # components of the velocity frames, FP64, an odd mesh size
        dict(name="pzt plate 61 f64 frames", kind="pzt", nex=61, discs=3, precision=64, steps=120, frames=40, graph=0),
        # the batched scenario sweep (training data): uneven damaged plates
        dict(name="batch 48 plates f32", kind="plate", n=48, nex=80, ney=80, edge_mm=6.25, precision=32, steps=300, graph=50),
        # a delaminated plate: split nodes, sub-laminates, so no grid numbering
        dict(name="delaminated 24x24 f64", kind="delam", nex=24, ney=24, precision=64, steps=200, graph=0),
        # a plate from the quad mesher: curvilinear numbering, distorted elements
        dict(name="quad mesh 97x71 f32", kind="quads", nex=97, ney=71, precision=32, steps=300, graph=50),
        # laminate as 3D solid elements, one per ply, delaminated interface
        dict(name="solid 64x64x8 f32", kind="solid", nex=64, precision=32, steps=150, graph=50),
        dict(name="solid 13x13x8 f64", kind="solid", nex=13, precision=64, steps=100, graph=0),
        # damage identification: misfit and per-element gradient, a batch of maps
        dict(name="gradient 16 maps f32", kind="adjoint", n=16, nex=50, mesh="grid", precision=32, steps=400, ckpt=100),
        # wavefield images of a solved plate, total displacement on the top surface
        dict(name="images 320x240x16 f32", kind="images", nex=80, ney=60, nx=320, ny=240, frames=16, motion=9, precision=32),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(("static", "plate", "plate", "pzt", "batch", "delam", "quads", "solid", "adjoint", "images"))
    prec = rng.choice((32, 64))
    graph = rng.choice((0, 50))
    if kind == "static":
        return dict(kind=kind, nex=_log(rng, 2, 60), ney=_log(rng, 2, 60))
    if kind == "plate":
        return dict(kind=kind, n=1, nex=_log(rng, 3, 70), ney=_log(rng, 3, 70), edge_mm=rng.choice((6.25, 10.0, 25.0)),
                    precision=prec, steps=rng.randint(100, 200), graph=graph)
    if kind == "pzt":
        nex = _log(rng, 24, 200 if prec == 32 else 72)
        return dict(kind=kind, nex=nex, discs=rng.choice((1, 3)), precision=prec, steps=rng.randint(80, 160),
                    frames=rng.choice((0, 40)), graph=graph)
    if kind == "batch":
        side = rng.randint(20, 80)
        return dict(kind="plate", n=rng.randint(2, 24), nex=side, ney=side, edge_mm=6.25, precision=32,
                    steps=rng.randint(100, 300), graph=50)
    if kind == "delam":
        return dict(kind=kind, nex=_log(rng, 12, 60), ney=_log(rng, 12, 60), precision=prec, steps=rng.randint(100, 200), graph=graph)
    if kind == "quads":
        hi = 90 if prec == 32 else 45
        return dict(kind=kind, nex=_log(rng, 5, hi), ney=_log(rng, 5, hi), precision=prec, steps=rng.randint(100, 300), graph=graph)
    if kind == "solid":
        return dict(kind=kind, nex=_log(rng, 6, 48 if prec == 32 else 20), precision=prec, steps=rng.randint(80, 150), graph=graph)
    if kind == "adjoint":
        mesh = rng.choice(("grid", "quads"))
        nex = _log(rng, 8, 50 if prec == 32 and mesh == "grid" else 20)
        return dict(kind=kind, n=rng.randint(1, 16 if mesh == "grid" else 2), nex=nex, mesh=mesh, precision=prec,
                    steps=rng.randint(100, 250), ckpt=rng.choice((50, 100, 200)))
    return dict(kind="images", nex=_log(rng, 12, 80), ney=_log(rng, 12, 80), nx=_log(rng, 40, 320), ny=_log(rng, 40, 300),
                frames=rng.randint(2, 16), motion=rng.randint(1, 9), precision=prec)


# ---------------------------------------------------------------------------
# inputs: the arrays that a program has in hand, from the case and the seed
# ---------------------------------------------------------------------------

@functools.lru_cache(maxsize=None)
def _dt(ax, ay, safety=0.9):
    return EL.stable_dt([EL.rect_nodes(ax, ay)], [M.cfrp_laminate()], safety)


def _damage(rng, mesh, zones):
    cen = MS.element_centres(mesh)
    lo, hi = cen.min(axis=0), cen.max(axis=0)
    keep = np.ones(cen.shape[0])
    for _ in range(zones):
        c = lo + rng.uniform(0.15, 0.85, 2) * (hi - lo)
        a = rng.uniform(0.05, 0.15, 2) * (hi - lo).max()
        t = rng.uniform(0, np.pi)
        d = cen - c
        u = (np.cos(t) * d[:, 0] + np.sin(t) * d[:, 1]) / a[0]
        v = (np.cos(t) * d[:, 1] - np.sin(t) * d[:, 0]) / a[1]
        keep[u * u + v * v <= 1.0] = 1.0 - rng.uniform(0.2, 0.8)
    return keep


def _burst(rng, dt, nft):
    f = float(rng.choice(CARRIERS))
    return rng.uniform(0.5, 2.0) * pkg.hanning_signal(dt, nft, f / 5, f, 0.0)[1]


def _circle(coords, xc, yc, r, n, phase):
    """1-based nodes nearest to n points of a circle (on any mesh)."""
    ang = phase + 2 * np.pi * np.arange(n) / n
    return np.array([MS.nearest_node(coords, xc + r * np.cos(t), yc + r * np.sin(t)) for t in ang], np.int32)


def _loaded(rng, mesh, reach, dt, nft, table, keep, n_out=8):
    """A point force at a random node, outputs on a circle that its wave reaches."""
    co = mesh["coords"]
    lo, hi = co.min(axis=0)[:2], co.max(axis=0)[:2]
    x, y = lo + rng.uniform(0.3, 0.7, 2) * (hi - lo)
    node = MS.nearest_node(co, x, y)
    outs = _circle(co, x, y, reach, n_out, rng.uniform(0, np.pi))
    return pkg.Scenario(mesh=mesh, mat_table=table, elem_keep=keep, force_dof=np.array([5 * node], np.int32),
                        force_val=np.array([1.0]), out_dof=(5 * outs).astype(np.int32), signal=_burst(rng, dt, nft))


def _jittered(rng, nex, ney, edge):
    """Quads with jittered corners through the mesher (its node numbering)."""
    X, Y = np.meshgrid(np.arange(nex + 1) * edge, np.arange(ney + 1) * edge)
    X[1:-1, 1:-1] += rng.uniform(-0.12, 0.12, X[1:-1, 1:-1].shape) * edge
    Y[1:-1, 1:-1] += rng.uniform(-0.12, 0.12, Y[1:-1, 1:-1].shape) * edge
    pos = np.stack([X.ravel(), Y.ravel(), np.zeros(X.size)], axis=1)
    c = (np.arange(ney)[:, None] * (nex + 1) + np.arange(nex)[None, :] + 1).ravel()
    quads = np.stack([c, c + 1, c + nex + 2, c + nex + 1], axis=1)
    nodes, coords, _ = MR.quad2spectral(MR.change_turn_quad(quads, pos), pos, 5)
    return dict(nodes=nodes, coords=coords, structured=False)


def _inputs(case, seed):
    """(scenarios, run parameters) of a case."""
    rng = np.random.default_rng([seed, 17])
    kind, lam = case["kind"], M.cfrp_laminate()
    table = M.table_row(lam)[None, :]
    run = dict(nn_first=2, eta_xy=W.ETA_XY, eta_z=W.ETA_Z, h=lam["h"])
    nft = case.get("steps", 1) + 1
    if kind == "plate":
        edge = case["edge_mm"] * 1e-3
        dt = _dt(edge, edge)
        scs = []
        for _ in range(case["n"]):
            lo = max(2, case["nex"] // 2)
            nex, ney = (case["nex"], case["ney"]) if case["n"] == 1 else (int(v) for v in rng.integers(lo, case["nex"] + 1, 2))
            mesh = MS.structured_plate(nex * edge, ney * edge, nex, ney)
            scs.append(_loaded(rng, mesh, 1.3 * edge, dt, nft, table, _damage(rng, mesh, int(rng.integers(1, 4)))))
        return scs, pkg.RunConfig(dt=dt, nft=nft, **run)
    if kind == "quads":
        edge = 6.25e-3
        dt = _dt(edge, edge, 0.5)
        mesh = _jittered(rng, case["nex"], case["ney"], edge)
        return [_loaded(rng, mesh, 0.7 * edge, dt, nft, table, _damage(rng, mesh, 2))], pkg.RunConfig(dt=dt, nft=nft, **run)
    if kind == "delam":
        # a square plate of nex x ney elements, the delamination near its centre
        L, few = 25e-3 * max(case["nex"], case["ney"]), min(case["nex"], case["ney"])
        zone = (*rng.uniform(0.4, 0.6, 2) * L, *rng.uniform(1.6, 3.0, 2) * L / few, rng.uniform(0, np.pi))
        scs, cfg = W.plate_delamination(nex=case["nex"], ney=case["ney"], L=L, zone=zone, layer=int(rng.integers(2, 7)),
                                        radius=32e-3, nft=nft)
        scs[0].signal = _burst(rng, cfg.dt, nft)
        return scs, cfg
    if kind == "pzt":
        if case["discs"] == 1:
            scs, cfg = W.plate_pzt(nex=case["nex"], L=case["nex"] * 5e-3, f=float(rng.choice(CARRIERS)), radius=8e-3,
                                   frames_every=case["frames"], nft=nft)
        else:
            scs, cfg = W.plate_multi_pzt(nex=case["nex"], L=case["nex"] * 5e-3, n_pzt=case["discs"],
                                         actuator_no=int(rng.integers(1, case["discs"] + 1)), nft=nft)
            cfg.frm_int, cfg.frame_dof, cfg.frame_kind = case["frames"], 0, 0
            act = np.unique((scs[0].force_dof - 1) // 5)
            x, y = scs[0].mesh["coords"][act].mean(axis=0)[:2]
            scs[0].out_dof = (5 * _circle(scs[0].mesh["coords"], x, y, 8e-3, 1, 0.3)).astype(np.int32)
        scs[0].elem_keep = _damage(rng, scs[0].mesh, 2)
        scs[0].signal = _burst(rng, cfg.dt, nft)
        return scs, cfg
    if kind == "solid":
        scs, cfg = W.solid_plate(nex=case["nex"], L=case["nex"] * 0.5 / 120, seed=int(seed), radius=5e-3, nft=nft)
        scs[0].signal = _burst(rng, cfg.dt, nft)
        return scs, cfg
    if kind == "adjoint":
        edge = 10e-3
        scs = []
        for _ in range(case["n"]):
            if case["mesh"] == "grid":
                mesh = MS.structured_plate(case["nex"] * edge, case["nex"] * edge, case["nex"], case["nex"])
            else:
                mesh = _jittered(rng, case["nex"], case["nex"], edge)
            scs.append(_loaded(rng, mesh, 0.7 * edge, 1.0, nft, table, _damage(rng, mesh, 2)))
        dt = _dt(edge, edge, 0.5 if case["mesh"] == "quads" else 0.9)
        for sc in scs:
            sc.signal = _burst(rng, dt, nft)
        return scs, pkg.RunConfig(dt=dt, nft=nft, **run)
    raise ValueError(kind)


def _target(case, seed, scs, dt):
    """Measured signals to fit: delayed bursts of the size that the plates' outputs have."""
    rng = np.random.default_rng([seed, 18])
    out = []
    for sc in scs:
        nft, n = len(sc.signal), len(sc.out_dof)
        t = np.arange(nft)[:, None] * dt
        late = rng.uniform(8e-6, 20e-6, n)[None, :]
        f = 50e3
        out.append(1e-8 * np.where(t > late, np.sin(2 * np.pi * f * (t - late)) * np.sin(np.pi * f / 5 * (t - late)) ** 2, 0.0))
    return out


def _wavefield(case, seed, coords, n):
    """Smooth five-component field number n: a few plane waves, [nnode, 5]."""
    rng = np.random.default_rng([seed, 19, n])
    U = np.zeros((coords.shape[0], 5))
    for f in range(5):
        for _ in range(2):
            k = rng.uniform(-200.0, 200.0, 2)
            U[:, f] += rng.uniform(0.2, 1.0) * 1e-6 * np.sin(coords[:, :2] @ k + rng.uniform(0, 6.0))
    return U


def _static_mesh(case, seed):
    rng = np.random.default_rng([seed, 20])
    mesh = _jittered(rng, case["nex"], case["ney"], 6.25e-3)
    nodes, nnode = mesh["nodes"], mesh["coords"].shape[0]
    fen = nodes.shape[0]
    keep = rng.uniform(0.3, 1.0, fen)
    lam = M.table_row(M.cfrp_laminate())[:21, None] * keep[None, :]
    U = rng.standard_normal(5 * nnode) * 1e-9
    # the reference's assembly maps (nodesMaps_Fiborek.m): each copy of a node,
    # in element order, to the least-filled of 12 baskets
    flat = nodes.reshape(-1).astype(np.int64)
    order = np.argsort(flat, kind="stable")
    fill = [0] * 12
    IG, IL = [[] for _ in range(12)], [[] for _ in range(12)]
    k = 0
    while k < order.size:
        g = flat[order[k]]
        m = k
        while m < order.size and flat[order[m]] == g:
            m += 1
        for b, q in zip(sorted(range(12), key=lambda b: fill[b]), range(k, m)):
            fill[b] += 1
            IG[b].append(int(g))
            IL[b].append(int(order[q]) + 1)
        k = m
    rows = max(fill)
    G, L = np.zeros((12, rows), np.int32), np.zeros((12, rows), np.int32)
    for b in range(12):
        G[b, :fill[b]], L[b, :fill[b]] = IG[b], IL[b]
    return mesh, lam, G, L, U


# ---------------------------------------------------------------------------
# what a program keeps, and one pass
# ---------------------------------------------------------------------------

def _plan(case, scs, run):
    if case["kind"] == "solid":
        return pkg.SolidPlan(scs, run, precision=case["precision"], steps_per_graph=case["graph"])
    return pkg.Plan(scs, run, precision=case["precision"], steps_per_graph=case.get("graph", 0))


def prepare(case, seed):
    kind = case["kind"]
    if kind == "static":
        mesh, lam, G, L, U = _static_mesh(case, seed)
        dev = torch.device("cuda:0")
        t = {k: torch.tensor(np.ascontiguousarray(v), device=dev) for k, v in
             dict(nodes=mesh["nodes"].T.astype(np.int32), coords=mesh["coords"].T, lam=lam, G=G, L=L, U=U).items()}
        return dict(kind=kind, t=t, F=torch.zeros_like(t["U"]), fen=mesh["nodes"].shape[0], nnode=mesh["coords"].shape[0],
                    rows=G.shape[1], lib=pkg.native.load())
    if kind == "images":
        edge = 6.25e-3
        mesh = MS.structured_plate(case["nex"] * edge, case["ney"] * edge, case["nex"], case["ney"])
        lam = M.cfrp_laminate()
        # a plan whose displacement frames 1..n are the given wavefields
        run = pkg.RunConfig(dt=_dt(edge, edge), nft=case["frames"], nn_first=1, h=1.0, frm_int=1, frame_dof=0, frame_kind=1)
        plan = pkg.Plan([pkg.Scenario(mesh=mesh, mat_table=M.table_row(lam)[None, :], signal=np.zeros(run.nft))], run,
                        precision=case["precision"])
        plan.set_signal()
        for n in range(case["frames"]):
            U = _wavefield(case, seed, mesh["coords"], n).reshape(-1)
            plan.set_state(U, U, n + 1)
            plan.advance(1)
        grid = pkg.wavefield.Grid(mesh, case["nx"], case["ny"], "top")
        return dict(kind=kind, plan=plan, grid=grid, motion=case["motion"], h=lam["h"], precision=case["precision"])
    scs, run = _inputs(case, seed)
    state = dict(kind=kind, plan=_plan(case, scs, run), precision=case["precision"])
    if kind == "adjoint":
        state["target"], state["ckpt"] = _target(case, seed, scs, run.dt), case["ckpt"]
    else:
        state["frames"] = run.frm_int > 0
    return state


def run(state):
    if state["kind"] == "static":
        t = state["t"]
        code = state["lib"].shm_stiffness_static(
            state["fen"], state["nnode"], t["nodes"].data_ptr(), t["coords"].data_ptr(), t["lam"].data_ptr(), state["rows"],
            t["G"].data_ptr(), t["L"].data_ptr(), t["U"].data_ptr(), state["F"].data_ptr(),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if code != 0:
            raise RuntimeError("shm_stiffness_static: status %d" % code)
        return state["F"]
    as_kept = (lambda a: a.astype(np.float32)) if state["precision"] == 32 else (lambda a: a)
    if state["kind"] == "images":
        return as_kept(state["grid"].from_plan(state["plan"], state["motion"], state["h"], "displacement"))
    if state["kind"] == "adjoint":
        misfit, grad = state["plan"].forward_backward(state["target"], ckpt_every=state["ckpt"])
        return dict(misfit=as_kept(misfit), grad=as_kept(np.concatenate(grad)))
    res = state["plan"].forward(want_frames=state["frames"])
    out = dict(displ=as_kept(res[0]["displ"] if len(res) == 1 else np.concatenate([r["displ"] for r in res], axis=1)))
    if res[0]["voltage"].size:
        out["voltage"] = as_kept(res[0]["voltage"])
    if state["frames"]:
        out["frames"] = as_kept(res[0]["frames"])
    return out


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------

def work(case):
    kind = case["kind"]
    word = case.get("precision", 64) // 8
    if kind == "static":
        fen = case["nex"] * case["ney"]
        nnode = (5 * case["nex"] + 1) * (5 * case["ney"] + 1)
        # U in, F out, connectivity, coordinates, laminate, maps
        return dict(bytes=nnode * (2 * 5 + 2) * 8.0 + fen * (36 * 4 + 21 * 8) + 2 * 36 * fen * 4.0, flops=fen * 16e3)
    if kind == "images":
        pts = case["nx"] * case["ny"]
        nnode = (5 * case["nex"] + 1) * (5 * case["ney"] + 1)
        fields = {1: 1, 2: 1, 3: 1, 4: 1, 5: 1, 6: 2, 7: 2, 8: 4, 9: 5}[case["motion"]]
        # the frames' fields in, the images out (FP64 by the interface)
        return dict(bytes=case["frames"] * (nnode * fields * word + pts * 8.0), flops=case["frames"] * pts * 36 * 2.0 * (1 + fields / 6))
    if kind == "solid":
        nodes = (5 * case["nex"] + 1) ** 2 * 17
        fen, fields, ops = 8 * case["nex"] ** 2, 3, 28e3
    else:
        ney = case.get("ney", case["nex"])
        n = case.get("n", 1)
        share = 1.0 if n == 1 or kind == "adjoint" else 0.75 ** 2   # sides spread over the upper half of the range
        nodes = n * share * (5 * case["nex"] + 1) * (5 * ney + 1)
        fen, fields, ops = n * share * case["nex"] * ney, 5, 12.8e3
    steps = case["steps"]
    # per DOF and step: u_n and u_{n-1} in, u_{n+1} out, the inverse mass in;
    # the gradient's second sweep reads the forward state as well
    passes = 1 if kind != "adjoint" else 2
    per = 4 * passes + (1 if kind == "adjoint" else 0)
    frames = steps // case["frames"] if case.get("frames") else 0
    kept = frames * nodes * (1 if case.get("discs") == 1 else 5) * 8.0
    return dict(bytes=float(steps) * nodes * fields * per * word + kept, flops=float(steps) * fen * ops * passes)


# ---------------------------------------------------------------------------
# the same in 64 bits, plainly
# ---------------------------------------------------------------------------

def _gll(n):
    P = np.polynomial.legendre.Legendre.basis(n - 1)
    x = np.concatenate(([-1.0], np.sort(P.deriv().roots().real), [1.0]))
    for _ in range(3):  # polish the interior roots
        x[1:-1] -= P.deriv()(x[1:-1]) / P.deriv(2)(x[1:-1])
    w = 2.0 / (n * (n - 1) * P(x) ** 2)
    D = np.zeros((n, n))
    for c in range(n):
        others = [m for m in range(n) if m != c]
        den = np.prod([x[c] - x[m] for m in others])
        for r in range(n):
            D[r, c] = sum(np.prod([x[r] - x[m] for m in others if m != q]) for q in others) / den
    D[np.abs(D) < 1e-12] = 0.0
    return x, w, D


def _dev():
    return torch.device("cuda:0" if torch.cuda.is_available() else "cpu")


def _t(a, dtype=torch.float64):
    return torch.tensor(np.ascontiguousarray(a), dtype=dtype, device=_dev())


class _Shell:
    """Flat-shell operator of a list of scenarios, numbered one after another."""

    def __init__(self, scs):
        _, w, D = _gll(6)
        self.D = _t(D)
        nodes, X, Y, C, keep, m11, I11, n0 = [], [], [], [], [], [], [], 0
        for sc in scs:
            el = np.asarray(sc.mesh["nodes"], np.int64) - 1
            co = np.asarray(sc.mesh["coords"], float)
            em = np.zeros(len(el), int) if sc.elem_mat is None else np.asarray(sc.elem_mat)
            tab = np.atleast_2d(sc.mat_table)
            Cm = np.zeros((len(tab), 8, 8))
            for q, r in enumerate(tab):
                A, B, Dm = (np.array([[v[0], v[1], v[2]], [v[1], v[3], v[4]], [v[2], v[4], v[5]]]) for v in (r[0:6], r[9:15], r[15:21]))
                Cm[q, :3, :3], Cm[q, :3, 3:6], Cm[q, 3:6, :3], Cm[q, 3:6, 3:6] = A, B, B, Dm
                Cm[q, 6:, 6:] = [[r[6], r[7]], [r[7], r[8]]]
            nodes.append(el + n0)
            X.append(co[el, 0])
            Y.append(co[el, 1])
            C.append(Cm[em])
            keep.append(np.ones(len(el)) if sc.elem_keep is None else sc.elem_keep)
            m11.append(tab[em, 21])
            I11.append(tab[em, 22])
            n0 += co.shape[0]
        self.nnode = n0
        self.nodes = _t(np.concatenate(nodes), torch.int64)
        self.fen = self.nodes.shape[0]
        X, Y = (_t(np.concatenate(v)).reshape(-1, 6, 6) for v in (X, Y))   # [e, eta k, xi i]
        J11, J21 = torch.einsum("ip,ekp->eki", self.D, X), torch.einsum("ip,ekp->eki", self.D, Y)
        J12, J22 = torch.einsum("kq,eqi->eki", self.D, X), torch.einsum("kq,eqi->eki", self.D, Y)
        det = J11 * J22 - J12 * J21
        self.i11, self.i12, self.i21, self.i22 = (v[..., None] for v in (J22 / det, -J12 / det, -J21 / det, J11 / det))
        self.Wt = (det * _t(np.outer(w, w)))[..., None]
        self.C = _t(np.concatenate(C))
        self.keep = _t(np.concatenate(keep))
        M_ = torch.zeros(n0, 2, dtype=torch.float64, device=_dev())
        mm = torch.stack([_t(np.concatenate(m11)), _t(np.concatenate(I11))], -1)
        M_.index_add_(0, self.nodes.reshape(-1), (self.Wt * mm[:, None, None, :]).reshape(-1, 2))
        self.minv = (1.0 / M_)[:, [0, 1, 0, 1, 0]]

    def parts(self, U):
        """Reference derivatives of the element values [e, 6, 6, 5] and the values."""
        ue = U[self.nodes].reshape(-1, 6, 6, 5)
        return ue, torch.einsum("ip,ekpf->ekif", self.D, ue), torch.einsum("kq,eqif->ekif", self.D, ue)

    def local(self, U):
        """K_e^0 u_e of every element, [e, 36, 5]."""
        ue, dx, de = self.parts(U)
        gx, gy = dx * self.i11 + de * self.i21, dx * self.i12 + de * self.i22
        s = torch.stack([gx[..., 0], gy[..., 2], gy[..., 0] + gx[..., 2], gx[..., 1], gy[..., 3], gy[..., 1] + gx[..., 3],
                         ue[..., 3] + gy[..., 4], ue[..., 1] + gx[..., 4]], -1)
        R = torch.einsum("eab,ekib->ekia", self.C, s) * self.Wt
        Sx, Sy = R[..., [0, 3, 2, 5, 7]], R[..., [2, 5, 1, 4, 6]]
        F = torch.einsum("ip,ekif->ekpf", self.D, Sx * self.i11 + Sy * self.i12)
        F += torch.einsum("kq,ekif->eqif", self.D, Sx * self.i21 + Sy * self.i22)
        F[..., 1] += R[..., 7]
        F[..., 3] += R[..., 6]
        return F.reshape(-1, 36, 5)

    def assemble(self, Fe):
        return torch.zeros(self.nnode, 5, dtype=torch.float64, device=_dev()).index_add_(0, self.nodes.reshape(-1), Fe.reshape(-1, 5))

    def force(self, U):
        return self.assemble(self.local(U) * self.keep[:, None, None])


class _Solid:
    """3D solid operator (6 x 6 x 3 nodes, box elements)."""

    def __init__(self, sc):
        x6, w6, D6 = _gll(6)
        _, w3, D3 = _gll(3)
        self.D6, self.D3 = _t(D6), _t(D3)
        el, co = np.asarray(sc.mesh["nodes"], np.int64) - 1, np.asarray(sc.mesh["coords"], float)
        self.nnode, self.nodes = co.shape[0], _t(el, torch.int64)
        P = co[el].reshape(-1, 3, 6, 6, 3)                                    # [e, z, y, x, component]
        size = np.stack([P[:, 0, 0, -1, 0] - P[:, 0, 0, 0, 0], P[:, 0, -1, 0, 1] - P[:, 0, 0, 0, 1], P[:, -1, 0, 0, 2] - P[:, 0, 0, 0, 2]], -1)
        self.s = _t(2.0 / size)[:, :, None, None, None]
        self.Wt = _t(np.einsum("z,y,x->zyx", w3, w6, w6))[None] * _t(np.prod(size / 2, axis=1))[:, None, None, None]
        d = np.asarray(sc.mat_table)[np.asarray(sc.elem_mat)]
        C = np.zeros((len(el), 6, 6))
        for q, (a, b) in enumerate([(0, 0), (0, 1), (0, 2), (0, 3), (1, 1), (1, 2), (1, 3), (2, 2), (2, 3), (3, 3), (4, 4), (4, 5), (5, 5)]):
            C[:, a, b] = C[:, b, a] = d[:, q]
        self.C = _t(C)
        Mn = torch.zeros(self.nnode, dtype=torch.float64, device=_dev())
        Mn.index_add_(0, self.nodes.reshape(-1), (self.Wt * _t(d[:, 13])[:, None, None, None]).reshape(-1))
        self.minv = (1.0 / Mn)[:, None].expand(-1, 3)

    def force(self, U):
        u = U[self.nodes].reshape(-1, 3, 6, 6, 3)
        gx = torch.einsum("ip,ezypf->ezyif", self.D6, u) * self.s[:, 0:1]
        gy = torch.einsum("iq,ezqxf->ezixf", self.D6, u) * self.s[:, 1:2]
        gz = torch.einsum("ir,eryxf->eiyxf", self.D3, u) * self.s[:, 2:3]
        E = torch.stack([gx[..., 0], gy[..., 1], gz[..., 2], gy[..., 0] + gx[..., 1], gz[..., 1] + gy[..., 2], gz[..., 0] + gx[..., 2]], -1)
        S = torch.einsum("eab,ezyxb->ezyxa", self.C, E) * self.Wt[..., None]
        F = torch.einsum("ip,ezyif->ezypf", self.D6, S[..., [0, 3, 5]] * self.s[:, 0:1])
        F += torch.einsum("iq,ezixf->ezqxf", self.D6, S[..., [3, 1, 4]] * self.s[:, 1:2])
        F += torch.einsum("ir,eiyxf->eryxf", self.D3, S[..., [5, 4, 2]] * self.s[:, 2:3])
        return torch.zeros(self.nnode, 3, dtype=torch.float64, device=_dev()).index_add_(0, self.nodes.reshape(-1), F.reshape(-1, 3))


class _March:
    """The central-difference loop's coefficients, forces and outputs."""

    def __init__(self, scs, run, nf):
        a0, a1 = 1 / run.dt ** 2, 1 / (2 * run.dt)
        eta = np.array([run.eta_xy, 0, run.eta_xy, 0, run.eta_z] if nf == 5 else [run.eta_xy, run.eta_xy, run.eta_z])
        self.a1, self.k1, self.k2 = a1, _t((a0 - a1 * eta) / (a0 + a1 * eta)), _t(1 / (a0 + a1 * eta))
        n0, fd, fv, fs, od = 0, [], [], [], []
        for k, sc in enumerate(scs):
            fd.append(np.asarray(sc.force_dof, np.int64) - 1 + nf * n0)
            fv.append(np.asarray(sc.force_val, float))
            fs.append(np.full(len(fd[-1]), k))
            od.append(np.asarray(sc.out_dof, np.int64) - 1 + nf * n0)
            n0 += np.asarray(sc.mesh["coords"]).shape[0]
        self.fd, self.fv, self.od = _t(np.concatenate(fd), torch.int64), _t(np.concatenate(fv)), _t(np.concatenate(od), torch.int64)
        self.st = _t(np.stack([sc.signal for sc in scs])[np.concatenate(fs)])          # [nforce, nft]
        self.shape = (n0, nf)

    def zeros(self):
        return torch.zeros(self.shape, dtype=torch.float64, device=_dev())

    def step(self, op, U, Uo, nn):
        F = -op.force(U)
        F.view(-1).index_add_(0, self.fd, self.fv * self.st[:, nn - 1])
        return U + self.k1 * (U - Uo) + self.k2 * op.minv * F


def _exact_forward(case, scs, run):
    solid = case["kind"] == "solid"
    op = _Solid(scs[0]) if solid else _Shell(scs)
    m = _March(scs, run, 3 if solid else 5)
    U, Uo = m.zeros(), m.zeros()
    displ = torch.zeros(run.nft, len(m.od), dtype=torch.float64, device=_dev())
    sens = scs[0].sensors if not solid else []
    volt, frames = torch.zeros(run.nft, len(sens), dtype=torch.float64, device=_dev()), []
    for nn in range(run.nn_first, run.nft + 1):
        displ[nn - 1] = U.reshape(-1)[m.od]
        if sens:
            # the sensor formula as the solver has it: invJ12 beside the
            # eta-derivative, invJ21 beside the xi-derivative
            _, dx, de = op.parts(U)
            p = scs[0].pzt
            sx, sy = dx * op.i11 + de * op.i12, dx * op.i21 + de * op.i22
            v = p["e31"] * (sx[..., 0] + run.h / 2 * sx[..., 1]) + p["e32"] * (sy[..., 2] + run.h / 2 * sy[..., 3])
            for k, els in enumerate(sens):
                volt[nn - 1, k] = (p["pzt_thickness"] / p["g33"] * v[torch.as_tensor(np.asarray(els, np.int64), device=_dev())]).mean()
        Un = m.step(op, U, Uo, nn)
        if run.frm_int and nn % run.frm_int == 0:
            vel = m.a1 * (Un - Uo)
            frames.append((vel if run.frame_dof == 0 else vel[:, run.frame_dof - 1:run.frame_dof]).T.clone())
        U, Uo = Un, U
    out = dict(displ=displ.cpu().numpy())
    if sens:
        out["voltage"] = volt.cpu().numpy()
    if run.frm_int:
        out["frames"] = torch.stack(frames).cpu().numpy()
    return out


def _exact_gradient(case, scs, run, target):
    op, m = _Shell(scs), _March(scs, run, 5)
    n0, N = run.nn_first, run.nft
    U, Uo, states = m.zeros(), m.zeros(), {}
    for nn in range(n0, N + 1):
        states[nn] = U
        U, Uo = m.step(op, U, Uo, nn), U
    tgt = _t(np.concatenate(target, axis=1))
    res = torch.zeros(N + 1, len(m.od), dtype=torch.float64, device=_dev())
    for nn in range(n0, N + 1):
        res[nn] = states[nn].reshape(-1)[m.od] - tgt[nn - 1]
    per = 0.5 * (res ** 2).sum(0)
    cuts = np.cumsum([0] + [len(sc.out_dof) for sc in scs])
    misfit = np.array([float(per[a:b].sum()) for a, b in zip(cuts[:-1], cuts[1:])])
    # reverse time: a_n = dJ/du_n of u_{n+1} = u_n + k1 (u_n - u_{n-1}) - k2 M^-1 (K u_n - f_n)
    a1, a2 = m.zeros(), m.zeros()
    grad = torch.zeros(op.fen, dtype=torch.float64, device=_dev())
    for nn in range(N, n0 - 1, -1):
        b = m.k2 * op.minv * a1
        grad += (b[op.nodes] * op.local(states[nn])).sum((1, 2))        # dJ/dd_e, d_e = 1 - keep_e
        a0 = (1 + m.k1) * a1 - m.k1 * a2 - op.force(b)
        a0.view(-1).index_add_(0, m.od, res[nn])
        a1, a2 = a0, a1
    return dict(misfit=misfit, grad=grad.cpu().numpy())


def _exact_images(case, seed):
    edge, h = 6.25e-3, M.cfrp_laminate()["h"]
    mesh = MS.structured_plate(case["nex"] * edge, case["ney"] * edge, case["nex"], case["ney"])
    x, _, _ = _gll(6)
    eps = 1e-8

    def along(n_el, n_pts):
        """Owner, Lagrange weights of the points along one axis: [n_pts], [n_pts, 6]."""
        L = n_el * edge
        p = eps + np.arange(n_pts) * (L - 2 * eps) / (n_pts - 1)
        own = np.minimum((p / edge).astype(int), n_el - 1)
        t = 2 * (p - own * edge) / edge - 1
        w = np.ones((n_pts, 6))
        for i in range(6):
            for q in range(6):
                if q != i:
                    w[:, i] *= (t - x[q]) / (x[i] - x[q])
        return own, w

    ox, wx = along(case["nex"], case["nx"])
    oy, wy = along(case["ney"], case["ny"])
    ix = torch.as_tensor(5 * ox[:, None] + np.arange(6), device=_dev())
    iy = torch.as_tensor(5 * oy[:, None] + np.arange(6), device=_dev())
    out = []
    for n in range(case["frames"]):
        u, fx, v, fy, w = (_t(_wavefield(case, seed, mesh["coords"], n)).reshape(mesh["NY"], mesh["NX"], 5)[..., f] for f in range(5))
        a, b = u + h / 2 * fx, v + h / 2 * fy
        val = {1: u, 2: v, 3: w, 4: fx, 5: fy, 6: a, 7: b, 8: (a * a + b * b).sqrt(), 9: (a * a + b * b + w * w).sqrt()}[case["motion"]]
        rows = (val[iy] * _t(wy)[:, :, None]).sum(1)                     # [ny, NX]
        out.append((rows[:, ix] * _t(wx)[None]).sum(-1))
    return torch.stack(out).cpu().numpy()


def exact(case, seed):
    if case["kind"] == "static":
        mesh, lam, _, _, U = _static_mesh(case, seed)
        fen = mesh["nodes"].shape[0]
        table = np.zeros((fen, 23))
        table[:, :21], table[:, 21:] = lam.T, 1.0
        op = _Shell([pkg.Scenario(mesh=mesh, mat_table=table, elem_mat=np.arange(fen))])
        return op.force(_t(U).reshape(-1, 5)).reshape(-1).cpu().numpy()
    if case["kind"] == "images":
        return _exact_images(case, seed)
    scs, run = _inputs(case, seed)
    if case["kind"] == "adjoint":
        return _exact_gradient(case, scs, run, _target(case, seed, scs, run.dt))
    return _exact_forward(case, scs, run)
