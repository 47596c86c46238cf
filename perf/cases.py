"""Performance cases: the calls a program makes into libpump, over their sizes.

Two listed cases are whole planning queries; the others are the stages such a
query is made of, each through its own entry point (include/pump.h), at the
sizes of the repository's configurations (``pump_gb300.workloads``) and
benchmark.  A case's ``kind`` names the entry point:

- ``plan``: pump_plan, host problem in, host path out.
- ``roadmap``: pump_roadmap, all pair costs, rn and the edges (precision).
- ``pairs``: pump_bvp_pairs, the pair matrix in one of the three arithmetics.
- ``waypoints``: pump_discretize_edges.
- ``edges``: pump_free_edges.
- ``halfspaces``: pump_cache_halfspaces, the dense cache of the reference.
- ``hsmc``: pump_hsmc_propagate_boxes, one wavefront.
- ``mc_cp``: pump_mc_cp, the full Monte Carlo CP of dense paths.
- ``refine``: pump_refine_bwd, objective and adjoint of node paths.
- ``path_cp``: pump_path_cp, candidate paths judged from host nodes.
"""
import ctypes as C
import math

import numpy as np
import torch

from pump_gb300 import lib, workloads

T_ROWS, DT = 400, 0.05
G = float(np.float32(-9.81))
TABLE_SEED = 0x9E3779B97F4A7C15


def listed():
    return [
        # whole queries: the reference's own size with the defaults (10 boxes,
        # bit-exact arithmetic, 128 particles), and the headline query (indoor
        # map, 4000 samples, 1024 particles)
        dict(name="plan_1000_parity", kind="plan", N=1000, mode=0, disc=9, particles=128, boxes=10,
             indoor=False, om=1e-3),
        dict(name="plan_4000_precision", kind="plan", N=4000, mode=1, disc=8, particles=1024, boxes=40,
             indoor=True, om=2e-3),
        # offline roadmap construction of that query
        dict(name="roadmap_4000", kind="roadmap", N=4000),
        # the pair matrix in the two bit-exact arithmetics, at the two sample
        # counts the repository has fixtures for
        dict(name="pairs_4000_parity", kind="pairs", N=4000, mode=0),
        dict(name="pairs_1000_parity_gpu", kind="pairs", N=1000, mode=2),
        # edge waypoints of the headline roadmap, as the reference computes them
        dict(name="waypoints_4000_parity", kind="waypoints", N=4000, mode=0, disc=8),
        # the eager collision check of every roadmap edge against the indoor map
        dict(name="edges_4000", kind="edges", N=4000, disc=8, boxes=40, indoor=True),
        # the reference's half-space cache for a 1000-sample roadmap
        dict(name="halfspaces_1000", kind="halfspaces", N=1000, disc=9, boxes=40, indoor=True, om=0.3),
        # one mid-search wavefront: 12,000 expansions, 1024 particles, noise
        # of the reference's example input
        dict(name="hsmc_12000", kind="hsmc", N=2000, disc=8, boxes=40, indoor=True, om=0.3, paths=12000,
             particles=1024),
        # re-judging 64 dense paths with 2048 particles
        dict(name="mc_cp_64", kind="mc_cp", paths=64, particles=2048, boxes=40, om=0.1),
        # gradient of the refinement objective over 1024 returned paths
        dict(name="refine_1024", kind="refine", paths=1024, W=8, om=2e-3),
        # the smallest call: a handful of candidate paths judged from the host
        dict(name="path_cp_8", kind="path_cp", paths=8, mode=0, particles=2048, boxes=10, om=0.1),
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["plan", "roadmap", "pairs", "waypoints", "edges", "halfspaces", "hsmc", "mc_cp",
                       "refine", "path_cp"])
    om = math.exp(rng.uniform(math.log(1e-3), math.log(0.3)))
    boxes = logint(5, 100)
    indoor = rng.random() < 0.5
    if indoor:
        boxes = 40
    disc = rng.randint(4, 16)
    if kind == "plan":
        return dict(kind=kind, N=logint(300, 4000), mode=rng.choice([0, 1]), disc=rng.randint(5, 10),
                    particles=rng.choice([128, 500, 1024]), boxes=boxes, indoor=indoor,
                    om=rng.choice([1e-3, 2e-3]))
    if kind == "roadmap":
        return dict(kind=kind, N=logint(300, 4000))
    if kind == "pairs":
        mode = rng.choice([0, 1, 2])
        return dict(kind=kind, N=logint(100, 2500 if mode == 2 else 4000), mode=mode)
    if kind == "waypoints":
        return dict(kind=kind, N=logint(300, 3000), mode=rng.choice([0, 1]), disc=disc)
    if kind == "edges":
        return dict(kind=kind, N=logint(300, 3000), disc=disc, boxes=boxes, indoor=indoor)
    if kind == "halfspaces":
        return dict(kind=kind, N=logint(300, 2500), disc=disc, boxes=boxes, indoor=indoor, om=om)
    if kind == "hsmc":
        return dict(kind=kind, N=logint(300, 2000), disc=disc, boxes=boxes, indoor=indoor, om=om,
                    paths=logint(100, 12000), particles=rng.choice([128, 500, 1000, 1024, 2048]))
    if kind == "mc_cp":
        return dict(kind=kind, paths=logint(1, 100), particles=rng.choice([1000, 2048]), boxes=max(boxes, 10),
                    om=rng.uniform(0.05, 0.3))
    if kind == "refine":
        return dict(kind=kind, paths=logint(4, 1024), W=rng.randint(4, 10), om=om)
    return dict(kind=kind, paths=logint(1, 64), mode=rng.choice([0, 1]), particles=2048, boxes=max(boxes, 10),
                om=rng.uniform(0.05, 0.3))


# ------------------------------------------------------------------ inputs
def _ptr(t):
    return t.data_ptr()


def _stream():
    return torch.cuda.current_stream().cuda_stream


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _empty(n, dtype):
    return torch.empty(int(n), dtype=dtype, device="cuda")


def _map(case, seed):
    """The case's boxes (n x 12 float32)."""
    if case.get("indoor"):
        return workloads.indoor(1000 + seed % 100000, boxes=case["boxes"] - 30)
    return workloads.random_boxes(case["boxes"], seed % 1000000)


def _samples(N, seed):
    """Uniform samples of the state box, init first and goal last."""
    g = np.random.Generator(np.random.PCG64(seed))
    lo, hi = np.asarray(workloads.LO), np.asarray(workloads.HI)
    s = (lo + (hi - lo) * g.random((N, 6))).astype(np.float32)
    s[0], s[-1] = workloads.INIT, workloads.GOAL
    return s


def _coefs(x0, x1):
    """Coefficients of c(t) = A0/t^3 + A1/t^2 + A2/t + A3 + A4 t."""
    D = x1[..., :3] - x0[..., :3]
    v0, v1 = x0[..., 3:], x1[..., 3:]
    A0 = 12 * (D * D).sum(-1)
    A1 = -12 * (D * (v0 + v1)).sum(-1)
    A2 = 4 * (v0 * v0 + v0 * v1 + v1 * v1).sum(-1)
    A3 = 2 * G * (v0[..., 2] - v1[..., 2])
    return A0, A1, A2, A3, 1 + G * G


def _cost(A, t):
    r = 1 / t
    return ((A[0] * r + A[1]) * r + A[2]) * r + A[3] + A[4] * t


def _roadmap_edges(s):
    """The 5 % cheapest ordered pairs of the samples: (src, dst, time), by source."""
    N = s.shape[0]
    k = int(N * (N - 1) * 0.05)
    costs, times = _empty(N * N, torch.float32).view(N, N), _empty(N * N, torch.float32).view(N, N)
    grid = np.geomspace(0.05, 5.0, 40)
    for r0 in range(0, N, 1000):
        A = _coefs(s[r0:r0 + 1000, None, :], s[None, :, :])
        best = torch.full_like(A[0], float("inf"))
        bt = torch.full_like(A[0], 1.0)
        for t in grid:
            c = _cost(A, float(t))
            bt = torch.where(c < best, float(t), bt)
            best = torch.minimum(best, c)
        for _ in range(3):
            q = ((A[4] * bt * bt - A[2]) * bt - 2 * A[1]) * bt - 3 * A[0]
            dq = (4 * A[4] * bt * bt - 2 * A[2]) * bt - 2 * A[1]
            n = bt - q / dq
            bt = torch.where((n > 0.8 * bt) & (n < 1.25 * bt) & (n <= 5.0), n, bt)
        costs[r0:r0 + 1000], times[r0:r0 + 1000] = _cost(A, bt), bt
    costs.fill_diagonal_(float("inf"))
    rn = torch.sort(costs.view(-1)).values[k]
    at = torch.nonzero(costs < rn)
    src, dst = at[:, 0].to(torch.int32).contiguous(), at[:, 1].to(torch.int32).contiguous()
    return src, dst, times[at[:, 0], at[:, 1]].contiguous()


def _cubic(x0, x1, tau, sv):
    """States of the edge cubic at fractions sv (broadcast over the last axis but one)."""
    p0, v0, p1, v1 = x0[..., :3], x0[..., 3:], x1[..., :3], x1[..., 3:]
    s2, s3 = sv * sv, sv * sv * sv
    p = (2 * s3 - 3 * s2 + 1) * p0 + (3 * s2 - 2 * s3) * p1 + \
        tau * ((s3 - 2 * s2 + sv) * v0 + (s3 - s2) * v1)
    v = (6 * s2 - 6 * sv) * (p0 - p1) / tau + (3 * s2 - 4 * sv + 1) * v0 + (3 * s2 - 2 * sv) * v1
    return torch.cat([p, v], -1)


def _waypoints(s, src, dst, tau, disc):
    x0, x1 = s[src.long()], s[dst.long()]
    w = _empty(src.numel() * (disc + 1) * 6, s.dtype).view(-1, disc + 1, 6)
    for i in range(disc + 1):
        w[:, i] = _cubic(x0, x1, tau[:, None], i / disc)
    w[:, 0], w[:, disc] = x0, x1
    return w


def _table(particles):
    t = _empty(T_ROWS * particles * 3, torch.float32)
    lib.check(lib.load().pump_particle_tables(TABLE_SEED, particles, T_ROWS, _ptr(t), None, _stream()))
    return t


def _node_paths(n, seed, boxes):
    """Candidate paths of one query, as smoothing makes them: node sequences
    near one base path from init to goal, and boxes around the base path that
    leave it a little room.  Returns (nodes, offsets, counts, boxes)."""
    g = np.random.Generator(np.random.PCG64(seed))
    m = 9
    u = np.linspace(0, 1, m)[:, None]
    a, b = np.asarray(workloads.INIT[:3]), np.asarray(workloads.GOAL[:3])
    base = a * (1 - u) + b * u + 0.15 * np.sin(np.pi * u) * g.normal(size=3)
    vel = np.gradient(base, axis=0) * 1.5
    vel[0] = vel[-1] = 0
    fine = np.stack([np.interp(np.linspace(0, 1, 200), u[:, 0], base[:, d]) for d in range(3)], 1)
    obs = []
    while len(obs) < boxes:
        h = g.uniform(0.05, 0.2, 3) / 2
        c = fine[int(g.integers(200))] + g.normal(0, 0.15, 3)
        gap = np.abs(fine - c) - h
        if np.any(np.all(gap < 0.015, axis=1)):
            continue
        obs.append(workloads._box(c - h, c + h))
    obs = np.asarray(obs, np.float32).reshape(-1, 12)
    nodes, offs, cnts = [], [], []
    for k in range(n):
        keep = np.sort(g.choice(np.arange(1, m - 1), size=int(g.integers(3, m - 1)), replace=False))
        keep = np.concatenate([[0], keep, [m - 1]])
        x = np.concatenate([base[keep], vel[keep]], 1)
        x[1:-1] += g.normal(0, 0.01, x[1:-1].shape)
        offs.append(sum(cnts))
        cnts.append(len(keep))
        nodes.append(x.astype(np.float32))
    return np.concatenate(nodes), np.asarray(offs, np.int32), np.asarray(cnts, np.int32), obs


def _dense(nodes, offs, cnts):
    """Dense states at dt = 0.05 of node paths, 0.6 to 1 s a segment."""
    rows, off, ln = [], [], []
    for o, n in zip(offs, cnts):
        x = nodes[o:o + n].astype(np.float64)
        path = []
        for i in range(n - 1):
            tau = 0.6 + 0.4 * float(np.linalg.norm(x[i + 1, :3] - x[i, :3]))
            sv = np.arange(0, tau, DT)[:, None] / tau
            path.append(_cubic(torch.from_numpy(x[i]), torch.from_numpy(x[i + 1]), tau,
                               torch.from_numpy(sv)).numpy())
        path = np.concatenate(path)
        off.append(sum(ln))
        ln.append(len(path))
        rows.append(path.astype(np.float32))
    return np.concatenate(rows), np.asarray(off, np.int32), np.asarray(ln, np.int32)


_ctx = []


def _context():
    """The process's library context (a program keeps one per thread)."""
    if not _ctx:
        _ctx.append(lib.Context(0))
    return _ctx[0]


def prepare(case, seed):
    kind = case["kind"]
    s = dict(kind=kind, case=case)
    if kind == "plan":
        obs = _map(case, seed)
        pb, res = lib.Problem(), lib.PlanResult()
        lib.load().pump_problem_defaults(C.byref(pb))
        pb.N, pb.num_disc, pb.num_hsmc, pb.bvp_mode = case["N"], case["disc"], case["particles"], case["mode"]
        pb.num_obstacles, pb.obstacles = obs.shape[0], obs.ctypes.data
        for k in range(6):
            pb.init[k], pb.goal[k] = workloads.INIT[k], workloads.GOAL[k]
            pb.lo[k], pb.hi[k] = workloads.LO[k], workloads.HI[k]
        pb.offset_mult, pb.cp_target, pb.cp_factor = case["om"], 0.01, 2.0
        path, nodes = np.zeros((400, 6), np.float32), np.zeros(400, np.int32)
        res.path, res.path_cap, res.nodes, res.nodes_cap = path.ctypes.data, 400, nodes.ctypes.data, 400
        s.update(ctx=_context(), pb=pb, res=res, path=path, nodes=nodes, obs=obs)
        return s
    if kind in ("roadmap", "pairs"):
        N = case["N"]
        n = N * (N - 1)
        s.update(samples=_dev(_samples(N, seed)), copts=_empty(n, torch.float32), topts=_empty(n, torch.float32))
        if kind == "roadmap":
            k = int(np.float32(n) * np.float32(0.05))
            s.update(ctx=_context(), k=k, src=_empty(k, torch.int32), dst=_empty(k, torch.int32),
                     ce=_empty(k, torch.float32), te=_empty(k, torch.float32), go=_empty(N + 1, torch.int32))
        return s
    if kind in ("waypoints", "edges", "halfspaces", "hsmc"):
        x = _dev(_samples(case["N"], seed))
        src, dst, tau = _roadmap_edges(x)
        E, W = src.numel(), case["disc"] + 1
        s.update(samples=x, src=src, dst=dst, tau=tau, E=E, W=W)
        if kind == "waypoints":
            s.update(out=_empty(E * W * 6, torch.float32))
            return s
        s.update(disc=_waypoints(x, src, dst, tau, W - 1), obs=_dev(_map(case, seed)))
        if kind == "edges":
            s.update(out=_empty(E, torch.uint8))
            return s
        s.update(H=min(case["boxes"], 5), maxd2=float(np.float32(0.1 * case["om"] ** 2)))
        g = np.random.Generator(np.random.PCG64(seed + 1))
        if kind == "halfspaces":
            s.update(free=_dev((g.random(E) < 0.8).astype(np.uint8)), a=_empty(E * W * s["H"] * 3, torch.float32),
                     b=_empty(E * W * s["H"], torch.float32), n=_empty(E * W, torch.int32))
            return s
        M, P = case["paths"], case["particles"]
        words, base, pmc = (P + 31) // 32, 1 + M // 4, 2048
        live = g.random((base, P)) < g.choice([0.9, 0.97, 1.0], (base, 1))
        bits = np.zeros((base, words * 32), np.uint8)
        bits[:, :P] = live
        valid = np.zeros((base + M, words), np.uint32)
        valid[:base] = np.packbits(bits, axis=1, bitorder="little").view(np.uint32)
        s.update(edge=_dev(g.integers(0, E, M).astype(np.int32)), prev=_dev(g.integers(0, base, M).astype(np.int32)),
                 valid=_dev(valid.view(np.int32)), times=_dev((6 * g.random(base)).astype(np.float32)),
                 cp=torch.zeros(base + M, dtype=torch.float32, device="cuda"), base=base, table=_table(pmc),
                 pmc=pmc, err=torch.zeros(1, dtype=torch.int32, device="cuda"))
        return s
    if kind in ("mc_cp", "path_cp"):
        nodes, offs, cnts, obs = _node_paths(case["paths"], seed, case["boxes"])
        s.update(table=_table(case["particles"]), obs=_dev(obs))
        n = case["paths"]
        if kind == "path_cp":
            s.update(ctx=_context(), nodes=nodes, offs=offs, cnts=cnts, cp=np.zeros(n, np.float32),
                     cost=np.zeros(n, np.float32), len=np.zeros(n, np.int32))
            return s
        rows, off, ln = _dense(nodes, offs, cnts)
        s.update(rows=_dev(rows), off=_dev(off), len=_dev(ln), hits=_empty(n, torch.int32),
                 cp=_empty(n, torch.float32), err=torch.zeros(1, dtype=torch.int32, device="cuda"))
        return s
    # refine: paths of 8 to 40 nodes, the gradient's buffer sized for 40
    obs = workloads.indoor(1000 + seed % 100000)
    n = case["paths"]
    nodes, offs, cnts = workloads.perturbed_paths(n, seed, obs)
    g = np.random.Generator(np.random.PCG64(seed + 2))
    lam = np.exp(g.uniform(math.log(0.1), math.log(100.0), n)).astype(np.float32)
    keep = [_dev(nodes), _dev(offs), _dev(cnts), _dev(lam), _dev(obs)]
    var = _empty(T_ROWS, torch.float64)
    lib.check(lib.load().pump_position_variance(T_ROWS, _ptr(var), _stream()))
    a = lib.RefineArgs()
    a.d_nodes, a.n_nodes = _ptr(keep[0]), nodes.shape[0]
    a.d_node_offset, a.d_node_count, a.n_paths = _ptr(keep[1]), _ptr(keep[2]), n
    a.d_lambda, a.W, a.tmax = _ptr(keep[3]), case["W"], 5.0
    a.d_obstacles, a.num_obstacles, a.offset_mult = _ptr(keep[4]), obs.shape[0], case["om"]
    a.d_pos_var, a.T_rows, a.dt, a.sigma_floor = _ptr(var), T_ROWS, DT, 1e-3
    s.update(args=a, keep=keep + [var], grad=torch.zeros(n * 40 * 6, device="cuda"), J=_empty(n, torch.float32))
    return s


# -------------------------------------------------------------------- run
def run(s):
    L, kind, case = lib.load(), s["kind"], s["case"]
    if kind == "plan":
        res = s["res"]
        st = L.pump_plan(s["ctx"].handle, C.byref(s["pb"]), C.byref(res), _stream())
        if st != lib.PUMP_ERR_NO_SOLUTION:
            lib.check(st)
        return dict(path=s["path"], nodes=s["nodes"], path_len=int(res.path_len), num_nodes=int(res.num_nodes),
                    rn=res.rn, cost=res.soln_cost, cp=res.soln_cp, success=int(res.success), edges=int(res.num_edges),
                    stored=int(res.num_paths), considered=int(res.num_considered))
    if kind == "roadmap":
        rn, E = C.c_float(0), C.c_longlong(0)
        lib.check(L.pump_roadmap(s["ctx"].handle, _ptr(s["samples"]), case["N"], 5.0, lib.PUMP_BVP_PRECISION, s["k"],
                                 s["k"], _ptr(s["copts"]), _ptr(s["topts"]), _ptr(s["src"]), _ptr(s["dst"]),
                                 _ptr(s["ce"]), _ptr(s["te"]), _ptr(s["go"]), C.byref(rn), C.byref(E), None,
                                 _stream()))
        E = int(E.value)
        return dict(copts=s["copts"], topts=s["topts"], rn=rn.value, src=s["src"][:E], dst=s["dst"][:E],
                    edge_cost=s["ce"][:E], edge_time=s["te"][:E], go=s["go"])
    if kind == "pairs":
        lib.check(L.pump_bvp_pairs(_ptr(s["samples"]), case["N"], 5.0, case["mode"], _ptr(s["copts"]),
                                   _ptr(s["topts"]), _stream()))
        return dict(copts=s["copts"], topts=s["topts"])
    if kind == "waypoints":
        lib.check(L.pump_discretize_edges(_ptr(s["samples"]), _ptr(s["src"]), _ptr(s["dst"]), _ptr(s["tau"]), s["E"],
                                          s["W"] - 1, case["mode"], _ptr(s["out"]), _stream()))
        return s["out"]
    if kind == "edges":
        lib.check(L.pump_free_edges(_ptr(s["obs"]), case["boxes"], _ptr(s["disc"]), s["E"], s["W"] - 1,
                                    _ptr(s["out"]), _stream()))
        return s["out"]
    if kind == "halfspaces":
        lib.check(L.pump_cache_halfspaces(_ptr(s["obs"]), case["boxes"], _ptr(s["disc"]), _ptr(s["free"]), s["E"],
                                          s["W"], s["H"], s["maxd2"], _ptr(s["a"]), _ptr(s["b"]), _ptr(s["n"]),
                                          _stream()))
        return dict(a=s["a"], b=s["b"], count=s["n"])
    if kind == "hsmc":
        lib.check(L.pump_hsmc_propagate_boxes(
            case["paths"], s["W"], _ptr(s["edge"]), _ptr(s["prev"]), s["E"], s["base"], _ptr(s["obs"]),
            case["boxes"], _ptr(s["disc"]), s["maxd2"], s["H"], _ptr(s["times"]), _ptr(s["tau"]), DT,
            _ptr(s["table"]), s["pmc"], T_ROWS, case["om"], _ptr(s["valid"]), case["particles"], _ptr(s["cp"]),
            _ptr(s["err"]), _stream()))
        return dict(valid=s["valid"], cp=s["cp"], err=s["err"])
    if kind == "mc_cp":
        lib.check(L.pump_mc_cp(_ptr(s["rows"]), _ptr(s["off"]), _ptr(s["len"]), case["paths"], _ptr(s["table"]),
                               case["particles"], T_ROWS, case["om"], _ptr(s["obs"]), case["boxes"], _ptr(s["hits"]),
                               _ptr(s["cp"]), _ptr(s["err"]), _stream()))
        return dict(hits=s["hits"], cp=s["cp"], err=s["err"])
    if kind == "refine":
        lib.check(L.pump_refine_bwd(C.byref(s["args"]), _ptr(s["grad"]), _ptr(s["J"]), _stream()))
        return dict(grad=s["grad"], J=s["J"])
    lib.check(L.pump_path_cp(s["ctx"].handle, s["nodes"].ctypes.data, s["offs"].ctypes.data, s["cnts"].ctypes.data,
                             case["paths"], case["mode"], _ptr(s["table"]), case["particles"], T_ROWS, case["om"],
                             _ptr(s["obs"]), case["boxes"], s["cp"].ctypes.data, s["cost"].ctypes.data,
                             s["len"].ctypes.data, _stream()))
    return dict(cp=s["cp"], cost=s["cost"], len=s["len"])


def work(case):
    """Bytes of the inputs and outputs; operations: about 30 per pair (the
    five coefficients and one cost), 25 per waypoint, 12 per (edge, box) and
    (waypoint, box) test, 6 per (particle, slot) test of half a slot an
    expansion, 24 per (particle, state) plus one box test, 40 per (waypoint,
    box) term of the refinement."""
    kind = case["kind"]
    if kind in ("plan", "roadmap", "pairs"):
        N = case["N"]
        n, E = N * (N - 1), 0.05 * N * (N - 1)
        b, f = 24.0 * N + 8 * n, 30.0 * n
        if kind != "pairs":
            b += 16 * E
        if kind == "plan":
            W = case["disc"] + 1
            b = 48.0 * case["boxes"] + 24 * 400
            f += 25 * E * W + 12 * E * case["boxes"]
        return {"bytes": b, "flops": f}
    if kind in ("waypoints", "edges", "halfspaces"):
        E, W = 0.05 * case["N"] * (case["N"] - 1), case["disc"] + 1
        if kind == "waypoints":
            return {"bytes": 24.0 * case["N"] + 12 * E + 24 * E * W, "flops": 25 * E * W}
        if kind == "edges":
            return {"bytes": 24 * E * W + E, "flops": 12 * E * case["boxes"]}
        H = min(case["boxes"], 5)
        return {"bytes": E + 24 * E * W + E * W * (16 * H + 4), "flops": 12 * E * W * case["boxes"]}
    if kind == "hsmc":
        M, P, W = case["paths"], case["particles"], case["disc"] + 1
        return {"bytes": M * (12 + 24.0 * W + P / 4), "flops": M * (12.0 * W * case["boxes"] + 3 * P)}
    if kind in ("mc_cp", "path_cp"):
        n, P, rows = case["paths"], case["particles"], 80
        b = 24.0 * rows * n + 12 * rows * P + 8 * n
        return {"bytes": b if kind == "mc_cp" else 24.0 * 7 * n + 12 * n + 12 * rows * P,
                "flops": 36.0 * n * P * rows}
    n = case["paths"] * 24.0
    return {"bytes": 48 * n + 8 * case["paths"], "flops": 40.0 * n * case["W"] * 40}


# ------------------------------------------------------------------ exact
def _best(x0, x1, tmax):
    """Binary64 minimiser (time, cost) of the pair cost on (0, tmax]: the
    quartic's monotone pieces between the real roots of its derivative, each
    upward sign change by bisection."""
    A = _coefs(x0, x1)
    A0, A1, A2, A4 = A[0], A[1], A[2], A[4]

    def q(t):
        return ((A4 * t * t - A2) * t - 2 * A1) * t - 3 * A0

    # Q'/(4 A4) = t^3 + p t + w
    p, w = -A2 / (2 * A4), -A1 / (2 * A4)
    three = -4 * p ** 3 - 27 * w * w > 0
    m = 2 * torch.sqrt(torch.clamp(-p / 3, min=0))
    phi = torch.acos(torch.clamp(3 * w / torch.where(p * m == 0, torch.ones_like(p), p * m), -1, 1)) / 3
    cuts = [torch.zeros_like(A0)]
    roots = torch.stack([m * torch.cos(phi - 2 * math.pi * k / 3) for k in range(3)])
    roots = torch.sort(torch.where(three, roots, torch.zeros_like(roots)), 0).values
    # one real root: bisection on Q' over (0, tmax)
    lo, hi = torch.zeros_like(A0), torch.full_like(A0, tmax)
    for _ in range(55):
        mid = 0.5 * (lo + hi)
        up = (4 * A4 * mid * mid - 2 * A2) * mid - 2 * A1 > 0
        lo, hi = torch.where(up, lo, mid), torch.where(up, mid, hi)
    cuts += [torch.clamp(torch.where(three, r, lo), 0, tmax) for r in roots]
    cuts.append(torch.full_like(A0, tmax))
    bt = torch.full_like(A0, tmax)
    bc = _cost(A, bt)
    for a, b in zip(cuts[:-1], cuts[1:]):
        has = (q(a) < 0) & (q(b) > 0)
        if not bool(has.any()):
            continue
        lo, hi = a.clone(), b.clone()
        for _ in range(56):
            mid = 0.5 * (lo + hi)
            neg = q(mid) < 0
            lo, hi = torch.where(neg, mid, lo), torch.where(neg, hi, mid)
        t = torch.where(has, 0.5 * (lo + hi), torch.full_like(A0, tmax))
        c = _cost(A, t)
        take = has & (c < bc)
        bt, bc = torch.where(take, t, bt), torch.where(take, c, bc)
    return bt, bc


def _exact_pairs(N, seed):
    x = _dev(_samples(N, seed)).double()
    copts, topts = _empty(N * (N - 1), torch.float64), _empty(N * (N - 1), torch.float64)
    for i0 in range(0, N, 500):
        i1 = min(N, i0 + 500)
        t, c = _best(x[i0:i1, None, :], x[None, :, :], 5.0)
        off = torch.ones(i1 - i0, N, dtype=torch.bool, device="cuda")
        off[torch.arange(i1 - i0), torch.arange(i0, i1)] = False
        topts[i0 * (N - 1):i1 * (N - 1)], copts[i0 * (N - 1):i1 * (N - 1)] = t[off], c[off]
    return copts, topts


def _exact_refine(case, seed):
    s = prepare(case, seed)
    nodes, offs, cnts, lam, obs = s["keep"][:5]
    om, W, n = float(s["args"].offset_mult), case["W"], case["paths"]
    dt, sf2 = float(s["args"].dt), float(s["args"].sigma_floor) ** 2
    # the closed loop's position variance per step
    h2, kp, kd, sw = 0.5 * DT * DT, 16.0, 5.6, 4.0
    F = np.array([[1 - h2 * kp, DT - h2 * kd], [-DT * kp, 1 - DT * kd]])
    gg = np.array([h2, DT]) * sw
    S, var = np.zeros((2, 2)), []
    for _ in range(T_ROWS):
        var.append(S[0, 0])
        S = F @ S @ F.T + np.outer(gg, gg)
    var = torch.tensor(var, dtype=torch.float64, device="cuda")
    x = nodes.double().view(-1, 6).requires_grad_(True)
    cnt, off = cnts.cpu().numpy(), offs.cpu().numpy()
    i0 = torch.from_numpy(np.concatenate([o + np.arange(c - 1) for o, c in zip(off, cnt)])).cuda()
    path = torch.from_numpy(np.repeat(np.arange(n), cnt - 1)).cuda()
    x0, x1 = x[i0], x[i0 + 1]
    t = _best(x0.detach(), x1.detach(), 5.0)[0]
    A = _coefs(x0, x1)
    slope = -3 * A[0] / t ** 4 - 2 * A[1] / t ** 3 - A[2] / t ** 2 + A[4]
    curv = (12 * A[0] / t ** 5 + 6 * A[1] / t ** 4 + 2 * A[2] / t ** 3).detach()
    tau = torch.where(t >= 5.0, t, t - (slope - slope.detach()) / curv)
    cost = torch.zeros(n, dtype=torch.float64, device="cuda").index_add(0, path, _cost(A, tau))
    run_t = torch.cumsum(tau, 0) - tau
    first = torch.from_numpy(np.concatenate([[0], np.cumsum(cnt - 1)[:-1]])).cuda()
    T0 = run_t - run_t[first][path]
    sv = (torch.arange(W, device="cuda", dtype=torch.float64) / W)[None, :, None]
    st = _cubic(x0[:, None, :], x1[:, None, :], tau[:, None, None], sv)
    p, v = st[..., :3], st[..., 3:]
    u = (T0[:, None] + sv[..., 0] * tau[:, None]) / dt
    j = torch.clamp(torch.floor(u.detach()).long(), 0, T_ROWS - 2)
    V = torch.where(u < T_ROWS - 1, var[j] + (u - j) * (var[j + 1] - var[j]), var[-1])
    sig = om * torch.sqrt(V + sf2)
    vv = (v * v).sum(-1) + 1e-12
    bound = torch.zeros(n, dtype=torch.float64, device="cuda")
    for b in obs.double():
        r = torch.minimum(torch.maximum(p, b[0:3]), b[6:9]) - p
        beta = (r * v).sum(-1) / vv
        a = r - beta[..., None] * v
        z = torch.sqrt((a * a).sum(-1) + 1e-12) / sig
        bound = bound.index_add(0, path, (0.5 * torch.erfc(z * math.sqrt(0.5))).sum(-1))
    J = cost + lam.double() * bound
    J.sum().backward()
    grad = x.grad.clone()
    ends = torch.from_numpy(np.concatenate([off, off + cnt - 1])).cuda()
    grad[ends] = 0
    whole = torch.zeros(n * 40 * 6, dtype=torch.float64, device="cuda")
    whole[:grad.numel()] = grad.reshape(-1)
    return dict(grad=whole, J=J.detach())


def exact(case, seed):
    kind = case["kind"]
    if kind == "roadmap" or (kind == "pairs" and case["mode"] == 1):
        c, t = _exact_pairs(case["N"], seed)
        return dict(copts=c, topts=t)
    if kind == "waypoints":
        s = prepare(case, seed)
        return _waypoints(s["samples"].double(), s["src"], s["dst"], s["tau"].double(), s["W"] - 1).reshape(-1)
    if kind == "refine":
        return _exact_refine(case, seed)
    return None
