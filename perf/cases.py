"""The calls this library is timed on, from the smallest scene to the largest.

Every case is something a user's program does through the public interface: step
one scene (`Solver.step`), step it and read the positions back to the host, step a
batch of scenes (`Batch.step`), serve a burst of requests (`Server.run`), or build
a neighbour grid on device arrays of its own (`tss_grid_build`).

The scenes are dam breaks some way into their flow, which is where a run spends
its steps: the fluid has spread into a slope along the floor, the particles right
of a line have been split (their four children lie close together beside their
parent, as they do after a while in this model), and the front is still moving
into the region of interest.  They are made directly from the seed instead of by
thousands of steps.  Physical constants, walls, time step and masses are those of
`scenes.dam_break_small` at the spacing that the particle count gives.
"""
import ctypes
import dataclasses
import math

import numpy as np
import torch

from twoscalesplit_gb300 import _abi, scenes
from twoscalesplit_gb300.serving import Request, Server, footprint, pool_config
from twoscalesplit_gb300.solver import Batch, Solver

# The slope: heights HEIGHT * (1 - x / FRONT), the area of the dam breaks' blocks
# (0.4 x 0.8).
FRONT = 0.9
AREA = 0.32
HEIGHT = 2.0 * AREA / FRONT
# The region of interest reaches from the line that leaves the wanted share of the
# particles to its right, to here.
ROI_RIGHT, ROI_TOP = 0.95, 0.5


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _step(n, arith="exact", steps=1, split=0.25, relax=0, merge=False, readback=False):
    """One scene of n low-res particles, `split` of them split (4 children each)."""
    return {"kind": "step", "n": n, "arith": arith, "steps": steps, "split": split, "relax": relax, "merge": merge,
            "readback": readback}


def _batch(scenes_, n_min, n_max, arith, steps=1):
    return {"kind": "batch", "scenes": scenes_, "n_min": n_min, "n_max": n_max, "arith": arith, "steps": steps}


def _serve(requests, n_min, n_max, h_min, h_max):
    return {"kind": "serve", "requests": requests, "n_min": n_min, "n_max": n_max, "h_min": h_min, "h_max": h_max}


def _grid(n):
    return {"kind": "grid", "n": n}


def listed():
    return [
        # the smallest scene of the mixed-size workloads, stepped one step at a time
        # by a host loop that looks at it in between: launches and latency
        dict(_step(2003), name="scene_2k"),
        # the 5k dam break, the reference's own kind of scene
        dict(_step(5000, split=0.3), name="dam_5k"),
        # the same with its children relaxed before they couple, eight steps a call
        dict(_step(5000, steps=8, split=0.3, relax=4), name="dam_5k_relaxed_x8"),
        # the median scene of the serving workload, in the tolerance arithmetic
        dict(_step(22391, "fast"), name="scene_22k_fast"),
        # a large scene of the mixed-size workloads whose positions a program on the
        # host reads after every step (overlapped read-back into page-locked memory)
        dict(_step(161999, readback=True), name="scene_162k_readback"),
        # the 1M dam break with 1M high-res particles, both arithmetics
        dict(_step(999698), name="dam_1m"),
        dict(_step(999698, "fast"), name="dam_1m_fast"),
        # the 1M dam break before the flow reaches the region of interest
        dict(_step(999698, split=0.0), name="dam_1m_unsplit"),
        # adaptive stress: a region of interest that moves, with merging, no Q1 term
        dict(_step(3000001, split=0.28, merge=True), name="adaptive_3m"),
        # many scenes of uneven sizes in one launch set, both arithmetics by size
        dict(_batch(48, 2000, 60000, "exact"), name="batch_48"),
        # a burst of requests through the serving loop: admission, continuous
        # batching, extraction, retirement
        dict(_serve(12, 1000, 30000, 40, 160), name="serve_burst_12"),
        # the neighbour grid alone, on a program's own device arrays
        dict(_grid(1300021), name="grid_1300k"),
    ]


def _log_uniform(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["batch", "batch", "serve", "grid"])
    if kind == "step":
        n = _log_uniform(rng, 1500, 1100000)
        merge = rng.random() < 0.2
        small = n < 30000
        return _step(n, rng.choice(["exact", "exact", "fast"]), rng.choice([1, 1, 2, 3, 8]) if small else 1,
                     0.0 if rng.random() < 0.15 and not merge else round(rng.uniform(0.05, 0.4), 3),
                     rng.choice([0, 0, 4]) if small and not merge else 0, merge, rng.random() < 0.2)
    if kind == "batch":
        n_min = _log_uniform(rng, 1000, 8000)
        return _batch(rng.randint(2, 64), n_min, n_min * rng.randint(2, 8), rng.choice(["exact", "fast"]),
                      rng.choice([1, 1, 2]))
    if kind == "serve":
        n_min = _log_uniform(rng, 1000, 4000)
        h = rng.randint(10, 60)
        return _serve(rng.randint(3, 14), n_min, n_min * rng.randint(2, 8), h, 2 * h)
    return _grid(_log_uniform(rng, 1000, 1500000))


# ---------------------------------------------------------------------------
# scenes
# ---------------------------------------------------------------------------
def _sizes(count, a, b, salt):
    """Log-uniform sizes that belong to the case, not to the seed."""
    r = np.random.default_rng(1000 * count + salt)
    return [int(x) for x in np.exp(r.uniform(math.log(a), math.log(b), size=count)).round()]


def _fluid(n, rng):
    """n points of a turned square lattice in the slope, a little disordered, and its spacing."""
    dx = float(np.float32(math.sqrt(AREA / n)))
    th = rng.uniform(0.15, 0.6)
    k = int(1.3 / dx) + 2
    c, s = math.cos(th), math.sin(th)
    i = np.arange(-k, k + 1, dtype=np.float64) * dx
    # rows of the turned lattice that meet the box of the slope
    v = i[(i > -FRONT * s - 2 * dx) & (i < (HEIGHT + 0.1) * c + 2 * dx)]
    out = []
    for lo in range(0, len(v), 256):
        u, w = np.meshgrid(i[i > -2 * dx], v[lo:lo + 256])
        x, y = c * u - s * w + rng.uniform(0, 1e-9), s * u + c * w
        m = (x >= 0.5 * dx) & (y >= 0.5 * dx) & (x < FRONT) & (y < 1.1 * HEIGHT * (1.0 - x / FRONT) + 4 * dx)
        out.append(np.stack([x[m], y[m]], axis=1))
    p = np.concatenate(out)
    # the n points lowest in the slope
    score = p[:, 1] - HEIGHT * (1.0 - p[:, 0] / FRONT)
    p = p[np.argpartition(score, n - 1)[:n]] if len(p) > n else p
    assert len(p) == n, (len(p), n)
    p = p[np.argsort((p[:, 1] * c - p[:, 0] * s) // dx, kind="stable")]  # row by row, as a lattice is laid down
    p += rng.uniform(-0.03 * dx, 0.03 * dx, size=p.shape)
    return np.maximum(p, 0.4 * dx).astype(np.float32), dx


@dataclasses.dataclass
class _Flow:
    scene: object
    state: np.ndarray  # uint8 [n]: 1 for a split particle
    high: dict         # the children: id, pos, vel, state


def _flow(n, split, seed, relax=0, merge=False):
    rng = np.random.default_rng(seed)
    pos, dx = _fluid(n, rng)
    vel = np.stack([2.0 * pos[:, 0] / FRONT, -1.5 * pos[:, 1]], axis=1)
    vel = (vel + 0.02 * rng.standard_normal(vel.shape)).astype(np.float32)
    # the line with exactly k particles to its right, below the region's top
    k = int(split * n)
    below = np.sort(pos[pos[:, 1] < np.float32(ROI_TOP - 0.01), 0])[::-1]
    x0 = float(below[k])
    top = ROI_TOP - 0.01 if k else ROI_TOP
    roi = [x0, -1.0, ROI_RIGHT, top] if k else [FRONT + 0.04, 0.0, FRONT + 0.05, ROI_TOP]
    if merge:
        sc = scenes.adaptive_dam_break(2, 4, dx, cap_high=4 * n)
        sc.config.roi_velocity[:] = [0.5, 0.0]
    else:
        sc = scenes.dam_break_small(2, 4, dx=dx, relax_iters=relax, cap_high=4 * n)
    sc.config.roi[:] = roi
    sc.config.flags |= _abi.TSS_FLAG_TETHER_GUARD
    if relax:
        sc.config.flags |= _abi.TSS_FLAG_OLDER_PLACEMENT
    sc = dataclasses.replace(sc, low_pos=pos, low_vel=vel)
    state = np.zeros(n, np.uint8)
    if k:
        state[(pos[:, 0] > np.float32(x0)) & (pos[:, 1] < np.float32(top))] = 1
    par = np.flatnonzero(state)
    # children: in a clump beside their parent, most of them much closer to each
    # other than to it
    phi = 3.0 + 0.7 * rng.standard_normal(len(par))
    off = 0.34 * dx * rng.uniform(0.7, 1.0, len(par))[:, None] * np.stack([np.cos(phi), np.sin(phi)], axis=1)
    wide = dx * 10.0 ** rng.uniform(-2.5, -0.9, size=(len(par), 1, 1))
    cp = pos[par][:, None, :] + off[:, None, :] + wide * rng.standard_normal((len(par), 4, 2))
    cv = vel[par][:, None, :] + 0.3 * rng.standard_normal((len(par), 4, 2))
    high = {"id": (4 * par[:, None] + np.arange(4)).astype(np.int32).reshape(-1),
            "pos": np.maximum(cp, 0.05 * dx).astype(np.float32).reshape(-1, 2),
            "vel": cv.astype(np.float32).reshape(-1, 2), "state": np.ones(4 * len(par), np.uint8)}
    return _Flow(sc, state, high)


def _flows(case, seed):
    """The scenes of a step or batch case."""
    if case["kind"] == "step":
        return [_flow(case["n"], case["split"], seed, case["relax"], case["merge"])]
    sizes = _sizes(case["scenes"], case["n_min"], case["n_max"], 1)
    shares = np.random.default_rng(case["scenes"]).uniform(0.1, 0.4, len(sizes))
    return [_flow(n, float(s), seed * 1000 + j) for j, (n, s) in enumerate(zip(sizes, shares))]


# ---------------------------------------------------------------------------
# what a program has in hand, and one pass
# ---------------------------------------------------------------------------
class _View:
    """Device memory of a solver as __cuda_array_interface__; keeps the solver alive."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": typestr, "data": (int(ptr), False), "version": 3,
                                         "strides": None}


def _lists(solver, n_low, n_high, n_born):
    """The solver's device buffers as tensors: the low-res list, the high-res list
    as long as it is now, and the entries that new children take."""
    b = solver.device_buffers()
    out = {}
    for scale, name, first, count in ((0, "low", 0, n_low), (1, "high", 0, n_high), (1, "born", n_high, n_born)):
        part = {}
        for key, width, size, kind in (("pos", 2, 8, "<f4"), ("vel", 2, 8, "<f4"), ("dens", 1, 4, "<f4"),
                                       ("id", 1, 4, "<i4"), ("state", 1, 1, "|u1")):
            if name == "born" and key == "dens":
                continue
            shape = (count, 2) if width == 2 else (count,)
            ptr = getattr(b, key)[scale] + first * size
            part[key] = torch.as_tensor(_View(solver, ptr, shape, kind), device="cuda") if count else None
        out[name] = part
    out["counts"] = torch.as_tensor(_View(solver, b.counts, (2,), "<i4"), device="cuda")
    return out


def prepare(case, seed):
    if case["kind"] in ("step", "batch"):
        flows = _flows(case, seed)
        if case["kind"] == "step":
            solver = Solver.from_scene(flows[0].scene)
            bases = [0]
        else:
            solver = Batch([f.scene for f in flows])
            ids = solver.download(0)["id"]  # scene by scene
            bases = ids[np.cumsum([0] + [f.scene.n_low for f in flows[:-1]])].tolist()
        n_low = sum(f.scene.n_low for f in flows)
        n_high = sum(len(f.high["id"]) for f in flows)
        if n_high:
            solver.upload(0, {"id": np.concatenate([b + np.arange(f.scene.n_low) for b, f in zip(bases, flows)]),
                              "pos": np.concatenate([f.scene.low_pos for f in flows]),
                              "vel": np.concatenate([f.scene.low_vel for f in flows]),
                              "state": np.concatenate([f.state for f in flows])})
            solver.upload(1, {"id": np.concatenate([4 * b + f.high["id"] for b, f in zip(bases, flows)]),
                              **{k: np.concatenate([f.high[k] for f in flows]) for k in ("pos", "vel", "state")}})
        solver.set_arith(case["arith"])
        st = {"case": case, "solver": solver, "out": _lists(solver, n_low, n_high, min(8192, solver.cap_high - n_high))}
        if case.get("readback"):
            cap = min(solver.cap_high, n_high + 8192)
            st["host"] = [[torch.zeros((n_low, 2), pin_memory=True), torch.zeros((cap, 2), pin_memory=True),
                           torch.zeros(2, dtype=torch.int32, pin_memory=True)] for _ in range(2)]
            st["turn"], st["ticket"] = 0, None
        return st
    if case["kind"] == "serve":
        n = case["requests"]
        hs = np.random.default_rng(n).integers(case["h_min"], case["h_max"] + 1, n)
        reqs = [Request(_flow(m, 0.2, seed * 1000 + j).scene, int(h), 0.0, True)
                for j, (m, h) in enumerate(zip(_sizes(n, case["n_min"], case["n_max"], 2), hs))]
        feet = [footprint(r.scene) for r in reqs]
        # a pool for about two thirds of the burst, so that the rest waits for room
        room = {k: max(max(f[k] for f in feet), int(0.67 * sum(f[k] for f in feet)))
                for k in ("low_slots", "high_particles", "low_cells", "high_cells", "wall_particles")}
        pool = pool_config(room["low_slots"] + 256, room["high_particles"], room["low_cells"] + 64,
                           room["high_cells"] + 64, room["wall_particles"] + 64, max_scenes=n)
        # where the program gathers the results: per scale, all requests' lists end to end
        store = []
        for per in (1, 4):
            m = per * sum(r.scene.n_low for r in reqs)
            store.append({"id": np.zeros(m, np.int32), "pos": np.zeros((m, 2), np.float32), "vel": np.zeros((m, 2), np.float32),
                          "state": np.zeros(m, np.uint8), "dens": np.zeros(m, np.float32)})
        return {"case": case, "server": Server(pool, staging_bytes=1 << 28), "requests": reqs, "store": store}
    n = case["n"]
    rng = np.random.default_rng(seed)
    pos, dx = _fluid(n, rng)
    r = 2.0 * dx
    dims = int(math.ceil(1.0 / r)) + 4
    lib = _abi.load_library()
    ws = ctypes.c_size_t(0)
    _abi.check(lib.tss_grid_workspace_size(n, dims, dims, ctypes.byref(ws)))
    return {"case": case, "lib": lib, "dims": dims, "cell": r, "pos": torch.from_numpy(pos).cuda(),
            "id": torch.from_numpy(np.sort(rng.permutation(2 * n)[:n]).astype(np.int32)).cuda(),
            "order": torch.empty(n, dtype=torch.int32, device="cuda"),
            "off": torch.empty(dims * dims + 1, dtype=torch.int32, device="cuda"),
            "work": torch.empty(ws.value, dtype=torch.uint8, device="cuda"), "bytes": ws.value}


def run(state):
    case = state["case"]
    if case["kind"] in ("step", "batch"):
        solver = state["solver"]
        solver.step(case["steps"])
        if not case.get("readback"):
            return state["out"]
        # read these positions back while the next step runs; wait for the last ones
        host = state["host"][state["turn"]]
        ticket = solver.read_positions_async(*host)
        if state["ticket"] is not None:
            solver.read_wait(state["ticket"])
        state["ticket"], state["turn"] = ticket, 1 - state["turn"]
        return {"lists": state["out"], "host": {"low": host[0], "high": host[1], "counts": host[2]}}
    if case["kind"] == "serve":
        stats, _, results = state["server"].run(state["requests"])
        for scale, store in enumerate(state["store"]):
            at = 0
            for req, res in zip(state["requests"], results):
                for k, whole in store.items():
                    whole[at:at + len(res[scale][k])] = res[scale][k]
                at += (1, 4)[scale] * req.scene.n_low
        return {"status": np.array([s["status"] for s in stats], np.int32),
                "n": np.array([[s["n_low"], s["n_high"]] for s in stats], np.int32),
                "low": state["store"][0], "high": state["store"][1]}
    ptr = lambda t: ctypes.c_void_p(t.data_ptr())  # noqa: E731
    _abi.check(state["lib"].tss_grid_build(
        ptr(state["pos"]), ptr(state["id"]), case["n"], 0.0, 0.0, state["cell"], state["dims"], state["dims"],
        ptr(state["order"]), ptr(state["off"]), ptr(state["work"]), state["bytes"],
        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
    return {"order": state["order"], "off": state["off"]}


# ---------------------------------------------------------------------------
# the least a pass can do
# ---------------------------------------------------------------------------
# A step reads a particle's position, velocity, state and id (21 bytes) and writes
# them and its density (25 bytes).  Its sums have about 12 same-scale neighbours:
# some 25 operations each for the density (distance, two cubic splines) and 65 for
# the force (gradient and kernel of both scales, viscosity, two vector sums).
STEP_BYTES, STEP_FLOPS = 46, 12 * (25 + 65)


def work(case):
    if case["kind"] == "grid":
        dims = int(math.ceil(1.0 / (2.0 * math.sqrt(AREA / case["n"])))) + 4
        return {"bytes": 16 * case["n"] + 4 * dims * dims, "flops": 8 * case["n"]}
    if case["kind"] == "serve":
        n = case["requests"]
        hs = np.random.default_rng(n).integers(case["h_min"], case["h_max"] + 1, n)
        ps = 1.8 * float(np.dot(_sizes(n, case["n_min"], case["n_max"], 2), hs))
        return {"bytes": STEP_BYTES * ps, "flops": STEP_FLOPS * ps}
    if case["kind"] == "batch":
        sizes = _sizes(case["scenes"], case["n_min"], case["n_max"], 1)
        shares = np.random.default_rng(case["scenes"]).uniform(0.1, 0.4, len(sizes))
        n = float(np.dot(sizes, 1.0 + 4.0 * shares))
    else:
        n = case["n"] * (1.0 + 4.0 * case["split"])
    return {"bytes": STEP_BYTES * n * case["steps"] + (8 * n if case.get("readback") else 0),
            "flops": STEP_FLOPS * n * case["steps"]}


# ---------------------------------------------------------------------------
# one step in 64 bits
# ---------------------------------------------------------------------------
def _pairs(tp, sp, rad, visit):
    """Calls visit(j, ok) so that every source within rad of target i comes up once as
    (j[i], ok[i]); some that are further off come up too."""
    if len(tp) == 0 or len(sp) == 0:
        return
    lo = torch.minimum(tp.min(0).values, sp.min(0).values) - rad
    hi = torch.maximum(tp.max(0).values, sp.max(0).values) + rad
    w, h = (int(v) + 3 for v in ((hi - lo) / rad).tolist())
    cell = lambda p: ((p - lo) / rad).floor().long()  # noqa: E731
    sc, tc = cell(sp), cell(tp)
    order = torch.argsort(sc[:, 1] * w + sc[:, 0])
    off = torch.zeros(w * h + 1, dtype=torch.int64, device=tp.device)
    off[1:] = torch.cumsum(torch.bincount(sc[:, 1] * w + sc[:, 0], minlength=w * h)[: w * h], 0)
    for dy in (-1, 0, 1):
        row = (tc[:, 1] + dy).clamp(0, h - 1) * w
        live = (tc[:, 1] + dy >= 0) & (tc[:, 1] + dy < h)
        a, b = off[row + (tc[:, 0] - 1).clamp(0, w - 1)], off[row + (tc[:, 0] + 1).clamp(0, w - 1) + 1]
        for k in range(int((b - a).max())):
            visit(order[(a + k).clamp(max=len(sp) - 1)], live & (a + k < b))


class _Exact:
    """One step of one scene from its state, in 64 bits."""

    def __init__(self, flow):
        self.dev = "cuda" if torch.cuda.is_available() else "cpu"
        self.f, self.c = flow, flow.scene.config
        c = self.c
        self.r, self.rh = float(c.r_low), float(c.r_high)
        self.mL, self.mH, self.mB = (float(np.float32(m)) for m in (flow.scene.mass_low, flow.scene.mass_high,
                                                                     flow.scene.mass_wall))

    def t(self, a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(self.dev).double()

    @staticmethod
    def w(d, s):
        q, k = 2.0 * d / s, 20.0 / (14.0 * math.pi * s * s)
        a, b = (2.0 - q).clamp(min=0.0), (1.0 - q).clamp(min=0.0)
        return k * (a ** 3 - 4.0 * b ** 3)

    @staticmethod
    def dw_over_d(d, s):
        # with (2-q)^2 - 4(1-q)^2 = q (4 - 3q) where q < 1
        q, g = 2.0 * d / s, -120.0 / (14.0 * math.pi * s ** 3)
        return torch.where(q < 1, g * (2.0 / s) * (4.0 - 3.0 * q), torch.where(q < 2, g * (2.0 - q) ** 2 / d, 0.0 * d))

    def density(self, tp, sp, rad, keep):
        out = torch.zeros(len(tp), dtype=torch.float64, device=self.dev)

        def visit(j, ok):
            d = (tp - sp[j]).norm(dim=1)
            out.add_(torch.where(ok & keep[j] & (d <= rad), 0.5 * (self.w(d, self.r) + self.w(d, self.rh)), 0.0))

        _pairs(tp, sp, rad, visit)
        return out

    def force(self, tp, tv, tq, td, sp, sv, sq, sd, rad, h, keep):
        """Pressure and viscosity sum, and the sigma sum."""
        acc, ten = torch.zeros_like(tp), torch.zeros_like(tp)
        alpha, cs = float(self.c.alpha), float(self.c.speed_sound)

        def visit(j, ok):
            x, v = tp - sp[j], tv - sv[j]
            d = x.norm(dim=1)
            ok = ok & keep[j] & (d > 0) & (d < rad)
            d = torch.where(ok, d, 1.0)
            dvp = (x * v).sum(1)
            visc = dvp / (d * d + 0.01 * h * h) * 2.0 * h * alpha * cs / (td + sd[j])
            co = tq + sq[j] - torch.where(dvp < 0, visc, 0.0)
            g = 0.5 * co * (self.dw_over_d(d, self.r) + self.dw_over_d(d, self.rh))
            acc.add_(torch.where(ok, g, 0.0)[:, None] * x)
            ten.add_(torch.where(ok, 0.5 * (self.w(d, self.r) + self.w(d, self.rh)), 0.0)[:, None] * x)

        _pairs(tp, sp, rad, visit)
        return acc, ten

    def wall(self, tp, rad, share):
        acc, wp, cs = torch.zeros_like(tp), self.t(self.f.scene.wall_pos), float(self.c.speed_sound)

        def visit(j, ok):
            x = tp - wp[j]
            d = x.norm(dim=1)
            q = 2.0 * d / rad
            f = torch.where(q < 2 / 3, 2 / 3 + 0.0 * q, torch.where(q < 1, 2 * q - 1.5 * q * q, 0.5 * (2 - q) ** 2))
            acc.add_(torch.where(ok & (q < 2), share * 0.02 * cs * cs / (d * d) * f, 0.0)[:, None] * x)

        _pairs(tp, wp, rad, visit)
        return acc

    def order(self, pos, ids, cell, dims):
        """(cell, id) order; the cells as 32-bit arithmetic gives them."""
        f = np.float32
        o = [f(v) for v in self.c.domain_origin[:]]
        cx = np.clip(((pos[:, 0] - o[0]) / f(cell)).astype(np.int64), 0, dims[0] - 1)
        cy = np.clip(((pos[:, 1] - o[1]) / f(cell)).astype(np.int64), 0, dims[1] - 1)
        return np.lexsort((ids, cy * dims[0] + cx))

    def step(self):
        f, c, sc = self.f, self.c, self.f.scene
        dt, g = float(c.dt), float(c.gravity)
        merge, q1 = bool(c.flags & _abi.TSS_FLAG_MERGE), bool(c.flags & _abi.TSS_FLAG_Q1_COMPAT)
        n = sc.n_low
        p, v = self.t(sc.low_pos), self.t(sc.low_vel)
        split = torch.from_numpy(f.state).to(self.dev) == 1
        hp, hv = self.t(f.high["pos"]), self.t(f.high["vel"])
        every, hevery = (torch.ones(k, dtype=torch.bool, device=self.dev) for k in (n, len(hp)))
        tait = lambda d: float(c.tait_b) * ((d / float(c.rest_density)) ** 7 - 1.0)  # noqa: E731
        d = self.mL * self.density(p, p, self.r, every)
        dh = self.mH * self.density(hp, hp, self.rh, hevery)
        if not q1:
            dh = dh + self.mL * self.density(hp, p, self.rh, ~split)
        q, qh = tait(d) / d ** 2, tait(dh) / dh ** 2
        down = torch.tensor([0.0, g], dtype=torch.float64, device=self.dev)
        acc, ten = self.force(p, v, q, d, p, v, q, d, self.r, self.r, every)
        acc = -self.mL * acc - float(c.tension) * ten + self.wall(p, self.r, self.mB / (self.mL + self.mB)) - down
        v1 = v + dt * acc
        p1 = p + dt * v1
        roi = [float(x) for x in c.roi[:]]
        inside = (p1[:, 0] > roi[0]) & (p1[:, 0] < roi[2]) & (p1[:, 1] > roi[1]) & (p1[:, 1] < roi[3])
        free = ~inside if merge else ~inside & ~split  # in state 0 after the split marks
        acc, ten = self.force(hp, hv, qh, dh, hp, hv, qh, dh, self.rh, self.rh, hevery)
        accl, tenl = self.force(hp, hv, qh, dh, p, v, q, d, self.r, 0.5 * (self.r + self.rh), free)
        acc = (-self.mH * acc - self.mL * accl - float(c.tension) * (ten + tenl)
               + self.wall(hp, self.rh, self.mB / (self.mH + self.mB)) - down)
        hv1 = hv + dt * acc
        hp1 = hp + dt * hv1
        parent = torch.from_numpy(f.high["id"] >> 2).to(self.dev).long()
        x = hp1 - p1[parent]
        dist = x.norm(dim=1)
        lim = torch.minimum(dist, 0.75 * torch.sqrt(self.mL / (d[parent] * math.pi)))
        held = (dist > 0) & ~(free[parent] & split[parent])
        hp1 = torch.where(held[:, None], p1[parent] + (lim / dist)[:, None] * x, hp1)
        low = torch.from_numpy(self.order(sc.low_pos, np.arange(n), c.r_low, c.dims_low[:])).to(self.dev)
        high = torch.from_numpy(self.order(f.high["pos"], f.high["id"], c.r_high, c.dims_high[:])).to(self.dev)
        return ({"pos": p1[low], "vel": v1[low], "dens": d[low]},
                {"pos": hp1[high], "vel": hv1[high], "dens": dh[high]})


def exact(case, seed):
    """The lists after one step.  After more than one, the order of the list is that
    of the cells of positions that 64 bits round another way: no value then."""
    if case["kind"] not in ("step", "batch") or case["steps"] != 1:
        return None
    parts = [_Exact(f).step() for f in _flows(case, seed)]
    none = {k: None for k in ("pos", "vel", "dens", "id", "state")}
    lists = {}
    for at, name in enumerate(("low", "high")):
        lists[name] = dict(none)
        for k in ("pos", "vel", "dens"):
            whole = torch.cat([x[at][k] for x in parts])
            lists[name][k] = whole if len(whole) else None
    lists["born"] = {k: None for k in ("pos", "vel", "id", "state")}
    lists["counts"] = None
    if not case.get("readback"):
        return lists
    return {"lists": lists, "host": {"low": lists["low"]["pos"], "high": None, "counts": None}}
