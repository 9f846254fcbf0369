"""One particle per group of lanes (lists too short to fill the GPU) at the sizes where
it can go wrong: lists shorter than a warp's groups, partly filled last warps, and one
particle either side of each size where another form takes over.  Every result must
equal the FP32 oracle's bit for bit."""
import numpy as np
import pytest

import oracle as O
from twoscalesplit_gb300 import _abi, scenes
from twoscalesplit_gb300.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from twoscalesplit_gb300 import build
    build.build()


@pytest.mark.parametrize("q1", [True, False])
@pytest.mark.parametrize("n_low,n_high", [(1, 0), (2, 1), (3, 5), (7, 8), (9, 31), (33, 33), (257, 1001), (12000, 12001),
                                          (12001, 12000), (20000, 20001), (20001, 20000), (48000, 48001), (48001, 48000)])
def test_list_lengths(n_low, n_high, q1):
    # the lattice starts at the domain's lower left corner, among the walls
    nx = 180 if n_low > 300 else 12
    sc = scenes.dam_break_small(nx, -(-n_low // nx), seed=n_low, roi=[0.1, 0.1, 0.3, 0.6])
    rng = np.random.default_rng(n_high)
    n, dx = n_low, sc.dx
    pos = (sc.low_pos[:n] + rng.uniform(-0.1 * dx, 0.1 * dx, size=(n, 2))).astype(np.float32)
    vel = rng.standard_normal((n, 2)).astype(np.float32)
    sc.low_pos, sc.low_vel, sc.cap_high = pos, vel, 4 * n + n_high
    if not q1:
        sc.config.flags &= ~_abi.TSS_FLAG_Q1_COMPAT
    # children of the first particles, a few of them in state 0
    hid = np.arange(n_high, dtype=np.int32) % (4 * n)
    hid = np.unique(hid)
    m = len(hid)
    state = np.zeros(n, np.uint8)
    state[: (m + 3) // 4] = 1
    high = {"id": hid, "pos": (pos[hid >> 2] + rng.uniform(-0.3 * dx, 0.3 * dx, size=(m, 2))).astype(np.float32),
            "vel": rng.standard_normal((m, 2)).astype(np.float32), "state": (rng.random(m) > 0.02).astype(np.uint8)}
    sol, orc = Solver.from_scene(sc), O.Oracle(sc, 32)
    ids = np.arange(n, dtype=np.int32)
    sol.upload(0, {"id": ids, "pos": pos, "vel": vel, "state": state})
    orc.set_scale(0, ids, pos, vel, state)
    if m:
        sol.upload(1, high)
        orc.set_scale(1, high["id"], high["pos"], high["vel"], high["state"])
    for k in range(2):
        sol.step(1)
        orc.step()
        for s in (0, 1):
            assert np.array_equal(sol.copy(s, _abi.TSS_BUF_SORTED_ID), orc.get(s, "sorted_id")), (k, s)
            for which, name in ((_abi.TSS_BUF_DENSITY, "dens"), (_abi.TSS_BUF_ACCEL, "acc")):
                assert np.array_equal(sol.copy(s, which), orc.get(s, name).astype(np.float32), equal_nan=True), (k, s, name)
            d, st = sol.download(s), orc.state(s)
            assert np.array_equal(d["id"], st["id"]) and np.array_equal(d["state"], st["state"]), (k, s)
            for f in ("pos", "vel"):
                assert np.array_equal(d[f], st[f].astype(np.float32), equal_nan=True), (k, s, f)


@pytest.mark.parametrize("cells", [500, 140000])
def test_walls_of_wide_grids(cells):
    # a grid of more columns than the two-cell rule for wall windows is used for; the
    # particles stand on walls in its corners and outside it
    rng = np.random.default_rng(cells)
    r = 1.0 / cells
    dx = 0.5 * r
    cfg = _abi.config_init(0.0, 0.0, 1.0, 6 * r, r, dx, scenes.REST_DENSITY, scenes.TAIT_B, scenes.SPEED_SOUND,
                           scenes.ALPHA, scenes.SIGMA, 1e-9)
    cfg.roi[:] = [9.0, 9.0, 10.0, 10.0]
    x = np.concatenate([np.arange(20) * dx, 1.0 - np.arange(1, 21) * dx, 0.5 + np.arange(20) * dx])
    walls = np.stack([np.repeat(x, 2), np.tile([0.0, 0.5 * dx], len(x))], axis=1)
    pos = np.stack([np.repeat(x, 5), np.tile(1.5 * dx + np.arange(5) * dx, len(x))], axis=1)
    pos += rng.uniform(-0.2 * dx, 0.2 * dx, size=pos.shape)
    pos[::37] += [[-4 * r, -5 * r]]
    n = len(pos)
    pos, vel = pos.astype(np.float32), rng.standard_normal((n, 2)).astype(np.float32)
    m = scenes.REST_DENSITY * dx * dx
    sc = scenes.Scene("wide", cfg, pos, vel, m, m / 4, 4 * n, walls.astype(np.float32), m / 4, 1, dx)
    high = {"id": np.arange(4 * n, dtype=np.int32), "pos": (np.repeat(pos, 4, axis=0) + rng.uniform(-0.3 * dx, 0.3 * dx, size=(4 * n, 2))).astype(np.float32),
            "vel": np.repeat(vel, 4, axis=0), "state": np.ones(4 * n, np.uint8)}
    ids = np.arange(n, dtype=np.int32)
    sol, orc = Solver.from_scene(sc), O.Oracle(sc, 32)
    sol.upload(0, {"id": ids, "pos": pos, "vel": vel, "state": np.ones(n, np.uint8)})
    orc.set_scale(0, ids, pos, vel, np.ones(n, np.uint8))
    sol.upload(1, high)
    orc.set_scale(1, high["id"], high["pos"], high["vel"], high["state"])
    sol.step(1)
    orc.step()
    for s in (0, 1):
        assert np.array_equal(sol.copy(s, _abi.TSS_BUF_SORTED_ID), orc.get(s, "sorted_id")), s
        assert np.array_equal(sol.copy(s, _abi.TSS_BUF_ACCEL), orc.get(s, "acc").astype(np.float32), equal_nan=True), s


@pytest.mark.parametrize("nx", [3, 40, 80])
def test_relaxing_few_and_many_children(nx):
    # 4 nx^2 children relax at once: by groups of lanes, or (25,600) one per thread
    sc = scenes.dam_break_small(nx, nx, dx=0.4 / nx, seed=nx, relax_iters=2, roi=[-1.0, -1.0, 2.0, 2.0])
    sc.config.flags |= _abi.TSS_FLAG_OLDER_PLACEMENT
    sol, orc = Solver.from_scene(sc), O.Oracle(sc, 32)
    for k in range(3):
        sol.step(1)
        orc.step()
        for s in (0, 1):
            d, st = sol.download(s), orc.state(s)
            assert np.array_equal(d["id"], st["id"]), (k, s)
            for f in ("pos", "vel"):
                assert np.array_equal(d[f], st[f].astype(np.float32), equal_nan=True), (k, s, f)
    assert sol.counts()["n_high"] == 4 * nx * nx
