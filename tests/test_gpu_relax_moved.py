"""Children that the relaxation carries out of the cells they were sorted into, to a
place with about as many neighbours as a list holds: the particle itself is not in its
window then.  Every result must equal the FP32 oracle's bit for bit."""
import math

import numpy as np
import pytest

import oracle as O
from twoscalesplit_gb300 import _abi, scenes
from twoscalesplit_gb300._abi import config_init
from twoscalesplit_gb300.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from twoscalesplit_gb300 import build
    build.build()


def _rows(x0, x1, y0, dx, n):
    """n lattice points of spacing dx, row by row from y0 up."""
    nx = int((x1 - x0) / dx) + 1
    k = np.arange(n)
    return np.stack([x0 + dx * (k % nx), y0 + dx * (k // nx)], axis=1)


# the densities take a group of lanes a particle up to 12,000, the forces up to 48,000
@pytest.mark.parametrize("n_high", [3000, 13000, 21000, 49000])
def test_children_moved_into_a_crowd(n_high):
    rng = np.random.default_rng(n_high)
    r, rh, dt = 0.01, 0.005, 1e-4
    crowds = 40
    sizes = 22 + np.arange(crowds) % 6  # 22 ... 27 others within the support
    cx, cy = np.meshgrid(0.04 + 0.08 * np.arange(8), 0.04 + 0.04 * np.arange(5))
    centre = np.stack([cx.ravel(), cy.ravel()], axis=1)
    crowd = np.concatenate([c + rng.uniform(-0.2 * rh, 0.2 * rh, size=(m, 2)) for c, m in zip(centre, sizes)])
    start = np.stack([0.04 + 0.02 * (np.arange(crowds) % 10), 0.26 + 0.02 * (np.arange(crowds) // 10)], axis=1)
    rest = _rows(0.02, 0.78, 0.45, 1.5 * rh, n_high - len(crowd) - crowds)  # no neighbours
    n_low = (len(crowd) + len(rest) + 3) // 4 + crowds
    low = _rows(0.9, 1.5, 0.02, 1.2 * r, n_low).astype(np.float32)
    cfg = config_init(0.0, 0.0, 1.6, max(rest[:, 1].max(), low[:, 1].max()) + 0.1, r, rh, scenes.REST_DENSITY,
                      scenes.TAIT_B, scenes.SPEED_SOUND, scenes.ALPHA, scenes.SIGMA, dt)
    cfg.roi[:] = [math.inf] * 4
    cfg.relax_iters, cfg.relax_dt_div = 1, 1.0
    mass = scenes.REST_DENSITY * (r / 2) ** 2
    sc = scenes.Scene("moved", cfg, low, np.zeros_like(low), mass, mass / 4, 4 * n_low, np.zeros((0, 2), np.float32),
                      mass / 4, 1, r / 2)
    # the first `crowds` parents have one fresh child each, the others up to four older ones
    fresh = np.arange(crowds, dtype=np.int32)
    pos = np.concatenate([start, crowd, rest])
    vel = np.zeros_like(pos)
    vel[:crowds] = (centre - start) / dt
    ids = np.concatenate([4 * fresh + rng.integers(0, 4, crowds), 4 * crowds + np.arange(len(crowd) + len(rest))])
    high = {"id": ids.astype(np.int32), "pos": pos.astype(np.float32), "vel": vel.astype(np.float32),
            "state": np.ones(len(pos), np.uint8)}
    sol, orc = Solver.from_scene(sc), O.Oracle(sc, 32)
    sol.upload(1, high)
    orc.set_scale(1, high["id"], high["pos"], high["vel"], high["state"])
    sol.set_fresh(fresh)
    orc.set_fresh(fresh)
    for k in range(2):
        sol.step(1)
        orc.step()
        for s in (0, 1):
            assert np.array_equal(sol.copy(s, _abi.TSS_BUF_SORTED_ID), orc.get(s, "sorted_id")), (k, s)
            for which, name in ((_abi.TSS_BUF_DENSITY, "dens"), (_abi.TSS_BUF_ACCEL, "acc")):
                assert np.array_equal(sol.copy(s, which), orc.get(s, name).astype(np.float32), equal_nan=True), (k, s, name)
            d, st = sol.download(s), orc.state(s)
            for f in ("id", "pos", "vel"):
                assert np.array_equal(d[f], st[f].astype(d[f].dtype), equal_nan=True), (k, s, f)
        if k == 0:
            # the moved children did meet their crowds, which do not see them
            dens = dict(zip(orc.get(1, "sorted_id").tolist(), orc.get(1, "dens").tolist()))
            alone = dens[int(ids[-1])]
            got = np.array([dens[int(i)] for i in ids[:crowds]])
            assert (got > 0.7 * alone * sizes).all(), (got / alone, sizes)
