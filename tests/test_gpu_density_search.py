"""The density passes' two phases (search into a list, then the terms) at the sizes
where the list can go wrong: empty and one-entry lists, lists that are just full or
one over, clusters far over, and rows whose entries lie further than a 16-bit offset
from the particle.  Every result must equal the FP32 oracle's bit for bit."""
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


def _scene(low, r, size):
    cfg = config_init(0.0, 0.0, size[0], size[1], r, 0.5 * r, scenes.REST_DENSITY, scenes.TAIT_B,
                      scenes.SPEED_SOUND, scenes.ALPHA, scenes.SIGMA, 1e-6)
    cfg.roi[:] = [math.inf, math.inf, math.inf, math.inf]
    low = low.astype(np.float32)
    m = scenes.REST_DENSITY * (r / 2) ** 2
    return scenes.Scene("clusters", cfg, low, np.zeros_like(low), m, m / 4, 4 * len(low), np.zeros((0, 2), np.float32),
                        m / 4, 1, r / 2)


def _check(sc, high=None, state=None):
    sol, orc = Solver.from_scene(sc), O.Oracle(sc, 32)
    n = sc.n_low
    ids = np.arange(n, dtype=np.int32)
    if high is not None:
        sol.upload(0, {"id": ids, "pos": sc.low_pos, "vel": sc.low_vel, "state": state})
        sol.upload(1, high)
        orc.set_scale(0, ids, sc.low_pos, sc.low_vel, state)
        orc.set_scale(1, high["id"], high["pos"], high["vel"], high["state"])
    for _ in range(2):
        sol.step(1)
        orc.step()
        for s in (0, 1):
            assert np.array_equal(sol.copy(s, _abi.TSS_BUF_SORTED_ID), orc.get(s, "sorted_id")), s
            for which, name in ((_abi.TSS_BUF_DENSITY, "dens"), (_abi.TSS_BUF_ACCEL, "acc")):
                assert np.array_equal(sol.copy(s, which), orc.get(s, name).astype(np.float32)), (s, name)


def _clusters(m, r, rng):
    """m points within a neighbour distance of one another, 40 times, far apart; the
    clusters straddle cell corners, so a list spans several rows of its window."""
    c = np.stack(np.meshgrid(np.arange(1, 9), np.arange(1, 6)), axis=-1).reshape(-1, 1, 2) * (8 * r)
    return (c + rng.uniform(-0.3 * r, 0.3 * r, size=(40, m, 2))).reshape(-1, 2)


@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 19, 20, 21, 22, 23, 25, 26, 27, 28, 29, 33, 70])
def test_lists_up_to_and_past_their_length(m):
    rng = np.random.default_rng(m)
    r = 0.01
    low = _clusters(m, r, rng)
    _check(_scene(low, r, (0.8, 0.5)))
    # the same as high-res particles; every third in state 0, so that both masks are met
    n = 40 * m
    sc = _scene(rng.uniform(0.3, 0.31, size=(n, 2)) * [1, 1], r, (0.8, 0.5))
    high = {"id": np.arange(n, dtype=np.int32) * 4, "pos": _clusters(m, 0.5 * r, rng).astype(np.float32),
            "vel": np.zeros((n, 2), np.float32), "state": (np.arange(n) % 3 != 0).astype(np.uint8)}
    _check(sc, high, np.ones(n, np.uint8))


def test_rows_past_a_16_bit_offset():
    # 20,000 cells a row, two particles wide and two high: neighbouring rows of cells
    # are 80,000 entries apart
    nx, ny, dx = 40000, 6, 1.0 / 40000
    rng = np.random.default_rng(5)
    p = scenes.particle_box(0.5 * dx, 0.5 * dx, dx, nx, ny) + rng.uniform(-0.05 * dx, 0.05 * dx, size=(nx * ny, 2))
    sc = _scene(p, 2 * dx, (1.0, 8 * dx))
    _check(sc)


@pytest.mark.parametrize("low_states,high_states", [([0, 1], [1]), ([0, 1, 2], [1]), ([0, 1, 2, 3], [0, 1, 2, 3])])
def test_masks_of_every_state(low_states, high_states):
    # the force passes read a neighbour's state only when a mask can reject it
    rng = np.random.default_rng(8)
    r, n = 0.02, 900
    p = scenes.particle_box(0.1, 0.1, 0.5 * r, 30, 30) + rng.uniform(-0.1 * r, 0.1 * r, size=(n, 2))
    sc = _scene(p, r, (0.6, 0.6))
    hp = scenes.particle_box(0.15, 0.15, 0.25 * r, 40, 40) + rng.uniform(-0.05 * r, 0.05 * r, size=(1600, 2))
    high = {"id": rng.permutation(3600)[:1600].astype(np.int32), "pos": hp.astype(np.float32),
            "vel": rng.standard_normal((1600, 2)).astype(np.float32), "state": rng.choice(high_states, 1600).astype(np.uint8)}
    _check(sc, high, rng.choice(low_states, n).astype(np.uint8))
