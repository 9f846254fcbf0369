"""Scenes whose particles have more neighbours than a list holds cost what their pairs
cost: a support of 3 lattice spacings has 2.25 times the candidates and neighbours of
one of 2 spacings, and no stage may take more than twice that factor longer."""
import math

import numpy as np
import pytest

from twoscalesplit_gb300 import scenes
from twoscalesplit_gb300._abi import config_init
from twoscalesplit_gb300.solver import Solver

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from twoscalesplit_gb300 import build
    build.build()


def _stage_ms(spacings, stage, arith):
    nx, dx = 800, 1.0 / 800
    r = spacings * dx
    low = scenes.particle_box(0.5 * dx, 0.5 * dx, dx, nx, nx).astype(np.float32)
    low += np.random.default_rng(1).uniform(-0.05 * dx, 0.05 * dx, size=low.shape).astype(np.float32)
    cfg = config_init(0.0, 0.0, 1.0, 1.0, r, 0.5 * r, scenes.REST_DENSITY, scenes.TAIT_B, scenes.SPEED_SOUND,
                      scenes.ALPHA, scenes.SIGMA, 1e-9)
    cfg.roi[:] = [math.inf] * 4
    mass = scenes.REST_DENSITY / scenes.lattice_pair_kernel_sum(dx, r, 0.5 * r)
    sol = Solver.from_scene(scenes.Scene("lattice", cfg, low, np.zeros_like(low), mass, mass / 4, 4,
                                         np.zeros((0, 2), np.float32), mass / 4, 1, dx))
    sol.set_arith(arith)
    sol.profile(True)
    sol.step(5)
    t = []
    for _ in range(9):
        sol.step(1)
        sol.sync()
        t.append(sol.stage_times()[stage])
    return float(np.median(t))


@pytest.mark.parametrize("arith", ["exact", "fast"])
@pytest.mark.parametrize("stage", ["density_low", "force_low"])
def test_time_grows_with_the_pairs(stage, arith):
    assert _stage_ms(3.0, stage, arith) < 2 * 2.25 * _stage_ms(2.0, stage, arith)
