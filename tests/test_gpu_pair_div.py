"""The square root, reciprocals and quotients of the force pairs in the exact arithmetic
(tss_device.cuh) against the IEEE operations, and the tether radius against its FP64
expression, bit for bit; whole steps on both sides of the pairs' operand ranges."""
import os
import subprocess

import numpy as np
import pytest

import oracle as O
from twoscalesplit_gb300 import _abi, build, scenes
from twoscalesplit_gb300.solver import Solver

pytestmark = pytest.mark.gpu
HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.parametrize("probe", ["div_pair", "tether"])
def test_equal_to_the_plain_expressions(tmp_path, probe):
    build.build()
    exe = str(tmp_path / probe)
    subprocess.check_call([build.nvcc(), *build.flags(), os.path.join(HERE, "cuda", probe + ".cu"), "-o", exe])
    out = subprocess.check_output([exe], timeout=300).decode()
    assert out.strip().splitlines()[-1].startswith("mismatches 0 of"), out


# radius, velocity scale, density scale, viscosity, distance of close pairs in radii
@pytest.mark.parametrize("r,v,rho,alpha,near", [
    (0.01, 1.0, 1e3, 0.05, 1e-3), (0.01, 1.0, 1e3, 0.0, 1e-6), (0.01, 0.0, 1e3, 0.05, 1e-3),
    (0.01, 1e-24, 1e3, 0.05, 1e-3), (0.01, 1e12, 1e3, 0.05, 1e-3), (0.01, 1.0, 1e-5, 0.05, 1e-3),
    (0.01, 1.0, 1e7, 0.05, 1e-3), (1e-6, 1.0, 1e3, 0.05, 1e-3), (64.0, 1.0, 1e3, 0.05, 1e-3)])
def test_pairs_in_and_out_of_range(r, v, rho, alpha, near):
    build.build()
    rng = np.random.default_rng(3)
    nx, ny = 20, 20
    n, dx = nx * ny, 0.5 * r
    p = scenes.particle_box(3 * r, 3 * r, dx, nx, ny).astype(np.float64) + rng.uniform(-0.2 * dx, 0.2 * dx, size=(n, 2))
    p[1::4] = p[::4] + near * r * rng.standard_normal((n // 4, 2))  # close pairs
    cfg = _abi.config_init(0.0, 0.0, 20 * r, 20 * r, r, 0.5 * r, rho, 100.0 * rho, 30.0, alpha, 0.08, 1e-9 * r)
    cfg.roi[:] = [1e9, 1e9, 2e9, 2e9]
    m = rho * dx * dx
    vel = (v * rng.standard_normal((n, 2))).astype(np.float32)
    sc = scenes.Scene("pairs", cfg, p.astype(np.float32), vel, m, m / 4, n, np.zeros((0, 2), np.float32), m / 4, 1, dx)
    hp = (p[:, None, :] + rng.uniform(-0.25 * dx, 0.25 * dx, size=(n, 1, 2))).reshape(-1, 2)
    high = {"id": np.arange(n, dtype=np.int32) * 4, "pos": hp.astype(np.float32), "vel": vel[::-1].copy(),
            "state": np.ones(n, np.uint8)}
    st = (np.arange(n) % 2).astype(np.uint8)
    ids = np.arange(n, dtype=np.int32)
    sol, orc = Solver.from_scene(sc), O.Oracle(sc, 32)
    for o, put in ((sol, lambda s, d: sol.upload(s, d)),
                   (orc, lambda s, d: orc.set_scale(s, d["id"], d["pos"], d["vel"], d["state"]))):
        put(0, {"id": ids, "pos": sc.low_pos, "vel": vel, "state": st})
        put(1, high)
        o.step()
    for s in (0, 1):
        for which, name in ((_abi.TSS_BUF_DENSITY, "dens"), (_abi.TSS_BUF_ACCEL, "acc")):
            assert np.array_equal(sol.copy(s, which), orc.get(s, name).astype(np.float32), equal_nan=True), (s, name)
