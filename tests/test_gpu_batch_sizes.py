"""Batches whose shared lists are about as long as the sizes where the kernels change
from groups of lanes to a thread per particle.  A batch's slots are rounded up to whole
pages per scene and its scenes can be retired, so its capacity says nothing about the
side its lists are on.  Every scene must equal the same scene alone, bit for bit."""
import ctypes

import numpy as np
import pytest

from twoscalesplit_gb300 import _abi, scenes
from twoscalesplit_gb300.serving import Pool, footprint, pool_config, scene_desc
from twoscalesplit_gb300.solver import Batch, Solver

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from twoscalesplit_gb300 import build
    build.build()


def _scene(n, seed):
    """n particles standing on the walls, some of them in the region of interest."""
    nx = max(int(np.sqrt(0.5 * n)), 1)
    sc = scenes.dam_break_small(nx, -(-n // nx), seed=seed, relax_iters=0, roi=[-1.0, -1.0, 0.06, 0.1])
    rng = np.random.default_rng(seed)
    sc.low_pos = (sc.low_pos[:n] + rng.uniform(-0.1 * sc.dx, 0.1 * sc.dx, size=(n, 2))).astype(np.float32)
    sc.low_vel = rng.standard_normal((n, 2)).astype(np.float32)
    return sc


def _same(batch, k, alone):
    for scale in (0, 1):
        mine, theirs = alone.download(scale), batch.download_scene(k, scale)
        assert np.array_equal(mine["id"], theirs["id"]), (k, scale)
        for name in ("pos", "vel", "state", "dens"):
            assert np.array_equal(mine[name], theirs[name]), (k, scale, name)


@pytest.mark.parametrize("sizes", [[47900], [4750] * 10, [900] * 48, [5000, 7000], [5001, 7000], [9000, 11000],
                                   [9001, 11000], [23000, 25000], [23001, 25000]])
def test_batch_equals_scenes_alone(sizes):
    scs = [_scene(n, k) for k, n in enumerate(sizes)]
    batch = Batch(scs)
    alone = [Solver.from_scene(sc) for sc in scs]
    for _ in range(3):
        batch.step(1)
        for a in alone:
            a.step(1)
    assert batch.scene_counts()[1].sum() > 0
    for k, a in enumerate(alone):
        _same(batch, k, a)


# 49,000 particles, then 42,000, then 49,000 again; and either side of the 150,000 entries
# where the grid build changes (a list is longer than what is left of it after a scene left)
@pytest.mark.parametrize("count,n", [(7, 7000), (3, 52000)])
@pytest.mark.parametrize("kind", ["batch", "pool"])
def test_scenes_leave_and_come_back(kind, count, n):
    scs = [_scene(n, k) for k in range(count)]
    alone = [Solver.from_scene(sc) for sc in scs]
    if kind == "batch":
        b = Batch(scs)
        slot = list(range(count))
    else:
        need = {k: count * footprint(scs[0])[k] for k in footprint(scs[0])}
        b = Pool(pool_config(need["low_slots"], need["high_particles"], need["low_cells"], need["high_cells"],
                             need["wall_particles"], max_scenes=count))
        slot = [b.admit(sc) for sc in scs]

    def check(live):
        for k in live:
            _same(b, slot[k], alone[k])

    def step(live):
        b.step(2)
        for k in live:
            alone[k].step(2)
        check(live)

    step(range(count))
    assert b.lib.tss_pool_retire(b.h, slot[2], None) == _abi.TSS_OK
    rest = [k for k in range(count) if k != 2]
    step(rest)
    alone[2] = Solver.from_scene(scs[2])
    desc, sid = scene_desc(scs[2], []), ctypes.c_int(-1)
    assert b.lib.tss_pool_admit(b.h, ctypes.byref(desc), None, ctypes.byref(sid)) == _abi.TSS_OK
    slot[2] = sid.value
    step(range(count))
