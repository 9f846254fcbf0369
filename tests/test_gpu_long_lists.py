"""The gathers' one-thread form (more than 12,000 particles of a scale for the densities,
more than 48,000 for the forces) where its neighbour lists can go wrong: lists just
full, one over and many times over, entries further than a 16-bit offset away, rows of
more than 32,768 candidates, and every state.  Every result must equal the FP32
oracle's bit for bit."""
import numpy as np
import pytest

from test_gpu_density_search import _check, _clusters, _scene
from twoscalesplit_gb300 import scenes

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", autouse=True)
def _built():
    from twoscalesplit_gb300 import build
    build.build()


def _fill(p, n, r, y0):
    """p and points without neighbours above y0 (80 a row), n in all."""
    k = np.arange(max(n - len(p), 0))
    return np.concatenate([p, np.stack([0.5 * r + 1.01 * r * (k % 80), y0 + 1.01 * r * (k // 80)], axis=1)])


# both scales' lists from 22 neighbours to 30, and up to twelve times a list's length
@pytest.mark.parametrize("n", [12001, 48001])
@pytest.mark.parametrize("m", [2, 3, 23, 24, 25, 26, 27, 28, 29, 30, 31, 49, 50, 51, 52, 75, 76, 300])
def test_lists_up_to_and_past_their_length(m, n):
    rng = np.random.default_rng(m)
    r = 0.01
    low = _fill(_clusters(m, r, rng), n, r, 0.55)
    size = (0.85, float(low[:, 1].max()) + 0.05)
    _check(_scene(low, r, size))
    # the same as high-res particles; every third in state 0, so that both masks are met
    high = _fill(_clusters(m, 0.5 * r, rng), n, 0.5 * r, 0.3)
    k = len(high)
    sc = _scene(np.stack([0.6 + 0.1 * rng.uniform(size=k), rng.uniform(size=k)], axis=1), r, (0.85, 1.6 * size[1]))
    _check(sc, {"id": rng.permutation(4 * k)[:k].astype(np.int32), "pos": high.astype(np.float32),
                "vel": rng.standard_normal((k, 2)).astype(np.float32), "state": (np.arange(k) % 3 != 0).astype(np.uint8)},
           np.ones(k, np.uint8))


@pytest.mark.parametrize("m", [4, 6, 26, 40])
def test_crowds_in_rows_past_a_16_bit_offset(m):
    # 6,000 cells a row with m particles at each cell corner: neighbouring rows of cells
    # are 6,000 m entries apart
    r = 1.0 / 6000
    rng = np.random.default_rng(m)
    c = np.stack(np.meshgrid(np.arange(1, 6000), np.arange(1, 3)), axis=-1).reshape(-1, 1, 2) * r
    p = (c + rng.uniform(-0.2 * r, 0.2 * r, size=(len(c), m, 2))).reshape(-1, 2)
    sc = _scene(p, r, (1.0, 4 * r))
    sc.config.dt = 1e-12  # the crowds stay together for the second step
    _check(sc)


def test_rows_of_more_candidates_than_16_bits():
    # particles beside the grid are all in its border cells: 40,000 candidates, few of
    # them near, and near ones far apart in the list
    rng = np.random.default_rng(9)
    r, n = 0.01, 40000
    beside = np.stack([-0.4 * r * (1 + rng.permutation(n)), 0.25 + rng.uniform(-0.3 * r, 0.3 * r, n)], axis=1)
    _check(_scene(_fill(beside, 48100, r, 0.5), r, (0.85, 1.6)))


@pytest.mark.parametrize("low_states,high_states", [([0, 1], [1]), ([0, 1, 2], [1]), ([0, 1, 2, 3], [0, 1, 2, 3])])
def test_masks_of_every_state(low_states, high_states):
    rng = np.random.default_rng(8)
    r, nx = 0.002, 222
    n = nx * nx
    p = scenes.particle_box(0.1, 0.1, 0.5 * r, nx, nx) + rng.uniform(-0.1 * r, 0.1 * r, size=(n, 2))
    sc = _scene(p, r, (0.6, 0.6))
    hp = scenes.particle_box(0.15, 0.15, 0.25 * r, nx, nx) + rng.uniform(-0.05 * r, 0.05 * r, size=(n, 2))
    high = {"id": rng.permutation(4 * n)[:n].astype(np.int32), "pos": hp.astype(np.float32),
            "vel": rng.standard_normal((n, 2)).astype(np.float32), "state": rng.choice(high_states, n).astype(np.uint8)}
    _check(sc, high, rng.choice(low_states, n).astype(np.uint8))
