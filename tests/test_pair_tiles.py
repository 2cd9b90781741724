"""The single-scene broadphase at the edges of its tiles: 32 leaves to a search
tile, 64 bodies to a block of the pair writer, 1024 leaves to a block of the tree
build, 128 partners to a bucket, with wide, static, coincident and non-finite
bodies, against the oracle's pairs and tree."""
import numpy as np
import pytest

from dyphur_b200 import scenes
from test_oracle_pins import _single_scene

pytestmark = pytest.mark.gpu


def _cloud(n, kind, seed):
    """n boxes and spheres in a cube with about ten partners each."""
    rng = np.random.default_rng(seed)
    side = max(2.0, 0.9 * n ** (1 / 3))
    pos = rng.uniform(0, side, (n, 3))
    shape = rng.integers(0, 3, n)
    mass = np.ones(n)
    if kind == "wide":  # several bodies longer than the scene is wide, first, last and in between
        shape[rng.integers(0, n, max(1, n // 40))] = 3
        shape[[0, n - 1]] = 3
    if kind == "static":  # every third body static
        mass[::3] = 0
    if kind == "heap":  # coincident centres: equal Morton codes, long buckets
        pos[: n // 2] = pos[0] + 0.02 * rng.normal(size=(n // 2, 3))
    if kind == "line":
        pos[:, 1:] = 0.5
        pos[:, 0] = np.linspace(0, 0.4 * n, n)
    shapes = [(0, 0.5, 0.4, 0.3), (1, 0.45, 0.45, 0.45), (0, 0.2, 0.7, 0.2), (0, side, 0.3, side)]
    s = _single_scene(shape, pos.astype(np.float32), shapes, mass, (mass == 0).astype(np.uint32))
    q = rng.normal(size=(n, 4)).astype(np.float32)
    s.rot = q / np.linalg.norm(q, axis=1, keepdims=True)
    hi = max(side, float(pos.max())) + 3
    s.bounds = np.array([[-3, -3, -3, hi, hi, hi]], np.float32)
    s.max_pairs, s.max_contacts = 300 * n + 64, 16 * n + 64
    return s


def _compare(oracle_mod, s, tree=True):
    from dyphur_b200 import device
    o = oracle_mod.World(s)
    o.stage(oracle_mod.STAGE_BROADPHASE)
    want, n_want = o.pairs()
    b, sh = device.DeviceBodies(s), device.DeviceShapes(s)
    bp = device.Broadphase(s.n_bodies, s.max_pairs)
    for _ in range(2):  # counters are left as they were found
        bp.build_and_query(b, sh, s.bounds[0])
    assert bp.download_count() == n_want
    assert np.array_equal(bp.pairs(), want[: s.max_pairs])
    if tree:
        got, ref = bp.bvh(s.n_bodies), o.bvh()
        for k in ("sorted_idx", "left", "right", "parent", "aabb"):
            assert np.array_equal(got[k], ref[k]), k
    assert device.device_error() == 0


@pytest.mark.parametrize("kind", ["plain", "wide", "static", "heap", "line"])
@pytest.mark.parametrize("n", [2, 3, 31, 32, 33, 63, 64, 65, 255, 257, 1023, 1024, 1025, 2049, 5000])
def test_pairs_and_tree_match_oracle(oracle_mod, n, kind):
    _compare(oracle_mod, _cloud(n, kind, n))


@pytest.mark.parametrize("n", [40, 300])
def test_pair_capacity_keeps_the_sorted_prefix(oracle_mod, n):
    s = _cloud(n, "heap", 3)
    s.max_pairs = 101
    _compare(oracle_mod, s, tree=False)


@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf, 7e4])
def test_non_finite_bodies(oracle_mod, value):
    """A NaN bound overlaps whatever its ancestors let it meet; infinite and
    past-fp16 positions have infinite bounds."""
    s = _cloud(200, "plain", 9)
    s.pos[[5, 77], [0, 2]] = value
    _compare(oracle_mod, s, tree=False)


@pytest.mark.parametrize("n", [20, 70, 300])
def test_unbounded_bodies(oracle_mod, n):
    """Half extents past fp16: boxes without bounds overlap every other one."""
    s = _cloud(n, "plain", 4)
    s.shape_half = np.concatenate([s.shape_half, np.full((1, 3), 1e6, np.float32)])
    s.shape_type = np.append(s.shape_type, np.uint32(0))
    s.shape_offset = np.array([0, len(s.shape_type)], np.uint32)
    s.shape[[0, n // 2]] = len(s.shape_type) - 1
    _compare(oracle_mod, s, tree=False)


def test_nan_bodies_and_long_buckets(oracle_mod):
    """A body with more partners than its bucket holds, next to NaN bodies and
    static ones: the later leaf of each two looks for the other."""
    for seed in range(6):
        s = _cloud(400, "heap", seed)
        rng = np.random.default_rng(seed)
        s.mass[rng.integers(0, 400, 40)] = 0
        s.pos[rng.integers(0, 400, 3), rng.integers(0, 3, 3)] = np.nan
        s.rot[rng.integers(0, 400), 1] = np.nan
        _compare(oracle_mod, s, tree=False)
