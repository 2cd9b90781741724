"""Ray walks over trees on both sides of the size rule, bit for bit against the
oracle's walk in leaf order: trees that fit the bodies, trees that bodies have
moved out of since, grazing and axis-parallel rays, capped and unbounded t_max,
and bodies and rays outside the fast walk's assumptions."""
import numpy as np
import pytest

from dyphur_b200 import scenes
from test_ray_sensor import _random_rays, bits

pytestmark = pytest.mark.gpu


def _rays(scene, pos, n, seed):
    rng = np.random.default_rng(seed)
    r = _random_rays(scene, n, seed)
    k = n // 4
    # from inside and next to bodies, grazing long ones, exact zeros, infinite and tiny spans
    j = rng.integers(0, scene.n_bodies, k)
    r[:k, :3] = pos[:, j].T + rng.normal(0, 0.3, (k, 3))
    r[:k, 3:6] = rng.normal(0, 1, (k, 3))
    r[k:k + 40, 3:6] *= 1e-3
    r[k + 40:k + 80, 3:6] *= 1e3
    r[k + 80:k + 120, 6] = np.inf
    r[k + 120:k + 130, 6] = 0.0
    r[k + 130:k + 140, 6] = -1.0
    r[k + 140:k + 150, 3] = 0.0
    r[k + 150:k + 155, 3:6] = 0.0
    r[k + 155:k + 158, 0] = np.nan
    r[k + 158:k + 160, 5] = np.inf
    r[k + 160:k + 200, :3] += 4000.0  # far away
    r[k + 160:k + 200, 3:6] = pos[:, j[:40]].T - r[k + 160:k + 200, :3]
    return r.astype(np.float32)


def _check(oracle_mod, scene, frames, moves, seed, n_rays=20000, before=None):
    """A tree built after `frames` frames (and `before`), bodies moved by `moves`, then cast."""
    from dyphur_b200 import device
    o = oracle_mod.World(scene)
    assert o.step(frames) == 0
    if before:
        st = o.state()
        before(st)
        o.set_state(st)
    o.stage(oracle_mod.STAGE_BROADPHASE)
    b, sh = device.DeviceBodies(scene), device.DeviceShapes(scene)
    b.set_state(o.state())
    bp = device.Broadphase(scene.n_bodies, scene.max_pairs)
    bp.build_and_query(b, sh, scene.bounds[0])
    st = o.state()
    moves(st)
    o.set_state(st)
    b.set_state(st)
    rays = _rays(scene, st[:3], n_rays, seed)
    want_t, want_b = o.ray_query(rays)
    t, body = device.ray_query(bp.bvh_view(scene.n_bodies), b, sh, rays)
    t, body = t.cpu().numpy(), body.cpu().numpy().view(np.uint32)
    bad = np.flatnonzero((body != want_b) | ((bits(t) != bits(want_t)) & ~(np.isnan(t) & np.isnan(want_t))))
    assert bad.size == 0, (bad[:5], rays[bad[:5]], t[bad[:5]], want_t[bad[:5]], body[bad[:5]], want_b[bad[:5]])
    assert device.device_error() == 0


def _still(st):
    pass


def _shift(amount):
    def f(st):
        rng = np.random.default_rng(1)
        st[:3] += rng.normal(0, amount, st[:3].shape).astype(np.float32)
    return f


def _bad_quaternion(st):
    st[3:7, 3] *= 1.3


def _nan_body(st):
    st[1, 5] = np.nan


def _burst(st):
    """Bodies across and beyond the range of the boxes' 16-bit bounds, on one or more axes."""
    rng = np.random.default_rng(2)
    far = rng.choice(np.arange(1, st.shape[1]), 240, replace=False)
    size = np.repeat([3e4, 65500.0, 65519.7, 7e4, 1e8, 1e20], 40).astype(np.float32)
    axes = rng.random((3, 240)) < 0.5
    axes[0] |= ~axes.any(0)
    st[:3, far] = np.where(axes, size * rng.choice([-1, 1], (3, 240)), st[:3, far]).astype(np.float32)


@pytest.mark.parametrize("n", [1, 2, 300, 16382, 16383, 20000])
@pytest.mark.parametrize("frames", [0, 30])
def test_walks_match_oracle(oracle_mod, n, frames):
    _check(oracle_mod, scenes.random_pile(n, seed=n), frames, _still, n)


@pytest.mark.parametrize("moves", [_shift(0.02), _shift(0.5), _bad_quaternion, _nan_body],
                         ids=["small", "large", "quaternion", "nan"])
def test_bodies_outside_their_boxes(oracle_mod, moves):
    _check(oracle_mod, scenes.random_pile(17000, seed=4), 30, moves, 5)


@pytest.mark.parametrize("moves", [_still, _shift(0.02), _shift(300.0)], ids=["still", "small", "huge"])
def test_bodies_past_the_bounds(oracle_mod, moves):
    _check(oracle_mod, scenes.random_pile(17000, seed=7), 30, moves, 8, before=_burst)


def test_box_stack(oracle_mod):
    """Touching boxes with equal distances: ties go to the earlier leaf."""
    _check(oracle_mod, scenes.stress_blocks(spacing=0.8, jitter=0.0, grid=(26, 26, 26)), 0, _still, 6)


@pytest.mark.parametrize("n", [300, 17000])
def test_captured_query(n):
    """A query recorded in a CUDA graph replays on new rays."""
    import torch
    from dyphur_b200 import device
    s = scenes.random_pile(n, seed=2)
    b, sh = device.DeviceBodies(s), device.DeviceShapes(s)
    bp = device.Broadphase(s.n_bodies, s.max_pairs)
    bp.build_and_query(b, sh, s.bounds[0])
    view = bp.bvh_view(s.n_bodies)
    first, second = (torch.from_numpy(_random_rays(s, 4096, k)).cuda() for k in (1, 2))
    want = [device.ray_query(view, b, sh, r) for r in (first, second)]
    rays = first.clone()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        t, body = device.ray_query(view, b, sh, rays)
    for r, (wt, wb) in zip((first, second), want):
        rays.copy_(r)
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(t.view(torch.int32), wt.view(torch.int32)) and torch.equal(body, wb)


@pytest.mark.parametrize("n_rays", [1, 7, 8, 9, 4000])
def test_few_and_short_rays(oracle_mod, n_rays):
    """On both sides of the rules on the number of rays (8 at this size) and on a ray's
    length, which is the same whether the direction or t_max carries it."""
    from dyphur_b200 import device
    scene = scenes.random_pile(16400, seed=3)
    o = oracle_mod.World(scene)
    assert o.step(20) == 0
    st = o.state()
    o.stage(oracle_mod.STAGE_BROADPHASE)
    b, sh = device.DeviceBodies(scene), device.DeviceShapes(scene)
    b.set_state(st)
    bp = device.Broadphase(scene.n_bodies, scene.max_pairs)
    bp.build_and_query(b, sh, scene.bounds[0])
    half = scene.shape_half[scene.shape]
    size = np.where(scene.shape_type[scene.shape] == 1, 3 * half[:, 0], half.sum(1)).mean()
    rng = np.random.default_rng(n_rays)
    d = rng.normal(size=(n_rays, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    length = 16 * size * rng.choice([0.1, 0.5, 0.999, 1.0, 1.001, 2.0, 30.0], n_rays)
    t_max = rng.choice([1e-3, 1.0, 50.0], n_rays)
    at = st[:3, rng.integers(0, scene.n_bodies, n_rays)].T
    rays = np.empty((n_rays, 7), np.float32)
    rays[:, 3:6] = d * (length / t_max)[:, None]
    rays[:, :3] = at - d * (length * rng.uniform(0, 1, n_rays))[:, None]
    rays[:, 6] = t_max
    want_t, want_b = o.ray_query(rays)
    t, body = device.ray_query(bp.bvh_view(scene.n_bodies), b, sh, rays)
    assert np.array_equal(bits(t.cpu().numpy()), bits(want_t))
    assert np.array_equal(body.cpu().numpy().view(np.uint32), want_b)
    assert (want_b != 0xFFFFFFFF).any()
    assert device.device_error() == 0
