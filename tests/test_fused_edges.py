"""The fused batched frame at the sizes where its tiles end: scenes of N bodies
resting apart on a ground, so that one level of the solve holds N contacts, with
the ground before or after them (the static body first or second in each pair),
and next to one another (chains of levels). Every scene bit for bit against the
oracle's run of that scene alone, on every kind of team."""
import numpy as np
import pytest

from dyphur_b200 import scenes
from test_batch import concat_scenes
from test_oracle_pins import _single_scene

pytestmark = pytest.mark.gpu

SIZES = (1, 2, 15, 16, 17, 31, 32, 33, 63, 64, 65, 95, 96, 97, 127, 128, 129, 160)


def _bed(n, ground_first, spacing, seed):
    """n spheres and boxes in a row-major bed on a ground, pressed in by 0.01."""
    rng = np.random.default_rng(seed)
    k = int(np.ceil(np.sqrt(n)))
    i = np.arange(n)
    half = 0.5 + 0.5 * k * spacing
    pos = np.stack([(i % k - k / 2) * spacing, np.full(n, 0.5 + 0.4 - 0.01), (i // k - k / 2) * spacing], 1)
    pos[:, 1] += rng.uniform(0, 0.005, n)
    kind, mass, flags = (i % 2).tolist(), [1.0] * n, [0] * n
    pos = pos.tolist()
    ground = ([2], [[0.0, 0.0, 0.0]], [0.0], [1])
    if ground_first:
        kind, pos, mass, flags = ground[0] + kind, ground[1] + pos, ground[2] + mass, ground[3] + flags
    else:
        kind, pos, mass, flags = kind + ground[0], pos + ground[1], mass + ground[2], flags + ground[3]
    s = _single_scene(kind, pos, [(0, 0.4, 0.4, 0.4), (1, 0.4, 0.4, 0.4), (0, half + 2, 0.5, half + 2)], mass, flags)
    dyn = np.asarray(mass) > 0
    s.vel[dyn] = rng.normal(0, 0.5, (n, 3))
    s.ang[dyn] = rng.normal(0, 0.5, (n, 3))
    s.inertia = np.tile(np.diag([0.1, 0.12, 0.09]).astype(np.float32).reshape(9), (n + 1, 1))
    b = half + 5
    s.bounds = np.array([[-b, -5, -b, b, 10, b]], np.float32)
    s.max_pairs, s.max_contacts = 48 * (n + 1) + 64, 16 * (n + 1) + 64
    s.vel, s.ang = s.vel.astype(np.float32), s.ang.astype(np.float32)
    return s


@pytest.mark.parametrize("mode", [1, 2])
@pytest.mark.parametrize("spacing", [1.2, 0.79])
@pytest.mark.parametrize("ground_first", [False, True])
def test_scene_sizes_match_oracle(oracle_mod, mode, spacing, ground_first):
    from dyphur_b200 import device
    parts = [_bed(n, ground_first, spacing, n) for n in SIZES]
    want = []
    for p in parts:
        o = oracle_mod.World(p)
        assert o.step(6, oracle_mod.SOLVER_SERIAL if mode == 1 else mode) == 0
        want.append(o.state())
    want = np.concatenate(want, 1)
    s = concat_scenes(parts)
    teams = set()
    for cfg in (None, (0, 0, 4), (60 << 10, 1, 4), (60 << 10, 2, 5), (1, 2, 6)):
        w = device.World(s, mode=mode)
        if cfg:
            w.set_fused_config(*cfg)
        c = w.fused_config()
        teams.add((c["warp_scenes"] > 0, c["half_scenes"] > 0, c["block_scenes"] > 0))
        w.step(6)
        assert w.stats()["status"] == 0 and device.device_error() == 0
        got = w.state()
        bad = np.flatnonzero((got.view(np.uint32) != want.view(np.uint32)).any(0))
        assert bad.size == 0, (cfg, np.unique(np.searchsorted(s.body_offset, bad, side="right") - 1))
    assert len(teams) >= 2
