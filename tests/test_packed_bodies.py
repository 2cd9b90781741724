"""Narrowphase contacts on both sides of the size from which bodies are packed,
bit for bit against the oracle, with one handle used for growing scenes and a
graph recorded before it grew."""
import numpy as np
import pytest

from dyphur_b200 import scenes
from test_ray_sensor import bits

pytestmark = pytest.mark.gpu


def _want(oracle_mod, scene, frames):
    o = oracle_mod.World(scene)
    assert o.step(frames) == 0
    st = o.state()
    o.stage(oracle_mod.STAGE_BROADPHASE)
    o.stage(oracle_mod.STAGE_NARROWPHASE)
    return st, o.contacts()


@pytest.mark.parametrize("n", [8191, 8192, 8193])
def test_contacts_match_oracle(oracle_mod, n):
    from dyphur_b200 import device
    s = scenes.random_pile(n - 1, seed=n)  # and the ground
    assert s.n_bodies == n
    st, (ab, p7) = _want(oracle_mod, s, 45)
    b, sh = device.DeviceBodies(s), device.DeviceShapes(s)
    b.set_state(st)
    bp, npz = device.Broadphase(n, s.max_pairs), device.Narrowphase(s.max_contacts)
    bp.build_and_query(b, sh, s.bounds[0])
    npz.run(bp, b, sh)
    got_ab, got_p7 = npz.contacts()
    assert len(ab) > 100
    assert np.array_equal(got_ab, ab) and np.array_equal(bits(got_p7), bits(p7))
    assert device.device_error() == 0


@pytest.mark.parametrize("n", [32767, 32768, 32769])
def test_contacts_match_oracle_at_the_line(oracle_mod, n):
    from dyphur_b200 import device
    s = scenes.random_pile(n - 1, seed=n)  # and the ground
    w = device.World(s)
    w.step(45)
    st = w.state()
    o = oracle_mod.World(s)
    o.set_state(st)
    o.stage(oracle_mod.STAGE_BROADPHASE)
    o.stage(oracle_mod.STAGE_NARROWPHASE)
    ab, p7 = o.contacts()
    bp, npz = device.Broadphase(n, s.max_pairs), device.Narrowphase(s.max_contacts)
    bp.build_and_query(w.bodies, w.shapes, s.bounds[0])
    npz.run(bp, w.bodies, w.shapes)
    got_ab, got_p7 = npz.contacts()
    assert len(ab) > 1000
    assert np.array_equal(got_ab, ab) and np.array_equal(bits(got_p7), bits(p7))
    assert device.device_error() == 0


@pytest.mark.parametrize("sizes", [(8200, 9000), (33000, 36000)])
def test_one_handle_grows(sizes):
    import torch
    from dyphur_b200 import device
    parts = []
    for n in sizes:
        s = scenes.random_pile(n, seed=n)
        w = device.World(s)
        w.step(45)
        b, sh, bp = w.bodies, w.shapes, device.Broadphase(s.n_bodies, 400000)
        bp.build_and_query(b, sh, s.bounds[0])
        parts.append((s, w, b, sh, bp))
    (_, _, b0, sh0, bp0), (_, _, b1, sh1, bp1) = parts
    contacts = max(p[0].max_contacts for p in parts)
    other, npz = device.Narrowphase(contacts), device.Narrowphase(contacts)
    other.run(bp1, b1, sh1)
    large = other.contacts()
    npz.run(bp0, b0, sh0)
    small = npz.contacts()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        npz.run(bp0, b0, sh0)
    npz.run(bp1, b1, sh1)
    got = npz.contacts()
    assert np.array_equal(got[0], large[0]) and np.array_equal(bits(got[1]), bits(large[1]))
    for _ in range(2):
        g.replay()
        torch.cuda.synchronize()
        got = npz.contacts()
        assert np.array_equal(got[0], small[0]) and np.array_equal(bits(got[1]), bits(small[1]))
    assert device.device_error() == 0
