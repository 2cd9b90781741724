"""A small single scene steps the frames of a call but the last on one block of
the fused kernel: the same frames, lists, colours and statistics as one call per
frame, bit for bit, on both sides of the size rule and at every capacity."""
import dataclasses

import numpy as np
import pytest

from dyphur_b200 import scenes

pytestmark = pytest.mark.gpu

SCENES = {
    "one_body": lambda: scenes.stress_blocks(grid=(1, 1, 1)).scene(0),
    "nine": lambda: scenes.stress_blocks(grid=(2, 2, 2)),
    "column": lambda: scenes.stress_blocks(grid=(1, 31, 1)),
    "below": lambda: scenes.random_pile(126, seed=5),
    "at": lambda: scenes.random_pile(127, seed=5),
    "above": lambda: scenes.random_pile(128, seed=5),
    "dense": lambda: _dense(100),
}


def _dense(n):
    """Bodies crowded into a small box: more than 256 contacts, so that the
    reference order colours them."""
    s = scenes.random_pile(n, seed=8)
    s.pos[:n] = np.random.default_rng(8).uniform(0, 2.2, (n, 3)).astype(np.float32) + np.float32([0, 0.6, 0])
    return s


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def _same(a, b, frames):
    assert np.array_equal(bits(a.state()), bits(b.state()))
    assert a.stats() == b.stats()
    for x, y in zip(a.history(), b.history()):
        assert len(x) == frames and np.array_equal(x, y)
    assert np.array_equal(a.pairs(), b.pairs())
    (ab, pa), (bb, pb) = a.contacts(), b.contacts()
    assert np.array_equal(ab, bb) and np.array_equal(bits(pa), bits(pb))
    assert a.solver_stats() == b.solver_stats()
    ca, cb = a.colors(len(ab)), b.colors(len(ab))
    assert np.array_equal(ca[0], cb[0]) and ca[1] == cb[1]


@pytest.mark.parametrize("mode", [0, 1, 2, 3])
@pytest.mark.parametrize("name", list(SCENES))
def test_call_of_frames_equals_calls_per_frame(name, mode):
    from dyphur_b200 import device
    s = SCENES[name]()
    a, b, c = (device.World(s, mode=mode) for _ in range(3))
    for _ in range(40):
        a.step(1)
    b.step(2)
    b.step(38)
    c.capture_episode(40)
    c.run_episode()
    _same(a, b, 40)
    _same(a, c, 40)
    assert device.device_error() == 0


def test_more_frames_than_a_launch(oracle_mod):
    from dyphur_b200 import device
    s = SCENES["nine"]()
    w = device.World(s)
    w.step(300)
    o = oracle_mod.World(s)
    assert o.step(300) == 0
    assert np.array_equal(bits(w.state()), bits(o.state()))


@pytest.mark.parametrize("pairs,contacts", [(50, 4096), (4096, 40), (30, 20)])
def test_capacities(pairs, contacts):
    from dyphur_b200 import device
    s = dataclasses.replace(_dense(100), max_pairs=pairs, max_contacts=contacts)
    a, b = device.World(s), device.World(s)
    for _ in range(12):
        a.step(1)
    b.step(12)
    assert a.stats()["status"] != 0
    _same(a, b, 12)


def test_trajectory_records_every_frame():
    import torch
    from dyphur_b200 import device
    s = SCENES["nine"]()
    a, b = device.World(s), device.World(s)
    out = torch.zeros((20, s.n_bodies, 7)).pin_memory()
    b.set_trajectory(out, 1)
    b.step(20)
    torch.cuda.synchronize()
    for f in range(20):
        a.step(1)
        assert np.array_equal(bits(a.state()[:7].T), bits(out[f].numpy()))


def _alike(a, b):
    """Equal bits, or both a NaN (whose payload is not part of the contract)."""
    a, b = np.asarray(a, np.float32), np.asarray(b, np.float32)
    return np.array_equal(np.isnan(a), np.isnan(b)) and np.array_equal(bits(a)[~np.isnan(a)], bits(b)[~np.isnan(b)])


@pytest.mark.parametrize("rows,bodies", [([0], [50]), ([0], [-2]), ([1], [-1]), ([2, 0], [7, 8]), ([3], [-2]), ([6, 1], [20, -1]),
                                         ([0, 1, 2], [9, 9, 9])])
@pytest.mark.parametrize("n,start", [(8, 20), (99, 200), (127, 60), (200, 120)])
def test_nan_bodies_meet_what_the_tree_lets_them(oracle_mod, n, start, rows, bodies):
    """A NaN bound overlaps every other one that a walk of the tree brings it to: the
    oracle's pairs, from one call of frames as from a call per frame."""
    from dyphur_b200 import device
    s = scenes.random_pile(n, seed=5)
    o = oracle_mod.World(s)
    assert o.step(start) == 0
    st = o.state()
    st[rows, [b % s.n_bodies for b in bodies]] = np.nan
    a, b = device.World(s), device.World(s)
    for w in (a, b):
        w.bodies.set_state(st)
    o.set_state(st)
    o.step(1)
    a.step(1)
    assert np.array_equal(a.pairs(), o.pairs()[0]) and a.history()[0].tolist() == [o.pairs()[1]]
    for _ in range(3):
        a.step(1)
    b.step(4)
    for x, y in zip(a.history(), b.history()):
        assert np.array_equal(x, y)
    assert np.array_equal(a.pairs(), b.pairs()) and _alike(a.state(), b.state())
    assert device.device_error() == 0
