"""Fused batches step all frames of a call in one launch: the same frames, lists,
statistics, trajectory rows and checkpoints as one call per frame, bit for bit."""
import numpy as np
import pytest

from dyphur_b200 import scenes

pytestmark = pytest.mark.gpu


def _world(mode=1, n_scenes=7):
    from dyphur_b200 import device
    return device.World(scenes.batch(n_scenes, 5, 40, seed=12), mode=mode)


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("frames", [2, 31, 257])
def test_one_call_equals_a_call_per_frame(mode, frames):
    a, b = _world(mode), _world(mode)
    for _ in range(frames):
        a.step(1)
    b.step(frames)
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


# records per buffer (8) reached in the middle, at the end and never; a short
# host buffer; a record interval that does not divide the frames
@pytest.mark.parametrize("every,records,frames", [(1, 40, 37), (2, 11, 40), (3, 9, 25), (7, 2, 30), (50, 3, 20)])
@pytest.mark.parametrize("captured", [False, True])
def test_trajectory_rows_of_a_run(every, records, frames, captured):
    import torch
    a, b = _world(), _world()
    n = a.bodies.n
    want = np.zeros((records, n, 7), np.float32)
    for f in range(frames):
        a.step(1)
        if f % every == 0 and f // every < records:
            want[f // every] = a.state()[:7].T
    out = torch.zeros((records, n, 7)).pin_memory()
    b.set_trajectory(out, every)
    if captured:
        b.capture_episode(frames)
        b.run_episode()
    else:  # split over calls, so that frame numbers carry on
        b.step(frames // 3)
        b.step(frames - frames // 3)
    torch.cuda.synchronize()
    assert np.array_equal(bits(out.numpy()), bits(want))
    assert np.array_equal(bits(a.state()), bits(b.state()))


@pytest.mark.parametrize("frames,every", [(1, 1), (12, 1), (13, 5), (300, 128)])
def test_rollout_checkpoints_of_a_run(frames, every):
    import torch
    a, b = _world(), _world()
    n = a.bodies.n
    want = []
    for f in range(frames):
        if f % every == 0:
            want.append(a.state())
        a.step(1)
    ckpt = torch.full(((frames + every - 1) // every, 13, n), float("nan"), device="cuda")
    b.rollout_raw(frames, every, ckpt.data_ptr(), torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    assert np.array_equal(bits(ckpt.cpu().numpy()), bits(np.stack(want)))
    assert np.array_equal(bits(a.state()), bits(b.state()))


def _crowds():
    """Scene 0: 30 fixed spheres in one place, 435 pairs and contacts in every frame.
    Scene 1: 37 of them, and two that arrive after some frames, past its 688 contacts."""
    from test_batch import concat_scenes
    from test_oracle_pins import _single_scene
    parts = []
    for fixed, moving in ((30, 0), (37, 2)):
        n = fixed + moving
        pos = np.zeros((n, 3), np.float32)
        pos[fixed:, 0] = [1.4, -1.4][:moving]
        mass = np.r_[np.zeros(fixed), np.ones(moving)]
        s = _single_scene([0] * n, pos.tolist(), [(1, 0.5, 0.5, 0.5)], mass.tolist(), (mass == 0).astype(int).tolist())
        s.vel[fixed:, 0] = [-9.0, 9.0][:moving]
        s.bounds = np.array([[-9, -9, -9, 9, 9, 9]], np.float32)
        parts.append(s)
    return concat_scenes(parts)


@pytest.mark.parametrize("pairs,contacts", [(1000, 10**5), (10**5, 1000), (10**5, 10**5)])
def test_status_is_the_first_frames_to_overflow(pairs, contacts):
    """A run's status is that of its earliest frame past a capacity, the world's or a scene's."""
    from dyphur_b200 import device
    s = _crowds()
    a, b = (device.World(s, max_pairs=pairs, max_contacts=contacts) for _ in range(2))
    seen = []
    for _ in range(8):
        a.step(1)
        seen.append(a.stats()["status"])
    b.step(8)
    assert (seen[0] != 0) == (min(pairs, contacts) == 1000) and seen[-1] != 0
    assert a.stats() == b.stats()


def test_probed_episode_keeps_the_last_frames_lists():
    """Frames timed one by one store their lists as a call's do: the last one's are kept."""
    a, b = _world(), _world()
    a.step(9)
    b.capture_episode(9, probe_stage=0)
    b.run_episode()
    assert (b.probe_ms() > 0).all()
    assert np.array_equal(bits(a.state()), bits(b.state())) and a.stats() == b.stats()
    for x, y in zip(a.history(), b.history()):
        assert np.array_equal(x, y)
    assert len(a.pairs()) > 0 and np.array_equal(a.pairs(), b.pairs())
    (ab, pa), (bb, pb) = a.contacts(), b.contacts()
    assert np.array_equal(ab, bb) and np.array_equal(bits(pa), bits(pb)) and a.solver_stats() == b.solver_stats()
