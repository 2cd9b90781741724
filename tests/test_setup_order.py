"""What a handle fills when it is made or first used is there before the streams
that read it: each set-up runs while the default stream is busy, and the work
that needs it follows on a stream that does not wait for the default one."""
import numpy as np
import pytest

from dyphur_b200 import scenes

pytestmark = pytest.mark.gpu


def bits(a):
    return np.ascontiguousarray(a, np.float32).view(np.uint32)


def _busy(torch):
    torch.cuda.synchronize()
    torch.cuda._sleep(100_000_000)  # some 50 ms on the default stream


@pytest.mark.parametrize("n", [8, 200])
def test_first_frames_of_a_small_scene(n):
    import torch
    from dyphur_b200 import device
    s = scenes.random_pile(n, seed=n)
    a, b = device.World(s), device.World(s)
    for _ in range(12):
        a.step(1)
    side = torch.cuda.Stream()
    _busy(torch)
    b.step(12, stream=side)
    side.synchronize()
    assert np.array_equal(bits(a.state()), bits(b.state()))
    assert a.stats() == b.stats()
    for x, y in zip(a.history(), b.history()):
        assert np.array_equal(x, y)
    assert device.device_error() == 0


@pytest.mark.parametrize("cap", [0, 56 << 10])
def test_batch_laid_out_again(cap):
    import torch
    from dyphur_b200 import device
    s = scenes.batch(9, 5, 60, seed=3)
    a, b = device.World(s), device.World(s)
    a.step(12)
    side = torch.cuda.Stream()
    _busy(torch)
    b.set_fused_config(cap, 1)
    b.step(12, stream=side)
    side.synchronize()
    assert np.array_equal(bits(a.state()), bits(b.state()))
    assert a.stats() == b.stats()
    assert device.device_error() == 0


@pytest.mark.parametrize("every", [1, 4])
def test_first_backward_pass(every):
    import torch
    from dyphur_b200 import device
    s = scenes.push(6)
    frames, got = 8, []
    for busy in (False, True):
        w = device.World(s, mode=1)
        n = w.bodies.n
        ckpt = torch.zeros(((frames + every - 1) // every, 13, n), device="cuda")
        g = torch.Generator(device="cuda").manual_seed(7)
        g_final = torch.randn((13, n), generator=g, device="cuda")
        g_init, g_im = torch.zeros((13, n), device="cuda"), torch.zeros(n, device="cuda")
        stream = torch.cuda.Stream() if busy else torch.cuda.current_stream()
        w.rollout_raw(frames, every, ckpt.data_ptr(), torch.cuda.current_stream().cuda_stream)
        if busy:
            _busy(torch)
        w.rollout_backward_raw(frames, every, ckpt.data_ptr(), g_final.data_ptr(), g_init.data_ptr(), g_im.data_ptr(),
                               stream.cuda_stream)
        stream.synchronize()
        torch.cuda.synchronize()
        got.append((bits(g_init.cpu().numpy()), bits(g_im.cpu().numpy())))
    assert np.any(got[0][0]) and all(np.array_equal(x, y) for x, y in zip(*got))
    assert device.device_error() == 0


def test_backward_pass_after_one_that_ran_out_of_memory():
    """Some of a pass's record sets were made, then the memory ran out: a smaller pass
    that finds enough of them there runs on them."""
    import torch
    from dyphur_b200 import capi, device
    s = scenes.push(128)
    n = s.n_bodies

    def gradients(w, frames):
        ckpt = torch.zeros((1, 13, n), device="cuda")
        w.bodies.fbuf[:13, :n] = w.initial_rows()[:13, :n]
        w.rollout_raw(frames, frames, ckpt.data_ptr(), torch.cuda.current_stream().cuda_stream)
        g_final, g_init, g_im = torch.ones((13, n), device="cuda"), torch.zeros((13, n), device="cuda"), \
            torch.zeros(n, device="cuda")
        w.rollout_backward_raw(frames, frames, ckpt.data_ptr(), g_final.data_ptr(), g_init.data_ptr(), g_im.data_ptr(),
                               torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        return bits(g_init.cpu().numpy()), bits(g_im.cpu().numpy())

    w, fresh = device.World(s, mode=1), device.World(s, mode=1)
    gradients(w, 1)  # two sets
    before = torch.cuda.mem_get_info()[0]
    want = gradients(fresh, 2)  # four sets
    four = before - torch.cuda.mem_get_info()[0]
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    hog = torch.empty(free - four, dtype=torch.uint8, device="cuda")  # room for some four more
    with pytest.raises(capi.DyphError):
        gradients(w, 12)
    del hog
    torch.cuda.empty_cache()
    got = gradients(w, 2)
    assert all(np.array_equal(a, b) for a, b in zip(got, want))
    assert device.device_error() == 0
