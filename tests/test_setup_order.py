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
