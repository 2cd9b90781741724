"""Calls beside a caller's stream capture leave the capture as it is."""
import numpy as np
import pytest

from dyphur_b200 import scenes
from test_ray_sensor import bits

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [8, 200])
def test_frames_beside_a_capture(n):
    """The first call of several frames, while another stream captures."""
    import torch
    from dyphur_b200 import device
    s = scenes.random_pile(n, seed=n)
    a, b = device.World(s), device.World(s)
    for w in (a, b):
        w.step(1)
    for _ in range(5):
        a.step(1)
    x, other = torch.zeros(64, device="cuda"), torch.cuda.Stream()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        x.add_(1)
        b.step(5, stream=other)
    g.replay()
    torch.cuda.synchronize()
    assert float(x.sum()) == 64
    assert np.array_equal(bits(a.state()), bits(b.state())) and a.stats() == b.stats()
    assert device.device_error() == 0
