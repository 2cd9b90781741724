"""Calls inside a caller's stream capture and beside one: what is recorded is
kernels alone, and a call on another stream leaves the capture as it is."""
import ctypes as C
import os
import subprocess
import sys

import numpy as np
import pytest

from dyphur_b200 import capi, scenes
from test_ray_sensor import _random_rays, bits

pytestmark = pytest.mark.gpu

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


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


@pytest.mark.parametrize("kind", ["small", "single", "batch"])
def test_steps_are_not_recorded(kind):
    """A world's frames are refused inside a capture, which goes on without them."""
    import torch
    from dyphur_b200 import device
    s = {"small": scenes.random_pile(40, seed=1), "single": scenes.random_pile(600, seed=1),
         "batch": scenes.batch(5, 5, 30, seed=1)}[kind]
    a, b = device.World(s), device.World(s)
    for w in (a, b):
        w.step(1)
    x, ckpt = torch.zeros(64, device="cuda"), torch.zeros((1, 13, s.n_bodies), device="cuda")
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        x.add_(1)
        for frames in (1, 4):
            with pytest.raises(capi.DyphError):
                b.step(frames)
        with pytest.raises(capi.DyphError):
            b.rollout_raw(2, 2, ckpt.data_ptr(), torch.cuda.current_stream().cuda_stream)
    g.replay()
    torch.cuda.synchronize()
    assert float(x.sum()) == 64
    a.step(4)
    b.step(4)
    assert np.array_equal(bits(a.state()), bits(b.state())) and a.stats() == b.stats()
    assert device.device_error() == 0


def test_large_narrowphase_beside_a_capture():
    """A handle's first run on a scene whose bodies it packs, while another stream captures."""
    import torch
    from dyphur_b200 import device
    small, large = scenes.random_pile(50, seed=2), scenes.random_pile(33000, seed=2)
    npz, other_npz = device.Narrowphase(large.max_contacts), device.Narrowphase(large.max_contacts)
    parts = []
    for s in (small, large):
        w = device.World(s)
        w.step(45)
        bp = device.Broadphase(s.n_bodies, 400000)
        bp.build_and_query(w.bodies, w.shapes, s.bounds[0])
        parts.append((bp, w.bodies, w.shapes, w))
    npz.run(*parts[0][:3])
    other_npz.run(*parts[1][:3])
    want = other_npz.contacts()
    x, other = torch.zeros(64, device="cuda"), torch.cuda.Stream()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        x.add_(1)
        npz.run(*parts[1][:3], stream=other)
    g.replay()
    torch.cuda.synchronize()
    got = npz.contacts()
    assert float(x.sum()) == 64 and len(want[0]) > 1000
    assert np.array_equal(got[0], want[0]) and np.array_equal(bits(got[1]), bits(want[1]))
    assert device.device_error() == 0


FIRST_QUERY = """
import ctypes as C
import torch
from dyphur_b200 import capi, device, scenes
s = scenes.random_pile(17000, seed=2)
b, sh = device.DeviceBodies(s), device.DeviceShapes(s)
bp = device.Broadphase(s.n_bodies, s.max_pairs)
bp.build_and_query(b, sh, s.bounds[0])
view = bp.bvh_view(s.n_bodies)
rays = torch.zeros((64, 7), device="cuda")
rays[:, 1] = 30
rays[:, 4] = -1
rays[:, 6] = 1e3
hits = torch.zeros((2, 64, 2), dtype=torch.int32, device="cuda")
x, other = torch.zeros(64, device="cuda"), torch.cuda.Stream()
torch.cuda.synchronize()
g = torch.cuda.CUDAGraph()
def query(k, stream):
    return capi.lib().dyph_ray_query(C.byref(view), C.byref(b.view), C.byref(sh.view), rays.data_ptr(),
                                     hits[k].data_ptr(), 64, stream.cuda_stream)
with torch.cuda.graph(g):
    x.add_(1)
    if INSIDE:
        assert query(0, torch.cuda.current_stream()) == 0
    else:
        assert query(0, other) == 0
g.replay()
torch.cuda.synchronize()
assert float(x.sum()) == 64
assert query(1, torch.cuda.current_stream()) == 0
torch.cuda.synchronize()
assert torch.equal(hits[0], hits[1]) and (hits[0, :, 1] >= 0).any()
assert device.device_error() == 0
"""


@pytest.mark.parametrize("inside", [True, False])
def test_first_large_query_of_a_process(inside):
    run = subprocess.run([sys.executable, "-c", f"INSIDE = {inside}\n" + FIRST_QUERY], cwd=ROOT, capture_output=True,
                         text=True, timeout=300)
    assert run.returncode == 0, run.stderr[-2000:]


def _cudart():
    """The runtime that torch has loaded."""
    import torch
    torch.cuda.init()
    with open("/proc/self/maps") as f:
        path = next(p for p in (line.split()[-1] for line in f) if "libcudart.so" in p)
    return C.CDLL(path)


def test_captured_large_query_instantiates_twice():
    """A recorded query is kernels: its graph can be instantiated as often as the
    program likes, and be part of another graph."""
    import torch
    from dyphur_b200 import device
    s = scenes.random_pile(17000, seed=2)
    b, sh = device.DeviceBodies(s), device.DeviceShapes(s)
    bp = device.Broadphase(s.n_bodies, s.max_pairs)
    bp.build_and_query(b, sh, s.bounds[0])
    view = bp.bvh_view(s.n_bodies)
    rays = torch.from_numpy(_random_rays(s, 4096, 1)).cuda()
    want_t, want_b = device.ray_query(view, b, sh, rays)
    hits = torch.zeros((4096, 2), dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    rt, stream = _cudart(), torch.cuda.Stream()
    graph, cs = C.c_void_p(), C.c_void_p(stream.cuda_stream)
    assert rt.cudaStreamBeginCapture(cs, 0) == 0
    st = capi.lib().dyph_ray_query(C.byref(view), C.byref(b.view), C.byref(sh.view), rays.data_ptr(), hits.data_ptr(),
                                   4096, stream.cuda_stream)
    assert rt.cudaStreamEndCapture(cs, C.byref(graph)) == 0 and st == 0
    execs = [C.c_void_p(), C.c_void_p()]
    codes = [rt.cudaGraphInstantiate(C.byref(e), graph, C.c_ulonglong(0)) for e in execs]
    parent, node = C.c_void_p(), C.c_void_p()
    codes.append(rt.cudaGraphCreate(C.byref(parent), 0))
    codes.append(rt.cudaGraphAddChildGraphNode(C.byref(node), parent, None, C.c_size_t(0), graph))
    for e in execs:
        if e.value:
            hits.zero_()
            torch.cuda.synchronize()
            assert rt.cudaGraphLaunch(e, cs) == 0
            stream.synchronize()
            assert torch.equal(hits[:, 0].view(torch.float32), want_t) and torch.equal(hits[:, 1], want_b)
            rt.cudaGraphExecDestroy(e)
    rt.cudaGraphDestroy(parent)
    rt.cudaGraphDestroy(graph)
    assert codes == [0, 0, 0, 0]
    assert device.device_error() == 0
