"""The work that programs have this framework do, as timed cases.

Six kinds of call, each through the package's public entry points:

  step    a single scene stepped some frames (World.step): the example's frame loop
  batch   many independent scenes stepped together (World.step on a batched world)
  episode a captured batch episode from host memory and back: the state uploaded
          from pinned memory, the poses of every other frame recorded to the host
  grad    a differentiable rollout and its gradients (autograd.rollout)
  rays    batched ray casts through a built tree (ray_query)
  loop    one frame of a program that drives the stages itself: integrate,
          broadphase, narrowphase, solve, a contact sensor read back, a ray scan

Scenes are the repository's own builders (scenes.py): the jittered box stacks of
the stress example, the random pile of boxes and spheres, the batch of stacks
and sphere piles, the mixed batch, the push setups. Frames start from a state
some frames into the episode, where bodies are in contact.

Frames are bit-identical to the reference's CPU build, which is the framework's
contract, so every forward output is compared exactly. A frame has no 64-bit
value apart from its float one: contact sets and branches are decided on the
float values and the scenes are chaotic, so `exact` gives one for ray casts only.
"""
import math

import numpy as np
import torch

from dyphur_b200 import autograd, capi, device, scenes

MODES = {"reference": capi.SOLVER_REFERENCE, "sequential": capi.SOLVER_SEQUENTIAL, "colored": capi.SOLVER_COLORED}


def listed():
    return [
        # The reference's sim-determinism size: 8 boxes and a ground. Launches and latency are all of it.
        dict(name="step_9", kind="step", scene="blocks", nx=2, ny=2, nz=2, mode="reference", start=30, frames=20),
        # The reference's stress example: 1024 boxes in a stack, its own solver order.
        dict(name="step_blocks_1025", kind="step", scene="blocks", nx=8, ny=16, nz=8, mode="reference", start=60,
             frames=20),
        # A pile of odd size in the sequential order (set_force_serial), the order that programs replay exactly.
        dict(name="step_pile_20002_seq", kind="step", scene="pile", n=20001, mode="sequential", start=120, frames=5),
        # The large single scene of the benchmark, settled into dense contact.
        dict(name="step_pile_65537", kind="step", scene="pile", n=65536, mode="reference", start=200, frames=10),
        # A handful of environments, as in interactive use or evaluation.
        dict(name="batch_64", kind="batch", builder="batch", scenes=64, lo=8, hi=64, mode="reference", tuned=False,
             start=30, frames=30),
        # The benchmark's batch: 4096 environments of 8 to 256 bodies, the layout tuned once per world.
        dict(name="batch_4096", kind="batch", builder="batch", scenes=4096, lo=8, hi=256, mode="sequential", tuned=True,
             start=60, frames=40),
        # Mixed boxes and spheres of every size, up to 512 bodies, reference order, as created.
        dict(name="batch_mixed_1024", kind="batch", builder="mixed", scenes=1024, lo=16, hi=512, mode="reference",
             tuned=False, start=60, frames=30),
        # Simulated data for a learner: episodes in from pinned memory, trajectories out.
        dict(name="episode_1024", kind="episode", scenes=1024, lo=8, hi=256, mode="sequential", frames=40),
        # Policy gradients through contact: the push task, a checkpoint every ten frames.
        dict(name="grad_push_256", kind="grad", builder="push", scenes=256, lo=0, hi=0, start=0, frames=20, every=10),
        # Gradients on mixed scenes with a checkpoint at every frame.
        dict(name="grad_mixed_512", kind="grad", builder="mixed", scenes=512, lo=16, hi=512, start=0, frames=8, every=1),
        # A million visibility rays into the settled pile.
        dict(name="rays_1m", kind="rays", n=65536, rays=1 << 20, camera=False, start=200),
        # One frame of a real-time program with a contact sensor on the ground and a 4096-ray scan.
        dict(name="loop_1025", kind="loop", nx=8, ny=16, nz=8, mode="reference", start=60, rays=4096),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step", "step", "batch", "batch", "episode", "grad", "rays", "loop"])
    mode = rng.choice(["reference", "sequential", "colored"])
    if kind == "step" and rng.random() < 0.5:
        return dict(kind=kind, scene="blocks", nx=rng.randint(1, 9), ny=rng.randint(1, 16), nz=rng.randint(1, 9),
                    mode=mode, start=rng.randint(20, 80), frames=rng.randint(1, 20))
    if kind == "step":
        return dict(kind=kind, scene="pile", n=_log_int(rng, 500, 65536), mode=mode, start=rng.randint(100, 200),
                    frames=rng.randint(1, 10))
    if kind == "batch":
        lo = rng.randint(4, 32)
        builder = rng.choice(["batch", "mixed"])
        return dict(kind=kind, builder=builder, scenes=_log_int(rng, 2, 4096 if builder == "batch" else 1024), lo=lo,
                    hi=lo + _log_int(rng, 8, 224 if builder == "batch" else 480), mode=mode, tuned=False,
                    start=rng.randint(20, 80), frames=rng.randint(1, 40))
    if kind == "episode":
        return dict(kind=kind, scenes=_log_int(rng, 8, 1024), lo=8, hi=_log_int(rng, 32, 256), mode=mode,
                    frames=2 * rng.randint(4, 20))
    if kind == "grad":
        frames = rng.randint(2, 20)
        if rng.random() < 0.5:
            return dict(kind=kind, builder="push", scenes=_log_int(rng, 4, 256), lo=0, hi=0, start=0, frames=frames,
                        every=rng.randint(1, frames))
        return dict(kind=kind, builder="mixed", scenes=_log_int(rng, 4, 512), lo=16, hi=_log_int(rng, 48, 512), start=0,
                    frames=min(frames, 8), every=rng.randint(1, 4))
    if kind == "rays":
        return dict(kind=kind, n=_log_int(rng, 256, 65536), rays=_log_int(rng, 1024, 1 << 20),
                    camera=rng.random() < 0.5, start=rng.randint(0, 120))
    return dict(kind=kind, nx=rng.randint(2, 9), ny=rng.randint(1, 16), nz=rng.randint(2, 9), mode=mode,
                start=rng.randint(20, 80), rays=_log_int(rng, 64, 16384))


def _scene(case, seed):
    seed = seed % (1 << 31) + 1
    if case["kind"] in ("step", "loop") and case.get("scene", "blocks") == "blocks":
        return scenes.stress_blocks(grid=(case["nx"], case["ny"], case["nz"]), seed=seed)
    if case["kind"] in ("step", "rays"):
        return scenes.random_pile(case["n"], seed=seed)
    # A batch is the same set of environments for every seed, each reset to
    # its own positions and to initial velocities drawn from the seed.
    if case.get("builder") == "push":
        scene = scenes.push(case["scenes"])
    elif case.get("builder") == "mixed":
        scene = scenes.batch_mixed(case["scenes"], case["lo"], case["hi"])
    else:
        scene = scenes.batch(case["scenes"], case["lo"], case["hi"])
    kick = np.random.default_rng(seed).normal(0.0, 0.2, (scene.n_bodies, 3)).astype(np.float32)
    scene.vel = scene.vel + np.where(scene.mass[:, None] > 0, kick, np.float32(0))
    return scene


def _rays(scene, pos, n_rays, camera, seed):
    """(n, 7) rays at the bodies: a pinhole camera above the scene, or random
    origins in its box aimed near random bodies."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    lo = torch.from_numpy(scene.bounds[0, :3].astype(np.float32)).cuda()
    hi = torch.from_numpy(scene.bounds[0, 3:].astype(np.float32)).cuda()
    rays = torch.empty((n_rays, 7), device="cuda")
    if camera:
        side = int(math.ceil(math.sqrt(n_rays)))
        k = torch.arange(n_rays, device="cuda")
        eye = torch.stack([lo[0], hi[1], lo[2]]) + torch.rand(3, generator=g, device="cuda")
        at = pos.mean(1)
        fwd = (at - eye) / (at - eye).norm()
        right = torch.linalg.cross(fwd, torch.tensor([0.0, 1.0, 0.0], device="cuda"))
        right = right / right.norm()
        up = torch.linalg.cross(right, fwd)
        u = ((k % side).float() + 0.5) / side - 0.5
        v = (torch.div(k, side, rounding_mode="floor").float() + 0.5) / side - 0.5
        rays[:, :3] = eye
        rays[:, 3:6] = fwd + u[:, None] * right + v[:, None] * up
    else:
        j = torch.randint(0, pos.shape[1], (n_rays,), generator=g, device="cuda")
        target = pos[:, j].T + 0.3 * torch.randn((n_rays, 3), generator=g, device="cuda")
        origin = lo + (hi - lo) * torch.rand((n_rays, 3), generator=g, device="cuda")
        rays[:, :3] = origin
        rays[:, 3:6] = target - origin
    rays[:, 6] = 200.0
    return rays


def prepare(case, seed):
    kind = case["kind"]
    scene = _scene(case, seed)
    n = scene.n_bodies
    if kind in ("rays", "loop"):
        world = device.World(scene, mode=MODES[case.get("mode", "reference")])
        world.step(case["start"])
        start = world.bodies.fbuf[:13, :n].clone()
        bodies, shapes = world.bodies, world.shapes
        st = {"kind": kind, "scene": scene, "bodies": bodies, "shapes": shapes, "start": start,
              "bp": device.Broadphase(n, scene.max_pairs),
              "rays": _rays(scene, start[:3], case["rays"], case.get("camera", True), seed)}
        torch.cuda.synchronize()
        world.close()
        if kind == "rays":
            st["bp"].build_and_query(bodies, shapes, scene.bounds[0])
            st["view"] = st["bp"].bvh_view(n)
        else:
            st["np"] = device.Narrowphase(scene.max_contacts)
            st["solver"] = device.XpbdSolver(scene.n_iters, scene.max_contacts, n, scene.friction)
            st["solver"].set_mode(MODES[case["mode"]])
            st["sensor"] = device.ContactSensor(int(scene.shape[-1]))  # the ground
            st["touching"], st["points"] = np.zeros((n, 2), np.uint32), np.zeros((n, 7), np.float32)
        return st
    mode = MODES[case.get("mode", "sequential")]
    world = device.World(scene, mode=mode)
    st = {"kind": kind, "world": world, "n": n}
    if kind in ("step", "batch"):
        if case.get("tuned"):
            world.autotune(8)
        world.step(case["start"])
        st["start"] = world.bodies.fbuf[:13].clone()
        st["frames"] = case["frames"]
    elif kind == "episode":
        st["host_in"] = world.bodies.fbuf.cpu().pin_memory()
        st["host_out"] = torch.empty((13, world.bodies.fbuf.shape[1])).pin_memory()
        st["traj"] = torch.empty(((case["frames"] + 1) // 2, n, 7)).pin_memory()
        world.set_trajectory(st["traj"], 2)
        world.capture_episode(case["frames"])
    else:
        dyn = np.flatnonzero(scene.mass > 0) if case["builder"] == "mixed" else \
            np.concatenate([np.arange(a, a + 64) for a in scene.body_offset[:-1]])
        fb = world.bodies.fbuf
        st.update(vel=fb[7:10, :n].T.clone().requires_grad_(True), ang=fb[10:13, :n].T.clone().requires_grad_(True),
                  im=fb[13, :n].clone().requires_grad_(True), boxes=torch.from_numpy(dyn).cuda(),
                  targets=torch.from_numpy(scene.targets[dyn]).cuda(), frames=case["frames"], every=case["every"])
    torch.cuda.synchronize()
    return st


def run(st):
    kind = st["kind"]
    if kind in ("step", "batch"):
        w = st["world"]
        w.bodies.fbuf[:13] = st["start"]
        w.step(st["frames"])
        return w.bodies.fbuf[:13, :st["n"]]
    if kind == "episode":
        w = st["world"]
        w.bodies.fbuf.copy_(st["host_in"], non_blocking=True)
        w.run_episode()
        st["host_out"].copy_(w.bodies.fbuf[:13], non_blocking=True)
        return st["traj"], st["host_out"]
    if kind == "grad":
        final = autograd.rollout(st["world"], st["vel"], st["ang"], st["im"], st["frames"], every=st["every"])
        loss = ((final[:3, st["boxes"]].T - st["targets"]) ** 2).sum(-1).mean()
        grads = torch.autograd.grad(loss, [st["vel"], st["ang"], st["im"]])
        return (final.detach(), loss.detach()) + tuple(grads)
    bodies, shapes, scene = st["bodies"], st["shapes"], st["scene"]
    if kind == "rays":
        return device.ray_query(st["view"], bodies, shapes, st["rays"])
    bodies.fbuf[:13, :scene.n_bodies] = st["start"]
    device.integrate(bodies, scene.gravity, scene.dt, scene.n_substeps)
    st["bp"].build_and_query(bodies, shapes, scene.bounds[0])
    st["np"].run(st["bp"], bodies, shapes)
    contacts = st["np"].contacts_view()
    st["solver"].solve(contacts, bodies, scene.dt)
    st["sensor"].query(contacts, bodies)
    touching, points = st["sensor"].rows()
    t, body = device.ray_query(st["bp"].bvh_view(scene.n_bodies), bodies, shapes, st["rays"])
    m = len(touching)  # into arrays of one size: a body touches the ground once at most
    st["touching"][:m], st["points"][:m] = touching, points
    st["touching"][m:], st["points"][m:] = 0, 0
    return bodies.fbuf[:13, :scene.n_bodies], m, st["touching"], st["points"], t, body


# Candidate pairs and contacts per body and frame, as measured on these scenes
# (settled; a pair costs the separating-axis test, a contact one projection).
_PER_BODY = {"blocks": (4.0, 2.5), "pile": (8.0, 3.0), "batch": (3.3, 1.9), "mixed": (6.0, 2.5), "push": (5.0, 2.8)}


def _bodies(case):
    kind = case["kind"]
    if "nx" in case:
        return case["nx"] * case["ny"] * case["nz"] + 1
    if kind in ("step", "rays"):
        return case["n"] + 1
    if case.get("builder") == "push":
        return 66 * case["scenes"]
    lo, hi = case["lo"], case["hi"]  # log-uniform sizes and a ground each
    return int(case["scenes"] * ((hi - lo) / math.log((hi + 1) / lo) + 1))


def work(case):
    """Bytes: the state, inverse masses and inertias, shapes and flags read once
    and the outputs written once per pass. Operations: per frame, 250 a body
    (integration, leaf box, renormalisation), 700 a candidate pair, 500 a contact;
    a backward pass is twice the forward's; a ray reads the boxes of about
    2 log2(n) nodes at 20 operations each."""
    n, kind = _bodies(case), case["kind"]
    scene = "mixed" if case.get("builder") == "mixed" else "push" if case.get("builder") == "push" else \
        "batch" if kind in ("batch", "episode") else "pile" if "n" in case else "blocks"
    pairs, contacts = _PER_BODY[scene]
    frame = n * (250.0 + 700.0 * pairs + 500.0 * contacts)
    state = n * (13 + 13 + 7 + 5) * 4.0
    if kind == "rays":
        return {"bytes": case["rays"] * 36.0 + n * (7 + 4) * 4.0 + 32.0 * n,
                "flops": case["rays"] * 40.0 * math.log2(n)}
    if kind == "loop":
        return {"bytes": state + case["rays"] * 36.0, "flops": frame + case["rays"] * 40.0 * math.log2(n)}
    frames = case["frames"]
    if kind == "episode":
        return {"bytes": state + (frames + 1) // 2 * n * 28.0, "flops": frames * frame}
    if kind == "grad":
        return {"bytes": state + n * (13 + 13 + 14) * 4.0, "flops": 3.0 * frames * frame}
    return {"bytes": state, "flops": frames * frame}


def tolerance(case):
    if case["kind"] == "grad":
        # The gradient against FP64 dual numbers along the same branches: 3.3e-6
        # relative after 10 frames of the push task, 1.9e-6 on the mixed scenes;
        # rounding grows with the frames.
        return {"rel": 2e-5}
    return "exact"


def exact(case, seed):
    """Ray casts in 64 bits against every body (no tree); None where that takes too long."""
    if case["kind"] != "rays" or float(case["rays"]) * case["n"] > 4e9:
        return None
    st = prepare(case, seed)
    scene = st["scene"]
    p = st["start"].double()
    sh = torch.from_numpy(scene.shape.astype(np.int64)).cuda()
    typ = torch.from_numpy(scene.shape_type.astype(np.int64)).cuda()[sh]
    half = torch.from_numpy(scene.shape_half).cuda().double()[sh]
    pos, w, u = p[:3].T, p[3], p[4:7].T
    rays = st["rays"].double()
    t_out = rays[:, 6].clone()
    b_out = torch.full((rays.shape[0],), -1, dtype=torch.int64, device="cuda")
    step = max(1, int(4e6) // pos.shape[0])

    def to_body(v):  # rotate by the conjugate quaternion
        t = 2.0 * torch.linalg.cross(-u.expand_as(v), v)
        return v + w[None, :, None] * t + torch.linalg.cross(-u.expand_as(v), t)

    for i in range(0, rays.shape[0], step):
        r = rays[i:i + step]
        oc = r[:, None, :3] - pos
        d = r[:, None, 3:6].expand_as(oc)
        lo, ld = to_body(oc), to_body(d)
        t1, t2 = (-half - lo) / ld, (half - lo) / ld
        tmin, tmax = torch.minimum(t1, t2).amax(-1), torch.maximum(t1, t2).amin(-1)
        tb = torch.where(tmin >= 0, tmin, tmax)
        tb = torch.where((tmax < 0) | (tmin > tmax), torch.inf, tb)
        a, b = (d * d).sum(-1), (d * oc).sum(-1)
        disc = b * b - a * ((oc * oc).sum(-1) - half[:, 0] ** 2)
        sq = disc.clamp(min=0).sqrt()
        ts = torch.where((-b - sq) / a < 0, (-b + sq) / a, (-b - sq) / a)
        ts = torch.where((disc < 0) | (ts < 0), torch.inf, ts)
        t, body = torch.where(typ == 1, ts, tb).min(-1)
        hit = t < r[:, 6]
        t_out[i:i + step] = torch.where(hit, t, r[:, 6])
        b_out[i:i + step] = torch.where(hit, body, -1)
    return t_out, None
