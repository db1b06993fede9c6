"""Timed workloads of the public entry points: single worlds from a few dozen to 100k bodies, jointed
chains with convex hulls, a world whose bodies go through host memory every step, batches of small
worlds, ray queries, and the adjoint.

Inputs are built directly in their working state (bodies at rest on one another at the contact
margin, joints at their anchors) from the seed alone, so that no solver run is needed to prepare
them. A world steps on from where the pass before left it, as a simulation does.
"""

from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), 'three-avbd_b200'))

import avbd_b200  # noqa: E402
from avbd_b200 import _abi, hulls as hull_shapes, scenes  # noqa: E402

GAP = 0.0095        # bodies at rest overlap by about the contact margin (0.01 m)
PITCH = 1.08        # a pile's lattice spacing
DT = 1.0 / 60.0
FLAG_FACE_BIAS, FLAG_START_AT_REST, FLAG_MASS_PENALTY = _abi.FLAG_FACE_BIAS, _abi.FLAG_START_AT_REST, _abi.FLAG_MASS_PENALTY


# --- the cases -----------------------------------------------------------------------------------------

def listed():
    return [
        # one small scene a frame, as an editor or a demo steps it: launches and latency
        dict(name='step 48 boxes', kind='step', bodies=48, spheres=0.0, rules='reference', iterations=10),
        # a game level's world with the production rules
        dict(name='step 300 world rules', kind='step', bodies=300, spheres=0.3, rules='world', iterations=10),
        dict(name='step 3001', kind='step', bodies=3001, spheres=0.3, rules='reference', iterations=10),
        dict(name='step 20000 world rules', kind='step', bodies=20000, spheres=0.3, rules='world', iterations=10),
        # the headline size
        dict(name='step 100000', kind='step', bodies=100000, spheres=0.3, rules='reference', iterations=10),
        # fracture debris on hanging chains: hull narrowphase and joint rows
        dict(name='hulls and chains', kind='chains', hulls=4000, chains=200, links=50, iterations=15),
        # a host program that edits bodies between steps: records in and out of pinned memory each step
        dict(name='host loop 8000', kind='host', bodies=8000, spheres=0.3, rules='reference', iterations=10),
        # rollouts of many small worlds (learning, sampling): a few, and as many as fill the GPU
        dict(name='batch 96', kind='batch', worlds=96, median=64, shape='default', steps=1, iterations=10),
        dict(name='batch 4096', kind='batch', worlds=4096, median=64, shape='tuned', steps=2, iterations=10),
        # sensors and picking: rays into a pile
        dict(name='rays 4096 in 20000', kind='rays', rays=4096, bodies=20000, spheres=0.3),
        # gradients of a rollout: a handful of worlds, and a batch
        dict(name='adjoint 16 x 24', kind='adjoint', worlds=16, bodies=24, steps=12, iterations=10),
        dict(name='adjoint 1024 x 64', kind='adjoint', worlds=1024, bodies=64, steps=8, iterations=10),
    ]


def draw(rng):
    log = lambda lo, hi: int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    kind = rng.choice(['step', 'step', 'step', 'host', 'chains', 'batch', 'rays', 'adjoint'])
    if kind in ('step', 'host'):
        return dict(kind=kind, bodies=log(20, 100000) if kind == 'step' else log(100, 30000), spheres=rng.choice([0.0, 0.3, 0.6]),
                    rules=rng.choice(['reference', 'world']), iterations=rng.choice([4, 10, 15]))
    if kind == 'chains':
        return dict(kind=kind, hulls=log(20, 4000), chains=log(4, 200), links=rng.randrange(5, 51), iterations=15)
    if kind == 'batch':
        return dict(kind=kind, worlds=log(8, 4096), median=rng.choice([32, 48, 64]), shape=rng.choice(['default', 'tuned']), steps=rng.choice([1, 2]),
                    iterations=10)
    if kind == 'rays':
        return dict(kind=kind, rays=log(1, 4096), bodies=log(50, 20000), spheres=rng.choice([0.0, 0.3]))
    return dict(kind=kind, worlds=log(1, 512), bodies=rng.randrange(5, 65), steps=rng.randrange(3, 13), iterations=10)


# --- inputs --------------------------------------------------------------------------------------------

def _quat_mul(a, b):
    ax, ay, az, aw = np.moveaxis(a, -1, 0)
    bx, by, bz, bw = np.moveaxis(b, -1, 0)
    return np.stack([aw * bx + ax * bw + ay * bz - az * by, aw * by - ax * bz + ay * bw + az * bx, aw * bz + ax * by - ay * bx + az * bw,
                     aw * bw - ax * bx - ay * by - az * bz], -1)


def _records(pos, rot, size, mass, moment, radius, friction, vel, ang, shape, up):
    r = np.zeros(len(pos), dtype=avbd_b200.BODY_DTYPE)
    r['pos'], r['rot'], r['size'], r['mass'], r['moment'], r['radius'] = pos, rot, size, mass, moment, radius
    r['friction'], r['vel'], r['ang_vel'], r['shape'] = friction, vel, ang, shape
    r['flags'] = 1.0
    r['initial_pos'], r['initial_rot'], r['inertial_pos'], r['inertial_rot'] = r['pos'], r['rot'], r['pos'], r['rot']
    r['prev_up_vel'] = r['vel'][:, up]
    return r


def _box_moment(size, mass):
    s2 = size * size
    return np.stack([s2[:, 1] + s2[:, 2], s2[:, 0] + s2[:, 2], s2[:, 0] + s2[:, 1]], 1) * (mass / 12.0)[:, None]


def _pile(counts, seed, spheres, up=2):
    """Settled piles, one per entry of `counts` (dynamic bodies each), as records in world order: per
    world a static ground box, then boxes and spheres in staggered layers, each layer's bodies of one
    thickness and resting on up to four below, a little turned and moving a little."""
    rng = np.random.default_rng(seed)
    counts = np.asarray(counts, dtype=np.int64)
    W, total = len(counts), int(counts.sum())
    layers = np.clip(np.round(counts ** (1.0 / 3.0)), 1, 10).astype(np.int64)
    side = np.ceil(np.sqrt(counts / layers)).astype(np.int64)
    w = np.repeat(np.arange(W), counts)
    k = np.arange(total) - np.repeat(np.cumsum(counts) - counts, counts)
    s = side[w]
    gx, gy, gz = k % s, (k // s) % s, k // (s * s)
    thick = rng.uniform(0.6, 1.0, (W, 12))
    below = np.cumsum(thick, 1) - thick
    t = thick[w, gz]
    is_sphere = rng.random(total) < spheres
    size = np.stack([rng.uniform(0.7, 1.0, total), rng.uniform(0.7, 1.0, total), t], 1)
    size = np.where(is_sphere[:, None], t[:, None], size)
    pos = np.stack([(gx - (s - 1) / 2 + 0.5 * (gz % 2)) * PITCH, (gy - (s - 1) / 2 + 0.5 * (gz % 2)) * PITCH,
                    below[w, gz] + t / 2 - GAP * (gz + 1)], 1)
    pos[:, :2] += rng.uniform(-0.04, 0.04, (total, 2))
    yaw = rng.uniform(-0.2, 0.2, total)
    tilt = rng.normal(0.0, 1e-3, (total, 2))
    rot = np.stack([tilt[:, 0], tilt[:, 1], np.sin(yaw / 2), np.cos(yaw / 2)], 1)
    rot /= np.linalg.norm(rot, axis=1, keepdims=True)
    mass = rng.uniform(0.5, 2.0, total) * np.where(is_sphere, math.pi / 6.0, 1.0) * size.prod(1)
    moment = np.where(is_sphere[:, None], (0.1 * mass * t * t)[:, None], _box_moment(size, mass))
    radius = np.where(is_sphere, t / 2, np.sqrt((size * size).sum(1)) / 2)
    friction = rng.uniform(0.3, 0.8, total)
    vel, ang = rng.normal(0.0, 0.05, (total, 3)), rng.normal(0.0, 0.05, (total, 3))
    first = np.cumsum(counts) - counts  # dynamic bodies before each world
    put = np.arange(total) + w + 1
    n = total + W

    def both(dynamic, ground):
        out = np.empty((n,) + dynamic.shape[1:])
        out[put] = dynamic
        out[first + np.arange(W)] = ground
        return out

    extent = side * PITCH + 20.0
    gsize = np.stack([extent, extent, np.ones(W)], 1)
    pos, size = both(pos, [0.0, 0.0, -0.5]), both(size, gsize)
    rot, moment, vel, ang = both(rot, [0.0, 0.0, 0.0, 1.0]), both(moment, 0.0), both(vel, 0.0), both(ang, 0.0)
    mass, radius, friction = both(mass, 0.0), both(radius, np.sqrt((gsize * gsize).sum(1)) / 2), both(friction, 0.5)
    shape = both(is_sphere.astype(np.float64), 0.0)
    if up == 1:  # turn z up into y up: (x, y, z) -> (y, z, x)
        turn = lambda a: a[:, [1, 2, 0]]
        pos, size, moment, vel, ang = (turn(a) for a in (pos, size, moment, vel, ang))
        rot = rot[:, [1, 2, 0, 3]]
    return _records(pos, rot, size, mass, moment, radius, friction, vel, ang, shape, up)


def _world_counts(case):
    """The worlds' dynamic body counts: the same for every seed, as a user's set of scenes is."""
    rng = np.random.default_rng([case['worlds'], 7])
    return np.clip(np.round(case['median'] * np.exp(0.5 * rng.standard_normal(case['worlds']))), 16, 512).astype(np.int64)


def _params(rules, iterations):
    """'reference': the solver's own defaults; 'world': what a production world runs with."""
    if rules == 'world':
        p = _abi.Params()
        if _abi.load().avbd_world_params(p) != _abi.AVBD_OK:
            raise RuntimeError('avbd_world_params')
    else:
        p = avbd_b200.solver.to_params(scenes.Params())
    p.gravity = -9.81
    p.iterations = iterations
    return p


class _DeviceArray:
    """One of the world's device arrays by address, for torch.as_tensor, which keeps this object and
    so the world that owns the memory."""

    def __init__(self, world, address, n):
        self.world = world
        self.__cuda_array_interface__ = {'shape': (n, 4), 'typestr': '<f4', 'data': (address, False), 'version': 2, 'strides': None}


def _views(world):
    """The world's body state as torch tensors on its own storage: position, rotation, velocity,
    angular velocity."""
    v = world.body_storage()
    rows = {'pos': 0, 'rot': 1, 'vel': 8, 'ang': 9}
    full = {k: torch.as_tensor(_DeviceArray(world, v['fields'][i], v['count']), device='cuda') for k, i in rows.items()}
    return {k: t if k == 'rot' else t[:, :3] for k, t in full.items()}


def _chains(case, seed):
    """Chains of boxes hanging from static anchors by ball joints, and convex hulls heaped between them."""
    rng = np.random.default_rng(seed)
    C, L, H = case['chains'], case['links'], case['hulls']
    side = max(1, math.ceil(math.sqrt(C)))
    step, top = 3.2, L * 0.5 + 2.0
    cx, cy = (np.arange(C) % side - (side - 1) / 2) * step, (np.arange(C) // side - (side - 1) / 2) * step
    ground = dict(pos=[[0.0, 0.0, -0.5]], size=[[side * step + 20.0, side * step + 20.0, 1.0]], mass=[0.0])
    anchors = dict(pos=np.stack([cx, cy, np.full(C, top + 0.1)], 1), size=np.tile([0.4, 0.4, 0.2], (C, 1)), mass=np.zeros(C))
    z = top - 0.25 - 0.5 * np.arange(L)
    links = dict(pos=np.stack([np.repeat(cx, L), np.repeat(cy, L), np.tile(z, C)], 1), size=np.tile([0.2, 0.2, 0.5], (C * L, 1)),
                 mass=np.full(C * L, 0.02))
    links['pos'] += rng.normal(0.0, 1e-3, (C * L, 3))
    shapes = []
    while len(shapes) < min(48, H):
        pts = rng.standard_normal((int(rng.integers(8, 33)), 3))
        pts /= np.linalg.norm(pts, axis=1, keepdims=True)
        h = hull_shapes.build_hull((pts * rng.uniform(0.3, 1.0, 3)).reshape(-1))
        if h is not None:
            shapes.append(h)
    offset = np.cumsum([0] + [h.vec4s for h in shapes[:-1]]) if shapes else np.zeros(0)
    which = rng.integers(0, max(len(shapes), 1), H)
    i = np.arange(H)
    hp = np.stack([(i % side - (side - 1) / 2 + 0.5) * step, ((i // side) % side - (side - 1) / 2 + 0.5) * step, 0.7 + 1.2 * (i // (side * side))], 1)
    hp[:, :2] += rng.uniform(-0.5, 0.5, (H, 2))
    q = rng.standard_normal((H, 4))
    q /= np.linalg.norm(q, axis=1, keepdims=True)
    pick = lambda f: np.array([f(shapes[k]) for k in which], dtype=np.float64)
    boxes = {k: np.concatenate([np.asarray(p[k], np.float64) for p in (ground, anchors, links)]) for k in ground}
    nb = len(boxes['mass'])
    pos = np.concatenate([boxes['pos'], hp])
    size = np.concatenate([boxes['size'], pick(lambda h: h.size).reshape(-1, 3)])
    mass = np.concatenate([boxes['mass'], pick(lambda h: h.volume)])
    moment = np.concatenate([_box_moment(boxes['size'], boxes['mass']), pick(lambda h: h.moments).reshape(-1, 3)])
    radius = np.concatenate([np.sqrt((boxes['size'] ** 2).sum(1)) / 2, pick(lambda h: h.radius)])
    rot = np.concatenate([np.tile([0.0, 0.0, 0.0, 1.0], (nb, 1)), q])
    shape = np.concatenate([np.zeros(nb), 3.0 + offset[which]])
    vel = rng.normal(0.0, 0.1, (nb + H, 3)) * (mass > 0)[:, None]
    friction = np.concatenate([np.full(nb, 0.5), rng.uniform(0.3, 0.8, H)])
    bodies = _records(pos, rot, size, mass, moment, radius, friction, vel, np.zeros((nb + H, 3)), shape, 2)
    # the joint from an anchor to its first link, and the one between links
    sample = [scenes.Body([0.0] * 3, s, 1.0, [1.0] * 3, 0.5, 1.0) for s in ([0.4, 0.4, 0.2], [0.2, 0.2, 0.5], [0.2, 0.2, 0.5])]
    ball = dict(stiffness_lin=math.inf, stiffness_ang=0.0, fracture=1e4, fracture_linear=True)
    head, head_info = avbd_b200.pack_force(scenes.Force('joint', 0, 1, [0.0, 0.0, -0.1], [0.0, 0.0, 0.25], **ball), sample)
    link, _ = avbd_b200.pack_force(scenes.Force('joint', 1, 2, [0.0, 0.0, -0.25], [0.0, 0.0, 0.25], **ball), sample)
    joints, info = np.full(C * L, link), np.full(C * L, head_info)
    joints[::L] = head
    b = 1 + C + np.arange(C * L)
    info['b'] = b
    info['a'] = np.where(np.arange(C * L) % L == 0, 1 + np.arange(C * L) // L, b - 1)
    return bodies, joints, info, shapes


def _recording(n, steps, iterations, seed):
    """One world's contact structure for the adjoint: n boxes in columns of up to four on the ground,
    sliding and swaying, the same contacts every step (a box's four lower corners on what is below it)."""
    rng = np.random.default_rng(seed)
    height = 4
    k = np.arange(n)
    col, lev = k // height, k % height
    side = math.ceil(math.sqrt(max(1, math.ceil(n / height))))
    pos = np.stack([(col % side) * 1.6, (col // side) * 1.6, 0.4 + 0.8 * lev - GAP * (lev + 1)], 1)
    pos[:, :2] += rng.uniform(-0.1, 0.1, (n, 2))
    yaw = rng.uniform(-0.1, 0.1, n)
    rot = np.stack([rng.normal(0, 1e-3, n), rng.normal(0, 1e-3, n), np.sin(yaw / 2), np.cos(yaw / 2)], 1)
    rot /= np.linalg.norm(rot, axis=1, keepdims=True)
    bodies = np.zeros((n + 1, 13))
    bodies[0] = [0, 0, -0.5, 0, 0, 0, 1, 0, 0, 0, 0, 0, 0.5]
    bodies[1:, :3], bodies[1:, 3:7] = pos, rot
    bodies[1:, 7] = rng.normal(0.0, 0.1, n)               # last step's velocity along up
    bodies[1:, 8:11] = 0.64 / 6.0                          # moments of a unit mass
    bodies[1:, 11] = 1.0
    bodies[1:, 12] = 0.5
    full_pos, full_rot = bodies[:, :3], bodies[:, 3:7]
    a = k + 1
    b = np.where(lev == 0, 0, k)
    normal = np.stack([rng.normal(0, 2e-3, n), rng.normal(0, 2e-3, n), np.ones(n)], 1)
    normal /= np.linalg.norm(normal, axis=1, keepdims=True)
    t1 = np.cross(normal, np.cross(np.tile([1.0, 0.0, 0.0], (n, 1)), normal))
    t1 /= np.linalg.norm(t1, axis=1, keepdims=True)
    basis = np.stack([normal, t1, np.cross(normal, t1)], 1)
    corner = np.array([[x, y, -0.4] for x in (-0.4, 0.4) for y in (-0.4, 0.4)])
    ra = np.repeat(corner[None], n, 0) * rng.uniform(0.9, 1.0, (n, 4, 1))
    xa = pos[:, None] + _turn(rot[:, None], ra)
    xb = xa + normal[:, None] * GAP + rng.normal(0.0, 2e-4, (n, 4, 3))
    conj = full_rot[b] * [-1, -1, -1, 1]
    rb = _turn(conj[:, None], xb - full_pos[b][:, None])
    anchors = np.concatenate([ra, rb], -1).reshape(-1, 6)
    m, p = n, 4 * n
    prev = np.concatenate([np.full(p, -1), np.arange((steps - 1) * p)])
    return {'n': n + 1, 'steps': steps, 'bodies': bodies.reshape(-1), 'step_man': np.arange(steps + 1) * m, 'step_pt': np.arange(steps + 1) * p,
            'man_bodies': np.tile(np.stack([a, b], 1).reshape(-1), steps), 'basis': np.tile(basis.reshape(-1), steps),
            'anchors': np.tile(anchors.reshape(-1), steps), 'pt_man': np.repeat(np.arange(steps * m), 4), 'pt_prev': prev,
            'colors': np.tile(np.concatenate([[-1], lev % 2]), steps), 'ncol': np.full(steps, 2 if n > 1 else 1),
            'params': dict(iterations=iterations, dt=DT, gravity=-9.81, alpha=0.99, gamma=0.999, beta_lin=10000.0, contact_margin=0.01)}


def _turn(q, v):
    """v rotated by q (arrays, last axis)."""
    u, w = q[..., :3], q[..., 3:]
    t = 2.0 * np.cross(u, v)
    return v + w * t + np.cross(u, t)


def _adjoint_inputs(case, seed):
    """Recordings of 8 distinct worlds shared round-robin, and every world's own parameters and target."""
    recs = [_recording(case['bodies'], case['steps'], case['iterations'], [seed, k]) for k in range(min(8, case['worlds']))]
    recs = [recs[w % len(recs)] for w in range(case['worlds'])]
    rng = np.random.default_rng([seed, 99])
    nb = sum(r['n'] for r in recs)
    start = np.concatenate([r['bodies'].reshape(-1, 13) for r in recs])
    dyn = start[:, 11] > 0
    params = np.zeros((nb, 8))
    params[:, :2] = rng.uniform(-1, 1, (nb, 2))
    params[:, 2] = rng.uniform(-0.2, 0.2, nb)
    params[:, 3:6] = rng.uniform(-0.5, 0.5, (nb, 3))
    params[:, 6] = 0.512 * rng.uniform(0.5, 2.0, nb)
    params *= dyn[:, None]
    params[:, 7] = np.where(dyn, rng.uniform(0.3, 0.8, nb), 0.5)
    target = start[:, :7] + np.where(dyn[:, None], rng.normal(0.0, 0.2, (nb, 7)), 0.0)
    return recs, params.reshape(-1), target.reshape(-1)


def _rays(case, seed):
    """Rays from around and above a pile into it."""
    bodies = _pile([case['bodies']], seed, case['spheres'])
    rng = np.random.default_rng([seed, 5])
    n = case['rays']
    lo, hi = bodies['pos'][1:].min(0), bodies['pos'][1:].max(0)
    origin = np.stack([rng.uniform(lo[0] - 2, hi[0] + 2, n), rng.uniform(lo[1] - 2, hi[1] + 2, n), rng.uniform(hi[2] + 1, hi[2] + 6, n)], 1)
    aim = rng.uniform(lo, hi, (n, 3))
    d = (aim - origin) * rng.uniform(0.5, 2.0, (n, 1))
    return bodies, origin.astype(np.float32), d.astype(np.float32)


def _pinned(n):
    t = torch.empty(n * avbd_b200.BODY_DTYPE.itemsize, dtype=torch.uint8, pin_memory=True)
    return t, t.numpy().view(avbd_b200.BODY_DTYPE)


def _world(bodies, params, joints=None, info=None, shapes=()):
    w = avbd_b200.CudaSolver3D(body_capacity=len(bodies), joint_capacity=len(joints) if joints is not None else None)
    w.params = params
    for h in shapes:
        w.add_hull(h.packed)
    w.add_bodies(bodies)
    if joints is not None:
        w.add_joints(joints, info)
    return w


def prepare(case, seed):
    kind = case['kind']
    if kind in ('step', 'host'):
        bodies = _pile([case['bodies']], seed, case['spheres'], 1 if case['rules'] == 'world' else 2)
        w = _world(bodies, _params(case['rules'], case['iterations']))
        if kind == 'step':
            return {'kind': kind, 'world': w, 'out': _views(w)}
        hold, records = _pinned(len(bodies))
        records[:] = bodies
        return {'kind': kind, 'world': w, 'hold': hold, 'records': records}
    if kind == 'chains':
        bodies, joints, info, shapes = _chains(case, seed)
        w = _world(bodies, _params('reference', case['iterations']), joints, info, shapes)
        return {'kind': 'step', 'world': w, 'out': _views(w)}
    if kind == 'batch':
        counts = _world_counts(case)
        bodies = _pile(counts, seed, 0.3)
        b = avbd_b200.BatchSolver3D(len(counts), len(bodies), params=_params('reference', case['iterations']))
        ends = np.cumsum(counts + 1)
        for lo, hi in zip(ends - counts - 1, ends):
            b.add_world(bodies[lo:hi])
        if case['shape'] == 'tuned':  # what avbd_batch_tune settles on for many worlds of this size
            b.set_launch(128, 0, 4, 64)
        hold, records = _pinned(len(bodies))
        return {'kind': kind, 'batch': b, 'steps': case['steps'], 'hold': hold, 'records': records}
    if kind == 'rays':
        bodies, origin, d = _rays(case, seed)
        return {'kind': kind, 'world': _world(bodies, _params('reference', 10)), 'origin': origin, 'direction': d}
    recs, params, target = _adjoint_inputs(case, seed)
    a = avbd_b200.Adjoint(recs, checkpoint=10)
    a.set_target(target)
    return {'kind': kind, 'adjoint': a, 'params': params}


def _fields(r):
    return {'pos': r['pos'], 'rot': r['rot'], 'vel': r['vel'], 'ang': r['ang_vel']}


def run(state):
    kind = state['kind']
    if kind == 'step':
        state['world'].step()
        return state['out']
    if kind == 'host':
        state['world'].write_bodies_async(state['records'])
        state['world'].step()
        state['world'].read_bodies_into(state['records'])
        return _fields(state['records'])
    if kind == 'batch':
        state['batch'].step(state['steps'])
        state['batch'].read_all_bodies_into(state['records'])
        return _fields(state['records'])
    if kind == 'rays':
        h = state['world'].raycast(state['origin'], state['direction'])
        return {'body': h['body'], 'distance': h['distance'], 'point': h['point'], 'normal': h['normal']}
    loss, pose = state['adjoint'].forward(state['params'])
    loss_again, grad = state['adjoint'].backward(state['params'])
    return {'loss': loss, 'pose': pose, 'grad': grad, 'loss_again': loss_again}


def work(case):
    """Bytes: each record read and written once (a body 160 B, a contact point 64, a pair 32, a joint
    176). Flops: a point's rows seen from its two bodies each iteration and its dual, a body's 6x6
    solve, a pair's narrowphase. A pile has about 3 pairs and 7 points a body."""
    kind = case['kind']
    if kind == 'rays':
        n, r = case['bodies'], case['rays']
        return {'bytes': 64.0 * n + 64.0 * r, 'flops': 20.0 * n * r}
    if kind == 'adjoint':
        b, p = case['worlds'] * case['bodies'], case['worlds'] * case['bodies'] * 4
        # per step: the recorded structure read by the replay and by the reverse sweep
        return {'bytes': 2.0 * case['steps'] * (p * 56 + b * 96) + b * 300.0,
                'flops': float(case['steps']) * case['iterations'] * (p * 2 * (400 + 400 + 900) + b * 900)}
    if kind == 'batch':
        n, steps = float(_world_counts(case).sum()), case['steps']
    elif kind == 'chains':
        n, steps = float(case['hulls'] + case['chains'] * case['links']), 1
    else:
        n, steps = float(case['bodies']), 1
    pairs, points, joints = 3.0 * n, 7.0 * n, 0.0
    if kind == 'chains':
        pairs, points, joints = 2.0 * case['hulls'], 4.0 * case['hulls'], float(case['chains'] * case['links'])
    it = case['iterations']
    flops = it * (points * 3 * 250 + joints * 3 * 500 + n * 300) + pairs * 1500
    moved = 2 * (n * 160 + points * 64 + pairs * 32 + joints * 176)
    return {'bytes': steps * moved + (2 * 160.0 * n if kind in ('host', 'batch') else 0.0), 'flops': steps * flops}


# --- the same in 64 bits -------------------------------------------------------------------------------

D = torch.float64


def exact(case, seed):
    kind = case['kind']
    if kind in ('step', 'host') and case['bodies'] <= 3500:
        up = 1 if case['rules'] == 'world' else 2
        bodies = _pile([case['bodies']], seed, case['spheres'], up)
        return _exact_steps(bodies, [len(bodies)], case['rules'], case['iterations'], up)
    if kind == 'batch' and case['steps'] == 1 and case['worlds'] * case['median'] <= 6500:
        counts = _world_counts(case)
        return _exact_steps(_pile(counts, seed, 0.3), counts + 1, 'reference', case['iterations'], 2)
    if kind == 'rays':
        return _exact_rays(*_rays(case, seed))
    if kind == 'adjoint' and case['worlds'] * case['bodies'] * case['steps'] <= 20000:
        return _exact_adjoint(case, seed)
    return None  # the narrowphase of so many pairs (or of hulls), or many steps' warm starts: too slow here


def _cross(a, b):
    return torch.linalg.cross(a, b, dim=-1)


def _qmul(a, b):
    ax, ay, az, aw = a.unbind(-1)
    bx, by, bz, bw = b.unbind(-1)
    return torch.stack([aw * bx + ax * bw + ay * bz - az * by, aw * by - ax * bz + ay * bw + az * bx, aw * bz + ax * by - ay * bx + az * bw,
                        aw * bw - ax * bx - ay * by - az * bz], -1)


def _rotate(q, v):
    u = q[..., :3]
    t = 2.0 * _cross(u, v)
    return v + q[..., 3:] * t + _cross(u, t)


def _qadd(q, v):
    s = q + 0.5 * _qmul(torch.cat([v, torch.zeros_like(v[..., :1])], -1), q)
    return s / s.norm(dim=-1, keepdim=True)


def _qsub(a, b):
    inv = b * torch.tensor([-1.0, -1.0, -1.0, 1.0], dtype=D) / (b * b).sum(-1, keepdim=True)
    return 2.0 * _qmul(a, inv)[..., :3]


def _ldlt_solve(A, b):
    """Each 6x6 system by LDL^T with every pivot kept above 1e-5 of its diagonal entry."""
    L = [[None] * 6 for _ in range(6)]
    Dg = [None] * 6
    for j in range(6):
        d = A[:, j, j]
        for k in range(j):
            d = d - L[j][k] ** 2 * Dg[k]
        Dg[j] = d if j == 0 else torch.maximum(d, A[:, j, j] * 1e-5)
        for i in range(j + 1, 6):
            s = A[:, i, j]
            for k in range(j):
                s = s - L[i][k] * L[j][k] * Dg[k]
            L[i][j] = s / Dg[j]
    y = []
    for i in range(6):
        s = b[:, i]
        for k in range(i):
            s = s - L[i][k] * y[k]
        y.append(s)
    x = [None] * 6
    for i in reversed(range(6)):
        s = y[i] / Dg[i]
        for k in range(i + 1, 6):
            s = s - L[k][i] * x[k]
        x[i] = s
    return torch.stack(x, 1)


def _rows(pt, dl, r, q, pen, lam, alpha):
    """The points' constraint values and forces at displacements dl and rotations r since the step's
    start (q: the whole rotation)."""
    a, b = pt['a'], pt['b']
    roll = pt['rolling'][:, None]
    raw = _rotate(torch.where(roll, pt['q0'][a], q[a]), pt['ra'])
    rbw = _rotate(torch.where(roll, pt['q0'][b], q[b]), pt['rb'])
    dp = dl[a] - dl[b] + _cross(2.0 * r[a, :3], raw) - _cross(2.0 * r[b, :3], rbw)
    C = pt['c0'] * (1.0 - alpha) + (pt['basis'] * dp[:, None]).sum(-1)
    F = pen * C + lam
    fx = torch.clamp(F[:, 0], max=0.0)
    bound = fx.abs() * pt['mu']
    f2 = F[:, 1] ** 2 + F[:, 2] ** 2
    slide = f2.detach().sqrt() > bound.detach()
    scale = torch.where(slide, bound / torch.where(slide, f2, torch.ones_like(f2)).sqrt(), torch.ones_like(f2))
    return raw, rbw, C, torch.stack([fx, F[:, 1] * scale, F[:, 2] * scale], 1), slide


def _iterate(pt, colors, mass, moment, ylin, yrot, dl, r, q0, pen, lam, P):
    """The coloured Newton sweeps and duals of one step; every body's displacement and rotation, and the
    points' penalties and multipliers, after them."""
    dt2 = P['dt'] ** 2
    q = _qmul(r, q0)
    plan = []
    for c in range(int(colors.max()) + 1 if len(colors) else 0):
        body = torch.nonzero(colors == c).flatten()
        if not len(body):
            continue
        where = torch.full((len(colors),), -1, dtype=torch.long)
        where[body] = torch.arange(len(body))
        pa, pb = torch.nonzero(where[pt['a']] >= 0).flatten(), torch.nonzero(where[pt['b']] >= 0).flatten()
        use = torch.cat([pa, pb])
        slot = torch.cat([where[pt['a'][pa]], where[pt['b'][pb]]])
        sign = torch.cat([torch.ones(len(pa), dtype=D), -torch.ones(len(pb), dtype=D)])
        sub = {k: (v[use] if k not in ('q0',) else v) for k, v in pt.items()}
        plan.append((body, use, slot, sign, sub))
    for _ in range(P['iterations']):
        for body, use, slot, sign, sub in plan:
            raw, rbw, _, F, _ = _rows(sub, dl, r, q, pen[use], lam[use], P['alpha'])
            arm = torch.where(sign[:, None] > 0, raw, rbw)
            lin = sub['basis'] * sign[:, None, None]
            J = torch.cat([lin, _cross(arm[:, None].expand_as(lin), lin)], -1)
            H = torch.zeros(len(body), 6, 6, dtype=D).index_add(0, slot, torch.einsum('pk,pki,pkj->pij', pen[use], J, J))
            g = torch.zeros(len(body), 6, dtype=D).index_add(0, slot, torch.einsum('pk,pki->pi', F, J))
            diag = torch.cat([mass[body, None].expand(-1, 3), moment[body]], 1) / dt2
            H = H + torch.diag_embed(diag)
            g = g + diag * torch.cat([dl[body] - ylin[body], _qsub(r[body], yrot[body])], 1)
            x = _ldlt_solve(H, g)
            dl = dl.index_copy(0, body, dl[body] - x[:, :3])
            r = r.index_copy(0, body, _qadd(r[body], -x[:, 3:]))
            q = _qmul(r, q0)
        _, _, C, F, slide = _rows(pt, dl, r, q, pen, lam, P['alpha'])
        ramp = torch.stack([F[:, 0] < 0, ~slide, ~slide], 1)
        pen = torch.where(ramp, torch.clamp(pen + P['beta_lin'] * C.abs(), max=1e10), pen)
        lam = F
    return dl, r, pen, lam


def _hash32(x):
    x = np.asarray(x, dtype=np.uint64) & 0xFFFFFFFF
    x ^= x >> 16
    x = (x * 0x7FEB352D) & 0xFFFFFFFF
    x ^= x >> 15
    x = (x * 0x846CA68B) & 0xFFFFFFFF
    return x ^ (x >> 16)


def _colors(n, dynamic, edges):
    """Jones-Plassmann by the hashed index: a body takes the least colour its neighbours of higher
    priority left free."""
    near = [[] for _ in range(n)]
    for a, b in edges:
        near[a].append(b)
        near[b].append(a)
    pri = _hash32(np.arange(n) + 0x9E3779B9)
    color = np.full(n, -1)
    for i in sorted(np.flatnonzero(dynamic), key=lambda i: (-int(pri[i]), -int(i))):
        taken = {color[j] for j in near[i]}
        color[i] = next(c for c in range(64) if c not in taken)
    return color


def _collide_boxes(ca, ha, Ra, cb, hb, Rb, face_bias):
    """Box against box: the axis of least penetration (columns of R are a box's axes), then the incident
    face clipped to the reference face, or two edges' closest points. (normal from A to B, points)"""
    delta = cb - ca
    cand = []
    for kind, axes in (('A', Ra.T), ('B', Rb.T), ('E', [np.cross(Ra[:, i], Rb[:, j]) for i in range(3) for j in range(3)])):
        for k, ax in enumerate(axes):
            l2 = ax @ ax
            if l2 < 1e-6:
                continue
            n = ax / math.sqrt(l2)
            if n @ delta < 0:
                n = -n
            sep = abs(delta @ n) - (ha @ np.abs(n @ Ra) + hb @ np.abs(n @ Rb))
            if sep > 0:
                return None
            cand.append((kind, k, sep, n))
    face = max((c for c in cand if c[0] != 'E'), key=lambda c: c[2])
    best = face
    edges = [c for c in cand if c[0] == 'E']
    if edges:
        e = max(edges, key=lambda c: c[2])
        if (e[2] > 0.95 * face[2] + 0.01) if face_bias else (0.95 * e[2] > face[2] + 0.01):
            best = e
    kind, k, _, n = best
    points = []

    def keep(xa, xb):
        if len(points) < 8 and all(((xa + xb - u - v) * 0.5) @ ((xa + xb - u - v) * 0.5) >= 1e-6 for u, v in points):
            points.append((xa, xb))

    sgn = lambda v: np.where(v >= 0, 1.0, -1.0)
    if kind == 'E':
        ia, ib = divmod(k, 3)

        def edge(c, h, R, i, d):
            s = sgn(d @ R) * h
            s[i] = 0.0
            mid = c + R @ s
            return mid - R[:, i] * h[i], mid + R[:, i] * h[i]

        p0, p1 = edge(ca, ha, Ra, ia, n)
        q0, q1 = edge(cb, hb, Rb, ib, -n)
        d1, d2, w = p1 - p0, q1 - q0, p0 - q0
        a, e, f, c, b = d1 @ d1, d2 @ d2, d2 @ w, d1 @ w, d1 @ d2
        den = a * e - b * b
        s = min(max((b * f - c * e) / den, 0.0), 1.0) if abs(den) > 1e-6 else 0.0
        t = (b * s + f) / e
        if t < 0:
            t, s = 0.0, min(max(-c / a, 0.0), 1.0)
        elif t > 1:
            t, s = 1.0, min(max((b - c) / a, 0.0), 1.0)
        keep(p0 + d1 * s, q0 + d2 * t)
    else:
        is_a = kind == 'A'
        (cr, hr, Rr), (ci, hi, Ri) = ((ca, ha, Ra), (cb, hb, Rb)) if is_a else ((cb, hb, Rb), (ca, ha, Ra))
        out = n if is_a else -n
        rn = Rr[:, k] * (1.0 if out @ Rr[:, k] >= 0 else -1.0)
        rc = cr + rn * hr[k]
        inc = int(np.argmax(np.abs(rn @ Ri)))
        fn = Ri[:, inc] * (-1.0 if Ri[:, inc] @ rn > 0 else 1.0)
        fc = ci + fn * hi[inc]
        u, v = [j for j in range(3) if j != inc]
        poly = [fc + Ri[:, u] * (su * hi[u]) + Ri[:, v] * (sv * hi[v]) for su, sv in ((1, 1), (-1, 1), (-1, -1), (1, -1))]
        for j in [j for j in range(3) if j != k]:
            for s in (1.0, -1.0):
                pn = Rr[:, j] * s
                off = pn @ rc + hr[j]
                nxt = []
                for i in range(len(poly)):
                    x, y = poly[i - 1], poly[i]
                    dx, dy = pn @ x - off, pn @ y - off
                    if (dx <= 1e-5) != (dy <= 1e-5):
                        t = min(max(dx / (dx - dy), 0.0), 1.0) if abs(dx - dy) > 1e-6 else 0.0
                        nxt.append(x + (y - x) * t)
                    if dy <= 1e-5:
                        nxt.append(y)
                poly = nxt
        if not poly:
            return n, []
        for p in poly:
            d = (p - rc) @ rn
            if d <= 1e-5:
                on = p - rn * d
                keep(on if is_a else p, p if is_a else on)
    if not points:
        points.append((ca + Ra @ (sgn(n @ Ra) * ha), cb + Rb @ (sgn(-n @ Rb) * hb)))
    return n, points


def _collide(i, j, pos, half, R, sphere, face_bias):
    if sphere[i] and sphere[j]:
        d = pos[j] - pos[i]
        dist = math.sqrt(d @ d)
        if dist > half[i][0] + half[j][0]:
            return None
        n = d / dist
        return n, [(pos[i] + n * half[i][0], pos[j] - n * half[j][0])]
    if sphere[i] or sphere[j]:
        s, x = (i, j) if sphere[i] else (j, i)
        p = (pos[s] - pos[x]) @ R[x]
        c = np.clip(p, -half[x], half[x])
        if (p != c).any():
            dist = math.sqrt((p - c) @ (p - c))
            if dist > half[s][0]:
                return None
            nl = (p - c) / dist
        else:
            k = int(np.argmin(half[x] - np.abs(p)))
            nl = np.zeros(3)
            nl[k] = 1.0 if p[k] >= 0 else -1.0
            c = c.copy()
            c[k] = nl[k] * half[x][k]
        out = R[x] @ nl
        on_s, on_x = pos[s] - out * half[s][0], pos[x] + R[x] @ c
        return (-out, [(on_s, on_x)]) if s == i else (out, [(on_x, on_s)])
    return _collide_boxes(pos[i], half[i], R[i], pos[j], half[j], R[j], face_bias)


def _exact_steps(bodies, counts, rules, iterations, up):
    """One step of fresh worlds (no contact history)."""
    p = _params(rules, iterations)
    P = dict(dt=float(p.dt), iterations=iterations, alpha=float(p.alpha), beta_lin=float(p.beta_lin))
    f8 = lambda name: bodies[name].astype(np.float64)
    pos, rot, half, mass, vel, ang = f8('pos'), f8('rot'), f8('size') / 2, f8('mass'), f8('vel'), f8('ang_vel')
    eye = np.eye(3)
    R = np.stack([_turn(rot, np.tile(e, (len(rot), 1))) for e in eye], -1)
    sphere = bodies['shape'] == 1
    reach = np.where(sphere[:, None], half, (np.abs(R) * half[:, None]).sum(-1))
    found, color = [], np.full(len(pos), -1)
    lo = 0
    for n in counts:
        hi = lo + int(n)
        edges = set()
        for b in range(lo, hi):
            over = (np.abs(pos[b + 1:hi] - pos[b]) <= reach[b + 1:hi] + reach[b] + 1e-4).all(1) & ((mass[b + 1:hi] > 0) | (mass[b] > 0))
            for a in b + 1 + np.flatnonzero(over):
                hit = _collide(a, b, pos, half, R, sphere, bool(p.flags & FLAG_FACE_BIAS))
                if hit is None or not hit[1]:
                    continue
                if mass[a] > 0 and mass[b] > 0:
                    edges.add((a - lo, b - lo))
                for xa, xb in hit[1]:
                    found.append((a, b, -hit[0], R[a].T @ (xa - pos[a]), R[b].T @ (xb - pos[b])))
        color[lo:hi] = _colors(hi - lo, mass[lo:hi] > 0, edges)
        lo = hi
    a, b = np.array([f[0] for f in found], np.int64), np.array([f[1] for f in found], np.int64)
    n, ra, rb = (np.array([f[k] for f in found]).reshape(-1, 3) for k in (2, 3, 4))
    t1 = np.where((np.abs(n[:, 0]) > np.abs(n[:, 2]))[:, None], np.stack([-n[:, 1], n[:, 0], 0 * n[:, 0]], 1), np.stack([0 * n[:, 0], -n[:, 2], n[:, 1]], 1))
    t1 /= np.linalg.norm(t1, axis=1, keepdims=True)
    basis = np.stack([n, t1, np.cross(n, t1)], 1)
    d = pos[a] - pos[b] + (R[a] @ ra[..., None])[..., 0] - (R[b] @ rb[..., None])[..., 0]
    c0 = (basis * d[:, None]).sum(-1) + np.array([float(p.contact_margin), 0.0, 0.0])
    fr = f8('friction')
    T = lambda x: torch.from_numpy(np.ascontiguousarray(x))
    q0 = T(rot)
    pt = dict(a=T(a), b=T(b), ra=T(ra), rb=T(rb), basis=T(basis), c0=T(c0), mu=T(np.sqrt(fr[a] * fr[b])), rolling=T(sphere[a] | sphere[b]), q0=q0)
    least = np.ones(len(a))
    if p.flags & FLAG_MASS_PENALTY:
        m = np.where(mass > 0, mass, np.inf)
        least = np.clip(np.minimum(m[a], m[b]) / P['dt'] ** 2, 1.0, 1e10)
    pen = T(np.stack([least, np.ones(len(a)), np.ones(len(a))], 1))
    dynamic = mass > 0
    fall = np.zeros(3)
    fall[up] = float(p.gravity) * P['dt'] ** 2
    turn = _qadd(torch.tensor([[0.0, 0.0, 0.0, 1.0]], dtype=D).expand(len(rot), 4), T(ang * P['dt']))
    move = dynamic.copy()
    if p.flags & FLAG_START_AT_REST:
        move &= ~(np.linalg.norm(vel, axis=1) + np.linalg.norm(ang, axis=1) * f8('radius') < 0.1)
    gain = np.clip((vel[:, up] - f8('prev_up_vel')) / P['dt'] * np.sign(p.gravity) / abs(p.gravity), 0.0, 1.0)
    dl = T(np.where(move[:, None], vel * P['dt'] + gain[:, None] * fall, 0.0))
    still = torch.zeros(len(rot), 4, dtype=D)
    still[:, 3] = 1.0
    r = torch.where(T(move)[:, None], turn, still)
    ylin = T(vel * P['dt'] + fall * dynamic[:, None])
    dl, r, pen, lam = _iterate(pt, T(color), T(mass), T(f8('moment')), ylin, turn, dl, r, q0, pen, torch.zeros_like(pen), P)
    q = _qmul(r, q0)
    dyn = T(dynamic)[:, None]
    q = torch.where(dyn, q / q.norm(dim=1, keepdim=True), q0)
    return {'pos': T(pos) + dl, 'rot': q, 'vel': torch.where(dyn, dl / P['dt'], T(vel)), 'ang': torch.where(dyn, 2.0 * r[:, :3] / P['dt'], T(ang))}


def _exact_rays(bodies, origin, direction):
    f8 = lambda name: bodies[name].astype(np.float64)
    pos, rot, half, radius, sphere = f8('pos'), f8('rot'), f8('size') / 2, f8('radius'), bodies['shape'] == 1
    o = origin.astype(np.float64)
    d = direction.astype(np.float64)
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    n = len(o)
    distance, point, normal = np.full(n, -1.0), np.zeros((n, 3)), np.zeros((n, 3))
    for k in range(n):
        rel = pos - o[k]
        along = rel @ d[k]
        near = np.flatnonzero((rel * rel).sum(1) - along * along <= radius * radius * (1 + 1e-9))
        q = rot[near] * [-1, -1, -1, 1]
        lo, ld = _turn(q, -rel[near]), _turn(q, np.tile(d[k], (len(near), 1)))
        with np.errstate(divide='ignore', invalid='ignore'):
            b = (lo * ld).sum(1)
            disc = b * b - (lo * lo).sum(1) + half[near, 0] ** 2
            ts = np.where(disc >= 0, -b - np.sqrt(np.maximum(disc, 0)), np.inf)
            t0, t1 = (-half[near] - lo) / ld, (half[near] - lo) / ld
            enter, leave = np.minimum(t0, t1), np.maximum(t0, t1)
            axis = np.argmax(enter, 1)
            tb = np.where(enter.max(1) <= leave.min(1), enter.max(1), np.inf)
        t = np.where(sphere[near], ts, tb)
        t = np.where(t >= 0, t, np.inf)
        if not len(t) or not np.isfinite(t.min()):
            continue
        h = int(np.argmin(t))
        local = (lo[h] + ld[h] * t[h]) / half[near[h], 0] if sphere[near[h]] else -np.sign(ld[h]) * (np.arange(3) == axis[h])
        distance[k] = t[h]
        point[k] = o[k] + d[k] * t[h]
        normal[k] = _turn(rot[near[h]], local)
    return {'body': None, 'distance': distance, 'point': point, 'normal': normal}


def _exact_adjoint(case, seed):
    recs, params, target = _adjoint_inputs(case, seed)
    P = recs[0]['params']
    base = np.cumsum([0] + [r['n'] for r in recs])
    nb = int(base[-1])
    start = torch.from_numpy(np.concatenate([r['bodies'].reshape(-1, 13) for r in recs]))
    world = torch.from_numpy(np.repeat(np.arange(len(recs)), [r['n'] for r in recs]))
    theta = torch.from_numpy(params.reshape(-1, 8).copy()).requires_grad_(True)
    dyn = start[:, 11:12] > 0
    x, q = start[:, :3], start[:, 3:7]
    vel, ang = theta[:, :3] * dyn, theta[:, 3:6] * dyn
    before = start[:, 7]
    mass = torch.where(dyn[:, 0], theta[:, 6], torch.ones(nb, dtype=D))
    moment = start[:, 8:11] * mass[:, None]
    mu = torch.where(dyn[:, 0], theta[:, 7], start[:, 12])
    # every step has the same contacts: the first step's, over all worlds
    man = [r['man_bodies'].reshape(-1, 2)[:r['n'] - 1] + b for r, b in zip(recs, base)]
    a, b = (torch.from_numpy(np.repeat(np.concatenate(man)[:, k], 4)) for k in (0, 1))
    basis = torch.from_numpy(np.repeat(np.concatenate([r['basis'].reshape(-1, 3, 3)[:r['n'] - 1] for r in recs]), 4, 0))
    anchors = torch.from_numpy(np.concatenate([r['anchors'].reshape(-1, 6)[:4 * (r['n'] - 1)] for r in recs]))
    colors = torch.from_numpy(np.concatenate([r['colors'][:r['n']] for r in recs]).astype(np.int64))
    pen, lam = torch.zeros(len(a), 3, dtype=D), torch.zeros(len(a), 3, dtype=D)
    dt, g = P['dt'], P['gravity']
    fall = torch.tensor([0.0, 0.0, g * dt * dt], dtype=D)
    for _ in range(case['steps']):
        lam, pen = lam * (P['alpha'] * P['gamma']), torch.clamp(pen * P['gamma'], 1.0, 1e10)
        d = (_rotate(q[a], anchors[:, :3]) + x[a]) - (_rotate(q[b], anchors[:, 3:]) + x[b])
        c0 = (basis * d[:, None]).sum(-1) + torch.tensor([P['contact_margin'], 0.0, 0.0], dtype=D)
        pt = dict(a=a, b=b, ra=anchors[:, :3], rb=anchors[:, 3:], basis=basis, c0=c0, mu=(mu[a] * mu[b]).sqrt(),
                  rolling=torch.zeros(len(a), dtype=torch.bool), q0=q)
        gain = torch.clamp((vel[:, 2] - before) / dt * math.copysign(1.0, g) / abs(g), 0.0, 1.0)
        one = torch.tensor([0.0, 0.0, 0.0, 1.0], dtype=D).expand(nb, 4)
        turn = torch.where(dyn, _qadd(one, ang * dt), one)
        ylin = (vel * dt + fall) * dyn
        dl = (vel * dt + fall * gain[:, None]) * dyn
        dl, r, pen, lam = _iterate(pt, colors, mass, moment, ylin, turn, dl, turn, q, pen, lam, P)
        before = vel[:, 2]
        vel, ang = dl / dt, 2.0 * r[:, :3] / dt
        x, q = x + dl, _qmul(r, q)
    pose = torch.cat([x, q], 1)
    off = ((pose - torch.from_numpy(target.reshape(-1, 7))) * dyn) ** 2
    loss = torch.zeros(len(recs), dtype=D).index_add(0, world, off.sum(1))
    loss.sum().backward()
    grad = (theta.grad * dyn).reshape(-1)
    return {'loss': loss.detach(), 'pose': pose.detach(), 'grad': grad, 'loss_again': loss.detach()}
