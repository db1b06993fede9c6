"""The passes a World runs around the step, through the C ABI, against their CPU restatement
(oracle/queries.py) on the same f32 records: impulses on bodies (Pusher, src/lib/push.ts), contact
begin/end events (ContactWatch, src/lib/contacts.ts) and nearest-hit raycasts (Raycaster,
src/lib/raycast.ts)."""

import numpy as np
import pytest

import avbd_b200
from avbd_b200 import _abi
from avbd_b200.scenes import Scene, drop_pile, hull_pile
import queries

pytestmark = pytest.mark.gpu


def test_pushes_match_oracle(cuda_lib):
    scene = drop_pile(400, seed=3, spacing=1.6, layers=3)
    w = avbd_b200.CudaSolver3D(scene)
    w.step(20)
    w.set_lifecycle(7, 2)  # disabled: left alone
    before = w.read_bodies()
    rng = np.random.default_rng(1)
    others = np.setdiff1d(np.arange(len(before)), [0, 7])
    # the static ground and the disabled body are left alone; 58 others are pushed
    slots = np.concatenate([[0, 7], rng.choice(others, size=58, replace=False)])
    p = np.zeros(len(slots), dtype=_abi.PUSH_DTYPE)
    p['body'] = slots
    p['lin'] = rng.normal(0, 5, (len(slots), 3))
    p['off_lin'] = p['lin'] * rng.uniform(0, 1, (len(slots), 1))
    at = before['pos'][slots] + rng.normal(0, 0.3, (len(slots), 3))
    p['moment'] = np.cross(at, p['off_lin']) + rng.normal(0, 0.5, (len(slots), 3))
    w.apply_pushes(p)
    after = w.read_bodies()
    vel, avel = queries.apply_pushes(before, p)
    assert np.allclose(after['vel'], vel, rtol=1e-5, atol=1e-5) and np.allclose(after['ang_vel'], avel, rtol=1e-5, atol=1e-4)
    assert np.array_equal(after['vel'][[0, 7]], before['vel'][[0, 7]])
    moved = np.abs(after['vel'] - before['vel']).max(axis=1) > 0
    assert moved.sum() == len(slots) - 2
    for bad in (np.r_[p[:2], p[:1]], p[:1].copy()):
        if len(bad) == 1:
            bad['body'] = len(before)  # not a slot
        with pytest.raises(avbd_b200.AvbdError):
            w.apply_pushes(bad)
    w.destroy()


def _bouncing_boxes():
    s = Scene('boxes dropped and kicked')
    s.box([40, 40, 1], 0, 0.5, [0, 0, -0.5])
    for k in range(24):
        s.box([0.6, 0.6, 0.6], 1, 0.5, [(k % 6) * 1.5 - 4, (k // 6) * 1.5 - 2, 0.8 + 0.4 * (k % 3)])
    return s


def test_contact_events_match_oracle(cuda_lib):
    """24 boxes land (begins), some are kicked up off the ground (ends) and land again (begins); half
    of them report. Every event, its step, point, impulse and normal against the restatement run on
    the same contacts read back after each step."""
    s = _bouncing_boxes()
    w = avbd_b200.CudaSolver3D(s)
    n = len(s.bodies)
    watch = w.contact_watch(pairs=256, capacity=4096)
    ids = np.arange(n) + 100
    on = (np.arange(n) % 2 == 1)
    on[0] = False  # the ground does not report; its pairs with reporting boxes do
    watch.set_watched(np.arange(n), ids, on)
    model = {i: (int(ids[i]), bool(on[i])) for i in range(n)}
    dt = s.params.dt
    prev, want = set(), []
    for step in range(1, 121):
        if step == 50:  # the reporting boxes kicked up at 4 m/s: they leave the ground and land again
            b = w.read_bodies()
            kick = np.zeros(12, dtype=_abi.PUSH_DTYPE)
            kick['body'] = np.arange(1, 25, 2)
            kick['lin'][:, 2] = 4.0 * b['mass'][kick['body']]
            w.apply_pushes(kick)
        w.step()
        watch.run(step, dt)
        m, c = w.read_contacts()
        events, prev = queries.contact_events(prev, m, c, w.read_bodies(), model, step, dt)
        want += events
    got, dropped, full = watch.read()
    assert dropped == 0 and not full
    kinds = {k: sum(1 for e in want if e[0] == k) for k in (1, 2)}
    assert kinds[1] >= 20 and kinds[2] >= 10, kinds
    key = lambda e: (e[3], e[0], e[1], e[2])
    want.sort(key=key)
    got_l = sorted(got.tolist(), key=lambda e: (e[3], e[0], e[1], e[2]))
    assert [key(e) for e in want] == [(e[3], e[0], e[1], e[2]) for e in got_l]
    for wv, g in zip(want, got_l):
        if wv[0] == 1:
            assert np.allclose(g[4], wv[4], atol=1e-5) and abs(g[5] - wv[5]) <= 1e-5 * max(1.0, wv[5]) and np.allclose(g[6], wv[6], atol=1e-6)
    assert np.all(np.diff(got['step'].astype(np.int64)) >= 0)  # read gives step order
    # a capacity too small drops the rest and says how many
    small = w.contact_watch(pairs=256, capacity=2)
    small.set_watched(np.arange(n), ids, np.ones(n, bool))
    w.step()
    small.run(121, dt)
    ev, dropped, _ = small.read()
    assert len(ev) == 2 and dropped > 0
    small.destroy()
    watch.destroy()
    w.destroy()


def test_raycast_matches_oracle(cuda_lib):
    """Rays among hulls, boxes and spheres: the nearest body (the lowest slot on a tie), its distance
    and the world normal there; rays from inside a body; a distance cap; ignored slots and a group mask."""
    s = hull_pile(90, seed=4)
    w = avbd_b200.CudaSolver3D(s)
    w.step(40)
    bodies = w.read_bodies()
    rng = np.random.default_rng(7)
    n = 300
    origins = rng.uniform(-6, 6, (n, 3)) + np.array([0, 0, 3.0])
    origins[:20] = bodies['pos'][1:21]  # inside bodies: distance 0
    directions = rng.normal(0, 1, (n, 3))
    maxd = np.where(rng.uniform(size=n) < 0.2, rng.uniform(0.5, 3, n), 3.0e38).astype(np.float32)
    groups = np.ones(len(bodies), np.uint32)
    groups[5:15] = 2
    w.set_filters(0, np.stack([groups, np.full(len(bodies), 0xFFFFFFFF, np.uint32)], axis=1))
    filters = np.stack([groups, groups], axis=1)
    ignore = [3, 30, 31]
    for mask in (0xFFFFFFFF, 1):
        hits = w.raycast(origins, directions, maxd, ignore=ignore, mask=mask)
        rays = np.zeros(n, _abi.RAY_DTYPE)  # the f32 inputs the device traced
        rays['origin'], rays['direction'], rays['max_distance'] = origins, directions, maxd
        agree = 0
        for k in range(n):
            d = rays['direction'][k].astype(float)
            d = (d / np.linalg.norm(d)).astype(np.float32)
            want = queries.raycast(bodies, s.hull_words, filters, rays['origin'][k], d, float(rays['max_distance'][k]), ignore=ignore, mask=mask)
            h = hits[k]
            if want is None:
                assert h['body'] == -1, f'ray {k}: hit {h["body"]}, none expected'
                continue
            b, t, nrm = want
            assert h['body'] >= 0, f'ray {k}: no hit, body {b} expected'
            assert abs(h['distance'] - t) <= 1e-5 * max(1.0, t), f'ray {k}: distance {h["distance"]} vs {t}'
            if h['body'] == b:
                if not np.allclose(h['normal'], nrm, atol=1e-4):  # faces that tie, or a grazing ray on a sphere
                    ties = queries.normals_at(bodies[b], s.hull_words, rays['origin'][k], d, float(h['distance']), 1e-5 * max(1.0, t))
                    assert any(np.allclose(h['normal'], m, atol=1e-4) for m in ties), f'ray {k}: normal {h["normal"]} vs {nrm}'
                agree += 1
            else:  # only where two surfaces lie at the same distance
                other = queries.ray_trace(bodies[h['body']], s.hull_words, rays['origin'][k], d, float(rays['max_distance'][k]))
                assert other is not None and abs(other[0] - t) <= 1e-5 * max(1.0, t)
            assert h['body'] not in ignore and (groups[h['body']] & mask)
        assert agree > n // 4
    with pytest.raises(avbd_b200.AvbdError):
        w.raycast(origins[:1], directions[:1], ignore=list(range(17)))
    w.destroy()


@pytest.mark.parametrize('n, rays', [(1, 1), (31, 9), (255, 63), (1022, 65), (1023, 40), (1024, 40), (1100, 4800)])
def test_raycast_tiles_and_far_origins(cuda_lib, n, rays):
    """Rays at the edges of the ray and body tiles, from near and from 2 km away, on long, flat and
    unnormalised bodies: all in one call as in calls of 32, and a sample of the distances against the
    restatement (f32 rounds a ray's offset from a body to 2^-23 of the distance, a few times over)."""
    rng = np.random.default_rng(n)
    scene = drop_pile(n, seed=4, spacing=1.6, layers=3)
    for b in scene.bodies[1::3]:
        b.size = [float(x) for x in rng.uniform(0.02, 1.5, 3)] if b.shape == 0 else b.size
    for b in scene.bodies[1::5]:
        b.rot = [1.3 * x for x in b.rot]
    w = avbd_b200.CudaSolver3D(scene)
    bodies = w.read_bodies()
    at = bodies['pos'][rng.integers(0, n + 1, rays)] + rng.normal(0, 0.3, (rays, 3))
    d = rng.standard_normal((rays, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o = (at - d * rng.choice([0.0, 3.0, 2000.0], (rays, 1))).astype(np.float32)
    d[0] = 0.0
    hits = w.raycast(o, d)
    parts = np.concatenate([w.raycast(o[k:k + 32], d[k:k + 32]) for k in range(0, rays, 32)])
    assert hits.tobytes() == parts.tobytes()
    filters = np.full((n + 1, 2), 0xFFFFFFFF, np.uint32)
    for k in range(0, rays, max(1, rays // 40)):
        dk = d[k].astype(np.float32).astype(float)
        dk = (dk / (np.linalg.norm(dk) or 1.0)).astype(np.float32)
        want = queries.raycast(bodies, None, filters, o[k], dk)
        tol = 1e-5 * (1.0 + float(np.abs(o[k]).max()))
        if want is None or hits['body'][k] < 0:
            # only a ray that grazes: the other view finds it within the tolerance of a surface
            grown = bodies.copy()
            grown['size'] += np.float32(20 * tol)
            assert (want is None) == (hits['body'][k] < 0) or queries.raycast(grown, None, filters, o[k], dk) is not None
        elif hits['body'][k] == want[0]:
            assert abs(hits['distance'][k] - want[1]) <= 20 * tol
    w.destroy()


def test_pose_capture_frames_match_the_world_and_round_trip(cuda_lib):
    """Pose cache frames gathered on the device every 3 steps of a pile equal the poses read back at
    those steps bit for bit, stamped with the world's step word; frames past max_frames are dropped and
    counted; the capture encodes to the pose cache format (src/bake/pose-cache.ts) and decodes to the
    same frames."""
    from avbd_b200 import pose_cache as pc
    from avbd_b200.scenes import drop_pile
    w = avbd_b200.CudaSolver3D(drop_pile(500, seed=2))
    cap = w.pose_capture(max_frames=5)
    seen, words = [], []
    for _ in range(6):
        w.step(3)
        cap.frame()
        b = w.read_bodies()
        seen.append(np.concatenate([b['pos'], b['rot']], axis=1).astype(np.float32))
        words.append(w.read_counters()['steps'])
    steps, poses, dropped = cap.read()
    assert len(steps) == 5 and dropped == 1
    assert list(steps) == words[:5]
    assert np.array_equal(poses.view(np.uint32), np.stack(seen[:5]).view(np.uint32))
    cache = cap.to_pose_cache(77, provenance={'tool': 'test'})
    manifest, chunks = pc.encode_pose_cache(cache, frames_per_chunk=2)
    back = pc.decode_pose_cache(manifest, chunks)
    assert np.array_equal(back.poses.view(np.uint32), poses.view(np.uint32)) and np.array_equal(back.steps, steps)
    assert back.bodies[0].fixed and not back.bodies[1].fixed  # the ground is static
    cap.reset()
    cap.frame()
    assert len(cap.read()[0]) == 1
    cap.destroy()
    w.destroy()


def _turned(rng, length2):
    """A random rotation scaled to the squared length, as f32."""
    q = rng.standard_normal(4)
    return (q / np.linalg.norm(q) * np.sqrt(length2)).astype(np.float32)


def _frame(q):
    """The matrix by which the trace takes a world offset into the body's frame."""
    return np.stack([queries.rotate(queries.conj(q.astype(float)), np.eye(3)[k]) for k in range(3)], 1)


@pytest.mark.parametrize('shape, length2, distance', [
    ('box', 0.9997, 2.0), ('box', 0.9991, 2.0), ('box', 0.99993, 30.0), ('box', 1.0009, 3.0),
    ('sphere', 0.9991, 2.0), ('sphere', 1.0009, 60.0), ('sphere', 1.00002, 200.0), ('sphere', 0.999995, 5.0), ('sphere', 1.0000015, 500.0)])
def test_raycast_grazes_bodies_of_inexact_rotation(cuda_lib, shape, length2, distance):
    """Rotations a little off unit length, as typed by hand, change what a ray hits: a box is as much larger or
    smaller as the rotation stretches, and a sphere more the farther the ray comes from. Rays at the edge of
    what the restatement hits, most of them outside the body's own bounding sphere. What the device finds is
    compared where the hit or miss holds for the body made smaller and larger: by 1e-4, and a sphere's squared
    radius also by ten f32 roundings of the squared distance, which its discriminant cancels."""
    rng = np.random.default_rng(17)
    size = np.array([1.0, 0.6, 0.8] if shape == 'box' else [1.0, 1.0, 1.0])
    bound = np.sqrt((size ** 2).sum()) / 2 if shape == 'box' else 0.5
    hit = outside = missed = 0
    for _ in range(12):
        s = Scene('one body')
        at = rng.uniform(-1, 1, 3)
        s.box(size, 0, 0.5, at) if shape == 'box' else s.sphere(0.5, 0, 0.5, at)
        s.bodies[0].rot = [float(x) for x in _turned(rng, length2)]
        w = avbd_b200.CudaSolver3D(s)
        body = w.read_bodies()[0]
        small, large = body.copy(), body.copy()
        slack = 1.2e-6 * distance ** 2 if shape == 'sphere' else 0.0
        small['size'] = 2 * np.sqrt(np.maximum(0.0, (size / 2 * (1 - 1e-4)) ** 2 - slack))
        large['size'] = 2 * np.sqrt((size / 2 * (1 + 1e-4)) ** 2 + slack)
        stretch = _frame(body['rot'])
        n = 120
        o, d = np.zeros((n, 3), np.float32), np.zeros((n, 3), np.float32)
        for k in range(n):
            if shape == 'box':  # past a corner, across the direction to it
                corner = np.linalg.solve(stretch, size / 2 * rng.choice([-1, 1], 3))
                across = np.cross(corner, rng.standard_normal(3))
                aim, along = corner * rng.uniform(1 - 3e-3, 1 + 1e-3), across / np.linalg.norm(across)
            else:  # past the silhouette, which the stretch moves by up to 4 |e| of the squared distance
                along, x = rng.standard_normal(3), rng.standard_normal(3)
                along /= np.linalg.norm(along)
                x -= along * (x @ along)
                extra = 4 * (length2 - 1) * distance ** 2
                aim = x / np.linalg.norm(x) * np.sqrt(0.25 * rng.uniform(0.99, 1.01) + extra * rng.uniform(0, 1.1))
            o[k] = body['pos'].astype(float) + aim - along * distance
            d[k] = along
        hits = w.raycast(o, d)
        w.destroy()
        for k in range(n):
            dk = d[k].astype(float)
            dk = (dk / np.linalg.norm(dk)).astype(np.float32)
            rel = body['pos'].astype(float) - o[k]
            perp = np.sqrt(max(0.0, rel @ rel - (rel @ dk) ** 2))
            inner, outer = (queries.ray_trace(b, None, o[k], dk, 3e38) for b in (small, large))
            if inner is not None:
                assert hits['body'][k] == 0, (k, perp)
                hit += 1
                outside += perp > bound * (1 + 1e-5)
            elif outer is None:
                assert hits['body'][k] == -1, (k, perp)
                missed += 1
    assert hit >= 100 and missed >= 100
    assert outside >= (20 if shape == 'box' and length2 < 0.9998 or shape == 'sphere' and length2 > 1 else 0)


@pytest.mark.parametrize('n, rays', [(31, 65), (400, 900), (1023, 400), (2500, 500), (1100, 4800)])
def test_raycast_passes_over_no_hit(cuda_lib, n, rays):
    """Near and far rays into a pile of long, flat, round and unnormalised bodies, against the restatement: a
    miss on the device must be one of the bodies made smaller by the tolerance, a hit one of the bodies made
    larger, and the body that the device names must lie as near as the nearest one."""
    rng = np.random.default_rng(n + rays)
    scene = drop_pile(n, seed=4, spacing=1.3, layers=3)
    for b in scene.bodies[1::3]:
        b.size = [float(x) for x in rng.uniform(0.05, 1.5, 3)] if b.shape == 0 else b.size
    for b in scene.bodies[1::4]:
        b.rot = [float(x * rng.choice([0.99985, 1.0001, 0.9, 1.3])) for x in b.rot]
    w = avbd_b200.CudaSolver3D(scene)
    bodies = w.read_bodies()
    at = bodies['pos'][rng.integers(1, n + 1, rays)] + rng.normal(0, 0.3, (rays, 3))
    d = rng.standard_normal((rays, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o = (at - d * rng.choice([0.5, 3.0, 100.0], (rays, 1))).astype(np.float32)
    hits = w.raycast(o, d)
    filters = np.full((n + 1, 2), 0xFFFFFFFF, np.uint32)
    agree = 0
    for k in range(0, rays, max(1, rays // 24)):
        dk = d[k].astype(np.float32).astype(float)
        dk = (dk / np.linalg.norm(dk)).astype(np.float32)
        # f32 rounds a ray's offset to 2^-23 of its distance, a few times over; a grazing ray moves along by
        # the root of that
        tol = 2e-6 * (1.0 + float(np.linalg.norm(o[k] - at[k])))
        small, large = bodies.copy(), bodies.copy()
        small['size'] = np.maximum(0.0, small['size'] - np.float32(20 * tol))
        large['size'] += np.float32(20 * tol)
        inner, outer = queries.raycast(small, None, filters, o[k], dk), queries.raycast(large, None, filters, o[k], dk)
        b, t = int(hits['body'][k]), float(hits['distance'][k])
        if b < 0:
            assert inner is None, f'ray {k}: missed body {inner[0]}'
            continue
        assert outer is not None and t >= outer[1] - 20 * tol, f'ray {k}: body {b} at {t}, the nearest is {outer}'
        assert inner is None or t <= inner[1] + 20 * tol, f'ray {k}: body {b} at {t}, past body {inner[0]} at {inner[1]}'
        own = queries.ray_trace(large[b], None, o[k], dk, 3e38)
        assert own is not None and t >= own[0] - 20 * tol
        agree += 1
    assert agree >= 8
    w.destroy()
