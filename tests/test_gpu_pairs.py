"""The step's pair walk and the tables it shares between steps: pair sets against the no-allocation
broadphase (one thread a body) and the oracle's grid, over several steps."""

import numpy as np
import pytest

import avbd_b200
from avbd_b200.scenes import Scene, drop_pile
from oracle import Oracle

pytestmark = pytest.mark.gpu


def _pairs(a):
    return {(int(x), int(y)) for x, y in a}


@pytest.mark.parametrize('n', [1, 7, 15, 257, 4000])
def test_pairs_follow_the_bodies_over_steps(cuda_lib, n):
    """Boxes and spheres with large bodies among them, fixed and moving, some disabled: each step's pairs
    are those of the poses it starts from."""
    scene = drop_pile(n, seed=n, spacing=1.25, layers=3)
    rng = np.random.default_rng(n)
    if n >= 257:
        for k in range(4):  # large: two fixed slabs, two moving ones
            scene.box([9.0, 9.0, 0.5], 1.0 if k % 2 else 0, 0.5, [*rng.uniform(-6, 6, 2), 2.5 * k])
    w = avbd_b200.CudaSolver3D(scene)
    off = rng.choice(np.arange(1, n + 1), n // 20, replace=False) if n >= 257 else []
    for i in off:
        w.set_lifecycle(int(i), 2)
    for step in range(6):
        before = w.read_bodies()
        want = _pairs(avbd_b200.find_pairs_noalloc(before))
        w.step()
        got = w.read_pairs()
        assert len(got) == len(_pairs(got)), 'a pair twice'
        assert _pairs(got) == want, f'step {step}'
        w.step(3)
    assert w.read_counters()['error'] == 0
    w.destroy()


@pytest.mark.parametrize('n', [32766, 32767, 32768])
def test_pairs_on_both_sides_of_the_walks_widths(cuda_lib, n):
    """With the ground 32767, 32768 and 32769 bodies: sixteen lanes a body up to 32768, four past it."""
    scene = drop_pile(n, seed=3, spacing=1.3, layers=10)
    w = avbd_b200.CudaSolver3D(scene)
    o = Oracle(scene, fp32=True)
    want = _pairs(o.pairs())
    w.step()
    assert _pairs(w.read_pairs()) == want and len(want) > n // 2
    w.destroy()


def test_a_world_without_bodies_steps(cuda_lib):
    w = avbd_b200.CudaSolver3D(Scene('empty'), body_capacity=8)
    w.step(3)
    c = w.read_counters()
    assert c['steps'] == 3 and c['pairs'] == 0 and c['error'] == 0
    w.destroy()


@pytest.mark.parametrize('bodies', [3, 48, 700])
def test_capacity_above_the_population_changes_nothing(cuda_lib, bodies):
    """Tables made for many more bodies than there are are emptied by other launches than those of a world
    that is full (the warm-start table past 256 words a thread by a memset): the same steps bit for bit, also
    with kept manifolds between, and after bodies came that put the world on the other side of the rule."""
    scene = drop_pile(bodies, seed=3, spacing=1.3, layers=3)
    records, _, _, _ = avbd_b200.scene_records(scene)
    more = records[1:].copy()
    more['pos'][:, 2] += 8.0
    for f in ('initial_pos', 'inertial_pos'):
        more[f] = more['pos']
    out = []
    for capacity in (2 * bodies + 1, 20000, 300000):
        w = avbd_b200.CudaSolver3D(body_capacity=capacity)
        w.params = scene.params
        w.add_bodies(records)
        state = []
        for k in range(12):
            w.step(2)
            w.step(1, reuse_manifolds=True)
            if k == 5:
                w.add_bodies(more)
            c = w.read_counters()
            assert c['error'] == 0 and c['overflow'] == 0
            state.append((c['pairs'], c['contacts'], w.read_bodies().tobytes()))
        out.append(state)
        w.destroy()
    assert out[0][-1][1] > 0
    for state in out[1:]:
        for k, (a, b) in enumerate(zip(out[0], state)):
            assert a == b, f'round {k}'


@pytest.mark.parametrize('n, slabs', [(300, 0), (300, 1), (300, 2), (300, 16), (300, 17), (3000, 60), (33000, 6), (33000, 60)])
def test_many_large_bodies(cuda_lib, n, slabs):
    """Large bodies up to the most there may be (64), fixed and moving, through a pile: the walk's places for
    the first ones and its lanes' strides over the rest, sixteen lanes a body and four, find the restated
    grid's pairs."""
    scene = drop_pile(n, seed=n, spacing=1.25, layers=6)
    rng = np.random.default_rng(n)
    side = max(abs(x) for b in scene.bodies[1:] for x in b.pos[:2])
    for k in range(slabs):
        scene.box([9.0, 9.0, 0.5], 1.0 if k % 3 else 0, 0.5, [*rng.uniform(-side, side, 2), float(rng.uniform(0, 8))])
    w = avbd_b200.CudaSolver3D(scene)
    before = w.read_bodies()
    want = _pairs(avbd_b200.find_pairs_noalloc(before)) if n <= 4000 else _pairs(Oracle(scene, fp32=True).pairs())
    w.step()
    got = w.read_pairs()
    assert len(got) == len(_pairs(got)) and _pairs(got) == want
    first = n + 1
    assert sum(max(p) >= first for p in want) >= 5 * slabs
    assert w.read_counters()['error'] == 0
    w.destroy()
