"""Touching bodies of one colour: colours given by the caller, and more bodies touching one another than
there are colours. The colour-by-colour sweep solves them side by side; the dataflow sweep must neither
wait for a result that comes after their own nor leave its tags in the contact records."""

import numpy as np
import pytest

import avbd_b200
from avbd_b200.scenes import Scene, drop_pile

pytestmark = pytest.mark.gpu


def _stack(boxes, pitch):
    """Unit cubes straight above one another on a static ground box: C0's tangential parts are zero, whose
    bits are those of a tag that nothing has been written under."""
    s = Scene(f'{boxes} cubes')
    s.box([50, 50, 1], 0, 0.5, [0, 0, -0.5])
    for k in range(boxes):
        s.box([1, 1, 1], 1, 0.5, [0, 0, 0.495 + k * pitch])
    s.params.gravity = -9.81
    return s


def _contacts(w):
    m, c = w.read_contacts()
    return {(int(r['a']), int(r['b'])): c[r['first']:r['first'] + r['count']].copy() for r in m}


def _c0_kept(make, colors, warm, iterations):
    """Steps the scene once without iterations, which leaves the records as the narrowphase wrote them, and
    once with; the C0 of every point alike, and the step without an error. The records and counters."""
    out = []
    for it in (0, iterations):
        scene = make()
        w = avbd_b200.CudaSolver3D(scene)
        w.step(warm)
        if colors is not None:
            w.set_fixed_colors(colors(w.body_count))
        p = w.params
        p.iterations = it
        w.params = p
        w.step(1)
        w.synchronize()
        c = w.read_counters()
        assert c['error'] == 0 and c['overflow'] == 0
        out.append((_contacts(w), c))
        assert np.isfinite(w.read_bodies()['pos']).all()
        w.destroy()
    (before, _), (after, counters) = out
    assert before.keys() == after.keys() and len(after) > 0
    for k, c in before.items():
        for field in ('c0_n', 'c0_t1', 'c0_t2'):
            assert np.array_equal(c[field], after[k][field]), (k, field)
    return after, counters


@pytest.mark.parametrize('iterations', [1, 2, 3, 10])
@pytest.mark.parametrize('color', [0, 63, 255])
def test_touching_bodies_of_one_fixed_color(cuda_lib, iterations, color):
    """A stack whose colours are all alike (255: none given). Each pair's owner could write its last result
    before the other body has looked for the one before."""
    after, _ = _c0_kept(lambda: _stack(4, 0.99), lambda n: np.full(n, color, np.uint32), 0, iterations)
    between = [c for (a, b), c in after.items() if min(a, b) > 0]
    assert between and any((c['c0_t1'].view(np.uint32) == 0).any() for c in between)


@pytest.mark.parametrize('iterations', [1, 2, 10])
def test_pile_of_one_fixed_color(cuda_lib, iterations):
    """Settled piles in one colour: the touching bodies are in many chunks, on many SMs."""
    _c0_kept(lambda: drop_pile(300, seed=6, spacing=1.3, layers=3), lambda n: np.zeros(n, np.uint32), 20, iterations)


@pytest.mark.parametrize('iterations', [2, 10])
def test_more_overlapping_bodies_than_colors(cuda_lib, iterations):
    """A hundred bodies spawned into one another take all 64 colours, and the rest share the last."""
    after, c = _c0_kept(lambda: _stack(100, 0.004), None, 0, iterations)
    assert c['colors'] == 64 and len(after) >= 100 * 99 // 2


@pytest.mark.parametrize('iterations', [2, 10])
def test_one_color_steps_as_a_batched_world(cuda_lib, iterations):
    """At one block the sweep does what the batched kernel's colour pass does, also for bodies of one colour
    (28 lanes of rows, one warp: side by side in both), bit for bit over 30 steps."""
    scene = _stack(4, 0.99)
    scene.params.iterations = iterations
    w = avbd_b200.CudaSolver3D(scene)
    w.set_solve_blocks(1)
    w.set_fixed_colors(np.zeros(5, np.uint32))
    b = avbd_b200.BatchSolver3D(1, 5, params=scene.params)
    b.add_world_from(w)
    w.step(30)
    b.step(30)
    w.synchronize()
    b.synchronize()
    assert w.read_counters()['error'] == 0 and b.read_counters(0)['error'] == 0
    assert w.read_bodies().tobytes() == b.read_bodies(0).tobytes()
    w.destroy()
    b.destroy()
