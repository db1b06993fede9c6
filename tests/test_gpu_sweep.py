"""The dataflow sweep and its launch shapes: the launch chosen by a world's size gives, bit for bit,
what the launch of every co-resident block gives, run after run, and leaves the contact records as the
layout has them."""

import numpy as np
import pytest

import avbd_b200
from avbd_b200.scenes import demo_scene, drop_pile, hulls_and_chains

pytestmark = pytest.mark.gpu


def _stepped(scene, steps, blocks, iterations=None):
    if iterations is not None:
        scene.params.iterations = iterations
    w = avbd_b200.CudaSolver3D(scene)
    w.set_solve_blocks(blocks)
    w.step(steps)
    m, c = w.read_contacts()
    out = w.read_bodies(), w.read_joints()[0], m, c, w.read_counters()
    w.destroy()
    return out


def _by_pair(m, c):
    return {(int(r['a']), int(r['b'])): (r['normal'].tobytes(), c[r['first']:r['first'] + r['count']].tobytes()) for r in m}


SCENES = {**{f'pile {n}': (lambda n=n: drop_pile(n, seed=5, spacing=1.5, layers=4), 25) for n in (1, 15, 17, 130, 2369, 8191, 8192)},
          'rope': (lambda: demo_scene('Rope'), 40), 'soft body': (lambda: demo_scene('Soft Body'), 40), 'breakable': (lambda: demo_scene('Breakable'), 40),
          'chains': (lambda: hulls_and_chains(40, 9, 12, distinct=8), 40)}


@pytest.mark.parametrize('name', SCENES)
def test_every_launch_shape_gives_the_same_world(cuda_lib, name):
    """Sizes on both sides of the rule between the launch shapes (8192 bodies with the ground), joints and
    springs: the chosen launch, the full one and the chosen one again."""
    make, steps = SCENES[name]
    full = avbd_b200.device_info(0)[1] * 2
    runs = [_stepped(make(), steps, b) for b in (0, full, 0)]
    assert runs[0][4]['error'] == 0 and runs[0][4]['overflow'] == 0
    for r in runs[1:]:
        assert r[0].tobytes() == runs[0][0].tobytes() and r[1].tobytes() == runs[0][1].tobytes()
        assert _by_pair(r[2], r[3]) == _by_pair(runs[0][2], runs[0][3])


@pytest.mark.parametrize('iterations', [1, 2, 10])
def test_contact_records_keep_their_start_values(cuda_lib, iterations):
    """C0's tangential parts share their words with the sweep's tags: after a step the records hold what
    the narrowphase wrote, which a step without iterations leaves as it is."""
    worlds = []
    for it in (0, iterations):
        scene = drop_pile(300, seed=6, spacing=1.3, layers=3)
        scene.params.iterations = 10
        w = avbd_b200.CudaSolver3D(scene)
        w.step(20)
        p = w.params
        p.iterations = it
        w.params = p
        w.step(1)
        m, c = w.read_contacts()
        worlds.append({(int(r['a']), int(r['b'])): c[r['first']:r['first'] + r['count']] for r in m})
        w.destroy()
    assert len(worlds[0]) > 100 and worlds[0].keys() == worlds[1].keys()
    for k, c in worlds[0].items():
        for field in ('c0_n', 'c0_t1', 'c0_t2', 'r_a', 'r_b'):
            assert np.array_equal(c[field], worlds[1][k][field]), (k, field)
