"""The GPU adjoint (avbd_adjoint_*, double precision) against the oracle's FP64 tape adjoint on the
same recorded structures, world by world; the tape adjoint is itself checked against central
differences (tests/test_adjoint_cpu.py)."""

import numpy as np
import pytest

import avbd_b200
from avbd_b200.scenes import tumbling_world
from oracle import Oracle

pytestmark = pytest.mark.gpu


def _recordings(worlds=4, bodies=16, steps=40, seed=0):
    recs, cpu = [], []
    for w in range(worlds):
        s = tumbling_world(np.random.default_rng(seed + w), bodies)
        A = Oracle(s).adjoint(steps)
        recs.append(A.export())
        cpu.append(A)
    return recs, cpu


def test_gpu_adjoint_matches_the_tape_adjoint(cuda_lib):
    recs, cpu = _recordings()
    adj = avbd_b200.Adjoint(recs, checkpoint=10)
    params, targets = [], []
    rng = np.random.default_rng(7)
    for A in cpu:
        p0 = A.nominal()
        pt = p0.copy()
        pt[0::8] += rng.normal(0, 0.2, A.n)
        pt[5::8] += rng.normal(0, 0.5, A.n)
        _, t = A.loss(pt, final=True)
        A.set_target(t)
        params.append(p0)
        targets.append(t.reshape(-1))
    P = np.concatenate(params)
    adj.set_target(np.concatenate(targets))
    loss_f, fin = adj.forward(P)
    loss, g = adj.backward(P)
    assert np.allclose(loss, loss_f, rtol=1e-12)
    o = 0
    worst_g = worst_l = 0.0
    for w, A in enumerate(cpu):
        L, gc = A.gradient(params[w])
        worst_l = max(worst_l, abs(L - loss[w]) / abs(L))
        gw = g[8 * o:8 * (o + A.n)].reshape(-1, 8)
        dyn = recs[w]['bodies'].reshape(-1, 13)[:, 11] != 0  # static bodies have no parameters
        gc = gc.reshape(-1, 8)[dyn]
        gw = gw[dyn]
        worst_g = max(worst_g, np.abs(gw - gc).max() / np.abs(gc).max())
        o += A.n
    print(f'GPU adjoint vs FP64 tape adjoint: loss rel {worst_l:.2e}, gradient rel (to max) {worst_g:.2e}')
    # Both sides are FP64 but sum in different orders (a tape against hand-written cotangents with
    # atomics); contact penalties reach 1e10 against inertia m/dt^2 ~ 1e3, so the 6x6 solves have
    # condition numbers near 1e7 and floored pivots: agreement to 1e-5 of the largest entry.
    assert worst_l < 1e-9 and worst_g < 1e-5
    adj.destroy()


@pytest.mark.parametrize('bodies', [1, 15, 33, 70, 120])
def test_every_block_size_gives_the_same_gradients(cuda_lib, bodies):
    """One world, 200 and 300 of it (256, 128 and 64 threads a world; more bodies of one colour than are
    solved together): the same sums in other orders, so the same gradients to the solves' conditioning
    (1e7 times a double's rounding, of the largest entry), and the same in every copy."""
    A = Oracle(tumbling_world(np.random.default_rng(bodies), bodies)).adjoint(4)
    rec, p0 = A.export(), A.nominal()
    target = np.tile([0.3, -0.2, 0.1, 0.0, 0.0, 0.0, 1.0], A.n)
    grads = []
    for worlds in (1, 200, 300):
        adj = avbd_b200.Adjoint([rec] * worlds, checkpoint=3)
        adj.set_target(np.tile(target, worlds))
        loss, fin = adj.forward(np.tile(p0, worlds))
        loss_b, g = adj.backward(np.tile(p0, worlds))
        adj.destroy()
        g = g.reshape(worlds, -1)
        assert np.allclose(loss, loss[0], rtol=1e-12) and np.allclose(loss_b, loss, rtol=1e-12)
        assert np.abs(g - g[0]).max() <= 1e-7 * np.abs(g[0]).max()
        grads.append(g[0])
    for g in grads[1:]:
        assert np.abs(g - grads[0]).max() <= 1e-7 * np.abs(grads[0]).max()


@pytest.mark.parametrize('bodies, steps_clashing', [(4, 30), (16, 30), (16, 7), (40, 30), (70, 30)])
def test_touching_bodies_of_one_color(cuda_lib, bodies, steps_clashing):
    """A recording whose last `steps_clashing` steps have every body in one colour, touching ones among them:
    the tape solves such bodies one after another, by index, and so does the replay. Its gradients are the
    tape's, beside a properly coloured world's in the same batch (to the tolerances of
    test_gpu_adjoint_matches_the_tape_adjoint)."""
    from oracle import Adjoint
    steps = 30
    A = Oracle(tumbling_world(np.random.default_rng(bodies), bodies)).adjoint(steps)
    proper, p0 = A.export(), A.nominal()
    dyn = proper['bodies'].reshape(-1, 13)[:, 11] != 0
    man = proper['man_bodies'].reshape(-1, 2)[proper['step_man'][steps - steps_clashing]:]
    assert (dyn[man[:, 0]] & dyn[man[:, 1]]).any()
    clash = dict(proper)
    colors, ncol = proper['colors'].reshape(steps, -1).copy(), proper['ncol'].copy()
    colors[steps - steps_clashing:] = np.where(dyn, 0, -1)
    ncol[steps - steps_clashing:] = 1
    clash['colors'], clash['ncol'] = colors.reshape(-1), ncol
    pt = p0.copy()
    pt[0::8] += np.random.default_rng(7).normal(0, 0.2, A.n)
    recs = [clash, proper]
    tapes = [Adjoint.from_record(r, p0) for r in recs]
    targets = [t.loss(pt, final=True)[1] for t in tapes]
    adj = avbd_b200.Adjoint(recs, checkpoint=4)
    adj.set_target(np.concatenate([t.reshape(-1) for t in targets]))
    P = np.tile(p0, 2)
    loss_f, _ = adj.forward(P)
    loss, g = adj.backward(P)
    adj.destroy()
    assert np.allclose(loss, loss_f, rtol=1e-12)
    for w, (tape, target) in enumerate(zip(tapes, targets)):
        tape.set_target(target)
        L, gc = tape.gradient(p0)
        gw, gc = g.reshape(2, -1, 8)[w][dyn], gc.reshape(-1, 8)[dyn]
        assert abs(L - loss[w]) < 1e-9 * abs(L), w
        assert np.abs(gw - gc).max() < 1e-5 * np.abs(gc).max(), w


@pytest.mark.parametrize('worlds', [1, 200, 300])
def test_adjoints_side_by_side(cuda_lib, worlds):
    """An adjoint of many points still runs, and gives what it gave, after one of few points was made for the
    same number of worlds, and the other way round."""
    made = []
    for bodies in (70, 2, 40):
        A = Oracle(tumbling_world(np.random.default_rng(bodies), bodies)).adjoint(30)
        adj = avbd_b200.Adjoint([A.export()] * worlds, checkpoint=4)
        adj.set_target(np.zeros(7 * A.n * worlds))
        P = np.tile(A.nominal(), worlds)
        made.append((adj, P, adj.forward(P), adj.backward(P)))
    points = [adj.info()['max_points'] for adj, _, _, _ in made]
    assert points[1] < points[2] < points[0]
    for adj, P, (loss, fin), (_, g) in made + made[::-1]:
        again, fin2 = adj.forward(P)
        loss_b, g2 = adj.backward(P)
        assert np.array_equal(again, loss) and np.array_equal(fin2, fin) and np.array_equal(loss_b, loss)
        # atomics of two runs may add in other orders: a double's rounding (1e-16) times the solves' condition
        # (1e7), a hundred of them in a row
        assert np.abs(g2 - g).max() <= 1e-7 * np.abs(g).max()
    for adj, _, _, _ in made:
        adj.destroy()
