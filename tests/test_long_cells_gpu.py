"""The neighbour search by cells (csrc/neighbors.cu k_cell_neighbors) where
cells hold many bodies: runs of equal keys around the length that a thread
looks through for itself, and a disk that a far body has squeezed into one
cell.  FoF labels bit for bit against the oracle's loop over all pairs,
impulses against numpy, and the time against the search through the tree."""
from __future__ import annotations

import numpy as np
import pytest

from test_cell_search_gpu import impulses

pytestmark = pytest.mark.gpu

SIDE = 2.0 * 1.001 * 1.001 / 1024.0  # of a finest cell of a cube of side 2


def runs(lengths, seed):
    """Bodies in the cube of side 2 about the origin, `lengths` of them in
    cells beside each other along x, most of them near the wall to the next,
    in random order."""
    rng = np.random.default_rng(seed)
    pos = [np.array([[-1.0, 1.0]] * 3)]
    lo = -1.001 * 1.001
    for k, m in enumerate(lengths):
        f = rng.uniform(0.0, 1.0, (3, m))
        near = rng.random(m) < 0.7
        f[0, near] = np.where(rng.random(near.sum()) < 0.5, 0.02, 0.98) + \
            rng.uniform(-0.015, 0.015, near.sum())
        pos.append(lo + SIDE * (np.array([[600 + k], [700], [512]]) + f))
    pos = np.concatenate(pos, 1).astype(np.float32)
    return pos[:, rng.permutation(pos.shape[1])]


LENGTHS = [(1, 2, 31, 32, 33, 34), (63, 64, 65, 66, 3), (128, 129, 130, 131), (200, 1, 97, 32),
           (700, 700)]


@pytest.mark.parametrize("lengths", LENGTHS)
@pytest.mark.parametrize("rel", [0.01, 0.05, 0.45])
def test_fof_of_long_runs(nb, cuda, port, lengths, rel):
    pos = runs(lengths, 5)
    ll = float(np.float32(rel * SIDE))
    l_ref, s_ref, g_ref = port.fof(*pos, ll)
    for fof in (nb.Octree(pos.shape[1]).fof, nb.fof_noalloc):
        lab, agg, g = fof(*[cuda.from_numpy(a).cuda() for a in pos], ll)
        assert g == g_ref
        np.testing.assert_array_equal(lab.cpu().numpy(), l_ref)
        np.testing.assert_array_equal(agg.cpu().numpy().view(np.uint16), s_ref)


def collide(nb, cuda, pos, vel, r, e):
    n = pos.shape[1]
    p = nb.allocate_particles_gpu(n)
    for k, a in zip(("x", "y", "z", "vx", "vy", "vz"), (*pos, *vel)):
        p.arrays[k].copy_(cuda.from_numpy(np.ascontiguousarray(a)))
    p.arrays["mass"].fill_(1e-9)
    t = nb.Octree(n)
    for f in (t.reset, lambda: t.bbox(p), lambda: t.build(p), t.summarize):
        f()
    t.collide(p, r, e)
    return t, p


@pytest.mark.parametrize("lengths", LENGTHS)
@pytest.mark.parametrize("rel", [0.05, 0.45])
def test_impulses_of_long_runs(nb, cuda, lengths, rel):
    pos = runs(lengths, 6)
    n, r = pos.shape[1], float(np.float32(rel * SIDE))
    vel = np.random.default_rng(2).standard_normal((3, n)).astype(np.float32)
    _, p = collide(nb, cuda, pos, vel, r, 0.2)
    got = np.stack([p.arrays[k].cpu().numpy() for k in ("vx", "vy", "vz")]).astype(np.float64)
    dv = impulses(pos, vel, r, 0.2)
    # terms of at most a few units, each rounded a dozen times in FP32 and added
    # one by one to a sum of up to as many units
    partners = np.array([((pos - pos[:, i:i + 1]) ** 2).sum(0) for i in range(n)])
    partners = (partners < 1.1 * r * r).sum(1)
    lim = 2.0**-23 * (16.0 * 8.0) * (partners + 1)
    assert (np.abs(got - (vel + dv)) <= lim).all()


def test_each_disk_s_own_runs(nb, cuda):
    """An ensemble of two disks of one long run each, whose keys differ in the
    disk alone: each as it moves by itself."""
    n, r = 300, 0.2 * SIDE
    states = []
    for k in range(2):
        pos = runs((n - 2,), 11 + k).astype(np.float64)
        states.append((pos, 0.1 * np.random.default_rng(20 + k).standard_normal((3, n))))
    prm = nb.sim_params(dt=1e-7, softening=1e-2, star_mass=0.0, r_coll=r,
                        state_precision=nb.STATE_F64)
    mass = np.full(n, 1e-12, np.float32)
    both = nb.Ensemble(prm, [{"n": n}, {"n": n}])
    x, v = (np.concatenate([s[k] for s in states], 1) for k in (0, 1))
    both.set_state(*x, *v, np.tile(mass, 2))
    both.step(1)
    g = both.get_state(double=True)
    for k, (x, v) in enumerate(states):
        one = nb.Sim(prm, n)
        one.set_state(*x, *v, mass)
        one.step(1)
        h = one.get_state(double=True)
        one.close()
        assert np.abs(h["vx"] - v[0]).max() > 1e-2
        for q in ("vx", "vy", "vz"):  # the same pairs, impulses and order of sums
            assert (g[q][k * n:(k + 1) * n] == h[q]).all()


def test_a_far_body_costs_no_more_than_the_tree_search(nb, cuda):
    n = 30011
    d = nb.make_disk(n, 0.5, 5.0, 0.01, 0.005, 1.0, 3)
    pos = np.stack([d[k] for k in "xyz"]).astype(np.float32)
    pos[:, 0] = 20000.0, 100.0, 3000.0  # one cell holds the others
    tree, p = collide(nb, cuda, pos, np.zeros((3, n), np.float32), 3.9e-5, 0.0)

    def best(call):
        e0, e1 = (cuda.cuda.Event(enable_timing=True) for _ in range(2))
        times = []
        for _ in range(6):
            cuda.cuda.synchronize()
            e0.record()
            call()
            e1.record()
            cuda.cuda.synchronize()
            times.append(e0.elapsed_time(e1))
        return min(times)

    cells = best(lambda: tree.collide(p, 3.9e-5, 0.0))
    through_tree = best(lambda: tree.collision_report(3.9e-5))
    assert cells <= 1.5 * through_tree, (cells, through_tree)
