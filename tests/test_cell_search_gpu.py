"""The neighbour search by cells (csrc/neighbors.cu k_cell_neighbors) at the
edges of its rule: radii just below and above half a cell (above, the tree
search answers), bodies an ulp to either side of cell walls, buckets of equal
keys, the axes' ends, several disks.  FoF labels and sizes bit for bit against
the oracle's loop over all pairs; impulses against numpy over all pairs."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bodies(kind, n, seed):
    """Positions in a cube of side 2 about `centre`, with bodies at its corners
    so that the root cube, and with it the cell side, is known in advance."""
    rng = np.random.default_rng(seed)
    centre = {"origin": 0.0, "far": 20.0}[kind.split("-")[1]]
    half = np.float32(np.float32(1.0) * np.float32(1.001) * np.float32(1.001))
    side = 2.0 * float(half) / 1024.0
    if kind.startswith("walls"):  # on the walls between cells, give or take an ulp or so
        walls = centre - float(half) + side * rng.integers(500, 520, (3, n))
        pos = walls + rng.normal(0.0, 0.3 * side, (3, n)) * (rng.random((3, n)) < 0.5)
    elif kind.startswith("crowd"):  # a few cells hold most bodies
        pos = centre + 0.3 + 0.2 * side * rng.normal(size=(3, n))
    else:
        pos = centre + rng.uniform(-0.02, 0.02, (3, n))
    pos = pos.astype(np.float32)
    pos[:, 0], pos[:, 1] = centre - 1.0, centre + 1.0
    return pos, side


KINDS = ["walls-origin", "walls-far", "crowd-origin", "cloud-far"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("rel", [1e-3, 0.1, 0.45, 0.55, 3.0])
def test_fof_at_the_rule(nb, cuda, port, kind, rel):
    n = 1500
    pos, side = bodies(kind, n, 7)
    ll = float(np.float32(rel * side))
    lab, agg, g = nb.Octree(n).fof(*[cuda.from_numpy(a).cuda() for a in pos], ll)
    l_ref, s_ref, g_ref = port.fof(*pos, ll)
    assert g == g_ref
    np.testing.assert_array_equal(lab.cpu().numpy(), l_ref)
    np.testing.assert_array_equal(agg.cpu().numpy().view(np.uint16), s_ref)
    lab, agg, g = nb.fof_noalloc(*[cuda.from_numpy(a).cuda() for a in pos], ll)
    assert g == g_ref and (lab.cpu().numpy() == l_ref).all()


@pytest.mark.parametrize("collisions", [False, True])
def test_engine_fof(nb, cuda, port, collisions):
    """The engine's FoF of its own state, with the records' boxes written by
    its steps (collisions on) or not, by cells and through the tree."""
    n = 3000
    pos, side = bodies("cloud-origin", n, 3)
    zero = np.zeros(n, np.float32)
    sim = nb.Sim(nb.sim_params(dt=1e-3, softening=1e-2, star_mass=0.0,
                               r_coll=1e-6 if collisions else 0.0), n)
    sim.set_state(*pos, zero, zero, zero, np.full(n, 1e-9, np.float32))
    sim.step(3)
    s = sim.get_state()
    for rel in (0.3, 4.0):
        ll = float(np.float32(rel * side))
        lab, agg, g = sim.fof(ll)
        l_ref, s_ref, g_ref = port.fof(s["x"], s["y"], s["z"], ll)
        assert g == g_ref
        np.testing.assert_array_equal(lab, l_ref)
        np.testing.assert_array_equal(agg, s_ref)
        sim.step(1)
        s = sim.get_state()
    sim.close()


def impulses(pos, vel, r, e):
    """dv of every body over all pairs, the pair test in FP32 as the kernels
    round it, the impulse in FP64; and the least distance of a pair's squared
    distance from the threshold, relative."""
    n, dv = pos.shape[1], np.zeros(pos.shape)
    r2 = np.float32(r) * np.float32(r)
    for i in range(n):
        d = (pos - pos[:, i:i + 1]).astype(np.float32).astype(np.float64)
        d2 = (d * d).sum(0)
        hit = (d2 < float(r2)) & (np.arange(n) != i)
        if not hit.any():
            continue
        nrm = d[:, hit] / (np.sqrt(d2[hit]) + 1e-10)
        dvn = np.minimum(((vel[:, hit] - vel[:, i:i + 1]).astype(np.float64) * nrm).sum(0), 0.0)
        dv[:, i] = 0.5 * (1.0 + e) * (dvn * nrm).sum(1)
    return dv


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("rel", [1e-2, 0.45, 0.55])
def test_impulses_at_the_rule(nb, cuda, kind, rel):
    n = 1500
    pos, side = bodies(kind, n, 11)
    r = float(np.float32(rel * side))
    rng = np.random.default_rng(2)
    vel = rng.standard_normal((3, n)).astype(np.float32)
    p = nb.allocate_particles_gpu(n)
    for k, a in zip(("x", "y", "z", "vx", "vy", "vz"), (*pos, *vel)):
        p.arrays[k].copy_(cuda.from_numpy(a))
    p.arrays["mass"].fill_(1e-9)
    t = nb.Octree(n)
    for f in (t.reset, lambda: t.bbox(p), lambda: t.build(p), t.summarize):
        f()
    t.collide(p, r, 0.2)
    got = np.stack([p.arrays[k].cpu().numpy() for k in ("vx", "vy", "vz")]).astype(np.float64)
    dv = impulses(pos, vel, r, 0.2)
    # a body's partners: terms of at most a few units, each rounded a dozen
    # times in FP32 and added one by one to a velocity of a few units
    partners = np.array([max(1, int(((pos - pos[:, i:i + 1]) ** 2).sum(0).min() >= 0) *
                             (((pos - pos[:, i:i + 1]) ** 2).sum(0) < 1.1 * r * r).sum())
                         for i in range(n)])
    lim = 2.0**-23 * (16.0 * 8.0) * (partners + 1)
    assert (np.abs(got - (vel + dv)) <= lim).all()


def test_each_disk_of_an_ensemble_by_its_own_rule(nb, cuda):
    """A disk searched by cells and one searched through the tree, in the same
    place: each as it moves alone.  Both collide: half of the wide disk's
    bodies sit half a radius from another, and a body of the small one has
    0.4 others within the radius on average."""
    n, r = 800, 2e-5
    rng = np.random.default_rng(4)
    wide = rng.uniform(-1.0, 1.0, (3, n))
    wide[:, n // 2:] = wide[:, :n // 2] + 0.5 * r * np.array([[1.0], [0.0], [0.0]])
    small = rng.uniform(-2e-4, 2e-4, (3, n))
    states = [(x, 0.1 * rng.standard_normal((3, n))) for x in (wide, small)]
    prm = nb.sim_params(dt=1e-7, softening=1e-2, star_mass=0.0, r_coll=r,
                        state_precision=nb.STATE_F64)
    mass = np.full(n, 1e-12, np.float32)
    both = nb.Ensemble(prm, [{"n": n}, {"n": n}])
    x, v = (np.concatenate([s[k] for s in states], 1) for k in (0, 1))
    both.set_state(*x, *v, np.tile(mass, 2))
    both.step(2)
    g = both.get_state(double=True)
    for k, (x, v) in enumerate(states):
        one = nb.Sim(prm, n)
        one.set_state(*x, *v, mass)
        one.step(2)
        h = one.get_state(double=True)
        one.close()
        assert np.abs(h["vx"] - v[0]).max() > 1e-3
        # impulses of ~0.1 in FP32, a few partners each, two steps
        for q in ("vx", "vy", "vz"):
            assert np.abs(g[q][k * n:(k + 1) * n] - h[q]).max() <= 1e-5
