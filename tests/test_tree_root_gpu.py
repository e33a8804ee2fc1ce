"""nbody_tree_stats_get's root mass and centre after each call that builds a
tree: those of that tree (a friends-of-friends search weighs every body 1)."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def cloud(n, seed):
    return np.random.default_rng(seed).uniform(0.5, 1.5, (3, n)).astype(np.float32)


def check(st, pos, mass):
    total = float(mass) * pos.shape[1]
    assert abs(st.root_mass - total) <= 1e-12 * total
    com = pos.astype(np.float64).mean(1)
    assert np.abs(np.array(st.root_com) - com).max() <= 1e-12 * 1.5


@pytest.mark.parametrize("n", [2, 33, 1000, 2048, 5000])
def test_root_of_the_last_tree(nb, cuda, n):
    pos, other = cloud(n, 1), cloud(n, 2)
    fof = lambda t, p: t.fof(*[cuda.from_numpy(a).cuda() for a in p], 0.01)
    t = nb.Octree(n)
    fof(t, pos)
    check(t.stats(), pos, 1.0)
    check(t.stats(), pos, 1.0)
    parts = nb.allocate_particles_gpu(n)
    for k, a in zip("xyz", other):
        parts.arrays[k].copy_(cuda.from_numpy(a))
    parts.arrays["mass"].fill_(0.25)
    t.reset()
    t.bbox(parts)
    t.build(parts)
    t.summarize()
    check(t.stats(), other, 0.25)
    fof(t, pos)
    check(t.stats(), pos, 1.0)


@pytest.mark.parametrize("n", [1, 700])
def test_root_of_a_search_smaller_than_the_handle(nb, cuda, n):
    t = nb.Octree(3000)
    pos = cloud(n, 3)
    t.fof(*[cuda.from_numpy(a).cuda() for a in pos], 0.01)
    check(t.stats(), pos, 1.0)


def test_no_tree_yet(nb, cuda):
    st = nb.Octree(100).stats()
    assert st.root_mass == 0.0 and list(st.root_com) == [0.0, 0.0, 0.0]
