"""Sim.fof answers for the state the engine holds, whichever call put it there:
a host round trip of no steps leaves positions that no tree has been built of.
Labels and sizes against the oracle's loop over all pairs; the steps that
follow are those of an engine that was not asked."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KEYS = ("x", "y", "z", "vx", "vy", "vz", "ax", "ay", "az")


def cloud(n, seed):
    rng = np.random.default_rng(seed)
    st = {k: rng.uniform(-1.0, 1.0, n).astype(np.float32) for k in KEYS}
    for k in KEYS[3:]:
        st[k] *= np.float32(0.01)
    return st


def check(port, sim, st, links):
    for ll in links:
        lab, agg, g = sim.fof(ll)
        l_ref, s_ref, g_ref = port.fof(st["x"], st["y"], st["z"], ll)
        assert g == g_ref
        np.testing.assert_array_equal(lab, l_ref)
        np.testing.assert_array_equal(agg, s_ref)


@pytest.mark.parametrize("n", [1, 2, 900, 3000])
@pytest.mark.parametrize("r_coll", [0.0, 1e-5])
def test_fof_of_a_state_no_step_has_sorted(nb, cuda, port, n, r_coll):
    links = [0.0006, 0.05]  # by cells, through the tree
    mass = np.full(n, 1e-9, np.float32)
    prm = nb.sim_params(dt=1e-3, softening=1e-2, star_mass=1.0, r_coll=r_coll)
    asked, other = nb.Sim(prm, n), nb.Sim(prm, n)
    first, second = cloud(n, 5), cloud(n, 6)
    for sim in (asked, other):
        st = {k: v.copy() for k, v in first.items()}
        sim.step_host(st, mass, 0)
        assert all((st[k] == first[k]).all() for k in KEYS)
        if sim is asked:  # no tree yet
            check(port, sim, first, links)
        sim.step(2)
        if sim is asked:
            check(port, sim, sim.get_state(), links)
        st = {k: v.copy() for k, v in second.items()}
        sim.step_host(st, mass, 0)
        if sim is asked:  # the tree is that of another state
            check(port, sim, second, links)
            check(port, sim, second, links)
        sim.step(1)
    a, b = asked.get_state(), other.get_state()
    assert all((a[k] == b[k]).all() for k in KEYS)
    check(port, asked, a, links)
    st = {k: v.copy() for k, v in first.items()}
    asked.step_host(st, mass, 1)  # a replayed step
    check(port, asked, st, links)
    for sim in (asked, other):
        sim.close()


def test_read_out_then_fof(nb, cuda):
    """Large read-outs lend the engine's tree buffers: a search after one is
    that of the positions read out."""
    n = (1 << 18) + 37
    st = cloud(n, 8)
    sim = nb.Sim(nb.sim_params(dt=1e-3, softening=1e-2, star_mass=1.0), n)
    sim.set_state(*[st[k] for k in KEYS[:6]], np.full(n, 1e-9, np.float32))
    sim.step(1)
    out = sim.get_state()
    pos = [cuda.from_numpy(out[k]).cuda() for k in "xyz"]
    tree = nb.Octree(n)
    for ll in (0.0006, 0.004):
        lab, agg, g = sim.fof(ll)
        l_ref, s_ref, g_ref = tree.fof(*pos, ll)
        assert g == g_ref and g > 0
        np.testing.assert_array_equal(lab, l_ref.cpu().numpy())
        np.testing.assert_array_equal(agg, s_ref.cpu().numpy().view(np.uint16))
    sim.close()
