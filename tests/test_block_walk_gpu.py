"""The walk with several warps to a group (csrc/walk.cu k_walk_block) against
the walk with one: the phase interface on the same tree, whose two-targets
form always runs one warp a group, gives another set of groups, so the
comparison is with the engine's walk mode 2 where no vote is taken (theta 0:
every node is opened and both walks sum every pair) and with the oracle's
forces where it is."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import disk

pytestmark = pytest.mark.gpu
STATE = ("x", "y", "z", "vx", "vy", "vz")


def accel(nb, st, n, **kw):
    prm = nb.sim_params(dt=0.01, softening=1e-3, star_mass=0.0, r_coll=0.0, **kw)
    sim = nb.Sim(prm, n)
    sim.set_state(*[st[k] for k in STATE], st["m"])
    sim.sync()
    g = sim.get_state()
    s = sim.stats()
    sim.close()
    return np.stack([g[k] for k in ("ax", "ay", "az")], 1).astype(np.float64), s


@pytest.mark.parametrize("n", [2, 31, 33, 129, 2000, 21504, 21505])
def test_every_pair(nb, cuda, n):
    """theta 0: all pairs, in FP32, in two orders of adding: each within n
    units in the last place of the sum of the terms' magnitudes (and a few for
    the terms themselves)."""
    st = disk(nb, n, 0.5, 5.0, seed=3, m=1e-6)
    a, sa = accel(nb, st, n, theta=0.0, walk_mode=1)
    b, sb = accel(nb, st, n, theta=0.0, walk_mode=2)
    assert sa.interactions == sb.interactions and sa.walk_nodes_visited == sb.walk_nodes_visited
    x = np.stack([st[k] for k in "xyz"], 1).astype(np.float64)
    idx = np.arange(n) if n <= 2000 else np.arange(0, n, 37)
    d = x[None, :, :] - x[idx, None, :]
    r2 = (d * d).sum(2) + 1e-6
    mag = (1e-6 * np.abs(d) / r2[:, :, None] ** 1.5).sum(1)
    lim = 2 * (n + 16) * 2.0**-24 * mag + 1e-30
    assert (np.abs(a[idx] - b[idx]) <= lim).all()


@pytest.mark.parametrize("n", [4096, 21504, 21505, 92160, 92161])
def test_votes_and_theta(nb, cuda, port, n):
    """theta 0.5: at the edges of the rule, no further from FP64 direct sums
    than the reference's own walk."""
    st = disk(nb, n, 0.5, 5.0, seed=9, m=1e-8)
    a, s = accel(nb, st, n, theta=0.5)
    assert s.status == 0
    tg = np.arange(0, n, max(1, n // 512))
    x = [st[k] for k in "xyz"]
    ref = np.stack(port.direct_f64(*x, st["m"], tg, 1e-3, 0.0, False), 1)
    err = np.linalg.norm(a[tg] - ref, axis=1) / np.linalg.norm(ref, axis=1)
    b, _ = accel(nb, st, n, theta=0.5, walk_mode=2)  # opens more than the vote walk
    err2 = np.linalg.norm(b[tg] - ref, axis=1) / np.linalg.norm(ref, axis=1)
    assert np.median(err) <= 2.0 * np.median(err2) + 1e-6
    # the same walk twice gives the same bits
    again, _ = accel(nb, st, n, theta=0.5)
    assert np.array_equal(a, again)
