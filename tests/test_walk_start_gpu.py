"""Where the walk of one warp a group (csrc/walk.cu k_walk) starts, how it
expands leaves, and the edge between four warps a group and two: the root accepted as a whole by every group, the root opened,
and cells of many bodies on one key."""
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


@pytest.mark.parametrize("n", [300, 1000, 5000])
def test_root_taken_whole(nb, cuda, n):
    """theta 1e4 and a centre of mass in no group's box (more bodies than one
    span of groups, the lone one a group of its own): every target gets the
    root's monopole, one node a group.  Each component is three products and
    sums of FP32 terms and the third power of a 2^-22 reciprocal root: within
    32 units of 2^-24 of the force, with the centre rounded to FP32."""
    st = disk(nb, n, 4.0, 5.0, seed=5, m=1e-6)
    x = np.stack([st[k] for k in "xyz"], 1).astype(np.float64)
    x[:, 0] += 40.0  # one side of a far lone body: the centre is between them
    x[0] = [-40.0 * (n - 1), 0.0, 0.0]
    st = dict(st, x=x[:, 0].astype(np.float32), y=x[:, 1].astype(np.float32),
              z=x[:, 2].astype(np.float32))
    x = np.stack([st[k] for k in "xyz"], 1).astype(np.float64)
    a, s = accel(nb, st, n, theta=1e4, walk_mode=2)
    assert s.status == 0 and s.interactions == n and s.walk_nodes_visited == s.walk_groups
    d = x.mean(0) - x
    r2 = (d * d).sum(1) + 1e-6
    ref = n * 1e-6 * d / r2[:, None] ** 1.5
    lim = 32 * 2.0**-24 * np.linalg.norm(ref, axis=1)
    # the centre itself, rounded to FP32, moves by half a unit in its last place
    lim += 3 * 2.0**-24 * np.abs(x.mean(0)).max() / np.sqrt(r2) * np.linalg.norm(ref, axis=1)
    assert (np.linalg.norm(a - ref, axis=1) <= lim).all()


@pytest.mark.parametrize("copies", [1, 8, 31, 33, 64, 300])
def test_cells_of_many_bodies(nb, cuda, copies):
    """theta 0 with clumps far below a cell's size: leaves of `copies` bodies,
    all pairs summed in FP32, within n + 16 units in the last place of the sum
    of the terms' magnitudes of the FP64 sum."""
    rng = np.random.default_rng(17)
    m = 40
    c = rng.uniform(-4.0, 4.0, (m, 3))
    x = (c[:, None, :] + rng.uniform(-1e-4, 1e-4, (m, copies, 3))).reshape(-1, 3).astype(np.float32)
    n = len(x)
    st = {k: x[:, i].copy() for i, k in enumerate("xyz")}
    st.update({k: np.zeros(n, np.float32) for k in ("vx", "vy", "vz")},
              m=np.full(n, 1e-6, np.float32))
    a, s = accel(nb, st, n, theta=0.0, walk_mode=2)
    assert s.status == 0 and s.interactions == n * n
    x = x.astype(np.float64)
    for i in range(0, n, max(1, n // 200)):
        d = x - x[i]
        r2 = (d * d).sum(1) + np.float64(np.float32(1e-3)) ** 2
        t = np.float64(np.float32(1e-6)) * d / r2[:, None] ** 1.5
        # a term's own error: FP32 coordinates are exact, their differences and
        # the rest of the term round a dozen times, the root to 2^-22 (cubed)
        assert (np.abs(a[i] - t.sum(0)) <= (n + 32) * 2.0**-24 * np.abs(t).sum(0)).all()


@pytest.mark.parametrize("n", [25600, 25601])
def test_edge_of_four_warps(nb, cuda, port, n):
    """theta 0.5 on both sides of the rule: no further from FP64 direct sums
    than twice the walk that takes no votes and so opens more."""
    st = disk(nb, n, 0.5, 5.0, seed=9, m=1e-8)
    tg = np.arange(0, n, n // 512)
    ref = np.stack(port.direct_f64(*[st[k] for k in "xyz"], st["m"], tg, 1e-3, 0.0, False), 1)

    def err(a):
        return np.median(np.linalg.norm(a[tg] - ref, axis=1) / np.linalg.norm(ref, axis=1))

    a, s = accel(nb, st, n, theta=0.5)
    b, _ = accel(nb, st, n, theta=0.5, walk_mode=2)
    assert s.status == 0 and err(a) <= 2.0 * err(b) + 1e-6
