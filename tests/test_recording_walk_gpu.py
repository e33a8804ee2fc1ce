"""The recording walk's two warps (csrc/walk.cu, record_batches) at the edges
of their batches: the trajectory a replay of the tape gives is the recorded
one bit for bit, and one that adds in FP64 stays within the FP32 sums' rounding."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("theta", [0.0, 0.5])
@pytest.mark.parametrize("n", [2, 31, 32, 33, 63, 64, 65, 129, 1000, 5003])
def test_tape_gives_the_walk(nb, cuda, n, theta):
    """theta 0: every list holds all n bodies -- n below, at and above whole
    batches of 32, and (1000, 5003) lists of many.  The replay adds the tape's
    entries in their order, so equal bits mean that batches, chunks and counts
    are the lists that were summed."""
    prm = nb.sim_params(dt=0.005, theta=theta, softening=1e-3, star_mass=1.0, r_coll=0.0,
                        restitution=0.0, gas_drag_rate=0.0, perturber_enabled=0,
                        state_precision=nb.NBODY_STATE_F64)
    d = nb.make_disk(n, 0.5, 5.0, 0.01, 0.005, 1.0, 11)
    x0 = cuda.tensor(np.stack([d[k] for k in "xyz"]), dtype=cuda.float64, device="cuda")
    v0 = cuda.tensor(np.stack([d["v" + k] for k in "xyz"]), dtype=cuda.float64, device="cuda")
    mass = cuda.full((n,), 1e-6, dtype=cuda.float32, device="cuda")
    eng = nb.Adjoint(prm, n, 3)
    x, v = eng.forward(x0, v0, mass, 0.0, 5.2)
    xr, vr = eng.replay(x0, v0, 0.0, 5.2)
    assert cuda.equal(x, xr) and cuda.equal(v, vr)
    # FP64 interactions from the same lists: FP32 sums of n terms apart, over
    # three steps of dt (kicks of dt a): n + 32 units of 2^-24 of the largest
    # sum of magnitudes
    xd, vd = eng.replay(x0, v0, 0.0, 5.2, fp64=True)
    p = x0.cpu().numpy()
    r = p[:, :, None] - p[:, None, :]
    mag = (1e-6 * np.abs(r) / ((r * r).sum(0) + 1e-6) ** 1.5).sum(2).max()
    lim = 4 * 3 * 0.005 * (n + 32) * 2.0**-24 * mag
    assert float((v - vd).abs().max()) <= lim
    eng.close()


@pytest.mark.parametrize("state", ["F64", "F32X2"])
@pytest.mark.parametrize("n", [2, 31, 33, 64, 65, 129, 2000, 92160, 92161])
def test_fine_states_keep_the_order_of_the_sums(nb, cuda, n, state):
    """States finer than FP32: the walk with votes, by two warps a group up to
    92,160 bodies, sums in the order of the walk by one.  With theta 0 no node
    is accepted, so it lists what the walk without votes (always one warp)
    lists, and the accelerations are equal bit for bit."""
    d = nb.make_disk(n, 0.5, 5.0, 0.01, 0.005, 1.0, 3)
    out = []
    for mode in (1, 2):
        prm = nb.sim_params(dt=0.01, softening=1e-3, star_mass=0.0, r_coll=0.0, walk_mode=mode,
                            theta=0.0, state_precision=getattr(nb, "NBODY_STATE_" + state))
        sim = nb.Sim(prm, n)
        sim.set_state(*[d[k] for k in ("x", "y", "z", "vx", "vy", "vz")],
                      np.full(n, 1e-6, np.float32))
        sim.sync()
        g = sim.get_state()
        out.append(np.stack([np.asarray(g[k]) for k in ("ax", "ay", "az")]))
        assert sim.stats().status == 0
        sim.close()
    assert np.array_equal(out[0], out[1])
