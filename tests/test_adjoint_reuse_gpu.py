"""An adjoint engine whose tape pool an earlier run has sized, on an input that
outgrows it: the repeat starts from this input's positions.  (In checkpoint
mode the level slots rotate, so the run that ran out of tape has overwritten
level 0's.)"""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def disk(nb, n, far):
    """A disk, or one with a body so far off that one of the finest cells holds
    the rest: every group then lists every body."""
    st = nb.make_disk(n, 0.5, 5.0, 0.01, 0.005, 1.0, 3)
    x = np.stack([st[k] for k in "xyz"])
    v = np.stack([st["v" + k] for k in "xyz"])
    if far:
        x[:, 0] = (20000.0, 100.0, 3000.0)
        v[:, 0] = 0.0
    return x, v


@pytest.mark.parametrize("n", [2000, 3000])
@pytest.mark.parametrize("mode,steps", [("tape", 4), ("checkpoint", 3), ("checkpoint", 10)])
def test_a_run_that_outgrows_the_tape(nb, cuda, mode, steps, n):
    prm = nb.sim_params(dt=0.01, theta=1.0, softening=1e-3, star_mass=1.0, perturber_enabled=1,
                        perturber_mass_mjup=1.0, perturber_radius_au=5.2)
    mass = cuda.full((n,), 1e-8, device="cuda")

    def run(engine, far):
        x0, v0 = (cuda.from_numpy(a).cuda() for a in disk(nb, n, far))
        x, v = engine.forward(x0, v0, mass, 1.0, 5.2)
        return x, v, engine.backward(cuda.ones_like(x), cuda.zeros_like(v))

    used, fresh = (nb.Adjoint(prm, n, steps, mode, 4) for _ in range(2))
    run(used, False)
    small = used.stats().tape_bytes
    x, v, g = run(used, True)
    assert used.stats().tape_bytes > small, "the second input was to outgrow the pool"
    x1, v1, g1 = run(fresh, True)
    assert cuda.equal(x, x1) and cuda.equal(v, v1)
    for a, b in zip(g[:2], g1[:2]):  # up to the order of the FP64 adds
        assert (a - b).abs().max() <= 1e-11 * b.abs().max()
    used.close()
    fresh.close()
