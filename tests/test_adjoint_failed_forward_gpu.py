"""A forward pass that ends with an error leaves no recording behind: its
levels have replaced the last run's, so a backward or a replay would mix two
runs.  The engine serves the next forward as a fresh one does."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode", ["tape", "checkpoint"])
def test_no_recording_after_a_failed_forward(nb, cuda, mode):
    n, steps = 900, 5
    prm = nb.sim_params(dt=0.01, softening=1e-3, star_mass=1.0)
    mass = cuda.full((n,), 1e-8, device="cuda")
    st = nb.make_disk(n, 0.5, 5.0, 0.01, 0.005, 1.0, 3)
    x0, v0 = (cuda.from_numpy(np.stack([st[p + k] for k in "xyz"])).cuda() for p in ("", "v"))
    one, zero = cuda.ones_like(x0), cuda.zeros_like(v0)
    eng, fresh = (nb.Adjoint(prm, n, steps, mode, 2) for _ in range(2))
    eng.forward(x0, v0, mass, 1.0, 5.2)
    bad = x0.clone()
    bad[1, 17] = float("nan")
    with pytest.raises(nb.NBodyError):
        eng.forward(bad, v0, mass, 1.0, 5.2)
    with pytest.raises(nb.NBodyError, match="no recorded forward"):
        eng.backward(one, zero)
    if mode == "tape":
        with pytest.raises(nb.NBodyError, match="no recorded forward"):
            eng.replay(x0, v0, 1.0, 5.2)
    x, v = eng.forward(x0, v0, mass, 1.0, 5.2)
    x1, v1 = fresh.forward(x0, v0, mass, 1.0, 5.2)
    assert cuda.equal(x, x1) and cuda.equal(v, v1)
    for a, b in zip(eng.backward(one, zero)[:2], fresh.backward(one, zero)[:2]):
        assert (a - b).abs().max() <= 1e-11 * b.abs().max()  # up to the order of the FP64 adds
    eng.close()
    fresh.close()
