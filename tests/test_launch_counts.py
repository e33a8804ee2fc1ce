"""The kernels that the engines say they launched, against those that a
stand-in for the CUDA runtime saw, over the sizes at which a step, a read-out
or a level changes its kernels."""
from __future__ import annotations

import numpy as np
import pytest
import torch

import fake_cuda


@pytest.fixture(scope="module")
def on_fake(tmp_path_factory):
    got = fake_cuda.load(tmp_path_factory.mktemp("fake"))
    if got is None:
        pytest.skip("the library's objects are not built")
    return got


def state(n):
    return np.random.default_rng(n).random((6, n)), np.full(n, 1e-9, np.float32)


def counted(fake, stats, call):
    before = stats().launches
    fake.fake_reset()
    call()
    return stats().launches - before, fake.fake_launches()


STEPS = {"gravity": {}, "collisions": {"r_coll": 1e-5},
         "fused": {"r_coll": 1e-5, "fuse_collisions": 1},
         "planet": {"r_coll": 1e-5, "perturber_enabled": 1, "perturber_mass_mjup": 1.0,
                    "perturber_radius_au": 5.2},
         "spans": {"span_walk": 1, "group_span": 8}}


@pytest.mark.parametrize("n", [1, 2, 900, 40000, 70000, (1 << 18) + 1])
@pytest.mark.parametrize("kind", STEPS)
@pytest.mark.parametrize("graphs", [True, False])
def test_steps(on_fake, n, kind, graphs):
    nb, fake = on_fake
    for precision in (nb.STATE_F32, nb.STATE_F64):
        sim = nb.Sim(nb.sim_params(state_precision=precision, **STEPS[kind]), n)
        x, mass = state(n)
        sim.set_state(*x.astype(np.float32), mass)
        sim.set_graphs(graphs)
        for steps in (1, 3):
            said, seen = counted(fake, sim.stats, lambda: sim.step(steps))
            assert said == seen > 0
        sim.close()


@pytest.mark.parametrize("sizes", [(2, 2), (300, 400), (1 << 17, (1 << 17) + 1)])
@pytest.mark.parametrize("r_coll", [0.0, 1e-5])
def test_ensembles(on_fake, sizes, r_coll):
    nb, fake = on_fake
    n = sum(sizes)
    ens = nb.Ensemble(nb.sim_params(r_coll=r_coll, state_precision=nb.STATE_F64),
                      [{"n": k} for k in sizes])
    x, mass = state(n)
    host = dict(zip(("x", "y", "z", "vx", "vy", "vz"), x))
    host.update({k: np.zeros(n, np.float32) for k in ("ax", "ay", "az")})
    for call in (lambda: ens.set_state(*x, mass), lambda: ens.step(1), lambda: ens.step(2),
                 lambda: ens.get_state(double=True), lambda: ens.get_state(double=False),
                 lambda: ens.step_host(host, mass, 1), lambda: ens.step_host(host, mass, 0)):
        said, seen = counted(fake, ens.stats, call)
        assert said == seen > 0
    ens.close()


@pytest.mark.parametrize("n", [64, 40000, 70000])
@pytest.mark.parametrize("mode", ["tape", "checkpoint", "direct"])
def test_gradients(on_fake, n, mode):
    nb, fake = on_fake
    eng = nb.Adjoint(nb.sim_params(gas_drag_rate=1e-3, perturber_enabled=1,
                                   perturber_mass_mjup=1.0, perturber_radius_au=5.2), n, 7, mode, 3)
    x, v = (torch.rand(3, n, dtype=torch.float64) for _ in range(2))
    mass = torch.full((n,), 1e-9)
    for _ in range(2):
        for call in (lambda: eng.forward(x, v, mass, 1.0, 5.2), lambda: eng.backward(x, v)):
            said, seen = counted(fake, eng.stats, call)
            assert said == seen > 0
    eng.close()
