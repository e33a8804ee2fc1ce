"""What a call that fails leaves in its handle, with the failure made on the
host by a stand-in for the CUDA runtime: the calls after it do what they do on
a new handle."""
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


@pytest.fixture
def nb(on_fake):
    on_fake[1].fake_reset()
    yield on_fake[0]
    on_fake[1].fake_reset()


@pytest.fixture
def fake(on_fake):
    return on_fake[1]


def particles(nb, n):
    p = nb.ParticleData(n, {k: torch.zeros(n, dtype=torch.int32 if k == "id" else torch.float32)
                            for k in nb.FIELDS + ("id",)})
    return p


def names(fake):
    return fake.fake_names().decode()


@pytest.mark.parametrize("kernel", [b"k_cells", b"k_emit"])
def test_a_failed_search_leaves_the_tree_its_masses(nb, fake, kernel):
    n = 700
    x = torch.rand(3, n)
    p = particles(nb, n)
    tree = nb.Octree(n)
    fake.fake_fail_launch(kernel, 1)
    with pytest.raises(nb.NBodyError):
        tree.fof(*x, 0.1)
    fake.fake_reset()
    tree.build(p)
    tree.summarize()
    assert "k_moment_tiles" in names(fake)
    tree.close()


@pytest.mark.parametrize("mode", ["tape", "checkpoint"])
@pytest.mark.parametrize("nth", [1, 2, 3])
def test_a_tape_pool_that_cannot_grow(nb, fake, mode, nth):
    """Its freed parts are neither used nor freed again."""
    n, steps = 64, 3
    eng = nb.Adjoint(nb.sim_params(dt=0.01, softening=1e-3, star_mass=1.0), n, steps, mode, 2)
    x, v = torch.rand(3, n, dtype=torch.float64), torch.rand(3, n, dtype=torch.float64)
    mass = torch.full((n,), 1e-8)
    eng.forward(x, v, mass, 1.0, 5.2)
    size = eng.stats().tape_bytes
    fake.fake_next_word(16)  # the next status read: the tape is full
    fake.fake_next_word(1 << 20)  # and the read after it: chunks in use
    fake.fake_fail_alloc(nth)
    with pytest.raises(nb.NBodyError, match="out of memory"):
        eng.forward(x, v, mass, 1.0, 5.2)
    fake.fake_fail_alloc(0)
    with pytest.raises(nb.NBodyError, match="no recorded forward"):
        eng.backward(x, v)
    eng.forward(x, v, mass, 1.0, 5.2)
    eng.backward(x, v)
    assert eng.stats().tape_bytes == size
    eng.close()
    assert fake.fake_bad_frees() == 0


@pytest.mark.parametrize("n", [40000, 65536])  # four keys a thread: a key kernel of its own
def test_a_failed_key_kernel_leaves_the_buffers_in_place(nb, fake, n):
    tree, p = nb.Octree(n), particles(nb, n)

    def buffers():
        tree.build(p)
        return [fake.fake_pointer(b"k_sorted_keys", k) for k in (3, 7)]

    before = buffers()
    fake.fake_fail_launch(b"k_keys", 1)
    with pytest.raises(nb.NBodyError):
        tree.build(p)
    fake.fake_reset()
    assert buffers() == before and before[0] != before[1]
    tree.close()


def test_a_search_of_the_engine_leaves_its_records(nb, fake):
    """Steps without collisions write no boxes; the search that adds them leaves
    the nodes' masses and centres as the walk read them."""
    n = 700
    sim = nb.Sim(nb.sim_params(dt=0.01, softening=1e-3, star_mass=1.0), n)
    sim.set_state(*np.random.default_rng(1).random((6, n), np.float32), np.ones(n, np.float32))
    sim.step(1)
    fake.fake_reset()
    sim.fof(0.1)
    assert "k_boxes" in names(fake) and "k_emit" not in names(fake)
    sim.close()


@pytest.mark.parametrize("kernel", [b"k_stream", b"k_permute", b"k_emit", b"k_walk"])
@pytest.mark.parametrize("engine", ["sim", "profiled", "ensemble"])
def test_a_step_whose_capture_fails(nb, fake, engine, kernel):
    """The capture is ended and the engine steps on its own stream again."""
    n = 700

    def make():
        if engine == "ensemble":
            e = nb.Ensemble(nb.sim_params(r_coll=1e-5), [{"n": 300}, {"n": 400}])
        else:
            e = nb.Sim(nb.sim_params(r_coll=1e-5), n)
            e.set_profiling(engine == "profiled")
        e.set_state(*np.random.default_rng(1).random((6, n), np.float32), np.ones(n, np.float32))
        return e

    def step(e):
        fake.fake_reset()
        before = e.stats()
        e.step(2)
        after = e.stats()
        return (names(fake), after.launches - before.launches,
                after.graph_launches - before.graph_launches)

    failed, new = make(), make()
    fake.fake_reset()
    fake.fake_fail_launch(kernel, 1)
    with pytest.raises(nb.NBodyError):
        failed.step(2)
    got = step(failed)
    assert got == step(new) and got[0].count("\n") == got[1] and got[2] == 2
    failed.close()
    new.close()
