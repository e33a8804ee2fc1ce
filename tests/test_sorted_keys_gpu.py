"""The body order of the octree build (csrc/keysort.cu and the one-sweep sort)
against numpy: keys made with the same FP64 operations from the root cube, and
a stable sort of them, at the edges of each form's range of sizes."""
from __future__ import annotations

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def morton(pos, centre, half):
    lo = np.array(centre, np.float64) - float(half)
    c = np.clip((pos.astype(np.float64) - lo[:, None]) * (512.0 / float(half)), 0, 1023)
    c = c.astype(np.int64)
    keys = np.zeros(pos.shape[1], np.int64)
    for b in range(10):
        for k in range(3):
            keys |= ((c[k] >> b) & 1) << (3 * b + k)
    return keys


@pytest.mark.parametrize("n", [1, 2, 31, 1023, 1024, 1025, 2049, 16384, 16385, 32769, 65535, 65536, 65537,
                               131071, 131072, 131073])
def test_body_order(nb, cuda, n):
    rng = np.random.default_rng(n)
    pos = rng.uniform(-1.0, 1.0, (3, n)).astype(np.float32)
    pos[:, rng.random(n) < 0.4] *= np.float32(1e-3)  # long runs of equal keys
    p = nb.allocate_particles_gpu(n)
    for k, a in zip("xyz", pos):
        p.arrays[k].copy_(cuda.from_numpy(a))
    p.arrays["mass"].fill_(1.0)
    t = nb.Octree(n)
    t.reset()
    t.bbox(p)
    t.build(p)
    t.sort()
    st = t.stats()
    keys = morton(pos, st.root_center, st.root_half) if n > 1 else np.zeros(1)
    assert (t.sort_idx() == np.argsort(keys, kind="stable")).all()
