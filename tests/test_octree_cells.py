"""The octree and target groups straight from sorted keys (csrc/tree.cu
k_cells, k_emit), restated on the CPU against plain recursive constructions.

The octree: a cell with more than `prune` bodies is split by the next three
key bits, chains of one-child cells are skipped, buckets of one key (level 10)
stay whole.  The groups: maximal nodes of <= span bodies of the binary radix
tree (index bits break ties), found by splitting key ranges bit by bit.  Keys
cover runs of equal keys (longer than a span, too), single bodies, thin
distributions and several disks in the bits above the 30 Morton bits."""
from __future__ import annotations

import numpy as np
import pytest

LEVELS = 10


def lev(a, b):
    x = int(a) ^ int(b)
    if x >> 30:
        return -1
    return LEVELS if x == 0 else (30 - x.bit_length()) // 3


# ------------------------------------------------------- plain constructions
def octree_plain(keys, prune):
    """{(first, end): (level, [(first, end) of its children])} from the roots."""
    out = {}

    def node(lo, hi):
        level = LEVELS if hi - lo == 1 else lev(keys[lo], keys[hi - 1])
        kids = []
        if hi - lo > max(prune, 1) and level < LEVELS:
            cuts = [lo] + [k for k in range(lo + 1, hi) if lev(keys[k - 1], keys[k]) == level] + [hi]
            kids = list(zip(cuts[:-1], cuts[1:]))
        out[lo, hi] = (level, kids)
        for c in kids:
            node(*c)

    edges = [0] + [k for k in range(1, len(keys)) if keys[k - 1] >> 30 != keys[k] >> 30] + [len(keys)]
    for lo, hi in zip(edges[:-1], edges[1:]):
        node(lo, hi)
    return out


def groups_plain(keys, span):
    """Maximal nodes of <= span bodies of the binary tree over (key, index)."""
    full = [(int(k) << 32) | i for i, k in enumerate(keys)]
    out = []

    def split(lo, hi):
        if hi - lo <= span and full[lo] >> 62 == full[hi - 1] >> 62:
            out.append((lo, hi - lo))
            return
        bit = (full[lo] ^ full[hi - 1]).bit_length() - 1
        mid = next(k for k in range(lo, hi) if (full[k] >> bit) & 1)
        split(lo, mid)
        split(mid, hi)

    split(0, len(keys))
    return out


# ------------------------------------------------------------- the kernels'
def prefix(x, ix):
    return ((1 << x.bit_length()) - 1, 2**32 - 1) if x else (0, (1 << ix.bit_length()) - 1)


def group_node(keys, i, span):
    """Bodies of the group node that starts at body i, 0 if none does."""
    n = len(keys)

    def shares(j, p):
        return 0 <= j < n and (int(keys[i]) ^ int(keys[j])) <= p[0] and (i ^ j) <= p[1]

    top = 1 << (span.bit_length() - 1)
    x = int(keys[i]) ^ int(keys[i - 1])
    if i > 0 and not x >> 30:
        p, h = prefix(x, i ^ (i - 1)), (span + 1) // 2
        if not shares(i - h, p) and not shares(i + h, p):
            return 0
        x, step = 0, top
        while step:
            if x + step <= span and shares(i - x - step, p):
                x += step
            step >>= 1
        if x < span and not shares(i - x + span, p):
            return 0
        q = (p[0] >> 1, 2**32 - 1 if p[0] else p[1] >> 1)
    else:
        q = ((1 << 30) - 1, 2**32 - 1)
    if i + span < n:
        r = prefix(int(keys[i]) ^ int(keys[i + span]), i ^ (i + span))
        q = min(q, (r[0] >> 1, 2**32 - 1 if r[0] else r[1] >> 1))
    t, step = 0, top
    while step:
        if t + step < span and shares(i + t + step, q):
            t += step
        step >>= 1
    return t + 1


def cells(keys, prune):
    """Candidates as k_cells takes them; child slots kept by first or last body."""
    n, past = len(keys), max(prune, 1)
    slot, by_lo, by_hi, roots = {}, {}, {}, []
    for k in range(n):
        l = lev(keys[k - 1], keys[k]) if k else -1
        if l < 0:
            end = next((j for j in range(k, n) if keys[j] >> 30 != keys[k] >> 30), n)
            roots.append((k, end, False))
        q = min(LEVELS - 1, lev(keys[k], keys[k + past])) if k + past < n else -1
        for level in range(l + 1, q + 1):
            shift = 3 * (LEVELS - 1 - level)
            ends, e = [], k
            for o in range(8):
                target = (((int(keys[k]) >> (shift + 3)) << 3) + o + 1) << shift
                while e < n and int(keys[e]) < target:
                    e += 1
                ends.append(e)
            starts = [k] + ends[:-1]
            kids = [(s, e, s == k) for s, e in zip(starts, ends) if e > s]
            if len(kids) < 2:
                continue
            end = ends[-1]
            first = end < n and lev(keys[end - 1], keys[end]) > l
            table, at = (by_hi, end - 1) if first else (by_lo, k)
            assert at not in table
            table[at] = kids
    return roots, by_lo, by_hi


def cases():
    rng = np.random.default_rng(5)
    out = []
    for n in (1, 2, 3, 31, 33, 200, 700):
        out.append(np.sort(rng.integers(0, 1 << 30, n)))
        out.append(np.sort(rng.integers(0, 1 << 9, n)))           # long runs, shallow
        out.append(np.sort(rng.integers(0, 40, n) << 14))         # buckets and gaps
        out.append(np.sort((rng.integers(0, 5, n) << 30) | rng.integers(0, 1 << 12, n) << 9))
    out.append(np.zeros(300, np.int64))
    out.append(np.full(70, (1 << 30) - 1, np.int64))
    out.append(np.sort((rng.integers(0, 300, 400) << 30) | (1 << 30) - 1))  # disks of one or two
    return out


@pytest.mark.parametrize("prune", [0, 1, 8, 12])
def test_cells_are_the_octree(prune):
    for keys in cases():
        want = octree_plain(keys, prune)
        roots, by_lo, by_hi = cells(keys, prune)
        seen, todo = {}, list(roots)
        while todo:
            lo, hi, first = todo.pop()
            level = LEVELS if hi - lo == 1 else lev(keys[lo], keys[hi - 1])
            kids = []
            if hi - lo > max(prune, 1) and level < LEVELS:  # as k_emit looks them up
                kids = by_hi[hi - 1] if first else by_lo[lo]
            assert (lo, hi) not in seen
            seen[lo, hi] = (level, [c[:2] for c in kids])
            todo += kids
        assert seen == want
        # and nothing else was given slots
        assert sum(map(len, by_lo.values())) + sum(map(len, by_hi.values())) \
            == sum(len(k) for _, k in want.values())


@pytest.mark.parametrize("span", [32, 64, 96, 256])
def test_group_nodes(span):
    for keys in cases():
        got = [(i, group_node(keys, i, span)) for i in range(len(keys))]
        assert [g for g in got if g[1]] == groups_plain(keys, span)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [2, 511, 512, 513, 2600, (1 << 18) - 1, (1 << 18) + 1])
def test_node_count_on_the_gpu(nb, cuda, n):
    """Every record of the full tree (one a distinct key, one a cell whose
    bodies fill two or more octants), at the edges of the blocks and of the
    rule on sizes; half of the bodies crowd into a few cells."""
    import torch
    rng = np.random.default_rng(n)
    pos = rng.uniform(-1.0, 1.0, (3, n)).astype(np.float32)
    pos[1] *= 0.01
    crowd = rng.random(n) < 0.5
    pos[:, crowd] = np.float32(0.3) + pos[:, crowd] * np.float32(0.004)
    p = nb.allocate_particles_gpu(n)
    for k, a in zip("xyz", pos):
        p.arrays[k].copy_(torch.from_numpy(a))
    p.arrays["mass"].fill_(1.0)
    t = nb.Octree(n)
    t.reset()
    t.bbox(p)
    t.build(p)
    t.summarize()
    st = t.stats()
    lo = np.array(st.root_center, np.float64) - float(st.root_half)
    c = np.clip((pos.astype(np.float64) - lo[:, None]) * (512.0 / float(st.root_half)), 0, 1023)
    keys = np.zeros(n, np.int64)
    for b in range(10):
        for k in range(3):
            keys |= ((c[k].astype(np.int64) >> b) & 1) << (3 * b + k)
    want = len(np.unique(keys))
    for level in range(LEVELS):
        kids = np.unique(keys >> (3 * (LEVELS - 1 - level)))
        want += int((np.unique(kids >> 3, return_counts=True)[1] > 1).sum())
    assert st.n_nodes == want
    assert abs(st.root_mass - n) < 1e-9 * n
