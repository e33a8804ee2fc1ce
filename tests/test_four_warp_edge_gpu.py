"""The checks of test_block_walk_gpu.py on both sides of where four warps a
group become two."""
from __future__ import annotations

import pytest

import test_block_walk_gpu as block

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [25600, 25601])
def test_every_pair(nb, cuda, n):
    block.test_every_pair(nb, cuda, n)


@pytest.mark.parametrize("n", [25600, 25601])
def test_votes_and_theta(nb, cuda, port, n):
    block.test_votes_and_theta(nb, cuda, port, n)
