"""Sample ranks of texts whose ranking groups have given sizes (copies of one stretch at the same
residue modulo the cover period): around the sizes at which a group changes from one thread to a block
to segmented passes, with keys that differ in one digit only and with keys that differ in all."""
import numpy as np
import pytest

import oracle
import sadcs_b200 as sa

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("sigma", [4, 30, 256])
@pytest.mark.parametrize("copies", [2, 8, 9, 31, 33, 256, 1023, 1024, 1025, 1500])
def test_groups(copies, sigma):
    rng = np.random.default_rng([copies, sigma])
    piece = rng.integers(0, sigma, 96)
    blocks = []
    for k in range(copies):
        tail = rng.integers(0, sigma, 32)
        if k % 3 == 0:  # these differ from one another in their last character only
            tail[:31] = piece[:31]
        blocks += [piece, tail]
    text = np.concatenate(blocks).astype(np.uint8)
    expected = oracle.sample_ranks_from_sa(oracle.doubling_sa(text), len(text))
    assert np.array_equal(sa.rank_sample(text), expected)


def test_equal_runs():
    text = np.concatenate([np.full(70_000, 5, np.uint8), np.resize(np.arange(7, dtype=np.uint8), 70_000)])
    expected = oracle.sample_ranks_from_sa(oracle.doubling_sa(text), len(text))
    assert np.array_equal(sa.rank_sample(text), expected)
