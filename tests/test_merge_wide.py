"""The merge kernel for texts with few long repeats (merge_wide.cuh), against the oracle: sizes around
one tile and around a level's first tiles, every code width it takes, ties that its words do not
decide (below the share of deep samples that sends a text to the other kernel), long common prefixes
inside a tile, and many texts in one tile."""
import numpy as np
import pytest

import oracle
import sadcs_b200 as sa

pytestmark = pytest.mark.gpu

TILE = 32 * ((253 * 7 - 187) // 32) + 187  # the records a tile holds


def _check(text):
    text = np.ascontiguousarray(text, dtype=np.uint8)
    expected = oracle.doubling_sa(text)
    eb, ep = oracle.bwt_from_sa(text, expected)
    s, b, p = sa.build(text)
    assert np.array_equal(s, expected)
    assert np.array_equal(b, eb) and p == ep


@pytest.mark.parametrize("sigma", [5, 20, 50, 100, 256])
@pytest.mark.parametrize("n", [1, 40, TILE - 1, TILE, TILE + 1, 2 * TILE + 3, 32 * TILE + 17, 200_003])
def test_sizes(sigma, n):
    _check(np.random.default_rng([sigma, n]).integers(0, sigma, n))


@pytest.mark.parametrize("sigma,copies,length", [(20, 2, 1500), (20, 5, 400), (200, 40, 60), (60, 3, 700)])
def test_ties(sigma, copies, length):
    """Copies of one stretch: groups of `copies` suffixes that agree beyond a record's words, ending
    with the text in one case in two."""
    rng = np.random.default_rng([sigma, copies])
    n = 40 * copies * length
    text = rng.integers(0, sigma, n)
    piece = rng.integers(0, sigma, length)
    for k in range(copies):
        at = n - length if k == 0 and copies % 2 else int(rng.integers(0, n - length))
        text[at:at + length] = piece
    _check(text)


def test_long_prefix_in_a_tile():
    """A run of one byte longer than a tile: the tile's common prefix exceeds the bits left out."""
    rng = np.random.default_rng(9)
    text = rng.integers(0, 250, 400_000)
    text[1000:1000 + 3 * TILE] = 7
    _check(text)
    text[-2 * TILE:] = 0  # the run ends with the text, in the smallest code
    _check(text)


@pytest.mark.parametrize("sigma", [20, 256])
def test_many_texts_in_a_tile(sigma):
    rng = np.random.default_rng(sigma)
    lengths = np.concatenate([np.ones(700, int), rng.integers(1, 40, 300), [5000, 1, 1, 70_000, 2, 33]])
    texts = [rng.integers(0, sigma, n).astype(np.uint8) for n in lengths]
    sas, bwts, primaries = sa.build_batch(texts)
    for t, s, b, p in zip(texts, sas, bwts, primaries):
        expected = oracle.doubling_sa(t)
        eb, ep = oracle.bwt_from_sa(t, expected)
        assert np.array_equal(s, expected) and np.array_equal(b, eb) and p == ep
