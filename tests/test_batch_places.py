"""Batches whose texts begin and end at every offset of a 16-byte piece, of a cover period and of a class
histogram's block, and one DNA text at every length modulo a stream word: each text's suffix array and
BWT against the oracle."""
import numpy as np
import pytest

import oracle
import sadcs_b200 as sa

pytestmark = pytest.mark.gpu


def _check_batch(texts):
    sas, bwts, primaries = sa.build_batch(texts)
    for t, s, b, p in zip(texts, sas, bwts, primaries):
        expected = oracle.doubling_sa(t)
        eb, ep = oracle.bwt_from_sa(t, expected)
        assert np.array_equal(s, expected) and np.array_equal(b, eb) and p == ep


@pytest.mark.parametrize("sigma", [4, 20, 256])
def test_offsets(sigma):
    rng = np.random.default_rng(sigma)
    lengths = list(range(1, 70)) + [65_535, 1, 65_536, 3, 131_073, 17]
    _check_batch([rng.integers(0, sigma, n).astype(np.uint8) for n in lengths])


@pytest.mark.parametrize("copies", [3, 700])
def test_large_groups_of_several_texts(copies):
    """Texts of the same repeats: groups past a block's size, every digit pass from one histogram."""
    rng = np.random.default_rng(copies)
    piece = rng.integers(0, 4, 128)
    texts = []
    for k in range(5):
        text = np.tile(piece, copies)
        text[rng.integers(0, len(text), 4)] = 3
        texts.append(text.astype(np.uint8))
    _check_batch(texts)


@pytest.mark.parametrize("n", list(range(2047, 2082)) + [(1 << 16) + 1])
def test_dna_lengths(n):
    text = np.frombuffer(b"ACGT", np.uint8)[np.random.default_rng(n).integers(0, 4, n)]
    s, b, p = sa.build(text)
    expected = oracle.doubling_sa(text)
    eb, ep = oracle.bwt_from_sa(text, expected)
    assert np.array_equal(s, expected) and np.array_equal(b, eb) and p == ep
