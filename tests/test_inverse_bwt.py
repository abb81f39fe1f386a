"""The inverse BWT's walk (check.cuh: pieces between splitter rows, chunks of 16 characters), against
the text: sizes around a splitter's 64 rows and a chunk, texts whose rows advance by multiples of the
splitters' spacing, runs, and BWTs that do not invert."""
import numpy as np
import pytest

import oracle
import sadcs_b200 as sa
from sadcs_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _device(a):
    import torch

    return torch.from_numpy(np.array(a, dtype=np.uint8)).cuda()


def _invert(bwt, primary):
    import torch

    d = _device(bwt)
    out = torch.empty_like(d)
    sa.inverse_bwt_device(d.data_ptr(), len(bwt), primary, out.data_ptr())
    return out.cpu().numpy()


def _texts(n):
    rng = np.random.default_rng(n)
    yield rng.integers(0, 256, n).astype(np.uint8)
    yield rng.integers(97, 99, n).astype(np.uint8)
    yield W.run_text(n)
    yield np.resize(np.arange(64, dtype=np.uint8), n)  # rows advance by n / 64
    yield np.resize(rng.integers(0, 4, 128).astype(np.uint8), n)
    yield W.fibonacci_text(n) if n >= 2 else W.run_text(n)


@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 63, 64, 65, 127, 129, 4096, 64 * 64, 64 * 64 * 4 + 1, 100_003])
def test_inverse(n):
    for text in _texts(n):
        bwt, primary = oracle.bwt_from_sa(text, oracle.doubling_sa(text))
        assert np.array_equal(_invert(bwt, primary), text)
        ok, index = sa.check_bwt(text, bwt, primary)
        assert ok and index == -1


@pytest.mark.parametrize("n", [2, 64, 1000, 50_001])
def test_not_invertible(n):
    """Exchanged characters and other primary rows: the same verdict as the oracle's walk."""
    rng = np.random.default_rng(n)
    text = rng.integers(0, 3, n).astype(np.uint8)
    bwt, primary = oracle.bwt_from_sa(text, oracle.doubling_sa(text))
    rejected = 0
    for k in range(12):
        b, p = bwt.copy(), primary
        if k % 3 == 2:
            p = int(rng.integers(1, n + 1))
        else:
            i, j = rng.integers(0, n, 2)
            b[i], b[j] = b[j], b[i]
        expected_ok, _ = oracle.check_bwt(text, b, p)
        ok, _ = sa.check_bwt(text, b, p)
        assert ok == expected_ok
        try:
            _invert(b, p)
        except sa.GpuError:
            rejected += 1
            assert not ok
    if n >= 64:
        assert rejected  # some of them miss rows
