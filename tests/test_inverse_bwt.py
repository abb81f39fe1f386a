"""The inverse BWT's walk (check.cuh: pieces between splitter rows, chunks of 16 characters), against
the text: sizes around a splitter's 128 rows and a chunk, texts whose rows advance by multiples of the
splitters' spacing, runs, and BWTs that do not invert, which must leave the memory beside the output alone.
The CPU tests run the kernels' own place arithmetic (tests/inverse_emulation.cu, built with nvcc)."""
import ctypes
import shutil
import subprocess
from pathlib import Path

import numpy as np
import pytest

import oracle
import sadcs_b200 as sa
from sadcs_b200 import workloads as W

HERE = Path(__file__).resolve().parent
SOURCE = HERE / "inverse_emulation.cu"
HEADERS = [HERE.parent / "sadcs_b200" / "csrc" / name for name in ("check.cuh", "common.cuh", "primitives.cuh")]
BUILT = HERE / "_build" / "libinverse_emulation.so"
_u8p = ctypes.POINTER(ctypes.c_uint8)


@pytest.fixture(scope="module")
def emulation():
    newest = max(p.stat().st_mtime for p in [SOURCE, *HEADERS])
    if not BUILT.exists() or BUILT.stat().st_mtime < newest:
        nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
        if not Path(nvcc).exists():
            pytest.skip("nvcc is needed to build the host run of the inverse's walk")
        BUILT.parent.mkdir(exist_ok=True)
        tmp = BUILT.with_suffix(".so.tmp")
        subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O2", "-Xcompiler", "-fPIC",
                        "-shared", "-o", str(tmp), str(SOURCE)], check=True)
        tmp.replace(BUILT)
    library = ctypes.CDLL(str(BUILT))
    library.inverse_emulate.argtypes = [_u8p, ctypes.c_int64, ctypes.c_int64, _u8p, ctypes.POINTER(ctypes.c_int64)]

    def run(bwt, primary):
        """(valid, text, characters placed outside the text)"""
        b = np.ascontiguousarray(bwt, dtype=np.uint8)
        text = np.zeros(len(b), np.uint8)
        outside = ctypes.c_int64()
        valid = library.inverse_emulate(b.ctypes.data_as(_u8p), len(b), primary, text.ctypes.data_as(_u8p),
                                        ctypes.byref(outside))
        return bool(valid), text, outside.value

    run.library = library
    return run


def _broken(n, count, seed):
    """Random bytes, and BWTs with two bytes exchanged or another primary row: (bwt, primary)."""
    rng = np.random.default_rng([n, seed])
    text = rng.integers(0, 3, n).astype(np.uint8)
    bwt, primary = oracle.bwt_from_sa(text, oracle.doubling_sa(text))
    for k in range(count):
        b, p = bwt.copy(), primary
        if k % 3 == 0:
            i, j = rng.integers(0, n, 2)
            b[i], b[j] = b[j], b[i]
        elif k % 3 == 1:
            p = int(rng.integers(1, n + 1))
        else:
            b = rng.integers(0, 4, n).astype(np.uint8)
        yield b, p


# a little under 128 * 2^k, where the laps that the jumps add up come closest to n, and other sizes
BROKEN_SIZES = [1, 2, 127, 128, 200, 250, 500, 510, 1000, 1020, 2040, 3000, 4090, 16_000]


@pytest.mark.parametrize("n", BROKEN_SIZES)
def test_places_of_broken_bwts(n, emulation):
    invalid = 0
    for bwt, primary in _broken(n, 90, 1):
        valid, text, outside = emulation(bwt, primary)
        assert outside == 0
        if n <= 3000:
            expected, _ = oracle.check_bwt(text, bwt, primary)
            assert not valid or expected
        invalid += not valid
    assert invalid or n < 127


@pytest.mark.parametrize("n", [1, 129, 257, 4096, 20_000])
def test_places(n, emulation):
    for text in _texts(n):
        bwt, primary = oracle.bwt_from_sa(text, oracle.doubling_sa(text))
        valid, inverse, outside = emulation(bwt, primary)
        assert valid and outside == 0 and np.array_equal(inverse, text)


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


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 2, 15, 16, 17, 63, 64, 65, 127, 128, 129, 255, 256, 257, 383, 384, 385, 4096,
                               64 * 64 * 4 + 1, 100_003])
def test_inverse(n):
    for text in _texts(n):
        bwt, primary = oracle.bwt_from_sa(text, oracle.doubling_sa(text))
        assert np.array_equal(_invert(bwt, primary), text)
        ok, index = sa.check_bwt(text, bwt, primary)
        assert ok and index == -1


@pytest.mark.gpu
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


@pytest.mark.gpu
@pytest.mark.parametrize("offset", [64, 65, 67, 78])
@pytest.mark.parametrize("n", BROKEN_SIZES)
def test_memory_beside_the_output(n, offset):
    """The output lies inside a larger buffer whose bytes before and after it stay as they were, whether the
    BWT inverts or not."""
    import torch

    margin = torch.full((n + 256,), 0xA5, dtype=torch.uint8, device="cuda")
    for bwt, primary in _broken(n, 30, 2):
        d = _device(bwt)
        torch.cuda.synchronize()
        try:
            sa.inverse_bwt_device(d.data_ptr(), n, primary, margin.data_ptr() + offset)
        except sa.GpuError:
            pass
        assert bool((margin[:offset] == 0xA5).all()) and bool((margin[offset + n:] == 0xA5).all())


@pytest.mark.gpu
@pytest.mark.parametrize("n", [1, 130, 100_000])
def test_walk_after_a_sort_that_gave_up(n, emulation):
    """The walk follows no order that its sort has not finished (every entry of this one leads to row 0)."""
    order = np.zeros(n, np.uint32)
    chunks = ctypes.c_int64(-1)
    walk = emulation.library.inverse_walk_after_time_out
    walk.restype = ctypes.c_int64
    walk.argtypes = [ctypes.POINTER(ctypes.c_uint32), ctypes.c_int64, ctypes.c_int64, ctypes.POINTER(ctypes.c_int64)]
    walked = walk(order.ctypes.data_as(ctypes.POINTER(ctypes.c_uint32)), n, 1, ctypes.byref(chunks))
    assert walked == 0 and chunks.value == 0
