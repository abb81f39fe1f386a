"""Large texts of mutated repeats, whose small ranking groups are finished by comparing the suffixes
directly (lists of 8M samples and more in groups of about two): the device checker accepts the
suffix array (which is then the only correct one). Narrow and wide codes, exact copies that agree beyond
the direct comparison, and a copy that ends with the text. The CPU tests run the comparison and the sort
by it (tests/direct_emulation.cu, built with nvcc) on groups of every size."""
import ctypes
import itertools
import os
import re
import shutil
import subprocess
import sys
from pathlib import Path

import numpy as np
import pytest

import sadcs_b200 as sa

HERE = Path(__file__).resolve().parent
SOURCE = HERE / "direct_emulation.cu"
HEADERS = [HERE.parent / "sadcs_b200" / "csrc" / name
           for name in ("segsort.cuh", "alphabet.cuh", "common.cuh", "primitives.cuh")]
BUILT = HERE / "_build" / "libdirect_emulation.so"
_u8p, _u32p = ctypes.POINTER(ctypes.c_uint8), ctypes.POINTER(ctypes.c_uint32)


@pytest.fixture(scope="module")
def direct():
    newest = max(p.stat().st_mtime for p in [SOURCE, *HEADERS])
    if not BUILT.exists() or BUILT.stat().st_mtime < newest:
        nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
        if not Path(nvcc).exists():
            pytest.skip("nvcc is needed to build the host run of the direct comparison")
        BUILT.parent.mkdir(exist_ok=True)
        tmp = BUILT.with_suffix(".so.tmp")
        subprocess.run([nvcc, "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O2", "-Xcompiler", "-fPIC",
                        "-shared", "-o", str(tmp), str(SOURCE)], check=True)
        tmp.replace(BUILT)
    library = ctypes.CDLL(str(BUILT))
    library.direct_sort.argtypes = [_u8p, ctypes.c_int64, ctypes.c_uint32, ctypes.c_uint32, ctypes.c_uint32, _u32p, _u32p]
    library.direct_sort.restype = None

    def run(codes, bits, depth, positions):
        """(positions in the order found, their group numbers)"""
        t = np.ascontiguousarray(codes, dtype=np.uint8)
        p = np.array(positions, dtype=np.uint32)
        number = np.zeros(len(p), np.uint32)
        library.direct_sort(t.ctypes.data_as(_u8p), len(t), bits, depth, len(p), p.ctypes.data_as(_u32p),
                            number.ctypes.data_as(_u32p))
        return p.tolist(), number.tolist()

    run.words = library.direct_words()
    return run


def _check_group(direct, codes, bits, depth, positions):
    """Suffixes of different numbers are in suffix order, members of one number are any order of a group."""
    found, number = direct(codes, bits, depth, positions)
    assert sorted(found) == sorted(positions) and number == sorted(number)
    suffixes = [bytes(np.asarray(codes[p:], np.uint8)) for p in found]
    for i, j in itertools.combinations(range(len(found)), 2):
        assert number[i] == number[j] or suffixes[i] < suffixes[j], (found, number, i, j)


@pytest.mark.parametrize("bits", [2, 3, 5, 8])
def test_a_suffix_that_ends_in_the_last_word(bits, direct):
    """One suffix ends inside the last word compared and is a prefix of the others, which differ after its
    end within that word: it comes first whatever order the group is in."""
    rng = np.random.default_rng(bits)
    depth, per_word = 46, 64 // bits
    for inside in range(1, per_word + 1):
        length = depth + (direct.words - 1) * per_word + inside
        piece = rng.integers(0, 1 << bits, length)
        gap = rng.integers(0, 1 << bits, 70)
        codes = np.concatenate([piece, [2, 0], gap, piece, [1, 3], gap, piece, [1, 0], gap, piece])
        starts = [0, length + 72, 2 * (length + 72), 3 * (length + 72)]
        for order in itertools.permutations(starts):
            number = _check_group(direct, codes, bits, depth, list(order))


@pytest.mark.parametrize("bits", [2, 4, 6, 8])
def test_groups_of_every_size(bits, direct):
    """Copies of a stretch with changes at every distance, some of them the text's last suffixes."""
    rng = np.random.default_rng([bits, 7])
    reach = 20 + direct.words * (64 // bits)
    for trial in range(400):
        size = int(rng.integers(2, 9))
        length = int(rng.integers(20, reach + 40))
        piece = rng.integers(0, 1 << bits, length)
        blocks, starts, at = [], [], 0
        for k in range(size):
            copy = piece.copy()
            if length > 21 and rng.random() < 0.7:
                change = rng.integers(20, length, int(rng.integers(1, 3)))
                copy[change] = rng.integers(0, 1 << bits, len(change))
            starts.append(at)
            blocks.append(copy)
            if k + 1 < size or rng.random() < 0.3:
                blocks.append(rng.integers(0, 2, int(rng.integers(1, 40))))
            at = sum(map(len, blocks))
        starts = [int(s) for s in rng.permutation(starts)]
        _check_group(direct, np.concatenate(blocks).astype(np.uint8), bits, 20, starts)


def _text(sigma, n, seed):
    import torch

    g = torch.Generator(device="cuda").manual_seed(seed)
    text = torch.randint(65, 65 + sigma, (n,), dtype=torch.uint8, device="cuda", generator=g)
    piece, base = 1 << 20, n * 6 // 10
    at = base
    k = 0
    while at < n:
        m = min(piece, n - at)
        start = 0 if at + m == n else int(torch.randint(0, base - piece, (1,), device="cuda", generator=g))
        copy = text[start:start + m].clone()
        if k % 7:  # every seventh copy stays exact
            changed = torch.rand(m, device="cuda", generator=g) < 0.01
            fresh = torch.randint(65, 65 + sigma, (m,), dtype=torch.uint8, device="cuda", generator=g)
            copy = torch.where(changed, fresh, copy)
        text[at:at + m] = copy
        at += m
        k += 1
    return text


@pytest.mark.gpu
@pytest.mark.parametrize("sigma,n", [(4, 450_000_001), (20, 260_000_003)])
def test_repeats(sigma, n):
    import torch

    text = _text(sigma, n, sigma)
    # Every length of a last suffix: copies of the text's end that go on differently, the larger one first.
    for k, tail in enumerate(range(40, 400)):
        piece = text[n - tail:].clone()
        for c, (last, at) in enumerate(((66, 0), (65, 1))):
            start = ((k * 2 + at) * 65536 + 32) // 32 * 32 + (n - tail) % 32  # the same residue: sampled together
            text[start:start + tail] = piece
            text[start + tail] = last
    suffixes = torch.empty(n, dtype=torch.int32, device="cuda")
    bwt = torch.empty(n, dtype=torch.uint8, device="cuda")
    torch.cuda.synchronize()
    stats = sa.Stats()
    with sa.Context(n) as context:
        primary = sa.build_device(text.data_ptr(), n, suffixes.data_ptr(), bwt.data_ptr(), context, stats=stats)
    assert stats.doubling_rounds > 0
    assert sa.check_suffix_array_device(text.data_ptr(), n, suffixes.data_ptr()) == (True, -1, None)
    out = torch.empty_like(text)
    sa.inverse_bwt_device(bwt.data_ptr(), n, primary, out.data_ptr())
    assert torch.equal(out, text)


TRACED = """
import sys
import torch
import sadcs_b200 as sa

sigma, copies, rate = int(sys.argv[1]), int(sys.argv[2]), float(sys.argv[3])
n = 32 << 20
g = torch.Generator(device="cuda").manual_seed(sigma)
x = torch.randint(0, sigma, (n,), dtype=torch.uint8, device="cuda", generator=g)
parts = [x]
for _ in range(copies):
    changed = torch.rand(n, device="cuda", generator=g) < rate
    parts.append(torch.where(changed, torch.randint(0, sigma, (n,), dtype=torch.uint8, device="cuda", generator=g), x))
text = torch.cat(parts)
out = torch.empty(text.numel(), dtype=torch.int32, device="cuda")
torch.cuda.synchronize()
sa.build_device(text.data_ptr(), text.numel(), out.data_ptr(), None)
assert sa.check_suffix_array_device(text.data_ptr(), text.numel(), out.data_ptr()) == (True, -1, None)
"""


@pytest.mark.gpu
@pytest.mark.parametrize("sigma,copies,rate,passes", [(4, 1, 0.0, 1), (256, 2, 0.0, 1), (4, 1, 0.02, 1), (256, 1, 0.03, 1)])
def test_direct_comparison_is_tried_and_left(sigma, copies, rate, passes):
    """A text and copies of it: with changes the sample is decided and so are the groups; exact copies are sampled in
    one pass, not compared beyond the sample, and not sampled again."""
    done = subprocess.run([sys.executable, "-c", TRACED, str(sigma), str(copies), str(rate)], capture_output=True,
                          text=True, cwd=HERE.parent, env={**os.environ, "SADCS_TRACE": "1"}, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
    found = [tuple(map(int, m)) for m in re.findall(
        r"direct comparison decided (\d+) of (\d+) sampled, (\d+) in all", done.stderr)]
    assert len(found) == passes, done.stderr
    decided, sampled, total = found[0]
    assert sampled > 0
    if rate:
        assert 4 * decided >= sampled and total > 32 * decided
    else:
        assert decided == 0 and total == 0
