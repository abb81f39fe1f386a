"""Which merge kernel a construction takes: the count of its ties from the ranking's lists and the rule on it (host
code, through tests/plan_harness.cu), and on the GPU the choice for texts with and without repeats that the wide
kernel's words cannot tell apart, whose suffix arrays the device check accepts."""
import ctypes
import os
import re
import subprocess
import sys

import pytest

from tests.test_memory_plan import HERE, harness

_u64 = ctypes.c_uint64


def _ties(chars, live, passes):
    library = harness()
    library.tie_count.restype = _u64
    depth = (_u64 * len(passes))(*[p[0] for p in passes])
    left = (_u64 * len(passes))(*[p[1] for p in passes])
    return library.tie_count(_u64(chars), _u64(live), depth, left, len(passes))


def test_tie_count():
    assert _ties(16, 1000, [(7, 600), (14, 400), (21, 50)]) == 300  # two of seven characters past 14
    assert _ties(14, 1000, [(7, 600), (14, 400), (21, 50)]) == 400
    assert _ties(21, 1000, [(7, 600), (14, 400), (28, 50)]) == 225
    assert _ties(16, 1000, [(7, 600), (14, 0)]) == 0  # nothing left before the depth asked for
    assert _ties(37, 1000, [(17, 900), (34, 900), (66, 900), (132, 10)]) == 900
    assert _ties(5, 1000, [(10, 0)]) == 500
    assert _ties(30, 1000, [(20, 100), (40, 120)]) == 100  # decided directly: never more than before
    assert _ties(0, 1000, [(20, 100)]) == 1000
    live = (1 << 32) - 1
    assert _ties(42, live, [(10, live), (29, live), (48, live - 1)]) == live


@pytest.mark.parametrize("bits,share", [(3, 128), (4, 128), (5, 64), (6, 64), (7, 32), (8, 32)])
def test_rule(bits, share):
    library = harness()
    samples = 12_345_678
    assert library.wide_merge(bits, _u64(samples // share), _u64(samples))
    assert not library.wide_merge(bits, _u64(samples // share + 1), _u64(samples))
    assert not library.wide_merge(2, _u64(0), _u64(samples)) and not library.wide_merge(1, _u64(0), _u64(samples))


def test_characters_the_words_hold():
    library = harness()
    library.wide_merge_chars.restype = _u64
    for bits in range(3, 9):
        for outputs in (1, 1000, 1 << 20, 1 << 28, (1 << 32) - 1):
            chars = library.wide_merge_chars(bits, _u64(outputs))
            assert 112 // bits <= chars <= (112 + 32) // bits


CHILD = """
import sys
import torch
import sadcs_b200 as sa

sigma, length, copies = map(int, sys.argv[1:4])
n = 8 << 20
g = torch.Generator(device="cuda").manual_seed(length)
slots = n // length
words = torch.randint(0, sigma, (slots // copies, length), dtype=torch.uint8, device="cuda", generator=g)
text = words[torch.randperm(slots, device="cuda", generator=g) % len(words)].reshape(-1).contiguous()
out = torch.empty(text.numel(), dtype=torch.int32, device="cuda")
torch.cuda.synchronize()
sa.build_device(text.data_ptr(), text.numel(), out.data_ptr(), None)
assert sa.check_suffix_array_device(text.data_ptr(), text.numel(), out.data_ptr()) == (True, -1, None)
"""


@pytest.mark.gpu
@pytest.mark.parametrize("sigma,length,copies,kernel", [
    (256, 1000, 1, "wide"),  # no repeats
    (256, 12, 16, "wide"),   # shorter than the words
    (256, 19, 16, "tree"),   # longer than the 16 characters they hold, shorter than the next pass reaches
    (256, 100, 4, "tree"),
    (8, 1000, 1, "wide"),
    (8, 30, 16, "wide"),     # the words hold 42 characters of 3 bits
    (8, 100, 4, "tree"),
    (4, 1000, 1, "tree"),
])
def test_choice(sigma, length, copies, kernel):
    done = subprocess.run([sys.executable, "-c", CHILD, str(sigma), str(length), str(copies)], capture_output=True,
                          text=True, cwd=HERE.parent, env={**os.environ, "SADCS_TRACE": "1"}, timeout=300)
    assert done.returncode == 0, done.stderr[-2000:]
    assert re.findall(r"sadcs: merge (\w+),", done.stderr) == [kernel], done.stderr
