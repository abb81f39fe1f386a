"""The suffix array check's fast path (sliced inverse, one pass) and its hand-over to the kernels that
name the first failing index, on both sides of the size where the inverse is written by slices, and
the LCP array there: verdict, index and reason as the one-pass kernels give them."""
import numpy as np
import pytest

import sadcs_b200 as sa

pytestmark = pytest.mark.gpu

SLICED = 16 << 20  # entries from which arrays are written by slices


def _lcp_of_neighbours(text, suffixes, limit=64):
    """LCPs of neighbouring suffixes that are below `limit`, by comparing character by character."""
    import torch

    n = text.numel()
    a, b = suffixes[:-1], suffixes[1:]
    out = torch.zeros(n, dtype=torch.int64, device="cuda")
    open_ = torch.ones(n - 1, dtype=torch.bool, device="cuda")
    for k in range(limit):
        inside = (a + k < n) & (b + k < n)
        open_ &= inside & (text[(a + k).clamp(max=n - 1)] == text[(b + k).clamp(max=n - 1)])
        out[1:] += open_
    return out


@pytest.mark.parametrize("n,full", [(257, False), (100_000, False), (SLICED - 1, False), (SLICED, False),
                                    (SLICED + 4097, False), (SLICED, True), (SLICED + 4097, True)])
def test_verdicts(n, full):
    """full: the device's memory is filled until the pairs of the sliced writes (8n bytes) are not to be had and the
    inverse and the LCP array's Phi (4n) are."""
    import torch

    g = torch.Generator(device="cuda").manual_seed(n)
    text = torch.randint(0, 7, (n,), dtype=torch.uint8, device="cuda", generator=g)
    suffixes = torch.empty(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    sa.build_device(text.data_ptr(), n, suffixes.data_ptr(), None)

    def check():
        torch.cuda.synchronize()
        return sa.check_suffix_array_device(text.data_ptr(), n, suffixes.data_ptr())

    lcp = torch.empty_like(suffixes)
    correct = suffixes.clone()
    if full:
        check(), sa.lcp_device(text.data_ptr(), n, suffixes.data_ptr(), lcp.data_ptr())  # the kernels are loaded
        expected_lcp = _lcp_of_neighbours(text, suffixes.to(torch.int64))
        torch.cuda.empty_cache()
        sa.query_device()
        leave = 8 * n  # the check takes 4n, then 8n; the LCP array 12.13n, then 4.13n
        filler = torch.empty(torch.cuda.mem_get_info()[0] - leave, dtype=torch.uint8, device="cuda")
        assert 5 * n < torch.cuda.mem_get_info()[0] <= leave
        assert check() == (True, -1, None)
        sa.lcp_device(text.data_ptr(), n, suffixes.data_ptr(), lcp.data_ptr())
        suffixes[n // 2] = correct[n // 3]
        verdict = check()
        suffixes.copy_(correct)
        del filler
        torch.cuda.empty_cache()
        assert torch.equal(lcp.to(torch.int64), expected_lcp)
        assert verdict == (False, n // 3, "duplicate entry")
    assert check() == (True, -1, None)  # no error is left over
    sa.lcp_device(text.data_ptr(), n, suffixes.data_ptr(), lcp.data_ptr())
    assert torch.equal(lcp.to(torch.int64), _lcp_of_neighbours(text, suffixes.to(torch.int64)))
    i, j = n // 3, n - 2
    suffixes[[i, i + 1]] = correct[[i + 1, i]]  # neighbours exchanged: the pair itself or one beside it
    ok, index, reason = check()
    assert not ok and index in (i - 1, i) and reason == "SA[index] and SA[index + 1] out of order"
    suffixes.copy_(correct)
    suffixes[j] = correct[i]  # the earlier of two equal entries is reported
    assert check() == (False, i, "duplicate entry")
    suffixes.copy_(correct)
    suffixes[31] = n
    suffixes[j] = n + 5
    assert check() == (False, 31, "entry out of range")
    suffixes.copy_(correct)
    suffixes[0], suffixes[n - 1] = correct[n - 1], correct[0]
    assert not check()[0]
