"""Large texts of mutated repeats, whose small ranking groups are finished by comparing the suffixes
directly (lists of 8M samples and more in groups of about two): the device checker accepts the
suffix array (which is then the only correct one). Narrow and wide codes, exact copies that agree beyond
the direct comparison, and a copy that ends with the text."""
import pytest

import sadcs_b200 as sa

pytestmark = pytest.mark.gpu


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


@pytest.mark.parametrize("sigma,n", [(4, 450_000_001), (20, 260_000_003)])
def test_repeats(sigma, n):
    import torch

    text = _text(sigma, n, sigma)
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
