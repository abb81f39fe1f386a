"""The temporary memory of the calls without a context is kept between calls, up to a bound, and given
back before free memory is counted for a context or a server; threads on their own streams share it."""
import threading

import numpy as np
import pytest

import oracle
import sadcs_b200 as sa
from sadcs_b200 import workloads as W

pytestmark = pytest.mark.gpu


def _check(text, suffixes):
    sa.check_suffix_array_device(text.data_ptr(), text.numel(), suffixes.data_ptr())


def _inputs(n):
    import torch

    text = torch.randint(0, 256, (n,), dtype=torch.uint8, device="cuda")
    suffixes = torch.zeros(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    _check(text, suffixes)  # loads the kernels
    return text, suffixes


def _free():
    """The device's free memory, as it is: sadcs_gpu_query_device would give the kept memory back first."""
    import torch

    return torch.cuda.mem_get_info()[0]


def test_kept_and_given_back():
    n = 32 << 20
    text, suffixes = _inputs(n)
    sa.query_device()
    before = _free()
    _check(text, suffixes)
    kept = before - _free()
    assert kept >= 12 * n  # the inverse and the pairs of a check
    for _ in range(3):
        _check(text, suffixes)
    assert before - _free() == kept
    assert sa.query_device()["free_bytes"] == _free() >= before


def test_kept_memory_is_bounded():
    n = 256 << 20  # 3 GiB of temporary memory
    text, suffixes = _inputs(n)
    sa.query_device()
    before = _free()
    _check(text, suffixes)
    assert before - _free() <= (2 << 30) + (64 << 20)
    sa.query_device()


def test_kept_memory_is_had_by_others():
    """With the device full but for what the pool keeps, a context, a server's construction that its budget was
    promised before, and an allocation of another library are made from it."""
    import torch

    n = 120 << 20
    text, suffixes = _inputs(n)
    torch.cuda.empty_cache()
    request = W.natural_text(40 << 20, seed=6)
    expected = sa.build(request)
    room = 300 << 20  # the reserve that a context leaves free, and some
    with sa.Server(memory_budget=1 << 30, workers=1) as server:
        for use in ("context", "server", "allocation"):
            sa.query_device()
            _check(text, suffixes)
            filler = torch.empty(_free() - room, dtype=torch.uint8, device="cuda")
            assert _free() <= room
            if use == "context":
                with sa.Context(64 << 20):
                    pass
            elif use == "server":
                got = server.wait(server.submit(request))
                assert np.array_equal(got[0], expected[0]) and np.array_equal(got[1], expected[1])
            else:
                torch.empty(1 << 30, dtype=torch.uint8, device="cuda")
            del filler
            torch.cuda.empty_cache()


def test_threads_and_streams():
    import torch

    texts = [W.natural_text(200_000 + 1000 * k, seed=k) for k in range(4)]
    failures = []

    def work(text):
        try:
            expected = oracle.doubling_sa(text)
            bwt, primary = oracle.bwt_from_sa(text, expected)
            stream = torch.cuda.Stream()
            with torch.cuda.stream(stream):
                d_text = torch.from_numpy(text.copy()).cuda()
                d_sa = torch.from_numpy(expected.view(np.int32).copy()).cuda()
                d_bwt = torch.from_numpy(bwt.copy()).cuda()
                out = torch.empty_like(d_text)
                lcp = torch.empty_like(d_sa)
            stream.synchronize()
            for _ in range(5):
                h = stream.cuda_stream
                assert sa.check_suffix_array_device(d_text.data_ptr(), len(text), d_sa.data_ptr(), stream=h)[0]
                sa.inverse_bwt_device(d_bwt.data_ptr(), len(text), primary, out.data_ptr(), stream=h)
                sa.lcp_device(d_text.data_ptr(), len(text), d_sa.data_ptr(), lcp.data_ptr(), stream=h)
                stream.synchronize()
                assert np.array_equal(out.cpu().numpy(), text)
                assert np.array_equal(lcp.cpu().numpy().view(np.uint32), oracle.lcp(text, expected))
        except BaseException as e:  # noqa: BLE001 - reported by the test's thread
            failures.append(e)

    threads = [threading.Thread(target=work, args=(t,)) for t in texts]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures
