"""The temporary memory of the calls without a context is kept between calls, up to a bound, and given
back before free memory is counted for a context or a server; threads on their own streams share it."""
import threading

import numpy as np
import pytest

import oracle
import sadcs_b200 as sa
from sadcs_b200 import workloads as W

pytestmark = pytest.mark.gpu


def test_given_back():
    import torch

    n = 8 << 20
    text = torch.randint(0, 256, (n,), dtype=torch.uint8, device="cuda")
    suffixes = torch.zeros(n, dtype=torch.int32, device="cuda")
    torch.cuda.synchronize()
    sa.check_suffix_array_device(text.data_ptr(), n, suffixes.data_ptr())  # loads the kernels
    before = sa.query_device()["free_bytes"]
    for _ in range(3):
        sa.check_suffix_array_device(text.data_ptr(), n, suffixes.data_ptr())
    assert sa.query_device()["free_bytes"] >= before


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
