"""Lines of different lengths filtered by several host threads at once: the
same kernel with different amounts of shared memory."""
import threading

import pytest
import torch

from nitorch_b200 import coeff

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("lengths", [(400, 200, 256), (1000, 5000, 20000)])
def test_lengths_in_parallel(lengths):
    inputs = [torch.randn(64, n, device="cuda") for n in lengths]
    refs = [coeff.spline_coeff(x, 3, 3) for x in inputs]
    torch.cuda.synchronize()
    failures = []

    def work(x, ref):
        try:
            with torch.cuda.stream(torch.cuda.Stream()):
                for _ in range(1500):
                    out = coeff.spline_coeff(x, 3, 3)
                torch.cuda.current_stream().synchronize()
            assert torch.equal(out, ref)
        except Exception as e:  # (raised in the test's own thread below)
            failures.append(e)

    threads = [threading.Thread(target=work, args=a) for a in zip(inputs, refs)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures[0]
