"""GPU parity of the dot and the sum where their form changes: the one-block
form's limit, its loads per thread, remainders of one to three elements, bases
that are not 32-byte aligned; the allocation-free dot gives the same bits."""
import math

import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("n", [1, 2, 255, 1023, 1025, 4096, 4099, 16_383, 16_384, 16_385, 16_387, 65_537, 311_297])
def test_sizes(hc, dev, n, shift):
    rng = np.random.default_rng(n)
    hx, hy = rng.uniform(-1, 1, size=n), rng.uniform(-1, 1, size=n)
    x, y = (torch.empty(n + shift, dtype=torch.float64, device=dev)[shift:] for _ in range(2))
    x.copy_(torch.from_numpy(hx))
    y.copy_(torch.from_numpy(hy))
    out = torch.full((3,), 9.0, dtype=torch.float64, device=dev)
    hc.dot_f64(x, y, out[0:1])
    hc.sum_f64(x, out[1:2])
    hc.call("hyd_cuda_dot_f64_noalloc", hc.ptr(x), hc.ptr(y), n, hc.ptr(out[2:3]), hc.stream_handle())
    d, s, d2 = out.cpu().tolist()
    # one rounding per operation of a chain or tree of fewer than 64 + n / 300 of them
    bound = (64 + n / 300) * 2.0 ** -53
    assert abs(d - math.fsum(hx * hy)) <= bound * np.abs(hx * hy).sum() + 2.0 ** -53 * np.abs(hx * hy).sum()
    assert abs(s - math.fsum(hx)) <= bound * np.abs(hx).sum()
    assert d == d2


def test_stream_handle_follows_the_current_stream(hc, dev):
    s = torch.cuda.Stream()
    with torch.cuda.stream(s):
        assert hc.stream_handle() == s.cuda_stream
    assert hc.stream_handle() == torch.cuda.current_stream().cuda_stream and hc.stream_handle(s) == s.cuda_stream
