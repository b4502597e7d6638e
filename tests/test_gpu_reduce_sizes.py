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


@pytest.mark.parametrize("shift", [0, 1])  # 32-byte aligned, and not
@pytest.mark.parametrize("op,limit", [("dot", 0.0242), ("sum", 0.0182)])
def test_short_arrays_round_no_more_than_long_ones(hc, dev, op, limit, shift):
    """Root mean square error over 200 arrays of 16000 elements in [-1, 1), in
    units of 2^-53 of the sum of magnitudes: at most 1.3 times the 0.0186 and
    0.0140 that the form for long arrays has at this size."""
    n, err = 16000, []
    b = [torch.empty(n + shift, dtype=torch.float64, device=dev)[shift:] for _ in range(2)]
    out = torch.zeros(1, dtype=torch.float64, device=dev)
    for seed in range(200):
        rng = np.random.default_rng(seed)
        x, y = rng.uniform(-1, 1, n), rng.uniform(-1, 1, n)
        b[0].copy_(torch.from_numpy(x))
        b[1].copy_(torch.from_numpy(y))
        if op == "dot":
            hc.dot_f64(b[0], b[1], out)
            hi = x * y
            # the products' rounding errors, exactly (Dekker's splitting)
            s = [a - (a * 134217729.0 - (a * 134217729.0 - a)) for a in (x, y)]
            t = [a - lo for a, lo in zip((x, y), s)]
            lo = ((t[0] * t[1] - hi) + t[0] * s[1] + s[0] * t[1]) + s[0] * s[1]
            exact, mag = math.fsum(np.concatenate([hi, lo]).tolist() + [-out.item()]), np.abs(hi).sum()
        else:
            hc.call("hyd_cuda_sum_f64", hc.ptr(b[0]), n, hc.ptr(out), hc.stream_handle())
            exact, mag = math.fsum(x.tolist() + [-out.item()]), np.abs(x).sum()
        err.append(exact / mag * 2.0 ** 53)
    assert float(np.sqrt(np.mean(np.square(err)))) <= limit
