"""GPU parity of the scans at the edges of their splits: the 256-element steps
and per-warp ranges of the two-launch form, the 4096-element tiles of the
float64 look-back and the size where float64 changes from one to the other;
unaligned arrays; int64 bit-exact, float64 within the scan's tolerance."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
VARIANTS = [(False, False), (False, True), (True, False), (True, True)]  # (reverse, inclusive)


def _dev(a, dev, shift):
    t = torch.empty(len(a) + shift, dtype=torch.int64 if a.dtype == np.int64 else torch.float64, device=dev)[shift:]
    t.copy_(torch.from_numpy(a))
    return t


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("n", [255, 256, 257, 2047, 2048, 2049, 131_071, 131_072, 131_073, 1_245_184, 1_245_185,
                               3_000_001])
def test_scan_sizes(hc, orc, dev, n, shift):
    rng = np.random.default_rng(n)
    xi = rng.integers(-(1 << 62), 1 << 62, size=n).astype(np.int64)
    xf = rng.uniform(-1, 1, size=n)
    ti, tf = _dev(xi, dev, shift), _dev(xf, dev, shift)
    oi, of = torch.empty_like(_dev(xi, dev, shift)), torch.empty_like(tf)
    for rev, inc in VARIANTS:
        hc.scan(ti, oi, -3, rev, inc)
        hc.scan(tf, of, 0.5, rev, inc)
        hc.check(hc.device_check())
        assert np.array_equal(oi.cpu().numpy(), orc.scan_i64(xi, -3, rev, inc))
        bound = orc.scan_f64(np.abs(xf), 0.5, rev, inc)
        assert np.all(np.abs(of.cpu().numpy() - orc.scan_f64(xf, 0.5, rev, inc)) <= 1e-12 * np.maximum(bound, 1.0))


@pytest.mark.parametrize("n,limit", [(50_000, 2.7), (300_000, 3.4)])
def test_scan_f64_rounds_few_times_at_the_prefix_size(hc, dev, n, limit):
    """The largest error of a scan of n positive elements, in units of 2^-53 of
    the last value, on average over 10 arrays.  A value takes about four
    roundings at its own size, whatever the tile's (2.2 and 3.0 measured; five
    and more, with the small sums added to the prefix one by one, gave 3.6 and
    3.7)."""
    worst = []
    for seed in range(10):
        x = np.random.default_rng(seed).uniform(0, 1, n)
        t = torch.from_numpy(x).to(dev)
        out = torch.empty_like(t)
        hc.scan(t, out, inclusive=True)
        exact = np.cumsum(x.astype(np.longdouble))
        worst.append(float(np.abs(out.cpu().numpy().astype(np.longdouble) - exact).max() / exact[-1]) * 2.0 ** 53)
    assert float(np.mean(worst)) <= limit
