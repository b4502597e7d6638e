"""GPU parity of the histogram's remainder by a bin count that is no power of
two: values at the edges of its 32-bit and 64-bit forms (mixed inside one
32-byte group), multiples of the divisor, the most negative value; a negative
value with a remainder is out of range, reported and left out, as in C."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("strategy", [0, 4])  # AUTO, GLOBAL
@pytest.mark.parametrize("bins", [3, 5, 7, 1000, 1023, 1025, 65_537, 99_991])
@pytest.mark.parametrize("negative", [False, True])
def test_remainders(hc, dev, bins, negative, strategy):
    rng = np.random.default_rng(bins)
    edge = np.array([0, 1, (1 << 31) - 1, 1 << 31, (1 << 32) - 1, 1 << 32, (1 << 62) + 1, (1 << 63) - 1], dtype=np.int64)
    x = np.concatenate([edge, edge // bins * bins, edge // bins * bins - 1 + (edge < bins),
                        rng.integers(0, 1 << 20, size=40_000), rng.integers(0, (1 << 63) - 1, size=10_001),
                        rng.integers(0, 1 << 32, size=10_000)]).astype(np.int64)
    if negative:
        x[::17] = -(x[::17] // 2)
        x[5], x[4001] = np.iinfo(np.int64).min, -bins
    data = torch.from_numpy(x).to(dev)
    hist = torch.zeros(bins, dtype=torch.int64, device=dev)
    hc.weighted_histogram(data, hist, strategy=strategy)
    bin_ = np.array([int(np.sign(v)) * (abs(int(v)) % bins) for v in x], dtype=np.int64)
    ok = bin_ >= 0
    assert hc.device_check() == (hc.OK if ok.all() else hc.ERR_BOUNDS)
    want = np.zeros(bins, dtype=np.uint64)
    u = x[ok].view(np.uint64)
    with np.errstate(over="ignore"):
        np.add.at(want, bin_[ok], u * u)
    assert np.array_equal(hist.cpu().numpy().view(np.uint64), want)
