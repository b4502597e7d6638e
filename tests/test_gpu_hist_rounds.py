"""GPU parity of the shared-memory histogram at the edges of its rounds (every
thread of the grid takes one group of four values per round, two rounds are
loaded ahead of the two being added), with power-of-two bins and without,
negative values inside a group, and an unaligned array."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("bins", [64, 1000, 4096])
@pytest.mark.parametrize("rounds", [1, 2, 3, 4, 5, 6])
@pytest.mark.parametrize("off", [-1, 0, 1])
def test_rounds(hc, dev, bins, rounds, off):
    threads = torch.cuda.get_device_properties(dev).multi_processor_count * 2 * 512
    n = 4 * (rounds * threads + off) + 3
    rng = np.random.default_rng(rounds)
    x = rng.integers(0, 1 << 20, size=n, dtype=np.int64)
    bad = rng.integers(0, n, size=7)
    for skip in (0, 1):  # 32-byte aligned, and not
        for negative in (False, True):
            y = x[skip:].copy()
            if negative:
                y[bad % len(y)] = -1  # bin -1: out of range, reported
            data = torch.from_numpy(np.concatenate([x[:skip], y])).to(dev)[skip:]
            hist = torch.zeros(bins, dtype=torch.int64, device=dev)
            hc.weighted_histogram(data, hist)
            assert hc.device_check() == (hc.ERR_BOUNDS if negative else hc.OK)
            ok = y >= 0
            b = y[ok] % bins
            # 20-bit squares: the sums of the low and the high parts are exact in float64
            sq = y[ok] * y[ok]
            want = np.bincount(b, weights=sq & 0xFFFFF, minlength=bins).astype(np.int64) + (
                np.bincount(b, weights=sq >> 20, minlength=bins).astype(np.int64) << 20)
            assert np.array_equal(hist.cpu().numpy(), want)
