"""GPU parity of the one-pass coo_sum_duplicates and the fused CSR build where
their tiles can go wrong: sizes around the 2048-entry tile, runs over many
tiles, unaligned arrays, wrapping sums, rows out of order."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _t(a, dev, shift):
    t = torch.empty(len(a) + shift, dtype=torch.int64, device=dev)[shift:]
    t.copy_(torch.from_numpy(a))
    return t


@pytest.mark.parametrize("shift", [0, 1])
@pytest.mark.parametrize("nnz", [1, 7, 8, 9, 255, 2047, 2048, 2049, 4096, 100_001])
@pytest.mark.parametrize("run", [1, 3, 256, 5000])  # entries per run (about)
def test_runs_and_tiles(hc, orc, dev, nnz, run, shift):
    rng = np.random.default_rng(nnz + run)
    head = rng.random(nnz) < 1.0 / run
    seg = np.cumsum(head)
    rows, cols = seg // 7, seg % 7  # neighbouring runs share a row
    vals = rng.integers(-(1 << 63), (1 << 63) - 1, size=nnz)
    r, c, v, k = hc.coo_sum_duplicates(_t(rows, dev, shift), _t(cols, dev, shift), _t(vals, dev, shift))
    hc.check(hc.device_check())
    orr, oc, ov, ok = orc.coo_sum_duplicates(rows, cols, vals)
    assert int(k.item()) == ok
    assert np.array_equal(r.cpu().numpy(), orr) and np.array_equal(c.cpu().numpy(), oc)
    assert np.array_equal(v.cpu().numpy(), ov)


@pytest.mark.parametrize("nnz", [1, 31, 33, 70_001])
@pytest.mark.parametrize("order", ["sorted", "shuffled"])
def test_csr_counts(hc, orc, dev, nnz, order):
    rng = np.random.default_rng(nnz)
    rows = rng.integers(0, 500, size=nnz)
    if order == "sorted":
        rows.sort()
    cols, vals = rng.integers(0, 99, size=nnz), rng.integers(-9, 9, size=nnz)
    rp, ci, cv = hc.csr_from_sorted_coo(500, nnz, _t(rows, dev, 0), _t(cols, dev, 0), _t(vals, dev, 0))
    hc.check(hc.device_check())
    orp, oci, ocv = orc.csr_from_sorted_coo(500, nnz, rows, cols, vals)
    assert np.array_equal(rp.cpu().numpy(), orp)
    assert np.array_equal(ci.cpu().numpy(), oci) and np.array_equal(cv.cpu().numpy(), ocv)


def test_csr_without_rows(hc, dev):
    rp, ci, cv = hc.csr_from_sorted_coo(0, 3, *(_t(np.array([0, 1, 2]), dev, 0) for _ in range(3)))
    assert hc.device_check() == hc.ERR_BOUNDS
    assert rp.cpu().tolist() == [0] and ci.cpu().tolist() == [0, 0, 0]
