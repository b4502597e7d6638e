"""GPU parity of the batched pipeline's bucket sorts on the shapes that decide
which of them a bucket takes: scattered and banded columns, rows with an
outlier, clusters beyond what a bin can rank, equal (row, col) entries, buckets
around 1024, 1536 and 2048 entries, one column, alternating kinds in a batch.
CSR bit-exact (equal entries in COO order), y within the tolerance."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _entries(kind, n, ncols, per_row, rng):
    L = np.full(n, per_row)
    if kind == "uneven":
        L = rng.integers(0, 2 * per_row + 1, size=n)
    r = np.repeat(np.arange(n), L)
    j = np.concatenate([np.arange(k) for k in L]) if n else np.zeros(0, dtype=np.int64)
    if kind == "band":
        c = r + j
    elif kind == "clusters":
        c = r * 7 + (j // 20) * (ncols // 3) + j % 20
    elif kind == "outlier":
        c = np.where(j == 0, ncols - 1, r + j)
    elif kind == "equal":
        c = r * 31 + (j // 5) * 17
    elif kind == "one":
        c = np.full(len(r), 3)
    else:  # scattered, uneven
        c = rng.integers(0, ncols, size=len(r))
    p = rng.permutation(len(r))
    return r[p].astype(np.int32), (c % ncols)[p].astype(np.int32)


def _check(hc, orc, dev, insts):
    rng = np.random.default_rng(1)
    rows, cols = (np.concatenate([i[k] for i in insts]) for k in (2, 3))
    vals = rng.uniform(-1, 1, size=len(rows))
    xs = [rng.uniform(-1, 1, size=i[1]) for i in insts]
    desc = np.array([[i[0], i[1], len(i[2])] for i in insts], dtype=np.int64)
    out = hc.batched_coo_csr_spmv(desc, *(torch.from_numpy(a).to(dev) for a in (rows, cols, vals, np.concatenate(xs))))
    hc.check(hc.device_check())
    rp, cc, cv, y = (t.cpu().numpy() for t in out)
    e = r = 0
    for k, (n, ncols, rr, ci) in enumerate(insts):
        v = vals[e:e + len(rr)]
        order = np.lexsort((np.arange(len(rr)), ci, rr))  # stable: equal entries in COO order
        assert np.array_equal(rp[r + k:r + k + n + 1], np.concatenate([[0], np.cumsum(np.bincount(rr, minlength=n))]))
        assert np.array_equal(cc[e:e + len(rr)], ci[order]) and np.array_equal(cv[e:e + len(rr)], v[order])
        want = np.bincount(rr, weights=v * xs[k][ci], minlength=n)
        bound = np.bincount(rr, weights=np.abs(v * xs[k][ci]), minlength=n)
        assert np.all(np.abs(y[r:r + n] - want) <= 1e-12 * np.maximum(bound, 1e-300))
        e += len(rr)
        r += n


@pytest.mark.parametrize("kind", ["scattered", "uneven", "band", "clusters", "outlier", "equal", "one"])
@pytest.mark.parametrize("per_row", [1, 12, 16, 17, 24, 25, 32, 33, 100])  # buckets of 64 .. 6400 entries
def test_kinds(hc, orc, dev, kind, per_row):
    rng = np.random.default_rng(per_row)
    n, ncols = 300, 200_003
    _check(hc, orc, dev, [(n, ncols, *_entries(kind, n, ncols, per_row, rng))])


@pytest.mark.parametrize("ncols", [1, 2, 65, (1 << 18) - 1, 1 << 18, (1 << 18) + 1])
def test_column_counts(hc, orc, dev, ncols):
    rng = np.random.default_rng(ncols)
    _check(hc, orc, dev, [(130, ncols, *_entries("scattered", 130, ncols, 9, rng))])


def test_mixed_batch(hc, orc, dev):
    rng = np.random.default_rng(2)
    kinds = ["scattered", "clusters", "band", "one", "uneven", "equal"]
    insts = []
    for k in range(60):
        n, ncols = int(rng.integers(1, 900)), int(rng.integers(1, 5000))
        insts.append((n, ncols, *_entries(kinds[k % 6], n, ncols, int(rng.integers(1, 40)), rng)))
    _check(hc, orc, dev, insts)
