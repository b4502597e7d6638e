"""GPU parity of the batched pipeline's entry tiles (6144 entries, put into
bucket order in shared memory) at their edges: entry counts around one and two
tiles, one bucket, 4096 buckets (the most a tile counts in shared memory) and
one more, more tiles than blocks; and of the SpMV's chunks of rows at the
totals where their size changes.  CSR bit-exact (equal entries in COO order),
y within the tolerance; an invalid column is reported."""
import numpy as np
import pytest
import torch

from test_gpu_bucket_place import _check

pytestmark = pytest.mark.gpu


def _random(n, ncols, nnz, rng):
    """nnz entries, at most 200 in a row."""
    r = (rng.permutation(nnz) + int(rng.integers(0, n))) % n
    return n, ncols, r.astype(np.int32), rng.integers(0, ncols, size=nnz).astype(np.int32)


@pytest.mark.parametrize("nnz", [0, 1, 31, 511, 6143, 6144, 6145, 12287, 12288, 12289])
@pytest.mark.parametrize("n", [64, 65, 5000])
def test_tile_edges(hc, orc, dev, nnz, n):
    rng = np.random.default_rng(nnz + n)
    _check(hc, orc, dev, [_random(n, 977, min(nnz, 200 * n), rng)])


@pytest.mark.parametrize("n", [(1 << 18) - 64, 1 << 18, (1 << 18) + 1])
def test_bucket_count_edges(hc, orc, dev, n):
    rng = np.random.default_rng(n)
    _check(hc, orc, dev, [_random(n, 300_001, 20_001, rng), _random(n, 5, 7001, rng)])


def test_more_tiles_than_blocks(hc, orc, dev):
    rng = np.random.default_rng(3)
    _check(hc, orc, dev, [_random(40_001 + 64 * k, 30_000, 400_003 + 2 * k, rng) for k in range(8)])


@pytest.mark.parametrize("chunk", [32, 64, 128, 256])
@pytest.mark.parametrize("off", [-1, 0, 1])
def test_chunk_sizes(hc, orc, dev, chunk, off):
    # a chunk has 64, 128 or 256 rows once there is one such chunk per resident warp
    rows = torch.cuda.get_device_properties(dev).multi_processor_count * 32 * chunk + off
    rng = np.random.default_rng(chunk)
    insts = []
    for n in (rows // 3, 1, 33, rows - rows // 3 - 34):
        r = np.concatenate([rng.integers(0, n, size=n // 2), np.full(150, n // 2), np.full(100, n - 1)])
        insts.append((n, 999, rng.permutation(r).astype(np.int32), rng.integers(0, 999, size=len(r)).astype(np.int32)))
    _check(hc, orc, dev, insts)


@pytest.mark.parametrize("vals_off", [0, 1, 2, 3])
@pytest.mark.parametrize("cols_off", [0, 1, 2])
def test_output_alignments(hc, dev, vals_off, cols_off):
    """The SpMV reads the CSR by 4, 16 or 32 bytes, as it is aligned: the same bits."""
    rng = np.random.default_rng(5)
    n, ncols, r, c = _random(700, 800, 20_011, rng)
    desc = np.array([[n, ncols, len(r)]], dtype=np.int64)
    args = [torch.from_numpy(a).to(dev) for a in (r, c, rng.uniform(-1, 1, len(r)), rng.uniform(-1, 1, ncols))]
    want = hc.batched_coo_csr_spmv(desc, *args)
    got = [torch.empty(n + 1, dtype=torch.int64, device=dev),
           torch.empty(len(r) + cols_off, dtype=torch.int32, device=dev)[cols_off:],
           torch.empty(len(r) + vals_off, dtype=torch.float64, device=dev)[vals_off:],
           torch.empty(n, dtype=torch.float64, device=dev)]
    hc.call("hyd_cuda_batched_coo_csr_spmv_f64", 1, desc.ctypes.data, *(hc.ptr(t) for t in args + got),
            hc.stream_handle(None))
    hc.check(hc.device_check())
    assert all(torch.equal(a, b) for a, b in zip(got, want))


def test_invalid_column_is_reported(hc, orc, dev):
    rng = np.random.default_rng(4)
    n, ncols, r, c = _random(3000, 500, 13_000, rng)
    for bad in (500, -1):
        cb = c.copy()
        cb[6200] = bad
        desc = np.array([[n, ncols, len(r)]], dtype=np.int64)
        args = [torch.from_numpy(a).to(dev) for a in (r, cb, rng.uniform(-1, 1, len(r)), rng.uniform(-1, 1, ncols))]
        hc.batched_coo_csr_spmv(desc, *args)
        assert hc.device_check() == hc.ERR_BOUNDS
    _check(hc, orc, dev, [(n, ncols, r, c)])
