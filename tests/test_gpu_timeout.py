"""GPU test of the timeout path of the runtime's bounded device waits.

Every device-side wait of this runtime (the mbarrier waits of the TMA kernels,
the tile-status waits of the decoupled look-back scans) gives up after a poll
limit, sets the device error word and returns, instead of hanging.  Here
hyd_cuda_selftest_timeout runs each of those two waits on a condition that
nothing satisfies (an mbarrier no thread arrives at; 32 tile flags no tile
publishes) with a short poll limit.  The test checks that hyd_cuda_check then
reports HYD_CUDA_ERR_TIMEOUT once, that the error is cleared by reading it, and
that a normal call right after gives the right result on the same context."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("which", [0, 1])
def test_bounded_wait_times_out_and_context_stays_usable(hc, orc, dev, which):
    L = hc.lib()
    s = torch.cuda.current_stream().cuda_stream
    assert hc.device_check() == hc.OK
    assert L.hyd_cuda_selftest_timeout(which, 1 << 12, s) == hc.OK, hc.last_error()
    assert L.hyd_cuda_check(s) == hc.ERR_TIMEOUT
    assert L.hyd_cuda_check(s) == hc.OK  # read and cleared
    n = 100_003
    xs = torch.empty(n, dtype=torch.float64, device=dev)
    ys = torch.empty(n, dtype=torch.float64, device=dev)
    hc.fill_uniform_f64(xs, 31, -1.0, 1.0)
    hc.fill_uniform_f64(ys, 32, -1.0, 1.0)
    out = torch.zeros(1, dtype=torch.float64, device=dev)
    hc.dot_f64(xs, ys, out)
    assert L.hyd_cuda_check(s) == hc.OK
    ref = orc.dot_compensated(orc.uniform_f64(n, 31, -1.0, 1.0), orc.uniform_f64(n, 32, -1.0, 1.0))
    assert abs(out.item() - ref) <= 1e-12 * max(1.0, abs(ref))
    # a scan (which uses the look-back wait) still completes normally
    x = torch.arange(1 << 16, dtype=torch.int64, device=dev)
    y = torch.empty_like(x)
    hc.scan(x, y)
    assert L.hyd_cuda_check(s) == hc.OK
    assert np.array_equal(y.cpu().numpy(), orc.scan_i64(x.cpu().numpy()))


def test_selftest_timeout_rejects_bad_arguments(hc, dev):
    L = hc.lib()
    assert L.hyd_cuda_selftest_timeout(2, 16, None) == hc.ERR_INVALID
    assert L.hyd_cuda_selftest_timeout(0, 0, None) == hc.ERR_INVALID
    assert L.hyd_cuda_selftest_timeout(0, (1 << 20) + 1, None) == hc.ERR_INVALID


@pytest.mark.parametrize("nnz", [2049, 70_001, 300_000])
def test_coo_sum_that_gives_up_writes_nothing_outside_its_outputs(hc, orc, dev, nnz):
    """One run of equal entries over all tiles, the first of which never
    publishes: the others have no place to write to (the first of them would be
    one before the outputs).  They leave their stores out, the outputs are zeros
    with a count of 0, the time-out is reported, and the next call is right."""
    L, s, guard, mark = hc.lib(), torch.cuda.current_stream().cuda_stream, 64, 0x5A5A5A5A5A5A
    rows = torch.zeros(nnz, dtype=torch.int64, device=dev)
    rows[nnz - 1:] = 3
    cols, vals = torch.ones_like(rows), torch.arange(nnz, dtype=torch.int64, device=dev)
    outs = [torch.full((nnz + 2 * guard,), mark, dtype=torch.int64, device=dev) for _ in range(3)]
    count = torch.full((2 * guard + 1,), mark, dtype=torch.int64, device=dev)
    inner = [o[guard:guard + nnz] for o in outs]
    assert hc.device_check() == hc.OK
    assert L.hyd_cuda_selftest_coo_timeout(rows.data_ptr(), cols.data_ptr(), vals.data_ptr(), nnz,
                                           *(o.data_ptr() for o in inner), count[guard:].data_ptr(), 1 << 10,
                                           s) == hc.OK, hc.last_error()
    assert L.hyd_cuda_check(s) == hc.ERR_TIMEOUT
    for o in outs:
        assert torch.all(o[:guard] == mark) and torch.all(o[guard + nnz:] == mark)
        assert torch.all(o[guard:guard + nnz] == 0)
    assert int(count[guard]) == 0 and torch.all(count[:guard] == mark) and torch.all(count[guard + 1:] == mark)
    assert L.hyd_cuda_check(s) == hc.OK  # read and cleared
    r, c, v, k = hc.coo_sum_duplicates(rows, cols, vals)
    assert hc.device_check() == hc.OK
    n = nnz - 1
    assert int(k) == 2 and r[:3].tolist() == [0, 3, 0] and v[:3].tolist() == [n * (n - 1) // 2, n, 0]


def test_selftest_coo_timeout_rejects_bad_arguments(hc, dev):
    L = hc.lib()
    t = torch.zeros(4096, dtype=torch.int64, device=dev)
    p = t.data_ptr()
    assert L.hyd_cuda_selftest_coo_timeout(p, p, p, 2048, p, p, p, p, 16, None) == hc.ERR_INVALID
    assert L.hyd_cuda_selftest_coo_timeout(p, p, p, 4096, p, p, p, p, 0, None) == hc.ERR_INVALID
    assert L.hyd_cuda_selftest_coo_timeout(p, p, p, 4096, p, p, p, None, 16, None) == hc.ERR_INVALID
