"""GPU parity of the evenly split segment sums (segmented_reduce and the SpMV
with the default row split) where the split can go wrong: boundaries at the
edges of the 256-value chunks and of the warps' ranges, pieces that cross many
warps, unaligned bases, row pointers that do not start at 0 or do not ascend."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _seg(hc, orc, dev, offsets, nv, shift):
    rng = np.random.default_rng(nv + shift)
    vi = rng.integers(-(1 << 62), 1 << 62, size=nv).astype(np.int64)
    vf = rng.uniform(-1, 1, size=nv)
    off = torch.from_numpy(offsets).to(dev)
    oi = torch.empty(len(offsets) - 1, dtype=torch.int64, device=dev)
    of = torch.empty(len(offsets) - 1, dtype=torch.float64, device=dev)
    ti = torch.empty(nv + shift, dtype=torch.int64, device=dev)[shift:]
    tf = torch.empty(nv + shift, dtype=torch.float64, device=dev)[shift:]
    ti.copy_(torch.from_numpy(vi))
    tf.copy_(torch.from_numpy(vf))
    hc.segmented_reduce(off, ti, oi, init=-5)
    hc.segmented_reduce(off, tf, of, init=0.5)
    hc.check(hc.device_check())
    assert np.array_equal(oi.cpu().numpy(), orc.segmented_reduce_i64(offsets, vi, -5))
    absum = orc.segmented_reduce_f64(offsets, np.abs(vf), 0.0)
    ref = orc.segmented_reduce_f64(offsets, vf, 0.5)
    assert np.all(np.abs(of.cpu().numpy() - ref) <= 1e-12 * np.maximum(absum, 1.0))


@pytest.mark.parametrize("shift", [0, 1, 2])  # 32-byte aligned values, and not
@pytest.mark.parametrize("step", [255, 256, 257, 2047, 2048, 1])
def test_segment_ends_at_chunk_and_range_edges(hc, orc, dev, step, shift):
    ends = np.arange(step, 200_001, step, dtype=np.int64)
    offsets = np.concatenate([[0, 0], np.repeat(ends, 1 + (np.arange(len(ends)) % 3 == 0))])
    _seg(hc, orc, dev, offsets, int(offsets[-1]) + 3, shift)


@pytest.mark.parametrize("n", [1, 256, 257, (1 << 21) + 5])
def test_one_segment_over_many_warps_between_short_ones(hc, orc, dev, n):
    lens = np.concatenate([[1, 0, 2], [n], [0, 3, 300]])
    _seg(hc, orc, dev, np.concatenate([[7], 7 + np.cumsum(lens)]).astype(np.int64), 7 + int(lens.sum()), 0)


def _csr(rng, nrows, ncols, kind):
    lens = np.minimum(rng.zipf(1.5, size=nrows), 256)
    if kind == "empty":
        lens[rng.random(nrows) < 0.9] = 0
    if kind == "long":
        lens[[3, nrows // 2, nrows - 1]] = [1000, 300_000, 257]
    row_ptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    nnz = int(row_ptr[-1])
    return row_ptr, rng.integers(0, ncols, size=nnz), rng.uniform(-1, 1, size=nnz), rng.uniform(-1, 1, size=ncols)


def _spmv(hc, dev, row_ptr, cols, vals, x, dtype, lanes=0, shift=0):
    def up(a, dt):
        t = torch.empty(len(a) + shift, dtype=dt, device=dev)[shift:]
        t.copy_(torch.from_numpy(a))
        return t
    y = torch.full((len(row_ptr) - 1,), -7.0, dtype=torch.float64, device=dev)
    hc.spmv_csr(torch.from_numpy(row_ptr).to(dev), up(cols, dtype), up(vals, torch.float64),
                torch.from_numpy(x).to(dev), y, lanes_per_row=lanes)
    return y


@pytest.mark.parametrize("dtype", [torch.int64, torch.int32])
@pytest.mark.parametrize("kind,shift", [("zipf", 0), ("zipf", 1), ("empty", 0), ("long", 0)])
def test_spmv_even_split(hc, orc, dev, kind, shift, dtype):
    nrows, ncols = (3 << 18) + 37, 70_001
    row_ptr, cols, vals, x = _csr(np.random.default_rng(5), nrows, ncols, kind)
    y = _spmv(hc, dev, row_ptr, cols, vals, x, dtype, shift=shift)
    hc.check(hc.device_check())
    assert torch.equal(y, _spmv(hc, dev, row_ptr, cols, vals, x, dtype, shift=shift))
    ref = orc.spmv_csr(row_ptr, cols, vals, x)
    bound = orc.spmv_csr(row_ptr, cols, np.abs(vals), np.abs(x))
    assert np.all(np.abs(y.cpu().numpy() - ref) <= 1e-12 * np.maximum(bound, 1e-300))


@pytest.mark.parametrize("case", ["starts_later", "descending_inside", "bad_column"])
def test_spmv_even_split_matches_the_lane_split(hc, dev, case):
    """Row pointers that do not start at 0 or do not ascend, and columns out of
    range, give what the lanes-per-row form gives (rows take what their two
    pointers span; a bad column is left out and reported)."""
    nrows, ncols = 3 << 18, 5000
    row_ptr, cols, vals, x = _csr(np.random.default_rng(6), nrows, ncols, "zipf")
    if case == "starts_later":
        row_ptr = row_ptr[1001:]
    elif case == "descending_inside":
        row_ptr[[500, 1000]] = row_ptr[[1000, 500]]
    else:
        cols[12345] = ncols
        cols[777] = -1
    if case == "starts_later":  # still enough rows for the even split
        row_ptr = np.concatenate([row_ptr, np.full(2000, row_ptr[-1])])
    y = _spmv(hc, dev, row_ptr, cols, vals, x, torch.int64)
    st = hc.device_check()
    want = _spmv(hc, dev, row_ptr, cols, vals, x, torch.int64, lanes=8)
    assert hc.device_check() == st == (hc.ERR_BOUNDS if case == "bad_column" else hc.OK)
    assert np.allclose(y.cpu().numpy(), want.cpu().numpy(), rtol=0, atol=1e-12 * 60_000)


@pytest.mark.parametrize("dtype", [torch.int32, torch.int64])
@pytest.mark.parametrize("per_row,lanes", [(1, False), (5, False), (8, False), (40, True), (100, True)])
def test_spmv_even_rows(hc, dev, per_row, lanes, dtype):
    """Rows of one length go by entries or by lanes, whichever the model says is
    faster; by lanes the sums are those of the lanes-per-row form, bit for bit."""
    nrows, ncols = (3 << 18) + 3, 9001
    rng = np.random.default_rng(per_row)
    row_ptr = np.arange(nrows + 1, dtype=np.int64) * per_row
    cols = rng.integers(0, ncols, size=nrows * per_row)
    vals, x = rng.uniform(-1, 1, size=nrows * per_row), rng.uniform(-1, 1, size=ncols)
    y = _spmv(hc, dev, row_ptr, cols, vals, x, dtype)
    want = _spmv(hc, dev, row_ptr, cols, vals, x, dtype, lanes=8)
    hc.check(hc.device_check())
    if lanes:
        assert torch.equal(y, want)
    assert np.allclose(y.cpu().numpy(), want.cpu().numpy(), rtol=0, atol=1e-12 * per_row)


def _with_empty_run(rng, n, where, filled):
    """Lengths of n rows, `filled` of them (the others empty in one run, or two)."""
    lens = np.zeros(n, dtype=np.int64)
    at = {"front": n - filled, "end": 0, "middle": 0}[where]
    lens[at:at + filled] = np.minimum(rng.zipf(1.5, size=filled), 256)
    if where == "middle":  # half of the filled rows move to the other end
        lens[n - filled // 2:], lens[filled // 2:filled] = lens[filled // 2:filled][-(filled // 2):].copy(), 0
    return lens


def _us(f, reps=5):
    """Fastest of a few timed runs on the current stream."""
    f()
    best = float("inf")
    for _ in range(reps):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        f()
        b.record()
        b.synchronize()
        best = min(best, 1e3 * a.elapsed_time(b))
    return best


@pytest.mark.parametrize("dtype", [torch.int64, torch.int32])
@pytest.mark.parametrize("where", ["front", "middle", "end"])
@pytest.mark.parametrize("nrows,filled", [(1 << 20, 1 << 19), (4_000_001, 40_000), (1 << 20, 2)])
def test_spmv_run_of_empty_rows(hc, orc, dev, nrows, filled, where, dtype):
    """Rows that are empty in one run, whose boundaries all stand at one entry,
    cost no more than they do with 8 lanes per row (twice that, for noise)."""
    rng = np.random.default_rng(filled)
    row_ptr = np.concatenate([[0], np.cumsum(_with_empty_run(rng, nrows, where, filled))]).astype(np.int64)
    nnz, ncols = int(row_ptr[-1]), 70_001
    cols, vals, x = rng.integers(0, ncols, size=nnz), rng.uniform(-1, 1, size=nnz), rng.uniform(-1, 1, size=ncols)
    rp, ci = torch.from_numpy(row_ptr).to(dev), torch.from_numpy(cols).to(dev, dtype)
    v, xt = torch.from_numpy(vals).to(dev), torch.from_numpy(x).to(dev)
    y = torch.full((nrows,), -7.0, dtype=torch.float64, device=dev)
    y8 = torch.empty_like(y)
    now = _us(lambda: hc.spmv_csr(rp, ci, v, xt, y))
    lanes = _us(lambda: hc.spmv_csr(rp, ci, v, xt, y8, lanes_per_row=8))
    hc.check(hc.device_check())
    bound = orc.spmv_csr(row_ptr, cols, np.abs(vals), np.abs(x))
    assert np.all(np.abs(y.cpu().numpy() - orc.spmv_csr(row_ptr, cols, vals, x)) <= 1e-12 * bound)
    assert now <= 2 * lanes


@pytest.mark.parametrize("where", ["front", "middle", "end"])
@pytest.mark.parametrize("nseg,filled", [(1_000_000, 2), (1 << 20, 1 << 19), (3_000_001, 100_000)])
def test_run_of_empty_segments(hc, orc, dev, nseg, filled, where):
    """Segments that are empty in one run cost about what as many cost with the
    empty ones spread between the others (four times that, for noise and the
    shares' unevenness)."""
    rng = np.random.default_rng(nseg)
    lens = _with_empty_run(rng, nseg, where, filled)
    offsets = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    _seg(hc, orc, dev, offsets, int(offsets[-1]), 0)
    spread = np.concatenate([[0], np.cumsum(rng.permutation(lens))]).astype(np.int64)
    v = torch.rand(int(offsets[-1]), dtype=torch.float64, device=dev)
    o = torch.empty(nseg, dtype=torch.float64, device=dev)
    a, b = torch.from_numpy(offsets).to(dev), torch.from_numpy(spread).to(dev)
    now = _us(lambda: hc.segmented_reduce(a, v, o, init=0.0))
    assert now <= 4 * _us(lambda: hc.segmented_reduce(b, v, o, init=0.0))


@pytest.mark.parametrize("nwords", [1, 37, 63, 64, 65, 129, 1000])
@pytest.mark.parametrize("step", [1, 3, 64, 255, 256, 300])
def test_equal_offsets_where_ranges_are_cut(hc, orc, dev, nwords, step):
    """`nwords` equal offsets every `step` values: cuts between the warps fall
    inside such a group, at its edges and around the 64 boundaries up to which
    a cut moves to a whole chunk."""
    ends = np.repeat(np.arange(0, 20_000, step, dtype=np.int64), nwords)[:1_500_000]
    offsets = np.concatenate([ends, np.full(nwords, ends[-1] + 100)])
    _seg(hc, orc, dev, offsets, int(offsets[-1]) + 100, 0)


@pytest.mark.parametrize("dtype", [torch.int64, torch.int32])
@pytest.mark.parametrize("per_row,long,count", [(8, 1_000_000, 1), (32, 1_000_000, 1), (32, 10_000_000, 1), (32, 1025, 9),
                                                (32, 5000, 3000), (100, 20_000, 70)])
def test_spmv_even_rows_and_a_few_long_ones(hc, orc, dev, per_row, long, count, dtype):
    """Rows of one length but for a few long ones that a sample of the rows does
    not show (neighbours among them): right, the same over runs, and the long
    rows are not left to 8 lanes each (a fifth of the time those take for the
    longest, 0.4 us per 8 entries, beside the time for the even rows alone)."""
    nrows, ncols = (3 << 18) + 3, 9001
    rng = np.random.default_rng(count)
    lens = np.full(nrows, per_row, dtype=np.int64)
    at = 4 * rng.integers(0, nrows // 4 - 1, size=count) + 1
    at[count // 2:] = at[:count - count // 2] + 1
    lens[np.minimum(at, nrows - 1)] = long
    row_ptr = np.concatenate([[0], np.cumsum(lens)]).astype(np.int64)
    nnz = int(row_ptr[-1])
    cols, vals, x = rng.integers(0, ncols, size=nnz), rng.uniform(-1, 1, size=nnz), rng.uniform(-1, 1, size=ncols)
    y = _spmv(hc, dev, row_ptr, cols, vals, x, dtype)
    assert torch.equal(y, _spmv(hc, dev, row_ptr, cols, vals, x, dtype))
    hc.check(hc.device_check())
    ref = orc.spmv_csr(row_ptr, cols, vals, x)
    bound = orc.spmv_csr(row_ptr, cols, np.abs(vals), np.abs(x))
    assert np.all(np.abs(y.cpu().numpy() - ref) <= 1e-12 * bound)
    rp, ci = torch.from_numpy(row_ptr).to(dev), torch.from_numpy(cols).to(dev, dtype)
    v, xt = torch.from_numpy(vals).to(dev), torch.from_numpy(x).to(dev)
    even = torch.arange(nrows + 1, device=dev) * per_row
    now = _us(lambda: hc.spmv_csr(rp, ci, v, xt, y))
    assert now <= 2 * _us(lambda: hc.spmv_csr(even, ci, v, xt, y)) + long / 8 * 0.4 / 5


def _big_matrix(dev, seed):
    """Row pointers, columns and values of an uneven matrix that the even split takes."""
    rng = np.random.default_rng(seed)
    nrows = (3 << 18) + 5
    row_ptr, cols, vals, x = _csr(rng, nrows, 9001, "zipf")
    return (torch.from_numpy(row_ptr).to(dev), torch.from_numpy(cols).to(dev), torch.from_numpy(vals).to(dev),
            torch.from_numpy(x).to(dev))


def test_spmv_first_call_on_a_stream_is_captured(hc, dev):
    """A captured SpMV needs nothing prepared, keeps no scratch of the stream it
    was captured on, and gives the sums of 8 lanes per row."""
    rp, ci, v, x = _big_matrix(dev, 8)
    y = torch.full((len(rp) - 1,), -7.0, dtype=torch.float64, device=dev)
    want = torch.empty_like(y)
    hc.spmv_csr(rp, ci, v, x, want, lanes_per_row=8)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=torch.cuda.Stream()):
        hc.spmv_csr(rp, ci, v, x, y)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, want)


def test_spmv_does_not_disturb_a_capture_on_another_stream(hc, dev):
    rp, ci, v, x = _big_matrix(dev, 9)
    y, one = torch.empty(len(rp) - 1, dtype=torch.float64, device=dev), torch.zeros(1, device=dev)
    other = torch.cuda.Stream()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=torch.cuda.Stream()):
        one.add_(1)
        hc.spmv_csr(rp, ci, v, x, y, stream=other)  # the first call on that stream
    g.replay()
    torch.cuda.synchronize()
    want = torch.empty_like(y)
    hc.spmv_csr(rp, ci, v, x, want)
    assert float(one) == 1.0 and torch.equal(y, want)


def test_spmv_from_two_threads_on_one_stream(hc, dev):
    """Calls of several threads on one stream, with calls that use the stream's
    workspace between them, give what they give alone."""
    import threading
    rp, ci, v, x = _big_matrix(dev, 10)
    xs = [x, x * 3.0, x - 0.25]
    alone = []
    for xk in xs:
        y = torch.empty(len(rp) - 1, dtype=torch.float64, device=dev)
        hc.spmv_csr(rp, ci, v, xk, y)
        alone.append(y)
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    got = [[torch.empty_like(alone[0]) for _ in range(30)] for _ in xs]
    out = torch.zeros(1, dtype=torch.float64, device=dev)

    def work(k):
        torch.cuda.set_device(dev)
        for y in got[k]:
            hc.spmv_csr(rp, ci, v, xs[k], y, stream=stream)

    def sums():
        torch.cuda.set_device(dev)
        for _ in range(60):
            hc.dot_f64(v, v, out, stream=stream)

    threads = [threading.Thread(target=work, args=(k,)) for k in range(len(xs))] + [threading.Thread(target=sums)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for k, ys in enumerate(got):
        assert all(torch.equal(y, alone[k]) for y in ys)
