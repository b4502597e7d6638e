"""GPU parity of the stencil bodies that run on the integer pipe, bit for bit
against the same IEEE operations in numpy, on values at the edges of what they
take: ties, carries to the next power of two, nearly equal neighbours, wide and
borderline exponent gaps, the ends of the exponent range, and everything that
must go to the FP64 unit (zeros, subnormals, negatives, infinities, NaN)."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
KINDS = ["edges", "ties", "powers", "gaps", "low", "high", "near", "special"]


def _values(kind, n, rng):
    m = rng.integers(0, 1 << 52, size=n, dtype=np.uint64)
    e = np.full(n, 1023, dtype=np.uint64)
    if kind == "edges":
        e += rng.integers(0, 3, size=n, dtype=np.uint64)
    elif kind == "ties":  # few significant bits, gaps up to the grid's limit
        m &= ~((np.uint64(1) << rng.integers(0, 53, size=n, dtype=np.uint64)) - np.uint64(1))
        e += rng.integers(0, 9, size=n, dtype=np.uint64)
    elif kind == "powers":
        m |= np.uint64((1 << 52) - 1) & ~((np.uint64(1) << rng.integers(0, 12, size=n, dtype=np.uint64)) - np.uint64(1))
    elif kind == "gaps":
        e += rng.integers(0, 12, size=n, dtype=np.uint64)
    elif kind == "low":
        e = rng.integers(70, 90, size=n, dtype=np.uint64)
    elif kind == "high":
        e = rng.integers(2036, 2047, size=n, dtype=np.uint64)
    elif kind == "near":
        m &= np.uint64(0xFFF)
    else:
        e = rng.integers(0, 2048, size=n, dtype=np.uint64)
    x = ((e << np.uint64(52)) | m).view(np.float64)
    if kind == "special":
        pick = rng.integers(0, 12, size=n)
        for k, v in enumerate([0.0, -0.0, 5e-324, -1.5, np.inf, -np.inf, np.nan, np.finfo(float).tiny]):
            x[pick == k] = v
    return x


def _same(got, want):
    nan = np.isnan(want)
    assert np.array_equal(np.isnan(got), nan)
    assert np.array_equal(got[~nan].view(np.int64), want[~nan].view(np.int64))


def _step(kind, u):
    a, b = np.vstack([u[:1], u[:-1]]), np.vstack([u[1:], u[-1:]])
    c, d = np.hstack([u[:, :1], u[:, :-1]]), np.hstack([u[:, 1:], u[:, -1:]])
    t = ((a + b) + c) + d
    if kind == 0:
        return t + u * -4.0
    if kind == 1:
        return t / 4.0
    if kind == 2:
        return u + 0.1 * (t - 4.0 * u)
    return (t + u) / 5.0


@pytest.mark.parametrize("variant", [14, 20])  # a tiled and the plain kernel, everything on the integer pipe
@pytest.mark.parametrize("h,w", [(96, 128), (1300, 1024), (5600, 5600)])  # 1, 4 and 8 rows per thread
@pytest.mark.parametrize("values", KINDS)
def test_stencil_bodies(hc, dev, values, h, w, variant):
    if h * w > (1 << 24) and values not in ("edges", "gaps"):
        pytest.skip("the large grid takes two value sets")
    u = _values(values, h * w, np.random.default_rng(len(values) + h)).reshape(h, w)
    src = torch.from_numpy(u).to(dev)
    with np.errstate(all="ignore"):
        for kind in range(4):
            out = torch.empty_like(src)
            hc.stencil2d(kind, src, out, variant=variant)
            want = _step(kind, u)
            if kind == 0:  # e * -4 is rounded into the sum: exact unless it overflows
                fine = np.abs(u) < 1e307
                _same(np.where(fine, out.cpu().numpy(), 0.0), np.where(fine, want, 0.0))
            elif kind == 2:
                fine = np.abs(u) < 1e307
                _same(np.where(fine, out.cpu().numpy(), 0.0), np.where(fine, want, 0.0))
            else:
                _same(out.cpu().numpy(), want)


@pytest.mark.parametrize("values", KINDS)
def test_jacobi1d_mean(hc, dev, values):
    x = _values(values, 100_001, np.random.default_rng(1))
    src = torch.from_numpy(x).to(dev)
    out = torch.empty_like(src)
    hc.jacobi1d(src, out)
    with np.errstate(all="ignore"):
        want = ((np.concatenate([x[:1], x[:-1]]) + x) + np.concatenate([x[1:], x[-1:]])) / 3.0
    _same(out.cpu().numpy(), want)


@pytest.mark.parametrize("dt", [1.0, 0.5])
@pytest.mark.parametrize("values", KINDS)
def test_gray_scott_laplacians(hc, dev, values, dt):
    rng = np.random.default_rng(2)
    u, v = (_values(values, 97 * 130, rng).reshape(97, 130) for _ in range(2))
    p = hc.GrayScott(dt=dt)
    src = [torch.from_numpy(x).to(dev) for x in (u, v)]
    out = [torch.empty_like(x) for x in src]
    hc.gray_scott_step(*src, *out, params=p)

    def lap(x):
        return ((np.roll(x, 1, 0) + np.roll(x, -1, 0)) + np.roll(x, 1, 1)) + np.roll(x, -1, 1) - 4.0 * x

    with np.errstate(all="ignore"):
        uvv = u * v * v
        want = (u + dt * ((p.du * lap(u) - uvv) + p.feed * (1.0 - u)), v + dt * ((p.dv * lap(v) + uvv) - (p.feed + p.kill) * v))
    # 4x is exact unless it overflows
    fine = np.ones_like(u, dtype=bool)
    for x in (u, v):
        fine &= ~(np.abs(x) >= 1e307)
    for got, w in zip(out, want):
        _same(np.where(fine, got.cpu().numpy(), 0.0), np.where(fine, w, 0.0))


def _five(kind, p):
    """One step from a field padded by one on every side."""
    t = ((p[:-2, 1:-1] + p[2:, 1:-1]) + p[1:-1, :-2]) + p[1:-1, 2:]
    u = p[1:-1, 1:-1]
    return [t + u * -4.0, t / 4.0, u + 0.1 * (t - 4.0 * u), (t + u) / 5.0][kind]


@pytest.mark.parametrize("boundary,pad", [(1, dict(mode="wrap")), (2, dict(mode="reflect")),
                                          (3, dict(mode="constant", constant_values=0.25))])
@pytest.mark.parametrize("values", KINDS)
def test_boundary_bodies(hc, dev, values, boundary, pad):
    u = _values(values, 75 * 101, np.random.default_rng(boundary)).reshape(75, 101)
    src = torch.from_numpy(u).to(dev)
    fine = ~(np.abs(u) >= 1e307)  # 4e is exact unless it overflows
    with np.errstate(all="ignore"):
        for kind in range(4):
            out = torch.empty_like(src)
            hc.stencil2d_bnd(kind, boundary, src, out, fill=0.25)
            keep = fine if kind in (0, 2) else np.ones_like(fine)
            _same(np.where(keep, out.cpu().numpy(), 0.0), np.where(keep, _five(kind, np.pad(u, 1, **pad)), 0.0))


@pytest.mark.parametrize("values", KINDS)
def test_served_laplacian(hc, dev, values):
    u = _values(values, 130 * 257, np.random.default_rng(3)).reshape(130, 257)
    src = torch.from_numpy(u).to(dev)
    out = torch.empty_like(src)
    torch.cuda.synchronize()
    srv = hc.Server(budget_bytes=1 << 30)
    st, ticket = srv.submit(hc.Request(hc.REQ_LAPLACIAN, 130, 257, src.data_ptr(), None, None, None, out.data_ptr()))
    assert st == hc.OK
    srv.wait(ticket)
    fine = ~(np.abs(u) >= 1e307)
    with np.errstate(all="ignore"):
        want = _five(0, np.pad(u, 1, mode="edge"))
    _same(np.where(fine, out.cpu().numpy(), 0.0), np.where(fine, want, 0.0))
