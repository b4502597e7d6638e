"""GPU parity of the one-sweep radix sort and the vectorised gather where their
tiles and record formats change: sizes around a tile, every number of passes,
digits that all keys share, 2^30 keys; gathers of whole 32-byte groups,
remainders, unaligned arrays and indices out of range inside a group."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def _perm(hc, dev, keys, key_bits=None):
    k = torch.from_numpy(keys).to(dev)
    p = torch.full_like(k, -1)
    hc.sort_indices(k, p, key_bits=key_bits)
    hc.check(hc.device_check())
    return p.cpu().numpy()


@pytest.mark.parametrize("n", [31, 3071, 3072, 3073, 6143, 6144, 6145, 12289, 200_003])
@pytest.mark.parametrize("bits", [8, 16, 32, 40, 41, 48, 56, 63])  # 1, 2, 4, 5, 6, 6, 7, 8 passes
def test_sizes_and_passes(hc, orc, dev, n, bits):
    rng = np.random.default_rng(n + bits)
    keys = rng.integers(0, (1 << bits) - 1, size=n, dtype=np.int64, endpoint=True)
    keys[n // 2] = (1 << bits) - 1
    keys[rng.integers(0, n, size=n // 3)] = keys[0]
    ref = orc.sort_indices(keys)
    assert np.array_equal(_perm(hc, dev, keys), ref)
    assert np.array_equal(_perm(hc, dev, keys, key_bits=bits), ref)


@pytest.mark.parametrize("kind", ["shared_digits", "negative", "all_negative", "extremes"])
def test_digit_patterns(hc, orc, dev, kind):
    rng = np.random.default_rng(3)
    keys = rng.integers(0, 7, size=50_001, dtype=np.int64)
    if kind == "shared_digits":
        keys = keys * 256 + 0x5A00000077
    elif kind == "negative":
        keys = (keys - 3) * 1_000_003
    elif kind == "all_negative":
        keys = -1 - keys * 70_000
    else:
        keys[::5] = np.iinfo(np.int64).min
        keys[1::5] = np.iinfo(np.int64).max
    assert np.array_equal(_perm(hc, dev, keys), orc.sort_indices(keys))


def test_two_to_the_30_keys(hc, dev):
    """Above 2^30 keys counts and indices take 64 bits: the permutation sorts
    the keys, keeps the order of equal ones and has every index once."""
    n = (1 << 30) + 4097
    if torch.cuda.mem_get_info()[0] < 80 << 30:
        pytest.skip("needs 80 GB of device memory")
    keys = torch.empty(n, dtype=torch.int64, device=dev)
    hc.fill_uniform_i64(keys, 8, 1 << 20)
    perm = torch.empty_like(keys)
    hc.sort_indices(keys, perm)
    hc.check(hc.device_check())
    seen = torch.zeros(n, dtype=torch.bool, device=dev)
    seen[perm] = True
    assert bool(seen.all())
    del seen
    s = keys[perm]
    del keys
    for a in range(0, n - 1, 1 << 28):
        b = min(a + (1 << 28), n - 1)
        x, y = s[a:b], s[a + 1:b + 1]
        assert bool(((x < y) | ((x == y) & (perm[a:b] < perm[a + 1:b + 1]))).all())
    del s, perm
    hc.lib().hyd_cuda_cleanup()  # gives the large scratch back
    hc.check(hc.lib().hyd_cuda_init())


@pytest.mark.parametrize("dtype", [torch.int64, torch.float64, torch.int32])
@pytest.mark.parametrize("n,shift", [(400_003, 0), (400_000, 1), (1_000_000, 0), (1_300_001, 0)])
def test_gather_groups(hc, dev, n, shift, dtype):
    rng = np.random.default_rng(n)
    src = rng.integers(-1000, 1000, size=70_001)
    perm = torch.empty(n + shift, dtype=torch.int64, device=dev)[shift:]
    idx = rng.integers(0, len(src), size=n)
    perm.copy_(torch.from_numpy(idx))
    out = torch.full((n + shift,), -5, dtype=dtype, device=dev)[shift:]
    d_src = torch.from_numpy(src).to(dev).to(dtype)
    hc.gather(perm, d_src, out)
    hc.check(hc.device_check())
    assert np.array_equal(out.cpu().numpy(), src[idx].astype(out.cpu().numpy().dtype))
    # out of range: reported, left unwritten, the rest of its group served
    idx[[0, 5, n // 2, n - 1]] = [-1, len(src), 1 << 60, len(src)]
    perm.copy_(torch.from_numpy(idx))
    out.fill_(-5)
    hc.gather(perm, d_src, out)
    assert hc.device_check() == hc.ERR_BOUNDS
    ok = (idx >= 0) & (idx < len(src))
    want = np.where(ok, src[np.where(ok, idx, 0)], -5)
    assert np.array_equal(out.cpu().numpy(), want.astype(out.cpu().numpy().dtype))
