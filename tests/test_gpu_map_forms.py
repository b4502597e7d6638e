"""GPU parity of the fused element chains' two compiled forms, with and without
the (+) reduction, at the edges of a block's 512 vectors, on aligned, 16-byte
aligned and unaligned arrays, and with many inputs."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 1023, 1025, 2047, 2048, 2049, 4099, 700_001])
@pytest.mark.parametrize("shift", [0, 1, 2])
@pytest.mark.parametrize("nin", [1, 3, 5, 8])
def test_with_and_without_reduction(hc, dev, n, shift, nin):
    rng = np.random.default_rng(n)
    hx = [rng.uniform(-1, 1, size=n) for _ in range(nin)]
    xs = []
    for h in hx:
        t = torch.empty(n + shift, dtype=torch.float64, device=dev)[shift:]
        t.copy_(torch.from_numpy(h))
        xs.append(t)
    body = "v = x0 * (double)(i + 1)" + "".join(" + x%d" % k for k in range(1, nin)) + ";"
    want = hx[0] * np.arange(1, n + 1)
    for h in hx[1:]:
        want = want + h
    outs = [torch.full((n + shift,), 7.0, dtype=torch.float64, device=dev)[shift:] for _ in range(2)]
    hc.map_f64(body, xs, out=outs[0])
    _, s = hc.map_f64(body, xs, out=outs[1], want_sum=True)
    _, alone = hc.map_f64(body, xs, want_sum=True)
    assert np.array_equal(outs[0].cpu().numpy(), want) and torch.equal(outs[0], outs[1])
    assert abs(float(s) - want.sum()) <= 1e-12 * np.abs(want).sum()
    if shift == 0:  # the same path with and without an output: the same bits
        assert float(s) == float(alone)
