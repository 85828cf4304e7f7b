"""The tcgen05 training gradient over every count of tiles per CTA: below one
per SM, between one and two CTAs per SM, and past two, where CTAs take a second
tile, against the FP32 kernel's gradient on the same samples.  Both round the
forward pass to bf16 in the same places; the tcgen05 kernel also rounds dY and
dZ (relative 2^-9 each, two layers deep), hence 2e-2 normwise per block."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("count", [64, 128, 192, 148 * 128, 148 * 128 + 64, 296 * 128, 296 * 128 + 64, 600 * 128 + 64])
def test_gradient_tiles(gpu_ok, mpm, count):
    from mlp_ref import OFF
    rng = np.random.default_rng(count)
    n = 5000
    feats = rng.normal(0, 1, (n, 16)).astype(np.float32)
    targs = (np.tanh(feats[:, 9:12]) + 0.1 * rng.normal(0, 1, (n, 3))).astype(np.float32)
    idx = rng.integers(0, n, count)
    with mpm.Corrector(n) as c:
        c.add_data(feats, targs)
        c.init(seed=2)
        c.set_train_kernel("fp32")
        want, wl = c.gradient(idx)
        c.set_train_kernel("tcgen05")
        got, gl = c.gradient(idx)
        again, _ = c.gradient(idx)
    assert abs(gl - wl) <= 1e-4 * wl
    for name in ("W1", "b1", "W2", "b2", "W3", "b3"):
        o, m = OFF[name]
        scale = np.linalg.norm(want[o:o + m])
        assert np.linalg.norm(got[o:o + m] - want[o:o + m]) <= 2e-2 * scale, name
        assert np.linalg.norm(got[o:o + m] - again[o:o + m]) <= 1e-5 * scale, name
