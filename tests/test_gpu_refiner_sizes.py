"""The refiner's training kernels over the edges of their split (groups of eight samples, one partial gradient per
SM): outputs, loss and every parameter block's gradient against the FP64 oracle; the forward pass gives the same
bits for a sample whatever batch it is in."""
import numpy as np
import pytest

import refiner_oracle as ro
import xcorr_gb300 as xg

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _batch(n, seed):
    r = np.random.default_rng(seed)
    yy, xx = np.mgrid[0:9, 0:9]
    t = r.uniform(-0.5, 0.5, (n, 2)).astype(np.float32)
    w = r.uniform(0.8, 2.0, (n, 1, 1))
    f = np.exp(-((xx - 4 - t[:, :1, None]) ** 2 + (yy - 4 - t[:, 1:, None]) ** 2) / (2 * w * w))
    return (f + r.normal(0, 0.05, f.shape)).reshape(n, 81).astype(np.float32), t


@pytest.mark.parametrize("n", [1, 2, 7, 8, 9, 65, 607, 1217])
def test_gradient_sizes(n):
    theta = ro.init(n).astype(np.float32)
    f, t = _batch(n, n + 1)
    ref = xg.Refiner(0, max_batch=n)
    ref.set_params(theta)
    df, dt = torch.from_numpy(f).cuda(), torch.from_numpy(t).cuda()
    loss, g, out = ref.gradient(df.data_ptr(), dt.data_ptr(), n)
    l64, g64, o64 = ro.loss_grad(theta.astype(np.float64), f, t)
    np.testing.assert_allclose(out, o64, rtol=1e-4, atol=1e-5)
    assert abs(loss - l64) <= 1e-5 * max(1.0, abs(l64))
    o = 0
    for name, shape in ro.PARAM_LAYOUT:
        k = int(np.prod(shape))
        blk = np.linalg.norm(g[o:o + k] - g64[o:o + k]) / max(np.linalg.norm(g64[o:o + k]), 1e-30)
        assert blk < 1e-3, (name, blk)
        o += k


def test_forward_bits_do_not_depend_on_the_batch():
    theta = ro.init(5).astype(np.float32)
    f, _ = _batch(1217, 9)
    df = torch.from_numpy(f).cuda()
    got = []
    for most in (1217, 100, 3):              # one pass, passes of 100 and of 3 samples
        ref = xg.Refiner(0, max_batch=most)
        ref.set_params(theta)
        o = torch.zeros((len(f), 3), device="cuda")
        ref.forward(df.data_ptr(), len(f), o.data_ptr(), tensor_cores=False)
        torch.cuda.synchronize()
        got.append(o.cpu().numpy())
        ref.close()
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])
