"""The refiner's training kernels over the edges of their split: groups of four samples in the convolutions, 32 samples
per CTA in the dense layers, one CTA per SM and longer ranges from 609 samples on (152 groups of four), and a context
made for more samples than a call brings: outputs, loss and every parameter block's gradient against the FP64 oracle."""
import numpy as np
import pytest

import refiner_oracle as ro
import xcorr_gb300 as xg
from test_gpu_refiner_sizes import _batch

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,most", [(3, 3), (4, 4), (5, 5), (31, 31), (32, 32), (33, 33), (608, 608), (609, 609), (5, 700), (33, 40)])
def test_gradient_at_the_edges(n, most):
    theta = ro.init(n).astype(np.float32)
    f, t = _batch(n, n + 1)
    ref = xg.Refiner(0, max_batch=most)
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
