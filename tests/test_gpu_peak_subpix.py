"""Peak and subpixel stages over their template sizes: every interpolation factor and transform length against the
FP32 oracle (peaks, values), on windows with and without the range interpolation."""
import numpy as np
import pytest

import xcorr_gb300 as xg
import xcorr_oracle as xo
from xcorr_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ifc", [8, 16, 32, 64])
@pytest.mark.parametrize("xs,ys,ri", [(16, 16, 1), (32, 64, 2), (64, 32, 4), (128, 64, 2), (256, 32, 1)])
def test_peaks_and_fractions(xs, ys, ri, ifc):
    nx, ny = 8 * xs + 301, 8 * ys + 203
    m, s = synth.make_pair(synth.PairSpec(nx=nx, ny=ny, dx=1.4, dy=-2.3, noise_frac=0.05, seed=xs + ifc))
    locs = xg.grid(nx, ny, 3, 3, xs, ys)
    with xg.Context(xg.params(xs, ys, ri=ri, interp_factor=ifc)) as ctx:
        r = ctx.correlate(m, s, locs, strip_len=3)
    o = xo.run(xo.params(xs, ys, ri=ri, ifc=ifc), m, s, locs, precision=xo.F32, strip_len=3)
    for k in ("ip", "jp", "fip", "fjp"):
        assert np.array_equal(r[k], o[k]), k
    for k in ("gamma", "cmax", "cave", "fmax"):
        assert np.max(np.abs(r[k] - o[k]) / np.maximum(np.abs(o[k]), 1e-30)) < 1e-4, k
