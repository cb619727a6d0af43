"""The time-domain modes on shared row segments against one row stage per window.

Both give the same amplitudes and chunk sums, and everything after them is exact
or a fixed sequence of operations, so the records must be identical."""
import pytest

import xcorr_gb300 as xg
from xcorr_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("xs,ys,mode,ri,fmt", [(64, 64, 0, 2, 0), (32, 128, 1, 1, 0), (128, 32, 0, 4, 1), (64, 128, 1, 8, 0),
                                               (256, 32, 0, 2, 0)])
def test_time_modes_share_row_segments(xs, ys, mode, ri, fmt):
    nx, ny = 10 * xs + 160, 14 * ys + 210
    m, s = synth.make_pair(synth.PairSpec(nx=nx, ny=ny, dx=0.8, dy=-1.3, noise_frac=0.1, seed=xs + ys, real=fmt == 1))
    locs = xg.grid(nx, ny, 16, 17, xs, ys)               # 272 patches of 2^16 pixels or more: enough to share
    locs[-1] = 3, ny - 2                                 # partly outside both images
    with xg.Context(xg.params(xs, ys, corr_mode=mode, ri=ri, fmt=fmt), max_batch=100) as ctx:
        shared = ctx.correlate(m, s, locs, 3, -4, 1e-3, strip_len=16)
        launches = ctx.stats().launches
        ctx.set_row_sharing(False)
        alone = ctx.correlate(m, s, locs, 3, -4, 1e-3, strip_len=16)
        assert launches > ctx.stats().launches           # the planners'
    assert shared.tobytes() == alone.tobytes()
