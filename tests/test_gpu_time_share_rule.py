"""Which -time and -time4 jobs run on shared row segments (their planners are launches of their own), at both lines of
the rule: patches of 2^15 pixels, and 2^24 pixels of them."""
import numpy as np
import pytest

import xcorr_gb300 as xg
from xcorr_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,xs,ys,n,shares", [(0, 32, 32, 1024, False), (1, 32, 32, 1100, False), (0, 64, 32, 511, False),
                                                 (0, 64, 32, 512, True), (1, 32, 64, 512, True), (0, 64, 64, 255, False), (0, 64, 64, 256, True)])
def test_jobs_that_share(mode, xs, ys, n, shares):
    nx, ny = 8 * xs + 260, 8 * ys + 300
    m, s = synth.make_pair(synth.PairSpec(nx=nx, ny=ny, dx=1.2, dy=-0.7, noise_frac=0.1, seed=n))
    r = np.random.default_rng(n)
    locs = np.stack([r.integers(4 * xs, nx - 4 * xs, n), r.integers(4 * ys, ny - 4 * ys, n)], 1).astype(np.int32)
    with xg.Context(xg.params(xs, ys, corr_mode=mode)) as ctx:
        ctx.set_batches(1)
        got = ctx.correlate(m, s, locs)
        launches = ctx.stats().launches
        ctx.set_row_sharing(False)
        alone = ctx.correlate(m, s, locs)
        assert (launches != ctx.stats().launches) == shares
    assert got.tobytes() == alone.tobytes()
