"""The peak stage on a cluster of four CTAs per window and on one CTA give the same bits, at the edges of the rule that
chooses between them (a lone batch, two batches) and for every transform length that has a cluster form."""
import numpy as np
import pytest

import xcorr_gb300 as xg
from xcorr_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("xs,ys,n", [(64, 64, 152), (64, 64, 153), (64, 64, 200), (64, 64, 202), (64, 128, 202), (64, 128, 306), (32, 64, 30), (128, 128, 9),
                                     (128, 32, 152), (128, 32, 153), (256, 64, 72), (256, 64, 73), (256, 32, 76), (256, 32, 78),
                                     (256, 16, 5)])
def test_cluster_and_single_cta(xs, ys, n):
    nx, ny = 8 * xs + 170, 8 * ys + 260
    m, s = synth.make_pair(synth.PairSpec(nx=nx, ny=ny, dx=1.7, dy=-2.6, noise_frac=0.1, seed=n + xs))
    side = int(np.ceil(np.sqrt(n)))
    locs = xg.grid(nx, ny, side, side, xs, ys)[:n]
    locs[-1] = 3, ny - 2                              # partly outside both images
    with xg.Context(xg.params(xs, ys)) as ctx:
        for batches in (1, 2):
            ctx.set_batches(batches)
            got = []
            for cfg in (0, 1, 2):
                ctx.set_launch_shapes(0, cfg)
                got.append(ctx.correlate(m, s, locs, strip_len=side))
            for name in xg.RESULT_DTYPE.names:
                for g in got[1:]:
                    assert np.array_equal(got[0][name], g[name], equal_nan=g[name].dtype.kind == "f"), (batches, name)
