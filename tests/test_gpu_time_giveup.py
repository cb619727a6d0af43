"""A tensor-core wait of the time modes that runs out (without a poll: nothing on the device times out).  The lag tile
that gives up ends with its matrix instructions, the window's other tiles run on, and the integer kernel forms the
window's sums: 64-bit integers either way, so the records must be the same, the next call's too."""
import pytest

import xcorr_gb300 as xg
from xcorr_gb300 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("xs,ys,mode", [(64, 64, 0), (128, 128, 0), (32, 64, 0), (64, 64, 1), (32, 32, 1), (128, 64, 1)])
def test_a_wait_that_runs_out_leaves_the_window_to_the_integer_kernel(xs, ys, mode):
    nx, ny = 12 * xs, 12 * ys
    m, s = synth.make_pair(synth.PairSpec(nx=nx, ny=ny, dx=1.7, dy=-2.2, noise_frac=0.1, seed=xs + 2 * ys + mode))
    locs = xg.grid(nx, ny, 4, 6, xs, ys)
    with xg.Context(xg.params(xs, ys, corr_mode=mode)) as ctx:
        ctx.set_profiling(True)
        ms = []
        for _ in range(4):
            usual = ctx.correlate(m, s, locs, strip_len=4)
            ms.append(ctx.stats().kernel_ms[1])
        ctx.inject_stage_timeout()
        given_up = ctx.correlate(m, s, locs, strip_len=4)
        if (xs, ys, mode) != (128, 64, 1):                   # (too bright for digits: the integer kernel's either way)
            assert ctx.stats().kernel_ms[1] > 1.2 * min(ms)  # both kernels took every window
        after = ctx.correlate(m, s, locs, strip_len=4)
    assert not (usual["flags"] & xg.FLAG_STAGE_TIMEOUT).any()
    assert given_up.tobytes() == usual.tobytes() and after.tobytes() == usual.tobytes()
