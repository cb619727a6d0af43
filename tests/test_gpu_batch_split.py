"""Which jobs run as two batches, at the edges of the rule, and that a split gives the same records as one batch,
called, captured and through the host entry.  A strip is never cut by these rules."""
import numpy as np
import pytest

import xcorr_gb300 as xg
from xcorr_gb300 import synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("xs,mode,nxl,nyl,strip,batches", [
    (64, 2, 5, 19, 5, 1), (64, 2, 8, 12, 8, 2),              # 95, 96 windows
    (32, 2, 1, 127, 1, 1), (32, 2, 16, 8, 16, 2),            # below, at 2^21 pixels of patches
    (32, 2, 24, 16, 24, 2), (32, 2, 11, 35, 11, 1),          # 384, 385 windows
    (64, 2, 120, 1, 120, 1), (64, 2, 60, 2, 60, 2), (64, 2, 10, 11, 0, 2),      # one strip, two, no strips
    (64, 0, 21, 19, 21, 1), (64, 0, 20, 20, 20, 2), (32, 1, 20, 20, 20, 2),     # time modes: 399, 400 windows
    (64, 1, 20, 20, 20, 1), (64, 0, 8, 64, 512, 1)])                            # large -time4 windows, one strip
def test_split_of_a_job(xs, mode, nxl, nyl, strip, batches):
    n, nx, ny = nxl * nyl, 8 * xs + 3 * nxl + 70, 8 * xs + 3 * nyl + 90
    m, s = synth.make_pair(synth.PairSpec(nx=nx, ny=ny, dx=1.2, dy=-0.7, noise_frac=0.1, seed=n))
    y, x = np.meshgrid(np.arange(nyl), np.arange(nxl), indexing="ij")
    locs = np.ascontiguousarray(np.stack([4 * xs + 2 + 3 * x, 4 * xs + 5 + 3 * y], -1).reshape(n, 2), np.int32)
    dm, ds = (torch.from_numpy(a.view(np.int32).reshape(ny, nx)).cuda() for a in (m, s))
    dl = torch.from_numpy(locs).cuda()
    res = torch.zeros((n, xg.RESULT_DTYPE.itemsize), dtype=torch.uint8, device="cuda")
    with xg.Context(xg.params(xs, xs, corr_mode=mode)) as ctx:
        def call():
            ctx.correlate_device(dm.data_ptr(), nx, ny, ds.data_ptr(), nx, ny, dl.data_ptr(), n, res.data_ptr(),
                                 stream=torch.cuda.current_stream().cuda_stream, strip_len=strip)

        def fresh(run):
            res.zero_()
            run()
            torch.cuda.synchronize()
            return res.cpu().numpy().tobytes()

        split = fresh(call)
        assert ctx.stats().batches == batches
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            call()
        assert fresh(g.replay) == split
        assert ctx.correlate(m, s, locs, strip_len=strip).tobytes() == split
        ctx.set_batches(1)
        assert fresh(call) == split
