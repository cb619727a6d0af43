"""A call's kernels follow each other as programmatic dependents, plainly inside a captured graph, and on several
streams when it is split into batches: the same bits every way, call after call on the same context."""
import numpy as np
import pytest

import xcorr_gb300 as xg
from xcorr_gb300 import synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("xs,ys,n", [(16, 32, 7), (64, 64, 60), (32, 32, 700), (128, 64, 24)])
def test_every_way_of_running_a_call_gives_the_same_bits(xs, ys, n):
    nx, ny = 8 * xs + 190, 8 * ys + 260
    m, s = synth.make_pair(synth.PairSpec(nx=nx, ny=ny, dx=1.7, dy=-2.6, noise_frac=0.1, seed=n))
    side = int(np.ceil(np.sqrt(n)))
    locs = xg.grid(nx, ny, side, side, xs, ys)[:n]
    dm, ds = (torch.from_numpy(a.view(np.int32).reshape(ny, nx)).cuda() for a in (m, s))
    dl = torch.from_numpy(locs).cuda()
    res = torch.zeros((n, xg.RESULT_DTYPE.itemsize), dtype=torch.uint8, device="cuda")
    with xg.Context(xg.params(xs, ys)) as ctx:
        def call(stream):
            ctx.correlate_device(dm.data_ptr(), nx, ny, ds.data_ptr(), nx, ny, dl.data_ptr(), n, res.data_ptr(),
                                 stream=stream, strip_len=side)

        def fresh(run):
            torch.cuda.synchronize()
            res.zero_()
            torch.cuda.synchronize()
            run()
            torch.cuda.synchronize()
            return res.cpu().numpy().copy()

        want = fresh(lambda: call(0))
        st = torch.cuda.Stream()
        got = {"side stream": fresh(lambda: call(st.cuda_stream)), "twice": fresh(lambda: (call(0), call(0)))}
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g):
            call(torch.cuda.current_stream().cuda_stream)
        got["graph"] = fresh(g.replay)
        for b in (1, 2, 5):
            ctx.set_batches(b)
            got["%d batches" % b] = fresh(lambda: call(st.cuda_stream))
        ctx.set_batches(0)
        got["host entry"] = ctx.correlate(m, s, locs, strip_len=side).view(np.uint8).reshape(n, -1)
        for name, r in got.items():
            a, b = (np.frombuffer(x.tobytes(), xg.RESULT_DTYPE) for x in (r, want))
            for f in xg.RESULT_DTYPE.names:
                assert np.array_equal(a[f], b[f], equal_nan=a[f].dtype.kind == "f"), (name, f)
