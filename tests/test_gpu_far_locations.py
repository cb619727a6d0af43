"""Locations far outside the images, beyond what the row-segment planner's sort keys hold (20 bits of columns, 24 of
rows): each window is wholly outside, its patches are zeros and flagged, and the windows beside it are what they are
without it."""
import numpy as np
import pytest

import xcorr_gb300 as xg
from xcorr_gb300 import synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

FAR = [(600000, 500), (-700000, 500), (500, 9000000), (500, -9000000), (1 << 20, 1 << 24), (-(1 << 30), 1 << 30), (1 << 30, -(1 << 30)),
       (-1, -(1 << 23)), ((1 << 19) + 512, 300), (-(1 << 19) + 100, 700)]


@pytest.mark.parametrize("mode,xs", [(2, 64), (0, 64), (1, 64), (2, 16), (2, 128)])
def test_windows_far_outside(mode, xs):
    nx, ny = 10 * xs + 160, 14 * xs + 210
    m, s = synth.make_pair(synth.PairSpec(nx=nx, ny=ny, dx=0.8, dy=-1.3, noise_frac=0.1, seed=xs + mode))
    near = xg.grid(nx, ny, 16, 17, xs, xs)
    locs = near.copy()
    at = np.arange(7, 7 + 13 * len(FAR), 13)
    locs[at] = FAR
    rest = np.setdiff1d(np.arange(len(locs)), at)
    with xg.Context(xg.params(xs, xs, corr_mode=mode)) as ctx:
        for xo, yo in ((3, -4), (-300000, 5000000)):      # the second: the slave's windows all far outside
            res = ctx.correlate(m, s, locs, xo, yo, 0.0)
            want = ctx.correlate(m, s, near, xo, yo, 0.0)
            ctx.set_row_sharing(False)
            alone = ctx.correlate(m, s, locs, xo, yo, 0.0)
            ctx.set_row_sharing(True)
            for k in ("mean1", "mean2", "flags"):
                assert np.array_equal(res[k], alone[k]) and np.array_equal(res[k][rest], want[k][rest])
            assert (res["mean1"][at] == 0).all() and (res["flags"][at] & xg.FLAG_OOB).all()
            for name in res.dtype.names:
                assert np.array_equal(res[name][rest], want[name][rest], equal_nan=res[name].dtype.kind == "f"), name
                if mode < 2:
                    assert np.array_equal(res[name], alone[name], equal_nan=res[name].dtype.kind == "f"), name


def test_far_location_in_a_stack():
    nx, ny = 700, 900
    m, s = synth.make_pair(synth.PairSpec(nx=nx, ny=ny, dx=0.8, dy=-1.3, noise_frac=0.1, seed=3))
    dm, ds = (torch.from_numpy(a.view(np.int32).reshape(ny, nx)).cuda() for a in (m, s))
    near = xg.grid(nx, ny, 5, 6, 32, 32)
    out = []
    for far in (False, True):
        locs = near.copy()
        if far:
            locs[3::3] = FAR[:len(locs[3::3])]
        res = [torch.zeros((len(locs), xg.RESULT_DTYPE.itemsize), dtype=torch.uint8, device="cuda") for _ in range(2)]
        pairs = []
        for r in res:
            p = xg.Pair()
            p.d_master, p.m_nx, p.m_ny = dm.data_ptr(), nx, ny
            p.d_slave, p.s_nx, p.s_ny = ds.data_ptr(), nx, ny
            p.xsearch = p.ysearch = 32
            p.locs, p.nlocs, p.strip_len, p.d_results = locs.ctypes.data, len(locs), 0, r.data_ptr()
            pairs.append(p)
        st = xg.Stack(xg.params(32, 32))
        st.run(pairs, torch.cuda.current_stream().cuda_stream)
        torch.cuda.synchronize()
        st.close()
        out.append([np.frombuffer(r.cpu().numpy().tobytes(), xg.RESULT_DTYPE) for r in res])
    keep = np.setdiff1d(np.arange(len(near)), np.arange(3, len(near), 3))
    for a, b in zip(*out):
        assert (b["flags"][3::3] & xg.FLAG_OOB).all() and (b["mean1"][3::3] == 0).all()
        for k in ("ip", "jp", "fip", "fjp", "mean1", "mean2", "gamma"):
            assert np.array_equal(a[k][keep], b[k][keep]), k
