"""xcg_fit_offsets on 16, 8 and 1 CTAs per axis (what a part of a GPU without room for 16 takes), over the edges of each
split, against the float64 numpy oracle; the tolerance is that of the other fit tests."""
import ctypes

import numpy as np
import pytest

import fit_oracle as fo
import xcorr_gb300 as xg

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("ctas,n", [(1, 0), (1, 5), (1, 257), (1, 8192), (1, 8193), (8, 1), (8, 2049), (8, 40003),
                                    (8, 8 * 8192 + 7), (16, 4097), (0, 1000)])
def test_forms(ctas, n):
    r = np.random.default_rng(n + ctas)
    locs = np.stack([r.integers(100, 9000, n), r.integers(200, 30000, n)], 1).astype(np.int32)
    res = np.zeros(n, xg.RESULT_DTYPE)
    res["xoff"], res["yoff"] = r.integers(-4, 5, n) + np.rint(locs[:, 0] * 2e-4), r.integers(-4, 5, n)
    res["xfrac"], res["yfrac"] = r.integers(-8, 8, n) / 16, r.integers(-8, 8, n) / 16
    res["corr"] = 90.0
    if n > 1000:
        res["xoff"][::97] = 500.0           # outliers the weights take out
        res["yfrac"][::211] = np.nan        # not finite: left out of both axes
    npar = 1 if n == 1 else 3
    dl, dr = torch.from_numpy(locs.reshape(-1)).cuda(), torch.from_numpy(res.view(np.uint8)).cuda()
    out = torch.zeros(ctypes.sizeof(xg.Fit), dtype=torch.uint8, device="cuda")
    keep = torch.zeros(256, dtype=torch.uint8, device="cuda")      # a buffer to point at where there is no record
    xg.fit_offsets((dr if n else keep).data_ptr(), (dl if n else keep).data_ptr(), n, out.data_ptr(), y_offset=3,
                   astretcha=2e-4, npar_range=npar, npar_azimuth=npar, robust_iters=2, ctas=ctas)
    torch.cuda.synchronize()
    f = xg.Fit.from_buffer_copy(out.cpu().numpy().tobytes())
    o = fo.fit(res, locs, y_offset=3, astretcha=2e-4, npar_range=npar, npar_azimuth=npar, robust_iters=2)
    for axis in ("range", "azimuth"):
        g, e = getattr(f, axis), o[axis]
        assert g.npts == e["npts"] and g.ishift == e["ishift"]
        for k in ("shift", "stretch", "a_stretch", "rms", "weight"):
            assert abs(getattr(g, k) - e[k]) <= 1e-9 * max(1.0, abs(e[k])), (axis, k, getattr(g, k), e[k])


def test_other_forms_are_refused():
    buf = torch.zeros(1024, dtype=torch.uint8, device="cuda")
    with pytest.raises(xg.XcgError):
        xg.fit_offsets(buf.data_ptr(), buf.data_ptr(), 1, buf.data_ptr(), ctas=4)
