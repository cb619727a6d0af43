"""xcg_fit_offsets over the edges of its split: no point, one, a CTA's first round and one more, several rounds,
and more points than the CTAs keep in shared memory, against the float64 numpy oracle."""
import ctypes

import numpy as np
import pytest

import fit_oracle as fo
import xcorr_gb300 as xg

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("n,npar,robust", [(0, 3, 1), (1, 1, 0), (5, 3, 2), (255, 2, 1), (257, 3, 4), (4096, 3, 1),
                                           (4097, 1, 2), (40003, 3, 3), (16 * 8192 + 4099, 3, 2)])
def test_fit_sizes(n, npar, robust):
    r = np.random.default_rng(n + 7)
    locs = np.stack([r.integers(100, 9000, n), r.integers(200, 30000, n)], 1).astype(np.int32)
    res = np.zeros(n, xg.RESULT_DTYPE)
    res["xoff"], res["yoff"] = r.integers(-4, 5, n) + np.rint(locs[:, 0] * 2e-4), r.integers(-4, 5, n)
    res["xfrac"], res["yfrac"] = r.integers(-8, 8, n) / 16, r.integers(-8, 8, n) / 16
    res["corr"] = r.uniform(10, 95, n) if n > 5 else 90.0
    if n > 1000:
        res["xoff"][::97] = 500.0           # outliers the weights take out
        res["yfrac"][::211] = np.nan        # not finite: left out of both axes
    dl, dr = torch.from_numpy(locs.reshape(-1)).cuda(), torch.from_numpy(res.view(np.uint8)).cuda()
    out = torch.zeros(ctypes.sizeof(xg.Fit), dtype=torch.uint8, device="cuda")
    keep = torch.zeros(256, dtype=torch.uint8, device="cuda")      # a buffer to point at where there is no record
    xg.fit_offsets((dr if n else keep).data_ptr(), (dl if n else keep).data_ptr(), n, out.data_ptr(), y_offset=3,
                   astretcha=2e-4, npar_range=npar, npar_azimuth=npar, robust_iters=robust)
    torch.cuda.synchronize()
    f = xg.Fit.from_buffer_copy(out.cpu().numpy().tobytes())
    o = fo.fit(res, locs, y_offset=3, astretcha=2e-4, npar_range=npar, npar_azimuth=npar, robust_iters=robust)
    for axis in ("range", "azimuth"):
        g, e = getattr(f, axis), o[axis]
        assert g.npts == e["npts"] and (n < 100 or g.npts > 0.8 * n)
        assert g.ishift == e["ishift"]
        for k in ("shift", "stretch", "a_stretch", "rms", "weight"):
            assert abs(getattr(g, k) - e[k]) <= 1e-9 * max(1.0, abs(e[k])), (axis, k, getattr(g, k), e[k])
