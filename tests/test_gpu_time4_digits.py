"""-time4 windows with so much energy that three digits leave less than eight rows per drain: four digits of eight
rows where the digits' largest values allow it, else the integer kernel.  The
surfaces must equal the sums modulo 2^64 formed by numpy on every side of both lines."""
import numpy as np
import pytest

import xcorr_gb300 as xg
from test_gpu_time_exact import _surface, _values

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("xs,ys,top", [(64, 64, 2500), (64, 64, 6000), (64, 64, 16000), (64, 32, 9000), (64, 32, 22000),
                                       (128, 32, 5000), (128, 32, 21000), (32, 64, 22000)])
def test_bright_windows(xs, ys, top):
    npx, npy, nx, ny = 4 * xs, 4 * ys, 2 * xs, 2 * ys
    r = np.random.default_rng(xs + 3 * ys + top)
    W, H = npx + 9, npy + 6
    m = np.rint(r.uniform(0, top, (H, W)))
    s = np.rint(np.clip(np.roll(m, (2, -3), (0, 1)) + r.normal(0, top / 20, (H, W)), 0, top))
    m, s = m.astype(np.float32), s.astype(np.float32)
    locs = np.array([[npx // 2 + 1, npy // 2 + 2]], np.int32)
    with xg.Context(xg.params(xs, ys, ri=1, interp_factor=16, fmt=1, corr_mode=1)) as ctx:
        res = ctx.correlate(m, s, locs)
    x, y = locs[0]
    pa, pb = (im[y - npy // 2: y + npy // 2, x - npx // 2: x + npx // 2] for im in (m, s))
    ma, mb = np.float64(pa.astype(np.float64).mean()), np.float64(pb.astype(np.float64).mean())
    assert res["mean1"][0] == ma and res["mean2"][0] == mb
    ia = (pa - np.float32(ma)).astype(np.int64)
    ib = (pb - np.float32(mb)).astype(np.int64)[ys: ys + ny, xs: xs + nx]
    v = _values(*_surface(ia, ib, nx, ny, 1), 1)
    top_v = np.nanmax(v)
    f, flat = np.float32(top_v), v.ravel()
    pk = np.flatnonzero(flat > np.float64(f))[-1] if np.float64(f) < top_v else np.flatnonzero(flat.astype(np.float32) == f)[0]
    assert (res["ip"][0], res["jp"][0]) == divmod(int(pk), nx)
    assert res["cmax"][0] == top_v and res["corr"][0] == f
    assert res["corr0n"][0] == flat[0] or (np.isnan(flat[0]) and np.isnan(res["corr0n"][0]))
