"""-time / -time4 cross sums, exactly: -real images whose samples are small multiples of a power of two make every
amplitude, patch mean and (int) demeaned value known exactly, so the correlation surface's maximum, its position and
its first value must equal the int64 (time4: modulo 2^64) sums formed by numpy, whatever the integers' size: digits of
a few bits, full int16 range, and integers too large for the tensor cores' digits (the integer kernel)."""
import numpy as np
import pytest

import xcorr_gb300 as xg

pytestmark = pytest.mark.gpu


def _surface(a, b, nxc, nyc, mode):
    """int64 cross sums and energies of every lag, and sum b*b, as the reference forms them."""
    if mode == 1:
        a, b = a * a, b * b
    ny, nx = b.shape
    win = np.lib.stride_tricks.sliding_window_view
    num = np.zeros((nyc, nxc), np.int64)
    for x in range(nx):                    # wraps modulo 2^64 as int64 does
        col = win(a[:, x: x + nxc], ny, axis=0)[:nyc]          # (nyc, nxc, ny)
        num += col @ b[:, x]
    sq = a * a
    cs = np.zeros((sq.shape[0] + 1, sq.shape[1] + 1), np.int64)
    cs[1:, 1:] = np.cumsum(np.cumsum(sq, axis=0), axis=1)
    en = cs[ny: ny + nyc, nx: nx + nxc] - cs[:nyc, nx: nx + nxc] - cs[ny: ny + nyc, :nxc] + cs[:nyc, :nxc]
    return num, en, np.sum(b * b)


def _values(num, en, d2, mode):
    with np.errstate(invalid="ignore", divide="ignore"):
        dd = 1.0 * en.astype(np.float64) * np.float64(d2)
        den = np.sqrt(dd)
        g = np.where(den == 0, 0.0, np.abs(num.astype(np.float64) / den))
        if mode == 0:
            return 100.0 * g
        return np.where(g <= 0.5, 0.0, 100.0 * np.sqrt(g * 2.0 - 1.0))


@pytest.mark.parametrize("mode", [0, 1])
@pytest.mark.parametrize("xs,ys,top,unit", [(32, 32, 3, 1), (32, 32, 15000, 1), (64, 32, 700, 1), (32, 64, 9000, 1),
                                            (64, 64, 15000, 1), (128, 32, 4000, 1), (32, 128, 15000, 1),
                                            (32, 32, 4000, 4096), (64, 32, 4000, 4096)])
def test_cross_sums_are_exact(xs, ys, top, unit, mode):
    npx, npy, nx, ny = 4 * xs, 4 * ys, 2 * xs, 2 * ys
    r = np.random.default_rng(xs + 7 * ys + top + mode)
    W, H = npx + 37, npy + 21
    # a few strong samples over weak ones, the slave a noisy shifted copy
    m = np.rint(np.minimum(r.rayleigh(top / 5, (H, W)), top))
    s = np.rint(np.minimum(np.abs(np.roll(m, (3, -5), (0, 1)) + r.normal(0, top / 10, (H, W))), top))
    m, s = (m * unit).astype(np.float32), (s * unit).astype(np.float32)
    locs = np.array([[npx // 2 + 1, npy // 2 + 2], [npx // 2 + 30, npy // 2 + 17]], np.int32)
    with xg.Context(xg.params(xs, ys, ri=1, interp_factor=16, fmt=1, corr_mode=mode)) as ctx:
        res = ctx.correlate(m, s, locs)
    for k, (x, y) in enumerate(locs):
        pa, pb = (im[y - npy // 2: y + npy // 2, x - npx // 2: x + npx // 2] for im in (m, s))
        ma, mb = np.float64(pa.astype(np.float64).mean()), np.float64(pb.astype(np.float64).mean())
        assert res["mean1"][k] == ma and res["mean2"][k] == mb
        ia = (pa - np.float32(ma)).astype(np.int64)
        ib = (pb - np.float32(mb)).astype(np.int64)[ys: ys + ny, xs: xs + nx]
        v = _values(*_surface(ia, ib, nx, ny, mode), mode)
        top_v = np.nanmax(v)
        f = np.float32(top_v)
        flat = v.ravel()
        pk = np.flatnonzero(flat > np.float64(f))[-1] if np.float64(f) < top_v else np.flatnonzero(flat.astype(np.float32) == f)[0]
        assert (res["ip"][k], res["jp"][k]) == divmod(int(pk), nx)
        assert res["cmax"][k] == top_v and res["corr"][k] == f
        assert res["corr0n"][k] == flat[0] or (np.isnan(flat[0]) and np.isnan(res["corr0n"][k]))
