"""The time modes' cross sums at the largest windows they take: 512 lag rows (operands of 766 rows, slabs of 16 and 32
columns) and 512 lag columns, as test_gpu_time_exact: every integer is known, so the surface's maximum, its place and its
first value equal the sums modulo 2^64.  The sums come from products of 8-bit digits by FFT (each below 2^34 and
rounded, an error of about 1e-5)."""
import numpy as np
import pytest

import xcorr_gb300 as xg
from test_gpu_time_exact import _values

pytestmark = pytest.mark.gpu


def _cross(a, b, nyc, nxc):
    """sum of b[y, x] a[y + i, x + j] modulo 2^64 for the lags (i, j), a and b of up to 40 bits."""
    shape = [1 << int(np.ceil(np.log2(p + q - 1))) for p, q in zip(a.shape, b.shape)]

    def digits(v):
        out, sign, v = [], np.sign(v), np.abs(v)
        for _ in range(5):
            out.append(np.fft.rfft2(sign * (v & 255), shape))
            v = v >> 8
        assert not v.any()
        return out
    num = np.zeros((nyc, nxc), np.uint64)
    fa, fb = digits(a), digits(b[::-1, ::-1])
    for i, x in enumerate(fa):
        for j, y in enumerate(fb):
            c = np.rint(np.fft.irfft2(x * y, shape)[b.shape[0] - 1:][:nyc, b.shape[1] - 1:][:, :nxc]).astype(np.int64)
            num += c.astype(np.uint64) << np.uint64(8 * (i + j))
    return num.astype(np.int64)


def _window_sums(v, ny, nx, nyc, nxc):
    cs = np.zeros((v.shape[0] + 1, v.shape[1] + 1), np.int64)
    cs[1:, 1:] = np.cumsum(np.cumsum(v, axis=0), axis=1)
    return cs[ny: ny + nyc, nx: nx + nxc] - cs[:nyc, nx: nx + nxc] - cs[ny: ny + nyc, :nxc] + cs[:nyc, :nxc]


@pytest.mark.parametrize("mode,xs,ys,top", [(0, 256, 256, 15000), (0, 32, 256, 9000), (0, 64, 256, 300), (0, 256, 32, 15000),
                                            (1, 256, 256, 60), (1, 256, 256, 700), (1, 32, 256, 60), (1, 32, 256, 900),
                                            (1, 32, 256, 15000), (1, 256, 32, 700), (1, 256, 64, 60)])
def test_largest_windows(mode, xs, ys, top):
    npx, npy, nx, ny = 4 * xs, 4 * ys, 2 * xs, 2 * ys
    r = np.random.default_rng(xs + 5 * ys + top + mode)
    m = np.rint(np.minimum(r.rayleigh(top / 5, (npy + 6, npx + 9)), top))
    s = np.rint(np.minimum(np.abs(np.roll(m, (7, -11), (0, 1)) + r.normal(0, top / 10, m.shape)), top))
    m, s = m.astype(np.float32), s.astype(np.float32)
    x, y = npx // 2 + 3, npy // 2 + 2
    with xg.Context(xg.params(xs, ys, ri=1, interp_factor=16, fmt=1, corr_mode=mode)) as ctx:
        res = ctx.correlate(m, s, np.array([[x, y]], np.int32))
    pa, pb = (im[y - npy // 2: y + npy // 2, x - npx // 2: x + npx // 2] for im in (m, s))
    ma, mb = pa.astype(np.float64).mean(), pb.astype(np.float64).mean()
    assert res["mean1"][0] == ma and res["mean2"][0] == mb
    a = (pa - np.float32(ma)).astype(np.int64)[: ny + ny - 1, : nx + nx - 1]
    b = (pb - np.float32(mb)).astype(np.int64)[ys: ys + ny, xs: xs + nx]
    if mode == 1:
        a, b = a * a, b * b
    v = _values(_cross(a, b, ny, nx), _window_sums(a * a, ny, nx, ny, nx), np.sum(b * b), mode)
    top_v = np.nanmax(v)
    f, flat = np.float32(top_v), v.ravel()
    pk = np.flatnonzero(flat > np.float64(f))[-1] if np.float64(f) < top_v else np.flatnonzero(flat.astype(np.float32) == f)[0]
    assert (res["ip"][0], res["jp"][0]) == divmod(int(pk), nx)
    assert res["cmax"][0] == top_v and res["corr"][0] == f
    assert res["corr0n"][0] == flat[0] or (np.isnan(flat[0]) and np.isnan(res["corr0n"][0]))
