"""Performance cases of the xcorr library: what its users run, through its public entry points.

listed() holds the cases, draw(rng) gives more of the same ranges, prepare() what a program has in hand
before the call (images on the device or in pinned host memory, the context), run() one call, work() the
bytes and operations the call cannot do without, exact() the same outputs computed in 64 bits by torch.
"""
import ctypes
import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "gmtsar-gpu_gb300", "python")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import xcorr_gb300 as xg  # noqa: E402
from xcorr_gb300 import refiner_train  # noqa: E402

#: a correlation case before its own values: the reference's defaults on a 2048 x 4096 pair
_CORR = {"kind": "device", "nx": 2048, "ny": 4096, "nxl": 20, "nyl": 50, "xs": 64, "ys": 64, "ri": 2, "ifc": 16,
         "fmt": 0, "mode": 2, "dx": 3.37, "dy": -5.81, "noise": 0.1, "xoff": 0, "yoff": 0, "stretch": 0.0}


def _corr(name, **kw):
    return {"name": name, **_CORR, **kw}


def listed():
    return [
        # one strip of locations, what the drop-in program hands over when a band of lines has arrived
        _corr("strip_128", nyl=1),
        # a quick look at a small image: 10 x 10 small windows from host memory
        _corr("host_64", kind="host", nx=1024, ny=1536, nxl=10, nyl=10, xs=32, ys=32),
        # the headline grid: 1000 windows of 128 x 128, images resident
        _corr("grid_128"),
        # the same through host buffers
        _corr("host_128", kind="host"),
        # a full frame: 40,000 windows of 256 x 256
        _corr("frame_256", nx=10240, ny=30720, nxl=100, nyl=400, xs=128, ys=128, dx=2.1, dy=-4.7, noise=0.01),
        # -real images, unequal search, finer range and subpixel interpolation, PRM shifts and stretch, odd sizes
        _corr("real_128x64", nx=2999, ny=2501, nxl=17, nyl=23, xs=64, ys=32, ri=4, ifc=32, fmt=1, dx=9.6, dy=-21.3,
              xoff=8, yoff=-22, stretch=3.1e-4),
        # a stack of eight pairs, windows of 32 to 256, one captured graph
        {"name": "stack_mixed", "kind": "stack", "pairs": 8, "nx": 2560, "ny": 4096, "nxl": 25, "nyl": 40, "ri": 2,
         "ifc": 16, "noise": 0.05},
        # -time: full search in the time domain on the headline grid
        _corr("time_128", mode=0),
        # -time4 on small windows
        _corr("time4_64", nx=1500, ny=2100, nxl=20, nyl=20, xs=32, ys=32, mode=1),
        # the surrogate form: no range interpolation, the learned subpixel refiner
        _corr("refined_128", kind="refined", ri=1),
        # one training batch of the refiner: outputs, loss, parameter gradient
        {"name": "gradient_4096", "kind": "gradient", "n": 4096},
        # the offset model fitted to a full frame's results, with reweighted passes
        {"name": "fit_40000", "kind": "fit", "n": 40000, "robust": 3, "npar": 3},
    ]


def _spread(rng, lo, hi):
    """A whole number between lo and hi, spread over its logarithm."""
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["device", "device", "device", "host", "host", "time", "time", "refined", "stack", "gradient", "fit"])
    if kind == "gradient":
        return {"kind": "gradient", "n": _spread(rng, 60, 4096)}
    if kind == "fit":
        return {"kind": "fit", "n": _spread(rng, 400, 40000), "robust": rng.randint(0, 4), "npar": rng.randint(1, 3)}
    if kind == "stack":
        return {"kind": "stack", "pairs": rng.randint(2, 8), "nx": _spread(rng, 2100, 3000), "ny": _spread(rng, 2500, 4500),
                "nxl": rng.randint(8, 25), "nyl": rng.randint(10, 40), "ri": rng.choice([1, 2, 2]),
                "ifc": rng.choice([8, 16, 16]), "noise": 0.05}
    c = dict(_CORR)
    if kind == "time":
        c["mode"], c["xs"], c["ys"] = rng.choice([0, 0, 1]), rng.choice([32, 64]), rng.choice([32, 64])
        most = 700
    elif kind == "refined":
        c["kind"], c["ri"] = "refined", rng.choice([1, 2])
        most = 2000
    else:
        c["kind"] = kind
        c["xs"] = rng.choice([16, 32, 64, 64, 128])
        c["ys"] = c["xs"] if rng.random() < 0.7 else rng.choice([32, 64, 128])
        c["ri"], c["ifc"], c["fmt"] = rng.choice([1, 2, 2, 2, 4]), rng.choice([8, 16, 16, 32]), rng.choice([0, 0, 0, 1])
        most = 2500
    n = _spread(rng, 12, most)
    c["nxl"] = max(1, min(n, _spread(rng, 4, 40)))
    c["nyl"] = max(1, n // c["nxl"])
    c["nx"] = 8 * c["xs"] + 3 + _spread(rng, 600, 3000)
    c["ny"] = 8 * c["ys"] + 5 + _spread(rng, 600, 5000)
    c["dx"], c["dy"] = round(rng.uniform(-7, 7), 2), round(rng.uniform(-7, 7), 2)
    c["noise"] = round(rng.uniform(0.003, 0.2), 3)
    if rng.random() < 0.4:
        c["xoff"], c["yoff"], c["stretch"] = rng.randint(-9, 9), rng.randint(-9, 9), round(rng.uniform(-4e-4, 4e-4), 6)
        c["dx"], c["dy"] = c["dx"] + c["xoff"], c["dy"] + c["yoff"]
    return c


# ------------------------------------------------------------------ inputs

def _grid(nx, ny, nxl, nyl, xs, ys):
    """The program's location grid: nxl x nyl window centres."""
    xi, yi = (nx - 6 * xs) // (nxl + 3), (ny - 6 * ys) // (nyl + 1)
    return np.array([(4 * xs + i * xi, 4 * ys + j * yi) for j in range(1, nyl + 1) for i in range(2, nxl + 2)], np.int32)


def _speckle_pair(nx, ny, dx, dy, noise, fmt, seed):
    """Complex speckle (sigma 1000) and its copy delayed by (dx, dy) pixels with noise, as the files hold them."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    m = torch.randn((ny, nx, 2), generator=g, device="cuda").mul_(1000.0).round_().clamp_(-32768, 32767)
    f = torch.fft.fft2(torch.view_as_complex(m))
    f *= torch.exp(-2j * math.pi * dy * torch.fft.fftfreq(ny, device="cuda", dtype=torch.float64)).to(torch.complex64)[:, None]
    f *= torch.exp(-2j * math.pi * dx * torch.fft.fftfreq(nx, device="cuda", dtype=torch.float64)).to(torch.complex64)[None, :]
    s = torch.view_as_real(torch.fft.ifft2(f))
    del f
    s = (s + torch.randn((ny, nx, 2), generator=g, device="cuda").mul_(1000.0 * math.sqrt(noise))).round_().clamp_(-32768, 32767)
    if fmt == 1:
        return torch.hypot(m[..., 0], m[..., 1]), torch.hypot(s[..., 0], s[..., 1])
    return m.to(torch.int16), s.to(torch.int16)


def _pair_of_case(c, seed):
    return _speckle_pair(c["nx"], c["ny"], c["dx"], c["dy"], c["noise"], c["fmt"], seed)


def _stack_pairs(c, seed):
    """Each pair of a stack: its search size, shift and images; windows of 32, 64, 128 and 256 in turn."""
    r = np.random.default_rng(seed)
    for k in range(c["pairs"]):
        xs = (64, 16, 128, 32)[k % 4]
        dx, dy = (float(v) for v in r.uniform(-8, 8, 2))
        yield xs, _speckle_pair(c["nx"], c["ny"], dx, dy, c["noise"], 0, seed * 64 + k + 1)


def _refiner_params(seed):
    """He-normal weights, log-variance bias -4, in the library's parameter order."""
    r, parts = np.random.default_rng(seed), []
    for shape, gain in (((32, 9), 1), ((32,), 0), ((32, 288), 1), ((32,), 0), ((32, 288), 1), ((32,), 0), ((64, 288), 1),
                        ((64,), 0), ((3, 64), 0.1), ((3,), 0)):
        parts.append((r.standard_normal(shape) * math.sqrt(2.0 / shape[-1]) * gain).astype(np.float32).ravel())
    parts[-1][2] = -4.0
    return np.concatenate(parts)


def _refiner_batch(n, seed):
    """9 x 9 neighbourhoods of correlation peaks at subpixel positions, with noise, and those positions."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    p = torch.rand((n, 2), generator=g, device="cuda") - 0.5
    k = torch.arange(-4, 5, device="cuda", dtype=torch.float32)
    wide = 0.8 + 0.6 * torch.rand((n, 1), generator=g, device="cuda")
    ex, ey = torch.exp(-((k - p[:, :1]) / wide) ** 2), torch.exp(-((k - p[:, 1:]) / wide) ** 2)
    f = ey[:, :, None] * ex[:, None, :]
    f = f + 0.1 * torch.rand((n, 9, 9), generator=g, device="cuda")
    return (f / f[:, 4:5, 4:5]).reshape(n, 81).contiguous(), p.contiguous()


def _fit_inputs(n, seed):
    """Result records and locations as a correlation leaves them: an affine offset field, noise, poor windows."""
    r = np.random.default_rng(seed)
    side = max(1, int(math.sqrt(n / 4)))
    locs = np.stack([300 + 96 * (np.arange(n) % side), 512 + 74 * (np.arange(n) // side)], 1).astype(np.int32)
    ox = 2.1 + 1e-5 * locs[:, 0] - 3e-6 * locs[:, 1] + 0.06 * r.standard_normal(n)
    oy = -4.7 + 2e-6 * locs[:, 0] + 8e-6 * locs[:, 1] + 0.15 * r.standard_normal(n)
    poor = r.random(n) < 0.03
    ox, oy = np.where(poor, r.uniform(-60, 60, n), ox), np.where(poor, r.uniform(-60, 60, n), oy)
    res = np.zeros(n, xg.RESULT_DTYPE)
    res["xoff"], res["yoff"] = np.rint(2 * ox), np.rint(oy)
    res["xfrac"], res["yfrac"] = np.rint((res["xoff"] - 2 * ox) * 16) / 16, np.rint((res["yoff"] - oy) * 16) / 16
    res["corr"] = np.where(poor, r.uniform(2, 40, n), r.uniform(30, 95, n))
    return res, locs


# ------------------------------------------------------------------ prepare and run

def prepare(case, seed):
    c, kind = case, case["kind"]
    stream = torch.cuda.current_stream().cuda_stream
    if kind == "gradient":
        net = xg.Refiner(max_batch=c["n"])
        net.set_params(_refiner_params(seed))
        feat, target = _refiner_batch(c["n"], seed)
        return {"case": c, "net": net, "feat": feat, "target": target, "stream": stream}
    if kind == "fit":
        res, locs = _fit_inputs(c["n"], seed)
        return {"case": c, "res": torch.from_numpy(res.view(np.uint8).reshape(len(res), -1)).cuda(),
                "locs": torch.from_numpy(locs).cuda(), "stream": stream,
                "fit": torch.zeros(ctypes.sizeof(xg.Fit), dtype=torch.uint8, device="cuda")}
    if kind == "stack":
        st = {"case": c, "stack": xg.Stack(xg.params(ri=c["ri"], interp_factor=c["ifc"])), "pairs": [], "keep": [], "res": [],
              "stream": torch.cuda.Stream()}
        st["stack"].set_graph(True)
        for xs, (m, s) in _stack_pairs(c, seed):
            locs = _grid(c["nx"], c["ny"], c["nxl"], c["nyl"], xs, xs)
            res = torch.zeros((len(locs), xg.RESULT_DTYPE.itemsize), dtype=torch.uint8, device="cuda")
            p = xg.Pair()
            p.d_master, p.m_nx, p.m_ny = m.data_ptr(), c["nx"], c["ny"]
            p.d_slave, p.s_nx, p.s_ny = s.data_ptr(), c["nx"], c["ny"]
            p.locs, p.nlocs, p.strip_len, p.xsearch, p.ysearch = locs.ctypes.data, len(locs), c["nxl"], xs, xs
            p.d_results = res.data_ptr()
            st["pairs"].append(p)
            st["keep"].append((m, s, locs))
            st["res"].append(res)
        torch.cuda.synchronize()
        return st
    m, s = _pair_of_case(c, seed)
    locs = _grid(c["nx"], c["ny"], c["nxl"], c["nyl"], c["xs"], c["ys"])
    ctx = xg.Context(xg.params(c["xs"], c["ys"], ri=c["ri"], interp_factor=c["ifc"], fmt=c["fmt"], corr_mode=c["mode"]))
    st = {"case": c, "ctx": ctx, "stream": stream}
    if kind == "host":
        st["m"], st["s"] = (t.cpu().pin_memory() for t in (m, s))
        st["master"], st["slave"], st["locs"] = st["m"].numpy(), st["s"].numpy(), locs
        return st
    st["m"], st["s"], st["locs"] = m, s, torch.from_numpy(locs).cuda()
    st["res"] = torch.zeros((len(locs), xg.RESULT_DTYPE.itemsize), dtype=torch.uint8, device="cuda")
    if kind == "refined":
        st["net"] = xg.Refiner(max_batch=64)
        st["net"].set_params(refiner_train.load_weights(refiner_train.weights_path(c["ri"])))
    return st


def _record(buf):
    """The result records (104 bytes each) as their fields: a byte tensor's views, or those of a record array."""
    if isinstance(buf, np.ndarray):
        f, i, d = (buf.view(t).reshape(len(buf), -1) for t in (np.float32, np.int32, np.float64))
    else:
        f, i, d = buf.view(torch.float32), buf.view(torch.int32), buf.view(torch.float64)
    return {"offset": f[:, 0:2], "fraction": f[:, 2:4], "corr": f[:, 4], "peaks": i[:, 5:9], "flags": i[:, 9],
            "fmax": f[:, 10], "diagnostics": d[:, 6:13]}


def run(state):
    st, c = state, state["case"]
    kind = c["kind"]
    if kind == "gradient":
        loss, grad, out = st["net"].gradient(st["feat"].data_ptr(), st["target"].data_ptr(), c["n"], stream=st["stream"])
        return {"loss": loss, "grad": grad, "out": out}
    if kind == "fit":
        xg.fit_offsets(st["res"].data_ptr(), st["locs"].data_ptr(), c["n"], st["fit"].data_ptr(), npar_range=c["npar"],
                       npar_azimuth=c["npar"], robust_iters=c["robust"], stream=st["stream"])
        d, i = st["fit"].view(torch.float64), st["fit"].view(torch.int32)
        return {"range": d[0:6], "azimuth": d[7:13], "whole": [i[12:14], i[26:28]]}
    if kind == "stack":
        st["stack"].run(st["pairs"], stream=st["stream"].cuda_stream)
        return [_record(r) for r in st["res"]]
    how = {"x_offset": c["xoff"], "y_offset": c["yoff"], "astretcha": c["stretch"], "strip_len": c["nxl"]}
    if kind == "host":
        return _record(st["ctx"].correlate(st["master"], st["slave"], st["locs"], **how))
    where = (st["m"].data_ptr(), c["nx"], c["ny"], st["s"].data_ptr(), c["nx"], c["ny"], st["locs"].data_ptr(),
             st["locs"].shape[0], st["res"].data_ptr())
    if kind == "refined":
        st["ctx"].correlate_device_refined(st["net"], *where, stream=st["stream"],
                                           max_sigma=0.15 if c["ri"] == 1 else 0.08,
                                           max_disagree=0.4 if c["ri"] == 1 else 0.25, **how)
    else:
        st["ctx"].correlate_device(*where, stream=st["stream"], **how)
    return _record(st["res"])


# ------------------------------------------------------------------ the work a pass cannot do without

def _corr_work(c, xs, ys):
    npx, npy, nw = 4 * xs, 4 * ys, c["nxl"] * c["nyl"]
    xi, yi = (c["nx"] - 6 * xs) // (c["nxl"] + 3), (c["ny"] - 6 * ys) // (c["nyl"] + 1)
    cols, rows = min(c["nx"], (c["nxl"] - 1) * xi + npx), min(c["ny"], (c["nyl"] - 1) * yi + npy)
    lx, ly = math.log2(npx), math.log2(npy)
    segments = c["nxl"] * min(c["nyl"] * npy, (c["nyl"] - 1) * max(yi, 0) + npy) * 2      # row segments of both images
    fl = segments * 5 * npx * lx * c["ri"]
    if c.get("mode", 2) < 2:
        fl += nw * 2.0 * (4 * xs * ys) ** 2
    else:
        fl += segments * 2.5 * npx * lx + nw * (1.5 * npx * 5 * npy * ly + ys * 5 * npx * lx + 6 * 4 * xs * ys)
    fl += nw * 4 * (8 * 8 * c["ifc"] * 8 + 64 * c["ifc"] ** 2 * 8)
    return {"bytes": 2 * 4 * cols * rows + 112 * nw, "flops": fl}


def work(case):
    c = case
    if c["kind"] == "gradient":
        macs = 49 * 9 * 32 + 25 * 288 * 32 + 9 * 288 * 32 + 288 * 64 + 64 * 3
        return {"bytes": c["n"] * (83 + 3) * 4 + 2 * 4 * 37507, "flops": 6.0 * c["n"] * macs}
    if c["kind"] == "fit":
        return {"bytes": c["n"] * (20 + 8) + 112, "flops": c["n"] * 50.0 * (1 + c["robust"])}
    if c["kind"] == "stack":
        each = [_corr_work(c, xs, xs) for xs in ((64, 16, 128, 32) * 2)[: c["pairs"]]]
        return {k: sum(w[k] for w in each) for k in ("bytes", "flops")}
    return _corr_work(c, c["xs"], c["ys"])


# ------------------------------------------------------------------ the outputs in 64 bits

def _interp(x, n, factor, dim):
    """FFT zero-pad interpolation of n samples along dim: bins below n/2 stay, the others move to the top."""
    f = torch.fft.fft(x, dim=dim)
    lo, hi = f.narrow(dim, 0, n // 2), f.narrow(dim, n // 2, n - n // 2)
    shape = list(f.shape)
    shape[dim] = n * factor - n
    return torch.fft.ifft(torch.cat([lo, torch.zeros(shape, dtype=f.dtype, device=f.device), hi], dim=dim), dim=dim) * factor


def _patches(img, fmt, x0, y0, npx, npy, ri):
    """Amplitudes of the range-interpolated patches that start at (x0, y0), zero outside the image."""
    ny, nx = img.shape[:2]
    xx, yy = x0[:, None] + torch.arange(npx, device="cuda"), y0[:, None] + torch.arange(npy, device="cuda")
    inside = ((yy >= 0) & (yy < ny))[:, :, None] & ((xx >= 0) & (xx < nx))[:, None, :]
    at = (yy.clamp(0, ny - 1)[:, :, None], xx.clamp(0, nx - 1)[:, None, :])
    z = img[at].double()
    z = (z.to(torch.complex128) if fmt == 1 else torch.view_as_complex(z)) * inside
    if ri > 1:
        z = _interp(z, npx, ri, 2)[:, :, npx // 2: npx // 2 + npx]
    return z.abs(), ~inside.all(dim=2).all(dim=1)


def _exact_windows(img, locs, c, xs, ys, first):
    """The records of windows `locs` in 64 bits; first: the next window's first surface value per window (a call-back)."""
    npx, npy, nxc, nyc = 4 * xs, 4 * ys, 2 * xs, 2 * ys
    x, y = locs[:, 0].long(), locs[:, 1].long()
    shift = (y.double() * c.get("stretch", 0.0)).trunc().long()
    a, o1 = _patches(img[0], c.get("fmt", 0), x - npx // 2, y - npy // 2, npx, npy, c["ri"])
    b, o2 = _patches(img[1], c.get("fmt", 0), x + c.get("xoff", 0) - npx // 2, y + c.get("yoff", 0) + shift - npy // 2, npx, npy, c["ri"])
    n = len(x)
    m1, m2 = a.mean(dim=(1, 2)), b.mean(dim=(1, 2))
    a, b = a - m1[:, None, None], b - m2[:, None, None]
    mask = torch.zeros((npy, npx), dtype=torch.float64, device="cuda")
    mask[ys: npy - ys, xs: npx - xs] = 1
    b = b * mask
    ia, ib = a.trunc(), b.trunc()
    mode = c.get("mode", 2)

    def lags(u, v):
        r = torch.fft.irfft2(torch.fft.rfft2(u) * torch.fft.rfft2(v).conj(), s=(npy, npx))
        return torch.roll(r, (ys, xs), (1, 2))[:, :nyc, :nxc]

    if mode == 2:
        surf = lags(a, b).abs()
    else:
        u, v = (ia, ib) if mode == 0 else (ia * ia, ib * ib)
        num, d1, d2 = lags(u, v), lags(u * u, mask.expand_as(u)), (v * v).sum(dim=(1, 2))
        den = torch.sqrt(d1 * d2[:, None, None])
        surf = torch.where(den == 0, torch.zeros_like(den), (num / den).abs())
        surf = 100 * surf if mode == 0 else torch.where(surf <= 0.5, torch.zeros_like(surf), 100 * torch.sqrt((2 * surf - 1).clamp_min(0)))
    flat = surf.reshape(n, -1)
    cmax, pk = flat.max(dim=1)
    ip, jp = pk // nxc, pk % nxc
    di, dj = ip - ys, jp - xs
    zero = torch.zeros_like(cmax)
    if mode == 2:
        e = torch.arange(nxc * nyc, device="cuda")
        half = (e & 512) == 0 if nxc * nyc > 1024 else e < 512
        cave, ctrue = (flat * half).mean(dim=1), flat.mean(dim=1)
        ry, rx = ys + di[:, None] + torch.arange(nyc, device="cuda"), xs + dj[:, None] + torch.arange(nxc, device="cuda")
        w = torch.arange(n, device="cuda")[:, None, None]
        p, q = ia[w, ry[:, :, None], rx[:, None, :]], ib[:, ys: npy - ys, xs: npx - xs]
        gamma = 100 * (p * q).sum(dim=(1, 2)).abs() / torch.sqrt((p * p).sum(dim=(1, 2)) * (q * q).sum(dim=(1, 2)))
        flat = flat / (cmax / gamma)[:, None]
    else:
        cave, ctrue, gamma = zero, zero, cmax
    md_at = (nyc // 2 - 4 + di)[:, None, None] + torch.arange(8, device="cuda")[None, :, None]
    md_at = md_at * nxc + (nxc // 2 - 4 + dj)[:, None, None] + torch.arange(8, device="cuda")[None, None, :]
    ns = nxc * nyc
    md = torch.gather(flat, 1, md_at.clamp(0, ns - 1).reshape(n, -1)).reshape(n, 8, 8)
    md = torch.where((md_at >= 0) & (md_at < ns), md, torch.where(md_at == ns, first(flat[:, 0])[:, None, None], torch.zeros_like(md)))
    fine = _interp(_interp((md ** 0.25).to(torch.complex128), 8, c["ifc"], 2), 8, c["ifc"], 1).real.reshape(n, -1)
    fmax, fk = fine.max(dim=1)
    side = 8 * c["ifc"]
    frac = torch.stack([(fk % side) - side / 2, torch.div(fk, side, rounding_mode="floor") - side / 2], 1).double() / c["ifc"]
    return {"offset": torch.stack([-dj, -di], 1).double(), "fraction": frac, "corr": gamma, "fmax": fmax,
            "diagnostics": torch.stack([cmax, cave, ctrue, gamma, m1, m2, flat[:, 0]], 1)}


def _exact_corr(img, c, xs, ys):
    locs = torch.from_numpy(_grid(c["nx"], c["ny"], c["nxl"], c["nyl"], xs, ys)).cuda()
    got, step = [], max(1, min(64, (1 << 22) // (16 * xs * ys * c["ri"]))) * c["nxl"]

    def first(v):      # whole strips at a time: the next window of the strip, 0 past its end
        nxt = torch.cat([v[1:], v[:1] * 0])
        nxt[c["nxl"] - 1:: c["nxl"]] = 0
        return nxt

    for k in range(0, len(locs), step):
        got.append(_exact_windows(img, locs[k: k + step], c, xs, ys, first))
    r = {k: torch.cat([g[k] for g in got]) for k in got[0]}
    r["peaks"] = r["flags"] = None
    return r


def exact(case, seed):
    c = case
    if c["kind"] == "gradient":
        feat, target = (t.double() for t in _refiner_batch(c["n"], seed))
        theta = torch.from_numpy(_refiner_params(seed)).cuda().double().requires_grad_(True)
        p, o = [], 0
        for shape in ((32, 1, 3, 3), (32,), (32, 32, 3, 3), (32,), (32, 32, 3, 3), (32,), (64, 288), (64,), (3, 64), (3,)):
            p.append(theta[o: o + math.prod(shape)].reshape(shape))
            o += math.prod(shape)
        x = feat.reshape(-1, 1, 9, 9)
        for k in range(3):
            win = torch.nn.functional.unfold(x, 3)
            side = x.shape[-1] - 2
            x = torch.nn.functional.gelu(p[2 * k].reshape(32, -1) @ win + p[2 * k + 1][:, None]).reshape(-1, 32, side, side)
        z = torch.nn.functional.gelu(x.reshape(-1, 288) @ p[6].T + p[7])
        out = z @ p[8].T + p[9]
        r2 = ((out[:, :2] - target) ** 2).sum(dim=1)
        each = 0.5 * r2 + 0.5 * r2.detach() * torch.exp(-out[:, 2]) + out[:, 2]
        grad, = torch.autograd.grad(each.mean(), theta)
        return {"loss": float(each.mean()), "grad": grad, "out": out.detach()}
    if c["kind"] == "fit":
        return _exact_fit(c, seed)
    if c["kind"] == "stack":
        return [_exact_corr(img, c, xs, xs) for xs, img in _stack_pairs(c, seed)]
    if c["nxl"] * c["nyl"] * c["xs"] * c["ys"] > 2500 * 64 * 64 * 2:      # the full frame: minutes in 64 bits
        return None
    r = _exact_corr(_pair_of_case(c, seed), c, c["xs"], c["ys"])
    if c["kind"] == "refined":     # the network's fractions have no value but its own
        r["fraction"] = r["fmax"] = None
    return r


def _exact_fit(c, seed):
    res, locs = _fit_inputs(c["n"], seed)
    f = np.float32
    o_r = (res["xoff"] / f(2) - res["xfrac"] / f(2)).astype(np.float64)
    o_a = (res["yoff"] - res["yfrac"]).astype(np.float64)
    use = res["corr"] > f(20.0)
    x, y = locs[use, 0].astype(np.float64), locs[use, 1].astype(np.float64)
    cx, cy = 0.5 * (x.min() + x.max()), 0.5 * (y.min() + y.max())
    hx, hy = 0.5 * (x.max() - x.min()) or 1.0, 0.5 * (y.max() - y.min()) or 1.0
    phi = np.stack([np.ones_like(x), (x - cx) / hx, (y - cy) / hy], 1)
    out = {"whole": None}
    for name, o in (("range", o_r[use]), ("azimuth", o_a[use])):
        k, scale, co = c["npar"], 0.0, np.zeros(3)
        for _ in range(c["robust"] + 1):
            w = np.ones_like(o)
            if scale > 0:
                t = (o - phi @ co) / (4.685 * scale)
                w = np.where(np.abs(t) < 1, (1 - t * t) ** 2, 0.0)
            co = np.zeros(3)
            co[:k] = np.linalg.solve((phi[:, :k] * w[:, None]).T @ phi[:, :k], (phi[:, :k] * w[:, None]).T @ o)
            e = o - phi @ co
            scale = math.sqrt(float((w * e * e).sum() / w.sum()))
        st, at = co[1] / hx, co[2] / hy
        shift = co[0] - st * cx - at * cy
        out[name] = np.array([shift, st, at, shift - int(shift), scale, w.sum()])
    return out
