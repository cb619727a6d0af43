// Affine fit of a pair's offsets on the device: the step GMTSAR runs after
// xcorr (fitoffset.csh, called out at xcorr.cu:52; the script is not part of
// the reference sources) to turn freq_xcorr.dat into the PRM resampling
// parameters rshift, sub_int_r, stretch_r, a_stretch_r and their azimuth
// counterparts.  It reads the correlation results where they already are (the
// device result array), so a correlate-then-fit pipeline never copies
// offsets to the host.
//
// Model per axis: o(x, y) = c0 + c1*x + c2*y (npar 3), c0 + c1*x (npar 2) or
// c0 (npar 1), over the locations whose correlation exceeds snr_min, with the
// offsets computed exactly as print_results.c:37-38 writes them (float
// arithmetic).  Coordinates are centred and scaled to [-1, 1] for the normal
// equations, which are accumulated in double with a fixed reduction order
// (deterministic).  robust_iters > 0 adds iteratively reweighted passes with
// Tukey's biweight (c = 4.685 times the weighted rms residual of the
// previous pass).
#include <cooperative_groups.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "fit_solve.cuh"
#include "xcorr_gb300.h"

namespace xcg {
void set_last_error(const char *msg);
}

namespace {

namespace cg = cooperative_groups;

constexpr int FIT_THREADS = 256;
constexpr int NS = 10;         // per axis: w, wu, wv, wuu, wuv, wvv, wo, wuo, wvo, woo
// points a CTA keeps in shared memory between passes (u, v, o: 20 bytes
// each); a call's further points are formed again from the records each pass
constexpr int FIT_KEEP = 8192;

struct AxisModel {
    double c[3];           // in normalised coordinates
    double scale;          // robust weight scale (0: unweighted pass)
};

// One axis's offset of location l as print_results.c:37-38 forms it (float
// arithmetic); false: left out (corr too low, or either offset not finite).
__device__ __forceinline__ bool offset_of(const xcg_result *__restrict__ r, int ly, int axis, int ri, int x_offset,
                                          int y_offset, double astretcha, float snr_min, float &o) {
    const int ishft = (int)((double)ly * astretcha);
    const float orng = (r->xoff / (float)ri) - (r->xfrac / (float)ri) + (float)x_offset;
    const float oazi = r->yoff - r->yfrac + (float)y_offset + (float)ishft;
    o = axis ? oazi : orng;
    return (r->corr > snr_min) && isfinite(orng) && isfinite(oazi);
}

// Sums of the warp's NS values, value k ending in lane bitrev5-ordered slots:
// each step a lane keeps half of its values and adds its partner's share of
// them, 12 additions per lane instead of 5 per value (FP64 additions are what
// a pass costs).  v[0] of lane l holds the warp's sum of value slot(l).
__device__ __forceinline__ void warp_split_sum(double *v) {
    const int lane = threadIdx.x & 31;
    auto step = [&](int n, int half, int bit) {       // lanes with the bit keep [half, n), the others [0, half)
        const bool up = (lane & bit) != 0;
#pragma unroll
        for (int k = 0; k < 5; k++) {
            if (k >= half) break;
            const double hi = (half + k < n) ? v[half + k] : 0.0;
            const double mine = up ? hi : v[k], theirs = up ? v[k] : hi;
            v[k] = mine + __shfl_xor_sync(0xffffffffu, theirs, bit);
        }
    };
    step(NS, 5, 16);       // 10 -> 5
    step(5, 3, 8);         // 5 -> 3 (or 2 and a zero)
    step(3, 2, 4);         // 3 -> 2
    step(2, 1, 2);         // 2 -> 1
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 1);
}
// the value whose sum warp_split_sum leaves in v[0] of `lane`, or -1 (a padding slot)
__device__ __forceinline__ int split_slot(int lane) {
    int lo = 0, n = NS;
    const int half[4] = {5, 3, 2, 1}, bit[4] = {16, 8, 4, 2};
#pragma unroll
    for (int s = 0; s < 4; s++) {
        if (lane & bit[s]) { lo += half[s]; n -= half[s]; }
        else n = n < half[s] ? n : half[s];
    }
    return (n >= 1 && (lane & 1) == 0) ? lo : -1;
}

// One cluster of CTAS CTAs per axis (the axes share nothing but the points
// used).  GB300 issues two FP64 operations per SM and cycle, and a pass is
// about 20 of them per point and axis, so the FP64 pipe bounds the fit: one
// CTA for both axes took 3466 us for 40,000 points and four passes; 2 x 16
// SMs, coordinates normalised once and kept in shared memory, multiplications
// by reciprocals instead of divisions and a split reduction take 92 us.  A
// cluster's barriers order the passes, so there is no workspace in device
// memory: calls on several streams stay independent.
template <int CTAS>
__global__ void __launch_bounds__(FIT_THREADS, 1) k_fit(const xcg_result *__restrict__ res, const xcg_loc *__restrict__ locs,
                                                     int n, int ri, int x_offset, int y_offset, double astretcha,
                                                     float snr_min, int npar_r, int npar_a, int robust_iters, int keep,
                                                     xcg_fit *out) {
    extern __shared__ double pts[];                   // [keep] u, [keep] v, then [keep] o as float
    double *pu = pts, *pv = pts + keep;
    float *po = reinterpret_cast<float *>(pts + 2 * keep);
    __shared__ int ext[5];                            // this CTA's min x, max x, min y, max y, points
    __shared__ int wext[FIT_THREADS / 32][5];
    __shared__ double part[2][NS];                    // this CTA's sums, by the parity of the pass
    __shared__ double wpart[FIT_THREADS / 32][NS];
    __shared__ double total[NS];
    __shared__ AxisModel mod;
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank(), axis = (int)blockIdx.x / CTAS;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int stride = CTAS * FIT_THREADS, first = rank * FIT_THREADS + (int)threadIdx.x;

    // pass 0: extent of the used locations; a point left out is kept as NaN
    int e0 = INT32_MAX, e1 = INT32_MIN, e2 = INT32_MAX, e3 = INT32_MIN, cnt = 0;
    {
        int j = threadIdx.x;
#pragma unroll 4
        for (int i = first; i < n; i += stride, j += FIT_THREADS) {
            const xcg_loc l = locs[i];
            float o;
            const bool use = offset_of(res + i, l.y, axis, ri, x_offset, y_offset, astretcha, snr_min, o);
            if (use) {
                e0 = min(e0, l.x); e1 = max(e1, l.x);
                e2 = min(e2, l.y); e3 = max(e3, l.y);
                cnt++;
            }
            if (j < keep) po[j] = use ? o : NAN;
        }
    }
    e0 = __reduce_min_sync(0xffffffffu, e0); e1 = __reduce_max_sync(0xffffffffu, e1);
    e2 = __reduce_min_sync(0xffffffffu, e2); e3 = __reduce_max_sync(0xffffffffu, e3);
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (lane == 0) { wext[warp][0] = e0; wext[warp][1] = e1; wext[warp][2] = e2; wext[warp][3] = e3; wext[warp][4] = cnt; }
    if (threadIdx.x == 0) { mod.c[0] = mod.c[1] = mod.c[2] = 0.0; mod.scale = 0.0; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int w = 1; w < FIT_THREADS / 32; w++) {
            e0 = min(e0, wext[w][0]); e1 = max(e1, wext[w][1]);
            e2 = min(e2, wext[w][2]); e3 = max(e3, wext[w][3]);
            cnt += wext[w][4];
        }
        ext[0] = e0; ext[1] = e1; ext[2] = e2; ext[3] = e3; ext[4] = cnt;
    }
    cl.sync();
    e0 = INT32_MAX; e1 = INT32_MIN; e2 = INT32_MAX; e3 = INT32_MIN; cnt = 0;
    for (int r = 0; r < CTAS; r++) {
        const int *q = cl.map_shared_rank(ext, r);
        e0 = min(e0, q[0]); e1 = max(e1, q[1]); e2 = min(e2, q[2]); e3 = max(e3, q[3]); cnt += q[4];
    }
    const int ntot = cnt;
    if (ntot == 0) e0 = e1 = e2 = e3 = 0;
    const double cx = 0.5 * ((double)e0 + (double)e1), hx = (e1 > e0) ? 0.5 * ((double)e1 - (double)e0) : 1.0;
    const double cy = 0.5 * ((double)e2 + (double)e3), hy = (e3 > e2) ? 0.5 * ((double)e3 - (double)e2) : 1.0;
    const double ihx = 1.0 / hx, ihy = 1.0 / hy;
    {
        int j = threadIdx.x;
        for (int i = first; i < n && j < keep; i += stride, j += FIT_THREADS) {
            const xcg_loc l = locs[i];
            pu[j] = ((double)l.x - cx) * ihx;
            pv[j] = ((double)l.y - cy) * ihy;
        }
    }

    const int np = axis == 0 ? npar_r : npar_a;
    for (int pass = 0; pass <= robust_iters; pass++) {
        const double scale = mod.scale;
        const bool weighted = scale > 0.0;
        const double inv = weighted ? 1.0 / (4.685 * scale) : 0.0;
        const double c0 = mod.c[0] * inv, c1 = mod.c[1] * inv, c2 = mod.c[2] * inv;
        double S[NS];
#pragma unroll
        for (int k = 0; k < NS; k++) S[k] = 0.0;
        int used = 0;
        int j = threadIdx.x;
        for (int i = first; i < n; i += stride, j += FIT_THREADS) {
            double u, v;
            float of;
            if (j < keep) {
                of = po[j];
                if (of != of) continue;
                u = pu[j];
                v = pv[j];
            } else {
                const xcg_loc l = locs[i];
                if (!offset_of(res + i, l.y, axis, ri, x_offset, y_offset, astretcha, snr_min, of)) continue;
                u = ((double)l.x - cx) * ihx;
                v = ((double)l.y - cy) * ihy;
            }
            const double o = (double)of;
            if (weighted) {
                // residual over 4.685 scale, and 1 - rr^2: > 0 where |rr| < 1
                const double rr = fma(-c2, v, fma(-c1, u, fma(o, inv, -c0)));
                const double q = fma(-rr, rr, 1.0);
                if (__double2hiint(q) <= 0) continue;          // weight 0
                const double w = q * q;
                const double wu = w * u, wv = w * v, wo = w * o;
                S[0] += w; S[1] += wu; S[2] += wv;
                S[3] = fma(wu, u, S[3]); S[4] = fma(wu, v, S[4]); S[5] = fma(wv, v, S[5]);
                S[6] += wo; S[7] = fma(wu, o, S[7]); S[8] = fma(wv, o, S[8]);
                S[9] = fma(wo, o, S[9]);
            } else {
                used++;
                S[1] += u; S[2] += v;
                S[3] = fma(u, u, S[3]); S[4] = fma(u, v, S[4]); S[5] = fma(v, v, S[5]);
                S[6] += o; S[7] = fma(u, o, S[7]); S[8] = fma(v, o, S[8]);
                S[9] = fma(o, o, S[9]);
            }
        }
        if (!weighted) S[0] = (double)used;
        warp_split_sum(S);
        const int slot = split_slot(lane);
        if (slot >= 0) wpart[warp][slot] = S[0];
        __syncthreads();
        if (threadIdx.x < NS) {
            double s[FIT_THREADS / 32];
#pragma unroll
            for (int w = 0; w < FIT_THREADS / 32; w++) s[w] = wpart[w][threadIdx.x];
            part[pass & 1][threadIdx.x] = ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
        }
        cl.sync();             // the parity keeps a slow CTA's reads apart from the next pass's sums
        if (threadIdx.x < NS) {
            double s[CTAS];
#pragma unroll
            for (int r = 0; r < CTAS; r++) s[r] = cl.map_shared_rank(part[pass & 1], r)[threadIdx.x];
#pragma unroll
            for (int h = CTAS / 2; h > 0; h /= 2)
#pragma unroll
                for (int r = 0; r < h; r++) s[r] += s[r + h];
            total[threadIdx.x] = s[0];
        }
        __syncthreads();
        if (threadIdx.x == 0) {          // every CTA solves the same system
            double c[3];
            const double *s = total;
            xcg::fit_solve_regular(s, np, c);
            // weighted residual sum of squares from the sums:
            // sum w (o - c.phi)^2 = woo + c.(M c - 2 (wo, wuo, wvo))
            const double r0 = fma(c[0], s[0], fma(c[1], s[1], fma(c[2], s[2], -2.0 * s[6])));
            const double r1 = fma(c[0], s[1], fma(c[1], s[3], fma(c[2], s[4], -2.0 * s[7])));
            const double r2 = fma(c[0], s[2], fma(c[1], s[4], fma(c[2], s[5], -2.0 * s[8])));
            const double q = fma(c[0], r0, fma(c[1], r1, fma(c[2], r2, s[9])));
            mod.c[0] = c[0]; mod.c[1] = c[1]; mod.c[2] = c[2];
            // scale 0 (an exact fit) keeps the next pass unweighted
            mod.scale = s[0] > 0.0 ? sqrt(fmax(q, 0.0) / s[0]) : 0.0;
        }
        __syncthreads();
    }
    if (rank == 0 && threadIdx.x == 0) {
        xcg_fit_axis f;
        // back to pixel coordinates: o = c0 + c1 (x - cx)/hx + c2 (y - cy)/hy
        f.stretch = mod.c[1] / hx;
        f.a_stretch = mod.c[2] / hy;
        f.shift = mod.c[0] - f.stretch * cx - f.a_stretch * cy;
        f.ishift = (int32_t)f.shift;            // truncation, as (int) and awk int() do
        f.sub_int = f.shift - (double)f.ishift;
        f.weight = total[0];
        f.rms = mod.scale;
        f.npts = ntot;
        if (axis == 0) out->range = f; else out->azimuth = f;
    }
    cl.sync();                 // no CTA leaves while another may still read its sums
}

constexpr size_t fit_smem(int keep) { return (size_t)keep * (2 * sizeof(double) + sizeof(float)); }

struct FitCall {
    const xcg_result *res;
    const xcg_loc *locs;
    int n, ri, x_offset, y_offset;
    double astretcha;
    float snr_min;
    int npar_range, npar_azimuth, robust_iters;
    xcg_fit *out;
    cudaStream_t stream;
};

// Launches the fit on clusters of CTAS CTAs; with `ask`, only where the device
// has room for such a cluster (ran: whether it was launched).
template <int CTAS>
cudaError_t launch_fit(const FitCall &f, bool ask, bool &ran) {
    ran = false;
    const long long per = (long long)CTAS * FIT_THREADS;           // points a cluster takes at a time
    const int keep = (int)std::min<long long>(FIT_KEEP, (f.n + per - 1) / per * FIT_THREADS);
    // the kernel's attributes, per device (idempotent: every call may set them);
    // up to 46 KB need none
    cudaError_t e = CTAS > 8 ? cudaFuncSetAttribute(k_fit<CTAS>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) : cudaSuccess;
    if (e == cudaSuccess && fit_smem(keep) > 46 * 1024)
        e = cudaFuncSetAttribute(k_fit<CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fit_smem(FIT_KEEP));
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * CTAS);
    cfg.blockDim = dim3(FIT_THREADS);
    cfg.dynamicSmemBytes = fit_smem(keep);
    cfg.stream = f.stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = CTAS;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    if (ask) {
        int clusters = 0;
        if (cudaOccupancyMaxActiveClusters(&clusters, k_fit<CTAS>, &cfg) != cudaSuccess) {
            cudaGetLastError();        // not an error of the call: the next form is tried
            clusters = 0;
        }
        if (clusters < 1) return cudaSuccess;
    }
    ran = true;
    return cudaLaunchKernelEx(&cfg, k_fit<CTAS>, f.res, f.locs, f.n, f.ri, f.x_offset, f.y_offset, f.astretcha, f.snr_min,
                              f.npar_range, f.npar_azimuth, f.robust_iters, keep, f.out);
}

// ctas: CTAs per axis, 16, 8 or 1; 0: the most of them that fit.  A cluster lies
// in one GPC, and a part of a GPU (an instance, a partition) may have none with
// 16 SMs free for it.  The same sums in another order.
xcg_status fit_offsets(const FitCall &f, int ctas) {
    if (!f.res || !f.locs || !f.out || f.n < 0 || f.ri < 1 || f.npar_range < 1 || f.npar_range > 3 || f.npar_azimuth < 1 ||
        f.npar_azimuth > 3 || f.robust_iters < 0 || f.robust_iters > 100) {
        xcg::set_last_error("xcg_fit_offsets: invalid argument");
        return XCG_ERR_ARG;
    }
    const bool any = ctas == 0;
    bool ran = false;
    cudaError_t e = cudaSuccess;
    if (any || ctas == 16) e = launch_fit<16>(f, any, ran);
    if (e == cudaSuccess && !ran && (any || ctas == 8)) e = launch_fit<8>(f, any, ran);
    if (e == cudaSuccess && !ran && (any || ctas == 1)) e = launch_fit<1>(f, false, ran);
    if (e == cudaSuccess) e = cudaGetLastError();
    if (e != cudaSuccess) {
        xcg::set_last_error(cudaGetErrorString(e));
        return XCG_ERR_CUDA;
    }
    return XCG_OK;
}

}  // namespace

extern "C" xcg_status xcg_fit_offsets(const xcg_result *d_results, const xcg_loc *d_locs, int32_t nlocs, int32_t ri,
                                      int32_t x_offset, int32_t y_offset, double astretcha, float snr_min,
                                      int32_t npar_range, int32_t npar_azimuth, int32_t robust_iters, xcg_fit *d_out,
                                      void *stream) {
    return fit_offsets({d_results, d_locs, nlocs, ri, x_offset, y_offset, astretcha, snr_min, npar_range, npar_azimuth,
                        robust_iters, d_out, (cudaStream_t)stream}, 0);
}

extern "C" xcg_status xcg_debug_fit_offsets(int32_t ctas, const xcg_result *d_results, const xcg_loc *d_locs, int32_t nlocs,
                                            int32_t ri, int32_t x_offset, int32_t y_offset, double astretcha, float snr_min,
                                            int32_t npar_range, int32_t npar_azimuth, int32_t robust_iters,
                                            xcg_fit *d_out, void *stream) {
    if (ctas != 1 && ctas != 8 && ctas != 16) {
        xcg::set_last_error("xcg_debug_fit_offsets: 1, 8 or 16 CTAs per axis");
        return XCG_ERR_ARG;
    }
    return fit_offsets({d_results, d_locs, nlocs, ri, x_offset, y_offset, astretcha, snr_min, npar_range, npar_azimuth,
                        robust_iters, d_out, (cudaStream_t)stream}, ctas);
}
