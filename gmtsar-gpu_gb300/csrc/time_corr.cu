// The -time and -time4 modes: a full-search time-domain correlation surface
// in place of the FFT surface (do_time_corr, do_time_int_xcorr.cu:146-189).
// The reference's GPU build leaves these modes without data (its host ints
// are never filled, xcorr.cu:364-368 with :413-414); this restores what the
// CPU code computes: for every lag (ioff, joff) in [-ysearch, ysearch) x
// [-xsearch, xsearch), calc_time_corr (:30-68) or calc_time_corr_hat
// (:103-144) over the ny_corr x nx_corr window of (int) demeaned amplitudes,
// the peak rule of do_time_corr (|corr| above the float-rounded running
// maximum, scan order ioff then joff), and the same 8x8 neighbourhood and
// subpixel stage as the frequency path.
//
//   k_tprep     per window: the patch means; sum b*b; the sum a*a under every
//               lag from sliding sums; and how the cross sums can be formed
//               exactly on the tensor cores (TimePlan)
//   k_tcorr_tc  per (lag tile, window): the cross sums as f16 matmuls of the
//               integers' digits, FP32 accumulation in tensor memory, every
//               partial sum an integer below 2^24 and so exact
//   k_tcorr     the same sums with 64-bit integer multiply-adds, for the
//               windows whose integers are too large for that (-real images
//               beyond 2^20; squares beyond 2^31) or where a wait of k_tcorr_tc
//               ran out
//   k_tpeak     per window: the scan-order peak, outputs, 8x8 neighbourhood
// All sums are 64-bit (time: exact; time4: modulo 2^64 like the reference's
// long long).
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "tc_umma.cuh"
#include "time_corr.cuh"

namespace xcg {
namespace {

constexpr int TC_THREADS = 256;
constexpr int TI = 32;      // lag rows per tile (ioff) of k_tcorr
constexpr int TJ = 64;      // lag columns per tile (joff)
constexpr int RI = 2, RJ = 4;

// How one window's cross sums are formed: every integer is split into `limbs`
// digits of `shift` bits, the lower ones balanced in [-2^(shift-1),
// 2^(shift-1)), and the digit products of `rows` master rows accumulate in
// tensor memory before they are drained; limbs 0: k_tcorr takes the window.
// k_tcorr_tc only reads these: its CTAs share a window and decide by them which
// barriers they take.  What it reports goes into `failed`: 0, 1 where one of its
// waits ran out (k_tcorr forms the window's sums), 2 where its instructions had
// not ended by the limit of a second wait either (the record says so).
struct TimePlan {
    long long d2;          // sum of b*b (time4: of v*v, modulo 2^64)
    int limbs, failed, shift, rows;      // (k_tcorr reads the first two at once)
};
// A window's amplitudes: the master patch (rows of npx) and the slave's centre
// (row stride a2s), its own or rows of its chunks of shared row segments
struct TimeAmps {
    const float *a1, *a2;
    int a2s;
};
__device__ __forceinline__ TimeAmps time_amps(const Plan &P, int w) {
    if (P.rc) {
        const int2 wc = P.rc_wch[w];
        return {P.rc_amp + (size_t)wc.x * P.rpc * P.npx,
                P.rc_amp + ((size_t)wc.y * P.rpc + P.ysearch) * P.npx + P.xsearch, P.npx};
    }
    return {P.amp1 + (size_t)w * P.npy * P.npx, P.amp2c + (size_t)w * P.ny_corr * P.nx_corr, P.nx_corr};
}

// A window's arrays in the row-spectrum scratch (npx*npy*8 bytes per window,
// P.zrow; with shared row segments the chunks' spectra, both unused in these modes): cross sums and master energies [nyc][nxc], the plan.
__device__ __forceinline__ char *time_base(const Plan &P, int w) {
    return reinterpret_cast<char *>(P.zrow + (size_t)w * P.npy * P.npx);
}
__device__ __forceinline__ long long *time_num(const Plan &P, int w) { return reinterpret_cast<long long *>(time_base(P, w)); }
__device__ __forceinline__ long long *time_energy(const Plan &P, int w) { return time_num(P, w) + (size_t)P.nyc * P.nxc; }
__device__ __forceinline__ TimePlan *time_plan(const Plan &P, int w) {
    return reinterpret_cast<TimePlan *>(time_energy(P, w) + (size_t)P.nyc * P.nxc);
}

template <int MODE>
struct TcTraits;
template <>
struct TcTraits<0> {        // -time: a, b and sums of a*b, a*a
    using E = int32_t;
    using S = long long;
    static constexpr int YB = 32;
    __device__ static E elem(int v) { return v; }
    __device__ static S prod(E a, E b) { return (S)a * (S)b; }
};
template <>
struct TcTraits<1> {        // -time4: u = a^2, v = b^2 and sums of u*v, u*u, wrapping
    using E = unsigned long long;
    using S = unsigned long long;
    static constexpr int YB = 8;
    __device__ static E elem(int v) { return (E)((long long)v * (long long)v); }
    __device__ static S prod(E a, E b) { return a * b; }
};

template <int MODE>
__host__ __device__ constexpr int tc_aw(int nx_corr) { return nx_corr + TJ - 1; }

__host__ __device__ constexpr size_t align16(size_t b) { return (b + 15) & ~(size_t)15; }

// shared layout: A band [YB+TI-1][AW] | B band [YB][nx_corr]
template <int MODE>
__host__ __device__ size_t tc_off_b(int nx_corr) {
    using Tr = TcTraits<MODE>;
    return align16((size_t)(Tr::YB + TI - 1) * tc_aw<MODE>(nx_corr) * sizeof(typename Tr::E));
}
template <int MODE>
size_t tcorr_smem(int nx_corr) {
    using Tr = TcTraits<MODE>;
    return tc_off_b<MODE>(nx_corr) + align16((size_t)Tr::YB * nx_corr * sizeof(typename Tr::E));
}

__device__ __forceinline__ double warp_sum_d(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// (int) of a demeaned amplitude, the expression of d_mean_mask_strip
// (conv_ampl_demean.cu:129-136) as the frequency path's gamma uses it
__device__ __forceinline__ int demeaned_int(float amp, float mean) {
    float v = amp - mean;
    v = v * 1.0f;
    return (int)v;
}

// ------------------------------------------------------------------ k_tprep

// the digits of an integer (time4: of its square), lowest first
template <int MODE>
__device__ __forceinline__ void digits_of(float amp, float mean, int L, int s, short *d) {
    const int v = demeaned_int(amp, mean);
    if (MODE == 0) {
        const int half = 1 << (s - 1), lo = ((v + half) & ((1 << s) - 1)) - half;
        d[0] = (short)lo;
        d[1] = (short)((v - lo) >> s);
    } else if (L < 4) {                        // squares below 2^27
        const int u = v * v, half = 1 << (s - 1), mask = (1 << s) - 1;
        const int lo = ((u + half) & mask) - half, u1 = (u - lo) >> s;
        const int mid = ((u1 + half) & mask) - half;
        d[0] = (short)lo;
        d[1] = (short)(L == 2 ? u1 : mid);
        d[2] = (short)((u1 - mid) >> s);
    } else {
        long long u = (long long)v * v;
        const int half = 1 << (s - 1), mask = (1 << s) - 1;
#pragma unroll
        for (int l = 0; l < 3; l++) {
            const int lo = (((int)u + half) & mask) - half;
            d[l] = (short)lo;
            u = (u - lo) >> s;
        }
        d[3] = (short)u;
    }
}

// Digits for integers up to vmax in magnitude (time4: their squares): the
// fewest that keep the lower digits near the square (cube, fourth) root of the
// largest value; squares are small compared with their largest, so a bit less.
// The top digit must be an integer an f16 holds (2048).  limbs 0: none.
template <int MODE>
__device__ void choose_digits(TimePlan &t, float vmax) {
    t.limbs = t.shift = t.rows = t.failed = 0;
    if (!(vmax >= 0.f) || !(vmax < 1e9f)) return;
    const float top = MODE == 0 ? vmax : vmax * vmax;
    const float lg = log2f(fmaxf(top, 2.f));
    const int L = MODE == 0 ? 2 : (lg < 13.f ? 2 : (lg < 27.f ? 3 : 4));
    int s = MODE == 0 ? (int)(0.5f * lg + 0.5f) : (int)ceilf(lg / (float)L) - 1;
    s = max(s, 3);
    while (s <= 11 && top / exp2f((float)(s * (L - 1))) + 2.f > 2048.f) s++;
    if (s > 11) return;
    t.limbs = L;
    t.shift = s;
}

// Master rows per drain so that every partial sum stays below 2^24: a segment
// of rows accumulates, for a lag, as many slave rows, so by Cauchy-Schwarz no
// sum of digit products exceeds the root of the product of the two operands'
// digit energies over those rows.  ga / gb: energies per group of eight
// rows and digit.
__device__ int rows_per_drain(const float (*ga)[128], const float (*gb)[64], int L, int nr, int tiles_i, int gbn, int lane) {
    constexpr float LIMIT = 16777216.f * 0.95f;
    for (int segs = 1;; segs++) {
        int rows = (nr + segs - 1) / segs;
        rows = (rows + 7) & ~7;
        const int ng = rows / 8;
        // slave: the largest energy of ng + 1 consecutive groups (rows not aligned to groups)
        float eb[4], ea[4];
#pragma unroll
        for (int l = 0; l < 4; l++) {
            eb[l] = ea[l] = 0.f;
            if (l >= L) continue;
            for (int g0 = lane; g0 < gbn; g0 += 32) {
                float e = 0.f;
                for (int g = g0; g < min(g0 + ng + 1, gbn); g++) e += gb[l][g];
                eb[l] = fmaxf(eb[l], e);
            }
            for (int q = lane; q < tiles_i * segs; q += 32) {       // every tile's every segment
                const int t = q / segs, r0 = (q - t * segs) * rows;
                float e = 0.f;
                for (int g = (128 * t + r0) / 8; g < (128 * t + min(r0 + rows, nr) + 7) / 8 && g < 128; g++) e += ga[l][g];
                ea[l] = fmaxf(ea[l], e);
            }
            for (int o = 16; o > 0; o >>= 1) {
                eb[l] = fmaxf(eb[l], __shfl_xor_sync(0xffffffffu, eb[l], o));
                ea[l] = fmaxf(ea[l], __shfl_xor_sync(0xffffffffu, ea[l], o));
            }
            eb[l] = sqrtf(eb[l]);
            ea[l] = sqrtf(ea[l]);
        }
        float worst = 0.f;
#pragma unroll
        for (int w = 0; w < 7; w++) {
            float sum = 0.f;
#pragma unroll
            for (int l = 0; l < 4; l++)
                if (w - l >= 0 && w - l < 4) sum += eb[l] * ea[w - l];
            worst = fmaxf(worst, sum);
        }
        if (worst * 1.002f < LIMIT) return rows;
        if (rows <= 8) return 0;
    }
}

// -time4 windows whose energies leave less than eight rows per drain with three
// digits: four digits and eight rows, if the digits' largest values alone keep
// every partial sum of 8 nx products below 2^24.  (The integer kernel takes 1.5 ms
// for such a window however few there are: 60 windows of 128 x 128 2663 -> 1378 us,
// 600 of them 13.7 -> 8.6 ms.)
__device__ bool four_digits(TimePlan &t, float vmax, int nx) {
    for (int s = 7; s <= 8; s++) {
        const float low = exp2f((float)(s - 1)), top = vmax * vmax * exp2f((float)(-3 * s)) + 2.f;
        const float d[4] = {low, low, low, top};
        float worst = 0.f;
        for (int w = 0; w < 7; w++) {
            float sum = 0.f;
            for (int i = 0; i < 4; i++)
                if (w - i >= 0 && w - i < 4) sum += d[i] * d[w - i];
            worst = fmaxf(worst, sum);
        }
        if (top <= 2048.f && worst * 8.f * (float)nx < 16777216.f * 0.95f) {
            t.limbs = 4;
            t.shift = s;
            t.rows = 8;
            return true;
        }
    }
    return false;
}

// CPT: window columns nxc + nx_corr - 1 (below 256 CPT) per thread
template <int MODE, int CPT>
__global__ void __launch_bounds__(TC_THREADS) k_tprep(Plan P) {
    using Tr = TcTraits<MODE>;
    using S = typename Tr::S;
    constexpr int WP = 256 * CPT, LMAX = MODE == 0 ? 2 : 4;
    extern __shared__ float4 smem_raw[];
    S *D = reinterpret_cast<S *>(smem_raw);            // [8][WP] column sums, then their prefix sums
    __shared__ double mean_sh[2];
    __shared__ float ga[4][128], gb[4][64];            // digit energies per eight rows
    __shared__ TimePlan plan_sh;
    __shared__ float vmax_sh;
    __shared__ unsigned long long red[8];
    const int w = blockIdx.x, tid = threadIdx.x, l32 = tid & 31, warp = tid >> 5;
    const int N = P.npx, nx = P.nx_corr, ny = P.ny_corr, nxc = P.nxc, nyc = P.nyc;
    const int W = nxc + nx - 1;
    for (int i = tid; i < 4 * 128; i += TC_THREADS) (&ga[0][0])[i] = 0.f;
    for (int i = tid; i < 4 * 64; i += TC_THREADS) (&gb[0][0])[i] = 0.f;
    if (warp == 0) {   // patch means, as the frequency path forms them, and the digits for the extremes
        double s1 = 0.0, s2 = 0.0;
        float lo1 = INFINITY, hi1 = -INFINITY, lo2 = INFINITY, hi2 = -INFINITY;
        if (P.rc) {         // the slave's extremes over its mask rows, as k_peak takes them
            const int2 wc = P.rc_wch[w];
            for (int i = l32; i < P.nchunks; i += 32) {
                s1 += (double)P.rc_part[wc.x + i];
                s2 += (double)P.rc_part[wc.y + i];
                const float2 a = P.rc_minmax[wc.x + i];
                lo1 = fminf(lo1, a.x); hi1 = fmaxf(hi1, a.y);
                const int r0 = i * P.rpc;
                if (r0 >= P.ysearch && r0 < P.npy - P.ysearch) {
                    const float2 b = P.rc_minmax[wc.y + i];
                    lo2 = fminf(lo2, b.x); hi2 = fmaxf(hi2, b.y);
                }
            }
        } else {
            const float *pb = P.part + (size_t)w * 2 * P.nchunks, *mm = P.minmax + (size_t)w * 4 * P.nchunks;
            for (int i = l32; i < P.nchunks; i += 32) {
                s1 += (double)pb[i];
                s2 += (double)pb[P.nchunks + i];
                lo1 = fminf(lo1, mm[i]); hi1 = fmaxf(hi1, mm[P.nchunks + i]);
                lo2 = fminf(lo2, mm[2 * P.nchunks + i]); hi2 = fmaxf(hi2, mm[3 * P.nchunks + i]);
            }
        }
        s1 = warp_sum_d(s1);
        s2 = warp_sum_d(s2);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo1 = fminf(lo1, __shfl_xor_sync(0xffffffffu, lo1, o)); hi1 = fmaxf(hi1, __shfl_xor_sync(0xffffffffu, hi1, o));
            lo2 = fminf(lo2, __shfl_xor_sync(0xffffffffu, lo2, o)); hi2 = fmaxf(hi2, __shfl_xor_sync(0xffffffffu, hi2, o));
        }
        if (l32 == 0) {
            const double inv = __longlong_as_double((long long)(1023 - (31 - __clz(N * P.npy))) << 52);   // 1/(N npy), a power of two
            s1 *= inv;
            s2 *= inv;
            mean_sh[0] = s1; mean_sh[1] = s2;
            P.means[2 * w] = s1; P.means[2 * w + 1] = s2;
            const float m1 = (float)s1, m2 = (float)s2;
            vmax_sh = fmaxf(fmaxf(hi1 - m1, m1 - lo1), fmaxf(hi2 - m2, m2 - lo2)) * 1.001f + 1.f;
            choose_digits<MODE>(plan_sh, vmax_sh);
        }
    }
    __syncthreads();
    const float m1f = (float)mean_sh[0], m2f = (float)mean_sh[1];
    const TimeAmps amps = time_amps(P, w);
    const float *amp1 = amps.a1, *amp2 = amps.a2;
    const int L = plan_sh.limbs, sh = plan_sh.shift;
    // adds this thread's digit energies of one group of rows to the group's
    auto publish = [&](float *e, float (*g)[128], float (*g2)[64], int at) {
#pragma unroll
        for (int l = 0; l < LMAX; l++) {
            float x = e[l];
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
            if (l32 == 0 && l < L) atomicAdd(g ? &g[l][at] : &g2[l][at], x);
            e[l] = 0.f;
        }
    };
    auto add_energy = [&](float amp, float mean, float *e) {
        short d[LMAX];
        digits_of<MODE>(amp, mean, L, sh, d);
#pragma unroll
        for (int l = 0; l < LMAX; l++)
            if (l < L) e[l] = fmaf((float)d[l], (float)d[l], e[l]);
    };
    unsigned long long d2 = 0;
    for (int g = warp; g < ny / 8; g += 8) {           // the slave's window: a warp per eight rows
        float e[LMAX] = {};
        for (int q = 0; q < 8; q++) {
            const float *row = amp2 + (size_t)(g * 8 + q) * amps.a2s;
            for (int c = l32; c < nx; c += 32) {
                const typename Tr::E v = Tr::elem(demeaned_int(row[c], m2f));
                d2 += (unsigned long long)Tr::prod(v, v);
                if (L) add_energy(row[c], m2f, e);
            }
        }
        publish(e, nullptr, gb, g);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) d2 += __shfl_xor_sync(0xffffffffu, d2, o);
    if (l32 == 0) red[warp] = d2;
    // master energies: column sums over the window's rows slide down the lag
    // rows, eight at a time; a warp per lag row turns them into prefix sums,
    // and a lag's energy is a difference of two.  Each row's digits are
    // weighed when it is first read.
    long long *en = time_energy(P, w);
    auto sq = [&](float a) -> S {
        const typename Tr::E e = Tr::elem(demeaned_int(a, m1f));
        return Tr::prod(e, e);
    };
    S run[CPT];
#pragma unroll
    for (int k = 0; k < CPT; k++) run[k] = 0;
    for (int y = 0; y < ny; y += 8) {
        float e[LMAX] = {};
#pragma unroll
        for (int k = 0; k < CPT; k++) {
            const int c = tid + 256 * k;
            if (c < W) {
                float a[8];
#pragma unroll
                for (int q = 0; q < 8; q++) a[q] = amp1[(size_t)(y + q) * N + c];
#pragma unroll
                for (int q = 0; q < 8; q++) {
                    run[k] += sq(a[q]);
                    if (L) add_energy(a[q], m1f, e);
                }
            }
        }
        publish(e, ga, nullptr, y / 8);
    }
    for (int ib = 0; ib < nyc; ib += 8) {
        // the rows that enter: ny + ib - 1, the last of one group, then seven of the next
        float e0[LMAX] = {}, e[LMAX] = {};
#pragma unroll
        for (int k = 0; k < CPT; k++) {
            const int c = tid + 256 * k;
            float in[8], out[8];
            if (c < W) {
#pragma unroll
                for (int q = 0; q < 8; q++) {          // lag row ib + q takes row in - 1 + ny and leaves row - 1
                    const int i = ib + q;
                    in[q] = (i > 0) ? amp1[(size_t)(i - 1 + ny) * N + c] : 0.f;
                    out[q] = (i > 0) ? amp1[(size_t)(i - 1) * N + c] : 0.f;
                }
            }
#pragma unroll
            for (int q = 0; q < 8; q++) {
                if (c < W && ib + q > 0) {
                    run[k] += sq(in[q]) - sq(out[q]);
                    if (L) add_energy(in[q], m1f, q == 0 ? e0 : e);
                }
                D[q * WP + c] = run[k];
            }
        }
        if (ib > 0) publish(e0, ga, nullptr, (ib + ny) / 8 - 1);
        publish(e, ga, nullptr, (ib + ny) / 8);
        __syncthreads();
        S *d = D + warp * WP;
        S carry = 0;
        for (int t = l32; t < WP; t += 32) {
            S x = d[t];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const S u = __shfl_up_sync(0xffffffffu, x, o);
                if (l32 >= o) x += u;
            }
            x += carry;
            d[t] = x;
            carry = __shfl_sync(0xffffffffu, x, 31);
        }
        __syncwarp();
        for (int j = l32; j < nxc; j += 32)
            en[(size_t)(ib + warp) * nxc + j] = (long long)(d[j + nx - 1] - (j ? d[j - 1] : (S)0));
        __syncthreads();
    }
    if (warp == 0) {
        int rows = 0;
        if (L) rows = rows_per_drain(ga, gb, L, min(128, nyc) + ny - 1, (nyc + 127) / 128, ny / 8, l32);
        if (l32 == 0) {
            TimePlan t = plan_sh;
            t.rows = rows;
            if (rows == 0 && !(MODE == 1 && L == 3 && four_digits(t, vmax_sh, nx))) t.limbs = 0;
            t.d2 = 0;
            for (int i = 0; i < 8; i++) t.d2 += (long long)red[i];
            *time_plan(P, w) = t;
        }
    }
}

// ------------------------------------------------------------------ k_tcorr_tc

// The cross sums of a tile of lags i in [i0, i0 + 128), j in [j0, j0 + JT) are
// sum over master rows r and window columns x of b[r - i][x] * a[r][x + j]:
// per master row a matmul over x of
//   A (128 x KS): slave rows r - i, kept in shared memory in reverse order
//     between zero rows, so that the next master row's operand is the same
//     array one row (16 bytes of the no-swizzle K-major layout) further;
//   B (KS x JT): the Hankel matrix a[r][x + j], of whose core matrices (8 x 8)
//     only KS/8 + JT/8 - 1 differ.  JT 128: the producers write those, per
//     digit, and both strides of the descriptor are one core matrix.  JT 64: an
//     instruction of 64 columns takes as long as one of 128 (66 and 74 cycles
//     measured), so the digits of a stand side by side, 64 columns each, the
//     core matrices written out in full, and one instruction covers them;
// for every pair of digits (l of b, m of a), accumulated in the JT columns of
// weight l + m in tensor memory.  FP32 holds every partial sum exactly
// (TimePlan); the drains combine the weights in 64 bits.  The tensor pipe
// bounds it (an instruction of 128 x 128 x 16 per 66 cycles); half of its
// products meet the zero rows.  1000 windows of 128 x 128 lags: 2.35 ms (the
// tensor pipe 81% busy; seven waves of 152 windows), 31.5 ms with 64-bit integer
// multiply-adds; 400 windows of 64 x 64 in -time4: 0.38 ms against 2.15 ms.
constexpr int TCT_STAGES = 3;
constexpr int TCT_PROD = 224;                       // producer threads: warps 1 to 7
constexpr uint32_t TCT_POLLS = 1u << 18;
constexpr int TCT_GIVEUP_ROW = 5;                   // Plan::time_giveup: the master row before which a tile gives up

struct TcLayout {
    int rows, hc, rw;                               // A rows, Hankel core matrices, row-buffer halves
    size_t a_limb, stage, rowbuf, bars, bytes;      // sizes and offsets in bytes
};
template <int MODE>
__host__ __device__ TcLayout tc_layout(int ny, int nyc, int ks, int jt) {
    constexpr int LMAX = MODE == 0 ? 2 : 4;
    TcLayout t;
    const int ilags = nyc < 128 ? nyc : 128;
    t.rows = ilags + ny + 126;
    t.hc = ks / 8 + jt / 8 - 1;
    t.rw = jt + ks + 8;
    t.a_limb = (size_t)(ks / 8) * t.rows * 16;
    t.stage = jt == 128 ? (size_t)LMAX * t.hc * 128 : (size_t)LMAX * ks * 128;
    t.rowbuf = LMAX * t.a_limb + TCT_STAGES * t.stage;
    t.bars = t.rowbuf + align16((size_t)2 * LMAX * t.rw * 2);
    t.bytes = t.bars + (2 * TCT_STAGES + 1) * 8 + 32;
    return t;
}

__device__ __forceinline__ uint32_t half_bits(short d) { return (uint32_t)__half_as_ushort(__short2half_rn(d)); }

// The matrix instructions of one master row, issued by one lane of a
// converged warp: L x L digit pairs, KST steps of 16 columns.  alo / blo: the
// low words of the operands' descriptors for digit 0 (start address and K
// stride in 16-byte units); the high words are the same for both.
template <int L, int KST>
__device__ __forceinline__ void issue_row(uint32_t leader, uint32_t tmem, uint32_t jt, uint32_t alo, uint32_t a_digit, uint32_t a_step,
                                          uint32_t blo, uint32_t b_digit, uint32_t hi, uint32_t idesc, uint32_t first) {
#pragma unroll
    for (int l = 0; l < L; l++)
#pragma unroll
        for (int m = 0; m < L; m++) {
            const bool fresh = l == 0 || m == L - 1;       // the row's first product of this weight
#pragma unroll
            for (int k = 0; k < KST; k++) {
                const uint64_t ad = ((uint64_t)hi << 32) | (alo + (uint32_t)l * a_digit + (uint32_t)k * a_step);
                const uint64_t bd = ((uint64_t)hi << 32) | (blo + (uint32_t)m * b_digit + (uint32_t)k * 16u);
                tc::mma_f16_uniform(leader, tmem + (uint32_t)(l + m) * jt, ad, bd, idesc, (fresh && k == 0) ? first : 1u);
            }
        }
}
// JT 64: one instruction per digit of b and step covers all digits of a (64 L
// columns, weights l .. l + L - 1).  In a segment's first row the highest
// weight of digits l > 0 is new while the others accumulate: two instructions.
template <int L, int KST>
__device__ __forceinline__ void issue_row64(uint32_t leader, uint32_t tmem, uint32_t alo, uint32_t a_digit, uint32_t a_step,
                                            uint32_t blo, uint32_t hi, uint32_t first) {
    constexpr uint32_t id_all = tc::idesc_f16_f32(128, 64 * L), id_old = tc::idesc_f16_f32(128, 64 * (L - 1)),
                       id_one = tc::idesc_f16_f32(128, 64);
#pragma unroll
    for (int l = 0; l < L; l++) {
        const uint32_t d = tmem + (uint32_t)l * 64u;
#pragma unroll
        for (int k = 0; k < KST; k++) {
            const uint64_t ad = ((uint64_t)hi << 32) | (alo + (uint32_t)l * a_digit + (uint32_t)k * a_step);
            const uint64_t bd = ((uint64_t)hi << 32) | (blo + (uint32_t)k * (128u * L));
            if (k == 0 && l > 0 && !first) {
                tc::mma_f16_uniform(leader, d, ad, bd, id_old, 1u);
                tc::mma_f16_uniform(leader, d + 64u * (L - 1), ad, bd + 64u * (L - 1), id_one, 0u);
            } else {
                tc::mma_f16_uniform(leader, d, ad, bd, id_all, (k == 0 && l == 0) ? first : 1u);
            }
        }
    }
}
template <int L>
__device__ __forceinline__ void issue_row64_k(int kst, uint32_t leader, uint32_t tmem, uint32_t alo, uint32_t a_digit,
                                              uint32_t a_step, uint32_t blo, uint32_t hi, uint32_t first) {
    if (kst == 4) issue_row64<L, 4>(leader, tmem, alo, a_digit, a_step, blo, hi, first);
    else if (kst == 2) issue_row64<L, 2>(leader, tmem, alo, a_digit, a_step, blo, hi, first);
    else issue_row64<L, 1>(leader, tmem, alo, a_digit, a_step, blo, hi, first);
}

template <int MODE, int JT>
__global__ void __launch_bounds__(256, 1) k_tcorr_tc(Plan P, int KS) {
    constexpr int LMAX = MODE == 0 ? 2 : 4;
    extern __shared__ __align__(128) uint8_t tsm[];
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int w = blockIdx.y;
    TimePlan *plan = time_plan(P, w);
    // (the shuffles tell the compiler that these are the same for the warp)
    const int L = __shfl_sync(0xffffffffu, plan->limbs, 0), sh = __shfl_sync(0xffffffffu, plan->shift, 0);
    const int seg_rows = __shfl_sync(0xffffffffu, plan->rows, 0);
    if (L == 0) return;                                       // k_tcorr's window (the same for every warp: nothing here writes limbs)
    // a test's give-up before this row's wait, with matrix instructions issued already
    const int giveup = (P.time_giveup && blockIdx.x == 0) ? TCT_GIVEUP_ROW : -1;
    const int nx = P.nx_corr, ny = P.ny_corr, nxc = P.nxc, N = P.npx;
    const int tiles_j = nxc / JT;
    const int i0 = ((int)blockIdx.x / tiles_j) * 128, j0 = ((int)blockIdx.x % tiles_j) * JT;
    const int ilags = min(128, P.nyc), rmax = ilags + ny - 2, nr = rmax + 1;
    const TcLayout lay = tc_layout<MODE>(ny, P.nyc, KS, JT);
    const int R = lay.rows, HC = lay.hc, RW = lay.rw;
    uint8_t *stages = tsm + LMAX * lay.a_limb;
    uint32_t *rowbuf = reinterpret_cast<uint32_t *>(tsm + lay.rowbuf);     // [2][LMAX][RW / 2] pairs of halves
    uint64_t *full = reinterpret_cast<uint64_t *>(tsm + lay.bars);
    uint64_t *empty = full + TCT_STAGES, *done = empty + TCT_STAGES;
    uint32_t *tmem_sh = reinterpret_cast<uint32_t *>(done + 1);
    volatile int *abort_sh = reinterpret_cast<volatile int *>(tmem_sh + 1);
    volatile int *go = abort_sh + 1;                                       // [2] by the parity of the row step
    const float m1f = (float)P.means[2 * w], m2f = (float)P.means[2 * w + 1];
    const TimeAmps amps = time_amps(P, w);
    const float *amp1 = amps.a1 + (size_t)i0 * N + j0;
    long long *num = time_num(P, w) + (size_t)i0 * nxc + j0;
    uint32_t tcols = 32;
    while (tcols < (uint32_t)((2 * L - 1) * JT)) tcols <<= 1;

    if (warp == 0) {
        tc::tmem_alloc(tmem_sh, tcols);
        tc::tmem_relinquish();
    }
    if (tid == 32) {
        for (int i = 0; i < TCT_STAGES; i++) { tc::mbar_init(&full[i], TCT_PROD / 32); tc::mbar_init(&empty[i], 1); }
        tc::mbar_init(done, 1);
        *abort_sh = 0;
        tc::mbar_fence_init();
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = __shfl_sync(0xffffffffu, *tmem_sh, 0);
    constexpr uint32_t idesc = tc::idesc_f16_f32(128, JT);

    int step = 0, seg = 0;                                    // row steps and drains so far
    bool fail = false;
    float v0 = 0.f, v1 = 0.f;                                 // producers: the next row's values
    // sums of the drains so far: in registers (-time4, which drains every few
    // rows and has one CTA per SM anyway), else in num
    constexpr bool KEEP = MODE == 1;
    unsigned long long kept[KEEP ? 32 : 1];
#pragma unroll
    for (int e = 0; e < (KEEP ? 32 : 1); e++) kept[e] = 0;
    for (int x0 = 0; x0 < nx && !fail; x0 += KS) {
        // A: row q of the array is slave row ny - 1 - p, p = q - (ilags - 1)
        for (int it = tid; it < R * (KS / 8); it += 256) {
            const int kb = it / R, q = it - kb * R, p = q - (ilags - 1);
            uint32_t pk[LMAX][4];
#pragma unroll
            for (int l = 0; l < LMAX; l++)
#pragma unroll
                for (int e = 0; e < 4; e++) pk[l][e] = 0u;
            if (p >= 0 && p < ny) {
                const float4 *src = reinterpret_cast<const float4 *>(amps.a2 + (size_t)(ny - 1 - p) * amps.a2s + x0 + 8 * kb);
                const float4 u = __ldg(src), v = __ldg(src + 1);
                const float f[8] = {u.x, u.y, u.z, u.w, v.x, v.y, v.z, v.w};
#pragma unroll
                for (int e = 0; e < 4; e++) {
                    short d0[LMAX], d1[LMAX];
                    digits_of<MODE>(f[2 * e], m2f, L, sh, d0);
                    digits_of<MODE>(f[2 * e + 1], m2f, L, sh, d1);
#pragma unroll
                    for (int l = 0; l < LMAX; l++)
                        if (l < L) pk[l][e] = half_bits(d0[l]) | (half_bits(d1[l]) << 16);
                }
            }
#pragma unroll
            for (int l = 0; l < LMAX; l++)
                if (l < L) *reinterpret_cast<uint4 *>(tsm + l * lay.a_limb + (size_t)it * 16) =
                    make_uint4(pk[l][0], pk[l][1], pk[l][2], pk[l][3]);
        }
        tc::fence_async_smem();
        __syncthreads();
        for (int r0 = 0; r0 < nr && !fail; r0 += seg_rows) {
            const int r1 = min(r0 + seg_rows, nr);
            if (warp == 0) {                                  // MMA issuer: the warp stays together, lane 0 issues
                const uint32_t leader = lane == 0 ? 1u : 0u;
                int st = step % TCT_STAGES;
                uint32_t ph = (uint32_t)(step / TCT_STAGES) & 1u;
                uint32_t alo = ((tc::smem_addr(tsm) >> 4) + (uint32_t)(rmax - r0)) | ((uint32_t)R << 16);
                const uint32_t hi = (uint32_t)(tc::sdesc(0, 0, 128) >> 32);
                const uint32_t ad = (uint32_t)(lay.a_limb >> 4), as = 2u * (uint32_t)R, bd = (uint32_t)HC * 8u;
                const uint32_t sb = (tc::smem_addr(stages) >> 4) | ((JT == 128 ? 8u : 64u * (uint32_t)L) << 16), ss = (uint32_t)(lay.stage >> 4);
                const int rend = (giveup >= r0 && giveup < r1) ? giveup : r1;
                for (int r = r0; r < rend; r++) {
                    if (!__all_sync(0xffffffffu, !*abort_sh && tc::mbar_wait(&full[st], ph, TCT_POLLS))) {
                        *abort_sh = 1;
                        break;
                    }
                    tc::fence_after_sync();
                    const uint32_t blo = sb + (uint32_t)st * ss, first = r == r0 ? 0u : 1u;
                    if constexpr (JT == 128) {                // -time: two digits
                        if (KS == 128) issue_row<2, 8>(leader, tmem, JT, alo, ad, as, blo, bd, hi, idesc, first);
                        else issue_row<2, 4>(leader, tmem, JT, alo, ad, as, blo, bd, hi, idesc, first);
                    } else if (MODE == 0 || L == 2) {
                        issue_row64_k<2>(KS / 16, leader, tmem, alo, ad, as, blo, hi, first);
                    } else if (L == 3) {
                        issue_row64_k<3>(KS / 16, leader, tmem, alo, ad, as, blo, hi, first);
                    } else {
                        issue_row64_k<4>(KS / 16, leader, tmem, alo, ad, as, blo, hi, first);
                    }
                    if (leader) tc::mma_commit(&empty[st]);
                    __syncwarp();
                    alo -= 1u;                                // the next master row: the slave rows one further
                    if (++st == TCT_STAGES) { st = 0; ph ^= 1u; }
                }
                if (rend < r1) *abort_sh = 1;
                if (leader) tc::mma_commit(done);
                __syncwarp();
            } else {                                          // producers of the Hankel core matrices
                const int p = tid - 32, cols = JT + KS - 1;
                const float *row = amp1 + (size_t)r0 * N + x0;
                if (r0 == 0) {                                // a slab's first row; later ones are in flight
                    v0 = p < cols ? row[p] : 0.f;
                    v1 = (p + TCT_PROD < cols) ? row[p + TCT_PROD] : 0.f;
                }
                // this thread's core-matrix rows (16 bytes each), the same in
                // every step: row n of core matrix k is halves 8 k + n .. + 7
                // of the digit's row, from two-half words shifted by 0 or 16
                uint32_t src[3], sft[3];
                int at[3], cnt[3];                            // JT 64: the first place in the stage, places
                const int items = L * HC * 8;
#pragma unroll
                for (int k = 0; k < 3; k++) {
                    const int it = p + k * TCT_PROD, l = it / (HC * 8), o = it - l * (HC * 8);
                    src[k] = (uint32_t)(l * (RW / 2) + (o >> 1));
                    sft[k] = (uint32_t)(o & 1) * 16u;
                    const int c = o >> 3, kb0 = max(0, c - 7), kb1 = min(KS / 8 - 1, c);
                    at[k] = (kb0 * 8 * L + l * 8 + (c - kb0)) * 8 + (o & 7);
                    cnt[k] = kb1 - kb0 + 1;
                }
                int st = step % TCT_STAGES;
                uint32_t ph = (uint32_t)(step / TCT_STAGES) & 1u;             // the stage's phase for this step
                for (int r = r0; r < r1; r++) {
                    const int c = step + r - r0, par = c & 1;
                    if (warp == 1 && lane == 0)
                        go[par] = (c < TCT_STAGES || (!*abort_sh && tc::mbar_wait(&empty[st], ph ^ 1u, TCT_POLLS))) ? 1 : 0;
                    uint32_t *rw = rowbuf + (size_t)par * LMAX * (RW / 2);
                    unsigned short *rb = reinterpret_cast<unsigned short *>(rw) + p;
                    {
                        short d[LMAX];
                        if (p < cols) {
                            digits_of<MODE>(v0, m1f, L, sh, d);
#pragma unroll
                            for (int l = 0; l < LMAX; l++)
                                if (l < L) rb[l * RW] = (unsigned short)half_bits(d[l]);
                        }
                        if (p + TCT_PROD < cols) {
                            digits_of<MODE>(v1, m1f, L, sh, d);
#pragma unroll
                            for (int l = 0; l < LMAX; l++)
                                if (l < L) rb[l * RW + TCT_PROD] = (unsigned short)half_bits(d[l]);
                        }
                    }
                    if (r + 1 < nr) {                         // in flight while this row's matrices are built
                        row += N;
                        v0 = p < cols ? row[p] : 0.f;
                        v1 = (p + TCT_PROD < cols) ? row[p + TCT_PROD] : 0.f;
                    }
                    __syncwarp();
                    asm volatile("bar.sync 1, 224;\n" ::: "memory");
                    if (!go[par]) { *abort_sh = 1; break; }   // one decision for every producer
                    uint4 *dst = reinterpret_cast<uint4 *>(stages + (size_t)st * lay.stage);
#pragma unroll
                    for (int k = 0; k < 3; k++) {
                        if (p + k * TCT_PROD < items) {
                            const uint32_t *q = rw + src[k];
                            const uint32_t q0 = q[0], q1 = q[1], q2 = q[2], q3 = q[3], q4 = q[4];
                            const uint4 v = make_uint4(__funnelshift_r(q0, q1, sft[k]), __funnelshift_r(q1, q2, sft[k]),
                                                       __funnelshift_r(q2, q3, sft[k]), __funnelshift_r(q3, q4, sft[k]));
                            if constexpr (JT == 128) {
                                dst[p + k * TCT_PROD] = v;
                            } else {                          // wherever K core matrix kb and N core matrix c - kb meet
                                uint4 *o = dst + at[k];
#pragma unroll
                                for (int n = 0; n < 8; n++, o += (8 * L - 1) * 8)
                                    if (n < cnt[k]) *o = v;
                            }
                        }
                    }
                    tc::fence_async_smem();
                    __syncwarp();
                    if (lane == 0) tc::mbar_arrive(&full[st]);
                    if (++st == TCT_STAGES) { st = 0; ph ^= 1u; }
                }
            }
            step += r1 - r0;
            // drain: lane i of the accumulator is lag row i0 + i
            const int mine = tc::mbar_wait(done, seg & 1, TCT_POLLS) ? 1 : 0;
            fail = __syncthreads_and(mine && !*abort_sh) == 0;
            tc::fence_after_sync();
            if (!fail) {
                const int i = 32 * (warp & 3) + lane, jh = (warp >> 2) * (JT / 2);
                const uint32_t tl = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)jh;
                // columns jc .. jc + 15 of every weight, the highest first
                auto combine = [&](int jc, unsigned long long *acc) {
#pragma unroll
                    for (int e = 0; e < 16; e++) acc[e] = 0;
#pragma unroll 1
                    for (int wt = 2 * L - 2; wt >= 0; wt--) {
                        float v[16];
                        tc::tmem_ld16(tl + (uint32_t)(wt * JT + jc), v);
#pragma unroll
                        for (int e = 0; e < 16; e++)
                            acc[e] = (acc[e] << sh) + (unsigned long long)(long long)__float2int_rn(v[e]);
                    }
                };
                if constexpr (KEEP) {
#pragma unroll
                    for (int jc = 0; jc < 32; jc += 16) {
                        unsigned long long acc[16];
                        combine(jc, acc);
#pragma unroll
                        for (int e = 0; e < 16; e++) kept[jc + e] += acc[e];
                    }
                } else {
#pragma unroll 1
                    for (int jc = 0; jc < JT / 2; jc += 16) {
                        unsigned long long acc[16];
                        combine(jc, acc);
                        if (i < ilags) {
                            ulonglong2 *dst = reinterpret_cast<ulonglong2 *>(num + (size_t)i * nxc + jh + jc);
#pragma unroll
                            for (int e = 0; e < 8; e++) {
                                ulonglong2 o = make_ulonglong2(acc[2 * e], acc[2 * e + 1]);
                                if (seg > 0) {
                                    const ulonglong2 b = dst[e];
                                    o.x += b.x;
                                    o.y += b.y;
                                }
                                dst[e] = o;
                            }
                        }
                    }
                }
            }
            seg++;
            tc::fence_before_sync();
            __syncthreads();
            tc::fence_after_sync();
        }
    }
    if constexpr (KEEP) {
        const int i = 32 * (warp & 3) + lane, jh = (warp >> 2) * (JT / 2);
        if (!fail && i < ilags) {
            ulonglong2 *dst = reinterpret_cast<ulonglong2 *>(num + (size_t)i * nxc + jh);
#pragma unroll
            for (int e = 0; e < 16; e++) dst[e] = make_ulonglong2(kept[2 * e], kept[2 * e + 1]);
        }
    }
    if (fail) {
        // a wait ran out: k_tcorr forms this window's sums.  The instructions
        // committed to `done` may still read shared memory and write tensor
        // memory, so they end before either is given back
        const int ended = tc::mbar_wait(done, (seg - 1) & 1, 8 * TCT_POLLS) ? 1 : 0;
        const bool all = __syncthreads_and(ended) != 0;
        if (tid == 0) atomicMax(&plan->failed, all ? 1 : 2);
    }
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    if (warp == 0) tc::tmem_dealloc(tmem, tcols);
}

// ------------------------------------------------------------------ k_tcorr

template <int MODE>
__global__ void __launch_bounds__(TC_THREADS) k_tcorr(Plan P) {
    using Tr = TcTraits<MODE>;
    using E = typename Tr::E;
    using S = typename Tr::S;
    constexpr int YB = Tr::YB;
    extern __shared__ float4 smem_raw[];
    const int nx_corr = P.nx_corr, ny_corr = P.ny_corr;
    const int AW = tc_aw<MODE>(nx_corr);
    char *sb = reinterpret_cast<char *>(smem_raw);
    E *As = reinterpret_cast<E *>(sb);                                          // [YB+TI-1][AW]
    E *Bs = reinterpret_cast<E *>(sb + tc_off_b<MODE>(nx_corr));                // [YB][nx_corr]
    const int tiles_j = P.nxc / TJ, tiles = (P.nyc / TI) * tiles_j;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int N = P.npx;
#pragma unroll 1
    for (int item = blockIdx.x; item < P.nwin * tiles; item += gridDim.x) {
        const int w = item / tiles, t0 = item - w * tiles;
        const int2 lf = *reinterpret_cast<const int2 *>(&time_plan(P, w)->limbs);
        if (lf.x != 0 && lf.y == 0) continue;                            // formed on the tensor cores
        const int i0 = (t0 / tiles_j) * TI, j0 = (t0 % tiles_j) * TJ;    // first lag row and column of the tile
        const float m1f = (float)P.means[2 * w], m2f = (float)P.means[2 * w + 1];
        const TimeAmps amps = time_amps(P, w);
        const float *amp1 = amps.a1;
        const int lgx = 31 - __clz(nx_corr);                             // a power of two
        S sab[RI][RJ];
#pragma unroll
        for (int a = 0; a < RI; a++)
#pragma unroll
            for (int b = 0; b < RJ; b++) sab[a][b] = 0;
#pragma unroll 1
        for (int y0 = 0; y0 < ny_corr; y0 += YB) {
            // master rows y0 + i0 + [0, YB+TI-1), columns j0 + [0, AW)
            for (int t = threadIdx.x; t < (YB + TI - 1) * AW; t += TC_THREADS) {
                const int r = t / AW, cc = t - r * AW;
                As[t] = Tr::elem(demeaned_int(amp1[(size_t)(y0 + i0 + r) * N + j0 + cc], m1f));
            }
            for (int t = threadIdx.x; t < YB * nx_corr; t += TC_THREADS)
                Bs[t] = Tr::elem(demeaned_int(amps.a2[(size_t)(y0 + (t >> lgx)) * amps.a2s + (t & (nx_corr - 1))], m2f));
            __syncthreads();
#pragma unroll 1
            for (int yy = 0; yy < YB; yy++) {
                const E *brow = Bs + (size_t)yy * nx_corr;
                const E *arow0 = As + (size_t)(yy + RI * ty) * AW + RJ * tx;
                const E *arow1 = arow0 + AW;
                E wa[RI][RJ];
#pragma unroll
                for (int b = 0; b < RJ - 1; b++) { wa[0][b + 1] = arow0[b]; wa[1][b + 1] = arow1[b]; }
#pragma unroll 4
                for (int x = 0; x < nx_corr; x++) {
#pragma unroll
                    for (int b = 0; b < RJ - 1; b++) { wa[0][b] = wa[0][b + 1]; wa[1][b] = wa[1][b + 1]; }
                    wa[0][RJ - 1] = arow0[x + RJ - 1];
                    wa[1][RJ - 1] = arow1[x + RJ - 1];
                    const E bv = brow[x];
#pragma unroll
                    for (int a = 0; a < RI; a++)
#pragma unroll
                        for (int b = 0; b < RJ; b++) sab[a][b] += Tr::prod(wa[a][b], bv);
                }
            }
            __syncthreads();
        }
        long long *num = time_num(P, w);
#pragma unroll
        for (int a = 0; a < RI; a++)
#pragma unroll
            for (int b = 0; b < RJ; b++)
                num[(size_t)(i0 + RI * ty + a) * P.nxc + j0 + RJ * tx + b] = (long long)sab[a][b];
    }
}

// ------------------------------------------------------------------ k_tpeak

// One lag's correlation (calc_time_corr, calc_time_corr_hat).
template <int MODE>
__device__ __forceinline__ double time_value(long long num, long long d1, long long d2) {
    const double dd = 1.0 * (double)d1 * (double)d2;
    const double den = sqrt(dd);
    double g;
    if (MODE == 0) {
        g = (den == 0.0) ? 0.0 : 100.0 * fabs((double)num / den);
    } else {
        g = (den == 0.0) ? 0.0 : fabs((double)num / den);
        g = (g <= 0.5) ? 0.0 : 100.0 * sqrt((g * 2.0) - 1.0);
    }
    return g;
}

// Scan-order peak of do_time_corr: with v* the largest |corr| and F = (float)v*,
// the running-maximum scan ends on the last element above F when F < v*, else
// on the first element that rounds to F.  Only the lags whose ratio in FP32 is
// within 1e-5 of the largest can be either (the FP32 ratio is good to 5e-7),
// and only those are formed in FP64: GB300 issues two FP64 operations per SM
// and cycle, and a square root and a division for every lag of 1000 windows of
// 128 x 128 would take 1.4 ms.
template <int MODE>
__global__ void __launch_bounds__(TC_THREADS) k_tpeak(Plan P) {
    __shared__ float rf[8];
    __shared__ double rd[8];
    __shared__ int ri_[8];
    __shared__ int flags_sh;
    const int w = blockIdx.x;
    const int nxc = P.nxc, nyc = P.nyc, ns = nxc * nyc;
    const long long *num = time_num(P, w), *en = time_energy(P, w);
    const long long d2 = time_plan(P, w)->d2;
    const float d2f = (float)d2;
    const int l32 = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // |num| / sqrt(d1 d2) in FP32; -1 where the reference's value is not a number
    auto ratio_of = [&](long long n, long long d1) {
        const float e = (float)d1 * d2f;
        const float r = fabsf((float)n) * rsqrtf(e);
        return e == 0.f ? 0.f : (e < 0.f ? -1.f : r);
    };
    auto ratio = [&](int k) { return ratio_of(num[k], en[k]); };
    // the value of lag k, given its ratio; in time4 ratios clearly below 1/2 are 0
    auto value = [&](int k, float r) { return (MODE == 1 && r < 0.49999f) ? 0.0 : time_value<MODE>(num[k], en[k], d2); };

    float mine = -1.f;
    {
        const longlong2 *n2 = reinterpret_cast<const longlong2 *>(num), *e2 = reinterpret_cast<const longlong2 *>(en);
#pragma unroll 4
        for (int k = threadIdx.x; k < ns / 2; k += TC_THREADS) {
            const longlong2 a = n2[k], b = e2[k];
            mine = fmaxf(mine, fmaxf(ratio_of(a.x, b.x), ratio_of(a.y, b.y)));
        }
    }
    float top = mine;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
    if (l32 == 0) rf[warp] = top;
    if (warp == 0) {          // the record's flags: any chunk that read outside an image, reduced by one warp
        int f = 0;
        const int2 wc = P.rc ? P.rc_wch[w] : make_int2(0, 0);
        for (int i = l32; i < P.nchunks; i += 32)
            f |= P.rc ? P.rc_oob[wc.x + i] | P.rc_oob[wc.y + i] : P.oobmap[(size_t)w * P.nchunks + i];
        f = __any_sync(0xffffffffu, f != 0);
        if (l32 == 0) flags_sh = (f ? XCG_FLAG_OOB : 0) | (time_plan(P, w)->failed > 1 ? XCG_FLAG_STAGE_TIMEOUT : 0);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TC_THREADS / 32; i++) top = fmaxf(top, rf[i]);
    // (time4 near 1/2: every lag may be the first of value 0)
    const float thr = (MODE == 1 && top <= 0.50002f) ? 0.f : top * (1.f - 1e-5f);
    double vmax = 0.0;
    if (mine >= thr)                        // this thread's lags, as above
        for (int q = 2 * threadIdx.x; q < ns; q += 2 * TC_THREADS)
            for (int k = q; k < q + 2; k++) {
                const float r = ratio(k);
                if (r >= thr) vmax = fmax(vmax, value(k, r));
            }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) vmax = fmax(vmax, __shfl_xor_sync(0xffffffffu, vmax, o));
    if (l32 == 0) rd[warp] = vmax;
    __syncthreads();
    double vstar = rd[0];
    for (int i = 1; i < TC_THREADS / 32; i++) vstar = fmax(vstar, rd[i]);
    const float F = (float)vstar;
    const bool down = (double)F < vstar;
    int pick = down ? -1 : ns;
    if (mine >= thr)
        for (int q = 2 * threadIdx.x; q < ns; q += 2 * TC_THREADS)
            for (int k = q; k < q + 2; k++) {
                const float r = ratio(k);
                if (!(r >= thr)) continue;
                const double v = value(k, r);
                if (down) { if (v > (double)F) pick = max(pick, k); }
                else if ((float)v == F) pick = min(pick, k);
            }
    pick = down ? __reduce_max_sync(0xffffffffu, pick) : __reduce_min_sync(0xffffffffu, pick);
    if (l32 == 0) ri_[warp] = pick;
    __syncthreads();
    int pk = ri_[0];
    for (int i = 1; i < TC_THREADS / 32; i++) pk = down ? max(pk, ri_[i]) : min(pk, ri_[i]);
    if (pk < 0 || pk >= ns) pk = 0;         // not reached: some element attains v*
    const int ip = pk / nxc, jp = pk % nxc;
    const float jpeak = (float)(jp - P.xsearch), ipeak = (float)(ip - P.ysearch);
    if (threadIdx.x == 0) {
        int local, pidx;
        const PairDev pd = pair_of(P, w, local, pidx);
        xcg_result &o = pd.out[local];
        const double first = time_value<MODE>(num[0], en[0], d2);
        o.xoff = -1 * jpeak;
        o.yoff = -1 * ipeak;
        o.corr = F;
        o.ip = ip; o.jp = jp;
        o.flags = flags_sh;
        o.cmax = vstar;
        o.cave = 0.0;
        o.cave_true = 0.0;
        o.gamma = (double)F;
        o.mean1 = P.means[2 * w];
        o.mean2 = P.means[2 * w + 1];
        o.corr0n = first;
        o.fip = -1; o.fjp = -1; o.fmax = 0.f; o.xfrac = 0.f; o.yfrac = 0.f;
        P.corr0n[w] = first;
    }
    // 8x8 neighbourhood with the reference's flat bounds test (conv_ampl_demean.cu:82-93)
    if (P.interp_flag) {
        const int n2 = P.n2x * P.n2y;
        const int jc = (nxc / 2) - P.n2x / 2 - (int)(-1 * jpeak);
        const int ic = (nyc / 2) - P.n2y / 2 - (int)(-1 * ipeak);
        for (int t = threadIdx.x; t < n2; t += TC_THREADS) {
            const int iy = t / P.n2x, ix = t - iy * P.n2x;
            const long long k = (long long)(ic + iy) * nxc + (jc + ix);
            float v = 0.f;
            unsigned char nx = 0;
            if (k >= 0 && k < ns) v = powf((float)time_value<MODE>(num[k], en[k], d2), 0.25f);
            else if (k == ns) nx = 1;
            P.md[(size_t)w * n2 + t] = v;
            P.mdnext[(size_t)w * n2 + t] = nx;
        }
    }
}

// Tile and slab widths of k_tcorr_tc: 128 lag columns per tile where two
// digits' three weights fit tensor memory (-time), else 64 (-time4: up to
// seven weights); the widest slab whose operands fit shared memory.
constexpr size_t SMEM_MAX = 227 * 1024;
struct TcGeom { int ks, jt; };            // columns of the window per slab, lag columns per tile
template <int MODE>
TcGeom tc_geom(const Plan &P) {
    TcGeom g;
    g.jt = (MODE == 0 && P.nxc >= 128) ? 128 : 64;
    g.ks = std::min(P.nx_corr, g.jt);
    while (g.ks > 16 && tc_layout<MODE>(P.ny_corr, P.nyc, g.ks, g.jt).bytes > SMEM_MAX) g.ks >>= 1;
    return g;
}
int prep_cpt(const Plan &P) { return P.nxc + P.nx_corr - 1 <= 256 ? 1 : (P.nxc + P.nx_corr - 1 <= 512 ? 2 : 4); }
template <int MODE>
cudaError_t time_setup_t(const Plan &P) {
    cudaError_t e = cudaFuncSetAttribute(k_tcorr<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)tcorr_smem<MODE>(512));
    if (!e) e = cudaFuncSetAttribute(k_tprep<MODE, 4>, cudaFuncAttributeMaxDynamicSharedMemorySize, 8 * 1024 * 8);
    if (!e) e = cudaFuncSetAttribute(k_tcorr_tc<MODE, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MAX);
    if (!e && MODE == 0)
        e = cudaFuncSetAttribute(k_tcorr_tc<MODE, MODE == 0 ? 128 : 64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM_MAX);
    return e;
}
template <int MODE>
void launch_tcorr_t(const Plan &P, cudaStream_t s) {
    const TcGeom g = tc_geom<MODE>(P);
    const int cpt = prep_cpt(P);
    const size_t psm = (size_t)8 * 256 * cpt * 8;
    if (cpt == 1) k_tprep<MODE, 1><<<P.nwin, TC_THREADS, psm, s>>>(P);
    else if (cpt == 2) k_tprep<MODE, 2><<<P.nwin, TC_THREADS, psm, s>>>(P);
    else k_tprep<MODE, 4><<<P.nwin, TC_THREADS, psm, s>>>(P);
    const dim3 grid(((P.nyc + 127) / 128) * (P.nxc / g.jt), P.nwin);
    const size_t sm = tc_layout<MODE>(P.ny_corr, P.nyc, g.ks, g.jt).bytes;
    if constexpr (MODE == 0) {
        if (g.jt == 128) k_tcorr_tc<MODE, 128><<<grid, 256, sm, s>>>(P, g.ks);
        else k_tcorr_tc<MODE, 64><<<grid, 256, sm, s>>>(P, g.ks);
    } else {
        k_tcorr_tc<MODE, 64><<<grid, 256, sm, s>>>(P, g.ks);
    }
    const int items = P.nwin * (P.nyc / TI) * (P.nxc / TJ);
    k_tcorr<MODE><<<std::min(items, 152 * 3), TC_THREADS, tcorr_smem<MODE>(P.nx_corr), s>>>(P);
}

}  // namespace

cudaError_t time_setup(const Plan &P) { return P.corr_mode == 0 ? time_setup_t<0>(P) : time_setup_t<1>(P); }

void launch_tcorr(const Plan &P, cudaStream_t s) {
    if (P.corr_mode == 0) launch_tcorr_t<0>(P, s);
    else launch_tcorr_t<1>(P, s);
}

void launch_tpeak(const Plan &P, cudaStream_t s) {
    if (P.corr_mode == 0) k_tpeak<0><<<P.nwin, TC_THREADS, 0, s>>>(P);
    else k_tpeak<1><<<P.nwin, TC_THREADS, 0, s>>>(P);
}

}  // namespace xcg
