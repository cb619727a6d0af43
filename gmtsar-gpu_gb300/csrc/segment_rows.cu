// Shared row segments: the row stage of the frequency-domain path computed
// once per image row segment rather than once per window that reads it.
//
// Windows of one column of the location grid read the same columns of the
// same image rows: with y_inc = 72 and 256-row patches (the 128 x 128
// configuration) each master and slave row segment belongs to about 3.5
// windows, with 512-row patches and y_inc = 74 (the full frame) to about 7.
// The reference cuts, range-interpolates and transforms every window's
// patch on its own (xcorr.cu:330-338, 237-292); the amplitudes of a row
// segment do not depend on the window, so they are computed once here and
// every window's means, (int) copies and time correlation see the same
// numbers the per-window path computes.  The demean and mask enter in the
// frequency domain by linearity (k_cols_rc), so the row spectra do not depend
// on the window either.
//
//   k_rc_plan   one CTA per batch, or one per image when the chunks need no
//               row-band order: every window contributes a master and a
//               slave entry (pair, image, first column, first row); entries
//               with the same pair, image, first column and first row modulo
//               the rows of a chunk are sorted by row and merged where their
//               row ranges overlap or touch; each merged run gets a range of
//               1024-sample chunks, so a window's patch is a run of
//               consecutive chunk rows
//   k_segrows   one warp per chunk (rows per chunk = 1024 / npx): the patch
//               rows of k_rows (read, range interpolation, amplitude, the
//               reference's FP32 chunk sums, extremes, out-of-image flags),
//               then the half spectra of the chunk's rows, two real rows per
//               complex FFT separated by Hermitian symmetry
//   k_cols_rc   per group of columns kx of one window: the column FFTs of
//               the master's and the masked slave's half spectra, the
//               product with the demean/mask corrections and the inverse
//               column FFT of the surface rows, as k_cols; the default form
//               (k_cols_rcp) is persistent, each CTA taking (window, column
//               group) tiles from a counter, the next tile's rows staged while
//               the current one is transformed
#include <cuda_runtime.h>
#include <algorithm>
#include <math.h>
#include <stdint.h>

#include "kernel_util.cuh"
#include "segment_rows.cuh"
#include "team_fft.cuh"
#include "tile_walk.cuh"

namespace xcg {

// ------------------------------------------------------------------ planner

constexpr int RC_ENTRIES = 2 * RC_MAX_WINDOWS;   // sort capacity, a power of two
// Sort key: pair (15 bits) | image (1) | first column + 2^19 (20) | first row
// modulo the chunk rows (4) | first row + 2^23 (24).  The group of an entry is
// the key without its low 24 bits.
constexpr int KEY_Y_BITS = 24;
constexpr int KEY_Y_BIAS = 1 << 23;
constexpr int KEY_X_BIAS = 1 << 19;
bool rc_fits(const PairDev &p) {
    return std::max(p.m_nx, p.s_nx) < KEY_X_BIAS && std::max(p.m_ny, p.s_ny) < KEY_Y_BIAS;
}

// In-place exclusive scan of a[0, ns) by the whole CTA (ns a multiple of NT,
// at most PER_THREAD of them); returns the total.
template <int NT, int PER_THREAD>
__device__ int block_exclusive_scan(int *a, int *wsum, int ns) {
    const int t = threadIdx.x, l32 = t & 31, wp = t >> 5;
    const int per = ns / NT;
    int v[PER_THREAD];
    int s = 0;
#pragma unroll
    for (int k = 0; k < PER_THREAD; k++) { v[k] = (k < per) ? a[t * per + k] : 0; s += v[k]; }
    int inc = s;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int u = __shfl_up_sync(0xffffffffu, inc, o);
        if (l32 >= o) inc += u;
    }
    if (l32 == 31) wsum[wp] = inc;
    __syncthreads();
    if (wp == 0) {
        int x = (l32 < NT / 32) ? wsum[l32] : 0;
        int xi = x;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, xi, o);
            if (l32 >= o) xi += u;
        }
        wsum[32 + l32] = xi - x;                  // exclusive prefix of the warp totals
        if (l32 == 31) wsum[64] = xi;             // CTA total
    }
    __syncthreads();
    int run = wsum[32 + wp] + inc - s;
#pragma unroll
    for (int k = 0; k < PER_THREAD; k++)
        if (k < per) { a[t * per + k] = run; run += v[k]; }
    const int total = wsum[64];
    __syncthreads();
    return total;
}

__device__ __forceinline__ int key_y(unsigned long long k) {
    return (int)(k & ((1ull << KEY_Y_BITS) - 1)) - KEY_Y_BIAS;
}

// One ascending sort of 32 (key, payload) pairs across a warp.
__device__ __forceinline__ void warp_sort(unsigned long long &k, int &p) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int kk = 2; kk <= 32; kk <<= 1)
#pragma unroll
        for (int j = kk >> 1; j > 0; j >>= 1) {
            const unsigned long long ok = __shfl_xor_sync(0xffffffffu, k, j);
            const int op = __shfl_xor_sync(0xffffffffu, p, j);
            const bool small = ((lane & j) == 0) == ((lane & kk) == 0);     // this lane keeps the smaller key
            if (small ? ok < k : ok > k) { k = ok; p = op; }
        }
}

// Latency bounds the planner (one SM per image), so its sort has few
// barriers: each warp sorts 32 entries by shuffles, then runs are merged by
// rank, an entry's place being its index in its run plus the entries of the
// sibling run before it (a binary search), two barriers a level.  Two batches
// of 500 windows: 32 us of planners with their launches, 41 us with a bitonic
// network and a barrier per step.  CTAs are as small as the entries allow.
// (Chunk descriptors of 8 bytes instead of 16 save 1 us more here and cost the
// row stage 1.6%, unpacking them.)
template <int NT, int PER>
__global__ void __launch_bounds__(NT, 1) k_rc_plan(Plan P) {
    const int tid = threadIdx.x;
    // Two CTAs (no row bands): CTA i plans image i's entries alone, its runs
    // never meeting the other image's, and numbers its chunks from
    // i * nwin * nchunks (the most chunks the master entries can need), so
    // neither waits for the other's total.  One CTA: both images.
    const bool split = (gridDim.x == 2);
    const int nent = split ? P.nwin : 2 * P.nwin;
    const int cbase = (split && blockIdx.x == 1) ? P.nwin * P.nchunks : 0;
    const int npx = P.npx, npy = P.npy, rpc = P.rpc;
    int n = 2;
    while (n < nent || n < 32) n <<= 1;
    const int ns = n > NT ? n : NT;               // the entries the loops and scans cover
    extern __shared__ unsigned long long plan_smem[];
    unsigned long long *key = plan_smem;          // [ns] sort keys
    int *pay = reinterpret_cast<int *>(key + ns); // [ns] entry = 2 w + image
    int *cnt = pay + ns;                          // [ns] run starts before each entry
    int *rlen = cnt + ns;                         // [ns] chunks of each run, then its first chunk
    int *rhead = rlen + ns;                       // [ns] first entry of each run
    int *rtail = rhead + ns;                      // [ns] last entry of each run
    int *wsum = rtail + ns;                       // [72] scan scratch
#pragma unroll
    for (int q = 0; q < PER; q++) {
        const int e = tid + q * NT;
        if (e >= ns) continue;                    // warp-uniform: ns is a multiple of 32
        unsigned long long k = ~0ull;             // padding sorts last
        const int ge = split ? 2 * e + (int)blockIdx.x : e;    // the entry: 2 w + image
        if (e < nent) {
            const int w = ge >> 1, img = ge & 1;
            const xcg_loc loc = P.locs[w];
            int local, pidx;
            const PairDev pd = pair_of(P, w, local, pidx);
            int x0 = img ? loc.x + pd.x_offset - npx / 2 : loc.x - npx / 2;
            int y0 = img ? loc.y + pd.y_offset + slave_row_shift(pd, loc.y) - npy / 2 : loc.y - npy / 2;
            // a patch wholly outside its image is the same wherever it lies: at
            // the image's edge its place fits the key (rc_fits)
            x0 = min(max(x0, -npx), img ? pd.s_nx : pd.m_nx);
            y0 = min(max(y0, -npy), img ? pd.s_ny : pd.m_ny);
            const int ym = ((y0 % rpc) + rpc) % rpc;
            k = ((unsigned long long)pidx << 49) | ((unsigned long long)img << 48) |
                ((unsigned long long)(x0 + KEY_X_BIAS) << 28) | ((unsigned long long)ym << KEY_Y_BITS) |
                (unsigned long long)(y0 + KEY_Y_BIAS);
        }
        int pe = ge;
        warp_sort(k, pe);
        key[e] = k;
        pay[e] = pe;
        rlen[e] = 0;
    }
    __syncthreads();
    for (int len = 32; len < n; len <<= 1) {      // runs of len into runs of 2 len
        unsigned long long k[PER];
        int pe[PER], at[PER];
#pragma unroll
        for (int q = 0; q < PER; q++) at[q] = -1;      // none: beyond the n entries
#pragma unroll
        for (int q = 0; q < PER; q++) {
            const int e = tid + q * NT;
            if (e >= n) continue;
            k[q] = key[e];
            pe[q] = pay[e];
            const int run = e / len;
            const bool left = (run & 1) == 0;     // equal keys: the left run's first
            const unsigned long long *sib = key + (run ^ 1) * len;
            int c = 0;
            for (int h = len >> 1; h > 0; h >>= 1) {
                const unsigned long long o = sib[c + h - 1];
                if (left ? o < k[q] : o <= k[q]) c += h;
            }
            const unsigned long long o = sib[c];
            if (left ? o < k[q] : o <= k[q]) c++;
            at[q] = (run & ~1) * len + (e & (len - 1)) + c;
        }
        __syncthreads();
#pragma unroll
        for (int q = 0; q < PER; q++)
            if (at[q] >= 0) { key[at[q]] = k[q]; pay[at[q]] = pe[q]; }
        __syncthreads();
    }
    // a run starts where the group changes or the next patch leaves a gap of rows
    auto is_head = [&](int i) {
        return i == 0 || (key[i] >> KEY_Y_BITS) != (key[i - 1] >> KEY_Y_BITS) || key_y(key[i]) > key_y(key[i - 1]) + npy;
    };
    for (int i = tid; i < ns; i += NT) cnt[i] = (i < nent && is_head(i)) ? 1 : 0;
    __syncthreads();
    const int nruns = block_exclusive_scan<NT, PER>(cnt, wsum, ns);
    for (int i = tid; i < nent; i += NT) {
        const bool h = is_head(i);
        const int r = cnt[i] + (h ? 0 : -1);
        if (h) rhead[r] = i;
        if (i == nent - 1 || is_head(i + 1)) rtail[r] = i;
    }
    __syncthreads();
    // every patch spans npy rows, so a run ends npy rows below its last entry's first row
    for (int r = tid; r < nruns; r += NT)
        rlen[r] = (key_y(key[rtail[r]]) - key_y(key[rhead[r]]) + npy) / rpc;
    __syncthreads();
    const int total = block_exclusive_scan<NT, PER>(rlen, wsum, ns);   // rlen[r] <- first chunk of run r
    for (int i = tid; i < nent; i += NT) {
        const int r = cnt[i] + (is_head(i) ? 0 : -1);
        const int c0 = rlen[r] + (key_y(key[i]) - key_y(key[rhead[r]])) / rpc;
        reinterpret_cast<int *>(P.rc_wch)[pay[i]] = cbase + c0;   // rc_wch[w].x for the master, .y for the slave
    }
    // chunk descriptors: one warp per run, its lanes writing consecutive chunks
    {
        const int wp = tid >> 5, l32 = tid & 31;
        for (int r = wp; r < nruns; r += NT / 32) {
            const unsigned long long k = key[rhead[r]];
            const int pidx = (int)(k >> 49), img = (int)((k >> 48) & 1);
            const int x0 = (int)((k >> 28) & ((1u << 20) - 1)) - KEY_X_BIAS;
            const int y0 = key_y(k);
            const int c0 = rlen[r], c1 = (r + 1 < nruns) ? rlen[r + 1] : total;
            for (int c = c0 + l32; c < c1; c += 32) P.rc_desc[cbase + c] = make_int4(pidx, img, x0, y0 + (c - c0) * rpc);
        }
    }
    if (tid == 0) {
        // chunks of the master entries' numbering, then of the slave's (from nwin * nchunks)
        if (split) {
            P.rc_count[blockIdx.x] = total;
        } else {
            P.rc_count[0] = total;
            P.rc_count[1] = 0;
        }
        if (P.rc_tile_next && blockIdx.x == 0) *P.rc_tile_next = 0;   // the persistent column stage's tile counter
    }
    if (P.rc_nbands > 0) {
        // the chunks listed band by band (order within a band is free).  A
        // chunk belongs to the first band whose end row lies beyond its last
        // row (the last band takes the rest).  Chunk k of a run covers rows
        // y0 + k rpc .. y0 + k rpc + rpc - 1, increasing with k, so each band's
        // chunks are one range of the run, found from the band ends alone:
        // one warp per run counts them, then writes its ranges at offsets
        // taken from per-band counters
        int *bcnt = wsum;                         // [0, 8) counts, [8, 16) fill, [16, 24) starts
        const int nb = P.rc_nbands;
        const int wp = tid >> 5, l32 = tid & 31;
        __syncthreads();                          // wsum free (the scans are done)
        if (tid < 24) wsum[tid] = 0;
        __syncthreads();
        // chunks of a run (first row y0, len chunks) whose last row is below row e
        auto below = [&](long long e, int y0, int len) {
            const long long num = e - (long long)y0 - rpc + 1;     // k rpc < num
            const long long k = (num <= 0) ? 0 : (num + rpc - 1) / rpc;
            return (int)(k < len ? k : len);
        };
        for (int pass = 0; pass < 2; pass++) {
            for (int r = wp; r < nruns; r += NT / 32) {
                const unsigned long long k = key[rhead[r]];
                const int img = (int)((k >> 48) & 1), y0 = key_y(k);
                const int c0 = rlen[r], len = ((r + 1 < nruns) ? rlen[r + 1] : total) - c0;
                int lo = 0, n = 0;                // lane b < nb: band b's chunks c0 + [lo, lo + n)
                if (l32 < nb) {
                    lo = (l32 == 0) ? 0 : below(P.rc_band_end[img][l32 - 1], y0, len);
                    n = ((l32 == nb - 1) ? len : below(P.rc_band_end[img][l32], y0, len)) - lo;
                }
                if (pass == 0) {
                    if (n > 0) atomicAdd(&bcnt[l32], n);
                } else {
                    const int off = (n > 0) ? bcnt[16 + l32] + atomicAdd(&bcnt[8 + l32], n) : 0;
                    for (int b = 0; b < nb; b++) {
                        const int ob = __shfl_sync(0xffffffffu, off, b);
                        const int lb = __shfl_sync(0xffffffffu, lo, b);
                        const int nn = __shfl_sync(0xffffffffu, n, b);
                        for (int j = l32; j < nn; j += 32) P.rc_order[ob + j] = c0 + lb + j;
                    }
                }
            }
            __syncthreads();
            if (pass == 0 && tid == 0) {
                int acc = 0;
                for (int b = 0; b < nb; b++) { bcnt[16 + b] = acc; P.rc_band_start[b] = acc; acc += bcnt[b]; }
                P.rc_band_start[nb] = acc;
            }
            __syncthreads();
        }
    }
}

// ------------------------------------------------------------------ row stage

// twiddle entries k_segrows holds: the transform's, and those with the
// half-sample shift where factor 2 uses them
template <int N, int LG>
__host__ __device__ constexpr int segrows_twiddles() { return (N <= 512 && LG < 2) ? 2 * fft_twiddle_len(N) : fft_twiddle_len(N); }

// row buffer of a team in shared memory: two rows of amplitudes in natural
// order, padded (factor 1 keeps them in registers)
__host__ __device__ constexpr int segrows_rowbuf(int n, int lg) { return lg == 0 ? 0 : 2 * n + 32; }

// Sum over the warp of t[m] at index (lane / T) (PER T) + lane % T + T m, in the
// tree order of h_reduceFD_strip (strides halving from the top).  A level whose
// stride is a lane distance leaves each lane half of its values: it sends the
// other half, and the next index bit takes the lane bit's place, so PER values
// cost PER shuffles however many lanes the top levels span.
template <int T, int PER>
__device__ __forceinline__ float chunk_tree(float (&t)[PER], int l32) {
    constexpr int C = (T == 32) ? 0 : (T == 16) ? 1 : (T == 8) ? 2 : 3;      // index bits above a team
    constexpr int LEVELS = C + ((PER == 32) ? 5 : 4);
    static_assert((T << C) == 32 && (PER == 16 || PER == 32), "layout of the sums");
#pragma unroll
    for (int i = 0; i < LEVELS; i++) {
        const int half = (PER >> i) / 2, bit = C ? 16 >> (i % (C ? C : 1)) : 0;
        if (C == 0) {
#pragma unroll
            for (int q = 0; q < half; q++) t[q] = t[q] + t[q + half];
        } else if (half >= 1) {
            const bool hi = (l32 & bit) != 0;
#pragma unroll
            for (int q = 0; q < half; q++) {
                const float mine = hi ? t[q + half] : t[q], other = hi ? t[q] : t[q + half];
                t[q] = mine + __shfl_xor_sync(0xffffffffu, other, bit);
            }
        } else {
            t[0] = t[0] + __shfl_xor_sync(0xffffffffu, t[0], bit);
        }
    }
    float x = t[0];
#pragma unroll
    for (int o = T / 2; o > 0; o >>= 1) x = x + __shfl_xor_sync(0xffffffffu, x, o);
    return x;
}

// Shared-memory wavefronts bound it (88% of the pipe at 512 points, 61% of the
// issue slots), so what a lane can get by shuffles does not go through memory:
// the last pass of a 512-point transform, the mirrored element of the two rows'
// split and the chunk's sum (40,000 patches of 512 x 512: 17.1 -> 15.6 ms; 1000
// of 256 x 256: 156 -> 151 us).
//
// One warp per chunk of rows of one image segment; the structure of k_rows
// (teams of T lanes, the rows t and t + 512 of the chunk through one team,
// rows in registers in the team layout) with one image instead of a window's
// two.  Range interpolation and amplitudes are k_rows' (xcorr.cu:237-250,
// fft_interpolate_routines.cu:76-113, conv_ampl_demean.cu:98-108), the chunk
// sum is h_reduceFD_strip's block sum (conv_ampl_demean.cu:703-726).
// SPEC: the row spectra too; the -time and -time4 modes need none.  (One kernel
// with a branch took fewer registers, and then its CTAs shared an SM with the peak
// stage's: 40,000 windows of 256 x 256 52.3 -> 53.0 ms.)
template <int N, int LG, bool SPEC>
__global__ void __launch_bounds__(128, (N >= 1024) ? 2 : (N >= 512 ? 3 : 4)) k_segrows(Plan P) {
    constexpr int T = fft_lanes(N);
    constexpr int TPW = 32 / T;
    constexpr int PADN = fft_padded_len(N);
    constexpr int RPC = (N >= 1024) ? 1 : 1024 / N;
    constexpr int RPT = (N >= 1024) ? 1 : 2;
    static_assert(RPT * TPW == RPC, "chunk rows");
    constexpr int TWL = fft_twiddle_len(N);
    constexpr int PER = N / T;
    constexpr int NH = N / 2;
    constexpr bool HSHIFT = (LG == 1) && (N <= 512);
    constexpr int TWS = segrows_twiddles<N, LG>();
    constexpr int RBF = segrows_rowbuf(N, LG);
    constexpr int GOFF = 32 / TPW;
    constexpr bool KEEPS = LG >= 2;                     // the row's spectrum is kept for the phases after the first

    extern __shared__ float4 smem_raw[];
    float2 *tw = reinterpret_cast<float2 *>(smem_raw);
    const int warp = threadIdx.x >> 5, l32 = threadIdx.x & 31;
    const int lane = l32 % T;
    const int tm = l32 / T;
    const int team = warp * TPW + tm;
    char *tbase = reinterpret_cast<char *>(tw + TWS) + (size_t)team * (PADN * sizeof(float2) + RBF * sizeof(float));
    float2 *ex = reinterpret_cast<float2 *>(tbase);
    float *rb = reinterpret_cast<float *>(ex + PADN) + tm * GOFF;
    const int rbx = tm & 1;
    float *const rbE = rb + rbx, *const rbO = rb - rbx;
    float *const rbL = (lane & 1) ? rbO : rbE;
    float ar[(LG == 0) ? RPT : 1][PER];                 // factor 1: the amplitudes of the team's rows
    char *after = reinterpret_cast<char *>(tw + TWS) +
                  (size_t)(blockDim.x / T) * (PADN * sizeof(float2) + RBF * sizeof(float));
    // KEEPS: each thread's spectrum elements, [PER][32] per warp
    float2 *spec = reinterpret_cast<float2 *>(after) + (size_t)warp * PER * 32 + l32;

    for (int i = threadIdx.x; i < TWL; i += blockDim.x) tw[i] = P.tw_row[i];
    if constexpr (HSHIFT)
        for (int i = threadIdx.x; i < TWL; i += blockDim.x) tw[TWL + i] = P.phase[i];
    grid_dep_wait();                 // the planner's chunks
    __syncthreads();

    constexpr int ri = 1 << LG;
    constexpr int KM0 = (LG == 0) ? 0 : PER / (2 * ri), KM1 = (LG == 0) ? PER : 3 * PER / (2 * ri);
    // this launch's chunks: all of them in planned order, or one row band's
    const bool banded = P.rc_nbands > 0;
    const int begin = banded ? P.rc_band_start[P.rc_band] : 0;
    // unbanded: the first planner's chunks, then the second's from nwin * nchunks
    const int cm = banded ? 0 : P.rc_count[0];
    const int end = banded ? P.rc_band_start[P.rc_band + 1] : cm + P.rc_count[1];
    const int cbase = P.nwin * P.nchunks;
    const bool iq16 = (P.format == 0);

    // Chunks are taken four per CTA, one per warp; warps share no state between
    // chunks, so a warp that runs out leaves without a barrier.  A warp's next
    // descriptor is read at the start of a chunk and the next chunk's first row
    // during the current one's last, so neither is waited for (40,000
    // patches of 512 x 512: 15.6 -> 13.7 ms; 1000 of 256 x 256: 151 -> 140 us).
    const int step = 4 * gridDim.x;
    auto chunk_of = [&](int i) { return banded ? P.rc_order[i] : (i < cm ? i : cbase + (i - cm)); };
    const void *base;
    int nx, ny, x0, y0, img;
    auto take = [&](const int4 &d) {
        img = d.y;
        const PairDev *q = P.pairs ? P.pairs + d.x : nullptr;
        base = q ? (img ? q->slave : q->master) : (img ? P.single.slave : P.single.master);
        nx = q ? (img ? q->s_nx : q->m_nx) : (img ? P.single.s_nx : P.single.m_nx);
        ny = q ? (img ? q->s_ny : q->m_ny) : (img ? P.single.s_ny : P.single.m_ny);
        x0 = d.z;
        y0 = d.w;
    };
    bool oob = false;                                    // of the chunk whose rows are loaded
    auto load_row = [&](int r, uint32_t *raw) {
        const int y = y0 + r;
        const bool rowok = (y >= 0 && y < ny);
        const uint32_t *row = reinterpret_cast<const uint32_t *>(base) + (size_t)(rowok ? y : 0) * (size_t)nx;
        if (rowok && x0 >= 0 && x0 + N <= nx) {
#pragma unroll
            for (int m = 0; m < PER; m++) raw[m] = __ldg(row + x0 + lane + T * m);
        } else {
#pragma unroll
            for (int m = 0; m < PER; m++) {
                const int x = x0 + lane + T * m;
                if (rowok && x >= 0 && x < nx) raw[m] = __ldg(row + x);
                else { raw[m] = 0u; oob = true; }
            }
        }
    };
    int i = begin + 4 * blockIdx.x + warp;
    if (i >= end) return;
    int c = chunk_of(i);
    take(P.rc_desc[c]);
    uint32_t raw[PER];
    load_row(tm, raw);
    for (;;) {
        const bool more = i + step < end;
        const int cn = more ? chunk_of(i + step) : c;
        const int4 dn = P.rc_desc[cn];
        float mn = INFINITY, mx = -INFINITY;

        auto to_complex = [&](const uint32_t *raw, float2 *v) {
            if (iq16) {
#pragma unroll
                for (int m = 0; m < PER; m++) {
                    const short lo = (short)(raw[m] & 0xffffu), hi = (short)(raw[m] >> 16);
                    v[m] = make_float2((float)lo, (float)hi);
                }
            } else {
#pragma unroll
                for (int m = 0; m < PER; m++) v[m] = make_float2(__uint_as_float(raw[m]), 0.f);
            }
        };
        // amplitudes of one row into rb slot s (natural order of the kept fine samples)
        auto amp_row = [&](int s, int r, const uint32_t *raw) {
            float *const rowE = rbE + s * N, *const rowO = rbO + s * N;
            float2 v[PER];
            to_complex(raw, v);
            if (LG == 0) {
#pragma unroll
                for (int m = 0; m < PER; m++) ar[s][m] = hypotf(v[m].x, v[m].y);
                return;
            }
#pragma unroll
            for (int m = KM0; m < KM1; m++) {
                const int k = ((lane + T * m) << LG) - N / 2;
                rowE[k] = amp_of(v[m]);
            }
            if constexpr (KEEPS) {
                // ri > 2: one forward transform, its elements kept by the
                // thread that holds them (registers have no room).  Transforming
                // the row again for each phase took 150 us where this takes 122
                // (factor 4, 391 windows of 128 x 64)
                team_fft_reg<N, -1>(v, ex, tw, lane);
#pragma unroll
                for (int m = 0; m < PER; m++) spec[32 * m] = v[m];
            }
#pragma unroll 1
            for (int p = 1; p < ri; p++) {
                if constexpr (KEEPS) {
#pragma unroll
                    for (int m = 0; m < PER; m++) v[m] = spec[32 * m];
                } else {
                    team_fft_reg<N, -1>(v, ex, tw, lane);
                }
                if constexpr (HSHIFT) {
                    team_ifft_half_shift<N>(v, ex, tw + TWL, lane);
                } else {
                    const float2 *ph = P.phase + (size_t)(p - 1) * N;
#pragma unroll
                    for (int m = 0; m < PER; m++) v[m] = cmulf(v[m], __ldg(ph + lane + T * m));
                    team_fft_reg<N, +1>(v, ex, tw, lane);
                }
#pragma unroll
                for (int m = KM0; m < KM1; m++) {
                    const int k = ((lane + T * m) << LG) + p - N / 2;
                    ((p & 1) ? rowO : rowE)[k] = amp_of(v[m]);
                }
            }
        };

        int cur_img = img;
        bool any_oob = false;
        constexpr int UNR = (LG == 0) ? RPT : 1;
#pragma unroll UNR
        for (int ir = 0; ir < RPT; ir++) {
            uint32_t cur[PER];
#pragma unroll
            for (int m = 0; m < PER; m++) cur[m] = raw[m];
            // the chunk's next row or the next chunk's first, in flight during this one
            const bool last = (ir + 1 == RPT);
            if (last) {
                cur_img = img;
                any_oob = __ballot_sync(0xffffffffu, oob) != 0u;
                oob = false;
                take(dn);
            }
            if (!last || more) load_row(last ? tm : (ir + 1) * TPW + tm, raw);
            amp_row(ir, ir * TPW + tm, cur);
        }
        __syncwarp();
        // amplitudes out, first reduction level (rows t and t + 512 of the
        // chunk), extremes, and the FFT input: two real rows in one complex
        // sequence; the slave's rows carry its mask columns [N/4, 3N/4) only
        float *ag = P.rc_amp + (size_t)c * RPC * N;
        float2 v[PER];
        float sums[PER];
#pragma unroll
        for (int m = 0; m < PER; m++) {
            const int e = lane + T * m;
            const float a0 = (LG == 0) ? ar[0][m] : rbL[e];
            const float a1 = (RPT == 1) ? 0.f : (LG == 0) ? ar[(LG == 0) ? RPT - 1 : 0][m] : rbL[N + e];
            const bool cin = (m >= PER / 4) && (m < 3 * PER / 4);
            const bool use = (cur_img == 0) || cin;
            // the slave's amplitudes are read only inside its mask columns
            // (the time-correlation window, [xsearch, xsearch + nx_corr))
            if (use) {
                ag[(size_t)tm * N + e] = a0;
                if (RPT == 2) ag[(size_t)(TPW + tm) * N + e] = a1;
            }
            sums[m] = (RPT == 2) ? a0 + a1 : a0;
            if (use) {
                mn = fminf(mn, a0); mx = fmaxf(mx, a0);
                if (RPT == 2) { mn = fminf(mn, a1); mx = fmaxf(mx, a1); }
            }
            v[m] = use ? make_float2(a0, a1) : make_float2(0.f, 0.f);
        }
        {
            const float x = chunk_tree<T>(sums, l32);    // the remaining tree levels
            if (l32 == 0) P.rc_part[c] = x;
        }
        if constexpr (SPEC) {
            team_fft_reg<N, -1>(v, ex, tw, lane);
            // half spectra k in [0, N/2) of both rows; bin 0 carries (DC, Nyquist),
            // both real for a real row.  Element N - k of k = lane + T m is in lane
            // T - lane's register PER - 1 - m (lane 0: in its own PER - m)
            float2 *s0 = P.rc_spec + ((size_t)c * RPC + tm) * NH;
            float2 *s1 = P.rc_spec + ((size_t)c * RPC + TPW + tm) * NH;
            const int mir = (l32 - lane) + ((T - lane) & (T - 1));
            const float2 xn = v[PER / 2];                    // k = 0's lane: the Nyquist bin
#pragma unroll
            for (int m = 0; m < PER / 2; m++) {
                const int k = lane + T * m;
                const float2 z1 = v[m];
                if (RPT == 2) {
                    float2 A, B, z2 = (lane == 0) ? v[(PER - m) % PER] : v[PER - 1 - m];
                    z2.x = __shfl_sync(0xffffffffu, z2.x, mir);
                    z2.y = __shfl_sync(0xffffffffu, z2.y, mir);
                    if (k == 0) {
                        A = make_float2(z1.x, xn.x);
                        B = make_float2(z1.y, xn.y);
                    } else {
                        A = make_float2(0.5f * (z1.x + z2.x), 0.5f * (z1.y - z2.y));
                        B = make_float2(0.5f * (z1.y + z2.y), -0.5f * (z1.x - z2.x));
                    }
                    s0[k] = A;
                    s1[k] = B;
                } else {
                    s0[k] = (k == 0) ? make_float2(z1.x, xn.x) : z1;
                }
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
            mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        }
        if (l32 == 0) {
            P.rc_minmax[c] = make_float2(mn, mx);
            P.rc_oob[c] = any_oob ? 1 : 0;
        }
        if (!more) break;
        i += step;
        c = cn;
        __syncwarp();        // ex and rb are reused by the warp's next chunk
    }
}

// ------------------------------------------------------------------ column stage

// k_cols on the cached half spectra: team kx transforms the master's and the
// masked slave's column kx (rows of the window's chunks); kx = 0 holds the
// packed (DC, Nyquist) columns, separated by Hermitian symmetry in ky.  The
// product, demean/mask corrections (conv_ampl_demean.cu:111-139, applied by
// linearity), (-1)^(kx+ky) shift and inverse column FFT of the surface rows
// are k_cols' (do_freq_xcorr.cu:32-64, 106-114).
template <int M, int THR>
__global__ void __launch_bounds__(THR, ColsGeom<M, THR>::BLOCKS) k_cols_rc(Plan P) {
    using G = ColsGeom<M, THR>;
    constexpr int T = G::T, CS = G::CS, CP = G::CP, TWL = G::TWL;
    constexpr int PER = M / T;
    static_assert((CP & (CP - 1)) == 0 && T % 2 == 0, "columns per CTA: a power of two");
    static_assert(THR == 128, "four warps: two partial chunk sums per patch");

    extern __shared__ float4 smem_raw[];
    float2 *tw = reinterpret_cast<float2 *>(smem_raw);
    float2 *cols = tw + TWL;                   // [2*CP + 1][CS]: master, slave, kx = N/2 product
    float2 *boxy = cols + (2 * CP + 1) * CS;    // [M] DFT of the row mask
    float2 *boxx = boxy + M;                    // [CP + 1] DFT of the column mask at this CTA's kx, then N/2
    double *dsum = reinterpret_cast<double *>(boxx + CP + 1);   // [4] per-warp partial chunk sums

    const int w = blockIdx.y, b = blockIdx.x;
    const int N = P.npx, NH = N / 2;
    const int kx0 = b * CP;
    const int warp = threadIdx.x >> 5, l32 = threadIdx.x & 31;
    const int lane = l32 % T;
    const int team = warp * (32 / T) + l32 / T;
    const int2 wc = P.rc_wch[w];
    const float2 *ms = P.rc_spec + (size_t)wc.x * P.rpc * NH;   // window's master rows, stride NH
    const float2 *ss = P.rc_spec + (size_t)wc.y * P.rpc * NH;   // window's slave rows

    for (int i = threadIdx.x; i < TWL; i += blockDim.x) tw[i] = P.tw_col[i];
    {   // thread t stages slot t % CP for rows t / CP + k * THR/CP: the slave's
        // mask rows [M/4, 3M/4) first (zeros elsewhere), then the master
        constexpr int RSTEP = THR / CP;
        constexpr int NLD = M / RSTEP;
        const int sl = threadIdx.x % CP, row0 = threadIdx.x / CP;
        float2 *sslot = cols + (CP + sl) * CS, *mslot = cols + sl * CS;
#pragma unroll 8
        for (int k = 0; k < NLD; k++) {
            const int r = row0 + k * RSTEP;
            if (r >= M / 4 && r < 3 * M / 4) cp_async8(sslot + fft_pad(r), ss + (size_t)r * NH + kx0 + sl);
            else sslot[fft_pad(r)] = make_float2(0.f, 0.f);
        }
        cp_async_commit();
#pragma unroll 8
        for (int k = 0; k < NLD; k++) {
            const int r = row0 + k * RSTEP;
            cp_async8(mslot + fft_pad(r), ms + (size_t)r * NH + kx0 + sl);
        }
        cp_async_commit();
    }
    // the mask spectra this CTA uses, staged once (per-element reads missed
    // the L1 left beside the column slots)
    for (int i = threadIdx.x; i < M; i += THR) boxy[i] = __ldg(P.box_y + i);
    if (threadIdx.x <= CP) boxx[threadIdx.x] = __ldg(P.box_x + (threadIdx.x < CP ? kx0 + threadIdx.x : NH));
    {
        // patch means (conv_ampl_demean.cu:719-724) from the chunk sums,
        // warps 0-1 the master's, 2-3 the slave's: the FP32 chunk sums of a
        // patch are exact in double, so any order gives the reference's bits
        const int nch = P.nchunks;
        const int base = (warp < 2) ? wc.x : wc.y;
        double sp = 0.0;
        for (int i = (warp & 1) * 32 + l32; i < nch; i += 64) sp += (double)P.rc_part[base + i];
        sp = warp_sum_f64(sp);
        if (l32 == 0) dsum[warp] = sp;
    }
    cp_async_wait<1>();                          // slave columns in (this thread's copies)
    __syncthreads();                             // ... and everyone's
    float dc1, m2;
    {
        const double inv = pow2_inv(N * M);
        const double s1 = (dsum[0] + dsum[1]) * inv, s2 = (dsum[2] + dsum[3]) * inv;
        dc1 = (float)(s1 * (double)N * (double)M);   // the master's DC term, m1 N M
        m2 = (float)s2;
        if (b == 0 && threadIdx.x == 0) { P.means[2 * w] = s1; P.means[2 * w + 1] = s2; }
    }

    const int kx = kx0 + team;
    float2 *a = cols + team * CS;               // master column, later the result
    float2 *pa = cols + (CP + team) * CS;       // slave column
    float2 z[PER];
#pragma unroll
    for (int m = 0; m < PER; m++) z[m] = pa[fft_pad(lane + T * m)];
    __syncwarp();
    team_fft_reg_mid<M, -1>(z, pa, tw, lane);    // zero outside the mask rows
#pragma unroll
    for (int m = 0; m < PER; m++) pa[fft_pad(lane + T * m)] = z[m];
    cp_async_wait<0>();                          // master columns in
    __syncthreads();
#pragma unroll
    for (int m = 0; m < PER; m++) z[m] = a[fft_pad(lane + T * m)];
    __syncwarp();
    team_fft_reg<M, -1>(z, a, tw, lane);
#pragma unroll
    for (int m = 0; m < PER; m++) a[fft_pad(lane + T * m)] = z[m];
    __syncwarp();

    // the kx = 0 team also emits column N/2 (its product goes through the
    // extra slot first); the trip count stays warp-uniform because
    // team_fft_reg synchronises the whole warp
    const bool dc = (kx == 0);
    const int nout = __any_sync(0xffffffffu, dc) ? 2 : 1;
    float2 *xs = cols + 2 * CP * CS;
    auto product = [&](int kxx, float2 A1, float2 A2, int ky) {
        if (kxx == 0 && ky == 0) A1.x -= dc1;
        const float2 bm = cmulf(boxx[kxx == NH ? CP : kxx - kx0], boxy[ky]);
        A2.x -= m2 * bm.x;
        A2.y -= m2 * bm.y;
        float2 pr = cmulf_conj(A1, A2);
        if ((kxx + ky) & 1) { pr.x = -pr.x; pr.y = -pr.y; }
        return pr;
    };
#pragma unroll 1
    for (int o = 0; o < nout; o++) {
        if (o == 0) {
#pragma unroll
            for (int m = 0; m < PER; m++) {
                const int ky = lane + T * m;
                const float2 zm = a[fft_pad(ky)], zs = pa[fft_pad(ky)];
                if (!dc) {
                    z[m] = product(kx, zm, zs, ky);
                } else {
                    // columns kx = 0 and N/2 from the packed (DC, Nyquist) column
                    const int kyn = (M - ky) & (M - 1);
                    const float2 wm = a[fft_pad(kyn)], ws = pa[fft_pad(kyn)];
                    const float2 D1 = make_float2(0.5f * (zm.x + wm.x), 0.5f * (zm.y - wm.y));
                    const float2 D2 = make_float2(0.5f * (zs.x + ws.x), 0.5f * (zs.y - ws.y));
                    const float2 Q1 = make_float2(0.5f * (zm.y + wm.y), -0.5f * (zm.x - wm.x));
                    const float2 Q2 = make_float2(0.5f * (zs.y + ws.y), -0.5f * (zs.x - ws.x));
                    z[m] = product(0, D1, D2, ky);
                    xs[fft_pad(ky)] = product(NH, Q1, Q2, ky);
                }
            }
        } else {
#pragma unroll
            for (int m = 0; m < PER; m++) z[m] = xs[fft_pad(lane + T * m)];
        }
        float2 *dst = (o == 0) ? a : pa;
        __syncwarp();                            // every lane has read a, pa and xs before dst is reused
        team_fft_reg<M, +1>(z, dst, tw, lane);
#pragma unroll
        for (int m = PER / 4; m < 3 * PER / 4; m++) dst[fft_pad(lane + T * m)] = z[m];
        __syncwarp();
    }
    __syncthreads();
    // rows y in [ysearch, ysearch + nyc) of the half spectrum, kx <= N/2
    {
        constexpr int RS = THR / CP;
        float2 *qw = P.qspec + (size_t)w * P.nyc * P.qpitch;
        const int s = threadIdx.x % CP, y0 = threadIdx.x / CP;
        float2 *dstq = qw + (size_t)y0 * P.qpitch + kx0 + s;
        const float2 *srcc = cols + s * CS;
        for (int k = 0; k < (M / 2) / RS; k++) {
            const int sy = (RS % 16 == 0) ? fft_pad(y0 + M / 4) + k * (RS + RS / 16) : fft_pad(y0 + M / 4 + k * RS);
            dstq[(size_t)k * RS * P.qpitch] = srcc[sy];
        }
        if (b == 0)                                // column N/2: the kx = 0 team's slave slot
            for (int yq = threadIdx.x; yq < M / 2; yq += blockDim.x)
                qw[(size_t)yq * P.qpitch + NH] = cols[CP * CS + fft_pad(yq + M / 4)];
    }
}

// The column stage as a persistent, software-pipelined kernel (the default;
// k_cols_rc above is one CTA per tile).  A tile is (window, group of CP
// columns); CTAs take tiles a quarter window at a time from a counter, so a
// CTA's consecutive tiles are mostly the next column groups of one window:
// the twiddles and the row mask's spectrum are staged once per CTA and the
// patch means once per run of a window's tiles.  Per tile: the slave's mask
// rows (staged during the previous tile's inverse transform) are
// transformed first, then the master's (staged during the previous tile's
// copy-out and the slave transform); the master's spectrum stays in
// registers for the product, after which the slave slots are free and the
// next tile's slave rows are requested.  Rows outside the slave's mask are
// zero in registers, never staged, and the slave's first FFT pass skips
// their butterflies.  The arithmetic is k_cols_rc's, operation for
// operation, so the results are the same bits.  Tiles of column group 0 (the
// packed DC/Nyquist column, whose second output goes through the slave slot)
// request the next tile's slave rows only after their copy-out.
// KEEP: the slave's column spectrum stays in registers for the product
// (the default form up to 512-point columns).  LANES: lanes of a column's team;
// MINB: CTAs per SM.
//
// 512-point columns go to teams of 16 lanes with 32 elements each: the
// exchanges through shared memory bound this kernel, and such a team needs one
// per transform where 32 lanes need two.  The registers leave two CTAs per SM
// (205 a thread).  40,000 patches of 512 x 512: 31.2 ms, without the slave's
// spectrum in registers 32.3, with 32 lanes at three CTAs per SM 37.7.
template <int M, int THR, bool KEEP, int LANES, int MINB>
__global__ void __launch_bounds__(THR, MINB) k_cols_rcp(Plan P) {
    using G = ColsGeom<M, THR, LANES>;
    constexpr int T = G::T, CS = G::CS, CP = G::CP, TWL = G::TWL;
    constexpr int PER = M / T;
    constexpr int RSTEP = THR / CP;            // rows a staging pass covers
    static_assert((CP & (CP - 1)) == 0 && T % 2 == 0, "columns per CTA: a power of two");
    static_assert(THR == 128, "four warps: two partial chunk sums per patch");
    static_assert(PER % 4 == 0 && (M / 2) % RSTEP == 0, "mask rows: whole registers and staging passes");

    extern __shared__ float4 smem_raw[];
    float2 *tw = reinterpret_cast<float2 *>(smem_raw);
    float2 *cols = tw + TWL;                   // [2*CP + 1][CS]: master, slave, kx = N/2 product
    float2 *boxy = cols + (2 * CP + 1) * CS;    // [M] DFT of the row mask
    float2 *boxx = boxy + M;                    // [CP + 1] DFT of the column mask at this tile's kx, then N/2
    double *dsum = reinterpret_cast<double *>(boxx + CP + 1);   // [4] per-warp partial chunk sums
    int *grab = reinterpret_cast<int *>(dsum + 4);              // [1] the next chunk of tiles (thread 0's grab)
    float *mval = reinterpret_cast<float *>(grab + 1);          // [2] the window's master DC term and slave mean

    const int N = P.npx, NH = N / 2;
    const int NG = NH / CP;                     // column groups per window
    const int ntiles = P.nwin * NG;
    // Tiles come in chunks from a counter the planner zeroed (a CTA that
    // starts late, behind the other batch's kernels, takes fewer), or,
    // without the counter, as one contiguous range per CTA.  A chunk is a
    // quarter window, or half of a CTA's even share of the tiles where that is
    // less: a strip of 20 windows of 128 x 128 (320 tiles) in quarter windows
    // ran on 80 CTAs, four tiles one after another (86.2 against 73.0 us per
    // call in single tiles).  Shorter chunks towards the end of a large batch
    // cost more in patch means than the shorter tail gives (1000 windows of
    // 128 x 128: 426 against 420 us).
    for (int i = threadIdx.x; i < TWL; i += THR) cp_async8(tw + i, P.tw_col + i);
    for (int i = threadIdx.x; i < M; i += THR) cp_async8(boxy + i, P.box_y + i);
    cp_async_commit();               // a group of its own, complete when the first tile's slave rows are
    grid_dep_wait();                 // the row stage's spectra and sums
    const bool dyn = (P.rc_tile_next != nullptr);
    const int K = max(1, min(NG / 4, ntiles / (2 * (int)gridDim.x)));
    TileWalk walk;
    walk.ntiles = ntiles;
    walk.K = K;
    if (dyn) {
        if (threadIdx.x == 0) *grab = atomicAdd(P.rc_tile_next, K);
        __syncthreads();
        walk.enter(*grab);
        __syncthreads();                        // every thread has read it before the next grab
    } else {
        walk.t = (int)((long long)ntiles * blockIdx.x / gridDim.x);
        walk.end = (int)((long long)ntiles * (blockIdx.x + 1) / gridDim.x);
    }
    if (walk.t >= walk.end) return;
    const int warp = threadIdx.x >> 5, l32 = threadIdx.x & 31;
    const int lane = l32 % T;
    // the columns of a warp: all even or all odd, this team's at 4 times tms;
    // two teams of 8 lanes in a half-warp 8 slots apart, four of 4 lanes 4 slots
    // apart, which puts them in distinct banks
    const int tm = l32 / T, tms = (T == 8) ? (tm >> 1) | ((tm & 1) << 1) : tm;
    const int sl = threadIdx.x % CP, row0 = threadIdx.x / CP;   // staging: slot, first row
    // tile t: window t / NG, column group t % NG (a CTA's consecutive tiles
    // are the next column groups of one window; taking the next windows at
    // one column group instead, so that windows sharing row chunks read them
    // at about the same time, was 29% slower: the means on every tile)
    auto tile = [&](int t, int &w, int &b) { w = t / NG; b = t - w * NG; };

    // tile t's slave mask rows [M/4, 3M/4) / master rows, into the slots (one commit group each)
    auto stage_slave = [&](int t) {
        int w, b;
        tile(t, w, b);
        const int kx0 = b * CP;
        const float2 *src = P.rc_spec + (size_t)P.rc_wch[w].y * P.rpc * NH + kx0 + sl;
        float2 *slot = cols + (CP + sl) * CS;
#pragma unroll 8
        for (int k = 0; k < (M / 2) / RSTEP; k++) {
            const int r = M / 4 + row0 + k * RSTEP;
            cp_async8(slot + fft_pad(r), src + (size_t)r * NH);
        }
        cp_async_commit();
    };
    auto stage_master = [&](int t) {
        int w, b;
        tile(t, w, b);
        const int kx0 = b * CP;
        const float2 *src = P.rc_spec + (size_t)P.rc_wch[w].x * P.rpc * NH + kx0 + sl;
        float2 *slot = cols + sl * CS;
#pragma unroll 8
        for (int k = 0; k < M / RSTEP; k++) {
            const int r = row0 + k * RSTEP;
            cp_async8(slot + fft_pad(r), src + (size_t)r * NH);
        }
        cp_async_commit();
    };

    stage_slave(walk.t);
    stage_master(walk.t);

    int cur_w = -1;
    for (;;) {
        int w, b;
        const int t = walk.t;
        tile(t, w, b);
        // the last tile of a chunk: the next chunk, read after the barrier below
        if (dyn && walk.last() && threadIdx.x == 0) *grab = atomicAdd(P.rc_tile_next, K);
        const int kx0 = b * CP;
        const bool neww = (w != cur_w);
        // (the previous tile's last barrier ordered every read of boxx and dsum before these writes)
        if (threadIdx.x <= CP) boxx[threadIdx.x] = __ldg(P.box_x + (threadIdx.x < CP ? kx0 + threadIdx.x : NH));
        if (neww) {
            // patch means from the chunk sums (conv_ampl_demean.cu:719-724),
            // warps 0-1 the master's, 2-3 the slave's (exact in double: any order)
            const int2 wc = P.rc_wch[w];
            const int base = (warp < 2) ? wc.x : wc.y;
            double sp = 0.0;
            for (int i = (warp & 1) * 32 + l32; i < P.nchunks; i += 64) sp += (double)P.rc_part[base + i];
            sp = warp_sum_f64(sp);
            if (l32 == 0) dsum[warp] = sp;
        }
        cp_async_wait<1>();                      // this tile's slave rows in (this thread's copies)
        __syncthreads();                         // ... and everyone's; boxx, dsum, tw, boxy, grab written
        const int tn = walk.next(dyn && walk.last() ? *grab : ntiles);      // the next tile, none: -1
        if (neww && warp == 0) {                 // one warp: GB300 issues two FP64 operations per SM and cycle
            const double inv = pow2_inv(N * M);
            const double s1 = (dsum[0] + dsum[1]) * inv, s2 = (dsum[2] + dsum[3]) * inv;
            if (l32 == 0) {
                mval[0] = (float)(s1 * (double)N * (double)M);
                mval[1] = (float)s2;
                if (b == 0) { P.means[2 * w] = s1; P.means[2 * w + 1] = s2; }
            }
        }
        cur_w = w;

        // even and odd columns differ in work (below), so the warps take turns
        const int par = (warp ^ t) & 1, slot = par + 2 * (warp >> 1) + 4 * tms;
        const int kx = kx0 + slot;               // kx0 is even
        float2 *a = cols + slot * CS;            // master column, later the result
        float2 *pa = cols + (CP + slot) * CS;    // slave column
        float2 z[PER];
#pragma unroll
        for (int m = 0; m < PER; m++)
            z[m] = (m >= PER / 4 && m < 3 * PER / 4) ? pa[fft_pad(lane + T * m)] : make_float2(0.f, 0.f);
        __syncwarp();
        team_fft_reg_mid<M, -1, T>(z, pa, tw, lane);    // zero outside the mask rows
        float2 zs[KEEP ? PER : 1];
        if constexpr (KEEP) {
#pragma unroll
            for (int m = 0; m < PER; m++) zs[m] = z[m];
        }
        if (!KEEP || b == 0) {                   // column group 0 splits the packed column from the slot
#pragma unroll
            for (int m = 0; m < PER; m++) pa[fft_pad(lane + T * m)] = z[m];
        }
        cp_async_wait<0>();                      // master rows in
        __syncthreads();
        const float dc1 = mval[0], m2 = mval[1];
#pragma unroll
        for (int m = 0; m < PER; m++) z[m] = a[fft_pad(lane + T * m)];
        __syncwarp();
        team_fft_reg<M, -1, T>(z, a, tw, lane);

        // The shift's sign (-1)^(kx + ky): the half in ky swaps the halves of the
        // inverse transform's output, bit for bit (the sign is the same for all
        // inputs of a butterfly until the pass that adds even and odd inputs, and
        // swaps its sums and differences), so the stores below swap them instead.
        // The mask's spectrum is zero in even kx but 0: those columns take no
        // correction, and in odd ones the sign goes into it (with the warps' columns
        // of one parity, the column stage of 1000 windows of 128 x 128 187 -> 182
        // us; of 391 of 128 x 64, also by the banks, 51 -> 43).
        auto product = [&](int kxx, float2 A1, float2 A2, int ky) {
            if (kxx == 0 && ky == 0) A1.x -= dc1;
            const float2 bm = cmulf(boxx[kxx == NH ? CP : kxx - kx0], boxy[ky]);
            A2.x -= m2 * bm.x;
            A2.y -= m2 * bm.y;
            float2 pr = cmulf_conj(A1, A2);
            if (kxx & 1) { pr.x = -pr.x; pr.y = -pr.y; }
            return pr;
        };
        auto product_odd = [&](float2 bx, float2 A1, float2 A2, int ky) {
            const float2 bm = cmulf(bx, boxy[ky]);
            return cmulf_conj(A1, make_float2(m2 * bm.x - A2.x, m2 * bm.y - A2.y));
        };
        // the product of column kx: from the master spectrum in registers, or
        // in column group 0 (CTA-uniform) through the master slot, where the
        // kx = 0 team splits the packed (DC, Nyquist) column and puts column
        // N/2's product in the extra slot
        const bool dc = (kx == 0);
        const int nout = (b == 0 && __any_sync(0xffffffffu, dc)) ? 2 : 1;    // warp-uniform
        float2 *xs = cols + 2 * CP * CS;
        if (b != 0 && par == 0) {
#pragma unroll
            for (int m = 0; m < PER; m++) {
                if constexpr (KEEP) z[m] = cmulf_conj(z[m], zs[m]);
                else z[m] = cmulf_conj(z[m], pa[fft_pad(lane + T * m)]);
            }
        } else if (b != 0) {
            const float2 bx = boxx[slot];
#pragma unroll
            for (int m = 0; m < PER; m++) {
                const int ky = lane + T * m;
                if constexpr (KEEP) z[m] = product_odd(bx, z[m], zs[m], ky);
                else z[m] = product_odd(bx, z[m], pa[fft_pad(ky)], ky);
            }
        } else {
#pragma unroll
            for (int m = 0; m < PER; m++) a[fft_pad(lane + T * m)] = z[m];
            __syncwarp();
#pragma unroll
            for (int m = 0; m < PER; m++) {
                const int ky = lane + T * m;
                const float2 zm = a[fft_pad(ky)], zs = pa[fft_pad(ky)];
                if (!dc) {
                    z[m] = product(kx, zm, zs, ky);
                } else {
                    const int kyn = (M - ky) & (M - 1);
                    const float2 wm = a[fft_pad(kyn)], ws = pa[fft_pad(kyn)];
                    const float2 D1 = make_float2(0.5f * (zm.x + wm.x), 0.5f * (zm.y - wm.y));
                    const float2 D2 = make_float2(0.5f * (zs.x + ws.x), 0.5f * (zs.y - ws.y));
                    const float2 Q1 = make_float2(0.5f * (zm.y + wm.y), -0.5f * (zm.x - wm.x));
                    const float2 Q2 = make_float2(0.5f * (zs.y + ws.y), -0.5f * (zs.x - ws.x));
                    z[m] = product(0, D1, D2, ky);
                    xs[fft_pad(ky)] = product(NH, Q1, Q2, ky);
                }
            }
        }
        __syncthreads();                         // every team has read its slave column
        // outside column group 0 the slave slots are free: the next tile's slave rows
        if (b != 0 && tn >= 0) stage_slave(tn);
        // inverse of column kx into its master slot; in column group 0 the
        // kx = 0 team's second output, column N/2, into its slave slot (one
        // call site of the transform for both cases)
#pragma unroll 1
        for (int o = 0; o < nout; o++) {
            if (o == 1) {
#pragma unroll
                for (int m = 0; m < PER; m++) z[m] = xs[fft_pad(lane + T * m)];
            }
            float2 *dst = (o == 0) ? a : pa;
            __syncwarp();
            team_fft_reg<M, +1, T>(z, dst, tw, lane);
#pragma unroll
            for (int m = PER / 4; m < 3 * PER / 4; m++) dst[fft_pad(lane + T * m)] = z[(m + PER / 2) % PER];
            __syncwarp();
        }
        __syncthreads();
        {   // rows y in [ysearch, ysearch + nyc) of the half spectrum, kx <= N/2
            constexpr int RS = THR / CP;
            float2 *qw = P.qspec + (size_t)w * P.nyc * P.qpitch;
            float2 *dstq = qw + (size_t)row0 * P.qpitch + kx0 + sl;
            const float2 *srcc = cols + sl * CS;
            for (int k = 0; k < (M / 2) / RS; k++) {
                const int sy = (RS % 16 == 0) ? fft_pad(row0 + M / 4) + k * (RS + RS / 16)
                                              : fft_pad(row0 + M / 4 + k * RS);
                dstq[(size_t)k * RS * P.qpitch] = srcc[sy];
            }
            if (b == 0)
                for (int yq = threadIdx.x; yq < M / 2; yq += THR)
                    qw[(size_t)yq * P.qpitch + NH] = cols[CP * CS + fft_pad(yq + M / 4)];
        }
        __syncthreads();                         // the slots are read: the next tile's rows may land
        if (tn < 0) break;
        if (b == 0) stage_slave(tn);
        stage_master(tn);
        walk.go(tn);
    }
}

// ------------------------------------------------------------------ launchers

// threads of the planner for nent entries per CTA: one entry each up to 512,
// then up to eight (a CTA of 1024 threads waits for an SM without other work)
static int plan_threads(int nent) { return nent <= 128 ? 128 : 512; }
static size_t rc_plan_smem_bytes(int nent) {
    int n = plan_threads(nent);
    while (n < nent) n <<= 1;
    return (size_t)n * (sizeof(unsigned long long) + 5 * sizeof(int)) + 72 * sizeof(int);
}
template <int N, int LG>
static size_t segrows_smem() {
    constexpr int T = fft_lanes(N);
    const int teams = 128 / T;
    return segrows_twiddles<N, LG>() * sizeof(float2) +
           (size_t)teams * (fft_padded_len(N) * sizeof(float2) + segrows_rowbuf(N, LG) * sizeof(float)) +
           (LG >= 2 ? (size_t)128 * (N / T) * sizeof(float2) : 0);
}
template <int M, int LANES = fft_lanes(M)>
static size_t cols_rc_smem() {
    using G = ColsGeom<M, 128, LANES>;
    return G::TWL * sizeof(float2) + (size_t)(2 * G::CP + 1) * G::CS * sizeof(float2) +
           (size_t)(M + G::CP + 1) * sizeof(float2) + 4 * sizeof(double) + 16;
}

template <int N, bool SPEC>
static cudaError_t setup_segrows_t() {
    cudaError_t e = cudaSuccess;
    auto set = [&](auto kern, size_t bytes) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
    };
    set(k_segrows<N, 0, SPEC>, segrows_smem<N, 0>());
    set(k_segrows<N, 1, SPEC>, segrows_smem<N, 1>());
    set(k_segrows<N, 2, SPEC>, segrows_smem<N, 2>());
    set(k_segrows<N, 3, SPEC>, segrows_smem<N, 3>());
    return e;
}
// The persistent column stage in a form: WIDE (512 points: 16 lanes per
// column) or not, the slave's spectrum kept in registers or not (at one CTA
// per SM fewer).
template <int M, bool WIDE, bool KEEP>
struct ColsForm {
    static constexpr int LANES = WIDE ? 16 : fft_lanes(M);
    static constexpr int MINB = WIDE ? 2 : (KEEP ? ColsGeom<M, 128>::BLOCKS - 1 : ColsGeom<M, 128>::BLOCKS);
    static constexpr int CP = ColsGeom<M, 128, LANES>::CP;
    static size_t smem() { return cols_rc_smem<M, LANES>(); }
    static auto kernel() { return k_cols_rcp<M, 128, KEEP, LANES, MINB>; }
    static cudaError_t setup() {
        return cudaFuncSetAttribute(kernel(), cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem());
    }
    static void launch(const Plan &P, int sms, cudaStream_t s) {
        const int ntiles = (P.npx / 2) / CP * P.nwin;
        launch_chain(P, kernel(), dim3(std::min(ntiles, sms * MINB)), 128, smem(), s);
    }
};
// the default form of a size and the one launch shape 2 takes
template <int M>
struct ColsForms {
    using Default = ColsForm<M, M == 512, (M <= 512)>;
    using Other = ColsForm<M, false, (M >= 1024)>;
};
template <int M>
static cudaError_t setup_cols_rc_t() {
    cudaError_t e = cudaFuncSetAttribute(k_cols_rc<M, 128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)cols_rc_smem<M>());
    if (!e) e = ColsForms<M>::Default::setup();
    return e ? e : ColsForms<M>::Other::setup();
}

cudaError_t segrows_setup(const Plan &P) {
    cudaError_t e = cudaFuncSetAttribute(k_rc_plan<512, RC_ENTRIES / 512>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         (int)rc_plan_smem_bytes(RC_ENTRIES));
    if (e) return e;
    const bool spec = (P.corr_mode == 2);           // the time modes have 128 columns or more
    switch (P.npx) {
        case 64: e = setup_segrows_t<64, true>(); break;
        case 128: e = spec ? setup_segrows_t<128, true>() : setup_segrows_t<128, false>(); break;
        case 256: e = spec ? setup_segrows_t<256, true>() : setup_segrows_t<256, false>(); break;
        case 512: e = spec ? setup_segrows_t<512, true>() : setup_segrows_t<512, false>(); break;
        case 1024: e = spec ? setup_segrows_t<1024, true>() : setup_segrows_t<1024, false>(); break;
        default: return cudaErrorInvalidValue;
    }
    if (e) return e;
    switch (P.npy) {
        case 64: return setup_cols_rc_t<64>();
        case 128: return setup_cols_rc_t<128>();
        case 256: return setup_cols_rc_t<256>();
        case 512: return setup_cols_rc_t<512>();
        case 1024: return setup_cols_rc_t<1024>();
    }
    return cudaErrorInvalidValue;
}

size_t rc_max_chunks(int npx, int npy, int nwin) {
    const int rpc = npx >= 1024 ? 1 : 1024 / npx;
    return (size_t)2 * nwin * (size_t)(npy / rpc);
}

void launch_rc_plan(const Plan &P, cudaStream_t s) {
    // one CTA per image unless the host entry wants the chunks listed by row band
    const int ctas = P.rc_nbands > 0 ? 1 : 2, nent = ctas == 1 ? 2 * P.nwin : P.nwin;
    const size_t sm = rc_plan_smem_bytes(nent);
    if (nent <= 128) k_rc_plan<128, 1><<<ctas, 128, sm, s>>>(P);
    else if (nent <= 512) k_rc_plan<512, 1><<<ctas, 512, sm, s>>>(P);
    else k_rc_plan<512, RC_ENTRIES / 512><<<ctas, 512, sm, s>>>(P);
}

template <int N, bool SPEC = true>
static void launch_segrows_t(const Plan &P, cudaStream_t s) {
    // a grid-stride walk over the planned chunks, four per CTA; the grid is
    // sized for the chunks the batch would have without sharing, capped at
    // a multiple of the CTAs that fit the GPU at once: four (a warp reads ahead
    // from its second chunk on; with an earlier form of it 1000 windows of 128 x 128
    // took 387 us at eight, 381 at four, 379 at two, where 40,000 of 256 x 256 took
    // 52.6 ms, 52.5, 52.6), one for a row band, a share of the chunks (1000
    // windows through host buffers: 547 us, at a half 568, at two 559)
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const size_t maxq = (rc_max_chunks(P.npx, P.npy, P.nwin) + 3) / 4;
    const int per_sm = (N >= 1024) ? 2 : (N >= 512 ? 3 : 4);
    const size_t cap = (size_t)sms * per_sm * (P.rc_nbands > 0 ? 1 : 4);
    const int grid = (int)((maxq < cap) ? maxq : cap);
    switch (P.log2ri) {
        case 0: launch_chain(P, k_segrows<N, 0, SPEC>, dim3(grid), 128, segrows_smem<N, 0>(), s); break;
        case 1: launch_chain(P, k_segrows<N, 1, SPEC>, dim3(grid), 128, segrows_smem<N, 1>(), s); break;
        case 2: launch_chain(P, k_segrows<N, 2, SPEC>, dim3(grid), 128, segrows_smem<N, 2>(), s); break;
        default: launch_chain(P, k_segrows<N, 3, SPEC>, dim3(grid), 128, segrows_smem<N, 3>(), s); break;
    }
}
void launch_segrows(const Plan &P, cudaStream_t s) {
    if (P.corr_mode < 2) {
        switch (P.npx) {
            case 128: launch_segrows_t<128, false>(P, s); break;
            case 256: launch_segrows_t<256, false>(P, s); break;
            case 512: launch_segrows_t<512, false>(P, s); break;
            case 1024: launch_segrows_t<1024, false>(P, s); break;
        }
        return;
    }
    switch (P.npx) {
        case 64: launch_segrows_t<64>(P, s); break;
        case 128: launch_segrows_t<128>(P, s); break;
        case 256: launch_segrows_t<256>(P, s); break;
        case 512: launch_segrows_t<512>(P, s); break;
        case 1024: launch_segrows_t<1024>(P, s); break;
    }
}

template <int M>
static void launch_cols_rc_t(const Plan &P, cudaStream_t s) {
    using G = ColsGeom<M, 128>;
    if (P.cols_cfg == 1) {                       // one CTA per tile
        dim3 grid((P.npx / 2) / G::CP, P.nwin);
        k_cols_rc<M, 128><<<grid, 128, cols_rc_smem<M>(), s>>>(P);      // (not a dependent: it does not wait)
        return;
    }
    // persistent: one CTA per resident slot, tiles from a counter (leaving
    // one slot per SM to the other batch's kernels measured the same on the
    // device entry and slower on the host entry)
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (P.cols_cfg == 2) ColsForms<M>::Other::launch(P, sms, s);
    else ColsForms<M>::Default::launch(P, sms, s);
}
void launch_cols_rc(const Plan &P, cudaStream_t s) {
    switch (P.npy) {
        case 64: launch_cols_rc_t<64>(P, s); break;
        case 128: launch_cols_rc_t<128>(P, s); break;
        case 256: launch_cols_rc_t<256>(P, s); break;
        case 512: launch_cols_rc_t<512>(P, s); break;
        case 1024: launch_cols_rc_t<1024>(P, s); break;
    }
}

}  // namespace xcg
