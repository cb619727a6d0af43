// Subpixel refiner: a small CNN that reads the normalised 9x9 correlation
// surface around the integer peak and predicts the subpixel peak position
// (fx, fy, in surface pixels, the quantities highres_corr returns as
// xfrac/yfrac, highres_corr.cu:67-76) and the log variance s of that
// estimate.  No counterpart in the reference; it stands in for the FFT
// zero-pad interpolation where it is confident.
//
// Network (valid 3x3 convolutions, GELU): 9x9 -> 32@7x7 -> 32@5x5 -> 32@3x3
// -> dense 64 -> dense 3.  37,507 parameters, FP32 master copy.
//   training:  k_ref_fwd (the convolutions, FP32, keeps activations and GELU
//              derivatives) -> k_ref_dense (the dense layers forward, the
//              loss, and back) -> k_ref_bwd (the convolutions back) ->
//              k_ref_wgrad (partial parameter gradients) -> k_ref_reduce ->
//              k_ref_adam
//   inference: k_ref_infer, BF16 weights and activations on the tensor cores
//              (mma.sync m16n8k16, FP32 accumulation), conv+GELU fused with
//              the activations channel-last in shared memory, one CTA per
//              window at a time.
// Loss per sample: 0.5 r^2 + 0.5 stopgrad(r^2) exp(-s) + s.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include <algorithm>

#include "refiner.cuh"

namespace xcg {

__device__ __forceinline__ float gelu_f(float x) { return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f)); }

__device__ __forceinline__ void cp_async16(void *smem, const void *gmem) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gmem) : "memory");
}

// ---------------------------------------------------------------- training kernels
// FP32 multiply-adds bound them: 1.04 M per sample in all, 0.11 ms per 4096
// samples at the measured FP32 rate.  In the convolutions a thread holds all
// outputs of one channel of one sample, so a shared-memory read (a row that the
// whole warp shares, or one weight per lane) feeds 4 to 10 of them; the layers
// run as roles of different warps on successive groups of four samples, one
// barrier per group, every scheduler with one warp of each role.  One CTA per SM
// takes a contiguous range of samples.  A gradient of 4096 samples with its host
// copies: 338 us (layer after layer on one group at a time, a barrier between
// layers: 437; a thread per output in one kernel each way: 4340).

// Activation rows are padded to 8 floats (4 for the 3-wide rows), channels to
// strides whose 16-byte accesses by consecutive lanes hit distinct banks.
constexpr int TR_S = 4;                        // samples of a group
constexpr int X0_S = 108, X0_R = 12;           // input: sample stride, row stride
constexpr int A3_SS = 292;                     // dense input: sample stride in shared memory

__device__ __forceinline__ void ld4(float *d, const float *s) {
    const float4 v = *reinterpret_cast<const float4 *>(s);
    d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
}
// GELU and, when G, its derivative from one erff
template <bool G>
__device__ __forceinline__ float gelu_both(float x, float &grad) {
    const float e = erff(x * 0.70710678118654752f);
    if (G) grad = 0.5f * (1.0f + e) + x * 0.39894228040143268f * expf(-0.5f * x * x);
    return 0.5f * x * (1.0f + e);
}
// a shared array (size and addresses multiples of 16 bytes) to global memory, by one thread
__device__ __forceinline__ void bulk_out(float *gmem, const float *smem, int bytes) {
    asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;\n" ::"l"(gmem),
                 "r"((unsigned)__cvta_generic_to_shared(smem)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;\n" ::: "memory"); }
// all but the N newest groups have read their shared memory / are complete
template <int N>
__device__ __forceinline__ void bulk_wait_read() { asm volatile("cp.async.bulk.wait_group.read %0;\n" ::"n"(N) : "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;\n" ::: "memory"); }
__device__ __forceinline__ void fence_bulk() { asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory"); }

// A valid 3x3 convolution of one sample for output channel c: WO x WO sums, 32
// input channels in_cs apart at `in` (rows of 8), weights [k][tap][c].  Each
// sum runs over the input channels, then the taps.
template <int WO>
__device__ __forceinline__ void conv_all(float (&y)[WO][WO], const float *in, int in_cs, const float *W, int c) {
#pragma unroll 1
    for (int k = 0; k < 32; k++) {
        float w[9];
#pragma unroll
        for (int d = 0; d < 9; d++) w[d] = W[(k * 9 + d) * 32 + c];
#pragma unroll
        for (int r = 0; r < WO + 2; r++) {
            float x[8];
            ld4(x, in + k * in_cs + r * 8);
            ld4(x + 4, in + k * in_cs + r * 8 + 4);
#pragma unroll
            for (int di = 0; di < 3; di++) {
                if (r - di < 0 || r - di >= WO) continue;
#pragma unroll
                for (int dj = 0; dj < 3; dj++)
#pragma unroll
                    for (int j = 0; j < WO; j++) y[r - di][j] = fmaf(w[di * 3 + dj], x[j + dj], y[r - di][j]);
            }
        }
    }
}

// The convolutions' forward pass.  Warps 0-3: conv2, 4-7: conv3, 8-11: conv1,
// a warp per sample, a lane per channel; in one step conv1 works on group t,
// conv2 on t - 1, conv3 on t - 2.  TRAIN: the activations and the GELU
// derivatives go to the sample's record, else only conv3's activations.
constexpr int FWD_THREADS = 384;
template <bool TRAIN>
__global__ void __launch_bounds__(FWD_THREADS, 1) k_ref_fwd(RefPlan R, const float *__restrict__ feat, int n) {
    extern __shared__ float4 smem_v[];
    float *W2 = reinterpret_cast<float *>(smem_v);     // [k*9 + tap][c]
    float *W3 = W2 + 9216;
    float *a1 = W3 + 9216;                             // [2][TR_S][A1_LEN] by the group's parity
    float *a2 = a1 + 2 * TR_S * A1_LEN;                // [2][TR_S][A2_LEN]
    float *x0 = a2 + 2 * TR_S * A2_LEN;                // [TR_S][X0_S]
    const int tid = threadIdx.x, c = tid & 31, warp = tid >> 5, s = warp & 3, role = warp >> 2;
    const int per = (n + gridDim.x - 1) / gridDim.x;
    const int s_beg = blockIdx.x * per, s_end = min(n, s_beg + per);
    if (s_beg >= s_end) return;
    for (int i = tid; i < 9216 / 4; i += FWD_THREADS) {
        reinterpret_cast<float4 *>(W2)[i] = reinterpret_cast<const float4 *>(R.w2t)[i];
        reinterpret_cast<float4 *>(W3)[i] = reinterpret_cast<const float4 *>(R.w3t)[i];
    }
    const float *P = R.theta;
    const int groups = (s_end - s_beg + TR_S - 1) / TR_S;
    float w1[9], bias = P[(role == 0 ? RP_B2 : role == 1 ? RP_B3 : RP_B1) + c];
#pragma unroll
    for (int d = 0; d < 9; d++) w1[d] = __ldg(P + RP_W1 + c * 9 + d);
    float nx[3] = {0.f, 0.f, 0.f};                     // conv1: the next group's input, 81 values over the lanes
    auto fetch = [&](int g) {
        const int at = s_beg + g * TR_S + s;
#pragma unroll
        for (int q = 0; q < 3; q++) nx[q] = (at < s_end && c + 32 * q < 81) ? feat[(size_t)at * 81 + c + 32 * q] : 0.f;
    };
    if (role == 2) fetch(0);
    __syncthreads();
    for (int t = 0; t < groups + 2; t++) {
        const int g = t - (role == 2 ? 0 : role == 0 ? 1 : 2);      // this role's group
        const int at = s_beg + g * TR_S + s;
        const bool have = g >= 0 && g < groups && at < s_end;
        float *rec = R.act + (size_t)(have ? at : s_beg) * REF_ACT;
        const int buf = g & 1;
        if (role == 2) {                               // conv1
            float *xs = x0 + s * X0_S;
#pragma unroll
            for (int q = 0; q < 3; q++) {
                const int e = c + 32 * q;
                if (e < 81) xs[(e / 9) * X0_R + e % 9] = nx[q];
            }
            __syncwarp();
            fetch(g + 1);
            if (have) {
                float *out = a1 + (buf * TR_S + s) * A1_LEN + c * A1_CS;
#pragma unroll 1
                for (int row = 0; row < 7; row++) {
                    float y[7], a[8], gd[8];
#pragma unroll
                    for (int j = 0; j < 7; j++) y[j] = bias;
#pragma unroll
                    for (int di = 0; di < 3; di++) {
                        float x[12];
                        const float *xr = xs + (row + di) * X0_R;
                        ld4(x, xr); ld4(x + 4, xr + 4); ld4(x + 8, xr + 8);
#pragma unroll
                        for (int dj = 0; dj < 3; dj++)
#pragma unroll
                            for (int j = 0; j < 7; j++) y[j] = fmaf(w1[di * 3 + dj], x[j + dj], y[j]);
                    }
                    a[7] = gd[7] = 0.f;
#pragma unroll
                    for (int j = 0; j < 7; j++) a[j] = gelu_both<TRAIN>(y[j], gd[j]);
#pragma unroll
                    for (int v = 0; v < 2; v++) {
                        *reinterpret_cast<float4 *>(out + row * 8 + 4 * v) = make_float4(a[4 * v], a[4 * v + 1], a[4 * v + 2], a[4 * v + 3]);
                        if (TRAIN)
                            *reinterpret_cast<float4 *>(rec + ACT_D1 + c * 56 + row * 8 + 4 * v) =
                                make_float4(gd[4 * v], gd[4 * v + 1], gd[4 * v + 2], gd[4 * v + 3]);
                    }
                }
            }
            __syncwarp();
        } else if (role == 0) {                        // conv2
            if (have) {
                float y[5][5];
#pragma unroll
                for (int i = 0; i < 5; i++)
#pragma unroll
                    for (int j = 0; j < 5; j++) y[i][j] = bias;
                conv_all<5>(y, a1 + (buf * TR_S + s) * A1_LEN, A1_CS, W2, c);
                float *out = a2 + (buf * TR_S + s) * A2_LEN + c * A2_CS;
#pragma unroll
                for (int i = 0; i < 5; i++) {
                    float a[8], gd[8];
#pragma unroll
                    for (int j = 5; j < 8; j++) a[j] = gd[j] = 0.f;
#pragma unroll
                    for (int j = 0; j < 5; j++) a[j] = gelu_both<TRAIN>(y[i][j], gd[j]);
#pragma unroll
                    for (int v = 0; v < 2; v++) {
                        *reinterpret_cast<float4 *>(out + i * 8 + 4 * v) = make_float4(a[4 * v], a[4 * v + 1], a[4 * v + 2], a[4 * v + 3]);
                        if (TRAIN)
                            *reinterpret_cast<float4 *>(rec + ACT_D2 + c * 40 + i * 8 + 4 * v) =
                                make_float4(gd[4 * v], gd[4 * v + 1], gd[4 * v + 2], gd[4 * v + 3]);
                    }
                }
            }
        } else if (have) {                             // conv3
            float y[3][3];
#pragma unroll
            for (int i = 0; i < 3; i++)
#pragma unroll
                for (int j = 0; j < 3; j++) y[i][j] = bias;
            conv_all<3>(y, a2 + (buf * TR_S + s) * A2_LEN, A2_CS, W3, c);
#pragma unroll
            for (int i = 0; i < 3; i++)
#pragma unroll
                for (int j = 0; j < 3; j++) {
                    float gd;
                    const float a = gelu_both<TRAIN>(y[i][j], gd);
                    rec[ACT_A3 + c * 9 + i * 3 + j] = a;
                    if (TRAIN) rec[ACT_D3 + c * 9 + i * 3 + j] = gd;
                }
        }
        // the activations written in this step go out while the next step reads
        // them; a buffer is written again two steps later
        if (TRAIN) {
            if (c == 0 && role != 1) bulk_wait_read<0>();      // this warp's copy of the step before
            fence_bulk();
        }
        __syncthreads();
        if (TRAIN && c == 0 && have) {
            if (role == 2) bulk_out(rec + ACT_A1, a1 + (buf * TR_S + s) * A1_LEN, A1_LEN * 4);
            if (role == 0) bulk_out(rec + ACT_A2, a2 + (buf * TR_S + s) * A2_LEN, A2_LEN * 4);
            bulk_commit();
        }
    }
    if (TRAIN && c == 0) bulk_wait_all();
}

// The dense layers of 32 samples per CTA, forward (288 -> 64 -> 3), and in
// training the loss and the gradients back to conv3's pre-activations.  A
// thread's forward tile is 4 outputs x 2 samples (each sum over the inputs in
// order), its backward tile 9 inputs x 4 samples.
constexpr int DN_S = 32, DN_THREADS = 256, F1_S = 68, Z_S = 68;    // samples, threads, padded row strides
template <bool TRAIN>
__global__ void __launch_bounds__(DN_THREADS, 1) k_ref_dense(RefPlan R, const float *__restrict__ target, int n) {
    extern __shared__ float4 smem_v[];
    float *F1 = reinterpret_cast<float *>(smem_v);     // [288][F1_S]: (input, output)
    float *a3 = F1 + 288 * F1_S;                       // [DN_S][A3_SS]
    float *g1 = a3 + DN_S * A3_SS;                     // [DN_S][Z_S] outputs of the first layer, then their gradients
    float *dg = g1 + DN_S * Z_S;                       // [DN_S][Z_S] GELU derivatives
    float *F2 = dg + DN_S * Z_S;                       // [3][64]
    float *dout = F2 + 192;                            // [DN_S][4]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int s0 = blockIdx.x * DN_S, m = min(DN_S, n - s0);
    const float *P = R.theta;
    for (int i = tid; i < 288 * 16; i += DN_THREADS) cp_async16(F1 + (i >> 4) * F1_S + 4 * (i & 15), R.f1t + 4 * i);
    for (int i = tid; i < DN_S * 72; i += DN_THREADS) {
        const int ss = i / 72, e = i - 72 * ss;
        if (ss < m) cp_async16(a3 + ss * A3_SS + 4 * e, R.act + (size_t)(s0 + ss) * REF_ACT + ACT_A3 + 4 * e);
        else *reinterpret_cast<float4 *>(a3 + ss * A3_SS + 4 * e) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    if (tid < 192) F2[tid] = P[RP_F2 + tid];
    __syncthreads();
    {
        const int o = 4 * (tid & 15), sp = 2 * (tid >> 4);
        float z[2][4];
#pragma unroll
        for (int k = 0; k < 4; k++) z[0][k] = z[1][k] = P[RP_C1 + o + k];
        const float *p0 = a3 + sp * A3_SS, *p1 = p0 + A3_SS;
#pragma unroll 4
        for (int h = 0; h < 288; h += 4) {
            float u0[4], u1[4];
            ld4(u0, p0 + h);
            ld4(u1, p1 + h);
#pragma unroll
            for (int q = 0; q < 4; q++) {
                float w[4];
                ld4(w, F1 + (h + q) * F1_S + o);
#pragma unroll
                for (int k = 0; k < 4; k++) { z[0][k] = fmaf(w[k], u0[q], z[0][k]); z[1][k] = fmaf(w[k], u1[q], z[1][k]); }
            }
        }
#pragma unroll
        for (int b = 0; b < 2; b++) {
            float a[4], g[4];
#pragma unroll
            for (int k = 0; k < 4; k++) a[k] = gelu_both<TRAIN>(z[b][k], g[k]);
            const float4 av = make_float4(a[0], a[1], a[2], a[3]);
            *reinterpret_cast<float4 *>(g1 + (sp + b) * Z_S + o) = av;
            if (TRAIN) {
                *reinterpret_cast<float4 *>(dg + (sp + b) * Z_S + o) = make_float4(g[0], g[1], g[2], g[3]);
                if (sp + b < m) *reinterpret_cast<float4 *>(R.act + (size_t)(s0 + sp + b) * REF_ACT + ACT_G1 + o) = av;
            }
        }
    }
    __syncthreads();
    if (tid < 3 * DN_S) {
        const int ss = tid / 3, o = tid - 3 * ss;
        float v = P[RP_C2 + o];
#pragma unroll 8
        for (int k = 0; k < 64; k++) v = fmaf(F2[o * 64 + k], g1[ss * Z_S + k], v);
        if (R.out && ss < m) R.out[(size_t)(s0 + ss) * 3 + o] = v;
        dout[ss * 4 + o] = v;
    }
    if (!TRAIN) return;
    __syncthreads();
    if (tid < DN_S) {
        float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
        if (tid < m) {
            const int sg = s0 + tid;
            const float inv_n = 1.0f / (float)n;
            const float lv = dout[tid * 4 + 2];
            const float rx = dout[tid * 4] - target[2 * sg], ry = dout[tid * 4 + 1] - target[2 * sg + 1];
            const float r2 = rx * rx + ry * ry;
            d.x = rx * inv_n;
            d.y = ry * inv_n;
            d.z = (1.0f - 0.5f * r2 * expf(-lv)) * inv_n;
            if (R.loss) R.loss[sg] = 0.5f * r2 + 0.5f * r2 * expf(-lv) + lv;
            *reinterpret_cast<float4 *>(R.grad_act + (size_t)sg * REF_GRAD + GRD_OUT) = d;
        }
        *reinterpret_cast<float4 *>(dout + tid * 4) = d;
    }
    __syncthreads();
    for (int i = tid; i < DN_S * 64; i += DN_THREADS) {
        const int ss = i >> 6, o = i & 63;
        float g = 0.f;
#pragma unroll
        for (int e = 0; e < 3; e++) g = fmaf(F2[e * 64 + o], dout[ss * 4 + e], g);
        const float v = g * dg[ss * Z_S + o];
        g1[ss * Z_S + o] = v;
        if (ss < m) R.grad_act[(size_t)(s0 + ss) * REF_GRAD + GRD_Z + o] = v;
    }
    __syncthreads();
    {   // inputs lane + 32 j of samples 4 warp .. 4 warp + 3
        float g[9][4] = {}, dv[9][4];
#pragma unroll
        for (int j = 0; j < 9; j++)
#pragma unroll
            for (int b = 0; b < 4; b++)
                dv[j][b] = 4 * warp + b < m ? R.act[(size_t)(s0 + 4 * warp + b) * REF_ACT + ACT_D3 + lane + 32 * j] : 0.f;
        const float *dz = g1 + 4 * warp * Z_S;
#pragma unroll 2
        for (int o = 0; o < 64; o += 4) {
            float d[4][4];
#pragma unroll
            for (int b = 0; b < 4; b++) ld4(d[b], dz + b * Z_S + o);
#pragma unroll
            for (int j = 0; j < 9; j++) {
                float w[4];
                ld4(w, F1 + (lane + 32 * j) * F1_S + o);
#pragma unroll
                for (int b = 0; b < 4; b++)
#pragma unroll
                    for (int e = 0; e < 4; e++) g[j][b] = fmaf(w[e], d[b][e], g[j][b]);
            }
        }
#pragma unroll
        for (int j = 0; j < 9; j++) {
            const int h = lane + 32 * j, cc = h / 9, q = h - 9 * cc, at = cc * 12 + (q / 3) * 4 + q % 3;
#pragma unroll
            for (int b = 0; b < 4; b++) {
                const int ss = 4 * warp + b;
                if (ss < m) R.grad_act[(size_t)(s0 + ss) * REF_GRAD + GRD_Y3 + at] = g[j][b] * dv[j][b];
            }
        }
    }
}

// The input gradient of a valid 3x3 convolution of one sample for input channel
// k: (WO + 2)^2 sums over the WO x WO output gradients of 32 channels dy_cs
// apart at `dy` (rows RS apart), weights [c][tap][k].
template <int WO, int RS>
__device__ __forceinline__ void conv_back_all(float (&g)[WO + 2][WO + 2], const float *dy, int dy_cs, const float *W, int k) {
#pragma unroll 1
    for (int c = 0; c < 32; c++) {
        float w[9];
#pragma unroll
        for (int d = 0; d < 9; d++) w[d] = W[(c * 9 + d) * 32 + k];
#pragma unroll
        for (int r = 0; r < WO; r++) {
            float v[WO > 4 ? 8 : 4];
            ld4(v, dy + c * dy_cs + r * RS);
            if constexpr (WO > 4) ld4(v + 4, dy + c * dy_cs + r * RS + 4);
#pragma unroll
            for (int di = 0; di < 3; di++)
#pragma unroll
                for (int dj = 0; dj < 3; dj++)
#pragma unroll
                    for (int j = 0; j < WO; j++) g[r + di][j + dj] = fmaf(w[di * 3 + dj], v[j], g[r + di][j + dj]);
        }
    }
}

// The convolutions' input gradients times the GELU derivatives: from conv3's
// pre-activation gradients to conv2's and conv1's.  Warps 0-3: conv2 of group
// t - 1, 4-7: conv3 of group t, a warp per sample, a lane per channel; the
// derivatives are loaded ahead of the sums they multiply.
constexpr int BWD_THREADS = 256, DY2_LEN = 32 * 40, DY3_LEN = 32 * 12;
__global__ void __launch_bounds__(BWD_THREADS, 1) k_ref_bwd(RefPlan R, int n) {
    extern __shared__ float4 smem_v[];
    float *W2 = reinterpret_cast<float *>(smem_v);     // [c*9 + tap][k]
    float *W3 = W2 + 9216;
    float *dy2 = W3 + 9216;                            // [2][TR_S][DY2_LEN] by the group's parity
    float *dy3 = dy2 + 2 * TR_S * DY2_LEN;             // [2][TR_S][DY3_LEN]
    float *dy1 = dy3 + 2 * TR_S * DY3_LEN;             // [TR_S][A1_LEN]
    const int tid = threadIdx.x, k = tid & 31, warp = tid >> 5, s = warp & 3, role = warp >> 2;
    const int per = (n + gridDim.x - 1) / gridDim.x;
    const int s_beg = blockIdx.x * per, s_end = min(n, s_beg + per);
    if (s_beg >= s_end) return;
    for (int i = tid; i < 9216 / 4; i += BWD_THREADS) {
        reinterpret_cast<float4 *>(W2)[i] = reinterpret_cast<const float4 *>(R.w2b)[i];
        reinterpret_cast<float4 *>(W3)[i] = reinterpret_cast<const float4 *>(R.w3b)[i];
    }
    const int groups = (s_end - s_beg + TR_S - 1) / TR_S;
    // conv3's warps copy their sample's gradients ahead, a group at a time
    auto fetch = [&](int g) {
        const int at = s_beg + g * TR_S + s;
        if (at < s_end)
#pragma unroll
            for (int q = 0; q < 3; q++)
                cp_async16(dy3 + ((g & 1) * TR_S + s) * DY3_LEN + 4 * (k + 32 * q),
                           R.grad_act + (size_t)at * REF_GRAD + GRD_Y3 + 4 * (k + 32 * q));
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    if (role == 1) fetch(0);
    __syncthreads();
    for (int t = 0; t < groups + 1; t++) {
        const int g = t - (role == 0 ? 1 : 0);
        const int at = s_beg + g * TR_S + s;
        const bool have = g >= 0 && g < groups && at < s_end;
        const float *rec = R.act + (size_t)(have ? at : s_beg) * REF_ACT;
        float *gr = R.grad_act + (size_t)(have ? at : s_beg) * REF_GRAD;
        const int buf = g & 1;
        if (role == 1) {
            fetch(g + 1);
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
            __syncwarp();
            if (have) {
                float d[5][8], a[5][5] = {};
#pragma unroll
                for (int i = 0; i < 5; i++) { ld4(d[i], rec + ACT_D2 + k * 40 + i * 8); ld4(d[i] + 4, rec + ACT_D2 + k * 40 + i * 8 + 4); }
                conv_back_all<3, 4>(a, dy3 + (buf * TR_S + s) * DY3_LEN, 12, W3, k);
                float *out = dy2 + (buf * TR_S + s) * DY2_LEN + k * 40;
#pragma unroll
                for (int i = 0; i < 5; i++) {
                    *reinterpret_cast<float4 *>(out + i * 8) =
                        make_float4(a[i][0] * d[i][0], a[i][1] * d[i][1], a[i][2] * d[i][2], a[i][3] * d[i][3]);
                    *reinterpret_cast<float4 *>(out + i * 8 + 4) = make_float4(a[i][4] * d[i][4], 0.f, 0.f, 0.f);
                }
            }
        } else if (have) {
            float d[7][8], a[7][7] = {};
#pragma unroll
            for (int i = 0; i < 7; i++) { ld4(d[i], rec + ACT_D1 + k * 56 + i * 8); ld4(d[i] + 4, rec + ACT_D1 + k * 56 + i * 8 + 4); }
            conv_back_all<5, 8>(a, dy2 + (buf * TR_S + s) * DY2_LEN, 40, W2, k);
            if (k == 0) bulk_wait_read<0>();           // the sample before has left this warp's rows
            __syncwarp();
            float *out = dy1 + s * A1_LEN + k * A1_CS;
#pragma unroll
            for (int i = 0; i < 7; i++) {
                *reinterpret_cast<float4 *>(out + i * 8) =
                    make_float4(a[i][0] * d[i][0], a[i][1] * d[i][1], a[i][2] * d[i][2], a[i][3] * d[i][3]);
                *reinterpret_cast<float4 *>(out + i * 8 + 4) = make_float4(a[i][4] * d[i][4], a[i][5] * d[i][5], a[i][6] * d[i][6], 0.f);
            }
            fence_bulk();
            __syncwarp();
            if (k == 0) { bulk_out(gr + GRD_Y1, dy1 + s * A1_LEN, A1_LEN * 4); bulk_commit(); }
        }
        if (role == 1) {
            if (k == 0) bulk_wait_read<0>();           // this warp's copy of the step before
            fence_bulk();
        }
        __syncthreads();
        if (role == 1 && k == 0 && have) { bulk_out(gr + GRD_Y2, dy2 + (buf * TR_S + s) * DY2_LEN, DY2_LEN * 4); bulk_commit(); }
    }
    if (k == 0) bulk_wait_all();
}

// ---------------------------------------------------------------- parameter gradients
// Each CTA sums the gradients of its range of samples in registers (the whole
// parameter vector is spread over its 256 threads) and writes one partial
// vector; k_ref_reduce adds the partials in a fixed order (no atomics,
// reproducible).  Per sample a thread of warps 0-3 takes 8 x 1 channel pairs
// of conv2 (9 taps each), of warps 4-7 the same of conv3, and every thread an
// 8 x 9 tile of the dense layer; the next sample's record is copied to shared
// memory meanwhile.
constexpr int WG_THREADS = 256;
// one sample's staged operands (floats): activations, then gradients, then the input
constexpr int WS_A2 = A1_LEN, WS_A3 = WS_A2 + A2_LEN, WS_G1 = WS_A3 + 288, WS_GRD = WS_G1 + 64,
              WS_X = WS_GRD + REF_GRAD, WS_LEN = WS_X + 84;

template <int WO, int IN_CS, int DY_CS, int RS>
__device__ __forceinline__ void wgrad_tile(float (&acc)[8][9], const float *dy, const float *a) {
#pragma unroll 1
    for (int r = 0; r < WO; r++) {
        float x[3][8];
#pragma unroll
        for (int di = 0; di < 3; di++) { ld4(x[di], a + (r + di) * 8); ld4(x[di] + 4, a + (r + di) * 8 + 4); }
#pragma unroll
        for (int c = 0; c < 8; c++) {
            float v[8];
            ld4(v, dy + c * DY_CS + r * RS);
            if constexpr (WO > 4) ld4(v + 4, dy + c * DY_CS + r * RS + 4);
#pragma unroll
            for (int j = 0; j < WO; j++)
#pragma unroll
                for (int d = 0; d < 9; d++) acc[c][d] = fmaf(v[j], x[d / 3][j + d % 3], acc[c][d]);
        }
    }
}

__global__ void __launch_bounds__(WG_THREADS, 1) k_ref_wgrad(RefPlan R, const float *__restrict__ feat, int n) {
    extern __shared__ float4 smem_v[];
    float *buf = reinterpret_cast<float *>(smem_v);    // [2][WS_LEN]
    __shared__ float fold[8][32][10];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int per = (n + gridDim.x - 1) / gridDim.x;
    const int s_beg = blockIdx.x * per, s_end = min(n, s_beg + per);
    auto stage = [&](int s, float *d) {
        const float *rec = R.act + (size_t)s * REF_ACT, *gr = R.grad_act + (size_t)s * REF_GRAD;
        for (int i = tid; i < A1_LEN / 4; i += WG_THREADS) cp_async16(d + 4 * i, rec + ACT_A1 + 4 * i);
        for (int i = tid; i < A2_LEN / 4; i += WG_THREADS) cp_async16(d + WS_A2 + 4 * i, rec + ACT_A2 + 4 * i);
        for (int i = tid; i < 288 / 4; i += WG_THREADS) cp_async16(d + WS_A3 + 4 * i, rec + ACT_A3 + 4 * i);
        for (int i = tid; i < 64 / 4; i += WG_THREADS) cp_async16(d + WS_G1 + 4 * i, rec + ACT_G1 + 4 * i);
        for (int i = tid; i < REF_GRAD / 4; i += WG_THREADS) cp_async16(d + WS_GRD + 4 * i, gr + 4 * i);
        if (tid < 81) {
            const unsigned dst = (unsigned)__cvta_generic_to_shared(d + WS_X + tid);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(dst), "l"(feat + (size_t)s * 81 + tid) : "memory");
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    float acc[8][9], af[8][9], aw[9], ab1 = 0.f, ab2 = 0.f, ab3 = 0.f, ac = 0.f, af2 = 0.f;
#pragma unroll
    for (int c = 0; c < 8; c++)
#pragma unroll
        for (int d = 0; d < 9; d++) { acc[c][d] = 0.f; af[c][d] = 0.f; }
#pragma unroll
    for (int d = 0; d < 9; d++) aw[d] = 0.f;
    if (s_beg < s_end) stage(s_beg, buf);
    for (int s = s_beg; s < s_end; s++) {
        const float *b = buf + ((s - s_beg) & 1) * WS_LEN;
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();                               // staged for all, and the other buffer is read
        if (s + 1 < s_end) stage(s + 1, buf + ((s + 1 - s_beg) & 1) * WS_LEN);
        const float *g = b + WS_GRD;
        if (warp < 4) wgrad_tile<5, A1_CS, 40, 8>(acc, g + GRD_Y2 + warp * 8 * 40, b + lane * A1_CS);
        else wgrad_tile<3, A2_CS, 12, 4>(acc, g + GRD_Y3 + (warp - 4) * 8 * 12, b + WS_A2 + lane * A2_CS);
        {   // dense: outputs 8 warp .. 8 warp + 7, inputs 9 lane .. 9 lane + 8
            float z[8], x[9];
            ld4(z, g + GRD_Z + 8 * warp);
            ld4(z + 4, g + GRD_Z + 8 * warp + 4);
#pragma unroll
            for (int e = 0; e < 9; e++) x[e] = b[WS_A3 + 9 * lane + e];
#pragma unroll
            for (int o = 0; o < 8; o++)
#pragma unroll
                for (int e = 0; e < 9; e++) af[o][e] = fmaf(z[o], x[e], af[o][e]);
        }
        if (warp < 7) {                                // conv1 and its bias: channel lane, output row warp
            float v[8];
            ld4(v, g + GRD_Y1 + lane * A1_CS + warp * 8);
            ld4(v + 4, g + GRD_Y1 + lane * A1_CS + warp * 8 + 4);
#pragma unroll
            for (int di = 0; di < 3; di++) {
                float x[9];
#pragma unroll
                for (int e = 0; e < 9; e++) x[e] = b[WS_X + (warp + di) * 9 + e];
#pragma unroll
                for (int dj = 0; dj < 3; dj++)
#pragma unroll
                    for (int j = 0; j < 7; j++) aw[di * 3 + dj] = fmaf(v[j], x[j + dj], aw[di * 3 + dj]);
            }
#pragma unroll
            for (int j = 0; j < 7; j++) ab1 += v[j];
        }
        if (warp < 5) {
            const float *y = g + GRD_Y2 + lane * 40 + warp * 8;
            ab2 += ((y[0] + y[1]) + (y[2] + y[3])) + y[4];
        } else {
            const float *y = g + GRD_Y3 + lane * 12 + (warp - 5) * 4;
            ab3 += (y[0] + y[1]) + y[2];
        }
        if (tid < 64) ac += g[GRD_Z + tid];
        if (tid < 192) af2 = fmaf(g[GRD_OUT + tid / 64], b[WS_G1 + (tid & 63)], af2);
        else if (tid < 195) af2 += g[GRD_OUT + tid - 192];
    }
    float *o = R.part + (size_t)blockIdx.x * RP_N;
    {
        const int base = warp < 4 ? RP_W2 : RP_W3, c0 = (warp & 3) * 8;
#pragma unroll
        for (int c = 0; c < 8; c++)
#pragma unroll
            for (int d = 0; d < 9; d++) o[base + (c0 + c) * 288 + lane * 9 + d] = acc[c][d];
#pragma unroll
        for (int c = 0; c < 8; c++)
#pragma unroll
            for (int d = 0; d < 9; d++) o[RP_F1 + (8 * warp + c) * 288 + 9 * lane + d] = af[c][d];
    }
#pragma unroll
    for (int d = 0; d < 9; d++) fold[warp][lane][d] = aw[d];
    fold[warp][lane][9] = ab1;
    __syncthreads();
    for (int i = tid; i < 320; i += WG_THREADS) {      // conv1's rows folded
        const int cc = i / 10, d = i - 10 * cc;
        float t = 0.f;
        for (int w = 0; w < 7; w++) t += fold[w][cc][d];
        o[d < 9 ? RP_W1 + cc * 9 + d : RP_B1 + cc] = t;
    }
    __syncthreads();
    fold[warp][lane][0] = warp < 5 ? ab2 : ab3;
    __syncthreads();
    if (tid < 32) {
        float t = 0.f;
        for (int w = 0; w < 5; w++) t += fold[w][tid][0];
        o[RP_B2 + tid] = t;
        o[RP_B3 + tid] = (fold[5][tid][0] + fold[6][tid][0]) + fold[7][tid][0];
    }
    if (tid < 64) o[RP_C1 + tid] = ac;
    if (tid < 195) o[RP_F2 + tid] = af2;               // F2, then c2
}

// The partial vectors summed: 64 parameters per CTA, four threads each taking
// every fourth partial.
__global__ void __launch_bounds__(256) k_ref_reduce(RefPlan R, int parts) {
    __shared__ float sh[4][64];
    const int e = threadIdx.x & 63, q = threadIdx.x >> 6, i = blockIdx.x * 64 + e;
    float t = 0.f;
    if (i < RP_N) {
#pragma unroll 8
        for (int p = q; p < parts; p += 4) t += R.part[(size_t)p * RP_N + i];
    }
    sh[q][e] = t;
    __syncthreads();
    if (q == 0 && i < RP_N) R.grad[i] = (sh[0][e] + sh[1][e]) + (sh[2][e] + sh[3][e]);
}

// ---------------------------------------------------------------- Adam + derived copies
__global__ void k_ref_adam(RefPlan R, float lr, float b1, float b2, float eps, float c1, float c2) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < RP_N; i += gridDim.x * blockDim.x) {
        const float gi = R.grad[i];
        const float m = b1 * R.m[i] + (1.f - b1) * gi;
        const float v = b2 * R.v[i] + (1.f - b2) * gi * gi;
        R.m[i] = m;
        R.v[i] = v;
        R.theta[i] = R.theta[i] - lr * (m / c1) / (sqrtf(v / c2) + eps);
    }
}

// transposed FP32 copies for the training forward and BF16 copies for inference
__global__ void k_ref_derive(RefPlan R) {
    __nv_bfloat16 *wb = reinterpret_cast<__nv_bfloat16 *>(R.wpack);
    float *ws = reinterpret_cast<float *>(R.wpack + INF_ROWS * INF_KS * 2);
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < INF_ROWS * INF_KS; e += gridDim.x * blockDim.x) {
        const int n = e / INF_KS, kk = e % INF_KS;
        float v = 0.f;
        if (kk < 288) {
            const int hi = kk >> 5, lo = kk & 31;        // tap (or dense input position), input channel
            const int base = (n < 32) ? RP_W2 + n * 288 : (n < 64) ? RP_W3 + (n - 32) * 288 : RP_F1 + (n - 64) * 288;
            v = R.theta[base + lo * 9 + hi];
        }
        wb[e] = __float2bfloat16_rn(v);
    }
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < INF_SMALL; e += gridDim.x * blockDim.x) {
        float v = 0.f;
        if (e < 288) v = R.theta[RP_W1 + e];
        else if (e < 320) v = R.theta[RP_B1 + e - 288];
        else if (e < 352) v = R.theta[RP_B2 + e - 320];
        else if (e < 384) v = R.theta[RP_B3 + e - 352];
        else if (e < 448) v = R.theta[RP_C1 + e - 384];
        else if (e < 643) v = R.theta[RP_F2 + e - 448];       // F2 (192) then c2 (3)
        ws[e] = v;
    }
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < RP_N; i += gridDim.x * blockDim.x) {
        const float t = R.theta[i];
        if (i >= RP_W2 && i < RP_W2 + 9216) { const int e = i - RP_W2, c = e / 288, kk = e % 288; R.w2t[kk * 32 + c] = t; R.w2b[(c * 9 + kk % 9) * 32 + kk / 9] = t; }
        if (i >= RP_W3 && i < RP_W3 + 9216) { const int e = i - RP_W3, c = e / 288, kk = e % 288; R.w3t[kk * 32 + c] = t; R.w3b[(c * 9 + kk % 9) * 32 + kk / 9] = t; }
        if (i >= RP_F1 && i < RP_F1 + 18432) { const int e = i - RP_F1, o = e / 288, h = e % 288; R.f1t[h * 64 + o] = t; }
    }
}

// ---------------------------------------------------------------- inference, BF16 tensor cores
// mma.sync m16n8k16 row.col bf16 -> f32.  Fragment layout (PTX ISA): with
// g = lane/4, t = lane%4, A regs {a0: (g, 2t..2t+1), a1: (g+8, 2t..), a2: (g, 2t+8..),
// a3: (g+8, 2t+8..)}, B regs {b0: (k=2t..2t+1, n=g), b1: (k=2t+8.., n=g)},
// C {c0,c1: (g, 2t..2t+1), c2,c3: (g+8, 2t..2t+1)}.
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Per-CTA shared memory of the inference kernel after the parameter pack:
// the window's input (81 f32, padded to 84) and its activations, channel-last
// with a padded channel stride INF_CS (conv1 out 7x7, conv2 out 5x5, conv3
// out 3x3, BF16), then the dense layer's 64 outputs (f32).
constexpr int INF_CS = 40;
constexpr int INF_ACT_BYTES = 84 * 4 + (49 + 25 + 9) * INF_CS * 2 + 64 * 4;
constexpr int INF_GROUPS = 2;      // windows per CTA at a time (four warps each)

// One warp's share of a convolution or dense layer as m16n8k16 tiles: rows are
// output positions (mt: 16-row tile), columns output channels (n-tiles nt0,
// nt0 + 1), K = 288 walked tap by tap (k' = 32 tap + c_in).  a_row(m) is the
// BF16 activation row of output position m's tap-0 input (nullptr: padding
// row), step(tap) the offset of tap's input row from it; B rows are INF_KS apart.
template <class ARow, class Step>
__device__ __forceinline__ void warp_gemm_288(float (&acc)[2][4], ARow a_row, Step step, const __nv_bfloat16 *B,
                                              int mt, int nt0, int lane) {
    const int g = lane >> 2, t = lane & 3;
    const __nv_bfloat16 *r0 = a_row(mt * 16 + g), *r1 = a_row(mt * 16 + g + 8);
    const __nv_bfloat16 *b0p = B + (size_t)(nt0 * 8 + g) * INF_KS + 2 * t;
    const __nv_bfloat16 *b1p = b0p + 8 * INF_KS;
#pragma unroll 3
    for (int ks = 0; ks < 18; ks++) {
        const int off = step(ks >> 1) + (ks & 1) * 16 + 2 * t;
        uint32_t a[4];
        a[0] = r0 ? *reinterpret_cast<const uint32_t *>(r0 + off) : 0u;
        a[1] = r1 ? *reinterpret_cast<const uint32_t *>(r1 + off) : 0u;
        a[2] = r0 ? *reinterpret_cast<const uint32_t *>(r0 + off + 8) : 0u;
        a[3] = r1 ? *reinterpret_cast<const uint32_t *>(r1 + off + 8) : 0u;
        const int k0 = ks * 16;
        mma_bf16(acc[0], a, *reinterpret_cast<const uint32_t *>(b0p + k0), *reinterpret_cast<const uint32_t *>(b0p + k0 + 8));
        mma_bf16(acc[1], a, *reinterpret_cast<const uint32_t *>(b1p + k0), *reinterpret_cast<const uint32_t *>(b1p + k0 + 8));
    }
}

// A CTA of four warps per window at a time (grid-stride over the windows):
// conv1 on the SIMT pipes in FP32 (K = 9), conv2, conv3 and the dense
// 288 -> 64 layer as tensor-core tiles with bias + GELU applied to the
// accumulators, the 64 -> 3 layer as warp dot products.  With the
// activations channel-last, each A-fragment element pair is one 32-bit load.
// the decision of RefDecide for window w: r3 = (fx, fy, s), f its 9x9 neighbourhood
__device__ static void ref_decide(const RefDecide &D, int w, const float *r3, const float *f) {
    const float fx = r3[0], fy = r3[1], sg = expf(0.5f * r3[2]);
    auto vertex = [](float a, float b, float c) {
        const float den = a - 2.f * b + c;
        return (den < 0.f) ? 0.5f * (a - c) / den : 0.f;
    };
    const float px = vertex(f[4 * 9 + 3], f[4 * 9 + 4], f[4 * 9 + 5]);
    const float py = vertex(f[3 * 9 + 4], f[4 * 9 + 4], f[5 * 9 + 4]);
    const bool ok = (sg < D.max_sigma) && fabsf(fx - px) < D.max_dis && fabsf(fy - py) < D.max_dis &&
                    isfinite(fx) && isfinite(fy) && f[4 * 9 + 4] > 0.f;
    D.skip[w] = ok ? 1 : 0;
    if (ok) {
        xcg_result &o = D.res[w];
        o.xfrac = fx;
        o.yfrac = fy;
        o.fip = -1;
        o.fjp = -1;
        o.flags |= XCG_FLAG_REFINED;
    }
}

__global__ void __launch_bounds__(128 * INF_GROUPS) k_ref_infer(RefPlan R, const float *__restrict__ feat,
                                                                 float *__restrict__ out, int n, RefDecide D) {
    extern __shared__ __align__(16) unsigned char smc[];
    const __nv_bfloat16 *B2 = reinterpret_cast<const __nv_bfloat16 *>(smc);    // [32][INF_KS]
    const __nv_bfloat16 *B3 = B2 + 32 * INF_KS;
    const __nv_bfloat16 *BF = B3 + 32 * INF_KS;                                 // [64][INF_KS]
    const float *small = reinterpret_cast<const float *>(smc + INF_ROWS * INF_KS * 2);
    // one group of four warps per window; each group has its own activations
    const int grp = threadIdx.x >> 7, gt = threadIdx.x & 127;
    float *x0 = reinterpret_cast<float *>(smc + INF_PACK_BYTES + (size_t)grp * INF_ACT_BYTES);   // [84]
    __nv_bfloat16 *a1 = reinterpret_cast<__nv_bfloat16 *>(x0 + 84);             // [49][INF_CS]
    __nv_bfloat16 *a2 = a1 + 49 * INF_CS;                                       // [25][INF_CS]
    __nv_bfloat16 *a3 = a2 + 25 * INF_CS;                                       // [9][INF_CS]
    float *g1 = reinterpret_cast<float *>(a3 + 9 * INF_CS);                     // [64]
    const float *W1 = small, *b1 = small + 288, *b2 = small + 320, *b3 = small + 352, *c1 = small + 384;
    const float *F2 = small + 448, *c2 = small + 448 + 192;

    // the parameter pack, 16 bytes per copy (no waits on flags: cp.async groups)
    for (int i = threadIdx.x; i < INF_PACK_BYTES / 16; i += blockDim.x) cp_async16(smc + 16 * i, R.wpack + 16 * i);
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();

    const int warp = gt >> 5, lane = threadIdx.x & 31;      // warp within the group
    const int g = lane >> 2, t = lane & 3;
    // the groups of a CTA take windows base + grp; barriers stay CTA-wide, so
    // a group without a window in the last round still takes part in them
    for (int base = blockIdx.x * INF_GROUPS; base < n; base += gridDim.x * INF_GROUPS) {
        const int w = base + grp;
        const bool have = w < n;
        if (gt < 81) x0[gt] = have ? feat[(size_t)w * 81 + gt] : 0.f;
        __syncthreads();
        // conv1 (FP32): lane = output channel, warps take positions in turn
        for (int p = warp; p < 49; p += 4) {
            const int i = p / 7, j = p % 7;
            float y = b1[lane];
#pragma unroll
            for (int d = 0; d < 9; d++) y = fmaf(W1[lane * 9 + d], x0[(i + d / 3) * 9 + j + d % 3], y);
            a1[p * INF_CS + lane] = __float2bfloat16_rn(gelu_f(y));
        }
        __syncthreads();
        // conv2: 25 positions (2 row tiles) x 32 channels (4 n-tiles); warp: tile mt = warp/2, n-tiles 2 (warp%2) +0/1
        {
            float acc[2][4] = {};
            auto row = [&](int m) -> const __nv_bfloat16 * {
                return (m < 25) ? a1 + ((m / 5) * 7 + m % 5) * INF_CS : nullptr;
            };
            auto step = [&](int tap) { return ((tap / 3) * 7 + tap % 3) * INF_CS; };
            const int mt = warp >> 1, nt0 = 2 * (warp & 1);
            warp_gemm_288(acc, row, step, B2, mt, nt0, lane);
#pragma unroll
            for (int q = 0; q < 2; q++)
#pragma unroll
                for (int h = 0; h < 4; h++) {
                    const int m = mt * 16 + g + (h >> 1) * 8, ch = (nt0 + q) * 8 + 2 * t + (h & 1);
                    if (m < 25) a2[m * INF_CS + ch] = __float2bfloat16_rn(gelu_f(acc[q][h] + b2[ch]));
                }
        }
        __syncthreads();
        // conv3: 9 positions (1 row tile) x 32 channels; warps 0, 1 take two n-tiles each
        if (warp < 2) {
            float acc[2][4] = {};
            auto row = [&](int m) -> const __nv_bfloat16 * {
                return (m < 9) ? a2 + ((m / 3) * 5 + m % 3) * INF_CS : nullptr;
            };
            auto step = [&](int tap) { return ((tap / 3) * 5 + tap % 3) * INF_CS; };
            const int nt0 = 2 * warp;
            warp_gemm_288(acc, row, step, B3, 0, nt0, lane);
#pragma unroll
            for (int q = 0; q < 2; q++)
#pragma unroll
                for (int h = 0; h < 4; h++) {
                    const int m = g + (h >> 1) * 8, ch = (nt0 + q) * 8 + 2 * t + (h & 1);
                    if (m < 9) a3[m * INF_CS + ch] = __float2bfloat16_rn(gelu_f(acc[q][h] + b3[ch]));
                }
        }
        __syncthreads();
        // dense 288 -> 64: one row (this window), k' = 32 position + channel; warp: n-tiles 2 warp +0/1
        {
            float acc[2][4] = {};
            auto row = [&](int m) -> const __nv_bfloat16 * { return (m == 0) ? a3 : nullptr; };
            auto step = [&](int pos) { return pos * INF_CS; };
            const int nt0 = 2 * warp;
            warp_gemm_288(acc, row, step, BF, 0, nt0, lane);
            if (g == 0)
#pragma unroll
                for (int q = 0; q < 2; q++)
#pragma unroll
                    for (int h = 0; h < 2; h++) {
                        const int o = (nt0 + q) * 8 + 2 * t + h;
                        g1[o] = gelu_f(acc[q][h] + c1[o]);
                    }
        }
        __syncthreads();
        // 64 -> 3, then the decision (x0 still holds the neighbourhood)
        if (warp == 0 && have) {
            float r3[3];
#pragma unroll
            for (int o = 0; o < 3; o++) {
                float v = fmaf(F2[o * 64 + lane], g1[lane], F2[o * 64 + 32 + lane] * g1[32 + lane]);
#pragma unroll
                for (int s = 16; s > 0; s >>= 1) v += __shfl_xor_sync(0xffffffffu, v, s);
                r3[o] = v + c2[o];
                if (lane == 0) out[(size_t)w * 3 + o] = r3[o];
            }
            if (D.skip && lane == 0) ref_decide(D, w, r3, x0);
        }
        __syncthreads();                           // x0 .. g1 are reused by the next window
    }
}

size_t ref_fwd_smem() { return (size_t)(2 * 9216 + TR_S * (2 * (A1_LEN + A2_LEN) + X0_S)) * sizeof(float); }
size_t ref_dense_smem() { return (size_t)(288 * F1_S + DN_S * (A3_SS + 2 * Z_S + 4) + 192) * sizeof(float); }
size_t ref_bwd_smem() { return (size_t)(2 * 9216 + TR_S * (2 * (DY2_LEN + DY3_LEN) + A1_LEN)) * sizeof(float); }
size_t ref_wgrad_smem() { return (size_t)2 * WS_LEN * sizeof(float); }
size_t ref_infer_smem() { return (size_t)INF_PACK_BYTES + (size_t)INF_GROUPS * INF_ACT_BYTES; }

cudaError_t ref_setup() {
    cudaError_t e = cudaFuncSetAttribute(k_ref_fwd<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ref_fwd_smem());
    if (!e) e = cudaFuncSetAttribute(k_ref_fwd<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ref_fwd_smem());
    if (!e) e = cudaFuncSetAttribute(k_ref_dense<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ref_dense_smem());
    if (!e) e = cudaFuncSetAttribute(k_ref_dense<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ref_dense_smem());
    if (!e) e = cudaFuncSetAttribute(k_ref_bwd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ref_bwd_smem());
    if (!e) e = cudaFuncSetAttribute(k_ref_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ref_wgrad_smem());
    if (!e) e = cudaFuncSetAttribute(k_ref_infer, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)ref_infer_smem());
    return e;
}

// CTAs of the forward and backward kernels: a group of four samples each
// until every SM has one, then longer ranges
static int train_grid(int n) { return std::min((n + TR_S - 1) / TR_S, REF_SMS); }
void ref_launch_fwd(const RefPlan &R, const float *feat, const float *target, int n, cudaStream_t s) {
    const int dense = (n + DN_S - 1) / DN_S;
    if (target) {
        k_ref_fwd<true><<<train_grid(n), FWD_THREADS, ref_fwd_smem(), s>>>(R, feat, n);
        k_ref_dense<true><<<dense, DN_THREADS, ref_dense_smem(), s>>>(R, target, n);
    } else {
        k_ref_fwd<false><<<train_grid(n), FWD_THREADS, ref_fwd_smem(), s>>>(R, feat, n);
        k_ref_dense<false><<<dense, DN_THREADS, ref_dense_smem(), s>>>(R, nullptr, n);
    }
}
void ref_launch_bwd(const RefPlan &R, int n, cudaStream_t s) {
    k_ref_bwd<<<train_grid(n), BWD_THREADS, ref_bwd_smem(), s>>>(R, n);
}
// partial gradient vectors of a batch of n: at least four samples each, one per SM at most
int ref_wgrad_parts(int n) { return std::min((n + 3) / 4, REF_SMS); }
void ref_launch_wgrad(const RefPlan &R, const float *feat, int n, cudaStream_t s) {
    const int parts = ref_wgrad_parts(n);
    k_ref_wgrad<<<parts, WG_THREADS, ref_wgrad_smem(), s>>>(R, feat, n);
    k_ref_reduce<<<(RP_N + 63) / 64, 256, 0, s>>>(R, parts);
}
void ref_launch_adam(const RefPlan &R, float lr, int step, cudaStream_t s) {
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - powf(b1, (float)step), c2 = 1.f - powf(b2, (float)step);
    k_ref_adam<<<(RP_N + 255) / 256, 256, 0, s>>>(R, lr, b1, b2, 1e-8f, c1, c2);
}
void ref_launch_derive(const RefPlan &R, cudaStream_t s) { k_ref_derive<<<(RP_N + 255) / 256, 256, 0, s>>>(R); }
void ref_launch_infer(const RefPlan &R, const float *feat, float *out, int n, cudaStream_t s, const RefDecide *D) {
    // INF_GROUPS windows per CTA at a time, two CTAs per SM (91 KB of shared memory each)
    const int need = (n + INF_GROUPS - 1) / INF_GROUPS;
    const int blocks = need < 2 * 152 ? need : 2 * 152;
    const RefDecide none{nullptr, nullptr, 0.f, 0.f};
    k_ref_infer<<<blocks > 0 ? blocks : 1, 128 * INF_GROUPS, ref_infer_smem(), s>>>(R, feat, out, n, D ? *D : none);
}

}  // namespace xcg
