// Element-wise stages of the AUSSM block around the scan operator, in the
// scan's own (batch, channel, time) layout, so that the block needs no
// transposing copies and no separate bias / activation passes:
//
//   causal depthwise convolution + bias   u[b][i][t] = bias[i] + sum_k w[i][k] xs[b][i][t - (K-1) + k]
//       (the reference transposes to (b, d, l), calls nn.Conv1d with padding K-1, cuts the result back to l
//        steps and transposes again: ai-modules/wavesAI/model/aussm.py:858-864)
//   step size                             dt[b][i][t] = softplus(pre[b][i][t] + scale * bias[i])
//       (the reference adds dt_proj's bias a second time and applies softplus as two passes, aussm.py:878-880)
//
// and their adjoints.  All four are streaming kernels: one pass over the rows, 128-bit accesses where the rows
// are 16-byte aligned.  Sums over batch and time (weight and bias gradients) are two-stage and deterministic:
// one block per (batch entry, channel) row leaves its partial sums, a second kernel adds them over the batch.
#include <cuda_runtime.h>
#include <stdint.h>

#include <algorithm>

#include "../../include/aussm_b200.h"
#include "common.cuh"
#include "host_common.cuh"

namespace aussm {
namespace {

constexpr int KMAX = AUSSM_MAX_CONV_TAPS;
constexpr int ROW_THREADS = 256;

// How a streaming kernel walks (rows, L): a row belongs to 32 to 256 threads (as many as it has quads), several short
// rows share a block, and a long row is cut into chunks when there are too few rows to fill the GPU.  Threads take
// whole quads, 128-bit where the rows are 16-byte aligned.
constexpr int MAX_CHUNKS = 16;
struct RowPlan {
    long long rows;
    int L, quads, vec;
    int tpr;                 // threads per row (32, 64, 128, 256)
    int chunks, qpc;         // chunks per row and quads per chunk (1 chunk when several rows share a block)
    unsigned blocks;
};
inline int row_chunks_max(long long rows) { return rows < 148 * 16 ? MAX_CHUNKS : 1; }
RowPlan row_plan(long long rows, int L, bool vec) {
    RowPlan p;
    p.rows = rows;
    p.L = L;
    p.quads = (int)(((long long)L + 3) / 4);
    p.vec = vec ? 1 : 0;
    p.tpr = 32;
    while (p.tpr < ROW_THREADS && p.tpr < p.quads) p.tpr *= 2;
    p.chunks = p.tpr < ROW_THREADS ? 1 : std::max(1, std::min(row_chunks_max(rows), p.quads / (2 * ROW_THREADS)));
    p.qpc = (p.quads + p.chunks - 1) / p.chunks;
    const long long rpb = ROW_THREADS / p.tpr;
    p.blocks = (unsigned)((rows + rpb - 1) / rpb * p.chunks);
    return p;
}
struct RowSlot {
    long long row;
    int chunk, lane;         // lane: thread of the row
    int q0, q1;              // its first quad, end of the chunk (empty for a row that does not exist)
    __device__ __forceinline__ explicit RowSlot(const RowPlan& p) {
        chunk = (int)(blockIdx.x % (unsigned)p.chunks);
        row = (long long)(blockIdx.x / (unsigned)p.chunks) * (ROW_THREADS / p.tpr) + threadIdx.x / p.tpr;
        lane = threadIdx.x % p.tpr;
        q0 = chunk * p.qpc + lane;
        q1 = row < p.rows ? min(p.quads, (chunk + 1) * p.qpc) : 0;
    }
};

// quad t .. t+3 of a row (t a multiple of 4), zero outside [0, L)
__device__ __forceinline__ void load_quad(const float* row, int t, int L, int vec, float* v) {
    if (t < 0 || t >= L) {
        v[0] = v[1] = v[2] = v[3] = 0.f;
    } else if (vec) {
        const float4 f = *reinterpret_cast<const float4*>(row + t);
        v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
    } else {
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = t + e < L ? row[t + e] : 0.f;
    }
}
__device__ __forceinline__ void store_quad(float* row, int t, int L, int vec, const float* v) {
    if (vec) {
        *reinterpret_cast<float4*>(row + t) = make_float4(v[0], v[1], v[2], v[3]);
    } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (t + e < L) row[t + e] = v[e];
    }
}

// Sums of n values over the threads of a row, in a fixed order; thread k < n of the row gets value k.
template <int n>
__device__ __forceinline__ float row_sums(float (&acc)[n], const RowPlan& p, const RowSlot& s) {
    __shared__ float red[ROW_THREADS / 32][n];
#pragma unroll
    for (int k = 0; k < n; ++k) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
        if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5][k] = acc[k];
    }
    __syncthreads();
    float sum = 0.f;
    if (s.lane < n) {
        const int first = (threadIdx.x - s.lane) >> 5;
        for (int w = 0; w < p.tpr / 32; ++w) sum += red[first + w][s.lane];
    }
    return sum;
}

// The filter right-aligned in a window of KMAX taps: u[t] = sum_m w[m] x[t - (KMAX-1) + m], m >= KMAX - K.
struct Taps {
    float w[KMAX];
};

__device__ __forceinline__ Taps load_taps(const float* w, int i, int K) {
    Taps t;
#pragma unroll
    for (int m = 0; m < KMAX; ++m) t.w[m] = m >= KMAX - K ? w[(long long)i * K + m - (KMAX - K)] : 0.f;
    return t;
}
static_assert(KMAX == 4, "a quad's window is the quad and its neighbour");

// ---- forward: u = conv(xs) + bias -------------------------------------------------------------
__global__ void __launch_bounds__(ROW_THREADS) conv_pre_fwd_kernel(const float* __restrict__ xs, const float* __restrict__ w,
                                                                   const float* __restrict__ bias, float* __restrict__ u,
                                                                   int D, int K, const RowPlan p) {
    const RowSlot s(p);
    if (s.q0 >= s.q1) return;
    const int i = (int)(s.row % D);
    const float* x = xs + s.row * p.L;
    const Taps tp = load_taps(w, i, K);
    const float bv = bias ? bias[i] : 0.f;
    for (int q = s.q0; q < s.q1; q += p.tpr) {
        float win[8], out[4];                                   // x[t0 - 4 .. t0 + 3]
        load_quad(x, 4 * q - 4, p.L, p.vec, win);
        load_quad(x, 4 * q, p.L, p.vec, win + 4);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            out[e] = bv;
#pragma unroll
            for (int m = 0; m < KMAX; ++m)
                if (m >= KMAX - K) out[e] = fmaf(tp.w[m], win[1 + e + m], out[e]);
        }
        store_quad(u + s.row * p.L, 4 * q, p.L, p.vec, out);
    }
}

// ---- backward: dxs = conv^T(du); per-row partial sums of dw and dbias ---------------------------
// partial[(row * chunks + chunk) * (KMAX + 1) + m] = sum_t du[t] xs[t - (KMAX-1) + m], [KMAX] = sum_t du[t].  Bound by HBM
// (12 bytes a step): B1 D512 L65536 231 us with one block per row and scalar loads, 101 us now (4.0 TB/s).
__global__ void __launch_bounds__(ROW_THREADS) conv_pre_bwd_kernel(const float* __restrict__ du,
                                                                   const float* __restrict__ xs,
                                                                   const float* __restrict__ w,
                                                                   float* __restrict__ dxs,
                                                                   float* __restrict__ partial, int D, int K,
                                                                   const RowPlan p) {
    const RowSlot s(p);
    const float* g = du + s.row * p.L;
    const float* x = xs + s.row * p.L;
    float acc[KMAX + 1];
#pragma unroll
    for (int k = 0; k <= KMAX; ++k) acc[k] = 0.f;
    if (s.q0 < s.q1) {
        const Taps tp = load_taps(w, (int)(s.row % D), K);
        for (int q = s.q0; q < s.q1; q += p.tpr) {
            float xw[8], gw[8], d[4];                           // x[t0 - 4 .. t0 + 3], du[t0 .. t0 + 7]
            load_quad(x, 4 * q - 4, p.L, p.vec, xw);
            load_quad(x, 4 * q, p.L, p.vec, xw + 4);
            load_quad(g, 4 * q, p.L, p.vec, gw);
            load_quad(g, 4 * q + 4, p.L, p.vec, gw + 4);
            const bool inner = q > 0 && 4 * q + 7 < p.L;        // no term outside the row (nor a product with its zero)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int t = 4 * q + e;
                d[e] = 0.f;
#pragma unroll
                for (int m = 0; m < KMAX; ++m) {
                    if (m >= KMAX - K) {                        // dxs[t] = sum_m w[m] du[t + (KMAX-1) - m]
                        if (inner || t + (KMAX - 1) - m < p.L) d[e] = fmaf(tp.w[m], gw[e + (KMAX - 1) - m], d[e]);
                        if (inner || (t - (KMAX - 1) + m >= 0 && t < p.L)) acc[m] = fmaf(gw[e], xw[1 + e + m], acc[m]);
                    }
                }
                acc[KMAX] += gw[e];
            }
            store_quad(dxs + s.row * p.L, 4 * q, p.L, p.vec, d);
        }
    }
    const float sum = row_sums(acc, p, s);
    if (s.row < p.rows && s.lane <= KMAX) partial[(s.row * p.chunks + s.chunk) * (KMAX + 1) + s.lane] = sum;
}

// dw[i][k] and dbias[i] = sums of the partials over batch entries and chunks, in a fixed order
__global__ void __launch_bounds__(256) conv_pre_reduce_kernel(const float* __restrict__ partial, float* __restrict__ dw,
                                                              float* __restrict__ dbias, int B, int D, int K,
                                                              int chunks) {
    const int o = blockIdx.x * 256 + threadIdx.x;
    if (o >= D * (K + 1)) return;
    const int i = o / (K + 1), k = o % (K + 1);
    const int slot = k < K ? KMAX - K + k : KMAX;
    float s = 0.f;
    for (int b = 0; b < B; ++b)
        for (int c = 0; c < chunks; ++c) s += partial[(((long long)b * D + i) * chunks + c) * (KMAX + 1) + slot];
    if (k < K) dw[(long long)i * K + k] = s;
    else if (dbias) dbias[i] = s;
}

// ---- step size: dt = softplus(pre + scale * bias) ---------------------------------------------------
// torch.nn.functional.softplus with its defaults (beta 1, threshold 20): x above 20 passes through
__device__ __forceinline__ float softplus_(float x) { return x > 20.f ? x : log1pf(__expf(x)); }

__global__ void __launch_bounds__(ROW_THREADS) softplus_bias_fwd_kernel(const float* __restrict__ pre,
                                                                        const float* __restrict__ bias, float scale,
                                                                        float* __restrict__ dt, int D, const RowPlan p) {
    const RowSlot s(p);
    if (s.q0 >= s.q1) return;
    const float bv = bias ? scale * bias[s.row % D] : 0.f;
    for (int q = s.q0; q < s.q1; q += p.tpr) {
        float v[4];
        load_quad(pre + s.row * p.L, 4 * q, p.L, p.vec, v);
#pragma unroll
        for (int e = 0; e < 4; ++e) v[e] = softplus_(v[e] + bv);
        store_quad(dt + s.row * p.L, 4 * q, p.L, p.vec, v);
    }
}

// dpre = ddt * sigmoid(pre + scale bias), with sigmoid recovered from the output: 1 - exp(-dt) (exact also
// above the threshold, where the forward passed x through and sigmoid(x) = 1 to float32 accuracy; expm1
// keeps the relative accuracy for very negative arguments, where dt is tiny);
// partial[row * chunks + chunk] = sum_t dpre
__global__ void __launch_bounds__(ROW_THREADS) softplus_bias_bwd_kernel(const float* __restrict__ ddt,
                                                                        const float* __restrict__ dt,
                                                                        float* __restrict__ dpre,
                                                                        float* __restrict__ partial, const RowPlan p) {
    const RowSlot s(p);
    float acc[1] = {0.f};
    for (int q = s.q0; q < s.q1; q += p.tpr) {
        float g[4], y[4];
        load_quad(ddt + s.row * p.L, 4 * q, p.L, p.vec, g);
        load_quad(dt + s.row * p.L, 4 * q, p.L, p.vec, y);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            g[e] *= -expm1f(-y[e]);
            acc[0] += g[e];
        }
        store_quad(dpre + s.row * p.L, 4 * q, p.L, p.vec, g);
    }
    const float sum = row_sums(acc, p, s);
    if (s.row < p.rows && s.lane == 0) partial[s.row * p.chunks + s.chunk] = sum;
}

__global__ void __launch_bounds__(256) bias_reduce_kernel(const float* __restrict__ partial, float scale,
                                                          float* __restrict__ dbias, int B, int D, int chunks) {
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= D) return;
    float s = 0.f;
    for (int b = 0; b < B; ++b)
        for (int c = 0; c < chunks; ++c) s += partial[((long long)b * D + i) * chunks + c];
    dbias[i] = scale * s;
}

// ---- RMS norm over the channels of token-major rows ---------------------------------------------
// y = x rstd w,  rstd = rsqrt(mean(x^2) + eps);  one warp per row, the row in registers (d <= 128 V, d a multiple of
// 4), so x is read once.  Bound by HBM: 8 bytes per element forward, 12 backward (16 with `extra`); as separate
// torch passes (square, mean, scale, weight and their adjoints) the block's norm moved about 24 and 60.
constexpr int NORM_WARPS = 8;

template <int V>
__device__ __forceinline__ void load_row(const float* row, int d4, int lane, float4 (&v)[V]) {
#pragma unroll
    for (int k = 0; k < V; ++k) {
        const int q = k * 32 + lane;
        v[k] = q < d4 ? reinterpret_cast<const float4*>(row)[q] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
}
__device__ __forceinline__ float dot4(const float4& a, const float4& b) {
    return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, a.w * b.w)));
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <int V>
__global__ void __launch_bounds__(32 * NORM_WARPS) rms_norm_fwd_kernel(const float* __restrict__ x,
                                                                       const float* __restrict__ w, float eps,
                                                                       float* __restrict__ y,
                                                                       float* __restrict__ rstd, long long rows, int d) {
    const int lane = threadIdx.x & 31, d4 = d / 4;
    float4 wv[V];
    load_row<V>(w, d4, lane, wv);
    for (long long r = (long long)blockIdx.x * NORM_WARPS + (threadIdx.x >> 5); r < rows; r += (long long)gridDim.x * NORM_WARPS) {
        float4 xv[V];
        load_row<V>(x + r * d, d4, lane, xv);
        float ss = 0.f;
#pragma unroll
        for (int k = 0; k < V; ++k) ss += dot4(xv[k], xv[k]);
        const float rs = rsqrtf(warp_sum(ss) / (float)d + eps);
        if (lane == 0) rstd[r] = rs;
#pragma unroll
        for (int k = 0; k < V; ++k) {
            const int q = k * 32 + lane;
            if (q < d4)
                reinterpret_cast<float4*>(y + r * d)[q] =
                    make_float4(xv[k].x * rs * wv[k].x, xv[k].y * rs * wv[k].y, xv[k].z * rs * wv[k].z,
                                xv[k].w * rs * wv[k].w);
        }
    }
}

// dx = rstd (g w - x rstd^2 mean(g w x)) [+ extra];  partial[block][c] = sum over the block's rows of g x rstd
template <int V>
__global__ void __launch_bounds__(32 * NORM_WARPS) rms_norm_bwd_kernel(const float* __restrict__ g,
                                                                       const float* __restrict__ extra,
                                                                       const float* __restrict__ x,
                                                                       const float* __restrict__ w,
                                                                       const float* __restrict__ rstd,
                                                                       float* __restrict__ dx,
                                                                       float* __restrict__ partial, long long rows,
                                                                       int d) {
    __shared__ float4 sums[NORM_WARPS][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, d4 = d / 4;
    float4 wv[V], acc[V];
    load_row<V>(w, d4, lane, wv);
#pragma unroll
    for (int k = 0; k < V; ++k) acc[k] = make_float4(0.f, 0.f, 0.f, 0.f);
    for (long long r = (long long)blockIdx.x * NORM_WARPS + warp; r < rows; r += (long long)gridDim.x * NORM_WARPS) {
        float4 xv[V], gv[V];
        load_row<V>(x + r * d, d4, lane, xv);
        load_row<V>(g + r * d, d4, lane, gv);
        const float rs = rstd[r];
        float dot = 0.f;
#pragma unroll
        for (int k = 0; k < V; ++k) {
            acc[k].x = fmaf(gv[k].x, xv[k].x * rs, acc[k].x);
            acc[k].y = fmaf(gv[k].y, xv[k].y * rs, acc[k].y);
            acc[k].z = fmaf(gv[k].z, xv[k].z * rs, acc[k].z);
            acc[k].w = fmaf(gv[k].w, xv[k].w * rs, acc[k].w);
            gv[k] = make_float4(gv[k].x * wv[k].x, gv[k].y * wv[k].y, gv[k].z * wv[k].z, gv[k].w * wv[k].w);
            dot += dot4(gv[k], xv[k]);
        }
        const float m = warp_sum(dot) / (float)d * rs * rs;
#pragma unroll
        for (int k = 0; k < V; ++k) {
            const int q = k * 32 + lane;
            if (q >= d4) continue;
            float4 o = make_float4(rs * fmaf(-xv[k].x, m, gv[k].x), rs * fmaf(-xv[k].y, m, gv[k].y),
                                   rs * fmaf(-xv[k].z, m, gv[k].z), rs * fmaf(-xv[k].w, m, gv[k].w));
            if (extra) {
                const float4 e = reinterpret_cast<const float4*>(extra + r * d)[q];
                o.x += e.x; o.y += e.y; o.z += e.z; o.w += e.w;
            }
            reinterpret_cast<float4*>(dx + r * d)[q] = o;
        }
    }
    // the block's warps in a fixed order
#pragma unroll
    for (int k = 0; k < V; ++k) {
        __syncthreads();
        sums[warp][lane] = acc[k];
        __syncthreads();
        if (warp == 0 && k * 32 + lane < d4) {
            float4 s = sums[0][lane];
#pragma unroll
            for (int v = 1; v < NORM_WARPS; ++v) {
                const float4 a = sums[v][lane];
                s.x += a.x; s.y += a.y; s.z += a.z; s.w += a.w;
            }
            reinterpret_cast<float4*>(partial + (long long)blockIdx.x * d)[k * 32 + lane] = s;
        }
    }
}

// dw[c] = sum over blocks: one warp per 32 columns and 8 strands of blocks, strands added in order
__global__ void __launch_bounds__(256) norm_weight_reduce_kernel(const float* __restrict__ partial,
                                                                 float* __restrict__ dw, int blocks, int d) {
    __shared__ float sums[8][32];
    const int c = blockIdx.x * 32 + (threadIdx.x & 31), strand = threadIdx.x >> 5;
    float s = 0.f;
    if (c < d)
        for (int b = strand; b < blocks; b += 8) s += partial[(long long)b * d + c];
    sums[strand][threadIdx.x & 31] = s;
    __syncthreads();
    if (strand == 0 && c < d) {
        for (int k = 1; k < 8; ++k) s += sums[k][threadIdx.x];
        dw[c] = s;
    }
}

// ---- polar form of the operator's B and C -------------------------------------------------------
// r = softplus(re) (re above 20 passes through, as torch's softplus), angle = im; both parameters in one launch each
// way: the views, softplus, copies and their adjoints were 16 launches of a training call (B8 D16 N4 L256: 41 -> 23
// launches with the zero states gone too).
__global__ void __launch_bounds__(128) polar_params_fwd_kernel(const float2* __restrict__ B, const float2* __restrict__ C,
                                                               float* __restrict__ out, int N) {
    const int j = blockIdx.x * 128 + threadIdx.x;
    if (j >= 2 * N) return;
    const float2 v = j < N ? B[j] : C[j - N];
    float* o = out + (j < N ? j : N + j);                     // rows B_r, B_theta, C_r, C_theta
    o[0] = v.x > 20.f ? v.x : log1pf(expf(v.x));
    o[N] = v.y;
}

__global__ void __launch_bounds__(128) polar_params_bwd_kernel(const float* __restrict__ dBr, const float* __restrict__ dBt,
                                                               const float* __restrict__ dCr, const float* __restrict__ dCt,
                                                               const float2* __restrict__ B, const float2* __restrict__ C,
                                                               float2* __restrict__ dB, float2* __restrict__ dC, int N) {
    const int j = blockIdx.x * 128 + threadIdx.x;
    if (j >= 2 * N) return;
    const bool b = j < N;
    const int i = b ? j : j - N;
    const float x = b ? B[i].x : C[i].x;
    const float *gr = b ? dBr : dCr, *gt = b ? dBt : dCt;
    const float e = expf(x), g = gr ? gr[i] : 0.f;
    (b ? dB : dC)[i] = make_float2(x > 20.f ? g : g * e / (e + 1.f), gt ? gt[i] : 0.f);
}

// four resident blocks per SM, fewer when there are fewer rows
unsigned norm_blocks(long long rows) {
    return (unsigned)std::min<long long>((rows + NORM_WARPS - 1) / NORM_WARPS, 148LL * 4);
}

bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int stage_dims_ok(const char* who, int B, int D, int L) {
    if (B <= 0 || D <= 0 || L <= 0 || (long long)B * D > 0x7fffffffLL) {
        set_error("%s: sizes must be positive and B*D fit 31 bits (B=%d D=%d L=%d)", who, B, D, L);
        return AUSSM_EINVAL;
    }
    return AUSSM_OK;
}

int launch_ok(const char* who) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error("%s launch: %s", who, cudaGetErrorString(e));
        return AUSSM_ECUDA;
    }
    return AUSSM_OK;
}

}  // namespace
}  // namespace aussm

using namespace aussm;

extern "C" {

int aussm_b200_conv_pre_fwd(const float* xs, const float* w, const float* bias, float* u, int B, int D, int L, int K,
                            aussm_stream_t stream) {
    if (int rc = stage_dims_ok("conv_pre_fwd", B, D, L)) return rc;
    if (!xs || !w || !u || K < 1 || K > KMAX) {
        set_error("conv_pre_fwd: null pointer or unsupported filter length %d (1..%d)", K, KMAX);
        return AUSSM_EINVAL;
    }
    const RowPlan p = row_plan((long long)B * D, L, L % 4 == 0 && al16(xs) && al16(u));
    conv_pre_fwd_kernel<<<p.blocks, ROW_THREADS, 0, (cudaStream_t)stream>>>(xs, w, bias, u, D, K, p);
    count_launch();
    return launch_ok("conv_pre_fwd");
}

size_t aussm_b200_conv_pre_bwd_workspace_bytes(int B, int D) {
    if (B <= 0 || D <= 0) return 0;
    const long long rows = (long long)B * D;
    return ((size_t)rows * row_chunks_max(rows) * (KMAX + 1) * sizeof(float) + 255) / 256 * 256;
}

int aussm_b200_conv_pre_bwd(const float* du, const float* xs, const float* w, float* dxs, float* dw, float* dbias,
                            int B, int D, int L, int K, void* workspace, size_t workspace_bytes,
                            aussm_stream_t stream_) {
    if (int rc = stage_dims_ok("conv_pre_bwd", B, D, L)) return rc;
    if (!du || !xs || !w || !dxs || !dw || K < 1 || K > KMAX) {
        set_error("conv_pre_bwd: null pointer or unsupported filter length %d (1..%d)", K, KMAX);
        return AUSSM_EINVAL;
    }
    if (!workspace || workspace_bytes < aussm_b200_conv_pre_bwd_workspace_bytes(B, D)) {
        set_error("conv_pre_bwd: workspace of %zu bytes required, got %zu", aussm_b200_conv_pre_bwd_workspace_bytes(B, D),
                  workspace_bytes);
        return AUSSM_EWORKSPACE;
    }
    cudaStream_t stream = (cudaStream_t)stream_;
    float* partial = static_cast<float*>(workspace);
    const RowPlan p = row_plan((long long)B * D, L, L % 4 == 0 && al16(du) && al16(xs) && al16(dxs));
    conv_pre_bwd_kernel<<<p.blocks, ROW_THREADS, 0, stream>>>(du, xs, w, dxs, partial, D, K, p);
    count_launch();
    if (int rc = launch_ok("conv_pre_bwd")) return rc;
    conv_pre_reduce_kernel<<<(D * (K + 1) + 255) / 256, 256, 0, stream>>>(partial, dw, dbias, B, D, K, p.chunks);
    count_launch();
    return launch_ok("conv_pre_bwd reduction");
}

int aussm_b200_softplus_bias_fwd(const float* pre, const float* bias, float scale, float* dt, int B, int D, int L,
                                 aussm_stream_t stream) {
    if (int rc = stage_dims_ok("softplus_bias_fwd", B, D, L)) return rc;
    if (!pre || !dt) {
        set_error("softplus_bias_fwd: null pointer");
        return AUSSM_EINVAL;
    }
    const RowPlan p = row_plan((long long)B * D, L, L % 4 == 0 && al16(pre) && al16(dt));
    softplus_bias_fwd_kernel<<<p.blocks, ROW_THREADS, 0, (cudaStream_t)stream>>>(pre, bias, scale, dt, D, p);
    count_launch();
    return launch_ok("softplus_bias_fwd");
}

size_t aussm_b200_softplus_bias_bwd_workspace_bytes(int B, int D) {
    if (B <= 0 || D <= 0) return 0;
    const long long rows = (long long)B * D;
    return ((size_t)rows * row_chunks_max(rows) * sizeof(float) + 255) / 256 * 256;
}

int aussm_b200_softplus_bias_bwd(const float* ddt, const float* dt, float scale, float* dpre, float* dbias, int B,
                                 int D, int L, void* workspace, size_t workspace_bytes, aussm_stream_t stream_) {
    if (int rc = stage_dims_ok("softplus_bias_bwd", B, D, L)) return rc;
    if (!ddt || !dt || !dpre) {
        set_error("softplus_bias_bwd: null pointer");
        return AUSSM_EINVAL;
    }
    if (!workspace || workspace_bytes < aussm_b200_softplus_bias_bwd_workspace_bytes(B, D)) {
        set_error("softplus_bias_bwd: workspace of %zu bytes required, got %zu",
                  aussm_b200_softplus_bias_bwd_workspace_bytes(B, D), workspace_bytes);
        return AUSSM_EWORKSPACE;
    }
    cudaStream_t stream = (cudaStream_t)stream_;
    float* partial = static_cast<float*>(workspace);
    const RowPlan p = row_plan((long long)B * D, L, L % 4 == 0 && al16(ddt) && al16(dt) && al16(dpre));
    softplus_bias_bwd_kernel<<<p.blocks, ROW_THREADS, 0, stream>>>(ddt, dt, dpre, partial, p);
    count_launch();
    if (int rc = launch_ok("softplus_bias_bwd")) return rc;
    if (dbias) {
        bias_reduce_kernel<<<(D + 255) / 256, 256, 0, stream>>>(partial, scale, dbias, B, D, p.chunks);
        count_launch();
        return launch_ok("softplus_bias_bwd reduction");
    }
    return AUSSM_OK;
}

static int norm_ok(const char* who, const void* a, const void* b, const void* c, long long rows, int d) {
    if (rows <= 0 || d <= 0 || d % 4 || d > AUSSM_MAX_NORM_CHANNELS) {
        set_error("%s: rows=%lld must be positive and d=%d a multiple of 4 up to %d", who, rows, d, AUSSM_MAX_NORM_CHANNELS);
        return AUSSM_EINVAL;
    }
    if (!a || !b || !c || !al16(a) || !al16(b) || !al16(c)) {
        set_error("%s: null or misaligned (16 bytes) pointer", who);
        return AUSSM_EINVAL;
    }
    return AUSSM_OK;
}

int aussm_b200_polar_params_fwd(const float* B, const float* C, float* out, int N, aussm_stream_t stream) {
    if (N <= 0 || N > 0x3fffffff || !B || !C || !out) {
        set_error("polar_params_fwd: null pointer or N=%d out of range", N);
        return AUSSM_EINVAL;
    }
    polar_params_fwd_kernel<<<(2 * N + 127) / 128, 128, 0, (cudaStream_t)stream>>>(
        reinterpret_cast<const float2*>(B), reinterpret_cast<const float2*>(C), out, N);
    count_launch();
    return launch_ok("polar_params_fwd");
}

int aussm_b200_polar_params_bwd(const float* dB_r, const float* dB_theta, const float* dC_r, const float* dC_theta,
                                const float* B, const float* C, float* dB, float* dC, int N, aussm_stream_t stream) {
    if (N <= 0 || N > 0x3fffffff || !B || !C || !dB || !dC) {
        set_error("polar_params_bwd: null pointer or N=%d out of range", N);
        return AUSSM_EINVAL;
    }
    polar_params_bwd_kernel<<<(2 * N + 127) / 128, 128, 0, (cudaStream_t)stream>>>(
        dB_r, dB_theta, dC_r, dC_theta, reinterpret_cast<const float2*>(B), reinterpret_cast<const float2*>(C),
        reinterpret_cast<float2*>(dB), reinterpret_cast<float2*>(dC), N);
    count_launch();
    return launch_ok("polar_params_bwd");
}

#define AUSSM_NORM(KERNEL, ...)                                                                        \
    do {                                                                                               \
        const dim3 grid(norm_blocks(rows)), block(32 * NORM_WARPS);                                    \
        if (d <= 128) KERNEL<1><<<grid, block, 0, (cudaStream_t)stream>>>(__VA_ARGS__);                \
        else if (d <= 256) KERNEL<2><<<grid, block, 0, (cudaStream_t)stream>>>(__VA_ARGS__);           \
        else if (d <= 512) KERNEL<4><<<grid, block, 0, (cudaStream_t)stream>>>(__VA_ARGS__);           \
        else KERNEL<8><<<grid, block, 0, (cudaStream_t)stream>>>(__VA_ARGS__);                         \
        count_launch();                                                                                \
    } while (0)

int aussm_b200_rms_norm_fwd(const float* x, const float* w, float eps, float* y, float* rstd, long long rows, int d,
                            aussm_stream_t stream) {
    if (int rc = norm_ok("rms_norm_fwd", x, w, y, rows, d)) return rc;
    if (!rstd) {
        set_error("rms_norm_fwd: null pointer");
        return AUSSM_EINVAL;
    }
    AUSSM_NORM(rms_norm_fwd_kernel, x, w, eps, y, rstd, rows, d);
    return launch_ok("rms_norm_fwd");
}

size_t aussm_b200_rms_norm_bwd_workspace_bytes(long long rows, int d) {
    if (rows <= 0 || d <= 0) return 0;
    return ((size_t)norm_blocks(rows) * d * sizeof(float) + 255) / 256 * 256;
}

int aussm_b200_rms_norm_bwd(const float* g, const float* extra, const float* x, const float* w, const float* rstd,
                            float* dx, float* dw, long long rows, int d, void* workspace, size_t workspace_bytes,
                            aussm_stream_t stream) {
    if (int rc = norm_ok("rms_norm_bwd", x, w, dx, rows, d)) return rc;
    if (!g || !rstd || !dw || !al16(g) || !al16(extra)) {
        set_error("rms_norm_bwd: null or misaligned (16 bytes) pointer");
        return AUSSM_EINVAL;
    }
    const size_t need = aussm_b200_rms_norm_bwd_workspace_bytes(rows, d);
    if (!workspace || workspace_bytes < need || !al16(workspace)) {
        set_error("rms_norm_bwd: workspace of %zu bytes (16-byte aligned) required, got %zu", need, workspace_bytes);
        return AUSSM_EWORKSPACE;
    }
    float* partial = static_cast<float*>(workspace);
    AUSSM_NORM(rms_norm_bwd_kernel, g, extra, x, w, rstd, dx, partial, rows, d);
    if (int rc = launch_ok("rms_norm_bwd")) return rc;
    norm_weight_reduce_kernel<<<(d + 31) / 32, 256, 0, (cudaStream_t)stream>>>(partial, dw, (int)norm_blocks(rows), d);
    count_launch();
    return launch_ok("rms_norm_bwd reduction");
}

}  // extern "C"
