// Real selective scan ("S6") for sm_100a, several-states-per-thread kernels for up to 32 states per channel.
//
// The S6 recurrence has a constant A, so unlike the unitary and complex scans it streams no per-state exponent:
// per (b, i, t) it moves 16 bytes forward and 28 backward for N states of arithmetic, and what has to be cheap is
// the arithmetic.  Here a channel is owned by LPC lanes (1, 2 or 4), each keeping NS / LPC of its states in
// registers (thread k of a channel owns states k, k + LPC, ...); a warp (one-warp blocks) owns 32 / LPC channels
// of ONE batch entry and walks time sequentially in 16-step tiles staged by coalesced 16-byte asynchronous copies
// through a two-stage ring:
//   * B_j(t), C_j(t) are the same for every channel of a batch entry: the lanes that own the same states read the
//     same shared-memory address (one wavefront per distinct address, and the LPC addresses of an instruction
//     fall into disjoint banks); with a thread per state and channel the shared-memory pipe was the bound;
//   * the sum over states is a chain in the thread plus log2(LPC) shuffles: no column-sum tiles;
//   * what depends on the channel and the step only (softplus, the gate and its derivative) is evaluated once per
//     tile by a pass in which the lanes of a channel share the tile's steps;
//   * dB and dC (sums over the channels of a batch entry) are added across the warp's channels through a padded
//     shared-memory tile and leave as one vector atomic per state and four steps.
// LPC is chosen per launch: one lane per channel is the cheapest per step, but a problem with few channels then has
// too few warps to hide the latency of its dependent chains (one warp per scheduler issues every third cycle).
// The recurrence contracts, so it cannot be run backwards: the forward kernel records the N states at every tile
// start, (channel, tile, state) with the states contiguous; the backward kernel recomputes a tile from there, keeping
// the states at every fourth step in shared memory, and then walks the tile's four-step groups in reverse, each
// group recomputed once more, state by state, with the state before every step held in registers.
//
// The operator is mamba_ssm.selective_scan_fn as called by MambaBlock.ssm_mamba (ai-modules/wavesAI/model/aussm.py:
// 771-805).
#include <stdint.h>

#include <algorithm>

#include "common.cuh"
#include "host_common.cuh"
#include "scan_s6.cuh"

namespace aussm {
namespace {

constexpr int WT = kS6Tile;          // steps per tile = checkpoint interval
constexpr int WTP = WT + 4;              // row pitch: a quarter-warp's 128-bit reads of eight rows hit disjoint banks
constexpr int NQ = WT / 4;
constexpr int WSTAGES = 2;
constexpr float kLog2e = 1.4426950408889634f;
constexpr float kLn2 = 0.6931471805599453f;

template <int NS_, int LPC_, bool BWD_>
struct WCfg {
    static constexpr int NS = NS_, LPC = LPC_;
    static constexpr int SPT = NS / LPC;                              // states per thread
    static constexpr int CPW = 32 / LPC;                              // channels per warp
    static constexpr int AUX = BWD_ ? 4 : 3;                          // u, delta, z [, gout]
    static constexpr int BC_FLOATS = 2 * NS * WTP;                    // B rows then C rows
    static constexpr int AUX_FLOATS = CPW * WTP;                      // one array: a row per channel
    static constexpr int STAGE_FLOATS = BC_FLOATS + AUX * AUX_FLOATS;
    // backward only: this thread's states at every fourth step [NQ][SPT][32]; channel-sum tile of four steps each,
    // [2 NS rows][CPW + 1] (pitch odd: the row-per-lane reads hit disjoint banks)
    static constexpr int SUB_FLOATS = BWD_ ? NQ * SPT * 32 : 0;
    static constexpr int RED_PITCH = CPW + 1;
    static constexpr int RED_FLOATS = BWD_ ? 2 * NS * RED_PITCH * 4 : 0;
    static constexpr size_t SMEM_BYTES = (size_t)(WSTAGES * STAGE_FLOATS + SUB_FLOATS + RED_FLOATS) * sizeof(float);
    static constexpr int BC_PIECES = (2 * NS * NQ + 31) / 32;         // 16-byte pieces per lane
    static constexpr int ROW_PIECES = (CPW * NQ + 31) / 32;           // per array
    static constexpr int PRE_STEPS = WT / LPC;                        // steps per lane in the per-channel passes
    static_assert(NS % LPC == 0 && PRE_STEPS % 4 == 0, "shape");
};

// Tile movement.  Piece id = i * 32 + lane -> row id / NQ, 16-byte column id % NQ.
template <class C>
struct WMap {
    long long row_off[C::ROW_PIECES];      // offset (floats) of this lane's pieces in a (nch, L) array, step 0
    const float* bc_ptr[C::BC_PIECES];     // nullptr: nothing to copy (state beyond N)
    int nvalid;

    __device__ __forceinline__ void init(int lane, int nvalid_, int N, long long L, const float* Bb, const float* Cb,
                                         long long ch0) {
        nvalid = nvalid_;
#pragma unroll
        for (int i = 0; i < C::ROW_PIECES; ++i) {
            const int id = i * 32 + lane;
            const int row = id / NQ, col = id % NQ;
            row_off[i] = (ch0 + min(row, nvalid - 1)) * L + col * 4;       // rows beyond the last channel shadow it
        }
#pragma unroll
        for (int i = 0; i < C::BC_PIECES; ++i) {
            const int id = i * 32 + lane;
            const int row = id / NQ, col = id % NQ;
            bc_ptr[i] = nullptr;
            if (row < 2 * C::NS) {
                const int j = row % C::NS;
                if (j < N) bc_ptr[i] = (row < C::NS ? Bb : Cb) + (long long)j * L + col * 4;
            }
        }
    }

    __device__ __forceinline__ void issue(float* stage, const float* const* aux_src, long long t0, int tlen,
                                          int lane) const {
        const int col = lane % NQ;
        if (col * 4 < tlen) {
#pragma unroll
            for (int i = 0; i < C::BC_PIECES; ++i) {
                const int id = i * 32 + lane;
                if (bc_ptr[i] != nullptr) cp_async16(stage + (id / NQ) * WTP + col * 4, bc_ptr[i] + t0);
            }
#pragma unroll
            for (int a = 0; a < C::AUX; ++a) {
                if (aux_src[a] == nullptr) continue;
                float* dst = stage + C::BC_FLOATS + a * C::AUX_FLOATS;
#pragma unroll
                for (int i = 0; i < C::ROW_PIECES; ++i) {
                    const int id = i * 32 + lane;
                    if (id / NQ < C::CPW) cp_async16(dst + (id / NQ) * WTP + col * 4, aux_src[a] + row_off[i] + t0);
                }
            }
        }
        cp_async_commit();
    }

    // coalesced store of one array's rows (real channels only) from the stage
    __device__ __forceinline__ void store(const float* src_rows, float* dst, long long t0, int tlen, int lane) const {
        const int col = lane % NQ;
        if (col * 4 >= tlen) return;
#pragma unroll
        for (int i = 0; i < C::ROW_PIECES; ++i) {
            const int row = (i * 32 + lane) / NQ;
            if (row < nvalid && row < C::CPW)
                *reinterpret_cast<float4*>(dst + row_off[i] + t0) = ld_shared_f4(src_rows + row * WTP + col * 4);
        }
    }
};

__device__ __forceinline__ float softplus_(float x) { return x > 20.f ? x : log1pf(__expf(x)); }

// sum over the LPC lanes of a channel (they are adjacent)
template <int LPC>
__device__ __forceinline__ float channel_sum(float v) {
#pragma unroll
    for (int o = 1; o < LPC; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

#define AUSSM_F4(v) {(v).x, (v).y, (v).z, (v).w}
// four consecutive steps as two pairs: what does not run along the recurrence is done two steps at a time with the
// packed float32x2 instructions (the kernels are bound by the shared-memory pipe and by what a few warps can issue, not by the FP32 pipe)
#define AUSSM_F22(v) {make_float2((v).x, (v).y), make_float2((v).z, (v).w)}

// multipliers exp(dlt A) of four steps
__device__ __forceinline__ void multipliers(const float2 (&dlt)[2], float2 A2, float2 (&a)[2]) {
#pragma unroll
    for (int p = 0; p < 2; ++p) {
        const float2 x = __fmul2_rn(dlt[p], A2);
        a[p] = make_float2(ex2_ftz(x.x), ex2_ftz(x.y));
    }
}
// four steps of h_t = a_t h_{t-1} + x_t; h receives the states after each step
__device__ __forceinline__ void four_steps(float h0, const float2 (&a)[2], const float2 (&x)[2], float2 (&h)[2]) {
    h[0].x = fmaf(a[0].x, h0, x[0].x);
    h[0].y = fmaf(a[0].y, h[0].x, x[0].y);
    h[1].x = fmaf(a[1].x, h[0].y, x[1].x);
    h[1].y = fmaf(a[1].y, h[1].x, x[1].y);
}

// ---------------------------------------------------------------------------
// Forward
// ---------------------------------------------------------------------------
template <int NS, int LPC>
__global__ void __launch_bounds__(32) s6w_fwd_kernel(const S6FwdParams p) {
    using C = WCfg<NS, LPC, false>;
    constexpr int SPT = C::SPT, CPW = C::CPW;
    extern __shared__ __align__(128) float smem[];
    const int lane = threadIdx.x;
    const int c = lane / LPC, k = lane % LPC;
    const int tasks_per_batch = (p.Dmod + CPW - 1) / CPW;
    const int tasks = tasks_per_batch * (p.nch / p.Dmod);
    const int seg = (int)(blockIdx.x / tasks), task = blockIdx.x % tasks;
    const int b = task / tasks_per_batch, i0 = (task % tasks_per_batch) * CPW;
    const int nvalid = min(CPW, p.Dmod - i0);
    const bool act = c < nvalid;
    const int i = i0 + min(c, nvalid - 1);
    const long long ch0 = (long long)b * p.Dmod + i0, ch = (long long)b * p.Dmod + i;
    const int N = p.N, L = p.L;
    const int ntiles = (L + WT - 1) / WT;
    const int first = seg * p.seg_tiles, last = p.nseg > 1 ? min(ntiles, first + p.seg_tiles) : ntiles;   // tiles

    float A2[SPT], h[SPT];
#pragma unroll
    for (int jj = 0; jj < SPT; ++jj) {
        const int j = jj * LPC + k;
        A2[jj] = j < N ? p.A[(long long)i * N + j] * kLog2e : 0.f;
        h[jj] = 0.f;
    }
    const float dskip = p.Dskip ? p.Dskip[i] : 0.f;
    const float bias = p.delta_bias ? p.delta_bias[i] : 0.f;
    const bool softplus = p.delta_softplus != 0, gate = p.z != nullptr;

    // rows of states beyond N are never copied: they must read as zero (B = C = 0 keeps such a state at zero)
    for (int x = lane; x < WSTAGES * C::STAGE_FLOATS; x += 32) smem[x] = 0.f;
    __syncwarp();

    const float* aux_src[C::AUX] = {p.u, p.delta, p.z};
    WMap<C> map;
    map.init(lane, nvalid, N, L, p.Bm + (long long)b * N * L, p.Cm + (long long)b * N * L, ch0);
    for (int s = 0; s < WSTAGES; ++s) {
        const int t = first + s;
        if (t < last) map.issue(smem + (t % WSTAGES) * C::STAGE_FLOATS, aux_src, (long long)t * WT, min(WT, L - t * WT), lane);
        else cp_async_commit();
    }
    float* ck = p.ckpt ? p.ckpt + ch * ntiles * N : nullptr;
    if (seg > 0) {                                          // left there by the segment chain
#pragma unroll
        for (int jj = 0; jj < SPT; ++jj)
            if (jj * LPC + k < N) h[jj] = ck[(long long)first * N + jj * LPC + k];
    }

    for (int tile = first; tile < last; ++tile) {
        float* st = smem + (tile % WSTAGES) * C::STAGE_FLOATS;
        float* urow = st + C::BC_FLOATS + c * WTP;
        float* drow = urow + C::AUX_FLOATS;
        float* zrow = drow + C::AUX_FLOATS;
        const long long t0 = (long long)tile * WT;
        const int tlen = min(WT, L - (int)t0);
        cp_async_wait<WSTAGES - 1>();
        __syncwarp();
        if (ck && act) {
#pragma unroll
            for (int jj = 0; jj < SPT; ++jj)
                if (jj * LPC + k < N) ck[(long long)tile * N + jj * LPC + k] = h[jj];
        }
        // per-channel pass: lane k of a channel takes steps [k PRE_STEPS, (k + 1) PRE_STEPS): the delta cells
        // receive dlt = softplus(delta + bias), the z cells silu(z)
#pragma unroll
        for (int x = 0; x < C::PRE_STEPS; x += 4) {
            const int t = k * C::PRE_STEPS + x;
            const float4 d4 = ld_shared_f4(drow + t);
            float dv[4] = AUSSM_F4(d4);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                dv[e] += bias;
                if (softplus) dv[e] = softplus_(dv[e]);
            }
            st_shared_f4(drow + t, make_float4(dv[0], dv[1], dv[2], dv[3]));
            if (gate) {
                const float4 z4 = ld_shared_f4(zrow + t);
                st_shared_f4(zrow + t, make_float4(siluf_(z4.x), siluf_(z4.y), siluf_(z4.z), siluf_(z4.w)));
            }
        }
        __syncwarp();
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            if (4 * q >= tlen) break;
            const float4 u4 = ld_shared_f4(urow + 4 * q), d4 = ld_shared_f4(drow + 4 * q);
            const float uv[4] = AUSSM_F4(u4);
            const float2 uv2[2] = AUSSM_F22(u4), dlt[2] = AUSSM_F22(d4);
            const float2 s[2] = {__fmul2_rn(dlt[0], uv2[0]), __fmul2_rn(dlt[1], uv2[1])};
            float2 y2[2] = {f2(0.f), f2(0.f)};
#pragma unroll
            for (int jj = 0; jj < SPT; ++jj) {
                const int j = jj * LPC + k;
                const float4 b4 = ld_shared_f4(st + j * WTP + 4 * q);               // one address per value of k
                const float4 c4 = ld_shared_f4(st + (NS + j) * WTP + 4 * q);
                const float2 bv[2] = AUSSM_F22(b4), cv[2] = AUSSM_F22(c4);
                float2 a[2], ht[2];
                multipliers(dlt, f2(A2[jj]), a);
                const float2 x[2] = {__fmul2_rn(s[0], bv[0]), __fmul2_rn(s[1], bv[1])};
                four_steps(h[jj], a, x, ht);
                h[jj] = ht[1].y;
#pragma unroll
                for (int p2 = 0; p2 < 2; ++p2) y2[p2] = __ffma2_rn(cv[p2], ht[p2], y2[p2]);
            }
            float y[4] = {y2[0].x, y2[0].y, y2[1].x, y2[1].y};
#pragma unroll
            for (int e = 0; e < 4; ++e) y[e] = fmaf(dskip, uv[e], channel_sum<LPC>(y[e]));
            if (gate) {
                const float4 z4 = ld_shared_f4(zrow + 4 * q);                       // silu(z)
                y[0] *= z4.x; y[1] *= z4.y; y[2] *= z4.z; y[3] *= z4.w;
            }
            __syncwarp();                       // every lane of the channel has read the u cells
            if (k == 0) st_shared_f4(urow + 4 * q, make_float4(y[0], y[1], y[2], y[3]));   // they now hold the output
        }
        __syncwarp();
        map.store(st + C::BC_FLOATS, p.out, t0, tlen, lane);
        __syncwarp();
        const int nt = tile + WSTAGES;
        if (nt < last) map.issue(st, aux_src, (long long)nt * WT, min(WT, L - nt * WT), lane);
        else cp_async_commit();
    }
    cp_async_wait<0>();
    if (act && p.last_state && last == ntiles) {
#pragma unroll
        for (int jj = 0; jj < SPT; ++jj)
            if (jj * LPC + k < N) p.last_state[ch * N + jj * LPC + k] = h[jj];
    }
}

// ---------------------------------------------------------------------------
// Backward
// ---------------------------------------------------------------------------
__device__ __forceinline__ void red_add_v4w(float* addr, const float4 v) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(addr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                 : "memory");
}

template <int NS, int LPC>
__global__ void __launch_bounds__(32) s6w_bwd_kernel(const S6BwdParams p) {
    using C = WCfg<NS, LPC, true>;
    constexpr int SPT = C::SPT, CPW = C::CPW, RP = C::RED_PITCH;
    extern __shared__ __align__(128) float smem[];
    const int lane = threadIdx.x;
    const int c = lane / LPC, k = lane % LPC;
    const int tasks_per_batch = (p.Dmod + CPW - 1) / CPW;
    const int tasks = tasks_per_batch * (p.nch / p.Dmod);
    const int seg = (int)(blockIdx.x / tasks), task = blockIdx.x % tasks;
    const int b = task / tasks_per_batch, i0 = (task % tasks_per_batch) * CPW;
    const int nvalid = min(CPW, p.Dmod - i0);
    const bool act = c < nvalid;
    const int i = i0 + min(c, nvalid - 1);
    const long long ch0 = (long long)b * p.Dmod + i0, ch = (long long)b * p.Dmod + i;
    const int N = p.N, L = p.L;
    const int ntiles = (L + WT - 1) / WT;
    const int first = seg * p.seg_tiles, last = p.nseg > 1 ? min(ntiles, first + p.seg_tiles) : ntiles;   // tiles

    float* sub = smem + WSTAGES * C::STAGE_FLOATS;          // [NQ][SPT][32]
    float* red = sub + C::SUB_FLOATS;                       // [2 NS][RP] float4: gB rows, then gC rows

    float A2[SPT], eps[SPT];
    float2 dA2[SPT];         // even and odd steps
#pragma unroll
    for (int jj = 0; jj < SPT; ++jj) {
        const int j = jj * LPC + k;
        A2[jj] = j < N ? p.A[(long long)i * N + j] * kLog2e : 0.f;
        eps[jj] = (p.nseg > 1 && act && j < N) ? p.seg_grad[(ch * p.nseg + seg) * N + j] : 0.f;       // a_{t+1} eta_{t+1}
        dA2[jj] = f2(0.f);
    }
    const float dskip = p.Dskip ? p.Dskip[i] : 0.f;
    const float bias = p.delta_bias ? p.delta_bias[i] : 0.f;
    const bool softplus = p.delta_softplus != 0, gate = p.z != nullptr;
    float dD_acc = 0.f, db_acc = 0.f;

    for (int x = lane; x < WSTAGES * C::STAGE_FLOATS; x += 32) smem[x] = 0.f;
    __syncwarp();

    const float* aux_src[C::AUX] = {p.u, p.delta, p.z, p.gout};
    WMap<C> map;
    map.init(lane, nvalid, N, L, p.Bm + (long long)b * N * L, p.Cm + (long long)b * N * L, ch0);
    for (int r = 0; r < WSTAGES; ++r) {
        const int tile = last - 1 - r;
        if (tile >= first)
            map.issue(smem + r * C::STAGE_FLOATS, aux_src, (long long)tile * WT, min(WT, L - tile * WT), lane);
        else cp_async_commit();
    }
    const float* ck = p.ckpt + ch * ntiles * N;
    float hn[SPT];                                          // state at the start of the tile taken next
#pragma unroll
    for (int jj = 0; jj < SPT; ++jj)
        hn[jj] = jj * LPC + k < N ? ck[(long long)(last - 1) * N + jj * LPC + k] : 0.f;
    // lane r of the channel-sum pass owns rows r, r + 32 of the tile: dB of state r (r < NS) or dC of state r - NS
    constexpr int RROWS = (2 * NS + 31) / 32;
    float* red_dst[RROWS];
    bool red_on[RROWS];
#pragma unroll
    for (int x = 0; x < RROWS; ++x) {
        const int row = x * 32 + lane, rj = row % NS;
        red_dst[x] = (row < NS ? p.dB : p.dC) + ((long long)b * N + min(rj, N - 1)) * L;
        red_on[x] = row < 2 * NS && rj < N;
    }

    for (int r = 0; r < last - first; ++r) {
        const int tile = last - 1 - r;
        float* st = smem + (r % WSTAGES) * C::STAGE_FLOATS;
        float* urow = st + C::BC_FLOATS + c * WTP;
        float* drow = urow + C::AUX_FLOATS;
        float* zrow = drow + C::AUX_FLOATS;
        float* grow = zrow + C::AUX_FLOATS;
        const long long t0 = (long long)tile * WT;
        const int tlen = min(WT, L - (int)t0);
        const int nq = tlen >> 2;
        float h[SPT];
#pragma unroll
        for (int jj = 0; jj < SPT; ++jj) h[jj] = hn[jj];
        if (tile > first) {
#pragma unroll
            for (int jj = 0; jj < SPT; ++jj)
                hn[jj] = jj * LPC + k < N ? ck[(long long)(tile - 1) * N + jj * LPC + k] : 0.f;
        }
        cp_async_wait<WSTAGES - 1>();
        __syncwarp();

        // per-channel pass (lane k of a channel: steps [k PRE_STEPS, (k + 1) PRE_STEPS)):
        //   delta cells <- dlt = softplus(delta + bias);  gout cells <- w = gout silu(z);  z cells <- gout silu'(z)
#pragma unroll
        for (int x = 0; x < C::PRE_STEPS; x += 4) {
            const int t = k * C::PRE_STEPS + x;
            const float4 d4 = ld_shared_f4(drow + t);
            float dv[4] = AUSSM_F4(d4);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                dv[e] += bias;
                if (softplus) dv[e] = softplus_(dv[e]);
            }
            st_shared_f4(drow + t, make_float4(dv[0], dv[1], dv[2], dv[3]));
            const float4 g4 = ld_shared_f4(grow + t);
            float gv[4] = AUSSM_F4(g4);
            if (gate) {
                const float4 z4 = ld_shared_f4(zrow + t);
                const float zv[4] = AUSSM_F4(z4);
                float zz[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float gz;
                    const float sz = silu_and_grad(zv[e], gz);
                    zz[e] = gv[e] * gz;
                    gv[e] *= sz;
                }
                st_shared_f4(zrow + t, make_float4(zz[0], zz[1], zz[2], zz[3]));
            }
            if (!act) gv[0] = gv[1] = gv[2] = gv[3] = 0.f;            // a shadow channel adds nothing to dB / dC
            st_shared_f4(grow + t, make_float4(gv[0], gv[1], gv[2], gv[3]));
        }
        __syncwarp();

        // first pass: this thread's states at the start of every four-step group
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            if (q >= nq) break;
#pragma unroll
            for (int jj = 0; jj < SPT; ++jj) sub[(q * SPT + jj) * 32 + lane] = h[jj];
            if (q + 1 >= nq) break;                                   // the last group's end state is not needed
            const float4 u4 = ld_shared_f4(urow + 4 * q), d4 = ld_shared_f4(drow + 4 * q);
            const float2 uv[2] = AUSSM_F22(u4), dlt[2] = AUSSM_F22(d4);
            const float2 s[2] = {__fmul2_rn(dlt[0], uv[0]), __fmul2_rn(dlt[1], uv[1])};
#pragma unroll
            for (int jj = 0; jj < SPT; ++jj) {
                const float4 b4 = ld_shared_f4(st + (jj * LPC + k) * WTP + 4 * q);
                const float2 bv[2] = AUSSM_F22(b4);
                const float2 x[2] = {__fmul2_rn(s[0], bv[0]), __fmul2_rn(s[1], bv[1])};
                float2 a[2], ht[2];
                multipliers(dlt, f2(A2[jj]), a);
                four_steps(h[jj], a, x, ht);
                h[jj] = ht[1].y;
            }
        }

        // second pass: the groups in reverse
#pragma unroll 1
        for (int q = nq - 1; q >= 0; --q) {
            const float4 u4 = ld_shared_f4(urow + 4 * q), d4 = ld_shared_f4(drow + 4 * q);
            const float4 w4 = ld_shared_f4(grow + 4 * q);
            const float uv[4] = AUSSM_F4(u4), dlt[4] = AUSSM_F4(d4), w[4] = AUSSM_F4(w4);
            const float2 uv2[2] = AUSSM_F22(u4), dlt2[2] = AUSSM_F22(d4), w2[2] = AUSSM_F22(w4);
            const float2 s[2] = {__fmul2_rn(dlt2[0], uv2[0]), __fmul2_rn(dlt2[1], uv2[1])};
            float2 SQ2[2] = {f2(0.f), f2(0.f)}, SY2[2] = {f2(0.f), f2(0.f)}, SP2[2] = {f2(0.f), f2(0.f)};
#pragma unroll
            for (int jj = 0; jj < SPT; ++jj) {
                const int j = jj * LPC + k;
                const float4 b4 = ld_shared_f4(st + j * WTP + 4 * q);
                const float4 c4 = ld_shared_f4(st + (NS + j) * WTP + 4 * q);
                const float2 bv[2] = AUSSM_F22(b4), cv2[2] = AUSSM_F22(c4);
                const float cv[4] = AUSSM_F4(c4);
                const float2 x[2] = {__fmul2_rn(s[0], bv[0]), __fmul2_rn(s[1], bv[1])};
                float2 a[2], ht[2];                    // multipliers; the states after each step of the group
                multipliers(dlt2, f2(A2[jj]), a);
                const float h0 = sub[(q * SPT + jj) * 32 + lane];
                four_steps(h0, a, x, ht);
                // eta_t = C_t w_t + a_{t+1} eta_{t+1}
                float2 g[2], ag[2];
                g[1].y = fmaf(cv[3], w[3], eps[jj]);
                ag[1].y = a[1].y * g[1].y;
                g[1].x = fmaf(cv[2], w[2], ag[1].y);
                ag[1].x = a[1].x * g[1].x;
                g[0].y = fmaf(cv[1], w[1], ag[1].x);
                ag[0].y = a[0].y * g[0].y;
                g[0].x = fmaf(cv[0], w[0], ag[0].y);
                ag[0].x = a[0].x * g[0].x;
                eps[jj] = ag[0].x;
                const float2 hp[2] = {make_float2(h0, ht[0].x), make_float2(ht[0].y, ht[1].x)};   // before each step
                float2 gB[2], gC[2];
#pragma unroll
                for (int p2 = 0; p2 < 2; ++p2) {
                    const float2 qa = __fmul2_rn(ag[p2], hp[p2]);                // a_t eta_t h_{t-1}
                    dA2[jj] = __ffma2_rn(qa, dlt2[p2], dA2[jj]);
                    SQ2[p2] = __ffma2_rn(qa, f2(A2[jj]), SQ2[p2]);               // times ln 2 below
                    SY2[p2] = __ffma2_rn(g[p2], bv[p2], SY2[p2]);
                    SP2[p2] = __ffma2_rn(cv2[p2], ht[p2], SP2[p2]);
                    gB[p2] = __fmul2_rn(g[p2], s[p2]);
                    gC[p2] = __fmul2_rn(w2[p2], ht[p2]);
                }
                st_shared_f4(red + (j * RP + c) * 4, make_float4(gB[0].x, gB[0].y, gB[1].x, gB[1].y));
                st_shared_f4(red + ((NS + j) * RP + c) * 4, make_float4(gC[0].x, gC[0].y, gC[1].x, gC[1].y));
            }
            const float SQ[4] = {SQ2[0].x, SQ2[0].y, SQ2[1].x, SQ2[1].y};
            const float SY[4] = {SY2[0].x, SY2[0].y, SY2[1].x, SY2[1].y};
            const float SP[4] = {SP2[0].x, SP2[0].y, SP2[1].x, SP2[1].y};
            __syncwarp();
            // dB, dC: lane r adds row r over the warp's channels, one vector atomic per state and group
#pragma unroll
            for (int x = 0; x < RROWS; ++x) {
                const int row = x * 32 + lane;
                if (row < 2 * NS) {
                    float4 acc = ld_shared_f4(red + (row * RP) * 4);
#pragma unroll
                    for (int l = 1; l < CPW; ++l) {
                        const float4 v = ld_shared_f4(red + (row * RP + l) * 4);
                        acc.x += v.x; acc.y += v.y; acc.z += v.z; acc.w += v.w;
                    }
                    if (red_on[x]) red_add_v4w(red_dst[x] + t0 + 4 * q, acc);
                }
            }
            // the channel's d delta, du, dz of the group replace delta, u, z in the stage
            float dd[4], du[4], dz[4];
            const float4 zz4 = gate ? ld_shared_f4(zrow + 4 * q) : make_float4(0.f, 0.f, 0.f, 0.f);   // gout silu'(z)
            const float zz[4] = AUSSM_F4(zz4);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float sy = channel_sum<LPC>(SY[e]), sq = channel_sum<LPC>(SQ[e]);
                float ddl = fmaf(uv[e], sy, sq * kLn2);
                if (softplus) ddl *= -expm1f(-dlt[e]);                // softplus'(x) = sigmoid(x) = 1 - exp(-softplus(x))
                dd[e] = ddl;
                du[e] = fmaf(dlt[e], sy, w[e] * dskip);
                if (gate) dz[e] = zz[e] * fmaf(dskip, uv[e], channel_sum<LPC>(SP[e]));
                db_acc += ddl;
                dD_acc = fmaf(w[e], uv[e], dD_acc);
            }
            __syncwarp();                       // every lane of the channel has read this group's cells
            if (k == 0) {
                st_shared_f4(urow + 4 * q, make_float4(du[0], du[1], du[2], du[3]));
                st_shared_f4(drow + 4 * q, make_float4(dd[0], dd[1], dd[2], dd[3]));
                if (gate) st_shared_f4(zrow + 4 * q, make_float4(dz[0], dz[1], dz[2], dz[3]));
            }
        }
        __syncwarp();
        map.store(st + C::BC_FLOATS, p.du, t0, tlen, lane);
        map.store(st + C::BC_FLOATS + C::AUX_FLOATS, p.ddelta, t0, tlen, lane);
        if (gate) map.store(st + C::BC_FLOATS + 2 * C::AUX_FLOATS, p.dz, t0, tlen, lane);
        __syncwarp();
        const int nr = r + WSTAGES;
        if (nr < last - first) {
            const int nt = last - 1 - nr;
            map.issue(st, aux_src, (long long)nt * WT, min(WT, L - nt * WT), lane);
        } else {
            cp_async_commit();
        }
    }
    cp_async_wait<0>();
    if (act) {
        const long long o = ((long long)b * max(1, p.nseg) + seg) * p.Dmod + i;
#pragma unroll
        for (int jj = 0; jj < SPT; ++jj)
            if (jj * LPC + k < N) p.part_A[o * N + jj * LPC + k] = dA2[jj].x + dA2[jj].y;
        if (k == 0) {
            p.part_D[o] = dD_acc;
            p.part_bias[o] = db_acc;
        }
    }
}

// ---------------------------------------------------------------------------
// Time-axis split: the segments' summaries and the chain through them.  With S the sum of a segment's step sizes its
// multipliers' product is exp(A S), so a segment is summed up by S and
//     forward    e = its end state from zero                     (the recurrence without the output)
//     backward   l = sum_t exp(A S_t) C_t w_t                    (S_t the sum up to step t, w = gout silu(z)): the
//                    gradient its outputs send to the state before it; no recurrence, 3 operations and one exponential
// Forward: e of segment s lies in the state record where segment s + 1 starts and S one tile into segment s (two
// entries that the real pass overwrites), the chain turns the e's into true start states in place.
// ---------------------------------------------------------------------------
template <int NS, int LPC>
__global__ void __launch_bounds__(32) s6w_fwd_summary_kernel(const S6FwdParams p) {
    using C = WCfg<NS, LPC, false>;
    constexpr int SPT = C::SPT, CPW = C::CPW;
    extern __shared__ __align__(128) float smem[];
    const int lane = threadIdx.x;
    const int c = lane / LPC, k = lane % LPC;
    const int tasks_per_batch = (p.Dmod + CPW - 1) / CPW;
    const int tasks = tasks_per_batch * (p.nch / p.Dmod);
    const int seg = (int)(blockIdx.x / tasks), task = blockIdx.x % tasks;
    const int b = task / tasks_per_batch, i0 = (task % tasks_per_batch) * CPW;
    const int nvalid = min(CPW, p.Dmod - i0);
    const bool act = c < nvalid;
    const int i = i0 + min(c, nvalid - 1);
    const long long ch0 = (long long)b * p.Dmod + i0, ch = (long long)b * p.Dmod + i;
    const int N = p.N, L = p.L, ntiles = (L + WT - 1) / WT;
    const int first = seg * p.seg_tiles, last = first + p.seg_tiles;      // never the last segment: whole tiles
    float A2[SPT], h[SPT], S = 0.f;
#pragma unroll
    for (int jj = 0; jj < SPT; ++jj) {
        const int j = jj * LPC + k;
        A2[jj] = j < N ? p.A[(long long)i * N + j] * kLog2e : 0.f;
        h[jj] = 0.f;
    }
    const float bias = p.delta_bias ? p.delta_bias[i] : 0.f;
    const bool softplus = p.delta_softplus != 0;
    for (int x = lane; x < WSTAGES * C::STAGE_FLOATS; x += 32) smem[x] = 0.f;
    __syncwarp();
    const float* aux_src[C::AUX] = {p.u, p.delta, nullptr};
    WMap<C> map;
    map.init(lane, nvalid, N, L, p.Bm + (long long)b * N * L, p.Cm + (long long)b * N * L, ch0);
    for (int s = 0; s < WSTAGES; ++s) {
        const int t = first + s;
        if (t < last) map.issue(smem + (t % WSTAGES) * C::STAGE_FLOATS, aux_src, (long long)t * WT, WT, lane);
        else cp_async_commit();
    }
    for (int tile = first; tile < last; ++tile) {
        float* st = smem + (tile % WSTAGES) * C::STAGE_FLOATS;
        float* urow = st + C::BC_FLOATS + c * WTP;
        float* drow = urow + C::AUX_FLOATS;
        cp_async_wait<WSTAGES - 1>();
        __syncwarp();
#pragma unroll
        for (int x = 0; x < C::PRE_STEPS; x += 4) {
            const int t = k * C::PRE_STEPS + x;
            const float4 d4 = ld_shared_f4(drow + t);
            float dv[4] = AUSSM_F4(d4);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                dv[e] += bias;
                if (softplus) dv[e] = softplus_(dv[e]);
                S += dv[e];
            }
            st_shared_f4(drow + t, make_float4(dv[0], dv[1], dv[2], dv[3]));
        }
        __syncwarp();
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const float4 u4 = ld_shared_f4(urow + 4 * q), d4 = ld_shared_f4(drow + 4 * q);
            const float uv[4] = AUSSM_F4(u4), dlt[4] = AUSSM_F4(d4);
#pragma unroll
            for (int jj = 0; jj < SPT; ++jj) {
                const float4 b4 = ld_shared_f4(st + (jj * LPC + k) * WTP + 4 * q);
                const float bv[4] = AUSSM_F4(b4);
#pragma unroll
                for (int e = 0; e < 4; ++e) h[jj] = fmaf(ex2_ftz(dlt[e] * A2[jj]), h[jj], dlt[e] * uv[e] * bv[e]);
            }
        }
        __syncwarp();
        const int nt = tile + WSTAGES;
        if (nt < last) map.issue(st, aux_src, (long long)nt * WT, WT, lane);
        else cp_async_commit();
    }
    cp_async_wait<0>();
    S = channel_sum<LPC>(S);
    if (act) {
        float* ck = p.ckpt + ch * ntiles * N;
#pragma unroll
        for (int jj = 0; jj < SPT; ++jj)
            if (jj * LPC + k < N) ck[(long long)last * N + jj * LPC + k] = h[jj];
        if (k == 0) ck[(long long)(first + 1) * N] = S;
    }
}

template <int NS, int LPC>
__global__ void __launch_bounds__(32) s6w_bwd_summary_kernel(const S6BwdParams p) {
    using C = WCfg<NS, LPC, false>;                       // rows: delta, z, gout
    constexpr int SPT = C::SPT, CPW = C::CPW;
    extern __shared__ __align__(128) float smem[];
    const int lane = threadIdx.x;
    const int c = lane / LPC, k = lane % LPC;
    const int tasks_per_batch = (p.Dmod + CPW - 1) / CPW;
    const int tasks = tasks_per_batch * (p.nch / p.Dmod);
    const int seg = 1 + (int)(blockIdx.x / tasks), task = blockIdx.x % tasks;
    const int b = task / tasks_per_batch, i0 = (task % tasks_per_batch) * CPW;
    const int nvalid = min(CPW, p.Dmod - i0);
    const bool act = c < nvalid;
    const int i = i0 + min(c, nvalid - 1);
    const long long ch0 = (long long)b * p.Dmod + i0, ch = (long long)b * p.Dmod + i;
    const int N = p.N, L = p.L, ntiles = (L + WT - 1) / WT;
    const int first = seg * p.seg_tiles, last = min(ntiles, first + p.seg_tiles);     // never segment 0
    float A2[SPT], l[SPT], S = 0.f;
#pragma unroll
    for (int jj = 0; jj < SPT; ++jj) {
        const int j = jj * LPC + k;
        A2[jj] = j < N ? p.A[(long long)i * N + j] * kLog2e : 0.f;
        l[jj] = 0.f;
    }
    const float bias = p.delta_bias ? p.delta_bias[i] : 0.f;
    const bool softplus = p.delta_softplus != 0, gate = p.z != nullptr;
    for (int x = lane; x < WSTAGES * C::STAGE_FLOATS; x += 32) smem[x] = 0.f;
    __syncwarp();
    const float* aux_src[C::AUX] = {p.delta, p.z, p.gout};
    WMap<C> map;
    map.init(lane, nvalid, N, L, p.Bm + (long long)b * N * L, p.Cm + (long long)b * N * L, ch0);
    for (int s = 0; s < WSTAGES; ++s) {
        const int t = first + s;
        if (t < last) map.issue(smem + (t % WSTAGES) * C::STAGE_FLOATS, aux_src, (long long)t * WT, min(WT, L - t * WT), lane);
        else cp_async_commit();
    }
    for (int tile = first; tile < last; ++tile) {
        float* st = smem + (tile % WSTAGES) * C::STAGE_FLOATS;
        float* drow = st + C::BC_FLOATS + c * WTP;
        float* zrow = drow + C::AUX_FLOATS;
        float* grow = zrow + C::AUX_FLOATS;
        const int tlen = min(WT, L - tile * WT);
        cp_async_wait<WSTAGES - 1>();
        __syncwarp();
#pragma unroll
        for (int x = 0; x < C::PRE_STEPS; x += 4) {
            const int t = k * C::PRE_STEPS + x;
            const float4 d4 = ld_shared_f4(drow + t);
            float dv[4] = AUSSM_F4(d4);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                dv[e] += bias;
                if (softplus) dv[e] = softplus_(dv[e]);
            }
            st_shared_f4(drow + t, make_float4(dv[0], dv[1], dv[2], dv[3]));
            if (gate) {
                const float4 z4 = ld_shared_f4(zrow + t), g4 = ld_shared_f4(grow + t);
                st_shared_f4(grow + t, make_float4(g4.x * siluf_(z4.x), g4.y * siluf_(z4.y), g4.z * siluf_(z4.z),
                                                   g4.w * siluf_(z4.w)));
            }
        }
        __syncwarp();
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            if (4 * q >= tlen) break;
            const float4 d4 = ld_shared_f4(drow + 4 * q), w4 = ld_shared_f4(grow + 4 * q);
            const float w[4] = AUSSM_F4(w4);
            const float at[4] = {S + d4.x, S + d4.x + d4.y, S + d4.x + d4.y + d4.z, S + d4.x + d4.y + d4.z + d4.w};
            S = at[3];
#pragma unroll
            for (int jj = 0; jj < SPT; ++jj) {
                const float4 c4 = ld_shared_f4(st + (NS + jj * LPC + k) * WTP + 4 * q);
                const float cv[4] = AUSSM_F4(c4);
#pragma unroll
                for (int e = 0; e < 4; ++e) l[jj] = fmaf(ex2_ftz(at[e] * A2[jj]), cv[e] * w[e], l[jj]);
            }
        }
        __syncwarp();
        const int nt = tile + WSTAGES;
        if (nt < last) map.issue(st, aux_src, (long long)nt * WT, min(WT, L - nt * WT), lane);
        else cp_async_commit();
    }
    cp_async_wait<0>();
    if (act) {
        const long long o = ch * p.nseg + seg;
#pragma unroll
        for (int jj = 0; jj < SPT; ++jj)
            if (jj * LPC + k < N) p.seg_grad[o * N + jj * LPC + k] = l[jj];
        if (k == 0) p.seg_delta[o] = S;
    }
}

// one thread per (channel, state): start states in place of the end states from zero
__global__ void __launch_bounds__(128) s6w_fwd_chain_kernel(const S6FwdParams p, int ntiles) {
    const long long id = (long long)blockIdx.x * 128 + threadIdx.x;
    if (id >= (long long)p.nch * p.N) return;
    const long long ch = id / p.N;
    const int j = (int)(id % p.N);
    const float A2 = p.A[(ch % p.Dmod) * p.N + j] * kLog2e;
    float* ck = p.ckpt + ch * ntiles * p.N;
    float h = 0.f;
    for (int seg = 0; seg + 1 < p.nseg; ++seg) {
        const float S = ck[((long long)seg * p.seg_tiles + 1) * p.N];
        float* at = ck + (long long)(seg + 1) * p.seg_tiles * p.N + j;
        h = fmaf(ex2_ftz(A2 * S), h, *at);
        *at = h;
    }
}

// one thread per (channel, state): seg_grad of segment s turns from l_s into the gradient of the state after s
__global__ void __launch_bounds__(128) s6w_bwd_chain_kernel(const S6BwdParams p) {
    const long long id = (long long)blockIdx.x * 128 + threadIdx.x;
    if (id >= (long long)p.nch * p.N) return;
    const long long ch = id / p.N;
    const int j = (int)(id % p.N);
    const float A2 = p.A[(ch % p.Dmod) * p.N + j] * kLog2e;
    float g = 0.f;
    for (int seg = p.nseg - 1; seg >= 0; --seg) {
        const long long o = ch * p.nseg + seg;
        const float l = seg > 0 ? p.seg_grad[o * p.N + j] : 0.f, S = seg > 0 ? p.seg_delta[o] : 0.f;
        p.seg_grad[o * p.N + j] = g;
        g = fmaf(ex2_ftz(A2 * S), g, l);
    }
}

// second stage of the parameter gradients: partials added over the batch entries (and segments) in a fixed order
__global__ void __launch_bounds__(256) s6_reduce_kernel(const S6ReduceParams p) {
    const long long o = (long long)blockIdx.x * 256 + threadIdx.x;
    const long long DN = (long long)p.D * p.N;
    if (o < DN) {
        float acc = 0.f;
        for (int b = 0; b < p.batch; ++b) acc += p.part_A[(long long)b * DN + o];
        p.dA[o] = acc;
    } else if (o < DN + p.D) {
        const long long i = o - DN;
        float aD = 0.f, ab = 0.f;
        for (int b = 0; b < p.batch; ++b) {
            aD += p.part_D[(long long)b * p.D + i];
            ab += p.part_bias[(long long)b * p.D + i];
        }
        if (p.dD) p.dD[i] = aD;
        if (p.dbias) p.dbias[i] = ab;
    }
}

// Lanes per channel for a launch.  Forward: one is the cheapest per step; more when the channels alone give too few
// warps (about three per scheduler hide the latencies of the dependent chains).  Backward: two measured best at
// every size tried (batch 8 x 2048 channels x 4096 steps: 2.75 / 2.32 / 3.37 ms with 1 / 2 / 4 lanes; batch 32 x
// 4096 x 1024: 4.83 / 4.14 / 4.64 ms) - one lane per channel needs every register there is, four repeat the
// per-channel work of a group four times; four only when even two give less than one warp per scheduler, and for more
// than 16 states, where four keep the eight states per thread that two keep for 16.
int lanes_per_channel(long long batches, int D, int NS, bool bwd) {
    static int sms = 0;                                     // the GPUs of a box are alike
    if (sms <= 0) {
        int dev = 0, n = 0;
        if (cudaGetDevice(&dev) == cudaSuccess &&
            cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess && n > 0)
            sms = n;
        else
            sms = 148;
    }
    auto warps = [&](int lpc) { return batches * ((D + 32 / lpc - 1) / (32 / lpc)); };
    if (bwd) return warps(2) < 4LL * sms ? 4 : 2;
    int lpc = NS > 16 ? 2 : 1;                              // 32 states of one thread do not fit its registers
    while (lpc < 4 && lpc * 2 <= NS && warps(lpc) < 12LL * sms) lpc *= 2;
    return lpc;
}

template <class C, class K, class P>
cudaError_t launch_w(K kern, const P& p, int segments, cudaStream_t stream) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    const long long tasks = (long long)(p.nch / p.Dmod) * ((p.Dmod + C::CPW - 1) / C::CPW);
    kern<<<(unsigned)(tasks * segments), 32, C::SMEM_BYTES, stream>>>(p);
    count_launch();
    return cudaGetLastError();
}

unsigned chain_blocks(long long nch, int N) { return (unsigned)((nch * N + 127) / 128); }

template <int NS, int LPC>
cudaError_t launch_w_fwd(const S6FwdParams& p, cudaStream_t stream) {
    using C = WCfg<NS, LPC, false>;
    return launch_w<C>(s6w_fwd_kernel<NS, LPC>, p, p.nseg > 1 ? p.nseg : 1, stream);
}

template <int NS, int LPC>
cudaError_t launch_w_bwd(const S6BwdParams& p, cudaStream_t stream) {
    using C = WCfg<NS, LPC, true>;
    return launch_w<C>(s6w_bwd_kernel<NS, LPC>, p, p.nseg > 1 ? p.nseg : 1, stream);
}

// lanes per channel of a launch that is cut along the time axis: eight states per thread at most
template <int NS>
constexpr int split_lanes() { return NS > 16 ? 4 : 2; }

template <int NS>
cudaError_t launch_w_fwd_split(const S6FwdParams& p, cudaStream_t stream) {
    constexpr int LPC = split_lanes<NS>();
    using C = WCfg<NS, LPC, false>;
    cudaError_t e = launch_w<C>(s6w_fwd_summary_kernel<NS, LPC>, p, p.nseg - 1, stream);
    if (e != cudaSuccess) return e;
    s6w_fwd_chain_kernel<<<chain_blocks(p.nch, p.N), 128, 0, stream>>>(p, (p.L + WT - 1) / WT);
    count_launch();
    e = cudaGetLastError();
    return e != cudaSuccess ? e : launch_w_fwd<NS, LPC>(p, stream);
}

template <int NS>
cudaError_t launch_w_bwd_split(const S6BwdParams& p, cudaStream_t stream) {
    constexpr int LPC = split_lanes<NS>();
    using C = WCfg<NS, LPC, false>;
    cudaError_t e = launch_w<C>(s6w_bwd_summary_kernel<NS, LPC>, p, p.nseg - 1, stream);
    if (e != cudaSuccess) return e;
    s6w_bwd_chain_kernel<<<chain_blocks(p.nch, p.N), 128, 0, stream>>>(p);
    count_launch();
    e = cudaGetLastError();
    return e != cudaSuccess ? e : launch_w_bwd<NS, LPC>(p, stream);
}

template <int NS>
cudaError_t launch_w_fwd_ns(const S6FwdParams& p, cudaStream_t stream) {
    if (p.nseg > 1) return launch_w_fwd_split<NS>(p, stream);
    switch (lanes_per_channel(p.nch / p.Dmod, p.Dmod, NS, false)) {
        case 4: return launch_w_fwd<NS, 4>(p, stream);
        case 2: return launch_w_fwd<NS, 2>(p, stream);
        default: return launch_w_fwd<NS, 1>(p, stream);
    }
}

template <int NS>
cudaError_t launch_w_bwd_ns(const S6BwdParams& p, cudaStream_t stream) {
    if (p.nseg > 1) return launch_w_bwd_split<NS>(p, stream);
    if constexpr (NS > 16) {
        return launch_w_bwd<NS, 4>(p, stream);
    } else {
        if (lanes_per_channel(p.nch / p.Dmod, p.Dmod, NS, true) == 4) return launch_w_bwd<NS, 4>(p, stream);
        return launch_w_bwd<NS, 2>(p, stream);
    }
}

}  // namespace

// A launch whose channels give few warps (two lanes per channel) is cut along the time axis.  The backward kernel
// holds 8 warps per SM (shared memory) and its summary pass costs an eighth of it: worth it below 4 warps per SM, as
// many segments as fill one wave.  The forward summary costs two thirds of the real pass, which reaches its rate at
// about 7 warps per SM: worth it below 3.  A segment keeps at least 64 steps; short sequences stay whole (the two
// extra launches cost what they save).  N = 16, forward + backward, whole -> split: B1 D512 L8192 3357 -> 368 us (forward
// alone 767 -> 140), B2 D1024 L2048 898 -> 348 us, B4 D512 L1024 487 -> 260 us, B4 D2048 L4096 (3.5 warps per SM)
// 2067 -> 1863 us; B2 D256 N4 L300 216 -> 224 us (bound by the host).
S6Plan s6_split_plan(long long batches, int D, int N, int L, bool bwd) {
    S6Plan plan = {1, (L + WT - 1) / WT};
    if (N > 32 || L < 512 || !time_split_option()) return plan;
    constexpr long long SMS = 148;                          // fixed: a workspace sized with the plan always fits
    const int per_warp = N > 16 ? 8 : 16;                   // channels
    const long long warps = batches * ((D + per_warp - 1) / per_warp);
    if (warps >= (bwd ? 4 : 3) * SMS) return plan;
    const long long want = std::min<long long>((bwd ? 8 : 14) * SMS / warps, L / 64);
    if (want < 2) return plan;
    const int tiles = plan.seg_tiles;
    plan.seg_tiles = (int)((tiles + want - 1) / want);
    plan.nseg = (tiles + plan.seg_tiles - 1) / plan.seg_tiles;
    return plan;
}

cudaError_t launch_s6_fwd(const S6FwdParams& p_, cudaStream_t stream) {
    if (p_.nch <= 0 || p_.L <= 0) return cudaSuccess;
    S6FwdParams p = p_;
    p.nseg = 1;
    if (p.ckpt) {                                           // the split hands states on through the record
        const S6Plan plan = s6_split_plan(p.nch / p.Dmod, p.Dmod, p.N, p.L, false);
        p.nseg = plan.nseg;
        p.seg_tiles = plan.seg_tiles;
    }
    if (p.N <= 4) return launch_w_fwd_ns<4>(p, stream);
    if (p.N <= 8) return launch_w_fwd_ns<8>(p, stream);
    if (p.N <= 16) return launch_w_fwd_ns<16>(p, stream);
    if (p.N <= 32) return launch_w_fwd_ns<32>(p, stream);
    return cudaErrorInvalidValue;
}

cudaError_t launch_s6_bwd(const S6BwdParams& p, cudaStream_t stream) {
    if (p.nch <= 0 || p.L <= 0) return cudaSuccess;
    if (p.N <= 4) return launch_w_bwd_ns<4>(p, stream);
    if (p.N <= 8) return launch_w_bwd_ns<8>(p, stream);
    if (p.N <= 16) return launch_w_bwd_ns<16>(p, stream);
    if (p.N <= 32) return launch_w_bwd_ns<32>(p, stream);
    return cudaErrorInvalidValue;
}

cudaError_t launch_s6_reduce(const S6ReduceParams& p, cudaStream_t stream) {
    const long long total = (long long)p.D * p.N + p.D;
    s6_reduce_kernel<<<(unsigned)((total + 255) / 256), 256, 0, stream>>>(p);
    count_launch();
    return cudaGetLastError();
}

}  // namespace aussm
