// Unitary selective-scan core for sm_100a: forward and backward kernels.
//
// Operator (per channel ch = (b, i), state j, step t), theta given:
//     h_t = exp(i*theta_t) h_{t-1} + Bc_j s_t,   s_t = dt_t * silu(u_t)
//     y_t = silu(z_t) * (D_i silu(u_t) + sum_j Re(Cc_j h_t))
// It replaces the scan part of the reference kernels
// csrc/cuda/ssm_adaptive_unitary_forward.cu:112-187 and
// csrc/cuda/ssm_adaptive_unitary_backward.cu:143-417 (the phase projection,
// forward.cu:83-110 / backward.cu:419-490, is a separate contraction).
//
// Work decomposition.  One thread owns SPT states of one channel and walks
// the time axis sequentially, so the recurrence costs four fused
// multiply-adds per step and needs no scan tree.  A warp owns 32/NL channels
// (NL lanes per channel) and is independent of every other warp: it has its
// own ring of shared-memory stages and the kernels contain no block-wide
// barrier.  The theta rows of a warp (contiguous in time in HBM, one row per
// state) are staged with 16-byte asynchronous copies, consecutive lanes
// fetching consecutive pieces of a row (fully coalesced 128-bit loads), into
// rows padded by 16 bytes so that the per-thread 128-bit shared loads of a
// quarter-warp hit disjoint banks.  Sums over the states of a channel go
// through the same tile: every thread overwrites the four phases it has just
// consumed with its four contributions, and after the tile the lanes switch
// roles (one lane = one channel and a few consecutive steps) to add the NL
// rows and emit y with coalesced vector stores.
//
// Lanes whose state or channel does not exist (N < NL*SPT, or the last warp
// of the grid) shadow a valid row: they load and process real data with a
// zero output weight and store nothing, so the inner loops carry no
// predicates.
//
// State normalisation: with Bc != 0 the kernels carry h/Bc instead of h, so
// that the input term is the real number s_t (two multiply-adds less per
// step) and the output projection uses the single constant M = Cc*Bc.
//
// Backward: because |exp(i*theta)| = 1 the recurrence is reversible,
// h_{t-1} = exp(-i*theta_t)(h_t - Bc s_t); the kernel starts from the final
// state that the forward pass returned and walks time backwards, regenerating
// the states while it runs the adjoint recurrence
//     eta_t = conj(Cc) w_t + exp(-i*theta_{t+1}) eta_{t+1},   w_t = gy_t silu(z_t)
// so nothing but the inputs and the final state is ever stored.  dtheta is
// written in place of theta in the stage and leaves with coalesced stores.
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "scan_unitary.cuh"

namespace aussm {

__device__ int g_device_status = 0;

int* device_status_ptr() {
    int* ptr = nullptr;
    if (cudaGetSymbolAddress(reinterpret_cast<void**>(&ptr), g_device_status) != cudaSuccess) return nullptr;
    return ptr;
}

cudaError_t read_and_clear_device_status(cudaStream_t stream, int* value) {
    cudaError_t e = cudaStreamSynchronize(stream);
    if (e != cudaSuccess) return e;
    e = cudaMemcpyFromSymbol(value, g_device_status, sizeof(int));
    if (e != cudaSuccess) return e;
    if (*value != 0) {
        const int zero = 0;
        e = cudaMemcpyToSymbol(g_device_status, &zero, sizeof(int));
    }
    return e;
}

namespace {

constexpr float kFloatMax = 3.402823466e38f;

constexpr int cmin(int a, int b) { return a < b ? a : b; }

// Shape of one warp's work.  NL lanes per channel, SPT states per thread,
// T steps per stage, TS steps per backward sub-block, AUX per-channel rows.
template <int NL_, int SPT_, int T_, int TS_, int STAGES_, int WARPS_, int AUX_, bool BWD_>
struct Cfg {
    static constexpr int NL = NL_, SPT = SPT_, T = T_, TS = TS_, STAGES = STAGES_, WARPS = WARPS_, AUX = AUX_;
    static constexpr int CPW = 32 / NL;                 // channels per warp
    static constexpr int TP = T + 4;                    // padded row pitch (floats)
    static constexpr int TSP = TS + 4;
    static constexpr int NROWS = 32 * SPT;
    static constexpr int STAGE_FLOATS = NROWS * TP + CPW * AUX * T;
    // backward only, not staged: two column-sum tiles and the s / w / silu'(u) rows of a sub-block
    static constexpr int SCRATCH_FLOATS = BWD_ ? 2 * 32 * TSP + CPW * 3 * TS : 0;
    static constexpr int WARP_FLOATS = STAGES * STAGE_FLOATS + SCRATCH_FLOATS;
    static constexpr size_t SMEM_BYTES = (size_t)WARPS * WARP_FLOATS * sizeof(float);
    // asynchronous-copy instructions per lane and tile
    static constexpr int CHUNKS_PER_ROW = T / 4;
    static constexpr int NCH_THETA = NROWS * CHUNKS_PER_ROW / 32;
    static constexpr int NCH_AUX = (CPW * AUX * CHUNKS_PER_ROW + 31) / 32;
    // per-(channel, step) passes: every lane owns VW consecutive steps of one channel
    static constexpr int EPL = CPW * TS / 32;           // elements per lane and sub-block
    static constexpr int VW = cmin(4, EPL);
    static constexpr int ITERS = EPL / VW;
    static_assert(T % TS == 0 && T % 4 == 0 && TS % 4 == 0, "tile shape");
    static_assert((NROWS * CHUNKS_PER_ROW) % 32 == 0, "theta chunks must fill whole warps");
    static_assert(CPW * TS >= 32 && (CPW * TS) % 32 == 0, "pass mapping");
};

template <int NL, int SPT, int T, int STAGES, int WARPS>
using FwdCfg = Cfg<NL, SPT, T, T, STAGES, WARPS, 3, false>;     // aux rows: u, dt (becomes s), z
template <int NL, int SPT, int T, int TS, int STAGES, int WARPS>
using BwdCfg = Cfg<NL, SPT, T, TS, STAGES, WARPS, 4, true>;     // aux rows: u, dt, z, gy

struct StateConsts {
    float mr, mi;      // M: projection constant (Cc*Bc normalised, Cc otherwise)
    float br, bi;      // Bc
    float kr, ki;      // state scale kappa (Bc normalised, 1 otherwise)
    bool act;
};

__device__ __forceinline__ void load_state_consts(StateConsts& sc, bool act, int j,
                                                  const float* B_r, const float* B_theta, const float* C_r,
                                                  const float* C_theta, bool& norm_ok) {
    sc.act = act;
    sc.mr = sc.mi = sc.br = sc.bi = 0.f;
    sc.kr = 1.f;
    sc.ki = 0.f;
    norm_ok = true;
    if (!act) return;
    float brad = B_r[j], bth = B_theta[j], crad = C_r[j], cth = C_theta[j];
    float sb, cb, scc, ccc;
    sincosf(bth, &sb, &cb);
    sincosf(cth, &scc, &ccc);
    sc.br = brad * cb;
    sc.bi = brad * sb;
    sc.mr = crad * ccc;   // Cc for now
    sc.mi = crad * scc;
    norm_ok = fabsf(brad) >= 1e-12f;
}

// switch the constants of an active state to the normalised representation
__device__ __forceinline__ void normalise_consts(StateConsts& sc, float& ccr, float& cci) {
    ccr = sc.mr;
    cci = sc.mi;
    if (!sc.act) return;
    sc.kr = sc.br;
    sc.ki = sc.bi;
    float mr = ccr * sc.br - cci * sc.bi;
    float mi = ccr * sc.bi + cci * sc.br;
    sc.mr = mr;
    sc.mi = mi;
}

// (ar + i ai) / (kr + i ki), scaled to stay in range for tiny |k|
__device__ __forceinline__ void cdiv(float ar, float ai, float kr, float ki, float& qr, float& qi) {
    float inv = rsqrtf(kr * kr + ki * ki);
    float ur = kr * inv, ui = ki * inv;     // unit vector of k
    float tr = ar * inv, ti = ai * inv;     // a / |k|
    qr = tr * ur + ti * ui;                 // times conj(unit)
    qi = ti * ur - tr * ui;
}

// A warp's work: CPW consecutive channels and, when the time axis is split, one segment of it.  The segments are
// seg_len steps (a multiple of the tile), the last one what is left; all channels of a warp share the segment.
// SEG = false: a launch without segments.  Length and start then come from the parameters and not from the warp's
// index, so loop bounds and addresses stay uniform.  It is compiled (FOLD at the launchers) for the tile shapes whose
// whole launches it makes faster; what it does to the others is the register allocation (N <= 4 forward: 114 -> 96, N <=
// 8 backward 110 -> 80, with fewer loads in flight).  Calls with / without the segment form, us:
//     N, B D L             forward      backward
//     4,  8 512 4096       168 / 191    308 / 284
//     8,  8 512 4096       191 / 200    345 / 365
//     16, 2 1024 8192      396 / 361    598 / 613
//     32, 8 512 2048       298 / 288    546 / 531
//     64, 8 256 2048       324 / 312    750 / 732
//     128, 4 256 2048      416 / 474    978 / 957
struct WarpTask {
    long long ch0;      // first channel
    int nvalid;         // channels that exist
    int seg, nseg;      // segment and number of segments (1: no split)
    long long t0;       // first step of the segment
    int L;              // its steps
    // entry of the per-segment state arrays that belongs to channel ch0 + c
    __device__ __forceinline__ long long entry(int c) const { return (ch0 + c) * nseg + seg; }
};
template <int CPW, bool SEG, class P>
__device__ __forceinline__ bool warp_task(const P& p, long long task, WarpTask& w) {
    const long long groups = ((long long)p.nch + CPW - 1) / CPW;
    if (!SEG) {
        if (task >= groups) return false;
        w.seg = 0;
        w.nseg = 1;
        w.ch0 = task * CPW;
        w.nvalid = (int)min((long long)CPW, (long long)p.nch - w.ch0);
        w.t0 = 0;
        w.L = p.L;
        return true;
    }
    w.nseg = p.nseg > 1 ? p.nseg : 1;
    if (task >= groups * w.nseg) return false;
    w.seg = w.nseg > 1 ? (int)(task / groups) : 0;
    w.ch0 = (task - w.seg * groups) * CPW;
    w.nvalid = (int)min((long long)CPW, (long long)p.nch - w.ch0);
    w.t0 = (long long)w.seg * p.seg_len;
    w.L = w.nseg > 1 ? (int)min((long long)p.seg_len, (long long)p.L - w.t0) : p.L;
    return true;
}

// ---------------------------------------------------------------------------
// Tile movement
// ---------------------------------------------------------------------------
// Where a warp's rows live in global memory, as seen by one lane: the source
// of every 16-byte piece this lane copies per tile (at step 0 of the launch).
template <class C>
struct TileMap {
    unsigned theta_off[C::NCH_THETA];     // byte offset from the warp's first theta row (32 bits: base + offset addressing)
    const float* aux_ptr[C::NCH_AUX];     // per-channel rows (nullptr: this lane has no piece)

    __device__ __forceinline__ void init(int lane, int nvalid, int N, long long ld_theta, const float* const* aux_src,
                                         long long aux_row0, long long ld_row) {
#pragma unroll
        for (int i = 0; i < C::NCH_THETA; ++i) {
            const int id = i * 32 + lane;
            const int slot = id / C::CHUNKS_PER_ROW, col = id % C::CHUNKS_PER_ROW;
            const int k = slot / 32, w = slot % 32;
            const int c = w / C::NL, j = (w % C::NL) + k * C::NL;
            const bool ok = c < nvalid && j < N;
            // missing rows shadow the warp's first row
            const long long row = ok ? (long long)(c * N + j) * ld_theta : 0;
            theta_off[i] = (unsigned)((row + col * 4) * (long long)sizeof(float));
        }
#pragma unroll
        for (int i = 0; i < C::NCH_AUX; ++i) {
            const int id = i * 32 + lane;
            const int row = id / C::CHUNKS_PER_ROW, col = id % C::CHUNKS_PER_ROW;
            aux_ptr[i] = nullptr;
            if (row < C::CPW * C::AUX) {
                const int cc = row / C::AUX, a = row % C::AUX;
                aux_ptr[i] = aux_src[a] + aux_row0 + (cc < nvalid ? cc : 0) * ld_row + col * 4;
            }
        }
    }

    // queue the asynchronous copies of one tile and close the group (FULL: a whole tile, no per-piece bound check).
    // Piece i of a lane lands at a compile-time distance from the lane's first piece, so every destination is
    // one register plus an immediate.
    template <bool FULL>
    __device__ __forceinline__ void issue_t(float* stage, const float* theta_t0, long long t0, int tlen,
                                            int lane) const {
        constexpr int CPR = C::CHUNKS_PER_ROW, RPI = 32 / CPR;       // rows covered by one warp-wide instruction
        static_assert(32 % CPR == 0, "pieces per row must divide the warp");
        const int col = lane % CPR;
        const uint32_t dst0 = smem_addr(stage) + (uint32_t)(((lane / CPR) * C::TP + col * 4) * sizeof(float));
#pragma unroll
        for (int i = 0; i < C::NCH_THETA; ++i) {
            if (FULL || col * 4 < tlen)
                cp_async16_s(dst0 + (uint32_t)(i * RPI * C::TP * sizeof(float)),
                             reinterpret_cast<const char*>(theta_t0) + theta_off[i]);
        }
        const uint32_t aux0 = smem_addr(stage) +
                              (uint32_t)((C::NROWS * C::TP + (lane / CPR) * C::T + col * 4) * sizeof(float));
#pragma unroll
        for (int i = 0; i < C::NCH_AUX; ++i) {
            if (aux_ptr[i] != nullptr && (FULL || col * 4 < tlen))
                cp_async16_s(aux0 + (uint32_t)(i * RPI * C::T * sizeof(float)), aux_ptr[i] + t0);
        }
        cp_async_commit();
    }
    __device__ __forceinline__ void issue(float* stage, const float* theta_warp, long long t0, int tlen,
                                          int lane) const {
        if (tlen == C::T) issue_t<true>(stage, theta_warp + t0, t0, tlen, lane);
        else issue_t<false>(stage, theta_warp + t0, t0, tlen, lane);
    }
};

// Tile copy for launches whose rows are not 16-byte aligned (odd lengths, shifted bases): the same asynchronous
// ring with 4-byte pieces, one warp-wide instruction per row of 32 steps (consecutive lanes, consecutive words, so
// the rows' start does not matter).  Missing rows shadow the warp's first row; steps beyond tlen are not written.
// Four times the copy instructions of the 16-byte path, 1.4 more issue slots per step of about 26; the synchronous
// loads this replaces exposed the full memory latency of every tile.  B6 D300 N10 L1021, forward + backward through
// the Python front end: 1238 -> 220 us.
template <class C>
__device__ __forceinline__ void issue_words(float* stage, const float* theta_warp, long long ld_theta,
                                            const float* const* aux_src, long long aux_row0, long long ld_row,
                                            int nvalid, int N, long long t0, int tlen, int lane) {
    static_assert(C::T == 32, "one lane per step");
    if (lane < tlen) {
        const float* src = theta_warp + t0 + lane;
        const uint32_t dst = smem_addr(stage) + (uint32_t)(lane * sizeof(float));
#pragma unroll
        for (int slot = 0; slot < C::NROWS; ++slot) {
            const int c = (slot % 32) / C::NL, j = slot % C::NL + (slot / 32) * C::NL;
            const long long row = (c < nvalid && j < N) ? (long long)(c * N + j) : 0;
            cp_async4_s(dst + (uint32_t)(slot * C::TP * sizeof(float)), src + row * ld_theta);
        }
        const uint32_t aux = dst + (uint32_t)(C::NROWS * C::TP * sizeof(float));
#pragma unroll
        for (int a = 0; a < C::AUX; ++a) {
            const float* asrc = aux_src[a] + aux_row0 + t0 + lane;
#pragma unroll
            for (int cc = 0; cc < C::CPW; ++cc)
                cp_async4_s(aux + (uint32_t)((cc * C::AUX + a) * C::T * sizeof(float)),
                            asrc + (cc < nvalid ? cc : 0) * ld_row);
        }
    }
    cp_async_commit();
}

// ---------------------------------------------------------------------------
// Forward
// ---------------------------------------------------------------------------
// VEC: rows are 16-byte aligned and L is a multiple of 4 (16-byte copies and vector stores).
template <class C, bool VEC, bool NORM>
__device__ __forceinline__ void fwd_warp(const ScanFwdParams& p, float* wsm, const WarpTask& wt, int lane,
                                         StateConsts (&sc)[C::SPT]) {
    constexpr int NL = C::NL, SPT = C::SPT, T = C::T, TP = C::TP, STAGES = C::STAGES, AUX = C::AUX, VW = C::VW;
    const int c = lane / NL, jl = lane % NL;
    const long long ch = wt.entry(c);
    const int N = p.N, L = wt.L, nvalid = wt.nvalid;
    const int ntiles = (L + T - 1) / T;
    const float* theta_warp = p.theta + wt.ch0 * N * p.ld_theta + wt.t0;
    const long long row0 = wt.ch0 * p.ld_row + wt.t0;           // this warp's first row of u, dt, z, y
    const float* aux_src[AUX] = {p.u, p.dt, p.z};

    float hr[SPT], hi[SPT];
#pragma unroll
    for (int k = 0; k < SPT; ++k) {
        const int j = jl + k * NL;
        hr[k] = hi[k] = 0.f;
        if (sc[k].act) {
            float ar = p.h0_re ? p.h0_re[ch * N + j] : 0.f;
            float ai = p.h0_im ? p.h0_im[ch * N + j] : 0.f;
            if (NORM) cdiv(ar, ai, sc[k].kr, sc[k].ki, hr[k], hi[k]);
            else { hr[k] = ar; hi[k] = ai; }
        }
    }
    // skip weight and output row of the channel each per-(channel, step) item of this lane belongs to
    float dval[C::ITERS];
    long long ybase[C::ITERS];
#pragma unroll
    for (int it = 0; it < C::ITERS; ++it) {
        const int cc = ((lane + 32 * it) * VW) / T;
        dval[it] = cc < nvalid ? p.Dskip[(wt.ch0 + cc) % p.Dmod] : 0.f;
        ybase[it] = row0 + (cc < nvalid ? cc : 0) * p.ld_row;
    }

    TileMap<C> map;
    if (VEC) map.init(lane, nvalid, N, p.ld_theta, aux_src, row0, p.ld_row);
    auto fetch = [&](float* stage, const int tile) {
        const int len = min(T, L - tile * T);
        if (VEC) map.issue(stage, theta_warp, (long long)tile * T, len, lane);
        else issue_words<C>(stage, theta_warp, p.ld_theta, aux_src, row0, p.ld_row, nvalid, N, (long long)tile * T, len,
                            lane);
    };
    for (int s = 0; s < STAGES; ++s) {
        if (s < ntiles) fetch(wsm + s * C::STAGE_FLOATS, s);
        else cp_async_commit();
    }

    for (int tile = 0; tile < ntiles; ++tile) {
        float* th = wsm + (tile % STAGES) * C::STAGE_FLOATS;
        float* aux = th + C::NROWS * TP;
        const long long t0 = (long long)tile * T;
        const int tlen = min(T, L - (int)t0);
        const int nq = (tlen + 3) >> 2;
        cp_async_wait<STAGES - 1>();
        __syncwarp();

        // pre-pass: v = silu(u) over the u row, s = dt * v over the dt row
#pragma unroll
        for (int it = 0; it < C::ITERS; ++it) {
            const int e0 = (lane + 32 * it) * VW;
            const int cc = e0 / T, t = e0 % T;
            if (t < tlen) {
                Vec<VW> u, d;
                u.ld(aux + (cc * AUX + 0) * T + t);
                d.ld(aux + (cc * AUX + 1) * T + t);
#pragma unroll
                for (int e = 0; e < VW; ++e) {
                    u.v[e] = siluf_(u.v[e]);
                    d.v[e] *= u.v[e];
                }
                u.st(aux + (cc * AUX + 0) * T + t);      // the u row now holds silu(u) for the post-pass
                d.st(aux + (cc * AUX + 1) * T + t);
            }
        }
        __syncwarp();

        // scan: SPT states per thread, four steps per shared-memory access
        const float* srow = aux + (c * AUX + 1) * T;
        auto quad = [&](const int q, auto whole) {
            const float4 s4 = ld_shared_f4(srow + 4 * q);
            const float sv[4] = {s4.x, s4.y, s4.z, s4.w};
            float pacc[4];
#pragma unroll
            for (int k = 0; k < SPT; ++k) {
                const float4 t4 = ld_shared_f4(th + (k * 32 + lane) * TP + 4 * q);
                const float tv[4] = {t4.x, t4.y, t4.z, t4.w};
                float sn[4], cs[4];
                sincos4(tv, sn, cs);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    if (!VEC && !whole.value && 4 * q + e >= tlen) {           // ragged tail
                        if (k == 0) pacc[e] = 0.f;
                        continue;
                    }
                    float nr, ni;
                    if (NORM) {
                        nr = fmaf(cs[e], hr[k], fmaf(-sn[e], hi[k], sv[e]));
                        ni = fmaf(cs[e], hi[k], sn[e] * hr[k]);
                    } else {
                        nr = fmaf(cs[e], hr[k], fmaf(-sn[e], hi[k], sc[k].br * sv[e]));
                        ni = fmaf(cs[e], hi[k], fmaf(sn[e], hr[k], sc[k].bi * sv[e]));
                    }
                    hr[k] = nr;
                    hi[k] = ni;
                    pacc[e] = (k == 0) ? fmaf(sc[k].mr, nr, -sc[k].mi * ni)
                                       : fmaf(sc[k].mr, nr, fmaf(-sc[k].mi, ni, pacc[e]));
                }
            }
            st_shared_f4(th + lane * TP + 4 * q, make_float4(pacc[0], pacc[1], pacc[2], pacc[3]));
        };
        if (tlen == T) {
#pragma unroll
            for (int q = 0; q < T / 4; ++q) quad(q, std::true_type{});
        } else {
            for (int q = 0; q < nq; ++q) quad(q, std::false_type{});
        }
        __syncwarp();

        // post-pass: one lane = one channel and VW steps
        if (p.y) {
#pragma unroll
            for (int it = 0; it < C::ITERS; ++it) {
                const int e0 = (lane + 32 * it) * VW;
                const int cc = e0 / T, t = e0 % T;
                if (t < tlen && cc < nvalid) {
                    Vec<VW> acc, u, z;
                    acc.ld(th + cc * NL * TP + t);
#pragma unroll
                    for (int r = 1; r < NL; ++r) {
                        Vec<VW> v;
                        v.ld(th + (cc * NL + r) * TP + t);
                        acc.add(v);
                    }
                    u.ld(aux + (cc * AUX + 0) * T + t);      // silu(u), left by the pre-pass
                    z.ld(aux + (cc * AUX + 2) * T + t);
#pragma unroll
                    for (int e = 0; e < VW; ++e) acc.v[e] = siluf_(z.v[e]) * fmaf(dval[it], u.v[e], acc.v[e]);
                    float* dst = p.y + ybase[it] + t0 + t;
                    if (VEC) {
                        acc.st(dst);      // global pointers take the same vector stores
                    } else {
                        for (int e = 0; e < VW; ++e)
                            if (t + e < tlen) dst[e] = acc.v[e];
                    }
                }
            }
        }
        __syncwarp();
        if (tile + STAGES < ntiles) fetch(th, tile + STAGES);
        else cp_async_commit();
    }
    cp_async_wait<0>();

#pragma unroll
    for (int k = 0; k < SPT; ++k) {
        if (sc[k].act && p.h1_re) {
            const int j = jl + k * NL;
            float orr = hr[k], oi = hi[k];
            if (NORM) {
                orr = sc[k].kr * hr[k] - sc[k].ki * hi[k];
                oi = sc[k].kr * hi[k] + sc[k].ki * hr[k];
            }
            p.h1_re[ch * N + j] = orr;
            p.h1_im[ch * N + j] = oi;
        }
    }
}

template <class C, bool VEC, bool SEG>
__global__ void __launch_bounds__(C::WARPS * 32) scan_unitary_fwd_kernel(const ScanFwdParams p) {
    extern __shared__ __align__(128) float smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    WarpTask wt;
    if (!warp_task<C::CPW, SEG>(p, (long long)blockIdx.x * C::WARPS + warp, wt)) return;   // no block barriers
    const int nvalid = wt.nvalid;
    float* wsm = smem + (size_t)warp * C::WARP_FLOATS;
    const int c = lane / C::NL, jl = lane % C::NL;
    StateConsts sc[C::SPT];
    bool ok = true;
#pragma unroll
    for (int k = 0; k < C::SPT; ++k) {
        const int j = jl + k * C::NL;
        bool okk;
        load_state_consts(sc[k], c < nvalid && j < p.N, j, p.B_r, p.B_theta, p.C_r, p.C_theta, okk);
        ok = ok && okk;
    }
    if (__all_sync(0xffffffffu, ok)) {
#pragma unroll
        for (int k = 0; k < C::SPT; ++k) {
            float a, b;
            normalise_consts(sc[k], a, b);
        }
        fwd_warp<C, VEC, true>(p, wsm, wt, lane, sc);
    } else {
        fwd_warp<C, VEC, false>(p, wsm, wt, lane, sc);
    }
}

// ---------------------------------------------------------------------------
// Backward
// ---------------------------------------------------------------------------
// SUMS (the drop-in pipeline): the sums of dtheta over time and its largest magnitude are collected.
template <class C, bool VEC, bool NORM, bool SUMS>
__device__ __forceinline__ void bwd_warp(const ScanBwdParams& p, float* wsm, const WarpTask& wt, int lane,
                                         StateConsts (&sc)[C::SPT], const float (&ccr)[C::SPT],
                                         const float (&cci)[C::SPT]) {
    constexpr int NL = C::NL, SPT = C::SPT, T = C::T, TS = C::TS, TP = C::TP, TSP = C::TSP, STAGES = C::STAGES,
                  AUX = C::AUX, VW = C::VW;
    const int c = lane / NL, jl = lane % NL;
    const long long ch = wt.entry(c);
    const int N = p.N, L = wt.L, nvalid = wt.nvalid;
    const int ntiles = (L + T - 1) / T;
    const float* theta_warp = p.theta + wt.ch0 * N * p.ld_theta + wt.t0;
    float* dtheta_warp = p.dtheta + wt.ch0 * N * p.ld_theta + wt.t0;      // launcher guarantees equal pitches
    const long long row0 = wt.ch0 * p.ld_row + wt.t0;

    float* scratch = wsm + STAGES * C::STAGE_FLOATS;
    float* pt = scratch;                    // [32][TSP] projections, summed over a thread's states
    float* et = pt + 32 * TSP;              // [32][TSP] Re(eta)
    float* sw = et + 32 * TSP;              // [CPW][3][TS]: s row, w row, d silu(u)/du row

    float hr[SPT], hi[SPT];     // state h_t (normalised), walking backwards
    float er[SPT], ei[SPT];     // exp(-i theta_{t+1}) eta_{t+1}
    float gmr[SPT], gmi[SPT];   // sum_t w_t conj(h_t)
    float sbr[SPT], sbi[SPT];   // sum_t eta_t s_t              (general representation only)
    float amax = 0.f;           // largest finite |dtheta| seen by this thread (spares its split a pass of its own)
    float rsum[SPT];            // sum_t dtheta_t
    float hlr[SPT], hli[SPT];   // conj(h_{L-1}) . gh   (boundary term of the Bc gradient)
#pragma unroll
    for (int k = 0; k < SPT; ++k) {
        const int j = jl + k * NL;
        hr[k] = hi[k] = er[k] = ei[k] = gmr[k] = gmi[k] = sbr[k] = sbi[k] = rsum[k] = hlr[k] = hli[k] = 0.f;
        if (sc[k].act) {
            const float ar = p.h1_re[ch * N + j], ai = p.h1_im[ch * N + j];
            const float gr = p.gh1_re ? p.gh1_re[ch * N + j] : 0.f;
            const float gi = p.gh1_im ? p.gh1_im[ch * N + j] : 0.f;
            if (NORM) {
                cdiv(ar, ai, sc[k].kr, sc[k].ki, hr[k], hi[k]);
                // gradient w.r.t. the normalised state: conj(kappa) * gh
                er[k] = sc[k].kr * gr + sc[k].ki * gi;
                ei[k] = sc[k].kr * gi - sc[k].ki * gr;
                // conj(h~_{L-1}) * gh
                if (wt.seg == wt.nseg - 1) {
                    hlr[k] = hr[k] * gr + hi[k] * gi;
                    hli[k] = hr[k] * gi - hi[k] * gr;
                }
            } else {
                hr[k] = ar; hi[k] = ai; er[k] = gr; ei[k] = gi;
            }
        }
    }
    float dval[C::ITERS], dacc[C::ITERS];
    long long obase[C::ITERS];
#pragma unroll
    for (int it = 0; it < C::ITERS; ++it) {
        const int cc = ((lane + 32 * it) * VW) / TS;
        dval[it] = cc < nvalid ? p.Dskip[(wt.ch0 + cc) % p.Dmod] : 0.f;
        dacc[it] = 0.f;
        obase[it] = row0 + (cc < nvalid ? cc : 0) * p.ld_row;
    }
    const float* aux_src[AUX] = {p.u, p.dt, p.z, p.gy};

    // r counts tiles in processing order (last tile first)
    TileMap<C> map;
    if (VEC) map.init(lane, nvalid, N, p.ld_theta, aux_src, row0, p.ld_row);
    auto fetch = [&](float* stage, const int tile) {
        const int len = min(T, L - tile * T);
        if (VEC) map.issue(stage, theta_warp, (long long)tile * T, len, lane);
        else issue_words<C>(stage, theta_warp, p.ld_theta, aux_src, row0, p.ld_row, nvalid, N, (long long)tile * T, len,
                            lane);
    };
    for (int r = 0; r < STAGES; ++r) {
        if (r < ntiles) fetch(wsm + r * C::STAGE_FLOATS, ntiles - 1 - r);
        else cp_async_commit();
    }

    for (int r = 0; r < ntiles; ++r) {
        const int tile = ntiles - 1 - r;
        float* th = wsm + (r % STAGES) * C::STAGE_FLOATS;
        float* aux = th + C::NROWS * TP;
        const long long t0 = (long long)tile * T;
        const int tlen = min(T, L - (int)t0);
        cp_async_wait<STAGES - 1>();
        __syncwarp();

        const int nsb = (tlen + TS - 1) / TS;
        for (int sb = nsb - 1; sb >= 0; --sb) {
            const int sbeg = sb * TS;                       // first step of the sub-block in the tile
            const int slen = min(TS, tlen - sbeg);
            const int nq = (slen + 3) >> 2;

            // pre-pass: every activation of the sub-block once.  s = dt silu(u), w = gy silu(z) feed the scan;
            // silu(u) and d silu(z)/dz replace the u and z rows, d silu(u)/du gets a row of its own.
#pragma unroll
            for (int it = 0; it < C::ITERS; ++it) {
                const int e0 = (lane + 32 * it) * VW;
                const int cc = e0 / TS, t = e0 % TS;
                if (t < slen) {
                    const int o = sbeg + t;
                    Vec<VW> u, d, z, g, gu;
                    u.ld(aux + (cc * AUX + 0) * T + o);
                    d.ld(aux + (cc * AUX + 1) * T + o);
                    z.ld(aux + (cc * AUX + 2) * T + o);
                    g.ld(aux + (cc * AUX + 3) * T + o);
#pragma unroll
                    for (int e = 0; e < VW; ++e) {
                        float gz;
                        u.v[e] = silu_and_grad(u.v[e], gu.v[e]);
                        d.v[e] *= u.v[e];
                        g.v[e] *= silu_and_grad(z.v[e], gz);
                        z.v[e] = gz;
                    }
                    u.st(aux + (cc * AUX + 0) * T + o);
                    z.st(aux + (cc * AUX + 2) * T + o);
                    d.st(sw + (cc * 3 + 0) * TS + t);
                    g.st(sw + (cc * 3 + 1) * TS + t);
                    gu.st(sw + (cc * 3 + 2) * TS + t);
                }
            }
            __syncwarp();

            // reverse scan
            float tmax = 0.f;
            auto quad = [&](const int q, auto whole) {
                const float4 s4 = ld_shared_f4(sw + (c * 3 + 0) * TS + 4 * q);
                const float4 w4 = ld_shared_f4(sw + (c * 3 + 1) * TS + 4 * q);
                const float sv[4] = {s4.x, s4.y, s4.z, s4.w};
                const float wv[4] = {w4.x, w4.y, w4.z, w4.w};
                float pacc[4], eacc[4];
#pragma unroll
                for (int k = 0; k < SPT; ++k) {
                    float* cell = th + (k * 32 + lane) * TP + sbeg + 4 * q;
                    const float4 t4 = ld_shared_f4(cell);
                    const float tv[4] = {t4.x, t4.y, t4.z, t4.w};
                    float sn[4], cs[4];
                    sincos4(tv, sn, cs);
                    float dth[4];
#pragma unroll
                    for (int e = 3; e >= 0; --e) {
                        if (!VEC && !whole.value && 4 * q + e >= slen) {
                            dth[e] = 0.f;
                            if (k == 0) { pacc[e] = 0.f; eacc[e] = 0.f; }
                            continue;
                        }
                        const float w = wv[e], s = sv[e];
                        // eta_t = carry + conj(M) w
                        const float nr = fmaf(sc[k].mr, w, er[k]);
                        const float ni = fmaf(-sc[k].mi, w, ei[k]);
                        // a = h_t - beta s  (= exp(i theta_t) h_{t-1})
                        float ar, ai;
                        if (NORM) { ar = hr[k] - s; ai = hi[k]; }
                        else { ar = fmaf(-sc[k].br, s, hr[k]); ai = fmaf(-sc[k].bi, s, hi[k]); }
                        // dtheta_t = -Im(conj(eta) a)
                        const float d = fmaf(ni, ar, -nr * ai);
                        dth[e] = d;
                        if (SUMS) { rsum[k] += d; tmax = fmaxf(tmax, fabsf(d)); }
                        const float pv = fmaf(sc[k].mr, hr[k], -sc[k].mi * hi[k]);
                        // gradient of the real drive s_t: Re(conj(eta) beta)
                        const float ev = NORM ? nr : fmaf(nr, sc[k].br, ni * sc[k].bi);
                        pacc[e] = (k == 0) ? pv : pacc[e] + pv;
                        eacc[e] = (k == 0) ? ev : eacc[e] + ev;
                        gmr[k] = fmaf(w, hr[k], gmr[k]);
                        gmi[k] = fmaf(-w, hi[k], gmi[k]);
                        if (!NORM) { sbr[k] = fmaf(nr, s, sbr[k]); sbi[k] = fmaf(ni, s, sbi[k]); }
                        // step back: h_{t-1} = conj(lambda) a ; carry = conj(lambda) eta
                        hr[k] = fmaf(cs[e], ar, sn[e] * ai);
                        hi[k] = fmaf(cs[e], ai, -sn[e] * ar);
                        er[k] = fmaf(cs[e], nr, sn[e] * ni);
                        ei[k] = fmaf(cs[e], ni, -sn[e] * nr);
                    }
                    st_shared_f4(cell, make_float4(dth[0], dth[1], dth[2], dth[3]));
                }
                st_shared_f4(pt + lane * TSP + 4 * q, make_float4(pacc[0], pacc[1], pacc[2], pacc[3]));
                st_shared_f4(et + lane * TSP + 4 * q, make_float4(eacc[0], eacc[1], eacc[2], eacc[3]));
            };
            if (slen == TS) {
#pragma unroll
                for (int q = TS / 4 - 1; q >= 0; --q) quad(q, std::true_type{});
            } else {
                for (int q = nq - 1; q >= 0; --q) quad(q, std::false_type{});
            }
            if (SUMS) {
                // an infinity (like a NaN, which fmaxf passes over) spoils its own row, not the scale of all others
                if (tmax > kFloatMax) {
                    tmax = 0.f;
#pragma unroll 1
                    for (int k = 0; k < SPT; ++k)
#pragma unroll 1
                        for (int t = 0; t < slen; ++t) {
                            const float d = fabsf(th[(k * 32 + lane) * TP + sbeg + t]);
                            if (d <= kFloatMax) tmax = fmaxf(tmax, d);
                        }
                }
                amax = fmaxf(amax, tmax);
            }
            __syncwarp();

            // post-pass: du, ddt, dz for one channel and VW steps per lane
#pragma unroll
            for (int it = 0; it < C::ITERS; ++it) {
                const int e0 = (lane + 32 * it) * VW;
                const int cc = e0 / TS, t = e0 % TS;
                if (t < slen && cc < nvalid) {
                    Vec<VW> P, E, v, d, gz, g, w, gu, du, ddt, dz;
                    P.ld(pt + cc * NL * TSP + t);
                    E.ld(et + cc * NL * TSP + t);
#pragma unroll
                    for (int rr = 1; rr < NL; ++rr) {
                        Vec<VW> a, b;
                        a.ld(pt + (cc * NL + rr) * TSP + t);
                        b.ld(et + (cc * NL + rr) * TSP + t);
                        P.add(a);
                        E.add(b);
                    }
                    const int o = sbeg + t;
                    v.ld(aux + (cc * AUX + 0) * T + o);       // silu(u)
                    d.ld(aux + (cc * AUX + 1) * T + o);
                    gz.ld(aux + (cc * AUX + 2) * T + o);      // d silu(z)/dz
                    g.ld(aux + (cc * AUX + 3) * T + o);
                    w.ld(sw + (cc * 3 + 1) * TS + t);         // gy silu(z)
                    gu.ld(sw + (cc * 3 + 2) * TS + t);
                    const float dv = dval[it];
#pragma unroll
                    for (int e = 0; e < VW; ++e) {
                        dz.v[e] = g.v[e] * fmaf(dv, v.v[e], P.v[e]) * gz.v[e];
                        ddt.v[e] = E.v[e] * v.v[e];
                        du.v[e] = fmaf(E.v[e], d.v[e], w.v[e] * dv) * gu.v[e];
                        if (VEC || t + e < slen) dacc[it] = fmaf(w.v[e], v.v[e], dacc[it]);
                    }
                    const long long off = obase[it] + t0 + o;
                    if (VEC) {
                        du.st(p.du + off);
                        ddt.st(p.ddt + off);
                        dz.st(p.dz + off);
                    } else {
                        for (int e = 0; e < VW; ++e) {
                            if (t + e < slen) {
                                p.du[off + e] = du.v[e];
                                p.ddt[off + e] = ddt.v[e];
                                p.dz[off + e] = dz.v[e];
                            }
                        }
                    }
                }
            }
            __syncwarp();
        }

        // dtheta leaves the stage: coalesced 16-byte stores, same piece-to-lane map as the loads
        if (VEC) {
            constexpr int CPR = C::CHUNKS_PER_ROW, RPI = 32 / CPR;
            const int col = lane % CPR;
            const float* src0 = th + (lane / CPR) * TP + col * 4;
            float* dst0 = dtheta_warp + t0;
            auto leave = [&](const int i) {
                *reinterpret_cast<float4*>(reinterpret_cast<char*>(dst0) + map.theta_off[i]) =
                    ld_shared_f4(src0 + i * RPI * TP);
            };
            if (nvalid == C::CPW && N == NL * SPT && tlen == T) {      // whole tile, every row real: no per-piece test
#pragma unroll
                for (int i = 0; i < C::NCH_THETA; ++i) leave(i);
            } else {
#pragma unroll
                for (int i = 0; i < C::NCH_THETA; ++i) {
                    const int slot = i * RPI + lane / CPR;
                    const int k = slot / 32, w = slot % 32;
                    const bool real_row = (w / NL) < nvalid && ((w % NL) + k * NL) < N;
                    if (real_row && col * 4 < tlen) leave(i);
                }
            }
        } else if (lane < tlen) {                       // one row of 32 steps per instruction
            float* dst = dtheta_warp + t0 + lane;
            const float* src = th + lane;
#pragma unroll
            for (int slot = 0; slot < C::NROWS; ++slot) {
                const int cc = (slot % 32) / NL, j = slot % NL + (slot / 32) * NL;
                if (cc < nvalid && j < N) dst[(long long)(cc * N + j) * p.ld_theta] = src[slot * TP];
            }
        }
        __syncwarp();
        if (r + STAGES < ntiles) fetch(th, ntiles - 1 - r - STAGES);
        else cp_async_commit();
    }
    cp_async_wait<0>();

    // ---- per-(channel, state) results ----
#pragma unroll
    for (int k = 0; k < SPT; ++k) {
        if (!sc[k].act) continue;
        const int j = jl + k * NL;
        const long long o = ch * N + j;                                          // states and their gradients
        const long long po = ((wt.ch0 + c) * p.part_nseg + wt.seg) * N + j;      // partial sums
        float dbr, dbi, dcr, dci, d0r, d0i, s0r, s0i;
        if (NORM) {
            const float kr = sc[k].kr, ki = sc[k].ki;
            // dCc = conj(Bc) G_M
            dcr = kr * gmr[k] + ki * gmi[k];
            dci = kr * gmi[k] - ki * gmr[k];
            // dBc = conj(Cc) G_M + conj(h~_{L-1}) gh - conj(h~_{-1} / Bc) carry.  The boundary terms of neighbouring
            // segments cancel; they are left out, because each is as large as the sum (with them dBc of B1 D200 N16
            // L20001 was off by several times the error of an unsplit launch).
            float qr, qi;
            cdiv(hr[k], hi[k], kr, ki, qr, qi);
            dbr = ccr[k] * gmr[k] + cci[k] * gmi[k];
            dbi = ccr[k] * gmi[k] - cci[k] * gmr[k];
            if (wt.seg == wt.nseg - 1) { dbr += hlr[k]; dbi += hli[k]; }
            if (wt.seg == 0) { dbr -= qr * er[k] + qi * ei[k]; dbi -= qr * ei[k] - qi * er[k]; }
            // dh0 = carry / conj(Bc) ;  h0 = Bc h~_{-1}
            cdiv(er[k], ei[k], kr, -ki, d0r, d0i);
            s0r = kr * hr[k] - ki * hi[k];
            s0i = kr * hi[k] + ki * hr[k];
        } else {
            dcr = gmr[k]; dci = gmi[k]; dbr = sbr[k]; dbi = sbi[k];
            d0r = er[k]; d0i = ei[k]; s0r = hr[k]; s0i = hi[k];
        }
        float4* pb = reinterpret_cast<float4*>(p.part_bc) + po;
        if (p.accumulate) {
            const float4 old = *pb;
            dbr += old.x; dbi += old.y; dcr += old.z; dci += old.w;
        }
        *pb = make_float4(dbr, dbi, dcr, dci);
        if (SUMS) p.part_rowsum[po] = rsum[k] + (p.accumulate ? p.part_rowsum[po] : 0.f);
        if (p.dh0_re) { p.dh0_re[o] = d0r; p.dh0_im[o] = d0i; }
        if (p.h0_re) { p.h0_re[o] = s0r; p.h0_im[o] = s0i; }
    }
    if (SUMS) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) amax = fmaxf(amax, __shfl_xor_sync(0xffffffffu, amax, o));
        if (lane == 0 && amax > 0.f) atomicMax(p.dtheta_amax, __float_as_uint(fminf(amax, 3.0e38f)));
    }
    // dD: add the lanes' partial sums channel by channel through the scratch tile
    __syncwarp();
#pragma unroll
    for (int it = 0; it < C::ITERS; ++it) pt[lane + 32 * it] = dacc[it];
    __syncwarp();
    if (lane < nvalid) {
        // item idx covers elements [idx*VW, idx*VW+VW) of the CPW*TS block: channel = idx*VW/TS
        float acc = 0.f;
        for (int idx = 0; idx < 32 * C::ITERS; ++idx)
            if ((idx * VW) / TS == lane) acc += pt[idx];
        const long long o = (wt.ch0 + lane) * p.part_nseg + wt.seg;
        p.part_d[o] = acc + (p.accumulate ? p.part_d[o] : 0.f);
    }
}

template <class C, bool VEC, bool SUMS, bool SEG>
__global__ void __launch_bounds__(C::WARPS * 32) scan_unitary_bwd_kernel(const ScanBwdParams p) {
    extern __shared__ __align__(128) float smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    WarpTask wt;
    if (!warp_task<C::CPW, SEG>(p, (long long)blockIdx.x * C::WARPS + warp, wt)) return;
    const int nvalid = wt.nvalid;
    float* wsm = smem + (size_t)warp * C::WARP_FLOATS;
    const int c = lane / C::NL, jl = lane % C::NL;
    StateConsts sc[C::SPT];
    float ccr[C::SPT], cci[C::SPT];
    bool ok = true;
#pragma unroll
    for (int k = 0; k < C::SPT; ++k) {
        const int j = jl + k * C::NL;
        bool okk;
        load_state_consts(sc[k], c < nvalid && j < p.N, j, p.B_r, p.B_theta, p.C_r, p.C_theta, okk);
        ccr[k] = sc[k].mr;
        cci[k] = sc[k].mi;
        ok = ok && okk;
    }
    if (__all_sync(0xffffffffu, ok)) {
#pragma unroll
        for (int k = 0; k < C::SPT; ++k) normalise_consts(sc[k], ccr[k], cci[k]);
        bwd_warp<C, VEC, true, SUMS>(p, wsm, wt, lane, sc, ccr, cci);
    } else {
        bwd_warp<C, VEC, false, SUMS>(p, wsm, wt, lane, sc, ccr, cci);
    }
}

// ---------------------------------------------------------------------------
// Segment summary of the time-axis split: what a segment does to the state and to the adjoint, from its inputs alone.
// With a_t the product of the segment's rotations up to step t (|a_t| = 1, so conj(a_t) is its inverse)
//     end state from zero          e = a_end Bc sum_t conj(a_t) s_t
//     gradient sent to its start   l = conj(Cc) sum_t conj(a_t) w_t          (BWD; w_t = gy_t silu(z_t))
// so one forward walk gives a_end and both sums: 8 multiply-adds per step after the sine and cosine, against two
// walks over theta (aggregate and adjoint) before.  Bound by the FP32 pipe and the loads' latency about equally: 1023 us
// for the two passes of B1 D512 N16 L65536 (2 x 2.1 GB of phases, 0.62 of the copy bandwidth), where the two aggregate
// passes and the adjoint pass took 1710 us.
// ---------------------------------------------------------------------------
template <class C, bool VEC, bool BWD>
__global__ void __launch_bounds__(C::WARPS * 32) scan_unitary_summary_kernel(const SegSummaryParams p) {
    constexpr int NL = C::NL, SPT = C::SPT, T = C::T, TP = C::TP, STAGES = C::STAGES, AUX = C::AUX, VW = C::VW;
    extern __shared__ __align__(128) float smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    WarpTask wt;
    if (!warp_task<C::CPW, true>(p, (long long)blockIdx.x * C::WARPS + warp, wt)) return;
    const int nvalid = wt.nvalid;
    float* wsm = smem + (size_t)warp * C::WARP_FLOATS;
    const int c = lane / NL, jl = lane % NL;
    const int N = p.N, L = wt.L;
    const int ntiles = (L + T - 1) / T;
    StateConsts sc[SPT];
#pragma unroll
    for (int k = 0; k < SPT; ++k) {
        bool okk;
        load_state_consts(sc[k], c < nvalid && jl + k * NL < N, jl + k * NL, p.B_r, p.B_theta, p.C_r, p.C_theta, okk);      // mr, mi hold Cc
    }
    const float* theta_warp = p.theta + wt.ch0 * N * p.ld_theta + wt.t0;
    const long long row0 = wt.ch0 * p.ld_row + wt.t0;
    const float* aux_src[4] = {p.u, p.dt, p.z, p.gy};
    float ar[SPT], ai[SPT], hr[SPT], hi[SPT], gr[SPT], gi[SPT];
#pragma unroll
    for (int k = 0; k < SPT; ++k) {
        ar[k] = 1.f;
        ai[k] = hr[k] = hi[k] = gr[k] = gi[k] = 0.f;
    }
    TileMap<C> map;
    if (VEC) map.init(lane, nvalid, N, p.ld_theta, aux_src, row0, p.ld_row);
    auto fetch = [&](float* stage, const int tile) {
        const int len = min(T, L - tile * T);
        if (VEC) map.issue(stage, theta_warp, (long long)tile * T, len, lane);
        else issue_words<C>(stage, theta_warp, p.ld_theta, aux_src, row0, p.ld_row, nvalid, N, (long long)tile * T, len,
                            lane);
    };
    for (int s = 0; s < STAGES; ++s) {
        if (s < ntiles) fetch(wsm + s * C::STAGE_FLOATS, s);
        else cp_async_commit();
    }
    for (int tile = 0; tile < ntiles; ++tile) {
        float* th = wsm + (tile % STAGES) * C::STAGE_FLOATS;
        float* aux = th + C::NROWS * TP;
        const int tlen = min(T, L - tile * T);
        // conj(a) stands for 1/a below: bring |a| back to 1 (one Newton step; 32 roundings move it by about 1e-6)
#pragma unroll
        for (int k = 0; k < SPT; ++k) {
            const float r = fmaf(-0.5f, fmaf(ar[k], ar[k], ai[k] * ai[k]), 1.5f);
            ar[k] *= r;
            ai[k] *= r;
        }
        cp_async_wait<STAGES - 1>();
        __syncwarp();
        // pre-pass: s = dt silu(u) replaces dt, w = gy silu(z) replaces gy
#pragma unroll
        for (int it = 0; it < C::ITERS; ++it) {
            const int e0 = (lane + 32 * it) * VW;
            const int cc = e0 / T, t = e0 % T;
            if (t < tlen) {
                Vec<VW> a, b;
                a.ld(aux + (cc * AUX + 0) * T + t);
                b.ld(aux + (cc * AUX + 1) * T + t);
#pragma unroll
                for (int e = 0; e < VW; ++e) b.v[e] *= siluf_(a.v[e]);
                b.st(aux + (cc * AUX + 1) * T + t);
                if (BWD) {
                    a.ld(aux + (cc * AUX + 2) * T + t);
                    b.ld(aux + (cc * AUX + 3) * T + t);
#pragma unroll
                    for (int e = 0; e < VW; ++e) b.v[e] *= siluf_(a.v[e]);
                    b.st(aux + (cc * AUX + 3) * T + t);
                }
            }
        }
        __syncwarp();
        auto quad = [&](const int q, auto whole) {
            const float4 s4 = ld_shared_f4(aux + (c * AUX + 1) * T + 4 * q);
            const float4 w4 = BWD ? ld_shared_f4(aux + (c * AUX + 3) * T + 4 * q) : make_float4(0.f, 0.f, 0.f, 0.f);
            const float sv[4] = {s4.x, s4.y, s4.z, s4.w}, wv[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
            for (int k = 0; k < SPT; ++k) {
                const float4 t4 = ld_shared_f4(th + (k * 32 + lane) * TP + 4 * q);
                const float tv[4] = {t4.x, t4.y, t4.z, t4.w};
                float sn[4], cs[4];
                sincos4(tv, sn, cs);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    if (!VEC && !whole.value && 4 * q + e >= tlen) continue;           // ragged tail
                    const float nr = fmaf(cs[e], ar[k], -sn[e] * ai[k]);
                    ai[k] = fmaf(cs[e], ai[k], sn[e] * ar[k]);
                    ar[k] = nr;
                    hr[k] = fmaf(ar[k], sv[e], hr[k]);
                    hi[k] = fmaf(-ai[k], sv[e], hi[k]);
                    if (BWD) {
                        gr[k] = fmaf(ar[k], wv[e], gr[k]);
                        gi[k] = fmaf(-ai[k], wv[e], gi[k]);
                    }
                }
            }
        };
        if (tlen == T) {
#pragma unroll
            for (int q = 0; q < T / 4; ++q) quad(q, std::true_type{});
        } else {
            for (int q = 0; q < (tlen + 3) >> 2; ++q) quad(q, std::false_type{});
        }
        __syncwarp();
        if (tile + STAGES < ntiles) fetch(th, tile + STAGES);
        else cp_async_commit();
    }
    cp_async_wait<0>();
#pragma unroll
    for (int k = 0; k < SPT; ++k) {
        if (!sc[k].act) continue;
        const long long o = wt.entry(c) * N + jl + k * NL;
        p.a_re[o] = ar[k];
        p.a_im[o] = ai[k];
        const float br = sc[k].br * hr[k] - sc[k].bi * hi[k], bi = sc[k].br * hi[k] + sc[k].bi * hr[k];
        p.e_re[o] = ar[k] * br - ai[k] * bi;
        p.e_im[o] = ar[k] * bi + ai[k] * br;
        if (BWD) {
            p.l_re[o] = sc[k].mr * gr[k] + sc[k].mi * gi[k];
            p.l_im[o] = sc[k].mr * gi[k] - sc[k].mi * gr[k];
        }
    }
}

// ---------------------------------------------------------------------------
// Segment chains of the time-axis split: one thread per (channel, state) walks the nseg segments.  The loads do not
// depend on the chain, so a few segments of them are in flight.
// ---------------------------------------------------------------------------
struct SegChainParams {
    const float *e_re, *e_im, *a_re, *a_im;
    const float *l_re, *l_im;           // backward
    const float *from_re, *from_im;     // forward: state before segment 0 (or nullptr = 0); backward: the final state
    const float *gh_re, *gh_im;         // backward: gradient of the final state, or nullptr
    float *at_re, *at_im;               // forward: state before every segment; backward: state after it
    float *g_re, *g_im;                 // backward: gradient of the state after every segment
    float *end_re, *end_im;             // forward: final state; backward: state before segment 0 (or nullptr)
    float *dh0_re, *dh0_im;             // backward: gradient of that state (or nullptr)
    long long total;
    int nseg, N;
};

__global__ void __launch_bounds__(128) segment_states_fwd_kernel(const SegChainParams p) {
    const long long id = (long long)blockIdx.x * 128 + threadIdx.x;      // ch * N + j
    if (id >= p.total) return;
    const float *__restrict__ e_re = p.e_re, *__restrict__ e_im = p.e_im;
    const float *__restrict__ a_re = p.a_re, *__restrict__ a_im = p.a_im;
    float *__restrict__ at_re = p.at_re, *__restrict__ at_im = p.at_im;
    float cr = p.from_re ? p.from_re[id] : 0.f, ci = p.from_im ? p.from_im[id] : 0.f;
    long long o = (id / p.N) * p.nseg * p.N + id % p.N;
#pragma unroll 4
    for (int s = 0; s < p.nseg; ++s, o += p.N) {
        const float ar = a_re[o], ai = a_im[o], er = e_re[o], ei = e_im[o];
        at_re[o] = cr;
        at_im[o] = ci;
        const float nr = fmaf(ar, cr, fmaf(-ai, ci, er));               // c_{s+1} = e_s + a_s c_s
        ci = fmaf(ar, ci, fmaf(ai, cr, ei));
        cr = nr;
    }
    if (p.end_re) { p.end_re[id] = cr; p.end_im[id] = ci; }
}

// walking back from the final state: c_s = conj(a_s) (c_{s+1} - e_s) (|a_s| = 1) and g_s = l_s + conj(a_s) g_{s+1}
__global__ void __launch_bounds__(128) segment_states_bwd_kernel(const SegChainParams p) {
    const long long id = (long long)blockIdx.x * 128 + threadIdx.x;
    if (id >= p.total) return;
    const float *__restrict__ e_re = p.e_re, *__restrict__ e_im = p.e_im, *__restrict__ l_re = p.l_re;
    const float *__restrict__ a_re = p.a_re, *__restrict__ a_im = p.a_im, *__restrict__ l_im = p.l_im;
    float *__restrict__ at_re = p.at_re, *__restrict__ at_im = p.at_im;
    float *__restrict__ g_re = p.g_re, *__restrict__ g_im = p.g_im;
    float cr = p.from_re[id], ci = p.from_im[id];
    float gr = p.gh_re ? p.gh_re[id] : 0.f, gi = p.gh_im ? p.gh_im[id] : 0.f;
    long long o = ((id / p.N) * p.nseg + p.nseg - 1) * p.N + id % p.N;
#pragma unroll 4
    for (int s = 0; s < p.nseg; ++s, o -= p.N) {
        const float ar = a_re[o], ai = a_im[o], er = e_re[o], ei = e_im[o], lr = l_re[o], li = l_im[o];
        at_re[o] = cr;
        at_im[o] = ci;
        g_re[o] = gr;
        g_im[o] = gi;
        const float dr = cr - er, di = ci - ei;
        cr = fmaf(ar, dr, ai * di);
        ci = fmaf(ar, di, -ai * dr);
        const float nr = fmaf(ar, gr, fmaf(ai, gi, lr));
        gi = fmaf(ar, gi, fmaf(-ai, gr, li));
        gr = nr;
    }
    if (p.end_re) { p.end_re[id] = cr; p.end_im[id] = ci; }
    if (p.dh0_re) { p.dh0_re[id] = gr; p.dh0_im[id] = gi; }
}

// ---------------------------------------------------------------------------
// Second stage: fixed-order sums of the per-channel partials (deterministic)
// and the polar chain rule  dr = Re(conj(G) e^{i phi}),  dphi = -Im(conj(G) w).
// ---------------------------------------------------------------------------
// One block per state walks that state's partials of all channels.  There are only N such blocks, so what bounds them is
// the latency of their loads: 1024 threads with four loads in flight each (16384 channels, N = 16: 30 us with 256
// threads and one).
constexpr int REDUCE_THREADS = 1024;
__global__ void __launch_bounds__(REDUCE_THREADS) reduce_param_grads_kernel(const ReduceParams p) {
    __shared__ float4 red[REDUCE_THREADS];
    const int tid = threadIdx.x;
    const int nseg = p.nseg > 1 ? p.nseg : 1;               // partial arrays: nseg entries per channel
    const long long nch = (long long)p.batch * p.D * nseg;
    if (blockIdx.x < p.N) {
        const int j = blockIdx.x;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
        for (long long ch = tid; ch < nch; ch += 4 * REDUCE_THREADS) {
            float4 v[4];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const long long at = ch + (long long)k * REDUCE_THREADS;
                v[k] = at < nch ? reinterpret_cast<const float4*>(p.part_bc)[at * p.N + j] : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                acc.x += v[k].x; acc.y += v[k].y; acc.z += v[k].z; acc.w += v[k].w;
            }
        }
        red[tid] = acc;
        __syncthreads();
        for (int s = REDUCE_THREADS / 2; s > 0; s >>= 1) {
            if (tid < s) {
                float4 a = red[tid], b = red[tid + s];
                red[tid] = make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w);
            }
            __syncthreads();
        }
        if (tid == 0) {
            const float4 g = red[0];
            float sb, cb, sc_, cc_;
            sincosf(p.B_theta[j], &sb, &cb);
            sincosf(p.C_theta[j], &sc_, &cc_);
            const float br = p.B_r[j], cr = p.C_r[j];
            p.dB_r[j] = g.x * cb + g.y * sb;
            p.dB_theta[j] = br * (g.y * cb - g.x * sb);
            p.dC_r[j] = g.z * cc_ + g.w * sc_;
            p.dC_theta[j] = cr * (g.w * cc_ - g.z * sc_);
        }
        return;
    }
    // remaining blocks: dD (D values) then dx_bias (D*N values), one thread per output
    const long long o = (long long)(blockIdx.x - p.N) * REDUCE_THREADS + tid;
    if (o < p.D) {
        float acc = 0.f;
        for (int b = 0; b < p.batch; ++b)
            for (int sg = 0; sg < nseg; ++sg) acc += p.part_d[((long long)b * p.D + o) * nseg + sg];
        p.dD[o] = acc;
    } else if (p.dx_bias && o - p.D < (long long)p.D * p.N) {
        const long long e = o - p.D;
        const long long i = e / p.N, j = e % p.N;
        float acc = 0.f;
        for (int b = 0; b < p.batch; ++b)
            for (int sg = 0; sg < nseg; ++sg)
                acc += p.part_rowsum[(((long long)b * p.D + i) * nseg + sg) * p.N + j];
        p.dx_bias[e] = acc;
    }
}

// ---------------------------------------------------------------------------
// Launchers
// ---------------------------------------------------------------------------
inline bool aligned16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// warp tasks of a launch: channel groups times segments
template <class C, class P>
long long warp_tasks(const P& p) {
    return (((long long)p.nch + C::CPW - 1) / C::CPW) * (p.nseg > 1 ? p.nseg : 1);
}

template <class C, bool VEC, bool SEG>
cudaError_t launch_fwd_cfg(const ScanFwdParams& p, cudaStream_t stream) {
    auto kern = scan_unitary_fwd_kernel<C, VEC, SEG>;
    const size_t smem = C::SMEM_BYTES;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const long long blocks = (warp_tasks<C>(p) + C::WARPS - 1) / C::WARPS;
    kern<<<(unsigned)blocks, C::WARPS * 32, smem, stream>>>(p);
    count_launch();
    return cudaGetLastError();
}

template <class C, bool VEC, bool SUMS, bool SEG>
cudaError_t launch_bwd_cfg(const ScanBwdParams& p, cudaStream_t stream) {
    auto kern = scan_unitary_bwd_kernel<C, VEC, SUMS, SEG>;
    const size_t smem = C::SMEM_BYTES;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const long long blocks = (warp_tasks<C>(p) + C::WARPS - 1) / C::WARPS;
    kern<<<(unsigned)blocks, C::WARPS * 32, smem, stream>>>(p);
    count_launch();
    return cudaGetLastError();
}

// Runtime properties -> template parameters.  FOLD: whole launches have a form of their own (see warp_task).
template <class C, bool FOLD>
cudaError_t launch_fwd_sel(const ScanFwdParams& p, bool vec, cudaStream_t s) {
    if (!vec) return launch_fwd_cfg<C, false, true>(p, s);
    if constexpr (FOLD) {
        if (p.nseg <= 1) return launch_fwd_cfg<C, true, false>(p, s);
    }
    return launch_fwd_cfg<C, true, true>(p, s);
}

template <class C, bool FOLD, bool SUMS>
cudaError_t launch_bwd_sums(const ScanBwdParams& p, bool vec, cudaStream_t s) {
    if (!vec) return launch_bwd_cfg<C, false, SUMS, true>(p, s);
    if constexpr (FOLD) {
        if (p.nseg <= 1) return launch_bwd_cfg<C, true, SUMS, false>(p, s);
    }
    return launch_bwd_cfg<C, true, SUMS, true>(p, s);
}

template <class C, bool FOLD>
cudaError_t launch_bwd_sel(const ScanBwdParams& p, bool vec, cudaStream_t s) {
    if ((p.dtheta_amax != nullptr) != (p.part_rowsum != nullptr)) return cudaErrorInvalidValue;
    return p.part_rowsum ? launch_bwd_sums<C, FOLD, true>(p, vec, s) : launch_bwd_sums<C, FOLD, false>(p, vec, s);
}

template <class C, bool VEC, bool BWD>
cudaError_t launch_summary_cfg(const SegSummaryParams& p, cudaStream_t stream) {
    auto kern = scan_unitary_summary_kernel<C, VEC, BWD>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)C::SMEM_BYTES);
    if (e != cudaSuccess) return e;
    const long long blocks = (warp_tasks<C>(p) + C::WARPS - 1) / C::WARPS;
    kern<<<(unsigned)blocks, C::WARPS * 32, C::SMEM_BYTES, stream>>>(p);
    count_launch();
    return cudaGetLastError();
}

// the summary pass stages (u, dt) or (u, dt, z, gy) and keeps no column-sum tiles
template <int NL, int SPT, int T, int STAGES, int WARPS>
cudaError_t launch_summary_sel(const SegSummaryParams& p, bool vec, cudaStream_t s) {
    using F = Cfg<NL, SPT, T, T, STAGES, WARPS, 2, false>;
    using B = Cfg<NL, SPT, T, T, STAGES, WARPS, 4, false>;
    if (p.gy) return vec ? launch_summary_cfg<B, true, true>(p, s) : launch_summary_cfg<B, false, true>(p, s);
    return vec ? launch_summary_cfg<F, true, false>(p, s) : launch_summary_cfg<F, false, false>(p, s);
}

// a warp's rows must be addressable with 32-bit byte offsets from its first row
inline bool offsets_fit(long long ld, int rows_per_warp) { return ld * (long long)rows_per_warp < (1LL << 29); }

}  // namespace

// Tile shapes per state count.  <lanes per channel, states per thread, tile
// steps, [sub-block,] stages, warps per block>.
cudaError_t launch_scan_unitary_fwd(const ScanFwdParams& p_, cudaStream_t stream) {
    if (p_.nch <= 0 || p_.L <= 0) return cudaSuccess;
    ScanFwdParams p = p_;
    p.status = device_status_ptr();
    if (!p.status) return cudaErrorInvalidSymbol;
    const bool vec = (p.L % 4 == 0) && (p.ld_theta % 4 == 0) && (p.ld_row % 4 == 0) && aligned16(p.theta) &&
                       aligned16(p.u) && aligned16(p.dt) && aligned16(p.z) && (p.y == nullptr || aligned16(p.y)) &&
                       offsets_fit(p.ld_theta, 128);
    const int N = p.N;
    if (N <= 4) return launch_fwd_sel<FwdCfg<4, 1, 32, 2, 4>, false>(p, vec, stream);
    if (N <= 8) return launch_fwd_sel<FwdCfg<8, 1, 32, 2, 4>, false>(p, vec, stream);
    if (N <= 16) return launch_fwd_sel<FwdCfg<16, 1, 32, 2, 4>, true>(p, vec, stream);
    if (N <= 32) return launch_fwd_sel<FwdCfg<32, 1, 32, 2, 4>, true>(p, vec, stream);
    if (N <= 64) return launch_fwd_sel<FwdCfg<32, 2, 32, 2, 4>, true>(p, vec, stream);
    if (N <= 128) return launch_fwd_sel<FwdCfg<32, 4, 32, 2, 2>, false>(p, vec, stream);
    return cudaErrorInvalidValue;
}

cudaError_t launch_scan_unitary_bwd(const ScanBwdParams& p_, cudaStream_t stream) {
    if (p_.nch <= 0 || p_.L <= 0) return cudaSuccess;
    ScanBwdParams p = p_;
    p.status = device_status_ptr();
    if (!p.status) return cudaErrorInvalidSymbol;
    if (p.ld_dtheta != p.ld_theta) return cudaErrorInvalidValue;
    if (p.part_nseg <= 0) p.part_nseg = p.nseg > 1 ? p.nseg : 1;
    const bool vec = (p.L % 4 == 0) && (p.ld_theta % 4 == 0) && (p.ld_row % 4 == 0) && aligned16(p.theta) &&
                       aligned16(p.dtheta) && aligned16(p.u) && aligned16(p.dt) && aligned16(p.z) &&
                       aligned16(p.gy) && aligned16(p.du) && aligned16(p.ddt) && aligned16(p.dz) &&
                       offsets_fit(p.ld_theta, 128);
    const int N = p.N;
    if (N <= 4) return launch_bwd_sel<BwdCfg<4, 1, 32, 32, 2, 2>, true>(p, vec, stream);
    if (N <= 8) return launch_bwd_sel<BwdCfg<8, 1, 32, 32, 2, 2>, false>(p, vec, stream);
    // one-warp blocks: a finished warp is replaced at once (measured 9.55 ms against 10.2 ms with two-warp blocks)
    if (N <= 16) return launch_bwd_sel<BwdCfg<16, 1, 32, 32, 2, 1>, false>(p, vec, stream);
    if (N <= 32) return launch_bwd_sel<BwdCfg<32, 1, 32, 32, 2, 2>, true>(p, vec, stream);
    if (N <= 64) return launch_bwd_sel<BwdCfg<32, 2, 32, 32, 2, 2>, true>(p, vec, stream);
    if (N <= 128) return launch_bwd_sel<BwdCfg<32, 4, 32, 32, 2, 2>, true>(p, vec, stream);
    return cudaErrorInvalidValue;
}

namespace {
cudaError_t launch_summary(const SegSummaryParams& p, cudaStream_t stream) {
    const bool vec = (p.L % 4 == 0) && (p.ld_theta % 4 == 0) && (p.ld_row % 4 == 0) && aligned16(p.theta) &&
                     aligned16(p.u) && aligned16(p.dt) && (!p.gy || (aligned16(p.z) && aligned16(p.gy))) &&
                     offsets_fit(p.ld_theta, 128);
    if (p.N <= 4) return launch_summary_sel<4, 1, 32, 2, 4>(p, vec, stream);
    if (p.N <= 8) return launch_summary_sel<8, 1, 32, 2, 4>(p, vec, stream);
    if (p.N <= 16) return launch_summary_sel<16, 1, 32, 2, 4>(p, vec, stream);
    if (p.N <= 32) return launch_summary_sel<32, 1, 32, 2, 4>(p, vec, stream);
    if (p.N <= 64) return launch_summary_sel<32, 2, 32, 2, 4>(p, vec, stream);
    if (p.N <= 128) return launch_summary_sel<32, 4, 32, 2, 2>(p, vec, stream);
    return cudaErrorInvalidValue;
}

unsigned chain_blocks(long long total) { return (unsigned)((total + 127) / 128); }

// Warps of a kernel that an SM holds by its shared memory (228 KB, 1 KB of it per block reserved), which is the limit for
// aligned rows.  The forward kernel for unaligned rows (128 registers at N = 16) and the summary for N > 64 hold fewer, 16
// instead of 20 warps; the plan must not depend on the rows' alignment, which a workspace query does not know.
template <class C>
constexpr long long warps_per_sm() {
    return (228 * 1024 / (long long)(C::SMEM_BYTES + 1024)) * C::WARPS;
}
}  // namespace

SegPlan scan_split_plan(long long nch, int N, int L, bool bwd) {
    SegPlan plan = {1, L};
    if (nch <= 0 || L <= 0 || N <= 0 || N > 128 || !time_split_option()) return plan;
    const int nl = N <= 4 ? 4 : N <= 8 ? 8 : N <= 16 ? 16 : 32;
    const long long warps = (nch + (32 / nl) - 1) / (32 / nl);
    long long per_sm = 0;
#define AUSSM_SLOTS(FWD, BWD) per_sm = bwd ? warps_per_sm<BWD>() : warps_per_sm<FWD>()
    using F4 = FwdCfg<4, 1, 32, 2, 4>; using B4 = BwdCfg<4, 1, 32, 32, 2, 2>;
    using F8 = FwdCfg<8, 1, 32, 2, 4>; using B8 = BwdCfg<8, 1, 32, 32, 2, 2>;
    using F16 = FwdCfg<16, 1, 32, 2, 4>; using B16 = BwdCfg<16, 1, 32, 32, 2, 1>;
    using F32 = FwdCfg<32, 1, 32, 2, 4>; using B32 = BwdCfg<32, 1, 32, 32, 2, 2>;
    using F64 = FwdCfg<32, 2, 32, 2, 4>; using B64 = BwdCfg<32, 2, 32, 32, 2, 2>;
    using F128 = FwdCfg<32, 4, 32, 2, 2>; using B128 = BwdCfg<32, 4, 32, 32, 2, 2>;
    if (N <= 4) AUSSM_SLOTS(F4, B4);
    else if (N <= 8) AUSSM_SLOTS(F8, B8);
    else if (N <= 16) AUSSM_SLOTS(F16, B16);
    else if (N <= 32) AUSSM_SLOTS(F32, B32);
    else if (N <= 64) AUSSM_SLOTS(F64, B64);
    else AUSSM_SLOTS(F128, B128);
#undef AUSSM_SLOTS
    // A split doubles the work (a summary pass before the real one), and an SM with a third of its warps resident is
    // already more than half busy, so it pays only when the launch fills less than a quarter.  As many segments as
    // fill a wave, and 32 of at least 256 steps where that is more: several waves of short segments keep the SMs
    // evenly busy to the end.  N = 16, 256 warps, L = 16384, forward + backward (device time): 1535 us whole, 850 with
    // 11 / 5 segments (one wave), 765 with 11, 738 with 16, 734 with 32, 772 with 64, 866 with 128; L = 65536: 3233 us
    // with 11 / 5, 2648 with 64; L = 3000 (150 warps): 292 whole, 131 with 11, 149 with 64.  Below 1024 steps a call is
    // bound by the host and two more launches cost more than the shorter chains save (B1 D64 L600: 204 us whole, 224
    // split).
    const long long slots = 148 * per_sm;
    if (warps * 4 > slots) return plan;
    const long long want = std::min<long long>(std::max<long long>(slots / warps, std::min(32, L / 256)), L / 128);
    if (want < 8) return plan;
    plan.seg_len = (int)(((L + want - 1) / want + 31) / 32 * 32);
    plan.nseg = (L + plan.seg_len - 1) / plan.seg_len;
    return plan;
}

// Forward with the time axis cut into segments: (A) every segment's summary: its end state from zero, e, and the
// product of its rotations, a; (B) the chain c_{s+1} = e_s + a_s c_s gives the state before every segment; (C) the
// real pass, every segment from its true initial state.
cudaError_t scan_unitary_fwd_split(const ScanFwdParams& p, const SegPlan& plan, float* scratch, cudaStream_t stream) {
    const long long VN = (long long)p.nch * plan.nseg * p.N;
    float *e_re = scratch, *e_im = e_re + VN, *a_re = e_im + VN, *a_im = a_re + VN, *b_re = a_im + VN,
          *b_im = b_re + VN;
    const SegSummaryParams sum = {p.theta, p.u, p.dt, nullptr, nullptr, p.B_r, p.B_theta, p.C_r, p.C_theta,
                                  e_re, e_im, a_re, a_im, nullptr, nullptr, p.nch, p.Dmod, p.N, p.L, p.ld_theta,
                                  p.ld_row, plan.nseg, plan.seg_len};
    cudaError_t err = launch_summary(sum, stream);
    if (err != cudaSuccess) return err;
    SegChainParams c = {};
    c.e_re = e_re; c.e_im = e_im; c.a_re = a_re; c.a_im = a_im; c.from_re = p.h0_re; c.from_im = p.h0_im;
    c.at_re = b_re; c.at_im = b_im; c.end_re = p.h1_re; c.end_im = p.h1_im;
    c.total = (long long)p.nch * p.N; c.nseg = plan.nseg; c.N = p.N;
    segment_states_fwd_kernel<<<chain_blocks(c.total), 128, 0, stream>>>(c);
    count_launch();
    err = cudaGetLastError();
    if (err != cudaSuccess || !p.y) return err;         // state-only call: the chain already gave the final state
    ScanFwdParams q = p;
    q.nseg = plan.nseg; q.seg_len = plan.seg_len;
    q.h0_re = b_re; q.h0_im = b_im; q.h1_re = q.h1_im = nullptr;
    return launch_scan_unitary_fwd(q, stream);
}

// Backward with the same cut: (A) the summaries, now with every segment's own contribution l to the gradient of the
// state before it; (B) one chain walks back from the final state and its gradient (the rotations are invertible);
// (C) the real backward pass, every segment with its true end state and incoming gradient.
cudaError_t scan_unitary_bwd_split(const ScanBwdParams& p, const SegPlan& plan, float* scratch, cudaStream_t stream) {
    const long long VN = (long long)p.nch * plan.nseg * p.N;
    float *e_re = scratch, *e_im = e_re + VN, *a_re = e_im + VN, *a_im = a_re + VN, *s_re = a_im + VN,
          *s_im = s_re + VN, *l_re = s_im + VN, *l_im = l_re + VN, *g_re = l_im + VN, *g_im = g_re + VN;
    const SegSummaryParams sum = {p.theta, p.u, p.dt, p.z, p.gy, p.B_r, p.B_theta, p.C_r, p.C_theta,
                                  e_re, e_im, a_re, a_im, l_re, l_im, p.nch, p.Dmod, p.N, p.L, p.ld_theta, p.ld_row,
                                  plan.nseg, plan.seg_len};
    cudaError_t err = launch_summary(sum, stream);
    if (err != cudaSuccess) return err;
    SegChainParams c = {};
    c.e_re = e_re; c.e_im = e_im; c.a_re = a_re; c.a_im = a_im; c.l_re = l_re; c.l_im = l_im;
    c.from_re = p.h1_re; c.from_im = p.h1_im; c.gh_re = p.gh1_re; c.gh_im = p.gh1_im;
    c.at_re = s_re; c.at_im = s_im; c.g_re = g_re; c.g_im = g_im;
    c.end_re = p.h0_re; c.end_im = p.h0_im; c.dh0_re = p.dh0_re; c.dh0_im = p.dh0_im;
    c.total = (long long)p.nch * p.N; c.nseg = plan.nseg; c.N = p.N;
    segment_states_bwd_kernel<<<chain_blocks(c.total), 128, 0, stream>>>(c);
    count_launch();
    err = cudaGetLastError();
    if (err != cudaSuccess) return err;
    ScanBwdParams q = p;
    q.nseg = plan.nseg; q.seg_len = plan.seg_len;
    q.h1_re = s_re; q.h1_im = s_im; q.gh1_re = g_re; q.gh1_im = g_im;
    q.dh0_re = q.dh0_im = nullptr; q.h0_re = q.h0_im = nullptr;
    return launch_scan_unitary_bwd(q, stream);
}

cudaError_t launch_reduce_param_grads(const ReduceParams& p, cudaStream_t stream) {
    const long long tail = (long long)p.D + (p.dx_bias ? (long long)p.D * p.N : 0);
    const unsigned blocks = (unsigned)(p.N + (tail + REDUCE_THREADS - 1) / REDUCE_THREADS);
    reduce_param_grads_kernel<<<blocks, REDUCE_THREADS, 0, stream>>>(p);
    count_launch();
    return cudaGetLastError();
}

}  // namespace aussm
