// tcgen05 / TMEM / TMA implementation of the float32-accurate GEMM used by the
// phase projection theta = x u and its two adjoints (replaces the d^2 inner
// loops of csrc/cuda/ssm_adaptive_unitary_forward.cu:83-110 and the atomics of
// ssm_adaptive_unitary_backward.cu:419-490 of the reference).
//
// Arithmetic: the three-term split  a*b ~ a_hi*b_hi + a_hi*b_lo + a_lo*b_hi  on
// FP16 parts.  split_f16 scales a tensor by the power of two S that brings its
// largest magnitude to about 2^14 and stores hi = fp16(S a), lo = fp16((S a -
// hi) 2^11): 2 x 11 significant bits over the whole float32 exponent range.
// The power-of-two scales come off exactly in the epilogue.
//
// One persistent CTA per SM walks 128 x 256 tiles of C.  Roles: warp 0 = TMA
// producer, warp 1 = MMA issuer (one lane; the warp also owns the 512-column
// TMEM allocation), warps 2-5 / 6-9 = accumulate/epilogue of the tile's left /
// right 128 columns (TMEM -> registers -> shared-memory transpose -> global).
// Per K block of 64 values and 128-column half of the tile the issuer runs, for
// each of the four K = 16 slices, one N = 256 tcgen05.mma  a_hi x [b_hi | b_lo]
// (accumulators [main | cross]) and one N = 128 tcgen05.mma  a_lo x b_hi  (cross).
//
// Shared-memory operand tiles use the 128-byte swizzle the TMA engine writes and
// the MMA descriptors expect.  K-major operand (K contiguous in memory): rows
// of 64 halves, 8-row groups 1024 B apart.  MN-major operand (row index
// contiguous): TMA boxes of 64 K-rows x 64 row-elements (8 KB) placed 8192 B
// apart along the row index, groups of 8 K-rows 1024 B apart inside a box.
//
// Every wait on an mbarrier is bounded; a wait that runs out records the reason
// in the device status word, and the CTA still frees its tensor memory.
#include "gemm_split3.cuh"

#include <cuda.h>
#include <cuda_fp16.h>
#include <stdint.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

#include "../../include/aussm_b200.h"
#include "common.cuh"
#include "host_common.cuh"

namespace aussm {
namespace {

constexpr int BM = 128, BN = 256;
constexpr int BK = 64;                               // K values per block
constexpr int KROW_BYTES = BK * 2;                   // a K-major row of a block: one swizzle row of 128 bytes
constexpr int MNBOX = 64;                            // row elements per MN-major TMA box (128-byte swizzle rows)
constexpr int MNBOX_BYTES = MNBOX * 2 * BK;          // 8 KB: BK rows of 128 bytes
constexpr int STAGES = 2;
constexpr int A_TILE_BYTES = BM * BK * 2;            // one part of the A tile: 16 KB
constexpr int B_HALF_BYTES = 128 * BK * 2;           // one part of one 128-column half: 16 KB
constexpr int STAGE_BYTES = 2 * A_TILE_BYTES + 4 * B_HALF_BYTES;   // hi + lo of both operands: 96 KB
// Epilogue staging: every accumulate warp turns its 32 x 32 blocks through shared memory (pitch 33 floats, free
// of bank conflicts both ways) so that C leaves - and, with beta, enters - as whole 128-byte row pieces.
constexpr int EPI_PITCH = 33;
constexpr int EPI_WARP_FLOATS = 32 * EPI_PITCH;
constexpr int EPI_WARPS = 8;                         // per column half one warp for each TMEM lane quarter
constexpr int EPI_BYTES = EPI_WARPS * EPI_WARP_FLOATS * 4;
constexpr int SMEM_BYTES = STAGES * STAGE_BYTES + 1024 + EPI_BYTES;    // + slack for 1024-byte alignment
// Tensor-memory accumulation truncates instead of rounding, so a long K loop drifts (measured 3.5e-5 relative
// at K = 4096).  The K loop is therefore cut into chunks of 256 K values: each chunk accumulates from zero in
// tensor memory and the epilogue warps add the finished chunk into float32 registers (round-to-nearest).  The
// hi*hi products and the two small cross terms go to separate accumulators (adding the tiny terms must not
// cost the big sum extra truncations).  The 512 columns hold such a pair for each 128-column half of the tile,
// and the halves take turns: while the tensor core works on one half of a chunk, the epilogue warps drain the
// other.
constexpr int MMA_N = 128;                           // the tile's two column halves take turns (see below)
constexpr int TMEM_COLS = 2 * BN;                    // 512: per column half a main and a cross accumulator
constexpr int NUM_THREADS = 32 * (2 + EPI_WARPS);

struct GemmKernelParams {
    float* C;
    long long ldc;
    long long c_batch_stride;
    int M, N, K;
    int kbatches;      // batch entries summed inside the K loop (1 when batches are independent)
    int a_batched;     // 0: operand shared by all batch entries (batch coordinate 0)
    int b_batched;
    int ksplit;        // partial outputs per output (runs of the contraction), c_part_stride floats apart
    long long c_part_stride;
    int beta;
    const float* row_bias;
    int* status;
    const unsigned* amax_a;   // FP16 parts: bit patterns of max|a|, max|b| (the parts are scaled by a power of two)
    const unsigned* amax_b;
    int c_vec;                // 1: C rows are 16-byte aligned (vector stores), 0: scalar stores
    int tiles_m, tiles_n, ntiles;   // one-CTA kernel: a CTA walks tiles blockIdx.x, blockIdx.x + gridDim.x, ...
};

// FP16 parts: the scaled low part is stored times 2^LO_SHIFT (see split_f16x4)
constexpr int LO_SHIFT = 11;

// Power-of-two scale that brings a tensor whose largest magnitude has the bit pattern `maxbits` to about 2^14
// (FP16 overflows at 65504), and its exact inverse.
__device__ __forceinline__ int scale_exponent(unsigned maxbits) {
    const int e = (int)((maxbits >> 23) & 0xffu) - 127;      // floor(log2(max)); -127 for zero / subnormal
    int k = 14 - e;
    if (k > 100) k = 100;
    if (k < -100) k = -100;
    return k;
}
__device__ __forceinline__ float pow2f(int k) { return __uint_as_float((unsigned)(127 + k) << 23); }

// The parts of four consecutive values, as the 8-byte words that are stored.  S = 2^k brings the tensor's largest
// magnitude to about 2^14:  hi = fp16(S a),  lo = fp16((S a - hi) 2^LO_SHIFT).
__device__ __forceinline__ void split_f16x4(const float4& v, float S, uint2& hi, uint2& lo) {
    constexpr float up = (float)(1 << LO_SHIFT);
    const float2 a = make_float2(v.x * S, v.y * S), b = make_float2(v.z * S, v.w * S);
    const __half2 ha = __float22half2_rn(a), hb = __float22half2_rn(b);
    const float2 fa = __half22float2(ha), fb = __half22float2(hb);
    const __half2 la = __float22half2_rn(make_float2((a.x - fa.x) * up, (a.y - fa.y) * up));
    const __half2 lb = __float22half2_rn(make_float2((b.x - fb.x) * up, (b.y - fb.y) * up));
    hi = make_uint2(*reinterpret_cast<const uint32_t*>(&ha), *reinterpret_cast<const uint32_t*>(&hb));
    lo = make_uint2(*reinterpret_cast<const uint32_t*>(&la), *reinterpret_cast<const uint32_t*>(&lb));
}

// ---- PTX wrappers ---------------------------------------------------------
__device__ __forceinline__ void tma_load_4d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1,
                                            int c2, int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(smem_addr(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_addr(bar)), "r"(c0), "r"(c1),
        "r"(c2), "r"(c3)
        : "memory");
}

__device__ __forceinline__ void tma_load_5d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1,
                                            int c2, int c3, int c4) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];"
        ::"r"(smem_addr(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_addr(bar)), "r"(c0), "r"(c1),
        "r"(c2), "r"(c3), "r"(c4)
        : "memory");
}

// One copy = both parts (hi then lo) of 128 rows of an operand for one K block: 32 KB.
template <int MN_MAJOR>
__device__ __forceinline__ void load_rows128(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int row0, int k0,
                                             int batch) {
    if (MN_MAJOR) tma_load_5d(smem_dst, map, bar, 0, k0, row0 / MNBOX, 0, batch);
    else tma_load_4d(smem_dst, map, bar, k0, row0, 0, batch);
}

__device__ __forceinline__ void tmem_alloc(uint32_t* smem_holder, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(smem_holder)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void umma_f16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// streaming store: the line is not read again, so it should be the first to leave the L2
__device__ __forceinline__ void st_global_cs_f4(float* dst, const float4& v) {
    asm volatile("st.global.cs.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(dst), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w)
                 : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(bar)) : "memory");
}

// arrives on the mbarrier when all MMAs issued so far by this thread have completed
__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
                 : "memory");
}

// two 16-column loads of this warp's 32 lanes in flight, one wait
__device__ __forceinline__ void tmem_ld16_pair(uint32_t ta, uint32_t tb, float (&va)[16], float (&vb)[16]) {
    uint32_t r[16], q[16];
#define AUSSM_LD16(R, T)                                                                                          \
    asm volatile(                                                                                                 \
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "                                                                 \
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"                          \
        : "=r"(R[0]), "=r"(R[1]), "=r"(R[2]), "=r"(R[3]), "=r"(R[4]), "=r"(R[5]), "=r"(R[6]), "=r"(R[7]),        \
          "=r"(R[8]), "=r"(R[9]), "=r"(R[10]), "=r"(R[11]), "=r"(R[12]), "=r"(R[13]), "=r"(R[14]), "=r"(R[15])   \
        : "r"(T)                                                                                                  \
        : "memory")
    AUSSM_LD16(r, ta);
    AUSSM_LD16(q, tb);
#undef AUSSM_LD16
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        va[i] = __uint_as_float(r[i]);
        vb[i] = __uint_as_float(q[i]);
    }
}

// Shared-memory matrix descriptors (64 bit): start address >> 4 in bits 0-13,
// leading byte offset >> 4 in bits 16-29, stride byte offset >> 4 in bits
// 32-45, descriptor version 1 in bits 46-47, 128-byte swizzle (2) in bits 61-63.
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo_bytes, uint32_t sbo_bytes,
                                              uint64_t layout_type) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo_bytes >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo_bytes >> 4) & 0x3FFFu) << 32) | (1ull << 46) | (layout_type << 61);
}

// descriptor of the kk-th slice (16 FP16 values of K) of an operand tile
template <int MN_MAJOR>
__device__ __forceinline__ uint64_t operand_desc(uint32_t tile_saddr, int kk) {
    if (MN_MAJOR) {
        // MN-major, 128-byte swizzle (type 2): TMA boxes of BK K-rows x 64 row-elements (8 KB) placed 8192 B
        // apart along the row index, groups of 8 K-rows 1024 B apart; a K = 16 slice is two groups
        return smem_desc(tile_saddr + kk * 2048, MNBOX_BYTES, 1024, 2);
    }
    // K-major, 128-byte swizzle (type 2): rows of 128 B (64 halves of K), 8-row groups 1024 B apart; a K = 16
    // slice starts 32 B further into the row
    return smem_desc(tile_saddr + kk * 32, 16, 8 * KROW_BYTES, 2);
}

// Accumulation chunks.  A chunk is KC consecutive K blocks accumulated in tensor memory before the epilogue warps
// add it to their float32 registers.  The chunks of the tile's two column halves are offset by KC/2 blocks, so the
// halves never finish a chunk at the same K block: the half that starts a new chunk is issued second and its
// drain hides behind the other half's MMAs.  The first chunk of half 1 is KC + KC/2 blocks long (not KC/2): at
// the start of a tile the warps that drain are still storing the previous tile.
__device__ __forceinline__ bool half_starts(int h, int it, int kc) {
    return it == 0 || (h ? ((it % kc) == kc / 2 && it > kc / 2) : (it % kc) == 0);
}
__device__ __forceinline__ bool half_ends(int h, int it, int total, int kc) {
    return it == total - 1 || half_starts(h, it + 1, kc);
}
__device__ __forceinline__ int first_half(int it, int kc) { return (it > 0 && half_starts(0, it, kc)) ? 1 : 0; }

// Instruction descriptor of kind::f16 with float32 accumulate: c_format = 1 (bits 4-5), a/b format F16 = 0
// (bits 7-9, 10-12), a/b major (bits 15, 16), N >> 3 (bits 17-22), M >> 4 (bits 24-28).
template <int A_MN, int B_MN>
__device__ __forceinline__ constexpr uint32_t instr_desc() {
    return (1u << 4) | ((uint32_t)A_MN << 15) | ((uint32_t)B_MN << 16) | ((uint32_t)(MMA_N >> 3) << 17) |
           ((uint32_t)(BM >> 4) << 24);
}

template <int A_MN, int B_MN>
__global__ void __launch_bounds__(NUM_THREADS, 1)
gemm_split3_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                   const GemmKernelParams p) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t full_bar[STAGES], empty_bar[STAGES], acc_full[2], acc_empty[2];
    __shared__ uint32_t tmem_holder;
    __shared__ int failed;

    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // Persistent CTA: tile t -> (row block fastest, then column block, then independent batch entry), so that CTAs
    // running side by side share a B tile in L2.  Barrier phases, stage indices and chunk counters run on across
    // tiles: the copies and MMAs of the next tile start while the epilogue warps still store the previous one.
    const int tiles_mn = p.tiles_m * p.tiles_n;
    constexpr int CHUNK_KB = 256 / BK;                         // K blocks per accumulation chunk (256 values)
    const int kblocks = (p.K + BK - 1) / BK;
    const int blocks_all = kblocks * p.kbatches;
    // tile t: which output, which run of its contraction (K blocks [begin, begin + total) of blocks_all)
    auto tile_batch = [&](int t) { return (t / tiles_mn) / p.ksplit; };
    auto tile_run = [&](int t) { return (t / tiles_mn) % p.ksplit; };
    auto run_begin = [&](int run) { return (int)((long long)blocks_all * run / p.ksplit); };

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        for (int h = 0; h < 2; ++h) {
            mbar_init(&acc_full[h], 1);
            mbar_init(&acc_empty[h], EPI_WARPS / 2);
        }
        failed = 0;
        fence_mbar_init();
        fence_proxy_async();
    }
    if (warp == 1) tmem_alloc(&tmem_holder, TMEM_COLS);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = tmem_holder;

    if (warp == 0) {
        // ---- TMA producer.  A stage is three copies: each tensor map covers both parts of its operand, and one
        // copy brings the hi and lo rows of 128 rows (the A tile; a 128-column half of the B tile).  clock64
        // stamps around the refill of a stage: the issuing warp is held 600-1000 cycles for the 96 KB of a stage
        // whether they go as ten copies or as three, from one lane or from several, and the data is complete
        // about 1500 cycles later - the refill of one stage takes longer than the 1536 tensor-core cycles of the
        // other, so the kernel runs at the rate the stage data arrives (about 42 bytes per cycle and SM) ----
        int g = 0;                                       // K blocks copied by this CTA so far
        bool okp = true;
        for (int t = blockIdx.x; t < p.ntiles && okp; t += gridDim.x) {
        const int zb = tile_batch(t), run = tile_run(t);
        const int m0 = ((t % tiles_mn) % p.tiles_m) * BM, n0 = ((t % tiles_mn) / p.tiles_m) * BN;
        const int begin = run_begin(run), total = run_begin(run + 1) - begin;
        for (int it = 0; it < total; ++it, ++g) {
            const int s = g % STAGES;
            const uint32_t ph = (uint32_t)(g / STAGES) & 1u;
            bool w = true;
            if (lane == 0) {
                w = mbar_wait_bounded(&empty_bar[s], ph ^ 1u, p.status);
                if (!w) failed = 1;
                else mbar_arrive_expect_tx(&full_bar[s], STAGE_BYTES);
            }
            w = __shfl_sync(0xffffffffu, w, 0);          // also orders the copies after the arming of the barrier
            if (!w) { okp = false; break; }
            const int kb = (begin + it) % kblocks;
            const int batch = zb * p.kbatches + (begin + it) / kblocks;
            const int ba = p.a_batched ? batch : 0, bb = p.b_batched ? batch : 0;
            uint8_t* st = smem + s * STAGE_BYTES;
            const int k0 = kb * BK;
            // the A tile [a_hi | a_lo], then per 128-column half [b_hi | b_lo] (one N = 256 descriptor covers a half)
            if (lane == 0) load_rows128<A_MN>(st, &mapA, &full_bar[s], m0, k0, ba);
            else if (lane < 3)
                load_rows128<B_MN>(st + 2 * A_TILE_BYTES + (lane - 1) * 2 * B_HALF_BYTES, &mapB, &full_bar[s],
                                   n0 + (lane - 1) * MMA_N, k0, bb);
        }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // ---- MMA issuer: per chunk of CHUNK_KB K-blocks, column half 0 then column half 1 ----
            constexpr uint32_t idesc = instr_desc<A_MN, B_MN>();                        // N = 128
            constexpr uint32_t idesc2 = idesc + ((uint32_t)(MMA_N >> 3) << 17);               // N = 256
            bool ok = true;
            int ch[2] = {0, 0};                       // chunks finished per column half
            int g = 0;                                // K blocks consumed so far
            for (int t = blockIdx.x; t < p.ntiles && ok; t += gridDim.x) {
            const int run = tile_run(t), total = run_begin(run + 1) - run_begin(run);
            for (int it = 0; it < total && ok; ++it, ++g) {
                const int s = g % STAGES;
                if (!mbar_wait_bounded(&full_bar[s], (uint32_t)(g / STAGES) & 1u, p.status)) { failed = 1; ok = false; break; }
                tc_fence_after();
                const uint32_t st = smem_addr(smem + s * STAGE_BYTES);
                const uint32_t a_hi = st, a_lo = st + A_TILE_BYTES;
                const int first = first_half(it, CHUNK_KB);
                for (int q = 0; q < 2 && ok; ++q) {
                    const int h = q == 0 ? first : 1 - first;
                    const bool starts = half_starts(h, it, CHUNK_KB);
                    if (starts) {
                        // the epilogue warps have taken this half's previous chunk out of tensor memory
                        if (!mbar_wait_bounded(&acc_empty[h], ((uint32_t)ch[h] & 1u) ^ 1u, p.status)) { failed = 1; ok = false; break; }
                        tc_fence_after();
                    }
                    const uint32_t acc_main = tmem_base + (uint32_t)(h * 2 * MMA_N), acc_cross = acc_main + MMA_N;
                    // [b_hi | b_lo] of this half are adjacent: a_hi meets both in one N = 256 instruction whose
                    // output columns are [main | cross] (one read of a_hi instead of two), then a_lo * b_hi
                    const uint32_t b_hi = st + 2 * A_TILE_BYTES + h * 2 * B_HALF_BYTES;
#pragma unroll
                    for (int kk = 0; kk < BK / 16; ++kk) {
                        const uint64_t ah = operand_desc<A_MN>(a_hi, kk), al = operand_desc<A_MN>(a_lo, kk);
                        const uint64_t bh = operand_desc<B_MN>(b_hi, kk);
                        const uint32_t acc_flag = (starts && kk == 0) ? 0u : 1u;
                        umma_f16(acc_main, ah, bh, idesc2, acc_flag);
                        umma_f16(acc_cross, al, bh, idesc, 1u);
                    }
                    if (half_ends(h, it, total, CHUNK_KB)) {
                        umma_commit(&acc_full[h]);          // chunk of this half complete
                        ++ch[h];
                    }
                }
                umma_commit(&empty_bar[s]);                 // frees the stage when these MMAs have read it
            }
            }
        }
    } else {
        // ---- accumulate + epilogue: warps 2..9; TMEM lane quarter = warp % 4, column half = (warp - 2) / 4.
        // The warps of a half depend on nothing the other half does: they store their half of a finished tile
        // while the tensor core works on the next one, and only have to be back when the first chunk of their
        // half of that tile is complete (four K blocks later for half 0, six for half 1).
        const int quarter = warp & 3;
        const int h = (warp - 2) >> 2;
        float acc[MMA_N];                        // scaled units (FP16 parts): the scales come off once, at the end
        const float cross_scale = pow2f(-LO_SHIFT);
        bool ok = true;
        int chn = 0;                                     // chunks drained
        // exact power-of-two scales, applied one after the other (read once: under the load of the operand
        // copies a global read takes thousands of cycles)
        const float ua = pow2f(-scale_exponent(*p.amax_a)), ub = pow2f(-scale_exponent(*p.amax_b));
        float* stg = reinterpret_cast<float*>(smem + STAGES * STAGE_BYTES) + (warp - 2) * EPI_WARP_FLOATS;
        const int rsub = lane >> 3, c4 = (lane & 7) * 4;           // coalesced phase: 4 rows x 8 quads per instruction
        const uint32_t t0 = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(h * 2 * MMA_N);
        for (int t = blockIdx.x; t < p.ntiles; t += gridDim.x) {
            const int zb = tile_batch(t), run = tile_run(t), total = run_begin(run + 1) - run_begin(run);
            const int m0 = ((t % tiles_mn) % p.tiles_m) * BM, n0 = ((t % tiles_mn) / p.tiles_m) * BN;
            const int own_row = m0 + quarter * 32 + lane;
            const float rb = (p.row_bias && own_row < p.M) ? p.row_bias[own_row] : 0.f;     // long before its use
#pragma unroll
            for (int i = 0; i < MMA_N; ++i) acc[i] = 0.f;
            for (int it = 0; it < total; ++it) {
                if (!half_ends(h, it, total, CHUNK_KB)) continue;
                // a chunk of this half is complete: add it to the registers and hand the columns back
                if (ok) ok = mbar_wait_bounded(&acc_full[h], (uint32_t)chn & 1u, p.status);
                tc_fence_after();
                if (ok) {
#pragma unroll
                    for (int part = 0; part < MMA_N / 16; ++part) {
                        float vm[16], vc[16];
                        tmem_ld16_pair(t0 + part * 16, t0 + MMA_N + part * 16, vm, vc);   // hi*hi ; hi*lo + lo*hi
#pragma unroll
                        for (int i = 0; i < 16; ++i)
                            acc[part * 16 + i] = fmaf(vc[i], cross_scale, acc[part * 16 + i] + vm[i]);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[h]);            // the issuer may start this half's next chunk
                ++chn;
            }
            // The 32 x 32 blocks of the warp turn through the staging tile: lane = row on the way in, 4 rows x 128
            // bytes per instruction on the way out.
            if (ok && !failed) {
                float* cbase = p.C + (long long)zb * p.c_batch_stride + (long long)run * p.c_part_stride;
#pragma unroll
                for (int blk = 0; blk < MMA_N / 32; ++blk) {
#pragma unroll
                    for (int c = 0; c < 32; ++c) stg[lane * EPI_PITCH + c] = (acc[blk * 32 + c] * ua) * ub + rb;
                    __syncwarp();
                    const int col = n0 + h * MMA_N + blk * 32 + c4;
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        const int rr = 4 * k + rsub;
                        const int row = m0 + quarter * 32 + rr;
                        const float* sp = stg + rr * EPI_PITCH + c4;
                        float4 o = make_float4(sp[0], sp[1], sp[2], sp[3]);
                        if (row < p.M) {
                            float* dst = cbase + (long long)row * p.ldc + col;
                            if (p.c_vec && col + 3 < p.N) {
                                if (p.beta) {
                                    const float4 cin = *reinterpret_cast<const float4*>(dst);
                                    o.x += cin.x; o.y += cin.y; o.z += cin.z; o.w += cin.w;
                                }
                                st_global_cs_f4(dst, o);           // written once, not read again by this kernel
                            } else {
                                if (col + 0 < p.N) dst[0] = o.x + (p.beta ? dst[0] : 0.f);
                                if (col + 1 < p.N) dst[1] = o.y + (p.beta ? dst[1] : 0.f);
                                if (col + 2 < p.N) dst[2] = o.z + (p.beta ? dst[2] : 0.f);
                                if (col + 3 < p.N) dst[3] = o.w + (p.beta ? dst[3] : 0.f);
                            }
                        }
                    }
                    __syncwarp();
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, TMEM_COLS);
}

// ---- hi/lo split ----------------------------------------------------------
// FP16 parts.  With S = 2^k the power of two that brings max|src| to about 2^14:
//   hi = fp16(S a),  lo = fp16((S a - hi) 2^LO_SHIFT)
// hi carries the first 11 significant bits and lo the next 11 (stored scaled up so that it stays in FP16's
// normal range); a*b ~ (hi_a hi_b + (hi_a lo_b + lo_a hi_b) 2^-LO_SHIFT) / (S_a S_b).
//
// Both passes walk the source four columns per thread and four such quads at a time, so that a thread has four loads
// in flight.  The walk carries (row, quad) and adds the grid's stride as (rows, quads) with one carry: no division
// per quad (with a 64-bit division per quad and an atomic per warp the maxima of a training pass of four AUSSM layers,
// B1 D512 N16 L65536, took 6.18 ms in 112 launches, now 1.61 ms).  VEC: rows of the
// source are 16-byte aligned and whole quads (one 128-bit load per thread); otherwise scalar loads with a bound check
// per column.  The destination pitch is always a multiple of 8 halves, so every thread stores its four halves as one
// 8-byte word, zeros after `cols`; what lies between that quad and the pitch stays undefined (the K extent of a
// K-major tensor map ends before it, and in an MN-major operand it meets columns of C that are never stored).
template <bool VEC>
__device__ __forceinline__ float4 load_quad(const float* row, long long c, long long cols) {
    if (VEC) return *reinterpret_cast<const float4*>(row + c);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c + 0 < cols) v.x = row[c + 0];
    if (c + 1 < cols) v.y = row[c + 1];
    if (c + 2 < cols) v.z = row[c + 2];
    if (c + 3 < cols) v.w = row[c + 3];
    return v;
}

struct QuadWalk {
    unsigned r, q;           // row, quad of the row
    unsigned dr, dq, nq;
    __device__ __forceinline__ QuadWalk(unsigned quads, unsigned block, unsigned blocks) : nq(quads) {
        const unsigned first = block * 256u + threadIdx.x, step = blocks * 256u;
        r = first / nq;
        q = first % nq;
        dr = step / nq;
        dq = step % nq;
    }
    __device__ __forceinline__ void next() {
        r += dr;
        q += dq;
        if (q >= nq) { q -= nq; ++r; }
    }
};
constexpr int QUADS_IN_FLIGHT = 4;

// The sources of a launch: source k owns blocks_of[k] consecutive blocks per batch entry.
struct SplitLaunch {
    SplitSource s[kSplitSources];
    unsigned blocks_of[kSplitSources];
    int vec[kSplitSources];
    unsigned second;             // first block of the second source
};

template <bool VEC>
__device__ __forceinline__ float quads_absmax(const float* __restrict__ src, long long ld_src, unsigned rows,
                                              unsigned cols, unsigned block, unsigned blocks) {
    float m = 0.f;
    for (QuadWalk w((cols + 3) / 4, block, blocks); w.r < rows;) {
        float4 v[QUADS_IN_FLIGHT];
#pragma unroll
        for (int k = 0; k < QUADS_IN_FLIGHT; ++k) {
            v[k] = w.r < rows ? load_quad<VEC>(src + w.r * ld_src, 4LL * w.q, cols) : make_float4(0.f, 0.f, 0.f, 0.f);
            w.next();
        }
#pragma unroll
        for (int k = 0; k < QUADS_IN_FLIGHT; ++k) {
            const float a[4] = {fabsf(v[k].x), fabsf(v[k].y), fabsf(v[k].z), fabsf(v[k].w)};
#pragma unroll
            for (int e = 0; e < 4; ++e)                  // no infinity, no NaN: these spoil their own rows and columns
                if (a[e] <= 3.402823466e38f) m = fmaxf(m, a[e]);
        }
    }
    return m;
}

__global__ void __launch_bounds__(256) absmax_kernel(const SplitLaunch p) {
    __shared__ float warp_max[8];
    const int k = blockIdx.x >= p.second ? 1 : 0;
    const SplitSource& s = p.s[k];
    const unsigned id = blockIdx.x - (k ? p.second : 0u), blocks = p.blocks_of[k];
    const float* src = s.src + (id / blocks) * s.src_batch_stride;
    float m = p.vec[k] ? quads_absmax<true>(src, s.ld_src, (unsigned)s.rows, (unsigned)s.cols, id % blocks, blocks)
                       : quads_absmax<false>(src, s.ld_src, (unsigned)s.rows, (unsigned)s.cols, id % blocks, blocks);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    if ((threadIdx.x & 31) == 0) warp_max[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll
        for (int w = 1; w < 8; ++w) m = fmaxf(m, warp_max[w]);
        // non-negative floats order like their bit patterns
        if (m > 0.f) atomicMax(s.amax, __float_as_uint(fminf(m, 3.0e38f)));
    }
}

template <bool VEC>
__device__ __forceinline__ void quads_split(const float* __restrict__ src, long long ld_src, __half* __restrict__ hi,
                                            __half* __restrict__ lo, long long ld_dst, unsigned rows, unsigned cols,
                                            float S, unsigned block, unsigned blocks) {
    for (QuadWalk w((cols + 3) / 4, block, blocks); w.r < rows;) {
        float4 v[QUADS_IN_FLIGHT];
        long long at[QUADS_IN_FLIGHT];
#pragma unroll
        for (int k = 0; k < QUADS_IN_FLIGHT; ++k) {
            const bool on = w.r < rows;
            v[k] = on ? load_quad<VEC>(src + w.r * ld_src, 4LL * w.q, cols) : make_float4(0.f, 0.f, 0.f, 0.f);
            at[k] = on ? w.r * ld_dst + 4LL * w.q : -1;
            w.next();
        }
#pragma unroll
        for (int k = 0; k < QUADS_IN_FLIGHT; ++k) {
            uint2 ph, pl;
            split_f16x4(v[k], S, ph, pl);
            if (at[k] >= 0) {
                *reinterpret_cast<uint2*>(hi + at[k]) = ph;
                *reinterpret_cast<uint2*>(lo + at[k]) = pl;
            }
        }
    }
}

__global__ void __launch_bounds__(256) split_f16_kernel(const SplitLaunch p) {
    const int k = blockIdx.x >= p.second ? 1 : 0;
    const SplitSource& s = p.s[k];
    const unsigned id = blockIdx.x - (k ? p.second : 0u), blocks = p.blocks_of[k];
    const long long b = id / blocks;
    const float* src = s.src + b * s.src_batch_stride;
    __half* hi = static_cast<__half*>(s.hi) + b * s.dst_batch_stride;
    __half* lo = static_cast<__half*>(s.lo) + b * s.dst_batch_stride;
    const float S = pow2f(scale_exponent(*s.amax));
    if (p.vec[k]) quads_split<true>(src, s.ld_src, hi, lo, s.ld_dst, (unsigned)s.rows, (unsigned)s.cols, S, id % blocks, blocks);
    else quads_split<false>(src, s.ld_src, hi, lo, s.ld_dst, (unsigned)s.rows, (unsigned)s.cols, S, id % blocks, blocks);
}

// ---- host side --------------------------------------------------------------
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* ptr = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(ptr);
    });
    return fn;
}

// Tensor map of a split operand (halves), both parts.  `part_stride` is the distance from the hi to the lo part
// in bytes.  K-major: dims (K, rows, part, batch), box (BK, 128, 2, 1), 128-byte swizzle.  MN-major: dims (64, K,
// rows / 64, part, batch), box (64, BK, 2, 2, 1), 128-byte swizzle: the row index is cut into the 64-element
// boxes the MMA descriptors expect, so one copy fills two boxes of each part.  Out-of-range K rows and boxes read
// as zero; the last box of an MN-major operand may reach up to 63 elements past `rows` (into the next row, or
// into the slack that split_part_halves() leaves behind the last row) - those values meet only rows or columns
// of C that are never stored.
int make_map(CUtensorMap* map, const void* base, long long part_stride, int mn_major, long long rows, long long K,
             long long ld, long long batch_stride, int batches) {
    EncodeTiledFn fn = encode_fn();
    if (!fn) {
        set_error("cuTensorMapEncodeTiled is not available from the driver");
        return AUSSM_ECUDA;
    }
    if (part_stride <= 0 || part_stride % 16) {
        set_error("gemm_split3: the lo part must follow the hi part at a multiple of 16 bytes (distance %lld)",
                  part_stride);
        return AUSSM_EINVAL;
    }
    cuuint64_t dims[5], strides[4];
    cuuint32_t box[5], estr[5] = {1, 1, 1, 1, 1};
    const cuuint64_t esize = 2;
    const cuuint64_t bstride = (cuuint64_t)(batches > 1 ? batch_stride : 8) * esize;   // unused when batches == 1
    int rank;
    if (mn_major) {
        rank = 5;
        dims[0] = MNBOX; dims[1] = (cuuint64_t)K; dims[2] = (cuuint64_t)((rows + MNBOX - 1) / MNBOX); dims[3] = 2;
        dims[4] = (cuuint64_t)batches;
        box[0] = MNBOX; box[1] = BK; box[2] = 128 / MNBOX; box[3] = 2; box[4] = 1;
        strides[0] = (cuuint64_t)ld * esize; strides[1] = MNBOX * esize; strides[2] = (cuuint64_t)part_stride;
        strides[3] = bstride;
    } else {
        rank = 4;
        dims[0] = (cuuint64_t)K; dims[1] = (cuuint64_t)rows; dims[2] = 2; dims[3] = (cuuint64_t)batches;
        box[0] = BK; box[1] = 128; box[2] = 2; box[3] = 1;
        strides[0] = (cuuint64_t)ld * esize; strides[1] = (cuuint64_t)part_stride; strides[2] = bstride;
    }
    CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, (cuuint32_t)rank, const_cast<void*>(base), dims, strides, box,
                    estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                    CU_TENSOR_MAP_SWIZZLE_128B,
                    CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed with code %d (rows=%lld K=%lld ld=%lld batches=%d mn_major=%d)", (int)r,
                  rows, K, ld, batches, mn_major);
        return AUSSM_ECUDA;
    }
    return AUSSM_OK;
}

template <int A_MN, int B_MN>
int launch(const CUtensorMap* maps, const GemmKernelParams& kp, dim3 grid, cudaStream_t stream) {
    auto kern = gemm_split3_kernel<A_MN, B_MN>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
    if (e != cudaSuccess) {
        set_error("gemm_split3: cudaFuncSetAttribute: %s", cudaGetErrorString(e));
        return AUSSM_ECUDA;
    }
    kern<<<grid, NUM_THREADS, SMEM_BYTES, stream>>>(maps[0], maps[1], kp);
    e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error("gemm_split3 launch: %s", cudaGetErrorString(e));
        return AUSSM_ECUDA;
    }
    count_launch();
    return AUSSM_OK;
}

bool ok16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

// SM count of the current device (cached per device ordinal)
int sm_count() {
    constexpr int kMaxDevices = 64;
    static int cached[kMaxDevices] = {};
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return 148;
    if (cached[dev] > 0) return cached[dev];
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    cached[dev] = n;
    return n;
}

}  // namespace

bool gemm_split3_supported(const SplitOperand& A, const SplitOperand& B, const float* C, const GemmShape& s) {
    if (s.M <= 0 || s.N <= 0 || s.K <= 0 || s.batches <= 0 || !C) return false;
    if (!A.amax || !B.amax) return false;
    // the parts are rows of halves whose pitch is a multiple of 16 bytes (split_f16 writes them that way)
    if (A.ld % 8 || B.ld % 8 || A.batch_stride % 8 || B.batch_stride % 8) return false;
    if (!ok16(A.hi) || !ok16(A.lo) || !ok16(B.hi) || !ok16(B.lo)) return false;
    return encode_fn() != nullptr;
}

long long gemm_split3_blocks(const GemmShape& s) {
    return (long long)((s.K + BK - 1) / BK) * (s.reduce_batches ? s.batches : 1);
}

int gemm_split3_runs(long long M, long long N, long long K, int batches, bool reduce_batches, int most) {
    constexpr long long SMS = 148;          // fixed, so that a workspace sized with it always fits
    const long long outputs = reduce_batches ? 1 : batches;
    const long long tiles = ((M + BM - 1) / BM) * ((N + BN - 1) / BN) * outputs;
    const long long blocks = ((K + BK - 1) / BK) * (reduce_batches ? batches : 1);
    const double part = 8.0 * (double)M * (double)N * (double)outputs / 7.8e6;
    int best = 1;
    double best_cost = 0.0;
    for (int g = 1; g <= most && (g == 1 || blocks / g >= 4); ++g) {
        const double waves = (double)((tiles * g + SMS - 1) / SMS);
        const double cost = waves * ((double)((blocks + g - 1) / g) + 6.0) + (g > 1 ? 2.0 + part * g : 0.0);
        if (g == 1 || cost < 0.97 * best_cost) {
            best = g;
            best_cost = cost;
        }
    }
    return best;
}

int gemm_split3(const SplitOperand& A, const SplitOperand& B, float* C, const GemmShape& s, cudaStream_t stream) {
    if (!gemm_split3_supported(A, B, C, s)) {
        set_error("gemm_split3: unsupported shape or alignment of the split operands (M=%d N=%d K=%d)", s.M, s.N, s.K);
        return AUSSM_EINVAL;
    }
    alignas(64) CUtensorMap maps[2];
    const int ab = A.batch_stride != 0 ? s.batches : 1, bb = B.batch_stride != 0 ? s.batches : 1;
    const long long a_ps = static_cast<const char*>(A.lo) - static_cast<const char*>(A.hi);
    const long long b_ps = static_cast<const char*>(B.lo) - static_cast<const char*>(B.hi);
    if (int rc = make_map(&maps[0], A.hi, a_ps, A.mn_major, s.M, s.K, A.ld, A.batch_stride, ab)) return rc;
    if (int rc = make_map(&maps[1], B.hi, b_ps, B.mn_major, s.N, s.K, B.ld, B.batch_stride, bb)) return rc;
    GemmKernelParams kp;
    kp.C = C; kp.ldc = s.ldc; kp.c_batch_stride = s.c_batch_stride;
    kp.M = s.M; kp.N = s.N; kp.K = s.K;
    kp.kbatches = s.reduce_batches ? s.batches : 1;
    kp.ksplit = std::max(1, std::min(s.ksplit, (s.K + BK - 1) / BK * kp.kbatches));
    kp.c_part_stride = s.c_part_stride;
    kp.beta = s.beta;
    kp.row_bias = s.row_bias;
    kp.a_batched = A.batch_stride != 0;
    kp.b_batched = B.batch_stride != 0;
    kp.amax_a = A.amax;
    kp.amax_b = B.amax;
    kp.c_vec = (ok16(C) && s.ldc % 4 == 0 && s.c_batch_stride % 4 == 0 && s.c_part_stride % 4 == 0) ? 1 : 0;
    kp.status = device_status_ptr();
    if (!kp.status) {
        set_error("gemm_split3: device status word unavailable");
        return AUSSM_ECUDA;
    }
    kp.tiles_m = (s.M + BM - 1) / BM;
    kp.tiles_n = (s.N + BN - 1) / BN;
    kp.ntiles = kp.tiles_m * kp.tiles_n * (s.reduce_batches ? 1 : s.batches) * kp.ksplit;
    const dim3 grid((unsigned)std::min(kp.ntiles, sm_count()), 1, 1);     // one persistent CTA per SM
    if (A.mn_major) return B.mn_major ? launch<1, 1>(maps, kp, grid, stream) : launch<1, 0>(maps, kp, grid, stream);
    return B.mn_major ? launch<0, 1>(maps, kp, grid, stream) : launch<0, 0>(maps, kp, grid, stream);
}

int split_f16_many(const SplitSource* sources, int count, cudaStream_t stream, bool have_amax) {
    SplitLaunch p = {};
    unsigned total_blocks = 0;
    int used = 0;
    for (int i = 0; i < count; ++i) {
        const SplitSource& s = sources[i];
        if (s.ld_dst % 8 || s.dst_batch_stride % 8 || s.ld_dst < (s.cols + 3) / 4 * 4 || !ok16(s.hi) || !ok16(s.lo) ||
            !s.amax || used == kSplitSources) {
            set_error("split_f16: destination rows must be 16-byte aligned and hold whole quads (cols=%lld ld_dst=%lld)",
                      s.cols, s.ld_dst);
            return AUSSM_EINVAL;
        }
        const long long total = s.rows * ((s.cols + 3) / 4);
        if (total <= 0 || s.batches <= 0) continue;
        // eight resident blocks per SM over all batch entries (all of one wave), fewer when there is less than one
        // round of four quads per thread to do
        const long long want = (total + 256 * QUADS_IN_FLIGHT - 1) / (256 * QUADS_IN_FLIGHT);
        const long long most = std::max<long long>(1, ((long long)sm_count() * 8 + s.batches - 1) / s.batches);
        p.s[used] = s;
        p.blocks_of[used] = (unsigned)std::min(want, most);
        p.vec[used] = s.cols % 4 == 0 && s.ld_src % 4 == 0 && s.src_batch_stride % 4 == 0 && ok16(s.src);
        total_blocks += p.blocks_of[used] * (unsigned)s.batches;
        if (++used == 1) p.second = total_blocks;
    }
    if (used == 0) return AUSSM_OK;
    if (!have_amax) {
        absmax_kernel<<<total_blocks, 256, 0, stream>>>(p);
        count_launch();
    }
    split_f16_kernel<<<total_blocks, 256, 0, stream>>>(p);
    count_launch();
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error("split_f16 launch: %s", cudaGetErrorString(e));
        return AUSSM_ECUDA;
    }
    return AUSSM_OK;
}

int split_f16(const float* src, long long ld_src, long long src_batch_stride, void* hi, void* lo, long long ld_dst,
              long long dst_batch_stride, long long rows, long long cols, int batches, unsigned* amax,
              cudaStream_t stream, bool have_amax) {
    const SplitSource s = {src, ld_src, src_batch_stride, hi, lo, ld_dst, dst_batch_stride, rows, cols, batches, amax};
    if (amax && !have_amax) {
        cudaError_t e = cudaMemsetAsync(amax, 0, sizeof(unsigned), stream);
        if (e != cudaSuccess) {
            set_error("split_f16: clearing the maximum: %s", cudaGetErrorString(e));
            return AUSSM_ECUDA;
        }
    }
    return split_f16_many(&s, 1, stream, have_amax);
}

}  // namespace aussm
