// Float32-accurate GEMM on the 5th-generation tensor cores (tcgen05, TMEM
// accumulators, TMA operand staging) by the three-term split
//     a*b ~ a_hi*b_hi + a_hi*b_lo + a_lo*b_hi
// on FP16 parts: with S the power of two that brings the tensor's largest
// magnitude to about 2^14,  hi = fp16(S a),  lo = fp16((S a - hi) 2^11).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "host_common.cuh"

namespace aussm {

// One operand, already split into its two FP16 parts by split_f16.  `mn_major == 0`: stored as [rows][K] with K
// contiguous; `mn_major == 1`: stored as [K][rows] with the row (M or N) index contiguous.  `ld` is the pitch of
// the slower index in halves (a multiple of 8), `batch_stride` the distance between batch entries (halves,
// multiple of 8, 0 for an operand shared by all batch entries).  `amax` points to the bit pattern of the
// tensor's largest magnitude on the device (the parts are scaled by a power of two derived from it).
struct SplitOperand {
    const void* hi;
    const void* lo;
    int mn_major;
    long long ld;
    long long batch_stride;
    const unsigned* amax;
};

struct GemmShape {
    int M, N, K;
    int batches;          // number of operand batch entries
    int reduce_batches;   // 0: one output per batch entry; 1: C = sum over the batch entries
    int beta;             // 0: overwrite C, 1: add to C
    long long ldc;        // floats; any value (rows that are not 16-byte aligned take scalar stores)
    long long c_batch_stride;
    int ksplit;           // 0 or 1: whole contraction per tile; g > 1: the contraction (all K blocks of all summed
                          // batch entries) is cut into g nearly equal runs, each a partial output of its own at
                          // C + run * c_part_stride, to be added by the caller
    long long c_part_stride;
    const float* row_bias;  // (M) added to every row of the result, or nullptr (with ksplit <= 1)
};

long long gemm_split3_blocks(const GemmShape& s);      // K blocks of one output: no more runs than these are made
// How many runs to cut a contraction into: few output tiles leave most SMs without work, and the time of a launch is
// its number of tile waves times the K blocks of a tile.  Counted in K blocks (64 values, about 1.3 us of a tile):
// a tile costs its blocks + 6 for its epilogue, and g > 1 adds the writing and reading of g partial outputs
// (8 bytes an element at 6 TB/s) and a launch (2 blocks).  A run keeps at least 4 blocks (one accumulation chunk).
int gemm_split3_runs(long long M, long long N, long long K, int batches, bool reduce_batches, int most);

// Halves to reserve for one part of a split operand that holds `halves` values: rounded up to 256 bytes, with
// room for the up to 63 halves that the last copy of an MN-major operand reads past the end of its last row.
// The lo part must follow the hi part (one tensor map covers both).
inline size_t split_part_halves(size_t halves) { return (halves + 64 + 127) / 128 * 128; }

// C[m][n] (+)= sum_k A(m,k) B(n,k).  Returns 0 or a negative AUSSM_E* code.
int gemm_split3(const SplitOperand& A, const SplitOperand& B, float* C, const GemmShape& s, cudaStream_t stream);

// true when the split operands meet the alignment rules of the TMA path (pitches multiple of 8 halves, 16-byte bases)
bool gemm_split3_supported(const SplitOperand& A, const SplitOperand& B, const float* C, const GemmShape& s);

// FP16 hi/lo split of a strided 2-D float32 array (rows x cols, cols contiguous, any pitch and alignment),
// batched.  ld_dst / dst_batch_stride count halves and are multiples of 8, ld_dst >= cols rounded up to 4.
// amax is a device word that receives the bit pattern of max|src|.
struct SplitSource {
    const float* src;
    long long ld_src, src_batch_stride;
    void *hi, *lo;
    long long ld_dst, dst_batch_stride, rows, cols;
    int batches;
    unsigned* amax;
};
// Several tensors (up to kSplitSources) with one launch for the maxima and one for the parts: on small operands the
// launches are what a split costs.  The amax words must be zero.  have_amax: they hold the maxima already (the
// producers found them) and the pass over the sources that does is skipped.
constexpr int kSplitSources = 2;
int split_f16_many(const SplitSource* sources, int count, cudaStream_t stream, bool have_amax = false);
int split_f16(const float* src, long long ld_src, long long src_batch_stride, void* hi, void* lo, long long ld_dst,
              long long dst_batch_stride, long long rows, long long cols, int batches, unsigned* amax,
              cudaStream_t stream, bool have_amax = false);

}  // namespace aussm
