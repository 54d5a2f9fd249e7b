// Phase projection and its adjoints as three-term split GEMMs on tcgen05.
#include "projection.cuh"

#include <stdint.h>

#include <algorithm>

#include "../../include/aussm_b200.h"
#include "gemm_split3.cuh"

namespace aussm {

namespace {
size_t up(size_t v, size_t a) { return (v + a - 1) / a * a; }

// Runs of the two adjoint contractions (the window's pitch stands for its length: one plan per operator call)
constexpr int MOST_RUNS = 16;
int dx_runs(int B, int D, long long M, long long ldw) { return gemm_split3_runs(M, D, ldw, B, true, MOST_RUNS); }
int du_runs(int B, int D, long long M, long long ldw) { return gemm_split3_runs(D, ldw, M, B, false, MOST_RUNS); }
size_t part_floats(int B, int D, long long M, long long ldw) {
    const int gx = dx_runs(B, D, M, ldw), gu = du_runs(B, D, M, ldw);
    const size_t nx = gx > 1 ? up((size_t)M * D, 4) * gx : 0, nu = gu > 1 ? (size_t)B * D * ldw * gu : 0;
    return std::max(nx, nu);                 // dx is finished before du begins
}

// dst (+)= part 0 + part 1 + ... in this order: rows of `cols` floats, ld_dst / ld_part apart
__global__ void __launch_bounds__(256) add_parts_kernel(float* __restrict__ dst, long long ld_dst,
                                                        const float* __restrict__ part, long long ld_part,
                                                        long long part_stride, int parts, unsigned cols,
                                                        long long total, int overwrite) {
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < total; i += (long long)gridDim.x * 256) {
        const long long r = i / cols, c = i % cols;
        const float* src = part + r * ld_part + c;
        float sum = src[0];
        for (int k = 1; k < parts; ++k) sum += src[k * part_stride];
        float* d = dst + r * ld_dst + c;
        *d = overwrite ? sum : *d + sum;
    }
}
// whole rows of quads, 16-byte aligned
__global__ void __launch_bounds__(256) add_parts_vec_kernel(float* __restrict__ dst, const float* __restrict__ part,
                                                            long long part_stride, int parts, long long n4,
                                                            int overwrite) {
    for (long long i = (long long)blockIdx.x * 256 + threadIdx.x; i < n4; i += (long long)gridDim.x * 256) {
        float4 o = reinterpret_cast<const float4*>(part)[i];
        for (int k = 1; k < parts; ++k) {
            const float4 b = reinterpret_cast<const float4*>(part + k * part_stride)[i];
            o.x += b.x; o.y += b.y; o.z += b.z; o.w += b.w;
        }
        if (!overwrite) {
            const float4 c = reinterpret_cast<const float4*>(dst)[i];
            o.x += c.x; o.y += c.y; o.z += c.z; o.w += c.w;
        }
        reinterpret_cast<float4*>(dst)[i] = o;
    }
}

int add_parts(float* dst, long long ld_dst, const float* part, long long ld_part, long long part_stride, int parts,
              long long rows, long long cols, bool overwrite, cudaStream_t stream) {
    const long long total = rows * cols;
    const bool flat = ld_dst == cols && ld_part == cols && total % 4 == 0 && part_stride % 4 == 0 &&
                      (reinterpret_cast<uintptr_t>(dst) & 15u) == 0 && (reinterpret_cast<uintptr_t>(part) & 15u) == 0;
    const long long items = flat ? total / 4 : total;
    const unsigned blocks = (unsigned)std::min<long long>((items + 255) / 256, 148 * 8);
    if (flat) add_parts_vec_kernel<<<blocks, 256, 0, stream>>>(dst, part, part_stride, parts, items, overwrite ? 1 : 0);
    else add_parts_kernel<<<blocks, 256, 0, stream>>>(dst, ld_dst, part, ld_part, part_stride, parts, (unsigned)cols,
                                                      items, overwrite ? 1 : 0);
    count_launch();
    if (cudaGetLastError() != cudaSuccess) {
        set_error("projection: launch of the partial-sum kernel failed");
        return AUSSM_ECUDA;
    }
    return AUSSM_OK;
}
}  // namespace

size_t proj_scratch_bytes(int B, int D, long long M_, long long ldw) {
    const size_t M = (size_t)M_, Dp = up((size_t)D, 8);
    const size_t halves = 2 * split_part_halves(M * Dp) + 2 * split_part_halves((size_t)B * D * ldw) +
                          2 * split_part_halves((size_t)B * M * ldw);
    return halves * 2 + up(part_floats(B, D, M_, ldw) * sizeof(float), 256) + 256;
}

void proj_scratch_bind(ProjScratch& s, void* base, int B, int D, long long M_, long long ldw) {
    const size_t M = (size_t)M_, Dp = up((size_t)D, 8);
    char* p = static_cast<char*>(base);
    auto take = [&](size_t halves) {
        void* r = p;
        p += split_part_halves(halves) * 2;          // every part starts 256-byte aligned
        return r;
    };
    s.x_hi = take(M * Dp);
    s.x_lo = take(M * Dp);
    s.u_hi = take((size_t)B * D * ldw);
    s.u_lo = take((size_t)B * D * ldw);
    s.dth_hi = take((size_t)B * M * ldw);
    s.dth_lo = take((size_t)B * M * ldw);
    s.part = reinterpret_cast<float*>(p);
    p += up(part_floats(B, D, M_, ldw) * sizeof(float), 256);
    s.dx_runs = dx_runs(B, D, M_, ldw);
    s.du_runs = du_runs(B, D, M_, ldw);
    s.amax = reinterpret_cast<unsigned*>(p);   // inside the 256 spare bytes
    s.Dp = (long long)Dp;
}

void proj_begin(const float* x, ProjScratch& s) { s.x = x; }

int proj_split_u(const ProjDims& d, const float* u, ProjScratch& s, cudaStream_t stream) {
    const int first = s.x ? 0 : 1;               // maxima to find anew: [x,] u, dtheta
    cudaError_t e = cudaMemsetAsync(s.amax + first, 0, (3 - first) * sizeof(unsigned), stream);
    if (e != cudaSuccess) {
        set_error("projection: clearing the maxima: %s", cudaGetErrorString(e));
        return AUSSM_ECUDA;
    }
    const SplitSource sources[2] = {
        {s.x, d.D, 0, s.x_hi, s.x_lo, s.Dp, 0, d.M, d.D, 1, s.amax + 0},
        // rows r (D of them per batch entry), tl columns of this window
        {u + d.t0, d.L, (long long)d.D * d.L, s.u_hi, s.u_lo, d.ldw, (long long)d.D * d.ldw, d.D, d.tl, d.B, s.amax + 1}};
    s.x = nullptr;
    return split_f16_many(sources + first, 2 - first, stream);
}

int proj_theta(const ProjDims& d, const float* u, const float* bias, float* theta_w, ProjScratch& s, cudaStream_t stream) {
    const int M = (int)d.M;
    if (int rc = proj_split_u(d, u, s, stream)) return rc;
    // theta_w[b] (M x tl) = x (M x D, K-major) * u_b (D x tl: K rows, N contiguous -> MN-major)
    const SplitOperand A = {s.x_hi, s.x_lo, 0, s.Dp, 0, s.amax + 0};
    const SplitOperand Bop = {s.u_hi, s.u_lo, 1, d.ldw, (long long)d.D * d.ldw, s.amax + 1};
    const GemmShape shape = {M, d.tl, d.D, d.B, 0, 0, d.ldw, (long long)M * d.ldw, 1, 0, bias};
    return gemm_split3(A, Bop, theta_w, shape, stream);
}

int proj_adjoints(const ProjDims& d, const float* dtheta_w, float* dx, float* du, bool overwrite_dx, ProjScratch& s,
                  cudaStream_t stream, bool dtheta_amax_known) {
    const int M = (int)d.M;
    if (int rc = split_f16(dtheta_w, d.ldw, (long long)M * d.ldw, s.dth_hi, s.dth_lo, d.ldw, (long long)M * d.ldw, M,
                           d.tl, d.B, s.amax + 2, stream, dtheta_amax_known))
        return rc;
    {
        // dx (M x D) (+)= sum_b dtheta_b (M x tl, K-major) * u_b^T (u_b: D rows x tl, K-major)
        const SplitOperand A = {s.dth_hi, s.dth_lo, 0, d.ldw, (long long)M * d.ldw, s.amax + 2};
        const SplitOperand Bop = {s.u_hi, s.u_lo, 0, d.ldw, (long long)d.D * d.ldw, s.amax + 1};
        // Few output tiles (M / 128 x D / 256) and a contraction over the whole batch and window: gemm_split3_runs
        // says into how many runs it is worth cutting; their partial results are added in a fixed order.  Kernel
        // times against one run (or two halves of the batch), dx / du: B8 D16 N4 L256 46 -> 15 / 11 us, B5 D181 N12
        // L1003 114 -> 31 / 70 -> 28 us, B64 D128 N16 L720 467 -> 133 / 141 us; adding the parts takes 4 us at
        // these sizes.
        GemmShape shape = {M, d.D, d.tl, d.B, 1, overwrite_dx ? 0 : 1, d.D, 0, 1, 0};
        if (s.dx_runs > 1) {
            shape.beta = 0;
            shape.ksplit = s.dx_runs;
            shape.c_part_stride = (long long)up((size_t)M * d.D, 4);
            if (int rc = gemm_split3(A, Bop, s.part, shape, stream)) return rc;
            const int runs = std::min<long long>(s.dx_runs, gemm_split3_blocks(shape));
            if (int rc = add_parts(dx, d.D, s.part, d.D, shape.c_part_stride, runs, M, d.D, overwrite_dx, stream)) return rc;
        } else if (int rc = gemm_split3(A, Bop, dx, shape, stream)) {
            return rc;
        }
    }
    {
        // du_b (D x tl) += x^T (x stored M rows x D: K rows, output-row index contiguous -> MN-major)
        //                  * dtheta_b (M x tl: K rows, N contiguous -> MN-major)
        const SplitOperand A = {s.x_hi, s.x_lo, 1, s.Dp, 0, s.amax + 0};
        const SplitOperand Bop = {s.dth_hi, s.dth_lo, 1, d.ldw, (long long)M * d.ldw, s.amax + 2};
        GemmShape shape = {d.D, d.tl, M, d.B, 0, 1, d.L, (long long)d.D * d.L, 1, 0};
        if (s.du_runs > 1) {
            shape.beta = 0;
            shape.ldc = d.tl;
            shape.c_batch_stride = (long long)d.D * d.tl;
            shape.ksplit = s.du_runs;
            shape.c_part_stride = (long long)d.B * d.D * d.ldw;
            if (int rc = gemm_split3(A, Bop, s.part, shape, stream)) return rc;
            const int runs = std::min<long long>(s.du_runs, gemm_split3_blocks(shape));
            // all rows of all batch entries: du's rows are L apart, the window's tl columns of each are added to
            return add_parts(du + d.t0, d.L, s.part, d.tl, shape.c_part_stride, runs, (long long)d.B * d.D, d.tl, false,
                             stream);
        }
        return gemm_split3(A, Bop, du + d.t0, shape, stream);
    }
}

}  // namespace aussm
