// Point-major [ng, ns] to species-major [ns, ng] copies and back, FP64.
//
// One matrix side is a few dozen to a few hundred species, the other the grid.
// A CTA moves 64 points x up to 64 species through shared memory, both sides in
// whole rows: a point's species are one contiguous run, a species' 64 points
// another (512 bytes).  The row stride of 65 doubles keeps the column reads free
// of bank conflicts.  Bound by L2/HBM bandwidth; on B200, 53 species, 32768
// points (13.9 MB each way): 8.5 us against 33 us for a strided copy; 2^20 points
// 174 us (5.1 TB/s) against 1091 us.  Streaming hints on both sides: without
// them four copies a step pushed the generated kernel's code out of L2, and
// that kernel took 218 us instead of 103.
#include <cuda_runtime.h>

#include <cstdint>

#include "../../include/chemgen_b200.h"

namespace {

constexpr int kT = 64, kThreads = 256;

// dst[c][r] = src[r][c] for r < rows, c < cols (src row stride cols, dst rows).
__global__ void __launch_bounds__(kThreads) transpose_kernel(const double* __restrict__ src, int64_t rows, int64_t cols,
                                                             double* __restrict__ dst) {
    __shared__ double s[kT][kT + 1];
    // neighbouring CTAs share the short side's rows
    const int64_t gr = (rows + kT - 1) / kT, gc = (cols + kT - 1) / kT;
    const int64_t r0 = (gr > gc ? blockIdx.x / gc : blockIdx.x % gr) * kT;
    const int64_t c0 = (gr > gc ? blockIdx.x % gc : blockIdx.x / gr) * kT;
    const int nr = (int)min((int64_t)kT, rows - r0), nc = (int)min((int64_t)kT, cols - c0);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int j = 0; j < kT / 8; ++j) {
        const int r = warp + 8 * j;
        if (r < nr) {
            const double* p = src + (r0 + r) * cols + c0;
            if (lane < nc) s[r][lane] = __ldcs(p + lane);
            if (lane + 32 < nc) s[r][lane + 32] = __ldcs(p + lane + 32);
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kT / 8; ++j) {
        const int c = warp + 8 * j;
        if (c < nc) {
            double* p = dst + (c0 + c) * rows + r0;
            if (lane < nr) __stcs(p + lane, s[lane][c]);
            if (lane + 32 < nr) __stcs(p + lane + 32, s[lane + 32][c]);
        }
    }
}

}  // namespace

extern "C" int chemgen_transpose(const double* src, int64_t rows, int64_t cols, double* dst, void* stream) {
    if (rows < 0 || cols < 0) return CHEMGEN_ERR_INVALID_ARGUMENT;
    if (rows == 0 || cols == 0) return CHEMGEN_OK;
    if (!src || !dst) return CHEMGEN_ERR_INVALID_ARGUMENT;
    if ((reinterpret_cast<uintptr_t>(src) & 7u) || (reinterpret_cast<uintptr_t>(dst) & 7u)) return CHEMGEN_ERR_MISALIGNED;
    const int64_t gr = (rows + kT - 1) / kT, gc = (cols + kT - 1) / kT;
    if (gr * gc > 0x7fffffff) return CHEMGEN_ERR_TOO_LARGE;
    transpose_kernel<<<(unsigned)(gr * gc), kThreads, 0, (cudaStream_t)stream>>>(src, rows, cols, dst);
    return cudaGetLastError() == cudaSuccess ? CHEMGEN_OK : CHEMGEN_ERR_CUDA;
}
