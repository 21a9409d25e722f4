// isf_tc.cuh -- the operand layout of the tensor-core F(q,tau), shared by the
// kernels that make the operands and the GEMMs that read them.
#pragma once

#include <cuda_bf16.h>
#include <cstddef>

#include "pgb_device.cuh"

namespace pgb {

constexpr int kTM = 128;          // rows per tile

// Element index of (r, k) in a tile-ordered [rows x K] bf16 operand whose
// tiles are TR rows x 64 K: tile (r / TR, k / 64) is one contiguous block of
// TR * 64 elements in core-matrix order (8-row groups of 1024 B, 16-byte core
// rows, 128 B between core matrices along K).
__host__ __device__ __forceinline__ size_t tiled_index(int r, int k, int K, int TR) {
    const int rt = r / TR, rr = r - rt * TR, kc = k >> 6, kk = k & 63;
    return ((size_t)rt * (size_t)(K >> 6) + (size_t)kc) * (size_t)(TR * 64) +
           (size_t)((rr >> 3) * 512 + (kk >> 3) * 64 + (rr & 7) * 8 + (kk & 7));
}

__device__ __forceinline__ void split_bf16(float x, __nv_bfloat16& h, __nv_bfloat16& l) {
    h = __float2bfloat16_rn(x);
    l = __float2bfloat16_rn(x - __bfloat162float(h));
}

}  // namespace pgb
