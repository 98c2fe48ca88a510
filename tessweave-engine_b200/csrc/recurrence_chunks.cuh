// What the recurrences in chunks of 64 tokens share (recurrence_chunks.cu, delta_chunks.cu): the key size of a head (TW_DK), 32-bit
// numbers as three bf16 terms, products of such terms on the tensor cores, and where a request's chunks lie in scratch memory.
#pragma once

#include "attention_common.cuh"

#ifndef TW_DK
#define TW_DK 128
#endif

namespace {

typedef __nv_bfloat16 bf16;
using tw_attn::ldmatrix_x4;
using tw_attn::ldmatrix_x4_trans;
using tw_attn::mma_bf16;

constexpr int L = 64, DK = TW_DK, KT = DK / 16, RS = DK + 8, MS = L + 8, THREADS = 256, WARPS = 8;
static_assert(DK == 32 || DK == 64 || DK == 128, "key sizes");

// (x, y) as three pairs of bf16 whose sum is the pair to 24 bits
__device__ __forceinline__ void split3(float x, float y, uint32_t& a, uint32_t& b, uint32_t& c) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    const float2 hf = __bfloat1622float2(h);
    x -= hf.x; y -= hf.y;
    const __nv_bfloat162 m = __floats2bfloat162_rn(x, y);
    const float2 mf = __bfloat1622float2(m);
    const __nv_bfloat162 l = __floats2bfloat162_rn(x - mf.x, y - mf.y);
    a = *reinterpret_cast<const uint32_t*>(&h);
    b = *reinterpret_cast<const uint32_t*>(&m);
    c = *reinterpret_cast<const uint32_t*>(&l);
}
// A product of the leading terms: sixteen products summed by the tensor core, added to the running sum by an fp32 addition
// that rounds to nearest (the tensor core's own additions truncate: chained over a whole sum they left errors of 2 to 3 times
// the token kernel's).  The products of the smaller terms are chained (mma_bf16), in sums of their own or before the others.
__device__ __forceinline__ void mma_top(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    float t[4] = {0.f, 0.f, 0.f, 0.f};
    mma_bf16(t, a, b0, b1);
    d[0] += t[0]; d[1] += t[1]; d[2] += t[2]; d[3] += t[3];
}

// Chunks of the requests before s that are served here: where the request's own chunks start.
__device__ __forceinline__ int first_chunk(const int* seq_q_len, int s, int min_len) {
    int n = 0;
    for (int r = threadIdx.x & 31; r < s; r += 32) {
        const int len = seq_q_len[r];
        n += len >= min_len ? (len + L - 1) / L : 0;
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) n += __shfl_xor_sync(0xffffffffu, n, o);
    return n;
}

// Two neighbouring channels of a token into rows of three terms [3][L][RS].
__device__ __forceinline__ void put3(bf16* dst, int t, int i, float x, float y) {
    uint32_t hi, mid, lo;
    split3(x, y, hi, mid, lo);
    *reinterpret_cast<uint32_t*>(dst + t * RS + i) = hi;
    *reinterpret_cast<uint32_t*>(dst + (L + t) * RS + i) = mid;
    *reinterpret_cast<uint32_t*>(dst + (2 * L + t) * RS + i) = lo;
}
}  // namespace
