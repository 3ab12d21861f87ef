// What the decode kernels (bd_decode.cu, bd_decode_short.cu) share: packed fields as MMA operands, where scales and zeros
// lie, the online-softmax step.
#pragma once

#include "bd_common.cuh"
#include "bd_kernels.h"

#ifndef BD_SUBNORMAL_CODES
#define BD_SUBNORMAL_CODES 1
#endif

namespace bd {

constexpr int kSmemLimit = 232448;     // 227 KB of shared memory per CTA
constexpr float kRescaleSlack = 8.0f;  // keep a stale row max until it is exceeded by 2^8

// A packed 32-bit register (two 16-bit words) and the helper word the field extraction
// needs: 4-bit: the high bytes of both words moved to the low bytes (one byte permute);
// 2-bit: the register shifted right by 10.
template <int BITS>
__device__ __forceinline__ uint32_t aux_word(uint32_t w) {
    if constexpr (BITS == 4) return __byte_perm(w, 0u, 0x4341u);
    else return w >> 10;
}
// Field j of a packed word as two fp16 lanes, every field inside the fp16 mantissa.
//
// 4-bit words are taken apart in PAIRS: an even field comes out together with the odd
// field above it (f_j + 16 f_{j+1}, a whole byte: still an exact fp16 subnormal), the odd
// field alone (16 f_{j+1}).  The products are linear, so the even field's sum is the
// difference of the two accumulators, taken once after the last MMA; that saves the
// shift and one of the masks on the high byte.  kFieldPairs tells the callers (with one field
// per quantization group, group 32, the two fields of a byte have different scales and every
// field is masked out alone).
template <int BITS, int J, bool PAIRS>
__device__ __forceinline__ uint32_t field(uint32_t w, uint32_t aux) {
    uint32_t x;
    if constexpr (BITS == 4) {
        if constexpr (J == 0) x = w & (PAIRS ? 0x00ff00ffu : 0x000f000fu);
        else if constexpr (J == 1) x = w & 0x00f000f0u;
        else if constexpr (J == 2) x = PAIRS ? aux : (aux & 0x000f000fu);
        else x = aux & 0x00f000f0u;
    } else {
        constexpr uint32_t m = 0x00030003u << (2 * (J < 5 ? J : J - 5));
        x = ((J < 5) ? w : aux) & m;
    }
#if !BD_SUBNORMAL_CODES
    x |= 0x64006400u;   // 1024 + value, then remove the 1024 exactly
    __half2 h = __hsub2(*reinterpret_cast<__half2 *>(&x), __half2half2(__ushort_as_half(0x6400)));
    x = *reinterpret_cast<uint32_t *>(&h);
#endif
    return x;
}
// Pairs need both fields of a byte to meet the same scale: two or more fields per group.
template <int BITS, int GROUP> constexpr bool kFieldPairs = (BITS == 4 && GROUP >= 64);
// Value of the fp16 lane produced by field<J> divided by the code.
template <int BITS>
__host__ __device__ constexpr float field_weight(int j) {
    float f = 1.0f;
    if (BITS == 4) {
        f = (j & 1) ? 16.0f : 1.0f;
    } else {
        int e = j < 5 ? j : j - 5;
        for (int i = 0; i < e; ++i) f *= 4.0f;
    }
#if BD_SUBNORMAL_CODES
    return f * (1.0f / 16777216.0f);
#else
    return f;
#endif
}

// Byte offset, inside a warp's K parameter tile, of the 8 scales of token group gk for channels
// 32a + 8l .. +7 (the zeros sit 256 bytes on), and inside its V parameter tile of the scales of
// tokens r0, r0 + 1 (hi = 0) or r0 + 8, r0 + 9 (hi = 1) of dim group gd, r0 even with r0 % 16 < 8.
// Natural order, except 4-bit with group 32: the reference's fragment order (element c of group g in
// row 2*(g%2) + (c/8)%2, column 16*(c/16) + 8*(g/2) + c%8; flash_fwd_kernel.h:939-957).
template <int BITS, int GROUP>
__device__ __forceinline__ uint32_t kprm_off(int gk, int a, int l) {
    if constexpr (BITS == 4 && GROUP == 32) return (2 * (gk & 1) + (l & 1)) * 512 + (16 * (2 * a + (l >> 1)) + 8 * (gk >> 1)) * 2;
    else return gk * 512 + (32 * a + 8 * l) * 2;
}
template <int BITS, int GROUP>
__device__ __forceinline__ uint32_t vprm_off(int gd, int r0, int hi) {
    constexpr int RUNS = (32 * (16 / BITS)) / 128;
    if constexpr (BITS == 4 && GROUP == 32) return (2 * (gd & 1) + hi) * 512 + (16 * (r0 >> 4) + 8 * (gd >> 1) + (r0 & 7)) * 2;
    else return gd * (RUNS * 512) + (r0 >> 7) * 512 + (r0 & 127) * 2 + 16 * hi;
}

// One online-softmax step for NT score tiles (m16n8 accumulators, columns = query
// rows).  On entry t holds the scores in log2 units MINUS the running maximum of
// their column (minus 0 while the column has no maximum yet); on exit it holds
// the probabilities.  The running max moves lazily: only when it is exceeded by
// more than 2^kRescaleSlack, so probabilities stay below 2^8 and the accumulators
// are rescaled a handful of times per sequence.  With ACC_L the probabilities are
// also added to l_run (otherwise the caller gets the row sums elsewhere).
// Returns true when a rescale happened (f holds the factor per column parity).
template <int NT, bool ACC_L, int NZ>
__device__ __forceinline__ bool softmax_step(float (&t)[NT][4], float (&m_run)[2], float (&l_run)[2],
                                             float (&O)[8][4], float (&ZS)[NZ][4], float (&f)[2]) {
    float cmax[2] = {-INFINITY, -INFINITY};
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) cmax[e & 1] = fmaxf(cmax[e & 1], t[j][e]);
#pragma unroll
    for (int c = 0; c < 2; ++c) {
        cmax[c] = fmaxf(cmax[c], __shfl_xor_sync(0xffffffffu, cmax[c], 4));
        cmax[c] = fmaxf(cmax[c], __shfl_xor_sync(0xffffffffu, cmax[c], 8));
        cmax[c] = fmaxf(cmax[c], __shfl_xor_sync(0xffffffffu, cmax[c], 16));
    }
    bool changed = false;
#pragma unroll
    for (int c = 0; c < 2; ++c)
        changed |= cmax[c] > kRescaleSlack || (m_run[c] == -INFINITY && cmax[c] != -INFINITY);
    const bool any = __any_sync(0xffffffffu, changed);
    if (any) {
        float shift[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const bool first = m_run[c] == -INFINITY;
            const bool move = cmax[c] > kRescaleSlack || (first && cmax[c] != -INFINITY);
            shift[c] = move ? cmax[c] : 0.f;
            f[c] = move ? (first ? 0.f : ex2f(-cmax[c])) : 1.f;
            if (move) m_run[c] = (first ? 0.f : m_run[c]) + cmax[c];
            l_run[c] *= f[c];
        }
#pragma unroll
        for (int mt = 0; mt < 8; ++mt)
#pragma unroll
            for (int e = 0; e < 4; ++e) O[mt][e] *= f[e & 1];
#pragma unroll
        for (int z = 0; z < NZ; ++z)
#pragma unroll
            for (int e = 0; e < 4; ++e) ZS[z][e] *= f[e & 1];
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) t[j][e] -= shift[e & 1];
    }
#pragma unroll
    for (int j = 0; j < NT; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            t[j][e] = ex2f(t[j][e]);
            if (ACC_L) l_run[e & 1] += t[j][e];
        }
    return any;
}

}  // namespace bd
