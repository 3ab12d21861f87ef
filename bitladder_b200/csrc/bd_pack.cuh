// Quantize-pack of a block's K or V by groups of kPackThreads threads, for the kernels that do it (bd_pack.cu; bd_decode_short.cu
// where a step fills a tail).  The arithmetic and its source are told in bd_pack.cu; what uses this is compiled without
// --use_fast_math (subnormal differences of bf16 rows must not be flushed).
#pragma once

#include <type_traits>
#include "bd_common.cuh"
#include "bd_kernels.h"

namespace bd {

template <bool BF16>
__device__ __forceinline__ float2 pair_to_float2(uint32_t w) {
    if constexpr (BF16) {
        return make_float2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
    } else {
        return __half22float2(*reinterpret_cast<__half2 *>(&w));
    }
}

// Running min / max of packed pairs in their own format (exact: no rounding is involved, and a
// NaN operand yields the other operand, like fminf / fmaxf).  +inf / -inf as the neutral starts.
template <bool BF16>
__device__ __forceinline__ uint32_t pair_min(uint32_t a, uint32_t b) {
    if constexpr (BF16) {
        __nv_bfloat162 r = __hmin2(*reinterpret_cast<__nv_bfloat162 *>(&a), *reinterpret_cast<__nv_bfloat162 *>(&b));
        return *reinterpret_cast<uint32_t *>(&r);
    } else {
        __half2 r = __hmin2(*reinterpret_cast<__half2 *>(&a), *reinterpret_cast<__half2 *>(&b));
        return *reinterpret_cast<uint32_t *>(&r);
    }
}
template <bool BF16>
__device__ __forceinline__ uint32_t pair_max(uint32_t a, uint32_t b) {
    if constexpr (BF16) {
        __nv_bfloat162 r = __hmax2(*reinterpret_cast<__nv_bfloat162 *>(&a), *reinterpret_cast<__nv_bfloat162 *>(&b));
        return *reinterpret_cast<uint32_t *>(&r);
    } else {
        __half2 r = __hmax2(*reinterpret_cast<__half2 *>(&a), *reinterpret_cast<__half2 *>(&b));
        return *reinterpret_cast<uint32_t *>(&r);
    }
}
template <bool BF16> constexpr uint32_t kPairPosInf = BF16 ? 0x7f807f80u : 0x7c007c00u;
template <bool BF16> constexpr uint32_t kPairNegInf = BF16 ? 0xff80ff80u : 0xfc00fc00u;

// Code of x as a bit field, in four instructions (subtract, multiply, add, logic op).
//   v = (x - mn) * scale_inv lies in [0, maxv + 1e-6] (x >= mn, and (mx - mn) * fl(maxv / (mx - mn))
//   exceeds maxv by a few ulps at most), or is NaN (NaN or infinite inputs), which the reference's
//   fminf(fmaxf(roundf(v), 0), maxv) turns into 0; its clamp from above never acts.
//   * The multiply is by scale_inv / 2^BITS (a power of two: the product is v / 2^BITS, rounded exactly
//     as v is) with saturation to [0, 1], which also turns NaN into 0: t = v / 2^BITS in [0, 1).
//   * t + (2^m + 2^-(BITS+1)), rounded toward zero, leaves floor(v + 0.5) = roundf(v) (v >= 0, ties
//     away from zero) in the mantissa at bit 23 - m - BITS and up: the ulp of the sum is 2^(m-23), the
//     half is representable beside 2^m for m <= 22 - BITS, and cutting first to that ulp and then to
//     the integer is one floor.  m is chosen per field so that the code lands where the field sits in
//     the 16-bit word (field 0 one bit higher, shifted down afterwards).
template <int BITS, int J>
__device__ __forceinline__ uint32_t put_field(uint32_t acc, float x, float mn, float scale_inv_div) {
    constexpr int kPos = (J == 0) ? 1 : BITS * J;                  // bit where the code lands
    constexpr int m = 23 - BITS - kPos;
    static_assert(m >= 0 && m <= 22 - BITS, "magic constant out of range");
    constexpr float kMagic = float(1u << m) + 1.0f / float(1u << (BITS + 1));
    float t;
    asm("mul.rn.sat.f32 %0, %1, %2;" : "=f"(t) : "f"(__fsub_rn(x, mn)), "f"(scale_inv_div));
    const uint32_t bits = __float_as_uint(__fadd_rz(t, kMagic));
    constexpr uint32_t kMask = ((1u << BITS) - 1u) << (BITS * J);
    if constexpr (J == 0) return acc | ((bits >> 1) & kMask);
    else return acc | (bits & kMask);
}

// approx_div: divide the way the reference does as it is shipped (built with --use_fast_math,
// setup.py:149): maxv / range becomes maxv times the GPU's approximate reciprocal, which is one ulp
// off the IEEE quotient in about a quarter of the groups and so moves a code by one step where
// (x - mn) * maxv / range is exactly k + 0.5.  Same bytes as that build on the same GPU; not
// reproducible on a CPU.  Default (0): IEEE division, the bytes the reference writes when built
// without that flag, and what a CPU evaluation of the formulas gives.
__device__ __forceinline__ void scale_from_minmax(float mn, float mx, float maxv, bool approx_div, float &scale_inv,
                                                  float &scale) {
    const float range = __fsub_rn(mx, mn);
    if (approx_div) {
        scale_inv = (range > 0.0f) ? __fdividef(maxv, range) : 0.0f;
        scale = (scale_inv == 0.0f) ? 0.0f : __fdividef(1.0f, scale_inv);
    } else {
        scale_inv = (range > 0.0f) ? __fdiv_rn(maxv, range) : 0.0f;
        scale = (scale_inv == 0.0f) ? 0.0f : __frcp_rn(scale_inv);
    }
}

// Where the parameters of (group g of the block / 128-token run, element c of 0..127) are stored:
// natural order, except 4-bit with group 32, where the reference keeps the order of its MMA
// fragments (csrc/bit_decode/src/flash_fwd_kernel.h:939-957 with num_params = 4): row
// 2*(g%2) + (c/8)%2, fp16 column 16*(c/16) + 8*(g/2) + c%8.  Pairs (c even, c + 1) stay adjacent.
template <int BITS, int GROUP>
__device__ __forceinline__ void param_slot(int g, int c, int &row, int &col) {
    if constexpr (BITS == 4 && GROUP == 32) {
        row = 2 * (g & 1) + ((c >> 3) & 1);
        col = 16 * (c >> 4) + 8 * (g >> 1) + (c & 7);
    } else {
        row = g;
        col = c;
    }
}

__device__ __forceinline__ const uint16_t *kin_of(const PackParams &p) { return static_cast<const uint16_t *>(p.k); }
__device__ __forceinline__ const uint16_t *vin_of(const PackParams &p) { return static_cast<const uint16_t *>(p.v); }

// A block of a head is the work of 2 * kPackSplit CTAs of 128 threads: kPackSplit share its K by channels, as many its
// V by tokens.  A CTA is three phases (load, reduce, quantize and store) that cannot overlap inside it, so what keeps
// HBM busy is eight small CTAs per SM in different phases (1024 threads of 64 registers), each thread with 32 words
// of input in flight.  Measured, 4 bits / 2 bits, 8 x 32768 x 8 heads and 2 x 16384 x 32 heads (group 64, bf16),
// graph replay: one CTA of 256 threads for K and then V (768 / 512 threads per SM) 212.5 / 135.7 us; split 2 ways
// 197.6 / 110.0, 4 ways 203.7 / 102.9; with fewer resident threads (768) 216.4 / 105.2.
template <int BITS> constexpr int kPackSplit = BITS == 4 ? 2 : 4;
template <int BITS> constexpr int kPackSubsets = BITS == 4 ? 4 : 8;         // token subsets of the K half
template <int BITS> constexpr int kPackThreads = (64 / kPackSplit<BITS>) * kPackSubsets<BITS>;

template <int BITS, int GROUP>
struct PackCfg {
    static constexpr int P = 16 / BITS;             // codes per 16-bit word
    static constexpr int NB = 32 * P;               // tokens per pack block
    static constexpr int SPLIT = kPackSplit<BITS>;  // parts of a block's K (by channels), and of its V (by tokens)
    static constexpr int KP = 64 / SPLIT;           // channel pairs of a part (K)
    static constexpr int NT = kPackSubsets<BITS>;   // token subsets (K)
    static constexpr int NTHREADS = KP * NT;
    static constexpr int PPT = 32 / NT;             // pack rows per thread (K)
    static constexpr int NGK = NB / GROUP;          // K token groups per block
    static constexpr int FPG = GROUP / 32;          // K fields per group
    static constexpr int DP = kHeadDim / P;         // words per V row
    static constexpr int NGD = kHeadDim / GROUP;    // V dim groups
    static constexpr int FPGV = P / NGD;            // V fields per dim group
    union Shared {
        struct {
            uint32_t red[NT][NGK][2][KP];   // K: minima and maxima of the token subsets, two channels each, in the input format
            float4 coef[NGK][KP];           //    and what the groups are quantized with: zeros and scaled inverses of two channels
        } k;
        __half vprm[NGD][2][NB / SPLIT];    // V: scales and zeros of the part's tokens
    };
};

// Part `part` of the K of block `blk` (of the source rows) of KV head ih of sequence ib, into block dst_blk; `sync` is a
// barrier of the group's threads, `tid` the thread's number among them.
template <int BITS, int GROUP, bool BF16, class Sync>
__device__ __forceinline__ void pack_k_part(const PackParams &p, typename PackCfg<BITS, GROUP>::Shared &sh, int tid, int ib, int ih,
                                            int part, int blk, int dst_blk, Sync sync) {
    using C = PackCfg<BITS, GROUP>;
    constexpr int P = C::P, NB = C::NB, KP = C::KP, NT = C::NT, NTHREADS = C::NTHREADS, PPT = C::PPT, NGK = C::NGK, FPG = C::FPG;
    constexpr int D = kHeadDim;
    const float maxv = static_cast<float>((1 << BITS) - 1);
    const bool approx_div = p.approx_div != 0;
    const int cl = tid % KP, T = tid / KP, cp = part * KP + cl;
    const uint16_t *kbase = kin_of(p) + ib * p.k_stride_b + static_cast<int64_t>(blk) * NB * p.k_stride_s +
                            ih * p.k_stride_h + 2 * cp;
    uint32_t raw[PPT][P];
#pragma unroll
    for (int pi = 0; pi < PPT; ++pi)
#pragma unroll
        for (int j = 0; j < P; ++j) {
            const int t = T * PPT + pi + 32 * j;
            raw[pi][j] = *reinterpret_cast<const unsigned int *>(kbase + t * p.k_stride_s);
        }
    {
        uint32_t pmn[NGK], pmx[NGK];        // both channels at once, in the input format
#pragma unroll
        for (int gk = 0; gk < NGK; ++gk) { pmn[gk] = kPairPosInf<BF16>; pmx[gk] = kPairNegInf<BF16>; }
#pragma unroll
        for (int pi = 0; pi < PPT; ++pi)
#pragma unroll
            for (int j = 0; j < P; ++j) {
                const int gk = j / FPG;
                pmn[gk] = pair_min<BF16>(pmn[gk], raw[pi][j]);
                pmx[gk] = pair_max<BF16>(pmx[gk], raw[pi][j]);
            }
#pragma unroll
        for (int gk = 0; gk < NGK; ++gk) {
            sh.k.red[T][gk][0][cl] = pmn[gk];
            sh.k.red[T][gk][1][cl] = pmx[gk];
        }
    }
    sync();
    // One thread per (group, channel pair) works out the scales (two IEEE divisions a channel cost as much as
    // twenty of its codes) and stores the parameters; the others take them from shared memory.
    for (int i = tid; i < NGK * KP; i += NTHREADS) {
        const int gk = i / KP, c = i % KP;
        uint32_t a = sh.k.red[0][gk][0][c], b = sh.k.red[0][gk][1][c];
#pragma unroll
        for (int t2 = 1; t2 < NT; ++t2) {
            a = pair_min<BF16>(a, sh.k.red[t2][gk][0][c]);
            b = pair_max<BF16>(b, sh.k.red[t2][gk][1][c]);
        }
        const float2 lo = pair_to_float2<BF16>(a), hi = pair_to_float2<BF16>(b);
        float si0, si1, sc0, sc1;
        scale_from_minmax(lo.x, hi.x, maxv, approx_div, si0, sc0);
        scale_from_minmax(lo.y, hi.y, maxv, approx_div, si1, sc1);
        constexpr float kDiv = 1.0f / float(1 << BITS);      // exact; see put_field
        sh.k.coef[gk][c] = make_float4(lo.x, lo.y, si0 * kDiv, si1 * kDiv);
        int prow, pcol;
        param_slot<BITS, GROUP>(gk, 2 * (cp - cl + c), prow, pcol);
        const int64_t grow = static_cast<int64_t>(dst_blk) * NGK + prow;
        __half *prm = reinterpret_cast<__half *>(p.k_params) + 2 * (ib * p.k_params_stride_b + (grow * p.h_k + ih) * D);
        *reinterpret_cast<__half2 *>(prm + pcol) = __floats2half2_rn(sc0, sc1);
        *reinterpret_cast<__half2 *>(prm + D + pcol) = __floats2half2_rn(lo.x, lo.y);
    }
    sync();
    float4 coef[NGK];
#pragma unroll
    for (int gk = 0; gk < NGK; ++gk) coef[gk] = sh.k.coef[gk][cl];
    uint16_t *kp = static_cast<uint16_t *>(p.k_pack) + ib * p.k_pack_stride_b +
                   ((static_cast<int64_t>(dst_blk) * 32 + T * PPT) * p.h_k + ih) * D + 2 * cp;
#pragma unroll
    for (int pi = 0; pi < PPT; ++pi) {
        uint32_t lo = 0, hi = 0;
        auto put = [&](auto jc) {
            constexpr int J = decltype(jc)::value;
            const float2 x = pair_to_float2<BF16>(raw[pi][J]);
            constexpr int gk = J / FPG;
            lo = put_field<BITS, J>(lo, x.x, coef[gk].x, coef[gk].z);
            hi = put_field<BITS, J>(hi, x.y, coef[gk].y, coef[gk].w);
        };
        put(std::integral_constant<int, 0>{}); put(std::integral_constant<int, 1>{});
        put(std::integral_constant<int, 2>{}); put(std::integral_constant<int, 3>{});
        if constexpr (P == 8) {
            put(std::integral_constant<int, 4>{}); put(std::integral_constant<int, 5>{});
            put(std::integral_constant<int, 6>{}); put(std::integral_constant<int, 7>{});
        }
        *reinterpret_cast<uint32_t *>(kp + static_cast<int64_t>(pi) * p.h_k * D) = lo | (hi << 16);
    }
}

// The same for a part of the block's V.
template <int BITS, int GROUP, bool BF16, class Sync>
__device__ __forceinline__ void pack_v_part(const PackParams &p, typename PackCfg<BITS, GROUP>::Shared &sh, int tid, int ib, int ih,
                                            int part, int blk, int dst_blk, Sync sync) {
    using C = PackCfg<BITS, GROUP>;
    constexpr int P = C::P, NB = C::NB, SPLIT = C::SPLIT, NTHREADS = C::NTHREADS, DP = C::DP, NGD = C::NGD, FPGV = C::FPGV;
    const float maxv = static_cast<float>((1 << BITS) - 1);
    const bool approx_div = p.approx_div != 0;
    // A thread owns 8 consecutive output words of one token (one 16-byte store) and so needs,
    // for every field j, the 8 dims  p0 + DP*j .. +7: P loads of 16 bytes.  DP/8 threads per token
    // (4 at 4 bits, 2 at 2 bits): the min/max over a token's group takes one or two shuffles.
    constexpr int TPT = DP / 8;              // threads per token
    constexpr int TPI = NTHREADS / TPT;      // tokens per iteration
    constexpr int VITER = NB / SPLIT / TPI;
    static_assert(VITER * TPI * SPLIT == NB, "token tiling");
    const int tok0 = part * (NB / SPLIT);                 // this part's tokens start here
    const int q8 = tid % TPT, tsub = tid / TPT;
    const uint16_t *vbase = vin_of(p) + ib * p.v_stride_b + static_cast<int64_t>(blk) * NB * p.v_stride_s +
                            ih * p.v_stride_h + 8 * q8;
    uint16_t *vp = static_cast<uint16_t *>(p.v_pack) + ib * p.v_pack_stride_b +
                   (static_cast<int64_t>(dst_blk) * NB * p.h_k + ih) * DP + 8 * q8;
    uint4 raw[VITER][P];
#pragma unroll
    for (int u = 0; u < VITER; ++u) {
        const int t = tok0 + u * TPI + tsub;
#pragma unroll
        for (int j = 0; j < P; ++j)
            raw[u][j] = *reinterpret_cast<const uint4 *>(vbase + t * p.v_stride_s + DP * j);
    }
    // Minima and maxima of all the thread's tokens first; then the lanes that share a token divide the (token, dim
    // group) pairs among themselves: one lane works out a pair's scales and hands the inverse to the others.
    float mn[VITER][NGD], mx[VITER][NGD], sinv[VITER][NGD];
#pragma unroll
    for (int u = 0; u < VITER; ++u)
#pragma unroll
        for (int gd = 0; gd < NGD; ++gd) {
            uint32_t pmn = kPairPosInf<BF16>, pmx = kPairNegInf<BF16>;
#pragma unroll
            for (int j = gd * FPGV; j < (gd + 1) * FPGV; ++j) {
                const uint32_t w4[4] = {raw[u][j].x, raw[u][j].y, raw[u][j].z, raw[u][j].w};
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    pmn = pair_min<BF16>(pmn, w4[r]);
                    pmx = pair_max<BF16>(pmx, w4[r]);
                }
            }
#pragma unroll
            for (int off = 1; off < TPT; off <<= 1) {
                pmn = pair_min<BF16>(pmn, __shfl_xor_sync(0xffffffffu, pmn, off));
                pmx = pair_max<BF16>(pmx, __shfl_xor_sync(0xffffffffu, pmx, off));
            }
            const float2 a = pair_to_float2<BF16>(pmn), b2 = pair_to_float2<BF16>(pmx);
            mn[u][gd] = fminf(a.x, a.y);
            mx[u][gd] = fmaxf(b2.x, b2.y);
        }
    constexpr int ITEMS = VITER * NGD;
#pragma unroll
    for (int i0 = 0; i0 < ITEMS; i0 += TPT) {
        float lo = mn[i0 / NGD][i0 % NGD], hi = mx[i0 / NGD][i0 % NGD];
#pragma unroll
        for (int i = 1; i < TPT; ++i)
            if (i0 + i < ITEMS && q8 == i) { lo = mn[(i0 + i) / NGD][(i0 + i) % NGD]; hi = mx[(i0 + i) / NGD][(i0 + i) % NGD]; }
        float si, sc;
        scale_from_minmax(lo, hi, maxv, approx_div, si, sc);
        si *= 1.0f / float(1 << BITS);                   // exact; see put_field
        if (i0 + q8 < ITEMS) {
            const int u = (i0 + q8) / NGD, gd = (i0 + q8) % NGD;
            sh.vprm[gd][0][u * TPI + tsub] = __float2half_rn(sc);
            sh.vprm[gd][1][u * TPI + tsub] = __float2half_rn(lo);
        }
#pragma unroll
        for (int i = 0; i < TPT; ++i)
            if (i0 + i < ITEMS) sinv[(i0 + i) / NGD][(i0 + i) % NGD] = __shfl_sync(0xffffffffu, si, i, TPT);
    }
#pragma unroll
    for (int u = 0; u < VITER; ++u) {
        const int t = u * TPI + tsub;
        uint32_t outw[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            uint32_t lo = 0, hi = 0;
            auto put = [&](auto jc) {
                constexpr int J = decltype(jc)::value;
                const uint32_t w = r == 0 ? raw[u][J].x : (r == 1 ? raw[u][J].y : (r == 2 ? raw[u][J].z : raw[u][J].w));
                const float2 x = pair_to_float2<BF16>(w);
                constexpr int gd = J / FPGV;
                lo = put_field<BITS, J>(lo, x.x, mn[u][gd], sinv[u][gd]);
                hi = put_field<BITS, J>(hi, x.y, mn[u][gd], sinv[u][gd]);
            };
            put(std::integral_constant<int, 0>{}); put(std::integral_constant<int, 1>{});
            put(std::integral_constant<int, 2>{}); put(std::integral_constant<int, 3>{});
            if constexpr (P == 8) {
                put(std::integral_constant<int, 4>{}); put(std::integral_constant<int, 5>{});
                put(std::integral_constant<int, 6>{}); put(std::integral_constant<int, 7>{});
            }
            outw[r] = lo | (hi << 16);
        }
        *reinterpret_cast<uint4 *>(vp + static_cast<int64_t>(tok0 + t) * p.h_k * DP) = make_uint4(outw[0], outw[1], outw[2], outw[3]);
    }
    sync();
    // scales / zeros of these tokens: per dim group, per run of 128 tokens, 128 scales then 128 zeros.
    constexpr int RUNS = NB / 128, W = NB / SPLIT / 2;      // W: token pairs of this CTA
    const int64_t run0 = static_cast<int64_t>(dst_blk) * RUNS;
    for (int i = tid; i < NGD * 2 * W; i += NTHREADS) {
        const int w = i % W, z = (i / W) & 1, gd = i / (2 * W);      // z: 0 scales, 1 zeros
        const int t = tok0 + 2 * w;
        int plane, pcol;
        param_slot<BITS, GROUP>(gd, t & 127, plane, pcol);
        __half *dst = reinterpret_cast<__half *>(p.v_params) +
                      2 * (ib * p.v_params_stride_b + plane * p.v_params_stride_g + ih * p.v_params_stride_h) +
                      256 * (run0 + (t >> 7)) + 128 * z + pcol;
        *reinterpret_cast<__half2 *>(dst) = *reinterpret_cast<const __half2 *>(&sh.vprm[gd][z][2 * w]);
    }
}

}  // namespace bd
