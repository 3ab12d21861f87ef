// Split-KV decode attention over the packed low-bit KV cache where there is little of it: steps that are bound by the
// latency of their parts, not by memory.
//
// The same arithmetic on the same operands as bd_decode.cu (and so as the reference's split-KV kernel,
// csrc/bit_decode/src/flash_fwd_kernel.h:66-728), cut for latency:
//
//  * A thread-block cluster of 1, 2, 4 or 8 CTAs per (sequence, KV head).  A CTA needs the lengths of its own sequence
//    only: no table of units, no partition arithmetic in front of the first copy.
//  * The work item of a warp is HALF a pack block (16 pack rows: 64 tokens at 4 bits, 128 at 2) or 16 tokens of the
//    unquantized tail, dealt out in turn over all warps of the cluster.
//  * The warps' results are merged by all of them together: deposits in shared memory, a barrier, every warp an eighth of
//    the output; then the CTAs' results the same way in the shared memory of the cluster's first CTA.  No second
//    kernel, no trip to L2.
//  * With rotary embedding, q and the new key are rotated where they are loaded (bd_rope.cu's arithmetic).
//  * A decoder step's bookkeeping is done here too: the lengths move on, and a tail that is full behind the step is
//    packed by the cluster that has just read it (bd_pack.cuh): one kernel a token.
//
// Measured against bd_decode.cu, and the rule that chooses between them: short_cluster in bd_api.cu.
#include <atomic>
#include <type_traits>

#include "bd_decode.cuh"
#include "bd_pack.cuh"

namespace bd {

namespace {

template <int BITS, int GROUP, int NQT>
struct ShortCfg {
    static constexpr int P = 16 / BITS;
    static constexpr int NB = 32 * P;
    static constexpr int NGK = NB / GROUP;              // K token groups per block
    static constexpr int FPG = GROUP / 32;              // K fields per token group
    static constexpr int NGD = kHeadDim / GROUP;        // V dim groups
    static constexpr int NZ = (NGD + 1) / 2;            // accumulators of sum_t p_t * zero_t (two dim groups each)
    static constexpr int FPGV = P / NGD;                // V fields per dim group
    static constexpr int DP = kHeadDim / P;             // 16-bit words per V row
    static constexpr int RUNS = NB / 128;               // 128-token runs per block (V params)
    static constexpr int PRM = 512 * NGK;               // scales and zeros of a block, K or V
    static constexpr int CODE = 4096;                   // K or V codes of half a block
    static constexpr int WARPS = kShortWarps;
    static constexpr int THREADS = 32 * WARPS;
    static constexpr int NACC = 8 * NQT * 4 + 4 * NQT;  // floats per thread handed over in a merge
    static constexpr int DEPOSIT = NACC * 128;          // bytes of one result
    static constexpr int LIMIT = kSmemLimit - 1024;
    static constexpr int STAGES = WARPS * 2 * (2 * CODE + 2 * PRM) + 2 * DEPOSIT <= LIMIT ? 2 : 1;
    static constexpr int OFF_PRM = WARPS * STAGES * 2 * CODE;
    static constexpr int OFF_MERGE = OFF_PRM + WARPS * STAGES * 2 * PRM;          // the CTAs' results (first CTA of a cluster)
    static constexpr int FIT = (LIMIT - OFF_MERGE) / DEPOSIT;
    static constexpr int CLUSTER = FIT >= 8 ? 8 : (FIT >= 4 ? 4 : (FIT >= 2 ? 2 : 1));
    static constexpr int OFF_BAR = OFF_MERGE + CLUSTER * DEPOSIT;
    static constexpr int OFF_FLAGS = OFF_BAR + WARPS * STAGES * 16;
    static constexpr int SMEM = OFF_FLAGS + WARPS * 4;
    static_assert(DEPOSIT <= STAGES * 2 * CODE, "a warp's result fits its own tiles");
    static_assert(SMEM <= kSmemLimit, "shared memory");
};

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
// Stores into the shared memory of the cluster's first CTA, at the place that `addr` names in this CTA's.
__device__ __forceinline__ uint32_t first_cta_addr(uint32_t addr) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(addr));
    return r;
}
__device__ __forceinline__ void st_cluster(uint32_t addr, float v) {
    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory");
}
__device__ __forceinline__ float ldsf(uint32_t addr) { return __uint_as_float(lds32(addr)); }
__device__ __forceinline__ void stsf(uint32_t addr, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }

__device__ __forceinline__ float half_value(uint32_t w, int hi, bool bf16) {
    const uint16_t h = uint16_t(hi ? w >> 16 : w);
    return bf16 ? __uint_as_float(uint32_t(h) << 16) : __half2float(__ushort_as_half(h));
}
__device__ __forceinline__ uint32_t half_pair(float lo, float hi, bool bf16) {
    if (bf16) {
        const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
        return *reinterpret_cast<const uint32_t *>(&v);
    }
    return pack_f16x2(lo, hi);
}
// Dims c0 .. c0 + 7 of a head's row `x` rotated at table row `pos` (bd_rope.cu's arithmetic, rounded to the input type):
// pairs half a rotary_dim apart, rotary_dim below 128 (the other kinds: Trig).
__device__ __forceinline__ void rotate8(const DecodeParams &p, const uint16_t *x, int c0, int pos, bool bf16, uint32_t (&r)[4]) {
    if (c0 >= p.rotary_dim) return;
    const int half = p.rotary_dim / 2;
    auto value = [&](uint32_t w, int hi) { return half_value(w, hi, bf16); };
    auto pack = [&](float lo, float hi) { return half_pair(lo, hi, bf16); };
    const uint16_t *cs = static_cast<const uint16_t *>(p.cos_tab) + int64_t(pos) * half;
    const uint16_t *sn = static_cast<const uint16_t *>(p.sin_tab) + int64_t(pos) * half;
    const bool low = c0 < half;
    const int col = low ? c0 : c0 - half;
    uint32_t o[4], cw[4], sw[4];
    ldg128_pinned(x + (low ? c0 + half : c0 - half), o);
    ldg128_pinned(cs + col, cw);
    ldg128_pinned(sn + col, sw);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float y[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const float c = value(cw[i], k), s = value(sw[i], k), a = value(r[i], k), b = value(o[i], k);
            y[k] = low ? __fsub_rn(__fmul_rn(a, c), __fmul_rn(b, s)) : __fadd_rn(__fmul_rn(b, s), __fmul_rn(a, c));
        }
        r[i] = pack(y[0], y[1]);
    }
}

// The table's words that this thread (dims 32 a + 8 l .. + 7) needs, all requested together: cosines, then sines.
// (Each chunk's words behind the chunk before it cost a step of 8 sequences 1.9 us, of 2 2.2; together 1.0 and 0.8.)
struct Trig {
    uint32_t w[2][8];
    bool near, far;               // pairs (2i, 2i + 1); pairs 64 apart; neither: rotate8
    __device__ __forceinline__ void load(const DecodeParams &p, int pos, int l) {
        near = p.rotary_interleaved != 0;
        far = !near && p.rotary_dim == kHeadDim;
        const int64_t row = int64_t(pos) * (p.rotary_dim / 2);
        const uint16_t *tab[2] = {static_cast<const uint16_t *>(p.cos_tab) + row, static_cast<const uint16_t *>(p.sin_tab) + row};
        if (near) {
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    const int c0 = 32 * a + 8 * l;
                    const uint2 v = *reinterpret_cast<const uint2 *>(tab[t] + (c0 < p.rotary_dim ? c0 / 2 : 0));
                    w[t][2 * a] = v.x;
                    w[t][2 * a + 1] = v.y;
                }
        } else if (far) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int t = 0; t < 2; ++t) {
                    const uint4 v = *reinterpret_cast<const uint4 *>(tab[t] + 32 * i + 8 * l);
                    w[t][4 * i] = v.x; w[t][4 * i + 1] = v.y; w[t][4 * i + 2] = v.z; w[t][4 * i + 3] = v.w;
                }
        }
    }
    // r[a]: the thread's dims of row x
    __device__ __forceinline__ void rotate(const DecodeParams &p, const uint16_t *x, int pos, int l, bool bf16, uint32_t (&r)[4][4]) const {
        if (near) {
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                if (32 * a + 8 * l >= p.rotary_dim) continue;
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float c = half_value(w[0][2 * a + (i >> 1)], i & 1, bf16), s = half_value(w[1][2 * a + (i >> 1)], i & 1, bf16);
                    const float x0 = half_value(r[a][i], 0, bf16), x1 = half_value(r[a][i], 1, bf16);
                    r[a][i] = half_pair(__fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, s)), __fadd_rn(__fmul_rn(x0, s), __fmul_rn(x1, c)), bf16);
                }
            }
        } else if (far) {
#pragma unroll
            for (int a = 0; a < 2; ++a)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    float lo[2], hi[2];
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const float c = half_value(w[0][4 * a + i], k, bf16), s = half_value(w[1][4 * a + i], k, bf16);
                        const float x0 = half_value(r[a][i], k, bf16), x1 = half_value(r[a + 2][i], k, bf16);
                        lo[k] = __fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, s));
                        hi[k] = __fadd_rn(__fmul_rn(x0, s), __fmul_rn(x1, c));
                    }
                    r[a][i] = half_pair(lo[0], lo[1], bf16);
                    r[a + 2][i] = half_pair(hi[0], hi[1], bf16);
                }
        } else {
#pragma unroll
            for (int a = 0; a < 4; ++a) rotate8(p, x, 32 * a + 8 * l, pos, bf16, r[a]);
        }
    }
};

}  // namespace

template <int BITS, int GROUP, int NQT>
__global__ void __launch_bounds__(ShortCfg<BITS, GROUP, NQT>::THREADS, 1)
bd_decode_short_kernel(const DecodeParams p, const PackParams roll, const __grid_constant__ CUtensorMap kmap,
                       const __grid_constant__ CUtensorMap vmap) {
    using C = ShortCfg<BITS, GROUP, NQT>;
    constexpr int P = C::P, NB = C::NB, NGK = C::NGK, FPG = C::FPG, NGD = C::NGD, FPGV = C::FPGV, NZ = C::NZ;
    constexpr int DP = C::DP, RUNS = C::RUNS, PRM = C::PRM, STAGES = C::STAGES, WARPS = C::WARPS;
    constexpr bool PAIRS = kFieldPairs<BITS, GROUP>;

    extern __shared__ __align__(1024) uint8_t smem[];
    const uint32_t smem_base = smem_u32(smem);
    // Whether a wait of a warp ran out; written by that warp, read by the others behind the barrier that follows the loop.
    volatile int *gave_up = reinterpret_cast<volatile int *>(smem + C::OFF_FLAGS);
    const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0), lane = tid & 31;
    const int g = lane >> 2, l = lane & 3;
    // a cluster's CTAs are consecutive, and so are the heads of a sequence
    const int ncta = p.cluster, rank = blockIdx.x % ncta, pair = blockIdx.x / ncta;
    const int ih = pair % p.h_k, ib = pair / p.h_k;
    const uint32_t code = smem_base + warp * STAGES * 2 * C::CODE;                       // K tile, V tile of a stage
    const uint32_t prm = smem_base + C::OFF_PRM + warp * STAGES * 2 * PRM;               // and their scales and zeros
    const uint32_t bars = smem_base + C::OFF_BAR + warp * STAGES * 16;

    if ((smem_base & 1023u) != 0) {                      // never seen (the swizzled tiles need it); refuse rather than read garbage
        asm volatile("griddepcontrol.wait;" ::: "memory");
        if (tid == 0) atomicExch(p.status, BD_ERR_ALIGNMENT);
        return;
    }
    if (lane == 0) {
        for (int i = 0; i < 2 * STAGES; ++i) mbar_init(bars + 8 * i, 1);
        gave_up[warp] = 0;
        fence_mbar_init();
        tma_prefetch_desc(&kmap);
        tma_prefetch_desc(&vmap);
    }
    __syncwarp();
    if (ncta > 1) cluster_arrive();          // "this CTA runs": waited for before anything is stored into another one
    // Nothing that an earlier kernel may have written is read before this wait (the set-up so far ran beside its end).
    asm volatile("griddepcontrol.wait;" ::: "memory");

    const bool bf16 = p.dtype == BD_BF16;
    // Query rows as B fragments: thread (g, l) holds q[row g][32a + 8l .. +7], a = 0..3; requested first.
    uint32_t qr[NQT][4][4];
    const uint16_t *qrow[NQT];
#pragma unroll
    for (int nq = 0; nq < NQT; ++nq) {
        const int r = nq * 8 + g;
        qrow[nq] = static_cast<const uint16_t *>(p.q) + ib * p.q_stride_b + (int64_t(ih) * p.gq + (r < p.gq ? r : 0)) * p.q_stride_h;
#pragma unroll
        for (int a = 0; a < 4; ++a) ldg128_pinned(qrow[nq] + 32 * a + 8 * l, qr[nq][a]);
    }
    const int cached = p.cache_seqlens ? p.cache_seqlens[ib] : p.s;
    const int in_tail = p.res_lens ? p.res_lens[ib] : p.res_len;
    const int seqlen = min(max(cached, 0), p.s);
    int res_old = 0, res_n = 0;              // tail rows in the buffers, and with this step's token
    if (p.k_res != nullptr) {
        res_n = res_old = min(max(in_tail, 0), min(kTailMax, p.res_cap));
        if (p.k_new != nullptr && res_n < min(kTailMax, p.res_cap)) res_n += 1;
    }
    // The items of this warp: every (WARPS * ncta)-th, tail items first (their loads are exposed; the copies run meanwhile).
    const int items_tail = (res_n + 15) / 16, items = items_tail + 2 * ((seqlen + NB - 1) / NB);
    const int stride = WARPS * ncta, first = warp * ncta + rank;
    int unit0 = first;                       // first half block of this warp, counted from the tail's first item
    if (unit0 < items_tail) unit0 += (items_tail - unit0 + stride - 1) / stride * stride;

    auto resolve = [&](int &ix, int &blk) -> bool {      // paged cache: see bd_decode.cu
        if (p.block_table == nullptr) return true;
        const int pg = blk / p.blocks_per_page;
        blk -= pg * p.blocks_per_page;
        const int page = p.block_table[int64_t(ix) * p.block_table_stride + pg];
        const bool ok = page >= 0 && page < p.num_pages;
        ix = ok ? page : 0;
        return ok;
    };
    bool starve = p.test_starve != 0 && blockIdx.x == 0;     // test hook: the first K copy of every warp of CTA 0
    auto issue = [&](int item, int st) {
        const int u = (item - items_tail) & 1;
        int blk = (item - items_tail) >> 1, ix = ib;
        if (elect_one()) {
            const uint32_t kt = code + st * 2 * C::CODE, vt = kt + C::CODE, kp = prm + st * 2 * PRM, vp = kp + PRM;
            const uint32_t kbar = bars + 16 * st, vbar = kbar + 8;
            resolve(ix, blk);
            mbar_arrive_expect_tx(kbar, C::CODE + PRM + (starve ? 16 : 0));
            const int row0 = ix * p.k_batch_rows + blk * 32 + 16 * u;
            tma_load_2d(kt, &kmap, kbar, ih * kHeadDim, row0);
            tma_load_2d(kt + 2048, &kmap, kbar, ih * kHeadDim + 64, row0);
            const uint16_t *ks = p.k_params + ix * p.k_params_stride_b;
#pragma unroll
            for (int gk = 0; gk < NGK; ++gk)
                bulk_load_1d(kp + gk * 512, ks + ((int64_t(blk) * NGK + gk) * p.h_k + ih) * (2 * kHeadDim), 512, kbar);
            mbar_arrive_expect_tx(vbar, C::CODE + PRM);
            // tokens 16 u + 32 j .. + 15 of the block: the tokens of the half block's pack rows
#pragma unroll
            for (int j = 0; j < P; ++j)
                tma_load_2d(vt + j * (32 * DP), &vmap, vbar, ih * DP, ix * p.v_batch_rows + blk * NB + 16 * u + 32 * j);
            const uint16_t *vs = p.v_params + ix * p.v_params_stride_b + ih * p.v_params_stride_h;
#pragma unroll
            for (int gd = 0; gd < NGD; ++gd)
                bulk_load_1d(vp + gd * (RUNS * 512), vs + gd * p.v_params_stride_g + int64_t(blk) * RUNS * 256, RUNS * 512, vbar);
        }
        starve = false;
    };
#pragma unroll
    for (int st = 0; st < STAGES; ++st)
        if (unit0 + st * stride < items) issue(unit0 + st * stride, st);
    __syncwarp();

    int pos = max(cached, 0) + max(in_tail, 0);          // of this step's token
    if (p.rotary_dim > 0 && pos >= p.rotary_positions) {
        if (tid == 0 && rank == 0) atomicExch(p.status, BD_ERR_POSITION);
        pos = p.rotary_positions - 1;
    }
    Trig trig;
    if (p.rotary_dim > 0) {
        trig.load(p, pos, l);
#pragma unroll
        for (int nq = 0; nq < NQT; ++nq) trig.rotate(p, qrow[nq], pos, l, bf16, qr[nq]);
    }
#pragma unroll
    for (int nq = 0; nq < NQT; ++nq)
#pragma unroll
        for (int a = 0; a < 4; ++a) {
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                if (bf16) qr[nq][a][x] = bf16x2_to_f16x2(qr[nq][a][x]);
                if (nq * 8 + g >= p.gq) qr[nq][a][x] = 0;
            }
        }

    // thread-constant shared-memory offsets (see bd_decode.cu)
    const uint32_t k_row_off = g * 128;
    const uint32_t k_chunk_off[2] = {uint32_t((l ^ g) << 4), uint32_t(((4 + l) ^ g) << 4)};
    const int v_slot = (lane & 7) + 8 * ((lane >> 4) & 1), v_cpar = (lane >> 3) & 1;
    uint32_t v_off[2];
    if constexpr (BITS == 4) {
        v_off[0] = v_slot * 64 + (((0 + v_cpar) ^ ((v_slot >> 1) & 3)) << 4);
        v_off[1] = v_slot * 64 + (((2 + v_cpar) ^ ((v_slot >> 1) & 3)) << 4);
    } else {
        v_off[0] = v_slot * 32 + ((v_cpar ^ ((v_slot >> 2) & 1)) << 4);
        v_off[1] = 0;
    }

    float O[NQT][8][4], ZS[NQT][NZ][4], m_run[NQT][2], l_run[NQT][2];
#pragma unroll
    for (int nq = 0; nq < NQT; ++nq) {
#pragma unroll
        for (int mt = 0; mt < 8; ++mt)
#pragma unroll
            for (int e = 0; e < 4; ++e) O[nq][mt][e] = 0.f;
#pragma unroll
        for (int z = 0; z < NZ; ++z)
#pragma unroll
            for (int e = 0; e < 4; ++e) ZS[nq][z][e] = 0.f;
        m_run[nq][0] = m_run[nq][1] = -INFINITY;
        l_run[nq][0] = l_run[nq][1] = 0.f;
    }

    // ---- unquantized tail (fp16 / bf16 rows): 16 tokens an item (as in bd_decode.cu) ----
#pragma unroll 1
    for (int item = first; item < items_tail; item += stride) {
        const int tok0 = 16 * item, tA = tok0 + g, tB = tA + 8;
        const bool okA = tA < res_n, okB = tB < res_n;
        // rows past the end are read from the last valid row (in bounds) and zeroed afterwards
        const int rA = min(tA, res_n - 1), rB = min(tB, res_n - 1);
        const bool newA = rA >= res_old, newB = rB >= res_old;       // this step's token, from where it comes in
        const int64_t row_base = ib * p.res_stride_b + ih * p.res_stride_h, new_base = ib * p.new_stride_b + ih * p.new_stride_h;
        const uint16_t *kres = static_cast<const uint16_t *>(p.k_res) + row_base, *vres = static_cast<const uint16_t *>(p.v_res) + row_base;
        const uint16_t *knew = static_cast<const uint16_t *>(p.k_new) + new_base, *vnew = static_cast<const uint16_t *>(p.v_new) + new_base;
        const uint16_t *kA = newA ? knew : kres + int64_t(rA) * p.res_stride_s, *kB = newB ? knew : kres + int64_t(rB) * p.res_stride_s;
        const uint16_t *vA = newA ? vnew : vres + int64_t(rA) * p.res_stride_s, *vB = newB ? vnew : vres + int64_t(rB) * p.res_stride_s;
        uint32_t ka[4][4], kb[4][4];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            ldg128_pinned(kA + 32 * a + 8 * l, ka[a]);
            ldg128_pinned(kB + 32 * a + 8 * l, kb[a]);
        }
        uint32_t va[16], vb[16];     // word i: dims 8 i + 2 l, + 1 of the two token rows
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            va[i] = *reinterpret_cast<const unsigned int *>(vA + 8 * i + 2 * l);
            vb[i] = *reinterpret_cast<const unsigned int *>(vB + 8 * i + 2 * l);
        }
        if (p.rotary_dim > 0 && (newA || newB)) {
            if (newA) trig.rotate(p, knew, pos, l, bf16, ka);
            if (newB) trig.rotate(p, knew, pos, l, bf16, kb);
        }
        // fused append: the four threads that hold this step's token also store it into its row of the tail buffers
        if (res_n > res_old && (tA == res_old || tB == res_old)) {
            const int64_t dst = row_base + int64_t(res_old) * p.res_stride_s;
            uint16_t *ko = static_cast<uint16_t *>(p.k_res_out) + dst, *vo = static_cast<uint16_t *>(p.v_res_out) + dst;
            const bool a_row = tA == res_old;
#pragma unroll
            for (int a = 0; a < 4; ++a)
                *reinterpret_cast<uint4 *>(ko + 32 * a + 8 * l) = a_row ? make_uint4(ka[a][0], ka[a][1], ka[a][2], ka[a][3])
                                                                        : make_uint4(kb[a][0], kb[a][1], kb[a][2], kb[a][3]);
#pragma unroll
            for (int i = 0; i < 16; ++i) *reinterpret_cast<uint32_t *>(vo + 8 * i + 2 * l) = a_row ? va[i] : vb[i];
        }
        if (bf16) {
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int x = 0; x < 4; ++x) { ka[a][x] = bf16x2_to_f16x2(ka[a][x]); kb[a][x] = bf16x2_to_f16x2(kb[a][x]); }
#pragma unroll
            for (int i = 0; i < 16; ++i) { va[i] = bf16x2_to_f16x2(va[i]); vb[i] = bf16x2_to_f16x2(vb[i]); }
        }
        uint32_t pb[NQT][2];
#pragma unroll
        for (int nq = 0; nq < NQT; ++nq) {
            float S[1][4] = {{0.f, 0.f, 0.f, 0.f}};
#pragma unroll
            for (int a = 0; a < 4; ++a) {
                mma_f16(S[0], ka[a][0], kb[a][0], ka[a][1], kb[a][1], qr[nq][a][0], qr[nq][a][1]);
                mma_f16(S[0], ka[a][2], kb[a][2], ka[a][3], kb[a][3], qr[nq][a][2], qr[nq][a][3]);
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float mu = m_run[nq][e & 1] == -INFINITY ? 0.f : m_run[nq][e & 1];
                S[0][e] = ((e < 2) ? okA : okB) ? fmaf(S[0][e], p.scale_log2, -mu) : -INFINITY;
            }
            float f[2];
            softmax_step<1, true, NZ>(S, m_run[nq], l_run[nq], O[nq], ZS[nq], f);
            pb[nq][0] = movmatrix_trans(pack_f16x2(S[0][0], S[0][1]));
            pb[nq][1] = movmatrix_trans(pack_f16x2(S[0][2], S[0][3]));
        }
#pragma unroll
        for (int mt = 0; mt < 8; ++mt) {
            const int jv = (BITS == 4) ? (mt & 3) : mt;
            // rows 0-7 of this m-tile are dims d0 .. d0+7, rows 8-15 are d0+8 .. d0+15
            const int i0 = (((BITS == 4) ? 16 * (mt >> 2) : 0) + DP * jv) / 8;
            const uint32_t a0 = movmatrix_trans(okA ? va[i0] : 0u), a1 = movmatrix_trans(okA ? va[i0 + 1] : 0u);
            const uint32_t a2 = movmatrix_trans(okB ? vb[i0] : 0u), a3 = movmatrix_trans(okB ? vb[i0 + 1] : 0u);
            const float fw = field_weight<BITS>(jv);   // O is kept in the units of its packed field
#pragma unroll
            for (int nq = 0; nq < NQT; ++nq) {
                float ot[4] = {0.f, 0.f, 0.f, 0.f};
                mma_f16(ot, a0, a1, a2, a3, pb[nq][0], pb[nq][1]);
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    O[nq][mt][e] = fmaf(ot[e], fw, O[nq][mt][e]);
                    if (PAIRS && (mt & 1)) O[nq][mt - 1][e] = fmaf(ot[e], fw, O[nq][mt - 1][e]);   // a pair's sum
                }
            }
        }
    }

    // Whether a copy has come is one answer for the warp: its lanes poll for themselves and could disagree on the last poll of
    // a wait that runs out, and what follows (MMAs, shuffles, an elected lane) needs them together.  (A vote per wait: 1 x 4096
    // tokens 6.47 -> 6.49 us, 8 x 2048 ragged 9.81 -> 9.79.)
    auto copied = [&](uint32_t bar, uint32_t parity) { return __all_sync(0xffffffffu, mbar_wait_bounded(bar, parity, p.spin_limit)); };

    // ---- half blocks ----
    int n = 0;
#pragma unroll 1
    for (int item = unit0; item < items; item += stride, ++n) {
        const int st = STAGES == 2 ? n & 1 : 0;
        const uint32_t par = (STAGES == 2 ? n >> 1 : n) & 1;
        const int u = (item - items_tail) & 1, blk = (item - items_tail) >> 1;
        const uint32_t kt = code + st * 2 * C::CODE, vt = kt + C::CODE, kp = prm + st * 2 * PRM, vp = kp + PRM;
        int seqlen_blk = seqlen;
        if (p.block_table != nullptr) {
            int ix = ib, pblk = blk;
            if (!resolve(ix, pblk)) {            // page index outside the pool: the whole block is masked
                seqlen_blk = 0;
                if (lane == 0) atomicExch(p.status, BD_ERR_PAGE);
            }
        }
        const bool need_mask = (blk + 1) * NB > seqlen_blk;
        if (!copied(bars + 16 * st, par)) { gave_up[warp] = 1; break; }

        // q . zero per token group, two groups at a time: rows 0-7 the one, rows 8-15 the other
        float Zc[NGK][NQT][2];
        {
            constexpr int NZP = (NGK + 1) / 2;
            float Z[NZP][NQT][4];
#pragma unroll
            for (int zp = 0; zp < NZP; ++zp)
#pragma unroll
                for (int nq = 0; nq < NQT; ++nq)
#pragma unroll
                    for (int e = 0; e < 4; ++e) Z[zp][nq][e] = 0.f;
#pragma unroll
            for (int zp = 0; zp < NZP; ++zp)
#pragma unroll
                for (int a = 0; a < 4; ++a) {
                    uint32_t z[4], y[4];
                    lds128(kp + kprm_off<BITS, GROUP>(2 * zp, a, l) + 256, z[0], z[1], z[2], z[3]);
#pragma unroll
                    for (int x = 0; x < 4; ++x) y[x] = z[x];
                    if constexpr (NGK > 1) lds128(kp + kprm_off<BITS, GROUP>(2 * zp + 1, a, l) + 256, y[0], y[1], y[2], y[3]);
#pragma unroll
                    for (int nq = 0; nq < NQT; ++nq) {
                        mma_f16(Z[zp][nq], z[0], y[0], z[1], y[1], qr[nq][a][0], qr[nq][a][1]);
                        mma_f16(Z[zp][nq], z[2], y[2], z[3], y[3], qr[nq][a][2], qr[nq][a][3]);
                    }
                }
#pragma unroll
            for (int gk = 0; gk < NGK; ++gk)
#pragma unroll
                for (int nq = 0; nq < NQT; ++nq) {
                    Zc[gk][nq][0] = Z[gk / 2][nq][2 * (gk & 1)] * p.scale_log2;
                    Zc[gk][nq][1] = Z[gk / 2][nq][2 * (gk & 1) + 1] * p.scale_log2;
                }
        }
        float S[P][NQT][4];
#pragma unroll
        for (int j = 0; j < P; ++j)
#pragma unroll
            for (int nq = 0; nq < NQT; ++nq)
#pragma unroll
                for (int e = 0; e < 4; ++e) S[j][nq][e] = 0.f;
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            // q * scale for the token groups of this block, channels 32a + 8l .. +7
            uint32_t qs[NGK][NQT][4];
#pragma unroll
            for (int gk = 0; gk < NGK; ++gk) {
                uint32_t s[4];
                lds128(kp + kprm_off<BITS, GROUP>(gk, a, l), s[0], s[1], s[2], s[3]);
#pragma unroll
                for (int nq = 0; nq < NQT; ++nq)
#pragma unroll
                    for (int x = 0; x < 4; ++x) qs[gk][nq][x] = hmul2_u32(qr[nq][a][x], s[x]);
            }
            uint32_t wl[4], wh[4];
            const uint32_t at = kt + (a >> 1) * 2048 + k_row_off + k_chunk_off[a & 1];
            lds128(at, wl[0], wl[1], wl[2], wl[3]);
            lds128(at + 1024, wh[0], wh[1], wh[2], wh[3]);
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const uint32_t w0 = wl[2 * half], w1 = wh[2 * half], w2 = wl[2 * half + 1], w3 = wh[2 * half + 1];
                const uint32_t s0 = aux_word<BITS>(w0), s1 = aux_word<BITS>(w1), s2 = aux_word<BITS>(w2), s3 = aux_word<BITS>(w3);
                auto do_kfield = [&](auto jc) {
                    constexpr int J = decltype(jc)::value;
#pragma unroll
                    for (int nq = 0; nq < NQT; ++nq)
                        mma_f16(S[J][nq], field<BITS, J, PAIRS>(w0, s0), field<BITS, J, PAIRS>(w1, s1), field<BITS, J, PAIRS>(w2, s2),
                                field<BITS, J, PAIRS>(w3, s3), qs[J / FPG][nq][2 * half], qs[J / FPG][nq][2 * half + 1]);
                };
                do_kfield(std::integral_constant<int, 0>{});
                do_kfield(std::integral_constant<int, 1>{});
                do_kfield(std::integral_constant<int, 2>{});
                do_kfield(std::integral_constant<int, 3>{});
                if constexpr (P == 8) {
                    do_kfield(std::integral_constant<int, 4>{});
                    do_kfield(std::integral_constant<int, 5>{});
                    do_kfield(std::integral_constant<int, 6>{});
                    do_kfield(std::integral_constant<int, 7>{});
                }
            }
        }
        uint32_t Pb[P][NQT][2];
#pragma unroll
        for (int nq = 0; nq < NQT; ++nq) {
            float t[P][4], zm[NGK][2];
#pragma unroll
            for (int gk = 0; gk < NGK; ++gk)
#pragma unroll
                for (int c = 0; c < 2; ++c) zm[gk][c] = Zc[gk][nq][c] - (m_run[nq][c] == -INFINITY ? 0.f : m_run[nq][c]);
#pragma unroll
            for (int j = 0; j < P; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float sv = S[j][nq][e];
                    if (PAIRS && (j & 1) == 0) sv -= S[j + (PAIRS ? 1 : 0)][nq][e];        // pair sum minus the odd field
                    t[j][e] = fmaf(sv, p.scale_log2 * (1.0f / field_weight<BITS>(j)), zm[j / FPG][e & 1]);
                    if (need_mask && blk * NB + 16 * u + 32 * j + g + 8 * (e >> 1) >= seqlen_blk) t[j][e] = -INFINITY;
                }
            float f[2];
            softmax_step<P, (NGD > 1), NZ>(t, m_run[nq], l_run[nq], O[nq], ZS[nq], f);
#pragma unroll
            for (int j = 0; j < P; ++j) {
                Pb[j][nq][0] = movmatrix_trans(pack_f16x2(t[j][0], t[j][1]));
                Pb[j][nq][1] = movmatrix_trans(pack_f16x2(t[j][2], t[j][3]));
            }
        }
        if (!copied(bars + 16 * st + 8, par)) { gave_up[warp] = 1; break; }
#pragma unroll
        for (int j = 0; j < P; ++j) {
            const int r0 = 16 * u + 32 * j + 2 * l;               // tokens of fragment register 0
            uint32_t sc0[NGD], sc1[NGD], ze0[NGD], ze1[NGD];      // tokens r0, r0+1 and r0+8, r0+9 (same run)
#pragma unroll
            for (int gd = 0; gd < NGD; ++gd) {
                const uint32_t b0 = vp + vprm_off<BITS, GROUP>(gd, r0, 0), b1 = vp + vprm_off<BITS, GROUP>(gd, r0, 1);
                sc0[gd] = lds32(b0);
                sc1[gd] = lds32(b1);
                ze0[gd] = lds32(b0 + 256);
                ze1[gd] = lds32(b1 + 256);
            }
            if (need_mask) {          // params of tokens past the end may be uninitialised
                const int tok = blk * NB + r0;
                const uint32_t k0 = (tok < seqlen_blk ? 0x0000ffffu : 0u) | (tok + 1 < seqlen_blk ? 0xffff0000u : 0u);
                const uint32_t k1 = (tok + 8 < seqlen_blk ? 0x0000ffffu : 0u) | (tok + 9 < seqlen_blk ? 0xffff0000u : 0u);
#pragma unroll
                for (int gd = 0; gd < NGD; ++gd) { sc0[gd] &= k0; ze0[gd] &= k0; sc1[gd] &= k1; ze1[gd] &= k1; }
            }
            uint32_t pv[NGD][NQT][2];
#pragma unroll
            for (int nq = 0; nq < NQT; ++nq) {
                // rows 0-7: sum_t p_t * zero_t of dim group 0; rows 8-15: of dim group 1 or, with a single one, sum_t p_t
                constexpr uint32_t kOnes = 0x3c003c00u;
#pragma unroll
                for (int z = 0; z < NZ; ++z)
                    mma_f16(ZS[nq][z], ze0[2 * z], NGD > 1 ? ze0[NGD > 1 ? 2 * z + 1 : 0] : kOnes, ze1[2 * z],
                            NGD > 1 ? ze1[NGD > 1 ? 2 * z + 1 : 0] : kOnes, Pb[j][nq][0], Pb[j][nq][1]);
#pragma unroll
                for (int gd = 0; gd < NGD; ++gd) {
                    pv[gd][nq][0] = hmul2_u32(Pb[j][nq][0], sc0[gd]);
                    pv[gd][nq][1] = hmul2_u32(Pb[j][nq][1], sc1[gd]);
                }
            }
            constexpr int NCB = (BITS == 4) ? 2 : 1;              // ldmatrix.x4 per slice of 16 tokens
#pragma unroll
            for (int cb = 0; cb < NCB; ++cb) {
                uint32_t w0, w1, w2, w3;
                ldsm_x4_trans(vt + j * (32 * DP) + v_off[cb], w0, w1, w2, w3);
                const uint32_t s0 = aux_word<BITS>(w0), s1 = aux_word<BITS>(w1), s2 = aux_word<BITS>(w2), s3 = aux_word<BITS>(w3);
                auto do_vfield = [&](auto jc) {
                    constexpr int JV = decltype(jc)::value;
                    const int mt = (BITS == 4) ? (cb * 4 + JV) : JV;
#pragma unroll
                    for (int nq = 0; nq < NQT; ++nq)
                        mma_f16(O[nq][mt], field<BITS, JV, PAIRS>(w0, s0), field<BITS, JV, PAIRS>(w1, s1), field<BITS, JV, PAIRS>(w2, s2),
                                field<BITS, JV, PAIRS>(w3, s3), pv[JV / FPGV][nq][0], pv[JV / FPGV][nq][1]);
                };
                do_vfield(std::integral_constant<int, 0>{});
                do_vfield(std::integral_constant<int, 1>{});
                do_vfield(std::integral_constant<int, 2>{});
                do_vfield(std::integral_constant<int, 3>{});
                if constexpr (P == 8) {
                    do_vfield(std::integral_constant<int, 4>{});
                    do_vfield(std::integral_constant<int, 5>{});
                    do_vfield(std::integral_constant<int, 6>{});
                    do_vfield(std::integral_constant<int, 7>{});
                }
            }
        }
        __syncwarp();
        if (item + STAGES * stride < items) {
            fence_proxy_async();
            issue(item + STAGES * stride, st);
            __syncwarp();
        }
    }
    // The kernel behind this one may be placed from here on (it waits for this grid before it reads anything).
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");

    // ---- this warp's result: O in final units (field weights and zero sums applied), then m, l ----
    const uint32_t mine = code;              // into its own tiles (nothing is in flight there unless the wait ran out: see the exit)
#pragma unroll
    for (int nq = 0; nq < NQT; ++nq) {
#pragma unroll
        for (int mt = 0; mt < 8; ++mt) {
            const int jv = (BITS == 4) ? (mt & 3) : mt;
            const int gd = jv / FPGV;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float ov = O[nq][mt][e];
                if (PAIRS && (mt & 1) == 0) ov -= O[nq][mt + (PAIRS ? 1 : 0)][e];      // pair sum minus the odd field
                stsf(mine + ((nq * 32 + mt * 4 + e) * 32 + lane) * 4,
                     fmaf(ov, 1.0f / field_weight<BITS>(jv), ZS[nq][gd >> 1][2 * (gd & 1) + (e & 1)]));
            }
        }
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            float sum = l_run[nq][c];
            sum += __shfl_xor_sync(0xffffffffu, sum, 4);
            sum += __shfl_xor_sync(0xffffffffu, sum, 8);
            sum += __shfl_xor_sync(0xffffffffu, sum, 16);
            if (NGD == 1) sum += ZS[nq][0][2 + c];      // every row of the ones block holds the column sum
            stsf(mine + ((32 * NQT + nq * 4 + c) * 32 + lane) * 4, m_run[nq][c]);
            stsf(mine + ((32 * NQT + nq * 4 + 2 + c) * 32 + lane) * 4, sum);
        }
    }
    __syncthreads();
    // The lengths move on when every CTA that works on the sequence has read them: each counts in, behind the barrier that
    // all of its warps have met at (a count per warp, each behind its own reads: a step of 8 sequences 11.05 -> 10.4 us, of 2
    // 13.1 -> 12.3), and the last one writes them where the others wait anyway.
    int arrived = -1;
    if (roll.roll_res_lens != nullptr && tid == C::THREADS - 32) {
        __threadfence();
        arrived = atomicAdd(roll.roll_arrivals + int64_t(ib) * p.h_k, 1);
    }
    // (the rule of bd_pack.cu's roll-over, for the lengths and for the block)
    auto room_for_block = [&]() { return cached >= 0 && cached % NB == 0 && cached <= roll.roll_s_cap - NB; };
    auto tail_behind_step = [&]() {
        const int r = min(max(in_tail, 0), roll.roll_res_cap);
        return r < roll.roll_res_cap ? r + 1 : r;
    };
    auto move_on = [&]() {
        if (arrived == p.h_k * ncta - 1) {
            const bool room = room_for_block();
            const int left = tail_behind_step();
            __threadfence();
            roll.roll_arrivals[int64_t(ib) * p.h_k] = 0;
            if (left == NB && room) roll.roll_cache_seqlens[ib] = cached + NB;
            if (left == NB && !room) atomicExch(roll.roll_status, BD_ERR_CAPACITY);
            roll.roll_res_lens[ib] = left == NB && room ? 0 : left;
        }
        __syncwarp();
    };

    // ---- merge: every warp sums EPW = 4 NQT values per thread of all results, in their order ----
    constexpr int EPW = 32 * NQT / WARPS;
    const int e0 = warp * EPW, mq = e0 / 32;             // first value, and the query tile it belongs to
    float o[EPW], M[2], L[2];
    auto merge = [&](uint32_t at, uint32_t step, int count) {
#pragma unroll
        for (int i = 0; i < EPW; ++i) o[i] = 0.f;
        M[0] = M[1] = -INFINITY;
        L[0] = L[1] = 0.f;
        float mm[8][2], ll[8][2];
#pragma unroll
        for (int d = 0; d < 8; ++d) {
            if (d >= count) continue;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                mm[d][c] = ldsf(at + d * step + ((32 * NQT + mq * 4 + c) * 32 + lane) * 4);
                ll[d][c] = ldsf(at + d * step + ((32 * NQT + mq * 4 + 2 + c) * 32 + lane) * 4);
                M[c] = fmaxf(M[c], mm[d][c]);
            }
        }
#pragma unroll
        for (int d = 0; d < 8; ++d) {
            if (d >= count) continue;
            float f[2];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                f[c] = mm[d][c] == -INFINITY ? 0.f : ex2f(mm[d][c] - M[c]);
                L[c] = fmaf(f[c], ll[d][c], L[c]);
            }
#pragma unroll
            for (int i = 0; i < EPW; ++i) o[i] = fmaf(f[i & 1], ldsf(at + d * step + ((e0 + i) * 32 + lane) * 4), o[i]);
        }
    };
    static_assert(WARPS <= 8 && C::CLUSTER <= 8 && EPW % 2 == 0, "eight results at most");
    merge(smem_base, STAGES * 2 * C::CODE, WARPS);
    if (ncta > 1) {
        // the CTA's result, laid out like a warp's, goes to the first CTA of the cluster, which merges them the same way
        cluster_wait();
        const uint32_t to = first_cta_addr(smem_base + C::OFF_MERGE + rank * C::DEPOSIT);
#pragma unroll
        for (int i = 0; i < EPW; ++i) st_cluster(to + ((e0 + i) * 32 + lane) * 4, o[i]);
        if (e0 % 32 == 0) {
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                st_cluster(to + ((32 * NQT + mq * 4 + c) * 32 + lane) * 4, M[c]);
                st_cluster(to + ((32 * NQT + mq * 4 + 2 + c) * 32 + lane) * 4, L[c]);
            }
        }
        cluster_arrive();
        move_on();
        cluster_wait();
        if (rank == 0) merge(smem_base + C::OFF_MERGE, C::DEPOSIT, ncta);
    }
    if (rank == 0) {
        const int64_t hq0 = int64_t(ih) * p.gq;
        float inv[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            inv[c] = L[c] > 0.f ? __fdividef(1.0f, L[c]) : 0.f;
            const int r = mq * 8 + 2 * l + c;
            if (p.lse && e0 % 32 == 0 && g == 0 && r < p.gq)
                p.lse[int64_t(ib) * p.h + hq0 + r] = L[c] > 0.f ? fmaf(M[c], 0.6931471805599453f, __logf(L[c])) : -INFINITY;
        }
#pragma unroll
        for (int i = 0; i < EPW; ++i) {
            // value (mt, e): query row 8 mq + 2 l + (e & 1), dims as in bd_decode.cu
            const int mt = (e0 % 32 + i) >> 2, e = (e0 + i) & 3, r = mq * 8 + 2 * l + (e & 1);
            if (r >= p.gq) continue;
            const int jv = (BITS == 4) ? (mt & 3) : mt;
            const int dim = ((BITS == 4) ? 16 * (mt >> 2) : 0) + 8 * (e >> 1) + DP * jv + g;
            const int64_t oi = ib * p.out_stride_b + (hq0 + r) * p.out_stride_h + dim;
            const float v = o[i] * inv[e & 1];
            if (p.out_dtype == BD_FP16) static_cast<__half *>(p.out)[oi] = __float2half_rn(v);
            else if (p.out_dtype == BD_BF16) static_cast<__nv_bfloat16 *>(p.out)[oi] = __float2bfloat16_rn(v);
            else static_cast<float *>(p.out)[oi] = v;
        }
    }
    int aborted = 0;
#pragma unroll
    for (int w = 0; w < WARPS; ++w) aborted |= gave_up[w];
    if (aborted != 0) {
        if (tid == 0) atomicExch(p.status, BD_ERR_TIMEOUT);
        // give copies that are still in flight time to land before a full tail is packed through the tiles, and before the
        // block's shared memory is released
        for (int it = 0; it < 2000; ++it) __nanosleep(1000);
        __syncthreads();
    }
    if (roll.roll_res_lens != nullptr) {
        if (ncta == 1) move_on();
        if (tail_behind_step() == NB && room_for_block()) {
            // (the token's own row, stored by one of the cluster's warps, is visible behind the barriers above)
            static_assert(PackCfg<BITS, GROUP>::NTHREADS == 128 && WARPS == 8, "two groups of threads pack");
            static_assert(sizeof(typename PackCfg<BITS, GROUP>::Shared) <= 16384 && C::OFF_PRM >= 32768, "in the warps' tiles");
            constexpr int SPLIT = PackCfg<BITS, GROUP>::SPLIT;
            const int group = warp >> 2, t = tid & 127;
            auto &sh = *reinterpret_cast<typename PackCfg<BITS, GROUP>::Shared *>(smem + group * 16384);
            auto sync = [&] { asm volatile("barrier.cta.sync %0, 128;" ::"r"(1 + group) : "memory"); };
            __syncthreads();
#pragma unroll 1
            for (int part = 2 * rank + group; part < 2 * SPLIT; part += 2 * ncta) {
                if (part < SPLIT) {
                    if (bf16) pack_k_part<BITS, GROUP, true>(roll, sh, t, ib, ih, part, 0, cached / NB, sync);
                    else pack_k_part<BITS, GROUP, false>(roll, sh, t, ib, ih, part, 0, cached / NB, sync);
                } else {
                    if (bf16) pack_v_part<BITS, GROUP, true>(roll, sh, t, ib, ih, part - SPLIT, 0, cached / NB, sync);
                    else pack_v_part<BITS, GROUP, false>(roll, sh, t, ib, ih, part - SPLIT, 0, cached / NB, sync);
                }
                sync();
            }
        }
    }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// The launch of a step, but for grid and stream; `at` holds the attributes.
template <int BITS, int GROUP, int NQT>
static cudaError_t short_config(int cluster, cudaLaunchConfig_t &cfg, cudaLaunchAttribute (&at)[2]) {
    using C = ShortCfg<BITS, GROUP, NQT>;
    static bool configured[64] = {};
    int dev = 0;
    cudaError_t err = cudaGetDevice(&dev);
    if (err != cudaSuccess) return err;
    if (dev >= 64 || !configured[dev]) {
        err = cudaFuncSetAttribute(bd_decode_short_kernel<BITS, GROUP, NQT>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(C::SMEM));
        if (err != cudaSuccess) return err;
        if (dev < 64) configured[dev] = true;
    }
    cfg = {};
    cfg.blockDim = dim3(C::THREADS);
    cfg.dynamicSmemBytes = C::SMEM;
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    at[1].id = cudaLaunchAttributeClusterDimension;
    at[1].val.clusterDim.x = unsigned(cluster);
    at[1].val.clusterDim.y = 1;
    at[1].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = cluster > 1 ? 2 : 1;
    return cudaSuccess;
}

template <int BITS, int GROUP, int NQT>
static cudaError_t launch_short(const DecodeParams &p, const PackParams &roll, const CUtensorMap &kmap, const CUtensorMap &vmap, cudaStream_t stream) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[2];
    cudaError_t err = short_config<BITS, GROUP, NQT>(p.cluster, cfg, at);
    if (err != cudaSuccess) return err;
    cfg.gridDim = dim3(unsigned(p.b) * unsigned(p.h_k) * unsigned(p.cluster));
    cfg.stream = stream;
    return cudaLaunchKernelEx(&cfg, bd_decode_short_kernel<BITS, GROUP, NQT>, p, roll, kmap, vmap);
}

// Clusters of a size that run at once: a cluster's CTAs take an SM each, all in one GPC, and the SMs that a GPC has beyond a
// multiple of the size stay without one.  Asked once per device.
template <int BITS, int GROUP, int NQT>
static int resident_short(int cluster, int dev) {
    static std::atomic<int> known[64][4] = {};           // one more than the answer for clusters of 1, 2, 4 and 8
    if (dev < 0 || dev >= 64) return 0;
    std::atomic<int> &slot = known[dev][cluster == 8 ? 3 : cluster / 2];
    if (slot > 0) return slot - 1;
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute at[2];
    int n = 0;
    cudaError_t err = short_config<BITS, GROUP, NQT>(cluster, cfg, at);
    cfg.gridDim = dim3(unsigned(cluster));
    if (err == cudaSuccess) err = cudaOccupancyMaxActiveClusters(&n, bd_decode_short_kernel<BITS, GROUP, NQT>, &cfg);
    if (err != cudaSuccess) {
        (void)cudaGetLastError();
        return 0;
    }
    slot = n + 1;
    return n;
}

#define BD_SHORT_PICK(RESULT)                                                                           \
    const bool one = gq <= 8;                                                                           \
    if (bits == 4 && group == 128) { if (one) RESULT(4, 128, 1) else RESULT(4, 128, 2) }                \
    if (bits == 4 && group == 64) { if (one) RESULT(4, 64, 1) else RESULT(4, 64, 2) }                   \
    if (bits == 4 && group == 32) { if (one) RESULT(4, 32, 1) else RESULT(4, 32, 2) }                   \
    if (bits == 2 && group == 128) { if (one) RESULT(2, 128, 1) else RESULT(2, 128, 2) }                \
    if (bits == 2 && group == 64) { if (one) RESULT(2, 64, 1) else RESULT(2, 64, 2) }                   \
    if (bits == 2 && group == 32 && one) RESULT(2, 32, 1)      /* two query tiles: a result does not fit the one stage there is */

cudaError_t launch_decode_short(const DecodeParams &p, const PackParams &roll, const CUtensorMap &kmap, const CUtensorMap &vmap,
                                int bits, int group, cudaStream_t stream) {
    const int gq = p.gq;
#define BD_SHORT_LAUNCH(B, G, Q) return launch_short<B, G, Q>(p, roll, kmap, vmap, stream);
    BD_SHORT_PICK(BD_SHORT_LAUNCH)
    return cudaErrorInvalidValue;
}

int decode_short_cluster(int bits, int group, int gq) {
#define BD_SHORT_CLUSTER(B, G, Q) return ShortCfg<B, G, Q>::CLUSTER;
    BD_SHORT_PICK(BD_SHORT_CLUSTER)
    return 0;
}

int decode_short_resident(int bits, int group, int gq, int cluster, int dev) {
#define BD_SHORT_RESIDENT(B, G, Q) return resident_short<B, G, Q>(cluster, dev);
    BD_SHORT_PICK(BD_SHORT_RESIDENT)
    return 0;
}

}  // namespace bd
