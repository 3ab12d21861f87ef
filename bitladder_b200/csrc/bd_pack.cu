// Quantize-pack kernel: K per channel (groups of G consecutive tokens), V per
// token (groups of G consecutive dims), asymmetric min-max to 4 or 2 bits.
//
// Arithmetic follows the reference quantizer step by step in IEEE fp32
// (reference: csrc/bit_decode/src/include/qpack.h:241-252 for range, scale_inv,
// stored scale and zero; :266-281 for subtract, multiply, roundf, clamp; :283-294
// for the field order inside a word).  Explicit round-to-nearest intrinsics keep
// the result independent of compiler flags, so codes, scales and zeros are
// bit-identical to a CPU evaluation of the same formulas, and to what the reference's kernel
// writes when it is built without --use_fast_math (4-bit, group 128 and 32).  PackParams::approx_div
// selects the division of the reference as shipped instead (see scale_from_minmax).
//
// The work is pure streaming (read 2*NB*d*2 bytes of a pack block, NB = 32 * 16/bits tokens of one KV head,
// write a quarter or an eighth of that): every thread keeps 32 words of input in flight, rows are read and
// written in segments of at least 64 bytes per row, and nothing is re-read.
#include "bd_pack.cuh"

namespace bd {

constexpr int kPackResident = 1024;                                         // threads per SM
template <int BITS, int GROUP, bool BF16>
__global__ void __launch_bounds__(kPackThreads<BITS>, kPackResident / kPackThreads<BITS>)
bd_pack_kernel(const PackParams p) {
    using C = PackCfg<BITS, GROUP>;
    constexpr int NB = C::NB, SPLIT = C::SPLIT, NTHREADS = C::NTHREADS;
    __shared__ typename C::Shared sh;

    const int tid = threadIdx.x;
    // heads vary fastest: CTAs that run together read neighbouring 256-byte pieces of the same token rows
    const int blk = blockIdx.y, ib = blockIdx.z;
    int dst_off = p.dst_token_offset;
    // Staged early behind the kernel in front; nothing in global memory is read or written before that one is done, and
    // what it may write is never read through the non-coherent path (__ldg), which promises constant memory.
    asm volatile("griddepcontrol.wait;" ::: "memory");
    if (p.roll_res_lens != nullptr) {          // roll-over: only sequences whose tail this step's token filled
        // The next step's kernel may be placed beside this short one; it waits for it before it reads anything.  Few sequences
        // gain in a graph (1 x 32768 tokens, group 64 25.4 -> 24.8 us a step, 8 x 8192 at 2 bits 26.0 -> 25.5) and lose nothing
        // in a stream; many short ones lose (16 of up to 2560 tokens, most of 128, stream 18.0 -> 18.9 us, graph 17.3 -> 17.5).
        if (p.b <= 8) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        // The lengths move only when all CTAs of the sequence have read them (the decode kernel in front is done with
        // them); a kernel of its own for that cost 0.4 us more per decoder step, and its launch.  One thread reads them
        // for its CTA, so that the fence in front of its count orders the CTA's only reads before the last one's writes.
        __shared__ int32_t roll[2];
        if (tid == 0) {
            roll[0] = p.roll_res_lens[ib];
            roll[1] = p.roll_cache_seqlens[ib];
        }
        __syncthreads();
        dst_off = roll[1];
        // The tail as this step leaves it: the decode kernel filed a token where there was room.  One rule for the block
        // and for the lengths: a tail of one pack block, full from the start or filled now, is packed if there is room.
        int left = min(max(roll[0], 0), p.roll_res_cap);
        if (left < p.roll_res_cap) left += 1;
        const bool room = dst_off >= 0 && dst_off % NB == 0 && dst_off <= p.roll_s_cap - NB;
        if (tid == 0) {
            int32_t *arrivals = p.roll_arrivals + static_cast<int64_t>(ib) * p.h_k;
            __threadfence();
            if (atomicAdd(arrivals, 1) == int(gridDim.x) - 1) {
                __threadfence();
                *arrivals = 0;
                if (left == NB && room) p.roll_cache_seqlens[ib] = dst_off + NB;
                if (left == NB && !room) atomicExch(p.roll_status, BD_ERR_CAPACITY);
                p.roll_res_lens[ib] = left == NB && room ? 0 : left;
            }
        }
        if (left != NB || !room) return;
    }
    if (p.fill_cache_seqlens != nullptr) {
        const int full = min(max(p.fill_cache_seqlens[ib], 0), min(p.s, p.fill_s_cap)) / NB;
        if (blk >= full) {
            // behind the whole blocks: one block's worth of rows to the tail, 16 bytes a thread, the K CTAs and the V CTAs
            // of a head a share of the rows each
            const int rest = blk > full ? 0 : min(min(p.fill_res_lens[ib], NB), p.s - blk * NB);
            const bool is_k = blockIdx.x < SPLIT * p.h_k;
            const int x = is_k ? blockIdx.x : blockIdx.x - SPLIT * p.h_k;
            const int ih = x / SPLIT, part = x % SPLIT, c = 8 * (tid & 15);
            const uint16_t *src = is_k ? kin_of(p) + ib * p.k_stride_b + ih * p.k_stride_h : vin_of(p) + ib * p.v_stride_b + ih * p.v_stride_h;
            const int64_t step = is_k ? p.k_stride_s : p.v_stride_s;
            uint16_t *dst = static_cast<uint16_t *>(is_k ? p.k_tail : p.v_tail) + ib * p.tail_stride_b + ih * p.tail_stride_h;
            constexpr int ROWS = NTHREADS / 16, STEPS = NB / SPLIT / ROWS;      // rows at a time
            const int t0 = part * (NB / SPLIT) + (tid >> 4);
            uint4 row[STEPS];
#pragma unroll
            for (int i = 0; i < STEPS; ++i)
                if (t0 + i * ROWS < rest) row[i] = *reinterpret_cast<const uint4 *>(src + (int64_t(blk) * NB + t0 + i * ROWS) * step + c);
#pragma unroll
            for (int i = 0; i < STEPS; ++i)
                if (t0 + i * ROWS < rest) *reinterpret_cast<uint4 *>(dst + (t0 + i * ROWS) * p.tail_stride_s + c) = row[i];
            return;
        }
    }
    const int dst_blk = blk + dst_off / NB;
    auto sync = [] { __syncthreads(); };
    if (blockIdx.x < SPLIT * p.h_k) {
        pack_k_part<BITS, GROUP, BF16>(p, sh, tid, ib, blockIdx.x / SPLIT, blockIdx.x % SPLIT, blk, dst_blk, sync);
    } else {
        const int xv = blockIdx.x - SPLIT * p.h_k;
        pack_v_part<BITS, GROUP, BF16>(p, sh, tid, ib, xv % p.h_k, xv / p.h_k, blk, dst_blk, sync);
    }
}

template <int BITS, int GROUP, bool BF16>
static cudaError_t launch_pack_t(const PackParams &p, cudaStream_t stream) {
    constexpr int NB = 32 * (16 / BITS);
    constexpr int NTHREADS = kPackThreads<BITS>;
    dim3 grid(2 * kPackSplit<BITS> * p.h_k, (p.s + NB - 1) / NB, p.b);       // (whole blocks, except for prompts)
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(NTHREADS);
    cfg.stream = stream;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;            // (one block of 8 sequences, stream launches: 4.15 -> 2.5 us a launch)
    return cudaLaunchKernelEx(&cfg, bd_pack_kernel<BITS, GROUP, BF16>, p);
}

cudaError_t launch_pack(const PackParams &p, int bits, int group, int dtype, cudaStream_t stream) {
    const bool bf = dtype == BD_BF16;
    if (bits == 4 && group == 128) return bf ? launch_pack_t<4, 128, true>(p, stream) : launch_pack_t<4, 128, false>(p, stream);
    if (bits == 4 && group == 64)  return bf ? launch_pack_t<4, 64, true>(p, stream)  : launch_pack_t<4, 64, false>(p, stream);
    if (bits == 2 && group == 128) return bf ? launch_pack_t<2, 128, true>(p, stream) : launch_pack_t<2, 128, false>(p, stream);
    if (bits == 2 && group == 64)  return bf ? launch_pack_t<2, 64, true>(p, stream)  : launch_pack_t<2, 64, false>(p, stream);
    if (bits == 4 && group == 32)  return bf ? launch_pack_t<4, 32, true>(p, stream)  : launch_pack_t<4, 32, false>(p, stream);
    if (bits == 2 && group == 32)  return bf ? launch_pack_t<2, 32, true>(p, stream)  : launch_pack_t<2, 32, false>(p, stream);
    return cudaErrorInvalidValue;
}

}  // namespace bd
