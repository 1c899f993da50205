// Prefill self-attention on the 5th-generation tensor cores (tcgen05 / TMEM), causal with optional left padding
// (LLaMA) or ALiBi bias (Baichuan-13B).
//
// Reference: q_k_mul + qk_softmax + attn_v_mul + transpose of LlamaMmha::forward_full
// (csrc/op/llama_mmha.cpp:354-426; softmax_kernel_gpt2 csrc/core/gpt2_self_softmax.cu:8-57; ALiBi variant
// masked_softmax_kernel :161-240): two cuBLAS batched GEMMs around a row-serial softmax over a materialised
// [B,H,S,S] fp16 score buffer.  Here one CTA owns 128 consecutive queries of one (batch, head) and walks the keys
// in blocks of 64, never past the diagonal and never left of the padding; nothing of size S x S exists.
//
// B200 design (two CTAs per SM, 256 tensor-memory columns and 97 KiB of shared memory each: what one CTA cannot
// overlap by itself the other fills):
//   warp 0 (one lane)  TMA producer: the Q tile once, then K and V tiles of 64 keys into two-stage rings (a K
//                      stage is free again when its Q.K^T has completed, a V stage when its P.V has); 3-D tensor
//                      maps with the 128-byte swizzle, rows past the prompt read as zeros.  It sets the barriers
//                      up itself and requests Q and the first two blocks before the block-wide barrier and the
//                      tensor-memory allocation.
//   warp 1 (one lane)  MMA issuer: S = Q.K^T (M128 x N64 x K16, eight per block, both operands K-major from
//                      shared memory) into one of two score buffers in tensor memory - the scores of block j+1
//                      are computed while the softmax of block j runs; O += P.V (four per block) with P read FROM
//                      TENSOR MEMORY as the A operand and V straight from its [key][dim] tile as an MN-major B
//                      operand - V is never transposed and P never touches shared memory.
//   warps 2-5          softmax, one thread per query row (= TMEM lane): tcgen05.ld of the row's 64 scores,
//                      scale / bias / masks, running max and sum, probabilities back INTO THE
//                      SCORE COLUMNS as fp16 pairs (tcgen05.st: a row only ever touches its own lane, and the
//                      tensor core overwrites a score buffer only after the P.V that read it, in issue order);
//                      the O accumulator is rescaled only when a row's maximum has outgrown the one that O is
//                      accumulated under by 2^8 (the conditional rescaling that FlashAttention-4 made known).  At the
//                      end they read O, normalise and store the context.
// Every wait is bounded (device status 2) and the CTA frees its tensor memory on every path.
//
// Numerics kept from the reference and from the mma.sync kernel this one replaces for long prompts: scores scaled
// by the fp16-rounded 1/sqrt(D), the ALiBi bias added in fp32, probabilities enter P.V as fp16, denominator + 1e-6, rows
// above the left padding are zero.  The scores stay in fp32: the reference stores them as fp16, which costs more than half of
// the error of the result (relative to 64 bits 4.4e-4 with that rounding, 2.6e-4 without it, 2 x 2048 tokens).
//
// Measured, 32 heads: 2 x 2048 tokens 85 us (136 with a rescale of O in nearly every block, one chain of 64 maxima, the
// tiles of a pair behind one another and the fp16 rounding), 8 x 512 46 us (57); 40 heads with a bias, 2 x 701 tokens 40 us
// (56).  Time stamps: a block takes 1650 cycles on each of an SM's two CTAs, and the issuing thread is the one that never waits: Q.K^T
// with 64 keys reads 6 KiB of shared memory per MMA (48 cycles) for 32 cycles of multiplications.
#include <cuda.h>

#include "common.cuh"
#include "kernels.h"

namespace eet {

namespace {

constexpr int kPtQ = 128;                      // queries per CTA
constexpr int kPtK = 64;                       // keys per block
constexpr int kPtThreads = 192;
constexpr int kPtQHalf = 128 * 128;            // bytes of the [128 queries][64 halves] swizzled half of the Q tile
constexpr int kPtQTile = 2 * kPtQHalf;         // dims 0-63, then dims 64-127
constexpr int kPtKvHalf = kPtK * 128;          // the same for a [64 keys][64 halves] half of a K or V tile
constexpr int kPtKvTile = 2 * kPtKvHalf;
constexpr int kPtStages = 2;
constexpr uint32_t kPtTmemCols = 256;
constexpr uint32_t kPtColS = 0;                // two score buffers of 64 fp32 columns; a block's probabilities
                                               // (32 columns: 64 fp16 as pairs) go over the first half of its scores
constexpr uint32_t kPtColO = 128;              // the context accumulator, 128 fp32 columns
constexpr int kPtSmem = kPtQTile + 2 * kPtStages * kPtKvTile + 1024;

struct PtSmem {
    uint64_t q_full;
    uint64_t k_full[kPtStages], k_empty[kPtStages];   // K tile landed / its Q.K^T has completed
    uint64_t v_full[kPtStages], v_empty[kPtStages];   // V tile landed / its P.V has completed
    uint64_t s_full[2];         // Q.K^T of a block has completed
    uint64_t p_ready[2];        // probabilities written, O rescaled (four softmax warps): P.V may be issued
    uint64_t pv_done[2];        // a block's P.V has completed (blocks alternate between the two: a softmax warp can
                                // be a whole block ahead of the slowest one, and one barrier's parity could then
                                // no longer tell "the previous P.V" from "the one before it")
    uint32_t tmem_base;
    volatile int abort;
};

__device__ __forceinline__ void tma_load_3d(void* smem_dst, const CUtensorMap* map, int x, int y, int z, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(
            smem_u32(smem_dst)),
        "l"(map), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ float ex2_approx(float x)
{
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// B operand held [k][n] with n contiguous (MN-major), 128-byte swizzle: 64 n-values per 128-byte row, 8 k-rows per
// 1024-byte group (stride byte offset), the next 64 n-values `lbo_bytes` further (leading byte offset).
__device__ __forceinline__ uint64_t umma_desc_mn_sw128(uint32_t smem_addr, uint32_t lbo_bytes)
{
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);
    d |= (uint64_t)(lbo_bytes >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// The ALiBi bias of one query for 64 keys, requested early: nine aligned 16-byte words that cover the 128 bytes (a row of
// the bias starts at any even address: its length is the prompt's).  Only words that hold a bias this query needs are
// read - keys up to min(i, key0 + 63); the others count as zero.  A word at either end may hold up to 14 bytes that are not
// this row's, at the ends of the tensor not the tensor's; they lie in the same aligned 16 bytes as one of its values, so
// in the same page, and are masked or shifted out.  40 heads, 2 x 701 tokens: 60 us, against 138 with 64 two-byte loads a thread, each touching 32 rows.
struct PtBias {
    uint32_t w[36];
    uint32_t shift;   // bytes from w[0] to the first bias

    __device__ __forceinline__ void load(const __half* row, int key0, int i, bool live)
    {
        const uintptr_t first = reinterpret_cast<uintptr_t>(row + key0);
        const uintptr_t last = reinterpret_cast<uintptr_t>(row + min(i, key0 + kPtK - 1));
        const uintptr_t base = first & ~(uintptr_t)15;
        shift = (uint32_t)(first & 15);
#pragma unroll
        for (int c = 0; c < 9; ++c) {
            uint4 v = make_uint4(0u, 0u, 0u, 0u);
            if (live && key0 <= i && base + 16 * c <= last) v = __ldg(reinterpret_cast<const uint4*>(base + 16 * c));
            w[4 * c] = v.x;
            w[4 * c + 1] = v.y;
            w[4 * c + 2] = v.z;
            w[4 * c + 3] = v.w;
        }
    }
    // w[k] becomes the biases of keys key0 + 2 k and key0 + 2 k + 1
    __device__ __forceinline__ void align()
    {
#pragma unroll
        for (int k = 0; k < 34; ++k) w[k] = (shift & 8) ? w[k + 2] : w[k];
#pragma unroll
        for (int k = 0; k < 33; ++k) w[k] = (shift & 4) ? w[k + 1] : w[k];
        const uint32_t sel = (shift & 2) ? 0x5432u : 0x3210u;
#pragma unroll
        for (int k = 0; k < 32; ++k) w[k] = __byte_perm(w[k], w[k + 1], sel);
    }
};

// 32 columns of tensor memory into 32 registers, without waiting for them
__device__ __forceinline__ void tmem_ld32_async(uint32_t taddr, uint32_t* v)
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];\n"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr));
}

// (the registers pass through the wait, so that nothing reads them above it)
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&v)[kPtK])
{
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int c = 0; c < kPtK; ++c) asm volatile("" : "+r"(v[c]));
}

// The FP32 operations of the softmax, two scores at a time (one instruction for a pair of registers).
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b)
{
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ uint64_t pair2(float a, float b)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 split2(uint64_t v)
{
    float2 f;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(f.x), "=f"(f.y) : "l"(v));
    return f;
}

__device__ __forceinline__ float max3(float a, float b, float c)
{
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// exp(s - m) of a row's 64 scores as one FMA and one ex2 each (-inf stays -inf and gives 0), as fp16 pairs; returns their sum
__device__ __forceinline__ float exponentials(const uint64_t (&sc)[kPtK / 2], float to_log2, float m, uint32_t (&pk)[kPtK / 2])
{
    const uint64_t to_log2_2 = pair2(to_log2, to_log2), m_l2 = pair2(-m * to_log2, -m * to_log2);
    uint64_t psum[2] = {0ull, 0ull};
#pragma unroll
    for (int c = 0; c < kPtK / 2; ++c) {
        const float2 e = split2(fma2(sc[c], to_log2_2, m_l2));
        const float p0 = ex2_approx(e.x), p1 = ex2_approx(e.y);
        psum[c & 1] = add2(psum[c & 1], pair2(p0, p1));
        const __half2 hp = __floats2half2_rn(p0, p1);
        pk[c] = *reinterpret_cast<const uint32_t*>(&hp);
    }
    const float2 ps = split2(add2(psum[0], psum[1]));
    return ps.x + ps.y;
}

template<bool kBias>
__global__ void __launch_bounds__(kPtThreads, 2)
prefill_mha_tc_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                      const __grid_constant__ CUtensorMap map_v, __half* __restrict__ ctx, int S, int H, int heads, int group,
                      const int64_t* __restrict__ pad_len, const __half* __restrict__ alibi, int alibi_stride)
{
    constexpr int D = 128;
    extern __shared__ __align__(1024) uint8_t pt_dyn[];
    __shared__ PtSmem sm;
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(pt_dyn) + 1023) & ~(uintptr_t)1023);
    uint8_t* q_tile = base;
    uint8_t* k_ring = q_tile + kPtQTile;
    uint8_t* v_ring = k_ring + kPtStages * kPtKvTile;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // Tiles in the order of their length, the longest (late queries) of all (batch, head) pairs of a group first, so that
    // short ones fill the end: with the tiles of one pair behind another a pair's longest tile began last.
    // A group is as many pairs as fit the L2 with their keys and values.
    const int q_tiles = (S + kPtQ - 1) / kPtQ;
    const int first_pair = (int)blockIdx.x / (q_tiles * group) * group;
    const int in_group = min(group, heads - first_pair);
    const int place = (int)blockIdx.x - first_pair * q_tiles;
    const int bh = first_pair + place % in_group;
    const int b = bh / H, h = bh % H;
    const int i0 = (q_tiles - 1 - place / in_group) * kPtQ;
    const int pad = (pad_len != nullptr && alibi == nullptr) ? (int)pad_len[b] : 0;
    const int kb_first = pad / kPtK;                                        // key blocks left of the padding are skipped
    const int kb_last = min((i0 + kPtQ - 1) / kPtK, (S - 1) / kPtK);        // causal: nothing above the diagonal
    const int n_blocks = kb_last - kb_first + 1;                            // <= 0: the whole tile lies inside the padding

    auto load_kv = [&](uint8_t* tile, const CUtensorMap* map, int key0, uint64_t* bar) {
        mbar_arrive_expect_tx(bar, (uint32_t)kPtKvTile);
        tma_load_3d(tile, map, 0, key0, bh, bar);
        tma_load_3d(tile + kPtKvHalf, map, 64, key0, bh, bar);
    };
    if (warp == 0 && elect_one()) {
        mbar_init(&sm.q_full, 1);
        for (int st = 0; st < kPtStages; ++st) {
            mbar_init(&sm.k_full[st], 1);
            mbar_init(&sm.k_empty[st], 1);
            mbar_init(&sm.v_full[st], 1);
            mbar_init(&sm.v_empty[st], 1);
        }
        for (int st = 0; st < 2; ++st) {
            mbar_init(&sm.s_full[st], 1);
            mbar_init(&sm.p_ready[st], 4);
        }
        mbar_init(&sm.pv_done[0], 1);
        mbar_init(&sm.pv_done[1], 1);
        sm.abort = 0;
        mbar_fence_init();
        // nobody else touches the barriers before the block-wide barrier below: the first loads go out now
        if (n_blocks > 0) {
            mbar_arrive_expect_tx(&sm.q_full, (uint32_t)kPtQTile);
            tma_load_3d(q_tile, &map_q, 0, i0, bh, &sm.q_full);
            tma_load_3d(q_tile + kPtQHalf, &map_q, 64, i0, bh, &sm.q_full);
            for (int jl = 0; jl < kPtStages && jl < n_blocks; ++jl) {
                load_kv(k_ring + jl * kPtKvTile, &map_k, (kb_first + jl) * kPtK, &sm.k_full[jl]);
                load_kv(v_ring + jl * kPtKvTile, &map_v, (kb_first + jl) * kPtK, &sm.v_full[jl]);
            }
        }
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)),
                     "r"(kPtTmemCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = sm.tmem_base;

    if (warp == 0) {
        // ------------------------------------------------------------------ TMA producer
        if (elect_one()) {
            for (int jl = kPtStages; jl < n_blocks; ++jl) {
                const int st = jl % kPtStages;
                const uint32_t ph = (uint32_t)((jl / kPtStages - 1) & 1);
                const int key0 = (kb_first + jl) * kPtK;
                if (!tc_wait(&sm.k_empty[st], ph, &sm.abort)) break;
                load_kv(k_ring + st * kPtKvTile, &map_k, key0, &sm.k_full[st]);
                if (!tc_wait(&sm.v_empty[st], ph, &sm.abort)) break;
                load_kv(v_ring + st * kPtKvTile, &map_v, key0, &sm.v_full[st]);
            }
        }
    }
    else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        if (n_blocks > 0 && elect_one()) {
            constexpr uint32_t idesc_qk = umma_idesc_f16(128, kPtK);                  // both operands K-major
            constexpr uint32_t idesc_pv = umma_idesc_f16(128, D) | (1u << 16);        // B operand MN-major
            const uint64_t q_desc = umma_desc_sw128(smem_u32(q_tile));
            const uint64_t k_desc0 = umma_desc_sw128(smem_u32(k_ring));
            const uint64_t v_desc0 = umma_desc_mn_sw128(smem_u32(v_ring), (uint32_t)kPtKvHalf);
            // Q.K^T of block jl into score buffer jl & 1.  That buffer last held the probabilities of block jl - 2,
            // whose P.V was issued before this: the tensor core executes in issue order.
            auto issue_qk = [&](int jl) -> bool {
                const int st = jl % kPtStages;
                if (!tc_wait(&sm.k_full[st], (uint32_t)((jl / kPtStages) & 1), &sm.abort)) return false;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t kd = k_desc0 + (uint64_t)(st * (kPtKvTile >> 4));
#pragma unroll
                for (int kk = 0; kk < 8; ++kk) {
                    // 16 head dims per MMA: 32 bytes along the swizzled row; dims 64-127 sit in the second half tile
                    const uint64_t qoff = (uint64_t)((kk >> 2) * (kPtQHalf >> 4) + (kk & 3) * 2);
                    const uint64_t koff = (uint64_t)((kk >> 2) * (kPtKvHalf >> 4) + (kk & 3) * 2);
                    umma_f16(tmem + kPtColS + (uint32_t)((jl & 1) * kPtK), q_desc + qoff, kd + koff, idesc_qk, kk != 0);
                }
                umma_commit(&sm.s_full[jl & 1]);
                umma_commit(&sm.k_empty[st]);
                return true;
            };
            bool ok = tc_wait(&sm.q_full, 0, &sm.abort) && issue_qk(0);
            for (int jl = 0; jl < n_blocks && ok; ++jl) {
                if (jl + 1 < n_blocks) ok = issue_qk(jl + 1);   // runs while the softmax of block jl does
                if (!ok) break;
                const int st = jl % kPtStages;
                if (!tc_wait(&sm.p_ready[jl & 1], (uint32_t)((jl >> 1) & 1), &sm.abort) ||
                    !tc_wait(&sm.v_full[st], (uint32_t)((jl / kPtStages) & 1), &sm.abort)) {
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint64_t vd = v_desc0 + (uint64_t)(st * (kPtKvTile >> 4));
#pragma unroll
                for (int kk = 0; kk < kPtK / 16; ++kk) {
                    // 16 keys per MMA: 8 columns of P, two 8-row groups (2048 bytes) of the V tile
                    umma_f16_ts(tmem + kPtColO, tmem + kPtColS + (uint32_t)((jl & 1) * kPtK + kk * 8),
                                vd + (uint64_t)(kk * (2048 >> 4)), idesc_pv, jl != 0 || kk != 0);
                }
                umma_commit(&sm.pv_done[jl & 1]);
                umma_commit(&sm.v_empty[st]);
            }
        }
    }
    else {
        // ------------------------------------------------------------------ softmax warps, then the epilogue
        const int lane_base = (warp & 3) * 32;               // the TMEM lanes this warp may access
        const int r = lane_base + lane;                      // query row inside the tile
        const int i = i0 + r;
        const uint32_t t_lane = (uint32_t)lane_base << 16;
        const float scalar = __half2float(__float2half(sqrtf(1.0f / D)));
        const uint64_t scalar2 = pair2(scalar, scalar);
        // From the scores as they are kept (scaled already with a bias, straight from the accumulator without) to powers of 2.
        const float to_log2 = kBias ? 1.4426950408889634f : 1.4426950408889634f * scalar;
        // m_ref: the maximum under which O and l_run are accumulated.  It follows the running maximum m_run only when that
        // has outgrown it by 2^8: until then the probabilities are at most 256, which fp16 holds as exactly as those
        // up to 1, and the common factor leaves with the division at the end.
        float m_run = -1e20f, m_ref = -1e20f, l_run = 0.f;
        const __half* arow = kBias ? alibi + ((size_t)h * alibi_stride + (i < S ? i : 0)) * alibi_stride : nullptr;
        bool ok = n_blocks > 0;
        for (int jl = 0; jl < n_blocks && ok; ++jl) {
            const int key0 = (kb_first + jl) * kPtK;
            PtBias bias;
            if (kBias) bias.load(arow, key0, i, i < S);   // on its way while the scores are computed
            const uint32_t t_s = tmem + t_lane + kPtColS + (uint32_t)((jl & 1) * kPtK);   // this block's score buffer
            if (!tc_wait_warp(&sm.s_full[jl & 1], (uint32_t)((jl >> 1) & 1), &sm.abort)) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            uint64_t sc[kPtK / 2];
            {
                uint32_t v[kPtK];
                tmem_ld32_async(t_s, v);
                tmem_ld32_async(t_s + 32, v + 32);
                if (kBias) bias.align();
                tmem_ld_wait(v);
#pragma unroll
                for (int c = 0; c < kPtK / 2; ++c) sc[c] = pair2(__uint_as_float(v[2 * c]), __uint_as_float(v[2 * c + 1]));
            }
            if (kBias) {
#pragma unroll
                for (int c = 0; c < kPtK / 2; ++c) {
                    const float2 b2 = __half22float2(*reinterpret_cast<const __half2*>(&bias.w[c]));
                    sc[c] = fma2(sc[c], scalar2, pair2(b2.x, b2.y));
                }
            }
            // a block left of the diagonal of all rows of the warp, right of the padding and inside the prompt needs no mask
            if (!((key0 + kPtK - 1 <= i0 + lane_base) && (key0 >= pad) && (key0 + kPtK <= S))) {
#pragma unroll
                for (int c = 0; c < kPtK / 2; ++c) {
                    const int j = key0 + 2 * c;
                    float2 f = split2(sc[c]);
                    f.x = (j <= i && j >= pad && j < S) ? f.x : -INFINITY;
                    f.y = (j + 1 <= i && j + 1 >= pad && j + 1 < S) ? f.y : -INFINITY;
                    sc[c] = pair2(f.x, f.y);
                }
            }
            // (four chains side by side: one of 64 dependent maxima took as long as the exponentials)
            float mx[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int c = 0; c < kPtK / 2; ++c) {
                const float2 f = split2(sc[c]);
                mx[c & 3] = max3(mx[c & 3], f.x, f.y);
            }
            m_run = fmaxf(m_run, fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])));
            float corr = 1.0f;
            const bool moves = (m_run - m_ref) * to_log2 > 8.0f;
            if (moves) {
                corr = ex2_approx((m_ref - m_run) * to_log2);
                m_ref = m_run;
            }
            uint32_t pk[kPtK / 2];
            l_run = l_run * corr + exponentials(sc, to_log2, m_ref, pk);
            // probabilities as the A operand of P.V: lane = query, 16-bit pairs along the columns, written over the
            // first half of this row's scores (which are in registers by now)
            tmem_st32(t_s, pk);
            // rescale O where a row of this warp has moved its reference, after the previous block's P.V has completed
            if (jl > 0 && __any_sync(0xffffffffu, moves)) {
                if (!tc_wait_warp(&sm.pv_done[(jl - 1) & 1], (uint32_t)(((jl - 1) >> 1) & 1), &sm.abort)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
                for (int c0 = 0; c0 < D; c0 += 32) {
                    uint32_t v[32];
                    tmem_ld32(tmem + t_lane + kPtColO + (uint32_t)c0, v);
#pragma unroll
                    for (int c = 0; c < 32; ++c) v[c] = __float_as_uint(__uint_as_float(v[c]) * corr);
                    tmem_st32(tmem + t_lane + kPtColO + (uint32_t)c0, v);
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.p_ready[jl & 1]);
        }

        // ---- normalise and store: context layout [B][S][H*D] (the transpose of llama_mmha.cpp:418-426) ----
        if (n_blocks > 0 && ok) {
            int done = 1;
            if (lane == 0) {
                done = tc_wait(&sm.pv_done[(n_blocks - 1) & 1], (uint32_t)(((n_blocks - 1) >> 1) & 1), &sm.abort) ? 1 : 0;
            }
            done = __shfl_sync(0xffffffffu, done, 0);
            ok = done != 0;
        }
        if (i < S) {
            __half* dst = ctx + (((size_t)b * S + i) * H + h) * D;
            if (n_blocks <= 0 || !ok) {
                // the whole tile lies inside the left padding (or a wait ran out): rows of zeros
                const uint4 z = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
                for (int c = 0; c < D / 8; ++c) reinterpret_cast<uint4*>(dst)[c] = z;
            }
        }
        if (n_blocks > 0 && ok) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            // rows above the left padding are zeroed by the reference (gpt2_self_softmax.cu:24-30)
            const float inv = (i < pad) ? 0.f : 1.0f / (l_run + 1e-6f * ex2_approx((m_run - m_ref) * to_log2));
#pragma unroll 1
            for (int c0 = 0; c0 < D; c0 += 32) {
                uint32_t v[32];
                tmem_ld32(tmem + t_lane + kPtColO + (uint32_t)c0, v);   // (warp-collective: rows past the prompt take part)
                if (i < S) {
                    __half* dst = ctx + (((size_t)b * S + i) * H + h) * D + c0;
#pragma unroll
                    for (int c = 0; c < 32; c += 8) {
                        uint4 o;
                        __half2* oh = reinterpret_cast<__half2*>(&o);
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            oh[e] = __floats2half2_rn(__uint_as_float(v[c + 2 * e]) * inv, __uint_as_float(v[c + 2 * e + 1]) * inv);
                        }
                        *reinterpret_cast<uint4*>(dst + c) = o;
                    }
                }
            }
        }
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kPtTmemCols) : "memory");
    }
}

// [rows_per_bh rows of 128 halves] x n_bh, of which the first `rows` of every (batch, head) are valid: reads past
// them return zeros, so a key block that reaches beyond the prompt never feeds stale cache rows (possibly NaN)
// into P.V.
int encode_rows_map(CUtensorMap* map, const __half* basep, int rows, size_t rows_per_bh, int n_bh, int box_rows)
{
    EncodeTiledFn encode = encode_tiled_fn();
    EET_CHECK(encode != nullptr, "prefill attention: cuTensorMapEncodeTiled is not available from the driver");
    const cuuint64_t dims[3] = {128, (cuuint64_t)rows, (cuuint64_t)n_bh};
    const cuuint64_t strides[2] = {256, (cuuint64_t)rows_per_bh * 256};
    const cuuint32_t box[3] = {64, (cuuint32_t)box_rows, 1};
    const cuuint32_t elem[3] = {1, 1, 1};
    const CUresult rc = encode(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<__half*>(basep), dims, strides, box, elem,
                               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    EET_CHECK(rc == CUDA_SUCCESS, "prefill attention: cuTensorMapEncodeTiled failed with code %d", (int)rc);
    return 0;
}

}  // namespace

// Prompts of at least this many tokens go to the tensor-core kernel (its tiles are 128 queries x 64 keys).
constexpr int kPrefillTcMinS = 96;
constexpr long long kPtGroupBytes = 64ll << 20;   // keys and values that are worked on at a time: half of the L2

bool prefill_mha_tc_supported(int S, int D)
{
    return D == 128 && S >= kPrefillTcMinS;
}

int launch_prefill_mha_tc(const __half* q, const __half* kcache, const __half* vcache, __half* ctx, int B, int S, int H,
                          int T_max, const int64_t* pad_len, const __half* alibi, int alibi_stride, cudaStream_t stream)
{
    EET_CHECK((long long)B * H <= 65535, "prefill attention: batch x heads = %lld exceeds 65535", (long long)B * H);
    CUtensorMap map_q, map_k, map_v;
    if (int rc = encode_rows_map(&map_q, q, S, (size_t)S, B * H, kPtQ)) return rc;
    if (int rc = encode_rows_map(&map_k, kcache, S, (size_t)T_max, B * H, kPtK)) return rc;
    if (int rc = encode_rows_map(&map_v, vcache, S, (size_t)T_max, B * H, kPtK)) return rc;
    auto kern = alibi != nullptr ? prefill_mha_tc_kernel<true> : prefill_mha_tc_kernel<false>;
    static bool attr_set[64][2] = {};
    int dev = 0;
    EET_CUDA(cudaGetDevice(&dev));
    dev &= 63;
    if (!attr_set[dev][alibi != nullptr]) {
        EET_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, kPtSmem));
        attr_set[dev][alibi != nullptr] = true;
    }
    const long long blocks = (long long)((S + kPtQ - 1) / kPtQ) * B * H;
    EET_CHECK(blocks <= 0x7fffffffLL, "prefill attention: %lld tiles exceed the grid limit", blocks);
    const long long fit = kPtGroupBytes / ((long long)S * 512);   // K and V of a pair: 512 bytes a token
    const int group = fit < 1 ? 1 : (fit < B * H ? (int)fit : B * H);
    kern<<<(unsigned)blocks, kPtThreads, kPtSmem, stream>>>(map_q, map_k, map_v, ctx, S, H, B * H, group, pad_len, alibi, alibi_stride);
    EET_LAUNCH_CHECK();
    return 0;
}

}  // namespace eet
