// W8A16 tensor-core GEMM for the prefill regime (and from 65 tokens on where its tiles fill the machine better than the
// stream-K kernel's units): C[M,N] = A[M,K] (fp16) x dequant(B), B in the W8T64 layout, per-channel fp16 scale (and
// optional fp16 residual or gated activation) in the epilogue.
//
// Replaces the reference's fpA_intB GEMM (kernel cutlass_extensions/.../gemm/kernel/fpA_intB_gemm.h:60-486,
// mainloop .../threadblock/dq_mma_multistage.h:490-583: mma.sync m16n8k16 with int8 -> fp16 conversion in
// registers after ldmatrix), which has no path for sm_90 or later.
//
// B200 design (tcgen05 / TMEM, one CTA per 256-channel x BN-token output tile, BN a multiple of 16 up to 256):
//  * "swap AB": the weights are the 128-row M operand of tcgen05.mma, the tokens the N operand (BN up to
//    256), so any batch of tokens fills the tensor core and the per-channel scale is per TMEM lane.
//  * Per 64-wide k-block the W8T64 tiles of the 256 channels come by 1-D bulk copies and the BN x 64 activation tile by
//    one 2-D tensor-map copy that lands in the 128-byte-swizzled K-major layout the MMA reads.
//  * Eight warps turn the int8 weights into fp16 (prmt + sub.f16x2, exact) and write them into shared
//    memory in the same swizzled K-major layout - the int8 bytes never go through the tensor core as int8
//    and the weights are never materialised as fp16 in global memory.
//  * After the last k-block the same warps read the accumulators with tcgen05.ld (lane = channel), multiply by
//    the channel's scale, round once to fp16, and pass 128 x 32 blocks through shared memory so that the
//    stores (and the residual loads) are 16-byte accesses of whole 256-byte row segments.
//  Every wait is bounded; a wait that runs out sets the device status word, and the CTA still frees its
//  tensor memory before it returns.
//
// (The weights in tensor memory as the MMA's A operand: gemm_ts.cu, which takes most shapes whose tiles fill a wave or less.  Here a
// k-block is bound by shared memory, 768 + 3 BN cycles, and by the 98 B/ns that an SM gets from L2.)
//
// Numerics: exact integer weights as fp16, fp32 accumulation, one multiply by the fp16 scale, one rounding
// to fp16 - the same as the skinny kernel's finalize step.
#include <cuda.h>
#include <cooperative_groups.h>

#include "common.cuh"
#include "kernels.h"

namespace eet {

namespace {

constexpr int kTcW8Bytes = 2 * kTileBytes;          // 128 channels x 64 k, int8
constexpr uint32_t kTcSpin = 1u << 24;

// Bounded wait of the warp-specialised kernels.  The roles that issue work are SINGLE threads whose loop
// is a chain of dependent instructions (a few cycles each at best): the common case - the phase has
// already completed - must cost one try_wait and nothing else.
__device__ __noinline__ bool tc_wait_slow(uint64_t* bar, uint32_t parity, volatile int* abort)
{
    for (uint32_t i = 0; i < kTcSpin; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if (*abort) return false;
    }
    *abort = 1;
    g_device_status = 2;
    return false;
}

__device__ __forceinline__ bool tc_wait(uint64_t* bar, uint32_t parity, volatile int* abort)
{
    if (mbar_try_wait(bar, parity)) return true;
    return tc_wait_slow(bar, parity, abort);
}

// The same for the 32 lanes of a converged warp: all of them get the same answer, so the warp cannot part on its way to a
// barrier.  (One vote where the phase is complete already, the usual case.)
__device__ __noinline__ bool tc_wait_warp_slow(uint64_t* bar, uint32_t parity, volatile int* abort)
{
    for (uint32_t i = 0; i < kTcSpin; ++i) {
        if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
        if (__any_sync(0xffffffffu, *abort)) return false;
    }
    *abort = 1;
    g_device_status = 2;
    return false;
}

__device__ __forceinline__ bool tc_wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort)
{
    if (__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) return true;
    return tc_wait_warp_slow(bar, parity, abort);
}

// shared-memory matrix descriptor: K-major, 128-byte swizzle, rows of 128 bytes, 8-row groups 1024 B apart
__device__ __forceinline__ uint64_t umma_desc_sw128(uint32_t smem_addr)
{
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFF) >> 4);        // start address, 16-byte units
    d |= (uint64_t)1 << 16;                             // leading byte offset (unused with swizzle)
    d |= (uint64_t)(1024 >> 4) << 32;                   // stride byte offset between 8-row groups
    d |= (uint64_t)1 << 46;                             // descriptor version of this architecture
    d |= (uint64_t)2 << 61;                             // SWIZZLE_128B
    return d;
}

// instruction descriptor for kind::f16: fp16 A and B, fp32 accumulate, both operands K-major
__host__ __device__ constexpr uint32_t umma_idesc_f16(int m, int n)
{
    return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(m >> 4) << 24);
}

__device__ __forceinline__ void umma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, bool accumulate)
{
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t"
        "}\n" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"((uint32_t)accumulate)
        : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t* bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* map, int x, int y, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(smem_dst)),
        "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32])
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
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Epilogue of one block of 128 channels x 32 tokens.  After tcgen05.ld every epilogue thread holds the 32
// token sums of ONE channel, while the output is channel-contiguous; the block therefore goes through a
// [32 tokens][128 channels] fp16 staging tile in shared memory (the operand rings are idle by then) and
// leaves as 16-byte stores of whole 256-byte row segments, with the residual fetched the same way and all
// four residual loads of a thread in flight before the first add.  Two staging tiles alternate so one named
// barrier per block is enough.  Called by all 128 epilogue threads.
constexpr int kEpiStageHalves = 32 * 128;

template<int kBarId = 1>
__device__ __forceinline__ void epilogue_block(const uint32_t (&v)[32], float sc, __half* stage, int channel, int tw,
                                               __half* C, const __half* residual, int gate, int m_first, int M, int N,
                                               int n_first)
{
#pragma unroll
    for (int j = 0; j < 32; ++j) stage[j * 128 + channel] = __float2half(__uint_as_float(v[j]) * sc);
    asm volatile("bar.sync %0, 128;" ::"n"(kBarId) : "memory");
    uint4 res[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int idx = tw + i * 128, row = idx >> 4, ch8 = idx & 15;
        res[i] = make_uint4(0u, 0u, 0u, 0u);
        if (residual != nullptr && m_first + row < M) {
            res[i] = *reinterpret_cast<const uint4*>(residual + (size_t)(m_first + row) * N + n_first + ch8 * 8);
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int idx = tw + i * 128, row = idx >> 4, ch8 = idx & 15;
        if (m_first + row < M) {
            uint4 o = *reinterpret_cast<const uint4*>(stage + row * 128 + ch8 * 8);
            if (residual != nullptr) {
                __half2* oh = reinterpret_cast<__half2*>(&o);
                const __half2* rh = reinterpret_cast<const __half2*>(&res[i]);
                if (gate) {
                    // the second operand is the gate projection: this GEMM is the up projection of a gated FFN
#pragma unroll
                    for (int e = 0; e < 4; ++e) oh[e] = gated_silu2(rh[e], oh[e]);
                }
                else {
#pragma unroll
                    for (int e = 0; e < 4; ++e) oh[e] = __hadd2(oh[e], rh[e]);
                }
            }
            *reinterpret_cast<uint4*>(C + (size_t)(m_first + row) * N + n_first + ch8 * 8) = o;
        }
    }
}

// ---------------------------------------------------------------------------------------------------
// Two accumulators (one per 128-channel half) fill the TMEM columns, and every activation tile fetched from L2 feeds both
// halves.  The three data streams have their own rings so that each can run as far ahead as its buffer allows (the launcher
// deals what shared memory has: BN = 256 three stages of activations and four of weights, BN = 128 five of each):
//   activations : BN x 128 bytes a stage, one 2-D TMA copy per k-block            (warp 0)
//   int8 weights: 16 KiB, four 4 KiB bulk copies per k-block                     (warp 6)
//   fp16 weights: 2 x 32 KiB (k-block x two 128-channel halves), written by warps 2-5 / 7-10, read by tcgen05.mma
// One commit per k-block ("done") releases the activation stage to its
// producer and the fp16 stage to the transform warps: the issuing thread pays for two waits, eight MMAs and
// one commit per k-block.  N is a multiple of 128: the last tile of a row may have a lower half only.
//
// Two ways to spread the tiles over the SMs:
//
// (a) Persistent CTAs (gridDim.z == 1), one per SM (fewer when there are fewer tiles): CTA i takes tiles i, i + G,
//     i + 2G, ... so that the CTAs of a wave walk the k-blocks in step: 16 CTAs want the same activation or
//     weight tile at about the same time (measured: out of step the k-loop runs 1.3x slower).  The rings and all
//     phase counters run on
//     across tiles: while the transform warps are busy with a tile's epilogue, the producers already fetch the
//     next tile's first k-blocks.  The epilogue's fp16 staging tiles live in the fp16 weight ring, which is idle
//     exactly then (all MMAs of the tile have completed, the next conversions come after).
//     Two ways of cutting the work so that no SM idles through the last, partial wave were built and measured
//     on 148 SMs, and dropped: (i) textbook stream-K (equal contiguous ranges of (tile, k-block) pairs, partial
//     accumulators handed on through a global scratch) ran 1.3x slower per k-block, because the CTAs no longer
//     read the same tiles at the same time (4096^2, M = 4096: 145 us against 109); (ii) whole tiles in waves and
//     only the left-over tiles cut along K into pieces that keep the k-blocks in step gained 0-3 % (4096 x 12288,
//     M = 4096: 328 us against 330; 11008 x 4096: 267 against 274) - exporting and importing 256 KiB accumulators
//     costs what the shorter wave saves.  What helps is a BN whose waves come out even (tc2_plan): 13696 x 5120 at M = 999
//     is 140 tiles of 144 tokens in one wave, 144 us, where 80 tiles of 256 found no form at all (264 us in a kernel
//     of 128-channel tiles that is gone).
//
// (b) Split-K over a thread-block cluster (gridDim.z = cluster size S = 2, 3 or 4) for shapes with fewer tiles
//     than SMs: the S CTAs of a cluster share one output tile (tile0 + blockIdx.x) and each walks 1/S of the
//     k-blocks.  The partial accumulators meet through distributed shared memory, never through global memory:
//     the tile's eight 32-token blocks are dealt out to the ranks (block b belongs to rank b % S), every CTA
//     stores its partial of a foreign block into the owner's shared memory (the operand rings are idle by then;
//     a warp's store instruction covers 512 contiguous bytes), and after one cluster barrier each owner adds
//     the S - 1 partials to its own accumulator in rank order and runs the usual epilogue for its blocks only.
// ---------------------------------------------------------------------------------------------------
constexpr int kTc2Threads = 352;   // X producer, MMA issuer, 4 + 4 transform/epilogue warps, W producer
constexpr int kTc2MaxNX = 8, kTc2MaxNW = 8, kTc2NH = 2, kTc2ND = 8;
constexpr int kTc2WBytes = 4 * kTileBytes, kTc2HBytes = 128 * 128;   // H: one half
constexpr int kTc2Smem = 224 * 1024;
constexpr int kTc2RedBlock = 256 * 128;               // one partial block: 256 channels x 32 tokens fp32
constexpr int kTc2StageBytes = 2 * 2 * kEpiStageHalves * 2;   // the epilogue's fp16 staging tiles (two per group)
// cluster mode: partial blocks received by one CTA (blocks owned, at most ceil(8 / S), x (S - 1) senders) follow
// the staging tiles at the start of the activation ring
static_assert(kTc2StageBytes + 6 * kTc2RedBlock <= kTc2Smem, "partials of S = 3 and S = 4 must fit behind the staging tiles");
static_assert(kTc2StageBytes <= kTc2NH * 2 * kTc2HBytes, "stream-K mode stages its output in the fp16 weight ring");

// Barrier of the 256 transform/epilogue threads of the 256 x 256 kernel that also ORs a predicate over them:
// every thread gets the same answer, so a decision taken on it cannot split the group before a later barrier.
template<int kThreads = 256>
__device__ __forceinline__ bool epi_bar_or(bool pred)
{
    uint32_t out;
    asm volatile(
        "{\n\t"
        ".reg .pred p, q;\n\t"
        "setp.ne.u32 q, %1, 0;\n\t"
        "bar.red.or.pred p, 3, %2, q;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}\n"
        : "=r"(out)
        : "r"((uint32_t)pred), "n"(kThreads)
        : "memory");
    return out != 0;
}

struct Tc2Smem {
    uint64_t x_full[kTc2MaxNX];
    uint64_t w_full[kTc2MaxNW], w_empty[kTc2MaxNW];
    uint64_t h_ready[kTc2NH];     // both halves of a k-block are written (8 transform warps)
    uint64_t done[kTc2ND];        // the MMAs of a k-block have completed
    uint64_t accum;               // all MMAs of a segment have completed
    uint64_t acc_free;            // the 8 epilogue warps have read the segment's accumulators
    uint32_t tmem_base;
    volatile int abort;
};

// One CTA's share of the work: `nseg` segments, processed in order.
struct Tc2Seg {
    int tile, kb0, kb1;
    bool cluster;   // a k-range of a tile shared with the other CTAs of the cluster
};

struct Tc2Work {
    int KT, G, i, tile0, nseg, cluster_kb0, cluster_kb1, cluster_tile;

    __device__ Tc2Seg seg(int p) const
    {
        Tc2Seg s;
        if (cluster_tile >= 0) {
            s.tile = cluster_tile;
            s.kb0 = cluster_kb0;
            s.kb1 = cluster_kb1;
            s.cluster = true;
            return s;
        }
        s.tile = tile0 + p * G + i;
        s.kb0 = 0;
        s.kb1 = KT;
        s.cluster = false;
        return s;
    }
};

__global__ void __launch_bounds__(kTc2Threads, 1)
gemm_tc2_kernel(const __grid_constant__ CUtensorMap tmap_x, const uint8_t* __restrict__ Bw, const __half* __restrict__ scale,
                __half* __restrict__ C, const __half* __restrict__ residual, int gate, int M, int N, int K, int bn, int nx, int nw,
                int tile0, int tile_count)
{
    // This launch covers tiles [tile0, tile0 + tile_count) of the output, numbered row-major over (token tile,
    // channel tile).
    extern __shared__ __align__(1024) uint8_t tc_dyn[];
    __shared__ Tc2Smem sm;
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(tc_dyn) + 1023) & ~(uintptr_t)1023);
    uint8_t* x_ring = base;                                   // 1024-byte aligned tiles (swizzled)
    const int x_bytes = bn * 128;                             // one k-block of activations
    uint8_t* h_ring = base + (size_t)nx * x_bytes;            // 1024-byte aligned tiles (swizzled)
    uint8_t* w_ring = h_ring + kTc2NH * 2 * kTc2HBytes;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = (int)gridDim.z, rank = (int)blockIdx.z;
    const int tiles_n = (N + 255) / 256;

    Tc2Work wk;
    wk.KT = K / kTile;
    wk.G = (int)gridDim.x;
    wk.i = (int)blockIdx.x;
    wk.cluster_tile = -1;
    wk.cluster_kb0 = wk.cluster_kb1 = 0;
    wk.tile0 = tile0;
    if (S > 1) {
        // cluster mode: the cluster is the gridDim.z CTAs of tile tile0 + blockIdx.x
        wk.cluster_tile = tile0 + (int)blockIdx.x;
        wk.cluster_kb0 = (int)((long long)wk.KT * rank / S);
        wk.cluster_kb1 = (int)((long long)wk.KT * (rank + 1) / S);
        wk.nseg = 1;
    }
    else {
        wk.nseg = (tile_count - wk.i + wk.G - 1) / wk.G;   // tiles tile0 + i, tile0 + i + G, ...
    }
    const int nseg = wk.nseg;

    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < nx; ++s) mbar_init(&sm.x_full[s], 1);
        for (int s = 0; s < kTc2ND; ++s) mbar_init(&sm.done[s], 1);
        for (int s = 0; s < nw; ++s) {
            mbar_init(&sm.w_full[s], 1);
            mbar_init(&sm.w_empty[s], 8);
        }
        for (int s = 0; s < kTc2NH; ++s) mbar_init(&sm.h_ready[s], 8);
        mbar_init(&sm.accum, 1);
        mbar_init(&sm.acc_free, 8);
        sm.abort = 0;
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = sm.tmem_base;
    bool epi_live = false;   // cluster mode: this epilogue thread has a complete accumulator to reduce

    if (warp == 0) {
        // ------------------------------------------------------------------ activation producer
        // (lane 0 and not elect.sync, here and for the weights: producers that run further ahead take the CTAs of a wave out of
        // step - 22016 x 8192 at M = 1426: 463 us, 448 so)
        if (lane == 0) {
            // (ring positions are counters: this loop is one thread's chain of dependent instructions)
            int s = 0, d = 0, it = 0;      // d: slot of done[] for k-block it - NX
            uint32_t phd = 0;
            bool ok = true;
            pdl_wait();            // the activations are the preceding kernel's output (the weights are not)
            for (int p = 0; p < nseg && ok; ++p) {
                const Tc2Seg sg = wk.seg(p);
                const int m0 = (sg.tile / tiles_n) * bn;
                for (int kb = sg.kb0; kb < sg.kb1; ++kb, ++it) {
                    if (it >= nx) {
                        if (!tc_wait(&sm.done[d], phd, &sm.abort)) {
                            ok = false;
                            break;
                        }
                        if (++d == kTc2ND) {
                            d = 0;
                            phd ^= 1;
                        }
                    }
                    mbar_arrive_expect_tx(&sm.x_full[s], (uint32_t)x_bytes);
                    tma_load_2d(x_ring + (size_t)s * x_bytes, &tmap_x, kb * kTile, m0, &sm.x_full[s]);
                    if (++s == nx) s = 0;
                }
            }
        }
    }
    else if (warp == 6) {
        // ------------------------------------------------------------------ int8 weight producer
        if (lane == 0) {
            int s = 0, it = 0;
            uint32_t ph = 1;
            bool ok = true;
            for (int p = 0; p < nseg && ok; ++p) {
                const Tc2Seg sg = wk.seg(p);
                const int n0 = (sg.tile % tiles_n) * 256;
                const int rows = n0 + 128 < N ? 4 : 2;   // tile rows of 64 channels
                const uint8_t* w0 = Bw + ((size_t)(n0 / kTile) * wk.KT + sg.kb0) * kTileBytes;
                for (int kb = sg.kb0; kb < sg.kb1; ++kb, ++it, w0 += kTileBytes) {
                    if (it >= nw && !tc_wait(&sm.w_empty[s], ph, &sm.abort)) {
                        ok = false;
                        break;
                    }
                    mbar_arrive_expect_tx(&sm.w_full[s], (uint32_t)(rows * kTileBytes));
                    uint8_t* dst = w_ring + (size_t)s * kTc2WBytes;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (i < rows) bulk_g2s(dst + i * kTileBytes, w0 + (size_t)i * wk.KT * kTileBytes, kTileBytes, &sm.w_full[s]);
                    }
                    if (++s == nw) {
                        s = 0;
                        ph ^= 1;
                    }
                }
            }
        }
    }
    else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        if (elect_one()) {
            const uint32_t idesc = umma_idesc_f16(128, bn);
            const uint64_t b_desc0 = umma_desc_sw128(smem_u32(x_ring));
            const uint64_t a_desc0 = umma_desc_sw128(smem_u32(h_ring));
            int sx = 0, sd = 0, it = 0;
            uint32_t phx = 0;
            bool ok = true;
            for (int p = 0; p < nseg && ok; ++p) {
                const Tc2Seg sg = wk.seg(p);
                const bool upper = (sg.tile % tiles_n) * 256 + 128 < N;
                // the accumulators are overwritten: the epilogue of the previous segment must have read them
                if (p > 0 && !tc_wait(&sm.acc_free, (uint32_t)((p - 1) & 1), &sm.abort)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int kb = sg.kb0; kb < sg.kb1; ++kb, ++it) {
                    const int sh = it & 1;
                    if (!tc_wait(&sm.x_full[sx], phx, &sm.abort) ||
                        !tc_wait(&sm.h_ready[sh], (uint32_t)((it >> 1) & 1), &sm.abort)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t b_desc = b_desc0 + (uint64_t)(sx * (x_bytes >> 4));
                    const uint64_t a0 = a_desc0 + (uint64_t)(sh * (2 * kTc2HBytes >> 4));
                    const uint64_t a1 = a0 + (uint64_t)(kTc2HBytes >> 4);
                    const bool acc = kb != sg.kb0;
                    umma_f16(tmem, a0, b_desc, idesc, acc);
                    umma_f16(tmem, a0 + 2, b_desc + 2, idesc, true);
                    umma_f16(tmem, a0 + 4, b_desc + 4, idesc, true);
                    umma_f16(tmem, a0 + 6, b_desc + 6, idesc, true);
                    if (upper) {
                        umma_f16(tmem + 256, a1, b_desc, idesc, acc);
                        umma_f16(tmem + 256, a1 + 2, b_desc + 2, idesc, true);
                        umma_f16(tmem + 256, a1 + 4, b_desc + 4, idesc, true);
                        umma_f16(tmem + 256, a1 + 6, b_desc + 6, idesc, true);
                    }
                    umma_commit(&sm.done[sd]);
                    if (++sd == kTc2ND) sd = 0;
                    if (++sx == nx) {
                        sx = 0;
                        phx ^= 1;
                    }
                }
                if (ok) umma_commit(&sm.accum);
            }
        }
    }
    else {
        // ------------------------------------------------------------------ transform warps, then epilogue
        // Two groups of four warps (2-5 and 7-10); group g owns the 128-channel half g of the tile: it converts
        // that half of every k-block and later runs that accumulator's epilogue.  One group alone could not
        // convert a k-block in the time the tensor core needs for it.
        const int grp = (warp >= 7) ? 1 : 0;
        const int tw = (warp - (grp ? 7 : 2)) * 32 + lane;  // 0..127 within the group
        const int lane_base = (warp & 3) * 32;              // the TMEM lanes this warp may read
        const int ch = grp * 128 + lane_base + lane;        // this thread's channel of the tile
        int sw = 0, d = 0, it = 0;     // d: slot of done[] for k-block it - NH
        uint32_t phw = 0, phd = 0;
        bool ok = true;
        for (int p = 0; p < nseg && ok; ++p) {
            const Tc2Seg sg = wk.seg(p);
            const bool mine = grp == 0 || (sg.tile % tiles_n) * 256 + 128 < N;   // (the last tile may have no upper half)
            for (int kb = sg.kb0; kb < sg.kb1; ++kb, ++it) {
                if (!tc_wait_warp(&sm.w_full[sw], phw, &sm.abort)) {
                    ok = false;
                    break;
                }
                const uint8_t* w8 = w_ring + (size_t)sw * kTc2WBytes;
                const int sh = it & 1;
                // (converted before the wait for the buffer: what follows that wait is on the chain from one k-block's
                // MMAs to the next but one's)
                uint4 o[4][2];
                const int qd = tw & 3;
                if (mine) {
#pragma unroll
                    for (int pass = 0; pass < 4; ++pass) {
                        const int r = pass * 32 + (tw >> 2);   // channel row of this half, 0..127
                        const uint4 raw = *reinterpret_cast<const uint4*>(w8 + (grp * 128 + r) * 64 + qd * 16);
                        cvt_u8x4_to_f16x4(raw.x, o[pass][0].x, o[pass][0].y);
                        cvt_u8x4_to_f16x4(raw.y, o[pass][0].z, o[pass][0].w);
                        cvt_u8x4_to_f16x4(raw.z, o[pass][1].x, o[pass][1].y);
                        cvt_u8x4_to_f16x4(raw.w, o[pass][1].z, o[pass][1].w);
                    }
                }
                if (it >= kTc2NH) {
                    if (!tc_wait_warp(&sm.done[d], phd, &sm.abort)) {
                        ok = false;
                        break;
                    }
                    if (++d == kTc2ND) {
                        d = 0;
                        phd ^= 1;
                    }
                }
                if (mine) {
                    uint8_t* wh = h_ring + (size_t)(sh * 2 + grp) * kTc2HBytes;
#pragma unroll
                    for (int pass = 0; pass < 4; ++pass) {
                        const int r = pass * 32 + (tw >> 2);
                        uint8_t* row = wh + r * 128;
                        *reinterpret_cast<uint4*>(row + (((2 * qd) ^ (r & 7)) << 4)) = o[pass][0];
                        *reinterpret_cast<uint4*>(row + (((2 * qd + 1) ^ (r & 7)) << 4)) = o[pass][1];
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                // (the int8 stage goes back only now: the stores above could not issue before their reads of it had returned)
                if (lane == 0) {
                    mbar_arrive(&sm.h_ready[sh]);
                    mbar_arrive(&sm.w_empty[sw]);
                }
                if (++sw == nw) {
                    sw = 0;
                    phw ^= 1;
                }
            }

            // ---- end of the segment: every epilogue warp gets here, also one that has left the loop above because a wait ran
            // out (the others may have finished theirs); the OR-reducing barrier gives all 256 epilogue threads the same
            // answer, whoever saw the abort flag first ----
            if (ok) tc_wait_warp(&sm.accum, (uint32_t)(p & 1), &sm.abort);
            if (epi_bar_or(sm.abort != 0)) {
                ok = false;
                break;
            }
            if (sg.cluster) {   // cluster split: the epilogue follows the cluster barriers below
                epi_live = true;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            pdl_wait();   // the output and the residual belong to the dependency chain
            const int n0 = (sg.tile % tiles_n) * 256, m0 = (sg.tile / tiles_n) * bn;
            const int m1 = min(M, m0 + bn);
            if (mine) {
                const float sc = __half2float(scale[n0 + ch]);
                __half* stage = reinterpret_cast<__half*>(h_ring) + grp * 2 * kEpiStageHalves;
                int blk = 0;
#pragma unroll 1
                for (int c0 = 0; m0 + c0 < m1; c0 += 32, ++blk) {
                    uint32_t v[32];
                    tmem_ld32(tmem + ((uint32_t)lane_base << 16) + (uint32_t)(grp * 256 + c0), v);
                    if (grp == 0) {
                        epilogue_block<1>(v, sc, stage + (blk & 1) * kEpiStageHalves, lane_base + lane, tw, C, residual, gate,
                                          m0 + c0, m1, N, n0);
                    }
                    else {
                        epilogue_block<2>(v, sc, stage + (blk & 1) * kEpiStageHalves, lane_base + lane, tw, C, residual, gate,
                                          m0 + c0, m1, N, n0 + 128);
                    }
                }
                // The staging tiles lie in this group's own part of the fp16 weight ring: its next conversions
                // must not start before every thread of the group has read its rows of the last tile.
                if (grp == 0) {
                    asm volatile("bar.sync 1, 128;" ::: "memory");
                }
                else {
                    asm volatile("bar.sync 2, 128;" ::: "memory");
                }
            }
            // accumulators read: the next segment's MMAs may overwrite them
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.acc_free);
        }
    }

    if (S > 1) {
        // ---- cluster split: reduce the S partial accumulators through distributed shared memory, then the
        // epilogue: TMEM lane = channel within the half, columns = tokens; group g takes accumulator g ----
        const bool epi_warp = (warp >= 2 && warp <= 5) || (warp >= 7 && warp <= 10);
        const int grp = (warp >= 7) ? 1 : 0;
        const int tw = (warp - (grp ? 7 : 2)) * 32 + lane;   // 0..127 within the group
        const int lane_base = (warp & 3) * 32;
        const int ch = grp * 128 + lane_base + lane;          // this thread's channel of the tile
        const int n0 = (wk.cluster_tile % tiles_n) * 256, m0 = (wk.cluster_tile / tiles_n) * bn;
        const int m1 = min(M, m0 + bn);
        if (grp == 1 && n0 + 128 >= N) epi_live = false;      // the last tile may have no upper half
        uint8_t* red = base + kTc2StageBytes;
        // All CTAs of the cluster have completed their MMAs: their rings may be overwritten.
        cooperative_groups::this_cluster().sync();
        if (epi_warp && epi_live) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            for (int b = 0; m0 + 32 * b < m1; ++b) {
                const int owner = b % S;
                if (owner == rank) continue;
                uint32_t v[32];
                tmem_ld32(tmem + ((uint32_t)lane_base << 16) + (uint32_t)(grp * 256 + 32 * b), v);
                // a partial block is laid out [4-token chunk][channel][16 bytes]: the 32 lanes of a warp store 512
                // contiguous bytes per instruction, and the owner reads them back the same way
                const int slot = (b / S) * (S - 1) + (rank < owner ? rank : rank - 1);
                const uint32_t local = smem_u32(red + (size_t)slot * kTc2RedBlock + (size_t)ch * 16);
                uint32_t remote;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(local), "r"((uint32_t)owner));
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(remote + (uint32_t)(j * 256 * 16)),
                                 "r"(v[4 * j]), "r"(v[4 * j + 1]), "r"(v[4 * j + 2]), "r"(v[4 * j + 3])
                                 : "memory");
                }
            }
        }
        // the partials of this CTA's blocks have arrived
        cooperative_groups::this_cluster().sync();
        if (epi_warp && epi_live) {
            pdl_wait();   // the output (and the residual) belong to the dependency chain
            __half* stage = reinterpret_cast<__half*>(x_ring) + grp * 2 * kEpiStageHalves;
            const float sc = __half2float(scale[n0 + ch]);
            int blk = 0;
#pragma unroll 1
            for (int b = rank; m0 + 32 * b < m1; b += S, ++blk) {
                const int c0 = 32 * b;
                uint32_t v[32];
                tmem_ld32(tmem + ((uint32_t)lane_base << 16) + (uint32_t)(grp * 256 + c0), v);
                for (int src = 0; src < S - 1; ++src) {
                    const uint8_t* p = red + (size_t)((b / S) * (S - 1) + src) * kTc2RedBlock + (size_t)ch * 16;
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        const uint4 q = *reinterpret_cast<const uint4*>(p + j * 256 * 16);
                        v[4 * j] = __float_as_uint(__uint_as_float(v[4 * j]) + __uint_as_float(q.x));
                        v[4 * j + 1] = __float_as_uint(__uint_as_float(v[4 * j + 1]) + __uint_as_float(q.y));
                        v[4 * j + 2] = __float_as_uint(__uint_as_float(v[4 * j + 2]) + __uint_as_float(q.z));
                        v[4 * j + 3] = __float_as_uint(__uint_as_float(v[4 * j + 3]) + __uint_as_float(q.w));
                    }
                }
                if (grp == 0) {
                    epilogue_block<1>(v, sc, stage + (blk & 1) * kEpiStageHalves, lane_base + lane, tw, C, residual, gate, m0 + c0, m1,
                                      N, n0);
                }
                else {
                    epilogue_block<2>(v, sc, stage + (blk & 1) * kEpiStageHalves, lane_base + lane, tw, C, residual, gate, m0 + c0, m1,
                                      N, n0 + 128);
                }
            }
        }
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled_fn()
{
    static EncodeTiledFn fn = nullptr;
    if (fn == nullptr) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess) {
            fn = reinterpret_cast<EncodeTiledFn>(p);
        }
    }
    return fn;
}

}  // namespace

// Smallest M this kernel accepts: below, the stream-K and skinny kernels serve.
constexpr int kTcMinM = 65;

// Clusters of `split` CTAs of the kernel that can be resident at once (0: that cluster size cannot be
// launched), asked of the occupancy calculator once per device and size.
static int tc2_max_clusters(int split)
{
    static int cached[64][5] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    dev &= 63;
    if (cached[dev][split] == 0) {
        const size_t smem = (size_t)kTc2Smem + 1024;
        int n = 0;
        if (cudaFuncSetAttribute(gemm_tc2_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(1, 1, split);
            cfg.blockDim = dim3(kTc2Threads, 1, 1);
            cfg.dynamicSmemBytes = smem;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = 1;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = split;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            if (cudaOccupancyMaxActiveClusters(&n, gemm_tc2_kernel, &cfg) != cudaSuccess) {
                (void)cudaGetLastError();
                n = 0;
            }
        }
        cached[dev][split] = n > 0 ? n : -1;
    }
    return cached[dev][split] > 0 ? cached[dev][split] : 0;
}

// How a shape is run (Tc2Plan): BN tokens per tile; the first `whole` tiles on persistent CTAs, the others (none, the last partial
// wave, or all) with their k-blocks split over clusters of `split` CTAs; and the modelled time.
//
// Time of a k-block of a 256 x BN tile with the machine full, measured at BN = 64 ... 256 on 4096 x 12288.  Below 128 tokens
// the conversion of the weights and the hand-overs set the pace, above it the tensor core and shared memory.
static double tc2_block_us(int bn)
{
    static const double at[9] = {0.57, 0.57, 0.58, 0.60, 0.62, 0.647, 0.69, 0.753, 0.80};   // at 0, 32, ..., 256
    const int i = bn / 32;
    return at[i] + (i < 8 ? (at[i + 1] - at[i]) * (bn % 32) / 32.0 : 0.0);
}

// The plan with the least modelled time over all BN and ways to treat the tiles that fill no wave.  A launch costs 5.5 us
// around its tiles, a tile's epilogue is not overlapped with its CTA's next tile, a cluster pays for two barriers and the
// exchange of partial sums, a second launch for its start.  When it was fitted, at M = 100 ... 4096 on the LLaMA-7B and
// Baichuan-13B shapes, the model was within 10 %; since the issuing thread is chosen by elect.sync calls below 50 us measure up to
// a fifth less (4096 x 4096, M = 100: 16.6 us for 20.9; 5120 x 13696, M = 256: 37.7 for 45.6; 11008 x 4096, M = 4096: 278 for 280).
// It knows no power limit, which makes calls of milliseconds longer by up to a sixth (8192 x 22016 at M = 8192: 2.0 ms here, 2.3
// measured) whatever the plan.
static Tc2Plan tc2_plan(int M, int N, int K)
{
    const int KT = K / kTile, G = sm_count();
    const int tiles_n = (N + 255) / 256;
    static int forced = -2;
    if (forced == -2) {
        const char* e = getenv("EET_TC2_SPLIT");
        forced = e ? atoi(e) : -1;
    }
    // (looked up once: this runs before every launch)
    int clusters[5];
    for (int sp = 2; sp <= 4; ++sp) clusters[sp] = tc2_max_clusters(sp);
    Tc2Plan best = {0, 0, 0, 1, 1e30};
    for (int bn = M < 256 ? (M + 15) / 16 * 16 : 256; bn >= 32; bn -= 16) {
        const long long tiles_ll = (long long)tiles_n * ((M + bn - 1) / bn);
        if (tiles_ll > 0x7fffffffLL) continue;
        const int tiles = (int)tiles_ll;
        const double block = tc2_block_us(bn), epilogue = 1.5 + 0.01 * bn;
        for (int sp = 1; sp <= 4; ++sp) {
            const int left = sp > 1 ? tiles % G : 0, whole = tiles - left;
            if (sp > 1 && (left == 0 || KT / sp < 4 || left > clusters[sp])) continue;
            if (forced >= 0 && sp != 1 && sp != forced) continue;
            // behind a wave of single CTAs the last few clusters of three find no room until others end and take a second turn
            // (8192 x 8192, M = 1200, 44 of them: 174 us; 12 clusters of four, BN = 256: 150)
            if (sp == 3 && whole > 0 && left > 40) continue;
            double us = 5.5 + (double)((whole + G - 1) / G) * (KT * block + epilogue);
            if (left > 0) us += (KT + sp - 1) / sp * block + epilogue + 4.0 + (whole > 0 ? 2.0 : 0.0);
            if (forced == sp && sp > 1 && whole == 0) us *= 0.1;
            if (us < best.us) best = Tc2Plan{bn, tiles, whole, sp, us};
        }
    }
    return best;
}

bool gemm_tc_supported(int M, int N, int K)
{
    return M >= kTcMinM && N % 128 == 0 && K % 64 == 0;
}

// Shapes that always go to tiles, whatever the models say: enough channels for 120 tiles of 256 x 256, or for 96 CTAs once
// their k-blocks are split over the largest cluster that fits.  A caller may rely on it: such a call needs no scratch and
// gives the same bits every time, which the stream-K kernel, whose sums meet in the order of arrival, does not.
bool gemm_tc_owns(int M, int N, int K)
{
    if (M < kTcMinM || N % 256 != 0) return false;
    const long long tiles = (long long)(N / 256) * ((M + 255) / 256);
    if (tiles >= 120) return true;
    for (int sp = 4; sp >= 2; --sp) {
        if (K / kTile / sp >= 4 && tiles <= tc2_max_clusters(sp)) return tiles * sp >= 96;
    }
    return false;
}

Tc2Plan gemm_tc_plan(int M, int N, int K)
{
    return gemm_tc_supported(M, N, K) ? tc2_plan(M, N, K) : Tc2Plan{0, 0, 0, 1, 1e30};
}

int launch_gemm_tc(const __half* A, const uint8_t* B, const __half* scale, __half* C, const __half* residual, int gate,
                   int M, int N, int K, const Tc2Plan& plan, cudaStream_t stream)
{
    EET_CHECK(gemm_tc_supported(M, N, K), "tensor-core GEMM: needs M >= 65, N %% 128 == 0, K %% 64 == 0");
    EncodeTiledFn encode = encode_tiled_fn();
    EET_CHECK(encode != nullptr, "tensor-core GEMM: cuTensorMapEncodeTiled is not available from the driver");
    static bool attr_set[64] = {};
    int dev = 0;
    EET_CUDA(cudaGetDevice(&dev));
    dev &= 63;
    const size_t smem = (size_t)kTc2Smem + 1024;
    if (!attr_set[dev]) {
        EET_CUDA(cudaFuncSetAttribute(gemm_tc2_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attr_set[dev] = true;
    }
    EET_CHECK(plan.bn > 0, "tensor-core GEMM: no plan for M=%d N=%d K=%d", M, N, K);
    CUtensorMap map;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)M};
    const cuuint64_t strides[1] = {(cuuint64_t)K * sizeof(__half)};
    const cuuint32_t box[2] = {64, (cuuint32_t)plan.bn};   // (rows past M read as zeros)
    const cuuint32_t elem[2] = {1, 1};
    const CUresult rc = encode(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half*>(A), dims, strides, box, elem,
                               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    EET_CHECK(rc == CUDA_SUCCESS, "tensor-core GEMM: cuTensorMapEncodeTiled failed with code %d", (int)rc);
    // the rings share what the fp16 weights (64 KiB) leave: as many stages of both as fit, the rest to the int8 weights
    const int x_bytes = plan.bn * 128, room = kTc2Smem - kTc2NH * 2 * kTc2HBytes;
    int nx = room / (x_bytes + kTc2WBytes);
    if (nx > kTc2MaxNX) nx = kTc2MaxNX;
    int nw = (room - nx * x_bytes) / kTc2WBytes;
    if (nw > kTc2MaxNW) nw = kTc2MaxNW;
    auto launch = [&](int tile0, int count, int grid_x, int cluster) -> cudaError_t {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3((unsigned)grid_x, 1, (unsigned)cluster);
        cfg.blockDim = dim3(kTc2Threads, 1, 1);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = stream;
        cudaLaunchAttribute attr[2];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 1;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = (unsigned)cluster;
        attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[1].val.programmaticStreamSerializationAllowed = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 2;
        return cudaLaunchKernelEx(&cfg, gemm_tc2_kernel, map, B, scale, C, residual, gate, M, N, K, plan.bn, nx, nw, tile0, count);
    };
    if (plan.whole > 0) {
        EET_CUDA(launch(0, plan.whole, plan.whole < sm_count() ? plan.whole : sm_count(), 1));
    }
    if (plan.whole < plan.tiles) {
        EET_CUDA(launch(plan.whole, plan.tiles - plan.whole, plan.tiles - plan.whole, plan.split));
    }
    return 0;
}

}  // namespace eet
