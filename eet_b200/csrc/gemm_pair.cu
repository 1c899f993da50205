// W8A16 tensor-core GEMM on CTA pairs (cta_group::2), for prompts long enough to fill the machine with its tiles: two SMs
// share one output tile of 256 channels x 2 BN tokens.
//
// The one-CTA kernel (gemm_tc.cu) is held back by what moves into and inside an SM: per 64-wide k-block of a 256 x 256 tile
// 48 KiB come from L2 (98 B/ns an SM was the most it took) and 192 KiB cross shared memory in the 1024 cycles that the
// tensor core needs.  A pair halves the weights of a CTA: each CTA converts 128 channels only, and holds one half of the
// rows of each activation tile, which the tensor cores of both read: 40 KiB from L2, 128 KiB through shared memory and
// half the conversion work for the same flops.
//
// Roles as in gemm_tc.cu, in each CTA of the pair: warp 0 activations (two tiles of BN/2 rows per k-block, signalled to the
// even CTA's barrier), warp 6 int8 weights, warps 2-5 and 7-10 conversion and epilogue (group g: accumulator g, i.e. tokens
// g BN ... of the tile, for this CTA's 128 channels), warp 1 of the even CTA issues for both.  Commits go to the barriers
// of both CTAs.  Plain TMA loads of this GPU's memory only, no multicast loads.
// The barriers between the two CTAs use the default (CTA) scope: what they guard is read and written by the tensor cores and
// the TMA engine, ordered by the proxy fence and the tensor-memory fences beside them.  With cluster-scope acquire in the
// waits a k-block took 1.25 us instead of 0.66, whatever the depth of the rings.
// Measured (a call, one-CTA kernel in brackets): 11008 x 4096 at M = 4096 246 us = 1.50 PF/s (278), at M = 2048 125 (137),
// 5120 x 13696 at M = 4096 398 (429), 4096 x 11008 at M = 2048 133 (148).
// Every wait is bounded (device status 2), tensor memory is freed on every path.
#include "common.cuh"
#include "kernels.h"

namespace eet {

namespace {

constexpr int kPrThreads = 352;
constexpr int kPrNX = 4, kPrNW = 4, kPrNH = 4, kPrND = 4;
constexpr int kPrXBytes = 256 * 128, kPrWBytes = 2 * kTileBytes, kPrHBytes = 128 * 128;
constexpr int kPrSmem = kPrNX * kPrXBytes + kPrNH * kPrHBytes + kPrNW * kPrWBytes;
static_assert(2 * 2 * kEpiStageHalves * 2 <= kPrNH * kPrHBytes, "the epilogue's staging tiles lie in the fp16 weight ring");

struct PrSmem {
    uint64_t x_full[kPrNX];                      // (even CTA) both CTAs' halves of a stage have landed
    uint64_t w_full[kPrNW], w_empty[kPrNW];
    uint64_t h_ready[kPrNH];                     // (even CTA) the fp16 weights of both CTAs are written (16 warps)
    uint64_t done[kPrND];                        // the MMAs of a k-block have completed
    uint64_t accum;                              // all MMAs of a tile have completed
    uint64_t acc_free;                           // (even CTA) the epilogue warps of both CTAs have read the accumulators
    uint32_t tmem_base;
    volatile int abort;
};

__device__ __forceinline__ uint32_t even_cta_addr(const void* p)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(r) : "r"(smem_u32(p)));
    return r;
}

__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr)
{
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* map, int x, int y, uint32_t bar_cluster_addr)
{
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
            smem_u32(smem_dst)),
        "l"(map), "r"(x), "r"(y), "r"(bar_cluster_addr)
        : "memory");
}

__device__ __forceinline__ void umma_f16_pair(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, bool accumulate)
{
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t"
        "}\n" ::"r"(d_tmem),
        "l"(a_desc), "l"(b_desc), "r"(idesc), "r"((uint32_t)accumulate)
        : "memory");
}

// arrives at the barrier of this offset in both CTAs once all MMAs issued so far have completed
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar)
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(smem_u32(bar)),
                 "h"((uint16_t)3)
                 : "memory");
}

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPrThreads, 1)
gemm_pair_kernel(const __grid_constant__ CUtensorMap tmap_x, const uint8_t* __restrict__ Bw, const __half* __restrict__ scale,
                 __half* __restrict__ C, const __half* __restrict__ residual, int gate, int M, int N, int K, int bn, int tiles)
{
    extern __shared__ __align__(1024) uint8_t pr_dyn[];
    __shared__ PrSmem sm;
    uint8_t* x_ring = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(pr_dyn) + 1023) & ~(uintptr_t)1023);
    uint8_t* h_ring = x_ring + kPrNX * kPrXBytes;
    uint8_t* w_ring = h_ring + kPrNH * kPrHBytes;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rank = (int)blockIdx.x & 1;
    const int pair = (int)blockIdx.x >> 1, pairs = (int)gridDim.x >> 1;
    const int KT = K / kTile;
    const int tiles_n = (N + 255) / 256;
    const int half_rows = bn >> 1;                 // rows of each activation tile that this CTA holds
    const int half_bytes = half_rows * 128;

    pdl_launch_dependents();
    if (threadIdx.x == 0) {
        for (int s = 0; s < kPrNX; ++s) mbar_init(&sm.x_full[s], 1);
        for (int s = 0; s < kPrND; ++s) mbar_init(&sm.done[s], 1);
        for (int s = 0; s < kPrNW; ++s) {
            mbar_init(&sm.w_full[s], 1);
            mbar_init(&sm.w_empty[s], 8);
        }
        for (int s = 0; s < kPrNH; ++s) mbar_init(&sm.h_ready[s], 16);
        mbar_init(&sm.accum, 1);
        mbar_init(&sm.acc_free, 16);
        sm.abort = 0;
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)),
                     "r"(512u)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cooperative_groups::this_cluster().sync();     // both CTAs' barriers are initialised and both have their tensor memory
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = sm.tmem_base;

    if (warp == 0) {
        // ------------------------------------------------------------------ activation producer
        if (elect_one()) {
            int s = 0, d = 0, it = 0;      // d: slot of done[] for k-block it - NX
            uint32_t phd = 0;
            bool ok = true;
            pdl_wait();            // the activations are the preceding kernel's output (the weights are not)
            for (int tile = pair; tile < tiles && ok; tile += pairs) {
                const int m0 = (tile / tiles_n) * 2 * bn + rank * half_rows;
                for (int kb = 0; kb < KT; ++kb, ++it) {
                    if (it >= kPrNX) {
                        if (!tc_wait(&sm.done[d], phd, &sm.abort)) {
                            ok = false;
                            break;
                        }
                        if (++d == kPrND) {
                            d = 0;
                            phd ^= 1;
                        }
                    }
                    if (rank == 0) mbar_arrive_expect_tx(&sm.x_full[s], (uint32_t)(4 * half_bytes));
                    const uint32_t bar = even_cta_addr(&sm.x_full[s]);
                    uint8_t* dst = x_ring + (size_t)s * kPrXBytes;
                    tma_load_2d_pair(dst, &tmap_x, kb * kTile, m0, bar);
                    tma_load_2d_pair(dst + half_bytes, &tmap_x, kb * kTile, m0 + bn, bar);
                    if (++s == kPrNX) s = 0;
                }
            }
        }
    }
    else if (warp == 6) {
        // ------------------------------------------------------------------ int8 weight producer: this CTA's 128 channels
        if (elect_one()) {
            int s = 0, it = 0;
            uint32_t ph = 1;
            bool ok = true;
            for (int tile = pair; tile < tiles && ok; tile += pairs) {
                const int n0 = (tile % tiles_n) * 256 + rank * 128;
                const uint8_t* w0 = Bw + (size_t)(n0 / kTile) * KT * kTileBytes;
                for (int kb = 0; kb < KT; ++kb, ++it, w0 += kTileBytes) {
                    if (it >= kPrNW && !tc_wait(&sm.w_empty[s], ph, &sm.abort)) {
                        ok = false;
                        break;
                    }
                    if (n0 < N) {
                        mbar_arrive_expect_tx(&sm.w_full[s], (uint32_t)kPrWBytes);
                        uint8_t* dst = w_ring + (size_t)s * kPrWBytes;
                        bulk_g2s(dst, w0, kTileBytes, &sm.w_full[s]);
                        bulk_g2s(dst + kTileBytes, w0 + (size_t)KT * kTileBytes, kTileBytes, &sm.w_full[s]);
                    }
                    else {
                        mbar_arrive(&sm.w_full[s]);   // the last tile has no upper half: nothing to load
                    }
                    if (++s == kPrNW) {
                        s = 0;
                        ph ^= 1;
                    }
                }
            }
        }
    }
    else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer of the pair
        if (rank == 0 && elect_one()) {
            const uint32_t idesc = umma_idesc_f16(256, bn);
            const uint64_t b_desc0 = umma_desc_sw128(smem_u32(x_ring));
            const uint64_t a_desc0 = umma_desc_sw128(smem_u32(h_ring));
            int sx = 0, sd = 0, it = 0, p = 0;
            uint32_t phx = 0;
            bool ok = true;
            for (int tile = pair; tile < tiles && ok; tile += pairs, ++p) {
                // the accumulators are overwritten: the epilogues of the previous tile must have read them
                if (p > 0 && !tc_wait(&sm.acc_free, (uint32_t)((p - 1) & 1), &sm.abort)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int kb = 0; kb < KT; ++kb, ++it) {
                    const int sh = it % kPrNH;
                    if (!tc_wait(&sm.x_full[sx], phx, &sm.abort) ||
                        !tc_wait(&sm.h_ready[sh], (uint32_t)((it / kPrNH) & 1), &sm.abort)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t b0 = b_desc0 + (uint64_t)(sx * (kPrXBytes >> 4));
                    const uint64_t b1 = b0 + (uint64_t)(half_bytes >> 4);
                    const uint64_t a = a_desc0 + (uint64_t)(sh * (kPrHBytes >> 4));
                    const bool acc = kb != 0;
                    umma_f16_pair(tmem, a, b0, idesc, acc);
                    umma_f16_pair(tmem, a + 2, b0 + 2, idesc, true);
                    umma_f16_pair(tmem, a + 4, b0 + 4, idesc, true);
                    umma_f16_pair(tmem, a + 6, b0 + 6, idesc, true);
                    umma_f16_pair(tmem + 256, a, b1, idesc, acc);
                    umma_f16_pair(tmem + 256, a + 2, b1 + 2, idesc, true);
                    umma_f16_pair(tmem + 256, a + 4, b1 + 4, idesc, true);
                    umma_f16_pair(tmem + 256, a + 6, b1 + 6, idesc, true);
                    umma_commit_pair(&sm.done[sd]);
                    if (++sd == kPrND) sd = 0;
                    if (++sx == kPrNX) {
                        sx = 0;
                        phx ^= 1;
                    }
                }
                if (ok) umma_commit_pair(&sm.accum);
            }
        }
    }
    else {
        // ------------------------------------------------------------------ transform warps, then epilogue
        const int grp = (warp >= 7) ? 1 : 0;
        const int tw = (warp - (grp ? 7 : 2)) * 32 + lane;  // 0..127 within the group
        const int te = grp * 128 + tw;                      // 0..255
        const int lane_base = (warp & 3) * 32;              // the TMEM lanes this warp may read
        const int ch = rank * 128 + lane_base + lane;       // this thread's channel of the tile
        const int qd = te & 3;
        uint32_t ready[kPrNH];
#pragma unroll
        for (int i = 0; i < kPrNH; ++i) ready[i] = even_cta_addr(&sm.h_ready[i]);
        const uint32_t acc_free = even_cta_addr(&sm.acc_free);
        int sw = 0, d = 0, it = 0, p = 0;     // d: slot of done[] for k-block it - NH
        uint32_t phw = 0, phd = 0;
        bool ok = true;
        for (int tile = pair; tile < tiles && ok; tile += pairs, ++p) {
            const int n0 = (tile % tiles_n) * 256;
            const bool mine = n0 + rank * 128 < N;
            for (int kb = 0; kb < KT; ++kb, ++it) {
                if (!tc_wait_warp(&sm.w_full[sw], phw, &sm.abort)) {
                    ok = false;
                    break;
                }
                const int sh = it % kPrNH;
                uint4 o[2][2];
                if (mine) {
                    const uint8_t* w8 = w_ring + (size_t)sw * kPrWBytes;
#pragma unroll
                    for (int pass = 0; pass < 2; ++pass) {
                        const int r = pass * 64 + (te >> 2);   // channel row, 0..127
                        const uint4 raw = *reinterpret_cast<const uint4*>(w8 + r * 64 + qd * 16);
                        cvt_u8x4_to_f16x4(raw.x, o[pass][0].x, o[pass][0].y);
                        cvt_u8x4_to_f16x4(raw.y, o[pass][0].z, o[pass][0].w);
                        cvt_u8x4_to_f16x4(raw.z, o[pass][1].x, o[pass][1].y);
                        cvt_u8x4_to_f16x4(raw.w, o[pass][1].z, o[pass][1].w);
                    }
                }
                if (it >= kPrNH) {
                    if (!tc_wait_warp(&sm.done[d], phd, &sm.abort)) {
                        ok = false;
                        break;
                    }
                    if (++d == kPrND) {
                        d = 0;
                        phd ^= 1;
                    }
                }
                if (mine) {
                    uint8_t* wh = h_ring + (size_t)sh * kPrHBytes;
#pragma unroll
                    for (int pass = 0; pass < 2; ++pass) {
                        const int r = pass * 64 + (te >> 2);
                        uint8_t* row = wh + r * 128;
                        *reinterpret_cast<uint4*>(row + (((2 * qd) ^ (r & 7)) << 4)) = o[pass][0];
                        *reinterpret_cast<uint4*>(row + (((2 * qd + 1) ^ (r & 7)) << 4)) = o[pass][1];
                    }
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                // (the int8 stage goes back only now: the stores above could not issue before their reads of it had returned)
                if (lane == 0) {
                    mbar_arrive_cluster(ready[sh]);
                    mbar_arrive(&sm.w_empty[sw]);
                }
                if (++sw == kPrNW) {
                    sw = 0;
                    phw ^= 1;
                }
            }

            // ---- end of the tile: every epilogue warp gets here, also one that has left the loop above because a wait ran out
            // (the others may have finished theirs); the OR-reducing barrier gives all 256 epilogue threads the same answer,
            // whoever saw the abort flag first ----
            if (ok) tc_wait_warp(&sm.accum, (uint32_t)(p & 1), &sm.abort);
            if (epi_bar_or(sm.abort != 0)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            pdl_wait();   // the output and the residual belong to the dependency chain
            if (mine) {
                const int m0 = (tile / tiles_n) * 2 * bn + grp * bn;
                const int m1 = min(M, m0 + bn);
                const float sc = __half2float(scale[n0 + ch]);
                __half* stage = reinterpret_cast<__half*>(h_ring) + grp * 2 * kEpiStageHalves;
                int blk = 0;
#pragma unroll 1
                for (int c0 = 0; m0 + c0 < m1; c0 += 32, ++blk) {
                    uint32_t v[32];
                    tmem_ld32(tmem + ((uint32_t)lane_base << 16) + (uint32_t)(grp * 256 + c0), v);
                    if (grp == 0) {
                        epilogue_block<1>(v, sc, stage + (blk & 1) * kEpiStageHalves, lane_base + lane, tw, C, residual, gate,
                                          m0 + c0, m1, N, n0 + rank * 128);
                    }
                    else {
                        epilogue_block<2>(v, sc, stage + (blk & 1) * kEpiStageHalves, lane_base + lane, tw, C, residual, gate,
                                          m0 + c0, m1, N, n0 + rank * 128);
                    }
                }
            }
            // The staging tiles lie in the fp16 weight ring, idle since the tile's last MMA: the next conversions must not
            // start before every thread has read its rows of the last block.
            asm volatile("bar.sync 3, 256;" ::: "memory");
            // accumulators read: the next tile's MMAs may overwrite them
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive_cluster(acc_free);
        }
    }

    // neither CTA may leave while the other's MMAs read its shared memory or commits arrive at its barriers
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    cooperative_groups::this_cluster().sync();
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
    }
}

// CTA pairs that can be resident at once, asked of the occupancy calculator once per device.
int max_pairs()
{
    static int cached[64] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    dev &= 63;
    if (cached[dev] == 0) {
        const size_t smem = (size_t)kPrSmem + 1024;
        int n = 0;
        if (cudaFuncSetAttribute(gemm_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(2, 1, 1);
            cfg.blockDim = dim3(kPrThreads, 1, 1);
            cfg.dynamicSmemBytes = smem;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = 2;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = 1;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            if (cudaOccupancyMaxActiveClusters(&n, gemm_pair_kernel, &cfg) != cudaSuccess) {
                (void)cudaGetLastError();
                n = 0;
            }
        }
        cached[dev] = n > 0 ? n : -1;
    }
    return cached[dev] > 0 ? cached[dev] : 0;
}

}  // namespace

// Token tile (per accumulator) and modelled time in microseconds; bn = 0 where the kernel does not take the shape.
PairPlan gemm_pair_plan(int M, int N, int K)
{
    PairPlan best = {0, 1e30};
    const int pairs = max_pairs();
    if (M < 256 || N % 128 != 0 || K % 64 != 0 || pairs == 0) return best;
    const int KT = K / kTile, tiles_n = (N + 255) / 256;
    for (int bn = 256; bn >= 128; bn -= 16) {
        const long long tiles = (long long)tiles_n * ((M + 2 * bn - 1) / (2 * bn));
        if (tiles > 0x3fffffffLL) continue;
        // a k-block with the machine full: fitted to 110 calls of 256 to 4096 rows at K from 4096 on, the smallest that was measured;
        // below, the constants from before the single threads were chosen by elect.sync.  Those are too long by 13 to 24 % (1024
        // x 4096 at M = 1024: 13.8 us for 18.1; 3072 x 8192 at M = 2048: 78 for 90), as the one-CTA kernel's are by 3 to 18 %
        // (15.1 for 18.2; 83 for 88)
        const double block = K >= 4096 ? 0.60 + 0.0018 * (bn - 192) : 0.65 + 0.00203 * (bn - 192);
        const double us = 7.0 + (double)((tiles + pairs - 1) / pairs) * (KT * block + 1.5 + 0.01 * bn);
        if (us < best.us) best = PairPlan{bn, us};
    }
    return best;
}

int launch_gemm_pair(const __half* A, const uint8_t* B, const __half* scale, __half* C, const __half* residual, int gate,
                     int M, int N, int K, int bn, cudaStream_t stream)
{
    EncodeTiledFn encode = encode_tiled_fn();
    EET_CHECK(encode != nullptr, "tensor-core GEMM: cuTensorMapEncodeTiled is not available from the driver");
    EET_CHECK(bn >= 32 && bn <= 256 && bn % 16 == 0 && max_pairs() > 0, "tensor-core GEMM: no CTA pairs for a token tile of %d", bn);
    CUtensorMap map;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)M};
    const cuuint64_t strides[1] = {(cuuint64_t)K * sizeof(__half)};
    const cuuint32_t box[2] = {64, (cuuint32_t)(bn / 2)};   // (rows past M read as zeros)
    const cuuint32_t elem[2] = {1, 1};
    const CUresult rc = encode(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half*>(A), dims, strides, box, elem,
                               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    EET_CHECK(rc == CUDA_SUCCESS, "tensor-core GEMM: cuTensorMapEncodeTiled failed with code %d", (int)rc);
    const int tiles = (N + 255) / 256 * ((M + 2 * bn - 1) / (2 * bn));
    const int pairs = tiles < max_pairs() ? tiles : max_pairs();
    EET_CUDA(launch_pdl(gemm_pair_kernel, dim3((unsigned)(2 * pairs)), dim3(kPrThreads), (size_t)kPrSmem + 1024, stream, map, B,
                        scale, C, residual, gate, M, N, K, bn, tiles));
    return 0;
}

}  // namespace eet
