// W8A16 tensor-core GEMM with the weights as an operand in TENSOR MEMORY, for 17 rows on (a batch of sequences in decode, a short
// prompt) up to the long prompts that CTA pairs serve better: C[M,N] = A[M,K] (fp16) x dequant(B), B in the W8T64 layout,
// per-channel fp16 scale, optional residual or gated activation, one launch, no scratch, the same bits every time.
//
// Replaces the reference's fpA_intB GEMM at these sizes (kernel cutlass_extensions/.../gemm/kernel/fpA_intB_gemm.h:60-486).
//
// What bounds it and why it looks like this.  The tile kernel of gemm_tc.cu converts the int8 weights into shared memory, and there
// per 64-wide k-block of 256 channels x BN tokens 768 + 3 BN cycles of shared-memory traffic meet 4 BN cycles of tensor core:
// 1100 cycles at BN = 112.  Converted into tensor memory (tcgen05.st, lane = channel), where the MMA reads its A operand, the
// traffic is 256 + 3 BN.  What bounds the loop then are the conversion warps (two instructions for four weights on half-rate
// pipes) and an MMA's 70 to 80 cycles with few tokens: 470 to 600 cycles a k-block up to 128 tokens, 760 at 192; with one
// token tile that is also about what HBM delivers to 129 SMs.
//  * warp 0 activations (2-D tensor map, 128-byte swizzle, one k-block a stage), warp 2 int8 weights (4-D tensor map, one copy a
//    unit of one or two k-blocks; the 64-byte swizzle spares the conversion a permutation of its registers), warp 1 issues, two
//    sets of eight warps convert alternate units and run the epilogue.
//  * Tiles that fill no wave are split along K over a cluster of up to eight CTAs.  Their partial sums meet through
//    distributed shared memory (about 20 bytes a cycle and SM, whether stored or copied: a third of the kernel at 100 rows),
//    announced by transaction barriers instead of cluster-wide ones.
//  * Otherwise persistent CTAs take tiles i, i + G, ... ordered so that CTAs side by side share a row of weight tiles.
// Measured, a call in a chain of calls (before: stream-K units and a finishing launch, or tiles with the weights in shared memory):
// 4096 x 11008: M = 17 12.8 us (16.7), 64 13.3 (19.1), 100 16.5 (22.8), 192 22.1 (24.8), 320 29 (40), 512 38 (48);
// 8192 x 8192: M = 64 16.7 (22.0), 128 21.4 (29.7); 4096 x 4096: M = 32 8.7 (11.2), 256 14.9 (20.6);
// 13696 x 5120 at M = 1024: 107 (152).
// Not taken: three sets of conversion warps (instruction issue is what they share: 850 cycles a k-block); one set and two CTAs per SM
// (4096 x 11008, M = 32: 14.9 us, 13.0 here); partial sums through the copy engine (16.9 us at M = 100, 16.5 as they are).
// Every wait is bounded (device status 2), tensor memory is freed on every path, and the CTAs of a cluster end together.
#include "common.cuh"
#include "kernels.h"

namespace eet {

namespace {

constexpr int kTsSets = 2;                            // sets of eight conversion warps
constexpr int kTsThreads = 96 + 256 * kTsSets;        // activation producer, MMA issuer, weight producer, conversion and epilogue
constexpr int kTsMaxNX = 8, kTsMaxNW = 10, kTsMaxNA = 6, kTsND = 8;
constexpr int kTsWBlock = 4 * kTileBytes;             // 256 channels x 64 k, int8
// tokens of a piece of the exchange between the CTAs of a cluster: few tokens are spread over more ranks
__host__ __device__ constexpr int ts_chunk(int bn) { return bn <= 64 ? 8 : 16; }
constexpr int kTsStageHalves = 16 * 128;              // staging of a group of 128 threads in the epilogue: 16 tokens, or twice 8
constexpr int kTsStageBytes = 2 * kTsSets * kTsStageHalves * 2;
constexpr int kTsMaxSplit = 8;
// k-blocks of a unit: two where two buffers of fp16 weights fit tensor memory beside the accumulators
__host__ __device__ constexpr int ts_unit(int bn) { return bn <= 128 ? 2 : 1; }
constexpr int kTsSmem = 224 * 1024, kTsCols = 512;

struct TsSmem {
    uint64_t x_full[kTsMaxNX];
    uint64_t w_full[kTsMaxNW], w_empty[kTsMaxNW];   // int8 tiles landed / read by the eight warps of a set
    uint64_t a_ready[kTsMaxNA];                     // fp16 weights of a k-block written (eight warps)
    uint64_t done[kTsND];                           // the MMAs of a k-block have completed
    uint64_t accum;                                 // all MMAs of a tile have completed
    uint64_t acc_free;                              // the epilogue warps have read the tile's accumulators
    uint64_t peers_done;                            // the MMAs of all other CTAs of the cluster have completed
    uint64_t partials;                              // their partial sums of this CTA's chunks have arrived
    uint32_t tmem_base;
    volatile int abort;
};

struct TsArgs {
    const uint8_t* B;
    const __half* scale;
    __half* C;
    const __half* residual;
    int gate, M, N, K;
    int bn, nx, nw, na, acc_cols;   // tokens per tile, stages, fp16 buffers, columns of an accumulator
    int tiles;                      // numbered row-major over (channel tile, token tile): CTAs side by side share the weights of a tile row
    int stream;                     // the weights are read once: let the L2 drop them
    uint32_t zero;                  // 0, see after_reads
};

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&v)[8])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// o <- o + res, or gated_silu(res, o): then this GEMM is the up projection of a gated FFN and `res` the gate projection
__device__ __forceinline__ void ts_combine(uint4& o, const uint4& res, int gate)
{
    __half2* oh = reinterpret_cast<__half2*>(&o);
    const __half2* rh = reinterpret_cast<const __half2*>(&res);
#pragma unroll
    for (int e = 0; e < 4; ++e) oh[e] = gate ? gated_silu2(rh[e], oh[e]) : __hadd2(oh[e], rh[e]);
}

__device__ __forceinline__ uint32_t cluster_addr32(uint32_t local, int rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(local), "r"(rank));
    return r;
}
__device__ __forceinline__ uint32_t cluster_addr(const void* p, int rank) { return cluster_addr32(smem_u32(p), rank); }

// This warp's part of a cluster-wide barrier; the CTAs of the cluster are past it when cluster_wait returns.
__device__ __forceinline__ void cluster_arrive()
{
    __syncwarp();
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
}
__device__ __forceinline__ void cluster_wait()
{
    __syncwarp();
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}

__device__ __forceinline__ void prefetch_map(const CUtensorMap* map)
{
    asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// A unit (k-blocks kb ... of the box) of 256 channels: W8T64 tiles, each 64 rows of 64 bytes, whose 16-byte pieces land in the order of the
// 64-byte swizzle (piece j of row r at j ^ (r / 2 % 4)): a warp that reads a piece of 32 rows meets no bank twice.
__device__ __forceinline__ void tma_load_w(void* smem_dst, const CUtensorMap* map, int kb, int tile_row, uint64_t policy, uint64_t* bar)
{
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %2, %3, %4}], [%5], %6;" ::"r"(
            smem_u32(smem_dst)),
        "l"(map), "r"(0), "r"(kb), "r"(tile_row), "r"(smem_u32(bar)), "l"(policy)
        : "memory");
}

// T tokens x 128 channels of the output by the 128 threads of a group: see epilogue_block.  One staging tile, so the caller
// keeps the group from writing it before everybody has read it.
template<int T>
__device__ __forceinline__ void ts_store(const uint32_t (&v)[T], float sc, __half* stage, int channel, int tw, int bar_id, __half* C,
                                         const __half* residual, int gate, int m_first, int M, int N, int n_first)
{
#pragma unroll
    for (int j = 0; j < T; ++j) stage[j * 128 + channel] = __float2half(__uint_as_float(v[j]) * sc);
    asm volatile("bar.sync %0, 128;" ::"r"(bar_id) : "memory");
    uint4 res[T / 8];
#pragma unroll
    for (int i = 0; i < T / 8; ++i) {
        const int idx = tw + i * 128, row = idx >> 4, ch8 = idx & 15;
        res[i] = make_uint4(0u, 0u, 0u, 0u);
        if (residual != nullptr && m_first + row < M) {
            res[i] = *reinterpret_cast<const uint4*>(residual + (size_t)(m_first + row) * N + n_first + ch8 * 8);
        }
    }
#pragma unroll
    for (int i = 0; i < T / 8; ++i) {
        const int idx = tw + i * 128, row = idx >> 4, ch8 = idx & 15;
        if (m_first + row < M) {
            uint4 o = *reinterpret_cast<const uint4*>(stage + row * 128 + ch8 * 8);
            if (residual != nullptr) {
                ts_combine(o, res[i], gate);
            }
            *reinterpret_cast<uint4*>(C + (size_t)(m_first + row) * N + n_first + ch8 * 8) = o;
        }
    }
}

template<int T>
__device__ __forceinline__ void tmem_ld_tokens(uint32_t taddr, uint32_t (&v)[T]);
template<>
__device__ __forceinline__ void tmem_ld_tokens<8>(uint32_t taddr, uint32_t (&v)[8]) { tmem_ld8(taddr, v); }
template<>
__device__ __forceinline__ void tmem_ld_tokens<16>(uint32_t taddr, uint32_t (&v)[16]) { tmem_ld16(taddr, v); }

// The S partial accumulators of a cluster meet through distributed shared memory.  The tile's tokens are dealt out to the ranks in
// chunks of T (chunk q belongs to rank q % S).  A CTA whose MMAs have completed (`summed`) has told the others that its rings may
// be overwritten; each stores its partials of foreign chunks into their owners' and, once all bytes of its own chunks have
// arrived, adds them to its own sums in rank order and finishes its chunks.  A CTA whose wait for its MMAs or for the others ran
// out stores nothing into anybody; who waits for its partials gives up in turn.  Behind its last store every thread arrives at
// the cluster barrier, which the kernel waits for before it ends: no CTA leaves while another may still address it.
template<int T>
__device__ __forceinline__ void ts_exchange(TsSmem& sm, const TsArgs& a, uint8_t* base, uint8_t* stage_base, uint32_t tmem, float sc, int warp,
                                            int lane, int S, int rank, int n0, int m0, bool summed)
{
    constexpr int kBytes = 256 * T * 4;   // the partial sums of a chunk
    const int set = (warp - 3) >> 3, grp = ((warp - 3) >> 2) & 1;
    if (warp < 3 || (grp == 1 && n0 + 128 >= a.N)) {   // (the last tile may have no upper half)
        cluster_arrive();
        return;
    }
    const int tw = ((warp - 3) & 3) * 32 + lane, lane_base = (warp & 3) * 32, r = lane_base + lane;
    const int chunks = (min(a.M, m0 + a.bn) - m0 + T - 1) / T;
    const uint32_t acc = tmem + ((uint32_t)lane_base << 16) + (uint32_t)(grp * a.acc_cols);
    const uint32_t mine = (uint32_t)(grp * 128 + r) * 16;     // this thread's channel in a chunk: [4 tokens][channel][16 bytes]
    pdl_wait();   // the output (and the residual) belong to the dependency chain
    // the 16-byte pieces of a chunk that this thread stores, and their residual, requested early
    const int col = n0 + grp * 128 + (tw & 15) * 8;
    uint4 res[T / 8];
    auto fetch = [&](int q) {
#pragma unroll
        for (int i = 0; i < T / 8; ++i) {
            const int m = m0 + q * T + (tw >> 4) + i * 8;
            res[i] = a.residual != nullptr && q < chunks && m < a.M ? *reinterpret_cast<const uint4*>(a.residual + (size_t)m * a.N + col)
                                                                    : make_uint4(0u, 0u, 0u, 0u);
        }
    };
    fetch(rank + S * set);
    const bool send = tc_wait_warp(&sm.peers_done, 0, &sm.abort) && summed;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t local = smem_u32(base) + mine, bar_local = smem_u32(&sm.partials);
    int owner = set, turn = 0;   // chunk q = turn * S + owner
    for (int q = set; q < chunks && send; q += kTsSets, owner += kTsSets) {
        while (owner >= S) {
            owner -= S;
            ++turn;
        }
        if (owner == rank) continue;
        uint32_t v[T];
        tmem_ld_tokens<T>(acc + (uint32_t)(q * T), v);
        const uint32_t to = cluster_addr32(local + (uint32_t)((turn * (S - 1) + (rank < owner ? rank : rank - 1)) * kBytes), owner);
        const uint32_t bar = cluster_addr32(bar_local, owner);
#pragma unroll
        for (int j = 0; j < T / 4; ++j) {   // (the 32 lanes of a warp store 512 contiguous bytes)
            asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, %4}, [%5];" ::"r"(
                             to + (uint32_t)(j * 256 * 16)),
                         "r"(v[4 * j]), "r"(v[4 * j + 1]), "r"(v[4 * j + 2]), "r"(v[4 * j + 3]), "r"(bar)
                         : "memory");
        }
    }
    cluster_arrive();
    // the partials of this CTA's chunks have arrived
    if (rank < chunks) tc_wait_warp(&sm.partials, 0, &sm.abort);
    __half* stage = reinterpret_cast<__half*>(stage_base) + (set * 2 + grp) * kTsStageHalves;
    const int bar_id = 4 + set * 2 + grp;
    turn = set;
#pragma unroll 1
    for (int q = rank + S * set; q < chunks; q += S * kTsSets, turn += kTsSets) {
        uint32_t v[T];
        tmem_ld_tokens<T>(acc + (uint32_t)(q * T), v);
        const uint8_t* p = base + (size_t)(turn * (S - 1)) * kBytes + mine;
#pragma unroll 2
        for (int src = 0; src < S - 1; ++src, p += kBytes) {
#pragma unroll
            for (int j = 0; j < T / 4; ++j) {
                const uint4 w = *reinterpret_cast<const uint4*>(p + j * 256 * 16);
                v[4 * j] = __float_as_uint(__uint_as_float(v[4 * j]) + __uint_as_float(w.x));
                v[4 * j + 1] = __float_as_uint(__uint_as_float(v[4 * j + 1]) + __uint_as_float(w.y));
                v[4 * j + 2] = __float_as_uint(__uint_as_float(v[4 * j + 2]) + __uint_as_float(w.z));
                v[4 * j + 3] = __float_as_uint(__uint_as_float(v[4 * j + 3]) + __uint_as_float(w.w));
            }
        }
        if (turn != set) asm volatile("bar.sync %0, 128;" ::"r"(bar_id) : "memory");   // the staging tile has been read
#pragma unroll
        for (int j = 0; j < T; ++j) stage[j * 128 + r] = __float2half(__uint_as_float(v[j]) * sc);
        asm volatile("bar.sync %0, 128;" ::"r"(bar_id) : "memory");
#pragma unroll
        for (int i = 0; i < T / 8; ++i) {
            const int m = m0 + q * T + (tw >> 4) + i * 8;
            if (m < a.M) {
                uint4 o = *reinterpret_cast<const uint4*>(stage + (tw + i * 128) * 8);
                if (a.residual != nullptr) ts_combine(o, res[i], a.gate);
                *reinterpret_cast<uint4*>(a.C + (size_t)m * a.N + col) = o;
            }
        }
        fetch(q + S * kTsSets);
    }
}

template<int kUnit>
__global__ void __launch_bounds__(kTsThreads, 1)
gemm_ts_kernel(const __grid_constant__ CUtensorMap tmap_x, const __grid_constant__ CUtensorMap tmap_w, const __grid_constant__ TsArgs a)
{
    extern __shared__ __align__(1024) uint8_t ts_dyn[];
    __shared__ TsSmem sm;
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(ts_dyn) + 1023) & ~(uintptr_t)1023);
    const int x_bytes = a.bn * 128;                           // one k-block of activations, 1024-byte aligned (swizzled)
    uint8_t* x_ring = base;
    uint8_t* w_ring = base + (size_t)a.nx * x_bytes;
    uint8_t* stage_base = base + kTsSmem - kTsStageBytes;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = (int)gridDim.z, rank = (int)blockIdx.z;
    const int tiles_m = (a.M + a.bn - 1) / a.bn;
    const int KU = (a.K / kTile + kUnit - 1) / kUnit;   // (k-blocks past the last read as zeros on both sides)
    // one tile shared by the S CTAs of a cluster, or tiles i, i + G, ... of a CTA
    const int u0 = S > 1 ? (int)((long long)KU * rank / S) : 0, u1 = S > 1 ? (int)((long long)KU * (rank + 1) / S) : KU;
    const int first = (int)blockIdx.x, last = a.tiles, step = (int)gridDim.x;

    pdl_launch_dependents();
    if (warp == 0 && elect_one()) {
        for (int s = 0; s < a.nx; ++s) mbar_init(&sm.x_full[s], 1);
        for (int s = 0; s < kTsND; ++s) mbar_init(&sm.done[s], 1);
        for (int s = 0; s < a.na; ++s) mbar_init(&sm.a_ready[s], 8);
        mbar_init(&sm.accum, 1);
        mbar_init(&sm.acc_free, 8 * kTsSets);
        mbar_init(&sm.peers_done, S > 1 ? S - 1 : 1);
        mbar_init(&sm.partials, 1);
        sm.abort = 0;
        mbar_fence_init();
        if (S > 1) {
            const int m0 = (first % tiles_m) * a.bn, T = ts_chunk(a.bn), chunks = (min(a.M, m0 + a.bn) - m0 + T - 1) / T;
            const int owned = rank < chunks ? (chunks - rank + S - 1) / S : 0, channels = (first / tiles_m) * 256 + 128 < a.N ? 256 : 128;
            mbar_arrive_expect_tx(&sm.partials, (uint32_t)(owned * (S - 1) * channels * T * 4));
        }
    }
    // the weights, constant inputs: the first ring is requested before the block-wide barrier and the tensor-memory allocation
    uint64_t w_policy = 0;
    int w_it = 0;
    if (warp == 2 && elect_one()) {
        prefetch_map(&tmap_w);
        prefetch_map(&tmap_x);
        for (int s = 0; s < a.nw; ++s) {
            mbar_init(&sm.w_full[s], 1);
            mbar_init(&sm.w_empty[s], 8);
        }
        mbar_fence_init();
        if (a.stream) asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(w_policy));
        else asm volatile("createpolicy.fractional.L2::evict_normal.b64 %0, 1.0;" : "=l"(w_policy));
        for (; w_it < a.nw && u0 + w_it < u1; ++w_it) {
            mbar_arrive_expect_tx(&sm.w_full[w_it], (uint32_t)(kUnit * kTsWBlock));
            tma_load_w(w_ring + (size_t)w_it * (kUnit * kTsWBlock), &tmap_w, (u0 + w_it) * kUnit, (first / tiles_m) * 4, w_policy, &sm.w_full[w_it]);
        }
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&sm.tmem_base)),
                     "n"(kTsCols)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (S > 1) cluster_arrive();   // waited for before the first remote access
    const uint32_t tmem = sm.tmem_base;
    const uint32_t a_cols = tmem + 2 * (uint32_t)a.acc_cols;   // the fp16 weights: [buffer][half of the channels][32 columns]
    float sc = 0.f;          // conversion warps: the scale of this thread's channel
    bool summed = false;     // and whether all MMAs of the last tile have completed, the same for a warp

    if (warp == 0) {
        // ------------------------------------------------------------------ activation producer
        if (elect_one()) {
            int s = 0, it = 0;     // k-blocks, counted over the tiles
            bool ok = true;
            pdl_wait();            // the activations are the preceding kernel's output (the weights are not)
            for (int tile = first; tile < last && ok; tile += step) {
                const int m0 = (tile % tiles_m) * a.bn;
                for (int kb = u0 * kUnit; kb < u1 * kUnit; ++kb, ++it) {
                    const int d = it - a.nx;   // the k-block that had this stage before
                    if (d >= 0 && !tc_wait(&sm.done[(d / kUnit) & (kTsND - 1)], (uint32_t)(d / kUnit / kTsND) & 1u, &sm.abort)) {
                        ok = false;
                        break;
                    }
                    mbar_arrive_expect_tx(&sm.x_full[s], (uint32_t)x_bytes);
                    tma_load_2d(x_ring + (size_t)s * x_bytes, &tmap_x, kb * kTile, m0, &sm.x_full[s]);
                    if (++s == a.nx) s = 0;
                }
            }
        }
    }
    else if (warp == 2) {
        // ------------------------------------------------------------------ int8 weight producer
        if (elect_one()) {
            int s = w_it == a.nw ? 0 : w_it;
            uint32_t ph = w_it == a.nw ? 0 : 1;      // parity of the slot's previous round
            bool ok = true;
            for (int tile = first, skip = w_it; tile < last && ok; tile += step, skip = 0) {
                const int row = (tile / tiles_m) * 4;   // (tile rows past the last of N read as zeros)
                for (int u = u0 + skip; u < u1; ++u, ++w_it) {
                    if (w_it >= a.nw && !tc_wait(&sm.w_empty[s], ph, &sm.abort)) {
                        ok = false;
                        break;
                    }
                    mbar_arrive_expect_tx(&sm.w_full[s], (uint32_t)(kUnit * kTsWBlock));
                    tma_load_w(w_ring + (size_t)s * (kUnit * kTsWBlock), &tmap_w, u * kUnit, row, w_policy, &sm.w_full[s]);
                    if (++s == a.nw) {
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
            const uint32_t idesc = umma_idesc_f16(128, a.bn);
            const uint64_t b_desc0 = umma_desc_sw128(smem_u32(x_ring));
            int sx = 0, sa = 0, it = 0, p = 0;
            uint32_t phx = 0, pha = 0;
            bool ok = true;
            for (int tile = first; tile < last && ok; tile += step, ++p) {
                const bool upper = (tile / tiles_m) * 256 + 128 < a.N;
                // the accumulators are overwritten: the epilogue of the previous tile must have read them
                if (p > 0 && !tc_wait(&sm.acc_free, (uint32_t)((p - 1) & 1), &sm.abort)) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int u = u0; u < u1; ++u, ++it) {
                    if (!tc_wait(&sm.a_ready[sa], pha, &sm.abort)) {
                        ok = false;
                        break;
                    }
                    const uint32_t a0 = a_cols + (uint32_t)(sa * kUnit * 64), d1 = tmem + (uint32_t)a.acc_cols;
#pragma unroll
                    for (int i = 0; i < kUnit; ++i) {
                        if (!tc_wait(&sm.x_full[sx], phx, &sm.abort)) {
                            ok = false;
                            break;
                        }
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        // 16 reduction indices per MMA: 8 columns of the weights, 32 bytes along the swizzled row of the activations
                        const uint64_t b = b_desc0 + (uint64_t)(sx * (x_bytes >> 4));
#pragma unroll
                        for (int k = 0; k < 4; ++k) umma_f16_ts(tmem, a0 + i * 64 + k * 8, b + 2 * k, idesc, u != u0 || i + k > 0);
                        if (upper) {
#pragma unroll
                            for (int k = 0; k < 4; ++k) umma_f16_ts(d1, a0 + i * 64 + 32 + k * 8, b + 2 * k, idesc, u != u0 || i + k > 0);
                        }
                        if (++sx == a.nx) {
                            sx = 0;
                            phx ^= 1;
                        }
                    }
                    if (!ok) break;
                    umma_commit(&sm.done[it & (kTsND - 1)]);
                    if (++sa == a.na) {
                        sa = 0;
                        pha ^= 1;
                    }
                }
                if (ok) umma_commit(&sm.accum);
            }
        }
    }
    else {
        // ------------------------------------------------------------------ conversion warps, then epilogue
        // Sets of eight warps take the units in turn; in a set four warps (one of each quarter of the TMEM lanes) for each
        // half of the channels, one thread per channel.
        const int set = (warp - 3) >> 3;
        const int grp = ((warp - 3) >> 2) & 1;
        const int tw = ((warp - 3) & 3) * 32 + lane;        // 0..127 within the group
        const int lane_base = (warp & 3) * 32;              // the TMEM lanes this warp may access
        const int r = lane_base + lane;                     // this thread's channel of its half
        const int sxr = (lane >> 1) & 3;                    // see tma_load_w
        const uint8_t* row0 = w_ring + (grp * 2 + (r >> 6)) * (kUnit * kTileBytes) + (r & 63) * 64;   // [tile row][k-block][row]
        const uint32_t a_mine = a_cols + ((uint32_t)lane_base << 16) + (uint32_t)(grp * 32);
        __half* stage = reinterpret_cast<__half*>(stage_base) + (set * 2 + grp) * kTsStageHalves;
        const int bar_id = 4 + set * 2 + grp;
        // Slots of unit `it`, the next of this set (counted over the tiles).  The number of weight stages is a multiple of the
        // sets: a stage belongs to one of them, which waits for every one of its phases (a set that skipped one could not
        // tell the phase before from the one after).
        int sw = set, sa = set, it = set, end = 0, p = 0;
        uint32_t phw = 0;
        bool ok = true;
        for (int tile = first; tile < last && ok; tile += step, ++p) {
            const int n0 = (tile / tiles_m) * 256;
            const bool mine = grp == 0 || n0 + 128 < a.N;   // (the last tile may have no upper half)
            sc = mine ? __half2float(a.scale[n0 + grp * 128 + r]) : 0.f;   // (constant like the weights: no wait)
            end += u1 - u0;
            for (; it < end; it += kTsSets) {
                if (!tc_wait_warp(&sm.w_full[sw], phw, &sm.abort)) {
                    ok = false;
                    break;
                }
                const uint8_t* row = row0 + sw * (kUnit * kTsWBlock);
                bool live = true;
#pragma unroll
                for (int i = 0; i < kUnit; ++i) {
                    uint32_t h[32], words = 0;
                    if (mine) {
                        uint4 c[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            c[j] = *reinterpret_cast<const uint4*>(row + i * kTileBytes + ((j ^ sxr) << 4));
                            words ^= c[j].x;
                        }
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            cvt_u8x4_to_f16x4(c[j].x, h[8 * j + 0], h[8 * j + 1]);
                            cvt_u8x4_to_f16x4(c[j].y, h[8 * j + 2], h[8 * j + 3]);
                            cvt_u8x4_to_f16x4(c[j].z, h[8 * j + 4], h[8 * j + 5]);
                            cvt_u8x4_to_f16x4(c[j].w, h[8 * j + 6], h[8 * j + 7]);
                        }
                    }
                    if (i == kUnit - 1) {
                        // the int8 stage is free again as soon as the bytes are in registers
                        __syncwarp();
                        if (lane == 0) mbar_arrive_after(&sm.w_empty[sw], after_reads(words, a.zero));
                    }
                    if (i == 0) {
                        const int d = it - a.na;
                        if (d >= 0) live = tc_wait_warp(&sm.done[d & (kTsND - 1)], (uint32_t)(d / kTsND) & 1u, &sm.abort);
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    }
                    if (mine && live) tmem_st32_async(a_mine + (uint32_t)((sa * kUnit + i) * 64), h);
                }
                if (!live) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&sm.a_ready[sa]);
                sw += kTsSets;
                if (sw >= a.nw) {
                    sw -= a.nw;
                    phw ^= 1;
                }
                sa += kTsSets;
                if (sa >= a.na) sa -= a.na;
            }

            // ---- end of the tile: every epilogue warp gets here, also one that has left the loop above because a wait ran out
            // (the others may have finished theirs); the OR-reducing barrier gives all epilogue threads the same answer, whoever
            // saw the abort flag first ----
            summed = ok && tc_wait_warp(&sm.accum, (uint32_t)(p & 1), &sm.abort);
            if (S > 1) break;   // the exchange and the epilogue follow below, whatever ran out
            if (epi_bar_or<256 * kTsSets>(sm.abort != 0)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            pdl_wait();   // the output and the residual belong to the dependency chain
            if (mine) {
                const int m0 = (tile % tiles_m) * a.bn, m1 = min(a.M, m0 + a.bn);
#pragma unroll 1
                for (int c0 = 16 * set; m0 + c0 < m1; c0 += 16 * kTsSets) {
                    uint32_t v[16];
                    tmem_ld16(tmem + ((uint32_t)lane_base << 16) + (uint32_t)(grp * a.acc_cols + c0), v);
                    asm volatile("bar.sync %0, 128;" ::"r"(bar_id) : "memory");   // the staging tile has been read
                    ts_store<16>(v, sc, stage, r, tw, bar_id, a.C, a.residual, a.gate, m0 + c0, m1, a.N, n0 + grp * 128);
                }
            }
            // accumulators read: the next tile's MMAs may overwrite them
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(&sm.acc_free);
        }
    }

    if (S > 1) {
        cluster_wait();   // (long since complete: all have started)
        if (warp == 3 && summed && lane < S && lane != rank) mbar_arrive_cluster(cluster_addr(&sm.peers_done, lane));
        const int n0 = (first / tiles_m) * 256, m0 = (first % tiles_m) * a.bn;
        if (ts_chunk(a.bn) == 8) ts_exchange<8>(sm, a, base, stage_base, tmem, sc, warp, lane, S, rank, n0, m0, summed);
        else ts_exchange<16>(sm, a, base, stage_base, tmem, sc, warp, lane, S, rank, n0, m0, summed);
        cluster_wait();   // nobody will address this CTA's memory any more
    }

    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (sm.abort) {
        // a wait has run out: give copies and MMAs that are still in flight the time to end before their memory goes
        for (int i = 0; i < 100; ++i) __nanosleep(1000);
    }
    if (warp == 1) {
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(kTsCols) : "memory");
    }
}

// Whether the partial sums that a CTA of a cluster of S receives fit the rings.
bool ts_fits(int bn, int S)
{
    const int T = ts_chunk(bn), chunks = (bn + T - 1) / T;
    return (chunks + S - 1) / S * (S - 1) * 256 * T * 4 <= kTsSmem - kTsStageBytes;
}

template<int kUnit>
int launch_ts(const __half* A, TsArgs a, int split, cudaStream_t stream)
{
    EncodeTiledFn encode = encode_tiled_fn();
    EET_CHECK(encode != nullptr, "tensor-core GEMM: cuTensorMapEncodeTiled is not available from the driver");
    static bool attr_set[64] = {};
    int dev = 0;
    EET_CUDA(cudaGetDevice(&dev));
    dev &= 63;
    const size_t smem = (size_t)kTsSmem + 1024;
    if (!attr_set[dev]) {
        EET_CUDA(cudaFuncSetAttribute(gemm_ts_kernel<kUnit>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attr_set[dev] = true;
    }
    CUtensorMap map, map_w;
    const int KT = a.K / kTile;
    const cuuint64_t wdims[4] = {64, 64, (cuuint64_t)KT, (cuuint64_t)(a.N / kTile)};
    const cuuint64_t wstrides[3] = {64, (cuuint64_t)kTileBytes, (cuuint64_t)KT * kTileBytes};
    const cuuint32_t wbox[4] = {64, 64, kUnit, 4}, welem[4] = {1, 1, 1, 1};
    const CUresult rw = encode(&map_w, CU_TENSOR_MAP_DATA_TYPE_UINT8, 4, const_cast<uint8_t*>(a.B), wdims, wstrides, wbox, welem,
                               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    EET_CHECK(rw == CUDA_SUCCESS, "tensor-core GEMM: cuTensorMapEncodeTiled failed with code %d", (int)rw);
    const cuuint64_t dims[2] = {(cuuint64_t)a.K, (cuuint64_t)a.M};
    const cuuint64_t strides[1] = {(cuuint64_t)a.K * sizeof(__half)};
    const cuuint32_t box[2] = {64, (cuuint32_t)a.bn};   // (rows past M read as zeros)
    const cuuint32_t elem[2] = {1, 1};
    const CUresult rc = encode(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<__half*>(A), dims, strides, box, elem,
                               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                               CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    EET_CHECK(rc == CUDA_SUCCESS, "tensor-core GEMM: cuTensorMapEncodeTiled failed with code %d", (int)rc);
    // weights as deep as four stages of activations leave room for, an even number of stages; the rest to the activations
    const int x_bytes = a.bn * 128, w_bytes = kUnit * kTsWBlock, room = kTsSmem - kTsStageBytes;
    a.nw = (room - 4 * x_bytes) / (kTsSets * w_bytes) * kTsSets;
    if (a.nw > kTsMaxNW) a.nw = kTsMaxNW;
    a.nx = (room - a.nw * w_bytes) / x_bytes;
    if (a.nx > kTsMaxNX) a.nx = kTsMaxNX;
    a.acc_cols = a.bn;
    a.na = (kTsCols - 2 * a.acc_cols) / (64 * kUnit);
    if (a.na > kTsMaxNA) a.na = kTsMaxNA;
    EET_CHECK(ts_fits(a.bn, split), "tensor-core GEMM: %d CTAs cannot share a tile of %d tokens", split, a.bn);
    EET_CHECK(a.bn % 16 == 0 && a.nx >= 2 && a.nw >= kTsSets && a.na >= kTsSets, "tensor-core GEMM: a token tile of %d does not fit", a.bn);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(split > 1 || a.tiles < sm_count() ? a.tiles : sm_count()), 1, (unsigned)split);
    cfg.blockDim = dim3(kTsThreads, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = (unsigned)split;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 2;
    EET_CUDA(cudaLaunchKernelEx(&cfg, gemm_ts_kernel<kUnit>, map, map_w, a));
    return 0;
}

}  // namespace

// Clusters of `split` CTAs of the kernel that can be resident at once (0: that cluster size cannot be launched), asked of the
// occupancy calculator once per device and size.
static int ts_max_clusters(int split)
{
    static int cached[64][kTsMaxSplit + 1] = {};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return 0;
    dev &= 63;
    if (cached[dev][split] == 0) {
        const size_t smem = (size_t)kTsSmem + 1024;
        int n = 0;
        if (cudaFuncSetAttribute(gemm_ts_kernel<1>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) == cudaSuccess) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(1, 1, split);
            cfg.blockDim = dim3(kTsThreads, 1, 1);
            cfg.dynamicSmemBytes = smem;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = 1;
            attr[0].val.clusterDim.y = 1;
            attr[0].val.clusterDim.z = split;
            cfg.attrs = attr;
            cfg.numAttrs = 1;
            if (cudaOccupancyMaxActiveClusters(&n, gemm_ts_kernel<1>, &cfg) != cudaSuccess) {
                (void)cudaGetLastError();
                n = 0;
            }
        }
        cached[dev][split] = n > 0 ? n : -1;
    }
    return cached[dev][split] > 0 ? cached[dev][split] : 0;
}

// The plan with the least modelled time over all token tiles and cluster sizes; us is large where the kernel does not take the shape.
// Times in microseconds, fitted to measured calls of 17 to 2048 rows on 4096 x 4096 to 8192 x 22016 (the 145 plans within
// 15 % of the best of their shape: spread 5 %; the choice is 0.5 % off the best plan on average, 5 % at most): a k-block of a 256 x BN tile with the machine full,
// or what HBM needs for the weights of a k-block of all CTAs that run; a tile's start, end and epilogue; in a cluster the
// exchange, by the tokens times senders (1 KiB each) that a CTA receives.
Tc2Plan gemm_ts_plan(int M, int N, int K)
{
    Tc2Plan best = {0, 0, 0, 1, 1e30};
    if (M < kTsMinM || N < kTsMinN || K < kTsMinK || K % 64 != 0 || N % 128 != 0 || (N % 256 != 0 && N < 2 * kTsMinN)) return best;
    static const struct { int bn; double us; } at[7] = {{32, 0.294}, {64, 0.280}, {96, 0.341}, {128, 0.391}, {144, 0.418}, {160, 0.444}, {192, 0.510}};
    const int G = sm_count(), KT = K / kTile, tiles_n = (N + 255) / 256;
    for (int tiles_m = (M + 191) / 192; tiles_m <= (M + 31) / 32; ++tiles_m) {
        int bn = ((M + tiles_m - 1) / tiles_m + 15) / 16 * 16;
        if (bn < 32) bn = 32;
        if ((M + bn - 1) / bn != tiles_m) continue;
        const long long tiles = (long long)tiles_n * tiles_m;
        if (tiles > 3LL * G) break;   // (beyond three waves the CTA pairs are faster)
        int i = 0;
        while (i < 5 && bn > at[i + 1].bn) ++i;
        const double block = at[i].us + (at[i + 1].us - at[i].us) * (bn - at[i].bn) / (at[i + 1].bn - at[i].bn);
        const int unit = ts_unit(bn), units = (KT + unit - 1) / unit;
        for (int S = 1; S <= kTsMaxSplit; ++S) {
            const int room = S == 1 ? G : ts_max_clusters(S);
            if (room == 0 || !ts_fits(bn, S) || units / S < kTsSets) continue;
            const int rounds = (int)((tiles + room - 1) / room);
            if (rounds > 1 && M > 512) continue;
            const double reading = (double)(tiles < room ? tiles : room) / tiles_m * S * (kTsWBlock / 6.1e6);
            const int chunk = ts_chunk(bn), chunks = (bn + chunk - 1) / chunk;
            double us = (units + S - 1) / S * unit * (block > reading ? block : reading) + 2.86 + 0.0214 * bn;
            if (S > 1) us += 1.13 + 0.0145 * ((chunks + S - 1) / S * (S - 1) * chunk) + (tiles_m > 1 ? 0.9 : 0.0);
            us = rounds * us - 0.34;
            // Up to 64 rows: CTAs without a second tile leave HBM to the others and their SM to the next kernel (149 to 400
            // tiles, measured 0.68 to 0.90 of full rounds); clusters of five to eight that end at different times do not
            // find room again at once (4 to 25 % longer).
            if (rounds > 1 && M < kTcMinM) us *= S == 1 ? 0.85 : (S > 4 ? 1.1 : 1.0);
            if (us < best.us) best = Tc2Plan{bn, (int)tiles, S == 1 ? (int)tiles : 0, S, us};
        }
    }
    return best;
}

int launch_gemm_ts(const __half* A, const uint8_t* B, const __half* scale, __half* C, const __half* residual, int gate, int M, int N,
                   int K, const Tc2Plan& plan, cudaStream_t stream)
{
    EET_CHECK(plan.bn > 0, "tensor-core GEMM: no plan for M=%d N=%d K=%d", M, N, K);
    TsArgs a = {};
    a.B = B;
    a.scale = scale;
    a.C = C;
    a.residual = residual;
    a.gate = gate;
    a.M = M;
    a.N = N;
    a.K = K;
    a.bn = plan.bn;
    a.tiles = plan.tiles;
    a.stream = M <= plan.bn;   // one token tile: the weights are read once
    return ts_unit(plan.bn) == 2 ? launch_ts<2>(A, a, plan.split, stream) : launch_ts<1>(A, a, plan.split, stream);
}

}  // namespace eet
