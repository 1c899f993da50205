// W8A16 GEMM for decode (M <= 16), finished in one launch: C[M,N] = A[M,K] (fp16) x dequant(B), scale, and the residual
// add or the gated activation, B in the W8T64 layout.  Optionally two weights of the same shape at once (gate and up
// projection): C = gated_silu(A x B, A x B2).
//
// gemm_skinny.cu deals equal shares of tiles to the CTAs, which balances perfectly but leaves fp32 partial sums in global
// memory for another launch to finish.  Here a CTA - or a cluster of 2 to 8 that splits the reduction - owns a whole
// tile row (64 channels) and stores fp16.  Equal shares are not what HBM needs: it needs about 10 MB in flight, which
// 150 CTAs with 64 KiB each give whatever the number of rows, so uneven rows per SM cost nothing until an SM has to
// convert faster than it can (about 90 B/cycle against the 24 of its share of HBM) - up to two rows per SM.  More rows run in
// waves, and a last wave of few CTAs has too little in flight: see gemm_row_wastes_a_wave.
//
//  * Eight warps, each with a ring of its own (two 4 KiB tiles, filled by 1-D bulk copies that its lane 0 issues):
//    warp w takes tiles w, w + 8, ... of the CTA's share of the row.  No producer warp, no barrier between warps until
//    the row is done.  The first two tiles are requested before anything else, without waiting for the preceding
//    kernel (weights are constants): 128 KiB an SM are on their way while that kernel drains.
//  * A warp multiplies its tile's 64 channels at once - four mma.m16n8k16 row groups, weights as the 16-row operand,
//    tokens as the 8 columns - so a fragment of the activations is loaded once per tile, straight from L2 into
//    registers one tile ahead, and four independent accumulator chains hide the latency of mma.sync.
//  * The two norms of a decoder layer need no launch of their own: a kernel that stores the residual stream also leaves
//    the sum of squares of its 64 channels of each token (`squares_out`, one float per row and token), and the kernel
//    behind it adds those up (`squares_in`) and normalises the activations as it loads them: a power of two next to
//    1 / rms times gamma goes onto the fp16 activations (two multiplies per pair, rounded once, as rmsnorm_kernel rounds
//    once), the rest of 1 / rms onto the sums.
//  * End of the row: the warps' accumulators meet in shared memory, the CTAs' in rank 0's (distributed shared memory,
//    one cluster barrier), added in a fixed order: results do not depend on timing.
//
// What bounds it: HBM, and for M > 8 the activations' way from L2 (half as many bytes as the weights).  LLaMA-7B shapes at
// M = 8, weights from HBM (kernel alone, back to back): QKV 9.0 us = 5.6 TB/s, output 4.8, gate and up together 15.4 us =
// 5.9 TB/s, down 9.0; the equal-share kernel 10.3, 5.0, 19 and 9.9 and a finishing launch behind each.  5120 x 15360 at
// M = 12: 15.7 us with everything, 20.2 as two launches.  The norm inside costs 0.7 us of a launch of 4.  Measured and not
// taken: three or four tiles per ring (0 to 40 % slower), two rows per CTA at M > 8 (20 to 120 % slower).
//
// Numerics: products of fp16 activations with exact integer weights, fp32 accumulation, one multiply by the fp16 scale,
// one rounding to fp16; then the fp16 residual add or the reference's gated activation.
#include "common.cuh"
#include "kernels.h"

namespace eet {

namespace {

constexpr int kRowWarps = 8;
constexpr int kRowThreads = kRowWarps * 32;
constexpr int kRowSlots = 2;
constexpr int kRowMaxSmem = 200 * 1024;
constexpr int kRowRing = kRowWarps * kRowSlots * kTileBytes;

// Float of token t, channel c in a warp's [token][64 channels] accumulators: the channel is permuted by the token so that
// the fragments' stores (4 token pairs x 8 channels) hit 32 banks; pairs of channels stay together.
__device__ __forceinline__ int row_red_at(int t, int c)
{
    return t * kTile + (c ^ (((t >> 1) & 3) << 3));
}

template<int NB>
__host__ __device__ constexpr int row_partial_floats()
{
    return 8 * NB * 64;   // one CTA's sums of one matrix
}

template<int NB, bool kPair, bool kNorm>
__global__ void __launch_bounds__(kRowThreads, 2)
gemm_row_kernel(RowGemmArgs a)
{
    extern __shared__ __align__(128) uint8_t row_dyn[];   // [warp][slot] tiles | partial sums of the other ranks
    __shared__ uint64_t full[kRowWarps][kRowSlots];
    pdl_launch_dependents();
    constexpr int kMats = kPair ? 2 : 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int S = a.splits, rank = (int)blockIdx.x % S, row = (int)blockIdx.x / S;
    const int KT = a.K / kTile;
    const int t0 = KT * rank / S, n_tiles = KT * (rank + 1) / S - t0;   // this CTA's tiles of each row
    uint8_t* ring = row_dyn + (size_t)warp * kRowSlots * kTileBytes;
    const size_t first = ((size_t)row * KT + t0) * kTileBytes;

    // ---- this warp's ring: tiles warp, warp + 8, ... of the share, of both matrices in turn ----
    const int mine = n_tiles > warp ? (n_tiles - warp + kRowWarps - 1) / kRowWarps : 0;
    auto issue = [&](int q, int slot, uint32_t offset) {
        const int i = warp + kRowWarps * (q / kMats);
        mbar_arrive_expect_tx(&full[warp][slot], kTileBytes);
        bulk_g2s_stream(ring + slot * kTileBytes, (q % kMats ? a.B2 : a.B) + first + (size_t)i * kTileBytes + offset, kTileBytes, &full[warp][slot]);
    };
    if (lane == 0) {
        for (int s = 0; s < kRowSlots; ++s) mbar_init(&full[warp][s], 1);
        mbar_fence_init();
        for (int s = 0; s < kRowSlots && s < kMats * mine; ++s) issue(s, s, 0);
    }
    __syncwarp();
    if (S > 1) asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory");   // waited for before the first remote store

    const int gq = lane >> 2, tq = lane & 3;   // mma fragment coordinates
    float acc[kMats][4][NB][4];
#pragma unroll
    for (int p = 0; p < kMats; ++p)
#pragma unroll
        for (int cg = 0; cg < 4; ++cg)
#pragma unroll
            for (int nb = 0; nb < NB; ++nb)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[p][cg][nb][c] = 0.f;

    // this CTA's norm weights (constants) into shared memory
    __half* gamma_s = reinterpret_cast<__half*>(row_dyn + kRowRing + (size_t)(S - 1) * kMats * row_partial_floats<NB>() * 4);
    if (kNorm) {
        for (int i = threadIdx.x; i < n_tiles * 8; i += kRowThreads) {
            reinterpret_cast<uint4*>(gamma_s)[i] = __ldg(reinterpret_cast<const uint4*>(a.gamma + (size_t)t0 * kTile) + i);
        }
    }

    // activations, residual and output belong to the dependency chain
    pdl_wait();

    // 1 / rms of every token from the sums of squares of its K/64 pieces, split into a power of two that scales the
    // activations exactly and a factor for the sums.  A warp per token and 128-byte requests: all CTAs want the same few
    // lines of L2 at the same time (every warp reading all tokens' pieces in small loads cost 16 us a launch).
    __shared__ float post_s[16], pre_s[16];
    float squares[NB];
    if (kNorm) {
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
            squares[nb] = 0.f;
            if (warp + 8 * nb < a.M) {
                for (int r = lane; r < KT; r += 32) squares[nb] += __ldcg(a.squares_in + (size_t)(warp + 8 * nb) * KT + r);
            }
        }
    }
    // fragment of the activations for a tile: token gq (+8), reduction indices 16 tq .. 16 tq + 15
    uint4 xr[NB][2];
    auto fetch_x = [&](int j) {
        const int i = warp + kRowWarps * j;
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
            xr[nb][0] = xr[nb][1] = make_uint4(0u, 0u, 0u, 0u);
            if (j < mine && gq + 8 * nb < a.M) {
                const uint4* p = reinterpret_cast<const uint4*>(a.A + (size_t)(gq + 8 * nb) * a.K + (size_t)(t0 + i) * kTile + tq * 16);
                xr[nb][0] = p[0];   // (not __ldg: the preceding kernel writes them during this one's lifetime)
                xr[nb][1] = p[1];
            }
        }
    };
    fetch_x(0);
    __half2 pre[NB];
    if (kNorm) {
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
            const float inv = rsqrtf(warp_sum(squares[nb]) / a.K + a.eps);
            const int e = min(max(((__float_as_int(inv) >> 23) & 255) - 127, -24), 15);
            const float p2 = __int_as_float((e + 127) << 23);
            if (lane == 0) {
                pre_s[warp + 8 * nb] = p2;
                post_s[warp + 8 * nb] = inv / p2;
            }
        }
        __syncthreads();   // (also: the norm weights are in shared memory)
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) pre[nb] = __float2half2_rn(pre_s[gq + 8 * nb]);
    }
    int slot = 0;
    uint32_t phase = 0;
    bool live = true;
    for (int j = 0; j < mine; ++j) {
        uint32_t xw[NB][8];
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
            xw[nb][0] = xr[nb][0].x; xw[nb][1] = xr[nb][0].y; xw[nb][2] = xr[nb][0].z; xw[nb][3] = xr[nb][0].w;
            xw[nb][4] = xr[nb][1].x; xw[nb][5] = xr[nb][1].y; xw[nb][6] = xr[nb][1].z; xw[nb][7] = xr[nb][1].w;
        }
        if (kNorm) {
            // fp16(x * 2^e * gamma): x * 2^e is of order one, so this rounds like the norm kernel's x * inv * gamma
            const uint4* p = reinterpret_cast<const uint4*>(gamma_s + (warp + kRowWarps * j) * kTile + tq * 16);
            const uint4 g0 = p[0], g1 = p[1];
            const uint32_t gw[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
#pragma unroll
            for (int nb = 0; nb < NB; ++nb)
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    const __half2 v = __hmul2(__hmul2(*reinterpret_cast<const __half2*>(&xw[nb][e]), pre[nb]),
                                              *reinterpret_cast<const __half2*>(&gw[e]));
                    xw[nb][e] = *reinterpret_cast<const uint32_t*>(&v);
                }
        }
        fetch_x(j + 1);
#pragma unroll
        for (int p = 0; p < kMats; ++p) {
            if (live && !mbar_wait_bounded(&full[warp][slot], phase)) {
                live = false;   // give up on this warp's tiles: no more waits and no more requests
                g_device_status = 1;
            }
            const uint8_t* w = ring + slot * kTileBytes + lane * 16;
            uint32_t words = 0;
#pragma unroll
            for (int cg = 0; cg < 4; ++cg) {
                const uint4 wa = *reinterpret_cast<const uint4*>(w + cg * 1024);
                const uint4 wb = *reinterpret_cast<const uint4*>(w + cg * 1024 + 512);
                const uint32_t wa4[4] = {wa.x, wa.y, wa.z, wa.w};
                const uint32_t wb4[4] = {wb.x, wb.y, wb.z, wb.w};
                words = wb.w;   // (the reads before this one have become operands of the MMAs)
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    uint32_t a0, a1, a2, a3;
                    cvt_u8x4_to_f16x4(wa4[i], a0, a2);
                    cvt_u8x4_to_f16x4(wb4[i], a1, a3);
#pragma unroll
                    for (int nb = 0; nb < NB; ++nb) {
                        mma_m16n8k16(acc[p][cg][nb], a0, a1, a2, a3, xw[nb][2 * i], xw[nb][2 * i + 1]);
                    }
                }
            }
            __syncwarp();
            const int q = kMats * j + p + kRowSlots;
            if (lane == 0 && live && q < kMats * mine) issue(q, slot, after_reads(words, a.zero));
            if (++slot == kRowSlots) {
                slot = 0;
                phase ^= 1;
            }
        }
    }

    // ---- the warps' accumulators meet: each leaves its own in its own ring, which is idle now ----
    constexpr int kRedFloats = 8 * NB * kTile;
    static_assert(kMats * kRedFloats * 4 <= kRowSlots * kTileBytes, "a warp's accumulators must fit into its ring");
    {
        float* red = reinterpret_cast<float*>(ring);
        if (kNorm) {
            // (a fragment's columns are tokens 2 tq and 2 tq + 1)
#pragma unroll
            for (int nb = 0; nb < NB; ++nb) {
                const float f0 = post_s[8 * nb + 2 * tq], f1 = post_s[8 * nb + 2 * tq + 1];
#pragma unroll
                for (int p = 0; p < kMats; ++p)
#pragma unroll
                    for (int cg = 0; cg < 4; ++cg)
#pragma unroll
                        for (int c = 0; c < 4; ++c) acc[p][cg][nb][c] *= (c & 1) ? f1 : f0;
            }
        }
#pragma unroll
        for (int p = 0; p < kMats; ++p)
#pragma unroll
            for (int cg = 0; cg < 4; ++cg)
#pragma unroll
                for (int nb = 0; nb < NB; ++nb)
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        // fragment element c: token 8 nb + 2 tq + (c & 1), channel 16 cg + gq + 8 (c >> 1)
                        red[p * kRedFloats + row_red_at(8 * nb + 2 * tq + (c & 1), cg * 16 + gq + 8 * (c >> 1))] = acc[p][cg][nb][c];
                    }
    }
    __syncthreads();
    // this thread: tokens warp (+8), channels 2 lane and 2 lane + 1
    float2 sum[kMats][NB];
#pragma unroll
    for (int p = 0; p < kMats; ++p)
#pragma unroll
        for (int nb = 0; nb < NB; ++nb) {
            sum[p][nb] = make_float2(0.f, 0.f);
#pragma unroll
            for (int w = 0; w < kRowWarps; ++w) {
                const float2 v = *reinterpret_cast<const float2*>(row_dyn + (size_t)w * kRowSlots * kTileBytes +
                                                                  4 * (p * kRedFloats + row_red_at(8 * nb + warp, 2 * lane)));
                sum[p][nb].x += v.x;
                sum[p][nb].y += v.y;
            }
        }

    // ---- and the CTAs' of the cluster: pushed into rank 0's shared memory ----
    constexpr int kPart = row_partial_floats<NB>();
    if (S > 1) {
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");   // every CTA of the cluster runs: its memory may be written
        float* part = reinterpret_cast<float*>(row_dyn + kRowRing);
        if (rank != 0) {
#pragma unroll
            for (int p = 0; p < kMats; ++p)
#pragma unroll
                for (int nb = 0; nb < NB; ++nb) {
                    const uint32_t local = smem_u32(part + ((rank - 1) * kMats + p) * kPart + (8 * nb + warp) * 64 + 2 * lane);
                    uint32_t remote;
                    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(remote) : "r"(local));
                    asm volatile("st.shared::cluster.v2.f32 [%0], {%1, %2};" ::"r"(remote), "f"(sum[p][nb].x), "f"(sum[p][nb].y) : "memory");
                }
        }
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (rank != 0) return;
        for (int r = 0; r < S - 1; ++r) {
#pragma unroll
            for (int p = 0; p < kMats; ++p)
#pragma unroll
                for (int nb = 0; nb < NB; ++nb) {
                    const float2 v = *reinterpret_cast<const float2*>(part + (r * kMats + p) * kPart + (8 * nb + warp) * 64 + 2 * lane);
                    sum[p][nb].x += v.x;
                    sum[p][nb].y += v.y;
                }
        }
    }

    const int n = row * kTile + 2 * lane;
    const float2 sc = __half22float2(*reinterpret_cast<const __half2*>(a.scale + n));
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
        const int m = 8 * nb + warp;
        if (m < a.M) {
            const size_t at = (size_t)m * a.N + n;
            __half2 o = __floats2half2_rn(sum[0][nb].x * sc.x, sum[0][nb].y * sc.y);
            if (kPair) {
                const float2 sc2 = __half22float2(*reinterpret_cast<const __half2*>(a.scale2 + n));
                o = gated_silu2(o, __floats2half2_rn(sum[kMats - 1][nb].x * sc2.x, sum[kMats - 1][nb].y * sc2.y));
            }
            else if (a.residual != nullptr) {
                const __half2 r = *reinterpret_cast<const __half2*>(a.residual + at);
                o = a.gate ? gated_silu2(r, o) : __hadd2(o, r);
            }
            *reinterpret_cast<__half2*>(a.C + at) = o;
            if (a.squares_out != nullptr) {   // (a warp holds the 64 channels of one token)
                const float2 f = __half22float2(o);
                const float ss = warp_sum(f.x * f.x + f.y * f.y);
                if (lane == 0) a.squares_out[(size_t)m * (a.N / kTile) + row] = ss;
            }
        }
    }
}

template<int NB, bool kPair, bool kNorm>
int launch_row(const RowGemmArgs& a, cudaStream_t stream)
{
    static bool attr_set[64] = {};
    int dev = 0;
    EET_CUDA(cudaGetDevice(&dev));
    dev &= 63;
    constexpr int kPartBytes = row_partial_floats<NB>() * (kPair ? 2 : 1) * 4;
    if (!attr_set[dev]) {
        EET_CUDA(cudaFuncSetAttribute(gemm_row_kernel<NB, kPair, kNorm>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      kRowMaxSmem));
        attr_set[dev] = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(a.N / kTile * a.splits));
    cfg.blockDim = dim3(kRowThreads);
    cfg.dynamicSmemBytes = (size_t)kRowRing + (size_t)(a.splits - 1) * kPartBytes;
    if (kNorm) cfg.dynamicSmemBytes += (size_t)((a.K / kTile + a.splits - 1) / a.splits) * kTile * sizeof(__half);
    EET_CHECK(cfg.dynamicSmemBytes <= (size_t)kRowMaxSmem, "decode GEMM: K=%d is too long for the norm inside it", a.K);
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = (unsigned)a.splits;
    attr[1].val.clusterDim.y = 1;
    attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = a.splits > 1 ? 2 : 1;
    EET_CUDA(cudaLaunchKernelEx(&cfg, gemm_row_kernel<NB, kPair, kNorm>, a));
    return 0;
}

}  // namespace

// A wide matrix whose last wave of tile rows is mostly empty: the equal shares of gemm_skinny.cu read it faster, with a finishing
// launch (3 us) and all, when what stays empty is worth more than 50 MB of weights.  M = 8: 8192 x 22016 (130 MB empty) 30.3 us
// against 34.1 here, 8192 x 24576 (109) 33.3, 35.6; 5120 x 22016 (81) 20.5, 24.3; 4096 x 24576 (55) 18.8, 20.4; 4096 x 28672
// (38) 21.3, 21.2; 4096 x 32000 (24) 23.7, 22.4.  Above 8 rows that kernel is bound by the activations (8192 x 22016 at M = 16
// 39.1, 36.9) and the faster one only where the last wave is as good as empty (8192 x 19456, 304 rows: 33.9, 35.4).
bool gemm_row_wastes_a_wave(int M, int N, int K)
{
    const int rows = N / kTile, slots = 2 * sm_count();
    const int empty = rows > slots ? (rows + slots - 1) / slots * slots - rows : 0;
    const double bytes = (double)empty * kTile * K;
    return M <= 8 ? bytes > 50e6 : bytes > 100e6 && empty > 0.85 * rows;
}

int launch_gemm_row(RowGemmArgs a, cudaStream_t stream)
{
    EET_CHECK(a.M <= kRowMaxM, "decode GEMM: M=%d exceeds %d", a.M, kRowMaxM);
    if (a.M == 0) return 0;
    // Two CTAs fit on an SM.  Fewer rows than SMs: as many CTAs per row as there is room for (4096 x 4096: four, 4.8 us),
    // each with at least one tile per warp.  More, up to two per SM: a row per CTA (4096 x 12288: 192 CTAs, 9.1 us).  More
    // than that run in waves; two CTAs per row where that leaves 70 MB less of the last wave empty (344 rows, 1.5 waves
    // instead of 2: 8192 x 22016 at M = 16 36.9 us instead of 41.0, gate and up together at M = 8 60.5 instead of 66.5;
    // 4096 x 22016, 39 MB: 22.2 instead of 20.5).
    const int rows = a.N / kTile, slots = 2 * sm_count(), KT = a.K / kTile;
    int s = 1;
    if (rows > slots) {
        const int half_waves = 2 * ((rows + slots - 1) / slots) - (2 * rows + slots - 1) / slots;   // saved by two CTAs per row
        if ((double)half_waves * slots * kTile * a.K * (a.B2 != nullptr ? 2 : 1) / 2 > 70e6) s = 2;
    }
    else {
        const int room = slots / rows;
        while (s < kRowMaxSplits && s + 1 <= room && KT / (s + 1) >= kRowWarps) ++s;
    }
    a.splits = s < 5 ? s : (s < 8 ? 4 : 8);
    const bool norm = a.gamma != nullptr;
    if (a.M <= 8) {
        if (a.B2 != nullptr) return norm ? launch_row<1, true, true>(a, stream) : launch_row<1, true, false>(a, stream);
        return norm ? launch_row<1, false, true>(a, stream) : launch_row<1, false, false>(a, stream);
    }
    if (a.B2 != nullptr) return norm ? launch_row<2, true, true>(a, stream) : launch_row<2, true, false>(a, stream);
    return norm ? launch_row<2, false, true>(a, stream) : launch_row<2, false, false>(a, stream);
}

}  // namespace eet
