// Symmetric per-output-channel int8 quantizer and the W8T64 weight packer.
//
// Replaces, for the int8 path, the reference's host-side symmetric_quantize
// (3rdparty/cutlass_kernels/cutlass_preprocessors.cc:581-678) and preprocess_weights_for_mixed_gemm
// (:497-534).  The arithmetic is kept operation for operation so that the int8 values and the scales
// are bit-identical: per-column max of |w| ignoring NaN, scale = amax * (1/128) in fp32, quotient by
// the un-rounded fp32 scale with IEEE division, C round() (half away from zero), clamp with the
// operand order of std::min / std::max (NaN -> 127).
//
// Layout produced ("W8T64"): tiles of 64 output channels x 64 reduction indices, ordered
// [N/64][K/64]; byte (n % 64) * 64 + (k % 64) inside a tile; each byte is q + 128.  One tile is a
// contiguous 4 KiB block, so a GEMM CTA streams its share of the weights as one linear byte range.
#include "common.cuh"
#include "kernels.h"

namespace eet {

namespace {

template<typename T>
struct Vec8;
template<>
struct Vec8<__half> {
    uint4 raw;
    __device__ __forceinline__ void load(const __half* p) { raw = *reinterpret_cast<const uint4*>(p); }
    __device__ __forceinline__ float get(int i) const
    {
        const __half* h = reinterpret_cast<const __half*>(&raw);
        return __half2float(h[i]);
    }
};
template<>
struct Vec8<float> {
    float4 a, b;
    __device__ __forceinline__ void load(const float* p)
    {
        a = *reinterpret_cast<const float4*>(p);
        b = *reinterpret_cast<const float4*>(p + 4);
    }
    __device__ __forceinline__ float get(int i) const
    {
        const float* f = reinterpret_cast<const float*>(&a);
        return i < 4 ? f[i] : reinterpret_cast<const float*>(&b)[i - 4];
    }
};

// max |w| of 8 columns over rows k0 + ty, k0 + ty + 8, ... of a slab of 64.  All eight rows are requested before the
// first is used.  NaN never becomes the maximum: fmaxf and __hmax2 return their non-NaN operand, as std::max(acc, x)
// does when x is NaN.
__device__ __forceinline__ void slab_max8(const float* p, size_t row_stride, float (&m)[8])
{
    Vec8<float> v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r].load(p + r * row_stride);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
#pragma unroll
        for (int r = 0; r < 8; ++r) m[i] = fmaxf(m[i], fabsf(v[r].get(i)));
    }
}
__device__ __forceinline__ void slab_max8(const __half* p, size_t row_stride, float (&m)[8])
{
    uint4 v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) v[r] = *reinterpret_cast<const uint4*>(p + r * row_stride);
    __half2 h[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        h[i] = __floats2half2_rn(0.f, 0.f);
#pragma unroll
        for (int r = 0; r < 8; ++r) h[i] = __hmax2(h[i], __habs2(reinterpret_cast<const __half2*>(&v[r])[i]));
        const float2 f = __half22float2(h[i]);
        m[2 * i] = f.x;
        m[2 * i + 1] = f.y;
    }
}

// Per-column max |w| over a slab of 64 rows x 256 columns, merged into amax[N] with an integer atomic
// max (valid because the values are non-negative floats).
template<typename T>
__global__ void __launch_bounds__(256) colmax_kernel(const T* __restrict__ w, int K, int N, float* __restrict__ amax)
{
    __shared__ float red[8][256];
    pdl_launch_dependents();
    const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
    const int n0 = blockIdx.x * 256 + tx * 8;
    const int k0 = blockIdx.y * 64;
    float m[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) m[i] = 0.f;
    if (n0 < N) slab_max8(w + (size_t)(k0 + ty) * N + n0, (size_t)8 * N, m);
#pragma unroll
    for (int i = 0; i < 8; ++i) red[ty][tx * 8 + i] = m[i];
    __syncthreads();
    const int c = threadIdx.x;
    float v = red[0][c];
#pragma unroll
    for (int r = 1; r < 8; ++r) v = fmaxf(v, red[r][c]);
    const int n = blockIdx.x * 256 + c;
    if (n < N) {
        atomicMax(reinterpret_cast<int*>(amax) + n, __float_as_int(v));
    }
}

__device__ __forceinline__ float col_scale(float amax, int variant)
{
    return variant ? __fdiv_rn(amax, 127.f) : amax * (1.f / 128.f);
}

__device__ __forceinline__ int quantize_one(float w, float s, float lo)
{
    float r = roundf(__fdiv_rn(w, s));
    float c = (r < 127.f) ? r : 127.f;  // std::min(127.f, r)
    c = (lo < c) ? c : lo;              // std::max(lo, c)
    return (int)c;
}

// Fast path of quantize_one for a column whose scale lies in [2^-100, 2^100] (then every |w / s| is at most 128 up to
// rounding): t = w * rcp(s) differs from the IEEE quotient fl(w / s) by less than 128 * (2^-23 + 2 * 2^-24) = 3.1e-5
// (one ulp of the reciprocal, one rounding of the product, one of the quotient), so unless t lies within 2^-14 of a
// half-integer both round to the same integer and the rounding mode does not matter; in that rare case
// (1.2e-4 of all values) the caller does the division.  min(t, 127) is the upper clamp and also what the reference's
// std::min makes of NaN; the lower clamp cannot act (t >= -128, or -127 for variant 1, up to the same 3.1e-5).
// Adding 1.5 * 2^23 + 128 leaves round(t) + 128 in the low byte.  Two values at a time: this GPU adds and multiplies
// pairs of floats in one instruction, and the kernel is bound by instruction issue before it is by memory.
constexpr float kQuantMagic = 12582912.0f + 128.0f;
constexpr float kQuantSure = 0.5f - 6.103515625e-5f;

__device__ __forceinline__ uint64_t pack_f32x2(float a, float b)
{
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack_f32x2(uint64_t v, float& a, float& b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}

__device__ __forceinline__ bool usual_scale(float s)
{
    return s >= 7.888609052210118e-31f && s <= 1.2676506002282294e30f;   // 2^-100, 2^100
}

// q0, q1: words whose low byte is the quantized value + 128; far: the largest distance from the rounded value so far
__device__ __forceinline__ void quantize_fast2(float w0, float w1, float inv, float& far, uint32_t& q0, uint32_t& q1)
{
    uint64_t t, f, d;
    float a, b;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(t) : "l"(pack_f32x2(w0, w1)), "l"(pack_f32x2(inv, inv)));
    unpack_f32x2(t, a, b);
    const uint64_t t2 = pack_f32x2(fminf(a, 127.f), fminf(b, 127.f));
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(f) : "l"(t2), "l"(pack_f32x2(kQuantMagic, kQuantMagic)));
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(f), "l"(pack_f32x2(-kQuantMagic, -kQuantMagic)));
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(t2), "l"(pack_f32x2(-1.f, -1.f)), "l"(d));
    unpack_f32x2(d, a, b);
    far = fmaxf(far, fmaxf(fabsf(a), fabsf(b)));
    unpack_f32x2(f, a, b);
    q0 = __float_as_uint(a);
    q1 = __float_as_uint(b);
}

// Four rows of one column by division: about one column in 70 of a warp's comes here, so the code is kept out of the
// way of the rest.
__device__ __noinline__ uint32_t quantize_by_division(float w0, float w1, float w2, float w3, float s, float lo)
{
    return (uint32_t)(quantize_one(w0, s, lo) + 128) | (uint32_t)(quantize_one(w1, s, lo) + 128) << 8 |
           (uint32_t)(quantize_one(w2, s, lo) + 128) << 16 | (uint32_t)(quantize_one(w3, s, lo) + 128) << 24;
}

// 128 * U(k) x 64(n) values per block (as many 64-row tiles as there are left at the end of K): quantize, optionally
// emit the row-major int8 matrix, and write the tiles' 4 KiB of the W8T64 layout with coalesced 16-byte stores after a
// transpose in shared memory.  Blocks that hold row 0 also write the scales.
//
// A thread owns 8 columns x 4 consecutive rows of U tiles (all loads in flight at once; U = 2 for fp16, 1 for fp32, the
// same 128 bytes), so the four bytes of a word of the packed layout meet in one thread's registers, and a warp's 4
// column groups x 8 row quads store to 32 different banks (rows of 17 words).  The row blocks are walked backwards: the
// column-max pass before this one read the matrix forwards, and what it read last is still in the L2.
// Bound by instruction issue (about 6 instructions a value; DRAM at 38 %).  4096 x 11008 fp16 on its own: 33 us, against
// 59 us with one IEEE division and one bank-conflicting byte store per value; the call (memset, maxima 18.5 us, this
// kernel) 51.8 us against 84.0.  The bytes of the call need 20 us read once, 34 us read twice.
// kVec: the caller's scratch is 16-byte aligned and the maxima come in two loads.  One float at a time costs 11 % of the call
// (4096 x 11008 fp16: 52.7 us, against 46.6), so that is left to scratch that begins elsewhere.
template<typename T, int U, bool kVec>
__global__ void __launch_bounds__(256, 4)
quant_pack_kernel(const T* __restrict__ w, int K, int N, const float* __restrict__ amax, int variant,
                  int8_t* __restrict__ q_rowmajor, uint8_t* __restrict__ packed, void* __restrict__ scales)
{
    __shared__ uint32_t tile[2 * U][64][17];
    const int nt = blockIdx.x, kt = 2 * U * (int)(gridDim.y - 1 - blockIdx.y);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int cg = (warp & 1) * 4 + (lane & 3);           // column group of 8
    const int quad = (warp >> 1) * 8 + (lane >> 2);       // row quad 0..31 of two tiles, then of the next two
    const int n0 = nt * 64 + cg * 8;
    Vec8<T> v[U][4];
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int k0 = kt * 64 + u * 128 + quad * 4;
        if (k0 < K) {
#pragma unroll
            for (int r = 0; r < 4; ++r) v[u][r].load(w + (size_t)(k0 + r) * N + n0);
        }
    }
    // The maxima are the preceding kernel's output.  The weights were complete before that kernel began (it is an
    // ordinary launch), so they are requested before the wait.
    pdl_wait();
    const float lo = variant ? -127.f : -128.f;
    float s[8];
    {
        float m[8];
        if (kVec) {
            const float4 m0 = __ldcg(reinterpret_cast<const float4*>(amax + n0)), m1 = __ldcg(reinterpret_cast<const float4*>(amax + n0) + 1);
            m[0] = m0.x; m[1] = m0.y; m[2] = m0.z; m[3] = m0.w;
            m[4] = m1.x; m[5] = m1.y; m[6] = m1.z; m[7] = m1.w;
        }
        else {
#pragma unroll
            for (int i = 0; i < 8; ++i) m[i] = __ldcg(amax + n0 + i);
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            s[i] = col_scale(m[i], variant);
            if (kt == 0 && quad == 0) {
                if (sizeof(T) == 4) {
                    reinterpret_cast<float*>(scales)[n0 + i] = s[i];
                }
                else {
                    reinterpret_cast<__half*>(scales)[n0 + i] = __float2half_rn(s[i]);
                }
            }
        }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
        const int k0 = kt * 64 + u * 128 + quad * 4;
        if (k0 >= K) break;
        uint32_t word[8];   // column i: rows k0 .. k0 + 3, value + 128 each
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            uint32_t q[4];
            float far = usual_scale(s[i]) ? 0.f : 1.f, inv;
            asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(s[i]));
            quantize_fast2(v[u][0].get(i), v[u][1].get(i), inv, far, q[0], q[1]);
            quantize_fast2(v[u][2].get(i), v[u][3].get(i), inv, far, q[2], q[3]);
            word[i] = __byte_perm(__byte_perm(q[0], q[1], 0x0040), __byte_perm(q[2], q[3], 0x0040), 0x5410);
            if (!(far < kQuantSure)) {
                word[i] = quantize_by_division(v[u][0].get(i), v[u][1].get(i), v[u][2].get(i), v[u][3].get(i), s[i], lo);
            }
        }
        uint32_t* dst = &tile[2 * u + (quad >> 4)][cg * 8][quad & 15];
#pragma unroll
        for (int i = 0; i < 8; ++i) dst[i * 17] = word[i];
        if (q_rowmajor != nullptr) {
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                uint32_t b[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t sel = (uint32_t)(r | ((4 + r) << 4));
                    b[h] = __byte_perm(__byte_perm(word[4 * h], word[4 * h + 1], sel),
                                       __byte_perm(word[4 * h + 2], word[4 * h + 3], sel), 0x5410) ^ 0x80808080u;
                }
                *reinterpret_cast<uint2*>(q_rowmajor + (size_t)(k0 + r) * N + n0) = make_uint2(b[0], b[1]);
            }
        }
    }
    __syncthreads();
    const int row = threadIdx.x >> 2, seg = threadIdx.x & 3;
    uint8_t* dst = packed + ((size_t)nt * (K / 64) + kt) * kTileBytes;
#pragma unroll
    for (int t = 0; t < 2 * U; ++t) {
        if ((kt + t) * 64 < K) {
            const uint32_t* src = &tile[t][row][seg * 4];
            __stcs(reinterpret_cast<uint4*>(dst + t * kTileBytes) + threadIdx.x, make_uint4(src[0], src[1], src[2], src[3]));
        }
    }
}

// Row-major int8 [K][N] -> W8T64 (the role of the reference's preprocess_weights, :536-544).
__global__ void __launch_bounds__(256)
pack_kernel(const int8_t* __restrict__ q, int K, int N, uint8_t* __restrict__ packed)
{
    __shared__ __align__(16) uint8_t tile[64][64 + 16];
    const int nt = blockIdx.x, kt = blockIdx.y;
    const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int kl = ty + half * 32;
        const uint2 v = *reinterpret_cast<const uint2*>(q + ((size_t)kt * 64 + kl) * N + nt * 64 + tx * 8);
        const uint8_t* b = reinterpret_cast<const uint8_t*>(&v);
#pragma unroll
        for (int i = 0; i < 8; ++i) tile[tx * 8 + i][kl] = (uint8_t)(b[i] ^ 0x80u);  // two's complement + 128
    }
    __syncthreads();
    const int row = threadIdx.x >> 2, seg = threadIdx.x & 3;
    uint8_t* dst = packed + ((size_t)nt * (K / 64) + kt) * kTileBytes;
    *reinterpret_cast<uint4*>(dst + threadIdx.x * 16) = *reinterpret_cast<const uint4*>(&tile[row][seg * 16]);
}

// W8T64 -> row-major int8 [K][N].
__global__ void __launch_bounds__(256)
unpack_kernel(const uint8_t* __restrict__ packed, int K, int N, int8_t* __restrict__ q)
{
    __shared__ __align__(16) uint8_t tile[64][64 + 16];
    const int nt = blockIdx.x, kt = blockIdx.y;
    const int row = threadIdx.x >> 2, seg = threadIdx.x & 3;
    const uint8_t* src = packed + ((size_t)nt * (K / 64) + kt) * kTileBytes;
    *reinterpret_cast<uint4*>(&tile[row][seg * 16]) = *reinterpret_cast<const uint4*>(src + threadIdx.x * 16);
    __syncthreads();
    const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int kl = ty + half * 32;
        uint2 v;
        uint8_t* b = reinterpret_cast<uint8_t*>(&v);
#pragma unroll
        for (int i = 0; i < 8; ++i) b[i] = (uint8_t)(tile[tx * 8 + i][kl] ^ 0x80u);
        *reinterpret_cast<uint2*>(q + ((size_t)kt * 64 + kl) * N + nt * 64 + tx * 8) = v;
    }
}

// Bytes packed by the reference for sm75-89 (cutlass_preprocessors.cc:497-534) -> W8T64.  The reference
// layout, in closed form: rows permuted in groups of 16 by {0,1,8,9,2,3,10,11,4,5,12,13,6,7,14,15},
// transposed, column pairs interleaved per 64-row tile (byte position
// (n/2)*2K + 128*(k/64) + 64*(n%2) + k%64), +128, bytes 1 and 2 of each 32-bit word swapped.
__global__ void __launch_bounds__(256)
repack_ref_kernel(const uint8_t* __restrict__ ref, int K, int N, uint8_t* __restrict__ packed)
{
    const int nt = blockIdx.x, kt = blockIdx.y;
    uint8_t* dst = packed + ((size_t)nt * (K / 64) + kt) * kTileBytes;
    for (int e = threadIdx.x; e < kTileBytes; e += 256) {
        const int n = nt * 64 + (e >> 6);
        const int k = kt * 64 + (e & 63);  // logical reduction index wanted at this byte
        // the reference stored logical row `k` at permuted row p where perm(p % 16) == k % 16
        const int t = k & 15;
        // inverse of perm(t) = 8*((t%4)/2) + t%2 + 2*(t/4)
        const int p16 = ((t & 7) >> 1) * 4 + ((t >> 3) << 1) + (t & 1);
        const int p = (k & ~15) + p16;
        size_t pos = (size_t)(n >> 1) * (2 * (size_t)K) + 128 * (p >> 6) + 64 * (n & 1) + (p & 63);
        const int in_word = (int)(pos & 3);
        pos = (pos & ~(size_t)3) | (in_word == 1 ? 2 : (in_word == 2 ? 1 : in_word));
        dst[e] = ref[pos];
    }
}

}  // namespace

int launch_quantize_w8(const void* w, bool fp32, int K, int N, int8_t* q_rowmajor, void* packed, void* scales,
                       int variant, float* amax_ws, cudaStream_t stream)
{
    EET_CUDA(cudaMemsetAsync(amax_ws, 0, sizeof(float) * N, stream));
    const dim3 g1((N + 255) / 256, K / 64), g2(N / 64, (K / 64 + (fp32 ? 1 : 3)) / (fp32 ? 2 : 4));
    const bool vec = reinterpret_cast<uintptr_t>(amax_ws) % 16 == 0;
    if (fp32) {
        colmax_kernel<float><<<g1, 256, 0, stream>>>((const float*)w, K, N, amax_ws);
        EET_LAUNCH_CHECK();
        EET_CUDA(launch_pdl(vec ? quant_pack_kernel<float, 1, true> : quant_pack_kernel<float, 1, false>, g2, dim3(256), 0, stream,
                            (const float*)w, K, N, (const float*)amax_ws, variant, q_rowmajor, (uint8_t*)packed, scales));
    }
    else {
        colmax_kernel<__half><<<g1, 256, 0, stream>>>((const __half*)w, K, N, amax_ws);
        EET_LAUNCH_CHECK();
        EET_CUDA(launch_pdl(vec ? quant_pack_kernel<__half, 2, true> : quant_pack_kernel<__half, 2, false>, g2, dim3(256), 0, stream,
                            (const __half*)w, K, N, (const float*)amax_ws, variant, q_rowmajor, (uint8_t*)packed, scales));
    }
    return 0;
}

int launch_pack_w8(const int8_t* q, int K, int N, void* packed, cudaStream_t stream)
{
    pack_kernel<<<dim3(N / 64, K / 64), 256, 0, stream>>>(q, K, N, (uint8_t*)packed);
    EET_LAUNCH_CHECK();
    return 0;
}

int launch_unpack_w8(const void* packed, int K, int N, int8_t* q, cudaStream_t stream)
{
    unpack_kernel<<<dim3(N / 64, K / 64), 256, 0, stream>>>((const uint8_t*)packed, K, N, q);
    EET_LAUNCH_CHECK();
    return 0;
}

int launch_repack_ref_w8(const void* ref_packed, int K, int N, void* packed, cudaStream_t stream)
{
    repack_ref_kernel<<<dim3(N / 64, K / 64), 256, 0, stream>>>((const uint8_t*)ref_packed, K, N, (uint8_t*)packed);
    EET_LAUNCH_CHECK();
    return 0;
}

}  // namespace eet
