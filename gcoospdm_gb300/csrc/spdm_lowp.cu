// spdm_lowp.cu -- the reduced-precision forms of the multiply on the FMA
// pipes (the tensor-core engine for block-structured matrices is in
// spdm_tc.cu). Same CTA/warp mapping as the FP32 row walk (one warp per row,
// the CTA's entries staged to shared memory with cp.async.bulk and used for
// several column tiles), with B read in a narrower format:
//   BF16        B as bf16 (8 columns per 128-bit load), A values rounded to
//               bf16, FP32 accumulation (the mixed-precision bf16 FMA of
//               sm_100+: no widening of the B values);
//   SPLIT_BF16  B = Bh + Bl and a = ah + al as bf16 pairs; acc += ah*Bh +
//               ah*Bl + al*Bh (three products, FP32 accumulation) -- FP32-level
//               accuracy from bf16 operands;
//   FP8_B       B as FP8 E4M3 scaled per column (s_j = the smallest power of
//               two with max_c |B[c][j]| / s_j <= 448), 16 columns per
//               128-bit load (narrow B: each value as the BF16 that equals
//               it), A kept FP32; the scale is applied once to the
//               accumulated column.
// B is converted into the handle's workspace by a pre-pass kernel per call.
#include <cuda_bf16.h>
#include <cuda_fp8.h>

#include "handle.hpp"

namespace gcoo {

struct LowpWork {
    DevBuf<uint16_t> bf;     // k*n bf16 (FP8: E4M3 values as bf16)
    DevBuf<uint32_t> split;  // k*n (hi | lo << 16) bf16 pairs
    DevBuf<uint8_t> f8;      // k*n e4m3 (wide B and the group walk)
    DevBuf<float> scale;     // n column scales
    DevBuf<unsigned> amax;   // n column absmax (float bits)
};

void destroy_lowp_work(LowpWork *w) { delete w; }

namespace {

constexpr int kChunk = 2048;
// Four-warp CTAs per SM (64 registers a thread) and entries per batch of the
// row walk. 4096^2 at 2 %, n = 4096 (us; BF16 / split / FP8, the latter two
// before their mixed-precision FMAs: 324 / 173 with them): batches of eight
// 152 / 398 / 192, of four 159 / 418 / 196, ten CTAs 154 / 406 / 200; before,
// two warps per row, a staging per tile, 16 KB of shared memory and the tail
// entry by entry: 220 / 443 / 222.
constexpr int kLowpCtas = 8, kLowpU = 8;
constexpr int kLowpCols = 1024; // columns per staging at most (512: 1-2 % slower)

__device__ __forceinline__ float bf_lo(uint32_t w) { return __uint_as_float(w << 16); }
__device__ __forceinline__ float bf_hi(uint32_t w) { return __uint_as_float(w & 0xffff0000u); }

enum Form { kBF16 = 1, kSplit = 2, kFP8 = 3, kFP8Wide = 4 };

// Columns per lane for each form (one 128-bit load per entry).
template <int F> struct FormTraits;
template <> struct FormTraits<kBF16> { static constexpr int V = 8; using T = uint16_t; };
template <> struct FormTraits<kSplit> { static constexpr int V = 4; using T = uint32_t; };
template <> struct FormTraits<kFP8> { static constexpr int V = 16; using T = uint8_t; };
template <> struct FormTraits<kFP8Wide> { static constexpr int V = 8; using T = uint16_t; };

// acc + a * b with bf16 a and b, one rounding (the mixed-precision FMA of
// sm_100+): the same result as fmaf on the widened values, since a product of
// two bf16 values is exact in FP32 -- without widening each B value first.
__device__ __forceinline__ float fma_bf16(uint16_t a, uint16_t b, float c)
{
    float d;
    asm("fma.rn.f32.bf16 %0, %1, %2, %3;" : "=f"(d) : "h"(a), "h"(b), "f"(c));
    return d;
}

// Two FP32 sums, each its own fma (one rounding each).
__device__ __forceinline__ void fma_pair(uint64_t &c, uint64_t a, float b0, float b1)
{
    uint64_t b;
    asm("mov.b64 %0, {%1, %2};" : "=l"(b) : "f"(b0), "f"(b1));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}

__device__ __forceinline__ uint64_t dup_f32(float a)
{
    uint64_t d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(a));
    return d;
}

__device__ __forceinline__ void split_f32x2(uint64_t x, float &lo, float &hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(x));
}

// An FP16 value in FP32 (1 * h - 0, exact, signed zeros too) by the
// mixed-precision FMA, which runs at the FMA's rate; the conversion
// instruction at half of it bounded the FP8 rows (4096^2 at 2 %, n = 4096: 189
// us with it, 173 without).
__device__ __forceinline__ float widen_f16(uint16_t h)
{
    float d;
    asm("fma.rn.f32.f16 %0, %1, %2, %3;" : "=f"(d) : "h"(h), "h"(static_cast<uint16_t>(0x3c00)), "f"(-0.0f));
    return d;
}

// A lane's V sums of one row tile, as the form multiplies them. BF16 and
// split-BF16: mixed-precision FMAs on the bf16 halves as they are (split, 4096^2
// at 2 %, n = 4096: 324 us; its halves widened and packed FMAs, half as many
// instructions for the products, 399). FP8: packed FMAs, A being FP32.
template <int F>
struct Sums {
    static constexpr int V = FormTraits<F>::V;
    uint64_t s[V / 2];
    __device__ __forceinline__ void clear()
    {
#pragma unroll
        for (int v = 0; v < V / 2; ++v)
            s[v] = 0ull;
    }
    __device__ __forceinline__ float get(int v) const
    {
        float lo, hi;
        split_f32x2(s[v / 2], lo, hi);
        return v & 1 ? hi : lo;
    }
    __device__ __forceinline__ void add(float val, const uint4 &w)
    {
        const uint32_t x[4] = {w.x, w.y, w.z, w.w};
        if constexpr (F == kFP8) {
            const uint64_t a = dup_f32(val);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const __half2_raw h01 = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(x[i] & 0xffffu), __NV_E4M3);
                const __half2_raw h23 = __nv_cvt_fp8x2_to_halfraw2(static_cast<__nv_fp8x2_storage_t>(x[i] >> 16), __NV_E4M3);
                fma_pair(s[(2 * i) % (V / 2)], a, widen_f16(h01.x), widen_f16(h01.y));
                fma_pair(s[(2 * i + 1) % (V / 2)], a, widen_f16(h23.x), widen_f16(h23.y));
            }
        } else {
            const uint64_t a = dup_f32(val);
#pragma unroll
            for (int i = 0; i < 4; ++i)
                fma_pair(s[i], a, bf_lo(x[i]), bf_hi(x[i]));
        }
    }
};

// BF16 and split-BF16
template <int F>
struct MixedSums {
    static constexpr int V = FormTraits<F>::V;
    float s[V];
    __device__ __forceinline__ void clear()
    {
#pragma unroll
        for (int v = 0; v < V; ++v)
            s[v] = 0.0f;
    }
    __device__ __forceinline__ float get(int v) const { return s[v]; }
    __device__ __forceinline__ void add(float val, const uint4 &w)
    {
        const uint32_t x[4] = {w.x, w.y, w.z, w.w};
        const __nv_bfloat16 a = __float2bfloat16_rn(val);
        const uint16_t ah = __bfloat16_as_ushort(a);
        if constexpr (F == kBF16) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                s[2 * i] = fma_bf16(ah, static_cast<uint16_t>(x[i] & 0xffffu), s[2 * i]);
                s[2 * i + 1] = fma_bf16(ah, static_cast<uint16_t>(x[i] >> 16), s[2 * i + 1]);
            }
        } else {
            const uint16_t al = __bfloat16_as_ushort(__float2bfloat16_rn(val - __bfloat162float(a)));
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint16_t bh = static_cast<uint16_t>(x[i] & 0xffffu), bl = static_cast<uint16_t>(x[i] >> 16);
                s[i] = fma_bf16(ah, bh, s[i]);
                s[i] = fma_bf16(ah, bl, s[i]);
                s[i] = fma_bf16(al, bh, s[i]);
            }
        }
    }
};
template <>
struct Sums<kBF16> : MixedSums<kBF16> {};
template <>
struct Sums<kSplit> : MixedSums<kSplit> {};

template <int F, int U>
__device__ __forceinline__ void lowp_batch(const Entry *__restrict__ s, const typename FormTraits<F>::T *__restrict__ Bj,
                                           int64_t n, Sums<F> &sum)
{
    Entry e[U];
    uint4 w[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
        e[u] = s[u];
#pragma unroll
    for (int u = 0; u < U; ++u)
        w[u] = __ldg(reinterpret_cast<const uint4 *>(Bj + static_cast<int64_t>(e[u].col) * n));
#pragma unroll
    for (int u = 0; u < U; ++u)
        sum.add(e[u].val, w[u]);
}

// One row's entries in order, U B loads in flight, the tail in halves too.
template <int F, int U>
__device__ __forceinline__ void row_chain_lowp(const Entry *__restrict__ s, int cnt,
                                               const typename FormTraits<F>::T *__restrict__ Bj, int64_t n, Sums<F> &sum)
{
    int i = 0;
#pragma unroll 1
    for (; i + U <= cnt; i += U)
        lowp_batch<F, U>(s + i, Bj, n, sum);
    if (U == 8 && i + 4 <= cnt) {
        lowp_batch<F, 4>(s + i, Bj, n, sum);
        i += 4;
    }
    if (i + 2 <= cnt) {
        lowp_batch<F, 2>(s + i, Bj, n, sum);
        i += 2;
    }
    if (i < cnt)
        lowp_batch<F, 1>(s + i, Bj, n, sum);
}

template <int F>
__device__ __forceinline__ void lowp_store(float *out, const float *__restrict__ scale, const Sums<F> &sum)
{
    constexpr int V = FormTraits<F>::V;
#pragma unroll
    for (int v = 0; v < V; v += 4) {
        float4 o = make_float4(sum.get(v), sum.get(v + 1), sum.get(v + 2), sum.get(v + 3));
        if constexpr (F == kFP8 || F == kFP8Wide) {
            const float4 s = __ldg(reinterpret_cast<const float4 *>(scale + v));
            o.x *= s.x; o.y *= s.y; o.z *= s.z; o.w *= s.w;
        }
        *reinterpret_cast<float4 *>(out + v) = o;
    }
}

// One CTA per (`cpg` rows, col_iters column tiles), one warp per row: the
// CTA's entries are staged once and each warp walks its row over all tiles
// from there, as in the FP32 row walk; entries beyond the staged chunk (its
// size is the launch's) are staged piecewise for each tile in turn. n must be
// a multiple of the form's V and B / C 16-byte aligned (host checks).
template <int F>
__global__ void __launch_bounds__(128, kLowpCtas)
spdm_lowp_kernel(const Entry *__restrict__ packed, const int32_t *__restrict__ row_ptr, int64_t m, int32_t cpg,
                 const typename FormTraits<F>::T *__restrict__ B, const float *__restrict__ col_scale, int64_t n,
                 float *__restrict__ C, int32_t col_iters, int32_t chunk, uint32_t *__restrict__ status)
{
    grid_wait_previous();
    row_ptr = written(row_ptr);
    col_scale = written(col_scale);
    constexpr int V = FormTraits<F>::V;
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem);
    Entry *s_nz = reinterpret_cast<Entry *>(smem + 128);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t r0 = static_cast<int64_t>(blockIdx.x) * cpg;
    const int64_t r_end = r0 + cpg < m ? r0 + cpg : m;
    const int64_t row = r0 + warp;
    const bool has_row = row < r_end;
    const int64_t j0 = static_cast<int64_t>(blockIdx.y) * col_iters * (32 * V) + static_cast<int64_t>(lane) * V;
    const int64_t gs = row_ptr[r0], ge = row_ptr[r_end];
    const int64_t rs = has_row ? row_ptr[row] : 0, re = has_row ? row_ptr[row + 1] : 0;
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        fence_mbar_init();
    }
    __syncthreads();
    const int64_t nchunks = (ge - gs + chunk - 1) / chunk;
    const bool once = nchunks <= 1;
    bool ok = true;
    uint32_t phase = 0;
    for (int it = 0; it < (once ? 1 : col_iters) && ok; ++it) {
        const int64_t j = j0 + it * (32 * V);
        Sums<F> sum;
        sum.clear();
        for (int64_t ch = 0; ch < nchunks; ++ch, ++phase) {
            const int64_t cs = gs + ch * chunk;
            const int64_t ce = cs + chunk < ge ? cs + chunk : ge;
            const int64_t a0 = cs & ~static_cast<int64_t>(1);
            const int64_t a1 = (ce + 1) & ~static_cast<int64_t>(1);
            if (threadIdx.x == 0) {
                fence_proxy_async();
                const uint32_t bytes = static_cast<uint32_t>((a1 - a0) * static_cast<int64_t>(sizeof(Entry)));
                mbar_arrive_expect_tx(bar, bytes);
                bulk_g2s(s_nz, packed + a0, bytes, bar);
            }
            const bool waited = mbar_wait(bar, phase & 1);
            ok = __syncthreads_and(waited) != 0;
            if (!ok) {
                if (threadIdx.x == 0)
                    atomicOr(status, kStatusWaitTimeout);
                mbar_wait(bar, phase & 1);
                break;
            }
            if (once)
                break; // staged for good: every tile below
            const int64_t lo = rs > cs ? rs : cs, hi = re < ce ? re : ce;
            if (j < n && lo < hi)
                row_chain_lowp<F, kLowpU>(s_nz + (lo - a0), static_cast<int>(hi - lo), B + j, n, sum);
            __syncthreads();
        }
        if (!once && has_row && j < n && ok)
            lowp_store<F>(C + row * n + j, col_scale + j, sum);
    }
    if (!once || !has_row || !ok)
        return;
    const Entry *s_row = s_nz + (rs - (gs & ~static_cast<int64_t>(1)));
    const int cnt = static_cast<int>(re - rs);
#pragma unroll 1
    for (int it = 0; it < col_iters; ++it) {
        const int64_t j = j0 + it * (32 * V);
        if (j >= n)
            break;
        Sums<F> sum;
        sum.clear();
        row_chain_lowp<F, kLowpU>(s_row, cnt, B + j, n, sum);
        lowp_store<F>(C + row * n + j, col_scale + j, sum);
    }
}

// ---- B pre-pass kernels (grid-stride over k*n / 4) ----------------------------------
__global__ void prep_bf16_kernel(const float4 *__restrict__ B, uint2 *__restrict__ out, int64_t n4)
{
    grid_launch_next();
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n4;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const float4 v = __ldcs(B + i);
        const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y);
        const __nv_bfloat162 b = __floats2bfloat162_rn(v.z, v.w);
        out[i] = make_uint2(*reinterpret_cast<const uint32_t *>(&a), *reinterpret_cast<const uint32_t *>(&b));
    }
}

__global__ void prep_split_kernel(const float4 *__restrict__ B, uint4 *__restrict__ out, int64_t n4)
{
    grid_launch_next();
    for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n4;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const float4 v = __ldcs(B + i);
        const float x[4] = {v.x, v.y, v.z, v.w};
        uint32_t w[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const __nv_bfloat16 h = __float2bfloat16_rn(x[q]);
            const __nv_bfloat16 l = __float2bfloat16_rn(x[q] - __bfloat162float(h));
            w[q] = static_cast<uint32_t>(*reinterpret_cast<const uint16_t *>(&h)) |
                   (static_cast<uint32_t>(*reinterpret_cast<const uint16_t *>(&l)) << 16);
        }
        out[i] = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// FP8 passes over B: a CTA takes 128 columns x 64 rows, a warp 8 of the rows,
// a lane 4 of the columns; the 8 rows' loads are in flight together (FP8 rows
// of 4096^2 at 2 %, n = 4096: 164 us; 4 rows 165, 16 169, 32 176).
constexpr int kStripCols = 128, kStripRows = 64, kWarpRows = 8;

// Column absmax: one atomic per column and CTA.
__global__ void __launch_bounds__(256)
colmax_kernel(const float *__restrict__ B, int64_t k, int64_t n, unsigned *__restrict__ amax)
{
    grid_launch_next();
    __shared__ float s_max[kStripRows / kWarpRows][kStripCols];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t j = static_cast<int64_t>(blockIdx.x) * kStripCols + lane * 4;
    const int64_t c0 = static_cast<int64_t>(blockIdx.y) * kStripRows + warp * kWarpRows;
    float4 mx = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 v[kWarpRows];
#pragma unroll
    for (int i = 0; i < kWarpRows; ++i)
        v[i] = j < n && c0 + i < k ? __ldg(reinterpret_cast<const float4 *>(B + (c0 + i) * n + j)) : mx;
#pragma unroll
    for (int i = 0; i < kWarpRows; ++i) {
        mx.x = fmaxf(mx.x, fabsf(v[i].x)); mx.y = fmaxf(mx.y, fabsf(v[i].y));
        mx.z = fmaxf(mx.z, fabsf(v[i].z)); mx.w = fmaxf(mx.w, fabsf(v[i].w));
    }
    *reinterpret_cast<float4 *>(&s_max[warp][lane * 4]) = mx;
    __syncthreads();
    const int t = threadIdx.x;
    const int64_t jt = static_cast<int64_t>(blockIdx.x) * kStripCols + t;
    if (t < kStripCols && jt < n) {
        float x = 0.0f;
#pragma unroll
        for (int w = 0; w < kStripRows / kWarpRows; ++w)
            x = fmaxf(x, s_max[w][t]);
        atomicMax(amax + jt, __float_as_uint(x));
    }
}

// Per-column scale: the smallest power of two s with absmax / s <= 448 (the
// largest E4M3 value). A power of two divides exactly, so both engines see
// the same E4M3 values, and the tensor engine can fold s into its BF16 tiles
// without a rounding (an E4M3 value times a power of two is a BF16 value).
__device__ __forceinline__ float fp8_scale(unsigned amax_bits)
{
    const float a = __uint_as_float(amax_bits);
    float s = 1.0f;
    if (a > 0.0f && a < INFINITY) {
        int e = 0;
        const float mant = frexpf(a / 448.0f, &e); // a / 448 = mant * 2^e, mant in [0.5, 1)
        s = ldexpf(1.0f, mant == 0.5f ? e - 1 : e);
    }
    return s;
}

__global__ void scale_kernel(const unsigned *__restrict__ amax, float *__restrict__ scale, int64_t n)
{
    const int64_t j = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (j < n)
        scale[j] = fp8_scale(amax[j]);
}

// B in units of its columns' scales as E4M3; the scales, computed where they
// are used, are written once for the multiply. WIDE: each E4M3 value as the
// BF16 that equals it.
template <bool WIDE>
__global__ void __launch_bounds__(256)
prep_fp8_kernel(const float *__restrict__ B, const unsigned *__restrict__ amax, float *__restrict__ scale,
                void *__restrict__ out, int64_t k, int64_t n)
{
    grid_wait_previous();
    amax = written(amax);
    grid_launch_next();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t j = static_cast<int64_t>(blockIdx.x) * kStripCols + lane * 4;
    const int64_t c0 = static_cast<int64_t>(blockIdx.y) * kStripRows + warp * kWarpRows;
    if (j >= n)
        return;
    float4 v[kWarpRows];
#pragma unroll
    for (int i = 0; i < kWarpRows; ++i)
        v[i] = c0 + i < k ? __ldcs(reinterpret_cast<const float4 *>(B + (c0 + i) * n + j)) : make_float4(0.f, 0.f, 0.f, 0.f);
    const uint4 am = *reinterpret_cast<const uint4 *>(amax + j);
    const float s[4] = {fp8_scale(am.x), fp8_scale(am.y), fp8_scale(am.z), fp8_scale(am.w)};
    if (blockIdx.y == 0 && warp == 0)
        *reinterpret_cast<float4 *>(scale + j) = make_float4(s[0], s[1], s[2], s[3]);
    // a power of two in the normal range has an exact reciprocal, so x * inv
    // is x / s exactly; otherwise divide
    bool by_inv = true;
    float inv[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        by_inv = by_inv && s[q] >= 1.17549435e-38f && s[q] <= 8.50705917e37f;
        inv[q] = 1.0f / s[q];
    }
#pragma unroll
    for (int i = 0; i < kWarpRows; ++i) {
        const float x[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
        __nv_fp8_storage_t f[4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
            f[q] = __nv_cvt_float_to_fp8(by_inv ? x[q] * inv[q] : x[q] / s[q], __NV_SATFINITE, __NV_E4M3);
        if (c0 + i >= k)
            break;
        if constexpr (WIDE) {
            uint32_t w[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) // an E4M3 value is an FP16 value and a BF16 value
                w[q] = __float_as_uint(__half2float(__half(__nv_cvt_fp8_to_halfraw(f[q], __NV_E4M3)))) >> 16;
            *reinterpret_cast<uint2 *>(static_cast<uint16_t *>(out) + (c0 + i) * n + j) =
                make_uint2(w[0] | (w[1] << 16), w[2] | (w[3] << 16));
        } else {
            *reinterpret_cast<uint32_t *>(static_cast<uint8_t *>(out) + (c0 + i) * n + j) =
                f[0] | (static_cast<uint32_t>(f[1]) << 8) | (static_cast<uint32_t>(f[2]) << 16) | (static_cast<uint32_t>(f[3]) << 24);
        }
    }
}

unsigned grid_for(int64_t items, int threads)
{
    int64_t b = (items + threads - 1) / threads;
    if (b > 152 * 32)
        b = 152 * 32;
    return static_cast<unsigned>(b < 1 ? 1 : b);
}

} // namespace

static dim3 strip_grid(int64_t k, int64_t n)
{
    return dim3(static_cast<unsigned>((n + kStripCols - 1) / kStripCols),
                static_cast<unsigned>((k + kStripRows - 1) / kStripRows));
}

static cudaError_t launch_colmax(const float *B, int64_t k, int64_t n, unsigned *amax, cudaStream_t st)
{
    const cudaError_t e = cudaMemsetAsync(amax, 0, sizeof(unsigned) * static_cast<size_t>(n), st);
    if (e != cudaSuccess)
        return e;
    colmax_kernel<<<strip_grid(k, n), 256, 0, st>>>(B, k, n, amax);
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_fp8_scales(const float *B, int64_t k, int64_t n, unsigned *amax, float *scale, cudaStream_t st)
{
    const cudaError_t e = launch_colmax(B, k, n, amax, st);
    if (e != cudaSuccess)
        return e;
    scale_kernel<<<static_cast<unsigned>((n + 255) / 256), 256, 0, st>>>(amax, scale, n);
    count_launches(1);
    return cudaGetLastError();
}

// Width constraint of each form on the FMA engine.
int lowp_vec(gcoo_precision prec) { return prec == GCOO_PREC_BF16 ? 8 : prec == GCOO_PREC_SPLIT_BF16 ? 4 : 16; }

// The group walk only where the caller asks for it: on 2946 multiplies of
// matrices whose groups share columns (blocks of 2 to 64 rows, aligned or not,
// with holes, unstructured from 25 %; 64^2 to 10000^2, n 16 to 2048) the row
// walk was up to 14 times as fast, 2.3 on average, and at most 13 % slower on
// the smallest (19 us against 17).
static bool lowp_groups(const gcoo_handle *h) { return h->p.fp32_order == 2 && group_order_chosen(h); }

// FP8-B: B's E4M3 values as one byte or as the BF16 that equals each. Bytes:
// half the gather, but two and a half instructions a value, and a warp's 16-byte
// loads span 512 columns; BF16: one and a half instructions. Measured (us;
// bytes / BF16): 4096^2 at 2 %, n = 4096 175 / 198, n = 1024 55 / 62, n = 512 39 /
// 41, n = 256 36 / 30; 2048^2 at 0.5 %, n = 512 21 / 20; 8192 x 1200 at 3 %,
// n = 128 33 / 27. The group walk reads bytes.
constexpr int64_t kFp8WideCols = 512;
static bool fp8_wide(const gcoo_handle *h, int64_t n) { return n <= kFp8WideCols && !lowp_groups(h); }

gcoo_status lowp_prepare(gcoo_handle *h, int64_t n, gcoo_precision prec)
{
    if (!h->lowp)
        h->lowp = new (std::nothrow) LowpWork();
    if (!h->lowp)
        return fail(GCOO_ERROR_ALLOC, "host allocation failed");
    const size_t kn = static_cast<size_t>(h->k) * static_cast<size_t>(n);
    bool ok = true;
    if (prec == GCOO_PREC_BF16)
        ok = h->lowp->bf.ensure(kn);
    else if (prec == GCOO_PREC_SPLIT_BF16)
        ok = h->lowp->split.ensure(kn);
    else
        // a width prepared once serves every smaller one, in either format
        ok = (lowp_groups(h) ||
              h->lowp->bf.ensure(static_cast<size_t>(h->k) * static_cast<size_t>(n < kFp8WideCols ? n : kFp8WideCols))) &&
             (fp8_wide(h, n) || h->lowp->f8.ensure(kn)) && h->lowp->scale.ensure(n) && h->lowp->amax.ensure(n);
    return ok ? GCOO_SUCCESS : fail(GCOO_ERROR_ALLOC, "device allocation of the form workspace failed");
}

// Converts B into the form's workspace (also used by the tensor engine for FP8 scales).
gcoo_status lowp_convert_b(gcoo_handle *h, const float *dB, int64_t n, gcoo_precision prec, cudaStream_t st)
{
    const int64_t n4 = h->k * n / 4;
    LowpWork *w = h->lowp;
    if (prec == GCOO_PREC_BF16) {
        prep_bf16_kernel<<<grid_for(n4, 256), 256, 0, st>>>(reinterpret_cast<const float4 *>(dB),
                                                            reinterpret_cast<uint2 *>(w->bf.ptr), n4);
        count_launches(1);
    } else if (prec == GCOO_PREC_SPLIT_BF16) {
        prep_split_kernel<<<grid_for(n4, 256), 256, 0, st>>>(reinterpret_cast<const float4 *>(dB),
                                                             reinterpret_cast<uint4 *>(w->split.ptr), n4);
        count_launches(1);
    } else {
        GCOO_CUDA(launch_colmax(dB, h->k, n, w->amax.ptr, st));
        if (!fp8_wide(h, n))
            GCOO_CUDA(launch_after(prep_fp8_kernel<false>, strip_grid(h->k, n), dim3(256), 0, st, dB, w->amax.ptr,
                                   w->scale.ptr, w->f8.ptr, h->k, n));
        else
            GCOO_CUDA(launch_after(prep_fp8_kernel<true>, strip_grid(h->k, n), dim3(256), 0, st, dB, w->amax.ptr,
                                   w->scale.ptr, w->bf.ptr, h->k, n));
        count_launches(1);
    }
    GCOO_LAUNCH("B conversion kernel");
    return GCOO_SUCCESS;
}

gcoo_status lowp_spdm(gcoo_handle *h, int64_t n, float *dC, gcoo_precision prec, cudaStream_t st)
{
    const bool wide = prec == GCOO_PREC_FP8_B && fp8_wide(h, n);
    const int V = wide ? 8 : lowp_vec(prec); // columns per lane
    if (h->p.rows_per_group > 16)
        return fail(GCOO_ERROR_UNSUPPORTED, "reduced-precision forms on the FMA engine support rows_per_group <= 16");
    LowpWork *w = h->lowp;
    if (prec != GCOO_PREC_SPLIT_BF16 && n % 8 == 0 && lowp_groups(h)) {
        // rows of a group share columns: decode each B segment once per group
        cudaError_t e = launch_spdm_lowp_group(
            h->vals.ptr, h->rc.ptr, h->rc.ptr + h->nnz, h->group_index(), h->m, h->ng,
            prec == GCOO_PREC_BF16 ? static_cast<const void *>(w->bf.ptr) : static_cast<const void *>(w->f8.ptr),
            w->scale.ptr, n, dC, prec, st);
        if (e != cudaSuccess)
            return cuda_fail(e, "spdm_group_kernel launch (reduced precision)");
        return GCOO_SUCCESS;
    }
    // one warp per row, up to four rows per CTA (any number gives the same
    // chains), fewer where that makes their entries fit one staging
    int rows = h->p.rows_per_group < 4 ? h->p.rows_per_group : 4;
    while (rows > 1 && h->max_row_nnz * rows + 2 > kChunk)
        rows /= 2;
    const int64_t most = h->max_row_nnz * rows + 2;
    const int chunk = static_cast<int>(most < kChunk ? (most < 64 ? 64 : most) : kChunk);
    // as the FP32 row walk: several tiles per staging, at least four waves of CTAs
    const int64_t tile = 32 * V, tiles = (n + tile - 1) / tile, groups = (h->m + rows - 1) / rows;
    const int64_t resident = static_cast<int64_t>(device_sms()) * kLowpCtas;
    int64_t ci = groups * tiles / (4 * resident);
    ci = ci > kLowpCols / tile ? kLowpCols / tile : ci;
    ci = ci < 1 ? 1 : ci;
    while ((tiles + ci - 1) / ci > 65535)
        ci *= 2;
    const int64_t ny = (tiles + ci - 1) / ci;
    // the widest B of this engine: 65535 strips of 8 warps over a group's rows
    const int64_t strip = 32 * lowp_vec(prec) * (h->p.rows_per_group < 8 ? 8 / h->p.rows_per_group : 1);
    if ((n + strip - 1) / strip > 65535 || groups > 0x7fffffffLL)
        return cuda_fail(cudaErrorInvalidConfiguration, "spdm_lowp_kernel launch");
    dim3 grid(static_cast<unsigned>(groups), static_cast<unsigned>(ny));
    const size_t smem = 128 + (static_cast<size_t>(chunk) + 2) * sizeof(Entry);
#define GCOO_LOWP(F, DATA, SCALE)                                                                               \
    GCOO_CUDA(launch_after(spdm_lowp_kernel<F>, grid, dim3(rows * 32), smem, st, h->packed.ptr, h->row_ptr.ptr,  \
                           h->m, rows, DATA, SCALE, n, dC, static_cast<int32_t>(ci), chunk, h->status.ptr))
    if (prec == GCOO_PREC_BF16)
        GCOO_LOWP(kBF16, w->bf.ptr, nullptr);
    else if (prec == GCOO_PREC_SPLIT_BF16)
        GCOO_LOWP(kSplit, w->split.ptr, nullptr);
    else if (wide)
        GCOO_LOWP(kFP8Wide, w->bf.ptr, w->scale.ptr);
    else
        GCOO_LOWP(kFP8, w->f8.ptr, w->scale.ptr);
#undef GCOO_LOWP
    count_launches(1);
    GCOO_LAUNCH("spdm_lowp_kernel");
    return GCOO_SUCCESS;
}

} // namespace gcoo
