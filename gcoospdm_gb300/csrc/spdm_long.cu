// spdm_long.cu -- the FP32 multiply of the long rows of a skewed matrix.
//
// A row is one sequential fmaf chain per output element (the reference's
// accumulation order, src/gcoo_spdm_kernels.cu:92-158), so a row of a few
// thousand entries is a long dependent chain; in the row kernel it keeps
// only a handful of B loads in flight and sets the whole launch's length.
// Here a CTA owns (long row, tile of 32 or 128 columns). Its copy warps keep a
// ring of the row's B pieces in flight in shared memory with cp.async:
//   * the row's entries arrive 2 kDepth steps ahead (an 8-byte copy per
//     entry), so the columns of the B pieces are on chip when their copies
//     are issued;
//   * the B pieces (a tile's columns of a B row per entry) arrive kDepth steps
//     of kBatch entries ahead;
// and its first warp does nothing but run its columns' chains over the landed
// step, in the row's column order starting from 0.0f -- the same fmaf chain
// as the row kernel and the reference, so results are bit-identical.
//
// What bounds it is instruction issue along one row: with one warp copying
// and multiplying (17 ns per entry) a row of 4096 took 70 us whatever else
// ran; with the copies in warps of their own and 128 entries per barrier it
// takes 24. Whole multiplies with Zipf rows of up to 4096 entries, us before
// and after: 16346 rows, n = 192 73 -> 44, n = 64 71 -> 33; 8192 rows, n = 256
// 68 -> 34; 65536 rows (1.2 M entries), n = 256 140 -> 119.
// Rows of at least long_row_min() = 256 entries come here, on the caller's
// stream; the others go to spdm_short_kernel (spdm_fp32.cu), which runs beside
// this kernel on the handle's side stream.
#include <algorithm>

#include "internal.cuh"

namespace gcoo {

namespace {

__device__ __forceinline__ void cp_async16(void *dst, const void *src)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async8(void *dst, const void *src)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__global__ void collect_long_kernel(const int32_t *__restrict__ row_ptr, int64_t m, int32_t min_len,
                                    int32_t *__restrict__ list, int64_t cap, unsigned long long *__restrict__ count)
{
    for (int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r < m;
         r += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int32_t len = row_ptr[r + 1] - row_ptr[r];
        if (len >= min_len) {
            const unsigned long long i = atomicAdd(count, 1ull);
            atomicAdd(count + 1, static_cast<unsigned long long>(len)); // the long rows' entries
            if (static_cast<int64_t>(i) < cap)
                list[i] = static_cast<int32_t>(r);
        }
    }
}

// The collected rows by length, longest first (to within kClassLen entries):
// one CTA counts the classes, then places the rows.
constexpr int kClasses = 64, kClassLen = 64, kOrderThreads = 1024;

__global__ void __launch_bounds__(kOrderThreads)
order_long_kernel(const int32_t *__restrict__ row_ptr, const int32_t *__restrict__ from, int64_t cap,
                  const unsigned long long *__restrict__ count, int32_t *__restrict__ list)
{
    __shared__ int s_at[kClasses];
    const int64_t n = static_cast<int64_t>(count[0]) < cap ? static_cast<int64_t>(count[0]) : cap;
    const auto cls = [&](int32_t r) { // class 0: the longest
        const int c = (row_ptr[r + 1] - row_ptr[r]) / kClassLen;
        return kClasses - 1 - (c < kClasses ? c : kClasses - 1);
    };
    if (threadIdx.x < kClasses)
        s_at[threadIdx.x] = 0;
    __syncthreads();
    for (int64_t i = threadIdx.x; i < n; i += kOrderThreads)
        atomicAdd(&s_at[cls(from[i])], 1);
    __syncthreads();
    if (threadIdx.x == 0) {
        int run = 0;
        for (int c = 0; c < kClasses; ++c) {
            const int x = s_at[c];
            s_at[c] = run;
            run += x;
        }
    }
    __syncthreads();
    for (int64_t i = threadIdx.x; i < n; i += kOrderThreads) {
        const int32_t r = from[i];
        list[atomicAdd(&s_at[cls(r)], 1)] = r;
    }
}

// acc (two columns) += {val, val} * b (two columns), each as fmaf
__device__ __forceinline__ void fma_pair(unsigned long long &acc, unsigned long long val, unsigned long long b)
{
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(val), "l"(b));
}

// V columns of shared memory in registers, and their chains
template <int V>
struct Chain;
template <>
struct Chain<4> {
    unsigned long long lo, hi; // two columns each
    __device__ __forceinline__ void zero() { lo = hi = 0ull; }
    __device__ __forceinline__ void add(float val, const float *b)
    {
        unsigned long long vv;
        asm("mov.b64 %0, {%1, %1};" : "=l"(vv) : "f"(val));
        const ulonglong2 t = *reinterpret_cast<const ulonglong2 *>(b);
        fma_pair(lo, vv, t.x);
        fma_pair(hi, vv, t.y);
    }
    __device__ __forceinline__ float at(int v) const
    {
        const unsigned long long two = v < 2 ? lo : hi;
        return __uint_as_float(static_cast<unsigned>(v & 1 ? two >> 32 : two));
    }
};
template <>
struct Chain<1> {
    float acc;
    __device__ __forceinline__ void zero() { acc = 0.0f; }
    __device__ __forceinline__ void add(float val, const float *b) { acc = fmaf(val, *b, acc); }
    __device__ __forceinline__ float at(int) const { return acc; }
};

template <int W>
__device__ __forceinline__ void cp_async_w(void *dst, const void *src)
{
    if (W == 4)
        cp_async16(dst, src);
    else if (W == 2)
        cp_async8(dst, src);
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}

// Columns per lane V: 1 where the CTAs are few and a row's chain is the time
// (a step of 32 entries instead of 128: 10 % more), 4 where there are many and
// their instructions are (half as many per column; 65536 rows, n = 256 119 us,
// V = 1 136, V = 2 123-126). Two copy warps instead of four: 1-10 % more;
// eight at V = 4: 7 % more.
constexpr int kCopyWarps = 4;
template <int V>
constexpr int kBatch = V == 1 ? 128 : 32; // entries per step
template <int V>
constexpr int kDepth = V == 1 ? 3 : 4; // steps of B pieces in flight
template <int V>
constexpr int kLongSmem = kDepth<V> * kBatch<V> * 32 * V * 4 + 2 * kDepth<V> * kBatch<V> * 8;
constexpr int kFewCtas = 12; // CTAs of V = 1 per SM up to which the chain is the time
constexpr int kMostSmem = 227 * 1024; // of one CTA

// The items (row, tile), longest rows first, over the CTAs that start
// together, `per_sm` on each SM: those of one SM, whether it gets consecutive
// CTAs or every sms-th, are of different lengths (item i of each of per_sm
// equal parts of the list), not the longest row's tiles.
struct Spread {
    unsigned per_sm, sms, together; // together: CTAs of the first wave
    __device__ __forceinline__ unsigned item(unsigned b) const
    {
        if (b >= together)
            return b;
        const unsigned q = together / per_sm, r = together % per_sm, k = b / per_sm;
        const unsigned part = (b % per_sm + (k < q ? k * per_sm / sms : 0u)) % per_sm;
        return part * q + (part < r ? part : r) + k;
    }
};

// V: columns per lane of the chain warp; W: floats per copy (B's alignment)
template <int V, int W>
__global__ void __launch_bounds__(32 * (1 + kCopyWarps))
spdm_long_kernel(const Entry *__restrict__ packed, const int32_t *__restrict__ row_ptr,
                 const int32_t *__restrict__ list, unsigned tiles, const Spread spread, const float *__restrict__ B,
                 int64_t n, float *__restrict__ C)
{
    constexpr int kCols = 32 * V, kChunks = kCols / W, kWarps = kCopyWarps;
    constexpr int BATCH = kBatch<V>, DEPTH = kDepth<V>, EDEPTH = 2 * DEPTH; // entries land before their pieces are requested
    extern __shared__ __align__(16) float s_b[]; // [DEPTH][BATCH][kCols]
    Entry *s_e = reinterpret_cast<Entry *>(s_b + DEPTH * BATCH * kCols); // [EDEPTH][BATCH]
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned item = spread.item(blockIdx.x);
    const int64_t r = list[item / tiles];
    const int64_t j0 = static_cast<int64_t>(item % tiles) * kCols;
    const Entry *row = packed + row_ptr[r];
    const int cnt = row_ptr[r + 1] - row_ptr[r]; // < 2^31 (int32 format)
    const int nb = (cnt + BATCH - 1) / BATCH;

    if (warp > 0) {
        // a batch's pieces in chunks of W floats, consecutive over lanes, then
        // over copy warps; chunks past n are not copied
        constexpr int kMine = BATCH * kChunks / (32 * kWarps); // copies of a lane per batch
        constexpr int kAhead = kMine < 8 ? kMine : 8;                       // their columns read together
        const int first = (warp - 1) * 32 + lane;
        // step g (g = -(EDEPTH-1) .. nb-1) commits one group: the entries of
        // batch g + EDEPTH - 1 and the B pieces of batch g + DEPTH - 1
        auto issue = [&](int g) {
            const int be = g + EDEPTH - 1;
            if (first < BATCH && be >= 0 && be * BATCH + first < cnt)
                cp_async8(&s_e[(be % EDEPTH) * BATCH + first], row + be * BATCH + first);
            const int bb = g + DEPTH - 1;
            if (bb >= 0 && bb < nb) {
                const Entry *es = s_e + (bb % EDEPTH) * BATCH;
                float *dst = s_b + (bb % DEPTH) * (BATCH * kCols);
                const int len = cnt - bb * BATCH;
#pragma unroll
                for (int i0 = 0; i0 < kMine; i0 += kAhead) {
                    const float *src[kAhead];
#pragma unroll
                    for (int i = 0; i < kAhead; ++i) {
                        const int c = (i0 + i) * (32 * kWarps) + first;
                        const int e = c / kChunks;
                        src[i] = B + static_cast<int64_t>(e < len ? es[e].col : 0) * n;
                    }
#pragma unroll
                    for (int i = 0; i < kAhead; ++i) {
                        const int c = (i0 + i) * (32 * kWarps) + first;
                        const int e = c / kChunks, col = (c % kChunks) * W;
                        if (e < len && j0 + col < n)
                            cp_async_w<W>(dst + e * kCols + col, src[i] + j0 + col);
                    }
                }
            }
            cp_async_commit();
        };
        // before step g requests B pieces, the entries they need (step
        // g - (EDEPTH - DEPTH)) have landed: at most DEPTH - 2 steps pending
        for (int g = -(EDEPTH - 1); g < nb; ++g) {
            cp_async_wait<DEPTH - 2>();
            __syncthreads();
            issue(g);
        }
        cp_async_wait<0>();
        return;
    }
    for (int g = -(EDEPTH - 1); g < 0; ++g)
        __syncthreads();
    Chain<V> chain;
    chain.zero();
    for (int b = 0; b < nb; ++b) {
        // step b - (DEPTH - 1), which carried B batch b, has landed; the
        // copies of step b go to the batch read before
        __syncthreads();
        const Entry *es = s_e + (b % EDEPTH) * BATCH;
        const float *bs = s_b + (b % DEPTH) * (BATCH * kCols) + lane * V;
        if (cnt - b * BATCH >= BATCH) {
#pragma unroll
            for (int e = 0; e < BATCH; e += 2) {
                const int4 two = *reinterpret_cast<const int4 *>(es + e); // (col, val) of two entries
                chain.add(__int_as_float(two.y), bs + e * kCols);
                chain.add(__int_as_float(two.w), bs + (e + 1) * kCols);
            }
        } else {
            const int len = cnt - b * BATCH;
            for (int e = 0; e < len; ++e)
                chain.add(es[e].val, bs + e * kCols);
        }
    }
#pragma unroll
    for (int v = 0; v < V; ++v)
        if (j0 + lane * V + v < n)
            C[r * n + j0 + lane * V + v] = chain.at(v);
}

template <int V, int W>
cudaError_t launch_long(const Entry *packed, const int32_t *row_ptr, const int32_t *list, int64_t n_long,
                        const float *B, int64_t n, float *C, cudaStream_t st)
{
    const int64_t tiles = (n + 32 * V - 1) / (32 * V), ctas = n_long * tiles;
    if (ctas > 0x7fffffffLL)
        return cudaErrorInvalidConfiguration;
    // as much shared memory each as spreads few CTAs evenly over the SMs:
    // beside the short rows the scheduler otherwise puts a dozen on one SM and
    // leaves others empty (25 rows of 4096, n = 192: 103 us against 36)
    const int64_t sms = device_sms();
    const int most = static_cast<int>(kMostSmem / (kLongSmem<V> + 1024));
    const int per_sm = static_cast<int>(std::min<int64_t>(most, (ctas + sms - 1) / sms));
    const int smem = std::max(kLongSmem<V>, kMostSmem / per_sm / 128 * 128 - 1024);
    const Spread spread{static_cast<unsigned>(per_sm), static_cast<unsigned>(sms),
                        static_cast<unsigned>(std::min<int64_t>(ctas, per_sm * sms))};
    // the most that any call asks for, not this call's: the attribute belongs to
    // every thread of the process, one of which may launch right after another
    const cudaError_t e = cudaFuncSetAttribute(spdm_long_kernel<V, W>, cudaFuncAttributeMaxDynamicSharedMemorySize, kMostSmem);
    if (e != cudaSuccess)
        return e;
    spdm_long_kernel<V, W><<<static_cast<unsigned>(ctas), 32 * (1 + kCopyWarps), smem, st>>>(
        packed, row_ptr, list, static_cast<unsigned>(tiles), spread, B, n, C);
    count_launches(1);
    return cudaGetLastError();
}

} // namespace

int32_t long_row_min() { return 256; }

// What this kernel and the short rows' can run: any alignment of B (copies of
// 16, 8 or 4 bytes), widths within their grids. Where they gain is another
// question (long_rows_pay, api.cu).
bool long_rows_ok(int64_t m, int64_t n)
{
    const int64_t tiles = (n + 31) / 32;
    return tiles <= 65535 && m <= 0x7fffffffLL / tiles;
}

cudaError_t launch_collect_long(const int32_t *row_ptr, int64_t m, int32_t *list, int64_t cap,
                                unsigned long long *count, cudaStream_t st)
{
    if (m <= 0)
        return cudaSuccess;
    int64_t blocks = (m + 255) / 256;
    if (blocks > 4096)
        blocks = 4096;
    int32_t *found = list + cap;
    collect_long_kernel<<<static_cast<unsigned>(blocks), 256, 0, st>>>(row_ptr, m, long_row_min(), found, cap, count);
    order_long_kernel<<<1, kOrderThreads, 0, st>>>(row_ptr, found, cap, count, list);
    count_launches(2);
    return cudaGetLastError();
}

cudaError_t launch_spdm_long(const Entry *packed, const int32_t *row_ptr, const int32_t *list, int64_t n_long,
                             const float *B, int64_t n, float *C, cudaStream_t st)
{
    if (n_long <= 0 || n <= 0)
        return cudaSuccess;
    const uintptr_t b = reinterpret_cast<uintptr_t>(B);
    const int w = n % 4 == 0 && !(b & 15) ? 4 : (n % 2 == 0 && !(b & 7) ? 2 : 1);
#define GCOO_LONG(V)                                                                          \
    return w == 4   ? launch_long<V, 4>(packed, row_ptr, list, n_long, B, n, C, st)           \
           : w == 2 ? launch_long<V, 2>(packed, row_ptr, list, n_long, B, n, C, st)           \
                    : launch_long<V, 1>(packed, row_ptr, list, n_long, B, n, C, st)
    if (n <= 32 || n_long * ((n + 31) / 32) <= static_cast<int64_t>(kFewCtas) * device_sms())
        GCOO_LONG(1);
    GCOO_LONG(4);
#undef GCOO_LONG
}

} // namespace gcoo
