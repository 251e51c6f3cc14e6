// convert.cu -- dense -> GCOO conversion on sm_103a.
//
// Replaces the reference's three conversion kernels
// (src/gcoo_spdm_kernels.cu:4-90 and :160-168, orchestrated by
// src/ShGCOOSpDM.cu:19-126) with:
//   1. row_count_kernel    one warp per row, 128-bit loads, per-row nonzero
//                          counts (a group count is the sum of its rows);
//   2. scan_*_kernels      a device-wide reduce-then-scan (three small
//                          launches, no single-thread serial scan) giving
//                          row pointers, group_index, nnz_per_group and the
//                          int64 total;
//   3. scatter_kernel      one CTA per group: ballot/popc ranks inside each
//                          warp, a warp-total exchange across the CTA, and
//                          a stable write of every entry twice: in the
//                          reference's GCOO order (column, then row) into
//                          vals/rows/cols, and in row order (row, then
//                          column) into the packed execution layout.
// The zero test is `v != 0.0f` everywhere, as in the reference.
#include "convert_load.cuh"

namespace gcoo {

namespace {

constexpr int kCountThreads = 256;
constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr int kScanTile = kScanThreads * kScanItems;
constexpr int kTopThreads = 1024;
constexpr int kScatterThreads = 256;

__device__ __forceinline__ int nz(float v) { return v != 0.0f ? 1 : 0; }

__global__ void __launch_bounds__(kCountThreads)
row_count_kernel(const float *__restrict__ A, int64_t m, int64_t k, int32_t *__restrict__ row_nnz)
{
    const int lane = threadIdx.x & 31;
    const int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
    for (int64_t r = warp; r < m; r += nwarps) {
        const float *row = A + r * k;
        int cnt = 0;
        // scalar head up to the first 16-byte boundary (rows start 4-byte aligned)
        const uintptr_t addr = reinterpret_cast<uintptr_t>(row);
        int64_t head = static_cast<int64_t>(((16u - (addr & 15u)) & 15u) >> 2);
        if (head > k)
            head = k;
        if (lane < head)
            cnt += nz(__ldg(row + lane));
        const float4 *body = reinterpret_cast<const float4 *>(row + head);
        const int64_t nb = (k - head) >> 2;
        int64_t i = lane;
#pragma unroll 1
        for (; i + 96 < nb; i += 128) {
            const float4 v0 = __ldcs(body + i);
            const float4 v1 = __ldcs(body + i + 32);
            const float4 v2 = __ldcs(body + i + 64);
            const float4 v3 = __ldcs(body + i + 96);
            cnt += nz(v0.x) + nz(v0.y) + nz(v0.z) + nz(v0.w);
            cnt += nz(v1.x) + nz(v1.y) + nz(v1.z) + nz(v1.w);
            cnt += nz(v2.x) + nz(v2.y) + nz(v2.z) + nz(v2.w);
            cnt += nz(v3.x) + nz(v3.y) + nz(v3.z) + nz(v3.w);
        }
        for (; i < nb; i += 32) {
            const float4 v = __ldcs(body + i);
            cnt += nz(v.x) + nz(v.y) + nz(v.z) + nz(v.w);
        }
        const int64_t t0 = head + nb * 4;
        if (t0 + lane < k)
            cnt += nz(__ldg(row + t0 + lane));
        cnt = __reduce_add_sync(0xffffffffu, cnt);
        if (lane == 0)
            row_nnz[r] = cnt;
    }
}

// Nonzeros per group: a group's rows are one contiguous range of A, counted
// by one warp or (from kGroupCtaFloats floats on) by a CTA's eight; the count
// goes into both arrays, nnz_per_group[ng] = 0. Against counts per row and a
// scan of those: two launches and two allocations less (4096^2: 20 us of
// kernels against 30, and no cudaMalloc / cudaFree in the call).
constexpr int64_t kGroupCtaFloats = 2048;

__global__ void __launch_bounds__(kCountThreads)
group_count_kernel(const float *__restrict__ A, int64_t m, int64_t k, int32_t cpg, int64_t ng, int wpg,
                   int32_t *__restrict__ group_index, int32_t *__restrict__ nnz_per_group)
{
    __shared__ int s_cnt[kCountThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per_cta = (kCountThreads / 32) / wpg;
    const int64_t g = static_cast<int64_t>(blockIdx.x) * per_cta + warp / wpg;
    int cnt = 0;
    if (g < ng) {
        const int64_t r1 = (g + 1) * cpg < m ? (g + 1) * cpg : m;
        const float *p = A + g * cpg * k;
        const int64_t len = (r1 - g * cpg) * k;
        int64_t head = static_cast<int64_t>(((16u - (reinterpret_cast<uintptr_t>(p) & 15u)) & 15u) >> 2);
        if (head > len)
            head = len;
        const int64_t nb = (len - head) >> 2, t0 = head + nb * 4;
        const float4 *body = reinterpret_cast<const float4 *>(p + head);
        const int sub = warp % wpg;
        if (sub == 0) {
            if (lane < head)
                cnt += nz(__ldg(p + lane));
            if (t0 + lane < len)
                cnt += nz(__ldg(p + t0 + lane));
        }
        const int64_t step = static_cast<int64_t>(wpg) * 32;
        int64_t i = static_cast<int64_t>(sub) * 32 + lane;
        for (; i + 3 * step < nb; i += 4 * step) {
            float4 v[4];
#pragma unroll
            for (int u = 0; u < 4; ++u)
                v[u] = __ldg(body + i + u * step);
#pragma unroll
            for (int u = 0; u < 4; ++u)
                cnt += nz(v[u].x) + nz(v[u].y) + nz(v[u].z) + nz(v[u].w);
        }
        for (; i < nb; i += step) {
            const float4 v = __ldg(body + i);
            cnt += nz(v.x) + nz(v.y) + nz(v.z) + nz(v.w);
        }
    }
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (wpg > 1) { // grid-uniform
        if (lane == 0)
            s_cnt[warp] = cnt;
        __syncthreads();
        cnt = 0;
        for (int w = warp / wpg * wpg; w < warp / wpg * wpg + wpg; ++w)
            cnt += s_cnt[w];
    }
    if (g < ng && lane == 0 && warp % wpg == 0) {
        group_index[g] = cnt;
        nnz_per_group[g] = cnt;
        if (g == 0)
            nnz_per_group[ng] = 0; // the reference memsets nGroup+1 entries
    }
}

// Block-wide exclusive scan of one int64 per thread; returns the exclusive
// prefix and writes the block total to *total (all threads).
template <int THREADS>
__device__ __forceinline__ int64_t block_exclusive_scan(int64_t x, int64_t *s_warp, int64_t *total)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t incl = x;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const int64_t y = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d)
            incl += y;
    }
    if (lane == 31)
        s_warp[warp] = incl;
    __syncthreads();
    constexpr int W = THREADS / 32;
    if (warp == 0) {
        int64_t v = lane < W ? s_warp[lane] : 0;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int64_t y = __shfl_up_sync(0xffffffffu, v, d);
            if (lane >= d)
                v += y;
        }
        if (lane < W)
            s_warp[lane] = v; // inclusive warp prefix
    }
    __syncthreads();
    const int64_t warp_excl = warp ? s_warp[warp - 1] : 0;
    *total = s_warp[W - 1];
    __syncthreads();
    return warp_excl + incl - x;
}

__global__ void __launch_bounds__(kScanThreads)
scan_reduce_kernel(const int32_t *__restrict__ cnt, int64_t m, int64_t *__restrict__ block_sums)
{
    __shared__ int64_t s_warp[32];
    const int64_t base = static_cast<int64_t>(blockIdx.x) * kScanTile + threadIdx.x * kScanItems;
    int64_t s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i)
        if (base + i < m)
            s += cnt[base + i];
    int64_t total;
    block_exclusive_scan<kScanThreads>(s, s_warp, &total);
    if (threadIdx.x == 0)
        block_sums[blockIdx.x] = total;
}

// One CTA: exclusive scan of the block sums in place; writes the grand total.
__global__ void __launch_bounds__(kTopThreads)
scan_top_kernel(int64_t *__restrict__ block_sums, int64_t nb, int64_t *__restrict__ d_total,
                int32_t *__restrict__ row_ptr, int64_t m, uint32_t *__restrict__ status)
{
    __shared__ int64_t s_warp[32];
    int64_t carry = 0;
    for (int64_t base = 0; base < nb; base += kTopThreads) {
        const int64_t i = base + threadIdx.x;
        const int64_t x = i < nb ? block_sums[i] : 0;
        int64_t total;
        const int64_t ex = block_exclusive_scan<kTopThreads>(x, s_warp, &total);
        if (i < nb)
            block_sums[i] = carry + ex;
        carry += total;
    }
    if (threadIdx.x == 0) {
        *d_total = carry;
        row_ptr[m] = static_cast<int32_t>(carry);
        if (carry > 0x7fffffffLL && status)
            atomicOr(status, kStatusOverflow);
    }
}

__global__ void __launch_bounds__(kScanThreads)
scan_down_kernel(int32_t *__restrict__ data, int64_t m, const int64_t *__restrict__ block_off)
{
    __shared__ int64_t s_warp[32];
    const int64_t base = static_cast<int64_t>(blockIdx.x) * kScanTile + threadIdx.x * kScanItems;
    int32_t v[kScanItems];
    int64_t s = 0;
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        v[i] = base + i < m ? data[base + i] : 0;
        s += v[i];
    }
    int64_t total;
    int64_t run = block_off[blockIdx.x] + block_exclusive_scan<kScanThreads>(s, s_warp, &total);
#pragma unroll
    for (int i = 0; i < kScanItems; ++i) {
        if (base + i < m)
            data[base + i] = static_cast<int32_t>(run);
        run += v[i];
    }
}

// The whole row scan of a matrix of up to kSmallScanRows rows by one CTA:
// row counts -> row_ptr (in place, row_ptr[m] = total), the total and the
// longest row into d_total[0] / d_total[1], and the group arrays when given.
// Same results as scan_reduce / scan_top / scan_down + group_arrays +
// row_max. d_total may be null. The counts are read past L1 (they may come from CTAs of the same
// launch). host_words (may be null; page-locked): d_total[0..3] as the CTA's
// thread 0 knows them at the end.
constexpr int kSmallScanItems = 8;
constexpr int64_t kSmallScanRows = 16384; // two chunks; the three-kernel scan is faster beyond

__device__ __forceinline__ void scan_small_cta(int32_t *__restrict__ data, int64_t m, int32_t cpg,
                                               int32_t *__restrict__ group_index, int32_t *__restrict__ nnz_per_group,
                                               int64_t *__restrict__ d_total, int64_t *__restrict__ host_words,
                                               uint32_t *__restrict__ status)
{
    __shared__ int64_t s_warp[32];
    __shared__ int s_max[32];
    constexpr int64_t kChunk = static_cast<int64_t>(kTopThreads) * kSmallScanItems;
    int64_t carry = 0;
    int mx = 0;
    for (int64_t c0 = 0; c0 < m; c0 += kChunk) {
        const int64_t base = c0 + static_cast<int64_t>(threadIdx.x) * kSmallScanItems;
        int32_t v[kSmallScanItems];
        int64_t sum = 0;
#pragma unroll
        for (int i = 0; i < kSmallScanItems; ++i) {
            v[i] = base + i < m ? __ldcg(data + base + i) : 0;
            sum += v[i];
            mx = v[i] > mx ? v[i] : mx;
        }
        int64_t total;
        int64_t run = carry + block_exclusive_scan<kTopThreads>(sum, s_warp, &total);
        // whole groups inside the thread's rows (rows_per_group dividing the item count): their
        // arrays straight from the registers
        const bool own_groups = group_index && kSmallScanItems % cpg == 0;
        int32_t gsum = 0;
        int64_t gstart = run;
#pragma unroll
        for (int i = 0; i < kSmallScanItems; ++i) {
            if (base + i < m)
                data[base + i] = static_cast<int32_t>(run);
            run += v[i];
            gsum += v[i];
            if (own_groups && (i + 1) % cpg == 0) {
                const int64_t r0 = base + i + 1 - cpg;
                if (r0 < m) {
                    group_index[r0 / cpg] = static_cast<int32_t>(gstart);
                    nnz_per_group[r0 / cpg] = gsum;
                }
                gsum = 0;
                gstart = run;
            }
        }
        carry += total;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        const int y = __shfl_xor_sync(0xffffffffu, mx, o);
        mx = y > mx ? y : mx;
    }
    if ((threadIdx.x & 31) == 0)
        s_max[threadIdx.x >> 5] = mx;
    __syncthreads(); // also orders the row_ptr writes above before the group reads below
    if (threadIdx.x == 0) {
        int best = 0;
        for (int w = 0; w < kTopThreads / 32; ++w)
            best = s_max[w] > best ? s_max[w] : best;
        if (d_total) {
            d_total[0] = carry;
            d_total[1] = best;
        }
        data[m] = static_cast<int32_t>(carry);
        if (carry > 0x7fffffffLL && status)
            atomicOr(status, kStatusOverflow);
        if (host_words) {
            host_words[0] = carry;
            host_words[1] = best;
            host_words[2] = d_total[2];
            host_words[3] = d_total[3];
        }
    }
    if (!group_index)
        return;
    const int64_t ng = (m + cpg - 1) / cpg;
    if (kSmallScanItems % cpg == 0) {
        if (threadIdx.x == 0) {
            group_index[ng] = static_cast<int32_t>(carry);
            nnz_per_group[ng] = 0; // the reference memsets nGroup+1 entries
        }
        return;
    }
    __syncthreads();
    for (int64_t g = threadIdx.x; g <= ng; g += kTopThreads) {
        if (g == ng) {
            group_index[ng] = data[m];
            nnz_per_group[ng] = 0; // the reference memsets nGroup+1 entries
        } else {
            const int64_t r0 = g * cpg;
            const int64_t r1 = r0 + cpg < m ? r0 + cpg : m;
            group_index[g] = data[r0];
            nnz_per_group[g] = data[r1] - data[r0];
        }
    }
}

__global__ void __launch_bounds__(kTopThreads)
scan_small_kernel(int32_t *__restrict__ data, int64_t m, int32_t cpg, int32_t *__restrict__ group_index,
                  int32_t *__restrict__ nnz_per_group, int64_t *__restrict__ d_total, uint32_t *__restrict__ status)
{
    scan_small_cta(data, m, cpg, group_index, nnz_per_group, d_total, nullptr, status);
}

// The segment prefixes of the tiled conversion and the row scan in one
// launch: one warp per row turns the row's segment counts into their
// exclusive prefix (in place) and its total into data[row]; the CTA that
// finishes last (*ticket, zeroed before the launch) scans the totals. No CTA
// waits for another. d_total[2] and [3] are inputs here (the counting
// kernel's). One launch and its gap less per conversion than two kernels
// (800 x 800: a launch and its gap, about 4 us of a rebuild).
__global__ void __launch_bounds__(kTopThreads)
prefix_scan_kernel(int32_t *__restrict__ cnt, int64_t S, int32_t *__restrict__ data, int64_t m, int32_t cpg,
                   int32_t *__restrict__ group_index, int32_t *__restrict__ nnz_per_group,
                   int64_t *__restrict__ d_total, unsigned int *__restrict__ ticket,
                   int64_t *__restrict__ host_words, uint32_t *__restrict__ status)
{
    grid_wait_previous();
    grid_launch_next();
    __shared__ bool s_last;
    const int lane = threadIdx.x & 31;
    const int64_t r = static_cast<int64_t>(blockIdx.x) * (kTopThreads / 32) + (threadIdx.x >> 5);
    if (r < m) {
        int32_t *row = cnt + r * S;
        int32_t carry = 0;
        for (int64_t b = 0; b < S; b += 32) {
            const int32_t x = b + lane < S ? row[b + lane] : 0;
            int32_t incl = x;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int32_t y = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d)
                    incl += y;
            }
            if (b + lane < S)
                row[b + lane] = carry + incl - x;
            carry += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0)
            data[r] = carry;
    }
    __threadfence(); // the totals before the ticket
    __syncthreads();
    if (threadIdx.x == 0)
        s_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!s_last)
        return;
    __threadfence();
    scan_small_cta(data, m, cpg, group_index, nnz_per_group, d_total, host_words, status);
}

__global__ void group_arrays_kernel(const int32_t *__restrict__ row_ptr, int64_t m, int32_t cpg,
                                    int64_t ng, int32_t *__restrict__ group_index,
                                    int32_t *__restrict__ nnz_per_group)
{
    for (int64_t g = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; g <= ng;
         g += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        if (g == ng) {
            group_index[ng] = row_ptr[m];
            nnz_per_group[ng] = 0; // the reference memsets nGroup+1 entries
        } else {
            const int64_t r0 = g * cpg;
            const int64_t r1 = r0 + cpg < m ? r0 + cpg : m;
            group_index[g] = row_ptr[r0];
            nnz_per_group[g] = row_ptr[r1] - row_ptr[r0];
        }
    }
}

// One CTA per group of CPG rows; the group is walked in column tiles of
// kScatterThreads columns, one column per thread.
template <int CPG>
__global__ void __launch_bounds__(kScatterThreads)
scatter_kernel(const float *__restrict__ A, int64_t m, int64_t k, const int32_t *__restrict__ group_index,
               const int32_t *__restrict__ row_ptr, float *__restrict__ vals, int32_t *__restrict__ rows,
               int32_t *__restrict__ cols, Entry *__restrict__ packed)
{
    constexpr int W = kScatterThreads / 32;
    __shared__ int s_col[W];
    __shared__ int s_row[W][CPG];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const unsigned lt = (1u << lane) - 1u;
    const int64_t g = blockIdx.x;
    const int64_t r0 = g * CPG;
    const int nrows = static_cast<int>(r0 + CPG <= m ? CPG : m - r0);

    const int64_t gbase = group_index ? group_index[g] : 0;
    int32_t row_base[CPG];
#pragma unroll
    for (int r = 0; r < CPG; ++r)
        row_base[r] = (r < nrows && packed) ? row_ptr[r0 + r] : 0;

    int64_t col_run = 0;
    int row_run[CPG];
#pragma unroll
    for (int r = 0; r < CPG; ++r)
        row_run[r] = 0;

    for (int64_t c0 = 0; c0 < k; c0 += kScatterThreads) {
        const int64_t c = c0 + threadIdx.x;
        float v[CPG];
        unsigned bal[CPG];
        int cc = 0;
#pragma unroll
        for (int r = 0; r < CPG; ++r) {
            v[r] = (r < nrows && c < k) ? __ldcs(A + (r0 + r) * k + c) : 0.0f;
            const int f = nz(v[r]);
            cc += f;
            bal[r] = __ballot_sync(0xffffffffu, f);
        }
        int incl = cc;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d)
                incl += y;
        }
        if (lane == 31)
            s_col[warp] = incl;
        if (lane == 0) {
#pragma unroll
            for (int r = 0; r < CPG; ++r)
                s_row[warp][r] = __popc(bal[r]);
        }
        __syncthreads();
        int col_before = 0, col_tile = 0;
#pragma unroll
        for (int w = 0; w < W; ++w) {
            const int x = s_col[w];
            col_before += w < warp ? x : 0;
            col_tile += x;
        }
        // GCOO order: (column, row)
        int64_t pos = gbase + col_run + col_before + (incl - cc);
#pragma unroll
        for (int r = 0; r < CPG; ++r) {
            int before = 0, tile = 0;
#pragma unroll
            for (int w = 0; w < W; ++w) {
                const int x = s_row[w][r];
                before += w < warp ? x : 0;
                tile += x;
            }
            if (v[r] != 0.0f) {
                if (vals) {
                    vals[pos] = v[r];
                    rows[pos] = static_cast<int32_t>(r0 + r);
                    cols[pos] = static_cast<int32_t>(c);
                }
                if (packed) {
                    const int64_t q = static_cast<int64_t>(row_base[r]) + row_run[r] + before + __popc(bal[r] & lt);
                    Entry e;
                    e.col = static_cast<int32_t>(c);
                    e.val = v[r];
                    packed[q] = e;
                }
                ++pos;
            }
            row_run[r] += tile;
        }
        col_run += col_tile;
        __syncthreads();
    }
}

// Vectorised scatter: each thread owns 4 consecutive columns of the group's
// rows (one 128-bit load per row, shifted where rows do not start on 16
// bytes), so a CTA covers 1024 columns per step. The per-row counts of a
// thread (0..4) are packed four to a word in 8-bit fields and one warp scan
// of the packed words gives, at once, every row's rank among the lanes (row
// order) and, summed over the rows, the column-major rank (the reference's
// GCOO order). (Issuing a step's loads ahead of the step before it: 23.5
// against 24.4 us at 4096^2, for 80 registers instead of 71.)
template <int CPG, bool AL>
__global__ void __launch_bounds__(kScatterThreads)
scatter_vec_kernel(const float *__restrict__ A, int64_t m, int64_t k, const int32_t *__restrict__ group_index,
                   const int32_t *__restrict__ row_ptr, float *__restrict__ vals, int32_t *__restrict__ rows,
                   int32_t *__restrict__ cols, Entry *__restrict__ packed)
{
    constexpr int W = kScatterThreads / 32;
    constexpr int NP = (CPG + 3) / 4;
    constexpr int kTileCols = kScatterThreads * 4;
    __shared__ uint32_t s_tot[W][NP];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t g = blockIdx.x;
    const int64_t r0 = g * CPG;
    const int nrows = static_cast<int>(r0 + CPG <= m ? CPG : m - r0);
    const int64_t gbase = group_index ? group_index[g] : 0;
    int32_t row_base[CPG];
    int row_run[CPG];
#pragma unroll
    for (int r = 0; r < CPG; ++r) {
        row_base[r] = (r < nrows && packed) ? row_ptr[r0 + r] : 0;
        row_run[r] = 0;
    }
    int64_t col_run = 0;

    for (int64_t c0 = 0; c0 < k; c0 += kTileCols) {
        const int64_t c = c0 + threadIdx.x * 4, cw = c0 + warp * 128;
        float4 v[CPG];
#pragma unroll
        for (int r = 0; r < CPG; ++r)
            v[r] = r < nrows && cw < k // warp-uniform
                       ? seg_load<AL, true>(A + (r0 + r) * k + cw, lane, k - cw, A, A + m * k)
                       : make_float4(0.f, 0.f, 0.f, 0.f);
        uint32_t bits[CPG];
        uint32_t word[NP];
#pragma unroll
        for (int i = 0; i < NP; ++i)
            word[i] = 0;
#pragma unroll
        for (int r = 0; r < CPG; ++r) {
            bits[r] = nz(v[r].x) | (nz(v[r].y) << 1) | (nz(v[r].z) << 2) | (nz(v[r].w) << 3);
            word[r / 4] |= static_cast<uint32_t>(__popc(bits[r])) << (8 * (r % 4));
        }
        uint32_t incl[NP];
#pragma unroll
        for (int i = 0; i < NP; ++i) {
            incl[i] = word[i];
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl[i], d);
                if (lane >= d)
                    incl[i] += y; // fields never carry: a field's prefix is at most 4 * 32
            }
            if (lane == 31)
                s_tot[warp][i] = incl[i];
        }
        __syncthreads();
        int before[CPG], tile[CPG], lane_ex[CPG];
#pragma unroll
        for (int r = 0; r < CPG; ++r) {
            before[r] = 0;
            tile[r] = 0;
            lane_ex[r] = static_cast<int>(((incl[r / 4] - word[r / 4]) >> (8 * (r % 4))) & 0xffu);
        }
#pragma unroll
        for (int w = 0; w < W; ++w) {
#pragma unroll
            for (int r = 0; r < CPG; ++r) {
                const int x = static_cast<int>((s_tot[w][r / 4] >> (8 * (r % 4))) & 0xffu);
                before[r] += w < warp ? x : 0;
                tile[r] += x;
            }
        }
        int64_t pos = gbase + col_run;
#pragma unroll
        for (int r = 0; r < CPG; ++r)
            pos += before[r] + lane_ex[r];
        // reference GCOO order: column, then row
#pragma unroll
        for (int q = 0; q < 4; ++q) {
#pragma unroll
            for (int r = 0; r < CPG; ++r) {
                if ((bits[r] >> q) & 1u) {
                    if (vals) {
                        const float x = q == 0 ? v[r].x : q == 1 ? v[r].y : q == 2 ? v[r].z : v[r].w;
                        vals[pos] = x;
                        rows[pos] = static_cast<int32_t>(r0 + r);
                        cols[pos] = static_cast<int32_t>(c + q);
                    }
                    ++pos;
                }
            }
        }
        // execution layout: row, then column
        if (packed) {
#pragma unroll
            for (int r = 0; r < CPG; ++r) {
                int64_t q_pos = static_cast<int64_t>(row_base[r]) + row_run[r] + before[r] + lane_ex[r];
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    if ((bits[r] >> q) & 1u) {
                        Entry e;
                        e.col = static_cast<int32_t>(c + q);
                        e.val = q == 0 ? v[r].x : q == 1 ? v[r].y : q == 2 ? v[r].z : v[r].w;
                        packed[q_pos++] = e;
                    }
                }
            }
        }
        int64_t tile_all = 0;
#pragma unroll
        for (int r = 0; r < CPG; ++r) {
            row_run[r] += tile[r];
            tile_all += tile[r];
        }
        col_run += tile_all;
        __syncthreads();
    }
}

int sm_count()
{
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (sms <= 0)
            sms = 152;
    }
    return sms;
}

} // namespace

cudaError_t launch_row_count(const float *A, int64_t m, int64_t k, int32_t *row_nnz, cudaStream_t st)
{
    if (m <= 0)
        return cudaSuccess;
    const int64_t warps_needed = m;
    const int64_t per_block = kCountThreads / 32;
    int64_t blocks = (warps_needed + per_block - 1) / per_block;
    const int64_t cap = static_cast<int64_t>(sm_count()) * 16;
    if (blocks > cap)
        blocks = cap;
    row_count_kernel<<<static_cast<unsigned>(blocks), kCountThreads, 0, st>>>(A, m, k, row_nnz);
    count_launches(1);
    return cudaGetLastError();
}

namespace {
__global__ void row_max_kernel(const int32_t *__restrict__ row_ptr, int64_t m, unsigned long long *__restrict__ out)
{
    long long mx = 0;
    for (int64_t r = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; r < m;
         r += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const long long len = row_ptr[r + 1] - row_ptr[r];
        mx = len > mx ? len : mx;
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        const long long y = __shfl_xor_sync(0xffffffffu, mx, o);
        mx = y > mx ? y : mx;
    }
    if ((threadIdx.x & 31) == 0 && mx > 0)
        atomicMax(out, static_cast<unsigned long long>(mx));
}
} // namespace

cudaError_t launch_row_max(const int32_t *row_ptr, int64_t m, int64_t *out, cudaStream_t st)
{
    int64_t blocks = (m + 255) / 256;
    if (blocks > 1024)
        blocks = 1024;
    row_max_kernel<<<static_cast<unsigned>(blocks < 1 ? 1 : blocks), 256, 0, st>>>(
        row_ptr, m, reinterpret_cast<unsigned long long *>(out));
    count_launches(1);
    return cudaGetLastError();
}

size_t scan_scratch_elems(int64_t m)
{
    const int64_t nb = (m + kScanTile - 1) / kScanTile;
    return static_cast<size_t>(nb + 1);
}

cudaError_t launch_row_scan(int32_t *data, int64_t m, int32_t cpg, int32_t *group_index,
                            int32_t *nnz_per_group, int64_t *d_total, int64_t *scratch,
                            uint32_t *status, cudaStream_t st)
{
    const int64_t nb = (m + kScanTile - 1) / kScanTile;
    if (nb > 0) {
        scan_reduce_kernel<<<static_cast<unsigned>(nb), kScanThreads, 0, st>>>(data, m, scratch);
        count_launches(1);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess)
            return e;
    }
    scan_top_kernel<<<1, kTopThreads, 0, st>>>(scratch, nb, d_total, data, m, status);
    count_launches(1);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        return e;
    if (nb > 0) {
        scan_down_kernel<<<static_cast<unsigned>(nb), kScanThreads, 0, st>>>(data, m, scratch);
        count_launches(1);
        e = cudaGetLastError();
        if (e != cudaSuccess)
            return e;
    }
    if (group_index) {
        const int64_t ng = (m + cpg - 1) / cpg;
        int64_t blocks = (ng + 1 + 255) / 256;
        if (blocks > 4096)
            blocks = 4096;
        group_arrays_kernel<<<static_cast<unsigned>(blocks), 256, 0, st>>>(data, m, cpg, ng, group_index,
                                                                           nnz_per_group);
        count_launches(1);
        e = cudaGetLastError();
    }
    return e;
}

cudaError_t launch_row_scan_max(int32_t *data, int64_t m, int32_t cpg, int32_t *group_index,
                                int32_t *nnz_per_group, int64_t *d_total, int64_t *scratch, uint32_t *status,
                                cudaStream_t st)
{
    if (m > 0 && m <= kSmallScanRows) {
        scan_small_kernel<<<1, kTopThreads, 0, st>>>(data, m, cpg, group_index, nnz_per_group, d_total, status);
        count_launches(1);
        return cudaGetLastError();
    }
    cudaError_t e = launch_row_scan(data, m, cpg, group_index, nnz_per_group, d_total, scratch, status, st);
    if (e != cudaSuccess)
        return e;
    return launch_row_max(data, m, d_total + 1, st);
}

bool group_counts_ok(const float *A, int64_t m, int64_t k, int64_t ng)
{
    return ng > 0 && ng <= kSmallScanRows && k <= 0x7fffffffLL / m && (reinterpret_cast<uintptr_t>(A) & 3) == 0;
}

cudaError_t launch_group_counts(const float *A, int64_t m, int64_t k, int32_t cpg, int32_t *group_index,
                                int32_t *nnz_per_group, cudaStream_t st)
{
    const int64_t ng = (m + cpg - 1) / cpg;
    const int wpg = cpg * k >= kGroupCtaFloats ? kCountThreads / 32 : 1; // warps per group
    const int64_t blocks = (ng * wpg + kCountThreads / 32 - 1) / (kCountThreads / 32);
    group_count_kernel<<<static_cast<unsigned>(blocks), kCountThreads, 0, st>>>(A, m, k, cpg, ng, wpg, group_index,
                                                                                nnz_per_group);
    scan_small_kernel<<<1, kTopThreads, 0, st>>>(group_index, ng, 1, nullptr, nullptr, nullptr, nullptr);
    count_launches(2);
    return cudaGetLastError();
}

bool prefix_scan_ok(int64_t m) { return m > 0 && m <= kSmallScanRows; }

cudaError_t launch_prefix_scan(int32_t *cnt, int64_t segments, int32_t *row_ptr, int64_t m, int32_t cpg,
                               int32_t *group_index, int32_t *nnz_per_group, int64_t *d_total, unsigned int *ticket,
                               int64_t *host_words, uint32_t *status, cudaStream_t st)
{
    const int64_t blocks = (m + kTopThreads / 32 - 1) / (kTopThreads / 32);
    count_launches(1);
    return launch_after(prefix_scan_kernel, dim3(static_cast<unsigned>(blocks)), dim3(kTopThreads), 0, st, cnt, segments,
                        row_ptr, m, cpg, group_index, nnz_per_group, d_total, ticket, host_words, status);
}

cudaError_t launch_scatter(const float *A, int64_t m, int64_t k, int32_t cpg, const int32_t *group_index,
                           const int32_t *row_ptr, float *vals, int32_t *rows, int32_t *cols, Entry *packed,
                           cudaStream_t st, bool dense)
{
    const int64_t ng = (m + cpg - 1) / cpg;
    if (ng <= 0)
        return cudaSuccess;
    const unsigned grid = static_cast<unsigned>(ng);
    // Rows that do not start on 16 bytes: the vector kernel up to 4 rows per group
    // (4000 x 4001 at 2 %: 1 row 43 us against 79 of 4-byte loads, 2 42 / 57, 4 44 /
    // 58); with 8 its shifted rows take too many registers (84 / 61; 5653 x 5910 at
    // 16 % 235 / 108). Known to be dense: one row per group only (4000 x 4001 at
    // 40 % 51 / 88, 2 69 / 67, 4 96 / 80).
    const bool al = k % 4 == 0 && (reinterpret_cast<uintptr_t>(A) & 15) == 0;
    if (al ? cpg <= 8 : (reinterpret_cast<uintptr_t>(A) & 3) == 0 && cpg <= (dense ? 1 : 4)) {
#define GCOO_SCATTER_VEC(C)                                                                                         \
    (al ? scatter_vec_kernel<C, true> : scatter_vec_kernel<C, false>)<<<grid, kScatterThreads, 0, st>>>(            \
        A, m, k, group_index, row_ptr, vals, rows, cols, packed)
        switch (cpg) {
        case 1: GCOO_SCATTER_VEC(1); break;
        case 2: GCOO_SCATTER_VEC(2); break;
        case 4: GCOO_SCATTER_VEC(4); break;
        case 8:
            scatter_vec_kernel<8, true><<<grid, kScatterThreads, 0, st>>>(A, m, k, group_index, row_ptr, vals, rows,
                                                                          cols, packed);
            break;
        default: return cudaErrorInvalidValue;
        }
#undef GCOO_SCATTER_VEC
        count_launches(1);
        return cudaGetLastError();
    }
    switch (cpg) {
    case 1: scatter_kernel<1><<<grid, kScatterThreads, 0, st>>>(A, m, k, group_index, row_ptr, vals, rows, cols, packed); break;
    case 2: scatter_kernel<2><<<grid, kScatterThreads, 0, st>>>(A, m, k, group_index, row_ptr, vals, rows, cols, packed); break;
    case 4: scatter_kernel<4><<<grid, kScatterThreads, 0, st>>>(A, m, k, group_index, row_ptr, vals, rows, cols, packed); break;
    case 8: scatter_kernel<8><<<grid, kScatterThreads, 0, st>>>(A, m, k, group_index, row_ptr, vals, rows, cols, packed); break;
    case 16: scatter_kernel<16><<<grid, kScatterThreads, 0, st>>>(A, m, k, group_index, row_ptr, vals, rows, cols, packed); break;
    case 32: scatter_kernel<32><<<grid, kScatterThreads, 0, st>>>(A, m, k, group_index, row_ptr, vals, rows, cols, packed); break;
    default: return cudaErrorInvalidValue;
    }
    count_launches(1);
    return cudaGetLastError();
}

} // namespace gcoo
