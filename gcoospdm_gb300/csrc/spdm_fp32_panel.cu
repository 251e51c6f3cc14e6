// spdm_fp32_panel.cu -- FP32 multiply of matrices whose rows share columns,
// sixteen rows at a time.
//
// The same product as the row and group walks and the reference's
// sparse_dense_groupcoo_mat_mul_kernel (src/gcoo_spdm_kernels.cu:92-158):
// every C element is one sequential fmaf chain over its row's entries in
// column order from 0.0f, so the bits are the same. What differs is how many
// rows one B value in a register serves: sixteen here (four groups), so that
// the FMA pipes and not the load path bound block-clustered matrices.
//
// One CTA per (16 rows, up to 4 x 128 output columns). The panel's entries
// are staged a window of 512 columns at a time: one pass sets every entry's
// row bit in its column's mask, the columns with entries are listed in order,
// and a second pass puts the values into s_a[place in the list][row]. Each
// row's part of a window is found without a search: the tiled conversion's
// per-(row, 128-column segment) prefixes give it. Each warp then walks the
// list with 4 output columns per lane and all 16 rows' sums in registers; the
// lane's B values come through its own slots of a ring of 16-byte cp.async
// copies eight columns deep (no barrier: a lane reads only what it copied),
// its 16 A values by four 16-byte broadcast loads. Where every listed column
// has all 16 rows the products are packed FMAs, two rows per fma.rn.f32x2
// (each half is the ordinary FP32 fma); otherwise each row's four FMAs run
// under the row's predicate, without branches: absent entries never touch a
// sum (0 * inf or a -0.0 sum would change the result).
//
// Bound: the FMA pipes and the registers' operand bandwidth. Measured at A
// 8192^2 (16 x 16 blocks, 25 %), B 8192 x 1024: 0.76 ms, 45 TFLOP/s, against
// 1.80 ms, 19 TFLOP/s of the group walk (each B value fetched for 4 rows: the
// L1 path and its shuffles bound it). A loop of nothing but these loads from
// shared memory and these FMAs (16 rows x 4 columns a lane) runs at 55
// TFLOP/s on the same GPU, the operands' register banks being what it waits
// for. Steps on the way: B loaded straight to registers 1.12 ms (its wait
// was exposed); the ring with branches on the masks 1.05 ms; values in list
// order with constant offsets 0.77 ms; entries loaded eight at a time 0.75
// ms. Lanes of 8 rows x 8 columns 0.81 ms, 16 x 8 0.79 ms, four CTAs per SM at
// 128 registers 0.80 ms, the next window's entries copied ahead 0.83 ms, a ring
// of four 0.98 ms, of sixteen 0.93 ms.
#include <type_traits>

#include "internal.cuh"

namespace gcoo {

namespace {

constexpr int kPanelRows = 16;
constexpr int kWinSegs = 4;              // 128-column segments per window
constexpr int kWinCols = kWinSegs * 128; // A values of a window: up to 32 KB
constexpr int kMaxWarps = 4;
constexpr int kV = 4;          // output columns per lane
constexpr int kCols = 32 * kV; // output columns per warp
constexpr int kRing = 8;       // B rows a warp keeps in flight, two per commit group
constexpr int kBatch = 8;      // entries a thread loads at once while staging

constexpr int panel_smem(int warps)
{
    return kWinCols * (kPanelRows * 4 + 8 + 4 + 4 + 2) + warps * kRing * kCols * 4 + kRing * 8 + 8;
}

__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c)
{
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

__device__ __forceinline__ uint64_t pack2(float lo, float hi)
{
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}

__device__ __forceinline__ void unpack2(uint64_t x, float &lo, float &hi)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(x));
}

// Two rows' sums of kV columns (row 0 low, row 1 high halves), each row
// multiplied only under its own (warp-uniform) predicate.
__device__ __forceinline__ void fma_masked(uint64_t (&c)[kV], uint32_t has0, uint32_t has1, uint64_t a, const float (&b)[kV])
{
    static_assert(kV == 4, "four sums per row below");
    float x[kV], y[kV], a0, a1;
    unpack2(a, a0, a1);
#pragma unroll
    for (int v = 0; v < kV; ++v)
        unpack2(c[v], x[v], y[v]);
    asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
        "@p fma.rn.f32 %0, %5, %6, %0;\n\t@p fma.rn.f32 %1, %5, %7, %1;\n\t"
        "@p fma.rn.f32 %2, %5, %8, %2;\n\t@p fma.rn.f32 %3, %5, %9, %3;\n\t}"
        : "+f"(x[0]), "+f"(x[1]), "+f"(x[2]), "+f"(x[3])
        : "r"(has0), "f"(a0), "f"(b[0]), "f"(b[1]), "f"(b[2]), "f"(b[3]));
    asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
        "@p fma.rn.f32 %0, %5, %6, %0;\n\t@p fma.rn.f32 %1, %5, %7, %1;\n\t"
        "@p fma.rn.f32 %2, %5, %8, %2;\n\t@p fma.rn.f32 %3, %5, %9, %3;\n\t}"
        : "+f"(y[0]), "+f"(y[1]), "+f"(y[2]), "+f"(y[3])
        : "r"(has1), "f"(a1), "f"(b[0]), "f"(b[1]), "f"(b[2]), "f"(b[3]));
#pragma unroll
    for (int v = 0; v < kV; ++v)
        c[v] = pack2(x[v], y[v]);
}

// kV output columns of a lane into its own ring slot. VEC4 (n % 4 == 0, B
// and C 16-byte aligned): one 16-byte copy; otherwise 4-byte copies at
// 32-column strides: contiguous across the warp whatever n is.
template <bool VEC4>
__device__ __forceinline__ void copy_b(uint32_t dst, const float *__restrict__ row, const int (&off)[VEC4 ? 1 : kV])
{
#pragma unroll
    for (int h = 0; h < (VEC4 ? 1 : kV); ++h) {
        if constexpr (VEC4)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + h * 512), "l"(row + off[h]) : "memory");
        else
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst + h * 128), "l"(row + off[h]) : "memory");
    }
}

__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }

template <int N>
__device__ __forceinline__ void copy_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

template <bool VEC4>
__global__ void __launch_bounds__(kMaxWarps * 32, 3)
spdm_panel_kernel(const Entry *__restrict__ packed, const int32_t *__restrict__ row_ptr,
                  const int32_t *__restrict__ pref, int64_t S, int64_t m, const float *__restrict__ B, int64_t n,
                  float *__restrict__ C)
{
    grid_wait_previous();
    row_ptr = written(row_ptr);
    pref = written(pref);
    grid_launch_next();
    extern __shared__ __align__(16) unsigned char smem[];
    float *s_a = reinterpret_cast<float *>(smem);                             // [listed column][kPanelRows]
    float *s_b = s_a + kWinCols * kPanelRows;                                 // [warp][kRing][kCols]
    int64_t *s_off = reinterpret_cast<int64_t *>(s_b + (blockDim.x >> 5) * (kRing * kCols)); // [listed]: offset of B's row
    uint32_t *s_mask = reinterpret_cast<uint32_t *>(s_off + kWinCols + kRing); // [column]: rows with an entry
    uint32_t *s_rows = s_mask + kWinCols;                                     // [listed]: the same, in list order
    uint16_t *s_pos = reinterpret_cast<uint16_t *>(s_rows + kWinCols + 2);      // [column]: its place in the list
    __shared__ int s_cnt[kWinCols / 32];

    const int tid = threadIdx.x, nthr = blockDim.x, warp = tid >> 5, lane = tid & 31;
    const int64_t r0 = static_cast<int64_t>(blockIdx.x) * kPanelRows;
    const int nrows = static_cast<int>(r0 + kPanelRows <= m ? kPanelRows : m - r0);
    const uint32_t full_mask = (1u << nrows) - 1u;
    const int64_t j0 = (static_cast<int64_t>(blockIdx.y) * (nthr >> 5) + warp) * kCols;
    const bool warp_live = j0 < n; // warp-uniform
    constexpr int NO = VEC4 ? 1 : kV;
    int off[NO]; // the lane's columns; past n: column 0, loaded and never stored
    bool has[NO];
#pragma unroll
    for (int h = 0; h < NO; ++h) {
        const int64_t j = j0 + (VEC4 ? h * 128 + lane * 4 : h * 32 + lane);
        has[h] = j < n;
        off[h] = has[h] ? static_cast<int>(j) : 0;
    }
    const float *my_b = s_b + warp * (kRing * kCols) + (VEC4 ? lane * 4 : lane);
    const uint32_t my_b_addr = smem_u32(my_b);

    uint64_t acc[kPanelRows / 2][kV]; // rows 2p | 2p + 1
#pragma unroll
    for (int p = 0; p < kPanelRows / 2; ++p)
#pragma unroll
        for (int v = 0; v < kV; ++v)
            acc[p][v] = 0ull;

    // staging: nthr / 16 threads per row
    const int tpr = nthr / kPanelRows, sr = tid / tpr, st = tid - sr * tpr;
    const int64_t row = r0 + sr;
    const bool srow = sr < nrows;
    const int32_t rbeg = srow ? row_ptr[row] : 0, rend = srow ? row_ptr[row + 1] : 0;
    const int32_t *rpref = pref + (srow ? row : r0) * S;

    const auto window_end = [&](int64_t s) { return srow ? (s < S ? rbeg + rpref[s] : rend) : 0; };
    int32_t lo = rbeg, hi = window_end(kWinSegs);
    for (int i = tid; i < kWinCols; i += nthr)
        s_mask[i] = 0;
    __syncthreads();
    for (int64_t s0 = 0; s0 < S; s0 += kWinSegs) {
        const int c0 = static_cast<int>(s0) * 128;
        const int32_t hi2 = window_end(s0 + 2 * kWinSegs);
        const Entry *ent = packed + lo; // the row's entries in this window
        const int len = hi - lo;
        int e = st;
#pragma unroll 1
        for (; e + (kBatch - 1) * tpr < len; e += kBatch * tpr) {
            int32_t c[kBatch];
#pragma unroll
            for (int u = 0; u < kBatch; ++u)
                c[u] = ent[e + u * tpr].col;
#pragma unroll
            for (int u = 0; u < kBatch; ++u)
                atomicOr(&s_mask[c[u] - c0], 1u << sr);
        }
#pragma unroll 4
        for (; e < len; e += tpr)
            atomicOr(&s_mask[ent[e].col - c0], 1u << sr);
        __syncthreads(); // masks set; the previous window consumed
        // the window's columns with entries, in order
        bool full = true; // every listed column has an entry in each of the panel's rows
        for (int b = warp; b < kWinCols / 32; b += nthr >> 5) {
            const uint32_t mk = s_mask[b * 32 + lane];
            const unsigned any = __ballot_sync(0xffffffffu, mk != 0);
            full = full && (mk == 0 || mk == full_mask);
            if (lane == 0)
                s_cnt[b] = __popc(any);
        }
        full = __syncthreads_and(full) != 0;
        const int mine = lane < kWinCols / 32 ? s_cnt[lane] : 0;
        int incl = mine;
#pragma unroll
        for (int d = 1; d < kWinCols / 32; d <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, incl, d);
            if (lane >= d)
                incl += y;
        }
        const int cnt = __shfl_sync(0xffffffffu, incl, kWinCols / 32 - 1);
        for (int b = warp; b < kWinCols / 32; b += nthr >> 5) {
            const uint32_t mk = s_mask[b * 32 + lane];
            const unsigned any = __ballot_sync(0xffffffffu, mk != 0);
            const int at = __shfl_sync(0xffffffffu, incl - mine, b) + __popc(any & ((1u << lane) - 1u));
            if (mk) {
                s_pos[b * 32 + lane] = static_cast<uint16_t>(at);
                s_off[at] = static_cast<int64_t>(c0 + b * 32 + lane) * n;
                s_rows[at] = mk;
            }
        }
        if (tid < kRing) // copied ahead of the end of the list, never multiplied
            s_off[cnt + tid] = static_cast<int64_t>(c0) * n;
        __syncthreads();
        for (int i = tid; i < kWinCols; i += nthr)
            s_mask[i] = 0; // for the next window
        e = st;
#pragma unroll 1
        for (; e + (kBatch - 1) * tpr < len; e += kBatch * tpr) {
            Entry t[kBatch];
#pragma unroll
            for (int u = 0; u < kBatch; ++u)
                t[u] = ent[e + u * tpr];
#pragma unroll
            for (int u = 0; u < kBatch; ++u)
                s_a[s_pos[t[u].col - c0] * kPanelRows + sr] = t[u].val;
        }
#pragma unroll 4
        for (; e < len; e += tpr) {
            const Entry t = ent[e];
            s_a[s_pos[t.col - c0] * kPanelRows + sr] = t.val;
        }
        lo = hi;
        hi = hi2;
        __syncthreads();
        if (!warp_live)
            continue;

        // slot u of the ring: listed columns u, u + kRing, ...; one commit group per two columns
        const auto refill = [&](int slot, const int64_t *o) { copy_b<VEC4>(my_b_addr + slot * (4 * kCols), B + o[slot], off); };
        const auto take_b = [&](int slot, float (&b)[kV]) {
            if constexpr (VEC4) {
#pragma unroll
                for (int h = 0; h < kV / 4; ++h) {
                    const float4 t = *reinterpret_cast<const float4 *>(my_b + slot * (kCols) + h * 128);
                    b[4 * h] = t.x; b[4 * h + 1] = t.y; b[4 * h + 2] = t.z; b[4 * h + 3] = t.w;
                }
            } else {
#pragma unroll
                for (int v = 0; v < kV; ++v)
                    b[v] = my_b[slot * (kCols) + v * 32];
            }
        };
        const auto dup = [&](const float (&b)[kV], uint64_t (&bb)[kV]) {
#pragma unroll
            for (int v = 0; v < kV; ++v)
                bb[v] = pack2(b[v], b[v]);
        };
        const auto fetch_a = [&](const float *sa, ulonglong2 (&a)[4]) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
                a[q] = reinterpret_cast<const ulonglong2 *>(sa)[q];
        };
        const auto fma_pair = [&](int p, uint64_t a, const uint64_t (&bb)[kV]) {
#pragma unroll
            for (int v = 0; v < kV; ++v)
                acc[p][v] = fma2(a, bb[v], acc[p][v]);
        };
        // the rows with an entry in the column, without branches: a predicate per row
        const auto apply_rows = [&](uint32_t has, const ulonglong2 (&a)[4], const float (&b)[kV]) {
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                fma_masked(acc[2 * q], has & (1u << (4 * q)), has & (2u << (4 * q)), a[q].x, b);
                fma_masked(acc[2 * q + 1], has & (4u << (4 * q)), has & (8u << (4 * q)), a[q].y, b);
            }
        };
        // Blocks of kRing listed columns. Column i + u is in a[u & 1],
        // b[u & 1] when it is multiplied, while the next one's A values and B
        // are read from shared memory; its ring slot is refilled after it.
#pragma unroll
        for (int u = 0; u < kRing; ++u) {
            refill(u, s_off);
            if (u & 1)
                copy_commit();
        }
        ulonglong2 a[2][4];
        float b[2][kV];
        uint32_t rows[2];
        int i = 0;
        copy_wait<kRing / 2 - 1>();
        fetch_a(s_a, a[0]);
        take_b(0, b[0]);
        const auto block = [&](auto all_rows) {
            const float *sa = s_a + i * kPanelRows;
            const int64_t *so = s_off + i + kRing;
#pragma unroll
            for (int u = 0; u < kRing; ++u) {
                // odd u: the next column is the first of its commit group
                if (u & 1)
                    copy_wait<kRing / 2 - 2>();
                fetch_a(sa + (u + 1) * kPanelRows, a[(u + 1) & 1]);
                take_b((u + 1) % kRing, b[(u + 1) & 1]);
                if constexpr (decltype(all_rows)::value) {
                    uint64_t bb[kV];
                    dup(b[u & 1], bb);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        fma_pair(2 * q, a[u & 1][q].x, bb);
                        fma_pair(2 * q + 1, a[u & 1][q].y, bb);
                    }
                } else {
                    rows[(u + 1) & 1] = s_rows[i + u + 1];
                    apply_rows(rows[u & 1], a[u & 1], b[u & 1]);
                }
                refill(u, so);
                if (u & 1)
                    copy_commit();
            }
        };
        if (full) {
#pragma unroll 1
            for (; i + kRing <= cnt; i += kRing)
                block(std::true_type());
        } else {
            rows[0] = s_rows[0];
#pragma unroll 1
            for (; i + kRing <= cnt; i += kRing)
                block(std::false_type());
        }
        copy_wait<0>();
#pragma unroll 1
        for (; i < cnt; ++i) { // fewer than kRing columns: all in the ring
            ulonglong2 ar[4];
            float br[kV];
            fetch_a(s_a + i * kPanelRows, ar);
            take_b(i & (kRing - 1), br);
            apply_rows(s_rows[i], ar, br);
        }
    }
    if (!warp_live)
        return;
#pragma unroll
    for (int p = 0; p < kPanelRows / 2; ++p) {
        float x[kV], y[kV];
#pragma unroll
        for (int v = 0; v < kV; ++v)
            unpack2(acc[p][v], x[v], y[v]);
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const int r = 2 * p + half;
            if (r >= nrows)
                break;
            float *out = C + (r0 + r) * n;
            if constexpr (VEC4) {
#pragma unroll
                for (int h = 0; h < kV / 4; ++h)
                    if (has[h])
                        *reinterpret_cast<float4 *>(out + off[h]) =
                            half ? make_float4(y[4 * h], y[4 * h + 1], y[4 * h + 2], y[4 * h + 3])
                                 : make_float4(x[4 * h], x[4 * h + 1], x[4 * h + 2], x[4 * h + 3]);
            } else {
#pragma unroll
                for (int v = 0; v < kV; ++v)
                    if (has[v])
                        out[off[v]] = half ? y[v] : x[v];
            }
        }
    }
}

// How many rows of a panel share a column, on up to gridDim.x panels spread
// over the matrix: out[0] += entries, out[1] += distinct columns, both of
// kShareCols columns from each panel's first one with an entry on. host (may be
// null; page-locked): out as the CTA that finishes last (*ticket, zeroed
// before) finds it. A CTA has one panel, and the build waits for it: many
// threads, eight entries' loads of each in flight, a byte per column (8192^2
// at 25 % in 16 x 16 blocks, 32768 entries a panel: 9.5 us; with 256 threads
// 42, 1024 threads that set bits with atomics 17).
constexpr int kShareCols = 1 << 15;
constexpr int kSharePanels = 64, kShareThreads = 1024, kShareBatch = 8;

__global__ void __launch_bounds__(kShareThreads)
panel_share_kernel(const Entry *__restrict__ packed, const int32_t *__restrict__ row_ptr, int64_t m, int64_t k,
                   int64_t panels, unsigned long long *__restrict__ out, unsigned int *__restrict__ ticket,
                   int64_t *__restrict__ host)
{
    __shared__ __align__(16) uint8_t s_seen[kShareCols]; // 0 or 1: stores of 1 need no atomics
    __shared__ int s_first, s_sum[2];
    const int64_t r0 = (blockIdx.x * panels / gridDim.x) * kPanelRows;
    const int64_t r1 = r0 + kPanelRows < m ? r0 + kPanelRows : m;
    const int used = static_cast<int>(k < kShareCols ? (k + 15) / 16 : kShareCols / 16);
    for (int i = threadIdx.x; i < used; i += kShareThreads)
        reinterpret_cast<uint4 *>(s_seen)[i] = make_uint4(0, 0, 0, 0);
    if (threadIdx.x == 0) {
        s_first = k > kShareCols ? 0x7fffffff : 0;
        s_sum[0] = s_sum[1] = 0;
    }
    grid_wait_previous();
    row_ptr = written(row_ptr);
    __syncthreads();
    const int64_t begin = row_ptr[r0], end = row_ptr[r1];
    if (k > kShareCols) {
        const int64_t r = r0 + threadIdx.x;
        if (r < r1 && row_ptr[r] < row_ptr[r + 1])
            atomicMin(&s_first, packed[row_ptr[r]].col);
        __syncthreads();
    }
    int entries = 0, distinct = 0;
    for (int64_t e0 = begin + threadIdx.x; e0 < end; e0 += kShareThreads * kShareBatch) {
        int c[kShareBatch];
#pragma unroll
        for (int u = 0; u < kShareBatch; ++u) {
            const int64_t e = e0 + u * kShareThreads;
            c[u] = e < end ? packed[e].col - s_first : kShareCols;
        }
#pragma unroll
        for (int u = 0; u < kShareBatch; ++u)
            if (c[u] < kShareCols) {
                ++entries;
                s_seen[c[u]] = 1;
            }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < 4 * used; i += kShareThreads)
        distinct += __popc(reinterpret_cast<const uint32_t *>(s_seen)[i]);
    entries = __reduce_add_sync(0xffffffffu, entries);
    distinct = __reduce_add_sync(0xffffffffu, distinct);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&s_sum[0], entries);
        atomicAdd(&s_sum[1], distinct);
    }
    __syncthreads();
    if (threadIdx.x != 0)
        return;
    atomicAdd(out, static_cast<unsigned long long>(s_sum[0]));
    atomicAdd(out + 1, static_cast<unsigned long long>(s_sum[1]));
    if (!host)
        return;
    __threadfence(); // the sums before the ticket
    if (atomicAdd(ticket, 1u) == gridDim.x - 1) {
        __threadfence();
        host[0] = static_cast<int64_t>(__ldcg(out));
        host[1] = static_cast<int64_t>(__ldcg(out + 1));
    }
}

// The same sample of A itself (k <= kShareCols), before the entries are placed:
// a conversion in two passes reads it with its totals, where the sample of the
// entries needs a wait of its own (builds, us: 2153 x 1929 at 36 % 75 -> 57,
// 6645 x 4381 227 -> 200, 8192^2 at 40 % 554 -> 522).
// totals: [0] entries, [2] distinct group columns; with fewer than `least` entries
// or, unless `any`, too little sharing to consider panels nothing is read. A CTA
// has 1024 columns of a panel.
constexpr int kDenseShareThreads = 256, kDenseShareCols = 1024;

__global__ void __launch_bounds__(kDenseShareThreads)
dense_share_kernel(const float *__restrict__ A, int64_t m, int64_t k, int64_t panels, int64_t least,
                   bool any, const int64_t *__restrict__ totals, unsigned long long *__restrict__ out)
{
    __shared__ int s_sum[2];
    if (threadIdx.x == 0)
        s_sum[0] = s_sum[1] = 0;
    grid_wait_previous();
    totals = written(totals);
    const int64_t nnz = totals[0], groups = totals[2];
    if (nnz < least || (!any && 2 * nnz < 3 * groups))
        return; // the same for all
    __syncthreads();
    const int64_t r0 = (blockIdx.x * panels / gridDim.x) * kPanelRows;
    const int rows = static_cast<int>(r0 + kPanelRows < m ? kPanelRows : m - r0);
    int entries = 0, distinct = 0;
#pragma unroll 1
    for (int q = 0; q < kDenseShareCols; q += kDenseShareThreads) {
        const int64_t c = static_cast<int64_t>(blockIdx.y) * kDenseShareCols + q + threadIdx.x;
        int x = 0;
#pragma unroll
        for (int r = 0; r < kPanelRows; ++r)
            x += c < k && r < rows && A[(r0 + r) * k + c] != 0.0f;
        entries += x;
        distinct += x != 0;
    }
    entries = __reduce_add_sync(0xffffffffu, entries);
    distinct = __reduce_add_sync(0xffffffffu, distinct);
    if ((threadIdx.x & 31) == 0) {
        atomicAdd(&s_sum[0], entries);
        atomicAdd(&s_sum[1], distinct);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        atomicAdd(out, static_cast<unsigned long long>(s_sum[0]));
        atomicAdd(out + 1, static_cast<unsigned long long>(s_sum[1]));
    }
}

} // namespace

bool dense_share_ok(int64_t k) { return k <= kShareCols; }

cudaError_t launch_dense_share(const float *A, int64_t m, int64_t k, int64_t least, bool any,
                               const int64_t *totals, unsigned long long *out, cudaStream_t st)
{
    const int64_t panels = (m + kPanelRows - 1) / kPanelRows;
    const dim3 grid(static_cast<unsigned>(panels < kSharePanels ? panels : kSharePanels),
                    static_cast<unsigned>((k + kDenseShareCols - 1) / kDenseShareCols));
    count_launches(1);
    return launch_after(dense_share_kernel, grid, dim3(kDenseShareThreads), 0, st, A, m, k, panels, least, any,
                        totals, out);
}

cudaError_t launch_panel_share(const Entry *packed, const int32_t *row_ptr, int64_t m, int64_t k,
                               unsigned long long *out, unsigned int *ticket, int64_t *host, cudaStream_t st)
{
    const int64_t panels = (m + kPanelRows - 1) / kPanelRows;
    const unsigned grid = static_cast<unsigned>(panels < kSharePanels ? panels : kSharePanels);
    count_launches(1);
    return launch_after(panel_share_kernel, dim3(grid), dim3(kShareThreads), 0, st, packed, row_ptr, m, k, panels, out,
                        ticket, host);
}

// Column tiles along the grid's y: wider B takes another walk (shared_walk,
// api.cu), whose tile count decides what is possible
bool panel_ok(int64_t n) { return n <= 1 << 20; }

cudaError_t launch_spdm_fp32_panel(const Entry *packed, const int32_t *row_ptr, const int32_t *pref, int64_t m,
                                   int64_t k, const float *B, int64_t n, float *C, cudaStream_t st)
{
    if (m <= 0 || n <= 0)
        return cudaSuccess;
    const bool vec4 = n % 4 == 0 && !((reinterpret_cast<uintptr_t>(B) | reinterpret_cast<uintptr_t>(C)) & 15);
    const int64_t strips = (n + kCols - 1) / kCols;
    const int warps = strips < kMaxWarps ? static_cast<int>(strips) : kMaxWarps;
    const int64_t ny = (strips + warps - 1) / warps;
    const int64_t nx = (m + kPanelRows - 1) / kPanelRows;
    if (!panel_ok(n) || nx > 0x7fffffffLL)
        return cudaErrorInvalidConfiguration;
    const dim3 grid(static_cast<unsigned>(nx), static_cast<unsigned>(ny));
    const int64_t S = conv_segments(k);
    const auto kern = vec4 ? spdm_panel_kernel<true> : spdm_panel_kernel<false>;
    // the most that any call asks for: the attribute belongs to every thread of the process
    const cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, panel_smem(kMaxWarps));
    if (e != cudaSuccess)
        return e;
    count_launches(1);
    return launch_after(kern, grid, dim3(warps * 32), panel_smem(warps), st, packed, row_ptr, pref, S, m, B, n, C);
}

} // namespace gcoo
