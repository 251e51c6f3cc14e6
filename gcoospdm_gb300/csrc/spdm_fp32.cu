// spdm_fp32.cu -- the plain FP32 GCOO x dense multiply on sm_103a.
//
// Replaces sparse_dense_groupcoo_mat_mul_kernel (src/gcoo_spdm_kernels.cu:
// 92-158). One CTA per (GCOO group, or part of one, and span of column tiles):
//   * one elected thread stages the CTA's nonzeros (the contiguous range
//     [row_ptr[g*cpg], row_ptr[(g+1)*cpg]) of the packed row-ordered layout)
//     into shared memory with cp.async.bulk, completing on an mbarrier;
//   * each warp owns one row and walks the span's tiles of 32*V output columns
//     from that one staging; for every entry of its row (a shared-memory
//     broadcast) each lane loads V B values, consecutive in one 128-bit load
//     (V = 4) or in pieces of W where n or B is not 16-byte aligned, and
//     updates V register accumulators with fmaf;
//   * rows of the group run side by side, so B rows shared by several rows of
//     a group are served from L1.
// Every C element is a sequential fmaf chain over its row's entries in
// column order starting from 0.0f -- the same chain the reference kernel
// evaluates (its entries of one row are visited in column order too), so
// the FP32 result is bit-identical to the reference's.
#include "internal.cuh"

namespace gcoo {

namespace {

constexpr int kChunk = 2048; // most entries staged per pass (16 KB)
// 4-warp CTAs of the row walk per SM: 48 registers a thread. Measured (us;
// 16384^2 at 0.1 %, 8192^2 at 1 % with its conversion, B 8192 x 1024 from the
// left): 8 CTAs 1067 / 1106 / 182, 9 1032 / 1096 / 179, 10 1011 / 1088 / 178,
// 12 1024 / 1092 / 194, against 1085 / 1104 / 183 with neither this bound nor
// batched row tails (44 registers). CTAs of 5 to 16 warps: 40 registers, as
// many as hold 48 warps on an SM (16 rows per group, 5396 x 1859, 18 entries a
// row, n = 1148 42 us; 80 registers, what they take without a bound, 62), but 64
// where a lane's columns come by narrow loads, which spill with 40 (8671 x 10332,
// 6 a row, n = 981 60 us with 40, 30 with 64).
constexpr int kRowCtas = 10;
// rows shorter than this walk two column tiles at once: twice the loads in
// flight (16384^2 at 0.1 %, rows of ~16: 1011 us below 16 entries, 959 below
// 24, 955 below 32 or 64; 8192^2 at 1 % is slower from 1000 on)
constexpr int kPairRows = 32;

// V output columns of a lane, in V / W loads of W consecutive columns at
// strides of 32 W: W = V where B's and C's rows are aligned for it, else the
// widest that they are. Each load is contiguous across the warp whatever W is.
template <int W>
struct Piece;
template <>
struct Piece<4> {
    static __device__ __forceinline__ void load(const float *p, float *o)
    {
        const float4 t = __ldg(reinterpret_cast<const float4 *>(p));
        o[0] = t.x; o[1] = t.y; o[2] = t.z; o[3] = t.w;
    }
    static __device__ __forceinline__ void store(float *p, const float *o)
    {
        *reinterpret_cast<float4 *>(p) = make_float4(o[0], o[1], o[2], o[3]);
    }
};
template <>
struct Piece<2> {
    static __device__ __forceinline__ void load(const float *p, float *o)
    {
        const float2 t = __ldg(reinterpret_cast<const float2 *>(p));
        o[0] = t.x; o[1] = t.y;
    }
    static __device__ __forceinline__ void store(float *p, const float *o)
    {
        *reinterpret_cast<float2 *>(p) = make_float2(o[0], o[1]);
    }
};
template <>
struct Piece<1> {
    static __device__ __forceinline__ void load(const float *p, float *o) { o[0] = __ldg(p); }
    static __device__ __forceinline__ void store(float *p, const float *o) { *p = o[0]; }
};

template <int V, int W>
struct Vec {
    static __device__ __forceinline__ void load(const float *p, float (&o)[V])
    {
#pragma unroll
        for (int h = 0; h < V / W; ++h)
            Piece<W>::load(p + h * 32 * W, o + h * W);
    }
    // the pieces whose first column, j + h * 32 W, is at least `from`
    static __device__ __forceinline__ void store(float *p, const float (&o)[V], int64_t j, int64_t from)
    {
#pragma unroll
        for (int h = 0; h < V / W; ++h)
            if (W == V || j + h * 32 * W >= from)
                Piece<W>::store(p + h * 32 * W, o + h * W);
    }
};

// A lane's columns in a 32 V-column tile. W == V: jt is the lane's first
// column. W < V: jt is the tile's, and the last tile of a ragged row starts
// early enough to be whole (n >= 32 V) and stores only its own columns.
template <int V, int W>
struct LaneCols {
    int64_t j, from;
    bool on;
    __device__ __forceinline__ LaneCols(int64_t jt, int lane, int64_t n) : j(jt), from(jt), on(jt < n)
    {
        if constexpr (W < V)
            j = (jt + 32 * V <= n ? jt : n - 32 * V) + lane * W;
    }
};

template <int V, int W, int U, bool PIPE>
__device__ __forceinline__ void row_chain(const Entry *__restrict__ s, int cnt, const float *__restrict__ Bj,
                                          int64_t n, float (&acc)[V])
{
    int i = 0;
    if (PIPE && cnt >= 2 * U) {
        // software pipeline: the B loads of batch i+1 are in flight while
        // batch i is accumulated (the fmaf order per element is unchanged)
        float a[U], b[U][V], a2[U], b2[U][V];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const Entry e = s[u];
            a[u] = e.val;
            Vec<V, W>::load(Bj + static_cast<int64_t>(e.col) * n, b[u]);
        }
#pragma unroll 1
        for (i = U; i + U <= cnt; i += U) {
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const Entry e = s[i + u];
                a2[u] = e.val;
                Vec<V, W>::load(Bj + static_cast<int64_t>(e.col) * n, b2[u]);
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int v = 0; v < V; ++v)
                    acc[v] = fmaf(a[u], b[u][v], acc[v]);
#pragma unroll
            for (int u = 0; u < U; ++u) {
                a[u] = a2[u];
#pragma unroll
                for (int v = 0; v < V; ++v)
                    b[u][v] = b2[u][v];
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int v = 0; v < V; ++v)
                acc[v] = fmaf(a[u], b[u][v], acc[v]);
    }
#pragma unroll 1
    for (; i + U <= cnt; i += U) {
        Entry e[U];
        float b[U][V];
#pragma unroll
        for (int u = 0; u < U; ++u)
            e[u] = s[i + u];
#pragma unroll
        for (int u = 0; u < U; ++u)
            Vec<V, W>::load(Bj + static_cast<int64_t>(e[u].col) * n, b[u]);
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int v = 0; v < V; ++v)
                acc[v] = fmaf(e[u].val, b[u][v], acc[v]);
    }
    // the tail in batches too: a row of 20 entries takes 4 round trips, not 6
    if (U == 8 && i + 4 <= cnt) {
        Entry e[4];
        float b[4][V];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            e[u] = s[i + u];
#pragma unroll
        for (int u = 0; u < 4; ++u)
            Vec<V, W>::load(Bj + static_cast<int64_t>(e[u].col) * n, b[u]);
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int v = 0; v < V; ++v)
                acc[v] = fmaf(e[u].val, b[u][v], acc[v]);
        i += 4;
    }
    if (i + 2 <= cnt) {
        Entry e[2];
        float b[2][V];
#pragma unroll
        for (int u = 0; u < 2; ++u)
            e[u] = s[i + u];
#pragma unroll
        for (int u = 0; u < 2; ++u)
            Vec<V, W>::load(Bj + static_cast<int64_t>(e[u].col) * n, b[u]);
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int v = 0; v < V; ++v)
                acc[v] = fmaf(e[u].val, b[u][v], acc[v]);
        i += 2;
    }
#pragma unroll 1
    for (; i < cnt; ++i) {
        const Entry e = s[i];
        float b[V];
        Vec<V, W>::load(Bj + static_cast<int64_t>(e.col) * n, b);
#pragma unroll
        for (int v = 0; v < V; ++v)
            acc[v] = fmaf(e.val, b[v], acc[v]);
    }
}

// One row's chain over two column tiles at once (same entries, same fmaf
// order per element as row_chain): U entries per batch, 2U B loads in flight.
template <int V, int W, int U>
__device__ __forceinline__ void row_chain_pair(const Entry *__restrict__ s, int cnt, const float *__restrict__ Ba,
                                               const float *__restrict__ Bb, int64_t n, float (&acc_a)[V],
                                               float (&acc_b)[V])
{
    int i = 0;
#pragma unroll 1
    for (; i + U <= cnt; i += U) {
        Entry e[U];
        float ba[U][V], bb[U][V];
#pragma unroll
        for (int u = 0; u < U; ++u)
            e[u] = s[i + u];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            Vec<V, W>::load(Ba + static_cast<int64_t>(e[u].col) * n, ba[u]);
            Vec<V, W>::load(Bb + static_cast<int64_t>(e[u].col) * n, bb[u]);
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int v = 0; v < V; ++v) {
                acc_a[v] = fmaf(e[u].val, ba[u][v], acc_a[v]);
                acc_b[v] = fmaf(e[u].val, bb[u][v], acc_b[v]);
            }
    }
    if (i + 2 <= cnt) {
        Entry e[2];
        float ba[2][V], bb[2][V];
#pragma unroll
        for (int u = 0; u < 2; ++u)
            e[u] = s[i + u];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            Vec<V, W>::load(Ba + static_cast<int64_t>(e[u].col) * n, ba[u]);
            Vec<V, W>::load(Bb + static_cast<int64_t>(e[u].col) * n, bb[u]);
        }
#pragma unroll
        for (int u = 0; u < 2; ++u)
#pragma unroll
            for (int v = 0; v < V; ++v) {
                acc_a[v] = fmaf(e[u].val, ba[u][v], acc_a[v]);
                acc_b[v] = fmaf(e[u].val, bb[u][v], acc_b[v]);
            }
        i += 2;
    }
#pragma unroll 1
    for (; i < cnt; ++i) {
        const Entry e = s[i];
        float ba[V], bb[V];
        Vec<V, W>::load(Ba + static_cast<int64_t>(e.col) * n, ba);
        Vec<V, W>::load(Bb + static_cast<int64_t>(e.col) * n, bb);
#pragma unroll
        for (int v = 0; v < V; ++v) {
            acc_a[v] = fmaf(e.val, ba[v], acc_a[v]);
            acc_b[v] = fmaf(e.val, bb[v], acc_b[v]);
        }
    }
}

// MAXT bounds the CTA size (rows_per_group * col_warps warps); the 1024-thread
// variant (rows_per_group 32) unrolls less to stay within 64 registers.
// col_iters > 1 (only when every group's entries fit one staging chunk): each
// warp walks col_iters column tiles, col_warps tiles apart, reusing the
// staged entries, so short rows do not pay one staging per tile.
template <int V, int W, int MAXT, bool PIPE, bool MULTI>
__global__ void __launch_bounds__(MAXT, MAXT == 128 ? kRowCtas : (MAXT == 512 && !PIPE ? (W == V ? 3 : 2) : 1))
spdm_fp32_kernel(const Entry *__restrict__ packed, const int32_t *__restrict__ row_ptr, int64_t m,
                 int32_t cpg, const float *__restrict__ B, int64_t n, float *__restrict__ C,
                 int32_t col_warps, int32_t col_iters, int32_t chunk_cap, uint32_t *__restrict__ status)
{
    grid_wait_previous();
    row_ptr = written(row_ptr);
    grid_launch_next();
    if (!MULTI)
        col_iters = 1;
    extern __shared__ __align__(128) unsigned char smem[];
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem);
    Entry *s_nz = reinterpret_cast<Entry *>(smem + 128);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int slot = warp / col_warps, sub = warp - slot * col_warps;
    const int64_t r0 = static_cast<int64_t>(blockIdx.x) * cpg;
    const int64_t r_end = r0 + cpg < m ? r0 + cpg : m;
    const int64_t row = r0 + slot;
    const bool has_row = slot < cpg && row < r_end;
    const int64_t tile_stride = static_cast<int64_t>(col_warps) * (32 * V);
    const int64_t j = (static_cast<int64_t>(blockIdx.y) * col_iters * col_warps + sub) * (32 * V) +
                      (W == V ? static_cast<int64_t>(lane) * V : 0);

    const int64_t gs = row_ptr[r0];
    const int64_t ge = row_ptr[r_end];
    if (gs < 0)
        return; // enqueued behind a conversion that did not fit (launch_place): C stays as it is
    int64_t rs = 0, re = 0;
    if (has_row) {
        rs = row_ptr[row];
        re = row_ptr[row + 1];
    }
    if (threadIdx.x == 0) {
        mbar_init(bar, 1);
        fence_mbar_init();
    }
    __syncthreads();

    float acc[V];
    // chunk: entries staged per pass, what the launch's shared memory holds
    const int64_t chunk = chunk_cap < kChunk ? chunk_cap : kChunk;
    const int64_t total = ge - gs;
    const int64_t nchunks = (total + chunk - 1) / chunk;
    // several column tiles per warp from one staging (the group fits one
    // chunk): every tile, the first included, is walked after the staging,
    // two at a time for short rows
    const bool multi_all = MULTI && col_iters > 1 && nchunks == 1;
    // otherwise each of the warp's tiles walks the group chunk by chunk
    const int tiles_staged = multi_all ? 1 : col_iters;
    bool ok = true;
    uint32_t phase = 0;
    for (int it = 0; it < tiles_staged && ok; ++it) {
        const LaneCols<V, W> at(j + it * tile_stride, lane, n);
        const float *Bj = B + at.j;
#pragma unroll
        for (int v = 0; v < V; ++v)
            acc[v] = 0.0f;
        for (int64_t ch = 0; ch < nchunks; ++ch, ++phase) {
            const int64_t cs = gs + ch * chunk;
            const int64_t ce = cs + chunk < ge ? cs + chunk : ge;
            const int64_t a0 = cs & ~static_cast<int64_t>(1); // 16-byte aligned superset
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
                mbar_wait(bar, phase & 1); // let the copy in flight land
                break;
            }
            const int64_t lo = rs > cs ? rs : cs;
            const int64_t hi = re < ce ? re : ce;
            if (!multi_all && at.on && lo < hi)
                row_chain<V, W, (MAXT > 512 ? 4 : 8), PIPE>(s_nz + (lo - a0), static_cast<int>(hi - lo), Bj, n, acc);
            __syncthreads(); // buffer free before the next copy
        }
        if (!multi_all && has_row && at.on && ok)
            Vec<V, W>::store(C + row * n + at.j, acc, at.j, at.from);
    }
    // all column tiles of the warp's row from the (single) staged chunk
    if (multi_all && ok && has_row) {
        const int64_t a0 = gs & ~static_cast<int64_t>(1);
        const Entry *s_row = s_nz + (rs - a0);
        const int cnt = static_cast<int>(re - rs);
        int it = 0;
        // very short rows: two tiles at a time, twice the B loads in flight
        // (longer rows already keep a batch of 8 loads in flight per tile)
        for (; cnt < kPairRows && it + 1 < col_iters; it += 2) {
            const LaneCols<V, W> aa(j + it * tile_stride, lane, n), ab(j + it * tile_stride + tile_stride, lane, n);
            if (!aa.on)
                break;
            float a2[V], b2[V];
#pragma unroll
            for (int v = 0; v < V; ++v)
                a2[v] = b2[v] = 0.0f;
            if (ab.on)
                row_chain_pair<V, W, 4>(s_row, cnt, B + aa.j, B + ab.j, n, a2, b2);
            else if (cnt > 0)
                row_chain<V, W, 4, false>(s_row, cnt, B + aa.j, n, a2);
            Vec<V, W>::store(C + row * n + aa.j, a2, aa.j, aa.from);
            if (ab.on)
                Vec<V, W>::store(C + row * n + ab.j, b2, ab.j, ab.from);
        }
        for (; it < col_iters; ++it) {
            const LaneCols<V, W> at(j + it * tile_stride, lane, n);
            if (!at.on)
                break;
#pragma unroll
            for (int v = 0; v < V; ++v)
                acc[v] = 0.0f;
            if (cnt > 0)
                row_chain<V, W, (MAXT > 512 ? 4 : 8), false>(s_row, cnt, B + at.j, n, acc);
            Vec<V, W>::store(C + row * n + at.j, acc, at.j, at.from);
        }
    }
}

// The short rows of a skewed matrix (its long rows go to spdm_long.cu or
// spdm_split.cu): one warp per (row, 32*V-column tile), nothing staged and no
// CTA barrier -- a row of a dozen entries is all latency, and a staging round
// trip and a group barrier would double it. The row's two pointers come in
// one load (lanes 0 and 1) and are shuffled to the warp. Lane i loads entry i
// of each 32-entry window; the B rows of U entries at a time are loaded
// with their columns shuffled from the owning lanes; each column's fmaf chain
// runs over the row's entries in column order from 0.0f, as in every other
// FP32 kernel. Measured slower on the Zipf workload (0.148 ms for this
// kernel with the long rows beside it): runs of 2-8 rows per warp with the
// next row's entries requested early (0.158-0.171 ms), bundles of 2-8 rows
// whose batches of eight entries run across row boundaries (0.159-0.211 ms),
// and one warp on both 128-column tiles of a row (0.167 ms): at a dozen
// entries per row, more independent warps in flight beat fewer round trips
// per warp. When B is larger than kShortTileMajorBytes the warps walk
// tile-major (every row's first column tile, then every row's second, ...),
// so one column slab of B is live in L2 instead of all of B: 0.150 -> 0.142
// ms with the long rows beside it (B 65536 x 256, 67 MB, was read from DRAM
// about twice in row-major order).
// Forty warps per SM with batches of four: 137 us on the Zipf workload with
// the long rows beside it, against 145 for thirty-two with batches of eight
// (forty-eight with four: 137, sixty-four 147, forty with eight 145).
// With the long rows in their copy-and-chain kernel: 118, forty-eight warps 118,
// thirty-two with batches of eight 127, of six 130.
// Thirty-two with batches of eight where all warps fit four waves and the long
// rows beside them take less time than the short ones (chains of up to 2500
// entries, or sums in pieces): a row of some hundred entries is then the time,
// and twice the loads in flight shorten it. Time with eight over time with four,
// 1379 multiplies, by waves and longest row: up to one wave, up to 600 entries
// .83, 1200 .86, 2500 .93, longer .99; two to four waves .89, .93, .96, .99;
// eight to sixteen .97, .98, 1.01, 1.0; more 1.02. Zipf rows of up to 4096: 16346
// warps 33.8 us with four, 35.2 with eight, 24000 34.6 / 36.7; the same with
// sums in pieces 29.8 / 28.1, 32.1 / 31.1, and 65536 52 / 58.
constexpr int64_t kShortDeepChain = 2500;
constexpr int64_t kShortDeepWaves = 4;
constexpr int short_ctas(int batch) { return batch == 4 ? 20 : 16; } // per SM

template <int V, int U>
__device__ __forceinline__ void short_window(const Entry &my, int nw, bool all_cols, bool has_col,
                                             const float *__restrict__ Bj, int64_t n, float (&acc)[V])
{
    int u0 = 0;
    if (all_cols) { // warp-uniform: every lane takes part in the shuffles below
        // whole batches: no per-entry predicates
        for (; u0 + U <= nw; u0 += U) {
            float a[U], b[U][V];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int col = __shfl_sync(0xffffffffu, my.col, u0 + u);
                a[u] = __shfl_sync(0xffffffffu, my.val, u0 + u);
                Piece<V>::load(Bj + static_cast<int64_t>(col) * n, b[u]);
            }
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int v = 0; v < V; ++v)
                    acc[v] = fmaf(a[u], b[u][v], acc[v]);
        }
    }
    // the tail batch (and lanes past n: shuffles only)
    for (; u0 < nw; u0 += U) {
        float a[U], b[U][V];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int col = __shfl_sync(0xffffffffu, my.col, (u0 + u) & 31);
            a[u] = __shfl_sync(0xffffffffu, my.val, (u0 + u) & 31);
            if (u0 + u < nw && has_col) {
                Piece<V>::load(Bj + static_cast<int64_t>(col) * n, b[u]);
            } else {
#pragma unroll
                for (int v = 0; v < V; ++v)
                    b[u][v] = 0.0f;
            }
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
            if (u0 + u < nw)
#pragma unroll
                for (int v = 0; v < V; ++v)
                    acc[v] = fmaf(a[u], b[u][v], acc[v]);
    }
}

// B larger than this walks tile-major (see spdm_short_kernel)
constexpr int64_t kShortTileMajorBytes = 32ll << 20;

template <int V, int U>
__global__ void __launch_bounds__(64, short_ctas(U))
spdm_short_kernel(const Entry *__restrict__ packed, const int32_t *__restrict__ row_ptr, int64_t m,
                  const float *__restrict__ B, int64_t n, float *__restrict__ C, int32_t tiles, int32_t long_min,
                  int32_t tile_major)
{
    const int lane = threadIdx.x & 31;
    const int64_t gw = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    int64_t row;
    int t;
    if (tile_major) { // every row's tile 0, then every row's tile 1, ...: one B column slab live in L2 at a time
        t = static_cast<int>(gw / m);
        row = gw - static_cast<int64_t>(t) * m;
        if (t >= tiles)
            return;
    } else {
        row = gw / tiles;
        if (row >= m)
            return;
        t = static_cast<int>(gw - row * tiles);
    }
    const int32_t rp = lane < 2 ? row_ptr[row + lane] : 0;
    const int32_t rs = __shfl_sync(0xffffffffu, rp, 0);
    const int cnt = __shfl_sync(0xffffffffu, rp, 1) - rs;
    if (long_min > 0 && cnt >= long_min)
        return; // the long-row kernel writes this row (warp-uniform)
    const int64_t j = static_cast<int64_t>(t) * (32 * V) + static_cast<int64_t>(lane) * V;
    const bool has_col = j < n;
    const bool all_cols = __all_sync(0xffffffffu, has_col);
    const float *Bj = B + (has_col ? j : 0);
    float acc[V];
#pragma unroll
    for (int v = 0; v < V; ++v)
        acc[v] = 0.0f;
    for (int w0 = 0; w0 < cnt; w0 += 32) {
        const int nw = cnt - w0 < 32 ? cnt - w0 : 32;
        Entry my;
        my.col = 0;
        my.val = 0.0f;
        if (lane < nw)
            my = packed[rs + w0 + lane];
        short_window<V, U>(my, nw, all_cols, has_col, Bj, n, acc);
    }
    if (has_col)
        Piece<V>::store(C + row * n + j, acc);
}

// A row tile's sums so far, from C (its own columns only, see LaneCols)
template <int V, int W>
__device__ __forceinline__ void view_resume(const float *c, const LaneCols<V, W> &at, bool resume, float (&acc)[V])
{
#pragma unroll
    for (int h = 0; h < V / W; ++h)
#pragma unroll
        for (int w = 0; w < W; ++w)
            acc[h * W + w] = resume && at.j + h * 32 * W >= at.from ? c[h * 32 * W + w] : 0.0f;
}

// Multiply straight from reference-layout arrays (entries of a group in
// column-then-row order, separate vals/rows/cols, any rows_per_group up to
// 32). One CTA per (group, strip of column tiles): the group's entries are
// staged in chunks and sorted by row in shared memory (each warp ranks its
// rows' entries with one ballot per 32, which keeps their column order), then
// each warp walks its rows over the strip's tiles as spdm_fp32_kernel does:
// the same fmaf chains. An entry whose row is not in its group is skipped.
// Bound like the row walk by the gather of B rows (nnz * n * 4 bytes from
// L2): 4096^2 at 1 %, n = 2048 76 us, against 306 us of a thread per column
// with one 4-byte load in flight and its sums in shared memory.
constexpr int kViewMaxWarps = 8;

template <int V, int W>
__global__ void __launch_bounds__(kViewMaxWarps * 32, 5)
spdm_view_kernel(const float *__restrict__ vals, const int32_t *__restrict__ rows,
                 const int32_t *__restrict__ cols, const int32_t *__restrict__ group_index,
                 const int32_t *__restrict__ nnz_per_group, int64_t m, int32_t cpg, int32_t chunk, int32_t col_iters,
                 const float *__restrict__ B, int64_t n, float *__restrict__ C)
{
    extern __shared__ __align__(128) unsigned char smem[];
    Entry *s_sorted = reinterpret_cast<Entry *>(smem); // by row
    Entry *s_raw = s_sorted + chunk;                   // as stored
    uint8_t *s_lr = reinterpret_cast<uint8_t *>(s_raw + chunk); // row in group, 255: none
    __shared__ int s_start[33];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nwarps = blockDim.x >> 5;
    const int64_t r0 = static_cast<int64_t>(blockIdx.x) * cpg;
    const int nrows = static_cast<int>(r0 + cpg <= m ? cpg : m - r0);
    const int64_t e0 = group_index[blockIdx.x];
    const int64_t total = nnz_per_group[blockIdx.x];
    const int64_t j0 = static_cast<int64_t>(blockIdx.y) * col_iters * (32 * V) + (W == V ? lane * V : 0);
    const unsigned lt = (1u << lane) - 1u;

    // entries [first, first + cnt) of the group into s_sorted, row r's at s_start[r]
    const auto stage = [&](int64_t first, int cnt) {
        __syncthreads(); // the previous chunk has been consumed
        for (int i = threadIdx.x; i < cnt; i += blockDim.x) {
            const int64_t e = e0 + first + i;
            const int64_t lr = rows[e] - r0;
            Entry t;
            t.col = cols[e];
            t.val = vals[e];
            s_raw[i] = t;
            s_lr[i] = lr >= 0 && lr < nrows ? static_cast<uint8_t>(lr) : 255;
        }
        __syncthreads();
        for (int r = warp; r < nrows; r += nwarps) {
            int c = 0;
            for (int i = 0; i < cnt; i += 32)
                c += __popc(__ballot_sync(0xffffffffu, i + lane < cnt && s_lr[i + lane] == r));
            if (lane == 0)
                s_start[r + 1] = c;
        }
        __syncthreads();
        if (warp == 0) {
            int x = lane < nrows ? s_start[lane + 1] : 0;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const int y = __shfl_up_sync(0xffffffffu, x, d);
                if (lane >= d)
                    x += y;
            }
            __syncwarp();
            if (lane < nrows)
                s_start[lane + 1] = x;
            if (lane == 0)
                s_start[0] = 0;
        }
        __syncthreads();
        for (int r = warp; r < nrows; r += nwarps) {
            int at = s_start[r];
            for (int i = 0; i < cnt; i += 32) {
                const bool mine = i + lane < cnt && s_lr[i + lane] == r;
                const unsigned bal = __ballot_sync(0xffffffffu, mine);
                if (mine)
                    s_sorted[at + __popc(bal & lt)] = s_raw[i + lane];
                at += __popc(bal);
            }
        }
        __syncwarp(); // a warp reads only the rows that it sorted
    };

    if (total <= chunk) {
        stage(0, static_cast<int>(total));
        for (int r = warp; r < nrows; r += nwarps) {
            const Entry *s_row = s_sorted + s_start[r];
            const int cnt = s_start[r + 1] - s_start[r];
            float *c_row = C + (r0 + r) * n;
            int it = 0;
            for (; cnt < kPairRows && it + 1 < col_iters; it += 2) {
                const LaneCols<V, W> aa(j0 + it * (32 * V), lane, n), ab(j0 + (it + 1) * (32 * V), lane, n);
                if (!aa.on)
                    break;
                float a2[V], b2[V];
#pragma unroll
                for (int v = 0; v < V; ++v)
                    a2[v] = b2[v] = 0.0f;
                if (ab.on)
                    row_chain_pair<V, W, 4>(s_row, cnt, B + aa.j, B + ab.j, n, a2, b2);
                else
                    row_chain<V, W, 4, false>(s_row, cnt, B + aa.j, n, a2);
                Vec<V, W>::store(c_row + aa.j, a2, aa.j, aa.from);
                if (ab.on)
                    Vec<V, W>::store(c_row + ab.j, b2, ab.j, ab.from);
            }
            for (; it < col_iters; ++it) {
                const LaneCols<V, W> at(j0 + it * (32 * V), lane, n);
                if (!at.on)
                    break;
                float acc[V];
#pragma unroll
                for (int v = 0; v < V; ++v)
                    acc[v] = 0.0f;
                row_chain<V, W, 8, false>(s_row, cnt, B + at.j, n, acc);
                Vec<V, W>::store(c_row + at.j, acc, at.j, at.from);
            }
        }
        return;
    }
    // more entries than one chunk: a tile's sums live in C between chunks
    for (int64_t first = 0; first < total; first += chunk) {
        stage(first, static_cast<int>(total - first < chunk ? total - first : chunk));
        for (int r = warp; r < nrows; r += nwarps) {
            const Entry *s_row = s_sorted + s_start[r];
            const int cnt = s_start[r + 1] - s_start[r];
            for (int it = 0; it < col_iters; ++it) {
                const LaneCols<V, W> at(j0 + it * (32 * V), lane, n);
                if (!at.on)
                    break;
                float acc[V];
                view_resume<V, W>(C + (r0 + r) * n + at.j, at, first > 0, acc);
                row_chain<V, W, 8, false>(s_row, cnt, B + at.j, n, acc);
                Vec<V, W>::store(C + (r0 + r) * n + at.j, acc, at.j, at.from);
            }
        }
    }
}

} // namespace

int device_sms()
{
    static int sms = 0;
    if (!sms) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms <= 0)
            sms = 152;
    }
    return sms;
}

bool row_lengths_skewed(int64_t m, int64_t nnz, int64_t max_row)
{
    const double mean = m > 0 ? static_cast<double>(nnz) / static_cast<double>(m) : 0.0;
    return max_row >= 256 && static_cast<double>(max_row) > 8.0 * (mean > 1.0 ? mean : 1.0);
}

constexpr int64_t kWideCols = 1 << 20;

LaunchShape pick_shape(const gcoo_params &p, int64_t m, int64_t n, int64_t nnz, int64_t max_row,
                       uintptr_t b_addr, uintptr_t c_addr)
{
    LaunchShape s;
    // Heavy-tailed row lengths (the longest row far above the mean): one row
    // per CTA, so a long row does not hold its group's other rows back, and
    // the next batch's B loads in flight, since a long row is one long
    // dependent chain. The per-element fmaf order is the same either way.
    const double mean = m > 0 ? static_cast<double>(nnz) / static_cast<double>(m) : 0.0;
    const bool skewed = row_lengths_skewed(m, nnz, max_row);
    s.rows = skewed ? 1 : p.rows_per_group;
    int w = 4; // the widest aligned load
    if (n % 4 != 0 || (b_addr & 15) || (c_addr & 15))
        w = 2;
    if (w == 2 && (n % 2 != 0 || (b_addr & 7) || (c_addr & 7)))
        w = 1;
    int v = p.vec > 0 ? p.vec : (n >= 128 ? 4 : (n >= 64 ? 2 : 1));
    if (v != 1 && v != 2 && v != 4)
        v = 1;
    // as many columns per lane from narrower loads: an entry read then serves
    // as many FMAs as in an aligned B (4001 x 3999 at 2 %: n = 2047 157 us
    // against 339 at one column per lane, n = 2046 149 against 185 at two,
    // n = 2048 135). Whole tiles only, two of them in pairs of columns (n =
    // 130 28 us against 26 at two columns per lane); and not where the number
    // of narrow tiles decides whether the launch is possible.
    while (v > w && (n < (w == 2 ? 64 : 32) * v || n > kWideCols))
        v /= 2;
    s.width = w < v ? w : v;
    s.vec = v;
    // Every group fits one staging chunk: one staging of a group's entries
    // can serve several column tiles per warp. With the launch shape left to
    // the library, a CTA takes fewer rows (down to one) where that makes its
    // group fit; rows of up to 2046 entries then stay on the one-warp-per-row
    // path (any rows per CTA gives the same fmaf chains). Where not even one
    // row fits, one row too: its CTA's passes wait for nobody else's (3000 x 5000
    // at 50 %, n = 1: 32 rows 1667 us, 4 rows 212, one 155; 300 x 8192, n = 16 7206 /
    // 840 / 216).
    const auto fits = [&](int rows) { return max_row > 0 && max_row * static_cast<int64_t>(rows) + 2 <= kChunk; };
    if (!skewed && p.warps <= 0 && p.col_warps <= 0 && max_row > 0) // 0: not known
        while (s.rows > 1 && !fits(s.rows))
            s.rows = s.rows / 2 > 0 ? s.rows / 2 : 1;
    const int cpg = s.rows;
    const bool one_chunk = fits(s.rows);
    int cw;
    if (p.col_warps > 0)
        cw = p.col_warps;
    else if (p.warps <= 0 && !skewed && one_chunk)
        // One warp per row, 4-warp CTAs, each warp walking several column
        // tiles of its row: measured on GB300 1.06 against 1.15 ms (8192^2,
        // 1 %) and 0.178 against 0.201 ms (8192^2, 0.1 %) for two warps per
        // row: twice the CTAs resident per SM keep more B loads in flight,
        // and the latency of the loads is what bounds these matrices.
        cw = 1;
    else {
        const int target = p.warps > 0 ? p.warps : 8;
        cw = target / cpg;
        if (cw < 1)
            cw = 1;
        // no wider than the matrix
        while (cw > 1 && static_cast<int64_t>(cw / 2) * 32 * v >= n)
            cw /= 2;
    }
    if (cw * cpg > 32)
        cw = 32 / cpg > 0 ? 32 / cpg : 1;
    s.col_warps = cw;
    s.warps = cw * cpg;
    s.depth = p.depth > 0 ? p.depth : (skewed ? 2 : 1);
    s.col_iters = 1;
    if (one_chunk) {
        const int64_t tile = static_cast<int64_t>(s.col_warps) * 32 * s.vec;
        const int64_t ny = (n + tile - 1) / tile;
        // about 768 columns per CTA (0.5-0.9 K columns measured best from
        // 2048^2 to 16384^2 at 1 % to 0.1 % density), but at least four waves
        // of CTAs on small matrices: the last wave's share of the time (4096^2
        // at 5 % 623 us with two, 604 with four; 2048^2 at 10 % 148 and 141;
        // 4096^2 at 1.5 %, n = 2048 108 with one, 107 and 100). Short rows: a
        // CTA's staging is the larger share, so one wave under 8 entries
        // (2048^2 at 0.1 % 8.1 us, 9.2 with two, 11.2 with four; 2880 x 1527
        // at 0.28 %, n = 1568 11.3, 11.4 and 14.0) and two under 16 (2048^2 at
        // 0.5 % 16.0, 15.1 and 16.5), as long as no row is much longer: its CTA
        // is then the time (6951 x 4723, 3 entries a row and up to 237, n = 728
        // 80 us with one wave, 45 with two, 26 with four; lines at 1/2 to 1/5 of
        // the longest row differ by less than 0.3 % over 2079 multiplies)
        int64_t ci = 768 / tile;
        const int64_t groups = (m + s.rows - 1) / s.rows;
        const int64_t resident = static_cast<int64_t>(device_sms()) * (s.warps <= 4 ? kRowCtas : 6);
        const double len = mean > max_row / 3.0 ? mean : max_row / 3.0;
        const int64_t waves = len < 8.0 ? 1 : (len < 16.0 ? 2 : 4);
        const int64_t by_grid = groups * ny / (waves * resident);
        ci = ci > by_grid ? by_grid : ci;
        ci = ci < 1 ? 1 : (ci > ny ? ny : ci);
        s.col_iters = static_cast<int>(ci > 64 ? 64 : ci);
        // shared memory for the largest possible group only, not a full
        // chunk: the rest of the SM's L1 array then holds B loads in flight
        // (measured 2-6 % faster at 0.1-1 % density)
        s.chunk = static_cast<int>(max_row * s.rows);
    }
    // Rows of some hundred entries and little more than one wave of CTAs: their
    // spread over the SMs is the time. Not started while the predecessor drains,
    // where they would take whichever slots come free first (1924 x 249, 154
    // entries a row, n = 236: 22.3 us behind another multiply, 18.9 so; shorter
    // rows gain by it, 6 % on average over 1504 multiplies, and so does less than
    // half a wave, which finds slots whoever drains: 355 x 11466, 122 a row, 16 rows
    // per group, n = 184 11.0 against 16.6); and with twelve 4-warp CTAs per SM
    // where that is one wave and kRowCtas are not (1199 x 4114, 170 a row, n = 728:
    // 42.5 us with ten, 34.3 with twelve).
    if (mean >= 100.0) {
        const int64_t tile = static_cast<int64_t>(s.col_warps) * 32 * s.vec * s.col_iters;
        const int64_t ctas = (m + s.rows - 1) / s.rows * ((n + tile - 1) / tile), sms = device_sms();
        const int64_t twelve = 48 / s.warps < 32 ? 48 / s.warps : 32; // of CTAs that wide as many as 48 warps
        const int64_t per_sm = s.warps <= 4 && 4 * kRowCtas / s.warps < twelve ? 4 * kRowCtas / s.warps : twelve;
        s.after = 10 * ctas > 13 * per_sm * sms || 10 * ctas < (mean < 500.0 ? 5 : 3) * per_sm * sms;
        s.tight = s.warps <= 4 && ctas > per_sm * sms && ctas <= twelve * sms;
    }
    return s;
}

cudaError_t launch_spdm_fp32(const Entry *packed, const int32_t *row_ptr, int64_t m, const float *B, int64_t n,
                             float *C, const LaunchShape &s, uint32_t *status, cudaStream_t st)
{
    const int32_t cpg = s.rows; // rows per CTA (any value gives the same fmaf chains)
    const int64_t ng = (m + cpg - 1) / cpg;
    const int64_t tile = static_cast<int64_t>(s.col_warps) * 32 * s.vec * (s.col_iters > 1 ? s.col_iters : 1);
    const int64_t ny = (n + tile - 1) / tile;
    if (ng <= 0 || ny <= 0)
        return cudaSuccess;
    if (ny > 65535)
        return cudaErrorInvalidConfiguration;
    dim3 grid(static_cast<unsigned>(ng), static_cast<unsigned>(ny));
    const int threads = s.warps * 32;
    // entries staged per pass and the shared memory that holds them (the
    // kernel stages any larger group in several passes)
    const int chunk = s.chunk > 0 && s.chunk < kChunk ? s.chunk : kChunk;
    const int smem = 128 + (chunk + 2) * static_cast<int>(sizeof(Entry));
    const auto go = [&](auto kernel, int32_t col_iters) {
        if (s.after)
            return launch_after(kernel, grid, dim3(threads), smem, st, packed, row_ptr, m, cpg, B, n, C, s.col_warps,
                                col_iters, chunk, status);
        kernel<<<grid, threads, smem, st>>>(packed, row_ptr, m, cpg, B, n, C, s.col_warps, col_iters, chunk, status);
        return cudaGetLastError();
    };
#define GCOO_FP32_LAUNCH(V, W, T, P)                                                                       \
    do {                                                                                                \
        if (s.col_iters > 1)                                                                            \
            le = go(spdm_fp32_kernel<V, W, T, P, true>, s.col_iters);                                    \
        else                                                                                            \
            le = go(spdm_fp32_kernel<V, W, T, P, false>, 1);                                             \
    } while (0)
#define GCOO_FP32_VEC(T, P)                                                                             \
    do {                                                                                                \
        if (s.vec == 4 && s.width == 4) GCOO_FP32_LAUNCH(4, 4, T, P);                                   \
        else if (s.vec == 4 && s.width == 2) GCOO_FP32_LAUNCH(4, 2, T, P);                              \
        else if (s.vec == 4) GCOO_FP32_LAUNCH(4, 1, T, P);                                              \
        else if (s.vec == 2 && s.width == 2) GCOO_FP32_LAUNCH(2, 2, T, P);                              \
        else if (s.vec == 2) GCOO_FP32_LAUNCH(2, 1, T, P);                                              \
        else GCOO_FP32_LAUNCH(1, 1, T, P);                                                              \
    } while (0)
    const bool pipe = s.depth >= 2;
    cudaError_t le = cudaSuccess;
    if (threads <= 128 && !pipe && !s.tight) {
        GCOO_FP32_VEC(128, false);
    } else if (threads <= 512) {
        if (pipe) GCOO_FP32_VEC(512, true);
        else GCOO_FP32_VEC(512, false);
    } else {
        if (pipe) GCOO_FP32_VEC(1024, true);
        else GCOO_FP32_VEC(1024, false);
    }
#undef GCOO_FP32_VEC
#undef GCOO_FP32_LAUNCH
    count_launches(1);
    return le;
}

cudaError_t launch_spdm_short(const Entry *packed, const int32_t *row_ptr, int64_t m, int64_t k, const float *B,
                              int64_t n, float *C, int32_t long_min, int64_t chain, cudaStream_t st)
{
    if (m <= 0 || n <= 0)
        return cudaSuccess;
    const uintptr_t b = reinterpret_cast<uintptr_t>(B), c = reinterpret_cast<uintptr_t>(C);
    int v = 1;
    if (n % 4 == 0 && !(b & 15) && !(c & 15))
        v = 4;
    else if (n % 2 == 0 && !(b & 7) && !(c & 7))
        v = 2;
    const int64_t tiles = (n + 32 * v - 1) / (32 * v);
    const int64_t warps = m * tiles;
    // two-warp CTAs: rows of very different lengths do not hold one another's
    // CTA slot (8-warp CTAs: 145 us on the Zipf workload, 2-warp: 127 us, 1-warp: 134 us)
    const int64_t blocks = (warps + 1) / 2;
    if (tiles > 0x7fffffffLL || blocks > 0x7fffffffLL)
        return cudaErrorInvalidConfiguration;
    const unsigned grid = static_cast<unsigned>(blocks);
    const int32_t nt = static_cast<int32_t>(tiles);
    const int32_t tm = tiles > 1 && k * n * 4 > kShortTileMajorBytes ? 1 : 0;
    const bool deep = chain <= kShortDeepChain && warps <= kShortDeepWaves * device_sms() * 2 * short_ctas(4);
#define GCOO_SHORT(V)                                                                                               \
    (deep ? spdm_short_kernel<V, 8> : spdm_short_kernel<V, 4>)<<<grid, 64, 0, st>>>(packed, row_ptr, m, B, n, C, nt, \
                                                                                    long_min, tm)
    if (v == 4)
        GCOO_SHORT(4);
    else if (v == 2)
        GCOO_SHORT(2);
    else
        GCOO_SHORT(1);
#undef GCOO_SHORT
    count_launches(1);
    return cudaGetLastError();
}

cudaError_t launch_spdm_view(const gcoo_view &a, const float *B, int64_t n, float *C, cudaStream_t st)
{
    if (a.n_group <= 0 || n <= 0)
        return cudaSuccess;
    if ((n + 127) / 128 > 65535) // the widest B this entry point takes
        return cudaErrorInvalidConfiguration;
    const int cpg = a.rows_per_group;
    // Short rows: a CTA's staging is most of it, and two warps of a few rows
    // each let more groups be resident (60000 x 1000, 1 entry a row, n = 1: 4 rows
    // per group 23.6 us, 19.6 so, 8 rows 23.7 / 17.2; 32 rows 18.5 / 18.9, n = 130
    // 27.9 / 40.0)
    const double len = a.m > 0 ? static_cast<double>(a.nnz) / static_cast<double>(a.m) : 0.0;
    const int most = len < 8.0 && cpg <= 8 ? 2 : kViewMaxWarps;
    const int warps = cpg < most ? cpg : most;
    gcoo_params p{};
    p.rows_per_group = cpg;
    p.warps = p.col_warps = 1;
    LaunchShape s = pick_shape(p, a.m, n, a.nnz, 0, reinterpret_cast<uintptr_t>(B), reinterpret_cast<uintptr_t>(C));
    // entries staged at once: a power of two above twice the mean group, at most
    // 256 (4.4 KB) per warp, so that the shared memory leaves room for as many
    // warps as the registers do (1873 x 2076 at 33 %, 1 row per group, n = 55 61 us
    // against 140 with 2048 entries, n = 800 218 / 652; 4 rows, n = 256 85 / 121)
    const int64_t mean = a.nnz / a.n_group;
    int chunk = 256;
    while (chunk < warps * 256 && chunk < 2 * mean + 64)
        chunk *= 2;
    // as the row walk: about 768 columns per CTA, but four waves of CTAs, two
    // of rows under 16 entries, one at most under 8 (1 entry a row, four waves /
    // as now, us: 5606 x 336, n = 218, 4 rows per group 13.1 / 9.8, n = 801 18.5 /
    // 12.2; 8000 x 300, n = 130 13.3 / 9.9)
    const int64_t tile = 32 * s.vec, tiles = (n + tile - 1) / tile;
    const int64_t resident = static_cast<int64_t>(device_sms()) * kRowCtas * 4 / warps;
    const int64_t waves = len < 8.0 ? 1 : (len < 16.0 ? 2 : 4);
    int64_t ci = (a.n_group * tiles + (len < 8.0 ? resident - 1 : 0)) / (waves * resident);
    ci = ci > 768 / tile ? 768 / tile : ci;
    ci = ci < 1 ? 1 : ci;
    while ((tiles + ci - 1) / ci > 65535)
        ci *= 2;
    const dim3 grid(static_cast<unsigned>(a.n_group), static_cast<unsigned>((tiles + ci - 1) / ci));
    const size_t smem = static_cast<size_t>(chunk) * (2 * sizeof(Entry) + 1);
#define GCOO_VIEW(V, W)                                                                                             \
    spdm_view_kernel<V, W><<<grid, warps * 32, smem, st>>>(a.vals, a.rows, a.cols, a.group_index, a.nnz_per_group, \
                                                           a.m, cpg, chunk, static_cast<int32_t>(ci), B, n, C)
    if (s.vec == 4 && s.width == 4) GCOO_VIEW(4, 4);
    else if (s.vec == 4 && s.width == 2) GCOO_VIEW(4, 2);
    else if (s.vec == 4) GCOO_VIEW(4, 1);
    else if (s.vec == 2 && s.width == 2) GCOO_VIEW(2, 2);
    else if (s.vec == 2) GCOO_VIEW(2, 1);
    else GCOO_VIEW(1, 1);
#undef GCOO_VIEW
    count_launches(1);
    return cudaGetLastError();
}

} // namespace gcoo
