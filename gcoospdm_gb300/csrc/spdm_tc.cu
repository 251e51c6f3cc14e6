// spdm_tc.cu -- tensor-core (tcgen05) engine for matrices whose nonzeros
// densify into 16-wide blocks.
//
// Plan (built once per handle and form, from the GCOO entries):
//   * A is cut into panels (256 rows for BF16 and FP8-B, 128 for split-BF16);
//     a tile is the panel's 16-column slice at column block cb, active when
//     it holds any entry;
//   * each active tile is stored densely (zeros where A has none) as BF16,
//     each 128-row half in the K-major, 32-byte-swizzled shared-memory layout
//     of tcgen05 (row r at r*32 bytes, 16-byte chunk c at
//     (c ^ ((r >> 2) & 1)) * 16), so a 4 KB copy lands a half ready for the
//     MMA; split-BF16 keeps two more tiles (lo = x - hi and lo2 = x - hi -
//     lo, each rounded to BF16: hi + lo + lo2 is x exactly), stored side by
//     side;
//   * B is converted per call into tiles of N output columns x 16 k (the
//     same layout, N rows of 32 bytes).
// BF16 / FP8-B kernel (spdm_tc_pair_kernel): a cluster of two CTAs on two
// SMs per (256-row panel, 256 or 512 output columns), or per equal share of
// the products where those would leave SMs idle; each CTA streams its 128-row
// half of four tiles and its 128-column halves of their B tiles per stage
// with tensor-map bulk copies (cta_group::2, completing on the first CTA's
// barrier), and the first CTA issues tcgen05.mma.cta_group::2 (M=256, N=256,
// K=16) into both CTAs' tensor memory, one accumulator per 256 columns.
// Split-BF16 kernel (spdm_tc_split_kernel): equal shares of the (tile, 128
// columns) products, or (panel, 128 columns) where panels have few tiles, two
// CTAs per SM, one stage per tile, six MMAs per tile. Every wait is bounded.
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_fp8.h>

#include <cuda.h>

#include <mutex>

#include "handle.hpp"

namespace gcoo {

constexpr int kPanel = 128;   // rows of a tile half (one CTA's MMA rows)
constexpr int kTileK = 16;    // columns per tile (MMA K)
constexpr int kTileBytes = kPanel * kTileK * 2; // one 128-row half
constexpr uint64_t kDrainNs = 2000000; // after a wait gives up: time for copies in flight to land

struct TcPlan {
    int64_t panels = 0, kb = 0, tiles = 0;
    int panel_rows = kPanel; // 256 for the pair kernel (two halves per tile), 128 for split-BF16
    bool split = false;
    int64_t nnz = 0;
    DevBuf<int32_t> pf;       // exclusive prefix over (panel, cb) flags, size panels*kb + 1
    DevBuf<int32_t> tile_cb;  // cb of each tile (ascending within a panel)
    DevBuf<int32_t> tile_panel; // panel of each tile
    DevBuf<uint16_t> a_hi;    // tiles * (panel_rows / 128) * 2048 bf16 (swizzled halves)
    DevBuf<uint16_t> a_lo;    // split only: tiles * 2 * 2048 bf16 (lo, then lo2, per tile)
    DevBuf<int64_t> scratch;
    // B workspace (per call)
    DevBuf<uint16_t> b_hi, b_lo; // b_lo (split only): lo then lo2 per B tile
    DevBuf<float> part;          // sums of (panel, strip of columns) that lie in several shares
    int64_t b_n = 0;
    // FP8-B: per-column power-of-two scales (and their absmax scratch)
    DevBuf<float> b_scale;
    DevBuf<unsigned> b_amax;
};

void destroy_tc_plan(TcPlan *p) { delete p; }

namespace {

// ---- small PTX wrappers for tcgen05 ----------------------------------------------
__device__ __forceinline__ uint64_t smem_desc_sw32(uint32_t saddr)
{
    // start address >> 4 | LBO (unused for swizzled K-major) = 1 | SBO = 256 B (8 rows x 32 B)
    // | version 1 (bits 46-47) | layout SWIZZLE_32B = 6 (bits 61-63)
    return static_cast<uint64_t>((saddr >> 4) & 0x3FFFu) | (static_cast<uint64_t>(1) << 16) |
           (static_cast<uint64_t>(256 >> 4) << 32) | (static_cast<uint64_t>(1) << 46) |
           (static_cast<uint64_t>(6) << 61);
}

__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N)
{
    // D f32 (bits 4-5 = 1), A bf16 (7-9 = 1), B bf16 (10-12 = 1), both K-major,
    // N >> 3 at bits 17-22, M >> 4 at bits 24-28.
    return (1u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(N >> 3) << 17) |
           (static_cast<uint32_t>(M >> 4) << 24);
}

__device__ __forceinline__ void tc_mma(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
                 "l"(a), "l"(b), "r"(idesc), "r"(acc)
                 : "memory");
}

__device__ __forceinline__ void tc_commit(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// One lane of a converged warp, the same at every call
__device__ __forceinline__ bool elect_one()
{
    uint32_t one;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(one));
    return one != 0;
}

__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float (&v)[32])
{
    uint32_t r[32];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
                 "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
                   "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]),
                   "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]),
                   "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i)
        v[i] = __uint_as_float(r[i]);
}

// 32 consecutive columns of a row of C, `left` of them inside it
__device__ __forceinline__ void store_row32(float *out, const float (&v)[32], int64_t left)
{
    if (left >= 32) {
#pragma unroll
        for (int q = 0; q < 32; q += 4)
            *reinterpret_cast<float4 *>(out + q) = make_float4(v[q], v[q + 1], v[q + 2], v[q + 3]);
    } else {
#pragma unroll
        for (int q = 0; q < 32; ++q)
            if (q < left)
                out[q] = v[q];
    }
}

// The same for a warp's 32 rows from C row `row`, columns from j, through a
// 32 x kStageRow staging tile of its own: each store instruction writes four
// rows' 128 contiguous bytes instead of 16 bytes of 32 rows. m, n: C's
// extents (n a multiple of 4).
constexpr int kStageRow = 36; // floats: 16-byte rows that a quarter warp writes without bank conflicts

__device__ __forceinline__ void store_warp32(float *stage, const float (&v)[32], float *__restrict__ C, int64_t row,
                                             int64_t j, int64_t m, int64_t n)
{
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < 32; q += 4)
        *reinterpret_cast<float4 *>(stage + lane * kStageRow + q) = make_float4(v[q], v[q + 1], v[q + 2], v[q + 3]);
    __syncwarp();
    const int r0 = lane >> 3, c = (lane & 7) * 4;
#pragma unroll
    for (int r = r0; r < 32; r += 4) {
        const float4 x = *reinterpret_cast<const float4 *>(stage + r * kStageRow + c);
        if (row + r < m && j + c < n)
            *reinterpret_cast<float4 *>(C + (row + r) * n + j + c) = x;
    }
    __syncwarp(); // the tile is rewritten by the next call
}

// Byte offset of element (row r, column c) of a 32-byte-row K-major tile in
// the 32B-swizzled layout.
__host__ __device__ __forceinline__ uint32_t sw32_offset(uint32_t r, uint32_t c)
{
    const uint32_t chunk = (c >> 3) ^ ((r >> 2) & 1u);
    return r * 32u + chunk * 16u + (c & 7u) * 2u;
}

// ---- plan building --------------------------------------------------------------------
__global__ void tile_flags_kernel(const Entry *__restrict__ packed, const int32_t *__restrict__ row_ptr, int64_t m,
                                  int64_t kb, int panel_rows, int32_t *__restrict__ flags)
{
    const int lane = threadIdx.x & 31;
    const int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
    for (int64_t r = warp; r < m; r += nw) {
        const int64_t base = (r / panel_rows) * kb;
        for (int64_t e = row_ptr[r] + lane; e < row_ptr[r + 1]; e += 32)
            flags[base + packed[e].col / kTileK] = 1;
    }
}

__global__ void tile_list_kernel(const int32_t *__restrict__ pf, int64_t total, int64_t kb, int32_t *__restrict__ tile_cb,
                                 int32_t *__restrict__ tile_panel)
{
    for (int64_t f = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; f < total;
         f += static_cast<int64_t>(gridDim.x) * blockDim.x)
        if (pf[f + 1] != pf[f]) {
            tile_cb[pf[f]] = static_cast<int32_t>(f % kb);
            tile_panel[pf[f]] = static_cast<int32_t>(f / kb);
        }
}

// lo (split-BF16 only) is filled with 128-row panels.
__global__ void tile_fill_kernel(const Entry *__restrict__ packed, const int32_t *__restrict__ row_ptr, int64_t m,
                                 int64_t kb, int panel_rows, const int32_t *__restrict__ pf,
                                 __nv_bfloat16 *__restrict__ hi, __nv_bfloat16 *__restrict__ lo)
{
    const int lane = threadIdx.x & 31;
    const int64_t warp = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
    const int64_t tile_elems = static_cast<int64_t>(panel_rows / kPanel) * (kTileBytes / 2);
    for (int64_t r = warp; r < m; r += nw) {
        const int64_t base = (r / panel_rows) * kb;
        const uint32_t lr = static_cast<uint32_t>(r % panel_rows);
        for (int64_t e = row_ptr[r] + lane; e < row_ptr[r + 1]; e += 32) {
            const Entry t = packed[e];
            const int64_t tile = pf[base + t.col / kTileK];
            const uint32_t off = (lr / kPanel) * (kTileBytes / 2) +
                                 sw32_offset(lr % kPanel, static_cast<uint32_t>(t.col % kTileK)) / 2;
            const __nv_bfloat16 h = __float2bfloat16_rn(t.val);
            hi[tile * tile_elems + off] = h;
            if (lo) {
                const float r1 = t.val - __bfloat162float(h); // exact
                const __nv_bfloat16 l1 = __float2bfloat16_rn(r1);
                lo[tile * kTileBytes + off] = l1;
                lo[tile * kTileBytes + kTileBytes / 2 + off] = __float2bfloat16_rn(r1 - __bfloat162float(l1));
            }
        }
    }
}

// B (k x n FP32, row-major) -> tiles [jt][cb] of N rows (output columns) x 16 k, swizzled.
// With fp8_scale (FP8-B): each value is first quantized to E4M3 in units of
// its column's power-of-two scale, then stored as the exact BF16 value of
// E4M3 x scale, so the BF16 MMA multiplies the FP8-B operand exactly.
// One CTA per 256-column tile (two 128-column ones): the 16 x N block of B is
// staged in shared memory with coalesced 16-byte loads, all of a thread's in
// flight together, then thread jj builds tile row jj (output column jt*N + jj: 16 values read down a
// shared-memory column, conflict-free across the warp) and writes its 32
// bytes with two 16-byte stores, so a warp writes 1 KB contiguous. B 8192 x
// 1024: 9.5 us (50 MB), split 17 us (84 MB); the terms computed whatever the
// form and the loads in a loop took 14 and 25.5 us.
__device__ __forceinline__ uint32_t pack_bf16(__nv_bfloat16 lo_half, __nv_bfloat16 hi_half)
{
    return static_cast<uint32_t>(__bfloat16_as_ushort(lo_half)) |
           (static_cast<uint32_t>(__bfloat16_as_ushort(hi_half)) << 16);
}

// N = 256 columns (the pair kernel), or 128 with SPLIT. SPLIT: the lo and lo2
// terms too; FP8: through E4M3 first. Needs n % 4 == 0 and B 16-byte aligned
// (the tensor engine takes n % 16 == 0).
template <bool SPLIT, bool FP8>
__global__ void __launch_bounds__(256)
b_tiles_kernel(const float *__restrict__ B, int64_t k, int64_t n, int64_t kb, __nv_bfloat16 *__restrict__ hi,
               __nv_bfloat16 *__restrict__ lo, const float *__restrict__ fp8_scale)
{
    grid_launch_next();
    constexpr int N = SPLIT ? 128 : 256, kT = 256 / N; // kT tiles (column blocks of 16 k) per CTA
    constexpr int kLoads = kTileK * N * kT / 4 / 256;  // float4 per thread
    __shared__ __align__(16) float blk[kT][kTileK][N];
    const int64_t cb0 = static_cast<int64_t>(blockIdx.x) * kT;
    const int64_t jt = blockIdx.y;
    constexpr size_t tile_elems = static_cast<size_t>(N) * kTileK;
    float4 v4[kLoads];
#pragma unroll
    for (int u = 0; u < kLoads; ++u) {
        const int i = u * 256 + threadIdx.x;
        const int r = i / (N / 4), c4 = i % (N / 4); // r: row inside the kT blocks
        const int64_t c = cb0 * kTileK + r, j = jt * N + c4 * 4;
        v4[u] = c < k && j < n ? __ldg(reinterpret_cast<const float4 *>(B + c * n + j)) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
#pragma unroll
    for (int u = 0; u < kLoads; ++u) {
        const int i = u * 256 + threadIdx.x;
        *reinterpret_cast<float4 *>(&blk[0][0][0] + i * 4) = v4[u];
    }
    __syncthreads();
    const int t = threadIdx.x / N, jj = threadIdx.x % N;
    const int64_t tile = jt * kb + cb0 + t;
    if (cb0 + t >= kb)
        return;
    const int64_t j = jt * N + jj;
    float sc = 1.0f;
    if (FP8 && j < n)
        sc = fp8_scale[j];
    // a power of two in the normal range has an exact reciprocal, so
    // v * inv is v / sc exactly; otherwise divide
    const bool by_inv = sc >= 1.17549435e-38f && sc <= 8.50705917e37f;
    const float inv = by_inv ? 1.0f / sc : 0.0f;
    uint32_t wh[8], wl[8], wl2[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        __nv_bfloat16 h2[2], l2[2], m2[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            float v = blk[t][q * 2 + e][jj];
            if (FP8 && j < n) {
                const __nv_fp8_storage_t f8 =
                    __nv_cvt_float_to_fp8(by_inv ? v * inv : v / sc, __NV_SATFINITE, __NV_E4M3);
                v = __half2float(__half(__nv_cvt_fp8_to_halfraw(f8, __NV_E4M3))) * sc;
            }
            h2[e] = __float2bfloat16_rn(v);
            if (SPLIT) {
                const float r1 = v - __bfloat162float(h2[e]); // exact
                l2[e] = __float2bfloat16_rn(r1);
                m2[e] = __float2bfloat16_rn(r1 - __bfloat162float(l2[e]));
            }
        }
        wh[q] = pack_bf16(h2[0], h2[1]);
        if (SPLIT) {
            wl[q] = pack_bf16(l2[0], l2[1]);
            wl2[q] = pack_bf16(m2[0], m2[1]);
        }
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const uint32_t off = sw32_offset(static_cast<uint32_t>(jj), static_cast<uint32_t>(half * 8)) / 2;
        const int w0 = half * 4;
        *reinterpret_cast<uint4 *>(hi + tile * tile_elems + off) = make_uint4(wh[w0], wh[w0 + 1], wh[w0 + 2], wh[w0 + 3]);
        if (SPLIT) {
            *reinterpret_cast<uint4 *>(lo + 2 * tile * tile_elems + off) =
                make_uint4(wl[w0], wl[w0 + 1], wl[w0 + 2], wl[w0 + 3]);
            *reinterpret_cast<uint4 *>(lo + (2 * tile + 1) * tile_elems + off) =
                make_uint4(wl2[w0], wl2[w0 + 1], wl2[w0 + 2], wl2[w0 + 3]);
        }
    }
}

// ---- split-BF16: one CTA per equal share of the tiles, or per panel and strip ----------
// The tile products (tile t of the plan x 128 output columns jt) are ordered
// w = jt * tiles + t and cut into equal consecutive shares, one per CTA, two
// CTAs per SM: no wave of CTAs is nearly empty and a few panels fill the GPU.
// Measured with 16 x 16 blocks at 25 % (us; a CTA per panel and 128 columns
// before): 8192^2, n = 1024 472-478 -> 436-453 by GPU and run (the MMAs 387 at
// their measured peak rate, 13 of fix-up), n = 128 216 -> 84; 2048 x 8192, n = 256 222 -> 57;
// 2048^2, n = 1024 67 -> 49; 1024^2 at 15 %, n = 64 32 -> 24. A share is
// walked panel by panel; a (panel, jt) that lies in one share is written to
// C, the others' sums go to a workspace and tc_fixup_kernel adds them in
// order. Every CTA's share and every place of the workspace follow from
// (tiles, columns, CTAs) alone, so the sums are the same on every run.
constexpr int kSplitN = 128;  // output columns of a tile product (MMA N)
constexpr int kSplitS = 4;    // stages of one tile each
constexpr int kSplitABytes = 3 * kTileBytes, kSplitBBytes = 3 * kSplitN * 32;
constexpr int kSplitStage = kSplitABytes + kSplitBBytes; // hi, lo, lo2 of both
constexpr int kSplitSmem = 1024 /* barriers, tmem slot */ + kSplitS * kSplitStage + 1024 /* alignment slack */;
constexpr int kSplitThreads = 192; // warps 0-3: epilogue (their tensor-memory lanes); 4: copies; 5: MMAs
constexpr int64_t kSplitMinTiles = 16; // tiles per CTA at least, where there are so many
constexpr int kPartFloats = kPanel * kSplitN;
static_assert(2 * kSplitSmem <= 227 * 1024, "two CTAs per SM: 2 x 256 tensor-memory columns");

struct ShareCut {
    int64_t work, shares, q, r; // the first r shares have q + 1 units, the others q
    __host__ explicit ShareCut(int64_t work_ = 0, int64_t shares_ = 1)
        : work(work_), shares(shares_), q(work_ / shares_), r(work_ % shares_)
    {
    }
    __host__ __device__ __forceinline__ int64_t begin(int64_t g) const { return g * q + (g < r ? g : r); }
    // the share of unit w < work
    __host__ __device__ __forceinline__ int64_t of(int64_t w) const
    {
        const int64_t big = r * (q + 1);
        return w < big ? w / (q + 1) : r + (w - big) / q;
    }
};

// The consecutive pieces of a share: (panel, jt, tiles [t0, t1)), `first`: the
// share starts with it; `whole`: all of the panel's tiles.
struct ShareWalk {
    const int32_t *pf, *tile_panel;
    int64_t kb, tiles, w, end, begin;
    int64_t panel, jt, t0, t1;
    bool first, whole;
    __device__ __forceinline__ ShareWalk(const int32_t *pf_, const int32_t *tile_panel_, int64_t kb_, int64_t tiles_,
                                         const ShareCut &cut, int64_t g)
        : pf(pf_), tile_panel(tile_panel_), kb(kb_), tiles(tiles_), w(cut.begin(g)), end(cut.begin(g + 1)), begin(w)
    {
    }
    // not a share: panel g % panels in strip g / panels, whole (maybe empty)
    __device__ __forceinline__ ShareWalk(const int32_t *pf_, const int32_t *tile_panel_, int64_t kb_, int64_t tiles_,
                                         int64_t panels, int64_t g)
        : pf(pf_), tile_panel(tile_panel_), kb(kb_), tiles(tiles_)
    {
        jt = g / panels;
        panel = g - jt * panels;
        w = begin = jt * tiles + pf[panel * kb];
        end = jt * tiles + pf[(panel + 1) * kb];
    }
    __device__ __forceinline__ bool next()
    {
        if (w >= end)
            return false;
        first = w == begin;
        jt = w / tiles;
        t0 = w - jt * tiles;
        panel = tile_panel[t0];
        const int64_t p0 = pf[panel * kb], p1 = pf[(panel + 1) * kb];
        const int64_t left = end - w;
        t1 = p1 - t0 <= left ? p1 : t0 + left;
        whole = t0 == p0 && t1 == p1;
        w += t1 - t0;
        return true;
    }
};

__global__ void __launch_bounds__(kSplitThreads, 1)
spdm_tc_split_kernel(const int32_t *__restrict__ pf, const int32_t *__restrict__ tile_cb,
                     const int32_t *__restrict__ tile_panel,
                     const uint16_t *__restrict__ a_hi, const uint16_t *__restrict__ a_lo,
                     const uint16_t *__restrict__ b_hi, const uint16_t *__restrict__ b_lo, int64_t m, int64_t n,
                     int64_t kb, int64_t panels, int64_t tiles, const ShareCut cut, bool shares,
                     float *__restrict__ C, float *__restrict__ part, uint32_t *__restrict__ status)
{
    constexpr int N = kSplitN, S = kSplitS;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    // carve: [0,1024) control, then 1024-aligned stages
    unsigned char *base = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(base);
    uint64_t *empty = full + S;
    uint64_t *done = empty + S;   // a piece's MMAs have completed
    uint64_t *drained = done + 1; // its sums have been read out of tensor memory
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drained + 1);
    volatile int *abort_flag = reinterpret_cast<volatile int *>(tmem_slot + 1);
    unsigned char *stages = base + 1024;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < S; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(done, 1);
        mbar_init(drained, 4); // one arrival per epilogue warp
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(2 * N)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    grid_wait_previous(); // barriers and tensor memory are the CTA's own
    grid_launch_next();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    // The leading products (ah * bh) go to bank 0 and the five correction
    // products to bank 1, so each correction is rounded at its own (2^-8
    // smaller) magnitude, not at the running total's; the epilogue adds bank
    // 1 to bank 0.
    ShareWalk sh = shares ? ShareWalk(pf, tile_panel, kb, tiles, cut, blockIdx.x)
                          : ShareWalk(pf, tile_panel, kb, tiles, panels, blockIdx.x);

    // Warps 4 and 5 walk together and one elected lane issues (a lane's own
    // branch costs the descriptors' moves to uniform registers at each MMA)
    if (warp == 4) {
        // copies: the ring runs on over the pieces
        int s = 0;
        uint32_t phase = 1; // the first turn of the ring waits for nothing
        bool ok = true;
        while (ok && sh.next()) {
            for (int64_t tile = sh.t0; tile < sh.t1; ++tile) {
                const int64_t btile = sh.jt * kb + tile_cb[tile];
                ok = mbar_wait(&empty[s], phase) && !*abort_flag;
                ok = __all_sync(0xffffffffu, ok ? 1 : 0);
                if (!ok) {
                    if (lane == 0) {
                        atomicOr(status, kStatusWaitTimeout);
                        *abort_flag = 1;
                    }
                    break;
                }
                unsigned char *st = stages + s * kSplitStage;
                if (elect_one()) {
                    mbar_arrive_expect_tx(&full[s], kSplitStage);
                    bulk_g2s(st, a_hi + tile * (kTileBytes / 2), kTileBytes, &full[s]);
                    bulk_g2s(st + kSplitABytes, b_hi + btile * (N * 16), N * 32, &full[s]);
                    // lo and lo2 of A, then of B: one contiguous copy each
                    bulk_g2s(st + kTileBytes, a_lo + tile * kTileBytes, 2 * kTileBytes, &full[s]);
                    bulk_g2s(st + kSplitABytes + N * 32, b_lo + btile * (N * 32), 2 * N * 32, &full[s]);
                }
                __syncwarp();
                if (++s == S) {
                    s = 0;
                    phase ^= 1;
                }
            }
        }
    } else if (warp == 5) {
        const uint32_t idesc = idesc_bf16(kPanel, N);
        int s = 0;
        uint32_t phase = 0, piece = 0;
        bool ok = true;
        while (ok && sh.next()) {
            // the piece before this one has been read out
            if (piece > 0)
                ok = __all_sync(0xffffffffu, mbar_wait(drained, (piece - 1) & 1) ? 1 : 0);
            tc_fence_after();
            for (int64_t tile = sh.t0; ok && tile < sh.t1; ++tile) {
                ok = __all_sync(0xffffffffu, mbar_wait(&full[s], phase) ? 1 : 0);
                if (!ok)
                    break;
                tc_fence_after();
                const uint32_t acc = tile > sh.t0 ? 1u : 0u;
                const uint64_t ah = smem_desc_sw32(smem_u32(stages + s * kSplitStage));
                if (elect_one()) {
                    const uint64_t bh = ah + (kSplitABytes >> 4);
                    tc_mma(tmem, ah, bh, idesc, acc);
                    // (ah + al + al2)(bh + bl + bl2): every product above 2^-24
                    // of the leading one (al * bl2, al2 * bl, al2 * bl2 dropped),
                    // into the correction bank
                    const uint32_t dx = tmem + static_cast<uint32_t>(N);
                    const uint64_t al = ah + (kTileBytes >> 4), al2 = ah + (2 * kTileBytes >> 4);
                    const uint64_t bl = bh + (N * 32 >> 4), bl2 = bh + (2 * N * 32 >> 4);
                    tc_mma(dx, ah, bl, idesc, acc);
                    tc_mma(dx, al, bh, idesc, 1u);
                    tc_mma(dx, al, bl, idesc, 1u);
                    tc_mma(dx, ah, bl2, idesc, 1u);
                    tc_mma(dx, al2, bh, idesc, 1u);
                    tc_commit(&empty[s]); // slot reusable once these MMAs have read it
                }
                __syncwarp();
                if (++s == S) {
                    s = 0;
                    phase ^= 1;
                }
            }
            if (elect_one())
                tc_commit(done); // arrives when every MMA issued above has completed
            __syncwarp();
            ++piece;
        }
        if (!ok && lane == 0) {
            atomicOr(status, kStatusWaitTimeout);
            *abort_flag = 1;
        }
    } else {
        // epilogue: warp w owns TMEM lanes 32w..32w+31 = panel rows
        uint32_t piece = 0;
        if (!shares && sh.w == sh.end) {
            // panel without entries: its C rows are zero, a warp's stores one row's 128 columns
            const int64_t j = sh.jt * N + lane * 4;
            for (int64_t row = sh.panel * kPanel + warp * 32, end = row + 32; row < end && row < m; ++row)
                if (j < n)
                    *reinterpret_cast<float4 *>(C + row * n + j) = make_float4(0.f, 0.f, 0.f, 0.f);
        }
        while (sh.next()) {
            const bool ok = mbar_wait(done, piece & 1);
            if (!__all_sync(0xffffffffu, ok ? 1 : 0) || *abort_flag) {
                if (lane == 0) {
                    atomicOr(status, kStatusWaitTimeout);
                    *abort_flag = 1;
                }
                break;
            }
            tc_fence_after();
            const int lr = warp * 32 + lane;
            const int64_t row = sh.panel * kPanel + lr;
            float *slot = part + (2 * static_cast<int64_t>(blockIdx.x) + (sh.first ? 0 : 1)) * kPartFloats;
#pragma unroll 1
            for (int c = 0; c < N; c += 32) {
                float v[32], w[32];
                tmem_ld32(tmem + (static_cast<uint32_t>(warp * 32) << 16) + static_cast<uint32_t>(c), v);
                tmem_ld32(tmem + (static_cast<uint32_t>(warp * 32) << 16) + static_cast<uint32_t>(N + c), w);
#pragma unroll
                for (int q = 0; q < 32; ++q)
                    v[q] += w[q];
                const int64_t j = sh.jt * N + c;
                if (!sh.whole) { // [column][row]: contiguous across the warp
#pragma unroll
                    for (int q = 0; q < 32; ++q)
                        slot[(c + q) * kPanel + lr] = v[q];
                } else if (row < m && j < n) {
                    store_row32(C + row * n + j, v, n - j);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0)
                mbar_arrive(drained);
            ++piece;
        }
    }
    __syncwarp(); // warps 4 and 5: their elected lanes are back
    __syncthreads();
    // after a wait gave up, copies already issued may still be landing in
    // this CTA's shared memory: give them a bounded time before it is released
    if (threadIdx.x == 0 && *abort_flag) {
        const uint64_t t_end = global_ns() + kDrainNs;
        while (global_ns() < t_end)
            __nanosleep(10000);
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 5) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * N) : "memory");
    }
}

// C of the (panel of `blockDim.x` rows, strip of `cols` columns) whose tiles
// lie in several shares (their parts added in order) or that have none
// (zeros). One thread per row, 32 of the columns per CTA.
__global__ void __launch_bounds__(2 * kPanel)
tc_fixup_kernel(const int32_t *__restrict__ pf, int64_t m, int64_t n, int64_t kb, int64_t tiles, const ShareCut cut,
                int cols, const float *__restrict__ part, float *__restrict__ C)
{
    grid_wait_previous();
    part = written(part);
    __shared__ __align__(16) float staging[2 * kPanel * kStageRow];
    const int R = blockDim.x;
    const int64_t panel = blockIdx.x, jt = blockIdx.y;
    const int c = blockIdx.z * 32;
    const int64_t j = jt * cols + c;
    if (j >= n)
        return;
    const int64_t p0 = pf[panel * kb], p1 = pf[(panel + 1) * kb];
    const int64_t w0 = jt * tiles + p0, w1 = jt * tiles + p1;
    int64_t g0 = 0, g1 = -1; // the shares with tiles of it
    if (p1 > p0) {
        g0 = cut.of(w0);
        if (cut.begin(g0 + 1) >= w1)
            return; // in one share: written there
        g1 = cut.of(w1 - 1);
    }
    const int64_t part_floats = static_cast<int64_t>(R) * cols;
    float v[32];
#pragma unroll
    for (int q = 0; q < 32; ++q)
        v[q] = 0.0f;
    for (int64_t g = g0; g <= g1; g += 2) { // two parts' loads in flight together
        float x[32], y[32];
        // a share's first piece starts where the share does
        const float *sx = part + (2 * g + (cut.begin(g) >= w0 ? 0 : 1)) * part_floats + c * R + threadIdx.x;
        const float *sy = part + 2 * (g + 1) * part_floats + c * R + threadIdx.x; // the share's first piece
        const bool two = g < g1;
#pragma unroll
        for (int q = 0; q < 32; ++q) {
            x[q] = sx[q * R];
            y[q] = two ? sy[q * R] : 0.0f;
        }
#pragma unroll
        for (int q = 0; q < 32; ++q) {
            v[q] += x[q];
            if (two)
                v[q] += y[q];
        }
    }
    const int warp = threadIdx.x >> 5;
    store_warp32(staging + warp * (32 * kStageRow), v, C, panel * R + warp * 32, j, m, n);
}

// ---- the pair kernel (BF16, FP8-B) ----------------------------------------------------
__device__ __forceinline__ uint32_t cluster_rank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}

// The shared::cluster address of `saddr` (a shared::cta address) in CTA `rank` of the cluster.
__device__ __forceinline__ uint32_t mapa_rank(uint32_t saddr, uint32_t rank)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(saddr), "r"(rank));
    return r;
}

__device__ __forceinline__ void cluster_sync_all()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// Arrives on an mbarrier of either CTA of the pair (a shared::cluster address)
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t addr)
{
    asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(addr) : "memory");
}

__device__ __forceinline__ void fence_cluster() { asm volatile("fence.acq_rel.cluster;" ::: "memory"); }

// One box of a 3-D / 4-D tensor map into this CTA's shared memory, completing
// on an mbarrier in either CTA of the pair.
__device__ __forceinline__ void tma_3d_pair(uint32_t dst, const CUtensorMap *map, int32_t y, int32_t z, uint32_t mbar)
{
    asm volatile("cp.async.bulk.tensor.3d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
                 " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(0), "r"(y), "r"(z), "r"(mbar)
                 : "memory");
}

__device__ __forceinline__ void tma_4d_pair(uint32_t dst, const CUtensorMap *map, int32_t y, int32_t z, int32_t w,
                                            uint32_t mbar)
{
    asm volatile("cp.async.bulk.tensor.4d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes"
                 " [%0], [%1, {%2, %3, %4, %5}], [%6];" ::"r"(dst),
                 "l"(reinterpret_cast<uint64_t>(map)), "r"(0), "r"(y), "r"(z), "r"(w), "r"(mbar)
                 : "memory");
}

__device__ __forceinline__ void tc_mma_pair(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                 "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
                 "l"(a), "l"(b), "r"(idesc), "r"(acc)
                 : "memory");
}

// Arrives on the mbarrier at the same offset in both CTAs once the MMAs issued so far have completed.
__device__ __forceinline__ void tc_commit_pair(uint64_t *bar)
{
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;"
                 ::"r"(smem_u32(bar)), "h"(static_cast<uint16_t>(3))
                 : "memory");
}

constexpr int kPairN = 256;                // output columns per accumulator (MMA N)
constexpr int kPairMaxNT = 2;              // accumulators per CTA: all 512 tensor-memory columns
constexpr int kPairK = 4;                  // tiles per stage
constexpr int kPairHalf = kTileBytes;      // 4 KB: a tile's 128-row half, or a B tile's 128-column half
// A stage holds the A halves of kPairK tiles, then per tile its B half of
// each accumulator: 32 KB or 48 KB, and the ring as many as fit 192 KB (with
// the one CTA per SM that the tensor memory allows).
constexpr int kPairRing = 192 * 1024;
constexpr int kPairMaxS = kPairRing / (2 * kPairK * kPairHalf);
constexpr int kPairStaging = 4 * 32 * kStageRow * 4; // the epilogue warps' staging tiles
constexpr int kPairSmem = 1024 + kPairRing + kPairStaging + 1024;
__host__ __device__ constexpr int pair_stages(int nt) { return kPairRing / ((1 + nt) * kPairK * kPairHalf); }
static_assert(kPairSmem <= 227 * 1024 && 2 * kPairSmem > 228 * 1024,
              "one pair CTA per SM: its tensor-memory allocation never waits for another");

// The MMAs of a stage's nq tiles into NT accumulators (of a strip's last
// column tile past n: the map's zeros). One thread's issue rate bounds the
// kernel, so the tiles are unrolled and a descriptor is one addition.
template <int NT>
__device__ __forceinline__ void pair_stage_mmas(uint32_t tmem, uint32_t st, uint32_t idesc, int nq, uint32_t acc)
{
    const uint64_t da = smem_desc_sw32(st), db = smem_desc_sw32(st + kPairK * kPairHalf);
#pragma unroll
    for (int q = 0; q < kPairK; ++q) {
        if (q >= nq)
            break;
#pragma unroll
        for (int t = 0; t < NT; ++t)
            tc_mma_pair(tmem + static_cast<uint32_t>(t * kPairN), da + static_cast<uint64_t>(q * kPairHalf >> 4),
                        db + static_cast<uint64_t>((q * NT + t) * kPairHalf >> 4), idesc, q > 0 ? 1u : acc);
    }
}

// A cluster of two CTAs per (256-row panel, nt * 256 output columns), or, with
// `shares`, per equal share of the (tile, 256 columns) products (a panel's
// parts go to the workspace, see the split kernel). CTA `rank` holds rows
// [128 rank, 128 rank + 128) of the panel: per stage its halves of up to
// kPairK of the panel's tiles and the matching 128-column halves of the B
// tiles, copied by its warp 4 with tensor-map bulk copies that complete on
// the first CTA's `full` barrier (which expects both CTAs' bytes). Warp 5 of
// the first CTA issues, per tile and accumulator, one
// tcgen05.mma.cta_group::2 (M=256, N=256, K=16) reading both CTAs' shared
// memory, and tcgen05.commit frees the slot in both CTAs. Warps 0-3 of each
// CTA drain its 128 rows of the accumulators from its own tensor memory.
//
// The MMAs bound it (8192^2 of 16 x 16 blocks at 25 %, n = 1024: 68 us at the
// peak rate of 128 SMs, 83 measured, 125 before), as long as one thread can
// issue them: a loop over run-time counts that built each descriptor took
// ~155 cycles per 128-cycle MMA and ~300 per stage, which is why an elected
// lane runs them unrolled, and a copy per tile and operand ~85 ns each, which
// is why one box carries A's stage and a lane each B's tiles. 4 tiles per
// stage and the ring as deep as 192 KB: 8 per stage is 5 % slower at two
// accumulators (and 5 % faster at one). C leaves through a staging tile, four
// rows' 128 bytes per store: 3 us of the 83 less than 16 bytes of 32 rows.
constexpr int kPairThreads = 192;

__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kPairThreads, 1)
spdm_tc_pair_kernel(const __grid_constant__ CUtensorMap tm_a, const __grid_constant__ CUtensorMap tm_b,
                    const int32_t *__restrict__ pf, const int32_t *__restrict__ tile_cb,
                    const int32_t *__restrict__ tile_panel, int64_t m, int64_t n, int64_t kb, int64_t panels,
                    int64_t tiles, const ShareCut cut, bool shares, int nt_cta,
                    float *__restrict__ C, float *__restrict__ part, uint32_t *__restrict__ status)
{
    constexpr int N = kPairN;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    // the same carve in both CTAs: the MMA reads the second CTA's operands at the first's offsets
    unsigned char *base = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(base);
    uint64_t *empty = full + kPairMaxS;
    uint64_t *done = empty + kPairMaxS; // [bank]: a piece's MMAs have completed
    uint64_t *drained = done + 2;       // [bank] (first CTA's): both CTAs have read a piece's sums
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(drained + 2);
    unsigned char *stages = base + 1024;
    float *staging = reinterpret_cast<float *>(stages + kPairRing);

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int64_t pair = blockIdx.x >> 1;
    const int S = pair_stages(nt_cta), stage_bytes = (1 + nt_cta) * kPairK * kPairHalf;
    const int64_t ntn = (n + N - 1) / N;
    bool gave_up = false;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kPairMaxS; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&done[b], 1);
            mbar_init(&drained[b], 8); // one arrival per epilogue warp of the two CTAs
        }
        fence_mbar_init();
    }
    if (warp == 5) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(kPairMaxNT * N)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    grid_wait_previous(); // barriers and tensor memory are the CTA's own
    grid_launch_next();
    tc_fence_before();
    cluster_sync_all(); // both CTAs' barriers initialised and tensor memory allocated
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    ShareWalk sh = shares ? ShareWalk(pf, tile_panel, kb, tiles, cut, pair)
                          : ShareWalk(pf, tile_panel, kb, tiles, panels, pair);
    // with one accumulator a piece's sums are drained while the next piece's
    // products go to the other half of the tensor memory
    const uint32_t bank_mask = nt_cta == 1 ? 1u : 0u;
    // accumulators of a strip of columns
    const auto strip_nt = [&](int64_t jt) { return static_cast<int>(ntn - jt * nt_cta < nt_cta ? ntn - jt * nt_cta : nt_cta); };

    if (warp == 4) {
        // copies (both CTAs); the ring runs on over the pieces. Lane 0 copies
        // the A halves of a stage's tiles (one box), lane q the B halves of
        // tile q (one box for all accumulators), so that no lane waits for
        // another tile's column block.
        int s = 0;
        uint32_t phase = 1; // the first turn of the ring waits for nothing
        while (!gave_up && sh.next()) {
            // read a stage ahead
            int32_t cb = 0, cb_next = lane < kPairK && lane < sh.t1 - sh.t0 ? tile_cb[sh.t0 + lane] : 0;
            for (int64_t q0 = sh.t0; q0 < sh.t1; q0 += kPairK) {
                const int nq = sh.t1 - q0 < kPairK ? static_cast<int>(sh.t1 - q0) : kPairK;
                cb = cb_next;
                if (lane < kPairK && q0 + kPairK + lane < sh.t1)
                    cb_next = tile_cb[q0 + kPairK + lane];
                const bool ok = mbar_wait(&empty[s], phase);
                if (!__all_sync(0xffffffffu, ok ? 1 : 0)) {
                    if (lane == 0)
                        atomicOr(status, kStatusWaitTimeout);
                    gave_up = true;
                    break;
                }
                const uint32_t st = smem_u32(stages + s * stage_bytes);
                const uint32_t leader_full = mapa_rank(smem_u32(&full[s]), 0);
                if (lane == 0) {
                    if (rank == 0) // both CTAs' bytes; boxes count whole, also past the maps' ends
                        mbar_arrive_expect_tx(&full[s], static_cast<uint32_t>(2 * (kPairK + nq * nt_cta) * kPairHalf));
                    tma_3d_pair(st, &tm_a, static_cast<int32_t>(rank * 8), static_cast<int32_t>(q0), leader_full);
                }
                __syncwarp();
                if (lane < nq)
                    tma_4d_pair(st + (kPairK + lane * nt_cta) * kPairHalf, &tm_b, static_cast<int32_t>(rank * 8), cb,
                                static_cast<int32_t>(sh.jt * nt_cta), leader_full);
                if (++s == S) {
                    s = 0;
                    phase ^= 1;
                }
            }
        }
    } else if (warp == 5) {
        if (rank == 0) {
            // MMA issuer (first CTA only): the warp walks together and one
            // elected lane issues a stage's MMAs, unrolled, descriptors
            // advanced by constants
            const uint32_t idesc = idesc_bf16(2 * kPanel, N);
            int s = 0;
            uint32_t phase = 0, piece = 0;
            while (!gave_up && sh.next()) {
                const uint32_t bank = piece & bank_mask, turn = piece >> bank_mask;
                const uint32_t acc0 = tmem + bank * N;
                if (turn > 0) {
                    const bool ok = mbar_wait(&drained[bank], (turn - 1) & 1);
                    if (!__all_sync(0xffffffffu, ok ? 1 : 0))
                        gave_up = true;
                    fence_cluster(); // the other CTA's arrivals
                }
                for (int64_t q0 = sh.t0; !gave_up && q0 < sh.t1; q0 += kPairK) {
                    const bool ok = mbar_wait(&full[s], phase);
                    if (!__all_sync(0xffffffffu, ok ? 1 : 0)) {
                        gave_up = true;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t st = smem_u32(stages + s * stage_bytes);
                    const int nq = sh.t1 - q0 < kPairK ? static_cast<int>(sh.t1 - q0) : kPairK;
                    const uint32_t acc = q0 > sh.t0 ? 1u : 0u;
                    if (elect_one()) {
                        if (nt_cta == 2)
                            pair_stage_mmas<2>(acc0, st, idesc, nq, acc);
                        else
                            pair_stage_mmas<1>(acc0, st, idesc, nq, acc);
                        tc_commit_pair(&empty[s]); // the slot is free in both CTAs once these MMAs have read it
                    }
                    __syncwarp();
                    if (++s == S) {
                        s = 0;
                        phase ^= 1;
                    }
                }
                if (elect_one())
                    tc_commit_pair(&done[bank]); // arrives in both CTAs when every MMA issued above has completed
                __syncwarp();
                ++piece;
            }
            if (gave_up && lane == 0)
                atomicOr(status, kStatusWaitTimeout);
        }
    } else {
        uint32_t piece = 0;
        const int lr = static_cast<int>(rank) * kPanel + warp * 32 + lane;
        if (!shares && sh.w == sh.end) {
            // panel without entries: its C rows are zero
            const int64_t row = sh.panel * (2 * kPanel) + lr;
            if (row < m)
                for (int64_t j = sh.jt * nt_cta * N; j < (sh.jt + 1) * nt_cta * N && j < n; ++j)
                    C[row * n + j] = 0.0f;
        }
        while (sh.next()) {
            const int nt = strip_nt(sh.jt);
            const uint32_t bank = piece & bank_mask, turn = piece >> bank_mask;
            const bool ok = mbar_wait(&done[bank], turn & 1);
            if (!__all_sync(0xffffffffu, ok ? 1 : 0)) {
                if (lane == 0)
                    atomicOr(status, kStatusWaitTimeout);
                gave_up = true;
                break;
            }
            tc_fence_after();
            const int64_t row = sh.panel * (2 * kPanel) + lr;
            float *slot = part + (2 * pair + (sh.first ? 0 : 1)) * static_cast<int64_t>(2 * kPanel) * nt_cta * N;
#pragma unroll 1
            for (int c = 0; c < nt * N; c += 32) {
                float v[32];
                tmem_ld32(tmem + bank * N + (static_cast<uint32_t>(warp * 32) << 16) + static_cast<uint32_t>(c), v);
                const int64_t j = sh.jt * nt_cta * N + c;
                if (!sh.whole) { // [column][row]: contiguous across the warp
                    if (j < n) {
#pragma unroll
                        for (int q = 0; q < 32; ++q)
                            slot[(c + q) * (2 * kPanel) + lr] = v[q];
                    }
                } else {
                    store_warp32(staging + warp * (32 * kStageRow), v, C, row - lane, j, m, n);
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0)
                mbar_arrive_cluster(mapa_rank(smem_u32(&drained[bank]), 0));
            ++piece;
        }
    }
    __syncwarp(); // warps 4 and 5: their elected lanes are back
    // after a wait gave up (in either CTA: the status word), copies already
    // issued may still be landing in this CTA or signalling the first CTA's
    // barriers: give them a bounded time before the pair leaves
    if (lane == 0 && (gave_up || (*reinterpret_cast<volatile uint32_t *>(status) & kStatusWaitTimeout))) {
        const uint64_t t_end = global_ns() + kDrainNs;
        while (global_ns() < t_end)
            __nanosleep(10000);
    }
    __syncwarp();
    tc_fence_before();
    cluster_sync_all(); // neither CTA leaves while the pair's MMAs or copies may touch it
    if (warp == 5) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kPairMaxNT * N)
                     : "memory");
    }
}

// Columns of a B tile: 256 for the pair kernel, 128 for split-BF16, whose
// two accumulator banks stay within half of the 512 tensor-memory columns so
// that two of its CTAs (~98 KB rings) share an SM. (Four banks in all 512
// columns, one CTA per SM with a 12-stage ring, measured 1.8x slower.)
int tile_n_for(bool split) { return split ? 128 : kPairN; }

// cuTensorMapEncodeTiled through the runtime's driver entry-point query (no
// driver library linked).
typedef CUresult (*EncodeTiledFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                   const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_tiled_fn()
{
    static EncodeTiledFn fn = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        cudaDriverEntryPointQueryResult q;
        void *f = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<EncodeTiledFn>(f);
    });
    return fn;
}

// A map of a buffer of tiles. Their bytes are already in the MMA's
// shared-memory layout, so the copies are unswizzled.
bool encode_map(CUtensorMap *map, const void *base, cuuint32_t rank, const cuuint64_t (&dims)[4],
                const cuuint64_t (&strides)[3], const cuuint32_t (&box)[4])
{
    EncodeTiledFn fn = encode_tiled_fn();
    if (!fn)
        return false;
    const cuuint32_t elem[4] = {1, 1, 1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, rank, const_cast<void *>(base), dims, strides, box, elem,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_NONE,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// How a BF16 / FP8-B multiply of `ntn` 256-column tiles is cut over the GPU's
// pairs of SMs. Whole: a pair per (panel, strip of one or two accumulators:
// two, each A half then feeding two MMAs, unless one per pair still leaves
// the grid within one wave). Shares: equal parts of the products with one
// accumulator, one per pair, where their estimate is shorter, in MMA times of
// one tile: a product of a share costs kPairShareRate (its A half feeds one
// MMA), the exposed last drain with the fix-up kPairShareCost, and each share
// that a panel's strip is cut into kPairSharePart (the fix-up adds them one
// after another: 206 x 4980, n = 192, 312 tiles in one panel 41 / 73). The choice
// takes 0.6 % longer than the better one over 768 multiplies of 64 x 400 to 10000
// x 14000 (2.9 % without the parts, up to 1.8 times). Measured, 16 x 16 blocks,
// whole / shares: 8192^2 at 25 %, n = 128 68 / 50 us, n = 512
// 72 / 80, n = 1024 94 / 125; 10240 x 8192 at 25 %, n = 1024 (80 units on 76
// pairs) 172 / 147; 2048 x 8192 at 25 %, n = 256 63 / 35; 1024 x 16384 at 10 %,
// n = 1024 110 / 61; 4096^2, n = 256 38 / 32; 2048^2, n = 1024 28 / 33;
// 12288 x 4096, n = 1024 102 / 105; 4096^2, n = 2048 61 / 84.
struct PairCut {
    int64_t pairs;
    int nt;
    bool shares;
};
constexpr double kPairShareRate = 1.45, kPairShareCost = 80.0, kPairSharePart = 7.0;
constexpr int64_t kPairShareCols = 128; // column tiles at most: beyond, whole units fill the waves

PairCut pair_cut(int64_t panels, int64_t tiles, int64_t ntn)
{
    const int64_t slots = static_cast<int64_t>(device_sms()) / 2;
    const int nt_whole = panels * ntn <= slots ? 1 : kPairMaxNT;
    const int64_t units = panels * ((ntn + nt_whole - 1) / nt_whole);
    const int64_t work = tiles * ntn;
    // in tiles of one accumulator
    const double whole = static_cast<double>((units + slots - 1) / slots) * nt_whole * tiles / (panels > 0 ? panels : 1);
    const double parts = static_cast<double>(slots) / static_cast<double>(panels * ntn > 0 ? panels * ntn : 1);
    const double share = kPairShareRate * static_cast<double>(work) / slots + kPairShareCost + kPairSharePart * parts;
    if (share < whole && work >= slots * kPairK && ntn <= kPairShareCols)
        return PairCut{slots, 1, true};
    return PairCut{units, nt_whole, false};
}

cudaError_t launch_pair(TcPlan &p, int64_t m, int64_t n, float *C, uint32_t *status, cudaStream_t st)
{
    const int64_t ntn = (n + kPairN - 1) / kPairN;
    const PairCut cut = pair_cut(p.panels, p.tiles, ntn);
    // a tile: 16 rows of 512 B, 8 per half. A: (512 B, row, tile), boxes of a
    // half of kPairK tiles; B: (512 B, row, column block, 256-column tile),
    // boxes of a half of one column block in cut.nt column tiles. Boxes past
    // the last tile are filled with zeros there.
    const cuuint64_t tiles = static_cast<cuuint64_t>(p.tiles > 0 ? p.tiles : 1);
    if (tiles > 0x7fffffffULL || p.kb > 0x7fffffffLL)
        return cudaErrorInvalidValue; // int32 coordinates
    CUtensorMap map_a, map_b; // passed by value
    if (!encode_map(&map_a, p.a_hi.ptr, 3, {256, 16, tiles, 1}, {512, 8192, 0}, {256, 8, kPairK, 1}) ||
        !encode_map(&map_b, p.b_hi.ptr, 4, {256, 16, static_cast<cuuint64_t>(p.kb), static_cast<cuuint64_t>(ntn)},
                    {512, 8192, 8192 * static_cast<cuuint64_t>(p.kb)}, {256, 8, 1, static_cast<cuuint32_t>(cut.nt)}))
        return cudaErrorInvalidValue;
    cudaError_t e = cudaFuncSetAttribute(spdm_tc_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kPairSmem);
    if (e != cudaSuccess)
        return e;
    const int64_t strips = (ntn + cut.nt - 1) / cut.nt;
    const ShareCut shares(p.tiles * strips, cut.pairs > 0 ? cut.pairs : 1);
    if (2 * p.panels > 0x7fffffffLL || strips > 65535 || 2 * cut.pairs > 0x7fffffffLL)
        return cudaErrorInvalidConfiguration;
    e = launch_after(
        spdm_tc_pair_kernel, dim3(static_cast<unsigned>(2 * cut.pairs)), dim3(kPairThreads), kPairSmem, st, map_a, map_b, p.pf.ptr, p.tile_cb.ptr, p.tile_panel.ptr, m, n, p.kb, p.panels, p.tiles, shares, cut.shares, cut.nt,
        C, p.part.ptr, status);
    if (e != cudaSuccess)
        return e;
    if (cut.shares) {
        const int cols = cut.nt * kPairN;
        const dim3 grid(static_cast<unsigned>(p.panels), static_cast<unsigned>(strips), static_cast<unsigned>(cols / 32));
        e = launch_after(tc_fixup_kernel, grid, dim3(2 * kPanel), 0, st, p.pf.ptr, m, n, p.kb, p.tiles, shares, cols,
                         p.part.ptr, C);
        if (e != cudaSuccess)
            return e;
        count_launches(1);
    }
    count_launches(1);
    return cudaGetLastError();
}

// CTAs of the split kernel: two per SM, fewer where a share would be short
int64_t split_ctas(int64_t work)
{
    const int64_t most = 2 * static_cast<int64_t>(device_sms());
    const int64_t by_work = work / kSplitMinTiles;
    return by_work < 1 ? 1 : (by_work > most ? most : by_work);
}

// Shares, or (few tiles per panel) a CTA per (panel, strip): a share of several
// panels walks them one after the other, some 4 us of drain each, and the
// fix-up is a launch more. Measured on 960 multiplies (64^2 to 12000^2, blocks
// and unstructured, n 16 to 2048), whole / shares, us: 5384 x 1267 at 0.2 %,
// n = 64 14 / 42; 2322 x 386 at 3 %, n = 96 16 / 28; 1024^2 at 15 % in blocks (48
// tiles a panel), n = 64 32 / 24. At 32 tiles the choice takes 0.6 % longer
// than the better of the two (16 and 48: 1.8 and 1.2 %; shares alone 32 %).
constexpr int64_t kSplitWholeTiles = 32;
bool split_shares(const TcPlan &p) { return p.tiles > kSplitWholeTiles * p.panels; }

cudaError_t launch_split(const TcPlan &p, int64_t m, int64_t n, float *C, uint32_t *status, cudaStream_t st)
{
    const int64_t njt = (n + kSplitN - 1) / kSplitN, work = p.tiles * njt;
    const bool shares = split_shares(p);
    const int64_t ctas = shares ? split_ctas(work) : p.panels * njt;
    const ShareCut cut(work, ctas);
    if (njt > 65535 || p.panels > 0x7fffffffLL || ctas > 0x7fffffffLL)
        return cudaErrorInvalidConfiguration;
    if (work > 0 || !shares) {
        cudaError_t e = cudaFuncSetAttribute(spdm_tc_split_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSplitSmem);
        if (e != cudaSuccess)
            return e;
        e = launch_after(
            spdm_tc_split_kernel, dim3(static_cast<unsigned>(ctas)), dim3(kSplitThreads), kSplitSmem, st, p.pf.ptr, p.tile_cb.ptr, p.tile_panel.ptr, p.a_hi.ptr, p.a_lo.ptr, p.b_hi.ptr, p.b_lo.ptr, m, n, p.kb, p.panels,
            p.tiles, cut, shares, C, p.part.ptr, status);
        if (e != cudaSuccess)
            return e;
        count_launches(1);
    }
    if (!shares)
        return cudaSuccess;
    const dim3 grid(static_cast<unsigned>(p.panels), static_cast<unsigned>(njt), kSplitN / 32);
    count_launches(1);
    return launch_after(tc_fixup_kernel, grid, dim3(kPanel), 0, st, p.pf.ptr, m, n, p.kb, p.tiles, cut, kSplitN,
                        p.part.ptr, C);
}

} // namespace

// Builds the densified tile plan (one synchronisation to size the tiles).
gcoo_status tc_build_plan(gcoo_handle *h, bool split, cudaStream_t st)
{
    if (h->tc && h->tc->split == split && h->tc->nnz == h->nnz)
        return GCOO_SUCCESS; // the same entries: built for this form already
    destroy_tc_plan(h->tc);
    h->tc = new (std::nothrow) TcPlan();
    if (!h->tc)
        return fail(GCOO_ERROR_ALLOC, "host allocation failed");
    TcPlan &p = *h->tc;
    p.split = split;
    p.nnz = h->nnz;
    p.panel_rows = split ? kPanel : 2 * kPanel;
    p.panels = (h->m + p.panel_rows - 1) / p.panel_rows;
    p.kb = (h->k + kTileK - 1) / kTileK;
    const int64_t L = p.panels * p.kb;
    const size_t sc = scan_scratch_elems(L);
    if (!p.pf.ensure(L + 1) || !p.scratch.ensure(sc + 1))
        return fail(GCOO_ERROR_ALLOC, "device allocation of the tile plan failed");
    GCOO_CUDA(cudaMemsetAsync(p.pf.ptr, 0, sizeof(int32_t) * (L + 1), st));
    unsigned blocks = static_cast<unsigned>(std::min<int64_t>((h->m + 7) / 8, 152 * 16));
    tile_flags_kernel<<<blocks, 256, 0, st>>>(h->packed.ptr, h->row_ptr.ptr, h->m, p.kb, p.panel_rows, p.pf.ptr);
    count_launches(1);
    GCOO_LAUNCH("tile_flags_kernel");
    GCOO_CUDA(launch_row_scan(p.pf.ptr, L, 1, nullptr, nullptr, p.scratch.ptr + sc, p.scratch.ptr, nullptr, st));
    int64_t total = 0;
    GCOO_CUDA(cudaMemcpyAsync(&total, p.scratch.ptr + sc, sizeof(total), cudaMemcpyDeviceToHost, st));
    GCOO_CUDA(cudaStreamSynchronize(st));
    p.tiles = total;
    const size_t tile_elems = static_cast<size_t>(p.panel_rows / kPanel) * (kTileBytes / 2);
    if (!p.tile_cb.ensure(total + 1) || !p.tile_panel.ensure(total + 1) || !p.a_hi.ensure(total * tile_elems + 1) ||
        (split && !p.a_lo.ensure(2 * total * tile_elems + 1)))
        return fail(GCOO_ERROR_ALLOC, "device allocation of the dense tiles failed");
    if (total > 0) {
        tile_list_kernel<<<static_cast<unsigned>(std::min<int64_t>((L + 255) / 256, 4096)), 256, 0, st>>>(
            p.pf.ptr, L, p.kb, p.tile_cb.ptr, p.tile_panel.ptr);
        GCOO_CUDA(cudaMemsetAsync(p.a_hi.ptr, 0, total * tile_elems * 2, st));
        if (split)
            GCOO_CUDA(cudaMemsetAsync(p.a_lo.ptr, 0, 2 * total * kTileBytes, st));
        tile_fill_kernel<<<blocks, 256, 0, st>>>(h->packed.ptr, h->row_ptr.ptr, h->m, p.kb, p.panel_rows, p.pf.ptr,
                                                 reinterpret_cast<__nv_bfloat16 *>(p.a_hi.ptr),
                                                 split ? reinterpret_cast<__nv_bfloat16 *>(p.a_lo.ptr) : nullptr);
        count_launches(2);
        GCOO_LAUNCH("tile plan kernels");
    }
    return GCOO_SUCCESS;
}

// Density of the stored tiles (entries / tile slots); 0 before a plan exists.
double tc_density(const gcoo_handle *h)
{
    if (!h->tc || h->tc->tiles == 0)
        return 0.0;
    return static_cast<double>(h->nnz) / (static_cast<double>(h->tc->tiles) * h->tc->panel_rows * kTileK);
}

gcoo_status tc_prepare_b(gcoo_handle *h, int64_t n, bool fp8)
{
    TcPlan &p = *h->tc;
    const int N = tile_n_for(p.split);
    const int64_t nt = (n + N - 1) / N;
    const size_t elems = static_cast<size_t>(nt) * p.kb * N * kTileK;
    // the parts of the shares, whatever the width: two per CTA (split) or pair
    size_t parts = 0;
    if (p.split)
        parts = split_shares(p) ? 4 * static_cast<size_t>(device_sms()) * kPartFloats : 0;
    else
        for (int64_t t = 1; t <= std::min<int64_t>(nt, kPairShareCols) && parts == 0; ++t)
            if (pair_cut(p.panels, p.tiles, t).shares)
                parts = static_cast<size_t>(device_sms()) * (2 * kPanel * kPairN);
    if (!p.b_hi.ensure(elems) || (p.split && !p.b_lo.ensure(2 * elems)) || (parts > 0 && !p.part.ensure(parts)) ||
        (fp8 && (!p.b_scale.ensure(static_cast<size_t>(n)) || !p.b_amax.ensure(static_cast<size_t>(n)))))
        return fail(GCOO_ERROR_ALLOC, "device allocation of the B tiles failed");
    p.b_n = n;
    return GCOO_SUCCESS;
}

gcoo_status tc_spdm(gcoo_handle *h, const float *dB, int64_t n, float *dC, bool fp8, cudaStream_t st)
{
    TcPlan &p = *h->tc;
    const int N = tile_n_for(p.split);
    if (fp8)
        GCOO_CUDA(launch_fp8_scales(dB, h->k, n, p.b_amax.ptr, p.b_scale.ptr, st));
    const int per_cta = p.split ? 2 : 1;
    dim3 g(static_cast<unsigned>((p.kb + per_cta - 1) / per_cta), static_cast<unsigned>((n + N - 1) / N));
    __nv_bfloat16 *hi = reinterpret_cast<__nv_bfloat16 *>(p.b_hi.ptr), *lo = reinterpret_cast<__nv_bfloat16 *>(p.b_lo.ptr);
    if (p.split)
        b_tiles_kernel<true, false><<<g, 256, 0, st>>>(dB, h->k, n, p.kb, hi, lo, nullptr);
    else if (fp8)
        b_tiles_kernel<false, true><<<g, 256, 0, st>>>(dB, h->k, n, p.kb, hi, nullptr, p.b_scale.ptr);
    else
        b_tiles_kernel<false, false><<<g, 256, 0, st>>>(dB, h->k, n, p.kb, hi, nullptr, nullptr);
    count_launches(1);
    GCOO_LAUNCH("b_tiles_kernel");
    if (p.split) {
        const cudaError_t e = launch_split(p, h->m, n, dC, h->status.ptr, st);
        if (e != cudaSuccess)
            return cuda_fail(e, "spdm_tc_split_kernel launch");
        return GCOO_SUCCESS;
    }
    const cudaError_t e = launch_pair(p, h->m, n, dC, h->status.ptr, st);
    if (e != cudaSuccess)
        return cuda_fail(e, "spdm_tc_pair_kernel launch (or its tensor maps)");
    return GCOO_SUCCESS;
}

} // namespace gcoo
