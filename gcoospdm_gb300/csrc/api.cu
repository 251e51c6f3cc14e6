// api.cu -- the C ABI (include/gcoo.h): validation, handle lifecycle, the
// conversion orchestration and dispatch to the kernels. Every entry point
// returns a status; CUDA errors are captured after each launch.
#include <math.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <mutex>
#include <string>

#include <nvtx3/nvToolsExt.h>

#include "handle.hpp"

namespace gcoo {

NvtxRange::NvtxRange(const char *name) { nvtxRangePushA(name); }
NvtxRange::~NvtxRange() { nvtxRangePop(); }

// ---- errors --------------------------------------------------------------------
static thread_local std::string t_last_error;

void set_error(const std::string &msg) { t_last_error = msg; }

gcoo_status fail(gcoo_status s, const std::string &msg)
{
    t_last_error = std::string(gcoo_status_string(s)) + ": " + msg;
    return s;
}

gcoo_status cuda_fail(cudaError_t e, const char *what)
{
    t_last_error = std::string("CUDA error in ") + what + ": " + cudaGetErrorName(e) + " (" +
                   cudaGetErrorString(e) + ")";
    return e == cudaErrorMemoryAllocation ? GCOO_ERROR_ALLOC : GCOO_ERROR_CUDA;
}

// ---- launch counter ------------------------------------------------------------------
static std::atomic<uint64_t> g_launches{0};
void count_launches(int n) { g_launches.fetch_add(static_cast<uint64_t>(n), std::memory_order_relaxed); }

// ---- allocator ---------------------------------------------------------------------
static gcoo_alloc_fn g_alloc = nullptr;
static gcoo_free_fn g_free = nullptr;
static void *g_alloc_ctx = nullptr;

void *dev_alloc(size_t bytes)
{
    if (g_alloc)
        return g_alloc(bytes, g_alloc_ctx);
    void *p = nullptr;
    if (cudaMalloc(&p, bytes) != cudaSuccess) {
        cudaGetLastError(); // clear the sticky-free error state of this call
        return nullptr;
    }
    return p;
}

void dev_free(void *p)
{
    if (!p)
        return;
    if (g_free)
        g_free(p, g_alloc_ctx);
    else
        cudaFree(p);
}

// coo.cu
gcoo_status coo_build(gcoo_handle *h, cudaStream_t st);
// left.cu
gcoo_status left_prepare(gcoo_handle *h, LeftPlan *&plan, int64_t p, cudaStream_t st);
gcoo_status left_spdm(gcoo_handle *h, const LeftPlan &L, const float *dD, int64_t p, float *dC, cudaStream_t st);

// Implemented in forms.cu / autotune.cpp.
gcoo_status run_form(gcoo_handle *h, const float *dB, int64_t n, float *dC, gcoo_precision prec,
                     cudaStream_t st, bool prepare_only);
bool form_uses_tensor(gcoo_handle *h, gcoo_precision prec);
bool tuned_params(int64_t m, int64_t k, int64_t nnz, int64_t n, gcoo_params *out);

static bool valid_cpg(int32_t c) { return c == 1 || c == 2 || c == 4 || c == 8 || c == 16 || c == 32; }

static gcoo_status check_dims(int64_t m, int64_t k)
{
    if (m <= 0 || k <= 0)
        return fail(GCOO_ERROR_INVALID_VALUE, "m and k must be positive");
    if (m >= (int64_t(1) << 31) || k >= (int64_t(1) << 31))
        return fail(GCOO_ERROR_INVALID_VALUE, "m and k must fit int32 indices");
    return GCOO_SUCCESS;
}

static gcoo_status check_n(int64_t n)
{
    if (n <= 0 || n >= (int64_t(1) << 31))
        return fail(GCOO_ERROR_INVALID_VALUE, "n must be in [1, 2^31)");
    return GCOO_SUCCESS;
}

// Whether the groups share enough columns for the FP32 multiply to consider
// the group and panel walks (shared_walk): forced by fp32_order, else when the
// conversion saw at least 1.5 entries per distinct (group, column) pair.
bool group_order_chosen(const gcoo_handle *h)
{
    if (h->coo || !group_order_ok(h->p.rows_per_group) || h->p.fp32_order == 1)
        return false;
    if (h->p.fp32_order == 2)
        return true;
    return h->distinct_cols > 0 && 2 * h->nnz >= 3 * h->distinct_cols;
}

// The split summation's partial sums for B of n columns (grown, never
// shrunk: allocated by the first multiply of a width, or by gcoo_prepare).
gcoo_status ensure_split_work(gcoo_handle *h, int64_t n)
{
    if (h->pieces_bound <= 0)
        return GCOO_SUCCESS;
    if (!h->split_part.ensure(static_cast<size_t>(h->pieces_bound) * static_cast<size_t>(n)))
        return fail(GCOO_ERROR_ALLOC, "device allocation of the long rows' partial sums failed");
    return GCOO_SUCCESS;
}

// Walk of a matrix whose groups share columns. The row walk reads a B row once
// per entry, the group walk once per column of a group (four rows), the panel
// walk once per column of sixteen rows, but their lanes also wait for the
// staging and the masks, and they have fewer CTAs. Measured on 4783 multiplies
// (64^2 to 10000^2, blocks of 2 to 64 rows, aligned or not, with holes,
// unstructured from 25 %, n 1 to 2048; rows / groups / panels, us):
//   4096^2, 16 x 16 blocks, 25 %: n 128 215 / 380 / 147, n 256 331 / 397 / 106, n 1024 1030 / 561 / 230
//           16 x 16 blocks,  5 %: n 128  42 /  93 /  57, n 256  60 /  97 /  46, n 1024  158 / 137 /  74
//           the same, 40 % holes: n 256  48 / 186 /  70, n 512  77 / 197 /  93, n 1024  140 / 229 / 133
//           4 x 4 blocks, 10 %:   n 128  59 / 154,       n 256 103 / 162,       n 1024  333 / 235
//           unstructured 30 %:    n 128 244 /1178 / 345, n 512 504 /1347 / 637, n 1024 1066 /1550 / 928
//           2 x 2 blocks, 10 %:   n 256  85 / 357 / 206, n 512 137 / 386 / 376, n 1024  267 / 451 / 542
//   8192^2, 2 x 2 blocks, 25 %:   n 256 1557 /2425 / 927, n 1024 5791 /3156 /2856
//   2048^2, 16 x 16, 40 % holes:  n 256  34 / 141 /  60, n 1024 78 / 154 / 84, n 2048 140 / 228 / 120
// Panels win with many rows per panel column (share) and much work, so that
// their CTAs fill the GPU: share^3 * nnz * n >= 5e10 * (5 + windows), a window
// of 512 columns taking some 4 us to stage whatever it holds (16 x 16 blocks at
// 1.7 %, rows / panels: 2747 x 7474, n = 272 30 / 61; 1758 x 9967, n = 280 34 / 71).
// Less counts of the work where the last strip of 128 columns is not full and
// where lanes copy B in 4-byte pieces, and rows of 1600 entries need twice as
// much (1139 x 5876, 3379 a row in 16 x 16 blocks with holes, n = 190 227 / 458).
// Groups win for blocks of four rows, wide and large. By this rule 5275
// multiplies (wide matrices and long rows among them) take 1.1 % longer than by
// the best walk of each (1 in 100 more than 1.27 times as long), by the row walk
// alone 5 % and up to 4 times; by the group walk alone twice.
enum SharedWalk { kWalkRows, kWalkGroups, kWalkPanels };

static SharedWalk shared_walk(const gcoo_handle *h, int64_t n, uintptr_t b, uintptr_t c)
{
    if (h->p.vec != 0)
        return kWalkGroups; // columns per lane chosen by the caller
    const double share = h->panel_share; // 0: no panels
    const double sharing4 = static_cast<double>(h->nnz) / static_cast<double>(h->distinct_cols);
    if (h->p.fp32_order == 2)
        return panel_ok(n) && share >= 1.75 * sharing4 ? kWalkPanels : kWalkGroups;
    const double work = static_cast<double>(h->nnz) * static_cast<double>(n);
    const bool vec4 = n % 4 == 0 && !((b | c) & 15);
    // a skewed matrix (its long rows have kernels of their own in the row walk):
    // panels once the work outweighs the one panel that walks the longest row's
    // columns (4308 x 667 in 16 x 16 blocks at 2 %, one full row, n = 1700: rows 36,
    // groups 111, panels 66 us)
    if (h->n_long > 0 && work < 5e5 * static_cast<double>(h->max_row_nnz))
        return kWalkRows;
    const double strips = static_cast<double>((n + 127) / 128 * 128), windows = static_cast<double>((h->k + 511) / 512);
    const double counts = work * (static_cast<double>(n) / strips) * (vec4 ? 1.0 : 0.6);
    const double enough = 5e10 * (5.0 + windows) * (h->nnz >= 1600 * h->m ? 2.0 : 1.0);
    if (panel_ok(n) && n >= 96 && share >= 4.0 && share * share * share * counts >= enough)
        return kWalkPanels;
    // a CTA per group and 1024 columns: with few of them the row walk (263 x 2693 at
    // 49 %, n = 940 107 / 420)
    const bool many = h->m * ((n + 1023) / 1024) >= 2000;
    return vec4 && n >= 640 && sharing4 >= 3.3 && work >= 3e8 && many && h->n_long == 0 ? kWalkGroups : kWalkRows;
}

static SharedWalk fp32_walk(const gcoo_handle *h, int64_t n, const float *dB, const float *dC)
{
    return group_order_chosen(h)
               ? shared_walk(h, n, reinterpret_cast<uintptr_t>(dB), reinterpret_cast<uintptr_t>(dC))
               : kWalkRows;
}

// Whether a skewed matrix's long and short rows get kernels of their own. B
// and C aligned for 16-byte accesses: yes, but where nearly all entries are in
// long rows and the work outweighs the longest one (8192^2, 410 entries a row
// and one full row, n = 1024: 1275 us, the row walk 716; 13622 x 5573, 286 a row,
// n = 976 1554 / 872). At other alignments a lane of those kernels has one column
// (two for even widths) where the row walk has four: only while the longest
// row's chain is the time of the row walk and not the work, sooner if more than
// half of the entries are in long rows. Measured on 869 multiplies of such
// widths, own kernels / row walk, us: 40000 Zipf rows of up to 4096 entries (38 %
// of all in long rows), n = 201 155 / 218; 65536, n = 255 340 / 376; 8609 x 2229
// with 1.7 M entries, n = 1767 1764 / 760; 6135 x 6475, 3.7 M, n = 1207 4426 /
// 1381; 6850^2, 504 a row, n = 33 411 / 232. The lines below take 3 % longer than
// the better one (always own kernels 7 %, up to 3.8 times; always the row walk
// 2 times on average).
static bool long_rows_pay(const gcoo_handle *h, int64_t n, const float *dB, const float *dC)
{
    const uintptr_t at = reinterpret_cast<uintptr_t>(dB) | reinterpret_cast<uintptr_t>(dC);
    const bool quads = n % 4 == 0 && !(at & 15), pairs = n % 2 == 0 && !(at & 7);
    if (quads && h->p.fp32_sum == GCOO_SUM_SPLIT)
        return true; // sums in pieces stay where they are asked for
    const int64_t tile = quads ? 128 : (pairs ? 64 : 32);
    const double cols = static_cast<double>(quads ? n : (n + tile - 1) / tile * tile); // walked
    const double work = static_cast<double>(h->nnz) * cols / static_cast<double>(h->max_row_nnz);
    if (quads)
        return work <= 2e5 || 20 * h->long_entries <= 17 * h->nnz;
    return work <= (pairs ? 1.5e5 : (2 * h->long_entries <= h->nnz ? 8e4 : 3e4));
}

gcoo_status spdm_fp32(gcoo_handle *h, const float *dB, int64_t n, float *dC, cudaStream_t st,
                      const gcoo_params *override_params)
{
    const SharedWalk walk = override_params ? kWalkRows : fp32_walk(h, n, dB, dC);
    if (walk == kWalkPanels) {
        const cudaError_t e = launch_spdm_fp32_panel(h->packed.ptr, h->row_ptr.ptr, h->tile_cnt.ptr, h->m, h->k, dB, n,
                                                     dC, st);
        if (e != cudaSuccess)
            return cuda_fail(e, "spdm_panel_kernel launch");
        return GCOO_SUCCESS;
    }
    if (walk == kWalkGroups) {
        // 8 columns per lane (two 16-byte loads: more FMAs per shuffled entry) where n allows
        int v = n % 8 == 0 ? 8 : 4;
        const uintptr_t b = reinterpret_cast<uintptr_t>(dB), c = reinterpret_cast<uintptr_t>(dC);
        if (n % 4 != 0 || (b & 15) || (c & 15))
            v = (n % 2 != 0 || (b & 7) || (c & 7)) ? 1 : 2;
        if (h->p.vec > 0 && h->p.vec < v)
            v = h->p.vec;
        cudaError_t e = launch_spdm_fp32_group(h->vals.ptr, h->rc.ptr, h->rc.ptr + h->nnz, h->group_index(), h->m,
                                               h->ng, dB, n, dC, v, st);
        if (e != cudaSuccess)
            return cuda_fail(e, "spdm_fp32_group_kernel launch");
        return GCOO_SUCCESS;
    }
    gcoo_params p = h->p;
    if (override_params) {
        p = *override_params;
        p.rows_per_group = h->p.rows_per_group;
    } else {
        gcoo_params t;
        if (tuned_params(h->m, h->k, h->nnz, n, &t)) {
            p.vec = t.vec;
            p.warps = t.warps;
            p.col_warps = t.col_warps;
            p.depth = t.depth;
        }
    }
    // a skewed matrix (explicit launch-shape overrides aside): its long rows go
    // to their own kernel, the short rest to a kernel without staging
    if (!override_params && h->n_long > 0 && h->side && h->ev_fork && h->ev_join && long_rows_ok(h->m, n) &&
        long_rows_pay(h, n, dB, dC)) {
        // the pieces' kernel copies 16 bytes at a time; other widths keep the chain
        const bool split = h->p.fp32_sum == GCOO_SUM_SPLIT && h->pieces_bound > 0 && n % 4 == 0 &&
                           (reinterpret_cast<uintptr_t>(dB) & 15) == 0;
        if (split) {
            gcoo_status ws = ensure_split_work(h, n);
            if (ws != GCOO_SUCCESS)
                return ws;
        }
        // The two kernels write disjoint rows of C: the short rows run on the
        // side stream, forked from and joined back into the caller's stream.
        // The long rows are on the caller's so that they start first: their
        // first wave spreads over idle SMs and the short rows, whose stream has
        // the priority from then on, fill what is left.
        GCOO_CUDA(cudaEventRecord(h->ev_fork, st));
        GCOO_CUDA(cudaStreamWaitEvent(h->side, h->ev_fork, 0));
        const cudaError_t el =
            split ? launch_spdm_split(h->packed.ptr, h->row_ptr.ptr, h->long_rows.ptr, h->n_long, h->piece_first.ptr,
                                      h->piece_row.ptr, h->piece_total.ptr, h->pieces_bound, dB, n,
                                      h->split_part.ptr, dC, st)
                  : launch_spdm_long(h->packed.ptr, h->row_ptr.ptr, h->long_rows.ptr, h->n_long, dB, n, dC, st);
        const cudaError_t es = el == cudaSuccess
                                   ? launch_spdm_short(h->packed.ptr, h->row_ptr.ptr, h->m, h->k, dB, n, dC,
                                                       long_row_min(), split ? 0 : h->max_row_nnz, h->side)
                                   : cudaSuccess;
        // joined whatever happened: nothing of this call runs past it on the side stream
        GCOO_CUDA(cudaEventRecord(h->ev_join, h->side));
        GCOO_CUDA(cudaStreamWaitEvent(st, h->ev_join, 0));
        if (el != cudaSuccess)
            return cuda_fail(el, split ? "spdm_piece_kernel launch" : "spdm_long_kernel launch");
        if (es != cudaSuccess)
            return cuda_fail(es, "spdm_short_kernel launch");
        return GCOO_SUCCESS;
    }
    const LaunchShape s = pick_shape(p, h->m, n, h->nnz, h->max_row_nnz, reinterpret_cast<uintptr_t>(dB),
                                     reinterpret_cast<uintptr_t>(dC));
    cudaError_t e = launch_spdm_fp32(h->packed.ptr, h->row_ptr.ptr, h->m, dB, n, dC, s, h->status.ptr, st);
    if (e != cudaSuccess)
        return cuda_fail(e, "spdm_fp32_kernel launch");
    return GCOO_SUCCESS;
}

} // namespace gcoo

using namespace gcoo;

extern "C" {

int gcoo_abi_version(void) { return GCOO_ABI_VERSION; }

uint64_t gcoo_kernel_launches(void) { return g_launches.load(std::memory_order_relaxed); }

const char *gcoo_status_string(gcoo_status s)
{
    switch (s) {
    case GCOO_SUCCESS: return "GCOO_SUCCESS";
    case GCOO_ERROR_INVALID_VALUE: return "GCOO_ERROR_INVALID_VALUE";
    case GCOO_ERROR_ALLOC: return "GCOO_ERROR_ALLOC";
    case GCOO_ERROR_CUDA: return "GCOO_ERROR_CUDA";
    case GCOO_ERROR_NOT_BUILT: return "GCOO_ERROR_NOT_BUILT";
    case GCOO_ERROR_UNSUPPORTED: return "GCOO_ERROR_UNSUPPORTED";
    case GCOO_ERROR_FORMAT: return "GCOO_ERROR_FORMAT";
    case GCOO_ERROR_TIMEOUT: return "GCOO_ERROR_TIMEOUT";
    case GCOO_ERROR_CAPACITY: return "GCOO_ERROR_CAPACITY";
    }
    return "GCOO_ERROR_UNKNOWN";
}

const char *gcoo_last_error(void) { return t_last_error.c_str(); }

gcoo_status gcoo_params_default(gcoo_params *p)
{
    if (!p)
        return fail(GCOO_ERROR_INVALID_VALUE, "params is NULL");
    memset(p, 0, sizeof(*p));
    p->rows_per_group = 4; // src/constants.h:4 COLUMN_PER_GROUP
    p->engine = GCOO_ENGINE_AUTO;
    return GCOO_SUCCESS;
}

gcoo_status gcoo_set_allocator(gcoo_alloc_fn alloc, gcoo_free_fn release, void *ctx)
{
    if ((alloc == nullptr) != (release == nullptr))
        return fail(GCOO_ERROR_INVALID_VALUE, "allocator and free function must be given together");
    g_alloc = alloc;
    g_free = release;
    g_alloc_ctx = ctx;
    return GCOO_SUCCESS;
}

gcoo_status gcoo_create(gcoo_handle **out, const float *dA, int64_t m, int64_t k, const gcoo_params *params)
{
    if (!out)
        return fail(GCOO_ERROR_INVALID_VALUE, "out is NULL");
    *out = nullptr;
    if (!dA)
        return fail(GCOO_ERROR_INVALID_VALUE, "dense matrix pointer is NULL");
    gcoo_status s = check_dims(m, k);
    if (s != GCOO_SUCCESS)
        return s;
    gcoo_params p;
    gcoo_params_default(&p);
    if (params)
        p = *params;
    if (!valid_cpg(p.rows_per_group))
        return fail(GCOO_ERROR_INVALID_VALUE, "rows_per_group must be a power of two in [1, 32]");
    if (p.vec != 0 && p.vec != 1 && p.vec != 2 && p.vec != 4)
        return fail(GCOO_ERROR_INVALID_VALUE, "vec must be 0, 1, 2 or 4");
    if (p.warps < 0 || p.warps > 32 || p.col_warps < 0 || p.col_warps > 32)
        return fail(GCOO_ERROR_INVALID_VALUE, "warps / col_warps out of range");
    if (p.engine < GCOO_ENGINE_AUTO || p.engine > GCOO_ENGINE_TENSOR)
        return fail(GCOO_ERROR_INVALID_VALUE, "unknown engine");
    if (p.depth < 0 || p.depth > 2)
        return fail(GCOO_ERROR_INVALID_VALUE, "depth must be 0, 1 or 2");
    if (p.fp32_order < 0 || p.fp32_order > 2)
        return fail(GCOO_ERROR_INVALID_VALUE, "fp32_order must be 0, 1 or 2");
    if (p.fp32_order == 2 && !group_order_ok(p.rows_per_group))
        return fail(GCOO_ERROR_UNSUPPORTED, "the group-order FP32 multiply needs rows_per_group 4");
    if (p.fp32_sum != GCOO_SUM_CHAIN && p.fp32_sum != GCOO_SUM_SPLIT)
        return fail(GCOO_ERROR_INVALID_VALUE, "fp32_sum must be GCOO_SUM_CHAIN (0) or GCOO_SUM_SPLIT (1)");
    gcoo_handle *h = new (std::nothrow) gcoo_handle();
    if (!h)
        return fail(GCOO_ERROR_ALLOC, "host allocation of the handle failed");
    h->dA = dA;
    h->m = m;
    h->k = k;
    h->p = p;
    h->ng = (m + p.rows_per_group - 1) / p.rows_per_group;
    *out = h;
    return GCOO_SUCCESS;
}

namespace {

constexpr size_t kReadbackWords = 8; // of a handle's page-locked readback
constexpr int64_t kSampleEntries = 34500; // 16^3 * entries * 2048 columns < 3e11 (shared_walk)

// How many rows of a panel (16 rows) share a column, for shared_walk; 0 where
// the panels cannot run or never pay. A sample of panels tells: share, when
// the build has read one back with its totals (a steady loop's on such a
// matrix), else one more readback. A panel's staging costs about the same
// whatever its window holds: at 2 % density (16 x 16 blocks, 4096^2) panels
// take 36 against the group walk's 53 us at n = 256 and 54 against 60 at n =
// 1024, so below 1/64 they are left out; and matrices so small that only B
// wider than 2048 columns would take them are not sampled, which is a tenth of
// a small matrix's rebuild (255 x 794 at 36 % 37 us with it, 32 without).
gcoo_status choose_panels(gcoo_handle *h, cudaStream_t st, const int64_t *share)
{
    h->panel_share = 0.0;
    h->sampled = false;
    if (!h->seg_prefix || !group_order_chosen(h) || h->nnz < kSampleEntries ||
        64.0 * static_cast<double>(h->nnz) < static_cast<double>(h->m) * h->k)
        return GCOO_SUCCESS;
    h->sampled = true;
    int64_t own[2] = {0, 0};
    if (!share) {
        // the build's words [6] and [7], zero as it left them
        unsigned long long *words = reinterpret_cast<unsigned long long *>(h->status.ptr + 2) + 6;
        GCOO_CUDA(launch_panel_share(h->packed.ptr, h->row_ptr.ptr, h->m, h->k, words, nullptr, nullptr, st));
        GCOO_CUDA(cudaMemcpyAsync(own, words, sizeof(own), cudaMemcpyDeviceToHost, st));
        GCOO_CUDA(cudaStreamSynchronize(st));
        share = own;
    }
    if (share[1] > 0)
        h->panel_share = static_cast<double>(share[0]) / static_cast<double>(share[1]);
    return GCOO_SUCCESS;
}

// The end of every successful build: plans derived from the old arrays go,
// and for a skewed matrix the list of its long rows (multiplied by their own
// kernel) is collected, one readback of its length. share: see choose_panels.
gcoo_status finish_build(gcoo_handle *h, cudaStream_t st, const int64_t *share = nullptr)
{
    if (h->tc)
        destroy_tc_plan(h->tc);
    h->tc = nullptr;
    destroy_left_plan(h->left);
    h->left = nullptr;
    const gcoo_status ps = choose_panels(h, st, share);
    if (ps != GCOO_SUCCESS)
        return ps;
    h->n_long = 0;
    h->long_entries = 0;
    h->pieces_bound = 0;
    if (row_lengths_skewed(h->m, h->nnz, h->max_row_nnz) && h->packed.count >= static_cast<size_t>(h->nnz) + 2) {
        const int64_t cap = h->nnz / long_row_min() + 1;
        if (!h->long_rows.ensure(2 * static_cast<size_t>(cap)) || !h->long_count.ensure(2))
            return fail(GCOO_ERROR_ALLOC, "device allocation of the long-row list failed");
        unsigned long long *d_cnt = h->long_count.ptr;
        GCOO_CUDA(cudaMemsetAsync(d_cnt, 0, 2 * sizeof(*d_cnt), st));
        GCOO_CUDA(launch_collect_long(h->row_ptr.ptr, h->m, h->long_rows.ptr, cap, d_cnt, st));
        const bool split = h->p.fp32_sum == GCOO_SUM_SPLIT;
        if (split) {
            // the piece plan, before the readback (its tables bounded without it)
            const int64_t pcap = split_piece_bound(cap, h->nnz);
            if (!h->piece_first.ensure(static_cast<size_t>(cap)) || !h->piece_row.ensure(static_cast<size_t>(pcap)) ||
                !h->piece_total.ensure(1))
                return fail(GCOO_ERROR_ALLOC, "device allocation of the long rows' piece plan failed");
            GCOO_CUDA(launch_split_plan(h->row_ptr.ptr, h->long_rows.ptr, d_cnt, cap, h->piece_first.ptr,
                                        h->piece_row.ptr, pcap, h->piece_total.ptr, st));
        }
        if (!h->readback && cudaMallocHost(&h->readback, kReadbackWords * sizeof(int64_t)) != cudaSuccess) {
            h->readback = nullptr;
            return fail(GCOO_ERROR_ALLOC, "page-locked allocation of the readback words failed");
        }
        GCOO_CUDA(cudaMemcpyAsync(h->readback, d_cnt, 2 * sizeof(int64_t), cudaMemcpyDeviceToHost, st));
        GCOO_CUDA(cudaStreamSynchronize(st));
        h->n_long = std::min<int64_t>(h->readback[0], cap);
        h->long_entries = h->readback[1];
        h->pieces_bound = split ? split_piece_bound(h->n_long, h->long_entries) : 0;
        if (h->n_long > 0) {
            // The short rows' stream, at the highest priority: long rows past the
            // first wave, the shorter ones, go behind the short rows, which are
            // the larger part of the gathers. Zipf rows, this against equal
            // priorities (and against the long rows first, at the highest): 65536
            // rows of 1.2 M entries, n = 256 118 us, 123 (124); of 3 M 224, 234
            // (237); of 2 M, n = 512 323, 333 (336); 40000 rows, n = 201 156, 161
            // (162); where one wave holds all long rows, and with split sums, equal.
            // (Each object made once; one that failed is retried by the next build.)
            if (!h->side) {
                int lo = 0, hi = 0;
                cudaStream_t side = nullptr;
                GCOO_CUDA(cudaDeviceGetStreamPriorityRange(&lo, &hi));
                GCOO_CUDA(cudaStreamCreateWithPriority(&side, cudaStreamNonBlocking, hi));
                h->side = side;
            }
            for (cudaEvent_t *ev : {&h->ev_fork, &h->ev_join}) {
                if (*ev)
                    continue;
                cudaEvent_t made = nullptr;
                GCOO_CUDA(cudaEventCreateWithFlags(&made, cudaEventDisableTiming));
                *ev = made;
            }
        }
    }
    h->built = true;
    return GCOO_SUCCESS;
}

} // namespace

// gcoo_build. mul (may be null): the multiply that follows (gcoo_multiply_by).
// A steady loop's multiply goes into the stream behind the one-read rebuild,
// before the rebuild's totals are back on the host, so the GPU does not wait
// for the host between the two (800^2 at 10 %, n = 800: 39.5 us a call
// against 54 with the wait, a second memset, a copy of the totals and one
// launch more); mul->done says so. Only the row walk of a matrix that was not skewed by the
// last build's totals goes ahead: any launch shape gives it the same chains,
// and where the arrays turn out too small the placing kernel voids the row
// pointers, so that it reads and writes nothing and the host multiplies again.
struct NextMultiply {
    const float *dB;
    int64_t n;
    float *dC;
    bool done;
};

// last density up to which one read of A takes any matrix (build_handle)
constexpr double kStagedDensity = 0.26;

static gcoo_status build_handle(gcoo_handle *h, cudaStream_t st, NextMultiply *mul)
{
    const bool ahead = mul && h->built && !h->coo && h->n_long == 0 && h->p.fp32_sum == GCOO_SUM_CHAIN &&
                       fp32_walk(h, mul->n, mul->dB, mul->dC) == kWalkRows;
    h->built = false;
    h->seg_prefix = false;
    if (h->coo) {
        gcoo_status s = coo_build(h, st);
        if (s != GCOO_SUCCESS)
            return s;
        return finish_build(h, st);
    }
    const int32_t cpg = h->p.rows_per_group;
    const bool tiled = tiled_convert_ok(h->dA, h->m, h->k, cpg);
    const bool one_scan = tiled && prefix_scan_ok(h->m); // needs no scan scratch
    if (!h->row_ptr.ensure(static_cast<size_t>(h->m) + 1) || !h->groups.ensure(2 * static_cast<size_t>(h->ng + 1)) ||
        (!one_scan && !h->scratch.ensure(scan_scratch_elems(h->m))) || !h->status.ensure(2 + 8 * 2))
        return fail(GCOO_ERROR_ALLOC, "device allocation of the GCOO index arrays failed");
    // [0] total nnz, [1] longest row, [2] distinct group columns, [3] staging status, [4] overflowed tiles,
    // [5] tickets of the prefix-and-scan and the sampling kernel, [6] entries and [7] distinct columns of the sample;
    // behind the status word: one memset clears all
    int64_t *d_total = reinterpret_cast<int64_t *>(h->status.ptr + 2);
    GCOO_CUDA(cudaMemsetAsync(h->status.ptr, 0, 8 + 8 * sizeof(int64_t), st));
    unsigned int *ticket = reinterpret_cast<unsigned int *>(d_total + 5);
    // One read of A when the entry arrays of an earlier build have room (a
    // steady loop of mutiplyBy / build); otherwise, or if they turn out too
    // small, the two-pass path below converts and sizes them exactly.
    const int64_t cap = std::min<int64_t>(static_cast<int64_t>(h->vals.count), static_cast<int64_t>(h->rc.count / 2));
    // Not where much lies above 26 % (the slots hold 25 %): nearly every tile
    // overflows and is read again (8192^2, 4 rows: at 40 % 635 us, two passes 521, at
    // 30 % 477 / 386, at 25 % 323 / 333; 4000 x 4001 at 40 % 184 / 139), sooner off
    // 16-byte boundaries, where the second pass is another kernel (3000 x 3001: at
    // 60 % 161 / 97, at 90 % 240 / 121; 2000 x 2001 at 90 % 97 / 74; aligned: 3000^2 at
    // 60 % 146 / 121, 2000^2 92 / 85 at 90 %). With few entries, and more of them where
    // a multiply is enqueued ahead, the wait between the passes costs more
    // (multiply_by, n = 8, of 7062 x 1257 at 40 % 167 / 166, 2000 x 2001 at 40 % 88 /
    // 92, 1000 x 1001 52 / 58; 2000^2 at 90 % 154 / 158, 3000^2 at 60 % 318 / 291).
    const double size = static_cast<double>(h->m) * static_cast<double>(h->k);
    const bool shifted = h->k % 4 != 0 || (reinterpret_cast<uintptr_t>(h->dA) & 15) != 0; // rows off 16 bytes
    const double above = static_cast<double>(h->nnz) - kStagedDensity * size;
    const double most = ahead ? (shifted ? 8e5 : 2.5e6) : (shifted ? 3e5 : 6e5);
    const bool one_read = above <= 0 || (size < 1.5e7 && above <= most);
    if (tiled && h->vals.ptr && h->rc.ptr && cap > 0 && one_read && staged_convert_ok(h->dA, h->m, h->k, cpg)) {
        const int64_t tiles = staged_tiles(h->m, h->k, cpg);
        const int32_t slot = staged_slot(h->nnz, tiles, cpg);
        if (!h->tile_cnt.ensure(static_cast<size_t>(h->m * conv_segments(h->k))) ||
            !h->stage.ensure(static_cast<size_t>(tiles) * static_cast<size_t>(slot)) ||
            !h->tile_tot.ensure(static_cast<size_t>(tiles)) || !h->over_list.ensure(static_cast<size_t>(tiles)))
            return fail(GCOO_ERROR_ALLOC, "device allocation of the staged conversion state failed");
        if (!h->readback && cudaMallocHost(&h->readback, kReadbackWords * sizeof(int64_t)) != cudaSuccess) {
            h->readback = nullptr;
            return fail(GCOO_ERROR_ALLOC, "page-locked allocation of the readback words failed");
        }
        if (!h->ev_totals) {
            cudaEvent_t made = nullptr;
            GCOO_CUDA(cudaEventCreateWithFlags(&made, cudaEventDisableTiming));
            h->ev_totals = made;
        }
        unsigned long long *over_count = reinterpret_cast<unsigned long long *>(d_total + 4);
        GCOO_CUDA(launch_stage(h->dA, h->m, h->k, cpg, slot, h->tile_cnt.ptr,
                               reinterpret_cast<unsigned long long *>(d_total + 2), h->stage.ptr, h->tile_tot.ptr,
                               h->over_list.ptr, over_count, reinterpret_cast<uint32_t *>(d_total + 3), st));
        if (one_scan) { // which also writes the readback words
            GCOO_CUDA(launch_prefix_scan(h->tile_cnt.ptr, conv_segments(h->k), h->row_ptr.ptr, h->m, cpg,
                                         h->group_index(), h->nnz_per_group(), d_total, ticket, h->readback,
                                         h->status.ptr, st));
        } else {
            GCOO_CUDA(launch_tile_prefix(h->tile_cnt.ptr, h->m, h->k, h->row_ptr.ptr, st));
            GCOO_CUDA(launch_row_scan_max(h->row_ptr.ptr, h->m, cpg, h->group_index(), h->nnz_per_group(), d_total,
                                          h->scratch.ptr, h->status.ptr, st));
        }
        // a matrix that needed the sample of its panels last time probably does again
        const bool sample = h->sampled;
        // placed on the device before the one readback (the kernel checks the fit itself)
        const int64_t packed_cap = static_cast<int64_t>(h->packed.count);
        GCOO_CUDA(launch_place(h->dA, h->m, h->k, cpg, slot, h->stage.ptr, h->tile_tot.ptr, h->over_list.ptr,
                               over_count, h->tile_cnt.ptr, h->group_index(), h->row_ptr.ptr, h->vals.ptr, h->rc.ptr,
                               h->packed.ptr, d_total, cap, packed_cap, ahead || sample ? h->row_ptr.ptr : nullptr, st));
        if (sample) // its totals with the others'
            GCOO_CUDA(launch_panel_share(h->packed.ptr, h->row_ptr.ptr, h->m, h->k,
                                         reinterpret_cast<unsigned long long *>(d_total + 6), ticket + 1,
                                         one_scan ? h->readback + 6 : nullptr, st));
        const int64_t *t3 = h->readback;
        if (!one_scan)
            GCOO_CUDA(cudaMemcpyAsync(h->readback, d_total, kReadbackWords * sizeof(int64_t), cudaMemcpyDeviceToHost, st));
        GCOO_CUDA(cudaEventRecord(h->ev_totals, st));
        if (ahead) {
            const gcoo_status s = spdm_fp32(h, mul->dB, mul->n, mul->dC, st, nullptr);
            if (s != GCOO_SUCCESS) {
                cudaEventSynchronize(h->ev_totals); // nothing of this build writes the readback words any more
                return s;
            }
        }
        GCOO_CUDA(cudaEventSynchronize(h->ev_totals));
        const int64_t total = t3[0];
        if (t3[3] == 0 && (total < 0 || total > 0x7fffffffLL))
            return fail(GCOO_ERROR_FORMAT, "nnz = " + std::to_string(total) + " exceeds the int32 GCOO format");
        if (t3[3] == 0 && total <= cap && total + 2 <= packed_cap) {
            h->max_row_nnz = t3[1];
            h->distinct_cols = t3[2];
            h->nnz = total;
            h->seg_prefix = true;
            if (mul)
                mul->done = ahead;
            return finish_build(h, st, sample ? t3 + 6 : nullptr);
        }
        GCOO_CUDA(cudaMemsetAsync(d_total, 0, 8 * sizeof(int64_t), st));
    }
    if (tiled) {
        if (!h->tile_cnt.ensure(static_cast<size_t>(h->m * conv_segments(h->k))))
            return fail(GCOO_ERROR_ALLOC, "device allocation of the tile counts failed");
        GCOO_CUDA(launch_tile_count(h->dA, h->m, h->k, cpg, h->tile_cnt.ptr,
                                    reinterpret_cast<unsigned long long *>(d_total + 2), st));
    } else {
        GCOO_CUDA(launch_row_count(h->dA, h->m, h->k, h->row_ptr.ptr, st));
    }
    if (one_scan) {
        GCOO_CUDA(launch_prefix_scan(h->tile_cnt.ptr, conv_segments(h->k), h->row_ptr.ptr, h->m, cpg, h->group_index(),
                                     h->nnz_per_group(), d_total, ticket, nullptr, h->status.ptr, st));
    } else {
        if (tiled)
            GCOO_CUDA(launch_tile_prefix(h->tile_cnt.ptr, h->m, h->k, h->row_ptr.ptr, st));
        GCOO_CUDA(launch_row_scan_max(h->row_ptr.ptr, h->m, h->p.rows_per_group, h->group_index(), h->nnz_per_group(),
                                      d_total, h->scratch.ptr, h->status.ptr, st));
    }
    // a matrix that needed the sample of its panels last time probably does again
    const bool sample2 = tiled && h->sampled && dense_share_ok(h->k);
    if (sample2)
        GCOO_CUDA(launch_dense_share(h->dA, h->m, h->k, kSampleEntries, h->p.fp32_order == 2, d_total,
                                     reinterpret_cast<unsigned long long *>(d_total + 6), st));
    int64_t tot2[kReadbackWords] = {};
    GCOO_CUDA(cudaMemcpyAsync(tot2, d_total, sizeof(tot2), cudaMemcpyDeviceToHost, st));
    GCOO_CUDA(cudaStreamSynchronize(st));
    const int64_t total = tot2[0];
    h->max_row_nnz = tot2[1];
    h->distinct_cols = tiled ? tot2[2] : 0; // 0: not counted
    if (total < 0 || total > 0x7fffffffLL)
        return fail(GCOO_ERROR_FORMAT, "nnz = " + std::to_string(total) + " exceeds the int32 GCOO format");
    const size_t nnz = static_cast<size_t>(total);
    // a little room beyond nnz lets later builds of a similar matrix take the one-pass path
    const size_t room = tiled ? nnz + nnz / 16 + 1024 : nnz;
    if (!h->vals.ensure(room) || !h->rc.ensure(2 * room) || !h->packed.ensure(room + 2))
        return fail(GCOO_ERROR_ALLOC, "device allocation of the GCOO entry arrays failed");
    // rows and cols live in one block, as in the reference (src/ShGCOOSpDM.cu:95-97)
    int32_t *rows = h->rc.ptr;
    int32_t *cols = h->rc.ptr + nnz;
    // dense rows off 16-byte boundaries: a CTA per group with 4-byte loads (4000 x
    // 4001 at 40 %, 4 rows: two passes 139 us, with shifted rows 161)
    const bool dense = static_cast<double>(total) > kStagedDensity * size && shifted && cpg > 1;
    if (tiled && !dense)
        GCOO_CUDA(launch_tile_scatter(h->dA, h->m, h->k, cpg, h->tile_cnt.ptr, h->group_index(), h->row_ptr.ptr,
                                      h->vals.ptr, rows, cols, h->packed.ptr, st));
    else
        GCOO_CUDA(launch_scatter(h->dA, h->m, h->k, cpg, h->group_index(), h->row_ptr.ptr, h->vals.ptr, rows,
                                 cols, h->packed.ptr, st, dense));
    h->nnz = total;
    h->seg_prefix = tiled;
    return finish_build(h, st, sample2 ? tot2 + 6 : nullptr);
}

gcoo_status gcoo_build(gcoo_handle *h, void *stream)
{
    NvtxRange nvtx("gcoo_build");
    if (!h)
        return fail(GCOO_ERROR_INVALID_VALUE, "handle is NULL");
    return build_handle(h, static_cast<cudaStream_t>(stream), nullptr);
}

gcoo_status gcoo_spdm_left(gcoo_handle *h, const float *dD, int64_t p, float *dC, void *stream)
{
    NvtxRange nvtx("gcoo_spdm_left");
    if (!h || !dD || !dC)
        return fail(GCOO_ERROR_INVALID_VALUE, "NULL handle or matrix pointer");
    if (!h->built)
        return fail(GCOO_ERROR_NOT_BUILT, "gcoo_build has not run");
    gcoo_status s = check_n(p);
    if (s != GCOO_SUCCESS)
        return s;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    s = left_prepare(h, h->left, p, st);
    if (s != GCOO_SUCCESS)
        return s;
    return left_spdm(h, *h->left, dD, p, dC, st);
}

gcoo_status gcoo_create_coo(gcoo_handle **out, int64_t m, int64_t k, const int32_t *d_rows, const int32_t *d_cols,
                            const float *d_vals, int64_t nnz, const gcoo_params *params)
{
    if (!out)
        return fail(GCOO_ERROR_INVALID_VALUE, "out is NULL");
    *out = nullptr;
    if (nnz < 0 || (nnz > 0 && (!d_rows || !d_cols || !d_vals)))
        return fail(GCOO_ERROR_INVALID_VALUE, "NULL triplet arrays or negative nnz");
    if (nnz > 0x7fffffffLL)
        return fail(GCOO_ERROR_FORMAT, "more triplets than the int32 GCOO format holds");
    // reuse the dense constructor's validation with a placeholder operand
    static const float placeholder = 0.0f;
    gcoo_status s = gcoo_create(out, &placeholder, m, k, params);
    if (s != GCOO_SUCCESS)
        return s;
    gcoo_handle *h = *out;
    h->dA = nullptr;
    h->coo = true;
    h->coo_rows = d_rows;
    h->coo_cols = d_cols;
    h->coo_vals = d_vals;
    h->coo_nnz = nnz;
    return GCOO_SUCCESS;
}

gcoo_status gcoo_export(const gcoo_handle *h, gcoo_view *out)
{
    if (!h || !out)
        return fail(GCOO_ERROR_INVALID_VALUE, "handle or view is NULL");
    if (!h->built)
        return fail(GCOO_ERROR_NOT_BUILT, "gcoo_build has not run");
    out->m = h->m;
    out->k = h->k;
    out->nnz = h->nnz;
    out->n_group = h->ng;
    out->rows_per_group = h->p.rows_per_group;
    out->group_index = h->groups.ptr;
    out->nnz_per_group = h->groups.ptr + (h->ng + 1);
    out->vals = h->vals.ptr;
    out->rows = h->rc.ptr;
    out->cols = h->rc.ptr + h->nnz;
    return GCOO_SUCCESS;
}

gcoo_status gcoo_spdm(gcoo_handle *h, const float *dB, int64_t n, float *dC, void *stream)
{
    NvtxRange nvtx("gcoo_spdm");
    if (!h || !dB || !dC)
        return fail(GCOO_ERROR_INVALID_VALUE, "NULL handle or matrix pointer");
    if (!h->built)
        return fail(GCOO_ERROR_NOT_BUILT, "gcoo_build has not run");
    gcoo_status s = check_n(n);
    if (s != GCOO_SUCCESS)
        return s;
    return spdm_fp32(h, dB, n, dC, static_cast<cudaStream_t>(stream), nullptr);
}

gcoo_status gcoo_spdm_ex(gcoo_handle *h, const float *dB, int64_t n, float *dC, gcoo_precision prec, void *stream)
{
    NvtxRange nvtx("gcoo_spdm_ex");
    if (!h || !dB || !dC)
        return fail(GCOO_ERROR_INVALID_VALUE, "NULL handle or matrix pointer");
    if (!h->built)
        return fail(GCOO_ERROR_NOT_BUILT, "gcoo_build has not run");
    gcoo_status s = check_n(n);
    if (s != GCOO_SUCCESS)
        return s;
    if (prec == GCOO_PREC_FP32)
        return spdm_fp32(h, dB, n, dC, static_cast<cudaStream_t>(stream), nullptr);
    if (prec < GCOO_PREC_FP32 || prec > GCOO_PREC_FP8_B)
        return fail(GCOO_ERROR_INVALID_VALUE, "unknown precision");
    return run_form(h, dB, n, dC, prec, static_cast<cudaStream_t>(stream), false);
}

gcoo_status gcoo_prepare(gcoo_handle *h, int64_t n, gcoo_precision prec, void *stream)
{
    if (!h)
        return fail(GCOO_ERROR_INVALID_VALUE, "handle is NULL");
    if (!h->built)
        return fail(GCOO_ERROR_NOT_BUILT, "gcoo_build has not run");
    gcoo_status s = check_n(n);
    if (s != GCOO_SUCCESS)
        return s;
    if (prec == GCOO_PREC_FP32) // the split summation's partial sums, if this handle sums in pieces
        return h->p.fp32_sum == GCOO_SUM_SPLIT && h->n_long > 0 ? ensure_split_work(h, n) : GCOO_SUCCESS;
    if (prec < GCOO_PREC_FP32 || prec > GCOO_PREC_FP8_B)
        return fail(GCOO_ERROR_INVALID_VALUE, "unknown precision");
    return run_form(h, nullptr, n, nullptr, prec, static_cast<cudaStream_t>(stream), true);
}

gcoo_status gcoo_multiply_by(gcoo_handle *h, const float *dB, int64_t n, float *dC, void *stream)
{
    NvtxRange nvtx("gcoo_multiply_by");
    if (!h || !dB || !dC)
        return fail(GCOO_ERROR_INVALID_VALUE, "NULL handle or matrix pointer");
    gcoo_status s = check_n(n);
    if (s != GCOO_SUCCESS)
        return s;
    NextMultiply mul{dB, n, dC, false};
    s = build_handle(h, static_cast<cudaStream_t>(stream), &mul);
    if (s != GCOO_SUCCESS || mul.done)
        return s;
    return spdm_fp32(h, dB, n, dC, static_cast<cudaStream_t>(stream), nullptr);
}

gcoo_status gcoo_destroy(gcoo_handle *h)
{
    delete h; // DevBuf members release through the allocator
    return GCOO_SUCCESS;
}

gcoo_status gcoo_query_engine(gcoo_handle *h, gcoo_precision prec, int32_t *tensor)
{
    if (!h || !tensor)
        return fail(GCOO_ERROR_INVALID_VALUE, "NULL argument");
    if (!h->built)
        return fail(GCOO_ERROR_NOT_BUILT, "gcoo_build has not run");
    *tensor = (prec != GCOO_PREC_FP32 && form_uses_tensor(h, prec)) ? 1 : 0;
    return GCOO_SUCCESS;
}

gcoo_status gcoo_device_status(gcoo_handle *h, void *stream, uint32_t *status)
{
    if (!h || !status)
        return fail(GCOO_ERROR_INVALID_VALUE, "NULL argument");
    *status = 0;
    if (!h->status.ptr)
        return GCOO_SUCCESS;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    GCOO_CUDA(cudaMemcpyAsync(status, h->status.ptr, sizeof(uint32_t), cudaMemcpyDeviceToHost, st));
    GCOO_CUDA(cudaStreamSynchronize(st));
    if (*status & kStatusWaitTimeout)
        return fail(GCOO_ERROR_TIMEOUT, "a bounded device wait gave up");
    return GCOO_SUCCESS;
}

gcoo_status gcoo_convert_count(const float *dA, int64_t m, int64_t k, int32_t rows_per_group, int32_t *d_group_index,
                               int32_t *d_nnz_per_group, int64_t *nnz, void *stream)
{
    if (!dA || !d_group_index || !d_nnz_per_group || !nnz)
        return fail(GCOO_ERROR_INVALID_VALUE, "NULL argument");
    gcoo_status s = check_dims(m, k);
    if (s != GCOO_SUCCESS)
        return s;
    if (!valid_cpg(rows_per_group))
        return fail(GCOO_ERROR_INVALID_VALUE, "rows_per_group must be a power of two in [1, 32]");
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const int64_t ng = (m + rows_per_group - 1) / rows_per_group;
    if (group_counts_ok(dA, m, k, ng)) {
        GCOO_CUDA(launch_group_counts(dA, m, k, rows_per_group, d_group_index, d_nnz_per_group, st));
        int32_t total = 0;
        GCOO_CUDA(cudaMemcpyAsync(&total, d_group_index + ng, sizeof(total), cudaMemcpyDeviceToHost, st));
        GCOO_CUDA(cudaStreamSynchronize(st));
        *nnz = total;
        return GCOO_SUCCESS;
    }
    DevBuf<int32_t> counts;
    DevBuf<int64_t> scratch;
    const size_t sc = scan_scratch_elems(m);
    if (!counts.ensure(static_cast<size_t>(m) + 1) || !scratch.ensure(sc + 1))
        return fail(GCOO_ERROR_ALLOC, "device allocation of conversion scratch failed");
    GCOO_CUDA(launch_row_count(dA, m, k, counts.ptr, st));
    GCOO_CUDA(launch_row_scan(counts.ptr, m, rows_per_group, d_group_index, d_nnz_per_group, scratch.ptr + sc,
                              scratch.ptr, nullptr, st));
    int64_t total = 0;
    GCOO_CUDA(cudaMemcpyAsync(&total, scratch.ptr + sc, sizeof(total), cudaMemcpyDeviceToHost, st));
    GCOO_CUDA(cudaStreamSynchronize(st));
    *nnz = total;
    if (total > 0x7fffffffLL)
        return fail(GCOO_ERROR_FORMAT, "nnz exceeds the int32 GCOO format");
    return GCOO_SUCCESS;
}

gcoo_status gcoo_convert_scatter(const float *dA, int64_t m, int64_t k, int32_t rows_per_group,
                                 const int32_t *d_group_index, float *d_vals, int32_t *d_rows, int32_t *d_cols,
                                 void *stream)
{
    if (!dA || !d_group_index || !d_vals || !d_rows || !d_cols)
        return fail(GCOO_ERROR_INVALID_VALUE, "NULL argument");
    gcoo_status s = check_dims(m, k);
    if (s != GCOO_SUCCESS)
        return s;
    if (!valid_cpg(rows_per_group))
        return fail(GCOO_ERROR_INVALID_VALUE, "rows_per_group must be a power of two in [1, 32]");
    GCOO_CUDA(launch_scatter(dA, m, k, rows_per_group, d_group_index, nullptr, d_vals, d_rows, d_cols, nullptr,
                             static_cast<cudaStream_t>(stream)));
    return GCOO_SUCCESS;
}

gcoo_status gcoo_spdm_view(const gcoo_view *a, const float *dB, int64_t n, float *dC, void *stream)
{
    if (!a || !dB || !dC || !a->group_index || !a->nnz_per_group)
        return fail(GCOO_ERROR_INVALID_VALUE, "NULL argument");
    if (a->nnz > 0 && (!a->vals || !a->rows || !a->cols))
        return fail(GCOO_ERROR_INVALID_VALUE, "NULL entry arrays");
    gcoo_status s = check_dims(a->m, a->k);
    if (s != GCOO_SUCCESS)
        return s;
    s = check_n(n);
    if (s != GCOO_SUCCESS)
        return s;
    if (a->rows_per_group < 1 || a->rows_per_group > 32 ||
        a->n_group != (a->m + a->rows_per_group - 1) / a->rows_per_group)
        return fail(GCOO_ERROR_INVALID_VALUE, "inconsistent rows_per_group / n_group");
    GCOO_CUDA(launch_spdm_view(*a, dB, n, dC, static_cast<cudaStream_t>(stream)));
    return GCOO_SUCCESS;
}

gcoo_status gcoo_error_norm(gcoo_handle *h, const float *dB, int64_t n, const float *dC, double *rel_fro,
                            void *stream)
{
    if (!h || !dB || !dC || !rel_fro)
        return fail(GCOO_ERROR_INVALID_VALUE, "NULL argument");
    if (!h->built)
        return fail(GCOO_ERROR_NOT_BUILT, "gcoo_build has not run");
    gcoo_status s = check_n(n);
    if (s != GCOO_SUCCESS)
        return s;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (!h->norm.ensure(2))
        return fail(GCOO_ERROR_ALLOC, "device allocation failed");
    GCOO_CUDA(cudaMemsetAsync(h->norm.ptr, 0, 2 * sizeof(double), st));
    GCOO_CUDA(launch_error_norm(h->packed.ptr, h->row_ptr.ptr, h->m, dB, n, dC, h->norm.ptr, st));
    double acc[2] = {0.0, 0.0};
    GCOO_CUDA(cudaMemcpyAsync(acc, h->norm.ptr, sizeof(acc), cudaMemcpyDeviceToHost, st));
    GCOO_CUDA(cudaStreamSynchronize(st));
    if (acc[1] == 0.0)
        *rel_fro = acc[0] == 0.0 ? 0.0 : INFINITY;
    else
        *rel_fro = sqrt(acc[0]) / sqrt(acc[1]);
    return GCOO_SUCCESS;
}

} // extern "C"
