/* gexs_internal.h — declarations shared by the library's translation units. */
#pragma once
#include <cstdint>
#include <string>
#include <cuda_runtime.h>
#include "../../include/gexs_b200.h"

namespace gexs {

/* kernel launchers (gexs_kernels.cu; tile kernels in gexs_tiles.cuh) */
int profile_class(const gexs_job& j);
int tile_bins(const gexs_launch_cfg& c);
/* Line slices of the tile kernels (the FP32 Voigt region-I kernel and
 * tile_kernel; the core kernel has its own, below): a tile whose line range
 * holds more than `lines_per_slice` lines is cut into
 * ceil(n / lines_per_slice) work items.  FP32 sums depend on the cut, which
 * therefore depends on the tile alone (unless the partial rows would pass
 * 1 GiB); FP64 sums do not (SUM_BLOCK).  A split tile's slices write
 * partial rows; the last one to finish sums them in slice order into the
 * output.  All arrays live in the launch table; the set-up kernel fills
 * them (and zeroes the tickets) before the kernel runs. */
struct SliceTables {
    int*       prefix;      /* ntiles + 1: first item of each tile       */
    int*       counts;      /* ntiles: slices per tile                   */
    int*       rowbase;     /* ntiles: first partial row of a split tile */
    int*       ticket;      /* ntiles: slices finished                   */
    long long* lohi;        /* 2 ntiles: each tile's line range          */
    int*       nitems;      /* 1: items of the launch                    */
    double*    rows;        /* max_rows x tile bins: partial rows        */
    int        max_rows;
    long long  lines_per_slice;
    int        round_rows;  /* core kernel: rows of a round (core_rows), 0: one round */
    int        split;       /* FP32 erf, Voigt: items are parts of a tile   */
};

/* One set-up launch (prep arrays, slice tables) where there is any to do,
 * then the kernels of one (profile class, precision).
 * d_prep: device array of per-job prep arrays (S | invw | y, 3 N doubles
 * each), filled here for lists of up to prep_lines lines, or NULL to derive
 * every line on load.
 * d_order: tile-major order tables of a launch with several jobs (F | R | P,
 * 3 njobs + 1 ints, see tile_order in gexs_capi.cu), or NULL for job-major
 * items.
 * d_counter: a 256-byte block of work counters, zeroed by the caller: int 0
 * the tile kernel's, 16 the set-up kernel's, 32 the core kernel's.
 * tiles_after: an event that the kernels after the set-up wait for, or NULL. */
cudaError_t launch_tiles(int pk, int prec, const gexs_job* d_jobs, const int* d_prefix,
                         int njobs, int nitems, int* d_counter, int* d_err,
                         double* const* d_prep, const gexs_launch_cfg& cfg, int nsm,
                         cudaStream_t st, const SliceTables* sl = nullptr,
                         const SliceTables* csl = nullptr, const int* d_order = nullptr,
                         int64_t prep_lines = 0, cudaEvent_t tiles_after = nullptr);
/* The FP64 tile kernel sums a bin's lines in order within blocks of this
 * many lines of the list (by index, so that a tile of any shape or cut has
 * the same block sums) and the blocks' sums as (hi, lo) pairs, whose
 * rounded total does not depend on their order but for a near tie (dd_add):
 * a result is the same for every tile shape, slice length and batch.
 * Sub-lists of one list start at multiples of it. */
constexpr int SUM_BLOCK = GEXS_LINE_BLOCK;

/* doubles of a partial row: a value per bin, (hi, lo) in the FP64 forms */
__host__ __device__ inline int row_doubles(int prec, int tile_w)
{
    return prec == GEXS_FP64 ? 2 * tile_w : tile_w;
}

/* which groups are sliced; lines_per_slice for a group and the bound on the
 * rows of its split tiles */
bool slices_apply(int pk, int prec);
long long slice_lines(const gexs_job* jobs, int njobs, int prec, int tile_w, int* max_rows);

/* bytes of partial rows held at a time */
constexpr long long ROW_BYTES = 1ll << 30;

/* The core kernel takes a tile in sub-tiles of at most CORE_W bins (a row of
 * doubles per warp in shared memory); a sliced tile of more bins is
 * core_subtiles core tiles.
 * Its own slices (its line range per core tile is reach_range's): FP32 only
 * when a tile is one sub-tile.  FP32 sums depend on the cut, so it depends
 * on the tile's lines and on the size of the job's whole grid alone: a
 * batch, a sub-range and a sub-list of a job are cut alike.
 * Lines per slice by the tiles of the grid, because a job of few tiles has
 * only its lines to fill the chip with.  Core of FP32 lists with slices of
 * 256, 512 and 2048 lines, us: 3e5 lines on 60 tiles 77, 90, 260; on 200
 * tiles 1e6 lines 234, 238, 306, 3e4 lines 45, 42, 43; 1e6 lines on 2000
 * tiles 432, 411, 381. */
constexpr int CORE_W = 1024;
__host__ __device__ constexpr int core_width(int tile_w) { return tile_w < CORE_W ? tile_w : CORE_W; }
__host__ __device__ constexpr int core_subtiles(int tile_w) { return (tile_w + CORE_W - 1) / CORE_W; }
__host__ __device__ inline long long core_cut(long long grid_points, int tile_w)
{
    const long long tiles = (grid_points + tile_w - 1) / tile_w;
    return tiles < 148 ? 256ll : tiles < 296 ? 512ll : 2048ll;
}
/* most slices of a tile (longer ones beyond): the rows of one job stay
 * within ROW_BYTES, and a thousand items, eight thousand for a job of few
 * tiles, fill the ~900 CTAs that fit */
__host__ __device__ inline long long core_max_slices(long long grid_points, int tile_w, int prec)
{
    const long long tiles = grid_points > tile_w ? (grid_points + tile_w - 1) / tile_w : 1;
    const long long fit = ROW_BYTES / (long long)sizeof(double) / (tiles * row_doubles(prec, tile_w));
    const long long use = 8192 / tiles > 1024 ? 8192 / tiles : 1024;
    return fit < 1 ? 1 : fit < use ? fit : use;
}
/* slices of a core tile with n lines (tile_w here and above: core_width) */
__host__ __device__ inline int core_slices(long long n, long long grid_points, int tile_w, int prec)
{
    const long long per = core_cut(grid_points, tile_w);
    if (n <= per) return 1;
    const long long ns = (n + per - 1) / per, most = core_max_slices(grid_points, tile_w, prec);
    return (int)(ns < most ? ns : most);
}
bool core_slices_apply(int pk, int prec, int tile_w);
/* partial rows of a launch's core slices: a bound on their number (false:
 * more than an int holds), the rows of a round (0: all are held and there is
 * one round) and those to allocate.  With several rounds the core
 * kernel is launched once for each range of round_rows rows, over the tiles
 * whose rows begin there, and the ranges share the memory; the last tile's
 * rows may reach past the range. */
struct CoreRows { int bound, round_rows, alloc; };
bool core_rows(const gexs_job* jobs, int njobs, int prec, int tile_w, CoreRows* out);
/* whether a tile's parts are items of their own: FP32 erf profiles, FP32
 * Voigt region I (4 bins x 4 warps) */
bool erf_split(const gexs_job* jobs, int njobs, int tile_w);
bool ws_split(const gexs_job* jobs, int njobs, int tile_w);
cudaError_t launch_count(const gexs_job* d_jobs, int njobs, unsigned long long* d_counts,
                         int nsm, cudaStream_t st);
cudaError_t launch_partition(const double* d_e, const int32_t* d_g, int64_t n,
                             const double* d_betas, int nt, double* d_partial, int nchunk,
                             double* d_q, cudaStream_t st);

/* small control writes done by kernels (gexs_kernels.cu): a launch table
 * passed as kernel parameters (at most kMaxParamUpload bytes) and zeroed
 * work counters, so that they never queue on a copy engine behind bulk
 * host-to-device copies of lines running on another stream */
const size_t kMaxParamUpload = 64 * 1024;
cudaError_t put_bytes(void* dst, const void* src, size_t n, cudaStream_t st);
cudaError_t zero_ints(int* p, int n, cudaStream_t st);
/* *out = the error word, which is set to zero in the same atomic step */
cudaError_t take_word(int* word, int* out, cudaStream_t st);

/* gexs_run with the kernels' error flags going to d_err (device int)
 * instead of the context's own word (NULL: the context's); the kernels after
 * the set-up wait for the event tiles_after (NULL: none) */
int run_jobs(gexs_ctx* ctx, const gexs_job* jobs, int njobs, const gexs_launch_cfg* cfg,
             void* stream, int* d_err, cudaEvent_t tiles_after = nullptr);

/* device scratch run_jobs takes from the context's pool for these jobs
 * (launch tables, per-job prep arrays, line-slice rows), in bytes */
int run_scratch_bytes(gexs_ctx* ctx, const gexs_job* jobs, int njobs, const gexs_launch_cfg* cfg,
                      size_t* bytes);

/* context accessors (gexs_capi.cu); ctx_pool may be NULL (then the
 * device's default pool serves the context) */
int ctx_device(gexs_ctx* c);
int ctx_sm_count(gexs_ctx* c);
cudaMemPool_t ctx_pool(gexs_ctx* c);
/* stream-ordered allocation from a pool (NULL: the device default); on an
 * out-of-memory the pool's unused pages are released and the call retried */
cudaError_t pool_alloc(cudaMemPool_t pool, void** p, size_t bytes, cudaStream_t s);

/* gexs_ctx_upload's worker (gexs_upload.cpp) */
struct Uploader;
Uploader* uploader_create(int device);
void uploader_destroy(Uploader* u);
cudaError_t upload(Uploader* u, const gexs_upload_piece* pieces, int n, cudaStream_t s);
Uploader* ctx_uploader(gexs_ctx* c);

/* error reporting (gexs_capi.cu): thread-local message, returns status */
int set_error(int status, const std::string& msg);
int cuda_error(cudaError_t e, const char* where);

/* validation shared by the run paths */
int validate_job(const gexs_job& j, int index);

}  // namespace gexs
