/*
 * gexs_kernels.cu — the set-up kernel (per-line prep arrays, slice tables),
 * exact evaluation counting, Q(T), and the front of the tile-kernel
 * dispatch (the tile kernels themselves are in gexs_tiles.cuh).
 */
#include <cmath>
#include <cstring>
#include <cub/cub.cuh>
#include "gexs_tiles.cuh"

namespace gexs {

/* ------------------------------------------------------------ prep
 * Per job, the FP64 per-line quantities once: S at base[i], invw at
 * base[N + i], y at base[2N + i] (N = line count).  The tile kernel then
 * reads 32 bytes per line instead of recomputing two exponentials, a power
 * and two divisions for every tile the line reaches.  Lines first + k
 * stride. */
__device__ __forceinline__ void prep_lines(const gexs_job& J, double* base, int64_t first,
                                           int64_t stride)
{
    const int64_t N = J.lines.count;
    const bool press = J.profile == GEXS_VOIGT || J.profile == GEXS_VOIGT_QUAD;
    const bool compact = J.lines.format == GEXS_LINES_COMPACT;
    for (int64_t i = first; i < N; i += stride) {
        RawLine L;
        L.nu = J.lines.nu[i];
        if (compact) {
            /* floats widened to FP64; aif holds g' A */
            L.elow = (double)reinterpret_cast<const float*>(J.lines.elow)[i];
            L.aif = (double)reinterpret_cast<const float*>(J.lines.aif)[i];
            L.g = 1;
        } else {
            L.elow = J.lines.elow[i]; L.aif = J.lines.aif[i];
            L.g = J.lines.gns[i];
        }
        LineQ q;
        if (press) {
            if (compact) {
                L.gam = (double)reinterpret_cast<const float*>(J.lines.gamma)[i];
                L.nexp = (double)reinterpret_cast<const float*>(J.lines.n)[i];
            } else {
                L.gam = J.lines.gamma[i]; L.nexp = J.lines.n[i];
            }
            q = line_quantities<true>(J, L);
        } else {
            L.gam = 0.0; L.nexp = 0.0;
            q = line_quantities<false>(J, L);
        }
        base[i] = q.S;
        base[N + i] = q.invw;
        base[2 * N + i] = q.y;
    }
}

/* ------------------------------------------------------ eval counting */
__global__ void count_kernel(const gexs_job* __restrict__ jobs, unsigned long long* counts)
{
    const gexs_job& J = jobs[blockIdx.y];
    unsigned long long local = 0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < J.lines.count;
         i += (int64_t)gridDim.x * blockDim.x) {
        double nu = J.lines.nu[i];
        if (nu == 0.0) nu = 1e-6;
        int64_t s0 = J.start_idx, s1 = J.start_idx + J.n_points;
        int64_t jl, jh;
        if (J.window_rule == GEXS_WINDOW_ROUNDED) {
            double ib = round(ddiv(dsub(dsub(nu, J.cutoff), J.nu_start), J.dnu));
            double ie = round(ddiv(dsub(dadd(nu, J.cutoff), J.nu_start), J.dnu));
            ib = fmax(ib, (double)s0); ie = fmin(ie, (double)s1);
            jl = (int64_t)ib; jh = (int64_t)ie; if (jh < jl) jh = jl;
        } else {
            auto in = [&](int64_t j) { return fabs(dsub(grid_f(J.nu_start, J.dnu, j), nu)) <= J.cutoff; };
            double c = ddiv(dsub(nu, J.nu_start), J.dnu), w = ddiv(J.cutoff, J.dnu);
            double le = floor(c - w) - 2.0, he = ceil(c + w) + 2.0;
            jl = (int64_t)fmax((double)s0, fmin(le, (double)s1));
            jh = (int64_t)fmax((double)s0, fmin(he, (double)s1));
            int guard = 0;
            while (jl > s0 && in(jl - 1) && guard++ < 64) --jl;
            while (jl < jh && !in(jl) && guard++ < 128) ++jl;
            while (jh < s1 && in(jh) && guard++ < 192) ++jh;
            while (jh > jl && !in(jh - 1) && guard++ < 256) --jh;
        }
        local += (unsigned long long)(jh - jl);
    }
    for (int o = 16; o > 0; o >>= 1) local += __shfl_down_sync(0xffffffffu, local, o);
    if ((threadIdx.x & 31) == 0 && local) atomicAdd(counts + blockIdx.y, local);
}

/* ------------------------------------------------ partition function Q(T) */
__global__ void partition_partial(const double* __restrict__ e, const int32_t* __restrict__ g,
                                  int64_t n, const double* __restrict__ betas, double* partial)
{
    /* block (x = chunk, y = temperature); fixed-order tree reduction */
    __shared__ double red[256];
    const double beta = betas[blockIdx.y];
    double s = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        s += (double)g[i] * exp(-beta * e[i]);
    red[threadIdx.x] = s;
    __syncthreads();
    for (int o = blockDim.x / 2; o > 0; o >>= 1) {
        if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
        __syncthreads();
    }
    if (threadIdx.x == 0) partial[blockIdx.y * gridDim.x + blockIdx.x] = red[0];
}

__global__ void partition_final(const double* partial, int nchunk, int nt, double* q)
{
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nt) return;
    double s = 0.0;
    for (int c = 0; c < nchunk; ++c) s += partial[t * nchunk + c];
    q[t] = s;
}

int profile_class(const gexs_job& j)
{
    if (j.profile == GEXS_VOIGT) return PK_VOIGT;
    if (j.profile == GEXS_DOPPLER || j.profile == GEXS_GAUSSIAN) return PK_ERF;
    if (j.profile == GEXS_VOIGT_QUAD) return j.quad_nodes == 16 ? PK_GH16 : PK_GH32;
    return -1;
}

int tile_bins(const gexs_launch_cfg& c) { return 32 * c.bins_per_lane * c.warps; }

/* ------------------------------------------------------------ set-up
 * One launch before the tile kernels: the line ranges and slice counts of
 * every tile (a warp per tile), their scans (the last of those blocks to
 * finish) and the prep arrays (the other blocks).  Its work is short and
 * bound by launch latency for small jobs: separate kernels for prep, two
 * plans, two one-CTA scans and a counter reset cost 26 us of a 170 us pass
 * with 3000 lines, this one 11. */
namespace {

/* a tile's line range, searched exactly as the region-I kernel's producers
 * search it, and its slice count */
__device__ __forceinline__ void plan_tile(const KArgs& a, const gexs_job& J, int ti, int tj, int lane)
{
    const int64_t j0 = J.start_idx + (int64_t)tj * a.tile_w;
    const int jn = (int)min((int64_t)a.tile_w, J.start_idx + J.n_points - j0);
    const double f0 = grid_f(J.nu_start, J.dnu, j0);
    const double fl = grid_f(J.nu_start, J.dnu, j0 + jn - 1);
    const int64_t nl = J.lines.count;
    const double margin = 2.0 * J.dnu + 1e-9 * (fabs(fl) + J.cutoff);
    const int64_t lo = warp_bound<false>(J.lines.nu, nl, f0 - J.cutoff - margin, lane);
    const int64_t hi = max(warp_bound<true>(J.lines.nu, nl, fl + J.cutoff + margin, lane), lo);
    if (lane == 0) {
        const long long n = hi - lo, per = a.sl.lines_per_slice;
        a.sl.lohi[2 * ti] = lo;
        a.sl.lohi[2 * ti + 1] = hi;
        a.sl.counts[ti] = n > per ? (int)((n + per - 1) / per) : 1;
        a.sl.ticket[ti] = 0;
    }
}

/* the same for core tile ti of the core kernel, bins [t0, t0 + CORE_W) of a
 * tile that ends at tend, with its own search (reach_range) */
__device__ __forceinline__ void plan_core_tile(const KArgs& a, const gexs_job& J, int ti, int64_t t0,
                                               int64_t tend, int lane)
{
    if (t0 >= tend) {
        if (lane == 0) {
            a.csl.lohi[2 * ti] = a.csl.lohi[2 * ti + 1] = 0;
            a.csl.counts[ti] = 1;
            a.csl.ticket[ti] = 0;
        }
        return;
    }
    const int jn = (int)min((int64_t)CORE_W, tend - t0);
    const double f0 = grid_f(J.nu_start, J.dnu, t0);
    const double fl = grid_f(J.nu_start, J.dnu, t0 + jn - 1);
    const int64_t nl = J.lines.count;
    double vlo, vhi;
    reach_range(J, f0, fl, vlo, vhi);
    const int64_t lo = warp_bound<false>(J.lines.nu, nl, vlo, lane);
    const int64_t hi = max(warp_bound<true>(J.lines.nu, nl, vhi, lane), lo);
    if (lane == 0) {
        const long long n = hi - lo;
        a.csl.lohi[2 * ti] = lo;
        a.csl.lohi[2 * ti + 1] = hi;
        a.csl.counts[ti] = core_slices(n, J.grid_points, core_width(a.tile_w), J.precision);
        a.csl.ticket[ti] = 0;
    }
}

constexpr int SETUP_NT = 256, SCAN_ITEMS = 8;
typedef cub::BlockScan<unsigned long long, SETUP_NT> SetupScan;

/* exclusive prefixes of the slice counts (items, upper word) and of the
 * slices of split tiles (partial rows, lower word), and the item count */
__device__ void scan_slices(const SliceTables& sl, int ntiles, int* err,
                            SetupScan::TempStorage& tmp)
{
    unsigned long long carry = 0;
    for (int base = 0; base < ntiles; base += SETUP_NT * SCAN_ITEMS) {
        unsigned long long v[SCAN_ITEMS], tot;
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; ++k) {
            const int i = base + (int)threadIdx.x * SCAN_ITEMS + k;
            const unsigned c = i < ntiles ? (unsigned)__ldcg(sl.counts + i) : 0u;
            v[k] = ((unsigned long long)c << 32) | (c > 1 ? c : 0u);
        }
        SetupScan(tmp).ExclusiveSum(v, v, tot);
#pragma unroll
        for (int k = 0; k < SCAN_ITEMS; ++k) {
            const int i = base + (int)threadIdx.x * SCAN_ITEMS + k;
            if (i >= ntiles) break;
            const unsigned long long e = carry + v[k];
            sl.prefix[i] = (int)(e >> 32);
            sl.rowbase[i] = (int)(unsigned)e;
        }
        carry += tot;
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        const unsigned items = (unsigned)(carry >> 32), rows = (unsigned)carry;
        if (rows > (unsigned)sl.max_rows || items > (unsigned)INT32_MAX) {
            /* cannot happen with the host's bound; run no item rather than
             * write past the partial rows */
            atomicOr(err, GEXS_KERR_SLICES);
            *sl.nitems = 0;
        } else {
            sl.prefix[ntiles] = (int)items;
            *sl.nitems = (int)items;
        }
    }
}

/* int of the counter block that the set-up kernel's plan blocks count in */
constexpr int SETUP_COUNTER = 16;

/* blocks [0, nplan): eight tiles each; then per_job blocks a job for prep */
__global__ void __launch_bounds__(SETUP_NT) setup_kernel(const KArgs a, int nplan, int per_job)
{
    __shared__ SetupScan::TempStorage tmp;
    __shared__ int s_last;
    if ((int)blockIdx.x >= nplan) {
        const int b = (int)blockIdx.x - nplan, j = b / per_job;
        prep_lines(a.jobs[j], a.prep[j], (int64_t)(b % per_job) * SETUP_NT + threadIdx.x,
                   (int64_t)per_job * SETUP_NT);
        return;
    }
    const int lane = threadIdx.x & 31;
    const int ti = blockIdx.x * (SETUP_NT / 32) + (threadIdx.x >> 5);
    if (ti < a.nitems) {
        int tj = 0;
        const gexs_job& J = a.jobs[tile_job(a, ti, &tj)];
        if (a.sl.prefix) plan_tile(a, J, ti, tj, lane);
        if (a.csl.prefix) {
            const int64_t t0 = J.start_idx + (int64_t)tj * a.tile_w;
            const int64_t tend = min((int64_t)(t0 + a.tile_w), J.start_idx + J.n_points);
            const int ns = core_subtiles(a.tile_w);
            for (int k = 0; k < ns; ++k)
                plan_core_tile(a, J, ti * ns + k, t0 + (int64_t)k * CORE_W, tend, lane);
        }
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(a.counter + SETUP_COUNTER, 1) == nplan - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (a.sl.prefix) scan_slices(a.sl, a.nitems, a.err, tmp);
    __syncthreads();
    if (a.csl.prefix) scan_slices(a.csl, a.nitems * core_subtiles(a.tile_w), a.err, tmp);
}
}  // namespace

/* max_lines: the longest list of the launch's jobs when they have prep
 * arrays, else 0 */
static cudaError_t launch_setup(const KArgs& a, int64_t max_lines, int nsm, cudaStream_t st)
{
    const bool plan = (a.sl.prefix || a.csl.prefix) && a.nitems > 0;
    const int nplan = plan ? (a.nitems + SETUP_NT / 32 - 1) / (SETUP_NT / 32) : 0;
    const int per_job = a.prep && max_lines > 0
                            ? (int)std::min<int64_t>((max_lines + SETUP_NT - 1) / SETUP_NT, (int64_t)nsm * 8)
                            : 0;
    const int64_t blocks = nplan + (int64_t)per_job * a.njobs;
    if (blocks == 0) return cudaSuccess;
    if (blocks > INT32_MAX) return cudaErrorInvalidValue;
    setup_kernel<<<(unsigned)blocks, SETUP_NT, 0, st>>>(a, nplan, per_job > 0 ? per_job : 1);
    return cudaGetLastError();
}

cudaError_t launch_tiles(int pk, int prec, const gexs_job* d_jobs, const int* d_prefix,
                         int njobs, int nitems, int* d_counter, int* d_err,
                         double* const* d_prep, const gexs_launch_cfg& cfg, int nsm,
                         cudaStream_t st, const SliceTables* sl, const SliceTables* csl,
                         const int* d_order, int64_t prep_lines, cudaEvent_t tiles_after)
{
    KArgs a;
    a.jobs = d_jobs; a.prefix = d_prefix; a.njobs = njobs; a.nitems = nitems;
    a.order = njobs > 1 ? d_order : nullptr;
    a.counter = d_counter; a.err = d_err; a.prep = d_prep;
    a.tile_w = tile_bins(cfg);
    a.row0 = 0;
    a.subs = 1;
    a.spin = cfg.wait_spins > 0 ? cfg.wait_spins : WS_SPIN;
    std::memset(&a.sl, 0, sizeof(a.sl));
    std::memset(&a.csl, 0, sizeof(a.csl));
    if (sl && slices_apply(pk, prec)) a.sl = *sl;
    if (csl && core_slices_apply(pk, prec, a.tile_w)) a.csl = *csl;
    cudaError_t e = launch_setup(a, prep_lines, nsm, st);
    if (e == cudaSuccess && tiles_after) e = cudaStreamWaitEvent(st, tiles_after, 0);
    if (e != cudaSuccess) return e;
    switch (pk) {
    case PK_VOIGT: return launch_tiles_voigt(prec, a, cfg, nsm, st);
    case PK_ERF:   return launch_tiles_erf(prec, a, cfg, nsm, st);
    case PK_GH16:  return launch_tiles_gh16(prec, a, cfg, nsm, st);
    case PK_GH32:  return launch_tiles_gh32(prec, a, cfg, nsm, st);
    }
    return cudaErrorInvalidValue;
}

bool slices_apply(int pk, int prec) { return !(pk == PK_ERF && prec == GEXS_FP64); }

bool core_slices_apply(int pk, int prec, int tile_w)
{
    return (pk == PK_VOIGT || (pk == PK_ERF && prec == GEXS_FP64)) &&
           (tile_w <= CORE_W || prec == GEXS_FP64);
}

/* A split tile of n lines has ceil(n / per) <= n / per + 1 slices, so for m
 * line entries in all of a job's tiles the slices of split tiles number at
 * most m / per + (split tiles), and a split tile holds more than per. */
static double row_bound(const gexs_job& j, double m, int tile_w, double per)
{
    const double tiles = std::ceil((double)j.n_points / (double)tile_w);
    return std::ceil(m / per) + std::min(tiles, std::floor(m / per));
}

/* a line lies in at most (2 (reach + margin)) / (tile width) + 2 tiles */
static double tile_entries(const gexs_job& j, double reach, int tile_w)
{
    const double tpl = std::floor((2.0 * reach + 8.0 * j.dnu) / ((double)tile_w * j.dnu)) + 3.0;
    return (double)j.lines.count * tpl;
}

static const double kMaxRowBytes = (double)ROW_BYTES;

/* reach_range's reach at the job's highest frequency */
static double scatter_reach(const gexs_job& j)
{
    const double z = j.profile == GEXS_VOIGT ? 15.0 : ERF_Z64, k = z * j.dop_coef;
    const double nu_hi = j.nu_start + (double)(j.start_idx + j.n_points) * j.dnu + j.cutoff;
    double reach = j.cutoff;
    if (j.profile == GEXS_GAUSSIAN) reach = std::min(reach, z / j.inv_width);
    else if (k < 1.0) reach = std::min(reach, (nu_hi + j.dnu) * k / (1.0 - k));
    return reach;
}

bool erf_split(const gexs_job* jobs, int njobs, int tile_w)
{
    /* a part repeats its tile's item set-up and some of its lines: worth it
     * where tiles are dense, or few and not nearly empty */
    double lines = 0.0, tiles = 0.0;
    for (int i = 0; i < njobs; ++i) {
        lines += tile_entries(jobs[i], scatter_reach(jobs[i]), tile_w);
        tiles += std::ceil((double)jobs[i].n_points / (double)tile_w);
    }
    return tiles < 1e8 && lines >= (tiles < 1184.0 ? 128.0 : 1024.0) * tiles;
}

bool ws_split(const gexs_job* jobs, int njobs, int tile_w)
{
    /* a quarter takes about 0.4 of a whole tile's time: worth it while the
     * whole tiles' items (about one per tile and 16384 lines) are fewer than
     * 1.5 per SM (manager segments of 300 to 500 items, which share the chip:
     * 14.7 against 13.7 ms with quarters), and a tile holds more than a few
     * lines */
    double lines = 0.0, tiles = 0.0;
    for (int i = 0; i < njobs; ++i) {
        lines += tile_entries(jobs[i], jobs[i].cutoff, tile_w);
        tiles += std::ceil((double)jobs[i].n_points / (double)tile_w);
    }
    return tiles + lines / 16384.0 < 222.0 && lines >= 64.0 * tiles;
}

bool core_rows(const gexs_job* jobs, int njobs, int prec, int tile_w, CoreRows* out)
{
    double total = 0.0;
    long long most = 1;
    for (int i = 0; i < njobs; ++i) {
        const gexs_job& j = jobs[i];
        const double tiles = std::ceil((double)j.n_points / (double)tile_w);
        /* reach_range's margins hold 2e-9 of the frequency as well */
        const double nu_hi = j.nu_start + (double)(j.start_idx + j.n_points) * j.dnu + j.cutoff;
        const double reach = scatter_reach(j) + 2e-9 * (std::fabs(nu_hi) + j.cutoff);
        const double m = std::min(tile_entries(j, reach, tile_w), (double)j.lines.count * tiles);
        const long long cap = core_max_slices(j.grid_points, tile_w, prec);
        if (cap < 2) continue;
        total += std::min(row_bound(j, m, tile_w, (double)core_cut(j.grid_points, tile_w)),
                          tiles * (double)cap);
        most = std::max(most, cap);
    }
    if (!(total < (double)INT32_MAX)) return false;
    const long long fit = ROW_BYTES / ((long long)sizeof(double) * row_doubles(prec, tile_w));
    out->bound = (int)total;
    /* never more than the jobs would take one by one */
    out->round_rows = total <= (double)(fit + most) ? 0 : (int)fit;
    out->alloc = out->round_rows ? (int)(fit + most) : out->bound;
    return true;
}

long long slice_lines(const gexs_job* jobs, int njobs, int prec, int tile_w, int* max_rows)
{
    /* FP32: slices of 16384 lines, more when the rows of split tiles, fewer
     * than 2 m / per, could pass 1 GiB.  Measured on one B200: the 1e8-line
     * workload is indifferent to 16k-128k, a dense band of 1e6 lines in 80
     * cm^-1 runs 25% faster than at 65536.
     * FP64 (any cut gives the same sums): about eight items for each of the
     * 740 (Voigt, 4 x 4) to 444 (quadrature, 4 x 8) CTAs that fit, of 512 to
     * 4096 lines.  Uncut, 2e5 lines on 194 tiles (GH32) took four times as
     * long. */
    double m = 0.0;
    for (int i = 0; i < njobs; ++i) m += tile_entries(jobs[i], jobs[i].cutoff, tile_w);
    long long per = 16384;
    if (prec == GEXS_FP64)
        for (per = 512; per < 4096 && (double)per * (8 * 888) < m; ) per *= 2;
    for (;; per *= 2) {
        double rows = 0.0, need = 0.0;
        for (int i = 0; i < njobs; ++i) {
            const double mi = tile_entries(jobs[i], jobs[i].cutoff, tile_w);
            rows += 2.0 * std::ceil(mi / (double)per);
            need += row_bound(jobs[i], mi, tile_w, (double)per);
        }
        if ((prec == GEXS_FP64 ? need : rows) * row_doubles(prec, tile_w) * sizeof(double) <= kMaxRowBytes) {
            *max_rows = (int)std::min(rows, need);
            return per;
        }
        if (per >= (1ll << 40)) { *max_rows = 0; return 1ll << 62; }
    }
}

/* ----------------------------------------------- control writes as kernels */
namespace {
const int kBlobBytes = 4000;                /* under the 4 KB kernel-parameter limit */
struct Blob { unsigned char b[kBlobBytes]; };

__global__ void put_blob_kernel(const Blob p, unsigned char* dst, int n)
{
    for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = p.b[i];
}

__global__ void zero_ints_kernel(int* p, int n)
{
    for (int i = threadIdx.x; i < n; i += blockDim.x) p[i] = 0;
}

__global__ void take_word_kernel(int* word, int* out)
{
    *out = atomicExch(word, 0);
}
}  // namespace

cudaError_t take_word(int* word, int* out, cudaStream_t st)
{
    take_word_kernel<<<1, 1, 0, st>>>(word, out);
    return cudaGetLastError();
}

cudaError_t put_bytes(void* dst, const void* src, size_t n, cudaStream_t st)
{
    if (n > kMaxParamUpload) return cudaMemcpyAsync(dst, src, n, cudaMemcpyHostToDevice, st);
    const unsigned char* s = static_cast<const unsigned char*>(src);
    unsigned char* d = static_cast<unsigned char*>(dst);
    for (size_t o = 0; o < n; o += kBlobBytes) {
        const int k = (int)std::min<size_t>(kBlobBytes, n - o);
        Blob b;
        std::memcpy(b.b, s + o, (size_t)k);
        put_blob_kernel<<<1, 256, 0, st>>>(b, d + o, k);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

cudaError_t zero_ints(int* p, int n, cudaStream_t st)
{
    zero_ints_kernel<<<1, 64, 0, st>>>(p, n);
    return cudaGetLastError();
}

cudaError_t launch_count(const gexs_job* d_jobs, int njobs, unsigned long long* d_counts,
                         int nsm, cudaStream_t st)
{
    dim3 grid(nsm * 4, njobs);
    count_kernel<<<grid, 256, 0, st>>>(d_jobs, d_counts);
    return cudaGetLastError();
}

cudaError_t launch_partition(const double* d_e, const int32_t* d_g, int64_t n,
                             const double* d_betas, int nt, double* d_partial, int nchunk,
                             double* d_q, cudaStream_t st)
{
    dim3 grid(nchunk, nt);
    partition_partial<<<grid, 256, 0, st>>>(d_e, d_g, n, d_betas, d_partial);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    partition_final<<<(nt + 127) / 128, 128, 0, st>>>(d_partial, nchunk, nt, d_q);
    return cudaGetLastError();
}

}  // namespace gexs
