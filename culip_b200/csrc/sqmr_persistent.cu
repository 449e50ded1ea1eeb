// Host side of the persistent SQMR solver (sqmr_persistent.cuh): workspaces,
// launches and results of the whole-grid, batched and many-system solves.
#include "sqmr_persistent.cuh"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdlib>
#include <memory>

namespace culipx {

using namespace persistent;

namespace {

// kernel arguments over a work area of kVecs n nr doubles + 8 nr (vectors, then out)
template <class TF>
PArgs<TF> make_args(Csr* A, Factor* M, double* base, double* partials, const double* b, double* x, double tol,
                    int max_it, int nr = 1)
{
    Pattern& p = *M->pat;
    const int n = A->m;
    PArgs<TF> a;
    a.n = n;
    a.nl = p.num_levels;
    a.max_it = max_it;
    a.fuse_l0 = (p.l0_diagonal && A->nnz == p.nnz && A->m == p.n) ? 1 : 0;
    a.tol = tol;
    a.rowptr = A->rowptr;
    a.colidx = A->colidx;
    a.kval = static_cast<const double*>(A->val);
    a.pk_col = M->pk_col.as<TF>();
    a.pk_row = M->pk_row.as<TF>();
    a.pk_off = M->pk_off.as<long long>();
    a.ndmask = M->ndmask.as<unsigned>();
    a.dg = M->dg.as<TF>();
    a.tri = M->tri.as<TF>();
    a.is_piv = M->is_piv.as<int>();
    a.perm = M->perm.as<int>();
    a.lvl_off = p.d_lvl_off.as<int>();
    a.lvl_rows = p.d_lvl_rows.as<int>();
    a.bs = p.d_bs.as<int>();
    a.u_rng = M->u_rng.as<int2>();
    a.u_colp = M->u_colp.as<int>();
    a.u_val = M->u_val.as<TF>();
    a.ut_rng = M->ut_rng.as<int2>();
    a.ut_col = M->ut_col.as<int>();
    a.ut_val = M->ut_val.as<TF>();
    a.rowflags = M->rowflags.as<int>();
    a.scan_s = M->scan_s.as<int>();
    a.scan_c = M->scan_c.as<int>();
    a.simple_rows = M->simple_rows.as<int>();
    a.cplx = M->cplx.as<int>();
    a.citem = M->citem.as<CItem>();
    const size_t vn = (size_t)n * nr;
    // the vectors that a solve reads before it writes them stand last (zero_vectors)
    a.v[0] = base;
    a.Av = base + vn;
    a.ev = base + 2 * vn;
    a.v[1] = base + 3 * vn;
    for (int i = 0; i < 2; ++i) a.p[i] = base + (size_t)(4 + i) * vn;
    a.xt = base + 6 * vn;
    a.out = base + (size_t)kVecs * vn;
    a.partials = partials;
    a.ts = nullptr;
    a.lvl_done = nullptr;
    a.wait_skew = 0;
    a.count_red = 0;
    a.red_skew = 0;
    a.x = x;
    a.b = b;
    return a;
}

// Whether the reductions of a fused two-level solve on G CTAs may use the
// counted barrier, whose wait is bounded (kWaitLimitNs, 200 ms).  They wait
// for the slowest thread of a phase; a thread walks a row of K and its run of
// U' serially.  At most kCountedSerial entries to a thread, each at most twice
// in a phase and each walk at most 1 us an entry (two dependent trips to
// memory for two entries with four right-hand sides), is 33 ms.  Longer rows
// (a dense constraint, say) keep grid.sync, which waits as long as they take:
// next to such a phase the 0.5 us that the counted barrier saves are nothing.
constexpr long long kCountedSerial = 16384;

bool reductions_counted(const Pattern& p, int G)
{
    if (p.num_levels != 2) return false;
    const long long items = p.lvl_off[2] - p.lvl_off[1];
    const long long rows = items / ((long long)G * kW) + p.n / ((long long)G * kT) + 2;  // of one thread
    return rows * p.longest_row <= kCountedSerial;
}

int ctas_per_sm()
{
    static int c = [] {
        const char* e = getenv("CULIPX_SQMR_CTAS");
        return (e && atoi(e) == 1) ? 1 : kCtasPerSm;
    }();
    return c;
}

template <class TF, int NR>
const void* persistent_kernel()
{
    return ctas_per_sm() == 1 ? persistent_fn<TF, 1, NR>() : persistent_fn<TF, 2, NR>();
}

// resident CTAs for the cooperative launch
template <class TF, int NR>
int persistent_grid(int dev, int* G)
{
    int per_sm = 0, sms = 0;
    CULIPX_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    // the resident item slots need more than the default 48 KB of dynamic shared memory
    CULIPX_CUDA(cudaFuncSetAttribute(persistent_kernel<TF, NR>(), cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)res_smem_bytes<TF>()));
    CULIPX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, persistent_kernel<TF, NR>(), kT,
                                                              res_smem_bytes<TF>()));
    if (per_sm < 1) return fail(CULIPX_NOT_SUPPORTED, "persistent SQMR kernel does not fit on an SM");
    *G = sms * std::min(per_sm, ctas_per_sm());
    return CULIPX_OK;
}

// Grid sizes depend on the device (SM count, occupancy), so each launch
// site keeps one entry per device of the current process.  Entries are
// written at most once with the same value, so concurrent first calls from
// several host threads at worst compute the size twice.
constexpr int kMaxDevices = 64;

struct DeviceGridCache {
    std::atomic<int> g[kMaxDevices];
};

// *G = the cached grid for the current device, computed by size(dev, &g) once
template <class SizeFn>
int cached_grid(DeviceGridCache& c, SizeFn size, int* G, int* dev_out = nullptr)
{
    int dev = 0;
    CULIPX_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= kMaxDevices) return fail(CULIPX_NOT_SUPPORTED, "device %d beyond %d devices", dev, kMaxDevices);
    int g = c.g[dev].load(std::memory_order_acquire);
    if (g == 0) {
        CULIPX_TRY(size(dev, &g));
        c.g[dev].store(g, std::memory_order_release);
    }
    *G = g;
    if (dev_out) *dev_out = dev;
    return CULIPX_OK;
}

// v_-1, p_-1, p_-2 and the iterate start at zero; everything else is written
// before it is read, the caller's x among it
template <class TF>
int zero_vectors(const PArgs<TF>& a, int nr, cudaStream_t s)
{
    CULIPX_CUDA(cudaMemsetAsync(a.v[1], 0, (size_t)4 * a.n * nr * sizeof(double), s));
    return CULIPX_OK;
}

// launch and wait; out_host receives 8 values per right-hand side
template <class TF, int NR>
int run_persistent(culipx_handle_t* h, PArgs<TF>& a, int G, double* out_host, bool wait = true)
{
    cudaStream_t s = h->stream;
    CULIPX_TRY(zero_vectors(a, NR, s));
    void* args[] = {&a};
    CULIPX_CUDA(cudaLaunchCooperativeKernel(persistent_kernel<TF, NR>(), dim3(G), dim3(kT), args,
                                            res_smem_bytes<TF>(), s));
    h->launches += 1;
    CULIPX_CUDA(cudaMemcpyAsync(out_host, a.out, (size_t)8 * NR * sizeof(double), cudaMemcpyDeviceToHost, s));
    if (wait) CULIPX_CUDA(cudaStreamSynchronize(s));
    return CULIPX_OK;
}

template <class TF, int NR>
int launch_persistent(culipx_handle_t* h, Csr* A, Factor* M, const double* b, double* x, double tol, int max_it,
                      Sqmr* w, double* out_host, bool wait = true)
{
    const int n = A->m;
    cudaStream_t s = h->stream;
    const size_t need = ((size_t)kVecs * n * NR + 8 * NR + 64) * sizeof(double);
    if (w->vecs.bytes() < need) {
        CULIPX_TRY(w->vecs.alloc(h, need));
        w->n = -1;  // the single-RHS workspace size is no longer known
    }
    static DeviceGridCache grid_cache;  // one per <TF, NR> instantiation
    int G = 0;
    CULIPX_TRY(cached_grid(grid_cache, persistent_grid<TF, NR>, &G));
    if ((size_t)(2 * kMaxNV * G) * sizeof(double) > w->partials.bytes())
        CULIPX_TRY(w->partials.alloc(h, (size_t)2 * kMaxNV * G * sizeof(double)));
    PArgs<TF> a = make_args<TF>(A, M, w->vecs.as<double>(), w->partials.as<double>(), b, x, tol, max_it, NR);
    // the level counter in the spare slots after the results (need: 8 NR + 64 values)
    a.lvl_done = reinterpret_cast<unsigned long long*>(a.out + 8 * kMaxNR);
    a.wait_skew = w->wait_skew;
    a.count_red = reductions_counted(*M->pat, G);
    a.red_skew = w->red_skew;
    if (w->profile && NR == 1) {
        if (w->ts.bytes() < (size_t)kTsIters * 8 * sizeof(unsigned long long))
            CULIPX_TRY(w->ts.alloc(h, (size_t)kTsIters * 8 * sizeof(unsigned long long)));
        CULIPX_CUDA(cudaMemsetAsync(w->ts.get(), 0, (size_t)kTsIters * 8 * sizeof(unsigned long long), s));
        a.ts = w->ts.as<unsigned long long>();
    }
    return run_persistent<TF, NR>(h, a, G, out_host, wait);
}

template <class TF>
int launch_nr(int nr, culipx_handle_t* h, Csr* A, Factor* M, const double* b, double* x, double tol, int max_it,
              Sqmr* w, double* out_host)
{
    switch (nr) {
    case 1: return launch_persistent<TF, 1>(h, A, M, b, x, tol, max_it, w, out_host);
    case 2: return launch_persistent<TF, 2>(h, A, M, b, x, tol, max_it, w, out_host);
    default: return launch_persistent<TF, 4>(h, A, M, b, x, tol, max_it, w, out_host);
    }
}

int status_of(const double* o, int max_it)
{
    if (o[6] != 0.0) return fail(CULIPX_TIMEOUT, "persistent SQMR: a bounded device wait gave up (results invalid)");
    if (o[2] != 0.0) return CULIPX_BREAKDOWN;
    if (o[3] == 0.0 && max_it > 0 && (int)o[1] >= max_it) return CULIPX_MAXIT;
    return CULIPX_OK;
}

}  // namespace

// nrhs right-hand sides (column-major n x nrhs) in launches of up to
// kMaxNR at a time; per right-hand side the quasi-residual, iterations and
// status (OK / MAXIT / BREAKDOWN)
int sqmr_solve_multi(culipx_handle_t* h, Csr* A, Factor* M, int nrhs, const double* B, double* X, double tol,
                     int max_it, double* h_res, int* h_its, int* h_status, Sqmr* w)
{
    if (!A || !M || !B || !X || !w || nrhs < 1) return fail(CULIPX_INVALID_ARG, "culipx_sqmr_solve_multi: bad argument");
    if (A->precision != CULIPX_F64 || A->m != A->n || !M->computed || M->pat->n != A->m)
        return fail(CULIPX_INVALID_ARG, "culipx_sqmr_solve_multi: A must be square FP64 and M its computed factor");
    if (M->solve_algorithm == CULIPX_SOLVE_JACOBI)
        return fail(CULIPX_NOT_SUPPORTED, "culipx_sqmr_solve_multi: SOLVE_JACOBI needs culipx_sqmr_solve");
    if (max_it < 0) return fail(CULIPX_INVALID_ARG, "culipx_sqmr_solve_multi: max_it < 0");
    const size_t n = A->m;
    double out[8 * kMaxNR];
    for (int r0 = 0; r0 < nrhs; r0 += kMaxNR) {
        const int nr = std::min(kMaxNR, nrhs - r0);
        // 3 right-hand sides run as 4, the fourth a copy of the third: it stops
        // when the third does and its x is dropped
        const int nl = (nr == 1) ? 1 : (nr == 2) ? 2 : 4;
        const double* b = B + r0 * n;
        double* x = X + r0 * n;
        DeviceBuffer pad_b, pad_x;
        if (nl != nr) {
            CULIPX_TRY(pad_b.alloc(h, nl * n * sizeof(double)));
            CULIPX_TRY(pad_x.alloc(h, nl * n * sizeof(double)));
            CULIPX_CUDA(cudaMemcpyAsync(pad_b.get(), b, nr * n * sizeof(double), cudaMemcpyDeviceToDevice, h->stream));
            CULIPX_CUDA(cudaMemcpyAsync(pad_b.as<double>() + nr * n, b + (nr - 1) * n, n * sizeof(double),
                                        cudaMemcpyDeviceToDevice, h->stream));
            b = pad_b.as<double>();
            x = pad_x.as<double>();
        }
        const int st = (M->precision == CULIPX_F64) ? launch_nr<double>(nl, h, A, M, b, x, tol, max_it, w, out)
                                                    : launch_nr<float>(nl, h, A, M, b, x, tol, max_it, w, out);
        if (st != CULIPX_OK) return st;
        if (nl != nr) {
            CULIPX_CUDA(cudaMemcpyAsync(X + r0 * n, x, nr * n * sizeof(double), cudaMemcpyDeviceToDevice, h->stream));
            CULIPX_CUDA(cudaStreamSynchronize(h->stream));
        }
        for (int j = 0; j < nr; ++j) {
            const double* o = out + 8 * j;
            if (h_res) h_res[r0 + j] = o[0];
            if (h_its) h_its[r0 + j] = (int)o[1];
            if (h_status) h_status[r0 + j] = status_of(o, max_it);
        }
    }
    return CULIPX_OK;
}

// The right-hand sides of one system in groups of 4 (then 2 and 1: no
// padding, so nothing is allocated per call) enqueued on h's stream without
// waiting; right-hand side r's 8 result values go to out_host + 8 r (pinned
// memory for a truly asynchronous call).  Groups run one after another on
// the stream and share the workspace.
int sqmr_solve_multi_async(culipx_handle_t* h, Csr* A, Factor* M, int nrhs, const double* B, double* X, double tol,
                           int max_it, Sqmr* w, double* out_host)
{
    if (!A || !M || !B || !X || !w || !out_host || nrhs < 1)
        return fail(CULIPX_INVALID_ARG, "sqmr_solve_multi_async: bad argument");
    if (A->precision != CULIPX_F64 || A->m != A->n || !M->computed || M->pat->n != A->m)
        return fail(CULIPX_INVALID_ARG, "sqmr_solve_multi_async: A must be square FP64 and M its computed factor");
    const size_t n = A->m;
    const bool f64 = M->precision == CULIPX_F64;
    for (int r0 = 0; r0 < nrhs;) {
        const int rem = nrhs - r0;
        const int nr = rem >= 4 ? 4 : (rem >= 2 ? 2 : 1);
        const double* b = B + r0 * n;
        double* x = X + r0 * n;
        double* o = out_host + (size_t)8 * r0;
        int st;
        if (nr == 4)
            st = f64 ? launch_persistent<double, 4>(h, A, M, b, x, tol, max_it, w, o, false)
                     : launch_persistent<float, 4>(h, A, M, b, x, tol, max_it, w, o, false);
        else if (nr == 2)
            st = f64 ? launch_persistent<double, 2>(h, A, M, b, x, tol, max_it, w, o, false)
                     : launch_persistent<float, 2>(h, A, M, b, x, tol, max_it, w, o, false);
        else
            st = f64 ? launch_persistent<double, 1>(h, A, M, b, x, tol, max_it, w, o, false)
                     : launch_persistent<float, 1>(h, A, M, b, x, tol, max_it, w, o, false);
        if (st != CULIPX_OK) return st;
        r0 += nr;
    }
    return CULIPX_OK;
}

// ---------------------------------------------------------------------------
// Batched solves (no counterpart in the reference, which solves one system
// per SQMR object): systems given as consecutive row ranges of one
// block-diagonal union pattern.
namespace {

// The whole-grid solve (a two-level factor, A on its pattern).
template <class TF>
int launch_lockstep(Batch* bt, const PArgs<TF>& a, const BatchArgs& ba, int rest_grid, Sqmr* w)
{
    culipx_handle_t* h = bt->h;
    const size_t need = lockstep_bytes(a.n, bt->num);
    if (w->lock.bytes() < need) CULIPX_TRY(w->lock.alloc(h, need));
    static DeviceGridCache grid_cache;  // one per factor precision
    int G = 0;
    CULIPX_TRY(cached_grid(
        grid_cache,
        [](int dev, int* g) {
            int per_sm = 0, sms = 0;
            CULIPX_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
            CULIPX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, lockstep_kernel<TF>(), kT, 0));
            if (per_sm < 1) return fail(CULIPX_NOT_SUPPORTED, "lockstep SQMR kernel does not fit on an SM");
            *g = sms * std::min(per_sm, kCtasPerSm);
            return (int)CULIPX_OK;
        },
        &G));
    CULIPX_TRY(lockstep_launch<TF>(a, bt->lock, ba, w->lock.get(), G, rest_grid, h->stream));
    h->launches += 2;
    return CULIPX_OK;
}

template <class TF>
int launch_batched(Batch* bt, Csr* A, Factor* M, const double* b, double* x, double tol, int max_it, Sqmr* w)
{
    culipx_handle_t* h = bt->h;
    cudaStream_t s = h->stream;
    const int n = A->m;
    CULIPX_TRY(sqmr_workspace(w, h, n));
    static DeviceGridCache grid_cache;  // one per factor precision
    int G = 0;
    CULIPX_TRY(cached_grid(
        grid_cache,
        [](int dev, int* g) {
            int per_sm = 0, sms = 0;
            CULIPX_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
            CULIPX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, batched_fn<TF>(), kT, 0));
            if (per_sm < 1) return fail(CULIPX_NOT_SUPPORTED, "batched SQMR kernel does not fit on an SM");
            *g = sms * std::min(per_sm, kCtasPerSm);
            return (int)CULIPX_OK;
        },
        &G));
    PArgs<TF> a = make_args<TF>(A, M, w->vecs.as<double>(), w->partials.as<double>(), b, x, tol, max_it);
    BatchArgs ba;
    ba.num = bt->num;
    ba.row_off = bt->d_row_off.as<int>();
    ba.qb = bt->d_qb.as<int>();
    ba.qe = bt->d_qe.as<int>();
    ba.out = bt->d_out.as<double>();
    ba.next = bt->d_next.as<int>();
    CULIPX_TRY(zero_vectors(a, 1, s));
    // static pivots or a threshold leave a factor whose level 0 is not known to be simple
    if (bt->lock.use && M->two_level && a.fuse_l0) return launch_lockstep<TF>(bt, a, ba, std::min(G, bt->num), w);
    CULIPX_CUDA(cudaMemsetAsync(ba.next, 0, sizeof(int), s));
    void* args[] = {&a, &ba};
    CULIPX_CUDA(cudaLaunchKernel(batched_fn<TF>(), dim3(std::min(G, bt->num)), dim3(kT), args, 0, s));
    h->launches += 1;
    return CULIPX_OK;
}

}  // namespace

namespace {

// The work units of the whole-grid solve, where it gains.  One CTA per system
// lasts as long as its largest system: measured 25 + 17.5 per 1000 rows us an
// iteration (FP32 and FP64 alike, the device not full); the whole grid takes
// 60 for its synchronisations, 0.15 per 1000 rows of all systems and 2.4 per
// 1000 rows of the largest for its sums.  256 systems of 750 to 30 000 rows:
// 0.84 ms against 0.46; one system of 30 000 rows: 0.55 against 0.09; 296
// systems of 4500 rows: 0.20 against 0.29, which keep a CTA each.  Small systems
// that outlast the large ones get a CTA each from there on (k_sqmr_rest).  Both
// kernels give the same bits, so the choice does not show in the results.
int lockstep_plan(culipx_handle_t* h, const Pattern& p, int num, const int* row_off, const std::vector<int>& qb,
                  const std::vector<int>& qe, LockPlan& plan)
{
    int largest = 0;
    for (int s = 0; s < num; ++s) largest = std::max(largest, row_off[s + 1] - row_off[s]);
    plan.use = largest > kLockRows && 25.0 + 17.5e-3 * largest > 60.0 + 0.15e-3 * p.n + 2.4e-3 * largest;
    if (!plan.use) return CULIPX_OK;
    std::vector<int4> chunk, tile;
    int pos = 0;  // level 0's fine rows in level-list order
    for (int s = 0; s < num; ++s) {
        int rows = 0;
        for (int q = qb[2 * s]; q < qe[2 * s]; ++q) rows += p.bs[p.lvl_rows[q] + 1] - p.bs[p.lvl_rows[q]];
        for (int r = 0; r < rows; r += 32) chunk.push_back(make_int4(pos + r, std::min(32, rows - r), s, 0));
        pos += rows;
        for (int q = qb[2 * s + 1]; q < qe[2 * s + 1]; ++q) {
            const int I = p.lvl_rows[q];
            tile.push_back(make_int4(I, p.bs[I], p.bs[I + 1] - p.bs[I], s));
        }
    }
    plan.chunks = (int)chunk.size();
    plan.tiles = (int)tile.size();
    chunk.insert(chunk.end(), tile.begin(), tile.end());
    return plan.units.upload(h, chunk.data(), chunk.size() * sizeof(int4));
}

}  // namespace

int batch_create(culipx_handle_t* h, const Pattern* p, int num, const int* h_row_off, Batch** out)
{
    if (!p || !h_row_off || !out || num < 1) return fail(CULIPX_INVALID_ARG, "culipx_batch_create: bad argument");
    if (h_row_off[0] != 0 || h_row_off[num] != p->n)
        return fail(CULIPX_INVALID_ARG, "culipx_batch_create: row offsets must run from 0 to n");
    const int cm = p->num_blocks, nl = p->num_levels;
    // system of every block row; every system boundary must be a block boundary
    std::vector<int> sys(cm);
    int s = 0;
    for (int I = 0; I < cm; ++I) {
        while (s < num && h_row_off[s + 1] <= p->bs[I]) ++s;
        if (s >= num || h_row_off[s] > p->bs[I] || p->bs[I + 1] > h_row_off[s + 1])
            return fail(CULIPX_INVALID_ARG, "culipx_batch_create: a system boundary splits block row %d", I);
        sys[I] = s;
    }
    for (int k = 0; k < num; ++k)
        if (h_row_off[k + 1] <= h_row_off[k]) return fail(CULIPX_INVALID_ARG, "culipx_batch_create: empty system %d", k);
    // the systems must be independent: no block of the (filled) pattern couples two of them
    for (int b = 0; b < p->coarse_nnz; ++b)
        if (sys[p->blk_row[b]] != sys[p->blk_col[b]])
            return fail(CULIPX_INVALID_ARG, "culipx_batch_create: block (%d, %d) couples systems %d and %d",
                        p->blk_row[b], p->blk_col[b], sys[p->blk_row[b]], sys[p->blk_col[b]]);
    // per system and level: its (contiguous) run in the level's ascending block list
    std::vector<int> qb((size_t)num * std::max(nl, 1), 0), qe((size_t)num * std::max(nl, 1), 0);
    for (int L = 0; L < nl; ++L)
        for (int q = p->lvl_off[L]; q < p->lvl_off[L + 1]; ++q) {
            const int k = sys[p->lvl_rows[q]];
            int& b0 = qb[(size_t)k * nl + L];
            int& e0 = qe[(size_t)k * nl + L];
            if (e0 == b0) b0 = q;
            else if (e0 != q) return fail(CULIPX_INVALID_ARG, "culipx_batch_create: level list not grouped by system");
            e0 = q + 1;
        }
    auto bt = std::make_unique<culipx_batch_t>();
    bt->h = h;
    bt->pat = p;
    bt->num = num;
    bt->nl = nl;
    bt->row_off.assign(h_row_off, h_row_off + num + 1);
    int st = bt->d_row_off.upload(h, h_row_off, (size_t)(num + 1) * sizeof(int));
    if (st == CULIPX_OK) st = bt->d_qb.upload(h, qb.data(), qb.size() * sizeof(int));
    if (st == CULIPX_OK) st = bt->d_qe.upload(h, qe.data(), qe.size() * sizeof(int));
    if (st == CULIPX_OK) st = bt->d_out.alloc(h, (size_t)num * 8 * sizeof(double));
    if (st == CULIPX_OK) st = bt->d_next.alloc(h, sizeof(int));
    if (st == CULIPX_OK && p->two_level) st = lockstep_plan(h, *p, num, h_row_off, qb, qe, bt->lock);
    if (st != CULIPX_OK) return st;
    *out = bt.release();
    return CULIPX_OK;
}

namespace {

// the batch's results (8 values per system) to per-system residual, iterations, status
int batch_results(Batch* bt, int max_it, double* h_res, int* h_its, int* h_status)
{
    std::vector<double> out((size_t)bt->num * 8);
    CULIPX_CUDA(cudaMemcpyAsync(out.data(), bt->d_out.get(), out.size() * sizeof(double), cudaMemcpyDeviceToHost,
                                bt->h->stream));
    CULIPX_CUDA(cudaStreamSynchronize(bt->h->stream));
    for (int k = 0; k < bt->num; ++k) {
        const double* o = out.data() + (size_t)k * 8;
        if (h_res) h_res[k] = o[0];
        if (h_its) h_its[k] = (int)o[1];
        if (h_status)
            h_status[k] = (o[2] != 0.0) ? CULIPX_BREAKDOWN
                          : (o[3] == 0.0 && max_it > 0 && (int)o[1] >= max_it) ? CULIPX_MAXIT
                                                                               : CULIPX_OK;
    }
    return CULIPX_OK;
}

int batch_check(Batch* bt, Csr* A, Factor* M, const double* b, double* x, int max_it, const char* what)
{
    if (!bt || !A || !M || !b || !x) return fail(CULIPX_INVALID_ARG, "%s: null argument", what);
    if (A->precision != CULIPX_F64 || A->m != A->n || A->m != bt->pat->n)
        return fail(CULIPX_INVALID_ARG, "%s: A must be the FP64 union matrix of the batch", what);
    if (M->pat != bt->pat) return fail(CULIPX_INVALID_ARG, "%s: M must be a factor of the batch's pattern", what);
    if (M->solve_algorithm == CULIPX_SOLVE_JACOBI) return fail(CULIPX_NOT_SUPPORTED, "%s: SOLVE_JACOBI is not batched", what);
    if (max_it < 0) return fail(CULIPX_INVALID_ARG, "%s: max_it < 0", what);
    return CULIPX_OK;
}

}  // namespace

Batch::~Batch()
{
    if (graph_exec) cudaGraphExecDestroy(graph_exec);
    if (graph) cudaGraphDestroy(graph);
    if (capture_stream) cudaStreamDestroy(capture_stream);
    delete gw;
}

// The numeric factorization of the union and the batched solve as one CUDA
// graph launch.  The first call for a given set of buffers (values, A, M, b,
// x) and settings factors and solves by ordinary launches -- which sizes
// every buffer, the batch's own solver workspace included -- and captures
// the same sequence on a stream of the batch's own; later calls replay it
// (the contents of the buffers may change in between).
int batch_factor_solve_graph(Batch* bt, Csr* A, Factor* M, const void* d_vals, int pivot, double threshold,
                             const double* b, double* x, double tol, int max_it, double* h_res, int* h_its,
                             int* h_status)
{
    CULIPX_TRY(batch_check(bt, A, M, b, x, max_it, "culipx_batch_factor_solve_graph"));
    if (!d_vals) return fail(CULIPX_INVALID_ARG, "culipx_batch_factor_solve_graph: null values");
    if (pivot < CULIPX_PIV_STATIC || pivot > CULIPX_PIV_ROOK)
        return fail(CULIPX_INVALID_ARG, "culipx_batch_factor_solve_graph: bad pivot method %d", pivot);
    culipx_handle_t* h = bt->h;
    if (!bt->gw) bt->gw = new Sqmr();
    Batch::Key key;
    key.vals = d_vals;
    key.A = A->serial;
    key.M = M->serial;
    key.b = b;
    key.x = x;
    key.pivot = pivot;
    key.max_it = max_it;
    key.threshold = threshold;
    key.tol = tol;
    key.piv64 = M->pivot_fp64;
    auto solve = [&]() -> int {
        return (M->precision == CULIPX_F64) ? launch_batched<double>(bt, A, M, b, x, tol, max_it, bt->gw)
                                            : launch_batched<float>(bt, A, M, b, x, tol, max_it, bt->gw);
    };
    if (!bt->graph_exec || !(bt->graph_key == key)) {
        CULIPX_TRY(factor_compute(M, d_vals, nullptr, pivot, threshold));
        CULIPX_TRY(solve());
        CULIPX_TRY(batch_results(bt, max_it, h_res, h_its, h_status));
        if (bt->graph_exec) cudaGraphExecDestroy(bt->graph_exec);
        if (bt->graph) cudaGraphDestroy(bt->graph);
        bt->graph_exec = nullptr;
        bt->graph = nullptr;
        if (!bt->capture_stream) CULIPX_CUDA(cudaStreamCreateWithFlags(&bt->capture_stream, cudaStreamNonBlocking));
        cudaStream_t s = h->stream;
        const long long launches0 = h->launches;
        CULIPX_CUDA(cudaStreamBeginCapture(bt->capture_stream, cudaStreamCaptureModeThreadLocal));
        h->stream = bt->capture_stream;
        M->capturing = true;
        int st = factor_compute(M, d_vals, nullptr, pivot, threshold);
        if (st == CULIPX_OK) st = solve();
        M->capturing = false;
        h->stream = s;
        bt->graph_launches = (int)(h->launches - launches0);
        h->launches = launches0;  // captured, not launched
        cudaGraph_t g = nullptr;
        const cudaError_t e = cudaStreamEndCapture(bt->capture_stream, &g);
        if (st != CULIPX_OK || e != cudaSuccess) {
            if (g) cudaGraphDestroy(g);
            cudaGetLastError();
            return st != CULIPX_OK ? st
                                   : fail(CULIPX_CUDA_ERROR, "culipx_batch_factor_solve_graph: capture failed: %s",
                                          cudaGetErrorString(e));
        }
        cudaGraphExec_t ge = nullptr;
        if (cudaGraphInstantiate(&ge, g, 0) != cudaSuccess) {
            cudaGraphDestroy(g);
            cudaGetLastError();
            return fail(CULIPX_CUDA_ERROR, "culipx_batch_factor_solve_graph: graph instantiation failed");
        }
        bt->graph = g;
        bt->graph_exec = ge;
        bt->graph_key = key;
        return CULIPX_OK;  // the ordinary run above factored and solved
    }
    CULIPX_CUDA(cudaGraphLaunch(bt->graph_exec, h->stream));
    h->launches += bt->graph_launches;
    M->pivot = pivot;
    M->threshold = threshold;
    M->two_level = M->pat->two_level && pivot != CULIPX_PIV_STATIC && threshold == 0.0;
    M->computed = true;
    return batch_results(bt, max_it, h_res, h_its, h_status);
}

int batch_sqmr_solve(Batch* bt, Csr* A, Factor* M, const double* b, double* x, double tol, int max_it,
                     double* h_res, int* h_its, int* h_status, Sqmr* w)
{
    if (!bt || !A || !M || !b || !x || !w) return fail(CULIPX_INVALID_ARG, "culipx_batch_sqmr_solve: null argument");
    if (A->precision != CULIPX_F64 || A->m != A->n || A->m != bt->pat->n)
        return fail(CULIPX_INVALID_ARG, "culipx_batch_sqmr_solve: A must be the FP64 union matrix of the batch");
    if (!M->computed || M->pat != bt->pat)
        return fail(CULIPX_INVALID_ARG, "culipx_batch_sqmr_solve: M must be a computed factor of the batch's pattern");
    if (M->solve_algorithm == CULIPX_SOLVE_JACOBI)
        return fail(CULIPX_NOT_SUPPORTED, "culipx_batch_sqmr_solve: SOLVE_JACOBI is not batched");
    if (max_it < 0) return fail(CULIPX_INVALID_ARG, "culipx_batch_sqmr_solve: max_it < 0");
    const int st = (M->precision == CULIPX_F64) ? launch_batched<double>(bt, A, M, b, x, tol, max_it, w)
                                                : launch_batched<float>(bt, A, M, b, x, tol, max_it, w);
    if (st != CULIPX_OK) return st;
    std::vector<double> out((size_t)bt->num * 8);
    CULIPX_CUDA(cudaMemcpyAsync(out.data(), bt->d_out.get(), out.size() * sizeof(double), cudaMemcpyDeviceToHost,
                                bt->h->stream));
    CULIPX_CUDA(cudaStreamSynchronize(bt->h->stream));
    for (int k = 0; k < bt->num; ++k) {
        const double* o = out.data() + (size_t)k * 8;
        if (h_res) h_res[k] = o[0];
        if (h_its) h_its[k] = (int)o[1];
        if (h_status)
            h_status[k] = (o[2] != 0.0) ? CULIPX_BREAKDOWN
                          : (o[3] == 0.0 && max_it > 0 && (int)o[1] >= max_it) ? CULIPX_MAXIT
                                                                               : CULIPX_OK;
    }
    return CULIPX_OK;
}

namespace {

// Enqueues one launch per (factor precision, right-hand sides per system)
// group on h's stream.  System k solves nr[k] (1, 2 or 4) right-hand sides,
// b[k] / x[k] each n x nr[k] column-major; its results (8 values per
// right-hand side) go to out_host + 8 (nr[0] + ... + nr[k-1]) (pinned
// memory for a truly asynchronous call).  One workspace allocation serves
// every group.
// every system's work area starts on a 256-byte boundary: with NR even the
// kernel reads the interleaved vectors with 16-byte loads
double* align256(double* p)
{
    return reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(p) + 255) & ~static_cast<uintptr_t>(255));
}

template <class TF>
int launch_many_prec(culipx_handle_t* h, const std::vector<int>& ks, const int* nr, Csr* const* A, Factor* const* M,
                     const double* const* b, double* const* x, const std::vector<size_t>& slot, double tol,
                     int max_it, double*& base, double* out_host)
{
    cudaStream_t s = h->stream;
    const int num = (int)ks.size();
    std::vector<PArgs<TF>> args(num);
    std::vector<int> nrs(num);
    for (int i = 0; i < num; ++i) {
        const int k = ks[i];
        const int r = nr ? nr[k] : 1;
        const size_t m = A[k]->m;
        base = align256(base);
        args[i] = make_args<TF>(A[k], M[k], base, nullptr, b[k], x[k], tol, max_it, r);
        base += (size_t)kVecs * m * r + 8 * r;
        nrs[i] = r;
        CULIPX_CUDA(cudaMemsetAsync(args[i].v[0], 0, (size_t)kVecs * m * r * sizeof(double), s));
        CULIPX_CUDA(cudaMemsetAsync(x[k], 0, m * r * sizeof(double), s));
    }
    // argument blocks after the vectors, then the right-hand-side counts and the counter
    base = align256(base);
    PArgs<TF>* d_args = reinterpret_cast<PArgs<TF>*>(base);
    int* d_nr = reinterpret_cast<int*>(d_args + num);
    int* d_next = d_nr + num;
    base = reinterpret_cast<double*>(d_args + num) + (num + 2) / 2 + 1;
    CULIPX_CUDA(cudaMemcpyAsync(d_args, args.data(), (size_t)num * sizeof(PArgs<TF>), cudaMemcpyHostToDevice, s));
    CULIPX_CUDA(cudaMemcpyAsync(d_nr, nrs.data(), (size_t)num * sizeof(int), cudaMemcpyHostToDevice, s));
    CULIPX_CUDA(cudaMemsetAsync(d_next, 0, sizeof(int), s));
    const bool multi = std::any_of(nrs.begin(), nrs.end(), [](int r) { return r != 1; });
    static DeviceGridCache grid_caches[2];  // single / multi right-hand-side variant, per factor precision
    auto many_grid = [](const void* kern) {
        return [kern](int dev, int* g) {
            int per_sm = 0, sms = 0;
            CULIPX_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
            CULIPX_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kT, 0));
            if (per_sm < 1) return fail(CULIPX_NOT_SUPPORTED, "batched SQMR kernel does not fit on an SM");
            *g = sms * std::min(per_sm, kCtasPerSm);
            return (int)CULIPX_OK;
        };
    };
    int G = 0;
    if (multi) CULIPX_TRY(cached_grid(grid_caches[1], many_grid(many_fn<TF, true>()), &G));
    else CULIPX_TRY(cached_grid(grid_caches[0], many_grid(many_fn<TF, false>()), &G));
    const PArgs<TF>* arg_sys = d_args;
    const int* arg_nr = d_nr;
    int arg_num = num;
    int* arg_next = d_next;
    void* kargs[] = {&arg_sys, &arg_nr, &arg_num, &arg_next};
    CULIPX_CUDA(cudaLaunchKernel(multi ? many_fn<TF, true>() : many_fn<TF, false>(), dim3(std::min(G, num)), dim3(kT),
                                 kargs, 0, s));
    h->launches += 1;
    for (int i = 0; i < num; ++i)
        CULIPX_CUDA(cudaMemcpyAsync(out_host + 8 * slot[ks[i]], args[i].out, (size_t)8 * nrs[i] * sizeof(double),
                                    cudaMemcpyDeviceToHost, s));
    return CULIPX_OK;
}

}  // namespace

int sqmr_solve_many_nr_async(culipx_handle_t* h, int num, Csr* const* A, Factor* const* M, const double* const* b,
                             double* const* x, const int* nr, double tol, int max_it, Sqmr* w, double* out_host)
{
    if (num == 0) return CULIPX_OK;
    // result slots in the caller's order; per factor precision one launch with
    // the systems longest first (rows x right-hand sides), so the CTAs that
    // take the last systems finish close together
    std::vector<size_t> slot(num);
    size_t total = 0, acc = 0;
    std::vector<int> groups[2];
    for (int k = 0; k < num; ++k) {
        const int r = nr ? nr[k] : 1;
        if (r != 1 && r != 2 && r != 4) return fail(CULIPX_INVALID_ARG, "sqmr_solve_many: nr must be 1, 2 or 4");
        slot[k] = acc;
        acc += r;
        total += (size_t)kVecs * A[k]->m * r + 8 * r + 32;  // + alignment
        groups[M[k]->precision == CULIPX_F64 ? 0 : 1].push_back(k);
    }
    size_t argbytes = 0;
    for (int p = 0; p < 2; ++p) {
        std::vector<int>& ks = groups[p];
        std::stable_sort(ks.begin(), ks.end(), [&](int a, int c) {
            return (long long)A[a]->m * (nr ? nr[a] : 1) > (long long)A[c]->m * (nr ? nr[c] : 1);
        });
        if (!ks.empty())
            argbytes += ks.size() * ((p == 0 ? sizeof(PArgs<double>) : sizeof(PArgs<float>)) + sizeof(int)) + 512;
    }
    const size_t need = total * sizeof(double) + argbytes + 256;
    if (w->many.bytes() < need) CULIPX_TRY(w->many.alloc(h, need));
    double* base = w->many.as<double>();
    if (!groups[0].empty())
        CULIPX_TRY(launch_many_prec<double>(h, groups[0], nr, A, M, b, x, slot, tol, max_it, base, out_host));
    if (!groups[1].empty())
        CULIPX_TRY(launch_many_prec<float>(h, groups[1], nr, A, M, b, x, slot, tol, max_it, base, out_host));
    return CULIPX_OK;
}

int sqmr_solve_many_async(culipx_handle_t* h, int num, Csr* const* A, Factor* const* M, const double* const* b,
                          double* const* x, double tol, int max_it, Sqmr* w, double* out_host)
{
    return sqmr_solve_many_nr_async(h, num, A, M, b, x, nullptr, tol, max_it, w, out_host);
}

void many_results(int num, int max_it, const double* out, double* h_res, int* h_its, int* h_status)
{
    for (int k = 0; k < num; ++k) {
        const double* o = out + (size_t)k * 8;
        if (h_res) h_res[k] = o[0];
        if (h_its) h_its[k] = (int)o[1];
        if (h_status)
            h_status[k] = (o[2] != 0.0) ? CULIPX_BREAKDOWN
                          : (o[3] == 0.0 && max_it > 0 && (int)o[1] >= max_it) ? CULIPX_MAXIT
                                                                               : CULIPX_OK;
    }
}

int sqmr_solve_many(culipx_handle_t* h, int num, Csr* const* A, Factor* const* M, const double* const* b,
                    double* const* x, double tol, int max_it, double* h_res, int* h_its, int* h_status, Sqmr* w)
{
    if (num < 0 || (num > 0 && (!A || !M || !b || !x)) || !w)
        return fail(CULIPX_INVALID_ARG, "culipx_sqmr_solve_many: bad argument");
    if (max_it < 0) return fail(CULIPX_INVALID_ARG, "culipx_sqmr_solve_many: max_it < 0");
    if (num == 0) return CULIPX_OK;
    const int prec = M[0] ? M[0]->precision : CULIPX_F64;
    for (int k = 0; k < num; ++k) {
        if (!A[k] || !M[k] || !b[k] || !x[k]) return fail(CULIPX_INVALID_ARG, "culipx_sqmr_solve_many: null system %d", k);
        if (A[k]->precision != CULIPX_F64 || A[k]->m != A[k]->n || !M[k]->computed || M[k]->pat->n != A[k]->m)
            return fail(CULIPX_INVALID_ARG, "culipx_sqmr_solve_many: system %d: A must be square FP64 and M its computed factor", k);
        if (M[k]->precision != prec)
            return fail(CULIPX_NOT_SUPPORTED, "culipx_sqmr_solve_many: all factors of one call must share a precision");
        if (M[k]->solve_algorithm == CULIPX_SOLVE_JACOBI)
            return fail(CULIPX_NOT_SUPPORTED, "culipx_sqmr_solve_many: SOLVE_JACOBI is not batched");
    }
    std::vector<double> out((size_t)num * 8, 0.0);
    CULIPX_TRY(sqmr_solve_many_async(h, num, A, M, b, x, tol, max_it, w, out.data()));
    CULIPX_CUDA(cudaStreamSynchronize(h->stream));
    many_results(num, max_it, out.data(), h_res, h_its, h_status);
    return CULIPX_OK;
}

int sqmr_solve_persistent(culipx_handle_t* h, Csr* A, Factor* M, const double* b, double* x, double tol, int max_it,
                          double* residual, int* iterations, Sqmr* w)
{
    double out[8];
    const int st = (M->precision == CULIPX_F64) ? launch_persistent<double, 1>(h, A, M, b, x, tol, max_it, w, out)
                                                : launch_persistent<float, 1>(h, A, M, b, x, tol, max_it, w, out);
    if (st != CULIPX_OK) return st;
    if (residual) *residual = out[0];
    if (iterations) *iterations = (int)out[1];
    if (out[6] != 0.0) return fail(CULIPX_TIMEOUT, "culipx_sqmr_solve: a bounded device wait gave up (results invalid)");
    if (out[2] != 0.0) return fail(CULIPX_BREAKDOWN, "culipx_sqmr_solve: breakdown (non-finite scalar)");
    if (out[3] == 0.0 && max_it > 0 && (int)out[1] >= max_it) return CULIPX_MAXIT;
    return CULIPX_OK;
}

// ---------------------------------------------------------------------------
// SQMR without device allocation.
//
// For callers that cannot allocate device memory when they solve: processes
// whose device memory is already handed out by another allocator (a caching
// allocator such as PyTorch's, or an application-wide pool that owns the
// GPU), and latency-critical request loops, where cudaMalloc / cudaFree can
// synchronize the device and take milliseconds.  The factor (and K) are set
// up beforehand through the regular entry points; this call then uses a
// fixed scratch area compiled into the library instead of the handle's
// workspace.
//
// The scratch is a file-scope device array of kNoAllocMaxRows x 8 doubles
// plus the per-CTA reduction slots (about 4.3 MB): every GPU that loads this
// library holds it until the process exits.  All calls share it and it keeps
// the last call's contents; the call clears what must start at zero.  Calls
// whose work overlaps on the GPU (two streams, two host threads) race on it.
// The first call on a device looks up the array's device address with
// cudaGetSymbolAddress (with that device current); make that first call
// before any stream capture.
namespace {

constexpr int kNoAllocMaxRows = 65536;
constexpr int kNoAllocMaxGrid = 1024;
constexpr size_t kNoAllocVecs = (kVecs + 1) * (size_t)kNoAllocMaxRows;
constexpr size_t kNoAllocSlots = kNoAllocVecs + (size_t)2 * kMaxNV * kNoAllocMaxGrid;

static __device__ __align__(256) double g_noalloc_scratch[kNoAllocSlots];

std::atomic<double*> g_noalloc_ptr[kMaxDevices];  // per-device address of g_noalloc_scratch

int noalloc_setup(int dev)
{
    if (g_noalloc_ptr[dev].load(std::memory_order_acquire)) return CULIPX_OK;
    void* ptr = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&ptr, g_noalloc_scratch);
    if (e != cudaSuccess || !ptr) {
        cudaGetLastError();
        return fail(CULIPX_CUDA_ERROR, "culipx_sqmr_solve_noalloc: cudaGetSymbolAddress failed: %s",
                    cudaGetErrorString(e));
    }
    g_noalloc_ptr[dev].store(static_cast<double*>(ptr), std::memory_order_release);
    return CULIPX_OK;
}

template <class TF>
int noalloc_grid(int dev, int* G)
{
    CULIPX_TRY((persistent_grid<TF, 1>(dev, G)));
    *G = std::min(*G, kNoAllocMaxGrid);
    return CULIPX_OK;
}

// out[0..3] = residual estimate, iterations, breakdown flag, converged flag
template <class TF>
int launch_noalloc(culipx_handle_t* h, Csr* A, Factor* M, const double* b, double* x, double tol, int max_it,
                   double (&out)[8])
{
    static DeviceGridCache grid_cache;  // one per factor precision
    int G = 0, dev = 0;
    CULIPX_TRY(cached_grid(grid_cache, noalloc_grid<TF>, &G, &dev));
    CULIPX_TRY(noalloc_setup(dev));
    double* base = g_noalloc_ptr[dev].load(std::memory_order_acquire);
    // run_persistent clears the recurrence vectors the scratch kept from the last call
    PArgs<TF> a = make_args<TF>(A, M, base, base + kNoAllocVecs, b, x, tol, max_it);
    // the level counter after the results (the vectors' region holds a spare row of kNoAllocMaxRows values)
    a.lvl_done = reinterpret_cast<unsigned long long*>(a.out + 8 * kMaxNR);
    a.wait_skew = h->sqmr ? h->sqmr->wait_skew : 0;
    a.count_red = reductions_counted(*M->pat, G);
    a.red_skew = h->sqmr ? h->sqmr->red_skew : 0;
    return run_persistent<TF, 1>(h, a, G, out);
}

}  // namespace

int sqmr_solve_noalloc(culipx_handle_t* h, Csr* A, Factor* M, const double* b, double* x, double tol, int max_it,
                       double* residual, int* iterations)
{
    if (!A || !M || !b || !x) return fail(CULIPX_INVALID_ARG, "culipx_sqmr_solve_noalloc: null argument");
    if (A->precision != CULIPX_F64 || A->m != A->n)
        return fail(CULIPX_INVALID_ARG, "culipx_sqmr_solve_noalloc: A must be square FP64");
    if (!M->computed || M->pat->n != A->m)
        return fail(CULIPX_INVALID_ARG, "culipx_sqmr_solve_noalloc: preconditioner not computed or wrong size");
    if (M->solve_algorithm == CULIPX_SOLVE_JACOBI)
        return fail(CULIPX_NOT_SUPPORTED, "culipx_sqmr_solve_noalloc: SOLVE_JACOBI needs culipx_sqmr_solve");
    if (A->m > kNoAllocMaxRows)
        return fail(CULIPX_INVALID_ARG,
                    "culipx_sqmr_solve_noalloc: n = %d exceeds the fixed scratch of %d rows; use culipx_sqmr_solve",
                    A->m, kNoAllocMaxRows);
    if (max_it < 0) return fail(CULIPX_INVALID_ARG, "culipx_sqmr_solve_noalloc: max_it < 0");
    double out[8] = {};
    const int st = M->precision == CULIPX_F64 ? launch_noalloc<double>(h, A, M, b, x, tol, max_it, out)
                                              : launch_noalloc<float>(h, A, M, b, x, tol, max_it, out);
    if (st != CULIPX_OK) return st;
    if (residual) *residual = out[0];
    if (iterations) *iterations = (int)out[1];
    if (out[6] != 0.0)
        return fail(CULIPX_TIMEOUT, "culipx_sqmr_solve_noalloc: a bounded device wait gave up (results invalid)");
    if (out[2] != 0.0) return fail(CULIPX_BREAKDOWN, "culipx_sqmr_solve_noalloc: breakdown (non-finite scalar)");
    return status_of(out, max_it);
}

}  // namespace culipx
