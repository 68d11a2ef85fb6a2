// Batched stepping of many independent lattices ("ensemble" and serving).
//
// The reference runs one lattice per program invocation; an ensemble of small
// lattices (different seeds, couplings and sizes) is a loop of separate runs.
// Here the lattices of a batch advance together: a persistent grid per kernel
// walks a table of work items, one item per (lattice, y/z tile, x-chunk) of the
// FP32 pair step (pair_step.cuh) or, for Moore lattices it does not take, the
// tiled step (tiled_step.cuh).  A call advancing K steps is one CUDA graph: a
// copy of the K per-step job tables from pinned host memory, then for each
// kernel its K steps.  The graph is reused as long as K is; lattices join and
// leave between calls by rewriting the tables.
//
// Each lattice's arithmetic uses only its own fields and coefficients and the
// same tile decomposition as the single-lattice path, and its diagnostics are
// reduced in a fixed order; so a lattice gives bitwise the same result alone,
// in any mix, and through lat_step on its own handle.
#include <algorithm>
#include <cstring>
#include <map>
#include <string>
#include <type_traits>
#include <vector>

#include "lattice_handle.hpp"
#include "pair_step.cuh"
#include "tiled_step.cuh"

namespace lat {

constexpr int kBatchMaxJobs = 256;

// Planes per diagnostic partial, by the lattice's size only: the partials, and
// so the sums, are the same for every chunk that is a multiple of it.  Short
// for small lattices, which march short chunks when few of them run.
constexpr int partial_planes(int64_t sites) { return sites <= (1 << 17) ? 2 : (sites <= (1 << 18) ? 4 : 8); }

struct BatchJob {
    Geom g;
    Fields<float, 7> f;     // AH uses the first 5 components
    union {
        StepCoefT<float> c;  // tiled step
        PairCoef pc;         // pair step
    };
    Charges<float> ch;
    DiagOut d;
    int diag;               // record diagnostics at this step
    int chunk;
    int psub;               // planes per diagnostic partial (0: one per item)
    int vec;                // tiled step: 16-byte staging
    int tiles_z, tiles_y;
    int items;              // tiles_z * tiles_y * x-chunks
    int partials;           // diagnostic partials of the step
    int item_begin;         // first work item of this job in its table
    int done;               // items finished (counted on the device at diagnostic steps)
    double* diag_out;       // finalized (energy, |G|) of this step
};

// One step kernel's share of a step: its jobs are jobs[first .. first+njobs).
struct BatchHead {
    int njobs, first, total_items, pad;
    int begin[kBatchMaxJobs];  // item_begin of its jobs, contiguous for the item -> job lookup
};

// x-planes per CTA of a served lattice's final diagnostics: its shape only, so
// that the sums do not depend on the other jobs.
int batch_chunk(const Geom& g)
{
    const int x = g.hix - g.lox;
    return std::min(x, x <= 32 ? 16 : 64);
}

namespace {

// the tiled step's tile in place of a PairShape
struct Tiled {};
template <class SH>
constexpr bool is_tiled = std::is_same<SH, Tiled>::value;
template <int NS, class SH>
using TileSmem = std::conditional_t<is_tiled<SH>, TiledSmem<float, NS>, PairSmem<NS>>;

template <int NS, class SH, bool DIAG, bool Q12>
__device__ __forceinline__ void run_item(unsigned char* smem_raw, const BatchJob& J, const Fields<float, 5>& f5,
                                         int bx, int by, int bz, const TileSums& sums)
{
    TileSmem<NS, SH>& sm = *reinterpret_cast<TileSmem<NS, SH>*>(smem_raw);
    if constexpr (is_tiled<SH>)
        tiled_tile<float, 2, DIAG>(sm, J.g, J.f, J.c, J.ch, J.d, bx, by, bz, J.chunk, sums, J.vec != 0);
    else if constexpr (NS == 1)
        pair_tile<1, DIAG, false, false>(sm, SH{}, J.g, f5, J.pc, J.ch, J.d, bx, by, bz, J.chunk, sums);
    else
        pair_tile<2, DIAG, false, Q12>(sm, SH{}, J.g, J.f, J.pc, J.ch, J.d, bx, by, bz, J.chunk, sums);
}

// Sum of a job's n diagnostic partials by the CTA that finished its last item:
// every thread a fixed strided subset with Neumaier compensation, then a fixed
// tree.  red: two doubles of shared memory for each warp.
template <int THREADS>
__device__ __forceinline__ void sum_partials(const double* partials, int n, double* out, double* red, int tid)
{
    double e = 0, ce = 0, g = 0, cg = 0;
    auto add = [](double& s, double& c, double x) {
        // |s| >= |x|, by integer instructions
        const bool larger = (unsigned long long)__double_as_longlong(s) << 1 >= (unsigned long long)__double_as_longlong(x) << 1;
        const double t = s + x, a = larger ? s : x, b = larger ? x : s;
        c += (a - t) + b;
        s = t;
    };
    for (int b = tid; b < n; b += THREADS) {
        const double2 v = __ldcg(reinterpret_cast<const double2*>(partials) + b);   // other CTAs wrote them
        add(e, ce, v.x);
        add(g, cg, v.y);
    }
    warp_sum2(e + ce, g + cg, red[tid >> 5], red[THREADS / 32 + (tid >> 5)], tid & 31);
    __syncthreads();
    store_sum2<THREADS / 32>(red, red + THREADS / 32, out, tid);
}

// Persistent step kernel for the lattices with NS scalars whose tile is SH: CTAs
// stride over the work items of all of them, four 4-warp CTAs per SM (tiled
// step: three 8-warp CTAs).  Q12: the Moore lattices with charges 1 and 2,
// whose link factors the tile forms in closed form (pair_step.cuh).  At a
// diagnostic step the CTA that finishes a job's last item also sums the job's
// partials (a separate launch after every step took 3 us of a 64^3 ensemble's
// step).
template <int NS, class SH, bool Q12>
__global__ void __launch_bounds__(is_tiled<SH> ? TT_THREADS : PT_THREADS, is_tiled<SH> ? 3 : 4)
batch_step_kernel(const BatchHead* __restrict__ tab, BatchJob* __restrict__ jobs)
{
    chain_wait();
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int THREADS = is_tiled<SH> ? TT_THREADS : PT_THREADS;
    __shared__ BatchJob sj;
    __shared__ Fields<float, 5> sf5;  // Abelian-Higgs view of sj.f
    __shared__ int s_job, s_last;
    const int total = tab->total_items;
    const int nj = tab->njobs;
    const int tid = threadIdx.y * TT_Z + threadIdx.x;
    for (int w = blockIdx.x; w < total; w += gridDim.x) {
        if (tid < 32) {
            // the job of item w: jobs whose first item is <= w, counted by one
            // warp over the contiguous begin[] (all loads independent)
            int cnt = 0;
#pragma unroll
            for (int r = 0; r < kBatchMaxJobs / 32; ++r) {
                const int q = r * 32 + tid;
                const bool le = q < nj && tab->begin[q] <= w;
                cnt += __popc(__ballot_sync(0xffffffffu, le));
            }
            if (tid == 0) s_job = tab->first + cnt - 1;
        }
        __syncthreads();
        // stage the job descriptor in shared memory (its coefficients are read
        // throughout the tile)
        {
            const int* src = reinterpret_cast<const int*>(&jobs[s_job]);
            int* dst = reinterpret_cast<int*>(&sj);
            for (int q = tid; q < (int)(sizeof(BatchJob) / sizeof(int)); q += THREADS) dst[q] = src[q];
            if (tid < 5) {
                sf5.now[tid] = jobs[s_job].f.now[tid];
                sf5.past[tid] = jobs[s_job].f.past[tid];
            }
        }
        __syncthreads();
        const int local = w - sj.item_begin;
        const int bx = local % sj.tiles_z;
        const int r = local / sj.tiles_z;
        const int by = r % sj.tiles_y;
        const int bz = r / sj.tiles_y;
        if (sj.diag) {
            const int per = sj.psub > 0 ? sj.chunk / sj.psub : 1;
            const TileSums s_sums{sj.d.partials + 2 * ((bz * per * sj.tiles_y + by) * sj.tiles_z + bx), sj.psub,
                                  2 * sj.tiles_y * sj.tiles_z};
            run_item<NS, SH, true, Q12>(smem_raw, sj, sf5, bx, by, bz, s_sums);
            if (tid == 0) {   // the thread that wrote the item's partials
                __threadfence();
                s_last = atomicAdd(&jobs[s_job].done, 1) == sj.items - 1;
            }
            __syncthreads();
            if (s_last) {
                __threadfence();
                sum_partials<THREADS>(sj.d.partials, sj.partials, sj.diag_out, reinterpret_cast<double*>(smem_raw), tid);
            }
        } else {
            run_item<NS, SH, false, Q12>(smem_raw, sj, sf5, bx, by, bz, TileSums{nullptr, 0, 0});
        }
        __syncthreads();  // sj and the tile's shared memory are reused by the next item
    }
}

// Job tables (step kernels): 0..3 Abelian-Higgs on 64x4 and 32x8 tiles with
// 16-byte staging, then with element staging; 4, 5 Moore on 64x4 tiles, with
// any charges and with 1 and 2; 6 Moore on the tiled step.
constexpr int kTables = 7;
enum { kMoorePair = 4, kMoorePair12 = 5, kMooreTiled = 6 };
using BatchKernel = void (*)(const BatchHead*, BatchJob*);
const BatchKernel kKernel[kTables] = {
    batch_step_kernel<1, PairShape<32, true>, false>, batch_step_kernel<1, PairShape<16, true>, false>,
    batch_step_kernel<1, PairShape<32, false>, false>, batch_step_kernel<1, PairShape<16, false>, false>,
    batch_step_kernel<2, PairShape<32, true>, false>, batch_step_kernel<2, PairShape<32, true>, true>,
    batch_step_kernel<2, Tiled, false>};
size_t table_smem(int table)
{
    return table == kMooreTiled ? sizeof(TiledSmem<float, 2>) : (table < kMoorePair ? sizeof(PairSmem<1>) : sizeof(PairSmem<2>));
}
dim3 table_block(int table) { return table == kMooreTiled ? dim3(TT_Z, TT_Y) : dim3(PT_TZ, PT_Y); }
constexpr size_t kMaxGraphs = 32;  // graphs kept per batch, by the set of tables they launch

}  // namespace

}  // namespace lat

using namespace lat;

struct lat_batch {
    struct Job {
        lat_handle* h;
        int32_t diag_every;
        int64_t stop_step;          // the job advances until its time step reaches this
        std::vector<lat_diag> diags;  // recorded, not yet taken
    };
    std::vector<Job> jobs;
    int device = 0;
    int max_jobs = 0;
    cudaStream_t stream = nullptr;
    int grid[kTables] = {};          // persistent CTAs of each step kernel
    int K = 0;                       // steps the buffers below hold and the graphs make
    int chunk = 0;                   // x-planes per work item; 0: lat_batch_advance's rule
    char* tab_host = nullptr;        // pinned, and its device copy: BatchHead[K][kTables], then BatchJob[K][max_jobs]
    char* tab_dev = nullptr;
    double* diag_dev = nullptr;      // [K][max_jobs][2]
    double* diag_host = nullptr;     // pinned copy
    std::map<unsigned, cudaGraphExec_t> exec;  // graphs of K steps, by the set of tables they launch
    cudaStream_t side[kTables] = {};           // one stream per table while a graph is captured
    cudaEvent_t fork = nullptr, join[kTables] = {};
    int64_t launches = 0;

    size_t heads_bytes() const { return sizeof(BatchHead) * kTables * (size_t)K; }
    size_t table_bytes() const { return heads_bytes() + sizeof(BatchJob) * (size_t)max_jobs * (size_t)K; }
    BatchHead* head(char* base, int s, int q) const { return (BatchHead*)base + kTables * s + q; }
    BatchJob* jobs_of(char* base, int s) const { return (BatchJob*)(base + heads_bytes()) + (size_t)max_jobs * s; }
};

#define BATCH_CK(call)                                                             \
    do {                                                                           \
        cudaError_t e_ = (call);                                                   \
        if (e_ != cudaSuccess) {                                                   \
            set_error(std::string(#call) + ": " + cudaGetErrorString(e_));         \
            return e_ == cudaErrorMemoryAllocation ? LAT_ERR_NOMEM : LAT_ERR_CUDA; \
        }                                                                          \
    } while (0)

static void release_graph(lat_batch* b)
{
    for (auto& e : b->exec) cudaGraphExecDestroy(e.second);
    b->exec.clear();
    cudaFreeHost(b->tab_host);
    cudaFree(b->tab_dev);
    cudaFree(b->diag_dev);
    cudaFreeHost(b->diag_host);
    b->tab_host = nullptr;
    b->tab_dev = nullptr;
    b->diag_dev = nullptr;
    b->diag_host = nullptr;
    b->K = 0;
}

// Build (or reuse) the graph of K steps for the tables in `mask`, and the
// buffers of K steps.  A lattice stays in one table for the whole call, so
// the tables' chains of K step kernels are independent and form parallel
// branches: 18 Abelian-Higgs and 6 Moore 64^3 lattices, which fill neither
// kernel's CTA slots alone, stepped one after the other before.  Graphs are
// kept per mask, as jobs of a model come and go between calls.
static int ensure_graph(lat_batch* b, int K, unsigned mask)
{
    if (b->K != K) {
        release_graph(b);
        b->K = K;
        cudaError_t e = cudaMallocHost((void**)&b->tab_host, b->table_bytes());
        if (e == cudaSuccess) e = cudaMalloc((void**)&b->tab_dev, b->table_bytes());
        if (e == cudaSuccess) e = cudaMalloc((void**)&b->diag_dev, sizeof(double) * 2 * (size_t)K * b->max_jobs);
        if (e == cudaSuccess) e = cudaMallocHost((void**)&b->diag_host, sizeof(double) * 2 * (size_t)K * b->max_jobs);
        if (e != cudaSuccess) {
            cudaGetLastError();
            release_graph(b);
            BATCH_CK(e);
        }
    }
    if (b->exec.count(mask)) return LAT_OK;
    if (b->exec.size() >= kMaxGraphs) {
        for (auto& e : b->exec) cudaGraphExecDestroy(e.second);
        b->exec.clear();
    }
    BATCH_CK(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal));
    cudaMemcpyAsync(b->tab_dev, b->tab_host, b->table_bytes(), cudaMemcpyHostToDevice, b->stream);
    cudaEventRecord(b->fork, b->stream);
    for (int q = 0; q < kTables; ++q) {
        if (!(mask & (1u << q))) continue;
        cudaStream_t st = b->side[q];
        cudaStreamWaitEvent(st, b->fork, 0);
        for (int s = 0; s < K; ++s)
            launch_chained(kKernel[q], b->grid[q], table_block(q), table_smem(q), st, b->head(b->tab_dev, s, q),
                           b->jobs_of(b->tab_dev, s));
        cudaEventRecord(b->join[q], st);
        cudaStreamWaitEvent(b->stream, b->join[q], 0);
    }
    cudaMemcpyAsync(b->diag_host, b->diag_dev, sizeof(double) * 2 * (size_t)K * b->max_jobs, cudaMemcpyDeviceToHost,
                    b->stream);
    cudaGraph_t graph = nullptr;
    BATCH_CK(cudaStreamEndCapture(b->stream, &graph));
    cudaGraphExec_t exec = nullptr;
    const cudaError_t e = cudaGraphInstantiate(&exec, graph, 0);
    cudaGraphDestroy(graph);
    BATCH_CK(e);
    b->exec[mask] = exec;
    return LAT_OK;
}

// The table (step kernel) of a lattice, by its model and tile, for a Moore
// lattice also whether its charges are 1 and 2: it depends on the lattice alone,
// never on its company.
static int table_of(const lat_handle* h, const Fields<float, 7>& fj)
{
    if (h->p.model == LAT_MODEL_MOORE) {
        if (!pair_moore_ok(h->geom, fj)) return kMooreTiled;
        return small_int_power(h->p.q1) == 1 && small_int_power(h->p.q2) == 2 ? kMoorePair12 : kMoorePair;
    }
    Fields<float, 5> f5;
    for (int c = 0; c < 5; ++c) f5.now[c] = fj.now[c];
    return (tiled_vec_ok(h->geom, f5) ? 0 : 2) + (pair_tz2(h->geom) == 32 ? 0 : 1);
}

static Fields<float, 7> level_fields(const lat_handle* h, int64_t n)
{
    const int tNow = (int)((n + 1) % 2), tPast = (int)(n % 2);
    Fields<float, 7> fj{};
    for (int c = 0; c < h->ncomp; ++c) {
        fj.now[c] = (const float*)h->slot(c, tNow);
        fj.past[c] = (float*)h->slot(c, tPast);
    }
    return fj;
}

extern "C" {

int lat_batch_create(int32_t max_jobs, lat_batch** out)
{
    if (!out || max_jobs < 1 || max_jobs > kBatchMaxJobs) {
        set_error("lat_batch_create: max_jobs must be in [1, 256]");
        return LAT_ERR_INVALID;
    }
    *out = nullptr;
    lat_batch* b = new lat_batch();
    b->max_jobs = max_jobs;
    cudaGetDevice(&b->device);
    if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess) {
        delete b;
        set_error("lat_batch_create: no CUDA device or stream");
        return LAT_ERR_NODEVICE;
    }
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, b->device);
    for (int q = 0; q < kTables; ++q) {
        const size_t smem = table_smem(q);
        cudaFuncSetAttribute(kKernel[q], cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        int per_sm = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kKernel[q], (int)(table_block(q).x * table_block(q).y), smem);
        b->grid[q] = std::max(1, sms * std::max(1, per_sm));
    }
    bool ok = cudaEventCreateWithFlags(&b->fork, cudaEventDisableTiming) == cudaSuccess;
    for (int q = 0; q < kTables; ++q)
        ok = ok && cudaStreamCreateWithFlags(&b->side[q], cudaStreamNonBlocking) == cudaSuccess &&
             cudaEventCreateWithFlags(&b->join[q], cudaEventDisableTiming) == cudaSuccess;
    if (!ok) {
        lat_batch_destroy(b);
        set_error("lat_batch_create: no CUDA streams or events");
        return LAT_ERR_CUDA;
    }
    *out = b;
    return LAT_OK;
}

int lat_batch_destroy(lat_batch* b)
{
    if (!b) return LAT_OK;
    cudaSetDevice(b->device);
    cudaStreamSynchronize(b->stream);
    release_graph(b);
    if (b->fork) cudaEventDestroy(b->fork);
    for (int q = 0; q < kTables; ++q) {
        if (b->side[q]) cudaStreamDestroy(b->side[q]);
        if (b->join[q]) cudaEventDestroy(b->join[q]);
    }
    cudaStreamDestroy(b->stream);
    delete b;
    return LAT_OK;
}

int lat_batch_add(lat_batch* b, lat_handle* h, int32_t diag_every, int64_t stop_step)
{
    if (!b || !h || diag_every < 0) {
        set_error("lat_batch_add: bad argument");
        return LAT_ERR_INVALID;
    }
    if (h->p.precision != LAT_F32 || h->p.kernel_variant != 0) {
        set_error("lat_batch_add: batches step FP32 lattices (LAT_F32, default kernels)");
        return LAT_ERR_INVALID;
    }
    if (h->p.bc > LAT_BC_FIXED || bc_z_kind(h->p) > LAT_BC_FIXED) {
        set_error("lat_batch_add: batches step lattices with periodic or fixed boundaries");
        return LAT_ERR_INVALID;
    }
    if ((int)b->jobs.size() >= b->max_jobs) {
        set_error("lat_batch_add: batch is full");
        return LAT_ERR_CAPACITY;
    }
    for (auto& j : b->jobs)
        if (j.h == h) {
            set_error("lat_batch_add: handle already in the batch");
            return LAT_ERR_STATE;
        }
    b->jobs.push_back({h, diag_every, stop_step, {}});
    return (int)b->jobs.size() - 1;
}

int lat_batch_remove(lat_batch* b, lat_handle* h)
{
    if (!b || !h) {
        set_error("lat_batch_remove: bad argument");
        return LAT_ERR_INVALID;
    }
    for (size_t q = 0; q < b->jobs.size(); ++q)
        if (b->jobs[q].h == h) {
            b->jobs.erase(b->jobs.begin() + (long)q);
            return LAT_OK;
        }
    set_error("lat_batch_remove: handle not in the batch");
    return LAT_ERR_STATE;
}

int lat_batch_size(const lat_batch* b) { return b ? (int)b->jobs.size() : LAT_ERR_INVALID; }

int lat_batch_set_chunk(lat_batch* b, int32_t chunk)
{
    if (!b || chunk < 0 || chunk > 4096) {
        set_error("lat_batch_set_chunk: chunk must be in [0, 4096]");
        return LAT_ERR_INVALID;
    }
    b->chunk = chunk;
    return LAT_OK;
}

int64_t lat_batch_kernel_launches(const lat_batch* b) { return b ? b->launches : LAT_ERR_INVALID; }

int lat_batch_advance(lat_batch* b, int32_t nsteps)
{
    if (!b || nsteps < 1) {
        set_error("lat_batch_advance: bad argument");
        return LAT_ERR_INVALID;
    }
    if (b->jobs.empty()) return 0;
    BATCH_CK(cudaSetDevice(b->device));
    const int K = nsteps;
    // previous work of the handles (uploads, single steps) must be complete
    for (auto& j : b->jobs) BATCH_CK(cudaStreamSynchronize(j.h->stream));
    // host-side schedule of every job over the K steps
    struct Plan {
        int steps;
        int64_t n0;
        int table;
    };
    std::vector<Plan> plan(b->jobs.size());
    unsigned mask = 0;
    for (size_t q = 0; q < b->jobs.size(); ++q) {
        auto& j = b->jobs[q];
        const int64_t left = j.stop_step - j.h->n;
        plan[q] = {(int)std::max<int64_t>(0, std::min<int64_t>(K, left)), j.h->n, table_of(j.h, level_fields(j.h, j.h->n))};
        if (plan[q].steps > 0) mask |= 1u << plan[q].table;
        // a diagnostic on the first step needs the divergence of the past level
        const int64_t n = j.h->n;
        if (plan[q].steps > 0 && j.diag_every > 0 && n % j.diag_every == 0 && j.h->p.g != 0 && !j.h->div_valid) {
            lat_handle* h = j.h;
            const int tPast = (int)(n % 2), th0 = h->ncomp - 3;
            cudaError_t e = launch_divergence_f32(h->geom, (const float*)h->slot(th0, tPast),
                                                  (const float*)h->slot(th0 + 1, tPast),
                                                  (const float*)h->slot(th0 + 2, tPast), make_coef(h->p, n),
                                                  (float*)h->divbuf, b->stream);
            if (e != cudaSuccess) {
                set_error(std::string("lat_batch_advance: ") + cudaGetErrorString(e));
                return LAT_ERR_CUDA;
            }
            ++b->launches;
        }
    }
    if (mask == 0) return 0;  // every lattice has reached its stop_step
    int rc = ensure_graph(b, K, mask);
    if (rc) return rc;
    std::vector<std::vector<int>> diag_slots(b->jobs.size());
    // x-planes per work item: the most of 2, 4, 8, 16 and 32 that leave the
    // running lattices together 1100 items, 1.8 for each of the 608 CTA slots.
    // Swept over 2..64 planes on 21 batches of 1..64 lattices of 32^3..256^3,
    // the rule is within 6 % of the best everywhere.  One lattice needs short
    // chunks to fill the SMs, sixty-four prefer long ones: against 64 planes,
    // or 16 below 33, for every lattice, a step of 4 x 32^3 takes 8.8 us
    // instead of 20.4, of 18 Abelian-Higgs and 6 Moore 64^3 105 instead of 172,
    // of 64 x 64^3 261 instead of 277.
    int chunk = 2;
    for (int c : {4, 8, 16, 32}) {
        int64_t items = 0;
        for (size_t q = 0; q < b->jobs.size(); ++q) {
            if (plan[q].steps == 0) continue;
            const Geom& g = b->jobs[q].h->geom;
            items += march_tiles(g, b->jobs[q].h->p.model == LAT_MODEL_MOORE) * ((g.hix - g.lox + c - 1) / c);
        }
        if (items >= 1100) chunk = c;
    }
    // what does not change from step to step
    std::vector<BatchJob> tmpl(b->jobs.size());
    for (size_t q = 0; q < b->jobs.size(); ++q) {
        const lat_handle* h = b->jobs[q].h;
        BatchJob& J = tmpl[q];
        std::memset(&J, 0, sizeof(J));
        J.g = h->geom;
        const bool moore = h->p.model == LAT_MODEL_MOORE;
        if (!moore) {
            J.ch.q[0] = 1;
            J.ch.qpow[0] = 1;
        } else {
            J.ch.q[0] = (float)h->p.q1;
            J.ch.q[1] = (float)h->p.q2;
            J.ch.qpow[0] = small_int_power(h->p.q1);
            J.ch.qpow[1] = small_int_power(h->p.q2);
        }
        J.ch.charge_current = h->p.moore_current == LAT_MOORE_CURRENT_CHARGE;
        J.d.partials = h->partials;
        J.d.divbuf = h->divbuf;
        J.d.use_div = 1;
        J.d.energy_form = h->p.energy_form;
        J.d.charge_current = J.ch.charge_current;
        J.d.write = 1;
        const int x = h->geom.hix - h->geom.lox;
        const int planes = partial_planes(h->N);
        J.chunk = b->chunk > 0 ? b->chunk : std::max(chunk, planes);   // may exceed x: one item, the same partials
        J.psub = J.chunk % planes == 0 ? planes : 0;
        J.vec = tiled_vec_ok(h->geom, level_fields(h, h->n)) ? 1 : 0;
        const dim3 tg = plan[q].table == kMooreTiled ? tiled_grid(h->geom, J.chunk)
                                                     : pair_shape_grid(h->geom, moore ? 32 : pair_tz2(h->geom), J.chunk);
        J.tiles_z = (int)tg.x;
        J.tiles_y = (int)tg.y;
        J.items = (int)(tg.x * tg.y * tg.z);
        J.partials = J.tiles_z * J.tiles_y * (J.psub > 0 ? (x + J.psub - 1) / J.psub : (int)tg.z);
        if (J.partials > h->nblocks) {
            set_error("lat_batch_advance: more diagnostic partials than a lattice has room for");
            return LAT_ERR_STATE;
        }
    }
    for (int s = 0; s < K; ++s) {
        BatchJob* const jobs = b->jobs_of(b->tab_host, s);
        int used = 0;
        for (int t = 0; t < kTables; ++t) {
            BatchHead& T = *b->head(b->tab_host, s, t);
            T.njobs = 0;
            T.first = used;
            T.total_items = 0;
            if (!(mask & (1u << t))) continue;
            for (size_t q = 0; q < b->jobs.size(); ++q) {
                if (plan[q].table != t || s >= plan[q].steps) continue;
                auto& j = b->jobs[q];
                lat_handle* h = j.h;
                const int64_t n = plan[q].n0 + s;
                BatchJob& J = jobs[used++];
                J = tmpl[q];
                J.f = level_fields(h, n);
                const StepCoef c64 = make_coef(h->p, n);
                if (t == kMooreTiled) J.c = coef_as<float>(c64);
                else J.pc = pair_coef(c64);
                const bool diag = j.diag_every > 0 && n % j.diag_every == 0;
                const bool next_diag = j.diag_every > 0 && (n + 1) % j.diag_every == 0;
                J.d.store_div = next_diag && h->p.g != 0;  // keep div(theta) for the next step's Gauss term
                J.diag = diag ? 1 : 0;
                J.item_begin = T.total_items;
                T.begin[T.njobs] = T.total_items;
                J.diag_out = b->diag_dev + 2 * ((size_t)s * b->max_jobs + q);
                T.total_items += J.items;
                ++T.njobs;
                if (diag) diag_slots[q].push_back(s);
            }
        }
    }
    BATCH_CK(cudaGraphLaunch(b->exec[mask], b->stream));
    BATCH_CK(cudaStreamSynchronize(b->stream));
    b->launches += (int64_t)__builtin_popcount(mask) * K;
    int active = 0;
    for (size_t q = 0; q < b->jobs.size(); ++q) {
        auto& j = b->jobs[q];
        lat_handle* h = j.h;
        for (int s : diag_slots[q]) {
            const double* v = b->diag_host + 2 * ((size_t)s * b->max_jobs + q);
            lat_diag dg;
            dg.energy = v[0];
            dg.gauss_abs_sum = v[1];
            const Geom& g = h->geom;
            dg.sites = (int64_t)(g.hix - g.lox) * (g.hiy - g.loy) * (g.hiz - g.loz);
            dg.time_step = plan[q].n0 + s;
            j.diags.push_back(dg);
        }
        if (plan[q].steps > 0) {
            const int64_t nlast = plan[q].n0 + plan[q].steps - 1;
            h->div_valid = j.diag_every > 0 && (nlast + 1) % j.diag_every == 0 && h->p.g != 0;
            h->n = plan[q].n0 + plan[q].steps;
            h->launches += 0;
        }
        if (h->n < j.stop_step) ++active;
    }
    return active;
}

int lat_batch_take_diags(lat_batch* b, lat_handle* h, lat_diag* out, int64_t cap, int64_t* count)
{
    if (!b || !h || !count || (cap > 0 && !out)) {
        set_error("lat_batch_take_diags: bad argument");
        return LAT_ERR_INVALID;
    }
    for (auto& j : b->jobs)
        if (j.h == h) {
            const int64_t n = std::min<int64_t>(cap, (int64_t)j.diags.size());
            for (int64_t q = 0; q < n; ++q) out[q] = j.diags[(size_t)q];
            *count = (int64_t)j.diags.size();
            j.diags.erase(j.diags.begin(), j.diags.begin() + n);
            return LAT_OK;
        }
    set_error("lat_batch_take_diags: handle not in the batch");
    return LAT_ERR_STATE;
}

}  // extern "C"
