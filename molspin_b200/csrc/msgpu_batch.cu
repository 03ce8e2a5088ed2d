// msgpu_batch.cu -- C ABI of the batching form (include/msgpu.h,
// msgpu_batch_*): many radical-pair systems of uneven dimension and
// trajectory count propagated together.  Systems below kStreamDim run the
// resident kernels (msgpu_resident.cuh, msgpu_resident_q.cuh), a CTA per
// trajectory with the Krylov basis in shared memory, one launch per kernel for all
// its systems, all launches at once on a few streams.  A system whose basis does not
// fit shared memory joins the persistent launch k_batch instead, replayed from a CUDA
// graph, with the team threshold and the grid size picked by an autotuner.  A large
// system is better served by the streamed single-system path, which advances all its trajectories in lockstep through the
// quartet-block SpMM (one read of H per 64 trajectories instead of one per
// trajectory): those systems get their own context and stream and run
// concurrently with the persistent launch and with each other.

#include "msgpu.h"

#include <algorithm>
#include <array>
#include <atomic>
#include <chrono>
#include <cmath>
#include <cstring>
#include <string>
#include <thread>
#include <vector>

#include "msgpu_batch.cuh"
#include "msgpu_quartet.h"

using namespace msgpu;

namespace {

struct Buf {
    void *p = nullptr;
    size_t bytes = 0;
};

// Systems of at least this dimension take the streamed single-system path: a
// trajectory's basis no longer fits a CTA's shared memory there, and of the other
// two the persistent launch wins below it and the lockstep SpMM above (the 64-system
// benchmark batch).
constexpr int kStreamDim = 2048;
constexpr int kStreamWorkers = 8;  // host threads driving streamed systems

struct BatchSystem {
    int D = 0, M = 0, nobs = 0, s1 = 0, s2 = 0;
    double kappa = 0.0, st_rate = 0.0;
    unsigned long long seed = 0;
    Buf rowptr, col, valf, obs, rates, psi, acc, comp, prev, pflip;
    // resident kernels: H in padded row order (ell: values, columns, lengths) up
    // to D = 128, by quartets (quart) above
    enum Kind { kNone, kRows, kQuartets, kUnassembled };  // kUnassembled: quartets from the next run on
    Buf ell, quart;
    Kind kind = kNone;
    int kmax = 0;
    ResidentQuartets rq{};
    msgpu_ctx *ctx = nullptr;  // streamed single-system path (D >= kStreamDim)
};

}  // namespace

struct msgpu_batch {
    int device = 0;
    size_t budget = 0, used = 0;
    cudaStream_t stream = nullptr;
    std::string err;
    std::vector<BatchSystem> sys;
    // systems below kStreamDim dropped by msgpu_batch_clear: their device
    // buffers serve the next msgpu_batch_add_system (no cudaMalloc / cudaFree per reuse)
    std::vector<BatchSystem> spare;
    Buf sys_d, items_d, queue_d, status_d, scratch, times_d, backup, many_d, first_d, jobs_d, found_d;
    int threshold = 512, ctas_per_sm = 2, tuned = 0;
    int sm_count = 0;
    cudaGraphExec_t graph = nullptr;
    size_t graph_key = 0;
    float last_ms = 0.f;
    int m = 0;
    long long launches = 0;  // kernels launched here (tuning probes included)
    cudaStream_t side[8] = {};  // the resident launches' streams, made on first use
    cudaEvent_t fork = nullptr, join[8] = {};
};

namespace {

int bfail(msgpu_batch *b, int code, const std::string &msg)
{
    if (b) b->err = msg;
    return code;
}

void brelease(msgpu_batch *b, Buf &x)
{
    if (x.p) {
        cudaFree(x.p);
        b->used -= x.bytes;
    }
    x.p = nullptr;
    x.bytes = 0;
}

int bensure(msgpu_batch *b, Buf &x, size_t bytes, const char *what)
{
    if (bytes == 0) bytes = 16;
    if (x.p && x.bytes >= bytes) return MSGPU_OK;
    brelease(b, x);
    if (b->budget && b->used + bytes > b->budget)
        return bfail(b, MSGPU_ERR_BUDGET, std::string("batch: device memory budget exceeded allocating ") + what);
    cudaError_t e = cudaMalloc(&x.p, bytes);
    if (e != cudaSuccess) {
        x.p = nullptr;
        return bfail(b, MSGPU_ERR_CUDA, std::string("batch: ") + what + ": " + cudaGetErrorString(e));
    }
    x.bytes = bytes;
    b->used += bytes;
    return MSGPU_OK;
}

int upload(msgpu_batch *b, Buf &x, const void *src, size_t bytes, const char *what)
{
    if (int rc = bensure(b, x, bytes, what)) return rc;
    cudaError_t e = cudaMemcpyAsync(x.p, src, bytes, cudaMemcpyHostToDevice, b->stream);
    if (e) return bfail(b, MSGPU_ERR_CUDA, std::string("batch: upload ") + what + ": " + cudaGetErrorString(e));
    return MSGPU_OK;
}

void drop_graph(msgpu_batch *b)
{
    if (b->graph) cudaGraphExecDestroy(b->graph);
    b->graph = nullptr;
    b->graph_key = 0;
}

double flip_prob(double st_rate, double h) { return -0.5 * std::expm1(-2.0 * (0.5 * st_rate) * h); }

// A system on the resident kernels (a CTA per trajectory).
struct ResidentRun {
    ResidentSystem S;
    ResidentManyShape shape;
    double cost;  // of one trajectory
};
constexpr size_t kSmemMax = 227 * 1024;
constexpr size_t kResidentSmemMax = kSmemMax - sizeof(ResidentSystem);  // beside the system's descriptor

// Queues the resident kernels, one launch for all systems of a kernel (a launch a
// system leaves a batch of small systems eight at a time: 500 systems of D = 64 with 8
// trajectories, 50 steps: 41 against 3.9 ms, 64 of them with 16, 20 steps: 2.24 against
// 0.47 ms), the longest trajectories first, over side streams between two events on
// the batch's stream.  Beside streamed systems (`streamed` of them), whose chains of
// short kernels set the time, they take one stream, or two beside a single one: nine
// kernels of 64 trajectories beside four systems of D = 2048 and 4096 8.6 ms with eight
// streams, 7.7 with one; of 8 trajectories beside one system of D = 2048 5.3, 5.3 with
// two, 6.1 with one.
int launch_resident(msgpu_batch *b, std::vector<ResidentRun> &runs, int streamed)
{
    if (runs.empty()) return MSGPU_OK;
    std::stable_sort(runs.begin(), runs.end(), [](const ResidentRun &x, const ResidentRun &y) { return x.cost > y.cost; });
    struct Launch {
        ResidentManyShape shape;
        std::vector<int> runs;
    };
    std::vector<Launch> launches;  // by their longest trajectory
    for (size_t i = 0; i < runs.size(); ++i) {
        size_t k = 0;
        while (k < launches.size() && launches[k].shape.fn != runs[i].shape.fn) ++k;
        if (k == launches.size()) launches.push_back(Launch{runs[i].shape, {}});
        launches[k].shape.smem = std::max(launches[k].shape.smem, runs[i].shape.smem);
        launches[k].runs.push_back(static_cast<int>(i));
    }
    // every launch's systems, then every launch's first CTAs (one more than systems)
    std::vector<ResidentSystem> sys;
    std::vector<int> first;
    for (const Launch &l : launches) {
        first.push_back(0);
        for (int i : l.runs) {
            sys.push_back(runs[i].S);
            first.push_back(first.back() + runs[i].S.M);
        }
    }
    int rc;
    if ((rc = upload(b, b->many_d, sys.data(), sizeof(ResidentSystem) * sys.size(), "resident systems")) ||
        (rc = upload(b, b->first_d, first.data(), sizeof(int) * first.size(), "resident work")))
        return rc;
    const int ns = std::min<int>(streamed > 1 ? 1 : streamed == 1 ? 2 : 8, static_cast<int>(launches.size()));
    cudaError_t e = cudaSuccess;
    if (!b->fork) e = cudaEventCreateWithFlags(&b->fork, cudaEventDisableTiming);
    for (int k = 0; k < ns && !e; ++k)
        if (!b->side[k] && !(e = cudaStreamCreateWithFlags(&b->side[k], cudaStreamNonBlocking)))
            e = cudaEventCreateWithFlags(&b->join[k], cudaEventDisableTiming);
    if (!e) e = cudaEventRecord(b->fork, b->stream);
    for (int k = 0; k < ns && !e; ++k) e = cudaStreamWaitEvent(b->side[k], b->fork, 0);
    int *status = static_cast<int *>(b->status_d.p);
    size_t at_sys = 0, at = 0;  // in sys and first
    for (size_t i = 0; i < launches.size() && !e; ++i) {
        const ResidentManyShape &r = launches[i].shape;
        const int n = static_cast<int>(launches[i].runs.size()), smem = static_cast<int>(r.smem);
        const bool one = n == 1 && r.one;
        if ((e = raise_smem_limit(one ? reinterpret_cast<const void *>(r.one) : reinterpret_cast<const void *>(r.fn), smem)))
            break;
        if (one)
            r.one<<<first[at + 1], 32 * r.warps, smem, b->side[i % ns]>>>(sys[at_sys], status);
        else
            r.fn<<<first[at + n], 32 * r.warps, smem, b->side[i % ns]>>>(
                static_cast<const ResidentSystem *>(b->many_d.p) + at_sys, static_cast<const int *>(b->first_d.p) + at, n,
                status);
        ++b->launches;
        e = cudaGetLastError();
        at_sys += n;
        at += n + 1;
    }
    for (int k = 0; k < ns && b->join[k]; ++k) {  // joined even after an error: nothing is left running behind it
        const cudaError_t je = cudaEventRecord(b->join[k], b->side[k]);
        const cudaError_t we = cudaStreamWaitEvent(b->stream, b->join[k], 0);
        if (!e) e = je ? je : we;
    }
    return e ? bfail(b, MSGPU_ERR_CUDA, std::string("batch: resident launch: ") + cudaGetErrorString(e)) : MSGPU_OK;
}

// The CSR arrays that the persistent launch reads.
int upload_csr(msgpu_batch *b, BatchSystem &s, const int *rowptr, const int *col, const std::vector<float> &val)
{
    const int nnz = rowptr[s.D];
    int rc;
    if ((rc = upload(b, s.rowptr, rowptr, sizeof(int) * (s.D + 1), "rowptr")) ||
        (nnz > 0 && (rc = upload(b, s.col, col, sizeof(int) * nnz, "col"))) ||
        (nnz > 0 && (rc = upload(b, s.valf, val.data(), sizeof(float) * val.size(), "values"))))
        return rc;
    return MSGPU_OK;
}

// Descriptors, work items and scratch for the given schedule, and the resident
// launches; returns the grid size through *grid.
int prepare(msgpu_batch *b, int ntimes, int m, int accumulate, long long step_offset, int threshold,
            int ctas_per_sm, int *grid, size_t *slice, size_t *smem, int *nlarge, int *nitems,
            std::vector<ResidentRun> *resident)
{
    std::vector<ResidentSystem> desc(b->sys.size());
    std::vector<ResidentWork> large, small;
    int dmax_large = 0, dmax_small = 0;
    for (size_t i = 0; i < b->sys.size(); ++i) {
        BatchSystem &s = b->sys[i];
        ResidentSystem S;
        std::memset(&S, 0, sizeof(S));
        S.rowptr = static_cast<const int *>(s.rowptr.p);
        S.col = static_cast<const int *>(s.col.p);
        S.valf = static_cast<const float2 *>(s.valf.p);
        S.kappa = s.kappa;
        S.D = s.D;
        S.M = s.M;
        S.acc_ld = s.M;
        S.m = std::min(m, s.D);
        S.s1 = s.s1;
        S.s2 = s.s2;
        S.nobs = s.nobs;
        S.obs = static_cast<const double2 *>(s.obs.p);
        S.rates = static_cast<const double *>(s.rates.p);
        S.nz.mode = s.st_rate > 0.0 ? MSGPU_NOISE_PHILOX : MSGPU_NOISE_NONE;
        S.nz.M = s.M;
        S.nz.seed = s.seed;
        S.psi = S.psi_out = s.psi.p;
        S.rs = 1;
        S.ts = s.D;
        S.acc = static_cast<double *>(s.acc.p);
        S.comp = static_cast<double *>(s.comp.p);
        S.prev = static_cast<double *>(s.prev.p);
        S.traj_values = nullptr;
        S.times = static_cast<const double *>(b->times_d.p);
        S.pflip = static_cast<const double *>(s.pflip.p);
        S.ntimes = ntimes;
        S.step_offset = step_offset;
        S.accumulate = accumulate;
        desc[i] = S;
        if (s.ctx) continue;  // streamed path: no work items here
        if (s.kind != BatchSystem::kNone) {
            const ResidentManyShape shape = s.kind == BatchSystem::kRows ? resident_shape_many(s.D, S.m) : resident_shape_q_many(s.D, S.m);
            if (shape.fn && shape.smem <= kResidentSmemMax) {
                if (s.kind == BatchSystem::kRows) {
                    const size_t slots = static_cast<size_t>(s.D) * s.kmax;
                    S.valf = static_cast<const float2 *>(s.ell.p);
                    S.col = reinterpret_cast<const int *>(S.valf + slots);
                    S.rowcnt = S.col + slots;
                    S.kstride = s.D;
                    S.kmax = s.kmax;
                } else {
                    S.rq = s.rq;
                }
                resident->push_back(ResidentRun{S, shape, static_cast<double>(s.D) * S.m});
                continue;
            }
        }
        auto &dst = s.D >= threshold ? large : small;
        for (int t = 0; t < s.M; ++t) dst.push_back(ResidentWork{static_cast<int>(i), t});
        if (s.D >= threshold) dmax_large = std::max(dmax_large, s.D);
        else dmax_small = std::max(dmax_small, s.D);
    }
    // largest systems first so that the long items start early
    auto byD = [&](const ResidentWork &x, const ResidentWork &y) {
        return b->sys[x.sys].D > b->sys[y.sys].D || (b->sys[x.sys].D == b->sys[y.sys].D && x.sys < y.sys);
    };
    std::stable_sort(large.begin(), large.end(), byD);
    std::stable_sort(small.begin(), small.end(), byD);
    std::vector<ResidentWork> items = large;
    items.insert(items.end(), small.begin(), small.end());
    *nlarge = static_cast<int>(large.size());
    *nitems = static_cast<int>(items.size());
    const size_t per_large = static_cast<size_t>(m + 1) * dmax_large;
    const size_t per_small = static_cast<size_t>(m + 1) * dmax_small * kBatchWarps;
    *slice = (std::max(per_large, per_small) + 63) / 64 * 64;
    *grid = std::max(1, b->sm_count * ctas_per_sm);
    *smem = sizeof(double2) * kBatchWarps * batch_expm_words(m);
    // the Krylov dimensions that the persistent launch takes, on every route
    if ((!items.empty() || !resident->empty()) && *smem > kSmemMax)
        return bfail(b, MSGPU_ERR_CUDA, std::string("batch: shared memory: ") + cudaGetErrorString(cudaErrorInvalidValue));
    int rc;
    if ((rc = bensure(b, b->status_d, sizeof(int), "status"))) return rc;
    if (items.empty()) return MSGPU_OK;
    if ((rc = upload(b, b->sys_d, desc.data(), sizeof(ResidentSystem) * desc.size(), "descriptors")) ||
        (rc = upload(b, b->items_d, items.data(), sizeof(ResidentWork) * items.size(), "items")) ||
        (rc = bensure(b, b->queue_d, 2 * sizeof(int), "queue")) ||
        (rc = bensure(b, b->scratch, sizeof(float2) * *slice * *grid, "scratch")))
        return rc;
    return MSGPU_OK;
}

int launch(msgpu_batch *b, int grid, size_t slice, size_t smem, int nlarge, int nitems, int m, bool use_graph)
{
    cudaError_t e;
    if ((e = raise_smem_limit(reinterpret_cast<const void *>(k_batch), static_cast<int>(smem))))
        return bfail(b, MSGPU_ERR_CUDA, std::string("batch: shared memory: ") + cudaGetErrorString(e));
    const size_t key = (static_cast<size_t>(grid) << 40) ^ (slice << 8) ^ (static_cast<size_t>(nlarge) << 20) ^
                       static_cast<size_t>(nitems) ^ (static_cast<size_t>(m) << 56) ^ reinterpret_cast<size_t>(b->scratch.p) ^
                       (reinterpret_cast<size_t>(b->sys_d.p) << 1) ^ (reinterpret_cast<size_t>(b->items_d.p) << 2) ^
                       (reinterpret_cast<size_t>(b->queue_d.p) << 3) ^ (reinterpret_cast<size_t>(b->status_d.p) << 4);
    auto enqueue = [&]() {
        cudaMemsetAsync(b->queue_d.p, 0, 2 * sizeof(int), b->stream);
        k_batch<<<grid, kBatchThreads, smem, b->stream>>>(
            static_cast<const ResidentSystem *>(b->sys_d.p), static_cast<const ResidentWork *>(b->items_d.p), nlarge,
            nitems, static_cast<int *>(b->queue_d.p), static_cast<float2 *>(b->scratch.p), slice, m,
            static_cast<int *>(b->status_d.p));
    };
    if (!use_graph) {
        enqueue();
    } else {
        if (!b->graph || b->graph_key != key) {
            drop_graph(b);
            cudaGraph_t g;
            if ((e = cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal)))
                return bfail(b, MSGPU_ERR_CUDA, std::string("batch: capture: ") + cudaGetErrorString(e));
            enqueue();
            if ((e = cudaStreamEndCapture(b->stream, &g)))
                return bfail(b, MSGPU_ERR_CUDA, std::string("batch: capture: ") + cudaGetErrorString(e));
            e = cudaGraphInstantiate(&b->graph, g, 0);
            cudaGraphDestroy(g);
            if (e) return bfail(b, MSGPU_ERR_CUDA, std::string("batch: instantiate: ") + cudaGetErrorString(e));
            b->graph_key = key;
        }
        if ((e = cudaGraphLaunch(b->graph, b->stream)))
            return bfail(b, MSGPU_ERR_CUDA, std::string("batch: graph launch: ") + cudaGetErrorString(e));
    }
    if ((e = cudaGetLastError())) return bfail(b, MSGPU_ERR_CUDA, std::string("batch: launch: ") + cudaGetErrorString(e));
    return MSGPU_OK;
}

// The resident kernels' forms of a system's H.  Without room for them in the
// memory budget the system takes the persistent launch (kind stays kNone).
void build_rows(msgpu_batch *b, BatchSystem &s, const int *rowptr, const int *col, const std::vector<float> &val, int max_row)
{
    const int D = s.D;
    const size_t slots = static_cast<size_t>(D) * max_row;
    if (slots == 0) return;
    std::vector<unsigned char> buf(slots * (sizeof(float2) + sizeof(int)) + D * sizeof(int), 0);
    float *v = reinterpret_cast<float *>(buf.data());
    int *c = reinterpret_cast<int *>(buf.data() + slots * sizeof(float2)), *n = c + slots;
    for (int r = 0; r < D; ++r) {
        n[r] = rowptr[r + 1] - rowptr[r];
        for (int k = 0; k < n[r]; ++k) {
            const size_t e = static_cast<size_t>(k) * D + r, from = rowptr[r] + k;
            v[2 * e] = val[2 * from];
            v[2 * e + 1] = val[2 * from + 1];
            c[e] = col[from];
        }
    }
    if (upload(b, s.ell, buf.data(), buf.size(), "rows") != MSGPU_OK) {
        (void)cudaGetLastError();
        b->err.clear();
        return;
    }
    s.kind = BatchSystem::kRows;
    s.kmax = max_row;
}

void build_quartets(msgpu_batch *b, BatchSystem &s, const int *rowptr, const int *col, const double *val)
{
    const int Q = s.D / 4;
    const QuartetForm f = quartet_form(s.D, s.s1, s.s2, rowptr, col, val, false, false);
    const QuartetSlots slots = quartet_slots(f);
    // one buffer: values (16-byte aligned), the resident arrays, blocks, row pointers, bases
    auto up = [](size_t n) { return (n + 15) / 16 * 16; };
    const size_t nval = up(f.val.size() * sizeof(float)), nrq = up(resident_q_bytes(Q, slots));
    const size_t nblk = up(f.blk.size() * sizeof(int2)), nrow = up(f.rowptr.size() * sizeof(int)), nbase = up(Q * sizeof(int));
    if (bensure(b, s.quart, nval + nrq + nblk + nrow + nbase, "quartets") != MSGPU_OK) {
        (void)cudaGetLastError();
        b->err.clear();
        return;
    }
    auto put = [&](size_t at, const void *from, size_t bytes) {
        return cudaMemcpyAsync(static_cast<unsigned char *>(s.quart.p) + at, from, bytes, cudaMemcpyHostToDevice, b->stream);
    };
    if (put(0, f.val.data(), f.val.size() * sizeof(float)) || put(nval + nrq, f.blk.data(), f.blk.size() * sizeof(int2)) ||
        put(nval + nrq + nblk, f.rowptr.data(), f.rowptr.size() * sizeof(int)) ||
        put(nval + nrq + nblk + nrow, f.base.data(), Q * sizeof(int)))
        return;
    unsigned char *p = static_cast<unsigned char *>(s.quart.p);
    s.rq = resident_q_build(p + nval, Q, s.s1, s.s2, slots, reinterpret_cast<const int *>(p + nval + nrq + nblk),
                            reinterpret_cast<const int2 *>(p + nval + nrq), reinterpret_cast<const float4 *>(p),
                            reinterpret_cast<const int *>(p + nval + nrq + nblk + nrow), b->stream);
    if (cudaGetLastError() != cudaSuccess) return;
    ++b->launches;
    s.kind = BatchSystem::kQuartets;
}

// The quartet forms that added systems still lack, all in one launch; a system whose
// blocks do not all get a slot there is assembled on the host from its CSR rows.
int assemble(msgpu_batch *b)
{
    std::vector<QuartetJob> jobs;
    std::vector<BatchSystem *> of;
    for (BatchSystem &s : b->sys)
        if (s.kind == BatchSystem::kUnassembled) {
            jobs.push_back(QuartetJob{static_cast<const int *>(s.rowptr.p), static_cast<const int *>(s.col.p),
                                      static_cast<const float2 *>(s.valf.p), s.quart.p, s.D, s.s1, s.s2});
            of.push_back(&s);
        }
    if (jobs.empty()) return MSGPU_OK;
    const size_t n = jobs.size();
    std::vector<QuartetFound> found(n);
    int rc;
    if ((rc = upload(b, b->jobs_d, jobs.data(), n * sizeof(QuartetJob), "quartet assembly")) ||
        (rc = bensure(b, b->found_d, n * sizeof(QuartetFound), "quartet assembly")))
        return rc;
    resident_q_assemble(static_cast<const QuartetJob *>(b->jobs_d.p), static_cast<int>(n),
                        static_cast<QuartetFound *>(b->found_d.p), b->stream);
    ++b->launches;
    if (cudaGetLastError() ||
        cudaMemcpyAsync(found.data(), b->found_d.p, n * sizeof(QuartetFound), cudaMemcpyDeviceToHost, b->stream) ||
        cudaStreamSynchronize(b->stream))
        return bfail(b, MSGPU_ERR_CUDA, "batch: quartet assembly failed");
    for (size_t i = 0; i < n; ++i) {
        BatchSystem &s = *of[i];
        if (found[i].nslot >= 0) {
            s.rq = resident_q_assembled(s.quart.p, s.D / 4, found[i]);
            s.kind = BatchSystem::kQuartets;
            continue;
        }
        std::vector<int> rowptr(s.D + 1);
        if (cudaMemcpyAsync(rowptr.data(), s.rowptr.p, sizeof(int) * rowptr.size(), cudaMemcpyDeviceToHost, b->stream) ||
            cudaStreamSynchronize(b->stream))
            return bfail(b, MSGPU_ERR_CUDA, "batch: quartet assembly failed");
        const size_t nnz = rowptr[s.D];
        std::vector<int> col(nnz);
        std::vector<float> valf(2 * nnz);
        if (cudaMemcpyAsync(col.data(), s.col.p, sizeof(int) * nnz, cudaMemcpyDeviceToHost, b->stream) ||
            cudaMemcpyAsync(valf.data(), s.valf.p, sizeof(float) * valf.size(), cudaMemcpyDeviceToHost, b->stream) ||
            cudaStreamSynchronize(b->stream))
            return bfail(b, MSGPU_ERR_CUDA, "batch: quartet assembly failed");
        const std::vector<double> val(valf.begin(), valf.end());
        s.kind = BatchSystem::kNone;
        build_quartets(b, s, rowptr.data(), col.data(), val.data());
    }
    return MSGPU_OK;
}

int set_times(msgpu_batch *b, const double *times, int ntimes)
{
    for (int s = 0; s < ntimes; ++s)
        if (!std::isfinite(times[s]) || (s > 0 && !(times[s] > times[s - 1])))
            return bfail(b, MSGPU_ERR_INVALID, "batch: times must be finite and strictly increasing");
    if (int rc = upload(b, b->times_d, times, sizeof(double) * ntimes, "times")) return rc;
    std::vector<double> pf(ntimes, 0.0);
    for (auto &s : b->sys) {
        if (s.ctx) continue;
        for (int k = 0; k + 1 < ntimes; ++k) pf[k] = flip_prob(s.st_rate, 0.5 * (times[k + 1] - times[k]));
        if (int rc = upload(b, s.pflip, pf.data(), sizeof(double) * ntimes, "flip probabilities")) return rc;
    }
    return MSGPU_OK;
}

int run_once(msgpu_batch *b, int ntimes, int m, int accumulate, long long step_offset, int threshold, int cps,
             bool graph, float *ms, const double *times = nullptr)
{
    int grid, nlarge, nitems;
    size_t slice, smem;
    std::vector<ResidentRun> resident;
    if (int rc = prepare(b, ntimes, m, accumulate, step_offset, threshold, cps, &grid, &slice, &smem, &nlarge, &nitems,
                         &resident))
        return rc;
    const bool here = nitems > 0 || !resident.empty();
    std::vector<int> routed;  // streamed systems (times given: a real run, not a tuning probe)
    if (times)
        for (size_t i = 0; i < b->sys.size(); ++i)
            if (b->sys[i].ctx) routed.push_back(static_cast<int>(i));
    const auto w0 = std::chrono::steady_clock::now();
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, b->stream);
    int rc = MSGPU_OK;
    if (here && cudaMemsetAsync(b->status_d.p, 0, sizeof(int), b->stream) != cudaSuccess)
        rc = bfail(b, MSGPU_ERR_CUDA, "batch: status reset failed");
    if (!rc) rc = launch_resident(b, resident, static_cast<int>(routed.size()));
    if (!rc && nitems > 0) rc = launch(b, grid, slice, smem, nlarge, nitems, m, graph);
    if (nitems > 0) b->launches += graph ? 1 : 2;  // a replay of the captured graph, or memset + kernel
    cudaEventRecord(e1, b->stream);
    // the streamed systems, each on its own context and stream, while the others run
    std::vector<int> rcs(routed.size(), MSGPU_OK);
    if (!routed.empty() && rc == MSGPU_OK) {
        msgpu_run_params p;
        std::memset(&p, 0, sizeof(p));
        p.times = times;
        p.ntimes = ntimes;
        p.krylov_dim = m;
        p.precision = MSGPU_PREC_C64;
        p.recurrence = MSGPU_REC_AUTO;
        p.propagator = MSGPU_PROP_KRYLOV;
        p.step_offset = step_offset;
        p.accumulate = accumulate;
        std::atomic<size_t> next{0};
        auto worker = [&]() {
            for (size_t k; (k = next.fetch_add(1)) < routed.size();) rcs[k] = msgpu_run(b->sys[routed[k]].ctx, &p);
        };
        std::vector<std::thread> pool;
        const int nw = std::min<int>(kStreamWorkers, static_cast<int>(routed.size()));
        for (int i = 0; i < nw; ++i) pool.emplace_back(worker);
        for (auto &th : pool) th.join();
        cudaSetDevice(b->device);
    }
    cudaError_t e = cudaEventSynchronize(e1);
    float t = 0.f;
    cudaEventElapsedTime(&t, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc) return rc;
    if (e) return bfail(b, MSGPU_ERR_CUDA, std::string("batch: run: ") + cudaGetErrorString(e));
    for (size_t k = 0; k < routed.size(); ++k)
        if (rcs[k])
            return bfail(b, rcs[k], "batch: system " + std::to_string(routed[k]) + ": " +
                                        msgpu_last_error(b->sys[routed[k]].ctx));
    int status = 0;
    if (here && (e = cudaMemcpy(&status, b->status_d.p, sizeof(int), cudaMemcpyDeviceToHost)))
        return bfail(b, MSGPU_ERR_CUDA, std::string("batch: status: ") + cudaGetErrorString(e));
    if (status & 2) return bfail(b, MSGPU_ERR_NONFINITE, "batch: non-finite observable on the device");
    if (status & 1) return bfail(b, MSGPU_ERR_EXPM, "batch: small matrix exponential failed");
    // persistent launch alone: its device time; with streamed systems: the
    // wall time of the whole run (host threads, several streams)
    if (ms)
        *ms = routed.empty() ? t
                             : std::chrono::duration<float, std::milli>(std::chrono::steady_clock::now() - w0).count();
    return MSGPU_OK;
}

}  // namespace

extern "C" {

msgpu_batch *msgpu_batch_create(int device, size_t hbm_budget_bytes)
{
    if (cudaSetDevice(device) != cudaSuccess) return nullptr;
    auto *b = new msgpu_batch();
    b->device = device;
    b->budget = hbm_budget_bytes;
    cudaDeviceGetAttribute(&b->sm_count, cudaDevAttrMultiProcessorCount, device);
    if (cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking) != cudaSuccess) {
        delete b;
        return nullptr;
    }
    return b;
}

void msgpu_batch_destroy(msgpu_batch *b)
{
    if (!b) return;
    cudaSetDevice(b->device);
    cudaStreamSynchronize(b->stream);
    drop_graph(b);
    for (auto *list : {&b->sys, &b->spare})
        for (auto &s : *list) {
            Buf *all[] = {&s.rowptr, &s.col, &s.valf, &s.obs, &s.rates, &s.psi, &s.acc, &s.comp, &s.prev, &s.pflip, &s.ell, &s.quart};
            for (Buf *x : all) brelease(b, *x);
            if (s.ctx) msgpu_destroy(s.ctx);
        }
    Buf *all[] = {&b->sys_d, &b->items_d, &b->queue_d, &b->status_d, &b->scratch, &b->times_d, &b->backup, &b->many_d, &b->first_d,
                  &b->jobs_d, &b->found_d};
    for (Buf *x : all) brelease(b, *x);
    for (int k = 0; k < 8; ++k) {
        if (b->join[k]) cudaEventDestroy(b->join[k]);
        if (b->side[k]) cudaStreamDestroy(b->side[k]);
    }
    if (b->fork) cudaEventDestroy(b->fork);
    cudaStreamDestroy(b->stream);
    delete b;
}

const char *msgpu_batch_last_error(const msgpu_batch *b) { return b ? b->err.c_str() : "null batch"; }

int msgpu_batch_clear(msgpu_batch *b)
{
    if (!b) return MSGPU_ERR_INVALID;
    cudaSetDevice(b->device);
    if (cudaStreamSynchronize(b->stream) != cudaSuccess) return bfail(b, MSGPU_ERR_CUDA, "batch: clear: stream failed");
    drop_graph(b);
    for (auto &s : b->sys) {
        if (s.ctx) {
            msgpu_destroy(s.ctx);  // a streamed system's context goes with it
            s.ctx = nullptr;
        } else {
            b->spare.push_back(s);
        }
    }
    b->sys.clear();
    b->tuned = 0;
    return MSGPU_OK;
}

int msgpu_batch_add_system(msgpu_batch *b, int dim, const int *rowptr, const int *col, const double *val,
                           double kappa, int stride1, int stride2, int nobs, const double *ops, const double *rates,
                           double st_rate, unsigned long long seed, int ntraj, const double *factors)
{
    if (!b) return -MSGPU_ERR_INVALID;
    if (dim < 4 || dim % 4 || !rowptr || !col || !val || ntraj <= 0 || !factors || nobs < 1 || nobs > 8 || !ops ||
        !rates || !std::isfinite(kappa) || !(st_rate >= 0.0))
        return -bfail(b, MSGPU_ERR_INVALID, "batch: invalid system arguments");
    const int hi = std::max(stride1, stride2), lo = std::min(stride1, stride2);
    if (lo <= 0 || hi == lo || hi % (2 * lo) || dim % (2 * hi))
        return -bfail(b, MSGPU_ERR_INVALID, "batch: electron strides do not belong to two spin-1/2 digits");
    cudaSetDevice(b->device);
    for (int k = 0; k < rowptr[dim]; ++k)
        if (col[k] < 0 || col[k] >= dim || !std::isfinite(val[2 * k]) || !std::isfinite(val[2 * k + 1]))
            return -bfail(b, MSGPU_ERR_INVALID, "batch: malformed Hamiltonian");
    if (dim >= kStreamDim) {
        // streamed single-system path: own context (charged to the batch budget)
        const size_t room = b->budget ? (b->budget > b->used ? b->budget - b->used : 1) : 0;
        msgpu_ctx *c = msgpu_create(b->device, room);
        if (!c) return -bfail(b, MSGPU_ERR_CUDA, "batch: cannot create a context for a large system");
        int rc = msgpu_upload_hamiltonian_csr(c, dim, rowptr, col, val);
        if (!rc) rc = msgpu_set_reaction_scalar(c, kappa);
        if (!rc) rc = msgpu_set_electron_pair(c, stride1, stride2);
        for (int o = 0; o < nobs && !rc; ++o) rc = msgpu_add_pair_observable(c, ops + 32 * static_cast<size_t>(o), rates[o]);
        if (!rc && st_rate > 0.0) rc = msgpu_set_st_noise(c, st_rate, MSGPU_NOISE_PHILOX, seed, nullptr, 0, 0);
        if (!rc) rc = msgpu_upload_factors(c, dim, ntraj, factors);
        if (rc) {
            const std::string why = msgpu_last_error(c);
            msgpu_destroy(c);
            return -bfail(b, rc, "batch: " + why);
        }
        BatchSystem s;
        s.D = dim;
        s.M = ntraj;
        s.nobs = nobs;
        s.s1 = std::max(stride1, stride2);
        s.s2 = std::min(stride1, stride2);
        s.kappa = kappa;
        s.st_rate = st_rate;
        s.seed = seed;
        s.ctx = c;
        b->sys.push_back(s);
        drop_graph(b);
        b->tuned = 0;
        return static_cast<int>(b->sys.size()) - 1;
    }
    BatchSystem s;
    if (!b->spare.empty()) {  // reuse a cleared system's buffers (upload keeps those large enough)
        s = b->spare.back();
        b->spare.pop_back();
    }
    s.D = dim;
    s.M = ntraj;
    s.nobs = nobs;
    s.s1 = hi;
    s.s2 = lo;
    s.kappa = kappa;
    s.st_rate = st_rate;
    s.seed = seed;
    const int nnz = rowptr[dim];
    std::vector<float> vf(2 * static_cast<size_t>(nnz));
    for (size_t i = 0; i < vf.size(); ++i) vf[i] = static_cast<float>(val[i]);
    // observables in the kernel pair basis (first digit = larger stride)
    const bool swapped = stride1 < stride2;
    const int perm[4] = {0, 2, 1, 3};
    std::vector<double> op(static_cast<size_t>(nobs) * 32);
    for (int o = 0; o < nobs; ++o)
        for (int a = 0; a < 4; ++a)
            for (int c = 0; c < 4; ++c) {
                const int ua = swapped ? perm[a] : a, uc = swapped ? perm[c] : c;
                op[o * 32 + 2 * (a * 4 + c)] = ops[o * 32 + 2 * (ua * 4 + uc)];
                op[o * 32 + 2 * (a * 4 + c) + 1] = ops[o * 32 + 2 * (ua * 4 + uc) + 1];
            }
    s.kind = BatchSystem::kNone;
    int max_row = 0;
    bool ascending = true;  // a column once in every row, then
    for (int r = 0; r < dim; ++r) {
        max_row = std::max(max_row, rowptr[r + 1] - rowptr[r]);
        for (int k = rowptr[r] + 1; k < rowptr[r + 1]; ++k) ascending = ascending && col[k] > col[k - 1];
    }
    if (dim <= 128) build_rows(b, s, rowptr, col, vf, max_row);
    // quartets: assembled on the device from the CSR rows, or here; the CSR rows stay
    // for a Krylov dimension whose basis does not fit shared memory
    const bool here = resident_q_takes(dim) && (max_row > kAssembleRow || !ascending);
    if (here && resident_shape_q_many(dim, kMaxKrylov).smem <= kResidentSmemMax) build_quartets(b, s, rowptr, col, val);
    std::vector<float> psi(2 * static_cast<size_t>(dim) * ntraj);
    for (size_t i = 0; i < psi.size(); ++i) psi[i] = static_cast<float>(factors[i]);
    const size_t sums = sizeof(double) * nobs * static_cast<size_t>(ntraj);
    int rc;
    if ((s.kind == BatchSystem::kNone && (rc = upload_csr(b, s, rowptr, col, vf))) ||
        (rc = upload(b, s.obs, op.data(), sizeof(double) * op.size(), "observables")) ||
        (rc = upload(b, s.rates, rates, sizeof(double) * nobs, "rates")) ||
        (rc = upload(b, s.psi, psi.data(), sizeof(float) * psi.size(), "factors")) ||
        (rc = bensure(b, s.acc, sums, "acc")) || (rc = bensure(b, s.comp, sums, "comp")) ||
        (rc = bensure(b, s.prev, sums, "prev"))) {
        b->spare.push_back(s);  // its buffers are freed with the batch
        return -rc;
    }
    for (Buf *x : {&s.acc, &s.comp, &s.prev})
        if (cudaMemsetAsync(x->p, 0, sums, b->stream) != cudaSuccess) {
            b->spare.push_back(s);
            return -bfail(b, MSGPU_ERR_CUDA, "batch: upload failed");
        }
    if (resident_q_takes(dim) && s.kind == BatchSystem::kNone) {
        if (here) {
            build_quartets(b, s, rowptr, col, val);
        } else if (bensure(b, s.quart, resident_q_assembled_bytes(dim / 4), "quartets") == MSGPU_OK) {
            s.kind = BatchSystem::kUnassembled;
        } else {  // no room: the persistent launch
            (void)cudaGetLastError();
            b->err.clear();
        }
    }
    if (cudaStreamSynchronize(b->stream) != cudaSuccess) {
        b->spare.push_back(s);
        return -bfail(b, MSGPU_ERR_CUDA, "batch: upload failed");
    }
    b->sys.push_back(s);
    drop_graph(b);
    b->tuned = 0;
    return static_cast<int>(b->sys.size()) - 1;
}

int msgpu_batch_tune(msgpu_batch *b, const double *times, int ntimes, int krylov_dim)
{
    if (!b) return MSGPU_ERR_INVALID;
    if (b->sys.empty() || !times || ntimes < 2 || krylov_dim < 1 || krylov_dim > kMaxKrylov)
        return bfail(b, MSGPU_ERR_INVALID, "batch: tune needs systems, >= 2 time points and krylov_dim in 1..32");
    cudaSetDevice(b->device);
    // back up every state, time a short run per candidate, restore
    size_t total = 0;
    for (auto &s : b->sys) total += s.psi.bytes;  // streamed systems hold no state here
    if (int rc = bensure(b, b->backup, total, "tuning backup")) return rc;
    size_t off = 0;
    for (auto &s : b->sys) {
        if (!s.psi.bytes) continue;
        cudaMemcpyAsync(static_cast<char *>(b->backup.p) + off, s.psi.p, s.psi.bytes, cudaMemcpyDeviceToDevice, b->stream);
        off += s.psi.bytes;
    }
    if (int rc = set_times(b, times, ntimes)) return rc;
    if (int rc = assemble(b)) return rc;
    const int thresholds[] = {256, 512, 1024, 2048};
    const int cps[] = {1, 2, 3, 4};
    float best = 1e30f;
    bool persistent = false;  // any system on the persistent launch, which these parameters shape
    for (auto &s : b->sys) {
        const int m = std::min(krylov_dim, s.D);
        persistent = persistent || (!s.ctx && !(s.kind != BatchSystem::kNone && (s.kind == BatchSystem::kRows ? resident_shape_many(s.D, m).smem
                                                                       : resident_shape_q_many(s.D, m).smem) <= kResidentSmemMax));
    }
    for (int th : thresholds)
        for (int c : cps) {
            if (!persistent) break;
            float ms = 0.f;
            if (int rc = run_once(b, ntimes, krylov_dim, 0, 0, th, c, false, &ms)) return rc;
            if (ms < best) {
                best = ms;
                b->threshold = th;
                b->ctas_per_sm = c;
            }
        }
    off = 0;
    for (auto &s : b->sys) {
        if (!s.psi.bytes) continue;
        cudaMemcpyAsync(s.psi.p, static_cast<char *>(b->backup.p) + off, s.psi.bytes, cudaMemcpyDeviceToDevice, b->stream);
        off += s.psi.bytes;
    }
    brelease(b, b->backup);
    if (cudaStreamSynchronize(b->stream) != cudaSuccess) return bfail(b, MSGPU_ERR_CUDA, "batch: restore failed");
    b->tuned = 1;
    drop_graph(b);
    return MSGPU_OK;
}

int msgpu_batch_run(msgpu_batch *b, const double *times, int ntimes, int krylov_dim, long long step_offset,
                    int accumulate)
{
    if (!b) return MSGPU_ERR_INVALID;
    if (b->sys.empty() || !times || ntimes < 1 || krylov_dim < 1 || krylov_dim > kMaxKrylov)
        return bfail(b, MSGPU_ERR_INVALID, "batch: run needs systems, time points and krylov_dim in 1..32");
    cudaSetDevice(b->device);
    if (int rc = set_times(b, times, ntimes)) return rc;
    if (int rc = assemble(b)) return rc;
    b->m = krylov_dim;
    return run_once(b, ntimes, krylov_dim, accumulate, step_offset, b->threshold, b->ctas_per_sm, true, &b->last_ms,
                    times);
}

int msgpu_batch_fetch_yields(msgpu_batch *b, int system, double *per_traj, double *ensemble)
{
    if (!b) return MSGPU_ERR_INVALID;
    if (system < 0 || system >= static_cast<int>(b->sys.size())) return bfail(b, MSGPU_ERR_INVALID, "batch: no such system");
    BatchSystem &s = b->sys[system];
    if (s.ctx) {
        const int rc = msgpu_fetch_yields(s.ctx, per_traj, ensemble);
        return rc ? bfail(b, rc, std::string("batch: ") + msgpu_last_error(s.ctx)) : MSGPU_OK;
    }
    std::vector<double> acc(static_cast<size_t>(s.nobs) * s.M);
    if (cudaMemcpy(acc.data(), s.acc.p, sizeof(double) * acc.size(), cudaMemcpyDeviceToHost) != cudaSuccess)
        return bfail(b, MSGPU_ERR_CUDA, "batch: fetch failed");
    for (int o = 0; o < s.nobs; ++o) {
        double sum = 0.0;
        for (int t = 0; t < s.M; ++t) {
            const double v = acc[static_cast<size_t>(o) * s.M + t];
            if (per_traj) per_traj[static_cast<size_t>(t) * s.nobs + o] = v;
            sum += v;
        }
        if (ensemble) ensemble[o] = sum;
    }
    return MSGPU_OK;
}

long long msgpu_batch_launch_count(const msgpu_batch *b)
{
    if (!b) return 0;
    long long n = b->launches;
    for (const auto &s : b->sys)
        if (s.ctx) n += msgpu_launch_count(s.ctx);
    return n;
}

int msgpu_batch_system_info(const msgpu_batch *b, int i, int *streamed, int *variant, int *tile, int *groups)
{
    if (!b || i < 0 || i >= static_cast<int>(b->sys.size())) return MSGPU_ERR_INVALID;
    const BatchSystem &s = b->sys[i];
    if (streamed) *streamed = s.ctx ? 1 : 0;
    if (s.ctx) return msgpu_spmm_choice(s.ctx, variant, tile, groups);
    if (variant) *variant = -1;
    if (tile) *tile = -1;
    if (groups) *groups = -1;
    return MSGPU_OK;
}

int msgpu_batch_stats(const msgpu_batch *b, double *last_run_ms, int *team_threshold, int *ctas_per_sm)
{
    if (!b) return MSGPU_ERR_INVALID;
    if (last_run_ms) *last_run_ms = b->last_ms;
    if (team_threshold) *team_threshold = b->threshold;
    if (ctas_per_sm) *ctas_per_sm = b->ctas_per_sm;
    return MSGPU_OK;
}

}  // extern "C"
