// engine.cu -- batched Foldy-Lax engine: persistent kernels over a device
// work queue, the runtime (device, workspace, jobs) and the msgpu_* C ABI.
//
// A team (one CTA, or a cluster of CTAs where the batch would leave SMs idle)
// takes the next (k, realisation) item from an atomic counter, assembles M(k)
// (and dM/dk) into its slot of the workspace, factors it and reduces the
// trace-log or the trace of M^-1 dM/dk, then takes the next item.  Items are dealt largest-n first, so uneven sizes balance.
#include <cuda_runtime.h>
#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "msgpu.h"
#include "fp64_engine.cuh"
#include "green_df.cuh"

using namespace msg;

namespace msg {

// Two CTAs of 256 threads per SM, every update on the FP64 pipe.
__global__ void __launch_bounds__(NT, 2) k_engine_fp64(EngineParams P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    run_items_fp64(P, *reinterpret_cast<LuSmem*>(smem_raw), this_team(), DfmaUpdate{});
}

// Four CTAs of 128 threads per SM, tiles of 32 rows: jobs of small matrices that
// fill the chip.  Such a matrix is a chain of short steps with the FP64 pipe idle
// in between; four of them interleave where two did.
constexpr int SMALL_NT = 128, SMALL_CTAS = 4;
using SmallSmem = LuSmemT<SMALL_NT, 32>;
__global__ void __launch_bounds__(SMALL_NT, SMALL_CTAS) k_engine_fp64_small(EngineParams P) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    run_items_fp64(P, *reinterpret_cast<SmallSmem*>(smem_raw), this_team(), DfmaUpdate{});
}

// single-matrix assembly for the drop-in layer (build_matrix.cu)
__global__ void __launch_bounds__(NT, 1) k_build_matrix(zc* A, int n, int d, const double* pos, msgpu_model m,
                                                        double kre, double kim, int deriv);

// device special functions for the checks against the reference goldens (special.cu)
__global__ void k_eval_special(int which, int d, msgpu_model m, int n, const double* ks, const double* rs,
                               double* out);

// FP64 FMA throughput probe: 8 independent chains per thread; the roofline
// denominator of the plain (FP64-pipe-bound) path.
__global__ void k_probe_dfma(double* sink, int iters, double a, double b) {
    double x0 = threadIdx.x, x1 = x0 + 1, x2 = x0 + 2, x3 = x0 + 3, x4 = x0 + 4, x5 = x0 + 5, x6 = x0 + 6,
           x7 = x0 + 7;
    for (int i = 0; i < iters; ++i) {
        x0 = fma(x0, a, b); x1 = fma(x1, a, b); x2 = fma(x2, a, b); x3 = fma(x3, a, b);
        x4 = fma(x4, a, b); x5 = fma(x5, a, b); x6 = fma(x6, a, b); x7 = fma(x7, a, b);
    }
    double s = x0 + x1 + x2 + x3 + x4 + x5 + x6 + x7;
    if (s == 12345.678) sink[blockIdx.x] = s;
}

// FP64 tensor-core throughput probe: 8 independent accumulators per warp of the
// warp-level m8n8k4 FP64 MMA (512 flops each), the other candidate of the FP64 path
__global__ void k_probe_dmma(double* sink, int iters, double a, double b) {
    double c[8][2];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
        c[u][0] = threadIdx.x + u;
        c[u][1] = 0.5 * u;
    }
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int u = 0; u < 8; ++u)
            asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                         : "+d"(c[u][0]), "+d"(c[u][1])
                         : "d"(a), "d"(b));
    }
    double s = 0.0;
#pragma unroll
    for (int u = 0; u < 8; ++u) s += c[u][0] + c[u][1];
    if (s == 12345.678) sink[blockIdx.x] = s;
}

}  // namespace msg

// ---------------------------------------------------------------------------
// runtime
// ---------------------------------------------------------------------------
namespace {

std::mutex g_mu;
std::string g_err;
int g_dev = -1;
int g_sms = 0;
int g_ctas_fp64 = 0;
int g_teams[2][5] = {};  // FP64 kernels (0: FP64 pipe, 1: tensor cores): clusters of 2^j CTAs the device holds at once
std::atomic<uint64_t> g_launches{0};
void* g_ws = nullptr;
size_t g_ws_bytes = 0;
unsigned long long g_ws_gen = 1;  // changes whenever g_ws moves (captured graphs hold its address)

// Launch choices per (kind, requested precision, size bucket): the engine that
// runs (a mixed request may be served by the FP64 engine, which is at least as
// accurate) and the resident CTAs per SM of the persistent grid.  0 = default
// (the requested engine, as many CTAs as fit).  Filled by msgpu_autotune or
// msgpu_tune_set; bucket b holds nmax in (2^(b-1), 2^b].
struct TuneEntry {
    int engine = 0;  // 0 default, 1 + MSGPU_FP64 / 1 + MSGPU_MIXED
    int ctas = 0;
};
constexpr int TUNE_BUCKETS = 17;
TuneEntry g_tune[3][2][TUNE_BUCKETS];

int size_bucket(int n) {
    int b = 0;
    while ((1 << b) < n && b < TUNE_BUCKETS - 1) ++b;
    return b;
}

int set_err(int code, const std::string& msg) {
    g_err = msg;
    return code;
}

#define CK(call)                                                                              \
    do {                                                                                      \
        cudaError_t e_ = (call);                                                              \
        if (e_ != cudaSuccess) return set_err(MSGPU_E_CUDA, std::string(#call) + ": " + cudaGetErrorString(e_)); \
    } while (0)

size_t smem_bytes() { return sizeof(LuSmem); }

int init_locked(int device) {
    if (g_dev >= 0) return 0;
    int ndev = 0;
    if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) return set_err(MSGPU_E_NODEV, "no CUDA device");
    if (device < 0) device = 0;
    CK(cudaSetDevice(device));
    cudaDeviceProp pr;
    CK(cudaGetDeviceProperties(&pr, device));
    g_sms = pr.multiProcessorCount;
    CK(cudaFuncSetAttribute(k_engine_fp64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes()));
    CK(cudaFuncSetAttribute(k_engine_fp64_small, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SmallSmem)));
    CK(cudaFuncSetAttribute(k_build_matrix, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes()));
    int occ = 0;
    CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k_engine_fp64, NT, smem_bytes()));
    g_ctas_fp64 = std::max(1, occ);
    CK(cudaFuncSetAttribute(k_engine_fp64, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    for (int j = 0; j < 5; ++j) {
        g_teams[0][j] = max_teams(k_engine_fp64, 1 << j, NT, smem_bytes());
        g_teams[1][j] = tc64_max_teams(1 << j);
    }
    g_teams[0][0] = g_sms * g_ctas_fp64;
    g_teams[1][0] = g_sms;
    g_dev = device;
    return 0;
}

void pool_trim();

int ensure_ws(size_t bytes, void** p) {
    if (bytes > g_ws_bytes) {
        if (g_ws) cudaFree(g_ws);
        g_ws = nullptr;
        g_ws_bytes = 0;
        ++g_ws_gen;
        if (cudaMalloc(&g_ws, bytes) != cudaSuccess) {
            cudaGetLastError();
            pool_trim();
            CK(cudaMalloc(&g_ws, bytes));
        }
        g_ws_bytes = bytes;
    }
    *p = g_ws;
    return 0;
}

// Device blocks of finished jobs, kept for the next ones: a job's arrays are one
// block, and cudaMalloc / cudaFree of a dozen of them took 0.8 of the 1.4 ms of
// a one-item call at n = 50.  At most POOL_BLOCKS blocks and POOL_BYTES in all;
// a block goes back to the driver when the pool is full or an allocation fails.
// Blocks change hands under g_mu, and only after the job's runs have completed.
struct PoolBlock {
    void* p;
    size_t bytes;
};
constexpr size_t POOL_BLOCKS = 8, POOL_BYTES = (size_t)64 << 20;
std::vector<PoolBlock> g_pool;

void pool_trim() {
    for (auto& b : g_pool) cudaFree(b.p);
    g_pool.clear();
}

// a block of at least `bytes` (rounded up in place); nullptr if the device has none
void* pool_get(size_t& bytes) {
    size_t want = (size_t)64 << 10;
    while (want < bytes && want < POOL_BYTES) want <<= 1;
    if (want < bytes) want = bytes;
    bytes = want;
    for (size_t i = 0; i < g_pool.size(); ++i)
        if (g_pool[i].bytes == want) {
            void* p = g_pool[i].p;
            g_pool.erase(g_pool.begin() + i);
            return p;
        }
    void* p = nullptr;
    if (cudaMalloc(&p, want) == cudaSuccess) return p;
    cudaGetLastError();
    pool_trim();
    if (cudaMalloc(&p, want) == cudaSuccess) return p;
    cudaGetLastError();
    return nullptr;
}

void pool_put(void* p, size_t bytes) {
    if (!p) return;
    size_t held = bytes;
    for (auto& b : g_pool) held += b.bytes;
    if (g_pool.size() >= POOL_BLOCKS || held > POOL_BYTES) cudaFree(p);
    else g_pool.push_back({p, bytes});
}

}  // namespace

// workspace budget for the per-CTA matrix slots
static size_t ws_budget() {
    size_t fr = 0, tot = 0;
    cudaMemGetInfo(&fr, &tot);
    size_t cap = (size_t)160 << 30;
    size_t avail = fr + g_ws_bytes;
    return std::min(cap, avail > ((size_t)4 << 30) ? avail - ((size_t)4 << 30) : avail / 2);
}

static int ilog2(int v) {
    int j = 0;
    while ((2 << j) <= v) ++j;
    return j;
}

// CTAs per matrix: the team size whose estimated time is least.  A matrix
// takes a part s of its time in steps one CTA does (the panels) and 1 - s in
// steps the team shares; the items go in waves of as many teams as the device
// holds at once (teams[j] of 2^j CTAs), CTAs that share an SM `share` slower.
static int pick_team(const int* teams, double s, double share, int nitem, int nmax) {
    int best = 1;
    double t_best = 0.0;
    for (int j = 0; j < 5; ++j) {
        const int team = 1 << j, held = teams[j];
        if (held < 1 || (team > 1 && nmax < 6 * team)) break;
        const double waves = (nitem + held - 1) / held;
        const double t = waves * ((double)std::min(nitem, held) * team > g_sms ? share : 1.0) * (s + (1.0 - s) / team);
        if (j == 0 || t < 0.95 * t_best) {
            best = team;
            t_best = t;
        }
    }
    return best;
}
static int pick_team_fp64(bool tc, int nitem, int nmax) {
    return pick_team(g_teams[tc], tc ? 0.2 : 0.3, tc ? 1.0 : 1.6, nitem, nmax);
}

struct msgpu_job {
    int kind = 0, precision = 0, nitem = 0, nmed = 0, nmax = 0;
    int cap = 0;  // item capacity of the device arrays
    double flops = 0.0;
    int grid = 0;
    std::vector<int> med_n;  // n of every medium (host copy)
    // mixed engine: per medium the smallest and largest pair distance (d = 3 with the
    // "maximum" model), or a negative smallest distance where the entry span is not predicted
    std::vector<double> med_rmin, med_rmax;
    bool wide = false;       // some item may need six-way slicing (sticky: captured graphs keep it)
    bool warm = false;       // kind 4: inverse iterations start from the vectors set by msgpu_job_set_vectors
    bool d3only = true;      // every medium has d = 3
    // the job's device arrays, all in one block
    void* block = nullptr;
    size_t block_bytes = 0;
    std::atomic<unsigned> runs{0}, done{0};  // runs queued, and how many of them are known to be over
    bool captured = false;   // a run went into a graph of the caller's, which may replay it at any time
    MedDev* d_media = nullptr;
    double* d_pos = nullptr;
    size_t items_b = 0;      // bytes from d_ks to the live count: the item arrays at full capacity
    double* d_ks = nullptr;
    int* d_item_med = nullptr;
    int* d_order = nullptr;
    double* d_out = nullptr;
    int* d_status = nullptr;
    unsigned* d_counter = nullptr;  // [0] work queue, [1] live items
    int* d_piv = nullptr;
    size_t slot = 0;
    size_t ws_bytes = 0;
    bool small = false;      // FP64: the kernel for small matrices
    bool tc = false;         // FP64: the kernel whose trailing updates run on the tensor cores
    int team = 1;            // CTAs that share one matrix
    size_t img_off = 0;      // tc: offset of the operand images in the workspace
    long long amp_total = 0, amp_cap = 0;
    double* d_amps = nullptr;
    long long* d_amp_off = nullptr;
    // graph mode: the run (queue reset + engine launch) captured once and replayed
    bool use_graph = false;
    cudaStream_t cap_stream = nullptr;
    cudaGraphExec_t gexec = nullptr;
    unsigned long long gen = 0;
};

extern "C" {

}  // extern "C"

namespace msg {
void count_launches(int n) { g_launches += n; }
// for entry points outside this file's lock (the allocation-free and eigenvalue entries)
int record_error(int code, const char* what) {
    std::lock_guard<std::mutex> lk(g_mu);
    return set_err(code, what);
}
}  // namespace msg

extern "C" {

int msgpu_init(int device) {
    std::lock_guard<std::mutex> lk(g_mu);
    return init_locked(device);
}

const char* msgpu_last_error(void) { return g_err.c_str(); }

int msgpu_sm_count(void) {
    std::lock_guard<std::mutex> lk(g_mu);
    if (init_locked(-1)) return 0;
    return g_sms;
}

uint64_t msgpu_launch_count(void) { return g_launches.load(); }

int msgpu_probe_fp64(double* tflops) {
    std::lock_guard<std::mutex> lk(g_mu);
    if (int e = init_locked(-1)) return e;
    double* sink = nullptr;
    CK(cudaMalloc(&sink, sizeof(double) * 4096));
    cudaEvent_t e0, e1;
    CK(cudaEventCreate(&e0));
    CK(cudaEventCreate(&e1));
    const int blocks = g_sms * 4, threads = 256, iters = 8192;
    k_probe_dfma<<<blocks, threads>>>(sink, 64, 0.999999, 1e-7);  // warm-up
    g_launches++;
    CK(cudaEventRecord(e0));
    k_probe_dfma<<<blocks, threads>>>(sink, iters, 0.999999, 1e-7);
    g_launches++;
    CK(cudaEventRecord(e1));
    CK(cudaEventSynchronize(e1));
    float ms = 0.f;
    CK(cudaEventElapsedTime(&ms, e0, e1));
    *tflops = 2.0 * 8.0 * iters * (double)blocks * threads / (ms * 1e-3) / 1e12;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(sink);
    return 0;
}

int msgpu_probe_fp64_mma(double* tflops) {
    std::lock_guard<std::mutex> lk(g_mu);
    if (int e = init_locked(-1)) return e;
    double* sink = nullptr;
    CK(cudaMalloc(&sink, sizeof(double) * 4096));
    cudaEvent_t e0, e1;
    CK(cudaEventCreate(&e0));
    CK(cudaEventCreate(&e1));
    const int blocks = g_sms * 4, threads = 256, iters = 2048;
    k_probe_dmma<<<blocks, threads>>>(sink, 16, 0.999999, 1e-7);  // warm-up
    g_launches++;
    CK(cudaEventRecord(e0));
    k_probe_dmma<<<blocks, threads>>>(sink, iters, 0.999999, 1e-7);
    g_launches++;
    CK(cudaEventRecord(e1));
    CK(cudaEventSynchronize(e1));
    float ms = 0.f;
    CK(cudaEventElapsedTime(&ms, e0, e1));
    // 512 flops per warp-level MMA, 8 per warp and iteration
    *tflops = 512.0 * 8.0 * iters * (double)blocks * (threads / 32) / (ms * 1e-3) / 1e12;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(sink);
    return 0;
}

int msgpu_eval_special(int which, int d, const msgpu_model* model, int n, const double* ks, const double* rs,
                       double* out) {
    std::lock_guard<std::mutex> lk(g_mu);
    if (int e = init_locked(-1)) return e;
    if (n <= 0) return 0;
    msgpu_model m{};
    if (model) m = *model;
    double *dk = nullptr, *dr = nullptr, *dout = nullptr;
    CK(cudaMalloc(&dk, sizeof(double) * 2 * n));
    CK(cudaMalloc(&dout, sizeof(double) * 2 * n));
    if (rs) CK(cudaMalloc(&dr, sizeof(double) * n));
    CK(cudaMemcpy(dk, ks, sizeof(double) * 2 * n, cudaMemcpyHostToDevice));
    if (rs) CK(cudaMemcpy(dr, rs, sizeof(double) * n, cudaMemcpyHostToDevice));
    k_eval_special<<<(n + 127) / 128, 128>>>(which, d, m, n, dk, dr, dout);
    g_launches++;
    CK(cudaGetLastError());
    CK(cudaMemcpy(out, dout, sizeof(double) * 2 * n, cudaMemcpyDeviceToHost));
    cudaFree(dk);
    cudaFree(dout);
    if (dr) cudaFree(dr);
    return 0;
}

int msgpu_build_matrix(const msgpu_medium* med, const double* k, int deriv, double* mat) {
    std::lock_guard<std::mutex> lk(g_mu);
    if (int e = init_locked(-1)) return e;
    if (!med || med->n < 1 || med->d < 1 || !med->pos || !k || !mat) return set_err(MSGPU_E_ARG, "bad argument");
    const int n = med->n, d = med->d;
    double* dpos = nullptr;
    zc* dA = nullptr;
    CK(cudaMalloc(&dpos, sizeof(double) * (size_t)n * d));
    CK(cudaMalloc(&dA, sizeof(zc) * (size_t)n * n));
    CK(cudaMemcpy(dpos, med->pos, sizeof(double) * (size_t)n * d, cudaMemcpyHostToDevice));
    int nt = (n + 31) / 32;
    k_build_matrix<<<std::min(nt, 4 * g_sms), NT, smem_bytes()>>>(dA, n, d, dpos, med->model, k[0], k[1], deriv);
    g_launches++;
    CK(cudaGetLastError());
    CK(cudaMemcpy(mat, dA, sizeof(zc) * (size_t)n * n, cudaMemcpyDeviceToHost));
    cudaFree(dpos);
    cudaFree(dA);
    return 0;
}

// Could the entries of M(k) (and of dM/dk for kind 1) of an item span more
// than the mixed engine's four-slice budget?  For d = 3 and the "maximum"
// model the moduli are known in closed form: off the diagonal
// |G| = e^{a r} / (4 pi r) (a = -Im k) and |dG/dk| = e^{a r} / (4 pi) over the
// pair distances [rmin, rmax], on the diagonal |k| / (4 pi) and 1 / (4 pi).
// The predicted span of the moduli, times 2 sqrt 2 (the engine measures
// max(|Re|, |Im|), within sqrt 2 of the modulus), is compared with the
// engine's threshold for the job kind; anything not covered counts as wide.
static bool item_may_be_wide(double rmin, double rmax, int kind, double kre, double kim) {
    // the engine's thresholds: 2^8, or 2^20 for amplitude items (refined to an FP64 residual)
    const double thr = kind == 2 ? 1048576.0 : 256.0;
    if (!(rmin > 0.0) || !(rmax >= rmin)) return true;
    const double a = -kim;
    auto g = [&](double r) { return std::exp(a * r) / r; };  // 4 pi |G|, up to the common factor
    double hi = std::max(g(rmin), g(rmax)), lo = std::min(g(rmin), g(rmax));
    if (a > 0.0 && 1.0 / a > rmin && 1.0 / a < rmax) lo = std::min(lo, g(1.0 / a));
    const double kabs = std::hypot(kre, kim);
    hi = std::max(hi, kabs);
    lo = std::min(lo, kabs);
    if (kind == 1) {
        const double e1 = std::exp(a * rmin), e2 = std::exp(a * rmax);
        hi = std::max({hi, e1, e2, 1.0});
        lo = std::min({lo, e1, e2, 1.0});
    }
    return !(hi <= lo * (thr / (2.0 * std::sqrt(2.0))));
}

// Items of a job: medium of each, k, the queue order (largest matrices
// first), the amplitude offsets (kind 2), the live count.  Caller holds g_mu.
static int set_items_locked(msgpu_job* J, int nitem, const int* item_med, const double* ks) {
    if (nitem < 1 || nitem > J->cap || !ks) return set_err(MSGPU_E_ARG, "job: bad item count");
    std::vector<int> med_of(nitem);
    double flops = 0.0;
    long long amp_total = 0;
    for (int i = 0; i < nitem; i++) {
        const int mi = item_med ? item_med[i] : 0;
        if (mi < 0 || mi >= J->nmed) return set_err(MSGPU_E_ARG, "job: bad item medium");
        med_of[i] = mi;
        // dlogf jobs always slice six ways (near a root M is ill-conditioned and tr(M^-1 dM/dk)
        // magnifies the factorisation's error by its condition number)
        if (J->precision == MSGPU_MIXED && !J->wide)
            J->wide = J->kind == 1 ||
                      item_may_be_wide(J->med_rmin[mi], J->med_rmax[mi], J->kind, ks[2 * i], ks[2 * i + 1]);
        const double n = J->med_n[mi], n3 = n * n * n, n2 = n * n;
        flops += (J->kind == 0) ? 8.0 / 3.0 * n3
                 : (J->kind == 1 || J->kind == 3) ? (8.0 / 3.0 + 8.0) * n3
                 : (J->kind == 2) ? 8.0 / 3.0 * n3 + 8.0 * n2
                                  : 8.0 / 3.0 * n3 + 50 * 8.0 * n2;  // kind 4: at most 50 solves
        amp_total += J->med_n[mi];
    }
    if ((J->kind == 2 || J->kind == 4) && J->d_amps && amp_total > J->amp_cap)
        return set_err(MSGPU_E_SIZE, "job: amplitudes exceed capacity");
    std::vector<int> order(nitem);
    for (int i = 0; i < nitem; i++) order[i] = i;
    std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return J->med_n[med_of[a]] > J->med_n[med_of[b]]; });
    std::vector<long long> off;
    if (J->d_amp_off) {
        off.resize(nitem);
        long long acc = 0;
        for (int i = 0; i < nitem; i++) { off[i] = acc; acc += J->med_n[med_of[i]]; }
    }
    const unsigned queue[2] = {0u, (unsigned)nitem};
    // small jobs: the item arrays (and the queue words behind them) in one copy
    std::vector<char> all(J->items_b <= ((size_t)64 << 10) ? J->items_b : 0);
    auto put = [&](void* dst, const void* src, size_t bytes) -> bool {
        if (bytes == 0) return true;
        if (all.empty()) return cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice) == cudaSuccess;
        std::memcpy(all.data() + ((char*)dst - (char*)J->d_ks), src, bytes);
        return true;
    };
    bool ok = put(J->d_ks, ks, sizeof(double) * 2 * nitem) && put(J->d_item_med, med_of.data(), sizeof(int) * nitem) &&
              put(J->d_order, order.data(), sizeof(int) * nitem) &&
              put(J->d_amp_off, off.data(), sizeof(long long) * off.size()) && put(J->d_counter, queue, sizeof(queue));
    if (ok && !all.empty()) ok = cudaMemcpy(J->d_ks, all.data(), all.size(), cudaMemcpyHostToDevice) == cudaSuccess;
    if (!ok) return set_err(MSGPU_E_CUDA, std::string("job: copy of the items: ") + cudaGetErrorString(cudaGetLastError()));
    J->nitem = nitem;
    J->flops = flops;
    J->amp_total = amp_total;
    return 0;
}

// (the block, if it is still the job's, is idle: it may be another job's next)
static void destroy_locked(msgpu_job* J) {
    if (J->gexec) cudaGraphExecDestroy(J->gexec);
    if (J->cap_stream) cudaStreamDestroy(J->cap_stream);
    pool_put(J->block, J->block_bytes);
    delete J;
}

msgpu_job* msgpu_job_create(int kind, int nmed, const msgpu_medium* media, int nitem, const int* item_med,
                            const double* ks, int precision) {
    std::lock_guard<std::mutex> lk(g_mu);
    if (init_locked(-1)) return nullptr;
    if (kind < 0 || kind > 4 || nmed < 1 || !media || nitem < 1 || !ks) {
        set_err(MSGPU_E_ARG, "job: bad argument");
        return nullptr;
    }
    if (precision != MSGPU_FP64 && precision != MSGPU_MIXED) {
        set_err(MSGPU_E_ARG, "job: unknown precision");
        return nullptr;
    }
    auto* J = new msgpu_job();
    J->kind = kind;
    J->precision = kind >= 3 ? MSGPU_FP64 : precision;  // traceinv, inverse iteration: FP64 engine
    J->cap = nitem;
    J->nmed = nmed;
    J->med_n.resize(nmed);
    std::vector<MedDev> hm(nmed);
    size_t npos = 0;
    for (int i = 0; i < nmed; i++) {
        const msgpu_medium& m = media[i];
        if (m.n < 1 || m.d < 1 || m.d > 20 || !m.pos || m.n > 50000) {
            set_err(MSGPU_E_ARG, "job: bad medium");
            delete J;
            return nullptr;
        }
        J->nmax = std::max(J->nmax, m.n);
        J->med_n[i] = m.n;
        if (m.d != 3) J->d3only = false;
        npos += (size_t)m.n * m.d;
    }
    // the engine that serves the job (the tuning table may hand a mixed request to the FP64 engine)
    const TuneEntry te = kind < 3 ? g_tune[kind][precision][size_bucket(J->nmax)] : TuneEntry{};
    if (te.engine) J->precision = te.engine - 1;
    // pair-distance range of every d = 3 "maximum" medium (mixed jobs: the entry span of M(k))
    J->med_rmin.assign(nmed, -1.0);
    J->med_rmax.assign(nmed, -1.0);
    if (J->precision == MSGPU_MIXED && (kind == 0 || kind == 2))  // dlogf jobs are wide whatever the span
        for (int i = 0; i < nmed; i++) {
            const msgpu_medium& m = media[i];
            if (m.d != 3 || m.model.type != MSGPU_MAXIMUM || m.n < 2) continue;
            double lo = INFINITY, hi = 0.0;
            for (int a = 0; a < m.n; a++)
                for (int b = a + 1; b < m.n; b++) {
                    const double dx = m.pos[3 * a] - m.pos[3 * b], dy = m.pos[3 * a + 1] - m.pos[3 * b + 1],
                                 dz = m.pos[3 * a + 2] - m.pos[3 * b + 2];
                    const double r2 = dx * dx + dy * dy + dz * dz;
                    lo = std::min(lo, r2);
                    hi = std::max(hi, r2);
                }
            J->med_rmin[i] = std::sqrt(lo);
            J->med_rmax[i] = std::sqrt(hi);
        }
    auto fail = [&](const char* what) -> msgpu_job* {
        set_err(MSGPU_E_CUDA, std::string("job: ") + what);
        destroy_locked(J);
        return nullptr;
    };
    // launch: the team, and as many slots as the device and the memory hold
    J->slot = (size_t)J->nmax * J->nmax;
    const bool fp64 = J->precision == MSGPU_FP64;
    // One launch takes the whole job, so its kernel goes by the largest medium: 1200 ln det of
    // n = 64 take 5.2 ms on the kernel for small matrices, 6.7 with one of n = 97 among them;
    // dlogf of 900 of n = 90 10.6, 16.7 with 30 of n = 110 (27 before there was a choice).
    J->tc = fp64 && J->nmax >= TC_NMIN;
    const size_t slot_b = slot_elems(kind, J->slot, J->nmax) * sizeof(zc);
    const size_t img_b = J->tc ? (tc64_image_bytes(J->nmax) + 127) / 128 * 128 : 0;
    const size_t per_cta = slot_b + img_b;
    const int ctas = te.ctas ? std::min(te.ctas, g_ctas_fp64) : g_ctas_fp64;
    int held = J->tc ? g_sms : g_sms * ctas;  // matrices on the device at once
    if (fp64) {
        J->team = pick_team_fp64(J->tc, nitem, J->nmax);
        if (J->team > 1) held = g_teams[J->tc][ilog2(J->team)];
        // (one CTA per SM asked for by the tuning table: as asked)
        J->small = J->nmax < TC_NMIN && J->team == 1 && te.ctas != 1 && nitem > held;
        if (J->small) held = g_sms * SMALL_CTAS;
    } else if (nitem < g_sms * g_ctas_fp64) {
        // (whatever the tuning table asks for a full chip: one wavefunction at n = 1024 takes
        // 31 ms on a cluster, 74 on a CTA)  A mixed job may turn wide with later points: count
        // the teams of the wide launch
        int teams[5] = {g_sms * g_ctas_fp64, 0, 0, 0, 0};
        for (int j = 1; j < 5; ++j) teams[j] = mixed_max_teams(kind, J->d3only, 1 << j);
        J->team = pick_team(teams, 0.25, 1.6, nitem, J->nmax);
        if (J->team > 1) held = teams[ilog2(J->team)];
    }
    int grid = std::min(nitem, held);
    if ((size_t)grid * per_cta + 128 > g_ws_bytes) {  // else the workspace that is there holds them
        const size_t budget = ws_budget();
        while (grid > 1 && (size_t)grid * per_cta > budget) grid--;
    }
    J->grid = grid;
    J->img_off = ((size_t)grid * slot_b + 127) / 128 * 128;
    J->ws_bytes = J->img_off + (size_t)grid * img_b;
    // one block: media, positions, then the item arrays, results, pivots, amplitudes
    const bool vecs = kind == 2 || kind == 4;
    if (vecs) J->amp_cap = (long long)nitem * J->nmax;  // nitem items of the largest medium
    size_t at = 0;
    auto take = [&](size_t bytes) {
        const size_t o = at;
        at = (at + bytes + 255) / 256 * 256;
        return o;
    };
    const size_t o_media = take(sizeof(MedDev) * nmed), o_pos = take(sizeof(double) * npos);
    const size_t o_ks = take(sizeof(double) * 2 * nitem), o_med = take(sizeof(int) * nitem), o_order = take(sizeof(int) * nitem);
    const size_t o_off = take(vecs ? sizeof(long long) * nitem : 0), o_counter = take(sizeof(unsigned) * 2);
    const size_t o_out = take(sizeof(double) * 2 * nitem), o_status = take(sizeof(int) * nitem);
    const size_t o_piv = take(sizeof(int) * (size_t)grid * J->nmax);
    const size_t o_amps = take(vecs ? sizeof(double) * 2 * (size_t)J->amp_cap : 0);
    J->block_bytes = at;
    char* base = static_cast<char*>(J->block = pool_get(J->block_bytes));
    if (!base) return fail("device allocation");
    J->d_media = reinterpret_cast<MedDev*>(base + o_media);
    J->d_pos = reinterpret_cast<double*>(base + o_pos);
    J->d_ks = reinterpret_cast<double*>(base + o_ks);
    J->d_item_med = reinterpret_cast<int*>(base + o_med);
    J->d_order = reinterpret_cast<int*>(base + o_order);
    J->d_amp_off = vecs ? reinterpret_cast<long long*>(base + o_off) : nullptr;
    J->d_counter = reinterpret_cast<unsigned*>(base + o_counter);
    J->items_b = o_counter + 2 * sizeof(unsigned) - o_ks;
    J->d_out = reinterpret_cast<double*>(base + o_out);
    J->d_status = reinterpret_cast<int*>(base + o_status);
    J->d_piv = reinterpret_cast<int*>(base + o_piv);
    J->d_amps = vecs ? reinterpret_cast<double*>(base + o_amps) : nullptr;
    std::vector<char> head(o_ks);
    size_t off = 0;
    for (int i = 0; i < nmed; i++) {
        const msgpu_medium& m = media[i];
        const size_t cnt = (size_t)m.n * m.d;
        std::memcpy(head.data() + o_pos + sizeof(double) * off, m.pos, sizeof(double) * cnt);
        hm[i] = MedDev{m.d, m.n, J->d_pos + off, m.model};
        off += cnt;
    }
    std::memcpy(head.data() + o_media, hm.data(), sizeof(MedDev) * nmed);
    if (cudaMemcpy(base, head.data(), head.size(), cudaMemcpyHostToDevice) != cudaSuccess) return fail("copy media");
    if (set_items_locked(J, nitem, item_med, ks)) {
        destroy_locked(J);
        return nullptr;
    }
    void* ws = nullptr;
    if (ensure_ws(J->ws_bytes, &ws)) {
        destroy_locked(J);
        return nullptr;
    }
    return J;
}

int msgpu_job_set_points(msgpu_job* J, int nitem, const int* item_med, const double* ks) {
    if (!J) return set_err(MSGPU_E_ARG, "null job");
    std::lock_guard<std::mutex> lk(g_mu);
    return set_items_locked(J, nitem, item_med, ks);
}

int msgpu_job_use_graph(msgpu_job* J, int on) {
    if (!J) return set_err(MSGPU_E_ARG, "null job");
    std::lock_guard<std::mutex> lk(g_mu);
    J->use_graph = on != 0;
    return 0;
}

// the work of one run on stream st: reset the queue, launch the engine
static int launch_locked(msgpu_job* J, void* ws, cudaStream_t st) {
    CK(cudaMemsetAsync(J->d_counter, 0, sizeof(unsigned), st));
    EngineParams P;
    P.media = J->d_media;
    P.ks = J->d_ks;
    P.item_med = J->d_item_med;
    P.order = J->d_order;
    P.nitem = J->cap;
    P.ws = reinterpret_cast<zc*>(ws);
    P.slot = J->slot;
    P.piv = J->d_piv;
    P.piv_stride = J->nmax;
    P.out = J->d_out;
    P.status = J->d_status;
    P.counter = J->d_counter;
    P.kind = J->kind;
    P.wide_ok = J->wide ? 1 : 0;
    P.warm = J->warm ? 1 : 0;
    P.given_n = 0;
    P.info = nullptr;
    P.first_wait = first_wait_limit();
    P.amps = J->d_amps;
    P.amp_off = J->d_amp_off;
    if (J->precision == MSGPU_MIXED) {
        int e = mixed_run(P, J->grid, J->team, J->nmax, J->d3only, st);
        if (e) return set_err(e, "mixed engine launch failed");
        return 0;
    }
    const int e = J->tc ? tc64_run(P, J->grid, J->team, J->nmax, static_cast<unsigned char*>(ws) + J->img_off, st)
                  : J->small ? launch_teams(k_engine_fp64_small, J->grid, 1, SMALL_NT, sizeof(SmallSmem), st, P)
                             : launch_teams(k_engine_fp64, J->grid, J->team, NT, smem_bytes(), st, P);
    if (e) return set_err(e, std::string("FP64 engine launch failed: ") + cudaGetErrorString(cudaGetLastError()));
    return 0;
}

// One matrix of the caller's through the FP64 engine, shared by a cluster of CTAs
// (n = 300: one CTA took 14 ms).  Its buffers are its own block of the pool, not the
// shared workspace: a job may still be running there, on a stream this one does not wait for.
static int tracelog_matrix_in(unsigned char* b, size_t img_off, size_t piv_off, size_t out_off, int n, const double* mat,
                              double* out, int* info) {
    const bool tc = n >= TC_NMIN;
    // results and queue: {out[2], info, status}, then the counter words {0, 1}
    const unsigned queue[2] = {0u, 1u};
    CK(cudaMemcpy(b, mat, sizeof(zc) * (size_t)n * n, cudaMemcpyHostToDevice));
    CK(cudaMemcpy(b + out_off + 128, queue, sizeof(queue), cudaMemcpyHostToDevice));
    EngineParams P{};
    P.nitem = 1;
    P.ws = reinterpret_cast<zc*>(b);
    P.slot = (size_t)n * n;
    P.piv = reinterpret_cast<int*>(b + piv_off);
    P.piv_stride = n;
    P.out = reinterpret_cast<double*>(b + out_off);
    P.info = reinterpret_cast<int*>(b + out_off + 16);
    P.status = P.info + 1;
    P.counter = reinterpret_cast<unsigned*>(b + out_off + 128);
    P.given_n = n;
    P.first_wait = first_wait_limit();
    const int team = pick_team_fp64(tc, 1, n);
    if (tc ? tc64_run(P, 1, team, n, b + img_off, nullptr)
           : launch_teams(k_engine_fp64, 1, team, NT, smem_bytes(), (cudaStream_t) nullptr, P))
        return set_err(MSGPU_E_CUDA, std::string("tracelog_matrix: ") + cudaGetErrorString(cudaGetLastError()));
    g_launches++;
    double h[3];
    CK(cudaMemcpy(h, b + out_off, sizeof(h), cudaMemcpyDeviceToHost));
    int st[2];
    std::memcpy(st, &h[2], sizeof(st));
    if (st[1] & MSGPU_S_TIMEOUT) return set_err(MSGPU_E_CUDA, "tracelog_matrix: a device wait ran out");
    out[0] = h[0];
    out[1] = h[1];
    if (info) *info = st[0];
    return 0;
}

int msgpu_tracelog_matrix(int n, const double* mat, double* out, int* info) {
    std::lock_guard<std::mutex> lk(g_mu);
    if (int e = init_locked(-1)) return e;
    if (n < 1 || !mat || !out) return set_err(MSGPU_E_ARG, "bad argument");
    const size_t img_off = (sizeof(zc) * (size_t)n * n + 127) / 128 * 128;
    const size_t piv_off = img_off + (n >= TC_NMIN ? (tc64_image_bytes(n) + 127) / 128 * 128 : 0);
    const size_t out_off = piv_off + (sizeof(int) * (size_t)n + 127) / 128 * 128;
    size_t bytes = out_off + 256;
    void* b = pool_get(bytes);
    if (!b) return set_err(MSGPU_E_CUDA, "tracelog_matrix: device allocation");
    const int e = tracelog_matrix_in(static_cast<unsigned char*>(b), img_off, piv_off, out_off, n, mat, out, info);
    if (e) cudaFree(b);  // (waits for what may still run on it)
    else pool_put(b, bytes);
    return e;
}

int msgpu_job_run(msgpu_job* J, void* stream) {
    if (!J) return set_err(MSGPU_E_ARG, "null job");
    std::lock_guard<std::mutex> lk(g_mu);
    cudaStream_t st = (cudaStream_t)stream;
    void* ws = nullptr;
    if (int e = ensure_ws(J->ws_bytes, &ws)) return e;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(st, &cs) == cudaSuccess && cs != cudaStreamCaptureStatusNone) J->captured = true;
    ++J->runs;
    if (!J->use_graph) {
        if (int e = launch_locked(J, ws, st)) return e;
        g_launches++;
        return 0;
    }
    if (J->precision == MSGPU_MIXED && mixed_prepare(J->grid, J->nmax)) return set_err(MSGPU_E_CUDA, "mixed scratch");
    // the graph holds the workspace and scratch addresses, the launch's shared-memory size
    // (wide) and the start-vector mode (warm)
    const unsigned long long gen =
        ((g_ws_gen * 0x9E3779B97F4A7C15ULL + mixed_generation()) * 2 + (J->wide ? 1 : 0)) * 2 + (J->warm ? 1 : 0);
    if (!J->gexec || J->gen != gen) {
        // (re)capture: the graph holds the workspace and scratch addresses
        if (J->gexec) cudaGraphExecDestroy(J->gexec);
        J->gexec = nullptr;
        if (!J->cap_stream) CK(cudaStreamCreateWithFlags(&J->cap_stream, cudaStreamNonBlocking));
        CK(cudaStreamBeginCapture(J->cap_stream, cudaStreamCaptureModeRelaxed));
        const int e = launch_locked(J, ws, J->cap_stream);
        cudaGraph_t g = nullptr;
        const cudaError_t ce = cudaStreamEndCapture(J->cap_stream, &g);
        if (e) {
            if (g) cudaGraphDestroy(g);
            return e;
        }
        CK(ce);
        const cudaError_t ie = cudaGraphInstantiate(&J->gexec, g, 0);
        cudaGraphDestroy(g);
        CK(ie);
        J->gen = gen;
    }
    CK(cudaGraphLaunch(J->gexec, st));
    g_launches++;
    return 0;
}

int msgpu_job_launches(const msgpu_job* J) { return J ? 1 : 0; }

int msgpu_engine_stats(double* out, int n) { return mixed_stats(out, n); }
double msgpu_job_flops(const msgpu_job* J) { return J ? J->flops : 0.0; }

int msgpu_job_results(msgpu_job* J, double* out, int* status) {
    if (!J) return set_err(MSGPU_E_ARG, "null job");
    const unsigned runs = J->runs;
    CK(cudaDeviceSynchronize());
    J->done = runs;
    if (out) CK(cudaMemcpy(out, J->d_out, sizeof(double) * 2 * J->nitem, cudaMemcpyDeviceToHost));
    if (status) CK(cudaMemcpy(status, J->d_status, sizeof(int) * J->nitem, cudaMemcpyDeviceToHost));
    return 0;
}

int msgpu_job_amplitudes(msgpu_job* J, double* amps) {
    if (!J || (J->kind != 2 && J->kind != 4) || !amps)
        return set_err(MSGPU_E_ARG, "job_amplitudes: not an amplitude or eigenvector job");
    CK(cudaDeviceSynchronize());
    CK(cudaMemcpy(amps, J->d_amps, sizeof(double) * 2 * (size_t)J->amp_total, cudaMemcpyDeviceToHost));
    return 0;
}

int msgpu_job_set_vectors(msgpu_job* J, const double* vecs) {
    if (!J || J->kind != 4 || !vecs || !J->d_amps)
        return set_err(MSGPU_E_ARG, "job_set_vectors: not an eigenvector job");
    std::lock_guard<std::mutex> lk(g_mu);
    CK(cudaMemcpy(J->d_amps, vecs, sizeof(double) * 2 * (size_t)J->amp_total, cudaMemcpyHostToDevice));
    J->warm = true;
    return 0;
}

void msgpu_job_destroy(msgpu_job* J) {
    if (!J) return;
    // The block is kept for the next job only if no run can be on the device: a run whose
    // results were not fetched may be, and a replay of a graph of the caller's.  Else it is
    // freed, which waits; outside the lock, so that other threads' calls go on meanwhile.
    if (J->captured || J->done != J->runs) {
        cudaFree(J->block);
        J->block = nullptr;
    }
    std::lock_guard<std::mutex> lk(g_mu);
    destroy_locked(J);
}

int msgpu_tune_set(int kind, int precision, int n, int engine, int ctas_per_sm) {
    if (kind < 0 || kind > 2 || (precision != MSGPU_FP64 && precision != MSGPU_MIXED) || n < 1 ||
        (engine != -1 && engine != MSGPU_FP64 && engine != MSGPU_MIXED) || ctas_per_sm < 0 || ctas_per_sm > 8)
        return set_err(MSGPU_E_ARG, "tune_set: bad argument");
    if (precision == MSGPU_FP64 && engine == MSGPU_MIXED)
        return set_err(MSGPU_E_ARG, "tune_set: an FP64 request cannot run on the mixed engine");
    std::lock_guard<std::mutex> lk(g_mu);
    TuneEntry& e = g_tune[kind][precision][size_bucket(n)];
    e.engine = engine < 0 ? 0 : engine + 1;
    e.ctas = ctas_per_sm;
    return 0;
}

int msgpu_tune_get(int kind, int precision, int n, int* engine, int* ctas_per_sm) {
    if (kind < 0 || kind > 2 || (precision != MSGPU_FP64 && precision != MSGPU_MIXED) || n < 1 || !engine ||
        !ctas_per_sm)
        return set_err(MSGPU_E_ARG, "tune_get: bad argument");
    std::lock_guard<std::mutex> lk(g_mu);
    const TuneEntry& e = g_tune[kind][precision][size_bucket(n)];
    *engine = e.engine - 1;
    *ctas_per_sm = e.ctas;
    return 0;
}

int msgpu_autotune(int kind, int precision, int d, int n, int nitem, double* seconds) {
    if (kind < 0 || kind > 2 || (precision != MSGPU_FP64 && precision != MSGPU_MIXED) || d < 2 || d > 3 ||
        n < 2 || nitem < 1 || !seconds)
        return set_err(MSGPU_E_ARG, "autotune: bad argument");
    {
        std::lock_guard<std::mutex> lk(g_mu);
        if (int e = init_locked(-1)) return e;
    }
    // probe: n scatterers of the reference's ball (seed 1), nitem k on the
    // real axis ... -0.05i (cross sections need real k)
    std::vector<double> pos((size_t)n * d), ks(2 * (size_t)nitem);
    if (int e = msgpu_fill_medium(d, n, MSGPU_BALL, 1.0, 1, pos.data())) return e;
    for (int i = 0; i < nitem; ++i) {
        ks[2 * i] = 0.5 + 2.5 * i / std::max(1, nitem - 1);
        ks[2 * i + 1] = kind == 2 ? 0.0 : -0.05;
    }
    const msgpu_medium med{d, n, pos.data(), {MSGPU_MAXIMUM, 0, {0.0, 0.0}}};
    const int engines[2] = {MSGPU_FP64, MSGPU_MIXED};
    double best = 0.0;
    int best_e = precision, best_c = 0;
    for (int ei = 0; ei < (precision == MSGPU_MIXED ? 2 : 1); ++ei)
        for (int c = 1; c <= 2; ++c) {
            const int eng = precision == MSGPU_MIXED ? engines[ei] : MSGPU_FP64;
            double& t = seconds[ei * 2 + (c - 1)];
            t = -1.0;
            if (c > g_ctas_fp64) continue;
            // above 96 rows the FP64 engine runs one CTA per SM whatever is asked: timed once
            const bool tc = eng == MSGPU_FP64 && n >= TC_NMIN;
            if (tc && c > 1) continue;
            if (int e = msgpu_tune_set(kind, precision, n, eng, c)) return e;
            msgpu_job* J = msgpu_job_create(kind, 1, &med, nitem, nullptr, ks.data(), precision);
            if (!J) return MSGPU_E_CUDA;
            cudaEvent_t e0, e1;
            cudaEventCreate(&e0);
            cudaEventCreate(&e1);
            int err = msgpu_job_run(J, nullptr);  // warm-up (allocations, first launch)
            if (!err) err = cudaDeviceSynchronize() == cudaSuccess ? 0 : MSGPU_E_CUDA;
            float ms = 0.0f;
            if (!err) {
                cudaEventRecord(e0, nullptr);
                err = msgpu_job_run(J, nullptr);
                cudaEventRecord(e1, nullptr);
                if (!err && cudaEventSynchronize(e1) == cudaSuccess) cudaEventElapsedTime(&ms, e0, e1);
            }
            cudaEventDestroy(e0);
            cudaEventDestroy(e1);
            msgpu_job_destroy(J);
            if (err) return err;
            t = 1e-3 * ms;
            if (best == 0.0 || t < best) {
                best = t;
                best_e = eng;
                best_c = tc ? 0 : c;
            }
        }
    return msgpu_tune_set(kind, precision, n, best_e, best_c);
}

static int run_batch(int kind, int nmed, const msgpu_medium* media, int nitem, const int* item_med, const double* ks,
                     double* out, int* status, int precision) {
    msgpu_job* J = msgpu_job_create(kind, nmed, media, nitem, item_med, ks, precision);
    if (!J) return g_err.empty() ? MSGPU_E_ARG : (g_err.find("CUDA") != std::string::npos ? MSGPU_E_CUDA : MSGPU_E_ARG);
    int e = msgpu_job_run(J, nullptr);
    if (!e) e = msgpu_job_results(J, out, status);
    msgpu_job_destroy(J);
    return e;
}

int msgpu_tracelog_batch(int nmed, const msgpu_medium* media, int nitem, const int* item_med, const double* ks,
                         double* out, int* status, int precision) {
    return run_batch(0, nmed, media, nitem, item_med, ks, out, status, precision);
}

int msgpu_dk_log_det_batch(int nmed, const msgpu_medium* media, int nitem, const int* item_med, const double* ks,
                           double* out, int* status, int precision) {
    return run_batch(1, nmed, media, nitem, item_med, ks, out, status, precision);
}

int msgpu_traceinv_batch(int nmed, const msgpu_medium* media, int nitem, const int* item_med, const double* ks,
                         double* out, int* status, int precision) {
    return run_batch(3, nmed, media, nitem, item_med, ks, out, status, precision);
}

int msgpu_inverse_iteration_batch(int nmed, const msgpu_medium* media, int nitem, const int* item_med,
                                  const double* ks, double* lambda, double* vecs, int* status, int precision) {
    msgpu_job* J = msgpu_job_create(4, nmed, media, nitem, item_med, ks, precision);
    if (!J) return MSGPU_E_ARG;
    int e = msgpu_job_run(J, nullptr);
    if (!e) e = msgpu_job_results(J, lambda, status);
    if (!e && vecs) e = msgpu_job_amplitudes(J, vecs);
    msgpu_job_destroy(J);
    return e;
}

int msgpu_amplitude_batch(int nmed, const msgpu_medium* media, int nitem, const int* item_med, const double* ks,
                          double* out, double* amps, int* status, int precision) {
    msgpu_job* J = msgpu_job_create(2, nmed, media, nitem, item_med, ks, precision);
    if (!J) return MSGPU_E_ARG;
    int e = msgpu_job_run(J, nullptr);
    if (!e) e = msgpu_job_results(J, out, status);
    if (!e && amps) e = msgpu_job_amplitudes(J, amps);
    msgpu_job_destroy(J);
    return e;
}

}  // extern "C"
