// engine_internal.h -- structures shared by the engine translation units.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>
#include "msgpu.h"
#include "cplx.cuh"
#include "error_text.h"

namespace msg {

struct MedDev {
    int d, n;
    const double* pos;
    msgpu_model model;
};

struct EngineParams {
    const MedDev* media;
    const double* ks;     // 2 * nitem
    const int* item_med;  // nitem
    const int* order;     // queue position -> item index
    int nitem;
    zc* ws;               // per-CTA slots
    size_t slot;          // complex elements per matrix slot
    int* piv;             // per-CTA pivots
    int piv_stride;
    double* out;          // 2 * nitem
    int* status;          // nitem
    unsigned* counter;    // [0] work queue; [1] live items (queue positions >= it are past the end)
    int kind;             // 0 ln det / n, 1 dlogf, 2 amplitudes a = M^-1 phi, 3 traceinv, 4 inverse iteration
    double* amps;         // kinds 2, 4: a (or the eigenvector) per item (2 * n_i doubles each) or nullptr
    const long long* amp_off;  // kind 2: offset (in complex elements) of item i in amps
    int wide_ok;          // mixed engine: the launch has the shared memory for six-way slicing
    int given_n;          // > 0: one item, the caller's matrix of given_n rows, already in the first slot
    int* info;            // given matrix: 1-based index of the first zero pivot, or 0
    int warm;             // kind 4: start each inverse iteration from the item's vector in amps
    int first_wait;       // FP64 engine on the tensor cores: poll limit of an update's first operand wait
};


#ifdef __CUDACC__
// An amplitude item without a result: NaN for its amplitudes, entries first, first + step, ...
// (the job's array is a pooled block and may hold another job's).
__device__ inline void void_amplitudes(const EngineParams& P, int it, int first, int step) {
    if (P.kind != 2 || !P.amps) return;
    double* a = P.amps + 2 * P.amp_off[it];
    const int n2 = 2 * P.media[P.item_med[it]].n;
    for (int i = first; i < n2; i += step) a[i] = nan("");
}
#endif

// adds to the library's count of kernel launches (msgpu_launch_count)
void count_launches(int n);

// Launches `teams` clusters of `team` CTAs (a plain launch for team = 1).
template <class... KArgs, class... Args>
int launch_teams(void (*kern)(KArgs...), int teams, int team, int threads, size_t smem, cudaStream_t st, Args... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)(teams * team));
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)team;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = team > 1 ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kern, KArgs(args)...) == cudaSuccess ? 0 : MSGPU_E_CUDA;
}

// clusters of `team` CTAs the device holds at once (0: none of that size)
template <class K>
int max_teams(K kern, int team, int threads, size_t smem) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)team);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)team;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

// FP64 engine with the trailing updates on the tensor cores (tc64.cu): `teams`
// matrices at a time, `team` CTAs on each; img: teams x tc64_image_bytes(nmax)
// rounded up to 128 bytes.
int tc64_run(const EngineParams& P, int teams, int team, int nmax, void* img, cudaStream_t st);
size_t tc64_image_bytes(int nmax);
int tc64_max_teams(int team);
// Rows from which an item's trailing updates run on the tensor cores.  Smaller items
// stay on the FP64 pipe: 912 ln det take 3.4 ms there against 3.9 at n = 96, 4.5
// against 4.5 at n = 97, 6.4 against 6.2 at n = 128; dlogf 8.4 against 8.7, 12.1 against
// 10.3 and 16.5 against 13.4.  The rule looks at the item alone, so that no result
// depends on the batch it is in.
constexpr int TC_NMIN = 97;

// Mixed-precision engine (mixed.cu).  Returns 0 when it ran the job, a
// negative MSGPU_E* code on error.
// d3only: every medium of the job has d = 3 (selects the d = 3 kernel instantiation);
// P.wide_ok: launch with the shared memory for six-way slicing; grid matrices at a time,
// `team` CTAs on each.
int mixed_run(const EngineParams& P, int grid, int team, int nmax, bool d3only, cudaStream_t st);
// clusters of `team` CTAs of that variant's wide launch the device holds at once (0: none of that size)
int mixed_max_teams(int kind, bool d3only, int team);
// Allocates the mixed engine's scratch for `grid` matrices up to nmax
// (mixed_run does so itself; called before a stream capture, which must not allocate).
int mixed_prepare(int grid, int nmax);
// poll limit of the first operand wait of every tensor-core update (msgpu_debug_first_wait_limit)
int first_wait_limit();
// Changes whenever the mixed engine's scratch is reallocated or that limit is set (captured
// graphs hold both).
unsigned long long mixed_generation();
// per-phase SM cycles of the last mixed run made with MSGPU_STATS set:
// assemble, panel, trsm, slice, tiles, solve, items
int mixed_stats(double* out, int n);

}  // namespace msg
