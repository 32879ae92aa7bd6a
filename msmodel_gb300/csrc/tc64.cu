// tc64.cu -- the FP64 engine on the tensor cores: the kernel (one CTA of 512
// threads per SM, or a cluster of them per matrix) and its launch.
#include "tc64.cuh"
#include "fp64_engine.cuh"

namespace msg {

__global__ void __launch_bounds__(TC_NT, 1) k_engine_tc64(EngineParams P, uint8_t* img, size_t img_stride) {
    extern __shared__ uint8_t smem_raw[];
    Tc64Smem& s = *reinterpret_cast<Tc64Smem*>((reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    const int tid = threadIdx.x, warp = tid >> 5;
    if (warp == 0) {
        tmem_alloc(&s.tmem, TC_TMEM);
        tmem_relinquish();
    }
    if (tid == 0) {
        mbar_init(&s.bar_b, 1);
        mbar_init(&s.bar_mma, 1);
        s.err = 0;
        s.mma_stuck = 0;
        fence_mbar_init();
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const ClusterTeam tm = this_team();
    TcState t{img + (size_t)(blockIdx.x / tm.size) * img_stride, s.tmem, 0, 0, P.first_wait, false};
    run_items_fp64(P, s, tm, TcUpdate{t});
    // an MMA completion wait that ran out may leave MMAs in flight: give them a bounded chance to land
    if (s.mma_stuck && tid == 0) mbar_wait(&s.bar_mma, (uint32_t)(s.mma_stuck - 1), 1 << 20);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(t.tmem, TC_TMEM);
}

size_t tc64_image_bytes(int nmax) { return (size_t)((nmax + TC_N - 1) / TC_N) * TC_BTILE + 256; }

static size_t tc64_smem() { return sizeof(Tc64Smem) + 128; }

// the kernel's attributes, on the current device
static int tc64_attributes() {
    static bool done[64] = {false};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return MSGPU_E_CUDA;
    if (dev < 64 && done[dev]) return 0;
    if (cudaFuncSetAttribute(k_engine_tc64, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tc64_smem()) != cudaSuccess ||
        cudaFuncSetAttribute(k_engine_tc64, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
        return MSGPU_E_CUDA;
    if (dev < 64) done[dev] = true;
    return 0;
}

int tc64_max_teams(int team) {
    return tc64_attributes() ? 0 : max_teams(k_engine_tc64, team, TC_NT, tc64_smem());
}

int tc64_run(const EngineParams& P, int teams, int team, int nmax, void* img, cudaStream_t st) {
    if (int e = tc64_attributes()) return e;
    return launch_teams(k_engine_tc64, teams, team, TC_NT, tc64_smem(), st, P, static_cast<uint8_t*>(img),
                        (tc64_image_bytes(nmax) + 127) / 128 * 128);
}

}  // namespace msg
