// One variant of the mixed-precision engine: job kind 0 (ln det), media all of d = 3,
// a cluster of CTAs per matrix.
#define MSG_MIXED_KERNEL_BODY
#include "mixed_engine.cuh"

namespace msg {
int mixed_team_0_d3(const EngineParams& P, const MixScratch& X, const MixLaunch& L) {
    return mixed_variant<0, true, ClusterTeam>(P, X, L);
}
}  // namespace msg
