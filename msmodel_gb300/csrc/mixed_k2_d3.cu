// One variant of the mixed-precision engine: job kind 2 (amplitudes), media all of d = 3,
// one CTA per matrix.
#define MSG_MIXED_KERNEL_BODY
#include "mixed_engine.cuh"

namespace msg {
int mixed_variant_2_d3(const EngineParams& P, const MixScratch& X, const MixLaunch& L) {
    return mixed_variant<2, true, Solo>(P, X, L);
}
}  // namespace msg
