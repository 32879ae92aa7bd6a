// One variant of the mixed-precision engine: job kind 1 (dlogf), media of any dimension,
// one CTA per matrix.
#define MSG_MIXED_KERNEL_BODY
#include "mixed_engine.cuh"

namespace msg {
int mixed_variant_1_any(const EngineParams& P, const MixScratch& X, const MixLaunch& L) {
    return mixed_variant<1, false, Solo>(P, X, L);
}
}  // namespace msg
