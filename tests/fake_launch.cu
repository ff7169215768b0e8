// Kernel launchers that launch nothing, beside fake_cudart.cpp.
#include <cuda_runtime.h>

#include "rp_internal.h"

extern "C" void fake_note_sort(int whole);
extern "C" int fake_note_adj(int ordered);

namespace rp {

static bool whole(const SortBufs& b) { return b.keys && b.hist && b.sums && b.perm && b.gbase && b.nkeys > 0; }

cudaError_t launch_step(const RpStepArgs&, int, int, double*, cudaStream_t, int, int* n) { *n += 1; return cudaSuccess; }
cudaError_t launch_step_noalloc(const RpStepArgs&, int, int, int, cudaStream_t, int, int*) { return cudaSuccess; }
cudaError_t launch_step_mixed(const RpStepArgs&, int, int, float*, int, cudaStream_t, int, int* n) { *n += 1; return cudaSuccess; }
cudaError_t launch_stage_f32(int, const void*, const void*, float*, int64_t, int64_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_quantize(const float*, uint32_t*, float*, void*, int, int, int, int, int, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_mixed_convert(const RpParticlesDev&, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_clear_slot(void*, int, int64_t, int, int, cudaStream_t) { return cudaSuccess; }
int64_t sort_key_count(const RpStepArgs& A, uint32_t* gb) {
    int64_t k = 0;
    for (int g = 0; g < A.ngrid; g++) {
        gb[g] = (uint32_t)k;
        k += (int64_t)A.g[g].nx * A.g[g].ny;
    }
    return k;
}
cudaError_t launch_sort(const RpStepArgs&, int, const SortBufs& b, void*, cudaStream_t, int*) {
    fake_note_sort(whole(b));
    return cudaSuccess;
}
cudaError_t launch_order(const RpStepArgs&, int, const SortBufs& b, cudaStream_t, int*) {
    fake_note_sort(whole(b));
    return cudaGetLastError();
}
cudaError_t launch_unsort(int, const void*, void*, const uint32_t*, uint32_t, int64_t, int64_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_adj(int, const RpStepArgs&, const AdjFrames&, const AdjStateDev& s, double*, int, double, double*, double*,
                       double*, double*, double*, double*, int, cudaStream_t, int, int64_t* nlaunch) {
    *nlaunch += 2;
    return fake_note_adj(s.order != nullptr) ? cudaErrorLaunchFailure : cudaGetLastError();
}
cudaError_t launch_adj_store(const double*, const double*, double*, int, int, int, int64_t, int64_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_adj_tangent_init(double*, int64_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_ll2ij(const double*, const double*, const double*, int, int, int, const double*, const double*, int64_t,
                         double*, double*, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_locate(const RpStepArgs&, int, const double*, const double*, const double*, const double*, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_convert(int, int, const void*, const void*, void*, int, int, int, int, int64_t, int64_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_state_from_host(const RpParticlesDev&, const double*, const int32_t*, uint32_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_state_to_host(const RpParticlesDev&, double*, int32_t*, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_mask_slot(const uint8_t*, uint8_t*, int64_t, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_diag_reset(const RpParticlesDev&, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_output(const RpStepArgs&, const OutCols&, int, uint32_t, int64_t, int, cudaStream_t) { return cudaSuccess; }
}  // namespace rp
