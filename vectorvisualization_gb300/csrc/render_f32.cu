// Forward ray-cast instantiations for field storage VVLIC_STORAGE_F32.
#include "render_fwd.cuh"

namespace vvlic {

cudaError_t launch_raycast_f32(const RenderArgs& a, int sampler, int integ, bool grad, int num_sms, cudaStream_t s) {
  return launch_storage<VVLIC_STORAGE_F32>(a, sampler, integ, grad, num_sms, s);
}

}  // namespace vvlic
