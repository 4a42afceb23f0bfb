// Slicing / vector-field DVR / LIC-volume instantiations for field storage VVLIC_STORAGE_F16.
#include "techniques.cuh"

namespace vvlic {

cudaError_t launch_technique_f16(const RenderArgs& a, const TechArgs& t, int sampler, int integ, bool grad,
                                 int num_sms, cudaStream_t s) {
  return launch_tech_storage<VVLIC_STORAGE_F16>(a, t, sampler, integ, grad, num_sms, s);
}

}  // namespace vvlic
