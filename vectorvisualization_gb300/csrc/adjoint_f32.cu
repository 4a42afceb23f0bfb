// Adjoint instantiations for field storage VVLIC_STORAGE_F32.
#include "adjoint.cuh"

namespace vvlic {

cudaError_t launch_adjoint_f32(const RenderArgs& a, int sampler, int integ, bool lit, const float4* g_img,
                               long long* acc, unsigned* next, int num_sms, cudaStream_t s) {
  return launch_adjoint_storage<VVLIC_STORAGE_F32>(a, sampler, integ, lit, g_img, acc, next, num_sms, s);
}

}  // namespace vvlic
