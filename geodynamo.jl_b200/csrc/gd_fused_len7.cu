// gd_fused_len7.cu -- row lengths of the register-resident phase kernels (gd_fused_reg.cuh).
#include "gd_fused_reg.cuh"

namespace gd {

bool launch_fused_len7(cudaStream_t s, const Dims& d, int nlon, const void* tw, int phase, const FusedArgs& a) {
  switch (nlon) {
    case 720: return launch_fused_row<12, 5, 12>(s, d, tw, phase, a);
    case 900: return launch_fused_row<15, 4, 15>(s, d, tw, phase, a);
    default: return false;
  }
}

}  // namespace gd
