// gd_fused_len5.cu -- row lengths of the register-resident phase kernels (gd_fused_reg.cuh).
#include "gd_fused_reg.cuh"

namespace gd {

bool launch_fused_len5(cudaStream_t s, const Dims& d, int nlon, const void* tw, int phase, const FusedArgs& a) {
  switch (nlon) {
    case 360: return launch_fused_row<6, 5, 12>(s, d, tw, phase, a);
    case 432: return launch_fused_row<12, 3, 12>(s, d, tw, phase, a);
    case 1024: return launch_fused_row<32, 1, 32>(s, d, tw, phase, a);
    default: return false;
  }
}

}  // namespace gd
