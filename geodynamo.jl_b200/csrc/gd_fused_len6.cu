// gd_fused_len6.cu -- row lengths of the register-resident phase kernels (gd_fused_reg.cuh).
#include "gd_fused_reg.cuh"

namespace gd {

bool launch_fused_len6(cudaStream_t s, const Dims& d, int nlon, const void* tw, int phase, const FusedArgs& a) {
  switch (nlon) {
    case 500: return launch_fused_row<10, 5, 10>(s, d, tw, phase, a);
    case 576: return launch_fused_row<12, 4, 12>(s, d, tw, phase, a);
    case 600: return launch_fused_row<10, 6, 10>(s, d, tw, phase, a);
    default: return false;
  }
}

}  // namespace gd
