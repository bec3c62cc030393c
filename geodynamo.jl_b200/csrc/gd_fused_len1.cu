// gd_fused_len1.cu -- row lengths of the register-resident phase kernels (gd_fused_reg.cuh).
#include "gd_fused_reg.cuh"

namespace gd {

bool launch_fused_len1(cudaStream_t s, const Dims& d, int nlon, const void* tw, int phase, const FusedArgs& a) {
  switch (nlon) {
    case 24: return launch_fused_row<2, 3, 4>(s, d, tw, phase, a);
    case 40: return launch_fused_row<2, 5, 4>(s, d, tw, phase, a);
    case 48: return launch_fused_row<4, 3, 4>(s, d, tw, phase, a);
    case 64: return launch_fused_row<8, 1, 8>(s, d, tw, phase, a);
    case 80: return launch_fused_row<4, 5, 4>(s, d, tw, phase, a);
    case 768: return launch_fused_row<16, 3, 16>(s, d, tw, phase, a);
    default: return false;
  }
}

}  // namespace gd
