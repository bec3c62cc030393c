// gd_fused_len2.cu -- row lengths of the register-resident phase kernels (gd_fused_reg.cuh).
#include "gd_fused_reg.cuh"

namespace gd {

bool launch_fused_len2(cudaStream_t s, const Dims& d, int nlon, const void* tw, int phase, const FusedArgs& a) {
  switch (nlon) {
    case 96: return launch_fused_row<4, 3, 8>(s, d, tw, phase, a);
    case 100: return launch_fused_row<10, 1, 10>(s, d, tw, phase, a);
    case 108: return launch_fused_row<6, 3, 6>(s, d, tw, phase, a);
    case 128: return launch_fused_row<8, 2, 8>(s, d, tw, phase, a);
    case 144: return launch_fused_row<4, 3, 12>(s, d, tw, phase, a);
    case 160: return launch_fused_row<4, 5, 8>(s, d, tw, phase, a);
    case 180: return launch_fused_row<6, 5, 6>(s, d, tw, phase, a);
    default: return false;
  }
}

}  // namespace gd
