// gd_fused_len4.cu -- row lengths of the register-resident phase kernels (gd_fused_reg.cuh).
#include "gd_fused_reg.cuh"

namespace gd {

bool launch_fused_len4(cudaStream_t s, const Dims& d, int nlon, const void* tw, int phase, const FusedArgs& a) {
  switch (nlon) {
    case 320: return launch_fused_row<8, 5, 8>(s, d, tw, phase, a);
    case 384: return launch_fused_row<8, 3, 16>(s, d, tw, phase, a);
    case 400: return launch_fused_row<10, 4, 10>(s, d, tw, phase, a);
    case 450: return launch_fused_row<15, 2, 15>(s, d, tw, phase, a);
    case 512: return launch_fused_row<16, 2, 16>(s, d, tw, phase, a);
    default: return false;
  }
}

}  // namespace gd
