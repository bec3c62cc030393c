// gd_fused_len3.cu -- row lengths of the register-resident phase kernels (gd_fused_reg.cuh).
#include "gd_fused_reg.cuh"

namespace gd {

bool launch_fused_len3(cudaStream_t s, const Dims& d, int nlon, const void* tw, int phase, const FusedArgs& a) {
  switch (nlon) {
    case 192: return launch_fused_row<8, 3, 8>(s, d, tw, phase, a);
    case 200: return launch_fused_row<10, 2, 10>(s, d, tw, phase, a);
    case 216: return launch_fused_row<6, 3, 12>(s, d, tw, phase, a);
    case 256: return launch_fused_row<16, 1, 16>(s, d, tw, phase, a);
    case 288: return launch_fused_row<12, 2, 12>(s, d, tw, phase, a);
    case 300: return launch_fused_row<10, 3, 10>(s, d, tw, phase, a);
    default: return false;
  }
}

}  // namespace gd
