// dev_int3c_g0.cu — (mn|P) kernels with la = 4, lb = 0..2 (see dev_int3c.cuh).
#include "dev_int3c.cuh"

namespace ecg {
namespace dev {
namespace int3c {

Kernel pick_g0(int lb) {
  switch (lb) {
    case 0: return int3c_kernel<4, 0>;
    case 1: return int3c_kernel<4, 1>;
    default: return int3c_kernel<4, 2>;
  }
}

}  // namespace int3c
}  // namespace dev
}  // namespace ecg
