// dev_int3c_f.cu — (mn|P) kernels with la = 3, lb = 0..3 (see dev_int3c.cuh).
#include "dev_int3c.cuh"

namespace ecg {
namespace dev {
namespace int3c {

Kernel pick_f(int lb) {
  switch (lb) {
    case 0: return int3c_kernel<3, 0>;
    case 1: return int3c_kernel<3, 1>;
    case 2: return int3c_kernel<3, 2>;
    default: return int3c_kernel<3, 3>;
  }
}

}  // namespace int3c
}  // namespace dev
}  // namespace ecg
