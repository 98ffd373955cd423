// dev_int3c_g.cu — (mn|P) kernels with la = 4, lb = 3..4 (see dev_int3c.cuh).
#include "dev_int3c.cuh"

namespace ecg {
namespace dev {
namespace int3c {

Kernel pick_g(int lb) {
  switch (lb) {
    case 3: return int3c_kernel<4, 3>;
    default: return int3c_kernel<4, 4>;
  }
}

}  // namespace int3c
}  // namespace dev
}  // namespace ecg
