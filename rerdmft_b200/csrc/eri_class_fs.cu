// Class kernels of the integral engine: (fs| s, p, d, f), and f shells of the metric: one thread per aux component (eri_class.cuh).
#include "eri_class.cuh"

namespace rr {
namespace eri {

bool launch_class_fs(int la, int lb, int lc, const ClassArgs& args, cudaStream_t s) {
  if (la == 3 && lb == 0 && lc == 0) {
    launch_class<3, 0, 0, true>(args, s);
    return true;
  }
  if (la == 3 && lb == 0 && lc == 1) {
    launch_class<3, 0, 1, true>(args, s);
    return true;
  }
  if (la == 3 && lb == 0 && lc == 2) {
    launch_class<3, 0, 2, true>(args, s);
    return true;
  }
  if (la == 3 && lb == 0 && lc == 3) {
    launch_class<3, 0, 3, true>(args, s);
    return true;
  }
  return false;
}

}  // namespace eri
}  // namespace rr
