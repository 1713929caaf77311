// Class kernels of the integral engine: (dd| s, p, d, f): one thread per aux component (eri_class.cuh).
#include "eri_class.cuh"

namespace rr {
namespace eri {

bool launch_class_dd(int la, int lb, int lc, const ClassArgs& args, cudaStream_t s) {
  if (la == 2 && lb == 2 && lc == 0) {
    launch_class<2, 2, 0, true>(args, s);
    return true;
  }
  if (la == 2 && lb == 2 && lc == 1) {
    launch_class<2, 2, 1, true>(args, s);
    return true;
  }
  if (la == 2 && lb == 2 && lc == 2) {
    launch_class<2, 2, 2, true>(args, s);
    return true;
  }
  if (la == 2 && lb == 2 && lc == 3) {
    launch_class<2, 2, 3, true>(args, s);
    return true;
  }
  return false;
}

}  // namespace eri
}  // namespace rr
