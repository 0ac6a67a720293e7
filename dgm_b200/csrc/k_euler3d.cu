// Euler 3-D kernel instantiations (Hex, FP64), p = 1..7, q = p+2 (and p+1).
#include "dispatch.cuh"

namespace dgmx {
namespace {
struct RegEuler3D {
  RegEuler3D() {
    reg3<DGMX_EULER3D, 1, 3>();
#define R(P) reg3<DGMX_EULER3D, P, P + 1>(); reg3<DGMX_EULER3D, P, P + 2>();
    R(2) R(3) R(4) R(5) R(6) R(7)
#undef R
    // the prefetching persistent kernel, and the second-form stage kernels at
    // q = p+2 (every template instantiation of a tile lives in one
    // compilation unit: its launchers and its constant tables must come from
    // the same module)
    reg_pipe<DGMX_EULER3D, 3, 5, 1, 0, false>();
#define R2(P) reg2<DGMX_EULER3D, P, P + 2>();
    R2(2) R2(3) R2(4) R2(5)
#undef R2
  }
} reg_euler3d;
}  // namespace
}  // namespace dgmx
