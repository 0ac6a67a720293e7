// Navier-Stokes 2-D kernel instantiations (Quad, FP64 and the FP32 viscous
// form, BR1), p = 1..8, q = p+2 (q = p+1 in k_ns2d_q1.cu: a unit's tables share
// 64 KB of constant memory).
#include "dispatch.cuh"

namespace dgmx {
namespace {
struct RegNS2D {
  RegNS2D() {
#define R(P) reg2d_ns<DGMX_NS2D, P, P + 2>();
    R(1) R(2) R(3) R(4) R(5) R(6) R(7) R(8)
#undef R
  }
} reg_ns2d;
}  // namespace
}  // namespace dgmx
