// Navier-Stokes 2-D kernel instantiations, p = 1..8, q = p+1 (k_ns2d.cu has q = p+2).
#include "dispatch.cuh"

namespace dgmx {
namespace {
struct RegNS2Dq1 {
  RegNS2Dq1() {
#define R(P) reg2d_ns<DGMX_NS2D, P, P + 1>();
    R(1) R(2) R(3) R(4) R(5) R(6) R(7) R(8)
#undef R
  }
} reg_ns2d_q1;
}  // namespace
}  // namespace dgmx
