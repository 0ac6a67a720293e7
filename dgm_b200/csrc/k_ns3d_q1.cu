// Navier-Stokes 3-D kernel instantiations, p = 2..7, q = p+1 (k_ns3d.cu has q = p+2).
#include "dispatch.cuh"

namespace dgmx {
namespace {
struct RegNS3Dq1 {
  RegNS3Dq1() {
#define R(P) reg3_ns<DGMX_NS3D, P, P + 1>();
    R(2) R(3) R(4) R(5) R(6) R(7)
#undef R
  }
} reg_ns3d_q1;
}  // namespace
}  // namespace dgmx
