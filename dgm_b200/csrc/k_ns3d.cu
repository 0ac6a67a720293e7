// Navier-Stokes 3-D kernel instantiations (Hex, FP64 and the FP32 viscous form,
// BR1), p = 1..7, q = p+2 (q = p+1 in k_ns3d_q1.cu: a unit's tables share 64 KB
// of constant memory).
#include "dispatch.cuh"

namespace dgmx {
namespace {
struct RegNS3D {
  RegNS3D() {
#define R(P) reg3_ns<DGMX_NS3D, P, P + 2>();
    R(1) R(2) R(3) R(4) R(5) R(6) R(7)
#undef R
  }
} reg_ns3d;
}  // namespace
}  // namespace dgmx
