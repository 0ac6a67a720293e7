// Navier-Stokes 3-D kernel instantiations (Hex, FP64, BR1), p = 1..7, q = p+2 (and p+1 from p = 2).
#include "dispatch.cuh"

namespace dgmx {
namespace {
struct RegNS3D {
  RegNS3D() {
    // the third form (default), and the first-form tile whose FP32 viscous
    // kernels the mixed form runs
#define R(P, Q) reg3_ns<DGMX_NS3D, P, Q>(); reg_variant<DGMX_NS3D, P, Q, default_epb(3, Q), 0, false>();
    R(1, 3)
    R(2, 3) R(3, 4) R(4, 5) R(5, 6) R(6, 7) R(7, 8)
    R(2, 4) R(3, 5) R(4, 6) R(5, 7) R(6, 8)
#undef R
    reg3_ns<DGMX_NS3D, 7, 9>();
    // p = 7, q = 9: 729 points leave the one-thread-per-point stage tile
    // (736 threads, one CTA per SM by its shared memory) 80 registers and
    // about 1 KB of spills per thread; with 512 threads (some take two
    // points) it has 128 and no spills.
    reg_variant<DGMX_NS3D, 7, 9, 1, 0, false, 512>();
  }
} reg_ns3d;
}  // namespace
}  // namespace dgmx
