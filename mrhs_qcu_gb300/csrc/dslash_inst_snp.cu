// Packed FP32x2 instances for SU(N >= 4) FP32; registered at library load.
// At two RHS per thread these kernels run 8 warps an SM (255 registers) and
// are bound by latency and issue, which the packed form halves: 16^3x32,
// scalar / packed, us a hop: SU(4) nrhs 16 125 / 100, SU(6) nrhs 32 494 / 387.
// (SU(8) nrhs 32: 905 with one RHS per thread, 900 packed.)  Register caps
// (128 and 168) spill and are slower.
#include "dslash.h"

namespace qcu {
namespace {
struct RegisterSnPacked {
  RegisterSnPacked() {
    register_dslash(PREC_SINGLE, 4, 2, 1, 1, &launch_wilson_mrhs<PREC_SINGLE, 4, 2, 1, true>);
    register_dslash(PREC_SINGLE, 5, 2, 1, 1, &launch_wilson_mrhs<PREC_SINGLE, 5, 2, 1, true>);
    register_dslash(PREC_SINGLE, 6, 2, 1, 1, &launch_wilson_mrhs<PREC_SINGLE, 6, 2, 1, true>);
    register_dslash(PREC_SINGLE, 8, 2, 1, 1, &launch_wilson_mrhs<PREC_SINGLE, 8, 2, 1, true>);
  }
} register_sn_packed;
}  // namespace
}  // namespace qcu
