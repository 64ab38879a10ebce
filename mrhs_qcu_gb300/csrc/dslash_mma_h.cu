// Instances of the register-fragment MMA dslash (dslash_mma.cuh), tensor-core
// variant 5: FP16 with its per-(site, RHS) scale, N = 3..8.
#include "dslash_tc.h"

namespace qcu {
namespace {

template <int N>
void register_n() {
  register_tc(PREC_HALF, N, kMmaVariant, &launch_wilson_mma<PREC_HALF, N>);
}

struct RegisterMmaFp16 {
  RegisterMmaFp16() {
    register_n<3>();
    register_n<4>();
    register_n<5>();
    register_n<6>();
    register_n<7>();
    register_n<8>();
  }
} register_mma_fp16;

}  // namespace
}  // namespace qcu
