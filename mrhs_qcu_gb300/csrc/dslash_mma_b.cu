// Instances of the register-fragment MMA dslash (dslash_mma.cuh), tensor-core
// variant 5: BF16 of either layout, N = 3..8.
#include "dslash_tc.h"

namespace qcu {
namespace {

// the same launcher serves both BF16 layouts (the plan reads the layout)
template <int N>
void register_n() {
  register_tc(PREC_BF16, N, kMmaVariant, &launch_wilson_mma<PREC_BF16, N>);
  register_tc(PREC_BF16S, N, kMmaVariant, &launch_wilson_mma<PREC_BF16, N>);
}

struct RegisterMmaBf16 {
  RegisterMmaBf16() {
    register_n<3>();
    register_n<4>();
    register_n<5>();
    register_n<6>();
    register_n<7>();
    register_n<8>();
  }
} register_mma_bf16;

}  // namespace
}  // namespace qcu
