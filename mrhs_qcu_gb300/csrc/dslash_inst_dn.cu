// Dslash instances for PREC_DOUBLE; registered at library load.  All of them
// run the fixed-point hop (dslash_fix.cuh): R > 1 takes the RHS of a thread one
// after another, PK (and every shape from SU(5) on) is the split form.
#include "dslash.h"

namespace qcu {
namespace {
struct Register_dn {
  Register_dn() {
    register_dslash(PREC_DOUBLE, 4, 1, 1, 0, &launch_wilson_mrhs<PREC_DOUBLE, 4, 1, 1, false>);
    register_dslash(PREC_DOUBLE, 4, 1, 2, 0, &launch_wilson_mrhs<PREC_DOUBLE, 4, 1, 2, false>);
    register_dslash(PREC_DOUBLE, 4, 1, 7, 0, &launch_wilson_mrhs<PREC_DOUBLE, 4, 1, 7, false>);
    register_dslash(PREC_DOUBLE, 4, 1, 2, 1, &launch_wilson_mrhs<PREC_DOUBLE, 4, 1, 2, true>);
    register_dslash(PREC_DOUBLE, 4, 1, 7, 1, &launch_wilson_mrhs<PREC_DOUBLE, 4, 1, 7, true>);
    register_dslash(PREC_DOUBLE, 4, 2, 1, 0, &launch_wilson_mrhs<PREC_DOUBLE, 4, 2, 1, false>);
    register_dslash(PREC_DOUBLE, 5, 1, 1, 0, &launch_wilson_mrhs<PREC_DOUBLE, 5, 1, 1, false>);
    register_dslash(PREC_DOUBLE, 5, 1, 2, 0, &launch_wilson_mrhs<PREC_DOUBLE, 5, 1, 2, false>);
    register_dslash(PREC_DOUBLE, 6, 1, 1, 0, &launch_wilson_mrhs<PREC_DOUBLE, 6, 1, 1, false>);
    register_dslash(PREC_DOUBLE, 6, 1, 2, 0, &launch_wilson_mrhs<PREC_DOUBLE, 6, 1, 2, false>);
    register_dslash(PREC_DOUBLE, 7, 1, 1, 0, &launch_wilson_mrhs<PREC_DOUBLE, 7, 1, 1, false>);
    register_dslash(PREC_DOUBLE, 7, 1, 2, 0, &launch_wilson_mrhs<PREC_DOUBLE, 7, 1, 2, false>);
    register_dslash(PREC_DOUBLE, 8, 1, 1, 0, &launch_wilson_mrhs<PREC_DOUBLE, 8, 1, 1, false>);
    register_dslash(PREC_DOUBLE, 8, 1, 2, 0, &launch_wilson_mrhs<PREC_DOUBLE, 8, 1, 2, false>);
  }
} register_dn;
}  // namespace
}  // namespace qcu
