// Substitutions with plain U, for more than 160 wall-normal points.  A module of
// their own: beside the pre-scaled ones, whose machine code they leave as it is,
// they cost the 128 x 129 x 128 corrector 0.8% (191.9 -> 193.4 us) by where the
// code lies.
#include "imm_solve.cuh"

namespace dnsb {

const void* imm_solve_plain(int kl, int nu, bool split) {
  return imm_solve_fn<false>(kl, nu, split);
}

}  // namespace dnsb
