// Radices and CTA shapes of the x passes (csrc/x_pass.cu, csrc/x_transform.cu).
#pragma once

namespace dnsb {

// R: physical rows per CTA.  Every stage's items fit NT threads once (RM = 1,
// R1 <= 27 complex values a thread); the lengths where R1 = M / 8 would not
// fit the registers split it (288, 384), with several items per thread, 24
// complex values in all.  MINB: CTAs per SM the FP64 registers are held to.
template <int M>
struct XShape;
#define DNSB_X_SHAPE(M_, R1_, RM_, RB_, R_, NT_, MINB_)                            \
  template <>                                                                      \
  struct XShape<M_> {                                                              \
    static constexpr int R1 = R1_, RM = RM_, RB = RB_, R = R_, NT = NT_, MINB = MINB_; \
    static_assert(R1 * RM * RB == M_, "radices");                                  \
  };
DNSB_X_SHAPE(36, 6, 1, 6, 4, 96, 5)
DNSB_X_SHAPE(48, 6, 1, 8, 4, 96, 5)
DNSB_X_SHAPE(54, 9, 1, 6, 4, 96, 5)
DNSB_X_SHAPE(72, 9, 1, 8, 4, 96, 5)
DNSB_X_SHAPE(96, 12, 1, 8, 4, 96, 5)
DNSB_X_SHAPE(108, 18, 1, 6, 4, 96, 5)
DNSB_X_SHAPE(144, 18, 1, 8, 4, 96, 5)
DNSB_X_SHAPE(162, 27, 1, 6, 4, 128, 3)
DNSB_X_SHAPE(192, 24, 1, 8, 4, 96, 5)
DNSB_X_SHAPE(216, 27, 1, 8, 4, 128, 3)
DNSB_X_SHAPE(288, 6, 6, 8, 4, 144, 3)
DNSB_X_SHAPE(384, 6, 8, 8, 2, 96, 5)
#undef DNSB_X_SHAPE

}  // namespace dnsb
