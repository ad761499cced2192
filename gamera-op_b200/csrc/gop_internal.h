// Host-side helpers shared by the C ABI translation units.
#pragma once

#include <cmath>

#include "gamera_op.h"

namespace gop {
// validates a descriptor (0 or a GOP_E* code with the message set)
int check_desc(const gop_desc* d);
// sets the thread's last-error message and returns code
int set_error(int code, const char* fmt, ...);
// the pole ring average of a descriptor: poles reached (bit 0 theta = 0,
// bit 1 theta = pi), ring rows per pole - 1, phi blocks per ring row
struct RingSetup {
  int poles = 0;
  int jmax = 0;
  int nchunk[16] = {0};
};
int ring_setup(const gop_desc* d, RingSetup& r);
// ca^2 = m / s with a power of two for s that leaves m of the order of one
// where ca is above one.  The FP64 speeds and the Boris factor are quotients
// over b^2 + ca^2 rho, whose squares would leave the range of a double for a ca
// above 1e77 (1e100, say, to have no Boris limit); over b^2 s + m rho they do
// not, with the same bits wherever ca^2 did not overflow.
inline void split_ca2(double ca, double& m, double& s) {
  int e = 0;
  const double f = std::frexp(ca, &e);
  const bool big = std::fabs(ca) > 1.0 && std::isfinite(ca);
  m = big ? f * f : ca * ca;
  s = big ? std::ldexp(1.0, -2 * e) : 1.0;
}
}  // namespace gop
