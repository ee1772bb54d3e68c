// crshort.cu -- test infrastructure: the short forms of crmath.cuh next to the series
// they stand in for, on the host.
#include <cstdint>

#include "../../vecgeom_b200/csrc/crmath.cuh"

using namespace vgb;

// out: sin, cos of cr_sincos and of the series; fell: calls the short form left to it
extern "C" void cs_sincos(int64_t n, const double *x, double *s, double *c, double *ss, double *cs,
                          int64_t *fell) {
  for (int64_t i = 0; i < n; ++i) {
    cr_sincos(x[i], s + i, c + i);
    cr_sincos_series(x[i], ss + i, cs + i);
    if (fabs(x[i]) < 4.0) {
      crm::DD a, b;
      double ea, eb;
      crm::sincos_short(x[i], a, b, ea, eb);
      *fell += !(crm::rounds_to_hi(a, ea) && crm::rounds_to_hi(b, eb));
    }
  }
}
// per x: sin hi, lo, cos hi, lo and the two error bounds of the short form
extern "C" void cs_short(int64_t n, const double *x, double *out) {
  for (int64_t i = 0; i < n; ++i) {
    crm::DD a, b;
    double *o = out + 6 * i;
    crm::sincos_short(x[i], a, b, o[4], o[5]);
    o[0] = a.hi, o[1] = a.lo, o[2] = b.hi, o[3] = b.lo;
  }
}
extern "C" void cs_atan2(int64_t n, const double *y, const double *x, double *t, double *ts) {
  for (int64_t i = 0; i < n; ++i) {
    t[i] = cr_atan2(y[i], x[i]);
    ts[i] = cr_atan2_series(y[i], x[i], atan2(y[i], x[i]));
  }
}
