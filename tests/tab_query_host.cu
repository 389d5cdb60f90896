// Host-side C wrapper around the tabulated EOS's queries
// (asterx_b200/csrc/axb_tab.cuh) for tests/test_tab_query.py.  Test
// infrastructure: compiled by nvcc as host code.
#include "../asterx_b200/csrc/axb_tab.cuh"

namespace {
axb::EosTab make(const int *n, const double *lr, const double *lt, const double *ye,
                 const double *y, double shift, double eps_min, int monotone) {
  axb::EosTab t{};
  const double *ax[3] = {lr, lt, ye};
  for (int d = 0; d < 3; ++d) {
    t.n[d] = n[d];
    t.x[d] = ax[d];
    t.idx[d] = 1.0 / (ax[d][1] - ax[d][0]);
    t.x0[d] = ax[d][0];
    t.xlast[d] = ax[d][n[d] - 1];
  }
  t.y = y;
  t.shift = shift;
  t.monotone = monotone;
  t.rgrho = axb::Range{std::exp(t.x0[0]), std::exp(t.xlast[0])};
  t.rgtemp = axb::Range{std::exp(t.x0[1]), std::exp(t.xlast[1])};
  t.rgeps = axb::Range{eps_min, 1e300};
  return t;
}
} // namespace

// out[0..3]: face_thermo's eps, press, cs2, eps2; out[4..7]: the same from the
// separate queries
extern "C" __attribute__((visibility("default"))) void
tab_face(const int *n, const double *lr, const double *lt, const double *ye, const double *y,
         double shift, double eps_min, int monotone, double rho, double temp, double yeq,
         double *out) {
  const axb::EosTab t = make(n, lr, lt, ye, y, shift, eps_min, monotone);
  const auto o = t.face_thermo(rho, temp, yeq);
  out[0] = o.eps;
  out[1] = o.press;
  out[2] = o.cs2;
  out[3] = o.eps2;
  out[4] = t.eps_from_valid_rho_temp_ye(rho, temp, yeq);
  out[5] = t.press_from_valid_rho_temp_ye(rho, temp, yeq);
  double e = out[4];
  const double cs = t.csnd_from_valid_rho_eps_ye(rho, e, yeq);
  out[6] = cs * (!(e == out[4]) ? t.csnd_from_valid_rho_eps_ye(rho, e, yeq) : cs);
  out[7] = e;
}

// out[0..3]: press and eps of press_query, ln T and eps of logtemp_query
extern "C" __attribute__((visibility("default"))) int
tab_query(const int *n, const double *lr, const double *lt, const double *ye, const double *y,
          double shift, double eps_min, int monotone, double rho, double eps, double yeq,
          int hint, double *out) {
  const axb::EosTab t = make(n, lr, lt, ye, y, shift, eps_min, monotone);
  const auto p = t.press_query(rho, eps, yeq, hint);
  const auto l = t.logtemp_query(rho, eps, yeq, hint);
  out[0] = p.value;
  out[1] = p.eps;
  out[2] = l.value;
  out[3] = l.eps;
  return l.hint;
}
