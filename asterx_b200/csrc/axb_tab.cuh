// Tabulated 3D EOS on the device (EOSX eos_3p_tabulated3d).
//
//   queries        EOSX/src/eos_3p_tabulated3d/eos_3p_tabulated3d.hxx:197-350
//   interpolation  EOSX/src/utils/eos_linear_interp_ND.hxx:50-206 (uniform
//                  axes, index clamped to [0, n-2], linear along ln rho, then
//                  ln T, then Ye)
//   T inversion    the root of the interpolant, found exactly (logtemp_root);
//                  Brent's zero finder (EOSX/src/utils/eos_brent.hxx:7-170)
//                  where the table is not monotonic in T
//
// Layout: only the four variables the hot path reads are kept, interleaved
// per node as (ln P, ln(eps + shift), s, cs^2) -- variables 0, 1, 2 and 4 of
// the reference's 19 -- so that one trilinear corner is one 32-byte DRAM
// sector; the 200 x 100 x 60 synthetic table is 38 MB and stays resident in
// the 126 MB L2 across a step.  The values are copied bit for bit.
#pragma once

#include "axb_eos.cuh"

namespace axb {

// a query as a function call on the device (see EosTab::press_query)
#ifdef __CUDACC__
#define AXB_TAB_CALL __host__ __device__ __noinline__
#else
#define AXB_TAB_CALL
#endif

constexpr int TAB_NV = 4;
enum { TAB_PRESS = 0, TAB_EPS = 1, TAB_S = 2, TAB_CS2 = 3 };
// Iteration cap of the temperature root find.  The reference's loop has no
// cap; Brent's method needs at most about (log2(interval / tol))^2 ~ 2500
// steps here and in practice a few dozen.  A capped query sets
// AXB_EW_ROOT_CAP in the status word instead of spinning.
constexpr int TAB_BRENT_MAXIT = 10000;

struct EosTab {
  int n[3];
  const double *x[3]; // axis values (device)
  double idx[3];      // 1 / (x[d][1] - x[d][0])
  double x0[3], xlast[3];
  const double *y; // TAB_NV values per node, node = i + n0*(j + n1*k)
  double shift;
  Range rgrho, rgye, rgtemp, rgeps;
  // ln eps grows with T at every (rho, Ye) node by more than the rounding of
  // its interpolation (set where the table is read): any search along T then
  // finds the one cell that holds a value, so a query may start from a guess
  int monotone;
  unsigned int *err; // status error word (device descriptor only), or null

  static constexpr bool kTabulated = true;

  // The cell of the uniform axis d holding xin, clamped to [0, n - 2]
  // (eos_linear_interp_ND.hxx:50-65).  The clamps act on the floating-point
  // position before it becomes an integer, so a NaN query (the logarithm of
  // a non-positive temperature that press_from_valid_rho_temp_ye takes
  // before clamping) and an infinite one map to an end cell instead of an
  // undefined conversion; finite queries are unchanged.
  AXB_HD int find(int d, double xin) const {
    const double xL = xin - x0[d];
    if (!(xL > 0))
      return 0;
    const double t = xL * idx[d];
    if (!(t < double(n[d] - 2)))
      return n[d] - 2;
    return static_cast<int>(t);
  }
  // The rho and Ye cells of a query and the weights in them, found once: all
  // node values and interpolations of the query share them.
  struct Cell {
    int i, k;
    double u, v;
  };
  AXB_HD Cell locate(double lrho, double ye) const {
    Cell c;
    c.i = find(0, lrho);
    c.k = find(2, ye);
    c.u = (lrho - x[0][c.i]) / (x[0][c.i + 1] - x[0][c.i]);
    c.v = (ye - x[2][c.k]) / (x[2][c.k + 1] - x[2][c.k]);
    return c;
  }
  // linear in ln rho at temperature node j and Ye node c.k + o
  AXB_HD double at_rho(int var, const Cell &c, int j, int o) const {
    const double *p =
        y + TAB_NV * (c.i + (long long)n[0] * (j + (long long)n[1] * (c.k + o))) + var;
    const double y0 = p[0], y1 = p[TAB_NV];
    return (y1 - y0) * c.u + y0;
  }
  // ln eps at temperature node j
  AXB_HD double eps_node(const Cell &c, int j) const {
    const double a = at_rho(TAB_EPS, c, j, 0), b = at_rho(TAB_EPS, c, j, 1);
    return (b - a) * c.v + a;
  }
  // the trilinear interpolant, along ln rho, then ln T, then Ye
  AXB_HD double tri(int var, const Cell &c, double lt) const {
    const int j = find(1, lt);
    return tri_in(var, c, j, (lt - x[1][j]) / (x[1][j + 1] - x[1][j]));
  }
  // the same with the T cell and the weight in it given
  AXB_HD double tri_in(int var, const Cell &c, int j, double w) const {
    double B[2];
#pragma unroll
    for (int o = 0; o < 2; ++o) {
      const double a = at_rho(var, c, j, o), b = at_rho(var, c, j + 1, o);
      B[o] = (b - a) * w + a;
    }
    return (B[1] - B[0]) * c.v + B[0];
  }

  template <class Fn>
  AXB_HD static double zero_brent(double a, double b, double t, const Fn &f,
                                  bool &capped) {
    double sa = a, sb = b, fa = f(sa), fb = f(sb);
    double c = sa, fc = fa, e = sb - sa, d = e;
    const double macheps = 2.220446049250313e-16;
    capped = true;
    for (int it = 0; it < TAB_BRENT_MAXIT; ++it) {
      if (fabs(fc) < fabs(fb)) {
        sa = sb;
        sb = c;
        c = sa;
        fa = fb;
        fb = fc;
        fc = fa;
      }
      const double tol = 2.0 * macheps * fabs(sb) + t;
      const double m = 0.5 * (c - sb);
      if (fabs(m) <= tol || fb == 0.0) {
        capped = false;
        break;
      }
      if (fabs(e) < tol || fabs(fa) <= fabs(fb)) {
        e = m;
        d = e;
      } else {
        double s = fb / fa, p, q;
        if (sa == c) {
          p = 2.0 * m * s;
          q = 1.0 - s;
        } else {
          q = fa / fc;
          const double r = fb / fc;
          p = s * (2.0 * m * q * (q - r) - (sb - sa) * (r - 1.0));
          q = (q - 1.0) * (r - 1.0) * (s - 1.0);
        }
        if (0.0 < p)
          q = -q;
        else
          p = -p;
        s = e;
        e = d;
        if (2.0 * p < 3.0 * m * q - fabs(tol * q) && p < fabs(0.5 * s * q)) {
          d = p / q;
        } else {
          e = m;
          d = e;
        }
      }
      sa = sb;
      fa = fb;
      if (tol < fabs(d))
        sb = sb + d;
      else if (0.0 < m)
        sb = sb + tol;
      else
        sb = sb - tol;
      fb = f(sb);
      if ((0.0 < fb && 0.0 < fc) || (fb <= 0.0 && fc <= 0.0)) {
        c = sa;
        fc = fa;
        e = sb - sa;
        d = e;
      }
    }
    return sb;
  }

  // logtemp_from_valid_rho_eps_ye (:197-228): clamps eps in place.  `c` is
  // the cell of (ln of the clamped rho, Ye); `hint` a guess of the T cell
  // (any value), replaced by the cell found.
  AXB_HD double logtemp_at(const Cell &c, double lrho, double &eps, double ye, int &hint) const {
    eps = fmax(eps + shift, rgeps.min + shift) - shift;
    const double leps = log(eps + shift);
    if (monotone && hint >= 1 && hint < n[1] - 2 && c.u >= 0.0 && c.u <= 1.0 && c.v >= 0.0 &&
        c.v <= 1.0) {
      // strictly inside the table (Ye is not clamped, so the weights are
      // looked at) the bracketing cell is the search's result
      const double e0 = eps_node(c, hint), e1 = eps_node(c, hint + 1);
      if (e0 <= leps && leps < e1)
        return in_cell(hint, leps, e0, e1);
    }
    const double vmin = tri(TAB_EPS, c, x0[1]);
    const double vmax = tri(TAB_EPS, c, xlast[1]);
    if (leps <= vmin) {
      eps = exp(vmin) - shift;
      return x0[1];
    }
    if (leps >= vmax) {
      eps = exp(vmax) - shift;
      return xlast[1];
    }
    return logtemp_root(c, lrho, leps, ye, vmin, vmax, hint);
  }
  // the root of the linear equation in the T cell `j` with end values e0, e1
  AXB_HD double in_cell(int j, double leps, double e0, double e1) const {
    const double xa = x[1][j], xb = x[1][j + 1];
    const double lam = fmin(fmax((leps - e0) / (e1 - e0), 0.0), 1.0);
    return xa + lam * (xb - xa);
  }

  // The root in ln T of leps = interp(EPS, lrho, ln T, ye).  The
  // interpolant is linear in ln T within each cell of the T axis (the
  // trilinear scheme interpolates along ln T between the two T nodes of the
  // cell), so the root is found exactly: a bisection over the nodes' values
  // (which grow with T for a thermodynamic table) locates the cell, and the
  // linear equation of that cell gives the root.  The reference runs Brent's
  // method on the whole axis to 1e-14 (eos_3p_tabulated3d.hxx:219-225,
  // eos_brent.hxx); both land on the same root of the same interpolant,
  // here to rounding.  Where the node values are not increasing around the
  // root, the reference's Brent search is run instead.  The bisection
  // evaluates the interpolant at temperature nodes, where it is the bilinear
  // interpolant in (ln rho, Ye) of that node's four values.
  AXB_HD double logtemp_root(const Cell &c, double lrho, double leps, double ye, double vlo,
                             double vhi, int &hint) const {
    // vlo = interp at node 0 < leps < vhi = interp at the last node.
    int lo = 0, hi = n[1] - 1;
    while (hi - lo > 1) {
      const int mid = (lo + hi) >> 1;
      const double vm = eps_node(c, mid);
      if (vm <= leps) {
        lo = mid;
        vlo = vm;
      } else {
        hi = mid;
        vhi = vm;
      }
    }
    hint = lo;
    // the cell [x_lo, x_lo+1]: interp = e0 + (e1 - e0) * lambda, lambda in [0, 1]
    const double e0 = eps_node(c, lo), e1 = eps_node(c, lo + 1);
    if (!(vlo <= leps && leps <= vhi) || !(e1 > e0)) {
      bool capped;
      const double lt = zero_brent(
          x0[1], xlast[1], 1.e-14, [&](double l) { return leps - tri(TAB_EPS, c, l); }, capped);
#ifdef __CUDA_ARCH__
      if (capped && err)
        atomicOr(err, AXB_EW_ROOT_CAP);
#endif
      return lt;
    }
    return in_cell(lo, leps, e0, e1);
  }
  AXB_HD double lr_clamped(double rho) const {
    return log(fmin(fmax(rho, rgrho.min), rgrho.max));
  }
  AXB_HD double lt_clamped(double temp) const {
    return log(fmin(fmax(temp, rgtemp.min), rgtemp.max));
  }
  // The queries are function calls, not inlined: a recovery evaluates them
  // at a dozen places, and inlined the kernel did not fit the instruction
  // cache (16 of its 55 stalled cycles per issued instruction were fetches).
  struct Query {
    double value, eps; // eps as the query leaves it
    int hint;
  };
  AXB_TAB_CALL Query press_query(double rho, double eps, double ye, int hint) const {
    Query q{0.0, eps, hint};
    const double lr = lr_clamped(rho);
    const Cell c = locate(lr, ye);
    const double lt = logtemp_at(c, lr, q.eps, ye, q.hint);
    q.value = exp(tri(TAB_PRESS, c, lt));
    return q;
  }
  AXB_TAB_CALL Query logtemp_query(double rho, double eps, double ye, int hint) const {
    Query q{0.0, eps, hint};
    const double lr = lr_clamped(rho);
    q.value = logtemp_at(locate(lr, ye), lr, q.eps, ye, q.hint);
    return q;
  }
  AXB_TAB_CALL double interp(int var, double lrho, double lt, double ye) const {
    return tri(var, locate(lrho, ye), lt);
  }
  // eps, press and the product of two sound-speed queries of a face state
  // given by its temperature (fluxes.cxx:297-304,556-560): eps from the
  // clamped logarithms, press from the plain ones, as the two queries take
  // them; cs^2 at that eps.  eps2 is eps as the sound-speed query leaves it (it
  // may clamp).
  //
  // The sound-speed query inverts eps for the temperature eps came from.  Where
  // the state lies inside the table and eps grows with T there, that is the
  // temperature at hand, so cs^2 is read at it: no logarithm, node search,
  // root or product of square roots (96^3 RHS 2.36 -> 2.01 ms), and without the
  // rounding the inversion amplifies where eps hardly depends on T.
  struct FaceThermo {
    double eps, press, cs2, eps2;
  };
  AXB_TAB_CALL FaceThermo face_thermo(double rho, double temp, double ye) const {
    FaceThermo o;
    const double r = fmin(fmax(rho, rgrho.min), rgrho.max);
    const double T = fmin(fmax(temp, rgtemp.min), rgtemp.max);
    const double lr = log(r), lt = log(T);
    const Cell c = locate(lr, ye);
    const int j = find(1, lt);
    const double w = (lt - x[1][j]) / (x[1][j + 1] - x[1][j]);
    o.eps = exp(tri_in(TAB_EPS, c, j, w)) - shift;
    const bool plain = r == rho && T == temp;
    if (plain)
      o.press = exp(tri_in(TAB_PRESS, c, j, w));
    else
      o.press = exp(tri(TAB_PRESS, locate(log(rho), ye), log(temp)));
    if (plain && monotone && o.eps >= rgeps.min && c.u >= 0.0 && c.u <= 1.0 && c.v >= 0.0 &&
        c.v <= 1.0 && w >= 0.0 && w <= 1.0) {
      o.eps2 = (o.eps + shift) - shift;
      o.cs2 = tri_in(TAB_CS2, c, j, w);
      if (o.cs2 >= 0.0)
        return o; // else NaN, as the root below gives it
    }
    o.eps2 = o.eps;
    int hint = j;
    const double cs = sqrt(tri(TAB_CS2, c, logtemp_at(c, lr, o.eps2, ye, hint)));
    o.cs2 = cs * cs;
    if (!(o.eps2 == o.eps))
      o.cs2 = cs * sqrt(tri(TAB_CS2, c, logtemp_at(c, lr, o.eps2, ye, hint)));
    return o;
  }
  AXB_HD double press_over_rho(double rho, double &eps, double ye, int &hint) const {
    const Query q = press_query(rho, eps, ye, hint);
    eps = q.eps;
    hint = q.hint;
    return q.value / rho;
  }
  AXB_HD double press_from_valid_rho_eps_ye(double rho, double &eps, double ye) const {
    const Query q = press_query(rho, eps, ye, -1);
    eps = q.eps;
    return q.value;
  }
  // takes the logs of the unclamped inputs, as the reference does (:230-239)
  AXB_HD double press_from_valid_rho_temp_ye(double rho, double temp, double ye) const {
    return exp(interp(TAB_PRESS, log(rho), log(temp), ye));
  }
  AXB_HD double eps_from_valid_rho_temp_ye(double rho, double temp, double ye) const {
    return exp(interp(TAB_EPS, lr_clamped(rho), lt_clamped(temp), ye)) - shift;
  }
  // no inversion of eps(press) for the tabulated EOS: the reference prints a
  // warning, asserts, and with assertions compiled out returns 0
  // (eos_3p_tabulated3d.hxx:259-269); the recovery reaches it only when a
  // limit (v_lim, the table's largest rho, the pressure atmosphere) fires
  // with use_temperature off
  AXB_HD double eps_from_valid_rho_press_ye(double, double, double) const { return 0.0; }
  AXB_HD double logtemp(double rho, double &eps, double ye) const {
    const Query q = logtemp_query(rho, eps, ye, -1);
    eps = q.eps;
    return q.value;
  }
  AXB_HD double csnd_from_valid_rho_eps_ye(double rho, double &eps, double ye) const {
    const double lt = logtemp(rho, eps, ye);
    return sqrt(interp(TAB_CS2, lr_clamped(rho), lt, ye));
  }
  AXB_HD double temp_from_valid_rho_eps_ye(double rho, double &eps, double ye) const {
    return exp(logtemp(rho, eps, ye));
  }
  // press, temperature and entropy of a recovered state, one after another
  // (each may clamp eps, as the separate queries do); `hint` as above
  AXB_HD void press_temp_entropy(double rho, double &eps, double ye, int hint, double &press,
                                 double &temp, double &entropy) const {
    const Query p = press_query(rho, eps, ye, hint);
    press = p.value;
    Query q = logtemp_query(rho, p.eps, ye, p.hint);
    temp = exp(q.value);
    // kappa_from_valid_rho_eps_ye inverts once more: the same inversion
    // unless the last one moved eps
    if (!(q.eps == p.eps))
      q = logtemp_query(rho, q.eps, ye, q.hint);
    eps = q.eps;
    entropy = entropy_from_valid_rho_temp_ye(rho, exp(q.value), ye);
  }
  AXB_HD double entropy_from_valid_rho_temp_ye(double rho, double temp, double ye) const {
    return interp(TAB_S, lr_clamped(rho), lt_clamped(temp), ye);
  }
  AXB_HD double kappa_from_valid_rho_eps_ye(double rho, double &eps, double ye) const {
    return entropy_from_valid_rho_temp_ye(rho, temp_from_valid_rho_eps_ye(rho, eps, ye), ye);
  }
  // not defined for a table (the reference prints and asserts,
  // eos_3p_tabulated3d.hxx:315-333); the entry points reject the entropy
  // scheme with a tabulated EOS, so these are never reached
  AXB_HD double press_from_valid_rho_kappa_ye(double, double, double) const { return nan(""); }
  AXB_HD double eps_from_valid_rho_kappa_ye(double, double, double) const { return nan(""); }
};

} // namespace axb
