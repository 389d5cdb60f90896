// The fluid's stress-energy tensor on the vertices and the regrid error
// estimate: the two scheduled routines of AsterX outside the RHS and
// post-step groups that read the evolved state every step.
//
//   k_tmunu2<ZVEC>,        AsterX_Tmunu (AsterX/src/tmunu.cxx:19-178): the
//   k_tmunu4<ZVEC>         cell-centred primitives interpolated to each
//                          interior vertex (AsterUtils/src/aster_interp.hxx:
//                          97-148, order 2 or 4), T_{mu nu} of the ideal
//                          MHD fluid added to eTtt .. eTzz
//   k_regrid_error<M>      AsterX_EstimateError (AsterX/src/
//                          estimate_error.cxx:70-144) with the indicators of
//                          AsterX/src/estimate_error.hxx:14-86
//
// k_tmunu2 (a plane's vertices row after row, 72 loads a vertex through L1,
// which bounds it) and k_regrid_error (rows of 128 along x, HBM) run one thread
// per point; k_tmunu4 runs tiles.  This file is compiled without multiply-add
// contraction and keeps the reference's operation order (sums from left to
// right, products left-associated as written), so the results are the
// reference's bits: IEEE division and square root round the same on both.
#include <algorithm>

#include "axb_internal.hxx"

using namespace axb;

namespace {

// ---------------------------------------------------------------------------
// AsterX_Tmunu
// ---------------------------------------------------------------------------
struct TmunuArgs {
  BoxDev b;
  const double *f[9]; // rho, eps, press, B^x..B^z, v^x..v^z or z^x..z^z
  const double *g[6], *alp, *beta[3];
  double *eT[10];
};

// Order 2: the 8 cells around vertex I (cell I - di - dj - dk), summed in
// the reference's loop order (dk, dj, di), divided by 8.
AXB_D double c2v2(const double *__restrict__ f, long long I, long long sy, long long sz) {
  double s = 0.0;
#pragma unroll
  for (int dk = 0; dk < 2; ++dk)
#pragma unroll
    for (int dj = 0; dj < 2; ++dj)
#pragma unroll
      for (int di = 0; di < 2; ++di)
        s += __ldg(f + I - di - dj * sy - dk * sz);
  return s / 8.0;
}

// T_{mu nu} of the fluid at vertex I, added to the arrays (tmunu.cxx:76-178);
// `field(v)` is field v of TmunuArgs::f interpolated there.
template <bool ZVEC, class Field>
AXB_D void tmunu_point(const TmunuArgs &a, long long I, const Field &field) {
  const double rho_avg = field(0), eps_avg = field(1), press_avg = field(2);
  const double Bup[3] = {field(3), field(4), field(5)};
  const sym3 g{__ldg(a.g[0] + I), __ldg(a.g[1] + I), __ldg(a.g[2] + I),
               __ldg(a.g[3] + I), __ldg(a.g[4] + I), __ldg(a.g[5] + I)};
  const double alp = __ldg(a.alp + I);
  const double beta_up[3] = {__ldg(a.beta[0] + I), __ldg(a.beta[1] + I),
                             __ldg(a.beta[2] + I)};
  double beta_low[3];
  lower3(g, beta_up, beta_low);
  const double beta_sq = dot3(beta_low, beta_up);

  double vup[3], vlow[3], w;
  const double vz[3] = {field(6), field(7), field(8)};
  if constexpr (!ZVEC) {
    for (int d = 0; d < 3; ++d)
      vup[d] = vz[d];
    lower3(g, vup, vlow);
    w = 1.0 / sqrt(1.0 - dot3(vup, vlow));
  } else {
    double zlow[3];
    lower3(g, vz, zlow);
    w = sqrt(1.0 + dot3(vz, zlow));
    for (int d = 0; d < 3; ++d) {
      vup[d] = vz[d] / w;
      vlow[d] = zlow[d] / w;
    }
  }

  const double rhW2 = (rho_avg * (1.0 + eps_avg) + press_avg) * w * w;
  const double ut_low = -alp + dot3(beta_low, vup);
  double ui_up[3];
  for (int d = 0; d < 3; ++d)
    ui_up[d] = vup[d] - beta_up[d] / alp;
  const double bst_up = w * (dot3(Bup, vlow)) / alp;
  double bsi_up[3];
  for (int d = 0; d < 3; ++d)
    bsi_up[d] = (Bup[d] + alp * bst_up * w * ui_up[d]) / w;
  const double gtt = -alp * alp + beta_sq;
  const double bst_low = bst_up * gtt + dot3(bsi_up, beta_low);
  double gb[3], bsi_low[3];
  lower3(g, bsi_up, gb);
  for (int d = 0; d < 3; ++d)
    bsi_low[d] = bst_up * beta_low[d] + gb[d];
  const double bs2 = bst_up * bst_low + dot3(bsi_up, bsi_low);
  const double w2 = w * w;

  const double t00 = rhW2 * ut_low * ut_low + press_avg * gtt +
                     (w2 * ut_low * ut_low + 0.5 * gtt) * bs2 - bst_low * bst_low;
  double t0[3];
  for (int d = 0; d < 3; ++d)
    t0[d] = rhW2 * ut_low * vlow[d] + press_avg * beta_low[d] +
            (w2 * ut_low * vlow[d] + 0.5 * beta_low[d]) * bs2 - bst_low * bsi_low[d];
  auto tij = [&](int p, int q) {
    return rhW2 * vlow[p] * vlow[q] + press_avg * g(p, q) +
           (w2 * vlow[p] * vlow[q] + 0.5 * g(p, q)) * bs2 - bsi_low[p] * bsi_low[q];
  };
  const double t[10] = {t00,       t0[0],     t0[1],     t0[2],     tij(0, 0),
                        tij(0, 1), tij(0, 2), tij(1, 1), tij(1, 2), tij(2, 2)};
#pragma unroll
  for (int c = 0; c < 10; ++c)
    a.eT[c][I] = a.eT[c][I] + t[c];
}

// Order 2: one thread per interior vertex [ng, ng + n], a plane's vertices row
// after row (rows of n + 1 cut into blocks of 128 leave the second block of
// each with one thread at n = 128); the 8 cells around a vertex from L1/L2.
template <bool ZVEC> __global__ void __launch_bounds__(128) k_tmunu2(const TmunuArgs a) {
  const BoxDev &b = a.b;
  const int flat = blockIdx.x * blockDim.x + threadIdx.x, w = b.n[0] + 1;
  const int row = flat / w;
  if (row > b.n[1])
    return;
  const long long I = b.at(b.ng + flat - row * w, b.ng + row, b.ng + blockIdx.y);
  tmunu_point<ZVEC>(a, I, [&](int v) { return c2v2(a.f[v], I, b.sy, b.sz); });
}

// Order 4: the cubic Lagrange weights (-1, 9, 9, -1)/16 on cells I-2 .. I+1
// along each direction, applied direction i first, then j, then k, for the
// three cyclic orders (i, j, k) = (x, y, z), (y, z, x), (z, x, y), all
// twelve final terms accumulated in one running sum, divided by 3.
//
// A vertex alone needs 3 x 64 loads and 3 x 84 multiply-adds per field (one
// thread per vertex ran 4.5 k FP64 operations and 1.7 k loads, bound by L1
// and by instruction fetch: 2635 us for 129^3 vertices against 104 us of
// HBM traffic; now 611 us, bound by the shared-memory and shuffle traffic of
// 16 warps per SM).  The first- and second-direction sums of one vertex are those
// of its neighbours, so a block forms each once: a tile of 29 x 13 x 3
// vertices, 32 lanes along x (x sums by shuffles), 16 rows along y (y sums
// through shared memory), 6 planes in z per thread (z sums in registers).
// Every sum is the same terms in the same order as before, so the bits are
// the same.  One field at a time through a rolled loop (the code of nine
// unrolled fields does not fit the instruction cache), its results parked in
// the thread's own shared-memory slots; the next field's loads are issued
// ahead of this one's sums.
constexpr int T4_X = 29, T4_Y = 13, T4_Z = 3; // vertices of a tile
constexpr int T4_ROWS = T4_Y + 3, T4_P = T4_Z + 3;
constexpr int T4_N = 32 * T4_ROWS; // threads
constexpr int T4_SMEM = (2 * T4_P + T4_Z + 9 * T4_Z) * T4_N * int(sizeof(double));

AXB_D double cubic(double a, double b, double c, double d) {
  double s = -1.0 / 16.0 * a;
  s += 9.0 / 16.0 * b;
  s += 9.0 / 16.0 * c;
  s += -1.0 / 16.0 * d;
  return s;
}
// the cubic sum over lanes l-2 .. l+1 (lanes 2 .. 30 get theirs)
AXB_D double cubic_x(double v) {
  const double a = __shfl_up_sync(0xffffffffu, v, 2), b = __shfl_up_sync(0xffffffffu, v, 1),
               d = __shfl_down_sync(0xffffffffu, v, 1);
  return cubic(a, b, v, d);
}
// the cubic sum over rows r-2 .. r+1 of the plane at p (this thread's slot;
// `v` is its own value); rows without all four neighbours get no sum
AXB_D double cubic_y(const double *p, double v, bool ok) {
  return ok ? cubic(p[-64], p[-32], v, p[32]) : 0.0;
}

template <bool ZVEC> __global__ void __launch_bounds__(T4_N, 1) k_tmunu4(const TmunuArgs a) {
  extern __shared__ double sm[];
  const BoxDev &b = a.b;
  const int lane = threadIdx.x, row = threadIdx.y;
  const int t = row * 32 + lane;
  double *const s_f = sm + t;                  // the field's planes
  double *const s_x = s_f + T4_P * T4_N;       // their x sums
  double *const s_zx = s_x + T4_P * T4_N;      // x sums of the z sums
  double *const s_res = s_zx + T4_Z * T4_N;    // results, field by field
  const int i = b.ng + int(blockIdx.x) * T4_X + lane - 2;
  const int j = b.ng + int(blockIdx.y) * T4_Y + row - 2;
  const int k0 = b.ng + int(blockIdx.z) * T4_Z;
  // cells past ng + n + 1 are needed by no vertex of the box
  long long at[T4_P];
#pragma unroll
  for (int p = 0; p < T4_P; ++p)
    at[p] = b.at(min(i, b.ng + b.n[0] + 1), min(j, b.ng + b.n[1] + 1),
                 min(k0 - 2 + p, b.ng + b.n[2] + 1));
  const bool row_ok = row >= 2 && row < T4_ROWS - 1;
  double f[T4_P], fn[T4_P];
#pragma unroll
  for (int p = 0; p < T4_P; ++p)
    fn[p] = __ldg(a.f[0] + at[p]);
#pragma unroll 1
  for (int v = 0; v < 9; ++v) {
#pragma unroll
    for (int p = 0; p < T4_P; ++p)
      f[p] = fn[p];
    if (v < 8) {
      const double *nf = a.f[v + 1];
#pragma unroll
      for (int p = 0; p < T4_P; ++p)
        fn[p] = __ldg(nf + at[p]);
    }
    double gx[T4_P], gzx[T4_Z];
#pragma unroll
    for (int p = 0; p < T4_P; ++p)
      gx[p] = cubic_x(f[p]);
#pragma unroll
    for (int q = 0; q < T4_Z; ++q)
      gzx[q] = cubic_x(cubic(f[q], f[q + 1], f[q + 2], f[q + 3]));
    __syncthreads(); // the previous field's sums are read
#pragma unroll
    for (int p = 0; p < T4_P; ++p) {
      s_f[p * T4_N] = f[p];
      s_x[p * T4_N] = gx[p];
    }
#pragma unroll
    for (int q = 0; q < T4_Z; ++q)
      s_zx[q * T4_N] = gzx[q];
    __syncthreads();
    double avg[T4_Z], gy[T4_P];
    // (x, y, z): the y sums of the x sums, summed over z
    {
      double gxy[T4_P];
#pragma unroll
      for (int p = 0; p < T4_P; ++p)
        gxy[p] = cubic_y(s_x + p * T4_N, gx[p], row_ok);
#pragma unroll
      for (int q = 0; q < T4_Z; ++q)
        avg[q] = cubic(gxy[q], gxy[q + 1], gxy[q + 2], gxy[q + 3]);
    }
    // (y, z, x): the z sums of the y sums, summed over x
#pragma unroll
    for (int p = 0; p < T4_P; ++p)
      gy[p] = cubic_y(s_f + p * T4_N, f[p], row_ok);
#pragma unroll
    for (int q = 0; q < T4_Z; ++q) {
      const double s = cubic(gy[q], gy[q + 1], gy[q + 2], gy[q + 3]);
      const double sa = __shfl_up_sync(0xffffffffu, s, 2), sb = __shfl_up_sync(0xffffffffu, s, 1),
                   sd = __shfl_down_sync(0xffffffffu, s, 1);
      avg[q] += -1.0 / 16.0 * sa;
      avg[q] += 9.0 / 16.0 * sb;
      avg[q] += 9.0 / 16.0 * s;
      avg[q] += -1.0 / 16.0 * sd;
    }
    // (z, x, y): the x sums of the z sums, summed over y
    if (row_ok) {
#pragma unroll
      for (int q = 0; q < T4_Z; ++q) {
        const double *p = s_zx + q * T4_N;
        avg[q] += -1.0 / 16.0 * p[-64];
        avg[q] += 9.0 / 16.0 * p[-32];
        avg[q] += 9.0 / 16.0 * gzx[q];
        avg[q] += -1.0 / 16.0 * p[32];
        s_res[(v * T4_Z + q) * T4_N] = avg[q] / 3.0;
      }
    }
  }
  if (!row_ok || lane < 2 || lane > 30 || i > b.ng + b.n[0] || j > b.ng + b.n[1])
    return;
#pragma unroll 1
  for (int q = 0; q < T4_Z; ++q) {
    if (k0 + q > b.ng + b.n[2])
      break;
    tmunu_point<ZVEC>(a, b.at(i, j, k0 + q),
                      [&](int v) { return s_res[(v * T4_Z + q) * T4_N]; });
  }
}

template <bool ZVEC> int launch_tmunu(int order, const TmunuArgs &a, cudaStream_t s) {
  const int *n = a.b.n;
  if (order == 2) {
    const long long plane = (long long)(n[0] + 1) * (n[1] + 1);
    if (plane > 0x7fffff00LL)
      return AXB_ERR_TOO_LARGE;
    k_tmunu2<ZVEC><<<dim3(unsigned((plane + 127) / 128), n[2] + 1), 128, 0, s>>>(a);
    return AXB_OK;
  }
  if (cudaFuncSetAttribute(k_tmunu4<ZVEC>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           T4_SMEM) != cudaSuccess)
    return AXB_ERR_CUDA;
  const dim3 grid((n[0] + T4_X) / T4_X, (n[1] + T4_Y) / T4_Y, (n[2] + T4_Z) / T4_Z);
  k_tmunu4<ZVEC><<<grid, dim3(32, T4_ROWS), T4_SMEM, s>>>(a);
  return AXB_OK;
}

// ---------------------------------------------------------------------------
// AsterX_EstimateError
// ---------------------------------------------------------------------------
constexpr int MAXVARS = 9; // the reference asserts NregridVars < 10

struct ErrorArgs {
  BoxDev b;
  const double *var[MAXVARS];
  int nvars;
  double epsilon_err;
  double *err;
};

// std::max over an initializer list: the first largest, NaN kept only when
// it comes first
AXB_D double max_il(double a, double b) { return (a < b) ? b : a; }

template <int M>
AXB_D double indicator(const double *__restrict__ f, long long I, const long long st[3],
                       double epsilon_err) {
  if constexpr (M == AXB_REGRID_FIRST_GRAD) {
    double errp = 0.0, errm = 0.0;
    const double v0 = __ldg(f + I);
    for (int d = 0; d < 3; ++d) {
      const double vm = __ldg(f + I - st[d]), vp = __ldg(f + I + st[d]);
      errp += (vp - v0) * (vp - v0);
      errm += (v0 - vm) * (v0 - vm);
    }
    return sqrt(max_il(errp, errm));
  } else {
    double err = 0.0;
    const double v0 = __ldg(f + I);
    for (int d = 0; d < 3; ++d) {
      const double vm = __ldg(f + I - st[d]), vp = __ldg(f + I + st[d]);
      if constexpr (M == AXB_REGRID_FIRST_DERIV) {
        err = max_il(max_il(err, fabs(v0 - vm)), fabs(vp - v0));
      } else if constexpr (M == AXB_REGRID_SECOND_DERIV) {
        err = max_il(err, fabs(vp + vm - 2 * v0));
      } else {
        const double dp = vp - v0, dm = v0 - vm;
        const double varsigma = fabs(vp) + 2 * fabs(v0) + fabs(vm);
        const double num = fabs(dp - dm) * fabs(dp - dm);
        const double den = (fabs(dp) + fabs(dm) + epsilon_err * varsigma) *
                           (fabs(dp) + fabs(dm) + epsilon_err * varsigma);
        err = max_il(err, sqrt(num / den));
      }
    }
    return err;
  }
}

// Interior cells; x along the block's threads.
template <int M> __global__ void __launch_bounds__(128) k_regrid_error(const ErrorArgs a) {
  const BoxDev &b = a.b;
  const int i = b.ng + blockIdx.x * blockDim.x + threadIdx.x;
  const int j = b.ng + blockIdx.y;
  const int k = b.ng + blockIdx.z;
  if (i >= b.ng + b.n[0])
    return;
  const long long I = b.at(i, j, k);
  const long long st[3] = {1, b.sy, b.sz};
  double e = 0.0;
  for (int v = 0; v < a.nvars; ++v)
    e = max_il(e, indicator<M>(a.var[v], I, st, a.epsilon_err));
  a.err[I] = e;
}

template <int M> void launch_error(const ErrorArgs &a, cudaStream_t s) {
  const dim3 grid((a.b.n[0] + 127) / 128, a.b.n[1], a.b.n[2]);
  k_regrid_error<M><<<grid, 128, 0, s>>>(a);
}

bool grid_ok(const axb_box &b, int extra) {
  for (int d = 0; d < 3; ++d)
    if (b.n[d] < 1 || b.n[d] + extra > 65535)
      return false;
  return true;
}

} // namespace

AXB_API int axb_tmunu(axb_ctx *c, const axb_box *box, const axb_fields *f,
                      const axb_params *p, int interp_order, double *const eT[10],
                      void *stream) {
  if (!c || !box || !f || !p || !eT)
    return AXB_ERR_ARG;
  if (interp_order != 2 && interp_order != 4)
    return AXB_ERR_ARG;
  if (box->ng < (interp_order == 4 ? 2 : 1))
    return AXB_ERR_GHOSTS;
  if (!grid_ok(*box, 1))
    return AXB_ERR_ARG;
  if (p->recon_type != AXB_RECVAR_V && p->recon_type != AXB_RECVAR_Z &&
      p->recon_type != AXB_RECVAR_S)
    return AXB_ERR_ARG;
  TmunuArgs a;
  a.b = make_box(*box);
  // s_vec reconstructs svec at the faces; the vertex tensor interpolates
  // the velocity as v_vec does (tmunu.cxx:35 tests recon_type == "v_vec"
  // only, so s_vec takes the zvec branch there): the zvec grid functions
  // are read for both z_vec and s_vec
  const bool zv = p->recon_type != AXB_RECVAR_V;
  const double *req[] = {f->gf[AXB_GF_rho], f->gf[AXB_GF_eps], f->gf[AXB_GF_press],
                         f->gf[AXB_GF_alp]};
  for (const double *q : req)
    if (!q)
      return AXB_ERR_ARG;
  a.f[0] = f->gf[AXB_GF_rho];
  a.f[1] = f->gf[AXB_GF_eps];
  a.f[2] = f->gf[AXB_GF_press];
  a.alp = f->gf[AXB_GF_alp];
  for (int d = 0; d < 3; ++d) {
    a.f[3 + d] = f->gf[AXB_GF_Bvecx + d];
    a.f[6 + d] = f->gf[(zv ? AXB_GF_zvec_x : AXB_GF_velx) + d];
    a.beta[d] = f->gf[AXB_GF_betax + d];
    if (!a.f[3 + d] || !a.f[6 + d] || !a.beta[d])
      return AXB_ERR_ARG;
  }
  for (int q = 0; q < 6; ++q) {
    a.g[q] = f->gf[AXB_GF_gxx + q];
    if (!a.g[q])
      return AXB_ERR_ARG;
  }
  for (int q = 0; q < 10; ++q) {
    a.eT[q] = eT[q];
    if (!eT[q])
      return AXB_ERR_ARG;
  }
  cudaStream_t s = (cudaStream_t)stream;
  axb_mark(c, AXB_R_TMUNU, s, true);
  const int rc = zv ? launch_tmunu<true>(interp_order, a, s)
                    : launch_tmunu<false>(interp_order, a, s);
  axb_mark(c, AXB_R_TMUNU, s, false);
  if (rc)
    return rc;
  return cudaGetLastError() == cudaSuccess ? AXB_OK : AXB_ERR_CUDA;
}

AXB_API int axb_estimate_error(axb_ctx *c, const axb_box *box, const double *const *vars,
                               int nvars, int method, double epsilon_err,
                               double *regrid_error, void *stream) {
  if (!c || !box || !vars || !regrid_error || nvars < 1 || nvars > MAXVARS)
    return AXB_ERR_ARG;
  if (method < AXB_REGRID_FIRST_DERIV || method > AXB_REGRID_FIRST_GRAD)
    return AXB_ERR_ARG;
  if (box->ng < 1)
    return AXB_ERR_GHOSTS;
  if (!grid_ok(*box, 0))
    return AXB_ERR_ARG;
  ErrorArgs a;
  a.b = make_box(*box);
  a.nvars = nvars;
  a.epsilon_err = epsilon_err;
  a.err = regrid_error;
  for (int v = 0; v < nvars; ++v) {
    if (!vars[v])
      return AXB_ERR_ARG;
    a.var[v] = vars[v];
  }
  cudaStream_t s = (cudaStream_t)stream;
  axb_mark(c, AXB_R_ERROR, s, true);
  switch (method) {
  case AXB_REGRID_FIRST_DERIV:
    launch_error<AXB_REGRID_FIRST_DERIV>(a, s);
    break;
  case AXB_REGRID_SECOND_DERIV:
    launch_error<AXB_REGRID_SECOND_DERIV>(a, s);
    break;
  case AXB_REGRID_SECOND_DERIV_NORM:
    launch_error<AXB_REGRID_SECOND_DERIV_NORM>(a, s);
    break;
  default:
    launch_error<AXB_REGRID_FIRST_GRAD>(a, s);
    break;
  }
  axb_mark(c, AXB_R_ERROR, s, false);
  return cudaGetLastError() == cudaSuccess ? AXB_OK : AXB_ERR_CUDA;
}
