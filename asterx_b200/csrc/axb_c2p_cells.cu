// Independent-cell recovery with the optional learned initial guess.
#include "axb_c2p_box.cuh"
#include "axb_mlp.cuh"

using namespace axb;

// ---------------------------------------------------------------------------
// Independent-cell recovery (the per-cell body of AsterX_Con2Prim_typeEoS,
// con2prim.cxx:137-416, without grid, mask or graded atmosphere), with the
// optional learned initial guess.
// ---------------------------------------------------------------------------
namespace axb {
MlpDev mlp_device_view(const axb_mlp *m);
int mlp_nf(const axb_mlp *m);
int launch_mlp_guess(const axb_cells &c, const axb_mlp *m, float2 *guess, DevStatus *status,
                     cudaStream_t s);

struct C2PCellsArgs {
  axb_cells c;
  C2PParams cp;
  int c2p_prime, c2p_second, use_entropy_fix;
  Atmo atmo;
  double gamma_noble, Zmin, gfac_over_gamma;
  int use_mlp;
  double bracket;
  MlpDev mlp;
  DevStatus *status;
};

template <class EOS>
AXB_D void run_solver_cells(int which, const EOS &eos, const C2PCellsArgs &a, Prim &pv,
                            Prim &seeds, Cons &cv, const sym3 &glo, Report &rep,
                            double zguess, double vsqguess, double xlo, double xhi) {
  if (which == AXB_C2P_NOBLE)
    noble_solve(eos, a.cp, a.atmo, a.gamma_noble, a.Zmin, pv, seeds, cv, glo, rep, zguess,
                vsqguess);
  else if (which == AXB_C2P_PALENZUELA)
    palenzuela_solve(eos, a.cp, a.atmo, pv, cv, glo, rep, xlo, xhi);
  else if (which == AXB_C2P_ENTROPY)
    entropy_solve(eos, a.cp, a.atmo, pv, cv, glo, rep);
}

// A cell's outputs; any pointer may be null.
AXB_D void c2p_cells_store(const axb_cells &c, long long i, int code, int iters_first,
                           bool fallback, const Prim &pv) {
  if (c.flag)
    c.flag[i] = code;
  if (c.fallback)
    c.fallback[i] = fallback ? 1.0 : 0.0;
  if (c.iters)
    c.iters[i] = iters_first;
  if (c.rho)
    c.rho[i] = pv.rho;
  if (c.eps)
    c.eps[i] = pv.eps;
  if (c.press)
    c.press[i] = pv.press;
  for (int q = 0; q < 3; ++q)
    if (c.vel[q])
      c.vel[q][i] = pv.vel[q];
  if (c.w_lorentz)
    c.w_lorentz[i] = pv.w_lor;
  if (c.Ye)
    c.Ye[i] = pv.Ye;
  if (c.temperature)
    c.temperature[i] = pv.temperature;
  if (c.entropy)
    c.entropy[i] = pv.entropy;
}

// Failure count and iteration histogram (every thread of the block arrives).
AXB_D void c2p_cells_epilogue(const C2PCellsArgs &a, unsigned int *s_hist, int iters_first,
                              bool failed) {
  const unsigned nfail = __popc(__ballot_sync(0xffffffffu, failed));
  if (nfail && (threadIdx.x % 32) == 0) {
    atomicAdd(&a.status->c2p_fail_count, nfail);
    atomicOr(&a.status->error_word, AXB_EW_C2P_FAIL);
  }
  if (iters_first >= 0)
    atomicAdd(&s_hist[min(iters_first, 63)], 1u);
  __syncthreads();
  for (int q = threadIdx.x; q < 64; q += blockDim.x)
    if (s_hist[q])
      atomicAdd(&a.status->c2p_iter_hist[q], (unsigned long long)s_hist[q]);
}

// The whole cascade on cell i.
template <class EOS>
AXB_D void c2p_cells_one(const C2PCellsArgs &a, const EOS &eos, const long long i,
                         int &iters_first, bool &failed) {
  const axb_cells &c = a.c;
  Cons cv;
  sym3 glo;
  {
    cv.dens = c.dens[i];
    for (int q = 0; q < 3; ++q) {
      cv.mom[q] = c.mom[q][i];
      cv.dBvec[q] = c.dB[q][i];
    }
    cv.tau = c.tau[i];
    cv.DYe = c.DYe[i];
    cv.DEnt = c.DEnt ? c.DEnt[i] : 0.0;
    glo = sym3{c.g[0][i], c.g[1][i], c.g[2][i], c.g[3][i], c.g[4][i], c.g[5][i]};
  }
  // learned guess (x = h W, W) from k_mlp_guess_tc
  double zguess = -1.0, vsqguess = -1.0, xlo = -1.0, xhi = -1.0;
  if (a.use_mlp) {
    const float2 gs = reinterpret_cast<const float2 *>(c.guess)[i];
    const double x = gs.x, W = gs.y;
    zguess = cv.dens / sqrt(det3(glo)) * x; // Z = rho h W^2 = D (h W)
    vsqguess = 1.0 - 1.0 / (W * W);
    xlo = x * (1.0 - a.bracket);
    xhi = x * (1.0 + a.bracket);
    if (!(zguess > 0.0 && zguess < 1e300 && vsqguess >= 0.0 && vsqguess < 1.0))
      zguess = vsqguess = xlo = xhi = -1.0;
  }
  bool fallback = false;
  {
    const double sqrt_detg = sqrt(det3(glo));
    const double isg = 1.0 / sqrt_detg;
    const double Bup[3] = {cv.dBvec[0] * isg, cv.dBvec[1] * isg, cv.dBvec[2] * isg};
    Prim pv;
    pv.set_nan();
    Prim seeds;
    if (c.seed_rho) {
      seeds.rho = c.seed_rho[i];
      seeds.eps = c.seed_eps[i];
      seeds.Ye = c.seed_Ye[i];
      for (int q = 0; q < 3; ++q)
        seeds.vel[q] = c.seed_vel[q][i];
      seeds.temperature = c.seed_temperature ? c.seed_temperature[i] : a.atmo.temp;
    } else { // cold start
      seeds.rho = cv.dens / sqrt_detg;
      seeds.eps = a.atmo.eps;
      seeds.Ye = cv.DYe / cv.dens;
      for (int q = 0; q < 3; ++q)
        seeds.vel[q] = 0.0;
      seeds.temperature = a.atmo.temp;
    }
    // the seed velocity is limited as in con2prim.cxx:168-209
    double v_low[3];
    lower3(glo, seeds.vel, v_low);
    const double vsq = dot3(v_low, seeds.vel);
    double zsq;
    if (vsq >= 1.0) {
      const double wlim = sqrt(1.0 + a.cp.vw_lim * a.cp.vw_lim);
      const double vlim = a.cp.vw_lim / wlim;
      for (int q = 0; q < 3; ++q)
        seeds.vel[q] *= vlim / sqrt(vsq);
      zsq = a.cp.vw_lim * a.cp.vw_lim;
    } else {
      zsq = vsq / (1.0 - vsq);
    }
    {
      double e = seeds.eps;
      seeds.press = eos.press_from_valid_rho_eps_ye(seeds.rho, e, seeds.Ye);
    }
    seeds.entropy = 0.0;
    for (int q = 0; q < 3; ++q) {
      seeds.Bvec[q] = Bup[q];
      seeds.E[q] = 0.0;
    }
    seeds.w_lor = sqrt(1.0 + zsq);
    int code;
    if (cv.dens <= sqrt_detg * a.atmo.rho_cut) {
      for (int q = 0; q < 3; ++q)
        pv.Bvec[q] = Bup[q];
      a.atmo.set(pv, cv, glo);
      code = AXB_C2P_ATMO;
      cons_floors(cv, glo);
    } else {
      cons_floors(cv, glo);
      Report r1, r2;
      code = AXB_C2P_PRIME;
      const bool guessed = zguess >= 0.0;
      const Prim seeds_plain = seeds; // the first scheme may overwrite its seeds
      run_solver_cells(a.c2p_prime, eos, a, pv, seeds, cv, glo, r1, zguess, vsqguess, xlo,
                       xhi);
      iters_first = r1.iters;
      if (r1.failed() && guessed) {
        // the guess led the first scheme astray: the plain cold start
        // (c2p_2DNoble.hxx:374-393, the plain bracket), then the plain cascade
        fallback = true;
        seeds = seeds_plain;
        pv.set_nan();
        Report rr;
        run_solver_cells(a.c2p_prime, eos, a, pv, seeds, cv, glo, rr, -1.0, -1.0, -1.0, -1.0);
        iters_first += rr.iters;
        r1 = rr;
      }
      if (r1.failed()) {
        code = AXB_C2P_SECOND;
        run_solver_cells(a.c2p_second, eos, a, pv, seeds, cv, glo, r2, -1.0, -1.0, -1.0,
                         -1.0);
      }
      bool recovered = false;
      if (r1.failed() && r2.failed() && a.use_entropy_fix) {
        Report re;
        entropy_solve(eos, a.cp, a.atmo, pv, cv, glo, re);
        recovered = !re.failed();
        if (recovered)
          code = AXB_C2P_ENTROPY_OK;
      }
      if (r1.failed() && r2.failed() && !recovered) {
        code = AXB_C2P_FAIL;
        failed = true;
        for (int q = 0; q < 3; ++q) {
          cv.dBvec[q] = sqrt_detg * Bup[q];
          pv.Bvec[q] = Bup[q];
        }
        a.atmo.set(pv, cv, glo);
      }
    }
    c2p_cells_store(c, i, code, iters_first, fallback, pv);
  }
}

template <class EOS> AXB_D void c2p_cells_body(const C2PCellsArgs &a, const EOS &eos) {
  __shared__ unsigned int s_hist[64];
  for (int q = threadIdx.x; q < 64; q += blockDim.x)
    s_hist[q] = 0;
  __syncthreads();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  int iters_first = -1;
  bool failed = false;
  if (i < a.c.n)
    c2p_cells_one(a, eos, i, iters_first, failed);
  c2p_cells_epilogue(a, s_hist, iters_first, failed);
}
// The table's queries are calls that take its address, so it stays in the
// parameter space; the ideal gas's few constants are faster by value (4.0M cells
// with use_z, Noble first 1329 -> 1273 us, entropy first 4388 -> 4270 us,
// Palenzuela first 1389 -> 1405 us).
__global__ void __launch_bounds__(128, AXB_C2P_MINB)
    k_c2p_cells_tab(const C2PCellsArgs a, const __grid_constant__ EosTab eos) {
  c2p_cells_body(a, eos);
}
__global__ void __launch_bounds__(128, AXB_C2P_MINB)
    k_c2p_cells(const C2PCellsArgs a, const EosIdeal eos) {
  c2p_cells_body(a, eos);
}

// ---------------------------------------------------------------------------
// The fast form for the ideal gas with Noble first: only the first solver's
// common path, so that it fits 8 CTAs per SM where the whole cascade takes the
// registers of 4, and without what the cascade's general form repeats (a
// cell's metric determinant, its inverse and root once; no conserved
// variables to rebuild).  Any cell that needs more -- an invalid metric,
// non-finite or over-magnetised conserved variables, a Newton search that
// does not converge, a non-positive rho or eps -- calls the cascade of
// k_c2p_cells, out of line, having written nothing.
//
// With noble_root's cheaper step, 4.0M cells: plain 1156 -> 445 us, learned
// (recovery alone) 691 -> 297 us.
//
// The cascade's 128 registers are not there in 8 CTAs per SM: a cell that needs
// it costs 1.35 times as long there, and a launch of few blocks waits for one
// cell.  So a launch that leaves the SMs room takes the form with MINB = 4:
// 1027 cells, 1 % of them failing, 237 -> 185 us (177 in k_c2p_cells).  In a
// full launch 8 win: 4.0M cells, 0 / 1 / 10 / 50 % of them failing, 438 / 4717 /
// 8942 / 9037 us (k_c2p_cells, where every cell waits for its warp's, 1152 /
// 7307 / 10535 / 10537); over-magnetised instead, 3333 / 9545 / 11579 us (4724 /
// 10996 / 12836).  Slower than k_c2p_cells are launches where most cells fail
// their first search: max_iter = 8, with 12 steps a search, 1353 -> 1875 us.
// ---------------------------------------------------------------------------

// The common path on cell i; false, having written nothing, when it leaves it.
AXB_D bool c2p_cells_common(const C2PCellsArgs &a, const EosIdeal &eos, const long long i,
                            int &iters_first) {
  const axb_cells &c = a.c;
  const sym3 g{c.g[0][i], c.g[1][i], c.g[2][i], c.g[3][i], c.g[4][i], c.g[5][i]};
  const double det = det3(g);
  const double isg = rsqrt(det);
  const double idet = isg * isg;
  const double dens = c.dens[i];
  const double D = dens * isg;
  double S[3], B[3];
  for (int q = 0; q < 3; ++q) {
    S[q] = c.mom[q][i] * isg;
    B[q] = c.dB[q][i] * isg;
  }
  double tau = c.tau[i] * isg;
  const double DYe = c.DYe[i] * isg;
  const double DEnt = c.DEnt ? c.DEnt[i] : 0.0;
  double Bl[3], Sup[3];
  lower3(g, B, Bl);
  const double Bsq = dot3(Bl, B);
  sym3 u; // the inverse metric
  u.xx = (g.yy * g.zz - g.yz * g.yz) * idet;
  u.xy = (g.xz * g.yz - g.xy * g.zz) * idet;
  u.xz = (g.xy * g.yz - g.xz * g.yy) * idet;
  u.yy = (g.xx * g.zz - g.xz * g.xz) * idet;
  u.yz = (g.xy * g.xz - g.xx * g.yz) * idet;
  u.zz = (g.xx * g.yy - g.xy * g.xy) * idet;
  lower3(u, S, Sup);
  double Ssq = dot3(S, Sup);
  // cons_floors_and_ceilings (c2p.hxx:330-369), undensitised
  const double tau_lim = 0.5 * Bsq;
  if (tau <= tau_lim)
    tau = tau_lim;
  const double slim = D + tau;
  if (Ssq > slim * slim) {
    const double f = sqrt(slim * slim / Ssq);
    for (int q = 0; q < 3; ++q) {
      S[q] *= f;
      Sup[q] *= f;
    }
    Ssq = Ssq * (f * f);
  }
  const double BiSi = dot3(S, B);
  // Near the cut (D is a few ulps off) the densitised variables are compared,
  // as every other form of the recovery compares them: with atmo_tol zero a
  // cell set to the atmosphere lies on the cut itself.  One just above it may
  // fall below after the search, by its rounding: the cascade's.
  bool atmosphere = D <= a.atmo.rho_cut, at_cut = false;
  if (fabs(D - a.atmo.rho_cut) <= 1e-14 * a.atmo.rho_cut) {
    atmosphere = dens <= sqrt(det) * a.atmo.rho_cut;
    at_cut = !atmosphere;
  }
  bool common = g.xx > 0.0 && g.xx * g.yy - g.xy * g.xy > 0.0 && det > 0.0 && isfinite(D) &&
                isfinite(Ssq) && isfinite(Bsq) && isfinite(BiSi) && isfinite(DYe) &&
                isfinite(DEnt) && !(Bsq > a.cp.Bsq_lim) && !at_cut;
  Prim pv;
  int code = AXB_C2P_PRIME;
  if (common && atmosphere) {
    a.atmo.set(pv);
    code = AXB_C2P_ATMO;
  } else if (common) {
    // start: the learned guess, or the seeds' (Z, v^2)
    double x0 = -1.0, x1 = -1.0;
    if (a.use_mlp) {
      const float2 gs = reinterpret_cast<const float2 *>(c.guess)[i];
      const double x = gs.x, W = gs.y;
      x0 = D * x; // Z = rho h W^2 = D (h W)
      x1 = 1.0 - 1.0 / (W * W);
      if (!(x0 > 0.0 && x0 < 1e300 && x1 >= 0.0 && x1 < 1.0))
        x0 = x1 = -1.0;
    }
    if (!(x0 >= 0.0)) {
      double eps = a.atmo.eps, vsq = 0.0;
      if (c.seed_rho) {
        double v[3], vl[3];
        for (int q = 0; q < 3; ++q)
          v[q] = c.seed_vel[q][i];
        lower3(g, v, vl);
        vsq = dot3(vl, v);
        if (vsq >= 1.0) // limited to v_lim, as con2prim.cxx:168-209
          vsq = a.cp.v_lim * a.cp.v_lim;
        eps = fmax(c.seed_eps[i], a.atmo.eps);
      }
      // rho = D / W, Z = (rho + eps rho + P) W^2 = D W (1 + eps + P/rho)
      const double W = rsqrt(1.0 - vsq);
      x0 = fabs(D * W * (1.0 + eps + eos.gm1 * eps));
      x1 = vsq;
    }
    const NobleRoot r =
        noble_root<true>(D, tau, Ssq, Bsq, BiSi, a.gamma_noble, a.gfac_over_gamma, a.Zmin,
                         a.cp.tol, min(a.cp.maxIter, NOBLE_CHEAP_STEPS), x0, x1);
    common = !r.slow && r.finite;
    if (common) {
      // WZ2Prim (c2p_2DNoble.hxx:192-273): W = (1 - v^2)^-1/2, rho = D / W,
      // eps = (Z / (W^2 rho) - 1) / Gamma = (Z / (W D) - 1) / Gamma
      const double om = 1.0 - r.vsq;
      const double W = rsqrt(om);
      const double iW = om * W;
      const double iD = 1.0 / D;
      pv.rho = D * iW;
      pv.w_lor = W;
      const double iZZB = 1.0 / (r.Z * (r.Z + Bsq));
      const double iZB = r.Z * iZZB;
      for (int q = 0; q < 3; ++q)
        pv.vel[q] = fma(BiSi * iZZB, B[q], Sup[q] * iZB);
      pv.eps = fma(r.Z * iW, iD, -1.0) * eos.inv_gamma;
      pv.Ye = DYe * iD;
      common = pv.rho > 0.0 && pv.eps > 0.0;
      if (common) {
        pv.press = eos.press_from_valid_rho_eps_ye(pv.rho, pv.eps, pv.Ye);
        pv.temperature = eos.temp_from_valid_rho_eps_ye(pv.rho, pv.eps, pv.Ye);
        pv.entropy = eos.kappa_from_valid_rho_eps_ye(pv.rho, pv.eps, pv.Ye);
        iters_first = r.iters;
        if (pv.rho < a.atmo.rho_cut) {
          a.atmo.set(pv);
        } else {
          Report rep;
          Cons cv;
          cv.dens = D;
          prims_floors(eos, a.cp, a.atmo, pv, cv, g, rep);
        }
      }
    }
  }
  if (common)
    c2p_cells_store(c, i, code, iters_first, false, pv);
  else
    iters_first = -1;
  return common;
}

__device__ __noinline__ void c2p_cells_cascade(const C2PCellsArgs &a, const EosIdeal &eos,
                                               long long i, int &iters_first, bool &failed) {
  c2p_cells_one(a, eos, i, iters_first, failed);
}

template <int MINB>
__global__ void __launch_bounds__(128, MINB)
    k_c2p_cells_noble(const __grid_constant__ C2PCellsArgs a,
                      const __grid_constant__ EosIdeal eos) {
  __shared__ unsigned int s_hist[64];
  for (int q = threadIdx.x; q < 64; q += blockDim.x)
    s_hist[q] = 0;
  __syncthreads();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  int iters_first = -1;
  bool failed = false;
  const bool rest = i < a.c.n && !c2p_cells_common(a, eos, i, iters_first);
  // cells that left the common path early and late take the cascade together
  // (one after another, 10 % over-magnetised cells of 1027 took 391 us, not 220)
  __syncwarp();
  if (rest)
    c2p_cells_cascade(a, eos, i, iters_first, failed);
  c2p_cells_epilogue(a, s_hist, iters_first, failed);
}
// cells from which 8 CTAs per SM win: 100003 / 200000 / 400000 cells 30 / 43 /
// 90 us at 4 and 31 / 46 / 87 at 8 CTAs per SM
constexpr long long CELLS_FULL = 1 << 18;
} // namespace axb

AXB_API int axb_c2p_cells(axb_ctx *ctx, const axb_cells *cells, const axb_params *p,
                          const axb_eos *eos, const axb_mlp *mlp, void *stream) {
  if (!ctx || !cells || !p || !eos || cells->n < 0)
    return AXB_ERR_ARG;
  if (!cells->dens || !cells->tau || !cells->DYe)
    return AXB_ERR_ARG;
  for (int q = 0; q < 3; ++q)
    if (!cells->mom[q] || !cells->dB[q])
      return AXB_ERR_ARG;
  for (int q = 0; q < 6; ++q)
    if (!cells->g[q])
      return AXB_ERR_ARG;
  if (cells->seed_rho && (!cells->seed_eps || !cells->seed_Ye || !cells->seed_vel[0] ||
                          !cells->seed_vel[1] || !cells->seed_vel[2]))
    return AXB_ERR_ARG;
  auto ok_solver = [](int s) {
    return s == AXB_C2P_NOBLE || s == AXB_C2P_PALENZUELA || s == AXB_C2P_ENTROPY;
  };
  if (!ok_solver(p->c2p_prime) || !(ok_solver(p->c2p_second) || p->c2p_second == AXB_C2P_NONE))
    return AXB_ERR_UNSUPPORTED;
  const bool entropy = p->use_entropy_fix || p->c2p_prime == AXB_C2P_ENTROPY ||
                       p->c2p_second == AXB_C2P_ENTROPY;
  if (entropy && eos->kind != 0)
    return AXB_ERR_UNSUPPORTED; // p(rho, kappa) is not defined for a table
  if (entropy && !cells->DEnt)
    return AXB_ERR_ARG; // the entropy scheme reads the conserved entropy
  if (!(p->c2p_tol > 0) || p->max_iter < 1)
    return AXB_ERR_ARG;
  C2PCellsArgs a;
  a.c = *cells;
  a.cp = make_c2p_params(*p);
  a.c2p_prime = p->c2p_prime;
  a.c2p_second = p->c2p_second;
  a.use_entropy_fix = p->use_entropy_fix;
  a.status = ctx->status;
  a.use_mlp = mlp != nullptr;
  a.bracket = 0.0;
  if (mlp) {
    if (!cells->guess)
      return AXB_ERR_ARG;
    a.mlp = mlp_device_view(mlp);
    a.bracket = a.mlp.bracket;
    if (eos->kind == 1 && mlp_nf(mlp) != 9)
      return AXB_ERR_ARG; // the tabulated guess takes Ye as a ninth input
  }
  // uniform atmosphere as for a box inside r_atmo (host_atmosphere)
  C2PBoxArgs hb{};
  hb.thermal_eos_atmo = p->thermal_eos_atmo;
  hb.use_press_atmo = p->use_press_atmo;
  hb.rho_abs_min = p->rho_abs_min;
  hb.p_atmo = p->p_atmo;
  hb.t_atmo = p->t_atmo;
  hb.Ye_atmo = p->Ye_atmo;
  hb.atmo_tol = p->atmo_tol;
  hb.poly = eos->poly;
  if (eos->kind == 0) {
    a.gamma_noble = eos->ideal.gamma;
    a.gfac_over_gamma = (a.gamma_noble - 1.0) / a.gamma_noble;
    a.Zmin = eos->ideal.rgrho.min;
    a.atmo = host_atmosphere(hb, eos->ideal);
  } else if (eos->kind == 1) {
    if (p->thermal_eos_atmo && p->use_press_atmo)
      return AXB_ERR_UNSUPPORTED;
    a.gamma_noble = a.gfac_over_gamma = std::numeric_limits<double>::quiet_NaN();
    a.Zmin = eos->tab_h.rgrho.min;
    a.atmo = host_atmosphere(hb, eos->tab_h);
  } else {
    return AXB_ERR_UNSUPPORTED;
  }
  if (cells->n == 0)
    return AXB_OK;
  const long long blocks = (cells->n + 127) / 128;
  if (blocks > 0x7fffffffLL)
    return AXB_ERR_TOO_LARGE;
  cudaStream_t s = (cudaStream_t)stream;
  if (mlp) {
    axb_mark(ctx, AXB_R_MLP, s, true);
    const int rc = launch_mlp_guess(*cells, mlp, reinterpret_cast<float2 *>(cells->guess),
                                   ctx->status, s);
    axb_mark(ctx, AXB_R_MLP, s, false);
    if (rc)
      return rc;
  }
  axb_mark(ctx, AXB_R_C2P_CELLS, s, true);
  if (eos->kind == 1)
    k_c2p_cells_tab<<<(unsigned)blocks, 128, 0, s>>>(a, tab_for_launch(*eos, a.status));
  else if (a.c2p_prime == AXB_C2P_NOBLE && !a.cp.use_zprim && cells->n < CELLS_FULL)
    k_c2p_cells_noble<4><<<(unsigned)blocks, 128, 0, s>>>(a, eos->ideal);
  else if (a.c2p_prime == AXB_C2P_NOBLE && !a.cp.use_zprim)
    k_c2p_cells_noble<8><<<(unsigned)blocks, 128, 0, s>>>(a, eos->ideal);
  else
    k_c2p_cells<<<(unsigned)blocks, 128, 0, s>>>(a, eos->ideal);
  axb_mark(ctx, AXB_R_C2P_CELLS, s, false);
  return cudaGetLastError() == cudaSuccess ? AXB_OK : AXB_ERR_CUDA;
}

