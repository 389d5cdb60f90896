// RHS kernels (see axb_rhs.cuh for the overview).
#pragma once

#include "axb_internal.hxx"
#include "axb_rhs.cuh"

namespace axb {

template <int N>
AXB_D void load_pencil(const double *__restrict__ f, long long I, long long s,
                       double (&q)[N]) {
#pragma unroll
  for (int m = 0; m < N; ++m)
    q[m] = __ldg(f + I + (m - N / 2) * s);
}

AXB_D void prefetch_l2(const double *p) {
  asm volatile("prefetch.global.L2 [%0];" ::"l"(p));
}

AXB_D double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1)
    v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// ---------------------------------------------------------------------------
// Shared pieces of the flux passes.
// ---------------------------------------------------------------------------

// Reconstruct the NREC variables of the cell at I (stride sd along DIR);
// `win(v, m)` is variable v of the cell m - 2 cells on.  Only PPM reads the
// pressure (its own stencil when the temperature is reconstructed) and, with
// zone flattening, the velocity along the pencil.
template <int DIR, int RECON, class Win>
AXB_D void recon_cell_all(const RhsArgs &a, const Win &win, long long I, long long sd,
                          double (&lo)[NREC], double (&up)[NREC]) {
  double pr[5] = {}, vd[5] = {};
  if constexpr (RECON == AXB_RECON_PPM) {
    if (a.rec_temp) {
      load_pencil<5>(a.press, I, sd, pr);
    } else {
#pragma unroll
      for (int m = 0; m < 5; ++m)
        pr[m] = win(R_PRESS, m);
    }
    if (a.rp.ppm_zone_flattening)
      load_pencil<5>(a.vel[DIR], I, sd, vd);
  }
#pragma unroll
  for (int v = 0; v < NREC; ++v) {
    double q[5];
#pragma unroll
    for (int m = 0; m < 5; ++m)
      q[m] = win(v, m);
    const CellLoUp r = recon_cell<RECON>(q, pr, vd, v == R_RHO, a.rp);
    lo[v] = r.lo;
    up[v] = r.up;
  }
}

// The face between the cells at I - sd and I, given the left state L (upper
// values of the left cell) and the right state R (lower values of the right
// cell): low-order redo of a side with a non-positive rho, entropy, Ye or
// thermodynamic variable (fluxes.cxx:263-343), face metric, both states'
// conserved variables, fluxes and fast speeds, and the Riemann flux
// (HLLE or LxF, fluxes.cxx:162-200).  Stores the two transverse B fluxes
// when asked.
template <int DIR, bool UCT, class EOS>
AXB_D void face_fluxes(const RhsArgs &a, const EOS &eos,
                       const double *const (&fld)[NREC], long long I, long long sd,
                       double (&L)[NREC], double (&R)[NREC], double (&F)[10],
                       double &smax, bool &bad) {
  constexpr int D1 = (DIR + 1) % 3, D2 = (DIR + 2) % 3;
  const bool lo0 = (L[R_RHO] <= 0.0) || (L[R_ENT] <= 0.0) ||
                   (L[R_YE] <= 0.0) || (L[R_PRESS] <= 0.0);
  const bool lo1 = (R[R_RHO] <= 0.0) || (R[R_ENT] <= 0.0) ||
                   (R[R_YE] <= 0.0) || (R[R_PRESS] <= 0.0);
  if (lo0 || lo1) {
    for (int v = 0; v < NREC; ++v) {
      double q[5];
      if (lo0) {
        load_pencil<5>(fld[v], I - sd, sd, q);
        L[v] = recon_cell_lo(a.recon_lo, q).up;
      }
      if (lo1) {
        load_pencil<5>(fld[v], I, sd, q);
        R[v] = recon_cell_lo(a.recon_lo, q).lo;
      }
    }
  }
  const FaceMetric m = face_metric<DIR>(a, I);
  const double Bdir = __ldg(a.dBstag[DIR] + I) * m.isqrtg;
  SideOut sL, sR;
  side_physics<DIR, UCT>(m, L, Bdir, eos, a.rec_temp, a.recvar, sL);
  side_physics<DIR, UCT>(m, R, Bdir, eos, a.rec_temp, a.recvar, sR);
  const double cmax = fmax(0.0, fmax(fmax(sL.lam_p, sL.lam_m), fmax(sR.lam_p, sR.lam_m)));
  const double cmin = fmin(0.0, fmin(fmin(sL.lam_p, sL.lam_m), fmin(sR.lam_p, sR.lam_m)));
  smax = fmax(smax, fmax(cmax, -cmin));
  if (a.flux_type == AXB_FLUX_HLLE) {
    const double icpm = 1 / (cmax - cmin);
#pragma unroll
    for (int v = 0; v < 10; ++v)
      F[v] = hlle_flux(cmax, cmin, icpm, sL.U[v], sR.U[v], sL.F[v], sR.F[v]);
  } else {
    const double ch = fmax(cmax, -cmin);
#pragma unroll
    for (int v = 0; v < 10; ++v)
      F[v] = laxf_flux(ch, sL.U[v], sR.U[v], sL.F[v], sR.F[v]);
  }
#pragma unroll
  for (int v = 0; v < 10; ++v)
    bad |= isnan(F[v]);
  if (a.write_bflux) {
    // bflux slots per direction hold the two transverse components in
    // ascending order: x (y, z), y (x, z), z (x, y)
    constexpr int BLO = D1 < D2 ? D1 : D2, BHI = D1 < D2 ? D2 : D1;
    a.bflux[2 * DIR + 0][I] = F[7 + BLO];
    a.bflux[2 * DIR + 1][I] = F[7 + BHI];
  }
  if constexpr (UCT) {
    // upwind-CT face data (fluxes.cxx:776-794): the bounding speeds and the
    // transverse vtilde averaged with them
    const double amax = cmax, amin = -cmin;
    a.uct[4 * DIR + 0][I] = (amax * sL.vt1 + amin * sR.vt1) / (amax + amin);
    a.uct[4 * DIR + 1][I] = (amax * sL.vt2 + amin * sR.vt2) / (amax + amin);
    a.uct[4 * DIR + 2][I] = amax;
    a.uct[4 * DIR + 3][I] = amin;
  }
}

// Fold F(face c+1) - F(face c) into the partial divergence of cell c (at I),
// in the reference's summation order (rhs.cxx:188-207): x writes, y adds,
// z adds and forms the RHS.  Returns true when the z pass formed a
// non-finite hydro RHS (the reference asserts there, rhs.cxx:199-206).
template <int DIR>
AXB_D bool fold_divergence(const RhsArgs &a, long long I, double idxd,
                           const double (&Fhi)[NHYDRO], const double (&Flo)[NHYDRO]) {
  bool bad = false;
  // every load ahead of the first store: the arrays may not be told apart, and
  // one at a time each variable waited for memory on its own
  double r[NHYDRO], un[NHYDRO], uk[NHYDRO];
#pragma unroll
  for (int v = 0; v < NHYDRO; ++v) {
    const double dF = Fhi[v] - Flo[v];
    if (DIR == 0) {
      r[v] = idxd * dF;
    } else if (DIR == 1) {
      r[v] = a.acc[v][I] + idxd * dF;
    } else {
      r[v] = a.rhs[v][I] + (-(a.acc[v][I] + idxd * dF));
      bad |= !isfinite(r[v]);
    }
  }
  if (DIR == 2 && a.fuse_stage) {
#pragma unroll
    for (int v = 0; v < NHYDRO; ++v) {
      un[v] = a.st_un[v][I];
      uk[v] = a.st_uk[v][I];
    }
#pragma unroll
    for (int v = 0; v < NHYDRO; ++v)
      a.st_uk[v][I] = stage_combine(a.st_alpha, un[v], a.st_beta, uk[v], a.st_gdt, r[v]);
  } else {
#pragma unroll
    for (int v = 0; v < NHYDRO; ++v)
      (DIR == 2 ? a.rhs : a.acc)[v][I] = r[v];
  }
  return bad;
}

AXB_D void flux_status(const RhsArgs &a, double smax, bool bad, bool bad_rhs = false) {
  // characteristic-speed maximum: warp shuffle, then one atomic per warp that
  // raises it (all of them on one address would serialise; a stale read only
  // costs an atomic too many)
  smax = warp_max(smax);
  const bool lead = threadIdx.x % 32 == 0;
  if (lead && smax > __longlong_as_double(*(volatile long long *)&a.status->max_speed_bits))
    atomic_max_nonneg(&a.status->max_speed_bits, smax);
  const bool any_bad = __any_sync(0xffffffffu, bad);
  const bool any_rhs = __any_sync(0xffffffffu, bad_rhs);
  if (lead && (any_bad || any_rhs))
    atomicOr(&a.status->error_word,
             (any_bad ? AXB_EW_NAN_FLUX : 0u) | (any_rhs ? AXB_EW_NAN_RHS : 0u));
}

#ifndef AXB_FLUX_X_MINB
#define AXB_FLUX_X_MINB 4 // resident CTAs per SM the register budget must allow
#endif
constexpr int FLUX_T = 128;   // threads of a y/z pass block
constexpr int FLUX_MINB = 3;  // its resident CTAs per SM (shared memory, registers)
constexpr double FLUX_START = 1.2; // what starting a segment costs, in steps
// its dynamic shared memory: ring, upper values, fluxes
constexpr int FLUX_SMEM = (5 * NREC + NREC + NHYDRO) * FLUX_T * int(sizeof(double));

// asynchronous copy of one double into shared memory, and the wait for all of
// this thread's copies
AXB_D void cp_async8(double *smem, const double *g) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                   unsigned(__cvta_generic_to_shared(smem))),
               "l"(g)
               : "memory");
}
AXB_D void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
AXB_D void cp_async_wait() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// ---------------------------------------------------------------------------
// k_flux_pass (y and z): one thread marches one pencil segment along DIR.
// Per step it reconstructs one cell (both interface values, ReconX per-cell
// formulas), forms the face between the previous cell and this one, and
// folds F(face) - F(face-1) into the partial divergence of the previous cell.
// Threads of a warp are adjacent along x, so every load is a coalesced
// 256-byte row.
//
// What bounds it is latency: 16 warps per SM re-reading their stencils through
// the L1 that 147 KB of shared memory left them hit it 18 % of the time and
// waited 5 (y) to 7 (z) cycles per issued instruction for L2, with the FP64
// pipe at 36 / 31 %.  So each thread keeps its five stencil rows in shared
// memory, a ring of five slots per variable: the next cell's last row is
// copied asynchronously into the slot of the row just used while the face is
// computed, and a step reads 9 doubles from memory for its stencils instead of
// 45.  With the carried upper values and fluxes that is 488 bytes a thread;
// three CTAs per SM fit, whose 168 registers hold both face states: without
// spills for the ideal gas on one box, with 0.1 KB (stores; 0.14 KB loads) in a
// level's kernels, whose draw of tiles stays live, and 0.2 (0.3) KB on a table
// (four CTAs at 128 registers spilled, and kept the left state in shared memory).  256^3 WENO-Z: y 3.55 -> 2.87 ms, z 3.80 -> 3.09 ms (beside the
// sources; with fold_divergence's loads ahead of its stores, and the z pass's
// in two batches from U prefetched, 2.52 and 2.49 ms).  Not kept: a four-slot
// ring with the last row loaded directly at four CTAs (3.05 / 3.31 ms) or three
// (2.95 / 3.09); seven 64-thread CTAs at 128 registers (3.39 / 3.66).
// Transverse range: cells [ng-1, ng+n] (one ghost layer each side, needed
// by the edge electric field); faces along DIR: [ng, ng+n].
// ---------------------------------------------------------------------------
template <int DIR, int RECON, class EOS, bool UCT = false>
AXB_D void flux_pass_body(const RhsArgs &a, const EOS &eos, const int &seglen, const uint3 bid) {
  static_assert(DIR != 0, "the x pass is k_flux_x");
  constexpr int D1 = (DIR + 1) % 3, D2 = (DIR + 2) % 3;
  constexpr int T0 = 0;
  constexpr int T1 = (DIR == 2) ? 1 : 2;
  const BoxDev &b = a.b;
  const int ng = b.ng;
  constexpr int te = UCT ? 3 : 1; // transverse ghost layers covered
  // the block's threads walk the transverse plane [ng-te, ng+n+te-1]^2 row
  // after row
  const int w0 = b.n[T0] + 2 * te;
  const int flat = bid.x * FLUX_T + threadIdx.x;
  const int t0 = ng - te + flat % w0, t1 = ng - te + flat / w0;
  const bool active = flat < w0 * (b.n[T1] + 2 * te);
  double smax = 0.0;
  bool bad = false, bad_rhs = false;
  if (active) {
    const bool trans_int = (t0 >= ng) && (t0 < ng + b.n[T0]) && (t1 >= ng) &&
                           (t1 < ng + b.n[T1]);
    const int f0 = ng + bid.z * seglen;
    const int flast = min(f0 + seglen, ng + b.n[DIR]);
    const long long sd = b.stride(DIR);
    int ijk[3];
    ijk[T0] = t0;
    ijk[T1] = t1;
    ijk[DIR] = f0 - 1;
    long long I = b.at(ijk[0], ijk[1], ijk[2]);
    const double *const fld[NREC] = {a.rho,     a.entropy, a.Ye,       a.thermo,
                                     a.recv[0], a.recv[1], a.recv[2], a.Bvec[D1],
                                     a.Bvec[D2]};
    const double idxd = b.idx[DIR];
    extern __shared__ double s_dyn[];
    // the thread's slots: 5 rows of the stencil (a ring), the upper values of
    // the previous cell, the fluxes of the previous face
    double *const ring = s_dyn + threadIdx.x;
    double *const s_up = ring + 5 * NREC * FLUX_T;
    double *const s_fprev = s_up + NREC * FLUX_T;
    auto fetch = [&](int slot, long long J) { // a stencil row into a ring slot
#pragma unroll
      for (int v = 0; v < NREC; ++v)
        cp_async8(ring + (slot + v) * FLUX_T, fld[v] + J);
    };
    int o[5]; // ring slots of the rows c-2 .. c+2
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      o[m] = m * NREC;
      fetch(o[m], I + (m - 2) * sd);
    }
    cp_async_commit();
#pragma unroll 1
    for (int c = f0 - 1; c <= flast; ++c, I += sd) {
      // L2 prefetch of the rows the march first touches a step ahead: the
      // face metric's two vertex rows, the face's staggered B and the partial
      // divergences (and RHS) it will accumulate into
      if (c + 1 <= flast) {
        const long long J = I + sd;
        const long long so = (D1 == 0) ? b.stride(D2) : b.stride(D1);
        prefetch_l2(a.alp + J);
        prefetch_l2(a.alp + J + so);
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          prefetch_l2(a.beta[q] + J);
          prefetch_l2(a.beta[q] + J + so);
        }
#pragma unroll
        for (int q = 0; q < 6; ++q) {
          prefetch_l2(a.g[q] + J);
          prefetch_l2(a.g[q] + J + so);
        }
        prefetch_l2(a.dBstag[DIR] + J);
        if (trans_int) {
#pragma unroll
          for (int v = 0; v < NHYDRO; ++v) {
            prefetch_l2(a.acc[v] + I);
            if (DIR == 2) {
              prefetch_l2(a.rhs[v] + I);
              if (a.fuse_stage) {
                prefetch_l2(a.st_un[v] + I);
                prefetch_l2(a.st_uk[v] + I);
              }
            }
          }
        }
      }
      cp_async_wait(); // this thread's own copies: no barrier
      double lo[NREC], up[NREC];
      recon_cell_all<DIR, RECON>(
          a, [&](int v, int m) { return ring[(o[m] + v) * FLUX_T]; }, I, sd, lo, up);
      // the next cell's last row lands in the slot of this cell's first one
      // while the face is computed
      if (c < flast)
        fetch(o[0], I + 3 * sd);
      cp_async_commit();
      const int first = o[0];
#pragma unroll
      for (int m = 0; m < 4; ++m)
        o[m] = o[m + 1];
      o[4] = first;
      if (c >= f0) {
        // face c: left state = upper values of cell c-1, right = lower of c
        double L[NREC], F[10];
#pragma unroll
        for (int v = 0; v < NREC; ++v)
          L[v] = s_up[v * FLUX_T];
        // (stored ahead of the face: the face needs the registers)
#pragma unroll
        for (int v = 0; v < NREC; ++v)
          s_up[v * FLUX_T] = up[v];
        face_fluxes<DIR, UCT>(a, eos, fld, I, sd, L, lo, F, smax, bad);
        if (c > f0 && trans_int) {
          double Fc[NHYDRO], Fp[NHYDRO];
#pragma unroll
          for (int v = 0; v < NHYDRO; ++v) {
            Fc[v] = F[v];
            Fp[v] = s_fprev[v * FLUX_T];
          }
          bad_rhs |= fold_divergence<DIR>(a, I - sd, idxd, Fc, Fp);
        }
#pragma unroll
        for (int v = 0; v < NHYDRO; ++v)
          s_fprev[v * FLUX_T] = F[v];
      } else {
#pragma unroll
        for (int v = 0; v < NREC; ++v)
          s_up[v * FLUX_T] = up[v];
      }
    }
  }
  flux_status(a, smax, bad, bad_rhs);
}
// blocks that cover the transverse plane of a y or z pass once, and the steps of
// a box's pencils in it
inline long long flux_plane_blocks(const BoxDev &b, int dir, int te) {
  const long long plane = (long long)(b.n[0] + 2 * te) * (b.n[dir == 2 ? 1 : 2] + 2 * te);
  return (plane + FLUX_T - 1) / FLUX_T;
}
inline int flux_steps(const BoxDev &b, int dir, int te, int sms) {
  const long long plane = flux_plane_blocks(b, dir, te);
  const int n = b.n[dir];
  return split_steps(n, double(FLUX_MINB) * sms, FLUX_START,
                     [&](int seg) { return plane * ((n + seg - 1) / seg); });
}
template <int DIR, int RECON, class EOS, bool UCT = false>
__global__ void __launch_bounds__(FLUX_T, FLUX_MINB)
    k_flux_pass(const RhsArgs a, const __grid_constant__ EOS eos, const int seglen) {
  flux_pass_body<DIR, RECON, EOS, UCT>(a, eos, seglen, blockIdx);
}

// ---------------------------------------------------------------------------
// k_flux_x: the x pass with the lanes of a warp along x, so that every
// stencil load is a coalesced row segment (a thread marching along x would
// touch 32 rows per load and lose its sectors before coming back to them).
// The rows' cells [ng-1, ng+n] are laid end to end, and a warp takes 32
// consecutive ones, overlapping the next warp's by two: lane l reconstructs
// its cell once, takes the left state of its lower face from lane l - 1 by
// shuffle, computes the face, and takes the flux of the next face from lane
// l + 1 to form the divergence of its cell.  Lanes 1..31 compute faces (but
// that of a row's first cell), lanes 1..30 divergences.  (Rows cut into chunks
// of 30 one by one left the last chunk of each mostly idle: 50 % of the lanes
// at n = 32, 67 % at 64, 80 % at 128, against 88 to 93 % end to end.)
// ---------------------------------------------------------------------------
template <int RECON, class EOS, bool UCT = false>
AXB_D void flux_x_body(const RhsArgs &a, const EOS &eos, const uint3 bid) {
  const BoxDev &b = a.b;
  const int ng = b.ng;
  const int lane = threadIdx.x & 31;
  const long long warp = ((long long)bid.x * blockDim.x + threadIdx.x) >> 5;
  constexpr int te = UCT ? 3 : 1; // transverse ghost layers covered
  const int ny = b.n[1] + 2 * te; // rows j, k in [ng-te, ng+n+te-1]
  const int nz = b.n[2] + 2 * te;
  const int w = b.n[0] + 2; // cells of a row
  double smax = 0.0;
  bool bad = false;
  const long long total = (long long)w * ny * nz;
  const long long g = 30 * warp + lane;
  if (30 * warp < total) { // warp-uniform
    const bool has_cell = g < total;
    int p = 0; // the cell's place in its row
    int row = 0;
    if (total < 0x7fffffffLL) {
      row = int(unsigned(g) / unsigned(w));
      p = int(unsigned(g) - unsigned(row) * unsigned(w));
    } else {
      row = int(g / w);
      p = int(g - (long long)row * w);
    }
    const int j = ng - te + row % ny;
    const int k = ng - te + row / ny;
    const bool trans_int = (j >= ng) && (j < ng + b.n[1]) && (k >= ng) && (k < ng + b.n[2]);
    const double *const fld[NREC] = {a.rho,     a.entropy, a.Ye,      a.thermo, a.recv[0],
                                     a.recv[1], a.recv[2], a.Bvec[1], a.Bvec[2]};
    const double idxd = b.idx[0];
    const long long I = b.at(ng - 1 + p, j, k);
    double lo[NREC], up[NREC];
    if (has_cell) {
      recon_cell_all<0, RECON>(
          a, [&](int v, int m) { return __ldg(fld[v] + I + (m - 2)); }, I, 1, lo, up);
    } else {
#pragma unroll
      for (int v = 0; v < NREC; ++v)
        lo[v] = up[v] = 0.0;
    }
    double L[NREC], R[NREC], F[10];
#pragma unroll
    for (int v = 0; v < NREC; ++v) {
      L[v] = __shfl_up_sync(0xffffffffu, up[v], 1);
      R[v] = lo[v];
    }
    const bool has_face = lane >= 1 && has_cell && p >= 1; // face p of [1, n + 1]
    if (has_face) {
      face_fluxes<0, UCT>(a, eos, fld, I, 1, L, R, F, smax, bad);
    } else {
#pragma unroll
      for (int v = 0; v < 10; ++v)
        F[v] = 0.0;
    }
    double Fhi[NHYDRO], Flo[NHYDRO];
#pragma unroll
    for (int v = 0; v < NHYDRO; ++v) {
      Flo[v] = F[v];
      Fhi[v] = __shfl_down_sync(0xffffffffu, F[v], 1);
    }
    // a cell's divergence needs its two faces
    if (trans_int && has_face && lane <= 30 && p <= b.n[0])
      fold_divergence<0>(a, I, idxd, Fhi, Flo);
  }
  flux_status(a, smax, bad);
}
// blocks of four warps the x pass of a box takes
inline long long flux_x_blocks(const BoxDev &b, int te) {
  const long long cells = (long long)(b.n[0] + 2) * (b.n[1] + 2 * te) * (b.n[2] + 2 * te);
  return ((cells + 29) / 30 + 3) / 4;
}
template <int RECON, class EOS, bool UCT = false>
__global__ void __launch_bounds__(128, AXB_FLUX_X_MINB)
    k_flux_x(const RhsArgs a, const __grid_constant__ EOS eos) {
  flux_x_body<RECON, EOS, UCT>(a, eos, blockIdx);
}

} // namespace axb
