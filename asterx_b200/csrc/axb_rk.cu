// Runge-Kutta stage update of the evolved variables and the periodic ghost
// fill of one box (the single-box form of the driver's SYNC).
#include <algorithm>
#include <cstring>
#include <vector>

#include "axb_batch.cuh"
#include "axb_internal.hxx"

using namespace axb;

namespace {

constexpr int NEVOLVED = 11;
// evolved grid functions and their centring (1 = cell-centred along x,y,z)
const int kEvolved[NEVOLVED] = {AXB_GF_dens, AXB_GF_momx, AXB_GF_momy, AXB_GF_momz,
                                AXB_GF_tau,  AXB_GF_DYe,  AXB_GF_DEnt, AXB_GF_Avec_x,
                                AXB_GF_Avec_y, AXB_GF_Avec_z, AXB_GF_Psi};
const int kEvolvedRhs[NEVOLVED] = {
    AXB_GF_densrhs, AXB_GF_momxrhs, AXB_GF_momyrhs, AXB_GF_momzrhs,
    AXB_GF_taurhs,  AXB_GF_DYe_rhs, AXB_GF_DEntrhs, AXB_GF_Avec_x_rhs,
    AXB_GF_Avec_y_rhs, AXB_GF_Avec_z_rhs, AXB_GF_Psi_rhs};
const int kCent[NEVOLVED][3] = {{1, 1, 1}, {1, 1, 1}, {1, 1, 1}, {1, 1, 1},
                                {1, 1, 1}, {1, 1, 1}, {1, 1, 1}, {1, 0, 0},
                                {0, 1, 0}, {0, 0, 1}, {0, 0, 0}};

struct StageArgs {
  BoxDev b;
  double *out[NEVOLVED];
  const double *un[NEVOLVED], *uk[NEVOLVED], *rhs[NEVOLVED];
  int cent[NEVOLVED][3];
  double alpha, beta, gdt;
};

// U_out = alpha U_n + beta U_k + (gamma dt) RHS on the interior of each
// field's centring (cells for hydro, edges for A, vertices for Psi).
AXB_D void rk_stage_body(const StageArgs &a, double alpha, double beta, double gdt,
                         const uint3 bid) {
  const BoxDev &b = a.b;
  int i, j;
  const int k = b.ng + bid.z;
  if (!b.row_ij(b.ng, b.n[0] + 1, b.ng, b.n[1] + 1, bid, i, j))
    return;
  const long long I = b.at(i, j, k);
  const int ijk[3] = {i, j, k};
#pragma unroll
  for (int v = 0; v < NEVOLVED; ++v) {
    bool in = true;
#pragma unroll
    for (int d = 0; d < 3; ++d)
      in &= ijk[d] < b.ng + b.n[d] + (a.cent[v][d] ? 0 : 1);
    // explicit rounding order, the same as the stage update fused into the
    // z flux pass and the CT kernel (stage_combine)
    if (in)
      a.out[v][I] = fma(gdt, a.rhs[v][I], fma(beta, a.uk[v][I], alpha * a.un[v][I]));
  }
}
__global__ void __launch_bounds__(128)
    k_rk_stage(const StageArgs a) {
  rk_stage_body(a, a.alpha, a.beta, a.gdt, blockIdx);
}

// The fields of a ghost fill, those of one centring together: group q holds
// f[first[q] .. first[q + 1]).  Eight centrings at most; NF bounds the fields.
template <int NF> struct SyncArgsN {
  BoxDev b;
  double *f[NF];
  int first[9];
  int cent[8][3];
  int groups;
  int small; // ghost points fit 32 bits
};
using SyncArgs = SyncArgsN<AXB_NUM_GF>;
using SyncArgsBatch = SyncArgsN<16>; // a substep's fields (11 or up to 15)

// the periodic image of i; a ghost layer is no wider than the box (n >= ng),
// and a vertex-centred direction has one point more
AXB_D int wrap(int i, int ng, int n) {
  int r = i - ng;
  if (r < 0)
    r += n;
  else if (r >= n)
    r -= n;
  return ng + (r < n ? r : r - n);
}

// Periodic ghost fill: every point outside the interior of its centring
// takes the value of its periodic image inside the interior.  One thread per
// ghost point, enumerated slab below, slab above, then the ghost rows and
// row ends of the middle planes, so no thread idles on interior points.
// Ghost points are counted in 32 bits where they fit (Int = unsigned): the
// enumeration is four divisions per point, and 64-bit ones took most of the
// kernel's time.
template <class Int> struct Shell {
  Int plane, A, AB, Cm, G;
  int N[3], hi[3], ng;
  AXB_HD Shell(const BoxDev &b, const int c[3]) {
    ng = b.ng;
    for (int d = 0; d < 3; ++d) {
      N[d] = b.n[d] + 2 * ng + (c[d] ? 0 : 1);
      hi[d] = ng + b.n[d] + (c[d] ? 0 : 1);
    }
    plane = Int(N[0]) * Int(N[1]);
    A = Int(ng) * plane;
    AB = A + Int(N[2] - hi[2]) * plane;
    Cm = Int(ng + N[1] - hi[1]) * Int(N[0]) + Int(hi[1] - ng) * Int(ng + N[0] - hi[0]);
    G = AB + Int(hi[2] - ng) * Cm;
  }
  AXB_HD void point(Int g, int &i, int &j, int &k) const {
    if (g < AB) {
      const Int q = g < A ? g : g - A;
      const Int z = q / plane, r = q - z * plane;
      k = (g < A ? 0 : hi[2]) + int(z);
      j = int(r / Int(N[0]));
      i = int(r - Int(j) * Int(N[0]));
      return;
    }
    g -= AB;
    const Int z = g / Cm;
    Int r = g - z * Cm;
    k = ng + int(z);
    const Int lowrows = Int(ng) * Int(N[0]), rows = lowrows + Int(N[1] - hi[1]) * Int(N[0]);
    if (r < rows) {
      j = int(r / Int(N[0]));
      i = int(r - Int(j) * Int(N[0]));
      if (r >= lowrows)
        j += hi[1] - ng;
    } else {
      r -= rows;
      const Int per = Int(ng + N[0] - hi[0]);
      const Int y = r / per;
      const int q = int(r - y * per);
      j = ng + int(y);
      i = q < ng ? q : hi[0] + (q - ng);
    }
  }
};

// One ghost point of every field of a group: its place and its image are found
// once (a launch with a thread per field's point spent its time on them: 256^3,
// two fills 255 -> 218 us with 32-bit divisions -> 205 us in groups; a level
// of 64 boxes 718 -> 618 -> 304 us, where a tile's block of arguments cost
// more than its 128 points).
template <class Int, class Args>
AXB_D void sync_shell_point(const Args &a, const int group, const long long g) {
  const BoxDev &b = a.b;
  const Shell<Int> sh(b, a.cent[group]);
  if (g >= (long long)sh.G)
    return;
  int i, j, k;
  sh.point(Int(g), i, j, k);
  const int ng = b.ng;
  const int is = (i >= ng && i < sh.hi[0]) ? i : wrap(i, ng, b.n[0]);
  const int js = (j >= ng && j < sh.hi[1]) ? j : wrap(j, ng, b.n[1]);
  const int ks = (k >= ng && k < sh.hi[2]) ? k : wrap(k, ng, b.n[2]);
  const long long to = b.at(i, j, k), from = b.at(is, js, ks);
  const int last = a.first[group + 1];
  for (int q = a.first[group]; q < last; q += 4) {
    double v[4]; // four loads in flight
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (q + u < last)
        v[u] = a.f[q + u][from];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (q + u < last)
        a.f[q + u][to] = v[u];
  }
}
template <class Args> AXB_D void sync_shell_body(const Args &a, const uint3 bid) {
  const long long g = (long long)bid.x * blockDim.x + threadIdx.x;
  if (a.small)
    sync_shell_point<unsigned>(a, bid.z, g);
  else
    sync_shell_point<long long>(a, bid.z, g);
}
// whether a box's points can be counted in 32 bits
bool sync_small(const BoxDev &b) {
  double pts = 1;
  for (int d = 0; d < 3; ++d)
    pts *= b.n[d] + 2.0 * b.ng + 1;
  return pts < 2147483648.0;
}

__global__ void __launch_bounds__(128) k_sync_shell(const SyncArgs a) {
  sync_shell_body(a, blockIdx);
}

int centring_of(int gf, int c[3]) {
  c[0] = c[1] = c[2] = 1; // cell
  switch (gf) {
  case AXB_GF_Avec_x: case AXB_GF_Avec_x_rhs: c[1] = c[2] = 0; break;
  case AXB_GF_Avec_y: case AXB_GF_Avec_y_rhs: c[0] = c[2] = 0; break;
  case AXB_GF_Avec_z: case AXB_GF_Avec_z_rhs: c[0] = c[1] = 0; break;
  case AXB_GF_dBx_stag: case AXB_GF_fxBy: case AXB_GF_fxBz:
  case AXB_GF_vtilde_y_xface: case AXB_GF_vtilde_z_xface:
  case AXB_GF_amax_xface: case AXB_GF_amin_xface: c[0] = 0; break;
  case AXB_GF_dBy_stag: case AXB_GF_fyBx: case AXB_GF_fyBz:
  case AXB_GF_vtilde_z_yface: case AXB_GF_vtilde_x_yface:
  case AXB_GF_amax_yface: case AXB_GF_amin_yface: c[1] = 0; break;
  case AXB_GF_dBz_stag: case AXB_GF_fzBx: case AXB_GF_fzBy:
  case AXB_GF_vtilde_x_zface: case AXB_GF_vtilde_y_zface:
  case AXB_GF_amax_zface: case AXB_GF_amin_zface: c[2] = 0; break;
  default:
    if ((gf >= AXB_GF_gxx && gf <= AXB_GF_kzz) || gf == AXB_GF_Psi ||
        gf == AXB_GF_Psi_rhs || (gf >= AXB_GF_Fx && gf <= AXB_GF_G))
      c[0] = c[1] = c[2] = 0;
  }
  return 0;
}

// sorts the fields ids[0..n) of `f` into groups of one centring; false when
// one is missing
template <class Args>
bool sync_groups(Args &a, const axb_fields *f, const int *ids, int n) {
  a.groups = 0;
  int at = 0;
  for (int code = 0; code < 8; ++code) {
    const int before = at;
    for (int q = 0; q < n; ++q) {
      int c[3];
      centring_of(ids[q], c);
      if (c[0] + 2 * c[1] + 4 * c[2] != code)
        continue;
      if (!(a.f[at++] = f->gf[ids[q]]))
        return false;
      for (int d = 0; d < 3; ++d)
        a.cent[a.groups][d] = c[d];
    }
    if (at > before)
      a.first[a.groups++] = before;
  }
  a.first[a.groups] = at;
  return true;
}

} // namespace

// One Runge-Kutta stage of the 11 evolved variables (dens, mom, tau, DYe,
// DEnt, Avec, Psi) on the interior:
//   out = alpha * U_n + beta * U_k + gamma * dt * RHS
// (the stage combine of CarpetX's ODESolvers, which the reference's
// scheduled routines rely on; SSP-RK3 in Shu-Osher form uses
// (alpha, beta, gamma) = (0,1,1), (3/4,1/4,1/4), (1/3,2/3,2/3)).
// `out`, `un` and `uk` may alias; the RHS is read from `rhs`.
AXB_API int axb_rk_stage(axb_ctx *c, const axb_box *box, const axb_fields *out,
                         const axb_fields *un, const axb_fields *uk,
                         const axb_fields *rhs, double alpha, double beta,
                         double gamma, double dt, void *stream) {
  if (!c || !box || !out || !un || !uk || !rhs)
    return AXB_ERR_ARG;
  StageArgs a;
  a.b = make_box(*box);
  for (int v = 0; v < NEVOLVED; ++v) {
    a.out[v] = out->gf[kEvolved[v]];
    a.un[v] = un->gf[kEvolved[v]];
    a.uk[v] = uk->gf[kEvolved[v]];
    a.rhs[v] = rhs->gf[kEvolvedRhs[v]];
    if (!a.out[v] || !a.un[v] || !a.uk[v] || !a.rhs[v])
      return AXB_ERR_ARG;
    for (int d = 0; d < 3; ++d)
      a.cent[v][d] = kCent[v][d];
  }
  a.alpha = alpha;
  a.beta = beta;
  a.gdt = gamma * dt;
  const int T = 128;
  const dim3 grid((box->n[0] + 1 + T - 1) / T, box->n[1] + 1, box->n[2] + 1);
  axb_mark(c, AXB_R_STAGE, (cudaStream_t)stream, true);
  k_rk_stage<<<grid, T, 0, (cudaStream_t)stream>>>(a);
  axb_mark(c, AXB_R_STAGE, (cudaStream_t)stream, false);
  return cudaGetLastError() == cudaSuccess ? AXB_OK : AXB_ERR_CUDA;
}

// Periodic ghost fill of the grid functions listed in `ids` (each with its
// own centring) on one box: the single-box stand-in for the driver's SYNC
// with periodic outer boundaries.
AXB_API int axb_sync_periodic(axb_ctx *c, const axb_box *box,
                              const axb_fields *f, const int *ids, int nids,
                              void *stream) {
  if (!c || !box || !f || !ids || nids < 1 || nids > AXB_NUM_GF)
    return AXB_ERR_ARG;
  if (box->ng < 1)
    return AXB_ERR_GHOSTS;
  for (int d = 0; d < 3; ++d)
    if (box->n[d] < box->ng)
      return AXB_ERR_ARG; // a ghost layer must fit inside one period
  SyncArgs a;
  a.b = make_box(*box);
  a.small = sync_small(a.b);
  for (int q = 0; q < nids; ++q)
    if (ids[q] < 0 || ids[q] >= AXB_NUM_GF)
      return AXB_ERR_ARG;
  if (!sync_groups(a, f, ids, nids))
    return AXB_ERR_ARG;
  // one thread per ghost point of the largest centring among the fields
  long long gmax = 0;
  for (int q = 0; q < a.groups; ++q)
    gmax = std::max(gmax, Shell<long long>(a.b, a.cent[q]).G);
  const dim3 grid(unsigned((gmax + 127) / 128), 1, a.groups);
  axb_mark(c, AXB_R_SYNC, (cudaStream_t)stream, true);
  k_sync_shell<<<grid, 128, 0, (cudaStream_t)stream>>>(a);
  axb_mark(c, AXB_R_SYNC, (cudaStream_t)stream, false);
  return cudaGetLastError() == cudaSuccess ? AXB_OK : AXB_ERR_CUDA;
}

// ---------------------------------------------------------------------------
// batched forms (see axb_batch.cuh)
// ---------------------------------------------------------------------------
namespace {

__global__ void __launch_bounds__(128)
    k_sync_batch(const SyncArgsBatch *args, const TileTable t, unsigned long long *ctr) {
  batch_loop(args, t, ctr,
             [&](const SyncArgsBatch &a, const uint3 bid) { sync_shell_body(a, bid); });
}

template <class T> int upload(const std::vector<T> &h, void **out) {
  *out = nullptr;
  if (h.empty())
    return AXB_OK;
  if (cudaMalloc(out, h.size() * sizeof(T)) != cudaSuccess)
    return AXB_ERR_CUDA;
  if (cudaMemcpy(*out, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice) !=
      cudaSuccess)
    return AXB_ERR_CUDA;
  return AXB_OK;
}

} // namespace

namespace axb {

// Per-box ghost-fill argument blocks of a batch, in device memory.
int batch_sync_setup(int nbox, const axb_box *boxes, const axb_fields *f, int recvar,
                     void **sync_evolved, void **sync_prims) {
  // the 12 cell-centred primitives, plus the reconstructed zvec or svec
  // when the fluxes reconstruct one of those instead of the velocity
  int prims[15] = {AXB_GF_rho,   AXB_GF_velx, AXB_GF_vely,        AXB_GF_velz,
                   AXB_GF_eps,   AXB_GF_press, AXB_GF_temperature, AXB_GF_Ye,
                   AXB_GF_entropy, AXB_GF_Bvecx, AXB_GF_Bvecy,     AXB_GF_Bvecz};
  int nprims = 12;
  if (recvar == AXB_RECVAR_Z || recvar == AXB_RECVAR_S) {
    const int first = recvar == AXB_RECVAR_Z ? AXB_GF_zvec_x : AXB_GF_svec_x;
    for (int q = 0; q < 3; ++q)
      prims[nprims++] = first + q;
  }
  std::vector<SyncArgsBatch> se(nbox), sp(nbox);
  for (int b = 0; b < nbox; ++b) {
    const axb_box &box = boxes[b];
    if (box.ng < 1)
      return AXB_ERR_GHOSTS;
    for (int d = 0; d < 3; ++d)
      if (box.n[d] < box.ng)
        return AXB_ERR_ARG;
    for (int pass = 0; pass < 2; ++pass) {
      SyncArgsBatch &y = pass ? sp[b] : se[b];
      std::memset(&y, 0, sizeof y);
      y.b = make_box(box);
      y.small = sync_small(y.b);
      if (!sync_groups(y, f + b, pass ? prims : kEvolved, pass ? nprims : NEVOLVED))
        return AXB_ERR_ARG;
    }
  }
  int rc = upload(se, sync_evolved);
  if (!rc)
    rc = upload(sp, sync_prims);
  return rc;
}

// batched grid of a ghost fill over the ghost points of the largest centring;
// set 0: the evolved variables (cells, three edges, vertices); else the
// primitives (cells)
uint3 sync_grid(const axb_box &b, int set) {
  const BoxDev bd = make_box(b);
  const int cents[5][3] = {{1, 1, 1}, {1, 0, 0}, {0, 1, 0}, {0, 0, 1}, {0, 0, 0}};
  const int groups = set == 0 ? 5 : 1;
  long long g = 0;
  for (int q = 0; q < groups; ++q)
    g = std::max(g, Shell<long long>(bd, cents[q]).G);
  return make_uint3(unsigned((g + 127) / 128), 1, groups);
}

int launch_sync_batch(const void *args, const TileTable &t, unsigned long long *ctr,
                      int nblocks, cudaStream_t s) {
  if (t.total == 0)
    return AXB_OK;
  k_sync_batch<<<nblocks, 128, 0, s>>>(static_cast<const SyncArgsBatch *>(args), t, ctr);
  return cudaGetLastError() == cudaSuccess ? AXB_OK : AXB_ERR_CUDA;
}

} // namespace axb

namespace axb {
// The centring of a grid function (1 = cell-centred along x, y, z), for the
// other translation units of the library.
int gf_centring(int gf, int c[3]) { return centring_of(gf, c); }
} // namespace axb
