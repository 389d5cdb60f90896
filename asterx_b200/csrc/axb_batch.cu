// Batched RK substep over the boxes of a refinement level.
//
// The reference advances a level box by box: CarpetX launches each scheduled
// routine's loop once per box (AsterX/schedule.ccl:119-228 over the boxes of
// every level), so a level of 512 small boxes costs ~5600 kernel launches per
// substep.  Here every phase of the substep is ONE persistent launch over the
// tiles of all boxes (axb_batch.cuh), the per-box argument blocks live in
// device memory, and the whole substep (11 launches and a memset of the work
// counters; with Palenzuela first one more of each, for the queue of deferred
// cells) is stream-ordered and allocation-free, so a caller can
// capture it in a CUDA graph.  The pencil segments of the y and z flux passes
// follow from the level's size; the autotuner checks them, and the number of
// resident CTAs per SM of the persistent grids, by timing the batch's own boxes.
#include <algorithm>
#include <cstring>
#include <new>
#include <vector>

#include "axb_batch.cuh"
#include "axb_internal.hxx"
#include "axb_rhs.cuh"

using namespace axb;

namespace axb {
// from the kernel translation units
int batch_rhs_setup(axb_ctx *c, int nbox, const axb_box *boxes, const axb_fields *f,
                    const axb_fields *fn, const axb_params *p, const axb_eos *eos, void **out);
int batch_c2p_setup(axb_ctx *c, int nbox, const axb_box *boxes, const axb_fields *f,
                    const axb_params *p, const axb_eos *eos, void **out);
int batch_sync_setup(int nbox, const axb_box *boxes, const axb_fields *f, int recvar,
                     void **sync_evolved, void **sync_prims);
uint3 rhs_misc_grid(int which, const axb_box &b, int seg);
int batch_steps(int dir, const axb_box *boxes, int nbox, int sms);
uint3 flux_grid(int dir, const axb_box &b, int seglen);
uint3 sync_grid(const axb_box &b, int set);
uint3 c2p_grid(int which, const axb_box &b);
int launch_rhs_misc_batch(int which, const void *args, const TileTable &t,
                          unsigned long long *ctr, int seg, const BatchStage &stage, int nblocks,
                          cudaStream_t s);
int launch_flux_batch(int recon, int dir, const RhsArgs *args, const TileTable &t,
                      unsigned long long *ctr, const axb_eos &eos, DevStatus *status,
                      int seglen, const BatchStage &stage, int nblocks, cudaStream_t s);
int launch_sync_batch(const void *args, const TileTable &t, unsigned long long *ctr,
                      int nblocks, cudaStream_t s);
int launch_c2p_batch(int which, const void *args, const TileTable &t,
                     unsigned long long *ctr, const axb_eos &eos, DevStatus *status,
                     int nblocks, cudaStream_t s, unsigned long long *queue = nullptr,
                     int deferred_blocks = 0, bool noble = false);
bool c2p_batch_fast_ok(int nbox, const axb_box *boxes, const axb_params *p);
} // namespace axb

namespace {

enum Phase {
  P_SOURCES = 0,
  P_FLUX_X,
  P_FLUX_Y,
  P_FLUX_Z,
  P_AUX,
  P_CT,
  P_SYNC_E,
  P_BSTAG,
  P_C2P,
  P_SYNC_P,
  NPHASE
};
const int kRegion[NPHASE] = {AXB_R_SOURCES, AXB_R_FLUX_X, AXB_R_FLUX_Y, AXB_R_FLUX_Z,
                             AXB_R_AUX,     AXB_R_CT,     AXB_R_SYNC,
                             AXB_R_BSTAG,   AXB_R_C2P,    AXB_R_SYNC};
// candidate pencil segments of the y / z flux passes
const int kSeg[] = {8, 16, 32, 64};
constexpr int NSEG = 4;
// candidate persistent-grid sizes, in CTAs per SM
const int kCtas[] = {2, 4, 8, 16};
constexpr int NCTAS = 4;

struct DevTable {
  long long *prefix = nullptr;
  uint3 *grid = nullptr;
  TileTable t{};
};

} // namespace

struct axb_batch {
  int nbox = 0;
  int sms = 148;
  int recon = 0, fd_order = 2;
  bool noble = false; // Noble is the first solver
  const axb_eos *eos = nullptr;
  DevStatus *status = nullptr;
  void *rhs_args = nullptr, *c2p_args = nullptr;
  void *sync_e = nullptr, *sync_p = nullptr;
  DevTable tab[NPHASE];
  // y, z tables: the autotuner's candidate segments, then the one chosen by
  // the level's size (split_steps), which stands unless the autotuner finds
  // one of the others faster
  DevTable flux_seg[2][NSEG + 1];
  int steps[2] = {16, 16}; // that segment
  int seg[2] = {NSEG, NSEG}; // index of the table in use
  int src_steps = 16;        // cells of a sources column
  int ctas[NPHASE];           // CTAs per SM of each phase's persistent grid
  unsigned long long *ctr = nullptr; // one work counter per phase
  // deferred-cell queue of the recovery's fast pass (null: full cascade)
  unsigned long long *c2p_queue = nullptr;
  long long zones = 0;
};

namespace {

int make_table(const std::vector<axb_box> &boxes, uint3 (*g)(const axb_box &, int), int arg,
               DevTable &out) {
  const int n = int(boxes.size());
  std::vector<long long> prefix(n + 1, 0);
  std::vector<uint3> grid(n);
  for (int b = 0; b < n; ++b) {
    grid[b] = g(boxes[b], arg);
    prefix[b + 1] = prefix[b] + (long long)grid[b].x * grid[b].y * grid[b].z;
  }
  if (cudaMalloc(&out.prefix, (n + 1) * sizeof(long long)) != cudaSuccess ||
      cudaMalloc(&out.grid, n * sizeof(uint3)) != cudaSuccess)
    return AXB_ERR_CUDA;
  if (cudaMemcpy(out.prefix, prefix.data(), (n + 1) * sizeof(long long),
                 cudaMemcpyHostToDevice) != cudaSuccess ||
      cudaMemcpy(out.grid, grid.data(), n * sizeof(uint3), cudaMemcpyHostToDevice) !=
          cudaSuccess)
    return AXB_ERR_CUDA;
  out.t.prefix = out.prefix;
  out.t.grid = out.grid;
  out.t.nbox = n;
  out.t.total = prefix[n];
  return AXB_OK;
}

void free_table(DevTable &d) {
  cudaFree(d.prefix);
  cudaFree(d.grid);
  d = DevTable{};
}

uint3 g_sources(const axb_box &b, int seg) { return rhs_misc_grid(0, b, seg); }
uint3 g_aux(const axb_box &b, int) { return rhs_misc_grid(2, b, 1); }
uint3 g_ct(const axb_box &b, int) { return rhs_misc_grid(3, b, 1); }
uint3 g_flux(const axb_box &b, int dir_seg) { return flux_grid(dir_seg & 3, b, dir_seg >> 2); }
uint3 g_sync(const axb_box &b, int set) { return sync_grid(b, set); }
uint3 g_c2p(const axb_box &b, int which) { return c2p_grid(which, b); }

// the persistent grid of a phase, and the items its CTAs draw at a time
int nblocks_for(const axb_batch *B, int phase, TileTable &t) {
  const long long cap = (long long)B->ctas[phase] * B->sms;
  t.chunk = t.total >= 16 * cap ? BATCH_CHUNK : 1;
  return int(std::max(1LL, std::min((t.total + t.chunk - 1) / t.chunk, cap)));
}

int segment_of(const axb_batch *B, int d) {
  return B->seg[d] < NSEG ? kSeg[B->seg[d]] : B->steps[d];
}

const TileTable &table_of(const axb_batch *B, int phase) {
  if (phase == P_FLUX_Y)
    return B->flux_seg[0][B->seg[0]].t;
  if (phase == P_FLUX_Z)
    return B->flux_seg[1][B->seg[1]].t;
  return B->tab[phase].t;
}

// one phase; `stage`: the update the z pass and the CT kernel make (or the RHS
// they store)
int launch_phase(axb_ctx *c, const axb_batch *B, int phase, const BatchStage &stage,
                 cudaStream_t s) {
  TileTable t = table_of(B, phase);
  const int nb = nblocks_for(B, phase, t);
  unsigned long long *ctr = B->ctr + phase;
  axb_mark(c, kRegion[phase], s, true);
  int rc = AXB_OK;
  switch (phase) {
  case P_SOURCES:
    rc = launch_rhs_misc_batch(B->fd_order == 4 ? 1 : 0, B->rhs_args, t, ctr, B->src_steps, stage, nb, s);
    break;
  case P_FLUX_X:
  case P_FLUX_Y:
  case P_FLUX_Z: {
    const int dir = phase - P_FLUX_X;
    const int seg = dir == 0 ? 32 : segment_of(B, dir - 1);
    rc = launch_flux_batch(B->recon, dir, static_cast<const RhsArgs *>(B->rhs_args), t, ctr,
                           *B->eos, B->status, seg, stage, nb, s);
    break;
  }
  case P_AUX: rc = launch_rhs_misc_batch(2, B->rhs_args, t, ctr, 1, stage, nb, s); break;
  case P_CT: rc = launch_rhs_misc_batch(3, B->rhs_args, t, ctr, 1, stage, nb, s); break;
  case P_SYNC_E: rc = launch_sync_batch(B->sync_e, t, ctr, nb, s); break;
  case P_BSTAG: rc = launch_c2p_batch(0, B->c2p_args, t, ctr, *B->eos, B->status, nb, s); break;
  case P_C2P:
    rc = launch_c2p_batch(1, B->c2p_args, t, ctr, *B->eos, B->status, nb, s, B->c2p_queue,
                          4 * B->sms, B->noble);
    break;
  case P_SYNC_P: rc = launch_sync_batch(B->sync_p, t, ctr, nb, s); break;
  }
  axb_mark(c, kRegion[phase], s, false);
  return rc;
}

// one RHS evaluation, stored.  Every round of launches starts from zeroed work
// counters: a tile drawn from a counter that was never set can be negative
int run_rhs_phases(axb_ctx *c, const axb_batch *B, cudaStream_t s) {
  AXB_CUDA_TRY(cudaMemsetAsync(B->ctr, 0, NPHASE * sizeof(unsigned long long), s));
  for (int ph = P_SOURCES; ph <= P_CT; ++ph) {
    const int rc = launch_phase(c, B, ph, BatchStage{}, s);
    if (rc)
      return rc;
  }
  return AXB_OK;
}

} // namespace

// ---------------------------------------------------------------------------
// C ABI
// ---------------------------------------------------------------------------
AXB_API int axb_batch_destroy(axb_batch *B) {
  if (!B)
    return AXB_ERR_ARG;
  cudaFree(B->rhs_args);
  cudaFree(B->c2p_args);
  cudaFree(B->sync_e);
  cudaFree(B->sync_p);
  cudaFree(B->ctr);
  cudaFree(B->c2p_queue);
  for (auto &t : B->tab)
    free_table(t);
  for (auto &d : B->flux_seg)
    for (auto &t : d)
      free_table(t);
  delete B;
  return AXB_OK;
}

AXB_API int axb_batch_create(axb_ctx *c, int nbox, const axb_box *boxes,
                             const axb_fields *fields, const axb_fields *fields_n,
                             const axb_params *p, const axb_eos *eos, axb_batch **out) {
  if (!c || !boxes || !fields || !fields_n || !p || !eos || !out || nbox < 1)
    return AXB_ERR_ARG;
  *out = nullptr;
  axb_batch *B = new (std::nothrow) axb_batch();
  if (!B)
    return AXB_ERR_ARG;
  B->nbox = nbox;
  B->recon = p->reconstruction_method;
  B->fd_order = p->local_spatial_order;
  B->noble = p->c2p_prime == AXB_C2P_NOBLE;
  B->eos = eos;
  B->status = c->status;
  for (int ph = 0; ph < NPHASE; ++ph)
    B->ctas[ph] = 8;
  cudaDeviceGetAttribute(&B->sms, cudaDevAttrMultiProcessorCount, c->device);
  std::vector<axb_box> bx(boxes, boxes + nbox);
  for (const auto &b : bx)
    B->zones += (long long)b.n[0] * b.n[1] * b.n[2];
  int rc = batch_rhs_setup(c, nbox, boxes, fields, fields_n, p, eos, &B->rhs_args);
  if (!rc)
    rc = batch_c2p_setup(c, nbox, boxes, fields, p, eos, &B->c2p_args);
  if (!rc)
    rc = batch_sync_setup(nbox, boxes, fields, p->recon_type, &B->sync_e, &B->sync_p);
  B->src_steps = batch_steps(0, boxes, nbox, B->sms);
  for (int d = 0; d < 2; ++d)
    B->steps[d] = batch_steps(d + 1, boxes, nbox, B->sms);
  if (!rc)
    rc = make_table(bx, g_sources, B->src_steps, B->tab[P_SOURCES]);
  if (!rc)
    rc = make_table(bx, g_flux, 0, B->tab[P_FLUX_X]);
  for (int d = 0; d < 2 && !rc; ++d)
    for (int q = 0; q <= NSEG && !rc; ++q)
      rc = make_table(bx, g_flux, (d + 1) | ((q < NSEG ? kSeg[q] : B->steps[d]) << 2),
                      B->flux_seg[d][q]);
  if (!rc)
    rc = make_table(bx, g_aux, 0, B->tab[P_AUX]);
  if (!rc)
    rc = make_table(bx, g_ct, 0, B->tab[P_CT]);
  if (!rc)
    rc = make_table(bx, g_sync, 0, B->tab[P_SYNC_E]);
  if (!rc)
    rc = make_table(bx, g_c2p, 0, B->tab[P_BSTAG]);
  if (!rc)
    rc = make_table(bx, g_c2p, 1, B->tab[P_C2P]);
  if (!rc)
    rc = make_table(bx, g_sync,
                    p->recon_type == AXB_RECVAR_Z || p->recon_type == AXB_RECVAR_S ? 2 : 1,
                    B->tab[P_SYNC_P]);
  if (!rc && cudaMalloc(&B->ctr, NPHASE * sizeof(unsigned long long)) != cudaSuccess)
    rc = AXB_ERR_CUDA;
  if (!rc && c2p_batch_fast_ok(nbox, boxes, p) &&
      cudaMalloc(&B->c2p_queue, (B->zones + 1) * sizeof(unsigned long long)) != cudaSuccess)
    rc = AXB_ERR_CUDA;
  if (rc) {
    axb_batch_destroy(B);
    return rc;
  }
  *out = B;
  return AXB_OK;
}

// One RK substep of every box of the batch (as axb_substep does for one box):
// RHS group with the stage update in its last kernels, periodic fill of the
// evolved variables, post-step group, periodic fill of the primitives.
AXB_API int axb_batch_substep(axb_ctx *c, axb_batch *B, double alpha, double beta,
                              double gamma, double dt, int periodic, void *stream) {
  if (!c || !B)
    return AXB_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  AXB_CUDA_TRY(cudaMemsetAsync(B->ctr, 0, NPHASE * sizeof(unsigned long long), s));
  const BatchStage stage{1, alpha, beta, gamma * dt};
  for (int ph = 0; ph < NPHASE; ++ph) {
    if (!periodic && (ph == P_SYNC_E || ph == P_SYNC_P))
      continue;
    const int rc = launch_phase(c, B, ph, stage, s);
    if (rc)
      return rc;
  }
  return AXB_OK;
}

// Autotuner: times the RHS phases on the batch's own boxes for every
// candidate persistent-grid size and every candidate pencil segment of the y
// and z flux passes (the one axb_batch_create chose by the level's size is the
// first of them), the best of three samples each, and keeps the fastest.  The
// RHS phases overwrite what they read back (sources and the x pass write, y
// and z accumulate on top; timed storing the RHS, not with the stage update
// the substep makes in their place), so repeating them leaves the state as one
// RHS evaluation would; the stage update and the post-step are not touched.
// Synchronous; call it outside any stream capture.  out[0..1] receive the
// y / z segments in use, out[2] the CTAs per SM of the flux passes.
AXB_API int axb_batch_autotune(axb_ctx *c, axb_batch *B, int *out, void *stream) {
  if (!c || !B)
    return AXB_ERR_ARG;
  cudaStream_t s = (cudaStream_t)stream;
  cudaEvent_t e0, e1;
  AXB_CUDA_TRY(cudaEventCreate(&e0));
  AXB_CUDA_TRY(cudaEventCreate(&e1));
  const int saved_timing = c->timing;
  c->timing = 0;
  auto time_rhs = [&](int phase, float &best_ms) -> int {
    best_ms = 1e30f;
    for (int sample = 0; sample < 3; ++sample) {
      AXB_CUDA_TRY(cudaMemsetAsync(B->ctr, 0, NPHASE * sizeof(unsigned long long), s));
      for (int ph = P_SOURCES; ph <= P_CT; ++ph) {
        if (ph == phase)
          AXB_CUDA_TRY(cudaEventRecord(e0, s));
        const int rc = launch_phase(c, B, ph, BatchStage{}, s);
        if (rc)
          return rc;
        if (ph == phase)
          AXB_CUDA_TRY(cudaEventRecord(e1, s));
      }
      float ms = 0;
      AXB_CUDA_TRY(cudaEventSynchronize(e1));
      AXB_CUDA_TRY(cudaEventElapsedTime(&ms, e0, e1));
      best_ms = std::min(best_ms, ms);
    }
    return AXB_OK;
  };
  int rc = run_rhs_phases(c, B, s); // warm-up
  // grid size of each RHS phase (segments at their defaults)
  for (int ph = P_SOURCES; ph <= P_CT && !rc; ++ph) {
    int best = B->ctas[ph];
    float best_ms = 1e30f;
    for (int q = 0; q < NCTAS && !rc; ++q) {
      B->ctas[ph] = kCtas[q];
      float ms = 0;
      rc = time_rhs(ph, ms);
      if (!rc && ms < best_ms) {
        best_ms = ms;
        best = kCtas[q];
      }
    }
    B->ctas[ph] = best;
  }
  // segment length of the y and z passes
  for (int d = 0; d < 2 && !rc; ++d) {
    int best = B->seg[d] = NSEG; // the level's own choice is a candidate too
    float best_ms = 1e30f;
    for (int q = NSEG; q >= 0 && !rc; --q) {
      B->seg[d] = q;
      float ms = 0;
      rc = time_rhs(P_FLUX_Y + d, ms);
      if (!rc && ms < best_ms) {
        best_ms = ms;
        best = q;
      }
    }
    B->seg[d] = best;
  }
  // the light post-step phases take the auxiliaries' grid size.  The recovery
  // keeps its own: its kernels hold up to 8 CTAs per SM, the flux passes 3, and
  // at the 4 these often get it ran at half its warps (64 boxes: 824 us at 8,
  // 1129 us at 4)
  B->ctas[P_SYNC_E] = B->ctas[P_SYNC_P] = B->ctas[P_AUX];
  B->ctas[P_BSTAG] = B->ctas[P_AUX];
  if (!rc)
    rc = run_rhs_phases(c, B, s); // leave one consistent RHS evaluation behind
  if (!rc && cudaStreamSynchronize(s) != cudaSuccess)
    rc = AXB_ERR_CUDA;
  c->timing = saved_timing;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (out) {
    out[0] = segment_of(B, 0);
    out[1] = segment_of(B, 1);
    out[2] = B->ctas[P_FLUX_Y];
  }
  return rc;
}
