// Launch helper for k_flux_pass, instantiated per reconstruction scheme in
// its own translation unit (axb_flux_<scheme>.cu) to keep builds parallel.
#pragma once

#include "axb_batch.cuh"
#include "axb_internal.hxx"
#include "axb_rhs_kernels.cuh"

namespace axb {

// a y or z pass, with its dynamic shared memory allowed
template <class K, class... Args>
void launch_pass(K kernel, dim3 grid, dim3 block, cudaStream_t s, const Args &...args) {
  cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FLUX_SMEM);
  kernel<<<grid, block, FLUX_SMEM, s>>>(args...);
}

template <int RECON, class EOS, bool UCT>
int launch_flux_pass_uct(int dir, const RhsArgs &a, const EOS &eos, cudaStream_t s) {
  const BoxDev &b = a.b;
  if (dir == 0) {
    const long long blocks = flux_x_blocks(b, a.text);
    if (blocks > 0x7fffffffLL)
      return AXB_ERR_TOO_LARGE;
    k_flux_x<RECON, EOS, UCT><<<(unsigned)blocks, 128, 0, s>>>(a, eos);
    return cudaGetLastError() == cudaSuccess ? AXB_OK : AXB_ERR_CUDA;
  }
  // The threads walk the transverse plane [ng-1, ng+n]^2 row after row (as in
  // the batched kernels), so the 2 extra columns of the plane do not leave most
  // of a warp idle.  (Blocks of 32 columns x 4 rows, which MP5 was faster on
  // while its stencils came through L1: 128^3 substep 3.19 ms, 2.88 so; 96^3
  // tabulated RHS 3.49 ms, 2.48 so.)
  const int seglen = flux_steps(b, dir, a.text, sm_count());
  const dim3 grid(unsigned(flux_plane_blocks(b, dir, a.text)), 1,
                  (b.n[dir] + seglen - 1) / seglen);
  if (dir == 1)
    launch_pass(k_flux_pass<1, RECON, EOS, UCT>, grid, dim3(FLUX_T), s, a, eos, seglen);
  else
    launch_pass(k_flux_pass<2, RECON, EOS, UCT>, grid, dim3(FLUX_T), s, a, eos, seglen);
  return cudaGetLastError() == cudaSuccess ? AXB_OK : AXB_ERR_CUDA;
}

// the upwind-CT face data and the wider transverse range are a separate
// instantiation, so the flux-CT passes carry none of it
template <int RECON, class EOS>
int launch_flux_pass_eos(int dir, const RhsArgs &a, const EOS &eos, cudaStream_t s) {
  if (a.use_uct)
    return launch_flux_pass_uct<RECON, EOS, true>(dir, a, eos, s);
  return launch_flux_pass_uct<RECON, EOS, false>(dir, a, eos, s);
}

template <int RECON>
int launch_flux_pass_t(int dir, const RhsArgs &a, const axb_eos &eos, cudaStream_t s) {
  if (eos.kind == 0)
    return launch_flux_pass_eos<RECON>(dir, a, eos.ideal, s);
  if (eos.kind == 1)
    return launch_flux_pass_eos<RECON>(dir, a, tab_for_launch(eos, a.status), s);
  return AXB_ERR_UNSUPPORTED;
}

// Batched flux passes over the boxes of a batch (tile tables built by the
// batch with the grids of launch_flux_pass_eos).
template <int DIR, int RECON, class EOS>
__global__ void __launch_bounds__(FLUX_T, FLUX_MINB)
    k_flux_pass_batch(const RhsArgs *args, const TileTable t, unsigned long long *ctr,
                      const __grid_constant__ EOS eos, const int seglen, const BatchStage stage) {
  batch_loop(
      args, t, ctr,
      [&](const RhsArgs &a, const uint3 bid) {
        flux_pass_body<DIR, RECON, EOS>(a, eos, seglen, bid);
      },
      stage);
}

template <int RECON, class EOS>
__global__ void __launch_bounds__(128, AXB_FLUX_X_MINB)
    k_flux_x_batch(const RhsArgs *args, const TileTable t, unsigned long long *ctr, const __grid_constant__ EOS eos) {
  batch_loop(args, t, ctr, [&](const RhsArgs &a, const uint3 bid) {
    flux_x_body<RECON, EOS>(a, eos, bid);
  });
}

template <int RECON, class EOS>
int launch_flux_batch_eos(int dir, const RhsArgs *args, const TileTable &t,
                          unsigned long long *ctr, const EOS &eos, int seglen,
                          const BatchStage &stage, int nblocks, cudaStream_t s) {
  if (t.total == 0)
    return AXB_OK;
  if (dir == 0)
    k_flux_x_batch<RECON, EOS><<<nblocks, 128, 0, s>>>(args, t, ctr, eos);
  else if (dir == 1)
    launch_pass(k_flux_pass_batch<1, RECON, EOS>, dim3(nblocks), dim3(FLUX_T), s, args,
                t, ctr, eos, seglen, stage);
  else
    launch_pass(k_flux_pass_batch<2, RECON, EOS>, dim3(nblocks), dim3(FLUX_T), s, args,
                t, ctr, eos, seglen, stage);
  return cudaGetLastError() == cudaSuccess ? AXB_OK : AXB_ERR_CUDA;
}

template <int RECON>
int launch_flux_batch_t(int dir, const RhsArgs *args, const TileTable &t,
                        unsigned long long *ctr, const axb_eos &eos, DevStatus *status,
                        int seglen, const BatchStage &stage, int nblocks, cudaStream_t s) {
  if (eos.kind == 0)
    return launch_flux_batch_eos<RECON>(dir, args, t, ctr, eos.ideal, seglen, stage, nblocks,
                                        s);
  if (eos.kind == 1)
    return launch_flux_batch_eos<RECON>(dir, args, t, ctr, tab_for_launch(eos, status), seglen,
                                        stage, nblocks, s);
  return AXB_ERR_UNSUPPORTED;
}

int launch_flux_batch(int recon, int dir, const RhsArgs *args, const TileTable &t,
                      unsigned long long *ctr, const axb_eos &eos, DevStatus *status,
                      int seglen, const BatchStage &stage, int nblocks, cudaStream_t s);

int launch_flux_ppm(int dir, const RhsArgs &a, const axb_eos &eos, cudaStream_t s);
int launch_flux_wenoz(int dir, const RhsArgs &a, const axb_eos &eos, cudaStream_t s);
int launch_flux_mp5(int dir, const RhsArgs &a, const axb_eos &eos, cudaStream_t s);
int launch_flux_low(int recon, int dir, const RhsArgs &a, const axb_eos &eos, cudaStream_t s);

} // namespace axb
