// The split of the RHS group's marching kernels, as a host library
// (tests/test_steps.py).
#include "../asterx_b200/csrc/axb_rhs_kernels.cuh"
#include "../asterx_b200/csrc/axb_rhs_misc.cuh"

extern "C" void rhs_steps(const int *n, int te, int sms, int *out) {
  axb::BoxDev b{};
  for (int d = 0; d < 3; ++d)
    b.n[d] = n[d];
  out[0] = axb::flux_steps(b, 1, te, sms);
  out[1] = axb::flux_steps(b, 2, te, sms);
  const long long rows = (long long)((n[0] + 127) / 128) * n[1];
  const long long packed = ((long long)n[0] * n[1] + 127) / 128;
  out[2] = axb::sources_steps(n[2], packed < rows ? packed : rows, sms);
}
