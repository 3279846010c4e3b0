// Launches of the full-precision Lennard-Jones forces (xnb_force_pairs.cuh).
#include "xnb_force_pairs.cuh"
#include "xnb_launch.cuh"

namespace xnb {

namespace {

constexpr uint32_t kWarps = 4;

// Eight blocks per SM, 64 registers: what the loads that find short lists need
// (953,312 atoms at density 0.02, Newton: 228 us with the 72 registers it would take).
template <int P, bool PE, bool KICK, bool NEWTON>
__global__ void __launch_bounds__(kWarps * 32, 8) k_force_pairs(uint32_t n_part, BatchSource src, DevArrays a) {
  __shared__ pairs::WarpSmem sm[kWarps];
  const uint32_t w = threadIdx.x >> 5;
  pairs::eight_particles<P, PE, KICK, NEWTON>((blockIdx.x * kWarps + w) * pairs::kPer, n_part, src, a, sm[w]);
}

template <int P, bool NEWTON>
void go(const Extent& ex, const BatchSource& src, const DevArrays& a, bool with_pe, bool second_half,
        cudaStream_t stream) {
  const uint32_t group = kWarps * pairs::kPer;
  const unsigned grid = (ex.n_part + group - 1u) / group, threads = kWarps * 32u;
  if constexpr (NEWTON) {  // the kick follows in k_force_finish
    if (with_pe) k_force_pairs<P, true, false, true><<<grid, threads, 0, stream>>>(ex.n_part, src, a);
    else k_force_pairs<P, false, false, true><<<grid, threads, 0, stream>>>(ex.n_part, src, a);
  } else {
    if (with_pe && second_half) k_force_pairs<P, true, true, false><<<grid, threads, 0, stream>>>(ex.n_part, src, a);
    else if (with_pe) k_force_pairs<P, true, false, false><<<grid, threads, 0, stream>>>(ex.n_part, src, a);
    else if (second_half) k_force_pairs<P, false, true, false><<<grid, threads, 0, stream>>>(ex.n_part, src, a);
    else k_force_pairs<P, false, false, false><<<grid, threads, 0, stream>>>(ex.n_part, src, a);
  }
}

}  // namespace

int launch_force_pairs(const Extent& ex, const SysDesc* sys, const SysState* st, const DevArrays& a, int precision,
                       bool newton, bool with_pe, bool second_half, int sys_only, cudaStream_t stream) {
  const BatchSource src(sys, st, a, sys_only);
  if (precision == kFp64Exact) go<kFp64Exact, false>(ex, src, a, with_pe, second_half, stream);
  else if (newton) go<kFp64, true>(ex, src, a, with_pe, second_half, stream);
  else go<kFp64, false>(ex, src, a, with_pe, second_half, stream);
  return 1;
}

}  // namespace xnb
