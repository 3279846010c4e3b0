// Mixed-precision Lennard-Jones forces over full lists, in two stages per block:
// the form for batches too small to fill the GPU with one thread per particle.
//
// One thread walking a particle's list (k_force, xnb_step_kernels.cu) waits for
// ~40 dependent rounds of gathers; below some 10^5 particles nothing hides that
// latency. The values have to stay those of that walk, bit for bit: FP32 force
// factors pd, and the sums of pd x_b, pd y_b, pd z_b, pd (and the energies) in
// FP64, each added in list order.
//   Stage 1 (FP32): a warp takes one particle at a time, 32 list entries per
//     step: mirror gathers, r^2, the cutoff (FP64 inside the proven band) and
//     pd; a ballot appends the pairs within rc to the particle's rows in shared
//     memory, in list order: their FP64 coordinates (image applied) and pd.
//   Stage 2 (FP64): a lane per (particle, sum) runs its sequential FMA chain
//     over the rows, nothing but two shared loads and the FMA per term. A warp
//     issues one FP64 instruction per 64 cycles whatever else it does, so 32
//     chains share each.
#include <algorithm>

#include "xnb_launch.cuh"
#include "xnb_lj_pair.cuh"
#include "xnb_traverse.cuh"

namespace xnb {

namespace {

// A particle of the block.
struct Row {
  float4 own;            // the particle's mirror
  const uint32_t* list;
  uint32_t n;            // list length, 0 for a slot that is not walked
  uint32_t sys;          // kNone for such a slot
  uint32_t count;        // pairs in the row (this chunk)
  uint32_t pad;
};
constexpr uint32_t kNone = 0xFFFFFFFFu;

template <bool PE, bool KICK>
__global__ void __launch_bounds__(256, 4)
    k_force_mixed(uint32_t n_part, BatchSource src, DevArrays a, uint32_t group, uint32_t chunk) {
  constexpr uint32_t kSums = PE ? 5 : 4;   // x, y, z, pd and the energy
  constexpr uint32_t kPer = 32 / kSums;    // particles per warp in stage 2
  extern __shared__ __align__(16) unsigned char force_smem[];
  const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const uint32_t stride = chunk + 1u;  // odd: the rows of a warp's lanes start on different banks
  Row* const info = reinterpret_cast<Row*>(force_smem);
  double* const rows = reinterpret_cast<double*>(info + group);  // per particle kSums rows: x, y, z, pd (, energy)
  const uint32_t first = blockIdx.x * group;

  uint32_t my_n = 0;
  if (threadIdx.x < group) {
    const uint32_t i = first + threadIdx.x;
    uint32_t s = 0;
    const uint32_t* list = nullptr;
    const bool ok = i < n_part && src.locate(i, s, list, my_n);
    if (!ok) my_n = 0;
    Row r;
    r.own = ok ? src.pf[i] : make_float4(0.f, 0.f, 0.f, 0.f);
    r.list = list;
    r.n = my_n;
    r.sys = ok ? s : kNone;
    r.count = 0;
    r.pad = 0;
    info[threadIdx.x] = r;
  }
  __syncthreads();

  // the warps that sum: group / kPer of them, from another one in each block
  // (a warp's FP64 work runs on its own quarter of the SM)
  const uint32_t turn = (wib + blockIdx.x) % nwarp;
  const uint32_t row = turn * kPer + lane / kSums;
  const uint32_t ax = lane % kSums;
  const bool worker = lane < kPer * kSums && row < group && info[min(row, group - 1u)].sys != kNone;
  double acc = 0.0;

  for (uint32_t kb = 0;; kb += chunk) {
    // ---- stage 1 ----
    for (uint32_t p = wib; p < group; p += nwarp) {
      const Row r = info[p];
      uint32_t count = 0;
      double* const out = rows + static_cast<size_t>(p) * kSums * stride;
      if (r.n > kb) {
        const uint32_t i = first + p;
        const SysDesc& S = src.sys[r.sys];
        const uint32_t pbase = S.part_base;
        const float r2_in = S.rc2_f - S.rc_margin_f, r2_out = S.rc2_f + S.rc_margin_f, r2_min = S.rc_margin_f;
        const float sig2 = S.sig2_f, eps24 = S.eps24_f, step = S.lo_step_f;
        const uint32_t wa = __float_as_uint(r.own.w);
        const float qx = field_x(wa), qy = field_y(wa), qz = field_z(wa);
        const uint32_t* __restrict__ L = r.list;
        const uint32_t self_e = ((i - pbase) << 5) | static_cast<uint32_t>(kImageCenter);
        const uint32_t kend = min(r.n, kb + chunk);
        uint32_t e = kb + lane < kend ? __ldg(L + kb + lane) : self_e;
        for (uint32_t k0 = kb; k0 < kend; k0 += 32u) {
          const uint32_t ent = e, code = ent & 31u;
          const uint32_t j = pbase + (ent >> 5);
          const float4 hb = __ldg(src.pf + j);
          double xb = __ldg(src.rx + j), yb = __ldg(src.ry + j), zb = __ldg(src.rz + j);
          e = k0 + 32u + lane < kend ? __ldg(L + k0 + 32u + lane) : self_e;
          const bool valid = k0 + lane < kend;
          const uint32_t wb = __float_as_uint(hb.w);
          // within 2u|d| + 2 lo_step of the FP64 displacement (u = 2^-24)
          float dx = fmaf(field_x(wb) - qx, step, hb.x - r.own.x);
          float dy = fmaf(field_y(wb) - qy, step * 0.0009765625f, hb.y - r.own.y);
          float dz = fmaf(field_z(wb) - qz, step, hb.z - r.own.z);
          if (code != static_cast<uint32_t>(kImageCenter)) {
            const float4 lb = __ldg(src.pflo + j), la = __ldg(src.pflo + i);
            const uint32_t cx = code % 3u, cy = (code / 3u) % 3u, cz = code / 9u;
            const float tie = S.image_tie_f;
            bool sure = true;
            dx = image_axis(hb.x, r.own.x, lb.x, la.x, cx, S.period_f[0], S.period_lo_f[0], tie, sure);
            dy = image_axis(hb.y, r.own.y, lb.y, la.y, cy, S.period_f[1], S.period_lo_f[1], tie, sure);
            dz = image_axis(hb.z, r.own.z, lb.z, la.z, cz, S.period_f[2], S.period_lo_f[2], tie, sure);
            // image_coord: x + (+-1.0 * period)
            if (cx != 1u) xb = __dadd_rn(xb, cx == 2u ? S.period[0] : -S.period[0]);
            if (cy != 1u) yb = __dadd_rn(yb, cy == 2u ? S.period[1] : -S.period[1]);
            if (cz != 1u) zb = __dadd_rn(zb, cz == 2u ? S.period[2] : -S.period[2]);
            if (!sure) {
              dx = narrow_f64(__dsub_rn(xb, src.rx[i]));
              dy = narrow_f64(__dsub_rn(yb, src.ry[i]));
              dz = narrow_f64(__dsub_rn(zb, src.rz[i]));
            }
          }
          const float r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
          bool in = valid && r2 < r2_in && r2 > r2_min;
          if (valid && !in && !(r2 > r2_out)) {
            // inside the FP32 band: the FP64 decision
            const double d2 = norm2_rn(__dsub_rn(xb, src.rx[i]), __dsub_rn(yb, src.ry[i]), __dsub_rn(zb, src.rz[i]));
            in = d2 > 0.0 && d2 <= S.rcut2;
          }
          const unsigned m = __ballot_sync(0xffffffffu, in);
          if (in) {
            // the hardware reciprocal (within 1 ulp) is part of the FP32 force magnitude
            float ir2;
            asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(ir2) : "f"(r2));
            const float s2 = sig2 * ir2;
            const float s6 = s2 * s2 * s2;
            const float pd = eps24 * s6 * fmaf(-2.0f, s6, 1.0f) * ir2;
            double* const o = out + count + __popc(m & ((1u << lane) - 1u));
            o[0] = xb;
            o[stride] = yb;
            o[2u * stride] = zb;
            o[3u * stride] = widen_f32_fast(pd);
            if (PE) o[4u * stride] = widen_f32_fast(0.5f * fmaf(S.eps4_f * s6, s6 - 1.0f, -S.e_shift_f));
          }
          count += __popc(m);
        }
        // zero terms up to a multiple of four pairs
        if (lane < ((0u - count) & 3u)) {
#pragma unroll
          for (uint32_t t = 0; t < kSums; ++t) out[t * stride + count + lane] = 0.0;
        }
      }
      if (lane == 0) info[p].count = count;
    }
    __syncthreads();
    // ---- stage 2 ----
    if (worker) {
      const uint32_t count = (info[row].count + 3u) & ~3u;
      const double* const mine = rows + (static_cast<size_t>(row) * kSums + ax) * stride;
      const double* const factor = rows + (static_cast<size_t>(row) * kSums + 3u) * stride;
      const bool axis = ax < 3u;  // a coordinate times pd; pd and the energy are summed as they are
      for (uint32_t k = 0; k < count; k += 4u) {
        double x[4], f[4];
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          x[t] = mine[k + t];
          f[t] = axis ? factor[k + t] : 1.0;
        }
#pragma unroll
        for (int t = 0; t < 4; ++t) acc = fma(f[t], x[t], acc);
      }
    }
    if (!__syncthreads_or(my_n > kb + chunk)) break;
  }

  // ---- the particle's sums ----
  const double psum = __shfl_sync(0xffffffffu, acc, lane - ax + 3u);
  if (!worker || ax == 3u) return;
  const SysDesc& S = src.sys[info[row].sys];
  const uint32_t i = first + row;
  if (PE && ax == 4u) {
    a.pe[i] = acc;
    return;
  }
  // the FP64 displacement folded out of the sum: sum pd (r_b - r_a)
  double f = fma(-(ax == 0u ? src.rx : (ax == 1u ? src.ry : src.rz))[i], psum, acc);
  if (S.divide_by_mass) f = __ddiv_rn(f, S.mass);
  (ax == 0u ? a.fx : (ax == 1u ? a.fy : a.fz))[i] = f;
  if (KICK) {
    double* const v = ax == 0u ? a.vx : (ax == 1u ? a.vy : a.vz);
    v[i] = fma(f, S.dt_half, v[i]);
  }
}

template <bool PE, bool KICK>
void go(const Extent& ex, const SysDesc* sys, const SysState* st, const DevArrays& a, int sys_only,
        cudaStream_t stream) {
  constexpr uint32_t sums = PE ? 5 : 4, group = 32u / sums;
  const BatchSource src(sys, st, a, sys_only);
  // list entries per chunk: a multiple of 32 that the usual lists fit, up to the 96
  // that leave shared memory for the eight blocks per SM which the registers allow
  // (23,328 atoms, lists of up to 84, 98, 157 and 335 entries: 40 / 35, 43 / 38, 82 /
  // 60 and 201 / 118 us with chunks of up to 256 / 96; 64 costs lists of 87 a tenth)
  constexpr uint32_t longest = 96u;
  const uint32_t chunk = std::min(std::max((ex.list_slot * 2u / 3u + 31u) / 32u * 32u, 32u), longest);
  static_assert(group * (sizeof(Row) + (longest + 1u) * sums * sizeof(double)) <= 48u * 1024u,
                "more shared memory than a launch may have without raising its kernel's limit");
  const size_t smem = group * (sizeof(Row) + static_cast<size_t>(chunk + 1u) * sums * sizeof(double));
  const unsigned grid = (ex.n_part + group - 1u) / group;
  // stage 1: a warp per particle while every block has an SM of its own, then
  // two particles per warp (32,000 atoms: 43 us with 128 threads, 61 us with 256)
  const unsigned threads = grid <= static_cast<unsigned>(ex.sm_count) ? group * 32u : group * 16u;
  k_force_mixed<PE, KICK><<<grid, threads, smem, stream>>>(ex.n_part, src, a, group, chunk);
}

// ---------------------------------------------------------------------------
// One thread per particle, for batches of many waves: every list entry once, two at
// a time, their mirrors and position steps (DevArrays::pstep) in flight together;
// a pair's FP64 position is formed only within the cutoff. A pair costs 3 DFMA on
// the FP64 pipe, which bounds the walk: a warp makes about 100 rounds of three (its
// longest list), and at one million atoms the pipe is busy 82% of the time (the
// marking walk gathers the entries near the cutoff a second time: 73 rounds, the
// pipe at 58% and the L1 data stage at 66%). 64 registers hold 16 blocks of 64
// threads per SM. Marking walk with the sums of PairSum / this one: 25 steps of 4M
// atoms 74.9 / 69.4 ms (three such batches at once 75.0 / 67.0); 1M atoms with
// energies 728 / 690 us; a batch of 96 small systems, 20 steps, three at once 45.2 /
// 35.4 ms. With 56 registers 71.7 ms and 773 us, four entries at a time 80.8 ms.
struct WalkParticle {
  const double* rx;
  const double* ry;
  const double* rz;
  const float4* pf;
  const int4* pstep;
  const uint32_t* list;
  uint32_t i, n, pbase;
  float4 own;
};

// b's FP64 position from its mirror and steps.
__device__ __forceinline__ void position(const WalkParticle& w, uint32_t j, float4 hb, int4 d, double& x, double& y,
                                         double& z) {
  if (d.w) {
    x = w.rx[j];
    y = w.ry[j];
    z = w.rz[j];
    return;
  }
  x = step_coord(hb.x, d.x);
  y = step_coord(hb.y, d.y);
  z = step_coord(hb.z, d.z);
}

// One entry: the values of mixed_pair (xnb_lj_pair.cuh) with the packed residuals,
// handed to sink(pd, s6, x_b, y_b, z_b) for a pair within the cutoff.
template <class Sink>
__device__ __forceinline__ void walk_entry(const SysDesc& S, const WalkParticle& w, uint32_t e, float4 hb, int4 d,
                                           float step, float r2_in, float r2_out, float r2_min, const Sink& sink) {
  const uint32_t code = e & 31u, j = w.pbase + (e >> 5);
  float dx, dy, dz, r2;
  double x, y, z;
  if (code == static_cast<uint32_t>(kImageCenter)) {
    // within 2u|d| + 2 lo_step of the FP64 displacement (u = 2^-24)
    const uint32_t wb = __float_as_uint(hb.w), wa = __float_as_uint(w.own.w);
    dx = fmaf(field_x(wb) - field_x(wa), step, hb.x - w.own.x);
    dy = fmaf(field_y(wb) - field_y(wa), step * 0.0009765625f, hb.y - w.own.y);
    dz = fmaf(field_z(wb) - field_z(wa), step, hb.z - w.own.z);
    r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    if (r2 > r2_out) return;
    position(w, j, hb, d, x, y, z);
  } else {
    position(w, j, hb, d, x, y, z);
    x = image_coord(x, S.period[0], static_cast<int>(code % 3u));
    y = image_coord(y, S.period[1], static_cast<int>((code / 3u) % 3u));
    z = image_coord(z, S.period[2], static_cast<int>(code / 9u));
    dx = narrow_f64(__dsub_rn(x, w.rx[w.i]));
    dy = narrow_f64(__dsub_rn(y, w.ry[w.i]));
    dz = narrow_f64(__dsub_rn(z, w.rz[w.i]));
    r2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
    if (r2 > r2_out) return;
  }
  if (!(r2 < r2_in && r2 > r2_min)) {
    // inside the FP32 band: the FP64 decision
    const double d2 = norm2_rn(__dsub_rn(x, w.rx[w.i]), __dsub_rn(y, w.ry[w.i]), __dsub_rn(z, w.rz[w.i]));
    if (!(d2 > 0.0 && d2 <= S.rcut2)) return;
  }
  // the hardware reciprocal (within 1 ulp) is part of the FP32 force magnitude
  float ir2;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(ir2) : "f"(r2));
  const float s2 = S.sig2_f * ir2;
  const float s6 = s2 * s2 * s2;
  sink(S.eps24_f * s6 * fmaf(-2.0f, s6, 1.0f) * ir2, s6, x, y, z);
}

__device__ __forceinline__ float pair_energy(const SysDesc& S, float s6) {
  return 0.5f * fmaf(S.eps4_f * s6, s6 - 1.0f, -S.e_shift_f);
}

// Sum of pd, or of the energies, in FP64, in list order (where PairSum is not exact).
template <bool ENERGY>
__device__ __noinline__ double sum_in_order(const SysDesc& S, const double* rx, const double* ry, const double* rz,
                                            const float4* pf, const int4* pstep, uint32_t i, const uint32_t* list,
                                            uint32_t n) {
  const WalkParticle w{rx, ry, rz, pf, pstep, list, i, n, S.part_base, pf[i]};
  double sum = 0.0;
  for (uint32_t k = 0; k < n; ++k) {
    const uint32_t e = list[k], j = w.pbase + (e >> 5);
    walk_entry(S, w, e, pf[j], pstep[j], S.lo_step_f, S.rc2_f - S.rc_margin_f, S.rc2_f + S.rc_margin_f, S.rc_margin_f,
               [&](float pd, float s6, double, double, double) {
                 sum += widen_f32_fast(ENERGY ? pair_energy(S, s6) : pd);
               });
  }
  return sum;
}

template <bool PE, bool KICK>
__global__ void __maxnreg__(64) k_force_walk(uint32_t n_part, BatchSource src, DevArrays a) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  uint32_t s, n;
  const uint32_t* list;
  if (i >= n_part || !src.locate(i, s, list, n)) return;
  const SysDesc& S = src.sys[s];
  const WalkParticle w{src.rx, src.ry, src.rz, src.pf, a.pstep, list, i, n, S.part_base, src.pf[i]};
  const float step = S.lo_step_f, r2_in = S.rc2_f - S.rc_margin_f, r2_out = S.rc2_f + S.rc_margin_f,
              r2_min = S.rc_margin_f;
  const int pd_exp = S.sum_pd.exponent;
  double fx = 0.0, fy = 0.0, fz = 0.0;
  PairSum pds, pes;
  pds.clear();
  pes.clear();
  const auto add = [&](float pd, float s6, double x, double y, double z) {
    // the FP64 displacement folded into the accumulation (mixed_pair)
    const double pdd = widen_f32_fast(pd);
    fx = fma(pdd, x, fx);
    fy = fma(pdd, y, fy);
    fz = fma(pdd, z, fz);
    pds.add(pd_exp, pd);
    if (PE) pes.add(S.sum_pe.exponent, pair_energy(S, s6));
  };
  // entries past an odd list's end: the particle's own slot, not visited (list
  // slots are multiples of 8 entries, 32-byte aligned)
  const uint32_t self_e = ((i - w.pbase) << 5) | static_cast<uint32_t>(kImageCenter);
  uint2 next = n ? __ldg(reinterpret_cast<const uint2*>(list)) : make_uint2(self_e, self_e);
  for (uint32_t k = 0; k < n; k += 2u) {
    const uint32_t e0 = next.x, e1 = k + 1u < n ? next.y : self_e;
    const uint32_t j0 = w.pbase + (e0 >> 5), j1 = w.pbase + (e1 >> 5);
    const float4 h0 = __ldg(w.pf + j0);
    const int4 d0 = __ldg(w.pstep + j0);
    const float4 h1 = __ldg(w.pf + j1);
    const int4 d1 = __ldg(w.pstep + j1);
    if (k + 2u < n) next = __ldg(reinterpret_cast<const uint2*>(list + k + 2u));
    walk_entry(S, w, e0, h0, d0, step, r2_in, r2_out, r2_min, add);
    if (k + 1u < n) walk_entry(S, w, e1, h1, d1, step, r2_in, r2_out, r2_min, add);
  }
  const double psum = pds.exact(S.sum_pd) ? pds.value(S.sum_pd)
                                          : sum_in_order<false>(S, a.rx, a.ry, a.rz, a.pf, a.pstep, i, list, n);
  double pe = 0.0;
  if (PE)
    pe = pes.exact(S.sum_pe) ? pes.value(S.sum_pe)
                             : sum_in_order<true>(S, a.rx, a.ry, a.rz, a.pf, a.pstep, i, list, n);
  finish_mixed<PE, KICK>(S, a, i, fx, fy, fz, psum, pe);
}

template <bool PE, bool KICK>
void go_walk(const Extent& ex, const SysDesc* sys, const SysState* st, const DevArrays& a, int sys_only,
             cudaStream_t stream) {
  const unsigned threads = ex.force_block > 0 ? static_cast<unsigned>(ex.force_block) : 64u;
  // All of an SM's memory as L1: a block of it beside another batch's neighbour build,
  // whose stages leave little L1, gathers from L2 and holds that SM's launch up.
  // Three batches stepping at once: 25 steps of 4M atoms 69.6 to 77 -> 67.0 ms, 20
  // steps of 96 small systems 42.2 -> 35.4 ms; one alone 69.7 / 70.0 and 38.3 / 38.6.
  set_attribute(k_force_walk<PE, KICK>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxL1);
  k_force_walk<PE, KICK><<<(ex.n_part + threads - 1u) / threads, threads, 0, stream>>>(
      ex.n_part, BatchSource(sys, st, a, sys_only), a);
}

}  // namespace

int launch_force_mixed(const Extent& ex, const SysDesc* sys, const SysState* st, const DevArrays& a, bool with_pe,
                       bool second_half, int sys_only, cudaStream_t stream) {
  if (with_pe && second_half) go<true, true>(ex, sys, st, a, sys_only, stream);
  else if (with_pe) go<true, false>(ex, sys, st, a, sys_only, stream);
  else if (second_half) go<false, true>(ex, sys, st, a, sys_only, stream);
  else go<false, false>(ex, sys, st, a, sys_only, stream);
  return 1;
}

int launch_force_walk(const Extent& ex, const SysDesc* sys, const SysState* st, const DevArrays& a, bool with_pe,
                      bool second_half, int sys_only, cudaStream_t stream) {
  if (with_pe && second_half) go_walk<true, true>(ex, sys, st, a, sys_only, stream);
  else if (with_pe) go_walk<true, false>(ex, sys, st, a, sys_only, stream);
  else if (second_half) go_walk<false, true>(ex, sys, st, a, sys_only, stream);
  else go_walk<false, false>(ex, sys, st, a, sys_only, stream);
  return 1;
}

}  // namespace xnb
