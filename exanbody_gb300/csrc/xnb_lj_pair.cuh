// Pieces of the Lennard-Jones pair body shared by the mixed force traversals
// (xnb_step_kernels.cu: one thread per particle, marking first; xnb_force_mixed.cu:
// two stages, and one thread per particle visiting each entry once;
// xnb_force_staged.cu: cell segments staged in shared memory).
#pragma once

#include "xnb_launch.cuh"
#include "xnb_traverse.cuh"

namespace xnb {

// ---------------------------------------------------------------------------
// Double-precision reciprocal of d > 0 from an FP32 seed refined by two
// Newton-Raphson steps y <- y + y*(1 - d*y) in FP64, not correctly rounded.
// The seed stays off the FP64 pipe: d is truncated to binary32 by moving its
// exponent (re-biased by -896) and the top 23 fraction bits with one funnel
// shift, the exponent field clamped to [1, 252] so that the FP32 reciprocal is
// a positive normal, which widens back by the inverse bit move. For d in
// [2^-126, 2^126) the seed (truncation, then the hardware FP32 reciprocal,
// within 1 ulp) is within 2^-22 of 1/d, and the two steps take the error to
// 2^-44, then below the FP64 rounding.
__device__ __forceinline__ double rcp_nr(double d) {
  const int hi = min(max(__double2hiint(d) - 0x38000000, 0x00100000), 0x0fcfffff);
  const float s = __uint_as_float(__funnelshift_l(static_cast<uint32_t>(__double2loint(d)), static_cast<uint32_t>(hi), 3));
  float rf;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rf) : "f"(s));
  const uint32_t r = __float_as_uint(rf);
  double y = __hiloint2double(static_cast<int>((r >> 3) + 0x38000000u), static_cast<int>(r << 29));
  double e = fma(-d, y, 1.0);
  y = fma(y, e, y);
  e = fma(-d, y, 1.0);
  return fma(y, e, y);
}

// Sum of one FP32 term per pair, as FP64 additions in list order would give it,
// without the FP64 pipe: every term is a multiple of a quantum Q, 2^23 Q <= |term|
// < 2^53 Q, and while the sum of |term| stays within 2^52 Q every partial sum is
// exact in FP64, so the sum is Q times the integer sum of term / Q in any order. A
// term outside that range (a force factor near its zero crossing, some 10^-5 of
// the particles; an energy within 3e-6 sigma of a cutoff of 2.5 sigma, some 10^-4)
// sets `inexact`: that particle is summed in FP64, in order. An FP64 instruction
// holds a quarter of an SM's FP64 pipe for 64 cycles; these are about twelve on
// the integer pipes.
struct PairSum {
  long long units;  // sum of term / Q
  float size;       // sum of |term|
  bool inexact;

  __device__ __forceinline__ void clear() {
    units = 0;
    size = 0.f;
    inexact = false;
  }
  __device__ __forceinline__ void add(int exponent, float term) {
    const uint32_t u = __float_as_uint(term);
    const int shift = static_cast<int>((u >> 23) & 0xFFu) - exponent;
    inexact = inexact || static_cast<unsigned>(shift) > 29u;
    const int mantissa = static_cast<int>((u & 0x007fffffu) | 0x00800000u);
    const int power = 1 << (shift & 31);
    units += static_cast<long long>(mantissa) * static_cast<long long>((u >> 31) ? -power : power);
    size += fabsf(term);
  }
  // (a NaN size is not exact)
  __device__ __forceinline__ bool exact(const SumRange& R) const { return !inexact && size <= R.limit; }
  __device__ __forceinline__ double value(const SumRange& R) const {
    return __dmul_rn(static_cast<double>(units), R.quantum);
  }
};

// The packed residual fields as FP32 numbers (a 10-bit field, its sign bit
// flipped, under the exponent of 2^23): differences are exact, q_b - q_a for x
// and z, 1024 (q_b - q_a) for y.
__device__ __forceinline__ float field_x(uint32_t w) { return __uint_as_float((w & 0x3FFu) ^ 0x4B000200u); }
__device__ __forceinline__ float field_y(uint32_t w) { return __uint_as_float((w & 0xFFC00u) ^ 0x4B080000u); }
__device__ __forceinline__ float field_z(uint32_t w) { return __uint_as_float((w >> 20) ^ 0x4B000200u); }

// One axis of an image entry's displacement in FP32 pairs: hi_b - hi_a by
// TwoDiff (Knuth), the image offset added to its high part (exact: the two are
// within a factor of two of each other), the small parts summed. The rounded
// sum is the FP64 displacement's FP32 rounding unless its remainder lies within
// `tie` (the bound on both errors) of half an ulp: those entries take FP64.
__device__ __forceinline__ float image_axis(float hb, float ha, float lb, float la, uint32_t digit, float p, float pl,
                                            float tie, bool& sure) {
  const float s = __fadd_rn(hb, -ha);
  const float t = __fadd_rn(s, -hb);
  const float err = __fadd_rn(__fadd_rn(hb, -__fadd_rn(s, -t)), -__fadd_rn(ha, t));
  const float sh = digit == 1u ? 0.f : (digit == 2u ? p : -p), sl = digit == 1u ? 0.f : (digit == 2u ? pl : -pl);
  const float hi = __fadd_rn(s, sh);
  const float rest = __fadd_rn(__fadd_rn(err, sl), __fadd_rn(lb, -la));
  const float d = __fadd_rn(hi, rest);
  const float lo = __fadd_rn(__fadd_rn(hi, -d), rest);
  const uint32_t ex = __float_as_uint(d) & 0x7f800000u;
  const float half = __uint_as_float(ex - (24u << 23));  // half an ulp of d (ex checked below)
  sure = sure && ex > (40u << 23) && fabsf(__fadd_rn(fabsf(lo), -half)) > tie &&
         fabsf(__fadd_rn(fabsf(lo), -0.5f * half)) > tie;
  return d;
}

// One marked entry of the mixed path: r^2 in FP32 (the compensated mirror
// difference for an entry in the same periodic image: hi difference plus the
// difference of the residuals packed in .w; the FP64 displacement converted for
// an image entry), the cutoff decided in FP32 outside the proven band and in
// FP64 inside it, then the FP32 force factor pd and the FP64 accumulation of
// pd * r_b and pd.
// PACKED = false (batches holding a system of X >= 1024 sigma, whose packed
// residuals are too coarse) takes the gathered residual mirrors lb and pal.
template <bool PE, bool PACKED>
__device__ __forceinline__ void mixed_pair(const SysDesc& S, uint32_t e, double xb, double yb, double zb, float4 hb,
                                           float4 lb, double xa, double ya, double za, float4 paf, float4 pal,
                                           double rcut2, double& fx, double& fy, double& fz, double& psum,
                                           double& pe) {
  const uint32_t code = e & 31u;
  float dxf, dyf, dzf;
  if (code == static_cast<uint32_t>(kImageCenter)) {
    if constexpr (PACKED) {
      // within 2u|d| + 2 lo_step of the FP64 displacement (u = 2^-24), without FP64 work
      const uint32_t wb = __float_as_uint(hb.w), wa = __float_as_uint(paf.w);
      const float q = S.lo_step_f;
      dxf = fmaf(small_int_f(lo_field(wb, 0) - lo_field(wa, 0)), q, hb.x - paf.x);
      dyf = fmaf(small_int_f(lo_field(wb, 1) - lo_field(wa, 1)), q, hb.y - paf.y);
      dzf = fmaf(small_int_f(lo_field(wb, 2) - lo_field(wa, 2)), q, hb.z - paf.z);
    } else {
      // within 2u|d| of the FP64 displacement
      dxf = (hb.x - paf.x) + (lb.x - pal.x);
      dyf = (hb.y - paf.y) + (lb.y - pal.y);
      dzf = (hb.z - paf.z) + (lb.z - pal.z);
    }
  } else {
    xb = image_coord(xb, S.period[0], static_cast<int>(code % 3u));
    yb = image_coord(yb, S.period[1], static_cast<int>((code / 3u) % 3u));
    zb = image_coord(zb, S.period[2], static_cast<int>(code / 9u));
    dxf = narrow_f64(__dsub_rn(xb, xa));
    dyf = narrow_f64(__dsub_rn(yb, ya));
    dzf = narrow_f64(__dsub_rn(zb, za));
  }
  const float r2 = fmaf(dxf, dxf, fmaf(dyf, dyf, dzf * dzf));
  bool in;
  if (r2 > S.rc2_f + S.rc_margin_f) {
    in = false;
  } else if (r2 < S.rc2_f - S.rc_margin_f && r2 > S.rc_margin_f) {
    in = true;
  } else {
    const double d2 = norm2_rn(__dsub_rn(xb, xa), __dsub_rn(yb, ya), __dsub_rn(zb, za));
    in = (d2 > 0.0 && d2 <= rcut2);
  }
  if (in) {
    // FP64 displacement folded into the FP64 accumulation:
    //   sum_b pd_b (r_b - r_a) = sum_b pd_b r_b - r_a sum_b pd_b,
    // so a pair costs 3 DFMA + 1 DADD instead of 3 DADD + 3 DFMA; the
    // subtraction happens once per particle (cancellation error
    // <= ~u_64 |r| sum|pd|, about 1e-12 of |F| at box sizes of 10^3 sigma).
    // The hardware reciprocal (within 1 ulp) is part of the FP32 force magnitude.
    float ir2;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(ir2) : "f"(r2));
    const float s2 = S.sig2_f * ir2;
    const float s6 = s2 * s2 * s2;
    const float pd = S.eps24_f * s6 * fmaf(-2.0f, s6, 1.0f) * ir2;
    const double pdd = widen_f32_fast(pd);  // exact, on the integer pipes
    fx = fma(pdd, xb, fx);
    fy = fma(pdd, yb, fy);
    fz = fma(pdd, zb, fz);
    psum += pdd;
    if (PE) pe += widen_f32_fast(0.5f * fmaf(S.eps4_f * s6, s6 - 1.0f, -S.e_shift_f));
  }
}

// A particle's sums to its force (and energy): the FP64 displacement folded out
// of sum pd (r_b - r_a), the division by the mass, the second-half kick.
template <bool PE, bool KICK>
__device__ __forceinline__ void finish_mixed(const SysDesc& S, const DevArrays& a, uint32_t i, double fx, double fy,
                                             double fz, double psum, double pe) {
  fx = fma(-a.rx[i], psum, fx);
  fy = fma(-a.ry[i], psum, fy);
  fz = fma(-a.rz[i], psum, fz);
  if (S.divide_by_mass) {
    // divide_force_by_type_scalar (compute/vec3_typescalar_op.cu:156, math_functors.h:140)
    fx = __ddiv_rn(fx, S.mass);
    fy = __ddiv_rn(fy, S.mass);
    fz = __ddiv_rn(fz, S.mass);
  }
  a.fx[i] = fx;
  a.fy[i] = fy;
  a.fz[i] = fz;
  if (PE) a.pe[i] = pe;
  if (KICK) {
    // verlet_second_half: push_f_v with dt_scale 0.5 (numerical-scheme.msp:17-18)
    const double h = S.dt_half;
    a.vx[i] = fma(fx, h, a.vx[i]);
    a.vy[i] = fma(fy, h, a.vy[i]);
    a.vz[i] = fma(fz, h, a.vz[i]);
  }
}

// ---------------------------------------------------------------------------
// zero_particle_force + lennard_jones_force over the neighbour lists, as a
// functor of the pair-functor API (include/xnb_pair.cuh) run through the batch
// traversal. compute_cell_particle_pairs_cell (compute/include/exanb/compute/
// compute_cell_particle_pairs_impl_default.h:148-238) walks each particle's
// stream in (cell_enc, p_b) order with dr = r_b - r_a and keeps 0 < d2 <= rc^2;
// LennardJonesForceFunctor (contribs/md/lennard_jones/lennard_jones.cu:67-102)
// sums pair_de*dr sequentially and adds the sum onto the zeroed force.
// One thread per particle, full lists: no atomics, fixed summation order. The
// mixed path takes raw entries (the functor forms the displacement): FP64
// displacement and FP64 accumulation; r^2, r^-6 and the force magnitude in FP32;
// the cutoff decision is made in FP32 where a proven margin allows and in FP64
// otherwise, so the pair set is the FP64 one. The displacement is applied once
// per particle (sum pd*r_b - r_a*sum pd, all in FP64) and the FP32 factor is
// widened on the integer pipes: a pair costs 3 DFMA and 1 DADD on the FP64 pipe.
// (The FP64 paths: xnb_force_pairs.cuh; the common mixed batches, with these bits:
// xnb_force_mixed.cu.)
template <bool PE, bool KICK, bool PACKED = true>
struct LJForce {
  const SysDesc* __restrict__ sys;
  DevArrays a;
  struct Acc {
    double fx, fy, fz, psum, pe;
  };

  __device__ __forceinline__ double rcut2(const pair::ParticleContext& c) const { return sys[c.sys].rcut2; }
  __device__ __forceinline__ float prefilter_hi(const pair::ParticleContext& c) const {
    const SysDesc& S = sys[c.sys];
    return S.rc2_f + S.pre_margin_f;
  }
  __device__ __forceinline__ bool start(Acc& q, const pair::ParticleContext&) const {
    q.fx = q.fy = q.fz = q.psum = q.pe = 0.0;
    return true;
  }
  __device__ __forceinline__ void entry(Acc& q, const pair::ParticleContext& c, const pair::RawEntry& r) const {
    const SysDesc& S = sys[c.sys];
    mixed_pair<PE, PACKED>(S, r.e, r.xb, r.yb, r.zb, r.hb, r.lb, c.x, c.y, c.z, c.hi, c.lo, S.rcut2, q.fx, q.fy,
                           q.fz, q.psum, q.pe);
  }
  __device__ __forceinline__ void combine(Acc& q, const Acc& o) const {
    q.fx += o.fx;
    q.fy += o.fy;
    q.fz += o.fz;
    q.psum += o.psum;
    q.pe += o.pe;
  }
  __device__ __forceinline__ void stop(Acc& q, const pair::ParticleContext& c) const {
    finish_mixed<PE, KICK>(sys[c.sys], a, c.i, q.fx, q.fy, q.fz, q.psum, q.pe);
  }
};

}  // namespace xnb

namespace xnb {
namespace pair {
// Raw entries (their residuals come packed with the hi mirror, so the residual
// mirrors are gathered only without packing), two per iteration (both entries'
// gathers in flight together; list order unchanged).
template <bool PE, bool KICK, bool PACKED>
struct ComputePairTraits<LJForce<PE, KICK, PACKED>> : DefaultPairTraits {
  static constexpr bool RawEntries = true;
  static constexpr bool GatherMirrors = !PACKED;
  static constexpr int EntriesPerIteration = 2;
};
}  // namespace pair
}  // namespace xnb
