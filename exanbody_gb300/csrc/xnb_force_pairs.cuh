// Full-precision Lennard-Jones forces, a warp per eight particles.
//
// The FP64 pipe takes one warp instruction per 64 cycles from each quarter of an
// SM whatever its lanes do, so what counts is how few FP64 instructions carry
// the pairs and how full they are. One thread per particle ran the pair body as
// often as the warp's busiest lane had marked entries (86% of the lanes in use)
// and, for batches too small to fill the GPU, waited for every pair's gathers.
//   Stage 1 (FP32): the warp filters one particle's list at a time, up to 96
//     entries in flight, against rc^2 plus the proven FP32 error bound; ballots
//     append the entries to the particle's row in shared memory, in list order.
//     Entries inside the band around rc^2 carry a flag. Short lists (the eight hold
//     at most 96 entries) are filtered at once, a lane per entry: with one list at
//     a time forces below a density of 0.1 were slower than by one thread per
//     particle (953,312 atoms, kFp64 / Newton, at 0.02: 187 / 207 us by one thread
//     per particle, 320 / 294 one list at a time, 188 / 204 now; at 0.05: 325 / 345,
//     371 / 348 and 268 / 224).
//   Stage 2 (FP64), kFp64: four lanes per particle take every fourth of its pairs,
//     18 FP64 instructions each (24 with the exact d2, a reciprocal of two Newton
//     steps and a compare per pair); flagged entries take the reference's d2 test
//     first. The order of a particle's sums follows from its own list alone, so a
//     system's forces are the same bits whatever else the batch holds.
//     Half lists (NEWTON), whose lengths differ more and whose reactions arrive in
//     any order anyway: the rows of the eight particles lie one after the other
//     and every lane takes an equal run of pairs. Where a run passes from one
//     particle to the next the sums so far are put down; each particle's few
//     pieces are then added in order.
//   kFp64Exact: the functor's own operations and roundings, four lanes per
//     particle; a 4 x 4 transpose hands each lane one component of four
//     consecutive pairs, which it adds in list order: the bits of the sequential
//     walk.
// The FP64 pipe is busy 85% of the time (kFp64, 119,164 atoms: 422 us with one
// thread per particle, 280 now; 282 with equal runs of the eight particles' pairs
// for full lists too, whose rounds are not those of the longest of eight lists but
// whose ends cost as much; at density 0.35, 953,312 atoms, 1,181, 875 and 822 us).
// Newton half lists, 5 steps of 256,000 atoms: 3.94 -> 1.89 ms; kFp64Exact, 5
// host-synchronised steps of 8,788 atoms: 767 -> 424 us.
#pragma once

#include "xnb_lj_pair.cuh"
#include "xnb_traverse.cuh"

namespace xnb {
namespace pairs {

constexpr uint32_t kPer = 8;             // particles per warp
constexpr uint32_t kChunk = 96;          // list entries filtered per round
constexpr uint32_t kRow = kChunk + 1;    // full lists: odd, the rows start on different banks
constexpr uint32_t kCheck = 0x80000000u; // entry inside the FP32 band (list entries stay below 2^31)

// A warp's shared memory.
struct WarpSmem {
  double pos[kPer][3];          // the particles
  double piece[32 + kPer][4];   // half lists: piece (lane, particle) at lane + particle, unique along the runs
  uint32_t row[kPer * kRow];
  uint32_t start[kPer + 1];     // half lists: first pair of each particle
  uint32_t sys[kPer];
};

// 1/d from the FP32 seed of rcp_nr (within 2^-22) and one third-order step:
// y (1 + e + e^2), e = 1 - d y, is within 2^-66 before its rounding.
__device__ __forceinline__ double reciprocal(double d) {
  const int hi = min(max(__double2hiint(d) - 0x38000000, 0x00100000), 0x0fcfffff);
  const float s = __uint_as_float(__funnelshift_l(static_cast<uint32_t>(__double2loint(d)), static_cast<uint32_t>(hi), 3));
  float rf;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rf) : "f"(s));
  const uint32_t r = __float_as_uint(rf);
  const double y = __hiloint2double(static_cast<int>((r >> 3) + 0x38000000u), static_cast<int>(r << 29));
  const double e = fma(-d, y, 1.0);
  return fma(y, fma(e, e, e), y);
}

__device__ __forceinline__ double shfl_xor(double v, int mask) { return __shfl_xor_sync(0xffffffffu, v, mask); }

// Entry e, whose particle's mirror is hb, of a particle at o: false when it is surely
// beyond the cutoff, and e marked when FP32 does not decide.
__device__ __forceinline__ bool filter(const SysDesc& S, uint32_t& e, float4 hb, float ox, float oy, float oz) {
  const float r2_out = S.rc2_f + S.pre_margin_f, r2_in = S.rc2_f - S.pre_margin_f, r2_min = S.pre_margin_f;
  const uint32_t code = e & 31u;
  if (code != static_cast<uint32_t>(kImageCenter)) {
    hb.x = image_coord_f(hb.x, S.period_f[0], static_cast<int>(code % 3u));
    hb.y = image_coord_f(hb.y, S.period_f[1], static_cast<int>((code / 3u) % 3u));
    hb.z = image_coord_f(hb.z, S.period_f[2], static_cast<int>(code / 9u));
  }
  const float dx = hb.x - ox, dy = hb.y - oy, dz = hb.z - oz;
  const float d2 = fmaf(dx, dx, fmaf(dy, dy, dz * dz));
  e |= d2 < r2_in && d2 > r2_min ? 0u : kCheck;
  return d2 <= r2_out;
}

// Bits of the 32 from `base` on that lie below `end`.
__device__ __forceinline__ unsigned below(uint32_t end, uint32_t base) {
  return end <= base ? 0u : (end - base >= 32u ? 0xffffffffu : (1u << (end - base)) - 1u);
}

// Forces (and energies) of particles first .. first + 7; every lane of the warp
// calls. NEWTON (kFp64): the lower half of each list, the reactions and the
// particle's own sum by FP64 reductions into cleared fields.
template <int P, bool PE, bool KICK, bool NEWTON>
__device__ __forceinline__ void eight_particles(uint32_t first, uint32_t n_part, const BatchSource& src,
                                                const DevArrays& a, WarpSmem& sm) {
  const uint32_t lane = threadIdx.x & 31u, mine = lane >> 2, sub = lane & 3u;
  const unsigned full = 0xffffffffu, lt = (1u << lane) - 1u;
  const uint32_t i = first + mine;
  uint32_t s = 0, n = 0;
  const uint32_t* list = nullptr;
  const bool ok = i < n_part && src.locate(i, s, list, n);
  if (!ok) n = 0;
  if (NEWTON && ok) n = src.nbr_half[i];
  const float4 own = ok ? src.pf[i] : make_float4(0.f, 0.f, 0.f, 0.f);
  __syncwarp();  // the previous group's readers are done
  if (ok && sub < 3u) sm.pos[mine][sub] = (sub == 0u ? src.rx : (sub == 1u ? src.ry : src.rz))[i];
  if (sub == 3u) sm.sys[mine] = s;
  const SysDesc& S = src.sys[s];
  const uint32_t longest = __reduce_max_sync(full, n);
  uint32_t off = n;  // entries of the particles before `mine`
#pragma unroll
  for (int d = 4; d < 32; d <<= 1) {
    const uint32_t v = __shfl_up_sync(full, off, d);
    if (lane >= static_cast<uint32_t>(d)) off += v;
  }
  const uint32_t entries = __shfl_sync(full, off, 31);
  off -= n;
  double sum = 0.0;  // component `sub` of particle `mine`
  double part[4] = {0.0, 0.0, 0.0, 0.0};  // kFp64, full lists: the components over this lane's pairs

  for (uint32_t kb = 0; kb < longest; kb += kChunk) {
    // ---- stage 1 ----
    uint32_t count = 0, total = 0, row0 = mine * kRow;
    if (entries <= kChunk) {
      // short lists: all eight at once
      unsigned kept[3] = {0u, 0u, 0u};
#pragma unroll
      for (uint32_t t = 0; t < 3u; ++t) {
        if (32u * t >= entries) break;
        const uint32_t f = 32u * t + lane;
        int p = 0;  // f's particle: the last that starts at or before it
#pragma unroll
        for (int step = 4; step > 0; step >>= 1) {
          const uint32_t o = __shfl_sync(full, off, 4 * (p + step));
          if (o <= f) p += step;
        }
        const int from = 4 * p;
        const uint32_t k = f - __shfl_sync(full, off, from);
        const uint32_t* L = reinterpret_cast<const uint32_t*>(
            __shfl_sync(full, reinterpret_cast<unsigned long long>(list), from));
        const SysDesc& T = src.sys[__shfl_sync(full, s, from)];
        const float ox = __shfl_sync(full, own.x, from), oy = __shfl_sync(full, own.y, from),
                    oz = __shfl_sync(full, own.z, from);
        uint32_t e = 0;
        bool keep = false;
        if (f < entries) {
          e = __ldg(L + k);
          const float4 hb = src.pf[T.part_base + (e >> 5)];
          keep = filter(T, e, hb, ox, oy, oz);
        }
        kept[t] = __ballot_sync(full, keep);
        if (keep) sm.row[total + __popc(kept[t] & lt)] = e;
        total += __popc(kept[t]);
      }
      // entries kept before the particle's first, and before its end
      row0 = 0;
      uint32_t end = 0;
#pragma unroll
      for (uint32_t t = 0; t < 3u; ++t) {
        row0 += __popc(kept[t] & below(off, 32u * t));
        end += __popc(kept[t] & below(off + n, 32u * t));
      }
      count = end - row0;
      if (NEWTON && sub == 0) sm.start[mine] = row0;
    } else {
      for (uint32_t p = 0; p < kPer; ++p) {
        const int from = static_cast<int>(4u * p);
        const uint32_t np = __shfl_sync(full, n, from);
        if (NEWTON && lane == 0) sm.start[p] = total;
        if (np <= kb) continue;
        const uint32_t* L = reinterpret_cast<const uint32_t*>(
            __shfl_sync(full, reinterpret_cast<unsigned long long>(list), from));
        const SysDesc& T = src.sys[__shfl_sync(full, s, from)];
        const float ox = __shfl_sync(full, own.x, from), oy = __shfl_sync(full, own.y, from),
                    oz = __shfl_sync(full, own.z, from);
        const uint32_t base = T.part_base, left = np - kb;
        uint32_t e[3];
        float4 hb[3];
#pragma unroll
        for (uint32_t t = 0; t < 3u; ++t) e[t] = 32u * t + lane < left ? __ldg(L + kb + 32u * t + lane) : 0xFFFFFFFFu;
#pragma unroll
        for (uint32_t t = 0; t < 3u; ++t)
          hb[t] = e[t] != 0xFFFFFFFFu ? src.pf[base + (e[t] >> 5)] : make_float4(1.0e18f, 0.f, 0.f, 0.f);
        uint32_t* const out = sm.row + (NEWTON ? total : p * kRow);
        uint32_t c = 0;
#pragma unroll
        for (uint32_t t = 0; t < 3u; ++t) {
          const bool keep = e[t] != 0xFFFFFFFFu && filter(T, e[t], hb[t], ox, oy, oz);
          const unsigned m = __ballot_sync(full, keep);
          if (keep) out[c + __popc(m & lt)] = e[t];
          c += __popc(m);
        }
        if (mine == p) count = c;
        total += c;
      }
    }
    if (NEWTON && lane == 0) sm.start[kPer] = total;
    __syncwarp();
    // ---- stage 2 ----
    if constexpr (NEWTON) {
      const uint32_t run = (total + 31u) >> 5;
      const uint32_t f0 = min(total, lane * run), f1 = min(total, f0 + run);
      uint32_t p = 0, end = 0, pbase = 0, e = 0;
      double xa = 0.0, ya = 0.0, za = 0.0, sig2 = 0.0, pd_a = 0.0, pd_b = 0.0;
      double fx = 0.0, fy = 0.0, fz = 0.0, pe = 0.0, xb = 0.0, yb = 0.0, zb = 0.0;
      const SysDesc* T = src.sys;
      // the particle that pair f belongs to, from p on
      auto enter = [&](uint32_t f) {
        while (f >= sm.start[p + 1]) ++p;
        end = sm.start[p + 1];
        xa = sm.pos[p][0];
        ya = sm.pos[p][1];
        za = sm.pos[p][2];
        T = src.sys + sm.sys[p];
        pbase = T->part_base;
        sig2 = T->sig2;
        pd_a = T->pd_a;
        pd_b = T->pd_b;
        fx = fy = fz = pe = 0.0;
      };
      auto put = [&]() {
        double* const o = sm.piece[lane + p];
        o[0] = fx;
        o[1] = fy;
        o[2] = fz;
        if (PE) o[3] = pe;
      };
      // the next pair's coordinates load while this one is evaluated (a run
      // crosses systems only between particles: the entry's own particle decides)
      auto fetch = [&](uint32_t f) {
        e = sm.row[f];
        uint32_t base = pbase;
        if (f >= end) {
          uint32_t q = p;
          while (f >= sm.start[q + 1]) ++q;
          base = src.sys[sm.sys[q]].part_base;
        }
        const uint32_t j = base + ((e & ~kCheck) >> 5);
        xb = src.rx[j];
        yb = src.ry[j];
        zb = src.rz[j];
      };
      if (f0 < f1) {
        enter(f0);
        fetch(f0);
      }
      for (uint32_t f = f0; f < f1; ++f) {
        if (f >= end) {
          put();
          enter(f);
        }
        const uint32_t w = e, code = w & 31u;
        double x = xb, y = yb, z = zb;
        if (f + 1u < f1) fetch(f + 1u);
        if (code != static_cast<uint32_t>(kImageCenter)) {
          const uint32_t cx = code % 3u, cy = (code / 3u) % 3u, cz = code / 9u;
          if (cx != 1u) x = __dadd_rn(x, cx == 2u ? T->period[0] : -T->period[0]);
          if (cy != 1u) y = __dadd_rn(y, cy == 2u ? T->period[1] : -T->period[1]);
          if (cz != 1u) z = __dadd_rn(z, cz == 2u ? T->period[2] : -T->period[2]);
        }
        const double dx = __dsub_rn(x, xa), dy = __dsub_rn(y, ya), dz = __dsub_rn(z, za);
        bool in = true;
        if (w & kCheck) {
          const double d2 = norm2_rn(dx, dy, dz);
          in = d2 > 0.0 && d2 <= T->rcut2;
        }
        if (in) {
          const double s2 = sig2 * reciprocal(fma(dx, dx, fma(dy, dy, dz * dz)));
          const double s6 = s2 * s2 * s2;
          // 24 eps / sigma^2 (1 - 2 s6) s6 s2
          const double pd = fma(pd_b, s6, pd_a) * s6 * s2;
          fx = fma(pd, dx, fx);
          fy = fma(pd, dy, fy);
          fz = fma(pd, dz, fz);
          double en = 0.0;
          if (PE) {
            en = 0.5 * fma(T->eps4 * s6, s6 - 1.0, -T->e_shift);
            pe += en;
          }
          const uint32_t j = pbase + ((w & ~kCheck) >> 5);
          atomicAdd(a.fx + j, -(pd * dx));
          atomicAdd(a.fy + j, -(pd * dy));
          atomicAdd(a.fz + j, -(pd * dz));
          if (PE) atomicAdd(a.pe + j, en);
        }
      }
      if (f0 < f1) put();
      __syncwarp();
      // the particle's pieces, in order
      const uint32_t p0 = sm.start[mine], p1 = sm.start[mine + 1];
      if (p0 < p1 && (PE || sub < 3u))
        for (uint32_t l = p0 / run; l <= (p1 - 1u) / run; ++l) sum += sm.piece[l + mine][sub];
    } else if constexpr (P == kFp64) {
      // four lanes per particle, each every fourth of its pairs
      const uint32_t* const row = sm.row + row0;
      const uint32_t pbase = S.part_base;
      const double xa = sm.pos[mine][0], ya = sm.pos[mine][1], za = sm.pos[mine][2];
      const double sig2 = S.sig2, pd_a = S.pd_a, pd_b = S.pd_b;
      uint32_t e = 0;
      double xb = 0.0, yb = 0.0, zb = 0.0;
      auto fetch = [&](uint32_t k) {
        if (k < count) {
          e = row[k];
          const uint32_t j = pbase + ((e & ~kCheck) >> 5);
          xb = src.rx[j];
          yb = src.ry[j];
          zb = src.rz[j];
        }
      };
      fetch(sub);
      for (uint32_t k = sub; k < count; k += 4u) {
        const uint32_t w = e, code = w & 31u;
        double x = xb, y = yb, z = zb;
        fetch(k + 4u);  // the next pair's coordinates while this one is evaluated
        if (code != static_cast<uint32_t>(kImageCenter)) {
          const uint32_t cx = code % 3u, cy = (code / 3u) % 3u, cz = code / 9u;
          if (cx != 1u) x = __dadd_rn(x, cx == 2u ? S.period[0] : -S.period[0]);
          if (cy != 1u) y = __dadd_rn(y, cy == 2u ? S.period[1] : -S.period[1]);
          if (cz != 1u) z = __dadd_rn(z, cz == 2u ? S.period[2] : -S.period[2]);
        }
        const double dx = __dsub_rn(x, xa), dy = __dsub_rn(y, ya), dz = __dsub_rn(z, za);
        if (w & kCheck) {
          const double d2 = norm2_rn(dx, dy, dz);
          if (!(d2 > 0.0 && d2 <= S.rcut2)) continue;
        }
        const double s2 = sig2 * reciprocal(fma(dx, dx, fma(dy, dy, dz * dz)));
        const double s6 = s2 * s2 * s2;
        // 24 eps / sigma^2 (1 - 2 s6) s6 s2
        const double pd = fma(pd_b, s6, pd_a) * s6 * s2;
        part[0] = fma(pd, dx, part[0]);
        part[1] = fma(pd, dy, part[1]);
        part[2] = fma(pd, dz, part[2]);
        if (PE) part[3] += 0.5 * fma(S.eps4 * s6, s6 - 1.0, -S.e_shift);
      }
    } else {
      const uint32_t* const row = sm.row + row0;
      const uint32_t rounds = (__reduce_max_sync(full, count) + 3u) >> 2, pbase = S.part_base;
      const double xa = sm.pos[mine][0], ya = sm.pos[mine][1], za = sm.pos[mine][2];
      uint32_t e = 0;
      double xb = 0.0, yb = 0.0, zb = 0.0;
      auto fetch = [&](uint32_t k) {
        if (k < count) {
          e = row[k];
          const uint32_t j = pbase + ((e & ~kCheck) >> 5);
          xb = src.rx[j];
          yb = src.ry[j];
          zb = src.rz[j];
        }
      };
      fetch(sub);
      for (uint32_t r = 0; r < rounds; ++r) {
        const uint32_t k = 4u * r + sub;
        const uint32_t w = e, code = w & 31u;
        double x = xb, y = yb, z = zb;
        fetch(k + 4u);  // the next pair's coordinates while this one is evaluated
        double g[4] = {0.0, 0.0, 0.0, 0.0};
        if (k < count) {
          if (code != static_cast<uint32_t>(kImageCenter)) {
            const uint32_t cx = code % 3u, cy = (code / 3u) % 3u, cz = code / 9u;
            if (cx != 1u) x = __dadd_rn(x, cx == 2u ? S.period[0] : -S.period[0]);
            if (cy != 1u) y = __dadd_rn(y, cy == 2u ? S.period[1] : -S.period[1]);
            if (cz != 1u) z = __dadd_rn(z, cz == 2u ? S.period[2] : -S.period[2]);
          }
          const double dx = __dsub_rn(x, xa), dy = __dsub_rn(y, ya), dz = __dsub_rn(z, za);
          const double d2 = norm2_rn(dx, dy, dz);
          if (!(w & kCheck) || (d2 > 0.0 && d2 <= S.rcut2)) {
            // lj_compute_energy (lennard_jones.cu:46-56) then pair_de *= w / r with w = 1
            const double rr = __dsqrt_rn(d2);
            const double inv_r = __drcp_rn(rr);  // the rounded 1 / r, without the division's quotient steps
            const double ratio = __dmul_rn(S.sigma, inv_r);
            const double ratio2 = __dmul_rn(ratio, ratio);
            const double ratio6 = __dmul_rn(__dmul_rn(ratio2, ratio2), ratio2);
            const double ratio12 = __dmul_rn(ratio6, ratio6);
            // 2 ratio12 is exact: one rounding either way
            double de = __dmul_rn(__dmul_rn(S.m24eps, __fma_rn(2.0, ratio12, -ratio6)), inv_r);
            de = __dmul_rn(de, inv_r);
            g[0] = __dmul_rn(de, dx);
            g[1] = __dmul_rn(de, dy);
            g[2] = __dmul_rn(de, dz);
            if (PE) g[3] = __dmul_rn(0.5, __dsub_rn(__dmul_rn(S.eps4, __dsub_rn(ratio12, ratio6)), S.e_shift));
          }
        }
        // lane t holds pair t's components; after the transpose lane c holds component c of the four pairs
        const bool odd = (sub & 1u) != 0, high = (sub & 2u) != 0;
        double v = shfl_xor(odd ? g[0] : g[1], 1);
        if (odd) g[0] = v;
        else g[1] = v;
        v = shfl_xor(odd ? g[2] : g[3], 1);
        if (odd) g[2] = v;
        else g[3] = v;
        v = shfl_xor(high ? g[0] : g[2], 2);
        if (high) g[0] = v;
        else g[2] = v;
        v = shfl_xor(high ? g[1] : g[3], 2);
        if (high) g[1] = v;
        else g[3] = v;
        // zero terms leave the sum as it is (it is never -0)
#pragma unroll
        for (int t = 0; t < 4; ++t) sum = __dadd_rn(sum, g[t]);
      }
    }
    __syncwarp();  // the rows are refilled for the next round
  }

  if (P == kFp64 && !NEWTON) {
    // component c of the four lanes meets in lane c: (0 + 1) + (2 + 3)
    const bool odd = (sub & 1u) != 0, high = (sub & 2u) != 0;
    const double lo = (odd ? part[1] : part[0]) + shfl_xor(odd ? part[0] : part[1], 1);
    const double hi = (odd ? part[3] : part[2]) + shfl_xor(odd ? part[2] : part[3], 1);
    sum = (high ? hi : lo) + shfl_xor(high ? lo : hi, 2);
  }
  const uint32_t ax = sub;
  double v = sum;
  if (!ok || (!PE && ax == 3u)) return;
  double* const f = ax == 0u ? a.fx : (ax == 1u ? a.fy : (ax == 2u ? a.fz : a.pe));
  // (energies, and reductions, are stored as they are)
  if (NEWTON) {
    atomicAdd(f + i, v);
    return;
  }
  if (ax == 3u) {
    f[i] = v;
    return;
  }
  // the force field was zeroed (zero_particle_force.cu:39-46) and receives the sum
  if (P == kFp64Exact) v = __dadd_rn(0.0, v);
  // divide_force_by_type_scalar (compute/vec3_typescalar_op.cu:156, math_functors.h:140)
  if (S.divide_by_mass) v = __ddiv_rn(v, S.mass);
  f[i] = v;
  if (KICK) {
    // verlet_second_half: push_f_v with dt_scale 0.5 (numerical-scheme.msp:17-18)
    double* const vel = ax == 0u ? a.vx : (ax == 1u ? a.vy : a.vz);
    vel[i] = P == kFp64Exact ? __dadd_rn(vel[i], __dmul_rn(v, S.dt_half)) : fma(v, S.dt_half, vel[i]);
  }
}

}  // namespace pairs
}  // namespace xnb
