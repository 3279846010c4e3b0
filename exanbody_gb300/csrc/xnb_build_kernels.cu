// Rebuild-path kernels: move/rebin with periodic wrap, AMR in-cell ordering,
// backup_r, and the cell-grid neighbour build; plus the device scan they use.
#include <algorithm>

#include "xnb_build_common.cuh"
#include "xnb_grid_barrier.cuh"
#include "xnb_launch.cuh"

namespace xnb {

namespace {

using namespace build;
constexpr uint32_t kMoverBit = 0x80000000u;


// sub_grid_size (amr/include/exanb/amr/amr_grid_algorithm.h:66-78): the largest
// side s with s^3 <= n/density (1 below side 2, capped at 16), computed from the
// same double n/density the reference feeds to cbrt.
__device__ __forceinline__ int sub_grid_side(uint32_t n, double density) {
  if (n == 0) return 0;
  const double x = __ddiv_rn(static_cast<double>(n), density);
  if (x < 8.0) return 1;
  int s = 2;
  while (s < 16 && static_cast<double>((s + 1) * (s + 1) * (s + 1)) <= x) ++s;
  return s;
}

// ---------------------------------------------------------------------------
// K_r1: destination cell of each particle of a rebuilding system.
// move_particles_across_cells (grid_cell_particles/include/exanb/grid_cell_particles/
// move_particles_across_cells.h:115-152): dst = domain_periodic_location(r)
// (core/include/exanb/core/domain.h:160-191, wrapping r by whole cells), and the
// particle leaves its cell when dst differs or it lies >= epsilon outside dst's bounds.
__device__ __forceinline__ void rebin_dest(uint32_t n_part, const SysDesc* __restrict__ sys, SysState* st,
                                           const DevArrays& a) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_part; i += gridDim.x * blockDim.x) {
    const uint32_t c = a.pcell[i];
    if (c == kInvalid) continue;
    const uint32_t s = a.cell_sys[c];
    if (!sys_flagged(st, s)) continue;
    const SysDesc& S = sys[s];
    int ci, cj, ck;
    cell_ijk(S, c - S.cell_base, ci, cj, ck);
    {
      // FP32 pre-decision from the position mirror: a particle whose quotient lies
      // farther than q_margin_f from a cell boundary, inside the grid, gets the
      // reference's cell without the FP64 division, and lies strictly inside it
      // (distance to the cell bounds 0, no wrapping).
      const float4 pq = a.pf[i];
      const float qv[3] = {pq.x * S.inv_cell_f, pq.y * S.inv_cell_f, pq.z * S.inv_cell_f};
      int lf[3];
      bool sure = true;
      for (int ax = 0; ax < 3; ++ax) {
        const float fl = floorf(qv[ax]);
        const float fr = qv[ax] - fl;
        sure = sure && fr > S.q_margin_f && fr < 1.0f - S.q_margin_f && fl >= 0.0f &&
               fl < static_cast<float>(S.dims[ax]);
        lf[ax] = static_cast<int>(fl);
      }
      if (sure) {
        if (lf[0] == ci && lf[1] == cj && lf[2] == ck) {
          a.pdest[i] = c;
        } else {
          const int dd[3] = {pmod_i(lf[0] - ci, S.dims[0]), pmod_i(lf[1] - cj, S.dims[1]),
                             pmod_i(lf[2] - ck, S.dims[2])};
          for (int ax = 0; ax < 3; ++ax)
            if (!(dd[ax] == 0 || dd[ax] == 1 || dd[ax] == S.dims[ax] - 1)) atomicOr(&st[s].error, kErrFarMover);
          a.pdest[i] = (S.cell_base + static_cast<uint32_t>((lf[2] * S.dims[1] + lf[1]) * S.dims[0] + lf[0])) |
                       kMoverBit;
        }
        continue;
      }
    }
    const double ro[3] = {a.rx[i], a.ry[i], a.rz[i]};
    double r[3] = {ro[0], ro[1], ro[2]};
    int loc[3];
    bool bad = false;
    for (int ax = 0; ax < 3; ++ax) {
      const double rel = __dsub_rn(r[ax], S.origin[ax]);
      const double q = floor(__ddiv_rn(rel, S.cell_size));
      if (!(fabs(q) < 1.0e9)) {
        bad = true;
        loc[ax] = 0;
        continue;
      }
      int l = static_cast<int>(q);
      if (l < 0 || l >= S.dims[ax]) {
        const int old = l;
        l = pmod_i(l, S.dims[ax]);
        r[ax] = __dadd_rn(r[ax], __dmul_rn(static_cast<double>(l - old), S.cell_size));
      }
      loc[ax] = l;
    }
    if (bad) {
      atomicOr(&st[s].error, kErrCellIndex);
      a.pdest[i] = c;
      continue;
    }
    // min_distance2_between(ro, cell_bounds(dst)) >= epsilon_cell_size2 (grid.h:60,89-90; geometry.h:137-153)
    double d[3];
    for (int ax = 0; ax < 3; ++ax) {
      const double lo = cell_lo(S, ax, loc[ax]);
      const double hi = cell_lo(S, ax, loc[ax] + 1);
      d[ax] = 0.0;
      if (ro[ax] < lo) d[ax] = __dsub_rn(lo, ro[ax]);
      else if (ro[ax] > hi) d[ax] = __dsub_rn(ro[ax], hi);
    }
    const double md2 = norm2_rn(d[0], d[1], d[2]);
    const double eps = __dmul_rn(0x1p-48, S.cell_size);
    const bool same = (loc[0] == ci && loc[1] == cj && loc[2] == ck);
    const bool mover = !same || md2 >= __dmul_rn(eps, eps);
    const uint32_t dst = S.cell_base + static_cast<uint32_t>((loc[2] * S.dims[1] + loc[1]) * S.dims[0] + loc[0]);
    if (mover) {
      // arrivals are gathered from the 26 neighbouring cells only
      const int dd[3] = {pmod_i(loc[0] - ci, S.dims[0]), pmod_i(loc[1] - cj, S.dims[1]), pmod_i(loc[2] - ck, S.dims[2])};
      for (int ax = 0; ax < 3; ++ax)
        if (!(dd[ax] == 0 || dd[ax] == 1 || dd[ax] == S.dims[ax] - 1)) atomicOr(&st[s].error, kErrFarMover);
      a.rx[i] = r[0];
      a.ry[i] = r[1];
      a.rz[i] = r[2];
    }
    a.pdest[i] = mover ? (dst | kMoverBit) : c;
  }
}
__global__ void __launch_bounds__(256)
    k_rebin_dest(uint32_t n_part, const SysDesc* __restrict__ sys, SysState* st, DevArrays a) {
  if (*a.any_rebuild == 0) return;
  rebin_dest(n_part, sys, st, a);
}

// ---------------------------------------------------------------------------
// K_r2: per source cell, compaction of the staying particles and list of movers.
// The hole left by a mover is filled with the current last particle, scanning
// from the top (move_particles_across_cells.h:186-207).
__device__ __forceinline__ void rebin_compact(uint32_t n_cells, const SysDesc* __restrict__ sys, const SysState* st,
                                              const DevArrays& a) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < n_cells; c += warps) {
    const uint32_t s = a.cell_sys[c];
    if (s == kInvalid || !sys_flagged(st, s)) continue;
    const uint32_t start = a.cell_start[c];
    const uint32_t n = a.cell_n[c];
    // movers, in particle order, via ballots
    uint32_t nmov = 0;
    for (uint32_t q0 = 0; q0 < n; q0 += 32) {
      const uint32_t q = q0 + lane;
      const bool mv = q < n && (a.pdest[start + q] & kMoverBit);
      const unsigned m = __ballot_sync(0xffffffffu, mv);
      if (mv) a.mover_list[start + nmov + __popc(m & lanemask_lt())] = start + q;
      if (q < n) a.plocal[start + q] = mv ? kInvalid : q;
      nmov += __popc(m);
    }
    __syncwarp();
    if (lane == 0) {
      // the holes from the top (only they matter to the scan)
      uint32_t ncur = n;
      for (uint32_t m = nmov; m-- > 0;) {
        const uint32_t q = a.mover_list[start + m] - start;
        if (q + 1 < ncur) a.plocal[start + q] = a.plocal[start + ncur - 1];
        --ncur;
      }
      a.cell_stay[c] = ncur;
      a.cell_nmov[c] = nmov;
    }
  }
}
__global__ void __launch_bounds__(128)
    k_rebin_compact(uint32_t n_cells, const SysDesc* __restrict__ sys, const SysState* st, DevArrays a) {
  if (*a.any_rebuild == 0) return;
  rebin_compact(n_cells, sys, st, a);
}

// The (up to) 27 source cells around destination cell c, sorted by global cell
// index, duplicates removed: arrivals are appended in (source cell, source
// index) order, the order one thread of the reference's OpenMP loop produces.
struct SrcInfo {
  uint32_t src;    // source cell (kInvalid if unused / duplicate)
  uint32_t rank;   // position in sorted order
  uint32_t count;  // movers from src into c
  uint32_t offset; // exclusive prefix of counts in sorted order
};

__device__ __forceinline__ SrcInfo arrivals_of(const SysDesc& S, const DevArrays& a, uint32_t c, uint32_t lane) {
  int ci, cj, ck;
  cell_ijk(S, c - S.cell_base, ci, cj, ck);
  uint32_t src = kInvalid;
  if (lane < 27) {
    const int di = static_cast<int>(lane % 3) - 1, dj = static_cast<int>((lane / 3) % 3) - 1,
              dk = static_cast<int>(lane / 9) - 1;
    const int ni = pmod_i(ci + di, S.dims[0]), nj = pmod_i(cj + dj, S.dims[1]), nk = pmod_i(ck + dk, S.dims[2]);
    src = S.cell_base + static_cast<uint32_t>((nk * S.dims[1] + nj) * S.dims[0] + ni);
  }
  uint32_t rank = 0;
  bool dup = false;
  for (uint32_t m = 0; m < 27; ++m) {
    const uint32_t o = __shfl_sync(0xffffffffu, src, m);
    if (lane < 27) {
      if (o < src) ++rank;
      if (o == src && m < lane) dup = true;
    }
  }
  uint32_t count = 0;
  if (lane < 27 && !dup) {
    const uint32_t st0 = a.cell_start[src];
    const uint32_t nm = a.cell_nmov[src];
    for (uint32_t m = 0; m < nm; ++m) {
      const uint32_t p = a.mover_list[st0 + m];
      if ((a.pdest[p] & ~kMoverBit) == c) ++count;
    }
  }
  if (dup) src = kInvalid;
  // offset = sum of counts of lanes with smaller rank
  uint32_t offset = 0;
  for (uint32_t m = 0; m < 27; ++m) {
    const uint32_t rm = __shfl_sync(0xffffffffu, rank, m);
    const uint32_t cm = __shfl_sync(0xffffffffu, count, m);
    if (rm < rank) offset += cm;
  }
  return SrcInfo{src, rank, count, offset};
}

// K_r3: new particle count of every cell (flagged systems: stayers + arrivals).
__device__ __forceinline__ void rebin_count(uint32_t n_cells, const SysDesc* __restrict__ sys, const SysState* st,
                                            const DevArrays& a) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < n_cells; c += warps) {
    const uint32_t s = a.cell_sys[c];
    if (s == kInvalid) {
      if (lane == 0) a.cell_cnt[c] = 0;
      continue;
    }
    if (!sys_flagged(st, s)) {
      if (lane == 0) a.cell_cnt[c] = a.cell_n[c];
      continue;
    }
    const SrcInfo si = arrivals_of(sys[s], a, c, lane);
    uint32_t tot = si.count;
    for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
    if (lane == 0) a.cell_cnt[c] = a.cell_stay[c] + tot;
  }
}
__global__ void __launch_bounds__(128)
    k_rebin_count(uint32_t n_cells, const SysDesc* __restrict__ sys, const SysState* st, DevArrays a) {
  if (*a.any_rebuild == 0) return;
  rebin_count(n_cells, sys, st, a);
}

// K_r5: gather stayers then arrivals of each destination cell into the scratch arrays.
__device__ __forceinline__ void rebin_scatter(uint32_t n_cells, const SysDesc* __restrict__ sys, const SysState* st,
                                              const DevArrays& a) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < n_cells; c += warps) {
    const uint32_t s = a.cell_sys[c];
    if (s == kInvalid || !sys_flagged(st, s)) continue;
    const SysDesc& S = sys[s];
    const uint32_t ns = S.part_base + static_cast<uint32_t>(a.cell_scan[c] - a.cell_scan[S.cell_base]);
    const uint32_t start = a.cell_start[c];
    const uint32_t stay = a.cell_stay[c];
    for (uint32_t q = lane; q < stay; q += 32) {
      const uint32_t src = start + a.plocal[start + q];
      const uint32_t dst = ns + q;
      a.t_rx[dst] = a.rx[src]; a.t_ry[dst] = a.ry[src]; a.t_rz[dst] = a.rz[src];
      a.t_vx[dst] = a.vx[src]; a.t_vy[dst] = a.vy[src]; a.t_vz[dst] = a.vz[src];
      a.t_fx[dst] = a.fx[src]; a.t_fy[dst] = a.fy[src]; a.t_fz[dst] = a.fz[src];
      a.t_id[dst] = a.id[src];
      a.t_ptype[dst] = a.ptype[src];
    }
    const SrcInfo si = arrivals_of(S, a, c, lane);
    if (si.src != kInvalid && si.count > 0) {
      const uint32_t st0 = a.cell_start[si.src];
      const uint32_t nm = a.cell_nmov[si.src];
      uint32_t k = 0;
      for (uint32_t m = 0; m < nm; ++m) {
        const uint32_t p = a.mover_list[st0 + m];
        if ((a.pdest[p] & ~kMoverBit) != c) continue;
        const uint32_t dst = ns + stay + si.offset + k++;
        a.t_rx[dst] = a.rx[p]; a.t_ry[dst] = a.ry[p]; a.t_rz[dst] = a.rz[p];
        a.t_vx[dst] = a.vx[p]; a.t_vy[dst] = a.vy[p]; a.t_vz[dst] = a.vz[p];
        a.t_fx[dst] = a.fx[p]; a.t_fy[dst] = a.fy[p]; a.t_fz[dst] = a.fz[p];
        a.t_id[dst] = a.id[p];
        a.t_ptype[dst] = a.ptype[p];
      }
    }
  }
}
__global__ void __launch_bounds__(128)
    k_rebin_scatter(uint32_t n_cells, const SysDesc* __restrict__ sys, const SysState* st, DevArrays a) {
  if (*a.any_rebuild == 0) return;
  rebin_scatter(n_cells, sys, st, a);
}

// backup_r of one particle (io/backup_r.cpp:56-79): its 32-bit encoding relative
// to the cell, and what that restores to. The FP64 and mixed step loops keep the
// position itself instead: their displacement trigger then differs from the
// reference's by the encoding's quantum (cell_size / 2^32) at most.
__device__ __forceinline__ void store_backup(const SysDesc& S, const DevArrays& a, uint32_t i, const double (&lo)[3],
                                             double x, double y, double z) {
  const uint32_t bx = encode_u32(x, lo[0], S.cell_size, S.inv_cell);
  const uint32_t by = encode_u32(y, lo[1], S.cell_size, S.inv_cell);
  const uint32_t bz = encode_u32(z, lo[2], S.cell_size, S.inv_cell);
  a.bkx[i] = bx;
  a.bky[i] = by;
  a.bkz[i] = bz;
  const double rx = restore_u32(bx, lo[0], S.cell_size);
  const double ry = restore_u32(by, lo[1], S.cell_size);
  const double rz = restore_u32(bz, lo[2], S.cell_size);
  a.rbx[i] = rx;
  a.rby[i] = ry;
  a.rbz[i] = rz;
  a.rbf[i] = make_pf(S, rx, ry, rz);
}

// K_r6: final in-cell order (rebuild_amr's stable sort by sub-cell,
// amr_grid_algorithm.h:131-374, when the cell is dense enough for a sub-grid),
// cell table update, and backup_r (io/backup_r.cpp:56-79): kBackupExact keeps
// the encoding (store_backup), kBackupPlain the position itself, both while the
// position is in registers; kBackupNone leaves it to backup_particles.
constexpr int kBackupNone = 0, kBackupExact = 1, kBackupPlain = 2;
template <int BACKUP>
__device__ __forceinline__ void rebin_finalize(uint32_t n_cells, const SysDesc* __restrict__ sys, SysState* st,
                                               const DevArrays& a) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t warps = gridDim.x * (blockDim.x >> 5);
  for (uint32_t c = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); c < n_cells; c += warps) {
    const uint32_t s = a.cell_sys[c];
    if (s == kInvalid || !sys_flagged(st, s)) continue;
    const SysDesc& S = sys[s];
    const uint32_t ns = S.part_base + static_cast<uint32_t>(a.cell_scan[c] - a.cell_scan[S.cell_base]);
    const uint32_t n = a.cell_cnt[c];
    int ci, cj, ck;
    // the FP64 division of sub_grid_side only for counts that can give a side > 1
    // (a warp-wide FP64 instruction costs the same for one lane as for 32)
    const int side = (S.amr_enabled && n >= S.amr_min_n) ? sub_grid_side(n, S.sub_grid_density) : 1;
    if (lane == 0) a.cside[c] = static_cast<uint8_t>(side);
    double lo[3];
    if (side > 1 || BACKUP == kBackupExact) {
      cell_ijk(S, c - S.cell_base, ci, cj, ck);
      lo[0] = cell_lo(S, 0, ci);
      lo[1] = cell_lo(S, 1, cj);
      lo[2] = cell_lo(S, 2, ck);
    }
    if (side > 1) {
      // sub-cell key of each particle (Grid::particle_pcoord, grid.h:184-190), kept in pdest
      for (uint32_t q = lane; q < n; q += 32) {
        const double r[3] = {a.t_rx[ns + q], a.t_ry[ns + q], a.t_rz[ns + q]};
        int key = 0;
        int sidx[3];
        for (int ax = 0; ax < 3; ++ax) {
          const double pc = __ddiv_rn(__dsub_rn(r[ax], lo[ax]), S.cell_size);
          long long v = __double2ll_rz(__dmul_rn(pc, static_cast<double>(side)));
          v = v < 0 ? 0 : (v > side - 1 ? side - 1 : v);
          sidx[ax] = static_cast<int>(v);
        }
        key = (sidx[2] * side + sidx[1]) * side + sidx[0];
        a.pdest[ns + q] = static_cast<uint32_t>(key);
      }
      __syncwarp();
      for (uint32_t q = lane; q < n; q += 32) {
        const uint32_t kq = a.pdest[ns + q];
        uint32_t rank = 0;
        for (uint32_t p = 0; p < n; ++p) {
          const uint32_t kp = a.pdest[ns + p];
          rank += (kp < kq) || (kp == kq && p < q);
        }
        a.plocal[ns + q] = rank;
      }
      __syncwarp();
    }
    for (uint32_t q = lane; q < n; q += 32) {
      const uint32_t src = ns + q;
      const uint32_t dst = ns + (side > 1 ? a.plocal[ns + q] : q);
      const double x = a.t_rx[src], y = a.t_ry[src], z = a.t_rz[src];
      a.rx[dst] = x; a.ry[dst] = y; a.rz[dst] = z;
      a.vx[dst] = a.t_vx[src]; a.vy[dst] = a.t_vy[src]; a.vz[dst] = a.t_vz[src];
      a.fx[dst] = a.t_fx[src]; a.fy[dst] = a.t_fy[src]; a.fz[dst] = a.t_fz[src];
      a.id[dst] = a.t_id[src];
      a.ptype[dst] = a.t_ptype[src];
      float4 mhi, mlo;
      make_pf2(S, x, y, z, mhi, mlo);
      a.pf[dst] = mhi;
      a.pflo[dst] = mlo;
      if (a.pstep) a.pstep[dst] = make_steps(x, y, z, mhi);
      if constexpr (BACKUP == kBackupExact) {
        store_backup(S, a, dst, lo, x, y, z);
      } else if constexpr (BACKUP == kBackupPlain) {
        a.rbx[dst] = x;
        a.rby[dst] = y;
        a.rbz[dst] = z;
        a.rbf[dst] = make_float4(mhi.x, mhi.y, mhi.z, 0.f);
      }
      a.pcell[dst] = c;
      if (side > 1) a.skey[dst] = static_cast<uint16_t>(a.pdest[src]);
    }
    if (lane == 0) {
      a.cell_start[c] = ns;
      a.cell_n[c] = n;
      atomicMax(&st[s].max_cell, n);
    }
  }
}
template <int BACKUP>
__global__ void __launch_bounds__(128)
    k_rebin_finalize(uint32_t n_cells, const SysDesc* __restrict__ sys, SysState* st, DevArrays a) {
  if (*a.any_rebuild == 0) return;
  rebin_finalize<BACKUP>(n_cells, sys, st, a);
}

// backup_r (io/backup_r.cpp:42-79) for flagged systems, a thread per particle.
__device__ __forceinline__ void backup_particles(uint32_t n_part, const SysDesc* __restrict__ sys, const SysState* st,
                                                 const DevArrays& a) {
  for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n_part; i += gridDim.x * blockDim.x) {
    const uint32_t c = a.pcell[i];
    if (c == kInvalid) continue;
    const uint32_t s = a.cell_sys[c];
    if (!sys_flagged(st, s)) continue;
    const SysDesc& S = sys[s];
    int ci, cj, ck;
    cell_ijk(S, c - S.cell_base, ci, cj, ck);
    const double lo[3] = {cell_lo(S, 0, ci), cell_lo(S, 1, cj), cell_lo(S, 2, ck)};
    store_backup(S, a, i, lo, a.rx[i], a.ry[i], a.rz[i]);
  }
}
__global__ void __launch_bounds__(256)
    k_backup(uint32_t n_part, const SysDesc* __restrict__ sys, SysState* st, DevArrays a) {
  if (*a.any_rebuild == 0) return;
  backup_particles(n_part, sys, st, a);
}

// backup_r done for the flagged systems; after a rebin their sub-cell keys
// (k_rebin_finalize) also describe the current positions
__global__ void k_arm(int nsys, SysState* st, const unsigned int* any, bool rebinned) {
  if (*any == 0) return;
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s < nsys && st[s].rebuild) {
    st[s].rebuild_armed = 1;
    if (rebinned) st[s].keys_fresh = 1;
  }
}

// Exclusive scan of one batch's cell counts by one block (the fused rebin).
__device__ __forceinline__ void scan_cells_one_block(const uint32_t* in, uint32_t n, unsigned long long* out) {
  constexpr uint32_t kItems = 8;
  __shared__ unsigned long long wsum[32];
  __shared__ unsigned long long carry;
  const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  if (threadIdx.x == 0) carry = 0;
  for (uint32_t b0 = 0; b0 < n; b0 += blockDim.x * kItems) {
    const uint32_t base = b0 + threadIdx.x * kItems;
    uint32_t v[kItems];
    unsigned long long t = 0;
#pragma unroll
    for (uint32_t k = 0; k < kItems; ++k) {
      v[k] = base + k < n ? in[base + k] : 0u;
      t += v[k];
    }
    unsigned long long inc = t;
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, inc, off);
      if (lane >= static_cast<uint32_t>(off)) inc += y;
    }
    if (lane == 31u) wsum[wib] = inc;
    __syncthreads();
    unsigned long long run = carry + inc - t;
    for (uint32_t q = 0; q < wib; ++q) run += wsum[q];
    unsigned long long tot = 0;
    for (uint32_t q = 0; q < nwarp; ++q) tot += wsum[q];
#pragma unroll
    for (uint32_t k = 0; k < kItems; ++k) {
      if (base + k < n) out[base + k] = run;
      run += v[k];
      if (base + k + 1u == n) out[n] = run;
    }
    __syncthreads();
    if (threadIdx.x == 0) carry += tot;
    __syncthreads();
  }
}

// ---------------------------------------------------------------------------
// chunk_neighbors_execute (particle_neighbors/include/exanb/particle_neighbors/
// chunk_neighbors_execute.h:110-244, 286-372): for each particle of cell a, the
// particles of the 27 cells around a (periodic images included) with
// (cell_a != cell_b || p_a != p_b) && 0 < d2 <= nbh_dist^2, d2 = norm2(r_a - r_b),
// in (cell_enc, p_b) order. Ghost particles outside the partner block enlarged
// by ghost_dist are not candidates (update_ghosts_comm_scheme.cpp:462-469).
//
// Candidates are staged in shared memory as float4 (FP32 position relative to
// the system origin, entry bits in .w); lanes test 32 candidates at a time
// against one particle of the cell and a ballot keeps the hits in order. The FP32 distance decides whenever it lies farther than a
// proven error bound from the threshold; otherwise the reference's FP64 d2 (and
// the FP64 ghost filter) decide, so the pair set is bit-exact.
// Writes one particle's finished list: the buffered entries in full lines, its
// count, lower-half length and slot start.
__device__ __forceinline__ void finish_particle(const DevArrays& a, uint32_t* seg, const uint32_t* sbuf, bool buffered,
                                                uint32_t i, uint32_t base, uint32_t slot, uint32_t cursor,
                                                uint32_t half, bool first_round, uint32_t lane) {
  if (buffered) {
    __syncwarp();
    const uint32_t nw = min(cursor, slot);
    for (uint32_t q = lane; q < nw; q += 32) seg[base + q] = sbuf[q];
    __syncwarp();
  }
  if (lane == 0) {
    a.nbr_cnt[i] = cursor;
    a.nbr_half[i] = half;
    if (first_round) a.nbr_start[i] = base;
  }
}

// One block per cell, for the cells listed by k_neighbors_warp as too large for
// it (a.nbr_wide). The block stages the cell's candidates (up to `cap` per
// round) once in shared memory for all its warps; warp w takes the cell's
// particles w, w + 4, ... two at a time, so each candidate load serves two
// tests. Each particle's hits go into its fixed slot of S.list_slot entries at
// (i - part_base) * list_slot: no count pass, scan or second traversal. When the
// cell's candidates fit one round and the slot fits the warp's list buffers
// (lbuf entries each), a particle's hits are gathered in shared memory and its
// list leaves in full 128-byte lines; otherwise each ballot's hits are stored
// directly. A particle with more hits than the slot holds keeps its true count,
// writes nothing past the slot and flags the system (kErrListOverflow); max_nbr
// records the largest count for resizing.
__device__ __forceinline__ void neighbors_wide(uint32_t n_cells, const SysDesc* __restrict__ sys, SysState* st,
                                               const DevArrays& a, int cap, int lbuf, float4* stage_all) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t wib = threadIdx.x >> 5;
  const uint32_t nwarp = blockDim.x >> 5;
  float4* srel = stage_all;
  uint32_t* sbuf0 = reinterpret_cast<uint32_t*>(stage_all + cap) + static_cast<size_t>(wib) * 2 * lbuf;
  uint32_t* sbuf1 = sbuf0 + lbuf;
  const unsigned lt = lanemask_lt();
  uint32_t acc_s = kInvalid, acc_max = 0;
  unsigned long long acc_sum = 0;
  const uint32_t n_wide = min(*a.nbr_wide_n, n_cells);
  for (uint32_t it = blockIdx.x; it < n_wide; it += gridDim.x) {
    // every condition below depends on the cell only: the block stays together
    const uint32_t c = a.nbr_wide[it];
    const uint32_t s = a.cell_sys[c];
    if (s == kInvalid || !sys_flagged(st, s)) continue;
    const uint32_t na = a.cell_n[c];
    if (na == 0) continue;
    if (s != acc_s) {
      if (lane == 0) flush_list_stats(st, sys, acc_s, acc_max, acc_sum);
      acc_s = s;
      acc_max = 0;
      acc_sum = 0;
    }
    const SysDesc& S = sys[s];
    const uint32_t sa = a.cell_start[c];
    int ci, cj, ck;
    cell_ijk(S, c - S.cell_base, ci, cj, ck);

    // group table: lane g < 27 describes neighbour cell g in (dk, dj, di) order
    uint32_t g_start = 0, g_n = 0, g_code = kImageCenter;
    if (lane < 27) {
      const int di = static_cast<int>(lane % 3) - 1, dj = static_cast<int>((lane / 3) % 3) - 1,
                dk = static_cast<int>(lane / 9) - 1;
      int n3[3] = {ci + di, cj + dj, ck + dk};
      int img[3];
      for (int ax = 0; ax < 3; ++ax) {
        img[ax] = 1;
        if (n3[ax] < 0) { n3[ax] += S.dims[ax]; img[ax] = 0; }
        else if (n3[ax] >= S.dims[ax]) { n3[ax] -= S.dims[ax]; img[ax] = 2; }
      }
      const uint32_t src = S.cell_base + static_cast<uint32_t>((n3[2] * S.dims[1] + n3[1]) * S.dims[0] + n3[0]);
      g_start = a.cell_start[src];
      g_n = a.cell_n[src];
      g_code = static_cast<uint32_t>(img[0] + 3 * img[1] + 9 * img[2]);
    }
    uint32_t g_off = g_n;  // inclusive scan over lanes
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, g_off, off);
      if (lane >= static_cast<uint32_t>(off)) g_off += v;
    }
    const uint32_t ncand = __shfl_sync(0xffffffffu, g_off, 26);
    g_off -= g_n;
    float4 own = make_float4(0.f, 0.f, 0.f, 0.f);
    if (na <= 32 && lane < na) own = a.pf[sa + lane];
    // candidates before cell a's own group come first (groups g < 13), then cell a
    const uint32_t off_self = __shfl_sync(0xffffffffu, g_off, 13);

    const float nb_hi = S.nbh2_f + S.nbh_margin_f;
    const float nb_lo = S.nbh2_f - S.nbh_margin_f;
    const float nb_zero = S.nbh_margin_f;
    const uint32_t slot = S.list_slot;
    uint32_t* const seg = a.nbr + S.list_base;
    const bool buffered = ncand <= static_cast<uint32_t>(cap) && slot <= static_cast<uint32_t>(lbuf);

    for (uint32_t c0 = 0; c0 < ncand; c0 += static_cast<uint32_t>(cap)) {
      const uint32_t c1 = min(ncand, c0 + static_cast<uint32_t>(cap));
      const uint32_t m = c1 - c0;
      const uint32_t mpad = (m + 31u) & ~31u;  // <= cap (a multiple of 32)
      __syncthreads();  // the previous round's readers are done with srel
      // every thread of the block stages candidates t, t + blockDim, ...; the group
      // of candidate u is the last g with g_off[g] <= u (binary search over lanes
      // 0..26; empty groups share their successor's offset and are skipped by it)
      for (uint32_t t0 = 0; t0 < mpad; t0 += blockDim.x) {
        const uint32_t t = t0 + threadIdx.x;
        const uint32_t u = c0 + t;
        uint32_t g = 0;
        for (uint32_t step = 16; step > 0; step >>= 1) {
          const uint32_t probe = g + step;
          const uint32_t po = __shfl_sync(0xffffffffu, g_off, probe < 27u ? probe : 26u);
          if (probe < 27u && po <= u) g = probe;
        }
        const uint32_t gs = __shfl_sync(0xffffffffu, g_start, g);
        const uint32_t go = __shfl_sync(0xffffffffu, g_off, g);
        const uint32_t gc = __shfl_sync(0xffffffffu, g_code, g);
        if (t < m) {
          srel[t] = stage_candidate(S, a, gs + (u - go), gc);
        } else if (t < mpad) {
          // padding up to a whole ballot: unreachable dummies, so the test needs no bound check
          srel[t] = make_float4(1.0e18f, 1.0e18f, 1.0e18f, __uint_as_float(kInvalid));
        }
      }
      __syncthreads();
      const bool last_round = c1 == ncand;
      for (uint32_t pa = wib; pa < na; pa += 2 * nwarp) {
        const uint32_t pb = pa + nwarp;  // second particle of the pair
        const bool two = pb < na;
        const uint32_t i0 = sa + pa, i1 = sa + (two ? pb : pa);
        float4 p0, p1;
        if (na <= 32) {
          p0.x = __shfl_sync(0xffffffffu, own.x, pa);
          p0.y = __shfl_sync(0xffffffffu, own.y, pa);
          p0.z = __shfl_sync(0xffffffffu, own.z, pa);
          const uint32_t src1 = two ? pb : pa;
          p1.x = __shfl_sync(0xffffffffu, own.x, src1);
          p1.y = __shfl_sync(0xffffffffu, own.y, src1);
          p1.z = __shfl_sync(0xffffffffu, own.z, src1);
        } else {
          p0 = a.pf[i0];
          p1 = a.pf[i1];
        }
        // entries taken before candidate index lower_end form the lower half
        const uint32_t low0 = off_self + pa, low1 = off_self + (two ? pb : pa);
        const uint32_t self0 = ((i0 - S.part_base) << 5) | static_cast<uint32_t>(kImageCenter);
        const uint32_t self1 = ((i1 - S.part_base) << 5) | static_cast<uint32_t>(kImageCenter);
        const uint32_t base0 = (i0 - S.part_base) * slot;  // the host keeps npart * slot below 2^32
        const uint32_t base1 = (i1 - S.part_base) * slot;
        uint32_t cur0 = 0, half0 = 0, cur1 = 0, half1 = 0;
        if (c0 > 0) {
          cur0 = a.nbr_cnt[i0];
          half0 = a.nbr_half[i0];
          cur1 = a.nbr_cnt[i1];
          half1 = a.nbr_half[i1];
        }
        const uint32_t start0 = cur0, start1 = cur1;
        uint32_t sv0 = 0, sv1 = 0;  // lane k keeps the ballots of the round's k-th step (<= 32 steps)
        for (uint32_t t0 = 0; t0 < mpad; t0 += 32) {
          const float4 b = srel[t0 + lane];
          const uint32_t ent = __float_as_uint(b.w);
          const bool amb = (ent & kAmbiguousBit) != 0;
          const float ax = p0.x - b.x, ay = p0.y - b.y, az = p0.z - b.z;
          const float bx = p1.x - b.x, by = p1.y - b.y, bz = p1.z - b.z;
          const float d0 = fmaf(ax, ax, fmaf(ay, ay, az * az));
          const float d1 = fmaf(bx, bx, fmaf(by, by, bz * bz));
          bool hit0 = d0 < nb_lo && d0 > nb_zero && !amb;
          bool hit1 = two && d1 < nb_lo && d1 > nb_zero && !amb;
          const bool may0 = !hit0 && d0 <= nb_hi && ent != self0;
          const bool may1 = two && !hit1 && d1 <= nb_hi && ent != self1;
          if (__any_sync(0xffffffffu, may0 || may1)) {
            if (may0) hit0 = exact_neighbor_test(S, a, i0, ent);
            if (may1) hit1 = exact_neighbor_test(S, a, i1, ent);
          }
          const unsigned m0 = __ballot_sync(0xffffffffu, hit0);
          const unsigned m1 = __ballot_sync(0xffffffffu, hit1);
          const uint32_t e = ent & ~kAmbiguousBit;
          const uint32_t q0 = cur0 + __popc(m0 & lt);
          const uint32_t q1 = cur1 + __popc(m1 & lt);
          if (hit0 && q0 < slot) {
            if (buffered) sbuf0[q0] = e;
            else seg[base0 + q0] = e;
          }
          if (hit1 && q1 < slot) {
            if (buffered) sbuf1[q1] = e;
            else seg[base1 + q1] = e;
          }
          if ((t0 >> 5) == lane) {
            sv0 = m0;
            sv1 = m1;
          }
          cur0 += __popc(m0);
          cur1 += __popc(m1);
        }
        // the lower half ends at candidate lower_end: hits of the earlier rounds
        // plus, from the kept ballots, this round's hits below it
        const uint32_t w0 = low0 - c0, w1 = low1 - c0;
        if (w0 < m) {
          const uint32_t v = lane < (w0 >> 5) ? __popc(sv0)
                                             : (lane == (w0 >> 5) ? __popc(sv0 & ((1u << (w0 & 31u)) - 1u)) : 0u);
          half0 = start0 + __reduce_add_sync(0xffffffffu, v);
        }
        if (w1 < m) {
          const uint32_t v = lane < (w1 >> 5) ? __popc(sv1)
                                             : (lane == (w1 >> 5) ? __popc(sv1 & ((1u << (w1 & 31u)) - 1u)) : 0u);
          half1 = start1 + __reduce_add_sync(0xffffffffu, v);
        }
        finish_particle(a, seg, sbuf0, buffered, i0, base0, slot, cur0, half0, c0 == 0, lane);
        if (two) finish_particle(a, seg, sbuf1, buffered, i1, base1, slot, cur1, half1, c0 == 0, lane);
        if (last_round) {
          acc_max = max(acc_max, cur0);
          acc_sum += cur0;
          if (two) {
            acc_max = max(acc_max, cur1);
            acc_sum += cur1;
          }
        }
      }
    }
  }
  if (lane == 0) flush_list_stats(st, sys, acc_s, acc_max, acc_sum);
}

// 64 registers (8 blocks of 128 per SM): measured faster than the 90-register
// schedule despite a few spills.
__global__ void __launch_bounds__(128, 8)
    k_neighbors(uint32_t n_cells, const SysDesc* __restrict__ sys, SysState* st, DevArrays a, int cap, int lbuf) {
  if (*a.any_rebuild == 0) return;
  extern __shared__ float4 stage_all[];
  neighbors_wide(n_cells, sys, st, a, cap, lbuf, stage_all);
}

// ---------------------------------------------------------------------------
// Warp-per-cell form of the same build. The warp stages the candidates that can
// lie within nbh_dist of any of the cell's particles -- those within reach of
// the particles' bounding box, about 3/4 of the 27-cell block; the FP32 distance
// to the box rounds like the pair test and never exceeds it, so what is left out
// is what the test would refuse -- and tests up to
// kWarpP particles per staged load: lanes hold 32 candidates, and a ballot per
// particle appends its hits in order straight to the particle's list slot (an
// entry past the slot lands on its last word; the count flags the overflow).
// The candidates come as runs of x-adjacent cells, contiguous in memory, so no
// lane searches for its cell (few candidates: as a list of their entries); a
// ballot compacts them in order. Two rare cases
// leave the fast test through warp-uniform branches: a chunk holding a candidate
// whose ghost filter is undecided in FP32, and an FP32 distance inside the error
// band around nbh^2 (both then take the reference's FP64 decision). A cell whose
// kept candidates exceed the stage (cap) is appended to a.nbr_wide for
// k_neighbors.
// The build is bound by instruction issue: 418 warp instructions per atom, the
// schedulers busy 66% of the time (1,972,156 atoms: 1.52 ms with every candidate of
// the 27 cells tested, six particles per load and one chunk test; 1.29 with the box
// and the runs, 1.03 with nbr_chunk_clear, its rarely true conditions moved out). Four particles
// per staged load fit 95 registers, 5 blocks of 4 warps per SM; six spill there
// (1.18 against 1.03 ms per build of 1,972,156 atoms), four at 6 blocks 1.07 ms.
// The last particles of a cell are tested two at a time, not padded to four.
constexpr int kWarpP = 4;  // particles tested per staged candidate load in the warp-per-cell build

// Cells of at most this many candidates list them one by one and test whole steps of
// 32; more come as runs, whose last step of each is partly empty. A build of
// 1,972,156 atoms, runs alone / this: 2.88 / 1.78 ms at density 0.05, 2.01 / 1.12 at
// 0.2, 0.95 / 0.87 at 0.35 (8 particles per cell, 220 candidates), 0.99 / 1.02 at
// 0.5, 1.11 / 1.11 at 0.84; listing up to 128 takes 1.48 ms at 0.2.
constexpr uint32_t kPackedMax = 256;

// FP32 values as integers in the same order (no NaN).
__device__ __forceinline__ int ordered_int(float f) {
  const int b = __float_as_int(f);
  return b ^ ((b >> 31) & 0x7fffffff);
}
__device__ __forceinline__ float from_ordered(int k) { return __int_as_float(k ^ ((k >> 31) & 0x7fffffff)); }

// What one warp of the warp-per-cell build works on.
struct WarpCell {
  uint32_t sa, na;        // the cell's particles
  uint32_t off_self;      // stage index of its first particle
  uint32_t mpad;          // staged candidates, padded to whole chunks
  bool undecided;         // some have an undecided ghost filter
  uint32_t slot;
  uint32_t* seg;          // the system's list segment
  uint32_t* sink;
  float nb_lo, nb_hi, nb_zero, band;
  unsigned lt;
};

// List lengths of one cell: lane p's particle, and this lane's largest and sum.
struct CellCounts {
  uint32_t cnt, half;
  bool mine;
  uint32_t most, sum;
};

// Particles p0 .. p0 + NP - 1 of the cell against the whole stage.
template <int NP>
__device__ __forceinline__ void warp_pass(const SysDesc& S, const DevArrays& a, const WarpCell& w, const float4* srel,
                                          float4 own, uint32_t p0, uint32_t lane, CellCounts& counts) {
  // particles past the cell's end sit at -1e18: never within reach of a
  // candidate (real ones, or the +1e18 dummies), so they need no test
  float px[NP], py[NP], pz[NP];
  uint32_t cur[NP], half[NP];
#pragma unroll
  for (int k = 0; k < NP; ++k) {
    const uint32_t pk = p0 + k;
    float4 q;
    if (w.na <= 32) {
      q.x = __shfl_sync(0xffffffffu, own.x, pk & 31u);
      q.y = __shfl_sync(0xffffffffu, own.y, pk & 31u);
      q.z = __shfl_sync(0xffffffffu, own.z, pk & 31u);
    } else {
      q = pk < w.na ? a.pf[w.sa + pk] : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    const bool valid = pk < w.na;
    px[k] = valid ? q.x : -1.0e18f;
    py[k] = valid ? q.y : -1.0e18f;
    pz[k] = valid ? q.z : -1.0e18f;
    cur[k] = 0;
    half[k] = 0;
  }
  const uint32_t i0 = w.sa + p0;
  const uint32_t self0 = ((i0 - S.part_base) << 5) | static_cast<uint32_t>(kImageCenter);
  const uint32_t low0 = w.off_self + p0;
  // hits go straight to the particles' slots (consecutive particles, stride
  // slot); a system without slots yet (the sizing build) only counts, its
  // hits landing in the warp's sink
  uint32_t* const pslot = w.slot ? w.seg + static_cast<size_t>(i0 - S.part_base) * w.slot : w.sink;
  const uint32_t pstride = w.slot ? w.slot : 1u;
  unsigned long long px2[NP / 2], py2[NP / 2], pz2[NP / 2], minus_nbh2;
#pragma unroll
  for (int k = 0; k < NP / 2; ++k) {
    asm("mov.b64 %0, {%1, %2};" : "=l"(px2[k]) : "f"(px[2 * k]), "f"(px[2 * k + 1]));
    asm("mov.b64 %0, {%1, %2};" : "=l"(py2[k]) : "f"(py[2 * k]), "f"(py[2 * k + 1]));
    asm("mov.b64 %0, {%1, %2};" : "=l"(pz2[k]) : "f"(pz[2 * k]), "f"(pz[2 * k + 1]));
  }
  asm("mov.b64 %0, {%1, %1};" : "=l"(minus_nbh2) : "f"(-S.nbh2_f));
  const uint32_t self_t0 = low0 & ~31u, self_span = ((low0 + NP - 1u) & ~31u) - self_t0;
  uint32_t room = 0;  // chunks that fit every slot whatever they hold
  for (uint32_t t0 = 0; t0 < w.mpad; t0 += 32) {
    const float4 b = srel[t0 + lane];
    const uint32_t ent = __float_as_uint(b.w);
    // the particles' own entries (lower-half ends) sit at stage indices low0 + k;
    // entries in [kAmbiguousBit, kInvalid): ghost filter undecided in FP32
    if (room == 0) {
      uint32_t most = cur[0];
#pragma unroll
      for (int k = 1; k < NP; ++k) most = max(most, cur[k]);
      room = w.slot > most ? (w.slot - most) >> 5 : 0u;
    }
    const bool close = t0 - self_t0 <= self_span || room == 0 ||
                       (w.undecided && __any_sync(0xffffffffu, ent - kAmbiguousBit < kInvalid - kAmbiguousBit));
    if (close || !nbr_chunk_clear<NP>(b, px2, py2, pz2, w.nb_lo, w.nb_zero, minus_nbh2, w.band, w.lt, pslot, pstride,
                                      cur))
      nbr_chunk<NP, true, true>(S, a, b, px, py, pz, i0, self0, t0, low0, w.nb_lo, w.nb_hi, w.nb_zero, w.lt, pslot,
                                pstride, cur, half);
    room -= room != 0 ? 1u : 0u;
  }
  if (w.na <= 32) {
    // lane p keeps particle p's counts; they are written together
#pragma unroll
    for (int k = 0; k < NP; ++k)
      if (lane == p0 + k) {
        counts.cnt = cur[k];
        counts.half = half[k];
        counts.mine = lane < w.na;
      }
    return;
  }
#pragma unroll
  for (int k = 0; k < NP; ++k) {
    const uint32_t pk = p0 + k;
    if (pk < w.na) {
      const uint32_t i = w.sa + pk;
      if (lane == 0) {
        a.nbr_cnt[i] = cur[k];
        a.nbr_half[i] = half[k];
        a.nbr_start[i] = (i - S.part_base) * w.slot;  // the host keeps npart * slot below 2^32
        counts.most = max(counts.most, cur[k]);
        counts.sum += cur[k];
      }
    }
  }
}

// split warps share a cell (each stages it and takes every split-th group of
// particles): batches with fewer cells than the GPU holds warps.
// (Plain loads: in the fused rebin the mirrors were written by this launch.)
template <int WARPS>
__device__ __forceinline__ void neighbors_warp(uint32_t n_cells, const SysDesc* __restrict__ sys, SysState* st,
                                               const DevArrays& a, int cap, bool prune, bool half_form, uint32_t split,
                                               float4* stage) {
  const uint32_t lane = threadIdx.x & 31;
  const uint32_t wib = threadIdx.x >> 5;
  const uint32_t nwarp = blockDim.x >> 5;
  float4* srel = stage + static_cast<size_t>(wib) * cap;
  constexpr int kSteps = 32;
  __shared__ uint4 lists[WARPS][kSteps];
  uint4* const list = lists[wib];  // first candidate, candidates left, image code
  __shared__ uint32_t sink[WARPS][kWarpP];  // hits of systems without list slots
  WarpCell w;
  w.lt = lanemask_lt();
  w.sink = sink[wib];
  uint32_t acc_s = kInvalid, acc_max = 0;
  unsigned long long acc_sum = 0;
  const uint32_t nw_all = gridDim.x * nwarp;
  for (uint32_t u = blockIdx.x * nwarp + wib; u < n_cells * split; u += nw_all) {
    const uint32_t c = u / split, part = u - c * split;
    const uint32_t s = a.cell_sys[c];
    if (s == kInvalid || !sys_flagged(st, s)) continue;
    if (half_form && !st[s].half_bad) continue;  // built by the half-shell kernels
    const uint32_t na = a.cell_n[c];
    if (na <= part * kWarpP) continue;
    if (prune && a.cside[c] >= 2 && st[s].keys_fresh) {
      if (lane == 0 && part == 0) a.nbr_sub[atomicAdd(a.nbr_sub_n, 1u)] = c;
      continue;
    }
    const SysDesc& S = sys[s];
    const uint32_t sa = a.cell_start[c];
    int ci, cj, ck;
    cell_ijk(S, c - S.cell_base, ci, cj, ck);
    w.nb_hi = S.nbh2_f + S.nbh_margin_f;
    w.nb_lo = S.nbh2_f - S.nbh_margin_f;
    w.nb_zero = S.nbh_margin_f;
    w.band = 1.001f * fmaxf(w.nb_hi - S.nbh2_f, S.nbh2_f - w.nb_lo);

    // group table: lane g < 27 describes neighbour cell g in (dk, dj, di) order
    uint32_t g_start = 0, g_n = 0, g_code = kImageCenter;
    if (lane < 27) {
      const int di = static_cast<int>(lane % 3) - 1, dj = static_cast<int>((lane / 3) % 3) - 1,
                dk = static_cast<int>(lane / 9) - 1;
      int n3[3] = {ci + di, cj + dj, ck + dk};
      int img[3];
      for (int ax = 0; ax < 3; ++ax) {
        img[ax] = 1;
        if (n3[ax] < 0) { n3[ax] += S.dims[ax]; img[ax] = 0; }
        else if (n3[ax] >= S.dims[ax]) { n3[ax] -= S.dims[ax]; img[ax] = 2; }
      }
      const uint32_t src = S.cell_base + static_cast<uint32_t>((n3[2] * S.dims[1] + n3[1]) * S.dims[0] + n3[0]);
      g_start = a.cell_start[src];
      g_n = a.cell_n[src];
      g_code = static_cast<uint32_t>(img[0] + 3 * img[1] + 9 * img[2]);
    }
    // the particles' bounding box
    float4 own = make_float4(0.f, 0.f, 0.f, 0.f);
    float bl[3] = {3.0e38f, 3.0e38f, 3.0e38f}, bh[3] = {-3.0e38f, -3.0e38f, -3.0e38f};
    for (uint32_t q = lane; q < na; q += 32) {
      const float4 v = a.pf[sa + q];
      if (q == lane) own = v;
      bl[0] = fminf(bl[0], v.x);
      bl[1] = fminf(bl[1], v.y);
      bl[2] = fminf(bl[2], v.z);
      bh[0] = fmaxf(bh[0], v.x);
      bh[1] = fmaxf(bh[1], v.y);
      bh[2] = fmaxf(bh[2], v.z);
    }
#pragma unroll
    for (int ax = 0; ax < 3; ++ax) {
      bl[ax] = from_ordered(__reduce_min_sync(0xffffffffu, ordered_int(bl[ax])));
      bh[ax] = from_ordered(__reduce_max_sync(0xffffffffu, ordered_int(bh[ax])));
    }

    uint32_t m = 0, off_self = 0;
    bool undecided = false;  // a candidate whose ghost filter FP32 does not decide
    // this lane's candidate j through its image, kept if it lies within reach of the
    // box; candidate `self` of these 32 (if one is) is the cell's own first particle
    // (kept, as all its own are: distance 0)
    auto stage = [&](float4 pb, uint32_t j, uint32_t code, bool valid, uint32_t self) {
      float4 rb = pb;
      if (code == static_cast<uint32_t>(kImageCenter)) {
        rb.w = __uint_as_float(((j - S.part_base) << 5) | static_cast<uint32_t>(kImageCenter));
      } else {
        rb = stage_from(S, pb, j, code);
        undecided |= valid && __float_as_uint(rb.w) - kAmbiguousBit < kInvalid - kAmbiguousBit;
      }
      const float ex = fmaxf(fmaxf(bl[0] - rb.x, rb.x - bh[0]), 0.f);
      const float ey = fmaxf(fmaxf(bl[1] - rb.y, rb.y - bh[1]), 0.f);
      const float ez = fmaxf(fmaxf(bl[2] - rb.z, rb.z - bh[2]), 0.f);
      const bool keep = valid && fmaf(ex, ex, fmaf(ey, ey, ez * ez)) <= w.nb_hi;
      const unsigned km = __ballot_sync(0xffffffffu, keep);
      if (self < 32u) off_self = m + __popc(km & ((1u << self) - 1u));
      const uint32_t pos = m + __popc(km & w.lt);
      if (keep && pos < static_cast<uint32_t>(cap)) srel[pos] = rb;
      m += __popc(km);
    };
    uint32_t g_off = g_n;  // inclusive scan
    for (int off = 1; off < 32; off <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, g_off, off);
      if (lane >= static_cast<uint32_t>(off)) g_off += v;
    }
    const uint32_t ncand = __shfl_sync(0xffffffffu, g_off, 31);
    g_off -= g_n;
    if (ncand <= kPackedMax && ncand + kPackedMax / 4u <= static_cast<uint32_t>(cap)) {
      // few: entries listed one after the other (behind the stage), 32 per step
      uint32_t* const map = reinterpret_cast<uint32_t*>(srel + cap) - kPackedMax;
      for (uint32_t q = 0; q < g_n; ++q) map[g_off + q] = ((g_start + q - S.part_base) << 5) | g_code;
      __syncwarp();
      const uint32_t first = __shfl_sync(0xffffffffu, g_off, 13);
      for (uint32_t t0 = 0; t0 < ncand; t0 += 128u) {
        uint32_t ent[4];
        float4 pb[4];
#pragma unroll
        for (uint32_t q = 0; q < 4u; ++q) {
          const uint32_t u = t0 + 32u * q + lane;
          ent[q] = u < ncand ? map[u] : static_cast<uint32_t>(kImageCenter);
          pb[q] = u < ncand ? a.pf[S.part_base + (ent[q] >> 5)] : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (uint32_t q = 0; q < 4u; ++q) {
          const uint32_t u0 = t0 + 32u * q;
          if (u0 < ncand) stage(pb[q], S.part_base + (ent[q] >> 5), ent[q] & 31u, u0 + lane < ncand, first - u0);
        }
      }
    } else {
      // 32 candidates of a run per step, the steps listed first so that the loads
      // of four are in flight together. The three cells of a row are one contiguous
      // run unless x wraps around: the first lane of the row then takes them all
      const uint32_t n1 = __shfl_down_sync(0xffffffffu, g_n, 1), n2 = __shfl_down_sync(0xffffffffu, g_n, 2);
      if (ci > 0 && ci < S.dims[0] - 1) g_n = lane % 3u == 0u ? g_n + n1 + n2 : 0u;
      const uint32_t steps = lane < 27u ? (g_n + 31u) >> 5 : 0u;
      uint32_t at = steps;  // inclusive scan
      for (int off = 1; off < 32; off <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, at, off);
        if (lane >= static_cast<uint32_t>(off)) at += v;
      }
      const uint32_t total = __shfl_sync(0xffffffffu, at, 31);
      at -= steps;
      for (uint32_t t0 = 0; t0 < total; t0 += kSteps) {
        __syncwarp();  // the previous list's readers are done
        for (uint32_t q = 0; q < steps; ++q)
          if (at + q - t0 < kSteps) list[at + q - t0] = make_uint4(g_start + 32u * q, g_n - 32u * q, g_code, 0u);
        __syncwarp();
        const uint32_t t1 = min(total - t0, static_cast<uint32_t>(kSteps));
        for (uint32_t t = 0; t < t1; t += 4u) {
          uint4 run[4];
          float4 pb[4];
#pragma unroll
          for (uint32_t q = 0; q < 4u; ++q) {
            run[q] = list[min(t + q, t1 - 1u)];
            if (t + q >= t1) run[q].y = 0;
            pb[q] = lane < run[q].y ? a.pf[run[q].x + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
          }
#pragma unroll
          for (uint32_t q = 0; q < 4u; ++q) {
            const uint32_t self = sa - run[q].x;
            stage(pb[q], run[q].x + lane, run[q].z, lane < run[q].y,
                  run[q].z == static_cast<uint32_t>(kImageCenter) && self < run[q].y ? self : 32u);
          }
        }
      }
    }
    if (m > static_cast<uint32_t>(cap)) {
      __syncwarp();
      if (lane == 0 && part == 0) a.nbr_wide[atomicAdd(a.nbr_wide_n, 1u)] = c;
      continue;
    }
    const uint32_t mpad = (m + 31u) & ~31u;  // <= cap (a multiple of 32)
    if (m + lane < mpad) srel[m + lane] = make_float4(1.0e18f, 1.0e18f, 1.0e18f, __uint_as_float(kInvalid));
    __syncwarp();
    if (s != acc_s) {
      if (lane == 0) flush_list_stats(st, sys, acc_s, acc_max, acc_sum);
      acc_s = s;
      acc_max = 0;
      acc_sum = 0;
    }
    w.sa = sa;
    w.na = na;
    w.off_self = off_self;
    w.mpad = mpad;
    w.undecided = __any_sync(0xffffffffu, undecided);
    w.slot = S.list_slot;
    w.seg = a.nbr + S.list_base;
    CellCounts counts{0u, 0u, false, 0u, 0u};
    for (uint32_t p0 = part * kWarpP; p0 < na; p0 += kWarpP * split) {
      const uint32_t rest = na - p0;
      if (rest > 2u) warp_pass<4>(S, a, w, srel, own, p0, lane, counts);
      else warp_pass<2>(S, a, w, srel, own, p0, lane, counts);
    }
    if (counts.mine) {
      const uint32_t i = sa + lane;
      a.nbr_cnt[i] = counts.cnt;
      a.nbr_half[i] = counts.half;
      a.nbr_start[i] = (i - S.part_base) * w.slot;  // the host keeps npart * slot below 2^32
      counts.most = counts.cnt;
      counts.sum = counts.cnt;
    }
    acc_max = max(acc_max, __reduce_max_sync(0xffffffffu, counts.most));
    acc_sum += __reduce_add_sync(0xffffffffu, counts.sum);
    __syncwarp();  // the stage is refilled for the next cell
  }
  if (lane == 0) flush_list_stats(st, sys, acc_s, acc_max, acc_sum);
}

__global__ void __launch_bounds__(128, 5)
    k_neighbors_warp(uint32_t n_cells, const SysDesc* __restrict__ sys, SysState* st, DevArrays a, int cap,
                     bool prune, bool half_form, uint32_t split) {
  if (*a.any_rebuild == 0) return;
  extern __shared__ float4 stage_w[];
  neighbors_warp<4>(n_cells, sys, st, a, cap, prune, half_form, split, stage_w);
}

// The trigger's decision and the whole rebin (K_r1 .. K_r6, the resets of the
// build that follows) of a small batch in one cooperative launch. A step without
// a rebuild costs one launch that returns at once, where the separate kernels
// cost twelve (0.7 us each inside a graph, 2.3 us when launched one by one); a
// rebuild costs six grid barriers: 50 steps of 864 atoms 844 -> 511 us, of 32,000
// 2.78 -> 2.42 ms. The phases are the separate kernels' bodies.
// BUILD: the lists of the flagged systems too (the warp-per-cell form without
// sub-cell pruning, then the cells it passes on), two more barriers: a step
// without a rebuild is then three launches, push, this one and the forces.
template <bool EXACT, bool BUILD>
__global__ void __launch_bounds__(256)
    k_rebin_fused(uint32_t n_part, uint32_t n_cells, int nsys, const SysDesc* __restrict__ sys, SysState* st,
                  DevArrays a, int cap, int lbuf, uint32_t split, bool check) {
  extern __shared__ float4 fused_smem[];
  const auto triggered = [&](int s) {
    return __ldcg(&st[s].moved) != 0ull && !(__ldcg(&st[s].error) & kErrBarrier);
  };
  int flagged = 0;
  for (int s = static_cast<int>(threadIdx.x); s < nsys; s += static_cast<int>(blockDim.x))
    flagged |= triggered(s) ? 1 : 0;
  if (!__syncthreads_or(flagged)) {
    if (blockIdx.x == 0) {
      for (int s = static_cast<int>(threadIdx.x); s < nsys; s += static_cast<int>(blockDim.x)) st[s].rebuild = 0;
      if (threadIdx.x == 0) *a.any_rebuild = 0;
    }
    return;
  }
  if (blockIdx.x == 0) {
    // what the other blocks read before the first barrier is `moved` and `error`
    unsigned int mine = 0;
    for (int s = static_cast<int>(threadIdx.x); s < nsys; s += static_cast<int>(blockDim.x)) {
      const bool r = triggered(s);
      st[s].rebuild = r ? 1u : 0u;
      if (!r) continue;
      ++mine;
      st[s].rebuilds += 1;
      st[s].rebuild_armed = 1;
      st[s].keys_fresh = 1;
      // the build that follows (k_nbr_reset)
      st[s].list_used = 0;
      st[s].max_nbr = 0;
      st[s].lists_fresh = 1;
      st[s].compact_bad = 0;
      st[s].half_bad = 0;
    }
    if (threadIdx.x == 0) {
      *a.any_rebuild = 0;
      *a.nbr_wide_n = 0;
      *a.nbr_sub_n = 0;
    }
    __syncthreads();
    if (mine) atomicAdd(a.any_rebuild, mine);
  }
  // check: one block more than there are, for 20 ms
  bool ok = check ? grid_barrier(a.grid_ctl, gridDim.x + 1u, 20000000ull) : grid_barrier(a.grid_ctl, gridDim.x);
  if (ok) {
    if (blockIdx.x == 0)
      for (int s = static_cast<int>(threadIdx.x); s < nsys; s += static_cast<int>(blockDim.x)) st[s].moved = 0;
    rebin_dest(n_part, sys, st, a);
    ok = grid_barrier(a.grid_ctl, gridDim.x);
  }
  if (ok) {
    rebin_compact(n_cells, sys, st, a);
    ok = grid_barrier(a.grid_ctl, gridDim.x);
  }
  if (ok) {
    rebin_count(n_cells, sys, st, a);
    ok = grid_barrier(a.grid_ctl, gridDim.x);
  }
  if (ok) {
    if (blockIdx.x == 0) scan_cells_one_block(a.cell_cnt, n_cells, a.cell_scan);
    ok = grid_barrier(a.grid_ctl, gridDim.x);
  }
  if (ok) {
    rebin_scatter(n_cells, sys, st, a);
    ok = grid_barrier(a.grid_ctl, gridDim.x);
  }
  if (ok) {
    rebin_finalize<EXACT ? kBackupNone : kBackupPlain>(n_cells, sys, st, a);
    if (EXACT || BUILD) ok = grid_barrier(a.grid_ctl, gridDim.x);
  }
  if (EXACT && ok) backup_particles(n_part, sys, st, a);
  if (BUILD && ok) {
    neighbors_warp<8>(n_cells, sys, st, a, cap, false, false, split, fused_smem);
    ok = grid_barrier(a.grid_ctl, gridDim.x);
  }
  if (BUILD && ok) neighbors_wide(n_cells, sys, st, a, cap, lbuf, fused_smem);
  if (!ok && threadIdx.x == 0) {
    // a barrier ran out of time: the systems being rebuilt stop
    for (int s = 0; s < nsys; ++s)
      if (__ldcg(&st[s].rebuild)) atomicOr(&st[s].error, kErrBarrier);
  }
}

// Clears the per-build list statistics of the flagged systems.
__global__ void k_nbr_reset(int nsys, SysState* st, const unsigned int* any, unsigned int* wide_n,
                            unsigned int* sub_n) {
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    *wide_n = 0;
    *sub_n = 0;
  }
  if (*any == 0) return;
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nsys || !st[s].rebuild) return;
  st[s].list_used = 0;
  st[s].max_nbr = 0;
  st[s].lists_fresh = 1;  // the build that follows reads the current positions
  st[s].compact_bad = 0;
  st[s].half_bad = 0;
}

// ---------------------------------------------------------------------------
// Exclusive scan, u32 -> u64, three phases (tile sums, scan of sums, tiles).
constexpr int kScanThreads = 256;
constexpr int kScanItems = 8;
constexpr uint32_t kScanTile = kScanThreads * kScanItems;

__global__ void __launch_bounds__(kScanThreads) k_scan_tiles(const uint32_t* __restrict__ in, uint32_t n,
                                                              unsigned long long* sums, const unsigned int* gate) {
  if (gate && *gate == 0) return;
  __shared__ unsigned long long red[kScanThreads / 32];
  const uint32_t base = blockIdx.x * kScanTile;
  unsigned long long v = 0;
  for (int k = 0; k < kScanItems; ++k) {
    const uint32_t idx = base + threadIdx.x + k * kScanThreads;
    if (idx < n) v += in[idx];
  }
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long t = 0;
    for (int w = 0; w < kScanThreads / 32; ++w) t += red[w];
    sums[blockIdx.x] = t;
  }
}

__global__ void __launch_bounds__(1024) k_scan_sums(unsigned long long* sums, uint32_t nb, const unsigned int* gate) {
  if (gate && *gate == 0) return;
  __shared__ unsigned long long carry_s;
  __shared__ unsigned long long wsum[32];
  if (threadIdx.x == 0) carry_s = 0;
  __syncthreads();
  for (uint32_t b0 = 0; b0 < nb; b0 += 1024) {
    const uint32_t b = b0 + threadIdx.x;
    const unsigned long long x = b < nb ? sums[b] : 0ull;
    unsigned long long inc = x;
    const uint32_t lane = threadIdx.x & 31;
    for (int off = 1; off < 32; off <<= 1) {
      const unsigned long long y = __shfl_up_sync(0xffffffffu, inc, off);
      if (lane >= static_cast<uint32_t>(off)) inc += y;
    }
    if (lane == 31) wsum[threadIdx.x >> 5] = inc;
    __syncthreads();
    if (threadIdx.x < 32) {
      unsigned long long w = wsum[threadIdx.x];
      unsigned long long wi = w;
      for (int off = 1; off < 32; off <<= 1) {
        const unsigned long long y = __shfl_up_sync(0xffffffffu, wi, off);
        if (threadIdx.x >= static_cast<uint32_t>(off)) wi += y;
      }
      wsum[threadIdx.x] = wi - w;
    }
    __syncthreads();
    const unsigned long long carry = carry_s;
    if (b < nb) sums[b] = carry + wsum[threadIdx.x >> 5] + inc - x;
    __syncthreads();
    if (threadIdx.x == 1023) carry_s = carry + wsum[31] + inc;
    __syncthreads();
  }
}

__global__ void __launch_bounds__(kScanThreads) k_scan_final(const uint32_t* __restrict__ in, uint32_t n,
                                                              const unsigned long long* __restrict__ sums,
                                                              unsigned long long* out, const unsigned int* gate) {
  if (gate && *gate == 0) return;
  __shared__ unsigned long long wsum[kScanThreads / 32];
  const uint32_t base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  unsigned long long loc[kScanItems];
  unsigned long long t = 0;
  for (int k = 0; k < kScanItems; ++k) {
    const uint32_t idx = base + k;
    loc[k] = idx < n ? in[idx] : 0ull;
    t += loc[k];
  }
  const uint32_t lane = threadIdx.x & 31;
  unsigned long long inc = t;
  for (int off = 1; off < 32; off <<= 1) {
    const unsigned long long y = __shfl_up_sync(0xffffffffu, inc, off);
    if (lane >= static_cast<uint32_t>(off)) inc += y;
  }
  if (lane == 31) wsum[threadIdx.x >> 5] = inc;
  __syncthreads();
  unsigned long long wpre = 0;
  for (uint32_t w = 0; w < (threadIdx.x >> 5); ++w) wpre += wsum[w];
  unsigned long long run = sums[blockIdx.x] + wpre + inc - t;
  for (int k = 0; k < kScanItems; ++k) {
    const uint32_t idx = base + k;
    if (idx < n) out[idx] = run;
    run += loc[k];
    if (idx + 1 == n) out[n] = run;
  }
}

inline int warp_grid(uint32_t n_items, int warps_per_block, int sm_count) {
  long long want = (static_cast<long long>(n_items) + warps_per_block - 1) / warps_per_block;
  const long long cap = static_cast<long long>(sm_count) * 16;
  if (want > cap) want = cap;
  return static_cast<int>(want < 1 ? 1 : want);
}

inline int thread_grid(uint32_t n, int threads, int sm_count) {
  long long want = (static_cast<long long>(n) + threads - 1) / threads;
  const long long cap = static_cast<long long>(sm_count) * 8;
  if (want > cap) want = cap;
  return static_cast<int>(want < 1 ? 1 : want);
}

}  // namespace

size_t scan_scratch_elems(uint32_t n) { return (n + kScanTile - 1) / kScanTile + 1; }

int launch_scan_u32_to_u64(const uint32_t* in, unsigned long long* out, uint32_t n, unsigned long long* scratch,
                           cudaStream_t stream, const unsigned int* gate) {
  if (n == 0) {
    cudaMemsetAsync(out, 0, sizeof(unsigned long long), stream);
    return 0;
  }
  const uint32_t nb = (n + kScanTile - 1) / kScanTile;
  k_scan_tiles<<<nb, kScanThreads, 0, stream>>>(in, n, scratch, gate);
  k_scan_sums<<<1, 1024, 0, stream>>>(scratch, nb, gate);
  k_scan_final<<<nb, kScanThreads, 0, stream>>>(in, n, scratch, out, gate);
  return 3;
}

// The encoding inside the rebin's last pass costs a warp's FP64 instructions per cell,
// however few its particles: a pass of its own, a thread per particle, unless the
// cells fill the warps and the batch is too small to hide one more launch. Rebin and
// build, inside / alone: 8,788 atoms 111 / 112 us at density 0.35 (8 per cell), 111 /
// 123 at 0.84; 32,000 atoms 221 / 160 us at 0.1, 134 / 136 at 0.84; 97,556 atoms 197
// / 195 us at 0.84; 953,312 atoms 11.9 / 8.1 ms at 0.02, 1.06 / 1.00 ms at 0.84. (In
// the fused rebin the pass is never slower: 50 steps of 8,788 atoms 73.0 / 73.0 us
// each at 0.84, 69 / 63 at 0.02.)
constexpr uint32_t kFoldBackupMax = 50000, kFoldBackupPerCell = 8;

int launch_rebin(const Extent& ex, const SysDesc* sys, SysState* st, const DevArrays& a, cudaStream_t stream,
                 bool exact_backup) {
  if (ex.n_part == 0 || ex.n_cells == 0) return 0;
  k_rebin_dest<<<thread_grid(ex.n_part, 256, ex.sm_count), 256, 0, stream>>>(ex.n_part, sys, st, a);
  const int wg = warp_grid(ex.n_cells, 4, ex.sm_count);
  k_rebin_compact<<<wg, 128, 0, stream>>>(ex.n_cells, sys, st, a);
  k_rebin_count<<<wg, 128, 0, stream>>>(ex.n_cells, sys, st, a);
  const int ns = launch_scan_u32_to_u64(a.cell_cnt, a.cell_scan, ex.n_cells, a.scan_blocks, stream, a.any_rebuild);
  k_rebin_scatter<<<wg, 128, 0, stream>>>(ex.n_cells, sys, st, a);
  int nb = 0;
  if (!exact_backup) {
    k_rebin_finalize<kBackupPlain><<<wg, 128, 0, stream>>>(ex.n_cells, sys, st, a);
  } else if (ex.n_part <= kFoldBackupMax && ex.n_part >= kFoldBackupPerCell * ex.n_cells) {
    k_rebin_finalize<kBackupExact><<<wg, 128, 0, stream>>>(ex.n_cells, sys, st, a);
  } else {
    k_rebin_finalize<kBackupNone><<<wg, 128, 0, stream>>>(ex.n_cells, sys, st, a);
    k_backup<<<thread_grid(ex.n_part, 256, ex.sm_count), 256, 0, stream>>>(ex.n_part, sys, st, a);
    nb = 1;
  }
  k_arm<<<(ex.nsys + 127) / 128, 128, 0, stream>>>(ex.nsys, st, a.any_rebuild, true);
  return 6 + nb + ns;
}

bool fused_rebin_fits(const Extent& ex) {
  return ex.n_part > 0 && ex.n_part <= kFusedRebinMaxParticles && ex.n_cells > 0 && ex.n_cells <= kFusedRebinMaxCells;
}

bool fused_build_fits(const Extent& ex, int form, bool prune) {
  return ex.n_cells <= kFusedBuildMaxCells && form == kBuildWarp && ex.force_form != kForceStaged && !(prune && ex.dense);
}

int launch_rebin_fused(const Extent& ex, const SysDesc* sys, SysState* st, const DevArrays& a, bool exact_backup,
                       bool build, int cap, int lbuf, bool check, cudaStream_t stream) {
  constexpr unsigned warps = 8;
  // at most one block per SM: always co-resident. The rebin takes a warp per
  // cell, the build up to four
  const unsigned want = build ? ex.n_cells * 4u : ex.n_cells;
  const unsigned grid = std::min((want + warps - 1u) / warps, static_cast<unsigned>(ex.sm_count));
  const uint32_t split = ex.n_cells * 4u <= grid * warps ? 4u : (ex.n_cells * 2u <= grid * warps ? 2u : 1u);
  size_t smem = 0;
  if (build) {
    smem = std::max(static_cast<size_t>(warps) * cap * sizeof(float4),
                    static_cast<size_t>(cap) * sizeof(float4) + static_cast<size_t>(warps) * 2 * lbuf * sizeof(uint32_t));
  }
  auto kern = exact_backup ? (build ? k_rebin_fused<true, true> : k_rebin_fused<true, false>)
                           : (build ? k_rebin_fused<false, true> : k_rebin_fused<false, false>);
  if (build) raise_smem_limit(kern, warps * kStageCapMax * sizeof(float4));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(warps * 32u);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kern, ex.n_part, ex.n_cells, ex.nsys, sys, st, a, cap, lbuf, split, check);
  return 1;
}

int launch_backup(const Extent& ex, const SysDesc* sys, SysState* st, const DevArrays& a, cudaStream_t stream) {
  if (ex.n_part == 0) return 0;
  k_backup<<<thread_grid(ex.n_part, 256, ex.sm_count), 256, 0, stream>>>(ex.n_part, sys, st, a);
  k_arm<<<(ex.nsys + 127) / 128, 128, 0, stream>>>(ex.nsys, st, a.any_rebuild, false);
  return 2;
}

int launch_neighbors(const Extent& ex, const SysDesc* sys, SysState* st, const DevArrays& a, int cap, int lbuf,
                     cudaStream_t stream, int form, bool prune, bool reset) {
  if (ex.n_cells == 0) return 0;
  const size_t smem = static_cast<size_t>(cap) * sizeof(float4) + static_cast<size_t>(4) * 2 * lbuf * sizeof(uint32_t);
  // warp-per-cell form: the stage alone (hits go straight to the slots)
  const size_t smem_w = 4 * static_cast<size_t>(cap) * sizeof(float4);
  raise_smem_limit(k_neighbors, kStageCapMax * sizeof(float4) + 4u * 2u * kMaxListBuf * sizeof(uint32_t));
  raise_smem_limit(k_neighbors_warp, 4u * kStageCapMax * sizeof(float4));
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_neighbors_warp, 128, smem_w) != cudaSuccess || per_sm < 1)
    per_sm = 1;
  // four or two warps per cell while that leaves no warp of the GPU without one
  const long long warps = static_cast<long long>(per_sm) * ex.sm_count * 4;
  const uint32_t split = ex.n_cells * 4ll <= warps ? 4u : (ex.n_cells * 2ll <= warps ? 2u : 1u);
  const long long want_w = (static_cast<long long>(ex.n_cells) * split + 3) / 4;
  const int grid_w = static_cast<int>(std::max(1ll, std::min(want_w, static_cast<long long>(per_sm) * ex.sm_count)));
  if (reset) k_nbr_reset<<<(ex.nsys + 127) / 128, 128, 0, stream>>>(ex.nsys, st, a.any_rebuild, a.nbr_wide_n, a.nbr_sub_n);
  // half-shell form: masks first; systems it cannot take go through the warp-per-cell build
  const bool half = form == kBuildHalf && a.nmask != nullptr;
  const int nh = half ? launch_neighbors_half_test(ex, sys, st, a, stream) : 0;
  if (form == kBuildRows) launch_neighbors_rows(ex, sys, st, a, stream, prune);
  else k_neighbors_warp<<<grid_w, 128, smem_w, stream>>>(ex.n_cells, sys, st, a, cap, prune, half, split);
  const int ne = half ? launch_neighbors_half_emit(ex, sys, st, a, stream) : 0;
  // dense cells (sub-grid side >= 2), before the block-per-cell build, which takes the ones it passes on
  const int nsub = prune ? launch_neighbors_sub(ex, sys, st, a, cap, stream) : 0;
  k_neighbors<<<warp_grid(ex.n_cells, 1, ex.sm_count), 128, smem, stream>>>(ex.n_cells, sys, st, a, cap, lbuf);
  // compact entries for the staged force traversal
  const int nc = ex.force_form == kForceStaged ? launch_compact_lists(ex, sys, st, a, stream) : 0;
  return 2 + (reset ? 1 : 0) + nh + ne + nsub + nc;
}

}  // namespace xnb
