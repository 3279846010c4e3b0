// Host-side launchers of the xnb kernels (internal; the public C ABI is include/xnb_gpu.h).
#pragma once
#include <string>

#include "xnb_internal.cuh"

namespace xnb {

// Largest settings of a batch that a launch's shared memory follows.
constexpr int kStageCapMax = 1024;       // candidates per stage of the neighbour build
constexpr uint32_t kMaxListBuf = 1024;   // entries per list buffer of its block-per-cell form
constexpr size_t kSmemPerBlock = 227 * 1024;  // what a block of an sm_103 may have

// Sets a kernel's attribute on the current device. Setting one that succeeds clears the
// thread's last error: that of a launch refused before it is kept for check_launch.
template <class Kernel>
inline void set_attribute(Kernel kern, cudaFuncAttribute what, int value) {
  if (cudaPeekAtLastError() == cudaSuccess) cudaFuncSetAttribute(kern, what, value);
}
// Raises a kernel's limit on dynamic shared memory. `most` is the largest that any
// launch of the kernel asks for, not this launch's: the limit belongs to the kernel,
// and a second host thread's launch may follow it.
template <class Kernel>
inline void raise_smem_limit(Kernel kern, size_t most) {
  set_attribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(most));
}

enum Precision : int { kFp64Exact = 0, kFp64 = 1, kMixed = 2 };

// Every launcher returns the number of kernels it enqueued.

// Work extent of a batch: high-water marks of the particle and cell pools.
struct Extent {
  uint32_t n_part;   // particles [0, n_part) are scanned; free slots have pcell == ~0u
  uint32_t n_cells;  // cells [0, n_cells); free cells have cell_sys == ~0u
  int nsys;
  int sm_count;
  int force_block;   // threads per block of the force traversal (multiple of 32, <= 256)
  int force_lanes;   // threads per particle of the mixed full-list traversal above kMixedSplitMax (1, 2 or 4)
  int far_coords;    // some resident system lies far from the coordinate origin (SysDesc::far_coords)
  int unpacked;      // some resident system reads the residual mirror, not packed residuals (SysDesc::packed_lo)
  int general;       // some resident system is not one of launch_force_walk's: unpacked, its origin not zero or
                     // SysDesc::plain_sums
  int dense;         // some resident system's cells hold half of what gives them a sub-grid, on average
  uint32_t list_slot;  // largest list slot of the resident systems
  int force_form;    // kForceThread or kForceStaged (mixed full-list traversal)
  uint32_t n_seg;    // cell segments of the staged traversal (DevArrays::seg)
};

// Mixed-precision force traversal forms: one thread per particle over global
// memory, or cell segments staged in shared memory (xnb_force_staged.cu).
constexpr int kForceThread = 0;
constexpr int kForceStaged = 1;
constexpr int kStagedSegCells = 8;  // x-adjacent cells of one row per staged segment

// Fused first half of velocity Verlet plus the displacement trigger:
// push_f_v_r(dt_scale 1) ; push_f_v(dt_scale 0.5) ; particle_displ_over.
int launch_first_half(const Extent& ex, const SysDesc* sys, SysState* st, const DevArrays& a,
                       bool do_push_r, bool do_push_v, bool do_trigger, double dt_scale_r,
                       double dt_scale_v, bool exact, int sys_only, cudaStream_t stream);

// zero_particle_force + lennard_jones_force (+ divide_force_by_type_scalar when the
// system asks for it), optionally fused with the second-half kick push_f_v(0.5).
// newton: FP64 / mixed paths walk the lower half of each list and deliver
// reactions with FP64 reductions (three kernels: zero, traverse, finish).
int launch_force(const Extent& ex, const SysDesc* sys, SysState* st, const DevArrays& a, int precision,
                 bool with_pe, bool second_half, int sys_only, cudaStream_t stream, bool newton = false);

// The mixed full-list forces in the two-stage form (xnb_force_mixed.cu): the same
// bits as one thread per particle, faster while the particles are too few to fill
// the GPU that way. Per call, two-stage / one-thread: 864 atoms 10 / 87 us, 32,000
// 43 / 96 us, 62,500 72 / 105 us, 131,072 135 / 137 us (178 / 165 us with
// energies). The line lies where three batches stepping at once on their own
// streams lose at no density: 10 steps of 55,296 atoms at 0.75, 0.84 and 1.0
// 731 / 705, 757 / 780 and 808 / 858 us, of 62,500 atoms 832 / 770, 876 / 835 and
// 933 / 950 us (one batch alone 920 / 1268 and 998 / 1289 us at 0.84).
// Short lists leave its second stage little and one thread's walk short: batches of
// more particles than kMixedSplitPerSlot times the list slot (which holds about 1.6
// times the mean list, and 16) keep the walk. Per graph step, two-stage / one-thread:
// at density 0.02 (slot 24) 16,384 atoms 67.6 / 67.3 us, 32,000 101 / 95, 48,668
// 155 / 143; at 0.08 (32) 32,000 67.1 / 69.0, 42,592 78.4 / 76.1; at 0.15 (40)
// 42,592 73.5 / 76.1, 48,668 84.9 / 84.2; at 0.2 (48) 48,668 80.7 / 83.8.
constexpr uint32_t kMixedSplitMax = XNB_MIXED_SPLIT_MAX, kMixedSplitPerSlot = 1200;
int launch_force_mixed(const Extent& ex, const SysDesc* sys, const SysState* st, const DevArrays& a, bool with_pe,
                       bool second_half, int sys_only, cudaStream_t stream);

// The mixed full-list forces of large batches, each list entry visited once by one
// thread per particle (xnb_force_mixed.cu), the same bits again: systems with
// packed residuals, their origin at zero and terms that PairSum takes
// (Extent::general is 0; other batches keep the marking walk of
// xnb_step_kernels.cu). The marking walk has the shorter chain per particle and
// wins while a call is a few waves of blocks. A call, marking / single-visit: 78,732
// atoms 113 / 135 us, 157,216 179 / 195 us, 364,500 299 / 310 us, 562,432 402 / 404
// us (with energies 443 / 440), 1M 639 / 629 us (710 / 690), 2M 1201 / 1154 us (1334
// / 1253). 10 steps, three batches at once: 562,432 atoms 5.31 / 4.70 ms, 2M 19.3 /
// 16.3 ms.
constexpr uint32_t kMixedWalkMin = 500000;
int launch_force_walk(const Extent& ex, const SysDesc* sys, const SysState* st, const DevArrays& a, bool with_pe,
                      bool second_half, int sys_only, cudaStream_t stream);

// The kernel of launch_force for full lists.
enum class ForceRoute {
  kPairs,       // FP64, FP64_EXACT: launch_force_pairs
  kStaged,      // mixed: launch_force_staged
  kTwoStage,    // launch_force_mixed
  kShortLists,  // the marking walk in its place, one thread per particle
  kWalk,        // launch_force_walk
  kMarks,       // the marking walk, force_lanes threads per particle
};
ForceRoute force_route(const Extent& ex, const DevArrays& a, int precision);
// whether it reads the batch's threads per particle, and threads per block
inline bool reads_force_lanes(const Extent& ex, ForceRoute r) {
  return (r == ForceRoute::kMarks || r == ForceRoute::kWalk) && !ex.unpacked;
}
inline bool reads_force_block(ForceRoute r) {
  return r == ForceRoute::kMarks || r == ForceRoute::kWalk || r == ForceRoute::kShortLists;
}

// FP64 and FP64_EXACT forces over full lists, or FP64 over their lower halves
// with FP64 reductions into cleared fields (newton; no kick) (xnb_force_pairs.cu).
int launch_force_pairs(const Extent& ex, const SysDesc* sys, const SysState* st, const DevArrays& a, int precision,
                       bool newton, bool with_pe, bool second_half, int sys_only, cudaStream_t stream);

// Compact list entries of the flagged systems after a build, and the staged
// mixed force traversal (+ kick) over the cell segments (xnb_force_staged.cu).
// all = true: every resident system's current lists (when the staged form is switched on)
int launch_compact_lists(const Extent& ex, const SysDesc* sys, SysState* st, const DevArrays& a, cudaStream_t stream,
                         bool all = false);
int launch_force_staged(const Extent& ex, const SysDesc* sys, SysState* st, const DevArrays& a, bool with_pe,
                        bool second_half, int sys_only, cudaStream_t stream);
size_t staged_smem_bytes();

// Marks systems for rebuild: all of them (init), or those with moved > 0.
int launch_mark_rebuild(const Extent& ex, SysState* st, int mode, int sys_only, unsigned int* any,
                        cudaStream_t stream);
int launch_clear_moved(const Extent& ex, SysState* st, cudaStream_t stream);

// Control block of the persistent step loop (device memory, zeroed before each launch).
struct StepCtl {
  GridBarrier bar;
  unsigned int fired[2];    // per step parity: an armed system's displacement trigger fired
  unsigned int steps_done;  // whole steps completed by the launch
  unsigned int stopped;     // 1: stopped after the first half of step steps_done (the trigger fired)
};
// Up to max_steps whole MD steps (first half + trigger, grid barrier, forces with
// the second-half kick, grid barrier) in one cooperative launch, one thread per
// particle, full lists; it stops after the first half of a step whose trigger
// fired. check: the first barrier waits for one block more than the launch has,
// so every wait runs out after wait_ns and the launch returns before changing
// any state (a test of the timeout path). Returns the number of launches.
int launch_steps_persistent(const Extent& ex, const SysDesc* sys, SysState* st, const DevArrays& a, int precision,
                            bool with_pe, StepCtl* ctl, int max_steps, bool check, cudaStream_t stream);

// move_particles + migrate + rebuild_amr + backup_r for systems with rebuild != 0.
// exact_backup = false keeps the backup position unencoded (FP64 and mixed paths).
int launch_rebin(const Extent& ex, const SysDesc* sys, SysState* st, const DevArrays& a, cudaStream_t stream,
                 bool exact_backup = true);
// backup_r alone.
// The displacement trigger's decision, the rebin and the build's resets in one
// cooperative launch, for batches it fits: a step without a rebuild then takes
// one launch here instead of twelve (a 50-step graph of 864 atoms: 0.84 -> 0.51 ms).
// The gain shrinks as the phases want more warps than one block per SM has; one
// block scans the cell counts, hence the limit on cells. A step of a graph (of an
// eager loop), fused / separate, mixed, density 0.84: 32,000 atoms 66 / 78 us (78 /
// 119), 97,556 151 / 159 (164 / 197), 131,072 182 / 191 (193 / 228), 256,000 322 /
// 323 (334 / 359); density 0.1: 9,261 cells 54 / 58 us (68 / 99), 13,824 66 / 64 (80 /
// 101), 17,576 80 / 75 (95 / 113), 42,875 132 / 101 (147 / 141). Both limits are on
// the near side of where a graph breaks even.
constexpr uint32_t kFusedRebinMaxParticles = 100000;
constexpr uint32_t kFusedRebinMaxCells = 16384;
bool fused_rebin_fits(const Extent& ex);
// build: the neighbour lists as well, for batches of few cells too sparse for
// sub-cell pruning to matter. One block per SM builds the lists slower than a launch
// of their own and saves two launches in each step. A step of a graph (of an eager
// loop), in here / on their own: 343 cells 28.6 / 31.1 us (35 / 46), 1,000 51.7 / 53.9
// (57 / 68), 1,331 66.5 / 65.5 at 32,000 atoms (71 / 79) and 57.0 / 57.5 at 27,436,
// 2,744 129.5 / 128.7 (134 / 142), 4,096 151 / 149 (157 / 162): graphs break even from
// 1,331 cells on, eager steps not by 4,913. The line is the graph's.
constexpr uint32_t kFusedBuildMaxCells = 1024;
bool fused_build_fits(const Extent& ex, int form, bool prune);
int launch_rebin_fused(const Extent& ex, const SysDesc* sys, SysState* st, const DevArrays& a, bool exact_backup,
                       bool build, int cap, int lbuf, bool check, cudaStream_t stream);
int launch_backup(const Extent& ex, const SysDesc* sys, SysState* st, const DevArrays& a, cudaStream_t stream);
// chunk_neighbors for systems with rebuild != 0: one pass writing each list
// into its particle's slot (statistics reset, the warp-per-cell build, and the
// block-per-cell build of the cells too large for it: three kernels). lbuf: the
// largest slot rounded up to 32 entries, 0 above 1024 or when no system has a
// slot yet; it sizes the shared-memory list buffers.
// form: kBuildRows (lane per particle, rows of three cells bulk-copied into
// shared memory, xnb_build_rows.cu) or kBuildWarp (lane per candidate, the
// 27-cell block staged per warp); cells neither handles go to the
// block-per-cell build.
// prune: cells with a sub-grid go to the sub-cell pruned build (xnb_build_sub.cu)
// when their system's sub-cell keys still describe its positions (keys_fresh:
// set by the rebin, cleared when positions are pushed).
// reset: clear the flagged systems' list statistics first (the fused rebin has).
constexpr int kBuildRows = 0;
constexpr int kBuildWarp = 1;
constexpr int kBuildHalf = 2;
int launch_neighbors(const Extent& ex, const SysDesc* sys, SysState* st, const DevArrays& a, int stage_cap,
                     int lbuf, cudaStream_t stream, int form = kBuildRows, bool prune = false, bool reset = true);
// the lane-per-particle build alone (cells it cannot take are appended to a.nbr_wide)
int launch_neighbors_rows(const Extent& ex, const SysDesc* sys, SysState* st, const DevArrays& a, cudaStream_t stream,
                          bool prune);
// the half-shell build (xnb_build_half.cu): pair masks of the systems whose
// cells all hold at most 64 particles, then the lists from the masks
int launch_neighbors_half_test(const Extent& ex, const SysDesc* sys, SysState* st, const DevArrays& a,
                               cudaStream_t stream);
int launch_neighbors_half_emit(const Extent& ex, const SysDesc* sys, SysState* st, const DevArrays& a,
                               cudaStream_t stream);
// the sub-cell pruned build of the cells listed in a.nbr_sub (cells with a
// neighbour of sub-grid side above 3 are passed on to a.nbr_wide)
int launch_neighbors_sub(const Extent& ex, const SysDesc* sys, SysState* st, const DevArrays& a, int stage_cap,
                         cudaStream_t stream);

// Reference-format chunk-neighbour streams of system sid (xnb_stream.cu):
// per-cell lengths (u16 units), the streams at cell_off, and the checker
// (counts[6]: format, order, self, range, far, missing).
int launch_stream_lengths(uint32_t sid, uint32_t ncells, const SysDesc* sys, const DevArrays& a, int T,
                          uint32_t* cell_len, int sm_count, cudaStream_t stream);
int launch_stream_write(uint32_t sid, uint32_t ncells, const SysDesc* sys, const DevArrays& a, int T,
                        const unsigned long long* cell_off, uint16_t* out, unsigned int* errors, int sm_count,
                        cudaStream_t stream);
int launch_stream_verify(uint32_t sid, uint32_t ncells, const SysDesc* sys, const DevArrays& a, int T,
                         const uint16_t* stream_data, uint64_t stream_len, const unsigned long long* cell_off,
                         unsigned long long* counts, int sm_count, cudaStream_t stream);

// On-device observables (xnb_observe.cu): simulation_stats of system sid into a
// scratch area of stats_scratch_bytes() (copy_stats reads it back: kinetic
// sum, potential, min/max |v|, min/max |f| and the count), and id sampling.
size_t stats_scratch_bytes();
int launch_stats(uint32_t sid, uint32_t npart, const SysDesc* sys, const DevArrays& a, void* scratch, int sm_count,
                 cudaStream_t stream);
int copy_stats(void* scratch, double* out6, unsigned long long* count_out, cudaStream_t stream);
int launch_sample(uint32_t sid, uint32_t npart, const SysDesc* sys, const DevArrays& a, const uint64_t* ids,
                  uint32_t n, double* out, int32_t* found, int sm_count, cudaStream_t stream);

// gravitational_force over the per-particle lists (xnb_functors.cu). Masses per
// particle type (at most kMaxTypes); pre_hi_f = rcut^2 + the FP32 prefilter's
// proven margin. flags bit 0: a particle type without a mass.
constexpr int kMaxTypes = 16;
struct GravParams {
  double G;
  double rcut2;
  float pre_hi_f;
  int ntypes;
  double mass[kMaxTypes];
};
int launch_gravity(const Extent& ex, const SysDesc* sys, const SysState* st, const DevArrays& a, int precision,
                   bool with_pe, bool accumulate, int sys_only, const GravParams& gp, unsigned int* flags,
                   cudaStream_t stream);
// field::type by id for system sid (ids sorted ascending); matched += particles found
int launch_set_types(uint32_t sid, uint32_t npart, const SysDesc* sys, const DevArrays& a, const uint64_t* ids,
                     const uint8_t* types, uint32_t n, unsigned long long* matched, int sm_count, cudaStream_t stream);

// Device placement of a system uploaded in input order into the rebin scratch
// (xnb_place.cu). flags: bit 0 a position outside any representable cell, bit 1
// a cell above kPlaceMaxCell particles (the host then places the system).
constexpr uint32_t kPlaceMaxCell = 4096;
struct PlaceArgs {
  double origin[3];
  double cell_size;
  int dims[3];
  uint32_t poff, coff, n, ncells, sys_slot;
};
int launch_place(const PlaceArgs& P, const DevArrays& a, unsigned int* flags, int sm_count, cudaStream_t stream);

// Exclusive scan of u32 counts into u64 offsets (n elements; out has n+1 entries).
// With gate != nullptr the kernels return at once while *gate == 0.
int launch_scan_u32_to_u64(const uint32_t* in, unsigned long long* out, uint32_t n,
                           unsigned long long* block_scratch, cudaStream_t stream,
                           const unsigned int* gate = nullptr);
size_t scan_scratch_elems(uint32_t n);


// Allocation-free neighbour build of one system (xnb_static_scratch.cu): scratch
// in a file-scope device array; returns 0, -1 (size above the array's limit,
// *err says which) or -2 (CUDA error). cap is clamped to 2^32 - 1 entries.
int launch_neighbors_static(const SysDesc& S, uint64_t ncells, uint64_t n, const double* rx, const double* ry,
                            const double* rz, const uint32_t* cell_start, const uint32_t* cell_n, uint32_t* nbr,
                            uint64_t cap, uint32_t* nbr_start, uint32_t* nbr_cnt, unsigned long long* total_out,
                            cudaStream_t stream, std::string* err);

}  // namespace xnb
