// Heterogeneous batch: trajectories of several receptor-ligand systems (each
// with its own grids, atoms, reaction pairs and run parameters) share one slot
// pool and the launches of the split stepper.  The trajectory index space is the
// concatenation of the systems' ranges; a slot stores the global index, and the
// system is found by a binary search over the prefix sums.  Every per-system
// quantity is read from device tables of DevSystem / DevSim, and the step is that
// of the single-system split stepper (its kernels over a MultiTab).  No reference
// counterpart (the reference runs one system per process).
#pragma once

#include "bd_kernels.cuh"

namespace bd {

struct MultiTab {
  const DevSystem* sys_;    // n_sys systems
  const DevSim* sim_;       // n_sys run parameters (ctr: the shared counters)
  const long long* base;    // n_sys + 1: first global index of each system, then the total
  int n_sys;
  long long total;
  unsigned long long* ctr;  // shared counters: pending cursor over global indices, tallies
  int small, large;         // every ligand has at most 32, at least 128 atoms, and no contact forces
  int largest;              // atoms of the largest ligand

  // the interface of the split stepper's kernels (OneTab is the single-system one)
  __device__ __forceinline__ const DevSystem& sys(int k) const { return sys_[k]; }
  __device__ __forceinline__ const DevSim& sim(int k) const { return sim_[k]; }
  __device__ __forceinline__ int locate(int& id) const;
  __device__ __forceinline__ int global_id(int k, int id) const { return (int)(base[k] + id); }
  __device__ __forceinline__ bool large_ligands() const { return large; }
  __device__ __forceinline__ int largest_ligand() const { return largest; }
  __device__ __forceinline__ void refill(Traj& tr, int& k, bool& dead, int lane) const;
  __device__ __forceinline__ bool overlap(int k, const double cn[3], bool need, int lane, const RecView&) const;
};

// System of global trajectory index g (the last s with base[s] <= g).
__device__ __forceinline__ int sys_of(const MultiTab& T, long long g) {
  int lo = 0, hi = T.n_sys - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    if (T.base[mid] <= g) lo = mid;
    else hi = mid - 1;
  }
  return lo;
}

// Trajectory id (global) -> its system; id becomes the system's own.
__device__ __forceinline__ int MultiTab::locate(int& id) const {
  const int k = sys_of(*this, id);
  id = (int)(id - base[k]);
  return k;
}

// Overlap test where every lane's trajectory may belong to another system: from the lane's own
// occupancy grid, or the warp sweeping the receptor chunks of the lanes whose system has none.
__device__ __forceinline__ bool MultiTab::overlap(int k, const double cn[3], bool need, int lane,
                                                  const RecView&) const {
  const unsigned FULL = 0xffffffffu;
  const bool grid = need && sys_[k].ov_cell;
  bool mine = grid && overlap_cells(sys_[k], cn);
  unsigned m = __ballot_sync(FULL, need && !grid);
  while (m) {
    const int j = __ffs(m) - 1;
    m &= m - 1;
    double cj[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) cj[i] = __shfl_sync(FULL, cn[i], j);
    const bool hit = overlap_any<32>(sys_[__shfl_sync(FULL, k, j)], cj, lane, FULL, RecView{nullptr, nullptr});
    if (lane == j) mine = hit;
  }
  return mine;
}

// Lanes whose trajectory ended take the next global indices (one atomic per warp).
__device__ __forceinline__ void MultiTab::refill(Traj& tr, int& k, bool& dead, int lane) const {
  const unsigned FULL = 0xffffffffu;
  const bool want = !dead && tr.status != ST_RUNNING;
  const unsigned wm = __ballot_sync(FULL, want);
  if (!wm) return;
  const int leader = __ffs(wm) - 1;
  unsigned long long first = 0;
  if (lane == leader) first = atomicAdd(ctr + C_PENDING, (unsigned long long)__popc(wm));
  first = __shfl_sync(FULL, first, leader);
  if (want) {
    const long long g = (long long)(first + __popc(wm & ((1u << lane) - 1u)));
    if (g >= total) {
      tr.status = ST_EMPTY;
      dead = true;
    } else {
      k = sys_of(*this, g);
      start_trajectory(sim_[k], (int)(g - base[k]), tr);
    }
  }
}

static __global__ void init_slots_multi_kernel(MultiTab T, SlotBuf B, int n_slots) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_slots) return;
  const int s = sys_of(T, i);
  Traj tr;
  start_trajectory(T.sim(s), (int)(i - T.base[s]), tr);
  tr.id = i;  // slots hold global indices
  store_slot(B, i, tr);
}

}  // namespace bd
