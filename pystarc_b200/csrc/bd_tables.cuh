// The stepper and evaluation kernels of one precision and torque mode, as launchable pointers.  Each
// of the four combinations is compiled in a source of its own (bd_table_*.cu), so that the library
// builds in parallel.
#pragma once

#include "bd_kernels.cuh"
#include "bd_multi.cuh"
#include "bd_pose.cuh"
#include "bd_split.cuh"
#include "bd_surrogate.cuh"

namespace bd {

constexpr int kGroups[5] = {1, 4, 8, 16, 32};  // lanes per trajectory of step_kernel and eval_*_kernel

struct SplitKernels {
  void *first, *mid, *last;  // scalar kernel: begin, end + begin, end
  void *fwd, *fwd_long, *fwd_packed, *rev;  // packed: null in FP64
};

struct KernelTable {
  void *pose[5], *atoms[5], *step[5];  // by kGroups
  void *pose_block, *pose_block_contact, *pose_fwd, *pose_rev;  // evaluation by whole warps
  void *warp, *warp_capped;            // step_kernel_warp without a register cap and at 128
  void *sur_begin, *sur_end;
  SplitKernels split, multi;           // of one system, of a heterogeneous batch
};

template <typename FT, bool TQ, class TAB>
SplitKernels split_kernels() {
  void* packed = nullptr;
  if constexpr (sizeof(FT) == 4) packed = (void*)&split_fwd_kernel<FT, TQ, FWD_PACKED, TAB>;
  return {(void*)&split_step_kernel<FT, TQ, false, true, TAB>, (void*)&split_step_kernel<FT, TQ, true, true, TAB>,
          (void*)&split_step_kernel<FT, TQ, true, false, TAB>, (void*)&split_fwd_kernel<FT, TQ, FWD_ONE, TAB>,
          (void*)&split_fwd_kernel<FT, TQ, FWD_LONG, TAB>, packed, (void*)&split_rev_kernel<FT, TQ, TAB>};
}

template <typename FT, bool TQ>
KernelTable make_table() {
  return {{(void*)&eval_pose_kernel<FT, 1, TQ>, (void*)&eval_pose_kernel<FT, 4, TQ>, (void*)&eval_pose_kernel<FT, 8, TQ>,
           (void*)&eval_pose_kernel<FT, 16, TQ>, (void*)&eval_pose_kernel<FT, 32, TQ>},
          {(void*)&eval_atoms_kernel<FT, 1, TQ>, (void*)&eval_atoms_kernel<FT, 4, TQ>,
           (void*)&eval_atoms_kernel<FT, 8, TQ>, (void*)&eval_atoms_kernel<FT, 16, TQ>,
           (void*)&eval_atoms_kernel<FT, 32, TQ>},
          {(void*)&step_kernel<FT, 1, TQ>, (void*)&step_kernel<FT, 4, TQ>, (void*)&step_kernel<FT, 8, TQ>,
           (void*)&step_kernel<FT, 16, TQ>, (void*)&step_kernel<FT, 32, TQ>},
          (void*)&pose_block_kernel<FT, TQ, false>,
          (void*)&pose_block_kernel<FT, TQ, true>,
          (void*)&pose_fwd_kernel<FT, TQ>,
          (void*)&pose_rev_kernel<FT, TQ>,
          (void*)&step_kernel_warp<FT, TQ, 1>,
          (void*)&step_kernel_warp<FT, TQ, 2>,
          (void*)&sur_begin_kernel<FT, TQ>,
          (void*)&sur_end_kernel<FT, TQ>,
          split_kernels<FT, TQ, OneTab>(),
          split_kernels<FT, TQ, MultiTab>()};
}

KernelTable table_mixed();
KernelTable table_mixed_torque();
KernelTable table_fp64();
KernelTable table_fp64_torque();

}  // namespace bd
