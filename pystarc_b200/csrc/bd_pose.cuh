// Force evaluation of a batch of poses (the reference's __call__,
// pystarc/forces/gpu_batch_engine.py:531-605) by the split stepper's force code.
//
//   pose_block_kernel  one block per pose, for batches that would leave SMs idle otherwise: its
//                      eight warps share the ligand atoms and then the sweep of Born direction 2
//   pose_fwd_kernel    forces on the ligand atoms, one warp per pose
//   pose_rev_kernel    Born direction 2, one warp per pose, added to the forces of the former
//
// One kernel for both parts held 168 registers a thread (12 warps per SM); apart, the ligand atoms run at
// 128 and 16 warps, the sweep at 64 and 32 in mixed precision without torque, at 80 and 24 with torque, at
// 128 and 16 in FP64.  The last two run in blocks of one warp, handed out by the device: poses differ in
// cost, and resident blocks of eight warps that stride left the last of their rounds nearly empty (3,200 +
// 18 atoms, mixed, 8,000 poses 159 -> 99 us, 100,000 820 -> 700).  Every sum keeps the order of the one-warp
// evaluation.
#pragma once

#include "bd_split.cuh"

namespace bd {

// Poses as the two evaluation entry points give them: centroids with quaternions (w, x, y, z) or
// rotation matrices, and the ligand atoms placed from the body frame or given in the lab frame.
struct PoseBatch {
  long long n;
  const double* cen;
  const double* rot;
  int rot_is_matrix;
  const double* atoms;  // n * n_lig * 3 lab positions, or NULL: placed from the pose
  double *F, *T, *E;
};

struct BatchSrc {
  const PoseBatch& P;
  long long t;
  __device__ __forceinline__ void load(double c[3], double R[9]) const {
#pragma unroll
    for (int i = 0; i < 3; ++i) c[i] = P.cen[3 * t + i];
    if (P.rot_is_matrix) {
#pragma unroll
      for (int i = 0; i < 9; ++i) R[i] = P.rot[9 * t + i];
    } else {
      const double q[4] = {P.rot[4 * t], P.rot[4 * t + 1], P.rot[4 * t + 2], P.rot[4 * t + 3]};
      quat_to_rot(q, R);
    }
  }
};

// Ligand atom positions of a pose of the batch.
struct BatchPos {
  const double* R;
  const double* c;
  const double* atoms;  // this pose's lab positions, or NULL
  __device__ __forceinline__ void operator()(int i, const double4& a, double ro[3], double x[3]) const {
    if (atoms) PosFromAtoms{atoms, c}(i, a, ro, x);
    else PosFromPose{R, c}(i, a, ro, x);
  }
};

__device__ __forceinline__ bool needs_reverse(const DevSystem& S, const double c[3]) {
  return (S.terms & 4u) && S.born_rev && norm3(c[0], c[1], c[2]) - S.rec_max_r < S.lig_born_rho;
}

// Which form evaluates n poses, by the work of one pose that warps can share: units of 32 ligand atoms, or of
// 32 receptor atoms to sweep.
//   EVAL_BLOCK  a block per pose: short batches wait for one pose's chain, which eight warps shorten (3,200 +
//               18 atoms FP64, 37 poses: 55 us in one kernel, 58 by warps, 23 by blocks).  With little to
//               share a pose keeps one warp of eight busy, and contact forces come from one warp anyway
//   EVAL_ONE    both parts in one kernel, four warps a block: short batches of light poses, where a second
//               launch is a quarter of the time (87 + 18 atoms FP64, 600 poses: 13 us, 19 by warps, 21 by
//               blocks), and medium ones in FP64, whose registers the 128 of the other forms do not hold
//   EVAL_WARPS  a kernel for the ligand atoms and one for the sweep, a warp per pose
// The lines, us by blocks / by warps: 3,200 + 18 atoms FP64 1,500 poses 60 / 67, 2,000 75 / 71; 1,701 + 1,401
// mixed 1,184 177 / 189, 1,500 216 / 198; FP64 without a sweep 3,000 259 / 312; 213 + 176 FP64 600 28 / 36,
// 1,000 40 / 40 and 29 in one; contact forces, 213 + 176 FP64, 37 poses 443 / 460 and 426 in one.
enum { EVAL_ONE, EVAL_BLOCK, EVAL_WARPS };
inline int eval_form(long long n, int n_sm, int units, bool fp64, bool rev, bool wca) {
  const int block = units >= 32 ? (fp64 && !rev ? 24 : 12) : units >= 6 && !wca ? 6 : 0;  // poses per SM
  const int one = fp64 && units < 32 ? 9 : units < 8 ? (rev ? 20 : 6) : 0;
  return n <= (long long)block * n_sm ? EVAL_BLOCK : n <= (long long)one * n_sm ? EVAL_ONE : EVAL_WARPS;
}

// CONTACT: systems with contact forces.  One warp adds them to the lanes' sums, atom by atom as in the
// one-warp evaluation, while the others wait; a kernel of its own, so that systems without keep theirs.
template <typename FT, bool TORQUE, bool CONTACT>
__global__ void __launch_bounds__(256, 2) pose_block_kernel(const __grid_constant__ DevSystem S,
                                                            const __grid_constant__ PoseBatch P) {
  using V4 = typename Vec4<FT>::type;
  constexpr int NC = kForwardNc<TORQUE, true>;
  constexpr int NV = (TORQUE ? 16 : 8) * kSplitBuf<FT>;
  union Shared {
    double fwd[2 * 8 * NC * 32];
    V4 rev[NV];
    __device__ Shared() {}
  };
  __shared__ Shared sh;
  __shared__ double out[16];
  __shared__ double sums[CONTACT ? (TORQUE ? 6 : 3) : 1][32];
  __shared__ int cnts[16];
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  Counts cnt{0, 0, 0};
  for (long long t = blockIdx.x; t < P.n; t += gridDim.x) {
    const BatchSrc src{P, t};
    const Pose<BatchSrc> pose(src);
    double tot[4];
    const BatchPos pos{pose.R, pose.c, P.atoms ? P.atoms + t * S.n_lig * 3 : nullptr};
    auto contact = [&](double* tot) {
      if constexpr (CONTACT) {
        if (!(S.terms & 8u) || !(norm3(pose.c[0], pose.c[1], pose.c[2]) < S.wca_act)) return;
        constexpr int N = TORQUE ? 6 : 3;
        if (warp < N) sums[warp][lane] = tot[0];
        __syncthreads();
        if (warp == 0) {
          double f[3] = {sums[0][lane], sums[1][lane], sums[2][lane]}, u[3] = {0, 0, 0};
          if (TORQUE) {
#pragma unroll
            for (int i = 0; i < 3; ++i) u[i] = sums[N - 3 + i][lane];
          }
          group_contact<32, TORQUE>(S, pose.c, lane, FULL, pos, f, u);
#pragma unroll
          for (int i = 0; i < 3; ++i) {
            sums[i][lane] = f[i];
            if (TORQUE) sums[N - 3 + i][lane] = u[i];
          }
        }
        __syncthreads();
        if (warp < N) tot[0] = sums[warp][lane];
      }
    };
    group_forward<FT, TORQUE, true>(S, pos, lane, warp, 8, 1, sh.fwd, S.terms & 1u, S.terms & 2u, tot, cnt, contact);
    if (lane == 0 && warp < NC) out[warp] = tot[0];
    const bool rev = needs_reverse(S, pose.c);
    double r[3] = {0, 0, 0}, u[3] = {0, 0, 0};
    __syncthreads();
    if (rev) {
      unsigned nr = 0;
      group_reverse_born<FT, TORQUE, true>(S, src, lane, warp, 8, 1, sh.rev, TORQUE ? sh.rev + 8 * kSplitBuf<FT> : sh.rev,
                                     cnts, r, u, nr);
      const double* sum = warp == 0 ? r : u;
      if (warp < 2) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          const double v = gsum<32>(sum[i], FULL);
          if (lane == 0) out[8 + 3 * warp + i] = v;
        }
      }
      __syncthreads();
    }
    if (threadIdx.x < 3) {
      const int i = threadIdx.x;
      const double* v = out + 8;
      double f = out[i], tq = TORQUE ? out[3 + i] : 0.0;
      if (rev) {
        // the reverse-Born force on the receptor, rotated to the lab frame, acts on the ligand with the
        // opposite sign
        const double R0 = i == 0 ? pose.R[0] : i == 1 ? pose.R[3] : pose.R[6],
                     R1 = i == 0 ? pose.R[1] : i == 1 ? pose.R[4] : pose.R[7],
                     R2 = i == 0 ? pose.R[2] : i == 1 ? pose.R[5] : pose.R[8];
        f = f - (R0 * v[0] + R1 * v[1] + R2 * v[2]);
        if (TORQUE) tq = tq - (R0 * v[3] + R1 * v[4] + R2 * v[5]);
      }
      P.F[3 * t + i] = f;
      P.T[3 * t + i] = tq;
      if (i == 0) P.E[t] = out[NC - 1];
    }
    __syncthreads();
  }
}

template <typename FT, bool TORQUE>
__global__ void __launch_bounds__(32, 16) pose_fwd_kernel(const __grid_constant__ DevSystem S,
                                                          const __grid_constant__ PoseBatch P) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x;
  Counts cnt{0, 0, 0};
  for (long long t = blockIdx.x; t < P.n; t += gridDim.x) {
    const Pose<BatchSrc> pose(BatchSrc{P, t});
    double f[3], tq[3], e;
    group_forces<FT, 32, TORQUE, true, BatchPos, false>(
        S, pose.c, pose.R, lane, FULL, BatchPos{pose.R, pose.c, P.atoms ? P.atoms + t * S.n_lig * 3 : nullptr}, f, tq, e,
        cnt, RecView{nullptr, nullptr}, S.terms);
    if (lane < 3) P.F[3 * t + lane] = lane == 0 ? f[0] : lane == 1 ? f[1] : f[2];
    else if (lane < 6) P.T[3 * t + lane - 3] = lane == 3 ? tq[0] : lane == 4 ? tq[1] : tq[2];
    else if (lane == 6) P.E[t] = e;
  }
}

template <typename FT, bool TORQUE>
__global__ void __launch_bounds__(32, sizeof(FT) == 4 ? (TORQUE ? 24 : 32) : 16) pose_rev_kernel(
    const __grid_constant__ DevSystem S, const __grid_constant__ PoseBatch P) {
  using V4 = typename Vec4<FT>::type;
  __shared__ V4 buf[kSplitBuf<FT>];
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x;
  unsigned nr = 0;
  for (long long t = blockIdx.x; t < P.n; t += gridDim.x) {
    const double c[3] = {P.cen[3 * t], P.cen[3 * t + 1], P.cen[3 * t + 2]};
    if (!needs_reverse(S, c)) continue;
    const BatchSrc src{P, t};
    double r[3] = {0, 0, 0}, u[3] = {0, 0, 0};
    lean_reverse_born<FT, TORQUE, true>(S, src, lane, buf, r, u, nr);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
      r[i] = gsum<32>(r[i], FULL);
      if (TORQUE) u[i] = gsum<32>(u[i], FULL);
    }
    if (lane < 3) {
      const Pose<BatchSrc> pose(src);
      const double R0 = lane == 0 ? pose.R[0] : lane == 1 ? pose.R[3] : pose.R[6],
                   R1 = lane == 0 ? pose.R[1] : lane == 1 ? pose.R[4] : pose.R[7],
                   R2 = lane == 0 ? pose.R[2] : lane == 1 ? pose.R[5] : pose.R[8];
      P.F[3 * t + lane] = P.F[3 * t + lane] - (R0 * r[0] + R1 * r[1] + R2 * r[2]);
      if (TORQUE) P.T[3 * t + lane] = P.T[3 * t + lane] - (R0 * u[0] + R1 * u[1] + R2 * u[2]);
    }
  }
}

}  // namespace bd
