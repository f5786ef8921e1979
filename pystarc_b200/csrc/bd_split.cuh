// Split stepper: one BD step as a scalar kernel over the slots and two force kernels over lists
// of poses, instead of one fused persistent kernel.
//
//   split_step_kernel  one lane per slot: the end of the previous step (step_move, overlap test,
//                      step_end, statistics, refill of ended trajectories from the pending pool)
//                      and the beginning of the next one (reaction test, escape/return), which
//                      lists the poses whose forces are needed
//   split_fwd_kernel   forces on the ligand atoms (grid, far-field, contact) of the listed poses
//   split_rev_kernel   Born direction 2 of the listed poses that reach the ligand Born grid
//
// The force kernels take one pose per warp from their list, so the warps of a pool share its
// poses evenly whatever its size: with the forces inside the scalar kernel, a warp evaluated its
// own 32 trajectories one after another, and a pool of 8,000 kept 250 warps busy on 148 SMs
// (protein + small ligand, 8,000 slots: 74 us of forces in that kernel; 6,000 slots of a
// 1,401-atom ligand: 1,140 us).  Each kernel also gets the registers that suit it: the scalar
// step and the forward stencils 128, the latency-bound sweep of direction 2 64 in mixed precision (twice
// the warps), 80 with torque, 128 in FP64.
// Candidates of the sweep (receptor atoms inside the ligand's Born box, in the ligand frame) go
// to a per-warp buffer in shared memory and are drained in whole groups of 32, entry i by lane i
// mod 32, in the order of the fused kernel's ring: every lane sums the same terms in the same
// order, so the forces, and so the trajectories, are those of the fused stepper.  The same keyed
// Philox stream drives both (gpu_batch_simulator.py:783-1254 is the step being split).
#pragma once

#include "bd_kernels.cuh"

namespace bd {

// Candidate entries per warp of the sweep (whole groups of 32 are drained).
template <typename FT>
constexpr int kSplitBuf = sizeof(FT) == 4 ? 128 : 64;
constexpr int kStepBlock = 128;  // threads of a scalar-kernel block

// Per-slot scratch of one BD step.
struct SplitBuf {
  double* F;       // 3 * cap: forces on the ligand atoms; the step's total force once complete
  double* T;       // 3 * cap
  double* rv;      // 6 * cap: Born direction 2 sums r (ligand frame) and u, from the sweep (64-bit indexes:
                   // the pose arrays allow 2^29 slots)
  double* rprev;   // cap: |c| at the end of the previous step (statistics)
  int8_t* mode;    // 0: no step; 1: F, T to be used as they are; 2: reused (complete);
                   // 3: F, T plus the Born direction 2 sums in rv
  int* flist;      // slots listed for split_fwd_kernel this step
  int* rlist;      // slots listed for split_rev_kernel this step
  int* cnt;        // two sets of {flist length, rlist length, their cursors}, used by steps in
                   // turn: a step's scalar kernel fills one set and clears the other
};

// Where a force kernel reads a pose: here a slot of the stepper's pool.
struct SlotSrc {
  const SlotBuf& B;
  int slot;
  __device__ __forceinline__ void load(double c[3], double R[9]) const {
    const double q[4] = {B.q[slot], B.q[B.cap + slot], B.q[2 * B.cap + slot], B.q[3 * B.cap + slot]};
#pragma unroll
    for (int i = 0; i < 3; ++i) c[i] = B.c[i * B.cap + slot];
    quat_to_rot(q, R);
  }
};

// One receptor-ligand system for all slots.
struct OneTab {
  DevSystem S;
  DevSim P;
  __device__ __forceinline__ const DevSystem& sys(int) const { return S; }
  __device__ __forceinline__ const DevSim& sim(int) const { return P; }
  __device__ __forceinline__ int locate(int&) const { return 0; }  // trajectory id -> system, local id
  __device__ __forceinline__ int global_id(int, int id) const { return id; }
  // ligands worth sharing among warps: every one of at least 128 atoms, no contact forces
  __device__ __forceinline__ bool large_ligands() const { return S.n_lig >= 128 && !S.wca; }
  __device__ __forceinline__ int largest_ligand() const { return S.n_lig; }  // atoms
  __device__ __forceinline__ void refill(Traj& tr, int&, bool& dead, int lane) const { warp_refill(P, tr, dead, lane); }
  __device__ __forceinline__ bool overlap(int, const double cn[3], bool need, int lane, const RecView& v) const {
    return warp_overlap(S, cn, need, lane, v);
  }
};

// Append the lanes with `eval` to flist and those with `rev` (which have `eval` too) to rlist: one
// atomic per warp on the pair of their lengths.
__device__ __forceinline__ void warp_append(const SplitBuf& U, int set, bool eval, bool rev, int slot, int lane) {
  const unsigned me = __ballot_sync(0xffffffffu, eval), mr = __ballot_sync(0xffffffffu, rev);
  if (!me) return;
  unsigned long long at = 0;
  const int leader = __ffs(me) - 1;
  if (lane == leader)
    at = atomicAdd(reinterpret_cast<unsigned long long*>(U.cnt + set),
                   (unsigned long long)__popc(mr) << 32 | (unsigned long long)__popc(me));
  at = __shfl_sync(0xffffffffu, at, leader);
  const unsigned below = (1u << lane) - 1u;
  if (eval) U.flist[(int)(at & 0xffffffffull) + __popc(me & below)] = slot;
  if (rev) U.rlist[(int)(at >> 32) + __popc(mr & below)] = slot;
}

// END: finish the step begun by the previous launch of this kernel; BEGIN: begin the next one.
// Warp w of block b takes the slots of chunk w * gridDim.x + b, so a small pool spreads over the SMs.
template <typename FT, bool TORQUE, bool END, bool BEGIN, class TAB>
__global__ void __launch_bounds__(kStepBlock, 4) split_step_kernel(const __grid_constant__ TAB T, SlotBuf B,
                                                                   const int* __restrict__ n_live, SplitBuf U,
                                                                   int set) {
  const int live = *n_live;
  if (blockIdx.x == 0 && threadIdx.x < 4) {
    U.cnt[4 * (1 - set) + threadIdx.x] = 0;
    if (!BEGIN) U.cnt[4 * set + threadIdx.x] = 0;
  }
  if ((long long)blockIdx.x * 32 >= live) return;  // no slots for this block
  const DevSim& P0 = T.sim(0);
  const BlockShared sh = END ? block_shared_begin(T.sys(0), P0) : BlockShared{RecView{nullptr, nullptr}, nullptr};
  const int lane = threadIdx.x & 31;
  const int n_warps = (gridDim.x * blockDim.x) >> 5;
  Tally tl{};
  for (long long base = 32ll * ((threadIdx.x >> 5) * gridDim.x + blockIdx.x); base < live; base += 32ll * n_warps) {
    const int slot = (int)base + lane;
    const bool own = slot < live;
    Traj tr{};
    tr.status = ST_EMPTY;
    int k = 0;
    if (own) {
      load_slot(B, slot, tr);
      k = T.locate(tr.id);
    }
    bool keep = false;  // F, T in the scratch are the forces at the slot's pose
    if (END) {
      const DevSystem& S = T.sys(k);
      const DevSim& P = T.sim(k);
      // everything the slot may need is loaded at once, before its mode is known
      int mode = 0;
      double F[3] = {0, 0, 0}, Tq[3] = {0, 0, 0}, rv[6] = {0, 0, 0, 0, 0, 0};
      if (own) {
        mode = (int)U.mode[slot];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          F[i] = U.F[3 * slot + i];
          Tq[i] = U.T[3 * slot + i];
          rv[i] = U.rv[6 * (size_t)slot + i];
          rv[3 + i] = U.rv[6 * (size_t)slot + 3 + i];
        }
      }
      const bool need = mode != 0;
      double R[9] = {1, 0, 0, 0, 1, 0, 0, 0, 1}, r = 0;
      if (need) {
        quat_to_rot(tr.q, R);
        r = norm3(tr.c[0], tr.c[1], tr.c[2]);
        if (mode == 3) {
          // the reverse-Born force on the receptor, rotated to the lab frame, acts on the ligand
          // with the opposite sign
#pragma unroll
          for (int i = 0; i < 3; ++i) F[i] = F[i] - (R[3 * i] * rv[0] + R[3 * i + 1] * rv[1] + R[3 * i + 2] * rv[2]);
          if (TORQUE) {
#pragma unroll
            for (int i = 0; i < 3; ++i)
              Tq[i] = Tq[i] - (R[3 * i] * rv[3] + R[3 * i + 1] * rv[4] + R[3 * i + 2] * rv[5]);
          }
        }
      }
      const Keyed key = traj_key(P, tr.id);
      const uint32_t s = (uint32_t)tr.steps;
      double cn[3] = {0, 0, 0}, qn[4] = {1, 0, 0, 0}, dt = 0;
      bool ok = true;
      if (need) ok = step_move<FT>(S, P, key, s, tr, R, r, F, Tq, cn, qn, dt);
      int st = tr.status;
      if (need && !ok) {
        tl.nonfinite += 1;
        st = ST_ERROR;
      }
      const bool ovl = T.overlap(k, cn, need && ok && P.overlap, lane, sh.v);
      if (need && ok) {
        const double c0[3] = {tr.c[0], tr.c[1], tr.c[2]};
        st = step_end(S, P, key, s, tr, R, cn, qn, !ovl, dt, tl);
        if (P.stats) {
          stats_step(S, P, tr, s, U.rprev[slot], dt, c0, R, sh.stats);
          trace_step(P, tr, s, F, dt);
          if (st == ST_REACTED) stats_encounter(P, tr, s, true);
        }
      }
      if (need && st != ST_RUNNING) {
        tr.status = st;
        P.out_status[tr.id] = (int8_t)st;
        P.out_steps[tr.id] = tr.steps;
        P.out_returns[tr.id] = tr.rets;
        tl.reacted += st == ST_REACTED;
        tl.escaped += st == ST_ESCAPED;
        tl.maxsteps += st == ST_MAXSTEPS;
      }
      bool dead = !own;
      T.refill(tr, k, dead, lane);
      // rejected and still running: the next step starts from the same pose with these forces
      keep = need && ok && ovl && st == ST_RUNNING;
      if (BEGIN && keep && mode != 2) {
#pragma unroll
        for (int i = 0; i < 3; ++i) {
          U.F[3 * slot + i] = F[i];
          U.T[3 * slot + i] = Tq[i];
        }
      }
    }
    if (BEGIN) {
      const DevSystem& S = T.sys(k);
      const DevSim& P = T.sim(k);
      const bool run = own && tr.status == ST_RUNNING;
      const uint32_t s = (uint32_t)tr.steps;
      if (run && P.stats) U.rprev[slot] = norm3(tr.c[0], tr.c[1], tr.c[2]);
      double R[9], r = 0;
      int st = ST_EMPTY;
      const int rets0 = tr.rets;
      if (run) {
        st = step_begin(S, P, traj_key(P, tr.id), s, tr, R, r, tl);
        if (P.stats && st == ST_REACTED) stats_encounter(P, tr, s, false);
      }
      const bool need = run && st == ST_RUNNING;
      const bool reuse = need && keep && tr.rets == rets0;
      const bool eval = need && !reuse;
      const bool rev = eval && S.born_rev && r - S.rec_max_r < S.lig_born_rho;
      warp_append(U, 4 * set, eval, rev, slot, lane);
      if (run && st != ST_RUNNING) {
        tr.status = st;
        P.out_status[tr.id] = (int8_t)st;
        P.out_steps[tr.id] = tr.steps;
        P.out_returns[tr.id] = tr.rets;
        tl.reacted += st == ST_REACTED;
        tl.escaped += st == ST_ESCAPED;
        tl.maxsteps += st == ST_MAXSTEPS;
      }
      if (own) U.mode[slot] = (int8_t)(need ? (reuse ? 2 : rev ? 3 : 1) : 0);
    }
    if (own) {
      tr.id = T.global_id(k, tr.id);
      store_slot(B, slot, tr);
    }
  }
  flush_tally(P0, tl, true);
  if (END) stats_block_end(P0, sh.stats);
}

// The next turn of a warp after its first: the cursor counts the turns taken beyond one per warp.
__device__ __forceinline__ int next_item(int* cursor, int n_warps, int lane) {
  int j = 0;
  if (lane == 0) j = n_warps + atomicAdd(cursor, 1);
  return __shfl_sync(0xffffffffu, j, 0);
}

// The pose of a source: centre and rotation.  The rotation is left as a set of values, as the fused
// stepper has it: otherwise the compiler may fuse its arithmetic with the atoms' and round the
// positions differently.
template <class SRC>
struct Pose {
  double c[3], R[9];
  __device__ __forceinline__ explicit Pose(const SRC& src) {
    src.load(c, R);
#pragma unroll
    for (int i = 0; i < 9; ++i) asm volatile("" : "+d"(R[i]));
  }
};

// Lane i of 8 or 32 stores component i of the six.
__device__ __forceinline__ void store_force(const SplitBuf& U, int slot, int i, const double f[3], const double t[3]) {
  const double v = i == 0 ? f[0] : i == 1 ? f[1] : i == 2 ? f[2] : i == 3 ? t[0] : i == 4 ? t[1] : t[2];
  if (i < 3) U.F[3 * slot + i] = v;
  else if (i < 6) U.T[3 * slot + i - 3] = v;
}

// Forces on the ligand atoms of a pose for ligands of at most 32 atoms, by 8 lanes: lane l takes atoms
// l, l + 8, l + 16, l + 24.  Four poses share a warp, so an 18-atom ligand fills 18 of 24 lane turns
// instead of 18 of 32, and three reduction levels serve four poses.  The sums follow the tree of a
// whole warp with one atom per lane (levels 16 and 8 in the lane, 4, 2, 1 across): the same bits.
template <typename FT, bool TORQUE>
__device__ __forceinline__ void quarter_forces(const DevSystem& S, const double c[3], const double R[9], int l,
                                               double f[3], double t[3], Counts& cnt) {
  const PosFromPose pos{R, c};
  double even[3] = {0, 0, 0}, even_t[3] = {0, 0, 0}, t0 = 0, t1 = 0, t2 = 0;
  f[0] = f[1] = f[2] = 0.0;
#pragma unroll 1
  for (int k = 0; k < 4; ++k) {  // turns 0, 2, then 1, 3
    if (k == 2) {
#pragma unroll
      for (int d = 0; d < 3; ++d) {
        even[d] = f[d];
        f[d] = 0.0;
      }
      even_t[0] = t0;
      even_t[1] = t1;
      even_t[2] = t2;
      t0 = t1 = t2 = 0.0;
    }
    const int i = l + 8 * (k < 2 ? 2 * k : 2 * k - 3);
    if (i >= S.n_lig) continue;
    const double4 a = S.lig[i];
    if (fabs(a.w) < 1e-9) continue;
    double ro[3], x[3];
    pos(i, a, ro, x);
    FT fa[3], ea;
    if (!ligand_atom<FT, false>(S, a.w, x, true, true, fa, ea, cnt.grid, cnt.ff)) continue;
    f[0] += (double)fa[0];
    f[1] += (double)fa[1];
    f[2] += (double)fa[2];
    if (TORQUE) {
      t0 += ro[1] * (double)fa[2] - ro[2] * (double)fa[1];
      t1 += ro[2] * (double)fa[0] - ro[0] * (double)fa[2];
      t2 += ro[0] * (double)fa[1] - ro[1] * (double)fa[0];
    }
  }
  t[0] = t0;
  t[1] = t1;
  t[2] = t2;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    f[d] = even[d] + f[d];
    if (TORQUE) t[d] = even_t[d] + t[d];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) {
      f[d] += __shfl_xor_sync(0xffffffffu, f[d], o);
      if (TORQUE) t[d] += __shfl_xor_sync(0xffffffffu, t[d], o);
    }
  }
}

// A product rounded by itself: never fused into the sum it goes to.
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

// Barrier of the `threads` threads of a block that share named barrier `id`.
__device__ __forceinline__ void group_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

// Forces on the ligand atoms of a pose by W = 2, 4 or 8 warps of a block: in a round, warp w takes the
// 32 atoms after those of warp w - 1 and leaves every lane's terms in shared memory (`sh`: two rounds of
// W rows of NC components of 32 lanes); component k is then summed by warp k mod W, lane by lane in the
// order of the atoms, as a single warp sums them: the same bits.  tot[i] receives component gw + i * W
// (f0..f2, t0..t2 with TORQUE, the energy last with ENERGY), reduced over the lanes.  Contact forces are
// not included; `extra`, called by every warp with its lane's sums, may add them.
template <bool TORQUE, bool ENERGY>
constexpr int kForwardNc = 3 + (TORQUE ? 3 : 0) + (ENERGY ? 1 : 0);

struct NoExtra {
  __device__ __forceinline__ void operator()(double*) const {}
};

template <typename FT, bool TORQUE, bool ENERGY, class PosFn, class Extra = NoExtra>
__device__ __forceinline__ void group_forward(const DevSystem& S, const PosFn& pos, int lane, int gw, int W, int bar,
                                              double* sh, bool t_grid, bool t_ff, double tot[4], Counts& cnt,
                                              const Extra& extra = Extra{}) {
  constexpr int NC = kForwardNc<TORQUE, ENERGY>;
#pragma unroll
  for (int i = 0; i < 4; ++i) tot[i] = 0.0;
  int flip = 0;
  for (int i0 = 0; i0 < S.n_lig; i0 += 32 * W) {
    double f[3] = {0, 0, 0}, t[3] = {0, 0, 0}, e = 0;
    const int i = i0 + 32 * gw + lane;
    if (i < S.n_lig) {
      const double4 a = S.lig[i];
      double ro[3], x[3];
      pos(i, a, ro, x);
      FT fa[3], ea;
      if (fabs(a.w) >= 1e-9 && ligand_atom<FT, ENERGY, ENERGY>(S, a.w, x, t_grid, t_ff, fa, ea, cnt.grid, cnt.ff)) {
#pragma unroll
        for (int d = 0; d < 3; ++d) f[d] = (double)fa[d];
        if (ENERGY) e = (double)ea;
        if (TORQUE) {
          t[0] = ro[1] * (double)fa[2] - ro[2] * (double)fa[1];
          t[1] = ro[2] * (double)fa[0] - ro[0] * (double)fa[2];
          t[2] = ro[0] * (double)fa[1] - ro[1] * (double)fa[0];
        }
      }
    }
    double* row = sh + ((size_t)flip * W + gw) * NC * 32 + lane;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
      row[d * 32] = f[d];
      if (TORQUE) row[(3 + d) * 32] = t[d];
    }
    if (ENERGY) row[(NC - 1) * 32] = e;
    group_sync(bar, 32 * W);
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int c = gw + k * W;
      if (c < NC)
        for (int w = 0; w < W; ++w) tot[k] += sh[(((size_t)flip * W + w) * NC + c) * 32 + lane];
    }
    flip ^= 1;
  }
  extra(tot);
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (gw + k * W < NC) tot[k] = gsum<32>(tot[k], 0xffffffffu);
  group_sync(bar, 32 * W);  // every row is read before the next pose writes one
}

// Warps per pose of the forward forces of a large ligand, for a list of n poses on n_warps warps: only
// where the list leaves most warps idle.  1,401 atoms, mixed precision, 128 steps, GPU time with one
// warp per pose -> with this rule: 100 trajectories 15.7 -> 6.5 ms, 700 18.1 -> 10.8, 2,000 22.8 -> 21.9,
// 6,000 34.9 both (two or eight warps there: 10 % slower, the rounds' barriers).
__device__ __forceinline__ int fwd_warps(int n, int n_warps) {
  return n <= n_warps / 8 ? 8 : n <= n_warps / 4 ? 4 : n <= n_warps / 2 ? 2 : 1;
}

// List entries a warp takes at a time in split_fwd_kernel<FWD_LONG>: about eight turns per warp and at most 16
// entries, or 512 atoms of ligands above 64 (a last turn of long poses would leave other warps waiting).
// The cursor is one address, and the device adds to it about once a nanosecond: with an entry a turn, lists
// of 100,000 poses and more were bound by it (256 steps, far-field of 18 atoms, FP64: 300,000 poses
// 76.7 -> 61.4 ms, 100,000 27.4 -> 23.2; 18 atoms with grids and Born direction 2 160 -> 142; 40 atoms,
// mixed, 85.8 -> 71.7; 200 atoms, 300,000 246 -> 240, 100,000 level).  Neighbours in the list share the
// sectors of their poses and forces (a turn's entries far apart: 69 instead of 59 ms at 600,000).
constexpr int kLongTurns = 8;
__device__ __forceinline__ int fwd_turn(int n, int n_warps, int atoms) {
  return n < 2 * kLongTurns * n_warps ? 1
                                      : max(1, min(n / (kLongTurns * n_warps), atoms <= 64 ? 16 : min(16, 512 / atoms)));
}

// Forces on the ligand atoms of the listed poses: a warp per pose, or four poses per warp for small
// ligands in mixed precision and lists of several poses a warp (18 atoms, 150,000 slots: 155 -> 116 us;
// at 8,000 slots a warp per pose is the faster, 15.5 against 17.4 us, and in FP64 the quarter-warp
// form spills and is slower at 30,011).  Bound by latency at 13 warps per SM: issue slots 45 %, L1 43 %,
// the double-float conversions 22 %.  FORM: a kernel each for one list entry a turn, for several (pools that
// can list 16 poses per warp) and for four poses a warp (small ligands in mixed precision, which fall back to
// one a turn on short lists): the loop over a turn costs lists with one entry a turn 2 %, the code of the
// four poses 1 to 5 % (40 atoms, mixed with torque, 20,000 slots, 256 steps: 9.42 -> 9.03 ms).
enum { FWD_ONE, FWD_LONG, FWD_PACKED };
template <typename FT, bool TORQUE, int FORM, class TAB>
__global__ void __launch_bounds__(256, 2) split_fwd_kernel(const __grid_constant__ TAB T, SlotBuf B, SplitBuf U,
                                                           int set) {
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  const int n = U.cnt[4 * set], n_warps = (gridDim.x * blockDim.x) >> 5;
  const int first = (threadIdx.x >> 5) * gridDim.x + blockIdx.x;
  Counts cnt{0, 0, 0};
  // Entries of the list that go four to a warp.  With torque the one to three after them take a warp each, one
  // that has few of the others; without, the lanes past the end repeat a pose, uncounted (with the counts apart
  // the torque kernel spills 40 bytes more: 150,000 slots +1 %; the tail in the loop below costs the other 1 %).
  const int packed = FORM == FWD_PACKED && n > 4 * n_warps ? (TORQUE ? n & ~3 : n) : 0;
  if (packed) {
    // lanes read the poses of `m` list entries together, then hand them out four at a time
    const int m = min(32, 4 * ((packed + 4 * n_warps - 1) / (4 * n_warps)));
    for (long long base = (long long)first * m; base < packed; base += (long long)n_warps * m) {
      const int j = (int)base + lane;
      const bool have = lane < m && j < packed;
      const int slot = have ? U.flist[j] : U.flist[(int)base];
      const Pose<SlotSrc> pose(SlotSrc{B, slot});
      int id = B.traj[slot];
      const int sys = T.locate(id);
      for (int p = 0; p < m && base + p < packed; p += 4) {
        const int src = p + (lane >> 3);
        double c[3], R[9], f[3], t[3];
#pragma unroll
        for (int i = 0; i < 3; ++i) c[i] = __shfl_sync(FULL, pose.c[i], src);
#pragma unroll
        for (int i = 0; i < 9; ++i) R[i] = __shfl_sync(FULL, pose.R[i], src);
        const int to = __shfl_sync(FULL, slot, src);
        const DevSystem& S = T.sys(__shfl_sync(FULL, sys, src));
        if (TORQUE) {
          quarter_forces<FT, TORQUE>(S, c, R, lane & 7, f, t, cnt);
          store_force(U, to, lane & 7, f, t);
        } else {
          Counts mine{0, 0, 0};
          quarter_forces<FT, TORQUE>(S, c, R, lane & 7, f, t, mine);
          if (base + src < n) {
            store_force(U, to, lane & 7, f, t);
            cnt.grid += mine.grid;
            cnt.ff += mine.ff;
          }
        }
      }
    }
  }
  if (packed && !TORQUE) {
  } else if (const int W = T.large_ligands() ? fwd_warps(n, n_warps) : 1; W > 1) {
    constexpr int NC = kForwardNc<TORQUE, false>;
    __shared__ double sh[2 * 8 * NC * 32];
    const int warp = threadIdx.x >> 5, gw = warp & (W - 1), grp = warp / W;
    for (int j = grp * gridDim.x + blockIdx.x; j < n; j += n_warps / W) {
      const int slot = U.flist[j];
      int id = B.traj[slot];
      const DevSystem& S = T.sys(T.locate(id));
      const Pose<SlotSrc> pose(SlotSrc{B, slot});
      double tot[4];
      group_forward<FT, TORQUE, false>(S, PosFromPose{pose.R, pose.c}, lane, gw, W, 1 + grp, sh + 2 * grp * W * NC * 32,
                                       true, true, tot, cnt);
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int c = gw + k * W;
        if (lane == 0 && c < 3) U.F[3 * slot + c] = tot[k];
        if (lane == 0 && c >= 3 && c < 6) U.T[3 * slot + c - 3] = TORQUE ? tot[k] : 0.0;
      }
    }
  } else {
    const int m = FORM == FWD_LONG ? fwd_turn(n, n_warps, T.largest_ligand()) : 1;
    for (int j = TORQUE && packed ? packed + n_warps - 1 - first : first * m, left = m; j < n;) {
      const int slot = U.flist[j];
      int id = B.traj[slot];
      const DevSystem& S = T.sys(T.locate(id));
      const Pose<SlotSrc> pose(SlotSrc{B, slot});
      double f[3], t[3], e;
      group_forces<FT, 32, TORQUE, false, PosFromPose, false>(S, pose.c, pose.R, lane, FULL,
                                                             PosFromPose{pose.R, pose.c}, f, t, e, cnt,
                                                             RecView{nullptr, nullptr});
      store_force(U, slot, lane, f, t);
      if (FORM == FWD_LONG && --left) ++j;
      else if (TORQUE && packed) break;
      else {
        j = m * next_item(U.cnt + 4 * set + 2, n_warps, lane);
        left = m;
      }
    }
  }
  const unsigned ng = gsumu<32>(cnt.grid, FULL), nf = gsumu<32>(cnt.ff, FULL);
  unsigned long long* ctr = T.sim(0).ctr;
  if (lane == 0 && ng) atomicAdd(ctr + C_GRID_EVALS, (unsigned long long)ng);
  if (lane == 0 && nf) atomicAdd(ctr + C_FF_EVALS, (unsigned long long)nf);
}

// The pose of a source as the sweep of direction 2 needs it: rotation and centre in FT, and its
// tests of receptor chunks and atoms against the ligand Born grid's margin box in the ligand frame.
template <typename FT>
struct RevPose {
  using V4 = typename Vec4<FT>::type;
  FT Rt[9], cx, cy, cz;

  template <class SRC>
  __device__ __forceinline__ explicit RevPose(const SRC& src) {
    double c[3], R[9];
    src.load(c, R);
#pragma unroll
    for (int k = 0; k < 9; ++k) Rt[k] = (FT)R[k];
    cx = (FT)c[0];
    cy = (FT)c[1];
    cz = (FT)c[2];
  }

  // Chunk k's bounding sphere; past the last chunk one that reaches nothing.
  static __device__ __forceinline__ V4 sphere(const DevSystem& S, int k) {
    if (k >= S.n_chunks) return Vec4<FT>::make(0, 0, 0, (FT)-1);
    if constexpr (sizeof(FT) == 4) return S.chunks_f[k];
    else return S.chunks[k];
  }

  // A chunk's bounding sphere reaches the box.
  __device__ __forceinline__ bool reaches(const DevSystem& S, const V4& sp) const {
    if (sp.w < (FT)0) return false;
    const DevGrid& g = S.lig_born;
    const FT lox = in<FT>(g.lox, g.loxf), loy = in<FT>(g.loy, g.loyf), loz = in<FT>(g.loz, g.lozf);
    const FT hix = in<FT>(g.hix, g.hixf), hiy = in<FT>(g.hiy, g.hiyf), hiz = in<FT>(g.hiz, g.hizf);
    const FT d0 = (FT)sp.x - cx, d1 = (FT)sp.y - cy, d2 = (FT)sp.z - cz;
    const FT l0 = Rt[0] * d0 + Rt[3] * d1 + Rt[6] * d2;
    const FT l1 = Rt[1] * d0 + Rt[4] * d1 + Rt[7] * d2;
    const FT l2 = Rt[2] * d0 + Rt[5] * d1 + Rt[8] * d2;
    const FT ex = fmax(fmax(lox - l0, l0 - hix), (FT)0);
    const FT ey = fmax(fmax(loy - l1, l1 - hiy), (FT)0);
    const FT ez = fmax(fmax(loz - l2, l2 - hiz), (FT)0);
    // the radius is inflated against rounding; the extra margin covers FP32 geometry
    const FT lim = (FT)sp.w + (sizeof(FT) == 4 ? (FT)1e-3 : (FT)1e-9);
    return ex * ex + ey * ey + ez * ez < lim * lim;
  }

  // Receptor atom idx is charged and inside the box; e = its ligand-frame position and charge.
  static __device__ __forceinline__ V4 atom(const DevSystem& S, int idx) {
    if constexpr (sizeof(FT) == 4) return S.rec_f[idx];
    else return S.rec[idx];
  }

  template <class SRC>
  __device__ __forceinline__ bool candidate(const DevSystem& S, const SRC& src, int idx, const V4& at, V4& e) const {
    const DevGrid& g = S.lig_born;
    const FT lox = in<FT>(g.lox, g.loxf), loy = in<FT>(g.loy, g.loyf), loz = in<FT>(g.loz, g.lozf);
    const FT hix = in<FT>(g.hix, g.hixf), hiy = in<FT>(g.hiy, g.hiyf), hiz = in<FT>(g.hiz, g.hizf);
    if (!(fabs(at.w) >= (FT)1e-9)) return false;
    const FT d0 = (FT)at.x - cx, d1 = (FT)at.y - cy, d2 = (FT)at.z - cz;
    const FT l0 = Rt[0] * d0 + Rt[3] * d1 + Rt[6] * d2;
    const FT l1 = Rt[1] * d0 + Rt[4] * d1 + Rt[7] * d2;
    const FT l2 = Rt[2] * d0 + Rt[5] * d1 + Rt[8] * d2;
    bool cand = l0 > lox && l0 < hix && l1 > loy && l1 < hiy && l2 > loz && l2 < hiz;
    if constexpr (sizeof(FT) == 4) {
      // within 1e-3 A of a face the FP64 box test decides (the set of atoms is the FP64 one)
      const float m = fminf(fminf(fminf(l0 - lox, hix - l0), fminf(l1 - loy, hiy - l1)), fminf(l2 - loz, hiz - l2));
      if (fabsf(m) < 1e-3f) {
        double c[3], R[9];
        src.load(c, R);
        const double4 a64 = S.rec[idx];
        const double e0 = a64.x - c[0], e1 = a64.y - c[1], e2 = a64.z - c[2];
        cand = in_box(g, R[0] * e0 + R[3] * e1 + R[6] * e2, R[1] * e0 + R[4] * e1 + R[7] * e2,
                      R[2] * e0 + R[5] * e1 + R[8] * e2);
      }
    }
    e = Vec4<FT>::make(l0, l1, l2, (FT)at.w);
    return cand;
  }
};

// Born direction 2 of one pose by a whole warp (the same terms and order as warp_reverse_born):
// receptor chunks culled against the ligand Born grid's margin box in the ligand frame, in-box
// atoms gathered into `buf` and drained 32 at a time.  Adds this lane's share of the sums to
// r (ligand frame) and u; the caller reduces over the warp.
// AHEAD: the next hit chunk's atoms load while one chunk's are tested.  In FP64 and in the evaluation
// kernel that pays (30,011 FP64 trajectories 117 -> 113 ms of GPU time, 20,000 FP64 poses 390 -> 351 us,
// mixed 267 -> 248); in the mixed stepper the registers it takes from the 64 cost as much as it gains
// (150,000 trajectories 327 -> 332 ms).
template <typename FT, bool TORQUE, bool AHEAD, class SRC>
__device__ __forceinline__ void lean_reverse_born(const DevSystem& S, const SRC& src, int lane,
                                                  typename Vec4<FT>::type* buf, double r[3], double u[3],
                                                  unsigned& nr) {
  using V4 = typename Vec4<FT>::type;
  const unsigned FULL = 0xffffffffu;
  const DevGrid& g = S.lig_born;
  const RevPose<FT> pose(src);
  FT rs0 = 0, rs1 = 0, rs2 = 0;
  int k0 = 0, head = 0;
  int kk = -1;  // the chunk whose atoms `at` holds, -1: none
  unsigned hits = 0;
  V4 at{};
  bool done = false;
  for (;;) {
    // gather until the buffer has no room for another chunk, or every chunk is done
    while (head <= kSplitBuf<FT> - 32) {
      if (kk < 0) {
        if (!hits) {
          if (k0 >= S.n_chunks) {
            done = true;
            break;
          }
          hits = __ballot_sync(FULL, pose.reaches(S, pose.sphere(S, k0 + lane)));
          k0 += 32;
          continue;
        }
        kk = k0 - 32 + __ffs(hits) - 1;
        hits &= hits - 1;
        at = pose.atom(S, kk * BD_CHUNK + lane);
      }
      int kn = -1;
      V4 an = at;
      if (AHEAD) {
        kn = hits ? k0 - 32 + __ffs(hits) - 1 : -1;
        hits &= hits - 1;
        if (kn >= 0) an = pose.atom(S, kn * BD_CHUNK + lane);
      }
      V4 ent{};
      const bool cand = pose.candidate(S, src, kk * BD_CHUNK + lane, at, ent);
      const unsigned m = __ballot_sync(FULL, cand);
      if (cand) buf[head + __popc(m & ((1u << lane) - 1u))] = ent;
      head += __popc(m);
      at = an;
      kk = kn;
    }
    __syncwarp();
    // drain whole groups of 32 (everything once the chunks are done): entry e by lane e mod 32
    const int n_drain = done ? head : (head & ~31);
    const FT alpha = in<FT>(S.alpha, S.alpha_f);
#pragma unroll 1
    for (int e = lane; e < n_drain; e += 32) {
      const V4 v = buf[e];
      const StencilOut<FT, 1> st = stencil<FT, 1, FT>(g, v.x, v.y, v.z);
      const FT cf = -alpha * v.w * v.w;
      const FT g0 = cf * st.gx[0], g1 = cf * st.gy[0], g2 = cf * st.gz[0];
      rs0 += g0;
      rs1 += g1;
      rs2 += g2;
      if (TORQUE) {
        const double x = (double)v.x, y = (double)v.y, z = (double)v.z;
        u[0] += y * (double)g2 - z * (double)g1;
        u[1] += z * (double)g0 - x * (double)g2;
        u[2] += x * (double)g1 - y * (double)g0;
      }
      nr += 1;
    }
    if (done) break;
    // the remainder (fewer than 32 entries) moves to the front of the buffer
    __syncwarp();
    const int rem = head - n_drain;
    V4 keep{};
    if (lane < rem) keep = buf[n_drain + lane];
    __syncwarp();
    if (lane < rem) buf[lane] = keep;
    __syncwarp();
    head = rem;
  }
  __syncwarp();  // the buffer is reused by the next pose
  r[0] += (double)rs0;
  r[1] += (double)rs1;
  r[2] += (double)rs2;
}

// Born direction 2 of one pose by W = 2, 4 or 8 warps of a block: warp gw of the group gathers
// every W-th hit chunk, the entries land in `buf` (W * kSplitBuf of them) in the order of
// lean_reverse_born, every thread evaluates stencils, and the sums are then taken entry by entry
// as there, by lane e mod 32 in order: the same bits.  The force sums (r) end in warp 0 and the
// torque sums (u) in warp 1, per lane; the caller reduces them.  `val` holds the evaluated
// coefficient and gradient (it is `buf` itself when the positions are not needed again);
// cnt: two rows of W counts.  Every warp of the group takes the same path (the culls and counts
// it depends on are the same on each), so the group's barriers match.
template <typename FT, bool TORQUE, bool AHEAD, class SRC>
__device__ __forceinline__ void group_reverse_born(const DevSystem& S, const SRC& src, int lane, int gw, int W, int bar, typename Vec4<FT>::type* buf,
                                                   typename Vec4<FT>::type* val, int* cnt, double r[3], double u[3],
                                                   unsigned& nr) {
  using V4 = typename Vec4<FT>::type;
  const unsigned FULL = 0xffffffffu;
  const DevGrid& g = S.lig_born;
  const RevPose<FT> pose(src);
  const FT alpha = in<FT>(S.alpha, S.alpha_f);
  FT rs0 = 0, rs1 = 0, rs2 = 0;
  int head = 0, flip = 0;
  // evaluate and sum the first n entries (a multiple of 32, or all of them)
  auto drain = [&](int n) {
    group_sync(bar, 32 * W);
#pragma unroll 1
    for (int e = 32 * gw + lane; e < n; e += 32 * W) {
      const V4 v = buf[e];
      const StencilOut<FT, 1> st = stencil<FT, 1, FT>(g, v.x, v.y, v.z);
      val[e] = Vec4<FT>::make(-alpha * v.w * v.w, st.gx[0], st.gy[0], st.gz[0]);
      nr += 1;
    }
    group_sync(bar, 32 * W);
    if (gw == 0) {
#pragma unroll 4
      for (int e = lane; e < n; e += 32) {
        const V4 v = val[e];
        // lean_reverse_born rounds the products where it uses them twice (torque), and fuses them
        // into the sums otherwise
        if (TORQUE) {
          rs0 += mul_rn(v.x, v.y);
          rs1 += mul_rn(v.x, v.z);
          rs2 += mul_rn(v.x, v.w);
        } else {
          rs0 = fma(v.x, v.y, rs0);
          rs1 = fma(v.x, v.z, rs1);
          rs2 = fma(v.x, v.w, rs2);
        }
      }
    }
    if (TORQUE && gw == 1) {
#pragma unroll 4
      for (int e = lane; e < n; e += 32) {
        const V4 v = val[e], p = buf[e];
        const FT g0 = mul_rn(v.x, v.y), g1 = mul_rn(v.x, v.z), g2 = mul_rn(v.x, v.w);
        const double x = (double)p.x, y = (double)p.y, z = (double)p.z;
        u[0] += y * (double)g2 - z * (double)g1;
        u[1] += z * (double)g0 - x * (double)g2;
        u[2] += x * (double)g1 - y * (double)g0;
      }
    }
    group_sync(bar, 32 * W);
  };
  for (int c0 = 0; c0 < S.n_chunks; c0 += 1024) {
    // lane l keeps the hit mask of chunks c0 + 32 l .. + 31
    unsigned mine = 0;
    const int n_mask = min(32, (S.n_chunks - c0 + 31) / 32);
    for (int l = 0; l < n_mask; l += 4) {  // four loads in flight
      V4 sp[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) sp[j] = pose.sphere(S, c0 + 32 * (l + j) + lane);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const unsigned m = __ballot_sync(FULL, pose.reaches(S, sp[j]));
        if (lane == l + j) mine = m;
      }
    }
    int before = __popc(mine);  // exclusive prefix of the hit counts
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int t = __shfl_up_sync(FULL, before, o);
      if (lane >= o) before += t;
    }
    const int H = __shfl_sync(FULL, before, 31);
    before -= __popc(mine);
    // the chunk of hit h: its mask's lane, then the bit with that many hits below it
    auto chunk_of = [&](int h) {
      const unsigned has = __ballot_sync(FULL, before <= h && h < before + __popc(mine));
      const int ml = __ffs(has) - 1;
      const unsigned m = __shfl_sync(FULL, mine, ml);
      const int nth = h - __shfl_sync(FULL, before, ml);
      const unsigned bit = __ballot_sync(FULL, ((m >> lane) & 1u) && __popc(m & ((1u << lane) - 1u)) == nth);
      return c0 + 32 * ml + __ffs(bit) - 1;
    };
    int kk = -1;
    V4 at{};
    if (AHEAD && gw < H) {
      kk = chunk_of(gw);
      at = pose.atom(S, kk * BD_CHUNK + lane);
    }
    for (int h0 = 0; h0 < H; h0 += W) {
      // AHEAD: the warp's next chunk loads while this one's atoms are tested
      int kn = -1;
      V4 an = at, ent{};
      if (!AHEAD) {
        kk = h0 + gw < H ? chunk_of(h0 + gw) : -1;
        if (kk >= 0) at = pose.atom(S, kk * BD_CHUNK + lane);
      } else if (h0 + W + gw < H) {
        kn = chunk_of(h0 + W + gw);
        an = pose.atom(S, kn * BD_CHUNK + lane);
      }
      const bool cand = kk >= 0 && pose.candidate(S, src, kk * BD_CHUNK + lane, at, ent);
      if (AHEAD) {
        at = an;
        kk = kn;
      }
      const unsigned m = __ballot_sync(FULL, cand);
      if (lane == 0) cnt[flip * 8 + gw] = __popc(m);
      group_sync(bar, 32 * W);
      int place = head, total = 0;
      for (int w = 0; w < W; ++w) {
        const int k = cnt[flip * 8 + w];
        if (w < gw) place += k;
        total += k;
      }
      flip ^= 1;
      if (cand) buf[place + __popc(m & ((1u << lane) - 1u))] = ent;
      head += total;
      if (head > (kSplitBuf<FT> - 32) * W) {  // no room for another round
        const int n = head & ~31, rem = head - n;
        drain(n);
        V4 keep{};
        if (gw == 0 && lane < rem) keep = buf[n + lane];
        group_sync(bar, 32 * W);
        if (gw == 0 && lane < rem) buf[lane] = keep;
        head = rem;
      }
    }
  }
  drain(head);
  r[0] = (double)rs0;
  r[1] = (double)rs1;
  r[2] = (double)rs2;
}

// Warps per pose of the sweep for a list of n poses on n_warps resident warps: a list that leaves
// warps idle gives each pose more of them.  One warp takes 20-40 us for a pose in contact (a serial
// chain of chunk gathers and stencil drains), so a short list is bound by that latency: 1,000
// trajectories FP64 took 89 us a sweep with one warp per pose, and the whole run's GPU time fell
// from 120 to 40 ms with eight; 8,000 mixed 200 -> 136 ms, 30,011 FP64 170 -> 147 ms.  Lines twice
// and four times as far out are no better (8,000: 142 and 134 ms; 30,011 FP64: 172 and 168 ms).
__device__ __forceinline__ int rev_warps(int n, int n_warps) {
  return n <= n_warps / 4 ? 8 : n <= n_warps / 2 ? 4 : n <= n_warps ? 2 : 1;
}

// FP32 without torque: capped at 64 registers, 32 warps per SM (at 80 and 24 warps 150,000 trajectories
// take 330 instead of 312 ms of GPU time).  With torque that cap spills 164 bytes: at 80 it spills none,
// and 8,000 trajectories take 107 instead of 121 ms, 6,000 protein pairs 106 instead of 113, 150,000
// (768 steps) 249 instead of 252.  FP64: at 128; a cap of 80 spills 450 bytes and is slower (30,011
// trajectories 114 -> 128 ms).
template <typename FT, bool TORQUE, class TAB>
__global__ void __launch_bounds__(256, sizeof(FT) == 4 ? (TORQUE ? 3 : 4) : 2) split_rev_kernel(const __grid_constant__ TAB T,
                                                                                SlotBuf B, SplitBuf U, int set) {
  using V4 = typename Vec4<FT>::type;
  __shared__ V4 bufs[8][kSplitBuf<FT>];
  __shared__ V4 vals[TORQUE ? 8 : 1][TORQUE ? kSplitBuf<FT> : 1];
  __shared__ int cnts[4][16];
  const unsigned FULL = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int n = U.cnt[4 * set + 1], n_warps = (gridDim.x * blockDim.x) >> 5;
  const int W = rev_warps(n, n_warps);
  const int gw = warp & (W - 1), grp = warp / W;  // warp of the group, group of the block
  unsigned nr = 0;
  for (int j = grp * gridDim.x + blockIdx.x; j < n;
       j = W > 1 ? j + n_warps / W : next_item(U.cnt + 4 * set + 3, n_warps, lane)) {
    const int slot = U.rlist[j];
    int id = B.traj[slot];
    const DevSystem& S = T.sys(T.locate(id));
    double r[3] = {0, 0, 0}, u[3] = {0, 0, 0};
    if (W == 1) {
      lean_reverse_born<FT, TORQUE, sizeof(FT) == 8>(S, SlotSrc{B, slot}, lane, bufs[warp], r, u, nr);
    } else {
      V4* buf = bufs[grp * W];
      group_reverse_born<FT, TORQUE, sizeof(FT) == 8>(S, SlotSrc{B, slot}, lane, gw, W, 1 + grp, buf, TORQUE ? vals[grp * W] : buf,
                                     cnts[grp], r, u, nr);
    }
    if (gw == 0) {
      r[0] = gsum<32>(r[0], FULL);
      r[1] = gsum<32>(r[1], FULL);
      r[2] = gsum<32>(r[2], FULL);
      if (lane < 3) U.rv[6 * (size_t)slot + lane] = r[lane];
      if (!TORQUE && lane < 3) U.rv[6 * (size_t)slot + 3 + lane] = 0.0;
    }
    if (TORQUE && gw == (W > 1 ? 1 : 0)) {
      u[0] = gsum<32>(u[0], FULL);
      u[1] = gsum<32>(u[1], FULL);
      u[2] = gsum<32>(u[2], FULL);
      if (lane < 3) U.rv[6 * (size_t)slot + 3 + lane] = u[lane];
    }
  }
  nr = gsumu<32>(nr, FULL);
  if (lane == 0 && nr) atomicAdd(T.sim(0).ctr + C_REV_EVALS, (unsigned long long)nr);
}

}  // namespace bd
