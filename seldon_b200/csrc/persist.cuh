// Persistent-kernel plumbing: a bounded grid barrier that also performs the
// deterministic cross-CTA reduction, and the per-solve device state.
//
// The kernels using it are launched cooperatively (all CTAs co-resident).
// Every wait is bounded by a wall-clock limit read from %globaltimer: a CTA
// that waits too long sets `status` and the whole grid unwinds, so a solve can
// never hang the GPU.
#pragma once

#include <algorithm>

#include "spmv_core.cuh"

namespace sb2 {

constexpr int kMaxRed = 8;  // scalars reduced by one barrier at most

constexpr int kPersistMaxCtas = 160;  // one CTA per SM

struct GridSync {
  unsigned count;  // arrivals (grid_sync: since the launch; grid_sync_wide: at this barrier)
  unsigned gen;    // generation (grid_sync_wide)
  int status;      // 0 ok, 1 a wait ran out
  int pad;
};

struct SolveOut {
  int nb_iter;
  int error_code;
  int init_failed;
  int hist_len;
  double facteur_reste;
  double last_residual;
};

struct Persist {
  GridSync* sync;
  double* partials;  // deposits (grid_sync: [2 * kMaxRed * gridDim.x])
  unsigned long long wait_ns;
};

// Record of the relative residual of one Finished() test.
struct History {
  double* res;
  int* it;
  int cap;
};

// CTAs of 1024 threads for a solver on `rows` rows in `blocks` row blocks (of up
// to 2048 entries): a row a thread, and no more than four blocks a CTA.  No
// more than that, since a small grid makes the barriers cheap; no less, since a
// product by few CTAs leaves the other SMs' loads unused.  Cg, us an iteration,
// by rows alone against this: 8192 rows of 301 entries 94 -> 19, 4096 of 1001 194
// -> 20, 20,000 of 81 63 -> 21, 27,000 of 27 34 -> 25; Lsqr 98 -> 15, 210 -> 17, 60
// -> 17, 31 -> 26.  Two blocks a CTA: the same where rows are wide, Lsqr on the
// 27,000 rows 29.
inline int persist_ctas(int rows, int blocks, int most) {
  const int want = std::max((rows + 1023) / 1024, (blocks + 3) / 4);
  return std::max(1, std::min(most, want));
}

#ifdef __CUDACC__

// Grid barrier.  Each CTA deposits K block sums (s_vals[0..K), written by
// thread 0) and adds one to a counter; when all have, every CTA adds the
// deposits in CTA order (the same tree on every run and in every CTA).  On
// return s_vals holds the K grid sums.  False when a wait ran out; the other
// CTAs then run out of theirs.
// It costs one red.release and the polling load that sees it, and with K > 0
// one more trip for the deposits: 1.4 us and 2.2 us at 148 CTAs.  The form it
// replaced (the last CTA to arrive sums and releases the others, 592 CTAs of
// 256 threads) took 2.8 us; deposits that carry their own tags, polled by
// every CTA, 3.7 us: a line that 148 SMs poll is slow to write.
// The counter only grows; deposits alternate between two sets, since a CTA
// can be one barrier ahead of another, never two.
// grid_arrive and grid_wait are its halves: work between them overlaps the
// trip.  Asynchronous copies belong there (a release waits for those its
// thread has in flight), and then `fence` is false: without it grid_wait
// orders only the sums, not other data of other CTAs.
template <int NT>
__device__ __forceinline__ void grid_arrive(const Persist& P, unsigned& epoch, int K,
                                            const double* s_vals) {
  static_assert(NT / 32 >= kMaxRed, "one warp sums one value");
  const int lane = threadIdx.x & 31, G = gridDim.x;
  double* part = P.partials + (size_t)(epoch & 1u) * kMaxRed * G;
  epoch++;
  __syncthreads();
  if (threadIdx.x < 32) {
    if (lane < K) __stcg(part + (size_t)lane * G + blockIdx.x, s_vals[lane]);
    __syncwarp();
    if (lane == 0) red_release_u32(&P.sync->count, 1u);
  }
}

// grid_arrive with the CTA's sums made on the way: the warps leave theirs in
// s_red[K][NT / 32], warp 0 adds them and deposits (one CTA barrier instead of
// the block sums' two each and the arrival's own; the same tree).
template <int NT, int K>
__device__ __forceinline__ void grid_arrive_sums(const Persist& P, unsigned& epoch,
                                                 const double (&a)[K], double* s_red) {
  constexpr int NW = NT / 32;
  const int tid = threadIdx.x, G = gridDim.x;
  double* part = P.partials + (size_t)(epoch & 1u) * kMaxRed * G;
  epoch++;
#pragma unroll
  for (int k = 0; k < K; k++) {
    const double w = warp_sum(a[k]);
    if ((tid & 31) == 0) s_red[k * NW + (tid >> 5)] = w;
  }
  __syncthreads();
  if (tid < 32) {
#pragma unroll
    for (int k = 0; k < K; k++) {
      const double w = warp_sum(tid < NW ? s_red[k * NW + tid] : 0.0);
      if (tid == 0) __stcg(part + (size_t)k * G + blockIdx.x, w);
    }
    if (tid == 0) red_release_u32(&P.sync->count, 1u);
  }
}

// POLLER_SUMS: the warp that polled also adds the deposits, one value after
// the other, which saves the CTA barrier between the two.  With the fused
// arrival Cg on the 512^2 Laplacian goes from 9.4 to 8.4 us an iteration
// (3 sums in 2 barriers), BiCgStab on 56^3 from 12.0 to 10.3; Gmres, short of
// registers there, loses: 57 to 62 us a step on 64^3.
template <int NT, bool POLLER_SUMS = false>
__device__ __forceinline__ bool grid_wait(const Persist& P, unsigned epoch, int K, double* s_vals,
                                          bool fence) {
  __shared__ int s_late;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int G = gridDim.x;
  const double* part = P.partials + (size_t)((epoch - 1u) & 1u) * kMaxRed * G;
  const unsigned target = epoch * (unsigned)G;
  // one value's deposits, added by one warp
  auto sum_of = [&](int k) {
    double in[(kPersistMaxCtas + 31) / 32], v = 0.0;
#pragma unroll
    for (int q = 0; q < (kPersistMaxCtas + 31) / 32; q++) {
      const int c = lane + 32 * q;
      in[q] = c < G ? __ldcg(part + (size_t)k * G + c) : 0.0;
    }
#pragma unroll
    for (int q = 0; q < (kPersistMaxCtas + 31) / 32; q++) v = add_rn(v, in[q]);
    return warp_sum(v);
  };
  if (warp == 0) {
    if (lane == 0) {
      const unsigned long long t0 = global_timer_ns();
      int late = 0;
      while ((int)(ld_acquire_u32(&P.sync->count) - target) < 0) {
        if (global_timer_ns() - t0 > P.wait_ns) {
          atomicExch(&P.sync->status, 1);
          late = 1;
          break;
        }
      }
      // a gpu-scope fence after the wait, as cooperative groups' grid.sync
      // takes: with the CTA barrier below, the L1-cached gathers of the next
      // phase (XLoadCa) see every write made before the barrier
      if (fence) asm volatile("fence.acq_rel.gpu;" ::: "memory");
      s_late = late;
    }
    if (POLLER_SUMS) {
      __syncwarp();
#pragma unroll
      for (int k = 0; k < K; k++) {
        const double v = sum_of(k);
        if (lane == 0) s_vals[k] = v;
      }
    }
  }
  __syncthreads();
  if (s_late) return false;
  if (K && !POLLER_SUMS) {
    if (warp < K) {
      const double v = sum_of(warp);
      if (lane == 0) s_vals[warp] = v;
    }
    __syncthreads();
  }
  return true;
}

template <int NT>
__device__ __forceinline__ bool grid_sync(const Persist& P, unsigned& epoch, int K, double* s_vals) {
  grid_arrive<NT>(P, epoch, K, s_vals);
  return grid_wait<NT>(P, epoch, K, s_vals, true);
}

// K sums over the grid and the barrier (s_red: K * NT / 32, the caller's own:
// no block sum may be using it).
template <int NT, int K>
__device__ __forceinline__ bool grid_sums(const Persist& P, unsigned& epoch, const double (&a)[K],
                                          double* s_vals, double* s_red) {
  grid_arrive_sums<NT, K>(P, epoch, a, s_red);
  return grid_wait<NT, (K <= 2)>(P, epoch, K, s_vals, true);
}

// Gathers of the product's operand inside a persistent kernel: cached in L1
// (ld.ca), where a stencil's neighbouring columns hit.  The operand must have
// been written in an EARLIER phase, never in the phase that gathers it: every
// phase ends at grid_sync / grid_sync_wide, whose gpu-scope fences (the
// waiting thread's acquire and fence, the last CTA's fence) and CTA barrier
// order these loads after every write released before the barrier -- the
// guarantee ordinary loads have after cooperative groups' grid.sync.  The
// read-only matrix uses the streaming path.
template <typename T>
struct XLoadCa {
  const T* x;
  __device__ __forceinline__ T operator()(int j) const { return __ldca(x + j); }
  template <typename O>
  __device__ __forceinline__ void gather4(const int4& c, O (&o)[4]) const {
    T v[4];
    if (quad_contiguous(x, c)) {
      vld4_ca(x + c.x, v);
    } else {
      v[0] = __ldca(x + c.x); v[1] = __ldca(x + c.y); v[2] = __ldca(x + c.z); v[3] = __ldca(x + c.w);
    }
    o[0] = O(v[0]); o[1] = O(v[1]); o[2] = O(v[2]); o[3] = O(v[3]);
  }
};

#endif  // __CUDACC__

}  // namespace sb2
