// Batched replicas: many independent BD systems with hydrodynamic
// interactions (rpy / rpy_smith, Ermak-McCammon scheme) advanced together.
//
// Every replica follows Box.propagate (src/bdsim/pyBrown/box.py:150-250) on
// its own positions, radii, box and noise stream, exactly as a single system
// would: D from the RPY (or Smith-Ewald RPY) tensor, B = chol(D), the
// deterministic step (dt/kBT) D F, then attempts of the stochastic step
// sqrt(2 dt) B xi that are undone on a bead overlap and redrawn.
//
// Each replica owns its device buffers (allocated when it is added).  The
// per-replica descriptors and work lists that the kernels read are rebuilt
// only when the membership changes, so replicas can join and leave between
// steps while the others keep their state on the device.  One step is a
// fixed sequence of launches over all replicas: Ewald tiles (one work list),
// written to D and to B's lower triangle, one cooperative data-flow Cholesky
// over every replica's tiles (left-looking on the tcgen05 tensor cores in the
// mixed precision, right-looking DMMA tile tasks in FP64), then the
// per-replica vector kernels (replica = blockIdx.y).  Replicas never interact, and each one's arithmetic does not
// depend on which other replicas share the batch.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <utility>
#include <vector>

#include "common.cuh"
#include "kernels.cuh"
#include "propagate.cuh"
#include "pybrown_b200.h"

namespace pbg {

// The stream-ordered pool keeps freed replica memory for the next replica
// instead of returning it to the driver at every synchronisation.
inline void batch_pool_keep() {
  static std::mutex mu;
  static bool done[64] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    cudaGetLastError();
    return;
  }
  std::lock_guard<std::mutex> lk(mu);
  if (done[dev]) return;
  cudaMemPool_t pool;
  if (cudaDeviceGetDefaultMemPool(&pool, dev) == cudaSuccess) {
    uint64_t threshold = UINT64_MAX;
    cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &threshold);
  }
  cudaGetLastError();
  done[dev] = true;
}

struct BatchReplica {
  pbg_params p;
  int N = 0, n = 0, ld = 0, nt = 0;
  double scale = 0;  // kBT 1e19 / eta: D = scale * M (box.py:498)
  double *pos = nullptr, *radii = nullptr, *force = nullptr, *U = nullptr, *xi = nullptr;
  void *D = nullptr, *B = nullptr, *invdiag = nullptr;
  bool has_force = false;
  unsigned long long seed = 0, draws = 0;
  // this replica's Cholesky task list on the device (built once, when added)
  int4* tasks = nullptr;
  std::vector<int> seg_start;
};

// One piece of a merged task list: `count` tasks of replica `replica`.
struct GatherSeg {
  const int4* src;
  long long dst;
  int count, replica;
};

// Attempts of one replica that a round evaluates together once its first
// attempt of the step was rejected (see batch_trmv_kernel).
constexpr int SPEC = 8;

// An entry of a round's work list: replica q with `attempts` attempts, its first
// unit of the B xi product and of the overlap test.
struct RoundEntry {
  int q, attempts, trmv0, ovl0;
};
// Entry counts and units of the two lists (one being worked on, the next one
// being built), count << 48 | product units << 26 | overlap units, so that one
// atomic reserves a consistent place in all three; blocks done.
struct RoundState {
  unsigned long long packed[2];
  int done, pad;
};
constexpr int TRMV_ROWS = 16;  // rows per unit of the product: two per warp
constexpr int OVL_BEADS = 8;   // beads per unit of the overlap test: one per warp

// What the vector kernels need of one replica.  U: SPEC + 1 vectors of ld, xi:
// SPEC vectors of ld.
struct BatchDev {
  double* pos;
  const double* radii;
  const double* force;
  double* U;
  double* xi;
  const void* D;
  void* B;
  double L, thr, kBT;
  int N, n, ld, check, has_force, pad;
};

}  // namespace pbg

struct pbg_batch {
  int precision = PBG_PREC_MIXED;
  int hydrodynamics = PBG_HI_RPY_SMITH;
  double alpha = 0;
  int m_max = 0, n_max = 0;
  const pbg::EwaldTables* tables = nullptr;
  std::vector<pbg::BatchReplica*> slots;
  // active replicas (slot ids) in the order of the device arrays
  std::vector<int> active;
  bool dirty = true;
  double dt = 0;
  bool in_step = false;
  // device arrays of the current membership
  pbg::BatchDev* d_reps = nullptr;
  void* d_rpy = nullptr;
  int4* d_ework = nullptr;
  int n_ework = 0;
  pbg::CholRep* d_chol = nullptr;
  int4* d_tasks = nullptr;
  int ntasks = 0;
  pbg::GatherSeg* d_segs = nullptr;
  int4* d_eparts = nullptr;  // per replica: tiles per edge, offset in the Ewald work list
  // capacities (bytes) of the grow-only arrays above
  size_t cap_reps = 0, cap_rpy = 0, cap_ework = 0, cap_chol = 0, cap_tasks = 0, cap_segs = 0, cap_eparts = 0,
         cap_flags = 0;
  int* d_flags = nullptr;  // [4 ctl][per replica: upd nt^2, fin nt^2][R infos]
  size_t flag_ints = 0;
  int* d_info = nullptr;
  int* d_ovl = nullptr;                // [cap][SPEC] overlap flags of a round's candidates
  int* d_rejected = nullptr;           // [cap] outcome of a host-driven attempt
  int* d_spec = nullptr;               // [cap] attempts of the present round
  pbg::RoundEntry* d_lists = nullptr;  // [2][cap]
  pbg::RoundState* d_state = nullptr;
  unsigned char* d_mask = nullptr;
  unsigned long long* d_stream = nullptr;  // [R][2]: seed, draws of each noise stream
  int* h_ovl = nullptr;  // pinned, read after a stream synchronisation
  int* h_info = nullptr;
  std::vector<unsigned char> mask;  // of the last upload, active order
  size_t cap = 0;  // capacity of the per-replica device/pinned arrays
  int max_n = 0;
  // Schedule of the batched factorisation (pbg_batch_autotune): the order in
  // which the replicas' task segments are merged, and the resident CTAs per
  // SM (0 = as many as fit).  Neither changes any result.
  int merge_order = PBG_MERGE_LARGER_FIRST;
  int ctas_per_sm = 0;
  bool have_D = false;  // a step has built D (the autotuner factors it)
  // CUDA graph of the deterministic part of a step (Ewald build, copy into
  // B, the persistent factorisation, the deterministic move), captured once a
  // step repeats with the same membership and flags, replayed afterwards.
  cudaStream_t cap_stream = nullptr;   // private non-blocking stream for the capture
  cudaGraphExec_t begin_exec = nullptr;
  long long begin_kernels = 0;         // kernel launches inside the graph
  int key_build = -1, key_chol = -1, key_force = -1;
  double key_dt = 0;
  int key_repeats = 0;                 // steps in a row with the current key
  bool graph_refused = false;          // the driver refused the capture: direct launches
  // Whole steps on the device (pbg_batch_step): the start, the rounds of
  // attempts under a conditional WHILE node and the wrap, as one graph.
  cudaStream_t cap_stream2 = nullptr;  // captures the loop body
  cudaGraphExec_t step_exec = nullptr;
  long long step_fixed_kernels = 0;    // kernels of one replay besides the rounds
  int* d_att = nullptr;                // [R] attempts of this step (inside d_flags)
  int* d_words = nullptr;              // [4]: any replica still moving, error bits, rounds, 0
  int* d_maxatt = nullptr;             // [cap] max_move_attempts per replica
  int* h_step = nullptr;               // pinned: infos, attempts, words of the last step
  bool streams_on_device = false;      // d_stream holds every replica's (seed, draws)
  bool host_draws_stale = false;       // ... and the host copies are behind it
};

namespace pbg {

namespace {

// B = lower(D) with the identity beyond n and zeros above the diagonal.
template <typename T>
__global__ void batch_copy_lower_kernel(const BatchDev* __restrict__ reps) {
  const BatchDev& r = reps[blockIdx.y];
  const T* src = static_cast<const T*>(r.D);
  T* dst = static_cast<T*>(r.B);
  const int n = r.n, ld = r.ld;
  const long long total = (long long)ld * ld;
  for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < total;
       t += (long long)gridDim.x * blockDim.x) {
    const int row = (int)(t / ld), col = (int)(t % ld);
    T v;
    if (row < n && col < n) v = col <= row ? src[t] : (T)0;
    else v = (T)(row == col ? 1 : 0);
    dst[t] = v;
  }
}

// Deterministic step (box.py:353-362) for replicas with a force:
// pos += ((dt/kBT) D @ F * 1) * 1, one warp per row.
template <typename T>
__global__ void batch_det_kernel(const BatchDev* __restrict__ reps, double dt) {
  const BatchDev& r = reps[blockIdx.y];
  if (!r.has_force) return;
  const T* D = static_cast<const T*>(r.D);
  const double c = dt / r.kBT;
  const double* F = r.force;
  const int lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  for (int row = blockIdx.x * warps + (threadIdx.x >> 5); row < r.n; row += gridDim.x * warps) {
    const double s = row_dot(D + (size_t)row * r.ld, r.n, [&](int j, double a) { return (c * a) * F[j]; });
    // the displacement waits in U until every row is done (see batch_det_move)
    if (lane == 0) r.U[row] = (s * 1.0) * 1.0;
  }
}

__global__ void batch_det_move_kernel(const BatchDev* __restrict__ reps) {
  const BatchDev& r = reps[blockIdx.y];
  if (!r.has_force) return;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < r.n; i += gridDim.x * blockDim.x) r.pos[i] += r.U[i];
}

// ---- attempt rounds -------------------------------------------------------
// A replica's stochastic attempts (box.py:219-248) in rounds: xi, U = B xi and
// the move, the overlap test, the undo of rejected moves and the bookkeeping.
// The first attempt of a step goes alone; a replica whose attempt was rejected
// takes its next SPEC attempts in one round: their noise is at known places of
// its stream, B is read once for all of them, and the first accepted one
// counts, exactly as if they had been made one after the other (rejected moves
// are added and taken back in their order, so the positions agree to the last
// bit; draws and attempts count up to the accepted one).  A round works from a
// list of the moving replicas, so its cost is that of the replicas in it: one
// 1865-bead replica of 24 took 112 us for B xi (64 blocks) and 65 us for the
// overlap test per attempt before, with up to 70 attempts in a step.

// The list entry that unit u belongs to (product units, or overlap units).
__device__ __forceinline__ RoundEntry find_entry(const RoundEntry* list, int count, int u, bool trmv) {
  int lo = 0, hi = count - 1;
  while (lo < hi) {
    const int mid = (lo + hi + 1) >> 1;
    const int first = trmv ? list[mid].trmv0 : list[mid].ovl0;
    if (first <= u) lo = mid;
    else hi = mid - 1;
  }
  return list[lo];
}
__device__ __forceinline__ int packed_count(unsigned long long v) { return (int)(v >> 48); }
__device__ __forceinline__ int packed_trmv(unsigned long long v) { return (int)((v >> 26) & 0x3FFFFFu); }
__device__ __forceinline__ int packed_ovl(unsigned long long v) { return (int)(v & 0x3FFFFFFu); }

// Appends replica q to the list being built.
__device__ __forceinline__ void append_entry(const BatchDev& r, int q, int attempts, RoundEntry* list,
                                             unsigned long long* packed) {
  const unsigned long long tu = (r.n + TRMV_ROWS - 1) / TRMV_ROWS;
  const unsigned long long ou = r.check ? (unsigned long long)((r.N + OVL_BEADS - 1) / OVL_BEADS) * attempts : 0;
  const unsigned long long at = atomicAdd(packed, (1ULL << 48) | (tu << 26) | ou);
  list[packed_count(at)] = RoundEntry{q, attempts, packed_trmv(at), packed_ovl(at)};
}

__device__ __forceinline__ double warp_sum(double s) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}

// Two rows of B times a noise vector, in the term order of row_dot
// (propagate.cuh) for each.
template <typename T>
__device__ __forceinline__ void row_pair_dots(const T* __restrict__ b0, const T* __restrict__ b1, int j0, int j1,
                                              const double* __restrict__ xi, double& s0, double& s1) {
  using C = Chunk<T>;
  constexpr int W = C::W, U = 4;
  const int lane = threadIdx.x & 31, nchunks = (j1 + W - 1) / W;
  const typename C::V* v0 = reinterpret_cast<const typename C::V*>(b0);
  const typename C::V* v1 = reinterpret_cast<const typename C::V*>(b1);
  s0 = s1 = 0.0;
  for (int c0 = lane; c0 < nchunks; c0 += 32 * U) {
    typename C::V p0[U], p1[U];
#pragma unroll
    for (int u = 0; u < U; ++u)
      if (c0 + 32 * u < nchunks) {
        p0[u] = __ldg(v0 + c0 + 32 * u);
        p1[u] = __ldg(v1 + c0 + 32 * u);
      }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int c = c0 + 32 * u;
      if (c >= nchunks) continue;
      double e0[W], e1[W], x[W];
      C::get(p0[u], e0);
      C::get(p1[u], e1);
#pragma unroll
      for (int q = 0; q < W; q += 2) {
        const double2 y = *reinterpret_cast<const double2*>(xi + c * W + q);
        x[q] = y.x;
        x[q + 1] = y.y;
      }
      // a row's terms beyond its diagonal are left out
      const int k0 = j0 - c * W, k1 = j1 - c * W;
#pragma unroll
      for (int q = 0; q < W; ++q) {
        if (q < k0) s0 += e0[q] * x[q];
        if (q < k1) s1 += e1[q] * x[q];
      }
    }
  }
  s0 = warp_sum(s0);
  s1 = warp_sum(s1);
}

// The same for SPEC noise vectors (stride ld) by the whole CTA, rows row0 + 2 w and
// + 1 on warp w: the noise passes through shared memory, TRMV_COLS columns at
// a time, one block ahead, instead of every warp reading 64 bytes of it per
// element of B through L1: a round of 23 replicas with up to 5600
// unknowns 505 -> 189 us, one of 250 replicas 788 -> 316 us.
constexpr int TRMV_COLS = 256;
template <typename T>
__device__ __forceinline__ void row_pair_dots_staged(const BatchDev& r, int row0, double (*xs)[SPEC * TRMV_COLS],
                                                     double (&s0)[SPEC], double (&s1)[SPEC]) {
  using C = Chunk<T>;
  using V = typename C::V;
  constexpr int W = C::W, U = TRMV_COLS / W / 32;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int ra = min(row0 + 2 * warp, r.n - 1), rb = min(row0 + 2 * warp + 1, r.n - 1);
  const int j0 = ra + 1, j1 = rb + 1, nchunks = (j1 + W - 1) / W;
  const V* v0 = reinterpret_cast<const V*>(static_cast<const T*>(r.B) + (size_t)ra * r.ld);
  const V* v1 = reinterpret_cast<const V*>(static_cast<const T*>(r.B) + (size_t)rb * r.ld);
  const int nb = (min(row0 + TRMV_ROWS, r.n) + TRMV_COLS - 1) / TRMV_COLS;
  auto stage = [&](int k) {  // the pairs of a chunk 32 places apart: no bank conflicts below
    for (int i = threadIdx.x; i < SPEC * TRMV_COLS / 2; i += 256) {
      const int a = i / (TRMV_COLS / 2), q = i % (TRMV_COLS / 2), c = 2 * q / W, h = q % (W / 2);
      const int col = k * TRMV_COLS + 2 * q;
      if (col < r.ld) {
        const unsigned d = (unsigned)__cvta_generic_to_shared(&xs[k & 1][a * TRMV_COLS + 2 * ((c / 32 * (W / 2) + h) * 32 + c % 32)]);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(r.xi + (size_t)a * r.ld + col) : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  V p0[U], p1[U];
  auto load = [&](int k, V (&x)[U], V (&y)[U]) {
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int c = k * (TRMV_COLS / W) + lane + 32 * u;
      if (c < nchunks) {
        x[u] = __ldg(v0 + c);
        y[u] = __ldg(v1 + c);
      }
    }
  };
#pragma unroll
  for (int a = 0; a < SPEC; ++a) s0[a] = s1[a] = 0.0;
  stage(0);
  for (int k = 0; k < nb; ++k) {
    load(k, p0, p1);
    if (k + 1 < nb) {
      stage(k + 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    __syncthreads();
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int c = k * (TRMV_COLS / W) + lane + 32 * u;
      if (c < nchunks) {
        double e0[W], e1[W];
        C::get(p0[u], e0);
        C::get(p1[u], e1);
        const int k0 = j0 - c * W, k1 = j1 - c * W;
#pragma unroll
        for (int a = 0; a < SPEC; ++a) {
          double x[W];
#pragma unroll
          for (int h = 0; h < W / 2; ++h) {
            const double2 y = *reinterpret_cast<const double2*>(
                &xs[k & 1][a * TRMV_COLS + 2 * ((u * (W / 2) + h) * 32 + lane)]);
            x[2 * h] = y.x;
            x[2 * h + 1] = y.y;
          }
#pragma unroll
          for (int q = 0; q < W; ++q) {
            if (q < k0) s0[a] += e0[q] * x[q];
            if (q < k1) s1[a] += e1[q] * x[q];
          }
        }
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int a = 0; a < SPEC; ++a) {
    s0[a] = warp_sum(s0[a]);
    s1[a] = warp_sum(s1[a]);
  }
}

// One row's candidates: U[a][row] = the position after attempt a (the attempts
// before it added and taken back), U[attempts][row] = after all of them were
// taken back (box.py:366-375; every product and sum rounded on its own).
template <int NA>
__device__ __forceinline__ void write_candidates(const BatchDev& r, int row, const double (&s)[NA], int attempts,
                                                 double s1) {
  double p = r.pos[row];
#pragma unroll
  for (int a = 0; a < NA; ++a)
    if (a < attempts) {
      const double m = __dmul_rn(s[a], s1), c = __dadd_rn(p, m);
      r.U[(size_t)a * r.ld + row] = c;
      p = __dadd_rn(c, -m);
    }
  r.U[(size_t)attempts * r.ld + row] = p;
}

// U = B xi (box.py:371; B lower triangular) and the candidate positions of the
// listed replicas' attempts.  Bound by reading B (once for all attempts of a
// round): two rows per warp share the noise vectors' loads.  rounds: the
// step's round counter (its parity names the list), null for list 0.
template <typename T>
__global__ void __launch_bounds__(256, 2) batch_trmv_kernel(const BatchDev* __restrict__ reps,
                                                         const RoundEntry* __restrict__ lists, int cap,
                                                         const RoundState* __restrict__ state,
                                                         const int* __restrict__ rounds, double s1) {
  __shared__ __align__(16) double xs[2][SPEC * TRMV_COLS];
  const int par = rounds ? *rounds & 1 : 0;
  const unsigned long long pk = state->packed[par];
  const RoundEntry* list = lists + (size_t)par * cap;
  const int count = packed_count(pk), units = packed_trmv(pk), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int u = blockIdx.x; u < units; u += gridDim.x) {
    const RoundEntry e = find_entry(list, count, u, true);
    const BatchDev r = reps[e.q];
    const int row = (u - e.trmv0) * TRMV_ROWS + 2 * warp;
    const bool two = row + 1 < r.n;
    if (e.attempts == 1) {
      if (row >= r.n) continue;
      const T* b0 = static_cast<const T*>(r.B) + (size_t)row * r.ld;
      double x0[1], x1[1];
      row_pair_dots<T>(b0, two ? b0 + r.ld : b0, row + 1, two ? row + 2 : row + 1, r.xi, x0[0], x1[0]);
      if (lane == 0) write_candidates<1>(r, row, x0, 1, s1);
      if (lane == 1 && two) write_candidates<1>(r, row + 1, x1, 1, s1);
    } else {
      double x0[SPEC], x1[SPEC];
      row_pair_dots_staged<T>(r, row - 2 * warp, xs, x0, x1);
      if (lane == 0 && row < r.n) write_candidates<SPEC>(r, row, x0, e.attempts, s1);
      if (lane == 1 && two) write_candidates<SPEC>(r, row + 1, x1, e.attempts, s1);
    }
  }
}

// Overlap test of every candidate (bead.c:169-218), no bonded pairs: one warp
// per bead i and attempt over the beads j < i.
__global__ void __launch_bounds__(256) batch_overlap_kernel(const BatchDev* __restrict__ reps,
                                                            const RoundEntry* __restrict__ lists, int cap,
                                                            const RoundState* __restrict__ state,
                                                            const int* __restrict__ rounds, int* ovl) {
  const int par = rounds ? *rounds & 1 : 0;
  const unsigned long long pk = state->packed[par];
  const RoundEntry* list = lists + (size_t)par * cap;
  const int count = packed_count(pk), units = packed_ovl(pk), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int u = blockIdx.x; u < units; u += gridDim.x) {
    const RoundEntry e = find_entry(list, count, u, false);
    const BatchDev r = reps[e.q];
    const int blocks = (r.N + OVL_BEADS - 1) / OVL_BEADS, k = u - e.ovl0, a = k / blocks;
    const int i = (k % blocks) * OVL_BEADS + warp;
    int* flag = ovl + e.q * SPEC + a;
    // lane 0's view of the flag for the whole warp
    if (i >= r.N || __shfl_sync(0xffffffffu, *reinterpret_cast<volatile int*>(flag), 0)) continue;
    const double* pos = r.U + (size_t)a * r.ld;
    bool hit = false;
    for (int j = lane; j < i && !hit; j += 32) hit = pair_overlaps(pos, r.radii, i, j, r.L, r.thr);
    if (__any_sync(0xffffffffu, hit) && lane == 0) atomicOr(flag, 1);
  }
}

__global__ void batch_wrap_kernel(const BatchDev* __restrict__ reps) {
  const BatchDev& r = reps[blockIdx.y];
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < r.n; i += gridDim.x * blockDim.x)
    r.pos[i] = pbg_wrap(r.pos[i], r.L);
}

// Counter-based normal variates for a replica's noise stream: Philox-4x32-10
// (Salmon, Moraes, Dror, Shaw, "Parallel random numbers: as easy as 1, 2, 3",
// SC 2011) keyed by the replica's seed, counter = pair index of the draw,
// and the Box-Muller transform of two 53-bit uniforms.  Draw d of a stream
// depends only on (seed, d), never on the other replicas of the batch.
__device__ __forceinline__ void philox_round(uint32_t c[4], uint32_t k0, uint32_t k1) {
  const uint32_t m0 = 0xD2511F53u, m1 = 0xCD9E8D57u;
  const uint32_t hi0 = __umulhi(m0, c[0]), lo0 = m0 * c[0];
  const uint32_t hi1 = __umulhi(m1, c[2]), lo1 = m1 * c[2];
  const uint32_t n0 = hi1 ^ c[1] ^ k0, n2 = hi0 ^ c[3] ^ k1;
  c[0] = n0;
  c[1] = lo1;
  c[2] = n2;
  c[3] = lo0;
}

__device__ __forceinline__ void philox4x32_10(uint32_t c[4], uint32_t k0, uint32_t k1) {
#pragma unroll
  for (int r = 0; r < 10; ++r) {
    philox_round(c, k0, k1);
    k0 += 0x9E3779B9u;
    k1 += 0xBB67AE85u;
  }
}

__device__ __forceinline__ double u53(uint32_t hi, uint32_t lo) {
  const unsigned long long v = ((unsigned long long)hi << 32 | lo) >> 11;
  return ((double)v + 0.5) * (1.0 / 9007199254740992.0);  // (0, 1)
}

// Draws 2 pair and 2 pair + 1 of a stream.
__device__ __forceinline__ void philox_pair(unsigned long long seed, unsigned long long pair, double& x, double& y) {
  uint32_t c[4] = {(uint32_t)pair, (uint32_t)(pair >> 32), 0u, 0u};
  philox4x32_10(c, (uint32_t)seed, (uint32_t)(seed >> 32));
  const double u1 = u53(c[0], c[1]), u2 = u53(c[2], c[3]);
  const double rad = sqrt(-2.0 * log(u1));
  double sn, cs;
  sincospi(2.0 * u2, &sn, &cs);
  x = rad * cs;
  y = rad * sn;
}

__global__ void batch_noise_kernel(const BatchDev* __restrict__ reps, const unsigned char* __restrict__ mask,
                                   const unsigned long long* __restrict__ streams) {
  if (!mask[blockIdx.y]) return;
  const BatchDev& r = reps[blockIdx.y];
  const unsigned long long seed = streams[2 * blockIdx.y], base = streams[2 * blockIdx.y + 1] / 2;  // even
  const int pairs = (r.n + 1) / 2;
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < pairs; q += gridDim.x * blockDim.x) {
    double x, y;
    philox_pair(seed, base + (unsigned long long)q, x, y);
    r.xi[2 * q] = x;
    if (2 * q + 1 < r.n) r.xi[2 * q + 1] = y;
  }
}

// The noise of `attempts` attempts from stream position `base` (even): attempt a
// takes the n draws from base + a (n + (n & 1)) on.
__device__ __forceinline__ void stream_noise(const BatchDev& r, unsigned long long seed, unsigned long long base,
                                             int attempts) {
  const int pairs = (r.n + 1) / 2;
  for (int t = threadIdx.x; t < attempts * pairs; t += blockDim.x) {
    const int a = t / pairs, q = t - a * pairs;
    double x, y;
    philox_pair(seed, base / 2 + (unsigned long long)t, x, y);
    double* xi = r.xi + (size_t)a * r.ld;
    xi[2 * q] = x;
    if (2 * q + 1 < r.n) xi[2 * q + 1] = y;
  }
}

// Start of the attempt rounds of a device step (one block per replica): every
// replica moves, with one attempt; the attempt counts and the step words are
// cleared, the first noise drawn.
__global__ void batch_round_init_kernel(const BatchDev* __restrict__ reps, unsigned char* __restrict__ mask,
                                        int* __restrict__ att, int* __restrict__ words, int* __restrict__ ovl,
                                        int* __restrict__ spec, const unsigned long long* __restrict__ streams,
                                        RoundEntry* lists, RoundState* state) {
  const int q = blockIdx.x;
  const BatchDev r = reps[q];
  if (threadIdx.x < SPEC) ovl[q * SPEC + threadIdx.x] = 0;
  if (threadIdx.x == 0) {
    mask[q] = 1;
    att[q] = 0;
    spec[q] = 1;
    append_entry(r, q, 1, lists, &state->packed[0]);
  }
  if (q == 0 && threadIdx.x < 4) words[threadIdx.x] = 0;
  stream_noise(r, streams[2 * q], streams[2 * q + 1], 1);
}

// End of one round of attempts (one block per replica): the first accepted
// candidate (or, when all were rejected, the positions after all were taken
// back) becomes the position; the attempts taken and the draws consumed (3N
// per attempt, rounded up to even) are counted.  A replica stops when a move
// was accepted or it has used max_move_attempts (error bit ATTEMPTS, as
// box.py:248 asserts); otherwise it joins the next round's list and draws the
// noise of its next attempts.  The last block to finish closes the round:
// words[0] = whether any replica still moves; inside the step's graph the
// WHILE node's condition is set to it, and a round cap bounds every launch.
constexpr int BATCH_ROUND_CAP = 4096;
__global__ void __launch_bounds__(512) batch_round_end_kernel(
    const BatchDev* __restrict__ reps, unsigned char* __restrict__ mask, int* __restrict__ ovl, int* __restrict__ spec,
    int* __restrict__ att, const int* __restrict__ maxatt, unsigned long long* __restrict__ streams,
    int* __restrict__ words, RoundEntry* lists, int cap, RoundState* state, cudaGraphConditionalHandle handle,
    int use_handle) {
  __shared__ int s_take, s_next;
  const int q = blockIdx.x, par = words[2] & 1;
  const BatchDev r = reps[q];
  const bool moving = mask[q] != 0;
  __syncthreads();  // thread 0 changes mask[q] below
  if (moving) {
    if (threadIdx.x == 0) {
      const int n = spec[q];
      int k = 0;
      while (k < n && ovl[q * SPEC + k]) ++k;
      for (int a = 0; a < n; ++a) ovl[q * SPEC + a] = 0;
      s_take = k;  // n: none accepted, U[n] holds the positions after the undo
      const int used = k < n ? k + 1 : n, total = att[q] + used;
      att[q] = total;
      streams[2 * q + 1] += (unsigned long long)used * (unsigned long long)(r.n + (r.n & 1));
      s_next = 0;
      if (k < n) {
        mask[q] = 0;
      } else if (total >= maxatt[q]) {
        mask[q] = 0;
        atomicOr(words + 1, (int)PBG_DEV_ERR_ATTEMPTS);
      } else {
        s_next = spec[q] = min(SPEC, maxatt[q] - total);
        append_entry(r, q, s_next, lists + (size_t)(par ^ 1) * cap, &state->packed[par ^ 1]);
      }
    }
    __syncthreads();
    const double* src = r.U + (size_t)s_take * r.ld;
    for (int i = threadIdx.x; i < r.n; i += blockDim.x) r.pos[i] = src[i];
    if (s_next) stream_noise(r, streams[2 * q], streams[2 * q + 1], s_next);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    if (atomicAdd(&state->done, 1) == (int)gridDim.x - 1) {
      __threadfence();
      const int any = packed_count(atomicAdd(&state->packed[par ^ 1], 0ULL)) > 0;
      const int rounds = words[2] + 1;
      words[2] = rounds;
      words[0] = any;
      state->packed[par] = 0;
      state->done = 0;
      if (use_handle) cudaGraphSetConditional(handle, (any && rounds % BATCH_ROUND_CAP != 0) ? 1u : 0u);
    }
  }
}

// A host-driven attempt: the masked replicas' list (one attempt each), and its
// outcome -- the candidate or, on an overlap, the position after the undo.
__global__ void batch_attempt_list_kernel(const BatchDev* __restrict__ reps, int R,
                                          const unsigned char* __restrict__ mask, int* __restrict__ ovl,
                                          RoundEntry* lists, RoundState* state) {
  for (int q = threadIdx.x; q < R; q += blockDim.x) {
    ovl[q * SPEC] = 0;
    if (mask[q]) append_entry(reps[q], q, 1, lists, &state->packed[0]);
  }
}
__global__ void batch_attempt_end_kernel(const BatchDev* __restrict__ reps, const unsigned char* __restrict__ mask,
                                         int* __restrict__ ovl, int* __restrict__ rejected, RoundState* state) {
  const int q = blockIdx.y;
  if (q == 0 && blockIdx.x == 0 && threadIdx.x == 0) state->packed[0] = 0;
  if (!mask[q]) return;
  const BatchDev& r = reps[q];
  const int hit = ovl[q * SPEC];
  if (blockIdx.x == 0 && threadIdx.x == 0) rejected[q] = hit;
  const double* src = r.U + (hit ? r.ld : 0);
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < r.n; i += gridDim.x * blockDim.x) r.pos[i] = src[i];
}

inline size_t elem_size(int precision) { return precision == PBG_PREC_FP64 ? 8 : 4; }

// Replica buffers come from the stream-ordered pool on the legacy default
// stream: allocation and release are ordered after the batch's earlier work
// on that stream (and on every blocking stream) and need no device-wide sync.
void free_replica(BatchReplica* r) {
  if (!r) return;
  void* bufs[] = {r->pos, r->radii, r->force, r->U, r->xi, r->D, r->B, r->invdiag, r->tasks};
  for (void* p : bufs)
    if (p) cudaFreeAsync(p, 0);
  delete r;
}

bool pool_alloc(void* p, size_t bytes) {
  return cudaMallocAsync(static_cast<void**>(p), bytes, 0) == cudaSuccess;
}

template <typename P>
void free_dev(P*& p) {
  if (p) cudaFree(p);
  p = nullptr;
}

// Device array of at least `bytes`, kept between rebuilds (grow only).
template <typename P>
int ensure(P*& p, size_t& cap, size_t bytes) {
  if (bytes <= cap && p) return PBG_OK;
  if (p) cudaFree(p);
  p = nullptr;
  cap = 0;
  const size_t want = std::max<size_t>(bytes + bytes / 4, 256);
  if (cudaMalloc((void**)&p, want) != cudaSuccess) {
    cudaGetLastError();
    pbg_set_error_message("out of device memory for the batch descriptors (%zu bytes)", want);
    return PBG_ERR_NOMEM;
  }
  cap = want;
  return PBG_OK;
}

// Merged task list: copies every segment and writes its replica index.
__global__ void gather_tasks_kernel(const GatherSeg* __restrict__ segs, int nseg, int4* __restrict__ out) {
  for (int s = blockIdx.x; s < nseg; s += gridDim.x) {
    const GatherSeg g = segs[s];
    for (int t = threadIdx.x; t < g.count; t += blockDim.x) {
      int4 v = g.src[t];
      v.x = (v.x & 7) | (g.replica << 3);
      out[g.dst + t] = v;
    }
  }
}

// Ewald work list: replica q's lower-triangle bead tiles (I, J), I >= J, in
// row order, at parts[q].y; parts[q].x = tiles per edge.
__global__ void ewald_work_kernel(const int4* __restrict__ parts, int4* __restrict__ out) {
  const int q = blockIdx.y;
  const int T = parts[q].x;
  const long long off = parts[q].y;
  const int total = T * (T + 1) / 2;
  for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < total; t += gridDim.x * blockDim.x) {
    int I = (int)((sqrt(8.0 * t + 1.0) - 1.0) * 0.5);
    while ((I + 1) * (I + 2) / 2 <= t) ++I;
    while (I * (I + 1) / 2 > t) --I;
    out[off + t] = make_int4(q, I, t - I * (I + 1) / 2, 0);
  }
}

// After device steps the device streams are ahead of the host's draw
// counts: copy them back (active order) before anything reads or changes
// them on the host or reorders the replicas.
int pull_draws(pbg_batch* b) {
  if (!b->host_draws_stale) return PBG_OK;
  const int R = (int)b->active.size();
  std::vector<unsigned long long> h(2 * (size_t)R);
  if (R) PBG_CUDA_TRY(cudaMemcpy(h.data(), b->d_stream, h.size() * sizeof(unsigned long long),
                                 cudaMemcpyDeviceToHost));
  for (int q = 0; q < R; ++q) {
    BatchReplica* r = b->slots[b->active[q]];
    if (r) r->draws = h[2 * q + 1];
  }
  b->host_draws_stale = false;
  b->streams_on_device = false;
  return PBG_OK;
}

// Uploads every replica's (seed, draws) in the active order, unless the
// device copy is current.
int push_streams(pbg_batch* b, cudaStream_t st) {
  if (b->streams_on_device) return PBG_OK;
  const int R = (int)b->active.size();
  std::vector<unsigned long long> streams(2 * (size_t)R);
  for (int q = 0; q < R; ++q) {
    const BatchReplica* r = b->slots[b->active[q]];
    streams[2 * q] = r->seed;
    streams[2 * q + 1] = r->draws;
  }
  // pageable source: staged before the call returns
  if (R) PBG_CUDA_TRY(cudaMemcpyAsync(b->d_stream, streams.data(), streams.size() * sizeof(unsigned long long),
                                      cudaMemcpyHostToDevice, st));
  b->streams_on_device = true;
  return PBG_OK;
}

void drop_graphs(pbg_batch* b) {
  if (b->begin_exec) {
    cudaGraphExecDestroy(b->begin_exec);
    b->begin_exec = nullptr;
  }
  if (b->step_exec) {
    cudaGraphExecDestroy(b->step_exec);
    b->step_exec = nullptr;
  }
}

// One replica of a merged task list: its segments, tile rows and matrix bytes.
struct MergeItem {
  int segments, nt;
  size_t bytes;
};

// The order of the replicas' task segments (see cholesky_df.cu) in the one list, as
// (replica, segment): every replica's spread evenly over the longest one's, so
// that the smaller ones fill the waits of the longest to its end instead of its
// first columns only (a serving batch of 24: 3277 -> 3201 us; FP64, 40 replicas:
// 161 -> 150), at one place with larger matrices first (default), in the order the
// replicas were added, or smaller first; replica after replica (all of one
// replica's segments, larger replicas first); or larger first in chunks of
// replicas whose matrices fit a byte budget, chunk after chunk.  Each replica's own
// segments keep their order in every policy, so every task still depends
// only on earlier tasks.
std::vector<std::pair<int, int>> merge_segments(int merge_order, const std::vector<MergeItem>& r) {
  const int R = (int)r.size();
  int longest = 0;
  std::vector<int> order(R);
  for (int q = 0; q < R; ++q) {
    order[q] = q;
    longest = std::max(longest, r[q].segments);
  }
  if (merge_order != PBG_MERGE_ADDED) {
    const bool larger = merge_order != PBG_MERGE_SMALLER_FIRST;
    std::stable_sort(order.begin(), order.end(),
                     [&](int x, int y) { return larger ? r[x].nt > r[y].nt : r[x].nt < r[y].nt; });
  }
  std::vector<std::pair<int, int>> out;
  auto push = [&](int q, int sg) {
    if (sg < r[q].segments) out.emplace_back(q, sg);
  };
  if (merge_order == PBG_MERGE_REPLICA_MAJOR) {
    for (int q : order)
      for (int sg = 0; sg < longest; ++sg) push(q, sg);
  } else if (merge_order >= PBG_MERGE_CHUNK_32M) {
    // chunks of consecutive (larger-first) replicas within the byte budget
    const size_t budget = (size_t)32 << (20 + (merge_order - PBG_MERGE_CHUNK_32M));
    for (size_t c0 = 0; c0 < order.size();) {
      size_t c1 = c0, bytes = 0;
      do bytes += r[order[c1++]].bytes;
      while (c1 < order.size() && bytes + r[order[c1]].bytes <= budget);
      for (int sg = 0; sg < longest; ++sg)
        for (size_t q = c0; q < c1; ++q) push(order[q], sg);
      c0 = c1;
    }
  } else {
    std::vector<int> next(R, 0);
    for (int tick = 0; tick < longest; ++tick)
      for (int q : order)
        for (; next[q] < r[q].segments && next[q] * (long long)longest / r[q].segments == tick; ++next[q])
          push(q, next[q]);
  }
  return out;
}

// Rebuilds the device descriptors and work lists of the current membership:
// small per-replica descriptors from the host, the task and tile work lists
// assembled on the device from each replica's cached list.
int rebuild(pbg_batch* b, cudaStream_t st) {
  int rc0 = pull_draws(b);
  if (rc0) return rc0;
  b->streams_on_device = false;
  drop_graphs(b);
  b->key_repeats = 0;
  b->key_build = -1;
  b->active.clear();
  for (int s = 0; s < (int)b->slots.size(); ++s)
    if (b->slots[s]) b->active.push_back(s);
  const int R = (int)b->active.size();
  b->n_ework = b->ntasks = 0;
  if ((size_t)R > b->cap || !b->d_ovl) {
    // the kernels of earlier steps on this stream may still read the old
    // arrays: the stream-ordered frees wait for them, the host buffers are
    // released once the stream has drained
    PBG_CUDA_TRY(cudaStreamSynchronize(st));
    for (void* p : {(void*)b->d_ovl, (void*)b->d_mask, (void*)b->d_stream, (void*)b->d_maxatt, (void*)b->d_rejected,
                    (void*)b->d_spec, (void*)b->d_lists, (void*)b->d_state})
      if (p) PBG_CUDA_TRY(cudaFreeAsync(p, st));
    b->d_ovl = nullptr;
    b->d_mask = nullptr;
    b->d_stream = nullptr;
    b->d_maxatt = nullptr;
    b->d_rejected = b->d_spec = nullptr;
    b->d_lists = nullptr;
    b->d_state = nullptr;
    if (b->h_ovl) cudaFreeHost(b->h_ovl);
    if (b->h_info) cudaFreeHost(b->h_info);
    if (b->h_step) cudaFreeHost(b->h_step);
    b->h_ovl = b->h_info = b->h_step = nullptr;
    b->cap = std::max<size_t>(2 * R, 16);
    PBG_CUDA_TRY(cudaMallocAsync((void**)&b->d_ovl, b->cap * SPEC * sizeof(int), st));
    PBG_CUDA_TRY(cudaMallocAsync((void**)&b->d_rejected, b->cap * sizeof(int), st));
    PBG_CUDA_TRY(cudaMallocAsync((void**)&b->d_spec, b->cap * sizeof(int), st));
    PBG_CUDA_TRY(cudaMallocAsync((void**)&b->d_lists, 2 * b->cap * sizeof(RoundEntry), st));
    PBG_CUDA_TRY(cudaMallocAsync((void**)&b->d_state, sizeof(RoundState), st));
    PBG_CUDA_TRY(cudaMallocAsync((void**)&b->d_mask, b->cap, st));
    PBG_CUDA_TRY(cudaMallocAsync((void**)&b->d_stream, 2 * b->cap * sizeof(unsigned long long), st));
    PBG_CUDA_TRY(cudaMallocAsync((void**)&b->d_maxatt, b->cap * sizeof(int), st));
    PBG_CUDA_TRY(cudaMallocHost(&b->h_ovl, b->cap * sizeof(int)));
    PBG_CUDA_TRY(cudaMallocHost(&b->h_info, b->cap * sizeof(int)));
    PBG_CUDA_TRY(cudaMallocHost(&b->h_step, (2 * b->cap + 4) * sizeof(int)));
  }
  b->max_n = 0;
  if (R == 0) {
    b->dirty = false;
    return PBG_OK;
  }
  // grow-only arrays: the kernels of earlier steps must be done with them
  PBG_CUDA_TRY(cudaStreamSynchronize(st));
  std::vector<BatchDev> reps(R);
  std::vector<unsigned char> rpy(R * rpy_batch_arg_bytes());
  std::vector<int4> eparts(R);
  size_t flag_ints = 4, n_ework = 0, ntasks = 0;
  std::vector<size_t> flag_off(R);
  for (int q = 0; q < R; ++q) {
    const BatchReplica* r = b->slots[b->active[q]];
    flag_off[q] = flag_ints;
    flag_ints += 2 * (size_t)r->nt * r->nt;
    b->max_n = std::max(b->max_n, r->n);
    const int T = (r->N + 15) / 16;
    eparts[q] = make_int4(T, (int)n_ework, 0, 0);
    n_ework += (size_t)T * (T + 1) / 2;
    ntasks += r->seg_start.empty() ? 0 : r->seg_start.back();
  }
  // after the per-replica flags: the infos, the attempt counts and the step
  // words, contiguous so that one copy reports a step
  const size_t info_off = flag_ints;
  flag_ints += 2 * (size_t)R + 4;
  b->flag_ints = flag_ints;
  int rc;
  if ((rc = ensure(b->d_flags, b->cap_flags, flag_ints * sizeof(int)))) return rc;
  b->d_info = b->d_flags + info_off;
  b->d_att = b->d_info + R;
  b->d_words = b->d_att + R;
  std::vector<CholRep> chol(R);
  const bool smith = b->hydrodynamics == PBG_HI_RPY_SMITH;
  for (int q = 0; q < R; ++q) {
    BatchReplica* r = b->slots[b->active[q]];
    BatchDev& d = reps[q];
    d.pos = r->pos;
    d.radii = r->radii;
    d.force = r->force;
    d.U = r->U;
    d.xi = r->xi;
    d.D = r->D;
    d.B = r->B;
    d.L = r->p.box_length;
    d.thr = r->p.overlap_treshold;
    d.kBT = r->p.kBT;
    d.N = r->N;
    d.n = r->n;
    d.ld = r->ld;
    d.check = r->p.check_overlaps;
    d.has_force = r->has_force;
    d.pad = 0;
    rpy_batch_arg(r->pos, r->radii, r->N, r->p.box_length, smith, b->tables, r->scale, r->D, r->B, r->ld,
                  rpy.data() + q * rpy_batch_arg_bytes());
    CholRep& c = chol[q];
    c.A = r->B;
    c.invdiag = r->invdiag;
    c.upd = b->d_flags + flag_off[q];
    c.fin = c.upd + (size_t)r->nt * r->nt;
    c.info = b->d_info + q;
    c.ld = r->ld;
    c.n = r->n;
    c.nt = r->nt;
    c.pad = 0;
  }
  std::vector<MergeItem> items(R);
  for (int q = 0; q < R; ++q) {
    const BatchReplica* r = b->slots[b->active[q]];
    items[q] = MergeItem{(int)r->seg_start.size() - 1, r->nt, (size_t)r->ld * r->ld * elem_size(b->precision)};
  }
  std::vector<GatherSeg> segs;
  long long dst = 0;
  for (const auto& e : merge_segments(b->merge_order, items)) {
    const BatchReplica* r = b->slots[b->active[e.first]];
    const int start = r->seg_start[e.second], count = r->seg_start[e.second + 1] - start;
    if (count <= 0) continue;
    segs.push_back(GatherSeg{r->tasks + start, dst, count, e.first});
    dst += count;
  }
  if ((rc = ensure(b->d_reps, b->cap_reps, R * sizeof(BatchDev))) ||
      (rc = ensure(b->d_rpy, b->cap_rpy, rpy.size())) ||
      (rc = ensure(b->d_ework, b->cap_ework, n_ework * sizeof(int4))) ||
      (rc = ensure(b->d_chol, b->cap_chol, R * sizeof(CholRep))) ||
      (rc = ensure(b->d_tasks, b->cap_tasks, std::max<size_t>(ntasks, 1) * sizeof(int4))) ||
      (rc = ensure(b->d_segs, b->cap_segs, std::max<size_t>(segs.size(), 1) * sizeof(GatherSeg))) ||
      (rc = ensure(b->d_eparts, b->cap_eparts, R * sizeof(int4))))
    return rc;
  PBG_CUDA_TRY(cudaMemsetAsync(b->d_state, 0, sizeof(RoundState), st));
  PBG_CUDA_TRY(cudaMemsetAsync(b->d_ovl, 0, b->cap * SPEC * sizeof(int), st));
  // pageable sources: each copy is staged before the call returns
  PBG_CUDA_TRY(cudaMemcpyAsync(b->d_reps, reps.data(), R * sizeof(BatchDev), cudaMemcpyHostToDevice, st));
  PBG_CUDA_TRY(cudaMemcpyAsync(b->d_rpy, rpy.data(), rpy.size(), cudaMemcpyHostToDevice, st));
  PBG_CUDA_TRY(cudaMemcpyAsync(b->d_chol, chol.data(), R * sizeof(CholRep), cudaMemcpyHostToDevice, st));
  PBG_CUDA_TRY(cudaMemcpyAsync(b->d_eparts, eparts.data(), R * sizeof(int4), cudaMemcpyHostToDevice, st));
  std::vector<int> maxatt(R);
  for (int q = 0; q < R; ++q) maxatt[q] = std::max(1, b->slots[b->active[q]]->p.max_move_attempts);
  PBG_CUDA_TRY(cudaMemcpyAsync(b->d_maxatt, maxatt.data(), R * sizeof(int), cudaMemcpyHostToDevice, st));
  if (!segs.empty()) {
    PBG_CUDA_TRY(cudaMemcpyAsync(b->d_segs, segs.data(), segs.size() * sizeof(GatherSeg), cudaMemcpyHostToDevice,
                                 st));
    gather_tasks_kernel<<<(int)std::min<size_t>(segs.size(), 148 * 16), 256, 0, st>>>(b->d_segs, (int)segs.size(),
                                                                                      b->d_tasks);
    PBG_CHECK_LAUNCH();
  }
  ewald_work_kernel<<<dim3(8, R), 256, 0, st>>>(b->d_eparts, b->d_ework);
  PBG_CHECK_LAUNCH();
  b->n_ework = (int)n_ework;
  b->ntasks = (int)dst;
  b->dirty = false;
  return PBG_OK;
}

inline dim3 rows_grid(const pbg_batch* b, int per_block) {
  const int x = std::max(1, std::min(64, (b->max_n + per_block - 1) / per_block));
  return dim3(x, (unsigned)b->active.size());
}

// Copies the host mask (indexed by slot, or all when null) to the device in
// the order of the active replicas.  Returns the number of masked replicas.
// Small uploads go from pageable memory: the copy is staged before the call
// returns, so the host vectors can change right away.
int upload_mask(pbg_batch* b, const unsigned char* mask, cudaStream_t st, int* count) {
  const int R = (int)b->active.size();
  b->mask.assign(R, 0);
  int c = 0;
  for (int q = 0; q < R; ++q) {
    b->mask[q] = mask ? (mask[b->active[q]] ? 1 : 0) : 1;
    c += b->mask[q];
  }
  *count = c;
  if (R) PBG_CUDA_TRY(cudaMemcpyAsync(b->d_mask, b->mask.data(), R, cudaMemcpyHostToDevice, st));
  return PBG_OK;
}

}  // namespace
}  // namespace pbg

using namespace pbg;

extern "C" {

PBG_API int pbg_batch_create(const pbg_params* tmpl, pbg_batch** out) {
  if (!tmpl || !out) return PBG_ERR_ARG;
  if (tmpl->hydrodynamics != PBG_HI_RPY && tmpl->hydrodynamics != PBG_HI_RPY_SMITH) {
    pbg_set_error_message("batched replicas support the rpy and rpy_smith hydrodynamics");
    return PBG_ERR_ARG;
  }
  if (tmpl->precision != PBG_PREC_FP64 && tmpl->precision != PBG_PREC_MIXED) return PBG_ERR_ARG;
  if (tmpl->propagation_scheme != PBG_SCHEME_ERMAK) {
    pbg_set_error_message("batched replicas support the ermak propagation scheme");
    return PBG_ERR_ARG;
  }
  auto* b = new pbg_batch();
  b->precision = tmpl->precision;
  b->hydrodynamics = tmpl->hydrodynamics;
  if (b->hydrodynamics == PBG_HI_RPY_SMITH) {
    b->alpha = tmpl->ewald_alpha;
    b->m_max = tmpl->ewald_real;
    b->n_max = tmpl->ewald_imag;
    int rc = get_ewald_tables(b->alpha, b->m_max, b->n_max, &b->tables);
    if (rc) {
      delete b;
      return rc;
    }
  }
  *out = b;
  return PBG_OK;
}

PBG_API int pbg_batch_destroy(pbg_batch* b) {
  if (!b) return PBG_OK;
  cudaDeviceSynchronize();
  for (auto* r : b->slots) free_replica(r);
  free_dev(b->d_reps);
  free_dev(b->d_rpy);
  free_dev(b->d_ework);
  free_dev(b->d_chol);
  free_dev(b->d_tasks);
  free_dev(b->d_segs);
  free_dev(b->d_eparts);
  free_dev(b->d_flags);
  free_dev(b->d_ovl);
  free_dev(b->d_mask);
  free_dev(b->d_stream);
  free_dev(b->d_maxatt);
  free_dev(b->d_rejected);
  free_dev(b->d_spec);
  free_dev(b->d_lists);
  free_dev(b->d_state);
  if (b->h_ovl) cudaFreeHost(b->h_ovl);
  if (b->h_info) cudaFreeHost(b->h_info);
  if (b->h_step) cudaFreeHost(b->h_step);
  drop_graphs(b);
  if (b->cap_stream) cudaStreamDestroy(b->cap_stream);
  if (b->cap_stream2) cudaStreamDestroy(b->cap_stream2);
  delete b;
  return PBG_OK;
}

PBG_API int pbg_cholesky_task_list(int nt, int precision, int* tasks, int cap, int* seg, int seg_cap, int* n_tasks,
                                   int* n_segs) {
  if (nt < 1 || !tasks || !seg || !n_tasks || !n_segs) return PBG_ERR_ARG;
  std::vector<int4> list;
  std::vector<int> starts;
  cholesky_replica_tasks(nt, precision, list, starts);
  *n_tasks = (int)list.size();
  *n_segs = (int)starts.size();
  if ((int)list.size() > cap || (int)starts.size() > seg_cap) return PBG_ERR_ARG;
  for (size_t t = 0; t < list.size(); ++t) {
    tasks[4 * t + 0] = list[t].x;
    tasks[4 * t + 1] = list[t].y;
    tasks[4 * t + 2] = list[t].z;
    tasks[4 * t + 3] = list[t].w;
  }
  for (size_t q = 0; q < starts.size(); ++q) seg[q] = starts[q];
  return PBG_OK;
}

PBG_API int pbg_cholesky_merge_list(int precision, int merge_order, const int* nts, int n_replicas, int* out, int cap,
                                    int* n_out) {
  if (!nts || !out || !n_out || n_replicas < 1 || merge_order < 0 || merge_order >= PBG_MERGE_ORDERS)
    return PBG_ERR_ARG;
  std::vector<MergeItem> items;
  for (int q = 0; q < n_replicas; ++q) {
    if (nts[q] < 1) return PBG_ERR_ARG;
    std::vector<int4> list;
    std::vector<int> starts;
    cholesky_replica_tasks(nts[q], precision, list, starts);
    const size_t ld = (size_t)nts[q] * PBG_TILE;
    items.push_back(MergeItem{(int)starts.size() - 1, nts[q], ld * ld * elem_size(precision)});
  }
  const auto merged = merge_segments(merge_order, items);
  *n_out = (int)merged.size();
  if ((int)merged.size() > cap) return PBG_ERR_ARG;
  for (size_t e = 0; e < merged.size(); ++e) {
    out[2 * e] = merged[e].first;
    out[2 * e + 1] = merged[e].second;
  }
  return PBG_OK;
}

// Device bytes a replica of n_beads takes in a batch of this precision (the
// Ewald build keeps no per-bead tables, so the lattice does not enter).
PBG_API long long pbg_batch_footprint(int precision, int hydrodynamics, int ewald_imag, int n_beads) {
  (void)hydrodynamics;
  (void)ewald_imag;
  const long long n = 3LL * n_beads, ld = (n + PBG_TILE - 1) / PBG_TILE * PBG_TILE, nt = ld / PBG_TILE;
  const long long es = elem_size(precision);
  return 2 * ld * ld * es + nt * PBG_TILE * PBG_TILE * es + ((2 * SPEC + 2) * ld + 4 * n_beads) * 8 + 2 * nt * nt * 4;
}

PBG_API int pbg_batch_add(pbg_batch* b, const pbg_params* p, const double* pos, const double* radii, int* slot) {
  if (!b || !p || !pos || !radii || !slot || p->n_beads <= 0 || !(p->box_length > 0) || !(p->kBT > 0) ||
      !(p->viscosity > 0))
    return PBG_ERR_ARG;
  if (b->in_step) {
    pbg_set_error_message("pbg_batch_add inside a step");
    return PBG_ERR_STATE;
  }
  int prc = pull_draws(b);
  if (prc) return prc;
  auto* r = new BatchReplica();
  r->p = *p;
  r->N = p->n_beads;
  r->n = 3 * r->N;
  r->ld = (r->n + PBG_TILE - 1) / PBG_TILE * PBG_TILE;
  r->nt = r->ld / PBG_TILE;
  r->scale = p->kBT * 1e19 / p->viscosity;
  const size_t es = elem_size(b->precision), ld = r->ld;
  batch_pool_keep();
  bool ok = pool_alloc(&r->pos, r->n * sizeof(double)) && pool_alloc(&r->radii, r->N * sizeof(double)) &&
            pool_alloc(&r->force, ld * sizeof(double)) && pool_alloc(&r->U, (SPEC + 1) * ld * sizeof(double)) &&
            pool_alloc(&r->xi, SPEC * ld * sizeof(double)) && pool_alloc(&r->D, ld * ld * es) &&
            pool_alloc(&r->B, ld * ld * es) && pool_alloc(&r->invdiag, (size_t)r->nt * PBG_TILE * PBG_TILE * es);
  std::vector<int4> tasks;
  cholesky_replica_tasks(r->nt, b->precision, tasks, r->seg_start);
  if (ok && !tasks.empty()) {
    ok = pool_alloc(&r->tasks, tasks.size() * sizeof(int4)) &&
         cudaMemcpyAsync(r->tasks, tasks.data(), tasks.size() * sizeof(int4), cudaMemcpyHostToDevice, 0) ==
             cudaSuccess;
  }
  if (!ok) {
    cudaGetLastError();
    free_replica(r);
    pbg_set_error_message("out of device memory adding a replica of %d beads", p->n_beads);
    return PBG_ERR_NOMEM;
  }
  cudaMemsetAsync(r->force, 0, ld * sizeof(double), 0);
  cudaMemsetAsync(r->U, 0, (SPEC + 1) * ld * sizeof(double), 0);
  cudaMemsetAsync(r->xi, 0, SPEC * ld * sizeof(double), 0);
  // ordered on the legacy stream after the allocations; a pageable source is
  // staged before the call returns
  PBG_CUDA_TRY(cudaMemcpyAsync(r->pos, pos, r->n * sizeof(double), cudaMemcpyDefault, 0));
  PBG_CUDA_TRY(cudaMemcpyAsync(r->radii, radii, r->N * sizeof(double), cudaMemcpyDefault, 0));
  int s = 0;
  while (s < (int)b->slots.size() && b->slots[s]) ++s;
  if (s == (int)b->slots.size()) b->slots.push_back(nullptr);
  b->slots[s] = r;
  b->dirty = true;
  *slot = s;
  return PBG_OK;
}

static BatchReplica* slot_of(pbg_batch* b, int slot) {
  if (!b || slot < 0 || slot >= (int)b->slots.size()) return nullptr;
  return b->slots[slot];
}

PBG_API int pbg_batch_remove(pbg_batch* b, int slot) {
  BatchReplica* r = slot_of(b, slot);
  if (!r) return PBG_ERR_ARG;
  if (b->in_step) {
    pbg_set_error_message("pbg_batch_remove inside a step");
    return PBG_ERR_STATE;
  }
  int rc = pull_draws(b);
  if (rc) return rc;
  free_replica(r);
  b->slots[slot] = nullptr;
  b->dirty = true;
  return PBG_OK;
}

PBG_API int pbg_batch_slots(pbg_batch* b) { return b ? (int)b->slots.size() : 0; }

PBG_API int pbg_batch_set_positions(pbg_batch* b, int slot, const double* pos) {
  BatchReplica* r = slot_of(b, slot);
  if (!r || !pos) return PBG_ERR_ARG;
  PBG_CUDA_TRY(cudaMemcpy(r->pos, pos, r->n * sizeof(double), cudaMemcpyDefault));
  return PBG_OK;
}

PBG_API int pbg_batch_get_positions(pbg_batch* b, int slot, double* out) {
  BatchReplica* r = slot_of(b, slot);
  if (!r || !out) return PBG_ERR_ARG;
  PBG_CUDA_TRY(cudaMemcpy(out, r->pos, r->n * sizeof(double), cudaMemcpyDefault));
  return PBG_OK;
}

// Stream-ordered copy of one replica's positions into `out` (pinned host
// memory for the copy to be asynchronous); the caller waits on the stream.
PBG_API int pbg_batch_get_positions_async(pbg_batch* b, int slot, double* out, void* stream) {
  BatchReplica* r = slot_of(b, slot);
  if (!r || !out) return PBG_ERR_ARG;
  PBG_CUDA_TRY(cudaMemcpyAsync(out, r->pos, r->n * sizeof(double), cudaMemcpyDefault, (cudaStream_t)stream));
  return PBG_OK;
}

PBG_API int pbg_batch_set_force(pbg_batch* b, int slot, const double* F) {
  BatchReplica* r = slot_of(b, slot);
  if (!r) return PBG_ERR_ARG;
  if (F) PBG_CUDA_TRY(cudaMemcpy(r->force, F, r->n * sizeof(double), cudaMemcpyDefault));
  else PBG_CUDA_TRY(cudaMemset(r->force, 0, r->n * sizeof(double)));
  if (r->has_force != (F != nullptr)) b->dirty = true;
  r->has_force = F != nullptr;
  return PBG_OK;
}

// Noise for the next attempt of one replica (3N normals, host or device memory).
PBG_API int pbg_batch_set_noise(pbg_batch* b, int slot, const double* xi) {
  BatchReplica* r = slot_of(b, slot);
  if (!r || !xi) return PBG_ERR_ARG;
  PBG_CUDA_TRY(cudaMemcpy(r->xi, xi, r->n * sizeof(double), cudaMemcpyDefault));
  return PBG_OK;
}

PBG_API int pbg_batch_set_seed(pbg_batch* b, int slot, unsigned long long seed, unsigned long long draws) {
  BatchReplica* r = slot_of(b, slot);
  if (!r) return PBG_ERR_ARG;
  int rc = pull_draws(b);
  if (rc) return rc;
  r->seed = seed;
  r->draws = draws + (draws & 1);
  b->streams_on_device = false;
  return PBG_OK;
}

PBG_API int pbg_batch_get_draws(pbg_batch* b, int slot, unsigned long long* draws) {
  BatchReplica* r = slot_of(b, slot);
  if (!r || !draws) return PBG_ERR_ARG;
  int rc = pull_draws(b);
  if (rc) return rc;
  *draws = r->draws;
  return PBG_OK;
}

// Fills the masked replicas' noise from their counter-based streams and
// advances each stream by 3N draws (rounded up to even).
PBG_API int pbg_batch_fill_noise(pbg_batch* b, const unsigned char* mask, void* stream) {
  if (!b) return PBG_ERR_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  int rc;
  if (b->dirty && (rc = rebuild(b, st))) return rc;
  const int R = (int)b->active.size();
  if (!R) return PBG_OK;
  int count = 0;
  if ((rc = upload_mask(b, mask, st, &count))) return rc;
  if (!count) return PBG_OK;
  // the stream positions of this fill (the host counts are authoritative here)
  if ((rc = pull_draws(b))) return rc;
  b->streams_on_device = false;
  if ((rc = push_streams(b, st))) return rc;
  batch_noise_kernel<<<rows_grid(b, 512), 256, 0, st>>>(b->d_reps, b->d_mask, b->d_stream);
  PBG_CHECK_LAUNCH();
  for (int q = 0; q < R; ++q)
    if (b->mask[q]) {
      BatchReplica* r = b->slots[b->active[q]];
      r->draws += (unsigned long long)(r->n + (r->n & 1));
    }
  b->streams_on_device = false;  // the device copy is now behind the host counts
  return PBG_OK;
}

// The device work of a step's start: D (build_D), B = chol(D) (cholesky) of
// every replica and the deterministic move of the replicas with a force.
static int enqueue_begin(pbg_batch* b, double dt, int build_D, int cholesky, bool any_force, cudaStream_t st) {
  const int R = (int)b->active.size();
  const bool f64 = b->precision == PBG_PREC_FP64;
  const bool smith = b->hydrodynamics == PBG_HI_RPY_SMITH;
  int rc;
  // a step that builds and factors D has the Ewald build write D's lower
  // triangle (and the padding) into B as well
  if (build_D && (rc = launch_rpy_batch(b->precision, smith, b->tables, b->d_rpy, b->d_ework, b->n_ework,
                                        cholesky != 0, st)))
    return rc;
  if (cholesky) {
    if (!build_D) {
      const dim3 g(64, R);
      if (f64) batch_copy_lower_kernel<double><<<g, 256, 0, st>>>(b->d_reps);
      else batch_copy_lower_kernel<float><<<g, 256, 0, st>>>(b->d_reps);
      PBG_CHECK_LAUNCH();
    }
    PBG_CUDA_TRY(cudaMemsetAsync(b->d_flags, 0, b->flag_ints * sizeof(int), st));
    if ((rc = launch_cholesky_batch(b->precision, b->d_chol, b->d_tasks, b->ntasks, b->d_flags, b->ctas_per_sm, st)))
      return rc;
  }
  if (any_force) {
    if (f64) batch_det_kernel<double><<<rows_grid(b, 8), 256, 0, st>>>(b->d_reps, dt);
    else batch_det_kernel<float><<<rows_grid(b, 8), 256, 0, st>>>(b->d_reps, dt);
    PBG_CHECK_LAUNCH();
    batch_det_move_kernel<<<rows_grid(b, 256), 256, 0, st>>>(b->d_reps);
    PBG_CHECK_LAUNCH();
  }
  return PBG_OK;
}

// Captures enqueue_begin into b->begin_exec on the private stream.  A refusal
// by the driver (capture or instantiation) leaves graph_refused set and the
// step runs its launches directly; any other error is returned.
static int capture_begin(pbg_batch* b, double dt, int build_D, int cholesky, bool any_force) {
  if (!b->cap_stream) PBG_CUDA_TRY(cudaStreamCreateWithFlags(&b->cap_stream, cudaStreamNonBlocking));
  const long long l0 = pbg_launch_count();
  if (cudaStreamBeginCapture(b->cap_stream, cudaStreamCaptureModeRelaxed) != cudaSuccess) {
    cudaGetLastError();
    b->graph_refused = true;
    return PBG_OK;
  }
  int rc = enqueue_begin(b, dt, build_D, cholesky, any_force, b->cap_stream);
  cudaGraph_t graph = nullptr;
  const cudaError_t end = cudaStreamEndCapture(b->cap_stream, &graph);
  const long long kernels = pbg_launch_count() - l0;
  pbg_count_launches(-kernels);  // nothing ran yet
  pbg_count_host_calls(-kernels);
  if (rc != PBG_OK || end != cudaSuccess || !graph) {
    if (graph) cudaGraphDestroy(graph);
    cudaGetLastError();
    b->graph_refused = true;
    return PBG_OK;
  }
  const cudaError_t inst = cudaGraphInstantiate(&b->begin_exec, graph, 0);
  cudaGraphDestroy(graph);
  if (inst != cudaSuccess) {
    cudaGetLastError();
    b->begin_exec = nullptr;
    b->graph_refused = true;
    return PBG_OK;
  }
  b->begin_kernels = kernels;
  return PBG_OK;
}

// Builds D (build_D) and B = chol(D) (cholesky) of every replica and applies
// the deterministic step of the replicas with a force.  The second and later
// steps with the same membership, flags and dt replay one CUDA graph.
PBG_API int pbg_batch_step_begin(pbg_batch* b, double dt, int build_D, int cholesky, void* stream) {
  if (!b || !(dt > 0)) return PBG_ERR_ARG;
  if (b->in_step) {
    pbg_set_error_message("pbg_batch_step_begin inside a step");
    return PBG_ERR_STATE;
  }
  cudaStream_t st = (cudaStream_t)stream;
  int rc;
  if (b->dirty && (rc = rebuild(b, st))) return rc;
  b->dt = dt;
  const int R = (int)b->active.size();
  if (!R) {
    b->in_step = true;
    return PBG_OK;
  }
  bool any_force = false;
  for (int s : b->active) any_force = any_force || b->slots[s]->has_force;
  const bool same = b->key_build == build_D && b->key_chol == cholesky && b->key_force == (int)any_force &&
                    b->key_dt == dt;
  if (!same) {
    if (b->begin_exec) {
      cudaGraphExecDestroy(b->begin_exec);
      b->begin_exec = nullptr;
    }
    b->key_build = build_D;
    b->key_chol = cholesky;
    b->key_force = (int)any_force;
    b->key_dt = dt;
    b->key_repeats = 0;
  }
  ++b->key_repeats;
  if (!b->begin_exec && !b->graph_refused && b->key_repeats >= 2 &&
      (rc = capture_begin(b, dt, build_D, cholesky, any_force)))
    return rc;
  if (b->begin_exec) {
    PBG_CUDA_TRY(cudaGraphLaunch(b->begin_exec, st));
    pbg_count_launches(b->begin_kernels);
    pbg_count_host_calls(1);
  } else if ((rc = enqueue_begin(b, dt, build_D, cholesky, any_force, st))) {
    return rc;
  }
  if (build_D) b->have_D = true;
  b->in_step = true;
  return PBG_OK;
}

// Blocks of the list-driven kernels: four (product) and eight per SM, fewer
// where the batch has fewer units.
static int round_blocks(const pbg_batch* b, int per_sm, int unit_rows, int rows) {
  const long long units = (long long)b->active.size() * ((rows + unit_rows - 1) / unit_rows);
  return (int)std::max<long long>(1, std::min<long long>(units, 148LL * per_sm));
}

static int enqueue_moves(pbg_batch* b, const int* rounds, cudaStream_t st) {
  const double s1 = std::sqrt(2 * b->dt);
  const int cap = (int)b->cap, blocks = round_blocks(b, 4, TRMV_ROWS, b->max_n);
  if (b->precision == PBG_PREC_FP64)
    batch_trmv_kernel<double><<<blocks, 256, 0, st>>>(b->d_reps, b->d_lists, cap, b->d_state, rounds, s1);
  else
    batch_trmv_kernel<float><<<blocks, 256, 0, st>>>(b->d_reps, b->d_lists, cap, b->d_state, rounds, s1);
  PBG_CHECK_LAUNCH();
  batch_overlap_kernel<<<round_blocks(b, 8, 1, b->max_n), 256, 0, st>>>(b->d_reps, b->d_lists, cap, b->d_state, rounds,
                                                                        b->d_ovl);
  PBG_CHECK_LAUNCH();
  return PBG_OK;
}

// One round of attempts of the replicas still moving: the product and the
// candidates, the overlap tests, the outcome.  Three kernels.
static int enqueue_round(pbg_batch* b, cudaStream_t st, cudaGraphConditionalHandle handle, int use_handle) {
  if (int rc = enqueue_moves(b, b->d_words + 2, st)) return rc;
  batch_round_end_kernel<<<(int)b->active.size(), 512, 0, st>>>(b->d_reps, b->d_mask, b->d_ovl, b->d_spec, b->d_att,
                                                                b->d_maxatt, b->d_stream, b->d_words, b->d_lists,
                                                                (int)b->cap, b->d_state, handle, use_handle);
  PBG_CHECK_LAUNCH();
  return PBG_OK;
}
constexpr int ROUND_KERNELS = 3;

// The wrap into the box and the step's report (infos, attempts, words) into
// pinned host memory.
static int enqueue_step_tail(pbg_batch* b, cudaStream_t st) {
  const int R = (int)b->active.size();
  batch_wrap_kernel<<<rows_grid(b, 256), 256, 0, st>>>(b->d_reps);
  PBG_CHECK_LAUNCH();
  PBG_CUDA_TRY(cudaMemcpyAsync(b->h_step, b->d_info, (2 * (size_t)R + 4) * sizeof(int), cudaMemcpyDeviceToHost, st));
  return PBG_OK;
}

static int enqueue_round_init(pbg_batch* b, cudaStream_t st) {
  const int R = (int)b->active.size();
  PBG_CUDA_TRY(cudaMemsetAsync(b->d_state, 0, sizeof(RoundState), st));
  batch_round_init_kernel<<<R, 256, 0, st>>>(b->d_reps, b->d_mask, b->d_att, b->d_words, b->d_ovl, b->d_spec,
                                             b->d_stream, b->d_lists, b->d_state);
  PBG_CHECK_LAUNCH();
  return PBG_OK;
}

// Captures a whole device step into b->step_exec: the start (enqueue_begin),
// the round initialisation, a conditional WHILE node whose body is one round
// (its last kernel sets the condition), and the tail.  A refusal by the
// driver leaves graph_refused set (direct launches from then on).
static int capture_step(pbg_batch* b, double dt, int build_D, int cholesky, bool any_force) {
  if (!b->cap_stream) PBG_CUDA_TRY(cudaStreamCreateWithFlags(&b->cap_stream, cudaStreamNonBlocking));
  if (!b->cap_stream2) PBG_CUDA_TRY(cudaStreamCreateWithFlags(&b->cap_stream2, cudaStreamNonBlocking));
  const long long l0 = pbg_launch_count();
  auto refuse = [&](cudaGraph_t g) {
    if (g) cudaGraphDestroy(g);
    cudaGetLastError();
    const long long k = pbg_launch_count() - l0;  // nothing ran
    pbg_count_launches(-k);
    pbg_count_host_calls(-k);
    b->graph_refused = true;
    return PBG_OK;
  };
  if (cudaStreamBeginCapture(b->cap_stream, cudaStreamCaptureModeRelaxed) != cudaSuccess) return refuse(nullptr);
  int rc = enqueue_begin(b, dt, build_D, cholesky, any_force, b->cap_stream);
  if (rc == PBG_OK) rc = enqueue_round_init(b, b->cap_stream);
  const long long fixed0 = pbg_launch_count() - l0;
  bool ok = rc == PBG_OK;
  cudaGraph_t g = nullptr;
  cudaGraphConditionalHandle handle = 0;
  cudaGraphNodeParams cp = {};
  if (ok) {
    cudaStreamCaptureStatus cs;
    const cudaGraphNode_t* deps = nullptr;
    size_t ndeps = 0;
    ok = cudaStreamGetCaptureInfo(b->cap_stream, &cs, nullptr, &g, &deps, &ndeps) == cudaSuccess &&
         cs == cudaStreamCaptureStatusActive &&
         cudaGraphConditionalHandleCreate(&handle, g, 1, cudaGraphCondAssignDefault) == cudaSuccess;
    cudaGraphNode_t wnode = nullptr;
    if (ok) {
      cp.type = cudaGraphNodeTypeConditional;
      cp.conditional.handle = handle;
      cp.conditional.type = cudaGraphCondTypeWhile;
      cp.conditional.size = 1;
      ok = cudaGraphAddNode(&wnode, g, deps, ndeps, &cp) == cudaSuccess &&
           cudaStreamUpdateCaptureDependencies(b->cap_stream, &wnode, 1, cudaStreamSetCaptureDependencies) ==
               cudaSuccess;
    }
    if (ok) {
      ok = cudaStreamBeginCaptureToGraph(b->cap_stream2, cp.conditional.phGraph_out[0], nullptr, nullptr, 0,
                                         cudaStreamCaptureModeRelaxed) == cudaSuccess;
      if (ok) {
        rc = enqueue_round(b, b->cap_stream2, handle, 1);
        cudaGraph_t body = nullptr;
        ok = cudaStreamEndCapture(b->cap_stream2, &body) == cudaSuccess && rc == PBG_OK;
      }
    }
  }
  if (ok) ok = enqueue_step_tail(b, b->cap_stream) == PBG_OK;
  cudaGraph_t graph = nullptr;
  const cudaError_t end = cudaStreamEndCapture(b->cap_stream, &graph);
  if (!ok || end != cudaSuccess || !graph) return refuse(graph);
  const cudaError_t inst = cudaGraphInstantiate(&b->step_exec, graph, 0);
  cudaGraphDestroy(graph);
  if (inst != cudaSuccess) {
    b->step_exec = nullptr;
    return refuse(nullptr);
  }
  // kernels per replay besides the rounds: the start, the initialisation and the wrap
  b->step_fixed_kernels = fixed0 + 1;
  const long long k = pbg_launch_count() - l0;  // nothing ran yet
  pbg_count_launches(-k);
  pbg_count_host_calls(-k);
  return PBG_OK;
}

// 1 while the start of a step (or, with pbg_batch_step, the whole step)
// replays a CUDA graph, 0 while it launches its kernels directly, -1 if the
// driver refused the capture.
PBG_API int pbg_batch_graph_state(pbg_batch* b) {
  if (!b) return 0;
  return b->graph_refused ? -1 : ((b->begin_exec || b->step_exec) ? 1 : 0);
}

// A whole step of every replica with device noise (see the header).
PBG_API int pbg_batch_step(pbg_batch* b, double dt, int build_D, int cholesky, int* status, int* attempts,
                           void* stream) {
  if (!b || !(dt > 0)) return PBG_ERR_ARG;
  if (b->in_step) {
    pbg_set_error_message("pbg_batch_step inside a step");
    return PBG_ERR_STATE;
  }
  cudaStream_t st = (cudaStream_t)stream;
  int rc;
  if (b->dirty && (rc = rebuild(b, st))) return rc;
  const int R = (int)b->active.size();
  if (!R) return PBG_OK;
  if ((rc = push_streams(b, st))) return rc;
  b->dt = dt;
  bool any_force = false;
  for (int s : b->active) any_force = any_force || b->slots[s]->has_force;
  const bool same = b->key_build == build_D && b->key_chol == cholesky && b->key_force == (int)any_force &&
                    b->key_dt == dt;
  if (!same) {
    drop_graphs(b);
    b->key_build = build_D;
    b->key_chol = cholesky;
    b->key_force = (int)any_force;
    b->key_dt = dt;
    b->key_repeats = 0;
  }
  ++b->key_repeats;
  if (!b->step_exec && !b->graph_refused && b->key_repeats >= 2 &&
      (rc = capture_step(b, dt, build_D, cholesky, any_force)))
    return rc;
  const int* words = b->h_step + 2 * R;
  if (b->step_exec) {
    PBG_CUDA_TRY(cudaGraphLaunch(b->step_exec, st));
    PBG_CUDA_TRY(cudaStreamSynchronize(st));
    pbg_count_launches(b->step_fixed_kernels + (long long)ROUND_KERNELS * words[2]);
    pbg_count_host_calls(1);
  } else {
    if ((rc = enqueue_begin(b, dt, build_D, cholesky, any_force, st)) || (rc = enqueue_round_init(b, st)))
      return rc;
  }
  // rounds launched from the host: all of them without a graph, or those
  // beyond the graph's round cap
  int* h_words = b->h_step + 2 * R;
  bool more = !b->step_exec;
  if (b->step_exec && words[0]) {
    more = true;
  }
  while (more) {
    if ((rc = enqueue_round(b, st, 0, 0))) return rc;
    PBG_CUDA_TRY(cudaMemcpyAsync(h_words, b->d_words, 4 * sizeof(int), cudaMemcpyDeviceToHost, st));
    PBG_CUDA_TRY(cudaStreamSynchronize(st));
    more = h_words[0] != 0;
  }
  if (!b->step_exec || words[0]) {
    // not replayed, or rounds were added: the tail runs here
    if ((rc = enqueue_step_tail(b, st))) return rc;
    PBG_CUDA_TRY(cudaStreamSynchronize(st));
  }
  b->have_D = b->have_D || build_D;
  b->streams_on_device = true;
  b->host_draws_stale = true;
  int worst = 0;
  for (int q = 0; q < R; ++q) {
    const int slot = b->active[q];
    if (status) status[slot] = b->h_step[q];
    if (attempts) attempts[slot] = b->h_step[R + q];
    if (b->h_step[q] < 0) worst = -1;
    else if (b->h_step[q] > 0 && worst == 0) worst = 1;
  }
  if (words[1] & PBG_DEV_ERR_ATTEMPTS) {
    pbg_set_error_message("maximal number of move attempts exceeded in a batched step");
    return PBG_ERR_ATTEMPTS;
  }
  if (worst < 0) {
    pbg_set_error_message("a device-wide wait in the batched factorisation gave up");
    return PBG_ERR_BARRIER;
  }
  if (worst > 0) {
    pbg_set_error_message("a replica's diffusion matrix is not positive definite");
    return PBG_ERR_NOT_SPD;
  }
  return PBG_OK;
}

PBG_API int pbg_batch_step_attempt(pbg_batch* b, const unsigned char* mask, unsigned char* accepted, void* stream) {
  if (!b) return PBG_ERR_ARG;
  if (!b->in_step) {
    pbg_set_error_message("pbg_batch_step_attempt outside a step");
    return PBG_ERR_STATE;
  }
  cudaStream_t st = (cudaStream_t)stream;
  const int R = (int)b->active.size();
  if (!R) return PBG_OK;
  int count = 0, rc;
  if ((rc = upload_mask(b, mask, st, &count))) return rc;
  if (!count) return PBG_OK;
  PBG_CUDA_TRY(cudaMemsetAsync(b->d_state, 0, sizeof(RoundState), st));
  batch_attempt_list_kernel<<<1, 256, 0, st>>>(b->d_reps, R, b->d_mask, b->d_ovl, b->d_lists, b->d_state);
  PBG_CHECK_LAUNCH();
  if ((rc = enqueue_moves(b, nullptr, st))) return rc;
  batch_attempt_end_kernel<<<rows_grid(b, 256), 256, 0, st>>>(b->d_reps, b->d_mask, b->d_ovl, b->d_rejected, b->d_state);
  PBG_CHECK_LAUNCH();
  PBG_CUDA_TRY(cudaMemcpyAsync(b->h_ovl, b->d_rejected, R * sizeof(int), cudaMemcpyDeviceToHost, st));
  PBG_CUDA_TRY(cudaStreamSynchronize(st));
  if (accepted)
    for (int q = 0; q < R; ++q)
      if (b->mask[q]) accepted[b->active[q]] = b->h_ovl[q] ? 0 : 1;
  return PBG_OK;
}

// Wraps every replica into its box and reports the factorisation status of
// the step: status[slot] (host, optional) = 0, or the first non-positive
// pivot (1-based), or -1 when a wait of the factorisation gave up.
PBG_API int pbg_batch_step_end(pbg_batch* b, int* status, void* stream) {
  if (!b) return PBG_ERR_ARG;
  if (!b->in_step) {
    pbg_set_error_message("pbg_batch_step_end outside a step");
    return PBG_ERR_STATE;
  }
  b->in_step = false;
  cudaStream_t st = (cudaStream_t)stream;
  const int R = (int)b->active.size();
  if (!R) return PBG_OK;
  batch_wrap_kernel<<<rows_grid(b, 256), 256, 0, st>>>(b->d_reps);
  PBG_CHECK_LAUNCH();
  PBG_CUDA_TRY(cudaMemcpyAsync(b->h_info, b->d_info, R * sizeof(int), cudaMemcpyDeviceToHost, st));
  PBG_CUDA_TRY(cudaStreamSynchronize(st));
  int worst = 0;
  for (int q = 0; q < R; ++q) {
    if (status) status[b->active[q]] = b->h_info[q];
    if (b->h_info[q] < 0) worst = -1;
    else if (b->h_info[q] > 0 && worst == 0) worst = 1;
  }
  if (worst < 0) {
    pbg_set_error_message("a device-wide wait in the batched factorisation gave up");
    return PBG_ERR_BARRIER;
  }
  if (worst > 0) {
    pbg_set_error_message("a replica's diffusion matrix is not positive definite");
    return PBG_ERR_NOT_SPD;
  }
  return PBG_OK;
}

// D or B (which = PBG_MAT_D / PBG_MAT_B) of one replica as a 3N x 3N FP64
// row-major host array.
PBG_API int pbg_batch_set_schedule(pbg_batch* b, int merge_order, int ctas_per_sm) {
  if (!b || merge_order < PBG_MERGE_LARGER_FIRST || merge_order >= PBG_MERGE_ORDERS || ctas_per_sm < 0)
    return PBG_ERR_ARG;
  if (b->in_step) {
    pbg_set_error_message("pbg_batch_set_schedule inside a step");
    return PBG_ERR_STATE;
  }
  if (merge_order != b->merge_order) b->dirty = true;
  b->merge_order = merge_order;
  b->ctas_per_sm = ctas_per_sm;
  return PBG_OK;
}

// Times the copy of D into B and the batched factorisation under each
// schedule.  Refactoring the current D reproduces the current B bit for bit
// (every tile's arithmetic is fixed by the task order of its replica).
PBG_API int pbg_batch_autotune(pbg_batch* b, int reps, int* best, float* ms, void* stream) {
  if (!b || reps < 1 || !best) return PBG_ERR_ARG;
  if (b->in_step || !b->have_D) {
    pbg_set_error_message("pbg_batch_autotune needs a completed step and must be called between steps");
    return PBG_ERR_STATE;
  }
  cudaStream_t st = (cudaStream_t)stream;
  const int R = (int)b->active.size();
  const bool f64 = b->precision == PBG_PREC_FP64;
  int max_ctas = 1, sms = 0;
  if (R) {
    const int rr = cholesky_batch_residency(b->precision, &max_ctas, &sms);
    if (rr) return rr;
  }
  max_ctas = std::min(max_ctas, 2);
  if (ms)
    for (int c = 0; c < 2 * PBG_MERGE_ORDERS; ++c) ms[c] = -1.0f;
  const int old_order = b->merge_order, old_ctas = b->ctas_per_sm;
  float best_ms = -1.0f;
  best[0] = old_order;
  best[1] = old_ctas;
  cudaEvent_t e0, e1;
  PBG_CUDA_TRY(cudaEventCreate(&e0));
  PBG_CUDA_TRY(cudaEventCreate(&e1));
  int rc = PBG_OK;
  for (int order = PBG_MERGE_LARGER_FIRST; order < PBG_MERGE_ORDERS && rc == PBG_OK && R; ++order) {
    for (int ctas = 1; ctas <= max_ctas && rc == PBG_OK; ++ctas) {
      b->merge_order = order;
      b->ctas_per_sm = ctas;
      b->dirty = true;
      if ((rc = rebuild(b, st))) break;
      float total = 0.0f;
      for (int r = 0; r <= reps && rc == PBG_OK; ++r) {  // the first run is a warm-up
        if (cudaEventRecord(e0, st) != cudaSuccess) { rc = PBG_ERR_CUDA; break; }
        const dim3 g(64, R);
        if (f64) batch_copy_lower_kernel<double><<<g, 256, 0, st>>>(b->d_reps);
        else batch_copy_lower_kernel<float><<<g, 256, 0, st>>>(b->d_reps);
        if (cudaGetLastError() != cudaSuccess) { rc = PBG_ERR_CUDA; break; }
        pbg_count_launch();
        if (cudaMemsetAsync(b->d_flags, 0, b->flag_ints * sizeof(int), st) != cudaSuccess) { rc = PBG_ERR_CUDA; break; }
        if ((rc = launch_cholesky_batch(b->precision, b->d_chol, b->d_tasks, b->ntasks, b->d_flags, ctas, st))) break;
        if (cudaEventRecord(e1, st) != cudaSuccess || cudaEventSynchronize(e1) != cudaSuccess) { rc = PBG_ERR_CUDA; break; }
        float t = 0.0f;
        cudaEventElapsedTime(&t, e0, e1);
        if (r) total += t;
      }
      if (rc != PBG_OK) break;
      const float mean = total / reps;
      if (ms) ms[order * 2 + ctas - 1] = mean;
      if (best_ms < 0.0f || mean < best_ms) {
        best_ms = mean;
        best[0] = order;
        best[1] = ctas;
      }
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  b->merge_order = rc == PBG_OK ? best[0] : old_order;
  b->ctas_per_sm = rc == PBG_OK ? best[1] : old_ctas;
  b->dirty = true;
  if (rc == PBG_OK) {
    // surface a failed factorisation like a step would
    PBG_CUDA_TRY(cudaMemcpyAsync(b->h_info, b->d_info, R * sizeof(int), cudaMemcpyDeviceToHost, st));
    PBG_CUDA_TRY(cudaStreamSynchronize(st));
    for (int q = 0; q < R; ++q)
      if (b->h_info[q] != 0) {
        pbg_set_error_message("factorisation failed during autotuning (replica %d, info %d)", q, b->h_info[q]);
        return b->h_info[q] < 0 ? PBG_ERR_BARRIER : PBG_ERR_NOT_SPD;
      }
  }
  return rc;
}

// Factors a copy of one replica's current D with the single-matrix kernel
// (the batch's precision) and returns its status in *info (0, a 1-based
// non-positive pivot, or -1): after a failed batched step, tells a matrix
// that is not positive definite from a factorisation that failed on a good
// one.  B and the replica's state are left as they are.
PBG_API int pbg_batch_check_factor(pbg_batch* b, int slot, int* info, void* stream) {
  BatchReplica* r = slot_of(b, slot);
  if (!r || !info) return PBG_ERR_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  const size_t es = elem_size(b->precision), ld = r->ld;
  void *A = nullptr, *work = nullptr;
  int* dinfo = nullptr;
  const size_t wbytes = cholesky_work_bytes(r->ld, b->precision);
  if (cudaMallocAsync(&A, ld * ld * es, st) != cudaSuccess || cudaMallocAsync(&work, wbytes, st) != cudaSuccess ||
      cudaMallocAsync((void**)&dinfo, sizeof(int), st) != cudaSuccess) {
    cudaGetLastError();
    if (A) cudaFreeAsync(A, st);
    if (work) cudaFreeAsync(work, st);
    pbg_set_error_message("out of device memory checking a replica's factorisation");
    return PBG_ERR_NOMEM;
  }
  int rc = PBG_OK;
  if (cudaMemcpyAsync(A, r->D, ld * ld * es, cudaMemcpyDeviceToDevice, st) != cudaSuccess) rc = PBG_ERR_CUDA;
  if (rc == PBG_OK) rc = launch_pad_identity(A, r->n, r->ld, b->precision, st);
  if (rc == PBG_OK) rc = launch_cholesky_ws(A, r->n, r->ld, b->precision, dinfo, work, st);
  int h = 0;
  if (rc == PBG_OK && (cudaMemcpyAsync(&h, dinfo, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
                       cudaStreamSynchronize(st) != cudaSuccess))
    rc = PBG_ERR_CUDA;
  cudaFreeAsync(A, st);
  cudaFreeAsync(work, st);
  cudaFreeAsync(dinfo, st);
  *info = h;
  return rc;
}

PBG_API int pbg_batch_get_matrix(pbg_batch* b, int slot, int which, double* out) {
  BatchReplica* r = slot_of(b, slot);
  if (!r || !out || (which != PBG_MAT_D && which != PBG_MAT_B)) return PBG_ERR_ARG;
  const size_t es = elem_size(b->precision), ld = r->ld;
  std::vector<unsigned char> h(ld * ld * es);
  PBG_CUDA_TRY(cudaMemcpy(h.data(), which == PBG_MAT_D ? r->D : r->B, h.size(), cudaMemcpyDeviceToHost));
  for (int i = 0; i < r->n; ++i)
    for (int j = 0; j < r->n; ++j) {
      double v;
      if (es == 8) v = reinterpret_cast<const double*>(h.data())[(size_t)i * ld + j];
      else v = reinterpret_cast<const float*>(h.data())[(size_t)i * ld + j];
      if (which == PBG_MAT_B && j > i) v = 0.0;
      out[(size_t)i * r->n + j] = v;
    }
  return PBG_OK;
}

}  // extern "C"
