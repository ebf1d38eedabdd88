// Data-flow tiled Cholesky factorisation on sm_100a (the factor of
// numpy.linalg.cholesky at src/bdsim/pyBrown/box.py:554).
//
// Single matrix: one persistent kernel, all CTAs co-resident (cooperative
// launch), one CTA per SM.  The 64 x 64 tiles of the lower triangle are
// processed as tasks:
//   F(k)     diagonal tile k: its last update (column k-1), the factorisation
//            by 8-column panels, and the solve blocks of L_kk (factor_tile);
//   S(i, k)  tile (i, k) below the diagonal: its last update, then
//            L_ik = A_ik L_kk^-T by forward substitution with 8 x 8 blocks
//            (solve_rows);
//   U(i,j,k) trailing update A_ij -= L_ik L_jk^T (j >= k+2): FP64 DMMA
//            (mma.sync m8n8k4 f64) in the FP64 path; in the mixed path
//            3xTF32 split products (hi*hi + hi*lo + lo*hi) on the tcgen05
//            tensor cores, up to four rows per task, accumulated in TMEM
//            (tc_tile.cuh);
//   LEAD(k, h) half h of row k+2 of panel k: S(k+2, k), U(k+2, k+1, k) as
//            one task, because the chain waits for them;
//   I(k)     inv(L_kk), only when the caller wants the inverted diagonal tiles.
// The diagonal tiles are factored in FP64 in every path, in the mixed path (FP32
// matrix) rounded to FP32 on store.
//
// The critical path of the factorisation is F(0), S(1,0), F(1), S(2,1), ...:
// block 0 (the chain CTA) runs exactly that sequence and keeps what one step
// hands to the next in shared memory (the solve blocks for S(k+1, k);
// L(k+1, k) for the update of F(k+1)), so the chain never waits on a round
// trip through L2.  The other CTAs take the remaining tasks in a fixed order
// from an atomic counter (df_task_list).  With an output X (the SPD inverse)
// the same list also forms X = inv(L) (XG / XZ tasks).  Every task depends only
// on chain tasks and on tasks earlier in the list, so with all CTAs resident
// the lowest unfinished task can always run.
//
// Batches of independent matrices: FP64 right-looking tile tasks
// (chol_batch_kernel<double>); mixed left-looking tasks that accumulate a
// whole K range on the tcgen05 tensor cores (chol_batch_ll_kernel).
//
// Dependencies are tracked per tile (per row in the left-looking batch):
// upd counts applied updates, fin marks final L tiles.  Waits spin on these
// flags with a bounded iteration count; on expiry the kernel raises an abort
// flag, marks info = -1 and every CTA returns.  Tile data written by other
// CTAs is read with L2-coherent loads (ld.global.cg, cp.async.cg).
#include <algorithm>
#include <map>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "kernels.cuh"
#include "tc_tile.cuh"

namespace pbg {

namespace {

constexpr int NB = 64;
constexpr int THREADS = 256;
constexpr int TILE_PER_THREAD = 64 * 64 / THREADS;  // elements of a 64 x 64 tile per thread
constexpr int LDA = NB + 4;   // staged tile row (bank-conflict-free fragment and row loads)
constexpr long long SPIN_LIMIT = 1LL << 24;

// TASK_U2 / TASK_U3 / TASK_U4: U(i, j, k) .. U(i+r-1, j, k) as one task (they
// share L_jk).  Groups of three and four rows only in the FP32 single-matrix
// list, whose update tasks run on the tcgen05 tensor cores.
enum : int { TASK_F = 0, TASK_S = 1, TASK_U = 2, TASK_I = 3, TASK_U2 = 4, TASK_U3 = 5, TASK_U4 = 6 };
// XG / XZ: the tasks that form X = inv(L) in the same list (single-matrix
// lists of an SPD inverse only; see inverse_update / inverse_finish).
enum : int { TASK_XG = 7, TASK_XZ = 8 };
// LEAD(k, h): half of the tile row k + 2 of panel k, on which the chain's next
// step waits (lead_task).
enum : int { TASK_LEAD = 9 };

// Pivots that a tile's factorisation takes: 1 / d of others is flushed to zero or
// infinite (pivot_rcp).  They are reported as non-positive.
constexpr double MIN_PIVOT = 2.2250738585072014e-308, MAX_PIVOT = 4.49423283715579e307;  // 2^-1022, 2^1022

struct DFArgs {
  void* A;
  int ld, n, nt, ntasks;
  const int4* tasks;
  int* ctl;      // [0] next task, [1] abort, [2] spin failures
  int* upd;      // nt * nt
  int* fin;      // nt * nt
  int* info;
  void* invdiag; // nt * 64 * 64: inv(L_kk), row-major tiles (I tasks)
  void* lp;      // nt * 64 * 64: the solve blocks of L_kk (factor_tile)
  unsigned* err;
  long long spin_limit;  // polls before a wait gives up
  void* X;       // or null: X = inv(L) is formed too (off-diagonal tiles of the ld x ld matrix)
  int* xupd;     // nt * nt: terms applied to X's tile (i, j)
  int* xfin;     // nt * nt: X's tile (i, j) final
  double min_pivot = MIN_PIVOT;  // a pivot below it counts as non-positive
};

__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.b32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

#ifdef PBG_TASK_TRACE
// Optional per-task timeline (build with -DPBG_TASK_TRACE): for task t,
// [fetch, waits done, end] in globaltimer ns and the SM id.  The chain tasks
// F(k), S(k+1, k) take the slots ntasks + 2k, ntasks + 2k + 1.
__device__ long long g_task_trace[4 * 65536];
__device__ __forceinline__ long long gtimer() {
  long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ int smid() {
  int s;
  asm volatile("mov.u32 %0, %%smid;" : "=r"(s));
  return s;
}
#define TRACE(slot, t) \
  if (threadIdx.x == 0 && (t) < 65536) g_task_trace[4 * (t) + (slot)] = (slot) == 3 ? smid() : gtimer()
// Phase totals of the left-looking batch workers: per CTA, 16 slots of
// clock64 cycles or counts (see ll_task).
__device__ long long g_ll_prof[1024 * 16];
#define LLPROF(slot, v) \
  if (threadIdx.x == 0 && blockIdx.x < 1024) g_ll_prof[blockIdx.x * 16 + (slot)] += (v)
#define LLCLK() clock64()
// Finer timeline of the chain: 8 stamps per panel k.
__device__ long long g_chain_trace[8 * 1024];
#define CTRACE(k, slot) \
  if (threadIdx.x == 0 && (k) < 1024) g_chain_trace[8 * (k) + (slot)] = gtimer()
#else
#define TRACE(slot, t)
#define CTRACE(k, slot)
#define LLPROF(slot, v) ((void)(v))
#define LLCLK() 0LL
#endif

__device__ __forceinline__ double ldcg(const double* p) { return __ldcg(p); }
__device__ __forceinline__ float ldcg(const float* p) { return __ldcg(p); }

// A bounded wait ran out: every CTA gives up, and the caller learns of it.
__device__ __forceinline__ void wait_expired(const DFArgs& a) {
  atomicExch(a.ctl + 1, 1);
  atomicAdd(a.ctl + 2, 1);
  atomicOr(a.err, PBG_DEV_ERR_BARRIER);
  atomicCAS(a.info, 0, -1);  // -1: the factorisation gave up waiting
}

// Warp 0 waits until every flags[q] >= targets[q] (count <= 9, bounded);
// returns false if the run was aborted.  Lane q polls flag q, so one round
// costs one L2 round trip whatever the count.  The acquire loads followed by
// the CTA barrier order every thread's later reads after the producers'
// release.
__device__ bool wait_all(const DFArgs& a, const int* const* flags, const int* targets, int count, int* s_ok) {
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    const int* flag = nullptr;
    int target = 0;
#pragma unroll
    for (int q = 0; q < 9; ++q)  // compile-time indices: the arrays stay in registers
      if (q < count && q == lane) {
        flag = flags[q];
        target = targets[q];
      }
    bool done = flag == nullptr;
    int ok = 1;
    for (long long it = 0;; ++it) {
      if (!done) done = ld_acquire(flag) >= target;
      if (__all_sync(0xffffffffu, done)) break;
      // the abort flag is polled every 16th round, so a round costs one L2 trip
      if ((it & 15) == 15) {
        const int ab = __shfl_sync(0xffffffffu, lane == 0 ? ld_acquire(a.ctl + 1) : 0, 0);
        if (ab) {
          ok = 0;
          break;
        }
      }
      if (it + 1 > a.spin_limit) {
        if (lane == 0) wait_expired(a);
        ok = 0;
        break;
      }
      if (it > 256) __nanosleep(200);
    }
    if (lane == 0) *s_ok = ok;
  }
  __syncthreads();
  return *s_ok != 0;
}

__device__ __forceinline__ bool wait_geq(const DFArgs& a, const int* flag, int target, int* s_ok) {
  return wait_all(a, &flag, &target, 1, s_ok);
}

// The CTA barrier makes every thread's tile stores happen-before thread 0's
// release store (release is cumulative), so no separate fence is needed.
__device__ __forceinline__ void publish(int* flag, int value) {
  __syncthreads();
  if (threadIdx.x == 0) st_release(flag, value);
}

__device__ __forceinline__ void cp_async16(void* smem_dst, const void* gmem_src) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem_dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s), "l"(gmem_src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
}

template <typename T>
__device__ __forceinline__ T* tile(const DFArgs& a, int i, int j) {
  return reinterpret_cast<T*>(a.A) + (size_t)i * NB * a.ld + (size_t)j * NB;
}

// Row-major asynchronous copy of a 64 x 64 tile into smem rows of `lds`
// elements, 16 bytes per cp.async (all issued before any wait).  The caller
// waits with cp_async_wait_all() and a barrier.
template <typename T>
__device__ __forceinline__ void stage_async(const T* g, int ld, T* s, int lds) {
  constexpr int per_row = NB * (int)sizeof(T) / 16;  // 16-byte chunks per row
  constexpr int elems = 16 / (int)sizeof(T);
#pragma unroll
  for (int q = 0; q < NB * per_row / THREADS; ++q) {
    const int t = threadIdx.x + q * THREADS;
    const int r = t / per_row, c = (t % per_row) * elems;
    cp_async16(s + r * lds + c, g + (size_t)r * ld + c);
  }
}

// Row-major copy of a 64 x 64 smem tile (rows of `lds`) to global, 16 bytes per store.
template <typename T>
__device__ __forceinline__ void store_tile(const T* s, int lds, T* g, int ld) {
  constexpr int elems = 16 / (int)sizeof(T);
  constexpr int per_row = NB / elems;
#pragma unroll
  for (int q = 0; q < NB * per_row / THREADS; ++q) {
    const int t = threadIdx.x + q * THREADS;
    const int r = t / per_row, c = (t % per_row) * elems;
    *reinterpret_cast<float4*>(g + (size_t)r * ld + c) = *reinterpret_cast<const float4*>(s + r * lds + c);
  }
}

// ---------------------------------------------------------------- tile GEMM
// Accumulator layout: 16 elements per thread; warp w owns rows 16*(w/2).. and
// columns 32*(w%2).. of the 64 x 64 tile.  Each thread holds two rows
// (row(rs), rs = 0, 1) times eight columns (col(cs), cs = 0..7); idx(rs, cs)
// is the element's place in the accumulator array.
__device__ __forceinline__ int acc_row(int rs) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  return 16 * (w >> 1) + 8 * rs + (lane >> 2);
}
__device__ __forceinline__ int acc_col(int cs) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  return 32 * (w & 1) + 8 * (cs >> 1) + 2 * (lane & 3) + (cs & 1);
}

template <typename T> struct TileMMA;

template <> struct TileMMA<double> {
  // mma.m8n8k4 f64: 2 m-tiles x 4 n-tiles of 8 x 8, 2 accumulators each.
  static __device__ __forceinline__ int idx(int rs, int cs) { return rs * 8 + cs; }
  // acc -= A B^T with A, B (64 x 64, rows = output row / column, cols = k) in smem.
  static __device__ __forceinline__ void sub(const double* sA, const double* sB, double acc[16]) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int m0 = 16 * (w >> 1), n0 = 32 * (w & 1), g = lane >> 2, t = lane & 3;
#pragma unroll 4
    for (int k0 = 0; k0 < NB; k0 += 4) {
      double a[2], b[4];
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) a[mt] = -sA[(m0 + 8 * mt + g) * LDA + k0 + t];
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) b[nt] = sB[(n0 + 8 * nt + g) * LDA + k0 + t];
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          double& c0 = acc[(mt * 4 + nt) * 2];
          double& c1 = acc[(mt * 4 + nt) * 2 + 1];
          asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                       : "+d"(c0), "+d"(c1)
                       : "d"(a[mt]), "d"(b[nt]));
        }
    }
  }
  // acc -= A B (AT false) or A^T B (AT true) with B, and A in the second case,
  // staged as they lie in memory (rows = k): a fragment's four k rows are 8
  // banks apart and its eight columns 2, so these loads are free of conflicts
  // where a transposing copy into shared memory meets 8-way ones.
  template <bool AT>
  static __device__ __forceinline__ void sub_rows(const double* sA, const double* sB, double acc[16]) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int m0 = 16 * (w >> 1), n0 = 32 * (w & 1), g = lane >> 2, t = lane & 3;
#pragma unroll 4
    for (int k0 = 0; k0 < NB; k0 += 4) {
      double a[2], b[4];
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
        a[mt] = AT ? -sA[(k0 + t) * LDA + m0 + 8 * mt + g] : -sA[(m0 + 8 * mt + g) * LDA + k0 + t];
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) b[nt] = sB[(k0 + t) * LDA + n0 + 8 * nt + g];
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) {
          double& c0 = acc[(mt * 4 + nt) * 2];
          double& c1 = acc[(mt * 4 + nt) * 2 + 1];
          asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                       : "+d"(c0), "+d"(c1)
                       : "d"(a[mt]), "d"(b[nt]));
        }
    }
  }
};


using tc::split_tf32;

template <> struct TileMMA<float> {
  // mma.m16n8k8 tf32: 1 m-tile of 16 x 4 n-tiles of 8, 4 accumulators each.
  // The product A B^T is accumulated from zero in its own registers and
  // subtracted from acc at the end: the tensor cores' accumulation rounds at
  // the magnitude of the product, not of the tile it updates, and acc takes
  // one FP32 rounding per product (accumulating into acc directly made the
  // factor's error grow with the number of panels, to 9e-6 at order 3072).
  static __device__ __forceinline__ int idx(int rs, int cs) { return (cs >> 1) * 4 + rs * 2 + (cs & 1); }
  static __device__ __forceinline__ void sub(const float* sA, const float* sB, float acc[16]) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int m0 = 16 * (w >> 1), n0 = 32 * (w & 1), g = lane >> 2, t = lane & 3;
    float prod[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) prod[e] = 0.0f;
#pragma unroll 2
    for (int k0 = 0; k0 < NB; k0 += 8) {
      // split the A fragment and the B fragments into tf32 hi + lo
      unsigned ah[4], al[4];
      {
        const float v[4] = {sA[(m0 + g) * LDA + k0 + t], sA[(m0 + g + 8) * LDA + k0 + t],
                            sA[(m0 + g) * LDA + k0 + t + 4], sA[(m0 + g + 8) * LDA + k0 + t + 4]};
#pragma unroll
        for (int q = 0; q < 4; ++q) split_tf32(v[q], ah[q], al[q]);
      }
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) {
        const float v0 = sB[(n0 + 8 * nt + g) * LDA + k0 + t];
        const float v1 = sB[(n0 + 8 * nt + g) * LDA + k0 + t + 4];
        unsigned bh0, bh1, bl0, bl1;
        split_tf32(v0, bh0, bl0);
        split_tf32(v1, bh1, bl1);
        float* c = prod + 4 * nt;
#define PBG_TF32_MMA(A0, A1, A2, A3, B0, B1)                                                        \
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, " \
               "{%8,%9}, {%0,%1,%2,%3};"                                                            \
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])                                     \
               : "r"(A0), "r"(A1), "r"(A2), "r"(A3), "r"(B0), "r"(B1))
        PBG_TF32_MMA(al[0], al[1], al[2], al[3], bh0, bh1);
        PBG_TF32_MMA(ah[0], ah[1], ah[2], ah[3], bl0, bl1);
        PBG_TF32_MMA(ah[0], ah[1], ah[2], ah[3], bh0, bh1);
#undef PBG_TF32_MMA
      }
    }
#pragma unroll
    for (int e = 0; e < 16; ++e) acc[e] -= prod[e];
  }
};

template <typename T>
__device__ __forceinline__ void load_acc(const T* g, int ld, T acc[16]) {
#pragma unroll
  for (int rs = 0; rs < 2; ++rs)
#pragma unroll
    for (int cs = 0; cs < 8; ++cs) acc[TileMMA<T>::idx(rs, cs)] = ldcg(g + (size_t)acc_row(rs) * ld + acc_col(cs));
}

template <typename T>
__device__ __forceinline__ void store_acc(T* g, int ld, const T acc[16]) {
#pragma unroll
  for (int rs = 0; rs < 2; ++rs)
#pragma unroll
    for (int cs = 0; cs < 8; ++cs) g[(size_t)acc_row(rs) * ld + acc_col(cs)] = acc[TileMMA<T>::idx(rs, cs)];
}

// Loads tile (i, j) into acc and applies update U(i, j, k): the two staged L
// tiles are copied asynchronously while the accumulator loads are in flight.
template <typename T>
__device__ __forceinline__ void load_and_update(const DFArgs& a, int i, int j, int k, T acc[16], T* sA, T* sB) {
  stage_async(tile<T>(a, i, k), a.ld, sA, LDA);
  if (i != j) stage_async(tile<T>(a, j, k), a.ld, sB, LDA);
  load_acc(tile<T>(a, i, j), a.ld, acc);
  cp_async_wait_all();
  __syncthreads();
  TileMMA<T>::sub(sA, i != j ? sB : sA, acc);
  __syncthreads();
}

// One warp's output tile D = A B of a small smem product on the tensor cores:
// A rows with stride lda (k contiguous), B k-major rows with stride ldb, K a
// multiple of 4: an 8 x 8 FP64 tile (mma m8n8k4), lane holds D[g][2t + h].
// (The diagonal tiles are inverted in FP64 in both paths.)
struct WarpTile64 {
  static constexpr int TM = 8;
  static __device__ __forceinline__ void mma(const double* A, int lda, const double* B, int ldb, int K, double d[4]) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    d[0] = d[1] = 0.0;
    for (int k0 = 0; k0 < K; k0 += 4) {
      const double a = A[g * lda + k0 + t], b = B[(k0 + t) * ldb + g];
      asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                   : "+d"(d[0]), "+d"(d[1])
                   : "d"(a), "d"(b));
    }
  }
  // element q of the lane's part of D: row, column within the tile
  static __device__ __forceinline__ int row(int q) { return (threadIdx.x & 31) >> 2; }
  static __device__ __forceinline__ int col(int q) { return 2 * (threadIdx.x & 3) + (q & 1); }
  static constexpr int NQ = 2;
};


// Inverse of the lower-triangular L_kk (in Lk, [64][LDA], zero above the
// diagonal) into X ([64][LDA]), with Rinv[j] = 1 / L_jj and scratch Tm
// (>= 32 x 36 T).  The eight 8 x 8 diagonal blocks are inverted by forward
// substitution (warp b, lane c < 8 owns column c of block b); then three
// doubling levels s = 8, 16, 32 fill the off-diagonal blocks:
//   inv([L11 0; L21 L22]) = [X11 0; -X22 (L21 X11) X22],  X_ii = inv(L_ii),
// each level two dependent block products: by one short dot product per
// thread at s = 8, by warp tensor-core tiles at s = 16 and 32.
template <typename T>
__device__ __forceinline__ void invert_factor(const T* Lk, const T* Rinv, T* X, T* Tm) {
  using WT = WarpTile64;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (lane < 8) {
    const T* D = Lk + 8 * warp * LDA + 8 * warp;
    const T* R = Rinv + 8 * warp;
    T x[8];
#pragma unroll
    for (int ii = 0; ii < 8; ++ii) {
      T sacc = 0;
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (q < ii && q >= lane) sacc += D[ii * LDA + q] * x[q];
      x[ii] = ii < lane ? T(0) : (ii == lane ? R[ii] : -sacc * R[ii]);
    }
#pragma unroll
    for (int ii = 0; ii < 8; ++ii) X[(8 * warp + ii) * LDA + 8 * warp + lane] = x[ii];
  }
  // blocks above the block diagonal are zero
  for (int t = tid; t < NB * NB; t += THREADS) {
    const int r = t >> 6, c = t & 63;
    if ((c >> 3) > (r >> 3)) X[r * LDA + c] = T(0);
  }
  __syncthreads();
  // s = 8: four 8 x 8 products per phase, one output per thread
  {
    const int m = tid >> 6, rr = (tid >> 3) & 7, cc = tid & 7, b0 = 16 * m;
    T v = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) v += Lk[(b0 + 8 + rr) * LDA + b0 + q] * X[(b0 + q) * LDA + b0 + cc];
    Tm[m * 64 + rr * 8 + cc] = v;
    __syncthreads();
    T u = 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) u += X[(b0 + 8 + rr) * LDA + b0 + 8 + q] * Tm[m * 64 + q * 8 + cc];
    X[(b0 + 8 + rr) * LDA + b0 + cc] = -u;
    __syncthreads();
  }
#pragma unroll
  for (int s = 16; s < NB; s *= 2) {
    const int ldt = s + 4;                              // Tm row stride
    const int tiles_r = s / WT::TM, tiles = (NB / (2 * s)) * tiles_r * (s / 8);
    // Tm = L21 X11 for every 2s x 2s diagonal block
    for (int q = warp; q < tiles; q += THREADS / 32) {
      const int m = q / (tiles_r * (s / 8)), tr = (q / (s / 8)) % tiles_r, tc = q % (s / 8), b0 = 2 * s * m;
      T d[4];
      WT::mma(Lk + (b0 + s + tr * WT::TM) * LDA + b0, LDA, X + b0 * LDA + b0 + 8 * tc, LDA, s, d);
      T* o = Tm + m * s * ldt + tr * WT::TM * ldt + 8 * tc;
#pragma unroll
      for (int e = 0; e < WT::NQ; ++e) o[WT::row(e) * ldt + WT::col(e)] = d[e];
    }
    __syncthreads();
    // X21 = -X22 Tm
    for (int q = warp; q < tiles; q += THREADS / 32) {
      const int m = q / (tiles_r * (s / 8)), tr = (q / (s / 8)) % tiles_r, tc = q % (s / 8), b0 = 2 * s * m;
      T d[4];
      WT::mma(X + (b0 + s + tr * WT::TM) * LDA + b0 + s, LDA, Tm + m * s * ldt + 8 * tc, ldt, s, d);
      T* o = X + (b0 + s + tr * WT::TM) * LDA + b0 + 8 * tc;
#pragma unroll
      for (int e = 0; e < WT::NQ; ++e) o[WT::row(e) * LDA + WT::col(e)] = -d[e];
    }
    __syncthreads();
  }
}

// inv(L_kk) from Lk ([64][LDA], zero above the diagonal) and Rinv = 1 / L_jj
// into X, then to the global invdiag array as S.  Scratch: Tm (>= 32 x 36).
template <typename T, typename S>
__device__ __forceinline__ void store_inverse(const DFArgs& a, int k, const T* Lk, const T* Rinv, T* X, T* Tm) {
  invert_factor(Lk, Rinv, X, Tm);
  S* inv = reinterpret_cast<S*>(a.invdiag) + (size_t)k * NB * NB;
  if constexpr (sizeof(S) == sizeof(T)) {
    store_tile(X, LDA, inv, NB);
  } else {
    for (int t = threadIdx.x; t < NB * NB; t += THREADS) inv[t] = (S)X[(t >> 6) * LDA + (t & 63)];
  }
}

template <typename T>
__device__ __forceinline__ void smem_to_acc(const T* s, T acc[16]) {
#pragma unroll
  for (int rs = 0; rs < 2; ++rs)
#pragma unroll
    for (int cs = 0; cs < 8; ++cs) acc[TileMMA<T>::idx(rs, cs)] = s[acc_row(rs) * LDA + acc_col(cs)];
}

template <typename T>
__device__ __forceinline__ void acc_to_smem(const T acc[16], T* s, int lds = LDA) {
#pragma unroll
  for (int rs = 0; rs < 2; ++rs)
#pragma unroll
    for (int cs = 0; cs < 8; ++cs) s[acc_row(rs) * lds + acc_col(cs)] = acc[TileMMA<T>::idx(rs, cs)];
}

// ---------------------------------------------------------------- F(k)
// The factorisation's critical path runs through the diagonal tiles: their
// 64 pivots are one dependent chain.  What a column costs is latency, not
// work (a 64 x 64 tile is 0.09 MFLOP), so everything here is arranged around
// the chain.  The tile is factored as LDL^T (one reciprocal per column; the
// square roots are taken off the chain) in FP64 on 8 x 8 blocks, which live in
// registers as MMA accumulator fragments, lane (g, t) = (lane / 4, lane % 4)
// holding the pair (row g, columns 2t and 2t + 1): with the K slots of the FP64
// m8n8k4 product chosen as columns 2t, 2t + 1 such a fragment is at once an A
// operand and (transposed) a B operand.  One warp takes the whole pivot chain
// from block to block: pivot block -> its factor and the inverse U of its unit
// triangle -> the next block row's X = S U^T (two MMAs) -> the next pivot block
// D - X M^T (two MMAs).  Everything else is done by the other warps while the
// next block is factored.
// Measured (order 1000, one B200 at 1965 MHz): F(k) 5.0 us, of which 3.4 the
// chain warp on its own (420 ns a block: 190 ns its eight reciprocal steps, the rest the
// hand-over of D, U and X through shared memory and registers), against 7.7 us
// (FP64) and 7.0 (FP32) with rows in lanes and one barrier of five warps per
// block; a chain step, F to F, 9.7 us against 13.5 and 12.2.  An FP32 variant
// would save reciprocal latency but pay for its products on the FMA pipe, so
// FP32 matrices are factored in FP64 too and rounded once on store.

// Rows of a staged 64 x 64 tile in the chain's and the solves' shared memory:
// 16-byte fragment loads of two FP64 rows fall on different banks.
template <typename T> struct ChainLd;
template <> struct ChainLd<double> { static constexpr int LT = NB + 8; };
template <> struct ChainLd<float> { static constexpr int LT = NB + 4; };

// 1 / d and 1 / sqrt(d) of a pivot: the PTX approximations refined to full
// precision -- the reciprocal by one third-order step
// y <- y + y g, g = e + e^2, e = 1 - d y (from ~2^-20 to ~2^-60; y and g are kept
// apart, see factor_chain), the square root by
// two Newton-Raphson steps y <- y + y (1 - d y^2) / 2.  d <= 0, NaN and d outside
// MIN_PIVOT .. MAX_PIVOT give values that factor_finish reports.
__device__ __forceinline__ void pivot_rcp(double d, double& y, double& g) {
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
  const double e = fma(-d, y, 1.0);
  g = fma(e, e, e);
}
__device__ __forceinline__ double pivot_rsqrt(double x) {
  double y;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  y = fma(0.5 * y, fma(-x * y, y, 1.0), y);
  return fma(0.5 * y, fma(-x * y, y, 1.0), y);
}

// Named barriers (0 is __syncthreads); __syncwarp first reconverges a warp
// after divergent code (the barrier instructions are warp-aligned).  bar_arrive
// does not wait; both order the calling warp's earlier shared-memory accesses
// before the barrier completes.
__device__ __forceinline__ void bar_wait(int id, int count) {
  __syncwarp();
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int count) {
  __syncwarp();
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(count) : "memory");
}

__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}
// d += A B^T and d -= A B^T for 8 x 8 fragments, two MMAs on separate accumulators
__device__ __forceinline__ void block_mul(double (&d)[2], const double (&a)[2], const double (&b)[2]) {
  double e[2] = {0.0, 0.0};
  dmma(e, a[1], b[1]);
  dmma(d, a[0], b[0]);
  d[0] += e[0];
  d[1] += e[1];
}
__device__ __forceinline__ void block_sub(double (&d)[2], const double (&a)[2], const double (&b)[2]) {
  const double n[2] = {-a[0], -a[1]};
  block_mul(d, n, b);
}
__device__ __forceinline__ void load_pair(const double* p, double (&d)[2]) {
  const double2 v = *reinterpret_cast<const double2*>(p);
  d[0] = v.x;
  d[1] = v.y;
}
__device__ __forceinline__ void load_pair(const float* p, float (&d)[2]) {
  const float2 v = *reinterpret_cast<const float2*>(p);
  d[0] = v.x;
  d[1] = v.y;
}
__device__ __forceinline__ void store_pair(double* p, double x, double y) {
  *reinterpret_cast<double2*>(p) = make_double2(x, y);
}
__device__ __forceinline__ void store_pair(float* p, float x, float y) {
  *reinterpret_cast<float2*>(p) = make_float2(x, y);
}

// Shared memory of a factorisation besides the tile and the solve blocks, in
// doubles: a panel's multiplier blocks twice, the inverses and pivots of eight
// panels, one word (the first non-positive pivot).
constexpr int RELEASE_WARP = 7;
constexpr int FETCH_WARP = 4;  // on the chain's SM quarter: takes no part in F(k)
constexpr int FRAG_LD = 10;  // rows of an 8 x 8 block read by rows and by columns
constexpr int FACTOR_SCRATCH = 2 * 8 * 64 + 8 * 8 * FRAG_LD + 16 * FRAG_LD + 2 * NB + 2;

// Its parts as shared-memory addresses (a pointer's state space would be lost in
// the struct, and generic accesses cost the chain half as much again).
struct FactorMem {
  uint32_t A;    // [64][LT] the tile, then x = L sqrt(d) column by column
  uint32_t V;    // [64][LT] its solve blocks
  uint32_t M;    // [2][8 block rows][64] a panel's multipliers x / d, fragment order
  uint32_t U;    // [8 panels][8][FRAG_LD] inverse of a pivot block's unit triangle, by columns
  uint32_t D;    // [16][FRAG_LD] the chain's pivot block and the identity
  uint32_t d;    // [64] pivots
  uint32_t r;    // [64] 1 / d
  int* bad;      // the first non-positive pivot (64: none)
  __device__ FactorMem(const double* tile_, const double* blocks, double* scratch)
      : A(tc::smem_u32(tile_)), V(tc::smem_u32(blocks)), M(tc::smem_u32(scratch)) {
    U = M + 8 * (2 * 8 * 64);
    D = U + 8 * (8 * 8 * FRAG_LD);
    d = D + 8 * (16 * FRAG_LD);
    r = d + 8 * NB;
    bad = reinterpret_cast<int*>(scratch + FACTOR_SCRATCH - 2);
  }
};
// A pair (16 bytes, aligned) and one double at element `i` of an array there.
__device__ __forceinline__ void lds_pair(uint32_t base, int i, double (&v)[2]) {
  asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v[0]), "=d"(v[1]) : "r"(base + 8 * i));
}
__device__ __forceinline__ double lds_one(uint32_t base, int i) {
  double v;
  asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(base + 8 * i));
  return v;
}
__device__ __forceinline__ void sts_pair(uint32_t base, int i, double x, double y) {
  asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(base + 8 * i), "d"(x), "d"(y) : "memory");
}

// Roles of the warps (FETCH_WARP takes no part; it shares the SM quarter with the
// chain, which any other role there slows by a fifth).  Panel p = columns 8p .. 8p + 7,
// block (r, c) = rows 8r .., columns 8c ...
//  - Warp 0, the chain: the pivot blocks and X of the block row below.
//  - Warp 3, the lead: block row p + 2, whose blocks (p + 2, p + 1) and
//    (p + 2, p + 2) the chain needs a panel later.
//  - Warps 1, 2, 5, 6: X of the other block rows and the update of the
//    trailing blocks with it.
//  - Warp 7: what leaves the tile, behind the others.
// Named barriers: 1 panel p is stored (the chain arrives and goes on), 3 the
// chain's next blocks (the lead arrives), 4 all X of the panel (the lead arrives).
// A barrier cannot be entered twice by one side before the other has left it, and
// the two halves of M cannot be overtaken: the chain stores panel p after barrier
// 3 of panel p - 1, which the lead reaches after barrier 1 of panel p - 1, that is
// when all helpers have done panel p - 2.  U, d, r and X keep a place per panel, so warp 7
// follows the count f.bad[1] of panels (panel p stored, and all of panel p - 1)
// at its own pace.  The count is published as a maximum: the lead stores its last one
// (6) after the barrier 3 that lets the chain go on to 7 and 8, in either order.
__device__ __forceinline__ void panels_done(const FactorMem& f, int n) {
  asm volatile("red.release.cta.shared::cta.max.s32 [%0], %1;" ::"r"(tc::smem_u32(f.bad) + 4), "r"(n) : "memory");
}

// The inverse of pivot block p's unit triangle as a fragment.
__device__ __forceinline__ void load_inverse(const FactorMem& f, int p, double (&u)[2]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  u[0] = lds_one(f.U, (8 * p + 2 * t) * FRAG_LD + g);
  u[1] = lds_one(f.U, (8 * p + 2 * t + 1) * FRAG_LD + g);
}

// Block (q, q) of the tile from its lower triangle.
__device__ __forceinline__ void load_symmetric(uint32_t A, int q, double (&v)[2]) {
  constexpr int LT = ChainLd<double>::LT;
  const int lane = threadIdx.x & 31, g = lane >> 2, c = 2 * (lane & 3);
  v[0] = lds_one(A, (8 * q + max(g, c)) * LT + 8 * q + min(g, c));
  v[1] = lds_one(A, (8 * q + max(g, c + 1)) * LT + 8 * q + min(g, c + 1));
}

// The chain.  Every lane factors the pivot block in its own registers (l, lower):
// reciprocal -> multiply-add per column, without a hand-over.  In the same
// instruction stream lanes 0 .. 7 eliminate the block's rows (x = L sqrt(d)) and
// lanes 8 .. 15 the rows of the identity, which become the columns of U = inv(unit
// triangle).
__device__ __forceinline__ void factor_chain(const FactorMem& f) {
  constexpr int LT = ChainLd<double>::LT;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  double a[2], s[2] = {0, 0}, next[2] = {0, 0};
  load_symmetric(f.A, 0, a);
  sts_pair(f.D, (8 + g) * FRAG_LD + 2 * t, g == 2 * t ? 1.0 : 0.0, g == 2 * t + 1 ? 1.0 : 0.0);
#pragma unroll 1
  for (int p = 0; p < 8; ++p) {
    sts_pair(f.D, g * FRAG_LD + 2 * t, a[0], a[1]);
    const double d0 = __shfl_sync(0xffffffffu, a[0], 0);
    __syncwarp();
    double l[8][8], x[8], d[8], r[8];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
      for (int c = 0; c <= i; c += 2) {
        double v[2];
        lds_pair(f.D, i * FRAG_LD + c, v);
        l[i][c] = v[0];
        l[i][c + 1] = v[1];
      }
#pragma unroll
    for (int c = 0; c < 8; c += 2) {
      double v[2];
      lds_pair(f.D, (lane & 15) * FRAG_LD + c, v);
      x[c] = v[0];
      x[c + 1] = v[1];
    }
    // lanes 16 .. 31 repeat lanes 0 .. 15, stores included: nothing here branches
    const uint32_t row =
        lane & 8 ? f.U + 8 * ((8 * p + (lane & 7)) * FRAG_LD) : f.A + 8 * ((8 * p + (lane & 7)) * LT + 8 * p);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      d[j] = j == 0 ? d0 : l[j][j];
      double y, gy, m = 0.0;
      pivot_rcp(d[j], y, gy);
      r[j] = fma(y, gy, y);
      if (j < 7) {
        // the next pivot less l (l / d), with l / d refined beside 1 / d: l^2 would
        // leave the FP64 range for matrices of 1e-154 or 1e154, at no gain
        const double u = l[j + 1][j] * y;
        m = fma(u, gy, u);
        l[j + 1][j + 1] = fma(-l[j + 1][j], m, l[j + 1][j + 1]);
      }
#pragma unroll
      for (int c = j + 1; c < 8; ++c) {
        const double e = c == j + 1 ? m : l[c][j] * r[j];
        x[c] = fma(-x[j], e, x[c]);
#pragma unroll
        for (int i = c; i < 8; ++i)
          if (i != j + 1) l[i][c] = fma(-l[i][j], e, l[i][c]);
      }
      if ((j & 1) == 0) sts_pair(row, j, x[j], x[j + 1]);  // final
      if (j == 4 && p < 7) {
        if (p > 0) bar_wait(3, 64);
        lds_pair(f.A, (8 * (p + 1) + g) * LT + 8 * p + 2 * t, s);
        load_symmetric(f.A, p + 1, next);
      }
    }
    __syncwarp();
    if (p < 7) {
      double u[2], rp[2], y[2] = {0, 0}, m[2];
      load_inverse(f, p, u);
#pragma unroll
      for (int c = 0; c < 8; c += 2) sts_pair(f.r, 8 * p + c, r[c], r[c + 1]);
      __syncwarp();
      lds_pair(f.r, 8 * p + 2 * t, rp);
      block_mul(y, s, u);
      m[0] = y[0] * rp[0];
      m[1] = y[1] * rp[1];
      a[0] = next[0];
      a[1] = next[1];
      block_sub(a, y, m);
      sts_pair(f.A, (8 * (p + 1) + g) * LT + 8 * p + 2 * t, y[0], y[1]);
      sts_pair(f.M, ((p & 1) * 8 + p + 1) * 64 + 2 * lane, m[0], m[1]);
    }
#pragma unroll
    for (int c = 0; c < 8; c += 2) sts_pair(f.d, 8 * p + c, d[c], d[c + 1]);
    if (p < 6) {
      bar_arrive(1, 192);
    } else {
      __syncwarp();
      if (lane == 0) panels_done(f, p + 1);
    }
  }
}

// The first helper: block row p + 2 and its blocks that the chain waits for.
__device__ __forceinline__ void factor_lead(const FactorMem& f) {
  constexpr int LT = ChainLd<double>::LT;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll 1
  for (int p = 0; p < 6; ++p) {
    const int at = (8 * (p + 2) + g) * LT + 8 * p + 2 * t;
    const uint32_t M = f.M + 8 * (((p & 1) * 8 + p) * 64 + 2 * lane);
    double u[2], r[2], s[2], b[2], c0[2], c1[2], x[2] = {0, 0}, m[2];
    bar_wait(1, 192);
    lds_pair(f.A, at, s);
    load_inverse(f, p, u);
    lds_pair(f.r, 8 * p + 2 * t, r);
    lds_pair(M, 64, b);
    lds_pair(f.A, at + 8, c0);
    lds_pair(f.A, at + 16, c1);
    block_mul(x, s, u);
    m[0] = x[0] * r[0];
    m[1] = x[1] * r[1];
    block_sub(c0, x, b);
    block_sub(c1, x, m);
    sts_pair(f.A, at + 8, c0[0], c0[1]);
    sts_pair(f.A, at + 16, c1[0], c1[1]);
    sts_pair(f.A, at, x[0], x[1]);
    sts_pair(M, 2 * 64, m[0], m[1]);
    bar_arrive(3, 64);
    if (p < 5) bar_arrive(4, 160);
    if (lane == 0) panels_done(f, p + 1);
  }
}

// The other helpers (h = 1 .. 4): block rows p + 7, 6, 3 and 4, 5.  One copy of each
// loop body: the code of the warps that run at once has to stay in the
// instruction cache (a chain step loses a third with four streams of 16 KB).
__device__ __forceinline__ void factor_help(const FactorMem& f, int h) {
  constexpr int LT = ChainLd<double>::LT;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int k1 = h == 1 ? 7 : h == 2 ? 6 : h == 3 ? 4 : 5, k0 = h == 3 ? 3 : k1;
#pragma unroll 1
  for (int p = 0; p < 6; ++p) {
    const uint32_t M = f.M + 8 * ((p & 1) * 8 * 64 + 2 * lane);
    const int last = min(p + k1, 7);
    bar_wait(1, 192);
    if (p == 5) break;
    double u[2], r[2];
    load_inverse(f, p, u);
    lds_pair(f.r, 8 * p + 2 * t, r);
    // X of the block rows, with the multipliers
#pragma unroll 1
    for (int row = p + k0; row <= last; ++row) {
      const int at = (8 * row + g) * LT + 8 * p + 2 * t;
      double s[2], x[2] = {0, 0};
      lds_pair(f.A, at, s);
      block_mul(x, s, u);
      sts_pair(f.A, at, x[0], x[1]);
      sts_pair(M, row * 64, x[0] * r[0], x[1] * r[1]);
    }
    bar_wait(4, 160);
    // blocks (row, p + 1 .. row) less X M^T, four at a time (past the end the last
    // one again, without a branch)
#pragma unroll 1
    for (int row = p + k0; row <= last; ++row) {
      const int base = (8 * row + g) * LT + 2 * t;
      double x[2];
      lds_pair(f.A, base + 8 * p, x);
#pragma unroll 1
      for (int col = p + 1; col <= row; col += 4) {
        double c[4][2], b[4][2];
        int at[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int q = min(col + i, row);
          at[i] = base + 8 * q;
          lds_pair(M, q * 64, b[i]);
          lds_pair(f.A, at[i], c[i]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) block_sub(c[i], x, b[i]);
#pragma unroll
        for (int i = 0; i < 4; ++i) sts_pair(f.A, at[i], c[i][0], c[i][1]);
      }
    }
  }
}

// Warp 7: the zeros above the block diagonal, then panel by panel the pivots'
// square roots, the first non-positive pivot, V_pp = inv(L_pp) = diag(1 / sqrt(d)) U
// and L_pp, and, a panel later, the block column below L_pp, to the factor and to
// the solve blocks.
template <typename S>
__device__ __forceinline__ void factor_finish(const DFArgs& a, int k, const FactorMem& f, S* V_out) {
  S* out = tile<S>(a, k, k);
  const int ld = a.ld;
  const double min_pivot = a.min_pivot;
  constexpr int LT = ChainLd<double>::LT;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  S* o = out + (size_t)g * ld + 2 * t;
#pragma unroll 1
  for (int p = 1; p < 8; ++p)
#pragma unroll 1
    for (int i = 0; i < p; ++i) store_pair(o + (size_t)8 * i * ld + 8 * p, S(0), S(0));
  double q0 = 0, q1 = 0;  // 1 / sqrt(d) of the previous panel's columns 2t, 2t + 1
#pragma unroll 1
  for (int p = 0; p < 8; ++p) {
    // bounded and reported like every wait, but not by the caller's limit: it depends
    // on no other CTA, and the panels take what they take.  The warp decides as one inside
    // the loop (__syncwarp hands on what the deciding lane acquired): with a vote after it
    // the factor of order 1008 took 179.5 us, 172 so.
    for (long long it = 0;; ++it) {
      int done;
      asm volatile("ld.acquire.cta.shared.b32 %0, [%1];" : "=r"(done) : "r"(tc::smem_u32(f.bad) + 4) : "memory");
      if (__any_sync(0xffffffffu, done > p)) break;
      if (it >= SPIN_LIMIT) {
        if (lane == 0) wait_expired(a);
        return;
      }
    }
    __syncwarp();
    const int c = 8 * p + 2 * t;
    const double d = lds_one(f.d, 8 * p + g);
    double u[2], x[2];
    load_inverse(f, p, u);
    lds_pair(f.A, (8 * p + g) * LT + c, x);
    // the column of the panel before
#pragma unroll 1
    for (int i = p > 0 ? p : 8; i < 8; i += 2) {
      double y[2], z[2];
      const int r0 = 8 * i + g, r1 = 8 * min(i + 1, 7) + g;
      lds_pair(f.A, r0 * LT + c - 8, y);
      lds_pair(f.A, r1 * LT + c - 8, z);
      y[0] *= q0;
      y[1] *= q1;
      z[0] *= q0;
      z[1] *= q1;
      sts_pair(f.V, r0 * LT + c - 8, y[0], y[1]);
      sts_pair(f.V, r1 * LT + c - 8, z[0], z[1]);
      store_pair(out + (size_t)r0 * ld + c - 8, (S)y[0], (S)y[1]);
      store_pair(out + (size_t)r1 * ld + c - 8, (S)z[0], (S)z[1]);
      if (V_out) {
        store_pair(V_out + r0 * NB + c - 8, (S)y[0], (S)y[1]);
        store_pair(V_out + r1 * NB + c - 8, (S)z[0], (S)z[1]);
      }
    }
    const unsigned bad = __ballot_sync(0xffffffffu, !(d >= min_pivot && d <= MAX_PIVOT));
    const double rg = pivot_rsqrt(d);
    q0 = __shfl_sync(0xffffffffu, rg, 8 * t);
    q1 = __shfl_sync(0xffffffffu, rg, 8 * t + 4);
    sts_pair(f.V, (8 * p + g) * LT + c, rg * u[0], rg * u[1]);
    if (V_out) store_pair(V_out + (8 * p + g) * NB + c, (S)(rg * u[0]), (S)(rg * u[1]));
    store_pair(o + (size_t)8 * p * ld + 8 * p, (S)(2 * t <= g ? x[0] * q0 : 0.0), (S)(2 * t + 1 <= g ? x[1] * q1 : 0.0));
    if (lane == 0 && bad) *f.bad = min(*f.bad, 8 * p + ((__ffs(bad) - 1) >> 2));
  }
}

// F(k) of the updated tile f.A (its lower triangle) by all warps but FETCH_WARP
// (which returns at once): L_kk to tile (k, k) of the factor (type S, zero above the diagonal),
// the solve blocks of L_kk to f.V and to V_out (global 64 x 64, type S, or
// null): with 8 x 8 blocks, V_jj = inv(L_jj) on the block diagonal and L_jq
// below it.  (Blocks above the block diagonal are neither written nor read.)
// A non-positive pivot is recorded in info.  f.bad: {64, 0} on entry; on
// return, after the caller's next CTA barrier, {64, 8}.  Ends with a barrier of the
// seven warps (named barrier 2).
template <typename S>
__device__ __forceinline__ void factor_tile(const DFArgs& a, int k, const FactorMem& f, S* V_out) {
  const int warp = threadIdx.x >> 5;
  if (warp == FETCH_WARP) return;
  if (warp == 0) factor_chain(f);
  else if (warp == 7) factor_finish<S>(a, k, f, V_out);
  else if (warp == 3) factor_lead(f);
  else factor_help(f, warp < 3 ? warp : warp - 2);
  bar_wait(2, 32 * 7);
  if (threadIdx.x == 0) {
    if (f.bad[0] < NB && k * NB + f.bad[0] < a.n) atomicCAS(a.info, 0, k * NB + f.bad[0] + 1);
    f.bad[0] = NB;
  }
}

// ---------------------------------------------------------------- S(i, k)
// W = C L_kk^-T for a 64 x 64 tile C (smem rows of ldc) with the solve blocks
// of L_kk (smem [64][LT], factor_tile), W_j = (C_j - sum_{q < j} W_q L_jq^T) V_jj^T
// block column by block column.  A warp keeps its rows' accumulators in
// registers; with the K slots chosen as columns 2t, 2t + 1 an accumulator
// fragment is at once the next products' A fragment, so the chain over
// the eight block columns is two MMAs and two adds per column, without shuffles
// or shared memory.  out(row, col, w0, w1) receives the pairs of W
// (columns col, col + 1).  G groups of eight rows per warp, so warps 0 .. 8 / G - 1;
// a warp's rows of C are read before its first out(), which may therefore
// overwrite them.
// Against the product with the explicit inverse: half the operations and no
// inversion before it.  FP64: DMMA, eight rows per warp (bound by the FP64
// tensor pipe: 576 DMMAs, 2.4k cycles, with one warp of sixteen rows per SM quarter as
// with two of eight).
template <int G, typename S, typename F>
__device__ __forceinline__ void solve_rows(const S* C, int ldc, const double* V, F out) {
  constexpr int LT = ChainLd<double>::LT;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, r0 = 8 * G * warp + g;
  double p[G][8][2], q[G][8][2], v[8][2];
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int i = 0; i < G; ++i) {
      S c[2];
      load_pair(C + (r0 + 8 * i) * ldc + 8 * j + 2 * t, c);
      p[i][j][0] = c[0];
      p[i][j][1] = c[1];
      q[i][j][0] = q[i][j][1] = 0.0;
    }
  __syncwarp();
  auto load_column = [&](int j) {  // V_jj, L_ij
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (i >= j) load_pair(V + (8 * i + g) * LT + 8 * j + 2 * t, v[i]);
  };
  load_column(0);
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    double w[G][2];
#pragma unroll
    for (int i = 0; i < G; ++i) {
      double d[2] = {0.0, 0.0}, e[2] = {0.0, 0.0};
      dmma(d, p[i][j][0] + q[i][j][0], v[j][0]);
      dmma(e, p[i][j][1] + q[i][j][1], v[j][1]);
      w[i][0] = d[0] + e[0];
      w[i][1] = d[1] + e[1];
    }
#pragma unroll
    for (int k = j + 1; k < 8; ++k)
#pragma unroll
      for (int i = 0; i < G; ++i) {
        dmma(p[i][k], -w[i][0], v[k][0]);
        dmma(q[i][k], -w[i][1], v[k][1]);
      }
    load_column(j + 1);  // ahead of this column's stores
#pragma unroll
    for (int i = 0; i < G; ++i) out(r0 + 8 * i, 8 * j + 2 * t, w[i][0], w[i][1]);
  }
}

// D (16 x 8) += A (16 x 8) B (8 x 8) in TF32; a = {(g, k0), (g + 8, k0),
// (g, k1), (g + 8, k1)}, b = {k0, k1} of column g, k0 / k1 the lane's K slots.
__device__ __forceinline__ void tf32_mma(float (&c)[4], const unsigned (&a)[4], const unsigned (&b)[2]) {
  asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// FP32: 3xTF32 m16n8k8, sixteen rows per warp (warps 0 .. 3), the hi * hi
// products and the two cross terms on separate accumulators.
template <typename F>
__device__ __forceinline__ void solve_rows_f32(const float* C, int ldc, const float* V, int warp, F out) {
  constexpr int LT = ChainLd<float>::LT;
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3, r0 = 16 * warp + g;
  float p[8][4], q[8][4];
  auto mul = [&](float (&p)[4], float (&q)[4], const unsigned (&ah)[4], const unsigned (&al)[4], const float* vb) {
    unsigned bh[2], bl[2];
    float v[2];
    load_pair(vb + g * LT + 2 * t, v);
#pragma unroll
    for (int e = 0; e < 2; ++e) split_tf32(v[e], bh[e], bl[e]);
    tf32_mma(p, ah, bh);
    tf32_mma(q, al, bh);
    tf32_mma(q, ah, bl);
  };
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    float c[2], e[2];
    load_pair(C + r0 * ldc + 8 * j + 2 * t, c);
    load_pair(C + (r0 + 8) * ldc + 8 * j + 2 * t, e);
    p[j][0] = c[0];
    p[j][1] = c[1];
    p[j][2] = e[0];
    p[j][3] = e[1];
#pragma unroll
    for (int u = 0; u < 4; ++u) q[j][u] = 0.0f;
  }
  __syncwarp();
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    // fragment order: (g, 2t), (g + 8, 2t), (g, 2t + 1), (g + 8, 2t + 1)
    constexpr int at[4] = {0, 2, 1, 3};
    unsigned ah[4], al[4];
    float w[4], d[4] = {0.0f, 0.0f, 0.0f, 0.0f}, e[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int u = 0; u < 4; ++u) tc::split_tf32_any(p[j][at[u]] + q[j][at[u]], ah[u], al[u]);
    mul(d, e, ah, al, V + 8 * j * LT + 8 * j);
#pragma unroll
    for (int u = 0; u < 4; ++u) w[u] = d[u] + e[u];
#pragma unroll
    for (int u = 0; u < 4; ++u) split_tf32(-w[at[u]], ah[u], al[u]);
#pragma unroll
    for (int i = j + 1; i < 8; ++i) mul(p[i], q[i], ah, al, V + 8 * i * LT + 8 * j);
    out(r0, 8 * j + 2 * t, w[0], w[1]);
    out(r0 + 8, 8 * j + 2 * t, w[2], w[3]);
  }
}

// 32 rows (rows of LDA) by the first four warps.
template <typename T, typename F>
__device__ __forceinline__ void solve_half(const T* C, const T* V, F out) {
  if constexpr (sizeof(T) == 8) solve_rows<1>(C, LDA, V, out);
  else if (threadIdx.x < 64) solve_rows_f32(C, LDA, V, threadIdx.x >> 5, out);
}
template <typename T, typename F>
__device__ __forceinline__ void solve_rows_t(const T* C, int ldc, const T* V, F out) {
  if constexpr (sizeof(T) == 8) solve_rows<1>(C, ldc, V, out);
  else if (threadIdx.x < 128) solve_rows_f32(C, ldc, V, threadIdx.x >> 5, out);
}

// ---------------------------------------------------------------- the chain's SYRK
// A = N - L L^T on and below the block diagonal (A, L: smem rows of
// ChainLd<double>::LT): the last update of the next diagonal tile, with the
// solve's result still in shared memory.  N (its rows of ChainLd<S>::LT) is not
// read before ready() returns, so that its way here overlaps with the products.
// The 36 lower 8 x 8 blocks, nine on each of warps 0 .. 3: rows 7 - w and w of
// blocks (bound by the FP64 tensor pipe, 2.4k cycles).
template <typename S, typename R>
__device__ __forceinline__ void syrk_lower(const S* N, const double* L, double* A, R ready) {
  constexpr int LT = ChainLd<double>::LT, LS = ChainLd<S>::LT;
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  int bi[9], bj[9];
  double d[9][2], e[9][2];
#pragma unroll
  for (int b = 0; b < 9; ++b) {
    const bool low = b < 8 - w;
    bi[b] = 8 * (low ? 7 - w : w);
    bj[b] = 8 * (low ? b : b - (8 - w));
    d[b][0] = d[b][1] = e[b][0] = e[b][1] = 0.0;
  }
#pragma unroll 1
  for (int k = 0; k < NB; k += 8)
#pragma unroll
    for (int b = 0; b < 9; ++b) {
      double x[2], y[2];
      load_pair(L + (bi[b] + g) * LT + k + 2 * t, x);
      load_pair(L + (bj[b] + g) * LT + k + 2 * t, y);
      dmma(d[b], x[0], y[0]);
      dmma(e[b], x[1], y[1]);
    }
  ready();
#pragma unroll
  for (int b = 0; b < 9; ++b) {
    S v[2];
    load_pair(N + (bi[b] + g) * LS + bj[b] + 2 * t, v);
    store_pair(A + (bi[b] + g) * LT + bj[b] + 2 * t, (double)v[0] - (d[b][0] + e[b][0]), (double)v[1] - (d[b][1] + e[b][1]));
  }
}

// ---------------------------------------------------------------- the chain CTA
// Shared memory of the chain CTA: three FP64 tiles (the diagonal tile, the
// solve's result, the solve blocks), two of the matrix's type (the solve's
// input, the next diagonal tile), and the factor scratch.
template <typename S>
constexpr size_t chain_smem_bytes() {
  return sizeof(double) * (3 * NB * ChainLd<double>::LT + FACTOR_SCRATCH) + 2 * sizeof(S) * NB * ChainLd<S>::LT;
}

// One warp's asynchronous copy of a 64 x 64 tile into smem rows of LT (the
// warp waits with cp_async_wait_all).
template <typename S>
__device__ __forceinline__ void fetch_tile_warp(const S* g, int ld, S* s) {
  constexpr int LT = ChainLd<S>::LT, per_row = NB * (int)sizeof(S) / 16, elems = 16 / (int)sizeof(S);
#pragma unroll 8
  for (int c = threadIdx.x & 31; c < NB * per_row; c += 32)
    cp_async16(s + (c / per_row) * LT + (c % per_row) * elems, g + (size_t)(c / per_row) * ld + (c % per_row) * elems);
}

// A single warp's bounded wait for *flag >= target (the abort polling and the
// expiry of wait_all) while the other warps of the CTA compute: lane 0 polls
// with relaxed loads and sleeps in between, because an acquire load per poll
// invalidates the SM's L1 each time and slowed the other warps' shared-memory
// accesses several times over.  The flag is then acquired once by every lane,
// which orders the lane's own later copies.
__device__ __forceinline__ int ld_relaxed(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ bool warp_wait_geq(const DFArgs& a, const int* flag, int target) {
  int ok = 1;
  if ((threadIdx.x & 31) == 0) {
    for (long long it = 0; ld_relaxed(flag) < target; ++it) {
      if ((it & 15) == 15 && ld_relaxed(a.ctl + 1)) {
        ok = 0;
        break;
      }
      if (it + 1 > a.spin_limit) {
        wait_expired(a);
        ok = 0;
        break;
      }
      __nanosleep(it > 256 ? 200 : 40);
    }
  }
  ok = __shfl_sync(0xffffffffu, ok, 0);
  return ok && __all_sync(0xffffffffu, ld_acquire(flag) >= target);
}

// The chain CTA: F(0), S(1, 0), F(1), S(2, 1), ... in FP64 on a matrix of
// type S.  For each k: F(k) on seven warps (L_kk to the factor, the solve
// blocks to a.lp for the workers' solves of column k, fin(k, k) = 1), while
// FETCH_WARP copies the solve's input A(k+1, k) as soon as its last update is
// in; S(k+1, k) on warps 0 .. 3 (one per SM quarter fills its FP64 tensor pipe),
// kept in shared memory and published as fin(k+1, k) = 1; the last update of
// A(k+1, k+1) from the result (syrk_lower, the same warps), whose tile FETCH_WARP
// copies meanwhile.  The flags are published by RELEASE_WARP, which has nothing else to
// do then: a release costs its warp 0.7 us.
template <typename S>
__device__ void run_chain(const DFArgs& a, unsigned char* smem, int* s_ok) {
  constexpr int LT = ChainLd<double>::LT, LS = ChainLd<S>::LT;
  double* A = reinterpret_cast<double*>(smem);
  double* L = A + NB * LT;
  double* V = L + NB * LT;
  const FactorMem f(A, V, V + NB * LT);
  S* C = reinterpret_cast<S*>(V + NB * LT + FACTOR_SCRATCH);
  S* N = C + NB * LS;
  const int nt = a.nt, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    *s_ok = 1;
    f.bad[0] = NB;
    f.bad[1] = 0;
  }
  for (int e = threadIdx.x; e < NB * NB; e += THREADS)
    A[(e >> 6) * LT + (e & 63)] = (double)ldcg(tile<S>(a, 0, 0) + (size_t)(e >> 6) * a.ld + (e & 63));
  __syncthreads();
  for (int k = 0; k < nt; ++k) {
    TRACE(0, a.ntasks + 2 * k);
    TRACE(3, a.ntasks + 2 * k);
    TRACE(1, a.ntasks + 2 * k);
    const int* next = a.upd + (k + 1) * nt + k + 1;
    if (warp != FETCH_WARP) {
      CTRACE(k, 0);
      factor_tile<S>(a, k, f, a.lp ? reinterpret_cast<S*>(a.lp) + (size_t)k * NB * NB : nullptr);
    } else if (k + 1 < nt) {
      const bool ok = warp_wait_geq(a, a.upd + (k + 1) * nt + k, k);
      if (ok) {
        fetch_tile_warp(tile<S>(a, k + 1, k), a.ld, C);
        cp_async_wait_all();
      } else if (lane == 0) {
        *s_ok = 0;
      }
    }
    TRACE(2, a.ntasks + 2 * k);
    CTRACE(k, 1);
    __syncthreads();
    if (threadIdx.x == 32 * RELEASE_WARP) st_release(a.fin + k * nt + k, 1);
    if (!*s_ok || k + 1 == nt) return;
    TRACE(0, a.ntasks + 2 * k + 1);
    TRACE(3, a.ntasks + 2 * k + 1);
    TRACE(1, a.ntasks + 2 * k + 1);
    CTRACE(k, 2);
    if (warp < 4) {
      S* out = tile<S>(a, k + 1, k);
      solve_rows<2>(C, LS, V, [&](int r, int c, double w0, double w1) {
        store_pair(L + r * LT + c, w0, w1);
        store_pair(out + (size_t)r * a.ld + c, (S)w0, (S)w1);
      });
      CTRACE(k, 3);
      bar_wait(5, 160);
      CTRACE(k, 4);
      TRACE(2, a.ntasks + 2 * k + 1);
      syrk_lower(N, L, A, [] { bar_wait(6, 160); });
    } else if (warp == RELEASE_WARP) {
      bar_wait(5, 160);
      if (lane == 0) st_release(a.fin + (k + 1) * nt + k, 1);
    } else if (warp == FETCH_WARP) {
      if (lane == 0) f.bad[1] = 0;
      if (warp_wait_geq(a, next, k)) {
        fetch_tile_warp(tile<S>(a, k + 1, k + 1), a.ld, N);
        cp_async_wait_all();
      } else if (lane == 0) {
        *s_ok = 0;
      }
      bar_arrive(6, 160);
    }
    __syncthreads();
    CTRACE(k, 5);
    if (!*s_ok) return;
  }
}

// U(i, j, k) with every tile moved by 16-byte copies: the target tile is
// staged into sC with cp.async together with L_ik, L_jk (instead of per-thread
// 4-byte loads), updated in registers, and written back through sC with
// 16-byte stores.  sC: a third [64][LDA] tile.
__device__ __forceinline__ void update_tile(const DFArgs& a, int i, int j, int k, double acc[16], double* sA, double* sB,
                                            double* sC) {
  using T = double;
  stage_async(tile<T>(a, i, k), a.ld, sA, LDA);
  if (i != j) stage_async(tile<T>(a, j, k), a.ld, sB, LDA);
  stage_async(tile<T>(a, i, j), a.ld, sC, LDA);
  cp_async_wait_all();
  __syncthreads();
  smem_to_acc(sC, acc);
  TileMMA<T>::sub(sA, i != j ? sB : sA, acc);
  acc_to_smem(acc, sC);  // each thread rewrites the elements it read
  __syncthreads();
  store_tile(sC, LDA, tile<T>(a, i, j), a.ld);
}

// U(i, j, k) and U(i+1, j, k) together: five tiles (L_ik, L_jk, L_{i+1,k} and
// both targets) staged with 16-byte copies in one round, two accumulators
// against the shared L_jk, one round of 16-byte stores.  s: five [64][LDA]
// FP64 tiles.
__device__ __forceinline__ void update_tile_pair(const DFArgs& a, int i, int j, int k, double acc[16], double* s) {
  using T = double;
  T* sA1 = s;
  T* sB = sA1 + NB * LDA;
  T* sC1 = sB + NB * LDA;
  T* sA2 = sC1 + NB * LDA;
  T* sC2 = sA2 + NB * LDA;
  if (i != j) stage_async(tile<T>(a, i, k), a.ld, sA1, LDA);
  stage_async(tile<T>(a, j, k), a.ld, sB, LDA);
  stage_async(tile<T>(a, i + 1, k), a.ld, sA2, LDA);
  stage_async(tile<T>(a, i, j), a.ld, sC1, LDA);
  stage_async(tile<T>(a, i + 1, j), a.ld, sC2, LDA);
  cp_async_wait_all();
  __syncthreads();
  T acc2[16];
  smem_to_acc(sC1, acc);
  smem_to_acc(sC2, acc2);
  TileMMA<T>::sub(i != j ? sA1 : sB, sB, acc);
  TileMMA<T>::sub(sA2, sB, acc2);
  acc_to_smem(acc, sC1);  // each thread rewrites the elements it read
  acc_to_smem(acc2, sC2);
  __syncthreads();
  store_tile(sC1, LDA, tile<T>(a, i, j), a.ld);
  store_tile(sC2, LDA, tile<T>(a, i + 1, j), a.ld);
}

// ---------------------------------------------------------------- tcgen05 updates
// The FP32 lists' update tasks run on the 5th-generation tensor cores: a task
// U(i .. i+rows-1, j, k) (rows <= 4, sharing L_jk) splits L_jk and the rows'
// L_ik into TF32 hi / lo halves in swizzled shared memory, one thread issues
// P = L_ik L_jk^T as 3xTF32 MMAs (M = 128: two row tiles per MMA, N = 64,
// K = 64) into TMEM accumulators (from zero), and the warps read P back with
// tcgen05.ld and subtract it from C_ij (C -= P once, as the mma.sync
// products do).  Each worker CTA allocates its 128 TMEM columns once.
struct TcWorker {
  uint64_t* mbar;       // MMA completion (one phase per task)
  uint32_t tmem;        // TMEM base: one accumulator of 64 columns per row pair
  uint32_t phase;
  int max_pairs;        // row pairs per task: 2 (single matrix) or 1 (batch)
  unsigned char* base;  // 1024-byte aligned operand area
};
constexpr uint32_t TC_A_BYTES = tc::operand_bytes(128);  // one M = 128 operand half (hi or lo)
constexpr uint32_t TC_B_BYTES = tc::operand_bytes(64);
// A hi, A lo (max_pairs row pairs each), B hi, B lo, and the alignment slack
constexpr size_t tc_worker_smem_bytes(int max_pairs) { return 2 * max_pairs * TC_A_BYTES + 2 * TC_B_BYTES + 1024; }
// TMEM columns: a power of two >= 32
__host__ __device__ constexpr uint32_t tc_cols(int max_pairs) { return max_pairs > 1 ? 128u : 64u; }

__device__ __forceinline__ void tc_worker_begin(uint64_t* mbar, uint32_t* s_tmem, unsigned char* smem, int max_pairs,
                                                TcWorker& w) {
  if (threadIdx.x == 0) tc::mbar_init(mbar, 1);
  if (threadIdx.x < 32) tc::tmem_alloc(s_tmem, tc_cols(max_pairs));
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  w.mbar = mbar;
  w.tmem = *s_tmem;
  w.phase = 0;
  w.max_pairs = max_pairs;
  w.base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem) + 1023) & ~uintptr_t(1023));
}

__device__ __forceinline__ void tc_worker_end(const TcWorker& w) {
  tc::fence_before_sync();
  __syncthreads();
  if (threadIdx.x < 32) tc::tmem_dealloc(w.tmem, tc_cols(w.max_pairs));
}

// U(i + r, j, k) for r < rows (rows <= 2 max_pairs) on the tensor cores (the
// dependencies are met).  Returns false if the MMAs did not complete within
// the spin limit (the run is then aborted like an expired flag wait).
__device__ bool update_rows_tc(const DFArgs& a, int i, int rows, int j, int k, TcWorker& w) {
  unsigned char* Ahi = w.base;
  unsigned char* Alo = Ahi + w.max_pairs * TC_A_BYTES;
  unsigned char* Bhi = Alo + w.max_pairs * TC_A_BYTES;
  unsigned char* Blo = Bhi + TC_B_BYTES;
  const int pairs = (rows + 1) >> 1;
  {
    // L_jk and the rows' L_ik, all loads in flight together
    tc::SplitTile t[5];
    t[0] = tc::SplitTile{tile<float>(a, j, k), 64, 0, Bhi, Blo};
#pragma unroll
    for (int r = 0; r < 4; ++r)
      t[1 + r] = tc::SplitTile{tile<float>(a, i + (r < rows ? r : 0), k), 128, 64 * (r & 1),
                               Ahi + (r >> 1) * TC_A_BYTES, Alo + (r >> 1) * TC_A_BYTES};
    tc::split_tiles_all<THREADS, 5>(t, 1 + rows, a.ld);
  }
  tc::fence_proxy_smem();
  __syncthreads();
  if (threadIdx.x == 0) {
    tc::fence_after_sync();
    for (int p = 0; p < pairs; ++p)
      tc::issue_product(w.tmem + 64 * p, tc::smem_u32(Ahi + p * TC_A_BYTES), tc::smem_u32(Alo + p * TC_A_BYTES),
                        tc::smem_u32(Bhi), tc::smem_u32(Blo));
    tc::mma_commit(w.mbar);
  }
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, q = warp & 3, g = warp >> 2;
  const int m = 32 * q + lane;  // accumulator row = TMEM lane
  const int p = pairs == 2 ? g : 0;
  const int c0 = pairs == 2 ? 0 : 32 * g;
  const int nh = pairs == 2 ? 2 : 1;  // 32-column halves this warp reads
  const int rr = 2 * p + (m >> 6);    // row tile in the group (warp-uniform)
  bool ok = tc::mbar_wait(w.mbar, w.phase, a.spin_limit);
  if (!ok) tc::mbar_wait(w.mbar, w.phase, a.spin_limit);  // the MMAs must not outlive the TMEM
  ok = __syncthreads_and(ok) != 0;                          // one verdict for the whole CTA
  if (!ok && threadIdx.x == 0) {
    atomicExch(a.ctl + 1, 1);
    atomicOr(a.err, PBG_DEV_ERR_BARRIER);
    atomicCAS(a.info, 0, -1);
  }
  w.phase ^= 1;
  tc::fence_after_sync();
  // P from TMEM into shared memory, row-major [rows * 64][LDA] over the A
  // operands (the MMAs that read them are complete) ...
  float* Ps = reinterpret_cast<float*>(w.base);
  if (ok && rr < rows) {
    for (int h = 0; h < nh; ++h) {
      float v[32];
      tc::tmem_ld32(w.tmem + ((uint32_t)(32 * q) << 16) + 64 * p + c0 + 32 * h, v);
      float* dst = Ps + (size_t)(64 * rr + (m & 63)) * LDA + c0 + 32 * h;
#pragma unroll
      for (int u = 0; u < 8; ++u)
        *reinterpret_cast<float4*>(dst + 4 * u) = make_float4(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
    }
  }
  __syncthreads();
  // ... then C -= P with coalesced 16-byte accesses (a row of 64 per 16 threads)
  if (ok)
    for (int e = threadIdx.x; e < rows * NB * 16; e += THREADS) {
      const int row = e >> 4, c4 = e & 15;
      float4* gp = reinterpret_cast<float4*>(tile<float>(a, i + (row >> 6), j) + (size_t)(row & 63) * a.ld) + c4;
      float4 cv = __ldcg(gp);
      const float4 pv = *reinterpret_cast<const float4*>(Ps + (size_t)row * LDA + 4 * c4);
      cv.x -= pv.x;
      cv.y -= pv.y;
      cv.z -= pv.z;
      cv.w -= pv.w;
      *gp = cv;
    }
  tc::fence_before_sync();
  __syncthreads();
  return ok;
}

// ---------------------------------------------------------------- inv(L) in the task list
// With DFArgs::X set, the factorisation's task list also forms X = inv(L)
// (its off-diagonal tiles; the diagonal ones are the inv(L_kk) in invdiag),
// right-looking over the columns of L:
//   X_ij = -X_ii sum_{k=j}^{i-1} L_ik X_kj    (i > j),
// accumulated as V_ij = -sum_k L_ik X_kj in X's own tile (i, j), in k order:
//   XG(i, j, k), j <= k <= i-2: V_ij -= L_ik X_kj for rows i and i+1 (they
//     share X_kj); needs L_ik final, X_kj final and the k - j earlier terms;
//   XZ(i, j): V_ij -= L_{i,i-1} X_{i-1,j}, then X_ij = X_ii V_ij; needs
//     L_{i,i-1}, X_{i-1,j}, inv(L_ii) (fin(i,i) = 2) and the earlier terms.
// xupd(i, j) counts the applied terms, xfin(i, j) = 1 marks X_ij final.  The
// list places XZ(k+1, .) and XG(., ., k) right after panel k's block, after
// every task (or chain step) they depend on.  Tiles written in this kernel
// are read through L2 (.cg loads, cp.async.cg).

template <typename T>
__device__ __forceinline__ const T* xtile(const DFArgs& a, int k, int j) {
  return k == j ? reinterpret_cast<const T*>(a.invdiag) + (size_t)j * NB * NB
                : reinterpret_cast<const T*>(a.X) + (size_t)k * NB * a.ld + (size_t)j * NB;
}
template <typename T>
__device__ __forceinline__ T* xtile_out(const DFArgs& a, int i, int j) {
  return reinterpret_cast<T*>(a.X) + (size_t)i * NB * a.ld + (size_t)j * NB;
}

// s[c][r] = g[r][c] through L2, all of a thread's loads in flight first.
template <typename T>
__device__ __forceinline__ void stage_transposed_cg(const T* g, int ld, T* s) {
  T v[TILE_PER_THREAD];
#pragma unroll
  for (int q = 0; q < TILE_PER_THREAD; ++q) {
    const int e = threadIdx.x + q * THREADS;
    v[q] = ldcg(g + (size_t)(e >> 6) * ld + (e & 63));
  }
#pragma unroll
  for (int q = 0; q < TILE_PER_THREAD; ++q) {
    const int e = threadIdx.x + q * THREADS;
    s[(e & 63) * LDA + (e >> 6)] = v[q];
  }
}

template <typename T>
__device__ __forceinline__ void acc_to_smem_transposed(const T acc[16], T* s) {
#pragma unroll
  for (int rs = 0; rs < 2; ++rs)
#pragma unroll
    for (int cs = 0; cs < 8; ++cs) s[acc_col(cs) * LDA + acc_row(rs)] = acc[TileMMA<T>::idx(rs, cs)];
}

// acc -= A X for the tile X of the inverse at g: staged as it lies (FP64) or
// transposed for the TF32 product's fragments (FP32).  stage_x starts the
// copy (the caller waits with cp_async_wait_all and a barrier).
template <typename T>
__device__ __forceinline__ void stage_x(const T* g, int ld, T* s) {
  if constexpr (sizeof(T) == 8) stage_async(g, ld, s, LDA);
  else stage_transposed_cg<T>(g, ld, s);
}
template <typename T>
__device__ __forceinline__ void sub_x(const T* sA, const T* sX, T acc[16]) {
  if constexpr (sizeof(T) == 8) TileMMA<T>::template sub_rows<false>(sA, sX, acc);
  else TileMMA<T>::sub(sA, sX, acc);
}

// XG(i, j, k) for rows i .. i+rows-1 (rows <= 2).  Shared memory: three tiles.
template <typename T>
__device__ void inverse_update(const DFArgs& a, int i, int rows, int j, int k, T* s) {
  T* sB = s;
  T* sA0 = s + NB * LDA;
  T* sA1 = s + 2 * NB * LDA;
  stage_async(tile<T>(a, i, k), a.ld, sA0, LDA);
  if (rows > 1) stage_async(tile<T>(a, i + 1, k), a.ld, sA1, LDA);
  T acc0[16], acc1[16];
  if (k > j) {
    load_acc(xtile_out<T>(a, i, j), a.ld, acc0);
    if (rows > 1) load_acc(xtile_out<T>(a, i + 1, j), a.ld, acc1);
  } else {
#pragma unroll
    for (int e = 0; e < 16; ++e) acc0[e] = acc1[e] = T(0);
  }
  stage_x<T>(xtile<T>(a, k, j), k == j ? NB : a.ld, sB);
  cp_async_wait_all();
  __syncthreads();
  sub_x<T>(sA0, sB, acc0);
  if (rows > 1) sub_x<T>(sA1, sB, acc1);
  store_acc(xtile_out<T>(a, i, j), a.ld, acc0);
  if (rows > 1) store_acc(xtile_out<T>(a, i + 1, j), a.ld, acc1);
}

// XZ(i, j).  Shared memory: three tiles.
template <typename T>
__device__ void inverse_finish(const DFArgs& a, int i, int j, T* s) {
  T* sB = s;
  T* sA = s + NB * LDA;
  T* sX = s + 2 * NB * LDA;
  stage_async(tile<T>(a, i, i - 1), a.ld, sA, LDA);
  stage_async(reinterpret_cast<const T*>(a.invdiag) + (size_t)i * NB * NB, NB, sX, LDA);  // X_ii
  T acc[16];
  if (i - 1 > j) {
    load_acc(xtile_out<T>(a, i, j), a.ld, acc);
  } else {
#pragma unroll
    for (int e = 0; e < 16; ++e) acc[e] = T(0);
  }
  stage_x<T>(xtile<T>(a, i - 1, j), i - 1 == j ? NB : a.ld, sB);
  cp_async_wait_all();
  __syncthreads();
  sub_x<T>(sA, sB, acc);  // V_ij complete
  __syncthreads();
  if constexpr (sizeof(T) == 8) acc_to_smem(acc, sB);
  else acc_to_smem_transposed(acc, sB);
  __syncthreads();
#pragma unroll
  for (int e = 0; e < 16; ++e) acc[e] = T(0);
  sub_x<T>(sX, sB, acc);  // -X_ii V
#pragma unroll
  for (int e = 0; e < 16; ++e) acc[e] = -acc[e];
  store_acc(xtile_out<T>(a, i, j), a.ld, acc);
}

// acc = A(i, j) with the updates of columns < j (the last one, with column
// j-1, applied here; the smem tiles are free again on return).
template <typename T>
__device__ bool solve_input(const DFArgs& a, int i, int j, T acc[16], T* sA, T* sB, int* s_ok) {
  const int nt = a.nt;
  if (j == 0) {
    load_acc(tile<T>(a, i, 0), a.ld, acc);
    return true;
  }
  const int* fl[3] = {a.fin + i * nt + j - 1, a.fin + j * nt + j - 1, a.upd + i * nt + j};
  const int tg[3] = {1, 1, j - 1};
  if (!wait_all(a, fl, tg, 3, s_ok)) return false;
  load_and_update(a, i, j, j - 1, acc, sA, sB);  // ends with a barrier
  return true;
}

// A B^T of a LEAD task: A 32 rows, B 64 rows (smem rows of LDA), 64 deep.  Warp w
// owns rows 16 (w / 4) .. and columns 16 (w % 4) .. of the 32 x 64 product;
// element 4 mt + 2 nt + h of `d` is row 8 mt + lane / 4, column 8 nt + 2 (lane % 4)
// + h of them (half_at).
__device__ __forceinline__ int half_row(int mt) { return 16 * (threadIdx.x >> 7) + 8 * mt + ((threadIdx.x & 31) >> 2); }
__device__ __forceinline__ int half_col(int nt) { return 16 * ((threadIdx.x >> 5) & 3) + 8 * nt + 2 * (threadIdx.x & 3); }
__device__ __forceinline__ void half_product(const double* sA, const double* sB, double (&d)[8]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const double* A = sA + (16 * (w >> 2) + g) * LDA + t;
  const double* B = sB + (16 * (w & 3) + g) * LDA + t;
  double c[4][2] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}}, e[4][2] = {{0, 0}, {0, 0}, {0, 0}, {0, 0}};
#pragma unroll 4
  for (int k0 = 0; k0 < NB; k0 += 8)
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      dmma(c[q], A[8 * (q >> 1) * LDA + k0], B[8 * (q & 1) * LDA + k0]);
      dmma(e[q], A[8 * (q >> 1) * LDA + k0 + 4], B[8 * (q & 1) * LDA + k0 + 4]);
    }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    d[2 * q] = c[q][0] + e[q][0];
    d[2 * q + 1] = c[q][1] + e[q][1];
  }
}
__device__ __forceinline__ void half_product(const float* sA, const float* sB, float (&d)[8]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, g = lane >> 2, t = lane & 3;
  const float* A = sA + (16 * (w >> 2) + g) * LDA + t;
  const float* B = sB + (16 * (w & 3) + g) * LDA + t;
  float c[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}}, e[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
#pragma unroll 2
  for (int k0 = 0; k0 < NB; k0 += 8) {
    unsigned ah[4], al[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) split_tf32(A[8 * (q & 1) * LDA + k0 + 4 * (q >> 1)], ah[q], al[q]);
#pragma unroll
    for (int n = 0; n < 2; ++n) {
      unsigned bh[2], bl[2];
      split_tf32(B[8 * n * LDA + k0], bh[0], bl[0]);
      split_tf32(B[8 * n * LDA + k0 + 4], bh[1], bl[1]);
      tf32_mma(c[n], ah, bh);
      tf32_mma(e[n], al, bh);
      tf32_mma(e[n], ah, bl);
    }
  }
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
      for (int h = 0; h < 2; ++h) d[4 * mt + 2 * n + h] = c[n][2 * mt + h] + e[n][2 * mt + h];
}
// 32 rows of a tile, as stage_async.
template <typename T>
__device__ __forceinline__ void stage_half(const T* g, int ld, T* s) {
  constexpr int per_row = NB * (int)sizeof(T) / 16, elems = 16 / (int)sizeof(T);
#pragma unroll
  for (int q = 0; q < 32 * per_row / THREADS; ++q) {
    const int t = threadIdx.x + q * THREADS, r = t / per_row, c = (t % per_row) * elems;
    cp_async16(s + r * LDA + c, g + (size_t)r * ld + c);
  }
}
// The second of two halves to arrive sets the flag: its counter's
// acquire-release and the flag's release order both halves' stores before it.
__device__ __forceinline__ void publish_half(int* counter, int* flag, int value) {
  int old;
  asm volatile("atom.add.acq_rel.gpu.global.s32 %0, [%1], 1;" : "=r"(old) : "l"(counter) : "memory");
  if (old == 1) st_release(flag, value);
}

// Shared memory of a worker's LEAD task: two tiles and two halves.
template <typename T>
constexpr size_t lead_smem_bytes() { return sizeof(T) * (NB * ChainLd<T>::LT + 2 * NB * LDA); }

// LEAD(k, h), rows 32 h .. 32 h + 31 of the tile row i = k + 2 of panel k: S(i, k),
// then U(i, k+1, k) -- the last update of the chain's next solve input -- with
// the rows of L(i, k) kept in shared memory in between.  Everything that does
// not need L_kk is done before the wait for it (the last update of A(i, k), the
// fetch of the target), so that from F(k) to the chain's input there are one
// solve, one product and two hand-overs.  The row is two tasks because both are
// bound by one SM's FP64 tensor pipe (a 64-row solve 1.6 us, a 64-row product
// 2.1 us): at order 1000 in FP64 the chain no longer waits, 174 us against 188.  The counters of the two
// halves are the flags of tile (k, k + 2), which is above the diagonal.
template <typename T>
__device__ bool lead_task(const DFArgs& a, int k, int h, T* s, int* s_ok) {
  constexpr int LT = ChainLd<T>::LT;
  const int nt = a.nt, i = k + 2, ld = a.ld;
  T* Li = s;                 // rows of A(i, k), then of L(i, k)
  T* sC = Li + 32 * LDA;     // rows of A(i, k+1)
  T* sB = sC + 32 * LDA;     // L(k, k-1), then L(k+1, k)
  T* sV = sB + NB * LDA;     // the solve blocks of L_kk
  auto rows = [&](int j) { return tile<T>(a, i, j) + (size_t)32 * h * ld; };
  T d[8];
  if (k > 0) {
    const int* fl[4] = {a.fin + i * nt + k - 1, a.fin + k * nt + k - 1, a.upd + i * nt + k, a.upd + i * nt + k + 1};
    const int tg[4] = {1, 1, k - 1, k};
    if (!wait_all(a, fl, tg, 3, s_ok)) return false;
    stage_half(rows(k), ld, Li);
    stage_half(rows(k - 1), ld, sC);
    stage_async(tile<T>(a, k, k - 1), ld, sB, LDA);
    cp_async_wait_all();
    __syncthreads();
    half_product(sC, sB, d);
#pragma unroll
    for (int q = 0; q < 8; ++q) Li[half_row(q >> 2) * LDA + half_col((q >> 1) & 1) + (q & 1)] -= d[q];
    if (!wait_geq(a, fl[3], tg[3], s_ok)) return false;  // (its barrier: sC is read)
  } else {
    stage_half(rows(0), ld, Li);
  }
  stage_half(rows(k + 1), ld, sC);
  if (!wait_geq(a, a.fin + k * nt + k, 1, s_ok)) return false;
  stage_async(reinterpret_cast<const T*>(a.lp) + (size_t)k * NB * NB, NB, sV, LT);
  cp_async_wait_all();
  __syncthreads();
  T* out = rows(k);
  if (threadIdx.x < 128)  // 32 rows: warps 0 .. 3 (FP64), 0 and 1 of them in FP32
    solve_half<T>(Li, sV, [&](int r, int c, T w0, T w1) {
      store_pair(Li + r * LDA + c, w0, w1);
      store_pair(out + (size_t)r * ld + c, w0, w1);
    });
  __syncthreads();
  // at once: the updates of row k + 2 that the next LEAD starts from wait for it
  int* counter = a.fin + k * nt + i;
  if (threadIdx.x == 32) publish_half(counter, a.fin + i * nt + k, 1);
  if (!wait_geq(a, a.fin + (k + 1) * nt + k, 1, s_ok)) return false;
  stage_async(tile<T>(a, k + 1, k), ld, sB, LDA);
  cp_async_wait_all();
  __syncthreads();
  half_product(Li, sB, d);
  T* o = rows(k + 1);
#pragma unroll
  for (int q = 0; q < 8; q += 2) {
    const int r = half_row(q >> 2), c = half_col((q >> 1) & 1);
    store_pair(o + (size_t)r * ld + c, sC[r * LDA + c] - d[q], sC[r * LDA + c + 1] - d[q + 1]);
  }
  __syncthreads();
  if (threadIdx.x == 0) publish_half(a.upd + k * nt + i, a.upd + i * nt + k + 1, k + 1);
  return true;
}

// The worker CTAs' task loop.  FP32 lists (T = float): every update task
// (one to four rows) runs on the tcgen05 tensor cores (update_rows_tc, w
// holds the CTA's TMEM); FP64 lists: DMMA tile products.
template <typename T>
__device__ void df_worker_loop(const DFArgs& a, unsigned char* smem, int* s_task_p, int* s_ok_p, TcWorker* w) {
  int& s_task = *s_task_p;
  int& s_ok = *s_ok_p;
  T* sA = reinterpret_cast<T*>(smem);
  T* sB = sA + NB * LDA;
  const int nt = a.nt;
  while (true) {
    if (threadIdx.x == 0) s_task = ld_acquire(a.ctl + 1) ? a.ntasks : atomicAdd(a.ctl, 1);
    __syncthreads();
    const int t = s_task;
    __syncthreads();
    if (t >= a.ntasks) return;
    const int4 tk = a.tasks[t];
    const int type = tk.x, i = tk.y, j = tk.z, k = tk.w;
    TRACE(0, t);
    TRACE(3, t);
    T acc[16];
    if (sizeof(T) == 4 && (type == TASK_U || type == TASK_U2 || type == TASK_U3 || type == TASK_U4)) {
      // U(i + r, j, k), r < rows: L_(i+r)k, L_jk final and the k previous updates of each (i + r, j)
      const int rows = type == TASK_U ? 1 : type == TASK_U2 ? 2 : type == TASK_U3 ? 3 : 4;
      const int* fl[9];
      int tg[9];
      fl[0] = a.fin + j * nt + k;
      tg[0] = 1;
#pragma unroll
      for (int r = 0; r < 4; ++r) {
        const int rr = r < rows ? r : 0;
        fl[1 + 2 * r] = a.fin + (i + rr) * nt + k;
        tg[1 + 2 * r] = 1;
        fl[2 + 2 * r] = a.upd + (i + rr) * nt + j;
        tg[2 + 2 * r] = k;
      }
      if (!wait_all(a, fl, tg, 1 + 2 * rows, &s_ok)) return;
      TRACE(1, t);
      if (!update_rows_tc(a, i, rows, j, k, *w)) return;
      if (threadIdx.x < rows) st_release(a.upd + (i + threadIdx.x) * nt + j, k + 1);
      TRACE(2, t);
    } else if (type == TASK_XG) {
      const int rows = i + 1 < nt ? 2 : 1;
      const int* fl[5] = {k == j ? a.fin + j * nt + j : a.xfin + k * nt + j, a.fin + i * nt + k,
                          a.xupd + i * nt + j, a.fin + (i + rows - 1) * nt + k, a.xupd + (i + rows - 1) * nt + j};
      const int tg[5] = {k == j ? 2 : 1, 1, k - j, 1, k - j};
      if (!wait_all(a, fl, tg, 5, &s_ok)) return;
      TRACE(1, t);
      inverse_update<T>(a, i, rows, j, k, sA);
      __syncthreads();
      if (threadIdx.x < rows) st_release(a.xupd + (i + threadIdx.x) * nt + j, k - j + 1);
      TRACE(2, t);
    } else if (type == TASK_XZ) {
      const int* fl[4] = {a.fin + i * nt + i - 1, i - 1 == j ? a.fin + j * nt + j : a.xfin + (i - 1) * nt + j,
                          a.fin + i * nt + i, a.xupd + i * nt + j};
      const int tg[4] = {1, i - 1 == j ? 2 : 1, 2, i - 1 - j};
      if (!wait_all(a, fl, tg, 4, &s_ok)) return;
      TRACE(1, t);
      inverse_finish<T>(a, i, j, sA);
      publish(a.xfin + i * nt + j, 1);
      TRACE(2, t);
    } else if (type == TASK_I) {
      // I(k): inv(L_kk) for the solves of column k, from the stored L_kk
      if (!wait_geq(a, a.fin + k * nt + k, 1, &s_ok)) return;
      TRACE(1, t);
      double* Lk = reinterpret_cast<double*>(smem);
      double* Xw = Lk + NB * LDA;
      double* Tm = Xw + NB * LDA;
      double* Rv = Tm + 32 * 36;
      const T* g = tile<T>(a, k, k);
      T v[TILE_PER_THREAD];  // all loads in flight before the first store
#pragma unroll
      for (int q = 0; q < TILE_PER_THREAD; ++q) {
        const int e = threadIdx.x + q * THREADS;
        v[q] = ldcg(g + (size_t)(e >> 6) * a.ld + (e & 63));
      }
#pragma unroll
      for (int q = 0; q < TILE_PER_THREAD; ++q) {
        const int e = threadIdx.x + q * THREADS, r = e >> 6, c = e & 63;
        Lk[r * LDA + c] = c <= r ? (double)v[q] : 0.0;
      }
      __syncthreads();
      if (threadIdx.x < NB) Rv[threadIdx.x] = 1.0 / Lk[threadIdx.x * LDA + threadIdx.x];
      __syncthreads();
      store_inverse<double, T>(a, k, Lk, Rv, Xw, Tm);
      publish(a.fin + k * nt + k, 2);
      TRACE(2, t);
    } else if (type == TASK_U) {
      if constexpr (sizeof(T) == 8) {  // FP32: on the tensor cores, above
        // U(i, j, k): needs L_ik, L_jk final and the k previous updates of (i, j)
        const int* fl[3] = {a.fin + i * nt + k, a.fin + j * nt + k, a.upd + i * nt + j};
        const int tg[3] = {1, 1, k};
        if (!wait_all(a, fl, tg, 3, &s_ok)) return;
        TRACE(1, t);
        update_tile(a, i, j, k, acc, sA, sB, sB + NB * LDA);
        publish(a.upd + i * nt + j, k + 1);
        TRACE(2, t);
      }
    } else if (type == TASK_U2) {
      if constexpr (sizeof(T) == 8) {  // FP32: on the tensor cores, above
        // U(i, j, k) and U(i+1, j, k): L_ik, L_{i+1,k}, L_jk final, k previous updates of both
        const int* fl[5] = {a.fin + i * nt + k, a.fin + (i + 1) * nt + k, a.fin + j * nt + k, a.upd + i * nt + j,
                            a.upd + (i + 1) * nt + j};
        const int tg[5] = {1, 1, 1, k, k};
        if (!wait_all(a, fl, tg, 5, &s_ok)) return;
        TRACE(1, t);
        update_tile_pair(a, i, j, k, acc, sA);
        __syncthreads();
        if (threadIdx.x == 0) {
          st_release(a.upd + i * nt + j, k + 1);
          st_release(a.upd + (i + 1) * nt + j, k + 1);
        }
        TRACE(2, t);
      }
    } else if (type == TASK_LEAD) {
      if (!lead_task<T>(a, k, i, sA, &s_ok)) return;
      TRACE(2, t);
    } else {
      // S(i, j), i >= j + 3: the tile after its last update, times L_jj^-T
      if (!solve_input<T>(a, i, j, acc, sA, sB, &s_ok)) return;
      if (!wait_geq(a, a.fin + j * nt + j, 1, &s_ok)) return;  // the solve blocks of L_jj are stored
      TRACE(1, t);
      constexpr int LT = ChainLd<T>::LT;
      stage_async(reinterpret_cast<const T*>(a.lp) + (size_t)j * NB * NB, NB, sB, LT);
      acc_to_smem(acc, sA);
      cp_async_wait_all();
      __syncthreads();
      T* out = tile<T>(a, i, j);
      solve_rows_t<T>(sA, LDA, sB, [&](int r, int c, T w0, T w1) { store_pair(out + (size_t)r * a.ld + c, w0, w1); });
      publish(a.fin + i * nt + j, 1);
      TRACE(2, t);
    }
    __syncthreads();
  }
}

// A matrix of type T; the chain CTA works in FP64.  The FP32 workers hold TMEM for their tensor-core
// updates from start to end.
template <typename T>
__global__ void __launch_bounds__(THREADS, 1) chol_df_kernel(DFArgs a) {
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int s_task, s_ok;
  if (blockIdx.x == 0) {
    run_chain<T>(a, smem, &s_ok);
    return;
  }
  if constexpr (sizeof(T) == 4) {
    __shared__ __align__(8) uint64_t s_mbar;
    __shared__ uint32_t s_tmem;
    TcWorker w;
    tc_worker_begin(&s_mbar, &s_tmem, smem, 2, w);
    df_worker_loop<T>(a, smem, &s_task, &s_ok, &w);
    tc_worker_end(w);
  } else {
    df_worker_loop<T>(a, smem, &s_task, &s_ok, nullptr);
  }
}

// Batched FP64 factorisation (right-looking; the mixed batch runs the
// left-looking chol_batch_ll_kernel below): every task comes from the shared
// list (there is no chain CTA); F(k) applies its last update itself.  Shared
// memory: two tiles (sA, sB) for the updates and solves; F uses two tiles
// (L_kk, its solve blocks) over the same bytes and the factor scratch after them.
constexpr size_t batch_smem_bytes() {
  // an F task's tile, solve blocks and factor scratch, or a paired update's five tiles
  return std::max(sizeof(double) * (2 * NB * ChainLd<double>::LT + FACTOR_SCRATCH),
                  5 * NB * LDA * sizeof(double));
}

// The FP64 batched kernel's task loop: DMMA updates in pairs (five tiles
// staged in one round, the loads overlapped with the math inside the CTA).
template <typename T>
__device__ void batch_worker_loop(const CholRep* __restrict__ reps, const int4* __restrict__ tasks, int ntasks,
                                  int* ctl, unsigned char* smem) {
  __shared__ int s_task, s_ok;
  T* sA = reinterpret_cast<T*>(smem);
  T* sB = sA + NB * LDA;
  constexpr int LT = ChainLd<T>::LT;
  T* Ft = reinterpret_cast<T*>(smem);  // F: the tile, its solve blocks, the scratch
  const FactorMem f(Ft, Ft + NB * LT, Ft + 2 * NB * LT);
  while (true) {
    if (threadIdx.x == 0) s_task = ld_acquire(ctl + 1) ? ntasks : atomicAdd(ctl, 1);
    __syncthreads();
    const int t = s_task;
    __syncthreads();
    if (t >= ntasks) return;
    const int4 tk = tasks[t];
    const int type = tk.x & 7, i = tk.y, j = tk.z, k = tk.w;
    const CholRep& R = reps[tk.x >> 3];
    DFArgs a;
    a.A = R.A;
    a.ld = R.ld;
    a.n = R.n;
    a.nt = R.nt;
    a.ntasks = ntasks;
    a.tasks = tasks;
    a.ctl = ctl;
    a.upd = R.upd;
    a.fin = R.fin;
    a.info = R.info;
    a.lp = R.invdiag;  // the solve blocks take the place of the inverses
    a.err = reinterpret_cast<unsigned*>(ctl + 3);
    a.spin_limit = SPIN_LIMIT;
    const int nt = a.nt;
    T acc[16];
    if (type == TASK_U) {
      const int* fl[3] = {a.fin + i * nt + k, a.fin + j * nt + k, a.upd + i * nt + j};
      const int tg[3] = {1, 1, k};
      if (!wait_all(a, fl, tg, 3, &s_ok)) return;
      load_and_update(a, i, j, k, acc, sA, sB);
      store_acc(tile<T>(a, i, j), a.ld, acc);
      publish(a.upd + i * nt + j, k + 1);
    } else if (type == TASK_U2) {
      const int* fl[5] = {a.fin + i * nt + k, a.fin + (i + 1) * nt + k, a.fin + j * nt + k, a.upd + i * nt + j,
                          a.upd + (i + 1) * nt + j};
      const int tg[5] = {1, 1, 1, k, k};
      if (!wait_all(a, fl, tg, 5, &s_ok)) return;
      update_tile_pair(a, i, j, k, acc, sA);
      __syncthreads();
      if (threadIdx.x == 0) {
        st_release(a.upd + i * nt + j, k + 1);
        st_release(a.upd + (i + 1) * nt + j, k + 1);
      }
    } else {
      const int col = j;
      if (col > 0) {
        const int* fl[3] = {a.fin + i * nt + col - 1, a.fin + col * nt + col - 1, a.upd + i * nt + col};
        const int tg[3] = {1, 1, col - 1};
        if (!wait_all(a, fl, tg, 3, &s_ok)) return;
        load_and_update(a, i, col, col - 1, acc, sA, sB);  // ends with a barrier: smem is free
      } else {
        load_acc(tile<T>(a, i, col), a.ld, acc);
      }
      if (type == TASK_F) {
        acc_to_smem(acc, Ft, LT);
        if (threadIdx.x == 0) {
          f.bad[0] = NB;
          f.bad[1] = 0;
        }
        __syncthreads();
        factor_tile<T>(a, col, f, reinterpret_cast<T*>(a.lp) + (size_t)col * NB * NB);
      } else {
        if (!wait_geq(a, a.fin + col * nt + col, 1, &s_ok)) return;
        stage_async(reinterpret_cast<const T*>(a.lp) + (size_t)col * NB * NB, NB, sB, LT);
        acc_to_smem(acc, sA);
        cp_async_wait_all();
        __syncthreads();
        T* out = tile<T>(a, i, col);
        solve_rows_t<T>(sA, LDA, sB, [&](int r, int c, T w0, T w1) { store_pair(out + (size_t)r * a.ld + c, w0, w1); });
      }
      publish(a.fin + i * nt + col, 1);
    }
    __syncthreads();
  }
}

template <typename T>
__global__ void __launch_bounds__(THREADS, 1) chol_batch_kernel(const CholRep* __restrict__ reps,
                                                                 const int4* __restrict__ tasks, int ntasks,
                                                                 int* ctl) {
  static_assert(sizeof(T) == 8, "the mixed batch runs chol_batch_ll_kernel");
  extern __shared__ __align__(16) unsigned char smem[];
  batch_worker_loop<T>(reps, tasks, ntasks, ctl, smem);
}

// ---------------------------------------------------------------- left-looking batched factorisation
// The mixed batch factors every replica left-looking on the tcgen05 tensor
// cores.  A task owns the row tiles i and i + 1 of column j of L (only i
// when i + 1 = nt) and forms
//   U_rj = A_rj - sum_{k < j} L_rk L_jk^T        (r = i, i + 1)
// as one M = 128, N = 64, K = 64 j product accumulated in TMEM: for each k
// the tiles L_ik, L_{i+1,k}, L_jk are split into TF32 hi / lo halves in
// shared memory and three MMAs per K-step add A_hi B_hi + A_hi B_lo + A_lo
// B_hi to the accumulator, while the tiles of k + 1 are split into a second
// operand buffer.  Then, by the task's kind:
//   LL_DIAG (i = j): F(j) (factor_tile, FP64 rounded on store), published at once,
//     then S(j + 1, j) with the solve blocks still in shared memory;
//   LL_UPDATE (i > j): U written over A's tiles, upd[r] = j + 1;
//   LL_SOLVE (i > j, a later segment): S(i, j), S(i + 1, j) from the stored
//     U once F(j) is published.
// Every tile is read as A once and written twice (U, then L), where a
// right-looking update reads and writes its tile once per panel.  Flags:
// fin[r] = the number of final tiles of row r, upd[r] = the columns of row r
// whose U is stored.  A row's tiles become final in column order (tile
// (r, j) needs (r, j - 1)), so one counter per row says which L_rk are
// ready.  Every task depends only on earlier tasks of the list.
constexpr uint32_t LL_A_BYTES = tc::operand_bytes(128);
constexpr uint32_t LL_B_BYTES = tc::operand_bytes(64);
constexpr uint32_t LL_OPERAND_BYTES = 2 * LL_A_BYTES + 2 * LL_B_BYTES;
// Two operand buffers from the 1024-byte aligned start of dynamic shared memory,
// then the worker's words (LLShared).  After the last product the first buffer's
// bytes hold P ([128][LDA] floats from 0), the U tiles ([64][LDA] at LL_U0 and
// LL_U1) and the factor scratch (from 0).
struct LLShared {
  uint64_t mbar[2], conv[2];
  uint32_t tmem;
  int task, ok, seen[3];
};
constexpr uint32_t LL_SHARED_OFFSET = 2 * LL_OPERAND_BYTES;
constexpr size_t ll_smem_bytes() { return LL_SHARED_OFFSET + sizeof(LLShared); }
static_assert(ll_smem_bytes() <= 227 * 1024, "the worker does not fit an SM");
// task kinds of the left-looking list
enum : int { LL_DIAG = 0, LL_UPDATE = 1, LL_SOLVE = 2 };
// K-steps (of 64) accumulated in TMEM before the sum is added in FP32
constexpr int LL_CHUNK = 4;
constexpr uint32_t LL_U0 = 40960, LL_U1 = 61440;
// F(j)'s tile, solve blocks and scratch take the second buffer's bytes
constexpr uint32_t LL_FACTOR_BYTES = sizeof(double) * (2 * NB * ChainLd<double>::LT + FACTOR_SCRATCH);
static_assert(LL_FACTOR_BYTES <= LL_OPERAND_BYTES, "the factor does not fit an operand buffer");
static_assert(sizeof(float) * 128 * LDA <= LL_U0, "P overlaps U0");
static_assert(LL_U1 + sizeof(float) * NB * LDA <= LL_OPERAND_BYTES, "U1 lies outside the operand bytes");

struct LLWorker {
  uint64_t* mbar;       // [2] completion of the products of one K-step, per operand buffer
  uint64_t* conv;       // [2] every thread's operands of a K-step written (THREADS arrivals)
  uint32_t tmem;        // TMEM base: two 128 x 128 FP32 accumulators (hi hi | cross terms)
  uint32_t phase;       // bit b: the parity of mbar[b]
  uint32_t conv_phase;  // thread 0's, of conv
  unsigned char* base;  // 1024-byte aligned operand buffers
};

__device__ __forceinline__ DFArgs batch_args(const CholRep& R, const int4* tasks, int ntasks, int* ctl) {
  DFArgs a;
  a.A = R.A;
  a.ld = R.ld;
  a.n = R.n;
  a.nt = R.nt;
  a.ntasks = ntasks;
  a.tasks = tasks;
  a.ctl = ctl;
  a.upd = R.upd;
  a.fin = R.fin;
  a.info = R.info;
  a.invdiag = nullptr;
  a.lp = R.invdiag;  // the solve blocks take the place of the inverses
  a.min_pivot = 1.17549435e-38;  // a smaller pivot is reported as non-positive
  a.err = reinterpret_cast<unsigned*>(ctl + 3);
  a.spin_limit = SPIN_LIMIT;
  a.X = nullptr;
  a.xupd = nullptr;
  a.xfin = nullptr;
  return a;
}

// Warp 0 waits until base[rows[q]] >= target for every slot q in mask
// (bounded, with the abort polling of wait_all).  seen[q] (touched by warp 0
// only) keeps the largest count observed for slot q in this task, so a wait
// that an earlier observation already satisfies costs no memory round trip.
// *s_ok only ever goes from 1 to 0.  Ends with a CTA barrier.
__device__ bool ll_wait_rows(const DFArgs& a, const int* base, const int (&rows)[3], unsigned mask, int target,
                             int* seen, int* s_ok) {
  if (threadIdx.x < 32) {
    const int lane = threadIdx.x;
    const bool mine = lane < 3 && ((mask >> lane) & 1u);
    const int* flag = mine ? base + rows[lane < 3 ? lane : 0] : nullptr;
    bool done = !mine || seen[lane] >= target;
    bool ok = true;
    for (long long it = 0;; ++it) {
      if (!done) {
        const int v = ld_acquire(flag);
        if (v >= target) {
          seen[lane] = v;
          done = true;
        }
      }
      if (__all_sync(0xffffffffu, done)) break;
      if ((it & 15) == 15) {
        const int ab = __shfl_sync(0xffffffffu, lane == 0 ? ld_acquire(a.ctl + 1) : 0, 0);
        if (ab) {
          ok = false;
          break;
        }
      }
      if (it + 1 > a.spin_limit) {
        if (lane == 0) wait_expired(a);
        ok = false;
        break;
      }
      if (it > 256) __nanosleep(200);
    }
    if (lane == 0 && !ok) *s_ok = 0;
  }
  __syncthreads();
  return *s_ok != 0;
}


// cp.async (16 bytes, through L2) of this thread's share of a 64 x 64 FP32
// tile into a row-major [64][64] stage; the same thread converts the same
// chunks later, so its own wait_group makes them visible to it.
__device__ __forceinline__ void ll_fetch_tile(const float* src, int ld, float* raw) {
#pragma unroll
  for (int e = 0; e < tc::TileShare<THREADS>::PER; ++e) {
    const int q = threadIdx.x + e * THREADS, r = q >> 4, c = q & 15;
    cp_async16(raw + r * NB + 4 * c, src + (size_t)r * ld + 4 * c);
  }
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait_group() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Per-thread bounded wait until base[rows[q]] >= target for q = 0, 1, 2,
// with the counts observed so far kept in the thread's registers (seen): a
// wait that an earlier observation satisfies costs nothing, and the thread's
// own acquire orders its later reads (no barrier).  false: the wait gave up
// (recorded like an expired wait_all) or the run was aborted.
__device__ bool ll_thread_wait_rows(const DFArgs& a, const int* base, const int (&rows)[3], int target,
                                    int (&seen)[3]) {
#pragma unroll
  for (int q = 0; q < 3; ++q) {
    for (long long it = 0; seen[q] < target; ++it) {
      const int v = ld_acquire(base + rows[q]);
      if (v >= target) {
        seen[q] = v;
        break;
      }
      if ((it & 63) == 63) {
        if (ld_acquire(a.ctl + 1)) return false;
        if (it > a.spin_limit) {
          wait_expired(a);
          return false;
        }
        __nanosleep(64);
      }
    }
  }
  return true;
}

__device__ __forceinline__ void ll_arrive(uint64_t* m) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_u32(m)) : "memory");
}

// P = sum_{k < j} [L_ik; L_{i+1,k}] L_jk^T into shared memory ([128][LDA]
// floats at the operand area's start), for j > 0, and A's tiles (i, j), (i + 1, j)
// into As.  Two operand buffers: the tiles of K-step k are split into one
// while the products of k - 1 run from the other, and a tile's registers take
// its successor (loaded straight from L2) as soon as it is split.  The first version had one
// buffer, and two raw stages in shared memory for the tiles on their way: split
// and products alternated, and every tile crossed shared memory twice more
// (3000 cycles a K-step of the 256-replica batch, 1730 now).  No
// CTA barrier inside the K loop: every thread loads and splits only its
// own chunks, waits for the products of k - 2 on their mbarrier before overwriting
// their operands, and arrives on the buffer's conversion mbarrier; thread 0 waits for
// all arrivals and issues the MMAs.  Returns false (after a CTA barrier) if the
// run was aborted, with no products of this CTA left in flight.
__device__ bool ll_products(const DFArgs& a, int i, int j, LLWorker& w, tc::TileShare<THREADS> (&As)[2]) {
  const int tid = threadIdx.x;
  const bool two = i + 1 < a.nt;
  const int rows[3] = {i, two ? i + 1 : i, j};
  int seen[3] = {0, 0, 0};
  if (!two) {
    // rows 64 .. 127 of the A halves stay zero for the whole task: bytes
    // 8192 .. 16383 of each of the two K blocks (16384 bytes each)
    for (int e = tid; e < 8 * 512; e += THREADS) {
      const int part = e >> 9, off = (e & 511) * 16;
      unsigned char* p = w.base + (part >> 2) * LL_OPERAND_BYTES + (part & 1) * LL_A_BYTES + ((part >> 1) & 1) * 16384 +
                         8192 + off;
      *reinterpret_cast<uint4*>(p) = make_uint4(0u, 0u, 0u, 0u);
    }
  }
  tc::TileShare<THREADS> sB;
  long long c0 = LLCLK();
  bool ok = ll_thread_wait_rows(a, a.fin, rows, 1, seen);
  if (ok) {
    tc::load_share(tile<float>(a, i, 0), a.ld, As[0]);
    if (two) tc::load_share(tile<float>(a, i + 1, 0), a.ld, As[1]);
    tc::load_share(tile<float>(a, j, 0), a.ld, sB);
  }
  LLPROF(2, LLCLK() - c0);
  // the products accumulate in TMEM for LL_CHUNK K-steps at a time, the chunks in
  // two accumulators in turn; each chunk's sum is added in FP32 to racc (this
  // thread's row m, columns 32 g .. 32 g + 31) while the next one runs, so no
  // accumulation runs longer than K = 64 LL_CHUNK in the tensor cores
  const int warp = tid >> 5, lane = tid & 31, q = warp & 3, g = warp >> 2;
  const int m = 32 * q + lane;
  const uint32_t tacc = w.tmem + ((uint32_t)(32 * q) << 16) + 32 * g;
  float racc[32];
#pragma unroll
  for (int u = 0; u < 32; ++u) racc[u] = 0.0f;
  auto fold = [&](int chunk) {
    float v[32], x[32];
    tc::tmem_ld32(tacc + 128 * (chunk & 1), v);
    tc::tmem_ld32(tacc + 128 * (chunk & 1) + 64, x);
#pragma unroll
    for (int u = 0; u < 32; ++u) racc[u] += v[u] + x[u];
  };
  auto finished = [&](int k) {  // waits for the products of K-step k
    const int b = k & 1;
    if (!tc::mbar_wait(w.mbar + b, (w.phase >> b) & 1u, a.spin_limit)) ok = false;
    w.phase ^= 1u << b;
  };
  for (int k = 0; k < j; ++k) {
    const int b = k & 1;
    unsigned char* Ahi = w.base + b * LL_OPERAND_BYTES;
    unsigned char* Alo = Ahi + LL_A_BYTES;
    unsigned char* B = Alo + LL_A_BYTES;
    c0 = LLCLK();
    if (k >= 2) {  // the products of k - 2 have read this buffer
      finished(k - 2);
      tc::fence_after_sync();
      if (k > LL_CHUNK && k % LL_CHUNK == 1) {
        // ... and were the last of a chunk; its accumulator is started again
        // LL_CHUNK - 1 steps from here (ordered by the conversion mbarriers)
        fold(k / LL_CHUNK - 1);
        tc::fence_before_sync();
      }
    }
    const long long c1 = LLCLK();
    LLPROF(3, c1 - c0);
    // the next step's tiles (or A's), where their rows are known to be final
    const bool last = k + 1 == j;
    const bool ready = __all_sync(0xffffffffu, ok && (last || min(seen[0], min(seen[1], seen[2])) >= k + 2));
    const int next = last ? j : k + 1;
    tc::store_share_split<THREADS>(As[0], 128, 0, Ahi, Alo);
    if (ready) tc::load_share(tile<float>(a, i, next), a.ld, As[0]);
    if (two) {
      tc::store_share_split<THREADS>(As[1], 128, 64, Ahi, Alo);
      if (ready) tc::load_share(tile<float>(a, i + 1, next), a.ld, As[1]);
    }
    tc::store_share_split<THREADS>(sB, 128, 0, B, B + 64 * 128);  // lo 64 rows below hi
    if (ready && !last) tc::load_share(tile<float>(a, j, next), a.ld, sB);
    tc::fence_proxy_smem();
    ll_arrive(w.conv + b);
    if (tid == 0) {
      if (!tc::mbar_wait(w.conv + b, (w.conv_phase >> b) & 1u, a.spin_limit)) ok = false;  // all operands written
      w.conv_phase ^= 1u << b;
      tc::fence_after_sync();
      tc::issue_product_wide(w.tmem + 128 * ((k / LL_CHUNK) & 1), tc::smem_u32(Ahi), tc::smem_u32(Alo), tc::smem_u32(B),
                             k % LL_CHUNK != 0 ? 1u : 0u);
      tc::mma_commit(w.mbar + b);
    }
    c0 = LLCLK();
    LLPROF(4, c0 - c1);
    if (!ready) {
      ok = ok && (last || ll_thread_wait_rows(a, a.fin, rows, k + 2, seen));
      if (ok) {
        tc::load_share(tile<float>(a, i, next), a.ld, As[0]);
        if (two) tc::load_share(tile<float>(a, i + 1, next), a.ld, As[1]);
        if (!last) tc::load_share(tile<float>(a, j, next), a.ld, sB);
      }
      LLPROF(2, LLCLK() - c0);
    }
  }
  c0 = LLCLK();
  if (j > 1) finished(j - 2);
  finished(j - 1);
  ok = __syncthreads_and(ok) != 0;
  LLPROF(3, LLCLK() - c0);
  if (!ok) {
    if (tid == 0) {
      atomicExch(a.ctl + 1, 1);
      atomicOr(a.err, PBG_DEV_ERR_BARRIER);
      atomicCAS(a.info, 0, -1);
    }
    return false;
  }
  tc::fence_after_sync();
  // P = racc + the chunks still in TMEM, into shared memory, row m = TMEM lane
  const int chunk = (j - 1) / LL_CHUNK;
  if (chunk > 0 && (j - 1) % LL_CHUNK == 0) fold(chunk - 1);
  fold(chunk);
  if (two || q < 2) {  // warp-uniform
    float* dst = reinterpret_cast<float*>(w.base) + (size_t)m * LDA + 32 * g;
#pragma unroll
    for (int u = 0; u < 8; ++u)
      *reinterpret_cast<float4*>(dst + 4 * u) =
          make_float4(racc[4 * u], racc[4 * u + 1], racc[4 * u + 2], racc[4 * u + 3]);
  }
  tc::fence_before_sync();
  __syncthreads();
  return true;
}

// U = A - P for rows i (and i + 1) of column j; A's tiles in As (this thread's
// chunks), no P for j = 0; into the [64][LDA] tiles U0 / U1 in shared memory,
// or in place into A when to_global.
__device__ __forceinline__ void ll_difference(const DFArgs& a, int i, int j, bool two, const float* Ps,
                                              const tc::TileShare<THREADS> (&As)[2], float* U0, float* U1,
                                              bool to_global) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    if (h == 1 && !two) break;
    float* gp = tile<float>(a, i + h, j);
    float* U = h == 0 ? U0 : U1;
#pragma unroll
    for (int e = 0; e < tc::TileShare<THREADS>::PER; ++e) {
      const int t = threadIdx.x + e * THREADS, r = t >> 4, c = 4 * (t & 15);
      float4 cv = As[h].v[e];
      if (j > 0) {
        const float4 pv = *reinterpret_cast<const float4*>(Ps + (size_t)(64 * h + r) * LDA + c);
        cv.x -= pv.x;
        cv.y -= pv.y;
        cv.z -= pv.z;
        cv.w -= pv.w;
      }
      if (to_global) *reinterpret_cast<float4*>(gp + (size_t)r * a.ld + c) = cv;
      else *reinterpret_cast<float4*>(U + r * LDA + c) = cv;
    }
  }
}

// One task of the left-looking list (kinds in cholesky_replica_tasks).
// Returns false if the run was aborted (nothing of this CTA in flight then).
__device__ bool ll_task(const DFArgs& a, int kind, int i, int j, LLWorker& w, int* seen, int* s_ok) {
  const int tid = threadIdx.x;
  const bool two = i + 1 < a.nt;
  const int rows[3] = {i, two ? i + 1 : i, j};
  if (tid < 3) seen[tid] = 0;
  float* Ps = reinterpret_cast<float*>(w.base);
  float* U0 = reinterpret_cast<float*>(w.base + LL_U0);
  float* U1 = reinterpret_cast<float*>(w.base + LL_U1);
  long long c0 = LLCLK();
  LLPROF(0, 1);
  LLPROF(1, j);
  if (kind != LL_SOLVE) {
    tc::TileShare<THREADS> As[2];
    if (j > 0) {
      if (!ll_products(a, i, j, w, As)) return false;
    } else {
      tc::load_share(tile<float>(a, i, 0), a.ld, As[0]);
      if (two) tc::load_share(tile<float>(a, i + 1, 0), a.ld, As[1]);
    }
    c0 = LLCLK();
    ll_difference(a, i, j, two, Ps, As, U0, U1, kind == LL_UPDATE);
    __syncthreads();
    LLPROF(5, LLCLK() - c0);
    c0 = LLCLK();
  }
  if (kind == LL_DIAG) {
    // F(j) in FP64, as the single-matrix chain does it, in the second buffer's bytes,
    // then S(j + 1, j) with the solve blocks still in shared memory
    LLPROF(11, 1);
    constexpr int LT = ChainLd<double>::LT;
    double* F = reinterpret_cast<double*>(w.base + LL_OPERAND_BYTES);
    double* V = F + NB * LT;
    const FactorMem f(F, V, V + NB * LT);
    for (int e = tid; e < NB * NB; e += THREADS) F[(e >> 6) * LT + (e & 63)] = U0[(e >> 6) * LDA + (e & 63)];
    if (tid == 0) {
      f.bad[0] = NB;
      f.bad[1] = 0;
    }
    __syncthreads();
    factor_tile<float>(a, j, f, reinterpret_cast<float*>(a.lp) + (size_t)j * NB * NB);
    publish(a.fin + j, j + 1);
    if (two) {
      float* out = tile<float>(a, j + 1, j);
      solve_rows<1>(U1, LDA, V,
                    [&](int r, int c, double w0, double w1) { store_pair(out + (size_t)r * a.ld + c, (float)w0, (float)w1); });
      publish(a.fin + j + 1, j + 1);
    }
    LLPROF(6, LLCLK() - c0);
  } else if (kind == LL_UPDATE) {
    // U_ij (and U_{i+1,j}) stay in A's tiles for the solve task
    if (tid == 0) {
      st_release(a.upd + i, j + 1);
      if (two) st_release(a.upd + i + 1, j + 1);
    }
  } else {
    if (!ll_wait_rows(a, a.upd, rows, two ? 3u : 1u, j + 1, seen, s_ok)) return false;  // U_ij in A
    if (!ll_wait_rows(a, a.fin, rows, 4u, j + 1, seen, s_ok)) return false;             // F(j)
    LLPROF(7, LLCLK() - c0);
    c0 = LLCLK();
    float* Vs = reinterpret_cast<float*>(w.base);
    stage_async(reinterpret_cast<const float*>(a.lp) + (size_t)j * NB * NB, NB, Vs, ChainLd<float>::LT);
    stage_async(tile<float>(a, i, j), a.ld, U0, LDA);
    if (two) stage_async(tile<float>(a, i + 1, j), a.ld, U1, LDA);
    cp_async_wait_all();
    __syncthreads();
    // a tile on four warps each
    const int h = tid >> 7;
    if (h == 0 || two) {
      float* out = tile<float>(a, i + h, j);
      solve_rows_f32(h ? U1 : U0, LDA, Vs, (tid >> 5) & 3,
                     [&](int r, int c, float w0, float w1) { store_pair(out + (size_t)r * a.ld + c, w0, w1); });
    }
    __syncthreads();
    if (tid == 0) {
      st_release(a.fin + i, j + 1);
      if (two) st_release(a.fin + i + 1, j + 1);
    }
    LLPROF(8, LLCLK() - c0);
  }
  __syncthreads();  // the next task overwrites the shared memory
  return true;
}

// One CTA per SM (192 KB of shared memory, 256 TMEM columns), all co-resident
// (cooperative launch).
__global__ void __launch_bounds__(THREADS, 1) chol_batch_ll_kernel(const CholRep* __restrict__ reps,
                                                                   const int4* __restrict__ tasks, int ntasks,
                                                                   int* ctl) {
  extern __shared__ __align__(1024) unsigned char ll_smem[];
  unsigned char* smem = ll_smem;
  if (tc::smem_u32(smem) & 1023u) {
    // the operands need a 1024-byte aligned start: give up on the whole run,
    // every replica reported as not factored (info -1)
    if (threadIdx.x == 0) {
      atomicExch(ctl + 1, 1);
      atomicOr(reinterpret_cast<unsigned*>(ctl + 3), PBG_DEV_ERR_BARRIER);
    }
    for (int t = blockIdx.x * blockDim.x + threadIdx.x; t < ntasks; t += gridDim.x * blockDim.x)
      atomicCAS(reps[tasks[t].x >> 3].info, 0, -1);
    return;
  }
  LLShared* sh = reinterpret_cast<LLShared*>(smem + LL_SHARED_OFFSET);
  if (threadIdx.x == 0) {
    for (int b = 0; b < 2; ++b) {
      tc::mbar_init(&sh->mbar[b], 1);
      tc::mbar_init(&sh->conv[b], THREADS);
    }
    sh->ok = 1;
  }
  if (threadIdx.x < 32) tc::tmem_alloc(&sh->tmem, 256);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  LLWorker w;
  w.mbar = sh->mbar;
  w.conv = sh->conv;
  w.tmem = sh->tmem;
  w.phase = 0;
  w.conv_phase = 0;
  w.base = smem;
  const long long k0 = LLCLK();
  while (true) {
    const long long f0 = LLCLK();
    if (threadIdx.x == 0) sh->task = ld_acquire(ctl + 1) ? ntasks : atomicAdd(ctl, 1);
    __syncthreads();
    const int t = sh->task;
    __syncthreads();
    LLPROF(9, LLCLK() - f0);
    if (t >= ntasks) break;
    const int4 tk = tasks[t];
    const DFArgs a = batch_args(reps[tk.x >> 3], tasks, ntasks, ctl);
    if (!ll_task(a, tk.x & 7, tk.y, tk.z, w, sh->seen, &sh->ok)) break;
  }
  LLPROF(10, LLCLK() - k0);
  tc::fence_before_sync();
  __syncthreads();
  if (threadIdx.x < 32) tc::tmem_dealloc(w.tmem, 256);
}

std::mutex g_task_mu;
std::map<int, std::pair<int4*, int>> g_task_tables;

// Task list of the worker CTAs for an nt x nt tile grid (see the file comment).
// group: updates per task down a column (2; 4 for the FP32 kernel, whose
// updates run on the tcgen05 tensor cores); inv_tasks: the I(k) tasks that
// store inv(L_kk); inverse: the tasks that form X = inv(L) as well (they need
// the I(k) tasks).
std::vector<int4> df_task_list(int nt, int group, bool inv_tasks, bool inverse) {
  // The chain tasks F(k) and S(k+1, k) run on the chain CTA and are left out.
  std::vector<int4> t;
  for (int k = 0; k < nt; ++k) {
    const int q = k - 1;  // the panel whose trailing updates this block holds
    if (k > 0 && k + 2 < nt) {
      // the two updates that LEAD(k) waits for
      t.push_back(make_int4(TASK_U, k + 2, k + 1, q));
      t.push_back(make_int4(TASK_U, k + 2, k + 2, q));
    }
    if (k + 2 < nt) {
      t.push_back(make_int4(TASK_LEAD, 0, 0, k));
      t.push_back(make_int4(TASK_LEAD, 1, 0, k));
      t.push_back(make_int4(TASK_U, k + 2, k + 2, k));  // the chain's next diagonal tile
    }
    for (int i = k + 3; i < nt; ++i) t.push_back(make_int4(TASK_S, i, k, k));
    if (inv_tasks) t.push_back(make_int4(TASK_I, 0, 0, k));
    // Column k of the update with panel q is fused into F(k), LEAD(k) and the
    // S(., k); U(k+1, k, q) belongs to LEAD(q) and U(k+1, k+1, q) follows it.  The plain
    // updates cover the rest, columns from the left (rows grouped:
    // U(i, jj, q), U(i+1, jj, q), ... share L(jj, q)).
    if (k > 0)
      for (int jj = k + 1; jj < nt; ++jj) {
        int i = std::max(jj, k + 3);
        if (group >= 4)
          for (; i + 3 < nt; i += 4) t.push_back(make_int4(TASK_U4, i, jj, q));
        if (group >= 3)
          for (; i + 2 < nt; i += 3) t.push_back(make_int4(TASK_U3, i, jj, q));
        for (; i + 1 < nt; i += 2) t.push_back(make_int4(TASK_U2, i, jj, q));
        if (i < nt) t.push_back(make_int4(TASK_U, i, jj, q));
      }
    if (inverse) {
      // X = inv(L): row k finished, then column q's contributions to the rows
      // below (pairs of rows)
      for (int j = 0; j < k; ++j) t.push_back(make_int4(TASK_XZ, k, j, 0));
      for (int j = 0; j <= q; ++j)
        for (int i = k + 1; i < nt; i += 2) t.push_back(make_int4(TASK_XG, i, j, q));
    }
  }
  return t;
}

int get_task_table(int nt, int group, bool inv_tasks, bool inverse, const int4** out, int* count) {
  std::lock_guard<std::mutex> lk(g_task_mu);
  const int key = ((nt * 8 + group) * 2 + (inv_tasks ? 1 : 0)) * 2 + (inverse ? 1 : 0);
  auto it = g_task_tables.find(key);
  if (it != g_task_tables.end()) {
    *out = it->second.first;
    *count = it->second.second;
    return PBG_OK;
  }
  const std::vector<int4> t = df_task_list(nt, group, inv_tasks, inverse);
  int4* d = nullptr;
  if (!t.empty()) {
    if (cudaMalloc(&d, t.size() * sizeof(int4)) != cudaSuccess) {
      cudaGetLastError();
      return PBG_ERR_NOMEM;
    }
    PBG_CUDA_TRY(cudaMemcpy(d, t.data(), t.size() * sizeof(int4), cudaMemcpyHostToDevice));
  }
  g_task_tables[key] = std::make_pair(d, (int)t.size());
  *out = d;
  *count = (int)t.size();
  return PBG_OK;
}

template <typename T>
size_t df_smem_bytes() {
  // the chain, a LEAD task, or a grouped update (the tensor-core operands in
  // FP32, five tiles in FP64)
  return std::max({chain_smem_bytes<T>(), lead_smem_bytes<T>(),
                   sizeof(T) == 4 ? tc_worker_smem_bytes(2) : 5 * NB * LDA * sizeof(T)});
}

// tasks_override / spin_limit: only for the wait-expiry self-test.
// inv_tasks: inv(L_kk) goes to invdiag.  X (or null): also form X = inv(L)
// (off-diagonal tiles); ints then holds the X flags after the factorisation's.
template <typename T>
int launch_df(T* A, int n, int ld, int* info, void* invdiag, bool inv_tasks, int* ints, void* lp, unsigned* err,
              cudaStream_t st, const int4* tasks_override = nullptr, int ntasks_override = 0,
              long long spin_limit = SPIN_LIMIT, T* X = nullptr, double min_pivot = MIN_PIVOT) {
  const int nt = ld / NB;
  const int4* tasks = nullptr;
  int ntasks = 0;
  if (tasks_override) {
    tasks = tasks_override;
    ntasks = ntasks_override;
  } else {
    int rc = get_task_table(nt, sizeof(T) == 4 ? 4 : 2, inv_tasks || X, X != nullptr, &tasks, &ntasks);
    if (rc) return rc;
  }
  const size_t smem = df_smem_bytes<T>();
  static int max_blocks_per_sm = -1;
  static int num_sms = 0;
  if (max_blocks_per_sm < 0) {
    PBG_CUDA_TRY(cudaFuncSetAttribute(chol_df_kernel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)smem));
    int dev;
    PBG_CUDA_TRY(cudaGetDevice(&dev));
    PBG_CUDA_TRY(cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev));
    PBG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&max_blocks_per_sm, chol_df_kernel<T>,
                                                               THREADS, smem));
    if (max_blocks_per_sm < 1) {
      pbg_set_error_message("cholesky kernel does not fit on an SM");
      return PBG_ERR_CUDA;
    }
  }
  // one CTA per SM: the chain CTA has its SM to itself
  int grid = num_sms;
  if (grid > ntasks + 1) grid = ntasks + 1;  // the chain CTA plus the shared tasks
  PBG_CUDA_TRY(cudaMemsetAsync(ints, 0, (3 + (X ? 4 : 2) * (size_t)nt * nt) * sizeof(int), st));
  PBG_CUDA_TRY(cudaMemsetAsync(info, 0, sizeof(int), st));
  DFArgs args;
  args.A = A;
  args.ld = ld;
  args.n = n;
  args.nt = nt;
  args.ntasks = ntasks;
  args.tasks = tasks;
  args.ctl = ints;
  args.upd = ints + 3;
  args.fin = ints + 3 + nt * nt;
  args.X = X;
  args.xupd = ints + 3 + 2 * nt * nt;
  args.xfin = ints + 3 + 3 * nt * nt;
  args.info = info;
  args.invdiag = invdiag;
  args.lp = lp;
  args.err = err;
  args.spin_limit = spin_limit;
  args.min_pivot = min_pivot;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  PBG_CUDA_TRY(cudaLaunchKernelEx(&cfg, chol_df_kernel<T>, args));
  PBG_CHECK_LAUNCH();
  return PBG_OK;
}

}  // namespace

// Self-test of the bounded waits (no counterpart in the reference): factors a
// 192 x 192 SPD matrix with a task list from which the host drops the update
// LEAD(0), so the chain's wait for U(2,1,0) can never be satisfied.  The wait
// gives up after spin_limit polls; the launch must end with info = -1 and the
// barrier error bit, the device must stay usable, and a normal
// factorisation right after must succeed.  Returns PBG_OK when all of that
// holds; *info_out and *err_out receive what the aborted launch reported.
extern "C" __attribute__((visibility("default"))) int pbg_selftest_wait_expiry(long long spin_limit, int* info_out,
                                                                                unsigned* err_out) {
  using namespace pbg;
  const int n = 192, ld = 192, nt = 3;
  if (spin_limit < 1 || spin_limit > (1LL << 24)) return PBG_ERR_ARG;
  const int4* full = nullptr;
  int nfull = 0;
  int rc = get_task_table(nt, 2, false, false, &full, &nfull);
  if (rc) return rc;
  std::vector<int4> tasks(nfull);
  PBG_CUDA_TRY(cudaMemcpy(tasks.data(), full, nfull * sizeof(int4), cudaMemcpyDeviceToHost));
  const auto dropped = std::remove_if(tasks.begin(), tasks.end(), [](const int4& t) {
    return t.x == TASK_LEAD && t.w == 0;
  });
  if (dropped == tasks.end()) return PBG_ERR_STATE;
  tasks.erase(dropped, tasks.end());
  std::vector<double> h((size_t)ld * ld, 0.0);
  for (int i = 0; i < n; ++i) {
    h[(size_t)i * ld + i] = 4.0;
    if (i > 0) h[(size_t)i * ld + i - 1] = h[(size_t)(i - 1) * ld + i] = 1.0;
  }
  double *A = nullptr, *lp = nullptr;
  int4* dt = nullptr;
  int* ints = nullptr;
  const size_t nints = 3 + 2 * (size_t)nt * nt + 2;
  bool ok = cudaMalloc(&A, h.size() * sizeof(double)) == cudaSuccess &&
            cudaMalloc(&lp, (size_t)nt * NB * NB * sizeof(double)) == cudaSuccess &&
            cudaMalloc(&dt, std::max<size_t>(tasks.size(), 1) * sizeof(int4)) == cudaSuccess &&
            cudaMalloc(&ints, nints * sizeof(int)) == cudaSuccess;
  int result = PBG_OK;
  if (!ok) {
    cudaGetLastError();
    result = PBG_ERR_NOMEM;
  } else {
    int* info = ints + nints - 2;
    unsigned* err = reinterpret_cast<unsigned*>(ints + nints - 1);
    int hinfo = 0;
    unsigned herr = 0;
    cudaMemcpy(A, h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice);
    cudaMemcpy(dt, tasks.data(), tasks.size() * sizeof(int4), cudaMemcpyHostToDevice);
    cudaMemset(err, 0, sizeof(unsigned));
    result = launch_df<double>(A, n, ld, info, nullptr, false, ints, lp, err, 0, dt, (int)tasks.size(), spin_limit);
    if (result == PBG_OK && cudaDeviceSynchronize() != cudaSuccess) result = PBG_ERR_CUDA;
    if (result == PBG_OK) {
      cudaMemcpy(&hinfo, info, sizeof(int), cudaMemcpyDeviceToHost);
      cudaMemcpy(&herr, err, sizeof(unsigned), cudaMemcpyDeviceToHost);
      if (info_out) *info_out = hinfo;
      if (err_out) *err_out = herr;
      if (hinfo != -1 || !(herr & PBG_DEV_ERR_BARRIER)) result = PBG_ERR_STATE;
    }
    if (result == PBG_OK) {
      // the context is still usable: the full task list factors the matrix
      cudaMemcpy(A, h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice);
      cudaMemset(err, 0, sizeof(unsigned));
      result = launch_df<double>(A, n, ld, info, nullptr, false, ints, lp, err, 0);
      if (result == PBG_OK && cudaDeviceSynchronize() != cudaSuccess) result = PBG_ERR_CUDA;
      if (result == PBG_OK) {
        cudaMemcpy(&hinfo, info, sizeof(int), cudaMemcpyDeviceToHost);
        if (hinfo != 0) result = PBG_ERR_STATE;
      }
    }
  }
  if (A) cudaFree(A);
  if (lp) cudaFree(lp);
  if (dt) cudaFree(dt);
  if (ints) cudaFree(ints);
  if (result != PBG_OK && result != PBG_ERR_CUDA)
    pbg_set_error_message("wait-expiry self-test: the aborted launch or the follow-up factorisation misbehaved");
  return result;
}

#ifdef PBG_TASK_TRACE
extern "C" __attribute__((visibility("default"))) int pbg_task_trace(long long* host, int ntasks) {
  PBG_CUDA_TRY(cudaMemcpyFromSymbol(host, g_task_trace, sizeof(long long) * 4 * ntasks));
  return PBG_OK;
}
extern "C" __attribute__((visibility("default"))) int pbg_ll_profile(long long* host, int ctas) {
  PBG_CUDA_TRY(cudaMemcpyFromSymbol(host, g_ll_prof, sizeof(long long) * 16 * ctas));
  return PBG_OK;
}
extern "C" __attribute__((visibility("default"))) int pbg_chain_trace(long long* host, int nt) {
  PBG_CUDA_TRY(cudaMemcpyFromSymbol(host, g_chain_trace, sizeof(long long) * 8 * nt));
  return PBG_OK;
}
#endif

// Scratch of one factorisation: task counter, abort flag, per-tile flags,
// error word; from the next 256-byte boundary the solve blocks.
static size_t df_flag_bytes(int nt) { return ((3 + 4 * (size_t)nt * nt + 1) * sizeof(int) + 255) / 256 * 256; }
size_t df_work_bytes(int ld) {
  const int nt = ld / NB;
  return df_flag_bytes(nt) + (size_t)nt * NB * NB * sizeof(double);
}

// Factors A in place; with want_inv (or X) the inverse of every diagonal
// factor tile goes to invdiag (nt x 64 x 64 row-major tiles, precision of A:
// the SPD inverse and the triangular solve of the midpoint scheme use them).
// A, invdiag and work start on 16-byte boundaries.
int launch_cholesky_df(void* A, int n, int ld, int precision, int* info, void* invdiag, bool want_inv, void* work,
                       cudaStream_t st, void* X) {
  const int nt = ld / NB;
  if (reinterpret_cast<uintptr_t>(A) % 16 != 0 || reinterpret_cast<uintptr_t>(invdiag) % 16 != 0 ||
      reinterpret_cast<uintptr_t>(work) % 16 != 0) {
    pbg_set_error_message("cholesky: the matrix and its workspace must start on 16-byte boundaries");
    return PBG_ERR_ARG;
  }
  int* ints = static_cast<int*>(work);
  unsigned* err = reinterpret_cast<unsigned*>(ints + 3 + 4 * (size_t)nt * nt);
  void* lp = static_cast<unsigned char*>(work) + df_flag_bytes(nt);
  if (precision == PBG_PREC_FP64)
    return launch_df<double>((double*)A, n, ld, info, invdiag, want_inv, ints, lp, err, st, nullptr, 0,
                                     SPIN_LIMIT, (double*)X);
  // PBG_PREC_MIXED reports a pivot below the smallest normal float as non-positive
  return launch_df<float>((float*)A, n, ld, info, invdiag, want_inv, ints, lp, err, st, nullptr, 0, SPIN_LIMIT, (float*)X,
                          precision == PBG_PREC_MIXED_FP64_DIAG ? MIN_PIVOT : 1.17549435e-38);
}


// One replica's tasks in its own order, cut into segments: segment 0 =
// F(0), S(i, 0); then for each k three segments F(k+1) | U(i, j, k) (j >= k+2)
// | S(i, k+1) (i >= k+2).  F(k+1) and S(., k+1) apply their update with panel
// k themselves.  seg_start holds 1 + 3(nt-1) segment starts and the end.
// A batch merges the replicas' lists segment by segment in one of several orders
// (merge_segments in batch.cu) that all keep each replica's own; the default
// spreads every replica's evenly over the longest one's.  With replicas of one size that
// is every replica's F(k+1), then every replica's U(., ., k), then every replica's
// S(., k+1), so the solves are fetched after their factorisations had the
// whole update phase to finish.  F(k+1) and U(., ., k) depend only on block
// k-1; S(., k+1) on F(k+1) and block k-1: every task depends only on earlier
// tasks.  The tasks carry replica tag 0; the merge writes the replica index.
//
// The mixed-precision lists are left-looking (chol_batch_ll_kernel), two
// segments per column j: LL_DIAG for rows (j, j + 1) and LL_UPDATE for the
// row pairs (j + 2, j + 3), (j + 4, j + 5), ...; then LL_SOLVE for the same
// pairs.  Column j + 1's tasks need column j's solves and come after them; among
// replicas of one size, every one's solves of column j come after every one's
// updates of it, so F(j) has had that phase to finish.
void cholesky_replica_tasks(int nt, int precision, std::vector<int4>& tasks, std::vector<int>& seg_start) {
  tasks.clear();
  seg_start.clear();
  if (nt < 1) return;
  if (precision != PBG_PREC_FP64) {
    for (int j = 0; j < nt; ++j) {
      seg_start.push_back((int)tasks.size());
      tasks.push_back(make_int4(LL_DIAG, j, j, 0));
      for (int i = j + 2; i < nt; i += 2) tasks.push_back(make_int4(LL_UPDATE, i, j, 0));
      seg_start.push_back((int)tasks.size());
      for (int i = j + 2; i < nt; i += 2) tasks.push_back(make_int4(LL_SOLVE, i, j, 0));
    }
    seg_start.push_back((int)tasks.size());
    return;
  }
  seg_start.push_back(0);
  tasks.push_back(make_int4(TASK_F, 0, 0, 0));
  for (int i = 1; i < nt; ++i) tasks.push_back(make_int4(TASK_S, i, 0, 0));
  for (int k = 0; k + 1 < nt; ++k) {
    seg_start.push_back((int)tasks.size());
    tasks.push_back(make_int4(TASK_F, k + 1, k + 1, k + 1));
    seg_start.push_back((int)tasks.size());
    for (int jj = k + 2; jj < nt; ++jj) {  // rows paired, as in the single-matrix list
      int i = jj;
      for (; i + 1 < nt; i += 2) tasks.push_back(make_int4(TASK_U2, i, jj, k));
      if (i < nt) tasks.push_back(make_int4(TASK_U, i, jj, k));
    }
    seg_start.push_back((int)tasks.size());
    for (int i = k + 2; i < nt; ++i) tasks.push_back(make_int4(TASK_S, i, k + 1, k + 1));
  }
  seg_start.push_back((int)tasks.size());
}

// Resident CTAs per SM of the batched factorisation kernel of this
// precision (the occupancy query, once per precision) and the SM count.
int cholesky_batch_residency(int precision, int* ctas_per_sm, int* sms) {
  const bool f64 = precision == PBG_PREC_FP64;
  const size_t smem = f64 ? batch_smem_bytes() : ll_smem_bytes();
  static int blocks_per_sm[2] = {-1, -1};
  static int num_sms = 0;
  int& bps = blocks_per_sm[f64 ? 0 : 1];
  if (bps < 0) {
    int dev;
    PBG_CUDA_TRY(cudaGetDevice(&dev));
    PBG_CUDA_TRY(cudaDeviceGetAttribute(&num_sms, cudaDevAttrMultiProcessorCount, dev));
    int b = 0;
    if (f64) {
      PBG_CUDA_TRY(cudaFuncSetAttribute(chol_batch_kernel<double>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      PBG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, chol_batch_kernel<double>, THREADS, smem));
    } else {
      PBG_CUDA_TRY(cudaFuncSetAttribute(chol_batch_ll_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
      PBG_CUDA_TRY(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, chol_batch_ll_kernel, THREADS, smem));
    }
    if (b < 1) {
      pbg_set_error_message("batched cholesky kernel does not fit on an SM");
      return PBG_ERR_CUDA;
    }
    bps = b;
  }
  *ctas_per_sm = bps;
  *sms = num_sms;
  return PBG_OK;
}

int launch_cholesky_batch(int precision, const CholRep* reps, const int4* tasks, int ntasks, int* ctl,
                          int ctas_per_sm, cudaStream_t st) {
  if (ntasks <= 0) return PBG_OK;
  const bool f64 = precision == PBG_PREC_FP64;
  const size_t smem = f64 ? batch_smem_bytes() : ll_smem_bytes();
  int bps = 0, num_sms = 0;
  int rc = cholesky_batch_residency(precision, &bps, &num_sms);
  if (rc) return rc;
  int grid = num_sms * (ctas_per_sm > 0 ? std::min(ctas_per_sm, bps) : bps);
  if (grid > ntasks) grid = ntasks;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(THREADS);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  if (f64) PBG_CUDA_TRY(cudaLaunchKernelEx(&cfg, chol_batch_kernel<double>, reps, tasks, ntasks, ctl));
  else {
    const cudaError_t e = cudaLaunchKernelEx(&cfg, chol_batch_ll_kernel, reps, tasks, ntasks, ctl);
    if (e == cudaErrorCooperativeLaunchTooLarge) {
      // say what the asked-for residency would need
      cudaGetLastError();
      size_t avail = 0;
      cudaFuncAttributes fa = {};
      cudaOccupancyAvailableDynamicSMemPerBlock(&avail, chol_batch_ll_kernel, grid / num_sms, THREADS);
      cudaFuncGetAttributes(&fa, chol_batch_ll_kernel);
      cudaGetLastError();
      pbg_set_error_message(
          "batched factorisation: %d CTAs per SM do not fit (%zu bytes of dynamic shared memory per CTA, %zu "
          "available at that residency; %d registers per thread, %zu bytes static shared memory)",
          grid / num_sms, smem, avail, fa.numRegs, fa.sharedSizeBytes);
      return PBG_ERR_CUDA;
    }
    PBG_CUDA_TRY(e);
  }
  PBG_CHECK_LAUNCH();
  return PBG_OK;
}


// ---------------------------------------------------------------- SPD inverse on the tensor cores
// inv(A) = X^T X with A = L L^T and X = inv(L): the data-flow factorisation
// forms X's off-diagonal tiles in the same launch (XG / XZ tasks, on TileMMA: FP64
// DMMA, or 3xTF32 split products with FP32 accumulation), then X^T X is formed.
// FP64 (lauum_kernel): one CTA per lower tile, X's diagonal tiles read from invdiag.
// FP32 (sym_tc_kernel, tcgen05): pairs of tiles, the diagonal ones copied into X
// first.  Used by the SPD inverse (cholesky.cu) and by the lubricated steps, which
// also read the factor of kBT inv(R) off X (launch_reversed_factor_tiles).
//
// Mixed workspace (tc_inverse_work_bytes): [inv(L_kk) tiles][data-flow
// scratch][X: ld x ld][F: ld x ld], F the matrix to factor (in place).

namespace {

// X_kk = inv(L_kk), upper triangle zero (one CTA per diagonal tile).
template <typename T>
__global__ void __launch_bounds__(THREADS) trtri_diag_kernel(const T* __restrict__ invdiag, T* X, int ld) {
  const int k = blockIdx.x;
  T* g = X + (size_t)k * NB * ld + (size_t)k * NB;
  const T* inv = invdiag + (size_t)k * NB * NB;
  T v[TILE_PER_THREAD];
#pragma unroll
  for (int q = 0; q < TILE_PER_THREAD; ++q) v[q] = inv[threadIdx.x + q * THREADS];
#pragma unroll
  for (int q = 0; q < TILE_PER_THREAD; ++q) {
    const int e = threadIdx.x + q * THREADS, r = e >> 6, c = e & 63;
    g[(size_t)r * ld + c] = c <= r ? v[q] : T(0);
  }
}

// out_IJ = scale (X^T X)_IJ = scale sum_{k >= I} X_kI^T X_kJ for the lower
// tile (I, J), written to (I, J) and (J, I), with `reversed` every element (r, c) to
// (ld-1-r, ld-1-c); FP64.  Off-diagonal tiles come from
// X, the diagonal ones from invdiag.  Bound by the FP64 tensor pipe (2.1 us per
// 64^3 product and SM): the tiles are used as they lie in memory (sub_rows),
// two K-steps in flight by cp.async; the CTAs with the longest K range start
// first.  Order 1536: 118 us with transposing copies through registers, 69 now.
constexpr size_t lauum_smem_bytes() { return 4 * NB * LDA * sizeof(double); }
__global__ void __launch_bounds__(THREADS) lauum_kernel(const double* __restrict__ X, const double* __restrict__ invdiag,
                                                        int ld, int nt, double scale, int reversed,
                                                        double* __restrict__ out) {
  extern __shared__ __align__(16) unsigned char smem[];
  double* st = reinterpret_cast<double*>(smem);  // [2][2][64][LDA]
  const int b = blockIdx.x;
  int I = (int)((sqrt(8.0 * b + 1.0) - 1.0) * 0.5);
  while ((I + 1) * (I + 2) / 2 <= b) ++I;
  while (I * (I + 1) / 2 > b) --I;
  const int J = b - I * (I + 1) / 2;
  auto fetch = [&](int k, double* s) {
    auto one = [&](int c, double* d) {
      if (k == c) stage_async(invdiag + (size_t)k * NB * NB, NB, d, LDA);
      else stage_async(X + (size_t)k * NB * ld + (size_t)c * NB, ld, d, LDA);
    };
    one(I, s);
    if (J != I) one(J, s + NB * LDA);
    cp_async_commit();
  };
  double acc[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) acc[e] = 0.0;
  fetch(I, st);
  for (int k = I; k < nt; ++k) {
    double* s = st + ((k - I) & 1) * 2 * NB * LDA;
    if (k + 1 < nt) {
      fetch(k + 1, st + ((k - I + 1) & 1) * 2 * NB * LDA);
      cp_async_wait_group<1>();
    } else {
      cp_async_wait_group<0>();
    }
    __syncthreads();
    TileMMA<double>::sub_rows<true>(s, J != I ? s + NB * LDA : s, acc);
    __syncthreads();
  }
#pragma unroll
  for (int rs = 0; rs < 2; ++rs)
#pragma unroll
    for (int cs = 0; cs < 8; ++cs) {
      const double v = -acc[TileMMA<double>::idx(rs, cs)] * scale;
      int r = I * NB + acc_row(rs), c = J * NB + acc_col(cs);
      if (reversed) {
        r = ld - 1 - r;
        c = ld - 1 - c;
      }
      out[(size_t)r * ld + c] = v;
      if (I != J) out[(size_t)c * ld + r] = v;  // a diagonal tile writes each element once
    }
}

// B[i][j] = scale X[ld-1-j][ld-1-i] for the lower triangle of B (32 x 32
// tiles through smem; tiles above the diagonal are not written).
template <typename T>
__global__ void reversed_transpose_kernel(const T* __restrict__ X, const T* __restrict__ Xdiag, int ld, T scale,
                                          T* __restrict__ B) {
  __shared__ T t[32][33];
  const int bi = blockIdx.y, bj = blockIdx.x;
  if (bj > bi) return;
  const int x0r = ld - 32 * (bj + 1), x0c = ld - 32 * (bi + 1);
  // a block within a diagonal tile of X
  const bool diag = Xdiag && x0r / NB == x0c / NB;
  const T* src = diag ? Xdiag + (size_t)(x0r / NB) * NB * NB + (x0r % NB) * NB + x0c % NB : X + (size_t)x0r * ld + x0c;
  const size_t lds = diag ? NB : ld;
  for (int r = threadIdx.y; r < 32; r += blockDim.y) t[r][threadIdx.x] = src[r * lds + threadIdx.x];
  __syncthreads();
  for (int rr = threadIdx.y; rr < 32; rr += blockDim.y)
    B[(size_t)(bi * 32 + rr) * ld + bj * 32 + threadIdx.x] = scale * t[31 - threadIdx.x][31 - rr];
}

// inv(B_II) for B = s J G^{-T} J (G lower, order ld, J the reversal of all ld
// indices): (1/s) J G_I'I'^T J with I' = nt-1-I, from the lower triangle of
// G's diagonal tile.
template <typename T>
__global__ void b_invdiag_kernel(const T* __restrict__ G, int ld, int nt, T inv_scale, T* __restrict__ invdiag) {
  const int I = blockIdx.x, Ip = nt - 1 - I;
  const T* g = G + (size_t)Ip * NB * ld + (size_t)Ip * NB;
  T* o = invdiag + (size_t)I * NB * NB;
  for (int e = threadIdx.x; e < NB * NB; e += blockDim.x) {
    const int r = e >> 6, c = e & 63;
    o[e] = r >= c ? inv_scale * g[(size_t)(NB - 1 - c) * ld + (NB - 1 - r)] : T(0);
  }
}

// ---------------------------------------------------------------- X^T X on tcgen05 (FP32)
// out = scale X^T X for the lower-triangular FP32 X (the SPD inverse's
// symmetric product in the mixed lubricated path): a CTA forms the output
// tiles (I, J) and (I + 1, J) (only (I, J) when I + 1 = nt) as one M = 128,
// N = 64 product over the K range k = I .. nt-1,
//   [X_kI^T; X_{k,I+1}^T] X_kJ    (X_{I,I+1} above the diagonal taken as 0),
// in 3xTF32 on the tensor cores.  Per K-step the three tiles arrive row-major
// by cp.async two K-steps ahead (raw stages); the transposition is done by
// the split into the K-major hi / lo operands (column m of X_kI becomes row
// m of A).  The accumulator restarts in TMEM every SYM_CHUNK K-steps and the
// chunk sums are added in FP32 (as in the left-looking batch kernel).
// Each element is written once: (r, c) and, off the diagonal tiles, (c, r);
// with `reversed`, (ld-1-r, ld-1-c) instead.
constexpr int SYM_CHUNK = 4;
constexpr uint32_t LL_RAW_BYTES = 3 * NB * NB * sizeof(float);  // one raw stage: X_kI, X_{k,I+1}, X_kJ
constexpr uint32_t SYM_SHARED_OFFSET = LL_OPERAND_BYTES + 2 * LL_RAW_BYTES;
constexpr size_t sym_smem_bytes() { return SYM_SHARED_OFFSET + 16; }  // mbarrier, TMEM address
static_assert(sym_smem_bytes() <= 227 * 1024, "the symmetric product does not fit an SM");

// Output tile pairs: for each J, I = J, J + 2, J + 4, ...
__host__ __device__ inline int sym_pairs(int nt) {
  int n = 0;
  for (int J = 0; J < nt; ++J) n += (nt - J + 1) / 2;
  return n;
}

// The K-step k tiles: X_kI, X_{k,I+1} (when it is a lower tile), X_kJ.
__device__ __forceinline__ void sym_fetch_step(const float* X, int ld, int I, int J, int k, bool two, float* raw) {
  const float* row = X + (size_t)k * NB * ld;
  ll_fetch_tile(row + (size_t)I * NB, ld, raw);
  if (two && k >= I + 1) ll_fetch_tile(row + (size_t)(I + 1) * NB, ld, raw + NB * NB);
  ll_fetch_tile(row + (size_t)J * NB, ld, raw + 2 * NB * NB);
  cp_async_commit();
}

__global__ void __launch_bounds__(THREADS, 1) sym_tc_kernel(const float* __restrict__ X, int ld, int nt, float scale,
                                                           int reversed, float* __restrict__ out, int* info) {
  extern __shared__ __align__(1024) unsigned char sym_smem[];
  unsigned char* base = sym_smem;
  const int tid = threadIdx.x;
  if (tc::smem_u32(base) & 1023u) {  // the operands need a 1024-byte aligned start
    if (tid == 0) atomicCAS(info, 0, -1);
    return;
  }
  uint64_t* mbar = reinterpret_cast<uint64_t*>(base + SYM_SHARED_OFFSET);
  uint32_t* s_tmem = reinterpret_cast<uint32_t*>(base + SYM_SHARED_OFFSET + 8);
  int b = blockIdx.x, J = 0;
  for (; J < nt; ++J) {
    const int cnt = (nt - J + 1) / 2;
    if (b < cnt) break;
    b -= cnt;
  }
  const int I = J + 2 * b;
  const bool two = I + 1 < nt;
  if (tid == 0) tc::mbar_init(mbar, 1);
  if (tid < 32) tc::tmem_alloc(s_tmem, 64);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *s_tmem;
  uint32_t phase = 0;
  unsigned char* Ahi = base;
  unsigned char* Alo = Ahi + LL_A_BYTES;
  unsigned char* Bhi = Alo + LL_A_BYTES;
  unsigned char* Blo = Bhi + LL_B_BYTES;
  float* raw[2] = {reinterpret_cast<float*>(base + LL_OPERAND_BYTES),
                   reinterpret_cast<float*>(base + LL_OPERAND_BYTES + LL_RAW_BYTES)};
  const int warp = tid >> 5, lane = tid & 31, q = warp & 3, g = warp >> 2;
  const uint32_t tacc = tmem + ((uint32_t)(32 * q) << 16) + 32 * g;
  // this thread's operand rows: A row ma (chunks 2e + tid / 128), B row nb
  // (chunks 4e + tid / 64)
  const int ma = tid & 127, nb = tid & 63;
  sym_fetch_step(X, ld, I, J, I, two, raw[0]);
  if (I + 1 < nt) sym_fetch_step(X, ld, I, J, I + 1, two, raw[1]);
  float racc[32];
#pragma unroll
  for (int u = 0; u < 32; ++u) racc[u] = 0.0f;
  bool ok = true;
  for (int k = I; k < nt; ++k) {
    const int s = k - I;
    float* st = raw[s & 1];
    if (k + 1 < nt) cp_async_wait_group<1>();
    else cp_async_wait_group<0>();
    __syncthreads();  // every thread's copies of this K-step are in
    if (s > 0) {      // the products of the previous K-step have read the operands
      if (!tc::mbar_wait(mbar, phase, SPIN_LIMIT)) ok = false;
      phase ^= 1;
      tc::fence_after_sync();
      if (s % SYM_CHUNK == 0) {
        float v[32];
        tc::tmem_ld32(tacc, v);
#pragma unroll
        for (int u = 0; u < 32; ++u) racc[u] += v[u];
        tc::fence_before_sync();
      }
    }
    // A row ma: column ma of X_kI (ma < 64) or of X_{k,I+1} (zero for k = I
    // or beyond the last tile); chunk c holds K = 4c .. 4c+3 (rows of X)
    {
      const bool zero = ma >= 64 && !(two && k >= I + 1);
      const float* src = st + (ma < 64 ? 0 : NB * NB) + (ma & 63);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        const int c = 2 * e + (tid >> 7);
        float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (!zero) x = make_float4(src[(4 * c) * NB], src[(4 * c + 1) * NB], src[(4 * c + 2) * NB], src[(4 * c + 3) * NB]);
        tc::store_split_chunk(x, tc::sw128_offset(128, ma, c), Ahi, Alo);
      }
      const float* srcb = st + 2 * NB * NB + nb;
#pragma unroll
      for (int e = 0; e < 4; ++e) {
        const int c = 4 * e + (tid >> 6);
        const float4 x =
            make_float4(srcb[(4 * c) * NB], srcb[(4 * c + 1) * NB], srcb[(4 * c + 2) * NB], srcb[(4 * c + 3) * NB]);
        tc::store_split_chunk(x, tc::sw128_offset(64, nb, c), Bhi, Blo);
      }
    }
    tc::fence_proxy_smem();
    __syncthreads();  // operands written; every thread is past its reads of this stage
    if (tid == 0) {
      tc::fence_after_sync();
      tc::issue_product(tmem, tc::smem_u32(Ahi), tc::smem_u32(Alo), tc::smem_u32(Bhi), tc::smem_u32(Blo),
                        s % SYM_CHUNK != 0 ? 1u : 0u);
      tc::mma_commit(mbar);
    }
    if (k + 2 < nt) sym_fetch_step(X, ld, I, J, k + 2, two, st);
  }
  if (!tc::mbar_wait(mbar, phase, SPIN_LIMIT)) ok = false;
  ok = __syncthreads_and(ok) != 0;
  tc::fence_after_sync();
  {
    float v[32];
    tc::tmem_ld32(tacc, v);
#pragma unroll
    for (int u = 0; u < 32; ++u) racc[u] += v[u];
  }
  const int m = 32 * q + lane, t = m >> 6;
  if (ok && (t == 0 || two)) {
    const int It = I + t;
    const int r0 = It * NB + (m & 63), c0 = J * NB + 32 * g;
#pragma unroll
    for (int u = 0; u < 32; ++u) {
      const float v = racc[u] * scale;
      int r = r0, c = c0 + u;
      if (reversed) {
        r = ld - 1 - r;
        c = ld - 1 - c;
      }
      out[(size_t)r * ld + c] = v;
      if (It != J) out[(size_t)c * ld + r] = v;
    }
  }
  if (!ok && tid == 0) atomicCAS(info, 0, -1);
  tc::fence_before_sync();
  __syncthreads();
  if (tid < 32) tc::tmem_dealloc(tmem, 64);
}

}  // namespace

int launch_trtri_diag(const float* invdiag, float* X, int ld, cudaStream_t st) {
  if (ld % NB != 0 || ld <= 0) return PBG_ERR_ARG;
  trtri_diag_kernel<float><<<ld / NB, THREADS, 0, st>>>(invdiag, X, ld);
  PBG_CHECK_LAUNCH();
  return PBG_OK;
}

int launch_lauum(const double* X, const double* invdiag, int ld, double scale, bool reversed, double* out,
                 cudaStream_t st) {
  if (ld % NB != 0 || ld <= 0) return PBG_ERR_ARG;
  const int nt = ld / NB;
  PBG_CUDA_TRY(cudaFuncSetAttribute(lauum_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)lauum_smem_bytes()));
  lauum_kernel<<<nt * (nt + 1) / 2, THREADS, lauum_smem_bytes(), st>>>(X, invdiag, ld, nt, scale, reversed ? 1 : 0,
                                                                    out);
  PBG_CHECK_LAUNCH();
  return PBG_OK;
}

// The data-flow scratch rounded up to 256 bytes, so X and F start aligned
// whatever the tile count (the scratch itself is 80 + 8 nt^2 bytes).
static size_t tc_scratch_bytes(int ld) { return (df_work_bytes(ld) + 255) / 256 * 256; }

size_t tc_inverse_work_bytes(int ld) {
  const size_t nt = ld / NB;
  return nt * NB * NB * sizeof(float) + tc_scratch_bytes(ld) + 2 * (size_t)ld * ld * sizeof(float);
}

TcInverseWork tc_inverse_work(void* work, int ld) {
  const size_t nt = ld / NB;
  unsigned char* p = static_cast<unsigned char*>(work);
  TcInverseWork w;
  w.invdiag = reinterpret_cast<float*>(p);
  w.scratch = p + nt * NB * NB * sizeof(float);
  w.X = reinterpret_cast<float*>(static_cast<unsigned char*>(w.scratch) + tc_scratch_bytes(ld));
  w.F = w.X + (size_t)ld * ld;
  return w;
}

int tc_factor_invert(int ld, int* info, void* work, cudaStream_t st) {
  if (ld % NB != 0 || ld <= 0) return PBG_ERR_ARG;
  const TcInverseWork w = tc_inverse_work(work, ld);
  if (reinterpret_cast<uintptr_t>(w.X) % 16 != 0) {
    pbg_set_error_message("tensor-core inverse: misaligned workspace");
    return PBG_ERR_ARG;
  }
  // the factorisation forms X's off-diagonal tiles in the same launch
  int rc = launch_cholesky_df(w.F, ld, ld, PBG_PREC_MIXED, info, w.invdiag, true, w.scratch, st, w.X);
  if (rc != PBG_OK) return rc;
  return launch_trtri_diag(w.invdiag, w.X, ld, st);
}

int tc_lauum(const float* X, int ld, float scale, bool reversed, float* out, int* info, cudaStream_t st) {
  if (ld % NB != 0 || ld <= 0) return PBG_ERR_ARG;
  const int nt = ld / NB;
  PBG_CUDA_TRY(cudaFuncSetAttribute(sym_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)sym_smem_bytes()));
  sym_tc_kernel<<<sym_pairs(nt), THREADS, sym_smem_bytes(), st>>>(X, ld, nt, scale, reversed ? 1 : 0, out, info);
  PBG_CHECK_LAUNCH();
  return PBG_OK;
}

template <typename T>
int launch_reversed_factor_tiles(const T* X, const T* Xdiag, const T* G, int ld, double s, T* B, T* invdiag,
                                 cudaStream_t st) {
  // first what reads G, which B may overwrite
  b_invdiag_kernel<T><<<ld / NB, THREADS, 0, st>>>(G, ld, ld / NB, (T)(1.0 / s), invdiag);
  PBG_CHECK_LAUNCH();
  reversed_transpose_kernel<T><<<dim3(ld / 32, ld / 32), dim3(32, 8), 0, st>>>(X, Xdiag, ld, (T)s, B);
  PBG_CHECK_LAUNCH();
  return PBG_OK;
}
template int launch_reversed_factor_tiles<double>(const double*, const double*, const double*, int, double, double*,
                                                  double*, cudaStream_t);

int tc_reversed_factor(const float* X, const float* G, int ld, double s, float* B, float* invdiag,
                       cudaStream_t st) {
  return launch_reversed_factor_tiles<float>(X, nullptr, G, ld, s, B, invdiag, st);
}

}  // namespace pbg
