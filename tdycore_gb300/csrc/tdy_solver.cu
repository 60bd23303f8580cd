// tdy_solver.cu -- device-resident backward-Euler Newton solve of one or many
// independent instances (the blocks of TDySetExtrudedMeshes) in one handle.
//
// Each Newton iteration evaluates the FP64 residual and the Jacobian with the
// handle's kernels for every instance at once, takes per-instance residual
// norms (the only values the host reads), and solves J y = F with
// right-preconditioned BiCGStab:
//   * Krylov vectors and the Jacobian copy in FP32 (default) or FP64; the
//     residual, the Newton update x -= y and the convergence test stay FP64;
//   * every instance keeps its own BiCGStab scalars and stops on its own
//     tolerance (device-side masks, no host round trip per iteration);
//   * preconditioner: exact solves of the vertical lines (the tridiagonal
//     coupling of each column of an extruded block, Thomas algorithm, one
//     thread per column), which carries the stiff vertical coupling of thin
//     layers;
//   * a solve is one launch: a cluster of CTAs per instance, or one
//     cooperative grid for all cells (bicgstab_block_kernel,
//     bicgstab_grid_kernel), whose loop ends with its last instance;
//   * the sparse matrix-vector product's threads per row (1, 2, 4 or 8) are
//     picked by timing the candidates on the first solve that uses them.
// No reference counterpart: the reference hands F and J to PETSc's SNES/KSP.
#include <cooperative_groups.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <climits>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <tuple>
#include <utility>
#include <vector>

#include "tdy_arena.h"
#include "tdy_device.h"

namespace tdy {

namespace {

#define SCUDA(call)                                                                             \
  do {                                                                                          \
    cudaError_t e_ = (call);                                                                    \
    if (e_ != cudaSuccess)                                                                      \
      return set_error(TDY_ERR_GPU, "%s failed: %s (%s:%d)", #call, cudaGetErrorString(e_), __FILE__, __LINE__); \
  } while (0)

inline unsigned nblk(long long n, int bs) { return (unsigned)((n + bs - 1) / bs); }

// per-instance scalars, [slot][nseg]
enum { S_RHO = 0, S_ALPHA, S_OMEGA, S_BETA, S_BNORM2, S_HALF, S_NSCAL };

// what the host reads of a set-up of clusters
struct ClusterCounts {
  unsigned long long both;  // clusters of 2..64 cells << 32 | cells in them
  unsigned long long lu;    // elements of their factors
  unsigned long long big;   // cells of larger clusters
  int settled;              // 0: the labels still changed in the last round
};

struct Krylov {
  bool ready = false;
  void *Jv = nullptr;                                  // matrix values (T)
  void *b = nullptr, *r = nullptr, *r0 = nullptr, *p = nullptr, *v = nullptr, *s = nullptr, *t = nullptr,
       *ph = nullptr, *sh = nullptr, *y = nullptr;     // vectors (T)
  void *la = nullptr, *lcp = nullptr, *linv = nullptr; // line factors (T)
  void *cinv = nullptr;                                // clusters: 1/diagonal of the other cells (T)
  void *sell = nullptr;                                // matrix values of the block schedule's instances (T)
  void *clu = nullptr;                                 // clusters: LU factors (T), grown on demand
  size_t clu_cap = 0;                                  // elements of clu
  int tpr = 0;  // spmv threads per row (autotuned)
  // instances of at most this many cells take the block schedule (-2: not
  // timed yet; the precisions differ in what fits shared memory)
  long long block_max_cells = -2;
};

}  // namespace

struct SolverState {
  int n = 0, nnz = 0, nseg = 0, nlines = 0;
  std::vector<int> h_seg_off;
  int *rowptr = nullptr, *colidx = nullptr, *seg_off = nullptr, *cell_seg = nullptr;
  int *line_off = nullptr, *line_cells = nullptr, *pos_d = nullptr, *pos_lo = nullptr, *pos_hi = nullptr;
  double *x = nullptr, *xb = nullptr, *F = nullptr, *J = nullptr, *norms = nullptr, *scal = nullptr, *lam = nullptr;
  int *trial = nullptr, *commit = nullptr;
  int *newt_active = nullptr, *lin_active = nullptr, *lin_its = nullptr;
  int nchunks = 0;
  int *chunk_off = nullptr, *seg_chunk = nullptr;  // chunks of the per-instance reductions
  double *part = nullptr;
  // the tile schedule's sums (accumulators and chunk sums), on its first use
  double *grid_acc = nullptr, *grid_part = nullptr;
  // what the host reads of a linear solve, in one copy: ||y||^2 and iterations
  // per instance, then the words of the tile schedule (GS_*; zeroed with lin_its)
  double *y2 = nullptr;
  unsigned *grid_sync = nullptr;
  std::vector<double> h_out;
  int *dpos = nullptr;  // position of each row's diagonal in the CSR values
  // strong-coupling clusters, rebuilt for every linear solve that uses them:
  // scratch of the set-up (cl_setup_kernel), label per cell, local index in
  // its cluster (-1: the cell
  // takes its diagonal), the members of the 2..64-cell clusters (cluster by
  // cluster, ascending cell index), their offsets and LU offsets, row orders
  unsigned char *cstrong = nullptr;
  int *ccnt = nullptr, *cid = nullptr;
  unsigned long long *ctotal = nullptr;
  unsigned *csync = nullptr;
  ClusterCounts *ccounts = nullptr;
  int *clab = nullptr, *cloc = nullptr, *cmem = nullptr, *coff = nullptr, *cperm = nullptr;
  long long *cluoff = nullptr;
  int ncl = 0;  // clusters of 2..64 cells in the current solve
  int ncl_cells = 0, ncl_big_cells = 0;  // cells in them; cells of clusters over 64 cells
  int precond_used = 0;
  Krylov k32, k64;
  // schedules of the line-preconditioned inner solve (block: a cluster per
  // instance; tile: one grid for all cells)
  int *inst_line_off = nullptr, *block_inst = nullptr, *block_mask = nullptr, *ticket = nullptr;
  std::vector<int> h_inst_line_off, h_order;  // h_order: instances by size, largest first
  // the block schedule's matrix layout (built on its first use): slices of 32
  // rows, entry k of the 32 rows side by side, column indices local to the
  // instance; only instances up to kBlockCap cells have slices
  int nslices = 0;
  std::vector<int> h_slice_off, h_slice_row;  // first slice per instance; first row per slice
  std::vector<long long> h_sell_off;          // first element per slice
  int *slice_off = nullptr, *slice_row = nullptr, *slice_end = nullptr;
  long long *sell_off = nullptr;
  uint16_t *sell_col = nullptr;
  // this solve's instances on the block schedule, class by class (CTAs per
  // instance 8, 4, 2, 1), each class largest first
  std::vector<int> h_block_list;
  cudaStream_t side[3] = {nullptr, nullptr, nullptr};  // the classes run side by side
  cudaEvent_t fork = nullptr, joined[3] = {nullptr, nullptr, nullptr};
  int device = 0;
  long long mask_for = -3;  // the split (block_max_cells) of block_mask
  int n_block = 0, n_tile = 0;
  std::vector<double> tune_ms;  // measured candidates of the last tuning (ms per linear solve)
  // phase timers on the solve's stream: evaluation, Jacobian cast and
  // preconditioner set-up, Krylov iterations (events of the current phase)
  cudaEvent_t tev[5] = {nullptr, nullptr, nullptr, nullptr, nullptr};
  // device memory: stream-ordered on the handle's stream (allocated there and
  // synchronised at init; freed there when the solver is destroyed, after
  // every solve has synchronised its stream)
  cudaStream_t st = nullptr;
  std::vector<void *> allocs;
  ~SolverState() {
    for (cudaEvent_t e : tev)
      if (e) cudaEventDestroy(e);
    // (joined into the solve's stream, which every solve synchronises)
    device_pool_release(device, nullptr, fork);
    for (int i = 0; i < 3; i++) device_pool_release(device, side[i], joined[i]);
    for (Krylov *k : {&k32, &k64})
      if (k->clu) dmem_free(k->clu, st);
    for (void *p : allocs) dmem_free(p, st);
  }
};

namespace {

template <class T>
int salloc(SolverState *s, T **p, size_t n) {
  int ierr = dmem_alloc((void **)p, std::max<size_t>(n, 1) * sizeof(T), s->st);
  if (ierr) return ierr;
  s->allocs.push_back(*p);
  return 0;
}
// (the host vector must stay alive until the stream is synchronised)
template <class T>
int sup(SolverState *s, T **p, const std::vector<T> &h) {
  int ierr = salloc(s, p, h.size());
  if (ierr) return ierr;
  if (h.empty()) return 0;
  cudaError_t e = cudaMemcpyAsync(*p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice, s->st);
  if (e != cudaSuccess) return set_error(TDY_ERR_GPU, "cudaMemcpyAsync: %s", cudaGetErrorString(e));
  return 0;
}

// ---------------------------------------------------------------------------
// kernels
//
// Two schedules run the BiCGStab iterations: "tile" (one grid works through
// all cells of the batch, instances masked as they converge, see
// bicgstab_grid_kernel) and "block" (a cluster per instance runs its whole
// Krylov loop, see bicgstab_block_kernel).  Both perform every floating-point operation of an
// instance in the same order with explicit roundings (the element operations
// below, the chunked reductions, the per-row lane split of the product), so
// an instance gets the same bits from either schedule.

__device__ __forceinline__ float e_fma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double e_fma(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ float e_mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double e_mul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float e_add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double e_add(double a, double b) { return __dadd_rn(a, b); }

// p = r + beta (p - omega v)
template <class T>
__device__ __forceinline__ T op_p(T r, T p, T v, T beta, T omega) {
  return e_fma(beta, e_fma(-omega, v, p), r);
}
// y += alpha ph (+ omega sh)
template <class T>
__device__ __forceinline__ T op_y(T y, T ph, T alpha) {
  return e_fma(alpha, ph, y);
}
template <class T>
__device__ __forceinline__ T op_y2(T y, T ph, T sh, T alpha, T omega) {
  return e_fma(omega, sh, e_fma(alpha, ph, y));
}
// the per-cell terms of the chunked dot products, in FP64
template <class TA, class TB>
__device__ __forceinline__ double op_dot(double acc, TA a, TB b) {
  return __fma_rn((double)a, (double)b, acc);
}

template <class T>
__global__ void cast_kernel(long long n, const double *a, T *b) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) b[i] = (T)a[i];
}

// the cells of the flagged instances: b = (float)a
__global__ void cast_masked_kernel(int n, const int *cell_seg, const int *flag, const double *a, float *b) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n && flag[cell_seg[i]]) b[i] = (float)a[i];
}

// Per-instance squared norms of one or two vectors in two deterministic
// passes: one block per chunk of at most kChunk cells (chunks counted from
// each instance's first cell, so an instance is reduced the same way alone and
// in a batch), then one thread per instance adding its chunks in order.
constexpr int kChunk = 4096;

template <class T>
__global__ void __launch_bounds__(256) chunk_norm_kernel(const int *chunk_off, int nchunks, const T *a, const T *b,
                                                         double *part) {
  __shared__ double sh[256];
  const int ch = blockIdx.x;
  const int i0 = chunk_off[ch], i1 = chunk_off[ch + 1];
  const T *v = blockIdx.y ? b : a;
  double acc = 0.0;
  for (int i = i0 + threadIdx.x; i < i1; i += blockDim.x) acc = op_dot(acc, v[i], v[i]);
  sh[threadIdx.x] = acc;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1) {
    if ((int)threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[(size_t)blockIdx.y * nchunks + ch] = sh[0];
}

__global__ void chunk_sum_kernel(int nseg, const int *seg_chunk, int nchunks, const double *part, double *out) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= nseg) return;
  double acc = 0.0;
  for (int k = seg_chunk[s]; k < seg_chunk[s + 1]; k++) acc += part[(size_t)blockIdx.y * nchunks + k];
  out[(size_t)blockIdx.y * nseg + s] = acc;
}

// y = A x over the CSR pattern with TPR threads per row
// One row of A x by TPR lanes (1, 2, 4 or 8) with the same bits for every
// TPR: the row's entries are split into 8 phases (entry k of the row in
// phase k mod 8), each phase summed by one FMA chain in entry order, and the
// 8 phase sums added by a fixed tree, ((P0+P4) + (P2+P6)) + ((P1+P5) +
// (P3+P7)).  Lane l holds phases l, l+TPR, ...; the tree levels whose pairs
// lie in one lane are added in registers, the others by shuffles, so the
// lane split can be tuned for speed without changing any result.  Lane 0
// returns the row's value.
template <class T, int TPR>
__device__ __forceinline__ T row_dot(bool valid, int k0, int k1, int lane, const int *colidx, const T *A, const T *x) {
  constexpr int NP = 8 / TPR;
  T P[NP];
#pragma unroll
  for (int q = 0; q < NP; q++) {
    T acc = 0;
    if (valid)
      for (int k = k0 + lane + TPR * q; k < k1; k += 8) acc = e_fma(A[k], x[colidx[k]], acc);
    P[q] = acc;
  }
#pragma unroll
  for (int o = 4; o >= TPR; o >>= 1) {  // pairs (p, p + o) within the lane: q and q + o / TPR
#pragma unroll
    for (int q = 0; q < o / TPR; q++) P[q] = e_add(P[q], P[q + o / TPR]);
  }
  T acc = P[0];
#pragma unroll
  for (int o = TPR / 2; o > 0; o >>= 1) acc = e_add(acc, __shfl_down_sync(0xffffffffu, acc, o, TPR));
  return acc;
}

template <class T, int TPR>
__global__ void __launch_bounds__(256) spmv_kernel(int n, const int *rowptr, const int *colidx, const T *A, const T *x,
                                                   T *y) {
  const long long gt = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const int row = (int)(gt / TPR), lane = (int)(gt % TPR);
  const T acc = row_dot<T, TPR>(row < n, row < n ? rowptr[row] : 0, row < n ? rowptr[row + 1] : 0, lane, colidx, A, x);
  if (row < n && lane == 0) y[row] = acc;
}

// Thomas factorisation of every vertical line from the FP64 Jacobian
template <class T>
__global__ void line_factor_kernel(int nlines, const int *line_off, const int *line_cells, const int *pd,
                                   const int *plo, const int *phi, const double *J, T *la, T *lcp, T *linv) {
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= nlines) return;
  double cp = 0.0;
  for (int k = line_off[l]; k < line_off[l + 1]; k++) {
    const double b = J[pd[k]], a = plo[k] >= 0 ? J[plo[k]] : 0.0, c = phi[k] >= 0 ? J[phi[k]] : 0.0;
    double den = b - a * cp;
    if (den == 0.0) den = (b != 0.0) ? b : 1.0;  // singular line: fall back to its diagonal
    const double inv = 1.0 / den;
    cp = c * inv;
    const int i = line_cells[k];  // factors by cell: the lines of a warp are neighbours in every layer
    la[i] = (T)a;
    lcp[i] = (T)cp;
    linv[i] = (T)inv;
  }
}

// ---------------------------------------------------------------------------
// Block schedule: C CTAs of kBlockThreads threads (a cluster; C = 1, 2, 4, 8)
// run an instance's whole BiCGStab loop with the line preconditioner,
// performing the tile schedule's operations in the tile schedule's order
// (reductions in kChunk-cell chunks with the same per-chunk tree and in-order
// chunk sum, each row's 8 phases and their tree), so the schedules and every C
// give the same bits.  Clusters take instances from a ticket counter, largest
// first; an instance's result does not depend on which cluster takes it.
//
// What bounds it is latency, then one SM's FP64 pipe (the dot products
// accumulate in FP64) and its L2 bandwidth (the matrix is read twice an
// iteration), hence
//   * the vector that the sparse product gathers from, z, sits in shared
//     memory, and the line solves work on it in place; so do, where they fit,
//     the other vectors and the line factors (read back from L2 they cost a
//     round trip in each of the ten passes of an iteration);
//   * the matrix is stored in slices of 32 rows (entry k of the rows side by
//     side, 16-bit column indices local to the instance), so the owner of a
//     row reads it with coalesced, independent loads;
//   * CTA q owns the cells with index [q, q + 1) * 256 / C modulo 256 in the
//     instance: the vector updates and products of its cells take all its
//     threads, and each of the 256 accumulators of a chunk reduction runs over
//     cells of one CTA;
//   * the tree of a reduction runs in one warp (7 additions from shared
//     memory, 5 shuffles) instead of 8 levels of block barriers, and thread 0
//     alone forms the scalars (a division by every thread would occupy the
//     FP64 pipe for thousands of cycles).
constexpr int kBlockThreads = 256;
static_assert(kBlockThreads == 256 && kChunk % kBlockThreads == 0,
              "the block schedule's reductions mirror the 256-thread chunk reductions");
// largest instance of the block schedule (16-bit column indices)
constexpr long long kBlockCap = 65536;

template <class T>
struct BlockSolve {
  int ninst;                 // instances of this launch
  const int *inst;           // their indices, largest first
  int *ticket;               // zeroed before the launch
  const int *seg_off;        // cells of instance g: [seg_off[g], seg_off[g + 1])
  const int *inst_line_off;  // lines of instance g: [inst_line_off[g], inst_line_off[g + 1])
  const int *slice_off;      // first slice of instance g
  const long long *sell_off;
  const int *rowptr;
  const T *A;
  const uint16_t *col;
  const T *la, *lcp, *linv;  // by cell
  const double *F;
  T *vec[8], *z, *x;  // V_*, z and the lines' cells where they exceed shared memory (y: the result)
  int slots;          // KEEP_MATRIX: matrix slots of a CTA
  int *lin_its;
  double tol2;
  int max_it;
};

// What of an instance lives in shared memory: everything (each CTA the cells,
// line factors and matrix rows it owns, and all of z), everything but the
// matrix, z only, or nothing.
enum { V_R0 = 0, V_R, V_P, V_V, V_S, V_T, V_PH, V_Y };
enum { KEEP_MATRIX = 0, KEEP_ALL = 1, KEEP_Z = 2, KEEP_NONE = 3 };
// chunks of an nc-cell instance that are reduced together, and the two sets of
// their accumulators
constexpr int kRedChunksMax = 2;
__host__ __device__ constexpr int red_chunks(int nc) { return nc > kChunk ? kRedChunksMax : 1; }
__host__ __device__ constexpr int red_doubles(int nc) { return 2 * red_chunks(nc) * 2 * kBlockThreads; }
// cells a CTA owns at most, and cells of the lines it solves
__host__ __device__ inline int owned_cells(int nc, int C) {
  return (nc + kBlockThreads - 1) / kBlockThreads * (kBlockThreads / C);
}
// The lines' cells and factors lie line by line in shared memory, nlp layers
// apart: 16-byte loads fetch kLineVec layers, and nlp is an odd multiple of
// kLineVec, which spreads the lines of a warp over the banks.
template <class T>
struct LineVec;
template <>
struct LineVec<float> {
  using type = float4;
};
template <>
struct LineVec<double> {
  using type = double2;
};
template <class T>
constexpr int kLineVec = 16 / (int)sizeof(T);
template <class T>
__host__ __device__ constexpr int line_pitch(int nl) {
  return ((nl + kLineVec<T> - 1) / kLineVec<T> | 1) * kLineVec<T>;
}

inline size_t up16(size_t b) { return (b + 15) & ~size_t(15); }
// (lines: lines a CTA solves at most; slots: matrix slots of one CTA's rows)
template <class T>
size_t block_smem(int keep, int nc, int lines, int nl, size_t slots, int C) {
  size_t b = sizeof(double) * red_doubles(nc);
  if (keep != KEEP_NONE) b += up16(sizeof(T) * nc);
  if (keep != KEEP_NONE) b += sizeof(T) * lines * line_pitch<T>(nl);
  if (keep <= KEEP_ALL)
    b += 3 * sizeof(T) * lines * line_pitch<T>(nl) + up16((8 * sizeof(T) + sizeof(unsigned)) * owned_cells(nc, C));
  if (keep == KEEP_MATRIX) b += (sizeof(T) + sizeof(uint16_t)) * slots;
  return b;
}

// exact conversion without the FP64 pipe (a conversion instruction costs as
// much there as an FMA); zeros, subnormals, infinities and NaN the plain way
__device__ __forceinline__ double to_f64(double x) { return x; }
__device__ __forceinline__ double to_f64(float x) {
  const unsigned u = __float_as_uint(x), e = u & 0x7f800000u;
  if (e == 0u || e == 0x7f800000u) return (double)x;
  return __hiloint2double((int)((u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + (896u << 20))), (int)(u << 29));
}

template <int C>
__device__ __forceinline__ void csync() {
  if constexpr (C == 1)
    __syncthreads();
  else
    cooperative_groups::this_cluster().sync();
}
// the same shared variable of CTA `rank` of the cluster
template <int C, class U>
__device__ __forceinline__ U *peer(U *p, int rank) {
  if constexpr (C == 1)
    return p;
  else
    return cooperative_groups::this_cluster().map_shared_rank(p, rank);
}

// G rows of the sliced matrix times z by TPR lanes each: the sums of row_dot,
// valid in lane 0.  Row u has rn[u] entries from element base[u] on.  The
// loads of all rows and of two steps of each phase are in flight together
// (one row at a time, every row waited for L2: 2.7 k cycles a row at 1 k
// cells, 1.1 k so).
template <class T, int TPR, int G, bool GLOBAL>
__device__ __forceinline__ void sell_dot(const unsigned *base, const int *rn, int lane, const T *A, const uint16_t *col,
                                         const T *z, T *out) {
  constexpr int NP = 8 / TPR;
  T P[G][NP];
  int most = 0;
#pragma unroll
  for (int u = 0; u < G; u++) {
    most = max(most, rn[u]);
#pragma unroll
    for (int q = 0; q < NP; q++) P[u][q] = 0;
  }
#pragma unroll 2
  for (int k0 = lane; k0 < most; k0 += 8) {
    T a[G][NP];
    int c[G][NP];
#pragma unroll
    for (int u = 0; u < G; u++)
#pragma unroll
      for (int q = 0; q < NP; q++) {
        const int k = k0 + TPR * q;
        if (k < rn[u]) {
          // (the read-only path lets loads pass the stores of earlier rows)
          a[u][q] = GLOBAL ? __ldg(A + base[u] + 32 * k) : A[base[u] + 32 * k];
          c[u][q] = GLOBAL ? __ldg(col + base[u] + 32 * k) : col[base[u] + 32 * k];
        }
      }
#pragma unroll
    for (int u = 0; u < G; u++)
#pragma unroll
      for (int q = 0; q < NP; q++)
        if (k0 + TPR * q < rn[u]) P[u][q] = e_fma(a[u][q], z[c[u][q]], P[u][q]);
  }
#pragma unroll
  for (int u = 0; u < G; u++) {
#pragma unroll
    for (int o = 4; o >= TPR; o >>= 1) {
#pragma unroll
      for (int q = 0; q < o / TPR; q++) P[u][q] = e_add(P[u][q], P[u][q + o / TPR]);
    }
    out[u] = P[u][0];
  }
#pragma unroll
  for (int o = TPR / 2; o > 0; o >>= 1)
#pragma unroll
    for (int u = 0; u < G; u++) out[u] = e_add(out[u], __shfl_down_sync(0xffffffffu, out[u], o, TPR));
}

// x <- (line-tridiagonal)^-1 x for n lines of nl layers, one thread per line;
// layer k of line l sits at [l * xp + k] of x and at [l * fl + k * fs] of the
// factors (VEC: fl = xp, fs = 1).  The recurrence is the critical path: a layer
// takes 9 cycles in FP32 and 126 in FP64 forward, half of that backward; with
// 4-byte loads, the load instructions took 27 in FP32.
template <class T, bool VEC>
__device__ __forceinline__ void block_lines(int n, int nl, int xp, int fl, int fs, const T *la, const T *lcp,
                                            const T *linv, T *x) {
  constexpr int V = kLineVec<T>, U = 8;
  using VT = typename LineVec<T>::type;
#pragma unroll 1
  for (int l = threadIdx.x; l < n; l += kBlockThreads) {
    T *const xl = x + l * xp;
    const T *const al = la + l * fl, *const cl = lcp + l * fl, *const dl = linv + l * fl;
    auto load = [&](T *dst, const T *src, int k, int step) {
      if constexpr (VEC) {
#pragma unroll
        for (int u = 0; u < U; u += V) *reinterpret_cast<VT *>(dst + u) = *reinterpret_cast<const VT *>(src + k + u);
      } else {
#pragma unroll
        for (int u = 0; u < U; u++) dst[u] = src[(k + u) * step];
      }
    };
    const int full = nl / U * U;
    T prev = 0;
#pragma unroll 1
    for (int k = 0; k < full; k += U) {
      alignas(16) T v[U], a[U], d[U];
      load(v, xl, k, 1);
      load(a, al, k, fs);
      load(d, dl, k, fs);
#pragma unroll
      for (int u = 0; u < U; u++) v[u] = prev = e_mul(e_fma(-a[u], prev, v[u]), d[u]);
      if constexpr (VEC) {
#pragma unroll
        for (int u = 0; u < U; u += V) *reinterpret_cast<VT *>(xl + k + u) = *reinterpret_cast<VT *>(v + u);
      } else {
#pragma unroll
        for (int u = 0; u < U; u++) xl[k + u] = v[u];
      }
    }
#pragma unroll 1
    for (int k = full; k < nl; k++) xl[k] = prev = e_mul(e_fma(-al[k * fs], prev, xl[k]), dl[k * fs]);
    T next = 0;
#pragma unroll 1
    for (int k = nl - 1; k >= full; k--) xl[k] = next = e_fma(-cl[k * fs], next, xl[k]);
#pragma unroll 1
    for (int k = full - U; k >= 0; k -= U) {
      alignas(16) T v[U], c[U];
      load(v, xl, k, 1);
      load(c, cl, k, fs);
#pragma unroll
      for (int u = U - 1; u >= 0; u--) v[u] = next = e_fma(-c[u], next, v[u]);
      if constexpr (VEC) {
#pragma unroll
        for (int u = 0; u < U; u += V) *reinterpret_cast<VT *>(xl + k + u) = *reinterpret_cast<VT *>(v + u);
      } else {
#pragma unroll
        for (int u = 0; u < U; u++) xl[k + u] = v[u];
      }
    }
  }
}

// (two CTAs per SM: the loops' loads hide behind the other CTA's barriers)
template <class T, int C, int KEEP>
__global__ void __launch_bounds__(kBlockThreads, sizeof(T) == 4 ? 2 : 1) bicgstab_block_kernel(const BlockSolve<T> B) {
  static_assert(KEEP != KEEP_NONE || C == 1, "clusters exchange z through shared memory");
  constexpr int NO = kBlockThreads / C;  // cells (of 256 consecutive ones) that a CTA owns
  // reductions (two sets in turn), z, the own lines, own vectors, line
  // factors, own rows (first element << 8 | entries)
  extern __shared__ double bsm[];
  __shared__ int cur, stop;
  __shared__ T c_alpha, c_beta, c_omega;
  __shared__ double c_sum[2][2 * kRedChunksMax], c_ratio, c_alpha64, c_omega64;
  const int tid = threadIdx.x;
  const int q = C == 1 ? 0 : (int)(blockIdx.x % C);
  int buf = 0;
  for (;;) {
    if (q == 0 && tid == 0) {
      const int k = atomicAdd(B.ticket, 1);
#pragma unroll
      for (int r = 0; r < C; r++) *peer<C>(&cur, r) = k;
    }
    csync<C>();
    const int k = cur;
    csync<C>();  // every thread has read the ticket before the next one is drawn
    if (k >= B.ninst) return;
    const int g = B.inst[k];
    const int c0 = B.seg_off[g], nc = B.seg_off[g + 1] - c0;
    const int nc2 = B.inst_line_off[g + 1] - B.inst_line_off[g], nl = nc / nc2;
    const int nj = (nc + kBlockThreads - 1) / kBlockThreads;
    const int *rowptr = B.rowptr + c0;
    const long long *so = B.sell_off + B.slice_off[g];
    const int nred = red_chunks(nc);
    constexpr bool SHARED = KEEP <= KEEP_ALL;
    const int nown = owned_cells(nc, C);
    // lines q, q + C, ... of the instance
    const int n1 = (nc2 - q + C - 1) / C, lines = (nc2 + C - 1) / C;
    const int nlp = KEEP == KEEP_NONE ? nl : line_pitch<T>(nl), nf = lines * nlp;
    char *at_byte = reinterpret_cast<char *>(bsm + red_doubles(nc));
    T *const z = KEEP == KEEP_NONE ? B.z + c0 : reinterpret_cast<T *>(at_byte);
    at_byte += (nc * sizeof(T) + 15) & ~size_t(15);
    T *const x = KEEP == KEEP_NONE ? B.x + c0 : reinterpret_cast<T *>(at_byte);
    T *const lf = x + nf;
    T *const w = lf + 3 * nf;
    unsigned *const rinfo = reinterpret_cast<unsigned *>(w + 8 * nown);
    // own cell e is cell i(e) of the instance
    auto cell = [&](int e) { return e / NO * kBlockThreads + q * NO + e % NO; };
    // vector k at own cell e (the base of each vector is formed where it is
    // used: held in registers they spill)
    auto at = [&](int k, int e) -> T & { return SHARED ? w[k * nown + e] : B.vec[k][c0 + cell(e)]; };
    // f(e, i) for the own cells
    auto each = [&](auto f) {
#pragma unroll 1
      for (int e = tid; e < nown; e += kBlockThreads) {
        const int i = cell(e);
        if (i < nc) f(e, i);
      }
    };
    const T *A = B.A + so[0];
    const uint16_t *col = B.col + so[0];
    if constexpr (SHARED) {
      for (int e = tid; e < n1 * nl; e += kBlockThreads) {
        const int kk = e / n1, l = e - kk * n1, i = c0 + kk * nc2 + q + C * l;
        lf[l * nlp + kk] = B.la[i];
        lf[nf + l * nlp + kk] = B.lcp[i];
        lf[2 * nf + l * nlp + kk] = B.linv[i];
      }
      if constexpr (KEEP == KEEP_ALL) {
        // (an instance whose vectors fit shared memory has far fewer than 2^24 entries)
        each([&](int e, int i) {
          rinfo[e] = (unsigned)(so[i >> 5] - so[0] + (i & 31)) << 8 | (unsigned)(rowptr[i + 1] - rowptr[i]);
        });
      } else {
        // the own rows in slices of 32 of their own: those of slice e / 32 as
        // wide as in HBM, where they are (parts of) neighbouring slices
        T *const As = reinterpret_cast<T *>(reinterpret_cast<char *>(w) +
                                            (((8 * sizeof(T) + sizeof(unsigned)) * nown + 15) & ~size_t(15)));
        uint16_t *const cs = reinterpret_cast<uint16_t *>(As + B.slots);
        // widths of the own slices, then their offsets
        const int ns = (nown + 31) / 32;
        unsigned off = 0;
        for (int sl = 0; sl < ns; sl++) {
          int width = 0;
          for (int e = sl * 32; e < min(nown, sl * 32 + 32); e += min(NO, 32)) {
            const int i = cell(e);
            if (i < nc) width = max(width, (int)(so[(i >> 5) + 1] - so[i >> 5]) / 32);
          }
          if (tid / 32 == sl % (kBlockThreads / 32)) {
            const int e = sl * 32 + (tid & 31), i = cell(e);
            if (e < nown && i < nc) {
              const int rn = rowptr[i + 1] - rowptr[i];
              rinfo[e] = (off + (tid & 31)) << 8 | (unsigned)rn;
              const T *src = A + (so[i >> 5] - so[0]) + (i & 31);
              const uint16_t *csrc = col + (so[i >> 5] - so[0]) + (i & 31);
#pragma unroll 4
              for (int k = 0; k < rn; k++) {
                As[off + (tid & 31) + 32 * k] = __ldg(src + 32 * k);
                cs[off + (tid & 31) + 32 * k] = __ldg(csrc + 32 * k);
              }
            }
          }
          off += 32 * width;
        }
        A = As;
        col = cs;
      }
    }
    auto row_info = [&](int e, int i, unsigned *base, int *rn) {
      if constexpr (SHARED) {
        *base = rinfo[e] >> 8;
        *rn = (int)(rinfo[e] & 255u);
      } else {
        *base = (unsigned)(so[i >> 5] - so[0]) + (i & 31);
        *rn = rowptr[i + 1] - rowptr[i];
      }
    };

    // (vector k0, vector k1) and, with k2 >= 0, (vector k2, vector k3): per
    // chunk the accumulators and the 256-way tree of chunk_norm_kernel, then the
    // chunks in order.  With C > 1 each sum and chunk has threads (and a part of
    // the FP64 pipe) of its own, and one warp does each tree (the additions of a
    // warp take 60 cycles each); another one does `side` meanwhile.  Thread 0 of
    // each CTA gets the sums; the cluster is synchronised in between.
    auto nothing = []() {};
    auto dots = [&](int k0, int k1, int k2, int k3, double *s0, double *s1, auto side) {
      constexpr int JC = kChunk / kBlockThreads;
      const int nsum = k2 >= 0 ? 2 : 1;
      double t0 = 0.0, t1 = 0.0;
      __syncthreads();  // the vectors are complete
      for (int jr = 0; jr < nj; jr += nred * JC) {
        double *red = bsm + buf * (nred * 2 * kBlockThreads);
        const int nch = min(nred, (nj - jr + JC - 1) / JC), np = nsum * nch;
        // pair p: sum p / nch of chunk p % nch; its accumulator of index
        // q * NO + o modulo 256
#pragma unroll 1
        for (int pr = tid / NO; pr < np; pr += C) {
          const int hs = pr >= nch, o = tid % NO, j0 = jr + (pr - hs * nch) * JC, j1 = min(j0 + JC, nj);
          const int ka = hs ? k2 : k0, kb = hs ? k3 : k1;
          double acc = 0.0;
#pragma unroll 4
          for (int j = j0; j < j1; j++)
            if (j * kBlockThreads + q * NO + o < nc)
              acc = __fma_rn(to_f64(at(ka, j * NO + o)), to_f64(at(kb, j * NO + o)), acc);
#pragma unroll
          for (int rk = 0; rk < C; rk++) peer<C>(red, rk)[pr * kBlockThreads + q * NO + o] = acc;
        }
        csync<C>();
        if (jr == 0 && tid == 128) side();
        if (tid / 32 < np) {
          const double *d = red + (tid / 32) * kBlockThreads + (tid & 31);
          double t = __dadd_rn(__dadd_rn(__dadd_rn(d[0], d[128]), __dadd_rn(d[64], d[192])),
                               __dadd_rn(__dadd_rn(d[32], d[160]), __dadd_rn(d[96], d[224])));
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) t = __dadd_rn(t, __shfl_down_sync(0xffffffffu, t, o));
          if ((tid & 31) == 0) c_sum[buf][tid / 32] = t;
        }
        __syncthreads();
        if (tid == 0)
          for (int ch = 0; ch < nch; ch++) {
            t0 = __dadd_rn(t0, c_sum[buf][ch]);
            if (nsum > 1) t1 = __dadd_rn(t1, c_sum[buf][nch + ch]);
          }
        buf ^= 1;
      }
      *s0 = t0;
      if (nsum > 1) *s1 = t1;
    };
    // vector `out` = A z at the own cells, two lanes per row (more lanes spend
    // FP64 additions on their tree: 3 for 4 rows with 8 lanes, 4 for 16 with 2)
    auto product = [&](int out, bool keep_z) {
      constexpr int TPR = 2, G = sizeof(T) == 4 ? 2 : 1, RP = kBlockThreads / TPR;
      const int lane = tid % TPR;
#pragma unroll 1
      for (int e0 = tid / TPR; e0 - tid / TPR < nown; e0 += G * RP) {
        unsigned base[G];
        int rn[G];
        T sum[G];
#pragma unroll
        for (int u = 0; u < G; u++) {
          const int e = e0 + u * RP, i = cell(e);
          base[u] = 0;
          rn[u] = 0;
          if (e < nown && i < nc) row_info(e, i, &base[u], &rn[u]);
        }
        sell_dot<T, TPR, G, KEEP != KEEP_MATRIX>(base, rn, lane, A, col, z, sum);
#pragma unroll
        for (int u = 0; u < G; u++) {
          const int e = e0 + u * RP, i = cell(e);
          if (lane == 0 && e < nown && i < nc) {
            at(out, e) = sum[u];
            if (keep_z) at(V_PH, e) = z[i];
          }
        }
      }
    };
    // the line solves' input goes to the CTA that solves the cell's line
    auto to_line = [&](int i, T v) {
      const int kk = i / nc2, l = i - kk * nc2;
      peer<C>(x, l & (C - 1))[l / C * nlp + kk] = v;
    };
    // M^-1 of the lines' input, to every CTA's z
    auto precondition = [&]() {
      csync<C>();
      if constexpr (SHARED)
        block_lines<T, true>(n1, nl, nlp, nlp, 1, lf, lf + nf, lf + 2 * nf, x);
      else
        block_lines<T, false>(n1, nl, nlp, C, nc2, B.la + c0 + q, B.lcp + c0 + q, B.linv + c0 + q, x);
      __syncthreads();
      for (int e = tid; e < n1 * nl; e += kBlockThreads) {
        const int kk = e / n1, l = e - kk * n1, i = kk * nc2 + q + C * l;
        const T v = x[l * nlp + kk];
#pragma unroll
        for (int rk = 0; rk < C; rk++) peer<C>(z, rk)[i] = v;
      }
      csync<C>();
    };

    // thread 0's scalars
    double bnorm2 = 0.0, tol = 0.0, rho = 1.0, alpha = 1.0, omega = 1.0, d0, d1;
    int its = 0;
    each([&](int e, int i) {
      const T f = (T)B.F[c0 + i];
      at(V_R0, e) = f;
      at(V_R, e) = f;
      at(V_P, e) = 0;
      at(V_V, e) = 0;
      at(V_Y, e) = 0;
    });
    dots(V_R0, V_R0, -1, -1, &bnorm2, nullptr, nothing);
    // the scalars of an iteration's first half, from rn = (r0, r)
    auto begin = [&](double rn, int it) {
      stop = it >= B.max_it || rn == 0.0;
      if (stop) return;
      const double beta = (rn / rho) * c_ratio;  // alpha / omega
      rho = rn;
      c_beta = (T)beta;
      c_omega = (T)omega;
    };
    if (tid == 0) {
      c_ratio = 1.0;
      tol = B.tol2 * bnorm2;
      if (bnorm2 > 0.0)
        begin(bnorm2, 0);  // r = r0
      else
        stop = 1;
    }
    __syncthreads();
    for (int it = 0; !stop; it++) {
      {
        const T tb = c_beta, to = c_omega;
        each([&](int e, int i) {
          const T pi = op_p(at(V_R, e), at(V_P, e), at(V_V, e), tb, to);
          at(V_P, e) = pi;
          to_line(i, pi);
        });
      }
      precondition();
      product(V_V, true);
      dots(V_R0, V_V, -1, -1, &d0, nullptr, nothing);
      if (tid == 0) {
        stop = d0 == 0.0;
        if (!stop) {
          alpha = rho / d0;
          c_alpha = (T)alpha;
        }
      }
      __syncthreads();
      if (stop) break;
      const T ta = c_alpha;
      each([&](int e, int i) {
        const T si = e_fma(-ta, at(V_V, e), at(V_R, e));
        at(V_S, e) = si;
        to_line(i, si);
      });
      dots(V_S, V_S, -1, -1, &d0, nullptr, nothing);
      if (tid == 0) {
        stop = d0 <= tol;  // converged at the half step
        if (stop) its++;
      }
      __syncthreads();
      if (stop) {
        each([&](int e, int) { at(V_Y, e) = op_y(at(V_Y, e), at(V_PH, e), ta); });
        break;
      }
      precondition();
      product(V_T, false);
      dots(V_T, V_T, V_T, V_S, &d0, &d1, nothing);
      if (tid == 0) {
        omega = d0 > 0.0 ? d1 / d0 : 0.0;
        c_omega = (T)omega;
        c_alpha64 = alpha;
        c_omega64 = omega;
      }
      __syncthreads();
      const T to = c_omega;
      each([&](int e, int i) {
        at(V_Y, e) = op_y2(at(V_Y, e), at(V_PH, e), z[i], ta, to);
        at(V_R, e) = e_fma(-to, at(V_T, e), at(V_S, e));
      });
      dots(V_R, V_R, V_R0, V_R, &d0, &d1, [&]() { c_ratio = c_alpha64 / c_omega64; });
      if (tid == 0) {
        its++;
        if (d0 <= tol || omega == 0.0)
          stop = 1;
        else
          begin(d1, it + 1);
      }
      __syncthreads();
    }
    if constexpr (SHARED) each([&](int e, int i) { B.vec[V_Y][c0 + i] = at(V_Y, e); });
    if (q == 0 && tid == 0) B.lin_its[g] = its;
  }
}

// Column indices of the sliced layout, local to the instance, and (each
// solve) the values of the active instances: one warp per slice, the rows read
// with coalesced loads and turned through shared memory.
constexpr int kSliceWarps = 4;
constexpr int kSliceCols = 32;  // entries of the rows turned at a time
template <class TO, class TI>
__global__ void __launch_bounds__(32 * kSliceWarps) sell_fill_kernel(int nslices, const int *slice_row,
                                                                      const int *slice_end, const long long *sell_off,
                                                                      const int *cell_seg, const int *active,
                                                                      const int *seg_off, const int *rowptr,
                                                                      const TI *in, TO *out) {
  __shared__ TO buf[kSliceWarps][32][kSliceCols + 1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int sl = blockIdx.x * kSliceWarps + warp;
  if (sl >= nslices) return;  // whole warp
  const int row0 = slice_row[sl], nrow = slice_end[sl] - row0, g = cell_seg[row0];
  if (active && !active[g]) return;
  const long long o0 = sell_off[sl];
  const int width = (int)((sell_off[sl + 1] - o0) / 32);
  const int c0 = seg_off[g];
  for (int k0 = 0; k0 < width; k0 += kSliceCols) {
    for (int rr = 0; rr < nrow; rr++) {
      const int p0 = rowptr[row0 + rr], k = k0 + lane;
      TO x = 0;
      if (k < rowptr[row0 + rr + 1] - p0) {
        if constexpr (sizeof(TO) == 2)
          x = (TO)(in[p0 + k] - c0);
        else
          x = (TO)in[p0 + k];
      }
      buf[warp][rr][lane] = x;
    }
    __syncwarp();
    const int n = min(kSliceCols, width - k0);
    if (lane < nrow)
      for (int k = 0; k < n; k++) out[o0 + (long long)(k0 + k) * 32 + lane] = buf[warp][lane][k];
    __syncwarp();
  }
}

// trial point of the line search: x = xb - lam_s y for the instances on
// trial, x = xb for the others (FP64 update)
template <class T>
__global__ void trial_kernel(int n, const int *cs, const int *trial, const double *lam, const T *y, const double *xb,
                             double *x) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int s = cs[i];
  x[i] = trial[s] ? xb[i] - lam[s] * (double)y[i] : xb[i];
}
// accepted trial points become the base
__global__ void commit_kernel(int n, const int *cs, const int *commit, const double *x, double *xb) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  if (commit[cs[i]]) xb[i] = x[i];
}

// ---------------------------------------------------------------------------
// Cooperative grids: words of their state (zeroed before the launch), then
// what each kernel counts in it.
enum { GS_BAR = 0, GS_ACTIVE, GS_ERR, GS_COUNT };

// Every CTA of the launch is past its phase; false if that took longer than
// seconds (a CTA that gives up flags the error for the others and the host).
__device__ __forceinline__ bool grid_barrier(unsigned *sync, unsigned &target, int *ok) {
  __syncthreads();
  if (threadIdx.x == 0) {
    target += gridDim.x;
    __threadfence();
    atomicAdd(&sync[GS_BAR], 1u);
    int good = 1;
    for (unsigned spin = 0;; spin++) {
      unsigned now;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(now) : "l"(&sync[GS_BAR]) : "memory");
      if ((int)(now - target) >= 0) break;
      if (spin > (1u << 23) || ((spin & 1023u) == 1023u && *(volatile unsigned *)&sync[GS_ERR])) {
        atomicExch(&sync[GS_ERR], 1u);
        good = 0;
        break;
      }
    }
    *ok = good;
  }
  __syncthreads();
  return *ok != 0;
}

// ---------------------------------------------------------------------------
// Strong-coupling clusters.  A coupling with |a_ij| >= tau sqrt(|a_ii a_jj|)
// joins cells i and j; the connected clusters are found by label
// propagation (every strong coupling hooks the labels of both cells to the
// smaller one, then every cell follows the labels to their root).  The labels
// converge to each cluster's smallest cell index whatever the order of the
// atomic updates, so the clusters are deterministic.

constexpr int kClusterMax = 64;
constexpr int kClusterLd = kClusterMax + 1;  // padded row of the staged block
constexpr int kClusterRounds = 64;           // of hooks, at most
constexpr int kClusterThreads = 512;
constexpr int kClusterRowLanes = 8;  // lanes of a row in the hooks

template <class T>
struct ClusterSetup {
  int n;
  double tau;
  const int *rowptr, *colidx, *dpos;
  const double *J;
  unsigned char *strong;      // by entry
  int *lab, *cnt, *id, *loc;  // by cell; cnt and id at a cluster's smallest cell
  int *coff, *cmem;
  long long *cluoff;
  T *inv;  // 1 / diagonal of the cells outside the clusters
  unsigned long long *total;  // [3][grid]
  ClusterCounts *out;
  unsigned *sync;  // the barrier's words, then a changed flag per round
};

// exclusive prefix sums of a and b over the block's threads; ta, tb the totals
__device__ __forceinline__ void block_scan(unsigned long long &a, unsigned long long &b, unsigned long long &ta,
                                           unsigned long long &tb, unsigned long long (*sh)[2]) {
  const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
  unsigned long long xa = a, xb = b;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long ua = __shfl_up_sync(0xffffffffu, xa, o), ub = __shfl_up_sync(0xffffffffu, xb, o);
    if (lane >= o) {
      xa += ua;
      xb += ub;
    }
  }
  __syncthreads();
  if (lane == 31) {
    sh[warp][0] = xa;
    sh[warp][1] = xb;
  }
  __syncthreads();
  a = xa - a;
  b = xb - b;
  ta = tb = 0;
  for (int w = 0; w < kClusterThreads / 32; w++) {
    if (w == warp) {
      a += ta;
      b += tb;
    }
    ta += sh[w][0];
    tb += sh[w][1];
  }
}

// Labels, numbering of the clusters of 2..kClusterMax cells in order of their
// smallest cell, members (in any order: cl_factor_kernel sorts them) and the
// other cells' diagonals, in one cooperative grid.  What bounds it is latency:
// two barriers a round and a few for the numbering.  Set-ups and factors of
// four Newton iterations, with a launch per step, a look at the flag per round
// and the numbering on the host, and now: 20,960 prisms 1.27 ms and 0.53,
// 82,400 prisms 3.41 and 1.00.
template <class T>
__global__ void __launch_bounds__(kClusterThreads, 2) cl_setup_kernel(const ClusterSetup<T> C) {
  __shared__ int ok;
  __shared__ unsigned long long sh[kClusterThreads / 32][2];
  unsigned target = 0;
  const int n = C.n, stride = gridDim.x * kClusterThreads, t0 = blockIdx.x * kClusterThreads + threadIdx.x;
  for (int i = t0; i < n; i += stride) {
    C.lab[i] = i;
    C.cnt[i] = 0;
  }
  if (!grid_barrier(C.sync, target, &ok)) return;
  unsigned *changed = C.sync + GS_COUNT;
  bool settled = false;
  for (int round = 0; round < kClusterRounds && !settled; round++) {
    bool any = false;
    for (long long e = t0; e < (long long)n * kClusterRowLanes; e += stride) {
      const int i = (int)(e / kClusterRowLanes);
      const double di = round ? 0.0 : fabs(C.J[C.dpos[i]]);
      for (int k = C.rowptr[i] + (int)(e % kClusterRowLanes); k < C.rowptr[i + 1]; k += kClusterRowLanes) {
        const int j = C.colidx[k];
        bool s;
        if (round) {
          s = C.strong[k];
        } else {
          const double aij = fabs(C.J[k]);
          s = j != i && aij > 0.0 && aij >= C.tau * sqrt(di * fabs(C.J[C.dpos[j]]));
          C.strong[k] = s;
        }
        if (!s) continue;
        const int li = __ldcg(&C.lab[i]), lj = __ldcg(&C.lab[j]);
        if (li == lj) continue;
        atomicMin(&C.lab[max(li, lj)], min(li, lj));
        any = true;
      }
    }
    if (any) changed[round] = 1;
    if (!grid_barrier(C.sync, target, &ok)) return;
    settled = __ldcg(&changed[round]) == 0;
    if (settled) break;
    for (int i = t0; i < n; i += stride) {
      int l = __ldcg(&C.lab[i]);
      for (int up = __ldcg(&C.lab[l]); up != l; up = __ldcg(&C.lab[l])) l = up;  // (labels only fall towards the root)
      C.lab[i] = l;
    }
    if (!grid_barrier(C.sync, target, &ok)) return;
  }
  if (!settled) {
    if (t0 == 0) C.out->settled = 0;
    return;
  }
  for (int i = t0; i < n; i += stride) atomicAdd(&C.cnt[C.lab[i]], 1);
  if (!grid_barrier(C.sync, target, &ok)) return;
  // numbering: this CTA's cells [b0, b1), the sums before them from every CTA's totals
  const long long per = (n + (long long)gridDim.x - 1) / gridDim.x;
  const long long b0 = min((long long)n, blockIdx.x * per), b1 = min((long long)n, b0 + per);
  auto value = [&](long long r, unsigned long long &a, unsigned long long &lu, unsigned long long &big) {
    const int c = r < b1 ? __ldcg(&C.cnt[r]) : 0;
    const bool in = c >= 2 && c <= kClusterMax;
    a = in ? (1ull << 32) | (unsigned)c : 0;
    lu = in ? (unsigned long long)c * c : 0;
    big = c > kClusterMax ? c : 0;
  };
  unsigned long long sa = 0, sl = 0, sb = 0, zero = 0, ta, tl, tb, none;
  for (long long r = b0 + threadIdx.x; r < b1; r += kClusterThreads) {
    unsigned long long a, lu, big;
    value(r, a, lu, big);
    sa += a;
    sl += lu;
    sb += big;
  }
  block_scan(sa, sl, ta, tl, sh);
  block_scan(sb, zero, tb, none, sh);
  if (threadIdx.x == 0) {
    C.total[blockIdx.x] = ta;
    C.total[gridDim.x + blockIdx.x] = tl;
    C.total[2 * gridDim.x + blockIdx.x] = tb;
  }
  if (!grid_barrier(C.sync, target, &ok)) return;
  sa = sl = sb = 0;
  for (int b = threadIdx.x; b < (int)blockIdx.x; b += kClusterThreads) {
    sa += __ldcg(&C.total[b]);
    sl += __ldcg(&C.total[gridDim.x + b]);
  }
  if (blockIdx.x == gridDim.x - 1)
    for (int b = threadIdx.x; b < (int)gridDim.x; b += kClusterThreads) sb += __ldcg(&C.total[2 * gridDim.x + b]);
  unsigned long long ca, cl;  // before this tile
  block_scan(sa, sl, ca, cl, sh);
  block_scan(sb, zero, tb, none, sh);
  for (long long r0 = b0; r0 < b1; r0 += kClusterThreads) {
    const long long r = r0 + threadIdx.x;
    unsigned long long a, lu, big;
    value(r, a, lu, big);
    const bool in = a != 0;
    block_scan(a, lu, ta, tl, sh);
    if (r < b1) {
      const int c = (int)((ca + a) >> 32);
      C.id[r] = in ? c : -1;
      C.cnt[r] = in ? (int)(unsigned)(ca + a) : 0;  // from here on: where the next member goes
      if (in) {
        C.coff[c] = (int)(unsigned)(ca + a);
        C.cluoff[c] = (long long)(cl + lu);
      }
    }
    ca += ta;
    cl += tl;
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == 0) {
    C.coff[ca >> 32] = (int)(unsigned)ca;
    C.cluoff[ca >> 32] = (long long)cl;
    *C.out = {ca, cl, tb, 1};
  }
  if (!grid_barrier(C.sync, target, &ok)) return;
  for (int i = t0; i < n; i += stride) {
    const int l = C.lab[i], c = C.id[l];
    C.loc[i] = c < 0 ? -1 : 0;
    if (c >= 0) {
      C.cmem[atomicAdd(&C.cnt[l], 1)] = i;
    } else {
      const double d = C.J[C.dpos[i]];
      C.inv[i] = d != 0.0 ? (T)(1.0 / d) : (T)1;
    }
  }
}

// One warp per cluster: sort its members, stage the cluster's block of J
// (every coupling between its cells) in shared memory, factor it by LU with
// partial pivoting (ties to the smaller row; a zero pivot becomes 1), store
// the factors column by column (the solves read a column at a time) and the
// order of the rows.
template <class T>
__global__ void __launch_bounds__(32) cl_factor_kernel(int ncl, const int *coff, const long long *luoff,
                                                       int *cmem, int *loc, const int *lab,
                                                       const int *rowptr, const int *colidx, const double *J, T *lu,
                                                       int *perm) {
  extern __shared__ unsigned char cl_smem[];
  __shared__ int order[kClusterMax], member[kClusterMax];
  T *B = reinterpret_cast<T *>(cl_smem);  // [kClusterMax][kClusterLd]
  const int cl = blockIdx.x, lane = threadIdx.x;
  if (cl >= ncl) return;
  const int c0 = coff[cl], sz = coff[cl + 1] - c0;
  for (int e = lane; e < sz * kClusterLd; e += 32) B[e] = (T)0;
  __syncwarp();
  for (int r = lane; r < sz; r += 32) order[r] = cmem[c0 + r];
  __syncwarp();
  for (int r = lane; r < sz; r += 32) {  // ascending cells
    const int m = order[r];
    int rank = 0;
    for (int q = 0; q < sz; q++) rank += order[q] < m;
    member[rank] = m;
    cmem[c0 + rank] = m;
    loc[m] = rank;
  }
  __syncwarp();
  for (int r = lane; r < sz; r += 32) {
    order[r] = r;
    const int m = member[r], L = lab[m];
    for (int k = rowptr[m]; k < rowptr[m + 1]; k++) {
      const int col = colidx[k];
      if (lab[col] == L) B[r * kClusterLd + loc[col]] = (T)J[k];
    }
  }
  __syncwarp();
  for (int kk = 0; kk < sz; kk++) {
    T best = (T)-1;
    int bi = kk;
    for (int i = kk + lane; i < sz; i += 32) {
      const T v = B[i * kClusterLd + kk] < (T)0 ? -B[i * kClusterLd + kk] : B[i * kClusterLd + kk];
      if (v > best) {
        best = v;
        bi = i;
      }
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
      const T ob = __shfl_down_sync(0xffffffffu, best, off);
      const int oi = __shfl_down_sync(0xffffffffu, bi, off);
      if (ob > best || (ob == best && oi < bi)) {
        best = ob;
        bi = oi;
      }
    }
    bi = __shfl_sync(0xffffffffu, bi, 0);
    if (lane == 0 && bi != kk) {
      const int t = order[kk];
      order[kk] = order[bi];
      order[bi] = t;
    }
    if (bi != kk)
      for (int j = lane; j < sz; j += 32) {
        const T t = B[kk * kClusterLd + j];
        B[kk * kClusterLd + j] = B[bi * kClusterLd + j];
        B[bi * kClusterLd + j] = t;
      }
    __syncwarp();
    T pv = B[kk * kClusterLd + kk];
    if (pv == (T)0) pv = (T)1;
    __syncwarp();
    if (lane == 0) B[kk * kClusterLd + kk] = pv;
    for (int i = kk + 1 + lane; i < sz; i += 32) {
      const T l = B[i * kClusterLd + kk] / pv;
      B[i * kClusterLd + kk] = l;
      for (int j = kk + 1; j < sz; j++) B[i * kClusterLd + j] -= l * B[kk * kClusterLd + j];
    }
    __syncwarp();
  }
  T *out = lu + luoff[cl];
  for (int e = lane; e < sz * sz; e += 32) out[e] = B[(e % sz) * kClusterLd + e / sz];
  for (int r = lane; r < sz; r += 32) perm[c0 + r] = order[r];
}

// ---------------------------------------------------------------------------
// Tile schedule: one cooperative grid runs the whole BiCGStab loop of every
// instance that is not on the block schedule, in seven phases an iteration
// with a grid barrier after each: update of p and preconditioner, product,
// (r0, v); update of s and preconditioner, product, (t, t), (t, s), (s, s);
// update of y and r, (r, r), (r0, r).  The vector updates run in the phase
// that first reads them, by the thread that owns the cell there.
//
// What bounds it up to some 100 k cells is latency: a barrier and a round trip
// to L2 per phase, the columns of a cluster's triangular solves, the chains of
// the FP64 sums.  Hence the accumulators of a chunk (256 chains over its
// cells) are spread warp by warp over the SMs; the warp that comes last in a
// chunk adds the tree, the last of an instance the chunks and forms the
// scalars, so that a sum costs one phase; loads go in groups ahead of the
// stores that the compiler cannot move them past; and the loop leaves with
// the last instance.  Four Newton iterations' inner solves in
// FP32, as some twenty kernels an iteration in a graph replayed eight times
// between looks at the flags, and now: 20,960 prisms with clusters 2.96 ms and
// 0.60 (8 iterations), 264,000 hexahedra with lines 16.5 and 11.2 (89),
// 1,122,000 of them 48.5 and 30.5 (78), 192 columns 77.7 and 38.9.
constexpr int kGridThreads = 512, kGridWarps = kGridThreads / 32;
constexpr int kGridSums = 3;    // sums of one phase at most
constexpr int kChainGroup = 4;  // cells of a chain whose loads go ahead of its stores

template <class T>
struct GridSolve {
  int n, ns, nchunks, nlines, ncl;
  int clusters;  // preconditioner: clusters, else lines
  const int *cell_seg, *newt_active, *block_mask;
  const int *chunk_off, *seg_chunk;
  const int *rowptr, *colidx;
  const T *A;
  const int *line_off, *line_cells;
  const T *la, *lcp, *linv;
  const int *cloc, *coff, *cmem, *cperm;
  const long long *cluoff;
  const T *cinv, *clu;
  const double *F;
  T *r, *r0, *p, *v, *sv, *tv, *ph, *sh, *y;
  int *act, *its;
  double *sc;         // [S_NSCAL][ns]
  double *acc;        // [nchunks][kGridSums][256]
  double *part;       // [kGridSums][nchunks]
  unsigned *sync;     // GS_*, then a counter per chunk and per instance
  double tol2;
  int max_it;
};

// whether this warp is the last of `of` to arrive; then it sees what the
// others wrote, and the counter is zero again
__device__ __forceinline__ bool last_arrival(unsigned *count, int of, int lane) {
  if (of == 1) {
    __syncwarp();
    return true;
  }
  __threadfence();
  __syncwarp();
  unsigned old = 0;
  if (lane == 0) old = atomicAdd(count, 1u);
  old = __shfl_sync(0xffffffffu, old, 0);
  if (old != (unsigned)of - 1) return false;
  if (lane == 0) *count = 0;
  __threadfence();
  return true;
}

// The accumulators 32 w + lane of chunk ch (of `cells` cells, instance g) are
// in a.  True in the warp that holds the instance's sums, in every lane: the
// tree of chunk_norm_kernel (levels 128, 64, 32 across the 8 values of a lane,
// the others by shuffles), then the chunks in order.
template <int ND, class T>
__device__ __forceinline__ bool chunk_sums(const GridSolve<T> &G, int ch, int w, int cells, int g, int lane,
                                           double (&a)[ND]) {
  const int parts = min(8, (cells + 31) / 32);
  double *acc = G.acc + (size_t)ch * kGridSums * 256;
  if (parts > 1) {
#pragma unroll
    for (int d = 0; d < ND; d++) __stcg(&acc[d * 256 + 32 * w + lane], a[d]);
    if (!last_arrival(&G.sync[GS_COUNT + ch], parts, lane)) return false;
  }
  const int c0 = G.seg_chunk[g], nch = G.seg_chunk[g + 1] - c0;
#pragma unroll
  for (int d = 0; d < ND; d++) {
    double x = a[d];
    if (parts > 1) {
      double e[8];
#pragma unroll
      for (int j = 0; j < 8; j++) e[j] = j < parts ? __ldcg(&acc[d * 256 + 32 * j + lane]) : 0.0;
#pragma unroll
      for (int o = 4; o > 0; o >>= 1)
#pragma unroll
        for (int j = 0; j < o; j++) e[j] = __dadd_rn(e[j], e[j + o]);
      x = e[0];
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) x = __dadd_rn(x, __shfl_down_sync(0xffffffffu, x, o));
    a[d] = __shfl_sync(0xffffffffu, x, 0);
    if (nch > 1 && lane == 0) __stcg(&G.part[(size_t)d * G.nchunks + ch], x);
  }
  if (nch == 1) return true;
  if (!last_arrival(&G.sync[GS_COUNT + G.nchunks + g], nch, lane)) return false;
#pragma unroll
  for (int d = 0; d < ND; d++) a[d] = 0.0;
  for (int k = 0; k < nch; k += 32) {
    double x[ND];
#pragma unroll
    for (int d = 0; d < ND; d++) x[d] = k + lane < nch ? __ldcg(&G.part[(size_t)d * G.nchunks + c0 + k + lane]) : 0.0;
    for (int j = 0; j < min(32, nch - k); j++)
#pragma unroll
      for (int d = 0; d < ND; d++) a[d] = __dadd_rn(a[d], __shfl_sync(0xffffffffu, x[d], j));
  }
  return true;
}

// y = A x for the rows of the active instances
template <class T, int TPR>
__device__ __forceinline__ void grid_spmv(const GridSolve<T> &G, const T *x, T *y) {
  constexpr int kRows = kGridThreads / TPR;
  const int lane = threadIdx.x % TPR;
  for (long long b = (long long)blockIdx.x * kRows; b < G.n; b += (long long)gridDim.x * kRows) {
    const long long row = b + threadIdx.x / TPR;
    const bool valid = row < G.n && G.act[G.cell_seg[row]];
    const T d = row_dot<T, TPR>(valid, valid ? G.rowptr[row] : 0, valid ? G.rowptr[row + 1] : 0, lane, G.colidx, G.A, x);
    if (valid && lane == 0) y[row] = d;
  }
}

// out = M^-1 in for the active instances; in(g) gives the entries of instance
// g's cells: value(i) reads, keep(i, value) stores what the update of the
// vector is.  Lines: a thread each, kLineGroup layers' loads ahead of their
// steps.  Clusters: a warp each, rows lane and lane + 32 in its registers (the
// rows' order, then the unit-lower and upper triangular solves, whose columns
// do not wait for the values); the other cells by their diagonal.
constexpr int kLineGroup = 4;

template <class T, class In>
__device__ __forceinline__ void grid_precondition(const GridSolve<T> &G, const In &in, T *out) {
  // neighbouring warps' work on different SMs
  const int warp = (threadIdx.x / 32) * gridDim.x + blockIdx.x, nwarps = gridDim.x * kGridWarps;
  const int lane = threadIdx.x % 32;
  if (!G.clusters) {
    for (int l = warp * 32 + lane; l < G.nlines; l += nwarps * 32) {
      const int k0 = G.line_off[l], len = G.line_off[l + 1] - k0;
      // a column's cells lie one layer apart
      const int first = G.line_cells[k0], step = len > 1 ? G.line_cells[k0 + 1] - first : 0;
      const int g = G.cell_seg[first];
      if (!G.act[g]) continue;
      const auto f = in(g);
      T prev = 0;
      for (int k = 0; k < len; k += kLineGroup) {
        T a[kLineGroup], d[kLineGroup], x[kLineGroup];
#pragma unroll
        for (int j = 0; j < kLineGroup; j++) {
          const int i = first + min(k + j, len - 1) * step;
          a[j] = G.la[i];
          d[j] = G.linv[i];
          x[j] = f.value(i);
        }
#pragma unroll
        for (int j = 0; j < kLineGroup; j++)
          if (k + j < len) {
            const int i = first + (k + j) * step;
            f.keep(i, x[j]);
            prev = e_mul(e_fma(-a[j], prev, x[j]), d[j]);
            out[i] = prev;
          }
      }
      T next = 0;
      for (int k = len - 1; k >= 0; k -= kLineGroup) {
        T c[kLineGroup], x[kLineGroup];
#pragma unroll
        for (int j = 0; j < kLineGroup; j++) {
          const int i = first + max(k - j, 0) * step;
          c[j] = G.lcp[i];
          x[j] = out[i];
        }
#pragma unroll
        for (int j = 0; j < kLineGroup; j++)
          if (k - j >= 0) {
            next = e_fma(-c[j], next, x[j]);
            out[first + (k - j) * step] = next;
          }
      }
    }
    return;
  }
  for (int cl = warp; cl < G.ncl; cl += nwarps) {
    const int c0 = G.coff[cl], sz = G.coff[cl + 1] - c0;
    const int g = G.cell_seg[G.cmem[c0]];
    if (!G.act[g]) continue;
    const auto f = in(g);
    const bool on0 = lane < sz, on1 = lane + 32 < sz;
    const int m0 = on0 ? G.cmem[c0 + lane] : 0, m1 = on1 ? G.cmem[c0 + lane + 32] : 0;
    const int s0 = on0 ? G.cperm[c0 + lane] : 0, s1 = on1 ? G.cperm[c0 + lane + 32] : 0;
    const T v0 = on0 ? f.value(m0) : (T)0, v1 = on1 ? f.value(m1) : (T)0;
    if (on0) f.keep(m0, v0);
    if (on1) f.keep(m1, v1);
    auto from = [&](int r) {  // row r's value (r differs by lane)
      const T a = __shfl_sync(0xffffffffu, v0, r & 31), b = __shfl_sync(0xffffffffu, v1, r & 31);
      return r < 32 ? a : b;
    };
    T x0 = from(s0), x1 = from(s1);
    const T *L = G.clu + G.cluoff[cl];
#pragma unroll 4
    for (int k = 0; k < sz; k++) {
      const T l0 = on0 ? L[k * sz + lane] : (T)0, l1 = on1 ? L[k * sz + lane + 32] : (T)0;
      const T xk = __shfl_sync(0xffffffffu, k < 32 ? x0 : x1, k & 31);
      if (lane > k) x0 -= l0 * xk;
      if (lane + 32 > k) x1 -= l1 * xk;
    }
#pragma unroll 4
    for (int k = sz - 1; k >= 0; k--) {
      const T l0 = on0 ? L[k * sz + lane] : (T)0, l1 = on1 ? L[k * sz + lane + 32] : (T)0;
      const T xk = __shfl_sync(0xffffffffu, k < 32 ? x0 : x1, k & 31) / L[k * sz + k];
      x0 = lane == k ? xk : lane < k ? x0 - l0 * xk : x0;
      x1 = lane + 32 == k ? xk : lane + 32 < k ? x1 - l1 * xk : x1;
    }
    if (on0) out[m0] = x0;
    if (on1) out[m1] = x1;
  }
  for (int i = blockIdx.x * kGridThreads + threadIdx.x; i < G.n; i += gridDim.x * kGridThreads) {
    if (G.cloc[i] >= 0) continue;
    const int g = G.cell_seg[i];
    if (!G.act[g]) continue;
    const auto f = in(g);
    const T x = f.value(i);
    f.keep(i, x);
    out[i] = G.cinv[i] * x;
  }
}

// p = r + beta (p - omega v)
template <class T>
struct UpdateP {
  const GridSolve<T> &G;
  T beta, omega;
  __device__ T value(int i) const { return op_p(G.r[i], G.p[i], G.v[i], beta, omega); }
  __device__ void keep(int i, T p) const { G.p[i] = p; }
};
// s = r - alpha v
template <class T>
struct UpdateS {
  const GridSolve<T> &G;
  T alpha;
  __device__ T value(int i) const { return e_fma(-alpha, G.v[i], G.r[i]); }
  __device__ void keep(int i, T s) const { G.sv[i] = s; }
};

// f(ch, w, i0, i1, g) for the accumulators 32 w .. 32 w + 31 of every chunk
template <class T, class Fn>
__device__ __forceinline__ void grid_chunks(const GridSolve<T> &G, const Fn &f) {
  for (int e = (threadIdx.x / 32) * gridDim.x + blockIdx.x; e < 8 * G.nchunks; e += gridDim.x * kGridWarps) {
    const int ch = e / 8, w = e % 8;
    const int i0 = G.chunk_off[ch], i1 = G.chunk_off[ch + 1];
    if (i0 + 32 * w < i1) f(ch, w, i0, i1, G.cell_seg[i0]);
  }
}

template <class T, int TPR>
__global__ void __launch_bounds__(kGridThreads, sizeof(T) == 4 ? 2 : 1) bicgstab_grid_kernel(const GridSolve<T> G) {
  __shared__ int ok;
  const int lane = threadIdx.x % 32, ns = G.ns;
  unsigned target = 0;
  auto S = [&](int slot, int g) -> double & { return G.sc[(size_t)slot * ns + g]; };
  auto retire = [&](int g) {
    G.act[g] = 0;
    atomicSub(&G.sync[GS_ACTIVE], 1u);
  };
  // rho = (r0, r) and the next beta
  auto beta = [&](int g, double rn, double rho, double alpha, double omega) {
    if (rn == 0.0) {
      retire(g);
      return;
    }
    S(S_BETA, g) = (rn / rho) * (alpha / omega);
    S(S_RHO, g) = rn;
  };
  // r = r0 = F, and ||F||^2
  grid_chunks(G, [&](int ch, int w, int i0, int i1, int g) {
    const bool on = G.newt_active[g];
    const bool mine = !G.block_mask[g];
    if (!on || !mine) {
      if (lane == 0 && w == 0 && ch == G.seg_chunk[g]) G.act[g] = 0;
      if (mine)
        for (int i = i0 + 32 * w + lane; i < i1; i += 256) G.y[i] = 0;
      return;
    }
    double a[1] = {0.0};
    for (int i = i0 + 32 * w + lane; i < i1; i += 256) {
      const T f = (T)G.F[i];
      G.r[i] = f;
      G.r0[i] = f;
      G.p[i] = 0;
      G.v[i] = 0;
      G.y[i] = 0;
      a[0] = op_dot(a[0], f, f);
    }
    if (chunk_sums(G, ch, w, i1 - i0, g, lane, a) && lane == 0) {
      S(S_BNORM2, g) = a[0];
      S(S_OMEGA, g) = S(S_ALPHA, g) = 1.0;
      const bool solve = a[0] > 0.0;
      G.act[g] = solve;
      if (solve) {
        atomicAdd(&G.sync[GS_ACTIVE], 1u);
        beta(g, a[0], 1.0, 1.0, 1.0);
      }
    }
  });
  if (!grid_barrier(G.sync, target, &ok)) return;
  for (int it = 0; it < G.max_it && __ldcg(&G.sync[GS_ACTIVE]) != 0; it++) {
    grid_precondition(
        G, [&](int g) { return UpdateP<T>{G, (T)S(S_BETA, g), (T)S(S_OMEGA, g)}; }, G.ph);
    if (!grid_barrier(G.sync, target, &ok)) return;
    grid_spmv<T, TPR>(G, G.ph, G.v);
    if (!grid_barrier(G.sync, target, &ok)) return;
    grid_chunks(G, [&](int ch, int w, int i0, int i1, int g) {
      if (!G.act[g]) return;
      double a[1] = {0.0};
#pragma unroll 8
      for (int i = i0 + 32 * w + lane; i < i1; i += 256) a[0] = op_dot(a[0], G.r0[i], G.v[i]);
      if (chunk_sums(G, ch, w, i1 - i0, g, lane, a) && lane == 0) {
        if (a[0] == 0.0)
          retire(g);
        else
          S(S_ALPHA, g) = S(S_RHO, g) / a[0];
      }
    });
    if (!grid_barrier(G.sync, target, &ok)) return;
    grid_precondition(
        G, [&](int g) { return UpdateS<T>{G, (T)S(S_ALPHA, g)}; }, G.sh);
    if (!grid_barrier(G.sync, target, &ok)) return;
    grid_spmv<T, TPR>(G, G.sh, G.tv);
    if (!grid_barrier(G.sync, target, &ok)) return;
    grid_chunks(G, [&](int ch, int w, int i0, int i1, int g) {
      if (!G.act[g]) return;
      double a[3] = {0.0, 0.0, 0.0};
#pragma unroll 8
      for (int i = i0 + 32 * w + lane; i < i1; i += 256) {
        const T t = G.tv[i], s = G.sv[i];
        a[0] = op_dot(a[0], t, t);
        a[1] = op_dot(a[1], t, s);
        a[2] = op_dot(a[2], s, s);
      }
      if (chunk_sums(G, ch, w, i1 - i0, g, lane, a) && lane == 0) {
        S(S_OMEGA, g) = a[0] > 0.0 ? a[1] / a[0] : 0.0;
        S(S_HALF, g) = a[2] <= G.tol2 * S(S_BNORM2, g) ? 1.0 : 0.0;  // converged at the half step
      }
    });
    if (!grid_barrier(G.sync, target, &ok)) return;
    grid_chunks(G, [&](int ch, int w, int i0, int i1, int g) {
      if (!G.act[g]) return;
      const T alpha = (T)S(S_ALPHA, g), omega = (T)S(S_OMEGA, g);
      const bool half = S(S_HALF, g) != 0.0;
      double a[2] = {0.0, 0.0};
      // kChainGroup cells' loads ahead of their stores
      for (int b = i0 + 32 * w + lane; b < i1; b += 256 * kChainGroup) {
        T y[kChainGroup], ph[kChainGroup], sh[kChainGroup], t[kChainGroup], sv[kChainGroup], r0[kChainGroup];
#pragma unroll
        for (int j = 0; j < kChainGroup; j++) {
          const int i = min(b + 256 * j, i1 - 1);
          y[j] = G.y[i];
          ph[j] = G.ph[i];
          sh[j] = G.sh[i];
          t[j] = G.tv[i];
          sv[j] = G.sv[i];
          r0[j] = G.r0[i];
        }
#pragma unroll
        for (int j = 0; j < kChainGroup; j++) {
          const int i = b + 256 * j;
          if (i >= i1) break;
          if (half) {
            G.y[i] = op_y(y[j], ph[j], alpha);
          } else {
            G.y[i] = op_y2(y[j], ph[j], sh[j], alpha, omega);
            const T r = e_fma(-omega, t[j], sv[j]);
            G.r[i] = r;
            a[0] = op_dot(a[0], r, r);
            a[1] = op_dot(a[1], r0[j], r);
          }
        }
      }
      if (chunk_sums(G, ch, w, i1 - i0, g, lane, a) && lane == 0) {
        G.its[g] += 1;
        const double om = S(S_OMEGA, g);
        if (half || a[0] <= G.tol2 * S(S_BNORM2, g) || om == 0.0)
          retire(g);
        else
          beta(g, a[1], S(S_RHO, g), S(S_ALPHA, g), om);
      }
    });
    if (!grid_barrier(G.sync, target, &ok)) return;
  }
}

// ---------------------------------------------------------------------------
template <class T>
void spmv(SolverState *s, const Krylov &k, const T *x, T *y, cudaStream_t st) {
  const T *A = (const T *)k.Jv;
  const unsigned g = nblk((long long)s->n * k.tpr, 256);
  switch (k.tpr) {
    case 1: spmv_kernel<T, 1><<<g, 256, 0, st>>>(s->n, s->rowptr, s->colidx, A, x, y); break;
    case 2: spmv_kernel<T, 2><<<g, 256, 0, st>>>(s->n, s->rowptr, s->colidx, A, x, y); break;
    case 4: spmv_kernel<T, 4><<<g, 256, 0, st>>>(s->n, s->rowptr, s->colidx, A, x, y); break;
    default: spmv_kernel<T, 8><<<g, 256, 0, st>>>(s->n, s->rowptr, s->colidx, A, x, y);
  }
}

// out = ||a||^2 per instance (, then ||b||^2)
template <class T>
void seg_norms(SolverState *s, const T *a, const T *b, double *out, cudaStream_t st) {
  const unsigned nv = b ? 2 : 1;
  chunk_norm_kernel<T><<<dim3(s->nchunks, nv), 256, 0, st>>>(s->chunk_off, s->nchunks, a, b, s->part);
  chunk_sum_kernel<<<dim3(nblk(s->nseg, 128), nv), 128, 0, st>>>(s->nseg, s->seg_chunk, s->nchunks, s->part, out);
}

// (one allocation for every vector; ordered on the solve's stream, which uses
// them next)
template <class T>
int krylov_alloc(SolverState *s, Krylov &k, cudaStream_t st) {
  // (the CSR copy Jv and the sliced copy are allocated by the schedules that use them)
  if (k.ready) return 0;
  Arena ar;
  T **vecs[] = {(T **)&k.b, (T **)&k.r,  (T **)&k.r0, (T **)&k.p,  (T **)&k.v,   (T **)&k.s,   (T **)&k.t,
                (T **)&k.ph, (T **)&k.sh, (T **)&k.y, (T **)&k.la, (T **)&k.lcp, (T **)&k.linv};
  for (T **vp : vecs) ar.work(vp, (size_t)s->n);
  int ierr = ar.commit(st);
  if (ierr) return ierr;
  s->allocs.push_back(ar.base);
  k.ready = true;
  return 0;
}

// Picks the threads per row of the tile schedule's product by timing
// spmv_kernel, the same product in a launch of its own, on the handle's first
// solve in each precision (the best split depends on the rows);
// options.spmv_threads forces one.  The results do not depend on it (row_dot).
// Inner solves in FP32 with the choice, then 1, 2, 4, 8 threads: 20,640 prisms
// 0.39 ms, 0.51, 0.39, 0.37, 0.39; 204 k prisms 0.64, 1.18, 0.75, 0.66, 0.64;
// 40,641 hexahedra 15.5, 16.0, 14.8, 15.6, 15.9; 264,000 215, 226, 217, 239,
// 289; 1,122,000 553, 558, 549, 641, 871; 192 columns 23.5, 26.4, 23.7, 23.5,
// 24.9.  (FP64 likewise: never more than 1 % from the best.)
template <class T>
int autotune_spmv(SolverState *s, Krylov &k, int forced, cudaStream_t st) {
  if (forced > 0) {
    k.tpr = forced;
    return 0;
  }
  if (k.tpr) return 0;
  cudaEvent_t e0, e1;
  SCUDA(cudaEventCreate(&e0));
  SCUDA(cudaEventCreate(&e1));
  float best = 1e30f;
  int best_tpr = 1;
  for (int tpr : {1, 2, 4, 8}) {
    k.tpr = tpr;
    spmv<T>(s, k, (const T *)k.b, (T *)k.v, st);  // warm-up
    cudaEventRecord(e0, st);
    for (int it = 0; it < 5; it++) spmv<T>(s, k, (const T *)k.b, (T *)k.v, st);
    cudaEventRecord(e1, st);
    SCUDA(cudaEventSynchronize(e1));
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    if (ms < best) {
      best = ms;
      best_tpr = tpr;
    }
  }
  k.tpr = best_tpr;
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  return 0;
}

// A cooperative launch: its CTAs are all resident, so that its barriers end.
template <class P>
int launch_cooperative(void (*kern)(const P), const P &arg, long long grid, int threads, cudaStream_t st) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)std::max(1LL, grid));
  cfg.blockDim = dim3(threads);
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  SCUDA(cudaLaunchKernelEx(&cfg, kern, arg));
  return 0;
}

// Clusters for the current Jacobian and their factors.  Returns 0 with
// precond_used = TDY_PRECOND_LINES when the labels have not settled in
// kClusterRounds rounds (the caller then factors the lines).
template <class T>
int cluster_setup(SolverState *s, Krylov &k, double tau, cudaStream_t st) {
  int ierr, dev = 0, nsm = 0, per_sm = 0;
  const int n = s->n;
  SCUDA(cudaGetDevice(&dev));
  SCUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  SCUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, cl_setup_kernel<T>, kClusterThreads, 0));
  const long long want = ((long long)n * kClusterRowLanes + kClusterThreads - 1) / kClusterThreads;
  const long long grid = std::max(1LL, std::min(want, (long long)nsm * per_sm));
  constexpr size_t nsync = GS_COUNT + kClusterRounds;
  if (!s->clab) {
    Arena ar;
    ar.work(&s->clab, n);
    ar.work(&s->cloc, n);
    ar.work(&s->cmem, n);
    ar.work(&s->cperm, n);
    ar.work(&s->ccnt, n);
    ar.work(&s->cid, n);
    ar.work(&s->coff, n + 1);
    ar.work(&s->cluoff, n + 1);
    ar.work(&s->cstrong, s->nnz);
    ar.work(&s->ctotal, 3 * (size_t)nsm * 4);  // (at most 2048 threads per SM)
    ar.work(&s->ccounts, 1 + (nsync * sizeof(unsigned) + sizeof(ClusterCounts) - 1) / sizeof(ClusterCounts));  // then csync
    if ((ierr = ar.commit(st))) return ierr;
    s->allocs.push_back(ar.base);
    s->csync = reinterpret_cast<unsigned *>(s->ccounts + 1);
  }
  if (!k.cinv) {
    T *p;
    if ((ierr = salloc(s, &p, n))) return ierr;
    k.cinv = p;
  }
  ClusterSetup<T> C;
  C.n = n;
  C.tau = tau;
  C.rowptr = s->rowptr;
  C.colidx = s->colidx;
  C.dpos = s->dpos;
  C.J = s->J;
  C.strong = s->cstrong;
  C.lab = s->clab;
  C.cnt = s->ccnt;
  C.id = s->cid;
  C.loc = s->cloc;
  C.coff = s->coff;
  C.cmem = s->cmem;
  C.cluoff = s->cluoff;
  C.inv = (T *)k.cinv;
  C.total = s->ctotal;
  C.out = s->ccounts;
  C.sync = s->csync;
  SCUDA(cudaMemsetAsync(s->csync, 0, nsync * sizeof(unsigned), st));
  if ((ierr = launch_cooperative(cl_setup_kernel<T>, C, grid, kClusterThreads, st))) return ierr;
  struct {
    ClusterCounts counts;
    unsigned sync[GS_COUNT];
  } out;
  SCUDA(cudaMemcpyAsync(&out, s->ccounts, sizeof(ClusterCounts) + sizeof(unsigned) * GS_COUNT, cudaMemcpyDeviceToHost, st));
  SCUDA(cudaStreamSynchronize(st));
  if (out.sync[GS_ERR]) return set_error(TDY_ERR_GPU, "solver: a wait of the cluster set-up ran out");
  const ClusterCounts &counts = out.counts;
  if (!counts.settled) {
    s->precond_used = TDY_PRECOND_LINES;
    return 0;
  }
  s->ncl = (int)(counts.both >> 32);
  s->ncl_cells = (int)(unsigned)counts.both;
  s->ncl_big_cells = (int)counts.big;
  if (s->ncl > 0) {
    const size_t need = (size_t)counts.lu;
    if (need > k.clu_cap) {  // stream-ordered: no device synchronisation
      if (k.clu) dmem_free(k.clu, st);
      k.clu = nullptr;
      k.clu_cap = 0;
      if ((ierr = dmem_alloc(&k.clu, need * sizeof(T), st))) return ierr;
      k.clu_cap = need;
    }
    cl_factor_kernel<T><<<s->ncl, 32, kClusterMax * kClusterLd * sizeof(T), st>>>(
        s->ncl, s->coff, s->cluoff, s->cmem, s->cloc, s->clab, s->rowptr, s->colidx, s->J, (T *)k.clu, s->cperm);
    SCUDA(cudaGetLastError());
  }
  s->precond_used = TDY_PRECOND_CLUSTERS;
  return 0;
}

// The sliced matrix layout of the block schedule, on its first use: offsets
// from the rows' lengths, column indices by sell_fill_kernel.  (sell_col is set
// when all of it is in place.)
int sell_setup(SolverState *s, cudaStream_t st) {
  if (s->sell_col) return 0;
  int ierr;
  std::vector<int> end(s->h_slice_row.size());
  for (size_t g = 0; g + 1 < s->h_seg_off.size(); g++)
    for (int k = s->h_slice_off[g]; k < s->h_slice_off[g + 1]; k++)
      end[k] = std::min(s->h_slice_row[k] + 32, s->h_seg_off[g + 1]);
  Arena ar;
  uint16_t *col = nullptr;
  ar.up(&s->slice_off, s->h_slice_off);
  ar.up(&s->slice_row, s->h_slice_row);
  ar.up(&s->slice_end, end);
  ar.up(&s->sell_off, s->h_sell_off);
  ar.work(&col, (size_t)s->h_sell_off.back());
  ierr = ar.commit(st);
  if (ar.base) s->allocs.push_back(ar.base);
  if (ierr) return ierr;
  if (s->nslices > 0)
    sell_fill_kernel<uint16_t, int><<<nblk(s->nslices, kSliceWarps), 32 * kSliceWarps, 0, st>>>(
        s->nslices, s->slice_row, s->slice_end, s->sell_off, s->cell_seg, nullptr, s->seg_off, s->rowptr, s->colidx,
        col);
  SCUDA(cudaGetLastError());
  SCUDA(cudaStreamSynchronize(st));  // the host vectors are read
  s->sell_col = col;
  return 0;
}

bool on_block(const SolverState *s, long long thr, int g) {
  const long long nc = s->h_seg_off[g + 1] - s->h_seg_off[g];
  return thr >= 0 && nc <= std::min(thr, kBlockCap);
}

// Instances on the block schedule for a split at `thr` cells (-1: none,
// LLONG_MAX: all up to kBlockCap): the per-instance mask.
int set_block_split(SolverState *s, long long thr, cudaStream_t st) {
  if (s->mask_for == thr) return 0;
  std::vector<int> mask(s->nseg, 0);
  s->n_block = 0;
  for (int g = 0; g < s->nseg; g++)
    if (on_block(s, thr, g)) {
      mask[g] = 1;
      s->n_block++;
    }
  s->n_tile = s->nseg - s->n_block;
  SCUDA(cudaMemcpyAsync(s->block_mask, mask.data(), sizeof(int) * s->nseg, cudaMemcpyHostToDevice, st));
  SCUDA(cudaStreamSynchronize(st));  // the host vector is read
  s->mask_for = thr;
  return 0;
}

// CTAs per instance: 256 cells each in FP32 and 128 in FP64 (whose arithmetic
// is the longer part), more in batches that fill the SMs eight times over.
// The launch lasts as long as its longest instance's iterations, not as the
// batch's work: 192 instances (217 k cells) take 50 times longer than their
// arithmetic and matrix traffic.
int block_ctas(long long cells, long long total, int nsm, size_t tsize) {
  const long long target = std::max<long long>(tsize == 4 ? 256 : 128, total / (8 * nsm));
  int c = 1;
  while (c < 8 && c * target < cells) c *= 2;
  return c;
}

// Launch classes of the block schedule: where the vectors live and the CTAs
// per instance, each split by shared memory (a class asks for what its largest
// instance needs, so small instances keep their residency beside large ones).
// The split by shared memory does not pay for its launches in the batches
// measured since: inner solves of a step with these steps and without, 28
// instances FP32 6.2 and 5.9 ms, 32 FP64 8.9 and 7.2, 192 FP32 15.6 and 13.5,
// 512 FP32 47 and 44, 512 FP64 77 and 75.
constexpr size_t kBlockSmemMax = 220 * 1024;  // dynamic shared memory of a CTA
constexpr size_t kBlockSmemSteps[3] = {36 * 1024, 72 * 1024, kBlockSmemMax};
constexpr int kBlockClasses = 2 * 4 * 3 + 2;

template <class T, int C, int KEEP>
int launch_block_class(const BlockSolve<T> &B, size_t smem, int nsm, cudaStream_t st) {
  auto kern = bicgstab_block_kernel<T, C, KEEP>;
  // (the 48 KB that need no attribute hold the static shared memory as well)
  if (smem > 47 * 1024) SCUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBlockSmemMax));
  int per_sm = 0;
  SCUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kBlockThreads, smem));
  const int grid = C * std::max(1, std::min(B.ninst, nsm * std::max(per_sm, 1) / C));
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(kBlockThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = C;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = C > 1 ? 1 : 0;
  SCUDA(cudaLaunchKernelEx(&cfg, kern, B));
  return 0;
}

// The active instances of the block schedule, one launch per class, side by
// side on streams of their own joined into st.
template <class T>
int launch_block(SolverState *s, Krylov &k, const TDyNewtonOptions &o, double tol2, long long thr,
                 const std::vector<int> &act, cudaStream_t st) {
  int ierr, dev = 0, nsm = 0;
  SCUDA(cudaGetDevice(&dev));
  SCUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  auto cells = [&](int g) { return s->h_seg_off[g + 1] - s->h_seg_off[g]; };
  // matrix slots of a CTA's rows at most: its slices are as wide as the widest in HBM
  auto slots_of = [&](int C, int g) {
    long long width = 0;
    for (int k = s->h_slice_off[g]; k < s->h_slice_off[g + 1]; k++)
      width = std::max(width, s->h_sell_off[k + 1] - s->h_sell_off[k]);
    return (size_t)width * ((owned_cells(cells(g), C) + 31) / 32);
  };
  auto smem_of = [&](int keep, int C, int g) {
    const int nc = cells(g), nc2 = s->h_inst_line_off[g + 1] - s->h_inst_line_off[g];
    return block_smem<T>(keep, nc, (nc2 + C - 1) / C, nc / nc2, keep == KEEP_MATRIX ? slots_of(C, g) : 0, C);
  };
  long long total = 0, ctas = 0;
  for (int g = 0; g < s->nseg; g++)
    if (act[g] && on_block(s, thr, g)) total += cells(g);
  for (int g = 0; g < s->nseg; g++)
    if (act[g] && on_block(s, thr, g)) ctas += block_ctas(cells(g), total, nsm, sizeof(T));
  struct Class {
    std::vector<int> inst;
    size_t smem = 0, slots = 0;
  } cls[kBlockClasses];
  constexpr size_t slot_bytes = sizeof(T) + sizeof(uint16_t);  // of a matrix entry
  for (int g : s->h_order) {
    if (!act[g] || !on_block(s, thr, g)) continue;
    int c = block_ctas(cells(g), total, nsm, sizeof(T)), lg = c == 8 ? 3 : c == 4 ? 2 : c == 2 ? 1 : 0;
    while (lg < 3 && smem_of(KEEP_ALL, 1 << lg, g) > kBlockSmemMax) lg++;
    int i = -1, keep = KEEP_ALL;
    // the matrix in shared memory, in batches of many CTAs where it leaves two
    // per SM (28 instances up to 5,264 cells: 2.0 ms against 2.5 ms with the
    // half limit; 192 instances: 4.6 against 3.8 ms)
    size_t smem = smem_of(KEEP_MATRIX, 1 << lg, g), slots = slots_of(1 << lg, g);
    auto class_of = [&] {
      int step = 0;
      while (smem > kBlockSmemSteps[step]) step++;
      return ((3 - lg) * 2 + keep) * 3 + 2 - step;  // larger instances first
    };
    if (smem <= (ctas <= 2 * nsm ? kBlockSmemMax : kBlockSmemMax / 2)) {
      // (the matrix lies behind everything else: its slots are the class's,
      // and with them the whole class has to fit)
      keep = KEEP_MATRIX;
      i = class_of();
      const size_t all = std::max(cls[i].smem, smem - slot_bytes * slots) + slot_bytes * std::max(cls[i].slots, slots);
      if (all > kBlockSmemMax) i = -1;
    }
    if (i < 0) {
      keep = KEEP_ALL;
      slots = 0;
      smem = smem_of(KEEP_ALL, 1 << lg, g);
    }
    if (i >= 0) {
    } else if (smem <= kBlockSmemMax) {
      i = class_of();
    } else if ((smem = smem_of(KEEP_Z, 8, g)) <= kBlockSmemMax) {
      i = kBlockClasses - 2;
    } else {
      smem = smem_of(KEEP_NONE, 1, g);
      i = kBlockClasses - 1;
    }
    cls[i].inst.push_back(g);
    cls[i].slots = std::max(cls[i].slots, slots);
    cls[i].smem = std::max(cls[i].smem, smem - slot_bytes * slots);
  }
  for (Class &c : cls) c.smem += slot_bytes * c.slots;
  s->h_block_list.clear();
  int first[kBlockClasses], used = 0;
  for (int i = 0; i < kBlockClasses; i++) {
    first[i] = (int)s->h_block_list.size();
    s->h_block_list.insert(s->h_block_list.end(), cls[i].inst.begin(), cls[i].inst.end());
    used += !cls[i].inst.empty();
  }
  if (!used) return 0;
  SCUDA(cudaMemcpyAsync(s->block_inst, s->h_block_list.data(), sizeof(int) * s->h_block_list.size(),
                        cudaMemcpyHostToDevice, st));
  SCUDA(cudaMemsetAsync(s->ticket, 0, kBlockClasses * sizeof(int), st));
  BlockSolve<T> B;
  B.seg_off = s->seg_off;
  B.inst_line_off = s->inst_line_off;
  B.slice_off = s->slice_off;
  B.sell_off = s->sell_off;
  B.rowptr = s->rowptr;
  B.A = (const T *)k.sell;
  B.col = s->sell_col;
  B.la = (const T *)k.la;
  B.lcp = (const T *)k.lcp;
  B.linv = (const T *)k.linv;
  B.F = s->F;
  T *const vec[8] = {(T *)k.r0, (T *)k.r, (T *)k.p, (T *)k.v, (T *)k.s, (T *)k.t, (T *)k.ph, (T *)k.y};
  for (int i = 0; i < 8; i++) B.vec[i] = vec[i];
  B.z = (T *)k.sh;
  B.x = (T *)k.b;
  B.lin_its = s->lin_its;
  B.tol2 = tol2;
  B.max_it = o.linear_max_it;
  if (used > 1) {
    // (each by itself: an earlier solve may have got some of them only)
    s->device = dev;
    if (!s->fork && (ierr = device_pool_event(&s->fork))) return ierr;
    for (int i = 0; i < 3; i++) {
      if (!s->side[i] && (ierr = device_pool_stream(&s->side[i]))) return ierr;
      if (!s->joined[i] && (ierr = device_pool_event(&s->joined[i]))) return ierr;
    }
    SCUDA(cudaEventRecord(s->fork, st));
    for (int i = 0; i < std::min(used - 1, 3); i++) SCUDA(cudaStreamWaitEvent(s->side[i], s->fork, 0));
  }
  int launched = 0;
  for (int i = 0; i < kBlockClasses; i++) {
    if (cls[i].inst.empty()) continue;
    B.ninst = (int)cls[i].inst.size();
    B.inst = s->block_inst + first[i];
    B.ticket = s->ticket + i;
    const size_t smem = cls[i].smem;
    const cudaStream_t ls = launched % 4 == 0 ? st : s->side[launched % 4 - 1];
    B.slots = (int)cls[i].slots;
    switch (i / 3) {
      case 0: ierr = launch_block_class<T, 8, KEEP_MATRIX>(B, smem, nsm, ls); break;
      case 1: ierr = launch_block_class<T, 8, KEEP_ALL>(B, smem, nsm, ls); break;
      case 2: ierr = launch_block_class<T, 4, KEEP_MATRIX>(B, smem, nsm, ls); break;
      case 3: ierr = launch_block_class<T, 4, KEEP_ALL>(B, smem, nsm, ls); break;
      case 4: ierr = launch_block_class<T, 2, KEEP_MATRIX>(B, smem, nsm, ls); break;
      case 5: ierr = launch_block_class<T, 2, KEEP_ALL>(B, smem, nsm, ls); break;
      case 6: ierr = launch_block_class<T, 1, KEEP_MATRIX>(B, smem, nsm, ls); break;
      case 7: ierr = launch_block_class<T, 1, KEEP_ALL>(B, smem, nsm, ls); break;
      default:
        ierr = i == kBlockClasses - 2 ? launch_block_class<T, 8, KEEP_Z>(B, smem, nsm, ls)
                                      : launch_block_class<T, 1, KEEP_NONE>(B, smem, nsm, ls);
    }
    if (ierr) return ierr;
    launched++;
  }
  for (int i = 0; i < std::min(launched - 1, 3); i++) {
    SCUDA(cudaEventRecord(s->joined[i], s->side[i]));
    SCUDA(cudaStreamWaitEvent(st, s->joined[i], 0));
  }
  return 0;
}

// The active instances of the tile schedule: as many CTAs as the product has
// rows for, up to what the GPU holds at once.
template <class T, int TPR>
int launch_grid_tpr(const GridSolve<T> &G, int nsm, cudaStream_t st) {
  auto kern = bicgstab_grid_kernel<T, TPR>;
  int per_sm = 0;
  SCUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kGridThreads, 0));
  const long long want = ((long long)G.n * TPR + kGridThreads - 1) / kGridThreads;
  return launch_cooperative(kern, G, std::min(want, (long long)nsm * per_sm), kGridThreads, st);
}

// words of the tile schedule behind lin_its
inline size_t grid_words(const SolverState *s) { return GS_COUNT + (size_t)s->nchunks + s->nseg; }

template <class T>
int launch_grid(SolverState *s, Krylov &k, const TDyNewtonOptions &o, double tol2, cudaStream_t st) {
  int ierr, dev = 0, nsm = 0;
  SCUDA(cudaGetDevice(&dev));
  SCUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
  if (!s->grid_acc) {
    Arena ar;
    ar.work(&s->grid_acc, (size_t)s->nchunks * kGridSums * 256);
    ar.work(&s->grid_part, (size_t)s->nchunks * kGridSums);
    if ((ierr = ar.commit(st))) return ierr;
    s->allocs.push_back(ar.base);
  }
  GridSolve<T> G;
  G.n = s->n;
  G.ns = s->nseg;
  G.nchunks = s->nchunks;
  G.nlines = s->nlines;
  G.clusters = s->precond_used == TDY_PRECOND_CLUSTERS;
  G.ncl = G.clusters ? s->ncl : 0;
  G.cell_seg = s->cell_seg;
  G.newt_active = s->newt_active;
  G.block_mask = s->block_mask;
  G.chunk_off = s->chunk_off;
  G.seg_chunk = s->seg_chunk;
  G.rowptr = s->rowptr;
  G.colidx = s->colidx;
  G.A = (const T *)k.Jv;
  G.line_off = s->line_off;
  G.line_cells = s->line_cells;
  G.la = (const T *)k.la;
  G.lcp = (const T *)k.lcp;
  G.linv = (const T *)k.linv;
  G.cloc = s->cloc;
  G.coff = s->coff;
  G.cmem = s->cmem;
  G.cperm = s->cperm;
  G.cluoff = s->cluoff;
  G.cinv = (const T *)k.cinv;
  G.clu = (const T *)k.clu;
  G.F = s->F;
  G.r = (T *)k.r;
  G.r0 = (T *)k.r0;
  G.p = (T *)k.p;
  G.v = (T *)k.v;
  G.sv = (T *)k.s;
  G.tv = (T *)k.t;
  G.ph = (T *)k.ph;
  G.sh = (T *)k.sh;
  G.y = (T *)k.y;
  G.act = s->lin_active;
  G.its = s->lin_its;
  G.sc = s->scal;
  G.acc = s->grid_acc;
  G.part = s->grid_part;
  G.sync = s->grid_sync;
  G.tol2 = tol2;
  G.max_it = o.linear_max_it;
  switch (k.tpr) {
    case 1: return launch_grid_tpr<T, 1>(G, nsm, st);
    case 2: return launch_grid_tpr<T, 2>(G, nsm, st);
    case 4: return launch_grid_tpr<T, 4>(G, nsm, st);
    default: return launch_grid_tpr<T, 8>(G, nsm, st);
  }
}

// One linear solve with instances of at most `thr` cells on the block
// schedule and the others on the tile schedule; its = inner iterations.
template <class T>
int solve_scheduled(SolverState *s, Krylov &k, const TDyNewtonOptions &o, double tol2, long long thr,
                    const std::vector<int> &newt_act, cudaStream_t st, std::vector<int> &its) {
  int ierr;
  const int ns = s->nseg;
  if ((ierr = set_block_split(s, thr, st))) return ierr;
  SCUDA(cudaMemsetAsync(s->lin_its, 0, sizeof(int) * (ns + grid_words(s)), st));
  if (s->n_block > 0 && (ierr = launch_block<T>(s, k, o, tol2, thr, newt_act, st))) return ierr;
  if (s->n_tile > 0 && (ierr = launch_grid<T>(s, k, o, tol2, st))) return ierr;
  SCUDA(cudaEventRecord(s->tev[4], st));
  seg_norms<T>(s, (const T *)k.y, nullptr, s->y2, st);
  SCUDA(cudaGetLastError());
  const size_t bytes = sizeof(double) * ns + sizeof(int) * ns + sizeof(unsigned) * GS_COUNT;
  s->h_out.resize((bytes + 7) / 8);
  SCUDA(cudaMemcpyAsync(s->h_out.data(), s->y2, bytes, cudaMemcpyDeviceToHost, st));
  SCUDA(cudaStreamSynchronize(st));
  const char *tail = reinterpret_cast<const char *>(s->h_out.data() + ns);
  its.resize(ns);
  std::memcpy(its.data(), tail, sizeof(int) * ns);
  unsigned err;
  std::memcpy(&err, tail + sizeof(int) * ns + sizeof(unsigned) * GS_ERR, sizeof(err));
  if (err) return set_error(TDY_ERR_GPU, "solver: a wait of the tile schedule ran out");
  return 0;
}

// Schedule autotuner.  The first line-preconditioned solve of a size class
// (arithmetic, number of instances, largest instance) times the candidate
// splits on the solve at hand: all instances on the tile schedule, all on the
// block schedule, and splits at 4096, 16384 and 65536 cells where they
// separate the instances; the fastest split is kept for the class for the
// rest of the process.  The schedules give the same bits, so the choice
// changes only the time.
std::mutex g_sched_mutex;
std::vector<std::pair<long long, long long>> g_sched;  // (class key, split)

template <class T>
long long sched_key(const SolverState *s) {
  long long maxc = 0;
  for (int g = 0; g < s->nseg; g++) maxc = std::max<long long>(maxc, s->h_seg_off[g + 1] - s->h_seg_off[g]);
  int lg = 0;
  while ((1LL << lg) < maxc) lg++;
  const int cls = s->nseg == 1 ? 0 : (s->nseg < 64 ? 1 : 2);
  return ((long long)sizeof(T) << 16) | ((long long)cls << 8) | lg;
}

// The split already chosen for this handle or its size class; false if none.
template <class T>
bool tuned_schedule(const SolverState *s, Krylov &k, long long *thr) {
  if (k.block_max_cells == -2) {
    const long long key = sched_key<T>(s);
    std::lock_guard<std::mutex> lk(g_sched_mutex);
    for (auto &e : g_sched)
      if (e.first == key) k.block_max_cells = e.second;
  }
  *thr = k.block_max_cells;
  return k.block_max_cells != -2;
}

template <class T>
int tune_schedule(SolverState *s, Krylov &k, const TDyNewtonOptions &o, double tol2, const std::vector<int> &act,
                  cudaStream_t st, long long *thr) {
  const long long key = sched_key<T>(s);
  std::vector<long long> cand = {-1};
  if (s->nslices > 0) cand.push_back(LLONG_MAX);
  for (long long c : {4096LL, 16384LL, 65536LL}) {
    int below = 0;
    for (int g = 0; g < s->nseg; g++) below += (s->h_seg_off[g + 1] - s->h_seg_off[g]) <= c;
    if (below > 0 && below < s->nseg) cand.push_back(c);
  }
  std::vector<int> its;
  s->tune_ms.clear();
  double best = 1e300;
  long long best_thr = -1;
  for (long long c : cand) {
    int ierr;
    if ((ierr = solve_scheduled<T>(s, k, o, tol2, c, act, st, its))) return ierr;  // warm-up
    const auto t0 = std::chrono::steady_clock::now();
    if ((ierr = solve_scheduled<T>(s, k, o, tol2, c, act, st, its))) return ierr;
    const double ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    s->tune_ms.push_back(ms);
    if (ms < best) {
      best = ms;
      best_thr = c;
    }
  }
  {
    std::lock_guard<std::mutex> lk(g_sched_mutex);
    g_sched.emplace_back(key, best_thr);
  }
  k.block_max_cells = *thr = best_thr;
  return 0;
}

// act: the instances to solve (the host's copy of newt_active)
template <class T>
int linear_solve(SolverState *s, Krylov &k, const TDyNewtonOptions &o, const std::vector<int> &act, cudaStream_t st,
                 long long *lin_total, std::vector<int> &inst_lin_its) {
  int ierr;
  if ((ierr = krylov_alloc<T>(s, k, st))) return ierr;
  // the schedule split: given by the options, chosen before, or (lines, below)
  // by timing on the first solve of this size class; clusters: tile only
  long long thr = -1;
  bool tune = false;
  if (o.precond != TDY_PRECOND_CLUSTERS) {
    if (o.schedule == TDY_SCHEDULE_BLOCK)
      thr = LLONG_MAX;
    else if (o.schedule != TDY_SCHEDULE_TILE)
      tune = !tuned_schedule<T>(s, k, &thr);
    // (FP64 solves within an FP32 step are of the few instances that need
    // them: too few to time the class on, so they follow the FP32 split)
    if (tune && sizeof(T) == 8 && o.linear_fp32) tune = !tuned_schedule<float>(s, s->k32, &thr);
  }
  bool tile = tune, block = tune && s->nslices > 0;
  if (!tune)
    for (int g = 0; g < s->nseg; g++) (on_block(s, thr, g) ? block : tile) = true;
  if (block) {
    if ((ierr = sell_setup(s, st))) return ierr;
    if (!k.sell) {
      if ((ierr = dmem_alloc(&k.sell, (size_t)s->h_sell_off.back() * sizeof(T), st))) return ierr;
      s->allocs.push_back(k.sell);
    }
  }
  if (tile) {
    if (!k.Jv) {
      if ((ierr = dmem_alloc(&k.Jv, (size_t)s->nnz * sizeof(T), st))) return ierr;
      s->allocs.push_back(k.Jv);
    }
    if ((ierr = autotune_spmv<T>(s, k, o.spmv_threads, st))) return ierr;  // uses b and v as scratch before they are set
  }
  const int ns = s->nseg;
  SCUDA(cudaEventRecord(s->tev[2], st));
  if (tile) cast_kernel<T><<<nblk(s->nnz, 256), 256, 0, st>>>(s->nnz, s->J, (T *)k.Jv);
  if (block)
    sell_fill_kernel<T, double><<<nblk(s->nslices, kSliceWarps), 32 * kSliceWarps, 0, st>>>(
        s->nslices, s->slice_row, s->slice_end, s->sell_off, s->cell_seg, s->newt_active, s->seg_off, s->rowptr, s->J,
        (T *)k.sell);
  s->precond_used = TDY_PRECOND_LINES;
  if (o.precond == TDY_PRECOND_CLUSTERS && (ierr = cluster_setup<T>(s, k, o.cluster_threshold, st))) return ierr;
  if (s->precond_used == TDY_PRECOND_LINES)
    line_factor_kernel<T><<<nblk(s->nlines, 128), 128, 0, st>>>(s->nlines, s->line_off, s->line_cells, s->pos_d,
                                                                 s->pos_lo, s->pos_hi, s->J, (T *)k.la, (T *)k.lcp,
                                                                 (T *)k.linv);
  SCUDA(cudaEventRecord(s->tev[3], st));
  const double tol2 = o.linear_rtol * o.linear_rtol;
  std::vector<int> its(ns);
  if (tune && (ierr = tune_schedule<T>(s, k, o, tol2, act, st, &thr))) return ierr;
  if ((ierr = solve_scheduled<T>(s, k, o, tol2, thr, act, st, its))) return ierr;
  for (int v : its) *lin_total += v;
  inst_lin_its = its;
  return 0;
}

int solver_init(_p_TDy *t) {
  if (t->solver) return 0;
  const MPFAOSetup &su = t->setup;
  SolverState *s = new SolverState();
  t->solver = s;
  s->st = (cudaStream_t)device_default_stream(t);
  for (cudaEvent_t &e : s->tev) SCUDA(cudaEventCreate(&e));
  s->n = t->mesh.nc;
  s->nnz = (int)su.colidx.size();
  // instances: the mesh blocks; lines: the columns of each block, bottom to top
  std::vector<int> seg_off(1, 0), cell_seg(s->n), line_off(1, 0), line_cells, pd, plo, phi;
  line_cells.reserve(s->n);
  auto find = [&](int i, int j) {
    const int *b = su.colidx.data() + su.rowptr[i], *e = su.colidx.data() + su.rowptr[i + 1];
    const int *q = std::lower_bound(b, e, j);
    return (q != e && *q == j) ? (int)(q - su.colidx.data()) : -1;
  };
  int c0 = 0;
  std::vector<int> inst_line_off(1, 0);
  for (const ExtrudedInput &blk : t->mesh_blocks) {
    const int nc2 = blk.nc2, nl = blk.nlayers;
    inst_line_off.push_back(inst_line_off.back() + nc2);
    for (int c2 = 0; c2 < nc2; c2++) {
      for (int k = 0; k < nl; k++) {
        const int i = c0 + k * nc2 + c2;
        line_cells.push_back(i);
        pd.push_back(find(i, i));
        plo.push_back(k > 0 ? find(i, i - nc2) : -1);
        phi.push_back(k + 1 < nl ? find(i, i + nc2) : -1);
        if (pd.back() < 0) return set_error(TDY_ERR_LIB, "solver: missing diagonal of cell %d", i);
      }
      line_off.push_back((int)line_cells.size());
    }
    for (int i = c0; i < c0 + nc2 * nl; i++) cell_seg[i] = (int)seg_off.size() - 1;
    c0 += nc2 * nl;
    seg_off.push_back(c0);
  }
  if (c0 != s->n) return set_error(TDY_ERR_LIB, "solver: blocks cover %d of %d cells", c0, s->n);
  s->nseg = (int)seg_off.size() - 1;
  s->nlines = (int)line_off.size() - 1;
  std::vector<int> chunk_off(1, 0), seg_chunk(1, 0);
  for (int g = 0; g < s->nseg; g++) {
    for (int i = seg_off[g]; i < seg_off[g + 1]; i += kChunk) chunk_off.push_back(std::min(i + kChunk, seg_off[g + 1]));
    seg_chunk.push_back((int)chunk_off.size() - 1);
  }
  s->nchunks = (int)chunk_off.size() - 1;
  // slices of the block schedule's matrix layout
  s->h_slice_off.assign(1, 0);
  s->h_sell_off.assign(1, 0);
  for (int g = 0; g < s->nseg; g++) {
    if (seg_off[g + 1] - seg_off[g] <= kBlockCap)
      for (int i = seg_off[g]; i < seg_off[g + 1]; i += 32) {
        int width = 0;
        for (int j = i; j < std::min(i + 32, seg_off[g + 1]); j++)
          width = std::max(width, su.rowptr[j + 1] - su.rowptr[j]);
        s->h_slice_row.push_back(i);
        s->h_sell_off.push_back(s->h_sell_off.back() + 32LL * width);
      }
    s->h_slice_off.push_back((int)s->h_slice_row.size());
  }
  s->nslices = (int)s->h_slice_row.size();
  s->h_seg_off = seg_off;
  s->h_inst_line_off = inst_line_off;
  s->h_order.resize(s->nseg);
  for (int g = 0; g < s->nseg; g++) s->h_order[g] = g;
  std::stable_sort(s->h_order.begin(), s->h_order.end(),
                   [&](int x, int y) { return seg_off[x + 1] - seg_off[x] > seg_off[y + 1] - seg_off[y]; });
  int ierr;
  // every array in one allocation, uploaded with one copy
  std::vector<int> dp(s->n);
  for (int i = 0; i < s->n; i++) dp[i] = find(i, i);  // every row has its diagonal (checked above per line cell)
  Arena ar;
  ar.up(&s->rowptr, su.rowptr);
  ar.up(&s->colidx, su.colidx);
  ar.up(&s->seg_off, seg_off);
  ar.up(&s->chunk_off, chunk_off);
  ar.up(&s->seg_chunk, seg_chunk);
  ar.work(&s->part, 2 * (size_t)s->nchunks);
  ar.up(&s->cell_seg, cell_seg);
  ar.up(&s->line_off, line_off);
  ar.up(&s->line_cells, line_cells);
  ar.up(&s->pos_d, pd);
  ar.up(&s->dpos, dp);
  ar.up(&s->pos_lo, plo);
  ar.up(&s->pos_hi, phi);
  ar.work(&s->x, s->n);
  ar.work(&s->xb, s->n);
  ar.work(&s->lam, s->nseg + (s->nseg + 1) / 2);  // then trial, copied with it
  ar.work(&s->commit, s->nseg);
  ar.work(&s->F, s->n);
  ar.work(&s->J, s->nnz);
  ar.work(&s->norms, 2 * s->nseg);
  ar.work(&s->scal, (size_t)S_NSCAL * s->nseg);
  ar.work(&s->newt_active, s->nseg);
  ar.work(&s->lin_active, s->nseg);
  ar.work(&s->y2, s->nseg + (s->nseg + grid_words(s) + 1) / 2);  // then lin_its and grid_sync
  ar.up(&s->inst_line_off, inst_line_off);
  ar.work(&s->block_inst, s->nseg);
  ar.work(&s->block_mask, s->nseg);
  ar.work(&s->ticket, kBlockClasses);
  if ((ierr = ar.commit(s->st))) return ierr;
  s->allocs.push_back(ar.base);
  s->trial = reinterpret_cast<int *>(s->lam + s->nseg);
  s->lin_its = reinterpret_cast<int *>(s->y2 + s->nseg);
  s->grid_sync = reinterpret_cast<unsigned *>(s->lin_its + s->nseg);
  // the allocations and uploads complete before any other stream uses them
  // (and before the host vectors above go out of scope)
  SCUDA(cudaStreamSynchronize(s->st));
  return 0;
}

}  // namespace

void device_solver_destroy(_p_TDy *t) {
  delete t->solver;
  t->solver = nullptr;
}

int device_num_instances(_p_TDy *t) { return (int)t->mesh_blocks.size(); }

// the last linear_solve's set-up and Krylov times (ms), once its events completed
static int add_linear_times(SolverState *s, double *prec, double *kry) {
  SCUDA(cudaEventSynchronize(s->tev[4]));
  float m1 = 0.f, m2 = 0.f;
  SCUDA(cudaEventElapsedTime(&m1, s->tev[2], s->tev[3]));
  SCUDA(cudaEventElapsedTime(&m2, s->tev[3], s->tev[4]));
  *prec += m1;
  *kry += m2;
  return 0;
}

static int be_solve(_p_TDy *t, double dt, double *dU, const TDyNewtonOptions &o, TDyNewtonStats *stats,
                    int *inst_its, double *inst_rel, cudaStream_t st) {
  int ierr;
  SolverState *s = t->solver;
  const int n = s->n, ns = s->nseg;
  t->dtime = dt;
  if ((ierr = device_presolve(t, dU, st, true))) return ierr;
  SCUDA(cudaMemcpyAsync(s->x, dU, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
  SCUDA(cudaMemcpyAsync(s->xb, dU, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
  std::vector<double> f0(ns, 0.0), fn(ns, 0.0), g2(2 * ns, 0.0);  // (g2: of F, then of x)
  std::vector<char> lam_trial((sizeof(double) + sizeof(int)) * ns);  // packed as on the device
  double *const lam = reinterpret_cast<double *>(lam_trial.data());
  int *const trial = reinterpret_cast<int *>(lam + ns);
  std::vector<int> act(ns, 1), its(ns, 0), commit(ns, 0), step_conv(ns, 0), failed(ns, 0);
  // instances retired by the caller are not advanced (TDySetActiveInstances)
  const bool masked = (int)t->inst_active.size() == ns;
  std::vector<int> live;
  for (int g = 0; g < ns; g++) {
    if (masked && !t->inst_active[g]) act[g] = 0;
    if (act[g]) live.push_back(g);
  }
  std::vector<double> y2(ns, 0.0), x2(ns, 0.0);
  std::vector<int> lin_its(ns, 0);  // inner iterations of the last solve, per instance
  long long lin_total = 0;
  int fell_back = 0;
  std::vector<int> trial_list;
  double t_eval = 0.0, t_prec = 0.0, t_kry = 0.0;  // ms on the stream
  int inner_redo = 0;  // FP32 inner solves redone in FP64 (instances x Newton iterations)
  // F and J at x (= xb for every instance after each evaluation below), and
  // the squared per-instance norms of F and x into g2
  // `sub` (host list of instances, or null for all): only those instances'
  // states changed since the last evaluation, the others keep F and J
  auto evaluate = [&](const std::vector<int> *sub = nullptr) -> int {
    int e;
    const bool part = sub && (int)sub->size() < ns && device_inst_ok(t);
    SCUDA(cudaEventRecord(s->tev[0], st));
    if (part)
      e = device_eval_instances(t, s->x, s->F, s->J, sub->data(), (int)sub->size(), st, true);
    else
      e = device_eval(t, FORM_SNES, 0.0, s->x, nullptr, 0.0, s->F, s->J, st, true);
    if (e) return e;
    SCUDA(cudaEventRecord(s->tev[1], st));
    seg_norms<double>(s, s->F, s->x, s->norms, st);
    SCUDA(cudaGetLastError());
    SCUDA(cudaMemcpyAsync(g2.data(), s->norms, sizeof(double) * 2 * ns, cudaMemcpyDeviceToHost, st));
    SCUDA(cudaStreamSynchronize(st));
    float ms = 0.f;
    SCUDA(cudaEventElapsedTime(&ms, s->tev[0], s->tev[1]));
    t_eval += ms;
    return 0;
  };
  if ((ierr = evaluate(masked ? &live : nullptr))) return ierr;
  for (int g = 0; g < ns; g++) {
    f0[g] = fn[g] = std::sqrt(g2[g]);
    x2[g] = g2[ns + g];
  }
  const double alpha = 1e-4;  // sufficient-decrease constant of PETSc's backtracking line search
  constexpr double kMaxStep = 1e8;  // PETSc's default SNESLineSearch maxstep
  const int max_backtracks = 12;
  for (int it = 0;; it++) {
    bool any = false;
    for (int g = 0; g < ns; g++) {
      if (act[g]) {
        if (!std::isfinite(fn[g]) || !std::isfinite(f0[g])) {  // diverged: stop, reported as not converged
          act[g] = 0;
          failed[g] = 1;
          continue;
        }
        const bool done = !(fn[g] > o.atol) || fn[g] <= o.rtol * f0[g];
        if (done || it == o.max_it) act[g] = 0;  // converged, or out of iterations (reported below)
        else its[g] = it + 1;
      }
      any |= act[g] != 0;
    }
    if (!any) break;
    SCUDA(cudaMemcpyAsync(s->newt_active, act.data(), sizeof(int) * ns, cudaMemcpyHostToDevice, st));
    // FP32 inner solves for the first fp32_max_it Newton iterations, FP64 after
    // (an instance still iterating then is one whose FP32 directions stall;
    // the switch depends only on the iteration number, so an instance takes it
    // at the same point alone and in a batch)
    const bool fp32 = o.linear_fp32 && (o.fp32_max_it < 0 || it < o.fp32_max_it);
    if (o.linear_fp32 && !fp32) fell_back = 1;
    const void *y;
    if (fp32) {
      // FP32 inner solves stop after a quarter of linear_max_it (at least 20
      // iterations); one that runs out (FP32 rounding can stall BiCGStab
      // above the tolerance on ill-conditioned Jacobians) is solved again in
      // FP64 with the full count, and the instance steps along that direction
      // (kept in the FP32 array).  The choice depends on the instance alone,
      // so it is the same alone and in a batch.
      TDyNewtonOptions o32 = o;
      o32.linear_max_it = std::min(o.linear_max_it, std::max(20, o.linear_max_it / 4));
      ierr = linear_solve<float>(s, s->k32, o32, act, st, &lin_total, lin_its);
      if (ierr) return ierr;
      if ((ierr = add_linear_times(s, &t_prec, &t_kry))) return ierr;
      std::vector<int> redo(ns, 0);
      bool any_redo = false;
      for (int g = 0; g < ns; g++)
        if (act[g] && lin_its[g] >= o32.linear_max_it) any_redo = redo[g] = 1;
      if (any_redo) {
        SCUDA(cudaMemcpyAsync(s->newt_active, redo.data(), sizeof(int) * ns, cudaMemcpyHostToDevice, st));
        std::vector<int> lin64;
        if ((ierr = linear_solve<double>(s, s->k64, o, redo, st, &lin_total, lin64))) return ierr;
        if ((ierr = add_linear_times(s, &t_prec, &t_kry))) return ierr;
        cast_masked_kernel<<<nblk(n, 256), 256, 0, st>>>(n, s->cell_seg, s->newt_active, (const double *)s->k64.y,
                                                         (float *)s->k32.y);
        SCUDA(cudaMemcpyAsync(s->newt_active, act.data(), sizeof(int) * ns, cudaMemcpyHostToDevice, st));
        seg_norms<float>(s, (const float *)s->k32.y, nullptr, s->y2, st);
        SCUDA(cudaGetLastError());
        SCUDA(cudaMemcpyAsync(s->h_out.data(), s->y2, sizeof(double) * ns, cudaMemcpyDeviceToHost, st));
        SCUDA(cudaStreamSynchronize(st));  // redo and act (host vectors) stay valid until here
        for (int g = 0; g < ns; g++)
          if (redo[g]) {
            lin_its[g] = lin64[g];
            inner_redo++;
          }
      }
      y = s->k32.y;
    } else {
      ierr = linear_solve<double>(s, s->k64, o, act, st, &lin_total, lin_its);
      if (!ierr) ierr = add_linear_times(s, &t_prec, &t_kry);
      y = s->k64.y;
    }
    if (ierr) return ierr;
    // ||y|| and ||x|| before the step (y2 and x2, from the solve and the last
    // accepted evaluation): PETSc's backtracking line search caps the step at
    // maxstep and ends with convergence by the step test when the full step
    // fails and ||y|| < stol ||x||
    for (int g = 0; g < ns; g++) y2[g] = s->h_out[g];
    // backtracking per instance: accept when ||F(x - lam y)||^2 <= (1 - 2 alpha lam) ||F(x)||^2
    // (initial slope -||F||^2 of the Newton direction), else a quadratic fit of
    // lam clamped to [0.1 lam, 0.5 lam] (PETSc SNESLineSearchApply_BT)
    for (int g = 0; g < ns; g++) {
      trial[g] = act[g];
      // ||lam y|| <= maxstep (SNESLineSearch maxstep, PETSc default 1e8): a
      // direction from a diverged inner solve cannot throw the state away
      const double yn = std::sqrt(y2[g]);
      lam[g] = yn > kMaxStep ? kMaxStep / yn : 1.0;
    }
    for (int ls = 0; ls <= max_backtracks; ls++) {
      SCUDA(cudaMemcpyAsync(s->lam, lam, (sizeof(double) + sizeof(int)) * ns, cudaMemcpyHostToDevice, st));
      if (fp32)
        trial_kernel<float><<<nblk(n, 256), 256, 0, st>>>(n, s->cell_seg, s->trial, s->lam, (const float *)y, s->xb,
                                                          s->x);
      else
        trial_kernel<double><<<nblk(n, 256), 256, 0, st>>>(n, s->cell_seg, s->trial, s->lam, (const double *)y, s->xb,
                                                           s->x);
      trial_list.clear();
      for (int g = 0; g < ns; g++)
        if (trial[g]) trial_list.push_back(g);
      if ((ierr = evaluate(&trial_list))) return ierr;
      bool pending = false;
      for (int g = 0; g < ns; g++) {
        commit[g] = 0;
        if (!trial[g]) continue;
        const double f = fn[g] * fn[g], gg = g2[g];
        const bool inner_ok = lin_its[g] < o.linear_max_it;
        if (std::isfinite(gg) &&
            (gg <= (1.0 - 2.0 * alpha * lam[g]) * f || (ls == max_backtracks && (inner_ok || gg <= 4.0 * f)))) {
          // sufficient decrease; or, at the smallest step, a Newton direction
          // from a converged inner solve (the next iteration's Jacobian at the
          // nearby state usually gives a better one; at the FP64 noise floor
          // no step lowers ||F|| and the step test ends the instance), or one
          // from an unconverged inner solve that at most doubles ||F||
          commit[g] = 1;
          trial[g] = 0;
          fn[g] = std::sqrt(gg);
          x2[g] = g2[ns + g];
        } else if (ls == max_backtracks) {
          // no finite residual along the step, or an unconverged inner solve
          // whose smallest step more than doubles ||F||: keep the last
          // accepted state and stop, converged by the step test if the step
          // is negligible, else failed
          trial[g] = 0;
          act[g] = 0;
          if (o.stol > 0.0 && std::sqrt(y2[g]) < o.stol * std::sqrt(x2[g]))
            step_conv[g] = 1;
          else
            failed[g] = 1;
        } else {
          const double slope = -f;
          double lt = std::isfinite(gg) ? -slope * lam[g] * lam[g] / (gg - f - 2.0 * slope * lam[g]) : 0.0;
          lt = std::min(lt, 0.5 * lam[g]);
          lam[g] = (lt <= 0.1 * lam[g]) ? 0.1 * lam[g] : lt;
          pending = true;
        }
      }
      SCUDA(cudaMemcpyAsync(s->commit, commit.data(), sizeof(int) * ns, cudaMemcpyHostToDevice, st));
      commit_kernel<<<nblk(n, 256), 256, 0, st>>>(n, s->cell_seg, s->commit, s->x, s->xb);
      SCUDA(cudaGetLastError());
      if (!pending) break;
    }
    // every instance still active now has x == xb, so its F and J rows hold
    // the accepted state (instances do not couple).
    // Step test (SNESConvergedDefault): ||y|| < stol ||x|| per instance, with
    // y the full Newton step (PETSc's backtracking line search reports the
    // norm of the step before its lambda scaling), so a step cut short by the
    // line search does not count as convergence.
    if (o.stol > 0.0)
      for (int g = 0; g < ns; g++)
        if (act[g] && std::sqrt(y2[g]) < o.stol * std::sqrt(x2[g])) {
          act[g] = 0;
          step_conv[g] = 1;
        }
  }
  SCUDA(cudaMemcpyAsync(dU, s->xb, sizeof(double) * n, cudaMemcpyDeviceToDevice, st));
  SCUDA(cudaStreamSynchronize(st));
  int conv = 0, conv_step = 0, maxit = 0;
  t->inst_status.assign(ns, TDY_INSTANCE_NOT_CONVERGED);
  double worst = 0.0;
  for (int g = 0; g < ns; g++) {
    const bool retired = masked && !t->inst_active[g];
    const double rel = (f0[g] > 0.0 && !retired) ? fn[g] / f0[g] : 0.0;
    const bool fin = !retired && !failed[g] && std::isfinite(fn[g]);
    const bool ok = fin && (!(fn[g] > o.atol) || rel <= o.rtol);
    conv += ok ? 1 : 0;
    conv_step += (fin && !ok && step_conv[g]) ? 1 : 0;
    t->inst_status[g] = retired ? TDY_INSTANCE_INACTIVE
                                : ok ? TDY_INSTANCE_CONVERGED
                                     : (fin && step_conv[g]) ? TDY_INSTANCE_STEP_TEST : TDY_INSTANCE_NOT_CONVERGED;
    worst = std::max(worst, rel);
    maxit = std::max(maxit, its[g]);
    if (inst_its) inst_its[g] = its[g];
    if (inst_rel) inst_rel[g] = rel;
  }
  if (stats) {
    stats->newton_iterations = maxit;
    stats->linear_iterations = lin_total;
    stats->converged = conv;
    stats->ninstances = ns;
    stats->max_rel_residual = worst;
    stats->step_converged = conv_step;
    stats->precond_used = s->precond_used;
    stats->clusters = s->precond_used == TDY_PRECOND_CLUSTERS ? s->ncl : 0;
    stats->cluster_cells = s->precond_used == TDY_PRECOND_CLUSTERS ? s->ncl_cells : 0;
    stats->cluster_cells_diagonal = s->precond_used == TDY_PRECOND_CLUSTERS ? s->ncl_big_cells : 0;
    stats->fp64_fallback = fell_back;
    stats->eval_schedule = 0;
    stats->eval_s = 1e-3 * t_eval;
    stats->precond_s = 1e-3 * t_prec;
    stats->krylov_s = 1e-3 * t_kry;
    stats->fp64_inner_redo = inner_redo;
    stats->block_instances = s->precond_used == TDY_PRECOND_LINES ? s->n_block : 0;
    stats->block_max_cells = s->precond_used == TDY_PRECOND_LINES ? s->mask_for : -1;
  }
  return 0;
}

int device_be_solve(_p_TDy *t, double dt, double *dU, const TDyNewtonOptions &o, TDyNewtonStats *stats,
                    int *inst_its, double *inst_rel, void *stream) {
  int ierr;
  if ((ierr = solver_init(t))) {
    device_solver_destroy(t);
    return ierr;
  }
  // the caller's stream, else the handle's own
  cudaStream_t st = (cudaStream_t)(stream ? stream : device_default_stream(t));
  ierr = be_solve(t, dt, dU, o, stats, inst_its, inst_rel, st);
  if (ierr) {
    // some of the solve may still run, on the side streams without a join: its
    // memory and its streams are free for other uses once this returns
    for (cudaStream_t side : t->solver->side)
      if (side) cudaStreamSynchronize(side);
    cudaStreamSynchronize(st);
  }
  return ierr;
}

}  // namespace tdy
