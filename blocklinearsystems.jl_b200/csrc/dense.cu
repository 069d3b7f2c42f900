// Dense Cholesky factorisation and solve of the reduced system on sm_100a: the reduced solve that follows
// reduce_schur_dense! when S is small enough to hold dense (the reference hands its dense S to DampedLinearSolve's
// Cholesky, src/schur_linear_systems.jl:312-320). S is read from its upper triangle in its storage type (FP64 or the
// mixed form's FP32) into the lower triangle of an FP64 working matrix owned by the solver, padded to whole 64 x 64
// tiles with an identity, and factored in place as S = L L' by a blocked Cholesky: panels of 64 columns in groups of
// four. One CTA factors the diagonal tiles one after the other; beside it, the rows below a tile are solved against it and
// the panel updates the group's remaining columns and the next group's first one (rank 64), and a finished group updates everything right of
// those (rank 256) beside the next panels. A pivot that is not positive (or
// not finite) stops the factorisation; its column is reported, 1-based. The solve is one cooperative kernel: a CTA owns
// tiles of 64 rows, the tiles' solutions pass from owner to all others through memory.
#include <algorithm>
#include <cmath>
#include <memory>
#include <type_traits>

#include "common.cuh"

namespace bls {

constexpr int NB = 64;      // panel width and tile size
constexpr int GROUP = 4;    // panels per group
constexpr int TS = NB + 2;  // row stride of a tile in shared memory (16-byte rows)

constexpr int64_t kWaitLimit = 1 << 22;   // some seconds

struct DenseSolver {
  bls_ctx* ctx = nullptr;
  int64_t n = 0, ld = 0;   // ld: n rounded up to whole tiles, the order and leading dimension of W
  DevBuf mem;      // what follows, in one allocation (a solver's creation and destruction cost what its allocations do)
  double* W = nullptr;        // ld x ld FP64, column-major; L in its lower triangle after a successful factorisation
  double* rows = nullptr;     // the 64 rows below the next diagonal tile, two buffers
  double* dinv = nullptr;     // 1 / L[j, j]
  double* inv = nullptr;      // per panel the inverse of its 64 x 64 diagonal tile (column-major), for the solve
  long long* status = nullptr;   // [0]: first failing column (0-based) or -1; [1]: 1 after a solve whose wait gave up
  int64_t wait_limit = kWaitLimit;   // polls of a value before a wait of the solve gives up
  bool factored = false;
  bool prepared = false;   // k_step's shared-memory limit is set
  // The diagonal tiles run on one high-priority stream, the panels below them and the updates they wait for on another,
  // while the rest of a group's update runs on the caller's stream (created at the first factorisation).
  cudaStream_t panel_stream = nullptr;
  cudaStream_t update_stream = nullptr;
  cudaEvent_t ev_join = nullptr, ev_panel = nullptr, ev_next = nullptr, ev_tile = nullptr, ev_update = nullptr;
  int panel_priority = 0;
  // Everything after the load of S (the launches depend on n only) as one CUDA graph, captured at the first
  // factorisation; the panel kernels carry the high priority as a launch attribute, so the graph keeps it.
  cudaStream_t cap_stream = nullptr;
  cudaGraphExec_t factor_graph = nullptr;
  double* y = nullptr;    // the solve's exchange: ld forward and ld backward values, all bits set until written
  int solve_grid = 0;     // resident CTAs of k_solve (set at the first solve)
  ~DenseSolver() {
    if (factor_graph) cudaGraphExecDestroy(factor_graph);
    if (cap_stream) cudaStreamDestroy(cap_stream);
    if (ev_join) cudaEventDestroy(ev_join);
    if (ev_panel) cudaEventDestroy(ev_panel);
    for (cudaEvent_t e : {ev_next, ev_tile, ev_update})
      if (e) cudaEventDestroy(e);
    if (update_stream) cudaStreamDestroy(update_stream);
    if (panel_stream) cudaStreamDestroy(panel_stream);
  }
};

// The lower triangle of W = S' (S's upper triangle), in FP64, plus lambda s_r[j] on the diagonal when s_r is given, and
// the identity in the padding; a CTA per 32 x 32 tile on or below the diagonal, turned in shared memory so that both
// sides are read and written in contiguous runs.
template <class T>
__global__ void __launch_bounds__(256) k_dense_load(int64_t n, int64_t ld, const T* __restrict__ S, double* __restrict__ W, double lambda,
                                                    const double* __restrict__ s_r, double* __restrict__ rows, long long* __restrict__ status) {
  __shared__ double t[32][33];
  if (blockIdx.x == 0 && blockIdx.y == 0 && threadIdx.x == 0) status[0] = -1;
  if (blockIdx.y > blockIdx.x) return;
  const int64_t i0 = 32 * (int64_t)blockIdx.x, j0 = 32 * (int64_t)blockIdx.y;   // rows i0.., columns j0.. of W
  const int x = threadIdx.x & 31, y = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < 32; k += 8) {
    const int64_t j = j0 + x, i = i0 + y + k;
    t[y + k][x] = j <= i && i < n ? (double)S[j + n * i] : i == j ? 1.0 : 0.0;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 32; k += 8) {
    const int64_t i = i0 + x, j = j0 + y + k;
    double v = t[x][y + k];
    if (s_r && i == j && i < n) v += lambda * s_r[j];
    W[i + ld * j] = v;
    if (j0 < NB && i0 >= NB && i0 < 2 * NB) rows[(i - NB) + NB * j] = v;   // the rows below tile 0, for the first k_step
  }
}

// The lower triangle of the diagonal tile [d0, d0 + 64) of W into t by 256 threads, all 16 loads of a thread in flight
// (zeros above the diagonal)
__device__ __forceinline__ void load_tile(double (*t)[TS], const double* __restrict__ W, int64_t ld, int64_t d0, int tid) {
  double v[NB * NB / 256];
#pragma unroll
  for (int k = 0; k < NB * NB / 256; ++k) {
    const int e = tid + 256 * k, rr = e & 63, cc = e >> 6;
    v[k] = cc <= rr ? W[(d0 + rr) + ld * (d0 + cc)] : 0.0;
  }
#pragma unroll
  for (int k = 0; k < NB * NB / 256; ++k) {
    const int e = tid + 256 * k;
    t[e & 63][e >> 6] = v[k];
  }
}

// An asynchronous 8-byte global -> shared copy (cp.async).
__device__ __forceinline__ void cp_async8(double* smem, const double* gmem) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}

// The diagonal tile T (lower triangle, in shared memory) factored in place by 256 threads, by 16-column sub-panels: warps 0
// and 1 factor a sub-panel's rows (lane i holds row c0 + i, in warp 1 row c0 + 32 + i, of its 16 columns in registers): per
// column warp 0 forms L[j, j] = pivot * rsqrt(pivot) and the entries below it, which go to T, and both warps update their
// rows with them, read back as broadcasts; the next pivot is row j + 1's own, so the chain of a column is rsqrt, a product,
// the exchange through shared memory and one multiply-add. The test of a pivot is off it: a bad one only makes what follows
// useless. (One warp holding two rows a lane and shuffling the 15 entries of a column: a 64-bit shuffle takes 11 cycles of
// issue and an FP64 multiply-add 5, 430 cycles a column.) Then all warps subtract the sub-panel's rank-16
// product from the rest of the tile (3 x 3 entries a thread, or 2 x 2, or one). The sub-panels from column `cols` on are the
// identity padding and stay as they are. Returns (to every thread) the first column whose pivot is not positive or not finite, or -1.
template <int NA>
__device__ __forceinline__ void rank16(double (*T)[TS], int c0, int tid) {   // rows and columns c0 + 16 .. c0 + 16 + 16 NA
  const int tx = tid & 15, ty = tid >> 4, base = c0 + 16;
  double acc[NA][NA];
#pragma unroll
  for (int a = 0; a < NA; ++a)
#pragma unroll
    for (int b = 0; b < NA; ++b) acc[a][b] = 0.0;
#pragma unroll
  for (int c = 0; c < 16; c += 2) {
    double2 x[NA], y[NA];
#pragma unroll
    for (int a = 0; a < NA; ++a) {
      x[a] = *reinterpret_cast<const double2*>(&T[base + tx + 16 * a][c0 + c]);
      y[a] = *reinterpret_cast<const double2*>(&T[base + ty + 16 * a][c0 + c]);
    }
#pragma unroll
    for (int a = 0; a < NA; ++a)
#pragma unroll
      for (int b = 0; b <= a; ++b) acc[a][b] = fma(x[a].y, y[b].y, fma(x[a].x, y[b].x, acc[a][b]));
  }
#pragma unroll
  for (int a = 0; a < NA; ++a)
#pragma unroll
    for (int b = 0; b <= a; ++b)
      if (a > b || ty <= tx) T[base + tx + 16 * a][base + ty + 16 * b] -= acc[a][b];
}

__device__ int factor_tile(double (*T)[TS], double* dv, int* failed, int cols) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int c0 = 0; c0 < cols; c0 += 16) {
    if (warp < 2) {
      const int r = c0 + 32 * warp + lane;
      const bool own = r < NB;
      double a[16];
#pragma unroll
      for (int k = 0; k < 16; ++k) a[k] = own ? T[r][c0 + k] : 0.0;
      int bad = -1;
      double d = __shfl_sync(0xffffffffu, a[0], 0);   // warp 0: the pivot
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        double l = 0.0;
        if (warp == 0) {
          if (bad < 0 && (!(d > 0.0) || !isfinite(d))) bad = c0 + j;   // uniform
          const double inv = rsqrt(d);
          l = a[j] * inv;
          if (own && lane >= j) T[r][c0 + j] = l;
          if (lane == j) dv[c0 + j] = inv;
          if (j < 15) d = __shfl_sync(0xffffffffu, fma(-l, l, a[j + 1 < 16 ? j + 1 : 15]), j + 1);
        }
        asm volatile("bar.sync 1, 64;" ::: "memory");   // column j is in T for both warps
        if (warp == 1) {
          l = a[j] * dv[c0 + j];
          if (own) T[r][c0 + j] = l;
        }
#pragma unroll
        for (int k = j + 1; k < 16; ++k) a[k] = fma(-l, T[c0 + k][c0 + j], a[k]);
      }
      if (tid == 0) *failed = bad;
    }
    __syncthreads();
    if (*failed >= 0) return *failed;   // uniform
    const bool more = c0 + 16 < cols;
    if (more) {
      if (c0 == 0) rank16<3>(T, 0, tid);
      else if (c0 == 16) rank16<2>(T, 16, tid);
      else rank16<1>(T, 32, tid);
    }
    if (more) __syncthreads();
  }
  __syncthreads();
  return -1;
}

// The 64 rows of X solved against the factored tile (X L' = A), by 256 threads in four steps of 16 columns: a thread
// subtracts from 4 columns of one row the products of the columns already solved, then a thread per row substitutes through
// the 16 x 16 diagonal block, its 16 values in registers (dv: 1 / L[j, j]). X[c][r] in place; Z is scratch; the steps from
// column `cols` on (identity padding) are left out. (A thread per row with its 64 entries in registers, fully unrolled, was
// bound by fetching its 64 KB of instructions: 25 us a panel. The diagonal blocks applied through explicit inverses took
// longer than this with the inverses' own time, n = 1000 0.477 ms in all against 0.440, and cost backward stability, see k_solve.)
__device__ __forceinline__ void solve_rows(double (*X)[NB], double (*Z)[NB], const double (*T)[TS], const double* dv, int tid, int cols = NB) {
  const int r = tid & 63, q = 4 * (tid >> 6);
  for (int b = 0; b < cols; b += 16) {
    double acc[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[j] = X[b + q + j][r];
#pragma unroll 4
    for (int k = 0; k < b; k += 2) {
      const double x0 = X[k][r], x1 = X[k + 1][r];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const double2 l = *reinterpret_cast<const double2*>(&T[b + q + j][k]);
        acc[j] = fma(-x1, l.y, fma(-x0, l.x, acc[j]));
      }
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) Z[q + j][r] = acc[j];
    __syncthreads();
    if (tid < NB) {
      double z[16];
#pragma unroll
      for (int j = 0; j < 16; ++j) z[j] = Z[j][r];
#pragma unroll
      for (int j = 0; j < 16; ++j) {
        z[j] *= dv[b + j];
#pragma unroll
        for (int k = j + 1; k < 16; ++k) z[k] = fma(-z[j], T[b + k][b + j], z[k]);
      }
#pragma unroll
      for (int j = 0; j < 16; ++j) X[b + j][r] = z[j];
    }
    __syncthreads();
  }
}

// shared memory of the panel kernels: the diagonal tile, 1 / L[j, j], the CTA's 64 panel rows and their scratch
struct PanelSmem {
  double T[NB][TS];
  double dv[NB];
  double X[NB][NB];   // X[column][row]
  double Z[16][NB];
};

// The 64 x 64 inverse of the factored tile T: the identity solved against it (X L' = I, so X[i][j] = inverse[i][j]), for
// the solve.
__device__ __forceinline__ void tile_inverse(PanelSmem& s, const double (*T)[TS], double* __restrict__ inv, int64_t k0, int tid, int cols = NB) {
#pragma unroll
  for (int k = 0; k < NB * NB / 256; ++k) {
    const int e = tid + 256 * k;
    s.X[e >> 6][e & 63] = (e >> 6) == (e & 63) ? 1.0 : 0.0;
  }
  __syncthreads();
  solve_rows(s.X, s.Z, T, s.dv, tid, cols);
#pragma unroll
  for (int k = 0; k < NB * NB / 256; ++k) {
    const int e = tid + 256 * k, i = e & 63, j = e >> 6;
    inv[NB * k0 + i + NB * j] = s.X[i][j];
  }
}

// The diagonal tiles, one CTA after the other: the chain that every panel waits for. For panel k (k0 = 64 k) it solves the
// 64 rows below the diagonal tile (a copy of them, `rows`: k_trsm_panel solves the same rows in W meanwhile), subtracts
// their rank-64 product from the next diagonal tile and factors that; `first`: it factors tile 0. `cols`: columns of the
// tile to factor that are not padding. A non-positive or
// non-finite pivot records its column and nothing is written. Bound by the latency of its 64 columns, one after another
// (with the rows' solve and the update as launches of their own between the tiles a panel took 33 us): a factorisation takes
// 27 us a panel where the updates do not bound it (n = 1000: 0.535 -> 0.440 ms).
struct StepSmem {
  PanelSmem p;
  double next[NB][TS];
};
__global__ void __launch_bounds__(256, 1) k_step(int64_t ld, double* __restrict__ W, const double* __restrict__ rows, double* __restrict__ dinv,
                                                 double* __restrict__ inv, int64_t k0, int first, int cols, long long* __restrict__ status) {
  extern __shared__ __align__(16) unsigned char dense_smem[];
  StepSmem& s = *reinterpret_cast<StepSmem*>(dense_smem);
  __shared__ int failed;
  if (status[0] >= 0) return;   // uniform
  const int tid = threadIdx.x;
  const int64_t d0 = first ? k0 : k0 + NB;   // the tile to factor
  if (!first) {
#pragma unroll
    for (int k = 0; k < NB * NB / 256; ++k) {
      const int e = tid + 256 * k, r = e & 63, c = e >> 6;
      cp_async8(&s.p.X[c][r], rows + e);
      cp_async8(&s.p.T[r][c], W + (k0 + r) + ld * (k0 + c));   // entries above the diagonal are not used
    }
    if (tid < NB) cp_async8(s.p.dv + tid, dinv + k0 + tid);
  }
  run_cp_commit();
  load_tile(s.next, W, ld, d0, tid);
  if (tid == 0) failed = -1;
  run_cp_wait<0>();
  __syncthreads();
  if (!first) {
    solve_rows(s.p.X, s.p.Z, s.p.T, s.p.dv, tid);
    // next -= X X', 4 x 4 entries a thread: rows 2 tx + {0, 1, 32, 33}, columns 2 ty + {0, 1, 32, 33}
    const int tx = tid & 15, ty = tid >> 4;
    double acc[4][4];
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[p][q] = 0.0;
#pragma unroll 4
    for (int c = 0; c < NB; ++c) {
      const double2 a0 = *reinterpret_cast<const double2*>(&s.p.X[c][2 * tx]), a1 = *reinterpret_cast<const double2*>(&s.p.X[c][32 + 2 * tx]);
      const double2 b0 = *reinterpret_cast<const double2*>(&s.p.X[c][2 * ty]), b1 = *reinterpret_cast<const double2*>(&s.p.X[c][32 + 2 * ty]);
      const double ra[4] = {a0.x, a0.y, a1.x, a1.y}, rb[4] = {b0.x, b0.y, b1.x, b1.y};
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[p][q] = fma(ra[p], rb[q], acc[p][q]);
    }
#pragma unroll
    for (int p = 0; p < 4; ++p)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int i = 2 * tx + (p & 1) + 32 * (p >> 1), j = 2 * ty + (q & 1) + 32 * (q >> 1);
        if (j <= i) s.next[i][j] -= acc[p][q];
      }
    __syncthreads();
  }
  const int bad = factor_tile(s.next, s.p.dv, &failed, cols);
  if (bad >= 0) {
    if (tid == 0) status[0] = d0 + bad;
    return;
  }
#pragma unroll
  for (int k = 0; k < NB * NB / 256; ++k) {
    const int e = tid + 256 * k, rr = e & 63, cc = e >> 6;
    if (cc <= rr) W[(d0 + rr) + ld * (d0 + cc)] = s.next[rr][cc];
  }
  if (tid < NB) dinv[d0 + tid] = s.p.dv[tid];
  if (d0 + NB == ld) tile_inverse(s.p, s.next, inv, d0, tid, cols);   // no panel below it: its inverse is formed here
}

// Whether a pivot has failed, as thread 0 sees it (false in every other thread). k_step runs beside the kernels that ask
// and may record its failure at any time: threads that each read the word could disagree, and some would leave before a
// barrier that the others wait at. A kernel asks once and decides for the whole CTA by __syncthreads_or.
__device__ __forceinline__ bool stopped(const long long* status) {
  return threadIdx.x == 0 && *reinterpret_cast<const volatile long long*>(status) >= 0;
}

// The panel below a diagonal tile factored by k_step: a CTA per 64 rows, and one for the tile's inverse.
__global__ void __launch_bounds__(256) k_trsm_panel(int64_t ld, double* __restrict__ W, const double* __restrict__ dinv,
                                                    double* __restrict__ inv, int64_t k0, const long long* __restrict__ status) {
  extern __shared__ __align__(16) unsigned char dense_smem[];
  PanelSmem& s = *reinterpret_cast<PanelSmem*>(dense_smem);
  const int tid = threadIdx.x;
  const bool stop = stopped(status);
  const bool rows = blockIdx.x + 1 < gridDim.x;
  const int64_t row0 = k0 + NB + (int64_t)blockIdx.x * NB;
#pragma unroll
  for (int k = 0; k < NB * NB / 256; ++k) {
    const int e = tid + 256 * k, r = e & 63, c = e >> 6;
    if (rows) cp_async8(&s.X[c][r], W + (row0 + r) + ld * (k0 + c));
    cp_async8(&s.T[r][c], W + (k0 + r) + ld * (k0 + c));   // entries above the diagonal are not used
  }
  if (tid < NB) cp_async8(s.dv + tid, dinv + k0 + tid);
  run_cp_commit();
  run_cp_wait<0>();
  if (__syncthreads_or(stop)) return;
  if (!rows) {
    tile_inverse(s, s.T, inv, k0, tid);
    return;
  }
  solve_rows(s.X, s.Z, s.T, s.dv, tid);
#pragma unroll
  for (int k = 0; k < NB * NB / 256; ++k) {
    const int e = tid + 256 * k, r = e & 63, c = e >> 6;
    W[(row0 + r) + ld * (k0 + c)] = s.X[c][r];
  }
}

// W[i, j] -= sum over c in [k0, k0 + K) of L[i, c] L[j, c] for the lower triangle of the tile columns
// [j0 + 64 blockIdx.y, + 64) of W: CTAs of 256 threads over tiles of MT x 64 (MT = 128: 8 x 4 entries a thread, MT = 64:
// 4 x 4), those above the diagonal leave at once. The two row panels pass through a ring of three 16-column chunks in
// shared memory (16-byte cp.async, two chunks ahead of the products). With 4 x 4 entries a thread a warp needs 6
// shared-memory wavefronts per 32 cycles of FP64 multiply-adds, 24 of every 32 for the SM's four, with 8 x 4 half of that;
// rank 256 reads and writes the output a quarter as often as rank 64 (n = 6000: 5.9 ms of updates before, 4.3 now, 20 TFLOP/s in the 128-row form).
// The panels wait for the rank-64 updates on their stream: those (AHEAD) have all four chunks and the output tile in
// flight at once, so that such a launch costs one round trip to memory.
template <int MT, bool AHEAD>
__host__ __device__ constexpr int syrk_smem() { return (AHEAD ? 4 : 3) * 16 * (MT + NB) * (int)sizeof(double); }
template <int MT, bool AHEAD>
__global__ void __launch_bounds__(256, AHEAD ? 3 : MT == 128 ? 2 : 4) k_syrk(int64_t ld, double* __restrict__ W, int64_t k0, int K, int64_t j0, double* __restrict__ rows,
                                                                 const long long* __restrict__ status) {
  constexpr int KC = 16, RM = MT / 16, ST = AHEAD ? 4 : 3;   // RM: rows a thread holds
  extern __shared__ __align__(16) unsigned char dense_smem[];
  double* ring = reinterpret_cast<double*>(dense_smem);
  const int64_t bj = j0 + NB * (int64_t)blockIdx.y, bi = j0 + MT * (int64_t)blockIdx.x;
  if (bi + MT <= bj) return;   // above the diagonal
  if (AHEAD && blockIdx.x == 0 && blockIdx.y == 0) return;   // the next diagonal tile is k_step's
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const bool stop = stopped(status);
  const int nch = K / KC;
  auto A = [&](int ch) { return reinterpret_cast<double (*)[MT]>(ring + (ch % ST) * KC * (MT + NB)); };
  auto B = [&](int ch) { return reinterpret_cast<double (*)[NB]>(ring + (ch % ST) * KC * (MT + NB) + KC * MT); };
  auto issue = [&](int ch) {
    if (ch < nch) {
      const double* src = W + ld * (k0 + KC * ch);
      auto a = A(ch);
      auto b = B(ch);
#pragma unroll
      for (int k = 0; k < KC * MT / 512; ++k) {
        const int e = tid + 256 * k, c = e / (MT / 2), r = 2 * (e % (MT / 2));
        const bool in = MT == NB || bi + r < ld;   // the last 128-row tile may hang over W's end
        run_cp16(&a[c][r], in ? src + ld * c + bi + r : src, in ? 16 : 0);
      }
#pragma unroll
      for (int k = 0; k < KC * NB / 512; ++k) {
        const int e = tid + 256 * k, c = e / (NB / 2), r = 2 * (e % (NB / 2));
        run_cp16(&b[c][r], src + ld * c + bj + r, 16);
      }
    }
    run_cp_commit();   // an empty group keeps the count of groups in flight uniform
  };
  // rows bi + 2 tx + 32 (p / 2) + (p & 1), columns bj + 2 ty + 32 (q / 2) + (q & 1) are this thread's
  auto out_row = [&](int p) { return bi + 2 * tx + 32 * (p >> 1) + (p & 1); };
  auto out_col = [&](int q) { return bj + 2 * ty + 32 * (q >> 1) + (q & 1); };
  auto is_out = [&](int p, int q) { return out_row(p) < ld && out_col(q) <= out_row(p); };
#pragma unroll
  for (int ch = 0; ch < ST - 1; ++ch) issue(ch);
  double acc[RM][4];
#pragma unroll
  for (int p = 0; p < RM; ++p)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[p][q] = 0.0;
  double out[AHEAD ? RM : 1][4];
  if constexpr (AHEAD) {
    issue(ST - 1);
#pragma unroll
    for (int p = 0; p < RM; ++p)
#pragma unroll
      for (int q = 0; q < 4; ++q) out[p][q] = is_out(p, q) ? W[out_row(p) + ld * out_col(q)] : 0.0;
  }
  if (__syncthreads_or(stop)) {   // the panels are useless from the failing column on
    run_cp_wait<0>();
    return;
  }
  for (int ch = 0; ch < nch; ++ch) {
    run_cp_wait<ST - 2 + (AHEAD ? 1 : 0)>();
    __syncthreads();   // chunk ch is in for every thread, and chunk ch - 1 has been used
    if (AHEAD) run_cp_commit();   // nch is ST: nothing left to issue
    else issue(ch + ST - 1);      // into the stage of chunk ch - 1
    auto a = A(ch);
    auto b = B(ch);
#pragma unroll 4
    for (int c = 0; c < KC; ++c) {
      double ra[RM], rb[4];
#pragma unroll
      for (int p = 0; p < RM; p += 2) {
        const double2 v = *reinterpret_cast<const double2*>(&a[c][2 * tx + 16 * p]);
        ra[p] = v.x;
        ra[p + 1] = v.y;
      }
#pragma unroll
      for (int q = 0; q < 4; q += 2) {
        const double2 v = *reinterpret_cast<const double2*>(&b[c][2 * ty + 16 * q]);
        rb[q] = v.x;
        rb[q + 1] = v.y;
      }
#pragma unroll
      for (int p = 0; p < RM; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[p][q] = fma(ra[p], rb[q], acc[p][q]);
    }
  }
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    double old[RM];
#pragma unroll
    for (int p = 0; p < RM; ++p) old[p] = AHEAD ? out[AHEAD ? p : 0][q] : is_out(p, q) ? W[out_row(p) + ld * out_col(q)] : 0.0;
#pragma unroll
    for (int p = 0; p < RM; ++p)
      if (is_out(p, q)) {
        W[out_row(p) + ld * out_col(q)] = old[p] - acc[p][q];
        // the rows below the next diagonal tile, finished here, also for k_step
        if (AHEAD && blockIdx.x == 1 && blockIdx.y == 0) rows[(out_row(p) - bi) + NB * (out_col(q) - bj)] = old[p] - acc[p][q];
      }
  }
}

// L L' x = g in one cooperative launch, CTA b owning the 64 rows of tile b. Forward: it takes y_k of every earlier tile in
// order (polling it: each value is 8 bytes, all bits set until it is written), subtracts L[b, k] y_k from its rows, then
// multiplies them by the inverse of its diagonal tile and posts y_b. Backward the same from the last tile up with L'. A
// tile's 64 x 64 block of L is loaded before its poll. The diagonal tile's inverse alone would cost backward stability:
// ||S x - g|| / (||S|| ||x||) reached 6e-12, 8e-10 and 1e-8 on Gaussian kernel matrices of condition 1e8, 1e10 and 1e12, where
// substitution leaves 5e-17. One step of refinement against the tile itself brings it back to 5e-17, for two more products of
// 64 x 64 from shared memory: n = 1000 51 -> 60 us, 10000 0.55 -> 0.58 ms. A poll that gives up after `limit` tries
// raises the fault word, which the next synchronising call reports, and passes NaNs on, so that nothing waits for ever.
// n = 10000: 2.3 ms as two launches per tile with a substitution by one warp in each, 0.58 ms now.
constexpr unsigned long long kUnwritten = ~0ull;
__device__ __forceinline__ double poll_value(const double* p, int64_t limit, long long* fault) {
  unsigned long long v = kUnwritten;
  for (int64_t i = 0; i < limit; ++i) {
    asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
    if (v != kUnwritten) break;
  }
  if (v != kUnwritten) return __longlong_as_double((long long)v);
  asm volatile("st.relaxed.gpu.global.u64 [%0], 1;" ::"l"(fault) : "memory");
  return __longlong_as_double(0x7ff8000000000000ll);
}
__device__ __forceinline__ void post_value(double* p, double v) {
  unsigned long long b = (unsigned long long)__double_as_longlong(v);
  if (b == kUnwritten) b = 0x7ff8000000000000ull;   // a NaN of another payload
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(b) : "memory");
}

struct SolveSmem {   // the tile of L and its inverse, [column][row], strides that serve both directions without conflicts
  double L[NB][NB + 1];
  double inv[NB][NB + 1];
};
__global__ void __launch_bounds__(256, 2) k_solve(int64_t n, int64_t ld, const double* __restrict__ W, const double* __restrict__ inv,
                                               const double* g, double* x, double* y, int64_t limit, long long* fault) {
  __shared__ double rt[NB];   // the tile's current right-hand side
  __shared__ double xk[NB];
  __shared__ double part[4][NB];
  extern __shared__ __align__(16) unsigned char dense_smem[];
  SolveSmem& sm = *reinterpret_cast<SolveSmem*>(dense_smem);
  const int tid = threadIdx.x, r = tid & 63, q = tid >> 6, lane = tid & 31, warp = tid >> 5;
  const int nt = (int)(ld / NB), b = blockIdx.x;
  const int64_t row0 = NB * (int64_t)b;
  // the diagonal tile and its inverse come in while the earlier tiles are waited for
#pragma unroll
  for (int k = 0; k < NB * NB / 256; ++k) {
    const int c = q + 4 * k;
    cp_async8(&sm.L[c][r], W + (row0 + r) + ld * (row0 + c));   // entries above the diagonal are not used
    cp_async8(&sm.inv[c][r], inv + NB * row0 + r + NB * c);
  }
  run_cp_commit();
  double* yf = y;
  double* yb = y + ld;
  if (tid < NB) rt[tid] = row0 + tid < n ? g[row0 + tid] : 0.0;
  double w[16];   // a 64 x 64 block: row r, columns 16 q ..
  auto load = [&](const double* M, int64_t stride) {
#pragma unroll
    for (int c = 0; c < 16; ++c) w[c] = M[r + stride * (16 * q + c)];
  };
  auto mul = [&](const double* xs) {   // (M xs)[r], in every thread
    double s = 0.0;
#pragma unroll
    for (int c = 0; c < 16; ++c) s = fma(w[c], xs[16 * q + c], s);
    part[q][r] = s;
    __syncthreads();
    return (part[0][r] + part[1][r]) + (part[2][r] + part[3][r]);
  };
  for (int k = 0; k < b; ++k) {
    load(W + row0 + ld * NB * (int64_t)k, ld);
    if (tid < NB) xk[tid] = poll_value(yf + NB * (int64_t)k + tid, limit, fault);
    __syncthreads();
    const double v = mul(xk);
    if (q == 0) rt[r] -= v;
    // the next xk and part are written after the barrier that every thread passes once it has read these: mul's own
    // barrier orders xk, the one below part and rt
    __syncthreads();
  }
  run_cp_wait<0>();
  __syncthreads();   // the tile and its inverse, rt (b = 0: as it was read from g)
  // the tile's system (T: transposed) for rt, in every thread: through the inverse, with one step of refinement
  auto product = [&](const double (*M)[NB + 1], auto t, bool lower) {
    double s = 0.0;
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      const int k = 16 * q + c, row = decltype(t)::value ? k : r, col = decltype(t)::value ? r : k;
      s = fma(lower && row < col ? 0.0 : M[col][row], xk[k], s);
    }
    part[q][r] = s;
    __syncthreads();
    return (part[0][r] + part[1][r]) + (part[2][r] + part[3][r]);
  };
  auto tile_solve = [&](auto t) {
    if (q == 0) xk[r] = rt[r];
    __syncthreads();
    const double x0 = product(sm.inv, t, false);
    if (q == 0) xk[r] = x0;   // every thread has passed the barrier in product after reading xk
    __syncthreads();          // and part is read
    const double res = rt[r] - product(sm.L, t, true);
    if (q == 0) xk[r] = res;
    __syncthreads();
    return x0 + product(sm.inv, t, false);
  };
  const double yv = tile_solve(std::false_type());
  if (q == 0) post_value(yf + row0 + r, yv);
  __syncthreads();   // every thread has read rt and part
  if (q == 0) rt[r] = yv;
  // backward: a block's column sums, a warp per 8 columns, lanes over its rows
  double w0[8], w1[8];
  auto load_t = [&](const double* M, int64_t stride) {
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      w0[m] = M[lane + stride * (8 * warp + m)];
      w1[m] = M[lane + 32 + stride * (8 * warp + m)];
    }
  };
  auto mul_t = [&](const double* xs) {   // (M' xs)[8 warp + lane] in lanes below 8
    const double x0 = xs[lane], x1 = xs[lane + 32];
    double v = 0.0;
#pragma unroll
    for (int m = 0; m < 8; ++m) {
      double s = w0[m] * x0 + w1[m] * x1;
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
      if (lane == m) v = s;
    }
    return v;
  };
  for (int k = nt - 1; k > b; --k) {
    load_t(W + NB * (int64_t)k + ld * row0, ld);
    __syncthreads();   // every thread has read the previous xk (first: rt is written)
    if (tid < NB) xk[tid] = poll_value(yb + NB * (int64_t)k + tid, limit, fault);
    __syncthreads();
    const double v = mul_t(xk);
    if (lane < 8) rt[8 * warp + lane] -= v;
  }
  __syncthreads();   // rt, and xk is read
  const double xv = tile_solve(std::true_type());
  if (q == 0) {
    post_value(yb + row0 + r, xv);
    if (row0 + r < n) x[row0 + r] = xv;
  }
}

// Launches kernel on stream st with the given priority (a launch attribute, so that a captured graph keeps it).
template <class... Args>
static void launch_prio(void (*kernel)(Args...), dim3 grid, unsigned block, size_t smem, cudaStream_t st, int prio, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributePriority;
  attr[0].val.priority = prio;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  BLS_CUDA(cudaLaunchKernelEx(&cfg, kernel, args...));
}

// The factorisation after the load of S into W: the diagonal tiles on the panel stream p, the panels below them and the
// updates that the next panels wait for on u, the rest of each group's update on s, joined on s.
static void launch_factor_body(DenseSolver* D, cudaStream_t s, cudaStream_t p) {
  const int64_t ld = D->ld, nt = ld / NB;
  double* W = D->W;
  double* dinv = D->dinv;
  double* inv = D->inv;
  long long* st = D->status;
  const long long* cst = st;
  const int prio = D->panel_priority;
  cudaStream_t u = D->update_stream;
  double* rows = D->rows;   // two buffers, by the parity of the panel
  double* none = nullptr;
  auto then = [](cudaStream_t from, cudaEvent_t ev, cudaStream_t to) {
    BLS_CUDA(cudaEventRecord(ev, from));
    BLS_CUDA(cudaStreamWaitEvent(to, ev, 0));
  };
  then(s, D->ev_join, p);
  BLS_CUDA(cudaStreamWaitEvent(u, D->ev_join, 0));
  auto step = [&](int64_t k0, int first, const double* below_rows) {
    const int64_t d0 = first ? k0 : k0 + NB;
    launch_prio(k_step, dim3(1), 256, sizeof(StepSmem), p, prio, ld, W, below_rows, dinv, inv, k0, first, (int)std::min<int64_t>(NB, D->n - d0), st);
  };
  step(0, 1, rows);
  bool next_pending = false;
  for (int64_t g0 = 0; g0 < nt; g0 += GROUP) {
    const int64_t g1 = std::min(nt, g0 + GROUP);   // the group's panels
    for (int64_t k = g0; k < g1; ++k) {
      const int64_t below = nt - k - 1;
      if (below == 0) break;   // the last tile's inverse is k_step's
      // u: the panel's rows, once its tile is factored; p: the next tile, once the previous panel's update (and, for a
      // group's first panel, the previous group's) is done
      then(p, D->ev_tile, u);
      if (k > 0) BLS_CUDA(cudaStreamWaitEvent(p, D->ev_update, 0));
      if (k == g0 && next_pending) {
        BLS_CUDA(cudaStreamWaitEvent(p, D->ev_next, 0));
        BLS_CUDA(cudaStreamWaitEvent(u, D->ev_next, 0));
      }
      launch_prio(k_trsm_panel, dim3((unsigned)(below + 1)), 256, sizeof(PanelSmem), u, prio, ld, W, (const double*)dinv, inv, k * NB, cst);
      step(k * NB, 0, rows + (k & 1) * NB * NB);
      if (below == 1) break;   // nothing but the next diagonal tile is left
      // the group's remaining columns and the next group's first one, which the next panels need
      const int64_t cols = std::min(nt, g1 + 1) - k - 1;
      launch_prio(k_syrk<64, true>, dim3((unsigned)below, (unsigned)cols), 256, (size_t)syrk_smem<64, true>(), u, prio, ld, W, k * NB, NB,
                  (k + 1) * NB, rows + ((k + 1) & 1) * NB * NB, cst);
      BLS_CUDA(cudaEventRecord(D->ev_update, u));
    }
    if (g1 + 1 >= nt) continue;
    // everything right of that, beside the next panels: the next group's other columns first (they wait for them)
    const int K = (int)((g1 - g0) * NB);
    const int64_t j0 = g1 + 1, g2 = std::min(nt, g1 + GROUP + 1);
    then(u, D->ev_panel, s);
    k_syrk<64, false><<<dim3((unsigned)(nt - j0), (unsigned)(g2 - j0)), 256, syrk_smem<64, false>(), s>>>(ld, W, g0 * NB, K, j0 * NB, none, cst);
    BLS_CUDA(cudaEventRecord(D->ev_next, s));
    next_pending = true;
    if (g2 < nt) {
      const int64_t rest = nt - g2;
      k_syrk<128, false><<<dim3((unsigned)((rest + 1) / 2), (unsigned)rest), 256, syrk_smem<128, false>(), s>>>(ld, W, g0 * NB, K, g2 * NB, none, cst);
    }
  }
  then(p, D->ev_tile, s);
  then(u, D->ev_update, s);
}

// An earlier solve's fault word as read back: cleared and raised as an error.
static void report_fault(DenseSolver* D, long long fault) {
  if (fault == 0) return;
  BLS_CUDA(cudaMemsetAsync(D->status + 1, 0, sizeof(long long), D->ctx->stream));
  throw Error(BLS_ECUDA, "a wait of an earlier solve did not complete within its limit: that solve's x is not valid");
}

template <class T>
static int factor(DenseSolver* D, const T* S, double lambda, const double* s_r, int64_t* failed_column) {
  if (!S) throw Error(BLS_EINVAL, "S is NULL");
  cudaStream_t s = D->ctx->stream;
  const int64_t n = D->n;
  double* W = D->W;
  long long* st = D->status;
  if (!D->prepared) {
    BLS_CUDA(cudaFuncSetAttribute(k_step, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(StepSmem)));
    D->prepared = true;
  }
  if (D->ld > NB && !D->panel_stream) {
    int lo = 0, hi = 0;
    BLS_CUDA(cudaDeviceGetStreamPriorityRange(&lo, &hi));
    D->panel_priority = hi;
    BLS_CUDA(cudaStreamCreateWithPriority(&D->panel_stream, cudaStreamNonBlocking, hi));
    BLS_CUDA(cudaEventCreateWithFlags(&D->ev_join, cudaEventDisableTiming));
    BLS_CUDA(cudaEventCreateWithFlags(&D->ev_panel, cudaEventDisableTiming));
    for (cudaEvent_t* e : {&D->ev_next, &D->ev_tile, &D->ev_update}) BLS_CUDA(cudaEventCreateWithFlags(e, cudaEventDisableTiming));
    BLS_CUDA(cudaStreamCreateWithPriority(&D->update_stream, cudaStreamNonBlocking, hi));
    BLS_CUDA(cudaFuncSetAttribute(k_syrk<64, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, syrk_smem<64, true>()));
    BLS_CUDA(cudaFuncSetAttribute(k_syrk<64, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, syrk_smem<64, false>()));
    BLS_CUDA(cudaFuncSetAttribute(k_syrk<128, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, syrk_smem<128, false>()));
    BLS_CUDA(cudaFuncSetAttribute(k_trsm_panel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(PanelSmem)));
  }
  const unsigned tiles = (unsigned)(D->ld / 32);
  k_dense_load<T><<<dim3(tiles, tiles), 256, 0, s>>>(n, D->ld, S, W, lambda, s_r, D->rows, st);
  if (D->ld == NB) {   // one tile: one launch
    k_step<<<1, 256, sizeof(StepSmem), s>>>(D->ld, W, D->rows, D->dinv, D->inv, 0, 1, (int)n, st);
  } else if (!D->factor_graph) {
    if (!D->cap_stream) BLS_CUDA(cudaStreamCreateWithFlags(&D->cap_stream, cudaStreamNonBlocking));
    BLS_CUDA(cudaStreamBeginCapture(D->cap_stream, cudaStreamCaptureModeThreadLocal));
    cudaGraph_t gr = nullptr;
    try {
      launch_factor_body(D, D->cap_stream, D->panel_stream);
    } catch (...) {
      cudaStreamEndCapture(D->cap_stream, &gr);
      if (gr) cudaGraphDestroy(gr);
      throw;
    }
    BLS_CUDA(cudaStreamEndCapture(D->cap_stream, &gr));
    const cudaError_t e = cudaGraphInstantiate(&D->factor_graph, gr, 0);
    cudaGraphDestroy(gr);
    if (e != cudaSuccess) {
      D->factor_graph = nullptr;
      throw Error(BLS_ECUDA, std::string("instantiating the factorisation: ") + cudaGetErrorString(e));
    }
  }
  if (D->ld > NB) BLS_CUDA(cudaGraphLaunch(D->factor_graph, s));
  BLS_CUDA(cudaGetLastError());
  long long h[2] = {-1, 0};
  BLS_CUDA(cudaMemcpyAsync(h, st, sizeof(h), cudaMemcpyDeviceToHost, s));
  BLS_CUDA(cudaStreamSynchronize(s));
  D->factored = h[0] < 0;
  if (failed_column) *failed_column = h[0] < 0 ? 0 : h[0] + 1;
  report_fault(D, h[1]);
  return h[0] < 0 ? BLS_OK : BLS_NOT_PD;
}

}  // namespace bls

using namespace bls;

struct bls_dense_solver : DenseSolver {};

#define DENSE_GUARD(...)                      \
  try {                                       \
    __VA_ARGS__                               \
  } catch (const bls::Error& e) {             \
    bls::set_error(e.what());                 \
    return e.code;                            \
  } catch (const std::bad_alloc&) {           \
    bls::set_error("out of host memory");     \
    return BLS_ENOMEM;                        \
  }

extern "C" {

int bls_dense_solver_create(bls_ctx* ctx, int64_t n, bls_dense_solver** out) {
  DENSE_GUARD({
    if (!ctx || !out) throw Error(BLS_EINVAL, "null argument");
    if (n < 1 || n > 16384) throw Error(BLS_EUNSUPPORTED, "dense reduced systems of 1 to 16384 variables are supported");
    std::unique_ptr<bls_dense_solver> D(new bls_dense_solver());
    D->ctx = ctx;
    D->n = n;
    D->ld = (n + NB - 1) / NB * NB;
    const size_t w = (size_t)(D->ld * D->ld), r = 2 * NB * NB, dv = (size_t)D->ld, v = NB * (size_t)D->ld, y = 2 * (size_t)D->ld;
    D->mem.alloc(sizeof(double) * (w + r + dv + v + y) + 2 * sizeof(long long));   // every part a multiple of 64 doubles
    D->W = D->mem.as<double>();
    D->rows = D->W + w;
    D->dinv = D->rows + r;
    D->inv = D->dinv + dv;
    D->y = D->inv + v;
    D->status = reinterpret_cast<long long*>(D->y + y);
    BLS_CUDA(cudaMemsetAsync(D->status, 0, 2 * sizeof(long long), ctx->stream));
    *out = D.release();
    return BLS_OK;
  })
}

int bls_dense_solver_destroy(bls_dense_solver* D) {
  delete D;
  return BLS_OK;
}

int bls_dense_cholesky(bls_dense_solver* D, int dtype, const void* S, int64_t* failed_column) {
  DENSE_GUARD({
    if (!D) throw Error(BLS_EINVAL, "solver is NULL");
    if (dtype == BLS_F64) return factor<double>(D, (const double*)S, 0.0, nullptr, failed_column);
    if (dtype == BLS_F32) return factor<float>(D, (const float*)S, 0.0, nullptr, failed_column);
    throw Error(BLS_EINVAL, "unknown dtype");
  })
}

int bls_dense_cholesky_shifted(bls_dense_solver* D, int dtype, const void* S, double lambda, const double* s_r, int64_t* failed_column) {
  DENSE_GUARD({
    if (!D || !s_r) throw Error(BLS_EINVAL, "null argument");
    if (!(std::isfinite(lambda) && lambda >= 0))
      throw Error(BLS_EINVAL, "lambda must be finite and non-negative, got " + std::to_string(lambda));
    if (dtype == BLS_F64) return factor<double>(D, (const double*)S, lambda, s_r, failed_column);
    if (dtype == BLS_F32) return factor<float>(D, (const float*)S, lambda, s_r, failed_column);
    throw Error(BLS_EINVAL, "unknown dtype");
  })
}

int bls_dense_cholesky_solve(bls_dense_solver* D, const double* g, double* x) {
  DENSE_GUARD({
    if (!D || !g || !x) throw Error(BLS_EINVAL, "null argument");
    if (!D->factored) throw Error(BLS_EINVAL, "the solver holds no factorisation (bls_dense_cholesky first, and it must succeed)");
    const int64_t n = D->n;
    const double* W = D->W;
    cudaStream_t s = D->ctx->stream;
    // the tiles' CTAs must be resident at once (256 at the largest n)
    const int64_t nt = D->ld / NB;
    if (D->solve_grid == 0) {
      int per_sm = 0, nsm = 0, dev = 0;
      BLS_CUDA(cudaGetDevice(&dev));
      BLS_CUDA(cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev));
      BLS_CUDA(cudaFuncSetAttribute(k_solve, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(SolveSmem)));
      BLS_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_solve, 256, sizeof(SolveSmem)));
      if (nt > (int64_t)nsm * per_sm) throw Error(BLS_EUNSUPPORTED, "the device is too small for this system's solve");
      D->solve_grid = (int)nt;
    }
    double* y = D->y;
    BLS_CUDA(cudaMemsetAsync(y, 0xff, sizeof(double) * 2 * (size_t)D->ld, s));
    int64_t n_arg = n, ld_arg = D->ld;
    const double* inv = D->inv;
    long long* fault = D->status + 1;
    void* args[] = {&n_arg, &ld_arg, &W, &inv, &g, &x, &y, &D->wait_limit, &fault};
    BLS_CUDA(cudaLaunchCooperativeKernel((const void*)k_solve, dim3((unsigned)D->solve_grid), dim3(256), args, sizeof(SolveSmem), s));
    BLS_CUDA(cudaGetLastError());
    return BLS_OK;
  })
}

int bls_dense_solver_check(bls_dense_solver* D) {
  DENSE_GUARD({
    if (!D) throw Error(BLS_EINVAL, "solver is NULL");
    long long fault = 0;
    BLS_CUDA(cudaMemcpyAsync(&fault, D->status + 1, sizeof(fault), cudaMemcpyDeviceToHost, D->ctx->stream));
    BLS_CUDA(cudaStreamSynchronize(D->ctx->stream));
    report_fault(D, fault);
    return BLS_OK;
  })
}

int bls_dense_solver_set_wait_limit(bls_dense_solver* D, int64_t polls) {
  if (!D || polls < 1 || polls > kWaitLimit) return BLS_EINVAL;
  D->wait_limit = polls;
  return BLS_OK;
}

}  // extern "C"
