// ngd.cu - the damped Gauss-Newton step of app/optimizer_module.f90:221-469
// (primal route, ABS damping) on the device:
//   G = J^T J / nb + mu I,  u = G^{-1} (b / nb),
// with the metric formed from the residual-Jacobian rows J[nrow][nw] and
// solved by an FP64 Cholesky factorization (the reference eliminates with
// partial pivoting, gauss_solve :472-522; G is symmetric positive definite
// once damped, so the factorization is the natural device form).
//
// The metric build is a GEMM: in the split path J is carried as three bf16
// terms and the six cross products are accumulated in FP32 over runs of at most
// 512 rows on the tensor cores, the runs summed in FP64; in the plain path it
// runs on the FP64 tensor cores.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>
#include <string>

#include "engine.hpp"
#include "gemm_tc.hpp"
#include "scratch.hpp"

namespace dnnf90 {

#define CKN(call)                                                      \
  do {                                                                 \
    cudaError_t e_ = (call);                                           \
    if (e_ != cudaSuccess) {                                           \
      set_error(std::string(#call) + ": " + cudaGetErrorString(e_));   \
      return e_ == cudaErrorMemoryAllocation ? RC_NOMEM : RC_DEVICE;   \
    }                                                                  \
  } while (0)

constexpr int NB = 64;

// ------------------------------------------------------------ FP64 products
// 64 x 64 output tiles on the FP64 tensor cores (mma.sync m8n8k4 f64): four
// warps of 32 x 32 (4 x 4 fragments).  Lane coordinates r8 = lane / 4, c4 =
// lane % 4; the fragments take rows, columns and k so that every shared load
// is 16 bytes (the layouts of gemm_f64.cu): from [k][x] tiles (the metric)
// fragment i holds rows 16 (i >> 1) + 2 r8 + (i & 1), from [x][k] tiles (the
// trailing update) rows 8 i + r8 with k = 16 kb + 4 c4 + ks.
__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}
// asynchronous copies, zero-filled when ok is false
__device__ __forceinline__ void cp8(double *dst, const double *src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(ok ? 8 : 0)
               : "memory");
}
__device__ __forceinline__ void cp16(double *dst, const double *src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src), "r"(ok ? 16 : 0)
               : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// (ti, tj), tj <= ti, of the e-th tile of a lower triangle
__device__ __forceinline__ void low_tile(int e, int &ti, int &tj) {
  int i = (int)((sqrt(8.0 * e + 1.0) - 1.0) * 0.5);
  while (i > 0 && (long long)i * (i + 1) / 2 > e) --i;
  while ((long long)(i + 1) * (i + 2) / 2 <= e) ++i;
  ti = i;
  tj = e - (int)((long long)i * (i + 1) / 2);
}

constexpr int GK = 16, GST = 68, GNS = 3;  // k-block, row stride, stages of the metric's ring
constexpr size_t GRAM_SMEM = (size_t)GNS * 2 * GK * GST * 8;

// G[i][j] += sum_r J[r][i] J[r][j] for the lower tiles, rows [z rchunk, ...)
// of slab z: a three-stage cp.async ring of 16-row blocks.  V16: 16-byte
// pieces (an even nw and 16-byte aligned rows), else 8-byte ones.  ATOMIC:
// several slabs add into G (zeroed before), else one slab writes it.
// Bound: the FP64 tensor pipe (4096 rows of 4481: 2.8 ms, 29 TFLOP/s useful;
// the CUDA-core tiles before took 4.8 ms).
template <bool V16, bool ATOMIC>
__global__ void __launch_bounds__(128, 4) k_syrk_f64(const double *J, int nrow, int nw, double *G,
                                                     int rchunk) {
  extern __shared__ __align__(16) double gsm[];
  int ti, tj;
  low_tile(blockIdx.x, ti, tj);
  const int i0 = ti * 64, j0 = tj * 64;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, r8 = lane >> 2, c4 = lane & 3;
  const int wm = (warp & 1) * 32, wn = (warp >> 1) * 32;
  const int r0 = blockIdx.y * rchunk, r1 = min(nrow, r0 + rchunk);
  const int nkb = (r1 - r0 + GK - 1) / GK;
  auto load = [&](int kb) {
    double *sa = gsm + (kb % GNS) * 2 * GK * GST, *sb = sa + GK * GST;
    const int k0 = r0 + kb * GK;
    if (V16) {
#pragma unroll
      for (int p = 0; p < GK * 32 / 128; ++p) {
        const int e = t + p * 128, kk = e >> 5, c = (e & 31) * 2;
        const bool rk = k0 + kk < r1, oa = rk && i0 + c < nw, ob = rk && j0 + c < nw;
        const double *row = J + (size_t)(rk ? k0 + kk : r0) * nw;
        cp16(sa + kk * GST + c, row + (oa ? i0 + c : 0), oa);
        cp16(sb + kk * GST + c, row + (ob ? j0 + c : 0), ob);
      }
    } else {
#pragma unroll
      for (int p = 0; p < GK * 64 / 128; ++p) {
        const int e = t + p * 128, kk = e >> 6, c = e & 63;
        const bool rk = k0 + kk < r1, oa = rk && i0 + c < nw, ob = rk && j0 + c < nw;
        const double *row = J + (size_t)(rk ? k0 + kk : r0) * nw;
        cp8(sa + kk * GST + c, row + (oa ? i0 + c : 0), oa);
        cp8(sb + kk * GST + c, row + (ob ? j0 + c : 0), ob);
      }
    }
  };
  double acc[4][4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;
#pragma unroll
  for (int p = 0; p < GNS - 1; ++p) {
    if (p < nkb) load(p);
    cp_commit();
  }
  for (int kb = 0; kb < nkb; ++kb) {
    cp_wait<GNS - 2>();
    __syncthreads();  // this k-block is in; every warp is done with the previous one
    if (kb + GNS - 1 < nkb) load(kb + GNS - 1);
    cp_commit();
    const double *sa = gsm + (kb % GNS) * 2 * GK * GST, *sb = sa + GK * GST;
#pragma unroll
    for (int ks = 0; ks < GK / 4; ++ks) {
      const double *pa = sa + (4 * ks + c4) * GST + wm + 2 * r8;
      const double *pb = sb + (4 * ks + c4) * GST + wn + 2 * r8;
      double a[4], b[4];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const double2 va = *(const double2 *)(pa + 16 * h), vb = *(const double2 *)(pb + 16 * h);
        a[2 * h] = va.x;
        a[2 * h + 1] = va.y;
        b[2 * h] = vb.x;
        b[2 * h + 1] = vb.y;
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) dmma(acc[i][j], a[i], b[j]);
    }
  }
  cp_wait<0>();
  // product column 2 c4 + e of fragment j is column 16 (j >> 1) + 2 (2 c4 + e) + (j & 1)
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = i0 + wm + 16 * (i >> 1) + 2 * r8 + (i & 1);
    if (r >= nw) continue;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = j0 + wn + 16 * (j >> 1) + 2 * (2 * c4 + e) + (j & 1);
        if (c > r) continue;
        double *g = G + (size_t)r * nw + c;
        if (ATOMIC) atomicAdd(g, acc[i][j][e]);
        else *g = acc[i][j][e];
      }
  }
}

// G (lower triangle, zeroed before) += J^T J in FP64
static int syrk_f64(const double *J, int nrow, int nw, double *G, cudaStream_t st) {
  const int tiles = (nw + 63) / 64, low = tiles * (tiles + 1) / 2;
  // the rows are split while there are fewer tiles than resident blocks
  int split = std::max(1, std::min(grid_sms() * 4 / low, (nrow + 63) / 64));
  int rchunk = (nrow + split - 1) / split;
  rchunk = std::max(GK, (rchunk + GK - 1) / GK * GK);
  split = std::max(1, (nrow + rchunk - 1) / rchunk);
  const bool v16 = nw % 2 == 0 && ((uintptr_t)J & 15) == 0;
  const dim3 grid(low, split);
#define SYRK(V, A)                                                                              \
  do {                                                                                          \
    CKN(cudaFuncSetAttribute(k_syrk_f64<V, A>, cudaFuncAttributeMaxDynamicSharedMemorySize,     \
                             (int)GRAM_SMEM));                                                  \
    LAUNCH("k_syrk_f64", st, (k_syrk_f64<V, A><<<grid, 128, GRAM_SMEM, st>>>(J, nrow, nw, G, rchunk))); \
  } while (0)
  if (v16 && split > 1) SYRK(true, true);
  else if (v16) SYRK(true, false);
  else if (split > 1) SYRK(false, true);
  else SYRK(false, false);
#undef SYRK
  CKN(cudaGetLastError());
  return RC_OK;
}

// G = G / nb + mu I on the lower triangle, one block per row; rhs = b / nb
// (null: none)
__global__ void k_scale_damp(double *G, int n, double inv_nb, double mu, const double *b,
                             double *rhs) {
  const int i = blockIdx.x;
  double *row = G + (size_t)i * n;
  for (int j = threadIdx.x; j <= i; j += blockDim.x) row[j] = row[j] * inv_nb + (i == j ? mu : 0.0);
  if (rhs && threadIdx.x == 0) rhs[i] = b[i] * inv_nb;
}

// ------------------------------------------------------------ Cholesky
// Right-looking with 64-wide panels, G = L L^T in place (lower triangle),
// the right-hand side carried along as one more row of the matrix, so that
// the forward substitution L y = b costs no pass of its own.  Per panel two
// launches: k_trsm_panel solves the rows below the diagonal block, and
// k_syrk_trail updates the trailing tiles, whose first block factors the
// next diagonal block as soon as its own tile is updated, behind the other
// tiles' products.  The backward substitution takes one launch per block of
// 64 unknowns (k_back_step).
// Measured at n = 4481 (30 GFLOP): 4.2 ms, of it k_syrk_trail 33 us a panel,
// k_trsm_panel 6, a backward step 8; unblocked panel kernels of one thread per
// row and a one-block solve a row at a time took 38 ms.

// Both panel steps work on 64 x 64 blocks in shared memory eight columns at
// a time: the short serial part (the 8 x 8 factor, a row's eight unknowns)
// by one thread per row, the rank-8 update of the remaining columns as 8 x 8
// tiles on the FP64 tensor cores by every warp.  A lone warp issues an
// instruction every five or so cycles, so long per-thread loops (one barrier
// per column, or a whole row per thread) leave the chain four to five times
// longer.

constexpr int PS = 66;   // row stride of the trailing update's strips (16-byte loads)
constexpr int QS = 68;   // row stride of the panel steps' blocks (8-byte fragment loads)

// C[8 ti ..][8 tj ..] -= X[8 ti ..][q ..] Y[8 tj ..][q ..]^T for the tiles
// tj0 <= tj <= tj1 among tb .. tb + 3, eight columns q, all with row stride
// QS; one warp.  The tiles' loads all go ahead of their products, so that
// one tile's latency is paid, not each tile's.
__device__ __forceinline__ void rank8_quad(double *C, const double *X, const double *Y, int ti,
                                           int tb, int tj0, int tj1, int q) {
  const int lane = threadIdx.x & 31, r8 = lane >> 2, c4 = lane & 3;
  double *cr = C + (8 * ti + r8) * QS + 8 * tb + 2 * c4;
  const double *x = X + (8 * ti + r8) * QS + q + c4, *y = Y + (8 * tb + r8) * QS + q + c4;
  const double x0 = -x[0], x1 = -x[4];
  double d[4][2], y0[4], y1[4];
#pragma unroll
  for (int t = 0; t < 4; ++t)
    if (tb + t >= tj0 && tb + t <= tj1) {
      const double2 v = *(const double2 *)(cr + 8 * t);
      d[t][0] = v.x;
      d[t][1] = v.y;
      y0[t] = y[8 * t * QS];
      y1[t] = y[8 * t * QS + 4];
    }
#pragma unroll
  for (int t = 0; t < 4; ++t)
    if (tb + t >= tj0 && tb + t <= tj1) dmma(d[t], x0, y0[t]);
#pragma unroll
  for (int t = 0; t < 4; ++t)
    if (tb + t >= tj0 && tb + t <= tj1) {
      dmma(d[t], x1, y1[t]);
      *(double2 *)(cr + 8 * t) = make_double2(d[t][0], d[t][1]);
    }
}
__device__ __forceinline__ void rank8_row(double *C, const double *X, const double *Y, int ti,
                                          int tj0, int tj1, int q) {
  if (tj0 < 4) rank8_quad(C, X, Y, ti, 0, tj0, tj1, q);
  if (tj1 >= 4) rank8_quad(C, X, Y, ti, 4, tj0, tj1, q);
}

// v <- v L^{-T} for eight unknowns; l[i][k] and the reciprocal diagonal id
// of the 8 x 8 triangle at L (row stride QS)
__device__ __forceinline__ void solve8(double (&v)[8], const double *L, const double (&id)[8]) {
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    v[i] *= id[i];
#pragma unroll
    for (int k = i + 1; k < 8; ++k) v[k] = fma(-v[i], L[k * QS + i], v[k]);
  }
}

// Factor of the 64 x 64 diagonal block in A (row stride QS, lower triangle;
// rows and columns past the matrix are those of the identity), by 128
// threads.  Threads 0..63 each factor the 8 x 8 diagonal block in registers
// and solve their own row against it.  info[0] receives the first
// non-positive pivot (1-based), which then counts as 1.  Bound: the serial
// chain of 64 reciprocal square roots.
__device__ __forceinline__ void potrf64(double *A, int k0, int *info) {
  const int t = threadIdx.x, warp = t >> 5;
#pragma unroll 1
  for (int p = 0; p < NB; p += 8) {
    double l[8][8], id[8];
    if (t < 64) {
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int k = 0; k <= i; ++k) l[i][k] = A[(p + i) * QS + p + k];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        double d = l[k][k];
        if (!(d > 0.0)) {
          if (t == 0 && info[0] == 0) info[0] = k0 + p + k + 1;
          d = 1.0;
        }
        id[k] = rsqrt(d);
        l[k][k] = d * id[k];
#pragma unroll
        for (int i = k + 1; i < 8; ++i) l[i][k] *= id[k];
#pragma unroll
        for (int i = k + 1; i < 8; ++i)
#pragma unroll
          for (int m = k + 1; m <= i; ++m) l[i][m] = fma(-l[i][k], l[m][k], l[i][m]);
      }
      if (t >= p + 8) {
        double v[8];
        double2 *r = (double2 *)(A + t * QS + p);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const double2 w = r[i];
          v[2 * i] = w.x;
          v[2 * i + 1] = w.y;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          v[i] *= id[i];
#pragma unroll
          for (int k = i + 1; k < 8; ++k) v[k] = fma(-v[i], l[k][i], v[k]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) r[i] = make_double2(v[2 * i], v[2 * i + 1]);
      }
    }
    __syncthreads();
    // the diagonal block itself: read by every thread above, by no one below
    if (t == 0)
#pragma unroll
      for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int k = 0; k <= i; ++k) A[(p + i) * QS + p + k] = l[i][k];
    // rows 7 - w and 3 - w of the remaining tiles to warp w
    const int b0 = p / 8 + 1;
    if (7 - warp >= b0) rank8_row(A, A, A, 7 - warp, b0, 7 - warp, p);
    if (3 - warp >= b0) rank8_row(A, A, A, 3 - warp, b0, 3 - warp, p);
    __syncthreads();
  }
}

// the diagonal block at k0 of G into A (identity beyond nb, upper part zero),
// row stride QS
template <int NTHR>
__device__ __forceinline__ void load_diag(double *A, const double *G, int n, int k0, int nb) {
  // every address is one of the block's, so the loads are unconditional
  // and all in flight together
#pragma unroll 16
  for (int p = 0; p < NB * NB / NTHR; ++p) {
    const int e = threadIdx.x + p * NTHR, i = e >> 6, j = e & 63, r = min(i, nb - 1);
    const double v = G[(size_t)(k0 + r) * n + k0 + min(j, r)];
    A[i * QS + j] = i < nb && j <= i ? v : i == j ? 1.0 : 0.0;
  }
}
__device__ __forceinline__ void store_diag(const double *A, double *G, int n, int k0, int nb) {
  for (int e = threadIdx.x; e < NB * NB; e += blockDim.x) {
    const int i = e >> 6, j = e & 63;
    if (i < nb && j <= i) G[(size_t)(k0 + i) * n + k0 + j] = A[i * QS + j];
  }
}

// the first diagonal block
__global__ void __launch_bounds__(128) k_potrf_diag(double *G, int n, int nb, int *info) {
  __shared__ __align__(16) double A[NB * QS];
  load_diag<128>(A, G, n, 0, nb);
  __syncthreads();
  potrf64(A, 0, info);
  store_diag(A, G, n, 0, nb);
}

// L21 = A21 L11^{-T} for the rows below the panel and, as row n, the
// right-hand side x: 64 rows per block.
constexpr size_t TRSM_SMEM = (size_t)(2 * NB * QS + NB) * 8;
__global__ void __launch_bounds__(256) k_trsm_panel(double *G, int n, int k0, int nb, double *x) {
  extern __shared__ __align__(16) double tsm[];
  double *L = tsm, *X = L + NB * QS, *id = X + NB * QS;  // id: 1 / L[j][j]
  const int r0 = k0 + nb + blockIdx.x * 64, t = threadIdx.x, warp = t >> 5;
  load_diag<256>(L, G, n, k0, nb);
#pragma unroll
  for (int p = 0; p < NB * NB / 256; ++p) {
    const int e = t + p * 256, i = e >> 6, j = min(e & 63, nb - 1), r = min(r0 + i, n);
    X[i * QS + (e & 63)] = *(r < n ? G + (size_t)r * n + k0 + j : x + k0 + j);
  }
  __syncthreads();
  if (t < 64) id[t] = 1.0 / L[t * QS + t];
  __syncthreads();
#pragma unroll 1
  for (int p = 0; p < NB; p += 8) {
    if (t < 64) {
      double v[8], d[8];
      double2 *r = (double2 *)(X + t * QS + p);
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        const double2 w = r[i];
        v[2 * i] = w.x;
        v[2 * i + 1] = w.y;
      }
#pragma unroll
      for (int i = 0; i < 8; ++i) d[i] = id[p + i];
      solve8(v, L + p * QS + p, d);
#pragma unroll
      for (int i = 0; i < 4; ++i) r[i] = make_double2(v[2 * i], v[2 * i + 1]);
    }
    __syncthreads();
    // warp w updates rows 8 w .. of the remaining column groups
    rank8_row(X, X, L, warp, p / 8 + 1, 7, p);
    __syncthreads();
  }
#pragma unroll
  for (int p = 0; p < NB * NB / 256; ++p) {
    const int e = t + p * 256, i = e >> 6, j = e & 63, r = r0 + i;
    if (j < nb && r <= n) {
      if (r < n) G[(size_t)r * n + k0 + j] = X[i * QS + j];
      else x[k0 + j] = X[i * QS + j];
    }
  }
}

// Trailing update A22 -= L21 L21^T on the lower 64 x 64 tiles (block e the
// e-th tile of the triangle, accumulators starting from A22), on the
// diagonal tiles also the right-hand side x -= L21 y, and in block 0 the
// factor of the next diagonal block.  The panel's two strips of 64 rows sit
// in shared memory whole (64 k).  Bound: the FP64 tensor pipe and A22's
// traffic while the triangle is large, the factor's chain in the last
// dozen panels.
constexpr size_t TRAIL_SMEM = (size_t)2 * NB * PS * 8;
__global__ void __launch_bounds__(128, 3) k_syrk_trail(double *G, int n, int k0, double *x,
                                                       int *info) {
  extern __shared__ __align__(16) double ssm[];
  int ti, tj;
  low_tile(blockIdx.x, ti, tj);
  const int base = k0 + NB, i0 = base + ti * 64, j0 = base + tj * 64;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, r8 = lane >> 2, c4 = lane & 3;
  const int wm = (warp & 1) * 32, wn = (warp >> 1) * 32;
  __shared__ double ys[NB];  // the panel's part of the right-hand side
  if (t < NB) ys[t] = x[k0 + t];
  double *sa = ssm, *sb = ti == tj ? sa : sa + NB * PS;
#pragma unroll 8
  for (int p = 0; p < NB * NB / 128; ++p) {
    const int e = t + p * 128, r = e >> 6, k = e & 63;
    const bool ok = i0 + r < n;
    cp8(sa + r * PS + k, G + (ok ? (size_t)(i0 + r) * n + k0 + k : 0), ok);
  }
  if (ti != tj)
#pragma unroll 8
    for (int p = 0; p < NB * NB / 128; ++p) {
      const int e = t + p * 128, r = e >> 6, k = e & 63;
      const bool ok = j0 + r < n;
      cp8(sb + r * PS + k, G + (ok ? (size_t)(j0 + r) * n + k0 + k : 0), ok);
    }
  cp_commit();
  double acc[4][4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = i0 + wm + 8 * i + r8;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        // clamped, so that the loads are unconditional and all in flight
        // (what lies outside is computed and never stored)
        const int c = j0 + wn + 8 * j + 2 * c4 + e;
        acc[i][j][e] = G[(size_t)min(r, n - 1) * n + min(c, n - 1)];
      }
  }
  cp_wait<0>();
  __syncthreads();
#pragma unroll 1
  for (int kb = 0; kb < NB / 16; ++kb) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      double2 a[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a[i] = *(const double2 *)(sa + (wm + 8 * i + r8) * PS + 16 * kb + 4 * c4 + 2 * h);
        a[i].x = -a[i].x;
        a[i].y = -a[i].y;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const double2 b = *(const double2 *)(sb + (wn + 8 * j + r8) * PS + 16 * kb + 4 * c4 + 2 * h);
#pragma unroll
        for (int i = 0; i < 4; ++i) dmma(acc[i][j], a[i].x, b.x);
#pragma unroll
        for (int i = 0; i < 4; ++i) dmma(acc[i][j], a[i].y, b.y);
      }
    }
  }
  if (ti == tj && t < 64 && i0 + t < n) {
    double s = 0.0;
#pragma unroll 8
    for (int k = 0; k < NB; ++k) s = fma(sa[t * PS + k], ys[k], s);
    x[i0 + t] -= s;
  }
  if (blockIdx.x != 0) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = i0 + wm + 8 * i + r8;
#pragma unroll
      for (int j = 0; j < 4; ++j)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int c = j0 + wn + 8 * j + 2 * c4 + e;
          if (r < n && c <= r) G[(size_t)r * n + c] = acc[i][j][e];
        }
    }
    return;
  }
  __syncthreads();  // the strip is done with: the tile takes its place
  const int nb = min(NB, n - base);
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = wm + 8 * i + r8;
#pragma unroll
    for (int j = 0; j < 4; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = wn + 8 * j + 2 * c4 + e;
        sa[r * QS + c] = r < nb && c <= r ? acc[i][j][e] : r == c ? 1.0 : 0.0;
      }
  }
  __syncthreads();
  potrf64(sa, base, info);
  store_diag(sa, G, n, base, nb);
}

// One step of L^T u = y, from the last block of 64 unknowns to the first:
// block c takes the unknowns of block c, subtracts the part of the block
// solved by the last step (rows p0 .. p0 + pn), and block j, the one whose
// parts are then all in, solves its own 64 unknowns.  x holds y and then u.
__global__ void __launch_bounds__(256) k_back_step(const double *G, int n, int j, int p0, int pn,
                                                   double *x) {
  __shared__ double L[NB * QS];
  __shared__ double red[4][64], up[NB];
  const int c = blockIdx.x, c0 = c * NB, cn = min(NB, n - c0);
  const int t = threadIdx.x, col = t & 63, grp = t >> 6;
  if (c == j) load_diag<256>(L, G, n, c0, cn);
  if (t < pn) up[t] = x[p0 + t];
  __syncthreads();
  double s = 0.0;
  if (col < cn)
#pragma unroll 16
    for (int r = grp; r < pn; r += 4) s = fma(G[(size_t)(p0 + r) * n + c0 + col], up[r], s);
  red[grp][col] = s;
  __syncthreads();
  if (t >= 64) return;
  double y = 0.0;
  if (t < cn) y = x[c0 + t] - (red[0][t] + red[1][t] + red[2][t] + red[3][t]);
  if (c != j) {
    if (t < cn) x[c0 + t] = y;
    return;
  }
  red[0][t] = y;
  __syncwarp();
  asm volatile("bar.sync 1, 64;" ::: "memory");
  if (t >= 32) return;
  // lane t holds unknowns t and t + 32
  double y0 = red[0][t], y1 = red[0][t + 32];
  const double d0 = 1.0 / L[t * QS + t], d1 = 1.0 / L[(t + 32) * QS + t + 32];
#pragma unroll 4
  for (int k = 63; k >= 32; --k) {
    const double u = __shfl_sync(0xffffffffu, y1 * d1, k - 32);
    if (t == k - 32) y1 = u;
    else if (t < k - 32) y1 = fma(-L[k * QS + t + 32], u, y1);
    y0 = fma(-L[k * QS + t], u, y0);
  }
#pragma unroll 4
  for (int k = 31; k >= 0; --k) {
    const double u = __shfl_sync(0xffffffffu, y0 * d0, k);
    if (t == k) y0 = u;
    else if (t < k) y0 = fma(-L[k * QS + t], u, y0);
  }
  if (t < cn) x[c0 + t] = y0;
  if (t + 32 < cn) x[c0 + t + 32] = y1;
}

// FP32 copy of the rows with a padded leading dimension (zero past nw), the
// operand of the tensor-core metric; one block per row
__global__ void __launch_bounds__(256) k_rows_f32(const double *rows, int nw, float *J, int ldj) {
  const double *src = rows + (size_t)blockIdx.x * nw;
  float *dst = J + (size_t)blockIdx.x * ldj;
#pragma unroll 4
  for (int c = threadIdx.x; c < ldj; c += 256) dst[c] = c < nw ? (float)__ldcs(src + c) : 0.f;
}

// G[nc][nc] (lower triangle, zeroed here) = A^T A for A[nr][nc]: on the
// tensor cores in the split precision (split-BF16 products of an FP32 copy,
// FP32 accumulation per 512 rows, FP64 across them), else FP64 tiles
static int gram(const double *A, int nr, int nc, double *G, int prec, cudaStream_t st) {
  CKN(cudaMemsetAsync(G, 0, sizeof(double) * (size_t)nc * nc, st));
  int rc = RC_UNSUPPORTED;
  if (prec == PREC_SPLIT && gemm_tc_available()) {
    const int ldj = (nc + 15) / 16 * 16;
    DevScratch J;
    if (J.take(sizeof(float) * (size_t)nr * ldj, st) == cudaSuccess) {
      LAUNCH("k_rows_f32", st, k_rows_f32<<<nr, 256, 0, st>>>(A, nc, J.as<float>(), ldj));
      rc = gemm_tc_syrk(J.as<float>(), nr, nc, ldj, G, st);
    } else {
      cudaGetLastError();  // no room for the copy: the FP64 tiles need none
    }
  }
  if (rc != RC_UNSUPPORTED) return rc;
  return syrk_f64(A, nr, nc, G, st);
}

// Cholesky factorization of the damped G[n][n] (lower triangle) and the
// solve G x = x; -1 with the first non-positive pivot in the error text
static int chol_solve(double *G, int n, double *x, int *info, cudaStream_t st) {
  CKN(cudaMemsetAsync(info, 0, sizeof(int), st));
  CKN(cudaFuncSetAttribute(k_trsm_panel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)TRSM_SMEM));
  CKN(cudaFuncSetAttribute(k_syrk_trail, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)TRAIL_SMEM));
  LAUNCH("k_potrf_diag", st, k_potrf_diag<<<1, 128, 0, st>>>(G, n, std::min(NB, n), info));
  CKN(cudaGetLastError());
  for (int k0 = 0; k0 < n; k0 += NB) {
    const int nbk = std::min(NB, n - k0), rem = n - k0 - nbk;
    // the rows below the panel and the right-hand side
    LAUNCH("k_trsm_panel", st, (k_trsm_panel<<<(rem + 1 + 63) / 64, 256, TRSM_SMEM, st>>>(G, n, k0, nbk, x)));
    CKN(cudaGetLastError());
    if (rem > 0) {
      const int tt = (rem + 63) / 64;
      LAUNCH("k_syrk_trail", st, (k_syrk_trail<<<tt * (tt + 1) / 2, 128, TRAIL_SMEM, st>>>(G, n, k0, x, info)));
      CKN(cudaGetLastError());
    }
  }
  for (int j = (n - 1) / NB; j >= 0; --j) {
    const int p0 = std::min(n, (j + 1) * NB), pn = std::min(NB, n - p0);
    LAUNCH("k_chol_back", st, (k_back_step<<<j + 1, 256, 0, st>>>(G, n, j, p0, pn, x)));
    CKN(cudaGetLastError());
  }
  int hinfo = 0;
  CKN(cudaMemcpyAsync(&hinfo, info, sizeof(int), cudaMemcpyDeviceToHost, st));
  CKN(cudaStreamSynchronize(st));
  if (hinfo) {
    set_error("the damped metric is not positive definite at column " + std::to_string(hinfo));
    return RC_BAD_ARG;
  }
  return RC_OK;
}

int ngd_device(const double *rows, int nrow, int nw, const double *b, int nb,
               double mu, double *u, int prec, cudaStream_t st) {
  DevScratch G;
  CKN(G.take(sizeof(double) * (size_t)nw * nw, st));
  const int rc = gram(rows, nrow, nw, G.as<double>(), prec, st);
  return rc ? rc : ngd_solve_device(G.as<double>(), nw, b, nb, mu, u, st);
}

// The two halves of the primal step, for a step whose rows are spread over
// ranks: each rank forms its own J^T J, the caller sums the metrics (and
// the gradients) over the ranks, and every rank solves the summed system,
// as app/optimizer_module.f90:310-321 does with sum_over_ranks.
int ngd_gram_device(const double *rows, int nrow, int nw, double *G, int prec, cudaStream_t st) {
  return gram(rows, nrow, nw, G, prec, st);
}

int ngd_solve_device(double *G, int nw, const double *b, int nb, double mu, double *u,
                     cudaStream_t st) {
  DevScratch info;
  CKN(info.take(sizeof(int), st));
  LAUNCH("k_scale_damp", st, k_scale_damp<<<nw, 256, 0, st>>>(G, nw, 1.0 / (double)nb, mu, b, u));
  CKN(cudaGetLastError());
  return chol_solve(G, nw, u, info.as<int>(), st);
}

// ------------------------------------------------- dual (Gram-space) route
// The dual route of app/optimizer_module.f90:408-446: with G = J^T J / nb
// and the damping mu, the push-through identity gives
//   (G + mu I)^{-1} b' = (1 / mu) (b' - J^T K^{-1} (J b') / nb),
//   K = mu I + J J^T / nb  (nrow x nrow),  b' = b / nb,
// so the nw x nw metric is never formed: an nrow x nrow solve and two
// passes over the rows.  The step is the primal one to roundoff.

// T[nc][nr] = A^T for A[nr][nc], 32 x 32 tiles through shared memory
__global__ void k_transpose(const double *A, int nr, int nc, double *T) {
  __shared__ double tile[32][33];
  const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int r = r0 + i, c = c0 + threadIdx.x;
    tile[i][threadIdx.x] = (r < nr && c < nc) ? A[(size_t)r * nc + c] : 0.0;
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int c = c0 + i, r = r0 + threadIdx.x;
    if (c < nc && r < nr) T[(size_t)c * nr + r] = tile[threadIdx.x][i];
  }
}

// y[r] = alpha sum_i J[r][i] x[i], one warp per row
__global__ void k_rows_dot(const double *J, int nrow, int nw, const double *x, double alpha,
                           double *y) {
  const int lane = threadIdx.x & 31;
  for (int r = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); r < nrow;
       r += gridDim.x * (blockDim.x >> 5)) {
    double s = 0.0;
    for (int i = lane; i < nw; i += 32) s += J[(size_t)r * nw + i] * x[i];
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (lane == 0) y[r] = alpha * s;
  }
}

// part[c][i] = sum_r J[r][i] y[r] over the rows of chunk c = blockIdx.y
__global__ void __launch_bounds__(128) k_cols_dot(const double *J, int nrow, int nw,
                                                  const double *y, int rchunk, double *part) {
  const int i = blockIdx.x * 128 + threadIdx.x;
  const int r0 = blockIdx.y * rchunk, r1 = min(nrow, r0 + rchunk);
  if (i >= nw) return;
  double v = 0.0;
#pragma unroll 8
  for (int r = r0; r < r1; ++r) v = fma(__ldcs(J + (size_t)r * nw + i), __ldg(y + r), v);
  part[(size_t)blockIdx.y * nw + i] = v;
}

// u[i] = (b[i] / nb - sum_c part[c][i] / nb) / mu, the chunks in order; u may
// be b
__global__ void k_dual_step(int nw, int nchunk, const double *part, const double *b, double inv_nb,
                            double inv_mu, double *u) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= nw) return;
  double s = 0.0;
#pragma unroll 8
  for (int c = 0; c < nchunk; ++c) s += part[(size_t)c * nw + i];
  u[i] = (b[i] * inv_nb - s * inv_nb) * inv_mu;
}

int ngd_device_dual(const double *rows, int nrow, int nw, const double *b, int nb, double mu,
                    double *u, int prec, cudaStream_t st) {
  if (!(mu > 0.0)) {
    set_error("the dual natural-gradient step needs a positive damping mu");
    return RC_BAD_ARG;
  }
  DevScratch Ks, JTs, ys, infos, parts;
  CKN(Ks.take(sizeof(double) * (size_t)nrow * nrow, st));
  CKN(JTs.take(sizeof(double) * (size_t)nrow * nw, st));
  CKN(ys.take(sizeof(double) * (size_t)nrow, st));
  CKN(infos.take(sizeof(int), st));
  // J^T y: about four blocks per SM share the rows, at least 16 rows each
  const int gx = (nw + 127) / 128;
  const int gy = std::max(1, std::min((nrow + 15) / 16, grid_sms() * 4 / gx));
  const int rchunk = (nrow + gy - 1) / gy, nchunk = (nrow + rchunk - 1) / rchunk;
  CKN(parts.take(sizeof(double) * (size_t)nchunk * nw, st));
  double *K = Ks.as<double>(), *JT = JTs.as<double>(), *y = ys.as<double>();
  int *info = infos.as<int>();
  // K = J J^T: the Gram product of the transposed rows, always in FP64.
  // The step ends with (b' - J^T y / nb) / mu, a cancellation divided by a
  // small damping, which magnifies the rounding of split-BF16 products in K
  // far past what the primal solve sees (measured backward error 6e-3
  // against 1e-7); K is only nrow x nrow, so FP64 costs little here.
  (void)prec;
  LAUNCH("k_transpose", st, k_transpose<<<dim3((nw + 31) / 32, (nrow + 31) / 32), dim3(32, 8), 0, st>>>(rows, nrow, nw, JT));
  int rc = cudaGetLastError() == cudaSuccess ? RC_OK : RC_DEVICE;
  if (!rc) rc = gram(JT, nw, nrow, K, PREC_F64, st);
  if (!rc) {
    const double inv_nb = 1.0 / (double)nb;
    LAUNCH("k_scale_damp", st, k_scale_damp<<<nrow, 256, 0, st>>>(K, nrow, inv_nb, mu, nullptr, nullptr));
    LAUNCH("k_rows_dot", st, k_rows_dot<<<std::max(1, std::min(4096, (nrow + 7) / 8)), 256, 0, st>>>(rows, nrow, nw, b, inv_nb, y));
    rc = cudaGetLastError() == cudaSuccess ? RC_OK : RC_DEVICE;
    if (!rc) rc = chol_solve(K, nrow, y, info, st);
    if (!rc) {
      double *part = parts.as<double>();
      LAUNCH("k_cols_dot", st, (k_cols_dot<<<dim3(gx, nchunk), 128, 0, st>>>(rows, nrow, nw, y, rchunk, part)));
      LAUNCH("k_dual_step", st, k_dual_step<<<(nw + 255) / 256, 256, 0, st>>>(nw, nchunk, part, b, inv_nb, 1.0 / mu, u));
      rc = cudaGetLastError() == cudaSuccess ? RC_OK : RC_DEVICE;
      if (!rc && cudaStreamSynchronize(st) != cudaSuccess) rc = RC_DEVICE;
    }
  }
  if (rc == RC_DEVICE) set_error("the dual natural-gradient step failed on the device");
  return rc;
}

// ------------------------------------------------- no-allocation variant
// dnnf90_ngd_step_noalloc runs the plain FP64 route above on caller
// buffers without allocating device memory: the damped metric and the
// pivot flag live in this fixed area instead.  The array belongs to every
// GPU that loads the library, for the life of the process (8 MiB).
constexpr int NGD_NOALLOC_MAXW = 1024;
static __device__ __align__(256) double
    g_ngd_scratch[(size_t)NGD_NOALLOC_MAXW * NGD_NOALLOC_MAXW + 32];

int ngd_noalloc_maxw() { return NGD_NOALLOC_MAXW; }

// Device address of the scratch on the current device, looked up once per
// device (host code cannot use the array's name as a device address) and
// kept for the life of the process: it does not survive cudaDeviceReset.
// With lazy module loading (the CUDA 12 default) the array is backed when
// this file's module first loads on a device, which the lookup itself
// triggers, so that first call may take the 8 MiB from the device.
static double *ngd_scratch_ptr() {
  static std::mutex mu;
  static double *ptr[256] = {};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 256) return nullptr;
  std::lock_guard<std::mutex> lk(mu);
  if (!ptr[dev]) {
    double *p = nullptr;
    cudaError_t e = cudaGetSymbolAddress((void **)&p, g_ngd_scratch);
    if (e != cudaSuccess) {
      set_error(std::string("cudaGetSymbolAddress(ngd scratch): ") + cudaGetErrorString(e));
      return nullptr;
    }
    ptr[dev] = p;
  }
  return ptr[dev];
}

int ngd_device_noalloc(const double *rows, int nrow, int nw, const double *b, int nb,
                       double mu, double *u, cudaStream_t st) {
  if (nw > NGD_NOALLOC_MAXW) {
    set_error("dnnf90_ngd_step_noalloc: nweights " + std::to_string(nw) +
              " is above the fixed scratch limit of " + std::to_string(NGD_NOALLOC_MAXW));
    return RC_BAD_ARG;
  }
  if (!(mu > 0.0)) {
    set_error("dnnf90_ngd_step_noalloc: the damping mu must be positive");
    return RC_BAD_ARG;
  }
  // the call reads the pivot flag back into host memory and waits for its
  // stream, neither of which a stream being captured allows
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
    set_error("dnnf90_ngd_step_noalloc cannot be captured into a CUDA graph (it waits for "
              "its stream and reads a status back)");
    return RC_UNSUPPORTED;
  }
  double *G = ngd_scratch_ptr();
  if (!G) return RC_DEVICE;
  int *info = (int *)(G + (size_t)NGD_NOALLOC_MAXW * NGD_NOALLOC_MAXW);
  // the scratch keeps the previous call's contents: clear what accumulates
  CKN(cudaMemsetAsync(G, 0, sizeof(double) * (size_t)nw * nw, st));
  int rc = syrk_f64(rows, nrow, nw, G, st);
  if (rc) return rc;
  LAUNCH("k_scale_damp", st, k_scale_damp<<<nw, 256, 0, st>>>(G, nw, 1.0 / (double)nb, mu, b, u));
  CKN(cudaGetLastError());
  return chol_solve(G, nw, u, info, st);
}

}  // namespace dnnf90
