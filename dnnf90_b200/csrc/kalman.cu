// kalman.cu - the extended Kalman filter of lib/kalman_module.f90 on the
// device: the rank-one update of kf_update_grad (:353-490) over a sequence
// of observation rows, for the dense (global) and the node-wise decoupled
// covariance.
//
// Covariance store.  P is symmetric block diagonal (one block of nw for the
// dense filter, one block per neuron over (bias, fan-in) for the decoupled
// one, kf_block_map :172-189).  Each block keeps only its upper triangle,
// as 32 x 32 FP64 tiles (I <= J, row-major inside the tile, zero padding
// past the block edge); the diagonal tiles are kept whole.  The downdate
// and the symmetrisation of the reference,
//     P <- (P - kv pj^T) / lambda,  P_ij <- (P_ij + P_ji) / 2,  P_ii += q,
// give, for an element whose old value a is the same on both sides,
//     P_ij <- ((a - kv_i pj_j) + (a - kv_j pj_i)) / (2 lambda),
// an expression symmetric in (i, j), so each stored element is updated from
// its own value alone and the triangle never needs the transposed entry
// (the reference divides each term by lambda before the average; the two
// differ by rounding only).
//
// One observation is two launches.  The tile pass applies observation k
// (downdate, process noise, and w += kv xi on the diagonal tiles) and, in
// the same read of each tile, forms the products of the NEW covariance with
// the next row: row sums of tile (I, J) land in partial slot J of the rows
// of I, column sums in slot I of the rows of J, so that every (slot, row)
// is written once and no atomics are needed.  The reduce pass sums the
// slots into P j for that row, forms j.Pj per row tile, and its last CTA
// (found with a counter, no waiting) sums the row tiles' shares in a fixed
// order into the global denominator, applies the innovation gate and
// advances lambda.  A call therefore reads and writes the covariance once
// per observation, plus one read-only pass for the first row.
//
// Calls of several observations on a dense filter that is not small apply
// eight of them per pass (grouped updates, below).
//
// Small filters run a whole call as one cooperative launch (k_kf_seq): the
// same tile code, reduce and scalar step as phases between bounded grid
// barriers, with the same summation orders, so both paths give the same
// bits.  The iterated EKF (kf_iekf_iter) reuses the two-launch kernels, and
// the per-point pass (dnnf90_kf_pass) calls kf_run once per point with
// that point's row formed on the device.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstring>
#include <string>
#include <vector>

#include "engine.hpp"
#include "scratch.hpp"

namespace dnnf90 {

#define CKK(call)                                                      \
  do {                                                                 \
    cudaError_t e_ = (call);                                           \
    if (e_ != cudaSuccess) {                                           \
      set_error(std::string(#call) + ": " + cudaGetErrorString(e_));   \
      return e_ == cudaErrorMemoryAllocation ? RC_NOMEM : RC_DEVICE;   \
    }                                                                  \
  } while (0)

// which update path kf_run takes: -1 by size (the one-launch sequence for
// small filters), 0 two launches per update, 1 the one-launch sequence
static std::atomic<int> g_kf_path{-1};

int kf_force_path(int path) {
  if (path < -1 || path > 1) return RC_BAD_ARG;
  g_kf_path = path;
  return RC_OK;
}

constexpr int KT = 32;          // tile side
constexpr int KTE = KT * KT;    // elements per tile
constexpr int RED_THREADS = 512;

// tile pass modes
constexpr int KM_PJ = 0;        // products with the first row only
constexpr int KM_UPD_PJ = 1;    // apply observation k, products with row k+1
constexpr int KM_UPD = 2;       // apply the last observation of the call

struct KfRowArgs {
  const double *rows;  // [nobs][ld]
  size_t ld;
  const double *xi;    // [nobs] innovations (target - prediction)
  const double *scale; // [nobs] or null (1)
};

// iterated EKF: the prior weights and the current ones (wprior null: a
// plain update)
struct KfIekf {
  const double *wprior;
  const double *w;
  int final;
};

__device__ __forceinline__ double row_scale(const KfRowArgs &a, int k) {
  return a.scale ? a.scale[k] : 1.0;
}

// (I, J) of tile t in the row-major upper triangle of tb x tb tiles, where
// row I starts at t0(I) = I tb - I (I - 1) / 2
__device__ __forceinline__ void tri_tile(int t, int tb, int &I, int &J) {
  const double b = 2.0 * tb + 1.0;
  int i = (int)((b - sqrt(b * b - 8.0 * t)) * 0.5);
  auto t0 = [tb](int r) { return (long long)r * tb - (long long)r * (r - 1) / 2; };
  while (i > 0 && t0(i) > t) --i;
  while (i + 1 < tb && t0(i + 1) <= t) ++i;
  I = i;
  J = i + (int)(t - t0(i));
}

// the scalars of the observation a tile pass applies
struct KfScal {
  double lam, denom, sg, xi, q;
};

// Where tile t sits: block offset o, block size n, tile (I, J) and the
// block's partial slots.  DENSE (a single block of nw) derives the position
// from the index, so that nothing the vector loads need waits on a table
// read; the decoupled filter reads its tile table.
template <bool DENSE>
__device__ __forceinline__ void kf_tile_at(int t, const int4 *__restrict__ tiles, int nw,
                                           double *part, int &o, int &n, int &I, int &J,
                                           double *&pslot) {
  if (DENSE) {
    o = 0;
    n = nw;
    tri_tile(t, (nw + KT - 1) / KT, I, J);
    pslot = part;
  } else {
    // x: block offset, y: block size, z: I | J << 16, w: the block's partial slots
    const int4 d = tiles[t];
    o = d.x;
    n = d.y;
    I = d.z & 0xffff;
    J = d.z >> 16;
    pslot = part + d.w;
  }
}

// One tile of the pass, its elements v already loaded: the update of
// observation k (MODE != KM_PJ) and the products of the result with the
// next row (MODE != KM_UPD).  Every thread of the CTA calls it.
template <int MODE, bool CG = false>
__device__ __forceinline__ void kf_tile_body(double *tp, double (&v)[4], int o, int n, int I,
                                             int J, double *pslot, const double *__restrict__ pj,
                                             const KfScal &sc, double *__restrict__ w,
                                             const double *__restrict__ wb, const KfRowArgs &ra,
                                             int knext) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int tb = (n + KT - 1) / KT;
  __shared__ double s_pjR[KT], s_kvR[KT], s_pjC[KT], s_kvC[KT], s_jR[KT], s_jC[KT];
  __shared__ double s_col[8][KT + 1];
  if (threadIdx.x < KT) {
    const int R = I * KT + lane, C = J * KT + lane;
    if (MODE != KM_PJ) {
      // CG: P j was written by other CTAs of the same launch (the
      // one-launch sequence), so it is read past L1
      const double pr = R < n ? sc.sg * (CG ? __ldcg(pj + o + R) : pj[o + R]) : 0.0;
      const double pc = C < n ? sc.sg * (CG ? __ldcg(pj + o + C) : pj[o + C]) : 0.0;
      s_pjR[lane] = pr;
      s_kvR[lane] = pr / sc.denom;
      s_pjC[lane] = pc;
      s_kvC[lane] = pc / sc.denom;
    }
    if (MODE != KM_UPD) {
      const double sn = row_scale(ra, knext);
      const double *jn = ra.rows + (size_t)knext * ra.ld;
      s_jR[lane] = R < n ? sn * jn[o + R] : 0.0;
      s_jC[lane] = C < n ? sn * jn[o + C] : 0.0;
    }
  }
  __syncthreads();
  const int C = J * KT + lane;
  if (MODE != KM_PJ) {
    // 1/lambda once per tile: an FP64 division per element would cost as
    // much as the element's HBM traffic (lambda = 1 is exact either way)
    const double rl = 1.0 / sc.lam, hl = 0.5 * rl;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int r = warp + 8 * m, R = I * KT + r;
      if (R < n && C < n) {
        const double a = v[m];
        if (R == C) {
          double d = __fma_rn(-s_kvR[r], s_pjR[r], a) * rl;
          if (sc.q > 0.0) d += sc.q;
          v[m] = d;
        } else {
          const double x = __fma_rn(-s_kvR[r], s_pjC[lane], a);
          const double y = __fma_rn(-s_kvC[lane], s_pjR[r], a);
          v[m] = (x + y) * hl;
        }
      }
      __stcs(tp + r * KT + lane, v[m]);
    }
    if (I == J && threadIdx.x < KT) {
      const int R = I * KT + lane;
      if (R < n) w[o + R] = __fma_rn(s_kvR[lane], sc.xi, wb[o + R]);
    }
  }
  if (MODE != KM_UPD) {
    // row sums -> slot J of the rows of tile I
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      double s = v[m] * s_jC[lane];
#pragma unroll
      for (int off = 16; off; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
      const int R = I * KT + warp + 8 * m;
      if (lane == 0 && R < n) pslot[((size_t)I * tb + J) * KT + warp + 8 * m] = s;
    }
    if (I != J) {  // column sums -> slot I of the rows of tile J
      double s = 0.0;
#pragma unroll
      for (int m = 0; m < 4; ++m) s = __fma_rn(v[m], s_jR[warp + 8 * m], s);
      s_col[warp][lane] = s;
      __syncthreads();
      if (threadIdx.x < KT) {
        double c = 0.0;
#pragma unroll
        for (int u = 0; u < 8; ++u) c += s_col[u][lane];
        if (C < n) pslot[((size_t)J * tb + I) * KT + lane] = c;
      }
    }
  }
}

// One CTA per tile.
template <int MODE, bool DENSE>
__global__ void __launch_bounds__(256, 8) k_kf_tiles(const int4 *__restrict__ tiles,
                                                     double *__restrict__ P, int nw,
                                                     const double *__restrict__ pj,
                                                     KfState *__restrict__ st,
                                                     double *__restrict__ w,
                                                     const double *__restrict__ wb,
                                                     KfRowArgs ra, int knext,
                                                     double *__restrict__ part) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // the tile's own elements first: their addresses depend on nothing else,
  // so the HBM reads are in flight while the scalars and vectors arrive.
  // The covariance streams through with evict-first loads and stores, so
  // that the partial slots written beside it stay in L2 for the reduce.
  double *tp = P + (size_t)blockIdx.x * KTE;
  double v[4];
#pragma unroll
  for (int m = 0; m < 4; ++m) v[m] = __ldcs(tp + (warp + 8 * m) * KT + lane);
  int o, n, I, J;
  double *pslot;
  kf_tile_at<DENSE>(blockIdx.x, tiles, nw, part, o, n, I, J, pslot);
  if (st->status) return;
  KfScal sc{1.0, 1.0, 1.0, 0.0, 0.0};
  if (MODE != KM_PJ) sc = KfScal{st->lamk, st->denom, st->sg, st->xi, st->q};
  kf_tile_body<MODE>(tp, v, o, n, I, J, pslot, pj, sc, w, wb, ra, knext);
}

// Sum of the row tiles' shares dotp[2b] (and dotp[2b + 1]) over b < n in a
// fixed order that does not depend on the block size: thread i < 256 adds
// b = i, i + 256, ... in turn, and the 256 partial sums are added pairwise
// (i + 128, i + 64, ...).  Every thread of the block calls it (at least 256
// of them); the sums are returned to all.  The shares come from other CTAs,
// so they are read past L1.
__device__ __forceinline__ void kf_dot_sum(const double *dotp, int n, double &dot, double &cor) {
  __shared__ double s_d[256], s_c[256];
  const int i = threadIdx.x;
  if (i < 256) {
    double d = 0.0, c = 0.0;
    for (int b = i; b < n; b += 256) {
      d += __ldcg(dotp + 2 * b);
      c += __ldcg(dotp + 2 * b + 1);
    }
    s_d[i] = d;
    s_c[i] = c;
  }
  __syncthreads();
  for (int h = 128; h > 0; h >>= 1) {
    if (i < h) {
      s_d[i] += s_d[i + h];
      s_c[i] += s_c[i + h];
    }
    __syncthreads();
  }
  dot = s_d[0];
  cor = s_c[0];
  __syncthreads();
}

// P j of row k from the partial slots, j.Pj per CTA, and in the last CTA
// the scalars of observation k (denominator, gate, lambda).  One CTA per
// row tile: its slots are contiguous ([slot][32]), warp g of 16 sums slots
// g, g + 16, ..., and the sixteen sums of a row are added in a fixed order.
__global__ void __launch_bounds__(RED_THREADS) k_kf_reduce(const int4 *__restrict__ rtl,
                                                           const double *__restrict__ part,
                                                           double *__restrict__ pj, KfRowArgs ra,
                                                           int k, int kbase, KfIekf ie,
                                                           double *__restrict__ dotp,
                                                           unsigned *__restrict__ ctr,
                                                           KfState *__restrict__ st) {
  if (st->status) return;
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int4 rt = rtl[blockIdx.x];  // x: first weight, y: rows, z: slots, w: slot offset
  const double *src = part + rt.w;
  __shared__ double s_sum[RED_THREADS / 32][33];
  __shared__ bool s_last;
  double s = 0.0;
#pragma unroll 8
  for (int i = g; i < rt.z; i += RED_THREADS / 32) s += src[(size_t)i * KT + lane];
  s_sum[g][lane] = s;
  __syncthreads();
  if (g == 0) {
    double p = 0.0, prod = 0.0, corr = 0.0;
#pragma unroll
    for (int u = 0; u < RED_THREADS / 32; ++u) p += s_sum[u][lane];
    if (lane < rt.y) {
      const int R = rt.x + lane;
      const double jf = row_scale(ra, k) * ra.rows[(size_t)k * ra.ld + R];
      pj[R] = p;
      prod = jf * p;
      if (ie.wprior) corr = jf * (ie.wprior[R] - ie.w[R]);
    }
#pragma unroll
    for (int off = 16; off; off >>= 1) {
      prod += __shfl_xor_sync(0xffffffffu, prod, off);
      corr += __shfl_xor_sync(0xffffffffu, corr, off);
    }
    if (lane == 0) {
      dotp[2 * blockIdx.x] = prod;
      dotp[2 * blockIdx.x + 1] = corr;
      __threadfence();
      s_last = atomicAdd(ctr, 1u) == gridDim.x - 1;
    }
  }
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  double dot, cor;
  kf_dot_sum(dotp, gridDim.x, dot, cor);
  if (threadIdx.x != 0) return;
  *ctr = 0;
  const double lam = st->lam;
  double denom = lam + dot;
  if (!(denom > 0.0)) {
    st->status = kbase + k + 1;
    return;
  }
  double xi, sg = 1.0;
  if (ie.wprior) {
    // iterated EKF (kf_iekf_iter :534-640): the innovation linearised at the
    // prior, xi = -scale R - jf.(w- - w_i); no gate; lambda advances only
    // with the covariance on the final iteration
    xi = -row_scale(ra, k) * ra.xi[k] - cor;
  } else {
    xi = row_scale(ra, k) * ra.xi[k];
    const double gate = st->gate;
    if (gate > 0.0) {
      const double jpj = denom - lam;
      if (xi * xi > gate * gate * denom) {
        const double s2 = gate * gate * lam / (xi * xi - gate * gate * jpj);
        sg = sqrt(s2);
        xi = sg * xi;
        denom = lam + s2 * jpj;
        st->ngated += 1;
      }
    }
  }
  st->lamk = lam;
  st->denom = denom;
  st->sg = sg;
  st->xi = xi;
  if (!ie.wprior || ie.final) st->lam = __dadd_rn(__dmul_rn(st->lam0, lam), 1.0) - st->lam0;
}

// w = w- + kv xi without touching the covariance (a non-final IEKF iteration)
__global__ void k_kf_wonly(int nw, double *__restrict__ w, const double *__restrict__ wb,
                           const double *__restrict__ pj, const KfState *__restrict__ st) {
  if (st->status) return;
  const int R = blockIdx.x * blockDim.x + threadIdx.x;
  if (R < nw) w[R] = wb[R] + (st->sg * pj[R] / st->denom) * st->xi;
}

// ---------------------------------------------------- whole sequence, one launch
// For a small filter the two launches of an update cost more than their
// work.  k_kf_seq runs a whole call as one cooperative launch: the tile
// pass, the reduce and the scalars of every observation as phases separated
// by grid barriers, with the same per-tile code and the same summation
// orders as the two-kernel path, so the results are bit-identical.  The
// scalars are formed by every CTA from the same values; lambda and the gate
// count live in registers and CTA 0 writes them back at the end.

constexpr long KF_BAR_LIMIT = 1L << 24;  // polls before a grid barrier gives up

// barrier among the CTAs of a cooperative launch (sense by generation);
// false, with status -1, when a wait runs out or another CTA gave up
__device__ bool kf_grid_sync(KfBar *b, KfState *st) {
  __shared__ int s_ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    const unsigned g = *(volatile unsigned *)&b->gen;
    __threadfence();
    if (atomicAdd(&b->count, 1u) == gridDim.x - 1) {
      atomicExch(&b->count, 0u);
      __threadfence();
      atomicAdd(&b->gen, 1u);
    } else {
      ok = 0;
      for (long i = 0; i < KF_BAR_LIMIT; ++i) {
        if (*(volatile unsigned *)&b->gen != g) {
          ok = 1;
          break;
        }
        if (*(volatile int *)&st->status < 0) break;
        if (i > 32) __nanosleep(32);
      }
      if (!ok) atomicCAS(&st->status, 0, -1);
    }
    __threadfence();
    s_ok = ok;
  }
  __syncthreads();
  return s_ok != 0;
}

// the tiles of this CTA (t = blockIdx, blockIdx + grid, ...)
template <int MODE, bool DENSE>
__device__ __forceinline__ void kf_seq_tiles(const int4 *__restrict__ tiles, int ntile,
                                             double *__restrict__ P, int nw,
                                             const double *__restrict__ pj, const KfScal &sc,
                                             double *__restrict__ w, const KfRowArgs &ra,
                                             int knext, double *__restrict__ part) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  for (int t = blockIdx.x; t < ntile; t += gridDim.x) {
    double *tp = P + (size_t)t * KTE;
    double v[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) v[m] = __ldcs(tp + (warp + 8 * m) * KT + lane);
    int o, n, I, J;
    double *pslot;
    kf_tile_at<DENSE>(t, tiles, nw, part, o, n, I, J, pslot);
    kf_tile_body<MODE, true>(tp, v, o, n, I, J, pslot, pj, sc, w, w, ra, knext);
    __syncthreads();  // the tile's vectors are read before the next tile writes them
  }
}

template <bool DENSE>
__global__ void __launch_bounds__(256) k_kf_seq(const int4 *__restrict__ tiles, int ntile,
                                                double *__restrict__ P, int nw,
                                                const int4 *__restrict__ rtl, int nred,
                                                double *__restrict__ part, double *__restrict__ pj,
                                                double *__restrict__ dotp,
                                                KfState *__restrict__ st, KfBar *__restrict__ bar,
                                                double *__restrict__ w, KfRowArgs ra, int nobs,
                                                int kbase, int first, int has_next) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __shared__ double s_sum[16][33];
  __shared__ KfScal s_sc;
  __shared__ int s_fail;
  if (*(volatile int *)&st->status) return;
  double lam = st->lam;
  const double lam0 = st->lam0, q = st->q, gate = st->gate;
  int ngated = st->ngated;
  KfScal sc{1.0, 1.0, 1.0, 0.0, q};
  if (first) {
    kf_seq_tiles<KM_PJ, DENSE>(tiles, ntile, P, nw, pj, sc, w, ra, 0, part);
    if (!kf_grid_sync(bar, st)) return;
  }
  for (int k = 0; k < nobs; ++k) {
    // reduce: P j of row k and the row tiles' shares of j.Pj, in the order
    // of k_kf_reduce (16 slot groups: this warp takes groups warp, warp + 8)
    for (int rt = blockIdx.x; rt < nred; rt += gridDim.x) {
      const int4 r = rtl[rt];
      const double *src = part + r.w;
      double s0 = 0.0, s1 = 0.0;
      for (int i = warp; i < r.z; i += 16) s0 += __ldcg(src + (size_t)i * KT + lane);
      for (int i = warp + 8; i < r.z; i += 16) s1 += __ldcg(src + (size_t)i * KT + lane);
      s_sum[warp][lane] = s0;
      s_sum[warp + 8][lane] = s1;
      __syncthreads();
      if (warp == 0) {
        double p = 0.0, prod = 0.0;
#pragma unroll
        for (int u = 0; u < 16; ++u) p += s_sum[u][lane];
        if (lane < r.y) {
          const int R = r.x + lane;
          pj[R] = p;
          prod = row_scale(ra, k) * ra.rows[(size_t)k * ra.ld + R] * p;
        }
#pragma unroll
        for (int off = 16; off; off >>= 1) prod += __shfl_xor_sync(0xffffffffu, prod, off);
        if (lane == 0) {
          dotp[2 * rt] = prod;
          dotp[2 * rt + 1] = 0.0;
        }
      }
      __syncthreads();
    }
    if (!kf_grid_sync(bar, st)) return;
    // the scalars of observation k, the same in every CTA
    double dot, cor;
    kf_dot_sum(dotp, nred, dot, cor);
    if (threadIdx.x == 0) {
      double denom = lam + dot;
      int fail = !(denom > 0.0);
      double xi = row_scale(ra, k) * ra.xi[k], sg = 1.0;
      if (!fail && gate > 0.0) {
        const double jpj = denom - lam;
        if (xi * xi > gate * gate * denom) {
          const double s2 = gate * gate * lam / (xi * xi - gate * gate * jpj);
          sg = sqrt(s2);
          xi = sg * xi;
          denom = lam + s2 * jpj;
          ++ngated;
        }
      }
      s_sc = KfScal{lam, denom, sg, xi, q};
      s_fail = fail;
    }
    __syncthreads();
    if (s_fail) {
      if (blockIdx.x == 0 && threadIdx.x == 0) {
        st->status = kbase + k + 1;
        st->lam = lam;
        st->ngated = ngated;
      }
      return;
    }
    sc = s_sc;
    lam = __dadd_rn(__dmul_rn(lam0, lam), 1.0) - lam0;
    if (k + 1 < nobs || has_next) {
      kf_seq_tiles<KM_UPD_PJ, DENSE>(tiles, ntile, P, nw, pj, sc, w, ra, k + 1, part);
      if (!kf_grid_sync(bar, st)) return;
    } else {
      kf_seq_tiles<KM_UPD, DENSE>(tiles, ntile, P, nw, pj, sc, w, ra, 0, part);
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    st->lam = lam;
    st->ngated = ngated;
    st->lamk = sc.lam;
    st->denom = sc.denom;
    st->sg = sc.sg;
    st->xi = sc.xi;
  }
}

// ---------------------------------------------------- grouped updates
// A call hands over all its rows at once, so up to GM = 8 observations share
// one pass over the covariance.  With P the covariance before the group and
// Y_k = P j_k (jf_k = scale_k j_k, written j below), the covariance before
// observation k of the group is
//     P_k = a_k P + c_k I - sum_{i<k} b_i p_i p_i^T,   p_i = s_i P_i j_i
// (s_i the gate's scale), because each update is P <- (P - p p^T / denom) /
// lambda + q I: a <- a / lambda, c <- c / lambda + q, b_i <- b_i / lambda and
// b_k = 1 / (lambda denom).  Every p_i is therefore a combination of the Y_l
// and j_l, l <= i.  Its coefficients, the denominators and the gates come from
// running the same update on 8 x 8 matrices: G = (j_l . P_k j_m) and the
// coefficients of P_k j_m in the Y_l and in the j_l.  Rows that resemble each
// other make G's update a difference of nearly equal numbers, whose rounding
// the single updates share out over the whole covariance, so the products
// j_l . Y_m, these matrices and the combinations of the Y_l are double-double.
// (300 weights, 24 rows of correlation 0.9999, p0 = 1e4, weights against 80-bit
// arithmetic: single updates 3.2e-13 to 6.6e-13, groups in doubles 3.1e-12 to
// 7.8e-12, so 2.6e-13 to 4.1e-13; correlation 0.9, p0 = 10: 4.0e-16 to 4.5e-16,
// 3.0e-16 to 4.9e-16, 1.5e-16 to 1.9e-16.  Here, 1217 weights, the error against
// the single updates': weights 0.35 without correlation, 0.5 at 0.99, 2.1 at
// 0.9999 (10.6 in doubles), covariance 0.5, 1.8 (4.2) and 1.5 (11.3).)  Per group
// three launches:
//   k_kf_greduce  sums the partial products into Y, forms the 8 x 8
//                 products, and its last CTA runs the recursion over k
//   k_kf_gvec     U_i = sqrt(b_i) p_i, w += sum_k p_k xi_k / denom_k, and the
//                 next group's rows packed as [weight][8]
//   k_kf_gtiles   P <- a P + c I - U U^T and, in the same read, the products
//                 of the new P with the next group's rows
// The covariance is read and written once per eight observations instead of
// once per observation.  A sum of squares -U U^T rounds alike on both sides
// of the diagonal, so P stays exactly symmetric.  A denominator that is not
// positive ends the group there: the observations before it are applied.

constexpr int GM = 8;            // observations per group
constexpr int GW = 8;            // warps of k_kf_gtiles: tile rows of a row block
constexpr int GVS = 12;          // row stride of the staged column vectors (doubles)

// double-double: h + l, |l| at most half an ulp of h
struct Dd {
  double h, l;
};
__device__ __forceinline__ Dd dd_norm(double h, double l) {
  const double s = h + l;
  return {s, l - (s - h)};
}
__device__ __forceinline__ double two_sum_err(double a, double b, double s) {
  const double t = s - a;
  return (a - (s - t)) + (b - t);
}
__device__ __forceinline__ Dd dd_add(Dd a, Dd b) {
  const double s = a.h + b.h;
  return dd_norm(s, two_sum_err(a.h, b.h, s) + (a.l + b.l));
}
__device__ __forceinline__ Dd dd_sub(Dd a, Dd b) { return dd_add(a, {-b.h, -b.l}); }
__device__ __forceinline__ Dd dd_mul(Dd a, Dd b) {
  const double p = __dmul_rn(a.h, b.h);  // not fused with the sum that follows
  return dd_norm(p, fma(a.h, b.l, fma(a.l, b.h, fma(a.h, b.h, -p))));
}
__device__ __forceinline__ Dd dd_div(Dd a, Dd b) {
  const double q = a.h / b.h, p = __dmul_rn(q, b.h);
  const double r = ((a.h - p) - fma(q, b.h, -p)) + fma(-q, b.l, a.l);
  return dd_norm(q, r / b.h);
}
__device__ __forceinline__ Dd dd_sqrt(Dd a) {  // a >= 0
  if (!(a.h > 0.0)) return {0.0, 0.0};
  const double s = sqrt(a.h);
  return dd_norm(s, (fma(-s, s, a.h) + a.l) / (2.0 * s));
}
// a running sum: h the sum in doubles, l what it has rounded off
__device__ __forceinline__ void dd_acc(Dd &a, double h, double l) {
  const double s = a.h + h;
  a.l += two_sum_err(a.h, h, s) + l;
  a.h = s;
}
// a running sum plus x y
__device__ __forceinline__ void dd_fma(Dd &a, Dd x, double y) {
  const double p = __dmul_rn(x.h, y);
  dd_acc(a, p, fma(x.l, y, fma(x.h, y, -p)));
}

struct KfGroup {
  int m;                         // observations to apply (0: none)
  double a, c;
  Dd ua[GM][GM], ub[GM][GM];     // U_i = sum_l ua[i][l] Y_l + ub[i][l] j_l
  Dd wa[GM], wb[GM];             // w += sum_l wa[l] Y_l + wb[l] j_l
};

__device__ __forceinline__ void kf_dmma(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}
__device__ __forceinline__ void kf_cp16(void *dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   (uint32_t)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}
// 16-byte chunk of (row, column pair c2) in a staged tile: the exclusive or
// spreads the rows so that both the fragment reads of 16 bytes (8 rows x 4
// pairs) and the transposed ones of 8 bytes (4 rows x 4 columns per half
// warp) meet each bank once
__device__ __forceinline__ int kf_chunk(int row, int c2) {
  return row * 16 + (c2 ^ (((row & 1) << 2) | (row & 2)));
}

// One CTA per item: a row block of eight tile rows I0 .. I0 + 7, one per
// warp, over the column tiles J0 .. J0 + Jn - 1.  A warp holds its 32 x 32
// tile as 4 x 4 fragments of the FP64 tensor cores (mma.sync m8n8k4, 32
// products each for the update and the two products with the next rows); the
// fragment of the updated tile is itself the left operand of the row
// products, with column 8 j + 2 c4 + e as the product's k; the column
// products read the tile transposed from shared memory.  The next column's
// tiles and vectors stream in by cp.async meanwhile.  Row products stay in
// registers along the item, column products are summed over the eight warps,
// so the partial sums are a tenth of the covariance's traffic.
// Bound: HBM; at nw = 17025 one pass takes 450 us for 2.32 GB (5.1 TB/s), 73 us
// per observation with the two small launches, against 569 for single updates.
template <int MODE>
__global__ void __launch_bounds__(GW * 32, 1)
    k_kf_gtiles(const int4 *__restrict__ items, int n, double *__restrict__ P,
                const double *__restrict__ U, const double *__restrict__ Jn,
                const KfGroup *__restrict__ grp, const KfState *__restrict__ st,
                double *__restrict__ rpart, double *__restrict__ cpart) {
  extern __shared__ __align__(16) double gsm[];
  double *tiles = gsm;                          // [2][GW][KTE]
  double *vec = tiles + 2 * GW * KTE;           // [2][2][KT * GVS]: U, J of the column tile
  double *colb = vec + 2 * 2 * KT * GVS;        // [GW][KT * GM]
  double ga = 1.0, gc = 0.0;
  if (MODE == KM_PJ) {
    if (st->status) return;
  } else {
    if (grp->m == 0) return;
    ga = grp->a;
    gc = grp->c;
  }
  const int4 ia = items[2 * blockIdx.x], ib = items[2 * blockIdx.x + 1];
  const int I0 = ia.x, J0 = ia.y, nJ = ia.z, rp = ib.x, cp = ib.y;
  const int tb = (n + KT - 1) / KT;
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31, r8 = lane >> 2, c4 = lane & 3;
  const int I = I0 + warp;
  // first tile of this warp's row: (I, J) sits at row0 + J
  double *row0 = P + ((size_t)I * tb - (size_t)I * (I - 1) / 2 - I) * KTE;
  auto stage = [&](int jj) {
    const int J = J0 + jj, buf = jj & 1;
    if (I < tb && I <= J) {
      double *dst = tiles + (buf * GW + warp) * KTE;
      const double *src = row0 + (size_t)J * KTE;
#pragma unroll
      for (int q = 0; q < KTE / 2 / 32; ++q) {
        const int e = q * 32 + lane;  // 16-byte chunk: row e / 16, pair e % 16
        kf_cp16(dst + 2 * kf_chunk(e >> 4, e & 15), src + 2 * e);
      }
    }
    // the vectors of the column tile: 32 rows of 8 doubles each
    {
      const int which = t >> 7, e = t & 127, r = e >> 2, c = (e & 3) * 2, R = J * KT + r;
      double *dst = vec + (buf * 2 + which) * KT * GVS + r * GVS + c;
      const double *src = which ? Jn : U;
      if (which ? MODE != KM_UPD : MODE != KM_PJ) {
        if (R < n) kf_cp16(dst, src + (size_t)R * GM + c);
        else *(double2 *)dst = make_double2(0.0, 0.0);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  stage(0);
  double ur[4][2], jr[4][2], yr[4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int s = 0; s < 2; ++s) {
      const int Ru = I * KT + 8 * i + r8, Rj = I * KT + 8 * i + c4 + 4 * s;
      ur[i][s] = MODE != KM_PJ && Ru < n ? -U[(size_t)Ru * GM + c4 + 4 * s] : 0.0;
      jr[i][s] = MODE != KM_UPD && Rj < n ? Jn[(size_t)Rj * GM + r8] : 0.0;
      yr[i][s] = 0.0;
    }
  for (int jj = 0; jj < nJ; ++jj) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();  // this column's vectors are in; every warp is done with the last column
    if (jj + 1 < nJ) stage(jj + 1);
    const int J = J0 + jj, buf = jj & 1;
    const bool act = I < tb && I <= J;
    double *tile = tiles + (buf * GW + warp) * KTE;
    const double *uc = vec + (buf * 2) * KT * GVS, *jc = uc + KT * GVS;
    double yc[4][2];
#pragma unroll
    for (int j = 0; j < 4; ++j) yc[j][0] = yc[j][1] = 0.0;
    if (act) {
      __syncwarp();  // this warp's copies of the tile
      double *gp = row0 + (size_t)J * KTE;
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        double v[4][2];
        const int row = 8 * i + r8;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const double2 x = *(const double2 *)(tile + 2 * kf_chunk(row, 4 * j + c4));
          v[j][0] = x.x;
          v[j][1] = x.y;
        }
        if (MODE != KM_PJ) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            v[j][0] *= ga;
            v[j][1] *= ga;
#pragma unroll
            for (int s = 0; s < 2; ++s)
              kf_dmma(v[j], ur[i][s], uc[(8 * j + r8) * GVS + c4 + 4 * s]);
            if (I == J && i == j && I * KT + row < n) {
              if (r8 == 2 * c4) v[j][0] += gc;
              if (r8 == 2 * c4 + 1) v[j][1] += gc;
            }
            const double2 x = make_double2(v[j][0], v[j][1]);
            if (MODE != KM_UPD) *(double2 *)(tile + 2 * kf_chunk(row, 4 * j + c4)) = x;
            __stcs((double2 *)(gp + row * KT + 8 * j + 2 * c4), x);
          }
        }
        if (MODE != KM_UPD)
#pragma unroll
          for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 2; ++e)
              kf_dmma(yr[i], v[j][e], jc[(8 * j + 2 * c4 + e) * GVS + r8]);
      }
      if (MODE != KM_UPD && I != J) {
        __syncwarp();  // the updated tile is in shared memory
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
          for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int s = 0; s < 2; ++s) {
              const int row = 8 * i + c4 + 4 * s, col = 8 * j + r8;
              kf_dmma(yc[j], tile[2 * kf_chunk(row, col >> 1) + (col & 1)], jr[i][s]);
            }
      }
    }
    if (MODE != KM_UPD) {
#pragma unroll
      for (int j = 0; j < 4; ++j)
        *(double2 *)(colb + warp * KT * GM + (8 * j + r8) * GM + 2 * c4) =
            make_double2(yc[j][0], yc[j][1]);
      __syncthreads();
      double v = 0.0;
#pragma unroll
      for (int w = 0; w < GW; ++w) v += colb[w * KT * GM + t];
      cpart[(size_t)(cp + jj) * KT * GM + t] = v;
    }
  }
  if (MODE != KM_UPD)
#pragma unroll
    for (int i = 0; i < 4; ++i)
      *(double2 *)(rpart + (size_t)(rp + warp) * KT * GM + (8 * i + r8) * GM + 2 * c4) =
          make_double2(yr[i][0], yr[i][1]);
}

// Y of one row tile from the partial sums (column partials of the row blocks
// 0 .. K / 8, then the row block's own segments, in that order), the tile's
// shares of j_l . Y_k and j_l . j_k, and in the last CTA (a counter, no
// waiting) their totals and the recursion over the group's observations.
constexpr int GRT = 512;
__global__ void __launch_bounds__(GRT)
    k_kf_greduce(int nw, const int4 *__restrict__ grt,
                 const double *__restrict__ rpart, const double *__restrict__ cpart,
                 const double *__restrict__ J, double *__restrict__ Y, KfRowArgs ra, int k0, int m,
                 int kbase, double2 *__restrict__ dots, unsigned *__restrict__ ctr,
                 KfGroup *__restrict__ grp, KfState *__restrict__ st) {
  __shared__ double ys[KT * GM], js[KT * GM], half[KT * GM];
  __shared__ Dd tot[4][2 * GM * GM];
  __shared__ Dd mat[3][GM][GM];        // G and the coefficients of P_k j_m in Y_l, in j_l
  __shared__ Dd al[GM][GM], be[GM][GM], bb[GM], wc[GM];
  __shared__ bool s_last;
  const int t = threadIdx.x;
  if (st->status) {  // an earlier group failed: nothing is applied from there on
    if (blockIdx.x == 0 && t == 0) grp->m = 0;
    return;
  }
  const int K = blockIdx.x, tb = gridDim.x, nb = K / GW;  // row tile, tiles per side
  const int4 gr = grt[K];            // x: its first row partial, y: segments of its row block
  {
    const int e = t & 255, h = t >> 8;  // even terms, odd terms
    const int terms = nb + 1 + gr.y;
    double v = 0.0;
#pragma unroll 8
    for (int q = h; q < terms; q += 2) {
      const double *src =
          q <= nb ? cpart + (size_t)(q * tb - GW / 2 * q * (q - 1) + K - GW * q) * KT * GM
                  : rpart + (size_t)(gr.x + (q - nb - 1) * GW) * KT * GM;
      v += __ldcg(src + e);
    }
    if (h) half[e] = v;
    __syncthreads();
    if (!h) {
      v += half[e];
      const bool ok = K * KT + (e >> 3) < nw;
      ys[e] = ok ? v : 0.0;
      js[e] = ok ? J[(size_t)K * KT * GM + e] : 0.0;
      if (ok) Y[(size_t)K * KT * GM + e] = v;
    }
  }
  __syncthreads();
  if (t < 2 * GM * GM) {  // j_l . Y_k, then j_l . j_k
    const int l = (t >> 3) & 7, k = t & 7;
    const double *b = t < GM * GM ? ys : js;
    Dd v = {0.0, 0.0};
#pragma unroll 8
    for (int r = 0; r < KT; ++r) {
      const double x = js[r * GM + l], y = b[r * GM + k], p = __dmul_rn(x, y);
      dd_acc(v, p, fma(x, y, -p));
    }
    dots[(size_t)blockIdx.x * 2 * GM * GM + t] = make_double2(v.h, v.l);
  }
  __threadfence();
  __syncthreads();
  if (t == 0) s_last = atomicAdd(ctr, 1u) == gridDim.x - 1;
  __syncthreads();
  if (!s_last) return;
  __threadfence();
  {
    const int e = t & 127, h = t >> 7;
    Dd v = {0.0, 0.0};
#pragma unroll 16
    for (int b = h; b < (int)gridDim.x; b += 4) {
      const double2 d = __ldcg(dots + (size_t)b * 2 * GM * GM + e);
      dd_acc(v, d.x, d.y);
    }
    tot[h][e] = v;
  }
  __syncthreads();
  if (t < 128) {
    Dd v = tot[0][t];
    for (int h = 1; h < 4; ++h) dd_acc(v, tot[h][t].h, tot[h][t].l);
    // an overflowed product keeps its infinity
    tot[0][t] = fabs(v.h) <= 1.7976931348623157e308 ? dd_norm(v.h, v.l) : Dd{v.h, 0.0};
  }
  __syncthreads();
  // the recursion: thread t < 192 holds entry (l, c) of one of the matrices
  const int which = t >> 6, l = (t >> 3) & 7, c8 = t & 7;
  const bool on = which < 3;
  if (on)
    mat[which][l][c8] =
        which == 0 ? tot[0][l * GM + c8] : Dd{which == 1 && l == c8 ? 1.0 : 0.0, 0.0};
  const double q = st->q > 0.0 ? st->q : 0.0, gate = st->gate, lam0 = st->lam0;
  double lam = st->lam;
  Dd a = {1.0, 0.0}, c = {0.0, 0.0}, b = {0.0, 0.0};  // b: of observation t, for t < 8
  int k = 0, ng = 0, fail = 0;
  double lamk = lam, denomk = 0.0, sgk = 1.0, xik = 0.0;
  __syncthreads();
  for (; k < m; ++k) {
    const Dd lm = {lam, 0.0}, jpj = mat[0][k][k];
    double den = lam + jpj.h;
    if (!(den > 0.0)) {
      fail = kbase + k0 + k + 1;
      break;
    }
    double xi = row_scale(ra, k0 + k) * ra.xi[k0 + k], sg = 1.0;
    Dd s2 = {1.0, 0.0};
    if (gate > 0.0 && xi * xi > gate * gate * den) {
      s2.h = gate * gate * lam / (xi * xi - gate * gate * jpj.h);
      sg = sqrt(s2.h);
      xi = sg * xi;
      s2 = dd_mul({sg, 0.0}, {sg, 0.0});
      ++ng;
    }
    // P_{k+1} j = (P_k j - p_k (s2 j_k . P_k j) / denom) / lambda + q j
    const bool inf = !(den <= 1.7976931348623157e308);
    const Dd dd = inf ? Dd{den, 0.0} : dd_add(lm, dd_mul(s2, jpj));
    den = dd.h;
    Dd v = {0.0, 0.0}, pa = v, pb = v;
    if (on) {
      v = mat[which][l][c8];
      if (!inf)
        v = dd_sub(v, dd_mul(mat[which][l][k], dd_div(dd_mul(s2, mat[0][k][c8]), dd)));
      v = dd_div(v, lm);
      if (q > 0.0) {
        if (which == 0) v = dd_add(v, dd_mul({q, 0.0}, tot[0][GM * GM + l * GM + c8]));
        else if (which == 2 && l == c8) v = dd_add(v, {q, 0.0});
      }
    }
    if (t < GM) {
      pa = dd_mul({sg, 0.0}, mat[1][t][k]);
      pb = dd_mul({sg, 0.0}, mat[2][t][k]);
      b = t == k ? (inf ? Dd{0.0, 0.0} : dd_div({1.0, 0.0}, dd_mul(lm, dd))) : dd_div(b, lm);
      al[k][t] = pa;
      be[k][t] = pb;
      if (t == k) wc[k] = inf ? Dd{0.0, 0.0} : dd_div({xi, 0.0}, dd);
    }
    a = dd_div(a, lm);
    c = dd_add(dd_div(c, lm), {q, 0.0});
    lamk = lam;
    denomk = den;
    sgk = sg;
    xik = xi;
    lam = __dadd_rn(__dmul_rn(lam0, lam), 1.0) - lam0;
    __syncthreads();  // every entry of step k is read
    if (on) mat[which][l][c8] = v;
    __syncthreads();
  }
  if (t < GM) bb[t] = dd_sqrt(b);
  __syncthreads();
  if (t < GM) {
    Dd wa = {0.0, 0.0}, wb = wa;
    for (int i = 0; i < k; ++i) {
      grp->ua[i][t] = dd_mul(bb[i], al[i][t]);
      grp->ub[i][t] = dd_mul(bb[i], be[i][t]);
      wa = dd_add(wa, dd_mul(wc[i], al[i][t]));
      wb = dd_add(wb, dd_mul(wc[i], be[i][t]));
    }
    for (int i = k; i < GM; ++i) grp->ua[i][t] = grp->ub[i][t] = {0.0, 0.0};
    grp->wa[t] = wa;
    grp->wb[t] = wb;
  }
  if (t == 0) {
    *ctr = 0;
    grp->m = k;
    grp->a = a.h;
    grp->c = c.h;
    st->lam = lam;
    st->ngated += ng;
    if (k > 0) {
      st->lamk = lamk;
      st->denom = denomk;
      st->sg = sgk;
      st->xi = xik;
    }
    if (fail) st->status = fail;
  }
}

// U, the weights and the next group's packed rows (grp null: only the rows);
// one thread per weight
__global__ void __launch_bounds__(128)
    k_kf_gvec(int nw, const KfGroup *__restrict__ grp, const double *__restrict__ Y,
              const double *J, double *__restrict__ U, double *__restrict__ w,
              KfRowArgs ra, int knext, int mnext, double *Jnext) {
  __shared__ KfGroup g;
  const int R = blockIdx.x * 128 + threadIdx.x;
  if (grp) {
    for (int e = threadIdx.x; e < (int)(sizeof(KfGroup) / 4); e += 128)
      ((int *)&g)[e] = ((const int *)grp)[e];
    __syncthreads();
    if (g.m == 0) return;
  }
  if (R >= nw) return;
  if (grp) {
    double y[GM], j[GM];
#pragma unroll
    for (int l = 0; l < GM; l += 2) {
      const double2 a = *(const double2 *)(Y + (size_t)R * GM + l);
      const double2 b = *(const double2 *)(J + (size_t)R * GM + l);
      // rows from a failed observation on take no part (they may hold NaN)
      y[l] = l < g.m ? a.x : 0.0;
      y[l + 1] = l + 1 < g.m ? a.y : 0.0;
      j[l] = l < g.m ? b.x : 0.0;
      j[l + 1] = l + 1 < g.m ? b.y : 0.0;
    }
    // sums of nearly opposite terms where the rows resemble each other
    const bool cj = g.c != 0.0;  // without process noise the j_l take no part
    Dd dw = {0.0, 0.0};
#pragma unroll
    for (int l = 0; l < GM; ++l) {
      dd_fma(dw, g.wa[l], y[l]);
      if (cj) dd_fma(dw, g.wb[l], j[l]);
    }
    w[R] += dw.h + dw.l;
#pragma unroll
    for (int i = 0; i < GM; i += 2) {
      double u[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        Dd v = {0.0, 0.0};
#pragma unroll
        for (int l = 0; l <= i + h; ++l) {
          dd_fma(v, g.ua[i + h][l], y[l]);
          if (cj) dd_fma(v, g.ub[i + h][l], j[l]);
        }
        u[h] = v.h + v.l;
      }
      *(double2 *)(U + (size_t)R * GM + i) = make_double2(u[0], u[1]);
    }
  }
  if (mnext > 0) {
    double v[GM];
#pragma unroll
    for (int k = 0; k < GM; ++k)
      v[k] = k < mnext ? row_scale(ra, knext + k) * ra.rows[(size_t)(knext + k) * ra.ld + R] : 0.0;
#pragma unroll
    for (int k = 0; k < GM; k += 2)
      *(double2 *)(Jnext + (size_t)R * GM + k) = make_double2(v[k], v[k + 1]);
  }
}

__global__ void k_kf_init_tiles(const int4 *__restrict__ tiles, double *__restrict__ P, double p0) {
  const int4 t = tiles[blockIdx.x];
  double *tp = P + (size_t)blockIdx.x * KTE;
  for (int e = threadIdx.x; e < KTE; e += blockDim.x) {
    const int r = e / KT, c = e - r * KT;
    const int R = (t.z & 0xffff) * KT + r, C = (t.z >> 16) * KT + c;
    tp[e] = (R == C && R < t.y) ? p0 : 0.0;
  }
}

void KfDev::release() {
  cudaFree(base);
  cudaFree(stage);
  *this = KfDev();
}

// Places of a filter's arrays in its one allocation
struct KfLayout {
  size_t cur = 0;
  size_t take(size_t bytes) {
    const size_t at = cur;
    cur = (cur + bytes + 255) / 256 * 256;
    return at;
  }
};

// Dense filters of at least this many tiles group the observations of a call
// (of at least KF_GROUP_OBS); smaller ones keep the one-launch sequence, whose
// bits do not depend on how a sequence is split into calls.
// The decoupled filter keeps single updates: its blocks share the denominators
// but each has products j_l . P j_k of its own, so that the recursion would
// run per block.
// Measured per observation, 64 (3) to a call, against the faster of the
// single-update paths: nw = 1217 6.6 (25) us against 14.1 (27), 4545 10.7 (36)
// against 50 (63), 17025 73 (233) against 566 (568).
constexpr int KF_GROUP_TILES = 512, KF_GROUP_OBS = 3;
constexpr size_t GT_SMEM =
    (size_t)(2 * GW * KTE + 2 * 2 * KT * GVS + GW * KT * GM) * sizeof(double);

// Work items of the grouped updates, the partial tiles they write (rows, columns)
static void group_items(int tb, std::vector<int4> &items, std::vector<int4> &grt, int &rp, int &cp) {
  long steps = 0;
  for (int I0 = 0; I0 < tb; I0 += GW) steps += tb - I0;
  // column tiles per item: about 12, so that its start-up is small beside
  // it, and a whole number of waves of one CTA per SM
  const long waves = std::max(1L, (steps + 6L * grid_sms()) / (12L * grid_sms()));
  const int seg = (int)std::max(2L, (steps + waves * grid_sms() - 1) / (waves * grid_sms()));
  cp = rp = 0;
  for (int I0 = 0; I0 < tb; I0 += GW) {
    const int rblock = rp, ns = (tb - I0 + seg - 1) / seg;
    for (int s = 0; s < ns; ++s) {
      const int J0 = I0 + s * seg, nJ = std::min(seg, tb - J0);
      items.push_back(make_int4(I0, J0, nJ, 0));
      items.push_back(make_int4(rp, cp, 0, 0));
      rp += GW;
      cp += nJ;
    }
    for (int K = I0; K < std::min(tb, I0 + GW); ++K) grt.push_back(make_int4(rblock + K - I0, ns, 0, 0));
  }
}

template <int MODE>
static int launch_gtiles(const KfDev &d, const double *Jn, cudaStream_t s) {
  CKK(cudaFuncSetAttribute(k_kf_gtiles<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)GT_SMEM));
  LAUNCH("k_kf_gtiles", s,
         (k_kf_gtiles<MODE><<<d.nitem, GW * 32, GT_SMEM, s>>>(
             d.gitems, d.nw, d.P, d.gU, Jn, (const KfGroup *)d.grp, d.st, d.grpart, d.gcpart)));
  CKK(cudaGetLastError());
  return RC_OK;
}

// the observations of one call, eight to a pass over the covariance
static int run_groups(KfDev &d, int nobs, const KfRowArgs &ra, double *w, cudaStream_t s,
                      int kbase) {
  KfGroup *grp = (KfGroup *)d.grp;
  const int gv = (d.nw + 127) / 128;
  int rc;
  LAUNCH("k_kf_gvec", s, (k_kf_gvec<<<gv, 128, 0, s>>>(d.nw, nullptr, d.gY, d.gJ[0], d.gU, w, ra, 0,
                                                       std::min(GM, nobs), d.gJ[0])));
  if ((rc = launch_gtiles<KM_PJ>(d, d.gJ[0], s))) return rc;
  for (int k0 = 0, b = 0; k0 < nobs; k0 += GM, b ^= 1) {
    const int m = std::min(GM, nobs - k0), mn = std::max(0, std::min(GM, nobs - k0 - GM));
    LAUNCH("k_kf_greduce", s,
           (k_kf_greduce<<<d.nred, GRT, 0, s>>>(d.nw, d.grt, d.grpart, d.gcpart, d.gJ[b], d.gY, ra,
                                                k0, m, kbase, d.gdots, d.ctr, grp, d.st)));
    LAUNCH("k_kf_gvec", s, (k_kf_gvec<<<gv, 128, 0, s>>>(d.nw, grp, d.gY, d.gJ[b], d.gU, w, ra,
                                                         k0 + GM, mn, d.gJ[b ^ 1])));
    if ((rc = mn ? launch_gtiles<KM_UPD_PJ>(d, d.gJ[b ^ 1], s)
                 : launch_gtiles<KM_UPD>(d, d.gJ[b ^ 1], s)))
      return rc;
  }
  CKK(cudaGetLastError());
  return RC_OK;
}

int kf_create(KfDev &d, const std::vector<int> &bsz, const std::vector<int> &boff, double p0,
              double lam_ini, double lam0, double q, double gate) {
  d.release();
  int nw = 0;
  for (size_t b = 0; b < bsz.size(); ++b) nw = std::max(nw, boff[b] + bsz[b]);
  // tiles (I <= J) of each block's triangle, and the block's partial slots:
  // [row tile K][slot s][32] at a per-block offset
  std::vector<int4> tl, rtl;
  size_t pslots = 0;
  for (size_t b = 0; b < bsz.size(); ++b) {
    const int n = bsz[b], o = boff[b], tb = (n + KT - 1) / KT;
    if (tb > 0xffff) {
      set_error("kalman: covariance block too large");
      return RC_UNSUPPORTED;
    }
    for (int I = 0; I < tb; ++I)
      for (int J = I; J < tb; ++J) tl.push_back(make_int4(o, n, I | J << 16, (int)pslots));
    for (int K = 0; K < tb; ++K)
      rtl.push_back(make_int4(o + K * KT, std::min(KT, n - K * KT), tb,
                              (int)(pslots + (size_t)K * tb * KT)));
    pslots += (size_t)tb * tb * KT;
    if (pslots > (size_t)INT32_MAX) {
      set_error("kalman: covariance too large for the partial-slot index");
      return RC_UNSUPPORTED;
    }
  }
  d.nw = nw;
  d.dense = bsz.size() == 1;
  d.ntile = (int)tl.size();
  d.nred = (int)rtl.size();
  // one allocation: the tables first, in the order of the host block that fills
  // them with one copy, the covariance last but for the groups' buffers, which
  // a filter does without where there is no memory for them
  const bool grouped = d.dense && d.ntile >= KF_GROUP_TILES;
  std::vector<int4> items, grt;
  int rp = 0, cp = 0;
  if (grouped) group_items((nw + KT - 1) / KT, items, grt, rp, cp);
  KfLayout L;
  const size_t ost = L.take(sizeof(KfState)), obar = L.take(sizeof(KfBar)),
               octr = L.take(sizeof(unsigned)), otl = L.take(tl.size() * sizeof(int4)),
               ort = L.take(rtl.size() * sizeof(int4)), oit = L.take(items.size() * sizeof(int4)),
               ogt = L.take(grt.size() * sizeof(int4)), head = L.cur;
  const size_t opart = L.take(pslots * sizeof(double)), opj = L.take(nw * sizeof(double)),
               odp = L.take(2 * d.nred * sizeof(double)), owp = L.take(nw * sizeof(double)),
               oP = L.take((size_t)d.ntile * KTE * sizeof(double)), single = L.cur;
  const size_t vb = (size_t)nw * GM * sizeof(double);
  const size_t oU = L.take(vb), oY = L.take(vb), oJ0 = L.take(vb), oJ1 = L.take(vb),
               orp = L.take((size_t)rp * KT * GM * 8), ocp = L.take((size_t)cp * KT * GM * 8),
               ods = L.take((size_t)d.nred * 2 * GM * GM * 16), ogr = L.take(sizeof(KfGroup));
  bool room = false;
  if (grouped) {
    room = cudaMalloc(&d.base, L.cur) == cudaSuccess;
    if (!room) cudaGetLastError();
  }
  if (!room) CKK(cudaMalloc(&d.base, single));
  char *p = (char *)d.base;
  d.st = (KfState *)(p + ost);
  d.bar = (KfBar *)(p + obar);
  d.ctr = (unsigned *)(p + octr);
  d.tiles = (int4 *)(p + otl);
  d.rtl = (int4 *)(p + ort);
  d.part = (double *)(p + opart);
  d.pj = (double *)(p + opj);
  d.dotp = (double *)(p + odp);
  d.wprior = (double *)(p + owp);
  d.P = (double *)(p + oP);
  if (room) {
    d.grouped = true;
    d.nitem = (int)items.size() / 2;
    d.gitems = (int4 *)(p + oit);
    d.grt = (int4 *)(p + ogt);
    d.gU = (double *)(p + oU);
    d.gY = (double *)(p + oY);
    d.gJ[0] = (double *)(p + oJ0);
    d.gJ[1] = (double *)(p + oJ1);
    d.grpart = (double *)(p + orp);
    d.gcpart = (double *)(p + ocp);
    d.gdots = (double2 *)(p + ods);
    d.grp = p + ogr;
  }
  {
    int coop = 0, dev = 0;
    CKK(cudaGetDevice(&dev));
    CKK(cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev));
    const int per_sm = blocks_per_sm(d.dense ? (const void *)k_kf_seq<true>
                                             : (const void *)k_kf_seq<false>, 256, 0);
    d.seq_grid = coop ? std::min(grid_sms() * per_sm, std::max(d.ntile, d.nred)) : 0;
  }
  std::vector<unsigned char> tab(head, 0);  // the barrier and the counter at zero
  KfState s{};
  s.lam = lam_ini;
  s.lam0 = lam0;
  s.q = q;
  s.gate = gate;
  std::memcpy(tab.data() + ost, &s, sizeof s);
  std::memcpy(tab.data() + otl, tl.data(), tl.size() * sizeof(int4));
  std::memcpy(tab.data() + ort, rtl.data(), rtl.size() * sizeof(int4));
  if (!items.empty()) std::memcpy(tab.data() + oit, items.data(), items.size() * sizeof(int4));
  if (!grt.empty()) std::memcpy(tab.data() + ogt, grt.data(), grt.size() * sizeof(int4));
  CKK(cudaMemcpy(d.base, tab.data(), head, cudaMemcpyHostToDevice));
  LAUNCH("k_kf_init_tiles", 0, k_kf_init_tiles<<<d.ntile, 256>>>(d.tiles, d.P, p0));
  CKK(cudaGetLastError());
  CKK(cudaDeviceSynchronize());
  return RC_OK;
}

int kf_run(KfDev &d, int nobs, const double *rows, size_t ld, const double *xi,
           const double *scale, double *w, cudaStream_t s, int kbase, bool has_next,
           bool first) {
  if (nobs <= 0) return RC_OK;
  KfRowArgs ra{rows, ld, xi, scale};
  int path = g_kf_path.load();
  // a call of several observations on a larger filter: every call of a
  // sequence comes here, so each forms its own first products
  if (path < 0 && d.grouped && nobs >= KF_GROUP_OBS) {
    if (kbase == 0) CKK(cudaMemsetAsync(&d.st->status, 0, sizeof(int), s));
    return run_groups(d, nobs, ra, w, s, kbase);
  }
  // one or two observations of a grouping filter: the call before, grouped,
  // formed no products for this one
  if (path < 0 && d.grouped) {
    first = true;
    has_next = false;
  }
  // a stream being captured into a graph takes the two-launch path, whose
  // kernels are plain launches
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone)
    path = 0;
  // measured: one launch wins up to about 2K tiles (MLP 3-32-32-1 dense, 741
  // tiles, 70K against 63K updates/s; 2-128-128-1 decoupled, 2063 tiles, 46K
  // against 43K) and loses from 10K tiles on (3-64-64-1: 13K against 21K)
  if (d.seq_grid > 0 && (path == 1 || (path < 0 && d.ntile <= 8 * d.seq_grid))) {
    if (kbase == 0) CKK(cudaMemsetAsync(&d.st->status, 0, sizeof(int), s));
    int fi = first ? 1 : 0, hn = has_next ? 1 : 0, ntile = d.ntile, nw = d.nw, nred = d.nred;
    void *args[] = {&d.tiles, &ntile, &d.P, &nw, &d.rtl, &nred, &d.part, &d.pj, &d.dotp,
                    &d.st, &d.bar, &w, &ra, &nobs, &kbase, &fi, &hn};
    const void *fn = d.dense ? (const void *)k_kf_seq<true> : (const void *)k_kf_seq<false>;
    CKK(cudaMemsetAsync(d.bar, 0, sizeof(KfBar), s));  // a barrier that gave up leaves a count
    int pi = prof_begin("k_kf_seq", s);
    const cudaError_t e = cudaLaunchCooperativeKernel(fn, d.seq_grid, 256, args, 0, s);
    prof_end(pi, s);
    note_launch();
    CKK(e);
    return RC_OK;
  }
  if (kbase == 0) CKK(cudaMemsetAsync(&d.st->status, 0, sizeof(int), s));
  if (first) {  // the products with the call's first row
    LAUNCH("k_kf_tiles_pj", s,
           (d.dense ? k_kf_tiles<KM_PJ, true> : k_kf_tiles<KM_PJ, false>)<<<d.ntile, 256, 0, s>>>(
               d.tiles, d.P, d.nw, d.pj, d.st, w, w, ra, 0, d.part));
  }
  const KfIekf plain{nullptr, nullptr, 0};
  for (int k = 0; k < nobs; ++k) {
    LAUNCH("k_kf_reduce", s,
           (k_kf_reduce<<<d.nred, RED_THREADS, 0, s>>>(d.rtl, d.part, d.pj, ra, k, kbase,
                                                       plain, d.dotp, d.ctr, d.st)));
    if (k + 1 < nobs || has_next)
      LAUNCH("k_kf_tiles", s,
             (d.dense ? k_kf_tiles<KM_UPD_PJ, true> : k_kf_tiles<KM_UPD_PJ, false>)<<<
                 d.ntile, 256, 0, s>>>(d.tiles, d.P, d.nw, d.pj, d.st, w, w, ra, k + 1, d.part));
    else
      LAUNCH("k_kf_tiles", s,
             (d.dense ? k_kf_tiles<KM_UPD, true> : k_kf_tiles<KM_UPD, false>)<<<
                 d.ntile, 256, 0, s>>>(d.tiles, d.P, d.nw, d.pj, d.st, w, w, ra, 0, d.part));
  }
  CKK(cudaGetLastError());
  return RC_OK;
}

int kf_iekf(KfDev &d, const double *row, const double *resid, const double *scale, double *w,
            bool final, cudaStream_t s, int kbase, bool reset) {
  KfRowArgs ra{row, (size_t)d.nw, resid, scale};
  const KfIekf ie{d.wprior, w, final ? 1 : 0};
  if (reset) CKK(cudaMemsetAsync(&d.st->status, 0, sizeof(int), s));
  LAUNCH("k_kf_tiles_pj", s,
         (d.dense ? k_kf_tiles<KM_PJ, true> : k_kf_tiles<KM_PJ, false>)<<<d.ntile, 256, 0, s>>>(
             d.tiles, d.P, d.nw, d.pj, d.st, w, w, ra, 0, d.part));
  LAUNCH("k_kf_reduce", s,
         (k_kf_reduce<<<d.nred, RED_THREADS, 0, s>>>(d.rtl, d.part, d.pj, ra, 0, kbase, ie,
                                                     d.dotp, d.ctr, d.st)));
  if (final)
    LAUNCH("k_kf_tiles", s,
           (d.dense ? k_kf_tiles<KM_UPD, true> : k_kf_tiles<KM_UPD, false>)<<<d.ntile, 256, 0,
                                                                              s>>>(
               d.tiles, d.P, d.nw, d.pj, d.st, w, d.wprior, ra, 0, d.part));
  else
    LAUNCH("k_kf_wonly", s,
           (k_kf_wonly<<<(d.nw + 255) / 256, 256, 0, s>>>(d.nw, w, d.wprior, d.pj, d.st)));
  CKK(cudaGetLastError());
  return RC_OK;
}

// xi = -R for one point from its output derivatives out[na][nout] (the
// first component) and a residual rule, in the order of the host's
// residual (R = sum_k c_k T_k, or c_k T_0 T_k for a nonlinear term)
__global__ void k_kf_resid(DevRule r, const double *__restrict__ out, int nout,
                           double *__restrict__ xi, double sign) {
  if (threadIdx.x != 0) return;
  double R = 0.0;
  for (int k = 0; k < r.nterm; ++k)
    R = r.nonlin[k] ? R + r.coeff[k] * out[0] * out[(size_t)r.ind[k] * nout]
                    : R + r.coeff[k] * out[(size_t)r.ind[k] * nout];
  *xi = sign * R;
}

int kf_resid_xi(const DevRule &r, const double *out, int nout, double *xi, cudaStream_t s,
                double sign) {
  LAUNCH("k_kf_resid", s, (k_kf_resid<<<1, 32, 0, s>>>(r, out, nout, xi, sign)));
  CKK(cudaGetLastError());
  return RC_OK;
}

// One observation of a system (the trainer's loop over sys_nres,
// app/sgd_batch_module.f90:497-545): from one point's output derivatives
// out[na][nout], residual ir of a system rule (calc_sys_residual,
// app/pinn_module.f90:86-125) as xi = sign * R_ir, and its seed dR_ir/dT
// in seed[nout][na] (set_sys_seed :127-162 with a one in slot ir, fac 1,
// unweighted).
__global__ void k_kf_sys_seed(DevRule r, const double *__restrict__ out, int na, int nout,
                              const double *__restrict__ src, int ir,
                              double *__restrict__ seed, double *__restrict__ xi, double sign) {
  for (int i = threadIdx.x; i < nout * na; i += blockDim.x) seed[i] = 0.0;
  __syncthreads();
  if (threadIdx.x != 0) return;
  auto T = [&](int f) {  // factor f: (component, slot), 0-based
    return out[(size_t)r.sfac[2 * f + 1] * nout + r.sfac[2 * f]];
  };
  double R = src ? -src[ir] : 0.0;
  for (int k = 0; k < r.nterm; ++k) {
    if (r.sys[3 * k] != ir) continue;
    const int nf = r.sys[3 * k + 1], f0 = r.sys[3 * k + 2];
    double prod = r.coeff[k];
    for (int m = 0; m < nf; ++m) prod = prod * T(f0 + m);
    R = R + prod;
    for (int m = 0; m < nf; ++m) {
      double other = r.coeff[k];
      for (int mm = 0; mm < nf; ++mm)
        if (mm != m) other = other * T(f0 + mm);
      const int at = r.sfac[2 * (f0 + m)] * na + r.sfac[2 * (f0 + m) + 1];
      seed[at] = seed[at] + other;
    }
  }
  *xi = sign * R;
}

int kf_sys_seed(const DevRule &r, const double *out, int na, int nout, const double *src,
                int ir, double *seed, double *xi, double sign, cudaStream_t s) {
  LAUNCH("k_kf_sys_seed", s,
         (k_kf_sys_seed<<<1, 256, 0, s>>>(r, out, na, nout, src, ir, seed, xi, sign)));
  CKK(cudaGetLastError());
  return RC_OK;
}

int kf_state(const KfDev &d, KfState *out, cudaStream_t s) {
  CKK(cudaMemcpyAsync(out, d.st, sizeof(KfState), cudaMemcpyDeviceToHost, s));
  CKK(cudaStreamSynchronize(s));
  return RC_OK;
}

int kf_read_cov(const KfDev &d, const std::vector<int> &bsz, const std::vector<int> &boff,
                bool dense, double *out, cudaStream_t s) {
  std::vector<double> h((size_t)d.ntile * KTE);
  std::vector<int4> tl(d.ntile);
  CKK(cudaMemcpyAsync(h.data(), d.P, h.size() * sizeof(double), cudaMemcpyDeviceToHost, s));
  CKK(cudaMemcpyAsync(tl.data(), d.tiles, tl.size() * sizeof(int4), cudaMemcpyDeviceToHost, s));
  CKK(cudaStreamSynchronize(s));
  // output offset of each block: dense [nw][nw]; decoupled blocks one after another
  std::vector<size_t> bout(bsz.size(), 0);
  for (size_t b = 1; b < bsz.size(); ++b) bout[b] = bout[b - 1] + (size_t)bsz[b - 1] * bsz[b - 1];
  size_t b = 0;
  for (int i = 0; i < d.ntile; ++i) {
    const int4 t = tl[i];
    while (boff[b] != t.x) ++b;
    const int n = t.y;
    for (int r = 0; r < KT; ++r)
      for (int c = 0; c < KT; ++c) {
        const int R = (t.z & 0xffff) * KT + r, C = (t.z >> 16) * KT + c;
        if (R >= n || C >= n) continue;
        const double v = h[(size_t)i * KTE + r * KT + c];
        if (dense) {
          out[(size_t)(t.x + R) * d.nw + t.x + C] = v;
          out[(size_t)(t.x + C) * d.nw + t.x + R] = v;
        } else {
          out[bout[b] + (size_t)R * n + C] = v;
          out[bout[b] + (size_t)C * n + R] = v;
        }
      }
  }
  return RC_OK;
}

}  // namespace dnnf90
