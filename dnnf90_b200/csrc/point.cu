// point.cu - the whole derivative-carrying step of a small network in one
// launch: one block per point runs the forward, the seed and the adjoint
// (lib/train_module.f90:241-489) with every plane in shared memory.
//
// A batch of few points, or one point, spends the layer-by-layer path in
// launches of nearly empty grids (ten to thirteen, each a chain of its own
// latencies, 4 to 70 us), and a filter pass pays that per point.  Here the
// layers follow one another between block barriers.  FP64 only (the split
// path's layer GEMMs are tensor-core kernels); it serves the batches for
// which point_applies() says so.
//
// Inside a block: layer products on the FP64 tensor cores (m8n8k4, 8 x 8 tiles
// dealt to the warps), the Bell step as the Horner form of tile_plan.hpp with
// eight lanes per (slot, eight neurons) and the pair lists of bell_col.hpp
// read through L1, the first layer from its monomials (see k_adj_l2a),
// gradients summed over the block's points in shared memory and added once
// per block.  A hidden layer keeps T and one more plane, in which S and then
// h follow each other, so that two blocks of 512 threads share an SM for most
// sets; a batch of no more points than SMs runs 1024 threads a point.
// Bound: barriers and dependent shared-memory loads, about 1 us a stage (a
// level of the Horner form, a product) at one point; shared-memory issue of
// the pair lists at several.  A training step, layer by layer -> here:
//   heat closure, 3-32-32-1, one point          59 -> 18 us
//   D0 = 4, K = 7, 4-8-8-1, one point          221 -> 61 us, 296 points 311 -> 94
//   D0 = 4, K = 3, 4-32-32-1, 600 points       139 -> 74 us
#include <cuda_runtime.h>

#include <algorithm>
#include <string>

#include "bell.hpp"
#include "engine.hpp"
#include "kernels.cuh"
#include "point.hpp"
#include "scratch.hpp"

namespace dnnf90 {

#define CKP(x)                                                     \
  do {                                                             \
    cudaError_t e_ = (x);                                          \
    if (e_ != cudaSuccess) {                                       \
      set_error(std::string("point: ") + cudaGetErrorString(e_));  \
      return RC_DEVICE;                                            \
    }                                                              \
  } while (0)

namespace {

constexpr int PT_LAYERS = 8;     // layers of a network here
constexpr int PT_RB = 4;       // items a warp holds between two barriers of q = 0
constexpr int PT_SMEM = 226 * 1024;

// Row stride (doubles) of a [slot][n] plane: a multiple of 4, and not of 16,
// so that the eight rows of a DMMA fragment start on different banks.
__host__ __device__ inline int ldp(int n) {
  const int v = (n + 3) / 4 * 4;
  return v % 16 ? v : v + 4;
}

struct PointArgs {
  int nl, na, d0, k, iact, npts, nout, nw;
  int dims[PT_LAYERS], woff[PT_LAYERS];   // per layer; offset of the layer's weights
  int ds[KMAX + 2];
  // shared-memory offsets (doubles): weights, gradient, powers of the first
  // layer's weights, s^(q) of the first and of the current layer, T and S (h
  // once formed) of each hidden layer, the two Horner buffers, out and seed
  int o_w, o_g, o_pw, o_sig, o_sg, o_t[PT_LAYERS], o_s[PT_LAYERS], o_m, o_a, o_b, o_out, o_seed;
  int train;
  const double *W, *X, *tpc, *sc, *src, *seeds;
  const int2 *fhdr, *ahdr;
  const uint32_t *frec, *arec, *ex;
  const short *dn;
  double *out, *grad, *rows, *loss, *xi;
  double xi_sign;
  int kind, nterm, nres;
  double fac;
  const double *coeff, *wres;
  const int *ind, *nonlin, *sys, *sfac;
};

// (row, column) of the elements t, t + NTH, ... of rows of n
template <int NTH>
struct RowCol {
  int r, j, n, dr, dj;
  __device__ RowCol(int n_) : r(threadIdx.x / n_), j(threadIdx.x % n_), n(n_), dr(NTH / n_), dj(NTH % n_) {}
  __device__ void next() {
    r += dr;
    j += dj;
    if (j >= n) {
      j -= n;
      ++r;
    }
  }
};

// Bell work of one layer, dealt to the warps in items of four units of eight
// lanes: a unit is eight neurons of one slot, or with parts (lgp) one half or
// quarter of its list
struct Units {
  int n, tiles, lgp, lane;
  unsigned magic;
  int r, j, part;
  bool act;
  __device__ Units(int n_, int lgp_)
      : n(n_), tiles((n_ + 7) / 8), lgp(lgp_), lane(threadIdx.x & 31) {
    magic = tiles > 1 ? 0xffffffffu / (unsigned)tiles + 1 : 0;
  }
  __device__ int items(int rows) const { return (((rows * tiles) << lgp) + 3) >> 2; }
  // this lane's slot, neuron and part of an item; idle lanes repeat entry 0
  __device__ void at(int item, int rows) {
    const int gi = item * 4 + (lane >> 3), unit = gi >> lgp;
    part = gi & ((1 << lgp) - 1);
    r = tiles > 1 ? (int)__umulhi((unsigned)unit, magic) : unit;
    j = (unit - r * tiles) * 8 + (lane & 7);
    act = r < rows && j < n;
    if (!act) r = j = 0;
  }
  __device__ double sum(double v) const {
    if (lgp > 0) v += __shfl_xor_sync(0xffffffffu, v, 8);
    if (lgp > 1) v += __shfl_xor_sync(0xffffffffu, v, 16);
    return v;
  }
};

// sum_b s~_b (D, E)_{q+1, a-b} of one unit's slot
__device__ __forceinline__ double2 horner(const Units &u, const int2 *hdr, const uint32_t *recs,
                                          const double *S, const double2 *Dr, int ls) {
  const int2 hd = __ldg(hdr + u.r);
  const uint32_t *rec = recs + hd.x;
  const double *sj = S + u.j;
  const double2 *dj = Dr + u.j;
  double2 c0 = make_double2(0.0, 0.0), c1 = c0;
  int i = 0;
#pragma unroll 2
  for (; i + 1 < hd.y; i += 2) {
    const uint2 w = __ldg((const uint2 *)(rec + i));
    const double s0 = sj[(w.x & 0xffffu) * ls], s1 = sj[(w.y & 0xffffu) * ls];
    const double2 e0 = dj[(w.x >> 16) * u.n], e1 = dj[(w.y >> 16) * u.n];
    c0.x = fma(s0, e0.x, c0.x);
    c0.y = fma(s0, e0.y, c0.y);
    c1.x = fma(s1, e1.x, c1.x);
    c1.y = fma(s1, e1.y, c1.y);
  }
  if (i < hd.y) {
    const uint32_t w = __ldg(rec + i);
    const double s0 = sj[(w & 0xffffu) * ls];
    const double2 e0 = dj[(w >> 16) * u.n];
    c0.x = fma(s0, e0.x, c0.x);
    c0.y = fma(s0, e0.y, c0.y);
  }
  return make_double2(c0.x + c1.x, c0.y + c1.y);
}

__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(d[0]), "+d"(d[1])
      : "d"(a), "d"(b));
}

// S[a][j] = (sum_i T[a][i] W[j][1 + i] (+ W[j][0] at a = 0)) / a!, 8 x 8 tiles
// dealt to the warps; rows and columns past the end repeat the last
template <int NTH>
__device__ __forceinline__ void prod_fwd(const double *T, const double *W, const double *ifact,
                                         double *S, int na, int n, int m) {
  const int lane = threadIdx.x & 31, r8 = lane >> 2, c4 = lane & 3, lt = ldp(m), ls = ldp(n);
  const int tn = (n + 7) / 8, tiles = (na + 7) / 8 * tn;
  for (int e = threadIdx.x >> 5; e < tiles; e += NTH / 32) {
    const int a0 = e / tn * 8, j0 = e % tn * 8;
    const double *t = T + min(a0 + r8, na - 1) * lt, *w = W + min(j0 + r8, n - 1) * (m + 1) + 1;
    double acc[2] = {0.0, 0.0};
#pragma unroll 4
    for (int k0 = 0; k0 < m; k0 += 4) {
      const int k = k0 + c4, kc = min(k, m - 1);
      const double tv = t[kc], wv = w[kc];
      dmma(acc, k < m ? tv : 0.0, k < m ? wv : 0.0);
    }
    const int r = a0 + r8;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int j = j0 + 2 * c4 + u;
      if (r < na && j < n) {
        double v = acc[u];
        if (r == 0) v += W[j * (m + 1)];
        S[r * ls + j] = v * __ldg(ifact + r);
      }
    }
  }
}

// Tb[a][i] = a! sum_j Sb[a][j] W[j][1 + i]
template <int NTH>
__device__ __forceinline__ void prod_dt(const double *Sb, const double *W, const double *fact,
                                        double *Tb, int na, int n, int m) {
  const int lane = threadIdx.x & 31, r8 = lane >> 2, c4 = lane & 3, lt = ldp(m), ls = ldp(n);
  const int tm = (m + 7) / 8, tiles = (na + 7) / 8 * tm;
  for (int e = threadIdx.x >> 5; e < tiles; e += NTH / 32) {
    const int a0 = e / tm * 8, i0 = e % tm * 8;
    const double *s = Sb + min(a0 + r8, na - 1) * ls, *w = W + min(i0 + r8, m - 1) + 1;
    double acc[2] = {0.0, 0.0};
#pragma unroll 4
    for (int k0 = 0; k0 < n; k0 += 4) {
      const int k = k0 + c4, kc = min(k, n - 1);
      const double sv = s[kc], wv = w[kc * (m + 1)];
      dmma(acc, k < n ? sv : 0.0, k < n ? wv : 0.0);
    }
    const int r = a0 + r8;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = i0 + 2 * c4 + u;
      if (r < na && i < m) Tb[r * lt + i] = acc[u] * __ldg(fact + r);
    }
  }
}

// G[j][0] += Sb[0][j], G[j][1 + i] += sum_a Sb[a][j] T[a][i].  With fewer
// tiles than warps the slots are split over the warps of a tile.
template <int NTH>
__device__ __forceinline__ void prod_dw(const double *Sb, const double *T, double *G, int na,
                                        int n, int m) {
  const int lane = threadIdx.x & 31, r8 = lane >> 2, c4 = lane & 3, lt = ldp(m), ls = ldp(n);
  const int tm = (m + 7) / 8, tiles = (n + 7) / 8 * tm, steps = (na + 3) / 4;
  const int parts = max(1, min(NTH / 32 / tiles, (steps + 3) / 4));
  for (int e = threadIdx.x >> 5; e < tiles * parts; e += NTH / 32) {
    const int p = e / tiles, q = e - p * tiles, j0 = q / tm * 8, i0 = q % tm * 8;
    const int s0 = steps * p / parts, s1 = steps * (p + 1) / parts;
    const double *s = Sb + min(j0 + r8, n - 1), *t = T + min(i0 + r8, m - 1);
    double acc[2] = {0.0, 0.0};
#pragma unroll 4
    for (int k0 = s0; k0 < s1; ++k0) {
      const int k = 4 * k0 + c4, kc = min(k, na - 1);
      const double sv = s[kc * ls], tv = t[kc * lt];
      dmma(acc, k < na ? sv : 0.0, k < na ? tv : 0.0);
    }
    const int j = j0 + r8;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const int i = i0 + 2 * c4 + u;
      if (j < n && i < m) {
        double *d = G + j * (m + 1) + 1 + i;
        if (parts > 1) atomicAdd(d, acc[u]);
        else *d += acc[u];
      }
    }
  }
  for (int j = threadIdx.x; j < n; j += NTH) G[j * (m + 1)] += Sb[j];
}

// s^(q) of n neurons from S_0 into sig[q][n]; tanh: one thread per (q, neuron)
template <int NTH>
__device__ __forceinline__ void sigmas(const PointArgs &a, const double *S0, double *sig, int n) {
  if (a.iact == 0) {
    for (int e = threadIdx.x; e < (a.k + 2) * n; e += NTH) {
      const int q = e / n, j = e - q * n;
      const double t = tanh(S0[j]);
      const double *row = a.tpc + q * (a.k + 3);
      double v = __ldg(row + q + 1);
      for (int i = q; i >= 0; --i) v = v * t + __ldg(row + i);
      sig[e] = v;
    }
  } else {
    for (int j = threadIdx.x; j < n; j += NTH) {
      double d[KMAX + 2];
      sigma_derivs(a.iact, a.tpc, a.k, S0[j], d);
      for (int q = 0; q <= a.k + 1; ++q) sig[q * n + j] = d[q];
    }
  }
}

// the rule's seed and loss from the output derivatives tl[nout][na] (one
// thread; the formulas of k_output_fwdv)
__device__ double point_seed(const PointArgs &a, const double *tl, double *sd, int pt) {
  const int na = a.na;
  for (int i = 0; i < a.nout * na; ++i) sd[i] = 0.0;
  if (a.kind == SEED_SYS) {
    double R[SYS_MAXRES];
    for (int r = 0; r < a.nres; ++r) R[r] = a.src ? -a.src[(size_t)pt * a.nres + r] : 0.0;
    for (int k = 0; k < a.nterm; ++k) {
      const int r = a.sys[3 * k], nf = a.sys[3 * k + 1], f0 = a.sys[3 * k + 2];
      double prod = a.coeff[k];
      for (int m = 0; m < nf; ++m)
        prod = prod * tl[a.sfac[2 * (f0 + m)] * na + a.sfac[2 * (f0 + m) + 1]];
      R[r] = R[r] + prod;
    }
    double l = 0.0;
    for (int r = 0; r < a.nres; ++r) l += a.wres[r] * R[r] * R[r];
    for (int k = 0; k < a.nterm; ++k) {
      const int r = a.sys[3 * k], nf = a.sys[3 * k + 1], f0 = a.sys[3 * k + 2];
      for (int m = 0; m < nf; ++m) {
        double other = a.fac * a.wres[r] * R[r] * a.coeff[k];
        for (int mm = 0; mm < nf; ++mm)
          if (mm != m) other = other * tl[a.sfac[2 * (f0 + mm)] * na + a.sfac[2 * (f0 + mm) + 1]];
        const int at = a.sfac[2 * (f0 + m)] * na + a.sfac[2 * (f0 + m) + 1];
        sd[at] = sd[at] + other;
      }
    }
    return 0.5 * a.fac * l;
  }
  double R0 = 0.0;
  for (int t = 0; t < a.nterm; ++t) {
    const int ind = a.ind[t];
    if (a.nonlin[t]) R0 = R0 + a.coeff[t] * tl[0] * tl[ind];
    else R0 = R0 + a.coeff[t] * tl[ind];
  }
  double Rs = R0, fac = a.fac, l = 0.0;
  if (a.xi) *a.xi = a.xi_sign * R0;  // one point's residual (see k_kf_resid)
  if (a.kind == SEED_JROW) { Rs = 1.0; fac = 1.0; }
  else l = 0.5 * a.fac * R0 * R0;
  for (int t = 0; t < a.nterm; ++t) {
    const int ind = a.ind[t];
    if (a.nonlin[t]) {
      sd[ind] = sd[ind] + fac * Rs * a.coeff[t] * tl[0];
      sd[0] = sd[0] + fac * Rs * a.coeff[t] * tl[ind];
    } else {
      sd[ind] = sd[ind] + fac * Rs * a.coeff[t];
    }
  }
  return l;
}

template <int NTH>
__global__ void __launch_bounds__(NTH, 1024 / NTH) k_point(PointArgs a) {
  extern __shared__ __align__(16) double sh[];
  __shared__ double s_loss;
  constexpr int NW = NTH / 32;
  const int t = threadIdx.x, warp = t >> 5, na = a.na, d0 = a.d0, K = a.k;
  const int H = a.nl - 2;  // hidden layers
  double *W = sh + a.o_w, *G = sh + a.o_g, *pw = sh + a.o_pw, *sig1 = sh + a.o_sig,
         *sg = sh + a.o_sg, *out = sh + a.o_out, *seed = sh + a.o_seed, *A = sh + a.o_a,
         *B = sh + a.o_b;
  const double *fact = a.sc, *ifact = a.sc + na;
  const int n1 = a.dims[1], l1 = ldp(n1);
  for (int i = t; i < a.nw; i += NTH) {
    W[i] = a.W[i];
    if (a.grad) G[i] = 0.0;
  }
  if (t == 0) s_loss = 0.0;
  __syncthreads();
  // pw[i][p][j] = W[j][i]^p / p!: a slot's monomial W^a / a! is a product of
  // d0 of them
  const double *W1 = W + a.woff[1];
  for (int e = t; e < d0 * n1; e += NTH) {
    const int i = e / n1, j = e - i * n1;
    const double w = W1[j * (d0 + 1) + 1 + i];
    double v = 1.0;
    for (int p = 0; p <= K; ++p) {
      pw[(i * (K + 1) + p) * n1 + j] = v;
      v = v * w / (double)(p + 1);
    }
  }
  auto mono = [&](int r, int j, int &deg) {
    const uint32_t ex = __ldg(a.ex + r);
    double v = 1.0;
    deg = 0;
    for (int i = 0; i < d0; ++i) {
      const int p = (ex >> (4 * i)) & 15;
      deg += p;
      v *= pw[(i * (K + 1) + p) * n1 + j];
    }
    return v;
  };
  for (int pt = blockIdx.x; pt < a.npts; pt += gridDim.x) {
    const double *x = a.X + (size_t)pt * d0;
    __syncthreads();
    // ---------------- first hidden layer: T_a = s^(|a|)(S_0) W^a
    for (int j = t; j < n1; j += NTH) {
      double s = W1[j * (d0 + 1)];
      for (int i = 0; i < d0; ++i) s = s + W1[j * (d0 + 1) + 1 + i] * __ldg(x + i);
      A[j] = s;
    }
    __syncthreads();
    sigmas<NTH>(a, A, sig1, n1);
    __syncthreads();
    {
      double *T = sh + a.o_t[1];
      for (RowCol<NTH> e(n1); e.r < na; e.next()) {
        int deg;
        const double m = mono(e.r, e.j, deg);
        T[e.r * l1 + e.j] = __ldg(fact + e.r) * m * sig1[deg * n1 + e.j];
      }
    }
    __syncthreads();
    // ---------------- hidden layers: product, then D_q, E_q (Horner)
    for (int l = 2; l <= H; ++l) {
      const int n = a.dims[l], ls = ldp(n);
      double *S = sh + a.o_s[l], *T = sh + a.o_t[l];
      prod_fwd<NTH>(sh + a.o_t[l - 1], W + a.woff[l], ifact, S, na, n, a.dims[l - 1]);
      __syncthreads();
      sigmas<NTH>(a, S, sg, n);  // row 0 holds S_0
      __syncthreads();
      {
        double2 *top = (double2 *)(K & 1 ? A : B);
        for (int j = t; j < n; j += NTH)
          top[j] = make_double2(sg[K * n + j], sg[(K + 1) * n + j]);
      }
      __syncthreads();
      Units u(n, 0);
      for (int q = K - 1; q >= 0; --q) {
        const double inv = 1.0 / (double)(q + 1);
        const double2 *Dr = (const double2 *)(q & 1 ? B : A);
        double2 *Dw = (double2 *)(q & 1 ? A : B);
        const int rows = a.ds[K - q + 1];  // slots of degree <= K - q
        const int items = u.items(rows);
        if (q > 0 || !a.train) {
          for (int e = warp; e < items; e += NW) {
            u.at(e, rows);
            double2 v = horner(u, a.fhdr, a.frec, S, Dr, ls);
            v = u.r == 0 ? make_double2(sg[q * n + u.j], sg[(q + 1) * n + u.j])
                         : make_double2(v.x * inv, v.y * inv);
            if (u.act) {
              if (q > 0) Dw[u.r * n + u.j] = v;
              else T[u.r * ls + u.j] = __ldg(fact + u.r) * v.x;
            }
          }
        } else {
          // q = 0 goes down the slots, PT_RB items of every warp at a time: an
          // output reads S of its own and lower slots only, so behind a
          // barrier h_a / a!, as the adjoint reads it, may take S's place
          constexpr int RND = NW * PT_RB;
          for (int base = (items - 1) / RND * RND; base >= 0; base -= RND) {
            double h[PT_RB];
            int to[PT_RB];
#pragma unroll
            for (int x = 0; x < PT_RB; ++x) {
              const int e = base + x * NW + warp;
              to[x] = -1;
              if (e >= items) continue;
              u.at(e, rows);
              double2 v = horner(u, a.fhdr, a.frec, S, Dr, ls);
              v = u.r == 0 ? make_double2(sg[u.j], sg[n + u.j]) : v;
              if (u.act) {
                to[x] = u.r * ls + u.j;
                T[to[x]] = __ldg(fact + u.r) * v.x;
              }
              h[x] = v.y;
            }
            __syncthreads();
#pragma unroll
            for (int x = 0; x < PT_RB; ++x)
              if (to[x] >= 0) S[to[x]] = h[x];
          }
        }
        __syncthreads();
      }
    }
    // ---------------- output layer: eight lanes per slot
    const int m = a.dims[H], lm = ldp(m);
    const double *WL = W + a.woff[H + 1], *TL = sh + a.o_t[H];
    for (int s = t >> 3; s < (a.nout * na + 3) / 4 * 4; s += NTH / 8) {
      const int sc = min(s, a.nout * na - 1), o = sc / na, r = sc - o * na;
      double v = 0.0;
      for (int i = t & 7; i < m; i += 8) v = fma(TL[r * lm + i], WL[o * (m + 1) + 1 + i], v);
      v += __shfl_xor_sync(0xffffffffu, v, 4);
      v += __shfl_xor_sync(0xffffffffu, v, 2);
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      if ((t & 7) == 0 && s < a.nout * na) {
        if (r == 0) v += WL[o * (m + 1)];
        out[s] = v;
        if (a.out) a.out[((size_t)pt * na + r) * a.nout + o] = v;
      }
    }
    if (!a.train) continue;
    __syncthreads();
    if (a.kind == SEED_GIVEN) {
      for (int s = t; s < a.nout * na; s += NTH) seed[s] = a.seeds[(size_t)pt * a.nout * na + s];
    } else if (a.kind == SEED_HALFSQ) {
      for (int s = t; s < a.nout * na; s += NTH) seed[s] = s < na ? out[s] : 0.0;
      if (t < 32) {
        double l = 0.0;
        for (int r = t; r < na; r += 32) l += out[r] * out[r];
        l = warp_sum(l);
        if (t == 0) s_loss += 0.5 * l;
      }
    } else if (t == 0) {
      s_loss += point_seed(a, out, seed, pt);
    }
    // a point's row of the Jacobian collects in G as a batch's gradient does
    if (a.rows)
      for (int i = t; i < a.nw; i += NTH) G[i] = 0.0;
    __syncthreads();
    // ---------------- adjoint: dW of the read-out, then a! Tb takes T's place
    const bool g = a.grad || a.rows;
    if (g) {
      double *gl = G + a.woff[H + 1];
      const int items = a.nout * m, parts = max(1, min(NTH / items, (na + 7) / 8));
      for (int e = t; e < items * parts; e += NTH) {
        const int p = e / items, q = e - p * items, o = q / m, i = q - o * m;
        const int a0 = na * p / parts, a1 = na * (p + 1) / parts;
        double v = 0.0;
        for (int r = a0; r < a1; ++r) v = fma(seed[o * na + r], TL[r * lm + i], v);
        double *d = gl + o * (m + 1) + 1 + i;
        if (parts > 1) atomicAdd(d, v);
        else *d += v;
      }
      for (int o = t; o < a.nout; o += NTH) gl[o * (m + 1)] += seed[o * na];
      __syncthreads();
    }
    double *Tb = B, *Sb = A;
    for (RowCol<NTH> e(m); e.r < na; e.next()) {
      double v = 0.0;
      for (int o = 0; o < a.nout; ++o) v = fma(WL[o * (m + 1) + 1 + e.j], seed[o * na + e.r], v);
      Tb[e.r * lm + e.j] = v * __ldg(fact + e.r);
    }
    __syncthreads();
    for (int l = H; l >= 2; --l) {
      const int n = a.dims[l], mm = a.dims[l - 1], ls = ldp(n);
      // Sb_b = (1 / b!) sum_g (a! Tb_a)(h_g / g!), a = b + g
      const double *h = sh + a.o_s[l];
      auto corr = [&](const Units &u) {
        int2 hd = __ldg(a.ahdr + u.r);
        if (!u.act) hd.y = 0;  // slot 0 has the longest list
        const uint32_t *rec = a.arec + hd.x;
        const double *tj = Tb + u.j, *hj = h + u.j;
        double c0 = 0.0, c1 = 0.0;
        int i = 2 * u.part;
        const int step = 2 << u.lgp;
#pragma unroll 2
        for (; i + 1 < hd.y; i += step) {
          const uint2 w = __ldg((const uint2 *)(rec + i));
          c0 = fma(tj[(w.x & 0xffffu) * ls], hj[(w.x >> 16) * ls], c0);
          c1 = fma(tj[(w.y & 0xffffu) * ls], hj[(w.y >> 16) * ls], c1);
        }
        if (i < hd.y) {
          const uint32_t w = __ldg(rec + i);
          c0 = fma(tj[(w & 0xffffu) * ls], hj[(w >> 16) * ls], c0);
        }
        return c0 + c1;
      };
      // the lists of the degrees 0 and 1 are the longest (|A| and its share
      // above e_i): four parts each, by the last warps, the rest from the first
      Units u(n, 2);
      const int low = a.ds[2];
      for (int e = NW - 1 - warp, items = u.items(low); e < items; e += NW) {
        u.at(e, low);
        const double v = u.sum(corr(u));
        if (u.act && u.part == 0) Sb[u.r * ls + u.j] = v * __ldg(ifact + u.r);
      }
      u.lgp = 0;
      for (int e = warp, items = u.items(na - low); e < items; e += NW) {
        u.at(e, na - low);
        u.r += u.act ? low : 0;
        const double v = corr(u);
        if (u.act) Sb[u.r * ls + u.j] = v * __ldg(ifact + u.r);
      }
      __syncthreads();
      if (g) prod_dw<NTH>(Sb, sh + a.o_t[l - 1], G + a.woff[l], na, n, mm);
      prod_dt<NTH>(Sb, W + a.woff[l], fact, Tb, na, n, mm);
      __syncthreads();
    }
    // ---------------- first layer (h^g = s^(|g|+1) W^g, see k_adj_l2a): with
    // c_a = a! Tb_a, Sb^0 = sum c_a s^(|a|+1) W^a / a! goes to the bias and,
    // times x, to the weights; e_i's share is sum c_a s^(|a|) W^(a-e_i) / (a-e_i)!
    if (g) {
      double *g1 = G + a.woff[1], *M = sh + a.o_m;
      for (RowCol<NTH> e(n1); e.r < na; e.next()) {
        int deg;
        M[e.r * l1 + e.j] = mono(e.r, e.j, deg);
      }
      __syncthreads();
      const int items = n1 * (d0 + 1), parts = max(1, min(NTH / items, (na + 3) / 4));
      for (int e = t; e < items * parts; e += NTH) {
        const int p = e / items, q = e - p * items, o = q / n1, j = q - o * n1;
        const int a0 = na * p / parts, a1 = na * (p + 1) / parts;
        double v = 0.0;
        int deg = 0;
        for (int r = a0; r < a1; ++r) {
          while (r >= a.ds[deg + 1]) ++deg;
          const int from = o == 0 ? r : __ldg(a.dn + r * d0 + o - 1);
          if (from < 0) continue;  // a_i = 0
          v = fma(Tb[r * l1 + j] * M[from * l1 + j], sig1[(deg + (o == 0)) * n1 + j], v);
        }
        double *gj = g1 + j * (d0 + 1);
        atomicAdd(gj + o, v);
        if (o == 0)
          for (int i = 0; i < d0; ++i) atomicAdd(gj + 1 + i, v * __ldg(x + i));
      }
    }
    if (a.rows) {
      double *row = a.rows + (size_t)pt * a.nw;
      __syncthreads();
      for (int i = t; i < a.nw; i += NTH) row[i] = G[i];
    }
  }
  __syncthreads();
  if (a.grad)
    for (int i = t; i < a.nw; i += NTH) atomicAdd(a.grad + i, G[i]);
  if (a.loss && t == 0) atomicAdd(a.loss, s_loss);
}

// shared-memory layout; returns the bytes
size_t layout(const DevTables &t, const DevNet &net, bool train, PointArgs &a) {
  const int na = t.na, L = net.nlayer, H = L - 2, n1 = net.dims[1], nout = net.dims[L - 1];
  long cur = 0;
  auto take = [&](long n) {
    const long at = cur;
    cur += (n + 1) / 2 * 2;
    return (int)std::min(at, (long)PT_SMEM);
  };
  int nmax = 0;
  for (int l = 1; l <= H; ++l) nmax = std::max(nmax, net.dims[l]);
  const long plane = (long)na * ldp(nmax);
  a.o_w = take(net.nw);
  a.o_g = take(train ? net.nw : 0);
  a.o_pw = take((long)t.d0 * (t.k + 1) * n1);
  a.o_sig = take((long)(t.k + 2) * n1);
  a.o_sg = take((long)(t.k + 2) * nmax);
  // T of the last hidden layer takes the buffer of the even D_q, which q = 0
  // does not read, and a! Tb follows it there; Sb takes the odd ones'
  const long odd = 2L * t.dstart[t.k] * nmax;                       // degree <= K - 1
  const long even = t.k >= 2 ? 2L * t.dstart[t.k - 1] * nmax : 2L * nmax;  // <= K - 2
  a.o_a = take(std::max(odd, train ? plane : (long)n1));
  a.o_b = take(std::max(even, plane));
  for (int l = 1; l < H; ++l) a.o_t[l] = take((long)na * ldp(net.dims[l]));
  a.o_t[H] = a.o_b;
  // the first layer's monomials, formed again for its gradient, take T_1's
  // place, or that of the odd D_q where T_1's holds a! Tb
  a.o_m = H > 1 ? a.o_t[1] : a.o_a;
  for (int l = 2; l <= H; ++l)
    a.o_s[l] = train || l == 2 ? take((long)na * ldp(train ? net.dims[l] : nmax)) : a.o_s[2];
  a.o_out = take((long)nout * na);
  a.o_seed = take(train ? (long)nout * na : 0);
  return (size_t)cur * sizeof(double);
}

// blocks of 512 threads an SM holds (0 after an error)
int point_blocks(size_t smem) {
  if (cudaFuncSetAttribute(k_point<512>, cudaFuncAttributeMaxDynamicSharedMemorySize, PT_SMEM))
    return 0;
  return blocks_per_sm((const void *)k_point<512>, 512, smem);
}

}  // namespace

bool point_set(const TableSet &t) {
  // the slots' exponents are packed four bits each
  if (t.d0 > 8 || t.k < 1 || t.k > 14 || t.na > 512) return false;
  for (int a = 1; a < t.na; ++a)
    if (t.deg[a] < t.deg[a - 1]) return false;
  return true;
}

void upload_point(const TableSet &t, const ColProg &p, PointDev &d, PlanBlock &b) {
  d = PointDev();
  const SlotIndex at(t);
  std::vector<uint32_t> ex(t.na, 0);
  for (int a = 0; a < t.na; ++a)
    for (int i = 0; i < t.d0; ++i) ex[a] |= (uint32_t)t.alpha[(size_t)a * t.d0 + i] << (4 * i);
  std::vector<short> dn((size_t)t.na * t.d0, -1);  // slot of a - e_i
  std::vector<int> al(t.d0);
  for (int a = 0; a < t.na; ++a)
    for (int i = 0; i < t.d0; ++i) {
      al.assign(t.alpha.begin() + (size_t)a * t.d0, t.alpha.begin() + (size_t)(a + 1) * t.d0);
      if (al[i]-- > 0) dn[(size_t)a * t.d0 + i] = (short)at.find(al.data());
    }
  b.add((int **)&d.fhdr, p.fhdr);
  b.add((int **)&d.ahdr, p.ahdr);
  b.add(&d.frec, p.frec);
  b.add(&d.arec, p.arec);
  b.add(&d.ex, ex);
  b.add(&d.dn, dn);
  d.ok = true;
}

// The rule: the plain path, a network whose planes fit shared memory, and up
// to 16 points per SM.  The layer-by-layer kernels cost 55 to 230 us at one
// point and little more at a few hundred; here the time goes up with each
// round of resident blocks.  Training steps, layer by layer against one
// launch, at the last count served and past it (148 SMs):
//   two blocks an SM, |A| <= 36 (the column kernels serve the other side):
//     8 points per SM: D0 = 4, K = 3, 32 wide 180 / 126 us, heat closure, 32
//     wide 103 / 65; at 16: 258 / 237 and 120 / 110, heat 8 wide 86 / 104
//   two blocks an SM, larger sets: 16 points per SM: D0 = 4, K = 4, 16 wide
//     328 / 253 us, K = 5 494 / 404; at 64: 1068 / 987, evaluation 415 / 426
//   one block an SM: 3 points per SM: D0 = 4, K = 5, 32 wide 248 / 178 us;
//     at 4: 293 / 286 and D0 = 4, K = 3, 64 wide 193 / 197
//   one hidden layer (no Bell step to save): 3 points per SM: heat closure,
//     16 wide 30 / 24 us; at 8: 35 / 38
bool point_applies(const DevTables &t, const DevNet &net, const DevRule &rule, int npts,
                   bool train, int prec) {
  const int L = net.nlayer, H = L - 2;
  const PointDev &d = t.bp.point;
  if (prec != PREC_F64 || !d.ok || !t.graded || H < 1 || L > PT_LAYERS || net.dims[L - 1] > 4 ||
      (int)t.dstart.size() < t.k + 2 || tune_pinned() || (train && rule.kind < 0))
    return false;
  PointArgs a;
  const size_t smem = layout(t, net, train, a);
  if (smem > PT_SMEM) return false;
  if (npts <= 3L * grid_sms()) return true;
  const int per = point_blocks(smem);
  return H > 1 && per >= 2 && npts <= (t.na > 36 ? 16L : 8L) * grid_sms();
}

int run_point(const DevTables &t, const DevNet &net, const DevRule &rule, const BatchArgs &b,
              cudaStream_t st) {
  PointArgs a{};
  const int L = net.nlayer;
  const size_t smem = layout(t, net, b.train, a);
  const PointDev &d = t.bp.point;
  a.nl = L; a.na = t.na; a.d0 = t.d0; a.k = t.k; a.iact = t.iact; a.npts = b.npts;
  a.nout = net.dims[L - 1]; a.nw = net.nw; a.train = b.train;
  for (int l = 0; l < L; ++l) {
    a.dims[l] = net.dims[l];
    a.woff[l] = l ? (int)net.woff[l] : 0;
  }
  for (int p = 0; p < KMAX + 2; ++p) a.ds[p] = p <= t.k + 1 ? t.dstart[p] : t.na;
  a.W = net.w64; a.X = b.X; a.tpc = t.tpc; a.sc = t.bp.sc64; a.src = b.src; a.seeds = b.seeds;
  a.fhdr = d.fhdr; a.ahdr = d.ahdr; a.frec = d.frec; a.arec = d.arec; a.ex = d.ex; a.dn = d.dn;
  a.out = b.out;
  if (b.train) {
    a.kind = rule.kind;
    a.rows = rule.kind == SEED_JROW ? b.rows : nullptr;
    a.grad = a.rows ? nullptr : b.grad;
    a.loss = rule.kind == SEED_GIVEN || rule.kind == SEED_JROW ? nullptr : b.loss;
    a.xi = b.xi; a.xi_sign = b.xi_sign;
    a.nterm = rule.nterm; a.nres = rule.nres; a.fac = rule.fac; a.coeff = rule.coeff;
    a.wres = rule.wres; a.ind = rule.ind; a.nonlin = rule.nonlin; a.sys = rule.sys;
    a.sfac = rule.sfac;
  }
  if (b.npts <= grid_sms()) {
    CKP(cudaFuncSetAttribute(k_point<1024>, cudaFuncAttributeMaxDynamicSharedMemorySize, PT_SMEM));
    LAUNCH("k_point", st, (k_point<1024><<<b.npts, 1024, smem, st>>>(a)));
  } else {
    const int grid = std::min(b.npts, grid_sms() * std::max(1, point_blocks(smem)));
    LAUNCH("k_point", st, (k_point<512><<<grid, 512, smem, st>>>(a)));
  }
  CKP(cudaGetLastError());
  return RC_OK;
}

}  // namespace dnnf90
