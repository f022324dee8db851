// bell_col.cu - Bell kernels with one thread per (point, neuron).
//
// Column kernels (small carried sets).  A set of a few tens of slots has too
// little work per neuron to share between warps: the block-per-point kernels
// of bell.cu spend such items in barriers (one per degree) and idle warps.
// Here every thread owns one neuron of one point and keeps its slots in its
// own column of shared memory ([slot][thread], so that a warp's access is
// one conflict-free row); no thread reads another's column, so the items
// need no barrier at all.  The pair lists are warp-uniform broadcasts.
// Forward: the Horner form of the Bell sum over factorial-normalised series
// (see tile_plan.hpp), with D and E side by side and updated in place: an
// output only reads slots of lower degree, so the slots are taken in
// descending order of degree.  Every sum is one chain that starts with the
// pair (a, 0), and the adjoint's sums keep the chains of the block-per-point
// kernels: up to K = 2 both then round exactly as those do (a natural-gradient step divides by a small damping what the
// rounding of its rows leaves).
//
// First-layer adjoint (every graded set).  The first hidden layer is
// analytic, h^g = s^(|g|+1)(S^0) W^g, so its adjoint needs the Tb plane once
// and per neuron tile a table of monomials.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <unordered_map>

#include "bell.hpp"
#include "bell_col.hpp"
#include "engine.hpp"
#include "kernels.cuh"
#include "scratch.hpp"

namespace dnnf90 {

#define CKC(x)                                                        \
  do {                                                                \
    cudaError_t e_ = (x);                                             \
    if (e_ != cudaSuccess) {                                          \
      set_error(std::string("bell_col: ") + cudaGetErrorString(e_));  \
      return e_ == cudaErrorMemoryAllocation ? RC_NOMEM : RC_DEVICE;  \
    }                                                                 \
  } while (0)

// ------------------------------------------------------------ the program
ColProg build_col_prog(const TableSet &t) {
  ColProg P;
  const int na = t.na, d0 = t.d0;
  for (int a = 0; a < na; ++a) P.kt = std::max(P.kt, t.deg[a]);
  // a multi-index as one word, four bits a component (K <= 15, D0 <= 16): no
  // component of a - b borrows from the next when b <= a
  std::unordered_map<uint64_t, int> at;
  std::vector<uint64_t> key(na, 0);
  at.reserve(2 * na);
  for (int a = 0; a < na; ++a) {
    for (int i = 0; i < d0; ++i) key[a] |= (uint64_t)t.alpha[(size_t)a * d0 + i] << (4 * i);
    at[key[a]] = a;
  }
  std::vector<std::vector<uint32_t>> f(na), adj(na);
  for (int a = 0; a < na; ++a)
    for (int b = 0; b < na; ++b) {
      bool le = t.deg[b] <= t.deg[a];
      const int *x = &t.alpha[(size_t)a * d0], *y = &t.alpha[(size_t)b * d0];
      for (int i = 0; le && i < d0; ++i) le = y[i] <= x[i];
      if (!le) continue;
      const int ig = at.at(key[a] - key[b]);  // the set is downward closed
      if (b != 0 && b == a) f[a].insert(f[a].begin(), (uint32_t)b);
      else if (b != 0) f[a].push_back((uint32_t)b | ((uint32_t)ig << 16));
      adj[b].push_back((uint32_t)a | ((uint32_t)ig << 16));
    }
  auto flat = [&](const std::vector<std::vector<uint32_t>> &v, std::vector<int> &hdr,
                  std::vector<uint32_t> &rec) {
    for (int a = 0; a < na; ++a) {
      if (rec.size() & 1) rec.push_back(0);
      hdr.push_back((int)rec.size());
      hdr.push_back((int)v[a].size());
      rec.insert(rec.end(), v[a].begin(), v[a].end());
    }
    if (rec.size() & 1) rec.push_back(0);
  };
  flat(f, P.fhdr, P.frec);
  flat(adj, P.ahdr, P.arec);
  P.dstart.assign(P.kt + 2, na);
  for (int a = na - 1; a >= 0; --a) P.dstart[t.deg[a]] = a;
  for (int p = P.kt; p >= 0; --p) P.dstart[p] = std::min(P.dstart[p], P.dstart[p + 1]);
  return P;
}

namespace {

constexpr int NT = 64;        // threads per block of the column kernels

template <typename R> struct Vec2;
template <> struct Vec2<float> { typedef float2 T; };
template <> struct Vec2<double> { typedef double2 T; };

struct ColArgs {
  int n, na, npts, k, kt, iact, nrec, gstride;
  const int *hdr;
  const uint32_t *rec;
  const int *dstart;
  const double *sc;        // [3][na]: a!, 1/a!, 1/a!
  const double *tpc;
  const void *A, *B;       // forward: S; adjoint: Tb, h
  void *C, *D;             // forward: T, h; adjoint: Sb
  double *gbias;
};

size_t col_tables(int na, int nrec, size_t rsz) {
  return (size_t)na * 8 + (size_t)nrec * 4 + (KMAX + 3) * 4 + 2 * (size_t)na * rsz + 64;
}
// columns: s~ and the (D, E) pairs (forward) or Tb and h (adjoint), the
// s^(q) rows
size_t col_fwd_smem(int na, int kt, int nrec, size_t rsz) {
  return (size_t)(3 * na + kt + 2) * NT * rsz + col_tables(na, nrec, rsz);
}
size_t col_adj_smem(int na, int nrec, size_t rsz) {
  return (size_t)2 * na * NT * rsz + col_tables(na, nrec, rsz);
}

// shared copies of the tables; the pointers are set by the caller's layout
template <typename R>
struct ColTab {
  int2 *hdr;
  uint32_t *rec;
  R *fact, *ifact;
  int *ds;
  __device__ void load(unsigned char *p, const ColArgs &a) {
    // records first: they are read as 8-byte pairs
    rec = (uint32_t *)p;
    hdr = (int2 *)(rec + (a.nrec + 1) / 2 * 2);
    fact = (R *)(hdr + a.na);
    ifact = fact + a.na;
    ds = (int *)(ifact + a.na);
    for (int i = threadIdx.x; i < a.nrec; i += NT) rec[i] = __ldg(a.rec + i);
    for (int i = threadIdx.x; i < a.na; i += NT) {
      hdr[i] = make_int2(__ldg(a.hdr + 2 * i), __ldg(a.hdr + 2 * i + 1));
      fact[i] = (R)__ldg(a.sc + i);
      ifact[i] = (R)__ldg(a.sc + a.na + i);
    }
    for (int i = threadIdx.x; i < a.kt + 2; i += NT) ds[i] = __ldg(a.dstart + i);
  }
};

__device__ __forceinline__ float2 madd2(float s, float2 d, float2 acc) {
  return __ffma2_rn(make_float2(s, s), d, acc);
}
__device__ __forceinline__ double2 madd2(double s, double2 d, double2 acc) {
  return make_double2(fma(s, d.x, acc.x), fma(s, d.y, acc.y));
}

// Bound: the loads and stores of the planes while the set is small (5 slots,
// 16384 points x 64 in FP64: 1020 us in the block-per-point kernels, 53 here,
// 126 MB at 2.4 TB/s), the shared-memory loads of the pairs beyond about 15
// slots.  NT = 64: small blocks, so that as many columns as fit are resident.
template <typename R, bool TRAIN>
__global__ void __launch_bounds__(NT) k_bell_fwd_col(ColArgs a) {
  typedef typename Vec2<R>::T R2;
  extern __shared__ __align__(16) unsigned char smc[];
  const int n = a.n, na = a.na, kt = a.kt;
  R2 *de = (R2 *)smc + threadIdx.x;                       // [na]
  R *s = (R *)((R2 *)smc + (size_t)na * NT) + threadIdx.x;  // [na]
  R *sig = s + (size_t)na * NT;                           // [kt + 2]
  ColTab<R> t;
  t.load((unsigned char *)((R *)((R2 *)smc + (size_t)na * NT) + (size_t)(na + kt + 2) * NT), a);
  __syncthreads();
  const long total = (long)a.npts * n, stride = (long)gridDim.x * NT;
  const size_t plane = (size_t)na * n;
  for (long e = (long)blockIdx.x * NT + threadIdx.x; e < total; e += stride) {
    const long pt = e / n;
    const size_t base = (size_t)pt * plane + (size_t)(e - pt * n);
    const R *S = (const R *)a.A + base;
    R s0 = S[0];
#pragma unroll 4
    for (int i = 1; i < na; ++i) s[i * NT] = S[(size_t)i * n] * t.ifact[i];
    if (a.iact == 0) {
      const double th = tanh((double)s0);
      const int ld = a.k + 3;
      for (int q = 0; q <= kt + 1; ++q) {
        double v = __ldg(a.tpc + q * ld + q + 1);
        for (int i = q; i >= 0; --i) v = v * th + __ldg(a.tpc + q * ld + i);
        sig[q * NT] = (R)v;
      }
    } else {
      double d[KMAX + 2];
      sigma_derivs(a.iact, a.tpc, a.k, (double)s0, d);
      for (int q = 0; q <= kt + 1; ++q) sig[q * NT] = (R)d[q];
    }
    R *T = (R *)a.C + base, *H = (R *)a.D + base;
    R2 top;
    top.x = sig[kt * NT];
    top.y = sig[(kt + 1) * NT];
    de[0] = top;
    for (int q = kt - 1; q >= 0; --q) {
      const R inv = (R)1 / (R)(q + 1);
      for (int i = t.ds[kt - q + 1] - 1; i >= 1; --i) {
        const int2 h = t.hdr[i];
        R2 acc;
        acc.x = acc.y = (R)0;
        const uint32_t *r = t.rec + h.x;
        int c = 0;
        for (; c + 1 < h.y; c += 2) {
          const uint2 u = *(const uint2 *)(r + c);
          acc = madd2(s[(u.x & 0xffffu) * NT], de[(u.x >> 16) * NT], acc);
          acc = madd2(s[(u.y & 0xffffu) * NT], de[(u.y >> 16) * NT], acc);
        }
        if (c < h.y) {
          const uint32_t u = r[c];
          acc = madd2(s[(u & 0xffffu) * NT], de[(u >> 16) * NT], acc);
        }
        acc.x *= inv;
        acc.y *= inv;
        if (q > 0) {
          de[i * NT] = acc;
        } else {
          T[(size_t)i * n] = t.fact[i] * acc.x;
          if (TRAIN) H[(size_t)i * n] = t.fact[i] * acc.y;
        }
      }
      if (q > 0) {
        R2 o;
        o.x = sig[q * NT];
        o.y = sig[(q + 1) * NT];
        de[0] = o;
      }
    }
    T[0] = sig[0];
    if (TRAIN) H[0] = sig[NT];
  }
}

// Sb_b b! = sum_g (a! Tb_a)(h_g / g!), a = b + g.  The threads stride over
// the (point, neuron) pairs by a multiple of n, so a thread's neuron is
// fixed and its share of the bias gradient stays in a register.  (5 slots,
// 16384 points x 64 in FP64: 550 us before, 40 here.)
template <typename R, int CHAINS>
__global__ void __launch_bounds__(NT) k_bell_adj_col(ColArgs a) {
  extern __shared__ __align__(16) unsigned char smc[];
  __shared__ double red[NT];
  const int n = a.n, na = a.na;
  R *tb = (R *)smc + threadIdx.x, *hh = tb + (size_t)na * NT;
  ColTab<R> t;
  t.load((unsigned char *)((R *)smc + (size_t)2 * na * NT), a);
  __syncthreads();
  const long total = (long)a.npts * n;
  const long stride = (long)gridDim.x * NT / n * n;
  const size_t plane = (size_t)na * n;
  const long e0 = (long)blockIdx.x * NT + threadIdx.x;
  double gb = 0.0;
  for (long e = e0 < stride ? e0 : total; e < total; e += stride) {
    const long pt = e / n;
    const size_t base = (size_t)pt * plane + (size_t)(e - pt * n);
    const R *Tb = (const R *)a.A + base, *H = (const R *)a.B + base;
#pragma unroll 4
    for (int i = 0; i < na; ++i) {
      tb[i * NT] = Tb[(size_t)i * n] * t.fact[i];
      hh[i * NT] = H[(size_t)i * n] * t.ifact[i];
    }
    R *Sb = (R *)a.C + base;
    for (int i = na - 1; i >= 0; --i) {
      const int2 h = t.hdr[i];
      const uint32_t *r = t.rec + h.x;
      R acc = (R)0, bcc = (R)0;
      int c = 0;
      for (; c + 1 < h.y; c += 2) {
        const uint2 u = *(const uint2 *)(r + c);
        acc = fma(tb[(u.x & 0xffffu) * NT], hh[(u.x >> 16) * NT], acc);
        R &second = CHAINS == 2 ? bcc : acc;
        second = fma(tb[(u.y & 0xffffu) * NT], hh[(u.y >> 16) * NT], second);
      }
      if (c < h.y) {
        const uint32_t u = r[c];
        acc = fma(tb[(u & 0xffffu) * NT], hh[(u >> 16) * NT], acc);
      }
      const R v = (CHAINS == 2 ? acc + bcc : acc) * t.ifact[i];
      Sb[(size_t)i * n] = v;
      if (i == 0) gb += (double)v;
    }
  }
  if (!a.gbias) return;
  red[threadIdx.x] = gb;
  __syncthreads();
  // threads n apart share a neuron
  if (threadIdx.x < n) {
    double v = 0.0;
    for (int i = threadIdx.x; i < NT; i += n) v += red[i];
    if (v != 0.0) atomicAdd(a.gbias + (size_t)(e0 % n) * a.gstride, v);
  }
}

int resident_grid(const void *k, int threads, size_t smem) {
  return grid_sms() * blocks_per_sm(k, threads, smem);
}

// ------------------------------------------------------------ first layer
struct L2aArgs {
  int n, na, npts, k, nt, ppw, zsplit;
  int chain;               // groups of slots to a run (k_adj_l2a)
  const int *up;           // [na][D0]: slot of g + e_i | (g_i + 1) << 16, or -1
  const int *par;          // [na]: slot of a - e_i | i << 16, i the first nonzero dimension
  const double *sc;        // [3][na]: a!, 1/a!, 1/a!
  const void *Tb, *sig;    // [P][na][n], [P][k + 2][n]
  const double *X, *W;     // [P][D0], [n][D0 + 1]
  double *g, *rows;
  size_t nw, woff;
  int ds[KMAX + 2];
};

constexpr int L2T = 256;   // threads per block

// bytes of k_adj_l2a's tables
__host__ __device__ inline size_t l2a_tables(int na, int nt, int d0, size_t msz) {
  return ((size_t)(na + 1) * nt + na + 3) * msz + (size_t)na * d0 * 4 + 16;
}

// a block's dW_2 sums, one set acc per thread: over the warps, then over the
// lanes that share a neuron, then one atomic per weight
template <int D0, int NTHR>
__device__ __forceinline__ void l2_reduce(const L2aArgs &a, double *red, const double (&acc)[D0 + 1],
                                          bool act, int j0) {
  __syncthreads();  // the tables are done with; red: [D0 + 1][NTHR]
#pragma unroll
  for (int o = 0; o <= D0; ++o) red[o * NTHR + threadIdx.x] = act ? acc[o] : 0.0;
  __syncthreads();
  for (int e = threadIdx.x; e < a.nt * (D0 + 1); e += NTHR) {
    const int o = e / a.nt, l = e - o * a.nt;
    if (j0 + l >= a.n) continue;
    double v = 0.0;
    for (int w = 0; w < NTHR / 32; ++w)
      for (int u = 0; u < a.ppw; ++u) v += red[o * NTHR + w * 32 + u * a.nt + l];
    if (v != 0.0) atomicAdd(a.g + (size_t)(j0 + l) * (D0 + 1) + o, v);
  }
}

// One point's dW_2 sums over the slots a0 .. a1 - 1, one product at a time and
// none for a slot without a_i, added to r.
template <typename R, typename MT, int D0>
__device__ __forceinline__ void l2a_plain(const L2aArgs &a, const MT *fact, const MT *Ml,
                                          const int *off, int j, long pt, int a0, int a1,
                                          double (&r)[D0 + 1]) {
  const R *Tb = (const R *)a.Tb + (size_t)pt * a.na * a.n + j;
  const R *sg = (const R *)a.sig + (size_t)pt * (a.k + 2) * a.n + j;
  double v = 0.0;
#pragma unroll 1
  for (int p = 0; p <= a.k; ++p)
#pragma unroll 1
    for (int q = max(a.ds[p], a0); q < min(a.ds[p + 1], a1); ++q) {
      const double x = (double)Tb[(size_t)q * a.n] * (double)fact[q];
      v += (double)sg[(size_t)(p + 1) * a.n] * (x * (double)Ml[q * a.nt]);
#pragma unroll
      for (int i = 0; i < D0; ++i) {
        const int o = off[q * D0 + i];
        if (o != a.na * a.nt) r[1 + i] += (double)sg[(size_t)p * a.n] * (x * (double)Ml[o]);
      }
    }
  r[0] += v;
#pragma unroll
  for (int i = 0; i < D0; ++i) r[1 + i] = fma(v, __ldg(a.X + (size_t)pt * D0 + i), r[1 + i]);
}
template <int N>
__device__ __forceinline__ bool any_odd(const double (&v)[N]) {  // not finite
  bool odd = false;
#pragma unroll
  for (int o = 0; o < N; ++o) odd |= !(fabs(v[o]) <= 1.7976931348623157e308);
  return odd;
}

// Sb^0 = sum_a Tb^a h^a and Sb^{e_i} = sum_a a_i Tb^a h^{a - e_i} with
// h^g = s^(|g|+1) W^g.  With M_a = W^a / a! and x_a = a! Tb^a both read
// x_a M_a and x_a M_{a - e_i}, and s depends on the degree alone, so each
// degree is summed first:
//   Sb^0 = sum_p s^(p+1) sum_{|a| = p} x_a M_a,
//   Sb^{e_i} = sum_p s^(p) sum_{|a| = p} x_a M_{a - e_i}.
// One lane per neuron of a tile (lanes beyond a narrow layer's neurons take
// further points) and PT points at a time per thread: the tile's M rows sit
// in shared memory and one read of a row serves PT points, and the slots go
// in groups of G whose values are loaded a group ahead, so the kernel streams
// Tb (32768 points x 128 at K = 7, D0 = 4 in FP32: 5.5 GB in 1.35 ms, 4.1
// TB/s; in FP64, 16384 points, 5.5 GB in 1.16).
// Precision: the degrees, the points and the blocks are added in FP64.  On
// the split path a degree is summed in FP32 runs of at most a.chain groups
// (BT = float), or in FP64 throughout (BT = MT = double) where a run would be
// shorter than a group: never longer than the |A| / 32 slots that one of
// k_adj_l2s's 32 warps sums, see l2a_k.
// Gradient mode sums over a thread's points and may split the slots over
// blockIdx.z (dW_2 is linear in each slot's share) when there are few
// points; row mode writes each point's sums, a warp's own (L2_ROWS) or, when
// there are few points, those of a block's eight warps, which share the
// slots of the same points (L2_ROWS8).
// A slot without a_i multiplies a row of zeros for e_i.  Where a value of Tb is
// not finite, neither are the sums, and the thread forms them again without
// those products, which are NaN (l2a_plain; behind the loop and from a fresh
// thread index, so that the loop keeps its registers: in the loop it cost a
// third of its speed).
enum L2Mode { L2_GRAD, L2_ROWS, L2_ROWS8 };
template <typename R, typename BT, typename MT, int D0, int PT, L2Mode MODE>
__global__ void __launch_bounds__(L2T, 2) k_adj_l2a(L2aArgs a) {
  constexpr int G = D0 == 1 ? 1 : 4;            // one slot a degree in one dimension
  extern __shared__ __align__(16) unsigned char sm2[];
  const int na = a.na, n = a.n, nt = a.nt;
  MT *fact = (MT *)sm2;                         // [na]
  MT *M = fact + (na + (na & 1));               // [na + 1][nt], row na zero
  int *off = (int *)(M + ((size_t)(na + 1) * nt + 1) / 2 * 2);  // [na][D0]: word offset of row a - e_i
  const int j0 = blockIdx.y * nt;
  for (int e = threadIdx.x; e < na * D0; e += L2T) off[e] = na * nt;
  for (int e = threadIdx.x; e < na; e += L2T) fact[e] = (MT)__ldg(a.sc + e);
  for (int e = threadIdx.x; e < nt; e += L2T) {
    M[e] = (MT)1;
    M[(size_t)na * nt + e] = (MT)0;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < na * D0; e += L2T) {
    const int g = e / D0, i = e - g * D0, u = __ldg(a.up + e);
    if (u >= 0) off[(u & 0xffff) * D0 + i] = g * nt;
  }
  for (int p = 1; p <= a.k; ++p) {
    const int r0 = a.ds[p], nr = a.ds[p + 1] - r0;
    for (int e = threadIdx.x; e < nr * nt; e += L2T) {
      const int r = r0 + e / nt, jl = e % nt, j = min(j0 + jl, n - 1);
      const int pk = __ldg(a.par + r), ps = pk & 0xffff, i = pk >> 16;
      // the exponent of dimension i: a! over (a - e_i)!
      const double f = __ldg(a.sc + ps) * __ldg(a.sc + na + r);
      M[(size_t)r * nt + jl] =
          (MT)((double)M[(size_t)ps * nt + jl] * (__ldg(a.W + (size_t)j * (D0 + 1) + 1 + i) * f));
    }
    __syncthreads();
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int jl = lane % nt, sub = lane / nt;
  const bool act = sub < a.ppw && j0 + jl < n;
  const int j = min(j0 + jl, n - 1);
  const MT *Ml = M + jl;
  // the slots of this block, or of this warp
  constexpr int NWP = L2T / 32;
  const int part = MODE == L2_ROWS8 ? warp : (int)blockIdx.z;
  const int nparts = MODE == L2_ROWS8 ? NWP : a.zsplit;
  const int a0 = (int)((long)na * part / nparts), a1 = (int)((long)na * (part + 1) / nparts);
  constexpr int NACC = MODE == L2_GRAD ? 1 : PT;  // sums over points, or each point's
  double acc[NACC][D0 + 1];
#pragma unroll
  for (int k = 0; k < NACC; ++k)
#pragma unroll
    for (int o = 0; o <= D0; ++o) acc[k][o] = 0.0;
  const long nwarp = MODE == L2_ROWS8 ? (long)gridDim.x : (long)gridDim.x * NWP;
  const long w0 = MODE == L2_ROWS8 ? (long)blockIdx.x : (long)blockIdx.x * NWP + warp;
  const int step = a.ppw;
  bool odd = false;  // a row that is not finite
  for (long w = w0; w * step * PT < a.npts; w += nwarp) {
    if (MODE != L2_ROWS8 && !act) continue;  // with shared slots every thread meets the barriers
    const R *Tb[PT], *sg[PT];
    bool on[PT];
    double v0[PT];
#pragma unroll
    for (int k = 0; k < PT; ++k) {
      const long pt = (w * PT + k) * step + sub;
      on[k] = pt < a.npts;
      const long q = on[k] ? pt : (long)a.npts - 1;  // read twice, times zero
      Tb[k] = (const R *)a.Tb + (size_t)q * na * n + j;
      sg[k] = (const R *)a.sig + (size_t)q * (a.k + 2) * n + j;
      v0[k] = 0.0;
    }
    if (MODE != L2_GRAD) {
#pragma unroll
      for (int k = 0; k < NACC; ++k)
#pragma unroll
        for (int o = 0; o <= D0; ++o) acc[k][o] = 0.0;
    }
    R xn[G][PT];  // the next G slots' values
    auto load = [&](int r) {
#pragma unroll
      for (int u = 0; u < G; ++u)
#pragma unroll
        for (int k = 0; k < PT; ++k)
          xn[u][k] = r + u < a1 ? __ldcs(Tb[k] + (size_t)(r + u) * n) : (R)0;
    };
    load(a0);
    for (int p = 0; p <= a.k; ++p) {
      const int r0 = max(a.ds[p], a0), r1 = min(a.ds[p + 1], a1);
      if (r0 >= r1) continue;
      R s1[PT], sp[PT];
#pragma unroll
      for (int k = 0; k < PT; ++k) {
        s1[k] = on[k] ? sg[k][(size_t)(p + 1) * n] : (R)0;
        sp[k] = on[k] ? sg[k][(size_t)p * n] : (R)0;
      }
      BT b[PT][D0 + 1];
#pragma unroll
      for (int k = 0; k < PT; ++k)
#pragma unroll
        for (int o = 0; o <= D0; ++o) b[k][o] = (BT)0;
      int left = a.chain;
      for (int q = r0; q < r1; q += G) {
        BT x[G][PT];
#pragma unroll
        for (int u = 0; u < G; ++u)
#pragma unroll
          for (int k = 0; k < PT; ++k) x[u][k] = (BT)xn[u][k];
        load(min(q + G, r1));
#pragma unroll
        for (int u = 0; u < G; ++u) {
          const int r = q + u;
          if (r >= r1) break;
          const BT f = (BT)fact[r], m0 = (BT)Ml[r * nt];
#pragma unroll
          for (int k = 0; k < PT; ++k) {
            x[u][k] *= f;
            b[k][0] = fma(x[u][k], m0, b[k][0]);
          }
#pragma unroll
          for (int i = 0; i < D0; ++i) {
            const BT m = (BT)Ml[off[r * D0 + i]];
#pragma unroll
            for (int k = 0; k < PT; ++k) b[k][1 + i] = fma(x[u][k], m, b[k][1 + i]);
          }
        }
        if (--left && q + G < r1) continue;
        left = a.chain;
#pragma unroll
        for (int k = 0; k < PT; ++k) {
          v0[k] = fma((double)s1[k], (double)b[k][0], v0[k]);
          b[k][0] = (BT)0;
#pragma unroll
          for (int i = 0; i < D0; ++i) {
            double &s = acc[MODE == L2_GRAD ? 0 : k][1 + i];
            s = fma((double)sp[k], (double)b[k][1 + i], s);
            b[k][1 + i] = (BT)0;
          }
        }
      }
    }
#pragma unroll
    for (int k = 0; k < PT; ++k) {
      if (!on[k]) continue;
      const long pt = (w * PT + k) * step + sub;
      const double *x = a.X + (size_t)pt * D0;
      double(&s)[D0 + 1] = acc[MODE == L2_GRAD ? 0 : k];
      s[0] += v0[k];
#pragma unroll
      for (int i = 0; i < D0; ++i) s[1 + i] = fma(v0[k], __ldg(x + i), s[1 + i]);
      if (MODE != L2_GRAD) odd |= any_odd(s);
      if (MODE == L2_ROWS) {
        double *row = a.rows + (size_t)pt * a.nw + a.woff + (size_t)j * (D0 + 1);
#pragma unroll
        for (int o = 0; o <= D0; ++o) row[o] = s[o];
      }
    }
    if (MODE == L2_ROWS8) {
      // [value][warp][lane], the warps added in order
      double *red = (double *)(sm2 + (l2a_tables(na, nt, D0, sizeof(MT)) + 15) / 16 * 16);
      __syncthreads();  // the last points' sums are written
#pragma unroll
      for (int k = 0; k < PT; ++k)
#pragma unroll
        for (int o = 0; o <= D0; ++o)
          red[((size_t)(k * (D0 + 1) + o) * NWP + warp) * 32 + lane] = acc[k][o];
      __syncthreads();
      for (int e = warp; e < PT * (D0 + 1); e += NWP) {
        const int k = e / (D0 + 1), o = e - k * (D0 + 1);
        const long pt = (w * PT + k) * step + sub;
        if (!act || pt >= a.npts) continue;
        double v = 0.0;
#pragma unroll
        for (int u = 0; u < NWP; ++u) v += red[((size_t)e * NWP + u) * 32 + lane];
        a.rows[(size_t)pt * a.nw + a.woff + (size_t)j * (D0 + 1) + o] = v;
      }
    }
  }
  if (MODE == L2_GRAD) odd = any_odd(acc[0]);
  if (MODE == L2_ROWS8) odd = __syncthreads_or(odd);
  if (odd) {
    int tid;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(tid));
    const int ln = tid & 31, wp = tid >> 5, jl2 = ln % a.nt, sub2 = ln / a.nt;
    const int j2 = blockIdx.y * a.nt + jl2;
    double r[D0 + 1];
#pragma unroll
    for (int o = 0; o <= D0; ++o) r[o] = 0.0;
    const bool mine = sub2 < a.ppw && j2 < a.n && (MODE != L2_ROWS8 || wp == 0);
    const long first = MODE == L2_ROWS8 ? (long)blockIdx.x : (long)blockIdx.x * NWP + wp;
    const long nw = MODE == L2_ROWS8 ? (long)gridDim.x : (long)gridDim.x * NWP;
    const int b0 = MODE == L2_GRAD ? (int)((long)a.na * blockIdx.z / a.zsplit) : 0;
    const int b1 = MODE == L2_GRAD ? (int)((long)a.na * (blockIdx.z + 1) / a.zsplit) : a.na;
#pragma unroll 1
    for (long w = first; mine && w * a.ppw * PT < a.npts; w += nw)
#pragma unroll 1
      for (int k = 0; k < PT; ++k) {
        const long pt = (w * PT + k) * a.ppw + sub2;
        if (pt >= a.npts) break;
        l2a_plain<R, MT, D0>(a, fact, M + jl2, off, j2, pt, b0, b1, r);
        if (MODE == L2_GRAD) continue;
        double *row = a.rows + (size_t)pt * a.nw + a.woff + (size_t)j2 * (D0 + 1);
        double old[D0 + 1];
#pragma unroll
        for (int o = 0; o <= D0; ++o) old[o] = row[o];
        const bool again = any_odd(old);
#pragma unroll
        for (int o = 0; o <= D0; ++o) {
          if (again) row[o] = r[o];
          r[o] = 0.0;
        }
      }
    if (MODE == L2_GRAD)
#pragma unroll
      for (int o = 0; o <= D0; ++o) acc[0][o] = r[o];
  }
  if (MODE == L2_GRAD && a.g) l2_reduce<D0, L2T>(a, (double *)sm2, acc[0], act, j0);
}

// The first-layer adjoint of a small set in the order of k_adj_l2s: slot g's
// products are formed as (g_i + 1) Tb^{g + e_i} h^g, h^g = s^(|g|+1) W^g, and
// summed over g = w, w + 32, ...; the sums of the 32 w are added in R in row
// mode and in FP64 (with the sums over the points) in gradient mode, so that
// a row or a gradient rounds as it does there.  Tb and h of a thread's
// (point, neuron) sit in its own columns of shared memory.  Bound: the rows
// written, or Tb read.
constexpr int L2RT = 128;
template <typename R, int D0>
__global__ void __launch_bounds__(L2RT) k_adj_l2r(L2aArgs a) {
  extern __shared__ __align__(16) unsigned char sm2[];
  const int na = a.na, n = a.n, nt = a.nt, j0 = blockIdx.y * nt;
  R *tb = (R *)sm2 + threadIdx.x, *hh = tb + (size_t)na * L2RT;
  R *M = (R *)sm2 + (size_t)2 * na * L2RT;      // [na][nt]
  int *up = (int *)(M + ((size_t)na * nt + 1) / 2 * 2);  // [na][D0]
  for (int e = threadIdx.x; e < na * D0; e += L2RT) up[e] = __ldg(a.up + e);
  for (int e = threadIdx.x; e < nt; e += L2RT) M[e] = (R)1;
  __syncthreads();
  for (int p = 1; p <= a.k; ++p) {
    const int r0 = a.ds[p], nr = a.ds[p + 1] - r0;
    for (int e = threadIdx.x; e < nr * nt; e += L2RT) {
      const int r = r0 + e / nt, jl = e % nt, j = min(j0 + jl, n - 1), pk = __ldg(a.par + r);
      M[(size_t)r * nt + jl] = (R)((double)M[(size_t)(pk & 0xffff) * nt + jl] *
                                   __ldg(a.W + (size_t)j * (D0 + 1) + 1 + (pk >> 16)));
    }
    __syncthreads();
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int jl = lane % nt, sub = lane / nt, j = j0 + jl;
  const bool act = sub < a.ppw && j < n;
  double acc[D0 + 1];
#pragma unroll
  for (int o = 0; o <= D0; ++o) acc[o] = 0.0;
  const long nwarp = (long)gridDim.x * (L2RT / 32);
  for (long w0 = (long)blockIdx.x * (L2RT / 32) + warp; w0 * a.ppw < a.npts; w0 += nwarp) {
    const long pt = w0 * a.ppw + sub;
    if (!act || pt >= a.npts) continue;
    const double *x = a.X + (size_t)pt * D0;
    const R *Tb = (const R *)a.Tb + (size_t)pt * na * n + j;
    const R *sg = (const R *)a.sig + (size_t)pt * (a.k + 2) * n + j;
    for (int p = 0; p <= a.k; ++p) {
      if (a.ds[p] >= a.ds[p + 1]) continue;
      const R dq = sg[(size_t)(p + 1) * n];
      for (int g = a.ds[p]; g < a.ds[p + 1]; ++g) {
        tb[g * L2RT] = __ldcs(Tb + (size_t)g * n);
        hh[g * L2RT] = dq * M[(size_t)g * nt + jl];
      }
    }
    R v[D0 + 1];
#pragma unroll
    for (int o = 0; o <= D0; ++o) v[o] = (R)0;
    for (int w = 0; w < min(32, na); ++w) {
      R s[D0 + 1];
#pragma unroll
      for (int o = 0; o <= D0; ++o) s[o] = (R)0;
      for (int g = w; g < na; g += 32) {
        const R hg = hh[g * L2RT];
        s[0] += tb[g * L2RT] * hg;
#pragma unroll
        for (int i = 0; i < D0; ++i) {
          const int u = up[g * D0 + i];
          if (u >= 0) s[1 + i] += (R)(u >> 16) * tb[(u & 0xffff) * L2RT] * hg;
        }
      }
      if (a.rows) {
#pragma unroll
        for (int o = 0; o <= D0; ++o) v[o] += s[o];
      } else {
        acc[0] += (double)s[0];
#pragma unroll
        for (int i = 0; i < D0; ++i) acc[1 + i] += (double)s[0] * __ldg(x + i) + (double)s[1 + i];
      }
    }
    if (!a.rows) continue;
    double *row = a.rows + (size_t)pt * a.nw + a.woff + (size_t)j * (D0 + 1);
    row[0] = (double)v[0];
#pragma unroll
    for (int i = 0; i < D0; ++i) row[1 + i] = (double)v[0] * __ldg(x + i) + (double)v[1 + i];
  }
  if (a.g) l2_reduce<D0, L2RT>(a, (double *)sm2, acc, act, j0);
}

// The rows of k_adj_l2r for few points, a block's eight warps to the points
// that one warp takes there: the warps share the loads and the 32 partial
// sums, which are then added in the same order, so that a row has the same
// bits from either.  Bound: one point's chain (28 slots x 128 neurons, one
// point: 21 -> 11 us).
template <typename R, int D0>
__global__ void __launch_bounds__(L2T) k_adj_l2r8(L2aArgs a) {
  extern __shared__ __align__(16) unsigned char sm2[];
  constexpr int NWP = L2T / 32;
  const int na = a.na, n = a.n, nt = a.nt, j0 = blockIdx.y * nt, nsum = min(32, na);
  R *tb = (R *)sm2, *hh = tb + (size_t)na * 32;      // [na][32]
  R *red = hh + (size_t)na * 32;                     // [nsum][D0 + 1][32]
  R *M = red + (size_t)nsum * (D0 + 1) * 32;         // [na][nt]
  int *up = (int *)(M + ((size_t)na * nt + 1) / 2 * 2);  // [na][D0]
  for (int e = threadIdx.x; e < na * D0; e += L2T) up[e] = __ldg(a.up + e);
  for (int e = threadIdx.x; e < nt; e += L2T) M[e] = (R)1;
  __syncthreads();
  for (int p = 1; p <= a.k; ++p) {
    const int r0 = a.ds[p], nr = a.ds[p + 1] - r0;
    for (int e = threadIdx.x; e < nr * nt; e += L2T) {
      const int r = r0 + e / nt, jl = e % nt, j = min(j0 + jl, n - 1), pk = __ldg(a.par + r);
      M[(size_t)r * nt + jl] = (R)((double)M[(size_t)(pk & 0xffff) * nt + jl] *
                                   __ldg(a.W + (size_t)j * (D0 + 1) + 1 + (pk >> 16)));
    }
    __syncthreads();
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int jl = lane % nt, sub = lane / nt, j = min(j0 + jl, n - 1);
  const bool act = sub < a.ppw && j0 + jl < n;
  tb += lane;
  hh += lane;
  red += lane;
  for (long w0 = blockIdx.x; w0 * a.ppw < a.npts; w0 += gridDim.x) {
    const long pt = w0 * a.ppw + sub, q = min(pt, (long)a.npts - 1);
    const R *Tb = (const R *)a.Tb + (size_t)q * na * n + j;
    const R *sg = (const R *)a.sig + (size_t)q * (a.k + 2) * n + j;
    for (int g = warp, p = 0; g < na; g += NWP) {
      while (g >= a.ds[p + 1]) ++p;
      tb[g * 32] = __ldcs(Tb + (size_t)g * n);
      hh[g * 32] = sg[(size_t)(p + 1) * n] * M[(size_t)g * nt + jl];
    }
    __syncthreads();
    for (int w = warp; w < nsum; w += NWP) {
      R s[D0 + 1];
#pragma unroll
      for (int o = 0; o <= D0; ++o) s[o] = (R)0;
      for (int g = w; g < na; g += 32) {
        const R hg = hh[g * 32];
        s[0] += tb[g * 32] * hg;
#pragma unroll
        for (int i = 0; i < D0; ++i) {
          const int u = up[g * D0 + i];
          if (u >= 0) s[1 + i] += (R)(u >> 16) * tb[(u & 0xffff) * 32] * hg;
        }
      }
#pragma unroll
      for (int o = 0; o <= D0; ++o) red[(w * (D0 + 1) + o) * 32] = s[o];
    }
    __syncthreads();  // the next points' values go in behind this too: they meet the one above
    if (!act || pt >= a.npts) continue;
    double *row = a.rows + (size_t)pt * a.nw + a.woff + (size_t)j * (D0 + 1);
    for (int o = warp; o <= D0; o += NWP) {
      R v0 = (R)0, v = (R)0;
#pragma unroll 8
      for (int w = 0; w < nsum; ++w) {
        v0 += red[(w * (D0 + 1)) * 32];
        v += red[(w * (D0 + 1) + o) * 32];
      }
      row[o] = o ? (double)v0 * __ldg(a.X + (size_t)pt * D0 + o - 1) + (double)v : (double)v0;
    }
  }
}

// neurons of a tile: the layer cut into equal tiles of at most 32
int l2a_tile(int n) { return (n + (n + 31) / 32 - 1) / ((n + 31) / 32); }

size_t l2a_smem(int na, int nt, int d0, size_t msz) {
  return std::max(l2a_tables(na, nt, d0, msz), (size_t)(d0 + 1) * L2T * 8);
}

size_t l2r_smem(int na, int nt, int d0, size_t rsz) {
  return std::max(((size_t)2 * na * L2RT + (size_t)na * nt + 1) * rsz + (size_t)na * d0 * 4 + 16,
                  (size_t)(d0 + 1) * L2RT * 8);
}
size_t l2r8_smem(int na, int nt, int d0, size_t rsz) {
  return ((size_t)2 * na * 32 + (size_t)std::min(32, na) * (d0 + 1) * 32 + (size_t)na * nt + 1) * rsz +
         (size_t)na * d0 * 4 + 16;
}
// points for which a block's warps share a point's rows: until a warp's own
// fill the SMs
bool l2_few(const L2aArgs &a) {
  return (long)a.npts * ((a.n + a.nt - 1) / a.nt) < 16L * grid_sms() * a.ppw;
}
// the sets k_adj_l2r takes: rows while the columns fit, and gradients on the
// split path while its conversions to FP64, one set per slot, cost less than
// the Tb plane's traffic (in FP64 both orders agree to rounding)
constexpr int L2R_ROWS = 36, L2R_GRAD = 16;

template <typename R, typename BT, typename MT, int D0, int PT, L2Mode MODE>
int l2a_launch(L2aArgs a, cudaStream_t st) {
  size_t smem = l2a_smem(a.na, a.nt, D0, sizeof(MT));
  if (MODE == L2_ROWS8) smem = (smem + 15) / 16 * 16 + (size_t)PT * (D0 + 1) * L2T * 8;
  if (smem > 227 * 1024) return RC_UNSUPPORTED;
  const void *k = (const void *)k_adj_l2a<R, BT, MT, D0, PT, MODE>;
  CKC(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const int gy = (a.n + a.nt - 1) / a.nt;
  // points per block and pass
  const long per = (MODE == L2_ROWS8 ? 1L : (long)(L2T / 32)) * a.ppw * PT;
  const int full = resident_grid(k, L2T, smem);
  const int gx = (int)std::max(1L, std::min((a.npts + per - 1) / per, (long)std::max(1, full / gy)));
  // few points: the slots are split over blocks too, at least 8 to a block
  // (300 points of 8 neurons, 330 slots: 113 us before, 19 here)
  a.zsplit = MODE != L2_GRAD ? 1 : std::max(1, std::min(a.na / 8, full / std::max(1, gx * gy)));
  LAUNCH("k_bell_adj_l2", st, (k_adj_l2a<R, BT, MT, D0, PT, MODE><<<dim3(gx, gy, a.zsplit), L2T, smem, st>>>(a)));
  CKC(cudaGetLastError());
  return RC_OK;
}

// Rows.  A block's warps share the points' slots while a warp's own would
// leave SMs idle (split path, 330 slots x 32 neurons: 1 point 56 -> 29 us, 512
// 80 -> 39, 2048 98 -> 95; without it 4096 points 105).
template <typename R, typename BT, int D0>
int l2a_rows(const L2aArgs &a, cudaStream_t st) {
  constexpr int PT = sizeof(R) == 4 && D0 <= 5 ? 3 : 2;
  if (l2_few(a)) {
    const int rc = l2a_launch<R, BT, BT, D0, 1, L2_ROWS8>(a, st);
    if (rc != RC_UNSUPPORTED) return rc;
  }
  return l2a_launch<R, BT, BT, D0, PT, L2_ROWS>(a, st);
}

template <typename R, int D0>
int l2a_k(L2aArgs a, cudaStream_t st) {
  if (a.rows && a.na <= L2R_ROWS && l2_few(a)) {
    const size_t smem = l2r8_smem(a.na, a.nt, D0, sizeof(R));
    const void *k = (const void *)k_adj_l2r8<R, D0>;
    CKC(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int gy = (a.n + a.nt - 1) / a.nt;
    const long groups = (a.npts + a.ppw - 1) / a.ppw;
    const int gx = (int)std::min(groups, (long)std::max(1, resident_grid(k, L2T, smem) / gy));
    LAUNCH("k_bell_adj_l2", st, (k_adj_l2r8<R, D0><<<dim3(gx, gy), L2T, smem, st>>>(a)));
    CKC(cudaGetLastError());
    return RC_OK;
  }
  if (a.na <= (a.rows ? L2R_ROWS : sizeof(R) == 4 ? L2R_GRAD : 0)) {
    const size_t smem = l2r_smem(a.na, a.nt, D0, sizeof(R));
    const void *k = (const void *)k_adj_l2r<R, D0>;
    CKC(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int gy = (a.n + a.nt - 1) / a.nt;
    const long per = (long)(L2RT / 32) * a.ppw;
    const int gx = (int)std::max(1L, std::min((a.npts + per - 1) / per,
                                              (long)std::max(1, resident_grid(k, L2RT, smem) / gy)));
    LAUNCH("k_bell_adj_l2", st, (k_adj_l2r<R, D0><<<dim3(gx, gy), L2RT, smem, st>>>(a)));
    CKC(cudaGetLastError());
    return RC_OK;
  }
  // Runs of FP32 sums: |A| / 32 slots in whole groups of four; below that a
  // gradient's sums are FP64 (65536 points x 128, 35 slots: 0.48 ms, 0.41 in
  // FP32).  k_adj_l2s added the parts of a row in FP32 too, so a row keeps its
  // runs of one group.
  const int run = (a.na + 31) / 32 / 4;
  if constexpr (sizeof(R) == 4) {
    a.chain = std::max(1, run);
    if (a.rows) return l2a_rows<R, float, D0>(a, st);
    if (run >= 1) return l2a_launch<R, float, float, D0, D0 <= 4 ? 4 : 3, L2_GRAD>(a, st);
  }
  a.chain = a.na;
  if constexpr (sizeof(R) == 8)
    if (a.rows) return l2a_rows<R, double, D0>(a, st);
  return l2a_launch<R, double, double, D0, sizeof(R) == 8 && D0 >= 4 ? 2 : 3, L2_GRAD>(a, st);
}

template <typename R>
int l2a_t(int d0, const L2aArgs &a, cudaStream_t st) {
  switch (d0) {
    case 1: return l2a_k<R, 1>(a, st);
    case 2: return l2a_k<R, 2>(a, st);
    case 3: return l2a_k<R, 3>(a, st);
    case 4: return l2a_k<R, 4>(a, st);
    case 5: return l2a_k<R, 5>(a, st);
    case 6: return l2a_k<R, 6>(a, st);
    case 7: return l2a_k<R, 7>(a, st);
    case 8: return l2a_k<R, 8>(a, st);
    default: return RC_UNSUPPORTED;
  }
}

template <typename R>
int fwd_col_t(const ColDev &d, const ColArgs &a, bool train, cudaStream_t st) {
  const size_t smem = col_fwd_smem(d.na, d.kt, d.nfrec, sizeof(R));
  const void *k = train ? (const void *)k_bell_fwd_col<R, true> : (const void *)k_bell_fwd_col<R, false>;
  CKC(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  const long total = (long)a.npts * a.n;
  const int grid = (int)std::max(1L, std::min((total + NT - 1) / NT, (long)resident_grid(k, NT, smem)));
  if (train) { LAUNCH("k_bell_fwd", st, (k_bell_fwd_col<R, true><<<grid, NT, smem, st>>>(a))); }
  else { LAUNCH("k_bell_fwd", st, (k_bell_fwd_col<R, false><<<grid, NT, smem, st>>>(a))); }
  CKC(cudaGetLastError());
  return RC_OK;
}

template <typename R>
int adj_col_t(const ColDev &d, const ColArgs &a, cudaStream_t st) {
  const size_t smem = col_adj_smem(d.na, d.narec, sizeof(R));
  // one chain per sum, as in k_bell_adj7, for launches too small for the
  // block-per-point kernels to have been timed on, where that one ran; two,
  // as in k_bell_adj5, beyond
  const bool one = (long)a.npts * ((a.n + 128 / (int)sizeof(R) - 1) / (128 / (int)sizeof(R))) <
                   8L * grid_sms();
  const void *k = one ? (const void *)k_bell_adj_col<R, 1> : (const void *)k_bell_adj_col<R, 2>;
  CKC(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
  // at least one neuron row of threads, so that the stride is not zero
  const long total = (long)a.npts * a.n;
  long grid = std::max(1L, std::min((total + NT - 1) / NT, (long)resident_grid(k, NT, smem)));
  grid = std::max(grid, (long)(a.n + NT - 1) / NT);
  if (one) { LAUNCH("k_bell_adj", st, (k_bell_adj_col<R, 1><<<(int)grid, NT, smem, st>>>(a))); }
  else { LAUNCH("k_bell_adj", st, (k_bell_adj_col<R, 2><<<(int)grid, NT, smem, st>>>(a))); }
  CKC(cudaGetLastError());
  return RC_OK;
}

}  // namespace

// ------------------------------------------------------------ host side
// The rule, by the forward and adjoint measured against the best of the
// block-per-point kernels (us, 8192 points, layers of 64; FP64):
//   |A|   10: 39 + 41 against 436 + 306     35: 352 + 284 against 660 + 482
//         21: 200 + 123 against 904 + 404   56: 1145 + 704 against 1150 + 706
// and in FP32 33 + 31 against 201 + 150 (10), 164 + 133 against 287 + 220
// (35), 558 + 288 against 465 + 293 (56): the columns win while the state
// leaves several warps per SM, up to 36 slots.  A launch of few neurons is a
// column's serial chain and hides nothing behind it; by neurons (points x
// width, the width in whole 128-byte rows of the other kernels), forward and
// adjoint, us, columns against the best of the others:
//   FP32  15 slots  4096: 17/11 14/8   16384: 17/19 14/12   65536: 19/43 15/27
//         28        4096: 28/12 20/9   16384: 29/23 21/15   32768: 30/33 21/21
//         35        8192: 22/13 21/10  32768: 23/25 23/21   65536: 25/43 25/33
//   FP64  15        2048: 17/10 15/8    8192: 17/19 15/13   16384: 17/27 15/19
//         28        8192: 31/25 21/15  16384: 31/35 21/23   32768: 33/62 23/37
// and half as many where the width is no multiple of 16 bytes, which the
// others' fast forms need.
constexpr int COL_MAX = 36, COL_SHORT = 16;
constexpr long COL_BYTES = 64 * 1024;  // of one slot's neurons; twice that beyond COL_SHORT

bool col_set(const TableSet &t) { return t.na <= COL_MAX && t.d0 <= D0MAX; }

void upload_col(const TableSet &t, const ColProg &P, ColDev &d, PlanBlock &b) {
  d = ColDev();
  b.add(&d.fhdr, P.fhdr);
  b.add(&d.ahdr, P.ahdr);
  b.add(&d.frec, P.frec);
  b.add(&d.arec, P.arec);
  b.add(&d.dstart, P.dstart);
  d.na = t.na;
  d.kt = P.kt;
  d.nfrec = (int)P.frec.size();
  d.narec = (int)P.arec.size();
  d.ok = true;
}

bool col_fits(const ColDev &d, int n, int prec) {
  const size_t rsz = prec == PREC_F64 ? 8 : 4;
  return d.ok && n >= 1 && col_fwd_smem(d.na, d.kt, d.nfrec, rsz) <= 227 * 1024 &&
         col_adj_smem(d.na, d.narec, rsz) <= 226 * 1024;
}

bool col_applies(const ColDev &d, int n, int npts, int prec) {
  const int row = prec == PREC_F64 ? 16 : 32;  // neurons of 128 bytes
  const long bytes = (long)npts * ((n + row - 1) / row) * 128;
  const long line = (d.na <= COL_SHORT ? 1 : 2) * COL_BYTES / (n % (row / 8) ? 2 : 1);
  return bytes >= line && col_fits(d, n, prec);
}

int bell_fwd_col(const ColDev &d, const DevTables &t, int n, int npts, const void *S, void *T,
                 void *h, bool train, int prec, cudaStream_t st) {
  ColArgs a{};
  a.n = n; a.na = d.na; a.npts = npts; a.k = t.k; a.kt = d.kt; a.iact = t.iact;
  a.nrec = d.nfrec; a.hdr = d.fhdr; a.rec = d.frec; a.dstart = d.dstart; a.sc = t.bp.sc64;
  a.tpc = t.tpc; a.A = S; a.C = T; a.D = h;
  return prec == PREC_F64 ? fwd_col_t<double>(d, a, train, st) : fwd_col_t<float>(d, a, train, st);
}

int bell_adj_col(const ColDev &d, const DevTables &t, int n, int npts, const void *Tb,
                 const void *h, void *Sb, double *gbias, int gstride, int prec,
                 cudaStream_t st) {
  ColArgs a{};
  a.n = n; a.na = d.na; a.npts = npts; a.k = t.k; a.kt = d.kt; a.iact = t.iact;
  a.nrec = d.narec; a.hdr = d.ahdr; a.rec = d.arec; a.dstart = d.dstart; a.sc = t.bp.sc64;
  a.A = Tb; a.B = h; a.C = Sb; a.gbias = gbias; a.gstride = gstride;
  return prec == PREC_F64 ? adj_col_t<double>(d, a, st) : adj_col_t<float>(d, a, st);
}

bool l2a_applies(int d0, int na, int n, int prec) {
  const size_t msz = prec == PREC_F64 ? 8 : 4;  // the smallest form of the monomials
  return d0 >= 1 && d0 <= 8 && n >= 1 && na <= 65535 &&
         l2a_smem(na, l2a_tile(n), d0, msz) <= 227 * 1024;
}

int bell_adj_l2a(const DevTables &t, int n, int npts, const void *Tb, const double *X, double *g,
                 double *rows, size_t nw, size_t woff, int prec, const L2Analytic &an,
                 cudaStream_t st) {
  if (npts <= 0) return RC_OK;
  L2aArgs a{};
  a.n = n; a.na = t.na; a.npts = npts; a.k = t.k; a.nt = l2a_tile(n);
  a.ppw = std::max(1, 32 / a.nt); a.zsplit = 1; a.up = t.l2up; a.par = an.par; a.sc = t.bp.sc64;
  a.Tb = Tb; a.sig = an.sig; a.X = X; a.W = an.W; a.g = g; a.rows = rows; a.nw = nw;
  a.woff = woff;
  for (int p = 0; p < KMAX + 2; ++p) a.ds[p] = p <= an.k + 1 ? an.dstart[p] : t.na;
  return prec == PREC_F64 ? l2a_t<double>(t.d0, a, st) : l2a_t<float>(t.d0, a, st);
}

}  // namespace dnnf90
