// bell_tile64.cu - the register-tiled Bell forward and adjoint of
// bell_tile.cu in FP64: the same recurrences, layout and records, with rows
// of 16 neurons (128 bytes) and the two half-warps working side by side.
//
// Forward: lanes 0-15 run the D chain and lanes 16-31 the E chain of the
// same 16 neurons.  Both multiply by the same s~ row (one broadcast read),
// and a (D, E) row is 32 doubles, so the shared memory is that of the FP32
// kernel (183 KB at D0 = 4, K = 7) and a side-8 triangle costs 36 + 36
// doubles in registers.
// Adjoint: the halves run two records of one tile side at a time, of two
// output tiles of one degree or of the two halves of one tile's records
// (TileAdj64).
//
// Twelve warps (a fourth warp per SM quarter would leave 128 registers, and
// a side-8 triangle needs 144 for its two tiles).
//
// Bound: issue and latency (ncu, 1184 points of 128 neurons: 35 % of issue
// slots, FP64 pipe 19 % in the forward and 11 % in the adjoint; 46 K warp
// instructions per item, 10.6 K of them multiply-adds).  One launch over 8191
// points of 128 neurons at D0 = 4, K = 7: forward 7.1 ms (7.8 before its
// records were read one ahead) against 15.1 for v8, adjoint 4.7 against 7.8 for v7 (bell.cu), which gather one operand per
// multiply-add.
#include <cuda_runtime.h>

#include <algorithm>
#include <string>
#include <vector>

#include "bell.hpp"
#include "bell_tile.cuh"
#include "engine.hpp"
#include "kernels.cuh"
#include "tile_plan.hpp"

namespace dnnf90 {

namespace {

constexpr int TWF = TILE_WARPS64_F, TWA = TILE_WARPS64_A;
constexpr int NPB = 16;                        // neurons per row
constexpr int LMAX = TILE_KMAX + 1;

// rows of a [na][n] plane slice (neurons j0 .. j0 + 15) into shared rows
// perm[r] of dst (128 bytes each), 16-byte pieces; n is even, so a piece is
// wholly in or out of the row
__device__ __forceinline__ void stage_perm(unsigned char *dst, const double *src, const int *perm,
                                           int na, int n, int j0) {
  for (int c = threadIdx.x; c < na * 8; c += blockDim.x) {
    const int r = c >> 3, piece = c & 7;
    const int col = j0 + piece * 2;
    const int ok = col < n ? 16 : 0;
    cp16(dst + perm[r] * 128 + piece * 16, src + (size_t)r * n + (ok ? col : 0), ok);
  }
}

// ------------------------------------------------------------ forward
struct Fwd64Args {
  int n, na, npts, gy, k, iact;
  int nunit, nrec;
  int o_s1, o_d0, o_d1, o_sig, o_list, o_unit, o_rec, o_perm, o_rowslot, o_fact, o_ifact;
  const double *tpc;
  const int *list;       // [k][TWF][2]
  const int4 *unit;      // [nunit]: L | origin << 8, first record, records, out row
  const uint32_t *rec;   // [nrec]: s row | d row << 16
  const int *perm, *rowslot;
  const double *fact, *ifact;
  const double *S;
  double *T, *h;
};

template <int TD, int C, int E, int EN>
struct FwdRow {
  static __device__ __forceinline__ void run(const double *sv, double dv, double *acc) {
    constexpr int o = tadd(TD, E, C);
    acc[o] = fma(sv[E], dv, acc[o]);
    FwdRow<TD, C, E + 1, EN>::run(sv, dv, acc);
  }
};
template <int TD, int C, int EN>
struct FwdRow<TD, C, EN, EN> {
  static __device__ __forceinline__ void run(const double *, double, double *) {}
};
template <int TD, int L, bool Z, int C, int CN>
struct FwdRows {
  static __device__ __forceinline__ void run(const double *sv, const double *d, double *acc) {
    const double dv = d[C * 32];
    FwdRow<TD, C, Z ? 1 : 0, tsize(TD, L - tdeg(TD, C))>::run(sv, dv, acc);
    FwdRows<TD, L, Z, C + 1, CN>::run(sv, d, acc);
  }
};
template <int TD, int L, bool Z, int CN>
struct FwdRows<TD, L, Z, CN, CN> {
  static __device__ __forceinline__ void run(const double *, const double *, double *) {}
};

template <int TD, int L, bool Z>
__device__ __forceinline__ void tile_fwd(const double *s, const double *d,
                                         double (&acc)[tsize(TD, L)]) {
  constexpr int NT = tsize(TD, L);
  constexpr int ND = tsize(TD, Z ? L - 1 : L);
  double sv[NT];
#pragma unroll
  for (int e = 0; e < NT; ++e) sv[e] = (Z && e == 0) ? 0.0 : s[e * NPB];
  FwdRows<TD, L, Z, 0, ND>::run(sv, d, acc);
}

struct FwdCtx {
  const double *S;        // this lane's neuron in the current S buffer
  const double *Dr;       // this lane's double of the buffer of (D, E)_{q+1}
  double *Dw;             // this lane's double of the buffer of (D, E)_q
  const uint32_t *rec;
  const int *rowslot;
  const double *fact;
  double *O;              // this lane's output plane (T or h) at its neuron; null: none
  int n;
};

template <int TD, int L>
__device__ __forceinline__ void fwd_unit(const FwdCtx &c, int4 u, int q, double inv, double sg) {
  constexpr int NT = tsize(TD, L);
  double acc[NT];
#pragma unroll
  for (int e = 0; e < NT; ++e) acc[e] = 0.0;
  {
    const uint32_t r = c.rec[u.y];
    tile_fwd<TD, L, true>(c.S + (r & 0xffffu) * NPB, c.Dr + (r >> 16) * 32, acc);
  }
  const int end = u.y + u.z;
  uint32_t rn = c.rec[u.y + 1];  // a record ahead (past the last: the next table's word)
  for (int i = u.y + 1; i < end; ++i) {
    const uint32_t r = rn;
    rn = c.rec[i + 1];
    tile_fwd<TD, L, false>(c.S + (r & 0xffffu) * NPB, c.Dr + (r >> 16) * 32, acc);
  }
#pragma unroll
  for (int e = 0; e < NT; ++e) acc[e] *= inv;
  if (u.x >> 8) acc[0] = sg;  // the origin: D_q(0) = sigma_q, E_q(0) = sigma_{q+1}
  if (q > 0) {
#pragma unroll
    for (int e = 0; e < NT; ++e) c.Dw[(u.w + e) * 32] = acc[e];
  } else if (c.O) {
#pragma unroll
    for (int e = 0; e < NT; ++e) {
      const int row = u.w + e;
      c.O[(size_t)c.rowslot[row] * c.n] = c.fact[row] * acc[e];
    }
  }
}

template <int TD, bool TRAIN>
__global__ void __launch_bounds__(TWF * 32, 1) k_bell_fwd64(Fwd64Args a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char *sm = smem_raw;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int l16 = lane & 15, half = lane >> 4;
  const int n = a.n, na = a.na, K = a.k;
  int *slist = (int *)(sm + a.o_list);
  int4 *sunit = (int4 *)(sm + a.o_unit);
  uint32_t *srec = (uint32_t *)(sm + a.o_rec);
  int *sperm = (int *)(sm + a.o_perm);
  int *srowslot = (int *)(sm + a.o_rowslot);
  double *sfact = (double *)(sm + a.o_fact);
  double *sifact = (double *)(sm + a.o_ifact);
  copy_words(slist, a.list, K * TWF * 2);
  copy_words(sunit, a.unit, a.nunit * 4);
  copy_words(srec, a.rec, a.nrec);
  copy_words(sperm, a.perm, na);
  copy_words(srowslot, a.rowslot, na);
  copy_words(sfact, a.fact, na * 2);
  copy_words(sifact, a.ifact, na * 2);
  __syncthreads();
  const size_t plane = (size_t)na * n;
  const long nitem = (long)a.npts * a.gy;
  long it0, it1;
  block_items(nitem, it0, it1);
  if (it0 < it1)
    stage_perm(sm, a.S + (it0 % a.npts) * plane, sperm, na, n, (int)(it0 / a.npts) * NPB);
  cp_commit();
  double *sig = (double *)(sm + a.o_sig) + l16;
  FwdCtx c;
  c.rec = srec;
  c.rowslot = srowslot;
  c.fact = sfact;
  c.n = n;
  int buf = 0;
  for (long it = it0; it < it1; ++it) {
    const int pt = (int)(it % a.npts);
    const int j = (int)(it / a.npts) * NPB + l16;
    cp_wait_all();
    __syncthreads();  // this item's S rows are in; every warp is done with the last item
    if (it + 1 < it1)
      stage_perm(sm + (buf ? 0 : a.o_s1), a.S + ((it + 1) % a.npts) * plane, sperm, na, n,
                 (int)((it + 1) / a.npts) * NPB);
    cp_commit();
    double *Sb = (double *)(sm + (buf ? a.o_s1 : 0)) + l16;
    // S_a -> S_a / a!, 16 bytes per thread at a time; the origin row keeps
    // S_0 (0! = 1) and is left alone, since the sigma warps read it next
    {
      unsigned char *sb0 = sm + (buf ? a.o_s1 : 0);
#pragma unroll 4
      for (int e = threadIdx.x + 8; e < na * 8; e += blockDim.x) {
        double2 *p = (double2 *)(sb0 + e * 16);
        const double f = sifact[e >> 3];
        double2 v = *p;
        v.x *= f;
        v.y *= f;
        *p = v;
      }
    }
    double *dk = (double *)(sm + ((K & 1) ? a.o_d1 : a.o_d0)) + lane;  // row 0 of buffer K & 1
    if (a.iact == 0) {
      // tanh: warp q forms sigma_q = P_q(tanh S_0) in the order of
      // sigma_derivs, the halves alike; D_K = sigma_K, E_K = sigma_{K+1}
      for (int q = warp; q <= K + 1; q += TWF) {
        const double t = tanh(Sb[0]);
        const double *row = a.tpc + q * (K + 3);
        double v = __ldg(row + q + 1);
        for (int i = q; i >= 0; --i) v = v * t + __ldg(row + i);
        if (half == 0) sig[q * NPB] = v;
        if (q == K + half) dk[0] = v;
      }
    } else if (warp == 0) {
      double d[TILE_KMAX + 2];
      sigma_derivs(a.iact, a.tpc, K, Sb[0], d);
#pragma unroll
      for (int q = 0; q <= TILE_KMAX + 1; ++q) {
        if (q <= K + 1 && half == 0) sig[q * NPB] = d[q];
        if (q == K + half) dk[0] = d[q];
      }
    }
    __syncthreads();
    c.S = Sb;
    c.O = j >= n ? nullptr
          : half == 0 ? a.T + pt * plane + j
          : TRAIN ? a.h + pt * plane + j
                  : nullptr;
    for (int q = K - 1; q >= 0; --q) {
      c.Dr = (const double *)(sm + (((q + 1) & 1) ? a.o_d1 : a.o_d0)) + lane;
      c.Dw = (double *)(sm + ((q & 1) ? a.o_d1 : a.o_d0)) + lane;
      const double inv = 1.0 / (double)(q + 1);
      const double sg = sig[(q + half) * NPB];
      const int u0 = slist[(q * TWF + warp) * 2], un = slist[(q * TWF + warp) * 2 + 1];
      for (int u = u0; u < u0 + un; ++u) {
        const int4 U = sunit[u];
        switch (U.x & 0xff) {
#define F64(LL) \
  case LL: fwd_unit<TD, LL>(c, U, q, inv, sg); break;
          F64(1) F64(2) F64(3) F64(4) F64(5) F64(6) F64(7) F64(8)
#undef F64
          default: break;
        }
      }
      if (q > 0) __syncthreads();
    }
    buf ^= 1;
  }
  cp_wait_all();
}

// ------------------------------------------------------------ adjoint
struct Adj64Args {
  int n, na, npts, gy, gstride;
  int nunit, nrec, nfin, nzero;
  int o_b1, o_scr, o_zero, o_list, o_unit, o_rec, o_flist, o_fin, o_perm, o_rowslot, o_fact,
      o_ifact;
  const int *list;       // [TWA][2]
  const int4 *unit;      // [nunit][2] (TileAdj64::unit)
  const uint2 *rec;      // [nrec]
  const int *flist;      // [TWA][2]
  const int4 *fin;       // [nfin]
  const int *perm, *rowslot;
  const double *fact, *ifact;
  const double *Tb, *h;
  double *Sb;
  double *gbias;
};

// one record: acc[a - c] += (a! Tb)_a (h / c!)_c over a in the Tb tile of
// side L and c <= a (componentwise)
template <int TD, int A, int C1, int C2, bool END = (C2 > tsecond(TD, A))>
struct AdjInner;
template <int TD, int A, int C1, int C2>
struct AdjInner<TD, A, C1, C2, false> {
  static __device__ __forceinline__ void run(double x, const double *hv, double *acc) {
    constexpr int o = tindex(TD, tfirst(TD, A) - C1, tsecond(TD, A) - C2);
    acc[o] = fma(x, hv[tindex(TD, C1, C2)], acc[o]);
    AdjInner<TD, A, C1, C2 + 1>::run(x, hv, acc);
  }
};
template <int TD, int A, int C1, int C2>
struct AdjInner<TD, A, C1, C2, true> {
  static __device__ __forceinline__ void run(double, const double *, double *) {}
};
template <int TD, int A, int C1, bool END = (C1 > tfirst(TD, A))>
struct AdjOuter;
template <int TD, int A, int C1>
struct AdjOuter<TD, A, C1, false> {
  static __device__ __forceinline__ void run(double x, const double *hv, double *acc) {
    AdjInner<TD, A, C1, 0>::run(x, hv, acc);
    AdjOuter<TD, A, C1 + 1>::run(x, hv, acc);
  }
};
template <int TD, int A, int C1>
struct AdjOuter<TD, A, C1, true> {
  static __device__ __forceinline__ void run(double, const double *, double *) {}
};
template <int TD, int A, int AN>
struct AdjRows {
  static __device__ __forceinline__ void run(const double *tb, const double *hv, double *acc) {
    const double x = tb[A * NPB];
    AdjOuter<TD, A, 0>::run(x, hv, acc);
    AdjRows<TD, A + 1, AN>::run(tb, hv, acc);
  }
};
template <int TD, int AN>
struct AdjRows<TD, AN, AN> {
  static __device__ __forceinline__ void run(const double *, const double *, double *) {}
};

// the steps of side L, L - 1, ..., 1 of a unit in turn (see AdjL of
// bell_tile.cu); every unit keeps the accumulators of the largest tile
template <int TD, int L>
struct AdjL {
  static __device__ __forceinline__ void run(const double *tbb, const double *hb,
                                             const double *zero, const uint2 *rec, int half,
                                             int i, uint32_t cw, int lo,
                                             double (&acc)[tsize(TD, LMAX)]) {
    const int cnt = lo >= L ? (int)((cw >> (4 * (lo - L))) & 15u) : 0;
    constexpr int NT = tsize(TD, L);
    for (int k = 0; k < cnt; ++k) {
      const uint2 rr = rec[i + k];
      const uint32_t r = half ? rr.y : rr.x;
      // a missing record is zeros times zeros: Tb may be infinite
      const bool null = r & TILE_NULL;
      const double *hp = null ? zero : hb + (r & (TILE_NULL - 1)) * NPB;
      const double *tp = null ? zero : tbb + ((r >> 14) & 0x3fffu) * NPB;
      double hv[NT];
#pragma unroll
      for (int e = 0; e < NT; ++e) hv[e] = hp[e * NPB];
      AdjRows<TD, 0, NT>::run(tp, hv, acc);
    }
    AdjL<TD, L - 1>::run(tbb, hb, zero, rec, half, i + cnt, cw, lo, acc);
  }
};
template <int TD>
struct AdjL<TD, 0> {
  static __device__ __forceinline__ void run(const double *, const double *, const double *,
                                             const uint2 *, int, int, uint32_t, int,
                                             double (&)[tsize(TD, LMAX)]) {}
};

// a unit's results: the halves' sums exchanged (one tile) or each half's own
// tile (pair), into scratch rows or scaled by 1/b! and stored
template <int TD, int LO>
__device__ __forceinline__ void adj_store(double (&acc)[tsize(TD, LMAX)], int flags, int row0,
                                          int half, double *scr, const int *rowslot,
                                          const double *ifact, double *Sb, int n, bool act,
                                          double &gb) {
  constexpr int NT = tsize(TD, LO);
  const bool pair = flags & 0x100, toscr = flags & 0x200;
  if (!pair)
#pragma unroll
    for (int e = 0; e < NT; ++e) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], 16);
  if (!pair && half) return;
  if (toscr) {
#pragma unroll
    for (int e = 0; e < NT; ++e) scr[(row0 + e) * NPB] = acc[e];
  } else {
#pragma unroll
    for (int e = 0; e < NT; ++e) {
      const int row = row0 + e;
      const double v = acc[e] * ifact[row];
      if (act) Sb[(size_t)rowslot[row] * n] = v;
      if (row == 0) gb += v;
    }
  }
}

template <int TD>
__global__ void __launch_bounds__(TWA * 32, 1) k_bell_adj64(Adj64Args a) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  unsigned char *sm = smem_raw;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int l16 = lane & 15, half = lane >> 4;
  const int n = a.n, na = a.na;
  int *slist = (int *)(sm + a.o_list);
  int4 *sunit = (int4 *)(sm + a.o_unit);
  uint2 *srec = (uint2 *)(sm + a.o_rec);
  int *sflist = (int *)(sm + a.o_flist);
  int4 *sfin = (int4 *)(sm + a.o_fin);
  int *sperm = (int *)(sm + a.o_perm);
  int *srowslot = (int *)(sm + a.o_rowslot);
  double *sfact = (double *)(sm + a.o_fact);
  double *sifact = (double *)(sm + a.o_ifact);
  copy_words(slist, a.list, TWA * 2);
  copy_words(sunit, a.unit, a.nunit * 8);
  copy_words(srec, a.rec, a.nrec * 2);
  copy_words(sflist, a.flist, TWA * 2);
  copy_words(sfin, a.fin, a.nfin * 4);
  copy_words(sperm, a.perm, na);
  copy_words(srowslot, a.rowslot, na);
  copy_words(sfact, a.fact, na * 2);
  copy_words(sifact, a.ifact, na * 2);
  for (int e = threadIdx.x; e < a.nzero * NPB; e += blockDim.x) ((double *)(sm + a.o_zero))[e] = 0.0;
  __syncthreads();
  double *scr = (double *)(sm + a.o_scr) + l16;
  const double *zero = (const double *)(sm + a.o_zero) + l16;
  const size_t plane = (size_t)na * n;
  const long nitem = (long)a.npts * a.gy;
  long it0, it1;
  block_items(nitem, it0, it1);
  // buffer b: Tb rows at b * o_b1, h rows na rows further
  auto stage = [&](int b, long it) {
    const size_t o = (it % a.npts) * plane;
    const int j0 = (int)(it / a.npts) * NPB;
    unsigned char *dst = sm + b * a.o_b1;
    stage_perm(dst, a.Tb + o, sperm, na, n, j0);
    stage_perm(dst + na * 128, a.h + o, sperm, na, n, j0);
  };
  if (it0 < it1) stage(0, it0);
  cp_commit();
  const int u0 = slist[warp * 2], un = slist[warp * 2 + 1];
  const int f0 = sflist[warp * 2], fn = sflist[warp * 2 + 1];
  // the bias gradient: Sb_0 of this lane's neuron, added once per neuron tile
  // (gb: the units' outputs; gbp: the split tiles', summed one item later)
  double gb = 0.0, gbp = 0.0;
  int gj = -1, gjp = -1;
  auto flush = [&](double &g, int &jj, int jn) {
    if (jj != jn) {
      if (a.gbias && jj >= 0 && jj < n && g != 0.0) atomicAdd(a.gbias + (size_t)jj * a.gstride, g);
      g = 0.0;
      jj = jn;
    }
  };
  // split output tiles of item itp: each element's parts summed in a fixed
  // order, the elements dealt over all half-warps
  auto finish = [&](long itp) {
    const int jp = (int)(itp / a.npts) * NPB + l16;
    flush(gbp, gjp, jp);
    double *Sbp = a.Sb + (itp % a.npts) * plane + jp;
    for (int f = f0 + half; f < f0 + fn; f += 2) {
      const int4 F = sfin[f];  // row, parts, first scratch row, part stride
      double v = 0.0;
      for (int p = 0; p < F.y; ++p) v += scr[(F.z + p * F.w) * NPB];
      v *= sifact[F.x];
      if (jp < n) Sbp[(size_t)srowslot[F.x] * n] = v;
      if (F.x == 0) gbp += v;
    }
    __syncwarp();
  };
  int buf = 0;
  for (long it = it0; it < it1; ++it) {
    const int pt = (int)(it % a.npts);
    const int j = (int)(it / a.npts) * NPB + l16;
    const bool act = j < n;
    flush(gb, gj, j);
    cp_wait_all();
    __syncthreads();  // this item's rows are in; every warp is done with the last item
    if (it + 1 < it1) stage(buf ^ 1, it + 1);
    cp_commit();
    // Tb_a -> a! Tb_a, h_g -> h_g / g!, 16 bytes per thread at a time
    {
      unsigned char *b0 = sm + buf * a.o_b1;
#pragma unroll 4
      for (int e = threadIdx.x; e < 2 * na * 8; e += blockDim.x) {
        const int r = e >> 3;
        const double f = r < na ? sfact[r] : sifact[r - na];
        double2 *p = (double2 *)(b0 + e * 16);
        double2 v = *p;
        v.x *= f;
        v.y *= f;
        *p = v;
      }
    }
    if (it > it0) finish(it - 1);  // the last item's split parts are in since the barrier
    __syncthreads();               // the rows are scaled, the scratch rows are free
    double *Sb = a.Sb + pt * plane + j;
    const double *tbb = (const double *)(sm + buf * a.o_b1) + l16, *hb = tbb + na * NPB;
    for (int u = u0; u < u0 + un; ++u) {
      const int4 U = sunit[2 * u], V = sunit[2 * u + 1];  // flags, first step, counts, row A; row B
      double acc[tsize(TD, LMAX)];
#pragma unroll
      for (int e = 0; e < tsize(TD, LMAX); ++e) acc[e] = 0.0;
      const int lo = U.x & 0xff;
      AdjL<TD, LMAX>::run(tbb, hb, zero, srec, half, U.y, (uint32_t)U.z, lo, acc);
      const int row0 = half ? V.x : U.w;
      switch (lo) {
#define ST64(LL)                                                                              \
  case LL:                                                                                    \
    adj_store<TD, LL>(acc, U.x, row0, half, scr, srowslot, sifact, Sb, n, act, gb);           \
    break;
        ST64(1) ST64(2) ST64(3) ST64(4) ST64(5) ST64(6) ST64(7) ST64(8)
#undef ST64
        default: break;
      }
      __syncwarp();
    }
    buf ^= 1;
  }
  cp_wait_all();
  __syncthreads();  // the last item's split parts are in
  if (it0 < it1) finish(it1 - 1);
  flush(gb, gj, -1);
  flush(gbp, gjp, -1);
}

}  // namespace

// ------------------------------------------------------------ host side
void upload_tile64_plan(const TableSet &t, Tile64Dev &d, PlanBlock &b) {
  d = Tile64Dev();
  const TilePlan P = build_tile_plan(t, TWF, TWA);
  if (!P.ok) return;
  const int na = P.na, K = P.k, lim = 227 * 1024;
  // what the adjoint's tables take beside its rows, scratch and zeros (an
  // upper bound, checked below)
  const int zrows = tile_size(P.td, K + 1);
  const int scr = (lim - 4 * na * 128 - zrows * 128 - na * 24 - 16 * 1024) / 128;
  const TileAdj64 A = scr > 0 ? build_tile_adj64(t, P, TWA, scr) : TileAdj64();
  std::vector<double> fact(na), ifact(na);
  for (int r = 0; r < na; ++r) {
    const int ia = P.rowslot[r];
    double f = 1.0;
    for (int i = 0; i < t.d0; ++i)
      for (int v = 2; v <= t.alpha[(size_t)ia * t.d0 + i]; ++v) f *= v;
    fact[r] = f;
    ifact[r] = 1.0 / f;
  }
  b.add(&d.flist, P.flist);
  b.add(&d.funit, P.funit);
  b.add(&d.frec, P.frec);
  b.add(&d.perm, P.perm);
  b.add(&d.rowslot, P.rowslot);
  b.add(&d.fact, fact);
  b.add(&d.ifact, ifact);
  if (A.ok) {
    b.add(&d.alist, A.list);
    b.add(&d.aunit, A.unit);
    b.add(&d.arec, A.rec);
    b.add(&d.aflist, A.flist);
    b.add(&d.afin, A.fin);
  }
  d.td = P.td;
  d.k = K;
  d.na = na;
  d.nfunit = (int)P.funit.size() / 4;
  d.nfrec = (int)P.frec.size();
  int o = 0;
  auto take = [&](int bytes, int align) {
    o = (o + align - 1) / align * align;
    const int at = o;
    o += bytes;
    return at;
  };
  take(2 * na * 128, 128);  // two S buffers
  d.f_o_d0 = take(std::max(1, P.nbuf[0]) * 256, 128);
  d.f_o_d1 = take(std::max(1, P.nbuf[1]) * 256, 128);
  d.f_o_sig = take((K + 2) * 128, 128);
  d.f_o_unit = take(d.nfunit * 16, 16);
  d.f_o_fact = take(na * 8, 8);
  d.f_o_ifact = take(na * 8, 8);
  d.f_o_list = take(K * TWF * 8, 4);
  d.f_o_rec = take(d.nfrec * 4, 4);
  d.f_o_perm = take(na * 4, 4);
  d.f_o_rowslot = take(na * 4, 4);
  d.f_smem = o;
  d.f_ok = d.f_smem <= lim;
  if (A.ok) {
    d.naunit = (int)A.unit.size() / 8;
    d.narec = (int)A.rec.size() / 2;
    d.nafin = (int)A.fin.size() / 4;
    d.nzero = zrows;
    o = 0;
    take(4 * na * 128, 128);  // two buffers of Tb and h rows
    d.a_o_scr = take(std::max(1, A.nscratch) * 128, 128);
    d.a_o_zero = take(zrows * 128, 128);
    d.a_o_unit = take(d.naunit * 32, 16);
    d.a_o_fin = take(d.nafin * 16, 16);
    d.a_o_fact = take(na * 8, 8);
    d.a_o_ifact = take(na * 8, 8);
    d.a_o_rec = take(d.narec * 8, 8);
    d.a_o_list = take(TWA * 8, 4);
    d.a_o_flist = take(TWA * 8, 4);
    d.a_o_perm = take(na * 4, 4);
    d.a_o_rowslot = take(na * 4, 4);
    d.a_smem = o;
    d.a_ok = d.a_smem <= lim;
  }
}

bool tile64_fwd_applies(const Tile64Dev &d, int n) { return d.f_ok && n % 2 == 0; }
bool tile64_adj_applies(const Tile64Dev &d, int n) { return d.a_ok && n % 2 == 0; }

int bell_fwd_tile64(const Tile64Dev &d, const DevTables &t, int n, int npts, const void *S,
                    void *T, void *h, bool train, cudaStream_t st) {
  if (!tile64_fwd_applies(d, n)) return RC_UNSUPPORTED;
  Fwd64Args a;
  a.n = n; a.na = d.na; a.npts = npts; a.gy = (n + NPB - 1) / NPB; a.k = d.k; a.iact = t.iact;
  a.nunit = d.nfunit; a.nrec = d.nfrec;
  a.o_s1 = d.na * 128; a.o_d0 = d.f_o_d0; a.o_d1 = d.f_o_d1; a.o_sig = d.f_o_sig;
  a.o_list = d.f_o_list; a.o_unit = d.f_o_unit; a.o_rec = d.f_o_rec; a.o_perm = d.f_o_perm;
  a.o_rowslot = d.f_o_rowslot; a.o_fact = d.f_o_fact; a.o_ifact = d.f_o_ifact;
  a.tpc = t.tpc; a.list = d.flist; a.unit = (const int4 *)d.funit; a.rec = d.frec;
  a.perm = d.perm; a.rowslot = d.rowslot; a.fact = d.fact; a.ifact = d.ifact;
  a.S = (const double *)S; a.T = (double *)T; a.h = (double *)h;
  auto k = d.td == 2 ? (train ? k_bell_fwd64<2, true> : k_bell_fwd64<2, false>)
                     : (train ? k_bell_fwd64<1, true> : k_bell_fwd64<1, false>);
  CKT(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, d.f_smem));
  const int grid = grid_for((const void *)k, TWF * 32, d.f_smem, (long)npts * a.gy);
  LAUNCH("k_bell_fwd", st, (k<<<grid, TWF * 32, d.f_smem, st>>>(a)));
  CKT(cudaGetLastError());
  return RC_OK;
}

int bell_adj_tile64(const Tile64Dev &d, int n, int npts, const void *Tb, const void *h, void *Sb,
                    double *gbias, int gstride, cudaStream_t st) {
  if (!tile64_adj_applies(d, n)) return RC_UNSUPPORTED;
  Adj64Args a;
  a.n = n; a.na = d.na; a.npts = npts; a.gy = (n + NPB - 1) / NPB; a.gstride = gstride;
  a.nunit = d.naunit; a.nrec = d.narec; a.nfin = d.nafin; a.nzero = d.nzero;
  a.o_b1 = 2 * d.na * 128; a.o_scr = d.a_o_scr; a.o_zero = d.a_o_zero; a.o_list = d.a_o_list;
  a.o_unit = d.a_o_unit; a.o_rec = d.a_o_rec; a.o_flist = d.a_o_flist; a.o_fin = d.a_o_fin;
  a.o_perm = d.a_o_perm; a.o_rowslot = d.a_o_rowslot; a.o_fact = d.a_o_fact;
  a.o_ifact = d.a_o_ifact;
  a.list = d.alist; a.unit = (const int4 *)d.aunit; a.rec = (const uint2 *)d.arec;
  a.flist = d.aflist; a.fin = (const int4 *)d.afin; a.perm = d.perm; a.rowslot = d.rowslot;
  a.fact = d.fact; a.ifact = d.ifact; a.Tb = (const double *)Tb; a.h = (const double *)h;
  a.Sb = (double *)Sb; a.gbias = gbias;
  auto k = d.td == 2 ? k_bell_adj64<2> : k_bell_adj64<1>;
  CKT(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, d.a_smem));
  const int grid = grid_for((const void *)k, TWA * 32, d.a_smem, (long)npts * a.gy);
  LAUNCH("k_bell_adj", st, (k<<<grid, TWA * 32, d.a_smem, st>>>(a)));
  CKT(cudaGetLastError());
  return RC_OK;
}

}  // namespace dnnf90
