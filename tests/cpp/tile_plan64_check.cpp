// The FP64 tiled kernels' work lists (TilePlan with their warp counts,
// TileAdj64) on the CPU, in the kernels' loop order: every row a record,
// unit or scratch entry names lies inside its buffer, every output row is
// written once per item, and the forward and the adjoint reproduce the Bell
// recurrence's pair sums to 1e-12.  Built and run by tests/test_tile_plan64.py.
#include <cmath>
#include <cstdio>
#include <cstdint>
#include <random>
#include <vector>

#include "tables.hpp"
#include "tile_plan.hpp"
using namespace dnnf90;

static void untri(int td, int e, int &a1, int &a2) {
  a2 = 0;
  if (td == 1) { a1 = e; return; }
  int s = 0;
  while ((s + 1) * (s + 2) / 2 <= e) ++s;
  a2 = e - s * (s + 1) / 2;
  a1 = s - a2;
}
static int tri(int td, int a1, int a2) {
  return td == 1 ? a1 : (a1 + a2) * (a1 + a2 + 1) / 2 + a2;
}
#define NEED(c) do { if (!(c)) { printf("line %d: %s (d0=%d k=%d)\n", __LINE__, #c, d0, k); return 1; } } while (0)

static int check(int d0, int k) {
  TableSet t;
  if (!build_tables(d0, k, 0, nullptr, t).empty()) return 1;
  const int FW = TILE_WARPS64_F, AW = TILE_WARPS64_A, na = t.na;
  const TilePlan P = build_tile_plan(t, FW, AW);
  NEED(P.ok);
  const int td = P.td, z = tile_size(td, k + 1);
  const int maxscr = (227 * 1024 - 4 * na * 128 - z * 128 - na * 24 - 16 * 1024) / 128;
  std::vector<double> fact(na, 1.0);
  for (int ia = 0; ia < na; ++ia)
    for (int j = 0; j < d0; ++j)
      for (int v = 2; v <= t.alpha[ia * d0 + j]; ++v) fact[ia] *= v;
  std::mt19937_64 g(7 + d0 * 10 + k);
  std::normal_distribution<double> nd(0, 0.7);

  // forward: D chain over the units of every warp
  std::vector<double> S(na), sig(k + 2);
  for (auto &v : S) v = nd(g);
  for (auto &v : sig) v = nd(g);
  std::vector<double> st(na);
  for (int r = 0; r < na; ++r) st[r] = S[P.rowslot[r]] / fact[P.rowslot[r]];
  std::vector<double> buf[2] = {std::vector<double>(std::max(1, P.nbuf[0])),
                                std::vector<double>(std::max(1, P.nbuf[1]))};
  std::vector<double> T(na, 0.0);
  std::vector<int> wrote(na, 0);
  buf[k & 1][0] = sig[k];
  for (int q = k - 1; q >= 0; --q) {
    const auto &Dr = buf[(q + 1) & 1];
    auto &Dw = buf[q & 1];
    std::vector<double> out = Dw;
    for (int w = 0; w < FW; ++w)
      for (int u = P.flist[(q * FW + w) * 2]; u < P.flist[(q * FW + w) * 2] + P.flist[(q * FW + w) * 2 + 1]; ++u) {
        const int *U = &P.funit[4 * u];
        const int L = U[0] & 0xff, nt = tile_size(td, L);
        NEED(L >= 1 && L <= TILE_KMAX + 1);
        std::vector<double> acc(nt, 0.0);
        for (int i = 0; i < U[2]; ++i) {
          const uint32_t r = P.frec[U[1] + i];
          const int sr = r & 0xffff, dr = r >> 16, LD = i == 0 ? L - 1 : L;
          NEED(sr + nt <= na);
          NEED(LD == 0 || dr + tile_size(td, LD) <= (int)Dr.size());
          for (int c = 0; c < tile_size(td, LD); ++c)
            for (int e = i == 0 ? 1 : 0; e < nt; ++e) {
              int b1, b2, c1, c2;
              untri(td, e, b1, b2);
              untri(td, c, c1, c2);
              if (b1 + b2 + c1 + c2 <= L - 1) acc[tri(td, b1 + c1, b2 + c2)] += st[sr + e] * Dr[dr + c];
            }
        }
        for (auto &v : acc) v /= q + 1;
        if (U[0] >> 8) acc[0] = sig[q];
        for (int e = 0; e < nt; ++e) {
          if (q > 0) {
            NEED(U[3] + e < (int)out.size());
            out[U[3] + e] = acc[e];
          } else {
            NEED(U[3] + e < na);
            wrote[U[3] + e]++;
            T[U[3] + e] = fact[P.rowslot[U[3] + e]] * acc[e];
          }
        }
      }
    if (q > 0) Dw = out;
  }
  for (int r = 0; r < na; ++r) NEED(wrote[r] == 1);
  // the Faa di Bruno sum by powers: B_q = s~^q / q!
  auto find = [&](const std::vector<int> &a) { return t.find(a.data()); };
  std::vector<double> s(na), pw(na, 0.0), ref(na, 0.0);
  for (int a = 0; a < na; ++a) s[a] = a == 0 ? 0.0 : S[a] / fact[a];
  pw[0] = 1.0;
  std::vector<std::vector<int>> sub(na * 1);
  std::vector<int> al(d0);
  for (int q = 0; q <= k; ++q) {
    for (int a = 0; a < na; ++a) ref[a] += sig[q] * pw[a];
    std::vector<double> nx(na, 0.0);
    for (int a = 0; a < na; ++a)
      for (int b = 0; b < na; ++b) {
        bool le = true;
        for (int j = 0; j < d0; ++j) {
          al[j] = t.alpha[a * d0 + j] - t.alpha[b * d0 + j];
          if (al[j] < 0) le = false;
        }
        if (le && b) nx[a] += s[b] * pw[find(al)];
      }
    for (auto &v : nx) v /= q + 1;
    pw = nx;
  }
  double err = 0, mx = 0;
  for (int a = 0; a < na; ++a) {
    err = std::max(err, std::fabs(T[P.perm[a]] - fact[a] * ref[a]));
    mx = std::max(mx, std::fabs(fact[a] * ref[a]));
  }
  NEED(err <= 1e-12 * mx);

  // adjoint
  const TileAdj64 A = build_tile_adj64(t, P, AW, maxscr);
  NEED(A.ok && A.nscratch <= maxscr);
  std::vector<double> Tb(na), h(na), tb(na), hh(na), scr(std::max(1, A.nscratch), NAN), Sb(na, 0.0);
  for (auto &v : Tb) v = nd(g);
  for (auto &v : h) v = nd(g);
  for (int r = 0; r < na; ++r) {
    tb[r] = Tb[P.rowslot[r]] * fact[P.rowslot[r]];
    hh[r] = h[P.rowslot[r]] / fact[P.rowslot[r]];
  }
  std::fill(wrote.begin(), wrote.end(), 0);
  std::vector<int> wscr(A.nscratch, 0);
  int units = 0;
  for (int w = 0; w < AW; ++w)
    for (int u = A.list[2 * w]; u < A.list[2 * w] + A.list[2 * w + 1]; ++u, ++units) {
      const int *U = &A.unit[8 * u];
      const int lo = U[0] & 0xff, pair = U[0] >> 8 & 1, toscr = U[0] >> 9 & 1;
      NEED(lo >= 1 && lo <= TILE_KMAX + 1);
      std::vector<double> acc[2] = {std::vector<double>(z, 0.0), std::vector<double>(z, 0.0)};
      int i = U[1];
      for (int L = TILE_KMAX + 1; L >= 1; --L) {
        const int cnt = lo >= L ? (U[2] >> (4 * (lo - L))) & 15 : 0;
        for (int c = 0; c < cnt; ++c, ++i)
          for (int hf = 0; hf < 2; ++hf) {
            NEED(2 * i + hf < (int)A.rec.size());
            const uint32_t r = A.rec[2 * i + hf];
            const bool null = r & TILE_NULL;
            const int hr = r & (TILE_NULL - 1), tr = r >> 14 & 0x3fff, nt = tile_size(td, L);
            NEED((int)(r >> 28) == L && hr + nt <= na && tr + nt <= na && nt <= z);
            for (int a = 0; a < nt; ++a)
              for (int e = 0; e < nt; ++e) {
                int a1, a2, c1, c2;
                untri(td, a, a1, a2);
                untri(td, e, c1, c2);
                if (c1 <= a1 && c2 <= a2)
                  acc[hf][tri(td, a1 - c1, a2 - c2)] += tb[tr + a] * (null ? 0.0 : hh[hr + e]);
              }
          }
      }
      const int nt = tile_size(td, lo);
      for (int e = nt; e < z; ++e) NEED(acc[0][e] == 0.0 && acc[1][e] == 0.0);
      if (!pair) for (int e = 0; e < nt; ++e) acc[0][e] += acc[1][e];
      for (int hf = 0; hf < 1 + pair; ++hf)
        for (int e = 0; e < nt; ++e) {
          const int row = U[3 + hf] + e;
          if (toscr) {
            NEED(row < A.nscratch);
            scr[row] = acc[hf][e];
            wscr[row]++;
          } else {
            NEED(row < na);
            Sb[row] = acc[hf][e] / fact[P.rowslot[row]];
            wrote[row]++;
          }
        }
    }
  NEED(units == (int)A.unit.size() / 8);
  for (int r = 0; r < A.nscratch; ++r) NEED(wscr[r] == 1);
  int fins = 0;
  for (int w = 0; w < AW; ++w)
    for (int f = A.flist[2 * w]; f < A.flist[2 * w] + A.flist[2 * w + 1]; ++f, ++fins) {
      const int *F = &A.fin[4 * f];
      double v = 0;
      for (int p = 0; p < F[1]; ++p) {
        NEED(F[2] + p * F[3] < A.nscratch);
        v += scr[F[2] + p * F[3]];
      }
      NEED(F[0] < na);
      Sb[F[0]] = v / fact[P.rowslot[F[0]]];
      wrote[F[0]]++;
    }
  NEED(fins == (int)A.fin.size() / 4);
  for (int r = 0; r < na; ++r) NEED(wrote[r] == 1);
  err = mx = 0;
  for (int b = 0; b < na; ++b) {
    double v = 0;
    for (int p = t.pair_start[b]; p < t.pair_start[b] + t.pair_num[b]; ++p)
      v += Tb[t.pair_ia[p]] * t.pair_binom[p] * h[t.pair_id[p]];
    if (b == 0) {
      v = 0;
      for (int a = 0; a < na; ++a) v += Tb[a] * h[a];
    }
    err = std::max(err, std::fabs(v - Sb[P.perm[b]]));
    mx = std::max(mx, std::fabs(v));
  }
  NEED(err <= 1e-12 * mx);
  printf("d0=%d k=%d na=%d units %d steps %zu fma %ld scratch %d\n", d0, k, na, units,
         A.rec.size() / 2, A.steps_fma, A.nscratch);
  return 0;
}

int main() {
  int bad = 0;
  for (int d0 = 1; d0 <= 4; ++d0)
    for (int k = 1; k <= TILE_KMAX; ++k) bad += check(d0, k);
  printf(bad ? "FAILED\n" : "ALL OK\n");
  return bad ? 1 : 0;
}
