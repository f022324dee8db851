// bell_col.hpp - Bell kernels of small carried sets and the analytic
// first-layer adjoint (see bell_col.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "plan_block.hpp"
#include "tables.hpp"

namespace dnnf90 {

struct DevTables;
struct L2Analytic;

// device copy of the column kernels' program (host form: ColProg)
struct ColDev {
  bool ok = false;
  int na = 0, kt = 0, nfrec = 0, narec = 0;
  int *fhdr = nullptr, *ahdr = nullptr;      // [na][2]: first record, records
  uint32_t *frec = nullptr, *arec = nullptr;
  int *dstart = nullptr;                     // [kt + 2]: first slot of each degree
};

// The pair lists of a downward-closed set, per output slot.  Forward: the
// pairs (b, a - b), b != 0, of output a.  Adjoint: the pairs (b + g, g) of
// output b.  Records are x | y << 16; every list starts at an even index.
struct ColProg {
  int kt = 0;                                // top degree of the set
  std::vector<int> fhdr, ahdr, dstart;
  std::vector<uint32_t> frec, arec;
};
ColProg build_col_prog(const TableSet &t);
// whether a set is one of the column kernels'
bool col_set(const TableSet &t);
void upload_col(const TableSet &t, const ColProg &p, ColDev &d, PlanBlock &b);

// whether the column kernels can run on this set, and whether they are the
// faster ones for npts points of n neurons
bool col_fits(const ColDev &d, int n, int prec);
bool col_applies(const ColDev &d, int n, int npts, int prec);
int bell_fwd_col(const ColDev &d, const DevTables &t, int n, int npts, const void *S, void *T,
                 void *h, bool train, int prec, cudaStream_t st);
int bell_adj_col(const ColDev &d, const DevTables &t, int n, int npts, const void *Tb,
                 const void *h, void *Sb, double *gbias, int gstride, int prec,
                 cudaStream_t st);

// The first hidden layer's adjoint fused with dW_2, h formed from the s^(q)
// the forward kept; l2a_applies tells for which shapes (graded slots).
bool l2a_applies(int d0, int na, int n, int prec);
int bell_adj_l2a(const DevTables &t, int n, int npts, const void *Tb, const double *X, double *g,
                 double *rows, size_t nw, size_t woff, int prec, const L2Analytic &an,
                 cudaStream_t st);

}  // namespace dnnf90
