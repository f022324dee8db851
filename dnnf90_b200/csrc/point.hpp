// point.hpp - the whole step of small networks in one launch (point.cu).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "bell_col.hpp"
#include "tables.hpp"

namespace dnnf90 {

struct DevTables;
struct DevNet;
struct DevRule;
struct BatchArgs;

// device copy of the pair lists (ColProg) and of the slots' exponents
struct PointDev {
  bool ok = false;
  int2 *fhdr = nullptr, *ahdr = nullptr;
  uint32_t *frec = nullptr, *arec = nullptr, *ex = nullptr;
  short *dn = nullptr;
};
bool point_set(const TableSet &t);  // the sets it takes
void upload_point(const TableSet &t, const ColProg &p, PointDev &d, PlanBlock &b);

// whether one launch serves the batch, and the launch: the same results as
// run_batch, with no plane in device memory
bool point_applies(const DevTables &t, const DevNet &net, const DevRule &rule, int npts,
                   bool train, int prec);
int run_point(const DevTables &t, const DevNet &net, const DevRule &rule, const BatchArgs &b,
              cudaStream_t st);

}  // namespace dnnf90
