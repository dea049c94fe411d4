// The Cleanup phase's first checks, shared by their own kernel and by the small
// models' fused one.
#pragma once

#include "engine.cuh"

namespace gpp {

// What the first checks of the four cleanup rules find on the current plan, in
// one pass: a thread reads one column and one row and flags the rules that may
// act.
//  - fixed variables: a kept column whose finite bounds lie within bound_tol;
//  - empty columns: any kept empty column (fixed, infeasible or unbounded);
//  - empty rows: any kept row without live entries;
//  - singleton rows: a row that gives a bound, or, when there is none (the
//    candidate bounds are then the columns' own), a column whose bounds cross
//    by more than bound_tol or are NaN.
// Bound by its reads, 18 bytes a column and 6 a row; the four detection kernels
// of the rules, which also fill the arrays that the rules go on with, took 7
// launches and copies and about 230 bytes a column.
struct ProbeArgs {
  int m, n;
  uint32_t rules;
  const uint8_t *keep_row, *keep_col;
  const double *l, *u;
  const uint8_t* empty_col;
  const int32_t* row_nnz;
  const uint8_t* singleton_row;
  const int32_t* scol;
  const double* sval;
  double bound_tol, zero_tol;
  int32_t *sc_owner, *sc_words;   // the singleton-column rule's scratch, which it needs cleared
};
__device__ __forceinline__ uint32_t probe_part(const ProbeArgs& g) {
  uint32_t f = 0;
  const int top = g.n > g.m ? g.n : g.m;
  for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < top; k += gridDim.x * blockDim.x) {
    if (k < g.n) {
      const double lj = g.l[k], uj = g.u[k];
      if (g.keep_col[k]) {
        if (isfinite(lj) && isfinite(uj) && lj <= uj && uj - lj <= g.bound_tol) f |= kProbeFixed;
        if (g.empty_col[k]) f |= kProbeEmptyColumns;
      }
      if (lj > uj + g.bound_tol || lj != lj || uj != uj) f |= kProbeSingletonRows;
    }
    if (k < g.m) g.sc_owner[k] = kUnclaimedRow;
    if (k < g.m && g.keep_row[k]) {
      if (g.row_nnz[k] == 0) f |= kProbeEmptyRows;
      if (g.singleton_row[k]) {
        const int col = g.scol[k];
        if (col >= 0 && col < g.n && fabs(g.sval[k]) > g.zero_tol) f |= kProbeSingletonRows;
      }
    }
  }
  return f & g.rules;
}

}  // namespace gpp
