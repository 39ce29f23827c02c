// The FP64 complex product C = A B shared by its two forms: the FP64 tensor cores (epb_f64gemm.cu) and 8-bit digits
// on the integer tensor cores (epb_f64oz.cu).
#pragma once

#include "epb_common.cuh"

namespace epb {

constexpr int GT_MAX = 16;      // max per-axis extent of R handled by the phase tables
constexpr int GK_MAX = 4096;    // max R vectors whose table indices are kept in shared memory

// B is a matrix; the phase from per-axis tables; the phase evaluated directly (R lists too wide for tables).
enum { B_MATRIX = 0, B_TABLE = 1, B_DIRECT = 2 };

struct F64GemmArgs {
  const double2* A;    // column-major, leading dimension lda
  int64_t lda, M, K, N;
  const double2* B;    // K x N matrix, leading dimension ldb (matrix form)
  int64_t ldb;
  const int4* rv;      // K lattice vectors and 3 x N points (phase form)
  const double* xk;
  double2* C;          // leading dimension ldc
  int64_t ldc;
  int lo0, lo1, lo2, L0, L1, L2;
  bool serial;         // one chain of FMAs over K per output (no split of K, no digits)
  int tri_n;           // > 0: A is a stack of tri_n x tri_n matrices, its rows run over i <= j only (M of them)
};

bool oz_pays(epb_ctx* ctx, const F64GemmArgs& a);
int oz_gemm(epb_ctx* ctx, const F64GemmArgs& a, int mode);
int f64_gemm_guarded(epb_ctx* ctx, const F64GemmArgs& a, int mode, const int* words);

}  // namespace epb
