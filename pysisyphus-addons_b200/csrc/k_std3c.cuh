// Launch interface of the explicit three-center blocks of the std tensors
// (k_std3c_impl.cuh, one translation unit per LAB).
#pragma once

#include "k_df3c.cuh"

namespace pa {

// Arguments of one class (LAB, LC) launch.
struct Std3cArgs {
  Df3cArgs x;                        // auxiliary basis, tables, Boys mode, Schwarz threshold
  DevBasis B;                        // orbital basis
  const int* bra = nullptr;          // class's shell pairs (diag: its shells), n_bra of them
  int n_bra = 0;
  const int2* pair_ab = nullptr;
  const int* pair_unit0 = nullptr;   // pair -> first primitive pair
  const double4* unit_pP = nullptr;
  const double* esph = nullptr;
  const long long* unit_esph = nullptr;
  const double* Qab = nullptr;       // pair -> Schwarz value
  const int* aux = nullptr;          // class's auxiliary shells of this launch, n_aux of them
  int n_aux = 0;
  const double* Qc = nullptr;        // auxiliary shell -> Schwarz value
  // Integral (r of pair q | function m of auxiliary shell i of the launch) goes
  // to out[(row0[q] + r) * ld + col0 + i * (2 LC + 1) + m]; with diag, (i i|P)
  // of shell pair (a, a) goes to out[(first function of a + i) * ld + P].
  const int* row0 = nullptr;
  int col0 = 0;
  int diag = 0;
  long long ld = 0;
  double* out = nullptr;
};

int launch_std3c_class(int lab, int lc, const Std3cArgs& a, cudaStream_t s);

struct Std3cRow {
  using LaunchFn = int (*)(const Std3cArgs&, cudaStream_t);
  LaunchFn launch[PA_LAUXMAX + 1] = {};
  cudaError_t (*upload_rownorm)(const double*, cudaStream_t) = nullptr;
};
void std3c_row_0(Std3cRow*);
void std3c_row_1(Std3cRow*);
void std3c_row_2(Std3cRow*);
void std3c_row_3(Std3cRow*);
void std3c_row_4(Std3cRow*);
void std3c_row_5(Std3cRow*);
void std3c_row_6(Std3cRow*);
void std3c_row_7(Std3cRow*);
void std3c_row_8(Std3cRow*);
// Row normalization of the solid harmonics (constant memory of every class
// translation unit).
cudaError_t upload_std3c_rownorm(const double* rownorm, cudaStream_t s);

}  // namespace pa
