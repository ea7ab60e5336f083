// Launch interface of the sTDDFT ("std") tensor kernels (k_std.cu).
#pragma once

#include "pa_internal.h"

namespace pa {

struct StdArgs {
  DevBasis B;                        // orbital basis
  DevBasis X;                        // auxiliary basis
  DeviceTables dt;
  int boys_mode = 1;
  double thresh = 0.0;               // Schwarz threshold on Q_ab * Q_c
  const int2* pair_ab = nullptr;     // pair -> (a, b), a >= b
  const int* pair_unit0 = nullptr;   // pair -> first bra unit
  const double4* unit_pP = nullptr;  // unit -> (p, P)
  const double* esph = nullptr;      // E_sph blocks
  const long long* unit_esph = nullptr;
  const double* Qab = nullptr;       // pair -> Schwarz value
  const double* Qc = nullptr;        // aux shell -> Schwarz value
};

// Layout of the block matrix (k_std.cu): Schwarz values of the class-ordered
// pairs, rows of the sorted pairs and their number, columns of the sorted
// auxiliary shells.
int launch_std_pair_keys(int n, const int* class_pair, const double* Qab, double* keys, int* vals, cudaStream_t s);
int launch_std_pair_size(const StdArgs& a, int n, const double* Q, const int* pair, const int* off, int nseg,
                         const double* qmax, int* size, int* nclass, cudaStream_t s);
int launch_std_pair_row(int n, const int* pair, const int* size, const int* first, int* row0, int* total,
                        cudaStream_t s);
int launch_std_columns(int n, const int* sorted, const double* Q, const int* off, int nseg, const int4* shell,
                       int* col_fn, double* col_Q, cudaStream_t s);

// fn_shell[nu] = shell of orbital function nu; Ct[nu * pld + p] = C[nu, p]
// (zero for nmos <= p < pld). mo is C (nbf x nmos, column-major).
int launch_std_orbitals(const DevBasis& B, const double* mo, int nmos, int pld, int* fn_shell, double* Ct,
                        cudaStream_t s);

// First half-transformation of intor_df2c_mo (std/intor.f90:207-261) over the
// block matrix I of nk auxiliary columns (ld even, >= nk):
// W[(nu * nmos + p) * ld + k] = sum_a skip(sum_(i in a) C[i, p] (i nu|k)).
struct StdHalfArgs {
  DevBasis B;
  const double* Qab = nullptr;
  const int* row0 = nullptr;      // pair -> first row of I, -1: none
  const int* fn_shell = nullptr;
  const double* col_Q = nullptr;  // Schwarz value of each of the nk columns
  double thresh = 0.0;
  const double* I = nullptr;
  const double* Ct = nullptr;
  int nk = 0, ld = 0, pld = 0, nmos = 0;  // pld: multiple of 16 std_half_pt(nmos)
  double* W = nullptr;
};
int std_half_pt(int nmos);
int launch_std_half(const StdHalfArgs& h, cudaStream_t s);

// Raw[col_fn[k] + naux * (p(p+1)/2 + q)] = Res[k + ld * (p + nmos * q)], k < nk, q <= p.
int launch_std_pack(const double* Res, int nk, int ld, int nmos, const int* col_fn, int naux, double* Raw,
                    cudaStream_t s);

// out[kp * nshells_aux + c] = ||(ab|c)||_2 for pair rec_pair[kp] (kp < npairs)
// and every auxiliary shell c.
int launch_std_block_norms(const StdArgs& a, const int* rec_pair, int npairs, double* out, cudaStream_t s);

// out[i + rows * j] = in[j + cols * i] (out: rows x cols, column-major).
int launch_transpose(const double* in, int rows, int cols, double* out, cudaStream_t s);

}  // namespace pa
