// Dense FP64 linear algebra of the density-fitting path (column-major):
//  * blocked right-looking Cholesky of the metric, lower triangle
//    (replaces dpotrf("L"), common/linalg.f90:78); one launch per 64 columns takes
//    the panel and the next diagonal block with its inverse, another the
//    trailing matrix beside the next step;
//  * L^-1 df as a blocked forward substitution on the density columns, using
//    the inverted diagonal blocks (replaces dtrtri("L","N"), common/linalg.f90:81,
//    followed by dtrmm("L","L","N","N"), diabatization/intor.f90:198: the
//    explicit inverse is never formed);
//  * a tiled FP64 GEMM C := beta C + alpha op(A) op(B) on the FP64 tensor
//    cores, used by the sTDDFT tensors and by the Gram matrix of the Coulomb
//    tensor for many densities;
//  * the 8-fold-symmetric scatter of the Coulomb tensor
//    (diabatization/intor.f90:241-269).
#include <algorithm>

#include "k_linalg.cuh"

#include <cstdint>
#include <type_traits>

namespace pa {

namespace {

constexpr int NB = 64;

__device__ __forceinline__ void dmma_m8n8k4(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

__device__ __forceinline__ void cp_async8(double* smem_dst, const double* gmem_src) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(gmem_src));
}

__device__ __forceinline__ void cp_async16_ld(double* smem_dst, const double* gmem_src) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(smem_dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(gmem_src));
}

// Cholesky factor of the 64 x 64 block S (lower triangle) in
// place, its inverse in X (undefined right of its 32 x 32 diagonal blocks), T scratch; all 256
// threads, S complete on entry (after a barrier). Rows and columns from nb on
// hold the identity. The serial chain is kept short: per pivot one reciprocal
// square root (CUDA's; the roots follow after it, one per lane), per 16-column
// sub-block
//  * warp 0 factors the 16 x 16 diagonal sub-block (lane r holds row r, pivots
//    and L(j, k) move by shuffles; two columns per link of the chain, through
//    the 2 x 2 determinant, was slower: more dependent FP64 operations);
//  * one thread per row below solves x L11^T = a in registers;
//  * the trailing lower triangle is updated on the FP64 tensor cores.
// Inverse: four warps invert the diagonal sub-blocks (lane c holds column c,
// right-looking, so a row's updates are independent), then the off-diagonal
// blocks follow by doubling: X_21 = -X_22 (L_21 X_11) at 16 and at 32 columns,
// on the FP64 tensor cores as well.
constexpr int SB = 16;
constexpr int kPanLd = NB + 4;  // 4 (mod 16): conflict-free m8n8k4 fragment loads

__device__ __forceinline__ void factor_invert_64(double (*S)[kPanLd], double (*X)[kPanLd], double (*T)[kPanLd],
                                                 double* invd, int nb, int pivot0, int* info) {
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t4 = lane & 3;
  for (int k0 = 0; k0 < NB; k0 += SB) {
    if (warp == 0) {
      // lanes 16..31 repeat lanes 0..15 (they only feed the shuffles)
      const int r = lane & (SB - 1);
      // row r and, apart from it, its diagonal element: the next pivot then
      // needs no shuffle but its own. No branches on r: they cost a third of the time
      double v[SB], dg = S[k0 + r][k0 + r];
      int bad = -1;  // first non-positive pivot
#pragma unroll
      for (int j = 0; j < SB; ++j) v[j] = (j < r) ? S[k0 + r][k0 + j] : 0.0;
#pragma unroll
      for (int k = 0; k < SB; ++k) {
        double dkk = __shfl_sync(0xffffffffu, dg, k);
        const bool ok = dkk > 0.0;
        bad = (!ok && bad < 0) ? k : bad;
        dkk = ok ? dkk : 1.0;  // keep the factor finite; the error is reported through info
        const double id = rsqrt(dkk);
        const double l = v[k] * id;  // L(r, k) of the rows below
        v[k] = r > k ? l : v[k];
        const double g2 = fma(-l, l, dg);
        dg = r > k ? g2 : dg;
#pragma unroll
        for (int j = 1; j < SB; ++j) {  // fixed trip count: j > k folds once k is unrolled
          if (j <= k) continue;
          const double ljk = __shfl_sync(0xffffffffu, v[k], j);  // L(j, k) from lane j
          const double u = fma(-v[k], ljk, v[j]);
          v[j] = r > j ? u : v[j];
        }
        if (lane == k) invd[k0 + k] = id;
      }
      if (lane == 0 && bad >= 0 && k0 + bad < nb) atomicCAS(info, 0, pivot0 + k0 + bad + 1);
      if (lane < SB) {
#pragma unroll
        for (int j = 0; j < SB; ++j)
          if (j < r) S[k0 + r][k0 + j] = v[j];
        S[k0 + r][k0 + r] = sqrt(dg > 0.0 ? dg : 1.0);  // dg has stayed this row's pivot
      }
    }
    __syncthreads();
    // panel rows below: x L11^T = a, right-looking in registers, one thread per row
    const int pr = k0 + SB + tid;
    if (pr < NB) {
      double v[SB];
#pragma unroll
      for (int j = 0; j < SB; ++j) v[j] = S[pr][k0 + j];
#pragma unroll
      for (int j = 0; j < SB; ++j) {
        v[j] *= invd[k0 + j];
#pragma unroll
        for (int jj = 1; jj < SB; ++jj)
          if (jj > j) v[jj] = fma(-v[j], S[k0 + jj][k0 + j], v[jj]);
      }
#pragma unroll
      for (int j = 0; j < SB; ++j) S[pr][k0 + j] = v[j];
    }
    __syncthreads();
    // trailing lower triangle: S -= P P^T of the sub-block's columns P, one 8 x 8
    // tile per warp and turn
    const int m8 = (NB - k0 - SB) / 8, tiles = m8 * (m8 + 1) / 2;  // 8-row tiles, at most 21
    if (tiles == 0) break;
    int tr[3], tc[3];
    double d[3][2];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
      const int t = warp + 8 * q;
      const int bi = (t >= 1) + (t >= 3) + (t >= 6) + (t >= 10) + (t >= 15);
      tr[q] = k0 + SB + 8 * bi + g;
      tc[q] = k0 + SB + 8 * (t - bi * (bi + 1) / 2);
      d[q][0] = d[q][1] = 0.0;
    }
#pragma unroll
    for (int k = 0; k < SB; k += 4)
#pragma unroll
      for (int q = 0; q < 3; ++q)
        if (warp + 8 * q < tiles) dmma_m8n8k4(d[q][0], d[q][1], S[tr[q]][k0 + k + t4], S[tc[q] + g][k0 + k + t4]);
#pragma unroll
    for (int q = 0; q < 3; ++q)
      if (warp + 8 * q < tiles) {
        S[tr[q]][tc[q] + 2 * t4] -= d[q][0];
        S[tr[q]][tc[q] + 2 * t4 + 1] -= d[q][1];
      }
    __syncthreads();
  }
  if (warp < NB / SB) {
    const int o = warp * SB, c = lane & (SB - 1);
    double x[SB];
#pragma unroll
    for (int i = 0; i < SB; ++i) x[i] = (i == c) ? 1.0 : 0.0;
#pragma unroll
    for (int i = 0; i < SB; ++i) {
      x[i] *= invd[o + i];
#pragma unroll
      for (int k = 1; k < SB; ++k)
        if (k > i) x[k] = fma(-S[o + k][o + i], x[i], x[k]);
    }
    if (lane < SB) {
#pragma unroll
      for (int i = 0; i < SB; ++i) {
        X[o + i][o + c] = i >= c ? x[i] : 0.0;
        if (warp % 2 == 0) X[o + i][o + SB + c] = 0.0;  // right of it: read as part of the 32-column block
      }
    }
  }
  __syncthreads();
  // doubling: blocks of w columns, T = L_21 X_11, then X_21 = -X_22 T, 8 x 8
  // tiles over the warps
  auto level = [&](auto wc) {
    constexpr int w = decltype(wc)::value;
    constexpr int turns = (NB / (2 * w)) * (w / 8) * (w / 8) / 8;
    int o[turns], i[turns], j[turns];
#pragma unroll
    for (int t = 0; t < turns; ++t) {
      const int id = warp + 8 * t;
      o[t] = id / ((w / 8) * (w / 8)) * 2 * w;
      i[t] = o[t] + w + id / (w / 8) % (w / 8) * 8 + g;
      j[t] = id % (w / 8) * 8;
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
      double d[turns][2][2] = {};  // per tile two chains of products
#pragma unroll
      for (int k = 0; k < w; k += 4)
#pragma unroll
        for (int t = 0; t < turns; ++t) {
          const double a = half == 0 ? S[i[t]][o[t] + k + t4] : X[i[t]][o[t] + w + k + t4];
          const double b = half == 0 ? X[o[t] + k + t4][o[t] + j[t] + g] : T[o[t] + w + k + t4][j[t] + g];
          dmma_m8n8k4(d[t][k / 4 & 1][0], d[t][k / 4 & 1][1], a, b);
        }
#pragma unroll
      for (int t = 0; t < turns; ++t)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const double v = d[t][0][e] + d[t][1][e];
          if (half == 0)
            T[i[t]][j[t] + 2 * t4 + e] = v;
          else
            X[i[t]][o[t] + j[t] + 2 * t4 + e] = -v;
        }
      __syncthreads();
    }
  };
  level(std::integral_constant<int, SB>{});
  level(std::integral_constant<int, 2 * SB>{});
}

// acc += A^T-layout tile product over [0, kq): As[k][row], Bs[k][col] with row
// stride kPanLd; warp w owns rows 16 (w % 4) and columns 32 (w / 4).
__device__ __forceinline__ void panel_mma(double (&acc)[2][4][2], const double* As, const double* Bs, int kq) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int wm = (warp & 3) * 16, wn = (warp >> 2) * 32;
#pragma unroll 4
  for (int q = 0; q < kq; q += 4) {
    double a[2], b[4];
#pragma unroll
    for (int mt = 0; mt < 2; ++mt) a[mt] = As[(q + t4) * kPanLd + wm + 8 * mt + g];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) b[nt] = Bs[(q + t4) * kPanLd + wn + 8 * nt + g];
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) dmma_m8n8k4(acc[mt][nt][0], acc[mt][nt][1], a[mt], b[nt]);
  }
}

// One step of the blocked Cholesky factorization: the panel of block column c,
// and (block 0) the next diagonal block. Block x owns row block i = c + 1 + x:
//   P(i, c) = (A(i, c) - P(i, c - 1) P(c, c - 1)^T) L(c, c)^-T,
// and for i = c + 1 then
//   A(i, i) -= P(i, c - 1) P(i, c - 1)^T + P(i, c) P(i, c)^T, factor, inverse.
// The contributions of columns below c - 1 came from the trailing updates
// (k_syrk_update), which leave out what this kernel takes itself: the next
// block column and the diagonal block after it. So the chain from one
// diagonal block to the next is one launch, and the trailing update of a step
// runs beside the next step. c = -1: the first diagonal block alone.
//
// Bound: latency of block 0's path, four 64^3 products on one SM (13 thousand
// cycles) and the factor with its inverse (25 us alone; 27 with a reciprocal root
// written out here and the roots on the chain). With the trailing update beside the
// next step 30 us a step at n = 448, 33 us at 2240 and 36 us at 3360; in one
// stream, step, update, step, 33, 41 and 47 us. With a launch each for the factor
// (40 us), the panel and the next column's update it was ~100 us.
constexpr size_t kCholSmem = sizeof(double) * 3 * NB * kPanLd;
__global__ void __launch_bounds__(256, 2) k_chol_step(double* A, long long lda, int n, int c, double* dinv,
                                                      int* info) {
  extern __shared__ __align__(16) double csm[];
  double* As = csm;                    // [p][r] P(i, c - 1), later the inverse
  double* Bs = As + NB * kPanLd;       // [p][r] P(c, c - 1), later [p][r] of the updated A(i, c), then S
  double* Ds = Bs + NB * kPanLd;       // [p][j] L(c, c)^-1, later [p][r] P(i, c), then scratch
  __shared__ double invd[NB];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int wm = (warp & 3) * 16, wn = (warp >> 2) * 32;
  const int i = c + 1 + blockIdx.x, r0 = i * NB, nr = min(NB, n - r0);
  const bool diag = blockIdx.x == 0;
  if (c >= 0) {
    const double* dc = dinv + static_cast<size_t>(c) * NB * NB;
    for (int idx = tid; idx < NB * NB; idx += 256) {
      const int r = idx & (NB - 1), p = idx >> 6;
      if (c > 0) {
        const double* col = A + lda * ((c - 1) * NB + p);
        if (r < nr)
          cp_async8(As + p * kPanLd + r, col + r0 + r);
        else
          As[p * kPanLd + r] = 0.0;
        cp_async8(Bs + p * kPanLd + r, col + c * NB + r);
      }
      cp_async8(Ds + p * kPanLd + r, dc + r + NB * p);
    }
    asm volatile("cp.async.commit_group;\n" ::);
  }
  // this thread's entries of A(i, c), in flight with the copies
  double cv[2][4][2];
  double* Ac = A + r0 + lda * (static_cast<long long>(c) * NB);
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = wm + 8 * mt + g, j = wn + 8 * nt + 2 * t4 + e;
        cv[mt][nt][e] = (c >= 0 && r < nr) ? Ac[r + lda * j] : 0.0;
      }
  // block 0: its entries of the next diagonal block (rows past n: identity)
  double* Ai = A + r0 + lda * static_cast<long long>(r0);
  double dv[2][4][2];
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = wm + 8 * mt + g, j = wn + 8 * nt + 2 * t4 + e;
        dv[mt][nt][e] = (diag && r < nr && j <= r) ? Ai[r + lda * j] : (r == j ? 1.0 : 0.0);
      }
  double acc[2][4][2];
  auto clear = [&] {
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) acc[mt][nt][0] = acc[mt][nt][1] = 0.0;
  };
  if (c >= 0) {
    asm volatile("cp.async.wait_group 0;\n" ::);
    __syncthreads();
    if (c > 0) {
      clear();
      panel_mma(acc, As, Bs, NB);
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt)
#pragma unroll
          for (int e = 0; e < 2; ++e) cv[mt][nt][e] -= acc[mt][nt][e];
      __syncthreads();  // Bs is rewritten
    }
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e) Bs[(wn + 8 * nt + 2 * t4 + e) * kPanLd + wm + 8 * mt + g] = cv[mt][nt][e];
    __syncthreads();
    clear();
    panel_mma(acc, Bs, Ds, wn + 32);  // row j of the inverse ends at column j
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const int r = wm + 8 * mt + g, j = wn + 8 * nt + 2 * t4 + e;
          if (r < nr) Ac[r + lda * j] = acc[mt][nt][e];
        }
    if (!diag) return;
    __syncthreads();  // Bs and Ds are rewritten
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e)
          Ds[(wn + 8 * nt + 2 * t4 + e) * kPanLd + wm + 8 * mt + g] = acc[mt][nt][e];
  }
  // the next diagonal block
  __syncthreads();
  for (int term = 0; term < 2; ++term) {  // columns c - 1, then c
    if (c < 1 - term) continue;
    clear();
    if (wm + 15 >= wn) panel_mma(acc, term == 0 ? As : Ds, term == 0 ? As : Ds, NB);
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int nt = 0; nt < 4; ++nt)
#pragma unroll
        for (int e = 0; e < 2; ++e) dv[mt][nt][e] -= acc[mt][nt][e];
  }
  double(*S)[kPanLd] = reinterpret_cast<double(*)[kPanLd]>(Bs);
  double(*X)[kPanLd] = reinterpret_cast<double(*)[kPanLd]>(As);
  double(*T)[kPanLd] = reinterpret_cast<double(*)[kPanLd]>(Ds);
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int r = wm + 8 * mt + g, j = wn + 8 * nt + 2 * t4 + e;
        S[r][j] = j <= r ? dv[mt][nt][e] : 0.0;
      }
  __syncthreads();  // As and Ds are free as well
  factor_invert_64(S, X, T, invd, nr, r0, info);
  double* di = dinv + static_cast<size_t>(i) * NB * NB;
  for (int q = 0; q < NB * NB / 256; ++q) {  // a warp's 8 x 4 pieces: no bank conflicts, 64 contiguous bytes
    const int r = 8 * warp + g, j = 4 * q + t4;
    if (r < nr && j <= r) Ai[r + lda * j] = S[r][j];
    di[r + NB * j] = (r < nr && j <= r) ? X[r][j] : 0.0;
  }
}

// One launch of the blocked forward substitution X = L^-1 B over R 64-row
// blocks of L from row k0 (a super-step). Two kinds of blocks, 8 warps each:
//  * the first nsolve blocks, one per 8 columns of B: apply X of the previous
//    super-step to the rows of this one, then solve them 64 at a time with the
//    inverted diagonal blocks, X_j = Dinv_j (B_j - sum_(l < j) L_jl X_l);
//  * the others, one per 64 rows below and 8 NT columns: B -= L X of the previous
//    super-step.
// So a super-step is one launch, its serial part overlaps the update below it,
// and nothing is solved twice. Products on the FP64 tensor cores (mma.sync
// m8n8k4): warp w owns rows 8 w.. of a 64-row block and reads its L fragments
// straight from global memory (8 rows = 64 contiguous bytes), ahead of the
// barriers that guard X, which is shared through shared memory.
//
// Bound: for few columns the solving blocks' chain of loads and barriers, so
// R = 2 with every fragment of a step in registers (one block per SM); for many
// the FP64 tensor pipe, so R = 4 (half the passes over B, two blocks per SM).
// Measured (n = 2240 / 3360, R = 2 against 4): 64 columns 213 against 223 / 321
// against 338 us, 128: 214, 227 / 382, 385, 192: 248, 235 / 456, 426, 1000: 699,
// 391 / 1534, 802.
constexpr int kTrsmFew = 128;
constexpr int kTrsmLdx = 12;  // 4 or 12 (mod 16): conflict-free fragment loads
constexpr size_t trsm_smem(int nt, int nblk) {
  return sizeof(double) * std::max(nblk * NB * (8 * nt + 4), nblk * NB * kTrsmLdx + 2 * NB * kTrsmLdx);
}

template <int NT, int R>
__global__ void __launch_bounds__(256, R == 2 ? 1 : 2) k_trsm_step(const double* __restrict__ L, long long lda, int n,
                                                                   int k0, const double* __restrict__ dinv, double* B,
                                                                   long long ldb, int nrhs, double* C, long long ldc,
                                                                   int nsolve) {
  extern __shared__ __align__(16) double tsm[];
  constexpr int kRows = R * NB, kQ = NB / 4;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int kp = k0 - kRows;  // rows of the previous super-step (all below n)
  if (static_cast<int>(blockIdx.x) < nsolve) {
    double* Xp = tsm;                        // [k][col] X of the previous super-step
    double* T = Xp + kRows * kTrsmLdx;       // [row][col] right-hand side of one block
    double* Xn = T + NB * kTrsmLdx;          // [row][col] its solution
    const int c0 = blockIdx.x * 8, row0 = k0 + 8 * warp + g;
    double bv[R][2], acc[R][2];
#pragma unroll
    for (int j = 0; j < R; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int row = row0 + NB * j, col = c0 + 2 * t4 + e;
        bv[j][e] = (row < n && col < nrhs) ? B[row + ldb * col] : 0.0;
        acc[j][e] = 0.0;
      }
    if (kp >= 0) {
      // fragments of 64 columns of L at a time, the next ones in flight while
      // the current ones are multiplied
      const double* l = L + row0 + lda * (kp + t4);
      double a[2][R][kQ];
      auto fetch = [&](int h, double (&f)[R][kQ]) {
#pragma unroll
        for (int j = 0; j < R; ++j)
#pragma unroll
          for (int q = 0; q < kQ; ++q) f[j][q] = row0 + NB * j < n ? l[NB * j + lda * (NB * h + 4 * q)] : 0.0;
      };
      if constexpr (R == 2) fetch(0, a[0]);
      for (int idx = tid; idx < kRows * 8; idx += 256) {
        const int r = idx & (kRows - 1), c = idx / kRows;
        Xp[r * kTrsmLdx + c] = c0 + c < nrhs ? C[(kp + r) + ldc * (c0 + c)] : 0.0;
      }
      __syncthreads();
      if constexpr (R == 2) {
        double part[R][4][2] = {};  // independent chains of products
#pragma unroll
        for (int h = 0; h < R; ++h) {
          if (h + 1 < R) fetch(h + 1, a[(h + 1) & 1]);
#pragma unroll
          for (int q = 0; q < kQ; ++q) {
            const double b = Xp[(NB * h + 4 * q + t4) * kTrsmLdx + g];
#pragma unroll
            for (int j = 0; j < R; ++j) dmma_m8n8k4(part[j][q & 3][0], part[j][q & 3][1], a[h & 1][j][q], b);
          }
        }
#pragma unroll
        for (int j = 0; j < R; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) acc[j][e] = (part[j][0][e] + part[j][1][e]) + (part[j][2][e] + part[j][3][e]);
      } else {
#pragma unroll 8
        for (int k = 0; k < kRows; k += 4) {
          const double b = Xp[(k + t4) * kTrsmLdx + g];
#pragma unroll
          for (int j = 0; j < R; ++j)
            dmma_m8n8k4(acc[j][0], acc[j][1], row0 + NB * j < n ? l[NB * j + lda * k] : 0.0, b);
        }
      }
    }
#pragma unroll
    for (int j = 0; j < R; ++j) {
      if (k0 + NB * j >= n) break;
      const int row = row0 + NB * j;
      const bool rowok = row < n;
      // Dinv_j and the tile of L that the next block waits for, before the barrier
      const double* dj = dinv + static_cast<size_t>(k0 / NB + j) * NB * NB + 8 * warp + g;
      const double* l = L + row0 + lda * (k0 + NB * j + t4);
      double da[kQ], ln[kQ];
#pragma unroll
      for (int q = 0; q < kQ; ++q) da[q] = 4 * q < 8 * (warp + 1) ? dj[NB * (4 * q + t4)] : 0.0;
      if (j + 1 < R)
#pragma unroll
        for (int q = 0; q < kQ; ++q) ln[q] = row + NB < n ? l[NB * (j + 1) + lda * (4 * q)] : 0.0;
#pragma unroll
      for (int e = 0; e < 2; ++e) T[(8 * warp + g) * kTrsmLdx + 2 * t4 + e] = rowok ? bv[j][e] - acc[j][e] : 0.0;
      __syncthreads();
      double x[4][2] = {};  // independent chains of products
#pragma unroll
      for (int q = 0; q < kQ; ++q)  // columns past the warp's rows of Dinv are zero
        if (4 * q < 8 * (warp + 1)) dmma_m8n8k4(x[q & 3][0], x[q & 3][1], da[q], T[(4 * q + t4) * kTrsmLdx + g]);
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const double v = (x[0][e] + x[1][e]) + (x[2][e] + x[3][e]);
        const int col = c0 + 2 * t4 + e;
        Xn[(8 * warp + g) * kTrsmLdx + 2 * t4 + e] = v;
        if (rowok && col < nrhs) C[row + ldc * col] = v;
      }
      if (j + 1 >= R) break;
      __syncthreads();
      double y[4][2] = {};
#pragma unroll
      for (int q = 0; q < kQ; ++q)
        dmma_m8n8k4(y[q & 3][0], y[q & 3][1], ln[q], Xn[(4 * q + t4) * kTrsmLdx + g]);
#pragma unroll
      for (int e = 0; e < 2; ++e) acc[(j + 1) % R][e] += (y[0][e] + y[1][e]) + (y[2][e] + y[3][e]);
      if constexpr (R > 2) {
#pragma unroll 4
        for (int k = 0; k < NB; k += 4) {
          const double b = Xn[(k + t4) * kTrsmLdx + g];
#pragma unroll
          for (int q = 2; q < R; ++q) {
            if (q <= j + 1) continue;
            dmma_m8n8k4(acc[q][0], acc[q][1], row0 + NB * q < n ? l[NB * q + lda * k] : 0.0, b);
          }
        }
      }
    }
    return;
  }
  constexpr int kLd = 8 * NT + 4;
  double* Xs = tsm;  // [k][col]
  const int r1 = k0 + kRows, nrow = (n - r1 + NB - 1) / NB;
  const int blk = blockIdx.x - nsolve, c0 = (blk / nrow) * 8 * NT;
  const int row = r1 + (blk % nrow) * NB + 8 * warp + g;
  const bool rowok = row < n;
  for (int idx = tid; idx < kRows * 8 * NT; idx += 256) {
    const int r = idx & (kRows - 1), c = idx / kRows;
    Xs[r * kLd + c] = c0 + c < nrhs ? C[(kp + r) + ldc * (c0 + c)] : 0.0;
  }
  double bv[NT][2], acc[NT][2];
#pragma unroll
  for (int q = 0; q < NT; ++q)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int col = c0 + 8 * q + 2 * t4 + e;
      bv[q][e] = (rowok && col < nrhs) ? B[row + ldb * col] : 0.0;
      acc[q][e] = 0.0;
    }
  __syncthreads();
  const double* l = L + row + lda * (kp + t4);
#pragma unroll 16
  for (int k = 0; k < kRows; k += 4) {
    const double a = rowok ? l[lda * k] : 0.0;
#pragma unroll
    for (int q = 0; q < NT; ++q) dmma_m8n8k4(acc[q][0], acc[q][1], a, Xs[(k + t4) * kLd + 8 * q + g]);
  }
#pragma unroll
  for (int q = 0; q < NT; ++q)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int col = c0 + 8 * q + 2 * t4 + e;
      if (rowok && col < nrhs) B[row + ldb * col] = bv[q][e] - acc[q][e];
    }
}

// C[m x n] := beta C + alpha op(A) op(B); op(A) is m x k, op(B) is k x n.
// 64 x 64 tiles, k-steps of 16 staged in shared memory, products on the FP64
// tensor cores (mma.sync m8n8k4): warp w owns rows 16 (w % 4) .. + 16 and
// columns 32 (w / 4) .. + 32 of the tile.
// lower_c: skip output tiles strictly above the diagonal (and entries above it).
constexpr int TM = 64, TN = 64, TK = 16;
template <bool TA, bool TB>
__global__ void __launch_bounds__(256) k_gemm(int m, int n, int k, double alpha,
                                              const double* __restrict__ A, long long lda,
                                              const double* __restrict__ B, long long ldb,
                                              double beta, double* C, long long ldc,
                                              int lower_c) {
  const int bi = blockIdx.x, bj = blockIdx.y;
  if (lower_c && bj > bi) return;
  __shared__ double As[TK][TM + 1];
  __shared__ double Bs[TK][TN + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int wm = (warp & 3) * 16, wn = (warp >> 2) * 32;
  const int i0 = bi * TM, j0 = bj * TN;
  double acc[2][4][2] = {};
  for (int kk = 0; kk < k; kk += TK) {
    for (int idx = threadIdx.x; idx < TK * TM; idx += 256) {
      int r, c;  // r in tile rows (m), c in k
      if (TA) {  // A stored k x m: op(A)(r, c) = A[c + lda * r]
        c = idx % TK;
        r = idx / TK;
      } else {
        r = idx % TM;
        c = idx / TM;
      }
      const int gi = i0 + r, gk = kk + c;
      double v = 0.0;
      if (gi < m && gk < k) v = TA ? A[gk + lda * gi] : A[gi + lda * gk];
      As[c][r] = v;
    }
    for (int idx = threadIdx.x; idx < TK * TN; idx += 256) {
      int r, c;  // r in k, c in tile cols (n)
      if (TB) {  // B stored n x k: op(B)(r, c) = B[c + ldb * r]
        c = idx % TN;
        r = idx / TN;
      } else {
        r = idx % TK;
        c = idx / TK;
      }
      const int gk = kk + r, gj = j0 + c;
      double v = 0.0;
      if (gk < k && gj < n) v = TB ? B[gj + ldb * gk] : B[gk + ldb * gj];
      Bs[r][c] = v;
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < TK; q += 4) {
      double a[2], b[4];
#pragma unroll
      for (int mt = 0; mt < 2; ++mt) a[mt] = As[q + t4][wm + 8 * mt + g];
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) b[nt] = Bs[q + t4][wn + 8 * nt + g];
#pragma unroll
      for (int mt = 0; mt < 2; ++mt)
#pragma unroll
        for (int nt = 0; nt < 4; ++nt) dmma_m8n8k4(acc[mt][nt][0], acc[mt][nt][1], a[mt], b[nt]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int gi = i0 + wm + 8 * mt + g, gj = j0 + wn + 8 * nt + 2 * t4 + i;
        if (gi < m && gj < n && (!lower_c || gi >= gj)) {
          double* c = C + gi + ldc * gj;
          *c = (beta == 0.0 ? 0.0 : beta * *c) + alpha * acc[mt][nt][i];
        }
      }
}

// Trailing update of the Cholesky factorization: C -= P P^T on the lower part
// (i >= j) of C (m x m, column-major, ldc) without its first 64 x 64 diagonal
// tile (k_chol_step takes that one), P (m x k, column-major, ldp, k <= NB).
// One block per 64 x 64 tile of that lower part, row by row. Both panels of a tile are staged whole (every k at
// once) by cp.async copies (16 bytes when the columns are 16-byte aligned,
// else 8 bytes: ldp may be odd), in rows of 68 doubles
// (4 mod 16: conflict-free m8n8k4 fragment loads); two blocks per SM (128
// registers: the C prefetch spills at three) keep one block's copies in
// flight during another's products (standalone 13400 x 13400 factor: 66.0 ms
// with three blocks and 8-byte copies, 49.2 ms now). The products run
// in k_gemm's order (k ascending, four at a time, zeros up to a multiple of
// 16), so the factor is the same bit for bit.
constexpr int kSyrkLd = TM + 4;
constexpr size_t kSyrkSmem = sizeof(double) * 2 * NB * kSyrkLd;

// V16: the panel columns start on 16-byte boundaries (ldp even, P aligned), so
// pairs of rows are copied 16 bytes at a time. The block's entries of C are
// loaded into registers before the panels arrive, so their latency overlaps
// the copies and the products.
template <bool V16>
__global__ void __launch_bounds__(256, 2) k_syrk_update(int m, int k, const double* __restrict__ P,
                                                        long long ldp, double* C, long long ldc) {
  extern __shared__ __align__(16) double sm[];
  double* As = sm;                  // As[c * kSyrkLd + r] = P[i0 + r, c]
  double* Bs = sm + NB * kSyrkLd;   // Bs[c * kSyrkLd + r] = P[j0 + r, c]
  const int t = blockIdx.x + 1;  // tile (0, 0) is left out
  int bi = static_cast<int>((sqrt(8.0 * t + 1.0) - 1.0) * 0.5);
  while ((bi + 1) * (bi + 2) / 2 <= t) ++bi;
  while (bi * (bi + 1) / 2 > t) --bi;
  const int bj = t - bi * (bi + 1) / 2;
  const int i0 = bi * TM, j0 = bj * TN;
  const int kq = (k + TK - 1) / TK * TK;
  if constexpr (V16) {
    for (int idx = threadIdx.x; idx < kq * (TM / 2); idx += 256) {
      const int r = 2 * (idx % (TM / 2)), c = idx / (TM / 2);
      double* da = As + c * kSyrkLd + r;
      double* db = Bs + c * kSyrkLd + r;
      if (c < k && i0 + r + 1 < m) {
        cp_async16_ld(da, P + (i0 + r) + ldp * c);
      } else {
        da[0] = (c < k && i0 + r < m) ? P[(i0 + r) + ldp * c] : 0.0;
        da[1] = 0.0;
      }
      if (c < k && j0 + r + 1 < m) {
        cp_async16_ld(db, P + (j0 + r) + ldp * c);
      } else {
        db[0] = (c < k && j0 + r < m) ? P[(j0 + r) + ldp * c] : 0.0;
        db[1] = 0.0;
      }
    }
  } else {
    for (int idx = threadIdx.x; idx < kq * TM; idx += 256) {
      const int r = idx % TM, c = idx / TM;
      double* da = As + c * kSyrkLd + r;
      double* db = Bs + c * kSyrkLd + r;
      if (c < k && i0 + r < m)
        cp_async8(da, P + (i0 + r) + ldp * c);
      else
        *da = 0.0;
      if (c < k && j0 + r < m)
        cp_async8(db, P + (j0 + r) + ldp * c);
      else
        *db = 0.0;
    }
  }
  asm volatile("cp.async.commit_group;\n" ::);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int wm = (warp & 3) * 16, wn = (warp >> 2) * 32;
  // this thread's entries of C, in flight while the panels arrive
  double cv[2][4][2];
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int gi = i0 + wm + 8 * mt + g, gj = j0 + wn + 8 * nt + 2 * t4 + i;
        cv[mt][nt][i] = (gi < m && gj < m && gi >= gj) ? C[gi + ldc * gj] : 0.0;
      }
  asm volatile("cp.async.wait_group 0;\n" ::);
  __syncthreads();
  double acc[2][4][2] = {};
#pragma unroll 4
  for (int q = 0; q < kq; q += 4) {
    double a[2], b[4];
#pragma unroll
    for (int mt = 0; mt < 2; ++mt) a[mt] = As[(q + t4) * kSyrkLd + wm + 8 * mt + g];
#pragma unroll
    for (int nt = 0; nt < 4; ++nt) b[nt] = Bs[(q + t4) * kSyrkLd + wn + 8 * nt + g];
#pragma unroll
    for (int mt = 0; mt < 2; ++mt)
#pragma unroll
      for (int nt = 0; nt < 4; ++nt) dmma_m8n8k4(acc[mt][nt][0], acc[mt][nt][1], a[mt], b[nt]);
  }
#pragma unroll
  for (int mt = 0; mt < 2; ++mt)
#pragma unroll
    for (int nt = 0; nt < 4; ++nt)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int gi = i0 + wm + 8 * mt + g, gj = j0 + wn + 8 * nt + 2 * t4 + i;
        if (gi < m && gj < m && gi >= gj) C[gi + ldc * gj] = cv[mt][nt][i] + -1.0 * acc[mt][nt][i];
      }
}

// Gram matrix G[i + nd j] = sum_k df[k + naux i] df[k + naux j] of the fitted
// densities, one warp per entry: lanes stride over k (contiguous columns),
// then a fixed-order shuffle reduction. Used for nd <= kGramWarpMax, where the
// tiled GEMM would run as a single block over the whole k range.
constexpr int kGramWarpMax = 128;
__global__ void __launch_bounds__(256) k_gram_warp(const double* __restrict__ df, int naux, int nd,
                                                   double* G) {
  const int w = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
  if (w >= nd * nd) return;
  const int i = w % nd, j = w / nd;
  const double* a = df + static_cast<long long>(naux) * i;
  const double* b = df + static_cast<long long>(naux) * j;
  double s = 0.0;
  for (int k = lane; k < naux; k += 32) s = fma(a[k], b[k], s);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) G[i + static_cast<long long>(nd) * j] = s;
}

// R(i,j,k,l) = Gram[pair(i,j)][pair(k,l)], pair(i,j) = max(max+1)/2 + min.
__global__ void k_coulomb4d(const double* __restrict__ gram, int ndens, int ns, double* R) {
  const long long total = static_cast<long long>(ns) * ns * ns * ns;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    long long t = idx;
    const int i = t % ns;
    t /= ns;
    const int j = t % ns;
    t /= ns;
    const int k = t % ns;
    const int l = static_cast<int>(t / ns);
    const int a = max(i, j), b = min(i, j), c = max(k, l), d = min(k, l);
    const int p1 = a * (a + 1) / 2 + b, p2 = c * (c + 1) / 2 + d;
    R[idx] = gram[p1 + static_cast<long long>(ndens) * p2];
  }
}

__global__ void k_add_diagonal(double* A, int n, double shift) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) A[i + static_cast<long long>(n) * i] += shift;
}

// C -= P P^T on the lower part of C (m x m) without its first diagonal tile, P m x k (k <= NB).
int syrk_update(int m, int k, const double* P, long long ldp, double* C, long long ldc, cudaStream_t s) {
  if (m <= 0) return 0;
  const long long nbr = (m + TM - 1) / TM, tiles = nbr * (nbr + 1) / 2 - 1;
  if (tiles <= 0) return 0;
  if (ldp % 2 == 0 && reinterpret_cast<uintptr_t>(P) % 16 == 0)
    k_syrk_update<true><<<static_cast<unsigned>(tiles), 256, kSyrkSmem, s>>>(m, k, P, ldp, C, ldc);
  else
    k_syrk_update<false><<<static_cast<unsigned>(tiles), 256, kSyrkSmem, s>>>(m, k, P, ldp, C, ldc);
  return 1;
}

}  // namespace

int gemm(bool ta, bool tb, int m, int n, int k, double alpha, const double* A, long long lda,
         const double* B, long long ldb, double beta, double* C, long long ldc, bool lower_only,
         cudaStream_t s) {
  if (m <= 0 || n <= 0) return 0;
  dim3 grid((m + TM - 1) / TM, (n + TN - 1) / TN);
  const int lc = lower_only ? 1 : 0;
  if (!ta && !tb)
    k_gemm<false, false><<<grid, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, lc);
  else if (!ta && tb)
    k_gemm<false, true><<<grid, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, lc);
  else if (ta && !tb)
    k_gemm<true, false><<<grid, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, lc);
  else
    k_gemm<true, true><<<grid, 256, 0, s>>>(m, n, k, alpha, A, lda, B, ldb, beta, C, ldc, lc);
  return 1;
}

size_t linalg_workspace_doubles(int n) {
  const int nblk = (n + NB - 1) / NB;
  return static_cast<size_t>(nblk) * NB * NB;
}

int cholesky_lower(double* A, int n, int* d_info, double* work, cudaStream_t s,
                   const CholLookahead* la) {
  int launches = 0;
  cudaFuncSetAttribute(k_chol_step, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kCholSmem));
  cudaFuncSetAttribute(k_syrk_update<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSyrkSmem));
  cudaFuncSetAttribute(k_syrk_update<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(kSyrkSmem));
  cudaMemsetAsync(d_info, 0, sizeof(int), s);
  const int nblk = (n + NB - 1) / NB;
  // Step c (k_chol_step) on s; its trailing update of block columns c + 2.. on
  // the aux stream beside step c + 1, which takes column c itself and needs the
  // updates up to that of step c - 1 only.
  bool pending[2] = {false, false};  // an update of a step of this parity is queued on la->aux
  for (int c = -1; c + 1 < nblk; ++c) {
    if (la && c >= 2 && pending[c & 1]) {
      cudaStreamWaitEvent(s, la->ev_rest[c & 1], 0);  // update of step c - 2
      pending[c & 1] = false;
    }
    k_chol_step<<<c < 0 ? 1 : nblk - 1 - c, 256, kCholSmem, s>>>(A, n, n, c, work, d_info);
    ++launches;
    if (c < 0) continue;
    const int j0 = (c + 2) * NB, rest = n - j0;
    if (rest <= NB) continue;  // nothing beyond the diagonal tile of the next steps
    const double* P = A + j0 + static_cast<long long>(n) * (c * NB);
    double* C = A + j0 + static_cast<long long>(n) * j0;
    if (!la) {
      launches += syrk_update(rest, NB, P, n, C, n, s);
      continue;
    }
    cudaEventRecord(la->ev_panel, s);
    cudaStreamWaitEvent(la->aux, la->ev_panel, 0);
    launches += syrk_update(rest, NB, P, n, C, n, la->aux);
    cudaEventRecord(la->ev_rest[c & 1], la->aux);
    pending[c & 1] = true;
  }
  for (int p = 0; p < 2; ++p)
    if (pending[p]) cudaStreamWaitEvent(s, la->ev_rest[p], 0);
  return launches;
}

namespace {

template <int NT, int R>
int trsm_launches(const double* L, int n, const double* dinv, double* B, long long ldb, int nrhs, double* C,
                  long long ldc, cudaStream_t s) {
  constexpr int kRows = R * NB;
  const size_t smem = trsm_smem(NT, R);
  cudaFuncSetAttribute(k_trsm_step<NT, R>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  const int nsolve = (nrhs + 7) / 8, ct = (nrhs + 8 * NT - 1) / (8 * NT);
  int launches = 0;
  for (int k0 = 0; k0 < n; k0 += kRows, ++launches) {
    const int below = k0 > 0 ? std::max(0, n - k0 - kRows) : 0;
    const long long blocks = nsolve + static_cast<long long>((below + NB - 1) / NB) * ct;
    k_trsm_step<NT, R><<<static_cast<unsigned>(blocks), 256, smem, s>>>(L, n, n, k0, dinv, B, ldb, nrhs, C, ldc, nsolve);
  }
  return launches;
}

}  // namespace

int trsm_lower_left(const double* L, int n, const double* dinv, double* B, long long ldb, int nrhs,
                    double* C, long long ldc, cudaStream_t s) {
  if (n <= 0 || nrhs <= 0) return 0;
  if (nrhs <= 40) return trsm_launches<5, 2>(L, n, dinv, B, ldb, nrhs, C, ldc, s);
  if (nrhs <= kTrsmFew) return trsm_launches<4, 2>(L, n, dinv, B, ldb, nrhs, C, ldc, s);
  return trsm_launches<4, 4>(L, n, dinv, B, ldb, nrhs, C, ldc, s);
}

int add_diagonal(double* A, int n, double shift, cudaStream_t s) {
  if (shift == 0.0 || n <= 0) return 0;
  k_add_diagonal<<<(n + 255) / 256, 256, 0, s>>>(A, n, shift);
  return 1;
}

int coulomb_4d(const double* df, int naux, int ndens, int nstates, double* gram_scratch,
               double* R, cudaStream_t s) {
  int launches = 0;
  if (ndens <= kGramWarpMax) {
    const long long threads = 32LL * ndens * ndens;
    k_gram_warp<<<static_cast<int>((threads + 255) / 256), 256, 0, s>>>(df, naux, ndens, gram_scratch);
    launches = 1;
  } else {
    launches = gemm(true, false, ndens, ndens, naux, 1.0, df, naux, df, naux, 0.0, gram_scratch, ndens,
                    false, s);
  }
  const long long total = static_cast<long long>(nstates) * nstates * nstates * nstates;
  const int blocks = static_cast<int>(std::min<long long>((total + 255) / 256, 4096));
  k_coulomb4d<<<std::max(blocks, 1), 256, 0, s>>>(gram_scratch, ndens, nstates, R);
  return launches + 1;
}

}  // namespace pa
