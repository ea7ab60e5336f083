// Explicit spherical blocks (ab|c) of the std tensors (std/intor.f90:66-111,
// 207-261) by class (LAB = la + lb, LC = l_aux):
//   (ab|c)[(ma,mb)][m] = sum_(units u of ab) sum_tuv E_u[(ma,mb)][tuv] X_(u,c)[tuv][m].
//
// X is the Hermite-by-auxiliary tile of the density-folded contraction
// (k_df3c_impl.cuh) and is built by the same code; in the place of the folded
// density the product takes the expansion E_u itself. A block (8 warps, two per
// SM) owns UB shell pairs x TC auxiliary shells and walks the pairs' primitive
// pairs in step: X of the UB x TC triplets, then E X -- on the FP64 tensor cores
// (mma.sync m8n8k4, 8 block rows x up to 32 auxiliary columns per warp task) for
// LAB > 2, per thread below, where a pair has at most nine rows and ten
// Hermite components. Every output element has one owner thread, which adds the
// pair's primitive pairs in order (in place: most pairs have one).
//
// What bounds it: as in k_df3c, the X build (Boys, recurrence and their
// barriers); the blocks written are one pass over the output. Measured on B200,
// 40 atoms (lmax 3, lauxmax 4, 60 orbitals, 2240 auxiliary functions): all
// classes ~4 ms, k_std_half 3.5 ms; one block per (c, b) that built one triple
// at a time between barriers took 261 ms for both. One-center blocks of 60 atoms:
// 0.47 ms for 3.5 ms.
#pragma once

#include "k_df3c_impl.cuh"
#include "k_std3c.cuh"

namespace pa {

namespace {

// std/intor.f90:247: integrals of magnitude <= 1e-10 (REAL(4)) are dropped
constexpr double kSkipInt = static_cast<double>(1e-10f);

constexpr int max_block_rows(int lab) {
  int r = 0;
  for (int la = 0; la <= PA_LMAX; ++la) {
    const int lb = lab - la;
    if (lb < 0 || lb > PA_LMAX) continue;
    const int n = (2 * la + 1) * (2 * lb + 1);
    if (n > r) r = n;
  }
  return r;
}

template <int LAB, int LC>
struct StdCfg : Cfg<LAB, LC, 0> {
  using B = Cfg<LAB, LC, 0>;
  static constexpr int kTeam = B::kPerThread ? 0 : B::NTRIP * B::kTeamStride + 2 * B::NR;
  static constexpr int SMEM = B::KP * B::MPAD + 1024 + kTeam;
  static constexpr int kRows = max_block_rows(LAB);
  static constexpr bool kTensor = LAB > 2;
  static constexpr int kRowTiles = (kRows + 7) / 8;
  static constexpr int kColGroups = (B::MT + 3) / 4;
};

template <int LAB, int LC>
__global__ void __launch_bounds__(kThreads, 2) k_std3c(Std3cArgs a) {
  using C = StdCfg<LAB, LC>;
  extern __shared__ __align__(16) double smem[];
  double* Xs = smem;                                       // [KP][MPAD]
  double* misc = Xs + C::KP * C::MPAD;
  double* Rteam = misc + 1024;                             // team scratch
  double4* u_pP = reinterpret_cast<double4*>(misc);        // [UB <= 64]
  double* u_Q = misc + 256;                                // [UB]
  double4* c_C = reinterpret_cast<double4*>(misc + 320);   // [TC <= 128] (x, y, z, Q)
  int* c_info = reinterpret_cast<int*>(misc + 320 + 512);  // [TC] (nprim, prim_off)
  int* c_col = c_info + 256;                               // [TC] first output column
  __shared__ const double* u_E[64];                        // expansion of the current unit
  __shared__ long long u_row[64];                          // first output row
  __shared__ int u_nrow[64], u_nu[64], u_unit0[64];
  static_assert(C::UB <= 64 && C::TC <= 128, "sizes of the parameter arrays");

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nbx = (a.n_aux + C::TC - 1) / C::TC;
  const int bx = blockIdx.x % nbx;
  const int q0 = static_cast<int>(blockIdx.x / nbx) * C::UB;
  const int c0 = bx * C::TC;
  const int tile_n = min(C::TC, a.n_aux - c0);
  const int nvalid = min(C::UB, a.n_bra - q0);
  const double thr = a.x.thresh;

  if (tid < C::TC) {
    if (tid < tile_n) {
      const int sh = a.aux[c0 + tid];
      const int4 info = a.x.X.shell[sh];
      const double4 cen = a.x.X.center[sh];
      c_C[tid] = make_double4(cen.x, cen.y, cen.z, a.Qc[sh]);
      c_info[2 * tid] = info.y;
      c_info[2 * tid + 1] = info.z;
      c_col[tid] = a.diag ? info.w : a.col0 + (c0 + tid) * C::NC;
    } else {
      c_C[tid] = make_double4(0.0, 0.0, 0.0, 0.0);
      c_info[2 * tid] = 0;
      c_info[2 * tid + 1] = 0;
      c_col[tid] = 0;
    }
  }
  if (tid < C::UB) {
    u_nu[tid] = 0;
    u_nrow[tid] = 0;
    u_pP[tid] = make_double4(1.0, 0.0, 0.0, 0.0);
    u_Q[tid] = 0.0;
    if (tid < nvalid) {
      int q = a.bra[q0 + tid];
      if (a.diag) q = q * (q + 1) / 2 + q;
      const int2 ab = a.pair_ab[q];
      const int4 sa = a.B.shell[ab.x], sb = a.B.shell[ab.y];
      u_Q[tid] = a.Qab[q];
      u_nu[tid] = sa.y * sb.y;
      u_unit0[tid] = a.pair_unit0[q];
      u_nrow[tid] = a.diag ? 2 * sa.x + 1 : (2 * sa.x + 1) * (2 * sb.x + 1);
      u_row[tid] = a.diag ? sa.w : a.row0[q];
    }
  }
  if constexpr (!C::kPerThread) {
    uchar4* txyz = reinterpret_cast<uchar4*>(Rteam + C::NTRIP * C::kTeamStride);
    fill_team_tables<C::L>(txyz, reinterpret_cast<int*>(txyz + C::NR), a.x.dt, tid);
  }
  __syncthreads();
  int maxprim = 0, maxu = 0;
  for (int i = 0; i < tile_n; ++i) maxprim = max(maxprim, c_info[2 * i]);
  for (int i = 0; i < nvalid; ++i) maxu = max(maxu, u_nu[i]);

  // result v of row r of pair ui, tile column col, at unit k of the pair
  auto emit = [&](int ui, int r, int col, int k, double v) {
    const int ci = col / C::NC, m = col - ci * C::NC;
    if (ci >= tile_n) return;
    double* o = a.out + (u_row[ui] + r) * a.ld + c_col[ci] + m;
    if (k > 0) v += *o;
    if (!a.diag && k + 1 == u_nu[ui] && fabs(v) <= kSkipInt) v = 0.0;
    *o = v;
  };

  for (int k = 0; k < maxu; ++k) {
    if (k > 0) __syncthreads();  // the previous unit's products are done with X and u_E
    if (tid < nvalid && k < u_nu[tid]) {
      const int u = u_unit0[tid] + k;
      u_pP[tid] = a.unit_pP[u];
      u_E[tid] = a.esph + a.unit_esph[u];
    }
    __syncthreads();

    // X; screened triplets get zero rows, so their block is zero
    if constexpr (C::kPerThread) {
      const int part = warp % C::TPT;
      for (int tr = lane + 32 * (warp / C::TPT); tr < C::NTRIP; tr += 32 * (kWarps / C::TPT)) {
        const int ui = tr / C::TC, ci = tr - ui * C::TC;
        if (ci >= tile_n || ui >= nvalid || k >= u_nu[ui]) continue;
        const double4 cc = c_C[ci];
        double* xrow0 = Xs + (ui * C::NH) * C::MPAD + ci * C::NC;
        if (u_Q[ui] * cc.w < thr) {
          x_rows_zero<LAB, LC, C::TPT>(xrow0, C::MPAD, part);
          continue;
        }
        const double4 up = u_pP[ui];
        x_triplet_thread<LAB, LC, C::NR, C::MPAD, C::TPT, double>(a.x, up.x, up.y - cc.x, up.z - cc.y, up.w - cc.z,
                                                                  c_info[2 * ci], c_info[2 * ci + 1], xrow0, part);
      }
    } else {
      const uchar4* txyz = reinterpret_cast<const uchar4*>(Rteam + C::NTRIP * C::kTeamStride);
      const int* pdesc = reinterpret_cast<const int*>(txyz + C::NR);
      const int team = tid / C::TS, tl = tid - team * C::TS;
      const bool in_team = team < C::NTRIP;
      const int ui = in_team ? team / C::TC : 0, ci = in_team ? team - ui * C::TC : 0;
      double* rbuf = Rteam + (in_team ? team : 0) * C::kTeamStride;
      const double4 cc = c_C[ci];
      const bool valid = in_team && ci < tile_n && ui < nvalid && k < u_nu[ui];
      const bool active = valid && !(u_Q[ui] * cc.w < thr);
      const double4 up = u_pP[ui];
      double* xrow = Xs + (ui * C::NH) * C::MPAD + ci * C::NC;
      if (valid && !active)
        for (int t = tl; t < C::NH; t += C::TS)
#pragma unroll
          for (int m = 0; m < C::NC; ++m) xrow[t * C::MPAD + m] = 0.0;
      x_triplet_team<LAB, LC, C::TS, double>(a.x, txyz, pdesc, rbuf, team, tl, active, active ? c_info[2 * ci] : 0,
                                             c_info[2 * ci + 1], maxprim, up.x, up.y - cc.x, up.z - cc.y,
                                             up.w - cc.z, xrow, C::MPAD);
    }
    __syncthreads();

    // E X
    const int rstep = a.diag ? 1 : 0;  // diag: row i is (i, i), E row i * (rows + 1)
    if constexpr (C::kTensor) {
      const int g = lane >> 2, t4 = lane & 3;
      for (int task = warp; task < C::UB * C::kRowTiles * C::kColGroups; task += kWarps) {
        const int cg = task % C::kColGroups, ur = task / C::kColGroups;
        const int rt = ur % C::kRowTiles, ui = ur / C::kRowTiles;
        if (ui >= nvalid || k >= u_nu[ui] || 8 * rt >= u_nrow[ui] || 32 * cg >= tile_n * C::NC) continue;
        const int row = 8 * rt + g;
        const bool rowok = row < u_nrow[ui];
        const double* e = u_E[ui] + static_cast<long long>(rstep ? row * (u_nrow[ui] + 1) : row) * C::NH;
        const double* xs = Xs + ui * C::NH * C::MPAD + 32 * cg + g;
        double acc[4][2];
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[j][0] = acc[j][1] = 0.0;
#pragma unroll 4
        for (int k4 = 0; k4 < (C::NH + 3) / 4; ++k4) {
          const int kr = 4 * k4 + t4;
          const bool kin = kr < C::NH;
          const double av = kin && rowok ? __ldg(e + kr) : 0.0;
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (4 * cg + j >= C::MT) continue;
            const double bv = kin ? xs[kr * C::MPAD + 8 * j] : 0.0;
            dmma_m8n8k4(acc[j][0], acc[j][1], av, bv);
          }
        }
        if (rowok)
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (4 * cg + j >= C::MT) continue;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
              const int col = 32 * cg + 8 * j + 2 * t4 + i;
              if (col < C::M) emit(ui, row, col, k, acc[j][i]);
            }
          }
      }
    } else {
      for (int idx = tid; idx < C::UB * C::kRows * C::M; idx += kThreads) {
        const int col = idx % C::M, ur = idx / C::M;
        const int r = ur % C::kRows, ui = ur / C::kRows;
        if (ui >= nvalid || k >= u_nu[ui] || r >= u_nrow[ui]) continue;
        const double* e = u_E[ui] + static_cast<long long>(rstep ? r * (u_nrow[ui] + 1) : r) * C::NH;
        const double* xs = Xs + ui * C::NH * C::MPAD + col;
        double v = 0.0;
#pragma unroll
        for (int t = 0; t < C::NH; ++t) v = fma(__ldg(e + t), xs[t * C::MPAD], v);
        emit(ui, r, col, k, v);
      }
    }
  }
}

template <int LAB, int LC>
int launch_std3c(const Std3cArgs& a, cudaStream_t s) {
  using C = StdCfg<LAB, LC>;
  if (a.n_bra <= 0 || a.n_aux <= 0) return 0;
  const size_t smem = sizeof(double) * C::SMEM;
  cudaFuncSetAttribute(k_std3c<LAB, LC>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  const long long blocks =
      static_cast<long long>((a.n_aux + C::TC - 1) / C::TC) * ((a.n_bra + C::UB - 1) / C::UB);
  k_std3c<LAB, LC><<<static_cast<unsigned>(blocks), kThreads, smem, s>>>(a);
  return 1;
}

template <int LAB, int LC>
void fill_std3c_row(Std3cRow* row) {
  row->launch[LC] = &launch_std3c<LAB, LC>;
  if constexpr (LC < PA_LAUXMAX) fill_std3c_row<LAB, LC + 1>(row);
}

}  // namespace

}  // namespace pa

// Defines std3c_row_<LAB>(): the dispatch row of this translation unit's LAB.
#define PA_STD3C_ROW(LAB)                  \
  namespace pa {                           \
  void std3c_row_##LAB(Std3cRow* row) {    \
    fill_std3c_row<LAB, 0>(row);           \
    row->upload_rownorm = &upload_rownorm; \
  }                                        \
  }
