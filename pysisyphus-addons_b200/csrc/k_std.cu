// Kernels of the sTDDFT ("std") density-fitting tensors (std/intor.f90). The
// explicit blocks (ab|c) come from the class kernels of k_std3c_impl.cuh; here:
//  * k_std_pair_size, k_std_pair_row, k_std_columns  the layout of the block
//                     matrix: rows are the function pairs of the shell pairs
//                     that meet the largest auxiliary Schwarz value, columns
//                     the auxiliary functions in sorted class order;
//  * k_std_half       the first half-transformation of intor_df2c_mo
//                     (std/intor.f90:207-261) with the reference's skip of
//                     half-transformed values (:269), summed over the partner
//                     shell a for every target function nu; the second half
//                     (:263-279) is then one GEMM per batch of auxiliary
//                     functions, followed by k_std_pack;
//  * k_std_block_norm ||(ab|c)|| of single blocks (the estimator study);
//  * k_transpose      column-major transposition of the L^-1-applied results.
//
// The reference drops individual integrals |(ab|c)| <= 1e-10 (REAL(4) literal)
// and individual half-transformed values <= 1e-10 before summing; at the 8-atom
// workload these skips move intor_df2c_mo by ~4e-9, so they are reproduced
// triple by triple, which is why the blocks are stored and not contracted on
// the way.
#include "boys.cuh"
#include "k_std.cuh"
#include "k_std3c.cuh"
#include "md.cuh"

#include <algorithm>
#include <mutex>

namespace pa {

namespace {

struct BlockSync {
  __device__ void operator()() const { __syncthreads(); }
};

constexpr int kStdThreads = 128;
constexpr int kLtot = 2 * PA_LMAX + PA_LAUXMAX;           // highest la + lb + lc
constexpr int kNR = ncum(kLtot);                           // R entries of one build
constexpr int kNHMax = ncum(2 * PA_LMAX);                  // Hermite components of a bra
constexpr int kNCMax = 2 * PA_LAUXMAX + 1;                 // spherical aux functions
constexpr int kNSMax = 2 * PA_LMAX + 1;                    // spherical orbital functions
constexpr int kNabMax = kNSMax * kNSMax;
constexpr double kSkipHalf = 1e-10;                        // std/intor.f90:269

// Shared scratch of block_3c.
struct Blk3cScratch {
  double* Rn;  // 32
  double* R0;  // kNR
  double* R1;  // kNR
  double* Xs;  // kNHMax * kNCMax
  double* I;   // kNabMax * kNCMax
};
constexpr int kBlk3cDoubles = 32 + 2 * kNR + kNHMax * kNCMax + kNabMax * kNCMax;

__device__ __forceinline__ Blk3cScratch blk3c_scratch(double* base) {
  Blk3cScratch s;
  s.Rn = base;
  s.R0 = s.Rn + 32;
  s.R1 = s.R0 + kNR;
  s.Xs = s.R1 + kNR;
  s.I = s.Xs + kNHMax * kNCMax;
  return s;
}

__device__ __forceinline__ int cidx_sum(const IndexTables* __restrict__ it, int i, int j) {
  const uchar4 a = *reinterpret_cast<const uchar4*>(it->xyz[i]);
  const uchar4 b = *reinterpret_cast<const uchar4*>(it->xyz[j]);
  return cidx(a.x + b.x, a.y + b.y, a.z + b.z);
}

// I[(ma * nsb + mb) * NC + m] = (a_ma b_mb | c_m) for pair = (a, b), a >= b, by
// the whole block. Starts and ends with a block barrier.
__device__ void block_3c(const StdArgs& a, int pair, int c, Blk3cScratch s) {
  const IndexTables* it = a.dt.idx;
  const int tid = threadIdx.x, nthr = blockDim.x;
  const int2 ab = a.pair_ab[pair];
  const int4 sa = a.B.shell[ab.x], sb = a.B.shell[ab.y];
  const int nab = (2 * sa.x + 1) * (2 * sb.x + 1);
  const int NH = ncum(sa.x + sb.x);
  const int4 sc = a.X.shell[c];
  const int lc = sc.x, NC = 2 * lc + 1;
  const int L = sa.x + sb.x + lc;
  const int offc = ncum(lc - 1);
  const double4 C = a.X.center[c];
  __syncthreads();  // previous readers of I are done
  for (int i = tid; i < nab * NC; i += nthr) s.I[i] = 0.0;
  const int u0 = a.pair_unit0[pair], nu = sa.y * sb.y;
  for (int u = u0; u < u0 + nu; ++u) {
    const double4 up = a.unit_pP[u];
    const double* E = a.esph + a.unit_esph[u];
    const double p = up.x;
    const double X = up.y - C.x, Y = up.z - C.y, Z = up.w - C.z;
    const double RPC2 = X * X + Y * Y + Z * Z;
    for (int kc = 0; kc < sc.y; ++kc) {
      const double2 gp = a.X.prim[sc.z + kc];
      const double gam = gp.x, pg = p + gam, alpha = p * gam / pg;
      double pref = kTwoPi52 / (p * gam * sqrt(pg)) * gp.y;
      for (int l = 0; l < lc; ++l) pref *= -0.5 / gam;  // (-1)^lc (2 gam)^-lc
      __syncthreads();  // previous users of Rn / R / Xs are done
      if (tid <= L) {
        double f = pref;
        for (int k = 0; k < tid; ++k) f *= -2.0 * alpha;
        s.Rn[tid] = f * boys_n(a.dt, a.boys_mode, tid, alpha * RPC2);
      }
      __syncthreads();
      hermite_R(a.dt.rdesc, L, s.Rn, X, Y, Z, s.R0, s.R1, tid, nthr, BlockSync());
      for (int idx = tid; idx < NH * NC; idx += nthr) {
        const int t = idx / NC, m = idx - t * NC;
        const int row = lc * lc + m;
        double y = 0.0;
        for (int k = a.dt.sph_start[row]; k < a.dt.sph_start[row + 1]; ++k)
          y = fma(a.dt.sph_val[k], s.R0[cidx_sum(it, t, offc + a.dt.sph_col[k])], y);
        s.Xs[idx] = y;
      }
      __syncthreads();
      for (int idx = tid; idx < nab * NC; idx += nthr) {
        const int r = idx / NC, m = idx - r * NC;
        const double* e = E + static_cast<long long>(r) * NH;
        double v = 0.0;
        for (int t = 0; t < NH; ++t) v = fma(__ldg(e + t), s.Xs[t * NC + m], v);
        s.I[idx] += v;
      }
    }
  }
  __syncthreads();
}

// ||(ab|c)||_2 of the block of pair rec_pair[blockIdx.y] and auxiliary shell
// blockIdx.x (the estimator study of intor/benchmark.f90:96-118).
__global__ void __launch_bounds__(kStdThreads) k_std_block_norm(StdArgs a, const int* __restrict__ rec_pair,
                                                                int nx, double* __restrict__ out) {
  __shared__ double scratch[kBlk3cDoubles];
  __shared__ double s_red[kStdThreads / 32];
  const int c = blockIdx.x, kp = blockIdx.y;
  const int pair = rec_pair[kp];
  Blk3cScratch s = blk3c_scratch(scratch);
  block_3c(a, pair, c, s);
  const int2 ab = a.pair_ab[pair];
  const int n = (2 * a.B.shell[ab.x].x + 1) * (2 * a.B.shell[ab.y].x + 1) * (2 * a.X.shell[c].x + 1);
  double ss = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) ss = fma(s.I[i], s.I[i], ss);
  for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = ss;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < kStdThreads / 32; ++w) t += s_red[w];
    out[static_cast<long long>(kp) * nx + c] = sqrt(t);
  }
}

// keys[i] = Schwarz value of the i-th pair of the class-ordered list.
__global__ void k_std_pair_keys(int n, const int* __restrict__ class_pair, const double* __restrict__ Qab,
                                double* keys, int* vals) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  keys[i] = Qab[class_pair[i]];
  vals[i] = i;
}

// Rows of the sorted pair i in the block matrix: all of its function pairs when
// it meets the largest auxiliary Schwarz value, else none. The sorted values
// fall within a class, so its surviving pairs are a prefix: nclass[c].
__global__ void k_std_pair_size(StdArgs a, int n, const double* __restrict__ Q, const int* __restrict__ pair,
                                const int* __restrict__ off, int nseg, const double* __restrict__ qmax, int* size,
                                int* nclass) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double qm = *qmax;
  const int2 ab = a.pair_ab[pair[i]];
  const bool alive = !(Q[i] * qm < a.thresh);
  size[i] = alive ? (2 * a.B.shell[ab.x].x + 1) * (2 * a.B.shell[ab.y].x + 1) : 0;
  int c = 0;
  while (c + 1 < nseg && i >= off[c + 1]) ++c;
  if (alive && (i + 1 == off[c + 1] || Q[i + 1] * qm < a.thresh)) nclass[c] = i + 1 - off[c];
}

// First row per pair id (-1: no rows); the number of rows goes to *total.
__global__ void k_std_pair_row(int n, const int* __restrict__ pair, const int* __restrict__ size,
                               const int* __restrict__ first, int* row0, int* total) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  row0[pair[i]] = size[i] > 0 ? first[i] : -1;
  if (i == n - 1) *total = first[i] + size[i];
}

// Columns: function m of sorted auxiliary shell i of class L is column
// (functions of lower classes) + (i - off[L]) (2L + 1) + m.
__global__ void k_std_columns(int n, const int* __restrict__ sorted, const double* __restrict__ Q,
                              const int* __restrict__ off, int nseg, const int4* __restrict__ shell, int* col_fn,
                              double* col_Q) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  int L = 0, base = 0;
  while (L + 1 < nseg && i >= off[L + 1]) {
    base += (off[L + 1] - off[L]) * (2 * L + 1);
    ++L;
  }
  base += (i - off[L]) * (2 * L + 1);
  for (int m = 0; m < 2 * L + 1; ++m) {
    col_fn[base + m] = shell[sorted[i]].w + m;
    col_Q[base + m] = Q[i];
  }
}

// Shell of every orbital function.
__global__ void k_std_fn_shell(int n, const int4* __restrict__ shell, int* fn_shell) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  for (int m = 0; m < 2 * shell[i].x + 1; ++m) fn_shell[shell[i].w + m] = i;
}

// Ct[i * pld + p] = C[i, p], zero for p >= nmos.
__global__ void k_std_mo_rows(const double* __restrict__ mo, int nbf, int nmos, int pld, double* __restrict__ Ct) {
  const long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x;
  if (idx >= static_cast<long long>(nbf) * pld) return;
  const int i = static_cast<int>(idx / pld), p = static_cast<int>(idx - static_cast<long long>(i) * pld);
  Ct[idx] = p < nmos ? mo[i + static_cast<long long>(nbf) * p] : 0.0;
}

// W[nu][p][k] = sum_a skip(sum_(i in a) C[i, p] (i nu|k)), partner shells a in
// ascending order (the reference's), skip(h) = h where |h| > 1e-10, else 0.
//
// A block owns one target function nu, 64 columns k and 16 PT orbitals p; a
// thread a PT x 4 tile of them, its partial sum over the functions of the
// current shell beside its accumulator. The functions of the surviving partner
// shells form one list of rows (a shell survives when its pair has rows and
// meets the tile's largest auxiliary Schwarz value); 16 rows of (i nu|k) and of
// C are staged at a time through three cp.async buffers, so a shell may
// straddle two stages. Bound: the FP64 pipe (52 % busy at 40 atoms, 64 % SM
// throughput), (functions + 2 per shell)
// operations per (nu, k, p) and partner shell; no tensor cores, because the
// skip needs every shell's sum on its own, and padding shells of 1, 3, 5, 7
// functions to the depth of an FP64 mma (4) would cost 1.7 times the products.
constexpr int kHalfCols = 64, kHalfRows = 16, kHalfStages = 3;
constexpr int kHalfThreads = 256;
constexpr int kHalfList = kHalfThreads * kNSMax;  // rows of one group of partner shells

constexpr size_t half_smem(int pt) {
  return sizeof(double) * kHalfStages * kHalfRows * (kHalfCols + 16 * pt) + sizeof(int) * 2 * kHalfList;
}

__device__ __forceinline__ void half_cp16(double* dst, const double* src) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src));
}

template <int PT>
__global__ void __launch_bounds__(kHalfThreads, 2) k_std_half(StdHalfArgs h) {
  constexpr int P = 16 * PT;
  extern __shared__ __align__(16) double sm[];
  double* Is = sm;                                             // [stage][row][kHalfCols]
  double* Cs = Is + kHalfStages * kHalfRows * kHalfCols;       // [stage][row][P]
  int* s_row = reinterpret_cast<int*>(Cs + kHalfStages * kHalfRows * P);  // row of the block matrix
  int* s_fn = s_row + kHalfList;                               // partner function * 2 + (last of its shell)
  __shared__ int s_cnt[kHalfThreads / 32];
  __shared__ double s_q[kHalfThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nkt = (h.nk + kHalfCols - 1) / kHalfCols;
  const int nu = blockIdx.x / nkt, k0 = (blockIdx.x - nu * nkt) * kHalfCols;
  const int p0 = blockIdx.y * P;
  const int b = h.fn_shell[nu];
  const int4 sb = h.B.shell[b];
  const int nb = 2 * sb.x + 1, j = nu - sb.w;
  const int ncol2 = min(kHalfCols, h.ld - k0) / 2;  // 16-byte pieces of the tile's rows (ld is even)

  double qmax = tid < kHalfCols && k0 + tid < h.nk ? h.col_Q[k0 + tid] : 0.0;
  for (int o = 16; o > 0; o >>= 1) qmax = fmax(qmax, __shfl_xor_sync(0xffffffffu, qmax, o));
  if (lane == 0) s_q[warp] = qmax;
  __syncthreads();
  qmax = fmax(s_q[0], s_q[1]);

  const int kt = tid & 15, pt = tid >> 4;
  double acc[PT][4], hh[PT][4];
#pragma unroll
  for (int q = 0; q < PT; ++q)
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[q][i] = hh[q][i] = 0.0;

  for (int sh0 = 0; sh0 < h.B.nshells; sh0 += kHalfThreads) {
    // rows of this group's surviving partner shells, in shell order
    const int sh = sh0 + tid;
    int na = 0, r0 = -1, fn0 = 0;
    if (sh < h.B.nshells) {
      const int hi = max(sh, b), lo = min(sh, b);
      const long long pair = static_cast<long long>(hi) * (hi + 1) / 2 + lo;
      r0 = h.row0[pair];
      if (r0 >= 0 && !(h.Qab[pair] * qmax < h.thresh)) {
        const int4 sa = h.B.shell[sh];
        na = 2 * sa.x + 1;
        fn0 = sa.w;
      }
    }
    int incl = na;
    for (int o = 1; o < 32; o <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += v;
    }
    if (lane == 31) s_cnt[warp] = incl;
    __syncthreads();
    int off = incl - na, total = 0;
    for (int w = 0; w < kHalfThreads / 32; ++w) {
      if (w < warp) off += s_cnt[w];
      total += s_cnt[w];
    }
    for (int i = 0; i < na; ++i) {
      s_row[off + i] = r0 + (sh >= b ? i * nb + j : j * na + i);
      s_fn[off + i] = 2 * (fn0 + i) + (i == na - 1 ? 1 : 0);
    }
    __syncthreads();
    const int nch = (total + kHalfRows - 1) / kHalfRows;
    auto issue = [&](int c) {
      if (c < nch) {
        double* is = Is + (c % kHalfStages) * kHalfRows * kHalfCols;
        double* cs = Cs + (c % kHalfStages) * kHalfRows * P;
        const int nr = min(kHalfRows, total - c * kHalfRows);
        for (int e = tid; e < kHalfRows * (kHalfCols / 2); e += kHalfThreads) {
          const int r = e / (kHalfCols / 2), x = e % (kHalfCols / 2);
          if (r < nr && x < ncol2)
            half_cp16(is + r * kHalfCols + 2 * x,
                      h.I + static_cast<long long>(s_row[c * kHalfRows + r]) * h.ld + k0 + 2 * x);
        }
        for (int e = tid; e < kHalfRows * (P / 2); e += kHalfThreads) {
          const int r = e / (P / 2), x = e % (P / 2);
          if (r < nr)
            half_cp16(cs + r * P + 2 * x,
                      h.Ct + static_cast<long long>(s_fn[c * kHalfRows + r] >> 1) * h.pld + p0 + 2 * x);
        }
      }
      asm volatile("cp.async.commit_group;\n" ::);
    };
    issue(0);
    issue(1);
    for (int c = 0; c < nch; ++c) {
      asm volatile("cp.async.wait_group 1;\n" ::);
      __syncthreads();  // stage c has arrived; stage c - 1 is consumed
      issue(c + 2);
      const double* is = Is + (c % kHalfStages) * kHalfRows * kHalfCols + 2 * kt;
      const double* cs = Cs + (c % kHalfStages) * kHalfRows * P + pt * PT;
      const int nr = min(kHalfRows, total - c * kHalfRows);
#pragma unroll 2
      for (int r = 0; r < nr; ++r) {
        const double2 x0 = *reinterpret_cast<const double2*>(is + r * kHalfCols);
        const double2 x1 = *reinterpret_cast<const double2*>(is + r * kHalfCols + kHalfCols / 2);
#pragma unroll
        for (int q = 0; q < PT; ++q) {
          const double cv = cs[r * P + q];
          hh[q][0] = fma(cv, x0.x, hh[q][0]);
          hh[q][1] = fma(cv, x0.y, hh[q][1]);
          hh[q][2] = fma(cv, x1.x, hh[q][2]);
          hh[q][3] = fma(cv, x1.y, hh[q][3]);
        }
        if (s_fn[c * kHalfRows + r] & 1)
#pragma unroll
          for (int q = 0; q < PT; ++q)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
              if (fabs(hh[q][i]) > kSkipHalf) acc[q][i] += hh[q][i];
              hh[q][i] = 0.0;
            }
      }
    }
    asm volatile("cp.async.wait_group 0;\n" ::);
    __syncthreads();  // the lists and stages are rewritten by the next group
  }
#pragma unroll
  for (int q = 0; q < PT; ++q) {
    const int p = p0 + pt * PT + q;
    if (p >= h.nmos) continue;
    double* w = h.W + (static_cast<long long>(nu) * h.nmos + p) * h.ld + k0;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int c = i * (kHalfCols / 2) + 2 * kt;
      if (c / 2 < ncol2) *reinterpret_cast<double2*>(w + c) = make_double2(acc[q][2 * i], acc[q][2 * i + 1]);
    }
  }
}

__global__ void k_std_pack(const double* __restrict__ Res, int nk, int ld, int nmos, const int* __restrict__ col_fn,
                           int naux, double* __restrict__ Raw) {
  const long long npack = static_cast<long long>(nmos) * (nmos + 1) / 2;
  const long long total = npack * nk;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const long long pk = idx / nk;
    const int kk = static_cast<int>(idx - pk * nk);
    int p = static_cast<int>((sqrt(8.0 * static_cast<double>(pk) + 1.0) - 1.0) * 0.5);
    while (static_cast<long long>(p) * (p + 1) / 2 > pk) --p;
    while (static_cast<long long>(p + 1) * (p + 2) / 2 <= pk) ++p;
    const int q = static_cast<int>(pk - static_cast<long long>(p) * (p + 1) / 2);
    Raw[col_fn[kk] + static_cast<long long>(naux) * pk] =
        Res[kk + static_cast<long long>(ld) * (p + static_cast<long long>(nmos) * q)];
  }
}

__global__ void k_transpose(const double* __restrict__ in, int rows, int cols, double* __restrict__ out) {
  // out (rows x cols) = in^T, in (cols x rows); a block moves one 32 x 32 tile,
  // reading along in's leading dimension and writing along out's
  __shared__ double tile[32][33];  // [out row][out col] within the tile
  const int j0 = blockIdx.x * 32, i0 = blockIdx.y * 32;
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int j = j0 + threadIdx.x, i = i0 + k;
    if (i < rows && j < cols) tile[k][threadIdx.x] = in[j + static_cast<long long>(cols) * i];
  }
  __syncthreads();
  for (int k = threadIdx.y; k < 32; k += blockDim.y) {
    const int i = i0 + threadIdx.x, j = j0 + k;
    if (i < rows && j < cols) out[i + static_cast<long long>(rows) * j] = tile[threadIdx.x][k];
  }
}

}  // namespace

namespace {

const Std3cRow* std3c_rows() {
  static Std3cRow table[2 * PA_LMAX + 1];
  static std::once_flag once;
  std::call_once(once, [] {
    std3c_row_0(&table[0]);
    std3c_row_1(&table[1]);
    std3c_row_2(&table[2]);
    std3c_row_3(&table[3]);
    std3c_row_4(&table[4]);
    std3c_row_5(&table[5]);
    std3c_row_6(&table[6]);
    std3c_row_7(&table[7]);
    std3c_row_8(&table[8]);
  });
  return table;
}

template <int PT>
int launch_half(const StdHalfArgs& h, cudaStream_t s) {
  const size_t smem = half_smem(PT);
  cudaFuncSetAttribute(k_std_half<PT>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
  const long long tiles = static_cast<long long>((h.nk + kHalfCols - 1) / kHalfCols) * h.B.nsph;
  k_std_half<PT><<<dim3(static_cast<unsigned>(tiles), (h.nmos + 16 * PT - 1) / (16 * PT)), kHalfThreads, smem, s>>>(h);
  return 1;
}

}  // namespace

int launch_std3c_class(int lab, int lc, const Std3cArgs& a, cudaStream_t s) {
  return std3c_rows()[lab].launch[lc](a, s);
}

cudaError_t upload_std3c_rownorm(const double* rownorm, cudaStream_t s) {
  for (int lab = 0; lab <= 2 * PA_LMAX; ++lab) {
    const cudaError_t e = std3c_rows()[lab].upload_rownorm(rownorm, s);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

int launch_std_pair_keys(int n, const int* class_pair, const double* Qab, double* keys, int* vals, cudaStream_t s) {
  if (n <= 0) return 0;
  k_std_pair_keys<<<(n + 255) / 256, 256, 0, s>>>(n, class_pair, Qab, keys, vals);
  return 1;
}

int launch_std_pair_size(const StdArgs& a, int n, const double* Q, const int* pair, const int* off, int nseg,
                         const double* qmax, int* size, int* nclass, cudaStream_t s) {
  if (n <= 0) return 0;
  k_std_pair_size<<<(n + 255) / 256, 256, 0, s>>>(a, n, Q, pair, off, nseg, qmax, size, nclass);
  return 1;
}

int launch_std_pair_row(int n, const int* pair, const int* size, const int* first, int* row0, int* total,
                        cudaStream_t s) {
  if (n <= 0) return 0;
  k_std_pair_row<<<(n + 255) / 256, 256, 0, s>>>(n, pair, size, first, row0, total);
  return 1;
}

int launch_std_columns(int n, const int* sorted, const double* Q, const int* off, int nseg, const int4* shell,
                       int* col_fn, double* col_Q, cudaStream_t s) {
  if (n <= 0) return 0;
  k_std_columns<<<(n + 255) / 256, 256, 0, s>>>(n, sorted, Q, off, nseg, shell, col_fn, col_Q);
  return 1;
}

int launch_std_orbitals(const DevBasis& B, const double* mo, int nmos, int pld, int* fn_shell, double* Ct,
                        cudaStream_t s) {
  if (B.nshells <= 0 || nmos <= 0) return 0;
  k_std_fn_shell<<<(B.nshells + 255) / 256, 256, 0, s>>>(B.nshells, B.shell, fn_shell);
  const long long n = static_cast<long long>(B.nsph) * pld;
  k_std_mo_rows<<<static_cast<unsigned>((n + 255) / 256), 256, 0, s>>>(mo, B.nsph, nmos, pld, Ct);
  return 2;
}

// Orbitals per thread: the fewest that cover nmos with one block column, at
// most 4 (64 orbitals per block; PT = 4 keeps tile, sums and operands within
// the 128 registers of two blocks per SM).
int std_half_pt(int nmos) { return std::min(4, std::max(1, (nmos + 15) / 16)); }

int launch_std_half(const StdHalfArgs& h, cudaStream_t s) {
  if (h.nk <= 0 || h.B.nsph <= 0 || h.nmos <= 0) return 0;
  switch (std_half_pt(h.nmos)) {
    case 1: return launch_half<1>(h, s);
    case 2: return launch_half<2>(h, s);
    case 3: return launch_half<3>(h, s);
    default: return launch_half<4>(h, s);
  }
}

int launch_std_block_norms(const StdArgs& a, const int* rec_pair, int npairs, double* out, cudaStream_t s) {
  if (npairs <= 0 || a.X.nshells == 0) return 0;
  int done = 0;
  for (int p0 = 0; p0 < npairs; p0 += 65535) {  // grid y limit
    dim3 grid(a.X.nshells, std::min(65535, npairs - p0));
    k_std_block_norm<<<grid, kStdThreads, 0, s>>>(a, rec_pair + p0, a.X.nshells,
                                                 out + static_cast<long long>(p0) * a.X.nshells);
    ++done;
  }
  return done;
}

int launch_std_pack(const double* Res, int nk, int ld, int nmos, const int* col_fn, int naux, double* Raw,
                    cudaStream_t s) {
  const long long total = static_cast<long long>(nmos) * (nmos + 1) / 2 * nk;
  if (total == 0) return 0;
  const int blocks = static_cast<int>(std::min<long long>((total + 255) / 256, 148 * 16));
  k_std_pack<<<blocks, 256, 0, s>>>(Res, nk, ld, nmos, col_fn, naux, Raw);
  return 1;
}

int launch_transpose(const double* in, int rows, int cols, double* out, cudaStream_t s) {
  if (rows <= 0 || cols <= 0) return 0;
  dim3 grid((cols + 31) / 32, (rows + 31) / 32);
  k_transpose<<<grid, dim3(32, 8), 0, s>>>(in, rows, cols, out);
  return 1;
}

}  // namespace pa
