// Densities on grid points and the GDMA primitive density.
//
// f_eval_densities (grid/grid_wrapper.f90:12-38, driver grid/grid.f90:110-286):
//   rho_j(r) = sum_(nu <= mu) f D_j(mu, nu) chi_mu(r) chi_nu(r), f = 1 on the
//   diagonal and 2 off it, over Cartesian basis functions chi in pysisyphus
//   order, with the reference's per-block screening: the points are cut into
//   consecutive blocks of blk_size, and a pair (nu, mu) contributes to a block
//   only when |f D_j(mu, nu) mean_nu mean_mu| >= thresh, mean = the mean |chi|
//   over the block's points.
// f_eval_prim_density (gdma/prim_dens.f90:100-259): the density of the
//   primitive pairs whose total exponent is below `switch`, on grid points.
//
// Both are masked quadratic forms of basis functions at the points,
//   rho(r) = sum_(nu, mu) W(nu, mu) chi_nu(r) chi_mu(r),
// so both kernels run them as products on the FP64 tensor cores (mma.sync
// m8n8k4): a CTA (8 warps, two per SM, persistent over the blocks of points)
//   1. evaluates chi at its block's points into its slice of a scratch array
//      ([function][point]); functions that vanish at all of them are not written;
//   2. compacts the functions that can contribute into an ordered list;
//   3. per 64 functions nu: T[nu][point] = sum_mu W[nu][mu] chi_mu[point], W and
//      chi staged 32 functions mu at a time in shared memory (tiles without a
//      surviving pair are skipped), then rho += sum_nu chi_nu T[nu].
//
// f_eval_densities: W = f D(mu, nu), mu >= nu, where the pair passes the test of
// the block (the block means are sequential sums over the points in order, as
// the reference's, so the decisions are the reference's); the functions of the
// list are those with mean_x dmax_x max_mean >= thresh, dmax_x = the largest
// |f D| of x's pairs.
// f_eval_prim_density: chi are the components of the primitives that have a
// partner within `switch`. exp(-mu |A-B|^2) exp(-p |r-P|^2) of a pair is
// exp(-a |r-A|^2) exp(-b |r-B|^2), so no pair needs an exponential of its own;
// W = f P(a_nu, b_mu), a <= b, under the reference's two tests of the pair.
// The reference drops a pair at points with p |r-P|^2 >= 36; those terms, up to
// 1e-10 of the pair's largest value for two g shells (x^4 e^-x at x = 36 against
// its maximum) and 1e-11 for two f shells, are summed here. A primitive is
// dropped at a block of points where exp(-a |r-A|^2) < 1.8e-35 throughout.
// Non-finite densities, coefficients or centers and exponents that are not
// positive take k_prim_density, which evaluates the reference's pairs one by one.
//
// Bound: latency, of the loads and tests that make up the weight tiles and of the
// exponentials, at 16 warps per SM (counters: FP64 tensor pipe 13 % busy in the grid
// density and 27 % in the primitive density, FP64 pipe 9 and 10 %). Measured on
// B200: 64^3 points around 40 atoms 0.97 ms, 2.0 ms with a broadcast shared-memory
// load per multiply-add; primitive density of 20 atoms at 60 007 points 0.58 ms,
// 5.2 ms pair by pair.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <limits>
#include <mutex>
#include <string>
#include <vector>

#include "pa_internal.h"  // before pa_b200.h: its status macros would rename the enum
#include "pa_b200.h"

namespace pa {
int set_error(int code, const std::string& msg);

namespace {

constexpr double kExpCutoff = -36.0;  // grid.f90:9, prim_dens.f90:13
constexpr double kPrimCutoff = 80.0;  // exponent beyond which a primitive's factor is dropped
constexpr int kGridThreads = 256;
constexpr int kGridWarps = kGridThreads / 32;
constexpr int kTileNu = 64, kTileMu = 32;
constexpr int kLdW = kTileNu + 4;  // 4 (mod 16): conflict-free fragment loads
constexpr int kGridLmax = 4;  // cart_gto3d_rel / prefacts cover s..g

// 1 / sqrt((2i-1)!! (2j-1)!! (2k-1)!!) of every Cartesian component of
// degree <= 4 (cidx order): the NORM2 / NORM3 / NORM4 / NORM22 factors of
// grid.f90:9-13 and prim_dens.f90:7-10.
__constant__ double c_cart_norm[ncum(kGridLmax)];
__constant__ unsigned char c_cart_pow[ncum(kGridLmax)][3];

// Points per product: two column groups of NT 8-point tiles.
template <int NT>
struct QuadTile {
  static constexpr int P = 16 * NT;
  static constexpr int LdX = P + 4;
  static constexpr size_t smem = sizeof(double) * (kTileMu * (kLdW + LdX) + 4 * P);
};

__device__ __forceinline__ void grid_cp16(double* dst, const double* src) {
  const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src));
}

__device__ __forceinline__ void grid_dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// out[p] = sum over listed functions nu, mu of w(mu, nu) chi_nu[p] chi_mu[p] at
// the points p0 .. p0 + np - 1 (np <= P) of the block's slice chi (row stride bp,
// even, rows 16-byte aligned); list positions of mu below nu's tile are not
// visited, so w must vanish for mu < nu. All threads of the CTA; the sums end in
// red[4][P] (rows of the four row groups), complete after the closing barrier.
template <int NT, class W>
__device__ __forceinline__ void quad_form(const int* act, int na, const double* chi, int bp, int p0, int np, W w,
                                          double* sm) {
  using Q = QuadTile<NT>;
  double* Ws = sm;                       // [mu][nu]
  double* Xs = Ws + kTileMu * kLdW;      // [mu][point]
  double* red = Xs + kTileMu * Q::LdX;   // [row group][point]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int g = lane >> 2, t4 = lane & 3, wm = warp & 3, wn = warp >> 2;
  const int nt = min(NT, max(0, (np + 7) / 8 - wn * NT));  // tiles of this warp that hold points
  double sum[NT][2];
#pragma unroll
  for (int n = 0; n < NT; ++n) sum[n][0] = sum[n][1] = 0.0;
  for (int t0 = 0; t0 < na; t0 += kTileNu) {
    double acc[2][NT][2];
#pragma unroll
    for (int m = 0; m < 2; ++m)
#pragma unroll
      for (int n = 0; n < NT; ++n) acc[m][n][0] = acc[m][n][1] = 0.0;
    for (int s0 = t0; s0 < na; s0 += kTileMu) {
      for (int e = tid; e < kTileMu * (Q::P / 2); e += kGridThreads) {
        const int k = e / (Q::P / 2), x = 2 * (e % (Q::P / 2));
        if (s0 + k < na) {
          if (x < np) grid_cp16(Xs + k * Q::LdX + x, chi + static_cast<long long>(act[s0 + k]) * bp + p0 + x);
        } else {
          Xs[k * Q::LdX + x] = Xs[k * Q::LdX + x + 1] = 0.0;
        }
      }
      bool any = false;
#pragma unroll 4
      for (int e = tid; e < kTileMu * kTileNu; e += kGridThreads) {
        const int k = e % kTileMu, m = e / kTileMu;
        const double v = (t0 + m < na && s0 + k < na) ? w(act[s0 + k], act[t0 + m]) : 0.0;
        Ws[k * kLdW + m] = v;
        any = any || v != 0.0;
      }
      asm volatile("cp.async.wait_all;\n" ::);
      if (__syncthreads_or(any)) {
#pragma unroll 2
        for (int q = 0; q < kTileMu; q += 4) {
          double a[2];
#pragma unroll
          for (int m = 0; m < 2; ++m) a[m] = Ws[(q + t4) * kLdW + 16 * wm + 8 * m + g];
#pragma unroll
          for (int n = 0; n < NT; ++n) {
            if (n >= nt) continue;
            const double b = Xs[(q + t4) * Q::LdX + 8 * (wn * NT + n) + g];
#pragma unroll
            for (int m = 0; m < 2; ++m) grid_dmma(acc[m][n][0], acc[m][n][1], a[m], b);
          }
        }
      }
      __syncthreads();  // the tiles are rewritten
    }
#pragma unroll
    for (int m = 0; m < 2; ++m) {
      const int r = t0 + 16 * wm + 8 * m + g;
      if (r >= na) continue;
      const double* row = chi + static_cast<long long>(act[r]) * bp + p0;
#pragma unroll
      for (int n = 0; n < NT; ++n) {
        const int p = 8 * (wn * NT + n) + 2 * t4;
        if (p >= np) continue;
        const double2 x = *reinterpret_cast<const double2*>(row + p);
        sum[n][0] = fma(x.x, acc[m][n][0], sum[n][0]);
        sum[n][1] = fma(x.y, acc[m][n][1], sum[n][1]);
      }
    }
  }
#pragma unroll
  for (int n = 0; n < NT; ++n)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      double v = sum[n][e];
#pragma unroll
      for (int o = 4; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (g == 0) red[wm * Q::P + 8 * (wn * NT + n) + 2 * t4 + e] = v;
    }
  __syncthreads();
}

// Cartesian components of degree L at (x, y, z), times e, to out[c * bp].
template <int L>
__device__ __forceinline__ void write_cart(double x, double y, double z, double e, double* out, int bp) {
  double xp[L + 1], yp[L + 1], zp[L + 1];
  xp[0] = yp[0] = zp[0] = 1.0;
#pragma unroll
  for (int m = 1; m <= L; ++m) {
    xp[m] = xp[m - 1] * x;
    yp[m] = yp[m - 1] * y;
    zp[m] = zp[m - 1] * z;
  }
  int c = 0;
#pragma unroll
  for (int i = L; i >= 0; --i)
#pragma unroll
    for (int j = L - i; j >= 0; --j, ++c)
      out[static_cast<long long>(c) * bp] = c_cart_norm[ncum(L - 1) + c] * xp[i] * yp[j] * zp[L - i - j] * e;
}

__device__ __forceinline__ void write_cart_l(int L, double x, double y, double z, double e, double* out, int bp) {
  switch (L) {
    case 0: write_cart<0>(x, y, z, e, out, bp); break;
    case 1: write_cart<1>(x, y, z, e, out, bp); break;
    case 2: write_cart<2>(x, y, z, e, out, bp); break;
    case 3: write_cart<3>(x, y, z, e, out, bp); break;
    default: write_cart<4>(x, y, z, e, out, bp); break;
  }
}

// Ordered list of the x < n with keep(x), to act; returns its length. All threads.
template <class K>
__device__ __forceinline__ int compact(int n, K keep, int* act, int* s_cnt) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int na = 0;
  for (int base = 0; base < n; base += kGridThreads) {
    const int x = base + tid;
    const bool k = x < n && keep(x);
    const unsigned bal = __ballot_sync(0xffffffffu, k);
    if (lane == 0) s_cnt[warp] = __popc(bal);
    __syncthreads();
    int off = na, tot = 0;
    for (int w = 0; w < kGridWarps; ++w) {
      if (w < warp) off += s_cnt[w];
      tot += s_cnt[w];
    }
    if (k) act[off + __popc(bal & ((1u << lane) - 1u))] = x;
    na += tot;
    __syncthreads();
  }
  return na;
}

struct GridArgs {
  int nshells, ncart, npoints, ndens, nbfs, blk, bp, nblks;
  const int4* shell;      // (L, nprim, prim_off, cart_off)
  const double4* center;  // (x, y, z, 0)
  const double2* prim;    // (exponent, normalized coefficient)
  const double* grid;     // [npoints][3]
  const double* D;        // density j, element (mu, nu) at D[j sj + mu sm + nu sn]
  long long sj, sm, sn;
  const double* dmax;     // [ncart]
  double thresh;
  double* chi;            // [slot][ncart][bp]
  double* mean;           // [slot][ncart]
  int* act;               // [slot][ncart]
  double* rho;            // rho[j + ndens i]
};

// dmax[x] = the largest |f D_j(mu, nu)| of the pairs mu >= nu with x in them.
__global__ void __launch_bounds__(256) k_grid_dmax(GridArgs a, double* dmax) {
  __shared__ double s_red[8];
  const int x = blockIdx.x;
  double m = 0.0;
  for (int j = 0; j < a.ndens; ++j)
    for (int y = threadIdx.x; y < a.nbfs; y += 256) {
      const double d = a.D[j * a.sj + max(x, y) * a.sm + min(x, y) * a.sn];
      m = fmax(m, fabs((x == y ? 1.0 : 2.0) * d));
    }
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) s_red[threadIdx.x >> 5] = m;
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < 8; ++w) m = fmax(m, s_red[w]);
    dmax[x] = m;
  }
}

constexpr int kGridNT = 8;  // 128 points per product

__global__ void __launch_bounds__(kGridThreads, 2) k_grid_density(GridArgs a) {
  extern __shared__ __align__(16) double sm[];
  __shared__ int s_cnt[kGridWarps];
  __shared__ double s_red[kGridWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  double* chi = a.chi + static_cast<long long>(blockIdx.x) * a.ncart * a.bp;
  double* mean = a.mean + static_cast<long long>(blockIdx.x) * a.ncart;
  int* act = a.act + static_cast<long long>(blockIdx.x) * a.ncart;
  for (int blk = blockIdx.x; blk < a.nblks; blk += gridDim.x) {
    const int start = blk * a.blk;
    const int n = min(a.blk, a.npoints - start);
    // 1. chi: a warp per shell, 128 points at a time. A shell that vanishes at
    // all points of the block is marked (mean -1) and not written, unless the
    // test passes everything (thresh 0) or the block has several groups
    const bool whole = n > 128 || !(a.thresh > 0.0);
    for (int sh = warp; sh < a.nshells; sh += kGridWarps) {
      const int4 s = a.shell[sh];
      const double4 C = a.center[sh];
      bool live = whole;
      for (int g0 = 0; g0 < n; g0 += 128) {
        double e[4], x[4], y[4], z[4];
        bool any = false;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int i = g0 + lane + 32 * q;
          e[q] = 0.0;
          if (i < n) {
            const double* R = a.grid + 3LL * (start + i);
            x[q] = R[0] - C.x, y[q] = R[1] - C.y, z[q] = R[2] - C.z;
            const double dist = x[q] * x[q] + y[q] * y[q] + z[q] * z[q];
            for (int p = 0; p < s.y; ++p) {
              const double2 pr = a.prim[s.z + p];
              const double arg = -pr.x * dist;
              if (arg < kExpCutoff) continue;
              e[q] += pr.y * exp(arg);
            }
            // (0 * a non-finite coordinate is NaN: such points count as reached)
            any = any || e[q] != 0.0 || !isfinite(dist);
          }
        }
        live = live || __any_sync(0xffffffffu, any);
        if (live)
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int i = g0 + lane + 32 * q;
            if (i < n) write_cart_l(s.x, x[q], y[q], z[q], e[q], chi + static_cast<long long>(s.w) * a.bp + i, a.bp);
          }
      }
      if (lane < ncart(s.x)) mean[s.w + lane] = live ? 0.0 : -1.0;
    }
    __syncthreads();
    // 2. block means, summed over the points in order
    double mmax = 0.0;
    for (int nu = tid; nu < a.ncart; nu += kGridThreads) {
      double m = 0.0;
      if (mean[nu] == 0.0) {
        const double* row = chi + static_cast<long long>(nu) * a.bp;
#pragma unroll 8
        for (int i = 0; i < n; ++i) m += fabs(row[i]);
        m /= n;
      }
      mean[nu] = m;
      mmax = fmax(mmax, m);
    }
    for (int o = 16; o > 0; o >>= 1) mmax = fmax(mmax, __shfl_xor_sync(0xffffffffu, mmax, o));
    if (lane == 0) s_red[warp] = mmax;
    __syncthreads();
    mmax = s_red[0];
    for (int w = 1; w < kGridWarps; ++w) mmax = fmax(mmax, s_red[w]);
    // the functions that can pass the test (a superset: the bound is relaxed by
    // 1e-12 for rounding)
    const int na = compact(
        a.ncart, [&](int nu) { return mean[nu] * a.dmax[nu] * mmax >= a.thresh * (1.0 - 1e-12); }, act, s_cnt);
    // 3. masked pair products, per density and per group of points
    for (int j = 0; j < a.ndens; ++j) {
      const double* D = a.D + j * a.sj;
      auto w = [&](int mu, int nu) {
        if (mu < nu) return 0.0;
        const double f = nu == mu ? 1.0 : 2.0;
        const double d = D[mu * a.sm + nu * a.sn];
        const double contrib = f * d * mean[nu] * mean[mu];
        return fabs(contrib) >= a.thresh ? f * d : 0.0;
      };
      using Q = QuadTile<kGridNT>;
      for (int p0 = 0; p0 < n; p0 += Q::P) {
        const int np = min(Q::P, n - p0);
        quad_form<kGridNT>(act, na, chi, a.bp, p0, np, w, sm);
        const double* red = sm + kTileMu * (kLdW + Q::LdX);
        if (tid < np)
          a.rho[j + static_cast<long long>(a.ndens) * (start + p0 + tid)] =
              (red[tid] + red[Q::P + tid]) + (red[2 * Q::P + tid] + red[3 * Q::P + tid]);
        __syncthreads();
      }
    }
  }
}

// GDMA: a primitive that has partners, and a Cartesian function of it.
struct PrimFn {
  double ax, da, A[3];
  int L, fn0, i0, pad;  // first function, Cartesian start in P
};

struct PrimArgs {
  int nprim, nfn, npoints, blk, nblks;
  const PrimFn* prim;
  const int* fn_prim;     // function -> primitive
  const double* coords;   // [npoints][3]
  const double* P;        // element (i, j) at P[i si + j sj]
  long long si, sj;
  double sw;
  double* chi;            // [slot][nfn][blk]
  int* act;               // [slot][nfn]
  int* live;              // [slot][nprim]
  double* rho;
};

template <int NT>
__global__ void __launch_bounds__(kGridThreads, 2) k_prim_product(PrimArgs a) {
  extern __shared__ __align__(16) double sm[];
  __shared__ int s_cnt[kGridWarps];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  constexpr int P = QuadTile<NT>::P;
  double* chi = a.chi + static_cast<long long>(blockIdx.x) * a.nfn * P;
  int* act = a.act + static_cast<long long>(blockIdx.x) * a.nfn;
  int* live = a.live + static_cast<long long>(blockIdx.x) * a.nprim;
  for (int blk = blockIdx.x; blk < a.nblks; blk += gridDim.x) {
    const int start = blk * P;
    const int n = min(P, a.npoints - start);
    for (int k = warp; k < a.nprim; k += kGridWarps) {
      const PrimFn& f = a.prim[k];
      double e[P / 32], x[P / 32], y[P / 32], z[P / 32];
      bool any = false;
#pragma unroll
      for (int q = 0; q < P / 32; ++q) {
        const int i = lane + 32 * q;
        e[q] = x[q] = y[q] = z[q] = 0.0;
        if (i < n) {
          const double* R = a.coords + 3LL * (start + i);
          x[q] = R[0] - f.A[0], y[q] = R[1] - f.A[1], z[q] = R[2] - f.A[2];
          const double arg = f.ax * (x[q] * x[q] + y[q] * y[q] + z[q] * z[q]);
          if (arg >= kPrimCutoff)
            x[q] = y[q] = z[q] = 0.0;  // (a point at infinity: 0, as the reference's cutoff gives)
          else {
            e[q] = f.da * exp(-arg);
            any = true;
          }
        }
      }
      any = __any_sync(0xffffffffu, any);
      if (any)
#pragma unroll
        for (int q = 0; q < P / 32; ++q)
          write_cart_l(f.L, x[q], y[q], z[q], e[q], chi + static_cast<long long>(f.fn0) * P + lane + 32 * q, P);
      if (lane == 0) live[k] = any ? 1 : 0;
    }
    __syncthreads();
    const int na = compact(a.nfn, [&](int fn) { return live[a.fn_prim[fn]] != 0; }, act, s_cnt);
    auto w = [&](int mu, int nu) {
      // both orders of two functions of one primitive are taken at mu > nu
      if (mu < nu) return 0.0;
      const int ia = a.fn_prim[nu], ib = a.fn_prim[mu];
      const PrimFn& fa = a.prim[ia];
      const PrimFn& fb = a.prim[ib];
      const double px = fa.ax + fb.ax;
      if (px >= a.sw) return 0.0;
      // prim_dens.f90:212 squares the sum of the differences (kept as is)
      const double dsum = (fa.A[0] - fb.A[0]) + (fa.A[1] - fb.A[1]) + (fa.A[2] - fb.A[2]);
      const double mux = fa.ax * fb.ax / px;
      if (-mux * dsum * dsum <= kExpCutoff) return 0.0;
      const int i = fa.i0 + nu - fa.fn0, j = fb.i0 + mu - fb.fn0;
      const double p = a.P[i * a.si + j * a.sj];
      if (ia != ib) return 2.0 * p;
      return mu == nu ? p : p + a.P[j * a.si + i * a.sj];
    };
    quad_form<NT>(act, na, chi, P, 0, n, w, sm);
    const double* red = sm + kTileMu * (kLdW + QuadTile<NT>::LdX);
    if (tid < n) a.rho[start + tid] = (red[tid] + red[P + tid]) + (red[2 * P + tid] + red[3 * P + tid]);
    __syncthreads();  // the slice is rewritten by the next block
  }
}

__device__ __forceinline__ double ipow(double x, int n) {
  double r = 1.0;
  for (int m = 0; m < n; ++m) r *= x;
  return r;
}

// GDMA primitive pairs (host-filtered, in the reference's ai <= bi order).
struct PrimPairG {
  double K, px, P[3], A[3], B[3];
  int La, Lb, ia, ib;
};

__device__ __forceinline__ void cart_prefactors(int L, double x, double y, double z, double* out) {
  const int c0 = ncum(L - 1), nc = ncart(L);
  for (int c = 0; c < nc; ++c) {
    const unsigned char* pw = c_cart_pow[c0 + c];
    out[c] = c_cart_norm[c0 + c] * ipow(x, pw[0]) * ipow(y, pw[1]) * ipow(z, pw[2]);
  }
}

constexpr int kPairChunk = 64;

__global__ void __launch_bounds__(128) k_prim_density(const PrimPairG* __restrict__ pairs, int npairs,
                                                      const double* __restrict__ coords, int npoints,
                                                      const double* __restrict__ P, long long si, long long sj,
                                                      double* __restrict__ rho) {
  __shared__ PrimPairG sp[kPairChunk];
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const bool pt = i < npoints;
  double R[3] = {0.0, 0.0, 0.0};
  if (pt)
    for (int d = 0; d < 3; ++d) R[d] = coords[3LL * i + d];
  double acc = 0.0;
  double pa[ncart(kGridLmax)], pb[ncart(kGridLmax)];
  for (int c0 = 0; c0 < npairs; c0 += kPairChunk) {
    const int nc = min(kPairChunk, npairs - c0);
    __syncthreads();
    for (int k = threadIdx.x; k < nc; k += blockDim.x) sp[k] = pairs[c0 + k];
    __syncthreads();
    if (!pt) continue;
    for (int k = 0; k < nc; ++k) {
      const PrimPairG& q = sp[k];
      const double dx = R[0] - q.P[0], dy = R[1] - q.P[1], dz = R[2] - q.P[2];
      const double r2 = dx * dx + dy * dy + dz * dz;
      if (-q.px * r2 <= kExpCutoff) continue;
      const double pexp = exp(-q.px * r2);
      cart_prefactors(q.La, R[0] - q.A[0], R[1] - q.A[1], R[2] - q.A[2], pa);
      cart_prefactors(q.Lb, R[0] - q.B[0], R[1] - q.B[1], R[2] - q.B[2], pb);
      const int na = ncart(q.La), nb = ncart(q.Lb);
      double s = 0.0;
      for (int nu = 0; nu < na; ++nu) {
        double t = 0.0;
        for (int mu = 0; mu < nb; ++mu)
          t = fma(__ldg(P + (q.ia + nu) * si + (q.ib + mu) * sj), pb[mu], t);
        s = fma(pa[nu], t, s);
      }
      acc = fma(q.K * pexp, s, acc);
    }
  }
  if (pt) rho[i] = acc;
}

std::once_flag g_tables_once[64];
cudaError_t g_tables_err[64];

cudaError_t upload_cart_tables() {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  std::call_once(g_tables_once[dev], [dev]() {
    double norm[ncum(kGridLmax)];
    unsigned char pw[ncum(kGridLmax)][3];
    auto df = [](int k) {  // (2k - 1)!!
      double r = 1.0;
      for (int m = 2 * k - 1; m > 1; m -= 2) r *= m;
      return r;
    };
    int idx = 0;
    for (int L = 0; L <= kGridLmax; ++L)
      for (int x = L; x >= 0; --x)
        for (int y = L - x; y >= 0; --y, ++idx) {
          const int z = L - x - y;
          norm[idx] = 1.0 / std::sqrt(df(x) * df(y) * df(z));
          pw[idx][0] = static_cast<unsigned char>(x);
          pw[idx][1] = static_cast<unsigned char>(y);
          pw[idx][2] = static_cast<unsigned char>(z);
        }
    g_tables_err[dev] = cudaMemcpyToSymbol(c_cart_norm, norm, sizeof(norm));
    if (g_tables_err[dev] == cudaSuccess) g_tables_err[dev] = cudaMemcpyToSymbol(c_cart_pow, pw, sizeof(pw));
  });
  return g_tables_err[dev];
}

// Per device: a memory pool that keeps up to kPoolKeep bytes mapped between
// calls (a call's allocations otherwise map and unmap device memory, 2.7 of 8.9
// ms for 64^3 points) and up to kStreamsKeep idle streams; both are given back
// by release_grid_pools (pa_basis_cache_clear). Never destroyed: no CUDA calls
// run during process teardown.
constexpr unsigned long long kPoolKeep = 512ull << 20;
constexpr size_t kStreamsKeep = 8;
struct GridDevice {
  std::mutex mu;
  cudaMemPool_t pool = nullptr;
  std::vector<cudaStream_t> idle;
};
GridDevice& grid_device(int dev) {
  static GridDevice* d = new GridDevice[64];
  return d[dev];
}

// One call's stream and device memory (a single allocation), given back when
// the call returns.
struct CallBuf {
  int dev = -1;
  cudaStream_t s = nullptr;
  char* base = nullptr;
  size_t used = 0;
  cudaError_t open() {
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
    GridDevice& d = grid_device(dev);
    std::lock_guard<std::mutex> lk(d.mu);
    if (!d.pool) {
      cudaMemPoolProps props{};
      props.allocType = cudaMemAllocationTypePinned;
      props.location.type = cudaMemLocationTypeDevice;
      props.location.id = dev;
      e = cudaMemPoolCreate(&d.pool, &props);
      if (e != cudaSuccess) {
        d.pool = nullptr;
        return e;
      }
      unsigned long long keep = kPoolKeep;
      e = cudaMemPoolSetAttribute(d.pool, cudaMemPoolAttrReleaseThreshold, &keep);
      if (e != cudaSuccess) return e;
    }
    if (!d.idle.empty()) {
      s = d.idle.back();
      d.idle.pop_back();
      return cudaSuccess;
    }
    return cudaStreamCreateWithFlags(&s, cudaStreamNonBlocking);
  }
  // carving: count with base == nullptr, allocate, carve again
  template <class T>
  T* take(size_t n) {
    T* p = base ? reinterpret_cast<T*>(base + used) : nullptr;
    used += (n * sizeof(T) + 255) & ~size_t(255);
    return p;
  }
  cudaError_t allocate() {
    const cudaError_t e = cudaMallocFromPoolAsync(reinterpret_cast<void**>(&base), std::max<size_t>(used, 256),
                                                  grid_device(dev).pool, s);
    if (e != cudaSuccess) base = nullptr;
    used = 0;
    return e;
  }
  ~CallBuf() {
    if (!s) return;
    if (base) cudaFreeAsync(base, s);
    cudaStreamSynchronize(s);
    GridDevice& d = grid_device(dev);
    std::lock_guard<std::mutex> lk(d.mu);
    if (d.idle.size() < kStreamsKeep)
      d.idle.push_back(s);
    else
      cudaStreamDestroy(s);
  }
};

#define PA_GRID_CUDA(x)                                                                                  \
  do {                                                                                                   \
    const cudaError_t e_ = (x);                                                                          \
    if (e_ != cudaSuccess) return set_error(PA_ERR_CUDA, std::string(#x ": ") + cudaGetErrorString(e_)); \
  } while (0)


// Tables of a call in one host buffer, for one upload.
struct Staged {
  std::vector<char> bytes;
  template <class T>
  size_t put(const std::vector<T>& v) {
    const size_t off = bytes.size();
    bytes.resize(off + ((v.size() * sizeof(T) + 255) & ~size_t(255)));
    if (!v.empty()) std::memcpy(bytes.data() + off, v.data(), v.size() * sizeof(T));
    return off;
  }
};

// Density j, element (mu, nu) at densities[j sj + mu sm + nu sn].
int eval_densities(int nshells, int ndata, const int* bas_centers, const int* bas_spec, const double* bas_data,
                   int npoints, const double* grid3d, int ndens, int nbfs, const double* densities, long long sj,
                   long long sm, long long sn, double* grid_densities, int blk_size, double thresh) {
  HostBasis b;
  std::string err;
  int st = unpack_basis(nshells, ndata, bas_centers, bas_spec, bas_data, kGridLmax, &b, &err);
  if (st != PA_OK) return set_error(st, "f_eval_densities: " + err);
  int ncart_tot = 0;
  for (const HostShell& s : b.shells) ncart_tot += ncart(s.L);
  if (npoints < 0 || ndens < 0 || nbfs != ncart_tot)
    return set_error(PA_ERR_ARG, "f_eval_densities: nbfs (" + std::to_string(nbfs) +
                                     ") must equal the Cartesian size of the basis (" + std::to_string(ncart_tot) + ")");
  if (blk_size < 1 || blk_size > 4096) return set_error(PA_ERR_ARG, "f_eval_densities: blk_size must be in [1, 4096]");
  if (!(thresh >= 0.0) || !std::isfinite(thresh)) return set_error(PA_ERR_ARG, "f_eval_densities: thresh must be >= 0");
  if ((npoints > 0 && (!grid3d || !grid_densities)) || (ndens > 0 && nbfs > 0 && !densities))
    return set_error(PA_ERR_ARG, "f_eval_densities: null array");
  if (npoints == 0 || ndens == 0) return PA_OK;
  if (nbfs == 0) {
    std::fill(grid_densities, grid_densities + static_cast<size_t>(ndens) * npoints, 0.0);
    return PA_OK;
  }
  PA_GRID_CUDA(upload_cart_tables());
  std::vector<int4> shell(b.shells.size());
  std::vector<double4> center(b.shells.size());
  std::vector<double2> prim(b.exps.size());
  int off = 0;
  for (size_t k = 0; k < b.shells.size(); ++k) {
    const HostShell& s = b.shells[k];
    shell[k] = make_int4(s.L, s.nprim, s.prim_off, off);
    center[k] = make_double4(s.A[0], s.A[1], s.A[2], 0.0);
    off += ncart(s.L);
  }
  for (size_t p = 0; p < b.exps.size(); ++p) prim[p] = make_double2(b.exps[p], b.coefs[p]);
  Staged tab;
  const size_t o_shell = tab.put(shell), o_center = tab.put(center), o_prim = tab.put(prim);
  CallBuf buf;
  PA_GRID_CUDA(buf.open());
  GridArgs a;
  a.nshells = static_cast<int>(b.shells.size());
  a.ncart = nbfs;
  a.npoints = npoints;
  a.ndens = ndens;
  a.nbfs = nbfs;
  a.blk = blk_size;
  a.bp = (blk_size + 1) / 2 * 2;
  a.nblks = (npoints + blk_size - 1) / blk_size;
  a.thresh = thresh;
  a.sj = sj;
  a.sm = sm;
  a.sn = sn;
  int sms = 148;
  PA_GRID_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, buf.dev));
  // slots of the chi scratch: the resident CTAs (two per SM), at most ~1 GiB in total
  const size_t slot_bytes = sizeof(double) * (static_cast<size_t>(nbfs) * a.bp + nbfs) + sizeof(int) * nbfs;
  int slots = std::min(a.nblks, 2 * sms);
  slots = std::max(1, std::min<int>(slots, static_cast<int>((size_t(1) << 30) / slot_bytes)));
  const size_t nD = static_cast<size_t>(ndens) * nbfs * nbfs;
  char* d_tab = nullptr;
  double *d_grid = nullptr, *d_D = nullptr, *d_dmax = nullptr;
  for (int pass = 0; pass < 2; ++pass) {
    if (pass == 1) PA_GRID_CUDA(buf.allocate());
    d_tab = buf.take<char>(tab.bytes.size());
    d_grid = buf.take<double>(3 * static_cast<size_t>(npoints));
    d_D = buf.take<double>(nD);
    d_dmax = buf.take<double>(nbfs);
    a.chi = buf.take<double>(static_cast<size_t>(slots) * nbfs * a.bp);
    a.mean = buf.take<double>(static_cast<size_t>(slots) * nbfs);
    a.act = buf.take<int>(static_cast<size_t>(slots) * nbfs);
    a.rho = buf.take<double>(static_cast<size_t>(ndens) * npoints);
  }
  PA_GRID_CUDA(cudaMemcpyAsync(d_tab, tab.bytes.data(), tab.bytes.size(), cudaMemcpyHostToDevice, buf.s));
  PA_GRID_CUDA(cudaMemcpyAsync(d_D, densities, sizeof(double) * nD, cudaMemcpyHostToDevice, buf.s));
  a.shell = reinterpret_cast<const int4*>(d_tab + o_shell);
  a.center = reinterpret_cast<const double4*>(d_tab + o_center);
  a.prim = reinterpret_cast<const double2*>(d_tab + o_prim);
  a.grid = d_grid;
  a.D = d_D;
  a.dmax = d_dmax;
  k_grid_dmax<<<nbfs, 256, 0, buf.s>>>(a, d_dmax);  // runs while the points are copied
  PA_GRID_CUDA(cudaMemcpyAsync(d_grid, grid3d, sizeof(double) * 3 * npoints, cudaMemcpyHostToDevice, buf.s));
  const size_t smem = QuadTile<kGridNT>::smem;
  PA_GRID_CUDA(cudaFuncSetAttribute(k_grid_density, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  k_grid_density<<<slots, kGridThreads, smem, buf.s>>>(a);
  PA_GRID_CUDA(cudaGetLastError());
  PA_GRID_CUDA(cudaMemcpyAsync(grid_densities, a.rho, sizeof(double) * ndens * static_cast<size_t>(npoints),
                               cudaMemcpyDeviceToHost, buf.s));
  PA_GRID_CUDA(cudaStreamSynchronize(buf.s));
  return PA_OK;
}

template <int NT>
int launch_prim_product(PrimArgs a, Staged& tab, size_t o_prim, size_t o_fn, const double* coords3d, const double* P,
                        size_t nP, double* rho, int sms, CallBuf& buf) {
  constexpr int pts = QuadTile<NT>::P;
  a.blk = pts;
  a.nblks = (a.npoints + pts - 1) / pts;
  const size_t slot_bytes = sizeof(double) * static_cast<size_t>(a.nfn) * pts + sizeof(int) * (a.nfn + a.nprim);
  int slots = std::min(a.nblks, 2 * sms);
  slots = std::max(1, std::min<int>(slots, static_cast<int>((size_t(1) << 30) / std::max<size_t>(slot_bytes, 1))));
  char* d_tab = nullptr;
  double *d_coords = nullptr, *d_P = nullptr;
  for (int pass = 0; pass < 2; ++pass) {
    if (pass == 1) PA_GRID_CUDA(buf.allocate());
    d_tab = buf.take<char>(tab.bytes.size());
    d_coords = buf.take<double>(3 * static_cast<size_t>(a.npoints));
    d_P = buf.take<double>(nP);
    a.chi = buf.take<double>(static_cast<size_t>(slots) * a.nfn * pts);
    a.act = buf.take<int>(static_cast<size_t>(slots) * a.nfn);
    a.live = buf.take<int>(static_cast<size_t>(slots) * a.nprim);
    a.rho = buf.take<double>(a.npoints);
  }
  if (!tab.bytes.empty())
    PA_GRID_CUDA(cudaMemcpyAsync(d_tab, tab.bytes.data(), tab.bytes.size(), cudaMemcpyHostToDevice, buf.s));
  PA_GRID_CUDA(cudaMemcpyAsync(d_coords, coords3d, sizeof(double) * 3 * a.npoints, cudaMemcpyHostToDevice, buf.s));
  if (nP) PA_GRID_CUDA(cudaMemcpyAsync(d_P, P, sizeof(double) * nP, cudaMemcpyHostToDevice, buf.s));
  a.prim = reinterpret_cast<const PrimFn*>(d_tab + o_prim);
  a.fn_prim = reinterpret_cast<const int*>(d_tab + o_fn);
  a.coords = d_coords;
  a.P = d_P;
  const size_t smem = QuadTile<NT>::smem;
  PA_GRID_CUDA(cudaFuncSetAttribute(k_prim_product<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem)));
  k_prim_product<NT><<<slots, kGridThreads, smem, buf.s>>>(a);
  PA_GRID_CUDA(cudaGetLastError());
  PA_GRID_CUDA(cudaMemcpyAsync(rho, a.rho, sizeof(double) * a.npoints, cudaMemcpyDeviceToHost, buf.s));
  PA_GRID_CUDA(cudaStreamSynchronize(buf.s));
  return PA_OK;
}

// Element (i, j) of the density matrix at P[i si + j sj].
int eval_prim_density(int nprims, int npoints, int nbfs, const int* ls_inds, const double* primdata,
                      const double* coords3d, const double* P, long long si, long long sj, double sw, double* rho) {
  if (nprims < 0 || npoints < 0 || nbfs < 0) return set_error(PA_ERR_ARG, "f_eval_prim_density: negative size");
  if ((nprims > 0 && (!ls_inds || !primdata)) || (npoints > 0 && (!coords3d || !rho)) || (nbfs > 0 && !P))
    return set_error(PA_ERR_ARG, "f_eval_prim_density: null array");
  for (int ai = 0; ai < nprims; ++ai) {
    const int La = ls_inds[2 * ai], ia = ls_inds[2 * ai + 1];
    if (La < 0 || La > kGridLmax)
      return set_error(PA_ERR_LMAX, "f_eval_prim_density: primitive " + std::to_string(ai) + " has L = " +
                                        std::to_string(La) + " (s..g supported)");
    if (ia < 0 || ia + ncart(La) > nbfs)
      return set_error(PA_ERR_ARG, "f_eval_prim_density: primitive " + std::to_string(ai) +
                                       ": Cartesian index outside the density matrix");
  }
  if (npoints == 0) return PA_OK;
  PA_GRID_CUDA(upload_cart_tables());
  const size_t nP = static_cast<size_t>(nbfs) * nbfs;
  // the product form needs finite factors: 0 * inf of a dropped pair would be NaN
  double amin = std::numeric_limits<double>::infinity(), bad[8] = {};
  bool plain = true;
  for (int ai = 0; ai < nprims; ++ai) {
    for (int d = 0; d < 5; ++d) plain = plain && std::isfinite(primdata[5 * ai + d]);
    plain = plain && primdata[5 * ai + 1] > 0.0;
    amin = std::min(amin, primdata[5 * ai + 1]);
  }
  for (size_t k = 0; k + 8 <= nP; k += 8)
    for (int q = 0; q < 8; ++q) bad[q] += 0.0 * P[k + q];
  for (size_t k = nP / 8 * 8; k < nP; ++k) bad[0] += 0.0 * P[k];
  for (double b : bad) plain = plain && b == 0.0;
  CallBuf buf;
  PA_GRID_CUDA(buf.open());
  if (plain) {
    // primitives with a partner, in their order, and their functions
    std::vector<PrimFn> prim;
    std::vector<int> fn_prim;
    for (int ai = 0; ai < nprims; ++ai) {
      const double* d = primdata + 5 * ai;
      if (d[1] + amin >= sw) continue;
      PrimFn f;
      f.da = d[0];
      f.ax = d[1];
      for (int k = 0; k < 3; ++k) f.A[k] = d[2 + k];
      f.L = ls_inds[2 * ai];
      f.i0 = ls_inds[2 * ai + 1];
      f.fn0 = static_cast<int>(fn_prim.size());
      f.pad = 0;
      fn_prim.insert(fn_prim.end(), ncart(f.L), static_cast<int>(prim.size()));
      prim.push_back(f);
    }
    Staged tab;
    const size_t o_prim = tab.put(prim), o_fn = tab.put(fn_prim);
    PrimArgs a{};
    a.nprim = static_cast<int>(prim.size());
    a.nfn = static_cast<int>(fn_prim.size());
    a.npoints = npoints;
    a.si = si;
    a.sj = sj;
    a.sw = sw;
    int sms = 148;
    PA_GRID_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, buf.dev));
    // 64 points per block, 32 where 64 would leave SMs without a block
    if (npoints < 64 * sms) return launch_prim_product<2>(a, tab, o_prim, o_fn, coords3d, P, nP, rho, sms, buf);
    return launch_prim_product<4>(a, tab, o_prim, o_fn, coords3d, P, nP, rho, sms, buf);
  }
  std::vector<PrimPairG> pairs;
  for (int ai = 0; ai < nprims; ++ai) {
    const double da = primdata[5 * ai], ax = primdata[5 * ai + 1];
    const double* A = primdata + 5 * ai + 2;
    for (int bi = ai; bi < nprims; ++bi) {
      const double db = primdata[5 * bi], bx = primdata[5 * bi + 1];
      if (ax + bx >= sw) continue;
      const double* B = primdata + 5 * bi + 2;
      const double px = ax + bx, mux = ax * bx / px;
      // prim_dens.f90:212 squares the sum of the differences (kept as is)
      const double dsum = (A[0] - B[0]) + (A[1] - B[1]) + (A[2] - B[2]);
      if (-mux * dsum * dsum <= kExpCutoff) continue;
      const double AB2 = (A[0] - B[0]) * (A[0] - B[0]) + (A[1] - B[1]) * (A[1] - B[1]) + (A[2] - B[2]) * (A[2] - B[2]);
      PrimPairG q;
      q.K = da * db * (ai == bi ? 1.0 : 2.0) * std::exp(-mux * AB2);
      q.px = px;
      for (int d = 0; d < 3; ++d) {
        q.P[d] = (ax * A[d] + bx * B[d]) / px;
        q.A[d] = A[d];
        q.B[d] = B[d];
      }
      q.La = ls_inds[2 * ai];
      q.ia = ls_inds[2 * ai + 1];
      q.Lb = ls_inds[2 * bi];
      q.ib = ls_inds[2 * bi + 1];
      pairs.push_back(q);
    }
  }
  PrimPairG* d_pairs = nullptr;
  double *d_coords = nullptr, *d_P = nullptr, *d_rho = nullptr;
  for (int pass = 0; pass < 2; ++pass) {
    if (pass == 1) PA_GRID_CUDA(buf.allocate());
    d_pairs = buf.take<PrimPairG>(pairs.size());
    d_coords = buf.take<double>(3 * static_cast<size_t>(npoints));
    d_P = buf.take<double>(nP);
    d_rho = buf.take<double>(npoints);
  }
  if (!pairs.empty())
    PA_GRID_CUDA(cudaMemcpyAsync(d_pairs, pairs.data(), sizeof(PrimPairG) * pairs.size(), cudaMemcpyHostToDevice, buf.s));
  PA_GRID_CUDA(cudaMemcpyAsync(d_coords, coords3d, sizeof(double) * 3 * npoints, cudaMemcpyHostToDevice, buf.s));
  if (nP) PA_GRID_CUDA(cudaMemcpyAsync(d_P, P, sizeof(double) * nP, cudaMemcpyHostToDevice, buf.s));
  k_prim_density<<<(npoints + 127) / 128, 128, 0, buf.s>>>(d_pairs, static_cast<int>(pairs.size()), d_coords,
                                                           npoints, d_P, si, sj, d_rho);
  PA_GRID_CUDA(cudaGetLastError());
  PA_GRID_CUDA(cudaMemcpyAsync(rho, d_rho, sizeof(double) * npoints, cudaMemcpyDeviceToHost, buf.s));
  PA_GRID_CUDA(cudaStreamSynchronize(buf.s));
  return PA_OK;
}

}  // namespace

void release_grid_pools() {
  for (int dev = 0; dev < 64; ++dev) {
    GridDevice& d = grid_device(dev);
    std::lock_guard<std::mutex> lk(d.mu);
    for (cudaStream_t s : d.idle) cudaStreamDestroy(s);
    d.idle.clear();
    if (d.pool) cudaMemPoolTrimTo(d.pool, 0);
  }
}

}  // namespace pa

using namespace pa;

extern "C" {

int f_eval_densities(int nshells, int ndata, const int* bas_centers, const int* bas_spec, const double* bas_data,
                     int npoints, const double* grid3d, int ndens, int nbfs, const double* densities,
                     double* grid_densities, int blk_size, double thresh) {
  return eval_densities(nshells, ndata, bas_centers, bas_spec, bas_data, npoints, grid3d, ndens, nbfs, densities, 1,
                        ndens, static_cast<long long>(ndens) * nbfs, grid_densities, blk_size, thresh);
}

int pa_eval_densities(int nshells, int ndata, const int* bas_centers, const int* bas_spec, const double* bas_data,
                      int npoints, const double* grid3d, int ndens, int nbfs, const double* densities, int layout,
                      double* grid_densities, int blk_size, double thresh) {
  if (layout == PA_LAYOUT_FORTRAN)
    return f_eval_densities(nshells, ndata, bas_centers, bas_spec, bas_data, npoints, grid3d, ndens, nbfs, densities,
                            grid_densities, blk_size, thresh);
  if (layout != PA_LAYOUT_C) return set_error(PA_ERR_ARG, "unknown layout");
  return eval_densities(nshells, ndata, bas_centers, bas_spec, bas_data, npoints, grid3d, ndens, nbfs, densities,
                        static_cast<long long>(nbfs) * nbfs, nbfs, 1, grid_densities, blk_size, thresh);
}

int f_eval_prim_density(int nprims, int npoints, int nbfs, const int* ls_inds, const double* primdata,
                        const double* coords3d, const double* P, double sw, double* rho) {
  return eval_prim_density(nprims, npoints, nbfs, ls_inds, primdata, coords3d, P, 1, nbfs, sw, rho);
}

int pa_eval_prim_density(int nprims, int npoints, int nbfs, const int* ls_inds, const double* primdata,
                         const double* coords3d, const double* P, int layout, double sw, double* rho) {
  if (layout != PA_LAYOUT_FORTRAN && layout != PA_LAYOUT_C) return set_error(PA_ERR_ARG, "unknown layout");
  const bool c = layout == PA_LAYOUT_C;
  return eval_prim_density(nprims, npoints, nbfs, ls_inds, primdata, coords3d, P, c ? nbfs : 1, c ? 1 : nbfs, sw, rho);
}

}  // extern "C"
