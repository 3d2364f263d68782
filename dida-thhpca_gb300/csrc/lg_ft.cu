// lg_ft.cu -- FP64 transform of up to 64 members from the tridiagonal form,
// without eigenvalues: W = sqrt(k-1) A^(-1/2), A = C + (k-1)/rho I = Q T Q^T.
//
// letkf_core.F90:98-225 diagonalises A; only W x (the state rows, or every unit
// vector for an explicit trans) and overline_w = A^-1 t are used.  Both are
// functions of T applied to vectors, so after the Householder reduction
// (lg_tri.cu) this kernel computes, per vector, y = Q^T x, f(T) y and
// Q f(T) y, with
//   T^(-1/2) = sum_j w_j (T + s_j I)^-1,
// the N-point midpoint rule of (2/pi) int_0^inf (T + s^2)^-1 ds in the variable
// u of s = sqrt(m) sc(u | k'), k'^2 = 1 - m/M, which is periodic and analytic
// when the eigenvalues of T lie in [m, M] (N. Hale, N. J. Higham and
// L. N. Trefethen, "Computing A^alpha, log(A) and related matrix functions by
// contour integrals", SIAM J. Numer. Anal. 46, 2008).  Its relative error is
// 4 exp(-2 pi N K/K'), so 15 nodes reach 2^-54 at M/m = 100 and 33 at 10^6.
// Here m = (k-1)/rho bounds the spectrum from below and Gershgorin's circles
// bound it from above.  Every (T + s_j I) is positive definite: the LDL^T
// recurrences need no pivoting, all weights are positive, nothing cancels.
//
// Why: the FP64 pipe retires a warp instruction per 17 cycles per SM.  Per
// 64-member solve the QL iteration takes about 4000 rotations at 24 FP64
// instructions (one lane each) and their replay 8 per rotation and vector; the
// shifted solves take 3 per node, element and vector, plus 8 per node and
// element for the factors, which the lanes of a solve compute for different
// nodes.  overline_w . x = (T^(-1/2) y) . (T^(-1/2) Q^T t) needs no solve of its
// own.  The reflections (2 k^2 multiply-adds per vector) leave the FP64 pipe
// altogether: a vector's norm does not change, so they run in fixed point on the
// integer pipe as the reduction does (lg_tri.cu), to 2^-58 of the norm per step, two
// reflectors at a time (reading and rounding the vector once for both took the
// explicit trans of those cubes from 7.2 to 6.6 ms).
//   rows (analysis): reflect_kernel (Q^T), ft_kernel, reflect_kernel (Q) with the
//     rows' update -- three kernels, so that the integer ones are not held to the
//     two to four warps per SM that the solves' five arrays leave;
//   explicit trans: ft_matrix_kernel forms F = f(T) itself, whose upper triangle
//     takes 1 FP64 instruction per node and element (no right-hand side: with
//     T + s = L D L^T, G = (T + s)^-1 has G_jj = 1/D_j + L_{j+1}^2 G_{j+1,j+1} and
//     G_ij = -L_{i+1} G_{i+1,j} above it), then W = Q F Q^T by two reflect_kernel
//     passes and overline_w = W (W t) / (k - 1) in add_wbar_kernel.  A solve per
//     unit vector instead made this step 12.9 ms where it is 6.4 (32 768 cubes of
//     40 members).
// The sum over the nodes is kept in 64-bit integers: off the FP64 pipe, and the same
// in any order, so that a vector may be spread over several lanes (launch_ft) and the
// result does not depend on how many solves a launch has.
// Measured alone against QL + replay: 921 600 solves of 40 members 233 -> 55 ms,
// 129 600 of 64 members 93 -> 22 ms; explicit trans against the accumulating solver
// (lg_eig.cu), with the reduction: 32 768 cubes of 40 members 133 -> 8.3 ms.  Faster at
// every size from 7 to 64 members; above, five arrays leave an SM one warp.
#include <float.h>
#include <math.h>

#include <algorithm>
#include <mutex>
#include <type_traits>

#include "lg_device.cuh"
#include "lg_fixed.cuh"
#include "lg_internal.h"

namespace lg {
namespace ft {

// M/m up to 2^43: Gershgorin's bound is below 3 |C| + m, |C| at most 2^(kFtLog + 1) m
constexpr int kMaxLog = kFtLog + 3;
constexpr int kMaxNodes = 72;  // nodes per row of the table (65 at 2^43), padded with zero weight
// [log2(M/m)][node]: (s_j / m, w_j / sqrt(m))
__device__ double2 g_nodes[kMaxLog + 1][kMaxNodes];
__device__ int g_count[kMaxLog + 1];

// complete elliptic integral K of the modulus whose complementary modulus is kc
double agm_k(double kc) {
  double a = 1.0, b = kc;
  for (int i = 0; i < 40 && fabs(a - b) > 1e-15 * a; ++i) {
    const double t = 0.5 * (a + b);
    b = sqrt(a * b);
    a = t;
  }
  return acos(-1.0) / (a + b);
}

// S = sc(u | k') = sn / cn of the modulus with complementary modulus k, for u
// up to K(k')/2, by Gauss's transformation in its hyperbolic form (sc(u | k') =
// -i sn(iu | k)): S(u, k) = (1 + k1) S1 / (1 - k1 S1^2) with k1 = (1 - k*) / (1 +
// k*), k*^2 = 1 - k^2, S1 = S(u / (1 + k1), k1); sinh(u) at k = 0
double jacobi_sc(double u, double k) {
  if (k < 1e-18) return sinh(u);
  const double ks = sqrt((1.0 - k) * (1.0 + k));
  const double k1 = k * k / ((1.0 + ks) * (1.0 + ks));
  const double s1 = jacobi_sc(u / (1.0 + k1), k1);
  return (1.0 + k1) * s1 / (1.0 - k1 * s1 * s1);
}

}  // namespace ft

// the node table on the current device (once per device)
int prepare_ft_nodes() {
  constexpr int kMaxDevices = 64;
  static bool done[kMaxDevices] = {};
  static std::mutex mu;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return LG_ERR_CUDA;
  std::lock_guard<std::mutex> lock(mu);
  if (done[dev]) return LG_OK;
  static double2 nodes[ft::kMaxLog + 1][ft::kMaxNodes];
  static int count[ft::kMaxLog + 1];
  if (count[1] == 0) {
    const double pi = acos(-1.0);
    for (int q = 1; q <= ft::kMaxLog; ++q) {
      const double kk = exp2(-0.5 * q);                  // k = sqrt(m/M)
      const double Kp = ft::agm_k(kk);                   // K(k')
      const double K = ft::agm_k(sqrt((1.0 - kk) * (1.0 + kk)));
      const int N = (int)ceil((log(4.0) + 54.0 * log(2.0)) / (2.0 * pi * K / Kp));
      count[q] = N;
      const double c = 2.0 * Kp / (pi * N);
      for (int j = 0; 2 * j < N; ++j) {
        // u < K'/2 directly; the mirror node K' - u from sc(K'-u) = 1 / (k sc u),
        // dn/cn^2 (K'-u) = dn / (k sn^2) (u): both keep their relative accuracy
        const double sc = ft::jacobi_sc((j + 0.5) * Kp / N, kk);
        const double icn2 = 1.0 + sc * sc;                        // 1 / cn^2
        const double dn = sqrt((1.0 + kk * kk * sc * sc) / icn2);  // dn^2 = cn^2 + k^2 sn^2
        nodes[q][j] = make_double2(sc * sc, c * dn * icn2);
        nodes[q][N - 1 - j] = make_double2(1.0 / (kk * sc * kk * sc), c * dn * icn2 / (kk * sc * sc));
      }
    }
    for (int j = 0; j < ft::kMaxNodes; ++j) nodes[0][j] = nodes[1][j];
    count[0] = count[1];
  }
  // (a copy from pageable memory may return before its transfer is complete, and a caller's
  // stream need not wait for the legacy one)
  if (cudaMemcpyToSymbol(ft::g_nodes, nodes, sizeof nodes) != cudaSuccess ||
      cudaMemcpyToSymbol(ft::g_count, count, sizeof count) != cudaSuccess ||
      cudaStreamSynchronize(cudaStreamLegacy) != cudaSuccess) {
    cudaGetLastError();
    return LG_ERR_CUDA;
  }
  done[dev] = true;
  return LG_OK;
}

namespace ft {

__device__ inline double rcp(double x) {  // x normal: two Newton steps from the approximation
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  r = fma(r, fma(-x, r, 1.0), r);
  return fma(r, fma(-x, r, 1.0), r);
}

__device__ inline void cp_async8(void* dst, const void* src) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(
                   (unsigned)__cvta_generic_to_shared(dst)),
               "l"(src)
               : "memory");
}

// Vectors of an analysis call: vector v of solve s -- 0: t (kept in the t array's
// place), v >= 1: the state row v - 1 (in `vec`, element i at
// ((s (n + 1) + i) (per - 1) + v - 1), element n being overline_w . x).  Core
// calls: column v of the solve's n x n matrix in `vec` (trans).
struct Vecs {
  int per;
  double* t;
  double* vec;
};
__device__ inline double* vec_at(const Vecs& z, int n, size_t s, int v, int& stride) {
  if (v == 0) {
    stride = 1;
    return z.t + s * n;
  }
  stride = z.per - 1;
  return z.vec + s * (n + 1) * (z.per - 1) + (v - 1);
}
__device__ inline size_t out_index(const SolveBatch& b, int s) {
  return b.s_col ? (size_t)b.first_solve + s : (size_t)s;
}

// A vector of n elements over kL neighbouring lanes: lane part p holds elements
// p, p + kL, .. at 0, 32, 64, ..; own(n) of them.  All lanes of the warp call it.
template <int kL>
__device__ inline int own(int n, int part) {
  return kL == 1 ? n : (n - part + kL - 1) / kL;
}
template <int kL, typename T>
__device__ inline T sum_parts(T x) {
#pragma unroll
  for (int o = 1; o < kL; o *= 2) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}

// Sum of f(i) over a vector's elements (i: this lane's, of m) in an order that does
// not depend on kL: eight sums of the elements equal modulo 8, joined as a tree.
template <int kL, typename F>
__device__ inline double sum_elements(int m, F f) {
  constexpr int kC = 8 / kL;
  double c[kC];
#pragma unroll
  for (int q = 0; q < kC; ++q) c[q] = 0.0;
  for (int i = 0; i < m; i += kC) {
#pragma unroll
    for (int q = 0; q < kC; ++q)
      if (i + q < m) c[q] += f(i + q);
  }
#pragma unroll
  for (int q = 0; q < kC; ++q) c[q] = sum_parts<kL>(c[q]);
#pragma unroll
  for (int o = 1; o < kC; o *= 2)
#pragma unroll
    for (int q = 0; q < kC; q += 2 * o) c[q] += c[q + o];
  return c[0];
}

// a += x in units of 2^(top - 62), for |x| < 2^top, Eb = top + 1022 >= 62: sums of
// the nodes' terms, exact in any order and off the FP64 pipe
__device__ inline void add_fixed(long long& a, double x, int Eb) {
  const int hi = __double2hiint(x);
  const unsigned long long m =
      ((unsigned long long)((hi & 0xfffff) | 0x100000) << 32 | (unsigned)__double2loint(x)) << 9;
  const long long v = (long long)(m >> min(max(Eb - ((hi >> 20) & 0x7ff), 0), 63));
  a += hi < 0 ? -v : v;
}
// power of two above f(T)'s norm, sqrt(rho) at most
__device__ inline int f_top(double inflation) {
  return ((__double2hiint(1.01 * sqrt(inflation)) >> 20) & 0x7ff) - 1022;
}

// This vector V from FP64 to integers of 2^(ex): |V| < 2^(ex + 58), held as in
// lg_tri.cu; false if a value is not finite.  m: this lane's elements.
template <int kL>
__device__ inline bool to_fixed(double* V, int m, int& ex) {
  unsigned emax = 0;
  for (int i = 0; i < m; ++i)
    emax = max(emax, ((unsigned)__double2hiint(V[32 * i]) >> 20) & 0x7ffu);
#pragma unroll
  for (int o = 1; o < kL; o *= 2) emax = max(emax, __shfl_xor_sync(0xffffffffu, emax, o));
  // norm < 2^(emax - 1043) sqrt(squares), in integers (any order); the power of two
  // above it
  unsigned long long squares = 0;
  for (int i = 0; i < m; ++i) {
    const int hi = __double2hiint(V[32 * i]) & 0x7fffffff;
    const unsigned f =
        ((((unsigned)hi & 0xfffffu) | 0x100000u) + 1 >> min((int)emax - (hi >> 20), 31)) + 1;
    squares += (unsigned long long)f * f;
  }
  squares = sum_parts<kL>(squares);
  const int Eb = (int)emax - 20 + (65 - __clzll((long long)squares)) / 2;
  for (int i = 0; i < m; ++i) {
    const unsigned long long u = (unsigned long long)__double_as_longlong(V[32 * i]);
    const int e = (int)(u >> 52) & 0x7ff;
    long long x = 0;
    if (e) {
      const int sh = min(max(Eb - e, 1), 62);
      x = (long long)((((u & 0xfffffffffffffull) | 0x10000000000000ull) << 6) + (1ull << (sh - 1))) >> sh;
      if (u >> 63) x = -x;
    }
    reinterpret_cast<int2*>(V)[32 * i] = fixed_split(x);
  }
  ex = Eb - 1023 - 58;
  return emax < 2047;
}

}  // namespace ft

namespace ft {
// T of a solve that the reduction left to the eigenvalue route
__device__ inline bool left_alone(const double* T) {
  return (unsigned long long)__double_as_longlong(T[1]) == kLeftMark;
}
}  // namespace ft

// One vector over kL lanes, one warp per block, lanes numbered through the solves'
// vectors.  Analysis: y <- Q^T x (kFirst; P_{n-1} first) or Q z (P_1 first) with
// the rows' update.  Core, W = Q F Q^T: the first pass takes column j of the
// symmetric F from row j of the matrix and leaves Q F's column j there (the
// matrix then holds (Q F)^T); the second takes column j -- row j of Q F -- and
// leaves W's column j there, so that no lane reads what another one writes.
// Reflector rows of the (up to `slots`) solves that a warp spans come into shared
// memory, two at a time, a step ahead of their use.
template <bool kFirst, bool kCore, int kL>
__global__ void __launch_bounds__(32) reflect_kernel(Geometry g, SolveBatch b, ft::Vecs z,
                                                     int slots, const double* tri, const double* xb,
                                                     const double* axb, double* xa, double* axa) {
  const int n = g.ens;
  const int lane = threadIdx.x;
  // the rows' update needs no t: its vectors are v = 1 .. per - 1
  const int v0 = !kFirst && !kCore ? 1 : 0;
  const int per = z.per - v0;
  constexpr int kV = 32 / kL;  // vectors of a warp
  const long long id0 = (long long)blockIdx.x * kV, total = (long long)b.nsolves * per;
  const int s_first = (int)(id0 / per);
  const int nsl = (int)((min(id0 + kV, total) - 1) / per) - s_first + 1;
  const long long id = id0 + lane / kL;
  const int part = kL == 1 ? 0 : lane % kL, m = ft::own<kL>(n, part);
  const bool mine = id < total;
  const int s = mine ? (int)(id / per) : s_first;
  const int v = v0 + (mine ? (int)(id - (long long)s * per) : 0);
  extern __shared__ double sm[];
  double* const Y = sm + lane;                      // element part + kL i at 32 i
  int2* const Yi = reinterpret_cast<int2*>(Y);
  double* const ub = sm + 32 * ((n + kL - 1) / kL);  // two buffers of slots x 2 n
  const size_t tri_stride = (size_t)n * n;
  // pair m, 1 .. n / 2: reflectors 2 m and 2 m - 1 as rows A and B, B padded with a
  // zero, and w_A . w_B behind A; for even n the last pair is reflector n - 1 alone
  auto fetch = [&](int m, int buf) {
    if (m >= 1 && m <= n / 2)
      for (int sl = 0; sl < nsl; ++sl) {
        const double* T = tri + (size_t)(s_first + sl) * tri_stride;
        double* d = ub + (size_t)(buf * slots + sl) * 2 * n;
        const bool two = 2 * m < n;
        const int la = two ? 2 * m : n - 1;
        const double* u = T + 3 * n + (size_t)la * (la - 1) / 2;
        for (int c = lane; c < la; c += 32) {
          ft::cp_async8(d + c, u + c);
          if (two && c < la - 1)
            ft::cp_async8(d + n + c, u - (la - 1) + c);
          else
            d[n + c] = 0.0;
        }
        if (lane == 0) {
          if (two)
            ft::cp_async8(d + n - 1, T + 2 * n + la);
          else
            d[n - 1] = 0.0;
        }
      }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  constexpr bool kDown = kFirst && !kCore;  // Q^T
  const int step = kDown ? -1 : 1, m0 = kDown ? n / 2 : 1;
  fetch(m0, 0);
  // ---- the vector
  int r_state = -1;
  size_t ci = 0;
  double* out;
  int vs;
  if (kCore) {
    out = z.vec + ft::out_index(b, s) * n * n + (kFirst ? (size_t)v * n : (size_t)v);
    vs = kFirst ? 1 : n;
  } else {
    out = ft::vec_at(z, n, s, v, vs);
    const int col = b.first_col + s / b.levels;
    const int kk = s % b.levels + 1;
    const int glat = col % g.num_lat + 1, glon = col / g.num_lat + 1;
    ci = (size_t)(glat - 1 + g.halo) + (size_t)(g.num_lat + 2 * g.halo) * (size_t)(glon - 1 + g.halo);
    if (v >= 1) {
      if (g.vert_dist <= 0.0)
        r_state = v - 1;
      else if (g.var_lev[v - 1] > 1)
        r_state = g.var_start[v - 1] + kk - 1;
      else if (kk == g.nz)
        r_state = g.var_start[v - 1];
    }
  }
  const bool row = mine && r_state >= 0;  // analysis: this solve updates the row
  const double* const xr = xb + (row ? (size_t)n * (r_state + (size_t)g.n * ci) : 0);
  for (int i = 0; i < m; ++i) {
    const int e = part + kL * i;
    double x = 0.0;
    if (kCore)
      x = out[(size_t)e * vs];
    else if (kFirst)
      x = v == 0 ? out[e] : (row ? xr[e] : 0.0);
    else if (row)
      x = out[(size_t)e * vs];
    Y[32 * i] = x;
  }
  int ex;
  const bool finite = ft::to_fixed<kL>(Y, m, ex);
  // ---- two reflections at a time: y -= w1 d1 + w2 d2, d1 = w1 . y, d2 = w2 . y -
  // (w1 . w2) d1, so that y is read twice and rounded once for both
  for (int c = 0, mp = m0; c < n / 2; ++c, mp += step) {
    fetch(mp + step, (c + 1) & 1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    const int2* const ud =
        reinterpret_cast<const int2*>(ub + (size_t)((c & 1) * slots + (s - s_first)) * 2 * n);
    const int2 *uA = ud + part, *uB = ud + n + part;
    const int2 g2 = ud[n - 1];
    const int mi = ft::own<kL>(min(2 * mp, n - 1), part);
    long long hA = 0, hB = 0, mA = part == 0 ? 1 << 27 : 0, mB = mA;  // rounds the sum's cut
#pragma unroll 4
    for (int j = 0; j < mi; ++j) {
      const int2 y = Yi[32 * j], w = uA[kL * j], x = uB[kL * j];
      hA += (long long)y.y * w.y;
      mA += (long long)y.y * w.x;
      mA += (long long)y.x * w.y;
      hB += (long long)y.y * x.y;
      mB += (long long)y.y * x.x;
      mB += (long long)y.x * x.y;
    }
    long long dA = 4 * ft::sum_parts<kL>(hA) + (ft::sum_parts<kL>(mA) >> 28);
    long long dB = 4 * ft::sum_parts<kL>(hB) + (ft::sum_parts<kL>(mB) >> 28);
    const int2 D1 = fixed_split(kDown ? dA : dB);
    const long long cross = 4 * ((long long)D1.y * g2.y) +
                            (((long long)D1.y * g2.x + (long long)D1.x * g2.y + (1 << 27)) >> 28);
    const int2 D2 = fixed_split((kDown ? dB : dA) - cross);
    const int2 DA = kDown ? D1 : D2, DB = kDown ? D2 : D1;
    const int A4 = -4 * DA.y, B4 = -4 * DB.y;  // |D| < 2^58.5
#pragma unroll 4
    for (int j = 0; j < mi; ++j) {
      const int2 w = uA[kL * j], x = uB[kL * j], y = Yi[32 * j];
      long long c2 = (long long)DA.y * w.x + ((long long)DA.x * w.y + (1 << 27));
      c2 += (long long)DB.y * x.x;
      c2 += (long long)DB.x * x.y;
      Yi[32 * j] = fixed_split(fixed_join(y) + (long long)A4 * w.y + (long long)B4 * x.y - (c2 >> 28));
    }
    __syncwarp();
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  // ---- out
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  if (kFirst || kCore) {
    if (mine)
      for (int i = 0; i < m; ++i)
        out[(size_t)(part + kL * i) * vs] =
            finite ? fixed_to_double(fixed_join(Yi[32 * i]), ex) : nan;
    return;
  }
  // xa = axb + sqrt(rho) x + (W - sqrt(rho) I) x + overline_w . x, recentred
  const double srho = sqrt(g.inflation);
  const double ab = row ? axb[r_state + (size_t)g.n * ci] : 0.0;
  const double dotw = row ? out[(size_t)n * vs] : 0.0;
  const double mean = ft::sum_elements<kL>(m, [&](int i) {
    if (!row) return 0.0;
    const double d = finite ? fixed_to_double(fixed_join(Yi[32 * i]), ex) : nan;
    const double x = ab + (srho * xr[part + kL * i] + (d + dotw));
    Y[32 * i] = x;
    return x;
  }) / (double)n;
  if (!row) return;
  // ft_kernel made the rows of a solve left to the eigenvalue route NaN: they stay as that
  // route wrote them
  if (!finite && ft::left_alone(tri + (size_t)s * tri_stride)) return;
  double* xo = xa + (size_t)n * (r_state + (size_t)g.n * ci);
  for (int i = 0; i < m; ++i) xo[part + kL * i] = Y[32 * i] - mean;
  if (part == 0) axa[r_state + (size_t)g.n * ci] = mean;
}

namespace ft {

// One warp: T's diagonals of the solves s_first .. + nsl - 1 into Dg (with the
// shift) and Eg, and each one's row of the node table (Gershgorin in FP32,
// rounded up).  A non-finite T counts in *eig_fail, as a QL iteration that never
// converges, if its first vector id is not below id0 (a solve left alone has the mark
// for its second diagonal element: NaN, but not counted).
__device__ inline void load_t(int n, const double* tri, int s_first, int nsl, double shift, double* Dg,
                              double* Eg, int* s_row, bool* s_nan, int per, long long id0,
                              int* eig_fail) {
  const int lane = threadIdx.x;
  for (int q = 0; q < nsl; ++q) {
    const double* T = tri + (size_t)(s_first + q) * n * n;
    for (int i = lane; i < n; i += 32) {
      Dg[q * n + i] = T[i] + shift;
      Eg[q * n + i] = T[n + i];
    }
    __syncwarp();
    float mx = 0.0f;
    bool nf = false;
    for (int i = lane; i < n; i += 32) {
      const double d = Dg[q * n + i], e0 = Eg[q * n + i], e1 = i + 1 < n ? Eg[q * n + i + 1] : 0.0;
      nf |= ((__double2hiint(d) >> 20) & 0x7ff) == 0x7ff || ((__double2hiint(e0) >> 20) & 0x7ff) == 0x7ff;
      mx = fmaxf(mx, fabsf(d2f_bits(d)) + fabsf(d2f_bits(e0)) + fabsf(d2f_bits(e1)));
    }
    nf = __any_sync(0xffffffffu, nf);
    mx = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mx)));
    if (lane == 0) {
      // smallest power of two above the bound
      const int ex = (int)((__float_as_uint(mx * (1.0001f / (float)shift)) >> 23) & 0xffu) - 127 + 1;
      s_row[q] = nf ? 0 : min(max(ex, 1), kMaxLog);
      s_nan[q] = nf;
      if (nf && (long long)(s_first + q) * per >= id0 && !left_alone(T)) atomicAdd(eig_fail, 1);
    }
  }
  __syncwarp();
}

// reciprocal pivots R and multipliers L (L[32 i] of the edge i - 1, i) of T +
// sigma = L D L^T for this lane's (slot, node) pair
__device__ inline void factor(int n, const double* D, const double* E, double sigma, double* R,
                              double* L) {
  double r = rcp(D[0] + sigma);
  R[0] = r;
#pragma unroll 2
  for (int i = 1; i < n; ++i) {
    const double e = E[i], l = e * r;
    r = rcp(fma(-l, e, D[i] + sigma));
    L[32 * i] = l;
    R[32 * i] = r;
  }
}

// The same elimination from both ends, meeting at element m = n / 2: as many
// operations in two independent chains of half the length.
// R is scaled by the node's weight w, which makes the solution w (T + sigma)^-1 y.
template <int kPW>
__device__ inline void factor_twisted(int n, const double* D, const double* E, double sigma, double w,
                                      double* R, double* L) {
  const int m = n / 2, nd = n - 1 - m;  // nd elements below m, m >= nd above
  double r = rcp(D[0] + sigma), q = rcp(D[n - 1] + sigma);
  R[0] = w * r;
  R[kPW * (n - 1)] = w * q;
  for (int c = 1; c < nd; ++c) {
    const int b = n - 1 - c;
    const double e = E[c], l = e * r, h = E[b + 1], k = h * q;
    r = rcp(fma(-l, e, D[c] + sigma));
    q = rcp(fma(-k, h, D[b] + sigma));
    L[kPW * c] = l;
    R[kPW * c] = w * r;
    L[kPW * (b + 1)] = k;
    R[kPW * b] = w * q;
  }
  if (m > nd) {
    const double e = E[m - 1], l = e * r;
    r = rcp(fma(-l, e, D[m - 1] + sigma));
    L[kPW * (m - 1)] = l;
    R[kPW * (m - 1)] = w * r;
  }
  const double e = E[m], l = e * r, h = E[m + 1], k = h * q;
  L[kPW * m] = l;
  L[kPW * (m + 1)] = k;
  R[kPW * m] = w * rcp(fma(-k, h, fma(-l, e, D[m] + sigma)));
}

}  // namespace ft

// f(T) y per lane, one warp per block: t gives sqrt(k-1) T^(-1/2) y, the rows
// (f(T) - sqrt(rho)) y and overline_w . x.  A warp takes `slots` solves, each with t and
// its rows (at most 15: solves of more rows take the eigenvalue route, eig2_supported).
// Shared memory, [element][lane] so that lanes never conflict: Y (the vector),
// F (the forward solve), A (the sum over nodes), and for kPW (slot, node) pairs
// the reciprocal pivots R and multipliers L of T + s; T's diagonals per slot.
template <int kL, int kPW>
__global__ void __launch_bounds__(32) ft_kernel(Geometry g, SolveBatch b, ft::Vecs z, int slots,
                                                const double* tri, int* eig_fail) {
  const int n = g.ens;
  const int lane = threadIdx.x;
  const int lanes = z.per * kL;  // of a solve
  const int s_first = (int)blockIdx.x * slots;
  const int nsl = min(slots, b.nsolves - s_first);
  const int sl = lane / lanes < nsl ? lane / lanes : 0, s = s_first + sl;
  const int part = lane % kL;  // this lane's nodes: part, part + kL, ..
  const bool mine = lane / lanes < nsl;
  const int v = mine ? (lane - sl * lanes) / kL : 0;  // 0: t
  extern __shared__ double sm[];
  const int cap = n * 32;
  double *const Y = sm + lane, *const F = Y + cap;
  long long* const A = reinterpret_cast<long long*>(F + cap);  // in units of 2^(top - 62)
  double *const R = sm + 3 * cap, *const L = R + kPW * n;
  double* const Dg = L + kPW * n;         // slots x n: diagonal + shift
  double* const Eg = Dg + slots * n;  // slots x n: Eg[i] couples i - 1 and i
  __shared__ int s_row[32];
  __shared__ bool s_nan[32];
  const double shift = (double)(n - 1) / g.inflation;
  int vs;
  double* const io = ft::vec_at(z, n, s, v, vs);
  if (mine)
#pragma unroll 4
    for (int i = 0; i < n; ++i) Y[32 * i] = io[(size_t)i * vs];
  ft::load_t(n, tri, s_first, nsl, shift, Dg, Eg, s_row, s_nan, 1, 0, eig_fail);
  const int nb = kPW / slots;  // nodes per batch: pair (slot, node) = slot + slots * node
  int nmax = 0;
  for (int q = 0; q < nsl; ++q) nmax = max(nmax, ft::g_count[s_row[q]]);
  const int fs = lane % slots, fj = lane / slots;
  const double wscale = sqrt((double)(n - 1) * shift);  // sqrt(k - 1) sqrt(m)
  // |f(T) y| < 2^top.  From 128 on, so that add_fixed shifts a zero's leading one out: a
  // vector of zeros (a state row without spread, t of an empty list) stays exactly zero.
  unsigned emax = 128;
  for (int i = 0; i < n; ++i) {
    A[32 * i] = 0;
    if (mine) emax = max(emax, ((unsigned)__double2hiint(Y[32 * i]) >> 20) & 0x7ffu);
  }
  const int top = (int)emax - 1022 + 3 + ft::f_top(g.inflation), Eb = top + 1022;
  const int m = n / 2, nd = n - 1 - m;
  auto solve = [&](int pair) {
    // A += w (T + s)^-1 y with the pair's twisted factors: inwards, then outwards
    // from element m, both chains one fused multiply-add per element; the next
    // element's operands are read ahead of the chains' stores
    const double *Rp = R + pair, *Lp = L + pair;
    double f = Y[0], h = Y[32 * (n - 1)];
    F[0] = f;
    F[32 * (n - 1)] = h;
    double lf = Lp[kPW], yf = Y[32], lh = Lp[kPW * (n - 1)], yh = Y[32 * (n - 2)];
#pragma unroll 4
    for (int c = 1; c < nd; ++c) {
      const int b = n - 1 - c;
      f = fma(-lf, f, yf);
      h = fma(-lh, h, yh);
      lf = Lp[kPW * (c + 1)];
      yf = Y[32 * (c + 1)];
      lh = Lp[kPW * b];
      yh = Y[32 * (b - 1)];
      F[32 * c] = f;
      F[32 * b] = h;
    }
    if (m > nd) {
      f = fma(-lf, f, yf);
      F[32 * (m - 1)] = f;
    }
    double u = Rp[kPW * m] * fma(-Lp[kPW * (m + 1)], h, fma(-Lp[kPW * m], f, Y[32 * m]));
    ft::add_fixed(A[32 * m], u, Eb);
    double d = u;
    int iu = m - 1, id = m + 1;
    double lu = Lp[kPW * m], gu = Rp[kPW * iu] * F[32 * iu];
    double ld = Lp[kPW * id], gd = Rp[kPW * id] * F[32 * id];
#pragma unroll 4
    for (int c = 1; c < nd; ++c) {
      u = fma(-lu, u, gu);
      d = fma(-ld, d, gd);
      const int ju = iu - 1, jd = id + 1;
      lu = Lp[kPW * iu];
      gu = Rp[kPW * ju] * F[32 * ju];
      ld = Lp[kPW * jd];
      gd = Rp[kPW * jd] * F[32 * jd];
      ft::add_fixed(A[32 * iu], u, Eb);
      ft::add_fixed(A[32 * id], d, Eb);
      iu = ju;
      id = jd;
    }
    u = fma(-lu, u, gu);
    ft::add_fixed(A[32 * iu], u, Eb);
    ft::add_fixed(A[32 * id], fma(-ld, d, gd), Eb);
    if (m > nd) ft::add_fixed(A[0], fma(-Lp[kPW], u, Rp[0] * F[0]), Eb);
  };
  for (int j0 = 0; j0 < nmax; j0 += nb) {
    if (fs < nsl && fj < nb && j0 + fj < nmax) {
      const double2 node = ft::g_nodes[s_row[fs]][j0 + fj];
      ft::factor_twisted<kPW>(n, Dg + fs * n, Eg + fs * n, node.x * shift, node.y * wscale, R + lane,
                         L + lane);
    }
    __syncwarp();
    if (mine)
      for (int j = part; j < nb && j0 + j < nmax; j += kL) solve(sl + slots * j);
    __syncwarp();
  }
  // ---- out
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  const bool finite = emax < 2047u && !s_nan[sl];
  double* const Af = reinterpret_cast<double*>(A);
  for (int i = 0; i < n; ++i) {
    const long long a = ft::sum_parts<kL>(A[32 * i]);
    Af[32 * i] = finite ? fixed_to_double(a, top - 62) : nan;
  }
  __syncwarp();
  const bool row = mine && v > 0;
  const double srho = sqrt(g.inflation);
  const double* zt = sm + 2 * cap + sl * lanes;  // vector 0's A
  const double dotw = ft::sum_elements<kL>(ft::own<kL>(n, part), [&](int q) {
    if (!row) return 0.0;
    const int i = part + kL * q;
    const double a = Af[32 * i];
    io[(size_t)i * vs] = fma(-srho, Y[32 * i], a);
    return a * zt[32 * i];
  });
  if (row && part == 0) io[(size_t)n * vs] = dotw / (double)(n - 1);
}

// F = f(T) of each solve, symmetric, into its n x n matrix: one column per lane,
// lanes numbered through the solves' columns, one warp per block.  Shared memory
// as in ft_kernel: A (the column), and per (slot, node) pair L and the diagonal G
// of (T + s)^-1 (R first).
template <int kL>
__global__ void __launch_bounds__(32) ft_matrix_kernel(Geometry g, SolveBatch b, ft::Vecs z, int slots,
                                                       const double* tri, int* eig_fail) {
  const int n = g.ens;
  const int lane = threadIdx.x;
  constexpr int kV = 32 / kL;  // columns of a warp
  const long long id0 = (long long)blockIdx.x * kV, total = (long long)b.nsolves * n;
  const int s_first = (int)(id0 / n);
  const int nsl = (int)((min(id0 + kV, total) - 1) / n) - s_first + 1;
  const long long id = id0 + lane / kL;
  const int part = lane % kL;  // this lane's nodes: part, part + kL, ..
  const bool mine = id < total;
  const int s = mine ? (int)(id / n) : s_first, sl = s - s_first;
  const int v = mine ? (int)(id - (long long)s * n) : 0;
  extern __shared__ double sm[];
  const int cap = n * 32;
  long long* const A = reinterpret_cast<long long*>(sm) + lane;  // in units of 2^(top - 62)
  double *const G = sm + cap, *const L = G + cap;
  double* const Dg = L + cap;
  double* const Eg = Dg + slots * n;
  __shared__ int s_row[32];
  __shared__ bool s_nan[32];
  const double shift = (double)(n - 1) / g.inflation;
  ft::load_t(n, tri, s_first, nsl, shift, Dg, Eg, s_row, s_nan, n, id0, eig_fail);
  const int nb = 32 / slots;
  int nmax = 0;
  for (int q = 0; q < nsl; ++q) nmax = max(nmax, ft::g_count[s_row[q]]);
  const int fs = lane % slots, fj = lane / slots;
  const double wscale = sqrt((double)(n - 1) * shift);  // sqrt(k - 1) sqrt(m)
  for (int i = 0; i < n; ++i) A[32 * i] = 0;
  const int top = ft::f_top(g.inflation), Eb = top + 1022;
  const int vmax = (int)__reduce_max_sync(0xffffffffu, (unsigned)v);
  for (int j0 = 0; j0 < nmax; j0 += nb) {
    if (fs < nsl && fj < nb && j0 + fj < nmax) {
      const double2 node = ft::g_nodes[s_row[fs]][j0 + fj];
      ft::factor(n, Dg + fs * n, Eg + fs * n, node.x * shift, G + lane, L + lane);
      // the weighted diagonal w G_jj, from the last element up, in R's place
      const double w = node.y * wscale;
      double gd = w * G[32 * (n - 1) + lane];
      G[32 * (n - 1) + lane] = gd;
      for (int i = n - 2; i >= 0; --i) {
        const double l = L[32 * (i + 1) + lane];
        gd = fma(l, l * gd, w * G[32 * i + lane]);
        G[32 * i + lane] = gd;
      }
    }
    __syncwarp();
    // two nodes' chains at a time, one read of A for both (32 768 cubes 6.57 -> 6.40
    // ms); one past the last keeps x = 0
    const int nn = min(nb, nmax - j0);
    for (int j = part; j < nn; j += 2 * kL) {
      const bool two = j + kL < nn;
      const int p0 = sl + slots * j, p1 = two ? p0 + slots * kL : p0;
      const double *L0 = L + p0, *L1 = L + p1;
      const double g0 = G[32 * v + p0], g1 = two ? G[32 * v + p1] : 0.0;
      double x0 = 0.0, x1 = 0.0;
#pragma unroll 4
      for (int i = vmax; i >= 0; --i) {
        // above the diagonal x is not begun yet, on it it starts
        const double s0 = i < n - 1 ? -L0[32 * (i + 1)] * x0 : 0.0;
        const double s1 = i < n - 1 ? -L1[32 * (i + 1)] * x1 : 0.0;
        x0 = i == v ? g0 : s0;
        x1 = i == v ? g1 : s1;
        if (i <= v) {
          long long a = A[32 * i];
          ft::add_fixed(a, x0, Eb);
          ft::add_fixed(a, x1, Eb);
          A[32 * i] = a;
        }
      }
    }
    __syncwarp();
  }
  if (kL > 1)
    for (int i = 0; i <= vmax; ++i) A[32 * i] = ft::sum_parts<kL>(A[32 * i]);
  if (!mine) return;
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  const bool finite = !s_nan[sl];
  double* const out = z.vec + ft::out_index(b, s) * n * n;
  for (int i = part; i <= v; i += kL) {
    const double x = finite ? fixed_to_double(A[32 * i], top - 62) : nan;
    out[(size_t)i * n + v] = x;
    out[(size_t)v * n + i] = x;
  }
}

// overline_w = W (W t) / (k - 1), trans(i, j) = W(i, j) + overline_w(i),
// column-major (W is symmetric).  W comes into shared memory once, and a column's
// products are spread over 128 / k threads: 16.7 -> 9.7 us for one solve of 40
// members (a chain of loads before), 0.43 -> 0.36 ms for 32 768.
__global__ void __launch_bounds__(128) add_wbar_kernel(int n, SolveBatch b, const double* tin,
                                                       double* trans, double* wbar) {
  const int s = blockIdx.x, tid = threadIdx.x;
  const size_t so = ft::out_index(b, s);
  double* To = trans + so * n * n;
  extern __shared__ double W[];  // n x n
  __shared__ double t[64], sums[128];
  const int parts = 128 / n, part = tid / n, i0 = tid - part * n;
#pragma unroll 8
  for (int r = tid; r < n * n; r += 128) W[r] = To[r];
  if (tid < n) t[tid] = tin[(size_t)s * n + tid];
  __syncthreads();
#pragma unroll
  for (int pass = 0; pass < 2; ++pass) {  // t <- W t
    if (part < parts) {
      double d = 0.0;
#pragma unroll 4
      for (int j = part; j < n; j += parts) d = fma(W[i0 + n * j], t[j], d);
      sums[tid] = d;
    }
    __syncthreads();
    if (tid < n) {
      double d = sums[tid];
      for (int p = 1; p < parts; ++p) d += sums[p * n + tid];
      t[tid] = pass == 0 ? d : d / (double)(n - 1);
    }
    __syncthreads();
  }
  if (wbar && tid < n) wbar[so * n + tid] = t[tid];
  const int step = 128 - parts * n;
  for (int r = tid, i = i0; r < n * n; r += 128) {
    To[r] = W[r] + t[i];
    i += step;
    if (i >= n) i -= n;
  }
}

bool ft_supported(const Geometry& g) {
  // below 7 members the tridiagonal form does not fit the Gram matrix's place;
  // a lowered sweep limit asks for the QL iteration; a shift (k - 1) / rho far from any
  // inflation in use would leave FP32's range in load_t and the nodes' in factor
  const double shift = (double)(g.ens - 1) / g.inflation;
  return g.ens >= 7 && g.ens <= 64 && (g.ql_max_iter == 0 || g.ql_max_iter >= 60) &&
         shift > 0x1p-100 && shift < 0x1p100;
}

size_t ft_vec_doubles(const Geometry& g) {
  return (size_t)(g.ens + 1) * (g.vert_dist > 0.0 ? g.n_var : g.n);
}

void launch_ft(const Geometry& g, const SolveBatch& b, bool core, double* t, const double* tri,
               double* vec, const double* xb, const double* axb, double* xa, double* axa,
               double* wbar, int* eig_fail, cudaStream_t stream) {
  if (b.nsolves == 0) return;
  const int n = g.ens;
  const int per = core ? n : 1 + (g.vert_dist > 0.0 ? g.n_var : g.n);
  const ft::Vecs z{per, t, vec};
  auto with = [](int lanes, auto f) {
    switch (lanes) {
      case 8: f(std::integral_constant<int, 8>()); break;
      case 4: f(std::integral_constant<int, 4>()); break;
      case 2: f(std::integral_constant<int, 2>()); break;
      default: f(std::integral_constant<int, 1>());
    }
  };
  auto smem_of = [&](auto kernel, size_t doubles) {
    const size_t smem = sizeof(double) * doubles;
    allow_smem(kernel, smem);
    return smem;
  };
  // solves that the vectors of a warp can touch, p to a solve, and warps
  auto spans = [](int p, int vectors) { return (vectors + p - 2) / p + 1; };
  auto blocks = [&](int p, int vectors) {
    return (unsigned)(((long long)b.nsolves * p + vectors - 1) / vectors);
  };
  auto reflect = [&](auto first, int p, int lanes) {
    with(lanes, [&](auto l) {
      constexpr int kL = decltype(l)::value, kV = 32 / kL;
      constexpr bool kFirst = decltype(first)::value;
      const int sl = spans(p, kV);
      const size_t doubles = 32 * (size_t)((n + kL - 1) / kL) + 4 * (size_t)sl * n;
      auto run = [&](auto kernel) {
        kernel<<<blocks(p, kV), 32, smem_of(kernel, doubles), stream>>>(g, b, z, sl, tri, xb, axb, xa,
                                                                       axa);
      };
      if (core)
        run(reflect_kernel<kFirst, true, kL>);
      else if constexpr (kL > 1)  // (at least two lanes: below)
        run(reflect_kernel<kFirst, false, kL>);
    });
  };
  // Lanes per vector, for the solves (lf, which share its nodes) and the reflections
  // (lr, its elements).  Few vectors leave most schedulers idle and the time is one
  // lane's chain; many vectors fill the chip and the shares cost their sums -- except
  // that an analysis's reflections gain occupancy from a smaller array per warp at
  // every size (core ones read columns, which two lanes coalesce worse).  By warps of
  // vectors at one lane each; measured, us of a core call of 40 members with lf at 8 /
  // 4 / 2 / 1: 20 warps 312 / 315 / 324 / 346, 160 warps 349 / 322 / 326 / 344, 320
  // warps 411 / 374 / 354 / 371, 640 warps 520 / 446 / 423 / 408; with lr: 160 warps
  // 285 / 291 / 320 / 369, 640 warps 456 / 410 / 423 / 463, 2880 warps 1479 / 1277 /
  // 1204 / 1252, 41 000 warps 18.9 / 15.8 / 14.5 / 14.1 ms.  At 16, 28, 52 and 64 members
  // and 10 to 12 000 warps the same lines stay within 5 % of the best of the four (9 % at
  // 16 members and 450 warps).  Analysis of 16 members, lf:
  // 324 warps 122 / 123 / 143 / 188, 1296 warps 210 / 205 / 190 / 204, 2500 warps 321 /
  // 293 / 289 / 283; lr: 324 warps 73 / 92 / 122 / 198, 2500 warps 289 / 281 / 293 /
  // 365; of 40 members, 144 000 warps in eleven launches, lr 70.9 / 62.9 / 59.2 / 63.0 ms.
  const long long warps = ((long long)b.nsolves * per + 31) / 32;
  auto lanes_for = [&](int w8, int w4, int w2) {
    return warps < w8 ? 8 : warps < w4 ? 4 : warps < w2 ? 2 : 1;
  };
  using First = std::true_type;
  using Second = std::false_type;
  if (core) {
    const int lf = lanes_for(40, 200, 450), lr = lanes_for(200, 800, 6000);
    with(lf, [&](auto l) {
      constexpr int kL = decltype(l)::value, kV = 32 / kL;
      const int sl = spans(n, kV);
      const size_t smem = smem_of(ft_matrix_kernel<kL>, 3 * 32 * (size_t)n + 2 * (size_t)sl * n);
      ft_matrix_kernel<kL><<<blocks(n, kV), 32, smem, stream>>>(g, b, z, sl, tri, eig_fail);
    });
    reflect(First(), n, lr);
    reflect(Second(), n, lr);
    add_wbar_kernel<<<b.nsolves, 128, sizeof(double) * n * n, stream>>>(n, b, t, vec, wbar);
    return;
  }
  int lf = lanes_for(400, 700, 2000);
  const int lr = warps < 700 ? 8 : warps < 2000 ? 4 : 2;
  // a solve's vectors have to fit a warp, nearly filling it
  while (lf > 1 && (per * lf > 32 || 32 % (per * lf) > 4)) lf /= 2;
  reflect(First(), per, lr);
  with(lf, [&](auto l) {
    constexpr int kL = decltype(l)::value;
    const int sl = 32 / (per * kL);
    const unsigned grid = (unsigned)((b.nsolves + sl - 1) / sl);
    auto doubles = [&](int pairs) {
      return (3 * 32 + 2 * (size_t)pairs) * n + 2 * (size_t)sl * n;
    };
    auto run = [&](auto kernel, int pairs) {
      kernel<<<grid, 32, smem_of(kernel, doubles(pairs)), stream>>>(g, b, z, sl, tri, eig_fail);
    };
    // Factors of 32 (solve, node) pairs at a time, or 16 where 32 leave an SM two warps and
    // 16 leave three (228 KB, a KB and the kernel's 160 bytes a block; with four state
    // rows from 55 members on).  Transform of 129 600 solves, ms at 32 / 16: 40 members
    // 6.70 / 7.31, 48 10.1 / 10.4 (three warps / four), 52 11.0 / 13.5, 56 15.9 / 15.0,
    // 64 18.9 / 18.0.
    auto warps_per_sm = [&](int pairs) {
      return (int)((228 << 10) / (sizeof(double) * doubles(pairs) + 1024 + 160));
    };
    if (warps_per_sm(32) <= 2 && warps_per_sm(16) > warps_per_sm(32))
      run(ft_kernel<kL, 16>, 16);
    else
      run(ft_kernel<kL, 32>, 32);
  });
  reflect(Second(), per - 1, lr);
}

}  // namespace lg
