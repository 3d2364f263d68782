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
// shifted solves take 4 per node, element and vector, plus 8 per node and
// element for the factors, which the lanes of a solve compute for different
// nodes.  The reflections Q^T x and Q z (2 k^2 multiply-adds per vector) leave
// the FP64 pipe altogether: a vector's norm does not change, so they run in
// fixed point on the integer pipe as the reduction does (lg_tri.cu), to 2^-58 of
// the norm per step.  Three kernels, so that the integer ones are not held to
// the two to four warps per SM that the solves' five arrays leave:
//   reflect_kernel (Q^T)  vectors in, y out
//   ft_kernel             f(T) y, and T^-1 y of t
//   reflect_kernel (Q)    z in; the rows' update, or the columns of W, out
// and for an explicit trans add_wbar_kernel.  Measured alone against QL + replay:
// 921 600 solves of 40 members 233 -> 71 ms, 129 600 of 64 members 93 -> 33 ms;
// explicit trans against the accumulating solver (lg_eig.cu), with the
// reduction: 32 768 cubes of 40 members 133 -> 15 ms.  Faster at every size from
// 7 to 64 members; above, five arrays leave an SM one warp.
#include <float.h>
#include <math.h>

#include <algorithm>
#include <mutex>

#include "lg_device.cuh"
#include "lg_fixed.cuh"
#include "lg_internal.h"

namespace lg {
namespace ft {

constexpr int kMaxLog = 80;    // M/m up to 2^80
constexpr int kMaxNodes = 128;  // nodes per row of the table, padded with zero weight
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
  if (cudaMemcpyToSymbol(ft::g_nodes, nodes, sizeof nodes) != cudaSuccess ||
      cudaMemcpyToSymbol(ft::g_count, count, sizeof count) != cudaSuccess) {
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

// Which vectors a call works on: vector v of solve s -- 0: t (kept in the t
// array's place), v >= 1: the state row v - 1 (analysis; in `vec`, element i at
// ((s (n + 1) + i) (per - 1) + v - 1), element n being overline_w . x) or the
// unit vector v - 1 (core; in trans, element i at so n n + i n + v - 1).
struct Vecs {
  int core, per;
  double* t;
  double* vec;  // or trans
};
__device__ inline double* vec_at(const Vecs& z, int n, size_t so, size_t s, int v, int& stride) {
  if (v == 0) {
    stride = 1;
    return z.t + s * n;
  }
  stride = z.core ? n : z.per - 1;
  return (z.core ? z.vec + so * n * n : z.vec + s * (n + 1) * (z.per - 1)) + (v - 1);
}
__device__ inline size_t out_index(const SolveBatch& b, int s) {
  return b.s_col ? (size_t)b.first_solve + s : (size_t)s;
}

// This lane's vector V (element i at 32 i) from FP64 to integers of 2^(ex):
// |V| < 2^(ex + 58), held as in lg_tri.cu; false if a value is not finite.
__device__ inline bool to_fixed(double* V, int n, int& ex) {
  unsigned emax = 0;
  for (int i = 0; i < n; ++i)
    emax = max(emax, ((unsigned)__double2hiint(V[32 * i]) >> 20) & 0x7ffu);
  float fro = 0.0f;
  for (int i = 0; i < n; ++i) {
    const int hi = __double2hiint(V[32 * i]) & 0x7fffffff;
    const int d = (int)emax - (hi >> 20);
    const float f =
        d > 60 ? 0.0f : __int_as_float(((127 - d) << 23) | ((hi & 0xfffff) << 3)) * 1.00001f;
    fro = fmaf(f, f, fro);
  }
  // norm < 2^(emax - 1023) sqrt(fro) 1.001; the power of two above it
  const int Eb = (int)emax + (int)((__float_as_uint(sqrtf(fro) * 1.001f) >> 23) & 0xffu) - 126;
  for (int i = 0; i < n; ++i) {
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

// y <- Q^T x (kIn; P_{n-1} first) or Q z (P_1 first) of one vector per lane, one
// warp per block, lanes numbered through the solves' vectors.  Reflector rows of
// the (up to `slots`) solves that a warp spans come into shared memory a step
// ahead of their use.
template <bool kIn, bool kCore>
__global__ void __launch_bounds__(32) reflect_kernel(Geometry g, SolveBatch b, ft::Vecs z,
                                                     int slots, const double* tri, const double* xb,
                                                     const double* axb, double* xa, double* axa) {
  const int n = g.ens;
  const int lane = threadIdx.x;
  // the rows' update needs no t: its vectors are v = 1 .. per - 1
  const int v0 = !kIn && !kCore ? 1 : 0;
  const int per = z.per - v0;
  const long long id0 = (long long)blockIdx.x * 32, total = (long long)b.nsolves * per;
  const int s_first = (int)(id0 / per);
  const int nsl = (int)((min(id0 + 32, total) - 1) / per) - s_first + 1;
  const bool mine = id0 + lane < total;
  const int s = mine ? (int)((id0 + lane) / per) : s_first;
  const int v = v0 + (mine ? (int)((id0 + lane) - (long long)s * per) : 0);
  extern __shared__ double sm[];
  double* const Y = sm + lane;                      // element i at 32 i
  int2* const Yi = reinterpret_cast<int2*>(Y);
  double* const ub = sm + 32 * n;                   // two buffers of slots x n
  const size_t tri_stride = (size_t)n * n;
  auto fetch = [&](int i, int buf) {
    if (i >= 1 && i < n)
      for (int sl = 0; sl < nsl; ++sl) {
        const double* T = tri + (size_t)(s_first + sl) * tri_stride;
        const double* u = T + 3 * n + (size_t)i * (i - 1) / 2;
        double* d = ub + (size_t)(buf * slots + sl) * n;
        for (int c = lane; c < i; c += 32) ft::cp_async8(d + c, u + c);
        if (lane == 0) ft::cp_async8(d + n - 1, T + 2 * n + i);  // H (i <= n - 1: free)
      }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  const int step = kIn ? -1 : 1, i0 = kIn ? n - 1 : 1;
  fetch(i0, 0);
  // ---- the vector
  int r_state = -1;
  size_t ci = 0;
  if (!kCore) {
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
  int vs;
  double* const out = ft::vec_at(z, n, ft::out_index(b, s), s, v, vs);
  const double* const xr = xb + (row ? (size_t)n * (r_state + (size_t)g.n * ci) : 0);
  for (int i = 0; i < n; ++i) {
    double x = 0.0;
    if (kIn && kCore)
      x = v == 0 ? out[i] : (i == v - 1 ? 1.0 : 0.0);
    else if (kIn)
      x = v == 0 ? out[i] : (row ? xr[i] : 0.0);
    else if (kCore || row)
      x = out[(size_t)i * vs];
    Y[32 * i] = x;
  }
  int ex;
  const bool finite = ft::to_fixed(Y, n, ex);
  // ---- reflections: y -= w (w . y)
  for (int c = 0, i = i0; c < n - 1; ++c, i += step) {
    fetch(i + step, (c + 1) & 1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
    const double* ud = ub + (size_t)((c & 1) * slots + (s - s_first)) * n;
    const int2* u = reinterpret_cast<const int2*>(ud);
    if (__double2hiint(ud[n - 1]) != 0) {
      long long hs = 0, ms = 1 << 27;
#pragma unroll 4
      for (int j = 0; j < i; ++j) {
        const int2 w = u[j], y = Yi[32 * j];
        hs += (long long)y.y * w.y;
        ms += (long long)y.y * w.x;
        ms += (long long)y.x * w.y;
      }
      const int2 D = fixed_split(4 * hs + (ms >> 28));
      const int D4 = -4 * D.y;  // |D| < 2^58.5
#pragma unroll 4
      for (int j = 0; j < i; ++j) {
        const int2 w = u[j], y = Yi[32 * j];
        const long long m = (long long)D.y * w.x + ((long long)D.x * w.y + (1 << 27));
        Yi[32 * j] = fixed_split(fixed_join(y) + (long long)D4 * w.y - (int)(m >> 28));
      }
    }
    __syncwarp();
  }
  asm volatile("cp.async.wait_group 0;" ::: "memory");
  // ---- out
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  if (kIn || kCore) {
    if (mine)
      for (int i = 0; i < n; ++i)
        out[(size_t)i * vs] = finite ? fixed_to_double(fixed_join(Yi[32 * i]), ex) : nan;
  } else if (row) {
    // xa = axb + sqrt(rho) x + (W - sqrt(rho) I) x + overline_w . x, recentred
    const double srho = sqrt(g.inflation);
    const double ab = axb[r_state + (size_t)g.n * ci];
    const double dotw = out[(size_t)n * vs];
    double mean = 0.0;
    for (int i = 0; i < n; ++i) {
      const double d = finite ? fixed_to_double(fixed_join(Yi[32 * i]), ex) : nan;
      const double x = ab + (srho * xr[i] + (d + dotw));
      Y[32 * i] = x;
      mean += x;
    }
    mean /= (double)n;
    double* xo = xa + (size_t)n * (r_state + (size_t)g.n * ci);
    for (int i = 0; i < n; ++i) xo[i] = Y[32 * i] - mean;
    axa[r_state + (size_t)g.n * ci] = mean;
  }
}

// f(T) y per lane, one warp per block.  Analysis: slots = 32 / per solves per
// warp; v = 0 gives T^-1 y (overline_w in the reduced basis), the rows
// (f(T) - sqrt(rho)) y and overline_w . x.  Core: lanes numbered through the
// solves' vectors; unit vectors give f(T) y.
// Shared memory, [element][lane] so that lanes never conflict: Y (the vector),
// F (the forward solve), A (the sum over nodes), and for 32 (slot, node) pairs
// the reciprocal pivots R and multipliers L of T + s; T's diagonals per slot.
template <bool kCore>
__global__ void __launch_bounds__(32) ft_kernel(Geometry g, SolveBatch b, ft::Vecs z, int slots,
                                                const double* tri, int* eig_fail) {
  const int n = g.ens;
  const int lane = threadIdx.x;
  const int per = z.per;
  int s_first, nsl, s, v;
  bool mine;
  if (kCore) {
    const long long id0 = (long long)blockIdx.x * 32, total = (long long)b.nsolves * per;
    s_first = (int)(id0 / per);
    nsl = (int)((min(id0 + 32, total) - 1) / per) - s_first + 1;
    mine = id0 + lane < total;
    s = mine ? (int)((id0 + lane) / per) : s_first;
    v = mine ? (int)((id0 + lane) - (long long)s * per) : 0;
  } else {
    s_first = blockIdx.x * slots;
    nsl = min(slots, b.nsolves - s_first);
    const int q = lane / per;
    mine = q < nsl;
    s = s_first + (mine ? q : 0);
    v = mine ? lane - q * per : 0;
  }
  const int sl = s - s_first;
  extern __shared__ double sm[];
  const int cap = n * 32;
  double *const Y = sm + lane, *const F = Y + cap, *const A = F + cap;
  double *const R = sm + 3 * cap, *const L = R + cap;
  double* const Dg = L + cap;         // slots x n: diagonal + shift
  double* const Eg = Dg + slots * n;  // slots x n: Eg[i] couples i - 1 and i
  const double shift = (double)(n - 1) / g.inflation;
  int vs;
  double* const io = ft::vec_at(z, n, ft::out_index(b, s), s, v, vs);
  if (mine)
    for (int i = 0; i < n; ++i) Y[32 * i] = io[(size_t)i * vs];
  // T, and per slot the node row (Gershgorin in FP32, rounded up)
  __shared__ int s_row[32];
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
      s_row[q] = nf ? 0 : min(max(ex, 1), ft::kMaxLog);
      // as a QL iteration that never converges; once per solve
      if (nf && (!kCore || (long long)(s_first + q) * per >= (long long)blockIdx.x * 32))
        atomicAdd(eig_fail, 1);
    }
  }
  __syncwarp();
  const int nb = 32 / slots;  // nodes per batch: pair (slot, node) = slot + slots * node
  int nmax = 0;
  for (int q = 0; q < nsl; ++q) nmax = max(nmax, ft::g_count[s_row[q]]);
  const int fs = lane % slots, fj = lane / slots;
  const double wscale = sqrt((double)(n - 1) * shift);  // sqrt(k - 1) sqrt(m)
  for (int i = 0; i < n; ++i) A[32 * i] = 0.0;
  auto factor = [&](double sigma) {
    // T + sigma = U^T diag(1/R) U with U[i-1][i] = L[i], for this lane's pair
    const double *D = Dg + fs * n, *E = Eg + fs * n;
    double r = ft::rcp(D[0] + sigma);
    R[lane] = r;
#pragma unroll 2
    for (int i = 1; i < n; ++i) {
      const double e = E[i], l = e * r;
      r = ft::rcp(fma(-l, e, D[i] + sigma));
      L[32 * i + lane] = l;
      R[32 * i + lane] = r;
    }
  };
  auto solve = [&](int pair, double w) {
    // A += w (T + s)^-1 y with the factors of the pair; each recurrence's chain
    // is one fused multiply-add per element
    const double *Rp = R + pair, *Lp = L + pair;
    double f = Y[0];
    F[0] = f;
#pragma unroll 4
    for (int i = 1; i < n; ++i) {
      f = fma(-Lp[32 * i], f, Y[32 * i]);
      F[32 * i] = f;
    }
    double x = Rp[32 * (n - 1)] * f;
    A[32 * (n - 1)] = fma(w, x, A[32 * (n - 1)]);
#pragma unroll 4
    for (int i = n - 2; i >= 0; --i) {
      x = fma(-Lp[32 * (i + 1)], x, Rp[32 * i] * F[32 * i]);
      A[32 * i] = fma(w, x, A[32 * i]);
    }
  };
  for (int j0 = 0; j0 < nmax; j0 += nb) {
    if (fs < nsl && fj < nb && j0 + fj < nmax) factor(ft::g_nodes[s_row[fs]][j0 + fj].x * shift);
    __syncwarp();
    if (mine) {
      const int rowq = s_row[sl];
      for (int j = 0; j < nb && j0 + j < nmax; ++j)
        solve(sl + slots * j, ft::g_nodes[rowq][j0 + j].y * wscale);
    }
    __syncwarp();
  }
  if (lane < nsl) factor(0.0);  // pair (slot, 0)
  __syncwarp();
  if (mine && v == 0) {
    for (int i = 0; i < n; ++i) A[32 * i] = 0.0;
    solve(sl, 1.0);
  }
  __syncwarp();
  if (!mine) return;
  if (!kCore && v >= 1) {
    const double srho = sqrt(g.inflation);
    const double* zt = sm + 2 * cap + sl * per;  // vector 0's A
    double dotw = 0.0;
    for (int i = 0; i < n; ++i) {
      const double y = Y[32 * i];
      dotw = fma(y, zt[32 * i], dotw);
      io[(size_t)i * vs] = fma(-srho, y, A[32 * i]);
    }
    io[(size_t)n * vs] = dotw;
  } else if (kCore) {
    for (int i = 0; i < n; ++i) io[(size_t)i * vs] = A[32 * i];
  }
}

// trans(i, j) = W(i, j) + overline_w(i), column-major; W is symmetric, so its
// row j comes in place of column j
__global__ void add_wbar_kernel(int n, SolveBatch b, const double* t, double* trans, double* wbar) {
  const int s = blockIdx.x;
  const size_t so = ft::out_index(b, s);
  const double* w = t + (size_t)s * n;
  double* To = trans + so * n * n;
  for (int r = threadIdx.x, i = r % n; r < n * n; r += blockDim.x) {
    To[r] += w[i];
    i = (i + blockDim.x) % n;
  }
  if (wbar)
    for (int i = threadIdx.x; i < n; i += blockDim.x) wbar[so * n + i] = w[i];
}

bool ft_supported(const Geometry& g) {
  // below 7 members the tridiagonal form does not fit the Gram matrix's place;
  // a lowered sweep limit asks for the QL iteration
  return g.ens >= 7 && g.ens <= 64 && (g.ql_max_iter == 0 || g.ql_max_iter >= 60);
}

size_t ft_vec_doubles(const Geometry& g) {
  return (size_t)(g.ens + 1) * (g.vert_dist > 0.0 ? g.n_var : g.n);
}

void launch_ft(const Geometry& g, const SolveBatch& b, bool core, double* t, const double* tri,
               double* vec, const double* xb, const double* axb, double* xa, double* axa,
               double* wbar, int* eig_fail, cudaStream_t stream) {
  if (b.nsolves == 0) return;
  const int n = g.ens;
  const int per = core ? n + 1 : 1 + (g.vert_dist > 0.0 ? g.n_var : g.n);
  const ft::Vecs z{core ? 1 : 0, per, t, vec};
  // solves that 32 consecutive vectors can touch
  auto spans = [](int p) { return (32 + p - 2) / p + 1; };
  auto blocks = [&](int p) { return (unsigned)(((long long)b.nsolves * p + 31) / 32); };
  auto reflect = [&](auto kernel, int p) {
    const int sl = spans(p);
    const size_t smem = sizeof(double) * ((size_t)32 * n + 2 * (size_t)sl * n);
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    kernel<<<blocks(p), 32, smem, stream>>>(g, b, z, sl, tri, xb, axb, xa, axa);
  };
  auto solve = [&](auto kernel, int sl, unsigned grid) {
    const size_t smem = sizeof(double) * ((size_t)5 * 32 * n + 2 * (size_t)sl * n);
    cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    kernel<<<grid, 32, smem, stream>>>(g, b, z, sl, tri, eig_fail);
  };
  if (core) {
    reflect(reflect_kernel<true, true>, per);
    solve(ft_kernel<true>, spans(per), blocks(per));
    reflect(reflect_kernel<false, true>, per);
    add_wbar_kernel<<<b.nsolves, 128, 0, stream>>>(n, b, t, vec, wbar);
  } else {
    const int sl = 32 / per;
    reflect(reflect_kernel<true, false>, per);
    solve(ft_kernel<false>, sl, (unsigned)((b.nsolves + sl - 1) / sl));
    reflect(reflect_kernel<false, false>, per - 1);
  }
}

}  // namespace lg
