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
// shifted solves take 5 per node, element and vector, plus 7 per node and
// element for the factors, which the lanes of a solve compute for different
// nodes.  Measured alone against QL + replay: 921 600 solves of 40 members
// 233 -> 102 ms, 129 600 of 64 members 93 -> 46 ms; explicit trans against the
// accumulating solver (lg_eig.cu): 32 768 cubes of 40 members 133 -> 29 ms (with
// the reduction).  Faster at every size from 7 to 64 members; above, three
// vectors per lane no longer leave an SM two warps.  Bound by the FP64 pipe.
#include <float.h>
#include <math.h>

#include <algorithm>
#include <mutex>

#include "lg_device.cuh"
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

}  // namespace ft

// Lanes are (slot, vector): slots = 32 / per solves of a warp, per vectors each.
//   analysis (kCore false): vector 0 is t, vector v >= 1 the solve's state row
//     v - 1; one warp per block.
//   kCore: one solve per block, lane j of its ceil(k / 32) warps is the unit
//     vector e_j; trans and overline_w = W (W t) / (k - 1) come out.
// Shared memory per warp, [element][lane] so that lanes never conflict: Y (the
// vector), F (the forward solve), A (the sum over nodes); per block: the
// factors R of 32 (slot, node) pairs -- in the reductions' phases the same
// space holds two rows of reflectors per slot -- and T's two diagonals.
// tri: per solve D[n] | E[n] | H[n] (0: no reflector, else P = I - H u u^T) | U,
// stride tri_stride.
template <bool kCore>
__global__ void ft_kernel(Geometry g, SolveBatch b, const double* tin, const double* tri,
                          size_t tri_stride, const double* xb, const double* axb, double* xa,
                          double* axa, double* trans_out, double* wbar_out, int* eig_fail) {
  const int n = g.ens;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int warps = kCore ? blockDim.x / 32 : 1;
  const bool vertical = g.vert_dist > 0.0;
  const int per = kCore ? 32 : 1 + (vertical ? g.n_var : g.n);
  const int slots = 32 / per;
  const int q = lane / per, v = lane - q * per;
  const int s0 = kCore ? (int)blockIdx.x : (int)blockIdx.x * slots;
  const int nsl = kCore ? 1 : min(slots, b.nsolves - s0);  // solves of this warp
  extern __shared__ double sm[];
  const int cap = n * 32;
  double* const Y = sm + (size_t)warp * 3 * cap;
  double* const F = Y + cap;
  double* const A = F + cap;
  double* const R = sm + (size_t)warps * 3 * cap;  // n x 32
  double* const Dg = R + cap;                      // slots x n: diagonal + shift
  double* const Eg = Dg + slots * n;               // slots x n: Eg[i] couples i - 1 and i
#define AT(a, i) (a)[(i) * 32 + lane]
  const double shift = (double)(n - 1) / g.inflation;
  const bool mine = kCore ? warp * 32 + lane < n : q < nsl;
  const int s = s0 + (kCore ? 0 : q);
  // T, and per slot the node row (Gershgorin in FP32, rounded up)
  __shared__ int s_row[32], s_bad[32];
  for (int sl = warp; sl < nsl; sl += warps) {
    const double* T = tri + (size_t)(s0 + sl) * tri_stride;
    for (int i = lane; i < n; i += 32) {
      Dg[sl * n + i] = T[i] + shift;
      Eg[sl * n + i] = T[n + i];
    }
    __syncwarp();
    float mx = 0.0f;
    bool nf = false;
    for (int i = lane; i < n; i += 32) {
      const double d = Dg[sl * n + i], e0 = Eg[sl * n + i], e1 = i + 1 < n ? Eg[sl * n + i + 1] : 0.0;
      nf |= ((__double2hiint(d) >> 20) & 0x7ff) == 0x7ff || ((__double2hiint(e0) >> 20) & 0x7ff) == 0x7ff;
      mx = fmaxf(mx, fabsf(d2f_bits(d)) + fabsf(d2f_bits(e0)) + fabsf(d2f_bits(e1)));
    }
    nf = __any_sync(0xffffffffu, nf);
    mx = __uint_as_float(__reduce_max_sync(0xffffffffu, __float_as_uint(mx)));
    if (lane == 0) {
      // smallest power of two above the bound
      const int ex = (int)((__float_as_uint(mx * (1.0001f / (float)shift)) >> 23) & 0xffu) - 127 + 1;
      s_row[sl] = nf ? 0 : min(max(ex, 1), ft::kMaxLog);
      s_bad[sl] = nf;
      if (nf) atomicAdd(eig_fail, 1);  // as a QL iteration that never converges
    }
  }
  // ---- the vectors
  int r_state = -1;
  size_t ci = 0;
  bool work = false;
  if (kCore) {
    work = mine;
    for (int i = 0; i < n; ++i) AT(Y, i) = i == warp * 32 + lane ? 1.0 : 0.0;
  } else if (mine) {
    const int col = b.first_col + s / b.levels;
    const int kk = s % b.levels + 1;
    const int glat = col % g.num_lat + 1, glon = col / g.num_lat + 1;
    ci = (size_t)(glat - 1 + g.halo) + (size_t)(g.num_lat + 2 * g.halo) * (size_t)(glon - 1 + g.halo);
    if (v >= 1) {
      if (!vertical)
        r_state = v - 1;
      else if (g.var_lev[v - 1] > 1)
        r_state = g.var_start[v - 1] + kk - 1;
      else if (kk == g.nz)
        r_state = g.var_start[v - 1];
    }
    work = v == 0 || r_state >= 0;
    const double* x = v == 0 ? tin + (size_t)s * n : xb + (size_t)n * (max(r_state, 0) + (size_t)g.n * ci);
    for (int i = 0; i < n; ++i) AT(Y, i) = work ? x[i] : 0.0;
  }
  if (kCore) __syncthreads(); else __syncwarp();
  // ---- y <- P_{n-1} first (Q^T) or P_1 first (Q), in place in V.  Row i's
  // reflectors of every slot come into shared memory a step ahead.
  double* const ub = R;  // two buffers of slots x n
  auto fetch = [&](int i, int buf) {
    if (i >= 1 && i < n)
      for (int sl = warp; sl < nsl; sl += warps) {
        const double* T = tri + (size_t)(s0 + sl) * tri_stride;
        const double* u = T + 3 * n + (size_t)i * (i - 1) / 2;
        double* d = ub + (size_t)(buf * slots + sl) * n;
        for (int c = lane; c < i; c += 32) ft::cp_async8(d + c, u + c);
        if (lane == 0) ft::cp_async8(d + n - 1, T + 2 * n + i);  // H (i <= n - 1: free)
      }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  auto reflect_all = [&](double* V, bool transposed) {
    const int step = transposed ? -1 : 1, i0 = transposed ? n - 1 : 1;
    fetch(i0, 0);
    for (int c = 0, i = i0; c < n - 1; ++c, i += step) {
      fetch(i + step, (c + 1) & 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
      if (kCore) __syncthreads(); else __syncwarp();
      const double* u = ub + (size_t)((c & 1) * slots + (kCore ? 0 : min(q, slots - 1))) * n;
      const double ih = u[n - 1];
      if (ih != 0.0) {
        double d0 = 0.0, d1 = 0.0, d2 = 0.0, d3 = 0.0;
        int j = 0;
        for (; j + 3 < i; j += 4) {
          d0 = fma(u[j], AT(V, j), d0);
          d1 = fma(u[j + 1], AT(V, j + 1), d1);
          d2 = fma(u[j + 2], AT(V, j + 2), d2);
          d3 = fma(u[j + 3], AT(V, j + 3), d3);
        }
        for (; j < i; ++j) d0 = fma(u[j], AT(V, j), d0);
        const double dot = -((d0 + d1) + (d2 + d3)) * ih;
#pragma unroll 4
        for (j = 0; j < i; ++j) AT(V, j) = fma(u[j], dot, AT(V, j));
      }
      if (kCore) __syncthreads(); else __syncwarp();
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (kCore) __syncthreads(); else __syncwarp();
  };
  reflect_all(Y, true);
  // ---- A = sqrt(k - 1) sum_j w_j (T + s_j)^-1 y; the row lanes' last pass
  // leaves vector 0 (t) with A = T^-1 y
  const int nb = kCore ? 32 : 32 / slots;  // nodes per batch: lane = slot + slots * node
  int nmax = 0;
  for (int sl = 0; sl < nsl; ++sl) nmax = max(nmax, ft::g_count[s_row[sl]]);
  const int fs = kCore ? 0 : lane % slots, fj = kCore ? lane : lane / slots;
  const double wscale = sqrt((double)(n - 1) * shift);  // sqrt(k - 1) sqrt(m)
  for (int i = 0; i < n; ++i) AT(A, i) = 0.0;
  auto factor = [&](double sigma) {
    // R[i] = 1 / (pivot i of T + sigma) for this lane's (slot, node)
    const double *D = Dg + fs * n, *E = Eg + fs * n;
    double r = ft::rcp(D[0] + sigma);
    AT(R, 0) = r;
    for (int i = 1; i < n; ++i) {
      const double e = E[i];
      r = ft::rcp(fma(-(e * r), e, D[i] + sigma));
      AT(R, i) = r;
    }
  };
  auto solve = [&](int rl, double w) {
    // A += w (T + s)^-1 y with the factors of lane rl
    const double* E = Eg + (kCore ? 0 : min(q, slots - 1)) * n;
    const double* Rl = R + rl;
    double f = Rl[0] * AT(Y, 0);
    AT(F, 0) = f;
#pragma unroll 4
    for (int i = 1; i < n; ++i) {
      f = Rl[i * 32] * fma(-E[i], f, AT(Y, i));
      AT(F, i) = f;
    }
    double x = f;
    AT(A, n - 1) = fma(w, x, AT(A, n - 1));
#pragma unroll 4
    for (int i = n - 2; i >= 0; --i) {
      x = fma(-Rl[i * 32], E[i + 1] * x, AT(F, i));
      AT(A, i) = fma(w, x, AT(A, i));
    }
  };
  for (int j0 = 0; j0 < nmax; j0 += nb) {
    if (warp == 0 && fs < nsl && fj < nb && j0 + fj < nmax)
      factor(ft::g_nodes[s_row[fs]][j0 + fj].x * shift);
    if (kCore) __syncthreads(); else __syncwarp();
    for (int j = 0; j < nb && j0 + j < nmax; ++j) {
      if (mine) {
        const int row = s_row[kCore ? 0 : q];
        solve(kCore ? j : q + slots * j, ft::g_nodes[row][j0 + j].y * wscale);
      }
    }
    if (kCore) __syncthreads(); else __syncwarp();
  }
  if (!kCore) {
    if (lane < nsl) factor(0.0);  // lanes 0 .. slots - 1 are (slot, node 0)
    __syncwarp();
    if (mine && v == 0) {
      for (int i = 0; i < n; ++i) AT(A, i) = 0.0;
      solve(q, 1.0);
    }
    __syncwarp();
    // dot = overline_w . x in the reduced basis; A becomes (W - sqrt(rho) I) y
    const double srho = sqrt(g.inflation);
    double dotw = 0.0;
    if (mine && v >= 1) {
      const double* zt = A + q * per;
      for (int i = 0; i < n; ++i) {
        const double y = AT(Y, i);
        dotw = fma(y, zt[i * 32], dotw);
        AT(A, i) = fma(-srho, y, AT(A, i));
      }
    }
    __syncwarp();
    reflect_all(A, false);
    if (work && v >= 1) {
      // xa = axb + sqrt(rho) x + (W - sqrt(rho) I) x + overline_w . x, recentred
      const double ab = axb[r_state + (size_t)g.n * ci];
      const double* xr = xb + (size_t)n * (r_state + (size_t)g.n * ci);
      double mean = 0.0;
      for (int i = 0; i < n; ++i) {
        const double x = ab + (srho * xr[i] + (AT(A, i) + dotw));
        AT(A, i) = x;
        mean += x;
      }
      mean /= (double)n;
      double* xo = xa + (size_t)n * (r_state + (size_t)g.n * ci);
      for (int i = 0; i < n; ++i) xo[i] = AT(A, i) - mean;
      axa[r_state + (size_t)g.n * ci] = mean;
    }
  } else {
    reflect_all(A, false);  // lane j: column j of W
    // overline_w = W (W t) / (k - 1): each lane a dot product with its column
    double* const tv = R;         // t, then W t
    double* const wt = R + n;
    const double* t = tin + (size_t)s * n;
    for (int i = threadIdx.x; i < n; i += blockDim.x) tv[i] = t[i];
    __syncthreads();
    double d = 0.0;
    if (mine)
      for (int i = 0; i < n; ++i) d = fma(AT(A, i), tv[i], d);
    if (mine) wt[warp * 32 + lane] = d;
    __syncthreads();
    d = 0.0;
    if (mine) {
      for (int i = 0; i < n; ++i) d = fma(AT(A, i), wt[i], d);
      d /= (double)(n - 1);
      // trans(i, j) = W(i, j) + overline_w(i), column-major; W is symmetric, so
      // this lane's column is also row i = its index
      const size_t so = b.s_col ? (size_t)b.first_solve + s : (size_t)s;
      const int i = warp * 32 + lane;
      double* To = trans_out + so * n * n;
      for (int j = 0; j < n; ++j) To[i + (size_t)n * j] = AT(A, j) + d;
      if (wbar_out) wbar_out[so * n + i] = d;
    }
  }
#undef AT
}

bool ft_supported(const Geometry& g) {
  // below 7 members the tridiagonal form does not fit the Gram matrix's place;
  // a lowered sweep limit asks for the QL iteration
  return g.ens >= 7 && g.ens <= 64 && (g.ql_max_iter == 0 || g.ql_max_iter >= 60);
}

void launch_ft(const Geometry& g, const SolveBatch& b, bool core, const double* t,
               const double* tri, size_t tri_stride, const double* xb, const double* axb,
               double* xa, double* axa, double* trans, double* wbar, int* eig_fail,
               cudaStream_t stream) {
  if (b.nsolves == 0) return;
  const int n = g.ens;
  const bool vertical = g.vert_dist > 0.0;
  const int slots = core ? 1 : 32 / (1 + (vertical ? g.n_var : g.n));
  const int warps = core ? (n + 31) / 32 : 1;
  const size_t smem = sizeof(double) * ((size_t)(3 * warps + 1) * 32 * n + 2 * (size_t)slots * n);
  if (core) {
    cudaFuncSetAttribute(ft_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    ft_kernel<true><<<b.nsolves, 32 * warps, smem, stream>>>(g, b, t, tri, tri_stride, xb, axb, xa,
                                                             axa, trans, wbar, eig_fail);
  } else {
    cudaFuncSetAttribute(ft_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    ft_kernel<false><<<(b.nsolves + slots - 1) / slots, 32, smem, stream>>>(
        g, b, t, tri, tri_stride, xb, axb, xa, axa, trans, wbar, eig_fail);
  }
}

}  // namespace lg
