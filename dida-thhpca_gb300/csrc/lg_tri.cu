// lg_tri.cu -- Householder reduction C = Q T Q^T of up to 64 members in fixed
// point on the integer pipe (the FP64 path's tridiagonalisation).
//
// The FP64 pipe retires one warp instruction per 17 cycles per SM, the integer
// pipe up to four a cycle, so a multiply-add of 59-bit fixed-point numbers
// (three 32 x 32 -> 64-bit multiply-adds) costs less than a tenth of an FP64
// one.  Everything in the reduction is bounded by |C| once C is scaled, so fixed
// point loses nothing: C is scaled by a power of two 2^E just above its
// Frobenius norm and held as integers of 2^(E-59), where FP64 would round each
// result to 2^-53 of itself.
//
//   A   X = a 2^(59-E), |X| <= 2^59, held as Xh 2^30 + Xl, -2^29 <= Xl < 2^29
//   w   the reflector P = I - w w^T, |w|^2 = 2, as w 2^58, split the same way
//   p = A w, K = w^T p / 2, q = p - K w: integers of 2^(E-59);  A -= w q^T + q w^T
// A product of an A-type and a w-type number is 4 Xh Wh + (Xh Wl + Xl Wh) / 2^28
// (Xl Wl, below one unit, is dropped).  The row norms bound the sums (Cauchy):
// sum Xh Wh < 2^58, sum Xh Wl < 2^61, sum Xl Wh < 2^61: no 64-bit sum overflows.
// The two square roots of a step (the row's norm, and |u| of the reflector)
// start from the FP32 reciprocal square root and take one third-order step in
// integers, to about 2^-60.  No FP64 instruction is issued.
//
// One warp per matrix, the packed lower triangle in shared memory; lanes take
// rows (split over lanes where fewer than 32 are left) in A w and elements in
// the update, as in tridiag_kernel (lg_eig2.cu).  Output in the Gram matrix's
// place: D[n] | E[n] | G[n] (even i: w_i . w_{i-1}, for the transform, which applies
// two reflectors at a time) | w rows, zero where there is none (w and G in units of
// 2^-58 as pairs of 32-bit integers).
// A non-finite C gives a NaN diagonal, which the transform reports.  A finite one that may
// be beyond 2^kFtLog times (k - 1) / rho (by its largest element) is marked and left for the eigenvalue route: f(T) is
// formed in units of 2^-62 of sqrt(rho), so a C of full rank would lose half the bits of
// that ratio, and beyond 2^59 its rounding would reach the shift (k - 1) / rho itself.
//
// Measured alone against tridiag_kernel: 921 600 matrices of 40 members 116 ->
// 52 ms, 129 600 of 64 members 54 -> 27 ms, 2592 of 16 members 81 -> 52 us; a single
// matrix of 40 members 94 us.  Bound by instruction issue (at 64 members the
// triangles leave twelve warps per SM).
#include <math.h>

#include <algorithm>

#include "lg_device.cuh"
#include "lg_fixed.cuh"
#include "lg_internal.h"

namespace lg {
namespace tri {

__device__ inline int idx(int j) { return j * (j + 1) / 2; }

// Sum over the warp (which has to fit 64 bits) by three 32-bit reductions.
__device__ inline long long warp_add(long long v) {
  const unsigned p0 = __reduce_add_sync(0xffffffffu, (unsigned)v & 0x1fffffu);
  const unsigned p1 = __reduce_add_sync(0xffffffffu, (unsigned)(v >> 21) & 0x1fffffu);
  const int p2 = __reduce_add_sync(0xffffffffu, (int)(v >> 42));
  return (long long)p0 + ((long long)p1 << 21) + ((long long)p2 << 42);
}

// 1/sqrt(x / 2^64) in units of 2^-60 (to about 2^-59) for x in [2^62, 2^64).
// y0 from FP32 (error below 2^-22), then y = y0 (1 + e/2 + 3 e^2 / 8), e = 1 -
// x y0^2; the next term is below 2^-66.
__device__ inline unsigned long long rsqrt_fixed(unsigned long long x) {
  const float y0f = rsqrtf((float)(unsigned)(x >> 32) * 2.3283064365386963e-10f);
  const unsigned y0 = (unsigned)(y0f * 1073741824.0f);        // 2^30 y0, at most 2^31
  const unsigned long long y2 = (unsigned long long)y0 * y0;  // 2^60 y0^2
  const long long e = (1ll << 60) - (long long)__umul64hi(x, y2);
  const long long e8 = e >> 8;
  const long long c = (e >> 1) + ((3 * ((e8 * e8) >> 44)) >> 3);
  return ((unsigned long long)y0 << 30) +
         (unsigned long long)((((c >> 6) * (long long)y0) >> 24) +
                              (long long)(((unsigned long long)(c & 63) * y0) >> 30));
}

// byte offsets of (row, column) in an array of int4, per element of the packed
// triangle
struct Elements {
  unsigned v[64 * 65 / 2];
  constexpr Elements() : v() {
    int t = 0;
    for (unsigned j = 0; j < 64; ++j)
      for (unsigned c = 0; c <= j; ++c) v[t++] = (j * 16u) << 16 | (c * 16u);
  }
};
__device__ constexpr Elements g_elements{};

}  // namespace tri

__global__ void __launch_bounds__(32) tridiag_fixed_kernel(int n, int nsolves, int e_max, double* C,
                                                          int* list, int* count) {
  using namespace tri;
  const int s = blockIdx.x;
  if (s >= nsolves) return;
  const int lane = threadIdx.x;
  extern __shared__ int4 sm4[];
  int4* const WQ = sm4;                                // n: (wl, wh, ql, qh)
  int2* const A = reinterpret_cast<int2*>(sm4 + n);    // packed lower triangle
  double* const M = C + (size_t)s * n * n;
  const int np = idx(n);
  // ---- scale: 2^E just above the Frobenius norm (FP32 sum relative to the
  // largest exponent, rounded up)
  unsigned emax = 0;
  {
    int j = 0, c = lane;
    while (c > j) {
      c -= j + 1;
      ++j;
    }
    for (int t = lane; t < np; t += 32) {
      const double a = M[(size_t)j * n + c];
      A[t] = make_int2(__double2loint(a), __double2hiint(a));
      emax = max(emax, ((unsigned)__double2hiint(a) >> 20) & 0x7ffu);
      c += 32;
      while (c > j) {
        c -= j + 1;
        ++j;
      }
    }
  }
  emax = __reduce_max_sync(0xffffffffu, emax);
  __syncwarp();
  double* const D = M;
  double* const E = M + n;
  int2* const G = reinterpret_cast<int2*>(M + 2 * n);
  double* const U = M + 3 * n;
  if (emax == 0 || (int)emax >= e_max) {  // all zero, not finite: NaN, or left alone
    __syncwarp();
    if (emax && emax < 2047u) {
      if (lane == 0) {
        M[1] = __longlong_as_double((long long)kLeftMark);
        const int at = atomicAdd(count, 1);
        if (list) list[at] = s;
      }
      return;
    }
    for (int i = lane; i < n; i += 32) {
      D[i] = emax ? __longlong_as_double(0x7ff8000000000000ll) : 0.0;
      E[i] = 0.0;
      G[i] = make_int2(0, 0);
    }
    for (int t = lane; t < n * (n - 1) / 2; t += 32) U[t] = 0.0;
    return;
  }
  float fro = 0.0f;
  auto rough = [&](int t) {  // mantissa to 20 bits, rounded up, at 2^-d
    const int hi = A[t].y & 0x7fffffff;
    const int d = (int)emax - (hi >> 20);
    return d > 60 ? 0.0f : __int_as_float(((127 - d) << 23) | ((hi & 0xfffff) << 3)) * 1.00001f;
  };
  for (int t = lane; t < np; t += 32) {
    const float f = rough(t);
    fro = fmaf(f, f, fro);
  }
  fro *= 2.0f;  // both triangles; the diagonal once
  for (int j = lane; j < n; j += 32) {
    const float f = rough(idx(j) + j);
    fro = fmaf(-f, f, fro);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) fro += __shfl_xor_sync(0xffffffffu, fro, o);
  __syncwarp();
  // |C|_F < 2^(emax - 1023) sqrt(fro) 1.001; E = the exponent above
  const int ef = (int)((__float_as_uint(sqrtf(fro) * 1.001f) >> 23) & 0xffu) - 127 + 1;
  const int Eb = (int)emax + ef;  // E + 1023
  for (int t = lane; t < np; t += 32) {
    const int2 a = A[t];
    const unsigned long long u = (unsigned long long)(unsigned)a.y << 32 | (unsigned)a.x;
    const int e = (int)(u >> 52) & 0x7ff;
    long long x = 0;
    if (e) {
      const int sh = min(Eb - e, 62);  // >= 1
      x = (long long)((((u & 0xfffffffffffffull) | 0x10000000000000ull) << 7) +
                      (1ull << (sh - 1))) >> sh;
      if (u >> 63) x = -x;
    }
    A[t] = fixed_split(x);
  }
  __syncwarp();
  const int ex = Eb - 1023 - 59;  // a = X 2^ex
  for (int i = n - 1; i >= 1; --i) {
    const int l = i - 1;
    int2* const row = A + idx(i);
    // the row's integers, brought up to [2^56, 2^57) at the largest
    long long x0 = lane <= l ? fixed_join(row[lane]) : 0, x1 = lane + 32 <= l ? fixed_join(row[lane + 32]) : 0;
    const unsigned long long m0 = (unsigned long long)llabs(x0), m1 = (unsigned long long)llabs(x1);
    const unsigned long long mm = m0 | m1;  // the leading bit is what counts
    const unsigned mh = __reduce_or_sync(0xffffffffu, (unsigned)(mm >> 32));
    const unsigned ml = __reduce_or_sync(0xffffffffu, (unsigned)mm);
    int2* const u_out = reinterpret_cast<int2*>(U) + (size_t)i * (i - 1) / 2;
    if (l == 0 || (mh | ml) == 0) {
      // nothing to reduce: e is the element beside the diagonal
      const long long e = __shfl_sync(0xffffffffu, l < 32 ? x0 : x1, l & 31);
      for (int c = lane; c < i; c += 32) u_out[c] = make_int2(0, 0);
      if (lane == 0) WQ[i] = make_int4((int)e, (int)(e >> 32), ex, 0);
      __syncwarp();
      continue;
    }
    const int lead = mh ? 63 - __clz((int)mh) : 31 - __clz((int)ml);
    const int up = 56 - lead;  // may be negative (down to -3)
    x0 = up >= 0 ? x0 << up : x0 >> -up;
    x1 = up >= 0 ? x1 << up : x1 >> -up;
    // squared norm in units of 2^30
    const int2 s0 = fixed_split(x0), s1 = fixed_split(x1);
    long long S1 = (long long)s0.y * s0.y + (long long)s1.y * s1.y;
    long long S2 = 2 * ((long long)s0.y * s0.x + (long long)s1.y * s1.x) +
                   (((long long)s0.x * s0.x + (long long)s1.x * s1.x) >> 30);
    S1 = warp_add(S1);
    S2 = warp_add(S2);
    // N = |x|^2 / 2^56 in [2^56, 2^64) = xn 2^(-zn), zn even
    const unsigned long long N =
        ((unsigned long long)S1 << 4) + (unsigned long long)(S2 >> 26);
    const int zn = __clzll((long long)N) & ~1;
    const unsigned long long xn = N << zn;
    // |x| = sqrt(xn / 2^64) 2^(60 - zn / 2)
    const unsigned long long rt = __umul64hi(xn, rsqrt_fixed(xn));
    const long long alpha = (long long)((rt + ((1ull << (zn / 2)) >> 1)) >> (zn / 2));
    const long long f = __shfl_sync(0xffffffffu, l < 32 ? x0 : x1, l & 31);
    const long long af = llabs(f);
    // u_l = f + sign(f) alpha; h = |x|^2 + |f| alpha = hh 2^57 = xh 2^(57 - zh), zh odd
    const unsigned long long hh =
        (N >> 1) + __umul64hi((unsigned long long)af << 6, (unsigned long long)alpha << 1);
    const int zh = ((__clzll((long long)hh) + 1) & ~1) - 1;
    const unsigned long long xh = zh < 0 ? hh >> 1 : hh << zh;
    const int rh = (121 - zh) >> 1;  // sqrt(h) = sqrt(xh / 2^64) 2^rh
    const long long yh = (long long)(rsqrt_fixed(xh) << 1);
    const long long ul = f >= 0 ? f + alpha : f - alpha;
    if (lane == (l & 31)) {
      if (l < 32)
        x0 = ul;
      else
        x1 = ul;
    }
    // w 2^58 = u 2^(58 - rh) yh 2^-61; |u| < 2^(rh + 0.5), so u 2^(62 - rh) fits
    auto to_w = [&](long long x) { return (__mul64hi(x << (62 - rh), yh) + 1) >> 1; };
    const long long w0 = to_w(x0), w1 = to_w(x1);
    if (lane <= l) {
      const int2 w = fixed_split(w0);
      row[lane] = w;
      WQ[lane].x = w.x;
      WQ[lane].y = w.y;
      u_out[lane] = w;
    }
    if (lane + 32 <= l) {
      const int2 w = fixed_split(w1);
      row[lane + 32] = w;
      WQ[lane + 32].x = w.x;
      WQ[lane + 32].y = w.y;
      u_out[lane + 32] = w;
    }
    if (lane == 0) {
      const long long e = f >= 0 ? -alpha : alpha;
      WQ[i] = make_int4((int)e, (int)(e >> 32), ex - up, 1);  // column i is done with
    }
    __syncwarp();
    // ---- p = A w: rows 0 .. nfull - 1 a lane each, the rest split over f lanes
    const int R = l + 1;
    const int nfull = R > 32 ? 32 : 0;
    long long pf = 0, ps = 0;  // p of this lane's full row, of its split row
    if (nfull) {
      const int j = lane, tj = idx(j);
      long long hs = 0, ms = 1 << 27;
      int tc = 0;
#pragma unroll 4
      for (int c = 0; c < R; ++c) {
        const int2 a = A[(c <= j) ? tj + c : tc + j];
        const int2 w = row[c];
        hs += (long long)a.y * w.y;
        ms += (long long)a.y * w.x;
        ms += (long long)a.x * w.y;
        tc += c + 1;
      }
      pf = 4 * hs + (ms >> 28);
    }
    const int rr = R - nfull;                 // 1..32
    const int lf = 31 - __clz(32 / rr);       // 2^lf lanes a row
    const int fl = 1 << lf;
    const int cl = (R + fl - 1) >> lf;
    const int ri = lane >> lf, pi = lane & (fl - 1);
    const bool act = ri < rr;
    const int j = nfull + (act ? ri : 0);
    {
      const int c0 = act ? min(R, pi * cl) : 0, c1 = act ? min(R, c0 + cl) : 0;
      const int tj = idx(j);
      long long hs = 0, ms = 0;
      int tc = idx(c0);
#pragma unroll 4
      for (int c = c0; c < c1; ++c) {
        const int2 a = A[(c <= j) ? tj + c : tc + j];
        const int2 w = row[c];
        hs += (long long)a.y * w.y;
        ms += (long long)a.y * w.x;
        ms += (long long)a.x * w.y;
        tc += c + 1;
      }
      for (int o = fl >> 1; o > 0; o >>= 1) {  // the same fl in every lane
        hs += __shfl_xor_sync(0xffffffffu, hs, o);
        ms += __shfl_xor_sync(0xffffffffu, ms, o);
      }
      ps = 4 * hs + ((ms + (1 << 27)) >> 28);
    }
    const bool own = act && pi == 0;  // this lane holds p_j of the split row
    // ---- K = w^T p / 2
    long long kh = 0, km = 0;
    const int2 wf = nfull ? row[lane] : make_int2(0, 0), ws = own ? row[j] : make_int2(0, 0);
    {
      const int2 p = fixed_split(pf), p2 = fixed_split(ps);
      kh = (long long)p.y * wf.y + (long long)p2.y * ws.y;
      km = (long long)p.y * wf.x + (long long)p.x * wf.y + (long long)p2.y * ws.x +
           (long long)p2.x * ws.y;
    }
    kh = warp_add(kh);
    km = warp_add(km);
    const int2 K = fixed_split((4 * kh + (km >> 28)) >> 1);
    auto q_of = [&](long long p, int2 w) {
      const long long m = (long long)K.y * w.x + ((long long)K.x * w.y + (1 << 27));
      return fixed_split(p - (4 * ((long long)K.y * w.y) + (m >> 28)));
    };
    if (nfull) {
      const int2 q = q_of(pf, wf);
      WQ[lane].z = q.x;
      WQ[lane].w = q.y;
    }
    if (own) {
      const int2 q = q_of(ps, ws);
      WQ[j].z = q.x;
      WQ[j].w = q.y;
    }
    __syncwarp();
    // ---- A -= w q^T + q w^T over the packed rows 0 .. l
    {
      const int tot = idx(l + 1);
      const unsigned char* const wq = reinterpret_cast<const unsigned char*>(WQ);
      auto updated = [](int4 a, int4 b, int2 x) {
        const long long hs = (long long)a.y * b.w + (long long)a.w * b.y;
        long long ms = (long long)a.y * b.z + (1 << 27);
        ms += (long long)a.x * b.w;
        ms += (long long)a.w * b.x;
        ms += (long long)a.z * b.y;
        return fixed_split(fixed_join(x) - 4 * hs - (ms >> 28));
      };
      int t = lane;
      for (; t + 32 < tot; t += 64) {  // two elements a lane, loaded together
        const unsigned o0 = g_elements.v[t], o1 = g_elements.v[t + 32];
        const int4 a0 = *reinterpret_cast<const int4*>(wq + (o0 >> 16));
        const int4 b0 = *reinterpret_cast<const int4*>(wq + (o0 & 0xffffu));
        const int4 a1 = *reinterpret_cast<const int4*>(wq + (o1 >> 16));
        const int4 b1 = *reinterpret_cast<const int4*>(wq + (o1 & 0xffffu));
        const int2 e0 = A[t], e1 = A[t + 32];
        A[t] = updated(a0, b0, e0);
        A[t + 32] = updated(a1, b1, e1);
      }
      if (t < tot) {
        const unsigned o = g_elements.v[t];
        A[t] = updated(*reinterpret_cast<const int4*>(wq + (o >> 16)),
                       *reinterpret_cast<const int4*>(wq + (o & 0xffffu)), A[t]);
      }
    }
    __syncwarp();
  }
  for (int i = lane; i < n; i += 32) {
    D[i] = fixed_to_double(fixed_join(A[idx(i) + i]), ex);
    double e = 0.0;
    if (i > 0) {
      const int4 w = WQ[i];
      e = fixed_to_double((long long)w.y << 32 | (unsigned)w.x, w.z);
    }
    E[i] = e;
  }
  // w_i . w_{i-1}, a pair per lane (rows i - 1 and i follow each other)
  for (int i = 2 * lane + 2; i < n; i += 64) {
    const int2* const y = reinterpret_cast<const int2*>(U) + (size_t)i * (i - 1) / 2;
    const int2* const x = y - (i - 1);
    long long hs = 0, ms = 1 << 27;
#pragma unroll 8
    for (int c = 0; c < i - 1; ++c) {
      const int2 a = x[c], b = y[c];
      hs += (long long)a.y * b.y;
      ms += (long long)a.y * b.x;
      ms += (long long)a.x * b.y;
    }
    G[i] = fixed_split(4 * hs + (ms >> 28));
  }
}

void launch_tridiag_in_place(const Geometry& g, int nsolves, double* C, int* list, int* count,
                             cudaStream_t stream) {
  if (nsolves == 0) return;
  const int n = g.ens;
  // the first biased exponent of an element at which |C|, less than 64 times the largest
  // element, may be beyond 2^kFtLog (k - 1) / rho, or is not representable
  const int e_max = std::min(1023 + ilogb((double)(n - 1) / g.inflation) + kFtLog - 6, 2047 - 8);
  const size_t smem = sizeof(int4) * n + sizeof(int2) * ((size_t)n * (n + 1) / 2);
  allow_smem(tridiag_fixed_kernel, smem);
  tridiag_fixed_kernel<<<nsolves, 32, smem, stream>>>(n, nsolves, e_max, C, list, count);
}

}  // namespace lg
