// lg_cube.cu -- application of cube solves to the columns they cover.
//
// With da_block_interval cube_n > 1 (and da_vertical_interval cube_nz on the
// vertical path) the reference solves letkf_core once per cube of
// cube_n x cube_n columns of a block (and level group), from the list of the
// cube's centre grid point, and applies that trans to every column (and level)
// of the cube: letkf_compute_nooverlap (letkf_compute.F90:12-154, xb_2_xa
// :259-329), letkf_compute_nooverlap_vertical (:386-554).  With
// da_block_overlap > 0 the cubes step by cube_n - overlap and each column's
// analysis is the average over the cubes covering it (letkf_compute :156-256,
// xb_add2_xa :332-382).  The solves' trans (k x k, column-major: trans(i, e))
// are computed beforehand; this kernel forms, per column and row,
//   dist(e) = axb + sum_i xb(i) trans(i, e),   mean over e,   xa = dist - mean,
// accumulated over the covering cubes and divided by their number.
#include <limits.h>

#include <algorithm>

#include "lg_device.cuh"
#include "lg_fixed.cuh"
#include "lg_internal.h"

namespace lg {

namespace {

// block (0-based) of a global grid point: pro_info_get_indx inverted (the first
// res blocks hold sec + 1 points, the others sec)
__device__ inline int block_of(int p, int npts, int nblk) {
  const int sec = npts / nblk, res = npts % nblk;
  const int big = res * (sec + 1);
  return p <= big ? (p - 1) / (sec + 1) : res + (p - 1 - big) / sec;
}

// first cube (0-based) along one axis whose span [1 + m st, m st + cn] holds p
__device__ inline int first_cube(int p, int cn, int st) { return p > cn ? (p - cn + st - 1) / st : 0; }

// FP32 value of a double relative to 2^(emax - 1023), its magnitude rounded up
__device__ inline float rough(double a, unsigned emax) {
  const int hi = __double2hiint(a) & 0x7fffffff;
  const int d = (int)emax - (hi >> 20);
  return d > 60 ? 0.0f : __int_as_float(((127 - d) << 23) | ((hi & 0xfffff) << 3)) * 1.00001f;
}
// biased exponent Eb with norm < 2^(Eb - 1023), from the largest biased exponent
// and the sum of squares of rough()
__device__ inline int norm_exponent(unsigned emax, float fro) {
  return (int)emax + (int)((__float_as_uint(sqrtf(fro) * 1.001f) >> 23) & 0xffu) - 126;
}
// a in units of 2^(Eb - 1081): vectors of norm below 2^(Eb - 1023) stay below 2^58
__device__ inline int2 to_fixed(double a, int Eb) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(a);
  const int e = (int)(u >> 52) & 0x7ff;
  if (!e) return make_int2(0, 0);
  const int sh = min(max(Eb - e, 1), 62);
  const long long x =
      (long long)((((u & 0xfffffffffffffull) | 0x10000000000000ull) << 6) + (1ull << (sh - 1))) >> sh;
  return fixed_split(u >> 63 ? -x : x);
}

// p 2^ex; kBad: an input was not finite
constexpr int kBad = INT_MIN;
__device__ inline double scaled(long long p, int ex) {
  if (ex == kBad) return __longlong_as_double(0x7ff8000000000000ll);
  if (ex > 900) return scalbn((double)p, ex);  // may overflow
  return fixed_to_double(p, ex);
}

// Without overlap a block takes one solve with all its columns (so that trans is
// brought to fixed point once), with overlap one column with all its solves, whose
// average it takes.  Each thread forms one product sum_i xb(i) trans(i, e) of a
// batch of rows, threads numbered through the rows' members so that no lane idles
// at the ragged end of an ensemble.  The FP64 pipe retires a warp instruction per
// 17 cycles per SM, so the k^2 multiply-adds of a row run in fixed point on the
// integer pipe (three 32 x 32 -> 64-bit multiply-adds each): x and trans are
// rounded once to 2^-58 of their (Frobenius) norms, and by Cauchy-Schwarz no sum
// leaves 64 bits.  The mean is the mean of the products, so axb stays out of the
// perturbations.  Measured, 32 768
// solves of 40 members over 7200 columns of 97 rows: 4.4 -> 1.3 ms (a block per
// column, 1.8 ms; FP64 at full lanes would take 2.3).
template <int kThreads>
__global__ void __launch_bounds__(kThreads, 768 / kThreads)
    cube_apply_kernel(Geometry g, CubeDev cd, const double* trans, const double* xb, const double* axb,
                      double* xa, double* axa) {
  const int k = g.ens, n = g.n, LDT = k + 1;  // odd stride for even k: few conflicts in staging
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int half = kThreads / k, batch = 2 * half;  // rows at a time
  const int kx = (k + 1) & ~1;                      // rows of X begin on 16 bytes
  extern __shared__ __align__(16) int2 smi[];
  int2* const Tt = smi;                                               // trans(i, e) at e + LDT i
  int2* const X = Tt + k * LDT;                                       // batch x kx
  long long* const P = reinterpret_cast<long long*>(X + batch * kx);  // batch x k products
  double* const mean = reinterpret_cast<double*>(P + batch * k);      // batch
  long long* const row = reinterpret_cast<long long*>(mean + batch);  // r + n (cell) of a batch row
  int* const ex = reinterpret_cast<int*>(row + batch);
  __shared__ unsigned s_emax[kThreads / 32];
  __shared__ float s_fro[kThreads / 32];
  const double inv_k = 1.0 / (double)k;
  const int my_q = tid / k, my_e = tid - my_q * k;  // this thread's row of a batch and member
  // this thread's elements of trans: place in memory, place in Tt
  const int step_e = kThreads / k, step_i = kThreads - step_e * k;
  auto cell = [&](int glat, int glon) {
    return (size_t)(glat - 1 + g.halo) +
           (size_t)(g.num_lat + 2 * g.halo) * (size_t)(glon - 1 + g.halo);
  };
  auto each = [&](auto f) {
    int e = my_q, m = my_e;  // trans(m, e)
#pragma unroll 4
    for (int idx = tid; idx < k * k; idx += kThreads) {
      f(idx, e + LDT * m);
      e += step_e;
      m += step_i;
      if (m >= k) {
        m -= k;
        ++e;
      }
    }
  };
  // the block's cubes (mi, mj), level groups and columns
  int b, mi0, mi1, mj0, mj1, gi0 = 0, gi1 = cd.ngroups, lat0, lon0, nlat = 1, nlon = 1;
  const int st = cd.stride, cn = cd.cube_n;
  const bool per_solve = st == cn;
  if (per_solve) {
    const int cube = blockIdx.x / cd.ngroups;
    b = 0;
    int hi = g.global_nx * g.global_ny;  // cube_off[b] <= cube < cube_off[hi]
    while (hi - b > 1) {
      const int mid = (b + hi) / 2;
      if (cd.cube_off[mid] <= cube)
        b = mid;
      else
        hi = mid;
    }
    const int4 bk = g.blk[b];  // s_lat, e_lat, s_lon, e_lon (1-based)
    const int m = cube - cd.cube_off[b], ncj = (bk.y - bk.x) / st + 1;
    mi0 = mi1 = m / ncj;
    mj0 = mj1 = m - mi0 * ncj;
    gi0 = blockIdx.x - cube * cd.ngroups;
    gi1 = gi0 + 1;
    lat0 = bk.x + mj0 * st;
    lon0 = bk.z + mi0 * st;
    nlat = min(cn, bk.y - lat0 + 1);
    nlon = min(cn, bk.w - lon0 + 1);
  } else {
    lat0 = blockIdx.x % g.num_lat + 1;
    lon0 = blockIdx.x / g.num_lat + 1;
    b = block_of(lon0, g.num_lon, g.global_ny) * g.global_nx + block_of(lat0, g.num_lat, g.global_nx);
    const int j = lat0 - g.blk[b].x + 1, i = lon0 - g.blk[b].z + 1;
    mj0 = first_cube(j, cn, st);
    mj1 = (j - 1) / st;
    mi0 = first_cube(i, cn, st);
    mi1 = (i - 1) / st;
  }
  const int ncj = (g.blk[b].y - g.blk[b].x) / st + 1;
  const int count = (mj1 - mj0 + 1) * (mi1 - mi0 + 1);
  const int solves = count * (gi1 - gi0);
  for (int sv = 0; sv < solves; ++sv) {
    const int mm = sv / (gi1 - gi0), gi = gi0 + sv - mm * (gi1 - gi0);
    const int mi = mi0 + mm / (mj1 - mj0 + 1), mj = mj0 + mm % (mj1 - mj0 + 1);
    const int cube = cd.cube_off[b] + mi * ncj + mj;
    const bool first = mm == 0;
    const double* T = trans + ((size_t)cube * cd.ngroups + gi) * k * k;
    // rows of levels sk..ek of the 3-D variables; the 2-D ones with the last group
    const int sk = gi * cd.cube_nz + 1, ek = min(sk + cd.cube_nz - 1, g.nz);
    int nrows = n;
    if (cd.grouped) {
      nrows = 0;
      for (int v = 0; v < g.n_var; ++v)
        nrows += g.var_lev[v] == 1 ? (ek == g.nz ? 1 : 0) : ek - sk + 1;
    }
    // ---- trans in fixed point
    unsigned emax = 0;
    each([&](int idx, int at) {
      const double a = T[idx];
      Tt[at] = make_int2(__double2loint(a), __double2hiint(a));
      emax = max(emax, ((unsigned)__double2hiint(a) >> 20) & 0x7ffu);
    });
    emax = __reduce_max_sync(0xffffffffu, emax);
    if (lane == 0) s_emax[warp] = emax;
    __syncthreads();
    for (int w = 0; w < kThreads / 32; ++w) emax = max(emax, s_emax[w]);
    float fro = 0.0f;
    each([&](int, int at) {
      const float f = rough(__hiloint2double(Tt[at].y, Tt[at].x), emax);
      fro = fmaf(f, f, fro);
    });
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) fro += __shfl_xor_sync(0xffffffffu, fro, o);
    if (lane == 0) s_fro[warp] = fro;
    __syncthreads();
    fro = 0.0f;
    for (int w = 0; w < kThreads / 32; ++w) fro += s_fro[w];
    const bool t_bad = emax == 2047u;
    const int Et = norm_exponent(emax, fro);
    each([&](int, int at) { Tt[at] = to_fixed(__hiloint2double(Tt[at].y, Tt[at].x), Et); });
    // ---- rows
    const int total = nrows * nlat * nlon;
    for (int r0 = 0; r0 < total; r0 += batch) {
      const int nb = min(batch, total - r0);
      for (int q = warp; q < nb; q += kThreads / 32) {
        const int c = (r0 + q) / nrows, ci = c / nlat;
        int r = r0 + q - c * nrows;
        if (cd.grouped) {
          int left = r;
          for (int v = 0; v < g.n_var; ++v) {
            const int nv = g.var_lev[v] == 1 ? (ek == g.nz ? 1 : 0) : ek - sk + 1;
            if (left >= 0 && left < nv)
              r = g.var_start[v] + (g.var_lev[v] == 1 ? 0 : sk - 1 + left);
            left -= nv;
          }
        }
        const size_t place = r + (size_t)n * cell(lat0 + c - ci * nlat, lon0 + ci);
        const double* xr = xb + (size_t)k * place;
        double x[4];
        unsigned em = 0;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          x[u] = 0.0;
          if (32 * u >= k) continue;
          if (lane + 32 * u < k) x[u] = xr[lane + 32 * u];
          em = max(em, ((unsigned)__double2hiint(x[u]) >> 20) & 0x7ffu);
        }
        em = __reduce_max_sync(0xffffffffu, em);
        float f2 = 0.0f;
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          if (32 * u >= k) continue;
          const float f = rough(x[u], em);
          f2 = fmaf(f, f, f2);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) f2 += __shfl_xor_sync(0xffffffffu, f2, o);
        const int E = norm_exponent(em, f2);
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (lane + 32 * u < k) X[q * kx + lane + 32 * u] = to_fixed(x[u], E);
        if (lane == 0) {
          ex[q] = em == 2047u || t_bad ? kBad : E + Et - 2 * 1081 + 58;
          row[q] = (long long)place;
        }
      }
      __syncthreads();
      // x . trans(:, e) in units of 2^58, of this thread's rows my_q and my_q + half
      long long p[2] = {0, 0};
      if (my_q < min(nb, half)) {
        const int2* const t = Tt + my_e;
        const int2* const x0 = X + my_q * kx;
        const int2* const x1 = my_q + half < nb ? x0 + half * kx : x0;
        long long h0 = 0, h1 = 0, m0 = 1 << 27, m1 = 1 << 27;
        auto add = [](long long& hs, long long& ms, int xl, int xh, int2 w) {
          hs += (long long)xh * w.y;
          ms += (long long)xh * w.x;
          ms += (long long)xl * w.y;
        };
        const int2* tq = t;
#pragma unroll 2
        for (int q = 0; q + 1 < k; q += 2, tq += 2 * LDT) {
          const int4 a = *reinterpret_cast<const int4*>(x0 + q);
          const int4 c = *reinterpret_cast<const int4*>(x1 + q);
          const int2 w0 = tq[0], w1 = tq[LDT];
          add(h0, m0, a.x, a.y, w0);
          add(h1, m1, c.x, c.y, w0);
          add(h0, m0, a.z, a.w, w1);
          add(h1, m1, c.z, c.w, w1);
        }
        if (k & 1) {
          const int2 w = t[LDT * (k - 1)];
          add(h0, m0, x0[k - 1].x, x0[k - 1].y, w);
          add(h1, m1, x1[k - 1].x, x1[k - 1].y, w);
        }
        p[0] = 4 * h0 + (m0 >> 28);
        p[1] = 4 * h1 + (m1 >> 28);
        P[tid] = p[0];
        if (my_q + half < nb) P[tid + half * k] = p[1];
      }
      __syncthreads();
      for (int q = warp; q < nb; q += kThreads / 32) {
        long long sum = 0;
        for (int e = lane; e < k; e += 32) sum += P[q * k + e];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (lane == 0) {
          const double m = scaled(sum, ex[q]) * inv_k;
          double* ao = axa + row[q];
          const double ab = axb[row[q]];
          const bool fin = (((unsigned)__double2hiint(ab) >> 20) & 0x7ffu) != 2047u;
          mean[q] = fin ? m : ab - ab;  // NaN, as dist - mean
          *ao = first ? ab + m : *ao + (ab + m);
        }
      }
      __syncthreads();
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        const int q = my_q + u * half;
        if (my_q < half && q < nb) {
          double* xo = xa + (size_t)k * row[q] + my_e;
          const double v = scaled(p[u], ex[q]) - mean[q];
          *xo = first ? v : *xo + v;
        }
      }
      // (the next batch's rows are written after every read of X; ex, row and
      // mean are read here, written there)
      __syncthreads();
    }
  }
  if (count > 1) {
    const size_t ci = cell(lat0, lon0);
    __syncthreads();
    for (int r = 0; r < n; ++r) {
      double* xo = xa + (size_t)k * (r + (size_t)n * ci);
      if (tid < k) xo[tid] = xo[tid] / (double)count;
      if (tid == 0) axa[r + (size_t)n * ci] = axa[r + (size_t)n * ci] / (double)count;
    }
  }
}

}  // namespace

void launch_cube_apply(const Geometry& g, const CubeDev& cd, int nsolves, const double* trans,
                       const double* xb, const double* axb, double* xa, double* axa,
                       cudaStream_t stream) {
  const int k = g.ens;
  const bool per_solve = cd.stride == cd.cube_n;
  const int grid = per_solve ? nsolves : g.num_lat * g.num_lon;
  auto run = [&](auto kernel, int threads) {
    const size_t batch = 2 * (threads / k);
    const size_t smem = 8 * ((size_t)k * (k + 1) + batch * (((k + 1) & ~1) + k + 3));
    allow_smem(kernel, smem);
    kernel<<<grid, threads, smem, stream>>>(g, cd, trans, xb, axb, xa, axa);
  };
  // Smaller blocks hide the steps between barriers better; above 64 members 128 threads
  // hold a single row each time and idle, unless there are few rows.  At 128 / 256
  // threads: 32 768 solves of 28 rows of 40 members 1.28 / 1.52 ms; single levels, 12
  // rows of 15 members 19 / 24 us, 12 of 70 30 / 33 us, 27 of 85 84 / 56 us.
  const int rows = (cd.grouped ? g.n_var * cd.cube_nz : g.n) * (per_solve ? cd.cube_n * cd.cube_n : 1);
  if (k <= 64 || rows * k <= 1024)
    run(cube_apply_kernel<128>, 128);
  else
    run(cube_apply_kernel<256>, 256);
}

}  // namespace lg
