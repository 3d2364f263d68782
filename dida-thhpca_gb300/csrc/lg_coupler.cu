// lg_coupler.cu -- GMCORE state to the DA background layout.
//
// The step before the analysis in the coupled cycle: GMCORE's u and v live on
// the C grid (u at half longitudes, v at half latitudes), pt and ps at cell
// centres; gmcore2da_send_coupling (gmcore_coupler.F90:153-284) moves u and v
// to the centres,
//   u(i, j) = (u_f(i, j) + u_f(i-1, j)) / 2,
//   v(i, j) = 2 (v_f(i, j-1) area_subcell(1, j) + v_f(i, j) area_subcell(2, j)) / area_cell(j),
// and the coupler delivers the four fields as the DA's xb(ens, n, lat, lon)
// with n = ps, u levels, v levels, pt levels and the longitude halo filled
// periodically (module_da_coupler.F90:91-147, 350-414).  One GPU holds the
// whole globe, so the MCT transfer is one HBM-bound kernel, members fastest on
// both sides (coalesced reads and writes).
#include <algorithm>

#include "lg_internal.h"

namespace lg {

namespace {

// x / 2, exactly as the FP64 pipe rounds it: the exponent goes down by one on the
// bit pattern, except for values that are zero, near the subnormals, infinite or
// NaN, which are multiplied.
__device__ inline double halved(double x) {
  const int hi = __double2hiint(x);
  if ((unsigned)(((hi >> 20) & 0x7ff) - 2) < 2045u) return __hiloint2double(hi - (1 << 20), __double2loint(x));
  return x * 0.5;
}

// Threads along x take the members, one or two each (V: two where the ensemble
// size is even and every array is 16-byte aligned, so that a load moves 16
// bytes), threads along y neighbouring longitudes (with halo) of one latitude,
// each all levels; no integer division, reads and writes contiguous in the
// members.  The v weights 2 area_subcell(., j) / area_cell(j) are formed once
// per block (two FP64 operations per v value instead of a division; the result
// differs from the reference's expression by rounding only).
//
// The FP64 pipe retires a warp instruction per 17 cycles per SM, so the four FP64
// operations per level and member (244 us at 180 x 90 x 32 levels, 64 members)
// and two divisions per thread cost as much as the 1.6 GB of HBM traffic (240
// us): the halving of u is done on the bit pattern and the divisions once per
// block.  At that size the whole call went from 465 to 305 us (the kernel 292 us,
// 5.5 TB/s); levels spread over more threads, each with its own divisions, took
// 412 us.
template <typename V>
__global__ void __launch_bounds__(sizeof(V) == 16 ? 512 : 1024)
    gmcore_to_da_kernel(int ens, int num_lat, int num_lon, int nz, int halo,
                        const V* __restrict__ ps, const V* __restrict__ u_half,
                        const V* __restrict__ v_half, const V* __restrict__ pt,
                        const double* __restrict__ area_subcell,
                        const double* __restrict__ area_cell, V* __restrict__ xb) {
  const int le = blockIdx.x * blockDim.y + threadIdx.y;  // 0-based longitude with halo
  const int jj = blockIdx.y;  // 0-based latitude
  const int m = threadIdx.x;  // in units of V, as ens
  __shared__ double s_w[2];
  if (threadIdx.x < 2 && threadIdx.y == 0)
    s_w[threadIdx.x] = 2.0 * area_subcell[2 * jj + threadIdx.x] / area_cell[jj];
  __syncthreads();
  if (m >= ens || le >= num_lon + 2 * halo) return;
  const int n = 1 + 3 * nz;
  const int nlat_e = num_lat + 2 * halo;
  int ii = le - halo;  // 0-based longitude, periodic
  ii = ii < 0 ? ii + num_lon : (ii >= num_lon ? ii - num_lon : ii);
  const int iw = ii == 0 ? num_lon - 1 : ii - 1;
  const double w_s = s_w[0], w_n = s_w[1];
  const size_t plane = (size_t)num_lat * num_lon * ens;
  const size_t vplane = (size_t)(num_lat + 1) * num_lon * ens;
  const size_t cell = ((size_t)jj * num_lon + ii) * ens + m;
  const size_t west = ((size_t)jj * num_lon + iw) * ens + m;
  const size_t vs0 = ((size_t)jj * num_lon + ii) * ens + m, vn0 = vs0 + (size_t)num_lon * ens;
  V* out = xb + ((size_t)le * nlat_e + (jj + halo)) * n * ens + m;
  auto mean = [](V a, V b) {
    if constexpr (sizeof(V) == 16)
      return make_double2(halved(a.x + b.x), halved(a.y + b.y));
    else
      return halved(a + b);
  };
  auto weigh = [&](V north, V south) {
    if constexpr (sizeof(V) == 16)
      return make_double2(fma(north.x, w_n, south.x * w_s), fma(north.y, w_n, south.y * w_s));
    else
      return fma(north, w_n, south * w_s);
  };
  out[0] = ps[cell];
#pragma unroll 2
  for (int k = 0; k < nz; ++k) {
    const V uc = u_half[k * plane + cell], uw = u_half[k * plane + west];
    const V vn = v_half[k * vplane + vn0], vs = v_half[k * vplane + vs0], p = pt[k * plane + cell];
    out[(size_t)(1 + k) * ens] = mean(uc, uw);
    out[(size_t)(1 + nz + k) * ens] = weigh(vn, vs);
    out[(size_t)(1 + 2 * nz + k) * ens] = p;
  }
}

}  // namespace

cudaError_t launch_gmcore_to_da(int ens, int num_lat, int num_lon, int nz, int halo,
                                const double* ps, const double* u_half, const double* v_half,
                                const double* pt, const double* area_subcell,
                                const double* area_cell, double* xb, cudaStream_t stream) {
  // 16-byte loads where every row starts on a 16-byte boundary
  const uintptr_t at = (uintptr_t)ps | (uintptr_t)u_half | (uintptr_t)v_half | (uintptr_t)pt |
                       (uintptr_t)xb;
  auto run = [&](auto kernel, auto unit, int e) {
    using V = decltype(unit);
    const int bx = (e + 31) / 32 * 32;
    const int by = std::max(1, 128 / bx);
    const dim3 grid((num_lon + 2 * halo + by - 1) / by, num_lat);
    kernel<<<grid, dim3(bx, by), 0, stream>>>(
        e, num_lat, num_lon, nz, halo, reinterpret_cast<const V*>(ps),
        reinterpret_cast<const V*>(u_half), reinterpret_cast<const V*>(v_half),
        reinterpret_cast<const V*>(pt), area_subcell, area_cell, reinterpret_cast<V*>(xb));
  };
  if (ens % 2 == 0 && at % 16 == 0)
    run(gmcore_to_da_kernel<double2>, double2{}, ens / 2);
  else
    run(gmcore_to_da_kernel<double>, 0.0, ens);
  return cudaGetLastError();
}

}  // namespace lg
