// lg_gram64_tc.cu -- FP64 weighted Gram matrices of up to 64 members on the
// 5th-generation tensor cores, by exact integer slices.
//
// Same quantities as lg_gram.cu (letkf_core.F90:58-75,146-195):
//   z_e = y_e rr_e,  rr_e = sqrt(rdiaginv(e) rloc_k(e)),  d~_e = rr_e d_e
//   C = sum_e z_e z_e^T,   t = sum_e z_e d~_e
//
// Why: the FP64 pipe of this GPU multiplies 2 lanes per cycle per SM, so the
// k(k+1)/2 products of one 64-member entry take about 1040 cycles of an SM, and
// the plain FP64 Gram (gram64_kernel) was 80 to 95 % of a plain-FP64 analysis.
// Here each z_ei is rounded once to a 53-bit integer Z relative to the largest
// |z| of the chunk (below a power of two 2^S), and Z is cut into six signed
// 9-bit digits,
//   z = 2^(S-53) Z,   Z = sum_a d_a 2^(45-9a),   -256 <= d_a <= 256,
// which are exact in FP16 (the error-free splitting of K. Ozaki, T. Ogita, S. Oishi and S. M.
// Rump, "Error-free transformations of matrix multiplication by using fast routines of matrix
// multiplication and its applications", Numerical Algorithms 59, 2012).  A product of digits has at most 16 bits and a
// tcgen05.mma accumulator holds 24 exactly, so the FP32 sums of up to 256
// entries are exact integers; they are combined in 64-bit integers.  Pairs of
// slices (a, b) with a + b >= 7 (below 2^-63 of the largest product) are left
// out, and of the rest only one of (a, b) and (b, a) is formed (C is symmetric).
// Up to 40 members three slices make one M = 128 operand.  They lie as [zero zero
// 3 4 5 0 1 2], 40 rows each, followed by the slices of d~ as rows of their own:
//   A = [0;1;2] x B = [8 rows of zero, 3 4 5 0 1 2, d~] (N = 256)   01 .. 25, d~
//   A = [3;4;5] x B = d~ (N = 16), into the first 8 columns         d~
//   A = [zero;zero;3] x B = [3] (N = 48), onto 20                   33
// 256 tensor-memory columns, so two buffers alternate and the sums of one are
// taken out while the next is filled.  From 41 members on the slices lie as [zero
// 5 0 1 3 2 4], 64 rows each, and two neighbours make an operand ("first | second"):
//   block 0   A = [5;0] x B = [0]              50 | 00
//   1..4      A = [0;1] x B = [1 3 2 4]        01 03 02 04 | 11 13 12 14
//   5         A = [3;2] x B = [3]              33 | 23
//   6         A = [2;4] x B = [2], + [zero;5] x [1]   22 | 42 + 51
//   d~        A = [5;0], [1;3], [2;4] x B = the six slices of d~ (N = 16)
// 448 + 48 of the 512 tensor-memory columns: the sums are taken out before the
// next ones begin.  An element's error is about
// 2^-54 of the chunk's largest |z| times |z| per entry, adding up as a random
// walk; a chain of FP64 additions loses 2^-53 of the partial sum at each.
//
// One persistent CTA per SM (the accumulators fill tensor memory), 28 warps in
// four roles that work on neighbouring chunks of up to 1344 or 1536 entries:
//   weighing (7 warps)    drop the candidates whose vertical weight cannot be
//     non-zero by an integer compare of |ln p - ln p_e|, queue the others in list
//     order, and weigh the queue densely (the only FP64 work, some 35
//     instructions per kept entry);
//   converting (12)       64 entries at a time by integer arithmetic into one of
//     two operand buffers;
//   issuing (1)           the MMAs (a converting warp that issued them was late
//     for its next stage by the MMAs' own time, 2500 cycles);
//   adding up (8)         finished sums out of tensor memory, C and t.
// The rows' largest values and the levels' ln p come from small kernels before
// this one.  Roles meet at mbarriers with bounded waits (lg_set_wait_limit); the first
// that runs out raises s_abort, every role leaves its loop and the launch reports
// LG_ERR_TIMEOUT.
//
// Bound: the conversions, about 3000 issue slots of twelve warps a stage, beside
// the MMAs -- max(46, N / 2) cycles each, 220 a K = 16 chunk with three slices per
// operand, 432 with two, and about 800 while the conversions share the shared
// memory's bandwidth with their operands (22 and 50 KB a chunk).  Two slices per
// operand and one buffer at 40 members left the MMAs waiting for the sums to be
// taken out, and each sum's conversion to integers (16 lanes a cycle and SM) is
// kept to four or five per element.  Measured alone against gram64_kernel: 921 600
// solves of 40 members and 379 entries (of 1562 candidates) 727 -> 92 ms (126 with
// two slices per operand); 82 944 of 40 members, 24 entries 5.6 -> 2.7 ms; 2592 of
// 16 members, 51 entries 0.18 -> 0.08 ms; 129 600 of 64 members, 954 entries 595 ->
// 48 ms.  It wins at every size, so up to 64 members there is no other path.
// A solve with a non-finite weight, row or innovation, or with magnitudes
// outside 2^+-400, is marked by a bit pattern in its first Gram element that no
// other solve can produce, and redone by gram64_kernel.
#include "lg_device.cuh"
#include "lg_fixed.cuh"
#include "lg_internal.h"
#include "lg_tc.cuh"

namespace lg {
namespace g64 {

constexpr int kPWarps = 7, kXWarps = 12, kDWarps = 8;  // weighing, converting, adding up
constexpr int kMmaWarp = kPWarps;                     // issues the MMAs
constexpr int kX0 = kMmaWarp + 1, kD0 = kX0 + kXWarps;  // first warps (multiples of 4)
constexpr int kPThreads = 32 * kPWarps, kXThreads = 32 * kXWarps, kDThreads = 32 * kDWarps;
constexpr int kThreads = 32 * (kD0 + kDWarps);
constexpr int kStage = 64;                            // entries per stage (4 K = 16 chunks)
constexpr int kPer = 4;                               // candidates per thread and refill
constexpr int kRefill = kPer * kPThreads;
constexpr int kGroup = 4;                             // stages per exact FP32 sum (256 entries)
// Operands and sums in shared memory.  A slice is kRows rows x K = 16 FP16.
template <bool kThree>
struct Layout {
  static constexpr int kRows = kThree ? 40 : 64;
  static constexpr int kSlice = kRows * 16 * 2;
  // [zero zero 3 4 5 0 1 2], d~ (8 rows), d~ again (16 rows); [zero 5 0 1 3 2 4], d~ (16)
  static constexpr int kTileD = (kThree ? 8 : 7) * kSlice;
  static constexpr int kTileD2 = kTileD + 8 * 16 * 2;
  static constexpr int kChunk = kThree ? kTileD2 + 16 * 16 * 2 : kTileD + 16 * 16 * 2;
  static constexpr int kStageBytes = 4 * kChunk;
  static constexpr int kUStride = kThree ? 41 : 65;
  static constexpr int kURows = kThree ? 120 : 64;  // a row per accumulator row, or per member
  // entries of a chunk (one scale), and chunks in flight between the roles: one more
  // where the operands leave room for it, so that solves of different lengths even
  // out
  static constexpr int kQueue = kThree ? 1344 : 1536, kDepth = kThree ? 3 : 2;
  static constexpr int kQueueBytes = kQueue * (16 + 8);
  static constexpr int kSmem =
      2 * kStageBytes + kDepth * kQueueBytes + kURows * kUStride * 8;
  // memory position of slice a
  static __host__ __device__ constexpr int pos(int a) {
    return kThree ? (a >= 3 ? a - 1 : a + 5)
                  : a == 5 ? 1 : a == 0 ? 2 : a == 1 ? 3 : a == 3 ? 4 : a == 2 ? 5 : 6;
  }
};
// C's exact sums are kept in units of 2^-51 of the largest product times 2^-1:
// twice the sum of 1536 products stays below 2^63
constexpr int kDrop = 10;
// named barriers: the weighing and the adding warps' own
constexpr int kBarP = 1, kBarD = 2;
constexpr int kTmemCols = 512;
constexpr int kColD = 448;                            // first column of the d~ products
constexpr int kExLimit = 400;

constexpr long long bias() {  // 256 in every digit
  long long b = 0;
  for (int j = 0; j < 6; ++j) b += 256ll << (9 * j);
  return b;
}

// kind::f16, FP16 A/B, FP32 D, K-major, M = 128, N
__host__ __device__ constexpr uint32_t idesc(int n) {
  return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

__device__ inline void mma(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t id, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(da), "l"(db), "r"(id), "r"(acc));
}

// eight consecutive accumulator columns of this thread's lane (no wait)
__device__ inline void tmem_ld8(uint32_t taddr, float* v) {
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]),
                 "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ inline void tmem_ld4(uint32_t taddr, float* v) {
  uint32_t r[4];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 4; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ inline void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

__device__ inline void bar_sync(int id, int count) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}
__device__ inline void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(tc::smem_u32(bar)) : "memory");
}

// (hi 2^27 + lo) 2^ex rounded to nearest-even
__device__ inline double wide_to_double(long long hi, long long lo, int ex) {
  __int128 v = ((__int128)hi << 27) + lo;
  if (v == 0) return 0.0;
  const bool neg = v < 0;
  unsigned __int128 m = neg ? (unsigned __int128)(-v) : (unsigned __int128)v;
  const unsigned long long mh = (unsigned long long)(m >> 64), ml = (unsigned long long)m;
  const int p = mh ? 127 - __clzll((long long)mh) : 63 - __clzll((long long)ml);
  unsigned long long mant;
  if (p <= 52) {
    mant = ml << (52 - p);
  } else {
    const int drop = p - 52;
    mant = (unsigned long long)(m >> drop);
    const unsigned __int128 rest = m & (((unsigned __int128)1 << drop) - 1);
    const unsigned __int128 half = (unsigned __int128)1 << (drop - 1);
    if (rest > half || (rest == half && (mant & 1))) ++mant;  // may carry into the exponent
  }
  const unsigned long long bits = ((unsigned long long)(p + ex + 1023 - 1) << 52) + mant;
  return __longlong_as_double((long long)(bits | (neg ? 0x8000000000000000ull : 0ull)));
}

// 32 (Z + bias) and the sign of one element: y (bit pattern) times the entry's
// weight mantissa.  par: (R >> 29, R & (2^29 - 1), shift base, entry) with rr =
// R 2^(er - 1080), R < 2^58.  Y = |y| 2^(58 + ...) at the chunk's scale: the
// shift base is the row's largest biased exponent plus how far the row's bound
// lies below the chunk's, so Y R / 2^58 = 32 |Z| + at most two units.  The
// digits are those of |Z| (9 bits each from bit 5 on: three in each 32-bit
// word); the sign is applied to them in FP16.
__device__ inline unsigned long long digits_of(unsigned hi, unsigned lo, const int4& par) {
  const int e = (int)((hi << 1) >> 21);
  const unsigned mh = (hi & 0xfffffu) | 0x100000u;
  const int sh = min(par.z - e, 63);
  const unsigned long long Y = ((((unsigned long long)mh << 32) | lo) << 6) >> sh;
  const unsigned yh = (unsigned)(Y >> 29), yl = (unsigned)Y & 0x1fffffffu;
  const unsigned rh = (unsigned)par.x, rl = (unsigned)par.y;
  unsigned long long mid = (unsigned long long)yl * rh + (1ull << 28);
  mid += (unsigned long long)yh * rl;
  return (unsigned long long)yh * rh + (16ull + ((unsigned long long)bias() << 5)) +
         (unsigned)(mid >> 29);
}

// the digit pairs of two neighbouring entries as packed FP16, slice a = 0..5;
// hi0, hi1: words whose top bits are the two signs
__device__ inline void digit_pairs(unsigned long long z0, unsigned long long z1, unsigned hi0,
                                   unsigned hi1, uint32_t* out) {
  const unsigned a0 = (unsigned)z0, b0 = (unsigned)z1;
  const unsigned a1 = (unsigned)(z0 >> 32), b1 = (unsigned)(z1 >> 32);
  // u + 1024 in FP16 is 0x6400 | u for u < 1024; minus 1280 leaves the signed
  // digit: +-1 (u + 1024) -+ 1280, both exact
  const unsigned sg = ((hi0 >> 16) & 0x8000u) | (hi1 & 0x80000000u);
  const uint32_t one = sg | 0x3c003c00u, off = sg ^ 0xe500e500u;
  auto pack = [&](unsigned x, unsigned y, unsigned mask) -> uint32_t {
    const unsigned t = (x & (mask & 0xffffu)) | 0x64006400u;
    const unsigned h = (y & (mask & 0xffff0000u)) | t;
    uint32_t r;
    asm("fma.rn.f16x2 %0, %1, %2, %3;" : "=r"(r) : "r"(h), "r"(one), "r"(off));
    return r;
  };
  out[5] = pack(a0 >> 5, b0 << 11, 0x01ff01ffu);
  out[4] = pack(a0 >> 14, b0 << 2, 0x01ff01ffu);
  out[3] = pack(a0 >> 23, b0 >> 7, 0x01ff01ffu);
  out[2] = pack(a1, b1 << 16, 0x01ff01ffu);
  out[1] = pack(a1 >> 9, b1 << 7, 0x01ff01ffu);
  out[0] = pack(a1 >> 18, b1 >> 2, 0x03ff03ffu);
}

}  // namespace g64

// High word of the largest |y| of each H(x) row: its biased exponent from bit 20
// on (0: all zero; 2047: a non-finite value), the leading mantissa bits below.
__global__ void row_exponent_kernel(int ens, int64_t rows, const double* yb, int* yexp) {
  const int64_t r = (int64_t)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
  if (r >= rows) return;
  const int lane = threadIdx.x & 31;
  unsigned e = 0;
  for (int i = lane; i < ens; i += 32)
    e = max(e, (unsigned)__double2hiint(yb[(size_t)r * ens + i]) & 0x7fffffffu);
  e = __reduce_max_sync(0xffffffffu, e);
  if (lane == 0) yexp[r] = (int)e;
}

void launch_row_exponents(int ens, int64_t rows, const double* yb, int* yexp,
                          cudaStream_t stream) {
  if (rows == 0) return;
  row_exponent_kernel<<<(unsigned)((rows + 7) / 8), 256, 0, stream>>>(ens, rows, yb, yexp);
}

// ln p of each solve's level into the first element of its t (which
// gram64_tc_kernel reads before it writes t)
__global__ void level_lnp_kernel(Geometry g, SolveBatch b, const double* axb, double* t) {
  const int s = blockIdx.x * blockDim.x + threadIdx.x;
  if (s >= b.nsolves) return;
  int col, kk;
  solve_col_level(b, s, col, kk);
  const int glat = col % g.num_lat + 1, glon = col / g.num_lat + 1;
  const size_t ci = (size_t)(glat - 1 + g.halo) +
                    (size_t)(g.num_lat + 2 * g.halo) * (size_t)(glon - 1 + g.halo);
  t[(size_t)s * g.ens] = alnp_level(g, kk, axb[g.ps_row + (size_t)g.n * ci]);
}

// what the weighing warps tell the converting ones about a queue
struct QueueHead {
  int s;         // solve, < 0: no more
  int stages;    // stages of kStage entries (0: nothing with weight)
  int S, Sd;     // |z| < 2^S, |d~| < 2^Sd
  int first;     // the solve's first chunk: C and t are written, else added to
  int bad;       // leave the solve to gram64_kernel
};

// kR: units (member, 4 entries) of a stage per converting thread -- 2 up to 48
// members, 3 above.  kThree: three slices in an operand's 128 rows (up to 40
// members).  kLimited: waits end after wait_ns (a clock in the waits of every launch
// would cost them registers).
template <int kR, bool kThree, bool kLimited>
__global__ void __launch_bounds__(g64::kThreads, 1)
    gram64_tc_kernel(Geometry g, HxDev hx, ListDev l, SolveBatch b, int lower, long long wait_ns,
                     double* Cout, double* tout, int* err) {
  using namespace g64;
  using L = Layout<kThree>;
  constexpr int kSlice = L::kSlice, kTileD = L::kTileD, kChunkBytes = L::kChunk,
                kStageBytes = L::kStageBytes, kUStride = L::kUStride, kQueue = L::kQueue,
                kQueueBytes = L::kQueueBytes, kDepth = L::kDepth;
  constexpr int kBufs = kThree ? 2 : 1;  // accumulator buffers in tensor memory
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // operand buffer multiplied, converted; queue full, empty; exact sum complete,
  // taken out (one phase per group of stages: the adding warps wait for no stage
  // in between, so a stage barrier's parity would not tell them which phase it is)
  __shared__ uint64_t m_mma[2], m_conv[2], m_sum[2], m_drain[2], m_full[kDepth], m_empty[kDepth];
  __shared__ uint32_t tmem_base_sh;
  __shared__ int s_wcnt[2][kPWarps];
  __shared__ longlong2 s_t[kThree ? 3 : 2][64];
  __shared__ int s_kmax, s_dmax, s_nf;
  __shared__ int s_before[kPThreads];  // a weighing thread's count before the present solve
  __shared__ volatile int s_abort;
  __shared__ int s_stop[2];  // s_abort as the weighing and the adding warps agree on it
  __shared__ QueueHead s_head[kDepth];

  const int k = g.ens;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const bool batch = b.mode == 1;
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) {
      tc::mbar_init(&m_mma[i], 1);
      tc::mbar_init(&m_conv[i], kXWarps);
      tc::mbar_init(&m_sum[i], 1);
      tc::mbar_init(&m_drain[i], kDWarps);
    }
    for (int i = 0; i < kDepth; ++i) {
      tc::mbar_init(&m_full[i], kPThreads);
      tc::mbar_init(&m_empty[i], kXWarps + 1 + kDWarps);
    }
    s_abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // the operand buffers' rows that stay zero: zero slices, members above k, the
  // d~ tiles' other rows
  for (int i = tid; i < 2 * kStageBytes / 16; i += kThreads)
    reinterpret_cast<uint4*>(smem_raw)[i] = make_uint4(0, 0, 0, 0);
  tc::fence_proxy_async();
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     tc::smem_u32(&tmem_base_sh)),
                 "r"(kTmemCols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc::fence_before();
  __syncthreads();
  tc::fence_after();
  const uint32_t tmem = tmem_base_sh;
  auto q_par = [&](int qb) {
    return reinterpret_cast<int4*>(smem_raw + 2 * kStageBytes + qb * kQueueBytes);
  };
  auto q_d = [&](int qb) { return reinterpret_cast<long long*>(q_par(qb) + kQueue); };
  auto wait = [&](uint64_t* bar, uint32_t parity) {
    if (!s_abort && !(kLimited ? tc::mbar_wait_ns(bar, parity, wait_ns) : tc::mbar_wait(bar, parity)))
      s_abort = 1;
    __syncwarp();
  };
  // s_abort, the same for the lanes of a warp
  auto stopped = [&]() { return __any_sync(0xffffffffu, s_abort != 0); };

  if (warp < kX0) {
  // registers: 256 x 56 + 384 x 80 + 256 x 72 within the launch's 896 x 72
  asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
  if (warp < kPWarps) {
    // ================= weighing warps
    const bool vertical = !batch && g.vert_dist > 0.0;
    // |al - ln p| / vert_dist rounds to more than 2 exactly where |al - ln p| > 2
    // vert_dist, and to more than 1 where it is > vert_dist: the sides of the
    // localisation's boundaries are taken from these, not from the product with the
    // rounded reciprocal.  Compared on the bit patterns; a NaN stays a candidate.
    const long long lim_bits = __double_as_longlong(2.0 * g.vert_dist);
    const long long one_bits = __double_as_longlong(g.vert_dist);
    // (a product differs by less than two roundings from the quotient)
    const double inv_vd = 1.0 / g.vert_dist;
    int work = 0;     // entries with weight
    unsigned nq = 0;  // queues filled so far
    // 1: a queue is filled; 0: the solve is left to gram64_kernel; -1: stop
    auto fill = [&](int s, int64_t base, int p, double al, int& scan, bool& first) -> int {
      const int qb = nq % kDepth;
      int4* const par = q_par(qb);
      long long* const qd = q_d(qb);
      if (nq >= kDepth) wait(&m_empty[qb], (nq / kDepth - 1) & 1);
      bar_sync(kBarP, kPThreads);  // every thread has read the last queue's maxima
      if (tid == 0) {
        s_kmax = 0;
        s_dmax = 0;
        s_nf = 0;
        s_stop[0] = s_abort;
      }
      bar_sync(kBarP, kPThreads);
      if (s_stop[0]) return -1;
      int qn = 0;
      while (qn <= kQueue - kRefill && scan < p) {
        int ent[kPer];
        double dz[kPer];
        unsigned m[kPer];
        bool keep[kPer];
        const int i0 = scan + warp * (32 * kPer) + lane;
#pragma unroll
        for (int r = 0; r < kPer; ++r) {
          keep[r] = i0 + 32 * r < p;
          ent[r] = i0 + 32 * r;
          dz[r] = 0.0;
          if (keep[r] && !batch) ent[r] = l.ent[base + i0 + 32 * r];
        }
        if (vertical) {
#pragma unroll
          for (int r = 0; r < kPer; ++r)
            if (keep[r]) dz[r] = hx.lnp[ent[r]];
#pragma unroll
          for (int r = 0; r < kPer; ++r) {
            dz[r] = al - dz[r];
            const long long a = __double_as_longlong(dz[r]) & 0x7fffffffffffffffll;
            keep[r] = keep[r] && !(a > lim_bits && a <= 0x7ff0000000000000ll);
          }
        }
        int c = 0;
#pragma unroll
        for (int r = 0; r < kPer; ++r) {
          m[r] = __ballot_sync(0xffffffffu, keep[r]);
          c += __popc(m[r]);
        }
        const int pb = (scan / kRefill) & 1;  // double-buffered counts: one barrier per refill
        if (lane == 0) s_wcnt[pb][warp] = c;
        bar_sync(kBarP, kPThreads);
        int off = qn;
#pragma unroll
        for (int w = 0; w < kPWarps; ++w) {
          off += w < warp ? s_wcnt[pb][w] : 0;
          qn += s_wcnt[pb][w];
        }
#pragma unroll
        for (int r = 0; r < kPer; ++r) {
          if (keep[r]) {
            const int pos = off + __popc(m[r] & ((1u << lane) - 1u));
            par[pos] = make_int4(__double2loint(dz[r]), __double2hiint(dz[r]), i0 + 32 * r, ent[r]);
          }
          off += __popc(m[r]);
        }
        scan += kRefill;
      }
      bar_sync(kBarP, kPThreads);
      // weights, densely (FP64): rr into par, d~ into qd
      int kmax = 0, dmax = 0, cnt = 0;
      bool nf = false;
      for (int q0 = tid; q0 < qn; q0 += 2 * kPThreads) {
        // two entries at a time: their loads are in flight together
        double rl[2], dep[2], dz[2];
        float rdg[2];
        int e[2];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int q = q0 + r * kPThreads;
          rl[r] = dep[r] = dz[r] = 0.0;
          rdg[r] = 0.0f;
          e[r] = 0;
          if (q >= qn) continue;
          const int4 c = par[q];
          const int64_t i = base + c.z;
          dz[r] = __hiloint2double(c.y, c.x);
          if (batch) {
            rl[r] = b.b_rloc[i];
            rdg[r] = b.b_rdiag[i];
            dep[r] = b.b_dep[i];
            const double* y = b.b_hx + (size_t)i * k;
            unsigned em = 0;
            for (int j = 0; j < k; ++j) em = max(em, (unsigned)__double2hiint(y[j]) & 0x7fffffffu);
            e[r] = (int)em;
          } else {
            rl[r] = l.rloc[i];
            rdg[r] = hx.rdiag[c.w];
            dep[r] = hx.dis[c.w];
            e[r] = hx.yexp[c.w];
          }
        }
#pragma unroll
        for (int r = 0; r < 2; ++r) {
          const int q = q0 + r * kPThreads;
          if (q >= qn) continue;
          double x = rl[r];
          if (vertical) {
            double z = fabs(dz[r]) * inv_vd;
            if ((unsigned)__double2loint(z) + 4u < 8u) {  // within four roundings of 1 or 2
              const long long a = __double_as_longlong(fabs(dz[r])), b = __double_as_longlong(z);
              if (a <= one_bits)
                z = __longlong_as_double(min(b, 0x3ff0000000000000ll));  // at most 1
              else if (a <= lim_bits)
                z = __longlong_as_double(
                    min(max(b, 0x3ff0000000000001ll), 0x4000000000000000ll));  // in (1, 2]
            }
            x = x * (g.gc_filter_vertical ? taper_fast(z) : schr(z));
          }
          double w = sqrt((double)rdg[r] * x), d = 0.0;
          if (w != 0.0) {
            d = w * dep[r];
            const int ew = (__double2hiint(w) >> 20) & 0x7ff;
            const int ed = (__double2hiint(d) >> 20) & 0x7ff;
            ++cnt;
            nf |= (e[r] >> 20) == 2047 || ew == 2047 || ed == 2047;
            if (e[r] >> 20) {
              // the bound |z| < 2^(kz - 1022): the product of the mantissas (each
              // rounded up, so at most 4) decides whether it carries
              const double fy = __hiloint2double((e[r] & 0xfffff) | 0x3ff00000, -1);
              const double fw = __hiloint2double((__double2hiint(w) & 0xfffff) | 0x3ff00000, -1);
              kmax = max(kmax, (e[r] >> 20) + ew + ((__double2hiint(fy * fw) >> 20) - 1023));
              dmax = max(dmax, ed);
            } else {
              w = 0.0;  // a row of zeros
            }
          }
          *reinterpret_cast<double*>(&par[q]) = w;
          qd[q] = __double_as_longlong(d);
        }
      }
      work += cnt;
      kmax = (int)__reduce_max_sync(0xffffffffu, (unsigned)kmax);
      dmax = (int)__reduce_max_sync(0xffffffffu, (unsigned)dmax);
      nf = __any_sync(0xffffffffu, nf);
      if (lane == 0) {
        atomicMax(&s_kmax, kmax);
        atomicMax(&s_dmax, dmax);
        if (nf) s_nf = 1;
      }
      bar_sync(kBarP, kPThreads);
      kmax = s_kmax;
      dmax = s_dmax;
      const int S = kmax - 2045, Sd = dmax - 1022;  // |z| < 2^S
      const bool bad = s_nf != 0 || (kmax && (S > kExLimit || S < -kExLimit)) ||
                       (dmax && (Sd > kExLimit || Sd < -kExLimit));
      const int qr = kmax && !bad ? (qn + kStage - 1) / kStage * kStage : 0;
      for (int q = tid; q < qr; q += kPThreads) {
        int4 pr = make_int4(0, 0, 0, 0);
        long long dq = 0;
        unsigned long long u = 0;
        if (q < qn) {
          u = *reinterpret_cast<unsigned long long*>(&par[q]);
          pr.w = par[q].w;
        } else {
          pr.w = par[0].w;  // padding: weight zero, a valid row
        }
        if (u << 1) {
          const int ew = (int)(u >> 52) & 0x7ff;
          const unsigned long long R = ((u & 0xfffffffffffffull) | 0x10000000000000ull) << 5;
          pr = make_int4((int)(R >> 29), (int)(R & 0x1fffffffull), kmax - ew, pr.w);
          const unsigned long long dv = (unsigned long long)qd[q];
          const int ed = (int)(dv >> 52) & 0x7ff;
          if (ed > 0) {
            const int sh = min(dmax - ed, 62);
            const unsigned long long mnt = (dv & 0xfffffffffffffull) | 0x10000000000000ull;
            dq = (long long)((mnt + (sh ? 1ull << (sh - 1) : 0ull)) >> sh);
            dq = (long long)((unsigned long long)dq | (dv & 0x8000000000000000ull));
          }
        }
        par[q] = pr;
        // 32 (|D| + bias) and the sign in the top bit, as digits_of leaves Z
        qd[q] = ((dq & 0x7fffffffffffffffll) + bias()) * 32 | (dq & (1ll << 63));
      }
      if (tid == 0) s_head[qb] = QueueHead{s, qr / kStage, S, Sd, first ? 1 : 0, bad ? 1 : 0};
      if (bad) work = s_before[tid];  // gram64_kernel counts this solve's entries
      mbar_arrive(&m_full[qb]);
      ++nq;
      first = false;
      return bad ? 0 : 1;
    };
    for (int s = blockIdx.x; s < b.nsolves; s += gridDim.x) {
      int64_t base;
      int p, col = 0, kk = 1;
      if (batch) {
        base = b.b_off[s];
        p = b.b_nobsl[s];
      } else {
        solve_col_level(b, s, col, kk);
        base = l.off[col];
        p = l.cnt[col];
      }
      const double al = vertical ? tout[(size_t)s * k] : 0.0;
      int scan = 0;
      bool first = true;
      int r = 1;
      s_before[tid] = work;
      do {
        r = fill(s, base, p, al, scan, first);
      } while (r > 0 && scan < p);
      if (r < 0) break;
    }
    const int qb = nq % kDepth;
    if (nq >= kDepth) wait(&m_empty[qb], (nq / kDepth - 1) & 1);
    if (tid == 0) s_head[qb] = QueueHead{-1, 0, 0, 0, 0, 0};
    mbar_arrive(&m_full[qb]);
    work = (int)__reduce_add_sync(0xffffffffu, (unsigned)work);
    if (b.work && lane == 0 && work) atomicAdd(b.work, (unsigned long long)work);
  } else {
    // ================= the issuing warp
    const uint64_t desc0 = tc::make_desc(tc::smem_u32(smem_raw), 128, 256);
    unsigned n = 0, groups = 0;  // stages issued (buffer n & 1), exact sums begun
    for (unsigned nq = 0;; ++nq) {
      const int qb = nq % kDepth;
      wait(&m_full[qb], (nq / kDepth) & 1);
      if (stopped() || s_head[qb].s < 0) break;
      const int stages = s_head[qb].stages;
      __syncwarp();
      if (lane == 0) mbar_arrive(&m_empty[qb]);
      for (int st = 0; st < stages; ++st, ++n) {
        wait(&m_conv[n & 1], (n >> 1) & 1);
        if (st % kGroup == 0) {
          // a new exact sum: the finished one is out of tensor memory
          if (groups >= kBufs)
            wait(&m_drain[(groups - kBufs) % kBufs], ((groups - kBufs) / kBufs) & 1);
          ++groups;
        }
        if (stopped()) break;
        if (lane == 0) {
          tc::fence_after();
          // descriptors of an operand at `off` bytes into the buffer: its address is
          // in the low 14 bits, in units of 16 bytes
          const uint32_t lo = (uint32_t)desc0 + (n & 1) * (kStageBytes / 16);
          const uint32_t hi = (uint32_t)(desc0 >> 32);
          auto at = [&](int off) { return (uint64_t)hi << 32 | (lo + (uint32_t)off / 16); };
#pragma unroll
          for (int c = 0; c < 4; ++c) {
            const int o = c * kChunkBytes;
            const uint32_t more = (st % kGroup > 0 || c > 0) ? 1u : 0u;
            if constexpr (kThree) {
              const uint32_t d = tmem + ((groups - 1) & 1) * 256;
              // [0;1;2] x [zero 3 4 5 0 1 2 d~], [3;4;5] x d~, [zero;zero;3] x 3
              mma(d, at(o + 5 * kSlice), at(o + 2 * kSlice - 256), idesc(256), more);
              mma(d, at(o + 2 * kSlice), at(o + L::kTileD2), idesc(16), 1u);
              mma(d + 128, at(o), at(o + 2 * kSlice), idesc(48), 1u);
            } else {
              mma(tmem, at(o + kSlice), at(o + 2 * kSlice), idesc(64), more);           // [5;0] x 0
              mma(tmem + 64, at(o + 2 * kSlice), at(o + 3 * kSlice), idesc(256), more); // [0;1] x 1 3 2 4
              mma(tmem + 320, at(o + 4 * kSlice), at(o + 4 * kSlice), idesc(64), more); // [3;2] x 3
              mma(tmem + 384, at(o + 5 * kSlice), at(o + 5 * kSlice), idesc(64), more); // [2;4] x 2
              mma(tmem + 384, at(o), at(o + 3 * kSlice), idesc(64), 1u);                // [zero;5] x 1
              mma(tmem + kColD, at(o + kSlice), at(o + kTileD), idesc(16), more);
              mma(tmem + kColD + 16, at(o + 3 * kSlice), at(o + kTileD), idesc(16), more);
              mma(tmem + kColD + 32, at(o + 5 * kSlice), at(o + kTileD), idesc(16), more);
            }
          }
          tc::mma_commit(&m_mma[n & 1]);
          if (st % kGroup == kGroup - 1 || st == stages - 1) tc::mma_commit(&m_sum[(groups - 1) % kBufs]);
        }
        __syncwarp();
      }
    }
    // every MMA issued here is complete before tensor memory is given back (the wait with
    // its full bound, whatever s_abort says)
    if (n > 0 && !tc::mbar_wait(&m_mma[(n - 1) & 1], ((n - 1) >> 1) & 1)) s_abort = 1;
  }
  } else if (warp < kD0) {
    // ================= converting warps
    asm volatile("setmaxnreg.inc.sync.aligned.u32 80;");
    const int xt = tid - 32 * kX0;
    // unit u of a stage: entries 4 (u & 1) .. + 3 of the 8-entry group u / 2k, member
    // (u / 2) % k -- two lanes fill the 16 bytes of an operand row.  This thread's
    // units: member, first entry (< 0: none), place in the operand buffer
    int um[kR], uq[kR], ud[kR];
#pragma unroll
    for (int r = 0; r < kR; ++r) {
      const int u = xt + r * kXThreads, ug = (u >> 1) / k;
      um[r] = (u >> 1) - ug * k;
      uq[r] = u < 16 * k ? ug * 8 + (u & 1) * 4 : -1;
      ud[r] = (ug >> 1) * kChunkBytes + (um[r] >> 3) * 256 + (ug & 1) * 128 + (um[r] & 7) * 16 +
              (u & 1) * 8;
    }
    unsigned n = 0;  // stages converted (buffer n & 1)
    for (unsigned nq = 0;; ++nq) {
      const int qb = nq % kDepth;
      wait(&m_full[qb], (nq / kDepth) & 1);
      // the solve is read once: after an expired wait the weighing warps may put -1 here
      // between two reads, and it indexes b_off
      const int s = *(volatile const int*)&s_head[qb].s;
      if (stopped() || s < 0) break;
      const int stages = s_head[qb].stages;
      const int4* const par = q_par(qb);
      const long long* const qd = q_d(qb);
      const double* const ysrc = batch ? b.b_hx + (size_t)b.b_off[s] * k : hx.yb;
      uint2 y[kR][4];
      auto load = [&](int st, int r) {
        if (uq[r] < 0) return;
        const int q0 = st * kStage + uq[r];
#pragma unroll
        for (int e = 0; e < 4; ++e)
          y[r][e] = __ldg(reinterpret_cast<const uint2*>(ysrc + (size_t)par[q0 + e].w * k + um[r]));
      };
      if (stages > 0) {
#pragma unroll
        for (int r = 0; r < kR; ++r) load(0, r);
      }
      for (int st = 0; st < stages; ++st, ++n) {
        unsigned char* const buf = smem_raw + (n & 1) * kStageBytes;
        if (n >= 2) wait(&m_mma[n & 1], ((n - 2) >> 1) & 1);
        if (stopped()) break;
#pragma unroll
        for (int r = 0; r < kR; ++r) {
          if (uq[r] < 0) continue;
          const int q0 = st * kStage + uq[r];
          uint32_t o[2][6];
#pragma unroll
          for (int e = 0; e < 2; ++e)
            digit_pairs(digits_of(y[r][2 * e].y, y[r][2 * e].x, par[q0 + 2 * e]),
                        digits_of(y[r][2 * e + 1].y, y[r][2 * e + 1].x, par[q0 + 2 * e + 1]),
                        y[r][2 * e].y, y[r][2 * e + 1].y, o[e]);
          if (st + 1 < stages) load(st + 1, r);  // in flight beside the rest of this stage
          unsigned char* const dst = buf + ud[r];
#pragma unroll
          for (int a = 0; a < 6; ++a)
            *reinterpret_cast<uint2*>(dst + L::pos(a) * kSlice) = make_uint2(o[0][a], o[1][a]);
        }
        if (warp == kD0 - 1) {
          // d~ slices: row b of the 16-row tile, two entries per lane
          const int q0 = st * kStage + 2 * lane;
          uint32_t o[6];
          const unsigned long long d0 = (unsigned long long)qd[q0], d1 = (unsigned long long)qd[q0 + 1];
          digit_pairs(d0 & ~(1ull << 63), d1 & ~(1ull << 63), (unsigned)(d0 >> 32),
                      (unsigned)(d1 >> 32), o);
          unsigned char* const dst = buf + (lane >> 3) * kChunkBytes + kTileD +
                                     ((lane >> 2) & 1) * 128 + (lane & 3) * 4;
#pragma unroll
          for (int a = 0; a < 6; ++a) *reinterpret_cast<uint32_t*>(dst + a * 16) = o[a];
          if constexpr (kThree)
#pragma unroll
            for (int a = 0; a < 4; ++a)
              *reinterpret_cast<uint32_t*>(dst + L::kTileD2 - kTileD + a * 16) = o[a];
        }
        tc::fence_proxy_async();
        __syncwarp();
        if (lane == 0) mbar_arrive(&m_conv[n & 1]);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&m_empty[qb]);
    }
  } else {
    // ================= adding warps
    const int xt = tid - 32 * kD0;
    const uint32_t lane_addr = tmem + ((uint32_t)((warp & 3) * 32) << 16);
    // this thread's accumulator row: slice of the operand and member
    const int arow = (warp & 3) * 32 + lane;
    const int blk = kThree ? arow / 40 : arow / 64;
    const int row = kThree ? arow - 40 * blk : arow - 64 * blk;
    const bool low = blk == 0;
    // columns of this warp quadruple: groups of four, from j0
    const int cw = (k + 7) / 8 * 4;
    const int j0 = (warp - kD0) / 4 * cw;
    const int ng = (cw + 3) / 4, h0 = (ng + 1) / 2;
    // the chunk's sums: per member, or (kThree) per accumulator row
    long long* const U = reinterpret_cast<long long*>(smem_raw + 2 * kStageBytes + kDepth * kQueueBytes);
    // kThree: an off-diagonal pair counts twice, weight 2^(90 - 9 (a + b)) in units
    // of 2^(45 + kDrop); slice blk against slices 0 (times 2^32), 1, 2, 3 as
    // integers, and against 0, 2, 3, 4, 5 as the FP32 part.  33 shares its sum with 20,
    // which 02 takes off again: (U + U^T) sees 20 and 02 alike.
    //   0   00 2^35, 01 2^27, 02 2^18 - 2^-19, 03 2^9, 04 1, 05 2^-9
    //   1   11 2^17, 12 2^9, 13 1, 14 2^-9, 15 2^-18
    //   2   20+33 2^-19, 22 2^-1, 23 2^-9, 24 2^-18
    const int c00 = blk == 0 ? 8 : 0, h1 = blk == 0 ? 1 << 27 : blk == 1 ? 1 << 17 : 0;
    const int h2 = blk == 0 ? 1 << 18 : blk == 1 ? 1 << 9 : 0;
    const int h3 = blk == 0 ? 1 << 9 : 0;
    const float f0 = blk == 2 ? 0x1p-19f : 0.0f, f2 = blk == 0 ? -0x1p-19f : blk == 1 ? 0.0f : 0.5f;
    const float f3 = blk == 0 ? 0.0f : blk == 1 ? 1.0f : 0x1p-9f;
    const float f4 = blk == 0 ? 1.0f : blk == 1 ? 0x1p-9f : 0x1p-18f;
    const float f5 = blk == 0 ? 0x1p-9f : blk == 1 ? 0x1p-18f : 0.0f;
    // kDThreads elements further on in rows of k + 1
    const int step_a = kDThreads / (k + 1), step_c = kDThreads - step_a * (k + 1);
    unsigned groups = 0;  // exact sums taken out
    for (unsigned nq = 0;; ++nq) {
      const int qb = nq % kDepth;
      wait(&m_full[qb], (nq / kDepth) & 1);
      const QueueHead h = s_head[qb];
      __syncwarp();
      if (lane == 0) mbar_arrive(&m_empty[qb]);
      bar_sync(kBarD, kDThreads);  // the chunk before is written
      if (xt == 0) s_stop[1] = s_abort;
      bar_sync(kBarD, kDThreads);
      if (s_stop[1] || h.s < 0) break;
      double* const C = Cout + (size_t)h.s * k * k;
      double* const tv = tout + (size_t)h.s * k;
      long long thi = 0, tlo = 0;
      // four columns of the exact FP32 sums as one integer each, written or added to
      // U.  The products worth a unit or less (below 2^-50 of the largest product)
      // come together in FP32 first: 24 bits of at most 2^24 units.
      auto columns3 = [&](int g4, bool add) {
        const uint32_t at = lane_addr + (groups & 1) * 256 + 8u + (uint32_t)(j0 + 4 * g4);
        float v[6][4];  // against slices 3 4 5 0 1 2
#pragma unroll
        for (int m = 0; m < 6; ++m) tmem_ld4(at + 40u * m, v[m]);
        tmem_wait_ld();
        long long* const u = U + arow * kUStride + j0 + 4 * g4;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const float f = fmaf(f0, v[3][c], fmaf(f5, v[2][c], fmaf(f4, v[1][c],
                          fmaf(f3, v[0][c], f2 * v[5][c]))));
          long long A = add && arow < 120 ? u[c] : 0;
          A += __float2int_rn(f);
          if ((warp & 3) < 3) {  // the last warp's rows are all slice 2
            A += (long long)__float2int_rn(v[4][c]) * h1;
            A += (long long)__float2int_rn(v[5][c]) * h2;
          }
          if ((warp & 3) < 2) {
            A += (long long)__float2int_rn(v[0][c]) * h3;
            A += (long long)((unsigned long long)(unsigned)(__float2int_rn(v[3][c]) * c00) << 32);
          }
          if (arow < 120) u[c] = A;
        }
      };
      auto columns = [&](int g4, bool add) {
        const int j = j0 + 4 * g4;
        float v[7][4];
#pragma unroll
        for (int m = 0; m < 7; ++m) tmem_ld4(lane_addr + 64u * m + (uint32_t)j, v[m]);
        tmem_wait_ld();
        long long* const u = U + row * kUStride + j;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          // an off-diagonal pair counts twice (C = (U + U^T) / 2); weight
          // 2^(90 - 9 (a + b)) in units of 2^(45 + kDrop)
          long long A = add ? u[c] : 0;
          if (low) {  // 50 01 03 02 04 33 22
            A += (long long)__float2int_rn(v[1][c]) * (1 << 27);
            A += (long long)__float2int_rn(v[3][c]) * (1 << 18);
            A += (long long)__float2int_rn(v[2][c]) * (1 << 9);
            A += __float2int_rn(
                fmaf(0x1p-19f, v[5][c], fmaf(0x1p-9f, v[0][c], fmaf(0.5f, v[6][c], v[4][c]))));
          } else {    // 00 11 13 12 14 23 42+51
            A += (long long)((unsigned long long)(unsigned)(__float2int_rn(v[0][c]) * 8) << 32);
            A += (long long)__float2int_rn(v[1][c]) * (1 << 17);
            A += (long long)__float2int_rn(v[3][c]) * (1 << 9);
            A += __float2int_rn(
                fmaf(0x1p-18f, v[6][c], fmaf(0x1p-9f, v[4][c], fmaf(0x1p-9f, v[5][c], v[2][c]))));
          }
          u[c] = A;
        }
      };
      for (int st = 0; st < h.stages; st += kGroup, ++groups) {
        wait(&m_sum[groups % kBufs], (groups / kBufs) & 1);
        tc::fence_after();
        if constexpr (kThree) {
          for (int q = 0; q < ng; ++q) columns3(q, st > 0);
          if (j0 == 0) {
            const uint32_t at = lane_addr + (groups & 1) * 256;
            float v[8], z[4];
            tmem_ld8(at + 248u, v);
            tmem_ld4(at, z);
            tmem_wait_ld();
            long long x[6], y[4];  // slice blk, and blk + 3, against d~ slices 0..
#pragma unroll
            for (int j = 0; j < 6; ++j) x[j] = __float2int_rn(v[j]);
#pragma unroll
            for (int j = 0; j < 4; ++j) y[j] = __float2int_rn(z[j]);
            long long w6;
            if (blk == 0) {
              thi += (x[0] << 18) + (x[1] << 9) + x[2];
              tlo += (x[3] << 18) + (x[4] << 9) + x[5] + (y[0] << 18) + (y[1] << 9) + y[2];
              w6 = y[3];
            } else if (blk == 1) {
              thi += (x[0] << 9) + x[1];
              tlo += (x[2] << 18) + (x[3] << 9) + x[4] + (y[0] << 9) + y[1];
              w6 = x[5] + y[2];
            } else {
              thi += x[0];
              tlo += (x[1] << 18) + (x[2] << 9) + x[3] + y[0];
              w6 = x[4] + y[1];
            }
            tlo += (w6 + 256) >> 9;
          }
          tc::fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&m_drain[groups & 1]);
        } else {
          // The two halves' sums meet in U: one half takes the first columns while the
          // other takes the rest, then they change over
          const bool fresh = st == 0;
          for (int q = low ? 0 : h0; q < (low ? h0 : ng); ++q) columns(q, !fresh);
          if (j0 == 0) {
            float v[3][8];
#pragma unroll
            for (int m = 0; m < 3; ++m) tmem_ld8(lane_addr + kColD + 16u * m, v[m]);
            tmem_wait_ld();
            long long x[3][6];
#pragma unroll
            for (int m = 0; m < 3; ++m)
#pragma unroll
              for (int j = 0; j < 6; ++j) x[m][j] = __float2int_rn(v[m][j]);
            // rows 5|0, 1|3, 2|4 of z against d~ slices 0..5, a + b <= 6; thi in
            // units of weight 2, tlo of weight 5
            long long w6;
            if (low) {
              thi += (x[1][0] << 9) + x[1][1] + x[2][0];
              tlo += (x[1][2] << 18) + (x[1][3] << 9) + x[1][4] + (x[2][1] << 18) + (x[2][2] << 9) +
                     x[2][3] + x[0][0];
              w6 = x[0][1] + x[1][5] + x[2][4];
            } else {
              thi += (x[0][0] << 18) + (x[0][1] << 9) + x[0][2];
              tlo += (x[0][3] << 18) + (x[0][4] << 9) + x[0][5] + (x[1][0] << 18) + (x[1][1] << 9) +
                     x[1][2] + (x[2][0] << 9) + x[2][1];
              w6 = x[1][3] + x[2][2];
            }
            tlo += (w6 + 256) >> 9;
          }
          bar_sync(kBarD, kDThreads);
          for (int q = low ? h0 : 0; q < (low ? ng : h0); ++q) columns(q, true);
          tc::fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&m_drain[0]);
          if (st + kGroup < h.stages) bar_sync(kBarD, kDThreads);  // U's columns change hands again
        }
      }
      if (h.bad) {
        // (an earlier chunk's C is written: the barrier at the top)
        if (xt == 0) C[0] = __longlong_as_double((long long)kGramMark);
        continue;
      }
      if (h.stages == 0 && !h.first) continue;
      if (j0 == 0 && arow < (kThree ? 120 : 128)) s_t[blk][row] = make_longlong2(thi, tlo);
      bar_sync(kBarD, kDThreads);
      const int ex2 = 2 * h.S - 62 + kDrop, ext = h.S + h.Sd - 61;
      // C = (U + U^T) / 2 out, the lower triangle in rows (rows i and k - 1 - i of it
      // share one row of k + 1 elements), four elements' loads in flight; t by the
      // threads with the fewest elements
      const int total = (k + 1) / 2 * (k + 1);
      int a = xt / (k + 1), c = xt - a * (k + 1);
      for (int r0 = xt; r0 < total; r0 += 4 * kDThreads) {
        int ci[4], cj[4];
        long long u[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const int i = c <= a ? a : k - 1 - a, j = c <= a ? c : c - a - 1;
          // odd k: the middle row meets itself
          const bool mine = r0 + e * kDThreads < total && !(2 * a == k - 1 && c > a);
          ci[e] = mine ? i : -1;
          cj[e] = j;
          u[e] = 0;
          if (mine && h.stages > 0) {
            const int at = i * kUStride + j, ta = j * kUStride + i;
            u[e] = U[at] + U[ta];
            if constexpr (kThree)
              u[e] += U[at + 40 * kUStride] + U[ta + 40 * kUStride] + U[at + 80 * kUStride] +
                      U[ta + 80 * kUStride];
          }
          a += step_a;
          c += step_c;
          if (c > k) {
            c -= k + 1;
            ++a;
          }
        }
#pragma unroll
        for (int e = 0; e < 4; ++e)
          if (ci[e] >= 0) {
            double v = fixed_to_double(u[e], ex2);
            if (!h.first) v += C[ci[e] * k + cj[e]];
            C[ci[e] * k + cj[e]] = v;
            if (!lower) C[cj[e] * k + ci[e]] = v;
          }
      }
      if (kDThreads - 1 - xt < k) {
        const int i = kDThreads - 1 - xt;
        double v = 0.0;
        if (h.stages > 0) {
          long long hi = s_t[0][i].x + s_t[1][i].x, lo = s_t[0][i].y + s_t[1][i].y;
          if constexpr (kThree) {
            hi += s_t[2][i].x;
            lo += s_t[2][i].y;
          }
          v = wide_to_double(hi, lo, ext);
        }
        tv[i] = h.first ? v : tv[i] + v;
      }
    }
  }
  tc::fence_before();
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem),
                 "r"(kTmemCols));
  if (tid == 0 && s_abort) atomicExch(err, LG_ERR_TIMEOUT);
}

bool gram64_tc_supported(int ens) { return ens <= 64; }

void launch_gram64_tc(const Geometry& g, const HxDev& hx, const ListDev& l, const SolveBatch& b,
                      const double* axb, bool lower, double* C, double* t, int* err,
                      cudaStream_t stream) {
  if (b.nsolves == 0) return;
  const int grid = b.nsolves < 152 ? b.nsolves : 152;
  if (b.mode == 0 && g.vert_dist > 0.0)
    level_lnp_kernel<<<(b.nsolves + 127) / 128, 128, 0, stream>>>(g, b, axb, t);
  auto run = [&](auto kernel, int smem) {
    allow_smem(kernel, smem);
    kernel<<<grid, g64::kThreads, smem, stream>>>(g, hx, l, b, lower ? 1 : 0,
                                                  (long long)g.tc_wait_ns, C, t, err);
  };
  const bool limited = g.tc_wait_ns > 0;
  if (g.ens <= 40)
    run(limited ? gram64_tc_kernel<2, true, true> : gram64_tc_kernel<2, true, false>,
        g64::Layout<true>::kSmem);
  else if (g.ens <= 48)
    run(limited ? gram64_tc_kernel<2, false, true> : gram64_tc_kernel<2, false, false>,
        g64::Layout<false>::kSmem);
  else
    run(limited ? gram64_tc_kernel<3, false, true> : gram64_tc_kernel<3, false, false>,
        g64::Layout<false>::kSmem);
}

}  // namespace lg
