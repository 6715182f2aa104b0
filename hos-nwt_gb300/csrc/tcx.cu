// Transform passes on the tensor cores (sm_103a).
//
// A REDFT00 / RODFT00 pass over many lines (fourier_FFTW.f90:130-229) is a
// product of the lines with a cosine or sine matrix.  GB300 runs FP64 at 2
// operations per clock per SM and its FFT in double-float at the FP32 issue
// rate, but BF16 products at 4096 per clock per SM: so the pass is done as an
// exact product of digits (the splitting of Ozaki, Ogita, Oishi and Rump,
// 2012).  Every line is scaled by a power of two and cut into six BF16 digits,
// and so is the matrix, whose entries are known in advance:
//
//   x / 2^(E-8) = d_0 + d_1 2^-9 + d_2 2^-18 + d_3 2^-27 + d_4 + d_5
//
// with whole numbers |d_i| <= 256 for i < 4, and d_4, d_5 the remainder
// (below 2^-28) as two BF16 numbers.  The products d_i w_j are summed by
// tcgen05.mma into FP32 accumulators in tensor memory, one per level i + j =
// 0, 1, 2, 3, and one for the levels 4 and 5.  A sum of level 0 to 3 is a whole
// number below 2^24 units over 128 (levels 0, 1) or 64 terms (2, 3), so every
// addition is exact; then it is added to a 64-bit fixed-point sum (34
// fractional bits), which is exact too.  In the fifth accumulator the FP32 rounding is 2^-24 of
// products below 2^-36 of the largest: all that a result owes to the order and
// the split of the work.  What is left out (level 6 and the
// remainders of the sixth digits) is 2^-54 of the largest product per term.
//
// Half of the work is saved by one fold per pass:
//   form F (every output wanted): outputs k and D - k from the sums over even
//     and odd inputs, E(k) + O(k) and +-(E(k) - O(k));
//   form T (every input given, truncated outputs): even and odd outputs from
//     u_j + u_{D-j} and u_j - u_{D-j}.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <type_traits>
#include <vector>

#include "hosnwt_internal.h"

namespace hos {
namespace {

constexpr int kS = 6;             // digits
constexpr int kBM = 128;          // lines per tile (the accumulator's lanes)
constexpr int kBN = 96;           // outputs per tile and parity: five accumulators of 96 columns
                                  // fill 480 of the 512 columns of tensor memory
constexpr int kBK = 32;           // terms per stage (a 64-byte swizzle row)
constexpr int kStages = 2;
constexpr int kDrainHi = 4;       // stages between two drains of levels 0, 1: 2 x 128 x 2^16 = 2^24
constexpr int kDrainLo = 2;       // and of levels 2, 3: 4 x 64 x 2^16 = 2^24
constexpr int kFrac = 34;         // fractional bits of the fixed-point sums
// Roles: warps 0-7 drain the accumulators (two per 32 lanes, 48 columns
// each), 8-11 turn finished sums into outputs (one per 32 lines), 12 loads, 13
// issues the products; 14 and 15 complete the warpgroup.
constexpr int kDrainWarps = 8, kOutWarps = 4, kLoadWarp = 12, kMmaWarp = 13;
constexpr int kColsPerWarp = kBN / 2;
constexpr int kThreads = 512;
constexpr int kOutCols = 8;       // sums per line that an output warp has in flight
constexpr int kBufs = 3;          // sums of a parity handed to the output warps: two read, one written
constexpr int kABytes = kS * kBM * kBK * 2;
constexpr int kBBytes = kS * kBN * kBK * 2;
constexpr int kStageBytes = kABytes + kBBytes;
constexpr int kStageRow = kOutCols + 1;
constexpr size_t kOutBytes = (size_t)kOutWarps * 2 * 32 * kStageRow * sizeof(double);
constexpr size_t kPassSmem = 1024 + (size_t)kStages * kStageBytes + kOutBytes;
constexpr unsigned kWaitLimit = 1u << 22;
constexpr int kNonFinite = 0x7fffffff;  // row exponent of a line with an infinity or a NaN
constexpr long long kSums = (long long)kBM * kBN;  // sums of one parity of a tile
constexpr int kUnitsPerSm = 6;                     // sums kept per SM when the tiles are split

struct TcJob {
  double* out;
  long long out_sk, out_sl;
  int row0;                     // first line among the group's
  unsigned* cmax;               // x passes: largest high word of output k over the lines
};

struct TcGroup {
  CUtensorMap a, b;
  int rows, nkb, nout_p;        // lines; stages per parity; outputs per parity
  int tm, tn, tile0;            // tiles along lines and outputs, first tile
  int unit0, nseg, segk;        // first unit; segments per parity, stages per segment
  int form, sin_kind, D, ew;
  int job0, njobs;
  int nout, klo, khi;
  int xpass;                    // outputs of a line are contiguous
  double r0, rD;                // output scales at k = 0 and k = D over the interior's
  const int* rowexp;
};

template <int NJ>
struct TcBatchT {
  TcGroup grp[NJ];
  TcJob job[NJ];
  int ngroups, nunits;
  // A unit of work is a tile with all its terms (split = 0: kBufs buffers of
  // sums per CTA), or one segment of one parity of a tile (split = 1: a buffer
  // per unit; k_tc_finish adds them up and writes the outputs).
  int split;
  long long* sums;              // [buffer][output][line]
  unsigned* failed;             // set when a wait ran out: k_tc_finish writes NaN
  unsigned* expired;            // the same for the host (page-locked host memory)
};
using TcBatch = TcBatchT<kMaxJobs>;

struct DgJob {
  const double* in;
  long long in_sk, in_sl;
  const double* win;
  long long win_sk, win_sl;
  int nlines, jlo, jend;
  int D, form, sin_kind, kp;
  int half0, halfD;             // 1: the end input counts half
  int rows, row0;               // lines of the group, first row of this job
  __nv_bfloat16* a;             // the group's digits [parity][digit][row][kp]
  int* rowexp;
  int nsplit, cps;              // y passes: CTAs per 32 lines, chunks of 64 terms per CTA
  const unsigned* lmax;         // y passes: largest high word of each line, where known
  unsigned* cmax;               // x passes: the outputs' maxima to clear, ncmax of them
  int ncmax;
};

template <int NJ>
struct DgBatchT {
  DgJob job[NJ];
  int start[NJ + 1];
  int njobs;
  int wpl;                      // x passes: warps per line (1 or 8)
};
using DgBatch = DgBatchT<kMaxJobs>;

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, unsigned parity) {
  const unsigned a = smem_u32(bar);
  for (unsigned it = 0; it < kWaitLimit; ++it) {
    unsigned done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}
__device__ __forceinline__ void tma_load_4d(unsigned dst, const CUtensorMap* map, int x, int y, int z, int w,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], "
      "[%6];" ::"r"(dst),
      "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(smem_u32(bar))
      : "memory");
}
// K-major tile of 64-byte rows with the 64-byte swizzle: 8-row groups 512
// bytes apart, descriptor version 1, layout type 4
__device__ __forceinline__ uint64_t sw64_desc(unsigned saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)1 << 16) | ((uint64_t)(512 >> 4) << 32) |
         ((uint64_t)1 << 46) | ((uint64_t)4 << 61);
}
// FP32 accumulator, BF16 operands, both K-major, M = 128
constexpr uint32_t idesc_of(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(kBM >> 4) << 24);
}
constexpr uint32_t kIdesc = idesc_of(kBN), kIdescWide = idesc_of(2 * kBN);

// Issued by the elected lane of a converged warp: the branch stays inside
// the instruction, so that the descriptors live in uniform registers.
__device__ __forceinline__ void mma_bf16(uint32_t tmem_d, uint64_t a, uint64_t b, uint32_t idesc, int accumulate,
                                         uint32_t elected) {
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "setp.ne.b32 q, %5, 0;\n\t"
      "@q tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate), "r"(elected)
      : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar, uint32_t elected) {
  asm volatile(
      "{\n\t.reg .pred q;\n\t"
      "setp.ne.b32 q, %1, 0;\n\t"
      "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n\t}" ::"r"(smem_u32(bar)),
      "r"(elected)
      : "memory");
}
__device__ __forceinline__ uint32_t elect_one() {
  uint32_t e;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "elect.sync _|p, 0xffffffff;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(e));
  return e;
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* r) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// ---------------------------------------------------------------- digits

// The digits of q / 2^62, |q| <= 2^62, as floats in true scale (units of
// 2^54): whole numbers times 2^-9i, then the remainder, not yet rounded (host
// form, for the matrices).
void split_digits(long long q, float* d) {
  const long long d0 = (q + (1LL << 53)) >> 54;
  q -= d0 << 54;
  const long long d1 = (q + (1LL << 44)) >> 45;
  q -= d1 << 45;
  const long long d2 = (q + (1LL << 35)) >> 36;
  q -= d2 << 36;
  const long long d3 = (q + (1LL << 26)) >> 27;
  q -= d3 << 27;
  d[0] = (float)d0;
  d[1] = (float)d1 * 0x1p-9f;
  d[2] = (float)d2 * 0x1p-18f;
  d[3] = (float)d3 * 0x1p-27f;
  d[4] = (float)q * 0x1p-54f;
}

// The same of a double, |x| < 2^(emax - 1022), in 32-bit integer operations:
// the digits lie on the high word, whose additions never carry from the low.
// A digit becomes a float by the bits of 1.5 2^23 + d (conversions run at an
// eighth of that rate).
__device__ __forceinline__ void split_double(double x, int emax, float* d) {
  const unsigned bh = (unsigned)__double2hiint(x), bl = (unsigned)__double2loint(x);
  const int e = (int)((bh >> 20) & 0x7ff);
  const unsigned mh = (bh & 0xfffffu) | (e ? 0x100000u : 0u);
  // mantissa << 9, shifted right to the common exponent
  const int sh = emax - (e ? e : 1);
  unsigned h = __funnelshift_l(bl, mh, 9), l = bl << 9;
  if (sh >= 32) {
    l = h;
    h = 0;
  }
  l = sh < 64 ? __funnelshift_r(l, h, sh & 31) : 0u;
  h = sh < 64 ? h >> (sh & 31) : 0u;
  const unsigned neg = (unsigned)((int)bh >> 31);
  l = (l ^ neg) - neg;
  h = (h ^ neg) + ((neg && l == 0u) ? 1u : 0u);
  int q = (int)h;
  const int d0 = (q + (1 << 21)) >> 22;
  q -= d0 << 22;
  const int d1 = (q + (1 << 12)) >> 13;
  q -= d1 << 13;
  const int d2 = (q + (1 << 3)) >> 4;
  q -= d2 << 4;
  const unsigned lr = l + (1u << 26);
  const int d3 = (int)__funnelshift_r(lr, (unsigned)q + (lr < l ? 1u : 0u), 27);
  const int r = (int)(l - ((unsigned)d3 << 27));
  d[0] = __int_as_float(0x4b400000 + d0) - 12582912.0f;
  d[1] = fmaf(__int_as_float(0x4b400000 + d1), 0x1p-9f, -12582912.0f * 0x1p-9f);
  d[2] = fmaf(__int_as_float(0x4b400000 + d2), 0x1p-18f, -12582912.0f * 0x1p-18f);
  d[3] = fmaf(__int_as_float(0x4b400000 + d3), 0x1p-27f, -12582912.0f * 0x1p-27f);
  d[4] = (float)r * 0x1p-54f;
}

// x / 2 by its exponent (an FP64 product takes 64 issue cycles of a warp, also
// where no lane needs it); numbers below 2^-1021 become zero
__device__ __forceinline__ double half_of(double x) {
  const int h = __double2hiint(x), e = (h >> 20) & 0x7ff;
  const int nh = e == 0x7ff ? h : (e >= 2 ? h - 0x100000 : h & (int)0x80000000);
  return __hiloint2double(nh, e >= 2 || e == 0x7ff ? __double2loint(x) : 0);
}

// The terms t = 2 i, 2 i + 1 of both parities of one line: v[parity][0..1].
// u(j) is the weighted input.
template <typename U>
__device__ __forceinline__ void fold_terms(const DgJob& J, int i, U&& u, double v[2][2]) {
  if (J.form == 0) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int p = 0; p < 2; ++p) v[p][h] = u(4 * i + 2 * h + p);
  } else {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int j = 2 * i + h, m = J.D - j;
      double s = 0.0, r = 0.0;
      if (j < m) {
        const double a = u(j), b = u(m);
        s = a + b;
        r = a - b;
      } else if (j == m) {
        // the middle input stands alone: cos sees it in the even outputs,
        // sin in the odd ones
        s = u(j);
      }
      v[0][h] = J.sin_kind ? r : s;
      v[1][h] = J.sin_kind ? s : r;
    }
  }
}

__device__ __forceinline__ unsigned high_abs(double x) {
  return (unsigned)(__double2hiint(x)) & 0x7fffffffu;
}

// packed BF16 digits of the two terms: out[0..5]
__device__ __forceinline__ void pack_digits(const double* v, int emax, unsigned* out) {
  float a[5], b[5];
  split_double(v[0], emax, a);
  split_double(v[1], emax, b);
#pragma unroll
  for (int s = 0; s < 5; ++s) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a[s], b[s]);
    memcpy(&out[s], &h, 4);
    if (s == 4) {
      const __nv_bfloat162 g =
          __floats2bfloat162_rn(a[4] - __bfloat162float(h.x), b[4] - __bfloat162float(h.y));
      memcpy(&out[5], &g, 4);
    }
  }
}

__device__ __forceinline__ int row_exponent(unsigned mx) {
  const int e = (int)(mx >> 20);
  return e == 0x7ff ? kNonFinite : (e ? e : 1);
}

constexpr int kDgThreads = 256;
constexpr int kDgItems = 5;  // pairs of terms per thread and parity in registers: lines up to 2560 terms a parity

// x passes (points contiguous): wpl warps per line; the line's largest
// exponent first, then the digits.
template <int NJ>
__global__ void __launch_bounds__(kDgThreads) k_tc_digits_x(const __grid_constant__ DgBatchT<NJ> b) {
  __shared__ unsigned wmax[kDgThreads / 32];
  int jb = 0;
  while (jb + 1 < b.njobs && (int)blockIdx.x >= b.start[jb + 1]) ++jb;
  const DgJob& J = b.job[jb];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int wpl = b.wpl, lpc = (kDgThreads / 32) / wpl;
  const int line = ((int)blockIdx.x - b.start[jb]) * lpc + warp / wpl;
  const int i0 = (wpl == 1) ? lane : (int)threadIdx.x, step = 32 * wpl;
  pdl_wait();
  const bool valid = line < J.nlines;
  const double* __restrict__ x = J.in + (long long)(valid ? line : 0) * J.in_sl;
  const double* __restrict__ w = J.win ? J.win + (long long)(valid ? line : 0) * J.win_sl : nullptr;
  auto u = [&](int j) -> double {
    if (j < J.jlo || j >= J.jend) return 0.0;
    double v = __ldg(x + j);
    if (w) v *= __ldg(w + (long long)j * J.win_sk);
    if ((j == 0 && J.half0) || (j == J.D && J.halfD)) v = half_of(v);
    return v;
  };
  if (J.cmax) {
    const int nb = b.start[jb + 1] - b.start[jb];
    for (int k = ((int)blockIdx.x - b.start[jb]) * kDgThreads + threadIdx.x; k < J.ncmax; k += nb * kDgThreads) J.cmax[k] = 0;
  }
  const int ni = valid ? J.kp / 2 : 0;
  // a thread keeps its terms in registers between the two steps
  double v[kDgItems][2][2];
  unsigned mx = 0;
#pragma unroll
  for (int m = 0; m < kDgItems; ++m) {
    const int i = i0 + m * step;
    if (i < ni) {
      fold_terms(J, i, u, v[m]);
    } else {
      v[m][0][0] = v[m][0][1] = v[m][1][0] = v[m][1][1] = 0.0;
    }
    mx = max(mx, max(max(high_abs(v[m][0][0]), high_abs(v[m][0][1])), max(high_abs(v[m][1][0]), high_abs(v[m][1][1]))));
  }
  for (int i = i0 + kDgItems * step; i < ni; i += step) {  // longer lines: read twice
    double t[2][2];
    fold_terms(J, i, u, t);
    mx = max(mx, max(max(high_abs(t[0][0]), high_abs(t[0][1])), max(high_abs(t[1][0]), high_abs(t[1][1]))));
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  if (wpl > 1) {
    if (lane == 0) wmax[warp] = mx;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kDgThreads / 32; ++k) mx = max(mx, wmax[k]);
  }
  if (!valid) return;
  const int emax = row_exponent(mx);
  const int row = J.row0 + line;
  if (i0 == 0) J.rowexp[row] = emax == kNonFinite ? kNonFinite : emax - 1022 - 16 - kFrac;
  const long long ds = (long long)J.rows * J.kp / 2;  // between digits, in pairs
  unsigned* a = reinterpret_cast<unsigned*>(J.a + (long long)row * J.kp);
  auto put = [&](int i, const double t[2][2]) {
#pragma unroll
    for (int p = 0; p < 2; ++p) {
      unsigned o[kS] = {};
      if (emax != kNonFinite) pack_digits(t[p], emax, o);
#pragma unroll
      for (int s = 0; s < kS; ++s) a[(p * kS + s) * ds + i] = o[s];
    }
  };
#pragma unroll
  for (int m = 0; m < kDgItems; ++m)
    if (i0 + m * step < ni) put(i0 + m * step, v[m]);
#pragma unroll 1
  for (int i = i0 + kDgItems * step; i < ni; i += step) {
    double t[2][2];
    fold_terms(J, i, u, t);
    put(i, t);
  }
}

// y passes (lines contiguous, points strided): a CTA takes 32 lines, lane =
// line; the digits of 64 terms go through shared memory so that they leave
// as 128-byte rows.  nsplit CTAs share the terms of the same lines (each
// finds their exponents anew) when the lines alone would not fill the GPU.
constexpr size_t kDgySmem = (size_t)2 * kS * 32 * 32 * 4 + (kDgThreads / 32) * 32 * 4;
template <int NJ>
__global__ void __launch_bounds__(kDgThreads) k_tc_digits_y(const __grid_constant__ DgBatchT<NJ> b) {
  extern __shared__ __align__(16) unsigned dsm[];
  unsigned* wmax = dsm + 2 * kS * 32 * 32;
  int jb = 0;
  while (jb + 1 < b.njobs && (int)blockIdx.x >= b.start[jb + 1]) ++jb;
  const DgJob& J = b.job[jb];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int lb = (int)blockIdx.x - b.start[jb];
  const int split = lb % J.nsplit, line0 = (lb / J.nsplit) * 32;
  const int line = line0 + lane;
  pdl_wait();
  const bool valid = line < J.nlines;
  const double* __restrict__ x = J.in + (valid ? line : 0);
  const double* __restrict__ w = J.win ? J.win + (long long)(valid ? line : 0) * J.win_sl : nullptr;
  auto u = [&](int j) -> double {
    if (!valid || j < J.jlo || j >= J.jend) return 0.0;
    double v = __ldg(x + (long long)j * J.in_sk);
    if (w) v *= __ldg(w + (long long)j * J.win_sk);
    if ((j == 0 && J.half0) || (j == J.D && J.halfD)) v = half_of(v);
    return v;
  };
  const int ni = J.kp / 2;
  unsigned mx = 0;
  if (J.lmax) {
    // maxima left by the x pass; a sum or difference of two is below twice it
    mx = valid ? __ldcg(J.lmax + line) : 0;
  } else {
#pragma unroll 4
    for (int i = warp; i < ni; i += kDgThreads / 32) {
      double v[2][2];
      fold_terms(J, i, u, v);
      mx = max(mx, max(max(high_abs(v[0][0]), high_abs(v[0][1])), max(high_abs(v[1][0]), high_abs(v[1][1]))));
    }
    wmax[warp * 32 + lane] = mx;
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kDgThreads / 32; ++k) mx = max(mx, wmax[k * 32 + lane]);
  }
  int emax = row_exponent(mx);
  if (J.lmax && J.form == 1 && emax != kNonFinite) ++emax;
  if (split == 0 && warp == 0 && valid)
    J.rowexp[J.row0 + line] = emax == kNonFinite ? kNonFinite : emax - 1022 - 16 - kFrac;
  const int nch = (J.kp + 63) / 64;
  const int c1 = min(nch, (split + 1) * J.cps);
  for (int c = split * J.cps; c < c1; ++c) {
    // all loads of the warp's four pairs of terms first
    double v[4][2][2];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int i = c * 32 + warp + m * (kDgThreads / 32);
      if (i < ni) {
        fold_terms(J, i, u, v[m]);
      } else {
        v[m][0][0] = v[m][0][1] = v[m][1][0] = v[m][1][1] = 0.0;
      }
    }
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      const int q = warp + m * (kDgThreads / 32);
      const int word = lane * 32 + (((q >> 2) ^ (lane & 7)) << 2) + (q & 3);
#pragma unroll
      for (int p = 0; p < 2; ++p) {
        unsigned o[kS] = {};
        if (emax != kNonFinite) pack_digits(v[m][p], emax, o);
#pragma unroll
        for (int s = 0; s < kS; ++s) dsm[(p * kS + s) * 1024 + word] = o[s];
      }
    }
    __syncthreads();
    const int nl = min(32, J.nlines - line0);
    for (int t = threadIdx.x; t < 2 * kS * 32 * 8; t += kDgThreads) {
      const int ps = t >> 8, r = (t >> 3) & 31, q = t & 7;
      const int k = c * 64 + q * 8;
      if (r < nl && k < J.kp) {
        const uint4 d = *reinterpret_cast<const uint4*>(dsm + ps * 1024 + r * 32 + ((q ^ (r & 7)) << 2));
        *reinterpret_cast<uint4*>(J.a + ((long long)ps * J.rows + J.row0 + line0 + r) * J.kp + k) = d;
      }
    }
    __syncthreads();
  }
}

// ---------------------------------------------------------------- the product

// The 21 pairs (i, j) of digits.  Twelve are issued two at a time: digits j and
// j + 1 of the matrix are neighbours in shared memory and the accumulators of
// levels i + j and i + j + 1 neighbours in tensor memory, so one instruction of
// 192 columns takes digit i of the lines against both and reads it once.  The
// other nine go to accumulator 4, the smallest first.  What bounds the products
// is the tensor cores' sustained rate: 2850 cycles per stage are 1.8 PFLOP/s in
// BF16 (1.2 kW at 2070 MHz), with 21 narrow products 2900; a time step of 2052 x
// 1028 modes at order 9, 193.7 -> 190.2 ms.
constexpr int kNarrow = 9, kWide = 6;
__device__ constexpr signed char kNarrowI[kNarrow] = {0, 5, 1, 4, 2, 3, 0, 4, 2};
__device__ constexpr signed char kNarrowJ[kNarrow] = {5, 0, 4, 1, 3, 2, 4, 0, 2};
__device__ constexpr signed char kWideI[kWide] = {0, 0, 1, 2, 1, 3};
__device__ constexpr signed char kWideJ[kWide] = {0, 2, 0, 0, 2, 0};

// a 2^e, rounded to nearest, by integer arithmetic: conversions and products
// in FP64 cost 64 issue cycles of a warp each.  -1000 < e < 900
__device__ __forceinline__ double fixed_to_double(long long a, int e) {
  const unsigned long long u = (unsigned long long)(a < 0 ? -a : a);
  const int lz = __clzll((long long)u);
  const unsigned long long v = u << (lz & 63);
  const unsigned long long m = (v >> 11) + ((v >> 10) & 1ULL);  // 2^52 <= m <= 2^53
  const unsigned hi = (unsigned)(m >> 32) + ((unsigned)(1022 + 63 - lz + e) << 20);
  const unsigned sign = (unsigned)(a >> 63) & 0x80000000u;
  return u ? __hiloint2double((int)(hi | sign), (int)(unsigned)m) : 0.0;
}
// What unit u of a batch covers.
struct Unit {
  const TcGroup* g;
  int tile, m0, n0, po;   // tile of the batch; first line, output; parity of a form T tile
  int p0, np, k0, k1;     // parities and stages
  int first;              // split: first unit of the tile
};
template <int NJ>
__device__ __forceinline__ Unit unit_of(const TcBatchT<NJ>& b, int u) {
  int g = 0;
  while (g + 1 < b.ngroups && u >= b.grp[g + 1].unit0) ++g;
  const TcGroup& G = b.grp[g];
  Unit w;
  w.g = &G;
  const int lu = u - G.unit0, both = G.form == 0 ? 2 : 1;
  int lt = lu;
  w.p0 = 0;
  w.np = both;
  w.k0 = 0;
  w.k1 = G.nkb;
  w.first = u;
  if (b.split) {
    const int per = both * G.nseg;
    lt = lu / per;
    const int r = lu - lt * per;
    w.p0 = r / G.nseg;
    w.np = 1;
    w.k0 = (r - w.p0 * G.nseg) * G.segk;
    w.k1 = min(w.k0 + G.segk, G.nkb);
    w.first = u - r;
  }
  w.tile = G.tile0 + lt;
  w.m0 = (lt % G.tm) * kBM;
  const int rest = lt / G.tm;
  w.n0 = (rest % G.tn) * kBN;
  w.po = rest / G.tn;
  if (G.form != 0) w.p0 = w.po;
  return w;
}

// One warp turns the sums of 32 lines (quad) of a tile, outputs c of the
// tile in [c_begin, c_end), into outputs: parities combined, scaled, stored.
// even and odd point at the sums of the lane's line, nseg buffers each.
// stage: 64 rows of kStageRow doubles for the warp (x passes).
template <int NJ>
__device__ __forceinline__ void put_outputs(const TcBatchT<NJ>& b, const Unit& w, int quad, int lane,
                                            const long long* even, const long long* odd, int nseg, double* stage,
                                            bool ok, int c_begin, int c_end) {
  const TcGroup& G = *w.g;
  const int n0 = w.n0, po = w.po;
  // copies of the tile's parameters: loads through the references would be
  // repeated after every store
  const int form = G.form, D = G.D, nout = G.nout, nout_p = G.nout_p, klo = G.klo, khi = G.khi;
  const bool sin_kind = G.sin_kind != 0, xpass = G.xpass != 0;
  const double r0 = G.r0, rD = G.rD;
  const int row = w.m0 + quad * 32 + lane;
  const bool valid = row < G.rows;
  int jb = G.job0;
  while (jb + 1 < G.job0 + G.njobs && row >= b.job[jb + 1].row0) ++jb;
  const long long out_sk = b.job[jb].out_sk;
  double* const orow = valid ? b.job[jb].out + (long long)(row - b.job[jb].row0) * b.job[jb].out_sl : nullptr;
  const int ex = valid ? __ldcg(G.rowexp + row) : 0;
  // maxima over the lines of each output, for the digits of the y pass
  unsigned* const cmax = b.job[jb].cmax;
  const int jb0 = __shfl_sync(0xffffffffu, jb, 0);
  const bool one_job = __all_sync(0xffffffffu, !valid || jb == jb0);
  // the exponent in two parts, the second a rare factor; NaN for a line
  // that is not finite
  const int e_all = ex + G.ew, er = max(min(e_all, 899), -999);
  const bool bad = ex == kNonFinite || !ok, far = bad || er != e_all;
  const int nc = min(c_end, nout_p - n0);
  long long a[kOutCols], o[kOutCols];
  auto fetch = [&](int c0) {
#pragma unroll
    for (int i = 0; i < kOutCols; ++i) {
      a[i] = __ldcg(even + (c0 + i) * kBM);
      o[i] = form == 0 ? __ldcg(odd + (c0 + i) * kBM) : 0;
    }
  };
  if (c_begin < nc) fetch(c_begin);
#pragma unroll 1
  for (int c0 = c_begin; c0 < nc; c0 += kOutCols) {
    for (int q = 1; q < nseg; ++q) {
#pragma unroll
      for (int i = 0; i < kOutCols; ++i) {
        a[i] += __ldcg(even + q * kSums + (c0 + i) * kBM);
        if (form == 0) o[i] += __ldcg(odd + q * kSums + (c0 + i) * kBM);
      }
    }
    long long s[kOutCols][2];
#pragma unroll
    for (int i = 0; i < kOutCols; ++i) {
      s[i][0] = a[i] + o[i];
      s[i][1] = sin_kind ? o[i] - a[i] : a[i] - o[i];
    }
    if (c0 + kOutCols < nc) fetch(c0 + kOutCols);  // in flight during the conversions
    double y[kOutCols][2];
#pragma unroll
    for (int i = 0; i < kOutCols; ++i) {
      y[i][0] = fixed_to_double(s[i][0], er);
      y[i][1] = form == 0 ? fixed_to_double(s[i][1], er) : 0.0;
    }
    if (far) {
      int d = bad ? 0 : e_all - er;
      double f = bad ? __longlong_as_double(0x7ff8000000000000LL) : 1.0;
#pragma unroll 1
      for (int q = 0; q < 3; ++q) {
        const int dq = max(min(d, 1000), -1000);
        f = bad ? f : __hiloint2double((1023 + dq) << 20, 0);
        d -= dq;
#pragma unroll
        for (int i = 0; i < kOutCols; ++i) {
          y[i][0] *= f;
          y[i][1] *= f;
        }
      }
    }
    if (n0 + c0 == 0 && (form == 0 || po == 0)) {
      // the end outputs k = 0 and D have their own scales, or are zero
      y[0][0] = klo > 0 ? 0.0 : y[0][0] * r0;
      y[0][1] = khi <= D ? 0.0 : y[0][1] * rD;
    }
    // form F: outputs n and D - n; form T: output 2 n + parity
    if (!xpass) {
#pragma unroll
      for (int i = 0; i < kOutCols; ++i) {
        const int n = n0 + c0 + i, k = form == 0 ? n : 2 * n + po;
        if (!valid || n >= nout_p || k >= nout) continue;
        orow[(long long)k * out_sk] = y[i][0];
        if (form == 0 && 2 * n != D) orow[(long long)(D - n) * out_sk] = y[i][1];
      }
    } else {
      if (cmax) {
        unsigned mine = 0;
#pragma unroll
        for (int i = 0; i < kOutCols; ++i)
#pragma unroll
          for (int side = 0; side < 2; ++side) {
            const unsigned m = valid ? high_abs(y[i][side]) : 0u;
            const int n = n0 + c0 + i, k = form == 0 ? (side ? D - n : n) : 2 * n + po;
            if (one_job) {
              const unsigned all = __reduce_max_sync(0xffffffffu, m);
              if (lane == i + side * kOutCols) mine = all;
            } else if (valid && n < nout_p && k < nout && (side == 0 || form == 0)) {
              atomicMax(cmax + k, m);
            }
          }
        if (one_job && lane < 2 * kOutCols) {
          const int n = n0 + c0 + (lane & (kOutCols - 1)), side = lane / kOutCols;
          const int k = form == 0 ? (side ? D - n : n) : 2 * n + po;
          if (n < nout_p && k < nout && (side == 0 || form == 0)) atomicMax(b.job[jb0].cmax + k, mine);
        }
      }
      // lines are rows of the output: eight lanes per line
      __syncwarp();
#pragma unroll
      for (int i = 0; i < kOutCols; ++i) {
        stage[lane * kStageRow + i] = y[i][0];
        stage[(32 + lane) * kStageRow + i] = y[i][1];
      }
      __syncwarp();
      const int cl = lane & (kOutCols - 1);
      const int n = n0 + c0 + cl, k = form == 0 ? n : 2 * n + po;
#pragma unroll 4
      for (int r0w = 0; r0w < 32; r0w += 32 / kOutCols) {
        const int r = r0w + lane / kOutCols;
        double* op = reinterpret_cast<double*>(
            __shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(orow), r));
        if (op == nullptr || n >= nout_p || k >= nout) continue;
        op[k] = stage[r * kStageRow + cl];
        if (form == 0 && 2 * n != D) op[D - n] = stage[(32 + r) * kStageRow + cl];
      }
    }
  }
}

template <int NJ>
__global__ void __launch_bounds__(kThreads, 1) k_tc_pass(const __grid_constant__ TcBatchT<NJ> b) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  __shared__ uint64_t full_bar[kStages], empty_bar[kStages], acc_full[3], acc_empty[3];  // levels 0-1, 2-3, 4-5
  __shared__ uint64_t sum_full[kBufs], sum_empty[kBufs], mma_done;
  __shared__ uint32_t tmem_base;
  __shared__ volatile int abort_flag, keep_tmem;
  __shared__ volatile int n_loaded, n_used;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int s = 0; s < 3; ++s) {
      mbar_init(&acc_full[s], 1);
      mbar_init(&acc_empty[s], kDrainWarps);
    }
    for (int s = 0; s < kBufs; ++s) {
      mbar_init(&sum_full[s], kDrainWarps);
      mbar_init(&sum_empty[s], kOutWarps);
    }
    mbar_init(&mma_done, 1);
    abort_flag = keep_tmem = 0;
    n_loaded = n_used = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == kMmaWarp) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                 "r"(512)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base;
  pdl_wait();

  auto unit = [&](int u) { return unit_of(b, u); };

  if (warp >= kLoadWarp) {
    // register shares of the four warpgroups: 152 + 152 + 152 + 56 = 4 x 128
    asm volatile("setmaxnreg.dec.sync.aligned.u32 56;");
    if (warp == kLoadWarp && lane == 0) {
      // ---- loads
      int it = 0;
      for (int u = blockIdx.x; u < b.nunits && !abort_flag; u += gridDim.x) {
        const Unit w = unit(u);
        const TcGroup& G = *w.g;
        for (int p = w.p0; p < w.p0 + w.np && !abort_flag; ++p)
          for (int kb = w.k0; kb < w.k1; ++kb, ++it) {
            const int s = it % kStages;
            if (it >= kStages && !mbar_wait(&empty_bar[s], (unsigned)((it / kStages - 1) & 1))) {
              abort_flag = 1;
              break;
            }
            asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(&full_bar[s])),
                         "r"((unsigned)kStageBytes)
                         : "memory");
            const unsigned dst = smem_u32(base) + s * kStageBytes;
            tma_load_4d(dst, &G.a, kb * kBK, w.m0, 0, p, &full_bar[s]);
            tma_load_4d(dst + kABytes, &G.b, kb * kBK, w.n0, 0, p, &full_bar[s]);
            n_loaded = it + 1;
          }
      }
    }
    if (warp == kMmaWarp) {
      // ---- products
      const uint32_t elected = elect_one();
      int it = 0, nd[3] = {0, 0, 0};  // drains asked for so far
      bool ok = true;
      // the accumulators of class c hold the last sums until they are drained
      auto wait_drained = [&](int c) {
        if (nd[c] > 0 && !mbar_wait(&acc_empty[c], (unsigned)((nd[c] - 1) & 1))) ok = false;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        return ok;
      };
      for (int u = blockIdx.x; u < b.nunits && ok; u += gridDim.x) {
        const Unit w = unit(u);
        const int nk = w.k1 - w.k0;
        for (int p = 0; p < w.np && ok; ++p)
          for (int kb = 0; kb < nk; ++kb, ++it) {
            const int s = it % kStages;
            const bool last = kb + 1 == nk;
            const bool hi0 = kb % kDrainHi == 0, hi1 = last || kb % kDrainHi == kDrainHi - 1;
            const bool lo0 = kb % kDrainLo == 0, lo1 = last || kb % kDrainLo == kDrainLo - 1;
            if (!mbar_wait(&full_bar[s], (unsigned)((it / kStages) & 1))) {
              ok = false;
              break;
            }
            const unsigned sa = smem_u32(base) + s * kStageBytes;
            const uint64_t da = sw64_desc(sa), db = sw64_desc(sa + kABytes);
            auto product = [&](int i, int j, int g, uint32_t idesc, bool fresh) {
#pragma unroll
              for (int kk = 0; kk < 2; ++kk)
                mma_bf16(tmem + g * kBN, da + i * (kBM * kBK * 2 / 16) + 2 * kk,
                         db + j * (kBN * kBK * 2 / 16) + 2 * kk, idesc, !(fresh && kk == 0), elected);
            };
            auto wide = [&](int q, bool fresh) {
              product(kWideI[q], kWideJ[q], kWideI[q] + kWideJ[q], kIdescWide, fresh);
            };
            if (kb == 0 && !wait_drained(2)) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll
            for (int q = 0; q < kNarrow; ++q) product(kNarrowI[q], kNarrowJ[q], 4, kIdesc, kb == 0 && q == 0);
            if (hi0 && !wait_drained(0)) break;
            wide(0, hi0);
            if (lo0 && !wait_drained(1)) break;
            wide(1, lo0);
            wide(2, false);
            if (hi1) {
              mma_commit(&acc_full[0], elected);
              ++nd[0];
            }
#pragma unroll
            for (int q = 3; q < kWide; ++q) wide(q, false);
            if (lo1) {
              mma_commit(&acc_full[1], elected);
              ++nd[1];
            }
            if (last) {
              mma_commit(&acc_full[2], elected);
              ++nd[2];
            }
            mma_commit(&empty_bar[s], elected);
            if (elected) n_used = it + 1;
          }
      }
      if (!ok) abort_flag = 1;
      mma_commit(&mma_done, elected);  // also of the products of a stage left half issued
    }
  } else if (warp >= kDrainWarps) {
    // ---- outputs: parities combined, scaled, stored
    asm volatile("setmaxnreg.inc.sync.aligned.u32 152;");
    const int quad = warp - kDrainWarps;
    double* stage = reinterpret_cast<double*>(base + kStages * kStageBytes) + quad * 2 * 32 * kStageRow;
    int ph = 0;
    bool ok = true;
    // once a wait has run out, NaN to every later tile of the CTA, without waiting
    for (int u = b.split ? b.nunits : (int)blockIdx.x; u < b.nunits; u += gridDim.x) {
      const Unit w = unit(u);
      for (int p = 0; p < w.np && ok; ++p)
        if (!mbar_wait(&sum_full[(ph + p) % kBufs], (unsigned)(((ph + p) / kBufs) & 1))) ok = false;
      const long long* sums = b.sums + (long long)blockIdx.x * kBufs * kSums + quad * 32 + lane;
      put_outputs(b, w, quad, lane, sums + (ph % kBufs) * kSums, sums + ((ph + 1) % kBufs) * kSums, 1, stage, ok, 0, kBN);
      __syncwarp();
      if (lane == 0 && ok)  // else no buffer is given back: another output warp may be reading it
        for (int p = 0; p < w.np; ++p) mbar_arrive(&sum_empty[(ph + p) % kBufs]);
      ph += w.np;
    }
    if (!ok) abort_flag = 1;
  } else {
    // ---- drains
    asm volatile("setmaxnreg.inc.sync.aligned.u32 152;");
    const int quad = warp & 3, half = warp >> 2;
    const uint32_t tw = tmem + ((uint32_t)(quad * 32) << 16) + (uint32_t)(half * kColsPerWarp);
    long long* sums = b.sums + (long long)(half * kColsPerWarp) * kBM + quad * 32 + lane;
    unsigned nd[3] = {0, 0, 0};
    int ph = 0;
    bool ok = true;
    long long acc[kColsPerWarp];
    // add accumulator g, in units of 2^-9g, to the sums
    auto drain = [&](auto gc) {
      constexpr int g = decltype(gc)::value;
      constexpr float up = g == 0 ? 1.0f : (g == 1 ? 0x1p9f : (g == 2 ? 0x1p18f : (g == 3 ? 0x1p27f : 0x1p34f)));
      constexpr long long unit = g < 4 ? 1LL << (kFrac - 9 * (g & 3)) : 1LL;
#pragma unroll
      for (int h = 0; h < kColsPerWarp; h += 16) {
        uint32_t r[16];
        tmem_ld16(tw + g * kBN + h, r);
        tmem_wait_ld();
#pragma unroll
        for (int c = 0; c < 16; ++c) acc[h + c] += (long long)__float2int_rn(__uint_as_float(r[c]) * up) * unit;
      }
    };
    auto begin_drain = [&](int c) {
      if (!mbar_wait(&acc_full[c], nd[c] & 1u)) ok = false;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      return ok;
    };
    auto end_drain = [&](int c) {
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(&acc_empty[c]);
      ++nd[c];
    };
    for (int u = blockIdx.x; u < b.nunits && ok; u += gridDim.x) {
      const Unit w = unit(u);
      const int nkb = w.k1 - w.k0;
      for (int p = 0; p < w.np && ok; ++p, ++ph) {
#pragma unroll
        for (int c = 0; c < kColsPerWarp; ++c) acc[c] = 0;
        for (int kb = 0; kb < nkb; kb += kDrainLo) {
          const bool last = kb + kDrainLo >= nkb;
          if (last || kb % kDrainHi == kDrainHi - kDrainLo) {
            if (!begin_drain(0)) break;
            drain(std::integral_constant<int, 0>());
            drain(std::integral_constant<int, 1>());
            end_drain(0);
          }
          if (!begin_drain(1)) break;
          drain(std::integral_constant<int, 2>());
          drain(std::integral_constant<int, 3>());
          end_drain(1);
        }
        if (ok && begin_drain(2)) {
          drain(std::integral_constant<int, 4>());
          end_drain(2);
        }
        // 256 bytes per store: lane = line
        if (ok && !b.split && ph >= kBufs && !mbar_wait(&sum_empty[ph % kBufs], (unsigned)((ph / kBufs - 1) & 1)))
          ok = false;
        if (!ok) break;
        long long* dst = sums + (b.split ? (long long)u : (long long)blockIdx.x * kBufs + ph % kBufs) * kSums;
#pragma unroll
        for (int c = 0; c < kColsPerWarp; ++c) dst[c * kBM] = acc[c];
        __syncwarp();
        if (lane == 0 && !b.split) mbar_arrive(&sum_full[ph % kBufs]);
      }
    }
    if (!ok) abort_flag = 1;
  }
  __syncwarp();
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (threadIdx.x == 0) {
    // the loads and products in flight, and their arrivals, end before the CTA does;
    // products that never finish keep their tensor memory
    if (abort_flag)
      for (int i = n_used; i < n_loaded; ++i) (void)mbar_wait(&full_bar[i % kStages], (unsigned)((i / kStages) & 1));
    keep_tmem = mbar_wait(&mma_done, 0) ? 0 : 1;
    if (abort_flag || keep_tmem) {
      *b.failed = 1;
      *b.expired = keep_tmem ? 2 : 1;
      __threadfence_system();
    }
  }
  __syncthreads();
  if (warp == kMmaWarp && !keep_tmem)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
}

// The outputs of split tiles: a CTA of four warps (one per 32 lines) takes
// kOutCols outputs of a tile, so that the whole GPU shares what the last CTA
// of a tile would do alone (33 us a tile).
template <int NJ>
__global__ void __launch_bounds__(kOutWarps * 32) k_tc_finish(const __grid_constant__ TcBatchT<NJ> b) {
  __shared__ double stage[kOutWarps * 2 * 32 * kStageRow];
  constexpr int kParts = kBN / kOutCols;
  int g = 0;
  const int tile = (int)blockIdx.x / kParts, part = (int)blockIdx.x - tile * kParts;
  while (g + 1 < b.ngroups && tile >= b.grp[g + 1].tile0) ++g;
  const int per = b.grp[g].nseg * (b.grp[g].form == 0 ? 2 : 1);
  const int u = b.grp[g].unit0 + (tile - b.grp[g].tile0) * per;
  const Unit w = unit_of(b, u);
  const int quad = threadIdx.x >> 5, lane = threadIdx.x & 31;
  pdl_wait();
  const long long* even = b.sums + (long long)u * kSums + quad * 32 + lane;
  put_outputs(b, w, quad, lane, even, even + (long long)w.g->nseg * kSums, w.g->nseg,
              stage + quad * 2 * 32 * kStageRow, __ldcg(b.failed) == 0u, part * kOutCols, (part + 1) * kOutCols);
}

// The HOS accumulation on the outputs of a finished pass (AccEpi): in a kernel
// of its own, since its loads and FP64 sums (up to 14 per output) would hold
// up the output warps above.
__global__ void __launch_bounds__(256) k_tc_accumulate(AccEpi acc, const double* __restrict__ z1, int nlines,
                                                       int nout, long long sk) {
  pdl_wait();
  const int line = blockIdx.x * 256 + threadIdx.x;
  if (line >= nlines) return;
  for (int k = blockIdx.y; k < nout; k += gridDim.y) {
    const long long i = line + k * sk;
    acc_epilogue(acc, i, __ldcg(z1 + i));
  }
}

// ---------------------------------------------------------------- matrices

// digits of the entry q = (row x column index) mod 2 D from the host's table
// (eight BF16 per entry, six used), rows r < nrows of both parities
__global__ void k_tc_matrix(const uint4* __restrict__ tab, __nv_bfloat16* m, int D, int form, int nrows, int kp) {
  const long long n = 2LL * nrows * kp;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const int p = (int)(i / ((long long)nrows * kp));
    const int rem = (int)(i - (long long)p * nrows * kp);
    const int r = rem / kp, c = rem - r * kp;
    // form F: output r, input 2 c + p; form T: output 2 r + p, input c
    const int j = form == 0 ? 2 * c + p : c, k = form == 0 ? r : 2 * r + p;
    uint4 e = make_uint4(0, 0, 0, 0);
    if (form == 0 ? j <= D : 2 * j <= D) e = __ldg(tab + (int)((long long)j * k % (2 * D)));
    const unsigned w[3] = {e.x, e.y, e.z};
#pragma unroll
    for (int s = 0; s < kS; ++s) {
      const unsigned short h = (unsigned short)(w[s >> 1] >> (16 * (s & 1)));
      reinterpret_cast<unsigned short*>(m)[((long long)(p * kS + s) * nrows + r) * kp + c] = h;
    }
  }
}

unsigned short bf16_bits(float f) {  // round to nearest even (finite f)
  unsigned u;
  std::memcpy(&u, &f, 4);
  u += 0x7fffu + ((u >> 16) & 1u);
  return (unsigned short)(u >> 16);
}
float bf16_float(unsigned short h) {
  const unsigned u = (unsigned)h << 16;
  float f;
  std::memcpy(&f, &u, 4);
  return f;
}

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
EncodeTiledFn encode_fn() {
  static const EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      return (EncodeTiledFn)p;
    return (EncodeTiledFn) nullptr;
  }();
  return fn;
}

// [parity][digit][rows][kp] BF16, boxes of kBK x box_rows x kS
bool make_map(CUtensorMap* m, const void* ptr, int rows, int kp, int box_rows) {
  const EncodeTiledFn enc = encode_fn();
  if (!enc) return false;
  const cuuint64_t dims[4] = {(cuuint64_t)kp, (cuuint64_t)rows, kS, 2};
  const cuuint64_t strides[3] = {(cuuint64_t)kp * 2, (cuuint64_t)rows * kp * 2, (cuuint64_t)kS * rows * kp * 2};
  const cuuint32_t box[4] = {kBK, (cuuint32_t)box_rows, kS, 1};
  const cuuint32_t estr[4] = {1, 1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 4, const_cast<void*>(ptr), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int pad_k(int k) { return (k + kBK - 1) / kBK * kBK; }

// Jobs of one matrix and the same extents: their lines form one operand.
struct GroupShape {
  int tiles, nkb, np;  // tiles of all parities (form T), stages and parities of a tile
};
int terms_of(const AxisJob& J, const TcMat& m) {
  return m.form == 0 ? pad_k((std::min(J.jhi, J.nin) + 1) / 2) : m.kp;
}
GroupShape shape_of(const AxisJob& J, const TcMat& m, long long rows) {
  const int nout_p = m.form == 0 ? m.nrows : (J.nout + 1) / 2;
  const long long tiles = (rows + kBM - 1) / kBM * ((nout_p + kBN - 1) / kBN) * (m.form == 0 ? 1 : 2);
  return GroupShape{(int)tiles, terms_of(J, m) / kBK, m.form == 0 ? 2 : 1};
}
bool same_group(const AxisJob& a, const TcMat* ma, const AxisJob& b, const TcMat* mb) {
  return ma == mb && a.nin == b.nin && a.nout == b.nout;
}

// Whether the tiles are split, and how far: a wave of whole tiles leaves SMs
// idle when the tiles are few or the last wave is short.  Segments per parity
// (0: whole tiles) and the cycles of the product.  Measured on GB300: a stage of
// products 2900 cycles, a unit's drains 4000, the outputs of the last whole tile
// 30000, the launch that finishes split tiles 8000.
struct Split {
  int nseg;
  double cycles;
};
Split best_split(const std::vector<GroupShape>& groups, int nsm, long long sum_cap) {
  constexpr double kStage = 2900.0, kUnit = 4000.0, kOut = 30000.0, kFinish = 8000.0;
  auto waves = [&](long long n) { return (double)((n + nsm - 1) / nsm); };
  double whole = 0.0;
  long long tiles = 0;
  for (const GroupShape& g : groups) {
    whole = std::max(whole, g.np * (g.nkb * kStage + kUnit));
    tiles += g.tiles;
  }
  Split best{0, waves(tiles) * whole + kOut};
  for (int ns = 1; ns <= 8; ++ns) {
    long long units = 0;
    double unit = 0.0;
    for (const GroupShape& g : groups) {
      const int n = std::min(ns, g.nkb);
      units += (long long)g.tiles * n * g.np;
      unit = std::max(unit, (g.nkb + n - 1) / n * kStage + kUnit);
    }
    if (units > sum_cap) break;
    const double c = waves(units) * unit + kFinish * (1.0 + 0.1 * ns);
    if (c < 0.95 * best.cycles) best = Split{ns, c};
  }
  return best;
}


template <typename Fn>
void with_tc_capacity(int n, Fn&& f) {
  if (n <= 1) f(std::integral_constant<int, 1>());
  else if (n <= 4) f(std::integral_constant<int, 4>());
  else f(std::integral_constant<int, kMaxJobs>());
}

// HOSNWT_FFT = 0 or 1 forces the sum or the FFT passes, 2 these passes
// wherever a matrix exists; the FP64 DFT (HOSNWT_FFT_DF = 0) goes without
// them too.  Returns 0 off, 1 by the rule, 2 forced.
int tc_mode() {
  static const int m = [] {
    const char* d = std::getenv("HOSNWT_FFT_DF");
    if (d && d[0] == '0') return 0;
    const char* e = std::getenv("HOSNWT_FFT");
    if (!e || !e[0]) return 1;
    return e[0] == '2' ? 2 : (e[0] == '0' || e[0] == '1' ? 0 : 1);
  }();
  return m;
}

}  // namespace

// The matrix of one form of a pass of length D (see TcMat).  scale is the
// interior output scale times the interior input weight.
bool describe_tc_matrix(int D, int form, int sin_kind, double scale, int nout, TcMat* out) {
  if (D < 8 || D > kTcMaxD) return false;
  *out = TcMat{};
  out->D = D;
  out->form = form;
  out->sin_kind = sin_kind;
  out->scale = scale;
  out->nout = form == 0 ? D + 1 : nout;
  out->nrows = form == 0 ? D / 2 + 1 : (nout + 1) / 2;
  out->kp = pad_k(D / 2 + 1);
  return true;
}

// Its digits on the device.  quarter holds the first quarter turn's cosines,
// filled as they are asked for (the forms of a length share them); the table of
// entries passes through `scratch`.  The matrix is complete once the default
// stream is.
bool build_tc_matrix(TcMat* out, std::vector<long double>& quarter, double* scratch, std::vector<void*>& allocs) {
  const int D = out->D, form = out->form, sin_kind = out->sin_kind;
  const double scale = out->scale;
  if (!scratch) return false;
  int ew = 0;
  const long double c = frexpl((long double)scale, &ew);  // scale = c 2^ew, c in [1/2, 1)
  const long double pi = 3.141592653589793238462643383279502884L;
  if ((int)quarter.size() != D + 1) quarter.assign(D + 1, 2.0L);
  std::vector<unsigned short> tab((size_t)2 * D * 8, 0);
  for (int q = 0; q < 2 * D; ++q) {
    // cos(pi m / (2 D)) with the angle folded to the first quarter turn
    int m = 2 * q;
    if (sin_kind) m = ((m - D) % (4 * D) + 4 * D) % (4 * D);
    if (m > 2 * D) m = 4 * D - m;
    const bool neg = m > D;
    if (neg) m = 2 * D - m;
    long double& v = quarter[m];
    if (v > 1.0L)
      v = (m == D) ? 0.0L
                   : (2 * m > D ? sinl(pi * (long double)(D - m) / (2.0L * D)) : cosl(pi * (long double)m / (2.0L * D)));
    float d[5];
    split_digits(llrintl(ldexpl(v * (neg ? -c : c), 62)), d);
    unsigned short* t = &tab[(size_t)q * 8];
    for (int s = 0; s < 5; ++s) t[s] = bf16_bits(d[s]);
    t[5] = bf16_bits(d[4] - bf16_float(t[4]));
  }
  const int nrows = out->nrows, kp = out->kp;
  void* mat = nullptr;
  if (cudaMalloc(&mat, (size_t)2 * kS * nrows * kp * 2) != cudaSuccess) {
    cudaGetLastError();  // this refusal: the job keeps its other pass
    return false;
  }
  allocs.push_back(mat);
  if (cudaMemcpy(scratch, tab.data(), tab.size() * 2, cudaMemcpyHostToDevice) != cudaSuccess) return false;
  k_tc_matrix<<<1024, 256>>>((const uint4*)scratch, (__nv_bfloat16*)mat, D, form, nrows, kp);
  if (cudaPeekAtLastError() != cudaSuccess) return false;  // left for the caller
  out->ew = ew;
  out->dev = mat;
  return true;
}

long long tc_scratch_doubles(const TcNeed& need) {
  return kTcMaxBytes / 8 + need.units * kSums + need.digits / 8 + 512 * kMaxJobs;
}

const TcMat* tc_matrix_of(const AxisJob& J, const Tables& tb) {
  if (tc_mode() == 0 || tb.ntc == 0) return nullptr;
  const bool c1s1 = (J.aj == 2 && J.bj == 0 && J.ak == 1 && J.bk == 0);
  if (!c1s1 || J.wm == 0.0 || J.sm == 0.0 || J.nlines < 32) return nullptr;
  if ((J.in_sk == 1) == (J.in_sl == 1) || (J.in_sk == 1 && J.epi)) return nullptr;
  const int sin_kind = J.off != 0 ? 1 : 0;
  const int form = J.nout == J.N ? 0 : 1;
  if (form == 1 && J.nin < J.N) return nullptr;
  const double scale = J.wm * J.sm * J.gscale;
  // end inputs of full or half weight
  if ((J.w0 != J.wm && J.w0 != 0.5 * J.wm) || (J.wl != J.wm && J.wl != 0.5 * J.wm)) return nullptr;
  for (int i = 0; i < tb.ntc; ++i) {
    const TcMat& m = tb.tc[i];
    if (m.D == J.D && m.form == form && m.sin_kind == sin_kind && m.scale == scale && J.nout <= m.nout) return &m;
  }
  return nullptr;
}

// Which requests go to the tensor cores.  Their x and y passes go together (the
// x pass leaves the maxima that the y pass needs; without them the digits of
// a y pass cost twice).  A class of requests of the same lengths and extents
// goes if its digits and products take less than its other passes, and all
// of them together if they still do with the three launches of a pass.  The times
// (us), measured on GB300: 6 ps per digit set (a y pass without maxima 12),
// 17 us per pass for the launches and their latencies, 8 us for those of a pass
// elsewhere (pass_time counts its work alone).  On both sides of the
// line (one field of the dealiased grid, both passes): 258 x 66 points 37
// against 18 us by the FFT, 770 x 194 points 49 against 40, 642 x 627 points 59
// against 77, 1282 x 642 points 93 against 128, 4100 x 2052 points 985 against 1920.
void tc_choose(AxisJob* const* jobs, const double* const* alt, int npass, int n, const Tables& tb) {
  if (tc_mode() == 0 || tb.ntc == 0) return;
  std::vector<std::vector<int>> cls;
  std::vector<const TcMat*> mat((size_t)npass * n);
  for (int i = 0; i < n; ++i) {
    bool all = true;
    for (int p = 0; p < npass; ++p) all = all && (mat[(size_t)p * n + i] = tc_matrix_of(jobs[p][i], tb)) != nullptr;
    if (!all) continue;
    bool put = false;
    for (auto& g : cls) {
      bool same = true;
      for (int p = 0; p < npass; ++p)
        same = same && same_group(jobs[p][g[0]], mat[(size_t)p * n + g[0]], jobs[p][i], mat[(size_t)p * n + i]);
      if (same) {
        g.push_back(i);
        put = true;
        break;
      }
    }
    if (!put) cls.push_back({i});
  }
  const int nsm = std::max(tb.nsm, 1);
  std::vector<std::vector<GroupShape>> shapes(npass);
  std::vector<int> chosen;
  double tc = 0.0, other = 0.0;
  for (const auto& g : cls) {
    double t = 0.0, f = 0.0;
    std::vector<GroupShape> sh;
    for (int p = 0; p < npass; ++p) {
      const AxisJob& J = jobs[p][g[0]];
      const TcMat& m = *mat[(size_t)p * n + g[0]];
      long long rows = 0;
      for (int i : g) {
        rows += jobs[p][i].nlines;
        f += alt[p][i];
      }
      sh.push_back(shape_of(J, m, rows));
      const bool maxima = npass == 2 || J.in_sk == 1;
      t += (maxima ? 6e-6 : 12e-6) * (double)rows * terms_of(J, m) * 2.0;
      t += (double)sh[p].tiles * sh[p].np * sh[p].nkb * 2900.0 / nsm / 1900.0;
    }
    if (t < f || tc_mode() == 2) {
      chosen.insert(chosen.end(), g.begin(), g.end());
      other += f;
      for (int p = 0; p < npass; ++p) {
        shapes[p].push_back(sh[p]);
        tc -= (double)sh[p].tiles * sh[p].np * sh[p].nkb * 2900.0 / nsm / 1900.0;
      }
      tc += t;
    }
  }
  if (chosen.empty()) return;
  for (int p = 0; p < npass; ++p) {
    tc += 17.0 + best_split(shapes[p], nsm, tb.tc_units).cycles / 1900.0;
    other += 8.0;
  }
  if (tc > other && tc_mode() != 2) return;
  for (int i : chosen)
    for (int p = 0; p < npass; ++p) jobs[p][i].tc = mat[(size_t)p * n + i];
}

// A batch of one, a few and `most` requests of one kind: what a request gains does
// not fall with their number (the launches are shared), and in a mixed batch no
// kind gains more than alone.  The buffers of sums are those of kMaxJobs requests cut
// as far as best_split cuts, or the kBufs of every CTA, and at most kUnitsPerSm per
// SM; the digits those of `held` requests (a batch of more goes in parts).
void tc_need(const AxisJob* passes, const double* alt, int npass, const Tables& tb, int most, int held, TcNeed* need) {
  const int nsm = std::max(tb.nsm, 1);
  Tables full = tb;
  full.tc_units = nsm * kUnitsPerSm;
  bool any = false;
  for (int q : {1, (most + 1) / 2, most}) {
    std::vector<AxisJob> j[2];
    std::vector<double> a[2];
    AxisJob* jobs[2] = {};
    const double* alts[2] = {};
    for (int p = 0; p < npass; ++p) {
      j[p].assign(q, passes[p]);
      a[p].assign(q, alt[p]);
      jobs[p] = j[p].data();
      alts[p] = a[p].data();
    }
    tc_choose(jobs, alts, npass, q, full);
    if (!j[0][0].tc) continue;
    any = true;
    for (int p = 0; p < npass; ++p) {
      const TcMat& m = *j[p][0].tc;
      const GroupShape one = shape_of(passes[p], m, passes[p].nlines);
      const long long tiles = (long long)kMaxJobs * one.tiles;
      const long long units = std::max(tiles * std::min(8, one.nkb) * one.np, kBufs * std::min<long long>(nsm, tiles));
      need->units = std::max(need->units, std::min<long long>(units, full.tc_units));
      need->digits = std::max(need->digits, (long long)held * passes[p].nlines * (terms_of(passes[p], m) * 4LL * kS + 4));
    }
  }
  need->any = need->any || any;
}

bool launch_tc_jobs(const AxisBatch& in, const Tables& tb, cudaStream_t st) {
  const TcMat* mat[kMaxJobs];
  for (int i = 0; i < in.njobs; ++i) mat[i] = in.job[i].tc;
  const bool ymode = in.njobs > 0 && in.job[0].in_sk != 1;
  char* const scratch = reinterpret_cast<char*>(tb.cs) + kTcMaxBytes;  // after the maxima
  const long long cap = tb.cs_cap * (long long)sizeof(double) - kTcMaxBytes;
  const long long sum_cap = tb.tc_units;  // buffers of sums
  if (sum_cap < kBufs) return false;
  const long long stash_bytes = sum_cap * kSums * 8;
  // groups of jobs with the same matrix and extents
  std::vector<std::vector<int>> groups;
  for (int i = 0; i < in.njobs; ++i) {
    bool put = false;
    for (auto& g : groups) {
      if (same_group(in.job[g[0]], mat[g[0]], in.job[i], mat[i])) {
        g.push_back(i);
        put = true;
        break;
      }
    }
    if (!put) groups.push_back({i});
  }
  static PerDeviceOnce attr;
  attr.run([&] {
    for (int nj : {1, 4, kMaxJobs})
      with_tc_capacity(nj, [&](auto c) {
        constexpr int NJ = decltype(c)::value;
        cudaFuncSetAttribute(k_tc_pass<NJ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kPassSmem);
        cudaFuncSetAttribute(k_tc_digits_y<NJ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDgySmem);
      });
  });
  size_t gi = 0, gj = 0;  // next group, next job inside it
  while (gi < groups.size()) {
    // as many jobs as the scratch holds
    TcBatch B{};
    DgBatch Dg{};
    B.sums = reinterpret_cast<long long*>(scratch);
    B.failed = tb.tc_failed;
    B.expired = tb.tc_expired;
    int ntiles = 0;
    long long used = (stash_bytes + 1023) / 1024 * 1024;
    int nj = 0, dblocks = 0;
    while (gi < groups.size()) {
      const std::vector<int>& g = groups[gi];
      const int kp = terms_of(in.job[g[0]], *mat[g[0]]);
      size_t end = gj;
      long long rows = 0;
      while (end < g.size()) {
        const long long r = rows + in.job[g[end]].nlines;
        if (used + r * kp * 2 * kS * 2 + r * 4 + 2048 > cap) break;
        rows = r;
        ++end;
      }
      if (end == gj) break;
      const TcMat& m = *mat[g[0]];
      const AxisJob& J0 = in.job[g[0]];
      TcGroup& G = B.grp[B.ngroups];
      __nv_bfloat16* a = reinterpret_cast<__nv_bfloat16*>(scratch + used);
      used = (used + rows * kp * 2 * kS * 2 + 1023) / 1024 * 1024;
      int* rowexp = reinterpret_cast<int*>(scratch + used);
      used = (used + rows * 4 + 1023) / 1024 * 1024;
      if (!make_map(&G.a, a, (int)rows, kp, kBM)) return false;
      if (!make_map(&G.b, m.dev, m.nrows, m.kp, kBN)) return false;
      G.rows = (int)rows;
      G.nkb = kp / kBK;
      G.nout_p = m.form == 0 ? m.nrows : (J0.nout + 1) / 2;
      G.tm = (int)((rows + kBM - 1) / kBM);
      G.tn = (G.nout_p + kBN - 1) / kBN;
      G.tile0 = ntiles;
      ntiles += G.tm * G.tn * (m.form == 0 ? 1 : 2);
      G.form = m.form;
      G.sin_kind = m.sin_kind;
      G.D = m.D;
      G.ew = m.ew;
      G.job0 = nj;
      G.njobs = (int)(end - gj);
      G.nout = J0.nout;
      G.klo = J0.klo;
      G.khi = J0.khi;
      G.xpass = ymode ? 0 : 1;
      G.r0 = J0.s0 / J0.sm;
      G.rD = J0.sl / J0.sm;
      G.rowexp = rowexp;
      int row0 = 0;
      for (size_t q = gj; q < end; ++q, ++nj) {
        const AxisJob& J = in.job[g[q]];
        TcJob& T = B.job[nj];
        T.out = J.out;
        T.out_sk = J.out_sk;
        T.out_sl = J.out_sl;
        T.row0 = row0;
        T.cmax = ymode ? nullptr : J.cmax;
        DgJob& X = Dg.job[nj];
        X.in = J.in;
        X.in_sk = J.in_sk;
        X.in_sl = J.in_sl;
        X.win = J.win;
        X.win_sk = J.win_sk;
        X.win_sl = J.win_sl;
        X.nlines = J.nlines;
        X.jlo = J.jlo;
        X.jend = std::min(J.jhi, J.nin);
        X.D = m.D;
        X.form = m.form;
        X.sin_kind = m.sin_kind;
        X.kp = kp;
        X.half0 = J.w0 != J.wm;
        X.halfD = J.wl != J.wm;
        X.rows = (int)rows;
        X.row0 = row0;
        X.a = a;
        X.rowexp = rowexp;
        X.lmax = ymode && !J.win ? J.lmax : nullptr;
        X.cmax = T.cmax;
        X.ncmax = J.nout;
        row0 += J.nlines;
        g_xform_fmas += (double)J.nlines * G.nout_p * kp * 2.0;
      }
      ++B.ngroups;
      gj = end;
      if (gj < g.size()) break;  // scratch full inside a group
      ++gi;
      gj = 0;
    }
    if (nj == 0) return false;  // one job does not fit
    std::vector<GroupShape> shapes;
    for (int g = 0; g < B.ngroups; ++g)
      shapes.push_back(GroupShape{(g + 1 < B.ngroups ? B.grp[g + 1].tile0 : ntiles) - B.grp[g].tile0, B.grp[g].nkb,
                                  B.grp[g].form == 0 ? 2 : 1});
    const int nseg = best_split(shapes, std::max(tb.nsm, 1), sum_cap).nseg;
    B.split = nseg > 0;
    B.nunits = 0;
    for (int g = 0; g < B.ngroups; ++g) {
      TcGroup& G = B.grp[g];
      const int n = std::max(1, std::min(nseg, G.nkb));
      G.segk = (G.nkb + n - 1) / n;
      G.nseg = (G.nkb + G.segk - 1) / G.segk;
      G.unit0 = B.nunits;
      B.nunits += shapes[g].tiles * (B.split ? G.nseg * shapes[g].np : 1);
    }
    // digits
    Dg.njobs = nj;
    Dg.wpl = 1;
    long long lines = 0;
    for (int i = 0; i < nj; ++i) {
      if (Dg.job[i].kp > 128) Dg.wpl = kDgThreads / 32;
      lines += (Dg.job[i].nlines + 31) / 32;
    }
    for (int i = 0; i < nj; ++i) {
      DgJob& X = Dg.job[i];
      Dg.start[i] = dblocks;
      if (ymode) {
        const int nch = (X.kp + 63) / 64;
        X.nsplit = (int)std::min<long long>(nch, std::max<long long>(1, 4LL * tb.nsm / std::max(lines, 1LL)));
        X.cps = (nch + X.nsplit - 1) / X.nsplit;
        X.nsplit = (nch + X.cps - 1) / X.cps;
        dblocks += (X.nlines + 31) / 32 * X.nsplit;
      } else {
        const int lpc = (kDgThreads / 32) / Dg.wpl;
        dblocks += (X.nlines + lpc - 1) / lpc;
      }
    }
    Dg.start[nj] = dblocks;
    with_tc_capacity(nj, [&](auto c) {
      constexpr int NJ = decltype(c)::value;
      DgBatchT<NJ> d{};
      TcBatchT<NJ> t{};
      for (int i = 0; i < nj; ++i) {
        d.job[i] = Dg.job[i];
        t.job[i] = B.job[i];
      }
      for (int i = 0; i <= nj; ++i) d.start[i] = Dg.start[i];
      d.njobs = nj;
      d.wpl = Dg.wpl;
      for (int i = 0; i < B.ngroups; ++i) t.grp[i] = B.grp[i];
      t.ngroups = B.ngroups;
      t.nunits = B.nunits;
      t.split = B.split;
      t.sums = B.sums;
      t.failed = B.failed;
      t.expired = B.expired;
      if (ymode) launch_pdl(k_tc_digits_y<NJ>, dim3(dblocks), dim3(kDgThreads), kDgySmem, st, d);
      else launch_pdl(k_tc_digits_x<NJ>, dim3(dblocks), dim3(kDgThreads), 0, st, d);
      // whole tiles: kBufs buffers per CTA
      const int ctas = B.split ? tb.nsm : (int)std::min<long long>(tb.nsm, sum_cap / kBufs);
      launch_pdl(k_tc_pass<NJ>, dim3(std::min(B.nunits, ctas)), dim3(kThreads), kPassSmem, st, t);
      if (B.split) launch_pdl(k_tc_finish<NJ>, dim3(ntiles * (kBN / kOutCols)), dim3(kOutWarps * 32), 0, st, t);
    });
  }
  for (int i = 0; i < in.njobs; ++i) {
    const AxisJob& J = in.job[i];
    if (J.epi)
      launch_pdl(k_tc_accumulate, dim3((J.nlines + 255) / 256, std::min(J.nout, 2048)), dim3(256), 0, st, in.acc,
                 (const double*)J.out, J.nlines, J.nout, J.out_sk);
  }
  return true;
}

}  // namespace hos
