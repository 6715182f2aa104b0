// Spectral transforms of the HOS-NWT hot path on sm_103a.
//
// Replaces the FFTW r2r plans of fourier_FFTW.f90:89-653 (DCT_FFTW,
// IDCT_FFTW, DCT_FFTW_big, IDCT_FFTW_big, DCT_FFTW_add, IDCT_FFTW_add).
// The lengths of the dealiased grid, Nd = ((p+1) n)/2 (common_vars.f90:40-41),
// have large prime factors, so each pass is computed as an exact FP64 sum
// over a quarter-wave twiddle table indexed with integer arithmetic.  That
// works for every length and kind and keeps the normalisation fused.
//
// On GB300 the FP64 pipe (about 1.2 TFLOP/s) is the bound of these passes,
// not HBM: an x pass spreads one line over many CTAs (8 warps split the sum,
// lanes own outputs), a y pass gives one row per lane (coalesced loads,
// warp-uniform twiddles) and several outputs per thread.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <type_traits>

#include "hosnwt_internal.h"

namespace hos {

namespace {

__device__ __forceinline__ double twiddle(const double* __restrict__ q, int D, int m) {
  // m in [0, 4D): cos(pi*m/(2D)) from the quarter-wave table
  int mm = (m > 2 * D) ? 4 * D - m : m;
  return (mm > D) ? -__ldg(q + (2 * D - mm)) : __ldg(q + mm);
}

__device__ __forceinline__ int mod4d(long long v, int D4) {
  long long r = v % D4;
  return (int)(r < 0 ? r + D4 : r);
}

// input j of a first-pass line, times the optional weight
__device__ __forceinline__ double in_at(const double* __restrict__ x, long long sk,
                                       const double* __restrict__ w, long long wsk, int j) {
  const double v = __ldg(x + (long long)j * sk);
  return w ? v * __ldg(w + (long long)j * wsk) : v;
}

constexpr int kXThreads = 256;   // 8 warps
constexpr int kXWarps = kXThreads / 32;
constexpr int kMaxPairChunk = 1024;  // staged terms per CTA

__device__ __forceinline__ double twiddle_s(const double* q, int D, int m) {
  int mm = (m > 2 * D) ? 4 * D - m : m;
  return (mm > D) ? -q[2 * D - mm] : q[mm];
}

// x pass: one CTA = (job, line, tile of 32 lane outputs, chunk of the sum).
// The quarter-wave table of the job and the CTA's chunk of inputs are staged
// in shared memory; lanes own outputs (twiddles are gathered from shared
// memory, inputs are broadcast), the 8 warps split the chunk, and the chunks
// of one tile are combined in a fixed order by the last CTA to arrive.
//   mode 0: direct sum over the interior terms plus the two end terms
//   mode 1: output symmetry: lane k accumulates even-j and odd-j sums E, O
//           and writes out[k] and out[D-k] (full outputs, D = N-1)
//   mode 2: input symmetry: terms are pairs (j, D-j) staged as
//           u = x_j + x_{D-j}, v = x_j - x_{D-j} (outputs k <= D/2)
template <int NJ>
__global__ void __launch_bounds__(kXThreads) axis_pass_lanes_k(const AxisBatchT<NJ> b) {
  extern __shared__ double smem[];
  __shared__ double red[kXWarps][32][2];
  __shared__ bool amlast;
  int jb = 0;
  while (jb + 1 < b.njobs && (int)blockIdx.x >= b.start[jb + 1]) ++jb;
  const AxisJob& J = b.job[jb];
  int local = blockIdx.x - b.start[jb];
  const int chunk_id = local % J.nchunk;
  local /= J.nchunk;
  const int tile = local % J.ntile;
  const int line = local / J.ntile;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k = tile * 32 + lane;
  const int D = J.D, D4 = 4 * D;
  const double* __restrict__ x = J.in + (long long)line * J.in_sl;
  const int kk = J.ak * k + J.bk;
  const int inc = mod4d((long long)J.aj * kk, D4);
  const bool lane_on = k < J.nlane;
  const long long sk = J.in_sk;
  const double* __restrict__ wr = J.win ? J.win + (long long)line * J.win_sl : nullptr;

  double* q = smem;                    // D + 1 table entries
  double* su = smem + (D + 1);         // staged inputs (or u)
  double* sv = su + kMaxPairChunk;     // v (mode 2)
  if (b.early)
    for (int t = threadIdx.x; t <= D; t += kXThreads) q[t] = __ldg(J.q + t);
  pdl_wait();
  if (!b.early)
    for (int t = threadIdx.x; t <= D; t += kXThreads) q[t] = __ldg(J.q + t);
  const int ca = J.ta + chunk_id * J.chunk;
  const int cb = min(J.tb, ca + J.chunk);
  // cos: even k pairs with u; sin: even k pairs with v (mode 2)
  const bool use_v = (J.mode == 2) && (((k & 1) == 0) != (J.off == 0));
  double e = 0.0, o = 0.0;  // mode 1: even / odd j sums; else e only
  for (int sa = ca; sa < cb; sa += kMaxPairChunk) {
    const int sb = min(cb, sa + kMaxPairChunk);
    __syncthreads();  // previous stage consumed
    if (J.mode == 2) {
      for (int t = threadIdx.x; t < sb - sa; t += kXThreads) {
        const int j = sa + t;
        const double xa = in_at(x, sk, wr, J.win_sk, j);
        const double xb = in_at(x, sk, wr, J.win_sk, D - j);
        su[t] = xa + xb;
        sv[t] = xa - xb;
      }
    } else {
      for (int t = threadIdx.x; t < sb - sa; t += kXThreads) su[t] = in_at(x, sk, wr, J.win_sk, sa + t);
    }
    __syncthreads();
    const int len = sb - sa;
    const int per = (len + kXWarps - 1) / kXWarps;
    const int ja = sa + warp * per;
    const int jz = min(sb, ja + per);
    if (lane_on && jz > ja) {
      int m = mod4d((long long)(J.aj * ja + J.bj) * kk + J.off, D4);
      if (J.mode == 1) {
        int j = ja;
        if (j & 1) {  // align to an even j
          o = fma(su[j - sa], twiddle_s(q, D, m), o);
          m += inc;
          if (m >= D4) m -= D4;
          ++j;
        }
        for (; j + 1 < jz; j += 2) {
          const double te = twiddle_s(q, D, m);
          m += inc;
          if (m >= D4) m -= D4;
          const double to = twiddle_s(q, D, m);
          m += inc;
          if (m >= D4) m -= D4;
          e = fma(su[j - sa], te, e);
          o = fma(su[j + 1 - sa], to, o);
        }
        if (j < jz) e = fma(su[j - sa], twiddle_s(q, D, m), e);
      } else {
        const double* sp = use_v ? sv : su;
        double e2 = 0.0;
        int j = ja;
        for (; j + 1 < jz; j += 2) {
          const double t0 = twiddle_s(q, D, m);
          m += inc;
          if (m >= D4) m -= D4;
          const double t1 = twiddle_s(q, D, m);
          m += inc;
          if (m >= D4) m -= D4;
          e = fma(sp[j - sa], t0, e);
          e2 = fma(sp[j + 1 - sa], t1, e2);
        }
        if (j < jz) e = fma(sp[j - sa], twiddle_s(q, D, m), e);
        e += e2;
      }
    }
  }
  if (cb <= ca) __syncthreads();  // table staged even when this CTA has no terms
  e *= J.wm;
  o *= J.wm;
  // end terms and the unpaired middle term, once per tile (chunk 0, warp 0)
  if (chunk_id == 0 && warp == 0 && lane_on) {
    const int j_end = min(J.jhi, J.nin);
    if (J.mode == 2) {
      if (J.jlo == 0) {  // pair (0, D) with the end weight
        const double xa = in_at(x, sk, wr, J.win_sk, 0), xb = in_at(x, sk, wr, J.win_sk, D);
        const double t = ((k & 1) == 0) ? xa + xb : xa - xb;
        e = fma(J.w0 * t, twiddle_s(q, D, mod4d((long long)J.bj * kk + J.off, D4)), e);
      }
      if ((D & 1) == 0) {
        const int jm = D / 2;
        if (jm >= J.jlo && jm < J.jhi && jm > 0) {
          const int mm = mod4d((long long)(J.aj * jm + J.bj) * kk + J.off, D4);
          e = fma(J.wm * in_at(x, sk, wr, J.win_sk, jm), twiddle_s(q, D, mm), e);
        }
      }
    } else {
      if (J.jlo == 0 && 0 < j_end) {
        const int mm = mod4d((long long)J.bj * kk + J.off, D4);
        e = fma(J.w0 * in_at(x, sk, wr, J.win_sk, 0), twiddle_s(q, D, mm), e);
      }
      const int jl = J.N - 1;
      if (jl > 0 && jl >= J.jlo && jl < j_end) {
        const int mm = mod4d((long long)(J.aj * jl + J.bj) * kk + J.off, D4);
        const double t = J.wl * in_at(x, sk, wr, J.win_sk, jl) * twiddle_s(q, D, mm);
        if (J.mode == 1 && (jl & 1)) o += t;
        else e += t;
      }
    }
  }
  red[warp][lane][0] = e;
  red[warp][lane][1] = o;
  __syncthreads();
  double E = 0.0, O = 0.0;
  if (warp == 0) {
#pragma unroll
    for (int w = 0; w < kXWarps; ++w) {
      E += red[w][lane][0];
      O += red[w][lane][1];
    }
  }
  if (J.nchunk > 1) {
    double* pp = J.part + ((long long)(line * J.ntile + tile) * J.nchunk) * 64;
    if (warp == 0) {
      pp[chunk_id * 64 + 2 * lane] = E;
      pp[chunk_id * 64 + 2 * lane + 1] = O;
    }
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
      unsigned int* c = J.cnt + (line * J.ntile + tile);
      const unsigned int t = atomicAdd(c, 1u);
      amlast = (t == (unsigned int)J.nchunk - 1);
      if (amlast) *c = 0u;
    }
    __syncthreads();
    if (!amlast) return;
    if (warp == 0) {
      E = 0.0;
      O = 0.0;
      for (int c = 0; c < J.nchunk; ++c) {
        E += __ldcg(pp + c * 64 + 2 * lane);
        O += __ldcg(pp + c * 64 + 2 * lane + 1);
      }
    }
  }
  if (warp != 0 || !lane_on) return;
  const double g = J.gscale;
  auto scale = [&](int kq) { return (kq == 0) ? J.s0 : ((kq == J.N - 1) ? J.sl : J.sm); };
  auto active = [&](int kq) { return kq >= J.klo && kq < J.khi; };
  double* out = J.out + (long long)line * J.out_sl;
  if (J.mode == 1) {
    const bool is_sin = (J.off != 0);
    const double yk = E + O;
    const double yr = is_sin ? (O - E) : (E - O);
    if (k < J.nout) {
      const double v = active(k) ? yk * scale(k) * g : 0.0;
      out[(long long)k * J.out_sk] = v;
      if (J.epi) acc_epilogue(b.acc, (long long)line * J.out_sl + (long long)k * J.out_sk, v);
    }
    const int kr = D - k;
    if (kr != k && kr < J.nout) {
      const double v = active(kr) ? yr * scale(kr) * g : 0.0;
      out[(long long)kr * J.out_sk] = v;
      if (J.epi) acc_epilogue(b.acc, (long long)line * J.out_sl + (long long)kr * J.out_sk, v);
    }
  } else {
    if (k < J.nout) {
      const double v = active(k) ? E * scale(k) * g : 0.0;
      out[(long long)k * J.out_sk] = v;
      if (J.epi) acc_epilogue(b.acc, (long long)line * J.out_sl + (long long)k * J.out_sk, v);
    }
  }
}

constexpr int kYThreads = 64;
constexpr int kYR = 8;  // outputs per thread, or 4 or 2

// y pass: one thread = one line (consecutive lines are contiguous in memory)
// and R lane outputs; twiddles are warp-uniform.  The two symmetries of
// the x pass halve the FP64 work of REDFT00 / RODFT00 kinds:
//   mode 1: lane output k (k <= D/2) keeps even-j and odd-j sums E, O and
//           writes out[k] and out[D-k]
//   mode 2: inputs are paired, u = x_j + x_{D-j}, v = x_j - x_{D-j}
//           (outputs k <= D/2)
// The FP64 pipe bounds it: a warp's multiply-add takes its scheduler 64 cycles, so
// eight outputs over 72 terms are 18 us for a warp however few there are.  Where
// that is the longer part (lanes_line_outputs) a thread takes four or two outputs,
// and the loads of four pairs of terms are in flight (x and y pass of eight fields
// of 514 x 72 points 79 -> 44 us, of one field 37 -> 22 us).
// R consecutive twiddles of a y row (rows are 64-byte aligned)
template <int R>
__device__ __forceinline__ void twiddle_row(const double* __restrict__ p, double (&t)[R]) {
  const double2* q = reinterpret_cast<const double2*>(p);
#pragma unroll
  for (int i = 0; i < R / 2; ++i) {
    const double2 v = __ldg(q + i);
    t[2 * i] = v.x;
    t[2 * i + 1] = v.y;
  }
}

template <int NJ, int R>
__global__ void __launch_bounds__(kYThreads) axis_pass_lanes_line(const AxisBatchT<NJ> b) {
  pdl_wait();
  int jb = 0;
  while (jb + 1 < b.njobs && (int)blockIdx.x >= b.start[jb + 1]) ++jb;
  const AxisJob& J = b.job[jb];
  const int local = blockIdx.x - b.start[jb];
  const int nlb = (J.nlines + kYThreads - 1) / kYThreads;
  const int kgrp = local / nlb;
  const int lb = local - kgrp * nlb;
  const int line = lb * kYThreads + threadIdx.x;
  if (line >= J.nlines) return;
  const int k0 = kgrp * R;
  const int D = J.D, D4 = 4 * D;
  const double* __restrict__ x = J.in + (long long)line * J.in_sl;
  const long long sk = J.in_sk;
  // input weights (a y pass that runs first reads them along y)
  const double* __restrict__ wr = J.win ? J.win + (long long)line * J.win_sl : nullptr;
  auto X = [&](int j) { return in_at(x, sk, wr, J.win_sk, j); };
  const int j_end = min(J.jhi, J.nin);
  const bool is_sin = (J.off != 0);
  double* out = J.out + (long long)line * J.out_sl;
  auto put = [&](int k, double v) {
    if (k >= J.nout) return;
    const bool active = (k >= J.klo) && (k < J.khi);
    const double sc = (k == 0) ? J.s0 : ((k == J.N - 1) ? J.sl : J.sm);
    const double y = active ? v * sc * J.gscale : 0.0;
    out[(long long)k * J.out_sk] = y;
    if (J.epi) acc_epilogue(b.acc, (long long)line * J.out_sl + (long long)k * J.out_sk, y);
  };
  auto step = [&](int& m, int inc) {
    m += inc;
    if (m >= D4) m -= D4;
  };
  int m[R], inc[R];
  const int a0 = max(J.jlo, 1);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int kk = J.ak * (k0 + r) + J.bk;
    inc[r] = mod4d((long long)J.aj * kk, D4);
    m[r] = mod4d((long long)(J.aj * a0 + J.bj) * kk + J.off, D4);
  }
  if (J.mode == 1 && J.ty) {
    // twiddle rows: row j, columns k0 .. k0 + R - 1
    const double* __restrict__ T = J.ty + k0;
    const long long ld = J.ldy;
    double E[R], O[R], t[R];
#pragma unroll
    for (int r = 0; r < R; ++r) E[r] = O[r] = 0.0;
    const int a1 = min(j_end, J.N - 1);
    int j = a0;
    if (j < a1 && (j & 1)) {
      const double v = X(j);
      twiddle_row<R>(T + j * ld, t);
#pragma unroll
      for (int r = 0; r < R; ++r) O[r] = fma(v, t[r], O[r]);
      ++j;
    }
#pragma unroll(R < kYR ? 4 : 1)
    for (; j + 1 < a1; j += 2) {
      const double v0 = X(j), v1 = X(j + 1);
      double t1[R];
      twiddle_row<R>(T + j * ld, t);
      twiddle_row<R>(T + (j + 1) * ld, t1);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        E[r] = fma(v0, t[r], E[r]);
        O[r] = fma(v1, t1[r], O[r]);
      }
    }
    if (j < a1) {
      const double v = X(j);
      twiddle_row<R>(T + j * ld, t);
#pragma unroll
      for (int r = 0; r < R; ++r) E[r] = fma(v, t[r], E[r]);
    }
    double t0[R], tD[R];
    twiddle_row<R>(T, t0);
    twiddle_row<R>(T + D * ld, tD);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int k = k0 + r;
      if (k >= J.nlane) break;
      double e = J.wm * E[r], o = J.wm * O[r];
      if (J.jlo == 0 && 0 < j_end) e = fma(J.w0 * X(0), t0[r], e);
      if (D >= J.jlo && D < j_end) {
        const double tt = J.wl * X(D) * tD[r];
        if (D & 1) o += tt;
        else e += tt;
      }
      put(k, e + o);
      if (D - k != k) put(D - k, is_sin ? o - e : e - o);
    }
  } else if (J.mode == 2 && J.ty) {
    const double* __restrict__ T = J.ty + k0;
    const long long ld = J.ldy;
    double acc[R], t[R];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = 0.0;
    const int pe = (D + 1) / 2;  // interior pairs j < D - j
#pragma unroll(R < kYR ? 4 : 1)
    for (int j = 1; j < pe; ++j) {
      const double xa = X(j), xb = X(D - j);
      const double u = xa + xb, v = xa - xb;
      twiddle_row<R>(T + j * ld, t);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const bool use_v = (((k0 + r) & 1) == 0) != !is_sin;
        acc[r] = fma(use_v ? v : u, t[r], acc[r]);
      }
    }
    double t0[R], tm[R];
    twiddle_row<R>(T, t0);
    twiddle_row<R>(T + (D / 2) * ld, tm);
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int k = k0 + r;
      if (k >= J.nlane) break;
      double tt = J.wm * acc[r];
      if (J.jlo == 0) {
        const double xa = X(0), xb = X(D);
        tt = fma(J.w0 * (((k & 1) == 0) ? xa + xb : xa - xb), t0[r], tt);
      }
      if ((D & 1) == 0) {
        const int jm = D / 2;
        if (jm >= J.jlo && jm < J.jhi) tt = fma(J.wm * X(jm), tm[r], tt);
      }
      put(k, tt);
    }
  } else if (J.mode == 1) {
    double E[R], O[R];
#pragma unroll
    for (int r = 0; r < R; ++r) E[r] = O[r] = 0.0;
    const int a1 = min(j_end, J.N - 1);
    int j = a0;
    if (j < a1 && (j & 1)) {
      const double v = X(j);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        O[r] = fma(v, twiddle(J.q, D, m[r]), O[r]);
        step(m[r], inc[r]);
      }
      ++j;
    }
    for (; j + 1 < a1; j += 2) {
      const double v0 = X(j), v1 = X(j + 1);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        E[r] = fma(v0, twiddle(J.q, D, m[r]), E[r]);
        step(m[r], inc[r]);
        O[r] = fma(v1, twiddle(J.q, D, m[r]), O[r]);
        step(m[r], inc[r]);
      }
    }
    if (j < a1) {
      const double v = X(j);
#pragma unroll
      for (int r = 0; r < R; ++r) E[r] = fma(v, twiddle(J.q, D, m[r]), E[r]);
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int k = k0 + r;
      if (k >= J.nlane) break;
      double e = J.wm * E[r], o = J.wm * O[r];
      if (J.jlo == 0 && 0 < j_end) e = fma(J.w0 * X(0), twiddle(J.q, D, mod4d(J.off, D4)), e);
      if (D >= J.jlo && D < j_end) {
        const double t = J.wl * X(D) *
                         twiddle(J.q, D, mod4d((long long)2 * D * k + J.off, D4));
        if (D & 1) o += t;
        else e += t;
      }
      put(k, e + o);
      if (D - k != k) put(D - k, is_sin ? o - e : e - o);
    }
  } else if (J.mode == 2) {
    double acc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = 0.0;
    // cos: even k pairs with u; sin: even k pairs with v
    const int pe = (D + 1) / 2;  // interior pairs j < D - j
    for (int j = 1; j < pe; ++j) {
      const double xa = X(j), xb = X(D - j);
      const double u = xa + xb, v = xa - xb;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const bool use_v = (((k0 + r) & 1) == 0) != !is_sin;
        acc[r] = fma(use_v ? v : u, twiddle(J.q, D, m[r]), acc[r]);
        step(m[r], inc[r]);
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int k = k0 + r;
      if (k >= J.nlane) break;
      double t = J.wm * acc[r];
      if (J.jlo == 0) {  // the end pair (0, D) with the end weight
        const double xa = X(0), xb = X(D);
        t = fma(J.w0 * (((k & 1) == 0) ? xa + xb : xa - xb), twiddle(J.q, D, mod4d(J.off, D4)), t);
      }
      if ((D & 1) == 0) {
        const int jm = D / 2;
        if (jm >= J.jlo && jm < J.jhi)
          t = fma(J.wm * X(jm),
                  twiddle(J.q, D, mod4d((long long)2 * jm * k + J.off, D4)), t);
      }
      put(k, t);
    }
  } else {
    double acc[R];
#pragma unroll
    for (int r = 0; r < R; ++r) acc[r] = 0.0;
    const int a1 = min(j_end, J.N - 1);
    for (int j = a0; j < a1; ++j) {
      const double v = X(j);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        acc[r] = fma(v, twiddle(J.q, D, m[r]), acc[r]);
        step(m[r], inc[r]);
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int k = k0 + r;
      if (k >= J.nout) break;
      double t = J.wm * acc[r];
      const int kk = J.ak * k + J.bk;
      if (J.jlo == 0 && 0 < j_end) {
        const int mm = mod4d((long long)J.bj * kk + J.off, D4);
        t = fma(J.w0 * X(0), twiddle(J.q, D, mm), t);
      }
      const int jl = J.N - 1;
      if (jl > 0 && jl >= J.jlo && jl < j_end) {
        const int mm = mod4d((long long)(J.aj * jl + J.bj) * kk + J.off, D4);
        t = fma(J.wl * X(jl), twiddle(J.q, D, mm), t);
      }
      put(k, t);
    }
  }
}

// y pass of few lines (the wavemaker grids of narrow 3-D tanks): CTA = (job, 32
// lines, two lane outputs), lane = line, the 8 warps split the inputs, so that a
// warp's inputs have one parity and the sums E, O of mode 1 are sums over warps.
// One thread per line with eight outputs left this to two CTAs of one warp: 20 us
// for 30 lines of 32 points, 3.4 us here.
constexpr int kFewLines = 32;
template <int NJ>
__global__ void __launch_bounds__(256) axis_pass_few_lines(const AxisBatchT<NJ> b) {
  __shared__ double red[2][8][32];
  int jb = 0;
  while (jb + 1 < b.njobs && (int)blockIdx.x >= b.start[jb + 1]) ++jb;
  const AxisJob& J = b.job[jb];
  const int D = J.D, D4 = 4 * D;
  const bool paired = J.mode == 1;
  const int ngrp = (J.nlane + 1) / 2;
  const int local = blockIdx.x - b.start[jb];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int k0 = 2 * (local % ngrp), line = (local / ngrp) * 32 + lane;
  const bool on = line < J.nlines;
  const double* __restrict__ x = J.in + (long long)(on ? line : 0) * J.in_sl;
  const double* __restrict__ wr = J.win ? J.win + (long long)(on ? line : 0) * J.win_sl : nullptr;
  const int jlo = J.jlo, j_end = min(J.jhi, J.nin);
  const bool is_sin = J.off != 0;
  int m[2], inc[2];
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    m[r] = mod4d(2LL * (jlo + warp) * (k0 + r) + J.off, D4);
    inc[r] = mod4d(16LL * (k0 + r), D4);
  }
  pdl_wait();
  double acc[2] = {0.0, 0.0};
  if (on) {
#pragma unroll 4
    for (int j = jlo + warp; j < j_end; j += 8) {
      double v = in_at(x, J.in_sk, wr, J.win_sk, j);
      // end inputs count full or half of an interior one
      if ((j == 0 && J.w0 != J.wm) || (j == J.N - 1 && J.wl != J.wm)) v *= 0.5;
#pragma unroll
      for (int r = 0; r < 2; ++r) {
        acc[r] = fma(v, twiddle(J.q, D, m[r]), acc[r]);
        m[r] += inc[r];
        if (m[r] >= D4) m[r] -= D4;
      }
    }
  }
  red[0][warp][lane] = acc[0];
  red[1][warp][lane] = acc[1];
  __syncthreads();
  if (warp >= 2 || !on) return;
  const int k = k0 + warp;
  if (k >= J.nlane) return;
  double s[2] = {0.0, 0.0};  // over the warps of even and of odd inputs
#pragma unroll
  for (int w = 0; w < 8; w += 2) {
    s[0] += red[warp][w][lane];
    s[1] += red[warp][w + 1][lane];
  }
  const double e = (jlo & 1) ? s[1] : s[0], o = (jlo & 1) ? s[0] : s[1];
  auto put = [&](int kk, double v) {
    if (kk >= J.nout) return;
    const double sc = ((kk == 0) ? J.s0 : ((kk == J.N - 1) ? J.sl : J.sm)) * J.gscale * J.wm;
    const double y = (kk >= J.klo && kk < J.khi) ? v * sc : 0.0;
    const long long at = (long long)line * J.out_sl + (long long)kk * J.out_sk;
    J.out[at] = y;
    if (J.epi) acc_epilogue(b.acc, at, y);
  };
  put(k, e + o);
  if (paired && D - k != k) put(D - k, is_sin ? o - e : e - o);
}

// scale of output k; w: the interior weight, where pass 1 left it out
__device__ __forceinline__ double p2_scale(const AxisJob& J, int k, double w) {
  return ((k == 0) ? J.s0 : ((k == J.N - 1) ? J.sl : J.sm)) * J.gscale * w;
}
__device__ __forceinline__ void p2_put(const AxisJob& J, const AccEpi& acc, int line, int k, double y, double scale) {
  if (k >= J.nout) return;
  const bool on = k >= J.klo && k < J.khi;
  const long long e = (long long)line * J.out_sl + (long long)k * J.out_sk;
  const double v = on ? y * scale : 0.0;
  J.out[e] = v;
  if (J.epi) acc_epilogue(acc, e, v);
}

// x or -x by the sign bit
__device__ __forceinline__ double flip_if(double x, bool neg) {
  return __hiloint2double(__double2hiint(x) ^ (neg ? (int)0x80000000 : 0), __double2loint(x));
}

// Direct x pass of few lines (lengths that do not factor, 2-D tanks): CTA = (job,
// line, KO lane outputs); a warp holds KO outputs times 32 / KO slices of the sum,
// warp w the slices w, w + 4, ..., which meet by shuffles and in shared memory.  The
// quarter-wave table is staged before the wait for the previous kernel, and no
// FP64 operation but the FMAs of the sums is in the loop: a warp's holds its
// scheduler for 64 cycles, under which the index arithmetic of the next twiddle
// is free (a staged tile of the CTA's twiddles cost 40 instructions each, and an
// ensemble of six tanks 15 %).  With mode 1 a slice's inputs have one parity (an even
// number of slices): the sums E, O of the k <-> D - k pairs; with mode 2 (every
// input, truncated outputs) the slices run over u = x_j + x_{D-j} or v = x_j -
// x_{D-j}.  D = 257, one line: 5.8 us by axis_pass_lanes_k (9 CTAs), 3.6 us here.
constexpr int kDirThreads = 128;
constexpr int kDirMaxD = 4200;      // table and inputs within 68 KB: three CTAs per SM
constexpr int kDirMaxLines = 8;     // more lines fill the SMs by axis_pass_lanes_k
__host__ __device__ inline int dir_terms(const AxisJob& J) {  // lane terms of the sum
  return J.mode == 2 ? J.D / 2 + 1 : (J.jhi < J.nin ? J.jhi : J.nin);
}
template <int NJ, int KO>
__global__ void __launch_bounds__(kDirThreads) direct_pass(const AxisBatchT<NJ> b) {
  extern __shared__ double smd[];
  __shared__ double red[4][KO];
  constexpr int SL = 4 * (32 / KO);
  int jb = 0;
  while (jb + 1 < b.njobs && (int)blockIdx.x >= b.start[jb + 1]) ++jb;
  const AxisJob& J = b.job[jb];
  const int D = J.D, D4 = 4 * D, mode = J.mode;
  const int nkb = (J.nlane + KO - 1) / KO;
  const int local = blockIdx.x - b.start[jb];
  const int line = local / nkb, k0 = (local - line * nkb) * KO;
  const int jlo = J.jlo, j_end = min(J.jhi, J.nin), nt = dir_terms(J);
  const bool is_sin = J.off != 0;
  double* tq = smd;             // cos(pi m / (2 D)), m = 0 .. D
  double* xs = smd + D + 1;     // inputs, or u then v
  const double* __restrict__ q = J.q;
  auto stage_twiddles = [&]() {
    for (int t = threadIdx.x; t <= D; t += kDirThreads) tq[t] = __ldg(q + t);
  };
  if (b.early) stage_twiddles();
  const double* __restrict__ x = J.in + (long long)line * J.in_sl;
  const double* __restrict__ wr = J.win ? J.win + (long long)line * J.win_sl : nullptr;
  const bool half0 = J.w0 != J.wm, halfD = J.wl != J.wm;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int kl = lane % KO, slice = warp + 4 * (lane / KO);
  const int k = k0 + kl;
  const double sk = p2_scale(J, k, J.wm), sm = p2_scale(J, D - k, J.wm);
  const long long in_sk = J.in_sk, win_sk = J.win_sk;
  pdl_wait();
  if (!b.early) stage_twiddles();
  auto u = [&](int j) -> double {
    if (j < jlo || j >= j_end) return 0.0;
    double v = in_at(x, in_sk, wr, win_sk, j);
    if ((j == 0 && half0) || (j == D && halfD)) v *= 0.5;
    return v;
  };
  for (int j = threadIdx.x; j < nt; j += kDirThreads) {
    const double v = u(j);
    if (mode == 2) {
      const bool mid = 2 * j == D;
      const double m = mid ? 0.0 : u(D - j);
      xs[j] = v + m;
      xs[nt + j] = v - m;
    } else {
      xs[j] = v;
    }
  }
  __syncthreads();
  // cos: even k sees u, odd k sees v; sin the other way round
  const double* xp = xs + (mode == 2 && (((k & 1) == 0) == is_sin) ? nt : 0);
  int m = mod4d(2LL * slice * k + J.off, D4);
  const int inc = mod4d(2LL * SL * k, D4);
  auto next = [&]() -> double {
    const int mm = m > 2 * D ? D4 - m : m;
    const bool neg = mm > D;
    m += inc;
    if (m >= D4) m -= D4;
    return flip_if(tq[neg ? 2 * D - mm : mm], neg);
  };
  double acc = 0.0, acc2 = 0.0;  // two chains
  int j = slice;
#pragma unroll 2
  for (; j + SL < nt; j += 2 * SL) {
    acc = fma(xp[j], next(), acc);
    acc2 = fma(xp[j + SL], next(), acc2);
  }
  if (j < nt) acc = fma(xp[j], next(), acc);
  acc += acc2;
#pragma unroll
  for (int off = KO; off < 32; off <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if (lane < KO) red[warp][lane] = acc;
  __syncthreads();
  if (threadIdx.x < KO && k < J.nlane) {
    const double e = red[0][lane] + red[2][lane], o = red[1][lane] + red[3][lane];
    p2_put(J, b.acc, line, k, e + o, sk);
    if (mode == 1 && D - k != k) p2_put(J, b.acc, line, D - k, is_sin ? o - e : e - o, sm);
  }
}

// Two-level passes for REDFT00 / RODFT00 kinds when D = A * B.  With
// j = B j1 + j2, pi j k / D = pi j1 k / A + pi j2 k / D, so
//   cos-kind: y_k = sum_j2 [cos(pi j2 k/D) C(j2,k) - sin(pi j2 k/D) S(j2,k)]
//   sin-kind: y_k = sum_j2 [cos(pi j2 k/D) S(j2,k) + sin(pi j2 k/D) C(j2,k)]
// with C, S = sum_j1 w_j x_j cos / sin(pi j1 k / A), which depend on k only
// through k mod 2A (C even, S odd about A).  Pass 1 computes C, S for
// k' = 0..A; pass 2 combines them.  Work: about (A+2) nin + 2 B nout FMAs
// (B nout when outputs pair up, see pass 2) instead of about nin * nout / 2
// for the direct sum.
//
// Both passes first issue all of their global loads (inputs, partial sums
// and twiddles staged in shared memory), then run FMA loops over shared
// memory: one round trip to L2 per pass instead of a chain of dependent
// scattered loads.
//
// What bounds them on GB300 is FP64 issue: a warp's FP64 instruction holds its
// scheduler's pipe for 64 cycles, whatever the warps beside it do, so a pass over
// one line (150k to 250k FMAs, about 6000 warp instructions) takes under a
// microsecond only when it lies on most of the 608 schedulers.  So both passes cut
// their sums into parts until the CTAs cover the SMs, keep every FP64 operation that
// is not an FMA of the sum out of the loops (weights and signs by exponent and
// sign bits, scales in one product per output), and add the parts up by
// shuffles.  One line of D = 3074: pass 1 9.5 us -> 4.9, pass 2 5.0 -> 4.0 in the step of
// the irregular 2-D tank, where the former split used 54 and 33 CTAs.
constexpr int kP1Threads = 128;
constexpr int kP2Threads = 128;
constexpr int kP2Warps = kP2Threads / 32;

__host__ __device__ inline int p1_half(int A) { return A / 2; }
// Pass 1: a CTA takes nk values of k' <= A/2 times G of j2, every sum over j1 in
// P parts.
struct P1Shape {
  int nk, G, kblocks, jblocks;
};
__host__ __device__ inline P1Shape p1_shape(int A, int B, int P) {
  P1Shape s;
  const int items = kP1Threads / P;
  s.nk = p1_half(A) + 1 < items ? p1_half(A) + 1 : items;
  s.G = items / s.nk;
  if (s.G > B) s.G = B;
  s.kblocks = (p1_half(A) + s.nk) / s.nk;
  s.jblocks = (B + s.G - 1) / s.G;
  return s;
}

// pass 1: CTA = (job, line, nk values of k', G values of j2).  The even and odd
// j1 terms are summed apart: cos / sin(pi j1 (A - k') / A) = +-(-1)^j1 cos /
// sin(pi j1 k' / A), so the same four sums give C, S at k' and at A - k' and
// half of the k' are computed.  Threads own (k', j2, part) with k' fastest:
// inputs are broadcast, twiddles gathered from the 2 A pairs cos, sin(pi m / A).  The inputs
// enter with the interior weight 1; pass 2 multiplies the outputs by it.  STAGED:
// the pairs lie in shared memory; a longer table (A > 5119, so D > 20475 as B is
// 4 or more) is read from the quarter-wave table in global memory.
template <int NJ, bool STAGED>
__global__ void __launch_bounds__(kP1Threads) two_level_pass1(const AxisBatchT<NJ> b, int P) {
  extern __shared__ double sm1[];
  __shared__ double red[4 * kP1Threads];
  int jb = 0;
  while (jb + 1 < b.njobs && (int)blockIdx.x >= b.start[jb + 1]) ++jb;
  const AxisJob& J = b.job[jb];
  const int A = J.A, B = J.B, D = J.D, H = p1_half(A);
  const int j_end = min(J.jhi, J.nin), jlo = J.jlo;  // terms j in [jlo, j_end)
  const int K = (j_end + B - 1) / B, Kp = (K + 1) & ~1;
  const P1Shape sh = p1_shape(A, B, P);
  int local = blockIdx.x - b.start[jb];
  const int kb = local % sh.kblocks;
  local /= sh.kblocks;
  const int j20 = (local % sh.jblocks) * sh.G, line = local / sh.jblocks;
  const int kp0 = kb * sh.nk, nk = min(sh.nk, H + 1 - kp0), G = min(sh.G, B - j20);
  double2* tw = reinterpret_cast<double2*>(sm1);                    // cos, sin(pi m / A), m < 2 A
  double* xs = sm1 + (STAGED ? 4 * (size_t)A : 0);                  // [j1][j2] inputs, zero outside the sum
  const double* __restrict__ x = J.in + (long long)line * J.in_sl;
  const double* __restrict__ wr = J.win ? J.win + (long long)line * J.win_sl : nullptr;
  const double* __restrict__ q = J.q;
  auto pair_of = [&](int t) -> double2 {
    const int m = 2 * B * t;  // pi t / A = pi m / (2 D), m < 4 D
    return make_double2(twiddle(q, D, m), twiddle(q, D, m >= D ? m - D : m + 3 * D));
  };
  auto stage_twiddles = [&]() {
    if constexpr (STAGED)
      for (int t = threadIdx.x; t < 2 * A; t += kP1Threads) tw[t] = pair_of(t);
  };
  if (b.early) stage_twiddles();
  const bool half0 = J.w0 != J.wm, halfD = J.wl != J.wm;
  const int N = J.N;
  const long long in_sk = J.in_sk, win_sk = J.win_sk;
  pdl_wait();
  if (!b.early) stage_twiddles();
  for (int t = threadIdx.x; t < Kp * G; t += kP1Threads) {
    const int j1 = t / G, j = j1 * B + j20 + (t - j1 * G);
    double v = 0.0;
    if (j1 < K && j >= jlo && j < j_end) {
      v = in_at(x, in_sk, wr, win_sk, j);
      if ((j == 0 && half0) || (j == N - 1 && halfD)) v *= 0.5;
    }
    xs[t] = v;
  }
  __syncthreads();
  const int items = nk * G;
  const int r = threadIdx.x / nk, kpl = threadIdx.x - r * nk;
  const int part = r / G, j2l = r - part * G;
  double ce = 0.0, se = 0.0, co = 0.0, so = 0.0;
  if (part < P) {
    const int A2 = 2 * A, kp = kp0 + kpl;
    int m = (2 * part * kp) % A2;
    const int inc = (2 * P * kp) % A2;
#pragma unroll 4
    for (int p = part; p < Kp / 2; p += P) {
      const double v0 = xs[2 * p * G + j2l], v1 = xs[(2 * p + 1) * G + j2l];
      const int m1 = m + kp >= A2 ? m + kp - A2 : m + kp;
      const double2 t0 = STAGED ? tw[m] : pair_of(m), t1 = STAGED ? tw[m1] : pair_of(m1);
      m += inc;
      if (m >= A2) m -= A2;
      ce = fma(v0, t0.x, ce);
      se = fma(v0, t0.y, se);
      co = fma(v1, t1.x, co);
      so = fma(v1, t1.y, so);
    }
    double* rp = red + part * 4 * items + 4 * (j2l * nk + kpl);
    rp[0] = ce;
    rp[1] = se;
    rp[2] = co;
    rp[3] = so;
  }
  __syncthreads();
  // the parts' sums: R threads per value, then the folds between values v and
  // v ^ 2 of an item, by shuffles
  const int R = P >= 16 ? 4 : (P >= 8 ? 2 : 1);
  double* cs = J.cs + ((long long)line * B + j20) * (A + 1) * 2;
  for (int t0 = 0; t0 < 4 * items * R; t0 += kP1Threads) {
    const int t = t0 + threadIdx.x, iv = t / R;
    const bool on = iv < 4 * items;
    double f = 0.0;
    if (on) {
      f = red[(t % R) * 4 * items + iv];
      for (int p = t % R + R; p < P; p += R) f += red[p * 4 * items + iv];
    }
    if (R > 1) f += __shfl_xor_sync(0xffffffffu, f, 1);
    if (R > 2) f += __shfl_xor_sync(0xffffffffu, f, 2);
    const double o = __shfl_xor_sync(0xffffffffu, f, 2 * R);
    const int v = iv & 3;
    // C(k') = ce + co, S(k') = se + so, C(A - k') = ce - co, S(A - k') = so - se
    const double y = flip_if(f, v == 2) + flip_if(o, v == 3);
    if (on && t % R == 0) {
      const int it = iv >> 2, kp = kp0 + it % nk;
      double* c = cs + (long long)(it / nk) * (A + 1) * 2;
      if (v < 2) c[2 * kp + v] = y;
      else if (A - kp != kp) c[2 * (A - kp) + v - 2] = y;
    }
  }
}

// cos(pi m / (2 D)) from the staged quarter-wave table, negated where neg
__device__ __forceinline__ double twiddle_flip(const double* q, int D, int m, bool neg) {
  const int mm = m > 2 * D ? 4 * D - m : m;
  const bool second = mm > D;
  return flip_if(q[second ? 2 * D - mm : mm], second != neg);
}

// Paired jobs (mode 1: B even, every output wanted): with B even, (-1)^j =
// (-1)^j2, so y(D - k) = +-sum_j2 (-1)^j2 T_j2(k) for the terms T_j2(k) of
// y(k).  Lanes own k <= D/2, and the sums E, O over even and odd j2 give y(k)
// = E + O and y(D - k) = E - O (cos kind) or O - E (sin kind).
__host__ __device__ inline int p2_lanes(const AxisJob& J) { return J.mode == 1 ? J.D / 2 + 1 : J.nout; }

// pass 2: CTA = (job, line, KO outputs).  A warp holds KO outputs times 32 / KO
// slices of the j2 sum, warp w the slices w, w + 4, ...: every slice of a warp
// has the parity of w (paired jobs), its slices meet by shuffles and the four
// warps in shared memory.
template <int NJ, int KO>
__global__ void __launch_bounds__(kP2Threads) two_level_pass2(const AxisBatchT<NJ> b) {
  extern __shared__ double sm2[];
  __shared__ double red[kP2Warps][KO];
  constexpr int SL = kP2Warps * (32 / KO);
  int jb = 0;
  while (jb + 1 < b.njobs && (int)blockIdx.x >= b.start[jb + 1]) ++jb;
  const AxisJob& J = b.job[jb];
  const int A = J.A, B = J.B, D = J.D, D4 = 4 * D;
  const bool paired = J.mode == 1;
  const int nlane = p2_lanes(J);
  const int nkb = (nlane + KO - 1) / KO;
  const int local = blockIdx.x - b.start[jb];
  const int line = local / nkb;
  const int k0 = (local - line * nkb) * KO;
  const double* __restrict__ q = J.q;
  // the quarter-wave table: its gathers and their index arithmetic run under
  // the FP64 operations (a staged tile of twiddles cost 70 instructions a pair)
  auto stage_twiddles = [&]() {
    for (int t = threadIdx.x; t <= D; t += kP2Threads) sm2[t] = __ldg(q + t);
  };
  if (b.early) stage_twiddles();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int kl = lane % KO, slice = warp + kP2Warps * (lane / KO);
  const int k = k0 + kl;
  const bool on = paired ? k < nlane : (k < J.nout && k >= J.klo && k < J.khi);
  int kp = k % (2 * A);
  const bool sneg = kp > A;
  if (sneg) kp = 2 * A - kp;
  const bool is_sin = (J.off != 0);
  const double2* cs = reinterpret_cast<const double2*>(J.cs) + (long long)line * B * (A + 1) + kp;
  const double sck = p2_scale(J, k, J.wm), scm = p2_scale(J, D - k, J.wm);
  pdl_wait();
  if (!b.early) stage_twiddles();
  // cos kind: cw C - sw S; sin kind: sw C + cw S (S with the sign of its fold)
  const bool neg = sneg != !is_sin;
  constexpr int kOwn = 8;  // terms in flight
  double acc = 0.0, acc2 = 0.0;
  // j2 < D and k < N, so 2 j2 k fits in 32 bits for N < 32768
  int m = (int)((2u * (unsigned)slice * (unsigned)k) % (unsigned)D4);
  const int inc = (int)((2u * (unsigned)SL * (unsigned)k) % (unsigned)D4);
  double2 v[kOwn];
  auto load = [&](int j2) {
#pragma unroll
    for (int i = 0; i < kOwn; ++i)
      if (on && j2 + i * SL < B) v[i] = __ldcg(cs + (long long)(j2 + i * SL) * (A + 1));
  };
  load(slice);
  __syncthreads();
  for (int j2 = slice; j2 < B; j2 += kOwn * SL) {
    if (j2 != slice) load(j2);
#pragma unroll
    for (int i = 0; i < kOwn; ++i) {
      if (on && j2 + i * SL < B) {
        // cos(pi j2 k / D) at m, sin at m - D
        const int ms = m >= D ? m - D : m + 3 * D;
        const double t = twiddle_flip(sm2, D, is_sin ? ms : m, false);
        const double f = twiddle_flip(sm2, D, is_sin ? m : ms, neg);
        acc = fma(t, v[i].x, acc);
        acc2 = fma(f, v[i].y, acc2);
        m += inc;
        if (m >= D4) m -= D4;
      }
    }
  }
  acc += acc2;
#pragma unroll
  for (int off = KO; off < 32; off <<= 1) acc += __shfl_xor_sync(0xffffffffu, acc, off);
  if (lane < KO) red[warp][lane] = acc;
  __syncthreads();
  if (threadIdx.x < KO) {
    const double e = red[0][lane] + red[2][lane], o = red[1][lane] + red[3][lane];
    if (paired) {
      if (k < nlane) {
        p2_put(J, b.acc, line, k, e + o, sck);
        if (D - k != k) p2_put(J, b.acc, line, D - k, is_sin ? o - e : e - o, scm);
      }
    } else if (k < J.nout) {
      p2_put(J, b.acc, line, k, on ? e + o : 0.0, sck);
    }
  }
}

// pass 2 for lengths whose quarter-wave table is over the shared memory:
// CTA = (job, 32 outputs, group of lpc lines).  The B x 32 twiddle tile is
// staged once for the group; each warp takes lines in turn and sums all of
// their j2 terms, so no cross-warp reduction is needed.
template <int NJ>
__global__ void __launch_bounds__(kP2Threads) two_level_pass2_lines(const AxisBatchT<NJ> b, int lpc) {
  extern __shared__ double sm2[];
  int jb = 0;
  while (jb + 1 < b.njobs && (int)blockIdx.x >= b.start[jb + 1]) ++jb;
  const AxisJob& J = b.job[jb];
  const int A = J.A, B = J.B, D = J.D, D4 = 4 * D;
  const bool paired = J.mode == 1;
  const int nlane = p2_lanes(J);
  const int nkb = (nlane + 31) / 32;
  const int local = blockIdx.x - b.start[jb];
  const int kb = local % nkb;
  const int l0 = (local / nkb) * lpc;
  const int k0 = kb * 32;
  auto stage_twiddles = [&]() {
    for (int t = threadIdx.x; t < B * 32; t += kP2Threads) {
      const int j2 = t >> 5, k = k0 + (t & 31);
      const int m = (int)((2u * (unsigned)j2 * (unsigned)k) % (unsigned)D4);
      sm2[2 * t] = twiddle(J.q, D, m);
      sm2[2 * t + 1] = twiddle(J.q, D, m >= D ? m - D : m + 3 * D);
    }
  };
  if (b.early) stage_twiddles();
  pdl_wait();
  if (!b.early) stage_twiddles();
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int k = k0 + lane;
  const bool on = paired ? k < nlane : (k < J.nout && k >= J.klo && k < J.khi);
  int kp = k % (2 * A);
  double ssign = 1.0;
  if (kp > A) {
    kp = 2 * A - kp;
    ssign = -1.0;
  }
  const bool is_sin = (J.off != 0);
  const double2* tw = reinterpret_cast<const double2*>(sm2) + lane;
  const int l1 = min(J.nlines, l0 + lpc);
  for (int line = l0 + warp; line < l1; line += kP2Warps) {
    const double* cs = J.cs + ((long long)line * B * (A + 1) + kp) * 2;
    double ae = 0.0, ao = 0.0;  // even, odd j2 (paired jobs; else all in ae)
    if (on) {
#pragma unroll 4
      for (int j2 = 0; j2 < B; ++j2) {
        const long long o = (long long)j2 * (A + 1) * 2;
        const double C = __ldcg(cs + o), S = ssign * __ldcg(cs + o + 1);
        const double2 t = tw[j2 * 32];
        if (paired && (j2 & 1)) {  // j2 is warp-uniform
          if (is_sin) ao = fma(t.x, S, fma(t.y, C, ao));
          else ao = fma(t.x, C, fma(-t.y, S, ao));
        } else {
          if (is_sin) ae = fma(t.x, S, fma(t.y, C, ae));
          else ae = fma(t.x, C, fma(-t.y, S, ae));
        }
      }
    }
    if (paired) {
      if (k < nlane) {
        p2_put(J, b.acc, line, k, ae + ao, p2_scale(J, k, J.wm));
        if (D - k != k) p2_put(J, b.acc, line, D - k, is_sin ? ao - ae : ae - ao, p2_scale(J, D - k, J.wm));
      }
    } else {
      p2_put(J, b.acc, line, k, on ? ae : 0.0, p2_scale(J, k, J.wm));
    }
  }
}

// Fused two-level pass for launches with few lines (the x passes of 2-D
// tanks).  The outputs k whose folded class k' (k mod 2A, reflected about
// A) is g or A - g need the pass-1 values C, S at those two k' only, and
// pass 1 gives both from one even/odd j1 sum.  So one CTA per (job, line,
// class pair g <= A/2, output split u) computes C, S of its pair into
// shared memory and then the outputs of its pair: both passes in one
// launch, no partial sums through global memory, and no communication
// between CTAs.  A half-period cos table is staged whole in shared memory
// (before griddepcontrol.wait when it is constant).  With nsplit > 1 the
// outputs of a pair are dealt round-robin to nsplit CTAs, each of which
// repeats the (short) pass 1.
constexpr int kFThreads = 256;
constexpr int kFWarps = kFThreads / 32;

// distinct residues k mod 2A of class pair g, ascending: {g, A-g, A+g, 2A-g}
__host__ __device__ inline int fused_residues(int A, int g, int* r) {
  if (g == 0) { r[0] = 0; r[1] = A; return 2; }
  if (2 * g == A) { r[0] = g; r[1] = A + g; return 2; }
  r[0] = g; r[1] = A - g; r[2] = A + g; r[3] = 2 * A - g;
  return 4;
}
// residue i of fused_residues(A, g, .), without an indexed local array
__host__ __device__ inline int fused_residue(int A, int g, int i) {
  if (g == 0) return i == 0 ? 0 : A;
  if (2 * g == A) return i == 0 ? g : A + g;
  return i == 0 ? g : (i == 1 ? A - g : (i == 2 ? A + g : 2 * A - g));
}
// number of outputs k < nlane in class pair g
__host__ __device__ inline int fused_slots(int A, int g, int nlane) {
  int r[4];
  const int nr = fused_residues(A, g, r);
  const int per = nlane / (2 * A), rem = nlane - per * 2 * A;
  int n = per * nr;
  for (int i = 0; i < nr; ++i) n += r[i] < rem ? 1 : 0;
  return n;
}
// j2 parts of pass 2 for nsb blocks of 32 outputs (even: parts keep the
// parity of j2, which paired outputs need)
__host__ __device__ inline int fused_parts(int nsb) {
  if (nsb <= 0 || nsb >= kFWarps) return 2;
  const int p = (kFWarps / nsb) & ~1;
  return p < 2 ? 2 : p;
}
__host__ __device__ inline int fused_p1_parts(int B) { return B >= kFThreads ? 1 : kFThreads / B; }

template <int NJ>
__global__ void __launch_bounds__(kFThreads) two_level_fused(const AxisBatchT<NJ> b, int nsplit) {
  extern __shared__ double smf[];
  int jb = 0;
  while (jb + 1 < b.njobs && (int)blockIdx.x >= b.start[jb + 1]) ++jb;
  const AxisJob& J = b.job[jb];
  const int A = J.A, B = J.B, D = J.D, D2 = 2 * D, D4 = 4 * D, H = A / 2;
  const int local = blockIdx.x - b.start[jb];
  const int line = local / ((H + 1) * nsplit);
  const int rem = local - line * (H + 1) * nsplit;
  const int g = rem / nsplit, u = rem - g * nsplit;
  const bool paired = J.mode == 1;
  const bool is_sin = (J.off != 0);
  const int nlane = paired ? D / 2 + 1 : J.nout;
  const int j_end = min(J.jhi, J.nin);
  const int K = (j_end + B - 1) / B;
  const int Klp = (K + 1) & ~1;
  // FP64 work on this GPU is scarce (about 2 operations per clock per SM),
  // so the inner loops issue FMAs only: the table covers a half period, so
  // a lookup needs no sign change, and signs and weights are applied to
  // the few sums, not to the terms.
  double* qh = smf;                 // 2D + 1: cos(pi m / (2D)), m = 0..2D
  double* xs = qh + (D2 + 1);       // Klp * B inputs, zero outside the sum
  double* csm = xs + Klp * B;       // B x {C(g), S(g), C(A-g), S(A-g)}
  double* red = csm + 4 * B;        // partial sums of both passes
  auto stage_table = [&]() {
    // cos(pi m/(2D)) = -cos(pi (2D - m)/(2D)): the sign bit is flipped as an
    // integer
    for (int t = threadIdx.x; t <= D2; t += kFThreads)
      qh[t] = t <= D ? __ldg(J.q + t)
                     : __longlong_as_double(__double_as_longlong(__ldg(J.q + (D2 - t))) ^ (1LL << 63));
  };
  auto cosm = [&](int m) { return qh[m <= D2 ? m : D4 - m]; };                 // m in [0, 4D)
  auto sinm = [&](int m) { return cosm(m >= D ? m - D : m + 3 * D); };
  if (b.early) stage_table();
  pdl_wait();
  if (!b.early) stage_table();
  const double* __restrict__ x = J.in + (long long)line * J.in_sl;
  const double* __restrict__ wr = J.win ? J.win + (long long)line * J.win_sl : nullptr;
  // interior inputs enter with weight wm, applied to the sums below; the two
  // end points carry w0 / wm and wl / wm
  const double e0 = J.w0 / J.wm, el = J.wl / J.wm;
  for (int t = threadIdx.x; t < Klp * B; t += kFThreads) {
    double v = 0.0;
    if (t >= J.jlo && t < j_end) {
      v = wr ? __ldg(x + (long long)t * J.in_sk) * __ldg(wr + (long long)t * J.win_sk)
             : __ldg(x + (long long)t * J.in_sk);
      if (t == 0) v *= e0;
      else if (t == J.N - 1) v *= el;
    }
    xs[t] = v;
  }
  __syncthreads();
  // pass 1: items (j2, part); part sums the j1 pairs q = part, part + P1, ...
  const int P1 = fused_p1_parts(B);
  const int npair = Klp / 2;
  {
    const int stp = (int)((2LL * B * g) % D4);                      // angle index of j1 = 1
    const int inc = (int)((2LL * stp * (long long)P1) % D4);        // j1 -> j1 + 2 P1
    for (int it = threadIdx.x; it < P1 * B; it += kFThreads) {
      const int j2 = it % B, part = it / B;
      double ce = 0.0, se = 0.0, co = 0.0, so = 0.0;
      int m = (int)((2LL * stp * (long long)part) % D4);           // j1 = 2 part
      for (int q = part; q < npair; q += P1) {
        int m1 = m + stp;
        if (m1 >= D4) m1 -= D4;
        const double v0 = xs[(2 * q) * B + j2], v1 = xs[(2 * q + 1) * B + j2];
        ce = fma(v0, cosm(m), ce);
        se = fma(v0, sinm(m), se);
        co = fma(v1, cosm(m1), co);
        so = fma(v1, sinm(m1), so);
        m += inc;
        if (m >= D4) m -= D4;
      }
      red[4 * it] = ce + co;      // C(g)
      red[4 * it + 1] = se + so;  // S(g)
      red[4 * it + 2] = ce - co;  // C(A - g)
      red[4 * it + 3] = so - se;  // S(A - g)
    }
  }
  __syncthreads();
  for (int t = threadIdx.x; t < B; t += kFThreads) {
    double f[4] = {0.0, 0.0, 0.0, 0.0};
    for (int part = 0; part < P1; ++part)
#pragma unroll
      for (int v = 0; v < 4; ++v) f[v] += red[4 * (part * B + t) + v];
#pragma unroll
    for (int v = 0; v < 4; ++v) csm[4 * t + v] = f[v] * J.wm;
  }
  __syncthreads();
  // pass 2: this CTA's outputs are the slots s = t nsplit + u of the pair
  const int nr = (g == 0 || 2 * g == A) ? 2 : 4;
  const int nslot = fused_slots(A, g, nlane);
  const int nu = nslot > u ? (nslot - u + nsplit - 1) / nsplit : 0;
  const int nsb = (nu + 31) / 32;
  const int P = fused_parts(nsb);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int item = warp; item < nsb * P; item += kFWarps) {
    const int sb = item / P, p = item - sb * P;
    const int t = sb * 32 + lane;
    double y = 0.0;
    if (t < nu) {
      const int s = t * nsplit + u;
      const int k = 2 * A * (s / nr) + fused_residue(A, g, s % nr);
      int kp = k % (2 * A);
      double ssign = 1.0;
      if (kp > A) { kp = 2 * A - kp; ssign = -1.0; }
      const double* cp = csm + (kp == g ? 0 : 2);
      int m = (int)((2LL * p * k) % D4);
      const int inc = (int)((2LL * P * k) % D4);
      // cos kind: y = sum cw C - ssign sum sw S; sin kind: y = ssign sum cw S + sum sw C
      double a1 = 0.0, a2 = 0.0;
      if (is_sin) {
        for (int j2 = p; j2 < B; j2 += P) {
          a1 = fma(cosm(m), cp[4 * j2 + 1], a1);
          a2 = fma(sinm(m), cp[4 * j2], a2);
          m += inc;
          if (m >= D4) m -= D4;
        }
        y = fma(ssign, a1, a2);
      } else {
        for (int j2 = p; j2 < B; j2 += P) {
          a1 = fma(cosm(m), cp[4 * j2], a1);
          a2 = fma(sinm(m), cp[4 * j2 + 1], a2);
          m += inc;
          if (m >= D4) m -= D4;
        }
        y = fma(-ssign, a2, a1);
      }
    }
    red[item * 32 + lane] = y;
  }
  __syncthreads();
  for (int t = threadIdx.x; t < nu; t += kFThreads) {
    const int sb = t >> 5, ln = t & 31;
    double e = 0.0, o = 0.0;
    for (int p = 0; p < P; p += 2) {
      e += red[(sb * P + p) * 32 + ln];
      o += red[(sb * P + p + 1) * 32 + ln];
    }
    const int s = t * nsplit + u;
    const int k = 2 * A * (s / nr) + fused_residue(A, g, s % nr);
    if (paired) {
      p2_put(J, b.acc, line, k, e + o, p2_scale(J, k, 1.0));
      if (D - k != k) p2_put(J, b.acc, line, D - k, is_sin ? o - e : e - o, p2_scale(J, D - k, 1.0));
    } else {
      p2_put(J, b.acc, line, k, e + o, p2_scale(J, k, 1.0));
    }
  }
}

// Two-level y passes (REDFT00 / RODFT00 along a strided axis, lines
// contiguous): the same split as above, with lanes owning lines so that
// every load and store is coalesced and every twiddle is warp-uniform.
// The partial sums are stored [((j2 (A+1) + k') 2 + {C, S}) nlines + line].
constexpr int kYT = 128;   // lines per CTA
constexpr int kYKF = 9;    // k' <= A/2 per pass-1 CTA (four accumulators each)
constexpr int kYQ = 20;    // outputs of one k' class per pass-2 thread
constexpr int kYH = 12;    // outputs k <= D/2 of one class per thread (paired jobs)

// pass 1: CTA = (job, k' chunk, j2, block of kYT lines).  As in the x pass,
// the even and odd j1 terms are summed apart, which gives C, S at k' and at
// A - k' from the same sums: only k' <= A/2 are computed.
template <int NJ>
__global__ void __launch_bounds__(kYT) ytl_pass1(const AxisBatchT<NJ> b) {
  extern __shared__ double smy[];
  int jb = 0;
  while (jb + 1 < b.njobs && (int)blockIdx.x >= b.start[jb + 1]) ++jb;
  const AxisJob& J = b.job[jb];
  const int A = J.A, B = J.B, D = J.D, D4 = 4 * D, H = A / 2;
  const int nkc = (H + 1 + kYKF - 1) / kYKF;
  int local = blockIdx.x - b.start[jb];
  const int kc = local % nkc;
  local /= nkc;
  const int j2 = local % B;
  const int lb = local / B;
  const int kp0 = kc * kYKF, nkp = min(kYKF, H + 1 - kp0);
  const int j_end = min(J.jhi, J.nin);
  const int K = (j_end + B - 1) / B;
  const int Kp = (K + 1) & ~1;    // whole (even, odd) pairs
  double* tc = smy;               // Kp x kYKF cos(pi j1 k' / A), zero beyond K
  double* ts = tc + Kp * kYKF;    // Kp x kYKF sin(pi j1 k' / A)
  auto stage = [&]() {
    for (int t = threadIdx.x; t < Kp * kYKF; t += kYT) {
      const int j1 = t / kYKF, kpl = t - j1 * kYKF;
      double c = 0.0, sn = 0.0;
      if (kpl < nkp && j1 < K) {
        const unsigned step = (2u * (unsigned)B * (unsigned)(kp0 + kpl)) % (unsigned)D4;
        const int m = (int)((step * (unsigned)j1) % (unsigned)D4);
        c = twiddle(J.q, D, m);
        sn = twiddle(J.q, D, m >= D ? m - D : m + 3 * D);
      }
      tc[t] = c;
      ts[t] = sn;
    }
  };
  if (b.early) stage();
  pdl_wait();
  if (!b.early) stage();
  __syncthreads();
  const int line = lb * kYT + threadIdx.x;
  if (line >= J.nlines) return;
  const double* __restrict__ x = J.in + (long long)line * J.in_sl;
  const double* __restrict__ wr = J.win ? J.win + (long long)line * J.win_sl : nullptr;
  double ce[kYKF], co[kYKF], se[kYKF], so[kYKF];
#pragma unroll
  for (int r = 0; r < kYKF; ++r) ce[r] = co[r] = se[r] = so[r] = 0.0;
  for (int j1 = 0; j1 < K; j1 += 2) {
    const int j = B * j1 + j2, jo = j + B;
    double v0 = 0.0, v1 = 0.0;
    if (j >= J.jlo && j < j_end) {
      const double w = (j == 0) ? J.w0 : ((j == J.N - 1) ? J.wl : J.wm);
      v0 = w * in_at(x, J.in_sk, wr, J.win_sk, j);
    }
    if (j1 + 1 < K && jo >= J.jlo && jo < j_end) {
      const double w = (jo == J.N - 1) ? J.wl : J.wm;
      v1 = w * in_at(x, J.in_sk, wr, J.win_sk, jo);
    }
    const double* t0 = tc + j1 * kYKF;
    const double* s0 = ts + j1 * kYKF;
#pragma unroll
    for (int r = 0; r < kYKF; ++r) {
      ce[r] = fma(v0, t0[r], ce[r]);
      se[r] = fma(v0, s0[r], se[r]);
      co[r] = fma(v1, t0[kYKF + r], co[r]);
      so[r] = fma(v1, s0[kYKF + r], so[r]);
    }
  }
  const long long nl = J.nlines;
  double* o = J.cs + (long long)j2 * (A + 1) * 2 * nl + line;
#pragma unroll
  for (int r = 0; r < kYKF; ++r) {
    if (r < nkp) {
      const int kp = kp0 + r;
      o[(2 * kp) * nl] = ce[r] + co[r];
      o[(2 * kp + 1) * nl] = se[r] + so[r];
      if (A - kp != kp) {
        o[(2 * (A - kp)) * nl] = ce[r] - co[r];
        o[(2 * (A - kp) + 1) * nl] = so[r] - se[r];
      }
    }
  }
}

// output o of class k': k = 2 A o + k' when k' is 0 or A, else alternately
// 2 A q + k' and 2 A (q + 1) - k' (folded, S enters with a minus sign)
__device__ __forceinline__ int ytl_k(int o, int A, int kp, bool pair) {
  if (!pair) return 2 * A * o + kp;
  const int q = o >> 1;
  return (o & 1) ? 2 * A * (q + 1) - kp : 2 * A * q + kp;
}

__device__ __forceinline__ void ytl_put(const AxisJob& J, const AccEpi& acc, int line, int k, double y) {
  if (k >= J.nout) return;
  const bool on = k >= J.klo && k < J.khi;
  const double sc = (k == 0) ? J.s0 : ((k == J.N - 1) ? J.sl : J.sm);
  const double v = on ? y * sc * J.gscale : 0.0;
  const long long e = (long long)line * J.out_sl + (long long)k * J.out_sk;
  J.out[e] = v;
  if (J.epi) acc_epilogue(acc, e, v);
}

// pass 2: CTA = (job, k', block of kYT lines); each C, S value is read once
// and feeds every output of its class.  Paired jobs (mode 1: B even, every
// output wanted): outputs k and D - k are in the same class, and with B
// even y(D - k) = +-sum_j2 (-1)^j2 T_j2(k); the thread sums even and odd j2
// apart for the class's outputs k <= D/2 and writes both.
template <int NJ>
__global__ void __launch_bounds__(kYT, 1) ytl_pass2(const AxisBatchT<NJ> b) {
  extern __shared__ double smy[];
  int jb = 0;
  while (jb + 1 < b.njobs && (int)blockIdx.x >= b.start[jb + 1]) ++jb;
  const AxisJob& J = b.job[jb];
  const int A = J.A, B = J.B, D = J.D, D4 = 4 * D;
  const int local = blockIdx.x - b.start[jb];
  const int kp = local % (A + 1);
  const int lb = local / (A + 1);
  const bool pair = kp > 0 && kp < A;
  const bool paired = J.mode == 1;
  double* tw = smy;  // B x kYQ (cos, sin)(pi j2 k / D)
  auto stage = [&]() {
    for (int t = threadIdx.x; t < B * kYQ; t += kYT) {
      const int j2 = t / kYQ, oi = t - j2 * kYQ;
      const int k = ytl_k(oi, A, kp, pair);
      double c = 0.0, sn = 0.0;
      if (k < J.nout) {
        const int m = (int)((2u * (unsigned)j2 * (unsigned)k) % (unsigned)D4);
        c = twiddle(J.q, D, m);
        sn = twiddle(J.q, D, m >= D ? m - D : m + 3 * D);
      }
      tw[2 * t] = c;
      tw[2 * t + 1] = sn;
    }
  };
  if (b.early) stage();
  pdl_wait();
  if (!b.early) stage();
  __syncthreads();
  const int line = lb * kYT + threadIdx.x;
  if (line >= J.nlines) return;
  const bool is_sin = (J.off != 0);
  const long long nl = J.nlines;
  const double* cs = J.cs + (long long)kp * 2 * nl + line;
  // outputs of this class below nout (uniform over the CTA)
  int nq = 0;
  while (nq < kYQ && ytl_k(nq, A, kp, pair) < J.nout) ++nq;
  if (paired) {
    int nc = 0;  // outputs k <= D/2 (the class's outputs increase with oi)
    while (nc < nq && nc < kYH && ytl_k(nc, A, kp, pair) <= D / 2) ++nc;
    double ae[kYH], ao[kYH];
#pragma unroll
    for (int oi = 0; oi < kYH; ++oi) ae[oi] = ao[oi] = 0.0;
    for (int j2 = 0; j2 < B; j2 += 2) {
      const long long base = (long long)j2 * (A + 1) * 2 * nl;
      const long long step = (long long)(A + 1) * 2 * nl;
      const double C0 = __ldcg(cs + base), S0 = __ldcg(cs + base + nl);
      const double C1 = __ldcg(cs + base + step), S1 = __ldcg(cs + base + step + nl);
      const double2* t0 = reinterpret_cast<const double2*>(tw) + j2 * kYQ;
      const double2* t1 = t0 + kYQ;
#pragma unroll
      for (int oi = 0; oi < kYH; ++oi) {
        if (oi < nc) {
          const bool neg = pair && (oi & 1);
          const double Sa = neg ? -S0 : S0, Sb = neg ? -S1 : S1;
          const double2 w0 = t0[oi], w1 = t1[oi];
          if (is_sin) {
            ae[oi] = fma(w0.x, Sa, fma(w0.y, C0, ae[oi]));
            ao[oi] = fma(w1.x, Sb, fma(w1.y, C1, ao[oi]));
          } else {
            ae[oi] = fma(w0.x, C0, fma(-w0.y, Sa, ae[oi]));
            ao[oi] = fma(w1.x, C1, fma(-w1.y, Sb, ao[oi]));
          }
        }
      }
    }
#pragma unroll
    for (int oi = 0; oi < kYH; ++oi) {
      if (oi < nc) {
        const int k = ytl_k(oi, A, kp, pair);
        ytl_put(J, b.acc, line, k, ae[oi] + ao[oi]);
        if (D - k != k) ytl_put(J, b.acc, line, D - k, is_sin ? ao[oi] - ae[oi] : ae[oi] - ao[oi]);
      }
    }
    return;
  }
  double acc[kYQ];
#pragma unroll
  for (int oi = 0; oi < kYQ; ++oi) acc[oi] = 0.0;
#pragma unroll 2
  for (int j2 = 0; j2 < B; ++j2) {
    const long long base = (long long)j2 * (A + 1) * 2 * nl;
    const double C = __ldcg(cs + base), S = __ldcg(cs + base + nl);
    const double2* t = reinterpret_cast<const double2*>(tw) + j2 * kYQ;
#pragma unroll
    for (int oi = 0; oi < kYQ; ++oi) {
      if (oi < nq) {
        const double Ss = (pair && (oi & 1)) ? -S : S;
        const double2 w = t[oi];
        acc[oi] = is_sin ? fma(w.x, Ss, fma(w.y, C, acc[oi])) : fma(w.x, C, fma(-w.y, Ss, acc[oi]));
      }
    }
  }
#pragma unroll
  for (int oi = 0; oi < kYQ; ++oi) {
    const int k = ytl_k(oi, A, kp, pair);
    if (oi < nq) ytl_put(J, b.acc, line, k, acc[oi]);
  }
}

// Fill the kind-dependent parameters of a pass.
void set_kind(AxisJob& J, int kind, int N, const double* q) {
  J.N = N;
  J.q = q;
  J.off = 0;
  J.jlo = 0;
  J.jhi = N;
  J.klo = 0;
  J.khi = N;
  J.w0 = J.wm = J.wl = 1.0;
  J.s0 = J.sm = J.sl = 1.0;
  switch (kind) {
    case K_C1_S2F:
    case K_C1_F2S:
    case K_S1_S2F:
    case K_S1_F2S: {
      const int D = N - 1;
      J.D = D;
      J.aj = 2; J.bj = 0; J.ak = 1; J.bk = 0;
      if (kind == K_C1_S2F) {
        J.w0 = 1.0; J.wm = 2.0; J.wl = 1.0;
        J.s0 = 1.0 / (2.0 * D); J.sm = 1.0 / D; J.sl = 1.0 / (2.0 * D);
      } else if (kind == K_S1_S2F || kind == K_S1_F2S) {
        J.off = 3 * D;  // sin = cos shifted by -D
        J.jlo = 1; J.jhi = N - 1;
        J.klo = 1; J.khi = N - 1;
        if (kind == K_S1_S2F) { J.w0 = J.wm = J.wl = 2.0; J.s0 = J.sm = J.sl = 1.0 / D; }
      }
      break;
    }
    default: {
      const int D = N;
      J.D = D;
      const double inv = 1.0 / N;
      if (kind == K_ZC_S2F) {
        J.aj = 1; J.bj = 0; J.ak = 2; J.bk = 1;
        J.w0 = 1.0; J.wm = 2.0; J.wl = 2.0;
        J.s0 = J.sm = J.sl = inv;
      } else if (kind == K_ZS_S2F) {
        J.aj = 1; J.bj = 1; J.ak = 2; J.bk = 1; J.off = 3 * D;
        J.w0 = 2.0; J.wm = 2.0; J.wl = 1.0;
        J.s0 = J.sm = J.sl = inv;
      } else if (kind == K_ZC_F2S) {
        J.aj = 2; J.bj = 1; J.ak = 1; J.bk = 0;
      } else {  // K_ZS_F2S
        J.aj = 2; J.bj = 1; J.ak = 1; J.bk = 1; J.off = 3 * D;
      }
      break;
    }
  }
}

int axis_kind(int grid_axis_is_z, int dir, int cs) {
  if (grid_axis_is_z) {
    if (dir > 0) return cs ? K_ZS_S2F : K_ZC_S2F;
    return cs ? K_ZS_F2S : K_ZC_F2S;
  }
  if (dir > 0) return cs ? K_S1_S2F : K_C1_S2F;
  return cs ? K_S1_F2S : K_C1_F2S;
}

constexpr size_t kSmemCap = 200 * 1024;  // dynamic shared memory of a pass

// FMAs of a two-level pass pair on one line: pass 1 folds k' about A/2,
// pass 2 pairs outputs k, D - k when B is even and every output is wanted
double x_two_level_cost(int A, int B, int D, int nin, int nout) {
  const bool paired = (B % 2 == 0) && nout == D + 1;
  return 2.0 * (A / 2 + 1) * (double)nin + 2.0 * B * (paired ? (double)(D / 2 + 1) : (double)nout);
}
// Choose D = A * B minimising the two-level work x_two_level_cost; A = 0
// when the direct sum (about nin * nout / 2 FMAs) is cheaper.
void pick_factors(int D, int nin, int nout, int* Aout, int* Bout) {
  *Aout = *Bout = 0;
  const double direct = 0.5 * (double)nin * (double)nout;
  double best = 0.6 * direct;  // two passes must pay for the second launch
  for (int A = 2; A <= D / 2; ++A) {
    if (D % A) continue;
    const int B = D / A;
    if (B < 2 || B > 256) continue;  // two_level_pass2_lines stages B x 32 twiddle pairs
    if (8LL * (A + 2) > (long long)kSmemCap) continue;  // pass 1's inputs
    const double cost = x_two_level_cost(A, B, D, nin, nout);
    if (cost < best) {
      best = cost;
      *Aout = A;
      *Bout = B;
    }
  }
}

// Call f with the smallest batch capacity that holds b's jobs.
template <int NJ>
AxisBatchT<NJ> shrink(const AxisBatch& b) {
  AxisBatchT<NJ> s{};
  for (int i = 0; i < b.njobs; ++i) s.job[i] = b.job[i];
  for (int i = 0; i <= b.njobs; ++i) s.start[i] = b.start[i];
  s.njobs = b.njobs;
  s.early = b.early;
  s.acc = b.acc;
  return s;
}
template <typename F>
void with_capacity(int njobs, F&& f) {
  if (njobs <= 1) f(std::integral_constant<int, 1>{});
  else if (njobs <= 2) f(std::integral_constant<int, 2>{});
  else if (njobs <= 4) f(std::integral_constant<int, 4>{});
  else if (njobs <= 8) f(std::integral_constant<int, 8>{});
  else f(std::integral_constant<int, kMaxJobs>{});
}
template <typename K>
void allow_smem(K kern) {
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemCap);
}

int p1_terms(const AxisJob& J) { return (std::min(J.jhi, J.nin) + J.B - 1) / J.B; }
// Shared memory of the passes (the twiddles, pass 1 also the inputs).
size_t pass1_smem(const AxisJob& J, int P, bool staged) {
  const int K = p1_terms(J), Kp = (K + 1) & ~1;
  const P1Shape s = p1_shape(J.A, J.B, P);
  return sizeof(double) * ((staged ? 4 * (size_t)J.A : 0) + (size_t)Kp * s.G);
}
size_t pass2_smem(const AxisJob& J) { return sizeof(double) * ((size_t)J.D + 1); }
size_t pass2_lines_smem(const AxisJob& J) { return sizeof(double) * 2 * 32 * (size_t)J.B; }

// FMAs of a two-level pass pair on one line
double two_level_fmas(const AxisJob& J) {
  return x_two_level_cost(J.A, J.B, J.D, std::min(J.nin, J.N), J.nout);
}
// the y passes (ytl_pass1/2) fold and pair the same way (pairing when the
// job's mode is 1)
double y_two_level_fmas(const AxisJob& J) {
  return 2.0 * (J.A / 2 + 1) * (double)std::min(J.nin, J.N) +
         2.0 * J.B * (J.mode == 1 ? (double)(J.D / 2 + 1) : (double)J.nout);
}
// outputs k <= D/2 of one k' class of a y pass are at most this many
bool ytl_can_pair(int D, int A, int B, int nout, int N) {
  return B % 2 == 0 && nout == N && 2 * ((D / 2) / (2 * A)) + 2 <= kYH;
}

void launch_two_level(AxisBatch& b, int nsm, bool early, cudaStream_t st) {
  b.early = early ? 1 : 0;
  for (int i = 0; i < b.njobs; ++i) g_xform_fmas += (double)b.job[i].nlines * two_level_fmas(b.job[i]);
  static PerDeviceOnce attr_set;
  attr_set.run([&] {
    for (int nj : {1, 2, 4, 8, kMaxJobs})
      with_capacity(nj, [&](auto c) {
        constexpr int NJ = decltype(c)::value;
        allow_smem(two_level_pass1<NJ, true>);
        allow_smem(two_level_pass1<NJ, false>);
        allow_smem(two_level_pass2<NJ, 16>);
        allow_smem(two_level_pass2<NJ, 32>);
      });
  });
  // pass 1: as many parts per sum as keep the launch within half of the SMs.
  // The right-hand side runs three branches at a time, and the CTAs of their
  // next passes wait on the SMs too: with launches of two CTAs per SM and eight
  // outputs per CTA of pass 2 a step of 257 modes took 0.49 to 0.75 ms from
  // one to the next, with these it takes 0.48 to 0.50, one of 1025 modes
  // 0.91 ms for 1.07 (a third or a quarter of the SMs: 0.93 to 0.98).
  auto ctas1 = [&](int P) {
    long long n = 0;
    for (int i = 0; i < b.njobs; ++i) {
      const AxisJob& J = b.job[i];
      const P1Shape s = p1_shape(J.A, J.B, P);
      n += (long long)J.nlines * s.kblocks * s.jblocks;
    }
    return n;
  };
  int P = 16;
  while (P > 2 && 2 * ctas1(P) > std::max(nsm, 1)) P /= 2;
  size_t smem1 = 0, smem2 = 0;
  bool staged = true;
  for (int i = 0; i < b.njobs; ++i) staged = staged && pass1_smem(b.job[i], P, true) <= kSmemCap;
  int total = 0;
  for (int i = 0; i < b.njobs; ++i) {
    const AxisJob& J = b.job[i];
    const P1Shape s = p1_shape(J.A, J.B, P);
    smem1 = std::max(smem1, pass1_smem(J, P, staged));
    b.start[i] = total;
    total += J.nlines * s.kblocks * s.jblocks;
  }
  b.start[b.njobs] = total;
  if (total > 0)
    with_capacity(b.njobs, [&](auto c) {
      constexpr int NJ = decltype(c)::value;
      launch_pdl(staged ? two_level_pass1<NJ, true> : two_level_pass1<NJ, false>, dim3(total), dim3(kP1Threads), smem1, st,
                 shrink<NJ>(b), P);
    });
  // Pass 2 gathers from a staged quarter-wave table whatever the lines.  (Groups of
  // lines that shared a staged tile of B x 32 pairs took 16 lines and more: 16 of 1024
  // points 74 us for both passes, 14 with the gather; 513 of 1025 points 355 and 124;
  // nowhere less, from 66 to 8193 points.)  Lengths whose table is over the shared
  // memory (D > 25599) keep the tiles, of 128 KB at most.
  size_t table = 0;
  for (int i = 0; i < b.njobs; ++i) table = std::max(table, pass2_smem(b.job[i]));
  if (table > kSmemCap) {
    static PerDeviceOnce attr_l;
    attr_l.run([&] {
      for (int nj : {1, 2, 4, 8, kMaxJobs})
        with_capacity(nj, [&](auto c) { allow_smem(two_level_pass2_lines<decltype(c)::value>); });
    });
    long long blocks = 0;
    for (int i = 0; i < b.njobs; ++i) blocks += (long long)b.job[i].nlines * ((p2_lanes(b.job[i]) + 31) / 32);
    const int lpc = (int)std::min<long long>(16, std::max<long long>(4, blocks / (4LL * std::max(nsm, 1))));
    total = 0;
    for (int i = 0; i < b.njobs; ++i) {
      b.start[i] = total;
      total += ((b.job[i].nlines + lpc - 1) / lpc) * ((p2_lanes(b.job[i]) + 31) / 32);
      smem2 = std::max(smem2, pass2_lines_smem(b.job[i]));
    }
    b.start[b.njobs] = total;
    with_capacity(b.njobs, [&](auto c) {
      constexpr int NJ = decltype(c)::value;
      launch_pdl(two_level_pass2_lines<NJ>, dim3(total), dim3(kP2Threads), smem2, st, shrink<NJ>(b), lpc);
    });
    return;
  }
  // pass 2: 16 outputs per CTA where 32 do not cover the SMs
  auto ctas2 = [&](int KO) {
    long long n = 0;
    for (int i = 0; i < b.njobs; ++i) n += (long long)b.job[i].nlines * ((p2_lanes(b.job[i]) + KO - 1) / KO);
    return n;
  };
  const int KO = ctas2(32) < std::max(nsm, 1) ? 16 : 32;
  total = 0;
  for (int i = 0; i < b.njobs; ++i) {
    b.start[i] = total;
    total += b.job[i].nlines * ((p2_lanes(b.job[i]) + KO - 1) / KO);
    smem2 = std::max(smem2, pass2_smem(b.job[i]));
  }
  b.start[b.njobs] = total;
  if (total > 0)
    with_capacity(b.njobs, [&](auto c) {
      constexpr int NJ = decltype(c)::value;
      if (KO == 16) launch_pdl(two_level_pass2<NJ, 16>, dim3(total), dim3(kP2Threads), smem2, st, shrink<NJ>(b));
      else launch_pdl(two_level_pass2<NJ, 32>, dim3(total), dim3(kP2Threads), smem2, st, shrink<NJ>(b));
    });
}

// Shared memory of the fused pass for job J with nsplit CTAs per class pair.
size_t fused_smem(const AxisJob& J, int nsplit) {
  const int j_end = std::min(J.jhi, J.nin);
  const int K = (j_end + J.B - 1) / J.B;
  const int Klp = (K + 1) & ~1;
  const int nlane = J.mode == 1 ? J.D / 2 + 1 : J.nout;
  size_t red = (size_t)4 * fused_p1_parts(J.B) * J.B;
  for (int g = 0; g <= J.A / 2; ++g) {
    const int nslot = fused_slots(J.A, g, nlane);
    const int nu = (nslot + nsplit - 1) / nsplit;
    const int nsb = (nu + 31) / 32;
    red = std::max(red, (size_t)nsb * fused_parts(nsb) * 32);
  }
  return sizeof(double) * (2 * (size_t)J.D + 1 + (size_t)Klp * J.B + 4 * (size_t)J.B + red);
}

// The fused pass serves x-pass batches whose jobs have few lines in all
// (2-D tanks) and no accumulation epilogue, when its shared memory fits;
// returns false (launching nothing) otherwise.
bool launch_two_level_fused(AxisBatch& b, int nsm, bool early, cudaStream_t st) {
  if (!g_fused_enabled) return false;
  long long units = 0;
  for (int i = 0; i < b.njobs; ++i) {
    const AxisJob& J = b.job[i];
    if (J.epi || J.A < 2 || J.wm == 0.0) return false;
    units += (long long)J.nlines * (J.A / 2 + 1);
  }
  if (units == 0 || units > 4LL * std::max(nsm, 1)) return false;
  // a small launch spreads each pair's outputs over up to 4 CTAs
  const int nsplit = (int)std::max<long long>(1, std::min<long long>(4, std::max(nsm, 1) / units));
  size_t smem = 0;
  for (int i = 0; i < b.njobs; ++i) smem = std::max(smem, fused_smem(b.job[i], nsplit));
  if (smem > kSmemCap) return false;
  static PerDeviceOnce attr_set;
  attr_set.run([&] {
    for (int nj : {1, 2, 4, 8, kMaxJobs})
      with_capacity(nj, [&](auto c) { allow_smem(two_level_fused<decltype(c)::value>); });
  });
  b.early = early ? 1 : 0;
  int total = 0;
  for (int i = 0; i < b.njobs; ++i) {
    const AxisJob& J = b.job[i];
    b.start[i] = total;
    total += J.nlines * (J.A / 2 + 1) * nsplit;
    // pass 1 runs once per CTA of a pair
    g_xform_fmas += (double)J.nlines * (two_level_fmas(J) +
                                        (nsplit - 1) * 2.0 * (J.A / 2 + 1) * std::min(J.nin, J.N));
  }
  b.start[b.njobs] = total;
  with_capacity(b.njobs, [&](auto c) {
    constexpr int NJ = decltype(c)::value;
    launch_pdl(two_level_fused<NJ>, dim3(total), dim3(kFThreads), smem, st, shrink<NJ>(b), nsplit);
  });
  return true;
}

// Decide the symmetry mode and the split of every x-pass job, then launch.
// Jobs of few lines whose twiddles fit run direct_pass and leave the batch.
void launch_direct(AxisBatch& b, const Tables& tb, cudaStream_t st) {
  AxisBatch few{}, rest{};
  few.njobs = rest.njobs = 0;
  few.acc = rest.acc = b.acc;
  few.early = tb.q_const ? 1 : 0;
  long long lanes = 0;
  for (int i = 0; i < b.njobs; ++i) {
    AxisJob J = b.job[i];
    const bool c1s1 = (J.aj == 2 && J.bj == 0 && J.ak == 1 && J.bk == 0);
    J.mode = J.nout == J.N ? 1 : (J.nin >= J.N ? 2 : 0);
    J.nlane = J.mode == 1 ? J.D / 2 + 1 : J.nout;
    if (!c1s1 || J.D < 4 || J.nlines > kDirMaxLines || J.D > kDirMaxD) {
      rest.job[rest.njobs++] = b.job[i];
      continue;
    }
    lanes += (long long)J.nlines * J.nlane;
    few.job[few.njobs++] = J;
  }
  b = rest;
  if (few.njobs == 0) return;
  // fewer outputs per CTA until the launch covers the SMs
  int KO = 32;
  while (KO > 4 && lanes / KO < std::max(tb.nsm, 1)) KO /= 2;
  int total = 0;
  size_t smem = 0;
  for (int i = 0; i < few.njobs; ++i) {
    const AxisJob& J = few.job[i];
    const int nt = dir_terms(J);
    few.start[i] = total;
    total += J.nlines * ((J.nlane + KO - 1) / KO);
    smem = std::max(smem, sizeof(double) * ((size_t)J.D + 1 + (J.mode == 2 ? 2 : 1) * (size_t)nt));
    g_xform_fmas += (double)J.nlines * J.nlane * nt;
  }
  few.start[few.njobs] = total;
  static PerDeviceOnce attr;
  attr.run([&] {
    for (int nj : {1, 2, 4, 8, kMaxJobs})
      with_capacity(nj, [&](auto c) {
        constexpr int NJ = decltype(c)::value;
        allow_smem(direct_pass<NJ, 4>);
        allow_smem(direct_pass<NJ, 8>);
        allow_smem(direct_pass<NJ, 16>);
        allow_smem(direct_pass<NJ, 32>);
      });
  });
  with_capacity(few.njobs, [&](auto c) {
    constexpr int NJ = decltype(c)::value;
    if (KO == 4) launch_pdl(direct_pass<NJ, 4>, dim3(total), dim3(kDirThreads), smem, st, shrink<NJ>(few));
    else if (KO == 8) launch_pdl(direct_pass<NJ, 8>, dim3(total), dim3(kDirThreads), smem, st, shrink<NJ>(few));
    else if (KO == 16) launch_pdl(direct_pass<NJ, 16>, dim3(total), dim3(kDirThreads), smem, st, shrink<NJ>(few));
    else launch_pdl(direct_pass<NJ, 32>, dim3(total), dim3(kDirThreads), smem, st, shrink<NJ>(few));
  });
}

void launch_batch_x(AxisBatch& b, const Tables& tb, cudaStream_t st) {
  launch_direct(b, tb, st);
  if (b.njobs == 0) return;
  b.early = tb.q_const ? 1 : 0;
  long long tiles_total = 0;
  for (int i = 0; i < b.njobs; ++i) {
    AxisJob& J = b.job[i];
    const bool c1s1 = (J.aj == 2 && J.bj == 0 && J.ak == 1 && J.bk == 0);  // REDFT00 / RODFT00 kinds
    const int D = J.D;
    const int j_end = std::min(J.jhi, J.nin);
    if (c1s1 && J.nout == J.N && D >= 4) {
      J.mode = 1;
      J.nlane = D / 2 + 1;
      J.ta = std::max(J.jlo, 1);
      J.tb = std::min(j_end, J.N - 1);
    } else if (c1s1 && J.nin >= J.N && J.nout <= D / 2 + 1 && D >= 4 &&
               J.w0 == J.wl) {
      J.mode = 2;
      J.nlane = J.nout;
      J.ta = std::max(J.jlo, 1);
      J.tb = (D + 1) / 2;  // pairs j < D - j
    } else {
      J.mode = 0;
      J.nlane = J.nout;
      J.ta = std::max(J.jlo, 1);
      J.tb = std::min(j_end, J.N - 1);
    }
    if (J.tb < J.ta) J.tb = J.ta;
    J.ntile = (J.nlane + 31) / 32;
    tiles_total += (long long)J.nlines * J.ntile;
  }
  const long long target = 4LL * std::max(tb.nsm, 1);
  long long part_need = 0, cnt_need = 0;
  int total = 0;
  for (int i = 0; i < b.njobs; ++i) {
    AxisJob& J = b.job[i];
    int terms = J.tb - J.ta;
    int nchunk = 1;
    if (tiles_total < target && terms > 512)
      nchunk = std::min((int)((target + tiles_total - 1) / tiles_total), (terms + 255) / 256);
    int chunk = std::max(1, (terms + nchunk - 1) / std::max(nchunk, 1));
    nchunk = std::max(1, (terms + chunk - 1) / chunk);
    J.part = nullptr;
    J.cnt = nullptr;
    if (nchunk > 1) {
      const long long np = (long long)J.nlines * J.ntile * nchunk * 64;
      const long long nc = (long long)J.nlines * J.ntile;
      if (part_need + np <= tb.part_cap && cnt_need + nc <= tb.cnt_cap) {
        J.part = tb.part + part_need;
        J.cnt = tb.cnt + cnt_need;
        part_need += np;
        cnt_need += nc;
      } else {
        // not enough scratch for a split sum: one CTA per tile
        nchunk = 1;
        chunk = std::max(terms, 1);
      }
    }
    J.nchunk = nchunk;
    J.chunk = chunk;
    g_xform_fmas += (double)J.nlines * J.nlane * std::max(J.tb - J.ta, 1);
    b.start[i] = total;
    total += J.nlines * J.ntile * J.nchunk;
  }
  b.start[b.njobs] = total;
  size_t smem = 0;
  for (int i = 0; i < b.njobs; ++i)
    smem = std::max(smem, sizeof(double) * ((size_t)b.job[i].D + 1 + 2 * (size_t)kMaxPairChunk));
  static PerDeviceOnce attr_set;
  attr_set.run([&] {
    for (int nj : {1, 2, 4, 8, kMaxJobs})
      with_capacity(nj, [&](auto c) { allow_smem(axis_pass_lanes_k<decltype(c)::value>); });
  });
  if (total > 0)
    with_capacity(b.njobs, [&](auto c) {
      constexpr int NJ = decltype(c)::value;
      launch_pdl(axis_pass_lanes_k<NJ>, dim3(total), dim3(kXThreads), smem, st, shrink<NJ>(b));
    });
}

// Factor pair of a y pass: minimum 2 (A+1) nin + 2 B nout FMAs, with every
// k' class (at most 2 nout / (2A) + 2 outputs) held by one pass-2 thread;
// A = 0 when the direct sum (nin * nout FMAs) is cheaper.
void pick_factors_y(int D, int nin, int nout, int* Aout, int* Bout) {
  *Aout = *Bout = 0;
  double best = 0.6 * (double)nin * (double)nout;
  for (int A = 2; A <= D / 2; ++A) {
    if (D % A) continue;
    const int B = D / A;
    if (B < 2 || B > 256) continue;
    if (2 * ((nout + 2 * A - 1) / (2 * A)) + 1 > kYQ) continue;
    const bool paired = ytl_can_pair(D, A, B, nout, D + 1);
    const double cost = 2.0 * (A / 2 + 1) * (double)nin + 2.0 * B * (paired ? (double)(D / 2 + 1) : (double)nout);
    if (cost < best) {
      best = cost;
      *Aout = A;
      *Bout = B;
    }
  }
}

void launch_ytl(AxisBatch& b, bool early, cudaStream_t st) {
  b.early = early ? 1 : 0;
  for (int i = 0; i < b.njobs; ++i) g_xform_fmas += (double)b.job[i].nlines * y_two_level_fmas(b.job[i]);
  static PerDeviceOnce attr_set;
  attr_set.run([&] {
    for (int nj : {1, 2, 4, 8, kMaxJobs})
      with_capacity(nj, [&](auto c) {
        allow_smem(ytl_pass1<decltype(c)::value>);
        allow_smem(ytl_pass2<decltype(c)::value>);
      });
  });
  int total = 0;
  size_t smem1 = 0, smem2 = 0;
  for (int i = 0; i < b.njobs; ++i) {
    const AxisJob& J = b.job[i];
    const int nlb = (J.nlines + kYT - 1) / kYT;
    const int K = (std::min(J.jhi, J.nin) + J.B - 1) / J.B;
    b.start[i] = total;
    total += nlb * J.B * ((J.A / 2 + 1 + kYKF - 1) / kYKF);
    smem1 = std::max(smem1, sizeof(double) * 2 * (size_t)((K + 1) & ~1) * kYKF);
    smem2 = std::max(smem2, sizeof(double) * 2 * (size_t)J.B * kYQ);
  }
  b.start[b.njobs] = total;
  with_capacity(b.njobs, [&](auto c) {
    constexpr int NJ = decltype(c)::value;
    launch_pdl(ytl_pass1<NJ>, dim3(total), dim3(kYT), smem1, st, shrink<NJ>(b));
  });
  total = 0;
  for (int i = 0; i < b.njobs; ++i) {
    b.start[i] = total;
    total += ((b.job[i].nlines + kYT - 1) / kYT) * (b.job[i].A + 1);
  }
  b.start[b.njobs] = total;
  with_capacity(b.njobs, [&](auto c) {
    constexpr int NJ = decltype(c)::value;
    launch_pdl(ytl_pass2<NJ>, dim3(total), dim3(kYT), smem2, st, shrink<NJ>(b));
  });
}

// FP64 FMAs per line of the sum passes of a job, as its launcher picks them.
double sum_cost(const AxisJob& J, bool ypass) {
  const int nin = std::min(J.nin, J.N);
  int A = 0, B = 0;
  if (!ypass) {
    pick_factors(J.D, nin, J.nout, &A, &B);
    return A > 0 ? x_two_level_cost(A, B, J.D, nin, J.nout) : 0.5 * (double)nin * J.nout;
  }
  pick_factors_y(J.D, nin, J.nout, &A, &B);
  if (A == 0) return 0.5 * (double)nin * J.nout;
  AxisJob t = J;
  t.A = A;
  t.B = B;
  t.mode = ytl_can_pair(J.D, A, B, J.nout, J.N) ? 1 : 0;
  return y_two_level_fmas(t);
}

// Time (us) of a job off the tensor cores, measured on GB300 over 66 to 4100
// points: 2.2 ps per unit of the FFT plan's cost, 4 ps per FMA of the sums.
double pass_time(const AxisJob& J, const Tables& tb, bool ypass) {
  if (!(J.aj == 2 && J.bj == 0 && J.ak == 1 && J.bk == 0)) return 0.0;
  const double sums = sum_cost(J, ypass);
  const FftPlanInfo* f = fft_choice(J, tb, sums);
  return (double)J.nlines * (f ? 2.2e-6 * f->cost_line_df : 4e-6 * sums);
}

// The jobs that run on the tensor cores (tcx.cu) leave the batch.  `next`, if
// given, are the y jobs that read the outputs of b's x jobs.
void launch_tensor(AxisBatch& b, const Tables& tb, cudaStream_t st, AxisBatch* next = nullptr) {
  AxisBatch t{}, rest{};
  t.njobs = rest.njobs = 0;
  t.acc = rest.acc = b.acc;
  int from[kMaxJobs];
  for (int i = 0; i < b.njobs; ++i) {
    if (!b.job[i].tc) {
      rest.job[rest.njobs++] = b.job[i];
      continue;
    }
    from[t.njobs] = i;
    t.job[t.njobs] = b.job[i];
    if (next) t.job[t.njobs].cmax = reinterpret_cast<unsigned*>(tb.cs) + (long long)i * (kTcMaxD + 8);
    ++t.njobs;
  }
  if (t.njobs == 0 || !launch_tc_jobs(t, tb, st)) return;
  b = rest;
  if (next)
    for (int i = 0; i < t.njobs; ++i) next->job[from[i]].lmax = t.job[i].cmax;
}

// Outputs per thread of axis_pass_lanes_line: its time is the FP64 instructions of
// the longest warp and those of all warps over the schedulers.  Fewer outputs per
// thread shorten the first and lengthen the second where terms are paired (two
// additions per pair and thread); eight unless it saves a tenth, as more threads
// read the lines and the twiddles again.
int lanes_line_outputs(const AxisBatch& b, int nsm) {
  auto cost = [&](int r) {
    double longest = 0.0, all = 0.0;
    for (int i = 0; i < b.njobs; ++i) {
      const AxisJob& J = b.job[i];
      const double terms = J.mode == 2 ? (J.D + 1) / 2 : std::max(std::min(std::min(J.jhi, J.nin), J.N) - J.jlo, 1);
      const double ops = terms * (r + (J.mode == 2 ? 2 : 0));
      longest = std::max(longest, ops);
      all += ops * ((J.nlines + kYThreads - 1) / kYThreads) * (kYThreads / 32) * ((J.nlane + r - 1) / r);
    }
    return longest + all / (4.0 * std::max(nsm, 1));
  };
  int best = kYR;
  for (int r = kYR / 2; r >= 2; r /= 2)
    if (cost(r) < 0.9 * cost(kYR) && cost(r) < cost(best)) best = r;
  return best;
}

// y passes: two-level where the length factors well (scratch permitting),
// direct sums otherwise
void launch_batch_y(AxisBatch& in, const Tables& tb, cudaStream_t st) {
  AxisBatch b{}, b2{}, bf{};
  b.njobs = b2.njobs = bf.njobs = 0;
  b.acc = b2.acc = bf.acc = in.acc;
  const FftPlanInfo* fplan[kMaxJobs];
  if (tb.ntc) {
    // jobs whose x pass did not decide for them: a y pass alone
    AxisBatch alone{};
    int from[kMaxJobs];
    double alt[kMaxJobs];
    for (int i = 0; i < in.njobs; ++i)
      if (!in.job[i].tc && !in.job[i].tc_decided) {
        from[alone.njobs] = i;
        alt[alone.njobs] = pass_time(in.job[i], tb, true);
        alone.job[alone.njobs++] = in.job[i];
      }
    AxisJob* jobs[1] = {alone.job};
    const double* alts[1] = {alt};
    tc_choose(jobs, alts, 1, alone.njobs, tb);
    for (int i = 0; i < alone.njobs; ++i) in.job[from[i]].tc = alone.job[i].tc;
  }
  launch_tensor(in, tb, st);
  long long cs_used = tb.ntc ? kTcMaxBytes / (long long)sizeof(double) : 0;  // behind the maxima and the flag
  for (int i = 0; i < in.njobs; ++i) {
    AxisJob J = in.job[i];
    J.A = J.B = 0;
    J.cs = nullptr;
    const bool c1s1 = (J.aj == 2 && J.bj == 0 && J.ak == 1 && J.bk == 0);
    if (c1s1) {
      const int nin = std::min(J.nin, J.N);
      if (const FftPlanInfo* f = fft_choice(J, tb, sum_cost(J, true))) {
        fplan[bf.njobs] = f;
        bf.job[bf.njobs++] = J;
        continue;
      }
    }
    if (c1s1 && tb.cs) {
      int A = 0, B = 0;
      pick_factors_y(J.D, std::min(J.nin, J.N), J.nout, &A, &B);
      const long long need = (long long)J.nlines * B * (A + 1) * 2;
      if (A > 0 && cs_used + need <= tb.cs_cap) {
        J.A = A;
        J.B = B;
        J.mode = ytl_can_pair(J.D, A, B, J.nout, J.N) ? 1 : 0;
        J.cs = tb.cs + cs_used;
        cs_used += need;
        b2.job[b2.njobs++] = J;
        continue;
      }
    }
    b.job[b.njobs++] = J;
  }
  if (bf.njobs) launch_fft_jobs(bf, fplan, tb, st);
  if (b2.njobs) launch_ytl(b2, tb.q_const, st);
  {
    // few lines
    AxisBatch few{}, rest{};
    few.njobs = rest.njobs = 0;
    few.acc = rest.acc = b.acc;
    int total = 0;
    for (int i = 0; i < b.njobs; ++i) {
      AxisJob J = b.job[i];
      const bool c1s1 = (J.aj == 2 && J.bj == 0 && J.ak == 1 && J.bk == 0);
      if (!c1s1 || J.nlines > kFewLines || J.D < 4) {
        rest.job[rest.njobs++] = J;
        continue;
      }
      J.mode = J.nout == J.N ? 1 : 0;
      J.nlane = J.mode ? J.D / 2 + 1 : J.nout;
      g_xform_fmas += (double)J.nlines * J.nlane * (std::min(J.jhi, J.nin) - J.jlo);
      few.start[few.njobs] = total;
      total += (J.nlines + 31) / 32 * ((J.nlane + 1) / 2);
      few.job[few.njobs++] = J;
    }
    few.start[few.njobs] = total;
    if (total > 0)
      with_capacity(few.njobs, [&](auto c) {
        constexpr int NJ = decltype(c)::value;
        launch_pdl(axis_pass_few_lines<NJ>, dim3(total), dim3(256), 0, st, shrink<NJ>(few));
      });
    b = rest;
  }
  if (b.njobs == 0) return;
  for (int i = 0; i < b.njobs; ++i) {
    AxisJob& J = b.job[i];
    const bool c1s1 = (J.aj == 2 && J.bj == 0 && J.ak == 1 && J.bk == 0);
    J.mode = 0;
    J.nlane = J.nout;
    if (c1s1 && J.nout == J.N && J.D >= 4) {
      J.mode = 1;
      J.nlane = J.D / 2 + 1;
    } else if (c1s1 && J.nin >= J.N && J.nout <= J.D / 2 + 1 && J.D >= 4 && J.w0 == J.wl) {
      J.mode = 2;
    }
    {
      const int nin = std::min(std::min(J.jhi, J.nin), J.N) - J.jlo;
      g_xform_fmas += (double)J.nlines * J.nlane * (J.mode == 2 ? (J.D + 1) / 2 : std::max(nin, 1));
    }
  }
  const int R = lanes_line_outputs(b, tb.nsm);
  int total = 0;
  for (int i = 0; i < b.njobs; ++i) {
    b.start[i] = total;
    total += (b.job[i].nlines + kYThreads - 1) / kYThreads * ((b.job[i].nlane + R - 1) / R);
  }
  b.start[b.njobs] = total;
  if (total > 0)
    with_capacity(b.njobs, [&](auto c) {
      constexpr int NJ = decltype(c)::value;
      launch_pdl(R == 2   ? axis_pass_lanes_line<NJ, 2>
                 : R == 4 ? axis_pass_lanes_line<NJ, 4>
                          : axis_pass_lanes_line<NJ, kYR>,
                 dim3(total), dim3(kYThreads), 0, st, shrink<NJ>(b));
    });
}

}  // namespace

thread_local double g_xform_fmas = 0.0;
thread_local bool g_launch_no_pdl = false;
const bool g_fused_enabled = [] {
  const char* e = std::getenv("HOSNWT_FUSED_PASS");
  return e && e[0] == '1';
}();

std::vector<double> quarter_table(int D) {
  std::vector<double> q(D + 1);
  const long double pi = 3.141592653589793238462643383279502884L;
  for (int m = 0; m <= D; ++m) {
    q[m] = (double)cosl(pi * (long double)m / (2.0L * (long double)D));
  }
  if (D > 0) q[D] = 0.0;
  if (D % 3 == 0) q[2 * D / 3] = 0.5;  // cos(pi/3)
  return q;
}

std::vector<double> y_twiddle_rows(int N, bool sin_kind, int* ld) {
  const int D = N - 1;
  const int nk = D / 2 + 1;
  *ld = (nk + 7) / 8 * 8;
  const std::vector<double> q = quarter_table(D);
  std::vector<double> t((size_t)N * *ld, 0.0);
  const long long D4 = 4LL * D, off = sin_kind ? 3LL * D : 0;
  for (int j = 0; j < N; ++j)
    for (int k = 0; k < nk; ++k) {
      const long long m = (2LL * j * k + off) % D4;
      const long long mm = (m > 2LL * D) ? D4 - m : m;
      t[(size_t)j * *ld + k] = (mm > D) ? -q[2 * D - mm] : q[mm];
    }
  return t;
}

namespace {

// The passes of the requests idx[0..n), along x then y.  The first pass
// applies the input weights, the last the scale and the accumulation
// epilogue; tmp[idx[i]] holds the intermediate.
void launch_ordered(const XfReq* reqs, const int* idx, int n, const Tables& tb, double* const* tmp,
                    cudaStream_t st) {
  AxisBatch bx{}, by{};
  bx.njobs = by.njobs = 0;
  for (int i = 0; i < n; ++i)
    if (reqs[idx[i]].acc) bx.acc = by.acc = *reqs[idx[i]].acc;
  for (int i = 0; i < n; ++i) {
    const int r = idx[i];
    const XfReq& R = reqs[r];
    int Nx, Ny;
    const double *qx, *qy;
    const bool zaxis = (R.grid == GRID_ADD);
    if (R.grid == GRID_N) { Nx = tb.n1; Ny = tb.n2; qx = tb.q_n1; qy = tb.q_n2; }
    else if (R.grid == GRID_BIG) { Nx = tb.nd1; Ny = tb.nd2; qx = tb.q_nd1; qy = tb.q_nd2; }
    else { Nx = tb.n3_add; Ny = tb.n2; qx = tb.q_add; qy = tb.q_n2; }
    const bool twod = (tb.n2 != 1);
    // x (or z) pass
    AxisJob& X = bx.job[bx.njobs++];
    set_kind(X, axis_kind(zaxis, R.dir, R.csx), Nx, qx);
    X.nin = R.nin1;
    X.nout = R.nout1;
    X.out_sk = 1;
    X.win_sk = 1;
    if (!twod) {
      X.in = R.in;
      X.in_sk = 1;
      X.in_sl = R.in_ld;
      X.win = R.win;
      X.win_sl = R.win_ld;
      X.nlines = 1;
      X.out = R.out;
      X.out_sl = R.out_ld;
      X.gscale = R.scale;
      X.epi = R.acc ? 1 : 0;
      continue;
    }
    AxisJob& Y = by.job[by.njobs++];
    set_kind(Y, axis_kind(false, R.dir, R.csy), Ny, qy);
    Y.ty = (R.grid == GRID_BIG) ? tb.ty_nd2[R.csy ? 1 : 0] : tb.ty_n2[R.csy ? 1 : 0];
    Y.ldy = (R.grid == GRID_BIG) ? tb.ldy_nd2 : tb.ldy_n2;
    Y.nin = R.nin2;
    Y.nout = R.nout2;
    Y.out_sl = 1;
    // The y-sin plans zero the boundary columns of the input and output
    // (fourier_FFTW.f90:282-285, 296-299): the x pass skips the lines beyond
    // the input's extent.
    X.in = R.in;
    X.in_sk = 1;
    X.in_sl = R.in_ld;
    X.win = R.win;
    X.win_sl = R.win_ld;
    X.nlines = R.nin2;
    X.out = tmp[r];
    X.out_sl = R.nout1;
    X.gscale = 1.0;
    X.epi = 0;
    Y.in = tmp[r];
    Y.in_sk = R.nout1;
    Y.in_sl = 1;
    Y.nlines = R.nout1;
    Y.out = R.out;
    Y.out_sk = R.out_ld;
    Y.gscale = R.scale;
    Y.epi = R.acc ? 1 : 0;
  }
  // FFT passes for the x jobs over many lines where they cost less, then
  // two-level passes for the jobs whose length factors well
  AxisBatch b2{}, bd{}, bf{};
  b2.njobs = bd.njobs = bf.njobs = 0;
  b2.acc = bd.acc = bf.acc = bx.acc;
  const FftPlanInfo* fplan[kMaxJobs];
  if (tb.ntc && by.njobs == bx.njobs) {
    AxisJob* jobs[2] = {bx.job, by.job};
    double altx[kMaxJobs], alty[kMaxJobs];
    for (int i = 0; i < bx.njobs; ++i) {
      altx[i] = pass_time(bx.job[i], tb, false);
      alty[i] = pass_time(by.job[i], tb, true);
      // a y pass with a matrix whose x pass has none is looked at alone
      by.job[i].tc_decided = bx.job[i].D == bx.job[i].N - 1;
    }
    const double* alts[2] = {altx, alty};
    tc_choose(jobs, alts, 2, bx.njobs, tb);
  }
  launch_tensor(bx, tb, st, by.njobs ? &by : nullptr);
  long long cs_used = tb.ntc ? kTcMaxBytes / (long long)sizeof(double) : 0;  // behind the maxima and the flag
  for (int i = 0; i < bx.njobs; ++i) {
    AxisJob J = bx.job[i];
    J.A = J.B = 0;
    J.cs = nullptr;
    const bool c1s1 = (J.aj == 2 && J.bj == 0 && J.ak == 1 && J.bk == 0);
    if (c1s1) {
      const int nin = std::min(J.nin, J.N);
      if (const FftPlanInfo* f = fft_choice(J, tb, sum_cost(J, false))) {
        fplan[bf.njobs] = f;
        bf.job[bf.njobs++] = J;
        continue;
      }
    }
    if (c1s1 && tb.cs) {
      int A = 0, B = 0;
      pick_factors(J.D, std::min(J.nin, J.N), J.nout, &A, &B);
      const long long need = (long long)J.nlines * B * (A + 1) * 2;
      if (A > 0 && cs_used + need <= tb.cs_cap) {
        J.A = A;
        J.B = B;
        J.mode = (B % 2 == 0 && J.nout == J.N) ? 1 : 0;  // pass 2 pairs k, D - k
        J.cs = tb.cs + cs_used;
        cs_used += need;
        b2.job[b2.njobs++] = J;
        continue;
      }
    }
    bd.job[bd.njobs++] = J;
  }
  if (bf.njobs) launch_fft_jobs(bf, fplan, tb, st);
  if (b2.njobs && !launch_two_level_fused(b2, tb.nsm, tb.q_const, st))
    launch_two_level(b2, tb.nsm, tb.q_const, st);
  if (bd.njobs) launch_batch_x(bd, tb, st);
  if (by.njobs) launch_batch_y(by, tb, st);
}

}  // namespace

TcNeed tank_tc_need(const Tables& tb, int most, const std::vector<int>& lines) {
  TcNeed need;
  auto look = [&](int Nx, int Ny, int dir, int nin1, int nin2, int nout1, int nout2) {
    AxisJob p[2] = {};
    set_kind(p[0], axis_kind(0, dir, 0), Nx, nullptr);
    set_kind(p[1], axis_kind(0, dir, 0), Ny, nullptr);
    p[0].nin = nin1;
    p[0].nout = nout1;
    p[0].nlines = nin2;
    p[0].in_sk = 1;
    p[0].in_sl = nin1;
    p[1].nin = nin2;
    p[1].nout = nout2;
    p[1].nlines = p[1].in_sk = nout1;
    p[1].in_sl = 1;
    p[0].gscale = p[1].gscale = 1.0;
    const double alt[2] = {pass_time(p[0], tb, false), pass_time(p[1], tb, true)};
    tc_need(p, alt, 2, tb, most, kMaxJobs, &need);
    tc_need(p + 1, alt + 1, 1, tb, most, kMaxJobs, &need);  // the x pass without a matrix (sin kinds)
  };
  for (int dir : {1, -1}) {
    look(tb.n1, tb.n2, dir, tb.n1, tb.n2, tb.n1, tb.n2);
    look(tb.nd1, tb.nd2, dir, tb.nd1, tb.nd2, tb.nd1, tb.nd2);
  }
  look(tb.nd1, tb.nd2, 1, tb.nd1, tb.nd2, tb.n1, tb.n2);
  look(tb.nd1, tb.nd2, -1, tb.n1, tb.n2, tb.nd1, tb.nd2);
  for (int n : lines) {
    AxisJob y{};
    set_kind(y, K_C1_F2S, tb.n2, nullptr);
    y.nin = y.nout = tb.n2;
    y.nlines = y.in_sk = n;
    y.in_sl = 1;
    y.gscale = 1.0;
    const double alt = pass_time(y, tb, true);
    tc_need(&y, &alt, 1, tb, most, 1, &need);
  }
  return need;
}

void launch_transforms(const XfReq* reqs, int nreq, const Tables& tb, double* const* tmp,
                       cudaStream_t st) {
  // x then y for every request.  (Running the y pass first, where it takes
  // fewer FMAs, was measured slower on the 3-D big grid: the x pass over
  // the extra lines runs at a lower FP64 rate than the y pass it saves.)
  int idx[kMaxJobs];
  for (int r = 0; r < nreq; ++r) idx[r] = r;
  launch_ordered(reqs, idx, nreq, tb, tmp, st);
}

namespace {
__global__ void k_dfma_peak(double* out, int iters, double a, double b) {
  pdl_wait();
  double x0 = threadIdx.x * 1e-3, x1 = x0 + 1, x2 = x0 + 2, x3 = x0 + 3;
  double x4 = x0 + 4, x5 = x0 + 5, x6 = x0 + 6, x7 = x0 + 7;
  for (int i = 0; i < iters; ++i) {
    x0 = fma(x0, a, b); x1 = fma(x1, a, b); x2 = fma(x2, a, b); x3 = fma(x3, a, b);
    x4 = fma(x4, a, b); x5 = fma(x5, a, b); x6 = fma(x6, a, b); x7 = fma(x7, a, b);
  }
  out[blockIdx.x * blockDim.x + threadIdx.x] = x0 + x1 + x2 + x3 + x4 + x5 + x6 + x7;
}
}  // namespace

double measure_fp64_peak_gflops() {
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int blocks = sms * 4, threads = 256, iters = 2048;
  double* out = nullptr;
  if (cudaMalloc(&out, sizeof(double) * blocks * threads) != cudaSuccess) return -1.0;
  cudaEvent_t e0, e1;
  cudaEventCreate(&e0);
  cudaEventCreate(&e1);
  float best = 1e30f;
  for (int rep = 0; rep < 4; ++rep) {
    cudaEventRecord(e0);
    k_dfma_peak<<<blocks, threads>>>(out, iters, 0.999999, 1e-7);
    cudaEventRecord(e1);
    cudaEventSynchronize(e1);
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    if (rep > 0 && ms < best) best = ms;
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  cudaFree(out);
  const double flops = 2.0 * 8.0 * iters * (double)blocks * threads;
  return flops / (best * 1e-3) / 1e9;
}

bool lines_direct(int n, int nlines) { return nlines <= kDirMaxLines && n - 1 <= kDirMaxD; }

// Lines of a launch of direct sums.  Its tiles of 32 outputs go over the SMs in whole
// waves, while 16 lines at a time leave a rest whose sums are cut over idle SMs:
// 17 lines of 3000 points 344 us in one launch, 318 in two; 32 lines 568 and 576.
// The waves of both, and the chunks where they save a fiftieth.
int direct_lines(int D, int nlines, int nsm) {
  constexpr int kChunk = 16;
  if (nlines <= kChunk) return nlines;
  auto waves = [&](int lines) {
    const long long tiles = (long long)lines * ((D / 2 + 1 + 31) / 32), target = 4LL * nsm;
    const int cut = tiles > 0 && tiles < target && D - 1 > 512
                        ? std::min((int)((target + tiles - 1) / tiles), (D - 1 + 255) / 256) : 1;
    return (double)((tiles * cut + nsm - 1) / nsm) / cut;
  };
  const double launch = 0.1;  // of a wave, for the last launch
  const double chunks = nlines / kChunk * waves(kChunk) + (nlines % kChunk ? waves(nlines % kChunk) + launch : 0.0);
  return chunks < 0.98 * waves(nlines) ? kChunk : nlines;
}

// nlines contiguous lines of n points (no context): two-level passes in chunks
// that fit the scratch tb.part where the length factors, else the direct sums.
void launch_lines(const Tables& tb, int dir, int cs, int n, int nlines, const double* in, double* out,
                  cudaStream_t st) {
  AxisJob J{};
  set_kind(J, axis_kind(0, dir, cs), n, tb.q_n1);
  J.nin = J.nout = n;
  J.in_sk = J.out_sk = 1;
  J.in_sl = J.out_sl = n;
  J.gscale = 1.0;
  int A = 0, B = 0;
  if (nlines >= 4) pick_factors(J.D, n, n, &A, &B);
  const long long per = (long long)B * (A + 1) * 2;
  const long long chunk = A > 0 ? tb.part_cap / per : 0;
  // chunks of four lines and more: what is left to a last chunk of fewer is as
  // cheap (16 lines of 8193 points: 2.2 ms by the direct sums, 0.1 ms in chunks of 15)
  const bool two = chunk >= 4;
  const int step = two ? (int)std::min<long long>(chunk, nlines) : direct_lines(J.D, nlines, tb.nsm);
  for (int l0 = 0; l0 < nlines; l0 += step) {
    AxisBatch b{};
    b.njobs = 1;
    b.job[0] = J;
    AxisJob& X = b.job[0];
    X.in = in + (long long)l0 * n;
    X.out = out + (long long)l0 * n;
    X.nlines = std::min(step, nlines - l0);
    if (two) {
      X.A = A;
      X.B = B;
      X.mode = (B % 2 == 0) ? 1 : 0;
      X.cs = tb.part;
      launch_two_level(b, tb.nsm, tb.q_const, st);
    } else {
      launch_batch_x(b, tb, st);
    }
  }
}

void launch_y_f2s(const Tables& tb, const std::vector<YReq>& reqs, int nlines, long long y_stride,
                  long long out_y_stride, cudaStream_t st) {
  for (size_t r0 = 0; r0 < reqs.size(); r0 += kMaxJobs) {
    AxisBatch b{};
    b.njobs = (int)std::min<size_t>(kMaxJobs, reqs.size() - r0);
    for (int i = 0; i < b.njobs; ++i) {
      const YReq& r = reqs[r0 + i];
      AxisJob& J = b.job[i];
      set_kind(J, r.cs ? K_S1_F2S : K_C1_F2S, tb.n2, tb.q_n2);
      J.ty = tb.ty_n2[r.cs ? 1 : 0];
      J.ldy = tb.ldy_n2;
      J.in = r.in;
      J.in_sk = y_stride;
      J.in_sl = 1;
      J.nin = tb.n2;
      J.nlines = nlines;
      J.nout = tb.n2;
      J.out = r.out;
      J.out_sk = out_y_stride;
      J.out_sl = 1;
      J.gscale = 1.0;
    }
    launch_batch_y(b, tb, st);
  }
}

}  // namespace hos
