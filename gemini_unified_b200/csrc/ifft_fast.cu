// Inverse FFT of real seismogram traces, fast form (FP64, FMA).
//
// Computes the same time series as transformFrequencyTime (frequencyTime.f90:
// 55-113): the Hermitian spectrum of bins nf1..nf2, its unnormalised inverse
// transform of length N = ns, then ts(i) = x(ndec*(i-1)+1) * df * fac(i).  The
// reference runs a radix-2 transform with twiddle angles built on the
// single-precision pi (fourierTransform.f90:128-147); this form evaluates the
// exact inverse DFT, which differs from it by about 1e-7 relative.
//
// Real output from a half-length complex transform: with H = N/2,
//   Z_k = (X_k + conj X_{H-k}) + i w^k (X_k - conj X_{H-k}),  w = e^{2 pi i/N},
//   z_n = sum_k Z_k e^{2 pi i kn/H},  x_{2n} = Re z_n,  x_{2n+1} = Im z_n,
// where X_{H-k} stands for X_{k+H} of the Hermitian spectrum.  One CTA of T =
// H/16 threads per trace; each thread keeps 16 points in registers per pass and
// the passes exchange through shared memory.  With k = T d2 + RB d1 + d0 and n =
// o2 + 16 o1 + 256 o0 (RB = H/256),
//   z_n = sum_d0 e^{2 pi i d0 (o2 + 16 o1)/H} e^{2 pi i d0 o0/RB}
//         sum_d1 e^{2 pi i d1 o2/256} e^{2 pi i d1 o1/16} sum_d2 e^{2 pi i d2 o2/16} Z_k:
// radix 16, 16 and RB, each pass writing where it read, so that one barrier
// separates two passes (an autosorting transform needs two) and the last one
// leaves consecutive threads consecutive samples.
//
// Bound: the FP64 pipe (580 instructions per thread and trace of 4096 points, 2 clocks each) and
// the L1 pipe (340 wavefronts per warp), each busy half of the time with the 16 warps per SM that
// the points' registers leave.  So the butterflies are those of radix 2 in FMA form, p = a + w b
// and 2 a - p, 6 instructions with the twiddle factor included; a radix-16 pass with its 15
// twiddles needs 208 that way and 4 loads (268 and 3 in a 4 x 4 split).  12,001 traces of 8192
// samples from 410 bins: 0.254 -> 0.212 ms (three CTAs per SM of 80 registers spill: 0.240; one
// trace per CTA, nothing fetched ahead: 0.221); 72,000: 1.42 -> 1.20 ms (2.4 GB written).  9009 traces
// of 2048 samples, band above 1/16, one trace per CTA, 128 registers and loads without a branch
// around them: 0.129 -> 0.079 ms (many traces per CTA: 0.177).
#include <cuda_runtime.h>

#include <algorithm>

#include "synth.h"

namespace gem {

namespace {

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 times_i(double2 a) { return make_double2(-a.y, a.x); }

constexpr double C16 = 0.92387953251128675613, S16 = 0.38268343236508977173, R8 = 0.70710678118654752440;

// (a, b) <- (a + w b, a - w b)
__device__ __forceinline__ void bf(double2& a, double2& b, double2 w) {
  const double2 p = make_double2(fma(-w.y, b.y, fma(w.x, b.x, a.x)), fma(w.y, b.x, fma(w.x, b.y, a.y)));
  b = make_double2(fma(2.0, a.x, -p.x), fma(2.0, a.y, -p.y));
  a = p;
}
__device__ __forceinline__ void bf_i(double2& a, double2& b, double2 w) {   // i w for w
  b = times_i(b);
  bf(a, b, w);
}
__device__ __forceinline__ void bf(double2& a, double2& b) {   // w = 1
  const double2 p = make_double2(a.x + b.x, a.y + b.y);
  b = make_double2(a.x - b.x, a.y - b.y);
  a = p;
}
__device__ __forceinline__ void bf_i(double2& a, double2& b) {   // w = i
  b = times_i(b);
  bf(a, b);
}
__device__ __forceinline__ double2 times_w8(double2 w) { return make_double2((w.x - w.y) * R8, (w.x + w.y) * R8); }
__device__ __forceinline__ double2 times_w16(double2 w) { return cmul(w, make_double2(C16, S16)); }

// out_o = sum_{r < R} w^r v_r e^{2 pi i r o/R}, left in v[rev<R>(o)].  The pairs (r, r +
// R/2) meet with w^{R/2}; the sums go on with w for the even o, the differences with w
// e^{2 pi i/R} for the odd.  w1, w2, w4, w8: powers of w.
template <int R>
__device__ __forceinline__ constexpr int rev(int o) {
  int q = 0;
  for (int b = 1; b < R; b <<= 1) q = 2 * q + ((o & b) != 0);
  return q;
}
__device__ __forceinline__ void dft_tw(double2 (&v)[16], double2 w1, double2 w2, double2 w4, double2 w8) {
#pragma unroll
  for (int r = 0; r < 8; ++r) bf(v[r], v[r + 8], w8);
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    bf(v[r], v[r + 4], w4);
    bf_i(v[r + 8], v[r + 12], w4);
  }
  const double2 w2b = times_w8(w2);
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    bf(v[r], v[r + 2], w2);
    bf_i(v[r + 4], v[r + 6], w2);
    bf(v[r + 8], v[r + 10], w2b);
    bf_i(v[r + 12], v[r + 14], w2b);
  }
  const double2 wb = times_w8(w1), wc = times_w16(w1), wd = times_w16(wb);
  bf(v[0], v[1], w1);
  bf_i(v[2], v[3], w1);
  bf(v[4], v[5], wb);
  bf_i(v[6], v[7], wb);
  bf(v[8], v[9], wc);
  bf_i(v[10], v[11], wc);
  bf(v[12], v[13], wd);
  bf_i(v[14], v[15], wd);
}
__device__ __forceinline__ void dft_tw(double2 (&v)[8], double2 w1, double2 w2, double2 w4, double2) {
#pragma unroll
  for (int r = 0; r < 4; ++r) bf(v[r], v[r + 4], w4);
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    bf(v[r], v[r + 2], w2);
    bf_i(v[r + 4], v[r + 6], w2);
  }
  const double2 wb = times_w8(w1);
  bf(v[0], v[1], w1);
  bf_i(v[2], v[3], w1);
  bf(v[4], v[5], wb);
  bf_i(v[6], v[7], wb);
}
__device__ __forceinline__ void dft_tw(double2 (&v)[4], double2 w1, double2 w2, double2, double2) {
  bf(v[0], v[2], w2);
  bf(v[1], v[3], w2);
  bf(v[0], v[1], w1);
  bf_i(v[2], v[3], w1);
}
__device__ __forceinline__ void dft_tw(double2 (&v)[2], double2 w1, double2, double2, double2) { bf(v[0], v[1], w1); }

// the first pass, w = 1.  BAND: only v0, v1, v14 and v15 are not zero, whose first
// two levels are copies
template <bool BAND>
__device__ __forceinline__ void dft16(double2 (&v)[16]) {
  if constexpr (BAND) {
    auto minus = [](double2 a) { return make_double2(-a.x, -a.y); };
    const double2 a = v[14], b = v[15];
    v[2] = a; v[3] = b;
    v[4] = v[0]; v[5] = v[1]; v[6] = minus(a); v[7] = minus(b);
    v[12] = v[8] = v[0]; v[13] = v[9] = v[1];
    v[14] = times_i(a); v[15] = times_i(b);
    v[10] = minus(v[14]); v[11] = minus(v[15]);
  } else {
#pragma unroll
    for (int r = 0; r < 8; ++r) bf(v[r], v[r + 8]);
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      bf(v[r], v[r + 4]);
      bf_i(v[r + 8], v[r + 12]);
    }
  }
  const double2 w8 = make_double2(R8, R8), w16 = make_double2(C16, S16), w163 = make_double2(S16, C16);
#pragma unroll
  for (int r = 0; r < 2; ++r) {
    bf(v[r], v[r + 2]);
    bf_i(v[r + 4], v[r + 6]);
    bf(v[r + 8], v[r + 10], w8);
    bf_i(v[r + 12], v[r + 14], w8);
  }
  bf(v[0], v[1]);
  bf_i(v[2], v[3]);
  bf(v[4], v[5], w8);
  bf_i(v[6], v[7], w8);
  bf(v[8], v[9], w16);
  bf_i(v[10], v[11], w16);
  bf(v[12], v[13], w163);
  bf_i(v[14], v[15], w163);
}

}  // namespace

// tw[m] = e^{2 pi i m / N}, m < N, then the pass tables: tw + N + IFFT_TWA for the
// pass (NS 16, R 16) and tw + N + IFFT_TWB for the last pass (NS 256, R H/256),
// entry (r - 1) NS + k = e^{2 pi i r k / (NS R)}.  Both angles are the same double
// as the m = r k N / (NS R) of the full table, so the entries equal tw[m].
// fac[i] = e^{arg i}, arg = sigma times the sampling interval: the reference's running product
// (frequencyTime.f90:105-110) is one dependent chain of nsamp multiplications, 46 us of one thread
// for 8192 samples, and departs from the exponential by the rounding of its base times i.
__global__ void ifft_fast_twiddles(int N, double2* tw, int nsamp, double arg, double* fac) {
  const int H = N / 2, RB = H / 256;
  for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < N + IFFT_TW_EXTRA; m += blockDim.x * gridDim.x) {
    long long num = 0, den = 1;
    if (m < N) {
      num = m; den = N;
    } else if (m < N + IFFT_TWB) {
      const int a = m - N - IFFT_TWA;
      if (a < 15 * 16) { num = (long long)(a / 16 + 1) * (a % 16); den = 256; }
    } else {
      const int b = m - N - IFFT_TWB;
      if (b < (RB - 1) * 256) { num = (long long)(b / 256 + 1) * (b % 256); den = 256LL * RB; }
    }
    double s, c;
    sincospi(2.0 * (double)num / (double)den, &s, &c);
    tw[m] = make_double2(c, s);
  }
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nsamp; i += blockDim.x * gridDim.x) fac[i] = exp(arg * (double)i);
}

// keeps what follows from a loop-invariant value inside the loop: hoisted twiddle products
// would take the registers of the 16 points
__device__ __forceinline__ void in_loop(double2& a) { asm volatile("" : "+d"(a.x), "+d"(a.y)); }
__device__ __forceinline__ double2 load_in_loop(const double2* p) {
  double2 a;
  asm volatile("ld.global.nc.v2.f64 {%0, %1}, [%2];" : "=d"(a.x), "=d"(a.y) : "l"(p));
  return a;
}

// BAND: the band's bins lie below H/8, so that Z_k is not zero for k < 2 T and k > H - 2 T only.
// H = 4096: a CTA runs over the traces blockIdx.x, + gridDim.x, ..., and with BAND loads the next
// trace's bins while the current one is transformed; else one trace per CTA.  128 registers.
template <int H, bool BAND>
__global__ void __launch_bounds__(H / 16, H == 256 ? 16 : 8192 / H) ifft_fast_kernel(SynthDev S, long long ntr,
                                                          const double2* __restrict__ X,
                                                          const double2* __restrict__ tw,
                                                          const double* __restrict__ fac, float* traces) {
  constexpr bool MANY = H == 4096;   // more than one trace per CTA
  extern __shared__ double2 buf[];   // point p = T d2 + RB d1 + d0 at p + d2: the last pass reads along d2
  constexpr int T = H / 16, RB = H / 256;
  const int N = 2 * H;
  const int tid = threadIdx.x;
  const int lo = S.nf1 - 1, hi = S.nf2 - 1;   // 0-based bins of the spectrum
  const double2 zero = make_double2(0.0, 0.0);
  double2 in[4];
  auto fetch = [&](long long tr) {   // bins k and H - k of the blocks r = 0, 1 and 14, 15
    const double2* x = X + tr * S.ldx;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
      const int k = tid + r * T, kk = (2 - r) * T - tid;
      in[r] = (k >= lo && k <= hi) ? x[k] : zero;
      in[r + 2] = (kk >= lo && kk <= hi) ? x[kk] : zero;
    }
  };
  if (BAND && MANY) fetch(blockIdx.x);
  double2 w0 = tw[tid];
  double2 wb1 = RB == 16 ? tw[N + IFFT_TWB + tid] : zero;
  // H = 4096, ndec = 1: the last pass leaves thread tid the samples 2 tid + 512 q (+1), whose factors are
  // df fac(2 tid) fac(512)^q (+1), formed by products instead of 32 table loads (a few ulps of a double)
  const bool ratios = H == 4096 && S.ndec == 1 && S.nsamp > 512;
  const bool pairs = (S.nsamp & 1) == 0 && (reinterpret_cast<size_t>(traces) & 7) == 0;   // 8-byte stores
  for (long long tr = blockIdx.x; tr < ntr; tr += gridDim.x) {
    double2 v[16];
    in_loop(w0);
    in_loop(wb1);
    // ---- pass over d2: Z_k formed on the fly, k = tid + r T
    if constexpr (BAND) {
      if (!MANY) fetch(tr);
#pragma unroll
      for (int r = 0; r < 2; ++r) {   // e^{2 pi i k/N} = w0 e^{2 pi i r/32}
        constexpr double C1 = 0.98078528040323044913, S1 = 0.19509032201612826785;
        const double2 w = r ? cmul(w0, make_double2(C1, S1)) : w0;
        const double2 u = cmul(w0, r ? make_double2(-C1, S1) : make_double2(-C16, S16));
        const double2 a = in[r], b = make_double2(in[r + 2].x, -in[r + 2].y);
        v[r] = make_double2(a.x - w.y * a.x - w.x * a.y, a.y + w.x * a.x - w.y * a.y);
        v[r + 14] = make_double2(b.x + u.y * b.x + u.x * b.y, b.y - u.x * b.x + u.y * b.y);
      }
      if (MANY && tr + gridDim.x < ntr) fetch(tr + gridDim.x);
    } else {
      // Z = s + i w d of the bins k and H - k; the loads carry no branch, so that they are in flight together
      const double2* x = X + tr * S.ldx;
#pragma unroll
      for (int r = 0; r < 16; ++r) {
        const int k = tid + r * T, kk = H - k;
        const double2 a = (k >= lo && k <= hi) ? x[k] : zero;
        double2 b = (k > 0 && kk >= lo && kk <= hi) ? x[kk] : zero;
        b.y = -b.y;
        const double2 s = make_double2(a.x + b.x, a.y + b.y), d = make_double2(a.x - b.x, a.y - b.y), w = tw[k];
        v[r] = make_double2(s.x - w.y * d.x - w.x * d.y, s.y + w.x * d.x - w.y * d.y);
      }
    }
    dft16<BAND>(v);
#pragma unroll
    for (int o = 0; o < 16; ++o) buf[o * (T + 1) + tid] = v[rev<16>(o)];
    __syncthreads();
    // ---- pass over d1 of (o2, d0)
    {
      const int o2 = tid / RB;
      double2* p = buf + o2 * (T + 1) + tid % RB;
      const double2* t = tw + N + IFFT_TWA + o2;
#pragma unroll
      for (int r = 0; r < 16; ++r) v[r] = p[r * RB];
      dft_tw(v, load_in_loop(t), load_in_loop(t + 16), load_in_loop(t + 3 * 16), load_in_loop(t + 7 * 16));
      if constexpr (RB > 1) {
#pragma unroll
        for (int o = 0; o < 16; ++o) p[o * RB] = v[rev<16>(o)];
      }
      __syncthreads();
    }
    // ---- pass over d0 of j = o2 + 16 o1: out_of(q) is then the point n = tid + q T
    if constexpr (RB > 1) {
#pragma unroll
      for (int b = 0; b < 16 / RB; ++b) {
        const int j = tid + b * T;
        const double2* p = buf + (j % 16) * (T + 1) + j / 16 * RB;
        double2 u[RB];
#pragma unroll
        for (int r = 0; r < RB; ++r) u[r] = p[r];
        if constexpr (RB == 16) {
          { const double2 w4 = load_in_loop(tw + N + IFFT_TWB + 3 * 256 + tid); dft_tw(u, wb1, cmul(wb1, wb1), w4, cmul(w4, w4)); }
        } else {
          const double2* t = tw + N + IFFT_TWB + j;
          const double2 w1 = load_in_loop(t);
          dft_tw(u, w1, RB > 2 ? load_in_loop(t + 256) : w1, RB > 4 ? load_in_loop(t + 3 * 256) : w1, w1);
        }
#pragma unroll
        for (int o = 0; o < RB; ++o) v[b + o * (16 / RB)] = u[rev<RB>(o)];
      }
      if (MANY) __syncthreads();   // the next trace writes the buffer
    }
    auto out_of = [&](int q) -> double2 { return RB > 1 ? v[q] : v[rev<16>(q)]; };
    // ---- x_{2n} = Re z_n, x_{2n+1} = Im z_n; ts(i) = x(ndec i) df fac(i)
    float* out = traces + tr * S.nsamp;
    const int ndec = S.ndec;
    if (ratios) {
      const double2 f01 = load_in_loop(reinterpret_cast<const double2*>(fac + 2 * tid));
      double ratio;
      asm volatile("ld.global.nc.f64 %0, [%1];" : "=d"(ratio) : "l"(fac + 512));
      double g0 = S.df * f01.x, g1 = S.df * f01.y;
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const double2 z = out_of(q);
        const int t0 = 2 * tid + 512 * q, t1 = t0 + 1;
        const float y0 = (float)(z.x * g0), y1 = (float)(z.y * g1);
        if (pairs) {
          if (t1 < S.nsamp) *reinterpret_cast<float2*>(out + t0) = make_float2(y0, y1);
        } else {
          if (t0 < S.nsamp) out[t0] = y0;
          if (t1 < S.nsamp) out[t1] = y1;
        }
        g0 *= ratio;
        g1 *= ratio;
      }
      continue;
    }
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const double2 z = out_of(q);
      const int n = tid + q * T;
      const int t0 = 2 * n, t1 = 2 * n + 1;
      if (ndec == 1) {
        if (t1 < S.nsamp) {
          const double2 f = *reinterpret_cast<const double2*>(fac + t0);   // t0 even: 16-byte aligned
          const float y0 = (float)(z.x * S.df * f.x), y1 = (float)(z.y * S.df * f.y);
          if (pairs) {
            *reinterpret_cast<float2*>(out + t0) = make_float2(y0, y1);
          } else {
            out[t0] = y0;
            out[t1] = y1;
          }
        } else if (t0 < S.nsamp) {
          out[t0] = (float)(z.x * S.df * fac[t0]);
        }
      } else {
        if (t0 % ndec == 0 && t0 / ndec < S.nsamp) out[t0 / ndec] = (float)(z.x * S.df * fac[t0 / ndec]);
        if (t1 % ndec == 0 && t1 / ndec < S.nsamp) out[t1 / ndec] = (float)(z.y * S.df * fac[t1 / ndec]);
      }
    }
    if (!MANY) return;
  }
}

// Launch: ns in 512..8192.  tw: the ns + IFFT_TW_EXTRA twiddles of ifft_fast_twiddles; fac: nsamp factors.
cudaError_t ifft_fast_launch(const SynthDev& S, long long ntr, const double2* X, const double2* tw, const double* fac,
                             float* traces, cudaStream_t st) {
  const int H = S.ns / 2;
  const size_t smem = (size_t)(H + 16) * sizeof(double2);
  const bool band = S.nf2 - 1 < H / 8;   // the first pass has 4 blocks of 16 that are not zero: 84 of 148 instructions, no partner bins
  auto go = [&](auto kern, int threads) -> cudaError_t {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e == cudaSuccess)   // all of the unified L1 as shared memory: more CTAs of the longest transforms per SM
      e = cudaFuncSetAttribute(kern, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);
    if (e != cudaSuccess) return e;
    int dev = 0, sms = 0, per = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess ||
        (e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess ||
        (e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kern, threads, smem)) != cudaSuccess)
      return e;
    const long long grid = H == 4096 ? std::min<long long>(ntr, (long long)sms * std::max(per, 1)) : ntr;
    kern<<<(unsigned)grid, threads, smem, st>>>(S, ntr, X, tw, fac, traces);
    return cudaGetLastError();
  };
  switch (H) {
    case 256: return band ? go(ifft_fast_kernel<256, true>, 16) : go(ifft_fast_kernel<256, false>, 16);
    case 512: return band ? go(ifft_fast_kernel<512, true>, 32) : go(ifft_fast_kernel<512, false>, 32);
    case 1024: return band ? go(ifft_fast_kernel<1024, true>, 64) : go(ifft_fast_kernel<1024, false>, 64);
    case 2048: return band ? go(ifft_fast_kernel<2048, true>, 128) : go(ifft_fast_kernel<2048, false>, 128);
    case 4096: return band ? go(ifft_fast_kernel<4096, true>, 256) : go(ifft_fast_kernel<4096, false>, 256);
    default: return cudaErrorInvalidValue;
  }
}

cudaError_t ifft_fast_twiddles_launch(int N, double2* tw, int nsamp, double arg, double* fac, cudaStream_t st) {
  ifft_fast_twiddles<<<(N + IFFT_TW_EXTRA + 255) / 256, 256, 0, st>>>(N, tw, nsamp, arg, fac);
  return cudaGetLastError();
}

}  // namespace gem
