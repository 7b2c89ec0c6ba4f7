// Legendre tables of the fast form (legendreFunctions.f90:48-157).
//
// Same tables as legendre_kernel (synth.cu): tab[(kind * lcap + l) * nsta + sta],
// and their binary exponents for the scales of the tensor-core sums,
// with kinds plm_m (m), dP/dtheta (3 + m) and P/sin(theta) (5 + m), from the
// chains of legendre_chain.cuh.
#include <cuda_runtime.h>

#include "legendre_chain.cuh"
#include "synth.h"

namespace gem {

namespace {

// block (32 stations, m); 4000 stations x 3260 degrees: 0.20 ms (0.84 GB of tables
// and 0.21 GB of exponents)
__global__ void __launch_bounds__(LC_THREADS) legendre_fast_kernel(int nsta, int lmax, int lcap,
                                                                   const double* __restrict__ theta,
                                                                   double* __restrict__ tab,
                                                                   short* __restrict__ texp) {
  const int m = blockIdx.y, sta = blockIdx.x * 32 + (threadIdx.x & 31);
  const double th = theta[min(sta, nsta - 1)];
  const double ct = cos(th), st = sin(th), rst = 1.0 / st;
  const bool pole = !(st > 0.0);
  const double isct = ct >= 0.0 ? 1.0 : -1.0, md = (double)m;
  const long long plane = (long long)lcap * nsta;
  const long long op = m * plane + sta, od = (3 + m) * plane + sta, os = (5 + m) * plane + sta;
  legendre_chain(m, lmax, ct, st, [&](int l, double p, double pl1) {
    if (sta >= nsta) return;
    const double dl = (double)l;
    double dp, ps;
    if (!pole) {
      dp = l < m ? 0.0 : fma(dl * ct, p, -(dl + md) * pl1) * rst;
      ps = p * rst;
    } else {   // legendreFunctions.f90:116-127
      const double q = m == 1 ? 0.5 * (dl * (dl + 1.0)) : 0.0, odd = l & 1 ? isct : 1.0;
      dp = q * odd;
      ps = q * (l & 1 ? 1.0 : isct);
    }
    const long long o = (long long)l * nsta;
    tab[op + o] = p;
    texp[op + o] = tc_exponent(p);
    tab[od + o] = dp;
    texp[od + o] = tc_exponent(dp);
    if (m >= 1) {
      tab[os + o] = ps;
      texp[os + o] = tc_exponent(ps);
    }
  });
}

}  // namespace

bool legendre_fast_supported(int lmax) { return legendre_chain_supported(lmax); }

cudaError_t legendre_fast_launch(int nsta, int lmax, int lcap, const double* theta, double* tab, short* texp,
                                 cudaStream_t st) {
  const size_t smem = legendre_chain_bytes(lmax);
  if (!legendre_fast_supported(lmax)) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(legendre_fast_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  legendre_fast_kernel<<<dim3((nsta + 31) / 32, 3), LC_THREADS, smem, st>>>(nsta, lmax, lcap, theta, tab, texp);
  return cudaGetLastError();
}

}  // namespace gem
