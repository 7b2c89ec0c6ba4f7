// Associated Legendre functions P_l^m, l = 0..lmax, of 32 angles per block
// (legendreFunctions.f90:48-157), handed degree by degree to a functor that
// forms and stores the tables made of them.
//
// The upward recurrence is written as
//   p_l = alpha_l p_{l-1} + beta_l p_{l-2},
//   alpha_l = ct (2l - 1) / (l - m),  beta_l = -(l + m - 1) / (l - m),
// with 1/(l - m) read from a shared-memory table, so one FMA per degree sits on
// the dependent chain.  (The plain kernels divide by (l - m) at every degree;
// the values differ by rounding only, relative 1e-13 at l = 3200: the recurrence
// is the dominant solution and does not amplify them.)
//
// The chain is serial in l and there are only 3 angles' worth of chains per
// column (m = 0, 1, 2), too few to fill the chip with the derivatives, the
// exponents and the stores of the tables as well: one thread per chain that did
// all of it was bound by its own instructions (0.26 ms for 4000 stations x 3072
// degrees with exponents, 0.18 without, where the stores need 0.13; 0.38 and
// 0.19 ms for 1000 points of the coupling, 13 tables).  So one warp runs the
// chains of 32 columns a chunk of degrees ahead, through shared memory, of
// LC_OUT warps that form and store the tables: 0.20 and 0.15 ms with exponents.
#pragma once
#include <cuda_runtime.h>

namespace gem {

constexpr int LC_CHUNK = 32, LC_OUT = 8, LC_THREADS = 32 * (LC_OUT + 1);

// dynamic shared memory; the limit leaves room for the chunk buffers
inline size_t legendre_chain_bytes(int lmax) { return (size_t)(lmax + 1) * sizeof(double); }
inline bool legendre_chain_supported(int lmax) { return legendre_chain_bytes(lmax) <= 200 * 1024; }

// Of one block: order m, angle cosine and sine of this lane's column; out(l, p_l,
// p_{l-1}) is called for every degree by one of the output warps.  Poles (sin = 0)
// keep the plain form's division.  All LC_THREADS threads take part.
template <class Out>
__device__ __forceinline__ void legendre_chain(int m, int lmax, double ct, double st, Out&& out) {
  extern __shared__ double rcp[];   // rcp[n] = 1/n, n = 1..lmax
  __shared__ double buf[2][LC_CHUNK + 1][32];   // degrees l0 - 1 .. l0 + LC_CHUNK - 1
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int n = threadIdx.x + 1; n <= lmax; n += blockDim.x) rcp[n] = 1.0 / (double)n;
  __syncthreads();
  const bool pole = !(st > 0.0);
  const bool anypole = __any_sync(0xffffffffu, pole);
  double pmm = 1.0, fact = 1.0;
  for (int j = 1; j <= m; ++j) { pmm = pmm * fact * st; fact = fact + 2.0; }
  double pl2 = 0.0, pl1 = 0.0;
  const double mm1 = (double)(m - 1);
  const int nchunk = lmax / LC_CHUNK + 1;
  auto step = [&](int l, double r) {
    const double dl = (double)l;
    const double alpha = ct * fma(2.0, dl, -1.0) * r;
    const double bp = -(dl + mm1) * r * pl2;   // off the chain: pl2 is known a degree early
    return fma(alpha, pl1, bp);
  };
  for (int c = 0; c <= nchunk; ++c) {
    if (warp == 0 && c < nchunk) {
      const int l0 = c * LC_CHUNK, n = min(LC_CHUNK, lmax + 1 - l0);
      double(*b)[32] = buf[c & 1];
      b[0][lane] = pl1;
      if (l0 >= m + 2 && n == LC_CHUNK && !anypole) {
        const double* r = rcp + (l0 - m);
#pragma unroll 8
        for (int i = 0; i < LC_CHUNK; ++i) {
          const double p = step(l0 + i, r[i]);
          b[i + 1][lane] = p;
          pl2 = pl1;
          pl1 = p;
        }
      } else {
        for (int i = 0; i < n; ++i) {
          const int l = l0 + i;
          double p;
          if (l < m) p = 0.0;
          else if (l == m) p = pmm;
          else if (l == m + 1) p = ct * (double)(2 * m + 1) * pmm;
          else if (pole) p = (ct * (double)(2 * l - 1) * pl1 - (double)(l + m - 1) * pl2) / (double)(l - m);
          else p = step(l, rcp[l - m]);
          b[i + 1][lane] = p;
          pl2 = pl1;
          pl1 = p;
        }
      }
    }
    if (warp > 0 && c > 0) {
      const int l0 = (c - 1) * LC_CHUNK, n = min(LC_CHUNK, lmax + 1 - l0);
      const double(*b)[32] = buf[(c - 1) & 1];
      for (int i = warp - 1; i < n; i += LC_OUT) out(l0 + i, b[i + 1][lane], b[i][lane]);
    }
    __syncthreads();
  }
}

}  // namespace gem
