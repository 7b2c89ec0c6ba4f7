// Sliced-integer operands of the tensor-core sums (sums_tc.cu): power-of-two
// scales, the 7-bit slices of a number, and the coefficient rows, formed and
// sliced by one kernel.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "synth.h"

namespace gem {

// smallest power of two strictly above |x| (1 for 0 or non-finite)
__device__ __forceinline__ double pow2_above(double x) {
  if (!(x > 0.0) || !isfinite(x)) return 1.0;
  int e;
  frexp(x, &e);   // x = f 2^e, f in [0.5, 1)
  return ldexp(1.0, e);
}

// the 7-bit slices of x, |x| < 1: x = sum_i q_i 128^-(i+1) + O(128^-S).  The
// slices are the base-128 digits of u = trunc(|x| 128^S) with the sign of x
// (x 128^S is exact and the conversion truncates), the same digits as S
// rounds of x *= 128, q = trunc(x), x -= q, all of which are exact.
// Of four numbers y = x 128^S: w[i] holds the four bytes of slice i.  The upper
// three digits and the others are spread to bytes and signed four at a time, then
// transposed (about 25 instructions per number for 6 slices; one digit at a time, 80).
template <int NS>
__device__ __forceinline__ void slice_words(const double (&y)[4], unsigned (&w)[NS]) {
  static_assert(NS == 6 || NS == 7, "three digits above 21 or 28 bits");
  constexpr int LOW = 7 * (NS - 3);
  unsigned h[4], g[4];
#pragma unroll
  for (int b = 0; b < 4; ++b) {
    const unsigned long long u = __double2ull_rz(fabs(y[b]));
    const unsigned hi = (unsigned)(u >> LOW), lo = (unsigned)u;
    h[b] = (hi & 0x7fu) | ((hi << 1) & 0x7f00u) | ((hi << 2) & 0x7f0000u);
    g[b] = (lo & 0x7fu) | ((lo << 1) & 0x7f00u) | ((lo << 2) & 0x7f0000u) | (NS == 7 ? (lo << 3) & 0x7f000000u : 0u);
    if (__double2hiint(y[b]) < 0) {   // 128 - d in every byte, then its top bit flipped: -d
      h[b] = (0x80808080u - h[b]) ^ 0x80808080u;
      g[b] = (0x80808080u - g[b]) ^ 0x80808080u;
    }
  }
  auto transpose = [](const unsigned (&a)[4], unsigned& o0, unsigned& o1, unsigned& o2, unsigned& o3) {
    const unsigned p = __byte_perm(a[0], a[1], 0x5140), q = __byte_perm(a[2], a[3], 0x5140);
    const unsigned r = __byte_perm(a[0], a[1], 0x7362), s = __byte_perm(a[2], a[3], 0x7362);
    o0 = __byte_perm(p, q, 0x5410);
    o1 = __byte_perm(p, q, 0x7632);
    o2 = __byte_perm(r, s, 0x5410);
    o3 = __byte_perm(r, s, 0x7632);
  };
  unsigned none;
  transpose(h, w[2], w[1], w[0], none);
  transpose(g, w[NS - 1], w[NS - 2], w[NS - 3], NS == 7 ? w[3] : none);
}

// x 128^S / s of a power of two s, by one product where its factor is exact
struct SliceScale {
  double s, f;
};
template <int NS>
__device__ __forceinline__ SliceScale slice_scale(double s) {
  return {s, s >= 0x1p-900 && s <= 0x1p900 ? (double)(1ull << (7 * NS)) / s : 0.0};
}
template <int NS>
__device__ __forceinline__ double slice_scaled(double x, SliceScale k) {
  return k.f != 0.0 ? x * k.f : x / k.s * (double)(1ull << (7 * NS));
}

__device__ __forceinline__ double block_max(double m) {
  __shared__ double red[32];
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = m;
  __syncthreads();
  m = red[0];
  for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = fmax(m, red[w]);
  __syncthreads();
  return m;
}

// A8[i][row][l] = slice i of A[row][l] s_l / r_row for the row pair (re, im) of
// sum k of frequency slot, r_row the power of two above the row's largest
// |A s_l|.  One block per (slot, sum).  The coefficients A = F::weight times the
// spectrum are never stored: the row's weights stay in shared memory between the
// pass for the largest value and the slicing.  Slices are written up to the end
// of the k-loop of the row's 128-row tile, which is all the products read.
// F: nwn(slot), kind(sum), rank(sum), nsk(kind), nf(), nsum(), weight(slot, sum,
// l) for l < nwn, and index(slot, sum): position of degree 0 in gr and gi.
// Bound: the slices' bytes.  Coefficients to FP64 rows, then slices, took 0.40 +
// 0.52 ms for the coupling at 1000 points (34,440 rows, 883 MB of FP64 written
// once and read twice), 0.22 + 0.30 ms for the regional integrals of 1001
// stations, 0.17 + 0.17 ms for the network; in one kernel 0.41, 0.20 and 0.15 ms.
template <int NS, class F>
__global__ void __launch_bounds__(256) coef_rows_kernel(F f, const float* __restrict__ gr, const float* __restrict__ gi,
                                                        TcCoefSink K) {
  extern __shared__ double wgt[];   // [K.K]
  __shared__ int kext;
  const int k = blockIdx.x % f.nsum(), slot = blockIdx.x / f.nsum();
  const int kind = f.kind(k), nsk = f.nsk(kind), nwn = min(f.nwn(slot), K.K);
  const int row = 2 * (slot * nsk + f.rank(k));
  const int m0 = row / K.tile_rows * K.tile_rows, s0 = m0 / (2 * nsk), s1 = min(f.nf() - 1, (m0 + K.tile_rows - 1) / (2 * nsk));
  if (threadIdx.x == 0) kext = 1;
  __syncthreads();
  for (int s = s0 + threadIdx.x; s <= s1; s += blockDim.x) atomicMax(&kext, min(f.nwn(s), K.K));
  const double* sl = K.lscale + (long long)kind * K.Kp;
  const long long o = f.index(slot, k);
  double mr = 0.0, mi = 0.0;
  for (int l = threadIdx.x; l < nwn; l += blockDim.x) {
    const double w = f.weight(slot, k, l);
    wgt[l] = w;
    mr = fmax(mr, fabs(w * (double)gr[o + l] * sl[l]));
    mi = fmax(mi, fabs(w * (double)gi[o + l] * sl[l]));
  }
  const double rr = pow2_above(block_max(mr)), ri = pow2_above(block_max(mi));   // the barriers publish wgt and kext
  const SliceScale kr = slice_scale<NS>(rr), ki = slice_scale<NS>(ri);
  const long long r0 = K.rowoff[kind] + row, plane = K.mtot * K.Kp;
  if (threadIdx.x == 0) { K.rscale[r0] = rr; K.rscale[r0 + 1] = ri; }
  const int end = (kext + K.tile_k - 1) / K.tile_k * K.tile_k;   // <= Kp
  for (int l0 = 4 * threadIdx.x; l0 < end; l0 += 4 * blockDim.x) {
    double yr[4] = {}, yi[4] = {};
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int l = l0 + b;
      if (l < nwn) {
        yr[b] = slice_scaled<NS>(wgt[l] * (double)gr[o + l] * sl[l], kr);
        yi[b] = slice_scaled<NS>(wgt[l] * (double)gi[o + l] * sl[l], ki);
      }
    }
    unsigned qr[NS], qi[NS];
    slice_words<NS>(yr, qr);
    slice_words<NS>(yi, qi);
    signed char* a = K.A8 + r0 * K.Kp + l0;
#pragma unroll
    for (int i = 0; i < NS; ++i) {
      *reinterpret_cast<unsigned*>(a + i * plane) = qr[i];
      *reinterpret_cast<unsigned*>(a + i * plane + K.Kp) = qi[i];
    }
  }
}

template <class F>
cudaError_t coef_rows_launch(const F& f, int nblocks, const float* gr, const float* gi, const TcCoefSink& K, cudaStream_t st) {
  const size_t smem = (size_t)K.K * sizeof(double);
  auto go = [&](auto kern) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    kern<<<nblocks, 256, smem, st>>>(f, gr, gi, K);
    return cudaGetLastError();
  };
  return K.nslice == 7 ? go(coef_rows_kernel<7, F>) : go(coef_rows_kernel<6, F>);
}

}  // namespace gem
