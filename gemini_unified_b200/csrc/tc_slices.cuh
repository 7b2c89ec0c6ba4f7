// Sliced-integer operands of the tensor-core sums (sums_tc.cu): power-of-two
// scales, the 7-bit slices of a number, and the coefficient rows, formed and
// sliced by one kernel.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

#include "synth.h"

namespace gem {

// finite non-zero exponent, else 0
__device__ __forceinline__ int tc_finite(short e) { return e == 2047 ? 0 : e; }

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

// Scale 2^(e - 1022) of a row from its largest finite biased exponent e (no number above
// the subnormals: 1), and 128^S over it as two factors of half
// the shift, whose products with the row's numbers are exact
struct SliceScale {
  double s, f1, f2;
};
template <int NS>
__device__ __forceinline__ SliceScale slice_scale(int e) {
  if (e == 0) e = 1022;
  const int shift = 7 * NS - (e - 1022), a = shift / 2;
  auto pow2 = [](int n) { return __hiloint2double((1023 + n) << 20, 0); };
  return {pow2(e - 1022), pow2(a), pow2(shift - a)};
}

// A8[i][row][l] = slice i of A[row][l] s_l / r_row for the row pair (re, im) of
// sum k of frequency slot, r_row the power of two above the row's largest
// |A s_l|.  One block per (sum, slot).  The coefficients A = F's weight times the
// spectrum are never stored: the products stay in registers between the pass for
// the largest value and the slicing.  Slices are written up to the end
// of the k-loop of the row's 128-row tile, which is all the products read.
// F: nwn(slot), kind(sum), rank(sum), nsk(kind), nf(), row(slot,
// sum): the weights w(l), w.l0 <= l < nwn, and index(slot, sum): position of degree 0 in gr and gi.
// Bound: the slices' bytes.  Coefficients to FP64 rows, then slices, took 0.40 +
// 0.52 ms for the coupling at 1000 points (34,440 rows, 883 MB of FP64 written
// once and read twice), 0.22 + 0.30 ms for the regional integrals of 1001
// stations, 0.17 + 0.17 ms for the network; in one kernel that passed twice over
// the spectrum, weights in shared memory, 0.40, 0.20 and 0.14 ms, bound by its
// instructions (taper cosines per sum, divisions per block, scales by maxima of
// doubles).  Each thread now keeps the products of 4 R degrees between the passes,
// the scales come from the largest exponents behind one barrier, and the tapers from
// a table that the sums of a frequency share: 0.31, 0.14 and 0.10 ms.
template <int NS, int R, class F>
__global__ void __launch_bounds__(512, 2) coef_rows_kernel(F f, const float* __restrict__ gr, const float* __restrict__ gi,
                                                           TcCoefSink K) {
  __shared__ int red[2][16], tile_ext;
  const int k = blockIdx.x, slot = blockIdx.y;
  const int kind = f.kind(k), nsk = f.nsk(kind), nwn = min(f.nwn(slot), K.K);
  const int row = 2 * (slot * nsk + f.rank(k));
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
  const double* sl = K.lscale + (long long)kind * K.Kp;
  const long long o = f.index(slot, k);
  const float *pr = gr + o, *pi = gi + o;
  const auto weight = f.row(slot, k);
  if (warp == nwarp - 1) {   // largest count of the rows' tile
    const int m0 = row / K.tile_rows * K.tile_rows, s0 = m0 / (2 * nsk), s1 = min(f.nf() - 1, (m0 + K.tile_rows - 1) / (2 * nsk));
    int kext = 1;
    for (int s = s0 + lane; s <= s1; s += 32) kext = max(kext, min(f.nwn(s), K.K));
    kext = __reduce_max_sync(0xffffffffu, kext);
    if (lane == 0) tile_ext = kext;
  }
  int er = 0, ei = 0;   // upper words of the rows' largest finite absolute values
  double vr[R][4], vi[R][4];
  auto load = [&](int base) {
#pragma unroll
    for (int c = 0; c < R; ++c) {
      const int l0 = base + 4 * (threadIdx.x + c * blockDim.x);
#pragma unroll
      for (int b = 0; b < 4; ++b) vr[c][b] = vi[c][b] = 0.0;
      if (l0 >= nwn) continue;
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int l = l0 + b;
        if (l < nwn && l >= weight.l0) {   // a spectrum need not be defined below a sum's first degree
          const double w = weight(l), s = sl[l];
          vr[c][b] = w * (double)pr[l] * s;
          vi[c][b] = w * (double)pi[l] * s;
        }
      }
    }
  };
  const int part = 4 * R * blockDim.x;
  int base = 0;
  do {   // once for a frequency without degrees too: its products are the zeros that load() sets
    load(base);
#pragma unroll
    for (int c = 0; c < R; ++c)
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        const int hr = __double2hiint(vr[c][b]) & 0x7fffffff, hi = __double2hiint(vi[c][b]) & 0x7fffffff;
        er = max(er, hr < 0x7ff00000 ? hr : 0);
        ei = max(ei, hi < 0x7ff00000 ? hi : 0);
      }
    base += part;
  } while (base < nwn);
  er = __reduce_max_sync(0xffffffffu, er);
  ei = __reduce_max_sync(0xffffffffu, ei);
  if (lane == 0) { red[0][warp] = er; red[1][warp] = ei; }
  __syncthreads();
  const int q = min(lane, nwarp - 1);
  er = __reduce_max_sync(0xffffffffu, red[0][q]) >> 20;
  ei = __reduce_max_sync(0xffffffffu, red[1][q]) >> 20;
  const SliceScale kr = slice_scale<NS>(er), ki = slice_scale<NS>(ei);
  const long long r0 = K.rowoff[kind] + row, plane = K.mtot * K.Kp;
  if (threadIdx.x == 0) { K.rscale[r0] = kr.s; K.rscale[r0 + 1] = ki.s; }
  const int end = (tile_ext + K.tile_k - 1) / K.tile_k * K.tile_k;   // <= Kp
  for (base = 0; base < end; base += part) {
    if (base > 0 || nwn > part) load(base);   // a row that does not fit the registers is formed again
#pragma unroll
    for (int c = 0; c < R; ++c) {
      const int l0 = base + 4 * (threadIdx.x + c * blockDim.x);
      if (l0 >= end) break;
#pragma unroll
      for (int b = 0; b < 4; ++b) {
        vr[c][b] = vr[c][b] * kr.f1 * kr.f2;
        vi[c][b] = vi[c][b] * ki.f1 * ki.f2;
      }
      unsigned qr[NS], qi[NS];
      slice_words<NS>(vr[c], qr);
      slice_words<NS>(vi[c], qi);
      signed char* a = K.A8 + r0 * K.Kp + l0;
#pragma unroll
      for (int i = 0; i < NS; ++i) {
        *reinterpret_cast<unsigned*>(a + i * plane) = qr[i];
        *reinterpret_cast<unsigned*>(a + i * plane + K.Kp) = qi[i];
      }
    }
  }
}

// 8 degrees per thread; 512 threads when a row has more than 2048
template <class F>
cudaError_t coef_rows_launch(const F& f, int nsum, int nf, const float* gr, const float* gi, const TcCoefSink& K, cudaStream_t st) {
  const int threads = K.K > 2048 ? 512 : 256;
  const dim3 nblocks(nsum, nf);
  if (K.nslice == 7) coef_rows_kernel<7, 2, F><<<nblocks, threads, 0, st>>>(f, gr, gi, K);
  else coef_rows_kernel<6, 2, F><<<nblocks, threads, 0, st>>>(f, gr, gi, K);
  return cudaGetLastError();
}

}  // namespace gem
