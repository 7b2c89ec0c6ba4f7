// Degree sums on the 5th-generation tensor cores with sliced integer operands.
//
// The degree sums of harmonicDegreeSums.f90:95-351 are, for every Legendre
// table kind, the product C[row, station] = sum_l A[row, l] * T[l, station]
// (rows: frequency x sum x re/im; see synth.cu).  The FP64 form runs it on
// CUDA cores.  Here the Legendre recurrences and the coefficient weights stay
// FP64 and the product runs on tcgen05 as an exact integer computation:
//
//   T[l, n] = s_l c_n t,    s_l, c_n powers of two, |t| < 1
//   A[m, l] s_l = r_m a,    r_m a power of two,      |a| < 1
//   a = sum_i a_i 128^-(i+1), t = sum_j t_j 128^-(j+1), a_i, t_j in [-127, 127]
//   C[m, n] = r_m c_n sum_{w=0}^{S-1} 128^-(w+2) sum_{i+j=w} (sum_l a_i t_j)
//
// with S = 6 slices of 7 bits (42 bits of each operand relative to its row or
// column scale; terms with i + j >= S are dropped).  The slice products are
// accumulated exactly in INT32 by tcgen05.mma kind::i8 and combined in FP64,
// so the result keeps FP64-level accuracy even where the degree sum cancels by
// five orders of magnitude (near-antipodal stations), which FP16 operands with
// FP32 accumulation cannot.
//
// GEMM kernel: one CTA per 128 x BN output tile.  Up to 80 (7 slices: 64) columns
// one launch forms all weights w = i + j on tiles of that width; beyond, two launches
// form the weights from 3 up and then 0..2 on tiles of 160 (128) columns and pass
// the partial sums in FP64, in the same order of additions, so both forms give the
// same bits.  Per k-block of 64 degrees, warp 0 issues TMA loads (64-byte swizzle)
// of the launch's slices of A and of T into a shared-memory ring; warp 1 issues the
// slice products (2 MMAs of K 32 each) into one TMEM accumulator of BN columns per
// weight; warps 2-5 combine the accumulators in FP64 and write C.
// Bound: the tensor pipe's INT8 rate, 160 cycles for 128 x 160 x 32.  4000 stations
// (batched band): 2.24 ms in one launch of 80-column tiles, 1.01 + 0.63 ms in two of
// 160; coupling, 1000 points: 2.51 -> 1.10 + 0.51 ms.  Slower: all products of one A
// slice in a row (2.7 ms), and with the slice kept in the collector buffer (5.3 ms).  All mbarrier waits
// of the pipeline are bounded by a timer (1 s unless the context sets another
// limit): a wait that runs out records an error flag, the CTA stops issuing
// work, waits (bounded by 1 s, whatever the limit) for its own copies and
// products, frees its TMEM and returns.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cstdint>
#include <vector>

#include "synth.h"
#include "tc_slices.cuh"

namespace gem {

// Slices per operand.  Measured on the tensor-core-sums configuration (synthetics step,
// worst trace error against the FP64 form): 7: 12.6 ms; 6: 11.3 ms, both at the FFT's
// own 1.75e-7; 5: 10.1 ms, but near-zero traces of the global configuration then miss
// the 1e-5 per-trace bar (1.4e-4); 4: 9.1 ms, 2.5e-6 (all with 128 x 64 tiles).  With six
// slices, 128 x 80 tiles (480 of the 512 TMEM columns) take the step from 11.3 to 10.4 ms
// at the same error: each A tile is loaded for 80 stations instead of 64.
constexpr int TC_S = 6;
constexpr int TC_BM = 128, TC_BN = 80, TC_BK = 64;      // tile; BK int8 = one swizzle row (64 or 32 bytes)
// The coupling synthetics combine 42 sums into strain, stress and traction, whose cancellations amplify
// the products' error: with 6 slices their spectra reach 5e-8 of a spectrum's peak against the oracle,
// with 7 (49 bits; 7 accumulators of 64 columns) the FP64 level.
constexpr int TC_S_FINE = 7, TC_BN_FINE = 64;
constexpr int TC_BN2 = 160, TC_BN_FINE2 = 128;   // tiles of the two-launch form
static_assert(TC_BK == 64 || TC_BK == 32, "swizzle spans of 64 or 32 bytes");
// Two stages: measured on the same step, 3 stages at N = 64 (8.51 ms) and 5 stages of BK = 32
// at N = 80 (8.74 ms) both lose to 2 stages of BK = 64 at N = 80 (7.63 ms): the operand bytes
// per product from L2 bound the main loop, not the depth of the pipeline.
constexpr int TC_STAGES = 2;
constexpr int TC_A_BYTES = TC_BM * TC_BK;               // 8 KiB per slice
constexpr int TC_THREADS = 192;
constexpr int TC_TMEM_COLS = 512;                       // NS accumulators of BN columns (power-of-two allocation)
// One launch of the products: the weights WLO <= w < WHI on tiles of BN columns
// (stations), WHI - WLO accumulators of BN columns.  A product of K 32 reads its
// 4 KiB of A and 32 BN bytes of B from shared memory; at BN = 80 (all six weights
// at once) the products kept the tensor pipe 36 % busy and took 78 cycles instead
// of the 40 of their arithmetic.  Two launches of three weights at BN = 160 (the
// fine shape: four and three weights at BN = 128) read half of A per column.
template <int BN_, int WLO_, int WHI_> struct TcShape {
  static constexpr int BN = BN_, WLO = WLO_, WHI = WHI_, NACC = WHI - WLO;
  static constexpr int B_BYTES = BN * TC_BK;                         // per slice
  static constexpr int STAGE_BYTES = WHI * (TC_A_BYTES + B_BYTES);   // slices 0..WHI-1 of A and T
  static constexpr int STAGES = WHI <= 3 ? 4 : TC_STAGES;
  static constexpr int SMEM = STAGES * STAGE_BYTES + 1024 /* alignment */ + 256 /* barriers */;
  static_assert(NACC * BN <= TC_TMEM_COLS, "the accumulators must fit the tensor memory");
  static_assert(BN % 16 == 0 && BN >= 16 && BN <= 256, "MMA N of kind::i8 with M = 128");
  static_assert(B_BYTES % 1024 == 0, "swizzled slices start on 1024 bytes");
  static_assert(SMEM <= 227 * 1024, "stages must fit the shared memory of a CTA");
};
constexpr unsigned long long TC_WAIT_NS = 1000000000ull;   // default pipeline wait limit and the drain limit

constexpr int TC_COLMAX_NONE = (int)0x80808080u;   // a column of zeros (every byte 0x80)

// ---------------------------------------------------------------------------
//  Operand preparation (FP64 in, INT8 slices out)
// ---------------------------------------------------------------------------

// The scales are powers of two above the largest |T| of a degree and the largest
// |T / s_l| of a column, so they follow from the entries' exponents alone, a quarter
// of the table's bytes (from the FP64 table the two passes took 0.21 + 0.19 ms at
// 4000 stations, 835 MB each; from the exponents 0.06 + 0.05).

// s[kind][l], lexp[kind][l] its exponent: one warp per degree, 8 per block
__global__ void __launch_bounds__(256) tab_scale_kernel(int ncol, int lcap, int K, const short* __restrict__ texp,
                                                        double* lscale, short* lexp, int Kp) {
  const int l = blockIdx.x * 8 + (threadIdx.x >> 5), kind = blockIdx.y, lane = threadIdx.x & 31;
  if (l >= Kp) return;
  int e = 0;
  if (l < K) {
    const short* row = texp + ((long long)kind * lcap + l) * ncol;
#pragma unroll 8
    for (int i = lane; i < ncol; i += 32) e = max(e, tc_finite(row[i]));
  }
  for (int o = 16; o > 0; o >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
  if (e == 0) e = 1022;   // no finite largest value: scale 1
  if (lane == 0) {
    lscale[(long long)kind * Kp + l] = ldexp(1.0, e - 1022);
    lexp[(long long)kind * Kp + l] = (short)e;
  }
}

// per (kind, column) the largest exponent of T / s_l: blocks of 128 columns x 64 degrees
__global__ void __launch_bounds__(128) tab_colmax_kernel(int ncol, int lcap, int K, int Kp, const short* __restrict__ texp,
                                                         const short* __restrict__ lexp, int* colmax) {
  __shared__ int se[64];
  const int col = blockIdx.x * blockDim.x + threadIdx.x, kind = blockIdx.z;
  const int l0 = blockIdx.y * 64, l1 = min(l0 + 64, K);
  if (threadIdx.x < 64) se[threadIdx.x] = lexp[(long long)kind * Kp + l0 + threadIdx.x];
  __syncthreads();
  if (col >= ncol) return;
  int m = INT_MIN;
  const short* t = texp + ((long long)kind * lcap + l0) * ncol + col;
#pragma unroll 8
  for (int l = l0; l < l1; ++l, t += ncol) {
    const int e = tc_finite(*t);
    if (e) m = max(m, max(e - se[l - l0], -1000));
  }
  if (m != INT_MIN) atomicMax(colmax + (long long)kind * ncol + col, m);
}

// c[kind][col] = power of two above that maximum
__global__ void tab_colscale_kernel(int n, const int* __restrict__ colmax, double* cscale) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) cscale[i] = colmax[i] == TC_COLMAX_NONE ? 1.0 : ldexp(1.0, colmax[i]);
}

__global__ void tab_exponent_kernel(const double* __restrict__ tab, long long n, short* texp) {
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
    texp[i] = tc_exponent(tab[i]);
}

// T8[j][kind*nsta + sta][l] = slice j of T / (s_l c_sta) for a tile of 64 degrees x 64
// stations: each thread slices four degrees of a station at a time from coalesced reads
// (consecutive stations) into a shared byte tile [slice][station][degree], which is
// written back as 4-degree words.  Bound: memory (1.46 GB at 4000 stations); by single
// digits and bytes, 80 instructions per entry, 0.43 ms, so 0.26 ms.
template <int NS>
__global__ void __launch_bounds__(256) tab_slice_kernel(int nkind, int nsta, int lcap, int K, int Kp,
                                                        const double* __restrict__ tab,
                                                        const double* __restrict__ lscale,
                                                        const double* __restrict__ cscale, signed char* T8) {
  constexpr int ROW = 68;   // bytes per station row: 17 words, so the word accesses of a warp hit distinct banks
  __shared__ __align__(16) signed char dig[NS][64][ROW];
  __shared__ double sl[64], il[64];
  const int kind = blockIdx.z;
  const int l0 = blockIdx.x * 64, s0 = blockIdx.y * 64;
  const int tx = threadIdx.x & 63, ty = threadIdx.x >> 6;   // 256 threads: 64 x 4
  const int sta = s0 + tx;
  double v[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int b = 0; b < 4; ++b) {
      const int l = l0 + 4 * (ty + 4 * r) + b;
      v[r][b] = l < K && sta < nsta ? tab[((long long)kind * lcap + l) * nsta + sta] : 0.0;
    }
  const double cs = sta < nsta ? cscale[(long long)kind * nsta + sta] : 1.0;
  bool far = !(cs >= 0x1p-400 && cs <= 0x1p400);
  if (threadIdx.x < 64) {
    const int l = l0 + threadIdx.x;
    const double s = l < K ? lscale[(long long)kind * Kp + l] : 1.0;
    sl[threadIdx.x] = s;
    il[threadIdx.x] = 1.0 / s;
    far |= !(s >= 0x1p-400 && s <= 0x1p400);
  }
  const bool slow = __syncthreads_or(far);   // a factor 128^S / (s c) of the tile may not be exact
  const double unit = (double)(1ull << (7 * NS)), ic = unit / cs;
#pragma unroll
  for (int r = 0; r < 4; ++r) {
    const int l = 4 * (ty + 4 * r);
    double y[4];
    unsigned w[NS];
#pragma unroll
    for (int b = 0; b < 4; ++b) y[b] = slow ? v[r][b] / sl[l + b] / cs * unit : v[r][b] * (il[l + b] * ic);
    slice_words<NS>(y, w);
#pragma unroll
    for (int j = 0; j < NS; ++j) *reinterpret_cast<uint32_t*>(&dig[j][tx][l]) = w[j];
  }
  __syncthreads();
  const long long plane = (long long)nkind * nsta * Kp;
  for (int e = threadIdx.x; e < 64 * 16; e += 256) {
    const int r = e >> 4, w = e & 15;   // station row of the tile, word of 4 degrees
    if (s0 + r >= nsta) continue;
    const long long o = ((long long)kind * nsta + s0 + r) * Kp + l0 + 4 * w;   // Kp, l0: multiples of 64
#pragma unroll
    for (int j = 0; j < NS; ++j)
      *reinterpret_cast<uint32_t*>(T8 + j * plane + o) = *reinterpret_cast<const uint32_t*>(&dig[j][r][4 * w]);
  }
}

// ---------------------------------------------------------------------------
//  tcgen05 integer GEMM
// ---------------------------------------------------------------------------

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ unsigned long long global_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count));
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}

// Bounded wait: true when the phase completed, false after limit_ns or when
// another role of this CTA has already given up (abort flag).
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag,
                                          unsigned long long limit_ns) {
  if (mbar_try(bar, parity)) return true;
  const unsigned long long t0 = global_ns();
  while (true) {
    if (mbar_try(bar, parity)) return true;
    if (*abort_flag) return false;
    if (global_ns() - t0 > limit_ns) {
      *abort_flag = 1;
      return false;
    }
  }
}

// wait that ignores the abort flag (used to drain this CTA's own copies before exit)
__device__ __forceinline__ void mbar_drain(uint64_t* bar, uint32_t parity) {
  const unsigned long long t0 = global_ns();
  while (!mbar_try(bar, parity) && global_ns() - t0 < TC_WAIT_NS) {
  }
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
          smem_u32(dst)),
      "l"((unsigned long long)map), "r"(smem_u32(bar)), "r"(x), "r"(y)
      : "memory");
}

// K-major operand swizzled over rows of TC_BK bytes (64 or 32): 8-row groups 8 TC_BK bytes apart
__device__ __forceinline__ uint64_t smem_desc_kmajor(const void* p) {
  const uint64_t addr = smem_u32(p);
  uint64_t d = 0;
  d |= (addr >> 4) & 0x3FFFull;                   // start address
  d |= (uint64_t)1 << 16;                         // leading byte offset (unused for swizzled K-major)
  d |= (uint64_t)((8 * TC_BK) >> 4) << 32;        // stride byte offset: 8 rows x TC_BK bytes
  d |= (uint64_t)1 << 46;                         // descriptor version (tcgen05)
  d |= (uint64_t)(TC_BK == 64 ? 4 : 6) << 61;     // SWIZZLE_64B / SWIZZLE_32B
  return d;
}

// kind::i8 instruction descriptor: D s32, A/B signed 8-bit, both K-major, N = BN, M = 128
template <int BN>
__host__ __device__ constexpr uint32_t tc_idesc() {
  return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(BN >> 3) << 17) | ((uint32_t)(TC_BM >> 4) << 24);
}

// The 16 columns [taddr + k stride, + 16) of the NA accumulators k = 0..NA-1,
// loaded by one asm statement that ends with the wait for all of them: the NA
// loads are in flight together, and the compiler sees the registers defined
// only after the wait.
#define GEM_TM16(a, k)                                                                                        \
  "=r"(a[k][0]), "=r"(a[k][1]), "=r"(a[k][2]), "=r"(a[k][3]), "=r"(a[k][4]), "=r"(a[k][5]), "=r"(a[k][6]),    \
      "=r"(a[k][7]), "=r"(a[k][8]), "=r"(a[k][9]), "=r"(a[k][10]), "=r"(a[k][11]), "=r"(a[k][12]),             \
      "=r"(a[k][13]), "=r"(a[k][14]), "=r"(a[k][15])
template <int NA>
__device__ __forceinline__ void tmem_ld_acc16(uint32_t taddr, uint32_t stride, uint32_t (&v)[NA][16]) {
  static_assert(NA == 3 || NA == 4 || NA == 6 || NA == 7, "accumulators of a launch");
  if constexpr (NA == 3) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%48];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%49];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47}, [%50];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : GEM_TM16(v, 0), GEM_TM16(v, 1), GEM_TM16(v, 2)
        : "r"(taddr + 0u * stride), "r"(taddr + 1u * stride), "r"(taddr + 2u * stride));
  } else if constexpr (NA == 4) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%64];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%65];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47}, [%66];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,%61,%62,%63}, [%67];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : GEM_TM16(v, 0), GEM_TM16(v, 1), GEM_TM16(v, 2), GEM_TM16(v, 3)
        : "r"(taddr + 0u * stride), "r"(taddr + 1u * stride), "r"(taddr + 2u * stride), "r"(taddr + 3u * stride));
  } else if constexpr (NA == 6) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%96];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%97];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47}, [%98];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,%61,%62,%63}, [%99];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%64,%65,%66,%67,%68,%69,%70,%71,%72,%73,%74,%75,%76,%77,%78,%79}, [%100];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%80,%81,%82,%83,%84,%85,%86,%87,%88,%89,%90,%91,%92,%93,%94,%95}, [%101];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : GEM_TM16(v, 0), GEM_TM16(v, 1), GEM_TM16(v, 2), GEM_TM16(v, 3), GEM_TM16(v, 4), GEM_TM16(v, 5)
        : "r"(taddr + 0u * stride), "r"(taddr + 1u * stride), "r"(taddr + 2u * stride), "r"(taddr + 3u * stride), "r"(taddr + 4u * stride), "r"(taddr + 5u * stride));
  } else if constexpr (NA == 7) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%112];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%113];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%32,%33,%34,%35,%36,%37,%38,%39,%40,%41,%42,%43,%44,%45,%46,%47}, [%114];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%48,%49,%50,%51,%52,%53,%54,%55,%56,%57,%58,%59,%60,%61,%62,%63}, [%115];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%64,%65,%66,%67,%68,%69,%70,%71,%72,%73,%74,%75,%76,%77,%78,%79}, [%116];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%80,%81,%82,%83,%84,%85,%86,%87,%88,%89,%90,%91,%92,%93,%94,%95}, [%117];\n\t"
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%96,%97,%98,%99,%100,%101,%102,%103,%104,%105,%106,%107,%108,%109,%110,%111}, [%118];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : GEM_TM16(v, 0), GEM_TM16(v, 1), GEM_TM16(v, 2), GEM_TM16(v, 3), GEM_TM16(v, 4), GEM_TM16(v, 5), GEM_TM16(v, 6)
        : "r"(taddr + 0u * stride), "r"(taddr + 1u * stride), "r"(taddr + 2u * stride), "r"(taddr + 3u * stride), "r"(taddr + 4u * stride), "r"(taddr + 5u * stride), "r"(taddr + 6u * stride));
  }
}
#undef GEM_TM16

// ADD: part holds the unscaled sums of the weights from WHI on; FINAL: the sums
// are complete, scaled and written to C, otherwise left unscaled in part.  part is
// laid out as the epilogue's threads hold it, [tile][column][row of the tile], so
// its accesses are whole lines and a chunk's loads are in flight together, a chunk
// ahead (read from C row by row they took 1.3 of the 1.9 ms of the second launch).
template <class Sh, bool ADD, bool FINAL>
__global__ void __launch_bounds__(TC_THREADS, 1)
    sums_tc_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                   const int4* __restrict__ tiles, const int* __restrict__ kind_rows,
                   const long long* __restrict__ kind_rowoff, const long long* __restrict__ coff, int nkind, int nsta,
                   long long mtot, const double* __restrict__ rscale, const double* __restrict__ cscale,
                   double* C, double* part, int* err, unsigned long long wait_ns) {
  constexpr int BN = Sh::BN, WLO = Sh::WLO, WHI = Sh::WHI, STAGES = Sh::STAGES;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  uint64_t* full = (uint64_t*)(smem + STAGES * Sh::STAGE_BYTES);
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;
  uint32_t* tmem_slot = (uint32_t*)(acc_full + 1);
  volatile int* abort_flag = (volatile int*)(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // (kind, first row of the tile within the kind, k-blocks): the tile's rows are zero
  // beyond its largest wavenumber count, so its k-loop stops there
  const int4 t = tiles[blockIdx.y];
  const int kind = t.x, m0 = t.y, nkb = t.z;
  const int n0 = blockIdx.x * BN;
  const int Mk = kind_rows[kind];
  const long long rowA = kind_rowoff[kind] + m0;
  const long long rowB = (long long)kind * nsta + n0;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(acc_full, 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(TC_TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = *tmem_slot;

  if (warp == 0 && lane == 0) {
    // ---- producer: the slices of A and of T per k-block
    int issued = 0;
    for (int kb = 0; kb < nkb; ++kb) {
      const int s = kb % STAGES;
      if (kb >= STAGES && !mbar_wait(&empty[s], ((kb / STAGES) - 1) & 1, abort_flag, wait_ns)) break;
      unsigned char* st = smem + s * Sh::STAGE_BYTES;
      mbar_expect_tx(&full[s], Sh::STAGE_BYTES);
#pragma unroll 1
      for (int i = 0; i < WHI; ++i)
        tma_load_2d(st + i * TC_A_BYTES, &mapA, &full[s], kb * TC_BK, (int)(i * mtot + rowA));
#pragma unroll 1
      for (int j = 0; j < WHI; ++j)
        tma_load_2d(st + WHI * TC_A_BYTES + j * Sh::B_BYTES, &mapB, &full[s], kb * TC_BK,
                    (int)(j * (long long)nkind * nsta + rowB));
      ++issued;
    }
    for (int kb = (issued > STAGES ? issued - STAGES : 0); kb < issued; ++kb)
      mbar_drain(&full[kb % STAGES], (kb / STAGES) & 1);
  } else if (warp == 1 && lane == 0) {
    // ---- MMA issuer: accumulator w = i + j at TMEM columns BN (w - WLO)
    bool ok = true;
    for (int kb = 0; kb < nkb; ++kb) {
      const int s = kb % STAGES;
      if (!mbar_wait(&full[s], (kb / STAGES) & 1, abort_flag, wait_ns)) { ok = false; break; }
      asm volatile("tcgen05.fence::after_thread_sync;");
      const unsigned char* st = smem + s * Sh::STAGE_BYTES;
#pragma unroll 1
      for (int i = 0; i < WHI; ++i) {
        const uint64_t da = smem_desc_kmajor(st + i * TC_A_BYTES);
#pragma unroll 1
        for (int j = i < WLO ? WLO - i : 0; j + i < WHI; ++j) {
          const uint64_t db = smem_desc_kmajor(st + WHI * TC_A_BYTES + j * Sh::B_BYTES);
          const uint32_t dtm = tmem + (uint32_t)((i + j - WLO) * BN);
#pragma unroll
          for (int kk = 0; kk < TC_BK / 32; ++kk) {
            const uint64_t adv = (uint64_t)((kk * 32) >> 4);   // 32 int8 = 32 bytes along K
            const uint32_t acc = (kb > 0 || kk > 0 || i > 0) ? 1u : 0u;
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "setp.ne.b32 p, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(dtm),
                "l"(da + adv), "l"(db + adv), "r"(tc_idesc<BN>()), "r"(acc));
          }
        }
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                       smem_u32(&empty[s]))
                   : "memory");
    }
    // signals the epilogue once every product issued above has completed
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                     smem_u32(acc_full))
                 : "memory");
    if (!ok) *abort_flag = 1;
    // the products issued above write TMEM and read the stages.  After an abort
    // (set here or by the epilogue at any time) nobody else waits for them, so
    // they are always drained here, before the CTA's closing barrier frees the
    // tensor memory; without an abort the epilogue has waited for the same phase
    mbar_drain(acc_full, 0);
  } else if (warp >= 2) {
    // ---- epilogue: TMEM lanes 32*(warp % 4) .. +31 hold rows of the tile
    const int q = warp & 3;
    const bool done = mbar_wait(acc_full, 0, abort_flag, wait_ns);
    asm volatile("tcgen05.fence::after_thread_sync;");
    const int r = m0 + q * 32 + lane;   // row within the kind
    // the ring is idle once every product has completed: each warp stages its
    // 32 rows x 16 columns there and writes them row by row (a row's 16
    // doubles are one 128-byte segment), not as 32 strided rows per store
    const bool store = __all_sync(0xffffffffu, done && !*abort_flag);
    const double rs = (store && r < Mk) ? rscale[kind_rowoff[kind] + r] : 0.0;
    double* ck = C + coff[kind];
    const double* cs = cscale + (long long)kind * nsta;
    double* stg = reinterpret_cast<double*>(smem) + q * (32 * 17);   // 17: one pad double per row
    double* pt = part + ((long long)blockIdx.y * gridDim.x + blockIdx.x) * (TC_BM * BN) + q * 32 + lane;
    double nxt[16];
    if (ADD) {
#pragma unroll
      for (int jj = 0; jj < 16; ++jj) nxt[jj] = pt[jj * TC_BM];
    }
    // columns in chunks of 16 (BN is a multiple of 16); the accumulators of a
    // chunk are loaded together, then combined smallest weights first
#pragma unroll 1
    for (int c = 0; c < BN / 16; ++c) {
      double sum[16];
#pragma unroll
      for (int jj = 0; jj < 16; ++jj) sum[jj] = ADD ? nxt[jj] : 0.0;
      if (ADD && c + 1 < BN / 16) {
#pragma unroll
        for (int jj = 0; jj < 16; ++jj) nxt[jj] = pt[((c + 1) * 16 + jj) * TC_BM];
      }
      uint32_t v[Sh::NACC][16];
      tmem_ld_acc16<Sh::NACC>(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(c * 16), (uint32_t)BN, v);
#pragma unroll
      for (int w = WHI - 1; w >= WLO; --w) {
        const double wgt = ldexp(1.0, -7 * (w + 2));
#pragma unroll
        for (int jj = 0; jj < 16; ++jj) sum[jj] += (double)(int)v[w - WLO][jj] * wgt;
      }
      if (store && !FINAL) {
#pragma unroll
        for (int jj = 0; jj < 16; ++jj) pt[(c * 16 + jj) * TC_BM] = sum[jj];
      } else if (store) {
#pragma unroll
        for (int jj = 0; jj < 16; ++jj) stg[lane * 17 + jj] = sum[jj] * rs;
        __syncwarp();
        const int col = lane & 15, n = n0 + c * 16 + col;
        const double csn = n < nsta ? cs[n] : 0.0;
#pragma unroll 4
        for (int k = 0; k < 16; ++k) {
          const int row = 2 * k + (lane >> 4), rg = m0 + q * 32 + row;
          if (rg < Mk && n < nsta) ck[(long long)rg * nsta + n] = stg[row * 17 + col] * csn;
        }
        __syncwarp();
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TC_TMEM_COLS));
  }
  if (threadIdx.x == 0 && *abort_flag) atomicExch(err, 1);
}

}  // namespace gem

// ===========================================================================
//  Host side
// ===========================================================================
using namespace gem;

namespace {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = (EncodeTiledFn)p;
  }
  return fn;
}

// 2D map over int8 rows of Kp bytes, box TC_BK bytes x box_rows, swizzled over TC_BK bytes
bool make_map(CUtensorMap* map, const signed char* base, long long rows, long long kp, int box_rows) {
  EncodeTiledFn f = encode_fn();
  if (!f) return false;
  cuuint64_t dims[2] = {(cuuint64_t)kp, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)kp};
  cuuint32_t box[2] = {(cuuint32_t)TC_BK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  return f(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, (void*)base, dims, strides, box, estr,
           CU_TENSOR_MAP_INTERLEAVE_NONE, TC_BK == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
           CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

struct TcLayout {
  int Kp;
  bool part_in_tab;   // the partial sums take the place of the table, which is used up when they are written
  size_t off[11], total;
};

int tc_slices(const TcProblem& P) { return P.nslice == TC_S_FINE ? TC_S_FINE : TC_S; }

TcLayout tc_layout(const TcProblem& P, long long mtot) {
  TcLayout L{};
  const int K = P.lmax + 1, nk = P.nkind, ns = tc_slices(P);
  L.Kp = (K + 63) / 64 * 64;   // the slicing kernels work on 64-degree tiles
  const int bn = ns == TC_S_FINE ? TC_BN_FINE2 : TC_BN2;
  const bool two = P.ncol > (ns == TC_S_FINE ? TC_BN_FINE : TC_BN);   // launches of the products
  const size_t part = two ? (size_t)(mtot / TC_BM + nk + 1) * ((P.ncol + bn - 1) / bn) * TC_BM * bn * sizeof(double) : 0;
  L.part_in_tab = part <= (size_t)nk * P.lcap * P.ncol * sizeof(double);
  const size_t sz[11] = {(size_t)ns * nk * P.ncol * L.Kp,             // T8
                        (size_t)ns * mtot * L.Kp,                     // A8
                        (size_t)nk * L.Kp * sizeof(double),           // lscale
                        (size_t)nk * P.ncol * sizeof(double),         // cscale
                        (size_t)mtot * sizeof(double),                // rscale
                        (size_t)nk * L.Kp * sizeof(short),            // lexp
                        (size_t)(mtot / TC_BM + nk + 1) * sizeof(int4),   // tiles
                        (size_t)3 * TC_MAX_KIND * sizeof(long long),  // per-kind tables
                        (size_t)(TC_MAX_KIND + 8) * sizeof(int),      // kind rows + error flag
                        (size_t)nk * P.ncol * sizeof(int),            // column maxima
                        L.part_in_tab ? 0 : part};                    // partial sums
  size_t b = 0;
  for (int i = 0; i < 11; ++i) {
    L.off[i] = b;
    b += (sz[i] + 1023) / 1024 * 1024;
  }
  L.total = b + 1024;
  return L;
}

}  // namespace

namespace gem {

TcProblem tc_problem_of(const SynthDev& S) {
  TcProblem P{};
  P.nkind = 8; P.ncol = S.nsta; P.lcap = S.lcap; P.lmax = S.lmax; P.nf1 = S.nf1; P.nf2 = S.nf2;
  for (int k = 0; k < 8; ++k) { P.nsk[k] = S.nsk[k]; P.coff[k] = S.coff[k]; }
  return P;
}

size_t sums_tc_workspace(const TcProblem& P, long long mtot, int* Kp_out) {
  TcLayout L = tc_layout(P, mtot);
  if (Kp_out) *Kp_out = L.Kp;
  return L.total;
}

struct TcOperands {
  const TcProblem* P;
  long long mtot;
  int Kp;
  const signed char *T8, *A8;
  const double *cscale, *rscale;
  const int4* tiles;
  size_t ntiles;
  const int* ints;
  const long long* tabs;
  int nslice;
  double* part;
};

template <class Sh, bool ADD, bool FINAL>
const char* tc_products(const TcOperands& O, double* C, int* err, unsigned long long wait_ns, cudaStream_t st) {
  const int nk = O.P->nkind, ncol = O.P->ncol;
  // tensor maps over A8 [nslice mtot][Kp] and T8 [nslice * nkind * ncol][Kp]
  CUtensorMap mA, mB;
  if (!make_map(&mA, O.A8, O.nslice * O.mtot, O.Kp, TC_BM) ||
      !make_map(&mB, O.T8, O.nslice * (long long)nk * ncol, O.Kp, Sh::BN))
    return "sums_tc: cuTensorMapEncodeTiled failed";
  if (cudaFuncSetAttribute(sums_tc_kernel<Sh, ADD, FINAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, Sh::SMEM) !=
      cudaSuccess)
    return "sums_tc: shared-memory attribute";
  dim3 grid((ncol + Sh::BN - 1) / Sh::BN, (unsigned)O.ntiles);
  sums_tc_kernel<Sh, ADD, FINAL><<<grid, TC_THREADS, Sh::SMEM, st>>>(
      mA, mB, O.tiles, O.ints, O.tabs + TC_MAX_KIND, O.tabs + 2 * TC_MAX_KIND, nk, ncol, O.mtot, O.rscale, O.cscale, C,
      O.part, err, wait_ns ? wait_ns : TC_WAIT_NS);
  return cudaGetLastError() == cudaSuccess ? nullptr : "sums_tc: launch failed";
}

// operand slices of NS digits and the products (blocking)
template <int NS>
const char* tc_slice_and_multiply(const TcProblem& P, long long mtot, int K, int Kp, const double* tab,
                                  const TcCoefs& coefs, const double* lscale, const double* cscale, signed char* T8,
                                  signed char* A8, double* rscale, const int4* tiles, size_t ntiles, int* ints,
                                  const long long* tabs, double* part, double* C, unsigned long long wait_ns, cudaStream_t st) {
  const int nk = P.nkind, ncol = P.ncol;
  tab_slice_kernel<NS><<<dim3(Kp / 64, (ncol + 63) / 64, nk), 256, 0, st>>>(nk, ncol, P.lcap, K, Kp, tab, lscale,
                                                                            cscale, T8);
  const TcCoefSink sink{K, Kp, NS, TC_BM, TC_BK, mtot, lscale, tabs + TC_MAX_KIND, A8, rscale};
  if (coefs(sink, st) != cudaSuccess) return "sums_tc: launch of the coefficient rows failed";
  if (cudaMemsetAsync(ints + TC_MAX_KIND, 0, sizeof(int), st) != cudaSuccess) return "sums_tc: upload failed";
  const TcOperands O{&P, mtot, Kp, T8, A8, cscale, rscale, tiles, ntiles, ints, tabs, NS, part};
  int* err = ints + TC_MAX_KIND;
  const char* why;
  // Two launches on wide tiles, unless the columns fit one narrow tile: the wide
  // tiles' columns beyond ncol are work for nothing.
  if constexpr (NS == TC_S) {
    if (ncol <= TC_BN) {
      why = tc_products<TcShape<TC_BN, 0, TC_S>, false, true>(O, C, err, wait_ns, st);
    } else {
      why = tc_products<TcShape<TC_BN2, 3, TC_S>, false, false>(O, C, err, wait_ns, st);
      if (!why) why = tc_products<TcShape<TC_BN2, 0, 3>, true, true>(O, C, err, wait_ns, st);
    }
  } else {
    if (ncol <= TC_BN_FINE) {
      why = tc_products<TcShape<TC_BN_FINE, 0, TC_S_FINE>, false, true>(O, C, err, wait_ns, st);
    } else {
      why = tc_products<TcShape<TC_BN_FINE2, 3, TC_S_FINE>, false, false>(O, C, err, wait_ns, st);
      if (!why) why = tc_products<TcShape<TC_BN_FINE2, 0, 3>, true, true>(O, C, err, wait_ns, st);
    }
  }
  if (why) return why;
  int herr = 0;
  if (cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, st) != cudaSuccess ||
      cudaStreamSynchronize(st) != cudaSuccess)
    return "sums_tc: execution failed";
  if (herr) return "sums_tc: a pipeline wait timed out";
  return nullptr;
}

cudaError_t tc_exponents_launch(const double* tab, long long n, short* texp, cudaStream_t st) {
  tab_exponent_kernel<<<148 * 16, 256, 0, st>>>(tab, n, texp);
  return cudaGetLastError();
}

// Sliced-integer sums: from the FP64 tables tab[kind][l][col] with their exponents texp and the coefficient
// rows that coefs launches, write C[kind][row][col] in FP64.  tab and texp hold nothing of use afterwards;
// texp may lie in C.  ws: device workspace of sums_tc_workspace bytes; wait_ns: limit of each pipeline wait
// (0: 1 s).  Blocking (synchronises the stream).
const char* sums_tc_run(const TcProblem& P, const int* nwn, long long mtot, double* tab, const short* texp,
                        const TcCoefs& coefs,
                        double* C, void* ws, size_t ws_bytes, unsigned long long wait_ns, cudaStream_t st) {
  if (P.nkind < 1 || P.nkind > TC_MAX_KIND) return "sums_tc: table kinds outside 1..16";
  TcLayout L = tc_layout(P, mtot);
  if (ws_bytes < L.total) return "sums_tc: workspace too small";
  const int nk = P.nkind, ncol = P.ncol;
  if (7LL * mtot >= (1LL << 31) || 7LL * nk * ncol >= (1LL << 31)) return "sums_tc: operand rows exceed 2^31";
  if ((long long)L.Kp * tc_slices(P) * 127 * 127 >= (1LL << 31))
    return "sums_tc: degree range too large for INT32 accumulation";
  if (P.nslice != 0 && P.nslice != TC_S && P.nslice != TC_S_FINE) return "sums_tc: 6 or 7 slices per operand";
  const int K = P.lmax + 1, Kp = L.Kp;
  const int nf = P.nf2 - P.nf1 + 1;
  char* base = (char*)(((uintptr_t)ws + 1023) & ~(uintptr_t)1023);
  signed char* T8 = (signed char*)(base + L.off[0]);
  signed char* A8 = (signed char*)(base + L.off[1]);
  double* lscale = (double*)(base + L.off[2]);
  double* cscale = (double*)(base + L.off[3]);
  double* rscale = (double*)(base + L.off[4]);
  int4* tiles = (int4*)(base + L.off[6]);
  long long* tabs = (long long*)(base + L.off[7]);
  int* ints = (int*)(base + L.off[8]);   // [0..15] rows per kind, [16] error flag
  short* lexp = (short*)(base + L.off[5]);
  int* colmax = (int*)(base + L.off[9]);
  double* part = L.part_in_tab ? tab : (double*)(base + L.off[10]);
  int krows[TC_MAX_KIND + 8] = {0};
  long long htabs[3 * TC_MAX_KIND] = {0};
  std::vector<int4> htiles;
  long long ro = 0;
  for (int k = 0; k < nk; ++k) {
    krows[k] = 2 * nf * P.nsk[k];
    htabs[TC_MAX_KIND + k] = ro;
    htabs[2 * TC_MAX_KIND + k] = P.coff[k];
    for (int m = 0; m < krows[k]; m += TC_BM) {
      // rows 2 (slot nsk + rank) + re/im; the coefficients of frequency slot are zero
      // from degree nwn[nf1 - 1 + slot] on
      const int s0 = m / (2 * P.nsk[k]), s1 = std::min(nf - 1, (m + TC_BM - 1) / (2 * P.nsk[k]));
      int ext = 0;
      for (int s = s0; s <= s1; ++s) ext = std::max(ext, nwn[P.nf1 - 1 + s]);
      ext = std::min(ext, K);
      htiles.push_back(make_int4(k, m, std::max(1, (ext + TC_BK - 1) / TC_BK), 0));
    }
    ro += krows[k];
  }
  if (ro != mtot) return "sums_tc: row count mismatch";
  if (htiles.empty()) return nullptr;
  // longest k-loops first: the short tiles fill the last wave
  std::stable_sort(htiles.begin(), htiles.end(), [](const int4& a, const int4& b) { return a.z > b.z; });
  if (cudaMemcpyAsync(tiles, htiles.data(), htiles.size() * sizeof(int4), cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaMemcpyAsync(tabs, htabs, sizeof htabs, cudaMemcpyHostToDevice, st) != cudaSuccess ||
      cudaMemcpyAsync(ints, krows, sizeof krows, cudaMemcpyHostToDevice, st) != cudaSuccess)
    return "sums_tc: upload failed";
  // operands
  tab_scale_kernel<<<dim3((Kp + 7) / 8, nk), 256, 0, st>>>(ncol, P.lcap, K, texp, lscale, lexp, Kp);
  if (cudaMemsetAsync(colmax, 0x80, (size_t)nk * ncol * sizeof(int), st) != cudaSuccess)
    return "sums_tc: upload failed";
  tab_colmax_kernel<<<dim3((ncol + 127) / 128, (K + 63) / 64, nk), 128, 0, st>>>(ncol, P.lcap, K, Kp, texp, lexp, colmax);
  tab_colscale_kernel<<<(nk * ncol + 255) / 256, 256, 0, st>>>(nk * ncol, colmax, cscale);
  if (tc_slices(P) == TC_S_FINE)
    return tc_slice_and_multiply<TC_S_FINE>(P, mtot, K, Kp, tab, coefs, lscale, cscale, T8, A8,
                                                      rscale, tiles, htiles.size(), ints, tabs, part, C, wait_ns, st);
  return tc_slice_and_multiply<TC_S>(P, mtot, K, Kp, tab, coefs, lscale, cscale, T8, A8, rscale, tiles,
                                            htiles.size(), ints, tabs, part, C, wait_ns, st);
}

}  // namespace gem
