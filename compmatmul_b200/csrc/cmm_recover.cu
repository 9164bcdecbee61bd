// Recovery kernels: median decompression (matmul_fft.hpp:135-147,165-177;
// matmul_fwht.hpp:122-134,154-166; array.hpp:323-328), device top-K, and
// the exact FP64 GEMM behind `gemm` (array.hpp:85-95).
#include <cfloat>

#include "cmm_internal.h"

namespace cmm {

// ------------------------------------------------------------ decompress
// Estimate for one (i, j): value_t = s1_t(i) s2_t(j) p_t[idx], idx =
// (h1+h2) & (b-1) (FFT) or h1 ^ h2 (FWHT).  With codes c = h | (s>0)<<31:
// (c1 + c2) & mask == (h1 + h2) & mask because mask < 2^31, and the product
// of the signs is negative iff bit 31 of c1 ^ c2 is set.  The sign is
// applied by flipping the sign bit, which is exactly (-1) * p.
template <int VARIANT>
__device__ __forceinline__ double estimate(const double* __restrict__ pt, uint32_t c1, uint32_t c2,
                                           uint32_t mask) {
  const uint32_t idx = VARIANT == kVariantFFT ? ((c1 + c2) & mask) : ((c1 ^ c2) & mask);
  long long bits = __double_as_longlong(__ldg(pt + idx));
  bits ^= (long long)((c1 ^ c2) & 0x80000000u) << 32;
  return __longlong_as_double(bits);
}

// sorting network by odd-even transposition; returns element D/2 of the
// ascending order (the reference's nth_element at size/2)
template <int D>
__device__ __forceinline__ double median_of(double (&v)[D]) {
#pragma unroll
  for (int pass = 0; pass < D; ++pass) {
#pragma unroll
    for (int i = pass & 1; i + 1 < D; i += 2) {
      const double lo = fmin(v[i], v[i + 1]);
      const double hi = fmax(v[i], v[i + 1]);
      v[i] = lo;
      v[i + 1] = hi;
    }
  }
  return v[D / 2];
}

// The same entry for finite values, without the sort: of kKeep = D / 2 + 2
// values the smallest and the largest cannot be the median, so each further
// value replaces two (an even D counts one more value, +inf).  20 exchanges
// instead of 36 for D = 9, each one comparison and four selections (fmin and
// fmax, which look for NaNs, take three times that; ordered integers instead of
// doubles took 239 us against 165 at 4096 x 4096, b = 1024).  The comparison
// takes zeros of both signs as equal, so get() is right up to a zero's sign.
__device__ __forceinline__ void exchange(double& a, double& b) {
  const bool swap = b < a;
  const double lo = swap ? b : a, hi = swap ? a : b;
  a = lo;
  b = hi;
}
// moves the smallest of v[LO..HI] to v[LO] and the largest to v[HI]
template <int LO, int HI, int N>
__device__ __forceinline__ void ends(double (&v)[N]) {
#pragma unroll
  for (int i = 0; LO + i < HI - i; ++i) exchange(v[LO + i], v[HI - i]);
#pragma unroll
  for (int i = LO + 1; 2 * i <= LO + HI; ++i) exchange(v[LO], v[i]);
#pragma unroll
  for (int i = HI - 1; 2 * i >= LO + HI; --i) exchange(v[i], v[HI]);
}
template <int D>
struct Median {
  static constexpr int kOdd = D | 1, kKeep = D == 1 ? 1 : kOdd / 2 + 2;
  static __host__ __device__ constexpr int slot(int t) { return t < kKeep ? t : 0; }  // where value t goes
  // after value T is in its slot
  template <int T>
  static __device__ __forceinline__ void put(double (&v)[kKeep]) {
    if constexpr (D > 1 && T >= kKeep - 1) ends<0, kOdd + 1 - T>(v);
  }
  static __device__ __forceinline__ double get(double (&v)[kKeep]) {
    if constexpr (D % 2 == 0) {
      v[slot(D)] = __longlong_as_double(0x7ff0000000000000LL);
      put<D>(v);
    }
    return v[D == 1 ? 0 : 1];
  }
};
// A median of zero: -0 sorts below +0, so it is -0 where more than D / 2 values
// have the sign bit.
template <int D>
__device__ __forceinline__ double zero_median(const double (&x)[D]) {
  int minus = 0;
#pragma unroll
  for (int t = 0; t < D; ++t) minus += (int)((uint32_t)__double2hiint(x[t]) >> 31);
  return minus > D / 2 ? -0.0 : 0.0;
}
// the largest exponent so far; kNotFinite: an infinity or a NaN
__device__ __forceinline__ int top_exponent(int top, double v) { return max(top, __double2hiint(v) & 0x7ff00000); }
constexpr int kNotFinite = 0x7ff00000;

template <int D, int T = 0>
__device__ __forceinline__ void select_all(const double (&x)[D], double (&v)[Median<D>::kKeep], int& top) {
  v[Median<D>::slot(T)] = x[T];
  top = top_exponent(top, x[T]);
  Median<D>::template put<T>(v);
  if constexpr (T + 1 < D) select_all<D, T + 1>(x, v, top);
}

// Bound: for tables beyond L1 a 32-byte sector from L2 per value (300 G/s on the
// chip; shared memory, filled by asynchronous copies tile by tile, and the shared
// memory of a cluster were slower: 1.1 to 1.8 times, 5 times); below, the
// selection (4096 x 4096, d = 9, b = 1024: 267 us with the full sort, 165 now).
// A CTA takes up to kDecRows rows of 256 columns, fewer where that leaves SMs
// without work, since rows follow one another in a thread.
constexpr int kDecThreads = 256;
constexpr int kDecRows = 16;

template <int VARIANT, int D>
__global__ void __launch_bounds__(kDecThreads) k_decompress(const uint32_t* __restrict__ cA,
                                                            const uint32_t* __restrict__ cB,
                                                            const double* __restrict__ p, int b,
                                                            int64_t n_a, int64_t n_b, int64_t lda,
                                                            int per, double* __restrict__ C) {
  __shared__ uint32_t sA[D][kDecRows];
  const int64_t j = (int64_t)blockIdx.x * kDecThreads + threadIdx.x;
  const int64_t i0 = (int64_t)blockIdx.y * per;
  for (int e = threadIdx.x; e < D * kDecRows; e += kDecThreads) {
    const int t = e / kDecRows, ii = e % kDecRows;
    sA[t][ii] = (i0 + ii < n_a) ? cA[(size_t)t * lda + i0 + ii] : 0u;
  }
  __syncthreads();
  if (j >= n_b) return;
  uint32_t c2[D];
#pragma unroll
  for (int t = 0; t < D; ++t) c2[t] = __ldg(cB + (size_t)t * n_b + j);
  const uint32_t mask = (uint32_t)b - 1u;
  const int rows = (int)((n_a - i0) < per ? (n_a - i0) : per);
  for (int ii = 0; ii < rows; ++ii) {
    double v[D];
#pragma unroll
    for (int t = 0; t < D; ++t) v[t] = estimate<VARIANT>(p + (size_t)t * b, sA[t][ii], c2[t], mask);
    double keep[Median<D>::kKeep];
    int top = 0;
    select_all<D>(v, keep, top);
    double m = Median<D>::get(keep);
    if (m == 0.0) m = zero_median<D>(v);
    if (top == kNotFinite) m = median_of<D>(v);
    C[(size_t)(i0 + ii) * n_b + j] = m;
  }
}

// any d: rank selection (element with lt <= d/2 < le), O(d^2) gathers
template <int VARIANT>
__global__ void k_decompress_generic(const uint32_t* __restrict__ cA, const uint32_t* __restrict__ cB,
                                     const double* __restrict__ p, int d, int b, int64_t n_a,
                                     int64_t n_b, int64_t lda, double* __restrict__ C) {
  const int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int64_t i = blockIdx.y;
  if (j >= n_b || i >= n_a) return;
  const uint32_t mask = (uint32_t)b - 1u;
  const int mid = d / 2;
  double ans = 0.0;
  for (int a = 0; a < d; ++a) {
    const double va = estimate<VARIANT>(p + (size_t)a * b, cA[(size_t)a * lda + i], cB[(size_t)a * n_b + j], mask);
    int lt = 0, le = 0;
    for (int t = 0; t < d; ++t) {
      const double vt = estimate<VARIANT>(p + (size_t)t * b, cA[(size_t)t * lda + i], cB[(size_t)t * n_b + j], mask);
      lt += vt < va;
      le += vt <= va;
    }
    if (lt <= mid && mid < le) { ans = va; break; }
  }
  C[(size_t)i * n_b + j] = ans;
}

template <int VARIANT, int D>
static void dec_launch(const uint32_t* cA, const uint32_t* cB, const double* p, int b, int64_t n_a,
                       int64_t n_b, int64_t lda, double* C, cudaStream_t s) {
  const int64_t cols = (n_b + kDecThreads - 1) / kDecThreads;
  const int64_t fill = n_a * cols / (4 * num_sms()) + 1;
  const int per = (int)(fill < kDecRows ? fill : kDecRows);
  dim3 grid((unsigned)cols, (unsigned)((n_a + per - 1) / per));
  k_decompress<VARIANT, D><<<grid, kDecThreads, 0, s>>>(cA, cB, p, b, n_a, n_b, lda, per, C);
}

template <int VARIANT>
static void dec_dispatch(int d, const uint32_t* cA, const uint32_t* cB, const double* p, int b,
                         int64_t n_a, int64_t n_b, int64_t lda, double* C, cudaStream_t s) {
  switch (d) {
#define CMM_DEC_CASE(D) case D: dec_launch<VARIANT, D>(cA, cB, p, b, n_a, n_b, lda, C, s); return;
    CMM_DEC_CASE(1) CMM_DEC_CASE(2) CMM_DEC_CASE(3) CMM_DEC_CASE(4) CMM_DEC_CASE(5)
    CMM_DEC_CASE(6) CMM_DEC_CASE(7) CMM_DEC_CASE(8) CMM_DEC_CASE(9) CMM_DEC_CASE(10)
    CMM_DEC_CASE(11) CMM_DEC_CASE(12) CMM_DEC_CASE(13) CMM_DEC_CASE(14) CMM_DEC_CASE(15)
    CMM_DEC_CASE(16)
#undef CMM_DEC_CASE
    default: {
      if (n_a > 2147483647LL) throw unsupported("n_a too large for the generic-d decompression");
      dim3 grid((unsigned)((n_b + 255) / 256), (unsigned)n_a);
      k_decompress_generic<VARIANT><<<grid, 256, 0, s>>>(cA, cB, p, d, b, n_a, n_b, lda, C);
    }
  }
}

void launch_decompress_dense(int variant, int d, int b, int64_t n_a, int64_t n_b,
                             const uint32_t* dCodesA, const uint32_t* dCodesB, const double* dP,
                             double* dC, cudaStream_t s) {
  if (n_a <= 0 || n_b <= 0) return;
  if ((n_a + kDecRows - 1) / kDecRows > 2147483647LL) throw unsupported("n_a too large");
  ProfScope prof("decompress", s);
  count_launch();
  if (variant == kVariantFFT) dec_dispatch<kVariantFFT>(d, dCodesA, dCodesB, dP, b, n_a, n_b, n_a, dC, s);
  else dec_dispatch<kVariantFWHT>(d, dCodesA, dCodesB, dP, b, n_a, n_b, n_a, dC, s);
  CMM_CUDA(cudaGetLastError());
}

// rows [i0, i0 + rows) of the dense estimate into dCrows (rows x n_b)
void launch_decompress_dense_rows(int variant, int d, int b, int64_t n_a, int64_t n_b, int64_t i0,
                                  int64_t rows, const uint32_t* dCodesA, const uint32_t* dCodesB,
                                  const double* dP, double* dCrows, cudaStream_t s) {
  if (rows <= 0 || n_b <= 0) return;
  if (i0 < 0 || i0 + rows > n_a) throw invalid_argument("decompression rows out of range");
  if ((rows + kDecRows - 1) / kDecRows > 2147483647LL) throw unsupported("n_a too large");
  ProfScope prof("decompress", s);
  count_launch();
  if (variant == kVariantFFT) dec_dispatch<kVariantFFT>(d, dCodesA + i0, dCodesB, dP, b, rows, n_b, n_a, dCrows, s);
  else dec_dispatch<kVariantFWHT>(d, dCodesA + i0, dCodesB, dP, b, rows, n_b, n_a, dCrows, s);
  CMM_CUDA(cudaGetLastError());
}

// list form: codes are d x count, one column per listed entry
template <int VARIANT>
__global__ void k_decompress_list(const uint32_t* __restrict__ cI, const uint32_t* __restrict__ cJ,
                                  const double* __restrict__ p, int d, int b, int64_t count,
                                  double* __restrict__ out) {
  const int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= count) return;
  const uint32_t mask = (uint32_t)b - 1u;
  const int mid = d / 2;
  double ans = 0.0;
  for (int a = 0; a < d; ++a) {
    const double va = estimate<VARIANT>(p + (size_t)a * b, cI[(size_t)a * count + e], cJ[(size_t)a * count + e], mask);
    int lt = 0, le = 0;
    for (int t = 0; t < d; ++t) {
      const double vt = estimate<VARIANT>(p + (size_t)t * b, cI[(size_t)t * count + e], cJ[(size_t)t * count + e], mask);
      lt += vt < va;
      le += vt <= va;
    }
    if (lt <= mid && mid < le) { ans = va; break; }
  }
  out[e] = ans;
}

void launch_decompress_list(int variant, int d, int b, int64_t count, const uint32_t* dCodesI,
                            const uint32_t* dCodesJ, const double* dP, double* dOut,
                            cudaStream_t s) {
  if (count <= 0) return;
  const unsigned blocks = (unsigned)((count + 255) / 256);
  ProfScope prof("decompress", s);
  count_launch();
  if (variant == kVariantFFT) k_decompress_list<kVariantFFT><<<blocks, 256, 0, s>>>(dCodesI, dCodesJ, dP, d, b, count, dOut);
  else k_decompress_list<kVariantFWHT><<<blocks, 256, 0, s>>>(dCodesI, dCodesJ, dP, d, b, count, dOut);
  CMM_CUDA(cudaGetLastError());
}

// ------------------------------------------------------------------ top-K
// Order-preserving 64-bit key of a double (larger key <=> larger value;
// -0.0 sorts just below +0.0, NaN with the sign bit clear above +inf).
__device__ __forceinline__ uint64_t okey(double v) {
  const uint64_t b = (uint64_t)__double_as_longlong(v);
  return (b >> 63) ? ~b : (b | 0x8000000000000000ULL);
}

constexpr int kHistBits = 11;
constexpr int kHistBins = 1 << kHistBits;
constexpr int kLevels = 6;  // 5 x 11 bits + 9 bits = 64
constexpr int kCandMax = 4096;

__host__ __device__ __forceinline__ int digit_bits(int level) {
  return 64 - kHistBits * level < kHistBits ? 64 - kHistBits * level : kHistBits;
}

// Passes over the entries keep kTopUnroll loads a thread in flight, eight CTAs
// of 256 threads per SM (16.8 M entries: one load, four CTAs 71 and 29 us).
constexpr int kTopUnroll = 4;

// histogram of digit `level` of the keys whose higher bits (the first
// kHistBits * level) equal `prefix`
__global__ void k_topk_hist(const double* __restrict__ C, int64_t n, int level, uint64_t prefix,
                            unsigned long long* __restrict__ hist) {
  __shared__ unsigned int sh[kHistBins];
  for (int i = threadIdx.x; i < kHistBins; i += blockDim.x) sh[i] = 0;
  __syncthreads();
  const int w = digit_bits(level);
  const int pbits = kHistBits * level;
  const int shift = 64 - pbits - w;
  const uint64_t dmask = (1ULL << w) - 1ULL;
  const int lane = threadIdx.x & 31;
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 - lane < n; i0 += kTopUnroll * step) {
    double v[kTopUnroll];
#pragma unroll
    for (int u = 0; u < kTopUnroll; ++u) v[u] = i0 + u * step < n ? __ldg(C + i0 + u * step) : 0.0;
#pragma unroll
    for (int u = 0; u < kTopUnroll; ++u) {
      const uint64_t k = okey(v[u]);
      const bool in = i0 + u * step < n && (level == 0 || (k >> (64 - pbits)) == prefix);
      // warp-aggregated: one shared atomic per distinct digit in the warp
      // (values cluster in few digits, plain atomics would serialise)
      const uint32_t dg = in ? (uint32_t)((k >> shift) & dmask) : 0xffffffffu;
      const uint32_t peers = __match_any_sync(0xffffffffu, dg);
      if (in && lane == __ffs(peers) - 1) atomicAdd(&sh[dg], (unsigned)__popc(peers));
    }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kHistBins; i += blockDim.x)
    if (sh[i]) atomicAdd(&hist[i], (unsigned long long)sh[i]);
}

// The digit, from the top, where the running count reaches `need`: out =
// {digit, count_above_in_level, count_in_bin}, or {0, total, 0} if none does.
// One CTA: counts of pairs of bins, then their suffix sums (one thread walking
// 2048 bins took 54 us).
constexpr int kPickThreads = kHistBins / 2;
__global__ void __launch_bounds__(kPickThreads) k_topk_pick(const unsigned long long* __restrict__ hist, int nbins,
                                                            unsigned long long need,
                                                            unsigned long long* __restrict__ out) {
  __shared__ unsigned long long warp_sum[kPickThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  // thread x holds digits hi = kHistBins - 1 - 2 x and hi - 1
  const int hi = kHistBins - 1 - 2 * (int)threadIdx.x;
  const unsigned long long c0 = hi < nbins ? hist[hi] : 0, c1 = hi - 1 < nbins ? hist[hi - 1] : 0;
  unsigned long long sum = c0 + c1;  // becomes the count of this thread's and all higher digits
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned long long x = __shfl_up_sync(0xffffffffu, sum, o);
    if (lane >= o) sum += x;
  }
  if (lane == 31) warp_sum[w] = sum;
  __syncthreads();
  for (int i = 0; i < w; ++i) sum += warp_sum[i];
  const unsigned long long above = sum - c0 - c1;
  if (above < need && above + c0 >= need) {
    out[0] = (unsigned long long)hi;
    out[1] = above;
    out[2] = c0;
  } else if (above + c0 < need && sum >= need) {
    out[0] = (unsigned long long)(hi - 1);
    out[1] = above + c0;
    out[2] = c1;
  } else if (threadIdx.x == kPickThreads - 1 && sum < need) {
    out[0] = 0; out[1] = sum; out[2] = 0;
  }
}

// collect entries whose key prefix (top `pbits` bits) is >= pfx (strictly
// greater if `strict`) into the candidate buffer
__global__ void k_topk_collect(const double* __restrict__ C, int64_t n, int pbits, uint64_t pfx,
                               int strict, unsigned long long* __restrict__ keys,
                               unsigned long long* __restrict__ idxs, unsigned int* __restrict__ count,
                               unsigned int cap) {
  const int64_t step = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i0 = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i0 < n; i0 += kTopUnroll * step) {
    double v[kTopUnroll];
#pragma unroll
    for (int u = 0; u < kTopUnroll; ++u) v[u] = i0 + u * step < n ? __ldg(C + i0 + u * step) : 0.0;
#pragma unroll
    for (int u = 0; u < kTopUnroll; ++u) {
      const int64_t idx = i0 + u * step;
      const uint64_t k = okey(v[u]);
      const uint64_t top = pbits >= 64 ? k : (k >> (64 - pbits));
      if (idx < n && (strict ? top > pfx : top >= pfx)) {
        const unsigned int slot = atomicAdd(count, 1u);
        if (slot < cap) { keys[slot] = k; idxs[slot] = (unsigned long long)idx; }
      }
    }
  }
}

// ordered collection of the first `need` entries equal to key `tau`
// (ties broken by linear index = (i, j) order): per-block counts, then
// block-ordered writes.
__global__ void k_topk_tie_count(const double* __restrict__ C, int64_t n, uint64_t tau,
                                 int64_t chunk, unsigned long long* __restrict__ counts) {
  const int64_t beg = (int64_t)blockIdx.x * chunk;
  const int64_t end = beg + chunk < n ? beg + chunk : n;
  unsigned long long c = 0;
  for (int64_t idx = beg + threadIdx.x; idx < end; idx += blockDim.x) c += okey(__ldg(C + idx)) == tau;
  for (int o = 16; o > 0; o >>= 1) c += __shfl_xor_sync(0xffffffffu, c, o);
  __shared__ unsigned long long s[32];
  if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = c;
  __syncthreads();
  if (threadIdx.x == 0) {
    unsigned long long tot = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += s[w];
    counts[blockIdx.x] = tot;
  }
}

__global__ void k_topk_tie_write(const double* __restrict__ C, int64_t n, uint64_t tau, int64_t chunk,
                                 const unsigned long long* __restrict__ counts, int nblocks,
                                 unsigned long long need, unsigned long long* __restrict__ keys,
                                 unsigned long long* __restrict__ idxs, unsigned int base) {
  // serial within the block, in index order (only blocks that contribute)
  if (threadIdx.x != 0) return;
  unsigned long long before = 0;
  for (int blk = 0; blk < (int)blockIdx.x; ++blk) before += counts[blk];
  if (before >= need || counts[blockIdx.x] == 0) return;
  const int64_t beg = (int64_t)blockIdx.x * chunk;
  const int64_t end = beg + chunk < n ? beg + chunk : n;
  unsigned long long r = before;
  for (int64_t idx = beg; idx < end && r < need; ++idx) {
    if (okey(C[idx]) == tau) {
      keys[base + r] = tau;
      idxs[base + r] = (unsigned long long)idx;
      ++r;
    }
  }
}

// single-CTA bitonic sort of up to kCandMax candidates: key descending,
// index ascending; writes the first K as (i, j, value).  The network is that of
// the next power of two above the count (4096 always: 67 us).
__global__ void __launch_bounds__(1024) k_topk_sort(const unsigned long long* __restrict__ keys,
                                                     const unsigned long long* __restrict__ idxs,
                                                     const unsigned int* __restrict__ count,
                                                     int K, int64_t n_b, uint32_t* oi, uint32_t* oj,
                                                     double* ov) {
  extern __shared__ unsigned long long sdyn[];
  unsigned long long* sk = sdyn;
  unsigned long long* si = sdyn + kCandMax;
  const unsigned int n = *count < (unsigned)kCandMax ? *count : (unsigned)kCandMax;
  int total = 64;
  while (total < (int)n) total <<= 1;
  for (int e = threadIdx.x; e < total; e += blockDim.x) {
    if ((unsigned)e < n) { sk[e] = keys[e]; si[e] = idxs[e]; }
    else { sk[e] = 0ULL; si[e] = ~0ULL; }
  }
  __syncthreads();
  // "a before b" := key_a > key_b || (key_a == key_b && idx_a < idx_b)
  for (int size = 2; size <= total; size <<= 1) {
    for (int stride = size >> 1; stride > 0; stride >>= 1) {
      for (int e = threadIdx.x; e < total; e += blockDim.x) {
        const int partner = e ^ stride;
        if (partner > e) {
          const bool asc = (e & size) == 0;  // first half of each block: "before" order
          const unsigned long long ka = sk[e], kb = sk[partner];
          const unsigned long long ia = si[e], ib = si[partner];
          const bool b_before_a = (kb > ka) || (kb == ka && ib < ia);
          if (asc ? b_before_a : !b_before_a) {
            sk[e] = kb; sk[partner] = ka;
            si[e] = ib; si[partner] = ia;
          }
        }
      }
      __syncthreads();
    }
  }
  for (int e = threadIdx.x; e < K; e += blockDim.x) {
    const unsigned long long key = sk[e];
    const unsigned long long bits = (key >> 63) ? (key & 0x7fffffffffffffffULL) : ~key;
    const unsigned long long id = si[e];
    oi[e] = (uint32_t)(id / (unsigned long long)n_b);
    oj[e] = (uint32_t)(id % (unsigned long long)n_b);
    ov[e] = __longlong_as_double((long long)bits);
  }
}

void topk_dense(const double* dC, int64_t n_a, int64_t n_b, int K, uint32_t* dI, uint32_t* dJ,
                double* dV, cudaStream_t s) {
  const int64_t n = n_a * n_b;
  if (K <= 0) return;
  if (K > kCandMax) throw unsupported("K > 4096 is not supported by the device top-K");
  if ((int64_t)K > n) throw invalid_argument("K exceeds the number of entries");
  ProfScope prof("topk", s);
  DevBuf hist((size_t)kHistBins * 8, s), pick(3 * 8, s);
  DevBuf keys((size_t)kCandMax * 8, s), idxs((size_t)kCandMax * 8, s), cnt(8, s);
  int64_t blocks = (n + 255) / 256;
  if (blocks > 8 * num_sms()) blocks = 8 * num_sms();
  uint64_t prefix = 0;              // selected digits so far
  unsigned long long need = (unsigned long long)K;  // still to take at this prefix
  unsigned long long above = 0;     // taken strictly above the prefix (all levels)
  int level = 0;
  int pbits = 0;
  unsigned long long h_pick[3];
  bool tie = false;
  for (; level < kLevels; ++level) {
    const int w = digit_bits(level);
    CMM_CUDA(cudaMemsetAsync(hist.ptr, 0, hist.bytes, s));
    count_launch(2);
    k_topk_hist<<<(unsigned)blocks, 256, 0, s>>>(dC, n, level, prefix, hist.as<unsigned long long>());
    CMM_CUDA(cudaGetLastError());
    k_topk_pick<<<1, kPickThreads, 0, s>>>(hist.as<unsigned long long>(), 1 << w, need,
                                 pick.as<unsigned long long>());
    CMM_CUDA(cudaMemcpyAsync(h_pick, pick.ptr, sizeof(h_pick), cudaMemcpyDeviceToHost, s));
    CMM_CUDA(cudaStreamSynchronize(s));
    prefix = (prefix << w) | h_pick[0];
    pbits += w;
    above += h_pick[1];
    need -= h_pick[1];
    // everything at this prefix fits: collect >= prefix and sort
    if (above + h_pick[2] <= (unsigned long long)kCandMax) break;
    if (level == kLevels - 1) tie = true;  // > kCandMax entries share the K-th key exactly
  }
  CMM_CUDA(cudaMemsetAsync(cnt.ptr, 0, 8, s));
  count_launch(tie ? 4 : 2);
  if (!tie) {
    k_topk_collect<<<(unsigned)blocks, 256, 0, s>>>(dC, n, pbits, prefix, 0, keys.as<unsigned long long>(),
                                                    idxs.as<unsigned long long>(), cnt.as<unsigned int>(), kCandMax);
    CMM_CUDA(cudaGetLastError());
  } else {
    // strictly greater keys (< K of them), then the first `need` ties by index
    k_topk_collect<<<(unsigned)blocks, 256, 0, s>>>(dC, n, 64, prefix, 1, keys.as<unsigned long long>(),
                                                    idxs.as<unsigned long long>(), cnt.as<unsigned int>(), kCandMax);
    CMM_CUDA(cudaGetLastError());
    const int64_t chunk = 1 << 20;
    const int nb = (int)((n + chunk - 1) / chunk);
    DevBuf counts((size_t)nb * 8, s);
    k_topk_tie_count<<<nb, 256, 0, s>>>(dC, n, prefix, chunk, counts.as<unsigned long long>());
    k_topk_tie_write<<<nb, 32, 0, s>>>(dC, n, prefix, chunk, counts.as<unsigned long long>(), nb, need,
                                       keys.as<unsigned long long>(), idxs.as<unsigned long long>(),
                                       (unsigned int)above);
    CMM_CUDA(cudaGetLastError());
    const unsigned int total = (unsigned int)K;
    CMM_CUDA(cudaMemcpyAsync(cnt.ptr, &total, 4, cudaMemcpyHostToDevice, s));
  }
  const int ssmem = 2 * kCandMax * 8;
  CMM_CUDA(cudaFuncSetAttribute(k_topk_sort, cudaFuncAttributeMaxDynamicSharedMemorySize, ssmem));
  k_topk_sort<<<1, 1024, ssmem, s>>>(keys.as<unsigned long long>(), idxs.as<unsigned long long>(),
                                  cnt.as<unsigned int>(), K, n_b, dI, dJ, dV);
  CMM_CUDA(cudaGetLastError());
  CMM_CUDA(cudaStreamSynchronize(s));
}

// ------------------------------------------------------------------- GEMM
// C[i][j] = sum_k AT[k][i] B[k][j] in FP64, ascending k.
//
// Bound: the FP64 units (64 FMA per cycle and SM, 36.7 TFLOP/s), through the
// FP64 matrix instructions (m16n8k4), which take a third of the register
// operands of single FMAs: 8 x 8 entries a thread with plain FMAs reached 22
// TFLOP/s.  Tiles of 64 x 64 in CTAs of four warps (32 x 32 each), four CTAs
// per SM, so that the SMs finish together (tiles of 128 x 128 leave a fifth of
// the last wave empty at 3000 x 2500).  Slabs of 16 inner indices are copied
// with cp.async behind the previous slab's products, 16 bytes at a time where
// rows are aligned (V16); 68 doubles a row keep the fragment loads free of bank
// conflicts.  The form before, 4 x 4 entries a thread on one buffer, took 1.86
// ms (16.5 TFLOP/s) for 3000 x 2048 x 2500,
// now 1.02 ms (30.1; 32.6 at 6000^3).
constexpr int kGT = 64, kGP = 68, kGK = 16, kGThreads = 128;
template <bool V16>
__device__ __forceinline__ void gemm_stage(double (&S)[kGK][kGP], const double* __restrict__ X, int64_t n, int64_t n_inner,
                                           int64_t k0, int64_t c0) {
  constexpr int W = V16 ? 2 : 1;  // elements per copy
#pragma unroll
  for (int e = threadIdx.x * W; e < kGK * kGT; e += kGThreads * W) {
    const int kk = e / kGT, c = e % kGT;
    const bool ok = k0 + kk < n_inner && c0 + c < n;  // (V16: n is even)
    const double* src = ok ? X + (k0 + kk) * n + c0 + c : X;
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(&S[kk][c]);
    if (V16)
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
    else
      asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(dst), "l"(src), "r"(ok ? 8 : 0) : "memory");
  }
}
// D += A B for a 16 x 4 (rows lane / 4 and + 8, k = lane % 4) and a 4 x 8 tile
// (k = lane % 4, column lane / 4); D: rows lane / 4 and + 8, columns 2 (lane %
// 4) and + 1
__device__ __forceinline__ void mma_f64(double (&d)[4], double a0, double a1, double b) {
  asm volatile("mma.sync.aligned.m16n8k4.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};\n"
               : "+d"(d[0]), "+d"(d[1]), "+d"(d[2]), "+d"(d[3])
               : "d"(a0), "d"(a1), "d"(b));
}

template <bool V16>
__global__ void __launch_bounds__(kGThreads, 4) k_gemm(const double* __restrict__ AT, const double* __restrict__ B,
                                                       int64_t n_a, int64_t n_inner, int64_t n_b,
                                                       double* __restrict__ C) {
  __shared__ __align__(16) double As[2][kGK][kGP], Bs[2][kGK][kGP];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, gr = lane >> 2, tg = lane & 3;
  const int wi = (warp >> 1) * 32, wj = (warp & 1) * 32;
  const int64_t i0 = (int64_t)blockIdx.y * kGT, j0 = (int64_t)blockIdx.x * kGT;
  double acc[2][4][4] = {};
  auto stage = [&](int s, int64_t k0) {
    gemm_stage<V16>(As[s], AT, n_a, n_inner, k0, i0);
    gemm_stage<V16>(Bs[s], B, n_b, n_inner, k0, j0);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  stage(0, 0);
  int s = 0;
  for (int64_t k0 = 0; k0 < n_inner; k0 += kGK, s ^= 1) {
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();  // this slab is there, and the other buffer is no longer read
    if (k0 + kGK < n_inner) stage(s ^ 1, k0 + kGK);
#pragma unroll
    for (int kk = 0; kk < kGK; kk += 4) {
      double a[2][2], b[4];
#pragma unroll
      for (int u = 0; u < 2; ++u) {
        a[u][0] = As[s][kk + tg][wi + 16 * u + gr];
        a[u][1] = As[s][kk + tg][wi + 16 * u + gr + 8];
      }
#pragma unroll
      for (int v = 0; v < 4; ++v) b[v] = Bs[s][kk + tg][wj + 8 * v + gr];
#pragma unroll
      for (int u = 0; u < 2; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) mma_f64(acc[u][v], a[u][0], a[u][1], b[v]);
    }
  }
#pragma unroll
  for (int u = 0; u < 2; ++u)
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const int64_t i = i0 + wi + 16 * u + 8 * h + gr;
      if (i >= n_a) continue;
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const int64_t j = j0 + wj + 8 * v + 2 * tg;
        if (j < n_b) C[i * n_b + j] = acc[u][v][2 * h];
        if (j + 1 < n_b) C[i * n_b + j + 1] = acc[u][v][2 * h + 1];
      }
    }
}

void launch_gemm(int64_t n_a, int64_t n_inner, int64_t n_b, double* dC, const double* dAT,
                 const double* dB, cudaStream_t s) {
  if (n_a <= 0 || n_b <= 0) return;
  if (n_inner <= 0) {
    CMM_CUDA(cudaMemsetAsync(dC, 0, (size_t)n_a * n_b * sizeof(double), s));
    return;
  }
  dim3 grid((unsigned)((n_b + kGT - 1) / kGT), (unsigned)((n_a + kGT - 1) / kGT));
  const bool v16 = n_a % 2 == 0 && n_b % 2 == 0 &&
                   (reinterpret_cast<uintptr_t>(dAT) | reinterpret_cast<uintptr_t>(dB)) % 16 == 0;
  ProfScope prof("gemm", s);
  count_launch();
  if (v16) k_gemm<true><<<grid, kGThreads, 0, s>>>(dAT, dB, n_a, n_inner, n_b, dC);
  else k_gemm<false><<<grid, kGThreads, 0, s>>>(dAT, dB, n_a, n_inner, n_b, dC);
  CMM_CUDA(cudaGetLastError());
}

// ---------------------------------------------------------- conversion
__global__ void k_f32_to_f64(const float* __restrict__ src, double* __restrict__ dst, int64_t n) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    dst[i] = (double)src[i];
}

void launch_f32_to_f64(const float* src, double* dst, int64_t n, cudaStream_t s) {
  if (n <= 0) return;
  int64_t blocks = (n + 255) / 256;
  if (blocks > 8 * num_sms()) blocks = 8 * num_sms();
  count_launch();
  k_f32_to_f64<<<(unsigned)blocks, 256, 0, s>>>(src, dst, n);
  CMM_CUDA(cudaGetLastError());
}

}  // namespace cmm
