// Additions of the product sketch: p_t[idx(i, j)] += s1_t(i) s2_t(j) C[i][j] for
// every entry of C = A^T B and every repetition t (cmm_product.cu forms C).
//
// d n_a n_b additions of 8-byte values to pseudo-random buckets.  Done without
// atomics and in a fixed order, from the side of the buckets: for a row i the
// columns that fall into consecutive buckets [m, m + W) of p_t are
// consecutive in the order of h2 (FFT: h2 in [m - h1(i), + W) mod b; FWHT: the
// aligned block (m ^ h1(i)) / W), so a warp that owns W buckets reads its
// entries of the sorted columns coalesced, looks up their C[i][j] and adds.
// Three forms, chosen by product_geometry:
//  staged  b <= 2^16: rows of C staged in shared memory, a CTA of 16 windows;
//  lane    a block of columns holds 1.5 times the buckets and more: lane
//          = bucket, rows and sorted columns in shared memory;
//  gather  b > 2^16: values gathered from L2.
// Rows are split into G groups with partial sketches, added up by
// k_prod_reduce.
#include <algorithm>

#include "cmm_internal.h"
#include "cmm_product.h"
#include "cmm_product_dev.cuh"

namespace cmm {
namespace {

constexpr int kIdxThreads = 1024;
constexpr int kScCols = 4096;  // columns per block of the staged and lane forms (12 bits of an entry)
constexpr int kScWin = 16;     // windows (warps) per CTA of the staged form
constexpr int kScThreads = 32 * (kScWin + 1);
constexpr size_t kScSmemMax = 227 * 1024 - 1024, kScSmemHalf = 112 * 1024;
constexpr int kGaWarps = 8;    // windows (warps) per CTA of the gather form

// A sorted column, in the order in which the additions take it apart: rank |
// j << 3 | (s2 < 0) << (3 + JB) | h2 << (4 + JB) (low bits), JB = 12 (16 bits
// of h2) or, gather form, 17 (11 bits).  rank counts the entries of the same
// bucket before it (6: six or more; 7: no entry), j << 3 is the offset of the
// value in the row.  Every list is stored twice in a row, so that a run that
// wraps around b (FFT) is read without a test.
constexpr uint32_t kNoEntry = 7;
template <int JB>
constexpr uint32_t kColMask = ((1u << JB) - 1u) << 3;

// ------------------------------------------------------------ sorted columns
// One CTA per (t, block of kScCols columns, job).  The keys (h2, j) are unique,
// so a bitonic sort gives the fixed order without atomics.  Four keys a thread
// in registers: exchanges at distances below 4 stay in the thread, below 128 in
// the warp, so 15 of the 78 steps of 4096 keys go through shared memory and a
// barrier (all of them did before: 45 us at 4096 columns, d = 9, 27 now).
// cum[h] = entries below bucket h, 16 bits, row stride b + 8 (16-byte stores
// of eight: the first by binary search, the others by walking on).
__device__ __forceinline__ void key_exchange(uint32_t& a, uint32_t& b, bool up) {
  const uint32_t lo = min(a, b), hi = max(a, b);
  a = up ? lo : hi;
  b = up ? hi : lo;
}
// sorts the len (a power of two, 128 .. 4 kIdxThreads) keys 4 tid + u of the CTA
__device__ __forceinline__ void sort_keys(uint32_t (&k)[4], uint32_t len, uint4* buf) {
  const uint32_t i = 4 * threadIdx.x;
  key_exchange(k[0], k[1], true);
  key_exchange(k[2], k[3], false);
  int flip = 0;
  for (uint32_t size = 4; size <= len; size <<= 1) {
    const bool up = (i & size) == 0;
    for (uint32_t stride = size >> 1; stride >= 4; stride >>= 1) {
      const bool low = ((i & stride) == 0) == up;  // this thread keeps the smaller ones
      uint32_t x[4];
      if (stride >= 128) {
        uint4* at = buf + flip * kIdxThreads;
        at[threadIdx.x] = make_uint4(k[0], k[1], k[2], k[3]);
        __syncthreads();
        const uint4 o = at[threadIdx.x ^ (stride >> 2)];
        x[0] = o.x; x[1] = o.y; x[2] = o.z; x[3] = o.w;
        flip ^= 1;  // the next step's stores do not meet this step's loads
      } else {
#pragma unroll
        for (int u = 0; u < 4; ++u) x[u] = __shfl_xor_sync(0xffffffffu, k[u], stride >> 2);
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) k[u] = low ? min(k[u], x[u]) : max(k[u], x[u]);
    }
    key_exchange(k[0], k[2], up);
    key_exchange(k[1], k[3], up);
    key_exchange(k[0], k[1], up);
    key_exchange(k[2], k[3], up);
  }
}
__host__ __device__ inline size_t cum16_stride(int log2b) { return ((size_t)1 << log2b) + 8; }
__global__ void __launch_bounds__(kIdxThreads) k_prod_index_blocks(const ProdJob* __restrict__ jobs) {
  const ProdJob& J = jobs[blockIdx.z];
  const int t = blockIdx.x, jb = blockIdx.y;
  if (J.form == kAddGather || t >= J.d || (int64_t)jb * kScCols >= J.n_b) return;
  if (t == 0 && jb == 0 && threadIdx.x == 0) *J.flag = 0;
  __shared__ uint4 buf[2 * kIdxThreads];
  const int tid = threadIdx.x;
  const uint32_t b = 1u << J.log2b;
  const uint32_t n = (uint32_t)min((int64_t)kScCols, J.n_b - (int64_t)jb * kScCols);
  const uint32_t* codes = J.codesB + (size_t)t * J.n_b + (size_t)jb * kScCols;
  uint32_t len = 128;
  while (len < n) len <<= 1;
  // h2 << 13 | j << 1 | (s2 < 0): the sign does not change the order; padding is the largest
  uint32_t k[4];
#pragma unroll
  for (uint32_t u = 0; u < 4; ++u) {
    const uint32_t e = 4 * tid + u, c = e < n ? __ldg(codes + e) : 0u;
    k[u] = e < n ? (c & (b - 1)) << 13 | e << 1 | (~c) >> 31 : 0xffffffffu;
  }
  sort_keys(k, len, buf);
  __syncthreads();
  uint32_t* key = reinterpret_cast<uint32_t*>(buf);
  buf[tid] = make_uint4(k[0], k[1], k[2], k[3]);
  __syncthreads();
  auto bucket = [&](uint32_t e) { return key[e] >> 13; };
  uint32_t* ent = J.ent + 2 * ((size_t)t * J.n_b + (size_t)jb * kScCols);
  for (uint32_t e = tid; e < n; e += kIdxThreads) {
    uint32_t rank = 0;
    while (rank < 6 && rank < e && bucket(e - rank - 1) == bucket(e)) ++rank;
    const uint32_t x = rank | (key[e] >> 1 & 0xfffu) << 3 | (key[e] & 1u) << 15 | bucket(e) << 16;
    ent[e] = x;
    ent[n + e] = x;
  }
  uint16_t* cum = reinterpret_cast<uint16_t*>(J.cum) + ((size_t)t * J.blocks + jb) * cum16_stride(J.log2b);
  for (uint32_t h0 = tid * 8; h0 <= b; h0 += kIdxThreads * 8) {
    uint32_t lo = 0, hi = n;  // the first entry with bucket >= h0
    while (lo < hi) {
      const uint32_t mid = (lo + hi) >> 1;
      if (bucket(mid) >= h0) hi = mid;
      else lo = mid + 1;
    }
    uint32_t w[4];
#pragma unroll
    for (uint32_t u = 0; u < 8; ++u) {
      while (lo < n && bucket(lo) < h0 + u) ++lo;
      if (u & 1) w[u >> 1] |= lo << 16;
      else w[u >> 1] = lo;
    }
    *reinterpret_cast<uint4*>(cum + h0) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

// The same over all columns (at most 2^17) for the gather form: counting sort
// with shared-memory atomics; each bucket's entries are then put in ascending j,
// so the order does not depend on the atomics.  One CTA per (t, kIdxBuckets
// buckets, job): it reads all codes, places those of its buckets, and begins
// after the columns that it counts below them.  (One CTA for all buckets of a
// repetition took 1.15 us per 1024 of them: calls with a small product took 240 us at
// b = 2^17, 5.6 ms at 2^22, now 97 and 0.4.)
constexpr uint32_t kIdxBuckets = 8 * kIdxThreads;
__global__ void __launch_bounds__(kIdxThreads) k_prod_index(const ProdJob* __restrict__ jobs) {
  const ProdJob& J = jobs[blockIdx.z];
  const int t = blockIdx.x;
  const uint32_t b = 1u << J.log2b, h0 = blockIdx.y * kIdxBuckets;  // (b is a multiple of kIdxBuckets)
  if (J.form != kAddGather || t >= J.d || h0 >= b) return;
  if (t == 0 && h0 == 0 && threadIdx.x == 0) *J.flag = 0;
  const uint32_t n = (uint32_t)J.n_b;
  uint32_t* cum = reinterpret_cast<uint32_t*>(J.cum) + (size_t)t * (b + 1);
  uint32_t* ent = J.ent + 2 * (size_t)t * n;
  const uint32_t* codes = J.codesB + (size_t)t * n;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  __shared__ uint32_t cnt[kIdxBuckets];  // counts, then the place of the bucket's next entry
  __shared__ uint32_t ws[32], s_below;
  for (uint32_t e = tid; e < kIdxBuckets; e += kIdxThreads) cnt[e] = 0;
  if (tid == 0) s_below = 0;
  __syncthreads();
  uint32_t below = 0;
  for (uint32_t j = tid; j < n; j += kIdxThreads) {
    const uint32_t h = __ldg(codes + j) & (b - 1);
    if (h - h0 < kIdxBuckets) atomicAdd(cnt + (h - h0), 1u);
    else if (h < h0) ++below;
  }
  below = __reduce_add_sync(0xffffffffu, below);
  if (lane == 0 && below) atomicAdd(&s_below, below);
  __syncthreads();
  const uint32_t base = s_below;
  // exclusive scan: cum[h] = start of bucket h
  uint32_t v[8], sum = 0;
#pragma unroll
  for (int u = 0; u < 8; ++u) sum += v[u] = cnt[tid * 8 + u];
  uint32_t inc = sum;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const uint32_t x = __shfl_up_sync(0xffffffffu, inc, o);
    if (lane >= o) inc += x;
  }
  if (lane == 31) ws[warp] = inc;
  __syncthreads();
  uint32_t run = base + inc - sum;
  for (int w = 0; w < warp; ++w) run += ws[w];
#pragma unroll
  for (int u = 0; u < 8; ++u) {
    cum[h0 + tid * 8 + u] = run;
    cnt[tid * 8 + u] = run;
    run += v[u];
  }
  if (h0 + kIdxBuckets == b && tid == 0) cum[b] = n;
  __syncthreads();
  // placement moves cnt[h] from the start of bucket h to its end
  for (uint32_t j = tid; j < n; j += kIdxThreads) {
    const uint32_t c = __ldg(codes + j), h = c & (b - 1);
    if (h - h0 < kIdxBuckets)
      __stcg(ent + atomicAdd(cnt + (h - h0), 1u), j << 3 | ((~c) >> 31) << 20 | (h & 0x7ffu) << 21);
  }
  __syncthreads();
  for (uint32_t h = tid; h < kIdxBuckets; h += kIdxThreads) {
    const uint32_t beg = h ? cnt[h - 1] : base, end = cnt[h];
    for (uint32_t e = beg + 1; e < end; ++e) {  // insertion sort by j
      const uint32_t x = __ldcg(ent + e);
      uint32_t f = e;
      while (f > beg) {
        const uint32_t y = __ldcg(ent + f - 1);
        if ((y & kColMask<17>) <= (x & kColMask<17>)) break;
        __stcg(ent + f, y);
        --f;
      }
      if (f != e) __stcg(ent + f, x);
    }
    for (uint32_t e = beg; e < end; ++e) {
      const uint32_t x = __ldcg(ent + e) | min(e - beg, 6u);
      __stcg(ent + e, x);
      __stcg(ent + n + e, x);
    }
  }
}

// ----------------------------------------------------------------- additions
// The kernel of a job's additions: 0 gather, 1 and 2 staged (that many CTAs per
// SM), 3 .. 5 lane with b = 512 .. 2048
constexpr int kAddClasses = 6;
__host__ __device__ inline int add_class(const ProdJob& J) {
  return J.form == kAddGather ? 0 : (J.form == kAddStaged ? J.per_sm : J.log2b - 6);
}
// Work of a CTA: the job of its class that covers blockIdx.x, and its window
// group x, repetition t and row group g (x fastest: CTAs that run together
// share rows).
struct AddWork {
  int job, x, t, g;
};
__device__ __forceinline__ AddWork add_work(const ProdJob* __restrict__ jobs, int count, int cls) {
  __shared__ int s_job;
  const int id = (int)blockIdx.x;
  for (int j = threadIdx.x; j < count; j += blockDim.x)
    if (add_class(jobs[j]) == cls && id >= jobs[j].add_begin && id - jobs[j].add_begin < jobs[j].add_x * jobs[j].d * jobs[j].G)
      s_job = j;
  __syncthreads();
  AddWork w;
  w.job = s_job;
  const ProdJob& J = jobs[w.job];
  const int e = id - J.add_begin, xt = J.add_x * J.d;
  w.g = e / xt;
  w.t = (e - w.g * xt) / J.add_x;
  w.x = e - w.g * xt - w.t * J.add_x;
  return w;
}

// A warp's look-up of 32 rows (one a lane): first entry, count and key of the
// window in each row
struct RowKeys {
  uint32_t e0, cnt, key, neg1;
};
template <int VARIANT, int JB, typename CumT>
__device__ __forceinline__ RowKeys row_keys(const uint32_t* cA, const CumT* cum, int64_t i, int64_t ie, uint32_t m0,
                                            uint32_t W, uint32_t b, uint32_t cols) {
  RowKeys k{0, 0, 0, 0};
  if (i < ie) {
    const uint32_t c1 = __ldg(cA + i);
    const uint32_t h1 = c1 & (b - 1);
    const uint32_t s = VARIANT == kVariantFFT ? ((m0 - h1) & (b - 1)) : ((m0 ^ h1) & ~(W - 1u));
    k.key = (VARIANT == kVariantFFT ? s : h1) << (JB + 4);
    k.neg1 = ~c1 & 0x80000000u;
    k.e0 = __ldg(cum + s);
    const uint32_t se = s + W;
    k.cnt = se <= b ? __ldg(cum + se) - k.e0 : cols - k.e0 + __ldg(cum + se - b);
  }
  return k;
}
__device__ __forceinline__ uint32_t entry_at(const uint32_t* ent, uint32_t count, uint32_t at) {
  return at < count ? __ldg(ent + at) : kNoEntry;
}
template <int JB>
__device__ __forceinline__ double signed_value(double c, uint32_t e, uint32_t neg1) {
  return __longlong_as_double(__double_as_longlong(c) ^ ((long long)(((e << (28 - JB)) & 0x80000000u) ^ neg1) << 32));
}
__device__ __forceinline__ void load_if(double& v, uint32_t at, bool p) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q ld.shared.f64 %0, [%1];\n\t}" : "+d"(v) : "r"(at), "r"((uint32_t)p) : "memory");
}
__device__ __forceinline__ void store_if(uint32_t at, double v, bool p) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.u32 q, %2, 0;\n\t@q st.shared.f64 [%0], %1;\n\t}" ::"r"(at), "d"(v), "r"((uint32_t)p) : "memory");
}
// Adds Q batches of a row (an entry and its value a lane and batch) to the warp's
// window of W = wmask / 8 + 1 buckets.  Entries of one bucket are neighbours and
// are added one rank after the other; the entries of one rank are in different
// buckets, so the batches' loads, sums and stores overlap.  Bound by latency and
// issue (0.6 of the slots, a third of the shared memory cycles): with a batch at
// a time 4096 x 4096, b = 65536, d = 9 took 0.675 ms, now 0.57; b = 16384 products of
// a batch 4.5 -> 3.4 ms.  (Reading the next row's values before this row's
// additions took 0.83 ms: the ring holds three rows.)
template <int VARIANT, int JB, int Q>
__device__ __forceinline__ void add_row(uint32_t acc, const uint32_t (&e)[Q], const double (&c)[Q], uint32_t key, uint32_t neg1,
                                        uint32_t wmask, int lane) {
  double v[Q], s[Q];
  uint32_t at[Q], rank[Q];
#pragma unroll
  for (int q = 0; q < Q; ++q) {
    rank[q] = e[q] & 7u;
    v[q] = signed_value<JB>(c[q], e[q], neg1);
    at[q] = acc + (((VARIANT == kVariantFFT ? e[q] - key : e[q] ^ key) >> (JB + 1)) & wmask);
    s[q] = 0.0;
  }
  for (uint32_t k = 0; k < 6; ++k) {
#pragma unroll
    for (int q = 0; q < Q; ++q) load_if(s[q], at[q], rank[q] == k);
#pragma unroll
    for (int q = 0; q < Q; ++q) store_if(at[q], s[q] + v[q], rank[q] == k);
    __syncwarp();
    bool more = false;  // an entry of a higher rank
#pragma unroll
    for (int q = 0; q < Q; ++q) more |= rank[q] - (k + 1) < 6u - k;
    if (!__any_sync(0xffffffffu, more)) return;
  }
#pragma unroll
  for (int q = 0; q < Q; ++q)  // six or more: one lane at a time, in order
    for (uint32_t todo = __ballot_sync(0xffffffffu, rank[q] == 6u); todo; todo &= todo - 1u) {
      const bool now = lane == __ffs(todo) - 1;
      load_if(s[q], at[q], now);
      store_if(at[q], s[q] + v[q], now);
      __syncwarp();
    }
}

// ring of row blocks of C filled by one thread of warp kScWin with bulk copies
struct RowRing {
  unsigned char* base;
  uint32_t row_bytes;
  int stages;
};
// (returns the row blocks that it issued)
__device__ __forceinline__ unsigned produce_rows(const ProdJob& J, const RowRing& R, uint64_t* full, uint64_t* empty,
                                                 int64_t ib, int64_t ie, volatile int* wait) {
  unsigned it = 0, st = 0, ph = 0;
  bool ok = true;
  for (int jb = 0; jb < J.blocks && ok; ++jb) {
    const uint32_t cols = (uint32_t)min((int64_t)kScCols, J.n_b - (int64_t)jb * kScCols);
    const uint32_t bytes = ((cols + 1u) & ~1u) * 8u;  // the row stride is even
    for (int64_t i = ib; i < ie; ++i, ++it) {
      if (!bar_wait(&empty[st], ph ^ 1u, wait)) { ok = false; break; }
      bar_expect(&full[st], bytes);
      bulk_load(R.base + st * R.row_bytes, J.C + i * J.ldc + (int64_t)jb * kScCols, bytes, &full[st]);
      if (++st == (unsigned)R.stages) { st = 0; ph ^= 1u; }
    }
  }
  return it;
}
// a wait ran out: report, and let the copies in flight land before the CTA ends
__device__ __forceinline__ void give_up(const ProdJob& J, const RowRing& R, uint64_t* full, unsigned issued,
                                        const ProdWaits& waits, volatile int* wait) {
  *waits.flag = 1;
  *J.flag = 1;
  __threadfence_system();
  for (unsigned z = issued > (unsigned)R.stages ? issued - R.stages : 0; z < issued; ++z)
    bar_drain(&full[z % R.stages], (z / R.stages) & 1u, wait);
}

// Staged form.  A gather from global memory costs one L1 tag cycle per lane (32
// a batch), from shared memory about six wavefronts; what pays is that one CTA
// covers 16 windows, so every staged row serves up to 2^14 buckets.  Warp 16
// copies the row blocks, warps 0-15 own a window each; the next row's entries
// are read while a row is added.
template <int VARIANT>
__device__ __noinline__ void add_staged(const ProdJob& J, int x, int t, int g, uint32_t smem, const ProdWaits& waits) {
  extern __shared__ __align__(128) unsigned char ssm[];
  __shared__ uint64_t full[8], empty[8];
  __shared__ int s_wait[2];
  __shared__ unsigned s_issued;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t b = 1u << J.log2b, W = 1u << J.logW, wmask = (W - 1u) * 8u;
  const uint32_t win0 = x * kScWin, wins = b >> J.logW;
  const int nw = (int)min((uint32_t)kScWin, wins - win0);
  double* acc0 = reinterpret_cast<double*>(ssm);
  const uint32_t acc_bytes = ((uint32_t)kScWin << J.logW) * 8u;
  RowRing R;
  R.base = ssm + acc_bytes;
  R.row_bytes = (((uint32_t)min((int64_t)kScCols, J.n_b) + 15u) & ~15u) * 8u;
  R.stages = (int)min(8u, (smem - acc_bytes) / R.row_bytes);
  if (threadIdx.x == 0) {
    for (int s = 0; s < R.stages; ++s) { bar_init(&full[s], 1 + waits.extra); bar_init(&empty[s], nw); }
    s_wait[0] = 0;
    s_wait[1] = waits.limit_us;
    s_issued = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  volatile int* wait = s_wait;
  const int64_t per = (J.n_a + J.G - 1) / J.G;
  const int64_t ib = (int64_t)g * per, ie = min(ib + per, J.n_a);
  if (warp == kScWin) {
    if (lane == 0) s_issued = produce_rows(J, R, full, empty, ib, ie, wait);
  } else if (warp < nw) {
    const uint32_t m0 = (win0 + warp) << J.logW;
    double* acc = acc0 + (size_t)warp * W;
    for (uint32_t e = lane; e < W; e += 32) acc[e] = 0.0;
    __syncwarp();
    const uint32_t acc_at = smem_u32(acc);
    const uint32_t* cA = J.codesA + (size_t)t * J.n_a;
    int st = 0;
    unsigned ph = 0;
    bool ok = true;
    for (int jb = 0; jb < J.blocks && ok; ++jb) {
      const uint32_t cols = (uint32_t)min((int64_t)kScCols, J.n_b - (int64_t)jb * kScCols);
      const uint16_t* cum = reinterpret_cast<const uint16_t*>(J.cum) + ((size_t)t * J.blocks + jb) * cum16_stride(J.log2b);
      const uint32_t* ent = J.ent + 2 * ((size_t)t * J.n_b + (size_t)jb * kScCols);
      const char* C = reinterpret_cast<const char*>(J.C + (size_t)jb * kScCols);
      auto entries = [&](const RowKeys& k, int r, uint32_t (&x)[3]) {
        const uint32_t n = __shfl_sync(0xffffffffu, k.cnt, r);
        const uint32_t* at = ent + __shfl_sync(0xffffffffu, k.e0, r);
#pragma unroll
        for (int q = 0; q < 3; ++q) x[q] = entry_at(at, n, lane + 32 * q);
        return n;
      };
      auto values = [&](const uint32_t (&x)[3], uint32_t n, double (&y)[3]) {  // (a lane without an entry reads column 0)
        ok = __all_sync(0xffffffffu, bar_wait(&full[st], ph, wait));
        if (!ok) return;
        const char* row = reinterpret_cast<const char*>(R.base) + st * R.row_bytes;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
          y[q] = 0.0;
          if (n > 32 * q) y[q] = *reinterpret_cast<const double*>(row + (x[q] & kColMask<12>));
        }
      };
      auto release = [&] {
        __syncwarp();
        if (lane == 0) bar_arrive(&empty[st]);
        if (++st == R.stages) { st = 0; ph ^= 1u; }
      };
      auto rest = [&](uint32_t e0, uint32_t n, int64_t i, uint32_t key, uint32_t neg1) {  // entries from the 97th on
        for (uint32_t at = 96; at < n; at += 32) {
          const uint32_t x[1] = {entry_at(ent + e0, n, at + lane)};
          const double y[1] = {__ldg(reinterpret_cast<const double*>(C + i * J.ldc * 8 + (x[0] & kColMask<12>)))};
          add_row<VARIANT, 12>(acc_at, x, y, key, neg1, wmask, lane);
        }
      };
      for (int64_t r0 = ib; r0 < ie && ok; r0 += 32) {
        const RowKeys k = row_keys<VARIANT, 12>(cA, cum, r0 + lane, ie, m0, W, b, cols);
        const int rows = (int)min((int64_t)32, ie - r0);
        uint32_t f[3];
        uint32_t nf = entries(k, 0, f);
        for (int r = 0; r < rows; ++r) {
          const uint32_t e[3] = {f[0], f[1], f[2]}, ne = nf;
          if (r + 1 < rows) nf = entries(k, r + 1, f);
          const uint32_t key = __shfl_sync(0xffffffffu, k.key, r), neg1 = __shfl_sync(0xffffffffu, k.neg1, r);
          double v[3];
          values(e, ne, v);
          if (!ok) break;
          if (ne > 64) add_row<VARIANT, 12, 3>(acc_at, e, v, key, neg1, wmask, lane);
          else add_row<VARIANT, 12, 2>(acc_at, {e[0], e[1]}, {v[0], v[1]}, key, neg1, wmask, lane);
          if (ne > 96) rest(__shfl_sync(0xffffffffu, k.e0, r), ne, r0 + r, key, neg1);
          release();
        }
      }
    }
    double* out = J.part + ((size_t)g * J.d + t) * b + m0;
    for (uint32_t e = lane; e < W; e += 32) out[e] = acc[e];
  }
  __syncthreads();
  if (s_wait[0] && threadIdx.x == 0) give_up(J, R, full, s_issued, waits, wait);
}

template <int PER_SM>
__global__ void __launch_bounds__(kScThreads, PER_SM) k_prod_add_staged(const ProdJob* __restrict__ jobs, int count,
                                                                        uint32_t smem, const __grid_constant__ ProdWaits waits) {
  const AddWork w = add_work(jobs, count, PER_SM);
  const ProdJob& J = jobs[w.job];
  if (J.variant == kVariantFFT) add_staged<kVariantFFT>(J, w.x, w.t, w.g, smem, waits);
  else add_staged<kVariantFWHT>(J, w.x, w.t, w.g, smem, waits);
}

// Lane form: thread = NB buckets (sums in registers); for row i bucket m adds
// the run of entries of h2 = m - h1(i) (FWHT: m ^ h1(i)).  The sorted columns
// of the block and the rows are in shared memory.
template <int VARIANT, int NB>
__device__ __noinline__ void add_lane(const ProdJob& J, int t, int g, uint32_t smem, const ProdWaits& waits) {
  extern __shared__ __align__(128) unsigned char ssm[];
  __shared__ uint64_t full[8], empty[8];
  __shared__ int s_wait[2];
  __shared__ unsigned s_issued;
  constexpr uint32_t b = 512u * NB;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  uint32_t* es = reinterpret_cast<uint32_t*>(ssm);                         // kScCols entries
  uint16_t* cs = reinterpret_cast<uint16_t*>(ssm + kScCols * 4);           // b + 8 positions
  constexpr uint32_t list_bytes = kScCols * 4 + ((b + 8) * 2 + 127) / 128 * 128;
  RowRing R;
  R.base = ssm + list_bytes;
  R.row_bytes = (((uint32_t)min((int64_t)kScCols, J.n_b) + 15u) & ~15u) * 8u;
  R.stages = (int)min(8u, (smem - list_bytes) / R.row_bytes);
  if (tid == 0) {
    for (int s = 0; s < R.stages; ++s) { bar_init(&full[s], 1 + waits.extra); bar_init(&empty[s], kScWin); }
    s_wait[0] = 0;
    s_wait[1] = waits.limit_us;
    s_issued = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  volatile int* wait = s_wait;
  const int64_t per = (J.n_a + J.G - 1) / J.G;
  const int64_t ib = (int64_t)g * per, ie = min(ib + per, J.n_a);
  if (warp == kScWin) {
    if (lane == 0) s_issued = produce_rows(J, R, full, empty, ib, ie, wait);
  } else {
    const uint32_t* cA = J.codesA + (size_t)t * J.n_a;
    double acc[NB];
#pragma unroll
    for (int q = 0; q < NB; ++q) acc[q] = 0.0;
    int st = 0;
    unsigned ph = 0;
    bool ok = true;
    for (int jb = 0; jb < J.blocks; ++jb) {  // (every warp takes every block's barriers)
      const uint32_t cols = (uint32_t)min((int64_t)kScCols, J.n_b - (int64_t)jb * kScCols);
      const uint16_t* cum = reinterpret_cast<const uint16_t*>(J.cum) + ((size_t)t * J.blocks + jb) * cum16_stride(J.log2b);
      const uint32_t* ent = J.ent + 2 * ((size_t)t * J.n_b + (size_t)jb * kScCols);
      asm volatile("bar.sync 1, 512;" ::: "memory");  // the previous block's list is no longer read
      for (uint32_t e = tid; e < cols; e += 512) es[e] = __ldg(ent + e);
      for (uint32_t e = tid; e <= b; e += 512) cs[e] = __ldg(cum + e);
      asm volatile("bar.sync 1, 512;" ::: "memory");
      for (int64_t r0 = ib; r0 < ie && ok; r0 += 32) {
        const uint32_t codes = r0 + lane < ie ? __ldg(cA + r0 + lane) : 0u;
        const int rows = (int)min((int64_t)32, ie - r0);
        for (int r = 0; r < rows; ++r) {
          const uint32_t c1 = __shfl_sync(0xffffffffu, codes, r);
          const uint32_t h1 = c1 & (b - 1);
          ok = __all_sync(0xffffffffu, bar_wait(&full[st], ph, wait));
          if (!ok) break;
          const char* row = reinterpret_cast<const char*>(R.base) + st * R.row_bytes;
#pragma unroll
          for (int q = 0; q < NB; ++q) {
            const uint32_t m = q * 512 + tid;
            const uint32_t h2 = VARIANT == kVariantFFT ? ((m - h1) & (b - 1)) : (m ^ h1);
            const uint32_t end = cs[h2 + 1];
            double s = 0.0;
            for (uint32_t e = cs[h2]; e < end; ++e) {
              const uint32_t x = es[e];
              s += signed_value<12>(*reinterpret_cast<const double*>(row + (x & kColMask<12>)), x, 0u);
            }
            acc[q] += c1 >> 31 ? s : -s;
          }
          __syncwarp();
          if (lane == 0) bar_arrive(&empty[st]);
          if (++st == R.stages) { st = 0; ph ^= 1u; }
        }
      }
    }
    double* out = J.part + ((size_t)g * J.d + t) * b;
#pragma unroll
    for (int q = 0; q < NB; ++q) out[q * 512 + tid] = acc[q];
  }
  __syncthreads();
  if (s_wait[0] && tid == 0) give_up(J, R, full, s_issued, waits, wait);
}

template <int NB>
__global__ void __launch_bounds__(kScThreads, 1) k_prod_add_lane(const ProdJob* __restrict__ jobs, int count,
                                                                 uint32_t smem, const __grid_constant__ ProdWaits waits) {
  const AddWork w = add_work(jobs, count, NB == 1 ? 3 : (NB == 2 ? 4 : 5));
  const ProdJob& J = jobs[w.job];
  if (J.variant == kVariantFFT) add_lane<kVariantFFT, NB>(J, w.t, w.g, smem, waits);
  else add_lane<kVariantFWHT, NB>(J, w.t, w.g, smem, waits);
}

// Gather form: windows as in the staged form, values from L2.  Entries are read
// two rows ahead and values one row ahead of the additions, so a row's chain
// of two L2 latencies overlaps the rows before it.
template <int VARIANT>
__device__ __forceinline__ void add_gather(const ProdJob& J, int x, int t, int g) {
  extern __shared__ double sacc[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const uint32_t b = 1u << J.log2b, W = 1u << J.logW, wmask = (W - 1u) * 8u;
  const uint32_t m0 = (x * kGaWarps + warp) << J.logW;
  if (m0 >= b) return;
  double* acc = sacc + (size_t)warp * W;
  for (uint32_t e = lane; e < W; e += 32) acc[e] = 0.0;
  __syncwarp();
  const uint32_t acc_at = smem_u32(acc);
  const uint32_t cols = (uint32_t)J.n_b;
  const uint32_t* cum = reinterpret_cast<const uint32_t*>(J.cum) + (size_t)t * (b + 1);
  const uint32_t* ent = J.ent + 2 * (size_t)t * cols;
  const uint32_t* cA = J.codesA + (size_t)t * J.n_a;
  const int64_t per = (J.n_a + J.G - 1) / J.G;
  const int64_t ib = (int64_t)g * per, ie = min(ib + per, J.n_a);
  const size_t ldc = (size_t)J.ldc * 8;
  for (int64_t r0 = ib; r0 < ie; r0 += 32) {
    const RowKeys k = row_keys<VARIANT, 17>(cA, cum, r0 + lane, ie, m0, W, b, cols);
    const int rows = (int)min((int64_t)32, ie - r0);
    const char* row = reinterpret_cast<const char*>(J.C) + (size_t)r0 * ldc;  // of row r
    auto value = [&](const char* at, uint32_t e) {
      return e != kNoEntry ? __ldg(reinterpret_cast<const double*>(at + (e & kColMask<17>))) : 0.0;
    };
    auto entries = [&](int r, uint32_t (&x)[3]) {
      const uint32_t n = r < rows ? __shfl_sync(0xffffffffu, k.cnt, r) : 0u;
      const uint32_t* at = ent + __shfl_sync(0xffffffffu, k.e0, r & 31);
#pragma unroll
      for (int q = 0; q < 3; ++q) x[q] = entry_at(at, n, lane + 32 * q);
    };
    uint32_t e[3], f[3], h[3];  // rows r, r + 1, r + 2
    double v[3], w[3];          // rows r, r + 1
    entries(0, e);
    entries(1, f);
#pragma unroll
    for (int q = 0; q < 3; ++q) v[q] = value(row, e[q]);
    for (int r = 0; r < rows; ++r) {
#pragma unroll
      for (int q = 0; q < 3; ++q) w[q] = value(row + ldc, f[q]);
      entries(r + 2, h);
      const uint32_t key = __shfl_sync(0xffffffffu, k.key, r), neg1 = __shfl_sync(0xffffffffu, k.neg1, r);
      const uint32_t cc = __shfl_sync(0xffffffffu, k.cnt, r);
      if (cc > 64) add_row<VARIANT, 17, 3>(acc_at, e, v, key, neg1, wmask, lane);
      else add_row<VARIANT, 17, 2>(acc_at, {e[0], e[1]}, {v[0], v[1]}, key, neg1, wmask, lane);
      if (cc > 96) {
        const uint32_t* ec = ent + __shfl_sync(0xffffffffu, k.e0, r);
        for (uint32_t at = 96; at < cc; at += 32) {
          const uint32_t x[1] = {entry_at(ec, cc, at + lane)};
          const double y[1] = {value(row, x[0])};
          add_row<VARIANT, 17>(acc_at, x, y, key, neg1, wmask, lane);
        }
      }
#pragma unroll
      for (int q = 0; q < 3; ++q) {
        e[q] = f[q];
        f[q] = h[q];
        v[q] = w[q];
      }
      row += ldc;
    }
  }
  double* out = J.part + ((size_t)g * J.d + t) * b + m0;
  for (uint32_t e = lane; e < W; e += 32) out[e] = acc[e];
}

__global__ void __launch_bounds__(kGaWarps * 32) k_prod_add_gather(const ProdJob* __restrict__ jobs, int count) {
  const AddWork w = add_work(jobs, count, 0);
  const ProdJob& J = jobs[w.job];
  if (J.variant == kVariantFFT) add_gather<kVariantFFT>(J, w.x, w.t, w.g);
  else add_gather<kVariantFWHT>(J, w.x, w.t, w.g);
}

// p = sum of the row groups' partial sketches (NaN when the flag is set)
__global__ void __launch_bounds__(256) k_prod_reduce(const ProdJob* __restrict__ jobs) {
  const ProdJob& J = jobs[blockIdx.y];
  const int64_t db = (int64_t)J.d << J.log2b;
  const bool bad = *J.flag == 1;
  for (int64_t e = (int64_t)blockIdx.x * 256 + threadIdx.x; e < db; e += (int64_t)gridDim.x * 256) {
    double s = 0.0;
    for (int g = 0; g < J.G; ++g) s += J.part[(size_t)g * db + e];
    J.p[e] = bad ? __longlong_as_double(0x7ff8000000000000ll) : s;
  }
}

}  // namespace

bool product_supported(int b, int64_t n_a, int64_t n_inner, int64_t n_b) {
  return n_inner > 0 && n_a > 0 && n_b > 0 && n_a <= 0x7fffffff && n_b <= 0x7fffffff && n_a * n_b <= kProdMaxEntries &&
         b >= 512 && (b <= 65536 || n_b <= 131072) &&  // what the forms of the additions take
         n_b <= 65535ll * kScCols;                     // blocks of columns in a launch
}

// Shared memory of a staged or lane CTA: its windows or lists and a ring of up
// to eight row blocks; staged, where windows and three row blocks take no more
// than half an SM, two CTAs share it (1.2 to 1.4 times as fast: 4000 x 2048, b =
// 8192, d = 7 0.315 -> 0.252 ms).
static size_t add_fixed(const ProdJob& J) {
  return J.form == kAddStaged ? ((size_t)kScWin << J.logW) * 8 : (size_t)kScCols * 4 + ((size_t)2 << J.log2b) + 128;
}
static size_t add_row(const ProdJob& J) { return (((size_t)std::min<int64_t>(J.n_b, kScCols) + 15) & ~(size_t)15) * 8; }
static size_t add_smem(const ProdJob& J) {
  return std::min(add_fixed(J) + 8 * add_row(J), J.per_sm == 2 ? kScSmemHalf : kScSmemMax);
}

void product_geometry(ProdJob& J, int variant, int d, int b, int64_t n_a, int64_t n_b, int64_t kc, bool alone, int sms) {
  J.variant = variant;
  J.d = d;
  J.n_a = n_a;
  J.n_b = n_b;
  J.kc = kc;
  J.ldc = prod_ldc(n_b);
  J.tiles_a = J.tiles_p = (int)((n_a + 255) / 256);
  J.tiles_b = (int)((n_b + 255) / 256);
  J.tile0 = 0;
  J.accumulate = 0;
  J.log2b = 0;
  while ((1 << J.log2b) < b) ++J.log2b;
  const int64_t cols = std::max<int64_t>(std::min<int64_t>(n_b, kScCols), 1);
  J.blocks = (int)((n_b + kScCols - 1) / kScCols);
  // Lane where the columns of a block are 1.5 times the buckets and more (4000 x
  // 4000, b = 2048, d = 9: lane 0.46 ms, staged 0.64; 8000 x 8000, b = 4096, d = 7:
  // 2.39 and 2.11); among other jobs 2.5 times, since a launch of its own for a
  // few long CTAs costs more (64 uneven products: 12.55 ms a run at 1.5, 12.26).
  J.form = J.log2b > 16 ? kAddGather : (2 * cols >= (alone ? 3 : 5) * (int64_t)b ? kAddLane : kAddStaged);
  // Windows: 48 to 96 entries of a row (two or three batches a warp; 4000 x 1385, b =
  // 8192: 36 to 72 227 G/s, 48 to 96 275), at most 1024 buckets (8 KB of shared
  // memory a warp).  Half as many where that lets two CTAs share an SM and
  // leaves 36 (batches of b = 16384 products: 3.5 -> 3.4 ms).
  const int64_t per_row = J.form == kAddGather ? std::max<int64_t>(n_b, 1) : cols;
  J.logW = 5;
  while (J.logW < 10 && ((int64_t)2 << J.logW) * per_row <= 96 * (int64_t)b) ++J.logW;
  J.logW = std::min(J.logW, J.log2b);
  auto two = [&] { return J.form == kAddStaged && add_fixed(J) + 3 * add_row(J) <= kScSmemHalf; };
  if (J.form == kAddStaged && !two() && J.logW > 5 && ((int64_t)1 << J.logW) * per_row > 72 * (int64_t)b) {
    --J.logW;
    if (!two()) ++J.logW;
  }
  J.per_sm = two() ? 2 : 1;
  const int64_t wins = (int64_t)b >> J.logW, most = std::min<int64_t>((n_a + 31) / 32, 512);
  int64_t G;
  if (J.form == kAddGather) {
    // Row groups of at most 32 MB of C: the CTAs in flight then work on about
    // two groups, which stay in L2.  (16384 rows of 16384 columns, b = 2^18: 60
    // ms in 3 groups, whose CTAs drift apart and miss L2; 11.6 ms in 64.)
    const int64_t rows = std::max<int64_t>(32, ((int64_t)32 << 20) / (8 * per_row));
    const int64_t fill = alone ? 12 * (int64_t)sms / (d * ((wins + kGaWarps - 1) / kGaWarps)) : 0;
    G = std::max((n_a + rows - 1) / rows, fill);
  } else {
    // The CTAs that fit, and up to three times as many where they keep 512 rows,
    // since some SMs are faster than others (16384 rows, b = 65536: 9.45 -> 8.7
    // ms).  Among other jobs 256 rows, which outweigh a CTA's start and end (64
    // uneven products: 512 rows 13.4 ms a run, 256 12.3, 128 12.3).
    const int64_t ctas = J.form == kAddLane ? d : d * ((wins + kScWin - 1) / kScWin);
    if (alone) {
      G = std::min<int64_t>(J.per_sm * sms / ctas, 64);
      if (J.form == kAddStaged) G = std::max(G, std::min(3 * G, n_a / 512));
    } else {
      G = (n_a + 255) / 256;
    }
  }
  // (16384 rows of 16384 columns, b = 2^24, d = 9: 64 groups would take 77 GB)
  const int64_t fit = (int64_t)(kProdMaxBytes / ((size_t)d * (size_t)b * 8));
  J.G = (int)std::max<int64_t>(1, std::min({G, most, fit}));
}

// --------------------------------------------------------------- device memory
namespace {
size_t up256(size_t n) { return (n + 255) & ~(size_t)255; }
size_t cum_bytes(const ProdJob& J) {
  return J.form == kAddGather ? (size_t)J.d * (((size_t)1 << J.log2b) + 1) * 4
                              : (size_t)J.d * J.blocks * cum16_stride(J.log2b) * 2;
}
// residue planes of n columns (in tiles of 256)
size_t plane_bytes(int tiles, int64_t kc, bool f32) {
  return (size_t)prod_moduli(f32) * 2 * tiles * prod_ksteps(kc) * kProdSlab;
}
// visits the parts of the work space in order
template <typename F>
void work_parts(const ProdJob& J, bool f32, bool own_c, F&& part) {
  const size_t n = (size_t)(J.n_a + J.n_b), nb = (size_t)((J.kc + kProdColRows - 1) / kProdColRows);
  part(0, plane_bytes(J.tiles_a, J.kc, f32));
  part(1, plane_bytes(J.tiles_b, J.kc, f32));
  part(2, prod_residue_row(J, f32) * J.tiles_p);
  part(3, (n + (size_t)J.kc + 1) * 4);
  part(4, nb * n * 8);
  part(5, nb * n * 4);
  part(6, (size_t)J.G * ((size_t)J.d << J.log2b) * 8);
  if (own_c) part(7, (size_t)J.n_a * (size_t)J.ldc * 8);
}
}  // namespace

size_t product_list_bytes(const ProdJob& J) { return up256(cum_bytes(J)) + up256(2 * (size_t)J.d * (size_t)J.n_b * 4); }
void product_set_lists(ProdJob& J, void* base) {
  J.cum = base;
  J.ent = reinterpret_cast<uint32_t*>(static_cast<uint8_t*>(base) + up256(cum_bytes(J)));
}
// (rows are copied in 16-byte units)
bool product_usable_c(const ProdJob& J, const double* c) {
  return c && J.ldc == J.n_b && reinterpret_cast<uintptr_t>(c) % 16 == 0;
}
size_t product_work_bytes(const ProdJob& J, bool f32, bool own_c) {
  size_t total = 0;
  work_parts(J, f32, own_c, [&](int, size_t n) { total += up256(n); });
  return total;
}
void product_set_work(ProdJob& J, void* base, bool f32, double* c) {
  const bool own_c = !product_usable_c(J, c);
  J.C = c;
  uint8_t* at = static_cast<uint8_t*>(base);
  work_parts(J, f32, own_c, [&](int i, size_t n) {
    switch (i) {
      case 0: J.slA = at; break;
      case 1: J.slB = at; break;
      case 2: J.res = reinterpret_cast<uint32_t*>(at); break;
      case 3:
        J.flag = reinterpret_cast<int*>(at);
        J.cexpA = J.flag + 1;
        J.cexpB = J.cexpA + J.n_a;
        J.rexp = J.cexpB + J.n_b;
        break;
      case 4: J.csum = reinterpret_cast<double*>(at); break;
      case 5: J.cmax = reinterpret_cast<int*>(at); break;
      case 6: J.part = reinterpret_cast<double*>(at); break;
      default: J.C = reinterpret_cast<double*>(at);
    }
    at += up256(n);
  });
}

void launch_product_index(const ProdJob* hJobs, const ProdJob* dJobs, int count, cudaStream_t s) {
  if (count <= 0) return;
  int d[2] = {}, blocks = 0, parts = 0;
  for (int i = 0; i < count; ++i) {
    const bool gather = hJobs[i].form == kAddGather;
    int& m = d[gather ? 0 : 1];
    m = std::max(m, hJobs[i].d);
    if (gather) parts = std::max(parts, (int)((1u << hJobs[i].log2b) / kIdxBuckets));
    else blocks = std::max(blocks, hJobs[i].blocks);
  }
  ProfScope prof("plan", s);
  if (d[0]) {
    count_launch();
    k_prod_index<<<dim3((unsigned)d[0], (unsigned)parts, (unsigned)count), kIdxThreads, 0, s>>>(dJobs);
    CMM_CUDA(cudaGetLastError());
  }
  if (d[1]) {
    count_launch();
    k_prod_index_blocks<<<dim3((unsigned)d[1], (unsigned)blocks, (unsigned)count), kIdxThreads, 0, s>>>(dJobs);
    CMM_CUDA(cudaGetLastError());
  }
}

int product_launches(const ProdJob* hJobs, int count) {
  bool used[kAddClasses] = {}, cexp = false;
  for (int i = 0; i < count; ++i) {
    used[add_class(hJobs[i])] = true;
    cexp |= hJobs[i].kc > kProdColRows;
  }
  int n = 2 + (cexp ? 1 : 0) + 2 + 2 + 1;  // rows, columns, (their sums), planes, product, residues -> C, sums
  for (bool u : used) n += u ? 1 : 0;
  return n;
}

void product_layout(ProdJob* jobs, int count, bool f32) {
  int64_t items = 0, ctas[kAddClasses] = {};
  for (int i = 0; i < count; ++i) {
    ProdJob& J = jobs[i];
    items += (int64_t)J.tiles_p * J.tiles_b * prod_moduli(f32);
    J.item_end = items;
    const int64_t wins = ((int64_t)1 << J.log2b) >> J.logW;
    J.add_x = J.form == kAddLane ? 1 : (int)((wins + (J.form == kAddStaged ? kScWin : kGaWarps) - 1) / (J.form == kAddStaged ? kScWin : kGaWarps));
    int64_t& c = ctas[add_class(J)];
    J.add_begin = (int)c;
    c += (int64_t)J.add_x * J.d * J.G;
    if (c > 0x7fffffff) throw unsupported("product sketch: too many work items");
  }
}

namespace {

template <typename K, typename... A>
void launch_add(K kernel, int64_t ctas, size_t smem, int threads, cudaStream_t s, A... args) {
  if (!ctas) return;
  // (the same for every launch: threads launch these kernels at the same time)
  CMM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kScSmemMax));
  count_launch();
  kernel<<<(unsigned)ctas, threads, smem, s>>>(args...);
  CMM_CUDA(cudaGetLastError());
}

}  // namespace

void launch_product_add(const ProdJob* hJobs, const ProdJob* dJobs, int count, int* flag, cudaStream_t s) {
  if (count <= 0) return;
  ProfScope prof("finalize", s);
  int64_t ctas[kAddClasses] = {};
  size_t smem[kAddClasses] = {};
  for (int i = 0; i < count; ++i) {
    const ProdJob& J = hJobs[i];
    const int c = add_class(J);
    ctas[c] += (int64_t)J.add_x * J.d * J.G;
    smem[c] = std::max(smem[c], c == 0 ? ((size_t)kGaWarps << J.logW) * 8 : add_smem(J));
  }
  const ProdWaits waits = product_waits(flag, "add");
  launch_add(k_prod_add_gather, ctas[0], smem[0], kGaWarps * 32, s, dJobs, count);
  launch_add(k_prod_add_staged<1>, ctas[1], smem[1], kScThreads, s, dJobs, count, (uint32_t)smem[1], waits);
  launch_add(k_prod_add_staged<2>, ctas[2], smem[2], kScThreads, s, dJobs, count, (uint32_t)smem[2], waits);
  launch_add(k_prod_add_lane<1>, ctas[3], smem[3], kScThreads, s, dJobs, count, (uint32_t)smem[3], waits);
  launch_add(k_prod_add_lane<2>, ctas[4], smem[4], kScThreads, s, dJobs, count, (uint32_t)smem[4], waits);
  launch_add(k_prod_add_lane<4>, ctas[5], smem[5], kScThreads, s, dJobs, count, (uint32_t)smem[5], waits);
  int64_t db = 0;
  for (int i = 0; i < count; ++i) db = std::max<int64_t>(db, (int64_t)hJobs[i].d << hJobs[i].log2b);
  count_launch();
  k_prod_reduce<<<dim3((unsigned)std::min<int64_t>((db + 255) / 256, 2048), (unsigned)count), 256, 0, s>>>(dJobs);
  CMM_CUDA(cudaGetLastError());
}

}  // namespace cmm
