// Product sketch: the sketch of C = A^T B from C itself.
//
// p_t is the count sketch of the product: p_t[idx(i, j)] += s1_t(i) s2_t(j)
// C[i][j], idx = (h1 + h2) mod b (FFT variant) or h1 ^ h2 (FWHT variant).
// The transform kernels reach it through d length-b transforms per inner
// index; here C is formed once, to FP64 (FP32) accuracy, on the int8 tensor
// cores and then added into the d sketches.  Per inner index that is
// 2 n_a n_b flops of matrix product instead of d transforms of length b, and
// the matrix product runs on tcgen05 while the transforms run on the FP64 /
// FP32 units.
//
// The product is an exact integer product, by residues:
//  * Row pair k is balanced by a power of two e_k (A row * 2^-e_k, B row *
//    2^e_k: the same rule as the FFT packing).  Column c of A or B then gets
//    the power of two E_c >= its 2-norm over k, and an entry x is the integer
//    X = rint(x 2^(T - E_c)), so every column of integers has norm <= 2^T and
//    every entry of the integer product is below 2^(2T) (Cauchy-Schwarz),
//    whatever the number of inner indices.
//  * The integer product is formed modulo N pairwise coprime m_i <= 256: the
//    residues of X fit signed bytes, their products add up exactly in the
//    int32 accumulators, and with M = m_1 ... m_N > 2^(2T + 1) the residues
//    determine the entry (Chinese remainder theorem).  N = 15, T = 58 for
//    FP64 inputs, N = 8, T = 31 for FP32 inputs.  (Splitting X into base-256
//    digits instead needs 34 and 13 int8 products for the same accuracy.)
// The only rounding is that of X: an error of about 2^-59 (2^-32) |a_i| |b_j|
// per entry, in the norms of the balanced columns.  Balancing makes the two
// rows of a pair equally large, so this is normwise the error of FP64 (FP32)
// transforms or smaller.
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <utility>
#include <vector>

#include "cmm_internal.h"
#include "cmm_product.h"
#include "cmm_product_dev.cuh"

namespace cmm {
namespace {

constexpr int kNoExp = -1000000;     // column without a nonzero entry
constexpr int kMinExp = -960;        // smaller columns are scaled as if they were this large

// pairwise coprime, descending
__host__ __device__ constexpr int modulus(int i) {
  constexpr int m[15] = {256, 255, 253, 251, 247, 241, 239, 233, 229, 227, 223, 217, 211, 199, 197};
  return m[i];
}
constexpr int powmod2(int e, int m) {  // 2^e mod m
  int r = 1 % m;
  for (int i = 0; i < e; ++i) r = (r * 2) % m;
  return r;
}
constexpr int invmod(int a, int m) {  // a^-1 mod m (a, m coprime)
  for (int x = 1; x < m; ++x)
    if ((a % m) * x % m == 1) return x;
  return 0;
}
// (M / m_i)^-1 mod m_i for the first n moduli
constexpr int crt_inv(int i, int n) {
  int p = 1 % modulus(i);
  for (int j = 0; j < n; ++j)
    if (j != i) p = p * (modulus(j) % modulus(i)) % modulus(i);
  return invmod(p, modulus(i));
}
// floor(v / m) = umulhi(v, magic) >> 7 exactly for v < 2^31
__host__ __device__ constexpr uint32_t mod_magic(int m) {
  return (uint32_t)((m & (m - 1)) == 0 ? (1ull << 39) / m : (1ull << 39) / m + 1);
}

struct U128 {
  unsigned long long lo, hi;
};
// product of the first n moduli without m_skip (skip < 0: all), mod 2^128
constexpr U128 mod_product(int n, int skip) {
  unsigned __int128 p = 1;
  for (int j = 0; j < n; ++j)
    if (j != skip) p *= (unsigned)modulus(j);
  return U128{(unsigned long long)p, (unsigned long long)(p >> 64)};
}

template <typename Real>
struct Fix;
template <>
struct Fix<double> {
  static constexpr int N = 15, T = 58;
};
template <>
struct Fix<float> {
  static constexpr int N = 8, T = 31;
};

// ------------------------------------------------------------- row balance
// e_k = (expo(max |A row|) - expo(max |B row|)) / 2, within the range of pow2; kPSkip
// when a row is zero.  A row pair with a non-finite value makes the whole
// sketch NaN, as the transforms would (flag[0] = 1; the FFT form skips row
// pairs with a zero row first, as its transform kernels do).
//
// Bound by latency: a CTA of four warps per row pair keeps four loads a thread
// in flight and takes several rows, and the largest magnitude is that of the
// bit patterns, one integer maximum a value (256 threads, one load, FP64
// maxima: 56 us at 4096 x 4096, 52 now; 64 uneven FP32 products 510 -> 197 us).
constexpr int kRowThreads = 128, kRowUnroll = 4;
// largest magnitude's bits (FP64: of the high word, and whether any value is not zero)
struct RowMax {
  uint32_t hi = 0, any = 0;
};
__device__ __forceinline__ void row_take(RowMax& m, double v) {
  const uint32_t h = (uint32_t)__double2hiint(v) & 0x7fffffffu;
  m.hi = max(m.hi, h);
  m.any |= h | (uint32_t)__double2loint(v);
}
__device__ __forceinline__ void row_take(RowMax& m, float v) { m.hi = max(m.hi, __float_as_uint(v) & 0x7fffffffu); }
template <typename Real>
__device__ __forceinline__ RowMax row_max(const Real* __restrict__ x, int64_t n) {
  RowMax m;
  for (int64_t i = threadIdx.x; i < n; i += kRowUnroll * kRowThreads) {
    Real v[kRowUnroll];
#pragma unroll
    for (int u = 0; u < kRowUnroll; ++u) v[u] = i + u * kRowThreads < n ? __ldg(x + i + u * kRowThreads) : (Real)0;
#pragma unroll
    for (int u = 0; u < kRowUnroll; ++u) row_take(m, v[u]);
  }
  m.hi = __reduce_max_sync(0xffffffffu, m.hi);
  m.any = sizeof(Real) == 8 ? __reduce_or_sync(0xffffffffu, m.any) : m.hi;
  return m;
}
template <typename Real>
__global__ void __launch_bounds__(kRowThreads) k_prod_rows(const ProdJob* __restrict__ jobs) {
  const ProdJob& J = jobs[blockIdx.y];
  constexpr int kWarps = kRowThreads / 32;
  __shared__ uint32_t part[2][kWarps][4];  // (two rows: one barrier a row)
  const int w = threadIdx.x >> 5;
  int buf = 0;
  for (int64_t k = blockIdx.x; k < J.kc; k += gridDim.x, buf ^= 1) {
    const RowMax a = row_max(reinterpret_cast<const Real*>(J.A) + k * J.n_a, J.n_a);
    const RowMax b = row_max(reinterpret_cast<const Real*>(J.B) + k * J.n_b, J.n_b);
    if ((threadIdx.x & 31) == 0) {
      part[buf][w][0] = a.hi;
      part[buf][w][1] = a.any;
      part[buf][w][2] = b.hi;
      part[buf][w][3] = b.any;
    }
    constexpr uint32_t kInf = sizeof(Real) == 8 ? 0x7ff00000u : 0x7f800000u;
    const bool bad = __syncthreads_or(a.hi >= kInf || b.hi >= kInf);
    bool some = true;
    if (bad) {  // a row counts as zero when all its numbers are, whatever NaNs it has
      bool sa = false, sb = false;
      for (int64_t i = threadIdx.x; i < J.n_a; i += kRowThreads) sa |= fabs((double)reinterpret_cast<const Real*>(J.A)[k * J.n_a + i]) > 0.0;
      for (int64_t j = threadIdx.x; j < J.n_b; j += kRowThreads) sb |= fabs((double)reinterpret_cast<const Real*>(J.B)[k * J.n_b + j]) > 0.0;
      sa = __syncthreads_or(sa);
      some = __syncthreads_or(sb) && sa;
    }
    if (threadIdx.x == 0) {
      uint32_t ha = 0, na = 0, hb = 0, nb = 0;
      for (int i = 0; i < kWarps; ++i) {
        ha = max(ha, part[buf][i][0]);
        na |= part[buf][i][1];
        hb = max(hb, part[buf][i][2]);
        nb |= part[buf][i][3];
      }
      // exponent of the largest magnitude (-1023: an FP64 subnormal)
      auto ex = [](uint32_t h) {
        if (sizeof(Real) == 4) h = (uint32_t)__double2hiint((double)__uint_as_float(h));
        return (int)(h >> 20) - 1023;
      };
      int e;
      if (na == 0 || nb == 0 || !some) {
        e = kPSkip;
      } else {
        e = (ex(ha) - ex(hb)) / 2;
        e = e > 1000 ? 1000 : (e < -1000 ? -1000 : e);
      }
      J.rexp[k] = e;
      if (bad && (e != kPSkip || J.variant != kVariantFFT)) *J.flag = 1;
    }
  }
}

// --------------------------------------------------------- column exponents
// E_c = the least power of two at or above the 2-norm of balanced column c.
// Thread = column; block = 128 columns x kColRows inner indices, whose sums of
// squares and largest exponents go to csum / cmax (k_prod_cexp adds them up in
// a fixed order; with one block of rows it is done here).  When the sum of
// squares leaves the FP64 range, the bound from the largest entry serves.
constexpr int kColRows = kProdColRows;
__device__ __forceinline__ int norm_exp(double sum, int mx, int64_t kc) {
  if (mx <= kNoExp) return kNoExp;
  if (sum > 1e-270 && sum < 1e300) {
    const int q = (int)((__double_as_longlong(sum * (1.0 + 1e-9)) >> 52) & 0x7ff) - 1022;  // sum < 2^q
    return (q + 1) >> 1;
  }
  return mx + 1 + (64 - __clzll((unsigned long long)kc) + 1) / 2;
}
template <typename Real>
__global__ void __launch_bounds__(128) k_prod_cols(const ProdJob* __restrict__ jobs) {
  const ProdJob& J = jobs[blockIdx.z >> 1];
  const int side = blockIdx.z & 1;
  const int64_t n = side ? J.n_b : J.n_a;
  const int64_t c = (int64_t)blockIdx.x * 128 + threadIdx.x;
  if (c >= n) return;
  const Real* X = reinterpret_cast<const Real*>(side ? J.B : J.A) + c;
  for (int64_t r = blockIdx.y; r * kColRows < J.kc; r += gridDim.y) {
    const int64_t k0 = r * kColRows, k1 = k0 + kColRows < J.kc ? k0 + kColRows : J.kc;
    int m = 2 * kNoExp;
    double sum = 0.0;
#pragma unroll 16
    for (int64_t k = k0; k < k1; ++k) {
      const int e = __ldg(J.rexp + k);
      const double v = (double)__ldg(X + k * n);
      if (e != kPSkip && v != 0.0) {
        const int hi = __double2hiint(v) & 0x7fffffff;
        m = max(m, max((hi >> 20) - 1023, -1023) + (side ? e : -e));
        const double w = v * pow2(side ? e : -e);
        sum = fma(w, w, sum);
      }
    }
    if (J.kc <= kColRows) {
      (side ? J.cexpB : J.cexpA)[c] = norm_exp(sum, m, J.kc);
    } else {
      const size_t at = (size_t)r * (J.n_a + J.n_b) + (side ? J.n_a : 0) + c;
      J.csum[at] = sum;
      J.cmax[at] = m;
    }
  }
}
__global__ void __launch_bounds__(128) k_prod_cexp(const ProdJob* __restrict__ jobs) {
  const ProdJob& J = jobs[blockIdx.y];
  const int64_t n = J.n_a + J.n_b, c = (int64_t)blockIdx.x * 128 + threadIdx.x;
  if (c >= n || J.kc <= kColRows) return;
  const int nb = (int)((J.kc + kColRows - 1) / kColRows);
  double sum = 0.0;
  int m = 2 * kNoExp;
#pragma unroll 16
  for (int r = 0; r < nb; ++r) {
    sum += J.csum[(size_t)r * n + c];
    m = max(m, J.cmax[(size_t)r * n + c]);
  }
  (c < J.n_a ? J.cexpA[c] : J.cexpB[c - J.n_a]) = norm_exp(sum, m, J.kc);
}

// ------------------------------------------------------------ residue planes
// Planes in the order and layout that the tensor cores read: [modulus][tile of
// 128 columns][32 inner indices][16 inner indices][column][byte], i.e.
// no-swizzle K-major core matrices of 8 columns x 16 bytes.  Thread = column:
// it reads 16 rows (coalesced over the columns) and writes one 16-byte
// core-matrix row per modulus.  Columns and inner indices are padded with
// zeros to whole tiles and stages.  The residues of A carry the factor
// (M / m_i)^-1 mod m_i of the reconstruction.
//
// X + 2^T is taken byte by byte: the dot product of its bytes with the balanced
// residues of 256^i (two dp4a; one for FP32) is an integer below 2^19 with the
// right residue, and starting the sum at the bits of 1.5 2^23 leaves it in the
// mantissa of a float.  With q = round(v / m) by the same trick, v - q m is the
// balanced residue (m odd: v / m stays 1 / 2m = 0.0025 away from a tie, against
// errors of 1e-4; m = 256: both ends of a tie are the byte 0x80), and its low
// byte is that of the two bit patterns' difference, because 1.5 2^23's low byte
// is zero.  Five instructions a residue, bound by issue; with 20-bit parts and
// an exact division by multiplication it took eight (4096 x 4096 FP64, both
// sides: 0.28 -> 0.18 ms).
constexpr int balanced(int r, int m) {  // the residue in [-m / 2, m / 2)
  return r % m >= (m + 1) / 2 ? r % m - m : r % m;
}
// balanced residues of f 256^(4 h + i), i < 4, one a byte
constexpr uint32_t byte_weights(int f, int h, int m) {
  uint32_t w = 0;
  for (int i = 0; i < 4; ++i) w |= (uint32_t)(uint8_t)balanced(powmod2(8 * (4 * h + i), m) * f % m, m) << (8 * i);
  return w;
}
__device__ __forceinline__ uint32_t dp4a_us(uint32_t bytes, uint32_t weights, uint32_t sum) {
  uint32_t d;
  asm("dp4a.u32.s32 %0, %1, %2, %3;" : "=r"(d) : "r"(bytes), "r"(weights), "r"(sum));
  return d;
}
template <typename Real, int SIDE, int I>
__device__ __forceinline__ uint32_t residue(uint32_t lo, uint32_t hi) {
  constexpr int N = Fix<Real>::N, T = Fix<Real>::T, m = modulus(I);
  constexpr int f = SIDE == 0 ? crt_inv(I, N) : 1;
  constexpr uint32_t kBits = 0x4B400000u;  // 1.5 2^23
  constexpr uint32_t start = kBits + (uint32_t)balanced(m - powmod2(T, m) * f % m, m);
  uint32_t v = dp4a_us(lo, byte_weights(f, 0, m), start);
  if (sizeof(Real) == 8) v = dp4a_us(hi, byte_weights(f, 1, m), v);
  const float t = fmaf(__uint_as_float(v) - 12582912.f, 1.f / m, 12582912.f);
  return v - __float_as_uint(t) * (uint32_t)m;  // (the low byte counts)
}
template <typename Real, int SIDE, int I>
__device__ __forceinline__ void plane_store(const uint32_t (&lo)[16], const uint32_t (&hi)[16], uint8_t* dst, size_t plane) {
  constexpr int N = Fix<Real>::N;
  uint32_t w[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint32_t r[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) r[u] = residue<Real, SIDE, I>(lo[4 * q + u], hi[4 * q + u]);
    w[q] = __byte_perm(__byte_perm(r[0], r[1], 0x0040), __byte_perm(r[2], r[3], 0x0040), 0x5410);
  }
  *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
  if constexpr (I + 1 < N) plane_store<Real, SIDE, I + 1>(lo, hi, dst + plane, plane);
}

template <typename Real, int SIDE>
__global__ void __launch_bounds__(128) k_prod_slice(const ProdJob* __restrict__ jobs) {
  constexpr int T = Fix<Real>::T;
  const ProdJob& J = jobs[blockIdx.z];
  const int64_t n = SIDE ? J.n_b : J.n_a;
  const int tiles = 2 * (SIDE ? J.tiles_b : J.tiles_a);
  const int tile = blockIdx.x;
  if (tile >= tiles) return;
  const int KS = prod_ksteps(J.kc);
  const size_t plane = (size_t)tiles * KS * kProdSlab;
  const int64_t c = (int64_t)tile * kProdTile + threadIdx.x;
  const Real* X = reinterpret_cast<const Real*>(SIDE ? J.B : J.A) + c;
  uint8_t* out = (SIDE ? J.slB : J.slA) + (size_t)tile * KS * kProdSlab + threadIdx.x * 16;
  const int E = c < n ? (SIDE ? J.cexpB : J.cexpA)[c] : kNoExp;
  const bool live = E > kNoExp;
  const double g = live ? pow2(T - max(E, kMinExp)) : 0.0;
  for (int kh = blockIdx.y; kh < 2 * KS; kh += gridDim.y) {  // 16 inner indices
    const int64_t k0 = (int64_t)kh * 16;
    Real x[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) x[u] = live && k0 + u < J.kc ? __ldg(X + (k0 + u) * n) : (Real)0;
    uint32_t lo[16], hi[16];
#pragma unroll
    for (int u = 0; u < 16; ++u) {
      const int e = k0 + u < J.kc ? __ldg(J.rexp + k0 + u) : kPSkip;
      const double y = e == kPSkip ? 0.0 : (double)x[u] * pow2(SIDE ? e : -e) * g;
      const unsigned long long w = (unsigned long long)__double2ll_rn(y) + (1ull << T);
      lo[u] = (uint32_t)w;
      hi[u] = (uint32_t)(w >> 32);
    }
    plane_store<Real, SIDE, 0>(lo, hi, out + (size_t)(kh >> 1) * kProdSlab + (kh & 1) * (kProdSlab / 2), plane);
  }
}

// ------------------------------------------------------- tcgen05 primitives
// arrives on the barrier at the same offset in CTA 0 of the pair
__device__ __forceinline__ void bar_arrive_lead(uint64_t* bar) {
  asm volatile(
      "{\n\t.reg .b32 ra;\n\t"
      "mapa.shared::cluster.u32 ra, %0, 0;\n\t"
      "mbarrier.arrive.shared::cluster.b64 _, [ra];\n\t}\n" ::"r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void mma_i8(uint32_t d, uint64_t ad, uint64_t bd, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d),
      "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
}
// arrives on the barrier at this offset in both CTAs once the MMAs issued so
// far are done
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
          smem_u32(bar)),
      "h"((uint16_t)3)
      : "memory");
}
// every thread of both CTAs, whole warps at a time
__device__ __forceinline__ void pair_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, int (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
      "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int u = 0; u < 32; ++u) asm volatile("" : "+r"(r[u]));  // not used before the wait
}

// shared-memory matrix descriptor: start address >> 4, leading byte offset
// 2048 (between the two 16-byte K halves), stride byte offset 128 (between
// 8-row groups), descriptor version 1, no swizzle
__device__ __forceinline__ uint64_t plane_desc(uint32_t saddr) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)(2048 >> 4) << 16) | ((uint64_t)(128 >> 4) << 32) |
         (1ull << 46);
}
// instruction descriptor, kind::i8: D int32 (bits 4-5 = 2), A and B signed
// (bits 7-9 and 10-12 = 1), both K-major, N = 256 (>> 3 at bit 17), M = 256
// (>> 4 at bit 24)
constexpr uint32_t kIdescI8 = (2u << 4) | (1u << 7) | (1u << 10) | ((256u >> 3) << 17) | ((256u >> 4) << 24);

// ------------------------------------------------------------- the product
// One work item = (tile of 256 columns of B x 256 columns of A, modulus),
// computed by a pair of CTAs with tcgen05.mma.cta_group::2 (M = 256: CTA r
// holds the rows 128 r .. 128 r + 127 of the tile, columns of B, in its 128
// TMEM lanes; N = 256: each CTA stages half of the columns of A).  Per 32
// inner indices and CTA that is 8 KB of operands for 128 cycles of tensor
// core, half of what single-CTA tiles of 128 x 256 would stage.  TMEM holds
// two accumulators of 256 columns, so an item's epilogue (int32 -> residue
// byte) runs behind the next item's MMAs.  Roles in each CTA: warps 0-7 the
// epilogue, warp 8 the bulk copies of this CTA's half of both operands, warp
// 9 the MMAs (CTA 0) or the relay (CTA 1: passes "my half of the stage has
// landed" on to CTA 0).
constexpr int kStageK = 4;                               // 32-index steps per stage
constexpr int kStageBytes = 2 * kStageK * kProdSlab;     // 32 KB: both operands of this CTA
constexpr int kStages = 6;
constexpr int kProdThreads = 320;
constexpr int kProdSmem = kStages * kStageBytes + 128;

struct ProdItem {
  int job, mod, mt, nt;
};
// item index -> (job, modulus, tile of B, tile of A); indices ascend, `job` is
// kept.  The tiles of one modulus come in groups of 8 tiles of A, so that the
// pairs in flight share their planes through L2.
__device__ __forceinline__ ProdItem prod_item(const ProdJob* __restrict__ jobs, int64_t idx, int job, int nmod) {
  while (idx >= jobs[job].item_end) ++job;
  const int tm = jobs[job].tiles_b, tn = jobs[job].tiles_p;
  const int64_t tiles = (int64_t)tm * tn;
  const int64_t e = idx - (jobs[job].item_end - tiles * nmod);
  ProdItem p;
  p.job = job;
  p.mod = (int)(e / tiles);
  const int64_t w = e - p.mod * tiles;
  const int gh = 8;
  const int grp = (int)(w / ((int64_t)gh * tm));
  const int h = min(gh, tn - grp * gh);
  const int v = (int)(w - (int64_t)grp * gh * tm);
  p.mt = v / h;
  p.nt = grp * gh + v % h;
  return p;
}

__device__ __forceinline__ int prod_modulus(int i) {
  constexpr uint64_t lo = 0xE9EFF1F7FBFDFF00ull, hi = 0x00C5C7D3D9DFE3E5ull;  // modulus(i) mod 256, a byte each
  const int b = (int)(((i < 8 ? lo : hi) >> (8 * (i & 7))) & 0xff);
  return b ? b : 256;
}

// residues of the int32 accumulators (this warp's 32 lanes x 128 columns)
__device__ __forceinline__ void prod_epilogue(const ProdJob& J, const ProdItem& it, int rank, uint32_t tbase, int warp,
                                              int lane, int m, uint32_t magic) {
  const int64_t ldr = (int64_t)J.tiles_b * 256;
  const int64_t j = (int64_t)it.mt * 256 + 128 * rank + 32 * (warp & 3) + lane;
  uint32_t* out = J.res + ((int64_t)it.mod * J.tiles_p + it.nt) * 64 * ldr + j;
  const int up = (0x20000000 + m - 1) / m * m;  // a multiple of m above every |accumulator|
#pragma unroll 1
  for (int c0 = (warp >> 2) * 128; c0 < (warp >> 2) * 128 + 128; c0 += 32) {
    int a[32];
    tmem_ld32(tbase + ((uint32_t)(32 * (warp & 3)) << 16) + c0, a);
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      uint32_t r[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const uint32_t v = (uint32_t)(a[4 * q + u] + up);
        r[u] = v - (__umulhi(v, magic) >> 7) * (uint32_t)m;
      }
      out[(int64_t)(c0 / 4 + q) * ldr] = (r[0] | r[1] << 8) | (r[2] | r[3] << 8) << 16;
    }
  }
}

template <int NMOD>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(kProdThreads, 1)
    k_prod_gemm(const ProdJob* __restrict__ jobs, int64_t items, const ProdWaits waits) {
  extern __shared__ __align__(1024) unsigned char psm[];
  unsigned char* ring = reinterpret_cast<unsigned char*>(((uintptr_t)psm + 127) & ~(uintptr_t)127);
  __shared__ uint64_t full[kStages], empty[kStages], accfull[2], accempty[2], drain;
  __shared__ uint32_t tmem_base;
  __shared__ int s_wait[2];
  __shared__ unsigned s_issued;  // stages whose copies were issued
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = blockIdx.x & 1;
  const int64_t pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
  if (tid == 0) {
    // CTA 0's stage is full when both CTAs' halves are there
    for (int s = 0; s < kStages; ++s) { bar_init(&full[s], (rank == 0 ? 2 : 1) + waits.extra); bar_init(&empty[s], 1); }
    for (int s = 0; s < 2; ++s) { bar_init(&accfull[s], 1); bar_init(&accempty[s], 16); }
    bar_init(&drain, 1);
    s_wait[0] = 0;
    s_wait[1] = waits.limit_us;
    s_issued = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  pair_sync();  // both CTAs run
  if (warp == 0)
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                 "r"(512u)
                 : "memory");
  fence_before();
  pair_sync();
  fence_after();
  const uint32_t tbase = tmem_base;
  volatile int* wait = s_wait;

  if (warp == 8) {
    if (lane == 0) {
      unsigned it = 0;
      int job = 0;
      bool ok = true;
      for (int64_t idx = pair; idx < items && ok; idx += pairs) {
        const ProdItem p = prod_item(jobs, idx, job, NMOD);
        job = p.job;
        const ProdJob& J = jobs[job];
        const int KS = prod_ksteps(J.kc);
        const uint8_t* gm = J.slB + ((size_t)p.mod * 2 * J.tiles_b + 2 * p.mt + rank) * KS * kProdSlab;
        const uint8_t* gn = J.slA + ((size_t)p.mod * 2 * J.tiles_a + 2 * (J.tile0 + p.nt) + rank) * KS * kProdSlab;
        for (int ks = 0; ks < KS; ks += kStageK, ++it) {
          const unsigned st = it % kStages;
          if (!bar_wait(&empty[st], ((it / kStages) & 1u) ^ 1u, wait)) { ok = false; break; }
          unsigned char* dst = ring + st * kStageBytes;
          bar_expect(&full[st], kStageBytes);
          bulk_load(dst, gm + (size_t)ks * kProdSlab, kStageBytes / 2, &full[st]);
          bulk_load(dst + kStageBytes / 2, gn + (size_t)ks * kProdSlab, kStageBytes / 2, &full[st]);
        }
      }
      s_issued = it;
      // the last arrivals on this CTA's empty barriers come from the other CTA's MMAs
      for (unsigned z = it > kStages ? it - kStages : 0; ok && z < it; ++z)
        ok = bar_wait(&empty[z % kStages], (z / kStages) & 1u, wait);
    }
  } else if (warp == 9) {
    if (lane == 0) {
      unsigned it = 0, acc = 0;
      int job = 0;
      bool ok = true;
      for (int64_t idx = pair; idx < items && ok; idx += pairs, ++acc) {
        job = prod_item(jobs, idx, job, NMOD).job;
        const int KS = prod_ksteps(jobs[job].kc);
        const unsigned ab = acc & 1u;
        if (rank == 0) {
          if (!bar_wait(&accempty[ab], ((acc >> 1) & 1u) ^ 1u, wait)) break;
          fence_after();
        }
        for (int ks = 0; ks < KS; ks += kStageK, ++it) {
          const unsigned st = it % kStages;
          if (!bar_wait(&full[st], (it / kStages) & 1u, wait)) { ok = false; break; }
          if (rank == 1) {
            bar_arrive_lead(&full[st]);
            continue;
          }
          fence_after();
          const uint32_t sa = smem_u32(ring + st * kStageBytes);
          const uint64_t dm = plane_desc(sa), dn = plane_desc(sa + kStageBytes / 2);
#pragma unroll
          for (int q = 0; q < kStageK; ++q)
            mma_i8(tbase + ab * 256u, dm + (uint64_t)(q * (kProdSlab >> 4)), dn + (uint64_t)(q * (kProdSlab >> 4)),
                   kIdescI8, ks == 0 && q == 0 ? 0u : 1u);
          mma_commit(&empty[st]);
        }
        if (ok && rank == 0) mma_commit(&accfull[ab]);
      }
    }
  } else {
    unsigned acc = 0;
    int job = 0;
    for (int64_t idx = pair; idx < items; idx += pairs, ++acc) {
      const ProdItem p = prod_item(jobs, idx, job, NMOD);
      job = p.job;
      const unsigned ab = acc & 1u;
      int got = lane == 0 ? (bar_wait(&accfull[ab], (acc >> 1) & 1u, wait) ? 1 : 0) : 0;
      got = __shfl_sync(0xffffffffu, got, 0);
      if (!got) break;
      bar_test(&accfull[ab], (acc >> 1) & 1u);  // every lane observes the phase before it reads tensor memory
      fence_after();
      const int m = prod_modulus(p.mod);
      prod_epilogue(jobs[job], p, rank, tbase + ab * 256u, warp, lane, m, mod_magic(m));
      fence_before();
      __syncwarp();
      if (lane == 0) bar_arrive_lead(&accempty[ab]);
    }
  }
  __syncwarp();
  __syncthreads();
  if (s_wait[0]) {  // a wait ran out: report, and let this CTA's MMAs and copies end before it does
    if (rank == 0 && warp == 9 && lane == 0) {
      mma_commit(&drain);
      bar_drain(&drain, 0, wait);
    }
    if (tid == 0) {
      *waits.flag = 1;
      __threadfence_system();
      for (unsigned b = s_issued > kStages ? s_issued - kStages : 0; b < s_issued; ++b)
        bar_drain(&full[b % kStages], (b / kStages) & 1u, wait);
      int job = 0;
      for (int64_t idx = pair; idx < items; idx += pairs) {
        job = prod_item(jobs, idx, job, NMOD).job;
        *jobs[job].flag = 1;  // the sketch becomes NaN
      }
    }
    __syncthreads();
  }
  // Allocating and freeing pairs of CTAs' tensor memory are operations of one
  // warp of each CTA together, and CTA 0's MMAs read CTA 1's shared memory: the
  // pair starts them together, and neither CTA leaves before both are through.
  // (Left to end on their own, CTAs that shared their SMs with other streams'
  // kernels did now and then not end at all.)
  fence_before();
  pair_sync();
  fence_after();
  if (warp == 0) {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(512u) : "memory");
  }
  pair_sync();
}

// ------------------------------------------------------------ reconstruction
// C[i][j] (+)= the integer with the N residues, in (-M / 2, M / 2), times
// 2^(E_i + E_j - 2T).  S = sum r_i (M / m_i) in 32-bit limbs, minus t M with t =
// round(S / M) from S's top limb (in FP32, off by less than 2^-11; |entry| <=
// 2^2T < 0.34 M keeps S / M 0.16 away from a tie), modulo 2^128 (2^64).  The
// top limb of 15 moduli needs 32 bits only.  Thread = column j, four rows i at a
// time.  Bound by the multiply-adds of the limbs (4096 x 4096, 15 moduli: 168
// us with a fixed-point sum for t and 64-bit top limbs, 153 now).
template <int N, int I>
__device__ __forceinline__ void crt_terms(const uint32_t (&w)[16], uint32_t pick, unsigned long long (&s)[3], uint32_t& top) {
  constexpr U128 P = mod_product(N, I);
  const uint32_t r = __byte_perm(w[I], 0, pick);
  s[0] += (unsigned long long)r * (uint32_t)P.lo;
  s[1] += (unsigned long long)r * (uint32_t)(P.lo >> 32);
  if (N > 8) {
    s[2] += (unsigned long long)r * (uint32_t)P.hi;
    top += r * (uint32_t)(P.hi >> 32);
  }
  if constexpr (I + 1 < N) crt_terms<N, I + 1>(w, pick, s, top);
}
constexpr double two_to(int e) { return e <= 0 ? 1.0 : 2.0 * two_to(e - 1); }
template <typename Real>
__global__ void __launch_bounds__(256) k_prod_crt(const ProdJob* __restrict__ jobs) {
  constexpr int N = Fix<Real>::N, T = Fix<Real>::T;
  constexpr U128 M = mod_product(N, -1);
  const ProdJob& J = jobs[blockIdx.z];
  const int64_t ldr = (int64_t)J.tiles_b * 256, quads = (int64_t)J.tiles_p * 64;
  const int64_t j = (int64_t)blockIdx.x * 256 + threadIdx.x;
  if (j >= J.n_b) return;
  const int eB = max(__ldg(J.cexpB + j), kMinExp) - 2 * T;
  for (int64_t r = blockIdx.y; r < quads; r += gridDim.y) {
    const int64_t i = (int64_t)J.tile0 * 256 + r * 4;
    if (i >= J.n_a) break;
    uint32_t w[16];
#pragma unroll
    for (int q = 0; q < N; ++q) w[q] = __ldcs(J.res + ((int64_t)q * quads + r) * ldr + j);
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (i + u >= J.n_a) break;
      unsigned long long s[3] = {0, 0, 0};
      uint32_t top = 0;
      crt_terms<N, 0>(w, 0x4440u + u, s, top);
      double v;
      if (N > 8) {
        constexpr float inv = (float)(two_to(96) / ((double)M.hi * two_to(64)));
        const uint32_t t = (uint32_t)__float2int_rn((float)(top + (uint32_t)(s[2] >> 32)) * inv);
        unsigned __int128 x = (unsigned __int128)s[0] + ((unsigned __int128)s[1] << 32) + ((unsigned __int128)s[2] << 64) +
                              ((unsigned __int128)top << 96);
        x -= (((unsigned __int128)M.hi << 64) | M.lo) * t;
        const bool neg = (__int128)x < 0;
        if (neg) x = -x;
        v = fma((double)(unsigned long long)(x >> 64), 18446744073709551616.0, (double)(unsigned long long)x);
        if (neg) v = -v;
      } else {
        constexpr float inv = (float)(two_to(36) / (double)M.lo);
        const uint32_t t = (uint32_t)__float2int_rn((float)(uint32_t)(s[1] >> 4) * inv);
        v = (double)(long long)(s[0] + (s[1] << 32) - M.lo * t);
      }
      const int e = min(max(__ldg(J.cexpA + i + u), kMinExp) + eB, 2046), h = e >> 1;
      v = v * pow2(h) * pow2(e - h);
      double* C = J.C + (i + u) * J.ldc + j;
      *C = J.accumulate ? *C + v : v;
    }
  }
}

}  // namespace

// Flags come from pages of host-mapped memory that stay for the process.
namespace {
std::mutex g_flag_mu;
std::vector<std::pair<int*, int*>> g_flags;  // free ones: host and device address
}  // namespace

WaitFlag::WaitFlag() {
  constexpr int kPage = 256;
  std::lock_guard<std::mutex> g(g_flag_mu);
  if (g_flags.empty()) {
    int *host = nullptr, *dev = nullptr;
    CMM_CUDA(cudaHostAlloc(reinterpret_cast<void**>(&host), kPage * sizeof(int), cudaHostAllocMapped | cudaHostAllocPortable));
    CMM_CUDA(cudaHostGetDevicePointer(reinterpret_cast<void**>(&dev), host, 0));
    for (int i = 0; i < kPage; ++i) g_flags.emplace_back(host + i, dev + i);
  }
  host_ = g_flags.back().first;
  dev_ = g_flags.back().second;
  g_flags.pop_back();
  __atomic_store_n(host_, 0, __ATOMIC_RELEASE);
}
WaitFlag::~WaitFlag() {
  std::lock_guard<std::mutex> g(g_flag_mu);
  g_flags.emplace_back(host_, dev_);
}
bool WaitFlag::take() { return __atomic_exchange_n(host_, 0, __ATOMIC_ACQ_REL) != 0; }

// (never given back: kernels of an ended thread may still run)
WaitFlag& thread_wait_flag() {
  static thread_local WaitFlag* f = nullptr;
  if (!f) f = new WaitFlag();
  return *f;
}

ProdWaits product_waits(int* flag, const char* kernel) {
  ProdWaits w{flag, kWaitUs, 0};
  const char* e = getenv("CMM_TEST_PRODUCT_WAIT");  // test hook: waits that cannot complete
  if (e && !strcmp(e, kernel)) {
    w.limit_us = 1000;
    w.extra = 1;
  }
  return w;
}

namespace {

template <int NMOD>
void launch_gemm(const ProdJob* dJobs, int64_t items, int* flag, cudaStream_t s) {
  CMM_CUDA(cudaFuncSetAttribute(k_prod_gemm<NMOD>, cudaFuncAttributeMaxDynamicSharedMemorySize, kProdSmem));
  const int grid = 2 * (int)std::min<int64_t>(items, num_sms() / 2);
  count_launch();
  k_prod_gemm<NMOD><<<grid, kProdThreads, kProdSmem, s>>>(dJobs, items, product_waits(flag, "product"));
  CMM_CUDA(cudaGetLastError());
}

}  // namespace

// CTAs along a dimension that kernels stride over, of `want` useful ones, next to
// `others` in the other dimensions: the grid is sized for the largest job, so
// among many jobs most CTAs find nothing to do, and 250,000 of them take 0.1 ms.
static unsigned spread(int64_t want, int64_t others) {
  return (unsigned)std::max<int64_t>(1, std::min(want, std::max<int64_t>(8, 32768 / others)));
}

void launch_product_planes(const ProdJob* hJobs, const ProdJob* dJobs, int count, bool f32, cudaStream_t s) {
  if (count <= 0) return;
  int64_t kc = 0, n = 0, nn = 0;
  int ta = 0, tb = 0;
  for (int i = 0; i < count; ++i) {
    const ProdJob& J = hJobs[i];
    kc = std::max(kc, J.kc);
    n = std::max(n, std::max(J.n_a, J.n_b));
    nn = std::max(nn, J.n_a + J.n_b);
    ta = std::max(ta, J.tiles_a);
    tb = std::max(tb, J.tiles_b);
  }
  {
    ProfScope prof("scale", s);
    const dim3 gr(spread(kc, count), (unsigned)count);
    const unsigned cx = (unsigned)((n + 127) / 128);
    const dim3 gc(cx, spread((kc + kColRows - 1) / kColRows, 2 * (int64_t)cx * count), (unsigned)(2 * count));
    count_launch(kc > kColRows ? 3 : 2);
    if (f32) {
      k_prod_rows<float><<<gr, kRowThreads, 0, s>>>(dJobs);
      k_prod_cols<float><<<gc, 128, 0, s>>>(dJobs);
    } else {
      k_prod_rows<double><<<gr, kRowThreads, 0, s>>>(dJobs);
      k_prod_cols<double><<<gc, 128, 0, s>>>(dJobs);
    }
    if (kc > kColRows) k_prod_cexp<<<dim3((unsigned)((nn + 127) / 128), (unsigned)count), 128, 0, s>>>(dJobs);
    CMM_CUDA(cudaGetLastError());
  }
  ProfScope prof("materialize", s);
  count_launch(2);
  const unsigned ky = spread(2 * prod_ksteps(kc), 2 * (int64_t)std::max(ta, tb) * count);
  const dim3 ga((unsigned)(2 * ta), ky, (unsigned)count), gb((unsigned)(2 * tb), ky, (unsigned)count);
  if (f32) {
    k_prod_slice<float, 0><<<ga, 128, 0, s>>>(dJobs);
    k_prod_slice<float, 1><<<gb, 128, 0, s>>>(dJobs);
  } else {
    k_prod_slice<double, 0><<<ga, 128, 0, s>>>(dJobs);
    k_prod_slice<double, 1><<<gb, 128, 0, s>>>(dJobs);
  }
  CMM_CUDA(cudaGetLastError());
}

void launch_product_gemm(const ProdJob* hJobs, const ProdJob* dJobs, int count, bool f32, int* flag, cudaStream_t s) {
  if (count <= 0) return;
  ProfScope prof("sketch", s);
  if (f32) launch_gemm<Fix<float>::N>(dJobs, hJobs[count - 1].item_end, flag, s);
  else launch_gemm<Fix<double>::N>(dJobs, hJobs[count - 1].item_end, flag, s);
  int64_t n_b = 0, rows = 0;
  for (int i = 0; i < count; ++i) {
    n_b = std::max(n_b, hJobs[i].n_b);
    rows = std::max<int64_t>(rows, (int64_t)hJobs[i].tiles_p * 64);
  }
  count_launch();
  const unsigned gx = (unsigned)((n_b + 255) / 256);
  const int64_t gy = std::max<int64_t>(1, std::min<int64_t>(rows, 32768 / ((int64_t)gx * count)));
  const dim3 g(gx, (unsigned)gy, (unsigned)count);
  if (f32) k_prod_crt<float><<<g, 256, 0, s>>>(dJobs);
  else k_prod_crt<double><<<g, 256, 0, s>>>(dJobs);
  CMM_CUDA(cudaGetLastError());
}

// ------------------------------------------------------------------- dispatch
// Estimates in microseconds, fitted to single calls on B200 (random shapes, n 1 to
// 20,000, b 2^9 to 2^23, both routes timed: the product within 10 % rms, the
// transforms within 5 to 20).  Of 640 shapes 6 take the route that is slower by
// more than a tenth; with the formula before, which counted the entries of C
// only, 61 did (8953 x 32 x 6096, b = 2^21, d = 5: 13.7 ms, transforms 3.0).
namespace {

// Additions: a warp's step over one row and window costs the same with one entry
// or twenty, so sparse rows (few columns, many buckets) pay per step.
struct AddCost {
  double spread;   // work that any number of SMs share
  double cta, row; // of a CTA: its rows, us for one
  double load;     // CTAs per place on the device
};
AddCost additions_cost(const ProdJob& J, int sms) {
  const double db = (double)J.d * (double)(1u << J.log2b), wins = (double)((1u << J.log2b) >> J.logW);
  const double cols = (double)std::min<int64_t>(J.n_b, 4096);
  AddCost c{(double)J.G * db * 8.0 * 1.5 / 6.5e6, 0, 0, 0};  // partial sketches, written and read
  if (J.form == kAddGather) {
    c.spread += 7e-6 * db + (double)J.n_a * J.d * (wins * 1.09e-4 + (double)J.n_b * 2.0e-6);
    return c;
  }
  c.cta = (double)J.n_a / J.G * J.blocks;
  c.row = J.form == kAddLane ? 0.3 + 2.1e-4 * cols : J.per_sm == 1 ? 0.43 + 1.5e-3 * cols / wins : 0.5 + 3.6e-3 * cols / wins;
  c.load = J.d * (J.form == kAddLane ? 1.0 : std::ceil(wins / 16.0)) * (double)J.G / ((double)J.per_sm * sms);
  return c;
}
double product_work(const ProdJob& J, bool f32, int64_t n_inner, double per_plane, double per_entry) {
  const double na = (double)J.n_a, nb = (double)J.n_b, k = (double)n_inner;
  return 65536.0 * J.tiles_a * J.tiles_b * std::ceil(k / 128.0) * 128.0 * 2.0 * prod_moduli(f32) / 3.0e9 +
         k * (na + nb) * per_plane + na * nb * per_entry;
}
double product_us(const ProdJob& J, bool f32, int64_t n_inner, int sms) {
  const AddCost c = additions_cost(J, sms);
  return 85.0 + product_work(J, f32, n_inner, 9.3e-6, f32 ? 1e-5 : 2e-5) + c.spread + std::max(1.0, c.load) * c.cta * c.row;
}

// Among other jobs, fitted to plans of 1 to 32 equal products (240 of them, 9 % rms;
// transforms 20): the work of all, a chain of launches, and the longest CTA of the
// additions, however few there are.
struct JobCost {
  double work, load, chain;
};
JobCost job_cost(const ProdJob& J, bool f32, int sms) {
  const AddCost c = additions_cost(J, sms);
  const double wins = (double)((1u << J.log2b) >> J.logW), cols = (double)std::min<int64_t>(J.n_b, 4096);
  const double row = J.form == kAddLane ? 0.155 + 9.6e-5 * cols : 0.155 + 4.2e-3 * cols / wins + 7e-3 * std::min(wins, 16.0);
  return {1.61 * (product_work(J, f32, J.kc, f32 ? 5e-6 : 8e-6, f32 ? 4e-6 : 9e-6) + c.spread), 1.07 * c.load * c.cta * c.row,
          c.cta * row};
}
// the batch transform kernel: fixed, per 4096 buckets, per d k b log b, per d k (n_a +
// n_b), per d b log b; FFT FP64, FP32, FWHT FP64, FP32
struct BatchCost {
  double fixed, buckets, work, rows, inverse;
};
constexpr BatchCost kBatchCost[4] = {{75, 17.3, 9.6e-7, 2.6e-5, 1.45e-6}, {58, 14.2, 5.4e-7, 1.27e-5, 1.3e-7},
                                     {86, 2.4, 6.2e-7, 1.7e-5, 0}, {63, 1.3, 4.05e-7, 1.24e-5, 0}};
const BatchCost& batch_cost(int variant, bool f32) { return kBatchCost[(variant == kVariantFFT ? 0 : 2) + (f32 ? 1 : 0)]; }
double batch_transforms_us(const ProdJob& J, bool f32) {
  const BatchCost& c = batch_cost(J.variant, f32);
  const double blog = (double)(1u << J.log2b) * J.log2b;
  return J.d * ((double)J.kc * (c.work * blog + c.rows * (double)(J.n_a + J.n_b)) + c.inverse * blog);
}

// The transform kernels that would run: launches and plan, the inverse per d b
// log b, the work per d k b log b (FP64, FP32) and per d k (n_a + n_b).
struct TransformCost {
  double fixed, inverse, work, work32, rows;
};
double transforms_us(int variant, bool f32, int d, int b, double k, double n) {
  const bool fft = variant == kVariantFFT;
  double log2b = 0;
  while ((1 << (int)log2b) < b) ++log2b;
  const double blog = (double)b * log2b;
  static const TransformCost kSmall[2] = {{55, 0, 2.6e-6, 2.4e-6, 4.5e-6}, {52, 0, 2.2e-6, 2.1e-6, 7.5e-6}};
  static const TransformCost kSlab[2] = {{135, 7e-6, 7.2e-7, 4.2e-7, 8e-6}, {138, 2e-6, 3.6e-7, 4.4e-7, 6e-6}};
  static const TransformCost kGroup[2] = {{135, 7.6e-6, 8e-7, 4.2e-7, 8e-6}, {132, 4e-6, 4.5e-7, 3.1e-7, 1.3e-5}};
  static const TransformCost kSlabBig[2] = {{140, 5.1e-6, 4.5e-7, 2.7e-7, 7e-4}, {150, 1.4e-6, 2.3e-7, 2.9e-7, 3.3e-4}};
  static const TransformCost kBig[2] = {{170, 4.7e-6, 1.7e-6, 1.7e-6, 7e-3}, {130, 1.3e-6, 8.5e-7, 8.2e-7, 2.5e-3}};
  const bool mixed = f32 && sketch_mixed_applicable(variant, b), slab = mixed || sketch_v1_applicable(variant, b, 0, 0);
  const bool small_b = !slab && b <= 65536;
  const TransformCost& c = (sketch_cluster_applicable(variant, f32, b) ? kGroup
                            : slab ? (b < (1 << 20) ? kSlab : kSlabBig)
                            : small_b ? kSmall : kBig)[fft ? 0 : 1];
  return c.fixed + (small_b && fft ? 0.005 * b : 0.0) + c.inverse * d * blog +
         d * k * ((f32 && (mixed || !slab) ? c.work32 : c.work) * blog + c.rows * n);
}

}  // namespace

bool product_faster(int variant, bool f32, int d, int b, int64_t n_a, int64_t n_inner, int64_t n_b) {
  ProdJob J{};
  product_geometry(J, variant, d, b, n_a, n_b, std::min(n_inner, kProdMaxK), true, num_sms());
  return product_us(J, f32, n_inner, num_sms()) <
         transforms_us(variant, f32, d, b, (double)n_inner, (double)(n_a + n_b));
}

bool product_among_others(int variant, bool f32, int d, int b, int64_t n_a, int64_t n_inner, int64_t n_b) {
  const int choice = sketch_kernel_choice();
  if (choice == 1 || choice == 2 || n_inner > kProdMaxK || !product_supported(b, n_a, n_inner, n_b)) return false;
  if (choice == 3) return true;
  ProdJob J{};
  product_geometry(J, variant, d, b, n_a, n_b, n_inner, false, num_sms());
  const JobCost c = job_cost(J, f32, num_sms());
  return 5.0 + c.work + c.load < batch_transforms_us(J, f32);
}

bool products_pay(const ProdJob* jobs, int count, bool f32, bool others) {
  if (sketch_kernel_choice() == 3) return true;
  double work = 57.0, load = 0.0, chain = 0.0, transforms = 0.0, fixed = 0.0;
  for (int i = 0; i < count; ++i) {
    const JobCost c = job_cost(jobs[i], f32, num_sms());
    work += c.work;
    load += c.load;
    chain = std::max(chain, c.chain);
    transforms += batch_transforms_us(jobs[i], f32);
    const BatchCost& b = batch_cost(jobs[i].variant, f32);
    fixed = std::max(fixed, b.fixed + b.buckets * (double)(1u << jobs[i].log2b) / 4096.0);
  }
  return work + std::sqrt(std::hypot(load * load, chain * chain)) < transforms + (others ? 0.0 : fixed);
}

}  // namespace cmm
