// Batched natural-order Walsh-Hadamard transform of FP32 rows, with a
// Hadamard-128 stage on the 5th-generation tensor cores (tcgen05.mma: BF16
// operands from shared memory, FP32 accumulators in tensor memory), beside
// the same transform with every stage on CUDA cores.
//
// y[r] = H_L x[r] for each row r, L = 2^LOGL (11 <= LOGL <= 13), H_L the
// unnormalised Sylvester matrix H[i][j] = (-1)^popc(i & j): the forward
// transform of the reference's fwht_transformer (transform.hpp:94-144, FXT
// walsh_wak in natural order; golden values in tests.cpp:621-671).
//
// Rows are contiguous, so both forms work on tiles of 8192 elements (8192 / L
// rows; one row where there are few), seen as 64 blocks of 128: H_L = H_{L/128}
// (x) H_128, whose factors commute.
//   * Index bits 7 and up: thread c holds element c of all blocks in
//     registers, as they come from global memory (coalesced over c), and runs
//     the L/128-point transforms there.
//   * Index bits 0-6: Y = H_128 X for the 128 x 64 matrix of the tile, on the
//     tensor cores or through shared memory.
//
// Tensor-core form.  H_128 is the M operand (exact in BF16), the tile the N
// operand: every FP32 value is split into BF16 hi + mid + lo (each part the
// round-to-nearest BF16 of what the earlier parts leave; the sum equals x to
// about 2^-27 |x|), so products are exact and only the FP32 accumulation
// rounds.  K = 128 runs as two accumulators of K = 64, added on the CUDA
// cores, the small parts first, so that only four accumulations see full-size
// sums.  D's lanes are the elements of a block: the epilogue's stores are
// coalesced.  Persistent CTAs of 13 warps, one per SM: two groups of four
// loader warps (load, transform, split; three operand buffers), one MMA warp,
// four epilogue warps (two accumulator buffers).
//
// Bound: HBM, 8 bytes a value; per tile and SM 1.5 us at 6.5 TB/s against some
// 1000 cycles of loader issue and 1150 of tensor core.  The earlier form (two
// Hadamard-16 stages, each a split, an MMA and a TMEM round trip in 128-thread
// CTAs) waited on its chain of phases: 16384 rows of 8192 took 1.00 ms, now 0.236
// ms (4.6 TB/s).  The CUDA-core form went from 0.268 to 0.219 ms (4.9 TB/s): its
// stages made eight passes over shared memory, now four.
//
// Waits: every mbarrier wait is bounded; when one runs out the CTA records it
// in a host-mapped flag, waits (bounded) for the MMAs it issued, frees its
// tensor memory and returns.
#include <cuda_bf16.h>

#include <mutex>

#include "cmm_fft_device.cuh"
#include "cmm_internal.h"
#include "cmm_product_dev.cuh"

namespace cmm {
namespace {

// A tile is NB blocks of 128: 64, or those of one row where there are few rows
// (wht_launch_rows).

// element c of the tile's blocks (zero beyond `left` elements)
template <int NB>
__device__ __forceinline__ void load_column(const float* __restrict__ src, int c, int64_t left, float (&v)[NB]) {
  if (left >= NB * 128) {
#pragma unroll
    for (int g = 0; g < NB; ++g) v[g] = __ldcs(src + g * 128 + c);
  } else {
#pragma unroll
    for (int g = 0; g < NB; ++g) v[g] = g * 128 + c < left ? __ldcs(src + g * 128 + c) : 0.f;
  }
}
// index bits 7 and up: transforms over the F = L / 128 blocks of each row
template <int LOGL, int NB>
__device__ __forceinline__ void block_transform(float (&v)[NB]) {
  constexpr int F = 1 << (LOGL - 7);
#pragma unroll
  for (int h = 1; h < F; h <<= 1)
#pragma unroll
    for (int g = 0; g < NB; ++g)
      if (!(g & h)) {
        const float a = v[g], b = v[g + h];
        v[g] = a + b;
        v[g + h] = a - b;
      }
}

// ---------------------------------------------------------------- CUDA cores
// 128 threads per tile; the 128-point transforms as NB-point transforms in
// registers (TP = 128 / NB threads a block, through shared memory) and exchanges
// between those neighbouring lanes.  X[g][c] at g (128 + TP) + c + c / NB: both
// access patterns touch every bank once (NB = 16: one of them twice).
constexpr int kCcThreads = 128;

template <int LOGL, int NB>
__global__ void __launch_bounds__(kCcThreads, 5) k_wht_rows(const float* x, float* y, int64_t elements) {
  constexpr int TP = 128 / NB, kTile = NB * 128, kRow = 128 + TP;
  __shared__ float X[NB * kRow];
  const int tid = threadIdx.x;
  for (int64_t e0 = (int64_t)blockIdx.x * kTile; e0 < elements; e0 += (int64_t)gridDim.x * kTile) {
    const int64_t left = elements - e0;
    float v[NB];
    load_column<NB>(x + e0, tid, left, v);
    block_transform<LOGL, NB>(v);
#pragma unroll
    for (int g = 0; g < NB; ++g) X[g * kRow + tid + tid / NB] = v[g];
    __syncthreads();
    const int part = tid % TP, at = tid / TP * kRow + part * (NB + 1);
#pragma unroll
    for (int j = 0; j < NB; ++j) v[j] = X[at + j];
    dev::whtr<float, NB>(v);
#pragma unroll
    for (int h = 1; h < TP; h <<= 1)
#pragma unroll
      for (int j = 0; j < NB; ++j) {
        const float o = __shfl_xor_sync(0xffffffffu, v[j], h);
        v[j] = part & h ? o - v[j] : v[j] + o;
      }
#pragma unroll
    for (int j = 0; j < NB; ++j) X[at + j] = v[j];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NB; ++q)
      if (left >= kTile || q * 128 + tid < left) __stcs(y + e0 + q * 128 + tid, X[q * kRow + tid + tid / NB]);
    __syncthreads();
  }
}

// -------------------------------------------------------------- tensor cores
constexpr int kLoaders = 256, kTcThreads = kLoaders + 128 + 32;
constexpr int kBufs = 3;
// operand layouts, no-swizzle K-major core matrices (8 rows x 16 bytes, 8-row
// groups 128 bytes apart): H128 with 2048 bytes between 8-element K units; the
// tile's splits with 1056 (64 rows x 16 bytes and 32 spare, which spread the
// loaders' stores over the banks)
constexpr int kUnitA = 2048, kUnitB = 1056;
constexpr int kSplitBytes = 16 * kUnitB, kBufBytes = 3 * kSplitBytes;
constexpr int kTcSmem = 16 * kUnitA + kBufs * kBufBytes + 128;

__device__ __forceinline__ uint64_t kmajor_desc(uint32_t saddr, int unit) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)(unit >> 4) << 16) | ((uint64_t)(128 >> 4) << 32) | (1ull << 46);
}
// instruction descriptor, kind::f16: D FP32 (bits 4-5 = 1), A and B BF16 (bits
// 7-9 and 10-12 = 1), both K-major, N (>> 3 at bit 17), M = 128 (>> 4 at bit 24)
template <int N>
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | (((uint32_t)N >> 3) << 17) | ((128u >> 4) << 24);

template <int N>
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(adesc), "l"(bdesc), "r"(kIdesc<N>), "r"(accumulate));
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
      "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_ld_wait(uint32_t (&a)[32], uint32_t (&b)[32]) {
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int u = 0; u < 32; ++u) asm volatile("" : "+r"(a[u]), "+r"(b[u]));  // not used before the wait
}
// (lo, hi) -> packed BF16 pair and what it leaves of both
__device__ __forceinline__ uint32_t take_bf16x2(float& a, float& b) {
  const __nv_bfloat162 p = __floats2bfloat162_rn(a, b);
  const uint32_t w = *reinterpret_cast<const uint32_t*>(&p);
  a -= __uint_as_float(w << 16);
  b -= __uint_as_float(w & 0xffff0000u);
  return w;
}

template <int LOGL, int NB>
__global__ void __launch_bounds__(kTcThreads, 1) k_wht_rows_tc(const float* x, float* y, int64_t elements, int* timeout) {
  constexpr int kTile = NB * 128;
  extern __shared__ __align__(128) unsigned char wsm[];
  unsigned char* As = reinterpret_cast<unsigned char*>(((uintptr_t)wsm + 127) & ~(uintptr_t)127);
  unsigned char* Bs = As + 16 * kUnitA;
  __shared__ uint64_t full[kBufs], empty[kBufs], accfull[2], accempty[2], drain;
  __shared__ uint32_t tmem_base;
  __shared__ int s_wait[2];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // H128[n][k] at unit k / 8, row n, eight elements of K a store
  for (int e = tid; e < 128 * 16; e += kTcThreads) {
    const int n = e & 127, u = e >> 7;
    const uint32_t row = __popc(n & (8 * u)) & 1 ? 0xbf80bf80u : 0x3f803f80u;
    uint32_t w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
      w[q] = row ^ ((__popc(n & (2 * q)) & 1) << 15) ^ ((uint32_t)(__popc(n & (2 * q + 1)) & 1) << 31);
    *reinterpret_cast<uint4*>(As + u * kUnitA + n * 16) = make_uint4(w[0], w[1], w[2], w[3]);
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base)),
                 "r"(256u)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (tid == 0) {
    for (int s = 0; s < kBufs; ++s) { bar_init(&full[s], 128); bar_init(&empty[s], 1); }
    for (int s = 0; s < 2; ++s) { bar_init(&accfull[s], 1); bar_init(&accempty[s], 4); }
    bar_init(&drain, 1);
    s_wait[0] = 0;
    s_wait[1] = kWaitUs;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // H128 -> visible to the tensor core
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = tmem_base;
  volatile int* wait = s_wait;
  const int64_t step = (int64_t)gridDim.x * kTile;

  if (tid < kLoaders) {
    // group w takes every second tile of this CTA
    const int w = tid >> 7, c = tid & 127;
    unsigned it = w;
    for (int64_t e0 = ((int64_t)blockIdx.x + (int64_t)w * gridDim.x) * kTile; e0 < elements; e0 += 2 * step, it += 2) {
      float v[NB];
      load_column<NB>(x + e0, c, elements - e0, v);
      block_transform<LOGL, NB>(v);
      const unsigned buf = it % kBufs;
      if (!__all_sync(0xffffffffu, bar_wait(&empty[buf], ((it / kBufs) & 1u) ^ 1u, wait))) break;
      // neighbouring lanes trade, so that each holds the pair (c, c + 1) of
      // half of the blocks: 4-byte stores, eight lanes 32 contiguous bytes
      unsigned char* dst = Bs + buf * kBufBytes + (c >> 3) * kUnitB + (c & 1) * 16 + ((c & 7) >> 1) * 4;
#pragma unroll
      for (int g = 0; g < NB; g += 2) {
        const float o = __shfl_xor_sync(0xffffffffu, c & 1 ? v[g] : v[g + 1], 1);
        float a = c & 1 ? o : v[g], b = c & 1 ? v[g + 1] : o;
#pragma unroll
        for (int s = 0; s < 3; ++s) *reinterpret_cast<uint32_t*>(dst + s * kSplitBytes + g * 16) = take_bf16x2(a, b);
      }
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      bar_arrive(&full[buf]);
    }
  } else if (tid < kLoaders + 128) {
    const int q = warp & 3;  // TMEM lanes 32 q .. 32 q + 31
    unsigned it = 0;
    for (int64_t e0 = (int64_t)blockIdx.x * kTile; e0 < elements; e0 += step, ++it) {
      const unsigned ab = it & 1u;
      const bool ok = __all_sync(0xffffffffu, bar_wait(&accfull[ab], (it >> 1) & 1u, wait));
      if (!ok) break;
      tc_fence_after();
      const int64_t left = elements - e0;
      float* out = y + e0 + 32 * q + lane;
#pragma unroll
      for (int n0 = 0; n0 < NB; n0 += 32) {  // (NB = 16: the other columns are not used)
        uint32_t a[32], b[32];
        const uint32_t t = tbase + ((uint32_t)(32 * q) << 16) + ab * 128u + n0;
        tmem_ld32(t, a);
        tmem_ld32(t + 64, b);
        tmem_ld_wait(a, b);
        if (n0 + 32 >= NB) {  // the accumulators are read
          tc_fence_before();
          __syncwarp();
          if (lane == 0) bar_arrive(&accempty[ab]);
        }
#pragma unroll
        for (int u = 0; u < (NB < 32 ? NB : 32); ++u) {
          const int at = (n0 + u) * 128;
          if (left >= kTile || at + 32 * q + lane < left) __stcs(out + at, __uint_as_float(a[u]) + __uint_as_float(b[u]));
        }
      }
    }
  } else if (lane == 0) {
    unsigned it = 0;
    const uint64_t da = kmajor_desc(smem_u32(As), kUnitA);
    for (int64_t e0 = (int64_t)blockIdx.x * kTile; e0 < elements; e0 += step, ++it) {
      const unsigned buf = it % kBufs, ab = it & 1u;
      if (!bar_wait(&accempty[ab], ((it >> 1) & 1u) ^ 1u, wait)) break;
      if (!bar_wait(&full[buf], (it / kBufs) & 1u, wait)) break;
      tc_fence_after();
      const uint64_t db = kmajor_desc(smem_u32(Bs + buf * kBufBytes), kUnitB);
#pragma unroll
      for (int s = 2; s >= 0; --s)  // lo, mid, hi
#pragma unroll
        for (int k = 0; k < 4; ++k)
#pragma unroll
          for (int half = 0; half < 2; ++half) {  // 16 elements of K: two units
            const int u = 2 * (4 * half + k);
            mma_bf16<NB>(tbase + ab * 128u + half * 64u, da + (uint64_t)(u * (kUnitA >> 4)),
                     db + (uint64_t)(s * (kSplitBytes >> 4) + u * (kUnitB >> 4)), s == 2 && k == 0 ? 0u : 1u);
          }
      mma_commit(&empty[buf]);
      mma_commit(&accfull[ab]);
    }
  }
  __syncthreads();
  if (s_wait[0] && tid == kLoaders + 128) {  // the MMAs this CTA issued, before their columns are freed
    atomicExch(timeout, 1);
    mma_commit(&drain);
    bar_drain(&drain, 0, wait);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(256u) : "memory");
}

template <int LOGL, int NB>
void wht_launch(bool tc, const float* x, float* y, int64_t rows, int* timeout, cudaStream_t s) {
  const int64_t elements = rows << LOGL, tiles = (elements + NB * 128 - 1) / (NB * 128);
  if (tc) {
    CMM_CUDA(cudaFuncSetAttribute(k_wht_rows_tc<LOGL, NB>, cudaFuncAttributeMaxDynamicSharedMemorySize, kTcSmem));
    k_wht_rows_tc<LOGL, NB><<<(unsigned)std::min<int64_t>(tiles, num_sms()), kTcThreads, kTcSmem, s>>>(x, y, elements, timeout);
  } else {
    k_wht_rows<LOGL, NB><<<(unsigned)std::min<int64_t>(tiles, (int64_t)num_sms() * 5), kCcThreads, 0, s>>>(x, y, elements);
  }
  CMM_CUDA(cudaGetLastError());
  count_launch();
}
// Few rows of 2^11 and 2^12: a tile a row, since four (two) rows one after another
// in a CTA take longer than side by side, as long as the CTAs are there at once
// (tensor form: one per SM).  A call with 148 rows of 2^11: CUDA cores 16.6 -> 15.6
// us, tensor 19.1 -> 17.7; with 500 in the tensor form, 64 blocks a tile take
// 18.8, 16 take 20.3.
template <int LOGL>
void wht_launch_rows(bool tc, const float* x, float* y, int64_t rows, int* timeout, cudaStream_t s) {
  constexpr int kRowBlocks = 1 << (LOGL - 7);
  if (rows <= (tc ? 1 : 2) * (int64_t)num_sms()) wht_launch<LOGL, kRowBlocks>(tc, x, y, rows, timeout, s);
  else wht_launch<LOGL, 64>(tc, x, y, rows, timeout, s);
}

// host-mapped timeout flag of the calling host thread (one per thread, so
// that concurrent calls from several threads do not clear each other's report)
int* wht_timeout_flag(int** dev) {
  thread_local int* host = nullptr;
  thread_local int* mapped = nullptr;
  if (!host) {
    int* h = nullptr;
    int* m = nullptr;
    CMM_CUDA(cudaHostAlloc(reinterpret_cast<void**>(&h), sizeof(int), cudaHostAllocMapped));
    *h = 0;
    if (cudaHostGetDevicePointer(reinterpret_cast<void**>(&m), h, 0) != cudaSuccess) {
      cudaFreeHost(h);
      throw cuda_error("cudaHostGetDevicePointer failed for the WHT timeout flag");
    }
    host = h;  // both set only once both calls succeeded
    mapped = m;
  }
  if (dev) *dev = mapped;
  return host;
}

}  // namespace

void wht_rows_f32(const float* x, float* y, int64_t rows, int log2n, int method, cudaStream_t s) {
  if (rows < 0) throw invalid_argument("rows must be non-negative");
  if (log2n < 11 || log2n > 13) throw unsupported("the row length must be 2^11, 2^12 or 2^13");
  if (method != 0 && method != 1) throw invalid_argument("method must be 0 (CUDA cores) or 1 (tensor cores)");
  if (rows == 0) return;
  if (!x || !y) throw invalid_argument("x and y must not be null");
  if ((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) & 15)
    throw invalid_argument("x and y must be 16-byte aligned");
  int* dflag = nullptr;
  volatile int* hflag = wht_timeout_flag(&dflag);
  *hflag = 0;
  const bool tc = method == 1;
  switch (log2n) {
    case 11: wht_launch_rows<11>(tc, x, y, rows, dflag, s); break;
    case 12: wht_launch_rows<12>(tc, x, y, rows, dflag, s); break;
    default: wht_launch<13, 64>(tc, x, y, rows, dflag, s); break;
  }
  CMM_CUDA(cudaStreamSynchronize(s));
  if (tc) {
    if (*hflag) {
      *hflag = 0;
      throw runtime_error("tensor-core WHT: an MMA completion wait ran out");
    }
  }
}

}  // namespace cmm
