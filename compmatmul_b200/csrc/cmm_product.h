// Product sketch (cmm_product.cu): device job description and launchers.
#pragma once
#include <algorithm>

#include "cmm_internal.h"

namespace cmm {

constexpr int kProdTile = 128;                 // columns per plane tile (two per output tile side)
constexpr int kProdK = 32;                     // inner indices per int8 MMA
constexpr int kProdSlab = kProdTile * kProdK;  // bytes of a plane tile per kProdK inner indices
constexpr int64_t kProdMaxK = 32768;           // inner indices per launch (int32 accumulators)

// kProdK-index steps of a launch over kc inner indices, in whole stages of 4
__host__ __device__ inline int prod_ksteps(int64_t kc) { return (int)((kc + 4 * kProdK - 1) / (4 * kProdK)) * 4; }

enum { kAddGather = 0, kAddStaged = 1, kAddLane = 2 };  // forms of the additions

struct ProdJob {
  const void *A, *B;      // kc x n_a, kc x n_b: the inner indices of this launch
  int64_t n_a, n_b, kc;
  int* rexp;              // kc: row balance exponents
  int *cexpA, *cexpB;     // column exponents
  double* csum;           // partial sums of squares and largest exponents of the columns:
  int* cmax;              //   ceil(kc / 256) x (n_a + n_b)
  int* flag;              // 1: a non-finite input or a failed wait
  uint8_t *slA, *slB;     // residue planes
  uint32_t* res;          // residues of the product: modulus x (64 tiles_p) x (256 tiles_b), four rows a word
  double* C;              // n_a x n_b, row stride ldc
  int64_t ldc;
  int64_t item_end;       // work items of this and all earlier jobs
  int tiles_a, tiles_b;   // output tiles of 256 columns of A and of B
  int tile0, tiles_p;     // the tiles of A of this launch (a panel of rows of C)
  int accumulate;         // add to C (later chunks of the inner index)
  // the sketch
  const uint32_t *codesA, *codesB;
  void* cum;              // sorted columns (cmm_product_add.cu): positions of the buckets
  uint32_t* ent;          //   and entries, 2 d x n_b
  double *part, *p;       // G x d x b partial sketches; d x b
  int d, log2b, variant;
  int form;               // which additions (plan_product_sketch)
  int logW, G;            // window of a warp, row groups
  int blocks;             // blocks of columns (staged and lane forms)
};

inline int prod_moduli(bool f32) { return f32 ? 8 : 15; }
inline int prod_tiles(int64_t n) { return (int)((n + 255) / 256); }
// residue planes of n columns x kc inner indices; residues of a panel
inline size_t prod_plane_bytes(int64_t n, int64_t kc, bool f32) {
  return (size_t)prod_moduli(f32) * 2 * prod_tiles(n) * prod_ksteps(kc) * kProdSlab;
}
inline size_t prod_residue_bytes(int tiles_p, int tiles_b, bool f32) {
  return (size_t)prod_moduli(f32) * 65536 * tiles_p * tiles_b;
}

// geometry of the additions of a job from its sizes (form, logW, G, blocks)
void plan_product_sketch(ProdJob& J, int sms);
size_t prod_cum_bytes(const ProdJob& J);
// C's row stride: even, so that rows can be copied in 16-byte units
inline int64_t prod_ldc(int64_t n_b) { return (n_b + 1) & ~(int64_t)1; }
// the largest n_a n_b whose product is formed (8 GiB of FP64)
constexpr int64_t kProdMaxEntries = (int64_t)1 << 30;

// hJobs: the host copy of dJobs.  Sorted columns (also clears the flags);
// exponents and residue planes; the product; the additions and their sum.
void launch_product_index(const ProdJob* hJobs, const ProdJob* dJobs, int count, cudaStream_t s);
void launch_product_planes(const ProdJob* hJobs, const ProdJob* dJobs, int count, bool f32, cudaStream_t s);
void launch_product_gemm(const ProdJob* hJobs, const ProdJob* dJobs, int count, bool f32, cudaStream_t s);
void launch_product_add(const ProdJob* hJobs, const ProdJob* dJobs, int count, cudaStream_t s);
// host-mapped flag set by a wait of these kernels that ran out (*dev: its device address)
int* product_timeout_flag(int** dev);
// true (and cleared) when such a wait ran out since the last call
bool product_timed_out();

}  // namespace cmm
