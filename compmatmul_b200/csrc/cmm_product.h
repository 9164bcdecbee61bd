// Product sketch (cmm_product.cu): device job description and launchers.
#pragma once
#include <algorithm>

#include "cmm_internal.h"

namespace cmm {

constexpr int kProdTile = 128;                 // columns per plane tile (two per output tile side)
constexpr int kProdK = 32;                     // inner indices per int8 MMA
constexpr int kProdSlab = kProdTile * kProdK;  // bytes of a plane tile per kProdK inner indices
constexpr int kProdColRows = 64;               // inner indices per partial sum of a column's squares
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
  int* cmax;              //   ceil(kc / kProdColRows) x (n_a + n_b)
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
  int form;               // which additions (product_geometry)
  int logW, G;            // window of a warp, row groups
  int per_sm;             // CTAs of the additions per SM
  int add_begin, add_x;   // their first CTA in the launch of their kind, CTAs per (t, row group)
  int blocks;             // blocks of columns (staged and lane forms)
};

inline int prod_moduli(bool f32) { return f32 ? 8 : 15; }
// C's row stride: even, so that rows can be copied in 16-byte units
inline int64_t prod_ldc(int64_t n_b) { return (n_b + 1) & ~(int64_t)1; }
// bytes of the residues of one output tile row (256 columns of A)
inline size_t prod_residue_row(const ProdJob& J, bool f32) { return (size_t)prod_moduli(f32) * 65536 * J.tiles_b; }
// the largest n_a n_b whose product is formed (8 GiB of FP64)
constexpr int64_t kProdMaxEntries = (int64_t)1 << 30;

// Whether the product sketch takes these sizes, and whether it is estimated to be
// faster than the transforms: for a single call, for a product of a batch plan or
// a request, and for the products of a plan together, whose launches come on top
// (others: the plan runs transforms for other products anyway).
bool product_supported(int b, int64_t n_a, int64_t n_inner, int64_t n_b);
bool product_faster(int variant, bool f32, int d, int b, int64_t n_a, int64_t n_inner, int64_t n_b);
bool product_among_others(int variant, bool f32, int d, int b, int64_t n_a, int64_t n_inner, int64_t n_b);
bool products_pay(const ProdJob* jobs, int count, bool f32, bool others);

// bytes of the residue planes of a chunk of k inner indices
inline size_t prod_plane_bytes(bool f32, int64_t n_a, int64_t n_b, int64_t k) {
  return (size_t)prod_moduli(f32) * 256 * (size_t)((n_a + 255) / 256 + (n_b + 255) / 256) * (size_t)((k + 127) / 128 * 128);
}
// A launch's planes (of 128 inner indices at least), and the partial sketches
// of its row groups (of one at least), take no more than this.
constexpr size_t kProdMaxBytes = (size_t)8 << 30;

// Sizes, tiles and additions of a job of kc inner indices (kc <= kProdMaxK)
// with all rows of C in one panel.  alone: the job has the device for itself
// (row groups to fill it); otherwise the row groups follow from the job's
// sizes only, so that it computes the same among any others.
void product_geometry(ProdJob& J, int variant, int d, int b, int64_t n_a, int64_t n_b, int64_t kc, bool alone, int sms);
// Device memory of a job: the sorted columns (they depend on the hash codes
// only), and the work space for J.kc inner indices and J.tiles_p tiles; with
// C in it, or in the caller's n_a x n_b doubles where those are usable.
size_t product_list_bytes(const ProdJob& J);
void product_set_lists(ProdJob& J, void* base);
bool product_usable_c(const ProdJob& J, const double* c);
size_t product_work_bytes(const ProdJob& J, bool f32, bool own_c);
void product_set_work(ProdJob& J, void* base, bool f32, double* c);

// Places of the jobs of one launch in its work lists (item_end, add_begin).
void product_layout(ProdJob* jobs, int count, bool f32);

// hJobs: the host copy of dJobs, laid out.  Sorted columns (also clears
// the flags); exponents and residue planes; the product; the additions.
void launch_product_index(const ProdJob* hJobs, const ProdJob* dJobs, int count, cudaStream_t s);
void launch_product_planes(const ProdJob* hJobs, const ProdJob* dJobs, int count, bool f32, cudaStream_t s);
// (flag: device address of the caller's WaitFlag)
void launch_product_gemm(const ProdJob* hJobs, const ProdJob* dJobs, int count, bool f32, int* flag, cudaStream_t s);
void launch_product_add(const ProdJob* hJobs, const ProdJob* dJobs, int count, int* flag, cudaStream_t s);
// kernels of one planes + product + additions sequence
int product_launches(const ProdJob* hJobs, int count);

// Set by a wait of these kernels that ran out; its sketch is NaN.  One for each
// caller that reports on its own: a host thread's single calls, a batch plan, a
// stream of a server.  Kernels that may set it have ended when it is destroyed.
class WaitFlag {
 public:
  WaitFlag();
  ~WaitFlag();
  WaitFlag(const WaitFlag&) = delete;
  WaitFlag& operator=(const WaitFlag&) = delete;
  int* dev() const { return dev_; }
  bool take();  // true (and cleared) when a wait ran out since the last call

 private:
  int *host_ = nullptr, *dev_ = nullptr;
};
WaitFlag& thread_wait_flag();
// How a kernel's waits end: the flag, the limit, and arrivals that its barriers
// wait for and do not get (the test hook CMM_TEST_PRODUCT_WAIT = product | add)
struct ProdWaits {
  int* flag;
  int limit_us, extra;
};
ProdWaits product_waits(int* flag, const char* kernel);

}  // namespace cmm
