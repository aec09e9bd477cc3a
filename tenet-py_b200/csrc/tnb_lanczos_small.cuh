// A whole Lanczos solve of a small problem as one CTA: what tnb_lanczos_solve hands the kernel
// in tnb_lanczos_small.cu.
#pragma once

#include "tnb_common.cuh"

namespace tnb {

constexpr int kSmallMaxStages = 12, kSmallMaxBufs = 32, kSmallMaxRows = 256;
constexpr int kSmallMaxSmem = 214 * 1024;  // (and 12.5 KB of the kernel's own)

// A stage of the recorded matvec.  Buffers are offsets (in doubles) into shared memory.
struct SmallStage {
  int gather;           // 1: a gather of warp items, 0: a grouped GEMM
  int width, count;     // words per item row and items; or the GEMM table's rows in `count`
  int rows_at;          // where a gather's item rows, or K and ldb per GEMM row, lie (bytes)
  int recs_at;          // the records of the stage's elements, 8 bytes each (bytes)
  int split_at;         // four bytes more per element of a gather of several terms (bytes)
  int src, n_src;       // the gather's source, or A
  int b, n_b;           // B
  int dst, n_dst;
  const void* rows;
  const int64_t* term_src;
  const double* term_coeff;
  const int64_t* term_ld;
  int64_t n_term;
};

// A buffer of the recorded launches: its copy in shared memory starts as it is.
struct SmallBuf {
  const double* from;
  int at, n;
};

struct SmallArgs {
  int n_stages, n_bufs;
  SmallStage st[kSmallMaxStages];
  SmallBuf buf[kSmallMaxBufs];
  int x, y, prev;       // the matvec's input and output, the vector before the input
  int weight;           // the weight of every element of a vector
  int order_at;         // n 16-bit words: the elements in the order the sums add them (bytes)
  int n_runs, n, ncv;
  double tol;
  const int64_t* run_start;
  const double* run_w;
  const double* x0;
  double* v;
  int64_t ldv;
  double* w;
  double* state;
  double* scal;
};

int launch_lanczos_small(const SmallArgs& a, int smem, cudaStream_t stream);

}  // namespace tnb
