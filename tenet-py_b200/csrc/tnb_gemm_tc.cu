// K2-TC: the grouped coupled-sector GEMM on the 5th-generation tensor cores (tcgen05).
//
// The precision form of the block GEMMs: the same descriptor table as the FP64 kernels,
// FP64 operands in and FP64 results out, but every product runs as tcgen05.mma with FP32
// accumulators held in tensor memory:
//   TNB_TILE_TC_TF32    A, B rounded to TF32 (kind::tf32);
//   TNB_TILE_TC_3XBF16  A = A_hi + A_lo, B = B_hi + B_lo split into BF16 pairs and the
//                       product taken as A_hi B_hi + A_hi B_lo + A_lo B_hi (kind::f16 with
//                       BF16 inputs), which keeps about 16 significand bits of every
//                       operand instead of 8.
//
// Two launches per table.  A pack kernel converts each operand once: every 128-row x
// 32 slab of A (and of B^T) becomes one 16 KB chunk of the work buffer, already in the
// canonical K-major, no-swizzle UMMA shared-memory layout (8-row x 16-byte core
// matrices, LBO = 128 B between the two core matrices of one K step, SBO between 8-row
// groups), parts (BF16 hi, lo) back to back.  Only the 8-row groups that hold rows of the
// operand are written and later copied (a prefix of each part): a row past M or N only
// reaches accumulators that are never stored, and the sectors of a symmetric tensor fill
// 14 to 40 of 128 rows.  The MMA kernel gives each CTA a 128 x 128
// output tile and runs a three-stage pipeline: one producer thread copies the next A and
// B slabs with cp.async.bulk (global -> shared, completion counted in bytes on the
// stage's "full" mbarrier), one issuer thread waits for "full", issues the MMAs into a
// 128-lane x 128-column TMEM accumulator and commits them to the stage's "empty"
// mbarrier, which the producer waits on before refilling the stage.  The epilogue reads
// TMEM with tcgen05.ld (warp w owns lanes 32w..32w+31) and writes FP64.  Every wait is
// bounded: past the limit the kernel raises TNB_ETIMEOUT, stops, and still frees its
// TMEM before returning.  No copy uses cluster multicast.
#include <cuda_bf16.h>

#include <string>

#include "tnb_common.cuh"

namespace tnb {

constexpr int kT2M = 128, kT2N = 128, kT2Bk = 32, kT2Threads = 128, kT2Stages = 3;
constexpr int kT2Slab = 16384;  // bytes of one packed operand slab, all parts
constexpr unsigned kT2TmemCols = 128;
constexpr long long kT2WaitCycles = 4000000000LL;  // ~2 s at the boost clock

struct T2Row {
  int64_t M, N, K, aoff, lda, boff, ldb, coff, ldc, tile_begin, tiles_n, a_chunk, b_chunk;
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// UMMA shared-memory descriptor, SWIZZLE_NONE, K-major, SM100 version 1.
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return static_cast<uint64_t>((saddr >> 4) & 0x3FFFu) |
         (static_cast<uint64_t>((lbo >> 4) & 0x3FFFu) << 16) |
         (static_cast<uint64_t>((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor: FP32 accumulate, both operands K-major, M = 128, N = 128.
__host__ __device__ constexpr uint32_t umma_idesc(uint32_t fmt) {
  return (1u << 4) | (fmt << 7) | (fmt << 10) | ((kT2N >> 3) << 17) | ((kT2M >> 4) << 24);
}

// Byte offset of element (r, k) of a K-major tile whose rows hold `row_bytes` bytes.
__device__ __forceinline__ uint32_t kmajor(int r, int k, int esz, int row_bytes) {
  const int bk = k * esz;
  return (r >> 3) * (row_bytes / 16) * 128 + (bk >> 4) * 128 + (r & 7) * 16 + (bk & 15);
}

__device__ __forceinline__ uint32_t to_tf32(double x) {
  uint32_t u;
  asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(u) : "f"(static_cast<float>(x)));
  return u;
}

__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t phase) {
  const long long t0 = clock64();
  while (true) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}"
        : "=r"(done) : "r"(mbar), "r"(phase) : "memory");
    if (done) return true;
    if (clock64() - t0 > kT2WaitCycles) return false;
  }
}

template <int MODE>
struct T2Layout {
  static constexpr int kEsz = MODE == 0 ? 4 : 2;
  static constexpr int kRowBytes = kT2Bk * kEsz;      // one 32-wide K row of one part
  static constexpr int kParts = MODE == 0 ? 1 : 2;
  static constexpr int kPartBytes = kT2M * kRowBytes;  // 16 KB (TF32) or 8 KB (BF16)
  static_assert(kParts * kPartBytes == kT2Slab, "a slab is 16 KB");
  static constexpr int kStageBytes = 2 * kT2Slab;      // A slab + B slab
  static constexpr int kSmemBytes = kT2Stages * kStageBytes + 1024;
};

__device__ __forceinline__ bool load_t2row(const int64_t* table, int64_t g, T2Row& r) {
  const int64_t* t = table + g * TNB_GEMM_WIDTH;
  r.M = t[0]; r.N = t[1]; r.K = t[2]; r.aoff = t[3]; r.lda = t[4]; r.boff = t[5];
  r.ldb = t[6]; r.coff = t[7]; r.ldc = t[8]; r.tile_begin = t[9]; r.tiles_n = t[10];
  r.a_chunk = t[12]; r.b_chunk = t[13];
  return r.M >= 0 && r.N >= 0 && r.K >= 0 && r.a_chunk >= 0 && r.b_chunk >= 0;
}

// One packed slab: its first element in the operand, the operand's leading dimension, and how
// many of its 128 rows and 32 columns of K the operand has.
struct Slab {
  int64_t off, ld;
  int rows, cols;
};

// The slab `chunk` of operand A (which == 0) or B (which == 1) from the GEMM table: its row
// is the last one whose first chunk is <= chunk (rows in chunk order), found by the warp in
// ceil(log32 n_gemm) rounds of 32 probes.
__device__ Slab find_slab(const int64_t* table, int64_t n_gemm, int64_t chunk, int which,
                          int lane) {
  int64_t lo = 0, n = n_gemm;  // the row is in [lo, lo + n)
  while (n > 1) {
    const int64_t step = (n + 31) / 32;
    const bool before = lane * step < n &&
                        table[(lo + lane * step) * TNB_GEMM_WIDTH + 12 + which] <= chunk;
    const int last = 31 - __clz(__ballot_sync(0xffffffffu, before || lane == 0));
    n = min(step, n - last * step);
    lo += last * step;
  }
  T2Row r;
  Slab s{0, 0, 0, 0};
  if (!load_t2row(table, lo, r)) return s;
  const int64_t ks = (r.K + kT2Bk - 1) / kT2Bk;
  const int64_t local = chunk - (which == 0 ? r.a_chunk : r.b_chunk);
  const int64_t rows = which == 0 ? r.M : r.N;
  if (ks == 0 || local < 0) return s;
  const int64_t t0 = (local / ks) * kT2M, k0 = (local % ks) * kT2Bk;
  if (t0 >= rows) return s;
  s.ld = which == 0 ? r.lda : r.ldb;
  s.off = which == 0 ? r.aoff + t0 * s.ld + k0 : r.boff + k0 * s.ld + t0;
  s.rows = static_cast<int>(min(rows - t0, int64_t(kT2M)));
  s.cols = static_cast<int>(min(r.K - k0, int64_t(kT2Bk)));
  return s;
}

// Eight consecutive K elements of one slab row in the UMMA layout: one 16-byte store per
// BF16 part, or two of TF32.
template <int MODE>
__device__ __forceinline__ void pack_eight(uint8_t* slab, int row, int kg, const double (&x)[8]) {
  using L = T2Layout<MODE>;
  if constexpr (MODE == 0) {
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      uint4 v;
      v.x = to_tf32(x[4 * h]);
      v.y = to_tf32(x[4 * h + 1]);
      v.z = to_tf32(x[4 * h + 2]);
      v.w = to_tf32(x[4 * h + 3]);
      *reinterpret_cast<uint4*>(slab + kmajor(row, 8 * kg + 4 * h, L::kEsz, L::kRowBytes)) = v;
    }
  } else {
    __align__(16) __nv_bfloat16 hi[8], lo[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      hi[j] = __double2bfloat16(x[j]);
      lo[j] = __double2bfloat16(x[j] - static_cast<double>(__bfloat162float(hi[j])));
    }
    uint8_t* const p = slab + kmajor(row, 8 * kg, L::kEsz, L::kRowBytes);
    *reinterpret_cast<uint4*>(p) = *reinterpret_cast<const uint4*>(hi);
    *reinterpret_cast<uint4*>(p + L::kPartBytes) = *reinterpret_cast<const uint4*>(lo);
  }
}

// Pack one slab of A (blocks [0, a_chunks): rows = M, read along K) or of B^T (blocks after
// them: rows = N, read along N) into its work-buffer chunk.  Warps work alone: one takes 8
// rows x 32 K of A or 32 rows x 8 K of B at a time, a lane eight K elements of one row, all
// eight loads in flight, and stores whole 16-byte core-matrix rows (a warp's stores fill 512
// contiguous bytes of A, 128-byte runs of B).  `slabs` (four words per slab: Slab with rows |
// cols << 32) makes a slab's description one load; without it each warp searches the table.
// Measured (before: slabs assembled element by element in shared memory behind a 12-step
// binary search, whole slabs written): the operands of the 64-member environment update's two
// products 130 us in all (566; 462 with the 32-way search alone), of a dense U(1) contraction
// 21 us (35).
constexpr int kPackThreads = 256;

template <int MODE>
__global__ void __launch_bounds__(kPackThreads)
tc_pack_kernel(const int64_t* __restrict__ table, int64_t n_gemm,
               const int64_t* __restrict__ slabs, const double* __restrict__ a, int64_t n_a,
               const double* __restrict__ b, int64_t n_b, uint8_t* __restrict__ work,
               int64_t work_bytes, int64_t a_chunks) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int which = blockIdx.x < a_chunks ? 0 : 1;
  Slab s;
  if (slabs != nullptr) {
    const int64_t* w = slabs + static_cast<int64_t>(blockIdx.x) * 4;
    s.off = __ldg(w);
    s.ld = __ldg(w + 1);
    const int64_t rc = __ldg(w + 2);
    s.rows = static_cast<int>(rc);
    s.cols = static_cast<int>(rc >> 32);
  } else {
    s = find_slab(table, n_gemm, which == 0 ? blockIdx.x : blockIdx.x - a_chunks, which, lane);
  }
  // the slab's own rows and columns inside the operand, its chunk inside the work buffer
  const int64_t last = which == 0 ? s.off + (s.rows - 1) * s.ld + s.cols
                                  : s.off + (s.cols - 1) * s.ld + s.rows;
  if (s.rows < 1 || s.rows > kT2M || s.cols < 1 || s.cols > kT2Bk || s.off < 0 || s.ld < 0 ||
      last > (which == 0 ? n_a : n_b) ||
      (static_cast<int64_t>(blockIdx.x) + 1) * kT2Slab > work_bytes) {
    if (threadIdx.x == 0) raise_bounds();
    return;
  }
  uint8_t* const slab = work + static_cast<int64_t>(blockIdx.x) * kT2Slab;
  pdl_wait();  // the operand may be the previous kernel's output
  const double* const src = (which == 0 ? a : b) + s.off;
  const int pieces = which == 0 ? (s.rows + 7) / 8 : 4 * ((s.rows + 31) / 32);
  for (int i = warp; i < pieces; i += kPackThreads / 32) {
    const int row = which == 0 ? 8 * i + (lane & 7) : 32 * (i >> 2) + lane;
    const int kg = which == 0 ? lane >> 3 : i & 3;
    const int64_t at = which == 0 ? row * s.ld + 8 * kg : 8 * kg * s.ld + row;
    const int64_t step = which == 0 ? 1 : s.ld;
    double x[8];
#pragma unroll
    for (int j = 0; j < 8; ++j)
      x[j] = row < s.rows && 8 * kg + j < s.cols ? __ldg(src + at + j * step) : 0.0;
    if (row < ((s.rows + 7) & ~7)) pack_eight<MODE>(slab, row, kg, x);
  }
}

__device__ __forceinline__ void bulk_copy(uint32_t dst, const void* src, uint32_t bytes,
                                          uint32_t mbar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
      :: "r"(dst), "l"(src), "r"(bytes), "r"(mbar) : "memory");
}

template <int MODE>
__global__ void __launch_bounds__(kT2Threads)
tc_mma_kernel(const int64_t* __restrict__ table, int64_t n_gemm,
              const int32_t* __restrict__ tile_map, const uint8_t* __restrict__ work,
              int64_t work_bytes, int64_t b_chunk0, double* __restrict__ c, int64_t n_c) {
  using L = T2Layout<MODE>;
  extern __shared__ uint8_t smem_dyn[];
  uint8_t* const smem = reinterpret_cast<uint8_t*>(
      (reinterpret_cast<uintptr_t>(smem_dyn) + 1023) & ~static_cast<uintptr_t>(1023));
  __shared__ __align__(8) uint64_t full[kT2Stages], empty[kT2Stages], done;
  __shared__ uint32_t s_tmem;
  __shared__ T2Row s_row;
  __shared__ int s_ok, s_fail, s_fills, s_drain_fail;

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    T2Row r{};
    const int64_t g = tile_map[blockIdx.x];
    bool ok = g >= 0 && g < n_gemm && load_t2row(table, g, r);
    const int64_t ks = ok ? (r.K + kT2Bk - 1) / kT2Bk : 0;
    if (ok) {
      const int64_t mt = (r.M + kT2M - 1) / kT2M, nt = (r.N + kT2N - 1) / kT2N;
      ok = r.M > 0 && r.N > 0 && r.tiles_n == nt && r.coff >= 0 &&
           r.coff + (r.M - 1) * r.ldc + r.N <= n_c &&
           (ks == 0 || ((r.a_chunk + mt * ks) * kT2Slab <= work_bytes &&
                        (b_chunk0 + r.b_chunk + nt * ks) * kT2Slab <= work_bytes));
    }
    if (!ok) raise_bounds();
    s_row = r;
    s_ok = ok;
    s_fail = 0;
    s_fills = 0;
    s_drain_fail = 0;
    for (int st = 0; st < kT2Stages; ++st) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&full[st])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&empty[st])) : "memory");
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&done)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {  // one warp owns the TMEM allocation
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(smem_u32(&s_tmem)), "r"(kT2TmemCols) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = s_tmem;
  const T2Row r = s_row;
  const bool ok = s_ok;
  const int64_t local = blockIdx.x - r.tile_begin;
  const int64_t mtile = ok ? local / r.tiles_n : 0, ntile = ok ? local % r.tiles_n : 0;
  const int64_t nk = ok ? (r.K + kT2Bk - 1) / kT2Bk : 0;
  const uint8_t* a_src = work + (r.a_chunk + mtile * nk) * kT2Slab;
  const uint8_t* b_src = work + (b_chunk0 + r.b_chunk + ntile * nk) * kT2Slab;
  // bytes of a part's written 8-row groups (nothing past them is read into a stored element)
  const int rows_a = ok ? static_cast<int>(min(r.M - mtile * kT2M, int64_t(kT2M))) : 0;
  const int rows_b = ok ? static_cast<int>(min(r.N - ntile * kT2N, int64_t(kT2N))) : 0;
  const uint32_t bytes_a = static_cast<uint32_t>(((rows_a + 7) & ~7) * L::kRowBytes);
  const uint32_t bytes_b = static_cast<uint32_t>(((rows_b + 7) & ~7) * L::kRowBytes);
  pdl_wait();  // the packed operands are the pack kernels' output

  if (tid == 0 && nk > 0) {  // producer
    uint32_t ephase[kT2Stages] = {0u, 0u, 0u};
    for (int64_t s = 0; s < nk; ++s) {
      const int st = static_cast<int>(s % kT2Stages);
      if (s >= kT2Stages) {
        if (!mbar_wait(smem_u32(&empty[st]), ephase[st])) {
          atomicCAS(&g_device_error, 0, TNB_ETIMEOUT);
          s_fail = 1;
          break;
        }
        ephase[st] ^= 1u;
      }
      const uint32_t fb = smem_u32(&full[st]);
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                   :: "r"(fb), "r"(L::kParts * (bytes_a + bytes_b)) : "memory");
      const uint32_t sa = smem_u32(smem + st * L::kStageBytes);
#pragma unroll
      for (int p = 0; p < L::kParts; ++p) {
        bulk_copy(sa + p * L::kPartBytes, a_src + s * kT2Slab + p * L::kPartBytes, bytes_a, fb);
        bulk_copy(sa + kT2Slab + p * L::kPartBytes, b_src + s * kT2Slab + p * L::kPartBytes,
                  bytes_b, fb);
      }
      s_fills = static_cast<int>(s + 1);
    }
  } else if (tid == 32 && nk > 0) {  // MMA issuer
    uint32_t fphase[kT2Stages] = {0u, 0u, 0u};
    constexpr uint32_t kLbo = 128, kSbo = (L::kRowBytes / 16) * 128;
    constexpr uint32_t kIdesc = umma_idesc(MODE == 0 ? 2u : 1u);
    constexpr int kSteps = L::kRowBytes / 32;  // one MMA consumes 32 bytes of K
    constexpr int kProducts = MODE == 0 ? 1 : 3;  // 3xBF16: hi.hi, hi.lo, lo.hi
    for (int64_t s = 0; s < nk; ++s) {
      const int st = static_cast<int>(s % kT2Stages);
      if (!mbar_wait(smem_u32(&full[st]), fphase[st])) {
        atomicCAS(&g_device_error, 0, TNB_ETIMEOUT);
        s_fail = 1;
        break;
      }
      fphase[st] ^= 1u;
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t sa = smem_u32(smem + st * L::kStageBytes), sb = sa + kT2Slab;
#pragma unroll
      for (int p = 0; p < kProducts; ++p) {
        const int pa = p == 2 ? 1 : 0, pb = p == 1 ? 1 : 0;
#pragma unroll
        for (int k = 0; k < kSteps; ++k) {
          const uint64_t ad = umma_desc(sa + pa * L::kPartBytes + k * 256, kLbo, kSbo);
          const uint64_t bd = umma_desc(sb + pb * L::kPartBytes + k * 256, kLbo, kSbo);
          const uint32_t acc = (s > 0 || p > 0 || k > 0) ? 1u : 0u;
          if constexpr (MODE == 0) {
            asm volatile(
                "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::tf32 [%0], %1, %2, %3, q;\n\t}"
                :: "r"(tmem), "l"(ad), "l"(bd), "r"(kIdesc), "r"(acc) : "memory");
          } else {
            asm volatile(
                "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %4, 0;\n\t"
                "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, q;\n\t}"
                :: "r"(tmem), "l"(ad), "l"(bd), "r"(kIdesc), "r"(acc) : "memory");
          }
        }
      }
      asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                   :: "r"(smem_u32(&empty[st])) : "memory");
    }
    // the last commit covers every MMA issued before it
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 :: "r"(smem_u32(&done)) : "memory");
  }
  __syncthreads();
  // Drain before the stages are reused and TMEM is freed, on the error path too: the
  // issuer commits `done` after whatever MMAs it issued, and every stage's last fill has
  // bulk copies that land whatever happened to the consumer.  A drain that itself gives
  // up leaves shared memory and TMEM possibly still being written, so the epilogue then
  // stores nothing.
  if (tid == 0 && nk > 0) {
    if (!mbar_wait(smem_u32(&done), 0u)) {
      atomicCAS(&g_device_error, 0, TNB_ETIMEOUT);
      s_fail = 1;
      s_drain_fail = 1;
    }
    if (s_fail) {
      const int fills = s_fills;
      for (int st = 0; st < kT2Stages && st < fills; ++st) {
        const int n_st = (fills - st + kT2Stages - 1) / kT2Stages;  // fills of stage st
        if (!mbar_wait(smem_u32(&full[st]), static_cast<uint32_t>((n_st - 1) & 1)))
          s_drain_fail = 1;
      }
    }
  }
  __syncthreads();

  // epilogue: TMEM -> registers -> shared memory -> FP64 C, 16 columns at a time (zeros
  // when K == 0 or a wait gave up).  Warp w owns TMEM lanes (tile rows) 32w..32w+31; its
  // 32 x 16 block is transposed through shared memory (the drained pipeline stages) so
  // that each store instruction writes two rows' 16 consecutive columns.
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const int64_t row0 = mtile * kT2M + warp * 32;
  const int64_t n0 = ntile * kT2N;
  const bool live = ok && nk > 0 && !s_fail;
  double* const stage = reinterpret_cast<double*>(smem) + warp * (32 * 17);
  // columns past N and warps whose rows all lie past M have nothing to store (both
  // conditions are uniform across the warp, as tcgen05.ld requires)
  const int64_t cols = ok ? r.N - n0 : 0;
  const int n_chunks = cols >= kT2N ? kT2N / 16 : static_cast<int>((cols + 15) / 16);
  const int warp_chunks = ok && row0 < r.M && !s_drain_fail ? n_chunks : 0;
#pragma unroll 1
  for (int chunk = 0; chunk < warp_chunks; ++chunk) {
    uint32_t v[16];
    if (live) {
      const uint32_t taddr = tmem + (static_cast<uint32_t>(warp * 32) << 16) + chunk * 16;
      asm volatile(
          "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,"
          "%13,%14,%15}, [%16];"
          : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]),
            "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]),
            "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
          : "r"(taddr));
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    } else {
#pragma unroll
      for (int j = 0; j < 16; ++j) v[j] = 0u;
    }
    __syncwarp();  // the previous chunk's reads of the stage are done
#pragma unroll
    for (int j = 0; j < 16; ++j) stage[lane * 17 + j] = static_cast<double>(__uint_as_float(v[j]));
    __syncwarp();
    if (ok) {
#pragma unroll
      for (int it = 0; it < 16; ++it) {
        const int e = it * 32 + lane, rr = e >> 4, cc = e & 15;
        const int64_t row = row0 + rr, col = n0 + chunk * 16 + cc;
        if (row < r.M && col < r.N) c[r.coff + row * r.ldc + col] = stage[rr * 17 + cc];
      }
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;"
                 :: "r"(tmem), "r"(kT2TmemCols) : "memory");
  }
}

template <int MODE>
cudaError_t launch_tc_mode(unsigned grid, cudaStream_t s, const int64_t* table, int64_t n_gemm,
                           const int32_t* tile_map, const int64_t* slabs, const double* a, int64_t n_a,
                           const double* b, int64_t n_b, double* c, int64_t n_c, void* work,
                           int64_t work_bytes, int64_t a_chunks, int64_t b_chunks) {
  using L = T2Layout<MODE>;
  static PerDeviceOnce opted;
  cudaError_t e = opted.once([] {
    return cudaFuncSetAttribute(tc_mma_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                L::kSmemBytes);
  });
  if (e != cudaSuccess) return e;
  auto* w = static_cast<uint8_t*>(work);
  if (a_chunks + b_chunks > 0)
    e = launch(tc_pack_kernel<MODE>, static_cast<unsigned>(a_chunks + b_chunks), kPackThreads, s,
               table, n_gemm, slabs, a, n_a, b, n_b, w, work_bytes, a_chunks);
  if (e == cudaSuccess)
    e = launch_dyn(tc_mma_kernel<MODE>, grid, kT2Threads, L::kSmemBytes, s, table, n_gemm,
                   tile_map, static_cast<const uint8_t*>(w), work_bytes, a_chunks, c, n_c);
  return e;
}

cudaError_t launch_gemm_tc(int kind, unsigned grid, cudaStream_t s, const int64_t* table,
                           int64_t n_gemm, const int32_t* tile_map, const int64_t* slabs,
                           const double* a, int64_t n_a, const double* b, int64_t n_b, double* c, int64_t n_c,
                           void* work, int64_t work_bytes, int64_t n_counters) {
  const int64_t a_chunks = n_counters & 0xFFFFFFFFll, b_chunks = (n_counters >> 32) & 0xFFFFFFFFll;
  if ((a_chunks + b_chunks) * kT2Slab > work_bytes || ((a_chunks + b_chunks) > 0 && !work))
    return cudaErrorInvalidValue;
  if (kind == TNB_TILE_TC_TF32)
    return launch_tc_mode<0>(grid, s, table, n_gemm, tile_map, slabs, a, n_a, b, n_b, c, n_c, work,
                             work_bytes, a_chunks, b_chunks);
  return launch_tc_mode<1>(grid, s, table, n_gemm, tile_map, slabs, a, n_a, b, n_b, c, n_c, work,
                           work_bytes, a_chunks, b_chunks);
}

}  // namespace tnb
