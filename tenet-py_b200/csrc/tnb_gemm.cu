// K2: grouped FP64 GEMM over the uneven coupled sectors of one composition.
//
// `compose` in the reference is one `ar.do("matmul", A_c, B_c)` per coupled sector c,
// with zeros for a sector carried by one operand only (ops/map.py:155-172).  Here every
// sector of a composition is one row of a descriptor table and the whole set runs in one
// launch: CTA b reads its (sector, tile) from a tile -> row map, so large and small
// sectors share the machine in a single wave instead of one launch each.
//
// Tile shapes, chosen by the host per composition:
//   TNB_TILE_64     64x64 output tile, 128 threads
//   TNB_TILE_32     32x32 output tile, 128 threads -- for compositions whose 64x64 tiles
//                   would not fill the 148 SMs (small M, N, long K)
//   TNB_TILE_SKINNY one thread per output row, for products with N <= 16 and K <= 16
//                   (the MPO links of a matvec: tall, 1-3 columns), B staged in shared
//                   memory; bandwidth-bound by construction
//   TNB_TILE_WIDE   a thread per output column (two for K <= 4), for products with M <= 16
//                   and K <= 16 (an MPO tensor as the left operand: a few rows, a long N)
#include <string>

#include "tnb_stages.cuh"

namespace tnb {

// The tiled kinds run on the FP64 tensor cores: mma.sync m16n8k8 (the tcgen05 unit has no
// FP64 kind), four warps per tile.  One instruction is 1,024 fused multiply-adds, 64 clocks of
// its scheduler's FP64 pipe, and a single dependent chain of them per warp already fills the
// pipe (8.5 of 9.2 TFLOP/s per scheduler over the chip), so four warps saturate an SM and
// 56 of 64 issue slots stay free for the loads.  The 4 x 4 register tiles of DFMAs that ran
// here took eight 64-bit shared loads per 16 multiply-adds and topped out at 14-16 TFLOP/s.
// Measured on B200: 4096^3 33.2 TFLOP/s (16.4 with DFMA tiles; cuBLAS DGEMM 35.5), a dense
// U(1) contraction's 1,466 tiles 29.4 (14.4), 3,520 products of about 108 x 82 x 24 8.7 (6.2,
// then bound by writing C), 95 MFLOP in 335 tiles 8.9 us (17.0).
//
// Each element's products are added in k order in one chain of fused multiply-adds, as
// before: the same bits (the instruction adds its eight products one after the other).
//
// Shared memory: A rows padded to 20 doubles, B rows to TN + 4, so the four k x eight rows (or
// columns) of a fragment load fall on 32 different banks per half warp.  K slabs of 16 arrive
// by cp.async, kMmaStages - 1 ahead; all threads read the tile's descriptor row themselves
// (one broadcast load each, no barrier before the first copy).
constexpr int kMmaThreads = 128, kMmaStages = 3, kMmaPadA = kBk + 4;

template <int TM, int TN>
struct MmaSmem {
  double As[kMmaStages][TM][kMmaPadA];
  double Bs[kMmaStages][kBk][TN + 4];
  int last;
};

__device__ __forceinline__ void mma_f64(double (&c)[4], const double (&a)[4],
                                        const double (&b)[2]) {
  asm volatile(
      "mma.sync.aligned.m16n8k8.row.col.f64.f64.f64.f64 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+d"(c[0]), "+d"(c[1]), "+d"(c[2]), "+d"(c[3])
      : "d"(a[0]), "d"(a[1]), "d"(a[2]), "d"(a[3]), "d"(b[0]), "d"(b[1]));
}

// The fragments of a finished tile (or K split of one) into C.  Element e of fragment (i, j) of
// a warp: row 16 i + lane / 4 + 8 (e / 2), column 8 j + 2 (lane % 4) + e % 2 of its part.
template <int TM, int TN>
__device__ __forceinline__ void flush_tile(const GemmArgs& g, const GemmRow& r, int64_t t2,
                                           int64_t split, int64_t m0, int64_t n0,
                                           double (&acc)[TM / 32][TN / 16][4],
                                           MmaSmem<TM, TN>& sm) {
  constexpr int FM = TM / 32, FN = TN / 16;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = (warp >> 1) * (TM / 2), wn = (warp & 1) * (TN / 2), fr = lane >> 2,
            fk = lane & 3;
  if (r.splits > 1) {
    // split K: park this partial tile, and let the last of the tile's splits to arrive
    // sum all of them in split order (a fixed order, so the result is deterministic)
    double* mine = g.parts + r.part_off + (t2 * r.splits + split) * (TM * TN);
#pragma unroll
    for (int i = 0; i < FM; ++i)
#pragma unroll
      for (int j = 0; j < FN; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          mine[(wm + 16 * i + fr + 8 * (e >> 1)) * TN + wn + 8 * j + 2 * fk + (e & 1)] =
              acc[i][j][e];
    __threadfence();
    __syncthreads();
    if (tid == 0) {
      const unsigned int prev = atomicAdd(g.counters + r.cnt_off + t2, 1u);
      sm.last = (prev == static_cast<unsigned int>(r.splits - 1));
    }
    __syncthreads();
    if (!sm.last) return;
    __threadfence();
    const double* base = g.parts + r.part_off + t2 * r.splits * (TM * TN);
    // splits outermost: each element sums its splits in split order from zero, and one
    // split's loads are in flight together
#pragma unroll
    for (int i = 0; i < FM; ++i)
#pragma unroll
      for (int j = 0; j < FN; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0;
    for (int64_t q = 0; q < r.splits; ++q) {
      double v[FM][FN][4];
#pragma unroll
      for (int i = 0; i < FM; ++i)
#pragma unroll
        for (int j = 0; j < FN; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            v[i][j][e] = __ldcg(base + q * (TM * TN) + (wm + 16 * i + fr + 8 * (e >> 1)) * TN +
                                wn + 8 * j + 2 * fk + (e & 1));
#pragma unroll
      for (int i = 0; i < FM; ++i)
#pragma unroll
        for (int j = 0; j < FN; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e) acc[i][j][e] += v[i][j][e];
    }
    if (tid == 0) g.counters[r.cnt_off + t2] = 0u;  // leave the counters zero for the next run
  }
  // through shared memory, so that a store instruction writes 32 consecutive columns of a row
  // (a fragment holds pairs of columns of eight rows: stored directly, half of each 32-byte
  // sector a time)
  constexpr int kPitch = TN + 4;
  static_assert(TM * kPitch <= kMmaStages * (TM * kMmaPadA + kBk * kPitch),
                "the tile fits the drained slabs");
  double* const stage = &sm.As[0][0][0];
  __syncthreads();  // every warp is done with the last slab
#pragma unroll
  for (int i = 0; i < FM; ++i)
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int j = 0; j < FN; ++j)
        *reinterpret_cast<double2*>(stage + (wm + 16 * i + fr + 8 * h) * kPitch + wn + 8 * j +
                                    2 * fk) = make_double2(acc[i][j][2 * h], acc[i][j][2 * h + 1]);
  __syncthreads();
  double* const pc = g.c + r.coff + m0 * r.ldc + n0;
  const int rows = static_cast<int>(min(r.M - m0, int64_t(TM)));
  const int cols = static_cast<int>(min(r.N - n0, int64_t(TN)));
  for (int row = warp; row < rows; row += kMmaThreads / 32)
#pragma unroll
    for (int c = 0; c < TN; c += 32)
      if (c + lane < cols) pc[row * r.ldc + c + lane] = stage[row * kPitch + c + lane];
}

// One TM x TN output tile, or one K split of it, by a CTA of four warps in a 2 x 2 grid.
template <int TM, int TN>
__global__ void __launch_bounds__(kMmaThreads, (TM == 64 ? 3 : 6))
gemm_f64_kernel(const GemmArgs g) {
  extern __shared__ __align__(16) uint8_t gemm_smem[];
  auto& sm = *reinterpret_cast<MmaSmem<TM, TN>*>(gemm_smem);
  constexpr int WM = TM / 2, WN = TN / 2;        // a warp's part of the tile
  constexpr int FM = WM / 16, FN = WN / 8;       // its m16 x n8 fragments
  constexpr int LA = TM * kBk / kMmaThreads, LB = TN * kBk / kMmaThreads;
  constexpr int RA = kMmaThreads / kBk, RB = kMmaThreads / TN;  // rows per round of copies
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int64_t tile = blockIdx.x;
  GemmRow r;
  bool ok = load_row(g, tile, r);
  ok = ok && footprint_ok(r, g.n_a, g.n_b, g.n_c);
  if (ok && r.splits > 1) {
    const int64_t nt = ((r.M + TM - 1) / TM) * r.tiles_n;
    ok = r.ksplit > 0 && r.ksplit % kBk == 0 && r.cnt_off >= 0 && r.cnt_off + nt <= g.n_cnt &&
         r.part_off >= 0 && r.part_off + nt * r.splits * TM * TN <= g.n_parts;
  }
  if (!ok) {
    if (tid == 0) raise_bounds();
    return;
  }
  // (a row's tiles are counted in 32 bits: the grid is; 64-bit divisions cost as much as the
  // tile's multiply-adds)
  const int64_t local = tile - r.tile_begin;
  if (local < 0 || r.splits > INT32_MAX || r.tiles_n < 1 || r.tiles_n > INT32_MAX) {
    if (tid == 0) raise_bounds();
    return;
  }
  uint32_t t2 = static_cast<uint32_t>(local), split = 0;
  if (r.splits > 1) {
    split = t2 % static_cast<uint32_t>(r.splits);
    t2 /= static_cast<uint32_t>(r.splits);
  }
  const uint32_t trow = t2 / static_cast<uint32_t>(r.tiles_n);
  const int64_t m0 = static_cast<int64_t>(trow) * TM;
  const int64_t n0 = static_cast<int64_t>(t2 - trow * static_cast<uint32_t>(r.tiles_n)) * TN;
  if (m0 >= r.M || n0 >= r.N) return;
  const int64_t kb = r.splits > 1 ? split * r.ksplit : 0;
  const int64_t ke = r.splits > 1 ? min(r.K, kb + r.ksplit) : r.K;
  const int kn = ke > kb ? static_cast<int>(min(ke - kb, int64_t(INT32_MAX - kBk))) : 0;
  const int nk = (kn + kBk - 1) / kBk;

  // this thread's copies: A element (ar + RA q, ac), B element (br + RB q, bc) of a slab
  const int ar = tid / kBk, ac = tid % kBk, br = tid / TN, bc = tid % TN;
  const double* const pa = g.a + r.aoff + (m0 + ar) * r.lda + kb + ac;
  const double* const pb = g.b + r.boff + (kb + br) * r.ldb + n0 + bc;
  const int64_t stepa = RA * r.lda, stepb = RB * r.ldb;
  const int rows = static_cast<int>(min(r.M - m0, int64_t(TM)));
  const int cols = static_cast<int>(min(r.N - n0, int64_t(TN)));
  const int rows_left = rows - ar;
  const bool b_in = bc < cols;
  auto issue = [&](int s, int buf) {
    const int k0 = s * kBk;
    const bool a_in = k0 + ac < kn;
#pragma unroll
    for (int q = 0; q < LA; ++q) {
      const bool in = a_in && RA * q < rows_left;
      cp_async8(&sm.As[buf][ar + RA * q][ac], in ? pa + k0 + q * stepa : g.a, in);
    }
#pragma unroll
    for (int q = 0; q < LB; ++q) {
      const bool in = b_in && k0 + br + RB * q < kn;
      cp_async8(&sm.Bs[buf][br + RB * q][bc], in ? pb + k0 * r.ldb + q * stepb : g.b, in);
    }
  };
  double acc[FM][FN][4];
#pragma unroll
  for (int i = 0; i < FM; ++i)
#pragma unroll
    for (int j = 0; j < FN; ++j)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][j][e] = 0.0;

  pdl_wait();  // A may be the previous kernel's output
#pragma unroll
  for (int s = 0; s < kMmaStages - 1; ++s) {
    if (s < nk) issue(s, s);
    cp_async_commit();
  }
  const int wm = (warp >> 1) * WM, wn = (warp & 1) * WN, fr = lane >> 2, fk = lane & 3;
  int buf = 0;
  for (int s = 0; s < nk; ++s) {
    cp_async_wait<kMmaStages - 2>();  // this thread's copies of slab s have landed
    __syncthreads();                  // everyone's have, and slab s - 1 is consumed
    // (a last slab of up to eight takes one step, a warp past the tile's edge none)
    const int steps = wm >= rows || wn >= cols ? 0 : (kn - s * kBk > 8 ? 2 : 1);
    auto fragments = [&](int h, double (&fa)[FM][4], double (&fb)[FN][2]) {
#pragma unroll
      for (int i = 0; i < FM; ++i) {
        const double* p = &sm.As[buf][wm + 16 * i + fr][8 * h + fk];
        fa[i][0] = p[0];
        fa[i][1] = p[8 * kMmaPadA];
        fa[i][2] = p[4];
        fa[i][3] = p[8 * kMmaPadA + 4];
      }
#pragma unroll
      for (int j = 0; j < FN; ++j) {
        const double* p = &sm.Bs[buf][8 * h + fk][wn + 8 * j + fr];
        fb[j][0] = p[0];
        fb[j][1] = p[4 * (TN + 4)];
      }
    };
    auto multiply = [&](const double (&fa)[FM][4], const double (&fb)[FN][2]) {
#pragma unroll
      for (int i = 0; i < FM; ++i)
#pragma unroll
        for (int j = 0; j < FN; ++j) mma_f64(acc[i][j], fa[i], fb[j]);
    };
    auto ahead = [&]() {
      if (s + kMmaStages - 1 < nk) issue(s + kMmaStages - 1, buf == 0 ? kMmaStages - 1 : buf - 1);
      cp_async_commit();
    };
    // 64-wide tiles issue the next slab's copies behind the first step's multiply-adds: with
    // two or three warps on a scheduler the pipe would idle through that address arithmetic
    // (dense 8 GF: 280 -> 273 us, 4096^3 32.6 -> 33.2 TFLOP/s). With up to six warps of
    // 32-wide tiles another warp fills the gap and the earlier copy is worth more (512^3
    // 18.8 us this way round, 21.7 the other).
    double fa[FM][4], fb[FN][2];
    if constexpr (TM == 32) ahead();
    if (steps > 0) {
      fragments(0, fa, fb);
      multiply(fa, fb);
    }
    if constexpr (TM == 64) ahead();
    if (steps > 1) {
      fragments(1, fa, fb);
      multiply(fa, fb);
    }
    buf = buf + 1 == kMmaStages ? 0 : buf + 1;
  }
  cp_async_wait<0>();

  flush_tile<TM, TN>(g, r, t2, split, m0, n0, acc, sm);
}

template <int TM, int TN>
cudaError_t launch_gemm_f64(unsigned grid, cudaStream_t s, const GemmArgs& g) {
  constexpr size_t kSmem = sizeof(MmaSmem<TM, TN>);
  static PerDeviceOnce opted;
  const cudaError_t e = opted.once([] {
    return cudaFuncSetAttribute(gemm_f64_kernel<TM, TN>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem);
  });
  if (e != cudaSuccess) return e;
  return launch_dyn(gemm_f64_kernel<TM, TN>, grid, kMmaThreads, kSmem, s, g);
}

__global__ void __launch_bounds__(kSkinnyThreads, 4)
gemm_f64_skinny_kernel(const GemmArgs g) {
  __shared__ SkinnySmem sm;
  skinny_tile<kSkinnyThreads, false>(g, blockIdx.x, sm, threadIdx.x, CtaSync{});
}

// kSkinnyThreads output columns, C[:, n] = A * B[:, n] for M, K <= 16 (the transpose of the
// skinny case: a few rows, a long N); loads of B and stores of C run along N, so both are
// coalesced.  Bound by HBM, and in a few waves by the chain of loads and sums of one CTA, so
// the tile's threads and the form of its sums go by the product:
//   K <= 4, M <= 4  A from broadcast loads, nothing staged: the
//            descriptor row is one round of loads and B's columns the next, and two columns a
//            thread at 48 registers keep ten CTAs on an SM;
//   K <= 16  A's rows in shared memory, padded with zeros to 4, 8, 12 or 16, one column after
//            the other;
//   K > 8 and M > 8  the FP64 tensor cores, eight columns a warp at a time.
// Each element is one chain of fused multiply-adds over k in all of them: the same bits.
//
// Threads per tile of 256 columns (builds of the one kernel): 256 up to four tiles an SM, where
// all CTAs run at once and one column a thread is the shortest chain; 128, two columns a
// thread, ten CTAs an SM, beyond; between five and eight tiles an SM with 64 registers instead
// of 48, since ten CTAs are not to be had there.
// Device times in us, before (a thread per column, A staged behind two barriers) / now: 2,020
// tiles M = 4 K = 4 10.3 / 5.7, M = 1 K = 16 8.9 / 7.7, M = 16 K = 16 30.4 / 27; 40 tiles M = 16
// K = 16 3.5 / 2.7, M = 4 K = 4 1.9 / 1.7; 760 tiles, the worst, M = 8 K = 14 7.3 / 8.6.  (Two
// passes of one column over K > 4 with A from broadcast loads took 59 us and 14.)  768 products
// of up to 4 x 25,790 x 4 (474 MB) 94.6 us, 5.0 TB/s (240 before).
template <int KM, int NT>
__device__ __forceinline__ void wide_columns(const GemmArgs& g, const GemmRow& r, int64_t n) {
  constexpr int NC = kSkinnyThreads / NT;
  const int M = static_cast<int>(r.M), K = static_cast<int>(r.K);
  const double* const pb = g.b + r.boff + n;
  double bv[NC][KM];
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int k = 0; k < KM; ++k)
      bv[c][k] = k < K && n + c * NT < r.N ? __ldg(pb + c * NT + k * r.ldb)
                                                     : 0.0;
  const double* const pa = g.a + r.aoff;
  double* const pc = g.c + r.coff + n;
#pragma unroll 1
  for (int m = 0; m < M; ++m) {
    double s[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) s[c] = 0.0;
#pragma unroll
    for (int k = 0; k < KM; ++k)
      if (k < K) {
        const double av = __ldg(pa + m * r.lda + k);
#pragma unroll
        for (int c = 0; c < NC; ++c) s[c] = fma(av, bv[c][k], s[c]);
      }
#pragma unroll
    for (int c = 0; c < NC; ++c)
      if (n + c * NT < r.N) pc[m * r.ldc + c * NT] = s[c];
  }
}

template <int KM, int NT>
__device__ __forceinline__ void wide_staged(const GemmArgs& g, const GemmRow& r, int64_t n0,
                                            double* sa) {
  const int M = static_cast<int>(r.M), K = static_cast<int>(r.K);
  for (int i = threadIdx.x; i < M * KM; i += NT)
    sa[i] = i % KM < K ? __ldg(g.a + r.aoff + (i / KM) * r.lda + (i % KM)) : 0.0;
  __syncthreads();
#pragma unroll 1
  for (int c = 0; c < kSkinnyThreads / NT; ++c) {
    const int64_t n = n0 + c * NT;
    if (n >= r.N) return;
    const double* pb = g.b + r.boff + n;
    double bv[KM];
#pragma unroll
    for (int k = 0; k < KM; ++k) bv[k] = k < K ? __ldg(pb + k * r.ldb) : 0.0;
    double* pc = g.c + r.coff + n;
#pragma unroll 2
    for (int m = 0; m < M; ++m, pc += r.ldc) {
      const double2* a = reinterpret_cast<const double2*>(sa + m * KM);
      double s = 0.0;
#pragma unroll
      for (int k = 0; k < KM; k += 2) {
        const double2 v = a[k / 2];
        s = fma(v.x, bv[k], s);
        s = fma(v.y, bv[k + 1], s);
      }
      *pc = s;
    }
  }
}

// (m8n8k4: ptxas takes no larger FP64 shape under the 48 registers of the many-wave build)
__device__ __forceinline__ void mma_f64_k4(double (&c)[2], double a, double b) {
  asm volatile(
      "mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
}

template <int NT>
__device__ __forceinline__ void wide_mma(const GemmArgs& g, const GemmRow& r, int64_t tile0) {
  constexpr int kCols = kSkinnyThreads / (NT / 32);  // a warp's columns
  const int M = static_cast<int>(r.M), K = static_cast<int>(r.K);
  const int lane = threadIdx.x & 31, fr = lane >> 2, fk = lane & 3;
  const int64_t n = tile0 + (threadIdx.x >> 5) * kCols;
  const int left = static_cast<int>(min(r.N - n, int64_t(kCols)));  // columns to do
  if (left <= 0) return;
  double fa[4][2], fb[4];
#pragma unroll
  for (int h = 0; h < 4; ++h)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int row = fr + 8 * e, k = 4 * h + fk;
      fa[h][e] = row < M && k < K ? __ldg(g.a + r.aoff + row * r.lda + k) : 0.0;
    }
  const double* pb = g.b + r.boff + n + fr + fk * r.ldb;
  auto load = [&](int c) {
#pragma unroll
    for (int h = 0; h < 4; ++h)
      fb[h] = c + fr < left && 4 * h + fk < K ? __ldg(pb + c + 4 * h * r.ldb) : 0.0;
  };
  double* const pc = g.c + r.coff + n + 2 * fk + fr * r.ldc;
  const bool pairs = (reinterpret_cast<uintptr_t>(pc) & 15) == 0 && (r.ldc & 1) == 0;
  load(0);
#pragma unroll 1
  for (int c = 0; c < left; c += 8) {
    double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}}, now[4];
#pragma unroll
    for (int h = 0; h < 4; ++h) now[h] = fb[h];
    if (c + 8 < left) load(c + 8);
#pragma unroll
    for (int h = 0; h < 4; ++h) {
      mma_f64_k4(acc[0], fa[h][0], now[h]);
      if (M > 8) mma_f64_k4(acc[1], fa[h][1], now[h]);
    }
    const int room = left - c - 2 * fk;  // of this lane's two columns
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      if (fr + 8 * h >= M) continue;
      double* const p = pc + c + 8 * h * r.ldc;
      if (pairs && room >= 2) {
        *reinterpret_cast<double2*>(p) = make_double2(acc[h][0], acc[h][1]);
      } else {
        if (room > 0) p[0] = acc[h][0];
        if (room > 1) p[1] = acc[h][1];
      }
    }
  }
}

template <int NT, int kMinBlocks>
__global__ void __launch_bounds__(NT, kMinBlocks)
gemm_f64_wide_kernel(const GemmArgs g) {
  __shared__ __align__(16) double sa[kSkinnyMax * kSkinnyMax];
  const int64_t tile = blockIdx.x;
  GemmRow r;
  if (!load_row(g, tile, r) || !footprint_ok(r, g.n_a, g.n_b, g.n_c) || r.M > kSkinnyMax ||
      r.K > kSkinnyMax || tile < r.tile_begin) {
    if (threadIdx.x == 0) raise_bounds();
    return;
  }
  pdl_wait();  // B may be the previous kernel's output
  const int64_t n0 = (tile - r.tile_begin) * kSkinnyThreads;
  if (r.K <= 4) {
    if (r.M <= 4)
      wide_columns<4, NT>(g, r, n0 + threadIdx.x);
    else
      wide_staged<4, NT>(g, r, n0 + threadIdx.x, sa);
  } else if (r.K <= 8) {
    wide_staged<8, NT>(g, r, n0 + threadIdx.x, sa);
  } else if (r.M > 8) {
    wide_mma<NT>(g, r, n0);
  } else if (r.K <= 12) {
    wide_staged<12, NT>(g, r, n0 + threadIdx.x, sa);
  } else {
    wide_staged<kSkinnyMax, NT>(g, r, n0 + threadIdx.x, sa);
  }
}

int device_sms();

static cudaError_t launch_wide(unsigned grid, cudaStream_t s, const GemmArgs& g) {
  const unsigned sms = static_cast<unsigned>(device_sms());
  if (grid <= 4 * sms)
    return launch(gemm_f64_wide_kernel<kSkinnyThreads, 4>, grid, kSkinnyThreads, s, g);
  if (grid > 5 * sms && grid <= 8 * sms)
    return launch(gemm_f64_wide_kernel<kSkinnyThreads / 2, 8>, grid, kSkinnyThreads / 2, s, g);
  return launch(gemm_f64_wide_kernel<kSkinnyThreads / 2, 10>, grid, kSkinnyThreads / 2, s, g);
}

}  // namespace tnb

extern "C" int tnb_grouped_gemm_f64(const int64_t* gemm_table, int64_t n_gemm,
                                    const int32_t* tile_map, int64_t total_tiles,
                                    int32_t tile_kind, const double* a, int64_t n_a,
                                    const double* b, int64_t n_b, double* c, int64_t n_c,
                                    void* work, int64_t work_bytes, int64_t n_counters,
                                    void* stream) {
  TNB_REQUIRE(n_gemm >= 0 && total_tiles >= 0, "tnb_grouped_gemm_f64: negative size");
  if (n_gemm == 0 || total_tiles == 0) return TNB_OK;
  TNB_REQUIRE(gemm_table != nullptr && tile_map != nullptr && c != nullptr,
              "tnb_grouped_gemm_f64: null table, tile map or C");
  TNB_REQUIRE(total_tiles < (int64_t(1) << 31), "tnb_grouped_gemm_f64: too many tiles");
  const bool tc = tile_kind == TNB_TILE_TC_TF32 || tile_kind == TNB_TILE_TC_3XBF16;
  TNB_REQUIRE(work_bytes >= 0 && n_counters >= 0 && (work_bytes == 0 || work != nullptr),
              "tnb_grouped_gemm_f64: bad work buffer");
  TNB_REQUIRE(tc || tnb::gemm_work_parts_offset(n_counters) <= work_bytes,
              "tnb_grouped_gemm_f64: work buffer too small for its counters");
  TNB_REQUIRE(!tc || ((n_counters & 0xFFFFFFFFll) + (n_counters >> 32)) * 16384 <= work_bytes,
              "tnb_grouped_gemm_f64: work buffer too small for the packed operands");
  auto* counters = static_cast<unsigned int*>(work);
  const int64_t poff = tnb::gemm_work_parts_offset(n_counters);
  double* parts = work_bytes > poff
                      ? reinterpret_cast<double*>(static_cast<char*>(work) + poff) : nullptr;
  const int64_t n_parts = work_bytes > poff ? (work_bytes - poff) / 8 : 0;
  const unsigned grid = static_cast<unsigned>(total_tiles);
  cudaStream_t s = tnb::as_stream(stream);
  cudaError_t e = cudaSuccess;
  const tnb::GemmArgs g{gemm_table, n_gemm, tile_map, a, n_a, b, n_b, c, n_c, counters,
                        n_counters, parts, n_parts};
  switch (tile_kind) {
    case TNB_TILE_64:
      e = tnb::launch_gemm_f64<64, 64>(grid, s, g);
      break;
    case TNB_TILE_32:
      e = tnb::launch_gemm_f64<32, 32>(grid, s, g);
      break;
    case TNB_TILE_SKINNY:
      e = tnb::launch(tnb::gemm_f64_skinny_kernel, grid, tnb::kSkinnyThreads, s, g);
      break;
    case TNB_TILE_WIDE:
      e = tnb::launch_wide(grid, s, g);
      break;
    case TNB_TILE_TC_TF32:
    case TNB_TILE_TC_3XBF16:
      e = tnb::launch_gemm_tc(tile_kind, grid, s, gemm_table, n_gemm, tile_map, nullptr, a, n_a,
                              b, n_b, c, n_c, work, work_bytes, n_counters);
      break;
    default:
      tnb::set_error("tnb_grouped_gemm_f64: unknown tile kind");
      return TNB_EINVAL;
  }
  if (e != cudaSuccess) {
    tnb::set_error(std::string("tnb_grouped_gemm_f64: ") + cudaGetErrorString(e));
    return TNB_ECUDA;
  }
  return tnb::check_launch("tnb_grouped_gemm_f64");
}

extern "C" int tnb_grouped_gemm_f64_rows(const int64_t* tile_rows, int64_t total_tiles,
                                         int32_t tile_kind, const double* a, int64_t n_a,
                                         const double* b, int64_t n_b, double* c, int64_t n_c,
                                         void* work, int64_t work_bytes, int64_t n_counters,
                                         void* stream) {
  TNB_REQUIRE(total_tiles >= 0, "tnb_grouped_gemm_f64_rows: negative size");
  if (total_tiles == 0) return TNB_OK;
  TNB_REQUIRE(tile_rows != nullptr && c != nullptr, "tnb_grouped_gemm_f64_rows: null rows or C");
  TNB_REQUIRE(total_tiles < (int64_t(1) << 31), "tnb_grouped_gemm_f64_rows: too many tiles");
  TNB_REQUIRE(tile_kind == TNB_TILE_64 || tile_kind == TNB_TILE_32 ||
                  tile_kind == TNB_TILE_SKINNY || tile_kind == TNB_TILE_WIDE,
              "tnb_grouped_gemm_f64_rows: FP64 tile kinds only");
  TNB_REQUIRE(work_bytes >= 0 && n_counters >= 0 && (work_bytes == 0 || work != nullptr) &&
                  tnb::gemm_work_parts_offset(n_counters) <= work_bytes,
              "tnb_grouped_gemm_f64_rows: bad work buffer");
  auto* counters = static_cast<unsigned int*>(work);
  const int64_t poff = tnb::gemm_work_parts_offset(n_counters);
  double* parts = work_bytes > poff
                      ? reinterpret_cast<double*>(static_cast<char*>(work) + poff) : nullptr;
  const int64_t n_parts = work_bytes > poff ? (work_bytes - poff) / 8 : 0;
  const unsigned grid = static_cast<unsigned>(total_tiles);
  cudaStream_t s = tnb::as_stream(stream);
  const tnb::GemmArgs g{nullptr, total_tiles, nullptr, a, n_a, b, n_b, c, n_c, counters,
                        n_counters, parts, n_parts, tile_rows};
  cudaError_t e = cudaSuccess;
  switch (tile_kind) {
    case TNB_TILE_64:
      e = tnb::launch_gemm_f64<64, 64>(grid, s, g);
      break;
    case TNB_TILE_32:
      e = tnb::launch_gemm_f64<32, 32>(grid, s, g);
      break;
    case TNB_TILE_SKINNY:
      e = tnb::launch(tnb::gemm_f64_skinny_kernel, grid, tnb::kSkinnyThreads, s, g);
      break;
    default:
      e = tnb::launch_wide(grid, s, g);
      break;
  }
  if (e != cudaSuccess) {
    tnb::set_error(std::string("tnb_grouped_gemm_f64_rows: ") + cudaGetErrorString(e));
    return TNB_ECUDA;
  }
  return tnb::check_launch("tnb_grouped_gemm_f64_rows");
}

extern "C" int tnb_grouped_gemm_tc(const int64_t* gemm_table, int64_t n_gemm,
                                   const int32_t* tile_map, int64_t total_tiles,
                                   const int64_t* slab_rows, int32_t tile_kind, const double* a,
                                   int64_t n_a, const double* b, int64_t n_b, double* c,
                                   int64_t n_c, void* work, int64_t work_bytes,
                                   int64_t n_counters, void* stream) {
  TNB_REQUIRE(n_gemm >= 0 && total_tiles >= 0, "tnb_grouped_gemm_tc: negative size");
  if (n_gemm == 0 || total_tiles == 0) return TNB_OK;
  TNB_REQUIRE(gemm_table != nullptr && tile_map != nullptr && c != nullptr,
              "tnb_grouped_gemm_tc: null table, tile map or C");
  TNB_REQUIRE(total_tiles < (int64_t(1) << 31), "tnb_grouped_gemm_tc: too many tiles");
  TNB_REQUIRE(tile_kind == TNB_TILE_TC_TF32 || tile_kind == TNB_TILE_TC_3XBF16,
              "tnb_grouped_gemm_tc: tensor-core tile kinds only");
  const int64_t n_slabs = (n_counters & 0xFFFFFFFFll) + (n_counters >> 32);
  TNB_REQUIRE(work_bytes >= 0 && n_counters >= 0 && (work_bytes == 0 || work != nullptr) &&
                  n_slabs * 16384 <= work_bytes && (n_slabs == 0 || slab_rows != nullptr),
              "tnb_grouped_gemm_tc: bad work buffer or slab rows");
  const cudaError_t e = tnb::launch_gemm_tc(
      tile_kind, static_cast<unsigned>(total_tiles), tnb::as_stream(stream), gemm_table, n_gemm,
      tile_map, slab_rows, a, n_a, b, n_b, c, n_c, work, work_bytes, n_counters);
  if (e != cudaSuccess) {
    tnb::set_error(std::string("tnb_grouped_gemm_tc: ") + cudaGetErrorString(e));
    return TNB_ECUDA;
  }
  return tnb::check_launch("tnb_grouped_gemm_tc");
}
