// A whole Lanczos solve of a small problem in one launch of one CTA.
//
// The stages of a recorded matvec (gathers of warp items, grouped FP64 GEMMs) and the
// recurrence run between CTA barriers, everything in shared memory: the stages' rows, the
// fixed operands, the buffers between the stages and the Krylov vectors at hand; only the
// vectors and the recurrence's state go to global memory.
//
// What bounds it: latency.  On the bonds of a 16-site SU(2) chain a vector has 2 to 194
// elements and a matvec 10 to 7,400 multiply-adds, but launched one by one a step of five
// stages and the recurrence took 9 to 19 us, most of it in starting kernels that each do a
// microsecond of dependent loads; the host needed 14 us to issue it.  Here a step is six
// stages of a few hundred clocks with a barrier each.
//
// Each element of a stage is worked out once, before the first step, into a record of its
// offsets, with every check of the launched stages made there: decoding the items in every step
// took 2,100 to 9,000 clocks a gather, a solve at 194 elements 305 us.
//
// Measured on B200, 20 vectors, from the call to the result read on the host (device times, and
// the rule that takes a matvec here: plan_small in tnb_seq.cu): 26 elements 365 -> 111 us, 134
// elements 399 -> 128, 420 elements 477 -> 203, 617 elements 482 -> 277; a 16-site sweep 28.8 ->
// 20.8 ms.
//
// Same arithmetic as the launches it replaces, in the same order (an element of a product as one
// chain of fused multiply-adds over k, gathers in table order, the recurrence rounded operation
// by operation, its sums as wdot_kernel adds one chunk): the same bits.
#include <string>

#include "tnb_gather_item.cuh"
#include "tnb_lanczos_small.cuh"

namespace tnb {

constexpr int kSmallThreads = 512, kSmallWarps = kSmallThreads / 32;
constexpr int kSumThreads = 256;  // threads that hold a sum's terms (wdot_kernel's)

// Sum of the first kSumThreads threads' `v` as block_sum orders it, valid in every thread.
// `part` is not written again before a barrier.
__device__ __forceinline__ double sum_total(double v, double* part) {
  const int tid = threadIdx.x, lane = tid & 31;
  if (tid < kSumThreads) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) part[tid >> 5] = v;
  }
  __syncthreads();
  v = part[lane & (kSumThreads / 32 - 1)];
#pragma unroll
  for (int o = kSumThreads / 64; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v + 0.0;
}

// The elements a sum's thread adds, in its order: indices, flagged where a run of equal weights
// starts and ends for this thread.
constexpr int kRunFirst = 1 << 15, kRunLast = 1 << 14, kRunIndex = kRunLast - 1;

template <class Term>  // (index) -> the two factors
__device__ __forceinline__ double run_sum(const uint16_t* mine, int count, const double* weight,
                                          Term term) {
  double acc = 0.0, s = 0.0;
#pragma unroll 4
  for (int k = 0; k < count; ++k) {
    const int e = mine[k], i = e & kRunIndex;
    const double2 f = term(i);
    s = fma(f.x, f.y, e & kRunFirst ? 0.0 : s);
    if (e & kRunLast) acc = fma(weight[i], s, acc);
  }
  return acc;
}

// Term i of an item's row: first source element, coefficient, leading dimension.
__device__ __forceinline__ void item_term(const SmallStage& st, const int* row, int i,
                                          int64_t& ts, double& cf, int& tl) {
  if (i == 0) {
    ts = item_i64(row[2], row[3]);
    cf = __hiloint2double(row[5], row[4]);
    tl = row[11];
  } else if (st.width == 64 && i <= kItemInline) {
    const int* r = row + 32 + 5 * (i - 1);
    ts = item_i64(r[0], r[1]);
    cf = __hiloint2double(r[3], r[2]);
    tl = r[4];
  } else {
    ts = __ldg(st.term_src + row[6] + i);
    cf = __ldg(st.term_coeff + row[6] + i);
    const int64_t ld = __ldg(st.term_ld + row[6] + i);
    tl = static_cast<int>(ld);
    if (ld != tl) ts = -1;
  }
}

// The checks tnb_block_gather_items makes of an item, by one thread.
__device__ bool item_ok(const SmallStage& st, const int* row) {
  const int base = row[8], n = row[9], rank = row[10] & 255;
  if (rank < 1 || rank > kItemMaxRank || ((row[10] >> 8) & 1) || n <= 0 || n > kItemMax ||
      base < 0 || row[6] < 0 || row[7] < row[6] || row[7] > st.n_term)
    return false;
  // row and column offsets of an item of several terms are kept in 16 bits each
  int64_t total = 1, lo = item_i64(row[0], row[1]), hi = lo;
  int64_t r_lo = 0, r_hi = 0, c_lo = 0, c_hi = 0;
  for (int d = 0; d < rank; ++d) {
    if (row[12 + d] <= 0) return false;
    total *= row[12 + d];
    if (total >= (int64_t(1) << 31)) return false;
    const int64_t x = static_cast<int64_t>(row[12 + d] - 1) * row[20 + d];
    lo += x < 0 ? x : 0;
    hi += x > 0 ? x : 0;
    const int64_t r = static_cast<int64_t>(row[12 + d] - 1) * row[24 + d];
    const int64_t c = static_cast<int64_t>(row[12 + d] - 1) * row[28 + d];
    (r < 0 ? r_lo : r_hi) += r;
    (c < 0 ? c_lo : c_hi) += c;
  }
  if (base + n > total || lo < 0 || hi >= st.n_dst) return false;
  if (row[7] - row[6] > 1 && (r_lo < INT16_MIN || r_hi > INT16_MAX || c_lo < INT16_MIN ||
                              c_hi > INT16_MAX))
    return false;
  for (int i = 0; i < row[7] - row[6]; ++i) {
    int64_t ts;
    double cf;
    int tl;
    item_term(st, row, i, ts, cf, tl);
    lo = hi = ts;
    for (int d = 0; d < rank; ++d) {
      const int64_t x = static_cast<int64_t>(row[12 + d] - 1) *
                        (static_cast<int64_t>(tl) * row[24 + d] + row[28 + d]);
      lo += x < 0 ? x : 0;
      hi += x > 0 ? x : 0;
    }
    if (lo < 0 || hi >= st.n_src) return false;
  }
  return true;
}

// A gathered element: its offset in shared memory and its first term's, how many terms and whose
// item.  Offsets fit 16 bits (kSmallMaxSmem); eight bytes an element and four more for several
// terms, with coefficients and lengths left in the rows, reach 617 elements a vector where
// records that held them too ended at 420.
struct __align__(8) SmallMove {
  uint16_t dst, src, terms, item;
};
// An element of a product: where its row of A, its column of B and itself lie, and its row.
struct __align__(8) SmallDot {
  uint16_t a, b, dst, row;
};
static_assert(sizeof(SmallMove) == 8 && sizeof(SmallDot) == 8, "records of 8 bytes");

__global__ void __launch_bounds__(kSmallThreads, 1)
lanczos_small_kernel(const __grid_constant__ SmallArgs g) {
  extern __shared__ __align__(16) unsigned char small_smem[];
  __shared__ double part[2][kSumThreads / 32];
  __shared__ int cursor;
  __shared__ int outs[kSmallMaxStages];               // elements of each stage
  __shared__ int first[kSmallMaxStages][kSmallMaxRows];  // of each item or product, -1: refused
  double* const sm = reinterpret_cast<double*>(small_smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = g.n, ncv = g.ncv;
  if (tid == 0) cursor = 0;

  // tables, fixed operands and the start vector
  for (int i = 0; i < g.n_bufs; ++i) {
    const SmallBuf& b = g.buf[i];
    for (int k = tid; k < b.n; k += kSmallThreads) sm[b.at + k] = b.from[k];
  }
  double* const weight = sm + g.weight;
  for (int i = tid; i < n; i += kSmallThreads) {
    int lo = 0, hi = g.n_runs - 1;  // the element's run
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (g.run_start[mid] <= i) lo = mid; else hi = mid - 1;
    }
    weight[i] = g.run_start[lo] <= i && i < g.run_start[lo + 1] ? g.run_w[lo] : 0.0;
    sm[g.x + i] = g.x0[i];
    sm[g.y + i] = 0.0;
  }
  for (int s = 0; s < g.n_stages; ++s) {
    const SmallStage& st = g.st[s];
    if (st.gather) {
      int* const rows = reinterpret_cast<int*>(small_smem + st.rows_at);
      const int* from = static_cast<const int*>(st.rows);
      for (int k = tid; k < st.width * st.count; k += kSmallThreads) rows[k] = from[k];
    }
  }
  for (int k = tid; k < 3 * ncv + 2; k += kSmallThreads) g.state[k] = 0.0;
  __syncthreads();
  // this thread's terms of a sum: elements a + tid, a + tid + kSumThreads, ... of every run
  uint16_t* mine = reinterpret_cast<uint16_t*>(small_smem + g.order_at);
  int terms = 0;
  if (tid < kSumThreads) {
    auto each = [&](auto&& use) {
      for (int r = 0; r < g.n_runs; ++r) {
        const int64_t a = __ldg(g.run_start + r), b = min(int64_t(n), __ldg(g.run_start + r + 1));
        if (a >= n) break;
        for (int64_t i = a < 0 ? b : a + tid; i < b; i += kSumThreads)
          use(static_cast<int>(i), i == a + tid, i + kSumThreads >= b);
      }
    };
    each([&](int, bool, bool) { ++terms; });
    const int at = atomicAdd(&cursor, terms);
    if (at + terms > n) {  // runs that overlap: no room for their terms
      if (terms > 0) raise_bounds();
      terms = 0;
    }
    mine += at;
    int k = 0;
    if (terms > 0)
      each([&](int i, bool head, bool tail) {
        mine[k++] = static_cast<uint16_t>(i | (head ? kRunFirst : 0) | (tail ? kRunLast : 0));
      });
  }
  for (int s = 0; s < g.n_stages; ++s) {  // each item's and product's elements, 0 where refused
    const SmallStage& st = g.st[s];
    for (int k = tid; k < st.count; k += kSmallThreads) {
      bool ok;
      int64_t elems = 0;
      if (st.gather) {
        const int* row = reinterpret_cast<const int*>(small_smem + st.rows_at) + k * st.width;
        ok = item_ok(st, row);
        elems = row[9];
      } else {
        const int64_t* t = static_cast<const int64_t*>(st.rows) + k * TNB_GEMM_WIDTH;
        const int64_t M = t[0], N = t[1], K = t[2];
        ok = M >= 0 && N >= 0 && K >= 0 && M <= st.n_dst && N <= st.n_dst;
        elems = ok ? M * N : 0;
        if (ok && elems > 0) {
          ok = elems <= st.n_dst && t[7] >= 0 && t[8] >= 0 && t[7] + (M - 1) * t[8] + N <= st.n_dst;
          if (K > 0)
            ok = ok && t[3] >= 0 && t[5] >= 0 && t[4] >= 0 && t[6] >= 0 &&
                 t[3] + (M - 1) * t[4] + K <= st.n_src && t[5] + (K - 1) * t[6] + N <= st.n_b;
        }
      }
      if (!ok) raise_bounds();
      first[s][k] = ok ? static_cast<int>(elems) : 0;
    }
  }
  __syncthreads();
  if (tid < g.n_stages) {
    int total = 0;
    for (int k = 0; k < g.st[tid].count; ++k) {
      const int e = first[tid][k];
      // (a table that writes an element twice keeps to what its records have room for)
      const bool fits = total + e <= g.st[tid].n_dst;
      if (!fits) raise_bounds();
      first[tid][k] = fits && e > 0 ? total : -1;
      total += fits ? e : 0;
    }
    outs[tid] = total;
  }
  __syncthreads();
  for (int s = 0; s < g.n_stages; ++s) {
    const SmallStage& st = g.st[s];
    for (int k = warp; k < st.count; k += kSmallWarps) {
      const int at = first[s][k];
      if (at < 0) continue;
      if (st.gather) {
        const int* row = reinterpret_cast<const int*>(small_smem + st.rows_at) + k * st.width;
        SmallMove* const rec = reinterpret_cast<SmallMove*>(small_smem + st.recs_at) + at;
        short2* const split = reinterpret_cast<short2*>(small_smem + st.split_at) + at;
        const int rank = row[10] & 255, terms = row[7] - row[6];
        for (int q = lane; q < row[9]; q += 32) {
          int rem = row[8] + q, to = row[0];
          int64_t rr = 0, cc = 0;
          for (int d = rank - 1; d >= 0; --d) {
            const int quo = d > 0 ? rem / row[12 + d] : 0;
            const int j = rem - quo * row[12 + d];
            rr += static_cast<int64_t>(j) * row[24 + d];
            cc += static_cast<int64_t>(j) * row[28 + d];
            to += j * row[20 + d];
            rem = quo;
          }
          SmallMove m;
          m.dst = static_cast<uint16_t>(st.dst + to);
          m.src = static_cast<uint16_t>(
              terms > 0 ? st.src + item_i64(row[2], row[3]) + row[11] * rr + cc : st.dst);
          m.terms = static_cast<uint16_t>(terms);
          m.item = static_cast<uint16_t>(k);
          rec[q] = m;
          if (st.width == 64) split[q] = make_short2(static_cast<short>(rr), static_cast<short>(cc));
        }
      } else {
        const int64_t* t = static_cast<const int64_t*>(st.rows) + k * TNB_GEMM_WIDTH;
        const int M = static_cast<int>(t[0]), N = static_cast<int>(t[1]), K = static_cast<int>(t[2]);
        SmallDot* const rec = reinterpret_cast<SmallDot*>(small_smem + st.recs_at) + at;
        if (lane == 0)
          reinterpret_cast<int2*>(small_smem + st.rows_at)[k] =
              make_int2(K, K > 1 ? static_cast<int>(t[6]) : 0);
        for (int q = lane; q < M * N; q += 32) {
          const int m = q / N, c = q - m * N;
          SmallDot d;
          d.a = static_cast<uint16_t>(K > 0 ? st.src + t[3] + m * t[4] : 0);
          d.b = static_cast<uint16_t>(K > 0 ? st.b + t[5] + c : 0);
          d.dst = static_cast<uint16_t>(st.dst + t[7] + m * t[8] + c);
          d.row = static_cast<uint16_t>(k);
          rec[q] = d;
        }
      }
    }
  }

  // v_0 = x0 / ||x0||
  double* const x = sm + g.x;
  double* const y = sm + g.y;
  double* const prev = sm + g.prev;
  {
    const double s2 = sum_total(
        run_sum(mine, terms, weight, [&](int i) { return make_double2(x[i], x[i]); }), part[0]);
    const double nrm = sqrt(s2);
    if (tid == 0) g.scal[0] = s2;
    for (int i = tid; i < n; i += kSmallThreads) g.v[i] = x[i] = __ddiv_rn(x[i], nrm);
  }
  double b = 0.0;  // beta of the step before
  for (int j = 0; j < ncv; ++j) {
    __syncthreads();
    for (int s = 0; s < g.n_stages; ++s) {
      const SmallStage& st = g.st[s];
      const int total = outs[s];
      if (st.gather) {
        const SmallMove* rec = reinterpret_cast<const SmallMove*>(small_smem + st.recs_at);
        for (int e = tid; e < total; e += kSmallThreads) {
          const SmallMove m = rec[e];
          const int* row = reinterpret_cast<const int*>(small_smem + st.rows_at) + m.item * st.width;
          double acc = m.terms > 0 ? fma(__hiloint2double(row[5], row[4]), sm[m.src], 0.0) : 0.0;
          if (m.terms > 1) {
            const short2 at = reinterpret_cast<const short2*>(small_smem + st.split_at)[e];
#pragma unroll 2
            for (int i = 1; i < m.terms; ++i) {
              int64_t ts;
              double cf;
              int tl;
              item_term(st, row, i, ts, cf, tl);
              acc = fma(cf, sm[st.src + static_cast<int>(ts) + tl * at.x + at.y], acc);
            }
          }
          sm[m.dst] = acc;
        }
      } else {
        const SmallDot* rec = reinterpret_cast<const SmallDot*>(small_smem + st.recs_at);
        for (int e = tid; e < total; e += kSmallThreads) {
          const SmallDot d = rec[e];
          const int2 len = reinterpret_cast<const int2*>(small_smem + st.rows_at)[d.row];
          const double* pa = sm + d.a;
          const double* pb = sm + d.b;
          double acc = 0.0;
#pragma unroll 8
          for (int i = 0; i < len.x; ++i, pb += len.y) acc = fma(pa[i], *pb, acc);
          sm[d.dst] = acc;
        }
      }
      __syncthreads();
    }
    const double a = sum_total(
        run_sum(mine, terms, weight, [&](int i) { return make_double2(x[i], y[i]); }), part[0]);
    for (int i = tid; i < n; i += kSmallThreads) {
      double t = __dsub_rn(y[i], __dmul_rn(x[i], a));
      if (j > 0) t = __dsub_rn(t, __dmul_rn(prev[i], b));
      y[i] = t;
    }
    __syncthreads();
    const double nrm2 = sum_total(
        run_sum(mine, terms, weight, [&](int i) { return make_double2(y[i], y[i]); }), part[1]);
    const double beta = sqrt(fmax(nrm2, 0.0));
    const bool stop_now = j + 1 == ncv || beta < g.tol;
    if (tid == 0) {
      g.state[j] = a;
      g.state[2 * ncv + j] = nrm2;
      g.state[3 * ncv] = static_cast<double>(stop_now ? j + 1 : j + 2);
      if (stop_now) g.state[3 * ncv + 1] = 1.0; else g.state[ncv + j] = beta;
    }
    if (stop_now) {
      for (int k = j + 1; k <= ncv; ++k)
        for (int i = tid; i < n; i += kSmallThreads) g.v[k * g.ldv + i] = 0.0;
      // (a recurrence that stops early leaves the matvec of a zero vector behind)
      for (int i = tid; i < n; i += kSmallThreads) g.w[i] = j + 1 == ncv ? y[i] : 0.0;
      return;
    }
    for (int i = tid; i < n; i += kSmallThreads) {
      const double t = __ddiv_rn(y[i], beta);
      prev[i] = x[i];
      x[i] = t;
      g.v[(j + 1) * g.ldv + i] = t;
    }
    b = beta;
  }
}

int launch_lanczos_small(const SmallArgs& a, int smem, cudaStream_t stream) {
  static PerDeviceInt ready;
  const int ok = ready.get([](int, int* out) {
    *out = 1;
    return cudaFuncSetAttribute(lanczos_small_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                kSmallMaxSmem);
  });
  if (!ok) {
    set_error("tnb_lanczos_solve: shared memory for a small solve");
    return TNB_ECUDA;
  }
  lanczos_small_kernel<<<1, kSmallThreads, smem, stream>>>(a);
  return check_launch("tnb_lanczos_solve: small solve");
}

}  // namespace tnb
