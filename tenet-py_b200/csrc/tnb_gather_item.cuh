// One item of a block gather from warp items (the kernel that runs tables of them is in
// tnb_gather_items.cu): the row's words, its checks and the move of its elements by one warp.
#pragma once

#include <type_traits>

#include "tnb_common.cuh"

namespace tnb {

constexpr int kItemMax = TNB_ITEM_MAX_ELEMS;  // elements of an item
constexpr int kItemEpl = kItemMax / 32;       // elements per lane
constexpr int kItemMaxRank = 4;
constexpr int kItemInline = 6;                // further terms inline in a 64-word row

struct ItemArgs {
  const int32_t* rows;
  int width;  // words per row: 32 (one term per segment) or 64
  int64_t n_items;
  const int64_t* term_src;
  const double* term_coeff;
  const int64_t* term_ld;
  int64_t n_term;
  const double* src0;
  int64_t n_src0;
  double* dst0;
  int64_t n_dst0;
  const double* src1;
  int64_t n_src1;
  double* dst1;
  int64_t n_dst1;
};

__device__ __forceinline__ int64_t item_i64(int lo, int hi) {
  return static_cast<int64_t>((static_cast<uint64_t>(static_cast<uint32_t>(hi)) << 32) |
                              static_cast<uint32_t>(lo));
}

// Decoded terms of a warp's item.
struct ItemTerms {
  int64_t src[32];
  double coeff[32];
  int ld[32];
};

// Word i of the row whose words 0..31 and 32..63 the lanes hold in w0 and w1.
struct ItemWords {
  int w0, w1;
  __device__ __forceinline__ int operator[](int i) const {
    return __shfl_sync(0xffffffffu, i < 32 ? w0 : w1, i & 31);
  }
};

// One item of rank R.  Every check is made once per item on the segment's whole box: the row's
// division constants and extents, and the box's lowest and highest destination and source
// offsets.  `load` reads a source element.  kSeveral: built for items of several terms (rows of
// 64 words), takes either width; the other takes rows of 32 words, items of several terms among
// them a term and an element at a time, so that its one-term body has the registers to itself
// (one build for both: 674 us for the batched environment update, 639 apart).
template <int R, bool kSeveral, class Load>
__device__ __forceinline__ void gather_item(const ItemArgs& g, const ItemWords& w, int lane,
                                            ItemTerms& terms, Load load) {
  const int base = w[8], n = w[9], meta = w[10], t0 = w[6], t1 = w[7];
  const bool second = ((meta >> 8) & 1) != 0;
  const double* __restrict__ src = second ? g.src1 : g.src0;
  double* __restrict__ dst = second ? g.dst1 : g.dst0;
  const int64_t n_src = second ? g.n_src1 : g.n_src0, n_dst = second ? g.n_dst1 : g.n_dst0;
  const int64_t dst_off = item_i64(w[0], w[1]);
  int dim[R], dstr[R], rstr[R], cstr[R];
  uint32_t mul[R];
  int shr[R];
  int64_t total = 1, d_lo = dst_off, d_hi = dst_off;
  bool ok = n > 0 && n <= kItemMax && base >= 0 && t0 >= 0 && t1 >= t0 && t1 <= g.n_term;
#pragma unroll
  for (int d = 0; d < R; ++d) {
    dim[d] = w[12 + d];
    dstr[d] = w[20 + d];
    rstr[d] = w[24 + d];
    cstr[d] = w[28 + d];
    ok = ok && dim[d] > 0;
    total *= dim[d];
    ok = ok && total < (int64_t(1) << 31);
    const int64_t x = static_cast<int64_t>(dim[d] - 1) * dstr[d];
    d_lo += x < 0 ? x : 0;
    d_hi += x > 0 ? x : 0;
    if (d > 0) {
      // floor(q / dim) = (q mul) >> (31 + l), l = ceil(log2 dim), for q < 2^31 whenever
      // 2^(31+l) <= mul dim < 2^(31+l) + 2^l (Granlund and Montgomery, 1994)
      mul[d] = static_cast<uint32_t>(w[15 + d]);
      shr[d] = (meta >> (11 + 5 * d)) & 31;
      const uint64_t prod = static_cast<uint64_t>(mul[d]) * static_cast<uint32_t>(dim[d]);
      const uint64_t p2 = 1ull << (32 + shr[d]);
      ok = ok && dim[d] > 1 && prod >= p2 && prod - p2 < (2ull << shr[d]);
    }
  }
  ok = ok && base + n <= total && d_lo >= 0 && d_hi < n_dst;
  // a term's source box
  auto inside = [&](int64_t ts, int tl) {
    int64_t lo = ts, hi = ts;
#pragma unroll
    for (int d = 0; d < R; ++d) {
      const int64_t x = static_cast<int64_t>(dim[d] - 1) *
                        (static_cast<int64_t>(tl) * rstr[d] + cstr[d]);
      lo += x < 0 ? x : 0;
      hi += x > 0 ? x : 0;
    }
    return lo >= 0 && hi < n_src;
  };
  if (!ok) {
    if (lane == 0) raise_bounds();
    return;
  }
  // the element's index in each extent, outermost last
  auto split = [&](int q, auto&& use) {
    uint32_t rem = static_cast<uint32_t>(q);
#pragma unroll
    for (int d = R - 1; d > 0; --d) {
      const uint32_t quo = __umulhi(rem, mul[d]) >> shr[d];
      use(d, static_cast<int>(rem - quo * static_cast<uint32_t>(dim[d])));
      rem = quo;
    }
    use(0, static_cast<int>(rem));
  };
  const int64_t ts0 = item_i64(w[2], w[3]);
  const double cf0 = __hiloint2double(w[5], w[4]);
  const int tl0 = w[11];
  if (t1 - t0 == 1) {
    if (!inside(ts0, tl0)) {
      if (lane == 0) raise_bounds();
      return;
    }
    int sstr[R];
#pragma unroll
    for (int d = 0; d < R; ++d) sstr[d] = tl0 * rstr[d] + cstr[d];
    const double* const s = src + ts0;
    double* const o = dst + dst_off;
    double v[kItemEpl];
    int to[kItemEpl];
#pragma unroll
    for (int k = 0; k < kItemEpl; ++k) {
      const int q = lane + 32 * k;
      if (32 * k < n) {  // uniform
        int from = 0;
        to[k] = 0;
        split(base + q, [&](int d, int j) {
          from += j * sstr[d];
          to[k] += j * dstr[d];
        });
        v[k] = q < n ? load(s + from) : 0.0;
      }
    }
#pragma unroll
    for (int k = 0; k < kItemEpl; ++k)
      if (lane + 32 * k < n) o[to[k]] = fma(cf0, v[k], 0.0);
    return;
  }
  const int nt = t1 - t0;
  bool bad = false;
  auto stored = [&](int i, int64_t& ts, double& cf, int& tl) {  // term i from the arrays
    ts = __ldg(g.term_src + t0 + i);
    cf = __ldg(g.term_coeff + t0 + i);
    const int64_t ld = __ldg(g.term_ld + t0 + i);
    tl = static_cast<int>(ld);
    if (ld != tl) ts = -1;  // refused below
  };
  if constexpr (!kSeveral) {
#pragma unroll 1
    for (int q = lane; q < n; q += 32) {
      int rr = 0, cc = 0, to = 0;
      split(base + q, [&](int d, int j) {
        rr += j * rstr[d];
        cc += j * cstr[d];
        to += j * dstr[d];
      });
      double acc = 0.0;
#pragma unroll 1
      for (int i = 0; i < nt; ++i) {
        int64_t ts;
        double cf;
        int tl;
        stored(i, ts, cf, tl);
        const bool in = inside(ts, tl);
        bad = bad || !in;
        acc = fma(cf, in ? load(src + ts + tl * rr + cc) : 0.0, acc);
      }
      dst[dst_off + to] = acc;
    }
    if (bad) raise_bounds();
    return;
  }
  // two terms (or none): both from the row, four elements per lane at a time
  if (nt <= 2) {
    int64_t ts1 = 0;
    double cf1 = 0.0;
    int tl1 = 0;
    if (nt == 2) {
      if (g.width == 64) {
        ts1 = item_i64(w[32], w[33]);
        cf1 = __hiloint2double(w[35], w[34]);
        tl1 = w[36];
      } else {
        stored(1, ts1, cf1, tl1);
      }
    }
    const bool in0 = nt == 2 && inside(ts0, tl0), in1 = nt == 2 && inside(ts1, tl1);
    if (nt == 2 && !(in0 && in1) && lane == 0) raise_bounds();
#pragma unroll 1
    for (int k0 = 0; 32 * k0 < n; k0 += 4) {
      double va[4], vb[4];
      int to[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const int q = lane + 32 * (k0 + k);
        int rr = 0, cc = 0;
        to[k] = 0;
        if (q < n)
          split(base + q, [&](int d, int j) {
            rr += j * rstr[d];
            cc += j * cstr[d];
            to[k] += j * dstr[d];
          });
        va[k] = in0 && q < n ? load(src + ts0 + tl0 * rr + cc) : 0.0;
        vb[k] = in1 && q < n ? load(src + ts1 + tl1 * rr + cc) : 0.0;
      }
#pragma unroll
      for (int k = 0; k < 4; ++k)
        if (lane + 32 * (k0 + k) < n)
          dst[dst_off + to[k]] = nt == 2 ? fma(cf1, vb[k], fma(cf0, va[k], 0.0)) : 0.0;
    }
    return;
  }
  // more terms.  The lanes decode and check up to 32 of them at a time into the
  // warp's shared memory; then E elements per lane at a time, the loads of 8 / E terms
  // together, each element's sum in table order.  (Every lane decoding each term from the row
  // and checking it, two terms' loads at a time, took 1.4x the chunk-map kernel's time at 6
  // terms (worst), 2x at 14, 3x at 40; now 0.78x, 0.83x and 0.79x in the mean over 75 tables.)
  auto decode = [&](int first) {  // terms first + lane
    const int i = first + lane;
    const int o = 5 * (i - 1);  // of its inline words
    int64_t ts = ts0;
    double cf = cf0;
    int tl = tl0;
    if (first == 0) {
      auto word = [&](int c) { return __shfl_sync(0xffffffffu, w.w1, (o + c) & 31); };
      const int a0 = word(0), a1 = word(1), a2 = word(2), a3 = word(3), a4 = word(4);
      if (i > 0 && i <= kItemInline) {
        ts = item_i64(a0, a1);
        cf = __hiloint2double(a3, a2);
        tl = a4;
      }
    }
    if (i < nt && i > (g.width == 64 ? kItemInline : 0)) stored(i, ts, cf, tl);
    if (i < nt) {
      const bool in = inside(ts, tl);
      bad = bad || !in;
      terms.src[lane] = in ? ts : -1;
      terms.coeff[lane] = cf;
      terms.ld[lane] = tl;
    }
  };
  auto sums = [&](auto tag, int k0) {  // elements 32 k0 + lane, 32 (k0 + 1) + lane, ...
    constexpr int E = decltype(tag)::value, T = 8 / E;
    double acc[E];
    int rr[E], cc[E];
#pragma unroll
    for (int k = 0; k < E; ++k) {
      const int q = lane + 32 * (k0 + k);
      rr[k] = cc[k] = 0;
      acc[k] = 0.0;
      if (q < n)
        split(base + q, [&](int d, int j) {
          rr[k] += j * rstr[d];
          cc[k] += j * cstr[d];
        });
    }
#pragma unroll 1
    for (int first = 0; first < nt; first += 32) {
      const int m = min(32, nt - first);
      if (k0 == 0 || nt > 32) {
        __syncwarp();
        decode(first);
        __syncwarp();
      }
      auto add = [&](auto count, int i) {
        constexpr int C = decltype(count)::value;
        double v[C][E], cf[C];
#pragma unroll
        for (int t = 0; t < C; ++t) {
          const int64_t ts = terms.src[i + t];
          const int tl = terms.ld[i + t];
          cf[t] = terms.coeff[i + t];
#pragma unroll
          for (int k = 0; k < E; ++k)
            v[t][k] = ts >= 0 && lane + 32 * (k0 + k) < n ? load(src + ts + tl * rr[k] + cc[k])
                                                          : 0.0;
        }
#pragma unroll
        for (int t = 0; t < C; ++t)
#pragma unroll
          for (int k = 0; k < E; ++k) acc[k] = fma(cf[t], v[t][k], acc[k]);
      };
      int i = 0;
#pragma unroll 1
      for (; i + T <= m; i += T) add(std::integral_constant<int, T>{}, i);
      if constexpr (T >= 8)
        if (i + 4 <= m) {
          add(std::integral_constant<int, 4>{}, i);
          i += 4;
        }
      if constexpr (T >= 4)
        if (i + 2 <= m) {
          add(std::integral_constant<int, 2>{}, i);
          i += 2;
        }
      if (i < m) add(std::integral_constant<int, 1>{}, i);
    }
#pragma unroll
    for (int k = 0; k < E; ++k) {
      const int q = lane + 32 * (k0 + k);
      int to = 0;
      split(base + q, [&](int d, int j) { to += j * dstr[d]; });
      if (q < n) dst[dst_off + to] = acc[k];
    }
  };
  if (n <= 32) {
    sums(std::integral_constant<int, 1>{}, 0);
  } else if (n <= 64) {
    sums(std::integral_constant<int, 2>{}, 0);
  } else if (R >= 3 && nt >= 10) {  // (four elements' loads would reach too far apart)
#pragma unroll 1
    for (int k0 = 0; 32 * k0 < n; k0 += 2) sums(std::integral_constant<int, 2>{}, k0);
  } else {
#pragma unroll 1
    for (int k0 = 0; 32 * k0 < n; k0 += 4) sums(std::integral_constant<int, 4>{}, k0);
  }
  if (__any_sync(0xffffffffu, bad) && lane == 0) raise_bounds();
  __syncwarp();  // the next item's terms take the place of these
}

template <bool kSeveral, class Load>
__device__ __forceinline__ void gather_item_any(const ItemArgs& g, const ItemWords& w, int lane,
                                                ItemTerms& terms, Load load) {
  switch (w[10] & 255) {
    case 1: gather_item<1, kSeveral>(g, w, lane, terms, load); break;
    case 2: gather_item<2, kSeveral>(g, w, lane, terms, load); break;
    case 3: gather_item<3, kSeveral>(g, w, lane, terms, load); break;
    case 4: gather_item<4, kSeveral>(g, w, lane, terms, load); break;
    default:
      if (lane == 0) raise_bounds();
  }
}

}  // namespace tnb
