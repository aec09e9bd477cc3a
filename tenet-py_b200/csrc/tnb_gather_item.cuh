// One item of a block gather from warp items (the kernel that runs tables of them is in
// tnb_gather_items.cu): the row's words, its checks and the move of its elements by one warp.
#pragma once

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

// Word i of the row whose words 0..31 and 32..63 the lanes hold in w0 and w1.
struct ItemWords {
  int w0, w1;
  __device__ __forceinline__ int operator[](int i) const {
    return __shfl_sync(0xffffffffu, i < 32 ? w0 : w1, i & 31);
  }
};

// One item of rank R.  Every check is made once per item on the segment's whole box (warp
// uniform): the row's division constants and extents, and the box's lowest and highest
// destination and source offsets.  `load` reads a source element.
template <int R, class Load>
__device__ __forceinline__ void gather_item(const ItemArgs& g, const ItemWords& w, int lane,
                                            Load load) {
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
  // several terms (or none): four elements per lane at a time, two terms' loads together,
  // each element's sum in table order
  const int nt = t1 - t0;
  auto term = [&](int i, int64_t& ts, double& cf, int& tl) {
    if (i == 0) {
      ts = ts0, cf = cf0, tl = tl0;
    } else if (g.width == 64 && i <= kItemInline) {
      const int o = 32 + 5 * (i - 1);
      ts = item_i64(w[o], w[o + 1]);
      cf = __hiloint2double(w[o + 3], w[o + 2]);
      tl = w[o + 4];
    } else {
      ts = __ldg(g.term_src + t0 + i);
      cf = __ldg(g.term_coeff + t0 + i);
      const int64_t ld = __ldg(g.term_ld + t0 + i);
      tl = static_cast<int>(ld);
      if (ld != tl) ts = -1;  // refused below
    }
  };
  bool bad = false;
#pragma unroll 1
  for (int k0 = 0; k0 < kItemEpl && 32 * k0 < n; k0 += 4) {
    double acc[4];
    int rr[4], cc[4], to[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int q = lane + 32 * (k0 + k);
      rr[k] = cc[k] = to[k] = 0;
      acc[k] = 0.0;
      if (q < n)
        split(base + q, [&](int d, int j) {
          rr[k] += j * rstr[d];
          cc[k] += j * cstr[d];
          to[k] += j * dstr[d];
        });
    }
    auto fetch = [&](int64_t ts, int tl, double (&v)[4]) {
      const bool in = inside(ts, tl);
      bad = bad || !in;
#pragma unroll
      for (int k = 0; k < 4; ++k)
        v[k] = in && lane + 32 * (k0 + k) < n ? load(src + ts + tl * rr[k] + cc[k]) : 0.0;
    };
    int i = 0;
#pragma unroll 1
    for (; i + 2 <= nt; i += 2) {
      int64_t sa, sb;
      double ca, cb, va[4], vb[4];
      int la, lb;
      term(i, sa, ca, la);
      term(i + 1, sb, cb, lb);
      fetch(sa, la, va);
      fetch(sb, lb, vb);
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[k] = fma(cb, vb[k], fma(ca, va[k], acc[k]));
    }
    if (i < nt) {
      int64_t sa;
      double ca, va[4];
      int la;
      term(i, sa, ca, la);
      fetch(sa, la, va);
#pragma unroll
      for (int k = 0; k < 4; ++k) acc[k] = fma(ca, va[k], acc[k]);
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (lane + 32 * (k0 + k) < n) dst[dst_off + to[k]] = acc[k];
  }
  if (bad && lane == 0) raise_bounds();
}

template <class Load>
__device__ __forceinline__ void gather_item_any(const ItemArgs& g, const ItemWords& w, int lane,
                                                Load load) {
  switch (w[10] & 255) {
    case 1: gather_item<1>(g, w, lane, load); break;
    case 2: gather_item<2>(g, w, lane, load); break;
    case 3: gather_item<3>(g, w, lane, load); break;
    case 4: gather_item<4>(g, w, lane, load); break;
    default:
      if (lane == 0) raise_bounds();
  }
}

}  // namespace tnb
