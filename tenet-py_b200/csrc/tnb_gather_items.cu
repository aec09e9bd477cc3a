// K1-I: the block gather from warp items.
//
// The same block maps as tnb_block_gather (permute, scale, sum the terms of one destination
// block, write once), the table cut into items of at most 256 consecutive elements of one
// segment, each one 128- or 256-byte row that a warp reads in one round of loads: offsets,
// the first terms inline, 32-bit extents, strides and division constants.  A warp moves its
// item alone, all loads of a one-term item in flight before the first store; an item of several
// terms decodes them into the warp's own shared memory.  Large tables of one term a segment and
// of several have a build each.
//
// What bounds it: a many-wave gather (the batched U(1) x U(1) x fZ2 update moves 0.13-0.53 GB
// a launch in segments of about 600 elements) wants some 45 KB in flight per SM to cover
// HBM's latency.  The chunk-row kernel (tnb_block_gather_direct) keeps about 20: a CTA of 256
// threads waits for its row, moves one 600-element segment at 2.3 elements per thread and
// holds 64 registers of 64-bit offsets.  An item's 32-bit indexing leaves room for eight
// elements per lane on 32 warps, and segments of any size fill whole warps (600 elements are
// three items of 224, 224 and 152).
//
// Measured on B200, a launch alone (chunk rows before): 531 MB in 46,848 segments 98.8 us, 5.4
// TB/s (334.6, 1.6); 473 MB of row copies 81.8 us, 5.8 TB/s (268.8); 132 MB, every source
// strided, 31.0 us (86.1); 122 MB in 26 segments 22.1 us (48.0); 974 elements 1.3 us (1.8).
#include <string>

#include "tnb_gather_item.cuh"

namespace tnb {

int device_sms();

template <int NT, int kMinBlocks, bool kRelease, bool kSeveral>
__global__ void __launch_bounds__(NT, kMinBlocks) gather_items_kernel(const ItemArgs g) {
  __shared__ ItemTerms terms[kSeveral ? NT / 32 : 1];  // (one-term items leave theirs unused)
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t item = static_cast<int64_t>(blockIdx.x) * (NT / 32) + warp;
  ItemWords w{0, 0};
  if (item < g.n_items) {
    const int32_t* r = g.rows + item * g.width;
    w.w0 = __ldg(r + lane);
    if (kSeveral && g.width == 64) w.w1 = __ldg(r + 32 + lane);
  }
  pdl_wait<kRelease>();  // the rows are static; the source may be the previous kernel's output
  if (item < g.n_items)
    gather_item_any<kSeveral>(g, w, lane, terms[kSeveral ? warp : 0],
                              [](const double* p) { return __ldg(p); });
}

// Items of several terms have more registers and fewer warps an SM: under the 64 of 32 warps they
// spill (3,240 elements of three terms 2.9 us, 2.3 so; 1.9 M of six 48, 40).  Small tables of
// either kind run the one build: a chain that alternates between two fetches its instructions
// anew at every launch (a matvec on the L = 64 mid bond 19.4 us, 18.1 so).
// A warp per item: two items a warp, their rows in flight together, spilled (1.9 M elements in
// 400 segments 11.2 us, one item 8.6; the batched update the same).  The next kernel is
// released early only by tables of up to eight warps an SM: from more, its CTAs start while most
// of this one's data is still to move and hold the SMs meanwhile (3,029 items, a grouped GEMM
// and 1,515 items of the 40-state U(1) contraction: 52 us released early, 37 not; a compiled
// matvec on the L = 64 mid bond, 14 to 75 items, gains 2 us a launch from the early release).
template <bool kSeveral>
static cudaError_t launch_items(const ItemArgs& g, cudaStream_t s) {
  const int64_t sms = device_sms(), n = g.n_items;
  if (n > 32 * sms)
    return launch(gather_items_kernel<256, kSeveral ? 3 : 4, false, kSeveral>,
                  static_cast<unsigned>((n + 7) / 8), 256, s, g);
  if (n > 8 * sms)
    return launch(gather_items_kernel<128, kSeveral ? 5 : 8, false, kSeveral>,
                  static_cast<unsigned>((n + 3) / 4), 128, s, g);
  return launch(gather_items_kernel<128, 5, true, true>,
                static_cast<unsigned>((n + 3) / 4), 128, s, g);
}

}  // namespace tnb

extern "C" int tnb_block_gather_items(const int32_t* item_rows, int32_t width, int64_t n_items,
                                      const int64_t* term_src, const double* term_coeff,
                                      const int64_t* term_ld, int64_t n_term,
                                      const double* src0, int64_t n_src0, double* dst0,
                                      int64_t n_dst0, const double* src1, int64_t n_src1,
                                      double* dst1, int64_t n_dst1, void* stream) {
  TNB_REQUIRE(n_items >= 0 && n_term >= 0, "tnb_block_gather_items: negative size");
  TNB_REQUIRE(width == 32 || width == 64, "tnb_block_gather_items: rows of 32 or 64 words");
  if (n_items == 0) return TNB_OK;
  TNB_REQUIRE(item_rows != nullptr, "tnb_block_gather_items: item_rows is null");
  TNB_REQUIRE(n_term == 0 || (term_src != nullptr && term_coeff != nullptr && term_ld != nullptr),
              "tnb_block_gather_items: term arrays are null");
  TNB_REQUIRE(dst0 != nullptr || dst1 != nullptr, "tnb_block_gather_items: no destination buffer");
  TNB_REQUIRE(n_items < (int64_t(1) << 31), "tnb_block_gather_items: too many items for one launch");
  const tnb::ItemArgs g{item_rows, width, n_items, term_src, term_coeff, term_ld, n_term,
                        src0, n_src0, dst0, n_dst0, src1, n_src1, dst1, n_dst1};
  const bool several = width == 64 || n_items <= 8 * static_cast<int64_t>(tnb::device_sms());
  const cudaError_t e = several ? tnb::launch_items<true>(g, tnb::as_stream(stream))
                                : tnb::launch_items<false>(g, tnb::as_stream(stream));
  if (e != cudaSuccess) {
    tnb::set_error(std::string("tnb_block_gather_items: ") + cudaGetErrorString(e));
    return TNB_ECUDA;
  }
  return tnb::check_launch("tnb_block_gather_items");
}
