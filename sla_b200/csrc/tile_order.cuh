// The order in which the dK/dV kernel's last CTAs take their 128-key tiles: longest list first.
//
// A key tile's work is the length of its column lists, and popular KV blocks are selected several times as often as
// the average (32760 tokens of a (21, 30, 52) latent grid, top-k 25 of 512: a tile's two lists merge to 34 entries in the
// mean, to 110-150 for the longest). In sequence order such a tile may start last and run alone. The tiles of the last
// heads are therefore taken longest first. List scheduling on 148 SMs, counting entries alone: the busiest SM gets 130
// instead of 174 with 2 heads (119 is the mean over the SMs), 696 instead of 783 with 12 (691). Measured, with 2 heads:
// dK/dV 271 -> 195 us. Only the last heads: the CTAs in flight share the Q and dO rows of their heads in the L2, and with
// every tile ordered (groups of 64 MB of rows) a uniform mask of 32 heads, where there is nothing to gain, ran 4 % slower.
#pragma once
#include "common.cuh"

namespace sla {

constexpr int kOrderBins = 1024;
constexpr int kOrderThreads = 256;

struct TileOrder {
  const int32_t* col_offsets = nullptr;   // [BH][nb + 1]
  int32_t* order = nullptr;               // for the tiles of heads [h0, bh): head * ntiles + tile; nullptr: not wanted
  int nb = 0, ntiles = 0, bh = 0, h0 = 0, shift = 0;
};
inline int order_heads(int ntiles, int D, int bh) {      // last heads with at most 64 MB of 16-bit Q and dO rows
  const int tiles = 1024 * 128 / D, heads = ntiles >= tiles ? 1 : tiles / ntiles;
  return heads < bh ? heads : bh;
}
// With at most one tile per SM every tile starts at once and the order does not matter.
inline TileOrder make_tile_order(const int32_t* col_offsets, int32_t* order, int nb, int mb, int D, int bh) {
  TileOrder o;
  o.nb = nb; o.ntiles = ceil_div(nb, 2); o.bh = bh;
  if (static_cast<long long>(o.ntiles) * bh <= kSms) return o;
  o.col_offsets = col_offsets; o.order = order;
  o.h0 = bh - order_heads(o.ntiles, D, bh);
  while ((2LL * mb >> o.shift) >= kOrderBins) ++o.shift;   // a tile's two lists hold at most 2 * mb entries
  return o;
}

#if defined(__CUDACC__)
// Counting sort by one CTA of kOrderThreads threads. Tiles of equal length come in any order: the order decides when a
// tile is worked on, never what is computed for it.
__device__ inline void order_tiles(const TileOrder& o) {
  __shared__ int hist[kOrderBins];
  __shared__ int wsum[kOrderThreads / 32];
  constexpr int BPT = kOrderBins / kOrderThreads;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int n = (o.bh - o.h0) * o.ntiles;
  for (int i = tid; i < kOrderBins; i += kOrderThreads) hist[i] = 0;
  __syncthreads();
  auto bin_of = [&](int i) {
    const int h = o.h0 + i / o.ntiles, t = i % o.ntiles;
    const int32_t* off = o.col_offsets + static_cast<size_t>(h) * (o.nb + 1);
    const int len = off[min(2 * t + 2, o.nb)] - off[2 * t];
    return kOrderBins - 1 - min(max(len, 0) >> o.shift, kOrderBins - 1);
  };
#pragma unroll 4
  for (int i = tid; i < n; i += kOrderThreads) atomicAdd(&hist[bin_of(i)], 1);
  __syncthreads();
  int c[BPT], sum = 0;
#pragma unroll
  for (int b = 0; b < BPT; ++b) { c[b] = hist[tid * BPT + b]; sum += c[b]; }
  int incl = sum;
#pragma unroll
  for (int d = 1; d < 32; d <<= 1) {
    const int up = __shfl_up_sync(0xffffffffu, incl, d);
    if (lane >= d) incl += up;
  }
  if (lane == 31) wsum[warp] = incl;
  __syncthreads();
  int base = incl - sum;
  for (int w = 0; w < warp; ++w) base += wsum[w];
#pragma unroll
  for (int b = 0; b < BPT; ++b) { hist[tid * BPT + b] = base; base += c[b]; }
  __syncthreads();
#pragma unroll 4
  for (int i = tid; i < n; i += kOrderThreads) o.order[atomicAdd(&hist[bin_of(i)], 1)] = o.h0 * o.ntiles + i;
}
#endif

}  // namespace sla
