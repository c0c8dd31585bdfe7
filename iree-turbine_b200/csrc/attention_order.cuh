// The order in which the persistent CTAs of the two attention forward kernels take their work items.
//
// An item is a query tile (one-tile kernel) or a pair of them (tile-pair kernel) of one head; its cost is
// the number of K/V tiles it visits, which differs between the tiles of a causal head and between the
// sequences of a paged call.  Every role of a CTA walks the same items, so the order is a function of the
// position alone and nothing is exchanged between CTAs.
//
//   * The list is sorted, heaviest first, and dealt out in serpentine order: round r of gridDim.x
//     positions goes to the CTAs forwards when r is even and backwards when it is odd, so that who got the
//     heavier item of one round gets the lighter one of the next.  Dealing it out always forwards from a
//     head-major list gave a CTA the same few tiles of every head it met (the stride of 148 shares a factor
//     with most tile counts): the busiest CTA had 1.13 to 1.45 times the mean work, here it has 1.00 to
//     1.07 over the same shapes.
//   * Dense causal: all heads cost the same, so sorted means tile by tile over `group` heads.  Heads that
//     are in flight together share L2 with their K/V, so a group is all heads only while those fit, else
//     about six rounds of items.  One-tile kernel, us, all heads / groups: 4x16x3000 (94 MB of K/V) 158 / 156,
//     3x16x4500 (105 MB) 249 / 241, 4x32x4096 (256 MB) 636 / 510; groups of four and eight rounds 554 and 511.
//   * Paged: the lengths are device data.  Each CTA sorts the (sequence, tile) entries by cost in shared
//     memory before it starts; an entry stands for the items of all heads.  Above kMaxSorted entries the
//     count of rounds makes up for the order, and the list stays sequence-major.
//   * Dense without a mask: all items cost the same; the list is head-major and dealt forwards.
#pragma once

#include "common.cuh"

namespace b200k {
namespace attn_order {

constexpr int kMaxSorted = 512;                   // entries of a paged call that are sorted
constexpr int kSortBytes = 2 * 2 * kMaxSorted;    // uint16 [order, cost][entry]
constexpr int64_t kSharedKvBytes = 100ll << 20;   // K/V of the heads in flight, of 126 MB of L2

struct ItemOrder {
  int32_t num_items;  // heads * tiles
  int32_t heads;      // batch * q_heads
  int32_t tiles;      // items per head, the last one the heaviest
  int32_t group;      // heads whose items are interleaved (1: head-major)
  int32_t serpentine;
  int32_t sorted;     // entries in the shared-memory table, 0 without one
  Divisor by_tiles, by_heads, by_q_heads;
};

// Positions of one CTA: `for (Walk w; w.pos < order.num_items; w.step(order))`.
struct Walk {
  int base, pos;
  bool back;
  __device__ __forceinline__ Walk() : base(0), pos(blockIdx.x), back(false) {}
  __device__ __forceinline__ void step(const ItemOrder& o) {
    base += gridDim.x;
    back = o.serpentine && !back;
    pos = base + static_cast<int>(back ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
  }
};

// PAGED decides at compile time whether there is a table: with a test at run time the items of a dense call were not
// uniform over a warp for the compiler, and calls of short items took longer (15x4 6954 queries over 367 keys, us: 118
// with the test, 115 without).
template <bool PAGED>
__device__ __forceinline__ void item_at(const ItemOrder& o, int pos, const uint16_t* table, int q_heads, int& batch, int& head,
                                        int& tile) {
  if (PAGED && o.sorted) {
    const int i = o.by_q_heads.quotient(pos);
    const int e = table[i];
    head = pos - i * q_heads;
    batch = o.by_tiles.quotient(e);
    tile = e - batch * o.tiles;
    return;
  }
  int bh, rank;
  if (o.group == 1) {
    bh = o.by_tiles.quotient(pos);
    rank = pos - bh * o.tiles;
  } else if (o.group == o.heads) {
    rank = o.by_heads.quotient(pos);
    bh = pos - rank * o.heads;
  } else {
    const int span = o.group * o.tiles;
    const int g = pos / span, in = pos - g * span;
    const int first = g * o.group;
    const int members = min(o.group, o.heads - first);
    rank = in / members;
    bh = first + in - rank * members;
  }
  tile = o.tiles - 1 - rank;
  batch = o.by_q_heads.quotient(bh);
  head = bh - batch * q_heads;
}

// Sorts entries 0..n-1 by cost, heaviest first, equal ones by number.  Called by all threads of the CTA.
template <typename Cost>
__device__ __forceinline__ void sort_entries(uint16_t* table, int n, Cost cost_of) {
  uint16_t* cost = table + kMaxSorted;
  for (int e = threadIdx.x; e < n; e += blockDim.x) cost[e] = static_cast<uint16_t>(min(cost_of(e), 65535));
  __syncthreads();
  for (int e = threadIdx.x; e < n; e += blockDim.x) {
    const int c = cost[e];
    int rank = 0;
    for (int f = 0; f < n; ++f) rank += cost[f] > c || (cost[f] == c && f < e);
    table[rank] = static_cast<uint16_t>(e);
  }
  __syncthreads();
}

// kv_bytes: K and V that the items of one query head read (its share of a grouped K/V head).
inline int fill_order(ItemOrder& o, const char* who, int64_t batch, int64_t q_heads, int64_t tiles, bool causal, bool paged,
                      int64_t kv_bytes) {
  const int64_t heads = batch * q_heads, items = heads * tiles, sms = num_sms();
  if (items > INT32_MAX) return set_error(B200K_ERR_BAD_SHAPE, "%s: too many query tiles", who);
  o.num_items = static_cast<int32_t>(items);
  o.heads = static_cast<int32_t>(heads);
  o.tiles = static_cast<int32_t>(tiles);
  o.sorted = paged && batch * tiles <= kMaxSorted ? static_cast<int32_t>(batch * tiles) : 0;
  o.serpentine = causal || paged;
  o.by_tiles.set(tiles);
  o.by_heads.set(heads);
  o.by_q_heads.set(q_heads);
  o.group = 1;
  if (causal && !paged) {
    const int64_t six_rounds = (6 * sms + tiles / 2) / tiles;
    const int64_t group = heads * kv_bytes <= kSharedKvBytes || six_rounds > heads ? heads : six_rounds;
    o.group = static_cast<int32_t>(group > 1 ? group : 1);
  }
  return B200K_OK;
}

}  // namespace attn_order
}  // namespace b200k
