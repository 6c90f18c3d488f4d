// How the attention kernel's work is cut into items.  Integer code without CUDA calls, so that it also compiles for the
// host alone, where a test walks all items of a problem.
#pragma once
#include <stdint.h>

#include "layout.h"

#ifdef __CUDACC__
#define B200TA_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define B200TA_HOST_DEVICE inline
#endif

namespace b200ta {

constexpr int kQTile = 128;  // queries per unit
constexpr int kUnits = 4;    // units per item

// A range of pair rows and how its units are put together: per (b, h) `pairs` x ceil(rows / rows_pair) items of two
// query blocks, then `singles` x ceil(rows / rows_single) items of one block.
struct RowGroup {
  int row0, row_end, rows_pair, rows_single;
  int items_pair, items_bh, num_items;
  uint32_t bh_mul, bh_shr;
};

// All items of a call: all (b, h) of group 0 come first.
struct ItemPlan {
  int pairs, singles;  // query blocks of a row: 2 * pairs + singles; the first go two by two
  uint32_t pairs_mul, pairs_shr, singles_mul, singles_shr;  // divisions as multiply-high and shift
  RowGroup group[2];
  int num_items;
};

struct Item {
  int b, h, r0, rows;  // first pair row and how many (1..4)
  int q0;
  bool two_blocks;  // unit u = row u / 2, query block u % 2; otherwise unit u = row u
};

// n / d for n < 2^31 with the constants of fast_div_constants(); mul == 0 stands for d == 1.
B200TA_HOST_DEVICE int fast_div(int n, uint32_t mul, uint32_t shr) {
  return mul ? int(uint32_t((uint64_t(uint32_t(n)) * mul) >> 32) >> shr) : n;
}

// Items are ordered (b, h, row group, query blocks) with the query blocks fastest: the CTAs that run at the same
// time work on the query blocks of neighbouring pair rows, so a row's K and V come from HBM once (and then from
// L2) while the head's bias, shared by all rows, stays in L2.
B200TA_HOST_DEVICE Item decode_item(const ItemPlan& p, int item) {
  Item it;
  const bool second = item >= p.group[0].num_items;
  const RowGroup& g = p.group[second];
  if (second) item -= p.group[0].num_items;
  const int bh = fast_div(item, g.bh_mul, g.bh_shr);
  int idx = item - bh * g.items_bh;
  it.h = bh % kHeads;
  it.b = bh / kHeads;
  it.two_blocks = idx < g.items_pair;
  if (it.two_blocks) {
    const int n = fast_div(idx, p.pairs_mul, p.pairs_shr);
    it.rows = g.rows_pair;
    it.r0 = g.row0 + n * g.rows_pair;
    it.q0 = (idx - n * p.pairs) * 2 * kQTile;
  } else {
    idx -= g.items_pair;
    const int n = fast_div(idx, p.singles_mul, p.singles_shr);
    it.rows = g.rows_single;
    it.r0 = g.row0 + n * g.rows_single;
    it.q0 = (2 * p.pairs + idx - n * p.singles) * kQTile;
  }
  if (it.r0 + it.rows > g.row_end) it.rows = g.row_end - it.r0;
  return it;
}

// Row of the item that `unit` belongs to; the item has no such unit if that is not below it.rows.
B200TA_HOST_DEVICE int unit_row(const Item& it, int unit) { return it.two_blocks ? unit >> 1 : unit; }
// The same for addresses, which have to stay inside the tensors for every unit: clamped to the item's rows.
B200TA_HOST_DEVICE int existing_row(const Item& it, int unit) {
  const int row = unit_row(it, unit);
  return row < it.rows ? row : it.rows - 1;
}

// Constants for fast_div: with l = ceil(log2 d) and mul = floor(2^(31+l) / d) + 1, floor(n / d) equals
// (n * mul) >> (31 + l) for every n < 2^31.
inline void fast_div_constants(uint32_t d, uint32_t* mul, uint32_t* shr) {
  if (d <= 1) {
    *mul = 0, *shr = 0;
    return;
  }
  uint32_t l = 0;
  while ((uint64_t(1) << l) < d) ++l;
  *mul = uint32_t((uint64_t(1) << (31 + l)) / d + 1);
  *shr = l - 1;
}

// How the units (128 queries of one row and head) of a (b, h) are put together into items of up to four.
// Normally the query blocks go two by two with two rows each and an odd last block with four rows.  A problem with
// too few units to fill the SMs that way takes fewer units per item instead: a CTA with one or two units finishes a
// tile in some 1000 to 1600 clocks of latency, one with four in some 2800.  For the same reason, when the last wave is at
// most half full, the rows that do not fill whole waves go to items of two units, provided that no CTA gets more items
// that way (with many (b, h) of few rows, rows in steps of four leave too much over: 20 x 16 rows of 384 97 us, undivided
// 89).  What it gives goes down with the number of waves: 6-7 % at 2-3 waves (225 tokens 39.3 -> 36.9 us), 3-4 % at 7 (360
// tokens 98.5 -> 95.6), 2 % at 11 (423 tokens 160.9 -> 157.4); at 12 to 16 it would still be 1.5 to 2.4 % (494 tokens
// 203.5 -> 199.9), from 18 on it was between +1.7 and -2.5 %, with runs that differ by up to 2.
inline ItemPlan split_items(int B, int R, int S, int num_sms) {
  ItemPlan p{};
  const int blocks = (S + kQTile - 1) / kQTile;
  const int64_t bh = int64_t(B) * kHeads;
  auto fill = [&](int which, int row0, int row_end, int rows_pair, int rows_single) -> int64_t {
    RowGroup& g = p.group[which];
    const int rows = row_end - row0;
    g.row0 = row0, g.row_end = row_end, g.rows_pair = rows_pair, g.rows_single = rows_single;
    g.items_pair = p.pairs * ((rows + rows_pair - 1) / rows_pair);
    g.items_bh = g.items_pair + p.singles * ((rows + rows_single - 1) / rows_single);
    g.num_items = int(bh * g.items_bh);
    fast_div_constants(uint32_t(g.items_bh), &g.bh_mul, &g.bh_shr);
    return bh * g.items_bh;
  };
  auto whole = [&](int pairs, int rows_pair, int rows_single) {
    p.pairs = pairs, p.singles = blocks - 2 * pairs;
    fill(1, R, R, 1, 1);
    return fill(0, 0, R, rows_pair, rows_single);
  };
  if (whole(0, 1, 1) > num_sms &&                                                 // one unit per item
      (blocks == 1 ? whole(0, 1, 2) : whole(blocks / 2, 1, 2)) > num_sms) {       // two units per item
    const int64_t items = whole(blocks / 2, R > 1 ? 2 : 1, R > 2 ? 4 : R);
    const int64_t waves = items / num_sms, rest = items % num_sms;
    if (waves >= 1 && waves < 12 && rest > 0 && 2 * rest <= num_sms) {
      // rows that fill the whole waves, in steps of four (one item of the odd block)
      const int64_t per_four = bh * (2 * p.pairs + p.singles);
      const int row = int(waves * num_sms / per_four) * 4;
      if (row > 0 && row < R && fill(0, 0, row, 2, 4) + fill(1, row, R, 1, 2) > (waves + 1) * num_sms)
        whole(blocks / 2, 2, 4);
    }
  }
  fast_div_constants(uint32_t(p.pairs), &p.pairs_mul, &p.pairs_shr);
  fast_div_constants(uint32_t(p.singles), &p.singles_mul, &p.singles_shr);
  p.num_items = p.group[0].num_items + p.group[1].num_items;
  return p;
}

}  // namespace b200ta
