// Walks the items of a sweep of problems: every unit (128 queries of a row and head) is in exactly one item, the row
// that the kernel addresses for a unit, existing or not, lies inside the tensor, and rows put into smaller items for the last
// wave do not make another wave.
#include <cstdio>
#include <vector>

#include "attention_items.h"

using namespace b200ta;

static int check(int B, int R, int S, int num_sms) {
  const ItemPlan plan = split_items(B, R, S, num_sms);
  const int blocks = (S + kQTile - 1) / kQTile;
  std::vector<int> seen(size_t(B) * kHeads * R * blocks, 0);
  for (int i = 0; i < plan.num_items; ++i) {
    const Item it = decode_item(plan, i);
    for (int u = 0; u < kUnits; ++u) {
      const long long br = (long long)it.b * R + it.r0 + existing_row(it, u);
      if (br < 0 || br >= (long long)B * R || it.q0 < 0 || it.q0 >= S) return std::printf("unit outside: %d %d %d %d\n", B, R, S, num_sms);
      if (unit_row(it, u) >= it.rows) continue;
      const int block = it.q0 / kQTile + (it.two_blocks ? u & 1 : 0);
      if (block >= blocks) return std::printf("block outside: %d %d %d %d\n", B, R, S, num_sms);
      ++seen[((size_t(it.b) * kHeads + it.h) * R + it.r0 + unit_row(it, u)) * blocks + block];
    }
  }
  const long long bh = (long long)B * kHeads;
  const long long undivided = bh * (blocks / 2 * ((R + 1) / 2) + blocks % 2 * ((R + 3) / 4));
  if (plan.group[1].num_items > 0 && plan.num_items > (undivided + num_sms - 1) / num_sms * num_sms)
    return std::printf("another wave: %d %d %d %d\n", B, R, S, num_sms);
  for (int n : seen)
    if (n != 1) return std::printf("unit %d times: %d %d %d %d\n", n, B, R, S, num_sms);
  return 0;
}

int main() {
  for (int num_sms : {1, 7, 148})
    for (int B : {1, 2, 5, 20})
      for (int R : {1, 2, 3, 4, 5, 7, 8, 16, 37, 63, 64, 65, 129, 201, 333})
        for (int S : {1, 127, 128, 129, 256, 257, 385, 512, 640, 1025})
          if (check(B, R, S, num_sms) != 0) return 1;
  std::puts("ok");
  return 0;
}
