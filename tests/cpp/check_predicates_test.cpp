// Host run of the bounds-check predicates of the checked build
// (ma57_b200/csrc/gpu/checked.cuh) on hand-made front tables, good and with
// planted mistakes: every planted mistake must be caught, no good entry
// flagged.
#include <cstdio>
#include <vector>

#include "checked.cuh"

using namespace symla_gpu;

static int failures = 0;
#define EXPECT(cond)                                              \
  do {                                                            \
    if (!(cond)) {                                                \
      std::printf("FAILED line %d: %s\n", __LINE__, #cond);       \
      ++failures;                                                 \
    }                                                             \
  } while (0)

int main() {
  // descriptor shapes: m, ld, ncols, nelig, nextra
  EXPECT(front_shape_ok(10, 10, 3, 3, 0));
  EXPECT(front_shape_ok(10, 10, 3, 5, 2));  // two delayed columns taken over
  EXPECT(front_shape_ok(0, 0, 0, 0, 0));
  EXPECT(!front_shape_ok(10, 9, 3, 3, 0));   // ld < m
  EXPECT(!front_shape_ok(10, 10, 3, 4, 0));  // nelig != ncols + nextra
  EXPECT(!front_shape_ok(4, 4, 3, 5, 2));    // more eligible columns than rows
  EXPECT(!front_shape_ok(-1, 0, 0, 0, 0));

  // storage: a 6 x 6 front (ld 6) inside a 100-double arena
  std::vector<double> arena(100);
  const double* lo = arena.data();
  const double* hi = arena.data() + arena.size();
  EXPECT(storage_ok(arena.data(), 6, 6, lo, hi));
  EXPECT(storage_ok(arena.data() + 64, 6, 6, lo, hi));    // ends exactly at the arena's end
  EXPECT(!storage_ok(arena.data() + 65, 6, 6, lo, hi));   // one past
  EXPECT(!storage_ok(arena.data() + 10, 10, 10, lo, hi));
  EXPECT(!storage_ok(nullptr, 6, 6, lo, hi));
  EXPECT(storage_ok(nullptr, 0, 0, lo, hi));               // an empty front has no storage

  // A scatter entries of a front with m = 8, 3 own columns, 1 delayed row:
  // positions < 3 are own columns, later ones move down by nextra
  const int m = 8, ncols = 3, nextra = 1;
  const long long nnz = 20;
  EXPECT(a_entry_ok(0, 0, 0, ncols, nextra, m, nnz));    // diagonal
  EXPECT(a_entry_ok(1, 6, 19, ncols, nextra, m, nnz));   // pos 6 -> row 7, the last
  EXPECT(!a_entry_ok(1, 7, 0, ncols, nextra, m, nnz));   // pos 7 -> row 8 = m
  EXPECT(!a_entry_ok(2, 1, 0, ncols, nextra, m, nnz));   // above the diagonal
  EXPECT(!a_entry_ok(3, 5, 0, ncols, nextra, m, nnz));   // not an own column
  EXPECT(!a_entry_ok(0, 4, 20, ncols, nextra, m, nnz));  // value index past A
  EXPECT(!a_entry_ok(0, -1, 0, ncols, nextra, m, nnz));

  // extend-add maps of a child with a 4-row contribution block into a
  // 6-row parent: invmap entries in [-1, 4), relmap entries in [0, 6)
  const int invmap[6] = {-1, 0, 1, -1, 2, 3};
  const int relmap[4] = {1, 2, 4, 5};
  for (int v : invmap) EXPECT(in_range(v, -1, 4));
  for (int v : relmap) EXPECT(in_range(v, 0, 6));
  const int bad_inv[2] = {4, -2}, bad_rel[2] = {6, -1};
  for (int v : bad_inv) EXPECT(!in_range(v, -1, 4));
  for (int v : bad_rel) EXPECT(!in_range(v, 0, 6));

  // assembly tasks of a 100-row front, at most 64 rows each: j0, i0, i1, m, rows,
  // then its children (of 10 offsets), then its A entries (of [20, 30))
  EXPECT(asm_task_ok(32, 32, 96, 100, 64, 0, 10, 10, 20, 30, 20, 30));
  EXPECT(asm_task_ok(96, 96, 100, 100, 64, 10, 0, 10, 0, 0, 20, 30));     // no children, no entries
  EXPECT(!asm_task_ok(33, 40, 96, 100, 64, 0, 10, 10, 20, 30, 20, 30));   // not a 32-column block
  EXPECT(!asm_task_ok(128, 128, 130, 100, 64, 0, 0, 10, 0, 0, 20, 30));   // past the front
  EXPECT(!asm_task_ok(32, 0, 64, 100, 64, 0, 10, 10, 20, 30, 20, 30));    // rows above the diagonal block
  EXPECT(!asm_task_ok(32, 64, 101, 100, 64, 0, 10, 10, 20, 30, 20, 30));  // a row past the front
  EXPECT(!asm_task_ok(0, 0, 65, 100, 64, 0, 10, 10, 20, 30, 20, 30));     // too many rows
  EXPECT(!asm_task_ok(0, 0, 64, 100, 64, 5, 6, 10, 20, 30, 20, 30));      // a child past the list
  EXPECT(!asm_task_ok(0, 0, 64, 100, 64, -1, 2, 10, 20, 30, 20, 30));
  EXPECT(!asm_task_ok(0, 0, 64, 100, 64, 0, 10, 10, 19, 30, 20, 30));     // another front's entry
  EXPECT(!asm_task_ok(0, 0, 64, 100, 64, 0, 10, 10, 20, 31, 20, 30));
  EXPECT(!asm_task_ok(0, 0, 64, 100, 64, 0, 10, 10, 25, 24, 20, 30));

  // packed operands of a 100-row front: 2 row tiles, 3 chunks of 8 doubles a tile
  EXPECT(packed_ok(arena.data(), 48, 2, 100, 3, 8, lo, hi));
  EXPECT(packed_ok(arena.data() + 4, 48, 2, 100, 3, 8, lo, hi));          // ends exactly at the end
  EXPECT(!packed_ok(arena.data() + 5, 48, 2, 100, 3, 8, lo, hi));
  EXPECT(!packed_ok(arena.data(), 47, 2, 100, 3, 8, lo, hi));             // too small
  EXPECT(!packed_ok(arena.data(), 48, 1, 100, 3, 8, lo, hi));             // a row tile missing
  EXPECT(!packed_ok(nullptr, 48, 2, 100, 3, 8, lo, hi));

  // solve tasks: tiny fronts, blocks with their flags, parts with their slots
  EXPECT(tiny_task_ok(0, 8, 8));
  EXPECT(tiny_task_ok(7, 1, 8));
  EXPECT(!tiny_task_ok(7, 2, 8));
  EXPECT(!tiny_task_ok(0, 9, 20));  // more than warps
  EXPECT(!tiny_task_ok(-1, 1, 8));
  EXPECT(!tiny_task_ok(0, 0, 8));
  EXPECT(block_task_ok(1, 65, 64, 5, 7));
  EXPECT(!block_task_ok(1, 64, 64, 5, 7));  // no such block
  EXPECT(!block_task_ok(1, 65, 64, 6, 7));  // its flag past the flags
  EXPECT(!block_task_ok(-1, 65, 64, 5, 7));
  EXPECT(!block_task_ok(0, 65, 64, -1, 7));
  EXPECT(part_task_ok(0, 1, 4, 4));   // no helpers
  EXPECT(part_task_ok(0, 4, 1, 4));
  EXPECT(part_task_ok(3, 4, 3, 4));
  EXPECT(!part_task_ok(0, 4, 2, 4));  // a helper's slot past the slots
  EXPECT(!part_task_ok(3, 4, 4, 4));
  EXPECT(!part_task_ok(4, 4, 0, 4));
  EXPECT(!part_task_ok(0, 0, 0, 4));

  if (failures) return 1;
  std::printf("check_predicates OK\n");
  return 0;
}
