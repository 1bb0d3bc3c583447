// Walks every CTA (pair) of a launch with the kernels' own iterator and checks the workspace slots of its units:
//   slot_check M N K first factor sk_per grid split_slots whole_slots    (tile sizes: SC_BM, SC_BN, SC_BK)
// Prints "OK <whole tiles that pass through a slot>".
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "work_iter.cuh"

int main(int argc, char** argv) {
  if (argc != 10) return 2;
  KcgGemmParams p;
  memset(&p, 0, sizeof(p));
  p.M = atoi(argv[1]), p.N = atoi(argv[2]), p.K = atoi(argv[3]);
  p.split_first_tile = atoi(argv[4]), p.split_factor = atoi(argv[5]), p.sk_per = atoi(argv[6]);
  const int grid = atoi(argv[7]), split_slots = atoi(argv[8]), whole_slots = atoi(argv[9]);
  const int tiles_m = (p.M + SC_BM - 1) / SC_BM, tiles_n = (p.N + SC_BN - 1) / SC_BN, num_kb = (p.K + SC_BK - 1) / SC_BK;
  p.whole_slot0 = split_slots;
  int whole = 0;
  for (int cta = 0; cta < grid; ++cta) {
    kcg::WorkIter<SC_BM, SC_BN, 8> units(p, cta, grid, tiles_m, tiles_n, num_kb);
    kcg::WorkUnit w;
    while (units.next(w)) {
      // what the fp32 kernels write to and sum: slots slot0 .. slot0 + nsplit - 1
      const int slot0 = w.nsplit > 1 ? w.slot - w.split : p.whole_slot0 + cta;
      const int end = w.nsplit > 1 ? split_slots : split_slots + whole_slots;
      const int begin = w.nsplit > 1 ? 0 : split_slots;
      whole += w.nsplit == 1;
      if (slot0 < begin || slot0 + w.nsplit > end) {
        printf("tile %d of CTA %d: slots %d..%d outside %d..%d\n", w.tile, cta, slot0, slot0 + w.nsplit - 1, begin, end - 1);
        return 1;
      }
    }
  }
  printf("OK %d\n", whole);
}
