// Prints what the host-side rules of a call decide (csrc/mmoe_common.cuh), for the CPU tests.  Host code only.
#include <stdio.h>
#include <string.h>

#include "../vllm_plugin_b200/csrc/mmoe_common.cuh"
#include "../vllm_plugin_b200/csrc/mmoe_plan_cache.h"

using namespace mmoe;

static const int kBlockMs[] = {16, 32, 64, 128, 192, 240};

// forms <ranks> <pair_above> <tile_select> <peers> <block_m> <m> <pairs> <small> <staged>
static void forms() {
  for (int ranks : {1, 2, 8})
    for (int pair_above : {192, kNeverPair, 0})
      for (int select : {0, 1, 2})
        for (int peers : {0, 1})
          for (int block_m : kBlockMs)
            for (int m : {0, 1, 7, 15, 16, 17, 64, 128, 129, 192, 193, 1000, 3840}) {
              static const void* peer[8] = {};
              Ctx c{};
              c.geo = MmoeGeometry{ranks, 0, 384, 6, 5120, 2304, 1, 3840};
              c.e_local = 384 / ranks;
              c.pair_above = pair_above;
              c.tile_select = select;
              c.peer_ws = peers ? peer : nullptr;
              const GemmForms f = gemm_forms(c, m, select != 1 && m > 0);
              printf("forms %d %d %d %d %d %d %d %d %d\n", ranks, pair_above, select, peers, block_m, m, f.pairs, f.small,
                     staged_tokens(c, m, block_m));
            }
}

// cache <keys in turn> <rounds> <built> <built from a sibling> <wrong values>, with 4 workspaces and room for 16
static void cache() {
  struct Key {
    int ws, layer;
    bool operator==(const Key& o) const { return ws == o.ws && layer == o.layer; }
    bool same_workspace(const Key& o) const { return ws == o.ws; }
  };
  for (int keys : {1, 3, 15, 16, 17, 40}) {
    PlanCache<Key, int, 16> plans;
    int built = 0, siblings = 0, wrong = 0;
    const Key first{0, 0};
    const std::shared_ptr<const int> held = plans.get(first, [&](const int*) { ++built; return std::make_shared<int>(0); });
    for (int round = 0; round < 3; ++round)
      for (int i = 0; i < keys; ++i) {
        const Key key{i % 4, i};
        plans.get(Key{9, 9}, [](const int*) { return std::shared_ptr<int>(); });     // fails: not kept
        const auto v = plans.get(key, [&](const int* sibling) {
          ++built;
          if (sibling != nullptr) siblings += *sibling % 4 == key.ws ? 1 : 1000;
          return std::make_shared<int>(i);
        });
        wrong += v == nullptr || *v != i;
      }
    printf("cache %d 3 %d %d %d\n", keys, built, siblings, wrong + (*held != 0));
  }
}

// cuts <block_m> <pair tiles> <cap> <n> <parts> <step> <non-empty tiles> <scale chunks of the expert's blocks>
static void cuts() {
  for (int block_m : kBlockMs) {
    bool caps[kSmallTileRows + 1] = {};
    for (int m = 0; m <= 300; ++m)
      for (int experts : {1, 63, 64, 512}) caps[small_only_cap(m, block_m, experts)] = true;
    caps[kDeepTileRows] = caps[kSmallTileRows] = true;                 // calls with pair tiles
    for (int cap = 0; cap <= kSmallTileRows; ++cap)
      for (int n = 1; caps[cap] && n <= 1100; ++n)
        for (int pairs = 0; pairs <= 1; ++pairs) {
          const Cut c = cut_rows(n, pairs != 0, cap);
          printf("cuts %d %d %d %d %d %d %d %d\n", block_m, pairs, cap, n, c.parts, c.step, (n + c.step - 1) / c.step,
                 (n + block_m - 1) / block_m * chunks_per_block(block_m));
        }
  }
}

// pairs <pair_above> <cap> <n> <on pairs> <tiles if not> <pair tasks if so>
static void pairs() {
  for (int pair_above : {192, kNeverPair, 0})
    for (int cap : {kDeepTileRows, kSmallTileRows})
      for (int n = 1; n <= 1100; ++n)
        printf("pairs %d %d %d %d %d %d\n", pair_above, cap, n, on_pairs(n, pair_above, cap), cut_rows(n, false, cap).parts,
               cut_rows(n, true, cap).parts / 2);
}

// abi <version> <bytes of MmoeGeometry> <MmoeLayout> <MmoeWeights> <MmoeOptions>
static void abi() {
  printf("abi %d %zu %zu %zu %zu\n", MMOE_ABI_VERSION, sizeof(MmoeGeometry), sizeof(MmoeLayout), sizeof(MmoeWeights), sizeof(MmoeOptions));
}

int main(int argc, char** argv) {
  for (int i = 1; i < argc; ++i)
    if (strcmp(argv[i], "forms") == 0) forms();
    else if (strcmp(argv[i], "cache") == 0) cache();
    else if (strcmp(argv[i], "abi") == 0) abi();
    else if (strcmp(argv[i], "cuts") == 0) cuts();
    else if (strcmp(argv[i], "pairs") == 0) pairs();
  return 0;
}
