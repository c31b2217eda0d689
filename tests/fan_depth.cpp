// Plans a deep circuit of gates as the engine does and reports, over its tile
// passes after merge_phases: ops, fans, the most constants of one fan, and the
// milliseconds that planning and merging took.
//   fan_depth <ops file> <tile qubits> <block units>
#include <algorithm>
#include <chrono>
#include <cstdio>
#include <cstdlib>
#include <fstream>
#include <iterator>
#include <vector>

#include "../code_mojo_gb300/csrc/bf_internal.h"

using namespace bf;

int main(int argc, char** argv) {
  if (argc < 4) return 2;
  std::ifstream fo(argv[1], std::ios::binary);
  std::vector<char> blob((std::istreambuf_iterator<char>(fo)), {});
  bf_oplist* list = nullptr;
  if (bf_ops_deserialize(blob.data(), blob.size(), &list) != BF_OK) return 3;
  const bf_op* ops;
  int64_t nops;
  int32_t n;
  bf_oplist_view(list, &ops, &nops, &n);
  std::vector<GateInstr> gates;
  for (int64_t i = 0; i < nops; ++i) gates.push_back(lower_gate(ops[i], BF_SPEC_ALL));
  const auto t0 = std::chrono::steady_clock::now();
  size_t total = 0;
  int fans = 0, most = 0, halvings = 0;
  std::vector<double> pool;
  for (const PlanStep& ps : plan_gates(n, gates, std::atoi(argv[2]), true, std::atof(argv[3]))) {
    if (!ps.is_tile) {
      ++total;
      continue;
    }
    std::vector<TileOp> merged;
    fans += merge_phases(ps.tile, merged, &pool, &halvings);
    total += merged.size();
    for (const TileOp& t : merged) most = std::max(most, (int)t.fan_consts);
  }
  const double ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
  std::printf("%zu %d %d %.3f\n", total, fans, most, ms);
  return 0;
}
