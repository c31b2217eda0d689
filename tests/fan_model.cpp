// Host model of the CUDA-core tile passes with phase fans: plans a circuit of
// gates and small unitaries as the engine does, merges each pass's phases
// (merge_phases), and applies the merged ops in FP64 from the fan tables and
// constants as the kernel reads them.
//   fan_model <ops file> <state in> <state out> <tile qubits> <block units>
// Prints: tile passes, gate steps, fans, phases left as ops of their own.
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <fstream>
#include <iterator>
#include <vector>

#include "../code_mojo_gb300/csrc/bf_internal.h"

using namespace bf;
using cd = std::complex<double>;

static std::vector<double> g_pool;

static void gate(std::vector<cd>& s, int target, uint64_t cmask, const double* m) {
  const uint64_t tb = 1ull << target;
  for (uint64_t i = 0; i < s.size(); ++i) {
    if ((i & tb) || (i & cmask) != cmask) continue;
    const cd a = s[i], b = s[i | tb];
    s[i] = cd(m[0], m[1]) * a + cd(m[2], m[3]) * b;
    s[i | tb] = cd(m[4], m[5]) * a + cd(m[6], m[7]) * b;
  }
}

static void unitary(std::vector<cd>& s, int t, int um, uint64_t cmask, const double* u) {
  const uint64_t D = 1ull << um, bits = (D - 1) << t;
  std::vector<cd> x(D);
  for (uint64_t i = 0; i < s.size(); ++i) {
    if ((i & bits) || (i & cmask) != cmask) continue;
    for (uint64_t c = 0; c < D; ++c) x[c] = s[i | (c << t)];
    for (uint64_t r = 0; r < D; ++r) {
      cd acc = 0;
      for (uint64_t c = 0; c < D; ++c) acc += cd(u[2 * (r * D + c)], u[2 * (r * D + c) + 1]) * x[c];
      s[i | (r << t)] = acc;
    }
  }
}

int main(int argc, char** argv) {
  if (argc < 6) return 2;
  std::ifstream fo(argv[1], std::ios::binary);
  std::vector<char> blob((std::istreambuf_iterator<char>(fo)), {});
  bf_oplist* list = nullptr;
  if (bf_ops_deserialize(blob.data(), blob.size(), &list) != BF_OK) return 3;
  const bf_op* ops;
  int64_t nops;
  int32_t n;
  bf_oplist_view(list, &ops, &nops, &n);
  std::vector<cd> s((size_t)1 << n);
  std::ifstream fi(argv[2], std::ios::binary);
  fi.read(reinterpret_cast<char*>(s.data()), (std::streamsize)(s.size() * sizeof(cd)));
  std::vector<GateInstr> gates;
  for (int64_t i = 0; i < nops; ++i) {
    const bf_op& o = ops[i];
    if (o.kind == BF_OP_UNITARY || o.kind == BF_OP_CUNITARY) {
      GateInstr g;
      std::memset(&g, 0, sizeof g);
      g.kind = GK_UNITARY;
      g.target = o.target;
      g.cmask = o.kind == BF_OP_CUNITARY ? o.controls : 0ull;
      g.um = o.target2;
      g.uoff = (int32_t)g_pool.size();
      g_pool.insert(g_pool.end(), o.data, o.data + 2 * ((size_t)1 << (2 * o.target2)));
      gates.push_back(g);
    } else if (o.kind == BF_OP_GATE) {
      gates.push_back(lower_gate(o, BF_SPEC_ALL));
    } else {
      return 4;
    }
  }
  int tiles = 0, singles = 0, fans = 0, phases = 0;
  for (const PlanStep& ps : plan_gates(n, gates, std::atoi(argv[4]), true, std::atof(argv[5]))) {
    if (!ps.is_tile) {
      ++singles;
      if (ps.gate.kind == GK_UNITARY) unitary(s, ps.gate.target, ps.gate.um, ps.gate.cmask, g_pool.data() + ps.gate.uoff);
      else gate(s, ps.gate.target, ps.gate.cmask, ps.gate.m);
      continue;
    }
    ++tiles;
    const TilePass& tp = ps.tile;
    std::vector<TileOp> merged;
    int halvings = 0, bare = 0;
    const int made = merge_phases(tp, merged, &g_pool, &halvings);
    fans += made;
    uint64_t tile_bits = 0;
    for (int j = 0; j < tp.K; ++j) tile_bits |= 1ull << tp.q[j];
    for (const TileOp& t : merged) {
      uint64_t cm = t.cmask_out;
      for (int j = 0; j < tp.K; ++j)
        if ((t.cmask_loc >> j) & 1u) cm |= 1ull << tp.q[j];
      if (t.kind == GK_PHASE) ++phases;
      if (t.fan) {
        if (t.fan > made || t.fan > kMaxPassFans || (t.fan_off & 1) || (t.fan_shape & 0xff) != tp.K / 2) return 5;
        if (t.kind != GK_FAN && (t.cmask_loc || t.cmask_out)) return 6;
        const int a = tp.K / 2;
        const size_t na = (size_t)1 << a, nb = (size_t)1 << (tp.K - a);
        const double* d = g_pool.data() + t.fan_off;
        const double* c = d + 2 * (na + nb);
        if (c[4 * t.fan_consts] != 1.0 || c[4 * t.fan_consts + 1] != 0.0) return 7;
        if (t.kind != GK_FAN && t.um) {  // the Hadamard before the fan
          const double r = t.um == GK_HU ? 1.0 : std::sqrt(0.5);
          const double m[8] = {r, 0, r, 0, r, 0, -r, 0};
          gate(s, tp.q[t.tloc], 0, m);
          bare += t.um == GK_HU;
        }
        for (uint64_t i = 0; i < s.size(); ++i) {
          if ((i & t.cmask_out) != t.cmask_out) continue;
          uint32_t x = 0;
          for (int j = 0; j < tp.K; ++j) x |= (uint32_t)((i >> tp.q[j]) & 1) << j;
          if (t.tloc >= 0 && !((x >> t.tloc) & 1)) continue;
          cd w(1.0, 0.0);
          for (int k = 0; k < t.fan_consts; ++k) {
            uint64_t m;
            std::memcpy(&m, c + 4 * k, sizeof m);
            if (m & tile_bits) return 8;
            if ((i & m) == m) w *= cd(c[4 * k + 2], c[4 * k + 3]);
          }
          if (t.fan_shape & kFanA) w *= cd(d[2 * (x & (na - 1))], d[2 * (x & (na - 1)) + 1]);
          if (t.fan_shape & kFanB) w *= cd(d[2 * (na + (x >> a))], d[2 * (na + (x >> a)) + 1]);
          s[i] *= w;
        }
        if (t.kind == GK_FAN) continue;
      }
      if (t.kind == GK_HU) {
        const double m[8] = {1, 0, 1, 0, 1, 0, -1, 0};
        gate(s, tp.q[t.tloc], cm, m);
        ++bare;
      } else if (t.kind == GK_UNITARY) {
        unitary(s, tp.q[t.tloc], t.um, cm, g_pool.data() + t.uoff);
      } else if (t.tloc >= 0) {
        gate(s, tp.q[t.tloc], cm, t.m);
      } else {
        for (uint64_t i = 0; i < s.size(); ++i)
          if ((i & cm) == cm) s[i] *= ((i >> t.tglob) & 1) ? cd(t.m[6], t.m[7]) : cd(t.m[0], t.m[1]);
      }
    }
    if (bare != 2 * halvings) return 9;
    for (cd& x : s) x *= std::ldexp(1.0, -halvings);
  }
  std::ofstream fw(argv[3], std::ios::binary);
  fw.write(reinterpret_cast<const char*>(s.data()), (std::streamsize)(s.size() * sizeof(cd)));
  std::printf("%d %d %d %d\n", tiles, singles, fans, phases);
  return 0;
}
