// planner.cpp — host-side lowering, validation and tile-pass planning.
// No device code: everything here runs (and is tested) without a GPU.
#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <deque>

#include "bf_internal.h"

namespace bf {

void fail(int code, const char* fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  throw Error{code, buf};
}

void check_cuda(cudaError_t e, const char* what) {
  if (e != cudaSuccess) {
    cudaGetLastError();
    fail(e == cudaErrorMemoryAllocation ? BF_ENOMEM : BF_ECUDA, "%s: %s", what, cudaGetErrorString(e));
  }
}

int current_device() {
  int dev = 0;
  BF_CUDA(cudaGetDevice(&dev));
  return dev;
}

// ---- validation: validate_circuit (executors.mojo:78-185) ----------------
static void check_qubit(int idx, int n, const char* label) {
  if (idx < 0 || idx >= n) fail(BF_EINVAL, "%s out of bounds: %d", label, idx);
}

void validate_ops(int n, const bf_op* ops, int64_t nops) {
  if (nops < 0) fail(BF_EINVAL, "negative op count");
  if (nops > 0 && ops == nullptr) fail(BF_EINVAL, "ops is null");
  for (int64_t i = 0; i < nops; ++i) {
    const bf_op& o = ops[i];
    switch (o.kind) {
      case BF_OP_GATE: {
        check_qubit(o.target, n, "Target");
        if (o.gate < 0 || o.gate > BF_GATE_CUSTOM) fail(BF_EINVAL, "Unknown gate kind: %d", o.gate);
        if (n < 64 && (o.controls >> n)) fail(BF_EINVAL, "Control out of bounds: %d", 63 - __builtin_clzll(o.controls));
        if (o.ncontrols < 0 || __builtin_popcountll(o.controls) != o.ncontrols)
          fail(BF_EINVAL, "Gate control kind mismatch: expected %d controls, mask holds %d", o.ncontrols,
               __builtin_popcountll(o.controls));
        if (o.flags & BF_OPF_FUSE_WITH_NEXT) {
          if (i + 1 >= nops || ops[i + 1].kind != BF_OP_GATE)
            fail(BF_EINVAL, "fused pair: the gate flagged FUSE_WITH_NEXT must be followed by a gate");
        }
        break;
      }
      case BF_OP_SWAP:
      case BF_OP_CSWAP:
        check_qubit(o.target, n, "Target");
        check_qubit(o.target2, n, "Target");
        break;
      case BF_OP_QREV:
      case BF_OP_BITREV:
      case BF_OP_PERMUTE:
      case BF_OP_GROVER_DIFFUSER:
      case BF_OP_GROVER_INVERSION0: {
        if (o.nqubits < 0 || (o.nqubits > 0 && o.qubits == nullptr)) fail(BF_EINVAL, "qubit list is null");
        for (int64_t k = 0; k < o.nqubits; ++k) check_qubit(o.qubits[k], n, "Target");
        if (o.kind == BF_OP_BITREV || o.kind == BF_OP_GROVER_DIFFUSER || o.kind == BF_OP_GROVER_INVERSION0) {
          uint64_t seen = 0;
          for (int64_t k = 0; k < o.nqubits; ++k) {
            if ((seen >> o.qubits[k]) & 1) fail(BF_EINVAL, "Duplicate target: %d", o.qubits[k]);
            seen |= 1ull << o.qubits[k];
          }
        }
        if (o.kind == BF_OP_PERMUTE && o.nqubits != 0) {
          if (o.nqubits != n) fail(BF_EINVAL, "Permutation size mismatch: %lld", (long long)o.nqubits);
          uint64_t seen = 0;
          for (int64_t k = 0; k < o.nqubits; ++k) {
            if ((seen >> o.qubits[k]) & 1) fail(BF_EINVAL, "Duplicate permutation value: %d", o.qubits[k]);
            seen |= 1ull << o.qubits[k];
          }
        }
        break;
      }
      case BF_OP_MODEXP:
      case BF_OP_MODEXP_INV: {  // apply_modexp(_inverse) checks (algos/shor.mojo:60-76, 103-119)
        const char* name = o.kind == BF_OP_MODEXP ? "MOD_EXP" : "MOD_EXP_INV";
        if (o.nqubits < 4 || !o.data) fail(BF_EINVAL, "%s expects 4 parameters: n_exp, n_value, a, N", name);
        for (int k = 0; k < 4; ++k)
          if (o.data[k] != std::floor(o.data[k]) || std::fabs(o.data[k]) > 9.0e15)
            fail(BF_EINVAL, "%s parameters must be integers", name);
        const int64_t ne = (int64_t)o.data[0], nv = (int64_t)o.data[1], a = (int64_t)o.data[2], N = (int64_t)o.data[3];
        if (ne <= 0 || nv <= 0) fail(BF_EINVAL, "%s expects positive register sizes", name);
        if (N <= 1) fail(BF_EINVAL, "%s expects modulus > 1", name);
        int64_t x = ((a % N) + N) % N, y = N;  // gcd(a, N)
        while (y != 0) {
          int64_t t = x % y;
          x = y;
          y = t;
        }
        if (x != 1) fail(BF_EINVAL, "%s expects a and modulus to be coprime", name);
        if (ne + nv != n) fail(BF_EINVAL, "State size mismatch for %s", name);
        break;
      }
      case BF_OP_CLASSICAL_ORACLE: {
        if (o.nqubits < 0 || (o.nqubits > 0 && o.data == nullptr)) fail(BF_EINVAL, "oracle index list is null");
        double N = std::ldexp(1.0, n);
        for (int64_t k = 0; k < o.nqubits; ++k) {
          double v = o.data[k];
          if (!(v >= 0 && v < N) || v != std::floor(v)) fail(BF_EINVAL, "Oracle index out of range: %.17g", v);
        }
        break;
      }
      case BF_OP_MEASURE: {
        if (o.nqubits < 0 || (o.nqubits > 0 && o.qubits == nullptr)) fail(BF_EINVAL, "qubit list is null");
        uint64_t seen = 0;
        for (int64_t k = 0; k < o.nqubits; ++k) {
          check_qubit(o.qubits[k], n, "Target");
          if ((seen >> o.qubits[k]) & 1) fail(BF_EINVAL, "Duplicate target: %d", o.qubits[k]);
          seen |= 1ull << o.qubits[k];
          if (o.data && !(o.data[k] == -1.0 || o.data[k] == 0.0 || o.data[k] == 1.0))
            fail(BF_EINVAL, "Measurement values must be -1 (free), 0 or 1");
        }
        break;
      }
      case BF_OP_UNITARY:
      case BF_OP_CUNITARY: {
        int m = o.target2;
        if (m > 0 && (o.target < 0 || o.target + m > n)) fail(BF_EINVAL, "Target range out of bounds");
        if (o.kind == BF_OP_CUNITARY) {
          if (o.ncontrols != 1 || __builtin_popcountll(o.controls) != 1)
            fail(BF_EINVAL, "Controlled unitary expects exactly one control");
          int c = __builtin_ctzll(o.controls);
          check_qubit(c, n, "Control");
          if (m > 0 && c >= o.target && c < o.target + m) fail(BF_EINVAL, "Control overlaps target range");
        }
        if (m > 0 && o.data == nullptr) fail(BF_EINVAL, "Unitary data is null");
        break;
      }
      default:
        fail(BF_EINVAL, "Unknown transformation type: %d", o.kind);
    }
  }
}

// ---- lowering: GateInfo kind/arg -> matrix (gates.mojo:5-61) ---------------
static void gate_matrix(int kind, double a, const double* mat, double* m) {
  const double s = std::sqrt(0.5);
  auto set = [&](double a0, double a1, double a2, double a3, double a4, double a5, double a6, double a7) {
    m[0] = a0; m[1] = a1; m[2] = a2; m[3] = a3; m[4] = a4; m[5] = a5; m[6] = a6; m[7] = a7;
  };
  switch (kind) {
    case BF_GATE_H: set(s, 0, s, 0, s, 0, -s, 0); break;
    case BF_GATE_P: set(1, 0, 0, 0, 0, 0, std::cos(a), std::sin(a)); break;
    case BF_GATE_X: set(0, 0, 1, 0, 1, 0, 0, 0); break;
    case BF_GATE_Y: set(0, 0, 0, -1, 0, 1, 0, 0); break;
    case BF_GATE_Z: set(1, 0, 0, 0, 0, 0, -1, 0); break;
    case BF_GATE_RX: set(std::cos(a / 2), 0, 0, -std::sin(a / 2), 0, -std::sin(a / 2), std::cos(a / 2), 0); break;
    case BF_GATE_RY: set(std::cos(a / 2), 0, -std::sin(a / 2), 0, std::sin(a / 2), 0, std::cos(a / 2), 0); break;
    case BF_GATE_RZ: set(std::cos(a / 2), -std::sin(a / 2), 0, 0, 0, 0, std::cos(a / 2), std::sin(a / 2)); break;
    default: std::memcpy(m, mat, 8 * sizeof(double)); break;
  }
}

static void split_pairs(const double* m, float* mhl) {
  for (int i = 0; i < 8; ++i) {
    float hi = (float)m[i];
    mhl[2 * i] = hi;
    mhl[2 * i + 1] = (float)(m[i] - (double)hi);
  }
}

// Chooses the cheapest kernel form that computes the same matrix: the
// reference's specialised H/P/X/RY/CP/CX/CRY kernels (transformations_scalar.mojo
// :178-566) plus diagonal and permutation detection for any other kind.
GateInstr lower_gate(const bf_op& o, uint32_t spec) {
  GateInstr g;
  std::memset(&g, 0, sizeof g);
  g.target = o.target;
  g.cmask = o.controls;
  gate_matrix(o.gate, o.arg, o.mat, g.m);
  const double* m = g.m;
  const bool ctl0 = o.ncontrols == 0, ctl1 = o.ncontrols == 1;
  bool off_zero = m[2] == 0 && m[3] == 0 && m[4] == 0 && m[5] == 0;
  bool diag_zero = m[0] == 0 && m[1] == 0 && m[6] == 0 && m[7] == 0;
  if (o.gate == BF_GATE_H && ctl0 && (spec & BF_SPEC_H)) {
    g.kind = GK_H;
  } else if (diag_zero && m[2] == 1 && m[3] == 0 && m[4] == 1 && m[5] == 0) {
    g.kind = GK_SWAP;  // X, CX, CCX, MCX (and a CUSTOM X)
  } else if (off_zero && m[0] == 1 && m[1] == 0) {
    g.kind = GK_PHASE;  // P, Z, CP, CZ, MCP
  } else if (off_zero) {
    g.kind = GK_DIAG;  // RZ and other diagonals
  } else if ((o.gate == BF_GATE_RY && ((ctl0 && (spec & BF_SPEC_RY)) || (ctl1 && (spec & BF_SPEC_CRY)))) ||
             (m[1] == 0 && m[3] == 0 && m[5] == 0 && m[7] == 0 && m[0] == m[6] && m[2] == -m[4])) {
    g.kind = GK_RY;  // real rotation [[c, -s], [s, c]]
  } else {
    g.kind = m[1] == 0 ? GK_DENSE_R : GK_DENSE;  // U3: m00 = cos(theta/2) is real
  }
  split_pairs(g.m, g.mhl);
  return g;
}

double gate_bytes_fraction(const GateInstr& g) {
  int c = __builtin_popcountll(g.cmask);
  double f = (g.kind == GK_PHASE) ? 1.0 : 2.0;  // P touches half the amplitudes
  return f / std::ldexp(1.0, c);
}

// ---- tile-pass planning -----------------------------------------------------
// Greedy, order-respecting grouping.  Scanning the remaining gates in order,
// a gate joins the current pass if it commutes with every gate deferred so
// far and its target is (or can become) a tile qubit; otherwise it is
// deferred.  Two gates commute when, on every qubit they share, both act
// diagonally (controls always do; a diagonal gate does on its target).
static TileOp to_tile_op(const GateInstr& g, const int* loc_of) {
  TileOp t;
  std::memset(&t, 0, sizeof t);
  t.kind = g.kind;
  t.tglob = g.target;
  t.tloc = loc_of[g.target];
  t.um = g.um;
  t.uoff = g.uoff;
  for (int b = 0; b < 64; ++b) {
    if (!((g.cmask >> b) & 1)) continue;
    if (loc_of[b] >= 0) t.cmask_loc |= 1u << loc_of[b];
    else t.cmask_out |= 1ull << b;
  }
  std::memcpy(t.m, g.m, sizeof t.m);
  std::memcpy(t.mhl, g.mhl, sizeof t.mhl);
  return t;
}

// ---- phase fans --------------------------------------------------------------
// A phase gate of a tile pass, by the bits that must all be 1 (target among
// them), inside and outside the tile.
struct PhaseTerm {
  const TileOp* op;
  uint32_t loc;
  uint64_t out;
};

// a diagonal factor that may join a fan: products of several others could leave
// FP32's range where the gates one by one do not
static bool unit_factor(const double* m) { return std::fabs(m[6] * m[6] + m[7] * m[7] - 1.0) <= 1e-6; }

// A number per qubit mask (open addressing; 0 for a mask not seen before).
class MaskTable {
 public:
  uint32_t& operator[](uint64_t mask) {  // (mask != 0)
    if (2 * used_ >= keys_.size()) grow();
    const size_t i = find(mask);
    if (keys_[i] == 0) {
      keys_[i] = mask;
      ++used_;
    }
    return vals_[i];
  }

 private:
  size_t find(uint64_t mask) const {
    size_t i = (size_t)((mask * 0x9e3779b97f4a7c15ull) >> 32) & (keys_.size() - 1);
    while (keys_[i] != 0 && keys_[i] != mask) i = (i + 1) & (keys_.size() - 1);
    return i;
  }
  void grow() {
    std::vector<uint64_t> k(keys_.empty() ? 256 : 2 * keys_.size(), 0);
    std::vector<uint32_t> v(k.size(), 0);
    k.swap(keys_);
    v.swap(vals_);
    for (size_t o = 0; o < k.size(); ++o)
      if (k[o] != 0) {
        const size_t i = find(k[o]);
        keys_[i] = k[o];
        vals_[i] = v[o];
      }
  }
  std::vector<uint64_t> keys_;
  std::vector<uint32_t> vals_;
  size_t used_ = 0;
};

// The phases of a pass that wait for a gate on one of their qubits: one per
// mask, so that what waits (and the constants of a fan) is bounded by the
// masks that differ, and found by tile bit, so that a gate looks at the phases
// it meets and at no others.  (With a list of all, rescanned at every gate, a
// pass of 40,000 gates took 590 ms to plan, now 7.5.)
class PendingPhases {
 public:
  explicit PendingPhases(const TilePass& tp) : q_(tp.q) {}
  void add(const PhaseTerm& t) {
    uint64_t mask = t.out;
    for (uint32_t b = t.loc; b; b &= b - 1) mask |= 1ull << q_[__builtin_ctz(b)];
    uint32_t& id = at_[mask];  // 1 + the latest term of the mask
    if (id != 0 && live_[id - 1]) {
      TileOp*& own = own_[id - 1];
      if (!own) {
        ops_.push_back(*terms_[id - 1].op);
        terms_[id - 1].op = own = &ops_.back();
      }
      const double r = own->m[6] * t.op->m[6] - own->m[7] * t.op->m[7];
      own->m[7] = own->m[6] * t.op->m[7] + own->m[7] * t.op->m[6];
      own->m[6] = r;
      split_pairs(own->m, own->mhl);
      return;
    }
    id = (uint32_t)terms_.size() + 1;
    for (uint32_t b = t.loc; b; b &= b - 1) by_bit_[__builtin_ctz(b)].push_back(id - 1);
    terms_.push_back(t);
    own_.push_back(nullptr);
    live_.push_back(1);
  }
  // removes the phases on a bit of x (~0: all), in order of arrival
  std::vector<PhaseTerm> take(uint32_t x) {
    std::vector<uint32_t> ids;
    if (x == ~0u) {
      for (uint32_t i = 0; i < terms_.size(); ++i)
        if (live_[i]) ids.push_back(i);
    } else {
      for (; x; x &= x - 1) {
        std::vector<uint32_t>& l = by_bit_[__builtin_ctz(x)];
        for (uint32_t i : l)
          if (live_[i]) {
            live_[i] = 0;
            ids.push_back(i);
          }
        l.clear();
      }
      std::sort(ids.begin(), ids.end());
    }
    std::vector<PhaseTerm> out;
    out.reserve(ids.size());
    for (uint32_t i : ids) {
      out.push_back(terms_[i]);
      live_[i] = 0;
    }
    return out;
  }

 private:
  const int32_t* q_;
  std::deque<TileOp> ops_;  // products of several phases of a mask
  std::vector<PhaseTerm> terms_;
  std::vector<TileOp*> own_;  // a term's product in ops_, null while it is one op of the pass
  std::vector<char> live_;
  MaskTable at_;
  std::vector<uint32_t> by_bit_[32];  // terms by tile bit; taken ones drop out when read
};

// A fan needs at least this many phases: one alone touches a quarter or half
// of the tile as its own op, a fan half of it with up to two products.  With 3
// instead, random circuits of 9 to 24 qubits (half of their gates phases) take
// 1 to 6% longer, ZZ layers of 11 qubits 27% (complex128) and 32%.
constexpr int kMinFanTerms = 2;
// tables stay below this many doubles (32-bit offsets); phases beyond it
// remain ops of their own
constexpr size_t kMaxFanPool = (size_t)1 << 30;

// Whether a phase, its centre taken off, is a factor of the fan's tables (its
// tile bits within one half) or of its constant (no tile bits).
static bool fan_takes(const PhaseTerm& t, uint32_t centre_loc, uint64_t centre_out, int a) {
  const uint32_t l = t.loc & ~centre_loc;
  if (l == 0) return true;
  if (t.out & ~centre_out) return false;
  return (l >> a) == 0 || (l & ((1u << a) - 1u)) == 0;
}

// Hadamards without factors: values grow by up to 2^kMaxHalvings inside a pass
// (run_tile makes room for it where they are large).
constexpr int kMaxHalvings = 12;

// |m| of rows and columns 1 and orthogonal, to well above rounding
static bool is_unitary(const double* m, int dim) {
  for (int r = 0; r < dim; ++r)
    for (int c = 0; c <= r; ++c) {
      double re = 0, im = 0;
      for (int k = 0; k < dim; ++k) {
        const double *x = m + 2 * (k * dim + r), *y = m + 2 * (k * dim + c);
        re += x[0] * y[0] + x[1] * y[1];
        im += x[0] * y[1] - x[1] * y[0];
      }
      if (!(std::fabs(re - (r == c ? 1.0 : 0.0)) <= 1e-6 && std::fabs(im) <= 1e-6)) return false;
    }
  return true;
}

// One table: entry x is the product of the factors whose mask is within x.
static void fan_table(const std::vector<std::pair<uint32_t, const double*>>& terms, int bits, int shift, double* out) {
  std::vector<double> one(2 * (size_t)bits, 0.0);  // product per single-bit mask
  for (int b = 0; b < bits; ++b) one[2 * b] = 1.0;
  auto mul = [](double* x, const double* f) {
    const double r = x[0] * f[0] - x[1] * f[1];
    x[1] = x[0] * f[1] + x[1] * f[0];
    x[0] = r;
  };
  for (auto& t : terms) {
    const uint32_t m = t.first >> shift;
    if ((m & (m - 1)) == 0) mul(&one[2 * __builtin_ctz(m)], t.second);
  }
  out[0] = 1.0;
  out[1] = 0.0;
  for (int b = 0; b < bits; ++b)
    for (uint32_t x = 0; x < (1u << b); ++x) {
      double* d = out + 2 * ((1u << b) + x);
      d[0] = out[2 * x];
      d[1] = out[2 * x + 1];
      mul(d, &one[2 * b]);
    }
  for (auto& t : terms) {
    const uint32_t m = t.first >> shift;
    if ((m & (m - 1)) == 0) continue;
    for (uint32_t x = 0; x < (1u << bits); ++x)
      if ((x & m) == m) mul(out + 2 * x, t.second);
  }
}

int merge_phases(const TilePass& tp, std::vector<TileOp>& out, std::vector<double>* pool, int* halvings) {
  const size_t first = out.size();
  const int K = tp.K, a = K / 2;
  PendingPhases pending(tp);
  int slots = 0;                   // of the pass's constants in shared memory
  std::vector<uint32_t> fan_bits;  // by fan (an op's uoff): the tile bits of its phases
  // fills op's fan from the terms around one centre
  auto make_fan = [&](TileOp& op, const std::vector<PhaseTerm>& terms, uint32_t centre_loc) {
    std::vector<std::pair<uint32_t, const double*>> ta, tb;
    std::vector<const PhaseTerm*> consts;
    for (const PhaseTerm& t : terms) {
      const uint32_t l = t.loc & ~centre_loc;
      if (l == 0) consts.push_back(&t);
      else if ((l >> a) == 0) ta.emplace_back(l, t.op->m + 6);
      else tb.emplace_back(l, t.op->m + 6);
    }
    op.fan = consts.empty() ? 1 : ++slots;  // (a fan without constants reads none)
    op.uoff = (int32_t)fan_bits.size();
    fan_bits.push_back(0u);
    for (const PhaseTerm& t : terms) fan_bits.back() |= t.loc;
    op.fan_shape = a | (ta.empty() ? 0 : kFanA) | (tb.empty() ? 0 : kFanB);
    op.fan_consts = (int32_t)consts.size();
    if (!pool) return;
    op.fan_off = (int32_t)pool->size();
    const size_t na = (size_t)1 << a, nb = (size_t)1 << (K - a);
    pool->resize(pool->size() + 2 * (na + nb));
    fan_table(ta, a, 0, pool->data() + op.fan_off);
    fan_table(tb, K - a, a, pool->data() + op.fan_off + 2 * na);
    for (const PhaseTerm* t : consts) {
      double mask;
      std::memcpy(&mask, &t->out, sizeof mask);
      const double e[4] = {mask, 0.0, t->op->m[6], t->op->m[7]};
      pool->insert(pool->end(), e, e + 4);
    }
    pool->push_back(1.0);  // the constants' product starts from here
    pool->push_back(0.0);
  };
  // Emits terms as fans around the centre given (a tile bit) or, without
  // one, around the qubit most of them share, the rest as ops of their own.
  // `gate`: an uncontrolled single-target gate that a fan around its target
  // can join; true when one did.
  auto flush = [&](std::vector<PhaseTerm> terms, uint32_t centre, TileOp* gate) {
    bool joined = false;
    while (!terms.empty() && (!pool || pool->size() < kMaxFanPool)) {
      uint32_t cl = centre;
      uint64_t co = 0;
      if (!centre) {
        int cnt[32 + 64] = {};  // tile bits, then outside qubits
        for (const PhaseTerm& t : terms) {
          for (uint32_t b = t.loc; b; b &= b - 1) cnt[__builtin_ctz(b)] += fan_takes(t, b & (0u - b), 0, a);
          for (uint64_t b = t.out; b; b &= b - 1) cnt[32 + __builtin_ctzll(b)] += fan_takes(t, 0, b & (0ull - b), a);
        }
        const int best = (int)(std::max_element(cnt, cnt + 96) - cnt);
        if (cnt[best] > 0) {
          cl = best < 32 ? 1u << best : 0u;
          co = best < 32 ? 0ull : 1ull << (best - 32);
        }
      }
      std::vector<PhaseTerm> in, rest;
      for (const PhaseTerm& t : terms) {
        const bool constant = (t.loc & ~cl) == 0;
        if (((t.loc & cl) || (t.out & co)) && fan_takes(t, cl, co, a) && (!constant || slots < kMaxPassFans))
          in.push_back(t);
        else
          rest.push_back(t);
      }
      // one phase of the target alone costs a gate in hand one product
      const bool lone = gate && centre && in.size() == 1 && (in[0].loc & ~cl) == 0;
      if ((int)in.size() < kMinFanTerms && !lone) break;
      if (gate && centre) {
        make_fan(*gate, in, cl);
        joined = true;
      } else {
        TileOp f;
        std::memset(&f, 0, sizeof f);
        f.kind = GK_FAN;
        f.tloc = cl ? __builtin_ctz(cl) : -1;
        f.tglob = cl ? tp.q[f.tloc] : __builtin_ctzll(co);
        f.cmask_out = co;
        make_fan(f, in, cl);
        out.push_back(f);
      }
      terms.swap(rest);
      if (centre) break;
    }
    for (const PhaseTerm& t : terms) out.push_back(*t.op);
    return joined;
  };
  for (const TileOp& op : tp.ops) {
    if (op.kind == GK_PHASE && unit_factor(op.m)) {
      PhaseTerm t;
      t.op = &op;
      t.loc = op.cmask_loc | (op.tloc >= 0 ? 1u << op.tloc : 0u);
      t.out = op.cmask_out | (op.tloc < 0 ? 1ull << op.tglob : 0ull);
      pending.add(t);
      continue;
    }
    if (op.kind == GK_PHASE || op.kind == GK_DIAG) {  // commutes with every phase
      out.push_back(op);
      continue;
    }
    const bool uni = op.kind == GK_UNITARY;
    const uint32_t x = uni ? ((1u << op.um) - 1u) << op.tloc : 1u << op.tloc;
    const std::vector<PhaseTerm> met = pending.take(x);
    TileOp g = op;
    const bool joins = !uni && op.kind != GK_SWAP && !op.cmask_loc && !op.cmask_out;
    if (!met.empty()) flush(met, uni ? 0u : x, joins ? &g : nullptr);
    out.push_back(g);
  }
  flush(pending.take(~0u), 0u, nullptr);
  // A Hadamard goes into the next op on its target where that has a fan and
  // nothing between them touches the target: the pair is read and written once.
  auto touches = [&](const TileOp& op) {
    if (op.kind < 0) return 0u;
    uint32_t m = op.cmask_loc | (op.fan ? fan_bits[(size_t)op.uoff] : 0u);
    if (op.kind == GK_UNITARY) m |= ((1u << op.um) - 1u) << op.tloc;
    else if (op.tloc >= 0) m |= 1u << op.tloc;
    return m;
  };
  for (size_t k = first; k < out.size(); ++k) {
    if (!out[k].fan || out[k].kind == GK_FAN) continue;
    const uint32_t t = 1u << out[k].tloc;
    size_t j = k;
    while (j > first && !(touches(out[j - 1]) & t)) --j;
    if (j == first) continue;
    TileOp& h = out[j - 1];
    if (h.kind != GK_H || h.fan || h.tloc != out[k].tloc || h.cmask_loc || h.cmask_out) continue;
    out[k].um = GK_H;
    h.kind = -1;
  }
  out.erase(std::remove_if(out.begin() + (std::ptrdiff_t)first, out.end(), [](const TileOp& op) { return op.kind < 0; }),
            out.end());
  // pairs of Hadamards without their factors: u + v and u - v take 44 of a
  // Hadamard's 72 double-float instructions, and the exact 1/2 per pair costs
  // the store nothing; at most kMaxHalvings, and none in a pass with gates
  // that may make values grow by themselves
  auto is_h = [](const TileOp& op, bool before) {
    return before ? op.kind != GK_UNITARY && op.um == GK_H : op.kind == GK_H;
  };
  int h = 0;
  for (size_t k = first; k < out.size(); ++k) h += is_h(out[k], true) + is_h(out[k], false);
  auto preserves = [&](const TileOp& op) {
    if (op.kind == GK_UNITARY) return pool && is_unitary(pool->data() + op.uoff, 1 << op.um);
    return is_unitary(op.m, 2);
  };
  *halvings = h >= 2 && std::all_of(tp.ops.begin(), tp.ops.end(), preserves) ? std::min(h / 2, kMaxHalvings) : 0;
  h = 2 * *halvings;
  for (size_t k = first; k < out.size(); ++k) {
    if (is_h(out[k], true) && h > 0 && h--) out[k].um = GK_HU;
    if (is_h(out[k], false) && h > 0 && h--) out[k].kind = GK_HU;
  }
  return (int)fan_bits.size();
}

// The work a tile pass counts a gate for when tiles are compared: a diagonal
// gate joins any tile, and merges into a fan of whichever pass it runs in.
static double gate_work(const GateInstr& g) {
  return gate_bytes_fraction(g) * (gk_is_diagonal(g.kind) ? 0.02 : 1.0);
}

// The work (per-gate bytes, in units of S) a tile pass over the qubit set
// inQ takes from the remaining gates: a gate joins when its non-diagonal
// target is in the set and it commutes with every gate deferred before it.
static double pass_work(const std::vector<const GateInstr*>& remaining, uint64_t inQ, uint64_t all) {
  uint64_t blockedX = 0, blockedAll = 0;
  double w = 0;
  for (const GateInstr* g : remaining) {
    const uint64_t Xg = gate_xmask(*g);
    const uint64_t Ag = gate_amask(*g);
    if (!(Xg & blockedAll) && !(Ag & blockedX) && !(Xg & ~inQ)) {
      w += gate_work(*g);
    } else {
      blockedX |= Xg;
      blockedAll |= Ag;
      if ((blockedX & all) == all) break;  // every later gate meets a deferred one
    }
  }
  return w;
}

// The tensor-core blocks a pass over inQ would need: its gates grouped into
// blocks of at most 5 tile qubits and 3 outside qubits, each gate into the
// earliest block at or after the last one that shares a tile qubit with it
// (the grouping of plan_blocks); large when a gate cannot be placed.
static int pass_blocks(const std::vector<const GateInstr*>& remaining, uint64_t inQ, uint64_t all) {
  uint64_t blockedX = 0, blockedAll = 0;
  uint64_t bq[64], bo[64];
  int nb = 0;
  for (const GateInstr* g : remaining) {
    const uint64_t Xg = gate_xmask(*g);
    const uint64_t Ag = gate_amask(*g);
    if ((Xg & blockedAll) || (Ag & blockedX) || (Xg & ~inQ)) {
      blockedX |= Xg;
      blockedAll |= Ag;
      if ((blockedX & all) == all) break;
      continue;
    }
    const uint64_t Q = Ag & inQ, O = Ag & ~inQ;
    if (__builtin_popcountll(Q) > 5 || __builtin_popcountll(O) > 3) return 1000;
    int last = -1;
    for (int b = 0; b < nb; ++b)
      if (bq[b] & Q) last = b;
    int place = -1;
    for (int b = std::max(last, 0); b < nb; ++b)
      if (__builtin_popcountll(bq[b] | Q) <= 5 && __builtin_popcountll(bo[b] | O) <= 3) {
        place = b;
        break;
      }
    if (place < 0) {
      if (nb == 64) return 1000;
      bq[nb] = 0;
      bo[nb] = 0;
      place = nb++;
    }
    bq[place] |= Q;
    bo[place] |= O;
  }
  return nb;
}

// The CUDA-core tile kernel's cost of the gates a pass over inQ takes, in
// dense-gate units (core_units of the same gates), its phases merged into
// fans and those no gate of the pass meets left to a later one.
static double pass_core_units(const std::vector<const GateInstr*>& remaining, uint64_t inQ, uint64_t all, bool fp32) {
  uint64_t blockedX = 0, blockedAll = 0;
  double u = 0;
  // the phases that wait for a gate, one per mask (1: waiting), by qubit
  std::vector<uint64_t> by_qubit[64];
  MaskTable pending;
  uint64_t after_h = 0;  // qubits that nothing touched since a Hadamard: a fan there takes it in
  for (const GateInstr* g : remaining) {
    const uint64_t Xg = gate_xmask(*g);
    const uint64_t Ag = gate_amask(*g);
    if ((Xg & blockedAll) || (Ag & blockedX) || (Xg & ~inQ)) {
      blockedX |= Xg;
      blockedAll |= Ag;
      if ((blockedX & all) == all) break;
      continue;
    }
    if (g->kind == GK_PHASE && unit_factor(g->m)) {
      uint32_t& waits = pending[Ag];
      if (!waits)
        for (uint64_t b = Ag; b; b &= b - 1) by_qubit[__builtin_ctzll(b)].push_back(Ag);
      waits = 1;
      continue;
    }
    u += core_units(g->kind, g->um, fp32);
    if (Xg) {
      size_t met = 0;
      for (uint64_t b = Xg; b; b &= b - 1) {
        std::vector<uint64_t>& l = by_qubit[__builtin_ctzll(b)];
        for (uint64_t p : l) {
          uint32_t& waits = pending[p];
          met += waits;
          waits = 0;
        }
        l.clear();
      }
      const bool joins = Ag == Xg && g->kind != GK_SWAP && g->kind != GK_UNITARY;
      if (met >= (size_t)kMinFanTerms) {
        u += core_units(GK_FAN, joins, fp32);
        if (joins && (after_h & Xg)) u += core_units(GK_HU, 1, fp32) - core_units(GK_H, 0, fp32);
      } else if (met) {
        u += core_units(GK_PHASE, 0, fp32);
      }
    }
    after_h &= ~Ag;
    if (g->kind == GK_H) after_h |= Xg;
  }
  return u;
}

// Measured per op of a 12-qubit tile of 26 qubits, against a dense gate's 161
// us (double-float) and 40 us (FP32): exchange 60 to 80 and 29 to 40, one phase
// 61 and 22, diagonal 99 and 40, Hadamard 90 and 40 (52 and 7 within a fan's
// op), fan 113 and 45 alone and 84 to 110 and 21 to 27 with a gate.  An m-qubit
// unitary does 2^m complex products per amplitude against a dense gate's 2.
double core_units(int kind, int um, bool fp32) {
  switch (kind) {
    case GK_SWAP: return fp32 ? 0.8 : 0.5;
    case GK_PHASE: return fp32 ? 0.55 : 0.4;
    case GK_DIAG: return fp32 ? 1.0 : 0.6;
    case GK_H:
    case GK_HU: return um ? (fp32 ? 0.17 : 0.32) : (fp32 ? 1.0 : 0.45);
    case GK_FAN: return um || !fp32 ? 0.6 : 1.1;
    case GK_UNITARY: return (double)(1 << (um - 1));
    default: return 1.0;
  }
}

std::vector<PlanStep> plan_gates(int n, const std::vector<GateInstr>& gates, int K, bool allow_single,
                                 double block_units, double pass_cost, bool keep_wide_unitaries, bool fp32) {
  std::vector<PlanStep> steps;
  if (gates.empty()) return steps;
  K = std::max(1, std::min(K, std::min(n, kMaxTileQubits)));
  // Low qubits always in the tile; when the tile is narrower than the state
  // at least one slot stays free, so every pass can take the next gate.
  const int L = (K >= n) ? std::min(K, kTileLowQubits) : std::min(K - 1, kTileLowQubits);
  const uint64_t low = (L >= 64) ? ~0ull : ((1ull << L) - 1);
  std::vector<const GateInstr*> remaining;
  for (auto& g : gates) remaining.push_back(&g);
  while (!remaining.empty()) {
    // the tile's qubits: first the targets in order of appearance among the
    // gates that could still join (first come), then single swaps of a chosen
    // qubit for another target while that improves the pass: more work, or
    // for passes that run as tensor-core blocks more work per unit of time
    // (a pass costs about as much as pass_cost blocks besides its blocks)
    uint64_t inQ = low;
    int nQ = L;
    // the qubits the remaining gates touch: once the deferred gates act
    // non-diagonally on all of them, no later gate can join a pass
    uint64_t all = 0, all_x = 0;  // all_x: the qubits they act on non-diagonally
    for (const GateInstr* g : remaining) {
      all |= gate_amask(*g);
      all_x |= gate_xmask(*g);
    }
    {
      uint64_t blockedX = 0, blockedAll = 0;
      for (const GateInstr* g : remaining) {
        const uint64_t Xg = gate_xmask(*g);
        const uint64_t Ag = gate_amask(*g);
        bool fits = false;
        if (!(Xg & blockedAll) && !(Ag & blockedX)) {
          const int extra = __builtin_popcountll(Xg & ~inQ);
          if (extra == 0) {
            fits = true;
          } else if (nQ + extra <= K) {
            inQ |= Xg;
            nQ += extra;
            fits = true;
          }
        }
        if (!fits) {
          blockedX |= Xg;
          blockedAll |= Ag;
          if ((blockedX & all) == all) break;
        }
      }
    }
    bool blocks_chosen = false;
    if (nQ == K && K < n) {
      const uint64_t targets = all_x;
      auto search = [&](uint64_t start, auto score) {
        uint64_t set = start;
        double best = score(set);
        for (int round = 0; round < 8; ++round) {
          uint64_t best_set = set;
          for (int a = 0; a < n; ++a) {
            if (!((set >> a) & 1) || ((low >> a) & 1)) continue;
            for (int b = 0; b < n; ++b) {
              if (((set >> b) & 1) || !((targets >> b) & 1)) continue;
              const uint64_t cand = (set & ~(1ull << a)) | (1ull << b);
              const double w = score(cand);
              if (w > best + 1e-9) {
                best = w;
                best_set = cand;
              }
            }
          }
          if (best_set == set) break;
          set = best_set;
        }
        return set;
      };
      auto work = [&](uint64_t set) { return pass_work(remaining, set, all); };
      const uint64_t start = inQ;
      const uint64_t by_work = search(start, work);
      if (block_units > 0) {
        // Passes that may run as tensor-core blocks: the tile that takes the
        // most work per unit of time as blocks (a pass costs about pass_cost
        // blocks besides its blocks), kept when its blocks beat the CUDA-core kernel
        // on the same gates and it does more work per unit of time than the
        // most-work tile does on the CUDA cores (same pass cost; a block
        // costs block_units dense gates).
        auto block_rate = [&](uint64_t c) { return work(c) / (pass_cost + pass_blocks(remaining, c, all)); };
        const uint64_t set = search(start, block_rate);
        const double core = pass_core_units(remaining, set, all, fp32);
        const double core_rate = work(by_work) / (pass_cost + pass_core_units(remaining, by_work, all, fp32) / block_units);
        if ((double)pass_blocks(remaining, set, all) * block_units < core && block_rate(set) >= core_rate) {
          inQ = set;
          blocks_chosen = true;
        }
      }
      if (!blocks_chosen) inQ = by_work;
    }
    // deferred: those passed over up to `tail`, from where no gate can join
    std::vector<const GateInstr*> taken, deferred;
    std::vector<size_t> taken_at, deferred_at;  // their places in `remaining`
    size_t tail = 0;
    {
      uint64_t blockedX = 0, blockedAll = 0;
      for (; tail < remaining.size(); ++tail) {
        const GateInstr* g = remaining[tail];
        const uint64_t Xg = gate_xmask(*g);
        const uint64_t Ag = gate_amask(*g);
        if (!(Xg & blockedAll) && !(Ag & blockedX) && !(Xg & ~inQ)) {
          taken.push_back(g);
          taken_at.push_back(tail);
        } else {
          deferred.push_back(g);
          deferred_at.push_back(tail);
          blockedX |= Xg;
          blockedAll |= Ag;
          if ((blockedX & all) == all) {
            ++tail;
            break;
          }
        }
      }
    }
    // A phase that no gate of this pass meets goes back when a deferred gate
    // acts non-diagonally on one of its qubits: there it joins a fan that
    // pass applies anyway (20-qubit QFT: no fan of its own in any pass).  A
    // tile chosen for tensor-core blocks keeps it, as part of a block.
    if (!blocks_chosen) {
      uint64_t later = 0, met = 0;
      for (const GateInstr* g : deferred) later |= gate_xmask(*g);
      for (size_t i = tail; i < remaining.size() && later != all_x; ++i) later |= gate_xmask(*remaining[i]);
      std::vector<char> back(taken.size(), 0);
      bool any = false;
      for (size_t k = taken.size(); k-- > 0;) {
        const uint64_t Xg = gate_xmask(*taken[k]);
        met |= Xg;
        if (taken[k]->kind != GK_PHASE) continue;
        const uint64_t Ag = gate_amask(*taken[k]);
        back[k] = !(Ag & met) && (Ag & later);
        any |= back[k] != 0;
      }
      if (any) {
        std::vector<const GateInstr*> keep, merged;
        size_t d = 0;
        for (size_t k = 0; k < taken.size(); ++k) {
          if (!back[k]) {
            keep.push_back(taken[k]);
            continue;
          }
          while (d < deferred.size() && deferred_at[d] < taken_at[k]) merged.push_back(deferred[d++]);
          merged.push_back(taken[k]);
        }
        merged.insert(merged.end(), deferred.begin() + (std::ptrdiff_t)d, deferred.end());
        if (!keep.empty()) {
          taken.swap(keep);
          deferred.swap(merged);
        }
      }
    }
    if (taken.empty()) fail(BF_EINVAL, "internal: tile planner made no progress (K=%d, n=%d)", K, n);
    double single_bytes = 0;
    bool wide_unitary = false;
    for (const GateInstr* g : taken) {
      single_bytes += gate_bytes_fraction(*g);
      wide_unitary |= g->kind == GK_UNITARY && g->um >= 4;
    }
    // a tile pass moves 2S; the gates on their own move no more.  With
    // keep_wide_unitaries a unitary of 4 or 5 qubits stays a pass (one
    // tensor-core block): on its own, a double-float kernel does 2^m complex
    // products per amplitude (at 26 qubits a lone 5-qubit unitary took 8.2
    // ms that way and 1.9 ms as a digit pass; a 3-qubit one 1.8 ms either
    // way, so it keeps its kernel)
    if (allow_single && single_bytes <= 2.0 && !(wide_unitary && keep_wide_unitaries)) {
      for (const GateInstr* g : taken) {
        PlanStep st;
        st.is_tile = false;
        st.gate = *g;
        steps.push_back(st);
      }
    } else {
      // pad the tile with the lowest unused qubits up to K
      for (int q = 0; q < n && nQ < K; ++q)
        if (!((inQ >> q) & 1)) {
          inQ |= 1ull << q;
          nQ++;
        }
      PlanStep st;
      st.is_tile = true;
      st.tile.K = nQ;
      st.tile.L = L;
      int loc_of[64];
      for (int q = 0; q < 64; ++q) loc_of[q] = -1;
      int j = 0;
      for (int q = 0; q < n; ++q)
        if ((inQ >> q) & 1) {
          st.tile.q[j] = q;
          loc_of[q] = j;
          ++j;
        }
      for (const GateInstr* g : taken) st.tile.ops.push_back(to_tile_op(*g, loc_of));
      steps.push_back(std::move(st));
    }
    deferred.insert(deferred.end(), remaining.begin() + (std::ptrdiff_t)tail, remaining.end());
    remaining.swap(deferred);
  }
  return steps;
}

}  // namespace bf
