// tile_body.cuh — the shared-memory tile pass body, used by the single-state
// tile kernel (tile.cu) and the batched persistent kernel (batch.cu).
#pragma once

#include <cstring>
#include <type_traits>

#include "amp_math.cuh"
#include "bf_internal.h"

namespace bf {

constexpr int kTileThreads = 256;

struct TileGeom {
  int32_t K;
  int32_t L;        // low qubits (q[j] = j for j < L)
  int32_t q[kMaxTileQubits];
};

// One in-tile gate over all its pairs: the gate kind and whether it has
// controls inside the tile are compile-time, so the pair loop carries no
// dispatch; indices are 32-bit (a tile has at most 2^13 amplitudes).
template <class P, int KIND, bool kCtl>
__device__ __forceinline__ void tile_pairs(typename P::Smem* amp, int TS, int tloc, uint32_t cml,
                                           const typename P::Coef& g) {
  using R = typename P::R;
  using S = typename P::Smem;
  const uint32_t low = (1u << tloc) - 1u, tb = 1u << tloc;
#pragma unroll 2
  for (int p = threadIdx.x; p < (TS >> 1); p += kTileThreads) {
    const uint32_t i0 = (((uint32_t)p & ~low) << 1) | ((uint32_t)p & low);
    if (kCtl && (i0 & cml) != cml) continue;
    const uint32_t i1 = i0 | tb;
    if (KIND == GK_SWAP) {
      S t = amp[i0];
      amp[i0] = amp[i1];
      amp[i1] = t;
    } else if (KIND == GK_PHASE) {
      R v = P::from_smem(amp[i1]);
      P::cmul(v, g, 6);
      amp[i1] = P::to_smem(v);
    } else {
      R u = P::from_smem(amp[i0]), v = P::from_smem(amp[i1]);
      apply_pair<P>(KIND, u, v, g);
      amp[i0] = P::to_smem(u);
      amp[i1] = P::to_smem(v);
    }
  }
}

template <class P, bool kCtl>
__device__ __forceinline__ void tile_gate(int kind, typename P::Smem* amp, int TS, int tloc, uint32_t cml,
                                          const typename P::Coef& g) {
  switch (kind) {
    case GK_DENSE: tile_pairs<P, GK_DENSE, kCtl>(amp, TS, tloc, cml, g); break;
    case GK_H: tile_pairs<P, GK_H, kCtl>(amp, TS, tloc, cml, g); break;
    case GK_HU: tile_pairs<P, GK_HU, kCtl>(amp, TS, tloc, cml, g); break;
    case GK_SWAP: tile_pairs<P, GK_SWAP, kCtl>(amp, TS, tloc, cml, g); break;
    case GK_PHASE: tile_pairs<P, GK_PHASE, kCtl>(amp, TS, tloc, cml, g); break;
    case GK_DIAG: tile_pairs<P, GK_DIAG, kCtl>(amp, TS, tloc, cml, g); break;
    case GK_DENSE_R: tile_pairs<P, GK_DENSE_R, kCtl>(amp, TS, tloc, cml, g); break;
    default: tile_pairs<P, GK_RY, kCtl>(amp, TS, tloc, cml, g); break;
  }
}

// Phase fans.  Bound by FP32 issue (double-float) and by the shared-memory
// round trip per op (complex64), so what a phase costs is its pass over the
// tile: as an op of its own it reads, multiplies and writes a quarter or half
// of it behind a barrier.  The n(n-1)/2 phases of a Fourier transform become
// at most one fan per Hadamard, multiplied into the pair the Hadamard has in
// registers anyway: one or two complex products per pair whatever the number
// of phases.  At 24 qubits, complex128, executing the value encoding (24 P, 276
// CP, 48 H) took 5.39 ms as 46 digit blocks in 4 passes and takes 1.68 ms in 3
// tile passes with fans; at 27 qubits, complex64, 18.2 against 5.1 ms; the
// 20-qubit QFT, complex128, 0.40 against 0.12 ms.
//
// A phase fan as the CTA holds it: tables in shared memory (the constant
// folded into one of them), or with neither table the constant alone.
template <class P>
struct FanView {
  const typename P::Smem* A;
  const typename P::Smem* B;
  uint32_t amask;
  int abits;
  bool use_a, use_b;
  typename P::R c;
};

template <class P>
__device__ __forceinline__ typename P::R cmul_r(typename P::R x, const typename P::R& w) {
  P::cmul_by(x, w.re, w.im);
  return x;
}

template <class P>
__device__ __forceinline__ typename P::R fan_apply(const FanView<P>& f, typename P::R v, uint32_t i) {
  if (f.use_a) v = cmul_r<P>(v, P::from_smem(f.A[i & f.amask]));
  if (f.use_b) v = cmul_r<P>(v, P::from_smem(f.B[i >> f.abits]));
  if (!f.use_a && !f.use_b) v = cmul_r<P>(v, f.c);
  return v;
}

// One uncontrolled in-tile gate with a fan on its target: the fan multiplies
// the pair's second amplitude on its way into the gate (GK_FAN: alone),
// after the Hadamard `before` (0: none).  With the first-layer Hadamards of a
// 24-qubit value encoding taken along like this its passes take 1.64 against
// 1.97 ms.
template <class P, int KIND>
__device__ __forceinline__ void tile_pairs_fan(typename P::Smem* amp, int TS, int tloc, int before,
                                               const typename P::Coef& g, const FanView<P>& f) {
  using R = typename P::R;
  const uint32_t low = (1u << tloc) - 1u, tb = 1u << tloc;
#pragma unroll 1
  for (int p = threadIdx.x; p < (TS >> 1); p += kTileThreads) {
    const uint32_t i0 = (((uint32_t)p & ~low) << 1) | ((uint32_t)p & low);
    const uint32_t i1 = i0 | tb;
    R v = P::from_smem(amp[i1]);
    if (KIND == GK_FAN) {
      amp[i1] = P::to_smem(fan_apply<P>(f, v, i1));
      continue;
    }
    R u = P::from_smem(amp[i0]);
    if (before == GK_HU) P::sum_difference(u, v);
    else if (before == GK_H) P::hadamard(u, v);
    v = fan_apply<P>(f, v, i1);
    apply_pair<P>(KIND, u, v, g);
    amp[i0] = P::to_smem(u);
    amp[i1] = P::to_smem(v);
  }
}

// ---- complex64: two amplitudes at a time ---------------------------------------
// An FP32 gate is a few instructions per pair, so what a pass costs is the
// shared-memory and index instructions around them: each thread takes the
// amplitudes 2k and 2k + 1 as one 16-byte word (two pairs that differ in
// local bit 0, or for a target on bit 0 one pair).  The passes of a 27-qubit
// value encoding take 4.74 against 6.66 ms, of six layers of U3 and CX at 24
// qubits 2.17 against 2.33.
// The loops stay rolled: unrolled by two, the kinds of a mixed circuit no longer
// fit the instruction cache (500 gates of every kind at 24 qubits 5.20 ms, 4.66
// like this, 4.80 one amplitude at a time; a batch of 128 circuits 702 and 665 us).
struct Pair32 {
  PolF32::R a, b;  // local bit 0 = 0, 1
};
__device__ __forceinline__ Pair32 pair32(float4 w) { return Pair32{PolF32::R{w.x, w.y}, PolF32::R{w.z, w.w}}; }
__device__ __forceinline__ float4 word32(const Pair32& p) { return make_float4(p.a.re, p.a.im, p.b.re, p.b.im); }

// the fan on amplitudes i and i + 1 (i even)
__device__ __forceinline__ void fan_apply2(const FanView<PolF32>& f, Pair32& v, uint32_t i) {
  if (f.use_a) {
    const Pair32 w = pair32(*reinterpret_cast<const float4*>(f.A + (i & f.amask)));
    v.a = cmul_r<PolF32>(v.a, w.a);
    v.b = cmul_r<PolF32>(v.b, w.b);
  }
  if (f.use_b) {
    const PolF32::R w = PolF32::from_smem(f.B[i >> f.abits]);
    v.a = cmul_r<PolF32>(v.a, w);
    v.b = cmul_r<PolF32>(v.b, w);
  }
  if (!f.use_a && !f.use_b) {
    v.a = cmul_r<PolF32>(v.a, f.c);
    v.b = cmul_r<PolF32>(v.b, f.c);
  }
}

template <int KIND>
__device__ __forceinline__ void pair_op32(PolF32::R& u, PolF32::R& v, const PolF32::Coef& g) {
  if (KIND == GK_SWAP) {
    const PolF32::R t = u;
    u = v;
    v = t;
  } else if (KIND != GK_FAN) {
    apply_pair<PolF32>(KIND, u, v, g);
  }
}

// kCtl: controls inside the tile; kFan: a fan on the target, after the
// Hadamard `before` (such ops have no controls)
template <int KIND, bool kCtl, bool kFan>
__device__ __forceinline__ void tile_words(float2* amp, int TS, int tloc, uint32_t cml, const PolF32::Coef& g,
                                           int before, const FanView<PolF32>& f) {
  using P = PolF32;
  float4* amp4 = reinterpret_cast<float4*>(amp);
  if (tloc == 0) {
#pragma unroll 1
    for (int k = threadIdx.x; k < (TS >> 1); k += kTileThreads) {
      if (kCtl && ((uint32_t)(2 * k) & cml) != cml) continue;
      Pair32 p = pair32(amp4[k]);
      if (kFan) {
        if (before == GK_HU) P::sum_difference(p.a, p.b);
        else if (before == GK_H) P::hadamard(p.a, p.b);
        const uint32_t i = 2 * (uint32_t)k + 1;
        if (f.use_a) p.b = cmul_r<P>(p.b, P::from_smem(f.A[i & f.amask]));
        if (f.use_b) p.b = cmul_r<P>(p.b, P::from_smem(f.B[i >> f.abits]));
        if (!f.use_a && !f.use_b) p.b = cmul_r<P>(p.b, f.c);
      }
      pair_op32<KIND>(p.a, p.b, g);
      amp4[k] = word32(p);
    }
    return;
  }
  const uint32_t low = (1u << (tloc - 1)) - 1u, tb = 1u << (tloc - 1);
  const uint32_t need = cml >> 1;
  const bool odd_only = kCtl && (cml & 1u);
#pragma unroll 1
  for (uint32_t q = threadIdx.x; q < (uint32_t)(TS >> 2); q += kTileThreads) {
    const uint32_t w0 = ((q & ~low) << 1) | (q & low), w1 = w0 | tb;
    if (kCtl && (w0 & need) != need) continue;
    Pair32 v = pair32(amp4[w1]);
    if (KIND == GK_PHASE || KIND == GK_FAN) {  // the target's 1 half alone
      if (kFan) {
        fan_apply2(f, v, 2 * w1);
      } else {
        if (!odd_only) P::cmul(v.a, g, 6);
        P::cmul(v.b, g, 6);
      }
      amp4[w1] = word32(v);
      continue;
    }
    Pair32 u = pair32(amp4[w0]);
    if (kFan) {
      if (before == GK_HU) {
        P::sum_difference(u.a, v.a);
        P::sum_difference(u.b, v.b);
      } else if (before == GK_H) {
        P::hadamard(u.a, v.a);
        P::hadamard(u.b, v.b);
      }
      fan_apply2(f, v, 2 * w1);
    }
    if (!odd_only) pair_op32<KIND>(u.a, v.a, g);
    pair_op32<KIND>(u.b, v.b, g);
    amp4[w0] = word32(u);
    amp4[w1] = word32(v);
  }
}

template <bool kCtl, bool kFan>
__device__ __forceinline__ void tile_words_of(int kind, float2* amp, int TS, int tloc, uint32_t cml,
                                              const PolF32::Coef& g, int before, const FanView<PolF32>& f) {
  switch (kind) {
    case GK_H: tile_words<GK_H, kCtl, kFan>(amp, TS, tloc, cml, g, before, f); break;
    case GK_HU: tile_words<GK_HU, kCtl, kFan>(amp, TS, tloc, cml, g, before, f); break;
    case GK_SWAP: tile_words<GK_SWAP, kCtl, kFan>(amp, TS, tloc, cml, g, before, f); break;
    case GK_PHASE: tile_words<GK_PHASE, kCtl, kFan>(amp, TS, tloc, cml, g, before, f); break;
    case GK_DIAG: tile_words<GK_DIAG, kCtl, kFan>(amp, TS, tloc, cml, g, before, f); break;
    case GK_RY: tile_words<GK_RY, kCtl, kFan>(amp, TS, tloc, cml, g, before, f); break;
    case GK_FAN: tile_words<GK_FAN, kCtl, kFan>(amp, TS, tloc, cml, g, before, f); break;
    default: tile_words<GK_DENSE, kCtl, kFan>(amp, TS, tloc, cml, g, before, f); break;
  }
}

// One in-tile dense unitary on the consecutive local bits tloc .. tloc+UM-1:
// each thread takes whole groups of 2^UM amplitudes (the other bits fixed),
// reads them, forms U x (rows of the row-major matrix `um` in shared memory)
// and writes it back in place.
template <class P, int UM, bool kCtl>
__device__ __forceinline__ void tile_unitary(typename P::Smem* amp, int TS, int tloc, uint32_t cml,
                                             const typename P::Smem* um) {
  using R = typename P::R;
  constexpr int D = 1 << UM;
  const uint32_t low = (1u << tloc) - 1u;
  for (int g = threadIdx.x; g < (TS >> UM); g += kTileThreads) {
    const uint32_t base = (((uint32_t)g & ~low) << UM) | ((uint32_t)g & low);
    if (kCtl && (base & cml) != cml) continue;
    R x[D];
#pragma unroll
    for (int c = 0; c < D; ++c) x[c] = P::from_smem(amp[base | ((uint32_t)c << tloc)]);
#pragma unroll
    for (int r = 0; r < D; ++r) {
      R acc = P::zero();
#pragma unroll
      for (int c = 0; c < D; ++c) acc = P::fma(P::from_smem(um[r * D + c]), x[c], acc);
      amp[base | ((uint32_t)r << tloc)] = P::to_smem(acc);
    }
  }
}

// A wider in-tile unitary (UM = 4 or 5 qubits): a thread's outputs (rows of
// groups) are formed from the group's inputs in shared memory into
// registers, 2 per thread at a time over whole groups, then written after
// a barrier (the groups of one round are disjoint from the next round's).
// The staged matrix is transposed (`umt[c * D + r]`), so that the lanes of a
// warp, which take consecutive rows of a group, read consecutive entries.
// Every thread runs the same number of rounds (the barriers are uniform).
template <class P, int UM, bool kCtl>
__device__ __forceinline__ void tile_unitary_wide(typename P::Smem* amp, int TS, int tloc, uint32_t cml,
                                                  const typename P::Smem* umt) {
  using R = typename P::R;
  constexpr int D = 1 << UM;
  constexpr int kPer = 2;  // outputs per thread per round (more cost registers of every unitary pass)
  const uint32_t low = (1u << tloc) - 1u;
  for (int round = 0; round < TS; round += kPer * kTileThreads) {
    R out[kPer];
    uint32_t where[kPer];
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
      const int o = round + j * kTileThreads + (int)threadIdx.x;
      where[j] = 0xffffffffu;
      if (o >= TS) continue;
      const uint32_t g = (uint32_t)o >> UM, r = (uint32_t)o & (D - 1);
      const uint32_t base = ((g & ~low) << UM) | (g & low);
      if (kCtl && (base & cml) != cml) continue;
      R acc = P::zero();
#pragma unroll 1
      for (int c = 0; c < D; ++c)
        acc = P::fma(P::from_smem(umt[c * D + r]), P::from_smem(amp[base | ((uint32_t)c << tloc)]), acc);
      out[j] = acc;
      where[j] = base | (r << tloc);
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kPer; ++j)
      if (where[j] != 0xffffffffu) amp[where[j]] = P::to_smem(out[j]);
  }
}

// bytes of shared memory before the staged unitary matrix (16-byte aligned)
template <class P>
__host__ __device__ inline size_t tile_umat_offset(int K, int L) {
  return ((((size_t)1 << K) * sizeof(typename P::Smem) + ((size_t)1 << (K - L)) * sizeof(uint64_t)) + 15) &
         ~(size_t)15;
}

// The arithmetic of a fan's constant and of its product with a table entry: at
// complex64 FP32 pairs, so that what an amplitude is multiplied by is rounded
// once whatever the number of factors.  With the products rounded one by one
// the error of a value encoding's state was 9.4e-8 at 9 and 1.8e-7 at 20
// qubits, 8.9e-8 and 1.2e-7 like this, for 5.50 against 5.44 ms at 27 qubits.
template <class P>
using FanPol = std::conditional_t<std::is_same<P, PolF32>::value, PolDF, P>;

// shared memory of the fans: the pass's constants, then the current op's
// tables (2^a + 2^(K-a) entries, a = K / 2)
template <class P>
__host__ __device__ inline size_t tile_fan_bytes(int K) {
  return kMaxPassFans * sizeof(typename FanPol<P>::Smem) +
         (((size_t)1 << (K / 2)) + ((size_t)1 << (K - K / 2))) * sizeof(typename P::Smem);
}

// One tile: load the 2^K amplitudes of tile `tile` (the non-tile qubits set
// to the bits of `tile`), apply ops[0..nops) in shared memory, store.  Called
// by every thread of a CTA of kTileThreads threads; `smem_raw` holds
// tile_smem_bytes(K, L) bytes.
// kL2Loads: read the state with L2-only loads (__ldcg).  Needed when other
// CTAs of the same launch wrote these amplitudes earlier (L1 is not coherent
// across SMs); a separate launch per pass does not need it.
// kUnitaries: the ops may include GK_UNITARY (their register-heavy loop is
// compiled only into this form; passes without them keep the lean one);
// pool then holds their matrices (row-major interleaved FP64), and
// `smem_raw` also holds the staged matrix.
// kFans: the ops may carry phase fans; pool then holds their tables and
// constants, and `smem_raw` also holds the staged ones (tile_smem_bytes).
// The results are stored times 2^-halvings; where an amplitude of the tile is
// so large that the factor-free Hadamards could leave the arithmetic's range,
// the tile is scaled before its ops instead: a vote at the barrier that follows
// the loads, 24-qubit value encoding 1683 against 1674 us without.  (A half at
// every second of these Hadamards, without a vote: 1775.)
template <class P, bool kL2Loads = false, bool kUnitaries = false, bool kFans = false>
__device__ __forceinline__ void run_tile(typename P::Glob* __restrict__ s, const TileOp* __restrict__ ops, int nops,
                                         const TileGeom& geo, uint64_t tile, unsigned char* smem_raw,
                                         const double* __restrict__ pool, int halvings) {
  using R = typename P::R;
  using S = typename P::Smem;
  const int K = geo.K, L = geo.L;
  const int TS = 1 << K;
  S* amp = reinterpret_cast<S*>(smem_raw);
  uint64_t* hoff = reinterpret_cast<uint64_t*>(smem_raw + (size_t)TS * sizeof(S));
  const int tid = threadIdx.x;

  // global index of local element 0: `tile` with zero bits inserted at the
  // tile positions (ascending).
  uint64_t obase = tile;
  for (int j = 0; j < K; ++j) obase = insert_zero_bit(obase, geo.q[j]);

  const int H = K - L;
  for (int h = tid; h < (1 << H); h += kTileThreads) {
    uint64_t off = 0;
    for (int j = 0; j < H; ++j)
      if ((h >> j) & 1) off |= 1ull << geo.q[L + j];
    hoff[h] = off;
  }
  __syncthreads();

  using FP = FanPol<P>;
  using FR = typename FP::R;
  using FS = typename FP::Smem;
  auto pool_at = [&](const double* d) { return FP::from_glob(__ldg(reinterpret_cast<const double2*>(d))); };
  FS* fan_c = reinterpret_cast<FS*>(smem_raw + tile_umat_offset<P>(K, L) +
                                    (kUnitaries ? ((size_t)1 << (2 * kTileUnitaryMax)) * sizeof(S) : 0));
  S* fan_a = reinterpret_cast<S*>(fan_c + kMaxPassFans);
  auto rounded = [](const FR& w) {
    if constexpr (std::is_same<P, PolF32>::value) return R{w.re.hi + w.re.lo, w.im.hi + w.im.lo};
    else return w;
  };
  if constexpr (kFans) {
    // the fans' constants for this CTA's outside bits, one warp per fan: the
    // lanes' factors multiplied by butterfly shuffles
    const int lane = tid & 31;
    for (int i = tid >> 5; i < nops; i += kTileThreads / 32) {
      const int slot = __ldg(&ops[i].fan), nc = __ldg(&ops[i].fan_consts);
      if (slot == 0 || nc == 0) continue;
      const double* c = pool + __ldg(&ops[i].fan_off) + 2 * ((1 << (K / 2)) + (1 << (K - K / 2)));
      FR acc = pool_at(c + 4 * nc);  // one
      for (int k = lane; k < nc; k += 32) {
        const uint64_t m = (uint64_t)__double_as_longlong(__ldg(c + 4 * k));
        if ((obase & m) == m) acc = cmul_r<FP>(acc, pool_at(c + 4 * k + 2));
      }
      int span = 1;
      while (span < nc && span < 32) span <<= 1;
      for (int off = span >> 1; off > 0; off >>= 1) {
        FS o = FP::to_smem(acc), r;
        constexpr int kWords = sizeof(FS) / 4;
        unsigned int w[kWords], x[kWords];
        memcpy(w, &o, sizeof o);
#pragma unroll
        for (int q = 0; q < kWords; ++q) x[q] = __shfl_xor_sync(0xffffffffu, w[q], off);
        memcpy(&r, x, sizeof r);
        acc = cmul_r<FP>(acc, FP::from_smem(r));
      }
      if (lane == 0) fan_c[slot - 1] = FP::to_smem(acc);
    }
  }

  const int lowmask = (1 << L) - 1;
  // complex64: two amplitudes per access where qubit 0 is a tile qubit
  const bool words = std::is_same<P, PolF32>::value && L > 0;
  bool large = false;
  if (words) {
    for (int k = tid; k < (TS >> 1); k += kTileThreads) {
      const uint64_t gi = obase | (uint64_t)((2 * k) & lowmask) | hoff[(2 * k) >> L];
      const float4* p = reinterpret_cast<const float4*>(s + gi);
      const float4 w = kL2Loads ? __ldcg(p) : *p;
      if constexpr (std::is_same<P, PolF32>::value) large |= P::large(R{w.x, w.y}) || P::large(R{w.z, w.w});
      reinterpret_cast<float4*>(amp)[k] = w;
    }
  } else {
    for (int e = tid; e < TS; e += kTileThreads) {
      uint64_t gi = obase | (uint64_t)(e & lowmask) | hoff[e >> L];
      const R r = P::from_glob(kL2Loads ? __ldcg(s + gi) : s[gi]);
      large |= P::large(r);
      amp[e] = P::to_smem(r);
    }
  }
  // (the warp reduction makes the branch uniform for the compiler: without it
  // the op loop keeps its descriptors in per-thread registers, 64 instead of 40)
  if (__reduce_or_sync(0xffffffffu, (unsigned)__syncthreads_or(large && halvings > 0)) != 0) {
#pragma unroll 1
    for (int e = tid; e < TS; e += kTileThreads) amp[e] = P::to_smem(P::scaled(P::from_smem(amp[e]), halvings));
    halvings = 0;
    __syncthreads();
  }

  for (int i = 0; i < nops; ++i) {
    const TileOp* op = ops + i;
    const uint64_t cmo = __ldg(&op->cmask_out);
    if ((obase & cmo) != cmo) continue;  // CTA-uniform
    const int kind = __ldg(&op->kind);
    const int tloc = __ldg(&op->tloc);
    const uint32_t cml = __ldg(&op->cmask_loc);
    if (kUnitaries && kind == GK_UNITARY) {
      // stage the matrix, then every group of the tile
      const int um = __ldg(&op->um);
      const double* u = pool + __ldg(&op->uoff);
      S* mat = reinterpret_cast<S*>(smem_raw + tile_umat_offset<P>(K, L));
      const int dim = 1 << um;
      for (int e = tid; e < dim * dim; e += kTileThreads) {
        typename P::Glob gv;
        if constexpr (sizeof(typename P::Glob) == 16) gv = make_double2(__ldg(u + 2 * e), __ldg(u + 2 * e + 1));
        else gv = make_float2((float)__ldg(u + 2 * e), (float)__ldg(u + 2 * e + 1));
        // row-major for the narrow forms, transposed for the wide ones
        const int at = um <= 3 ? e : (e % dim) * dim + e / dim;
        mat[at] = P::to_smem(P::from_glob(gv));
      }
      __syncthreads();
      switch (um) {
        case 2:
          if (cml) tile_unitary<P, 2, true>(amp, TS, tloc, cml, mat);
          else tile_unitary<P, 2, false>(amp, TS, tloc, 0u, mat);
          break;
        case 3:
          if (cml) tile_unitary<P, 3, true>(amp, TS, tloc, cml, mat);
          else tile_unitary<P, 3, false>(amp, TS, tloc, 0u, mat);
          break;
        case 4:
          if (cml) tile_unitary_wide<P, 4, true>(amp, TS, tloc, cml, mat);
          else tile_unitary_wide<P, 4, false>(amp, TS, tloc, 0u, mat);
          break;
        default:
          if (cml) tile_unitary_wide<P, 5, true>(amp, TS, tloc, cml, mat);
          else tile_unitary_wide<P, 5, false>(amp, TS, tloc, 0u, mat);
          break;
      }
      __syncthreads();
      continue;
    }
    const typename P::Coef g = P::coef(op->m, op->mhl);
    if (kFans && __ldg(&op->fan) != 0) {
      const int shape = __ldg(&op->fan_shape), nc = __ldg(&op->fan_consts);
      FanView<P> f;
      f.use_a = (shape & kFanA) != 0;
      f.use_b = (shape & kFanB) != 0;
      f.abits = K / 2;
      f.amask = (1u << f.abits) - 1u;
      f.A = fan_a;
      f.B = fan_a + (1 << f.abits);
      const FS* cs = fan_c + (__ldg(&op->fan) - 1);
      if (f.use_a || f.use_b) {
        // the tables, the constant folded into B (or the only table)
        const int na = 1 << f.abits, nt = na + (1 << (K - f.abits));
        if (tid < nt && (tid < na ? f.use_a : f.use_b)) {
          FR w = pool_at(pool + __ldg(&op->fan_off) + 2 * tid);
          if (nc && (tid >= na || !f.use_b)) w = cmul_r<FP>(w, FP::from_smem(*cs));
          fan_a[tid] = P::to_smem(rounded(w));
        }
        __syncthreads();
      } else {
        f.c = rounded(FP::from_smem(*cs));
      }
      if (tloc < 0) {  // the centre is outside the tile (and set): every amplitude
        for (int e = tid; e < TS; e += kTileThreads) amp[e] = P::to_smem(fan_apply<P>(f, P::from_smem(amp[e]), e));
      } else if constexpr (std::is_same<P, PolF32>::value) {
        tile_words_of<false, true>(kind, amp, TS, tloc, 0u, g, __ldg(&op->um), f);
      } else {
        const int before = __ldg(&op->um);
        switch (kind) {
          case GK_FAN: tile_pairs_fan<P, GK_FAN>(amp, TS, tloc, before, g, f); break;
          case GK_H: tile_pairs_fan<P, GK_H>(amp, TS, tloc, before, g, f); break;
          case GK_HU: tile_pairs_fan<P, GK_HU>(amp, TS, tloc, before, g, f); break;
          case GK_DENSE_R: tile_pairs_fan<P, GK_DENSE_R>(amp, TS, tloc, before, g, f); break;
          case GK_RY: tile_pairs_fan<P, GK_RY>(amp, TS, tloc, before, g, f); break;
          default: tile_pairs_fan<P, GK_DENSE>(amp, TS, tloc, before, g, f); break;
        }
      }
    } else if (tloc >= 0) {
      if constexpr (std::is_same<P, PolF32>::value) {
        const FanView<P> none{};
        if (cml) tile_words_of<true, false>(kind, amp, TS, tloc, cml, g, 0, none);
        else tile_words_of<false, false>(kind, amp, TS, tloc, 0u, g, 0, none);
      } else {
        if (cml) tile_gate<P, true>(kind, amp, TS, tloc, cml, g);
        else tile_gate<P, false>(kind, amp, TS, tloc, 0u, g);
      }
    } else {
      // diagonal gate, target outside the tile: one entry for the whole CTA
      const int tg = __ldg(&op->tglob);
      const int bit = (int)((obase >> tg) & 1);
      if (kind == GK_PHASE && bit == 0) continue;  // CTA-uniform
      const typename P::E c = bit ? g.v[6] : g.v[0], sn = bit ? g.v[7] : g.v[1];
      for (int e = tid; e < TS; e += kTileThreads) {
        if ((e & cml) != cml) continue;
        R x = P::from_smem(amp[e]);
        P::cmul_by(x, c, sn);
        amp[e] = P::to_smem(x);
      }
    }
    __syncthreads();
  }

  if (words) {
    const float f = __int_as_float((127 - halvings) << 23);
    for (int k = tid; k < (TS >> 1); k += kTileThreads) {
      const uint64_t gi = obase | (uint64_t)((2 * k) & lowmask) | hoff[(2 * k) >> L];
      const float4 w = reinterpret_cast<const float4*>(amp)[k];
      *reinterpret_cast<float4*>(s + gi) = make_float4(w.x * f, w.y * f, w.z * f, w.w * f);
    }
    return;
  }
  for (int e = tid; e < TS; e += kTileThreads) {
    uint64_t gi = obase | (uint64_t)(e & lowmask) | hoff[e >> L];
    s[gi] = P::to_glob_halved(P::from_smem(amp[e]), halvings);
  }
}

// shared memory of run_tile; with_unitary: room for a staged
// 2^kTileUnitaryMax-square matrix; with_fans: for the phase fans
template <class P>
inline size_t tile_smem_bytes(int K, int L, bool with_unitary = false, bool with_fans = false) {
  if (!with_unitary && !with_fans)
    return ((size_t)1 << K) * sizeof(typename P::Smem) + ((size_t)1 << (K - L)) * sizeof(uint64_t);
  return tile_umat_offset<P>(K, L) +
         (with_unitary ? ((size_t)1 << (2 * kTileUnitaryMax)) * sizeof(typename P::Smem) : 0) +
         (with_fans ? tile_fan_bytes<P>(K) : 0);
}

}  // namespace bf
