// measure.cu — measurement and readout of a device state.
//
//  * bf_probabilities: outcome probabilities over a list of qubits (the
//    reduction of apply_measure, state.mojo:466-501), optionally restricted
//    to amplitudes whose other listed qubits have fixed values.
//  * bf_measure: apply_measure (state.mojo:447-553) — reduction, the
//    reference's seeded draw (seed mod 2^31-1, times 48271 mod 2^31-1,
//    scaled by the total), collapse onto the drawn outcome and
//    renormalisation by 1/sqrt(p).
//  * bf_probs_topk: the k most probable basis states.
// Reductions accumulate |amp|^2 in double-float per thread and finish in
// FP64 on the host.
#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "amp_math.cuh"
#include "bf_internal.h"

namespace bf {

constexpr int kMeasThreads = 256;
constexpr int kMaxOutcomeBits = 20;
constexpr int kMargTileBits = 11;                                 // 2048 amplitudes: 32 KiB at complex128
constexpr int kMargCtas = 5;                                      // resident per SM (48 registers)
constexpr uint64_t kMargHostSums = 2048;
constexpr int kMargPer = (1 << kMargTileBits) / kMeasThreads;     // tile positions per thread

// Outcome probabilities.  The state is read in tiles of 2^T amplitudes: its
// lowest T index bits that no fixed qubit takes.  A CTA owns one setting of the
// listed free qubits above the tile and walks the settings of the summed-out
// ones there, each thread adding |amp|^2 to the same eight tile positions in
// registers.  Only then are the tile's own summed-out bits folded, once, in
// registers, between lanes and through shared memory, and the tile's outcomes
// written.  A long walk is cut into chunks so that the grid fills the GPU; the
// host or k_marginal_chunks adds the chunks' sums.
//
// A tile is contiguous when no fixed qubit lies in its range (kMargRun).  It
// was contiguous whatever is fixed before, and 11 low fixed qubits of 28 left
// one live amplitude of 2048 per step: 717 us, 32 like this.
//
// Bound by HBM: the state is read once in 32 KiB runs (8 independent 16-byte
// loads per thread in flight).  One CTA per outcome, which this replaces, read
// 2^20 outcomes of 16 amplitudes as 2^20 CTAs and finished them on the host.
// A 20-qubit register of 24 (complex128): 5.26 ms then, 0.64 ms now, most of
// it the 8 MiB result's copy; 16 of 28 (complex128): 2.64 against 0.75 ms,
// 0.84 of the copy bandwidth; 16 of 29 (complex64): 5.19 against 0.70 ms.
enum { kMargRun, kMargSpread, kMargPart };  // a contiguous tile, a whole one, less than one
struct MargArgs {
  int32_t tile_bits;       // T
  uint64_t tile_mask;      // the tile's index bits
  uint64_t row[kMargPer];  // index of tile position j * kMeasThreads
  int8_t lane_pos[8];      // index bits of the tile's lowest 8 (of all there are)
  uint64_t fixed_val;      // the fixed qubits' required bits
  uint64_t free_high;      // free listed qubits above the tile
  uint64_t sum_high;       // summed-out qubits above the tile
  uint64_t steps;          // 2^popcount(sum_high)
  uint64_t per_chunk;      // of them per CTA
  uint32_t chunks;         // CTAs per setting of free_high
  uint64_t outcomes;
  int32_t nfree_low;
  uint32_t keep;           // their bits in a tile position
  int8_t low_pos[kMaxOutcomeBits];   // tile positions of the free qubits inside it, ascending
  int8_t low_out[kMaxOutcomeBits];   // their bit in the outcome index
  int8_t high_out[kMaxOutcomeBits];  // outcome bits of free_high, ascending
};

template <class T>
__device__ __forceinline__ dfl prob_df(T a);
template <>
__device__ __forceinline__ dfl prob_df<double2>(double2 a) {
  dfl r = df_from_double(a.x), i = df_from_double(a.y);
  return df_dot2(r, r, i, i);
}
template <>
__device__ __forceinline__ dfl prob_df<float2>(float2 a) {
  return df_squares(a.x, a.y);
}

// the bits of x spread over the set positions of mask, ascending
__host__ __device__ __forceinline__ uint64_t deposit_mask(uint64_t x, uint64_t mask) {
  uint64_t r = 0;
  for (; x && mask; x >>= 1) {
    const uint64_t low = mask & (0 - mask);
    if (x & 1) r |= low;
    mask ^= low;
  }
  return r;
}

// A streaming load that stays where it is written: left to itself, the
// compiler moves each of a thread's loads to its use, and two instead of
// eight are in flight (16 of 28 qubits, complex128: 1.13 against 0.87 ms).
__device__ __forceinline__ void load_now(double2& v, const double2* p) {
  asm volatile("ld.global.cs.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
}
__device__ __forceinline__ void load_now(float2& v, const float2* p) {
  asm volatile("ld.global.cs.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
}

template <class T>
__global__ void __launch_bounds__(kMeasThreads, kMargCtas) k_marginal(const T* __restrict__ s, const MargArgs a,
                                                           double* __restrict__ out) {
  __shared__ dfl sum[1 << kMargTileBits];
  const uint64_t h = blockIdx.x / a.chunks, chunk = blockIdx.x % a.chunks;
  const uint32_t size = 1u << a.tile_bits;
  const bool run = a.tile_mask == (1u << kMargTileBits) - 1u;
  uint64_t lane = threadIdx.x;
  if (!run) {
    lane = 0;
#pragma unroll
    for (int b = 0; b < 8; ++b) lane |= (uint64_t)((threadIdx.x >> b) & 1u) << a.lane_pos[b];
  }
  const uint64_t base = a.fixed_val | deposit_mask(h, a.free_high) |
                        lane;
  dfl acc[kMargPer];
#pragma unroll
  for (int j = 0; j < kMargPer; ++j) acc[j] = dfl{0.f, 0.f};
  const uint64_t first = chunk * a.per_chunk, last = min(first + a.per_chunk, a.steps);
  // the summed-out bits step by masked addition: the ones between them carry
  uint64_t r = deposit_mask(first, a.sum_high);
  auto walk = [&](auto form) {
    for (uint64_t k = first; k < last; ++k, r = ((r | ~a.sum_high) + 1) & a.sum_high) {
      const T* p = s + (base | r);
      T v[kMargPer];
#pragma unroll
      for (int j = 0; j < kMargPer; ++j) {
        if constexpr (decltype(form)::value == kMargRun) load_now(v[j], p + j * kMeasThreads);
        if constexpr (decltype(form)::value == kMargSpread) load_now(v[j], p + a.row[j]);
        if constexpr (decltype(form)::value == kMargPart) {
          v[j] = T{};
          if (threadIdx.x + j * kMeasThreads < size) load_now(v[j], p + a.row[j]);
        }
      }
#pragma unroll
      for (int j = 0; j < kMargPer; ++j) acc[j] = df_add(acc[j], prob_df<T>(v[j]));
    }
  };
  if (run) walk(std::integral_constant<int, kMargRun>{});
  else if (a.tile_bits == kMargTileBits) walk(std::integral_constant<int, kMargSpread>{});
  else walk(std::integral_constant<int, kMargPart>{});
  // Fold the tile bits that are not outcome bits: the three highest between
  // the thread's own sums, the five lowest between the lanes, the three in
  // between through shared memory.
  const uint32_t gone = (size - 1u) & ~a.keep;
#pragma unroll
  for (int b = 2; b >= 0; --b) {
    if (!((gone >> (8 + b)) & 1u)) continue;
#pragma unroll
    for (int j = 0; j < kMargPer; ++j)
      if (!((j >> b) & 1)) acc[j] = df_add(acc[j], acc[j | (1 << b)]);
  }
  for (int b = 0; b < 5; ++b) {
    if (!((gone >> b) & 1u)) continue;
#pragma unroll
    for (int j = 0; j < kMargPer; ++j)
      if (!(((uint32_t)j << 8) & gone))
        acc[j] = df_add(acc[j], dfl{__shfl_xor_sync(0xffffffffu, acc[j].hi, 1 << b),
                                    __shfl_xor_sync(0xffffffffu, acc[j].lo, 1 << b)});
  }
#pragma unroll
  for (int j = 0; j < kMargPer; ++j) {
    const uint32_t e = threadIdx.x + j * kMeasThreads;
    if (e < size && !(e & gone & 0x71fu)) sum[e] = acc[j];
  }
  __syncthreads();
  uint64_t oh = 0;
  for (int i = 0; (h >> i) != 0; ++i) oh |= ((h >> i) & 1) << a.high_out[i];
  for (uint32_t k = threadIdx.x; k < (1u << a.nfree_low); k += kMeasThreads) {
    uint32_t e = 0;
    uint64_t o = oh;
    for (int i = 0; i < a.nfree_low; ++i) {
      e |= ((k >> i) & 1u) << a.low_pos[i];
      o |= (uint64_t)((k >> i) & 1u) << a.low_out[i];
    }
    dfl v = sum[e];
    if (gone & 0xe0u) {
      dfl w[8];
#pragma unroll
      for (uint32_t x = 0; x < 8; ++x) w[x] = (x << 5) & ~gone ? dfl{0.f, 0.f} : sum[e | (x << 5)];
#pragma unroll
      for (int half = 4; half > 0; half >>= 1)
        for (int x = 0; x < half; ++x) w[x] = df_add(w[x], w[x + half]);
      v = w[0];
    }
    out[chunk * a.outcomes + o] = (double)v.hi + (double)v.lo;
  }
}

// out[o] = sum over chunks of in[c * outcomes + o]: `width` outcomes (a power
// of two) by 256 / width chunk lanes per CTA, the lanes' sums folded by halves.
// The width leaves a lane about eight chunks: with 8 lanes whatever the counts,
// the 1024 chunks of one outcome at 22 qubits were a chain of 128 loads, and
// the call took 55 us (30 now).
__global__ void __launch_bounds__(256) k_marginal_chunks(const double* __restrict__ in, uint64_t outcomes,
                                                         uint32_t chunks, uint32_t width, double* __restrict__ out) {
  __shared__ double part[256];
  const uint32_t x = threadIdx.x & (width - 1), y = threadIdx.x / width, lanes = 256 / width;
  const uint64_t o = (uint64_t)blockIdx.x * width + x;
  double acc = 0;
  if (o < outcomes)
    for (uint32_t c = y; c < chunks; c += lanes) acc += in[c * outcomes + o];
  part[threadIdx.x] = acc;
  __syncthreads();
  for (uint32_t half = 128; half >= width; half >>= 1) {
    if (threadIdx.x < half) part[threadIdx.x] += part[threadIdx.x + half];
    __syncthreads();
  }
  if (y == 0 && o < outcomes) out[o] = part[x];
}

// collapse: keep (and scale) the amplitudes whose listed qubits read `want`
template <class P>
__global__ void __launch_bounds__(256) k_collapse(typename P::Glob* __restrict__ s, uint64_t N, uint64_t mask,
                                                  uint64_t want, double inv) {
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  typename P::Coef g;
  // coefficient (inv, 0) in the policy's representation
  double m[8] = {inv, 0, 0, 0, 0, 0, 0, 0};
  float hl[16];
  hl[0] = __double2float_rn(inv);  // one FP64 op per thread: negligible
  hl[1] = (float)(inv - (double)hl[0]);
  for (int i = 2; i < 16; ++i) hl[i] = 0.f;
  g = P::coef(m, hl);
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += step) {
    typename P::R x = P::from_glob(s[i]);
    if ((i & mask) == want) {
      P::cmul(x, g, 0);
    } else {
      x = P::zero();
    }
    s[i] = P::to_glob(x);
  }
}

static void check_qubits(const State& st, const int32_t* q, int32_t nq) {
  if (nq < 0 || (nq > 0 && !q)) fail(BF_EINVAL, "qubit list is null");
  uint64_t seen = 0;
  for (int i = 0; i < nq; ++i) {
    if (q[i] < 0 || q[i] >= st.n) fail(BF_EINVAL, "Target out of bounds: %d", q[i]);
    if ((seen >> q[i]) & 1) fail(BF_EINVAL, "Duplicate target: %d", q[i]);
    seen |= 1ull << q[i];
  }
}

// Outcome probabilities over the free qubits (values[k] < 0) of `q`; the
// others must read values[k].  out[o], bit k of o = k-th free qubit.
// The result stays in the state's pinned buffer until its next reduction.
const double* marginal_probs(State& st, const int32_t* q, const int8_t* values, int32_t nq, uint64_t* count) {
  check_qubits(st, q, nq);
  if (nq == 0) {  // the norm
    const double sum = reduce_norm2(st);
    st.h_partial[0] = sum;
    *count = 1;
    return st.h_partial;
  }
  MargArgs a;
  std::memset(&a, 0, sizeof a);
  uint64_t listed = 0, fixed = 0;
  int nfree = 0;
  int out_bit[64];
  for (int i = 0; i < nq; ++i) {
    const uint64_t bit = 1ull << q[i];
    listed |= bit;
    const int v = values ? values[i] : -1;
    if (v < 0) {
      if (nfree >= kMaxOutcomeBits) fail(BF_EUNSUPPORTED, "more than %d free measured qubits", kMaxOutcomeBits);
      out_bit[q[i]] = nfree++;
    } else {
      fixed |= bit;
      if (v) a.fixed_val |= bit;
    }
  }
  int nfh = 0;
  for (int p = 0; p < st.n; ++p) {
    const uint64_t bit = 1ull << p;
    if (fixed & bit) continue;
    const bool free_bit = (listed & bit) != 0;
    if (a.tile_bits < kMargTileBits) {
      a.tile_mask |= bit;
      if (a.tile_bits < 8) a.lane_pos[a.tile_bits] = (int8_t)p;
      if (free_bit) {
        a.keep |= 1u << a.tile_bits;
        a.low_pos[a.nfree_low] = (int8_t)a.tile_bits;
        a.low_out[a.nfree_low++] = (int8_t)out_bit[p];
      }
      ++a.tile_bits;
    } else if (free_bit) {
      a.free_high |= bit;
      a.high_out[nfh++] = (int8_t)out_bit[p];
    } else {
      a.sum_high |= bit;
    }
  }
  for (int j = 0; j < kMargPer; ++j) a.row[j] = deposit_mask((uint64_t)j * kMeasThreads, a.tile_mask);
  a.steps = 1ull << __builtin_popcountll(a.sum_high);
  a.outcomes = 1ull << nfree;
  // One wave of CTAs for one setting of the free high qubits (28 qubits, none
  // free, complex128: 742 against 800 us with 8 CTAs per SM), more where only
  // halves and quarters of a wave could be had (8 high ones free: 703 against
  // 883, complex64 365 against 351); a chunk is whole walk steps, at least one per 512
  // outcomes it writes (so that the sums stay a fraction of what is read), and
  // the chunks' sums stay within 32 MiB
  uint64_t chunks = std::max<uint64_t>(1, ((uint64_t)st.num_sms * (nfh ? 8 : kMargCtas)) >> nfh);
  chunks = std::min(chunks, std::max<uint64_t>(1, (1ull << 22) >> nfree));
  a.per_chunk = std::max((a.steps + chunks - 1) / chunks, std::min<uint64_t>(a.steps, ((1ull << a.nfree_low) + 511) / 512));
  a.chunks = (uint32_t)((a.steps + a.per_chunk - 1) / a.per_chunk);
  // Sums of the chunks, then (with more than one) the outcomes; a few sums are
  // added on the host, for less than a second launch costs.
  const uint64_t sums = (uint64_t)a.chunks * a.outcomes;
  const bool on_host = a.chunks > 1 && sums <= kMargHostSums;
  const uint64_t read = on_host ? sums : a.outcomes;
  ensure_partials(st, (size_t)(sums + a.outcomes + 1) / 2, (size_t)(read + 1) / 2);
  double* fin = a.chunks > 1 && !on_host ? st.d_partial + sums : st.d_partial;
  const dim3 grid((unsigned)((uint64_t)a.chunks << nfh));
  if (st.dtype == BF_C128)
    k_marginal<double2><<<grid, kMeasThreads, 0, st.stream>>>(static_cast<const double2*>(st.amp), a, st.d_partial);
  else
    k_marginal<float2><<<grid, kMeasThreads, 0, st.stream>>>(static_cast<const float2*>(st.amp), a, st.d_partial);
  BF_CUDA(cudaGetLastError());
  st.launches++;
  if (fin != st.d_partial) {
    uint32_t width = 1;
    while (width < 32 && width < a.outcomes && width * a.chunks < 2048) width *= 2;
    k_marginal_chunks<<<(unsigned)((a.outcomes + width - 1) / width), 256, 0, st.stream>>>(
        st.d_partial, a.outcomes, a.chunks, width, fin);
    BF_CUDA(cudaGetLastError());
    st.launches++;
  }
  BF_CUDA(cudaMemcpyAsync(st.h_partial, fin, read * sizeof(double), cudaMemcpyDeviceToHost, st.stream));
  sync_state(st);
  for (uint64_t k = a.outcomes; k < read; ++k) st.h_partial[k & (a.outcomes - 1)] += st.h_partial[k];
  *count = a.outcomes;
  return st.h_partial;
}

void measure(State& st, const int32_t* q, const int8_t* values, int32_t nq, int64_t seed, uint64_t* outcome,
             double* prob) {
  if (nq == 0) {
    if (outcome) *outcome = 0;
    if (prob) *prob = 1.0;
    return;
  }
  uint64_t outcomes = 0;
  const double* p = marginal_probs(st, q, values, nq, &outcomes);
  double total = 0;
  for (uint64_t i = 0; i < outcomes; ++i) total += p[i];
  if (!(total > 0)) fail(BF_EINVAL, "Measurement probability is zero");
  // the reference's draw (state.mojo:506-525); a negative seed is replaced
  // by a clock-derived one there as well
  if (seed < 0) seed = (int64_t)std::chrono::steady_clock::now().time_since_epoch().count() & 0x7fffffffffffll;
  int64_t rng = seed % 2147483647;
  rng = (rng * 48271) % 2147483647;
  double r = (double)rng / (double)2147483647 * total;
  uint64_t chosen = 0;
  double acc = 0;
  for (uint64_t i = 0; i < outcomes; ++i) {
    acc += p[i];
    if (r <= acc) {
      chosen = i;
      break;
    }
  }
  double cp = p[chosen];
  if (!(cp > 0)) fail(BF_EINVAL, "Measurement outcome probability is zero");
  double inv = 1.0 / std::sqrt(cp);
  uint64_t mask = 0, want = 0;
  int k = 0;
  for (int i = 0; i < nq; ++i) {
    mask |= 1ull << q[i];
    int v = values ? values[i] : -1;
    int bit = v >= 0 ? v : (int)((chosen >> k++) & 1);
    if (bit) want |= 1ull << q[i];
  }
  unsigned blocks = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((st.N + 255) / 256, (uint64_t)st.num_sms * 16));
  switch (st.prec) {
    case PREC_F64:
      k_collapse<PolF64><<<blocks, 256, 0, st.stream>>>(static_cast<double2*>(st.amp), st.N, mask, want, inv);
      break;
    case PREC_DF:
      k_collapse<PolDF><<<blocks, 256, 0, st.stream>>>(static_cast<double2*>(st.amp), st.N, mask, want, inv);
      break;
    default:
      k_collapse<PolF32><<<blocks, 256, 0, st.stream>>>(static_cast<float2*>(st.amp), st.N, mask, want, inv);
      break;
  }
  BF_CUDA(cudaGetLastError());
  st.launches++;
  if (outcome) *outcome = chosen;
  if (prob) *prob = cp;
}

// ---- top-k ------------------------------------------------------------------
// Each warp keeps a sorted list of its best candidates in registers: list
// position j sits in lane j % 32, slot j / 32.  One ballot tests 32
// probabilities against the warp's k-th best; the few lanes that beat it are
// inserted one at a time with shuffles.  After the first few thousand
// amplitudes almost no chunk holds one, so the pass streams the state at the
// cost of the ballot.  An FP32 estimate of |amp|^2 from the leading bits of
// each component skips the exact double-float square for amplitudes that
// cannot reach the k-th best.  The CTA's warps merge their lists through
// shared memory, and a one-CTA kernel merges the CTAs' lists, so the host
// reads back the k winners only.  Candidates are ordered by (probability
// desc, index asc).
constexpr int kTopK = 64;
constexpr int kTopUnroll = 4;            // loads in flight per thread
constexpr int kTopMergeThreads = 1024;
// The estimate is at least (1 - 2^-18) of the exact |amp|^2 and the k-th
// best's hi part is within 2^-24 of its value, so an amplitude that beats
// the k-th best has an estimate above its hi part times 1 - 2^-16.
constexpr float kTopSlack = 1.0f - 1.0f / 65536.0f;

struct Cand {
  float hi, lo;
  uint64_t idx;
};

__device__ __forceinline__ Cand cand_none() { return Cand{-1.f, 0.f, ~0ull}; }

__device__ __forceinline__ bool cand_better(const Cand& a, const Cand& b) {
  if (a.hi != b.hi) return a.hi > b.hi;
  if (a.lo != b.lo) return a.lo > b.lo;
  return a.idx < b.idx;
}

__device__ __forceinline__ Cand shfl_cand(const Cand& c, int src) {
  return Cand{__shfl_sync(0xffffffffu, c.hi, src), __shfl_sync(0xffffffffu, c.lo, src),
              __shfl_sync(0xffffffffu, c.idx, src)};
}

__device__ __forceinline__ Cand shfl_up_cand(const Cand& c) {
  return Cand{__shfl_up_sync(0xffffffffu, c.hi, 1), __shfl_up_sync(0xffffffffu, c.lo, 1),
              __shfl_up_sync(0xffffffffu, c.idx, 1)};
}

// |x| truncated to the 21 leading significant bits of the FP64 (its high
// word), as FP32; 0 below the FP32 range, +inf above it (and for Inf/NaN) so
// that the exact path decides those.
__device__ __forceinline__ float lead_abs(double x) {
  const unsigned hw = (unsigned)((unsigned long long)__double_as_longlong(x) >> 32);
  const int ef = (int)((hw >> 20) & 0x7ffu) - 896;
  if (ef <= 0) return 0.f;
  if (ef >= 255) return __int_as_float(0x7f800000);
  return __int_as_float((ef << 23) | (int)((hw & 0xfffffu) << 3));
}

// An FP32 estimate of |a|^2 that is at least (1 - 2^-18) of the exact value
// (two 2^-20 truncations squared, two FP32 roundings).
template <class T>
__device__ __forceinline__ float prob_estimate(T a);
template <>
__device__ __forceinline__ float prob_estimate<double2>(double2 a) {
  const float r = lead_abs(a.x), i = lead_abs(a.y);
  return fmaf(r, r, __fmul_rn(i, i));
}
template <>
__device__ __forceinline__ float prob_estimate<float2>(float2 a) {
  return fmaf(a.x, a.x, __fmul_rn(a.y, a.y));
}

// A warp's k best candidates, sorted, KB slots per lane (KB = 1 for k <= 32,
// 2 for k <= 64).  Unused positions hold cand_none().
template <int KB>
struct WarpTop {
  Cand s[KB];

  __device__ __forceinline__ void init() {
#pragma unroll
    for (int b = 0; b < KB; ++b) s[b] = cand_none();
  }
  // position k - 1, in every lane
  __device__ __forceinline__ Cand kth(int k) const {
    if (KB == 2 && k > 32) return shfl_cand(s[KB - 1], k - 33);
    return shfl_cand(s[0], k - 1);
  }
  // insert the warp-uniform x at its rank; the last position falls off
  __device__ __forceinline__ void insert(const Cand& x, int lane) {
    int pos = __popc(__ballot_sync(0xffffffffu, cand_better(s[0], x)));
    if (KB == 2) pos += __popc(__ballot_sync(0xffffffffu, cand_better(s[KB - 1], x)));
    const Cand up0 = shfl_up_cand(s[0]);
    if (KB == 2) {
      Cand up1 = shfl_up_cand(s[KB - 1]);
      const Cand last0 = shfl_cand(s[0], 31);
      if (lane == 0) up1 = last0;
      const int j = lane + 32;
      s[KB - 1] = j < pos ? s[KB - 1] : (j == pos ? x : up1);
    }
    s[0] = lane < pos ? s[0] : (lane == pos ? x : up0);
  }
  // one candidate per lane (where `valid`); thr is the k-th best and follows
  // the insertions
  __device__ __forceinline__ void offer(const Cand& c, bool valid, Cand& thr, int k, int lane) {
    unsigned m = __ballot_sync(0xffffffffu, valid && cand_better(c, thr));
    while (m) {
      const int src = __ffs(m) - 1;
      m &= m - 1;
      const Cand x = shfl_cand(c, src);
      if (cand_better(x, thr)) {
        insert(x, lane);
        thr = kth(k);
      }
    }
  }
  __device__ __forceinline__ void store(Cand* dst, int k, int lane) const {
#pragma unroll
    for (int b = 0; b < KB; ++b)
      if (lane + 32 * b < k) dst[lane + 32 * b] = s[b];
  }
};

// The CTA's WARPS lists -> warp 0's list (valid in warp 0 only).
template <int KB, int WARPS>
__device__ __forceinline__ void merge_warps(WarpTop<KB>& top, Cand& thr, Cand (*lists)[kTopK], int k) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  top.store(lists[warp], k, lane);
  __syncthreads();
  if (warp != 0) return;
  for (int w = 1; w < WARPS; ++w)
    for (int j0 = 0; j0 < k; j0 += 32) {
      const int j = j0 + lane;
      top.offer(j < k ? lists[w][j] : cand_none(), j < k, thr, k, lane);
    }
}

template <class T, int KB>
__global__ void __launch_bounds__(kMeasThreads) k_topk(const T* __restrict__ s, uint64_t N, int k,
                                                       Cand* __restrict__ out) {
  constexpr int kWarps = kMeasThreads / 32;
  __shared__ Cand lists[kWarps][kTopK];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  WarpTop<KB> top;
  top.init();
  Cand thr = cand_none();
  const uint64_t chunk = 32ull * kTopUnroll;
  const uint64_t step = (uint64_t)gridDim.x * kWarps * chunk;
  for (uint64_t base = ((uint64_t)blockIdx.x * kWarps + warp) * chunk; base < N; base += step) {
    T v[kTopUnroll];
#pragma unroll
    for (int u = 0; u < kTopUnroll; ++u) {
      const uint64_t i = base + 32 * u + lane;
      v[u] = i < N ? s[i] : T{};
    }
#pragma unroll
    for (int u = 0; u < kTopUnroll; ++u) {
      const uint64_t i = base + 32 * u + lane;
      const bool valid = i < N && prob_estimate<T>(v[u]) >= thr.hi * kTopSlack;
      Cand c{0.f, 0.f, i};
      if (valid) {
        const dfl p = prob_df<T>(v[u]);
        c.hi = p.hi;
        c.lo = p.lo;
      }
      top.offer(c, valid, thr, k, lane);
    }
  }
  merge_warps<KB, kWarps>(top, thr, lists, k);
  if (warp == 0) top.store(out + (size_t)blockIdx.x * k, k, lane);
}

// m candidates (the CTAs' lists) -> the k best, sorted.
template <int KB>
__global__ void __launch_bounds__(kTopMergeThreads) k_topk_merge(const Cand* __restrict__ in, int m, int k,
                                                                 Cand* __restrict__ out) {
  constexpr int kWarps = kTopMergeThreads / 32;
  __shared__ Cand lists[kWarps][kTopK];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  WarpTop<KB> top;
  top.init();
  Cand thr = cand_none();
  for (int j0 = warp * 32; j0 < m; j0 += kTopMergeThreads) {
    const int j = j0 + lane;
    top.offer(j < m ? in[j] : cand_none(), j < m, thr, k, lane);
  }
  merge_warps<KB, kWarps>(top, thr, lists, k);
  if (warp == 0) top.store(out, k, lane);
}

template <class T, int KB>
static void launch_topk(State& st, unsigned blocks, int k, Cand* part, Cand* fin) {
  k_topk<T, KB><<<blocks, kMeasThreads, 0, st.stream>>>(static_cast<const T*>(st.amp), st.N, k, part);
  BF_CUDA(cudaGetLastError());
  k_topk_merge<KB><<<1, kTopMergeThreads, 0, st.stream>>>(part, (int)blocks * k, k, fin);
  BF_CUDA(cudaGetLastError());
  st.launches += 2;
}

void probs_topk(State& st, int k, uint64_t* idx, double* probs) {
  if (k < 1 || k > kTopK) fail(BF_EINVAL, "k must be in [1, %d]", kTopK);
  if ((uint64_t)k > st.N) fail(BF_EINVAL, "k exceeds the number of amplitudes");
  static_assert(sizeof(Cand) == 2 * sizeof(double), "a candidate fills one partial-sum slot");
  const uint64_t per_cta = (uint64_t)kMeasThreads * kTopUnroll;
  const unsigned blocks = (unsigned)std::max<uint64_t>(
      1, std::min<uint64_t>((st.N + per_cta - 1) / per_cta, (uint64_t)st.num_sms * 4));
  ensure_partials(st, (size_t)blocks * k + k, (size_t)k);
  Cand* part = reinterpret_cast<Cand*>(st.d_partial);
  Cand* fin = part + (size_t)blocks * k;
  const bool wide = k > 32;
  if (st.dtype == BF_C128) {
    if (wide) launch_topk<double2, 2>(st, blocks, k, part, fin);
    else launch_topk<double2, 1>(st, blocks, k, part, fin);
  } else {
    if (wide) launch_topk<float2, 2>(st, blocks, k, part, fin);
    else launch_topk<float2, 1>(st, blocks, k, part, fin);
  }
  Cand* h = reinterpret_cast<Cand*>(st.h_partial);
  BF_CUDA(cudaMemcpyAsync(h, fin, (size_t)k * sizeof(Cand), cudaMemcpyDeviceToHost, st.stream));
  sync_state(st);
  for (int i = 0; i < k; ++i) {
    idx[i] = h[i].idx;
    probs[i] = (double)h[i].hi + (double)h[i].lo;
  }
}

}  // namespace bf
