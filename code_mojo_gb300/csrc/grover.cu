// grover.cu — the Grover diffuser and inversion about |0> as classical
// passes (apply_grover_diffuser / apply_grover_inversion_0,
// butterfly/algos/grover_classical.mojo:262-326), replacing their gate
// decompositions (H^k X^k MCP(pi) X^k H^k) with one reduction and one update.
//
// For every assignment b of the qubits outside `targets` (a block of 2^k
// amplitudes over the targets):
//   inversion:  x[b, 0] <- -x[b, 0]
//   diffuser:   x[b, t] <- 2 * mean_b - x[b, t],  mean_b = sum_t x[b, t] / 2^k
// The reference writes the imaginary part as -2 * mean_im - x_im
// (grover_classical.mojo:318); this pass uses 2 * mean - x for both parts,
// the inversion about the mean for complex amplitudes.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "amp_math.cuh"
#include "bf_internal.h"

namespace bf {

struct DiffArgs {
  int32_t low;               // 1: the targets are qubits 0..k-1 (index = b << k | t)
  int32_t k;                 // targets
  int8_t tpos[64];           // target positions, ascending
  int32_t nother;
  int8_t opos[64];           // other positions, ascending
  uint64_t blocks;           // 2^(n-k)
  uint64_t chunk;            // target-subspace amplitudes per CTA
  uint32_t chunks;           // CTAs per block
};

__device__ __forceinline__ uint64_t deposit_pos(uint64_t x, const int8_t* pos, int cnt) {
  uint64_t r = 0;
  for (int j = 0; j < cnt; ++j) r |= ((x >> j) & 1ull) << pos[j];
  return r;
}

__device__ __forceinline__ uint64_t diff_index(const DiffArgs& a, uint64_t b, uint64_t t) {
  if (a.low) return (b << a.k) | t;
  return deposit_pos(b, a.opos, a.nother) | deposit_pos(t, a.tpos, a.k);
}

// negate the amplitudes whose target bits are all zero (sign bits only: exact)
template <class T>
__global__ void __launch_bounds__(256) k_inversion0(T* __restrict__ s, uint64_t count, DiffArgs a) {
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; b < count; b += step) {
    uint64_t i = diff_index(a, b, 0);
    T v = s[i];
    v.x = -v.x;
    v.y = -v.y;
    s[i] = v;
  }
}

// CTA (block b, chunk c) sums its share of block b's amplitudes (double-float)
template <class T>
__device__ __forceinline__ void amp_df(T g, dfl& re, dfl& im);
template <>
__device__ __forceinline__ void amp_df<double2>(double2 g, dfl& re, dfl& im) {
  re = df_from_double(g.x);
  im = df_from_double(g.y);
}
template <>
__device__ __forceinline__ void amp_df<float2>(float2 g, dfl& re, dfl& im) {
  re = dfl{g.x, 0.f};
  im = dfl{g.y, 0.f};
}

template <class T>
__global__ void __launch_bounds__(256) k_diff_sum(const T* __restrict__ s, DiffArgs a, float4* __restrict__ partial) {
  const uint64_t b = blockIdx.x / a.chunks, c = blockIdx.x % a.chunks;
  const uint64_t sub = 1ull << a.k;
  const uint64_t begin = c * a.chunk, end = min(begin + a.chunk, sub);
  dfl sr{0.f, 0.f}, si{0.f, 0.f};
  for (uint64_t t = begin + threadIdx.x; t < end; t += blockDim.x) {
    dfl xr, xi;
    amp_df<T>(s[diff_index(a, b, t)], xr, xi);
    sr = df_add(sr, xr);
    si = df_add(si, xi);
  }
  __shared__ dfl wr[8], wi[8];
  for (int off = 16; off > 0; off >>= 1) {
    sr = df_add(sr, dfl{__shfl_down_sync(0xffffffffu, sr.hi, off), __shfl_down_sync(0xffffffffu, sr.lo, off)});
    si = df_add(si, dfl{__shfl_down_sync(0xffffffffu, si.hi, off), __shfl_down_sync(0xffffffffu, si.lo, off)});
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    wr[warp] = sr;
    wi[warp] = si;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    dfl r = wr[0], im = wi[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) {
      r = df_add(r, wr[w]);
      im = df_add(im, wi[w]);
    }
    partial[blockIdx.x] = make_float4(r.hi, r.lo, im.hi, im.lo);
  }
}

// one CTA per block b: 2 * mean_b in double-float from its chunk partials
__global__ void __launch_bounds__(256) k_diff_mean(const float4* __restrict__ partial, DiffArgs a,
                                                   float4* __restrict__ mean2) {
  const uint64_t b = blockIdx.x;
  dfl r{0.f, 0.f}, im{0.f, 0.f};
  for (uint32_t c = threadIdx.x; c < a.chunks; c += blockDim.x) {
    float4 p = partial[b * a.chunks + c];
    r = df_add(r, dfl{p.x, p.y});
    im = df_add(im, dfl{p.z, p.w});
  }
  __shared__ dfl wr[8], wi[8];
  for (int off = 16; off > 0; off >>= 1) {
    r = df_add(r, dfl{__shfl_down_sync(0xffffffffu, r.hi, off), __shfl_down_sync(0xffffffffu, r.lo, off)});
    im = df_add(im, dfl{__shfl_down_sync(0xffffffffu, im.hi, off), __shfl_down_sync(0xffffffffu, im.lo, off)});
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    wr[warp] = r;
    wi[warp] = im;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) {
      wr[0] = df_add(wr[0], wr[w]);
      wi[0] = df_add(wi[0], wi[w]);
    }
    // scale by 2 / 2^k: a power of two, exact on both parts
    const float sc = ldexpf(1.0f, 1 - a.k);
    mean2[b] = make_float4(wr[0].hi * sc, wr[0].lo * sc, wi[0].hi * sc, wi[0].lo * sc);
  }
}

template <class P>
__global__ void __launch_bounds__(256) k_diff_update(typename P::Glob* __restrict__ s, DiffArgs a,
                                                     const float4* __restrict__ mean2) {
  const uint64_t sub = 1ull << a.k;
  const uint64_t total = a.blocks * sub;
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; j < total; j += step) {
    const uint64_t b = j >> a.k, t = j & (sub - 1);
    const uint64_t i = diff_index(a, b, t);
    const float4 m = mean2[b];
    typename P::R x = P::from_glob(s[i]);
    if constexpr (std::is_same<P, PolDF>::value) {
      x.re = df_sub(dfl{m.x, m.y}, x.re);
      x.im = df_sub(dfl{m.z, m.w}, x.im);
    } else if constexpr (std::is_same<P, PolF32>::value) {
      x.re = (m.x + m.y) - x.re;
      x.im = (m.z + m.w) - x.im;
    } else {
      x.re = ((double)m.x + (double)m.y) - x.re;
      x.im = ((double)m.z + (double)m.w) - x.im;
    }
    s[i] = P::to_glob(x);
  }
}

// small target sets (k <= kSmallDiff): one thread per block, sum then update
constexpr int kSmallDiff = 8;

template <class P>
__global__ void __launch_bounds__(256) k_diff_small(typename P::Glob* __restrict__ s, DiffArgs a) {
  const uint64_t sub = 1ull << a.k;
  const uint64_t step = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; b < a.blocks; b += step) {
    const uint64_t base = deposit_pos(b, a.opos, a.nother);
    dfl sr{0.f, 0.f}, si{0.f, 0.f};
    for (uint64_t t = 0; t < sub; ++t) {
      dfl xr, xi;
      amp_df<typename P::Glob>(s[base | deposit_pos(t, a.tpos, a.k)], xr, xi);
      sr = df_add(sr, xr);
      si = df_add(si, xi);
    }
    const float sc = ldexpf(1.0f, 1 - a.k);
    const float4 m = make_float4(sr.hi * sc, sr.lo * sc, si.hi * sc, si.lo * sc);
    for (uint64_t t = 0; t < sub; ++t) {
      const uint64_t i = base | deposit_pos(t, a.tpos, a.k);
      typename P::R x = P::from_glob(s[i]);
      if constexpr (std::is_same<P, PolDF>::value) {
        x.re = df_sub(dfl{m.x, m.y}, x.re);
        x.im = df_sub(dfl{m.z, m.w}, x.im);
      } else if constexpr (std::is_same<P, PolF32>::value) {
        x.re = (m.x + m.y) - x.re;
        x.im = (m.z + m.w) - x.im;
      } else {
        x.re = ((double)m.x + (double)m.y) - x.re;
        x.im = ((double)m.z + (double)m.w) - x.im;
      }
      s[i] = P::to_glob(x);
    }
  }
}

static DiffArgs diff_args(const State& st, const int32_t* q, int32_t nq) {
  DiffArgs a;
  std::memset(&a, 0, sizeof a);
  uint64_t tm = 0;
  if (nq == 0) tm = (st.n >= 64) ? ~0ull : ((1ull << st.n) - 1);
  for (int i = 0; i < nq; ++i) {
    if (q[i] < 0 || q[i] >= st.n) fail(BF_EINVAL, "Target out of bounds: %d", q[i]);
    if ((tm >> q[i]) & 1) fail(BF_EINVAL, "Duplicate target: %d", q[i]);
    tm |= 1ull << q[i];
  }
  for (int b = 0; b < st.n; ++b) {
    if ((tm >> b) & 1) a.tpos[a.k++] = (int8_t)b;
    else a.opos[a.nother++] = (int8_t)b;
  }
  a.blocks = 1ull << a.nother;
  a.low = (a.k == 0) || (a.tpos[a.k - 1] == a.k - 1);  // ascending: targets are 0..k-1
  return a;
}

// classical_oracle (grover.mojo:64-66): negate listed amplitudes, eight per launch
struct OracleIdx {
  int32_t count;
  uint64_t idx[8];
};

template <class T>
__global__ void k_negate(T* s, OracleIdx a) {
  if ((int)threadIdx.x < a.count) {
    T v = s[a.idx[threadIdx.x]];
    v.x = -v.x;
    v.y = -v.y;
    s[a.idx[threadIdx.x]] = v;
  }
}

void launch_classical_oracle(State& st, const double* idx, int64_t count) {
  for (int64_t k = 0; k < count; k += 8) {
    OracleIdx a;
    a.count = (int32_t)std::min<int64_t>(8, count - k);
    for (int j = 0; j < a.count; ++j) a.idx[j] = (uint64_t)idx[k + j];
    // a repeated index is negated twice, as in the reference's loop
    bool dup = false;
    for (int i = 0; i < a.count; ++i)
      for (int j = i + 1; j < a.count; ++j) dup |= a.idx[i] == a.idx[j];
    if (dup) {
      for (int j = 0; j < a.count; ++j) {
        OracleIdx one;
        one.count = 1;
        one.idx[0] = a.idx[j];
        if (st.dtype == BF_C128) k_negate<double2><<<1, 32, 0, st.stream>>>(static_cast<double2*>(st.amp), one);
        else k_negate<float2><<<1, 32, 0, st.stream>>>(static_cast<float2*>(st.amp), one);
        st.launches++;
      }
    } else {
      if (st.dtype == BF_C128) k_negate<double2><<<1, 32, 0, st.stream>>>(static_cast<double2*>(st.amp), a);
      else k_negate<float2><<<1, 32, 0, st.stream>>>(static_cast<float2*>(st.amp), a);
      st.launches++;
    }
    BF_CUDA(cudaGetLastError());
  }
}

void launch_grover_inversion0(State& st, const int32_t* q, int32_t nq) {
  DiffArgs a = diff_args(st, q, nq);
  unsigned g = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((a.blocks + 255) / 256, (uint64_t)st.num_sms * 16));
  if (st.dtype == BF_C128) k_inversion0<double2><<<g, 256, 0, st.stream>>>(static_cast<double2*>(st.amp), a.blocks, a);
  else k_inversion0<float2><<<g, 256, 0, st.stream>>>(static_cast<float2*>(st.amp), a.blocks, a);
  BF_CUDA(cudaGetLastError());
  st.launches++;
}

template <class P>
static void diffuser_p(State& st, DiffArgs& a) {
  if (a.k <= kSmallDiff) {
    unsigned g = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((a.blocks + 255) / 256, (uint64_t)st.num_sms * 16));
    k_diff_small<P><<<g, 256, 0, st.stream>>>(static_cast<typename P::Glob*>(st.amp), a);
    BF_CUDA(cudaGetLastError());
    st.launches++;
    return;
  }
  const uint64_t sub = 1ull << a.k;
  // short CTAs (16 Ki amplitudes each) so that other streams' kernels get SMs
  // between them
  a.chunk = std::min<uint64_t>(sub, 1ull << 14);
  a.chunks = (uint32_t)((sub + a.chunk - 1) / a.chunk);
  uint64_t slots = a.blocks * a.chunks;
  if (slots > 0x7fffffffull) fail(BF_EUNSUPPORTED, "too many diffuser blocks");
  // partials (float4 per slot) then 2*mean (float4 per block), in the partials buffer
  size_t need = (size_t)(slots + a.blocks) * sizeof(float4);
  ensure_partials(st, (need + 2 * sizeof(double) - 1) / (2 * sizeof(double)), 0);
  float4* partial = reinterpret_cast<float4*>(st.d_partial);
  float4* mean2 = partial + slots;
  auto* s = static_cast<typename P::Glob*>(st.amp);
  k_diff_sum<typename P::Glob><<<(unsigned)slots, 256, 0, st.stream>>>(s, a, partial);
  if (a.blocks > 0x7fffffffull) fail(BF_EUNSUPPORTED, "too many diffuser blocks");
  k_diff_mean<<<(unsigned)a.blocks, 256, 0, st.stream>>>(partial, a, mean2);
  // one element per thread: short CTAs
  unsigned g = (unsigned)std::max<uint64_t>(1, std::min<uint64_t>((st.N + 255) / 256, 0x7fffffffull));
  k_diff_update<P><<<g, 256, 0, st.stream>>>(s, a, mean2);
  BF_CUDA(cudaGetLastError());
  st.launches += 3;
}

void launch_grover_diffuser(State& st, const int32_t* q, int32_t nq) {
  DiffArgs a = diff_args(st, q, nq);
  switch (st.prec) {
    case PREC_F64: diffuser_p<PolF64>(st, a); break;
    case PREC_DF: diffuser_p<PolDF>(st, a); break;
    default: diffuser_p<PolF32>(st, a); break;
  }
}

// ---- Grover search loop ------------------------------------------------------
// `iters` repetitions of (classical oracle, diffuser over every qubit) -- the
// body of grover_search with the classical replacements (grover.mojo:64-94,
// grover_classical.mojo:284-326) -- in one launch and one read-modify-write of
// the state, whatever the iteration count.
//
// With k marked amplitudes (sum W) and the N - k others (sum U), an iteration
// adds m = 2 (U - W) / N to every marked amplitude and maps every other one
// to m - x.  In the coordinates u = U / sqrt(N - k), w = W / sqrt(k) that is a
// rotation by 2 theta, sin(theta) = sqrt(k / N) (the two-dimensional picture
// of the search), so r iterations are the rotation by phi = 2 r theta, and
//   x -> (-1)^r x + c   (unmarked),  c = (U_r - (-1)^r U_0) / (N - k)
//   x -> x + d          (marked),    d = (W_r - W_0) / k
// with c and d linear in U_0 and W_0.  The host forms the four coefficients
// (grover_coefficients); the kernel sums the state, meets at one grid barrier
// (or ends there, and its second half is a launch of its own) and adds c or d.
//
// Bound by memory: one read for the sum, one read and one write for the
// update (3S; the sum's second read comes from L2 up to about 2^22
// amplitudes).  At 20 qubits, complex128, 804 iterations: 10.7 ms with a
// sweep and a grid barrier per iteration, 0.024 ms like this.  x is rounded
// once instead of once per iteration: served searches of 10 to 20 qubits went
// from 5.5e-13 to 2.6e-14 off the 64-bit probabilities.
struct LoopArgs {
  uint64_t N;
  uint64_t chunk;         // amplitudes per CTA
  int32_t nmarked;        // indices negated by the oracle (odd multiplicity)
  uint64_t marked[8];
  int32_t odd;            // 1: an odd number of iterations (the sign of x)
  double cu, cw;          // c = cu U_0 + cw W_0
  double du, dw;          // d = du U_0 + dw W_0
  uint32_t spin_limit;    // polls of 64 ns before a barrier wait gives up
  float4* partial;        // gridDim.x
  double2* saved;         // the split form: the marked amplitudes before the loop
  unsigned int* bar;      // arrival counter, zero at launch
  int* flag;              // set to 1 when a barrier wait expires
};

__device__ __forceinline__ unsigned int ld_acquire_u32(const unsigned int* p) {
  unsigned int v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

// all CTAs of the grid: returns false (CTA-uniform) when the wait expired
__device__ __forceinline__ bool loop_barrier(const LoopArgs& a, unsigned int target) {
  __shared__ int ok_sh;
  __syncthreads();
  if (threadIdx.x == 0) {
    int ok = 1;
    __threadfence();
    atomicAdd(a.bar, 1u);
    unsigned int polls = 0;
    while (ld_acquire_u32(a.bar) < target) {
      if (++polls > a.spin_limit) {
        ok = 0;
        atomicExch(a.flag, 1);
        break;
      }
      __nanosleep(64);
    }
    ok_sh = ok;
  }
  __syncthreads();
  return ok_sh != 0;
}

__device__ __forceinline__ void block_sum2(dfl& r, dfl& im, dfl* wr, dfl* wi) {
  for (int off = 16; off > 0; off >>= 1) {
    r = df_add(r, dfl{__shfl_down_sync(0xffffffffu, r.hi, off), __shfl_down_sync(0xffffffffu, r.lo, off)});
    im = df_add(im, dfl{__shfl_down_sync(0xffffffffu, im.hi, off), __shfl_down_sync(0xffffffffu, im.lo, off)});
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) {
    wr[warp] = r;
    wi[warp] = im;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) {
      wr[0] = df_add(wr[0], wr[w]);
      wi[0] = df_add(wi[0], wi[w]);
    }
    r = wr[0];
    im = wi[0];
  }
}

// sign * x + c: complex128 in FP64 (two DADD per amplitude stay under the
// pass's HBM time), complex64 with c as an FP32 pair
__device__ __forceinline__ double2 loop_shift(double2 x, bool neg, double cr, double ci) {
  return make_double2((neg ? -x.x : x.x) + cr, (neg ? -x.y : x.y) + ci);
}
__device__ __forceinline__ float2 loop_shift(float2 x, bool neg, float2 cr, float2 ci) {
  return make_float2((cr.x + (neg ? -x.x : x.x)) + cr.y, (ci.x + (neg ? -x.y : x.y)) + ci.y);
}
__device__ __forceinline__ float2 loop_pair(double v) {
  const float hi = (float)v;
  return make_float2(hi, (float)(v - (double)hi));
}

enum { kLoopWhole, kLoopSum, kLoopUpdate };  // both halves in one launch, or one each
template <class T, int kPart>
__global__ void __launch_bounds__(256) k_grover_loop(T* __restrict__ s, LoopArgs a) {
  __shared__ dfl wr[8], wi[8];
  __shared__ double shift[4];  // c (re, im), d (re, im)
  __shared__ double2 mk[8];    // the marked amplitudes before the loop
  const uint64_t begin = (uint64_t)blockIdx.x * a.chunk;
  const uint64_t end = min(begin + a.chunk, a.N);
  const unsigned int G = gridDim.x;
  // every CTA reads the marked amplitudes before any CTA writes the state
  if ((int)threadIdx.x < a.nmarked) {
    if constexpr (kPart == kLoopUpdate) {
      mk[threadIdx.x] = __ldcg(a.saved + threadIdx.x);
    } else {
      const T v = s[a.marked[threadIdx.x]];
      mk[threadIdx.x] = make_double2((double)v.x, (double)v.y);
      if (kPart == kLoopSum && blockIdx.x == 0) a.saved[threadIdx.x] = mk[threadIdx.x];
    }
  }
  // eight loads in flight per thread before any use
  constexpr int kU = 8;
  dfl sr{0.f, 0.f}, si{0.f, 0.f};
  for (uint64_t base = begin + threadIdx.x; base < end && kPart != kLoopUpdate; base += kU * blockDim.x) {
    T v[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const uint64_t i = base + (uint64_t)u * blockDim.x;
      v[u] = i < end ? s[i] : T{};
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      dfl xr, xi;
      amp_df<T>(v[u], xr, xi);
      sr = df_add(sr, xr);
      si = df_add(si, xi);
    }
  }
  if constexpr (kPart != kLoopUpdate) {
    block_sum2(sr, si, wr, wi);
    if (threadIdx.x == 0) a.partial[blockIdx.x] = make_float4(sr.hi, sr.lo, si.hi, si.lo);
    if constexpr (kPart == kLoopSum) return;
    if (G > 1) {
      if (!loop_barrier(a, G)) return;
    } else {
      __syncthreads();
    }
  }
  sr = si = dfl{0.f, 0.f};
  for (unsigned int c = threadIdx.x; c < G; c += blockDim.x) {
    const float4 q = __ldcg(a.partial + c);
    sr = df_add(sr, dfl{q.x, q.y});
    si = df_add(si, dfl{q.z, q.w});
  }
  block_sum2(sr, si, wr, wi);
  if (threadIdx.x == 0) {
    double w0 = 0, w1 = 0;
    for (int k = 0; k < a.nmarked; ++k) {
      w0 += mk[k].x;
      w1 += mk[k].y;
    }
    const double u0 = ((double)sr.hi + (double)sr.lo) - w0, u1 = ((double)si.hi + (double)si.lo) - w1;
    shift[0] = a.cu * u0 + a.cw * w0;
    shift[1] = a.cu * u1 + a.cw * w1;
    shift[2] = a.du * u0 + a.dw * w0;
    shift[3] = a.du * u1 + a.dw * w1;
  }
  __syncthreads();
  const bool neg = a.odd != 0;
  auto as_shift = [](double v) {
    if constexpr (sizeof(T) == 16) return v;
    else return loop_pair(v);
  };
  const auto cr = as_shift(shift[0]), ci = as_shift(shift[1]);
  for (uint64_t base = begin + threadIdx.x; base < end; base += kU * blockDim.x) {
    T v[kU];
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const uint64_t i = base + (uint64_t)u * blockDim.x;
      if (i < end) v[u] = s[i];
    }
#pragma unroll
    for (int u = 0; u < kU; ++u) {
      const uint64_t i = base + (uint64_t)u * blockDim.x;
      if (i < end) s[i] = loop_shift(v[u], neg, cr, ci);
    }
  }
  // the CTA's own marked amplitudes, once its unmarked update is done
  __syncthreads();
  if ((int)threadIdx.x < a.nmarked) {
    const uint64_t i = a.marked[threadIdx.x];
    if (i >= begin && i < end) {
      const double2 x = mk[threadIdx.x];
      T v;
      v.x = (decltype(v.x))(x.x + shift[2]);
      v.y = (decltype(v.y))(x.y + shift[3]);
      s[i] = v;
    }
  }
}

int grover_loop_max_marked() { return 8; }

// The coefficients of c and d (above).  Differences of nearly equal terms are
// taken as products of half-angle sines and cosines, so each coefficient is
// good to about phi 2^-53 relative to the larger of its two terms.
static void grover_coefficients(LoopArgs& a, int iters) {
  const double N = (double)a.N, k = (double)a.nmarked, rest = N - k;
  const double phi = 2.0 * iters * std::asin(std::sqrt(k / N));
  const double half_s = std::sin(0.5 * phi), half_c = std::cos(0.5 * phi), sn = std::sin(phi);
  a.odd = iters & 1;
  // cos(phi) - (-1)^r and cos(phi) - 1
  const double cos_sign = a.odd ? 2.0 * half_c * half_c : -2.0 * half_s * half_s;
  const double cos_one = -2.0 * half_s * half_s;
  const bool both = k > 0 && rest > 0;
  a.cu = rest > 0 ? cos_sign / rest : 0.0;
  a.cw = both ? -sn / std::sqrt(rest * k) : 0.0;
  a.du = both ? sn / std::sqrt(rest * k) : 0.0;
  a.dw = k > 0 ? cos_one / k : 0.0;
}

template <class T>
static void launch_grover_t(State& st, LoopArgs& a) {
  int per_sm = 0;
  BF_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_grover_loop<T, kLoopWhole>, 256, 0));
  const uint64_t resident = (uint64_t)std::max(1, per_sm) * (uint64_t)st.num_sms;
  // chunks of at least 4096 amplitudes
  uint64_t G = std::max<uint64_t>(1, std::min<uint64_t>(std::min((uint64_t)2 * st.num_sms, resident), st.N >> 12));
  a.chunk = (st.N + G - 1) / G;
  a.chunk = (a.chunk + 255) & ~255ull;
  G = (st.N + a.chunk - 1) / a.chunk;
  // partial sums (G float4), the marked amplitudes, the arrival counter
  const size_t bytes = G * sizeof(float4) + sizeof a.marked / sizeof a.marked[0] * sizeof(double2) + 16;
  ensure_partials(st, (bytes + 2 * sizeof(double) - 1) / (2 * sizeof(double)), 0);
  a.partial = reinterpret_cast<float4*>(st.d_partial);
  a.saved = reinterpret_cast<double2*>(a.partial + G);
  a.bar = reinterpret_cast<unsigned int*>(a.saved + sizeof a.marked / sizeof a.marked[0]);
  a.flag = state_flag(st);
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)G);
  cfg.blockDim = dim3(256);
  cfg.dynamicSmemBytes = 0;
  cfg.stream = st.stream;
  T* s = static_cast<T*>(st.amp);
  if (st.shared_gpu && G > 1) {
    // a server slot shares the GPU: CTAs that wait at a barrier would hold SMs
    // that the other slots' kernels need, so the two halves are launches of
    // their own, which wait for nothing.  A request of 26 qubits, complex128,
    // whatever the count: 4.9 ms; with the barrier and 16 CTAs 11.9 ms; with
    // the ops one by one 5.8 ms at 2 iterations and 15.3 ms at 16.  At 20
    // qubits 0.27 ms, 0.37 with 16 CTAs.
    BF_CUDA(cudaLaunchKernelEx(&cfg, k_grover_loop<T, kLoopSum>, s, a));
    BF_CUDA(cudaLaunchKernelEx(&cfg, k_grover_loop<T, kLoopUpdate>, s, a));
    st.launches += 2;
    return;
  }
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  if (G > 1) {
    BF_CUDA(cudaMemsetAsync(a.bar, 0, sizeof(unsigned int), st.stream));
    cfg.attrs = attr;
    cfg.numAttrs = 1;
  }
  BF_CUDA(cudaLaunchKernelEx(&cfg, k_grover_loop<T, kLoopWhole>, s, a));
  st.launches++;
}

void launch_grover_loop(State& st, const uint64_t* marked, int nmarked, int iters) {
  if (iters <= 0) return;
  if (nmarked < 0 || nmarked > 8) fail(BF_EINVAL, "internal: %d oracle indices in a Grover loop", nmarked);
  LoopArgs a;
  std::memset(&a, 0, sizeof a);
  a.N = st.N;
  a.nmarked = nmarked;
  for (int k = 0; k < nmarked; ++k) a.marked[k] = marked[k];
  grover_coefficients(a, iters);
  a.spin_limit = 1u << 25;  // x 64 ns sleeps: about 2 s
  if (st.dtype == BF_C128) launch_grover_t<double2>(st, a);
  else launch_grover_t<float2>(st, a);
}

}  // namespace bf
