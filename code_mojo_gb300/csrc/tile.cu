// tile.cu — fused tile pass: each CTA loads the 2^K amplitudes that share
// one assignment of the non-tile qubits into shared memory, applies an
// ordered list of gates there, and writes them back: one HBM read + write
// for the whole group of gates.
//
// GPU form of the reference's fused-grid strategy (GRID_FUSED: row-local
// groups applied one row at a time, executors.mojo:1062-1093) and of its
// L2 column tiling (transformations_grid.mojo:21, 367-555): the "row" is the
// set of K tile qubits, which need not be contiguous.  The low
// kTileLowQubits qubits are always part of the tile so that every global
// access moves runs of 2^5 contiguous amplitudes (512 B at complex128).
//
// A gate fits a tile pass when its target is a tile qubit; its controls may
// be anywhere (a control outside the tile is constant over the CTA, so the
// CTA applies the gate or skips it).  A diagonal gate fits whatever its
// qubits: a target outside the tile only selects which diagonal entry the
// whole CTA multiplies by.
#include <algorithm>

#include "tile_body.cuh"

namespace bf {

// kUnitaries: the pass holds dense unitaries; kFans: phase fans (separate
// forms, so that passes without them keep the gate loop's small register
// count and shared memory)
//
// A complex64 12-qubit tile leaves room for six CTAs per SM, and six of them
// hide the per-op latencies better than the five that 46 registers allow: the
// passes of a 27-qubit value encoding take 4.37 against 4.74 ms (7 or 8: 4.57).
// (0: unspecified; complex128 loses with more registers than the compiler
// takes by itself.)
template <class P, bool kUnitaries>
constexpr int kTileCtas = sizeof(typename P::Glob) == 8 && !kUnitaries ? 6 : 0;

template <class P, bool kUnitaries, bool kFans>
__global__ void __launch_bounds__(kTileThreads, (kTileCtas<P, kUnitaries>)) k_tile(typename P::Glob* __restrict__ s,
                                                       const TileOp* __restrict__ ops, int nops,
                                                       const TileGeom geo, const double* __restrict__ pool,
                                                       int halvings) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  run_tile<P, false, kUnitaries, kFans>(s, ops, nops, geo, blockIdx.x, smem_raw, pool, halvings);
}

template <class P, bool kUnitaries, bool kFans>
static void launch_tile_form(State& st, const TileOp* d_ops, int nops, const TileGeom& geo, const double* d_pool,
                             int halvings) {
  static PerDeviceOnce configured;  // one per instantiation
  configured.run(st.device, [] {
    BF_CUDA(cudaFuncSetAttribute(k_tile<P, kUnitaries, kFans>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)tile_smem_bytes<P>(kMaxTileQubits, 0, kUnitaries, kFans)));
  });
  const uint64_t blocks = st.N >> geo.K;
  if (blocks > 0x7fffffffull) fail(BF_EUNSUPPORTED, "tile grid too large");
  k_tile<P, kUnitaries, kFans><<<(unsigned)blocks, kTileThreads,
                                 tile_smem_bytes<P>(geo.K, geo.L, kUnitaries, kFans), st.stream>>>(
      static_cast<typename P::Glob*>(st.amp), d_ops, nops, geo, d_pool, halvings);
  BF_CUDA(cudaGetLastError());
  st.launches++;
}

template <class P>
static void launch_tile_p(State& st, const TileOp* d_ops, int nops, const TilePass& p, const double* d_pool,
                          bool unitaries, bool fans, int halvings) {
  TileGeom geo;
  geo.K = p.K;
  geo.L = p.L;
  if (geo.L < 0 || geo.L > std::min(p.K, kTileLowQubits)) fail(BF_EINVAL, "internal: bad tile low width %d", geo.L);
  for (int j = 0; j < p.K; ++j) geo.q[j] = p.q[j];
  for (int j = 0; j < geo.L; ++j)
    if (geo.q[j] != j) fail(BF_EINVAL, "internal: tile qubits must start with 0..%d", geo.L - 1);
  if (unitaries && fans) launch_tile_form<P, true, true>(st, d_ops, nops, geo, d_pool, halvings);
  else if (unitaries) launch_tile_form<P, true, false>(st, d_ops, nops, geo, d_pool, halvings);
  else if (fans) launch_tile_form<P, false, true>(st, d_ops, nops, geo, d_pool, halvings);
  else launch_tile_form<P, false, false>(st, d_ops, nops, geo, d_pool, halvings);
}

void launch_tile_pass(State& st, const TileOp* d_ops, int nops, const TilePass& p, const double* d_pool,
                      bool unitaries, bool fans, int halvings) {
  switch (st.prec) {
    case PREC_F64: launch_tile_p<PolF64>(st, d_ops, nops, p, d_pool, unitaries, fans, halvings); break;
    case PREC_DF: launch_tile_p<PolDF>(st, d_ops, nops, p, d_pool, unitaries, fans, halvings); break;
    default: launch_tile_p<PolF32>(st, d_ops, nops, p, d_pool, unitaries, fans, halvings); break;
  }
}

int tile_max_qubits(const State&) { return kMaxTileQubits; }

}  // namespace bf
