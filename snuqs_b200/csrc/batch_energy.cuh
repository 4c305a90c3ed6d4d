// Energies of the streamed (pool-resident) circuits of a batch, after their
// sweeps: the tiled Pauli expectation (pauli_tiles.cuh) over work items of all
// of them.  Deferred circuit k has passes(Hamiltonian) x 2^(n - m) tiles to
// work, pass by pass, in chunks of kEnergyTiles; its chunks are numbered from
// chunk_off[k].  partials[w], partials[nchunks + w] receive the carried sum of
// chunk w, and batch_energy_finalize adds a circuit's chunks in order (the sums
// do not depend on the grid).
//
// Bound: shared-memory reads (pauli_tiles.cuh); the states come from L2 (the
// chunks running at any one time belong to a few neighbouring circuits), once
// per pass.  One circuit look-up, one staging of a pass and one block sum per
// chunk: with one tile per chunk these took longer than the tile (512 VQE
// circuits of 8..20 qubits, 64 strings each: 4.0 ms, now 3.15 ms).
#pragma once
#include "jit_batch.cuh"
#include "pauli_tiles.cuh"

namespace sq {

constexpr uint32_t kEnergyTiles = 8;

template <typename Real>
__global__ void __launch_bounds__(kPauliThreads, 4)
    batch_energy_tiles(const typename Vec2<Real>::T *__restrict__ pool, const BatchCircuit *__restrict__ circuits,
                       const PauliTilePlan *__restrict__ plans, const uint32_t *__restrict__ deferred,
                       const uint32_t *__restrict__ chunk_off, uint32_t ndef, uint32_t nchunks, uint32_t max_terms,
                       double *__restrict__ partials) {
  extern __shared__ __align__(16) unsigned char pauli_raw[];
  PauliShared sh(pauli_raw, max_terms);
  for (uint32_t w = blockIdx.x; w < nchunks; w += gridDim.x) {
    // Deferred circuit k with chunk_off[k] <= w < chunk_off[k + 1].
    uint32_t k = 0, end = ndef;
    while (end - k > 1) {
      const uint32_t mid = (k + end) / 2;
      if (chunk_off[mid] <= w) k = mid;
      else end = mid;
    }
    const BatchCircuit &C = circuits[deferred[k]];
    const PauliTilePlan &T = plans[C.ham];
    const typename Vec2<Real>::T *psi = pool + C.state_off;
    const uint32_t tile_bits = T.n - T.m, items = T.npasses << tile_bits;
    const uint32_t first = (w - chunk_off[k]) * kEnergyTiles;
    const uint32_t last = first + kEnergyTiles < items ? first + kEnergyTiles : items;
    uint32_t staged = ~0u;
    CarriedSum acc{0.0, 0.0};
    for (uint32_t j = first; j < last; ++j) {
      const uint32_t pass = j >> tile_bits;
      if (pass != staged) pauli_stage(T, T.pass[pass], sh);
      staged = pass;
      carry_add(acc, pauli_tile<Real, true>(psi, T, T.pass[pass], j & ((1u << tile_bits) - 1u), sh), 0.0);
    }
    const CarriedSum s = block_sum(acc);
    if (threadIdx.x == 0) {
      partials[w] = s.hi;
      partials[nchunks + w] = s.lo;
    }
  }
}

// energies[deferred[k]] = sum of the chunks [chunk_off[k], chunk_off[k + 1]), in
// order.  One block per deferred circuit.
static __global__ void __launch_bounds__(kReduceThreads)
    batch_energy_finalize(const double *__restrict__ partials, const uint32_t *__restrict__ chunk_off,
                          uint32_t nchunks, const uint32_t *__restrict__ deferred, double *__restrict__ energies) {
  const uint32_t k = blockIdx.x;
  CarriedSum v{0.0, 0.0};
  for (uint32_t i = chunk_off[k] + threadIdx.x; i < chunk_off[k + 1]; i += blockDim.x)
    carry_add(v, partials[i], partials[nchunks + i]);
  v = block_sum(v);
  if (threadIdx.x == 0) energies[deferred[k]] = carried(v);
}

}  // namespace sq
