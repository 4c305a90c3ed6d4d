// Energies of the streamed (pool-resident) circuits of a batch, after their
// sweeps: the tiled Pauli expectation (pauli_tiles.cuh) over work items of all
// of them.  Deferred circuit k has passes(Hamiltonian) x 2^(n - m) items,
// numbered from item_off[k]; partials[w] receives the sum of item w, and
// batch_energy_finalize adds a circuit's items in order (the sums do not
// depend on the grid).
//
// Bound: the states are read from L2 (the items running at any one time
// belong to a few neighbouring circuits), once per pass instead of once per
// flip mask; see pauli_tiles.cuh for the arithmetic.
#pragma once
#include "jit_batch.cuh"
#include "pauli_tiles.cuh"

namespace sq {

template <typename Real>
__global__ void __launch_bounds__(kPauliThreads, 4)
    batch_energy_tiles(const typename Vec2<Real>::T *__restrict__ pool, const BatchCircuit *__restrict__ circuits,
                       const PauliTilePlan *__restrict__ plans, const uint32_t *__restrict__ deferred,
                       const uint32_t *__restrict__ item_off, uint32_t ndef, uint32_t nitems, uint32_t max_terms,
                       double *__restrict__ partials) {
  extern __shared__ __align__(16) unsigned char pauli_raw[];
  PauliShared sh(pauli_raw, max_terms);
  for (uint32_t w = blockIdx.x; w < nitems; w += gridDim.x) {
    // Deferred circuit k with item_off[k] <= w < item_off[k + 1].
    uint32_t k = 0, end = ndef;
    while (end - k > 1) {
      const uint32_t mid = (k + end) / 2;
      if (item_off[mid] <= w) k = mid;
      else end = mid;
    }
    const BatchCircuit &C = circuits[deferred[k]];
    const PauliTilePlan &T = plans[C.ham];
    const uint32_t j = w - item_off[k], tile_bits = T.n - T.m;
    const PauliTilePass &S = T.pass[j >> tile_bits];
    pauli_stage(T, S, sh);
    double s = pauli_tile<Real, true>(pool + C.state_off, T, S, j & ((1u << tile_bits) - 1u), sh);
    s = block_sum(s);
    if (threadIdx.x == 0) partials[w] = s;
  }
}

}  // namespace sq
