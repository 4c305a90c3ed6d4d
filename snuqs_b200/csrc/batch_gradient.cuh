// Gradients of K parameter sets of one circuit as multi-state sweeps: the parts
// between the forward and the reverse sweeps, and after them.
//
// Measured on B200, 64 sets of a QAOA circuit (16 qubits, p = 8, complex128):
// forward sweeps 414 us, batch_apply_kernel 65 us, 12 reverse sweeps
// (sq_jit_madjoint) 1150 us, sums 8 us; one CTA per circuit (64 of 148 SMs
// busy) took 5080 us.
#pragma once
#include "jit_batch.cuh"

namespace sq {

constexpr uint32_t kApplyBits = 12;  // amplitudes of one block

// lambda = H psi over K states of 2^n amplitudes that lie back to back (state c
// with Hamiltonian circuits[c].ham); partials[block] receives the block's
// share of Re <psi|lambda>, 2^(n - kApplyBits) blocks per state.  Bound: one read
// of psi per flip group and one for the energy, and one write of lambda.
template <typename Real>
__global__ void __launch_bounds__(kReduceThreads)
    batch_apply_kernel(const typename Vec2<Real>::T *__restrict__ psi, typename Vec2<Real>::T *__restrict__ lam,
                       const BatchCircuit *__restrict__ circuits, const PauliParams *__restrict__ hams, uint32_t n,
                       double *__restrict__ partials) {
  using C2 = typename Vec2<Real>::T;
  constexpr int U = 4;  // amplitudes in flight
  const uint32_t shift = n - kApplyBits;
  const uint64_t c = blockIdx.x >> shift;
  const PauliParams &H = hams[circuits[c].ham];
  const C2 *p = psi + (c << n);
  C2 *o = lam + (c << n);
  const uint64_t first = (uint64_t(blockIdx.x & ((1u << shift) - 1u)) << kApplyBits) + threadIdx.x;
  double e = 0.0;
  for (uint32_t j = 0; j < (1u << kApplyBits) / kReduceThreads; j += U) {
    double ar[U] = {}, ai[U] = {};
    for (uint32_t gi = 0; gi < H.ngroups; ++gi) {
      const PauliGroup &G = H.g[gi];
      C2 b[U];
      double w[U] = {};
#pragma unroll
      for (int u = 0; u < U; ++u) b[u] = p[(first + (j + u) * kReduceThreads) ^ G.x];
      for (uint32_t t = G.t0; t < G.t1; ++t) {
        const double f = H.f[t];
#pragma unroll
        for (int u = 0; u < U; ++u)
          w[u] += (__popcll((first + (j + u) * kReduceThreads) & H.zy[t]) & 1) ? -f : f;
      }
#pragma unroll
      for (int u = 0; u < U; ++u) {
        if (G.odd) {  // w * (-i) * b
          ar[u] += w[u] * double(b[u].y);
          ai[u] -= w[u] * double(b[u].x);
        } else {
          ar[u] += w[u] * double(b[u].x);
          ai[u] += w[u] * double(b[u].y);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const uint64_t i = first + (j + u) * kReduceThreads;
      C2 v;
      v.x = Real(ar[u]);
      v.y = Real(ai[u]);
      const C2 a = p[i];
      o[i] = v;
      e += double(a.x) * ar[u] + double(a.y) * ai[u];
    }
  }
  e = block_sum(e);
  if (threadIdx.x == 0) partials[blockIdx.x] = e;
}

// energies[c] = the sum of state c's `count` partials, in a fixed order.
static __global__ void __launch_bounds__(kReduceThreads)
    batch_apply_finalize(const double *__restrict__ partials, uint32_t count, double *__restrict__ energies) {
  const double *p = partials + uint64_t(blockIdx.x) * count;
  double v = 0.0;
  for (uint32_t i = threadIdx.x; i < count; i += blockDim.x) v += p[i];
  v = block_sum(v);
  if (threadIdx.x == 0) energies[blockIdx.x] = v;
}

// One slot of one reverse sweep: its rows (jit_madjoint_sweep) and the
// occurrence it feeds; entries are sorted by occurrence.
struct GradientEntry {
  uint64_t rows;      // first row of the sweep (doubles from the row buffer)
  uint64_t per;       // tiles per CTA of the sweep
  uint32_t rows_per;  // rows per state
  uint32_t tile_shift;
  uint32_t slot, pad;
};

// occ[c * nocc + g].x = sum over the entries of occurrence g (first[g] ..
// first[g + 1]) and their rows of state c, in a fixed order.  Block g + nocc c.
static __global__ void __launch_bounds__(128)
    gradient_reduce_kernel(const double *__restrict__ rows, const GradientEntry *__restrict__ entries,
                           const uint32_t *__restrict__ first, uint32_t nocc, double2 *__restrict__ occ) {
  const uint32_t g = blockIdx.x % nocc;
  const uint64_t c = blockIdx.x / nocc;
  double s = 0.0;
  for (uint32_t e = first[g]; e < first[g + 1]; ++e) {
    const GradientEntry E = entries[e];
    const uint64_t r0 = (c << E.tile_shift) / E.per, r1 = (((c + 1) << E.tile_shift) - 1) / E.per;
    for (uint32_t r = threadIdx.x; r <= uint32_t(r1 - r0); r += blockDim.x)
      s += rows[E.rows + (c * E.rows_per + r) * kMaxInner + E.slot];
  }
  s = block_sum(s);
  if (threadIdx.x == 0) occ[blockIdx.x] = make_double2(s, 0.0);
}

}  // namespace sq
