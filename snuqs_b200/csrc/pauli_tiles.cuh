// Kernels of the tiled Pauli-sum expectation (pauli_tiles.h has the plan),
// FP64 throughout for both state precisions.
//
// What bounds it: one read of the state per pass, against one shared-memory
// read and three FP64 operations per pair and group.  A block holds one tile
// of 2^11 amplitudes (32 KiB as complex doubles) and each of its 256 threads
// four of its amplitudes (r * 256 + tid, rows r = 0..3) in registers.  A group whose flip
// reaches the top tile bit (the plan makes nearly all do) has one amplitude
// of every pair in rows 0..3: four partners per thread, each one 16-byte
// shared read (lanes read an XOR of consecutive slots: conflict-free without
// a swizzle).  Signs (-1)^popc(i & zy) split over tile base, thread and row:
// the base's parities are computed once per tile and term, the rows' are two
// factors of +-1 that the sum over the rows takes in its FMAs.
// Bound by shared-memory reads (ncu: 80 % of their rate, DRAM 42 %).  Measured
// on B200: 64 random strings (8 passes) and 25 diagonal ones on 25 qubits
// complex128 1187 us together, with one read of the state per mask 6212 us;
// 2110 us with per-row sign flips and own amplitudes chosen at run time, 1670
// us with a group header and a term loop for every single string.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "pauli_tiles.h"
#include "reduce_kernels.cuh"

namespace sq {

constexpr int kPauliThreads = 256;
constexpr int kPauliRows = (1 << kPauliTileBits) / kPauliThreads;

// A sum and the rounding errors of its additions (hi is what adding alone
// gives).  Sums over whole states cancel: the ring sum of Z Z strings on a
// random state is 2^-(n/2) of its weights, while the partial sums of blocks
// that each hold one pattern of the high index bits are not.  Added plainly
// these left errors two to three times those of threads that stride over the
// whole state (19 to 21 qubits); with the errors carried along, a tenth.
struct CarriedSum {
  double hi, lo;
};
__device__ __forceinline__ void carry_add(CarriedSum &a, double hi, double lo) {
  const double s = __dadd_rn(a.hi, hi), b = __dsub_rn(s, a.hi);
  const double e = __dadd_rn(__dsub_rn(a.hi, __dsub_rn(s, b)), __dsub_rn(hi, b));
  a.lo = __dadd_rn(__dadd_rn(a.lo, lo), e);
  a.hi = s;
}
// The sum (hi alone where the errors are not numbers: infinite sums).
__device__ __forceinline__ double carried(const CarriedSum &a) {
  const double s = __dadd_rn(a.hi, a.lo);
  return s == s ? s : a.hi;
}

// block_sum of carried sums; valid in thread 0.
__device__ __forceinline__ CarriedSum block_sum(CarriedSum v) {
  __shared__ double red_hi[32], red_lo[32];
  auto warp = [](CarriedSum &x) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double h = __shfl_xor_sync(0xffffffffu, x.hi, o), l = __shfl_xor_sync(0xffffffffu, x.lo, o);
      carry_add(x, h, l);
    }
  };
  warp(v);
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (lane == 0) {
    red_hi[w] = v.hi;
    red_lo[w] = v.lo;
  }
  __syncthreads();
  v = CarriedSum{0.0, 0.0};
  if (w == 0) {
    if (lane < int(blockDim.x >> 5)) v = CarriedSum{red_hi[lane], red_lo[lane]};
    warp(v);
  }
  __syncthreads();
  return v;
}

// out[0] = sum of the n carried sums partial[i], partial[n + i], in a fixed
// order; out[1] takes *word (if any), for one copy to the host instead of two.
static __global__ void __launch_bounds__(kReduceThreads)
    finalize_carried_kernel(const double *__restrict__ partial, uint32_t n, double *__restrict__ out,
                            const uint32_t *__restrict__ word) {
  CarriedSum v{0.0, 0.0};
  for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) carry_add(v, partial[i], partial[n + i]);
  v = block_sum(v);
  if (threadIdx.x == 0) {
    out[0] = carried(v);
    if (word) *reinterpret_cast<uint32_t *>(out + 1) = *word;
  }
}

__device__ __forceinline__ double pauli_signed(double v, uint32_t bit31) {
  return __hiloint2double(__double2hiint(v) ^ int(bit31 & 0x80000000u), __double2loint(v));
}

struct alignas(16) PauliTerm {
  double f;
  uint32_t word;  // Z-or-Y mask in tile coordinates | parity of the tile base << 31
  uint32_t c;     // flip mask of its group
};
struct PauliShared {
  double2 *tile;
  PauliTerm *term;
  double2 *sign;  // per term: +-1 for row bits 0 and 1
  PauliTileGroup *group;
  __device__ PauliShared(unsigned char *raw, uint32_t terms) {
    tile = reinterpret_cast<double2 *>(raw);
    term = reinterpret_cast<PauliTerm *>(tile + (1u << kPauliTileBits));
    sign = reinterpret_cast<double2 *>(term + terms);
    group = reinterpret_cast<PauliTileGroup *>(sign + terms);
  }
};

// Pair product of one group: Re conj(a) b, or Im conj(a) b for an odd number
// of Y (either amplitude of the pair may be a: the signs make up for it).
template <bool ODD>
__device__ __forceinline__ double pauli_pair(const double2 &a, const double2 &b) {
  return ODD ? fma(a.x, b.y, -a.y * b.x) : fma(a.x, b.x, a.y * b.y);
}

// Pair products of the thread's four amplitudes in rows 0..3 under a flip
// that reaches the top tile bit.
template <bool ODD>
__device__ __forceinline__ void pauli_pairs_top(const double2 (&A)[4], const PauliShared &S, uint32_t c,
                                                double (&q)[4]) {
  const uint32_t at = threadIdx.x ^ c;
#pragma unroll
  for (int i = 0; i < 4; ++i) q[i] = pauli_pair<ODD>(A[i], S.tile[at ^ (i * kPauliThreads)]);
}

// acc + one term's share of such a group.
__device__ __forceinline__ double pauli_term_top(const PauliShared &S, const PauliTerm &T, uint32_t t,
                                                 const double (&q)[4], double acc) {
  const double2 g = S.sign[t];
  const double x = fma(g.y, fma(g.x, q[3], q[2]), fma(g.x, q[1], q[0]));
  return fma(pauli_signed(T.f, uint32_t(__popc(T.word & (threadIdx.x | 0x80000000u))) << 31), x, acc);
}

// The single-term groups [t0, t1) of a pass (terms in group order).
template <bool ODD>
__device__ __forceinline__ double pauli_singles(const double2 (&A)[4], const PauliShared &S, uint32_t t0, uint32_t t1,
                                                double acc) {
#pragma unroll 2
  for (uint32_t t = t0; t < t1; ++t) {
    const PauliTerm T = S.term[t];
    double q[4];
    pauli_pairs_top<ODD>(A, S, T.c, q);
    acc = pauli_term_top(S, T, t, q, acc);
  }
  return acc;
}

template <bool ODD>
__device__ __forceinline__ double pauli_group_top(const double2 (&A)[4], const PauliShared &S,
                                                  const PauliTileGroup &G, double acc) {
  double q[4];
  pauli_pairs_top<ODD>(A, S, G.c, q);
  for (uint32_t t = G.t0; t < G.t1; ++t) acc = pauli_term_top(S, S.term[t], t, q, acc);
  return acc;
}

// Any other off-diagonal group: the thread's four pairs are j ^ r_i and their
// partners, r_1 and r_2 one bit each, so a term's signs are again one parity
// of j and two factors over the rows.  A flip within 256 places: the threads
// with its highest bit clear take the pairs of rows 0..3, the others, each
// from its own place, those of rows 4..7 (consecutive places across the lanes:
// no bank conflicts).  Otherwise, and on a tile of 2^m < 2^11 amplitudes (zero
// above), pair k = i * 256 + tid with a zero inserted at the highest bit.
// The lowest qubit flipped, 28 qubits complex128: 887 us with a pair at a
// time, 691 us so (complex64 873, 671 us).
template <bool FULL, bool ODD>
__device__ __forceinline__ double pauli_group_any(const PauliShared &S, const PauliTileGroup &G, uint32_t m,
                                                  double acc) {
  if (!FULL && threadIdx.x >> (m - 1)) return acc;
  const uint32_t pivot = 31 - __clz(int(G.c));
  uint32_t j, r1, r2;
  if (FULL && pivot < 8) {
    j = threadIdx.x | ((threadIdx.x >> pivot) & 1u) << (kPauliTileBits - 1);
    r1 = 256u;
    r2 = 512u;
  } else {
    j = uint32_t(insert_zero(threadIdx.x, pivot));
    r1 = pivot > 8 ? 256u : 512u;
    r2 = pivot > 9 ? 512u : 1024u;
  }
  double2 a[4], b[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const uint32_t at = j ^ (i & 1 ? r1 : 0u) ^ (i & 2 ? r2 : 0u);
    a[i] = S.tile[at];
    b[i] = S.tile[at ^ G.c];
  }
  double q[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) q[i] = pauli_pair<ODD>(a[i], b[i]);
  for (uint32_t t = G.t0; t < G.t1; ++t) {
    const PauliTerm T = S.term[t];
    const double g1 = T.word & r1 ? -1.0 : 1.0, g2 = T.word & r2 ? -1.0 : 1.0;
    const double x = fma(g2, fma(g1, q[3], q[2]), fma(g1, q[1], q[0]));
    acc = fma(pauli_signed(T.f, uint32_t(__popc(T.word & (j | 0x80000000u))) << 31), x, acc);
  }
  return acc;
}

// The diagonal group: the eight rows' probabilities under the eight sign
// patterns of the row bits (a Walsh transform), then one weight per pattern.
__device__ __forceinline__ double pauli_diagonal(const PauliShared &S, const PauliTileGroup &G,
                                                 const uint16_t *diag) {
  double p[kPauliRows];
#pragma unroll
  for (int r = 0; r < kPauliRows; ++r) {
    const double2 a = S.tile[r * kPauliThreads + threadIdx.x];
    p[r] = fma(a.x, a.x, a.y * a.y);
  }
#pragma unroll
  for (int b = 1; b < kPauliRows; b <<= 1)
#pragma unroll
    for (int r = 0; r < kPauliRows; ++r)
      if (!(r & b)) {
        const double u = p[r], v = p[r | b];
        p[r] = u + v;
        p[r | b] = u - v;
      }
  const uint32_t tb = threadIdx.x | 0x80000000u;
  double s = 0.0;
#pragma unroll
  for (int z = 0; z < kPauliRows; ++z) {
    if (diag[z] == diag[z + 1]) continue;
    double w = 0.0;
    for (uint32_t t = G.t0 + diag[z]; t < uint32_t(G.t0 + diag[z + 1]); ++t)
      w += pauli_signed(S.term[t].f, uint32_t(__popc(S.term[t].word & tb)) << 31);
    s = fma(p[z], w, s);
  }
  return s;
}

// Copies a pass's groups and terms to shared memory (term numbers from 0).
// Ends without a barrier.
template <class Plan>
__device__ __forceinline__ void pauli_stage(const Plan &T, const PauliTilePass &S, PauliShared &sh) {
  const uint32_t t0 = T.group[S.g0].t0, t1 = T.group[S.g1 - 1].t1;
  const uint32_t singles = uint32_t(S.go - S.g0);  // their terms come first
  for (uint32_t i = threadIdx.x; i < t1 - t0; i += kPauliThreads) {
    const uint32_t z = T.zt[t0 + i];
    sh.term[i].f = T.f[t0 + i];
    sh.term[i].c = i < singles ? T.group[S.g0 + i].c : 0u;
    sh.sign[i] = make_double2(z & 256u ? -1.0 : 1.0, z & 512u ? -1.0 : 1.0);
  }
  for (uint32_t i = threadIdx.x; i < uint32_t(S.g1 - S.g0); i += kPauliThreads) {
    PauliTileGroup g = T.group[S.g0 + i];
    g.t0 = uint16_t(g.t0 - t0);
    g.t1 = uint16_t(g.t1 - t0);
    sh.group[i] = g;
  }
}

// Thread's share of all groups of one pass on tile `t`.  The pass is staged
// in sh (its barrier is the one below); ends with a barrier.
template <typename Real, bool FULL, class Plan>
__device__ __forceinline__ double pauli_tile(const typename Vec2<Real>::T *__restrict__ psi, const Plan &T,
                                             const PauliTilePass &S, uint64_t t, PauliShared &sh) {
  const uint32_t tid = threadIdx.x, low = T.low, m = T.m;
  uint64_t base = t << low;
  for (uint32_t i = 0; i < m - low; ++i) base = insert_zero(base, S.pivot[i]);
  uint64_t mine = base ^ (tid & ((1u << low) - 1u));
  for (uint32_t i = low; i < 8 && i < m; ++i)
    if ((tid >> i) & 1) mine ^= S.gen[i - low];
  const uint32_t rows = FULL ? kPauliRows : (m > 8 ? 1u << (m - 8) : (tid >> m) == 0 ? 1u : 0u);
  double2 A[4];
  {
    typename Vec2<Real>::T v[kPauliRows];
#pragma unroll
    for (int r = 0; r < kPauliRows; ++r) {
      uint64_t at = mine;
#pragma unroll
      for (int b = 0; b < 3; ++b)
        if ((r >> b) & 1) at ^= S.gen[8 + b - kPauliLowBits];
      if (FULL || uint32_t(r) < rows) {
        v[r] = psi[at];
      } else {
        v[r].x = 0;
        v[r].y = 0;
      }
    }
#pragma unroll
    for (int r = 0; r < kPauliRows; ++r) {
      const double2 a = make_double2(double(v[r].x), double(v[r].y));
      if (r < 4) A[r] = a;
      sh.tile[r * kPauliThreads + tid] = a;
    }
  }
  const uint32_t t0 = T.group[S.g0].t0, t1 = T.group[S.g1 - 1].t1;
  for (uint32_t i = tid; i < t1 - t0; i += kPauliThreads)
    sh.term[i].word = T.zt[t0 + i] | (uint32_t(__popcll(base & T.zy[t0 + i])) << 31);
  __syncthreads();
  const uint32_t even = uint32_t(S.ge - S.g0), odd = uint32_t(S.go - S.g0);
  double acc = pauli_singles<false>(A, sh, 0, even, 0.0), diagonal = 0.0;
  acc = pauli_singles<true>(A, sh, even, odd, acc);
  for (uint32_t g = odd; g < uint32_t(S.g1 - S.g0); ++g) {
    const PauliTileGroup G = sh.group[g];
    if (FULL && (G.c >> (kPauliTileBits - 1)))
      acc = G.odd ? pauli_group_top<true>(A, sh, G, acc) : pauli_group_top<false>(A, sh, G, acc);
    else if (G.c)
      acc = G.odd ? pauli_group_any<FULL, true>(sh, G, m, acc) : pauli_group_any<FULL, false>(sh, G, m, acc);
    else if (FULL || rows)
      diagonal += pauli_diagonal(sh, G, T.diag);
  }
  __syncthreads();
  return fma(2.0, acc, diagonal);  // pairs count twice (not in the weights: those may be near the range's end)
}

// The carried sum partial[blockIdx.x], partial[gridDim.x + blockIdx.x] (+)=
// this block's share of the plan's expectation.
template <typename Real, bool FULL, class Plan>
__global__ void __launch_bounds__(kPauliThreads, 4)
    pauli_expect_tiles(const typename Vec2<Real>::T *__restrict__ psi, const __grid_constant__ Plan T,
                       double *__restrict__ partial, int accumulate) {
  extern __shared__ __align__(16) unsigned char pauli_raw[];
  PauliShared sh(pauli_raw, T.max_terms);
  const uint32_t tile_bits = T.n - T.m;
  const uint64_t items = uint64_t(T.npasses) << tile_bits;
  uint32_t staged = ~0u;
  double acc = 0.0;  // a thread's tiles alternate over the state: its sum stays small
  for (uint64_t w = blockIdx.x; w < items; w += gridDim.x) {
    const uint32_t pass = uint32_t(w >> tile_bits);
    if (pass != staged) pauli_stage(T, T.pass[pass], sh);
    staged = pass;
    acc += pauli_tile<Real, FULL>(psi, T, T.pass[pass], w & ((uint64_t(1) << tile_bits) - 1), sh);
  }
  CarriedSum s = block_sum(CarriedSum{acc, 0.0});
  if (threadIdx.x == 0) {
    double *hi = partial + blockIdx.x, *lo = hi + gridDim.x;
    if (accumulate) carry_add(s, *hi, *lo);
    *hi = s.hi;
    *lo = s.lo;
  }
}

// A plan of one group that flips within the low bits, on a state of whole
// blocks: both amplitudes of a pair are in one line, so there is no tile to
// stage.  Bound: one read of the state, four pairs in flight.  (The tiles' form
// for such groups reads eight places a thread and group: the lowest qubit
// flipped, 28 qubits complex64, 671 us in tiles, 302 us here; complex128
// 691 and 636 us.)
template <typename Real, class Plan>
__global__ void __launch_bounds__(kPauliThreads)
    pauli_expect_low(const typename Vec2<Real>::T *__restrict__ psi, const __grid_constant__ Plan T,
                     double *__restrict__ partial, int accumulate) {
  constexpr int U = 4;
  const uint32_t x = T.group[0].c, top = 31 - __clz(int(x)), nt = T.group[0].t1;
  const bool odd = T.group[0].odd != 0;
  const uint64_t pairs = uint64_t(1) << (T.n - 1), step = uint64_t(gridDim.x) * (kPauliThreads * U);
  double acc = 0.0;
  for (uint64_t h = uint64_t(blockIdx.x) * (kPauliThreads * U) + threadIdx.x; h < pairs; h += step) {
    // insert_zero(h + u * 256, top): the steps lie above the inserted bit.
    const typename Vec2<Real>::T *p = psi + insert_zero(h, top);
    typename Vec2<Real>::T a[U], b[U];
#pragma unroll
    for (int u = 0; u < U; ++u) a[u] = p[u * 2 * kPauliThreads];
    p = psi + (insert_zero(h, top) ^ x);
#pragma unroll
    for (int u = 0; u < U; ++u) b[u] = p[u * 2 * kPauliThreads];
    double w[U] = {};
    for (uint32_t t = 0; t < nt; ++t) {
      const uint64_t zy = T.zy[t];
      const uint32_t own = uint32_t(__popcll(insert_zero(h, top) & zy));
#pragma unroll
      for (int u = 0; u < U; ++u)
        w[u] += pauli_signed(T.f[t], (own + __popc(uint32_t(u * 2 * kPauliThreads) & uint32_t(zy))) << 31);
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const double2 c = make_double2(double(a[u].x), double(a[u].y)), d = make_double2(double(b[u].x), double(b[u].y));
      acc = fma(odd ? pauli_pair<true>(c, d) : pauli_pair<false>(c, d), w[u], acc);
    }
  }
  CarriedSum s = block_sum(CarriedSum{2.0 * acc, 0.0});
  if (threadIdx.x == 0) {
    double *hi = partial + blockIdx.x, *lo = hi + gridDim.x;
    if (accumulate) carry_add(s, *hi, *lo);
    *hi = s.hi;
    *lo = s.lo;
  }
}

// Launches the kernel of a plan on `st` (2 x blocks partials).
template <typename Real, class Plan>
inline cudaError_t launch_pauli_plan(const void *psi, const Plan &P, double *partial, uint32_t blocks, int accumulate,
                                     cudaStream_t st) {
  uint32_t smem = pauli_tile_smem(P.max_terms, P.max_groups);
  auto fn = P.m == kPauliTileBits ? pauli_expect_tiles<Real, true, Plan> : pauli_expect_tiles<Real, false, Plan>;
  if (P.m == kPauliTileBits && P.npasses == 1 && P.pass[0].g1 == 1 && P.group[0].c && P.group[0].c < 8) {
    fn = pauli_expect_low<Real, Plan>;
    smem = 0;
  }
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               int(pauli_tile_smem(kPauliMaxTerms, kPauliMaxGroups)));
    if (e != cudaSuccess) return e;
  }
  fn<<<blocks, kPauliThreads, smem, st>>>(static_cast<const typename Vec2<Real>::T *>(psi), P, partial, accumulate);
  return cudaGetLastError();
}

template <typename Real>
inline cudaError_t launch_pauli_tiles(const void *psi, const PauliTilePlan &P, double *partial, uint32_t blocks,
                                      int accumulate, cudaStream_t st) {
  PauliSmallPlan S;
  return pauli_small_plan(P, S) ? launch_pauli_plan<Real>(psi, S, partial, blocks, accumulate, st)
                                : launch_pauli_plan<Real>(psi, P, partial, blocks, accumulate, st);
}

}  // namespace sq
