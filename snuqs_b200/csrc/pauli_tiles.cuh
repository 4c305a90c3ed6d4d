// Kernels of the tiled Pauli-sum expectation (pauli_tiles.h has the plan),
// FP64 throughout for both state precisions.
//
// What bounds it: one read of the state per pass, against one shared-memory
// read and three FP64 operations per pair and group.  A block holds one tile
// of 2^11 amplitudes (32 KiB as complex doubles) and each of its 256 threads
// the eight amplitudes r * 256 + tid of it in registers; a pair's partner is
// then one 16-byte shared read (lanes read an XOR of consecutive slots:
// conflict-free without a swizzle), and each pair is taken by one thread:
//  - the flip reaches register bits: the threads take the four of their
//    amplitudes with the lowest flipped register bit clear;
//  - else the thread with the highest flipped thread bit clear takes
//    amplitudes 0..3, its partner 4..7 (the term is symmetric in the pair).
// Signs (-1)^popc(i & zy) split over tile base, thread and register: the
// base's parities are computed once per tile and term, the rows' by the host.
// Measured on B200, 25 qubits complex128: 64 random strings (8 passes) and 25
// diagonal ones 2110 us together, before with one read of the state per mask
// 6212 us; the energy pass of 512 VQE circuits of 8..20 qubits 5.9 ms, before
// 11.9 ms.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "pauli_tiles.h"
#include "reduce_kernels.cuh"

namespace sq {

constexpr int kPauliThreads = 256;
constexpr int kPauliRows = (1 << kPauliTileBits) / kPauliThreads;

__device__ __forceinline__ double pauli_signed(double v, uint32_t bit31) {
  return __hiloint2double(__double2hiint(v) ^ int(bit31 & 0x80000000u), __double2loint(v));
}

struct PauliShared {
  double2 *tile;
  PauliTileGroup *group;
  double *f;
  uint32_t *word;  // thread bits of the Z-or-Y mask | row parities << 16 | parity of the tile base << 31
  __device__ PauliShared(unsigned char *raw, uint32_t terms, uint32_t groups) {
    tile = reinterpret_cast<double2 *>(raw);
    group = reinterpret_cast<PauliTileGroup *>(raw + (16u << kPauliTileBits));
    f = reinterpret_cast<double *>(group + groups);
    word = reinterpret_cast<uint32_t *>(f + terms);
  }
};

// Thread's share of one group.  PB: register bit the four amplitudes have
// clear; PB < 0: no register bit is flipped (half = the thread's pivot bit).
template <int PB, bool FULL>
__device__ __forceinline__ double pauli_group(const double2 (&A)[kPauliRows], const PauliShared &S,
                                              const PauliTileGroup &G, uint32_t tb, uint32_t rows, uint32_t half) {
  const uint32_t tid = threadIdx.x, c = G.c;
  const double2 *partner = S.tile + (tid ^ (c & (kPauliThreads - 1)));
  const uint32_t cr = c / kPauliThreads;
  double q[4];
  uint32_t row[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    double2 a;
    if constexpr (PB < 0) {
      row[i] = i + 4 * half;
      a.x = half ? A[i + 4].x : A[i].x;
      a.y = half ? A[i + 4].y : A[i].y;
    } else {
      constexpr int P = PB < 0 ? 0 : PB;
      const int r = ((i >> P) << (P + 1)) | (i & ((1 << P) - 1));
      row[i] = r;
      a = A[r];
    }
    const double2 b = partner[(row[i] ^ cr) * kPauliThreads];
    q[i] = G.odd ? fma(a.x, b.y, -a.y * b.x) : fma(a.x, b.x, a.y * b.y);
  }
  double s = 0.0;
  for (uint32_t t = G.t0; t < G.t1; ++t) {
    const uint32_t word = S.word[t], sg = uint32_t(__popc(word & tb)) << 31;
    double x = 0.0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const double v = pauli_signed(q[i], sg ^ (word << (15 - row[i])));
      if (FULL || row[i] < rows) x += v;
    }
    s = fma(S.f[t], x, s);
  }
  return s;
}

template <bool FULL>
__device__ __forceinline__ double pauli_diagonal(const double2 (&A)[kPauliRows], const PauliShared &S,
                                                 const PauliTileGroup &G, uint32_t tb, uint32_t rows) {
  double w[kPauliRows] = {};
  for (uint32_t t = G.t0; t < G.t1; ++t) {
    const uint32_t word = S.word[t];
    const double f = pauli_signed(S.f[t], uint32_t(__popc(word & tb)) << 31);
#pragma unroll
    for (int r = 0; r < kPauliRows; ++r) w[r] += pauli_signed(f, word << (15 - r));
  }
  double s = 0.0;
#pragma unroll
  for (int r = 0; r < kPauliRows; ++r)
    if (FULL || uint32_t(r) < rows) s = fma(fma(A[r].x, A[r].x, A[r].y * A[r].y), w[r], s);
  return s;
}

// Copies a pass's groups and terms to shared memory (term numbers from 0).
// Ends without a barrier.
__device__ __forceinline__ void pauli_stage(const PauliTilePlan &T, const PauliTilePass &S, PauliShared &sh) {
  const uint32_t t0 = T.group[S.g0].t0, t1 = T.group[S.g1 - 1].t1;
  for (uint32_t i = threadIdx.x; i < t1 - t0; i += kPauliThreads) sh.f[i] = T.f[t0 + i];
  for (uint32_t i = threadIdx.x; i < uint32_t(S.g1 - S.g0); i += kPauliThreads) {
    PauliTileGroup g = T.group[S.g0 + i];
    g.t0 = uint16_t(g.t0 - t0);
    g.t1 = uint16_t(g.t1 - t0);
    sh.group[i] = g;
  }
}

// Thread's share of all groups of one pass on tile `t`.  The pass is staged
// in sh (its barrier is the one below); ends with a barrier.
template <typename Real, bool FULL>
__device__ __forceinline__ double pauli_tile(const typename Vec2<Real>::T *__restrict__ psi, const PauliTilePlan &T,
                                             const PauliTilePass &S, uint64_t t, PauliShared &sh) {
  const uint32_t tid = threadIdx.x, low = T.low, m = T.m;
  uint64_t base = t << low;
  for (uint32_t i = 0; i < m - low; ++i) base = insert_zero(base, S.pivot[i]);
  uint64_t mine = base ^ (tid & ((1u << low) - 1u));
  for (uint32_t i = low; i < 8 && i < m; ++i)
    if ((tid >> i) & 1) mine ^= S.gen[i - low];
  const uint32_t rows = FULL ? kPauliRows : (m > 8 ? 1u << (m - 8) : (tid >> m) == 0 ? 1u : 0u);
  double2 A[kPauliRows];
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
    for (int r = 0; r < kPauliRows; ++r) A[r] = make_double2(double(v[r].x), double(v[r].y));
  }
#pragma unroll
  for (int r = 0; r < kPauliRows; ++r) sh.tile[r * kPauliThreads + tid] = A[r];
  const uint32_t t0 = T.group[S.g0].t0, t1 = T.group[S.g1 - 1].t1;
  for (uint32_t i = tid; i < t1 - t0; i += kPauliThreads)
    sh.word[i] = (T.zt[t0 + i] & 0xff00ffu) | (uint32_t(__popcll(base & T.zy[t0 + i])) << 31);
  __syncthreads();
  const uint32_t tb = tid | 0x80000000u;
  double acc = 0.0;
  for (uint32_t g = 0; g < uint32_t(S.g1 - S.g0); ++g) {
    const PauliTileGroup G = sh.group[g];
    const uint32_t cr = G.c / kPauliThreads;
    if (G.c == 0) {
      acc += pauli_diagonal<FULL>(A, sh, G, tb, rows);
    } else if (cr & 1) {
      acc += pauli_group<0, FULL>(A, sh, G, tb, rows, 0);
    } else if (cr & 2) {
      acc += pauli_group<1, FULL>(A, sh, G, tb, rows, 0);
    } else if (cr) {
      acc += pauli_group<2, FULL>(A, sh, G, tb, rows, 0);
    } else {
      const uint32_t half = (tid >> (31 - __clz(int(G.c)))) & 1u;
      if (FULL) {
        acc += pauli_group<-1, FULL>(A, sh, G, tb, rows, half);
      } else {
        // Fewer than eight rows: the thread with the pivot bit clear takes
        // all of its amplitudes (rows 4..7 do not exist below 2^11).
        const double s = pauli_group<-1, FULL>(A, sh, G, tb, rows, 0);
        acc += half ? 0.0 : s;
      }
    }
  }
  __syncthreads();
  return acc;
}

// partial[blockIdx.x] (+)= this block's share of the plan's expectation.
template <typename Real, bool FULL>
__global__ void __launch_bounds__(kPauliThreads, 3)
    pauli_expect_tiles(const typename Vec2<Real>::T *__restrict__ psi, const __grid_constant__ PauliTilePlan T,
                       double *__restrict__ partial, int accumulate) {
  extern __shared__ __align__(16) unsigned char pauli_raw[];
  PauliShared sh(pauli_raw, T.max_terms, T.max_groups);
  const uint32_t tile_bits = T.n - T.m;
  const uint64_t items = uint64_t(T.npasses) << tile_bits;
  uint32_t staged = ~0u;
  double acc = 0.0;
  for (uint64_t w = blockIdx.x; w < items; w += gridDim.x) {
    const uint32_t pass = uint32_t(w >> tile_bits);
    if (pass != staged) pauli_stage(T, T.pass[pass], sh);
    staged = pass;
    acc += pauli_tile<Real, FULL>(psi, T, T.pass[pass], w & ((uint64_t(1) << tile_bits) - 1), sh);
  }
  const double s = block_sum(acc);
  if (threadIdx.x == 0) partial[blockIdx.x] = accumulate ? partial[blockIdx.x] + s : s;
}

// Launches pauli_expect_tiles on `st`; returns the number of partials in
// *blocks (at most max_blocks).
template <typename Real>
inline cudaError_t launch_pauli_tiles(const void *psi, const PauliTilePlan &P, double *partial, uint32_t blocks,
                                      int accumulate, cudaStream_t st) {
  const uint32_t smem = pauli_tile_smem(P.max_terms, P.max_groups);
  auto fn = P.m == kPauliTileBits ? pauli_expect_tiles<Real, true> : pauli_expect_tiles<Real, false>;
  if (smem > 48 * 1024) {
    const cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               int(pauli_tile_smem(kPauliMaxTerms, kPauliMaxGroups)));
    if (e != cudaSuccess) return e;
  }
  fn<<<blocks, kPauliThreads, smem, st>>>(static_cast<const typename Vec2<Real>::T *>(psi), P, partial, accumulate);
  return cudaGetLastError();
}

}  // namespace sq
