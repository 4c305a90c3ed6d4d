// Result kernels beyond the expectation value: measurement sampling,
// amplitude lookup, marginal probabilities and Pauli-sum variance.
//
// The reference computes every result on the host after copying the whole
// state back: probabilities as |psi|^2 in numpy and shots with
// np.random.choice over them (src/braket/snuqs/simulation.py:208-220); its
// plugin registers no Expectation / Variance / Probability / Amplitude
// result types (src/braket/snuqs/result_types.py:149-151,
// src/braket/snuqs/simulator.py:578-580).  Here each is a device pass over
// the resident state and only the results cross PCIe.
//
// Sampling is an inverse CDF over |psi_i|^2 that is reproducible bit for bit:
// the probabilities are summed in one fixed binary tree (pairs of adjacent
// amplitudes, then pairs of pairs, ...), and a shot with uniform u walks that
// tree from the root with r = u * total: at a node with children sums (L, R)
// it goes left when r < L or R == 0, else subtracts L and goes right.  The
// tree is cut at nodes of 2^7 (2^5) amplitudes: the levels from there up stay in
// device memory, the levels inside a node are rebuilt in registers by the warp
// that serves a shot.  Any restatement that sums in the same tree and walks
// it the same way returns the same indices.
#include <cuda_runtime.h>

#include <algorithm>
#include <complex>
#include <cstring>
#include <functional>
#include <map>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/snuqs_b200.h"
#include "engine_internal.h"
#include "sweep_kernels.cuh"

namespace {

// Amplitudes of one block of the first pass, and the size of the nodes that
// the stored tree ends at: 2^7 amplitudes up to 30 qubits, then as large as
// keeps the stored tree at 2^24 doubles (128 MiB).  Nodes of 2^5 where the
// shots together would read more than the state in nodes of 2^7 and the two
// further levels are small (at most 16 MiB, up to 25 qubits), from 2^14 shots
// (below, a call is its launches and copies): 10^6 shots of 20 /
// 23 qubits complex128 195 / 231 us on the device, with nodes of 2^7 396 / 428 us
// (with leaves of 2^12 summed again by blocks 509 / 204 us).
constexpr int kBlockBits = 12;
constexpr uint32_t kBlockAmps = 1u << kBlockBits;
constexpr int kTreeThreads = 256;
constexpr uint32_t kPerLane = kBlockAmps / kTreeThreads;  // 16 amplitudes, 32 apart
constexpr uint32_t kNodeBits = 7, kFineBits = 5;
constexpr uint32_t kMaxTreeDepth = 23;

uint32_t node_bits(uint32_t n, uint64_t shots) {
  if (n <= 25 && shots >= std::max(uint64_t(1) << 14, (uint64_t(1) << n) >> kNodeBits)) return kFineBits;
  return n > kNodeBits + kMaxTreeDepth ? n - kMaxTreeDepth : kNodeBits;
}

template <typename C2>
__device__ __forceinline__ double prob_of(const C2 &a) {
  const double re = double(a.x), im = double(a.y);
  return __dadd_rn(__dmul_rn(re, re), __dmul_rn(im, im));
}

// First pass (bound: one read of the state): the sums of the fixed tree (pairs
// of consecutive amplitudes, level by level) from nodes of 2^node_bits up to
// 2^12 amplitudes.  Heap layout: the 2^d nodes of depth d at tree + 2^d, so the
// root is tree[1] and the children of node k are the 16-byte pair 2k, 2k + 1.
// Warp w covers the 512 amplitudes from 512 w; lane l reads amplitude 32 k + l
// for k = 0..15 (coalesced), the five lowest levels of each group of 32 are
// lane pairs l, l^1, l^2, ... (shuffles; a commutative add gives both partners
// the same value), the next four are the groups k in registers, then the
// warps pairwise through shared memory.
template <typename C2>
__global__ void __launch_bounds__(kTreeThreads) node_sum_kernel(const C2 *__restrict__ psi, uint32_t n,
                                                                uint32_t node, double *__restrict__ tree) {
  __shared__ double ws[kTreeThreads / 32];
  const uint64_t N = uint64_t(1) << n;
  const int depth = n > node ? int(n - node) : 0;  // of the nodes of 2^node amplitudes
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint64_t base = uint64_t(blockIdx.x) * kBlockAmps + uint64_t(warp) * (32 * kPerLane) + lane;
  double v[kPerLane];
#pragma unroll
  for (uint32_t k = 0; k < kPerLane; ++k)  // states below 2^12 amplitudes are padded with zeros
    v[k] = base + 32 * k < N ? prob_of(psi[base + 32 * k]) : 0.0;
  // Node j of this block at the level of 2^s amplitudes.
  auto put = [&](uint32_t s, uint32_t j, double x) {
    const int d = depth - int(s - node);
    if (d < 0) return;
    const uint64_t at = uint64_t(blockIdx.x) * (kBlockAmps >> s) + j;
    if (at < (uint64_t(1) << d)) tree[(uint64_t(1) << d) + at] = x;
  };
#pragma unroll
  for (int o = 1; o < 32; o <<= 1)
#pragma unroll
    for (uint32_t k = 0; k < kPerLane; ++k) v[k] = __dadd_rn(v[k], __shfl_xor_sync(0xffffffffu, v[k], o));
  if (node <= kFineBits && lane == 0) {
#pragma unroll
    for (uint32_t j = 0; j < kPerLane; ++j) put(kFineBits, warp * kPerLane + j, v[j]);
  }
#pragma unroll
  for (uint32_t w = kPerLane / 2, s = 6; w >= 1; w >>= 1, ++s) {
#pragma unroll
    for (uint32_t j = 0; j < w; ++j) v[j] = __dadd_rn(v[2 * j], v[2 * j + 1]);
    if (s >= node && lane == 0) {
#pragma unroll
      for (uint32_t j = 0; j < w; ++j) put(s, warp * w + j, v[j]);
    }
  }
  if (lane == 0) ws[warp] = v[0];
  __syncthreads();
  if (threadIdx.x == 0) {
    double w[kTreeThreads / 32];
#pragma unroll
    for (int j = 0; j < kTreeThreads / 32; ++j) w[j] = ws[j];
#pragma unroll
    for (uint32_t m = kTreeThreads / 64, s = 10; m >= 1; m >>= 1, ++s)
#pragma unroll
      for (uint32_t j = 0; j < m; ++j) {
        w[j] = __dadd_rn(w[2 * j], w[2 * j + 1]);
        if (s >= node) put(s, j, w[j]);
      }
  }
}

// `levels` (1..11) levels above depth `from`: block b sums the 2^levels nodes
// from node b << levels, through shared memory.
constexpr uint32_t kUpperLevels = 11;
__global__ void __launch_bounds__(1024) upper_tree_kernel(double *__restrict__ tree, uint32_t from, uint32_t levels) {
  __shared__ __align__(16) double buf[2][1u << (kUpperLevels - 1)];  // read in pairs
  uint32_t nodes = 1u << levels;
  const double2 *src = reinterpret_cast<const double2 *>(tree + ((uint64_t(1) << from) + (uint64_t(blockIdx.x) << levels)));
  for (uint32_t l = 1; l <= levels; ++l) {
    nodes >>= 1;
    const uint64_t at = (uint64_t(1) << (from - l)) + (uint64_t(blockIdx.x) << (levels - l));
    if (threadIdx.x < nodes) {
      const double2 c = l == 1 ? src[threadIdx.x] : reinterpret_cast<const double2 *>(buf[l & 1])[threadIdx.x];
      const double x = __dadd_rn(c.x, c.y);
      tree[at + threadIdx.x] = x;
      buf[(l + 1) & 1][threadIdx.x] = x;
    }
    __syncthreads();
  }
}

__device__ __forceinline__ bool go_left(double r, double l, double rr) { return r < l || rr == 0.0; }

// Four consecutive amplitudes' probabilities (zero past the end of the state).
template <typename C2>
__device__ __forceinline__ void prob4(const C2 *__restrict__ psi, uint64_t i, uint64_t N, double (&p)[4]) {
  if constexpr (sizeof(C2) == 8) {
    if (i + 4 <= N) {
      const float4 *q = reinterpret_cast<const float4 *>(psi + i);
      const float4 x = q[0], y = q[1];
      p[0] = prob_of(make_float2(x.x, x.y));
      p[1] = prob_of(make_float2(x.z, x.w));
      p[2] = prob_of(make_float2(y.x, y.y));
      p[3] = prob_of(make_float2(y.z, y.w));
      return;
    }
  }
#pragma unroll
  for (int j = 0; j < 4; ++j) p[j] = i + j < N ? prob_of(psi[i + j]) : 0.0;
}

// One warp per `per_warp` (1..32) shots.  First every lane walks one shot down
// the stored tree (one 16-byte pair of children per level; the warp's 32 walks
// overlap), then the warp serves its shots one by one: lane l holds amplitudes
// 4l..4l+3 of the shot's 128-amplitude node, the five levels above them are
// lane pairs as in node_sum_kernel, and the walk goes on in registers.
// EXTRA > 0 (more than 30 qubits): the stored nodes hold 2^EXTRA runs of 128
// amplitudes, whose sums are rebuilt first.  EXTRA = -2: nodes of 32, one
// amplitude a lane.
// A shot reads 128 amplitudes, wherever it falls; before, each leaf of 2^12
// amplitudes that any shot fell into was read and summed again by a block, for
// many shots the whole state a second time, after a counting sort of the
// shots by leaf.  10^6 shots of 28 qubits complex128 on B200: 424 us and 5 us
// for the tree's upper levels (2 GB of runs: 0.73 of the copy bandwidth),
// before 1760 us and 140 us for the sort and the upper levels; the first pass
// 681 us (0.97 of the copy bandwidth; 602 us without storing the lower levels).
template <typename C2, int EXTRA>
__global__ void __launch_bounds__(256) shot_kernel(const C2 *__restrict__ psi, uint32_t n,
                                                   const double *__restrict__ tree, const double *__restrict__ u,
                                                   uint64_t shots, uint32_t per_warp, uint64_t *__restrict__ out) {
  constexpr unsigned kAll = 0xffffffffu;
  const uint64_t N = uint64_t(1) << n;
  const uint32_t node = kNodeBits + EXTRA;
  const uint32_t depth = n > node ? n - node : 0;
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t first = ((uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5) * per_warp;
  if (first >= shots) return;  // uniform over the warp
  const uint32_t mine = uint32_t(shots - first < per_warp ? shots - first : per_warp);
  double r = 0.0;
  uint64_t k = 1;
  if (lane < mine) {
    r = __dmul_rn(u[first + lane], tree[1]);
    for (uint32_t d = 0; d < depth; ++d) {
      const double2 c = reinterpret_cast<const double2 *>(tree)[k];
      k = 2 * k;
      if (!go_left(r, c.x, c.y)) {
        r = __dsub_rn(r, c.x);
        ++k;
      }
    }
  }
  const uint64_t leaf = (k - (uint64_t(1) << depth)) << node;
  for (uint32_t j = 0; j < mine; ++j) {
    uint64_t base = __shfl_sync(kAll, leaf, j);
    double rr = __shfl_sync(kAll, r, j);
    double p[4];
    if constexpr (EXTRA > 0) {
      constexpr int B = 1 << EXTRA;
      double t[2 * B];  // heap of the node's 128-amplitude runs
#pragma unroll 1
      for (int b = 0; b < B; ++b) {
        prob4(psi, base + uint64_t(b) * 128 + 4 * lane, N, p);
        double s = __dadd_rn(__dadd_rn(p[0], p[1]), __dadd_rn(p[2], p[3]));
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) s = __dadd_rn(s, __shfl_xor_sync(kAll, s, o));
        t[B + b] = s;
      }
      for (int i = B - 1; i >= 1; --i) t[i] = __dadd_rn(t[2 * i], t[2 * i + 1]);
      int at = 1;
#pragma unroll 1
      for (int e = 0; e < EXTRA; ++e) {
        const double l = t[2 * at], q = t[2 * at + 1];
        at = 2 * at;
        if (!go_left(rr, l, q)) {
          rr = __dsub_rn(rr, l);
          ++at;
        }
      }
      base += uint64_t(at - B) * 128;
    }
    constexpr uint32_t PER = EXTRA < 0 ? 1 : 4;
    if constexpr (EXTRA < 0) p[0] = base + lane < N ? prob_of(psi[base + lane]) : 0.0;
    else prob4(psi, base + 4 * lane, N, p);
    double lo = p[0], hi = 0.0;
    if constexpr (EXTRA >= 0) {
      lo = __dadd_rn(p[0], p[1]);
      hi = __dadd_rn(p[2], p[3]);
    }
    // sum[e]: the run of 2^e lanes this lane belongs to.
    double sum[5];
    sum[0] = EXTRA < 0 ? lo : __dadd_rn(lo, hi);
#pragma unroll
    for (int e = 0; e < 4; ++e) sum[e + 1] = __dadd_rn(sum[e], __shfl_xor_sync(kAll, sum[e], 1 << e));
    uint32_t at = 0;  // first lane of the node walked to
#pragma unroll
    for (int e = 4; e >= 0; --e) {
      const double l = __shfl_sync(kAll, sum[e], at), q = __shfl_sync(kAll, sum[e], at + (1u << e));
      if (!go_left(rr, l, q)) {
        rr = __dsub_rn(rr, l);
        at += 1u << e;
      }
    }
    if (lane == at) {
      uint32_t a = 0;
      if constexpr (EXTRA >= 0) {
        double l = p[0], q = p[1];
        if (!go_left(rr, lo, hi)) {
          rr = __dsub_rn(rr, lo);
          a = 2;
          l = p[2];
          q = p[3];
        }
        if (!go_left(rr, l, q)) ++a;
      }
      out[first + j] = base + PER * lane + a;
    }
  }
}

template <typename C2>
__global__ void amplitude_kernel(const C2 *__restrict__ psi, uint64_t N, const uint64_t *__restrict__ idx,
                                 uint64_t count, double2 *__restrict__ out, uint32_t *__restrict__ bad) {
  const uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= count) return;
  const uint64_t j = idx[i];
  if (j >= N) {
    atomicOr(bad, 1u);
    out[i] = make_double2(0.0, 0.0);
    return;
  }
  const C2 a = psi[j];
  out[i] = make_double2(double(a.x), double(a.y));
}

// Marginal probabilities over k target bits: out[b] = sum of |psi_i|^2 over
// the indices i whose target bits spell b.
//
// Bound: one read of the state.  A warp's lanes sit on the `low` = 5 lowest
// index bits whatever the targets are, so every load covers a run of 32
// amplitudes; the other bits split into target and rest positions.  An item
// is one assignment of the high target bits and one chunk of the high rest
// bits: its indices are base | rest with rest walked in ascending order by
// (rest - mask) & mask (two integer operations instead of depositing n bits
// for every amplitude), eight loads in flight per lane.  With fewer than
// eight rest assignments (CL < 3) the eight loads cover 8 >> CL neighbouring
// target assignments instead.  Lanes on rest bits are summed by shuffles,
// lanes on target bits write different bins.
// Measured on B200 (device time): targets of 1 / 5 / 11 of 26 qubits
// complex128 514 us for the three (0.97 of the copy bandwidth), the 2^20
// probabilities of 20 qubits 6.5 us.  With one block per (bin, chunk) and a
// bit deposit per amplitude these took 3052 us and 3699 us.
constexpr int kMarginalThreads = 256;
constexpr uint32_t kMarginalWarps = kMarginalThreads / 32;
struct MarginalParams {
  uint32_t n, low;      // lane bits: min(n, 5) lowest index bits
  uint32_t th, rh;      // target / rest bits above them
  uint32_t log_chunks;  // chunks of the high rest assignments per bin: 0, or at least 3
  uint32_t lane_rest;   // lane bits that are not targets
  uint64_t rest_step;   // high rest bits except the lowest CL
  uint8_t tpos[64];     // high target positions, ascending
  uint8_t tout[64];     // and the output bit of each
  uint8_t rpos[64];     // high rest positions, ascending
  uint32_t lane_out[5]; // output weight of lane bit p (0: not a target)
};

template <typename C2, int CL>
__global__ void __launch_bounds__(kMarginalThreads)
    marginal_kernel(const C2 *__restrict__ psi, const __grid_constant__ MarginalParams P, double *__restrict__ out) {
  constexpr int U = 8, G = U >> CL;
  __shared__ double ws[kMarginalWarps][32];
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint64_t bins_hi = uint64_t(1) << P.th;
  const uint64_t items = ((bins_hi + G - 1) / G) << P.log_chunks;
  const uint64_t steps = (uint64_t(1) << (P.rh - P.log_chunks)) >> CL;
  const bool live = lane < (1u << P.low);
  uint64_t lane_o = 0;
#pragma unroll
  for (int p = 0; p < 5; ++p)
    if ((lane >> p) & 1) lane_o |= P.lane_out[p];
  uint64_t goff[U], gout[G];  // offsets of the eight loads, output offsets of the G targets
#pragma unroll
  for (int u = 0; u < U; ++u) {
    uint64_t x = 0;
#pragma unroll
    for (int b = 0; b < 3; ++b)
      if ((u >> b) & 1) {
        if (b < CL) x |= uint64_t(1) << P.rpos[b];
        else if (uint32_t(b - CL) < P.th) x |= uint64_t(1) << P.tpos[b - CL];
      }
    goff[u] = x;
  }
#pragma unroll
  for (int g = 0; g < G; ++g) {
    uint64_t x = 0;
#pragma unroll
    for (int b = 0; b < 3 - CL; ++b)
      if (((g >> b) & 1) && uint32_t(b) < P.th) x |= uint64_t(1) << P.tout[b];
    gout[g] = x;
  }
  // Blocks take kMarginalWarps consecutive items, one per warp (with chunks,
  // all of one bin: log_chunks >= 3); every warp of a block makes the same
  // number of rounds, so the barriers below are uniform.
  for (uint64_t i0 = uint64_t(blockIdx.x) * kMarginalWarps; i0 < items; i0 += uint64_t(gridDim.x) * kMarginalWarps) {
    const uint64_t item = i0 + warp;
    double acc[U] = {0, 0, 0, 0, 0, 0, 0, 0};
    uint64_t ob = 0;
    const uint64_t a = (item >> P.log_chunks) * G;
    if (item < items) {
      uint64_t base = lane;
      for (uint32_t i = 0; i < P.th; ++i)
        if ((a >> i) & 1) {
          base |= uint64_t(1) << P.tpos[i];
          ob |= uint64_t(1) << P.tout[i];
        }
      const uint64_t r0 = (item & ((uint64_t(1) << P.log_chunks) - 1)) * (steps << CL);
      uint64_t rest = 0;
      for (uint32_t i = 0; i < P.rh; ++i)
        if ((r0 >> i) & 1) rest |= uint64_t(1) << P.rpos[i];
      if (live) {
        const C2 *p = psi + base;
        for (uint64_t s = 0; s < steps; ++s) {
          C2 v[U];
#pragma unroll
          for (int u = 0; u < U; ++u) v[u] = p[rest | goff[u]];
#pragma unroll
          for (int u = 0; u < U; ++u) {
            const double re = double(v[u].x), im = double(v[u].y);
            acc[u] = fma(re, re, fma(im, im, acc[u]));
          }
          rest = (rest - P.rest_step) & P.rest_step;
        }
      }
    }
#pragma unroll
    for (int g = 0; g < G; ++g) {
      double x = 0.0;
#pragma unroll
      for (int r = 0; r < (1 << CL); ++r) x += acc[(g << CL) | r];
#pragma unroll
      for (int p = 0; p < 5; ++p)
        if ((P.lane_rest >> p) & 1) x += __shfl_xor_sync(0xffffffffu, x, 1 << p);
      acc[g] = x;
    }
    if (P.log_chunks == 0) {
      if (item < items && live && !(lane & P.lane_rest)) {
#pragma unroll
        for (int g = 0; g < G; ++g)
          if (a + g < bins_hi) out[ob | gout[g] | lane_o] = acc[g];
      }
    } else {  // CL == 3: one value per lane; the block's eight chunks are summed in order
      ws[warp][lane] = acc[0];
      __syncthreads();
      if (warp == 0 && live && !(lane & P.lane_rest)) {
        double x = 0.0;
#pragma unroll
        for (uint32_t w = 0; w < kMarginalWarps; ++w) x += ws[w][lane];
        const uint64_t chunk = (i0 & ((uint64_t(1) << P.log_chunks) - 1)) / kMarginalWarps;
        out[((ob | lane_o) << (P.log_chunks - 3)) + chunk] = x;
      }
      __syncthreads();
    }
  }
}

// One block per bin: its partials in a fixed order.
__global__ void __launch_bounds__(256) marginal_finalize_kernel(const double *__restrict__ partial, uint32_t count,
                                                                double *__restrict__ out) {
  const double *p = partial + uint64_t(blockIdx.x) * count;
  __shared__ double ws[8];
  double s = 0.0;
  for (uint32_t c = threadIdx.x; c < count; c += 256) s += p[c];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double x = 0.0;
    for (int w = 0; w < 8; ++w) x += ws[w];
    out[blockIdx.x] = x;
  }
}

// Distance between two states of the same size, any precisions: per block
// max |a_i - b_i| and the FP64 sums <a|b> (re, im), <a|a>, <b|b>.
template <typename CA, typename CB>
__global__ void __launch_bounds__(256) distance_kernel(const CA *__restrict__ a, const CB *__restrict__ b, uint64_t N,
                                                       double *__restrict__ part) {
  __shared__ double sm[5][8];
  double mx = 0.0, re = 0.0, im = 0.0, na = 0.0, nb = 0.0;
  for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < N; i += uint64_t(gridDim.x) * blockDim.x) {
    const double ar = double(a[i].x), ai = double(a[i].y), br = double(b[i].x), bi = double(b[i].y);
    mx = fmax(mx, hypot(ar - br, ai - bi));
    re += ar * br + ai * bi;  // conj(a) b
    im += ar * bi - ai * br;
    na += ar * ar + ai * ai;
    nb += br * br + bi * bi;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    re += __shfl_xor_sync(0xffffffffu, re, o);
    im += __shfl_xor_sync(0xffffffffu, im, o);
    na += __shfl_xor_sync(0xffffffffu, na, o);
    nb += __shfl_xor_sync(0xffffffffu, nb, o);
  }
  const int w = threadIdx.x >> 5;
  if ((threadIdx.x & 31) == 0) {
    sm[0][w] = mx;
    sm[1][w] = re;
    sm[2][w] = im;
    sm[3][w] = na;
    sm[4][w] = nb;
  }
  __syncthreads();
  if (threadIdx.x < 5) {
    double v = threadIdx.x == 0 ? 0.0 : 0.0;
    for (int j = 0; j < 8; ++j) v = threadIdx.x == 0 ? fmax(v, sm[0][j]) : v + sm[threadIdx.x][j];
    part[uint64_t(blockIdx.x) * 5 + threadIdx.x] = v;
  }
}

int fail(int code, const std::string &msg) { return sq_detail_fail(code, msg.c_str()); }

#define RQ_CUDA(call)                                                                         \
  do {                                                                                        \
    cudaError_t e_ = (call);                                                                  \
    if (e_ != cudaSuccess)                                                                    \
      return fail(e_ == cudaErrorMemoryAllocation ? SQ_ERR_OOM : SQ_ERR_CUDA,                 \
                  std::string(#call) + ": " + cudaGetErrorString(e_));                        \
  } while (0)

size_t align256(size_t x) { return (x + 255) & ~size_t(255); }

// Scratch bytes of sample_impl: the stored tree.
size_t sample_scratch_bytes(uint32_t n, uint64_t shots) {
  const uint32_t node = node_bits(n, shots);
  return align256((uint64_t(2) << (n > node ? n - node : 0)) * sizeof(double));
}

// u_ready (optional): an event the shot phase waits for before reading the
// uniforms (they may still be in flight on another stream while the
// probability tree is built).
template <typename C2>
int sample_impl(const C2 *psi, uint32_t n, const double *u, uint64_t shots, uint64_t *out, void *scr,
                cudaStream_t st, cudaEvent_t u_ready = nullptr, const std::function<int()> &before_shots = {}) {
  double *tree = static_cast<double *>(scr);
  const uint32_t node = node_bits(n, shots);
  const uint32_t blocks_log = n > uint32_t(kBlockBits) ? n - kBlockBits : 0;
  node_sum_kernel<C2><<<1u << blocks_log, kTreeThreads, 0, st>>>(psi, n, node, tree);
  RQ_CUDA(cudaGetLastError());
  for (uint32_t from = blocks_log; from > 0;) {
    const uint32_t lv = std::min(from, kUpperLevels);
    upper_tree_kernel<<<1u << (from - lv), 1024, 0, st>>>(tree, from, lv);
    RQ_CUDA(cudaGetLastError());
    from -= lv;
  }
  if (before_shots) {
    const int rc = before_shots();
    if (rc != SQ_OK) return rc;
  }
  if (u_ready) RQ_CUDA(cudaStreamWaitEvent(st, u_ready, 0));
  // Shots per warp: as many as leave a warp for every slot of the GPU, at most
  // 32 (a warp serves its shots one after the other).
  int dev = 0, sms = 0;
  RQ_CUDA(cudaGetDevice(&dev));
  RQ_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  uint32_t per_warp = 32;
  while (per_warp > 1 && shots / per_warp < uint64_t(sms) * 64) per_warp >>= 1;
  const uint64_t warps = (shots + per_warp - 1) / per_warp;
  const unsigned grid = unsigned((warps + 7) / 8);
  switch (int(node) - int(kNodeBits)) {
    case -2: shot_kernel<C2, -2><<<grid, 256, 0, st>>>(psi, n, tree, u, shots, per_warp, out); break;
    case 0: shot_kernel<C2, 0><<<grid, 256, 0, st>>>(psi, n, tree, u, shots, per_warp, out); break;
    case 1: shot_kernel<C2, 1><<<grid, 256, 0, st>>>(psi, n, tree, u, shots, per_warp, out); break;
    case 2: shot_kernel<C2, 2><<<grid, 256, 0, st>>>(psi, n, tree, u, shots, per_warp, out); break;
    case 3: shot_kernel<C2, 3><<<grid, 256, 0, st>>>(psi, n, tree, u, shots, per_warp, out); break;
    default: shot_kernel<C2, 4><<<grid, 256, 0, st>>>(psi, n, tree, u, shots, per_warp, out);
  }
  RQ_CUDA(cudaGetLastError());
  return SQ_OK;
}

}  // namespace

extern "C" {

int sq_sample(sq_state *s, const double *uniforms_device, uint64_t shots, uint64_t *out_device, void *stream) {
  if (!s || (shots && (!uniforms_device || !out_device))) return fail(SQ_ERR_INVALID, "sq_sample: null pointer");
  if (shots > (uint64_t(1) << 31)) return fail(SQ_ERR_UNSUPPORTED, "sq_sample: more than 2^31 shots per call");
  auto st = static_cast<cudaStream_t>(stream);
  const int rc = sq_flush(s, stream);
  if (rc != SQ_OK || shots == 0) return rc;
  const uint32_t n = sq_state_num_qubits(s);
  if (n > 34) return fail(SQ_ERR_UNSUPPORTED, "sq_sample: more than 34 qubits");
  void *scr = nullptr;
  const int sc = sq_detail_state_scratch(s, sample_scratch_bytes(n, shots), &scr);
  if (sc != SQ_OK) return sc;
  if (sq_state_dtype(s) == SQ_C64)
    return sample_impl(static_cast<const float2 *>(sq_state_data(s)), n, uniforms_device, shots, out_device, scr, st);
  return sample_impl(static_cast<const double2 *>(sq_state_data(s)), n, uniforms_device, shots, out_device, scr,
                     st);
}

int sq_sample_host(sq_state *s, const double *uniforms, uint64_t shots, uint64_t *out, void *stream) {
  if (!s || (shots && (!uniforms || !out))) return fail(SQ_ERR_INVALID, "sq_sample_host: null pointer");
  if (shots > (uint64_t(1) << 31)) return fail(SQ_ERR_UNSUPPORTED, "sq_sample_host: more than 2^31 shots per call");
  auto st = static_cast<cudaStream_t>(stream);
  int rc = sq_flush(s, stream);
  if (rc != SQ_OK || shots == 0) return rc;
  const uint32_t n = sq_state_num_qubits(s);
  if (n > 34) return fail(SQ_ERR_UNSUPPORTED, "sq_sample_host: more than 34 qubits");
  // The state's scratch holds the uniforms and the indices, then the sampler's own scratch.
  const size_t b_u = align256(shots * sizeof(double)), b_o = align256(shots * sizeof(uint64_t));
  void *scr = nullptr;
  rc = sq_detail_state_scratch(s, b_u + b_o + sample_scratch_bytes(n, shots), &scr);
  if (rc != SQ_OK) return rc;
  char *p = static_cast<char *>(scr);
  double *du = reinterpret_cast<double *>(p);
  uint64_t *dout = reinterpret_cast<uint64_t *>(p + b_u);
  // Pinned staging (the state's, reused): the uniforms are copied into it
  // and go up on a second stream while the probability tree is built; the
  // shot phase waits for them; the indices come back through it.
  void *hs = nullptr;
  rc = sq_detail_state_host_scratch(s, std::max(shots * sizeof(double), shots * sizeof(uint64_t)), &hs);
  if (rc != SQ_OK) return rc;
  cudaStream_t cs = nullptr;
  cudaEvent_t prior = nullptr, ready = nullptr;
  struct Release {
    cudaStream_t &cs;
    cudaEvent_t &a, &b;
    ~Release() {
      if (a) cudaEventDestroy(a);
      if (b) cudaEventDestroy(b);
      if (cs) cudaStreamDestroy(cs);
    }
  } release{cs, prior, ready};
  RQ_CUDA(cudaStreamCreateWithFlags(&cs, cudaStreamNonBlocking));
  RQ_CUDA(cudaEventCreateWithFlags(&prior, cudaEventDisableTiming));
  RQ_CUDA(cudaEventCreateWithFlags(&ready, cudaEventDisableTiming));
  RQ_CUDA(cudaEventRecord(prior, st));  // earlier work on the state's stream
  auto upload = [&]() -> int {
    std::memcpy(hs, uniforms, shots * sizeof(double));  // while the tree kernels run
    RQ_CUDA(cudaStreamWaitEvent(cs, prior, 0));
    RQ_CUDA(cudaMemcpyAsync(du, hs, shots * sizeof(double), cudaMemcpyHostToDevice, cs));
    RQ_CUDA(cudaEventRecord(ready, cs));
    return SQ_OK;
  };
  rc = sq_state_dtype(s) == SQ_C64
           ? sample_impl(static_cast<const float2 *>(sq_state_data(s)), n, du, shots, dout, p + b_u + b_o, st,
                         ready, upload)
           : sample_impl(static_cast<const double2 *>(sq_state_data(s)), n, du, shots, dout, p + b_u + b_o, st,
                         ready, upload);
  if (rc != SQ_OK) {
    cudaStreamSynchronize(cs);
    return rc;
  }
  RQ_CUDA(cudaMemcpyAsync(hs, dout, shots * sizeof(uint64_t), cudaMemcpyDeviceToHost, st));
  RQ_CUDA(cudaStreamSynchronize(st));
  std::memcpy(out, hs, shots * sizeof(uint64_t));
  return SQ_OK;
}

int sq_amplitudes(sq_state *s, const uint64_t *indices_device, uint64_t count, double *out_device, void *stream) {
  if (!s || (count && (!indices_device || !out_device))) return fail(SQ_ERR_INVALID, "sq_amplitudes: null pointer");
  auto st = static_cast<cudaStream_t>(stream);
  int rc = sq_flush(s, stream);
  if (rc != SQ_OK || count == 0) return rc;
  void *scr = nullptr;
  rc = sq_detail_state_scratch(s, 256, &scr);
  if (rc != SQ_OK) return rc;
  uint32_t *bad = static_cast<uint32_t *>(scr);
  RQ_CUDA(cudaMemsetAsync(bad, 0, sizeof(uint32_t), st));
  const uint64_t N = uint64_t(1) << sq_state_num_qubits(s);
  const unsigned grid = unsigned((count + 255) / 256);
  auto *o = reinterpret_cast<double2 *>(out_device);
  if (sq_state_dtype(s) == SQ_C64)
    amplitude_kernel<float2><<<grid, 256, 0, st>>>(static_cast<const float2 *>(sq_state_data(s)), N,
                                                   indices_device, count, o, bad);
  else
    amplitude_kernel<double2><<<grid, 256, 0, st>>>(static_cast<const double2 *>(sq_state_data(s)), N,
                                                    indices_device, count, o, bad);
  RQ_CUDA(cudaGetLastError());
  uint32_t h = 0;
  RQ_CUDA(cudaMemcpyAsync(&h, bad, sizeof(h), cudaMemcpyDeviceToHost, st));
  RQ_CUDA(cudaStreamSynchronize(st));
  if (h) return fail(SQ_ERR_INVALID, "sq_amplitudes: an index is >= 2^num_qubits (its output is 0)");
  return SQ_OK;
}

int sq_marginal_probabilities(sq_state *s, const uint32_t *qubits, uint32_t k, double *out_device, void *stream) {
  if (!s || !out_device || (k && !qubits)) return fail(SQ_ERR_INVALID, "sq_marginal_probabilities: null pointer");
  const uint32_t n = sq_state_num_qubits(s);
  if (k > n) return fail(SQ_ERR_INVALID, "sq_marginal_probabilities: more targets than qubits");
  if (k > 30) return fail(SQ_ERR_UNSUPPORTED, "sq_marginal_probabilities: more than 30 target qubits");
  uint64_t tmask = 0;
  uint8_t outbit[64] = {0};  // output bit of each target index bit
  for (uint32_t j = 0; j < k; ++j) {
    if (qubits[j] >= n) return fail(SQ_ERR_INVALID, "sq_marginal_probabilities: qubit out of range");
    const uint64_t bit = uint64_t(1) << (n - 1 - qubits[j]);
    if (tmask & bit) return fail(SQ_ERR_INVALID, "sq_marginal_probabilities: repeated qubit");
    tmask |= bit;
    outbit[n - 1 - qubits[j]] = uint8_t(k - 1 - j);
  }
  auto st = static_cast<cudaStream_t>(stream);
  int rc = sq_flush(s, stream);
  if (rc != SQ_OK) return rc;
  int sms = 0, dev = 0;
  RQ_CUDA(cudaGetDevice(&dev));
  RQ_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  MarginalParams P;
  std::memset(&P, 0, sizeof(P));
  P.n = n;
  P.low = std::min(n, 5u);
  for (uint32_t p = 0; p < n; ++p) {
    const bool target = (tmask >> p) & 1;
    if (p < P.low) {
      if (target) P.lane_out[p] = 1u << outbit[p];
      else P.lane_rest |= 1u << p;
    } else if (target) {
      P.tpos[P.th] = uint8_t(p);
      P.tout[P.th++] = outbit[p];
    } else {
      P.rpos[P.rh++] = uint8_t(p);
    }
  }
  const uint32_t cl = std::min(3u, P.rh);
  for (uint32_t i = cl; i < P.rh; ++i) P.rest_step |= uint64_t(1) << P.rpos[i];
  // Chunks: about 2^16 warp items in all (seven rounds of the resident warps,
  // so that the last one is nearly full), at least eight loads each.
  uint32_t lc = P.th < 16 && P.rh > 3 ? std::min(16 - P.th, P.rh - 3) : 0;
  if (lc < 3) lc = 0;
  P.log_chunks = lc;
  const uint64_t bins = uint64_t(1) << k;
  double *dst = out_device;
  if (lc) {
    void *scr = nullptr;
    rc = sq_detail_state_scratch(s, (bins << (lc - 3)) * sizeof(double), &scr);
    if (rc != SQ_OK) return rc;
    dst = static_cast<double *>(scr);
  }
  const uint64_t g = 8u >> cl;
  const uint64_t items = (((uint64_t(1) << P.th) + g - 1) / g) << lc;
  const unsigned grid =
      unsigned(std::min<uint64_t>((items + kMarginalWarps - 1) / kMarginalWarps, uint64_t(sms) * 8));
  auto launch = [&](auto *psi) {
    switch (cl) {
      case 0: marginal_kernel<std::remove_pointer_t<decltype(psi)>, 0><<<grid, kMarginalThreads, 0, st>>>(psi, P, dst); break;
      case 1: marginal_kernel<std::remove_pointer_t<decltype(psi)>, 1><<<grid, kMarginalThreads, 0, st>>>(psi, P, dst); break;
      case 2: marginal_kernel<std::remove_pointer_t<decltype(psi)>, 2><<<grid, kMarginalThreads, 0, st>>>(psi, P, dst); break;
      default: marginal_kernel<std::remove_pointer_t<decltype(psi)>, 3><<<grid, kMarginalThreads, 0, st>>>(psi, P, dst);
    }
  };
  if (sq_state_dtype(s) == SQ_C64) launch(static_cast<float2 *>(sq_state_data(s)));
  else launch(static_cast<double2 *>(sq_state_data(s)));
  RQ_CUDA(cudaGetLastError());
  if (lc) {
    marginal_finalize_kernel<<<unsigned(bins), 256, 0, st>>>(dst, 1u << (lc - 3), out_device);
    RQ_CUDA(cudaGetLastError());
  }
  return SQ_OK;
}

int sq_state_distance(sq_state *a, sq_state *b, double *max_abs, double *one_minus_fidelity, void *stream) {
  if (!a || !b || !max_abs || !one_minus_fidelity) return fail(SQ_ERR_INVALID, "sq_state_distance: null pointer");
  const uint32_t n = sq_state_num_qubits(a);
  if (sq_state_num_qubits(b) != n) return fail(SQ_ERR_INVALID, "sq_state_distance: states of different size");
  auto st = static_cast<cudaStream_t>(stream);
  int rc = sq_flush(a, stream);
  if (rc == SQ_OK) rc = sq_flush(b, stream);
  if (rc != SQ_OK) return rc;
  int sms = 0, dev = 0;
  RQ_CUDA(cudaGetDevice(&dev));
  RQ_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  const uint64_t N = uint64_t(1) << n;
  const unsigned blocks = unsigned(std::max<uint64_t>(1, std::min<uint64_t>((N + 255) / 256, uint64_t(sms) * 4)));
  void *scr = nullptr;
  rc = sq_detail_state_scratch(a, size_t(blocks) * 5 * sizeof(double), &scr);
  if (rc != SQ_OK) return rc;
  double *part = static_cast<double *>(scr);
  const bool a64 = sq_state_dtype(a) == SQ_C64, b64 = sq_state_dtype(b) == SQ_C64;
  const void *pa = sq_state_data(a), *pb = sq_state_data(b);
  if (!a64 && !b64)
    distance_kernel<<<blocks, 256, 0, st>>>(static_cast<const double2 *>(pa), static_cast<const double2 *>(pb), N, part);
  else if (!a64 && b64)
    distance_kernel<<<blocks, 256, 0, st>>>(static_cast<const double2 *>(pa), static_cast<const float2 *>(pb), N, part);
  else if (a64 && !b64)
    distance_kernel<<<blocks, 256, 0, st>>>(static_cast<const float2 *>(pa), static_cast<const double2 *>(pb), N, part);
  else
    distance_kernel<<<blocks, 256, 0, st>>>(static_cast<const float2 *>(pa), static_cast<const float2 *>(pb), N, part);
  RQ_CUDA(cudaGetLastError());
  std::vector<double> h(size_t(blocks) * 5);
  RQ_CUDA(cudaMemcpyAsync(h.data(), part, h.size() * sizeof(double), cudaMemcpyDeviceToHost, st));
  RQ_CUDA(cudaStreamSynchronize(st));
  double mx = 0, re = 0, im = 0, na = 0, nb = 0;
  for (unsigned i = 0; i < blocks; ++i) {
    mx = std::max(mx, h[5 * i]);
    re += h[5 * i + 1];
    im += h[5 * i + 2];
    na += h[5 * i + 3];
    nb += h[5 * i + 4];
  }
  *max_abs = mx;
  *one_minus_fidelity = (na > 0 && nb > 0) ? 1.0 - (re * re + im * im) / (na * nb) : 1.0;
  return SQ_OK;
}

}  // extern "C"
