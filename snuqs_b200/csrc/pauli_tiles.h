// Pauli-sum expectations by tiles: the plan the host makes and the kernels
// (pauli_tiles.cuh) run.
//
// A Pauli string with flip mask x pairs amplitude i with i ^ x, so a group of
// strings of one mask needs one read of the state when the pairs are fetched
// from memory.  Flip masks form a vector space over GF(2): a tile that holds
// a coset base ^ span(v_1 .. v_k) of index space holds both amplitudes of
// every pair of EVERY group whose mask lies in the span.  A pass therefore
// collects groups while their masks fit a span of kPauliTileBits dimensions
// (the kPauliLowBits lowest index bits, so that a tile is made of 128-byte
// runs of complex128 amplitudes, and eight more generators), and the state is
// read once per pass: 64 random strings of 25 qubits take 8 passes instead
// of 64 reads.
//
// The span's basis is chosen so that the top tile bit is set in the tile
// coordinates of every mask that made the span grow (a linear functional l
// with l(mask) = 1: possible because those masks are independent).  Both
// amplitudes of such a pair then lie in different halves of the tile, at
// places the kernel knows at compile time; a mask inside the span with l = 0
// takes the kernel's slower general form.
#pragma once
#include <stdint.h>

namespace sq {

constexpr uint32_t kPauliTileBits = 11;
constexpr uint32_t kPauliLowBits = 3;
constexpr uint32_t kPauliGens = kPauliTileBits - kPauliLowBits;
constexpr uint32_t kPauliMaxTerms = 1024;
constexpr uint32_t kPauliMaxGroups = 256;
constexpr uint32_t kPauliMaxPasses = 40;

struct alignas(8) PauliTileGroup {
  uint16_t c;       // flip mask in tile coordinates (0: diagonal)
  uint16_t odd;     // odd number of Y: the pair's imaginary part
  uint16_t t0, t1;  // terms
};

struct PauliTilePass {
  uint64_t gen[kPauliGens];    // global index vector of tile bit low + i
  uint8_t pivot[kPauliGens];   // ascending bits the tile base has clear
  // Groups: single terms that flip the top tile bit with an even number of Y
  // [g0, ge) and an odd one [ge, go), all others [go, g1).
  uint16_t g0, ge, go, g1;
};

// Tile index j stands for global index base ^ (j's low bits) ^ gens of its
// other bits; base runs over the indices with the low and pivot bits clear.
template <uint32_t TERMS, uint32_t GROUPS, uint32_t PASSES>
struct PauliPlanOf {
  uint32_t n;
  uint32_t m, low;   // tile bits, low bits (both at most n)
  uint32_t npasses;
  uint32_t max_terms, max_groups;  // of any pass (shared-memory sizes)
  PauliTilePass pass[PASSES];
  PauliTileGroup group[GROUPS];
  uint64_t zy[TERMS];   // Z-or-Y mask (global index bits)
  double f[TERMS];      // weight and phase
  uint32_t zt[TERMS];   // Z-or-Y mask in tile coordinates
  // Terms of the diagonal group (at most one), relative to its first: those
  // with row parities z (tile bits 8..10 of zt) are diag[z] .. diag[z + 1].
  uint16_t diag[9];
};
using PauliTilePlan = PauliPlanOf<kPauliMaxTerms, kPauliMaxGroups, kPauliMaxPasses>;
// A plan is a kernel argument: one of 26 KiB makes a call on a small state
// longer than its two kernels (a norm of 2 qubits 53 us, with this one of
// 3.4 KiB, which sums of up to some sixty strings fit, 41 us).
using PauliSmallPlan = PauliPlanOf<96, 64, 12>;

// Copies a plan to the small form; false when it does not fit.
inline bool pauli_small_plan(const PauliTilePlan &P, PauliSmallPlan &S) {
  const uint32_t groups = P.npasses ? P.pass[P.npasses - 1].g1 : 0, terms = groups ? P.group[groups - 1].t1 : 0;
  if (P.npasses > 12 || groups > 64 || terms > 96) return false;
  S.n = P.n;
  S.m = P.m;
  S.low = P.low;
  S.npasses = P.npasses;
  S.max_terms = P.max_terms;
  S.max_groups = P.max_groups;
  for (uint32_t i = 0; i < P.npasses; ++i) S.pass[i] = P.pass[i];
  for (uint32_t i = 0; i < groups; ++i) S.group[i] = P.group[i];
  for (uint32_t i = 0; i < terms; ++i) {
    S.zy[i] = P.zy[i];
    S.f[i] = P.f[i];
    S.zt[i] = P.zt[i];
  }
  for (uint32_t i = 0; i < 9; ++i) S.diag[i] = P.diag[i];
  return true;
}

// Dynamic shared memory of the kernels for passes of at most these sizes:
// the tile as complex doubles, two 16-byte records per term, the groups.
constexpr uint32_t pauli_tile_smem(uint32_t terms, uint32_t groups) {
  return (16u << kPauliTileBits) + groups * 8u + terms * 32u;
}

// Blocks of one launch: `most`, or as many as there are tiles to work.
inline uint32_t pauli_tile_blocks(const PauliTilePlan &P, uint32_t most) {
  const uint64_t items = uint64_t(P.npasses) << (P.n - P.m);
  return items < 1 ? 1 : items < most ? uint32_t(items) : most;
}

// Plans the groups that start at term position `pos` of the term order idx
// (sorted by flip mask, then parity of the Y count): as many groups as the
// plan holds, at least one.  xm / zym / ny / w: per term the flip mask,
// Z-or-Y mask, Y count and weight.  `items`: work items (tile x pass) that
// fill the GPU; a state of few tiles gets more passes of fewer groups.
// Returns the position after the last planned term; `pos` itself when one
// group has more than kPauliMaxTerms terms.  Allocates nothing.
template <class Index>
uint32_t plan_pauli_tiles(PauliTilePlan &P, uint32_t n, const Index *idx, uint32_t nterms, uint32_t pos,
                          const uint64_t *xm, const uint64_t *zym, const int *ny, const double *w,
                          uint32_t items) {
  P.n = n;
  P.m = n < kPauliTileBits ? n : kPauliTileBits;
  P.low = n < kPauliLowBits ? n : kPauliLowBits;
  P.npasses = P.max_terms = P.max_groups = 0;
  // Groups [first, last) of the term order.
  uint16_t first[kPauliMaxGroups], last[kPauliMaxGroups];
  uint16_t open[kPauliMaxGroups];  // groups not yet in a pass
  uint64_t mask[kPauliMaxGroups];  // flip masks without the low bits
  uint32_t ngroups = 0;
  const uint32_t base = pos;
  const uint64_t lowmask = (uint64_t(1) << P.low) - 1;
  while (pos < nterms && ngroups < kPauliMaxGroups) {
    uint32_t end = pos;
    while (end < nterms && xm[idx[end]] == xm[idx[pos]] && (ny[idx[end]] & 1) == (ny[idx[pos]] & 1)) ++end;
    if (end - base > kPauliMaxTerms) break;
    first[ngroups] = uint16_t(pos - base);
    last[ngroups] = uint16_t(end - base);
    mask[ngroups] = xm[idx[pos]] & ~lowmask;
    open[ngroups] = uint16_t(ngroups);
    ++ngroups;
    pos = end;
  }
  const uint32_t gens = P.m - P.low;
  const uint64_t tiles = uint64_t(1) << (n - P.m);
  // Groups per pass: all that fit when the tiles alone fill the GPU.
  uint32_t cap = kPauliMaxGroups;
  if (tiles < items && ngroups) {
    uint64_t passes = (items + tiles - 1) / tiles;
    if (passes > 32) passes = 32;
    cap = uint32_t((ngroups + passes - 1) / passes);
  }
  uint32_t ng = 0, nt = 0;
  for (uint32_t left = ngroups; left;) {
    if (P.npasses == kPauliMaxPasses) return base;  // cannot happen: see kPauliMaxPasses
    PauliTilePass &S = P.pass[P.npasses++];
    uint64_t gen[kPauliGens] = {};
    uint32_t piv[kPauliGens] = {}, dim = 0;
    bool val[kPauliGens];  // l(gen[i])
    // gen stays reduced: bit piv[i] is set in gen[i] only, so the part of x
    // outside the span follows from x's own pivot bits (every open group is
    // tried in every pass: without branches 300 random strings on 17 qubits are
    // planned in 54 us, with them in 170 us).  Adds x with l(x) = v.
    auto add = [&](uint64_t x, bool v) -> bool {
      uint64_t rest = x;
      for (uint32_t i = 0; i < kPauliGens; ++i) rest ^= gen[i] & (0 - ((x >> piv[i]) & 1));
      if (!rest) return true;
      if (dim == gens) return false;
      for (uint32_t i = 0; i < dim; ++i) v ^= val[i] & bool((x >> piv[i]) & 1);
      const uint32_t p = uint32_t(__builtin_ctzll(rest));
      for (uint32_t i = 0; i < dim; ++i)
        if ((gen[i] >> p) & 1) {
          gen[i] ^= rest;
          val[i] ^= v;
        }
      gen[dim] = rest;
      val[dim] = v;
      piv[dim++] = p;
      return true;
    };
    uint16_t member[kPauliMaxGroups];
    uint32_t nm = 0, kept = 0;
    for (uint32_t k = 0; k < left; ++k) {
      const uint16_t g = open[k];
      if (nm < cap && add(mask[g], true)) member[nm++] = g;
      else open[kept++] = g;
    }
    left = kept;
    for (uint32_t b = P.low; dim < gens; ++b) add(uint64_t(1) << b, false);  // fill with the lowest free bits
    // The top tile bit: a generator with l = 1, which the others with l = 1
    // then lose; the rest in ascending pivot order.
    auto exchange = [&](uint32_t i, uint32_t j) {
      const uint32_t tp = piv[i];
      piv[i] = piv[j];
      piv[j] = tp;
      const uint64_t tg = gen[i];
      gen[i] = gen[j];
      gen[j] = tg;
      const bool tv = val[i];
      val[i] = val[j];
      val[j] = tv;
    };
    for (uint32_t i = 0; i < gens; ++i)
      if (val[i]) {
        exchange(i, gens - 1);
        for (uint32_t j = 0; j + 1 < gens; ++j)
          if (val[j]) gen[j] ^= gen[gens - 1];
        break;
      }
    for (uint32_t i = 0; i + 1 < gens; ++i)
      for (uint32_t j = i + 1; j + 1 < gens; ++j)
        if (piv[j] < piv[i]) exchange(i, j);
    // The tile base has the pivots clear: ascending for its enumeration.
    uint64_t pivots = 0;
    for (uint32_t i = 0; i < gens; ++i) pivots |= uint64_t(1) << piv[i];
    for (uint32_t i = 0, p = 0; i < kPauliGens; ++i) {
      S.gen[i] = i < gens ? gen[i] : 0;
      while (pivots >> p && !((pivots >> p) & 1)) ++p;
      S.pivot[i] = uint8_t(i < gens ? p++ : 0);
    }
    S.g0 = uint16_t(ng);
    const uint32_t t_begin = nt;
    auto coordinate_of = [&](uint64_t x) {
      // Every pivot but the top generator's occurs in one generator only;
      // what is left then tells the top one's.
      uint64_t rest = x;
      uint32_t c = 0;
      for (uint32_t i = 0; i < gens; ++i)
        if (((i + 1 < gens ? x : rest) >> piv[i]) & 1) {
          c |= 1u << (P.low + i);
          rest ^= gen[i];
        }
      return c | uint32_t(rest);
    };
    for (uint32_t k = 0; k < 3 * nm; ++k) {
      if (k == nm) S.ge = uint16_t(ng);
      if (k == 2 * nm) S.go = uint16_t(ng);
      const uint32_t g = member[k % nm], i0 = idx[base + first[g]];
      const uint64_t x = xm[i0];
      const uint32_t c = coordinate_of(x);
      const bool single = last[g] - first[g] == 1 && (c >> (kPauliTileBits - 1));
      if ((single ? uint32_t(ny[i0] & 1) : 2u) != k / nm) continue;
      PauliTileGroup &G = P.group[ng++];
      G.c = uint16_t(c);
      G.odd = uint16_t(ny[i0] & 1);
      G.t0 = uint16_t(nt);
      auto put = [&](uint32_t t, uint32_t zt) {
        P.zy[nt] = zym[t];
        // (-i)^ny folded into a real factor: even ny (-1)^(ny/2), odd ny
        // (-1)^((ny-1)/2) for the imaginary part.
        P.f[nt] = w[t] * (((ny[t] / 2) & 1) ? -1.0 : 1.0);
        P.zt[nt++] = zt;
      };
      auto coordinates = [&](uint32_t t) {
        uint32_t zt = uint32_t(zym[t] & lowmask);
        for (uint32_t i = 0; i < gens; ++i)
          if (__builtin_popcountll(gen[i] & zym[t]) & 1) zt |= 1u << (P.low + i);
        return zt;
      };
      // The diagonal group's terms by row parities.
      for (uint32_t z = 0; z < (x ? 1u : 8u); ++z) {
        if (!x) P.diag[z] = uint16_t(nt - G.t0);
        for (uint32_t e = first[g]; e < last[g]; ++e) {
          const uint32_t t = idx[base + e], zt = coordinates(t);
          if (x || zt >> 8 == z) put(t, zt);
        }
      }
      if (!x) P.diag[8] = uint16_t(nt - G.t0);
      G.t1 = uint16_t(nt);
    }
    S.g1 = uint16_t(ng);
    if (nt - t_begin > P.max_terms) P.max_terms = nt - t_begin;
    if (nm > P.max_groups) P.max_groups = nm;
  }
  return pos;
}

}  // namespace sq
