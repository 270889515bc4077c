// Host partition of a body's rows over the blocks of one thread-block
// cluster (the device side is tl_cluster.cuh).  Plain C++, no CUDA types, so
// that the CPU tests compile it with g++.
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

#include "tl_sell_build.h"

namespace tl {

constexpr uint32_t CLUSTER_NO_PUSH = 0xffffffffu;
constexpr uint32_t CLUSTER_INLINE = 4;  // destinations of a row kept beside it

// First slice of block `rank` of a body of `slices` slices over `ctas` blocks.
#ifdef __CUDACC__
__host__ __device__
#endif
inline uint32_t clusterSlice(uint32_t slices, uint32_t ctas, uint32_t rank) {
  return uint32_t(uint64_t(slices) * rank / ctas);
}

struct ClusterHost {
  uint32_t maxEntries = 0;           // vector entries (own rows, then foreign ones) of one block
  uint32_t maxPositions = 0;         // block positions of one block
  std::vector<uint32_t> foreign;     // [ctas] foreign entries of each block's vector
  std::vector<uint16_t> local;       // [positions] entry of each column slot in its block's vector
  std::vector<uint32_t> push;        // [CLUSTER_INLINE * rows] (block << 16) | entry, or CLUSTER_NO_PUSH
  std::vector<uint32_t> overStart;   // [rows + 1] destinations beyond the inline ones
  std::vector<uint32_t> over;
};

// Block q owns the slices [clusterSlice(q), clusterSlice(q + 1)); its vector
// holds its own rows, then the foreign columns its rows read, ascending.  A
// row lists the (block, entry) places its value is sent to.  False when a
// block's vector has more entries than 16 bits address.
inline bool buildClusterHost(const SellHost& h, uint32_t ctas, ClusterHost& out) {
  const uint32_t rows = h.slices * SELL_ROWS;  // padding rows, past h.rows, hold no blocks
  out.local.assign(h.positions, 0);
  std::vector<uint32_t> mark(rows, ctas), entryOf(rows, 0), foreign, count(size_t(rows) + 1, 0);
  std::vector<std::pair<uint32_t, uint32_t>> sends;  // (row, code), in order of block then entry
  for (uint32_t q = 0; q < ctas; ++q) {
    const uint32_t sA = clusterSlice(h.slices, ctas, q), sB = clusterSlice(h.slices, ctas, q + 1);
    const uint32_t lo = sA * SELL_ROWS, hi = sB * SELL_ROWS;
    const uint32_t p0 = h.sliceStart[sA], p1 = h.sliceStart[sB];
    const auto column = [&](uint32_t p) {
      const uint32_t r = h.groupSlice[p / SELL_ROWS] * SELL_ROWS + p % SELL_ROWS;
      return r < h.rows ? h.col[p] : r;
    };
    foreign.clear();
    for (uint32_t p = p0; p < p1; ++p) {
      const uint32_t c = column(p);
      if ((c < lo || c >= hi) && mark[c] != q) {
        mark[c] = q;
        foreign.push_back(c);
      }
    }
    std::sort(foreign.begin(), foreign.end());
    const uint32_t own = hi - lo, entries = own + uint32_t(foreign.size());
    if (entries > 0xffffu) return false;
    out.maxPositions = std::max(out.maxPositions, p1 - p0);
    out.maxEntries = std::max(out.maxEntries, entries);
    out.foreign.push_back(uint32_t(foreign.size()));
    for (uint32_t f = 0; f < foreign.size(); ++f) {
      entryOf[foreign[f]] = own + f;
      sends.emplace_back(foreign[f], (q << 16) | (own + f));
      ++count[foreign[f] + 1];
    }
    for (uint32_t p = p0; p < p1; ++p) {
      const uint32_t c = column(p);
      out.local[p] = uint16_t(c >= lo && c < hi ? c - lo : entryOf[c]);
    }
  }
  out.push.assign(size_t(CLUSTER_INLINE) * rows, CLUSTER_NO_PUSH);
  out.overStart.assign(size_t(rows) + 1, 0);
  for (uint32_t r = 0; r < rows; ++r)
    out.overStart[r + 1] = out.overStart[r] + (count[r + 1] > CLUSTER_INLINE ? count[r + 1] - CLUSTER_INLINE : 0u);
  out.over.assign(out.overStart[rows], 0);
  std::fill(count.begin(), count.end(), 0u);
  for (const auto& s : sends) {
    const uint32_t k = count[s.first]++;
    if (k < CLUSTER_INLINE) out.push[size_t(CLUSTER_INLINE) * s.first + k] = s.second;
    else out.over[out.overStart[s.first] + k - CLUSTER_INLINE] = s.second;
  }
  return true;
}

}  // namespace tl
