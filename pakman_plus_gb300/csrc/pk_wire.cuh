// The ranking behind a macro-node's initial wiring, shared by the wiring kernel and the
// initial state of the compaction.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace pk {

// Ranks of a side's five slots (four base codes and the terminal entry) among the present
// ones; their visits land in vis[rank] and the list positions of the ranked entries come
// back four bits each.
__device__ __forceinline__ uint32_t wire_rank(const uint32_t raw[4], const int32_t v[5], int32_t* vis) {
  uint32_t pos = 0, ids = 0;  // pos: present slots so far
#pragma unroll
  for (int e = 0; e < 5; e++) {
    if (e < 4 && !raw[e]) continue;
    const int32_t ce = e < 4 ? (int32_t)raw[e] : 1;
    uint32_t rank = 0;
#pragma unroll
    for (int o = 0; o < 5; o++) {
      if (o == e || (o < 4 && !raw[o])) continue;
      const int32_t co = o < 4 ? (int32_t)raw[o] : 1;
      const bool same = v[o] == v[e] && co == ce;
      rank += (v[o] > v[e] || (v[o] == v[e] && co > ce) || (same && o < e)) ? 1u : 0u;
    }
    vis[rank] = v[e];
    ids |= pos << (4 * rank);
    pos++;
  }
  return ids;
}

}  // namespace pk
