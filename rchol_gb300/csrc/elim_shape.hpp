// How the columns of one tree depth are eliminated (factor.cu): buffer width
// of a column and warps per tree node.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>
#include <vector>

namespace rchol {

inline int pow2_at_least(int x) {
  int p = 32;
  while (p < x) p <<= 1;
  return p;
}

// Records that a column of each depth may have: its initial entries and its
// slab, or what a column of that depth was seen to have where that is more
// (records come from the pool and from the column before, too).  widest holds
// the widest column that did not fit, per depth: one wide separator column
// must not widen the buffers of the leaves.
inline std::vector<int> depth_widths(const std::vector<int> &coldepth, const std::vector<int> &initdeg,
                                     const std::vector<uint32_t> &cap, const std::vector<int> &widest) {
  std::vector<int> width(widest.size(), 32);
  for (size_t c = 0; c < coldepth.size(); ++c)
    width[coldepth[c]] = std::max(width[coldepth[c]], initdeg[c] + (int)cap[c]);
  for (size_t d = 0; d < widest.size(); ++d) width[d] = std::max(width[d], widest[d]);
  return width;
}

struct ElimShape {
  bool four_warps;   // one thread block of four warps per node, else one warp per node
  int emax;          // records of a column's buffers
  size_t node_smem;  // their bytes per node; 0: in global memory
  int nodes_per_block;
};

// smem: most dynamic shared memory of a thread block (2 KB of it go to the
// four-warp kernel's static arrays).
inline ElimShape elim_shape(int width, int64_t nodes, int sms, size_t smem) {
  ElimShape S;
  S.emax = std::max(256, pow2_at_least(width));
  S.node_smem = (size_t)S.emax * 96;
  S.nodes_per_block = 1;
  // four warps per node unless the nodes alone fill the GPU several times
  S.four_warps = nodes <= 8 * (int64_t)sms && S.node_smem <= smem - 2048;
  if (S.four_warps) return S;
  S.emax = pow2_at_least(std::max(width, 128));
  S.node_smem = (size_t)S.emax * 40;
  if (S.node_smem > smem) S.node_smem = 0;
  else S.nodes_per_block = (int)std::min<size_t>(4, smem / S.node_smem);
  return S;
}

}  // namespace rchol
