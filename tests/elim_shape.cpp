// CPU check of the elimination's shapes per tree depth (csrc/elim_shape.hpp):
//   elim_shape <smem> <sms> <depth> <initdeg> <cap> <widest> <nodes> ...
// one group of five per depth's only column; prints "four_warps emax
// node_smem nodes_per_block" per depth.
#include <cstdio>
#include <cstdlib>

#include "elim_shape.hpp"

int main(int argc, char **argv) {
  const size_t smem = std::strtoull(argv[1], nullptr, 10);
  const int sms = std::atoi(argv[2]);
  std::vector<int> depth, deg, widest(1, 0);
  std::vector<uint32_t> cap;
  std::vector<int64_t> nodes;
  for (int i = 3; i + 4 < argc; i += 5) {
    depth.push_back(std::atoi(argv[i]));
    deg.push_back(std::atoi(argv[i + 1]));
    cap.push_back((uint32_t)std::atoi(argv[i + 2]));
    widest.push_back(std::atoi(argv[i + 3]));
    nodes.push_back(std::atoll(argv[i + 4]));
  }
  const std::vector<int> width = rchol::depth_widths(depth, deg, cap, widest);
  for (size_t k = 0; k < depth.size(); ++k) {
    const rchol::ElimShape S = rchol::elim_shape(width[depth[k]], nodes[k], sms, smem);
    std::printf("%d %d %zu %d\n", (int)S.four_warps, S.emax, S.node_smem, S.nodes_per_block);
  }
  return 0;
}
