// CPU check of the shapes of the block solves (csrc/blocks.cu, included whole;
// nothing runs on a device):
//   block_shape <fit of clusters of 2> <of 4> <of 8> <of 16>
// prints for a range of stages "fp32 npieces maxrows cols halvings C B nown gl
// nv threads max_threads stride_vectors", with the block rows halved 0 to 4
// times as the plan does when a stage does not fit.

#include "../rchol_gb300/csrc/blocks.cu"

#include <cstdio>
#include <cstdlib>

namespace rchol {
void note_launch(int64_t) {}
void set_last_error(const std::string &) {}
void exclusive_scan_i64(int64_t *, int64_t, cudaStream_t) {}
}  // namespace rchol

using namespace rchol;

template <typename VT>
static int bound(int nv, int C) {
  if (C > 1)
    return nv == 1 ? BlkBounds<VT, 1, true>::threads : nv == 2 ? BlkBounds<VT, 2, true>::threads : BlkBounds<VT, 4, true>::threads;
  return nv == 1 ? BlkBounds<VT, 1, false>::threads : nv == 2 ? BlkBounds<VT, 2, false>::threads : BlkBounds<VT, 4, false>::threads;
}

int main(int argc, char **argv) {
  ClusterFit fit = {152, 0, 0, 0, 0};
  for (int i = 1; i < 5 && i < argc; ++i) fit[i] = std::atoi(argv[i]);
  const int pieces[] = {1, 2, 7, 8, 9, 18, 19, 36, 37, 76, 77, 152, 100000};
  const int rows[] = {1, 2, 31, 32, 33, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 1025, 16384};
  for (int fp32 = 0; fp32 < 2; ++fp32)
    for (int cols : {1, kBlkWideCols})
      for (int P : pieces)
        for (int R : rows) {
          BlkStage S;
          S.npieces = P;
          S.maxrows = R;
          choose_shape(S, fp32 != 0, cols, fit);
          for (int halved = 0; S.B >= 32; ++halved, S.B /= 2) {
            set_geometry(S, fp32 ? 4 : 8);
            const int nown = S.B / S.C, threads = nown / 4 * S.gl + S.helpers;
            std::printf("%d %d %d %d %d %d %d %d %d %d %d %d %lld\n", fp32, P, R, cols, halved, S.C, S.B, nown, S.gl, S.nv,
                        threads, fp32 ? bound<float>(S.nv, S.C) : bound<double>(S.nv, S.C), (long long)S.goff[nown / 4]);
          }
        }
  return 0;
}
