// Triangular-solve schedule of a factor (built once per factor, see trsv.cu).
#pragma once

#include <array>
#include <memory>
#include <mutex>
#include <utility>
#include <vector>

#include "common.hpp"

namespace rchol {

// Block stream of one direction (forward with L = G, backward with U = G^T).
//
// The rows of every tree node are cut into pieces (pieces of one node are
// solved one after another) and every piece into blocks of 32 consecutive
// rows.  A piece's entries are
//   * external (columns outside the piece, already solved): a CSR over rows,
//     ext_rp / ext_ci / ext_v, summed by an all-SM kernel before the stage;
//   * in an earlier block of the piece: kept sparse in the block's record;
//   * inside the block: folded into the exact inverse of the block's 32x32
//     triangle.
// Record formats (trsv.cu documents each): FMT_WARP, one warp per piece with
// a window of solved values (depths with many nodes); FMT_PIPE, one thread
// block per piece whose warps split a block's entries by distance (the few
// long chains at the top of the tree); FMT_KTEAM, a thread block per piece
// for 32 right-hand sides at once.
enum { FMT_WARP = 0, FMT_PIPE = 1, FMT_KTEAM = 2 };

struct NodeDesc {
  int64_t begin;    // first row of the piece
  int32_t rows;
  int32_t nblocks;
  int64_t blk0;     // offsets of its blocks: blk_off[blk0 .. blk0 + nblocks]
  int32_t maxrec;   // largest block record (bytes)
  int32_t wide;     // column indices are u32 (piece larger than 65535 rows)
  int32_t maxchunk; // pipeline / k-team formats: most chunks of one block
  int32_t pad_;
};

struct StreamDir {
  std::vector<int> stage_ptr;        // pieces of stage s: [stage_ptr[s], stage_ptr[s+1])
  std::vector<int> stage_rows;       // largest piece of the stage (rows)
  std::vector<int> stage_maxrec;     // largest block record of the stage (bytes)
  std::vector<int64_t> stage_row_ptr;  // rows of the stages: srows[stage_row_ptr[s] ..]
  std::vector<int> stage_fmt;        // FMT_WARP, FMT_PIPE or FMT_KTEAM
  std::vector<int> stage_warps;      // pipeline / k-team: warps of the stage's teams
  std::vector<int> stage_chunks;     // pipeline / k-team: most chunks of one block in the stage
  std::vector<int> stage_window;     // warp format: rows of the window of solved values (a power of two)
  std::vector<int> stage_ext;        // 1: the stage has external entries (else it reads the rhs directly)
  std::vector<int> stage_ext_lanes;  // lanes per row of the external sums (1, 4, 8 or 32)
  std::vector<std::array<int, 9>> stage_smem;  // pipeline / k-team: launch shared memory by ring depth
  DevBuf<int32_t> srows;
  DevBuf<NodeDesc> nodes;
  DevBuf<int64_t> ext_rp;
  DevBuf<int32_t> ext_ci;
  DevBuf<double> ext_v64;
  DevBuf<float> ext_v32;
  DevBuf<unsigned char> blocks;      // block records (FP32 or FP64 values, per the factor)
  DevBuf<int64_t> blk_off;
  int64_t ext_nnz = 0, sparse_nnz = 0, nblocks = 0;
  int64_t steps = 0;                 // sequential block steps on the critical path
};

// ---- block plan (blocks.cu) -------------------------------------------------------
//
// One direction of the triangular solves as sequential steps of up to 512
// rows, each step one exact triangular inverse.  A piece (a tree node, cut at
// kBlkMaxRows rows) is solved by a cluster of C thread blocks.  Positions
// count a piece's rows in processing order (backward: from its last row);
// block s holds positions [s B, (s+1) B), and its rows go to the ranks of the
// cluster in groups of four (group q to rank q mod C).  The entries in
// earlier blocks are in record rec0 + s C + rank, the inverse's rows at
// inv0 + (blk0 + s) C + rank times the stage's stride.

constexpr int kBlkMaxRows = 16384;  // a piece's unknowns in shared memory: 64 KB in FP32, 128 KB in FP64
constexpr int kBlkMaxGroups = 64;   // 4-row groups of a thread block
constexpr int kBlkCols = 32;        // right-hand sides of one traversal
// From kBlkWideFrom right-hand sides on, the solves run on a second plan whose
// shapes count every piece kBlkWideCols times: the columns fill the GPU, so
// clusters are smaller and blocks shorter.  us per preconditioner, first plan /
// second, FP32: 80^3 2 columns 651 / 693, 5 columns 926 / 784, 32 columns
// 4020 / 2605; 30^3 2 columns 134 / 164, 5 columns 192 / 168; FP64 80^3 2
// columns 1483 / 1622, 5 columns 2348 / 2139.  With pieces counted 4 times
// 32 columns take 2900 us, 32 times 2448 (but 5 columns 998).
constexpr int kBlkWideFrom = 5, kBlkWideCols = 8;

struct BlkPiece {
  int64_t begin;   // first row
  int32_t rows;
  int32_t nblocks;
  int64_t rec0;    // first record
  int64_t blk0;    // blocks of the stage before it
};

struct BlkStage {
  int piece0 = 0, npieces = 0;
  int C = 1, B = 32;
  int gl = 32;            // lanes of a 4-row group (row threads; a quarter of them per row)
  int helpers = 0;        // threads that prepare the next block (clusters)
  int nv = 1;             // vectors of the inverse per thread and row
  int maxrows = 0;        // longest piece
  int64_t rows = 0;       // rows of all pieces
  int64_t erow0 = 0;      // their place in erow
  bool fused = false;     // its records hold external entries
  int late_lanes = 0;     // > 0: its late external entries are summed before it
  int slot = 0;           // bytes of a ring slot
  int ring = 4;
  size_t smem = 0;
  int64_t inv0 = 0;       // its inverses (values)
  int64_t stride = 0;     // values per (block, rank)
  int32_t goff[kBlkMaxGroups + 1] = {};  // first vector of a group
};

struct BlkExt {  // CSR over the matrix's rows
  DevBuf<int64_t> rp;
  DevBuf<int32_t> ci;
  DevBuf<double> v64;
  DevBuf<float> v32;
  int lanes = 8;  // per row
};

struct BlkDir {
  std::vector<BlkStage> stages;
  DevBuf<BlkPiece> pieces;
  DevBuf<int64_t> rec_off;
  DevBuf<unsigned char> recs;
  DevBuf<double> inv64;
  DevBuf<float> inv32;
  // external entries summed by kernels of their own: those in columns of the
  // first stage after it, for all later rows; the rest before a stage
  BlkExt early, late;
  DevBuf<int32_t> erow;  // the later stages' rows
  int64_t early_rows = 0;
};

// Vectors of trsv and precond with up to `cols` right-hand sides: what lies
// between the two solves of the preconditioner, and on the block plan with
// several of them right-hand sides and solutions column after column.
struct SolveWork {
  int cols = 0;
  DevBuf<double> a, b, y64;
  DevBuf<float> y32;
};

// Workspace and captured CUDA graph of one PCG iteration for a given matrix
// and number of right-hand sides (solve.cu).
struct PcgWork {
  uint64_t key_uid = 0;  // the matrix the captured iteration reads
  int64_t n = 0, nnz = 0;
  int k = 0;
  DevBuf<double> r, z, p, q, x, sc;
  DevBuf<double> hb, hx;  // staging of the host-buffer entry point
  DevBuf<int> ic;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev_in = nullptr, ev_out = nullptr;
  cudaGraphExec_t exec = nullptr;
  int64_t graph_kernels = 0;
  ~PcgWork() {
    if (exec) cudaGraphExecDestroy(exec);
    if (ev_in) cudaEventDestroy(ev_in);
    if (ev_out) cudaEventDestroy(ev_out);
    if (stream) cudaStreamDestroy(stream);
  }
};

// Workspace and captured graph of the batched PCG: independent systems that
// are the diagonal blocks (row ranges seg[s] .. seg[s+1]) of one matrix.
struct SegWork {
  uint64_t key_uid = 0;
  std::vector<int64_t> seg_host;
  int64_t n = 0;
  bool one_block = false;  // short systems: a thread block per system makes its sums and updates
  DevBuf<int64_t> seg;
  DevBuf<double> r, z, p, q, x, sc;
  DevBuf<double> hb, hx;
  DevBuf<int> ic;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev_in = nullptr, ev_out = nullptr;
  cudaGraphExec_t exec = nullptr;
  int64_t graph_kernels = 0;
  ~SegWork() {
    if (exec) cudaGraphExecDestroy(exec);
    if (ev_in) cudaEventDestroy(ev_in);
    if (ev_out) cudaEventDestroy(ev_out);
    if (stream) cudaStreamDestroy(stream);
  }
};

// Launch-time choices of the single-right-hand-side solves (trsv.cu).  Any
// setting solves the same system with the same arithmetic; the tuner
// (rchol_gpu_factor_tune) times alternatives on the factor itself.
struct SolveKnobs {
  int pipe_pf = 0;    // pipeline format: records prefetched into L2 ahead of use (0: none)
  int w2_pf = 0;      // warp format: the same
  int pipe_ring = 8;  // pipeline format: most ring slots (5..8)
  int w2_wpb = 8;     // warp format: most warps (pieces) per thread block (1..8)
};

struct SolvePlan {
  std::mutex lock;  // solves on one factor are serialised (they share workspaces)
  SolveKnobs knobs;
  double tuned_ms = 0.0;  // preconditioner time with the tuned knobs (0: not tuned)
  std::vector<std::unique_ptr<PcgWork>> pcg;
  std::vector<std::unique_ptr<SegWork>> seg;
  unsigned int *status = nullptr;  // status word of the solve kernels
  bool blocked = false;    // trsv and precond run on bfwd / bbwd (else, and in PCG, on the record streams)
  bool blocked1 = false;   // the same for one right-hand side
  BlkDir bfwd, bbwd;
  BlkDir bkfwd, bkbwd;     // shapes for several right-hand sides (built on first use)
  bool kblocks = false, kwide = false;  // that was tried; it is there
  StreamDir sfwd, sbwd;
  StreamDir kfwd, kbwd;    // pieces for up to 32 right-hand sides (built on first use)
  bool kbuilt = false;
  int64_t dag_fwd = -1, dag_bwd = -1;  // dependency-chain lengths, computed on request
  DevBuf<double> ytmp;     // intermediate of PCG's preconditioner (FP64 path)
  DevBuf<float> ytmp32;    // the same (FP32 path)
  DevBuf<double> acc64;    // external partial sums of split stages
  DevBuf<float> acc32;
  DevBuf<double> acck64;   // the same for up to 32 right-hand sides (n x 32)
  DevBuf<float> acck32;
  std::vector<SolveWork> work;  // of trsv and precond; the last is in use
};

// Block plan of both directions.  Left out: G's rows are too dense for it, its
// entries have mixed signs, or it would be too large.
enum class BlkBuilt { kReady, kLeftOut, kNoMemory };
BlkBuilt build_blocks(const rchol_factor_s &F, SolvePlan &P, cudaStream_t s);
// Whether one right-hand side takes that plan.
bool blocks_for_one(const rchol_factor_s &F, const SolvePlan &P);
// The plan that k right-hand sides take, where it is another one.
void build_blocks_k(const rchol_factor_s &F, SolvePlan &P, int k, cudaStream_t s);
// Solve with G (upper = false) or G^T for k <= kBlkCols right-hand sides, one
// column after another; acc: n k values of G's precision.
void block_trsv(const rchol_factor_s &F, const SolvePlan &P, bool upper, const double *in64, const float *in32,
                double *out64, float *out32, void *acc, int k, cudaStream_t s);
// Device address of the status word of the solve kernels (current device).
unsigned int *solve_status_word();
void build_streams(const rchol_factor_s &F, SolvePlan &P, cudaStream_t s);
void build_streams_k(const rchol_factor_s &F, SolvePlan &P, cudaStream_t s);
// Solve with G (upper = false) or G^T for k right-hand sides, n x k
// row-major, in groups of up to 32 columns.
void stream_trsv_k(const rchol_factor_s &F, const SolvePlan &P, bool upper, const double *in64,
                   const float *in32, double *out64, float *out32, int k, cudaStream_t s);
// acc: n values of G's precision.
void stream_trsv(const rchol_factor_s &F, const SolvePlan &P, bool upper, const double *in64,
                 const float *in32, double *out64, float *out32, void *acc, cudaStream_t s);
// Times the preconditioner under alternative SolveKnobs and keeps the
// fastest; returns {ms with the knobs on entry, ms with the chosen ones}.
std::pair<double, double> tune_solves(const rchol_factor_s &F, SolvePlan &P, cudaStream_t s);

}  // namespace rchol
