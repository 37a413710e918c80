// Triangular solves with G and G^T in large blocks: rchol_gpu_trsv_d and
// rchol_gpu_precond_d (PCG applies the record streams of trsv.cu).
//
// Replaces the two MKL trsv calls of c++/util/pcg.cpp:141-159.
//
// Nested dissection leaves chains of thousands of rows (a separator of 16,384
// rows has about 9,000 levels), and a solve takes the chain's steps one after
// another.  Here a step retires a block of B rows (32 to 512):
//     t = rhs - (entries in earlier blocks) x,    x = T^-1 t
// with the exact inverse of the block's B x B triangle, made in FP64 when the
// plan is built.  T is a triangular M-matrix (nonpositive off-diagonal
// entries), so its inverse has no cancellation and the product is as accurate
// as substitution.  The rows of a block are dealt to the thread blocks of a
// cluster, each of which keeps all of the piece's unknowns in its own shared
// memory; t and x travel as remote stores that complete on the receivers'
// mbarriers, so a step has two one-way trips and no cluster barrier.
//
// Several right-hand sides lie column after column, and a cluster solves one
// column of a piece: the chain's length, not the arithmetic, is what a solve
// costs, and columns hide it from one another.  Preconditioner of 80^3 with
// 128 subdomains, record streams -> now: FP32 2 columns 8.9 -> 0.65 ms, 32
// columns 8.3 -> 2.5; FP64 49 -> 1.5 and 49 -> 8.8 ms.
//
// The plan is built on the GPU from the CSR of G (or G^T): count entries by
// distance, lay out the records, copy the entries, invert the triangles.

#include <algorithm>
#include <array>
#include <cstring>
#include <mutex>

#include "bulk.hpp"
#include "common.hpp"
#include "host.hpp"
#include "plan.hpp"

namespace rchol {

void exclusive_scan_i64(int64_t *d_data, int64_t n, cudaStream_t s);

namespace {

constexpr size_t kBlkSmem = 224 * 1024;  // dynamic shared memory of a launch
constexpr int kBlkRingMax = 8;
constexpr size_t kBlkBars = 8 * (kBlkRingMax + 2);  // mbarriers: the ring's, t's and x's

__host__ __device__ inline size_t up16(size_t x) { return (x + 15) & ~size_t(15); }

// Record of one step and rank (16-byte sections), nown = B / C rows:
//   u32 hdr[8]            byte offsets of ccol, ocol, ecol, cval, oval, eval; external entries; 0
//   u16 off[nown+1][4]    row offsets into the chain, old and external lists, in quads (external: pairs)
//   u16 ccol[]            chain: positions in the block before (single thread block: in all earlier blocks)
//   u16 ocol[]            old: positions in the blocks before that
//   u32 ecol[]            external: rows of the matrix
//   VT  cval[], oval[], eval[]
// A row's entries fill whole quads (pairs); free places have the position of
// a zero (no column) and the value 0.
constexpr uint32_t kBlkOff = 32;  // byte offset of off
constexpr uint32_t kNoCol = 0xffffffffu;
struct BlkLayout {
  uint32_t o_ccol, o_ocol, o_ecol, o_cval, o_oval, o_eval, len;
};
// nc, no: quads; ne: pairs
__host__ __device__ inline BlkLayout blk_layout(uint32_t nown, uint32_t nc, uint32_t no, uint32_t ne, uint32_t vsz) {
  BlkLayout L;
  L.o_ccol = kBlkOff + (uint32_t)up16(8 * (nown + 1));
  L.o_ocol = L.o_ccol + (uint32_t)up16(8 * nc);
  L.o_ecol = L.o_ocol + (uint32_t)up16(8 * no);
  L.o_cval = L.o_ecol + (uint32_t)up16(8 * ne);
  L.o_oval = L.o_cval + (uint32_t)up16(4 * vsz * nc);
  L.o_eval = L.o_oval + (uint32_t)up16(4 * vsz * no);
  L.len = L.o_eval + (uint32_t)up16(2 * vsz * ne);
  return L;
}

// Position in its block of own row j of a rank, and back.
__host__ __device__ inline int own_pos(int j, int rank, int C) { return ((j >> 2) * C + rank) * 4 + (j & 3); }

// ---- building the plan --------------------------------------------------------------------

struct BlkRec {
  int64_t row0;    // the block's rows [row0, row0 + nr)
  int64_t pb, pe;  // the piece's
  int32_t nr;
  int32_t B;
  int32_t rank, C;
  int32_t apart;  // external entries are not in the record
  int32_t pad;    // position of a zero
};

// first position in [a, b) of the sorted columns ci with ci >= c
__device__ __forceinline__ int64_t lower_pos(const int32_t *ci, int64_t a, int64_t b, int64_t c) {
  while (a < b) {
    const int64_t m = (a + b) >> 1;
    if (ci[m] < c) a = m + 1;
    else b = m;
  }
  return a;
}

// Per row the positions (relative to its start) where the classes of its
// sorted columns change.  Lower: external [0,x), old [x,y), chain [y,z),
// inside [z,len-1), diagonal.  Upper: diagonal, inside [1,x), chain [x,y),
// old [y,z), external [z,len).  Early entries (columns of the first stage,
// early[col] = 1; lower only) are counted per row in nearly.  One warp per
// record.
__global__ void __launch_bounds__(256) blk_count_kernel(const BlkRec *recs, int64_t nrec, const int64_t *rp,
                                                        const int32_t *ci, bool upper, const unsigned char *early, int4 *bnd,
                                                        int64_t *nearly, int4 *cnt) {
  const int64_t w = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= nrec) return;
  const BlkRec d = recs[w];
  int nc = 0, no = 0, ne = 0;  // quads, quads, pairs
  for (int j = lane; j < d.B / d.C; j += 32) {
    const int p = own_pos(j, d.rank, d.C);
    if (p >= d.nr) continue;
    const int64_t row = upper ? d.row0 + d.nr - 1 - p : d.row0 + p, q0 = rp[row], q1 = rp[row + 1];
    int x, y, z, c_n, o_n, e_n;
    if (!upper) {
      const int64_t e = lower_pos(ci, q0, q1, d.pb), o = lower_pos(ci, e, q1, d.row0 - d.B),
                    c = lower_pos(ci, o, q1, d.row0);
      x = (int)(e - q0), y = (int)(o - q0), z = (int)(c - q0);
      c_n = z - y, o_n = y - x, e_n = x;
    } else {
      const int64_t hi = d.row0 + d.nr, a = lower_pos(ci, q0, q1, hi),
                    c = lower_pos(ci, a, q1, min(hi + d.B, d.pe)), o = lower_pos(ci, c, q1, d.pe);
      x = (int)(a - q0), y = (int)(c - q0), z = (int)(o - q0);
      c_n = y - x, o_n = z - y, e_n = (int)(q1 - o);
    }
    bnd[row] = make_int4(x, y, z, (int)(q1 - q0));
    if (early) {
      int k = 0;
      for (int64_t q = q0; q < q0 + x; ++q) k += early[ci[q]];
      nearly[row] = k;
      e_n -= k;
    }
    if (d.C == 1) c_n += o_n, o_n = 0;
    nc += (c_n + 3) / 4, no += (o_n + 3) / 4, ne += (e_n + 1) / 2;
  }
  for (int o = 16; o; o >>= 1) {
    nc += __shfl_xor_sync(0xffffffffu, nc, o);
    no += __shfl_xor_sync(0xffffffffu, no, o);
    ne += __shfl_xor_sync(0xffffffffu, ne, o);
  }
  if (lane == 0) cnt[w] = make_int4(0, nc, no, ne);
}

// Entries of G^T that are not <= 0 (out[0]) and positive diagonal entries (out[1]).
__global__ void __launch_bounds__(256) blk_sign_kernel(int64_t n, int64_t nnz, const int64_t *rp, const double *v,
                                                       unsigned long long *out) {
  const int64_t t0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x, T = (int64_t)gridDim.x * blockDim.x;
  unsigned long long all = 0, diag = 0;
  for (int64_t q = t0; q < nnz; q += T) all += !(v[q] <= 0.0);
  for (int64_t i = t0; i < n; i += T) diag += v[rp[i]] > 0.0;
  for (int o = 16; o; o >>= 1) {
    all += __shfl_xor_sync(0xffffffffu, all, o);
    diag += __shfl_xor_sync(0xffffffffu, diag, o);
  }
  if ((threadIdx.x & 31) == 0) {
    if (all) atomicAdd(out, all);
    if (diag) atomicAdd(out + 1, diag);
  }
}

__global__ void blk_mark_kernel(const BlkPiece *pieces, int npieces, unsigned char *early) {
  for (int k = blockIdx.x; k < npieces; k += gridDim.x)
    for (int i = threadIdx.x; i < pieces[k].rows; i += blockDim.x) early[pieces[k].begin + i] = 1;
}

// Headers, row offsets and entries of the records; one thread block (4 warps)
// per record.
template <typename VT>
__global__ void __launch_bounds__(128) blk_fill_kernel(const BlkRec *recs, const int64_t *rec_off, const int4 *cnt,
                                                       const int64_t *rp, const int32_t *ci, const double *v,
                                                       const int4 *bnd, bool upper, const unsigned char *early,
                                                       const int64_t *nearly, unsigned char *out) {
  __shared__ uint32_t off[3][513];
  const BlkRec d = recs[blockIdx.x];
  const int4 k = cnt[blockIdx.x];
  const int nown = d.B / d.C, ne = d.apart ? 0 : k.w;
  unsigned char *p = out + rec_off[blockIdx.x];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  auto row_of = [&](int j) {  // own row j, or -1 past the block's rows
    const int q = own_pos(j, d.rank, d.C);
    return q >= d.nr ? (int64_t)-1 : upper ? d.row0 + d.nr - 1 - q : d.row0 + q;
  };
  if (warp < 3) {  // warps 0..2: running sums of the chain, old and external entries
    uint32_t carry = 0;
    if (lane == 0) off[warp][0] = 0;
    for (int j0 = 0; j0 < nown; j0 += 32) {
      const int j = j0 + lane;
      uint32_t c = 0;
      const int64_t row = j < nown ? row_of(j) : -1;
      if (row >= 0) {
        const int4 b = bnd[row];
        const int c_n = upper ? b.y - b.x : b.z - b.y, o_n = upper ? b.z - b.y : b.y - b.x;
        if (warp == 0) c = (c_n + (d.C == 1 ? o_n : 0) + 3) / 4;
        else if (warp == 1) c = d.C == 1 ? 0 : (o_n + 3) / 4;
        else c = d.apart ? 0 : ((upper ? b.w - b.z : b.x - (early ? (int)nearly[row] : 0)) + 1) / 2;
      }
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t t = __shfl_up_sync(0xffffffffu, c, o);
        if (lane >= o) c += t;
      }
      if (j < nown) off[warp][j + 1] = carry + c;
      carry += __shfl_sync(0xffffffffu, c, 31);
    }
  }
  __syncthreads();
  const BlkLayout L = blk_layout(nown, k.y, k.z, ne, sizeof(VT));
  if (tid == 0) {
    const uint32_t h[8] = {L.o_ccol, L.o_ocol, L.o_ecol, L.o_cval, L.o_oval, L.o_eval, (uint32_t)ne, 0};
    for (int i = 0; i < 8; ++i) reinterpret_cast<uint32_t *>(p)[i] = h[i];
  }
  uint16_t *po = reinterpret_cast<uint16_t *>(p + kBlkOff);
  for (int t = tid; t < 4 * (nown + 1); t += 128) po[t] = (t & 3) < 3 ? (uint16_t)off[t & 3][t >> 2] : 0;
  uint16_t *cc = reinterpret_cast<uint16_t *>(p + L.o_ccol), *oc = reinterpret_cast<uint16_t *>(p + L.o_ocol);
  uint32_t *ec = reinterpret_cast<uint32_t *>(p + L.o_ecol);
  VT *cv = reinterpret_cast<VT *>(p + L.o_cval), *ov = reinterpret_cast<VT *>(p + L.o_oval),
     *ev = reinterpret_cast<VT *>(p + L.o_eval);
  for (int i = tid; i < 4 * k.y; i += 128) cc[i] = (uint16_t)d.pad, cv[i] = VT(0);
  for (int i = tid; i < 4 * k.z; i += 128) oc[i] = (uint16_t)d.pad, ov[i] = VT(0);
  for (int i = tid; i < 2 * ne; i += 128) ec[i] = kNoCol, ev[i] = VT(0);
  __syncthreads();
  auto pos_of = [&](int32_t c) { return (uint16_t)(upper ? d.pe - 1 - c : c - d.pb); };
  for (int j = warp; j < nown; j += 4) {
    const int64_t row = row_of(j);
    if (row < 0) continue;
    const int64_t q0 = rp[row];
    const int4 b = bnd[row];
    const int c0 = upper ? b.x : b.y, c1 = upper ? b.y : b.z, o0 = upper ? b.y : b.x, o1 = upper ? b.z : b.y;
    const uint32_t oat = d.C == 1 ? 4 * off[0][j] : 4 * off[1][j], cat = 4 * off[0][j] + (d.C == 1 ? o1 - o0 : 0);
    for (int e = o0 + lane; e < o1; e += 32) {
      (d.C == 1 ? cc : oc)[oat + e - o0] = pos_of(ci[q0 + e]);
      (d.C == 1 ? cv : ov)[oat + e - o0] = (VT)v[q0 + e];
    }
    for (int e = c0 + lane; e < c1; e += 32) {
      cc[cat + e - c0] = pos_of(ci[q0 + e]);
      cv[cat + e - c0] = (VT)v[q0 + e];
    }
    if (d.apart) continue;
    const int e0 = upper ? b.z : 0, e1 = upper ? b.w : b.x;
    uint32_t k2 = 2 * off[2][j];
    for (int eb = e0; eb < e1; eb += 32) {
      const int e = eb + lane;
      const bool on = e < e1 && !(early && early[ci[q0 + e]]);
      const unsigned bal = __ballot_sync(0xffffffffu, on);
      if (on) {
        const uint32_t at = k2 + __popc(bal & ((1u << lane) - 1u));
        ec[at] = (uint32_t)ci[q0 + e];
        ev[at] = (VT)v[q0 + e];
      }
      k2 += __popc(bal);
    }
  }
}

// Entries of the late CSR per row: a row of an `apart` stage keeps its
// external entries that are not early.
__global__ void blk_late_count_kernel(int64_t nrows, const int32_t *rows, const int4 *bnd, const int64_t *nearly,
                                      int64_t *nlate) {
  const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (t < nrows) nlate[rows[t]] = bnd[rows[t]].x - nearly[rows[t]];
}

// The external entries with early[col] == want as a CSR.
__global__ void blk_ext_fill_kernel(int64_t nrows, const int32_t *rows, const int64_t *rp, const int32_t *ci,
                                    const double *v, const int4 *bnd, const unsigned char *early, int want,
                                    const int64_t *erp, int32_t *eci, float *ev32, double *ev64) {
  const int64_t t = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (t >= nrows) return;
  const int64_t i = rows[t];
  int64_t w = erp[i];
  if (erp[i + 1] == w) return;
  const int64_t q0 = rp[i];
  for (int eb = 0; eb < bnd[i].x; eb += 32) {
    const int e = eb + lane;
    const bool on = e < bnd[i].x && early[ci[q0 + e]] == want;
    const unsigned bal = __ballot_sync(0xffffffffu, on);
    if (on) {
      const int64_t k = w + __popc(bal & ((1u << lane) - 1u));
      eci[k] = ci[q0 + e];
      if (ev32) ev32[k] = (float)v[q0 + e];
      else ev64[k] = v[q0 + e];
    }
    w += __popc(bal);
  }
}

// Where the inverse's entry (position p, position c <= p) of a block sits in
// the values of p's rank: vector goff[g] + (v * 4 + r) * gl + l of group g's
// row r holds the positions of 16-byte chunk v * gl + l.
struct BlkInv {
  int C, gl;
  int64_t stride;
  int32_t goff[kBlkMaxGroups + 1];
};

// 32 columns of one block's inverse by one warp (lane = column), row after
// row in FP64 with the panel in shared memory.  recs points at the stage's
// first record, ranks of a block together.  Row facts (start, class bounds,
// reciprocal diagonal) are loaded 32 rows at a time.
template <typename VT>
__global__ void __launch_bounds__(32) blk_invert_kernel(const BlkRec *recs, BlkInv g, int panels, const int64_t *rp,
                                                        const int32_t *ci, const double *v, const int4 *bnd,
                                                        bool upper, VT *inv) {
  extern __shared__ double X[];  // [position - first][32]
  const int lane = threadIdx.x;
  const int64_t blk = blockIdx.x / panels;
  const int first = (int)(blockIdx.x % panels) * 32;
  const BlkRec d = recs[blk * g.C];
  const int nr = d.nr;
  if (first >= nr) return;
  constexpr int per = 16 / (int)sizeof(VT);
  auto row_of = [&](int p) { return upper ? d.row0 + nr - 1 - p : d.row0 + p; };
  int64_t rs = 0;
  int4 rb = make_int4(0, 0, 0, 0);
  double rd = 0.0;
  const int c = first + lane, q = c / per, cv = q / g.gl, cl = q % g.gl;
  for (int p = first; p < nr; ++p) {
    const int t = p - first;
    if ((t & 31) == 0 && p + lane < nr) {  // facts of positions p..p+31, one per lane
      const int64_t row = row_of(p + lane);
      rs = rp[row];
      rb = bnd[row];
      rd = 1.0 / v[upper ? rs : rs + rb.w - 1];
    }
    const int64_t q0 = __shfl_sync(0xffffffffu, rs, t & 31);
    const int z = __shfl_sync(0xffffffffu, upper ? rb.x : rb.z, t & 31), len = __shfl_sync(0xffffffffu, rb.w, t & 31);
    const double rdi = __shfl_sync(0xffffffffu, rd, t & 31);
    const int e0 = upper ? 1 : z, e1 = upper ? z : len - 1;  // entries inside the triangle
    double a[4] = {p == c ? 1.0 : 0.0, 0.0, 0.0, 0.0};
    for (int eb = e0; eb < e1; eb += 32) {
      const int e = eb + lane;
      const int32_t ncol = e < e1 ? (upper ? (int32_t)(d.row0 + nr - 1 - ci[q0 + e]) : (int32_t)(ci[q0 + e] - d.row0)) : -1;
      const double nval = e < e1 ? v[q0 + e] : 0.0;
      const int m = min(32, e1 - eb);
      for (int u = 0; u < m; u += 4) {
#pragma unroll
        for (int w = 0; w < 4; ++w) {
          const int col = __shfl_sync(0xffffffffu, ncol, (u + w) & 31);
          const double val = __shfl_sync(0xffffffffu, nval, (u + w) & 31);
          if (u + w < m && col >= first) a[w] = fma(-val, X[(col - first) * 32 + lane], a[w]);
        }
      }
    }
    const double x = ((a[0] + a[1]) + (a[2] + a[3])) * rdi;
    X[t * 32 + lane] = x;
    if (c <= p) {
      const int rank = (p >> 2) % g.C, grp = (p >> 2) / g.C;
      inv[(blk * g.C + rank) * g.stride + (int64_t)(g.goff[grp] + (cv * 4 + (p & 3)) * g.gl + cl) * per + c % per] = (VT)x;
    }
  }
}

// ---- solving ----------------------------------------------------------------------------------

// A solve is a chain of short kernels (two per tree depth and direction), so
// each may start while the one before it still runs (programmatic dependent
// launch): it sets up its barriers and loads what the plan holds, then waits
// here until the kernels before it are complete and their writes visible.  It
// must not touch vectors before that, and reads them with plain loads: the
// compiler may move read-only ones above the wait.  The next kernel's start is
// allowed as soon as all of this one's thread blocks run, so none of them ever
// waits for room that a waiting kernel holds.
__device__ __forceinline__ void allow_next() { asm volatile("griddepcontrol.launch_dependents;\n" ::: "memory"); }
__device__ __forceinline__ void wait_previous() { asm volatile("griddepcontrol.wait;\n" ::: "memory"); }

// acc_i = in_i - (entries of row i in a CSR of external ones) out, LANES
// lanes per row, four entries in flight per lane; in may be acc.  One
// right-hand side (KC = 1), or columns (n apart) KC blockIdx.y and on of k, so
// that a row's entries are read once for KC of them.
template <typename VT, typename InT, typename OutT, int LANES, int KC>
__global__ void __launch_bounds__(256) blk_ext_kernel(const int32_t *__restrict__ rows, int64_t nrows,
                                                        const int64_t *__restrict__ rp, const int32_t *__restrict__ ci,
                                                        const VT *__restrict__ v, const InT *in, const OutT *out,
                                                        VT *acc, int k, int64_t n) {
  allow_next();
  const int64_t t = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) / LANES;
  const int sub = threadIdx.x % LANES, col0 = KC == 1 ? 0 : blockIdx.y * KC;
  if (t >= nrows) {  // whole groups leave together
    wait_previous();
    return;
  }
  const int64_t i = rows[t], q0 = rp[i], q1 = rp[i + 1];
  wait_previous();
  const OutT *oc[KC];
#pragma unroll
  for (int j = 0; j < KC; ++j) oc[j] = KC == 1 ? out : out + min(col0 + j, k - 1) * n;
  VT s[KC][4] = {};
  for (int64_t q = q0 + sub; q < q1; q += 4 * LANES) {
    int32_t c[4];
    VT w[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const bool ok = q + u * LANES < q1;
      c[u] = ok ? ci[q + u * LANES] : -1;
      w[u] = ok ? v[q + u * LANES] : VT(0);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (c[u] >= 0) {
#pragma unroll
        for (int j = 0; j < KC; ++j) s[j][u] = fma(w[u], (VT)oc[j][c[u]], s[j][u]);
      }
  }
  const unsigned mask = LANES == 32 ? 0xffffffffu : (((1u << LANES) - 1u) << ((threadIdx.x & 31) / LANES * LANES));
#pragma unroll
  for (int j = 0; j < KC; ++j) {
    VT sum = (s[j][0] + s[j][1]) + (s[j][2] + s[j][3]);
#pragma unroll
    for (int o = LANES / 2; o; o >>= 1) sum += __shfl_xor_sync(mask, sum, o, LANES);
    const int64_t at = KC == 1 ? i : (col0 + j) * n + i;
    if (sub == 0 && (KC == 1 || col0 + j < k)) acc[at] = (VT)in[at] - sum;
  }
}

template <typename VT>
struct BlkArgs {
  const BlkPiece *pieces;  // of the stage
  const int64_t *rec_off;
  const unsigned char *recs;
  const VT *inv;  // of the stage
  unsigned int *status;
  int64_t stride;
  int C, B;
  int gl, helpers;
  int ring, slot;
  int fused;  // the records hold external entries
  int xrows;  // positions of the unknowns' array (four zeros follow)
  int k;      // right-hand sides, columns n apart
  int64_t n;
  int32_t goff[kBlkMaxGroups + 1];
};

__device__ __forceinline__ uint32_t map_rank(uint32_t addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(addr), "r"(rank));
  return r;
}
// Four consecutive values to another thread block's shared memory; their
// bytes count toward its mbarrier.
__device__ __forceinline__ void send4(uint32_t dst, const float (&x)[4], uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v4.f32 [%0], {%1, %2, %3, %4}, [%5];\n" ::"r"(dst),
               "f"(x[0]), "f"(x[1]), "f"(x[2]), "f"(x[3]), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void send4(uint32_t dst, const double (&x)[4], uint32_t bar) {
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];\n" ::"r"(dst),
               "d"(x[0]), "d"(x[1]), "r"(bar)
               : "memory");
  asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.v2.f64 [%0], {%1, %2}, [%3];\n" ::"r"(dst + 16),
               "d"(x[2]), "d"(x[3]), "r"(bar)
               : "memory");
}
__device__ __forceinline__ void mbar_expect(uint64_t *bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_addr(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
  __syncwarp();
  asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
// Barrier 1 over the first `n` threads.
__device__ __forceinline__ void row_barrier(int n) { asm volatile("bar.sync 1, %0;\n" ::"r"(n) : "memory"); }

// Shared-memory reads by 32-bit address, issued in program order: a batch of
// them is in flight before the first result is used.
__device__ __forceinline__ uint4 lds16(uint32_t a) {
  uint4 v;
  asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ uint2 lds8(uint32_t a) {
  uint2 v;
  asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];\n" : "=r"(v.x), "=r"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void lds_val(uint32_t a, float &v) { asm volatile("ld.shared.f32 %0, [%1];\n" : "=f"(v) : "r"(a) : "memory"); }
__device__ __forceinline__ void lds_val(uint32_t a, double &v) { asm volatile("ld.shared.f64 %0, [%1];\n" : "=d"(v) : "r"(a) : "memory"); }

// Whether any of four sums is a NaN or an infinity (FP32: or their sum, which
// is as good; FP64 additions are scarce).
__device__ __forceinline__ bool not_finite(const float (&x)[4]) {
  return (__float_as_uint((x[0] + x[1]) + (x[2] + x[3])) & 0x7f800000u) == 0x7f800000u;
}
__device__ __forceinline__ bool not_finite(const double (&x)[4]) {
  bool any = false;
#pragma unroll
  for (int r = 0; r < 4; ++r) any |= (__double2hiint(x[r]) & 0x7ff00000) == 0x7ff00000;
  return any;
}

// 16 bytes of values; dot_nonzero leaves out the terms where this one is zero.
template <typename VT>
struct Vec16;
template <>
struct Vec16<float> {
  float4 v;
  __device__ __forceinline__ void lds(uint32_t a) {
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];\n" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(a) : "memory");
  }
  __device__ __forceinline__ float get(int i) const { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }
  __device__ __forceinline__ float dot(const Vec16 &b, float s) const {
    return fmaf(v.w, b.v.w, fmaf(v.z, b.v.z, fmaf(v.y, b.v.y, fmaf(v.x, b.v.x, s))));
  }
  __device__ __forceinline__ float dot_nonzero(const Vec16 &b, float s) const {
    if (v.x != 0.f) s = fmaf(v.x, b.v.x, s);
    if (v.y != 0.f) s = fmaf(v.y, b.v.y, s);
    if (v.z != 0.f) s = fmaf(v.z, b.v.z, s);
    if (v.w != 0.f) s = fmaf(v.w, b.v.w, s);
    return s;
  }
};
template <>
struct Vec16<double> {
  double2 v;
  __device__ __forceinline__ void lds(uint32_t a) {
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];\n" : "=d"(v.x), "=d"(v.y) : "r"(a) : "memory");
  }
  __device__ __forceinline__ double get(int i) const { return i & 1 ? v.y : v.x; }
  __device__ __forceinline__ double dot(const Vec16 &b, double s) const {
    return fma(v.y, b.v.y, fma(v.x, b.v.x, s));
  }
  __device__ __forceinline__ double dot_nonzero(const Vec16 &b, double s) const {
    if (v.x != 0.0) s = fma(v.x, b.v.x, s);
    if (v.y != 0.0) s = fma(v.y, b.v.y, s);
    return s;
  }
};

// Quads [q, q1) of a list by step `lanes`: sum of value * unknown at the
// position (unknowns at xs_at).
template <typename VT>
__device__ __forceinline__ VT quad_sum(uint32_t cols, uint32_t vals, uint32_t q, uint32_t q1, uint32_t lanes,
                                       uint32_t xs_at, VT s0) {
  constexpr uint32_t vsz = sizeof(VT);
  VT s1 = VT(0);
  for (; q < q1; q += lanes) {
    const uint2 c = lds8(cols + 8 * q);
    Vec16<VT> w, w2;
    w.lds(vals + 4 * vsz * q);
    if (vsz == 8) w2.lds(vals + 4 * vsz * q + 16);
    VT y0, y1, y2, y3;
    lds_val(xs_at + vsz * (c.x & 0xffffu), y0);
    lds_val(xs_at + vsz * (c.x >> 16), y1);
    lds_val(xs_at + vsz * (c.y & 0xffffu), y2);
    lds_val(xs_at + vsz * (c.y >> 16), y3);
    s0 = fma(w.get(0), y0, s0), s1 = fma(w.get(1), y1, s1);
    s0 = fma(vsz == 8 ? w2.get(0) : w.get(2), y2, s0), s1 = fma(vsz == 8 ? w2.get(1) : w.get(3), y3, s1);
  }
  return s0 + s1;
}

// Pairs [q, q1) of external entries by step `lanes`, four pairs in flight.
template <typename VT, typename OutT>
__device__ __forceinline__ VT ext_sum(uint32_t cols, uint32_t vals, uint32_t q, uint32_t q1, uint32_t lanes,
                                      const OutT *out) {
  VT s0 = VT(0), s1 = VT(0);
  for (; q < q1; q += 4 * lanes) {
    uint2 c[4];
    OutT y[4][2];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      c[u] = make_uint2(kNoCol, kNoCol);
      if (q + u * lanes < q1) c[u] = lds8(cols + 8 * (q + u * lanes));
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      y[u][0] = c[u].x != kNoCol ? out[c[u].x] : OutT(0);
      y[u][1] = c[u].y != kNoCol ? out[c[u].y] : OutT(0);
    }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (q + u * lanes < q1) {
        VT w0, w1;
        lds_val(vals + 2 * (uint32_t)sizeof(VT) * (q + u * lanes), w0);
        lds_val(vals + 2 * (uint32_t)sizeof(VT) * (q + u * lanes) + (uint32_t)sizeof(VT), w1);
        s0 = fma(w0, (VT)y[u][0], s0), s1 = fma(w1, (VT)y[u][1], s1);
      }
  }
  return s0 + s1;
}

// One cluster (of one to 16 thread blocks) per piece.
// A step is bound by latency: two dependent shared-memory reads (entries),
// two exchanges of t and x (about 400 cycles each), one read and 4 NV FMAs
// (product) and the shuffles of two sums.  Measured at 128^3 (FP32 forward,
// the root's 16,384 rows, 32 steps of 512 by 16 thread blocks): 48 us, against
// 293 us for 512 steps of 32 rows by one thread block (pipe_kernel); all
// stages 507 us in turn, 447 us with early starts, against 1122 us.  The subdomains (512 pieces, 92% of the
// rows) take 132 us of it for 490 MB, 3.7 TB/s (w2_kernel: 200 us).
//   row threads: gl lanes per group of four own rows, a quarter of them per
//     row for the sparse sums.  Step s adds the row's entries in block s-1 to
//     the sum that is ready for it, sends t to every thread block, waits for
//     all of t, forms x = T^-1 t and sends x.  In the product every lane
//     multiplies its chunks of t with the four rows' vectors of the inverse,
//     which it holds in registers (loaded during the step before), and the
//     lanes' sums are folded so that each quarter ends with its own row's x.
//   helper threads (clusters): meanwhile sum block s+1's right-hand side,
//     external entries and entries in blocks up to s-1.  In a single thread
//     block the row threads do this themselves: several pieces share an SM
//     there and fewer instructions count.
// The thread after the row threads streams the records: record s+2 is waited
// for in step s.  One block-wide barrier per step, which also carries a
// failed wait.
// Registers: where many thread blocks share an SM, the compiler's choice would
// leave out one of them.  FP32 with one vector of the inverse per row is held
// to 64 (it would take 83 for the branch on infinities: 12^3 with 32 columns
// 52 -> 65 us), with two in a cluster to 80 (104: 64^3 with 32 columns 1.42 ->
// 1.49 ms; 64: with one column 246 -> 320 us).  A launch has 384 threads at
// most: 256 row threads and 128 helpers.
template <typename VT, int NV, bool CLUSTER>
struct BlkBounds {
  static constexpr bool pairs = NV == 2 && CLUSTER && sizeof(VT) == 4;
  static constexpr int threads = pairs ? 384 : 512;
  static constexpr int blocks = pairs || (NV == 1 && (CLUSTER || sizeof(VT) == 4)) ? 2 : 1;
};
template <typename VT, typename InT, typename OutT, bool UPPER, int NV, bool CLUSTER>
__global__ void __launch_bounds__(BlkBounds<VT, NV, CLUSTER>::threads, BlkBounds<VT, NV, CLUSTER>::blocks)
    blk_solve_kernel(BlkArgs<VT> a, const InT *in, OutT *out) {
  allow_next();
  extern __shared__ __align__(16) unsigned char smem[];
  const int C = CLUSTER ? a.C : 1;
  const int rank = CLUSTER ? (int)(blockIdx.x % (unsigned)C) : 0;
  // a cluster takes one column of a piece; the columns of a piece run side by
  // side, so its records and inverses come from L2 for all but one of them
  unsigned item = CLUSTER ? blockIdx.x / (unsigned)C : blockIdx.x;
  if (a.k > 1) {
    const int64_t col = item % (unsigned)a.k;
    item /= (unsigned)a.k;
    in += col * a.n;
    out += col * a.n;
  }
  const BlkPiece pc = a.pieces[item];
  const int tid = threadIdx.x, T = blockDim.x, B = a.B, nb = pc.nblocks, rows = pc.rows;
  const int nown = B / C, GL = a.gl, LD = GL >> 2, TC = nown * LD;
  constexpr int per = 16 / (int)sizeof(VT);
  constexpr uint32_t vsz = sizeof(VT);
  uint64_t *bar = reinterpret_cast<uint64_t *>(smem), *tbar = bar + kBlkRingMax, *xbar = tbar + 1;
  VT *tb = reinterpret_cast<VT *>(smem + kBlkBars);
  VT *ps = tb + B;         // [2][nown] sums for the coming blocks
  VT *xs = ps + 2 * nown;  // the piece's unknowns by position, then four zeros
  const uint32_t xs_at = smem_addr(xs), zero = xs_at + vsz * a.xrows;
  const uint32_t ring_at = zero + 4 * vsz;
  unsigned char *ring = smem + kBlkBars + vsz * (size_t)(B + 2 * nown + a.xrows + 4);
  auto block_bytes = [&](int s) { return (uint32_t)(min(B, (rows - s * B + 3) / 4 * 4)) * vsz; };
  const int64_t *roff = a.rec_off + pc.rec0 + rank;
  const bool streamer = tid == TC;
  // streamer: the next record to copy (its offsets loaded ahead) and to wait for
  int issued = 0, islot = 0, wslot = 0;
  uint32_t wpar = 0;
  int64_t o0 = 0, o1 = 0;
  auto issue = [&]() {
    bulk_load(ring + (size_t)islot * a.slot, a.recs + o0, (uint32_t)(o1 - o0), bar + islot);
    if (++islot == a.ring) islot = 0;
    if (++issued < nb) o0 = roff[(int64_t)issued * C], o1 = roff[(int64_t)issued * C + 1];
  };
  bool dead = false;  // a bounded wait of this thread gave up
  auto give_up = [&]() {
    dead = true;
    atomicOr(a.status, 1u);
  };
  auto wait_record = [&]() {
    if (!dead && !mbar_wait(bar + wslot, wpar)) give_up();
    if (++wslot == a.ring) wslot = 0, wpar ^= 1u;
  };
  auto stream = [&](int s, bool stop) {  // in step s: copy into record s-1's slot (free since the barrier), await s+2
    if (stop) return;
    if (s >= 1 && issued < nb) {
      fence_proxy_async();
      issue();
    }
    if (s + 2 < nb) wait_record();
  };
  if (streamer) {
    o0 = roff[0], o1 = roff[1];
    for (int i = 0; i < a.ring; ++i) mbar_init(bar + i, 1);
    mbar_init(tbar, 1);
    mbar_init(xbar, 1);
    fence_mbar_init();
    if (CLUSTER) {
      mbar_expect(tbar, block_bytes(0));
      mbar_expect(xbar, block_bytes(0));
    }
    while (issued < a.ring && issued < nb) issue();
    for (int s = 0; s < 2 && s < nb; ++s) wait_record();
  }
  for (int i = tid; i < B; i += T) tb[i] = VT(0);
  if (tid < 4) xs[a.xrows + tid] = VT(0);
  bool stop = __syncthreads_or(dead);
  if (CLUSTER) cluster_sync();  // every thread block's mbarriers exist before the first send

  // This thread's row: position in its block, place of its values in the
  // vectors (one block further per step), right-hand sides loaded a block
  // ahead.
  const bool row_thread = tid < TC;
  const int th = row_thread ? tid : tid - TC;
  const int L = row_thread || !CLUSTER ? LD : a.helpers / nown, j = th / L, l = th % L;
  const int pos = own_pos(j, rank, C);
  int64_t at = UPPER ? pc.begin + rows - 1 - pos : pc.begin + pos;  // block 0's row
  const int step = UPPER ? -B : B;
  int left = rows - pos;  // > 0: the current block has this row
  const InT *ip = in + at;
  int fleft = left;
  InT ri = InT(0);
  auto fetch = [&]() {  // past the last row: the piece's first one again
    ri = *(fleft > 0 ? ip : in + pc.begin);
    fleft -= B;
    ip += step;
  };
  auto next_rhs = [&]() {  // the next block's; the one after it is requested
    const VT r = (VT)ri;
    fetch();
    return r;
  };

  if (row_thread) {
    // ---- row threads
    const int lane = tid & 31, lg = lane & (GL - 1), grp = tid / GL;
    const int gfirst = pos & ~3;  // first position of the group
    const VT *inv = a.inv + (pc.blk0 * C + rank) * a.stride;
    const int64_t inv_step = (int64_t)C * a.stride;
    const uint32_t ioff = (uint32_t)(a.goff[grp] + lg) * per;
    const int nvec = (int)((uint32_t)(a.goff[grp + 1] - a.goff[grp]) / (uint32_t)(4 * GL));  // chunks of this lane
    Vec16<VT> m[NV][4];
    // In a single thread block every load is made, past the group's own chunks
    // of its last one again (multiplied with zeros): a load under a condition
    // would have to arrive before the loop goes on, and the step is short.  In
    // a cluster the loads that are not needed would cost more (the root of a
    // 128^3 grid: 74 us against 49).  Past the last block what follows is read.
    uint32_t i_at[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v) i_at[v] = ioff + (uint32_t)(min(v, nvec - 1) * 4 * GL * per);
    auto load_inv = [&]() {
#pragma unroll
      for (int v = 0; v < NV; ++v)
        if (!CLUSTER || v < nvec) {
#pragma unroll
          for (int r = 0; r < 4; ++r)
            m[v][r] = *reinterpret_cast<const Vec16<VT> *>(inv + (i_at[v] + (uint32_t)(r * GL * per)));
        }
      inv += inv_step;
    };
#pragma unroll
    for (int v = 0; v < NV; ++v)
#pragma unroll
      for (int r = 0; r < 4; ++r) m[v][r] = Vec16<VT>{};
    load_inv();
    // chunks of t past the group's positions are read as zeros
    uint32_t t_at[NV];
#pragma unroll
    for (int v = 0; v < NV; ++v)
      t_at[v] = (v * GL + lg) * per <= gfirst + 3 ? smem_addr(tb) + (uint32_t)(v * GL + lg) * 16 : zero;
    // sends: lane r of a group serves rank r
    uint32_t t_dst = 0, t_bar = 0, x_dst = 0, x_bar = 0;
    if (CLUSTER && lg < C) {
      t_dst = map_rank(smem_addr(tb + gfirst), lg);
      x_dst = map_rank(smem_addr(xs + gfirst), lg);
      t_bar = map_rank(smem_addr(tbar), lg);
      x_bar = map_rank(smem_addr(xbar), lg);
    }
    int gleft = lg < C ? rows - gfirst : 0;  // > 0: this lane sends the group's values
    auto send = [&](uint32_t dst, uint32_t bar_at, VT x) {
      VT v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = __shfl_sync(0xffffffffu, x, u * LD, GL);
      if (gleft > 0) send4(dst, v, bar_at);
    };
    VT rhs = VT(0), part = VT(0);
    uint32_t p = ring_at, q0 = 0, q1 = 0;  // the coming record and this thread's quads of its chain list
    uint32_t o_ccol = 0, o_cval = 0;
    OutT ey[2] = {OutT(0), OutT(0)};  // the first external pair, gathered before the barrier
    VT ew[2] = {VT(0), VT(0)};
    bool eon[2] = {false, false};
    int cslot = 0;
    auto open_record = [&]() {
      p = ring_at + (uint32_t)cslot * a.slot;
      if (++cslot == a.ring) cslot = 0;
      const uint4 h0 = lds16(p);
      const uint2 f0 = lds8(p + kBlkOff + 8 * j), f1 = lds8(p + kBlkOff + 8 * j + 8);
      o_ccol = p + h0.x, o_cval = p + h0.w;
      q0 = (f0.x & 0xffffu) + l, q1 = f1.x & 0xffffu;
      if (!CLUSTER) {
        const uint4 h1 = lds16(p + 16);
        part = VT(0);
        const uint32_t x0 = (f0.y & 0xffffu) + l, x1 = f1.y & 0xffffu;
        if (a.fused) {
          const bool on = x0 < x1;
          const uint2 c = lds8(on ? p + h0.z + 8 * x0 : zero);
          eon[0] = on;
          eon[1] = on && c.y != kNoCol;
          ey[0] = out[on ? c.x : (uint32_t)pc.begin];
          ey[1] = out[eon[1] ? c.y : (uint32_t)pc.begin];
          lds_val(on ? p + h1.y + 2 * vsz * x0 : zero, ew[0]);
          lds_val(on ? p + h1.y + 2 * vsz * x0 + vsz : zero, ew[1]);
          if (x0 + LD < x1) part = ext_sum<VT, OutT>(p + h0.z, p + h1.y, x0 + LD, x1, LD, out);
        }
      }
    };
    OutT *op = out + at;
    wait_previous();
    if (!CLUSTER) {
      fetch();
      rhs = next_rhs();
    }
    if (!stop) open_record();
    for (int s = 0; s < nb; ++s) {
      if (CLUSTER && s > 0) {
        if (!dead && !mbar_wait(xbar, (uint32_t)(s - 1) & 1u)) give_up();
        if (tid == 0 && !dead) mbar_expect(xbar, block_bytes(s));  // one arrival per phase
      }
      stop = __syncthreads_or(dead) || stop;
      VT sum = part;
      if (!CLUSTER && a.fused)
        sum = fma(ew[0], eon[0] ? (VT)ey[0] : VT(0), fma(ew[1], eon[1] ? (VT)ey[1] : VT(0), sum));
      if (!stop) sum = quad_sum<VT>(o_ccol, o_cval, q0, q1, LD, xs_at, sum);
      for (int o = LD >> 1; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (CLUSTER) {
        send(t_dst, t_bar, left > 0 ? ps[(s & 1) * nown + j] - sum : VT(0));
        if (!stop && s + 1 < nb) open_record();
        if (!dead && !mbar_wait(tbar, (uint32_t)s & 1u)) give_up();
        if (tid == 0 && !dead && s + 1 < nb) mbar_expect(tbar, block_bytes(s + 1));
        __syncwarp();
      } else {
        if (l == 0) tb[pos] = left > 0 ? rhs - sum : VT(0);
        row_barrier(TC);
      }
      VT x[4] = {VT(0), VT(0), VT(0), VT(0)};
      Vec16<VT> tv[NV];
#pragma unroll
      for (int v = 0; v < NV; ++v) tv[v].lds(t_at[v]);
#pragma unroll
      for (int v = 0; v < NV; ++v)
        if (vsz == 4 || v < nvec) {  // FP64 arithmetic is scarce: chunks past the group's rows are left out
#pragma unroll
          for (int r = 0; r < 4; ++r) x[r] = m[v][r].dot(tv[v], x[r]);
        }
      if (not_finite(x)) {
        // A NaN or an infinity in t: the inverse's zeros must not carry it to
        // rows that do not depend on it.
#pragma unroll
        for (int r = 0; r < 4; ++r) {
          x[r] = VT(0);
#pragma unroll
          for (int v = 0; v < NV; ++v) x[r] = m[v][r].dot_nonzero(tv[v], x[r]);
        }
      }
      {  // fold: after two exchanges each quarter of the group holds its own row
        const bool hi = lg & (GL >> 1), hi2 = lg & (GL >> 2);
        const VT y0 = hi ? x[2] : x[0], y1 = hi ? x[3] : x[1];
        const VT z0 = __shfl_xor_sync(0xffffffffu, hi ? x[0] : x[2], GL >> 1),
                 z1 = __shfl_xor_sync(0xffffffffu, hi ? x[1] : x[3], GL >> 1);
        const VT w0 = y0 + z0, w1 = y1 + z1;
        x[0] = (hi2 ? w1 : w0) + __shfl_xor_sync(0xffffffffu, hi2 ? w0 : w1, GL >> 2);
      }
      for (int o = GL >> 3; o; o >>= 1) x[0] += __shfl_xor_sync(0xffffffffu, x[0], o);
      if (CLUSTER) send(x_dst, x_bar, x[0]);
      else if (l == 0 && left > 0) xs[s * B + pos] = x[0];
      load_inv();
      if (l == 0 && left > 0) *op = (OutT)x[0];
      op += step;
      left -= B;
      gleft -= B;
      x_dst += (uint32_t)B * vsz;
      if (!CLUSTER && s + 1 < nb) {
        rhs = next_rhs();
        if (!stop) open_record();
      }
    }
  } else {
    // ---- helper threads (single thread blocks: one warp that only streams)
    int hslot = 0;
    auto prepare = [&](int s) {
      const VT r = next_rhs();
      VT sum = VT(0);
      if (!stop) {
        const uint32_t p = ring_at + (uint32_t)hslot * a.slot;
        const uint4 h0 = lds16(p), h1 = lds16(p + 16);
        const uint2 f0 = lds8(p + kBlkOff + 8 * j), f1 = lds8(p + kBlkOff + 8 * j + 8);
        if (h1.z) sum = ext_sum<VT, OutT>(p + h0.z, p + h1.y, (f0.y & 0xffffu) + l, f1.y & 0xffffu, L, out);
        sum = quad_sum<VT>(p + h0.y, p + h1.x, (f0.x >> 16) + l, f1.x >> 16, L, xs_at, sum);
      }
      if (++hslot == a.ring) hslot = 0;
      for (int o = L >> 1; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (l == 0) ps[(s & 1) * nown + j] = r - sum;
    };
    wait_previous();
    if (CLUSTER) {
      fetch();
      prepare(0);
    }
    for (int s = 0; s < nb; ++s) {
      if (CLUSTER && s > 0 && !dead && !mbar_wait(xbar, (uint32_t)(s - 1) & 1u)) give_up();
      stop = __syncthreads_or(dead) || stop;
      if (streamer) stream(s, stop);
      __syncwarp();
      if (CLUSTER && s + 1 < nb) prepare(s + 1);
    }
    if (streamer && (dead || stop)) {  // wait (bounded) for copies still in flight
      for (int s = max(0, issued - a.ring); s < issued; ++s) (void)mbar_wait(bar + s % a.ring, (uint32_t)(s / a.ring) & 1u);
    }
  }
  if (CLUSTER) {
    if (!dead && !mbar_wait(xbar, (uint32_t)(nb - 1) & 1u)) give_up();
    cluster_sync();  // nobody leaves while others may still send here
    // Without a completed phase the others' last stores, all issued by now, may
    // still be on their way: they take microseconds.
    if (dead) __nanosleep(1000000);
  }
}

}  // namespace

// ---- plan ----------------------------------------------------------------------------------------

namespace {

using ClusterFit = std::array<int, 5>;

// Cluster size, block rows and threads of a stage of npieces pieces, the
// longest with maxrows rows.
//
// The fewer the pieces, the larger the clusters that run side by side (7
// clusters of 16 fit the GB300's GPCs with one thread block per SM, 15 of 8,
// 36 of 4, 76 of 2; a stage that exceeds this by one or two still gains), and
// B grows with the cluster so that a thread block has 16 to 64 rows: a step
// costs about 1.3 us in a cluster (two exchanges, two barriers) whatever B
// is, against about 1 us in a single thread block.  Short pieces take smaller
// clusters: below maxrows the steps saved do not pay for the exchanges.
// 128^3 log-normal, 512 subdomains, FP32 forward solve, kernels in turn: 507 us
// with these lines; 528 with clusters of 8 only up to 9 pieces, 527 with single thread
// blocks from 40 pieces on, 1122 with the record streams of trsv.cu.
// In FP64 (2 FMA per clock and SM) the inverse's B / 2 products per row are
// what a step costs, so B is smaller: 417 us for 64^3 with 64 subdomains
// against 451 with B = 128 at the root and 1066 with the record streams.
// fit: clusters of 1, 2, 4, 8, 16 that the device runs at once; a size that it
// does not run at all gives way to the next smaller one.
void choose_shape(BlkStage &S, bool fp32, int cols, const ClusterFit &fit) {
  const int P = (int)std::min<int64_t>((int64_t)S.npieces * cols, 1 << 20), R = S.maxrows;
  int i = P <= 8 && R >= 512 ? 4 : P <= 18 && R >= 256 ? 3 : P <= 36 && R >= 128 ? 2 : P <= 76 && R >= 128 ? 1 : 0;
  while (i > 0 && fit[i] < 1) --i;
  static const int b32[] = {64, 128, 256, 256, 512}, b64[] = {32, 64, 128, 128, 256};
  static const int g32[] = {8, 16, 16, 32, 32}, g64[] = {16, 16, 32, 32, 32};
  S.C = 1 << i;
  S.B = fp32 ? b32[i] : b64[i];
  while (S.B > 32 && S.B / 2 >= R) S.B /= 2;
  S.gl = fp32 ? g32[i] : g64[i];
}

// Threads, vectors of the inverse and their places for the stage's C, B and gl.
void set_geometry(BlkStage &S, size_t vsz) {
  const int per = 16 / (int)vsz;
  S.C = std::min(S.C, S.B / 8);
  const int nown = S.B / S.C, chunks = S.B / per;
  while (S.gl > 8 && (nown / 4 * S.gl > 384 || S.gl > chunks)) S.gl /= 2;
  while (S.gl < 32 && (chunks > 4 * S.gl || nown / 4 * S.gl < 32 || S.gl < S.C)) S.gl *= 2;
  S.nv = chunks <= S.gl ? 1 : chunks <= 2 * S.gl ? 2 : 4;
  if (S.C == 1) {
    S.helpers = 32;
  } else {
    S.helpers = std::max(128, nown);  // 4 warps; 8 measured no faster in FP32 and slower in FP64
  }
  S.goff[0] = 0;
  for (int g = 0; g < nown / 4; ++g) {
    const int last = (g * S.C + S.C - 1) * 4 + 3;  // of any rank's group g
    S.goff[g + 1] = S.goff[g] + (last / (S.gl * per) + 1) * 4 * S.gl;
  }
  S.stride = (int64_t)S.goff[nown / 4] * per;
}

constexpr int kMaxDevices = 128;

// Clusters of 1, 2, 4, 8 and 16 thread blocks, one per SM, that run at once on
// the current device (152, 76, 36, 15 and 7 on a whole GB300); asked once.
const ClusterFit &cluster_fit() {
  static std::once_flag once[kMaxDevices];
  static ClusterFit fit[kMaxDevices];
  int dev = 0;
  RCHOL_CUDA(cudaGetDevice(&dev));
  RCHOL_CHECK_ARG(dev >= 0 && dev < kMaxDevices, "device ordinal out of range");
  std::call_once(once[dev], [&] {
    auto *kernel = blk_solve_kernel<float, float, double, true, 1, true>;
    RCHOL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBlkSmem));
    RCHOL_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
    RCHOL_CUDA(cudaDeviceGetAttribute(&fit[dev][0], cudaDevAttrMultiProcessorCount, dev));
    for (int i = 1; i < 5; ++i) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(1u << i);
      cfg.blockDim = dim3(256);
      cfg.dynamicSmemBytes = kBlkSmem;
      cudaLaunchAttribute at;
      at.id = cudaLaunchAttributeClusterDimension;
      at.val.clusterDim.x = 1u << i;
      at.val.clusterDim.y = at.val.clusterDim.z = 1;
      cfg.attrs = &at;
      cfg.numAttrs = 1;
      if (cudaOccupancyMaxActiveClusters(&fit[dev][i], kernel, &cfg) != cudaSuccess) {
        (void)cudaGetLastError();
        fit[dev][i] = 0;
      }
    }
  });
  return fit[dev];
}

size_t stage_smem(const BlkStage &S, size_t vsz, int ring) {
  return kBlkBars + vsz * (size_t)(S.B + 2 * (S.B / S.C) + (S.maxrows + 3) / 4 * 4 + 4) + (size_t)ring * S.slot;
}

template <typename VT>
bool build_dir(int64_t n, const DevBuf<int64_t> &rp, const DevBuf<int32_t> &ci, const DevBuf<double> &v,
               const std::vector<TreeNode> &tnodes, bool upper, int cols, BlkDir &D, DevBuf<VT> &inv, cudaStream_t s) {
  const ClusterFit &fit = cluster_fit();
  int maxdepth = 1;
  for (auto &nd : tnodes) maxdepth = std::max(maxdepth, nd.depth);
  std::vector<BlkPiece> pieces;
  D.stages.clear();
  std::vector<std::vector<std::pair<int64_t, int64_t>>> by_depth(maxdepth + 1);
  for (auto &nd : tnodes)
    if (std::min(nd.end, n) > nd.begin) by_depth[nd.depth].push_back({nd.begin, std::min(nd.end, n)});
  for (int st = 0; st < maxdepth; ++st) {
    const auto &nodes = by_depth[upper ? st + 1 : maxdepth - st];
    // piece number t of every node of this depth, in processing order
    for (int64_t t = 0;; ++t) {
      BlkStage S;
      S.piece0 = (int)pieces.size();
      for (auto &nd : nodes) {
        const int64_t len = nd.second - nd.first, np = (len + kBlkMaxRows - 1) / kBlkMaxRows;
        if (t >= np) continue;
        const int64_t u = upper ? np - 1 - t : t;  // equal pieces of whole 32-row groups
        const int64_t step = ((len + np - 1) / np + 31) / 32 * 32;
        const int64_t b = nd.first + std::min(len, u * step), e = nd.first + std::min(len, (u + 1) * step);
        if (e <= b) continue;
        pieces.push_back(BlkPiece{b, (int32_t)(e - b), 0, 0, 0});
        S.maxrows = std::max<int>(S.maxrows, (int)(e - b));
        S.rows += e - b;
      }
      S.npieces = (int)pieces.size() - S.piece0;
      if (!S.npieces) break;
      choose_shape(S, sizeof(VT) == 4, cols, fit);
      D.stages.push_back(S);
    }
  }
  DevBuf<int4> bnd(n);
  D.pieces.upload(pieces.data(), pieces.size(), s);
  // forward: the first stage's columns (nearly all of them) are summed for
  // all later rows at once after it
  DevBuf<unsigned char> early;
  DevBuf<int64_t> nearly;
  if (!upper && D.stages.size() > 1) {
    early.alloc(n);
    nearly.alloc(n + 1);
    RCHOL_CUDA(cudaMemsetAsync(early.p, 0, n, s));
    RCHOL_CUDA(cudaMemsetAsync(nearly.p, 0, nearly.bytes(), s));
    blk_mark_kernel<<<(unsigned)std::min(D.stages[0].npieces, 4096), 256, 0, s>>>(D.pieces.p, D.stages[0].npieces,
                                                                                 early.p);
    RCHOL_CUDA(cudaGetLastError());
  }
  for (int attempt = 0; attempt < 6; ++attempt) {
    std::vector<BlkRec> recs;
    std::vector<int64_t> stage_rec(1, 0);
    int64_t ninv = 0;
    for (auto &S : D.stages) {
      set_geometry(S, sizeof(VT));
      int64_t blocks = 0;
      for (int k = S.piece0; k < S.piece0 + S.npieces; ++k) {
        BlkPiece &pc = pieces[k];
        pc.nblocks = (pc.rows + S.B - 1) / S.B;
        pc.rec0 = (int64_t)recs.size();
        pc.blk0 = blocks;
        blocks += pc.nblocks;
        for (int t = 0; t < pc.nblocks; ++t) {
          const int32_t nr = std::min(S.B, pc.rows - t * S.B);
          const int64_t row0 = upper ? pc.begin + pc.rows - (int64_t)t * S.B - nr : pc.begin + (int64_t)t * S.B;
          for (int r = 0; r < S.C; ++r)
            recs.push_back(BlkRec{row0, pc.begin, pc.begin + pc.rows, nr, S.B, r, S.C,
                                  early.p && S.C > 1, (S.maxrows + 3) / 4 * 4});
        }
      }
      S.inv0 = ninv;
      ninv += blocks * S.C * S.stride;
      stage_rec.push_back((int64_t)recs.size());
    }
    const int64_t nrec = (int64_t)recs.size();
    DevBuf<BlkRec> d_recs(nrec);
    DevBuf<int4> d_cnt(nrec);
    d_recs.upload(recs.data(), nrec, s);
    blk_count_kernel<<<(unsigned)((nrec * 32 + 255) / 256), 256, 0, s>>>(d_recs.p, nrec, rp.p, ci.p, upper, early.p,
                                                                        bnd.p, nearly.p, d_cnt.p);
    RCHOL_CUDA(cudaGetLastError());
    std::vector<int4> cnt(nrec);
    d_cnt.download(cnt.data(), nrec, s);
    RCHOL_CUDA(cudaStreamSynchronize(s));
    std::vector<int64_t> off(nrec + 1, 0);
    bool refit = false;
    for (size_t st = 0; st < D.stages.size(); ++st) {
      BlkStage &S = D.stages[st];
      int64_t maxrec = 0, late = 0;
      bool fused = false;
      for (int64_t r = stage_rec[st]; r < stage_rec[st + 1]; ++r) {
        const int ne = recs[r].apart ? 0 : cnt[r].w;
        const bool fits16 = cnt[r].y <= 65535 && cnt[r].z <= 65535 && ne <= 65535;
        const int64_t len = fits16 ? blk_layout(S.B / S.C, cnt[r].y, cnt[r].z, ne, sizeof(VT)).len : (int64_t)1 << 30;
        late += recs[r].apart ? 2 * cnt[r].w : 0;
        fused |= ne > 0;
        off[r + 1] = off[r] + len;
        maxrec = std::max(maxrec, len);
      }
      S.slot = (int)maxrec;
      S.fused = fused;
      S.late_lanes = !late ? 0 : late < 6 * S.rows ? 2 : late < 32 * S.rows ? 8 : 32;
      if (stage_smem(S, sizeof(VT), 4) > kBlkSmem) {
        if (S.B <= 32) return false;
        S.B /= 2;
        refit = true;
        continue;
      }
      S.ring = 4;
      const int most = 6;
      while (S.ring < most && stage_smem(S, sizeof(VT), S.ring + 1) <= (S.C > 1 ? kBlkSmem / 2 : kBlkSmem / 4)) ++S.ring;
      S.smem = stage_smem(S, sizeof(VT), S.ring);
    }
    if (refit) continue;
    int64_t slack = 0;  // the kernel loads one block past a piece's last
    for (const BlkStage &S : D.stages) slack = std::max(slack, S.C * S.stride);
    // A plan of over an eighth of the device's memory per direction is left
    // out: the record streams (for several columns, the first plan) solve too.
    // The line is drawn by the problem alone, not by what is free just now:
    // the two plans round differently, and a program's results must not
    // depend on what else is resident.
    size_t room = 0, total = 0;
    RCHOL_CUDA(cudaMemGetInfo(&room, &total));
    const size_t need = (size_t)off[nrec] + (size_t)(ninv + slack) * sizeof(VT) + (size_t)v.n * (sizeof(VT) + 4);
    if (need > total / 8) return false;
    D.rec_off.upload(off.data(), nrec + 1, s);
    D.recs.alloc(off[nrec]);
    blk_fill_kernel<VT><<<(unsigned)nrec, 128, 0, s>>>(d_recs.p, D.rec_off.p, d_cnt.p, rp.p, ci.p, v.p, bnd.p, upper,
                                                      early.p, nearly.p, D.recs.p);
    RCHOL_CUDA(cudaGetLastError());
    inv.alloc(ninv + slack);
    RCHOL_CUDA(cudaMemsetAsync(inv.p, 0, inv.bytes(), s));
    RCHOL_CUDA(cudaFuncSetAttribute(blk_invert_kernel<VT>, cudaFuncAttributeMaxDynamicSharedMemorySize, 512 * 256));
    for (size_t st = 0; st < D.stages.size(); ++st) {
      const BlkStage &S = D.stages[st];
      const int64_t r0 = stage_rec[st], nblk = (stage_rec[st + 1] - r0) / S.C;
      const int panels = (S.B + 31) / 32;
      BlkInv g;
      g.C = S.C;
      g.gl = S.gl;
      g.stride = S.stride;
      std::copy(S.goff, S.goff + kBlkMaxGroups + 1, g.goff);
      blk_invert_kernel<VT><<<(unsigned)(nblk * panels), 32, (size_t)S.B * 256, s>>>(
          d_recs.p + r0, g, panels, rp.p, ci.p, v.p, bnd.p, upper, inv.p + S.inv0);
      RCHOL_CUDA(cudaGetLastError());
    }
    D.pieces.upload(pieces.data(), pieces.size(), s);
    D.early_rows = 0;
    if (early.p) {
      std::vector<int32_t> rows;
      for (size_t st = 1; st < D.stages.size(); ++st) {
        BlkStage &S = D.stages[st];
        S.erow0 = (int64_t)rows.size();
        for (int k = S.piece0; k < S.piece0 + S.npieces; ++k)
          for (int i = 0; i < pieces[k].rows; ++i) rows.push_back((int32_t)(pieces[k].begin + i));
      }
      const int64_t nr = D.early_rows = (int64_t)rows.size();
      D.erow.upload(rows.data(), nr, s);
      DevBuf<int64_t> nlate(n + 1);
      RCHOL_CUDA(cudaMemsetAsync(nlate.p, 0, nlate.bytes(), s));
      for (const BlkStage &S : D.stages)
        if (S.late_lanes)
          blk_late_count_kernel<<<(unsigned)((S.rows + 255) / 256), 256, 0, s>>>(S.rows, D.erow.p + S.erow0, bnd.p,
                                                                                nearly.p, nlate.p);
      RCHOL_CUDA(cudaGetLastError());
      auto make = [&](BlkExt &E, DevBuf<int64_t> &count, int want) {
        exclusive_scan_i64(count.p, n, s);
        int64_t ne = 0;
        RCHOL_CUDA(cudaMemcpyAsync(&ne, count.p + n, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
        RCHOL_CUDA(cudaStreamSynchronize(s));
        const double avg = (double)ne / (double)nr;
        E.lanes = avg < 6 ? 2 : avg < 48 ? 8 : 32;
        E.ci.alloc(std::max<int64_t>(ne, 1));
        if (sizeof(VT) == 4) E.v32.alloc(std::max<int64_t>(ne, 1));
        else E.v64.alloc(std::max<int64_t>(ne, 1));
        blk_ext_fill_kernel<<<(unsigned)((nr * 32 + 255) / 256), 256, 0, s>>>(
            nr, D.erow.p, rp.p, ci.p, v.p, bnd.p, early.p, want, count.p, E.ci.p, E.v32.p, E.v64.p);
        RCHOL_CUDA(cudaGetLastError());
        E.rp = std::move(count);
      };
      make(D.early, nearly, 1);
      make(D.late, nlate, 0);
    }
    RCHOL_CUDA(cudaStreamSynchronize(s));  // host arrays and temporaries end here
    return true;
  }
  return false;
}

// Launch of a kernel that calls wait_previous, in clusters of C thread blocks;
// early: it may start before the kernel ahead of it has ended.
template <typename... Params, typename... Args>
void chain_launch(void (*kernel)(Params...), dim3 grid, unsigned threads, size_t smem, int C, bool early,
                  cudaStream_t s, const Args &...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = early;
  at[1].id = cudaLaunchAttributeClusterDimension;
  at[1].val.clusterDim.x = (unsigned)C;
  at[1].val.clusterDim.y = at[1].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = C > 1 ? 2 : 1;
  RCHOL_CUDA(cudaLaunchKernelEx(&cfg, kernel, Params(args)...));
}

template <typename VT, typename InT, typename OutT, bool UPPER, int NV>
void launch_stage(const BlkStage &S, const BlkArgs<VT> &a, const InT *in, OutT *out, cudaStream_t s) {
  auto *single = blk_solve_kernel<VT, InT, OutT, UPPER, NV, false>;
  auto *multi = blk_solve_kernel<VT, InT, OutT, UPPER, NV, true>;
  static std::once_flag once[kMaxDevices];
  int dev = 0;
  RCHOL_CUDA(cudaGetDevice(&dev));
  RCHOL_CHECK_ARG(dev >= 0 && dev < kMaxDevices, "device ordinal out of range");
  std::call_once(once[dev], [&] {
    RCHOL_CUDA(cudaFuncSetAttribute(single, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBlkSmem));
    RCHOL_CUDA(cudaFuncSetAttribute(multi, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kBlkSmem));
    RCHOL_CUDA(cudaFuncSetAttribute(multi, cudaFuncAttributeNonPortableClusterSizeAllowed, 1));
  });
  const unsigned threads = (unsigned)(S.B / S.C / 4 * S.gl + S.helpers);
  const unsigned blocks = (unsigned)S.npieces * (unsigned)a.k * (unsigned)S.C;
  // A stage that starts early finds SMs busy with the one before, and its
  // thread blocks would share the free ones while others stay empty later (in
  // FP64, where an SM's arithmetic is what a step waits for, 700^2 took 1007 us
  // instead of 728).  So a stage that fits the GPU in `waves` thread blocks per
  // SM asks for the shared memory that admits no more.  Preconditioner, one
  // right-hand side, starting in turn -> early -> early with this rule, us:
  // FP32 80^3 547, 479, 444; 700^2 343, 273, 257; FP64 80^3 1283, 1354, 1199;
  // 700^2 728, 1007, 644; 12^3 72, 47, 48.  FP64 stages of more than one wave
  // start in turn: they run long, and early ones were up to 4% slower (700^2
  // with 5 columns 1534 -> 1594 us).
  const int fit = std::max(1, cluster_fit()[S.C == 1 ? 0 : S.C == 2 ? 1 : S.C == 4 ? 2 : S.C == 8 ? 3 : 4]);
  const int64_t waves = ((int64_t)S.npieces * a.k + fit - 1) / fit;
  const bool early = sizeof(VT) == 4 || waves == 1;
  size_t smem = S.smem;
  if (early && waves <= 4) smem = std::max(smem, kBlkSmem / 16 / (size_t)(waves + 1) * 16 + 2048);
  if (S.C == 1) chain_launch(single, blocks, threads, smem, 1, early, s, a, in, out);
  else chain_launch(multi, blocks, threads, smem, S.C, early, s, a, in, out);
  note_launch();
  RCHOL_CUDA(cudaGetLastError());
}

template <typename VT, typename InT, typename OutT, bool UPPER>
void launch_nv(const BlkStage &S, const BlkArgs<VT> &a, const InT *in, OutT *out, cudaStream_t s) {
  if (S.nv == 1) launch_stage<VT, InT, OutT, UPPER, 1>(S, a, in, out, s);
  else if (S.nv == 2) launch_stage<VT, InT, OutT, UPPER, 2>(S, a, in, out, s);
  else launch_stage<VT, InT, OutT, UPPER, 4>(S, a, in, out, s);
}

template <typename VT>
const VT *ext_values(const BlkExt &E);
template <>
const float *ext_values<float>(const BlkExt &E) {
  return E.v32.p;
}
template <>
const double *ext_values<double>(const BlkExt &E) {
  return E.v64.p;
}

template <typename VT, typename InT, typename OutT, int KC>
void launch_ext_kc(const BlkExt &E, int lanes, const int32_t *rows, int64_t nrows, const InT *in, const OutT *out,
                   VT *acc, int k, int64_t n, cudaStream_t s) {
  const dim3 grid((unsigned)((nrows * lanes + 255) / 256), (unsigned)((k + KC - 1) / KC));
  const VT *v = ext_values<VT>(E);
  if (lanes == 2) chain_launch(blk_ext_kernel<VT, InT, OutT, 2, KC>, grid, 256, 0, 1, true, s, rows, nrows, E.rp.p, E.ci.p, v, in, out, acc, k, n);
  else if (lanes == 8) chain_launch(blk_ext_kernel<VT, InT, OutT, 8, KC>, grid, 256, 0, 1, true, s, rows, nrows, E.rp.p, E.ci.p, v, in, out, acc, k, n);
  else chain_launch(blk_ext_kernel<VT, InT, OutT, 32, KC>, grid, 256, 0, 1, true, s, rows, nrows, E.rp.p, E.ci.p, v, in, out, acc, k, n);
  note_launch();
  RCHOL_CUDA(cudaGetLastError());
}

template <typename VT, typename InT, typename OutT>
void launch_ext(const BlkExt &E, int lanes, const int32_t *rows, int64_t nrows, const InT *in, const OutT *out, VT *acc,
                int k, int64_t n, cudaStream_t s) {
  if (k == 1) launch_ext_kc<VT, InT, OutT, 1>(E, lanes, rows, nrows, in, out, acc, k, n, s);
  else launch_ext_kc<VT, InT, OutT, 4>(E, lanes, rows, nrows, in, out, acc, k, n, s);
}

template <typename VT, typename InT, typename OutT, bool UPPER>
void launch_dir(const BlkDir &D, const VT *inv, const InT *in, OutT *out, VT *acc, int k, int64_t n,
                unsigned int *status, cudaStream_t s) {
  for (size_t st = 0; st < D.stages.size(); ++st) {
    const BlkStage &S = D.stages[st];
    if (st == 1 && D.early_rows)
      launch_ext<VT, InT, OutT>(D.early, D.early.lanes, D.erow.p, D.early_rows, in, out, acc, k, n, s);
    if (S.late_lanes) launch_ext<VT, VT, OutT>(D.late, S.late_lanes, D.erow.p + S.erow0, S.rows, acc, out, acc, k, n, s);
    BlkArgs<VT> a;
    a.pieces = D.pieces.p + S.piece0;
    a.rec_off = D.rec_off.p;
    a.recs = D.recs.p;
    a.inv = inv + S.inv0;
    a.status = status;
    a.stride = S.stride;
    a.C = S.C;
    a.B = S.B;
    a.gl = S.gl;
    a.helpers = S.helpers;
    a.ring = S.ring;
    a.slot = S.slot;
    a.fused = S.fused;
    a.xrows = (S.maxrows + 3) / 4 * 4;
    a.k = k;
    a.n = n;
    std::copy(S.goff, S.goff + kBlkMaxGroups + 1, a.goff);
    if (st > 0 && D.early_rows) launch_nv<VT, VT, OutT, UPPER>(S, a, acc, out, s);
    else launch_nv<VT, InT, OutT, UPPER>(S, a, in, out, s);
  }
}

// make() builds into fwd and bwd; kNoMemory where an allocation failed (the
// record streams or the first plan solve without this one).  Half a plan is
// given back.
template <typename Make>
BlkBuilt try_build(BlkDir &fwd, BlkDir &bwd, Make make) {
  BlkBuilt built = BlkBuilt::kLeftOut;
  try {
    if (make()) return BlkBuilt::kReady;
  } catch (const Error &e) {
    if (e.status != RCHOL_ERR_NOMEM) throw;
    built = BlkBuilt::kNoMemory;
  }
  fwd = BlkDir();
  bwd = BlkDir();
  return built;
}

bool build_block_dirs(const rchol_factor_s &F, int cols, BlkDir &fwd, BlkDir &bwd, cudaStream_t s) {
  if (F.precision == RCHOL_PREC_FP32)
    return build_dir<float>(F.n, F.lrp, F.lci, F.lv, F.nodes, false, cols, fwd, fwd.inv32, s) &&
           build_dir<float>(F.n, F.urp, F.uci, F.uv, F.nodes, true, cols, bwd, bwd.inv32, s);
  return build_dir<double>(F.n, F.lrp, F.lci, F.lv, F.nodes, false, cols, fwd, fwd.inv64, s) &&
         build_dir<double>(F.n, F.urp, F.uci, F.uv, F.nodes, true, cols, bwd, bwd.inv64, s);
}

// Inverses of large triangles are as accurate as substitution because nothing
// cancels in them: the diagonal is positive and no other entry is (true of
// every sampled factor).  Any other G keeps the record streams.
bool block_signs(const rchol_factor_s &F, cudaStream_t s) {
  DevBuf<unsigned long long> positive(2);
  RCHOL_CUDA(cudaMemsetAsync(positive.p, 0, positive.bytes(), s));
  blk_sign_kernel<<<1024, 256, 0, s>>>(F.n, F.nnz, F.urp.p, F.uv.p, positive.p);
  RCHOL_CUDA(cudaGetLastError());
  unsigned long long count[2];
  positive.download(count, 2, s);
  RCHOL_CUDA(cudaStreamSynchronize(s));
  return count[0] == (unsigned long long)F.n && count[1] == (unsigned long long)F.n;
}

}  // namespace

BlkBuilt build_blocks(const rchol_factor_s &F, SolvePlan &P, cudaStream_t s) {
  return try_build(P.bfwd, P.bbwd, [&] { return block_signs(F, s) && build_block_dirs(F, 1, P.bfwd, P.bbwd, s); });
}

// Whether one right-hand side is solved on the block plan, too (several always
// are).  Its clusters shorten the chain of stages with few pieces; where a
// stage's pieces take more than three rounds of all SMs, a warp per piece
// (w2_kernel) gets more done than a thread block per piece.  us per
// preconditioner, record streams / blocks: 400 systems of 512 rows FP32 33 /
// 19, FP64 95 / 87; 500 of 1024 FP32 60 / 73, FP64 185 / 257; 3000 of 256 FP32
// 55 / 90, FP64 199 / 267; 1000^2 grid with 4096 subdomains of 244 rows FP32 508
// / 302, FP64 1142 / 693.  The figures below are least-squares lines through 170
// such batches with 1 to 8 subdomains per system and single chains.
bool blocks_for_one(const rchol_factor_s &F, const SolvePlan &P) {
  const bool fp32 = F.precision == RCHOL_PREC_FP32;
  const int rounds = 3 * cluster_fit()[0];
  double gain = 0.0;  // us
  for (const BlkStage &S : P.bfwd.stages) {
    if (S.npieces <= rounds) gain += fp32 ? 9.0 + 0.028 * S.maxrows : 12.0 + 0.106 * S.maxrows;
    else if (fp32) gain += 10.0 - 1e-3 * (8.0 * S.npieces + 0.03 * (double)S.rows);
    else gain -= 1e-3 * (6.0 * S.npieces + 0.08 * (double)S.rows);
  }
  return gain >= 0.0;
}

void build_blocks_k(const rchol_factor_s &F, SolvePlan &P, int k, cudaStream_t s) {
  if (P.kblocks || k < kBlkWideFrom) return;
  P.kwide = try_build(P.bkfwd, P.bkbwd, [&] { return build_block_dirs(F, kBlkWideCols, P.bkfwd, P.bkbwd, s); }) ==
            BlkBuilt::kReady;
  P.kblocks = true;
}

void block_trsv(const rchol_factor_s &F, const SolvePlan &P, bool upper, const double *in64, const float *in32,
                double *out64, float *out32, void *acc, int k, cudaStream_t s) {
  unsigned int *st = P.status;
  float *a32 = static_cast<float *>(acc);
  double *a64 = static_cast<double *>(acc);
  const int64_t n = F.n;
  const bool wide = P.kwide && k >= kBlkWideFrom;
  const BlkDir &D = upper ? wide ? P.bkbwd : P.bbwd : wide ? P.bkfwd : P.bfwd;
  if (F.precision == RCHOL_PREC_FP32) {
    const float *inv = D.inv32.p;
    if (!upper && in64 && out32) launch_dir<float, double, float, false>(D, inv, in64, out32, a32, k, n, st, s);
    else if (!upper && in64 && out64) launch_dir<float, double, double, false>(D, inv, in64, out64, a32, k, n, st, s);
    else if (upper && in32 && out64) launch_dir<float, float, double, true>(D, inv, in32, out64, a32, k, n, st, s);
    else if (upper && in64 && out64) launch_dir<float, double, double, true>(D, inv, in64, out64, a32, k, n, st, s);
    else throw Error(RCHOL_ERR_INTERNAL, "unsupported triangular-solve operand types");
  } else {
    if (!in64 || !out64) throw Error(RCHOL_ERR_INTERNAL, "unsupported triangular-solve operand types");
    if (upper) launch_dir<double, double, double, true>(D, D.inv64.p, in64, out64, a64, k, n, st, s);
    else launch_dir<double, double, double, false>(D, D.inv64.p, in64, out64, a64, k, n, st, s);
  }
}

}  // namespace rchol
