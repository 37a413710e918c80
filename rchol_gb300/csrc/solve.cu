// SpMV with A, the transposed copy and FP32 copy of G, the solve plan, and
// the PCG loops of c++/util/pcg.cpp:57-159 on the GPU (one system with k
// right-hand sides, and many independent systems at once).  The triangular
// solves themselves are in trsv.cu.
//
// Several right-hand sides are stored row-major (n x k); every right-hand
// side keeps its own PCG scalars and stopping test.

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstring>
#include <future>
#include <numeric>
#include <vector>

#include "common.hpp"
#include "host.hpp"
#include "plan.hpp"

namespace rchol {

void exclusive_scan_i64(int64_t *d_data, int64_t n, cudaStream_t s);

void destroy_plan(SolvePlan *p) { delete p; }

namespace {

// ---- SpMV ---------------------------------------------------------------------

// y = A x for one right-hand side: LPR lanes per row.
template <int LPR>
__global__ void spmv1_kernel(int64_t n, const int64_t *__restrict__ rp, const int32_t *__restrict__ ci,
                             const double *__restrict__ v, const double *__restrict__ x,
                             double *__restrict__ y) {
  int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  int64_t row = t / LPR;
  int sub = (int)(t % LPR);
  double s = 0.0;
  if (row < n)  // no early return: every lane takes part in the shuffles
    for (int64_t q = rp[row] + sub; q < rp[row + 1]; q += LPR) s += v[q] * x[ci[q]];
#pragma unroll
  for (int o = LPR / 2; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o, LPR);
  if (sub == 0 && row < n) y[row] = s;
}

// Up to W entries of a row (`on` of them are there) times V right-hand sides,
// added in order.  All are read before the first is used.  W is the most that
// any row of the warp has, so entries that no row has cost nothing: under a
// condition the compiler keeps the multiply-add and selects, and at 2 of them
// a clock and SM they are what a product with many right-hand sides waits for
// (600^2 with 32: 156 us in rounds of 4 conditional entries).
template <int V, int W>
__device__ __forceinline__ void spmvk_add(double (&s)[V], const int32_t *__restrict__ ci, const double *__restrict__ v,
                                          const double *__restrict__ x, int64_t row, int k, int on) {
  double w[W], xv[W][V];
#pragma unroll
  for (int e = 0; e < W; ++e) {
    const int64_t c = e < on ? ci[e] : row;
    w[e] = e < on ? v[e] : 0.0;
    if (V == 2) {
      const double2 t = *reinterpret_cast<const double2 *>(x + c * k);
      xv[e][0] = t.x, xv[e][V - 1] = t.y;
    } else {
      xv[e][0] = x[c * k];
    }
  }
#pragma unroll
  for (int e = 0; e < W; ++e)
    if (e < on) {
#pragma unroll
      for (int u = 0; u < V; ++u) s[u] += w[e] * xv[e][u];
    }
}

// y = A x for k right-hand sides stored row-major.  A thread owns V (1 or 2)
// neighbouring right-hand sides of a row, k / V threads a row, so every load
// of x and store of y is contiguous across a row's threads; the row's entries
// are read in rounds of up to eight and summed in order.  Bound by FP64
// multiply-adds (2 a clock and SM): 80^3 with 8 takes 60 us, 47 of them for
// its 28.6 M, and a warp per row 193; 600^2 with 2 11 us against 101.
template <int V>
__global__ void __launch_bounds__(256) spmvk_kernel(int64_t n, int k, int rows, const int64_t *__restrict__ rp,
                                                    const int32_t *__restrict__ ci, const double *__restrict__ v,
                                                    const double *__restrict__ x, double *__restrict__ y) {
  const int per_row = k / V, lr = (int)threadIdx.x / per_row, r = ((int)threadIdx.x - lr * per_row) * V;
  const int64_t row = min(blockIdx.x * (int64_t)rows + lr, n - 1);
  const bool mine = lr < rows && blockIdx.x * (int64_t)rows + lr < n;
  const int64_t q0 = rp[row];
  const int len = mine ? (int)(rp[row + 1] - q0) : 0;
  const int most = __reduce_max_sync(0xffffffffu, len);
  ci += q0;
  v += q0;
  x += r;
  double s[V];
#pragma unroll
  for (int u = 0; u < V; ++u) s[u] = 0.0;
  for (int j = 0; j < most; j += 8, ci += 8, v += 8) switch (min(8, most - j)) {
      case 1: spmvk_add<V, 1>(s, ci, v, x, row, k, len - j); break;
      case 2: spmvk_add<V, 2>(s, ci, v, x, row, k, len - j); break;
      case 3: spmvk_add<V, 3>(s, ci, v, x, row, k, len - j); break;
      case 4: spmvk_add<V, 4>(s, ci, v, x, row, k, len - j); break;
      case 5: spmvk_add<V, 5>(s, ci, v, x, row, k, len - j); break;
      case 6: spmvk_add<V, 6>(s, ci, v, x, row, k, len - j); break;
      case 7: spmvk_add<V, 7>(s, ci, v, x, row, k, len - j); break;
      default: spmvk_add<V, 8>(s, ci, v, x, row, k, len - j);
    }
  if (!mine) return;
  if (V == 2) *reinterpret_cast<double2 *>(y + row * k + r) = make_double2(s[0], s[V - 1]);
  else y[row * k + r] = s[0];
}

// Rows of a thread block with `per_row` threads each: as many as 256 threads
// hold, fewer where that leaves over 5% of the last warp's round empty.
int spmvk_rows(int per_row) {
  auto fill = [per_row](int rows) { return (double)(rows * per_row) / ((rows * per_row + 31) / 32 * 32); };
  int rows = 256 / per_row;
  if (fill(rows) >= 0.95) return rows;
  for (int t = rows - 1; t * per_row >= 128; --t)
    if (fill(t) > fill(rows)) rows = t;
  return rows;
}

// The same by one warp per row, lanes over the right-hand sides.
__global__ void __launch_bounds__(256) spmvk_warp_kernel(int64_t n, int k, const int64_t *__restrict__ rp,
                                                         const int32_t *__restrict__ ci, const double *__restrict__ v,
                                                         const double *__restrict__ x, double *__restrict__ y) {
  const int64_t row = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  if (row >= n) return;
  for (int r = threadIdx.x & 31; r < k; r += 32) {
    double s = 0.0;
    for (int64_t q = rp[row]; q < rp[row + 1]; ++q) s += v[q] * x[(int64_t)ci[q] * k + r];
    y[row * k + r] = s;
  }
}

// Whether a warp per row serves k right-hand sides: where at least 7 of 8
// lanes have one.  us, a warp per row / threads with pairs: 600^2 grid k = 26
// 116 / 111, 28 117 / 117, 32 117 / 129, 48 201 / 172, 56 201 / 223, 64
// 201 / 247; 60^3 k = 28 86 / 85, 32 86 / 94, 48 164 / 127, 64 164 / 176.
bool spmvk_by_warps(int k) { return 8 * k >= 7 * ((k + 31) / 32 * 32); }

// W entries of a slice's row, all read before the first gather; even ones to
// s0, odd ones to s1.
template <int W>
__device__ __forceinline__ void sell_add(double &s0, double &s1, const int32_t *__restrict__ ci,
                                         const double *__restrict__ v, const double *__restrict__ x) {
  int32_t c[W];
  double a[W], b[W];
#pragma unroll
  for (int u = 0; u < W; ++u) c[u] = __ldg(ci + 32 * u), a[u] = __ldg(v + 32 * u);
#pragma unroll
  for (int u = 0; u < W; ++u) b[u] = __ldg(&x[c[u]]);
#pragma unroll
  for (int u = 0; u < W; ++u) {
    if (u & 1) s1 += a[u] * b[u];
    else s0 += a[u] * b[u];
  }
}

// y = A x, sliced ELL: one thread per row, each of a warp's loads is one
// contiguous 128/256-byte transaction.  A slice (a warp) reads its entries in
// rounds of eight and a last one of just what is left (six thread blocks an SM
// keep enough of them in flight).  Bound by HBM: 128^3 (226 MB) 39 us, 5.8
// TB/s; with two entries in flight 49, with rounds of eight under conditions
// and their 47 registers 48, where 2D grids, 5 of 8 entries, lost 20 to 40%
// (300^2 4.5 -> 6.3 us, now 4.4).
__global__ void __launch_bounds__(256, 6) spmv_sell_kernel(int64_t n, const int64_t *__restrict__ off,
                                                           const int32_t *__restrict__ ci,
                                                           const double *__restrict__ v,
                                                           const double *__restrict__ x, double *__restrict__ y) {
  const int64_t row = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (row >= n) return;
  const int64_t sl = row >> 5;
  const int64_t o0 = off[sl];
  int w = (int)((off[sl + 1] - o0) >> 5);
  ci += o0 + (row & 31);
  v += o0 + (row & 31);
  double s0 = 0.0, s1 = 0.0;
  for (; w > 8; w -= 8, ci += 256, v += 256) sell_add<8>(s0, s1, ci, v, x);
  switch (w) {
    case 1: sell_add<1>(s0, s1, ci, v, x); break;
    case 2: sell_add<2>(s0, s1, ci, v, x); break;
    case 3: sell_add<3>(s0, s1, ci, v, x); break;
    case 4: sell_add<4>(s0, s1, ci, v, x); break;
    case 5: sell_add<5>(s0, s1, ci, v, x); break;
    case 6: sell_add<6>(s0, s1, ci, v, x); break;
    case 7: sell_add<7>(s0, s1, ci, v, x); break;
    case 8: sell_add<8>(s0, s1, ci, v, x); break;
  }
  y[row] = s0 + s1;
}

void spmv(const rchol_matrix_s &A, const double *x, double *y, int k, cudaStream_t s) {
  const int64_t n = A.n;
  if (k == 1 && A.sell_off.p) {
    spmv_sell_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, A.sell_off.p, A.sell_ci.p, A.sell_v.p, x, y);
    note_launch();
  } else if (k == 1) {
    int64_t threads = n * 8;
    spmv1_kernel<8><<<(unsigned)((threads + 255) / 256), 256, 0, s>>>(n, A.rp.p, A.ci.p, A.v.p, x, y);
    note_launch();
  } else if (spmvk_by_warps(k)) {
    spmvk_warp_kernel<<<(unsigned)((n * 32 + 255) / 256), 256, 0, s>>>(n, k, A.rp.p, A.ci.p, A.v.p, x, y);
    note_launch();
  } else {
    // pairs of right-hand sides where every pair is 16-byte aligned
    const bool pairs = k % 2 == 0 && (reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(y)) % 16 == 0;
    const int per_row = pairs ? k / 2 : k, rows = spmvk_rows(per_row);
    const unsigned grid = (unsigned)((n + rows - 1) / rows), threads = (unsigned)(rows * per_row + 31) / 32 * 32;
    if (pairs) spmvk_kernel<2><<<grid, threads, 0, s>>>(n, k, rows, A.rp.p, A.ci.p, A.v.p, x, y);
    else spmvk_kernel<1><<<grid, threads, 0, s>>>(n, k, rows, A.rp.p, A.ci.p, A.v.p, x, y);
    note_launch();
  }
  RCHOL_CUDA(cudaGetLastError());
}

}  // namespace

void build_sell(rchol_matrix_s &A) {
  const HostCsr &H = A.host;
  const int64_t n = H.n, ns = (n + 31) / 32;
  std::vector<int64_t> off(ns + 1, 0);
  for (int64_t sl = 0; sl < ns; ++sl) {
    int64_t w = 0;
    for (int64_t r = sl * 32; r < std::min(n, sl * 32 + 32); ++r) w = std::max(w, H.rp[r + 1] - H.rp[r]);
    off[sl + 1] = off[sl] + 32 * w;
  }
  std::vector<int32_t> ci(off[ns]);
  std::vector<double> v(off[ns], 0.0);
  parallel_for(ns, [&](int64_t s0, int64_t s1) {
    for (int64_t sl = s0; sl < s1; ++sl) {
      const int64_t w = (off[sl + 1] - off[sl]) / 32;
      for (int t = 0; t < 32; ++t) {
        const int64_t r = sl * 32 + t;
        const int64_t len = r < n ? H.rp[r + 1] - H.rp[r] : 0;
        for (int64_t j = 0; j < w; ++j) {
          const int64_t o = off[sl] + 32 * j + t;
          if (j < len) {
            ci[o] = (int32_t)H.ci[H.rp[r] + j];
            v[o] = H.v[H.rp[r] + j];
          } else {
            ci[o] = (int32_t)std::min<int64_t>(r, n - 1);
            v[o] = 0.0;
          }
        }
      }
    }
  }, 1 << 12);
  A.sell_off.upload(off.data(), ns + 1);
  A.sell_ci.upload(ci.data(), off[ns]);
  A.sell_v.upload(v.data(), off[ns]);
  RCHOL_CUDA(cudaDeviceSynchronize());
}

namespace {

// ---- PCG --------------------------------------------------------------------------
//
// Per right-hand side r the device keeps: bnorm2, rnorm2, rz, rz_prev, pr, pq,
// alpha, beta, active, iters.  Every reduction is deterministic: a fixed grid,
// a fixed per-thread assignment, fixed-shape trees.

constexpr int RED_BLOCKS = 512;
constexpr int RED_THREADS = 256;

struct PcgState {
  double *bnorm2, *rnorm2, *rz, *rz_prev, *pr, *pq, *alpha, *beta;
  int *active, *iters;
  int *any_active;
  double *partial;  // RED_BLOCKS * k * 2
  int k;
  const double *tol;  // in device memory so that a captured graph serves any call
  const int *maxit;
};

enum RedOp { RED_DOT = 0, RED_DOT2 = 1, RED_UPDATE = 2, RED_RESID = 3 };

// Generic per-RHS reduction over rows.  Thread mapping: rhs = t % k,
// row lane = t / k with a power-of-two number of row lanes per block.
template <int OP>
__global__ void __launch_bounds__(RED_THREADS) reduce_kernel(int64_t n, PcgState st, const double *a,
                                                             const double *b, double *c, double *d,
                                                             const double *e) {
  __shared__ double sh[2][RED_THREADS];
  const int k = st.k;
  if (OP != RED_RESID && !*st.any_active) return;
  int lanes = 1;
  while (lanes * 2 * k <= RED_THREADS) lanes *= 2;
  const int t = threadIdx.x;
  const int r = t % k, rl = t / k;
  const bool act_t = (k <= RED_THREADS) && (rl < lanes);
  int64_t per = (n + gridDim.x - 1) / gridDim.x;
  int64_t i0 = blockIdx.x * per, i1 = min(n, i0 + per);
  double s0 = 0.0, s1 = 0.0;
  if (act_t) {
    if (OP == RED_DOT) {  // s0 = a.b
      for (int64_t i = i0 + rl; i < i1; i += lanes) s0 += a[i * k + r] * b[i * k + r];
    } else if (OP == RED_DOT2) {  // s0 = a.b, s1 = a.e  (p.q and p.r)
      for (int64_t i = i0 + rl; i < i1; i += lanes) {
        double pv = a[i * k + r];
        s0 += pv * b[i * k + r];
        s1 += pv * e[i * k + r];
      }
    } else if (OP == RED_UPDATE) {  // x += alpha p ; r -= alpha q ; s0 = r.r
      double al = st.active[r] ? st.alpha[r] : 0.0;
      bool on = st.active[r];
      for (int64_t i = i0 + rl; i < i1; i += lanes) {
        int64_t o = i * k + r;
        double rv = d[o];
        if (on) {
          c[o] += al * a[o];
          rv += -al * b[o];
          d[o] = rv;
        }
        s0 += rv * rv;
      }
    } else {  // RED_RESID: s0 = (a - b).(a - b)  with a = A x, b = rhs
      for (int64_t i = i0 + rl; i < i1; i += lanes) {
        double q = a[i * k + r] + -1.0 * b[i * k + r];
        s0 += q * q;
      }
    }
  }
  sh[0][t] = s0;
  sh[1][t] = s1;
  __syncthreads();
  for (int h = lanes / 2; h > 0; h >>= 1) {
    if (act_t && rl < h) {
      sh[0][t] += sh[0][t + h * k];
      sh[1][t] += sh[1][t + h * k];
    }
    __syncthreads();
  }
  if (act_t && rl == 0) {
    st.partial[(int64_t)blockIdx.x * k + r] = sh[0][t];
    st.partial[(int64_t)(gridDim.x + blockIdx.x) * k + r] = sh[1][t];
  }
}

// Sum the RED_BLOCKS partials of every rhs (one block per rhs, fixed tree).
__device__ double block_total(const double *part, int k, int r, int which) {
  __shared__ double sh[RED_THREADS];
  double s = 0.0;
  for (int bb = threadIdx.x; bb < RED_BLOCKS; bb += RED_THREADS)
    s += part[(int64_t)(which * RED_BLOCKS + bb) * k + r];
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int h = RED_THREADS / 2; h > 0; h >>= 1) {
    if (threadIdx.x < h) sh[threadIdx.x] += sh[threadIdx.x + h];
    __syncthreads();
  }
  double tot = sh[0];
  __syncthreads();
  return tot;
}

enum FinOp { FIN_INIT = 0, FIN_BETA = 1, FIN_ALPHA = 2, FIN_CONV = 3, FIN_RESID = 4 };

__global__ void finalize_kernel(PcgState st, int op, int first, double *relres) {
  const int r = blockIdx.x;
  if (op != FIN_INIT && op != FIN_RESID && !*st.any_active) return;
  double t0 = block_total(st.partial, st.k, r, 0);
  double t1 = block_total(st.partial, st.k, r, 1);
  if (threadIdx.x != 0) return;
  if (op == FIN_INIT) {  // t0 = b.b (r = b)
    st.bnorm2[r] = t0;
    st.rnorm2[r] = t0;
    st.iters[r] = 0;
    int act = (sqrt(t0) > sqrt(t0) * *st.tol) && (*st.maxit > 0);
    st.active[r] = act;
    if (act) atomicOr(st.any_active, 1);
  } else if (op == FIN_BETA) {  // t0 = r.z
    if (st.active[r]) {
      st.beta[r] = st.iters[r] == 0 ? 0.0 : t0 / st.rz_prev[r];
      st.rz[r] = t0;
    }
  } else if (op == FIN_ALPHA) {  // t0 = p.q, t1 = p.r
    if (st.active[r]) {
      st.pq[r] = t0;
      st.pr[r] = t1;
      st.alpha[r] = t1 / t0;
    }
  } else if (op == FIN_CONV) {  // t0 = r.r after the update
    if (st.active[r]) {
      st.rnorm2[r] = t0;
      st.rz_prev[r] = st.rz[r];
      int it = st.iters[r] + 1;
      st.iters[r] = it;
      st.active[r] = (sqrt(t0) > sqrt(st.bnorm2[r]) * *st.tol) && (it < *st.maxit);
    }
  } else {  // FIN_RESID
    relres[r] = sqrt(t0) / sqrt(st.bnorm2[r]);
  }
}

__global__ void any_active_kernel(PcgState st) {
  int a = 0;
  for (int r = 0; r < st.k; ++r) a |= st.active[r];
  *st.any_active = a;
}

// p = beta p + z (p = z on the first iteration), only for active right-hand sides.
__global__ void pupdate_kernel(int64_t nk, PcgState st, double *p, const double *z) {
  if (!*st.any_active) return;
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= nk) return;
  int r = (int)(i % st.k);
  if (!st.active[r]) return;
  if (st.iters[r] == 0) p[i] = z[i];
  else p[i] = st.beta[r] * p[i] + 1.0 * z[i];
}

__global__ void init_kernel(int64_t nk, const double *b, double *x, double *r) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= nk) return;
  x[i] = 0.0;
  r[i] = b[i];
}

}  // namespace

// ---- plan construction -----------------------------------------------------------

namespace {

__global__ void transpose_count_kernel(int64_t nnz, const int32_t *uci, unsigned long long *cnt) {
  int64_t q = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (q < nnz) atomicAdd(&cnt[uci[q]], 1ull);
}

__global__ void transpose_scatter_kernel(int64_t n, const int64_t *urp, const int32_t *uci,
                                         const double *uv, const int64_t *lrp,
                                         unsigned long long *cur, int32_t *tci, double *tv) {
  int64_t row = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  int lane = threadIdx.x & 31;
  if (row >= n) return;
  for (int64_t q = urp[row] + lane; q < urp[row + 1]; q += 32) {
    int32_t j = uci[q];
    unsigned long long slot = atomicAdd(&cur[j], 1ull);
    tci[lrp[j] + slot] = (int32_t)row;
    tv[lrp[j] + slot] = uv[q];
  }
}

// Sort each row of L by column (rank sort; columns within a row are unique).
__global__ void row_sort_kernel(int64_t n, const int64_t *lrp, const int32_t *tci, const double *tv,
                                int32_t *lci, double *lv) {
  int64_t row = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
  int lane = threadIdx.x & 31;
  if (row >= n) return;
  int64_t b = lrp[row], e = lrp[row + 1];
  for (int64_t q = b + lane; q < e; q += 32) {
    int32_t c = tci[q];
    int64_t rank = 0;
    for (int64_t f = b; f < e; ++f) rank += (tci[f] < c);
    lci[b + rank] = c;
    lv[b + rank] = tv[q];
  }
}


__global__ void to_f32_kernel(int64_t n, const double *a, float *b) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) b[i] = (float)a[i];
}

__global__ void i64_from_ull_kernel(int64_t n, const unsigned long long *a, int64_t *b) {
  int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) b[i] = (int64_t)a[i];
}

}  // namespace

void finish_factor(rchol_factor_s &F, cudaStream_t s) {
  const int64_t n = F.n, nnz = F.nnz;
  const auto t0 = std::chrono::steady_clock::now();
  // L = transpose(U)
  DevBuf<unsigned long long> cnt(n);
  RCHOL_CUDA(cudaMemsetAsync(cnt.p, 0, cnt.bytes(), s));
  transpose_count_kernel<<<(unsigned)((nnz + 255) / 256), 256, 0, s>>>(nnz, F.uci.p, cnt.p);
  note_launch();
  F.lrp.alloc(n + 1);
  i64_from_ull_kernel<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, cnt.p, F.lrp.p);
  note_launch();
  RCHOL_CUDA(cudaGetLastError());
  exclusive_scan_i64(F.lrp.p, n, s);
  RCHOL_CUDA(cudaMemsetAsync(cnt.p, 0, cnt.bytes(), s));
  {
    DevBuf<int32_t> tci(nnz);
    DevBuf<double> tv(nnz);
    transpose_scatter_kernel<<<(unsigned)((n * 32 + 255) / 256), 256, 0, s>>>(
        n, F.urp.p, F.uci.p, F.uv.p, F.lrp.p, cnt.p, tci.p, tv.p);
    note_launch();
    F.lci.alloc(nnz);
    F.lv.alloc(nnz);
    row_sort_kernel<<<(unsigned)((n * 32 + 255) / 256), 256, 0, s>>>(n, F.lrp.p, tci.p, tv.p, F.lci.p,
                                                                      F.lv.p);
    note_launch();
    RCHOL_CUDA(cudaGetLastError());
    RCHOL_CUDA(cudaStreamSynchronize(s));
  }
  if (F.precision == RCHOL_PREC_FP32) {
    F.uv32.alloc(nnz);
    F.lv32.alloc(nnz);
    to_f32_kernel<<<(unsigned)((nnz + 255) / 256), 256, 0, s>>>(nnz, F.uv.p, F.uv32.p);
    note_launch();
    to_f32_kernel<<<(unsigned)((nnz + 255) / 256), 256, 0, s>>>(nnz, F.lv.p, F.lv32.p);
    note_launch();
    RCHOL_CUDA(cudaGetLastError());
  }
  RCHOL_CUDA(cudaStreamSynchronize(s));
  const auto t1 = std::chrono::steady_clock::now();
  build_plan(F, s);
  RCHOL_CUDA(cudaStreamSynchronize(s));
  F.t_assemble = std::chrono::duration<double>(t1 - t0).count();
  F.t_plan = std::chrono::duration<double>(std::chrono::steady_clock::now() - t1).count();
}

void build_plan(rchol_factor_s &F, cudaStream_t s) {
  auto P = new SolvePlan();
  try {
    P->status = solve_status_word();
    // rchol_gpu_trsv_d and rchol_gpu_precond_d run in large blocks (blocks.cu)
    // where G allows it and RCHOL_TRSV_FORMAT does not ask for one of trsv.cu's
    // record formats.  The PCG loops always apply the record streams: CG
    // amplifies the rounding of the preconditioner, so another order of its
    // sums changes iteration counts (of 40 FP32 systems solved to 1e-8 five
    // took an iteration more or less, of 15 FP64 ones two, with x off by
    // 2e-9), and the same program has to give the same iterates as ever.  Both
    // plans are built at once, the records by the host's threads and the
    // blocks by the GPU.  Where memory is too short for that, the streams are
    // built alone and the block plan after them if it still fits.
    const bool wanted = !getenv("RCHOL_TRSV_FORMAT");
    BlkBuilt built = BlkBuilt::kLeftOut;
    std::future<BlkBuilt> other;
    if (wanted) {
      int dev = 0;
      RCHOL_CUDA(cudaGetDevice(&dev));
      other = std::async(std::launch::async, [&F, P, s, dev] {
        RCHOL_CUDA(cudaSetDevice(dev));
        return build_blocks(F, *P, s);
      });
    }
    try {
      build_streams(F, *P, s);
      if (wanted) built = other.get();
    } catch (const Error &e) {
      if (!wanted || e.status != RCHOL_ERR_NOMEM) throw;
      if (other.valid()) other.wait();
      P->bfwd = BlkDir();
      P->bbwd = BlkDir();
      P->sfwd = StreamDir();
      P->sbwd = StreamDir();
      build_streams(F, *P, s);
      built = BlkBuilt::kNoMemory;
    }
    if (built == BlkBuilt::kNoMemory) built = build_blocks(F, *P, s);
    P->blocked = built == BlkBuilt::kReady;
    P->blocked1 = P->blocked && blocks_for_one(F, *P);
  } catch (...) {
    delete P;
    throw;
  }
  destroy_plan(F.plan);
  F.plan = P;
}

// Grows PCG's intermediate vector.  Growing frees a buffer that captured PCG
// graphs point to, so every cached graph of this factor is dropped with it
// (a replay would otherwise read and write freed memory).  Callers hold P.lock.
static void ensure_scratch(SolvePlan &P, bool fp32, int64_t count) {
  bool grew = false;
  if (fp32) {
    if (P.ytmp32.n < (size_t)count) P.ytmp32.alloc(count), grew = true;
  } else {
    if (P.ytmp.n < (size_t)count) P.ytmp.alloc(count), grew = true;
  }
  if (grew) {
    P.pcg.clear();
    P.seg.clear();
  }
}

// One right-hand side, in large blocks or by the record streams.  acc: n
// values of G's precision.
static void trsv_one(const rchol_factor_s &F, const SolvePlan &P, bool blocks, bool upper, const double *in64,
                     const float *in32, double *out64, float *out32, void *acc, cudaStream_t s) {
  if (blocks) block_trsv(F, P, upper, in64, in32, out64, out32, acc, 1, s);
  else stream_trsv(F, P, upper, in64, in32, out64, out32, acc, s);
}

// z = (G G^T)^-1 r with the intermediate vector in y64 or y32.
static void precond_one(const rchol_factor_s &F, const SolvePlan &P, bool blocks, const double *r, double *z,
                        double *y64, float *y32, void *acc, cudaStream_t s) {
  trsv_one(F, P, blocks, false, r, nullptr, y64, y32, acc, s);
  trsv_one(F, P, blocks, true, y64, y32, z, nullptr, acc, s);
}

// The plan's partial-sum vector, sized for n values.
static void *ensure_acc(SolvePlan &P, bool fp32, int64_t n) {
  if (fp32) {
    if (P.acc32.n < (size_t)n) P.acc32.alloc(n);
    return P.acc32.p;
  }
  if (P.acc64.n < (size_t)n) P.acc64.alloc(n);
  return P.acc64.p;
}

// What PCG needs for k right-hand sides.
static void ensure_pcg(const rchol_factor_s &F, int k, cudaStream_t s) {
  SolvePlan &P = *F.plan;
  const bool fp32 = F.precision == RCHOL_PREC_FP32;
  ensure_scratch(P, fp32, F.n * k);
  if (k == 1) ensure_acc(P, fp32, F.n);
  else build_streams_k(F, P, s);
}

// What trsv and precond need for k right-hand sides on the block plan or the
// record streams: accumulator and workspace.  Columns come in a power of two.
// A workspace that is grown out of stays until the factor goes, because a
// caller's graph of a solve with fewer columns holds its addresses (all of
// them together are smaller than the last); PCG does not share them.
static const SolveWork &ensure_work(const rchol_factor_s &F, bool blocks, int k, cudaStream_t s) {
  SolvePlan &P = *F.plan;
  const bool fp32 = F.precision == RCHOL_PREC_FP32;
  const size_t n = (size_t)F.n;
  if (k == 1) {
    ensure_acc(P, fp32, F.n);
  } else if (blocks) {
    build_blocks_k(F, P, std::min(k, kBlkCols), s);
    if (fp32 && P.acck32.n < n * kBlkCols) P.acck32.alloc(n * kBlkCols);
    if (!fp32 && P.acck64.n < n * kBlkCols) P.acck64.alloc(n * kBlkCols);
  } else {
    build_streams_k(F, P, s);
  }
  const int need = blocks ? std::min(k, kBlkCols) : k;
  int cols = 1;
  while (cols < need) cols *= 2;
  if (P.work.empty() || P.work.back().cols < cols) {
    SolveWork w;
    w.cols = cols;
    if (fp32) w.y32.alloc(n * cols);
    else w.y64.alloc(n * cols);
    if (blocks && k > 1) w.a.alloc(n * cols), w.b.alloc(n * cols);
    P.work.push_back(std::move(w));
  }
  return P.work.back();
}

// Columns j0 .. j0 + g of an n x k row-major array, one after another
// (TO_COLS), or back.  A thread block moves 64 rows through shared memory, so
// both sides are read and written in runs.
template <bool TO_COLS>
__global__ void __launch_bounds__(256) blk_columns_kernel(int64_t n, int k, int j0, int g, const double *__restrict__ in,
                                                          double *__restrict__ out) {
  __shared__ double tile[64][kBlkCols + 1];
  const int64_t r0 = blockIdx.x * (int64_t)64;
  const int rows = (int)min((int64_t)64, n - r0);
  for (int e = threadIdx.x; e < 64 * g; e += 256) {
    const int r = TO_COLS ? e / g : e & 63, c = TO_COLS ? e - r * g : e >> 6;
    if (r < rows) tile[r][c] = TO_COLS ? in[(r0 + r) * k + j0 + c] : in[c * n + r0 + r];
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 64 * g; e += 256) {
    const int r = TO_COLS ? e & 63 : e / g, c = TO_COLS ? e >> 6 : e - r * g;
    if (r >= rows) continue;
    if (TO_COLS) out[c * n + r0 + r] = tile[r][c];
    else out[(r0 + r) * k + j0 + c] = tile[r][c];
  }
}

template <bool TO_COLS>
static void move_columns(int64_t n, int k, int j0, int g, const double *in, double *out, cudaStream_t s) {
  blk_columns_kernel<TO_COLS><<<(unsigned)((n + 63) / 64), 256, 0, s>>>(n, k, j0, g, in, out);
  note_launch();
  RCHOL_CUDA(cudaGetLastError());
}

// k right-hand sides (n x k row-major) on the block plan, up to kBlkCols
// columns at a time: the solve of direction `dir` (0, 1) or the preconditioner (2).
static void blocks_k(const rchol_factor_s &F, const SolvePlan &P, const SolveWork &w, int dir, const double *in,
                     double *out, int k, cudaStream_t s) {
  const int64_t n = F.n;
  const bool fp32 = F.precision == RCHOL_PREC_FP32;
  void *acc = fp32 ? (void *)P.acck32.p : (void *)P.acck64.p;
  double *a = w.a.p, *b = w.b.p;
  for (int j0 = 0; j0 < k; j0 += kBlkCols) {
    const int g = std::min(kBlkCols, k - j0);
    move_columns<true>(n, k, j0, g, in, a, s);
    if (dir < 2) {
      block_trsv(F, P, dir == 1, a, nullptr, b, nullptr, acc, g, s);
    } else if (fp32) {
      block_trsv(F, P, false, a, nullptr, nullptr, w.y32.p, acc, g, s);
      block_trsv(F, P, true, nullptr, w.y32.p, b, nullptr, acc, g, s);
    } else {
      block_trsv(F, P, false, a, nullptr, w.y64.p, nullptr, acc, g, s);
      block_trsv(F, P, true, w.y64.p, nullptr, b, nullptr, acc, g, s);
    }
    move_columns<false>(n, k, j0, g, b, out, s);
  }
}

// The preconditioner by the record streams with the intermediate vector(s) in
// y64 or y32, everything sized already.
static void precond_streams(const rchol_factor_s &F, const double *r, double *z, double *y64, float *y32, int k,
                            cudaStream_t s) {
  SolvePlan &P = *F.plan;
  const bool fp32 = F.precision == RCHOL_PREC_FP32;
  if (k == 1) {
    precond_one(F, P, false, r, z, y64, y32, ensure_acc(P, fp32, F.n), s);
  } else if (fp32) {
    stream_trsv_k(F, P, false, r, nullptr, nullptr, y32, k, s);
    stream_trsv_k(F, P, true, nullptr, y32, z, nullptr, k, s);
  } else {
    stream_trsv_k(F, P, false, r, nullptr, y64, nullptr, k, s);
    stream_trsv_k(F, P, true, y64, nullptr, z, nullptr, k, s);
  }
}

void trsv(const rchol_factor_s &F, bool upper, const double *in, double *out, int k, cudaStream_t s) {
  SolvePlan &P = *F.plan;
  std::lock_guard<std::mutex> guard(P.lock);
  const bool blocks = k == 1 ? P.blocked1 : P.blocked;
  const SolveWork &w = ensure_work(F, blocks, k, s);
  if (k == 1) trsv_one(F, P, blocks, upper, in, nullptr, out, nullptr, ensure_acc(P, F.precision == RCHOL_PREC_FP32, F.n), s);
  else if (blocks) blocks_k(F, P, w, upper, in, out, k, s);
  else stream_trsv_k(F, P, upper, in, nullptr, out, nullptr, k, s);
}

void precond(const rchol_factor_s &F, const double *r, double *z, int k, cudaStream_t s) {
  SolvePlan &P = *F.plan;
  std::lock_guard<std::mutex> guard(P.lock);
  const bool blocks = k == 1 ? P.blocked1 : P.blocked;
  const SolveWork &w = ensure_work(F, blocks, k, s);
  if (!blocks) precond_streams(F, r, z, w.y64.p, w.y32.p, k, s);
  else if (k == 1) precond_one(F, P, true, r, z, w.y64.p, w.y32.p, ensure_acc(P, F.precision == RCHOL_PREC_FP32, F.n), s);
  else blocks_k(F, P, w, 2, r, z, k, s);
}

// ---- preconditioner apply without allocation --------------------------------------------
//
// Some callers cannot allocate device memory at solve time: code that runs
// under a fixed memory budget decided at start-up, allocator-free real-time
// loops, or hosts that own all device memory themselves.  For them the
// preconditioner z = (G G^T)^-1 r can run with its two scratch vectors (the
// partial sums and the intermediate y = G^-1 r) in this fixed, file-scope
// device array instead of buffers allocated with the factor's plan.  Every
// GPU that loads the library holds the array until the process exits.
// The array is shared by all calls and keeps the last call's contents; nothing
// in it has to start at zero (both vectors are fully written before they are
// read), and calls that overlap on the GPU race on it.
constexpr size_t kNoAllocScratchBytes = size_t(16) << 20;  // 16 MiB
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

namespace {
constexpr size_t up16(size_t x) { return (x + 15) & ~size_t(15); }
constexpr int kNoAllocDevices = 128;
std::mutex g_noalloc_mutex;
void *g_noalloc_ptr[kNoAllocDevices] = {};  // device address of the array, per device ordinal
}  // namespace

size_t noalloc_scratch_bytes() { return kNoAllocScratchBytes; }

// Set-up on the current device: the array's host-side name is only a
// stand-in, so its device address is looked up with the device current.  The
// first call on a device does this (it should come before any stream
// capture); later calls whose stream is not capturing look it up again, so a
// device reset (which gives the array a new address) leaves no stale pointer.
static void *noalloc_scratch_address(cudaStream_t s) {
  int dev = 0;
  RCHOL_CUDA(cudaGetDevice(&dev));
  RCHOL_CHECK_ARG(dev >= 0 && dev < kNoAllocDevices, "device ordinal out of range");
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &cs) != cudaSuccess) {
    (void)cudaGetLastError();  // e.g. the legacy stream while another stream captures
    cs = cudaStreamCaptureStatusActive;
  }
  std::lock_guard<std::mutex> guard(g_noalloc_mutex);
  if (!g_noalloc_ptr[dev] || cs == cudaStreamCaptureStatusNone) {
    void *p = nullptr;
    RCHOL_CUDA(cudaGetSymbolAddress(&p, g_noalloc_scratch));
    g_noalloc_ptr[dev] = p;
  }
  return g_noalloc_ptr[dev];
}

void precond_noalloc(const rchol_factor_s &F, const double *r, double *z, cudaStream_t s) {
  const int64_t n = F.n;
  const bool fp32 = F.precision == RCHOL_PREC_FP32;
  const size_t vsz = fp32 ? 4 : 8;
  const size_t acc_bytes = up16((size_t)n * vsz);
  if (2 * acc_bytes > kNoAllocScratchBytes)
    throw Error(RCHOL_ERR_INVALID, "n = " + std::to_string(n) + " needs " + std::to_string(2 * acc_bytes) +
                                       " bytes of scratch; the allocation-free entry point has " +
                                       std::to_string(kNoAllocScratchBytes) + " (n <= " +
                                       std::to_string(kNoAllocScratchBytes / (2 * vsz)) + " for this precision)");
  unsigned char *base = static_cast<unsigned char *>(noalloc_scratch_address(s));
  void *y = base + acc_bytes;
  precond_one(F, *F.plan, F.plan->blocked1, r, z, fp32 ? nullptr : static_cast<double *>(y),
              fp32 ? static_cast<float *>(y) : nullptr, base, s);
}

void spmv_public(const rchol_matrix_s &A, const double *x, double *y, int k, cudaStream_t s) {
  spmv(A, x, y, k, s);
}

namespace {
// dL/dw_e = -(lambda_i - lambda_j)(x_i - x_j): the derivative of -lambda^T A(w) x
// with respect to one edge weight.
__global__ void edge_grad_kernel(int64_t m, const int64_t *__restrict__ ei, const int64_t *__restrict__ ej,
                                 const double *__restrict__ lam, const double *__restrict__ x,
                                 double *__restrict__ g) {
  const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (e >= m) return;
  const int64_t i = ei[e], j = ej[e];
  g[e] = -(lam[i] - lam[j]) * (x[i] - x[j]);
}
}  // namespace

void edge_grad(int64_t m, const int64_t *ei, const int64_t *ej, const double *lam, const double *x, double *g,
               cudaStream_t s) {
  if (m <= 0) return;
  edge_grad_kernel<<<(unsigned)((m + 255) / 256), 256, 0, s>>>(m, ei, ej, lam, x, g);
  note_launch();
  RCHOL_CUDA(cudaGetLastError());
}

// Longest dependency chain (levels of a level schedule) of the forward or
// backward solve, computed on first request from the CSR of G or G^T.
int64_t plan_levels(const rchol_factor_s &F, bool upper) {
  SolvePlan &P = *F.plan;
  std::lock_guard<std::mutex> guard(P.lock);
  int64_t &dag = upper ? P.dag_bwd : P.dag_fwd;
  if (dag >= 0) return dag;
  const int64_t n = F.n, nnz = F.nnz;
  std::vector<int64_t> rp(n + 1);
  std::vector<int32_t> ci(nnz);
  (upper ? F.urp : F.lrp).download(rp.data(), n + 1, 0);
  (upper ? F.uci : F.lci).download(ci.data(), nnz, 0);
  RCHOL_CUDA(cudaStreamSynchronize(0));
  std::vector<int32_t> lv(n, 0);
  int32_t mx = 0;
  if (!upper) {  // rows of G: diagonal last
    for (int64_t i = 0; i < n; ++i) {
      int32_t l = 0;
      for (int64_t q = rp[i]; q < rp[i + 1] - 1; ++q) l = std::max(l, lv[ci[q]] + 1);
      lv[i] = l;
      mx = std::max(mx, l);
    }
  } else {  // rows of G^T: diagonal first
    for (int64_t i = n - 1; i >= 0; --i) {
      int32_t l = 0;
      for (int64_t q = rp[i] + 1; q < rp[i + 1]; ++q) l = std::max(l, lv[ci[q]] + 1);
      lv[i] = l;
      mx = std::max(mx, l);
    }
  }
  dag = n ? (int64_t)mx + 1 : 0;
  return dag;
}

// PCG for k right-hand sides (device pointers), c++/util/pcg.cpp:57-127.
//
// One iteration (preconditioner, r.z, p update, SpMV with p.q and p.r, x/r
// update with ||r||^2, stopping test) is captured once per (matrix, factor, k)
// into a CUDA graph and replayed; every kernel returns at once when no
// right-hand side is active any more, so the host checks convergence only
// every few iterations.  The graph runs on the workspace's own stream, joined
// to the caller's stream with events.
static PcgWork &pcg_workspace(const rchol_matrix_s &A, const rchol_factor_s &F, int k) {
  SolvePlan &P = *F.plan;
  for (auto &w : P.pcg)
    if (w->key_uid == A.uid && w->n == A.n && w->nnz == A.nnz && w->k == k)
      return *w;
  if (P.pcg.size() >= 4) P.pcg.erase(P.pcg.begin());
  auto w = std::make_unique<PcgWork>();
  w->key_uid = A.uid;
  w->n = A.n;
  w->nnz = A.nnz;
  w->k = k;
  const int64_t nk = A.n * k;
  w->r.alloc(nk);
  w->z.alloc(nk);
  w->p.alloc(nk);
  w->q.alloc(nk);
  w->x.alloc(nk);
  w->sc.alloc(9 * (size_t)k + 2 * (size_t)RED_BLOCKS * k + 1);
  w->ic.alloc(2 * (size_t)k + 2);
  RCHOL_CUDA(cudaStreamCreateWithFlags(&w->stream, cudaStreamNonBlocking));
  RCHOL_CUDA(cudaEventCreateWithFlags(&w->ev_in, cudaEventDisableTiming));
  RCHOL_CUDA(cudaEventCreateWithFlags(&w->ev_out, cudaEventDisableTiming));
  P.pcg.push_back(std::move(w));
  return *P.pcg.back();
}

static PcgState pcg_state(PcgWork &w) {
  const int k = w.k;
  PcgState st;
  double *sc = w.sc.p;
  st.bnorm2 = sc;
  st.rnorm2 = sc + k;
  st.rz = sc + 2 * k;
  st.rz_prev = sc + 3 * k;
  st.pr = sc + 4 * k;
  st.pq = sc + 5 * k;
  st.alpha = sc + 6 * k;
  st.beta = sc + 7 * k;
  st.partial = sc + 8 * k;
  // [8k, 8k + 2*RB*k) partial sums, then k relres slots, then tol
  st.tol = sc + 9 * k + 2 * (size_t)RED_BLOCKS * k;
  st.active = w.ic.p;
  st.iters = w.ic.p + k;
  st.any_active = w.ic.p + 2 * k;
  st.maxit = w.ic.p + 2 * k + 1;
  st.k = k;
  return st;
}

static void pcg_iteration(const rchol_matrix_s &A, const rchol_factor_s &F, PcgWork &w, const PcgState &st,
                          cudaStream_t s) {
  const int k = w.k;
  const int64_t n = A.n, nk = n * k;
  const unsigned eb = (unsigned)((nk + 255) / 256);
  precond_streams(F, w.r.p, w.z.p, F.plan->ytmp.p, F.plan->ytmp32.p, k, s);
  reduce_kernel<RED_DOT><<<RED_BLOCKS, RED_THREADS, 0, s>>>(n, st, w.r.p, w.z.p, nullptr, nullptr, nullptr);
  finalize_kernel<<<k, RED_THREADS, 0, s>>>(st, FIN_BETA, 0, nullptr);
  pupdate_kernel<<<eb, 256, 0, s>>>(nk, st, w.p.p, w.z.p);
  spmv(A, w.p.p, w.q.p, k, s);
  reduce_kernel<RED_DOT2><<<RED_BLOCKS, RED_THREADS, 0, s>>>(n, st, w.p.p, w.q.p, nullptr, nullptr, w.r.p);
  finalize_kernel<<<k, RED_THREADS, 0, s>>>(st, FIN_ALPHA, 0, nullptr);
  reduce_kernel<RED_UPDATE><<<RED_BLOCKS, RED_THREADS, 0, s>>>(n, st, w.p.p, w.q.p, w.x.p, w.r.p, nullptr);
  finalize_kernel<<<k, RED_THREADS, 0, s>>>(st, FIN_CONV, 0, nullptr);
  any_active_kernel<<<1, 1, 0, s>>>(st);
  RCHOL_CUDA(cudaGetLastError());
}

// b_host / x_host: the host-buffer entry point (b copied in and x copied out
// on the workspace stream, through device staging kept with the workspace).
static void pcg_impl(const rchol_matrix_s &A, const rchol_factor_s &F, const double *b, double *x,
                     const double *b_host, double *x_host, int k, double tol, int maxit, double *relres,
                     int *itr, cudaStream_t s) {
  SolvePlan &P = *F.plan;
  std::lock_guard<std::mutex> guard(P.lock);
  const int64_t n = A.n, nk = n * k;
  ensure_pcg(F, k, s);
  PcgWork &w = pcg_workspace(A, F, k);
  PcgState st = pcg_state(w);
  cudaStream_t ws = w.stream;
  RCHOL_CUDA(cudaEventRecord(w.ev_in, s));
  RCHOL_CUDA(cudaStreamWaitEvent(ws, w.ev_in, 0));
  if (b_host) {
    if (w.hb.n < (size_t)nk) w.hb.alloc(nk);
    if (w.hx.n < (size_t)nk) w.hx.alloc(nk);
    RCHOL_CUDA(cudaMemcpyAsync(w.hb.p, b_host, nk * sizeof(double), cudaMemcpyHostToDevice, ws));
    b = w.hb.p;
    x = w.hx.p;
  }
  if (!w.exec) {
    cudaGraph_t g = nullptr;
    RCHOL_CUDA(cudaStreamBeginCapture(ws, cudaStreamCaptureModeThreadLocal));
    try {
      pcg_iteration(A, F, w, st, ws);
    } catch (...) {
      cudaStreamEndCapture(ws, &g);
      if (g) cudaGraphDestroy(g);
      throw;
    }
    RCHOL_CUDA(cudaStreamEndCapture(ws, &g));
    size_t nodes = 0;
    RCHOL_CUDA(cudaGraphGetNodes(g, nullptr, &nodes));
    w.graph_kernels = (int64_t)nodes;
    cudaError_t e = cudaGraphInstantiate(&w.exec, g, 0);
    cudaGraphDestroy(g);
    RCHOL_CUDA(e);
  }
  // setup: tolerances, x = 0, r = b, ||b||^2 and the initial stopping test
  double htol = tol;
  int hmax = maxit;
  RCHOL_CUDA(cudaMemsetAsync(w.sc.p, 0, w.sc.bytes(), ws));
  RCHOL_CUDA(cudaMemsetAsync(w.ic.p, 0, w.ic.bytes(), ws));
  RCHOL_CUDA(cudaMemcpyAsync(const_cast<double *>(st.tol), &htol, sizeof(double), cudaMemcpyHostToDevice, ws));
  RCHOL_CUDA(cudaMemcpyAsync(const_cast<int *>(st.maxit), &hmax, sizeof(int), cudaMemcpyHostToDevice, ws));
  const unsigned eb = (unsigned)((nk + 255) / 256);
  init_kernel<<<eb, 256, 0, ws>>>(nk, b, w.x.p, w.r.p);
  RCHOL_CUDA(cudaMemsetAsync(w.q.p, 0, w.q.bytes(), ws));
  reduce_kernel<RED_RESID><<<RED_BLOCKS, RED_THREADS, 0, ws>>>(n, st, b, w.q.p, nullptr, nullptr, nullptr);
  finalize_kernel<<<k, RED_THREADS, 0, ws>>>(st, FIN_INIT, 0, nullptr);
  note_launch(3);
  RCHOL_CUDA(cudaGetLastError());
  int h_any = 1;
  for (int it = 0; it < maxit;) {
    const int batch = it == 0 ? 8 : 4;
    for (int j = 0; j < batch && it < maxit; ++j, ++it) {
      RCHOL_CUDA(cudaGraphLaunch(w.exec, ws));
      note_launch(w.graph_kernels);
    }
    RCHOL_CUDA(cudaMemcpyAsync(&h_any, st.any_active, sizeof(int), cudaMemcpyDeviceToHost, ws));
    RCHOL_CUDA(cudaStreamSynchronize(ws));
    if (!h_any) break;
  }
  // x out, relres = ||A x - b|| / ||b||
  double *d_relres = w.sc.p + 8 * (size_t)k + 2 * (size_t)RED_BLOCKS * k;
  spmv(A, w.x.p, w.q.p, k, ws);
  reduce_kernel<RED_RESID><<<RED_BLOCKS, RED_THREADS, 0, ws>>>(n, st, w.q.p, b, nullptr, nullptr, nullptr);
  finalize_kernel<<<k, RED_THREADS, 0, ws>>>(st, FIN_RESID, 0, d_relres);
  note_launch(3);
  RCHOL_CUDA(cudaGetLastError());
  if (x_host) RCHOL_CUDA(cudaMemcpyAsync(x_host, w.x.p, nk * sizeof(double), cudaMemcpyDeviceToHost, ws));
  else RCHOL_CUDA(cudaMemcpyAsync(x, w.x.p, nk * sizeof(double), cudaMemcpyDeviceToDevice, ws));
  RCHOL_CUDA(cudaMemcpyAsync(relres, d_relres, k * sizeof(double), cudaMemcpyDeviceToHost, ws));
  RCHOL_CUDA(cudaMemcpyAsync(itr, st.iters, k * sizeof(int), cudaMemcpyDeviceToHost, ws));
  RCHOL_CUDA(cudaEventRecord(w.ev_out, ws));
  RCHOL_CUDA(cudaStreamWaitEvent(s, w.ev_out, 0));
  RCHOL_CUDA(cudaStreamSynchronize(ws));
}

void pcg_device(const rchol_matrix_s &A, const rchol_factor_s &F, const double *b, double *x, int k, double tol,
                int maxit, double *relres, int *itr, cudaStream_t s) {
  pcg_impl(A, F, b, x, nullptr, nullptr, k, tol, maxit, relres, itr, s);
}

void pcg_host(const rchol_matrix_s &A, const rchol_factor_s &F, const double *b, double *x, int k, double tol,
              int maxit, double *relres, int *itr) {
  pcg_impl(A, F, nullptr, nullptr, b, x, k, tol, maxit, relres, itr, 0);
}

// ---- batched PCG over independent systems ---------------------------------------------
//
// The systems are the diagonal blocks of one matrix (rows seg[s] .. seg[s+1])
// with a block-diagonal factor, so one SpMV and one preconditioner apply serve
// them all; the scalars of c++/util/pcg.cpp:57-127 are kept per system, and a
// system stops updating once it has converged.  A system's sum is 256 chains
// over rows 256 apart and a fixed tree over them (so results are
// deterministic).  Inside the iteration a warp owns 32 of the chains: a system
// is spread over 8 warps, which may sit on different SMs, each reads 24 rows
// of its chains ahead, and every kernel that needs a total redoes the tree.  With one
// thread block per system and a row in flight, 40 systems of 0.85 M rows in all
// took 170 and 110 us per iteration for the two updates; the sums, updates and
// stopping test take 77 us now (sums 52: the longest chain's loads).  The order
// of every sum is the same, which matters: with the
// factor in FP32, a different rounding here changes iteration counts.

namespace {

constexpr int SEG_THREADS = 256;

unsigned seg_sms() {
  int dev = 0, sms = 0;
  RCHOL_CUDA(cudaGetDevice(&dev));
  RCHOL_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  return (unsigned)sms;
}

struct SegState {
  const int64_t *seg;
  int nseg;
  double *bnorm2, *rz, *rz_prev, *relres;
  int *active, *iters, *any_active;
  const double *tol;
  const int *maxit;
  double *part;  // [3][nseg][256] chain sums: r.z or p.q, p.r, r.r
};

// Block-wide sum in a fixed tree; every thread gets the total.
__device__ double seg_sum(double v, double *sh) {
  sh[threadIdx.x] = v;
  __syncthreads();
  for (int h = SEG_THREADS / 2; h > 0; h >>= 1) {
    if (threadIdx.x < h) sh[threadIdx.x] += sh[threadIdx.x + h];
    __syncthreads();
  }
  const double t = sh[0];
  __syncthreads();
  return t;
}

// x = 0, r = b, ||b||^2 and the first stopping test (pcg.cpp:60-70).
__global__ void __launch_bounds__(SEG_THREADS) seg_init_kernel(SegState st, const double *b, double *x,
                                                               double *r) {
  __shared__ double sh[SEG_THREADS];
  const int s = blockIdx.x;
  const int64_t i0 = st.seg[s], i1 = st.seg[s + 1];
  double acc = 0.0;
  for (int64_t i = i0 + threadIdx.x; i < i1; i += SEG_THREADS) {
    const double bv = b[i];
    x[i] = 0.0;
    r[i] = bv;
    acc += bv * bv;
  }
  const double t = seg_sum(acc, sh);
  if (threadIdx.x == 0) {
    st.bnorm2[s] = t;
    st.iters[s] = 0;
    const int act = (sqrt(t) > sqrt(t) * *st.tol) && (*st.maxit > 0);
    st.active[s] = act;
    if (act) atomicOr(st.any_active, 1);
  }
}

constexpr int SEG_GROUPS = SEG_THREADS / 32;  // warps of a system
constexpr int SEG_AHEAD = 24;                 // rows of a chain read at a time
// Longest system of the one-block kernels.  Whole solves, chains over eight
// warps / one block: 50 systems of about 100 rows 834 / 622 us, 300 of 1024
// 2.85 / 2.36 ms, 300 of 4096 7.27 / 7.17, 300 of 8100 12.8 / 13.4, one of
// 4096 2.92 / 2.95, one of 16,384 10.0 / 11.3.
constexpr int64_t kSegOneRows = 4096;

// This warp's system (-1: none left, or converged) and chains.
struct SegLane {
  int s, chain;
  int64_t i0, i1;
};
__device__ __forceinline__ SegLane seg_lane(const SegState &st) {
  SegLane g{-1, 0, 0, 0};
  const int w = (int)(blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32), s = w / SEG_GROUPS;
  if (s >= st.nseg || !*st.any_active || !st.active[s]) return g;
  g.s = s;
  g.chain = (w % SEG_GROUPS) * 32 + (int)(threadIdx.x & 31);
  g.i0 = st.seg[s] + g.chain;
  g.i1 = st.seg[s + 1];
  return g;
}

// The tree of seg_sum over a system's 256 chain sums, by one warp: lane l holds
// chains l + 32 m.  Every lane gets the total.
__device__ __forceinline__ double seg_total(const double *chains) {
  const int lane = threadIdx.x & 31;
  double v[SEG_GROUPS];
#pragma unroll
  for (int m = 0; m < SEG_GROUPS; ++m) v[m] = chains[lane + 32 * m];
#pragma unroll
  for (int h = SEG_GROUPS / 2; h > 0; h >>= 1)
#pragma unroll
    for (int m = 0; m < h; ++m) v[m] += v[m + h];
#pragma unroll
  for (int h = 16; h > 0; h >>= 1) v[0] += __shfl_xor_sync(0xffffffffu, v[0], h);
  return v[0];
}

__device__ __forceinline__ double *seg_chains(const SegState &st, int which, int s) {
  return st.part + ((size_t)which * st.nseg + s) * SEG_THREADS;
}

// Chain sums of a.b, and of a.c where c is given (DUAL).
template <bool DUAL>
__global__ void __launch_bounds__(32) seg_dot_kernel(SegState st, int which, const double *__restrict__ a,
                                                     const double *__restrict__ b, const double *__restrict__ c) {
  const SegLane g = seg_lane(st);
  if (g.s < 0) return;
  double s0 = 0.0, s1 = 0.0;
  for (int64_t i = g.i0; i < g.i1; i += SEG_AHEAD * SEG_THREADS) {
    double av[SEG_AHEAD], bv[SEG_AHEAD], cv[SEG_AHEAD];
#pragma unroll
    for (int u = 0; u < SEG_AHEAD; ++u) {
      const int64_t k = i + u * SEG_THREADS;
      const bool on = k < g.i1;
      av[u] = on ? a[k] : 0.0;
      bv[u] = on ? b[k] : 0.0;
      if (DUAL) cv[u] = on ? c[k] : 0.0;
    }
#pragma unroll
    for (int u = 0; u < SEG_AHEAD; ++u)
      if (i + u * SEG_THREADS < g.i1) {
        s0 += av[u] * bv[u];
        if (DUAL) s1 += av[u] * cv[u];
      }
  }
  seg_chains(st, which, g.s)[g.chain] = s0;
  if (DUAL) seg_chains(st, which + 1, g.s)[g.chain] = s1;
}

// beta = rz / rz_prev, p = z (first iteration) or beta p + z; grid (systems, parts).
__global__ void __launch_bounds__(SEG_THREADS) seg_beta_kernel(SegState st, const double *z, double *p) {
  __shared__ double sh;
  const int s = blockIdx.x;
  if (!*st.any_active || !st.active[s]) return;
  if (threadIdx.x < 32) {
    const double rz = seg_total(seg_chains(st, 0, s));
    if (threadIdx.x == 0) sh = rz;
  }
  __syncthreads();
  const double rz = sh;
  const int it = st.iters[s];
  const double beta = it == 0 ? 0.0 : rz / st.rz_prev[s];
  const int64_t i1 = st.seg[s + 1];
  for (int64_t i = st.seg[s] + blockIdx.y * SEG_THREADS + threadIdx.x; i < i1; i += (int64_t)gridDim.y * SEG_THREADS)
    p[i] = it == 0 ? z[i] : beta * p[i] + 1.0 * z[i];
  if (threadIdx.x == 0 && blockIdx.y == 0) st.rz[s] = rz;
}

// alpha = p.r / p.q, x += alpha p, r -= alpha q; grid (systems, parts).
__global__ void __launch_bounds__(SEG_THREADS) seg_alpha_kernel(SegState st, const double *p, const double *q,
                                                                double *x, double *r) {
  __shared__ double sh;
  const int s = blockIdx.x;
  if (!*st.any_active || !st.active[s]) return;
  if (threadIdx.x < 32) {
    const double pq = seg_total(seg_chains(st, 0, s)), pr = seg_total(seg_chains(st, 1, s));
    if (threadIdx.x == 0) sh = pr / pq;
  }
  __syncthreads();
  const double alpha = sh;
  const int64_t i1 = st.seg[s + 1];
  for (int64_t i = st.seg[s] + blockIdx.y * SEG_THREADS + threadIdx.x; i < i1;
       i += (int64_t)gridDim.y * SEG_THREADS) {
    x[i] += alpha * p[i];
    r[i] = r[i] + -alpha * q[i];
  }
}

// The stopping test of system s, ||r||^2 = rr; one thread.
__device__ __forceinline__ void seg_stop(const SegState &st, int s, double rr) {
  const int it = st.iters[s] + 1;
  st.iters[s] = it;
  st.rz_prev[s] = st.rz[s];
  st.active[s] = (sqrt(rr) > sqrt(st.bnorm2[s]) * *st.tol) && (it < *st.maxit);
}

// One warp per system.
__global__ void __launch_bounds__(128) seg_conv_kernel(SegState st) {
  const int s = (int)(blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32);
  if (s >= st.nseg || !*st.any_active || !st.active[s]) return;
  const double t = seg_total(seg_chains(st, 2, s));
  if ((threadIdx.x & 31) == 0) seg_stop(st, s, t);
}

// Short systems: one thread block per system makes a system's sums and updates
// in one go, with two kernels an iteration instead of six.  (First of the two:
// beta and p as above.)
__global__ void __launch_bounds__(SEG_THREADS) seg_beta_one_kernel(SegState st, const double *r, const double *z,
                                                                   double *p) {
  __shared__ double sh[SEG_THREADS];
  const int s = blockIdx.x;
  if (!*st.any_active || !st.active[s]) return;
  const int64_t i0 = st.seg[s], i1 = st.seg[s + 1];
  double acc = 0.0;
  for (int64_t i = i0 + threadIdx.x; i < i1; i += SEG_THREADS) acc += r[i] * z[i];
  const double rz = seg_sum(acc, sh);
  const int it = st.iters[s];
  const double beta = it == 0 ? 0.0 : rz / st.rz_prev[s];
  for (int64_t i = i0 + threadIdx.x; i < i1; i += SEG_THREADS) p[i] = it == 0 ? z[i] : beta * p[i] + 1.0 * z[i];
  if (threadIdx.x == 0) st.rz[s] = rz;
}

// Second: alpha, x and r as above, then the stopping test.
__global__ void __launch_bounds__(SEG_THREADS) seg_alpha_one_kernel(SegState st, const double *p, const double *q,
                                                                    double *x, double *r) {
  __shared__ double sh[SEG_THREADS];
  const int s = blockIdx.x;
  if (!*st.any_active || !st.active[s]) return;
  const int64_t i0 = st.seg[s], i1 = st.seg[s + 1];
  double a0 = 0.0, a1 = 0.0;
  for (int64_t i = i0 + threadIdx.x; i < i1; i += SEG_THREADS) {
    const double pv = p[i];
    a0 += pv * q[i];
    a1 += pv * r[i];
  }
  const double pq = seg_sum(a0, sh), pr = seg_sum(a1, sh), alpha = pr / pq;
  double rr = 0.0;
  for (int64_t i = i0 + threadIdx.x; i < i1; i += SEG_THREADS) {
    x[i] += alpha * p[i];
    const double rv = r[i] + -alpha * q[i];
    r[i] = rv;
    rr += rv * rv;
  }
  const double t = seg_sum(rr, sh);
  if (threadIdx.x == 0) seg_stop(st, s, t);
}

__global__ void seg_any_kernel(SegState st) {
  __shared__ int any;
  if (threadIdx.x == 0) any = 0;
  __syncthreads();
  int a = 0;
  for (int s = threadIdx.x; s < st.nseg; s += blockDim.x) a |= st.active[s];
  if (a) atomicOr(&any, 1);
  __syncthreads();
  if (threadIdx.x == 0) *st.any_active = any;
}

// relres = ||A x - b|| / ||b|| per system (q = A x).
__global__ void __launch_bounds__(SEG_THREADS) seg_resid_kernel(SegState st, const double *q, const double *b) {
  __shared__ double sh[SEG_THREADS];
  const int s = blockIdx.x;
  const int64_t i0 = st.seg[s], i1 = st.seg[s + 1];
  double acc = 0.0;
  for (int64_t i = i0 + threadIdx.x; i < i1; i += SEG_THREADS) {
    const double d = q[i] + -1.0 * b[i];
    acc += d * d;
  }
  const double t = seg_sum(acc, sh);
  if (threadIdx.x == 0) st.relres[s] = sqrt(t) / sqrt(st.bnorm2[s]);
}

}  // namespace

// Whether a thread block per system serves (see the kernels).
static bool seg_one_block(int64_t nseg, const int64_t *seg) {
  int64_t most = 0;
  for (int64_t s = 0; s < nseg; ++s) most = std::max(most, seg[s + 1] - seg[s]);
  return most <= kSegOneRows;
}

static SegWork &seg_workspace(const rchol_matrix_s &A, const rchol_factor_s &F, int64_t nseg,
                              const int64_t *seg) {
  SolvePlan &P = *F.plan;
  for (auto &w : P.seg)
    if (w->key_uid == A.uid && (int64_t)w->seg_host.size() == nseg + 1 &&
        std::equal(w->seg_host.begin(), w->seg_host.end(), seg))
      return *w;
  if (P.seg.size() >= 4) P.seg.erase(P.seg.begin());
  auto w = std::make_unique<SegWork>();
  w->key_uid = A.uid;
  w->seg_host.assign(seg, seg + nseg + 1);
  w->n = A.n;
  w->seg.upload(seg, nseg + 1, 0);
  w->r.alloc(A.n);
  w->z.alloc(A.n);
  w->p.alloc(A.n);
  w->q.alloc(A.n);
  w->x.alloc(A.n);
  w->one_block = seg_one_block(nseg, seg);
  w->sc.alloc(4 * (size_t)nseg + 1 + (w->one_block ? 0 : 3 * (size_t)nseg * SEG_THREADS));
  w->ic.alloc(2 * (size_t)nseg + 2);
  RCHOL_CUDA(cudaStreamCreateWithFlags(&w->stream, cudaStreamNonBlocking));
  RCHOL_CUDA(cudaEventCreateWithFlags(&w->ev_in, cudaEventDisableTiming));
  RCHOL_CUDA(cudaEventCreateWithFlags(&w->ev_out, cudaEventDisableTiming));
  RCHOL_CUDA(cudaStreamSynchronize(0));
  P.seg.push_back(std::move(w));
  return *P.seg.back();
}

static SegState seg_state(SegWork &w) {
  const int S = (int)(w.seg_host.size() - 1);
  SegState st;
  st.seg = w.seg.p;
  st.nseg = S;
  st.bnorm2 = w.sc.p;
  st.rz = w.sc.p + S;
  st.rz_prev = w.sc.p + 2 * (size_t)S;
  st.relres = w.sc.p + 3 * (size_t)S;
  st.tol = w.sc.p + 4 * (size_t)S;
  st.active = w.ic.p;
  st.iters = w.ic.p + S;
  st.any_active = w.ic.p + 2 * (size_t)S;
  st.maxit = w.ic.p + 2 * (size_t)S + 1;
  st.part = w.sc.p + 4 * (size_t)S + 1;
  return st;
}

static void pcg_batch_impl(const rchol_matrix_s &A, const rchol_factor_s &F, int64_t nseg, const int64_t *seg,
                           const double *b, double *x, const double *b_host, double *x_host, double tol,
                           int maxit, double *relres, int *itr, cudaStream_t s) {
  SolvePlan &P = *F.plan;
  std::lock_guard<std::mutex> guard(P.lock);
  const int64_t n = A.n;
  ensure_pcg(F, 1, s);
  SegWork &w = seg_workspace(A, F, nseg, seg);
  SegState st = seg_state(w);
  const unsigned S = (unsigned)nseg;
  cudaStream_t ws = w.stream;
  RCHOL_CUDA(cudaEventRecord(w.ev_in, s));
  RCHOL_CUDA(cudaStreamWaitEvent(ws, w.ev_in, 0));
  if (b_host) {
    if (w.hb.n < (size_t)n) w.hb.alloc(n);
    if (w.hx.n < (size_t)n) w.hx.alloc(n);
    RCHOL_CUDA(cudaMemcpyAsync(w.hb.p, b_host, n * sizeof(double), cudaMemcpyHostToDevice, ws));
    b = w.hb.p;
    x = w.hx.p;
  }
  if (!w.exec) {
    cudaGraph_t g = nullptr;
    RCHOL_CUDA(cudaStreamBeginCapture(ws, cudaStreamCaptureModeThreadLocal));
    try {
      precond_streams(F, w.r.p, w.z.p, P.ytmp.p, P.ytmp32.p, 1, ws);
      if (w.one_block) {
        seg_beta_one_kernel<<<S, SEG_THREADS, 0, ws>>>(st, w.r.p, w.z.p, w.p.p);
        spmv(A, w.p.p, w.q.p, 1, ws);
        seg_alpha_one_kernel<<<S, SEG_THREADS, 0, ws>>>(st, w.p.p, w.q.p, w.x.p, w.r.p);
      } else {
        const unsigned C = S * SEG_GROUPS;
        // element updates: enough parts of a system for four thread blocks an SM
        const dim3 E(S, std::min(64u, (4 * seg_sms() + S - 1) / S));
        seg_dot_kernel<false><<<C, 32, 0, ws>>>(st, 0, w.r.p, w.z.p, nullptr);
        seg_beta_kernel<<<E, SEG_THREADS, 0, ws>>>(st, w.z.p, w.p.p);
        spmv(A, w.p.p, w.q.p, 1, ws);
        seg_dot_kernel<true><<<C, 32, 0, ws>>>(st, 0, w.p.p, w.q.p, w.r.p);
        seg_alpha_kernel<<<E, SEG_THREADS, 0, ws>>>(st, w.p.p, w.q.p, w.x.p, w.r.p);
        seg_dot_kernel<false><<<C, 32, 0, ws>>>(st, 2, w.r.p, w.r.p, nullptr);
        seg_conv_kernel<<<(S + 3) / 4, 128, 0, ws>>>(st);
      }
      seg_any_kernel<<<1, 256, 0, ws>>>(st);
      RCHOL_CUDA(cudaGetLastError());
    } catch (...) {
      cudaStreamEndCapture(ws, &g);
      if (g) cudaGraphDestroy(g);
      throw;
    }
    RCHOL_CUDA(cudaStreamEndCapture(ws, &g));
    size_t nodes = 0;
    RCHOL_CUDA(cudaGraphGetNodes(g, nullptr, &nodes));
    w.graph_kernels = (int64_t)nodes;
    cudaError_t e = cudaGraphInstantiate(&w.exec, g, 0);
    cudaGraphDestroy(g);
    RCHOL_CUDA(e);
  }
  double htol = tol;
  int hmax = maxit;
  RCHOL_CUDA(cudaMemsetAsync(w.sc.p, 0, w.sc.bytes(), ws));
  RCHOL_CUDA(cudaMemsetAsync(w.ic.p, 0, w.ic.bytes(), ws));
  RCHOL_CUDA(cudaMemcpyAsync(const_cast<double *>(st.tol), &htol, sizeof(double), cudaMemcpyHostToDevice, ws));
  RCHOL_CUDA(cudaMemcpyAsync(const_cast<int *>(st.maxit), &hmax, sizeof(int), cudaMemcpyHostToDevice, ws));
  seg_init_kernel<<<S, SEG_THREADS, 0, ws>>>(st, b, w.x.p, w.r.p);
  note_launch(1);
  RCHOL_CUDA(cudaGetLastError());
  int h_any = 1;
  for (int it = 0; it < maxit;) {
    const int batch = it == 0 ? 8 : 4;
    for (int j = 0; j < batch && it < maxit; ++j, ++it) {
      RCHOL_CUDA(cudaGraphLaunch(w.exec, ws));
      note_launch(w.graph_kernels);
    }
    RCHOL_CUDA(cudaMemcpyAsync(&h_any, st.any_active, sizeof(int), cudaMemcpyDeviceToHost, ws));
    RCHOL_CUDA(cudaStreamSynchronize(ws));
    if (!h_any) break;
  }
  spmv(A, w.x.p, w.q.p, 1, ws);
  seg_resid_kernel<<<S, SEG_THREADS, 0, ws>>>(st, w.q.p, b);
  note_launch(2);
  RCHOL_CUDA(cudaGetLastError());
  if (x_host) RCHOL_CUDA(cudaMemcpyAsync(x_host, w.x.p, n * sizeof(double), cudaMemcpyDeviceToHost, ws));
  else RCHOL_CUDA(cudaMemcpyAsync(x, w.x.p, n * sizeof(double), cudaMemcpyDeviceToDevice, ws));
  RCHOL_CUDA(cudaMemcpyAsync(relres, st.relres, nseg * sizeof(double), cudaMemcpyDeviceToHost, ws));
  RCHOL_CUDA(cudaMemcpyAsync(itr, st.iters, nseg * sizeof(int), cudaMemcpyDeviceToHost, ws));
  RCHOL_CUDA(cudaEventRecord(w.ev_out, ws));
  RCHOL_CUDA(cudaStreamWaitEvent(s, w.ev_out, 0));
  RCHOL_CUDA(cudaStreamSynchronize(ws));
}

void pcg_batch_device(const rchol_matrix_s &A, const rchol_factor_s &F, int64_t nseg, const int64_t *seg,
                      const double *b, double *x, double tol, int maxit, double *relres, int *itr,
                      cudaStream_t s) {
  pcg_batch_impl(A, F, nseg, seg, b, x, nullptr, nullptr, tol, maxit, relres, itr, s);
}

void pcg_batch_host(const rchol_matrix_s &A, const rchol_factor_s &F, int64_t nseg, const int64_t *seg,
                    const double *b, double *x, double tol, int maxit, double *relres, int *itr) {
  pcg_batch_impl(A, F, nseg, seg, nullptr, nullptr, b, x, tol, maxit, relres, itr, 0);
}

}  // namespace rchol
