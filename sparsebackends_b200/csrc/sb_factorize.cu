// Device kernels of the block factorisations (QR and SVD truncation).
//
// * Householder QR of a column-major m x n matrix with LAPACK's dlarfg
//   convention (beta = -sign(alpha) * ||x||, tau = (beta - alpha) / beta,
//   v = x / (alpha - beta), H = I when the sub-column is zero), so Q and R
//   agree with LAPACK geqrf/orgqr up to rounding.  Up to 1024 rows in panels of
//   16 or 32 reflectors in compact WY form (Schreiber and Van Loan 1989):
//   k_house_panel factors a panel in one CTA, its columns in registers;
//   k_house_block applies I - V T^T V^T to the columns behind it, one CTA per
//   column, and k_house_q forms Q column by column.  Beyond 1024 rows one
//   reflector at a time (k_house_gen, k_house_apply).
// * One-sided (Hestenes) Jacobi SVD of many small row-major matrices, one CTA
//   per matrix: rows are rotated pairwise until orthogonal, U accumulates the
//   rotations; singular values are the final row norms (high relative
//   accuracy, which the relative cutoff of the truncation needs).
// Every loop is bounded; a Jacobi solve that has not converged after
// max_sweeps sweeps raises a status flag the host reads.
#include <algorithm>

#include "sb_kernels.hpp"

namespace sb {
namespace {

constexpr int kFacThreads = 256;

__device__ __forceinline__ double block_sum(double v, double* red) {
  // fixed-order tree reduction over kFacThreads threads; result broadcast
  red[threadIdx.x] = v;
  __syncthreads();
#pragma unroll
  for (int s = kFacThreads / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] = __dadd_rn(red[threadIdx.x], red[threadIdx.x + s]);
    __syncthreads();
  }
  const double r = red[0];
  __syncthreads();
  return r;
}

__global__ void __launch_bounds__(kFacThreads)
    k_house_gen(double* __restrict__ M, int64_t ld, int64_t m, int64_t j, double* __restrict__ tau) {
  __shared__ double red[kFacThreads];
  __shared__ double scal;
  double* col = M + j * ld;
  double acc = 0.0;
  for (int64_t i = j + 1 + threadIdx.x; i < m; i += kFacThreads) acc = __fma_rn(col[i], col[i], acc);
  const double xn2 = block_sum(acc, red);
  if (threadIdx.x == 0) {
    const double alpha = col[j];
    if (xn2 == 0.0) {
      tau[j] = 0.0;
      scal = 0.0;
    } else {
      const double nrm = sqrt(__fma_rn(alpha, alpha, xn2));
      const double beta = alpha >= 0.0 ? -nrm : nrm;
      tau[j] = (beta - alpha) / beta;
      scal = 1.0 / (alpha - beta);
      col[j] = beta;
    }
  }
  __syncthreads();
  const double s = scal;
  if (s != 0.0)
    for (int64_t i = j + 1 + threadIdx.x; i < m; i += kFacThreads) col[i] = __dmul_rn(col[i], s);
}

// T[:, c] = (I - tau_j v v^T) T[:, c] for c in [c0, c0 + gridDim.x); v_j = 1,
// v_i = V[i + j*ldv] for i > j; rows below j only.
__global__ void __launch_bounds__(kFacThreads)
    k_house_apply(const double* __restrict__ V, int64_t ldv, double* __restrict__ T, int64_t ldt, int64_t m,
                  int64_t j, int64_t c0, const double* __restrict__ tau) {
  __shared__ double red[kFacThreads];
  const double t = tau[j];
  if (t == 0.0) return;
  const double* v = V + j * ldv;
  double* col = T + (c0 + blockIdx.x) * ldt;
  double acc = 0.0;
  for (int64_t i = j + 1 + threadIdx.x; i < m; i += kFacThreads) acc = __fma_rn(v[i], col[i], acc);
  const double s = block_sum(acc, red);
  const double w = __dmul_rn(t, __dadd_rn(col[j], s));
  if (threadIdx.x == 0) col[j] = __dsub_rn(col[j], w);
  for (int64_t i = j + 1 + threadIdx.x; i < m; i += kFacThreads) col[i] = __fma_rn(-v[i], w, col[i]);
}

// One panel of pb <= 16 * CPW reflectors: rows [p0, m) of columns [p0, p0 + pb)
// of M (m - p0 <= 32 * RPL).  Warp w owns columns w and w + 16; row p0 + r of
// a column is register r / 32 of lane r % 32, so the pivot of reflector j is
// register 0 of lane j.  Per reflector: its owner leaves the column below the
// pivot in shared memory (two buffers), one barrier, and every warp takes the
// norm and the products with its own columns in one reduction: the columns
// behind update, those before give V^T v for T.  Latency-bound: a barrier, one
// warp reduction, a square root, a division and the update per reflector, 1.35 us
// each at 256 rows.  The 256 x 160 factorisation took 2.0 ms as a launch per
// reflector and one per update (483), and takes 0.34 ms in 13 launches.
// The products are those of x, scaled afterwards: they stay in range and meet
// no infinity with x's zeros while every magnitude is at most 2^400; a panel
// that holds a larger one, an infinity or NaN goes to house_panel_plain.
constexpr int kPanelThreads = 512;
constexpr int kPanelMax = 32;    // reflectors of a panel
constexpr int kPanelRows = 1024;

// The panel in memory, a warp per column, with products of v over the rows below
// the pivot only and no step for a reflector with tau = 0, so that infinities
// and NaN reach what the reflectors one at a time let them reach.
__device__ __noinline__ void house_panel_plain(double* M, int64_t ld, int rows, int p0, int pb, double* T, double* taus,
                                               double (*z)[kPanelMax + 1], double (*ts)[kPanelMax + 1]) {
  const int warp = static_cast<int>(threadIdx.x) >> 5, lane = static_cast<int>(threadIdx.x) & 31;
  auto column = [&](int c) { return M + p0 + static_cast<int64_t>(p0 + c) * ld; };
  auto product = [&](const double* a, const double* b, int r0) {  // over rows [r0, rows)
    double s = 0.0;
    for (int r = r0 + lane; r < rows; r += 32) s = __fma_rn(a[r], b[r], s);
    for (int o = 16; o > 0; o >>= 1) s = __dadd_rn(s, __shfl_xor_sync(0xffffffffu, s, o));
    return s;
  };
  for (int j = 0; j < pb; ++j) {
    double* const v = column(j);
    const double alpha = v[j], xn2 = product(v, v, j + 1);
    double tau = 0.0, beta = alpha, scal = 0.0;
    if (xn2 != 0.0) {
      const double nrm = sqrt(__fma_rn(alpha, alpha, xn2));
      beta = alpha >= 0.0 ? -nrm : nrm;
      tau = (beta - alpha) / beta;
      scal = 1.0 / (alpha - beta);
    }
    __syncthreads();
    if (warp == (j & 15)) {
      if (scal != 0.0)
        for (int r = j + 1 + lane; r < rows; r += 32) v[r] = __dmul_rn(v[r], scal);
      if (lane == 0) {
        v[j] = beta;
        taus[j] = tau;
      }
    }
    __syncthreads();
    for (int c = warp; c < pb; c += kPanelThreads / 32) {
      if (c == j || (c > j && tau == 0.0)) continue;
      double* const col = column(c);
      const double cj = col[j], d = __dadd_rn(cj, product(v, col, j + 1)), w = __dmul_rn(tau, d);
      if (c < j) {
        if (lane == 0) z[c][j] = d;
        continue;
      }
      __syncwarp();
      if (lane == 0) col[j] = __dsub_rn(cj, w);
      for (int r = j + 1 + lane; r < rows; r += 32) col[r] = __fma_rn(-v[r], w, col[r]);
    }
    __syncthreads();
    if (warp == 0) {
      double s = 0.0;
      for (int i = lane; i < j; ++i)
        if (taus[i] != 0.0) s = __fma_rn(ts[lane][i], z[i][j], s);
      if (lane < j) ts[lane][j] = taus[lane] != 0.0 && tau != 0.0 ? -__dmul_rn(tau, s) : 0.0;
      else if (lane == j) ts[j][j] = tau;
      __syncwarp();
    }
  }
  if (warp == 0)
    for (int j = 0; j < pb; ++j) T[lane + kPanelMax * j] = lane <= j ? ts[lane][j] : 0.0;
}
template <int RPL, int CPW>
__global__ void __launch_bounds__(kPanelThreads, 1)
    k_house_panel(double* __restrict__ M, int64_t ld, int m, int p0, int pb, double* __restrict__ T) {
  __shared__ double xs[2][32 * RPL];
  __shared__ double alphas[2];
  __shared__ double taus[kPanelMax];
  __shared__ double z[kPanelMax][kPanelMax + 1];   // z[i][j] = v_i . v_j, i < j
  __shared__ double ts[kPanelMax][kPanelMax + 1];  // T, upper triangular
  const int warp = static_cast<int>(threadIdx.x) >> 5, lane = static_cast<int>(threadIdx.x) & 31;
  const int rows = m - p0;
  double a[CPW][RPL];
#pragma unroll
  for (int q = 0; q < CPW; ++q) {
    const int c = warp + 16 * q;
    const double* col = M + p0 + static_cast<int64_t>(p0 + c) * ld;
#pragma unroll
    for (int i = 0; i < RPL; ++i) a[q][i] = c < pb && lane + 32 * i < rows ? col[lane + 32 * i] : 0.0;
  }
  bool odd = false;
#pragma unroll
  for (int q = 0; q < CPW; ++q)
#pragma unroll
    for (int i = 0; i < RPL; ++i) odd = odd || !(fabs(a[q][i]) <= 0x1p400);
  if (__syncthreads_or(odd)) {
    house_panel_plain(M, ld, rows, p0, pb, T, taus, z, ts);
    return;
  }
  // T(0:j, j) = -tau_j * T(0:j, 0:j) * z(0:j, j), T(j, j) = tau_j, by one warp
  auto t_column = [&](int j) {
    double s0 = 0.0, s1 = 0.0;
    for (int i = 0; i < j; i += 2) {
      if (i >= lane) s0 = __fma_rn(ts[lane][i], z[i][j], s0);
      if (i + 1 >= lane && i + 1 < j) s1 = __fma_rn(ts[lane][i + 1], z[i + 1][j], s1);
    }
    if (lane < j) ts[lane][j] = -__dmul_rn(taus[j], __dadd_rn(s0, s1));
    else if (lane == j) ts[j][j] = taus[j];
    __syncwarp();
  };
  // reflector j = 16 * qj + jj belongs to warp jj's column qj (a constant index)
#pragma unroll
  for (int qj = 0; qj < CPW; ++qj)
    for (int jj = 0; jj < 16 && 16 * qj + jj < pb; ++jj) {
      const int j = 16 * qj + jj;
      double* const x = xs[j & 1];
      if (warp == jj) {
        x[lane] = lane > j ? a[qj][0] : 0.0;
#pragma unroll
        for (int i = 1; i < RPL; ++i) x[lane + 32 * i] = a[qj][i];
        if (lane == j) alphas[j & 1] = a[qj][0];
      }
      __syncthreads();
      // x . x and x . column together, in every warp
      double n0 = 0.0, n1 = 0.0, s0[CPW], s1[CPW];
#pragma unroll
      for (int q = 0; q < CPW; ++q) s0[q] = s1[q] = 0.0;
#pragma unroll
      for (int i = 0; i < RPL; i += 2) {
        const double u = x[lane + 32 * i], w = i + 1 < RPL ? x[lane + 32 * (i + 1)] : 0.0;
        n0 = __fma_rn(u, u, n0);
        n1 = __fma_rn(w, w, n1);
#pragma unroll
        for (int q = 0; q < CPW; ++q) {
          s0[q] = __fma_rn(u, a[q][i], s0[q]);
          if (i + 1 < RPL) s1[q] = __fma_rn(w, a[q][i + 1], s1[q]);
        }
      }
      double sum[CPW + 1];
      sum[CPW] = __dadd_rn(n0, n1);
#pragma unroll
      for (int q = 0; q < CPW; ++q) sum[q] = __dadd_rn(s0[q], s1[q]);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q <= CPW; ++q) sum[q] = __dadd_rn(sum[q], __shfl_xor_sync(0xffffffffu, sum[q], o));
      const double xn2 = sum[CPW], alpha = alphas[j & 1];
      double tau = 0.0, beta = alpha, scal = 1.0;
      if (xn2 != 0.0) {
        const double nrm = sqrt(__fma_rn(alpha, alpha, xn2));
        beta = alpha >= 0.0 ? -nrm : nrm;
        tau = (beta - alpha) / beta;
        scal = 1.0 / (alpha - beta);
      }
#pragma unroll
      for (int q = 0; q < CPW; ++q) {
        const int c = warp + 16 * q;
        // v . column, v = (1, scal * x) from row j on
        const double d = __fma_rn(scal, sum[q], __shfl_sync(0xffffffffu, a[q][0], j));
        if (c == j) {
          a[q][0] = lane > j ? __dmul_rn(a[q][0], scal) : lane == j ? beta : a[q][0];
#pragma unroll
          for (int i = 1; i < RPL; ++i) a[q][i] = __dmul_rn(a[q][i], scal);
          if (lane == 0) taus[j] = tau;
        } else if (c > j) {
          const double w = __dmul_rn(tau, d), ws = -__dmul_rn(w, scal);
          if (lane == j) a[q][0] = __dsub_rn(a[q][0], w);
#pragma unroll
          for (int i = 0; i < RPL; ++i) a[q][i] = __fma_rn(x[lane + 32 * i], ws, a[q][i]);
        } else if (lane == 0) {
          z[c][j] = d;
        }
      }
      // T's column j - 1, by a warp that is not about to own a reflector
      if (j > 0 && warp == ((jj + 8) & 15)) t_column(j - 1);
    }
#pragma unroll
  for (int q = 0; q < CPW; ++q) {
    const int c = warp + 16 * q;
    double* col = M + p0 + static_cast<int64_t>(p0 + c) * ld;
#pragma unroll
    for (int i = 0; i < RPL; ++i)
      if (c < pb && lane + 32 * i < rows) col[lane + 32 * i] = a[q][i];
  }
  __syncthreads();
  if (warp == 0) {
    t_column(pb - 1);
    for (int j = 0; j < pb; ++j)
      if (lane < kPanelMax) T[lane + kPanelMax * j] = lane <= j ? ts[lane][j] : 0.0;
  }
}

// x <- (I - V op(T) V^T) x for one column x (rows [p0, m), in shared memory),
// V the panel's reflectors in M (1 on the diagonal, 0 above).  A warp takes
// the dot products of a stride of the reflectors; V is read from L2 twice,
// coalesced along its columns.  A product that is not finite is taken again over
// the rows from the pivot on, and T's zeros (reflectors with tau = 0) skip it.
__device__ __forceinline__ void apply_block(const double* __restrict__ M, int64_t ld, int m, int p0, int pb,
                                            const double* __restrict__ T, bool trans, double* x, double* w, double* y) {
  const int tid = static_cast<int>(threadIdx.x), warp = tid >> 5, lane = tid & 31, rows = m - p0;
  constexpr int kPer = kPanelMax / (kFacThreads / 32);  // reflectors per warp, their loads in flight together
  double s4[kPer];
#pragma unroll
  for (int q = 0; q < kPer; ++q) s4[q] = 0.0;
#pragma unroll 4
  for (int r = lane; r < rows; r += 32) {
#pragma unroll
    for (int q = 0; q < kPer; ++q) {
      const int j = kPer * warp + q;
      const double vr = r > j && j < pb ? M[p0 + r + static_cast<int64_t>(p0 + j) * ld] : r == j ? 1.0 : 0.0;
      s4[q] = __fma_rn(vr, x[r], s4[q]);
    }
  }
#pragma unroll
  for (int q = 0; q < kPer; ++q) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s4[q] = __dadd_rn(s4[q], __shfl_xor_sync(0xffffffffu, s4[q], o));
    if (lane == 0) w[kPer * warp + q] = s4[q];
  }
  bool odd = false;
#pragma unroll
  for (int q = 0; q < kPer; ++q) odd = odd || !isfinite(s4[q]);
  odd = __syncthreads_or(odd);
  if (odd) {
    for (int j = kPer * warp; j < kPer * warp + kPer && j < pb; ++j) {
      double s = 0.0;
      for (int r = j + lane; r < rows; r += 32)
        s = __fma_rn(r > j ? M[p0 + r + static_cast<int64_t>(p0 + j) * ld] : 1.0, x[r], s);
      for (int o = 16; o > 0; o >>= 1) s = __dadd_rn(s, __shfl_xor_sync(0xffffffffu, s, o));
      if (lane == 0) w[j] = s;
    }
    __syncthreads();
  }
  if (tid < pb) {
    double s = 0.0;
    if (odd)
      for (int i = trans ? 0 : tid; i < (trans ? tid + 1 : pb); ++i) {
        const double t = T[trans ? i + kPanelMax * tid : tid + kPanelMax * i];
        if (t != 0.0) s = __fma_rn(t, w[i], s);
      }
    else if (trans)
      for (int i = 0; i <= tid; ++i) s = __fma_rn(T[i + kPanelMax * tid], w[i], s);
    else
      for (int j = tid; j < pb; ++j) s = __fma_rn(T[tid + kPanelMax * j], w[j], s);
    y[tid] = s;
  }
  __syncthreads();
  for (int r = tid; r < rows; r += kFacThreads) {
    const double* v = M + p0 + r + static_cast<int64_t>(p0) * ld;
    const int jn = r < pb ? r : pb;  // reflectors with a stored entry in this row
    double s0 = r < pb ? y[r] : 0.0, s1 = 0.0;
    int j = 0;
#pragma unroll 8
    for (; j + 1 < jn; j += 2) {
      s0 = __fma_rn(v[static_cast<int64_t>(j) * ld], y[j], s0);
      s1 = __fma_rn(v[static_cast<int64_t>(j + 1) * ld], y[j + 1], s1);
    }
    if (j < jn) s0 = __fma_rn(v[static_cast<int64_t>(j) * ld], y[j], s0);
    x[r] = __dsub_rn(x[r], __dadd_rn(s0, s1));
  }
  __syncthreads();
}

// Columns [c0, c0 + gridDim.x) of M through the panel at p0 (transposed T).
__global__ void __launch_bounds__(kFacThreads)
    k_house_block(double* __restrict__ M, int64_t ld, int m, int p0, int pb, int c0, const double* __restrict__ T) {
  __shared__ double x[kPanelRows], w[kPanelMax], y[kPanelMax];
  double* col = M + p0 + static_cast<int64_t>(c0 + blockIdx.x) * ld;
  for (int r = threadIdx.x; r < m - p0; r += kFacThreads) x[r] = col[r];
  __syncthreads();
  apply_block(M, ld, m, p0, pb, T, true, x, w, y);
  for (int r = threadIdx.x; r < m - p0; r += kFacThreads) col[r] = x[r];
}

// Column blockIdx.x = c of Q = H_0 H_1 ... H_{k-1} restricted to k columns: the
// panels of nb reflectors applied to the unit vector, last one first; the
// reflectors behind the c-th leave it alone.
__global__ void __launch_bounds__(kFacThreads)
    k_house_q(const double* __restrict__ M, int64_t ld, int m, int nb, const double* __restrict__ T,
              double* __restrict__ Q) {
  __shared__ double x[kPanelRows], w[kPanelMax], y[kPanelMax];
  const int c = static_cast<int>(blockIdx.x);
  for (int r = threadIdx.x; r < m; r += kFacThreads) x[r] = r == c ? 1.0 : 0.0;
  __syncthreads();
  for (int p = c / nb; p >= 0; --p)
    apply_block(M, ld, m, p * nb, min(nb, c + 1 - p * nb), T + static_cast<int64_t>(p) * kPanelMax * kPanelMax, false,
                x + p * nb, w, y);
  for (int r = threadIdx.x; r < m; r += kFacThreads) Q[r + static_cast<int64_t>(c) * m] = x[r];
}

__global__ void k_identity_cols(double* __restrict__ Q, int64_t m, int64_t k) {
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < m * k;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x)
    Q[e] = (e % m == e / m) ? 1.0 : 0.0;
}

__global__ void k_upper(const double* __restrict__ M, int64_t m, int64_t k, int64_t n, double* __restrict__ R) {
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < k * n;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const int64_t r = e % k, c = e / k;
    R[e] = r <= c ? M[r + c * m] : 0.0;
  }
}

// WARP: a warp per item (items of a few elements, the blocks of a sparse
// prefix); otherwise a row of CTAs per item.
template <bool WARP>
__global__ void k_gather_2d(const double* __restrict__ src, double* __restrict__ dst, const double* __restrict__ scale,
                            const Gather2D* __restrict__ items, int64_t nitems) {
  const int64_t i = WARP ? static_cast<int64_t>(blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5) : blockIdx.y;
  if (i >= nitems) return;
  const Gather2D it = items[i];
  const int64_t n = it.rows * it.cols, step = WARP ? 32 : static_cast<int64_t>(gridDim.x) * blockDim.x;
  for (int64_t e = WARP ? threadIdx.x & 31 : static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < n;
       e += step) {
    const int64_t r = e % it.rows, c = e / it.rows;
    const double v = src[it.src_off + r * it.src_rs + c * it.src_cs];
    dst[it.dst_off + r * it.dst_rs + c * it.dst_cs] = it.s_idx >= 0 ? __dmul_rn(v, scale[it.s_idx + c]) : v;
  }
}

__global__ void __launch_bounds__(kFacThreads)
    k_svd_rows(double* __restrict__ A, double* __restrict__ Vt, double* __restrict__ U, double* __restrict__ S,
               const SvdGroup* __restrict__ groups, int max_sweeps, int* __restrict__ status) {
  __shared__ double red[kFacThreads];
  __shared__ double Us[kSvdMaxRows * kSvdMaxRows];
  __shared__ double nrm[kSvdMaxRows];
  __shared__ int perm[kSvdMaxRows];
  const SvdGroup g = groups[blockIdx.x];
  const int m = g.m;
  const int64_t n = g.n;
  double* a = A + g.a_off;
  for (int e = threadIdx.x; e < m * m; e += kFacThreads) Us[e] = (e % m == e / m) ? 1.0 : 0.0;
  __syncthreads();
  // Rotation threshold |gamma| > tol * sqrt(alpha * beta) with tol = n * eps,
  // the rounding bound of the length-n dot products: below it the rows are
  // orthogonal to working accuracy.  (A tighter threshold makes rank-deficient
  // groups rotate rounding-level rows forever.)
  const double eps = 2.220446049250313e-16;
  const double tol = eps * static_cast<double>(n > 1 ? n : 1);
  // Rows with norm below eps * ||A||_F are rounding noise: they take part in
  // no rotation (rotating them against each other never settles).
  double fro = 0.0;
  for (int64_t i = threadIdx.x; i < static_cast<int64_t>(m) * n; i += kFacThreads) fro = __fma_rn(a[i], a[i], fro);
  const double tiny = eps * eps * block_sum(fro, red);
  bool rotated = true;
  int sweep = 0;
  for (; sweep < max_sweeps && rotated; ++sweep) {
    rotated = false;
    for (int p = 0; p < m - 1; ++p) {
      for (int q = p + 1; q < m; ++q) {
        double* rp = a + static_cast<int64_t>(p) * n;
        double* rq = a + static_cast<int64_t>(q) * n;
        double sa = 0.0, sb2 = 0.0, sc = 0.0;
        for (int64_t i = threadIdx.x; i < n; i += kFacThreads) {
          const double x = rp[i], y = rq[i];
          sa = __fma_rn(x, x, sa);
          sb2 = __fma_rn(y, y, sb2);
          sc = __fma_rn(x, y, sc);
        }
        const double alpha = block_sum(sa, red);
        const double beta = block_sum(sb2, red);
        const double gamma = block_sum(sc, red);
        // uniform across the CTA (reduced values)
        if (alpha <= tiny || beta <= tiny || gamma == 0.0 || fabs(gamma) <= tol * sqrt(alpha) * sqrt(beta)) continue;
        rotated = true;
        const double zeta = (beta - alpha) / (2.0 * gamma);
        const double t = (zeta >= 0.0 ? 1.0 : -1.0) / (fabs(zeta) + hypot(1.0, zeta));
        const double cs = 1.0 / sqrt(1.0 + t * t);
        const double sn = cs * t;
        for (int64_t i = threadIdx.x; i < n; i += kFacThreads) {
          const double x = rp[i], y = rq[i];
          rp[i] = cs * x - sn * y;
          rq[i] = sn * x + cs * y;
        }
        if (threadIdx.x < m) {
          const double x = Us[threadIdx.x + p * m], y = Us[threadIdx.x + q * m];
          Us[threadIdx.x + p * m] = cs * x - sn * y;
          Us[threadIdx.x + q * m] = sn * x + cs * y;
        }
        __syncthreads();
      }
    }
  }
  if (rotated && threadIdx.x == 0) atomicExch(status, 1);  // not converged within max_sweeps
  // singular values = row norms, sorted descending (stable in row index)
  for (int p = 0; p < m; ++p) {
    const double* rp = a + static_cast<int64_t>(p) * n;
    double s = 0.0;
    for (int64_t i = threadIdx.x; i < n; i += kFacThreads) s = __fma_rn(rp[i], rp[i], s);
    const double t = block_sum(s, red);
    if (threadIdx.x == 0) nrm[p] = sqrt(t);
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    for (int p = 0; p < m; ++p) perm[p] = p;
    for (int p = 1; p < m; ++p) {
      const int x = perm[p];
      int q = p - 1;
      while (q >= 0 && nrm[perm[q]] < nrm[x]) {
        perm[q + 1] = perm[q];
        --q;
      }
      perm[q + 1] = x;
    }
  }
  __syncthreads();
  for (int r = 0; r < m; ++r) {
    const int p = perm[r];
    const double s = nrm[p];
    const double inv = s > 0.0 ? 1.0 / s : 0.0;
    const double* rp = a + static_cast<int64_t>(p) * n;
    double* out = Vt + g.a_off + static_cast<int64_t>(r) * n;
    for (int64_t i = threadIdx.x; i < n; i += kFacThreads) out[i] = s > 0.0 ? rp[i] * inv : 0.0;
    if (threadIdx.x < m) U[g.u_off + threadIdx.x + static_cast<int64_t>(r) * m] = Us[threadIdx.x + p * m];
    if (threadIdx.x == 0) S[g.s_off + r] = s;
  }
}

unsigned grid_1d(int64_t n) {
  const int64_t g = (n + 255) / 256;
  return static_cast<unsigned>(g < 1 ? 1 : (g > 148 * 32 ? 148 * 32 : g));
}

}  // namespace

// Panels of 32 reflectors up to 512 rows, of 16 up to 1024 (a warp's columns
// have to stay in registers); 0 = one reflector at a time.
int householder_panel(int64_t m) { return m <= 512 ? 32 : m <= kPanelRows ? 16 : 0; }

int64_t householder_scalars(int64_t m, int64_t n) {
  const int64_t k = std::min(m, n);
  const int nb = householder_panel(m);
  return nb > 0 ? (k + nb - 1) / nb * kPanelMax * kPanelMax : k;
}

cudaError_t launch_householder_qr(double* M, int64_t m, int64_t n, double* tau, cudaStream_t s, int64_t* launches) {
  const int64_t k = std::min(m, n);
  if (const int nb = householder_panel(m); nb > 0) {
    for (int64_t p0 = 0; p0 < k; p0 += nb) {
      const int pb = static_cast<int>(std::min<int64_t>(nb, k - p0)), mi = static_cast<int>(m), pi = static_cast<int>(p0);
      double* T = tau + p0 / nb * kPanelMax * kPanelMax;
      const int64_t rows = m - p0;
      if (nb == 16) k_house_panel<32, 1><<<1, kPanelThreads, 0, s>>>(M, m, mi, pi, pb, T);
      else if (rows <= 128) k_house_panel<4, 2><<<1, kPanelThreads, 0, s>>>(M, m, mi, pi, pb, T);
      else if (rows <= 256) k_house_panel<8, 2><<<1, kPanelThreads, 0, s>>>(M, m, mi, pi, pb, T);
      else if (rows <= 384) k_house_panel<12, 2><<<1, kPanelThreads, 0, s>>>(M, m, mi, pi, pb, T);
      else k_house_panel<16, 2><<<1, kPanelThreads, 0, s>>>(M, m, mi, pi, pb, T);
      ++*launches;
      const int64_t nc = n - p0 - pb;
      if (nc > 0x7fffffffLL) return cudaErrorInvalidValue;
      if (nc > 0) {
        k_house_block<<<static_cast<unsigned>(nc), kFacThreads, 0, s>>>(M, m, mi, pi, pb, pi + pb, T);
        ++*launches;
      }
    }
    return cudaGetLastError();
  }
  for (int64_t j = 0; j < k; ++j) {
    k_house_gen<<<1, kFacThreads, 0, s>>>(M, m, m, j, tau);
    ++*launches;
    const int64_t nc = n - j - 1;
    for (int64_t c = 0; c < nc; c += 65535) {
      const unsigned g = static_cast<unsigned>(std::min<int64_t>(65535, nc - c));
      k_house_apply<<<g, kFacThreads, 0, s>>>(M, m, M, m, m, j, j + 1 + c, tau);
      ++*launches;
    }
  }
  return cudaGetLastError();
}

cudaError_t launch_householder_form_q(const double* M, int64_t m, int64_t k, const double* tau, double* Q,
                                      cudaStream_t s, int64_t* launches) {
  if (m <= 0 || k <= 0) return cudaSuccess;
  if (const int nb = householder_panel(m); nb > 0) {
    k_house_q<<<static_cast<unsigned>(k), kFacThreads, 0, s>>>(M, m, static_cast<int>(m), nb, tau, Q);
    ++*launches;
    return cudaGetLastError();
  }
  k_identity_cols<<<grid_1d(m * k), 256, 0, s>>>(Q, m, k);
  ++*launches;
  for (int64_t j = k - 1; j >= 0; --j) {
    const int64_t nc = k - j;
    for (int64_t c = 0; c < nc; c += 65535) {
      const unsigned g = static_cast<unsigned>(std::min<int64_t>(65535, nc - c));
      k_house_apply<<<g, kFacThreads, 0, s>>>(M, m, Q, m, m, j, j + c, tau);
      ++*launches;
    }
  }
  return cudaGetLastError();
}

cudaError_t launch_upper(const double* M, int64_t m, int64_t k, int64_t n, double* R, cudaStream_t s) {
  if (k <= 0 || n <= 0) return cudaSuccess;
  k_upper<<<grid_1d(k * n), 256, 0, s>>>(M, m, k, n, R);
  return cudaGetLastError();
}

cudaError_t launch_gather_2d(const double* src, double* dst, const double* scale, const Gather2D* d_items, int64_t n,
                             int64_t max_elems, cudaStream_t s) {
  if (n <= 0 || max_elems <= 0) return cudaSuccess;
  if (max_elems <= 64 && (n + 7) / 8 <= 0x7fffffffLL) {
    k_gather_2d<true><<<static_cast<unsigned>((n + 7) / 8), 256, 0, s>>>(src, dst, scale, d_items, n);
    return cudaGetLastError();
  }
  for (int64_t b = 0; b < n; b += 65535) {
    const unsigned gy = static_cast<unsigned>(std::min<int64_t>(65535, n - b));
    const unsigned gx = static_cast<unsigned>(std::min<int64_t>((max_elems + 255) / 256, 64));
    k_gather_2d<false><<<dim3(gx, gy), 256, 0, s>>>(src, dst, scale, d_items + b, gy);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

cudaError_t launch_svd_rows(double* A, double* Vt, double* U, double* S, const SvdGroup* d_groups, int64_t ngroups,
                            int max_sweeps, int* d_status, cudaStream_t s) {
  if (ngroups <= 0) return cudaSuccess;
  if (ngroups > 0x7fffffffLL) return cudaErrorInvalidValue;
  k_svd_rows<<<static_cast<unsigned>(ngroups), kFacThreads, 0, s>>>(A, Vt, U, S, d_groups, max_sweeps, d_status);
  return cudaGetLastError();
}

}  // namespace sb
