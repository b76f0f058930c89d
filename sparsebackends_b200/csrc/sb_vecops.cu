// Vector-space kernels for Krylov solvers: chunked deterministic dot products,
// elementwise maps (axpy / axpby / copy / multiply), scale, fill and the
// key-union block add.  All HBM-bound; every floating-point step is an
// explicitly rounded double operation so results do not depend on contraction
// choices of the compiler, and reductions run in a fixed order so repeated
// calls give identical bits.
#include <algorithm>

#include "sb_kernels.hpp"

namespace sb {
namespace {

constexpr int kDotThreads = 256;

// One CTA per chunk: partial[c] = sum_t (s*x[t]) * (s*y[t]) in a fixed
// thread-stride-then-tree order.  chunks NULL: one contiguous segment of n
// elements.  The CTA that finishes last (by the counter, which it zeroes again)
// sums the partials, in an order that does not depend on which CTA it is, and
// writes the result to host memory: one launch and no copies per scalar, where
// the chunk upload, the second launch and the read-back made a dot product of
// two 1 MB vectors a 25 us round trip (nine of them in a Lanczos solve of three
// steps: chi = 512 947 us, now 789).
__global__ void __launch_bounds__(kDotThreads)
    k_dot(const double* __restrict__ X, const double* __restrict__ Y, const double* __restrict__ S,
          const DotChunk* __restrict__ chunks, int64_t n, double* partial, unsigned* counter, double* out) {
  __shared__ double red[1024];
  __shared__ bool last;
  DotChunk c;
  if (chunks) {
    c = chunks[blockIdx.x];
  } else {
    const int64_t o = static_cast<int64_t>(blockIdx.x) * kDotChunk;
    c = DotChunk{o, o, -1, static_cast<int32_t>(n - o < kDotChunk ? n - o : kDotChunk), 0};
  }
  const double* x = X + c.x_off;
  const double* y = Y + c.y_off;
  // a chunk is at most kDotChunk = 4 * kDotThreads elements: every thread
  // issues its (up to) four loads of each operand before the first FMA
  constexpr int kPer = kDotChunk / kDotThreads;
  double xv[kPer], yv[kPer];
#pragma unroll
  for (int r = 0; r < kPer; ++r) {
    const int t = threadIdx.x + r * kDotThreads;
    xv[r] = t < c.len ? x[t] : 0.0;
    yv[r] = t < c.len ? y[t] : 0.0;
  }
  const double sc = c.s_idx < 0 ? 1.0 : S[c.s_idx];
  double acc = 0.0;
#pragma unroll
  for (int r = 0; r < kPer; ++r)
    acc = c.s_idx < 0 ? __fma_rn(xv[r], yv[r], acc) : __fma_rn(__dmul_rn(sc, xv[r]), __dmul_rn(sc, yv[r]), acc);
  red[threadIdx.x] = acc;
  __syncthreads();
#pragma unroll
  for (int s = kDotThreads / 2; s > 0; s >>= 1) {
    if (threadIdx.x < s) red[threadIdx.x] = __dadd_rn(red[threadIdx.x], red[threadIdx.x + s]);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = red[0];
    __threadfence();
    last = atomicAdd(counter, 1u) + 1 == gridDim.x;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  // sum of the partials: 1024 strided sums, then a tree
  const int64_t np = gridDim.x;
#pragma unroll
  for (int r = 0; r < 1024 / kDotThreads; ++r) {
    const int v = threadIdx.x + r * kDotThreads;
    double a = 0.0;
    for (int64_t i = v; i < np; i += 1024) a = __dadd_rn(a, __ldcg(partial + i));
    red[v] = a;
  }
  __syncthreads();
  for (int s = 512; s > 0; s >>= 1) {
    for (int v = threadIdx.x; v < s; v += kDotThreads) red[v] = __dadd_rn(red[v], red[v + s]);
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    *out = red[0];
    *counter = 0;
  }
}

__global__ void k_map(double* __restrict__ R, const double* __restrict__ A, int64_t n, int op, double alpha,
                      double beta) {
  for (int64_t i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
       i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    const double r = R[i];
    const double a = A ? A[i] : 0.0;
    double v;
    switch (op) {
      case kMapAxpy: v = __dadd_rn(r, __dmul_rn(alpha, a)); break;
      case kMapAxpby: v = __dadd_rn(__dmul_rn(beta, r), __dmul_rn(alpha, a)); break;
      case kMapCopy: v = a; break;
      case kMapMul: v = __dmul_rn(r, a); break;
      case kMapScale: v = __dmul_rn(alpha, r); break;
      default: v = alpha; break;  // kMapFill
    }
    R[i] = v;
  }
}

// C block = A block (A only), 0 + B block (B only) or A + B (both): the
// rounding of copy(A) followed by `c += b` over a zero-initialised new block.
__global__ void k_add_blocks(const double* __restrict__ A, const double* __restrict__ B, double* __restrict__ C,
                             const AddBlock* __restrict__ items) {
  const AddBlock it = items[blockIdx.y];
  for (int64_t e = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < it.len;
       e += static_cast<int64_t>(gridDim.x) * blockDim.x) {
    double v;
    if (it.b_off < 0) v = A[it.a_off + e];
    else v = __dadd_rn(it.a_off >= 0 ? A[it.a_off + e] : 0.0, B[it.b_off + e]);
    C[it.c_off + e] = v;
  }
}

unsigned grid_1d(int64_t n, int threads) {
  const int64_t g = (n + threads - 1) / threads;
  return static_cast<unsigned>(g < 1 ? 1 : (g > 148 * 32 ? 148 * 32 : g));
}

}  // namespace

cudaError_t launch_dot(const double* X, const double* Y, const double* S, const DotChunk* d_chunks, int64_t nchunks,
                       int64_t n, double* d_partial, unsigned* d_counter, double* out, cudaStream_t s) {
  if (nchunks <= 0 || nchunks > 0x7fffffffLL) return cudaErrorInvalidValue;
  k_dot<<<static_cast<unsigned>(nchunks), kDotThreads, 0, s>>>(X, Y, S, d_chunks, n, d_partial, d_counter, out);
  return cudaGetLastError();
}

cudaError_t launch_map(double* R, const double* A, int64_t n, int op, double alpha, double beta, cudaStream_t s) {
  if (n <= 0) return cudaSuccess;
  k_map<<<grid_1d(n, 256), 256, 0, s>>>(R, A, n, op, alpha, beta);
  return cudaGetLastError();
}

cudaError_t launch_add_blocks(const double* A, const double* B, double* C, const AddBlock* d_items, int64_t n,
                              int64_t max_len, cudaStream_t s) {
  if (n <= 0 || max_len <= 0) return cudaSuccess;
  if (n > 65535) {
    // grid.y is limited to 65535: launch in slices of items
    for (int64_t b = 0; b < n; b += 65535) {
      const cudaError_t e = launch_add_blocks(A, B, C, d_items + b, std::min<int64_t>(65535, n - b), max_len, s);
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  }
  const unsigned gx = static_cast<unsigned>(std::min<int64_t>((max_len + 255) / 256, 64));
  k_add_blocks<<<dim3(gx, static_cast<unsigned>(n)), 256, 0, s>>>(A, B, C, d_items);
  return cudaGetLastError();
}

}  // namespace sb
