// Grouped FP64 block GEMM on the fifth-generation tensor cores, through exact
// 8-bit integer products (error-free splitting, after Ozaki, Ogita, Oishi and
// Rump, "Error-free transformations of matrix multiplication", Numer.
// Algorithms 59, 2012).
//
// Why: sm_100a has no FP64 tcgen05.mma; DMMA reaches 30 TFLOP/s on these block
// lists, while kind::i8 multiplies 8192 pairs per clock and SM.
//
// Same plan as the DMMA kernels (GemmCBlock / GemmPair).  Every row of X and
// every column of Y of a pair gets a power-of-two scale from its largest
// magnitude (2^E <= max < 2^(E+1), E one larger above mantissa 1.99), and each
// element becomes the integer rint(x * 2^(54-E)), |.| < 2^55: 53 significant
// bits and two more for the largest element.  In balanced radix 256 that is
// seven signed 8-bit digits d_0 (most significant) .. d_6.  Products of digits
// s and t weigh 256^(12-s-t); all products with s + t <= 7 are summed exactly
// in INT32 accumulators, one per s + t ("diagonal"), 34 of the 49.
//
// Error against |row||column| (2-norms), K the length of a pair's sum.  Worst
// case: each side's rounding, at most 1.01 * 2^-55 of the row's largest magnitude
// per element, adds up to 1.01 sqrt(K) 2^-55, and the digit products left out (at
// most 5 * 2^14 * 2^32 units of 2^-108 per element, and little more) to
// K 2^-59.6; rows of one large and many equal small entries come near it (x = y =
// (1, c, ..., c), c with digits of 127: 27, 58 and 154 times 2^-55 at K = 700,
// 1500 and 4000; bounds 82, 140 and 293).  With entries whose roundings and low
// digits are independent of each other the two parts stay below 2^-55 in the
// root mean square, where the sums of a DMMA chain round at about 2^-55 too.  It
// is not a bound against sum_k |x_k||y_k|, which DMMA keeps: the path runs only
// for callers that chose it (prepare_i8).
//
// Four diagonals combine into one
// 64-bit integer, which converts to FP64 exactly; the sum over the chunks of K
// and the pairs is in FP64.  Rows whose scale lies outside 2^+-400, infinities
// and NaN set *flag, and the launch that follows (launch_gemm_f64_fallback)
// then recomputes everything with DMMA; so it does when a bounded wait ran out.
//
// Kernels.  k_i8_rowmax finds the scales (one atomic maximum per row and
// k-tile, of the high words), k_i8_pack writes the seven digit planes of each
// 64-deep k-tile of each 128-row tile of X and nbs-column tile of Y in the
// layout the tensor core reads from shared memory (K-major, 64-byte swizzle),
// (rows of several C blocks that read the same Y blocks are stacked, I8Group); with
// every K at most 768 k_i8_pack_strip does both in one pass;
// k_gemm_i8 is persistent, one CTA per SM: warp 0 moves images with bulk
// copies, warp 1 issues the MMAs, warps 4-11 drain.  A tile is 128 x nb (nb <=
// 128, a multiple of 16).  INT32 accumulators of 128 columns for four diagonals
// fill the 512 TMEM columns, so every chunk runs in two passes over its
// k-tiles: diagonals 0-3 (10 products, four planes of each side) and 4-7 (24
// products, all planes).  One pass over all diagonals with 64-wide tiles would
// run the tensor core at 48 cycles per MMA instead of 32 (measured: 64 cycles
// at 128 columns, 60 at 112, 56 at 96, 48 at 64).
//
// What bounds it (psi*L of the chi = 2048 H_eff, clock64 per role): of 1.70 M
// clocks, MMA 1.22 M (0.98 M at 64 clocks each; the operands take all of the
// shared memory's 128 bytes per clock and the copies come on top), waits for
// the drain 0.38 M (reading the accumulators back runs at about 64 bytes per
// clock and SM; overlapping it with the next pass, diagonal by diagonal, made
// both slower: 1231 against 913 us), waits for copies 0.10 M.  Measured against
// DMMA: psi*L 1831 -> 913 us + 119 packing, R*T3 1911 -> 870 + 414; with the
// rows of C blocks that share Y stacked, 827 + 119 and 808 + 402.
#include <algorithm>
#include <atomic>

#include "sb_kernels.hpp"
#include "sb_tcgen05.cuh"

namespace sb {
namespace {

constexpr int kI8Planes = 7;
constexpr int kI8BK = 64;                      // k-tile: 64 digits = one 64-byte swizzle row
constexpr int kI8Plane = 128 * kI8BK;          // bytes of one 128-row plane
constexpr int kI8Side = kI8Planes * kI8Plane;  // bytes reserved for one operand of a stage
constexpr int kI8Stages = 2;
constexpr int kI8SmemBytes = kI8Stages * 2 * kI8Side + 1024 /*alignment*/ + 128 /*barriers*/;
constexpr int kI8DrainWarps = 8;
// Warpgroup 0: producer, MMA and two idle warps; warpgroups 1 and 2 drain.
// Register split of the block's 384 x 168: 128 x 72 + 256 x 216.
constexpr int kI8Threads = (4 + kI8DrainWarps) * 32;
constexpr int kI8RegsLaunch = 168, kI8RegsIssue = 72, kI8RegsDrain = 216;
static_assert(128 * kI8RegsIssue + 256 * kI8RegsDrain <= kI8Threads * kI8RegsLaunch, "register split");
static_assert(kI8SmemBytes <= 227 * 1024, "shared memory of the integer GEMM");

// Exponent of the row scale from the high word of the row's largest magnitude.
__device__ __forceinline__ int scale_exp(uint32_t hi) {
  return static_cast<int>(hi >> 20) - 1023 + ((hi & 0xFFFFFu) >= 0xFD70Au ? 1 : 0);
}

__device__ __forceinline__ uint32_t abs_hi(double x) {
  const uint64_t b = static_cast<uint64_t>(__double_as_longlong(x));
  const uint32_t hi = static_cast<uint32_t>(b >> 32) & 0x7FFFFFFFu;
  return hi == 0 && static_cast<uint32_t>(b) != 0 ? 1u : hi;  // the smallest subnormals count as nonzero
}

// 2^e, -1022 <= e <= 1023
__device__ __forceinline__ double pow2(int e) {
  return __longlong_as_double(static_cast<long long>(e + 1023) << 52);
}

// Largest magnitude (high word) of every row of one k-tile image.  HBM-bound:
// each element is read once, coalesced along its contiguous direction.
__global__ void __launch_bounds__(256)
    k_i8_rowmax(const double* __restrict__ src, const I8Image* __restrict__ imgs, uint32_t* __restrict__ rowhi) {
  __shared__ uint32_t half[128];
  const I8Image im = imgs[blockIdx.x];
  const int tid = static_cast<int>(threadIdx.x);
  const double* s = src + im.src;
  if (im.kc) {
    // 16 lanes per row, 16 rows per pass
    const int l = tid & 15;
    for (int r = tid >> 4; r < (im.rows + 15) / 16 * 16; r += 16) {
      uint32_t m = 0;
      if (r < im.rows) {
        const double* p = s + static_cast<int64_t>(r) * im.ld;
#pragma unroll
        for (int j = 0; j < kI8BK / 16; ++j) {
          const int k = l + 16 * j;
          if (k < im.kv) m = max(m, abs_hi(p[k]));
        }
      }
#pragma unroll
      for (int o = 8; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
      if (l == 0 && r < im.rows && m > 0) atomicMax(&rowhi[im.scale + r], m);
    }
    return;
  }
  const int r = tid & 127, h = tid >> 7;
  uint32_t m = 0;
  if (r < im.rows) {
    const double* p = s + r;
    const int k1 = min(im.kv, 32 * (h + 1));
#pragma unroll 8
    for (int k = 32 * h; k < k1; ++k) m = max(m, abs_hi(p[static_cast<int64_t>(k) * im.ld]));
  }
  if (h) half[r] = m;
  __syncthreads();
  if (!h && r < im.rows) {
    m = max(m, half[r]);
    if (m > 0) atomicMax(&rowhi[im.scale + r], m);
  }
}

// K-major 64-byte swizzle: byte of image row ri, chunk c of 16 k in its plane.
__device__ __forceinline__ int digit_at(int ri, int c) {
  return (ri >> 3) * 512 + (ri & 7) * 64 + ((c ^ ((ri >> 1) & 3)) << 4);
}

// Seven digits of a row's 16 consecutive k (largest magnitude hi) into the
// planes at o.
__device__ __forceinline__ void put_digits(double (&x)[16], uint32_t hi, bool store, unsigned char* o, int plane,
                                           int* flag) {
      double f = 0.0;
      if (hi != 0) {
        const int e = scale_exp(hi);
        if (e < -400 || e > 400) {
          *flag = 1;  // the DMMA launch recomputes (also infinities and NaN)
#pragma unroll
          for (int j = 0; j < 16; ++j) x[j] = 0.0;
        } else {
          f = pow2(54 - e);
        }
      }
      uint32_t w[kI8Planes][4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint32_t lo[4], up[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          // balanced digits: add 128 to each of the seven bytes, then take 128 off
          // again byte by byte (flip the top bit)
          const uint64_t v = (static_cast<uint64_t>(__double2ll_rn(__dmul_rn(x[4 * q + j], f))) + 0x0080808080808080ull) ^
                             0x0080808080808080ull;
          lo[j] = static_cast<uint32_t>(v);
          up[j] = static_cast<uint32_t>(v >> 32);
        }
        // 4 x 4 byte transposes: plane 6 holds the lowest byte of each value
        const uint32_t a0 = __byte_perm(lo[0], lo[1], 0x5140), a1 = __byte_perm(lo[0], lo[1], 0x7362);
        const uint32_t b0 = __byte_perm(lo[2], lo[3], 0x5140), b1 = __byte_perm(lo[2], lo[3], 0x7362);
        w[6][q] = __byte_perm(a0, b0, 0x5410);
        w[5][q] = __byte_perm(a0, b0, 0x7632);
        w[4][q] = __byte_perm(a1, b1, 0x5410);
        w[3][q] = __byte_perm(a1, b1, 0x7632);
        const uint32_t c0 = __byte_perm(up[0], up[1], 0x5140), c1 = __byte_perm(up[0], up[1], 0x7362);
        const uint32_t d0 = __byte_perm(up[2], up[3], 0x5140), d1 = __byte_perm(up[2], up[3], 0x7362);
        w[2][q] = __byte_perm(c0, d0, 0x5410);
        w[1][q] = __byte_perm(c0, d0, 0x7632);
        w[0][q] = __byte_perm(c1, d1, 0x5410);
      }
  if (store)
#pragma unroll
    for (int q = 0; q < kI8Planes; ++q) st_global_v4(o + q * plane, w[q][0], w[q][1], w[q][2], w[q][3]);
}

// Digit planes of one k-tile image: a warp takes 8 rows, lane = 4*row + chunk
// of 16 k, so that its 16-byte stores cover 512 contiguous bytes per plane.
// k-contiguous rows go through a shared-memory copy (loads coalesced along k;
// the index 68*row + 17*chunk + j is free of bank conflicts both ways).
__global__ void __launch_bounds__(256)
    k_i8_pack(const double* __restrict__ src, const I8Image* __restrict__ imgs, const uint32_t* __restrict__ rowhi,
              unsigned char* __restrict__ dst, int* __restrict__ flag) {
  __shared__ double stage[8][8 * 68];
  const I8Image im = imgs[blockIdx.x];
  const int warp = static_cast<int>(threadIdx.x) >> 5, lane = static_cast<int>(threadIdx.x) & 31;
  const int plane = im.rows_img * kI8BK;
  unsigned char* const d = dst + im.dst;
  for (int g = im.row0 / 8 + warp; 8 * g < im.row_end; g += 8) {
    const int rl = lane >> 2, c = lane & 3;
    const int ri = 8 * g + rl, r = ri - im.row0;  // row of the image, of the block
    const double* s = src + im.src;
    double x[16];
    if (im.kc) {
      double* st = stage[warp];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int rr = 8 * g + q - im.row0;
        const double* p = s + static_cast<int64_t>(rr) * im.ld;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int k = lane + 32 * h;
          st[68 * q + 17 * (k >> 4) + (k & 15)] = rr >= 0 && rr < im.rows && k < im.kv ? p[k] : 0.0;
        }
      }
      __syncwarp();
#pragma unroll
      for (int j = 0; j < 16; ++j) x[j] = st[68 * rl + 17 * c + j];
      __syncwarp();
    } else {
      const double* p = s + r + static_cast<int64_t>(16 * c) * im.ld;
#pragma unroll
      for (int j = 0; j < 16; ++j)
        x[j] = r >= 0 && r < im.rows && 16 * c + j < im.kv ? p[static_cast<int64_t>(j) * im.ld] : 0.0;
    }
    const uint32_t hi = r >= 0 && r < im.rows ? rowhi[im.scale + r] : 0u;
    put_digits(x, hi, r >= 0 && ri < im.row_end, d + digit_at(ri, c), plane, flag);
  }
}

// Doubles from one row of a strip to the next in shared memory.
__host__ __device__ constexpr int strip_stride(int k) {
  const int n = (k + kI8BK - 1) / kI8BK;
  return 68 * n + ((4 - 4 * n) & 15);
}

__device__ __forceinline__ void cp_async8(double* smem, const double* g) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(smem))),
               "l"(g)
               : "memory");
}

// The same for strips: up to 16 image rows and all of their K, which is in
// shared memory while the scales are found and the digits written, so that HBM
// is read once and one launch does both.  Element (r, k) lies at r*ss + (r >> 2)
// + k + (k >> 4), ss = 4 modulo 16: no bank conflicts for 16 rows of one k, for
// a row's consecutive k, or for 4 rows x 4 chunks.  The issue of the conversion
// and the phases' latencies bound it (a double-buffered persistent form was
// slower, 163 us), not HBM: the packs of psi*L at chi = 2048 119 -> 103 us, 1400
// 74 -> 57, 1024 51 -> 40.
__global__ void __launch_bounds__(256)
    k_i8_pack_strip(const double* __restrict__ src, const I8Image* __restrict__ imgs, uint32_t* __restrict__ rowhi,
                    unsigned char* __restrict__ dst, int* __restrict__ flag) {
  extern __shared__ double strip[];
  __shared__ uint32_t top[8 * 16];
  const I8Image im = imgs[blockIdx.x];
  const int tid = static_cast<int>(threadIdx.x), warp = tid >> 5, lane = tid & 31;
  const int nkt = (im.kv + kI8BK - 1) / kI8BK, ss = strip_stride(im.kv);
  const int r16 = tid & 15;
  const double* s = src + im.src;
  if (im.kc) {
    for (int r = warp; r < im.rows; r += 8) {
      const double* p = s + static_cast<int64_t>(r) * im.ld;
      double* q = strip + r * ss + (r >> 2);
#pragma unroll 4
      for (int k = lane; k < im.kv; k += 32) cp_async8(q + k + (k >> 4), p + k);
    }
  } else if (r16 < im.rows) {
    double* q = strip + r16 * ss + (r16 >> 2);
#pragma unroll 4
    for (int k = tid >> 4; k < im.kv; k += 16) cp_async8(q + k + (k >> 4), s + r16 + static_cast<int64_t>(k) * im.ld);
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
  __syncthreads();
  uint32_t m = 0;
  if (r16 < im.rows) {
    const double* q = strip + r16 * ss + (r16 >> 2);
#pragma unroll 4
    for (int k = tid >> 4; k < im.kv; k += 16) m = max(m, abs_hi(q[k + (k >> 4)]));
  }
  m = max(m, __shfl_xor_sync(0xffffffffu, m, 16));
  if (lane < 16) top[16 * warp + lane] = m;
  __syncthreads();
  if (tid < 16) {
    for (int j = 1; j < 8; ++j) m = max(m, top[16 * j + tid]);
    top[tid] = m;
    if (tid < im.rows) rowhi[im.scale + tid] = m;
  }
  __syncthreads();
  const int plane = im.rows_img * kI8BK;
  const int g0 = im.row0 / 8, ng = (im.row_end + 7) / 8 - g0;
  for (int u = warp; u < ng * nkt; u += 8) {
    const int kt = u / ng, rl = lane >> 2, c = lane & 3;
    const int ri = 8 * (g0 + u - kt * ng) + rl, r = ri - im.row0, k0 = kt * kI8BK + 16 * c;
    const bool own = r >= 0 && r < im.rows;
    const double* p = strip + r * ss + (r >> 2) + k0 + (k0 >> 4);
    double x[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) x[j] = own && k0 + j < im.kv ? p[j] : 0.0;
    put_digits(x, own ? top[r] : 0u, r >= 0 && ri < im.row_end,
               dst + im.dst + static_cast<int64_t>(kt) * kI8Planes * plane + digit_at(ri, c), plane, flag);
  }
}

// Shared-memory descriptor of a K-major SWIZZLE_64B image: stride 512 bytes
// between 8-row groups, descriptor version 1, layout type 4.  A 32-deep step
// along K adds 32 bytes.
__device__ __forceinline__ uint64_t desc_sw64(uint32_t addr) {
  return static_cast<uint64_t>((addr & 0x3FFFFu) >> 4) | (1ull << 16) | (32ull << 32) | (1ull << 46) | (4ull << 61);
}

// Instruction descriptor of kind::i8: S32 accumulator, both operands signed
// 8-bit and K-major, M = 128, N = n (a multiple of 16).
__device__ __forceinline__ uint32_t idesc_i8(int n) {
  return (2u << 4) | (1u << 7) | (1u << 10) | (static_cast<uint32_t>(n >> 3) << 17) | ((128u >> 4) << 24);
}

__device__ __forceinline__ void mma_i8(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, int32_t (&v)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, "
      "%15}, [%16];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
        "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
      : "r"(taddr));
}

// d * M + c in 64 bits, one instruction (the drain's inner loop).
template <int M>
__device__ __forceinline__ long long mad_wide(int32_t d, long long c) {
  long long r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(d), "n"(M), "l"(c));
  return r;
}

// All products of the diagonals [LO, LO + 4) of one 64-deep k-tile.
// first: the tile that opens the accumulators (the first product of each
// diagonal overwrites).
template <int LO>
__device__ __forceinline__ void issue_ktile(uint32_t tmem, uint32_t sa, uint32_t sb, uint32_t bstride, uint32_t idesc,
                                            bool first) {
  // descriptors differ in their low words only (addresses below 2^18)
  const uint64_t dhi = desc_sw64(0);
  uint32_t open = first ? 0u : 1u;
#pragma unroll 1
  for (int k = 0; k < kI8BK / 32; ++k) {
    const uint32_t a = (sa + 32 * k) >> 4, b = (sb + 32 * k) >> 4;
#pragma unroll
    for (int d = LO; d < LO + 4; ++d) {
#pragma unroll
      for (int s = 0; s < kI8Planes; ++s) {
        const int t = d - s;
        if (t < 0 || t >= kI8Planes) continue;
        const bool opens = s == (d >= kI8Planes ? d - kI8Planes + 1 : 0);
        mma_i8(tmem + (d - LO) * 128, dhi | (a + (s * kI8Plane >> 4)), dhi | (b + t * bstride), idesc,
               opens ? open : 1u);
      }
    }
    open = 1u;
  }
}

__global__ void __launch_bounds__(kI8Threads, 1)
    k_gemm_i8(const unsigned char* __restrict__ pack, double* __restrict__ C, const I8Group* __restrict__ groups,
              const int64_t* __restrict__ row_off, const int32_t* __restrict__ row_ld, const I8Pack* __restrict__ packs, const uint32_t* __restrict__ rowhi, const TcTile* __restrict__ tiles,
              const int32_t* __restrict__ first, int32_t ntiles, int32_t nz_begin, double* __restrict__ partial,
              int* __restrict__ flag) {
  extern __shared__ unsigned char smem_raw[];
  const int tid = static_cast<int>(threadIdx.x);
  const int warp = tid >> 5, lane = tid & 31;
  const uint32_t raw = smem_u32(smem_raw);
  const uint32_t base = (raw + 1023u) & ~1023u;
  const uint32_t bars = base + kI8Stages * 2 * kI8Side;
  const uint32_t bar_full0 = bars, bar_empty0 = bars + 16, bar_accf = bars + 32, bar_acce = bars + 40;
  const uint32_t tmem_slot = bars + 48;
  unsigned char* const tmem_slot_ptr = smem_raw + (tmem_slot - raw);
  const int grid = static_cast<int>(gridDim.x);
  const int t0 = first[blockIdx.x], t1 = first[blockIdx.x + 1];  // this CTA's items

  if (tid == 0) {
    for (int s = 0; s < kI8Stages; ++s) {
      mbar_init(bar_full0 + 8 * s, 1);
      mbar_init(bar_empty0 + 8 * s, 1);
    }
    mbar_init(bar_accf, 1);
    mbar_init(bar_acce, kI8DrainWarps);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(tmem_slot));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(tmem_slot_ptr);

  // The k-tiles of an item in chunks: within one pair, cut at multiples of
  // kI8Chunk k-tiles of the pair (so the cuts do not depend on the item), the
  // accumulators' bound.  Every role walks the same chunks, each in two passes.
  struct Walk {
    int p, j, rem;  // pair, k-tile inside it, k-tiles left in the item
    __device__ int len(int nkt) const { return min(min(rem, nkt - j), kI8Chunk - j % kI8Chunk); }
    __device__ void step(int l, int nkt) {
      rem -= l;
      j += l;
      if (j >= nkt) {
        ++p;
        j = 0;
      }
    }
  };

  if (warp < 4) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kI8RegsIssue));
    if (warp == 0 && lane == 0) {
      bool failed = false;
      uint32_t g = 0;
      for (int t = t0; t < t1 && !failed; ++t) {
        const TcTile tl = tiles[t];
        for (Walk w{tl.p0, tl.k0 / kI8BK, tl.nkt}; w.rem > 0 && !failed;) {
          const I8Pack pk = packs[w.p];
          const int len = w.len(pk.nkt);
          const int64_t bimg = static_cast<int64_t>(kI8Planes) * pk.nbs * kI8BK;
          const unsigned char* ga = pack + pk.a_base + (static_cast<int64_t>(tl.a0 >> 7) * pk.nkt + w.j) * kI8Side;
          const unsigned char* gb = pack + pk.b_base + (static_cast<int64_t>(tl.b0 / pk.nbs) * pk.nkt + w.j) * bimg;
          for (int pass = 0; pass < 2 && !failed; ++pass) {
            const uint32_t np = pass == 0 ? 4u : static_cast<uint32_t>(kI8Planes);
            const uint32_t abytes = np * kI8Plane, bbytes = np * static_cast<uint32_t>(pk.nbs) * kI8BK;
            for (int i = 0; i < len; ++i, ++g) {
              const uint32_t s = g % kI8Stages;
              if (g >= kI8Stages) failed = !mbar_wait(bar_empty0 + 8 * s, ((g / kI8Stages) - 1) & 1, flag);
              if (failed) break;
              const uint32_t sa = base + s * 2 * kI8Side, full = bar_full0 + 8 * s;
              mbar_expect_tx(full, abytes + bbytes);
              bulk_g2s(sa, ga + static_cast<int64_t>(i) * kI8Side, abytes, full);
              bulk_g2s(sa + kI8Side, gb + i * bimg, bbytes, full);
            }
          }
          w.step(len, pk.nkt);
        }
      }
      // copies still in flight land before the CTA exits
      for (uint32_t q = g > kI8Stages ? g - kI8Stages : 0; q < g; ++q)
        mbar_wait(bar_full0 + 8 * (q % kI8Stages), (q / kI8Stages) & 1, flag);
    }
    if (warp == 1 && lane == 0) {
      bool failed = false;
      uint32_t g = 0, np = 0;  // stages, passes
      for (int t = t0; t < t1 && !failed; ++t) {
        const TcTile tl = tiles[t];
        const uint32_t idesc = idesc_i8(tl.nb);
        for (Walk w{tl.p0, tl.k0 / kI8BK, tl.nkt}; w.rem > 0 && !failed;) {
          const int nkt = packs[w.p].nkt;
          const uint32_t bstride = static_cast<uint32_t>(packs[w.p].nbs) * kI8BK >> 4;
          const int len = w.len(nkt);
          for (int pass = 0; pass < 2 && !failed; ++pass, ++np) {
            if (np >= 1) failed = !mbar_wait(bar_acce, (np - 1) & 1, flag);
            for (int i = 0; i < len && !failed; ++i, ++g) {
              const uint32_t s = g % kI8Stages;
              failed = !mbar_wait(bar_full0 + 8 * s, (g / kI8Stages) & 1, flag);
              if (failed) break;
              tc_fence_after();
              const uint32_t sa = base + s * 2 * kI8Side;
              if (pass == 0) issue_ktile<0>(tmem, sa, sa + kI8Side, bstride, idesc, i == 0);
              else issue_ktile<4>(tmem, sa, sa + kI8Side, bstride, idesc, i == 0);
              mma_commit(bar_empty0 + 8 * s);
            }
            if (!failed) mma_commit(bar_accf);
          }
          w.step(len, nkt);
        }
      }
    }
  } else {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kI8RegsDrain));
    // warp w drains TMEM lanes 32*(w % 4).. (rows) and columns [64h, 64h + 64)
    bool failed = false;
    const int q = warp & 3, h = (warp - 4) >> 2;
    const uint32_t lanes = static_cast<uint32_t>(32 * q) << 16;
    uint32_t np = 0;
    for (int t = t0; t < t1; ++t) {
      const TcTile tl = tiles[t];
      const I8Group gr = groups[tl.cb];
      const int row = tl.a0 + 32 * q + lane;
      const int cols = min(tl.nb, gr.N - tl.b0) - 64 * h;  // valid columns of this warp (may be <= 0)
      const bool row_ok = row < gr.rows;
      const int64_t c_off = row_ok ? row_off[gr.row0 + row] : 0;
      const int c_ld = row_ok ? row_ld[gr.row0 + row] : 0;
      double acc[64];
#pragma unroll
      for (int j = 0; j < 64; ++j) acc[j] = 0.0;
      for (Walk w{tl.p0, tl.k0 / kI8BK, tl.nkt}; w.rem > 0;) {
        const I8Pack pk = packs[w.p];
        const int len = w.len(pk.nkt);
        const uint32_t* ch = rowhi + pk.b_sc + tl.b0 + 64 * h;
        // scale exponents (rows the flag reports may be anything), the columns'
        // in lanes and shifted to the exponent's place in a high word
        auto ex = [](uint32_t hi) { return hi == 0 ? 0 : min(max(scale_exp(hi), -401), 401); };
        const int ea = ex(row_ok ? rowhi[pk.a_sc + row] : 0u);
        const int eb0 = (lane < cols ? ex(ch[lane]) : 0) * (1 << 20), eb1 = (lane + 32 < cols ? ex(ch[lane + 32]) : 0) * (1 << 20);
        for (int pass = 0; pass < 2; ++pass, ++np) {
          if (!failed) failed = __any_sync(0xffffffffu, !mbar_wait(bar_accf, np & 1, flag));
          tc_fence_after();
          const uint32_t acc0 = tmem + static_cast<uint32_t>(64 * h) + lanes;
          const int ehi = (ea + (pass == 0 ? -36 : -68) + 1023) * (1 << 20);
#pragma unroll
          for (int gp = 0; gp < 4; ++gp) {
            if (16 * gp < cols) {
              int32_t v4[4][16];
#pragma unroll
              for (int q4 = 0; q4 < 4; ++q4) tmem_ld16(acc0 + 128 * q4 + 16 * gp, v4[q4]);
              tmem_wait_ld();
#pragma unroll
              for (int j = 0; j < 16; ++j) {
                // the four diagonals as one integer below 2^51, made a double by
                // adding it to the bits of 1.5 * 2^52
                long long v = mad_wide<1>(v4[3][j], 0x4338000000000000ll);
                v = mad_wide<1 << 8>(v4[2][j], v);
                v = mad_wide<1 << 16>(v4[1][j], v);
                v = mad_wide<1 << 24>(v4[0][j], v);
                const double x = __dadd_rn(__longlong_as_double(v), -6755399441055744.0);
                const int e = ehi + __shfl_sync(0xffffffffu, gp < 2 ? eb0 : eb1, (16 * gp + j) & 31);
                acc[16 * gp + j] = __fma_rn(x, __hiloint2double(e, 0), acc[16 * gp + j]);
              }
            }
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(bar_acce);
        }
        w.step(len, pk.nkt);
      }
      if (!row_ok || failed) continue;
      if (tl.part >= 0) {
        double* pt = partial + static_cast<int64_t>(tl.part) * kI8PartElems + (64 * h) * 128 + 32 * q + lane;
#pragma unroll
        for (int j = 0; j < 64; ++j)
          if (j < cols) pt[j * 128] = acc[j];
      } else {
        double* c = C + c_off + static_cast<int64_t>(tl.b0 + 64 * h) * c_ld;
#pragma unroll
        for (int j = 0; j < 64; ++j) {
          if (j < cols) *c = acc[j];
          c += c_ld;
        }
      }
    }
    // C blocks without pairs (items [nz_begin, ntiles)): zeros
    for (int t = nz_begin + static_cast<int>(blockIdx.x); t < ntiles; t += grid) {
      const TcTile tl = tiles[t];
      const I8Group gr = groups[tl.cb];
      const int rows = min(128, gr.rows - tl.a0), cols = min(tl.nb, gr.N - tl.b0);
      for (int e = tid - 128; e < rows * cols; e += 32 * kI8DrainWarps) {
        const int r = gr.row0 + tl.a0 + e % rows;
        C[row_off[r] + static_cast<int64_t>(tl.b0 + e / rows) * row_ld[r]] = 0.0;
      }
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
  }
}

// Sum of the k-segment partial tiles of split tiles, in segment order.  One
// CTA per (split tile, 32 columns), reads and writes coalesced along the rows.
__global__ void __launch_bounds__(256) k_i8_reduce(const double* __restrict__ partial, double* __restrict__ C,
                                                   const I8Group* __restrict__ groups,
                                                   const int64_t* __restrict__ row_off,
                                                   const int32_t* __restrict__ row_ld,
                                                   const TcSplit* __restrict__ splits) {
  const TcSplit sp = splits[blockIdx.x >> 2];
  const int c0 = 32 * static_cast<int>(blockIdx.x & 3);
  const I8Group gr = groups[sp.cb];
  const int r = static_cast<int>(threadIdx.x) & 127, row = sp.a0 + r;
  const int cols = min(min(sp.nb, gr.N - sp.b0) - c0, 32);
  if (row >= gr.rows) return;
  const int64_t c_off = row_off[gr.row0 + row];
  const int c_ld = row_ld[gr.row0 + row];
  for (int c = static_cast<int>(threadIdx.x) >> 7; c < cols; c += 2) {
    const double* p = partial + static_cast<int64_t>(sp.part0) * kI8PartElems + r + (c0 + c) * 128;
    double acc = 0.0;
    for (int q = 0; q < sp.nparts; q += 4) {  // four loads in flight, added in segment order
      double v[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) v[j] = q + j < sp.nparts ? p[(q + j) * kI8PartElems] : 0.0;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (q + j < sp.nparts) acc = __dadd_rn(acc, v[j]);
    }
    C[c_off + static_cast<int64_t>(sp.b0 + c0 + c) * c_ld] = acc;
  }
}

// One CTA per block / run; latency-bound, a few microseconds once per plan.
__global__ void __launch_bounds__(256) k_i8_entries(const I8Block* __restrict__ blocks, I8Image* __restrict__ imgs) {
  const I8Block b = blocks[blockIdx.x];
  const int n = i8_entries(b);
  for (int p = static_cast<int>(threadIdx.x); p < n; p += 256) imgs[b.first + p] = i8_entry(b, p);
}

__global__ void __launch_bounds__(256) k_i8_rows(const I8RowRun* __restrict__ runs, int64_t* __restrict__ row_off,
                                                 int32_t* __restrict__ row_ld) {
  const I8RowRun q = runs[blockIdx.x];
  for (int r = static_cast<int>(threadIdx.x); r < q.M; r += 256) {
    row_off[q.row0 + r] = q.c_off + r;
    row_ld[q.row0 + r] = q.ldc;
  }
}

}  // namespace

cudaError_t launch_i8_entries(const I8Block* d_blocks, int64_t nblocks, I8Image* d_imgs, cudaStream_t s) {
  if (nblocks <= 0) return cudaSuccess;
  if (nblocks > 0x7fffffffLL) return cudaErrorInvalidValue;
  k_i8_entries<<<static_cast<unsigned>(nblocks), 256, 0, s>>>(d_blocks, d_imgs);
  return cudaGetLastError();
}

cudaError_t launch_i8_rows(const I8RowRun* d_runs, int64_t nruns, int64_t* d_row_off, int32_t* d_row_ld,
                           cudaStream_t s) {
  if (nruns <= 0) return cudaSuccess;
  if (nruns > 0x7fffffffLL) return cudaErrorInvalidValue;
  k_i8_rows<<<static_cast<unsigned>(nruns), 256, 0, s>>>(d_runs, d_row_off, d_row_ld);
  return cudaGetLastError();
}

cudaError_t launch_i8_pack(const double* src, const I8Image* d_imgs, int64_t nimg, int32_t strip_k, uint32_t* d_rowhi,
                           void* dst, int* d_flag, cudaStream_t s) {
  if (nimg <= 0) return cudaSuccess;
  if (nimg > 0x7fffffffLL || strip_k > kI8StripK) return cudaErrorInvalidValue;
  const unsigned g = static_cast<unsigned>(nimg);
  unsigned char* const d = static_cast<unsigned char*>(dst);
  if (strip_k > 0) {
    auto smem = [](int k) { return static_cast<size_t>(16 * strip_stride(k) + 4) * sizeof(double); };
    static std::atomic<unsigned long long> configured{0};  // as in launch_gemm_i8
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(configured & bit)) {
      e = cudaFuncSetAttribute(k_i8_pack_strip, cudaFuncAttributeMaxDynamicSharedMemorySize,
                               static_cast<int>(smem(kI8StripK)));
      if (e != cudaSuccess) return e;
      configured.fetch_or(bit);
    }
    k_i8_pack_strip<<<g, 256, smem(strip_k), s>>>(src, d_imgs, d_rowhi, d, d_flag);
    return cudaGetLastError();
  }
  k_i8_rowmax<<<g, 256, 0, s>>>(src, d_imgs, d_rowhi);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return e;
  k_i8_pack<<<g, 256, 0, s>>>(src, d_imgs, d_rowhi, d, d_flag);
  return cudaGetLastError();
}

cudaError_t launch_gemm_i8(const void* pack, double* C, const I8Group* d_groups, const int64_t* d_row_off,
                           const int32_t* d_row_ld, const I8Pack* d_packs, const uint32_t* d_rowhi,
                           const TcTile* d_tiles, const int32_t* d_first, int32_t nctas, int32_t ntiles,
                           int32_t nz_begin, double* d_partial, const TcSplit* d_splits, int32_t nsplits, int* d_flag,
                           cudaStream_t s) {
  if (ntiles <= 0) return cudaSuccess;
  if (nctas < 1 || (nsplits > 0 && (!d_partial || !d_splits))) return cudaErrorInvalidValue;
  static std::atomic<unsigned long long> configured{0};  // one bit per device ordinal (host threads may race)
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return e;
  const unsigned long long bit = 1ull << (dev & 63);
  if (!(configured & bit)) {
    e = cudaFuncSetAttribute(k_gemm_i8, cudaFuncAttributeMaxDynamicSharedMemorySize, kI8SmemBytes);
    if (e != cudaSuccess) return e;
    configured.fetch_or(bit);
  }
  const unsigned g = static_cast<unsigned>(nctas);
  k_gemm_i8<<<g, kI8Threads, kI8SmemBytes, s>>>(static_cast<const unsigned char*>(pack), C, d_groups, d_row_off,
                                                d_row_ld, d_packs, d_rowhi, d_tiles, d_first, ntiles, nz_begin, d_partial, d_flag);
  e = cudaGetLastError();
  if (e != cudaSuccess || nsplits <= 0) return e;
  k_i8_reduce<<<static_cast<unsigned>(nsplits) * 4, 256, 0, s>>>(d_partial, C, d_groups, d_row_off,
                                                                   d_row_ld, d_splits);
  return cudaGetLastError();
}

}  // namespace sb
