// Digit-slice packing of the exact-slice products (gemm_oz.cu): a strided FP64
// source becomes R rows of S slices of Kpad BF16 digits, each row scaled by
// the power of two above its largest element.  The source is gathered through
// the operand's strides, so the index permutation of a contraction costs
// nothing extra.
//
// HBM bound: 8 bytes read and 2 S written per element.  The row exponent is
// needed before the first digit, so where a row's share fits, one kernel reads
// it once into registers or shared memory (k the faster source index, up to 4096
// and 14080 columns) or into the shared memory of a block or cluster (row index
// faster, up to 176 and 1536 columns), reduces the exponent and cuts from there;
// longer rows, and few long ones, take an exponent pass of their own.
#include <cuda_bf16.h>

#include <algorithm>

#include "fcc_tc.cuh"
#include "fcc_tcgen05.cuh"

namespace fcc {

namespace {

constexpr int OZ_BK = 64;
constexpr int TILE_KMAX = 176;      // fused transposing pack: 33 x 176 doubles of shared memory (46 KB)

// frexp-style exponent of the row scale from the stored biased exponent
__device__ __forceinline__ int oz_row_exp(int be) { return be ? be - 1022 : 0; }

__device__ __forceinline__ int biased_exp(double x) { return (int)((__double_as_longlong(x) >> 52) & 0x7FF); }

// ex[r] = max over the row of the biased exponent (ex zeroed before), for
// sources whose k index is the faster one: a warp per (row, k-slab), each
// lane reading 4 consecutive k at a time
__global__ void __launch_bounds__(256) oz_exp_rows_kernel(const double* __restrict__ src, PackSpec ps, int64_t kslab,
                                                          int* __restrict__ ex) {
  const int lane = threadIdx.x & 31;
  const int64_t nks = (ps.K + kslab - 1) / kslab;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const bool k1 = pack_k_single(ps);
  for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < ps.R * nks; w += nw) {
    const int64_t r = w / nks, ka = (w % nks) * kslab, kb = min(ps.K, ka + kslab);
    const int64_t ro = pack_row_off(ps, r);
    int m = 0;
    for (int64_t k0 = ka + 4 * lane; k0 < kb; k0 += 128) {
      double xv[4];
      pack_load4(src, ps, k1, ro, k0, (int)min((int64_t)4, kb - k0), xv);
#pragma unroll
      for (int q = 0; q < 4; ++q) m = max(m, biased_exp(xv[q]));
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if (lane == 0 && m > 0) atomicMax(ex + r, m);
  }
}

// same for sources whose row index is the faster one: 32 rows x 8 k-lanes
// per block over one k-slab, the column offsets of each 32-column step in
// shared memory
__global__ void __launch_bounds__(256) oz_exp_tiles_kernel(const double* __restrict__ src, PackSpec ps, int64_t kslab,
                                                           int* __restrict__ ex) {
  __shared__ int red[8][32];
  __shared__ int64_t coff[32];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int64_t nrt = (ps.R + 31) / 32, nks = (ps.K + kslab - 1) / kslab;
  for (int64_t tb = blockIdx.x; tb < nrt * nks; tb += gridDim.x) {
    const int64_t r = (tb / nks) * 32 + tx;
    const int64_t ka = (tb % nks) * kslab, kb = min(ps.K, ka + kslab);
    const int64_t ro = r < ps.R ? pack_row_off(ps, r) : 0;
    int m = 0;
    for (int64_t kc = ka; kc < kb; kc += 32) {
      __syncthreads();   // the previous offsets are consumed
      if (ty == 0) coff[tx] = kc + tx < kb ? pack_col_off(ps, kc + tx) : 0;
      __syncthreads();
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int kk = ty + 8 * j;
        if (r < ps.R && kc + kk < kb) m = max(m, biased_exp(src[ro + coff[kk]]));
      }
    }
    red[ty][tx] = m;
    __syncthreads();
    if (ty == 0) {
      for (int j = 1; j < 8; ++j) m = max(m, red[j][tx]);
      if (r < ps.R && m > 0) atomicMax(ex + r, m);
    }
    __syncthreads();
  }
}

// bf16 bits (in the upper half) of the integer d (|d| < 2^22; exact in bf16
// for |d| <= 256): the float 1.5 * 2^23 + d, less the bias, is d exactly
__device__ __forceinline__ uint32_t oz_int_bits(int d) {
  return __float_as_uint(__int_as_float(0x4B400000 + d) - 12582912.0f);
}
// of byte `sel` of w, less 128
__device__ __forceinline__ uint32_t oz_byte_bits(uint32_t w, int sel) {
  return __float_as_uint(__uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440 | sel)) - 8388736.0f);
}
// bf16 of a and b (upper halves) as one word, a in the lower half
__device__ __forceinline__ uint32_t oz_pair(uint32_t a, uint32_t b) { return __byte_perm(a, b, 0x7632); }

// |x| 2^-e (|x| < 2^e; e includes the guard bits) times 2^bits, rounded to an integer; bits <= 64
__device__ __forceinline__ unsigned long long oz_fixed(unsigned long long x, int e, int bits) {
  const int be = (int)((x >> 52) & 0x7FF);
  unsigned long long Z = 0;
  if (be != 0) {
    const unsigned long long m = (x & ((1ull << 52) - 1)) | (1ull << 52);   // |x| = m 2^(be - 1075)
    const int sh = 1075 + e - bits - be;                                    // Z = m 2^-sh
    if (sh <= 0) Z = m << (-sh);
    else if (sh < 64) Z = (m >> sh) + ((m >> (sh - 1)) & 1ull);
  }
  return Z;
}

// The S balanced base-2^BITS digits of y = x 2^-e, as float bits whose upper
// halves are their bf16: Z = round(|y| 2^(BITS S)) with the sign of x is
// d_1 2^(BITS (S-1)) + ... + d_S with |d_S|, .., |d_2| <= 2^(BITS-1), d_1 the
// rest.  The low digits are the plain digits of Z plus half a digit at every
// low place, less that half (a digit at or above half carries one into the
// next).  Integer arithmetic only; |y - sum_s d_s 2^(-BITS s)| <= 2^(-BITS S) / 2.
// 8 bits: the signed Z is cut, each low digit is one byte (three instructions);
// otherwise (6 bits, or the 64 bits of S = 8, which leave no room for a sign)
// |Z| is cut and the digits take the sign.
template <int S, int BITS>
__device__ __forceinline__ void oz_digits(double x, int e, uint32_t (&d)[S]) {
  const unsigned long long xb = (unsigned long long)__double_as_longlong(x);
  const unsigned long long Z = oz_fixed(xb, e, BITS * S);
  const int neg = (int)(xb >> 63);
  constexpr unsigned long long HALF = 1ull << (BITS - 1);
  constexpr unsigned long long C = HALF * (((1ull << (BITS * (S - 1))) - 1) / ((1ull << BITS) - 1));
  if (BITS == 8 && S == 8) {
    const unsigned long long low = (Z & ((1ull << 56) - 1)) + C;   // C < 2^56: no carry out of 57 bits
    const uint32_t w[2] = {(uint32_t)low, (uint32_t)(low >> 32)};
    const uint32_t flip = neg ? 0x80000000u : 0u;
#pragma unroll
    for (int s = 1; s < S; ++s) d[s] = oz_byte_bits(w[(S - 1 - s) >> 2], (S - 1 - s) & 3) ^ flip;
    d[0] = oz_int_bits((int)(Z >> 56) + (int)(low >> 56)) ^ flip;
  } else if (BITS == 8) {
    const unsigned long long Zc = (neg ? 0ull - Z : Z) + C;
    const uint32_t w[2] = {(uint32_t)Zc, (uint32_t)(Zc >> 32)};
#pragma unroll
    for (int s = 1; s < S; ++s) d[s] = oz_byte_bits(w[(S - 1 - s) >> 2], (S - 1 - s) & 3);
    d[0] = oz_int_bits((int)((long long)Zc >> (8 * (S - 1))));
  } else {
    const unsigned long long Zc = Z + C;
#pragma unroll
    for (int s = 1; s < S; ++s) {
      const int dv = (int)((Zc >> (BITS * (S - 1 - s))) & (2 * HALF - 1)) - (int)HALF;
      d[s] = oz_int_bits(neg ? -dv : dv);
    }
    const int top = (int)(Zc >> (BITS * (S - 1)));
    d[0] = oz_int_bits(neg ? -top : top);
  }
}

// the digits of 4 consecutive k of row r as one 8-byte word per slice
template <int S, int BITS>
__device__ __forceinline__ void oz_store4(const double (&xv)[4], int e, __nv_bfloat16* d, int64_t Kpad) {
  uint32_t dg[4][S];
#pragma unroll
  for (int q = 0; q < 4; ++q) oz_digits<S, BITS>(xv[q], e, dg[q]);
#pragma unroll
  for (int s = 0; s < S; ++s)
    *reinterpret_cast<uint2*>(d + s * Kpad) = make_uint2(oz_pair(dg[0][s], dg[1][s]), oz_pair(dg[2][s], dg[3][s]));
}

// Row walk in one pass (k the faster source index, at most 4 groups of 4
// columns per thread): 2^lg threads read a row into registers, reduce its
// exponent and cut it.
template <int S, int BITS>
__global__ void __launch_bounds__(256) oz_pack_rows_fused_kernel(const double* __restrict__ src, PackSpec ps,
                                                                 int64_t Kpad, int guard, int* __restrict__ ex,
                                                                 __nv_bfloat16* __restrict__ dst, int lg) {
  __shared__ int red[8];
  const int tpr = 1 << lg, lane = threadIdx.x & (tpr - 1), rpb = 256 >> lg, sub = threadIdx.x >> lg;
  const int wpr = tpr >> 5, warp = threadIdx.x >> 5;
  const int ng = (int)(Kpad >> 2);
  const bool k1 = pack_k_single(ps);
  for (int64_t rb = (int64_t)blockIdx.x * rpb; rb < ps.R; rb += (int64_t)gridDim.x * rpb) {
    const int64_t r = rb + sub;
    const bool ok = r < ps.R;
    const int64_t ro = ok ? pack_row_off(ps, r) : 0;
    double xv[4][4];
    int m = 0;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const int64_t k0 = (int64_t)(lane + g * tpr) << 2;
#pragma unroll
      for (int q = 0; q < 4; ++q) xv[g][q] = 0.0;
      if (ok && k0 < ps.K) pack_load4(src, ps, k1, ro, k0, (int)min((int64_t)4, ps.K - k0), xv[g]);
    }
#pragma unroll
    for (int g = 0; g < 4; ++g)
#pragma unroll
      for (int q = 0; q < 4; ++q) m = max(m, biased_exp(xv[g][q]));
    m = __reduce_max_sync(0xffffffffu, m);
    if (lg > 5) {
      __syncthreads();   // the previous row's maxima are consumed
      if ((threadIdx.x & 31) == 0) red[warp] = m;
      __syncthreads();
      for (int w = 0; w < wpr; ++w) m = max(m, red[sub * wpr + w]);
    }
    if (!ok) continue;   // every thread of the block runs the same number of rounds
    if (lane == 0) ex[r] = m;
    const int e = oz_row_exp(m) + guard;
    __nv_bfloat16* drow = dst + r * (S * Kpad);
#pragma unroll
    for (int g = 0; g < 4; ++g) {
      const int grp = lane + g * tpr;
      if (grp < ng) oz_store4<S, BITS>(xv[g], e, drow + (grp << 2), Kpad);
    }
  }
}

// Transposing walk in one pass (row index the faster one, K <= TILE_KMAX): a
// block reads 32 rows x K into shared memory, coalesced along the rows,
// reduces the row exponents and cuts from there, two consecutive k per thread.
template <int S, int BITS>
__global__ void __launch_bounds__(256) oz_pack_tiles_fused_kernel(const double* __restrict__ src, PackSpec ps,
                                                                  int64_t Kpad, int guard, int* __restrict__ ex,
                                                                  __nv_bfloat16* __restrict__ dst) {
  extern __shared__ double ftile[];   // [K][33]
  __shared__ int64_t coff[TILE_KMAX];
  __shared__ int red[8][32];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int kp = threadIdx.x & 15, rw = threadIdx.x >> 4;   // write phase: k pair, row
  const int64_t ntr = (ps.R + 31) / 32;
  const int K = (int)ps.K;
  for (int k = threadIdx.x; k < K; k += 256) coff[k] = pack_col_off(ps, k);
  __syncthreads();
  for (int64_t tb = blockIdx.x; tb < ntr; tb += gridDim.x) {
    const int64_t r0 = tb * 32;
    const bool rok = r0 + tx < ps.R;
    const int64_t ro = rok ? pack_row_off(ps, r0 + tx) : 0;
    int m = 0;
#pragma unroll 8
    for (int kk = ty; kk < K; kk += 8) {
      const double x = rok ? src[ro + coff[kk]] : 0.0;
      m = max(m, biased_exp(x));
      ftile[kk * 33 + tx] = x;
    }
    red[ty][tx] = m;
    __syncthreads();
    if (ty == 0) {
#pragma unroll
      for (int j = 1; j < 8; ++j) m = max(m, red[j][tx]);
      red[0][tx] = m;
      if (rok) ex[r0 + tx] = m;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int rr = rw + 16 * j;
      const int64_t r = r0 + rr;
      if (r >= ps.R) continue;
      const int e = oz_row_exp(red[0][rr]) + guard;
      for (int k = 2 * kp; k < (int)Kpad; k += 32) {
        uint32_t da[S], db[S];
        oz_digits<S, BITS>(k < K ? ftile[k * 33 + rr] : 0.0, e, da);
        oz_digits<S, BITS>(k + 1 < K ? ftile[(k + 1) * 33 + rr] : 0.0, e, db);
        uint32_t* d = reinterpret_cast<uint32_t*>(dst + r * (S * Kpad) + k);
#pragma unroll
        for (int s = 0; s < S; ++s) d[(s * Kpad) >> 1] = oz_pair(da[s], db[s]);
      }
    }
    __syncthreads();   // the tile is consumed
  }
}

// The same for K up to 8 x TILE_KW: a cluster of up to eight blocks shares 32
// rows, each with its range of columns, and exchanges the maxima through
// distributed shared memory, so the source is read once and by one launch
// instead of a memset, an exponent pass and the cut.  With the rows through
// shared memory below: packs of a mixed solve at (H2O)8 99 -> 92 ms, of an exact
// step at (H2O)6 odd 2.08 -> 1.89.
constexpr int TILE_KW = 192;
template <int S, int BITS>
__global__ void __launch_bounds__(256) oz_pack_tiles_cluster_kernel(const double* __restrict__ src, PackSpec ps,
                                                                    int64_t Kpad, int guard, int* __restrict__ ex,
                                                                    __nv_bfloat16* __restrict__ dst, int nc, int kw) {
  extern __shared__ double ftile[];   // [kw][33]
  __shared__ int64_t coff[TILE_KW];
  __shared__ int red[8][32];
  __shared__ int own[32], tot[32];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int kp = threadIdx.x & 15, rw = threadIdx.x >> 4;   // write phase: k pair, row
  const int rank = (int)tc5::cluster_rank();
  const int64_t ntr = (ps.R + 31) / 32;
  const int ka = rank * kw, K = (int)min((int64_t)kw, ps.K - ka);   // columns here (<= 0: padding only)
  const int kend = (int)min((int64_t)kw, Kpad - ka);
  for (int k = threadIdx.x; k < K; k += 256) coff[k] = pack_col_off(ps, ka + k);
  __syncthreads();
  for (int64_t tb = blockIdx.x / nc; tb < ntr; tb += gridDim.x / nc) {
    const int64_t r0 = tb * 32;
    const bool rok = r0 + tx < ps.R;
    const int64_t ro = rok ? pack_row_off(ps, r0 + tx) : 0;
    int m = 0;
#pragma unroll 8
    for (int kk = ty; kk < K; kk += 8) {
      const double x = rok ? src[ro + coff[kk]] : 0.0;
      m = max(m, biased_exp(x));
      ftile[kk * 33 + tx] = x;
    }
    red[ty][tx] = m;
    __syncthreads();
    if (ty == 0) {
#pragma unroll
      for (int j = 1; j < 8; ++j) m = max(m, red[j][tx]);
      own[tx] = m;
    }
    tc5::cluster_sync();
    if (ty == 0) {
      const uint32_t at = tc5::smem_u32(&own[tx]);
      int part[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        part[q] = 0;
        if (q < nc)
          asm volatile("ld.shared::cluster.u32 %0, [%1];" : "=r"(part[q]) : "r"(tc5::cluster_addr(at, q)) : "memory");
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) m = max(m, part[q]);
      tot[tx] = m;
      if (rok && rank == 0) ex[r0 + tx] = m;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int rr = rw + 16 * j;
      const int64_t r = r0 + rr;
      if (r >= ps.R) continue;
      const int e = oz_row_exp(tot[rr]) + guard;
      for (int k = 2 * kp; k < kend; k += 32) {
        uint32_t da[S], db[S];
        oz_digits<S, BITS>(k < K ? ftile[k * 33 + rr] : 0.0, e, da);
        oz_digits<S, BITS>(k + 1 < K ? ftile[(k + 1) * 33 + rr] : 0.0, e, db);
        uint32_t* d = reinterpret_cast<uint32_t*>(dst + r * (S * Kpad) + ka + k);
#pragma unroll
        for (int s = 0; s < S; ++s) d[(s * Kpad) >> 1] = oz_pair(da[s], db[s]);
      }
    }
    tc5::cluster_sync();   // the tile and the maxima are consumed
  }
}

// Rows too long for registers, through shared memory: a block of 512 threads per
// row, two to an SM up to ROW_KMAX columns.
constexpr int ROW_KMAX = 14080;     // 110 KB
template <int S, int BITS>
__global__ void __launch_bounds__(512) oz_pack_rows_smem_kernel(const double* __restrict__ src, PackSpec ps,
                                                                int64_t Kpad, int guard, int* __restrict__ ex,
                                                                __nv_bfloat16* __restrict__ dst) {
  extern __shared__ double ftile[];   // [Kpad]
  __shared__ int red[16];
  const int ng = (int)(Kpad >> 2), t = threadIdx.x;
  const bool k1 = pack_k_single(ps);
  for (int64_t r = blockIdx.x; r < ps.R; r += gridDim.x) {
    const int64_t ro = pack_row_off(ps, r);
    int m = 0;
    for (int g0 = t; g0 < ng; g0 += 512 * 3) {
      double xv[3][4];
#pragma unroll
      for (int u = 0; u < 3; ++u) {
        const int64_t k0 = (int64_t)(g0 + 512 * u) << 2;
#pragma unroll
        for (int q = 0; q < 4; ++q) xv[u][q] = 0.0;
        if (k0 < ps.K) pack_load4(src, ps, k1, ro, k0, (int)min((int64_t)4, ps.K - k0), xv[u]);
      }
#pragma unroll
      for (int u = 0; u < 3; ++u) {
        const int g = g0 + 512 * u;
#pragma unroll
        for (int q = 0; q < 4; ++q) m = max(m, biased_exp(xv[u][q]));
        if (g < ng) {
          *reinterpret_cast<double2*>(ftile + 4 * g) = make_double2(xv[u][0], xv[u][1]);
          *reinterpret_cast<double2*>(ftile + 4 * g + 2) = make_double2(xv[u][2], xv[u][3]);
        }
      }
    }
    m = __reduce_max_sync(0xffffffffu, m);
    if ((t & 31) == 0) red[t >> 5] = m;
    __syncthreads();
#pragma unroll
    for (int w = 0; w < 16; ++w) m = max(m, red[w]);
    if (t == 0) ex[r] = m;
    const int e = oz_row_exp(m) + guard;
    __nv_bfloat16* drow = dst + r * (S * Kpad);
    for (int g = t; g < ng; g += 512) {
      const double2 a = *reinterpret_cast<const double2*>(ftile + 4 * g), b = *reinterpret_cast<const double2*>(ftile + 4 * g + 2);
      const double xv[4] = {a.x, a.y, b.x, b.y};
      oz_store4<S, BITS>(xv, e, drow + 4 * g, Kpad);
    }
    __syncthreads();   // the row and the maxima are consumed
  }
}

// dst[r][s*Kpad + k]: row walk (k the faster source index), 2^lg threads per
// row, each cutting 4 consecutive k and writing one 8-byte word per slice
// (zeros over the padding [K, Kpad))
template <int S, int BITS>
__global__ void __launch_bounds__(256) oz_pack_rows_kernel(const double* __restrict__ src, PackSpec ps, int64_t Kpad, int guard,
                                                           const int* __restrict__ ex, __nv_bfloat16* __restrict__ dst,
                                                           PackWalk pw) {
  const int tpr = 1 << pw.lg, lane = threadIdx.x & (tpr - 1), rpb = 256 >> pw.lg;
  const int64_t ng = Kpad >> 2;
  const bool k1 = pack_k_single(ps);
  const int64_t units = ps.R * pw.nseg;
  for (int64_t u = (int64_t)blockIdx.x * rpb + (threadIdx.x >> pw.lg); u < units; u += (int64_t)gridDim.x * rpb) {
    const int64_t r = pw.nseg == 1 ? u : u / pw.nseg;
    const int64_t g0 = (u - r * pw.nseg) * pw.gseg, g1 = min(ng, g0 + pw.gseg);
    const int e = oz_row_exp(ex[r]) + guard;
    const int64_t ro = pack_row_off(ps, r);
    __nv_bfloat16* drow = dst + r * (S * Kpad);
    for (int64_t g = g0 + lane; g < g1; g += tpr) {
      const int64_t k0 = g << 2;
      double xv[4] = {0.0, 0.0, 0.0, 0.0};
      if (k0 < ps.K) pack_load4(src, ps, k1, ro, k0, (int)min((int64_t)4, ps.K - k0), xv);
      oz_store4<S, BITS>(xv, e, drow + k0, Kpad);
    }
  }
}

// transposing walk through 32 x 32 tiles (row index faster in the source):
// source offsets of the tile's rows and columns in shared memory, coalesced
// reads along rows, and each thread cuts two consecutive k of one row and
// writes one 4-byte word per slice (the tiles cover [0, Kpad), zeros past K)
template <int S, int BITS>
__global__ void __launch_bounds__(256) oz_pack_tiles_kernel(const double* __restrict__ src, PackSpec ps, int64_t Kpad, int guard,
                                                            const int* __restrict__ ex,
                                                            __nv_bfloat16* __restrict__ dst) {
  __shared__ double tile[32][33];
  __shared__ int64_t roff[32], coff[32];
  const int64_t ntr = (ps.R + 31) / 32, ntk = Kpad / 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int kp = threadIdx.x & 15, rw = threadIdx.x >> 4;   // write phase: k pair, row
  for (int64_t tb = blockIdx.x; tb < ntr * ntk; tb += gridDim.x) {
    const int64_t r0 = (tb / ntk) * 32, k0 = (tb % ntk) * 32;
    __syncthreads();   // the previous tile is consumed
    if (ty == 0) roff[tx] = r0 + tx < ps.R ? pack_row_off(ps, r0 + tx) : 0;
    else if (ty == 1) coff[tx] = k0 + tx < ps.K ? pack_col_off(ps, k0 + tx) : 0;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int kk = ty + 8 * j;
      tile[kk][tx] = (r0 + tx < ps.R && k0 + kk < ps.K) ? src[roff[tx] + coff[kk]] : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int rr = rw + 16 * j;
      const int64_t r = r0 + rr;
      if (r >= ps.R) continue;
      const int e = oz_row_exp(ex[r]) + guard;
      uint32_t da[S], db[S];
      oz_digits<S, BITS>(tile[2 * kp][rr], e, da);
      oz_digits<S, BITS>(tile[2 * kp + 1][rr], e, db);
      uint32_t* d = reinterpret_cast<uint32_t*>(dst + r * (S * Kpad) + k0 + 2 * kp);
#pragma unroll
      for (int s = 0; s < S; ++s) d[(s * Kpad) >> 1] = oz_pair(da[s], db[s]);
    }
  }
}

bool pack_by_tiles(const PackSpec& ps) {
  const int64_t kfast = std::llabs(ps.kd3 > 1 ? ps.ks3 : (ps.kd2 > 1 ? ps.ks2 : ps.ks1));
  const int64_t rfast = std::llabs(ps.rd3 > 1 ? ps.rs3 : (ps.rd2 > 1 ? ps.rs2 : ps.rs1));
  return rfast < kfast && ps.R >= 32;
}

// exponent pass, then the cut
template <int S, int BITS>
void pack_two_pass(const double* src, const PackSpec& ps, int guard, __nv_bfloat16* dst, int* ex, bool tiles,
                   cudaStream_t s) {
  const int64_t Kpad = oz_kpad(ps.K);
  FCC_CUDA(cudaMemsetAsync(ex, 0, sizeof(int) * ps.R, s));
  // k-slabs so that the exponent pass has enough independent work
  const int64_t want = 152 * 64;
  const int64_t units = tiles ? (ps.R + 31) / 32 : ps.R;
  int64_t kslab = ps.K;
  if (units < want) kslab = std::max<int64_t>(256, (ps.K * units + want - 1) / want);
  const int64_t nks = (ps.K + kslab - 1) / kslab;
  if (tiles) {
    oz_exp_tiles_kernel<<<(unsigned)std::min<int64_t>(units * nks, 152 * 32), 256, 0, s>>>(src, ps, kslab, ex);
    FCC_CHECK_LAUNCH();
    const unsigned tgrid = (unsigned)std::min<int64_t>(((ps.R + 31) / 32) * (Kpad / 32), 152 * 16);
    oz_pack_tiles_kernel<S, BITS><<<tgrid, 256, 0, s>>>(src, ps, Kpad, guard, ex, dst);
  } else {
    const int64_t warps = units * nks;
    oz_exp_rows_kernel<<<(unsigned)std::min<int64_t>((warps + 7) / 8, 152 * 32), 256, 0, s>>>(src, ps, kslab, ex);
    FCC_CHECK_LAUNCH();
    const PackWalk pw = pack_walk(ps.R, Kpad / 4);
    oz_pack_rows_kernel<S, BITS><<<pack_walk_grid(pw, ps.R), 256, 0, s>>>(src, ps, Kpad, guard, ex, dst, pw);
  }
  FCC_CHECK_LAUNCH();
}

template <int S, int BITS>
void pack(const double* src, const PackSpec& ps, int guard, __nv_bfloat16* dst, int* ex, cudaStream_t s) {
  const int64_t Kpad = oz_kpad(ps.K);
  const bool tiles = pack_by_tiles(ps);
  const int64_t ntr = (ps.R + 31) / 32;
  if (tiles && ps.K <= TILE_KMAX) {
    oz_pack_tiles_fused_kernel<S, BITS><<<(unsigned)std::min<int64_t>(ntr, 152 * 16), 256, (size_t)ps.K * 33 * 8, s>>>(
        src, ps, Kpad, guard, ex, dst);
    FCC_CHECK_LAUNCH();
    return;
  }
  // few long rows: the two-pass walk cuts them into segments for more blocks
  if (!tiles && Kpad <= 4096 && (Kpad <= 512 || ps.R >= 64)) {
    int lg = 5;
    while ((int64_t(16) << lg) < Kpad) ++lg;
    const int64_t rpb = 256 >> lg;
    oz_pack_rows_fused_kernel<S, BITS><<<(unsigned)std::min<int64_t>((ps.R + rpb - 1) / rpb, 152 * 16), 256, 0, s>>>(
        src, ps, Kpad, guard, ex, dst, lg);
    FCC_CHECK_LAUNCH();
    return;
  }
  if (tiles && Kpad <= 8 * TILE_KW) {
    const int nc = (int)((Kpad + TILE_KW - 1) / TILE_KW);
    const int kw = (int)((Kpad / 64 + nc - 1) / nc * 64);
    static SmemLimit smem;
    smem.raise(oz_pack_tiles_cluster_kernel<S, BITS>, TILE_KW * 33 * 8);
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(std::min<int64_t>(ntr, 152 * 4) * nc));
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = (size_t)kw * 33 * 8;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = (unsigned)nc;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    FCC_CUDA(cudaLaunchKernelEx(&cfg, oz_pack_tiles_cluster_kernel<S, BITS>, src, ps, Kpad, guard, ex, dst, nc, kw));
    FCC_CHECK_LAUNCH();
    return;
  }
  if (!tiles && Kpad > 4096 && Kpad <= ROW_KMAX && ps.R >= 304) {
    static SmemLimit smem;
    smem.raise(oz_pack_rows_smem_kernel<S, BITS>, ROW_KMAX * 8);
    oz_pack_rows_smem_kernel<S, BITS><<<(unsigned)std::min<int64_t>(ps.R, 152 * 8), 512, (size_t)Kpad * 8, s>>>(
        src, ps, Kpad, guard, ex, dst);
    FCC_CHECK_LAUNCH();
    return;
  }
  pack_two_pass<S, BITS>(src, ps, guard, dst, ex, tiles, s);
}

}  // namespace

int64_t oz_kpad(int64_t K) { return ((K + OZ_BK - 1) / OZ_BK) * OZ_BK; }

void pack_oz(const double* src, const PackSpec& ps, int S, int bits, int guard, __nv_bfloat16* dst, int* ex,
             cudaStream_t s) {
  if (ps.R <= 0 || ps.K <= 0) return;
  if (ps.R >= (int64_t(1) << 31) || ps.K >= (int64_t(1) << 31)) fail(FCC_ERR_BAD_ARG, "pack extent too large");
  const int pidx = prof_begin(s);
  struct End { cudaStream_t s; int i; double b; ~End() { prof_end(s, i, PROF_PACK, b); } } pend{s, pidx,
      (double)ps.R * (double)ps.K * 8.0 + (double)ps.R * (double)(S * oz_kpad(ps.K)) * 2.0};
  switch (10 * bits + S) {
    case 61: pack<1, 6>(src, ps, guard, dst, ex, s); break;
    case 62: pack<2, 6>(src, ps, guard, dst, ex, s); break;
    case 63: pack<3, 6>(src, ps, guard, dst, ex, s); break;
    case 64: pack<4, 6>(src, ps, guard, dst, ex, s); break;
    case 65: pack<5, 6>(src, ps, guard, dst, ex, s); break;
    case 66: pack<6, 6>(src, ps, guard, dst, ex, s); break;
    case 67: pack<7, 6>(src, ps, guard, dst, ex, s); break;
    case 68: pack<8, 6>(src, ps, guard, dst, ex, s); break;
    case 81: pack<1, 8>(src, ps, guard, dst, ex, s); break;
    case 82: pack<2, 8>(src, ps, guard, dst, ex, s); break;
    case 83: pack<3, 8>(src, ps, guard, dst, ex, s); break;
    case 84: pack<4, 8>(src, ps, guard, dst, ex, s); break;
    case 85: pack<5, 8>(src, ps, guard, dst, ex, s); break;
    case 86: pack<6, 8>(src, ps, guard, dst, ex, s); break;
    case 87: pack<7, 8>(src, ps, guard, dst, ex, s); break;
    case 88: pack<8, 8>(src, ps, guard, dst, ex, s); break;
    default: fail(FCC_ERR_BAD_ARG, "bad slice count");
  }
}

}  // namespace fcc
