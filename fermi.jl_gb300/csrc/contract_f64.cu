// FP64 tensor contraction on the DMMA pipe (mma.sync m8n8k4 .f64) and the
// einsum-style front end used by the CCSD driver.
//
// Every contraction of the amplitude equations is C = alpha * A.B + beta * C
// where the M, N and K matrix indices are each a pair of tensor indices with
// arbitrary strides, so index permutations are folded into the loads and
// stores instead of separate transpose passes.  On GB300 the FP64 pipe
// (about 1 TFLOP/s per GPU) is the bound of this kernel; a 64x64 tile with
// 16-deep K steps staged through shared memory keeps it saturated.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <map>
#include <mutex>

#include "fcc_common.cuh"
#include "fcc_tc.cuh"

namespace fcc {

namespace {

constexpr int BM = 64, BN = 64, BK = 16, NT = 128;
constexpr int LDS = BM + 8;  // 72 doubles: rows 64 B apart modulo 128 B

__device__ __forceinline__ void dmma884(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// Offsets of a 3-level index x = (x1*D2 + x2)*D3 + x3.  Extents are below
// 2^31 (contract_f64_launch checks): a 64-bit division goes through the FP64
// pipe here (1/64 rate) and one per loaded element, as this file once had, cost
// more than the MMAs of a tile.
__device__ __forceinline__ int64_t off3(int64_t x, int64_t D2, int64_t D3, int64_t s1, int64_t s2, int64_t s3) {
  const uint32_t x3 = (uint32_t)x % (uint32_t)D3, r = (uint32_t)x / (uint32_t)D3;
  const uint32_t x2 = r % (uint32_t)D2, x1 = r / (uint32_t)D2;
  return (int64_t)x1 * s1 + (int64_t)x2 * s2 + (int64_t)x3 * s3;
}
// of a 2-level index
__device__ __forceinline__ int64_t off2(int64_t k, int64_t D2, int64_t s1, int64_t s2) {
  const uint32_t k1 = (uint32_t)k / (uint32_t)D2, k2 = (uint32_t)k - k1 * (uint32_t)D2;
  return (int64_t)k1 * s1 + (int64_t)k2 * s2;
}

// alpha * x + beta * c without FP64 instructions for the usual factors (a warp's
// FP64 instruction takes its SM's pipe for 16 clk)
__device__ __forceinline__ double f64_axpby(double x, double c, double alpha, double beta) {
  if (alpha == -1.0) x = -x;
  else if (alpha != 1.0) x *= alpha;
  if (beta == 1.0) x += c;
  else if (beta != 0.0) x += beta * c;
  return x;
}
__device__ __forceinline__ void f64_store(double* dst, double x, double alpha, double beta) {
  *dst = f64_axpby(x, beta != 0.0 ? *dst : 0.0, alpha, beta);
}

// The k loop of one 64 x 64 output tile: stage A (BM x BK) and B (BK x BN)
// into shared memory, then 4 k-steps of m8n8k4 per 16-deep slab.  EDGE tiles
// (the last row or column tile of a ragged extent) skip the MMAs of 8-wide
// blocks that lie wholly outside the output, so a v = 152 extent (tiles of
// 64 + 64 + 24) issues no DMMA work for the 40 missing columns.
template <bool EDGE>
__device__ __forceinline__ void f64_mainloop(const double* __restrict__ A, const double* __restrict__ B,
                                             const CtrDesc& d, int a_mfast, int b_nfast, int64_t kbeg,
                                             int64_t kend, double (&As)[BK][LDS], double (&Bs)[BK][LDS],
                                             const int64_t* rowA, const int64_t* colB, const int8_t* rowOK,
                                             const int8_t* colOK, int64_t m0, int64_t n0,
                                             double (&acc)[4][4][2]) {
  const int tid = threadIdx.x;
  const int warp = tid >> 5, lane = tid & 31;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
  // row (column) blocks of 8 of this warp that lie inside the output
  int ni = 4, nj = 4;
  if (EDGE) {
    ni = (int)max((int64_t)0, min((int64_t)4, (d.M - m0 - wm + 7) / 8));
    nj = (int)max((int64_t)0, min((int64_t)4, (d.N - n0 - wn + 7) / 8));
  }
  for (int64_t k0 = kbeg; k0 < kend; k0 += BK) {
    if (a_mfast) {
      int m = tid & 63, kb = tid >> 6;
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        int kk = kb + 2 * r;
        int64_t k = k0 + kk;
        double v = 0.0;
        if (rowOK[m] && k < kend) {
          v = A[rowA[m] + off2(k, d.K2, d.a_k1, d.a_k2)];
        }
        As[kk][m] = v;
      }
    } else {
      int kk = tid & 15, mb = tid >> 4;
      int64_t k = k0 + kk;
      bool kok = k < kend;
      int64_t koff = 0;
      if (kok) {
        koff = off2(k, d.K2, d.a_k1, d.a_k2);
      }
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        int m = mb + 8 * r;
        As[kk][m] = (kok && rowOK[m]) ? A[rowA[m] + koff] : 0.0;
      }
    }
    if (b_nfast) {
      int n = tid & 63, kb = tid >> 6;
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        int kk = kb + 2 * r;
        int64_t k = k0 + kk;
        double v = 0.0;
        if (colOK[n] && k < kend) {
          v = B[colB[n] + off2(k, d.K2, d.b_k1, d.b_k2)];
        }
        Bs[kk][n] = v;
      }
    } else {
      int kk = tid & 15, nb = tid >> 4;
      int64_t k = k0 + kk;
      bool kok = k < kend;
      int64_t koff = 0;
      if (kok) {
        koff = off2(k, d.K2, d.b_k1, d.b_k2);
      }
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        int n = nb + 8 * r;
        Bs[kk][n] = (kok && colOK[n]) ? B[colB[n] + koff] : 0.0;
      }
    }
    __syncthreads();
#pragma unroll
    for (int ks = 0; ks < BK; ks += 4) {
      double af[4], bf[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) af[i] = As[ks + (lane & 3)][wm + 8 * i + (lane >> 2)];
#pragma unroll
      for (int j = 0; j < 4; ++j) bf[j] = Bs[ks + (lane & 3)][wn + 8 * j + (lane >> 2)];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (!EDGE || (i < ni && j < nj)) dmma884(acc[i][j][0], acc[i][j][1], af[i], bf[j]);   // warp-uniform
    }
    __syncthreads();
  }
}

__global__ void __launch_bounds__(NT, 5) contract_f64_kernel(const double* __restrict__ A,
                                                          const double* __restrict__ B,
                                                          double* __restrict__ C, CtrDesc d,
                                                          int a_mfast, int b_nfast, int64_t k_chunk,
                                                          double* __restrict__ partial) {
  __shared__ double As[BK][LDS];
  __shared__ double Bs[BK][LDS];
  __shared__ int64_t rowA[BM], colB[BN], rowC[BM], colC[BN];
  __shared__ int8_t rowOK[BM], colOK[BN];

  if (d.sym && blockIdx.y < blockIdx.x) return;   // copied by mirror_kernel
  const int tid = threadIdx.x;
  const int64_t m0 = (int64_t)blockIdx.x * BM;
  const int64_t n0 = (int64_t)blockIdx.y * BN;
  // blockIdx.z: batch index, or the K slice when split over K (partial != 0)
  const int64_t bz = partial ? 0 : blockIdx.z;
  const int64_t kbeg = partial ? (int64_t)blockIdx.z * k_chunk : 0;
  const int64_t kend = partial ? min(d.K, kbeg + k_chunk) : d.K;
  A += bz * d.a_b;
  B += bz * d.b_b;
  C += bz * d.c_b;

  if (tid < BM) {
    const int64_t m = m0 + tid;
    const bool ok = m < d.M;
    rowA[tid] = ok ? off3(m, d.M2, d.M3, d.a_m1, d.a_m2, d.a_m3) : 0;
    rowC[tid] = ok ? off3(m, d.M2, d.M3, d.c_m1, d.c_m2, d.c_m3) : 0;
    rowOK[tid] = ok;
  } else {
    const int t = tid - BM;
    const int64_t n = n0 + t;
    const bool ok = n < d.N;
    colB[t] = ok ? off3(n, d.N2, d.N3, d.b_n1, d.b_n2, d.b_n3) : 0;
    colC[t] = ok ? off3(n, d.N2, d.N3, d.c_n1, d.c_n2, d.c_n3) : 0;
    colOK[t] = ok;
  }
  __syncthreads();

  const int warp = tid >> 5, lane = tid & 31;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
  double acc[4][4][2];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j][0] = acc[i][j][1] = 0.0;

  if (m0 + BM <= d.M && n0 + BN <= d.N)
    f64_mainloop<false>(A, B, d, a_mfast, b_nfast, kbeg, kend, As, Bs, rowA, colB, rowOK, colOK, m0, n0, acc);
  else
    f64_mainloop<true>(A, B, d, a_mfast, b_nfast, kbeg, kend, As, Bs, rowA, colB, rowOK, colOK, m0, n0, acc);

  // ---- epilogue: C = alpha * acc + beta * C with general output strides
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int ml = wm + 8 * i + (lane >> 2);
    const int64_t m = m0 + ml;
    if (m >= d.M) continue;
    const int64_t crow = rowC[ml];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int nl = wn + 8 * j + 2 * (lane & 3) + h;
        const int64_t n = n0 + nl;
        if (n >= d.N) continue;
        if (partial) {   // split-K: raw partial sums, reduced in a fixed order later
          partial[((int64_t)blockIdx.z * d.M + m) * d.N + n] = acc[i][j][h];
          continue;
        }
        f64_store(C + crow + colC[nl], acc[i][j][h], d.alpha, d.beta);
      }
    }
  }
}

// C(m, n) = C(n, m) for the 64 x 64 tiles below the diagonal, 32 x 32 elements a block.
__global__ void __launch_bounds__(256) mirror_kernel(double* __restrict__ C, CtrDesc d) {
  if (blockIdx.x / 2 <= blockIdx.y / 2) return;
  __shared__ double tile[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int64_t m0 = (int64_t)blockIdx.x * 32, n0 = (int64_t)blockIdx.y * 32;
  auto at = [&](int64_t m, int64_t n) {
    return off3(m, d.M2, d.M3, d.c_m1, d.c_m2, d.c_m3) + off3(n, d.N2, d.N3, d.c_n1, d.c_n2, d.c_n3);
  };
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int64_t r = n0 + ty + 8 * q, c = m0 + tx;
    if (r < d.M && c < d.N) tile[ty + 8 * q][tx] = C[at(r, c)];
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int64_t m = m0 + ty + 8 * q, n = n0 + tx;
    if (m < d.M && n < d.N) C[at(m, n)] = tile[tx][ty + 8 * q];
  }
}

// C = alpha * sum_z partial[z] + beta * C, summed in slice order.
__global__ void splitk_reduce_kernel(const double* __restrict__ partial, int splits, double* __restrict__ C,
                                     CtrDesc d) {
  const int64_t MN = d.M * d.N;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < MN; t += (int64_t)gridDim.x * blockDim.x) {
    double s = 0.0;
    for (int z = 0; z < splits; z += 8) {   // eight loads in flight, added in order
      double x[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) x[q] = z + q < splits ? partial[(int64_t)(z + q) * MN + t] : 0.0;
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (z + q < splits) s += x[q];
    }
    const uint32_t m = (uint32_t)((uint64_t)t >> 32 ? t / d.N : (uint32_t)t / (uint32_t)d.N);
    const int64_t n = t - (int64_t)m * d.N;
    f64_store(C + off3(m, d.M2, d.M3, d.c_m1, d.c_m2, d.c_m3) + off3(n, d.N2, d.N3, d.c_n1, d.c_n2, d.c_n3), s,
              d.alpha, d.beta);
  }
}

// The same for few outputs and many slices: 32 outputs per block, eight warps
// over interleaved slices, added in a fixed order.
__global__ void __launch_bounds__(256) splitk_reduce_few_kernel(const double* __restrict__ partial, int splits,
                                                                double* __restrict__ C, CtrDesc d) {
  __shared__ double part[8][32];
  const int x = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int64_t MN = d.M * d.N, t = (int64_t)blockIdx.x * 32 + x;
  double s = 0.0;
  if (t < MN) {
#pragma unroll 4
    for (int z = g; z < splits; z += 8) s += partial[(int64_t)z * MN + t];
  }
  part[g][x] = s;
  __syncthreads();
  if (g != 0 || t >= MN) return;
#pragma unroll
  for (int q = 1; q < 8; ++q) s += part[q][x];
  const uint32_t m = (uint32_t)t / (uint32_t)d.N, n = (uint32_t)t - m * (uint32_t)d.N;
  f64_store(C + off3(m, d.M2, d.M3, d.c_m1, d.c_m2, d.c_m3) + off3(n, d.N2, d.N3, d.c_n1, d.c_n2, d.c_n3), s,
            d.alpha, d.beta);
}

// Small contractions: a block of four warps per 8 x 8 output tile and K range,
// the k-steps of four dealt to the warps in turn, operands read straight into
// the fragments of m8n8k4.  An SM does two FP64 FMAs per clk, so one m8n8k4
// takes the SM 128 clk, its two loads are free, and what counts is that the work
// reaches all SMs: with 64 x 64 tiles the contractions of a dimer ran on 1-25
// SMs (a 46 x 46 x 46 product took 97 us on one), with 16 x 16 tiles a 90 x 90 x
// 90 one ran on 36 (13 us; 6 here).  Where the tiles are fewer than the SMs a
// cluster of up to eight blocks shares a tile's K and the first block adds the
// sums, read from the others' shared memory, in block order: no second launch
// and no partial sums in memory (15 x 190 x 190: 21 us with 16 x 16 tiles, 6
// here).
constexpr int SM_T = 8, SM_WARPS = 4;
__global__ void __launch_bounds__(32 * SM_WARPS) contract_f64_small_kernel(const double* __restrict__ A,
                                                                           const double* __restrict__ B,
                                                                           double* __restrict__ C, CtrDesc d,
                                                                           int k_chunk, int cl,
                                                                           double* __restrict__ partial) {
  __shared__ double part[SM_WARPS][SM_T * SM_T];
  __shared__ double sum[SM_T * SM_T];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t m0 = (int64_t)blockIdx.x * SM_T, n0 = (int64_t)blockIdx.y * SM_T;
  // z: K range of a partial product, or (batch, block of the cluster)
  const uint32_t zb = partial ? 0 : blockIdx.z / (uint32_t)cl;
  const int zk = partial ? (int)blockIdx.z : (int)(blockIdx.z - zb * (uint32_t)cl);
  // unsigned: K is below 2^31, a loop's last step may not be
  const uint32_t kbeg = (uint32_t)zk * (uint32_t)k_chunk;
  const uint32_t kend = min((uint32_t)d.K, kbeg + (uint32_t)k_chunk);
  A += (int64_t)zb * d.a_b;
  B += (int64_t)zb * d.b_b;
  C += (int64_t)zb * d.c_b;
  const int64_t m = m0 + (lane >> 2), n = n0 + (lane >> 2);
  const bool rok = m < d.M, cok = n < d.N;
  const int64_t ra = rok ? off3(m, d.M2, d.M3, d.a_m1, d.a_m2, d.a_m3) : 0;
  const int64_t cb = cok ? off3(n, d.N2, d.N3, d.b_n1, d.b_n2, d.b_n3) : 0;
  double acc[2][2] = {{0.0, 0.0}, {0.0, 0.0}};
  constexpr int U = 8;   // k-steps in flight
  for (uint32_t k0 = kbeg + 4 * warp; k0 < kend; k0 += 4 * SM_WARPS * U) {
    double a[U], b[U];
#pragma unroll
    for (int q = 0; q < U; ++q) {
      const uint32_t k = k0 + 4 * SM_WARPS * q + (lane & 3);
      a[q] = b[q] = 0.0;
      if (k < kend) {
        const uint32_t k1 = k / (uint32_t)d.K2, k2 = k - k1 * (uint32_t)d.K2;
        if (rok) a[q] = A[ra + (int64_t)k1 * d.a_k1 + (int64_t)k2 * d.a_k2];
        if (cok) b[q] = B[cb + (int64_t)k1 * d.b_k1 + (int64_t)k2 * d.b_k2];
      }
    }
#pragma unroll
    for (int q = 0; q < U; ++q) {
      if (k0 + 4 * SM_WARPS * q >= kend) break;
      dmma884(acc[q & 1][0], acc[q & 1][1], a[q], b[q]);
    }
  }
  // lane: row lane / 4, columns 2 (lane % 4) and the next
  part[warp][2 * lane] = acc[0][0] + acc[1][0];
  part[warp][2 * lane + 1] = acc[0][1] + acc[1][1];
  __syncthreads();
  double s = 0.0;
  if (tid < SM_T * SM_T) {
    s = part[0][tid];
#pragma unroll
    for (int w = 1; w < SM_WARPS; ++w) s += part[w][tid];
  }
  if (!partial && cl > 1) {
    if (tid < SM_T * SM_T) sum[tid] = s;
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (zk == 0 && tid < SM_T * SM_T) {
      const uint32_t own = (uint32_t)__cvta_generic_to_shared(&sum[tid]);
      double other[7];
#pragma unroll
      for (int q = 1; q < 8; ++q) {
        other[q - 1] = 0.0;
        if (q < cl) {
          uint32_t addr;
          asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(addr) : "r"(own), "r"(q));
          asm volatile("ld.shared::cluster.f64 %0, [%1];" : "=d"(other[q - 1]) : "r"(addr) : "memory");
        }
      }
#pragma unroll
      for (int q = 1; q < 8; ++q)
        if (q < cl) s += other[q - 1];
    }
    // the other blocks' shared memory stays until it is read
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
    if (zk != 0) return;
  }
  if (tid >= SM_T * SM_T) return;
  const int64_t mo = m0 + (tid >> 3), no = n0 + (tid & 7);
  if (mo >= d.M || no >= d.N) return;
  if (partial) {
    partial[((int64_t)blockIdx.z * d.M + mo) * d.N + no] = s;
  } else {
    f64_store(C + off3(mo, d.M2, d.M3, d.c_m1, d.c_m2, d.c_m3) + off3(no, d.N2, d.N3, d.c_n1, d.c_n2, d.c_n3), s,
              d.alpha, d.beta);
  }
}

// N == 1 (matrix-vector): one warp per output row, lanes stride over K.
__global__ void gemv_f64_kernel(const double* __restrict__ A, const double* __restrict__ B, double* __restrict__ C,
                                CtrDesc d) {
  const int lane = threadIdx.x & 31;
  const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  const int64_t bz = blockIdx.y;
  A += bz * d.a_b;
  B += bz * d.b_b;
  C += bz * d.c_b;
  for (int64_t m = warp; m < d.M; m += nwarps) {
    const double* a = A + off3(m, d.M2, d.M3, d.a_m1, d.a_m2, d.a_m3);
    double s = 0.0;
#pragma unroll 4
    for (int64_t k = lane; k < d.K; k += 32) s += a[off2(k, d.K2, d.a_k1, d.a_k2)] * B[off2(k, d.K2, d.b_k1, d.b_k2)];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (lane == 0) f64_store(C + off3(m, d.M2, d.M3, d.c_m1, d.c_m2, d.c_m3), s, d.alpha, d.beta);
  }
}

// N == 1 with the rows adjacent in memory (unit stride along m): 32 rows per
// block, lanes along the rows so that reads coalesce, a warp for each residue of
// k modulo 32.  The sums are those of gemv_f64_kernel bit for bit (lane k mod 32,
// then halves): the mixed form's digits are cut from what follows from them, and
// its iterates should not depend on the memory layout of an operand.
__global__ void __launch_bounds__(1024) gemv_cols_f64_kernel(const double* __restrict__ A, const double* __restrict__ B,
                                                             double* __restrict__ C, CtrDesc d) {
  __shared__ double part[32][33];
  const int x = threadIdx.x & 31, g = threadIdx.x >> 5;
  const int64_t m0 = (int64_t)blockIdx.x * 32, m = m0 + x;
  const int64_t bz = blockIdx.y;
  A += bz * d.a_b;
  B += bz * d.b_b;
  C += bz * d.c_b;
  double s = 0.0;
  if (m < d.M) {
    const double* a = A + off3(m, d.M2, d.M3, d.a_m1, d.a_m2, d.a_m3);
    if (d.K2 >= d.K) {
#pragma unroll 8
      for (int64_t k = g; k < d.K; k += 32) s = fma(a[k * d.a_k2], B[k * d.b_k2], s);
    } else {
#pragma unroll 4
      for (int64_t k = g; k < d.K; k += 32)
        s = fma(a[off2(k, d.K2, d.a_k1, d.a_k2)], B[off2(k, d.K2, d.b_k1, d.b_k2)], s);
    }
  }
  part[g][x] = s;
  __syncthreads();
  s = part[x][g];   // row m0 + g
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if (x == 0 && m0 + g < d.M) f64_store(C + off3(m0 + g, d.M2, d.M3, d.c_m1, d.c_m2, d.c_m3), s, d.alpha, d.beta);
}

// out[i0 i1 i2 i3] = alpha in + beta out: a warp per run of up to 128 elements
// of the last index (runs of equal length), so the index arithmetic is per run.
__global__ void __launch_bounds__(256) axpby4_kernel(const double* __restrict__ in, double* __restrict__ out,
                                                     uint32_t d1, uint32_t d2, uint32_t d3, int64_t si0, int64_t si1,
                                                     int64_t si2, int64_t si3, int64_t so0, int64_t so1, int64_t so2,
                                                     int64_t so3, double alpha, double beta, uint32_t nseg,
                                                     uint32_t seglen, int64_t runs) {
  const int lane = threadIdx.x & 31;
  const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < runs; w += nw) {
    uint32_t r = (uint32_t)w;
    const uint32_t seg = r % nseg;
    r /= nseg;
    const uint32_t i2 = r % d2;
    r /= d2;
    const uint32_t i1 = r % d1, i0 = r / d1;
    const double* src = in + (int64_t)i0 * si0 + (int64_t)i1 * si1 + (int64_t)i2 * si2;
    double* dst = out + (int64_t)i0 * so0 + (int64_t)i1 * so1 + (int64_t)i2 * so2;
    const uint32_t jend = min(d3, (seg + 1) * seglen), jw = seg * seglen, j0 = jw + lane;
    double v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t j = j0 + 32 * q;
      v[q] = j < jend ? src[(int64_t)j * si3] : 0.0;
    }
    double p[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t j = j0 + 32 * q;
      p[q] = beta != 0.0 && j < jend ? dst[(int64_t)j * so3] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t j = j0 + 32 * q;
      if (jw + 32 * q >= jend) break;   // an FP64 instruction takes its 16 clk also where no lane needs it
      if (j < jend) dst[(int64_t)j * so3] = f64_axpby(v[q], p[q], alpha, beta);
    }
  }
}

// The same where the source's fastest index is another one (tx) than the
// output's (the last): 32 x 32 tiles through shared memory, both sides
// coalesced.  The other two indices are (oa, ob).
__global__ void __launch_bounds__(256) axpby4_tr_kernel(const double* __restrict__ in, double* __restrict__ out,
                                                        uint32_t dx, uint32_t d3, uint32_t db, int64_t six,
                                                        int64_t si3, int64_t sia, int64_t sib, int64_t sox,
                                                        int64_t so3, int64_t soa, int64_t sob, double alpha,
                                                        double beta, uint32_t ntx, uint32_t nt3, uint32_t tiles) {
  __shared__ double tile[32][33];
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  for (uint32_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    uint32_t r = t;
    const uint32_t x0 = (r % ntx) * 32;
    r /= ntx;
    const uint32_t j0 = (r % nt3) * 32;
    r /= nt3;
    const uint32_t ib = r % db, ia = r / db;
    const double* src = in + (int64_t)ia * sia + (int64_t)ib * sib;
    double* dst = out + (int64_t)ia * soa + (int64_t)ib * sob;
    __syncthreads();   // the previous tile is consumed
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t x = x0 + tx, j = j0 + ty + 8 * q;
      if (x < dx && j < d3) tile[ty + 8 * q][tx] = src[(int64_t)x * six + (int64_t)j * si3];
    }
    __syncthreads();
    double p[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t x = x0 + ty + 8 * q, j = j0 + tx;
      p[q] = beta != 0.0 && x < dx && j < d3 ? dst[(int64_t)x * sox + (int64_t)j * so3] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const uint32_t x = x0 + ty + 8 * q, j = j0 + tx;
      if (x < dx && j < d3)
        dst[(int64_t)x * sox + (int64_t)j * so3] = f64_axpby(tile[tx][ty + 8 * q], p[q], alpha, beta);
    }
  }
}

}  // namespace

void contract_f64_launch(const double* A, const double* B, double* C, const CtrDesc& d, cudaStream_t s) {
  if (d.M <= 0 || d.N <= 0 || d.batch <= 0) return;
  if (d.M >= (int64_t(1) << 31) || d.N >= (int64_t(1) << 31) || d.K >= (int64_t(1) << 31))
    fail(FCC_ERR_BAD_ARG, "contraction extent too large");
  if (d.K <= 0) fail(FCC_ERR_BAD_ARG, "empty contraction index");
  int64_t gm = (d.M + BM - 1) / BM, gn = (d.N + BN - 1) / BN;
  if (gn > 65535 || d.batch > 65535) fail(FCC_ERR_BAD_ARG, "contraction grid too large");
  const int pidx = prof_begin(s);
  const double pflops = 2.0 * (double)d.M * (double)d.N * (double)d.K * (double)d.batch;
  // stage along M (N) when the fastest-moving M (N) index has unit stride
  const int a_fast = (d.M3 > 1 ? d.a_m3 : d.a_m2) == 1 ? 1 : 0;
  const int b_fast = (d.N3 > 1 ? d.b_n3 : d.b_n2) == 1 ? 1 : 0;
  if (d.N == 1) {
    if (a_fast && d.M >= 32) {
      gemv_cols_f64_kernel<<<dim3((unsigned)((d.M + 31) / 32), (unsigned)d.batch), 1024, 0, s>>>(A, B, C, d);
    } else {
      const int64_t blocks = std::min<int64_t>((d.M + 7) / 8, 152 * 16);
      gemv_f64_kernel<<<dim3((unsigned)blocks, (unsigned)d.batch), 256, 0, s>>>(A, B, C, d);
    }
    FCC_CHECK_LAUNCH();
    prof_end(s, pidx, PROF_F64, pflops);
    return;
  }
  auto workspace = [&](DBuf<double>& local, int64_t need) -> double* {
    DBuf<double>* ws = f64_workspace();
    if (!ws) ws = &local;
    if ((int64_t)ws->n < need) ws->alloc(need);
    return ws->p;
  };
  DBuf<double> local;
  const int64_t MN = d.M * d.N;
  const unsigned rgrid = (unsigned)std::min<int64_t>((MN + 255) / 256, 152 * 8);
  // 8 x 8 tiles while the 64 x 64 ones would leave SMs without work.  Up to
  // eight blocks share a tile while there are fewer than two blocks per SM and
  // each has 16 values of k; a longer K over few tiles (over 512 a block) is cut
  // into partial sums for all SMs, reduced in a fixed order by a second launch.
  const int64_t sm = (d.M + SM_T - 1) / SM_T, sn = (d.N + SM_T - 1) / SM_T;
  if (!d.wide && gm * gn * d.batch < 3 * 152 && sn <= 65535) {
    int64_t cl = 1;
    while (cl < 8 && sm * sn * d.batch * cl < 152 && d.K >= 32 * cl && d.batch * cl * 2 <= 65535) cl *= 2;
    const int64_t splits0 = (304 + sm * sn - 1) / (sm * sn);
    if (d.batch == 1 && splits0 > 8 && d.K > 4096) {
      const int64_t chunk = ((d.K + splits0 - 1) / splits0 + 15) / 16 * 16;
      const int64_t splits = (d.K + chunk - 1) / chunk;
      double* part = workspace(local, splits * MN);
      contract_f64_small_kernel<<<dim3((unsigned)sm, (unsigned)sn, (unsigned)splits), 32 * SM_WARPS, 0, s>>>(
          A, B, C, d, (int)chunk, 1, part);
      FCC_CHECK_LAUNCH();
      if (MN <= 152 * 32) {
        splitk_reduce_few_kernel<<<(unsigned)((MN + 31) / 32), 256, 0, s>>>(part, (int)splits, C, d);
      } else {
        splitk_reduce_kernel<<<rgrid, 256, 0, s>>>(part, (int)splits, C, d);
      }
    } else {
      const int chunk = (int)(((d.K + cl - 1) / cl + 3) / 4 * 4);
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3((unsigned)sm, (unsigned)sn, (unsigned)(d.batch * cl));
      cfg.blockDim = dim3(32 * SM_WARPS);
      cfg.stream = s;
      cudaLaunchAttribute at[1];
      at[0].id = cudaLaunchAttributeClusterDimension;
      at[0].val.clusterDim.x = at[0].val.clusterDim.y = 1;
      at[0].val.clusterDim.z = (unsigned)cl;
      cfg.attrs = at;
      cfg.numAttrs = 1;
      FCC_CUDA(cudaLaunchKernelEx(&cfg, contract_f64_small_kernel, A, B, C, d, chunk, (int)cl, (double*)nullptr));
    }
    FCC_CHECK_LAUNCH();
    prof_end(s, pidx, PROF_F64, pflops);
    return;
  }
  // fewer output tiles than one wave of resident CTAs (96 registers x 128
  // threads: 5 per SM) and a long K: split K so that about 8 CTAs per SM
  // share the work.  Under one wave the FP64 pipe idles on DMMA latency:
  // 387 CTAs ran at 0.8 TFLOP/s where 1216 reach 1.08.
  constexpr int64_t WAVE_CTAS = 5 * 152, SPLIT_CTAS = 8 * 152;
  if (d.batch == 1 && gm * gn < WAVE_CTAS && d.K >= 32 * BK) {
    int64_t splits = std::min<int64_t>((SPLIT_CTAS + gm * gn - 1) / (gm * gn), d.K / (8 * BK));
    splits = std::max<int64_t>(2, std::min<int64_t>(splits, 1024));
    const int64_t chunk = ((d.K + splits - 1) / splits + BK - 1) / BK * BK;
    splits = (d.K + chunk - 1) / chunk;
    double* part = workspace(local, splits * MN);
    dim3 grid((unsigned)gm, (unsigned)gn, (unsigned)splits);
    CtrDesc full = d;
    full.sym = false;
    contract_f64_kernel<<<grid, NT, 0, s>>>(A, B, C, full, a_fast, b_fast, chunk, part);
    FCC_CHECK_LAUNCH();
    splitk_reduce_kernel<<<rgrid, 256, 0, s>>>(part, (int)splits, C, d);
    FCC_CHECK_LAUNCH();
    prof_end(s, pidx, PROF_F64, pflops);
    return;
  }
  dim3 grid((unsigned)gm, (unsigned)gn, (unsigned)d.batch);
  contract_f64_kernel<<<grid, NT, 0, s>>>(A, B, C, d, a_fast, b_fast, d.K, nullptr);
  FCC_CHECK_LAUNCH();
  if (d.sym) {
    const unsigned t = (unsigned)((d.M + 31) / 32);
    mirror_kernel<<<dim3(t, t), 256, 0, s>>>(C, d);
    FCC_CHECK_LAUNCH();
  }
  prof_end(s, pidx, PROF_F64, pflops);
}

void tensor_axpby_launch(const TView& in, const TView& out, double alpha, double beta, cudaStream_t s) {
  int64_t total = 1;
  for (int k = 0; k < 4; ++k) {
    total *= out.dim[k];
    if (out.dim[k] >= (int64_t(1) << 31)) fail(FCC_ERR_BAD_ARG, "tensor extent too large");
  }
  if (total <= 0) return;
  // Indices slowest first by their stride in the output (unit extents in
  // front), so the last one is what the threads run along.
  int ord[4] = {0, 1, 2, 3};
  std::stable_sort(ord, ord + 4, [&](int a, int b) {
    const bool ua = out.dim[a] == 1, ub = out.dim[b] == 1;
    if (ua != ub) return ua;
    return std::llabs(out.str[a]) > std::llabs(out.str[b]);
  });
  int64_t dim[4], si[4], so[4];
  for (int k = 0; k < 4; ++k) {
    dim[k] = out.dim[ord[k]];
    si[k] = in.str[ord[k]];
    so[k] = out.str[ord[k]];
  }
  // neighbouring indices that are contiguous in both tensors become one
  for (int k = 2; k >= 0; --k) {
    int n = k + 1;                       // the next slower non-unit index is k
    if (dim[k] == 1) continue;
    if (dim[n] > 1 && si[k] == dim[n] * si[n] && so[k] == dim[n] * so[n] && dim[k] * dim[n] < (int64_t(1) << 31)) {
      dim[n] *= dim[k];
      for (int q = k; q > 0; --q) { dim[q] = dim[q - 1]; si[q] = si[q - 1]; so[q] = so[q - 1]; }
      dim[0] = 1;
      si[0] = so[0] = 0;
      ++k;                               // what moved into place k is looked at next
    }
  }
  // the source's fastest index, if it is another one than the output's
  int x = 3;
  for (int k = 0; k < 3; ++k)
    if (dim[k] > 1 && std::llabs(si[k]) < std::llabs(si[x])) x = k;
  if (x != 3 && dim[x] >= 8 && dim[3] >= 8) {
    const int o1 = x == 0 ? 1 : 0, o2 = x == 2 ? 1 : 2;   // the other two, slower first
    const int64_t ntx = (dim[x] + 31) / 32, nt3 = (dim[3] + 31) / 32;
    const int64_t tiles = ntx * nt3 * dim[o1] * dim[o2];
    if (tiles >= (int64_t(1) << 31)) fail(FCC_ERR_BAD_ARG, "tensor too large");
    axpby4_tr_kernel<<<(unsigned)std::min<int64_t>(tiles, 152 * 16), 256, 0, s>>>(
        in.p, out.p, (uint32_t)dim[x], (uint32_t)dim[3], (uint32_t)dim[o2], si[x], si[3], si[o1], si[o2], so[x], so[3],
        so[o1], so[o2], alpha, beta, (uint32_t)ntx, (uint32_t)nt3, (uint32_t)tiles);
    FCC_CHECK_LAUNCH();
    return;
  }
  const int64_t nseg = (dim[3] + 127) / 128, seglen = ((dim[3] + nseg - 1) / nseg + 31) / 32 * 32;
  const int64_t runs = dim[0] * dim[1] * dim[2] * nseg;
  if (runs >= (int64_t(1) << 31)) fail(FCC_ERR_BAD_ARG, "tensor too large");
  axpby4_kernel<<<(unsigned)std::min<int64_t>((runs + 7) / 8, 152 * 16), 256, 0, s>>>(
      in.p, out.p, (uint32_t)dim[1], (uint32_t)dim[2], (uint32_t)dim[3], si[0], si[1], si[2], si[3], so[0], so[1],
      so[2], so[3], alpha, beta, (uint32_t)nseg, (uint32_t)seglen, runs);
  FCC_CHECK_LAUNCH();
}

// ------------------------------------------------------------ einsum front end
namespace {

struct Operand {
  std::string idx;
  const TView* t;
  int pos(char c) const { auto p = idx.find(c); return p == std::string::npos ? -1 : (int)p; }
  int64_t stride(char c) const { int p = pos(c); return p < 0 ? 0 : t->str[p]; }
  int64_t dim(char c) const { int p = pos(c); return p < 0 ? 1 : t->dim[p]; }
};

// A merged index: extent plus the stride it has in each operand.
struct Ix {
  int64_t dim;
  int64_t s[3];
};

void parse(const char* spec, std::vector<std::string>& ins, std::string& out) {
  std::string s(spec);
  auto arrow = s.find("->");
  if (arrow == std::string::npos) fail(FCC_ERR_BAD_ARG, std::string("einsum spec without ->: ") + spec);
  out = s.substr(arrow + 2);
  std::string lhs = s.substr(0, arrow);
  size_t start = 0;
  while (true) {
    auto c = lhs.find(',', start);
    ins.push_back(lhs.substr(start, c == std::string::npos ? std::string::npos : c - start));
    if (c == std::string::npos) break;
    start = c + 1;
  }
}

// Fuse indices of a group until it has at most `cap` members; two indices x
// (slower) and y (faster) fuse when str[x] == dim[y] * str[y] in every operand.
bool try_fuse(std::vector<Ix>& g, int cap) {
  while ((int)g.size() > cap) {
    bool done = false;
    for (size_t x = 0; x < g.size() && !done; ++x)
      for (size_t y = 0; y < g.size() && !done; ++y) {
        if (x == y) continue;
        bool ok = true;
        for (int o = 0; o < 3; ++o) {
          bool zx = g[x].s[o] == 0, zy = g[y].s[o] == 0;
          if (zx != zy) { ok = false; break; }
          if (!zx && g[x].s[o] != g[y].dim * g[y].s[o]) { ok = false; break; }
        }
        if (ok) {
          g[y].dim *= g[x].dim;
          g.erase(g.begin() + x);
          done = true;
        }
      }
    if (!done) return false;
  }
  return true;
}

void fuse(std::vector<Ix>& g, int cap, const char* spec) {
  if (!try_fuse(g, cap)) fail(FCC_ERR_BAD_ARG, std::string("einsum group not reducible to ") + std::to_string(cap) + " indices: " + spec);
}

int64_t gdim(const std::vector<Ix>& g) {
  int64_t d = 1;
  for (auto& x : g) d *= x.dim;
  return d;
}

// pad a group to exactly 3 levels (slowest first)
void pad3(std::vector<Ix>& g) { while (g.size() < 3) g.insert(g.begin(), Ix{1, {0, 0, 0}}); }

bool same_spec(const PackSpec& a, const PackSpec& b) {
  return a.R == b.R && a.K == b.K && a.Kp == b.Kp && a.rd2 == b.rd2 && a.rd3 == b.rd3 && a.rs1 == b.rs1 &&
         a.rs2 == b.rs2 && a.rs3 == b.rs3 && a.kd2 == b.kd2 && a.kd3 == b.kd3 && a.ks1 == b.ks1 && a.ks2 == b.ks2 &&
         a.ks3 == b.ks3 && a.P == b.P && a.code == b.code && a.scale == b.scale;
}

// The entry of the engine's kept operands that belongs to the source `src` of
// operand A (nullptr: not one of the kept sources).
TcEngine::KeptPack* kept_of(TcEngine* tc, const double* src) {
  for (int i = 0; i < 2; ++i)
    if (src && tc->keep_src[i] == src) return &tc->kept[i];
  return nullptr;
}

// Whether a kept operand has to be packed now: (ps, lv) is not what it holds.
// lv.S = 0: the split scheme.
bool kept_stale(TcEngine::KeptPack* k, const PackSpec& ps, const OzLevel& lv) {
  if (k->valid && k->S == lv.S && k->bits == lv.bits && k->guard == lv.guard && same_spec(k->ps, ps)) return false;
  k->ps = ps;
  k->S = lv.S;
  k->bits = lv.bits;
  k->guard = lv.guard;
  k->valid = true;
  return true;
}

// Tensor-core evaluation of C = alpha * A.B + beta * C (no batch index): by
// exact-slice products of level lv, or (lv.S = 0) by the engine's split scheme.
// `optional`: false, with nothing done, where scratch cannot be had.
bool run_tc(TcEngine* tc, bool optional, OzLevel lv, double alpha, const TView& A, const TView& B, double beta, const TView& C,
            std::vector<Ix> gm, std::vector<Ix> gn, std::vector<Ix> gk, cudaStream_t s) {
  // fastest-moving member last: the one with the smallest stride in the operand that is read along it
  auto order = [](std::vector<Ix>& g, int op) {
    std::stable_sort(g.begin(), g.end(), [op](const Ix& a, const Ix& b) { return std::llabs(a.s[op]) > std::llabs(b.s[op]); });
  };
  order(gm, 2);
  order(gn, 2);
  order(gk, 0);
  pad3(gm); pad3(gn); pad3(gk);
  const int64_t M = gdim(gm), N = gdim(gn), K = gdim(gk);
  ScratchInUse in_use(tc);
  auto grow = [&](auto& buf, int64_t n) {
    if ((int64_t)buf.n >= n) return true;
    if (optional) return buf.try_alloc(n);
    buf.alloc(n);
    return true;
  };
  if (lv.S > 0) {
    // exact-slice products: S digit slices of each operand, FP64 output
    const int S = lv.S;
    const int64_t Kpad = oz_kpad(K), W = S * Kpad;
    TcEngine::KeptPack* ka = kept_of(tc, A.p);
    auto& bufA = ka ? ka->buf : tc->bufA;
    auto& exA = ka ? ka->ex : tc->exA;
    if (ka && ((int64_t)bufA.n < M * W || (int64_t)exA.n < M)) ka->valid = false;
    if (!grow(bufA, M * W) || !grow(tc->bufB, N * W) || !grow(exA, M) || !grow(tc->exB, N)) return false;
    PackSpec pa{M, K, W, gm[1].dim, gm[2].dim, gm[0].s[0], gm[1].s[0], gm[2].s[0],
                gk[1].dim, gk[2].dim, gk[0].s[0], gk[1].s[0], gk[2].s[0], S, 0};
    PackSpec pb{N, K, W, gn[1].dim, gn[2].dim, gn[0].s[1], gn[1].s[1], gn[2].s[1],
                gk[1].dim, gk[2].dim, gk[0].s[1], gk[1].s[1], gk[2].s[1], S, 0};
    if (!ka || kept_stale(ka, pa, lv)) pack_oz(A.p, pa, S, lv.bits, lv.guard, bufA.p, exA.p, s);
    pack_oz(B.p, pb, S, lv.bits, lv.guard, tc->bufB.p, tc->exB.p, s);
    EpiMap ep;
    ep.M = M; ep.N = N;
    ep.md2 = gm[1].dim; ep.md3 = gm[2].dim; ep.ms1 = gm[0].s[2]; ep.ms2 = gm[1].s[2]; ep.ms3 = gm[2].s[2];
    ep.nd2 = gn[1].dim; ep.nd3 = gn[2].dim; ep.ns1 = gn[0].s[2]; ep.ns2 = gn[1].s[2]; ep.ns3 = gn[2].s[2];
    ep.alpha = alpha; ep.beta = beta; ep.C = C.p;
    ep.work = 2.0 * (double)M * (double)N * (double)K * oz_pairs(lv);
    ep.no_loads = tc->no_loads_once;
    tc->no_loads_once = 0;
    gemm_oz(bufA.p, M, exA.p, tc->bufB.p, N, tc->exB.p, Kpad, lv, ep, tc->ozws, tc->err, s);
    tc->tc_calls++;
    tc->tc_flops += ep.work;
    return true;
  }
  const SplitScheme sc = tc->scheme;
  const int64_t Kp = packed_kp(K, sc.P);
  TcEngine::KeptPack* ka = kept_of(tc, A.p);
  auto& bufA = ka ? ka->buf : tc->bufA;
  if (ka && (int64_t)bufA.n < M * Kp) ka->valid = false;
  if (!grow(bufA, M * Kp) || !grow(tc->bufB, N * Kp)) return false;
  PackSpec pa{M, K, Kp, gm[1].dim, gm[2].dim, gm[0].s[0], gm[1].s[0], gm[2].s[0],
              gk[1].dim, gk[2].dim, gk[0].s[0], gk[1].s[0], gk[2].s[0], sc.P, sc.code_a};
  PackSpec pb{N, K, Kp, gn[1].dim, gn[2].dim, gn[0].s[1], gn[1].s[1], gn[2].s[1],
              gk[1].dim, gk[2].dim, gk[0].s[1], gk[1].s[1], gk[2].s[1], sc.P, sc.code_b};
  if (!ka || kept_stale(ka, pa, lv)) pack_split(A.p, pa, bufA.p, s);
  pack_split(B.p, pb, tc->bufB.p, s);
  EpiMap ep;
  ep.M = M; ep.N = N;
  ep.md2 = gm[1].dim; ep.md3 = gm[2].dim; ep.ms1 = gm[0].s[2]; ep.ms2 = gm[1].s[2]; ep.ms3 = gm[2].s[2];
  ep.nd2 = gn[1].dim; ep.nd3 = gn[2].dim; ep.ns1 = gn[0].s[2]; ep.ns2 = gn[1].s[2]; ep.ns3 = gn[2].s[2];
  ep.alpha = alpha; ep.beta = beta; ep.C = C.p;
  ep.work = 2.0 * (double)M * (double)N * (double)K * sc.P;
  ep.no_loads = tc->no_loads_once;
  tc->no_loads_once = 0;
  gemm_bf16x3(bufA.p, M, 0, tc->bufB.p, N, 0, Kp, ep, tc->err, s);
  tc->tc_calls++;
  tc->tc_flops += 2.0 * (double)M * (double)N * (double)K * sc.P;
  return true;
}

}  // namespace

bool TcEngine::scratch_fits(double growth) const {
  if (growth <= 0) return true;
  if (scratch_held() + growth > scratch_max) return false;
  if (growth < 2.5e8) return true;   // try_alloc sees to it, and it can be reclaimed: no need to ask the driver
  size_t f = 0, t = 0;
  return cudaMemGetInfo(&f, &t) == cudaSuccess && growth <= 0.5 * (double)f;
}

void TcEngine::release_scratch() {
  for (auto* b : {&bufA, &bufB, &bvvA, &bvvB}) b->release();
  for (auto* b : {&exA, &exB, &bvvEx}) b->release();
  ozws.release();
  for (KeptPack& k : kept) {
    k.valid = false;
    k.buf.release();
    k.ex.release();
  }
}

bool reclaim_scratch() {
  TcEngine* tc = tc_engine();
  if (!tc || tc->busy || tc->scratch_held() + (double)tc->ozws.bytes() == 0) return false;
  tc->release_scratch();
  return true;
}

static std::atomic<int64_t> g_launches{0};
void note_launch() { g_launches.fetch_add(1, std::memory_order_relaxed); }
int64_t launch_count() { return g_launches.load(std::memory_order_relaxed); }

TcEngine*& tc_engine() {
  thread_local TcEngine* e = nullptr;
  return e;
}

DBuf<double>*& f64_workspace() {
  thread_local DBuf<double>* w = nullptr;
  return w;
}

// bytes by which run_tc would grow the engine's buffers for a product
static double pack_growth(TcEngine* tc, const OzLevel& lv, const double* a, int64_t M, int64_t N, int64_t K) {
  const double w = (double)lv.S * (double)oz_kpad(K);
  const TcEngine::KeptPack* ka = kept_of(tc, a);
  const size_t na = ka ? ka->buf.n : tc->bufA.n, ne = ka ? ka->ex.n : tc->exA.n;
  auto more = [](double need, size_t have) { return std::max(0.0, need - (double)have); };
  return 2.0 * (more(M * w, na) + more(N * w, tc->bufB.n)) + 4.0 * (more(M, ne) + more(N, tc->exB.n));
}

void einsum(double alpha, const char* spec, const TView& A, const TView& B, double beta, const TView& C,
            cudaStream_t s) {
  std::vector<std::string> ins;
  std::string out;
  parse(spec, ins, out);
  if (ins.size() != 2) fail(FCC_ERR_BAD_ARG, std::string("einsum expects two operands: ") + spec);
  Operand oa{ins[0], &A}, ob{ins[1], &B}, oc{out, &C};
  if ((int)oa.idx.size() != A.rank || (int)ob.idx.size() != B.rank || (int)oc.idx.size() != C.rank)
    fail(FCC_ERR_BAD_ARG, std::string("einsum rank mismatch: ") + spec);
  std::string letters;
  for (auto& str : {oa.idx, ob.idx, oc.idx})
    for (char c : str)
      if (letters.find(c) == std::string::npos) letters += c;
  std::vector<Ix> gb, gm, gn, gk;
  for (char c : letters) {
    bool ia = oa.pos(c) >= 0, ib = ob.pos(c) >= 0, ic = oc.pos(c) >= 0;
    int64_t dim = std::max({oa.dim(c), ob.dim(c), oc.dim(c)});
    for (auto* op : {&oa, &ob, &oc})
      if (op->pos(c) >= 0 && op->dim(c) != dim)
        fail(FCC_ERR_BAD_ARG, std::string("einsum extent mismatch for '") + c + "': " + spec);
    Ix ix{dim, {oa.stride(c), ob.stride(c), oc.stride(c)}};
    if (ia && ib && ic) gb.push_back(ix);
    else if (ia && ic) gm.push_back(ix);
    else if (ib && ic) gn.push_back(ix);
    else if (ia && ib) gk.push_back(ix);
    else fail(FCC_ERR_BAD_ARG, std::string("einsum index in one operand only: ") + spec);
  }
  TcEngine* tc = tc_engine();
  if (tc && tc->enabled && gb.empty()) {
    const double flops = 2.0 * (double)gdim(gm) * (double)gdim(gn) * (double)gdim(gk);
    std::vector<Ix> m3 = gm, n3 = gn, k3 = gk;
    if (flops >= tc->min_flops && gdim(gm) >= tc->min_dim && gdim(gn) >= tc->min_dim && try_fuse(m3, 3) && try_fuse(n3, 3) &&
        try_fuse(k3, 3)) {
      run_tc(tc, false, tc->exact ? tc->oz : OzLevel{0, 0, 0, 0, 0}, alpha, A, B, beta, C, m3, n3, k3, s);
      return;
    }
  }
  // FP64: exact-slice products at the FP64 level from f64_min_flops on (see
  // TcEngine), DMMA below
  if (tc && gb.empty() && !tc->f64_wide) {
    const double flops = 2.0 * (double)gdim(gm) * (double)gdim(gn) * (double)gdim(gk);
    std::vector<Ix> m3 = gm, n3 = gn, k3 = gk;
    if (flops >= tc->f64_min_flops && gdim(gm) > 1 && gdim(gn) > 1 && oz_takes(gdim(gm), gdim(gn), gdim(gk)) &&
        try_fuse(m3, 3) && try_fuse(n3, 3) && try_fuse(k3, 3) &&
        tc->scratch_fits(pack_growth(tc, OZ_F64, A.p, gdim(gm), gdim(gn), gdim(gk))) &&
        run_tc(tc, true, OZ_F64, alpha, A, B, beta, C, m3, n3, k3, s))
      return;
  }
  fuse(gb, 1, spec);
  fuse(gm, 3, spec);
  fuse(gn, 3, spec);
  fuse(gk, 2, spec);
  if (tc) {
    tc->f64_calls++;
    tc->f64_flops += 2.0 * (double)gdim(gm) * (double)gdim(gn) * (double)gdim(gk) * (double)gdim(gb);
  }
  // order each group slowest first (the last member has the smallest stride
  // in the operand read along it), padded at the front with unit indices
  auto order = [](std::vector<Ix>& g, int op, size_t levels) {
    std::stable_sort(g.begin(), g.end(), [op](const Ix& a, const Ix& b) { return std::llabs(a.s[op]) > std::llabs(b.s[op]); });
    while (g.size() < levels) g.insert(g.begin(), Ix{1, {0, 0, 0}});
  };
  order(gm, 0, 3);
  order(gn, 1, 3);
  order(gk, 0, 2);
  if (gb.empty()) gb.push_back(Ix{1, {0, 0, 0}});
  CtrDesc d;
  d.M = gdim(gm); d.M2 = gm[1].dim; d.M3 = gm[2].dim;
  d.N = gdim(gn); d.N2 = gn[1].dim; d.N3 = gn[2].dim;
  d.K = gk[0].dim * gk[1].dim; d.K2 = gk[1].dim;
  d.batch = gb[0].dim;
  d.sym = tc && tc->f64_sym && beta == 0.0 && d.M == d.N && d.batch == 1;
  d.wide = tc && tc->f64_wide && 2.0 * (double)d.M * (double)d.N * (double)d.K >= 1e7;
  d.a_m1 = gm[0].s[0]; d.a_m2 = gm[1].s[0]; d.a_m3 = gm[2].s[0];
  d.a_k1 = gk[0].s[0]; d.a_k2 = gk[1].s[0]; d.a_b = gb[0].s[0];
  d.b_k1 = gk[0].s[1]; d.b_k2 = gk[1].s[1];
  d.b_n1 = gn[0].s[1]; d.b_n2 = gn[1].s[1]; d.b_n3 = gn[2].s[1]; d.b_b = gb[0].s[1];
  d.c_m1 = gm[0].s[2]; d.c_m2 = gm[1].s[2]; d.c_m3 = gm[2].s[2];
  d.c_n1 = gn[0].s[2]; d.c_n2 = gn[1].s[2]; d.c_n3 = gn[2].s[2]; d.c_b = gb[0].s[2];
  d.alpha = alpha;
  d.beta = beta;
  contract_f64_launch(A.p, B.p, C.p, d, s);
}

void einsum1(double alpha, const char* spec, const TView& A, double beta, const TView& C, cudaStream_t s) {
  std::vector<std::string> ins;
  std::string out;
  parse(spec, ins, out);
  if (ins.size() != 1 || (int)ins[0].size() != A.rank || (int)out.size() != C.rank || A.rank != C.rank)
    fail(FCC_ERR_BAD_ARG, std::string("einsum1 spec mismatch: ") + spec);
  TView src;
  src.p = A.p;
  src.rank = 4;
  TView dst = C;
  for (int k = C.rank; k < 4; ++k) { dst.dim[k] = 1; dst.str[k] = 0; }
  for (int k = 0; k < 4; ++k) { src.dim[k] = 1; src.str[k] = 0; }
  for (int k = 0; k < C.rank; ++k) {
    auto p = ins[0].find(out[k]);
    if (p == std::string::npos) fail(FCC_ERR_BAD_ARG, std::string("einsum1 index missing: ") + spec);
    if (A.dim[p] != C.dim[k]) fail(FCC_ERR_BAD_ARG, std::string("einsum1 extent mismatch: ") + spec);
    src.dim[k] = A.dim[p];
    src.str[k] = A.str[p];
  }
  tensor_axpby_launch(src, dst, alpha, beta, s);
}

}  // namespace fcc

// ===================================================== allocation-free GEMM
// fcc_gemm_f64_noalloc: the split-K FP64 (DMMA) contraction for callers that
// cannot allocate device memory: a host framework that owns every device
// allocation through its own pool and forbids others, or a latency-critical
// path where cudaMalloc's implicit device synchronisation is not acceptable.
// Such callers pass their own device inputs and output; the partial sums of
// the K slices live in the fixed file-scope array below instead of a
// cudaMalloc'd buffer.
//
// The array holds FCC_NOALLOC_SCRATCH doubles (16 MiB) and stays resident on
// every GPU that loads this library until the process exits.  Every call
// shares it and it keeps the last call's contents: each call writes every
// partial it later reads, so nothing needs clearing, but calls whose work
// overlaps on the GPU (different streams, or host threads without ordering)
// race on it and must be serialised by the caller.
namespace {

constexpr int64_t FCC_NOALLOC_SCRATCH = int64_t(1) << 21;
__device__ __align__(256) double g_noalloc_scratch[FCC_NOALLOC_SCRATCH];

// Device address of g_noalloc_scratch, looked up once per device with that
// device current (a host-side reference to the symbol is not a device address).
double* noalloc_scratch_ptr(int& status) {
  static std::mutex mu;
  static double* ptr[64] = {nullptr};
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { status = FCC_ERR_NO_DEVICE; return nullptr; }
  std::lock_guard<std::mutex> lock(mu);
  if (!ptr[dev]) {
    void* p = nullptr;
    if (cudaGetSymbolAddress(&p, g_noalloc_scratch) != cudaSuccess || !p) { status = FCC_ERR_CUDA; return nullptr; }
    ptr[dev] = static_cast<double*>(p);
  }
  status = FCC_OK;
  return ptr[dev];
}

}  // namespace

extern "C" int fcc_gemm_f64_noalloc(int64_t M, int64_t N, int64_t K, double alpha, const double* A, int64_t lda,
                                    const double* B, int64_t ldb, double beta, double* C, int64_t ldc, void* stream) {
  using namespace fcc;
  if (M <= 0 || N <= 0 || K <= 0 || !A || !B || !C || lda < K || ldb < N || ldc < N) return FCC_ERR_BAD_ARG;
  // M and N are bounded one at a time first, so M * N cannot overflow
  if (M > FCC_NOALLOC_SCRATCH / 2 || N > FCC_NOALLOC_SCRATCH / 2) return FCC_ERR_BAD_ARG;
  if (M * N > FCC_NOALLOC_SCRATCH / 2) return FCC_ERR_BAD_ARG;   // at least two K slices must fit
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  // the scratch address is the current device's: the stream must belong to it
  if (s) {
    int cur = -1, sdev = -1;
    if (cudaGetDevice(&cur) != cudaSuccess || cudaStreamGetDevice(s, &sdev) != cudaSuccess) return FCC_ERR_CUDA;
    if (cur != sdev) return FCC_ERR_BAD_ARG;
  }
  int st = FCC_OK;
  double* scratch = noalloc_scratch_ptr(st);
  if (!scratch) return st;
  // index arithmetic is 32-bit: a longer K goes in pieces added to C
  constexpr int64_t KMAX = int64_t(1) << 30;
  for (int64_t k0 = KMAX; k0 < K; k0 += KMAX) {
    const int rc = fcc_gemm_f64_noalloc(M, N, std::min(KMAX, K - k0), alpha, A + k0, lda, B + k0 * ldb, ldb,
                                        k0 == KMAX ? beta : 1.0, C, ldc, stream);
    if (rc != FCC_OK) return rc;
  }
  if (K > KMAX) {
    K = KMAX;
    beta = 1.0;
  }
  CtrDesc d;
  d.M = M; d.M2 = 1; d.N = N; d.N2 = N; d.K = K; d.K2 = K; d.batch = 1;
  d.a_m1 = lda; d.a_m2 = 0; d.a_k1 = 0; d.a_k2 = 1; d.a_b = 0;
  d.b_k1 = 0; d.b_k2 = ldb; d.b_n1 = 0; d.b_n2 = 1; d.b_b = 0;
  d.c_m1 = ldc; d.c_m2 = 0; d.c_n1 = 0; d.c_n2 = 1; d.c_b = 0;
  d.alpha = alpha;
  d.beta = beta;
  const int64_t gm = (M + BM - 1) / BM, gn = (N + BN - 1) / BN;
  if (gn > 65535) return FCC_ERR_BAD_ARG;
  int64_t splits = std::min<int64_t>(std::max<int64_t>(2, (2 * 152 + gm * gn - 1) / (gm * gn)), (K + BK - 1) / BK);
  splits = std::max<int64_t>(1, std::min<int64_t>(splits, FCC_NOALLOC_SCRATCH / (M * N)));
  const int64_t chunk = ((K + splits - 1) / splits + BK - 1) / BK * BK;
  splits = (K + chunk - 1) / chunk;
  dim3 grid((unsigned)gm, (unsigned)gn, (unsigned)splits);
  contract_f64_kernel<<<grid, NT, 0, s>>>(A, B, C, d, 0, 1, chunk, scratch);
  if (cudaGetLastError() != cudaSuccess) return FCC_ERR_CUDA;
  note_launch();
  const int64_t MN = M * N;
  splitk_reduce_kernel<<<(unsigned)std::min<int64_t>((MN + 255) / 256, 152 * 8), 256, 0, s>>>(scratch, (int)splits, C, d);
  if (cudaGetLastError() != cudaSuccess) return FCC_ERR_CUDA;
  note_launch();
  return FCC_OK;
}
