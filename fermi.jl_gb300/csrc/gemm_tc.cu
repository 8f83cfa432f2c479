// Split-BF16 tensor-core contraction for GB300 (sm_103a): tcgen05.mma with the
// accumulator in TMEM, operands staged by TMA (cp.async.bulk.tensor) into
// 128-byte-swizzled shared memory, an mbarrier pipeline between one producer
// thread, one MMA-issuing thread and four epilogue warps.
//
// A FP64 contraction C = alpha * A.B + beta * C is evaluated as one BF16 GEMM
// over a K-concatenated operand pair (three products, FP32 accumulation):
//   A' = [hi(A) | hi(A) | lo(A)],  B' = [hi(B) | lo(B) | hi(B)]
//   A'.B'^T = hi(A) hi(B) + hi(A) lo(B) + lo(A) hi(B)
// with hi(x) = bf16(x) and lo(x) = bf16(x - hi(x)).  The pack kernel gathers
// the operand from any strided tensor view (the index permutation of the
// contraction is folded into it) and the epilogue scatters into any strided
// output view, so no separate transpose pass exists.
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cstring>
#include <mutex>

#include "fcc_tc.cuh"
#include "fcc_tcgen05.cuh"

namespace fcc {

namespace {

using namespace tc5;

constexpr int BM = 128;
constexpr int BK = 64;                       // one 128-byte swizzle atom of bf16 per row
constexpr int TC_THREADS = 192;              // warp 0 TMA, warp 1 MMA, warps 2-5 epilogue

template <int BN>
struct TcCfg {
  static constexpr int STAGES = (BN == 256) ? 4 : 6;
  static constexpr int A_BYTES = BM * BK * 2;
  static constexpr int B_BYTES = BN * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int SMEM = STAGES * STAGE_BYTES + 1024;  // + alignment slack
};

// bf16 bits of (-1)^sgn * m * 2^e for 0 <= m <= 256; zero below the bf16
// normal range (|value| < 2^-126), infinity above it.
__device__ __forceinline__ uint16_t bf16_bits(uint32_t sgn, uint32_t m, int e) {
  if (m == 0) return 0;
  const int lz = __clz(m) - 24;              // m in [1, 255]: shift up to [128, 255]
  if (lz >= 0) { m <<= lz; e -= lz; }
  else { m >>= 1; e += 1; }                  // m == 256
  const int b = e + 7 + 127;                 // m * 2^e = (m / 128) * 2^(e + 7)
  if (b <= 0) return 0;
  if (b >= 255) return (uint16_t)((sgn << 15) | 0x7F80u);
  return (uint16_t)((sgn << 15) | ((uint32_t)b << 7) | (m & 0x7Fu));
}

// a (0 < a < 2^62) rounded to nearest-even at 8 significant bits: returns m
// in [1, 256] with a ~ m * 2^sh
__device__ __forceinline__ uint32_t round8(uint64_t a, int& sh) {
  const int n = 64 - __clzll((long long)a);
  if (n <= 8) { sh = 0; return (uint32_t)a; }
  sh = n - 8;
  const uint64_t q = a >> sh, rem = a & ((1ull << sh) - 1), half = 1ull << (sh - 1);
  return (uint32_t)(q + ((rem > half || (rem == half && (q & 1))) ? 1u : 0u));
}

// hi, mid, lo bf16 pieces of x, each the nearest (ties to even) 8-bit value to
// what the previous pieces leave, so |x - hi - mid - lo| <= 2^-24 |x|
// (typically ~2^-27; pieces below the bf16 range become zero).  Integer arithmetic on the
// FP64 bit pattern: the remainders are exact and no FP64 instruction (a slow
// pipe on this part) is issued.
__device__ __noinline__ void split3_int(double x, __nv_bfloat16 (&lv)[3]) {
  const uint64_t u = (uint64_t)__double_as_longlong(x);
  const int ex = (int)((u >> 52) & 0x7FF);
  uint16_t h = 0, m = 0, l = 0;
  if (ex == 0x7FF) {                         // inf keeps its sign, nan becomes the canonical bf16 nan
    const bool nan = (u & ((1ull << 52) - 1)) != 0;
    lv[0] = __ushort_as_bfloat16(nan ? (unsigned short)0x7FFF : (unsigned short)(((u >> 48) & 0x8000u) | 0x7F80u));
    lv[1] = lv[2] = __ushort_as_bfloat16((unsigned short)0);
    return;
  }
  if (ex != 0) {                             // zero and FP64 subnormals give zeros
    const uint64_t M = (u & ((1ull << 52) - 1)) | (1ull << 52);   // |x| = M 2^e0
    const int e0 = ex - 1075;
    uint32_t sg = (uint32_t)(u >> 63);
    int sh;
    uint32_t q = round8(M, sh);
    h = bf16_bits(sg, q, e0 + sh);
    int64_t r = (int64_t)M - ((int64_t)q << sh);
    if (r != 0) {
      if (r < 0) { sg ^= 1u; r = -r; }
      q = round8((uint64_t)r, sh);
      m = bf16_bits(sg, q, e0 + sh);
      r -= (int64_t)q << sh;
      if (r != 0) {
        if (r < 0) { sg ^= 1u; r = -r; }
        q = round8((uint64_t)r, sh);
        l = bf16_bits(sg, q, e0 + sh);
      }
    }
  }
  lv[0] = __ushort_as_bfloat16(h);
  lv[1] = __ushort_as_bfloat16(m);
  lv[2] = __ushort_as_bfloat16(l);
}

// float of an integer v < 2^23, exactly
__device__ __forceinline__ float small_uint_float(uint32_t v) { return __uint_as_float(0x4B000000u | v) - 8388608.0f; }

// bf16 bits of the nearest (ties to even) 8-bit value to a * scale, for an
// integer 0 < a < 2^46 and a power of two scale with a * scale in the normal
// float range.  a is cut at 24 significant bits with the last one set when
// anything below is nonzero (rounding to odd, Boldo & Melquiond, IEEE Trans.
// Comput. 57 (2008)), so that the float-to-bf16 rounding of that float equals
// the rounding of a itself: a = X + Y with X = (a >> 23) 2^23 and Y < 2^23,
// both exact floats; s = X + Y rounded toward zero is a cut at 24 bits, and
// s - X is exact (Sterbenz), so s - X != Y tells whether the cut lost bits.
__device__ __forceinline__ uint32_t rne8_bits(uint64_t a, float scale) {
  const float X = small_uint_float((uint32_t)(a >> 23)) * 8388608.0f;
  const float Y = small_uint_float((uint32_t)a & 0x7FFFFFu);
  const float sr = __fadd_rz(X, Y);
  const uint32_t odd = __fsub_rn(sr, X) != Y ? 1u : 0u;
  const float f = __fmul_rn(__uint_as_float(__float_as_uint(sr) | odd), scale);
  return (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(f));
}

// integer value of the positive bf16 piece pb in units of 2^e0
__device__ __forceinline__ uint64_t piece_units(uint32_t pb, int e0) {
  const uint64_t m8 = 0x80u | (pb & 0x7Fu);
  const int sh = (int)((pb >> 7) & 0xFFu) - 134 - e0;
  return sh >= 0 ? m8 << sh : m8 >> (-sh);
}

// The same three pieces as split3_int, computed with single-precision
// arithmetic where every piece is a normal float (2^-74 <= |x| < 2^127, so
// all pieces, multiples of the FP64 ulp of x, are at least 2^-126): the
// remainders stay exact 64-bit integers in units of that ulp, and each
// rounding to 8 bits goes through rne8_bits; other x take split3_int (not
// inlined, so the common path carries none of its instructions).
__device__ __forceinline__ void split3(double x, __nv_bfloat16 (&lv)[3]) {
  const uint64_t u = (uint64_t)__double_as_longlong(x);
  const int ex = (int)((u >> 52) & 0x7FF);
  if (ex < 949 || ex > 1149) {
    split3_int(x, lv);
    return;
  }
  const uint32_t sg = (uint32_t)(u >> 63);
  const int e0 = ex - 1075;                                       // |x| = M 2^e0
  const uint64_t M = (u & ((1ull << 52) - 1)) | (1ull << 52);
  // hi: the top 24 bits of M rounded to odd, as a float of the scale of x
  const uint32_t A = (uint32_t)(M >> 29) | ((M & ((1ull << 29) - 1)) != 0 ? 1u : 0u);
  const uint32_t hb =
      (uint32_t)__bfloat16_as_ushort(__float2bfloat16_rn(__uint_as_float(((uint32_t)(ex - 896) << 23) | (A & 0x7FFFFFu))));
  const int64_t r1 = (int64_t)M - (int64_t)piece_units(hb, e0);
  uint32_t m = 0, l = 0;
  if (r1 != 0) {
    const float scale = __uint_as_float((uint32_t)(e0 + 127) << 23);   // 2^e0
    const uint32_t sg1 = sg ^ (r1 < 0 ? 1u : 0u);
    const uint64_t a1 = (uint64_t)(r1 < 0 ? -r1 : r1);
    const uint32_t mb = rne8_bits(a1, scale);
    m = (sg1 << 15) | mb;
    const int64_t r2 = (int64_t)a1 - (int64_t)piece_units(mb, e0);
    if (r2 != 0) {
      const uint32_t sg2 = sg1 ^ (r2 < 0 ? 1u : 0u);
      l = (sg2 << 15) | rne8_bits((uint64_t)(r2 < 0 ? -r2 : r2), scale);
    }
  }
  lv[0] = __ushort_as_bfloat16((unsigned short)((sg << 15) | hb));
  lv[1] = __ushort_as_bfloat16((unsigned short)m);
  lv[2] = __ushort_as_bfloat16((unsigned short)l);
}

// piece `lev` (0 hi, 1 mid, 2 lo) without a dynamically indexed local array
__device__ __forceinline__ __nv_bfloat16 piece(const __nv_bfloat16 (&lv)[3], int lev) {
  return lev == 0 ? lv[0] : (lev == 1 ? lv[1] : lv[2]);
}

// Persistent: CTA b processes units b, b + gridDim.x, ...; unit u is K slice
// u / tiles of output tile u % tiles (grouped_tile).  Two TMEM accumulators, so
// the loads and MMAs of a unit run while the epilogue warps store the one
// before: with one CTA per unit the store stage (up to 60 us a tile while it
// issued FP64 instructions, even predicated off) added to every tile.  One
// W-build launch at (H2O)8 (2888 x 23104, K = 672) 1.05 -> 0.28 ms, a ring
// product (4864^3) 0.72 -> 0.43 ms.
template <int BN>
__global__ void __launch_bounds__(TC_THREADS, 1)
    gemm_bf16_tc_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, int a_row0,
                        int b_row0, int num_k, int k_chunk, uint32_t tm, uint32_t tn, uint32_t units,
                        const __grid_constant__ EpiMap ep, int* err) {
  using Cfg = TcCfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[Cfg::STAGES];
  __shared__ __align__(8) uint64_t empty_bar[Cfg::STAGES];
  __shared__ __align__(8) uint64_t accf_bar[2];   // accumulator b holds a finished unit
  __shared__ __align__(8) uint64_t acce_bar[2];   // accumulator b has been read out
  __shared__ __align__(8) uint64_t done_bar;      // every issued MMA has completed
  __shared__ uint32_t tmem_holder;
  __shared__ int abort_flag;
  __shared__ float epi_tile[4][32][33];   // per epilogue warp: 32 x 32 transpose

  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + Cfg::STAGES * Cfg::A_BYTES;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t tiles = tm * tn;

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::STAGES; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&accf_bar[b]), 1);
      mbar_init(smem_u32(&acce_bar[b]), 4);   // one arrival per epilogue warp
    }
    mbar_init(smem_u32(&done_bar), 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_holder)),
                 "r"(2 * BN)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_holder;

  if (warp == 0) {
    if (elect_one()) {
      // ---------------- TMA producer (none at all under the no_loads test hook:
      // nothing is then in flight, and the MMA thread's bounded wait gives up)
      int it = 0, s = 0;
      uint32_t ph = 0;
      bool stop = ep.no_loads != 0;
      for (uint32_t u = blockIdx.x; u < units && !stop; u += gridDim.x) {
        uint32_t mt, nt;
        grouped_tile(u % tiles, tm, tn, mt, nt);
        const int kb = (int)(u / tiles) * k_chunk, ke = min(num_k, kb + k_chunk);
        const int am = a_row0 + (int)mt * BM, bn = b_row0 + (int)nt * BN;
        for (int k = kb; k < ke; ++k, ++it) {
          if (!mbar_wait(smem_u32(&empty_bar[s]), ph ^ 1)) { atomicExch(&abort_flag, 1); stop = true; break; }
          const uint32_t fb = smem_u32(&full_bar[s]);
          mbar_expect_tx(fb, Cfg::STAGE_BYTES);
          tma_load_2d(smem_u32(sA + s * Cfg::A_BYTES), &tmA, k * BK, am, fb);
          tma_load_2d(smem_u32(sB + s * Cfg::B_BYTES), &tmB, k * BK, bn, fb);
          if (++s == Cfg::STAGES) { s = 0; ph ^= 1; }
        }
        if (*(volatile int*)&abort_flag) break;
      }
      // on an abort, wait (bounded) for the loads still in flight before the
      // shared memory can be released
      if (*(volatile int*)&abort_flag && !ep.no_loads) {
        for (int q = max(0, it - Cfg::STAGES); q < it; ++q)
          (void)mbar_wait(smem_u32(&full_bar[q % Cfg::STAGES]), (q / Cfg::STAGES) & 1);
      }
    }
  } else if (warp == 1) {
    if (elect_one()) {
      // ---------------- MMA issuer: the next stage's barrier is read between
      // the MMAs of a stage, while the tensor pipe has work queued
      constexpr uint32_t idesc = idesc_bf16(BM, BN);
      const uint64_t ad0 = sw128_desc(smem_u32(sA)), bd0 = sw128_desc(smem_u32(sB));
      uint32_t s = 0, ph = 0, lt = 0, peek = 0;
      bool ok = true;
      for (uint32_t u = blockIdx.x; u < units && ok; u += gridDim.x, ++lt) {
        const int kb = (int)(u / tiles) * k_chunk, nkt = min(num_k, kb + k_chunk) - kb;
        const uint32_t b = lt & 1;
        if (!mbar_wait(smem_u32(&acce_bar[b]), ((lt >> 1) & 1) ^ 1)) { atomicExch(&abort_flag, 1); break; }
        const uint32_t dcol = tmem + b * BN;
        for (int x = 0; x < nkt; ++x) {
          if (!peek && !mbar_wait(smem_u32(&full_bar[s]), ph)) { atomicExch(&abort_flag, 1); ok = false; break; }
          asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
          const uint64_t ad = ad0 + (uint64_t)(s * (Cfg::A_BYTES >> 4));
          const uint64_t bd = bd0 + (uint64_t)(s * (Cfg::B_BYTES >> 4));
          uint32_t s2 = s + 1, ph2 = ph;
          if (s2 == Cfg::STAGES) { s2 = 0; ph2 ^= 1; }
          mma_bf16(dcol, ad, bd, idesc, x > 0 ? 1u : 0u);
          peek = mbar_test(smem_u32(&full_bar[s2]), ph2);
          mma_bf16(dcol, ad + 2, bd + 2, idesc, 1u);
          mma_bf16(dcol, ad + 4, bd + 4, idesc, 1u);
          mma_bf16(dcol, ad + 6, bd + 6, idesc, 1u);
          tc_commit(smem_u32(&empty_bar[s]));
          s = s2;
          ph = ph2;
        }
        if (!ok) break;
        tc_commit(smem_u32(&accf_bar[b]));
      }
      // TMEM is freed only after every issued MMA has completed (also on an abort)
      tc_commit(smem_u32(&done_bar));
      if (!mbar_wait(smem_u32(&done_bar), 0)) atomicExch(&abort_flag, 1);
    }
  } else {
    // ---------------- epilogue: TMEM -> transposed 32 x 32 blocks -> strided global stores
    const int q = warp & 3;              // TMEM lane quadrant this warp may access
    float (*tile)[33] = epi_tile[q];
    const float alpha = (float)ep.alpha;
    // 0: store; 1: reduce into C (no load; beta = 1 or several K slices); 2: add to beta C
    const int mode = ep.atomic || ep.beta == 1.0 ? 1 : (ep.beta == 0.0 ? 0 : 2);
    uint32_t lt = 0;
    for (uint32_t u = blockIdx.x; u < units; u += gridDim.x, ++lt) {
      uint32_t mt, nt;
      grouped_tile(u % tiles, tm, tn, mt, nt);
      const uint32_t b = lt & 1;
      bool ok = mbar_wait(smem_u32(&accf_bar[b]), (lt >> 1) & 1);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok || __any_sync(0xffffffffu, *(volatile int*)&abort_flag != 0)) { atomicExch(&abort_flag, 1); break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int64_t m0 = (int64_t)mt * BM + q * 32, n0 = (int64_t)nt * BN;
      const int rows = (int)min((int64_t)32, ep.M - m0);
      // this lane's row offset; rows are broadcast to the warp below
      const int64_t crow = lane < rows ? epi_row_off(ep, (uint32_t)(m0 + lane)) : 0;
#pragma unroll 1
      for (int c0 = 0; c0 < BN; c0 += 32) {
        if (n0 + c0 >= ep.N) break;
        uint32_t r[32];
        tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + b * BN + (uint32_t)c0, r);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        // transpose the warp's 32 x 32 block through shared memory so each
        // store instruction writes 32 consecutive columns of one row
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 32; ++j) tile[lane][j] = __uint_as_float(r[j]);
        __syncwarp();
        const int64_t n = n0 + c0 + lane;
        const bool nok = n < ep.N;
        double* dst = static_cast<double*>(ep.C) + (nok ? epi_col_off(ep, (uint32_t)n) : 0);
        // The FP32 product becomes FP64 by integer arithmetic: an FP64
        // instruction takes its pipe for 16 clk per warp.
        if (mode == 0) {
#pragma unroll 8
          for (int jr = 0; jr < 32; ++jr) {
            const int64_t roff = __shfl_sync(0xffffffffu, crow, jr);
            if (jr < rows && nok) dst[roff] = f32_to_f64_scaled(alpha * tile[jr][lane], 0, false);
          }
        } else if (mode == 1) {
#pragma unroll 8
          for (int jr = 0; jr < 32; ++jr) {
            const int64_t roff = __shfl_sync(0xffffffffu, crow, jr);
            if (jr < rows && nok) atomicAdd(dst + roff, f32_to_f64_scaled(alpha * tile[jr][lane], 0, false));
          }
        } else {
#pragma unroll 1
          for (int j0 = 0; j0 < 32; j0 += 8) {
            double prev[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const int64_t roff = __shfl_sync(0xffffffffu, crow, j0 + j);
              prev[j] = j0 + j < rows && nok ? dst[roff] : 0.0;
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              const int64_t roff = __shfl_sync(0xffffffffu, crow, j0 + j);
              if (j0 + j < rows && nok)
                dst[roff] = f32_to_f64_scaled(alpha * tile[j0 + j][lane], 0, false) + ep.beta * prev[j];
            }
          }
        }
      }
      // the accumulator is free for the unit after next
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&acce_bar[b]));
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * BN) : "memory");
  }
  if (threadIdx.x == 0 && abort_flag) atomicExch(err, 1);
}

// ---------------------------------------------------------------- packing

// Scale modes of the split packing: the source times 1, times -1 (a sign flip
// of the bit pattern) or times a general factor (one FP64 multiply).
enum { PK_ONE = 0, PK_NEG = 1, PK_ANY = 2 };
template <int SM>
__device__ __forceinline__ double pk_scaled(double v, double scale) {
  if (SM == PK_ONE) return v;
  if (SM == PK_NEG) return __longlong_as_double(__double_as_longlong(v) ^ (long long)0x8000000000000000ull);
  return v * scale;
}

// dst[r][k'] (row pitch Kp) from src: piece p of k' = p*K + k holds hi, mid or
// lo of src(r, k) per `code`; columns >= P*K are zero.  Row walk (k the
// faster source index): 2^lg threads per row, each splitting 4 consecutive k
// once and writing all P pieces, or zeroing 4 of the pad columns.
template <int SM>
__global__ void __launch_bounds__(256) pack_rows_kernel(const double* __restrict__ src, PackSpec ps,
                                                        __nv_bfloat16* __restrict__ dst, PackWalk pw) {
  const int tpr = 1 << pw.lg, lane = threadIdx.x & (tpr - 1), rpb = 256 >> pw.lg;
  const int64_t kq = (ps.K + 3) >> 2, pk = ps.P * ps.K;
  const int64_t ng = kq + ((ps.Kp - pk + 3) >> 2);
  const bool k1 = pack_k_single(ps);
  const bool vec = (ps.K & 3) == 0 && (ps.Kp & 3) == 0 && (reinterpret_cast<uintptr_t>(dst) & 7) == 0;
  const int64_t units = ps.R * pw.nseg;
  for (int64_t u = (int64_t)blockIdx.x * rpb + (threadIdx.x >> pw.lg); u < units; u += (int64_t)gridDim.x * rpb) {
    const int64_t r = pw.nseg == 1 ? u : u / pw.nseg;
    const int64_t g0 = (u - r * pw.nseg) * pw.gseg, g1 = min(ng, g0 + pw.gseg);
    const int64_t ro = pack_row_off(ps, r);
    __nv_bfloat16* drow = dst + r * ps.Kp;
    for (int64_t g = g0 + lane; g < g1; g += tpr) {
      if (g < kq) {
        const int64_t k0 = g << 2;
        const int cnt = (int)min((int64_t)4, ps.K - k0);
        double xv[4];
        pack_load4(src, ps, k1, ro, k0, cnt, xv);
        __nv_bfloat16 lv[4][3];
#pragma unroll
        for (int q = 0; q < 4; ++q) split3(pk_scaled<SM>(xv[q], ps.scale), lv[q]);
        for (int p = 0; p < ps.P; ++p) {
          const int lev = (ps.code >> (2 * p)) & 3;
          __nv_bfloat16* d = drow + p * ps.K + k0;
          if (vec && cnt == 4) {
            __nv_bfloat162 v0 = __halves2bfloat162(piece(lv[0], lev), piece(lv[1], lev));
            __nv_bfloat162 v1 = __halves2bfloat162(piece(lv[2], lev), piece(lv[3], lev));
            uint2 u;
            u.x = *reinterpret_cast<uint32_t*>(&v0);
            u.y = *reinterpret_cast<uint32_t*>(&v1);
            *reinterpret_cast<uint2*>(d) = u;
          } else {
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (q < cnt) d[q] = piece(lv[q], lev);
          }
        }
      } else {
        const int64_t c0 = pk + ((g - kq) << 2);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (c0 + q < ps.Kp) drow[c0 + q] = __ushort_as_bfloat16((unsigned short)0);
      }
    }
  }
}

// Transposing walk through 32 x 32 tiles, for sources whose row index is the
// faster one in memory: the tile's row and column source offsets are
// computed once into shared memory, reads coalesce along rows, and each
// thread splits two consecutive k of one row and writes them as one 4-byte
// store per piece.
template <int SM>
__global__ void __launch_bounds__(256) pack_tiles_kernel(const double* __restrict__ src, PackSpec ps,
                                                         __nv_bfloat16* __restrict__ dst) {
  __shared__ double tile[32][33];
  __shared__ int64_t roff[32], coff[32];
  const int64_t ntr = (ps.R + 31) / 32, ntk = (ps.K + 31) / 32;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int kp = threadIdx.x & 15, rw = threadIdx.x >> 4;   // write phase: k pair, row
  const bool pair = (ps.K & 1) == 0 && (ps.Kp & 1) == 0 && (reinterpret_cast<uintptr_t>(dst) & 3) == 0;
  for (int64_t tb = blockIdx.x; tb < ntr * ntk; tb += gridDim.x) {
    const int64_t r0 = (tb / ntk) * 32, k0 = (tb % ntk) * 32;
    __syncthreads();   // the previous tile is consumed
    if (ty == 0) roff[tx] = r0 + tx < ps.R ? pack_row_off(ps, r0 + tx) : 0;
    else if (ty == 1) coff[tx] = k0 + tx < ps.K ? pack_col_off(ps, k0 + tx) : 0;
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int kk = ty + 8 * j;
      tile[kk][tx] =
          (r0 + tx < ps.R && k0 + kk < ps.K) ? pk_scaled<SM>(src[roff[tx] + coff[kk]], ps.scale) : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int rr = rw + 16 * j;
      const int64_t r = r0 + rr, k = k0 + 2 * kp;
      if (r >= ps.R || k >= ps.K) continue;
      const bool two = k + 1 < ps.K;
      __nv_bfloat16 a[3], b[3];
      split3(tile[2 * kp][rr], a);
      split3(two ? tile[2 * kp + 1][rr] : 0.0, b);
      __nv_bfloat16* d = dst + r * ps.Kp + k;
      for (int p = 0; p < ps.P; ++p) {
        const int lev = (ps.code >> (2 * p)) & 3;
        if (two && pair) {
          *reinterpret_cast<__nv_bfloat162*>(d + p * ps.K) = __halves2bfloat162(piece(a, lev), piece(b, lev));
        } else {
          d[p * ps.K] = piece(a, lev);
          if (two) d[p * ps.K + 1] = piece(b, lev);
        }
      }
    }
  }
}

// zero columns [P*K, Kp) of every row
__global__ void pack_pad_kernel(PackSpec ps, __nv_bfloat16* __restrict__ dst) {
  const int64_t w = ps.Kp - ps.P * ps.K;
  const int64_t total = ps.R * w;
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < total; t += (int64_t)gridDim.x * blockDim.x) {
    const int64_t r = t / w, c = t - r * w;
    dst[r * ps.Kp + ps.P * ps.K + c] = __float2bfloat16_rn(0.0f);
  }
}

// C = beta * C over an epilogue map (before split-K atomics): a row per block
// in turn, columns along the threads.
__global__ void __launch_bounds__(256) scale_out_kernel(EpiMap ep, double beta) {
  for (int64_t n = (int64_t)blockIdx.x * 256 + threadIdx.x; n < ep.N; n += (int64_t)gridDim.x * 256) {
    double* dst = static_cast<double*>(ep.C) + epi_col_off(ep, (uint32_t)n);
    for (int64_t m = blockIdx.y; m < ep.M; m += gridDim.y) {
      double* d = dst + epi_row_off(ep, (uint32_t)m);
      *d = beta == 0.0 ? 0.0 : beta * *d;
    }
  }
}

// -------------------------------------------------------- tensor maps
PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
std::once_flag g_encode_once;

void get_encoder() {
  std::call_once(g_encode_once, []() {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  });
  if (!g_encode) fail(FCC_ERR_CUDA, "cuTensorMapEncodeTiled is unavailable");
}

CUtensorMap make_map(const __nv_bfloat16* base, int64_t rows, int64_t Kp, int box_rows) {
  get_encoder();
  if (Kp % BK != 0 || (reinterpret_cast<uintptr_t>(base) & 15) != 0)
    fail(FCC_ERR_BAD_ARG, "packed operand misaligned for TMA");
  CUtensorMap tm;
  std::memset(&tm, 0, sizeof(tm));
  cuuint64_t dims[2] = {(cuuint64_t)Kp, (cuuint64_t)rows};
  cuuint64_t strides[1] = {(cuuint64_t)Kp * 2};
  cuuint32_t box[2] = {(cuuint32_t)BK, (cuuint32_t)box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = g_encode(&tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<__nv_bfloat16*>(base), dims, strides, box,
                        estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                        CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) fail(FCC_ERR_CUDA, "cuTensorMapEncodeTiled failed");
  return tm;
}

template <int BN>
void launch_tc(const __nv_bfloat16* A, int64_t a_rows, int64_t a_row0, const __nv_bfloat16* B, int64_t b_rows,
               int64_t b_row0, int64_t Kp, const EpiMap& ep, int* err, cudaStream_t s) {
  using Cfg = TcCfg<BN>;
  static SmemLimit smem;
  smem.raise(gemm_bf16_tc_kernel<BN>, Cfg::SMEM);
  CUtensorMap ta = make_map(A, a_rows, Kp, BM);
  CUtensorMap tb = make_map(B, b_rows, Kp, BN);
  const int64_t tm = (ep.M + BM - 1) / BM, tn = (ep.N + BN - 1) / BN;
  const int num_k = (int)(Kp / BK);
  // split K across CTAs when the output has too few tiles to fill the GPU
  int splits = 1;
  if (tm * tn < 152 && num_k >= 16)
    splits = (int)std::min<int64_t>((152 + tm * tn - 1) / (tm * tn), num_k / 8);
  splits = std::max(1, std::min(splits, 64));
  const int chunk = (num_k + splits - 1) / splits;
  splits = (num_k + chunk - 1) / chunk;
  EpiMap e2 = ep;
  if (splits > 1) {
    if (ep.beta != 1.0) {   // C = beta * C before the partial sums are added
      const int64_t x = std::min<int64_t>((ep.N + 255) / 256, 152 * 16);
      const int64_t y = std::max<int64_t>(1, std::min<int64_t>(ep.M, 152 * 16 / x));
      scale_out_kernel<<<dim3((unsigned)x, (unsigned)y), 256, 0, s>>>(ep, ep.beta);
      FCC_CHECK_LAUNCH();
    }
    e2.atomic = 1;
  }
  const int64_t units = tm * tn * splits;
  if (units >= (int64_t(1) << 31)) fail(FCC_ERR_BAD_ARG, "tensor-core grid too large");
  const int pidx = prof_begin(s);
  gemm_bf16_tc_kernel<BN><<<(unsigned)std::min<int64_t>(units, 152), TC_THREADS, Cfg::SMEM, s>>>(
      ta, tb, (int)a_row0, (int)b_row0, num_k, chunk, (uint32_t)tm, (uint32_t)tn, (uint32_t)units, e2, err);
  FCC_CHECK_LAUNCH();
  // executed BF16 flops (padded K included)
  prof_end(s, pidx, PROF_TC, ep.work > 0 ? ep.work : 2.0 * (double)ep.M * (double)ep.N * (double)Kp);
}

}  // namespace

int64_t packed_kp(int64_t K, int P) { return ((P * K + BK - 1) / BK) * BK; }

CUtensorMap tma_map_bf16(const __nv_bfloat16* base, int64_t rows, int64_t cols, int box_rows) {
  return make_map(base, rows, cols, box_rows);
}

void pack_split(const double* src, const PackSpec& ps, __nv_bfloat16* dst, cudaStream_t s) {
  if (ps.R <= 0 || ps.K <= 0) return;
  const int pidx = prof_begin(s);
  struct End { cudaStream_t s; int i; double b; ~End() { prof_end(s, i, PROF_PACK, b); } } pend{s, pidx,
      (double)ps.R * (double)ps.K * 8.0 + (double)ps.R * (double)ps.Kp * 2.0};
  if (ps.P < 1 || ps.P > 8 || ps.Kp < ps.P * ps.K) fail(FCC_ERR_BAD_ARG, "bad pack spec");
  if (ps.R >= (int64_t(1) << 31) || ps.K >= (int64_t(1) << 31)) fail(FCC_ERR_BAD_ARG, "pack extent too large");
  const int64_t kfast = std::llabs(ps.kd3 > 1 ? ps.ks3 : (ps.kd2 > 1 ? ps.ks2 : ps.ks1));
  const int64_t rfast = std::llabs(ps.rd3 > 1 ? ps.rs3 : (ps.rd2 > 1 ? ps.rs2 : ps.rs1));
  const int sm = ps.scale == 1.0 ? PK_ONE : (ps.scale == -1.0 ? PK_NEG : PK_ANY);
  if (rfast < kfast && ps.R >= 32) {
    const int64_t tiles = ((ps.R + 31) / 32) * ((ps.K + 31) / 32);
    const unsigned grid = (unsigned)std::min<int64_t>(tiles, 152 * 16);
    if (sm == PK_ONE) pack_tiles_kernel<PK_ONE><<<grid, 256, 0, s>>>(src, ps, dst);
    else if (sm == PK_NEG) pack_tiles_kernel<PK_NEG><<<grid, 256, 0, s>>>(src, ps, dst);
    else pack_tiles_kernel<PK_ANY><<<grid, 256, 0, s>>>(src, ps, dst);
    FCC_CHECK_LAUNCH();
    if (ps.Kp > ps.P * ps.K) {
      const int64_t tot = ps.R * (ps.Kp - ps.P * ps.K);
      pack_pad_kernel<<<(unsigned)std::min<int64_t>((tot + 255) / 256, 152 * 16), 256, 0, s>>>(ps, dst);
      FCC_CHECK_LAUNCH();
    }
  } else {
    const PackWalk pw = pack_walk(ps.R, (ps.K + 3) / 4 + (ps.Kp - ps.P * ps.K + 3) / 4);
    const unsigned grid = pack_walk_grid(pw, ps.R);
    if (sm == PK_ONE) pack_rows_kernel<PK_ONE><<<grid, 256, 0, s>>>(src, ps, dst, pw);
    else if (sm == PK_NEG) pack_rows_kernel<PK_NEG><<<grid, 256, 0, s>>>(src, ps, dst, pw);
    else pack_rows_kernel<PK_ANY><<<grid, 256, 0, s>>>(src, ps, dst, pw);
    FCC_CHECK_LAUNCH();
  }
}

void gemm_bf16x3(const __nv_bfloat16* A, int64_t a_rows, int64_t a_row0, const __nv_bfloat16* B, int64_t b_rows,
                 int64_t b_row0, int64_t Kp, const EpiMap& ep, int* err, cudaStream_t s) {
  if (ep.M <= 0 || ep.N <= 0) return;
  if (Kp <= 0 || Kp % BK || Kp >= (int64_t(1) << 31)) fail(FCC_ERR_BAD_ARG, "bad packed K");
  if (a_rows >= (int64_t(1) << 31) || b_rows >= (int64_t(1) << 31)) fail(FCC_ERR_BAD_ARG, "packed operand too large");
  if (ep.N >= 256) launch_tc<256>(A, a_rows, a_row0, B, b_rows, b_row0, Kp, ep, err, s);
  else launch_tc<128>(A, a_rows, a_row0, B, b_rows, b_row0, Kp, ep, err, s);
}

}  // namespace fcc
