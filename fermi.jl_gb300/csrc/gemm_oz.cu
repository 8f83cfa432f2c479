// Exact-slice BF16 tensor-core contraction (the Ozaki scheme) for GB300.
//
// C = alpha * A.B^T + beta * C for FP64 operands, evaluated from signed digit
// slices of A and B (pack_oz.cu, fcc_tc.cuh).  Every digit is an integer,
// |d| <= 2^bits (the first digit) or 2^(bits-1) (the others), exact in BF16,
// and tcgen05.mma accumulates products of such digits exactly in FP32 while
// |sum| <= 2^24.
//
// Slice pairs of one weight 2^(-bits g) (g = sa + sb, slices counted from 1)
// share an accumulator.  Two neighbouring groups g, g + 1 form a band and run
// together, because their pairs can be ordered so that each step shares one
// operand tile with the step before: the tiles
//   B_g, A_1, B_(g-1), A_2, ..., B_1, A_g
// arrive as one stream and step i multiplies tiles i and i + 1.  A step then
// moves one tile into shared memory instead of two.  What bounds long products
// is shared-memory bandwidth (128 B/clk per SM): the MMAs of a 128 x 128 x 64
// step read 32 KB in 256 clk while the incoming 16 KB are written, 384 clk (two
// thirds of the tensor rate; 512 with two new tiles).  So two CTAs on
// neighbouring SMs share a 256 x 128 tile where its rows allow (cta_group::2):
// each keeps half of every B tile, and reads 24 KB and writes 12 a step, 288
// clk.  Measured at M = N = K = 4864, 21 products of 6-bit digits: 3.03 ms and
// 1596 TFLOP/s executed (3.60 with single CTAs; 6.0 with two new tiles a step
// and roles in threads the compiler could not tell from warps, fcc_tcgen05.cuh
// elect_one); 36 products (9 groups) 5.05 ms, 1642.
//
// When an accumulator could reach 2^24 (a chunk: 2-16 k-blocks at the FP64 level,
// 25-64 of 6-bit digits) the eight epilogue warps add it, times its weight (a
// power of two), into a running double-FP32 sum (hi + lo, 2^-47 over K = 11628)
// held in registers, 64 columns per thread.  Registers instead of TMEM leave
// TMEM for two sets of two chunk accumulators, so the MMA thread fills one set
// while the other is drained, and a drain reads 4 bytes per element from TMEM
// instead of moving 20.  The additions run two per instruction (fma.rn.f32x2).
// The FP64 level's 8-bit digits close a chunk every 2-16 k-blocks and its drains
// show: 36 products of 4864^3 in 5.62 ms, 1473 TFLOP/s.
//
// Batches: products of the same shape whose rows lie apart by fixed steps in A,
// B and C run in one launch (EpiMap batch, ba, bb, bc), which fills the chip
// where one product has a few dozen tiles.
//
// `cut`: the first band (groups 2 and 3) and the rest get separate running
// sums ("parts"), each converted and added to C in FP64.  At the FP64 level
// with one chunk in the first band (K <= 1024) that band runs last and needs no
// sum of its own: its two accumulators are added to the others' sums in the store
// stage (`merged`), one conversion and one pass over C instead of two.
//
// Short products (K a few hundred, the (T) ones) are bound by that store stage:
// a 128 x 128 tile converts 64 elements a thread.  Integer conversion of hi,
// lo and tail, a short form where no exponent can leave the FP64 range, sums
// handed over through shared memory so that a warp stores whole rows, and
// red.add where C is added to (the read would wait in the warp, the addition
// is the L2's): 5776 x 1216 x 92 at the FP64 level 133 us.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>

#include "fcc_tc.cuh"
#include "fcc_tcgen05.cuh"

namespace fcc {

namespace {

using namespace tc5;

constexpr int OZ_BM = 128, OZ_BN = 128, OZ_BK = 64;
constexpr int OZ_SLOTS = 10;                     // tile ring
constexpr int OZ_TILE_BYTES = 128 * OZ_BK * 2;   // one operand tile, A or B
constexpr int OZ_EPI_WARPS = 8;
constexpr int OZ_THREADS = 128 + 32 * OZ_EPI_WARPS;   // warp 0 TMA of A, 1 MMA, 2 TMA of B, 3 idle, 4-11 epilogue
constexpr int OZ_XP_LD = 17;                     // transpose tile of an epilogue warp: 32 rows x 16 columns,
constexpr int OZ_XP_PLANE = 32 * OZ_XP_LD;       // three words per element
constexpr int OZ_XP_BYTES = OZ_EPI_WARPS * 3 * OZ_XP_PLANE * 4;
constexpr int OZ_SMEM = OZ_SLOTS * OZ_TILE_BYTES + OZ_XP_BYTES + 1024;
constexpr int OZ_MAXBANDS = 5, OZ_MAXJOBS = 152;

// One band: groups g (and g + 1 when ngrp = 2), ntile operand tiles per
// k-block, alternating B and A (bfirst) or A and B; the A tiles are slices 0,
// 1, ..., the B tiles btop, btop - 1, ...; ck k-blocks per chunk.  Step j
// multiplies tiles j and j + 1, and successive steps alternate between the
// two groups.
struct OzBand {
  int16_t ntile, ck, g, ngrp, bfirst, btop;
};
// One piece of an output tile's work: bands [b0, b1) over k-blocks [k0, k1).
struct OzJob {
  int16_t b0, b1;
  int32_t k0, k1;
};
struct OzParams {
  OzBand band[OZ_MAXBANDS];
  OzJob job[OZ_MAXJOBS];
  uint32_t njobs;
  int cut;                     // cut: bands of the first part (0: one part)
  int bits, guard;             // digit width, guard bits of the scales
  int merged;                  // the last band is added to the others' sums in the store stage
  int kper, kpad;              // k-blocks per L2 block; padded columns per slice
  uint32_t tm, tn, units;
  double* part;                // partial results [product][job][M][N] (nullptr: C itself)
};

// The bands of groups 2..G over S slices (G <= S + 2): {.., (G-3, G-2),
// (G-1, G)}, group 2 on its own when their number is odd.
int make_bands(OzLevel lv, OzBand* out) {
  const int S = lv.S, G = lv.G;
  const double first = std::ldexp(1.0, 1 - lv.guard);   // largest first digit over the largest other one
  int n = 0;
  for (int g = 2; g <= G;) {
    OzBand b;
    b.g = (int16_t)g;
    b.ngrp = (int16_t)(((G - 1) % 2 == 1 && g == 2) ? 1 : 2);
    b.bfirst = b.ngrp == 2 && g <= S;        // B_g, A_1, B_(g-1), A_2, ..., B_1, A_g
    b.btop = (int16_t)(b.ngrp == 1 ? 0 : (b.bfirst ? g - 1 : S - 1));
    b.ntile = (int16_t)(2 * (b.btop + 1));
    // units of 64 2^(2 bits - 2) (64 products of two digits after the first)
    // that one k-block adds to a group; the sum may reach 2^24
    double worst = 0;
    for (int q = 0; q < b.ngrp; ++q) {
      double u = 0;
      for (int a = 1; a < g + q; ++a) {
        const int c = g + q - a;
        if (a <= S && c <= S) u += (a == 1 ? first : 1.0) * (c == 1 ? first : 1.0);
      }
      worst = std::max(worst, u);
    }
    b.ck = (int16_t)std::max(1, (int)(std::ldexp(1.0, 20 - 2 * lv.bits) / worst));
    out[n++] = b;
    g += b.ngrp;
  }
  return n;
}

// frexp-style exponent of the row scale from the stored biased exponent
// (2^21 for a row with infinities or NaN)
__device__ __forceinline__ int oz_scale_exp(int be) { return be == 2047 ? (1 << 21) : (be ? be - 1022 : 0); }

__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
  uint64_t d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
__device__ __forceinline__ uint64_t add2(uint64_t a, uint64_t b) {
  uint64_t d;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
__device__ __forceinline__ uint64_t pack2(uint32_t x, uint32_t y) {
  uint64_t d;
  asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "r"(x), "r"(y));
  return d;
}
__device__ __forceinline__ void unpack2(uint64_t d, uint32_t& x, uint32_t& y) {
  asm("mov.b64 {%0, %1}, %2;" : "=r"(x), "=r"(y) : "l"(d));
}

// two independent (hi + lo) += v * w: TwoSum of hi and v * w (the product by a
// power of two is exact inside the fma), the error into lo.  lo grows by half a
// last place of hi an addition and ff_norm2 takes it back every second drain: 8.5
// packed operations an addition instead of ten with every one, and the FP32 pipe
// is what a drain takes (two clk per packed instruction).  Without it lo, and the
// last place it is rounded to, grew over all of a product: at K = 11628 the sums
// carried 2^-45.8 at nine groups and 2^-44.7 in the FP64 level's lower bands, now
// 2^-47.2 and 2^-47.5 (an FP64 step at (H2O)8 75.1 ms, 75.2 with it).
__device__ __forceinline__ void ff_add2(uint64_t& hi, uint64_t& lo, uint64_t v, uint64_t w, uint64_t m1) {
  const uint64_t s = fma2(v, w, hi);
  const uint64_t nbb = fma2(s, m1, hi);       // -(s - hi)
  const uint64_t t = add2(s, nbb);
  lo = add2(lo, add2(fma2(t, m1, hi), fma2(v, w, nbb)));
  hi = s;
}

__device__ __forceinline__ void ff_norm2(uint64_t& hi, uint64_t& lo, uint64_t m1) {
  const uint64_t h = add2(hi, lo);
  lo = fma2(fma2(hi, m1, h), m1, lo);   // lo - (h - hi)
  hi = h;
}

__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// (hi + lo + tail) * 2^e as one FP64 number by integer arithmetic: lo and tail
// are turned into units of the 53-bit last place of hi (lo at most 2^29, tail a
// few) and added to the bit pattern of hi.  The FP64 pipe (1/64 rate) would take
// three conversions and two additions per element.  |lo| <= ulp(hi) / 2; |hi| is
// 0 or at least 2^-72, the smallest weight.  e >= 2^20 marks a row or column
// with infinities or NaN.
__device__ __forceinline__ double ff_to_f64(float hf, float lf, float tail, int e, uint32_t neg) {
  const uint32_t h = __float_as_uint(hf);
  const int eh = (int)((h >> 23) & 0xFF);
  const uint32_t m = h & 0x7FFFFFu;
  const uint32_t rest = __float_as_uint(__fadd_rn(lf, tail));
  const int down = (m == 0 && (int)(h ^ rest) < 0) ? 1 : 0;   // hi a power of two, the sum in the binade below
  const float scale = __uint_as_float((uint32_t)(306 - eh + down) << 23);   // 1 / last place, 2^(179 - eh)
  int t = __float2int_rn(__fmul_rn(lf, scale)) + __float2int_rn(__fmul_rn(tail, scale));
  if ((int)h < 0) t = -t;
  const int ne = eh + 896 + e;                              // biased FP64 exponent of hi
  const uint32_t sign = (h ^ neg) & 0x80000000u;
  const uint64_t mag = ((uint64_t)(((uint32_t)ne << 20) | (m >> 3)) << 32 | (uint64_t)(m << 29)) + (uint64_t)(int64_t)t;
  uint32_t w1 = (uint32_t)(mag >> 32), w0 = (uint32_t)mag;
  if (eh == 0 || ne <= 0) w1 = w0 = 0;
  if (ne > 2046) { w1 = e >= (1 << 20) ? 0x7FF80000u : 0x7FF00000u; w0 = 0; }
  if (eh == 0 && e >= (1 << 20)) w1 = 0x7FF80000u;
  return __longlong_as_double((long long)((uint64_t)(w1 | sign) << 32 | w0));
}

// The same where no exponent can leave the FP64 range (es = (e + 896) << 20,
// |e| < 810): half the instructions.
__device__ __forceinline__ double ff_to_f64_safe(float hf, float lf, float tail, int es, uint32_t neg) {
  const uint32_t h = __float_as_uint(hf), a = h & 0x7FFFFFFFu, s = h ^ a;
  const float l = __uint_as_float(__float_as_uint(lf) ^ s);      // relative to the sign of hi
  const float x = __uint_as_float(__float_as_uint(tail) ^ s);
  const uint32_t down = ((h & 0x7FFFFFu) == 0u && (int)__float_as_uint(__fadd_rn(l, x)) < 0) ? 1u << 23 : 0u;
  const float scale = __uint_as_float((306u << 23) - (a & 0x7F800000u) + down);
  const int t = __float2int_rn(__fmul_rn(l, scale)) + __float2int_rn(__fmul_rn(x, scale));
  const uint64_t mag = ((uint64_t)((a >> 3) + (uint32_t)es) << 32 | (uint64_t)(h << 29)) + (uint64_t)(int64_t)t;
  const uint32_t w1 = (uint32_t)(mag >> 32) | ((s ^ neg) & 0x80000000u);
  return __hiloint2double(a ? (int)w1 : 0, a ? (int)(uint32_t)mag : 0);
}

// Persistent: worker b processes units b, b + workers, ...; unit u is output
// tile u % tiles of job (u / tiles) % njobs of product u / (tiles njobs).  The
// tile ring and the accumulator sets run on across units, so the loads and MMAs
// of a unit's first chunks overlap the previous unit's stores.  Every role walks
// the same sequence: parts, L2 blocks of kper k-blocks (units running at the
// same time share one, so the slices they stream stay in L2), bands, chunks of
// ck k-blocks.  PAIR: a cluster of two CTAs is one worker; each loads its rows
// of A and half of B, the loads of both count on the first CTA's barriers, which
// issues the MMAs for both; barriers that free tiles or hand over accumulators
// are signalled in both.
// F64: the FP64 level, whose store stage may take the last band's accumulators
// along (P.merged).
template <bool F64, bool PAIR>
__global__ void __launch_bounds__(OZ_THREADS, 1)
    gemm_oz_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                   const __grid_constant__ OzParams P, const int* __restrict__ exA, const int* __restrict__ exB,
                   const __grid_constant__ EpiMap ep, int* err) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[OZ_SLOTS];
  __shared__ __align__(8) uint64_t empty_bar[OZ_SLOTS];
  __shared__ __align__(8) uint64_t accf_bar[2];   // accumulator set b is complete
  __shared__ __align__(8) uint64_t acce_bar[2];   // accumulator set b is drained
  __shared__ __align__(8) uint64_t done_bar;      // every issued MMA has completed
  __shared__ uint32_t tmem_holder;
  __shared__ int abort_flag;

  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  float* xp = reinterpret_cast<float*>(smem + OZ_SLOTS * OZ_TILE_BYTES);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t tiles = P.tm * P.tn;
  // PAIR: two CTAs share a 256 x 128 tile; this one has 128 of its rows and
  // loads half of each B tile; the first issues the MMAs
  const uint32_t rank = PAIR ? cluster_rank() : 0u;
  const uint32_t wid = PAIR ? blockIdx.x >> 1 : blockIdx.x, nwork = PAIR ? gridDim.x >> 1 : gridDim.x;
  constexpr int UM = PAIR ? 2 * OZ_BM : OZ_BM;

  if (threadIdx.x == 0) {
    for (int s = 0; s < OZ_SLOTS; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&accf_bar[b]), 1);
      mbar_init(smem_u32(&acce_bar[b]), PAIR ? 2 * OZ_EPI_WARPS : OZ_EPI_WARPS);
    }
    mbar_init(smem_u32(&done_bar), 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    if (PAIR) {
      asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_holder)),
                   "r"(512)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    } else {
      asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_holder)),
                   "r"(512)
                   : "memory");
      asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (PAIR) cluster_sync();     // both CTAs' barriers are there before either is signalled
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_holder;

  if (warp < 4) {
    // 384 threads x 168 registers at launch; the epilogue warps take 224
    // (128 x 48 + 256 x 224 = 63488 <= 64512)
    asm volatile("setmaxnreg.dec.sync.aligned.u32 48;");
    if (warp == 0 || warp == 2) {
     if (elect_one()) {
      // ---------------- TMA producers: warp 0 streams the A tiles, warp 2 the
      // B tiles.  One load costs its thread ~300 clk of issue, more than the
      // 256 clk of a step's MMAs, so one thread could not feed both.
      const bool isB = warp == 2;
      const CUtensorMap* tm = isB ? &tmB : &tmA;
      int s = 0;                   // ring slot of the chain's first tile, and its phase
      uint32_t ph = 0;
      uint32_t issued = 0, parity = 0;   // slots loaded by this thread, phase parity of the last load of each
      bool stop = ep.no_loads != 0;
      for (uint32_t u = wid; u < P.units && !stop; u += nwork) {
        uint32_t mt, nt;
        grouped_tile(u % tiles, P.tm, P.tn, mt, nt);
        const uint32_t q = u / tiles;
        const OzJob jb = P.job[q % P.njobs];
        const int64_t bq = q / P.njobs;
        const int row = (int)(isB ? bq * ep.bb + nt * OZ_BN + rank * (OZ_BN / 2) : bq * ep.ba + mt * UM + rank * OZ_BM);
        int bb = jb.b0;
        while (bb < jb.b1 && !stop) {
          const int be = (bb < P.cut) ? min(P.cut, (int)jb.b1) : (int)jb.b1;   // this part's bands
          for (int zb = jb.k0; zb < jb.k1 && !stop; zb += P.kper) {
            const int ze = min(zb + P.kper, jb.k1);
            for (int b = bb; b < be && !stop; ++b) {
              const OzBand bd = P.band[b];
              const int off = (bd.bfirst != 0) == isB ? 0 : 1, np = bd.ntile >> 1;
              const int x0 = (isB ? (int)bd.btop : 0) * P.kpad, dx = isB ? -P.kpad : P.kpad;
              for (int kb = zb; kb < ze; ++kb) {
                int cs = s + off;
                uint32_t cp = ph;
                if (cs >= OZ_SLOTS) { cs -= OZ_SLOTS; cp ^= 1; }
                int x = x0 + kb * OZ_BK;
                for (int i = 0; i < np; ++i, x += dx) {
                  if (!mbar_wait(smem_u32(&empty_bar[cs]), cp ^ 1)) { atomicExch(&abort_flag, 1); stop = true; break; }
                  const uint32_t fb = smem_u32(&full_bar[cs]);
                  if (PAIR) {
                    // both CTAs' halves count on the first one's barrier
                    if (rank == 0) mbar_expect_tx(fb, isB ? OZ_TILE_BYTES : 2 * OZ_TILE_BYTES);
                    tma_load_2d_pair(smem_u32(smem + cs * OZ_TILE_BYTES), tm, x, row, cluster_addr(fb, 0));
                  } else {
                    mbar_expect_tx(fb, OZ_TILE_BYTES);
                    tma_load_2d(smem_u32(smem + cs * OZ_TILE_BYTES), tm, x, row, fb);
                  }
                  issued |= 1u << cs;
                  parity = (parity & ~(1u << cs)) | (cp << cs);
                  cs += 2;
                  if (cs >= OZ_SLOTS) { cs -= OZ_SLOTS; cp ^= 1; }
                }
                if (stop || *(volatile int*)&abort_flag) { stop = true; break; }
                s += bd.ntile;
                while (s >= OZ_SLOTS) { s -= OZ_SLOTS; ph ^= 1; }
              }
            }
          }
          bb = be;
        }
      }
      // on an abort, wait (bounded) for the loads still in flight before the
      // shared memory can be released
      // (a pair's first CTA waits for the loads of both)
      if (*(volatile int*)&abort_flag && rank == 0) {
        for (int c = 0; c < OZ_SLOTS; ++c)
          if ((issued >> c) & 1) (void)mbar_wait(smem_u32(&full_bar[c]), (parity >> c) & 1);
      }
     }
    } else if (warp == 1 && rank == 0) {
     if (elect_one()) {
      // ---------------- MMA issuer.  An MMA's issue waits until the one before
      // it has started, so whatever the thread does between two steps leaves
      // the tensor pipe idle unless it runs behind an issued MMA: the next
      // tile's barrier is read between the MMAs of a step, and a step's
      // descriptors need one addition each.
      constexpr uint32_t idesc = idesc_bf16(UM, OZ_BN);
      auto mma = [&](uint32_t d, uint64_t ad, uint64_t bd, uint32_t acc) {
        if (PAIR) mma_bf16_pair(d, ad, bd, idesc, acc);
        else mma_bf16(d, ad, bd, idesc, acc);
      };
      auto commit = [&](uint32_t bar) {
        if (PAIR) tc_commit_pair(bar);
        else tc_commit(bar);
      };
      const uint64_t desc0 = sw128_desc(smem_u32(smem));
      const uint32_t full0 = smem_u32(&full_bar[0]), empty0 = smem_u32(&empty_bar[0]);
      uint32_t s = 0, ph = 0;      // ring slot of the next tile, and its phase
      uint32_t chunk = 0;
      bool ok = true;
      for (uint32_t u = wid; u < P.units && ok; u += nwork) {
        const OzJob jb = P.job[(u / tiles) % P.njobs];
        int bb = jb.b0;
        while (bb < jb.b1 && ok) {
          const int be = (bb < P.cut) ? min(P.cut, (int)jb.b1) : (int)jb.b1;
          for (int zb = jb.k0; zb < jb.k1 && ok; zb += P.kper) {
            const int ze = min(zb + P.kper, jb.k1);
            for (int b = bb; b < be && ok; ++b) {
              const OzBand bd = P.band[b];
              const int nt_ = bd.ntile;
              const uint32_t par0 = (uint32_t)(bd.g + bd.bfirst) & 1u;
              for (int kc = zb; kc < ze && ok; kc += bd.ck, ++chunk) {
                const int set = chunk & 1;
                const int ntot = (min(kc + (int)bd.ck, ze) - kc) * nt_;
                if (!mbar_wait(smem_u32(&acce_bar[set]), ((chunk >> 1) & 1) ^ 1)) {
                  atomicExch(&abort_flag, 1);
                  ok = false;
                  break;
                }
                const uint32_t dset = tmem + (uint32_t)(set * 2 * OZ_BN);
                uint32_t started = 0;        // bit q: the accumulator of parity q holds a sum
                uint32_t pslot = 0, par = par0, peek = 0;
                uint32_t curB = (uint32_t)bd.bfirst;   // the tile at s is a B tile
                int t = 0;
                for (int x = 0; x < ntot; ++x) {
                  if (!peek && !mbar_wait(full0 + 8 * s, ph)) { atomicExch(&abort_flag, 1); ok = false; break; }
                  uint32_t s2 = s + 1, ph2 = ph;
                  if (s2 == OZ_SLOTS) { s2 = 0; ph2 ^= 1; }
                  if (t > 0) {
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t ad = desc0 + (uint64_t)((curB ? pslot : s) * (OZ_TILE_BYTES >> 4));
                    const uint64_t bdsc = desc0 + (uint64_t)((curB ? s : pslot) * (OZ_TILE_BYTES >> 4));
                    const uint32_t dcol = dset + par * OZ_BN;
                    const uint32_t acc = (started >> par) & 1u;
                    mma(dcol, ad, bdsc, acc);
                    peek = mbar_test(full0 + 8 * s2, ph2);
                    mma(dcol, ad + 2, bdsc + 2, 1u);
                    started |= 1u << par;
                    par ^= 1u;
                    mma(dcol, ad + 4, bdsc + 4, 1u);
                    mma(dcol, ad + 6, bdsc + 6, 1u);
                    commit(empty0 + 8 * pslot);                     // its last use
                  } else {
                    peek = 0;
                  }
                  pslot = s;
                  s = s2;
                  ph = ph2;
                  curB ^= 1u;
                  if (++t == nt_) {
                    commit(empty0 + 8 * pslot);
                    t = 0;
                    par = par0;
                  }
                }
                if (!ok) break;
                commit(smem_u32(&accf_bar[set]));
              }
            }
          }
          bb = be;
        }
      }
      commit(smem_u32(&done_bar));
     }
    }
  } else {
    // ---------------- epilogue warps: rows q*32 .. q*32+31, columns half*64 .. half*64+63 of each tile
    asm volatile("setmaxnreg.inc.sync.aligned.u32 224;");
    const int q = warp & 3, half = (warp - 4) >> 2;
    const uint32_t lanebase = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(half * 64);
    float* tile = xp + (warp - 4) * 3 * OZ_XP_PLANE;
    const uint64_t m1 = pack2(0xBF800000u, 0xBF800000u);   // -1, -1
    bool ok = true;
    uint32_t chunk = 0;
    auto drained = [&](int set) {   // an accumulator set is free for the MMA thread
      const uint32_t bar = smem_u32(&acce_bar[set]);
      if (PAIR) mbar_arrive_cluster(cluster_addr(bar, 0));
      else mbar_arrive(bar);
    };
    // alpha = +-2^ka folds into the exponent arithmetic; otherwise one FP64 multiply
    const double alpha = P.part ? 1.0 : ep.alpha;
    const unsigned long long ab = (unsigned long long)__double_as_longlong(alpha);
    const bool apow2 = (ab & ((1ull << 52) - 1)) == 0 && ((ab >> 52) & 0x7FF) != 0;
    const int ka = (apow2 ? (int)((ab >> 52) & 0x7FF) - 1023 : 0) + 2 * P.guard;
    const uint32_t aneg = apow2 && (ab >> 63) ? 0x80000000u : 0u;
    const double alpha_left = apow2 ? 1.0 : alpha;
    for (uint32_t u = wid; u < P.units && ok; u += nwork) {
      uint32_t mt, nt;
      grouped_tile(u % tiles, P.tm, P.tn, mt, nt);
      const uint32_t slot = u / tiles;           // (product, job)
      const OzJob jb = P.job[slot % P.njobs];
      const int64_t bq = slot / P.njobs;
      int bb = jb.b0;
      while (bb < jb.b1 && ok) {
        const int be = (bb < P.cut) ? min(P.cut, (int)jb.b1) : (int)jb.b1;
        // what the store stage needs, read ahead of the sums
        const int64_t m = (int64_t)mt * UM + rank * OZ_BM + q * 32 + lane;
        int64_t crow = 0;
        int erow = 0;
        if (m < ep.M) {
          crow = P.part ? ((int64_t)slot * ep.M + m) * ep.N : epi_row_off(ep, (uint32_t)m) + bq * ep.bc;
          erow = oz_scale_exp(exA[bq * ep.ba + m]) + ka;
        }
        // this lane's share of the column exponents: columns lane and lane + 32
        int ecl[2];
#pragma unroll
        for (int c = 0; c < 2; ++c) {
          const int64_t n = (int64_t)nt * OZ_BN + half * 64 + 32 * c + lane;
          ecl[c] = n < ep.N ? oz_scale_exp(exB[bq * ep.bb + n]) : 0;
        }
        int last = -1, drains = 0;
        uint64_t hi[32], lo[32];
#pragma unroll
        for (int c = 0; c < 32; ++c) hi[c] = lo[c] = 0ull;
        for (int zb = jb.k0; zb < jb.k1 && ok; zb += P.kper) {
          const int ze = min(zb + P.kper, jb.k1);
          for (int b = bb; b < be && ok; ++b) {
            const int ck = P.band[b].ck, g0 = P.band[b].g, ng = P.band[b].ngrp;
            for (int kc = zb; kc < ze; kc += ck, ++chunk) {
              const int set = chunk & 1;
              ok = mbar_wait(smem_u32(&accf_bar[set]), (chunk >> 1) & 1);
              ok = __all_sync(0xffffffffu, ok);
              if (!ok || __any_sync(0xffffffffu, *(volatile int*)&abort_flag != 0)) {
                atomicExch(&abort_flag, 1);
                ok = false;
                break;
              }
              asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
              if (F64 && P.merged && b == jb.b1 - 1) {   // its one chunk is read in the store stage
                last = set;
                continue;
              }
              // weight of the group, 2^(-bits g), exact in FP32; the
              // accumulators hold exact integers of at most 2^24.  16 columns
              // at a time, each read while the ones before are added.
              uint32_t x[2][16];
              tmem_ld16(lanebase + (uint32_t)(set * 2 * OZ_BN + (g0 & 1) * OZ_BN), x[0]);
#pragma unroll 1
              for (int gq = 0; gq < ng; ++gq) {
                const int g = g0 + gq;
                const uint32_t wb = (uint32_t)(127 - P.bits * g) << 23;
                const uint64_t w = pack2(wb, wb);
                const uint32_t col = lanebase + (uint32_t)(set * 2 * OZ_BN + (g & 1) * OZ_BN);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                  tmem_wait(x[c & 1]);
                  if (c < 3) tmem_ld16(col + 16 * (c + 1), x[(c + 1) & 1]);
                  else if (gq + 1 < ng) tmem_ld16(lanebase + (uint32_t)(set * 2 * OZ_BN + ((g + 1) & 1) * OZ_BN), x[0]);
#pragma unroll
                  for (int j = 0; j < 8; ++j)
                    ff_add2(hi[8 * c + j], lo[8 * c + j], pack2(x[c & 1][2 * j], x[c & 1][2 * j + 1]), w, m1);
                }
              }
              asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
              __syncwarp();
              if (lane == 0) drained(set);
              if ((++drains & 1) == 0) {
#pragma unroll
                for (int j = 0; j < 32; ++j) ff_norm2(hi[j], lo[j], m1);
              }
            }
          }
        }
        if (!ok) break;
        // ---- the part's sums, scaled, to the output
        const bool first = bb == jb.b0;
        // 0: store, 1: add to the output, 2: add to beta times the output
        const int bmode = first ? (P.part || ep.beta == 0.0 ? 0 : (ep.beta == 1.0 ? 1 : 2)) : 1;
        double* out = P.part ? P.part : static_cast<double*>(ep.C);
        // rows this lane stores: 2 j + lane / 16
        const int rows = (int)min((int64_t)32, ep.M - ((int64_t)mt * UM + rank * OZ_BM + q * 32));
        // the usual case: factors of a power of two, exponents well inside the FP64 range
        const bool plain = __all_sync(0xffffffffu, apow2 && bmode < 2 && abs(erow) < 400 && abs(ecl[0]) < 400 &&
                                                       abs(ecl[1]) < 400);
        const float w2 = __uint_as_float((uint32_t)(127 - P.bits * 2) << 23);
        const float w3 = __uint_as_float((uint32_t)(127 - P.bits * 3) << 23);
#pragma unroll
        for (int c0 = 0; c0 < 4; ++c0) {       // 16 columns at a time
          const int64_t nb = (int64_t)nt * OZ_BN + half * 64 + 16 * c0;
          if (nb >= ep.N) continue;
          __syncwarp();
#pragma unroll
          for (int c1 = 0; c1 < 2; ++c1) {
            uint32_t a2[8], a3[8];
            if (F64 && last >= 0) {            // groups 2 and 3, one chunk each
              const uint32_t col = lanebase + (uint32_t)(last * 2 * OZ_BN + 16 * c0 + 8 * c1);
              tmem_ld8(col, a2);
              tmem_ld8(col + OZ_BN, a3);
              tmem_wait(a2);
              tmem_wait(a3);
            }
#pragma unroll
            for (int j = 0; j < 8; ++j) {
              uint32_t x[2], y[2];
              unpack2(hi[8 * c0 + 4 * c1 + j / 2], x[0], x[1]);
              unpack2(lo[8 * c0 + 4 * c1 + j / 2], y[0], y[1]);
              // renormalised (|lo| is far below |hi| unless the sums cancelled,
              // where the difference is exact)
              const float h0 = __uint_as_float(x[j & 1]), l0 = __uint_as_float(y[j & 1]);
              float h = __fadd_rn(h0, l0), l = __fsub_rn(l0, __fsub_rn(h, h0));
              float* at = tile + lane * OZ_XP_LD + 8 * c1 + j;
              if (F64 && last >= 0) {
                // both groups are exact; their sum (f, r) and the others' (h, l)
                // become f' + l' + tail
                float f, r, g, d;
                two_sum(__fmul_rn(__uint_as_float(a2[j]), w2), __fmul_rn(__uint_as_float(a3[j]), w3), f, r);
                two_sum(r, h, g, d);
                d = __fadd_rn(d, l);
                two_sum(f, g, h, l);
                // where f and g cancelled (l = 0) the tail can be as large as h
                const bool z = l == 0.0f;
                two_sum(h, z ? d : l, f, r);
                h = f;
                l = r;
                at[2 * OZ_XP_PLANE] = z ? 0.0f : d;
              }
              at[0] = h;
              at[OZ_XP_PLANE] = l;
            }
          }
          __syncwarp();
          // Each lane turns into FP64 what it stores: two rows of 16 columns per
          // instruction, in a loop (unrolled over the registers of the sums, the
          // conversion was 50 KB of code run once per tile, bound by instruction
          // fetch).  Adding to the output is a reduction in L2 (red.add): no
          // load to wait for, and the order is fixed all the same: within a
          // launch one thread owns an element and its reductions reach it in
          // program order.  Other factors go apart, because an FP64 instruction
          // takes the pipe for 16 clk per warp even where it is predicated off.
          const int64_t nl = nb + (lane & 15);
          const bool nok = nl < ep.N;
          double* dst = out + (!nok ? 0 : (P.part ? nl : epi_col_off(ep, (uint32_t)nl)));
          const int ec = __shfl_sync(0xffffffffu, ecl[c0 >> 1], 16 * (c0 & 1) + (lane & 15));
          const float* src = tile + (lane >> 4) * OZ_XP_LD + (lane & 15);
          if (plain) {
            const int esr = (erow + 896) << 20, esc = ec << 20;
#pragma unroll 4
            for (int j = 0; j < 16; ++j) {
              const int r = 2 * j + (lane >> 4);
              const int64_t off = __shfl_sync(0xffffffffu, crow, r);
              const int es = __shfl_sync(0xffffffffu, esr, r) + esc;
              const float* at = src + 2 * j * OZ_XP_LD;
              const float tail = F64 && last >= 0 ? at[2 * OZ_XP_PLANE] : 0.0f;
              const double v = F64 ? ff_to_f64_safe(at[0], at[OZ_XP_PLANE], tail, es, aneg)
                                   : ff_to_f64_safe(at[0], at[OZ_XP_PLANE], 0.0f, es, aneg);
              if (!nok || r >= rows) continue;
              if (bmode == 0) dst[off] = v;
              else atomicAdd(dst + off, v);
            }
          } else {
#pragma unroll 1
            for (int j = 0; j < 16; ++j) {
              const int r = 2 * j + (lane >> 4);
              const int64_t off = __shfl_sync(0xffffffffu, crow, r);
              const int e = __shfl_sync(0xffffffffu, erow, r) + ec;
              const float* at = src + 2 * j * OZ_XP_LD;
              const float tail = F64 && last >= 0 ? at[2 * OZ_XP_PLANE] : 0.0f;
              const double v = alpha_left * ff_to_f64(at[0], at[OZ_XP_PLANE], tail, e, aneg);
              if (!nok || r >= rows) continue;
              if (bmode == 0) dst[off] = v;
              else if (bmode == 1) atomicAdd(dst + off, v);
              else dst[off] = v + ep.beta * dst[off];
            }
          }
          __syncwarp();
        }
        if (F64 && last >= 0) {
          asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
          __syncwarp();
          if (lane == 0) drained(last);
        }
        bb = be;
      }
    }
    // every MMA is complete before TMEM is freed
    bool dn = mbar_wait(smem_u32(&done_bar), 0);
    dn = __all_sync(0xffffffffu, dn);
    if (!dn) atomicExch(&abort_flag, 1);
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (PAIR) cluster_sync();     // neither CTA goes while the other may still signal it or read its tiles
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
  }
  if (threadIdx.x == 0 && abort_flag) atomicExch(err, 1);
}

// C = alpha * sum_j part[j] + beta * C, the jobs summed in order.  The first
// nhi jobs (all of them without a cut) are those of the first part: exact
// multiples of 2^-24 of the row and column scales whose sum fits 53 bits, so it
// is exact, and adding the sum of the others, 2^-12 of it or less, is the one
// rounding of the result.
__global__ void __launch_bounds__(256) oz_reduce_kernel(const double* __restrict__ part, int nhi, int njobs,
                                                        EpiMap ep) {
  const int64_t MN = ep.M * ep.N;
  part += (int64_t)blockIdx.y * njobs * MN;
  auto sum = [&](int64_t t, int j0, int j1) {
    double s = 0.0;
    for (int j = j0; j < j1; j += 8) {   // eight loads in flight, added in order
      double x[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) x[q] = j + q < j1 ? part[(int64_t)(j + q) * MN + t] : 0.0;
#pragma unroll
      for (int q = 0; q < 8; ++q)
        if (j + q < j1) s += x[q];
    }
    return s;
  };
  for (int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; t < MN; t += (int64_t)gridDim.x * blockDim.x) {
    double s = sum(t, 0, nhi);
    if (nhi < njobs) s += sum(t, nhi, njobs);
    const uint32_t m = (uint32_t)t / (uint32_t)ep.N, n = (uint32_t)t - m * (uint32_t)ep.N;
    double* dst = static_cast<double*>(ep.C) + blockIdx.y * ep.bc + epi_row_off(ep, m) + epi_col_off(ep, n);
    if (ep.alpha != 1.0) s *= ep.alpha;
    if (ep.beta == 1.0) s += *dst;
    else if (ep.beta != 0.0) s += ep.beta * *dst;
    *dst = s;
  }
}

}  // namespace

OzLevel oz_level(int groups) { return OzLevel{groups - 1, groups, 0, 6, 0}; }

void gemm_oz(const __nv_bfloat16* A, int64_t a_rows, const int* exA, const __nv_bfloat16* B, int64_t b_rows,
             const int* exB, int64_t Kpad, OzLevel lv, const EpiMap& ep0, DBuf<double>& ws, int* err, cudaStream_t s) {
  EpiMap ep = ep0;
  if (ep.M <= 0 || ep.N <= 0) return;
  if (lv.S < 1 || lv.S > OZ_MAXS || lv.G < 2 || lv.G > lv.S + 2 || (lv.bits != 6 && lv.bits != 8) || lv.guard < 0 || lv.guard > 2)
    fail(FCC_ERR_BAD_ARG, "bad exact-slice level");
  if (Kpad <= 0 || Kpad % OZ_BK || Kpad > OZ_KMAX) fail(FCC_ERR_BAD_ARG, "bad padded K");
  if (ep.batch < 1 || ep.batch > 65535 || a_rows < ep.M + (ep.batch - 1) * ep.ba || b_rows < ep.N + (ep.batch - 1) * ep.bb)
    fail(FCC_ERR_BAD_ARG, "packed operands smaller than the output");
  if (ep.M >= (int64_t(1) << 31) || ep.N >= (int64_t(1) << 31)) fail(FCC_ERR_BAD_ARG, "output extent too large");
  // Pairs of CTAs on 256 x 128 tiles (4864^3 at 6 bits 3.03 ms, 3.60 with single
  // CTAs on 128 x 128), unless the last tile would leave more than an eighth of
  // the rows' work to padding.  A long product whose columns fit pairs and whose
  // rows do not is turned over: its stores no longer coalesce, which 32 k-blocks
  // outweigh (528 x 2888 x 11628: 0.79 ms as it stands, 0.67 turned over).
  auto pairs = [](int64_t rows) {
    const int64_t t = (rows + OZ_BM - 1) / OZ_BM;
    return t % 2 == 0 || t >= 8;
  };
  if (!pairs(ep.M) && pairs(ep.N) && Kpad >= 32 * OZ_BK) {
    std::swap(A, B);
    std::swap(a_rows, b_rows);
    std::swap(exA, exB);
    std::swap(ep.M, ep.N);
    std::swap(ep.md2, ep.nd2);
    std::swap(ep.md3, ep.nd3);
    std::swap(ep.ms1, ep.ns1);
    std::swap(ep.ms2, ep.ns2);
    std::swap(ep.ms3, ep.ns3);
    std::swap(ep.ba, ep.bb);
  }
  const bool pair = pairs(ep.M);
  auto* const kernel = lv.cut ? (pair ? gemm_oz_kernel<true, true> : gemm_oz_kernel<true, false>)
                              : (pair ? gemm_oz_kernel<false, true> : gemm_oz_kernel<false, false>);
  static SmemLimit smem[2][2];
  smem[lv.cut != 0][pair].raise(kernel, OZ_SMEM);
  OzParams P;
  std::memset(&P, 0, sizeof(P));
  const int nb = make_bands(lv, P.band);
  P.bits = lv.bits;
  P.guard = lv.guard;
  P.cut = lv.cut;
  P.kpad = (int)Kpad;
  const int nkb = (int)(Kpad / OZ_BK);
  const int64_t rows_unit = pair ? 2 * OZ_BM : OZ_BM;
  const int64_t tm = (ep.M + rows_unit - 1) / rows_unit, tn = (ep.N + OZ_BN - 1) / OZ_BN;
  const int64_t workers = pair ? 76 : 152;
  const int64_t tiles = tm * tn;
  if (tiles * OZ_MAXJOBS * ep.batch >= (int64_t(1) << 31) || a_rows >= (int64_t(1) << 31) || b_rows >= (int64_t(1) << 31))
    fail(FCC_ERR_BAD_ARG, "tensor-core grid too large");
  P.tm = (uint32_t)tm;
  P.tn = (uint32_t)tn;
  // L2 blocks: the units that run at the same time (one per SM, about 8 tile
  // rows x 19 tile columns in the grouped order) stream the same k-blocks;
  // their panels (all S slices of a 128-row block) must fit in L2 together,
  // or every slice is fetched again from HBM for each pair that uses it (a
  // full-K ring launch at (H2O)8 read 17 GB for 0.76 GB of packed operands)
  const double panel = (double)OZ_BM * lv.S * OZ_BK * 2.0;   // bytes per k-block
  const int64_t conc = std::min<int64_t>(tiles, workers);
  const int64_t rtile = std::min<int64_t>(tm, 8);
  const int64_t cblk = std::min<int64_t>(tn, (conc + rtile - 1) / rtile), rblk = pair ? 2 * rtile : rtile;
  constexpr double L2_BUDGET = 48.0 * (1 << 20);
  P.kper = (int)std::max(4.0, L2_BUDGET / ((double)(rblk + cblk) * panel));
  P.kper = std::min(P.kper & ~3, std::max(4, nkb));          // whole chunks of every band
  // Jobs: one per output tile when there are enough tiles; otherwise each
  // band's k-blocks are cut into pieces of about `target` steps whose partial
  // results are summed in order by oz_reduce_kernel (one more launch).  A unit
  // costs about FIXED steps besides its own (ramp-up, the last drain, its
  // stores); a step is ~0.2 us.
  int steps_kb = 0;
  for (int b = 0; b < nb; ++b) steps_kb += P.band[b].ntile - 1;
  const double total = (double)steps_kb * nkb;
  constexpr double FIXED = 24.0, REDUCE = 16.0;
  auto build = [&](double target) {
    int n = 0;
    if (target <= 0) {
      P.job[n++] = OzJob{0, (int16_t)nb, 0, nkb};
      return n;
    }
    for (int b = 0; b < nb;) {
      // join bands while they stay within the target (never across the cut)
      int e = b + 1;
      double st = (double)(P.band[b].ntile - 1) * nkb;
      while (e < nb && e != lv.cut && st + (double)(P.band[e].ntile - 1) * nkb <= target) {
        st += (double)(P.band[e].ntile - 1) * nkb;
        ++e;
      }
      int pieces = std::max(1, std::min(nkb, (int)std::ceil(st / target)));
      const int len = (nkb + pieces - 1) / pieces;
      for (int k = 0; k < nkb; k += len) {
        if (n == OZ_MAXJOBS) return -1;
        P.job[n++] = OzJob{(int16_t)b, (int16_t)e, k, std::min(nkb, k + len)};
      }
      b = e;
    }
    return n;
  };
  double best = 1e300, best_target = 0;
  for (int q = 0; q < 12; ++q) {
    const double target = q == 0 ? 0.0 : total / (double)(q < 5 ? q + 1 : (q < 9 ? 4 * (q - 3) : 36 << (q - 9)));
    const int n = build(target);
    if (n < 1 || (q > 0 && (n == 1 || (double)n * ep.batch * ep.M * ep.N > (double)(32 << 20)))) continue;
    // longest CTA under the static assignment of units to CTAs
    const int64_t units = tiles * n * ep.batch;
    double t = 0;
    for (int c = 0; c < std::min<int64_t>(units, 4); ++c) {
      const int64_t cta = c == 0 ? 0 : (c == 1 ? std::min<int64_t>(units, workers) - 1 : (c == 2 ? workers / 2 : 3 * workers / 4));
      double l = 0;
      for (int64_t u = cta; u < units; u += workers) {
        const OzJob& j = P.job[(u / tiles) % n];
        double st = 0;
        for (int b = j.b0; b < j.b1; ++b) st += P.band[b].ntile - 1;
        l += st * (j.k1 - j.k0) + FIXED;
        if (units > workers * 64) { l *= (double)((units + workers - 1) / workers); break; }
      }
      t = std::max(t, l);
    }
    if (n > 1) t += REDUCE + (double)(n + 2) * ep.batch * ep.M * ep.N * 8.0 / 1e6;   // ~1 MB a step
    if (t < best * 0.97) { best = t; best_target = target; }
  }
  P.njobs = (uint32_t)build(best_target);
  P.units = (uint32_t)(tiles * P.njobs * ep.batch);
  if (P.njobs > 1) {
    const size_t need = (size_t)P.njobs * ep.batch * ep.M * ep.N;
    if (ws.n >= need || ws.try_alloc(need)) {
      P.part = ws.p;
    } else {   // no room for partial results: one job a tile
      P.njobs = (uint32_t)build(0.0);
      P.units = (uint32_t)(tiles * P.njobs * ep.batch);
    }
  }
  // One job and one chunk in the first band: the other bands go first, and the
  // store stage adds the first band's two accumulators to their sums, so the
  // output is converted and written once instead of twice.
  if (lv.cut == 1 && P.njobs == 1 && P.band[0].ngrp == 2 && nkb <= P.band[0].ck) {
    std::reverse(P.band, P.band + nb);
    P.cut = 0;
    P.merged = 1;
    P.kper = std::max(P.kper, nkb);
  }
  CUtensorMap ta = tma_map_bf16(A, a_rows, lv.S * Kpad, OZ_BM);
  CUtensorMap tb = tma_map_bf16(B, b_rows, lv.S * Kpad, pair ? OZ_BN / 2 : OZ_BN);
  // persistent: one CTA per SM
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(std::min<int64_t>(P.units, workers) * (pair ? 2 : 1)));
  cfg.blockDim = dim3(OZ_THREADS);
  cfg.dynamicSmemBytes = OZ_SMEM;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = pair ? 2 : 1;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const int pidx = prof_begin(s);
  FCC_CUDA(cudaLaunchKernelEx(&cfg, kernel, ta, tb, P, exA, exB, ep, err));
  FCC_CHECK_LAUNCH();
  if (P.njobs > 1) {
    const int64_t MN = ep.M * ep.N;
    int nhi = (int)P.njobs;
    if (lv.cut) {
      nhi = 0;
      while (nhi < (int)P.njobs && P.job[nhi].b0 < lv.cut) ++nhi;
    }
    oz_reduce_kernel<<<dim3((unsigned)std::min<int64_t>((MN + 255) / 256, 152 * 8), (unsigned)ep.batch), 256, 0, s>>>(
        ws.p, nhi, (int)P.njobs, ep);
    FCC_CHECK_LAUNCH();
  }
  prof_end(s, pidx, PROF_OZ, ep.work > 0 ? ep.work : 2.0 * ep.batch * (double)ep.M * (double)ep.N * (double)Kpad * steps_kb);
}

}  // namespace fcc
