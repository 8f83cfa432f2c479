// Grouped, K-segmented split-BF16 tensor-core GEMM for the (T) intermediates.
//
// For one pair (i, j) and a run of k, W_ijk[a][b][c] is the sum of twelve
// contractions (PerturbativeTriples/ijk.jl:109-114).  Each term carries one
// virtual index alone on one operand (c, b or a) and the other two together
// on the other operand; grouping the terms by that lone index gives three
// groups of four terms with the same (pair, lone) orientation:
//   group 0: rows (a,b), columns c    group 1: rows (a,c), columns b
//   group 2: rows (b,c), columns a
// so each group is ONE product whose K is the concatenation of the four
// terms' K ranges (two over d, two over l; the l terms' signs are folded
// into their packed operands).  One launch computes all groups for all k of
// the run: CTA (m-tile, group, k), four K segments, each read by TMA from
// its own packed operand.  The FP32 results are stored once, G_g[k][pair][lone]
// (no read-modify-write); the energy kernel adds the three groups.
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <cstring>

#include "fcc_t3.cuh"
#include "fcc_tcgen05.cuh"

namespace fcc {

namespace {

using namespace tc5;

constexpr int T3_BM = 128;
constexpr int T3_BK = 64;
constexpr int T3_THREADS = 192;   // warp 0 TMA, warp 1 MMA, warps 2-5 epilogue
template <int BN>
struct T3Cfg {
  static constexpr int STAGES = BN > 192 ? 6 : 7;
  static constexpr int A_BYTES = T3_BM * T3_BK * 2;
  static constexpr int B_BYTES = BN / 2 * T3_BK * 2;   // this CTA's half
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int SMEM = STAGES * STAGE_BYTES + 1024;
  static constexpr int TMEM_COLS = BN <= 32 ? 32 : BN <= 64 ? 64 : BN <= 128 ? 128 : 256;   // per accumulator (two)
};

__device__ __forceinline__ int t3_sel(int code, int i, int j, int k) { return code == 0 ? i : (code == 1 ? j : k); }

// tile t -> (m-tile, n-tile, group, k - k0), m-tile fastest.  Group 0 comes
// first for every k of the run (its A operands belong to i and j only, so
// they stay in L2 across the k sweep); then groups 1 and 2 alternate per k
// (they share the A operands of k, and each keeps its i- or j-operands).
// With the group outermost of all, group 0's A panels were evicted between
// consecutive k and read again from HBM for every k.
struct T3Tile {
  int mt, nt, g, kq;
};
__device__ __forceinline__ T3Tile t3_tile(int t, int tm, int tn, int nk) {
  T3Tile r;
  const int per = tm * tn;
  const int q = t / per, rem = t - q * per;
  r.mt = rem % tm;
  r.nt = rem / tm;
  if (q < nk) {
    r.g = 0;
    r.kq = q;
  } else {
    const int q2 = q - nk;
    r.kq = q2 >> 1;
    r.g = 1 + (q2 & 1);
  }
  return r;
}

// Persistent: each pair of CTAs (cta_group::2, a 256 x BN tile: 128 rows and
// half of every B tile each) walks tiles b, b + pairs, ...; a step of 128 x 160 x
// 64 in a single CTA moved 36 KB in and out of shared memory, 576 clk for 320 of
// MMAs, in a pair 26 KB (the GEMMs of a (T) at (H2O)8: 160 ms, 148 in pairs).
// The TMA thread streams the K segments of its tiles through a shared-memory
// ring, the MMA thread alternates two TMEM accumulators, and the epilogue
// warps store tile t while the MMAs of tile t+1 run.
template <int BN>
__global__ void __launch_bounds__(T3_THREADS, 1) gemm_t3_kernel(const __grid_constant__ T3Params P, int tm,
                                                                 int tn, int ntiles) {
  using Cfg = T3Cfg<BN>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full_bar[Cfg::STAGES];
  __shared__ __align__(8) uint64_t empty_bar[Cfg::STAGES];
  __shared__ __align__(8) uint64_t accf_bar[2];   // accumulator b holds a finished tile
  __shared__ __align__(8) uint64_t acce_bar[2];   // accumulator b has been read out
  __shared__ __align__(8) uint64_t done_bar;      // every issued MMA has completed
  __shared__ uint32_t tmem_holder;
  __shared__ int abort_flag;

  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* sA = smem;
  uint8_t* sB = smem + Cfg::STAGES * Cfg::A_BYTES;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int64_t v = P.v, o = P.o;

  if (threadIdx.x == 0) {
    for (int s = 0; s < Cfg::STAGES; ++s) {
      mbar_init(smem_u32(&full_bar[s]), 1);
      mbar_init(smem_u32(&empty_bar[s]), 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(smem_u32(&accf_bar[b]), 1);
      mbar_init(smem_u32(&acce_bar[b]), 8);   // one arrival per epilogue warp of the pair
    }
    mbar_init(smem_u32(&done_bar), 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_holder)),
                 "r"(2 * Cfg::TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync();     // both CTAs' barriers are there before either is signalled
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_holder;
  const uint32_t rank = cluster_rank();
  const int wid = blockIdx.x >> 1, nwork = gridDim.x >> 1;

  if (warp == 0) {
   if (elect_one()) {
    // ---------------- TMA producer over the tiles' K segments
    int it = 0;
    bool stop = P.no_loads != 0;
    for (int t = wid; t < ntiles && !stop; t += nwork) {
      const T3Tile tl = t3_tile(t, tm, tn, P.nk);
      const int kk = P.k0 + tl.kq;
      const int64_t m0 = (int64_t)tl.mt * (2 * T3_BM) + rank * T3_BM;
      for (int s = 0; s < T3_NSEG && !stop; ++s) {
        const T3Seg sg = P.seg[tl.g][s];
        const int32_t arow = (int32_t)(t3_sel(sg.asel, P.i, P.j, kk) * v * v + m0);
        const int32_t brow = (int32_t)((t3_sel(sg.bsel1, P.i, P.j, kk) * o + t3_sel(sg.bsel2, P.i, P.j, kk)) * v +
                                       (int64_t)tl.nt * BN + rank * (BN / 2));
        for (int kb = 0; kb < sg.nkb; ++kb, ++it) {
          const int st = it % Cfg::STAGES;
          const uint32_t ph = (it / Cfg::STAGES) & 1;
          if (!mbar_wait(smem_u32(&empty_bar[st]), ph ^ 1)) { atomicExch(&abort_flag, 1); stop = true; break; }
          if (*(volatile int*)&abort_flag) { stop = true; break; }
          const uint32_t fb = smem_u32(&full_bar[st]), f0 = cluster_addr(fb, 0);
          // both CTAs' loads count on the first one's barrier
          if (rank == 0) mbar_expect_tx(fb, 2 * Cfg::STAGE_BYTES);
          tma_load_2d_pair(smem_u32(sA + st * Cfg::A_BYTES), &P.maps[sg.amap], kb * T3_BK, arow, f0);
          tma_load_2d_pair(smem_u32(sB + st * Cfg::B_BYTES), &P.maps[sg.bmap], kb * T3_BK, brow, f0);
        }
      }
    }
    if (stop && rank == 0) {
      // wait (bounded) for both CTAs' loads still in flight before shared memory is released
      for (int q = max(0, it - Cfg::STAGES); q < it; ++q)
        (void)mbar_wait(smem_u32(&full_bar[q % Cfg::STAGES]), (q / Cfg::STAGES) & 1);
    }
   }
  } else if (warp == 1) {
   if (rank == 0 && elect_one()) {
    // ---------------- MMA issuer, for both CTAs
    constexpr uint32_t idesc = idesc_bf16(2 * T3_BM, BN);
    const uint64_t ad0 = sw128_desc(smem_u32(sA)), bd0 = sw128_desc(smem_u32(sB));
    uint32_t st = 0, ph = 0, peek = 0;
    int lt = 0;
    bool ok = true;
    for (int t = wid; t < ntiles && ok; t += nwork, ++lt) {
      const int g = t3_tile(t, tm, tn, P.nk).g;
      int total = 0;
      for (int s = 0; s < T3_NSEG; ++s) total += P.seg[g][s].nkb;
      const int b = lt & 1;
      if (!mbar_wait(smem_u32(&acce_bar[b]), ((lt >> 1) & 1) ^ 1)) { atomicExch(&abort_flag, 1); break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t dcol = tmem + (uint32_t)(b * Cfg::TMEM_COLS);
      for (int x = 0; x < total; ++x) {
        // the next stage's barrier is read between the MMAs of a stage, while
        // the tensor pipe has work queued
        if (!peek && !mbar_wait(smem_u32(&full_bar[st]), ph)) { atomicExch(&abort_flag, 1); ok = false; break; }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const uint64_t ad = ad0 + (uint64_t)(st * (Cfg::A_BYTES >> 4));
        const uint64_t bd = bd0 + (uint64_t)(st * (Cfg::B_BYTES >> 4));
        uint32_t st2 = st + 1, ph2 = ph;
        if (st2 == Cfg::STAGES) { st2 = 0; ph2 ^= 1; }
        mma_bf16_pair(dcol, ad, bd, idesc, x > 0 ? 1u : 0u);
        peek = mbar_test(smem_u32(&full_bar[st2]), ph2);
        mma_bf16_pair(dcol, ad + 2, bd + 2, idesc, 1u);
        mma_bf16_pair(dcol, ad + 4, bd + 4, idesc, 1u);
        mma_bf16_pair(dcol, ad + 6, bd + 6, idesc, 1u);
        tc_commit_pair(smem_u32(&empty_bar[st]));
        st = st2;
        ph = ph2;
      }
      if (!ok) break;
      tc_commit_pair(smem_u32(&accf_bar[b]));
    }
    // TMEM is freed only after every issued MMA has completed (also on an abort)
    tc_commit_pair(smem_u32(&done_bar));
    if (!mbar_wait(smem_u32(&done_bar), 0)) atomicExch(&abort_flag, 1);
   }
  } else if (warp >= 2) {
    // ---------------- epilogue: each lane has a row (x, y) and stores its columns
    // in whole 32-byte sectors straight from the registers.  (Transposed through
    // shared memory for 128-byte rows, an element took about eight instructions
    // of the warp instead of one and a half, and the shared memory shared with
    // the MMAs: 167 ms of a (T) at (H2O)8 where this took 160, 29 and 24 ms at
    // (H2O)6 with odd sizes.)
    const int q = warp & 3;
    const int64_t v2 = v * v;
    int lt = 0;
    for (int t = wid; t < ntiles; t += nwork, ++lt) {
      const T3Tile tl = t3_tile(t, tm, tn, P.nk);
      const int b = lt & 1;
      bool ok = mbar_wait(smem_u32(&accf_bar[b]), (lt >> 1) & 1);
      ok = __all_sync(0xffffffffu, ok);
      if (!ok || __any_sync(0xffffffffu, *(volatile int*)&abort_flag != 0)) { atomicExch(&abort_flag, 1); break; }
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const int64_t m0 = (int64_t)tl.mt * (2 * T3_BM) + rank * T3_BM;
      const int64_t nbk = t3_nb(v);
      float* out = P.G + ((int64_t)tl.g * P.nk + tl.kq) * t3_slab(v);
      const int64_t nb0 = (int64_t)tl.nt * BN;
      const int64_t mr = m0 + q * 32 + lane;
      const int x = (int)((uint32_t)mr / (uint32_t)P.v), y = (int)mr - x * P.v;
      float* dst = out + t3_cube(x >> 3, y >> 3, 0, nbk) + t3_run(x & 7, y & 7);
      const bool swap = ((x ^ y) & 4) != 0;
#pragma unroll 1
      for (int c0 = 0; c0 < BN; c0 += 32) {
        if (nb0 + c0 >= v) break;
        uint32_t r[32];
        tmem_ld32(tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * Cfg::TMEM_COLS + c0), r);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          const int64_t n = nb0 + c0 + 8 * g;
          if (mr < v2 && n < v) {   // columns past v in the last run are padding of the slab
            uint32_t w[8];
#pragma unroll
            for (int l = 0; l < 8; ++l) w[l] = swap ? r[8 * g + (l ^ 4)] : r[8 * g + l];
            asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(dst + ((n >> 3) << 9)), "r"(w[0]),
                         "r"(w[1]), "r"(w[2]), "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
                         : "memory");
          }
        }
      }
      // the accumulator is free for the tile after next
      asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(cluster_addr(smem_u32(&acce_bar[b]), 0));
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  cluster_sync();     // neither CTA goes while the other may still signal it or read its tiles
  if (warp == 1) {
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * Cfg::TMEM_COLS)
                 : "memory");
  }
  if (threadIdx.x == 0 && abort_flag) atomicExch(P.err, 1);
}

template <int BN>
void launch_t3(const T3Params& P, cudaStream_t s) {
  using Cfg = T3Cfg<BN>;
  static SmemLimit smem;
  smem.raise(gemm_t3_kernel<BN>, Cfg::SMEM);
  const int64_t tm = ((int64_t)P.v * P.v + 2 * T3_BM - 1) / (2 * T3_BM);
  const int64_t tn = (P.v + BN - 1) / BN;
  const int64_t ntiles = tm * tn * 3 * P.nk;
  if (ntiles > (int64_t)1 << 30) fail(FCC_ERR_BAD_ARG, "too many (T) tiles in one launch");
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(2 * std::min<int64_t>(ntiles, 76)));   // a CTA per SM, in pairs
  cfg.blockDim = dim3(T3_THREADS);
  cfg.dynamicSmemBytes = Cfg::SMEM;
  cfg.stream = s;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = 2;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  FCC_CUDA(cudaLaunchKernelEx(&cfg, gemm_t3_kernel<BN>, P, (int)tm, (int)tn, (int)ntiles));
  FCC_CHECK_LAUNCH();
}

}  // namespace

int t3_bn(int v) {
  if (v <= 128) return 128;
  if (v <= 160) return 160;
  if (v <= 192) return 192;
  return 256;   // v > 256: several column tiles
}

void gemm_t3(const T3Params& P, cudaStream_t s) {
  if (P.nk <= 0) return;
  if (P.nk > 65535) fail(FCC_ERR_BAD_ARG, "too many k in one (T) launch");
  const double flops = 2.0 * 3.0 * (double)P.nk * (double)P.v * P.v * P.v *
                       (double)(P.seg[0][0].nkb + P.seg[0][1].nkb + P.seg[0][2].nkb + P.seg[0][3].nkb) * T3_BK;
  const int pidx = prof_begin(s);
  switch (P.bn) {
    case 128: launch_t3<128>(P, s); break;
    case 160: launch_t3<160>(P, s); break;
    case 192: launch_t3<192>(P, s); break;
    case 256: launch_t3<256>(P, s); break;
    default: fail(FCC_ERR_BAD_ARG, "no (T) tile width for this v");
  }
  prof_end(s, pidx, PROF_TC, flops);
}

}  // namespace fcc
