// Split-BF16 tensor-core contraction: operand packing and the tcgen05 GEMM.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>

#include "fcc_common.cuh"

namespace fcc {

// Split schemes.  x = hi + mid + lo with hi = bf16(x), mid = bf16(x - hi),
// lo = bf16(x - hi - mid).  A product A.B is evaluated as a sum of P piece
// products, stored as P column blocks of the packed operands:
//   3 products: A' = [hi hi mid],          B' = [hi mid hi]          (~2^-16)
//   6 products: A' = [hi hi mid hi mid lo], B' = [hi mid hi lo mid hi] (~2^-24)
// Piece p of an operand holds level (code >> 2p) & 3 (0 hi, 1 mid, 2 lo).
struct SplitScheme {
  int P;
  uint32_t code_a, code_b;
};
constexpr SplitScheme SPLIT3{3, 0u | (0u << 2) | (1u << 4), 0u | (1u << 2) | (0u << 4)};
constexpr SplitScheme SPLIT6{6, 0u | (0u << 2) | (1u << 4) | (0u << 6) | (1u << 8) | (2u << 10),
                             0u | (1u << 2) | (0u << 4) | (2u << 6) | (1u << 8) | (0u << 10)};

// Gather spec of a packed operand: row r = (r1*rd2 + r2)*rd3 + r3 and column
// k = (k1*kd2 + k2)*kd3 + k3 of a strided FP64 source; the destination is
// R rows x Kp bf16 with split piece p at columns [p*K, (p+1)*K), zero from
// P*K to Kp.
struct PackSpec {
  int64_t R, K, Kp;
  int64_t rd2, rd3, rs1, rs2, rs3;
  int64_t kd2, kd3, ks1, ks2, ks3;
  int P = 3;
  uint32_t code = 0;
  double scale = 1.0;   // the source is multiplied by this (exact for +-1 and powers of two)
};

// Source offsets of packed row r and packed column k (32-bit index
// arithmetic: pack_split / pack_oz reject R or K of 2^31 or more).
__device__ __forceinline__ int64_t pack_row_off(const PackSpec& ps, int64_t r) {
  const uint32_t rr = (uint32_t)r, d3 = (uint32_t)ps.rd3, d2 = (uint32_t)ps.rd2;
  const uint32_t r3 = rr % d3, q = rr / d3;
  return (int64_t)(q / d2) * ps.rs1 + (int64_t)(q % d2) * ps.rs2 + (int64_t)r3 * ps.rs3;
}
__device__ __forceinline__ int64_t pack_col_off(const PackSpec& ps, int64_t k) {
  const uint32_t kk = (uint32_t)k, d3 = (uint32_t)ps.kd3, d2 = (uint32_t)ps.kd2;
  const uint32_t k3 = kk % d3, q = kk / d3;
  return (int64_t)(q / d2) * ps.ks1 + (int64_t)(q % d2) * ps.ks2 + (int64_t)k3 * ps.ks3;
}
// Walks consecutive packed columns k, k+1, ... without divisions.
struct PackColIter {
  uint32_t k2, k3;
  int64_t off;
  __device__ __forceinline__ PackColIter(const PackSpec& ps, int64_t k) {
    const uint32_t kk = (uint32_t)k, d3 = (uint32_t)ps.kd3, d2 = (uint32_t)ps.kd2;
    k3 = kk % d3;
    const uint32_t q = kk / d3;
    k2 = q % d2;
    off = (int64_t)(q / d2) * ps.ks1 + (int64_t)k2 * ps.ks2 + (int64_t)k3 * ps.ks3;
  }
  __device__ __forceinline__ void next(const PackSpec& ps) {
    if (++k3 < (uint32_t)ps.kd3) { off += ps.ks3; return; }
    k3 = 0;
    off += ps.ks2 - (ps.kd3 - 1) * ps.ks3;
    if (++k2 < (uint32_t)ps.kd2) return;
    k2 = 0;
    off += ps.ks1 - ps.kd2 * ps.ks2;   // from (k1, kd2, 0) to (k1 + 1, 0, 0)
  }
};

// k is one source index (k3 = k): column offset k * ks3, no divisions
__host__ __device__ inline bool pack_k_single(const PackSpec& ps) { return ps.kd2 == 1 && ps.kd3 >= ps.K; }

// Source values of packed columns k0 .. k0 + cnt - 1 (cnt <= 4) of the row at
// source offset ro; zeros past cnt.
__device__ __forceinline__ void pack_load4(const double* __restrict__ src, const PackSpec& ps, bool k1, int64_t ro,
                                           int64_t k0, int cnt, double (&x)[4]) {
  if (k1) {
    const double* sp = src + ro + k0 * ps.ks3;
    if (ps.ks3 == 1 && cnt == 4 && (reinterpret_cast<uintptr_t>(sp) & 15) == 0) {
      const double2 a = *reinterpret_cast<const double2*>(sp), b = *reinterpret_cast<const double2*>(sp + 2);
      x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
      return;
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) x[q] = q < cnt ? sp[q * ps.ks3] : 0.0;
  } else {
    PackColIter ci(ps, k0);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      x[q] = q < cnt ? src[ro + ci.off] : 0.0;
      if (q + 1 < cnt) ci.next(ps);
    }
  }
}

// Row walk of the row-major pack kernels: a unit is a segment of gseg
// 4-column groups of one packed row (nseg segments per row), walked by 2^lg
// threads (32 ... 256); 256 >> lg units per block of 256 threads.  Rows are
// cut into segments when there are too few of them to fill the GPU.
struct PackWalk {
  int lg;
  int64_t gseg, nseg;
};
inline PackWalk pack_walk(int64_t R, int64_t groups) {
  PackWalk w;
  w.lg = 5;
  while (w.lg < 8 && (int64_t(1) << w.lg) < groups) ++w.lg;
  const int64_t tpr = int64_t(1) << w.lg;
  // about 152 SMs x 2048 threads, up to 8 groups each
  const int64_t per_thread = std::max<int64_t>(1, std::min<int64_t>(8, R * groups / (152 * 2048)));
  w.gseg = std::min(groups, tpr * per_thread);
  w.nseg = (groups + w.gseg - 1) / w.gseg;
  return w;
}
inline unsigned pack_walk_grid(const PackWalk& w, int64_t R) {
  const int64_t upb = 256 >> w.lg;
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>((R * w.nseg + upb - 1) / upb, 152 * 32));
}

// Output scatter of the GEMMs: element (m, n) goes to the FP64 value
// C[m1*ms1 + m2*ms2 + m3*ms3 + n1*ns1 + n2*ns2 + n3*ns3] as alpha * acc + beta * C
// (atomic: reduced into C by several K slices).
struct EpiMap {
  int64_t M = 0, N = 0;
  int64_t md2 = 1, md3 = 1, ms1 = 0, ms2 = 0, ms3 = 0;
  int64_t nd2 = 1, nd3 = 1, ns1 = 0, ns2 = 0, ns3 = 0;
  double alpha = 1.0, beta = 0.0;
  void* C = nullptr;
  int atomic = 0;
  // exact-slice products only: `batch` products of the same extents, product q
  // over the packed rows q * ba.. of A and q * bb.. of B into C + q * bc
  int batch = 1;
  int64_t ba = 0, bb = 0, bc = 0;
  double work = 0.0;   // algorithmic BF16 flops for the timing log (0: use the padded count)
  int no_loads = 0;    // test hook: the producer issues no TMA loads, so the bounded waits give up
};

// Offsets of row m and column n in C (32-bit divisions: M, N < 2^31; a 64-bit
// one costs a thread about a microsecond on this part).
__device__ __forceinline__ int64_t epi_row_off(const EpiMap& ep, uint32_t m) {
  const uint32_t d3 = (uint32_t)ep.md3, d2 = (uint32_t)ep.md2;
  const uint32_t m3 = m % d3, r = m / d3;
  return (int64_t)(r / d2) * ep.ms1 + (int64_t)(r % d2) * ep.ms2 + (int64_t)m3 * ep.ms3;
}
__device__ __forceinline__ int64_t epi_col_off(const EpiMap& ep, uint32_t n) {
  const uint32_t d3 = (uint32_t)ep.nd3, d2 = (uint32_t)ep.nd2;
  const uint32_t n3 = n % d3, r = n / d3;
  return (int64_t)(r / d2) * ep.ns1 + (int64_t)(r % d2) * ep.ns2 + (int64_t)n3 * ep.ns3;
}

int64_t packed_kp(int64_t K, int P = 3);
void pack_split(const double* src, const PackSpec& ps, __nv_bfloat16* dst, cudaStream_t s);
// D = A' B'^T over Kp packed columns; rows a_row0.. of A' (a_rows total) and
// b_row0.. of B' (b_rows total); err set to 1 if a bounded wait gave up.
void gemm_bf16x3(const __nv_bfloat16* A, int64_t a_rows, int64_t a_row0, const __nv_bfloat16* B, int64_t b_rows,
                 int64_t b_row0, int64_t Kp, const EpiMap& ep, int* err, cudaStream_t s);

// 2-D TMA map over a row-major [rows][cols] BF16 array, boxes of 64 columns
// (one 128-byte swizzle atom) x box_rows rows; cols must be a multiple of 64.
CUtensorMap tma_map_bf16(const __nv_bfloat16* base, int64_t rows, int64_t cols, int box_rows);

// Exact-slice products (the Ozaki scheme: Ozaki, Ogita, Oishi & Rump, Numer.
// Algorithms 59, 95 (2012); on tensor cores: Mukunoki et al., ISC 2020).
// Each row r of an operand is scaled by 2^e_r (|x| < 2^e_r over the row) and
// cut into S balanced digit slices of b bits, x = 2^e_r sum_s d_s 2^(-b s),
// |d_1| <= 2^b, |d_s| <= 2^(b-1), stored exactly in BF16 (8-bit significand).
// A.B^T is the sum over slice pairs (s, t) with s + t <= G of the digit
// products; pairs of one weight 2^(-b (s+t)) are summed on the tensor cores in
// FP32 while |sum| <= 2^24, so every partial sum is an exact integer, and
// those are added in double-FP32 (2^-47 to 2^-48).  BF16 carries 8-bit digits
// exactly, and fewer, wider digits need fewer products for the same bits (48
// bits: S = 6 and 21 products instead of the 36 of eight 6-bit digits), which
// the FP64 level uses.  The levels of the mixed and exact forms keep 6-bit
// digits, the finish too: its iterates, and so its converged T1, depend on what
// a level drops.  (At (H2O)8 a finish of six 8-bit digits, as many bits, moved T1
// by 1.3e-9 of its norm and T2 by 4e-12, where repeated solves agree to 1e-12;
// 6-bit digits agree to 1e-11.)
// `cut` > 0: the first `cut` bands of groups get a running sum of their own
// (the FP64 level, see gemm_oz.cu).  guard: the digits are cut from x 2^-guard,
// |d_1| <= 2^(b - guard), so that sums reach 2^24 later.
struct OzLevel {
  int S, G, cut, bits, guard;
};
// FP64 level: 62 bits below the row maximum (two guard bits, so that sums of
// first digits stay below 2^24 over 16 k-blocks), the first 36 pairs, the first
// band summed apart.  Dropped pairs and cut digits are about 2^-62 of max|A_r|
// max|B_c| per term and the sums carry ~2^-59 of the result, where an FP64
// product accumulates roundings of 2^-53 of its partial sums.  Error against
// quadruple precision on the operands of (H2O)4 (2-norm of the difference over
// that of the result), this level / FP64 pipe: DF fit over J^-1/2 1.6e-15 /
// 1.8e-14, MO transform 5.9e-17 / 5.3e-16, (ia|jb) 2.5e-17 / 2.3e-16, (ab|cd)
// 2e-17 / 5.3e-16, ring 1.9e-17 / 2.7e-16, ladder 1.1e-16 / 9e-16, (T) over d
// 2.3e-17 / 3.2e-16, over l 3e-17 / 1.7e-16.  Seven slices would be 5% faster
// and nearly as far off as the pipe on the DF fit; eight leave a decade.
constexpr OzLevel OZ_F64{8, 9, 1, 8, 2};
constexpr int OZ_MAXS = 8;
constexpr int OZ_G_DEFAULT = 8;
// the level of `groups` weight groups of 6-bit digits, the unit the phases of
// the mixed form are counted in
OzLevel oz_level(int groups);
// slice pairs (BF16 products) of a level
inline double oz_pairs(OzLevel lv) {
  int n = 0;
  for (int a = 1; a <= lv.S; ++a) n += std::max(0, std::min(lv.S, lv.G - a));
  return n;
}
// packed layout: row r holds slice s at columns [s*Kpad, s*Kpad + K), zero up
// to (s+1)*Kpad; ex[r] = biased FP64 exponent of max_k |x_rk| (0: all zero,
// 2047: the row holds an infinity or NaN, and so will its products)
int64_t oz_kpad(int64_t K);
// the extents pack_oz and gemm_oz take
constexpr int64_t OZ_KMAX = int64_t(1) << 27;
inline bool oz_takes(int64_t M, int64_t N, int64_t K) {
  return M < (int64_t(1) << 31) && N < (int64_t(1) << 31) && K <= OZ_KMAX;
}
void pack_oz(const double* src, const PackSpec& ps, int S, int bits, int guard, __nv_bfloat16* dst, int* ex,
             cudaStream_t s);
// exact-slice product over packed operands, written to ep;
// ws holds the partial results of products cut into several jobs
void gemm_oz(const __nv_bfloat16* A, int64_t a_rows, const int* exA, const __nv_bfloat16* B, int64_t b_rows,
             const int* exB, int64_t Kpad, OzLevel lv, const EpiMap& ep, DBuf<double>& ws, int* err, cudaStream_t s);

// Engine state for einsum calls that run on the tensor cores: scratch for
// the packed operands, the device error flag, the routing threshold and
// counters of what ran.
struct TcEngine {
  bool enabled = false;
  SplitScheme scheme = SPLIT3;
  bool exact = false;      // exact-slice products instead of the split scheme
  OzLevel oz = oz_level(OZ_G_DEFAULT);
  DBuf<int> exA, exB;
  DBuf<double> ozws;       // partial results of exact-slice products cut into jobs
  double min_flops = 1e6;
  int64_t min_dim = 16;   // smallest M and N routed to the tensor cores
  // FP64 contractions of this size and more run as exact-slice products at the
  // FP64 level, whether `enabled` or not
  double f64_min_flops = 4e7;
  // FP64 contractions on the FP64 pipe, from 1e7 flop on in 64 x 64 tiles: the
  // integrals that every form starts from (setup_integrals)
  bool f64_wide = false;
  bool f64_sym = false;   // and the next ones' results are symmetric in (m, n)
  DBuf<__nv_bfloat16> bufA, bufB;
  int* err = nullptr;
  int no_loads_once = 0;   // test hook: the next tensor-core GEMM runs with EpiMap::no_loads
  // Packed A operands kept across calls: an A operand whose source is one of
  // keep_src (set by a KeepPackedA scope, whose caller guarantees that those
  // sources do not change meanwhile) is packed into its own entry and packed
  // again only when its layout or level changes, so an operand used by
  // every block of a loop is packed once.
  struct KeptPack {
    PackSpec ps{};
    int S = 0, bits = 0, guard = 0;
    bool valid = false;
    DBuf<__nv_bfloat16> buf;
    DBuf<int> ex;
  };
  const double* keep_src[2] = {nullptr, nullptr};
  KeptPack kept[2];
  // The ladder's dressed factors Bt[Q][x][y] (x, y virtual) packed once per
  // residual for every block's (ac|bd) product (rows (x, y), K = Q): digit
  // slices and row exponents, or the split pieces in the A and in the B order
  DBuf<__nv_bfloat16> bvvA, bvvB;
  DBuf<int> bvvEx;
  // Digit slices take twice the memory of an FP64 operand, and FP64 contractions
  // can do without: they take more scratch (from 250 MB on) only while that leaves
  // half of the free memory, and run on the FP64 pipe otherwise or where the
  // allocation fails.
  double scratch_max = 1e300;   // test hook: bytes of packed operands in all
  double scratch_held() const {
    double b = (double)(bufA.bytes() + bufB.bytes() + exA.bytes() + exB.bytes() + bvvA.bytes() + bvvB.bytes() + bvvEx.bytes());
    for (const KeptPack& k : kept) b += (double)(k.buf.bytes() + k.ex.bytes());
    return b;
  }
  bool scratch_fits(double growth) const;
  // Given back where another allocation of the thread's call finds no memory
  // (unless a product is using it), and at the end of a call that leaves more than
  // KEEP: the 1.7 GB of an FP64 run at (H2O)8 stay for the next call, the 4.6 of a
  // mixed one at (H2O)12 do not (such a call takes seconds, allocating them again
  // milliseconds).
  static constexpr double KEEP = 4e9;
  double scratch_keep = KEEP;
  int busy = 0;
  void release_scratch();
  int64_t tc_calls = 0, f64_calls = 0;
  double tc_flops = 0, f64_flops = 0;
};

// Keep the packed forms of the A operands with sources a0 and a1 over the
// following contractions; they are dropped when the scope ends.
struct KeepPackedA {
  TcEngine* tc;
  KeepPackedA(TcEngine* e, const double* a0, const double* a1) : tc(e) {
    if (!tc) return;
    tc->keep_src[0] = a0;
    tc->keep_src[1] = a1;
    for (auto& k : tc->kept) k.valid = false;
  }
  ~KeepPackedA() {
    if (!tc) return;
    tc->keep_src[0] = tc->keep_src[1] = nullptr;
    for (auto& k : tc->kept) k.valid = false;
  }
};

// Current engine of this host thread (nullptr: every contraction is on the
// FP64 pipe).
TcEngine*& tc_engine();

// While one is alive the engine's packed operands stay where they are.
struct ScratchInUse {
  TcEngine* tc;
  explicit ScratchInUse(TcEngine* e) : tc(e) { if (tc) ++tc->busy; }
  ~ScratchInUse() { if (tc) --tc->busy; }
  ScratchInUse(const ScratchInUse&) = delete;
  ScratchInUse& operator=(const ScratchInUse&) = delete;
};

// The end of an entry point: what it leaves beyond KEEP is given back.
struct ScratchBound {
  TcEngine* tc;
  explicit ScratchBound(TcEngine* e) : tc(e) {}
  ~ScratchBound() { if (tc && tc->scratch_held() + (double)tc->ozws.bytes() > tc->scratch_keep) tc->release_scratch(); }
  ScratchBound(const ScratchBound&) = delete;
  ScratchBound& operator=(const ScratchBound&) = delete;
};

struct TcScope {
  TcEngine* prev;
  explicit TcScope(TcEngine* e) : prev(tc_engine()) { tc_engine() = e; }
  ~TcScope() { tc_engine() = prev; }
};

}  // namespace fcc
