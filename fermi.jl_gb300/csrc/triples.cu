// RCCSD(T) perturbative triples on one GPU, FP64 form.
//
// Algorithm: Fermi.jl's default (T), src/Methods/CoupledCluster/
// PerturbativeTriples/ijk.jl:20-149.  For every occupied triplet i >= j >= k
// the v^3 intermediate W is the sum of the twelve contractions of
// ijk.jl:109-114 (six over a virtual index d, six over an occupied index l),
// V = W + the three T1 x (ia|jb) products of ijk.jl:116, and the energy is the
// six-fold permutation sum of ijk.jl:121-137 with weight
// (2 - d_ij - d_jk) / (D_ijkabc (1 + d_ab + d_bc)) over a >= b >= c.
//
// Two of the twelve terms always share the occupied index of their two-electron
// integral over virtuals and amplitude over l, so they are one product over the
// concatenated index [d, l] of two arrays,
//   F[x][y][z] = [ (xy|zd) | -t(x,l,y,z) ],  H[x][y][z] = [ t(x,y,z,d) | (ly|xz) ],
//   W_ijk(a,b,c) = F[i](a,b) H[k][j](c) + F[j](b,a) H[k][i](c) + F[k](c,a) H[j][i](b)
//                + F[i](a,c) H[j][k](b) + F[k](c,b) H[i][j](a) + F[j](b,c) H[i][k](a),
// and F and H are cut into digit slices once.  For one j, a run of i >= j and
// all k <= j the six terms are six exact-slice products at the FP64 level into
// W[i][k][a][b][c] (the runs of i and k join the rows or columns, or are a batch
// where their rows are not adjacent), with c or its run the columns so that
// stores coalesce.  (Twelve FP64-pipe contractions per pair and run of k took
// 0.54 s at (H2O)4 where this takes 0.04, of which the products' store stages
// are the larger part: K = v + o is short.)  Small systems, and those whose slices
// do not fit in memory, run the terms on the FP64 pipe.  The energy kernel then works on 8 x
// 8 x 8 sub-cubes (blocks A >= B >= C): it stages the six permutations of a
// sub-cube of W in shared memory with loads along W's stride-1 index, forms V
// from T1 and (ia|jb) blocks staged beside them, and reduces in FP64 into
// per-(i, k, sub-cube) partials that are summed in a fixed order at the end.
#include <algorithm>
#include <cmath>

#include "fcc_ctx.cuh"

namespace fcc {

namespace {

constexpr int EB = 256;          // threads per energy block

__device__ __forceinline__ double warp_sum(double x) {
  for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
  return x;
}

constexpr int ET = 8;            // sub-cube edge of the energy kernel

struct TileTri {
  int16_t a, b, c, pad;
};

// Energy of the triplets (i0 + blockIdx.y / nk, j, k0 + blockIdx.y % nk) on the
// sub-cube tiles[blockIdx.x] (blocks A >= B >= C), from W[blockIdx.y][a][b][c].
// part[(i * o + k) * ntiles + tile] accumulates over the calls in a fixed order.
__global__ void __launch_bounds__(EB) triples_energy_f64_kernel(const double* __restrict__ W,
                                                                const TileTri* __restrict__ tiles, int ntiles,
                                                                const double* __restrict__ t1,
                                                                const double* __restrict__ ovov,
                                                                const double* __restrict__ eps, int o, int v,
                                                                int i0, int j, int k0, int nk,
                                                                double* __restrict__ part) {
  __shared__ double Wt[6][ET][ET][ET + 1];   // W on the six permutations of the sub-cube
  __shared__ double Mjk[3][3][ET][ET + 1];   // (j y|k z) for y in block r1, z in block r2
  __shared__ double Mik[3][3][ET][ET + 1];
  __shared__ double Mij[3][3][ET][ET + 1];
  __shared__ double T1[3][3][ET];            // t1 of i, j, k on block r
  __shared__ double epsv[3][ET];
  __shared__ double red[EB / 32];
  const int kq = blockIdx.y, i = i0 + kq / nk, k = k0 + kq % nk;
  if (i == j && j == k) return;              // weight 2 - d_ij - d_jk = 0
  const TileTri tt = tiles[blockIdx.x];
  const int oa = tt.a * ET, ob = tt.b * ET, oc = tt.c * ET;
  auto org = [&](int r) { return r == 0 ? oa : (r == 1 ? ob : oc); };
  const int64_t v2 = (int64_t)v * v;
  const double* Wk = W + (int64_t)kq * v2 * v;
  // permutation p: roles (rx, ry, rz) of the sub-cube blocks, 2 bits each:
  // (0,1,2) (0,2,1) (1,0,2) (1,2,0) (2,0,1) (2,1,0)
  constexpr uint64_t PRC = (0ull | 1ull << 2 | 2ull << 4) | (0ull | 2ull << 2 | 1ull << 4) << 8 |
                           (1ull | 0ull << 2 | 2ull << 4) << 16 | (1ull | 2ull << 2 | 0ull << 4) << 24 |
                           (2ull | 0ull << 2 | 1ull << 4) << 32 | (2ull | 1ull << 2 | 0ull << 4) << 40;
  auto role = [](int p, int r) { return (int)((PRC >> (8 * p + 2 * r)) & 3); };
  const int t = threadIdx.x;
  // every thread issues all its global loads first, then writes shared memory
  constexpr int NE = 6 * ET * ET * ET / EB;
  constexpr int NM = (9 * ET * ET + EB - 1) / EB;
  double w[NE], mjk[NM], mik[NM], mij[NM];
  const int64_t mstr = (int64_t)o * v;
#pragma unroll
  for (int q = 0; q < NE; ++q) {
    const int e = t + q * EB;
    const int p = e / (ET * ET * ET), r = e % (ET * ET * ET);
    const int x = org(role(p, 0)) + r / (ET * ET), y = org(role(p, 1)) + (r / ET) % ET, z = org(role(p, 2)) + r % ET;
    w[q] = (x < v && y < v && z < v) ? Wk[((int64_t)x * v + y) * v + z] : 0.0;
  }
#pragma unroll
  for (int q = 0; q < NM; ++q) {
    const int e = t + q * EB;
    mjk[q] = mik[q] = mij[q] = 0.0;
    if (e < 9 * ET * ET) {
      const int rr = e / (ET * ET), qq = e % (ET * ET);
      const int Y = org(rr / 3) + qq / ET, Z = org(rr % 3) + qq % ET;
      if (Y < v && Z < v) {
        // ovov[p][y][q][z] = (p y|q z), row stride o*v
        mjk[q] = ovov[((int64_t)j * v + Y) * mstr + (int64_t)k * v + Z];
        mik[q] = ovov[((int64_t)i * v + Y) * mstr + (int64_t)k * v + Z];
        mij[q] = ovov[((int64_t)i * v + Y) * mstr + (int64_t)j * v + Z];
      }
    }
  }
  if (t < 3 * ET) {
    const int r = t / ET, x = t % ET, X = org(r) + x;
    T1[0][r][x] = X < v ? t1[(int64_t)i * v + X] : 0.0;
    T1[1][r][x] = X < v ? t1[(int64_t)j * v + X] : 0.0;
    T1[2][r][x] = X < v ? t1[(int64_t)k * v + X] : 0.0;
    epsv[r][x] = X < v ? eps[o + X] : 0.0;
  }
#pragma unroll
  for (int q = 0; q < NM; ++q) {
    const int e = t + q * EB;
    if (e < 9 * ET * ET) {
      const int rr = e / (ET * ET), qq = e % (ET * ET);
      Mjk[rr / 3][rr % 3][qq / ET][qq % ET] = mjk[q];
      Mik[rr / 3][rr % 3][qq / ET][qq % ET] = mik[q];
      Mij[rr / 3][rr % 3][qq / ET][qq % ET] = mij[q];
    }
  }
#pragma unroll
  for (int q = 0; q < NE; ++q) {
    const int e = t + q * EB;
    const int p = e / (ET * ET * ET), r = e % (ET * ET * ET);
    Wt[p][r / (ET * ET)][(r / ET) % ET][r % ET] = w[q];
  }
  __syncthreads();
  // V(x,y,z) for x in block rx at lx etc.: W + t1_ix (jy|kz) + (ix|kz) t1_jy + (ix|jy) t1_kz  (ijk.jl:116)
  auto V = [&](int rx, int lx, int ry, int ly, int rz, int lz, double wv) -> double {
    return wv + T1[0][rx][lx] * Mjk[ry][rz][ly][lz] + Mik[rx][rz][lx][lz] * T1[1][ry][ly] +
           Mij[rx][ry][lx][ly] * T1[2][rz][lz];
  };
  const double Dijk = eps[i] + eps[j] + eps[k];
  double acc = 0.0;
  for (int e = t; e < ET * ET * ET; e += EB) {
    const int la = e / (ET * ET), lb = (e / ET) % ET, lc = e % ET;
    const int a = oa + la, b = ob + lb, c = oc + lc;
    if (a >= v || b >= v || c >= v || b > a || c > b) continue;
    const double Wabc = Wt[0][la][lb][lc], Wacb = Wt[1][la][lc][lb], Wbac = Wt[2][lb][la][lc];
    const double Wbca = Wt[3][lb][lc][la], Wcab = Wt[4][lc][la][lb], Wcba = Wt[5][lc][lb][la];
    const double Vabc = V(0, la, 1, lb, 2, lc, Wabc), Vacb = V(0, la, 2, lc, 1, lb, Wacb);
    const double Vbac = V(1, lb, 0, la, 2, lc, Wbac), Vbca = V(1, lb, 2, lc, 0, la, Wbca);
    const double Vcab = V(2, lc, 0, la, 1, lb, Wcab), Vcba = V(2, lc, 1, lb, 0, la, Wcba);
    const double X = Wabc * Vabc + Wacb * Vacb + Wbac * Vbac + Wbca * Vbca + Wcab * Vcab + Wcba * Vcba;   // :129
    const double Y = Vabc + Vbca + Vcab;                                                                   // :130
    const double Z = Vacb + Vbac + Vcba;                                                                   // :131
    const double Ef = (Y - 2.0 * Z) * (Wabc + Wbca + Wcab) + (Z - 2.0 * Y) * (Wacb + Wbac + Wcba) + 3.0 * X;
    const double Dd = Dijk - epsv[0][la] - epsv[1][lb] - epsv[2][lc];
    acc += Ef / (Dd * (1.0 + (a == b) + (b == c)));                                                       // :133
  }
  acc = warp_sum(acc);
  if ((t & 31) == 0) red[t >> 5] = acc;
  __syncthreads();
  if (t == 0) {
    double s = 0.0;
    for (int q = 0; q < EB / 32; ++q) s += red[q];
    part[((int64_t)i * o + k) * ntiles + blockIdx.x] += (2.0 - (i == j) - (j == k)) * s;
  }
}

// sum of n values by one block, a fixed order
__global__ void __launch_bounds__(1024) sum_kernel(const double* part, int n, double* out) {
  __shared__ double sh[32];
  double s = 0.0;
#pragma unroll 4
  for (int b = threadIdx.x; b < n; b += 1024) s += part[b];
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x >= 32) return;
  s = warp_sum(sh[threadIdx.x]);
  if (threadIdx.x == 0) *out = s;
}

}  // namespace

double triples_fp64(fcc_ctx* c, const std::vector<int3>* subset, std::vector<double>* each) {
  cudaStream_t s = c->stream;
  TcScope scope(&c->tc);
  c->tc.enabled = false;
  reset_device_error(c);
  const int64_t o = c->o, v = c->v, Q = c->Q, n = c->n;
  const int64_t v2 = v * v, v3 = v2 * v;
  const int64_t Kc = v + o;
  TView B = rm(c->B.p, {Q, n, n});
  TView Boo = slice(slice(B, 1, 0, o), 2, 0, o);
  TView Bov = slice(slice(B, 1, 0, o), 2, o, v);
  TView Bvv = slice(slice(B, 1, o, v), 2, o, v);
  TView t2v = rm(c->t2.p, {o, o, v, v});
  // F and H in FP64, then their digit slices: F by (x, y, z) and by (x, z, y),
  // H by (x, y, z) and by (y, x, z), so that every run below is adjacent rows
  const OzLevel lv = OZ_F64;
  const int64_t Kpad = oz_kpad(Kc), rowlen = lv.S * Kpad;
  const int64_t RF = o * v2, RH = o * o * v;
  // one packed operand: its rows from a first row on
  struct Packed {
    DBuf<__nv_bfloat16> p;
    DBuf<int> e;
    void alloc(int64_t rows, int64_t rowlen) { p.alloc(rows * rowlen); e.alloc(rows); }
  };
  // Rows of F or H for a product: packed from one on (p, e, n of them), or in
  // FP64, row (x, y, z) of segment q at p + x sx + y sy + z sz with K columns ks
  // apart, times a.  The columns [d, l] are one segment, or two that read the
  // integrals and amplitudes where they are; r gives the indices of a product's
  // three row levels and of its batch as (x, y, z) = (0, 1, 2).
  struct Seg { const double* p; int64_t sx, sy, sz, ks, K; double a; };
  struct Rows { const __nv_bfloat16* p; const int* e; int64_t n; int64_t x, y, z; int r1, r2, r3, rb; };
  Packed pF, pF2, pHx, pHy, pFj;
  auto rows = [&](const Packed& pk, int64_t r0, int64_t x, int64_t y, int64_t z, int r1, int r2, int r3, int rb) {
    return Rows{pk.p.p + r0 * rowlen, pk.e.p + r0, (int64_t)pk.e.n - r0, x, y, z, r1, r2, r3, rb};
  };
  // W for a run of i and of k: at most ~2 GB
  const int64_t slots_max = std::max<int64_t>(1, (int64_t)(2ll << 30) / (8 * v3));
  int64_t slots = 0;   // the largest run of any j
  for (int64_t j = 0; j < o; ++j) slots = std::max(slots, (o - j) * (j + 1));
  slots = subset ? 1 : std::min(slots, c->t3_kc_override > 0 ? (int64_t)c->t3_kc_override : slots_max);
  const int64_t run = std::min(slots, o);
  // Small systems on the FP64 pipe: an exact-slice product takes 33 us however
  // short, a few us on the pipe while it has little to do (at (H2O)1 1.2 ms for
  // the 30 products, 0.2 on the pipe; at (H2O)2 the pipe would need 6 ms where
  // the slices take 2).  The line is 0.2 ms of the pipe's time.  Others too where
  // the slices of H and of a run of F, beside F and W, leave too little memory:
  // then without F and H, whose parts [d] and [l] are two products each.
  bool small = (double)o * o * o * (double)v3 * Kc < 1e8, split = false;
  size_t mfree = 0, mtotal = 0;
  if (!small) {
    FCC_CUDA(cudaMemGetInfo(&mfree, &mtotal));
    const double slices = (2.0 * rowlen + 4.0) * (2.0 * RH + (double)(2 * run + 1) * v2);
    split = slices > c->tc.scratch_max ||
            slices + 8.0 * ((double)std::max(RF, RH) * Kc + (double)slots * v3) + 2e9 > (double)mfree;
  }
  if (c->t3_form) {
    small = c->t3_form == 1;
    split = c->t3_form == 3;
  }
  const bool pipe = small || split;
  auto pack = [&](const double* src, int64_t d1, int64_t d2, int64_t d3, int64_t s1, int64_t s2, int64_t s3, Packed& dst) {
    PackSpec ps{};
    ps.R = d1 * d2 * d3;
    ps.K = Kc;
    ps.Kp = rowlen;
    ps.rd2 = d2; ps.rd3 = d3; ps.rs1 = s1 * Kc; ps.rs2 = s2 * Kc; ps.rs3 = s3 * Kc;
    ps.kd2 = 1; ps.kd3 = Kc; ps.ks3 = 1;
    pack_oz(src, ps, lv.S, lv.bits, lv.guard, dst.p.p, dst.e.p, s);
  };
  DBuf<double> H, F;
  // with split: (xy|zd) [x][y][z][d] and (ly|xz) [l][y][x][z]
  const int64_t Fk = split ? v : Kc;
  if (split) {
    H.alloc(o * o * o * v);
    einsum(1.0, "Qly,Qxz->lyxz", Boo, Bov, 0.0, rm(H.p, {o, o, o, v}), s);
  } else {
    H.alloc(RH * Kc);
    TView Hv = rm(H.p, {o, o, v, Kc});
    einsum1(1.0, "xyzd->xyzd", t2v, 0.0, slice(Hv, 3, 0, v), s);
    einsum(1.0, "Qly,Qxz->xyzl", Boo, Bov, 0.0, slice(Hv, 3, v, o), s);             // (ly|xz)
  }
  if (!pipe) {
    pHx.alloc(RH, rowlen);
    pHy.alloc(RH, rowlen);
    pack(H.p, o, o, v, o * v, v, 1, pHx);
    pack(H.p, o, o, v, v, o * v, 1, pHy);
    FCC_CUDA(cudaStreamSynchronize(s));
    H.release();
  }
  F.alloc(RF * Fk);
  TView Fv = rm(F.p, {o, v, v, Fk});
  einsum(1.0, "Qia,Qbd->iabd", Bov, Bvv, 0.0, slice(Fv, 3, 0, v), s);             // (xy|zd)
  if (!split) einsum1(-1.0, "xlyz->xyzl", t2v, 0.0, slice(Fv, 3, v, o), s);
  std::vector<Seg> segF, segH;
  if (split) {
    segF = {Seg{F.p, v3, v2, v, 1, v, 1.0}, Seg{c->t2.p, o * v2, v, 1, v2, o, -1.0}};
    segH = {Seg{c->t2.p, o * v2, v2, v, 1, v, 1.0}, Seg{H.p, v, o * v, 1, o * o * v, o, 1.0}};
  } else if (pipe) {
    segF = {Seg{F.p, v2 * Kc, v * Kc, Kc, 1, Kc, 1.0}};
    segH = {Seg{H.p, o * v * Kc, v * Kc, Kc, 1, Kc, 1.0}};
  }
  // The slices of F take four times the memory of F, twice that of the FP64
  // array in either order.  Where they do not fit beside the rest, F stays in
  // FP64 and the rows of a run are packed for each pair of runs (hook: t3_kc).
  if (!pipe) FCC_CUDA(cudaMemGetInfo(&mfree, &mtotal));
  const bool whole = !pipe && c->t3_kc_override <= 0 && 4.0 * (double)RF * (double)rowlen + 6e9 < (double)mfree;
  if (whole) {
    pF.alloc(RF, rowlen);
    pF2.alloc(RF, rowlen);
    pack(F.p, o, v, v, v2, v, 1, pF);
    pack(F.p, o, v, v, v2, 1, v, pF2);
    FCC_CUDA(cudaStreamSynchronize(s));
    F.release();
  }
  c->Wt.alloc(slots * v3);
  if (!whole && !pipe) {
    pF.alloc(run * v2, rowlen);
    pFj.alloc(v2, rowlen);
    pF2.alloc(run * v2, rowlen);
  }
  const int nt = (int)((v + ET - 1) / ET);
  std::vector<TileTri> th;
  for (int a = 0; a < nt; ++a)
    for (int b = 0; b <= a; ++b)
      for (int cc = 0; cc <= b; ++cc) th.push_back(TileTri{(int16_t)a, (int16_t)b, (int16_t)cc, 0});
  const int ntiles = (int)th.size();
  DBuf<TileTri> tiles;
  tiles.alloc(ntiles);
  FCC_CUDA(cudaMemcpyAsync(tiles.p, th.data(), sizeof(TileTri) * ntiles, cudaMemcpyHostToDevice, s));
  DBuf<double> part, out;
  part.alloc(o * o * ntiles);
  out.alloc(1);
  part.zero(s);

  // One product: rows m of A (packed rows ar0..), columns n of B (br0..), each a
  // three-level index with the given strides in W
  struct Ix3 { int64_t d2, d3, s1, s2, s3; };
  auto product = [&](bool a_is_f, Rows a, int64_t M, Ix3 m, Rows b, int64_t N, Ix3 nn, double beta, int64_t batch,
                     int64_t ba, int64_t bb, int64_t bc) {
    EpiMap ep;
    ep.M = M; ep.N = N;
    ep.md2 = m.d2; ep.md3 = m.d3; ep.ms1 = m.s1; ep.ms2 = m.s2; ep.ms3 = m.s3;
    ep.nd2 = nn.d2; ep.nd3 = nn.d3; ep.ns1 = nn.s1; ep.ns2 = nn.s2; ep.ns3 = nn.s3;
    ep.beta = beta;
    ep.C = c->Wt.p;
    ep.batch = (int)batch; ep.ba = ba; ep.bb = bb; ep.bc = bc;
    if (pipe) {
      for (size_t q = 0; q < segF.size(); ++q) {
        const Seg &sa = a_is_f ? segF[q] : segH[q], &sb = a_is_f ? segH[q] : segF[q];
        auto at = [](const Seg& g, const Rows& r) { return g.p + r.x * g.sx + r.y * g.sy + r.z * g.sz; };
        auto stride = [](const Seg& g, int r) { return r == 0 ? g.sx : (r == 1 ? g.sy : (r == 2 ? g.sz : 0)); };
        CtrDesc d{};
        d.M = M; d.M2 = m.d2; d.M3 = m.d3; d.N = N; d.N2 = nn.d2; d.N3 = nn.d3; d.K = d.K2 = sa.K; d.batch = batch;
        d.a_m1 = stride(sa, a.r1); d.a_m2 = stride(sa, a.r2); d.a_m3 = stride(sa, a.r3); d.a_k2 = sa.ks;
        d.b_n1 = stride(sb, b.r1); d.b_n2 = stride(sb, b.r2); d.b_n3 = stride(sb, b.r3); d.b_k2 = sb.ks;
        d.c_m1 = m.s1; d.c_m2 = m.s2; d.c_m3 = m.s3; d.c_n1 = nn.s1; d.c_n2 = nn.s2; d.c_n3 = nn.s3;
        d.a_b = batch > 1 && ba ? stride(sa, a.rb) : 0;
        d.b_b = batch > 1 && bb ? stride(sb, b.rb) : 0;
        d.c_b = bc;
        d.alpha = sa.a * sb.a;
        d.beta = q == 0 ? beta : 1.0;
        contract_f64_launch(at(sa, a), at(sb, b), c->Wt.p, d, s);
      }
      return;
    }
    ep.work = 2.0 * (double)batch * (double)M * (double)N * (double)Kc * oz_pairs(lv);
    gemm_oz(a.p, a.n, a.e, b.p, b.n, b.e, Kpad, lv, ep, c->tc.ozws, c->tc.err, s);
  };
  // W[i][k][a][b][c] for i in [i0, i0 + ni), k in [k0, k0 + nk) and one j
  auto build_w = [&](int64_t i0, int64_t ni, int64_t j, int64_t k0, int64_t nk) {
    const int64_t ws = nk * v3;   // stride of i
    if (!whole && !pipe) {
      pack(F.p + i0 * v2 * Kc, ni, v, v, v2, v, 1, pF);
      pack(F.p + j * v2 * Kc, 1, v, v, v2, v, 1, pFj);
      pack(F.p + k0 * v2 * Kc, nk, v, v, v2, 1, v, pF2);
    }
    // F[i] and F[j] by (x, y, z), F[k] by (x, z, y)
    const Rows fi = rows(pF, whole ? i0 * v2 : 0, i0, 0, 0, 0, 1, 2, -1);
    const Rows fj = rows(whole || pipe ? pF : pFj, whole ? j * v2 : 0, j, 0, 0, 0, 1, 2, -1);
    const Rows fk = rows(pF2, whole ? k0 * v2 : 0, k0, 0, 0, 0, 2, 1, -1);
    // H[x][y] over a run of x or of y (the second row level) and z
    auto h = [&](const Packed& ph, int64_t first, int64_t x, int64_t y, int r2, int rb) {
      return rows(ph, first * v, x, y, 0, -1, r2, 2, rb);
    };
    const Rows hk = h(pHy, j * o + k0, k0, j, 0, -1);          // H[k..][j]
    const Rows hki = h(pHy, i0 * o + k0, k0, i0, 0, 1);        // H[k..][i]
    const Rows hji = h(pHx, j * o + i0, j, i0, 1, -1), hjk = h(pHx, j * o + k0, j, k0, 1, -1);
    const Rows hij = h(pHy, j * o + i0, i0, j, 0, -1), hik = h(pHx, i0 * o + k0, i0, k0, 1, 0);
    // F[i](a,b) H[k][j](c): rows (i,a,b), columns (k,c)
    product(true, fi, ni * v2, {v, v, ws, v2, v}, hk, nk * v, {nk, v, 0, v3, 1}, 0.0, 1, 0, 0, 0);
    // F[j](b,a) H[k][i](c): rows (b,a), columns (k,c), a product per i
    product(true, fj, v2, {v, v, 0, v, v2}, hki, nk * v, {nk, v, 0, v3, 1}, 1.0, ni, 0, o * v, ws);
    // H[j][i](b) F[k](c,a): rows (i,b), columns (k,a,c)
    product(false, hji, ni * v, {ni, v, 0, ws, v}, fk, nk * v2, {v, v, v3, v2, 1}, 1.0, 1, 0, 0, 0);
    // H[j][k](b) F[i](a,c): rows (k,b), columns (i,a,c)
    product(false, hjk, nk * v, {nk, v, 0, v3, v}, fi, ni * v2, {v, v, ws, v2, 1}, 1.0, 1, 0, 0, 0);
    // H[i][j](a) F[k](c,b): rows (i,a), columns (k,b,c)
    product(false, hij, ni * v, {ni, v, 0, ws, v2}, fk, nk * v2, {v, v, v3, v, 1}, 1.0, 1, 0, 0, 0);
    // H[i][k](a) F[j](b,c): rows (k,a), columns (b,c), a product per i
    product(false, hik, nk * v, {nk, v, 0, v3, v2}, fj, v2, {v, v, 0, v, 1}, 1.0, ni, o * v, 0, ws);
  };
  auto energy = [&](int64_t i0, int64_t ni, int64_t j, int64_t k0, int64_t nk) {
    const int pe = prof_begin(s);
    dim3 g((unsigned)ntiles, (unsigned)(ni * nk));
    triples_energy_f64_kernel<<<g, EB, 0, s>>>(c->Wt.p, tiles.p, ntiles, c->t1.p, c->ovov.p, c->eps.p, (int)o, (int)v,
                                               (int)i0, (int)j, (int)k0, (int)nk, part.p);
    FCC_CHECK_LAUNCH();
    prof_end(s, pe, PROF_TRIPLES, (double)ni * (double)nk * (double)v * (v + 1) * (v + 2) / 6.0);
  };
  if (subset) {
    // one triplet at a time, each energy read separately
    each->assign(subset->size(), 0.0);
    for (size_t q = 0; q < subset->size(); ++q) {
      const int3 t = (*subset)[q];
      part.zero(s);
      build_w(t.x, 1, t.y, t.z, 1);
      energy(t.x, 1, t.y, t.z, 1);
      sum_kernel<<<1, 1024, 0, s>>>(part.p, (int)(o * o * ntiles), out.p);
      FCC_CHECK_LAUNCH();
      FCC_CUDA(cudaMemcpyAsync(&(*each)[q], out.p, sizeof(double), cudaMemcpyDeviceToHost, s));
    }
    FCC_CUDA(cudaStreamSynchronize(s));
  } else {
    for (int64_t j = 0; j < o; ++j) {
      const int64_t nk = std::min<int64_t>(j + 1, slots);
      const int64_t ni = std::min<int64_t>({std::max<int64_t>(1, slots / nk), 32768 / nk, o});
      for (int64_t k0 = 0; k0 <= j; k0 += nk)
        for (int64_t i0 = j; i0 < o; i0 += ni) {
          const int64_t kk = std::min(nk, j + 1 - k0), ii = std::min(ni, o - i0);
          if (ii == 1 && i0 == j && k0 == j) continue;   // i = j = k only: weight 0
          build_w(i0, ii, j, k0, kk);
          energy(i0, ii, j, k0, kk);
        }
    }
  }
  sum_kernel<<<1, 1024, 0, s>>>(part.p, (int)(o * o * ntiles), out.p);
  FCC_CHECK_LAUNCH();
  double et = 0.0;
  FCC_CUDA(cudaMemcpyAsync(&et, out.p, sizeof(double), cudaMemcpyDeviceToHost, s));
  check_device_error(c, "(T)");
  c->Wt.release();
  return subset ? 0.0 : et;
}

}  // namespace fcc
