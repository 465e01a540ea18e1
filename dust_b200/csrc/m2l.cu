// m2l.cu -- batched multipole-to-local translation (levels >= 2).
//
// M2L_multipole (src/fmm/mod_multipole.f90:282-356) in the form
//   g(m') = (-1)^|m'| / m'!  sum_n  Dhat(m'+n) x ahat(n),  |m'| <= p+1,
// Dhat = k! D(k) of compute_der_ker (:388-450), ahat(n) = a(n)/n!.
//
// Scalar form.  The vector kernel of compute_der_ker is a gradient: with
// Shat(j) = d^j phi the plain derivatives of the scalar kernel
// phi = 1 / (4 pi sqrt(r^2 + delta^2)), Dhat(k)_c = -Shat(k + e_c), so
//   (sum_n Dhat(m'+n) x ahat(n))_x = L_y(m'+e_z) - L_z(m'+e_y)   (and cyclic),
//   L_c(j) = sum_n Shat(j+n) ahat_c(n),   1 <= |j| <= p+2 (p+1 without
// stretching): three scalar sums per offset replace the cross products.
//
// The targets of a level are the non-empty active cells, grouped by their
// position in the parent (octant class q = key & 7): all targets of one class
// share the same 189 interaction offsets (children of the parent's 26
// neighbours that are not adjacent, mod_octree.f90:440-476).  For one offset
// L is a matrix product, (target, component) x n times n x j with the second
// factor Shat(j+n) shared by every target, and runs on the FP64 tensor
// instruction (details at k_m2l_batch).
//
// Scaling: with h the cell size of the level, the tables hold
// Shat(s) h^(|s|+1) and the sources a(n) / (n! h^|n|), so both stay of order
// one at every level and degree; the output is rescaled by h^-(|m'|+2).
//
// Both precisions run the same FP64 kernel: FP64 products at the tensor
// instruction's rate are faster than FP32 ones through shared memory were.
#include <cub/cub.cuh>

#include <algorithm>
#include <cstring>
#include <vector>

#include "dust_common.cuh"
#include "fmm_internal.h"
#include "tc_common.cuh"

#define M2L_NOFF 189     // interaction offsets of an octant class
#define M2L_OFFS 192     // row length of the offset table
#define M2L_NST 2        // stages of the copy pipeline
#define M2L_MAXW 12      // computing warps
#define M2L_SM (224 * 1024)  // shared memory of an SM's CTAs
#define M2L_MINB 14          // least targets of a batch with several CTAs per SM

// ksteps of 4 source monomials, and their padded count, of degree p
__host__ __device__ constexpr int m2l_ks(int p) { return ((p + 1) * (p + 2) * (p + 3) / 6 + 3) / 4; }
// j-tiles (8 indices j) that a warp carries together: as many as keep the
// table fragments (JT * ks doubles) in registers
__host__ __device__ constexpr int m2l_jt(int ks) { return ks <= 9 ? 3 : ks <= 14 ? 2 : 1; }
// targets of a unit (3 rows each, so whole row tiles): more of them share one
// gather of the table fragments, while the stages leave room for the sums
__host__ __device__ constexpr int m2l_tcx(int ks) { return ks <= 9 ? 16 : 8; }
// row stride of a staged source row in doubles: = 4 or 12 mod 16, so that the
// 4 rows x 4 monomials that a half-warp reads fall into distinct banks
__host__ __device__ constexpr int m2l_rs(int kp) { return (kp % 16 == 4 || kp % 16 == 12) ? kp : kp + 4; }

struct M2LArgs {
  const double *tab[DUST_MAXLEV + 1];  // per-level dimensionless tables
  const double *ahat;                  // scaled sources [cell][3][rs]
  const uint32_t *srcix;               // active cell index of a non-empty active cell, else ~0
  const uint16_t *offs;                // [8][M2L_OFFS] table row of each offset
  const uint2 *jix;                    // [group][ks][lane] positions of j + n (4 x u16)
  uint32_t c0;                         // active index of ahat's first cell
  int NB, NJT, nJ, P, OS, jix_smem;
};

__device__ __forceinline__ void dmma884(double (&c)[2], double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
      : "+d"(c[0]), "+d"(c[1])
      : "d"(a), "d"(b));
}
// J j-tiles (first jt0) of the rows of one staged chunk: acc += A B
template <int KS, int J>
__device__ __forceinline__ void m2l_tiles(const double *sA, const double *sT, const uint2 *jix,
                                          const int *tgt, int k, int jt0, int JP, int lane,
                                          double *s_acc) {
  constexpr int RS = m2l_rs(4 * KS);
  double b[J][KS];
#pragma unroll
  for (int q = 0; q < KS; ++q) {
    const uint2 w = jix[q * 32 + lane];
    b[0][q] = sT[w.x & 0xffffu];
    if constexpr (J > 1) b[1][q] = sT[w.x >> 16];
    if constexpr (J > 2) b[2][q] = sT[w.y & 0xffffu];
  }
  const double *ap = sA + (lane >> 2) * RS + (lane & 3);
  double *cp = s_acc + jt0 * 8 + 2 * (lane & 3);
  for (int r = lane >> 2; r - (lane >> 2) < 3 * k; r += 8, ap += 8 * RS) {
    const int x = r / 3;
    const int ro = x < k ? (tgt[x] * 3 + r - 3 * x) * JP : -1;
    double a[KS];
#pragma unroll
    for (int q = 0; q < KS; ++q) a[q] = ap[4 * q];
    double c[J][2];
#pragma unroll
    for (int j = 0; j < J; ++j) {
      c[j][0] = c[j][1] = 0.0;
      if (ro >= 0) {
        const double2 v = *(const double2 *)(cp + ro + 8 * j);
        c[j][0] = v.x;
        c[j][1] = v.y;
      }
    }
#pragma unroll
    for (int q = 0; q < KS; ++q) {
#pragma unroll
      for (int j = 0; j < J; ++j) dmma884(c[j], a[q], b[j][q]);
    }
    if (ro >= 0) {
#pragma unroll
      for (int j = 0; j < J; ++j)
        *(double2 *)(cp + ro + 8 * j) = make_double2(c[j][0], c[j][1]);
    }
  }
}

// One CTA per batch descriptor (level, class, first target, count <= NB <= 32)
// and share blockIdx.y of the 189 offsets (every OS-th; OS > 1 only where the
// batches alone would leave SMs idle).  The batches of all levels >= 2 run in
// one launch (M2L of different levels is independent; L2L follows).
//
// The last warp feeds the others.  Lane i looks up target i's source at each
// offset (four offsets' loads in flight), and for every offset the present
// ones go out in units of up to TCX targets: one bulk copy per source
// (3 rows, one per component, of RS doubles) and one of the offset's scalar
// table into one of M2L_NST stages, an mbarrier each for full and empty.
// A unit's rows are the M of the product, 3 per target without gaps, in
// tiles of 8; each computing warp owns j-tiles (N): it gathers their table
// values for all n into registers, once per unit, through the index table
// jix, and adds every row tile's product to the FP64 sums L_c(j) of the
// targets in shared memory (one 16-byte load and store per lane, row tile and
// j-tile; no other warp touches these columns).  All warps read the same A
// rows, a row fragment of 8 bytes per lane serving J multiplications.
//
// Bound: the FP64 tensor rate.  At p = 4, 9 x 11 multiplications of 8 x 8 x 4
// per 8 rows, 16 cycles each on a sub-core (37 TFLOP/s measured for the bare
// instruction).  Three CTAs of small batches per SM rather than one of a
// large batch, so that one's waits (gather, stage, row sums) are filled by
// another; two stages are enough then.  Measured against the SIMT tile kernel
// this replaces (FP64 / FP32 forms, sums added with shared-memory atomics):
// p = 4, 110k particles (1.69M pairs) 4.45 -> 1.43 ms; 1.1M particles (20.6M
// pairs) FP32 form 23.0 -> 14.8 ms (0.72 of the instruction's rate); p = 6,
// 40k particles 13.8 -> 2.2 ms; p = 4, 3,000 particles 335 -> 76 us.
template <int KS, int JT>
__global__ void __launch_bounds__((M2L_MAXW + 1) * 32)
    k_m2l_batch(FmmDev d, const int4 *batches, const uint32_t *list, M2LArgs A) {
  extern __shared__ __align__(16) unsigned char smraw[];
  constexpr int RS = m2l_rs(4 * KS), TCX = m2l_tcx(KS);
  const int4 bd = batches[blockIdx.x];
  const int l = bd.x, q = bd.y, t0 = bd.z, cnt = bd.w;
  const int NB = A.NB, JP = 8 * A.NJT, P = A.P, OS = A.OS;
  const int nthr = blockDim.x, NW = (nthr >> 5) - 1;
  const int nv = (M2L_NOFF - (int)blockIdx.y + OS - 1) / OS;
  const int ngrp = (A.NJT + JT - 1) / JT;
  const int stage_n = TCX * 3 * RS + P;
  double *s_acc = (double *)smraw;                           // NB x 3 x JP
  double *s_stg = s_acc + (size_t)NB * 3 * JP;               // stages: rows, table
  uint2 *s_jx = (uint2 *)(s_stg + M2L_NST * (size_t)stage_n);  // optional index table
  const size_t jxn = A.jix_smem ? (size_t)ngrp * KS * 32 : 0;
  const uint2 *jix = A.jix_smem ? s_jx : A.jix;
  __shared__ __align__(8) uint64_t s_full[M2L_NST], s_empty[M2L_NST];
  __shared__ int s_tgt[M2L_NST][TCX], s_cnt[M2L_NST], s_fail;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int e = tid; e < NB * 3 * JP; e += nthr) s_acc[e] = 0.0;
  for (int e = tid; e < (int)jxn; e += nthr) s_jx[e] = A.jix[e];
  if (tid == 0) {
    s_fail = 0;
    for (int s = 0; s < M2L_NST; ++s) {
      mbar_init(&s_full[s], 1);
      mbar_init(&s_empty[s], NW);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  __syncthreads();
  if (warp == NW) {
    int ti = -1000, tj = -1000, tk = -1000;
    if (lane < cnt) cart_of_key(d.G, l, d.act_key[list[t0 + lane]], ti, tj, tk);
    const uint32_t *six = A.srcix + d.G.lev_off[l];
    const uint16_t *offs = A.offs + q * M2L_OFFS + blockIdx.y;
    auto lookup = [&](int v, int &tab) {
      uint32_t s = ~0u;
      tab = v < nv ? offs[v * OS] : 0;
      const int si = ti + tab % 7 - 3, sj = tj + tab / 7 % 7 - 3, sk = tk + tab / 49 - 3;
      if (v < nv && lane < cnt && cart_in(d.G, l, si, sj, sk)) s = six[key_of(d.G, l, si, sj, sk)];
      return s;
    };
    unsigned npairs = 0;
    int u = 0;  // units issued
    bool ok = true;
    uint32_t sn[4];
    int tn[4];
#pragma unroll
    for (int g = 0; g < 4; ++g) sn[g] = lookup(g, tn[g]);
    for (int vb = 0; ok && vb < nv; vb += 4) {
      uint32_t sc[4];
      int tc[4];
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        sc[g] = sn[g], tc[g] = tn[g];
        sn[g] = lookup(vb + 4 + g, tn[g]);
      }
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const unsigned m = __ballot_sync(0xffffffffu, sc[g] != ~0u);
        const int np = __popc(m), rank = __popc(m & ((1u << lane) - 1u));
        npairs += np;
        for (int c = 0; ok && c < np; c += TCX, ++u) {
          const int st = u % M2L_NST, k = min(np - c, TCX), slot = rank - c;
          if (u >= M2L_NST)
            ok = mbar_wait_f(smem_u32(&s_empty[st]), (u / M2L_NST - 1) & 1, &s_fail);
          ok = __all_sync(0xffffffffu, ok);
          if (!ok) break;
          double *sA = s_stg + (size_t)st * stage_n;
          const bool in = sc[g] != ~0u && slot >= 0 && slot < k;
          if (in) s_tgt[st][slot] = lane;
          if (lane == 0) s_cnt[st] = k;
          __syncwarp();
          if (lane == 0) {
            mbar_expect_tx(&s_full[st], (uint32_t)(k * 3 * RS + P) * 8);
            bulk_g2s(smem_u32(sA + TCX * 3 * RS), A.tab[l] + (size_t)tc[g] * P, P * 8,
                     &s_full[st]);
          }
          __syncwarp();
          if (in)
            bulk_g2s(smem_u32(sA + slot * 3 * RS), A.ahat + (size_t)(sc[g] - A.c0) * 3 * RS,
                     3 * RS * 8, &s_full[st]);
        }
      }
    }
    if (lane == 0) {
      if (ok && u >= M2L_NST)
        ok = mbar_wait_f(smem_u32(&s_empty[u % M2L_NST]), (u / M2L_NST - 1) & 1, &s_fail);
      if (ok) {  // an empty unit ends the computing warps
        s_cnt[u % M2L_NST] = 0;
        mbar_arrive(&s_full[u % M2L_NST]);
      } else {  // gave up: let the copies in flight land before the CTA ends
        for (int w = max(0, u - M2L_NST); w < u; ++w)
          mbar_wait(smem_u32(&s_full[w % M2L_NST]), (w / M2L_NST) & 1);
      }
      if (npairs && d.counters)
        atomicAdd((unsigned long long *)d.counters, (unsigned long long)npairs);
    }
  } else {
    for (int u = 0;; ++u) {
      const int st = u % M2L_NST;
      if (!mbar_wait_f(smem_u32(&s_full[st]), (u / M2L_NST) & 1, &s_fail)) break;
      const int k = s_cnt[st];
      if (k == 0) break;
      const double *sA = s_stg + (size_t)st * stage_n, *sT = sA + TCX * 3 * RS;
      for (int g = warp; g < ngrp; g += NW) {
        const uint2 *jg = jix + (size_t)g * KS * 32;
        const int nj = A.NJT - g * JT;
        if (nj >= JT)
          m2l_tiles<KS, JT>(sA, sT, jg, s_tgt[st], k, g * JT, JP, lane, s_acc);
        else if (JT > 2 && nj == 2)
          m2l_tiles<KS, (JT > 2 ? 2 : 1)>(sA, sT, jg, s_tgt[st], k, g * JT, JP, lane, s_acc);
        else
          m2l_tiles<KS, 1>(sA, sT, jg, s_tgt[st], k, g * JT, JP, lane, s_acc);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&s_empty[st]);
    }
  }
  __syncthreads();
  if (s_fail) {
    if (tid == 0 && d.counters) d.counters[2] = 1;
    return;
  }
  // outputs: (sum_n Dhat(m'+n) x ahat(n)) from the L_c(j), rescaled
  const int nm = d.nm, nout = d.use_vs ? d.nm1 : d.nm;
  const double hi = 1.0 / d.G.csize[l];
  for (int e = tid; e < cnt * nout; e += nthr) {
    const int t = e / nout, mo = e - t * nout;
    int oi, oj, ok;
    mono_exp(mo, oi, oj, ok);
    double sc = (((oi + oj + ok) & 1) ? -1.0 : 1.0) * d.inv_fact[mo];
    for (int x = 0; x < oi + oj + ok + 2; ++x) sc *= hi;
    const double *Lx = s_acc + (size_t)t * 3 * JP, *Ly = Lx + JP, *Lz = Ly + JP;
    const int jx = mono_idx(oi + 1, oj, ok) - 1, jy = mono_idx(oi, oj + 1, ok) - 1,
              jz = mono_idx(oi, oj, ok + 1) - 1;
    const double g[3] = {sc * (Ly[jz] - Lz[jy]), sc * (Lz[jx] - Lx[jz]), sc * (Lx[jy] - Ly[jx])};
    const uint32_t ci = list[t0 + t];
    double *gx = d.Gx + (size_t)ci * 3 * d.nm1 + 3 * mo, *bb = d.B + (size_t)ci * 3 * nm + 3 * mo;
    for (int x = 0; x < 3; ++x) {
      if (OS == 1) {
        if (d.use_vs) gx[x] += g[x];
        if (mo < nm) bb[x] += g[x];
      } else {  // several CTAs share the target
        if (d.use_vs) atomicAdd(gx + x, g[x]);
        if (mo < nm) atomicAdd(bb + x, g[x]);
      }
    }
  }
}

// class keys of the active cells of levels >= 2: (level << 3 | key & 7) for
// non-empty cells and for empty leaves that hold evaluation points, 0xff for
// the other empty ones (dropped)
__global__ void k_m2l_keys(FmmDev d, uint32_t c0, uint32_t nact, uint32_t *keys,
                           uint32_t *vals, int *hist) {
  uint32_t ci = c0 + blockIdx.x * blockDim.x + threadIdx.x;
  if (ci >= nact) return;
  int l = d.act_lev[ci];
  uint32_t key = d.act_key[ci];
  int sh = 3 * (d.G.ll - l);
  bool ne = d.cstart[(key + 1u) << sh] > d.cstart[key << sh] ||
            (d.flags[d.G.lev_off[l] + key] & FL_PTS);
  uint32_t k = ne ? (uint32_t)((l << 3) | (key & 7)) : 0xffu;
  keys[ci - c0] = k;
  vals[ci - c0] = ci;
  if (ne) atomicAdd(hist + k, 1);
}

static inline unsigned nblk(size_t n, int t) { return (unsigned)((n + t - 1) / t); }

int m2l_batch_tables(dust_octree *o) {
  // dimensionless scalar tables T(s) = Shat(s) h^(|s|+1), |s| <= 2p+2, read
  // off the vector tables: Dhat(k)_c h^(|k|+2) = -Shat(k + e_c) h^(|k+e_c|+1).
  // Entry 0 (s = 0, never used by a sum) is zero: the index table points the
  // padding of j and n there.
  const int p = o->p, nD = o->nD;
  const int nS = n_mon(2 * p + 2);
  const int P = (nS + 1) / 2 * 2;
  const int jmax = o->prm.vortstretch ? p + 2 : p + 1;
  const int nJ = n_mon(jmax) - 1, nm = n_mon(p);
  const int KS = m2l_ks(p), JT = m2l_jt(KS), NJT = (nJ + 7) / 8, ngrp = (NJT + JT - 1) / JT;
  o->m2l_nJ = nJ;
  o->m2l_P = P;
  std::vector<int> deg(nD);
  for (int q = 0; q < nD; ++q) {
    int i, j, k;
    mono_exp(q, i, j, k);
    deg[q] = i + j + k;
  }
  // source of entry s: (vector entry s - e_c, component c) for the first c
  // with s_c >= 1
  std::vector<int> sq(nS, -1), scomp(nS, 0);
  for (int s = 1; s < nS; ++s) {
    int i, j, k;
    mono_exp(s, i, j, k);
    if (i >= 1) sq[s] = mono_idx(i - 1, j, k), scomp[s] = 0;
    else if (j >= 1) sq[s] = mono_idx(i, j - 1, k), scomp[s] = 1;
    else sq[s] = mono_idx(i, j, k - 1), scomp[s] = 2;
  }
  for (int l = 2; l <= o->G.ll; ++l) {
    const size_t n = (size_t)343 * nD * 3, nt = (size_t)343 * P;
    DUST_TRY(devbuf_grow(o->dtabs[l], nt * 8));
    std::vector<double> h(n), t64(nt, 0.0);
    DUST_CUDA(cudaMemcpy(h.data(), o->dtab[l].p, n * 8, cudaMemcpyDeviceToHost));
    const double cs = o->G.csize[l];
    std::vector<double> hp(2 * DUST_MAXP + 6, 1.0);
    for (size_t e = 1; e < hp.size(); ++e) hp[e] = hp[e - 1] * cs;
    for (size_t off = 0; off < 343; ++off)
      for (int s = 1; s < nS; ++s) {
        const int q = sq[s];
        t64[off * P + s] = -h[(off * nD + q) * 3 + scomp[s]] * hp[deg[q] + 2];
      }
    DUST_CUDA(cudaMemcpy(o->dtabs[l].p, t64.data(), nt * 8, cudaMemcpyHostToDevice));
  }
  // jix[group][k][lane] (4 x u16): table positions of j + n for the group's
  // j-tiles, j index 8 jt + lane / 4 and n = 4 k + lane % 4; then the offsets
  // of the 8 octant classes
  std::vector<uint16_t> js((size_t)ngrp * KS * 32 * 4 + 8 * M2L_OFFS, 0);
  for (int jt = 0; jt < NJT; ++jt)
    for (int k = 0; k < KS; ++k)
      for (int lane = 0; lane < 32; ++lane) {
        const int jj = 8 * jt + lane / 4, nn = 4 * k + lane % 4;
        if (jj >= nJ || nn >= nm) continue;
        int ji, jj2, jk, ni, nj, nk;
        mono_exp(jj + 1, ji, jj2, jk);
        mono_exp(nn, ni, nj, nk);
        js[(((size_t)(jt / JT) * KS + k) * 32 + lane) * 4 + jt % JT] =
            (uint16_t)mono_idx(ji + ni, jj2 + nj, jk + nk);
      }
  uint16_t *of = js.data() + (size_t)ngrp * KS * 32 * 4;
  for (int q = 0; q < 8; ++q) {
    int v = 0;
    for (int c = 0; c < 216; ++c) {
      const int ox = c % 6 - 2 - (q & 1), oy = c / 6 % 6 - 2 - (q >> 1 & 1),
                oz = c / 36 - 2 - (q >> 2 & 1);
      if (std::abs(ox) <= 1 && std::abs(oy) <= 1 && std::abs(oz) <= 1) continue;
      of[q * M2L_OFFS + v++] = (uint16_t)((ox + 3) + 7 * ((oy + 3) + 7 * (oz + 3)));
    }
  }
  DUST_TRY(devbuf_grow(o->jsum, js.size() * 2));
  DUST_CUDA(cudaMemcpy(o->jsum.p, js.data(), js.size() * 2, cudaMemcpyHostToDevice));
  return DUST_OK;
}

// Sorts the targets of levels >= 2 (level 1 is handled by the per-target
// kernel) by level and octant class.
int m2l_prepare(dust_octree *o, FmmDev &d, cudaStream_t st) {
  const int ll = o->G.ll;
  uint32_t c0 = (uint32_t)o->act_off[2 <= ll ? 2 : ll + 1];
  uint32_t nact = (uint32_t)o->n_active;
  uint32_t m = nact > c0 ? nact - c0 : 0;
  o->m2l_list = nullptr;
  memset(o->m2l_cnt, 0, sizeof(o->m2l_cnt));
  if (m == 0) return DUST_OK;
  DUST_TRY(devbuf_grow(o->m2l_buf, (size_t)m * 16 + 4096));
  uint32_t *k_in = (uint32_t *)o->m2l_buf.p, *v_in = k_in + m, *k_out = v_in + m,
           *v_out = k_out + m;
  int *hist = (int *)(v_out + m);
  DUST_CUDA(cudaMemsetAsync(hist, 0, 256 * sizeof(int), st));
  k_m2l_keys<<<nblk(m, 256), 256, 0, st>>>(d, c0, nact, k_in, v_in, hist);
  size_t tb = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, tb, k_in, k_out, v_in, v_out, (int)m, 0, 8, st);
  DUST_TRY(devbuf_grow(o->cub_tmp, tb));
  DUST_CUDA(cub::DeviceRadixSort::SortPairs(o->cub_tmp.p, tb, k_in, k_out, v_in, v_out, (int)m,
                                            0, 8, st));
  int h[256];
  DUST_CUDA(cudaMemcpyAsync(h, hist, sizeof(h), cudaMemcpyDeviceToHost, st));
  DUST_CUDA(cudaStreamSynchronize(st));
  memcpy(o->m2l_cnt, h, sizeof(int) * 8 * (DUST_MAXLEV + 1));
  o->m2l_list = v_out;
  // scaled source coefficients of the active cells of levels >= 2, written by
  // the upward pass beside the multipoles (put_multipole)
  DUST_TRY(devbuf_grow(o->ahat, (size_t)m * 3 * m2l_rs(4 * m2l_ks(o->p)) * 8 + 256));
  o->ahat_c0 = c0;
  d.ahat = (double *)o->ahat.p;
  d.ahat_c0 = c0;
  d.ahat_rs = m2l_rs(4 * m2l_ks(o->p));
  return DUST_OK;
}

template <int P_>
static int m2l_launch(const dim3 &grid, int NW, size_t sm, cudaStream_t st, FmmDev &d,
                      const dust_octree *o, const M2LArgs &A) {
  constexpr int KS = m2l_ks(P_), JT = m2l_jt(KS);
  if (sm > 48 * 1024)
    DUST_CUDA(cudaFuncSetAttribute(k_m2l_batch<KS, JT>,
                                   cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  k_m2l_batch<KS, JT><<<grid, (NW + 1) * 32, sm, st>>>(d, (const int4 *)o->m2l_bat.p, o->m2l_list, A);
  return DUST_OK;
}

int m2l_all_levels(dust_octree *o, FmmDev &d, cudaStream_t st) {
  if (!o->m2l_list) return DUST_OK;
  const int KS = m2l_ks(o->p), JT = m2l_jt(KS), RS = m2l_rs(4 * KS), TCX = m2l_tcx(KS);
  M2LArgs A;
  A.nJ = o->m2l_nJ;
  A.NJT = (A.nJ + 7) / 8;
  A.P = o->m2l_P;
  const int ngrp = (A.NJT + JT - 1) / JT;
  // every group of j-tiles its own warp, or shares as even as possible
  const int rounds = (ngrp + M2L_MAXW - 1) / M2L_MAXW, NW = (ngrp + rounds - 1) / rounds;
  const size_t jxb = (size_t)ngrp * KS * 32 * 8;
  A.jix_smem = jxb <= 16 * 1024;
  int n_tgt = 0;
  for (int k = 16; k < 8 * (DUST_MAXLEV + 1); ++k) n_tgt += o->m2l_cnt[k];
  if (n_tgt == 0) return DUST_OK;
  // targets per batch (up to 32): what three CTAs per SM can hold, unless a
  // batch of so few leaves its row tiles part empty; then two, then one
  const size_t fixed = M2L_NST * ((size_t)TCX * 3 * RS + A.P) * 8 + (A.jix_smem ? jxb : 0);
  const size_t per = (size_t)3 * 8 * A.NJT * 8;
  for (int c = 3; c >= 1; --c) {
    const size_t cap = (M2L_SM - c * 1024) / c;
    A.NB = std::min<int>(32, (int)((cap - std::min(cap, fixed)) / per));
    if (A.NB >= M2L_MINB) break;
  }
  std::vector<int4> bs;
  int start = 0;
  for (int k = 0; k < 8 * (DUST_MAXLEV + 1); ++k) {
    const int c = o->m2l_cnt[k], l = k >> 3, q = k & 7;
    if (l >= 2)
      for (int b = 0; b < c; b += A.NB)
        bs.push_back(make_int4(l, q, start + b, std::min(A.NB, c - b)));
    start += c;
  }
  // share the offsets of a batch among CTAs while the grid is short of about
  // five CTAs per resident slot (444): the 189 offsets of one CTA are a serial
  // chain, and its last wave is nearly empty otherwise.  Against one CTA per
  // batch: 3,000 particles 291 -> 76 us, 110k 1.77 -> 1.52 ms (three times
  // the line: 1.55 ms), 1.1M particles the same.
  A.OS = std::max(1, std::min(16, (int)(2368 / bs.size())));
  DUST_TRY(devbuf_grow(o->m2l_bat, bs.size() * sizeof(int4)));
  DUST_CUDA(cudaMemcpyAsync(o->m2l_bat.p, bs.data(), bs.size() * sizeof(int4),
                            cudaMemcpyHostToDevice, st));
  for (int l = 0; l <= DUST_MAXLEV; ++l)
    A.tab[l] = (l >= 2 && l <= o->G.ll) ? (const double *)o->dtabs[l].p : nullptr;
  A.ahat = (const double *)o->ahat.p;
  A.c0 = o->ahat_c0;
  A.srcix = (const uint32_t *)o->srcix.p;
  A.jix = (const uint2 *)o->jsum.p;
  A.offs = (const uint16_t *)o->jsum.p + (size_t)ngrp * KS * 32 * 4;
  const size_t sm = fixed + A.NB * per;
  const dim3 grid((unsigned)bs.size(), (unsigned)A.OS);
  o->kev_m2l = o->timing;
  if (o->timing) cudaEventRecord(o->ev[6], st);
  switch (o->p) {
    case 0: DUST_TRY(m2l_launch<0>(grid, NW, sm, st, d, o, A)); break;
    case 1: DUST_TRY(m2l_launch<1>(grid, NW, sm, st, d, o, A)); break;
    case 2: DUST_TRY(m2l_launch<2>(grid, NW, sm, st, d, o, A)); break;
    case 3: DUST_TRY(m2l_launch<3>(grid, NW, sm, st, d, o, A)); break;
    case 4: DUST_TRY(m2l_launch<4>(grid, NW, sm, st, d, o, A)); break;
    case 5: DUST_TRY(m2l_launch<5>(grid, NW, sm, st, d, o, A)); break;
    case 6: DUST_TRY(m2l_launch<6>(grid, NW, sm, st, d, o, A)); break;
    case 7: DUST_TRY(m2l_launch<7>(grid, NW, sm, st, d, o, A)); break;
    default: DUST_TRY(m2l_launch<8>(grid, NW, sm, st, d, o, A)); break;
  }
  if (o->timing) cudaEventRecord(o->ev[7], st);
  DUST_CUDA(cudaGetLastError());
  return DUST_OK;
}
