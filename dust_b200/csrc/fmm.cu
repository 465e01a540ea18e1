// fmm.cu -- octree FMM for vortex particles on sm_100a.
//
// Replaces the reference's mod_octree / mod_multipole path
// (src/fmm/mod_octree.f90:251-1429, src/fmm/mod_multipole.f90:224-450) and
// the particle kernels of src/aeroel/mod_vortpart.f90:139-336.
//
// Design (B200-first, not a translation):
//  * particles are binned at the finest level and stably radix-sorted by a
//    hierarchical Morton key, so every cell of every level owns a contiguous
//    particle range (the reference's pointer lists, mod_octree.f90:746-773
//    and 911-961, in the same order);
//  * the reference's leaf rule (npart >= min_octree_part at fixed depth,
//    siblings of leaves become leaves, :896-962) runs over Morton-ordered flag
//    arrays, three levels a launch; active cells and leaves are compacted with
//    one device scan;
//  * multipole data live in compact per-active-cell SoA blocks;
//  * M2L evaluates the degree-(p+1) velocity local expansion g once and
//    derives the reference's gradient coefficients from it exactly,
//    c(r,:,m) = (m_r+1) g(:, m+e_r); the velocity coefficients b (degree p)
//    and g are translated with the reference's own truncations in L2L;
//  * L2P is fused into the leaf-pair P2P kernel: one warp per leaf, or per item
//    of a leaf with a large near field; the near-field source ranges are
//    concatenated into one virtual index space streamed through shared memory in
//    32-particle tiles, lane groups split the sources of small leaves, and their
//    partial sums meet in shared memory.
#include <cub/cub.cuh>
#include <thrust/iterator/transform_iterator.h>
#include <thrust/iterator/transform_output_iterator.h>
#include <thrust/iterator/zip_iterator.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <type_traits>
#include <vector>

#include "dust_common.cuh"
#include "elements.cuh"
#include "fmm_internal.h"
#include "p2p_items.h"

static int build_shift_tables(dust_octree *o);

// ===================================================================== host
static int grow(DevBuf &b, size_t bytes) {
  if (bytes <= b.cap) return DUST_OK;
  if (b.p) cudaFree(b.p);
  b.p = nullptr;
  b.cap = 0;
  size_t want = bytes + bytes / 8 + 256;
  DUST_CUDA(cudaMalloc(&b.p, want));
  b.cap = want;
  return DUST_OK;
}
void devbuf_free(DevBuf &b) {
  if (b.p) cudaFree(b.p);
  b.p = nullptr;
  b.cap = 0;
}
int devbuf_grow(DevBuf &b, size_t bytes) { return grow(b, bytes); }

// compute_der_ker (mod_multipole.f90:388-450) for one offset, returning
// D(3, n_mon(2p+1)) scaled by the multi-index factorial of its monomial.
static void host_der_table(int p, const double diff[3], double delta, double *Dhat) {
  int deg = 2 * p + 2;
  int nm = n_mon(deg);
  std::vector<double> bk(nm, 0.0);
  double R2 = diff[0] * diff[0] + diff[1] * diff[1] + diff[2] * diff[2] + delta * delta;
  for (int k = 0; k <= deg; ++k)
    for (int j = 0; j <= deg - k; ++j)
      for (int i = 0; i <= deg - j - k; ++i) {
        double kmod = (double)(k + j + i);
        if (i == 0 && j == 0 && k == 0) {
          bk[0] = 1.0 / (4.0 * DUST_PI * sqrt(R2));
        } else {
          double s1 = 0.0, s2 = 0.0;
          if (i >= 1) s1 += diff[0] * bk[mono_idx(i - 1, j, k)];
          if (j >= 1) s1 += diff[1] * bk[mono_idx(i, j - 1, k)];
          if (k >= 1) s1 += diff[2] * bk[mono_idx(i, j, k - 1)];
          if (i >= 2) s2 += bk[mono_idx(i - 2, j, k)];
          if (j >= 2) s2 += bk[mono_idx(i, j - 2, k)];
          if (k >= 2) s2 += bk[mono_idx(i, j, k - 2)];
          bk[mono_idx(i, j, k)] =
              1.0 / (R2 * kmod) * ((2.0 * kmod - 1.0) * s1 - (kmod - 1.0) * s2);
        }
      }
  double fact[40];
  fact[0] = 1.0;
  for (int q = 1; q < 40; ++q) fact[q] = fact[q - 1] * q;
  int nD = n_mon(2 * p + 1);
  for (int q = 0; q < nD; ++q) {
    int i, j, k;
    mono_exp(q, i, j, k);
    double f = fact[i] * fact[j] * fact[k];
    Dhat[3 * q + 0] = -(1.0 + i) * bk[mono_idx(i + 1, j, k)] * f;
    Dhat[3 * q + 1] = -(1.0 + j) * bk[mono_idx(i, j + 1, k)] * f;
    Dhat[3 * q + 2] = -(1.0 + k) * bk[mono_idx(i, j, k + 1)] * f;
  }
}

static int build_tables(dust_octree *o) {
  int p = o->p;
  int nD = n_mon(2 * p + 1);
  std::vector<double> tab;
  for (int l = 1; l <= o->G.ll; ++l) {
    int L[3];
    for (int d = 0; d < 3; ++d)
      L[d] = (l == 1) ? std::max(o->G.nbox[d], 3) : 3;
    for (int d = 0; d < 3; ++d) o->kdlen[l][d] = L[d];
    size_t nofs = (size_t)(2 * L[0] + 1) * (2 * L[1] + 1) * (2 * L[2] + 1);
    tab.assign(nofs * nD * 3, 0.0);
    size_t q = 0;
    for (int k = -L[2]; k <= L[2]; ++k)
      for (int j = -L[1]; j <= L[1]; ++j)
        for (int i = -L[0]; i <= L[0]; ++i, ++q)
          if (std::abs(i) >= 2 || std::abs(j) >= 2 || std::abs(k) >= 2) {
            double diff[3] = {o->G.csize[l] * (double)(-i), o->G.csize[l] * (double)(-j),
                              o->G.csize[l] * (double)(-k)};
            host_der_table(p, diff, o->prm.rankine_rad, &tab[q * nD * 3]);
          }
    DUST_TRY(grow(o->dtab[l], tab.size() * sizeof(double)));
    DUST_CUDA(cudaMemcpy(o->dtab[l].p, tab.data(), tab.size() * sizeof(double),
                         cudaMemcpyHostToDevice));
  }
  // index table idxsum[n * nm1 + m'] = mono_idx(m' + n), and scale tables
  int nm = n_mon(p), nm1 = n_mon(p + 1);
  std::vector<uint16_t> isum((size_t)nm * nm1);
  for (int n = 0; n < nm; ++n) {
    int a, b, c;
    mono_exp(n, a, b, c);
    for (int m = 0; m < nm1; ++m) {
      int i, j, k;
      mono_exp(m, i, j, k);
      isum[(size_t)n * nm1 + m] = (uint16_t)mono_idx(i + a, j + b, k + c);
    }
  }
  DUST_TRY(grow(o->idxsum, isum.size() * sizeof(uint16_t)));
  DUST_CUDA(cudaMemcpy(o->idxsum.p, isum.data(), isum.size() * sizeof(uint16_t),
                       cudaMemcpyHostToDevice));
  return DUST_OK;
}

static int geom_init(dust_octree *o) {
  TreeGeom &G = o->G;
  const dust_fmm_params &p = o->prm;
  memset(&G, 0, sizeof(G));
  G.ll = p.n_octree_levels;
  uint64_t off = 0;
  for (int d = 0; d < 3; ++d) {
    G.nbox[d] = p.n_box[d];
    G.xmin[d] = p.origin[d];
    G.xmax[d] = p.origin[d] + (double)p.n_box[d] * p.box_length;
  }
  for (int l = 1; l <= G.ll; ++l) {
    uint64_t nc = 1;
    for (int d = 0; d < 3; ++d) {
      G.ncl[l][d] = p.n_box[d] << (l - 1);
      nc *= (uint64_t)G.ncl[l][d];
    }
    if (nc >= (1ull << 31)) return DUST_ERR_CAPACITY;
    G.ncell[l] = (uint32_t)nc;
    G.lev_off[l] = (uint32_t)off;
    off += nc;
    if (off >= (1ull << 31)) return DUST_ERR_CAPACITY;
    G.csize[l] = (l == 1) ? p.box_length : p.box_length / (double)(1 << (l - 1));
  }
  G.lev_off[G.ll + 1] = (uint32_t)off;
  o->ncell_tot = off;
  return DUST_OK;
}

extern "C" int dust_octree_create(const dust_fmm_params *prm, dust_octree **out) {
  if (!prm || !out) return DUST_ERR_BAD_ARG;
  *out = nullptr;
  if (prm->n_octree_levels < 1 || prm->n_octree_levels > 11 ||
      prm->multipole_degree < 0 || prm->multipole_degree > DUST_MAXP ||
      prm->box_length <= 0.0 || prm->n_box[0] < 1 || prm->n_box[1] < 1 ||
      prm->n_box[2] < 1 || prm->min_octree_part < 0)
    return DUST_ERR_BAD_ARG;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return DUST_ERR_NO_DEVICE;
  dust_octree *o = new dust_octree();
  o->prm = *prm;
  o->p = prm->multipole_degree;
  o->nm = n_mon(o->p);
  o->nm1 = n_mon(o->p + 1);
  o->nD = n_mon(2 * o->p + 1);
  int st = geom_init(o);
  if (st != DUST_OK) {
    delete o;
    return st;
  }
  if (cudaStreamCreateWithFlags(&o->stream, cudaStreamNonBlocking) != cudaSuccess) {
    delete o;
    return DUST_ERR_CUDA;
  }
  for (int e = 0; e < 12; ++e) cudaEventCreate(&o->ev[e]);
  st = build_tables(o);
  if (st == DUST_OK) st = grow(o->small, 64 * 8);
  if (st == DUST_OK && cudaMemset(o->small.p, 0, 64 * 8) != cudaSuccess) st = DUST_ERR_CUDA;
  if (st == DUST_OK) st = build_shift_tables(o);
  if (st == DUST_OK) st = m2l_batch_tables(o);
  if (st != DUST_OK) {
    dust_octree_destroy(o);
    return st;
  }
  *out = o;
  return DUST_OK;
}

extern "C" int dust_octree_destroy(dust_octree *o) {
  if (!o) return DUST_OK;
  cudaStreamSynchronize(o->stream);
  for (int l = 0; l <= DUST_MAXLEV; ++l) {
    devbuf_free(o->dtab[l]);
    devbuf_free(o->dtabs[l]);
  }
  devbuf_free(o->m2l_buf);
  devbuf_free(o->ahat);
  devbuf_free(o->m2l_bat);
  devbuf_free(o->jsum);
  devbuf_free(o->srcix);
  devbuf_free(o->p2p_work);
  devbuf_free(o->shift);
  devbuf_free(o->ffbuf);
  devbuf_free(o->near_buf);
  DevBuf *bufs[] = {&o->idxsum, &o->keys,   &o->keys_s, &o->vals,   &o->perm,
                    &o->cnt,    &o->cstart, &o->part,   &o->flags,
                    &o->cidx,   &o->lidx,   &o->act_key, &o->act_lev, &o->leaf_ci,
                    &o->mp,     &o->outs,   &o->cub_tmp, &o->small,  &o->h_in,
                    &o->h_out,  &o->h_pts,  &o->el_geo, &o->el_raw};
  for (DevBuf *b : bufs) devbuf_free(*b);
  for (int e = 0; e < 12; ++e) cudaEventDestroy(o->ev[e]);
  cudaStreamDestroy(o->stream);
  delete o;
  return DUST_OK;
}

extern "C" int dust_octree_get_stats(const dust_octree *o, dust_fmm_stats *st) {
  if (!o || !st) return DUST_ERR_BAD_ARG;
  *st = o->stats;
  return DUST_OK;
}
extern "C" int dust_octree_set_near_limit(dust_octree *o, long long pairs) {
  if (!o || pairs < 0) return DUST_ERR_BAD_ARG;
  o->near_limit = (size_t)pairs;
  return DUST_OK;
}

extern "C" int dust_octree_set_timing(dust_octree *o, int on) {
  if (!o) return DUST_ERR_BAD_ARG;
  o->timing = on != 0;
  return DUST_OK;
}

// ================================================================== kernels
__global__ void k_bin(int n, const double *__restrict__ cen, TreeGeom G,
                      uint32_t *__restrict__ keys, uint32_t *__restrict__ vals,
                      uint32_t *__restrict__ cnt, int *__restrict__ err) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  int ll = G.ll;
  double csize = G.csize[ll];
  int idx[3];
  bool bad = false;
  for (int d = 0; d < 3; ++d) {
    // idx = ceiling((cen - xmin)/csize) (mod_octree.f90:754)
    double c = ceil((cen[3 * t + d] - G.xmin[d]) / csize);
    if (!(c >= 1.0 && c <= (double)G.ncl[ll][d])) {
      bad = true;
      idx[d] = 1;
    } else {
      idx[d] = (int)c;
    }
  }
  if (bad) {
    atomicMin(err, t);
    keys[t] = 0xffffffffu;
    vals[t] = (uint32_t)t;
    return;
  }
  uint32_t key = key_of(G, ll, idx[0] - 1, idx[1] - 1, idx[2] - 1);
  keys[t] = key;
  vals[t] = (uint32_t)t;
  atomicAdd(&cnt[key], 1u);
}

// sorted SoA particle block: x y z ax ay az sigma (n each)
__global__ void k_gather(int n, const uint32_t *__restrict__ perm,
                         const double *__restrict__ cen, const double *__restrict__ dir,
                         const double *__restrict__ mag, const double *__restrict__ rv,
                         double *__restrict__ P) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= n) return;
  uint32_t ip = perm[t];
  double m = mag[ip];
  for (int d = 0; d < 3; ++d) {
    P[(size_t)d * n + t] = cen[3 * (size_t)ip + d];
    P[(size_t)(3 + d) * n + t] = m * dir[3 * (size_t)ip + d];
  }
  P[(size_t)6 * n + t] = rv[ip];
}

__device__ inline uint32_t cell_lo(const TreeGeom &G, const uint32_t *cstart, int l,
                                   uint32_t key) {
  return cstart[key << (3 * (G.ll - l))];
}
__device__ inline uint32_t cell_hi(const TreeGeom &G, const uint32_t *cstart, int l,
                                   uint32_t key) {
  return cstart[(key + 1u) << (3 * (G.ll - l))];
}

// one upward pass of the leaf rule (mod_octree.f90:911-962) at every
// level, three levels a launch: a CTA takes 512 consecutive cells of level lb (of the
// finest one: `fine`, from the particle counts; else as the launch before left
// them) and the cells above them up to level lt, in shared memory.  (A launch a
// level, six for 3,000 particles: 12 us; for 1,100,000 100 us; 5 and 88 us.)
#define FLG_T 256
#define FLG_C 512
__global__ void __launch_bounds__(FLG_T) k_flags(TreeGeom G, int lb, int lt, bool fine,
                                                 const uint32_t *__restrict__ cstart, int min_part,
                                                 uint8_t *__restrict__ flags) {
  __shared__ uint8_t s_f[FLG_C + FLG_C / 8 + FLG_C / 64 + FLG_C / 512];
  const uint32_t base = blockIdx.x * FLG_C, nb = min((uint32_t)FLG_C, G.ncell[lb] - base);
  for (uint32_t e = threadIdx.x; e < nb; e += FLG_T) {
    const uint32_t key = base + e;
    uint8_t f;
    if (fine) {
      const int np = (int)(cstart[key + 1] - cstart[key]);
      f = (np >= min_part || lb == 1) ? (FL_LEAF | FL_ACTIVE) : 0;
    } else {
      f = flags[G.lev_off[lb] + key];
    }
    s_f[e] = f;
  }
  uint8_t *below = s_f;
  uint32_t m = nb;
  for (int l = lb - 1; l >= lt; --l) {
    uint8_t *here = below + m;
    const uint32_t mu = m >> 3, key0 = base >> (3 * (lb - l));
    __syncthreads();
    for (uint32_t e = threadIdx.x; e < mu; e += FLG_T) {
      uint8_t *ch = below + 8 * e;
      bool got = false;
      for (int c = 0; c < 8; ++c) got |= (ch[c] & (FL_LEAF | FL_BRANCH)) != 0;
      if (got) {
        for (int c = 0; c < 8; ++c)
          if (!(ch[c] & (FL_LEAF | FL_BRANCH))) ch[c] = FL_LEAF | FL_ACTIVE;
        here[e] = FL_BRANCH | FL_ACTIVE;
      } else {
        for (int c = 0; c < 8; ++c) ch[c] = 0;
        const int np = (int)(cell_hi(G, cstart, l, key0 + e) - cell_lo(G, cstart, l, key0 + e));
        here[e] = (np >= min_part || l == 1) ? (FL_LEAF | FL_ACTIVE) : 0;
      }
    }
    below = here;
    m = mu;
  }
  __syncthreads();
  const uint8_t *f = s_f;
  for (int l = lb; l >= lt; --l) {
    const uint32_t ml = nb >> (3 * (lb - l)), key0 = base >> (3 * (lb - l));
    for (uint32_t e = threadIdx.x; e < ml; e += FLG_T) flags[G.lev_off[l] + key0 + e] = f[e];
    f += ml;
  }
}

// Evaluation points (panel centres) sorted into the tree as sort_particles
// sorts the panels (mod_octree.f90:776-799): the leaf above each point's
// finest cell gets FL_PTS, so that an empty leaf that holds a point still
// gets its local expansion (the particles' own M2L skips empty targets).  A
// point outside the box records its index in *err.
__global__ void k_mark_points(TreeGeom G, int npts, const double *__restrict__ pts,
                              uint8_t *__restrict__ flags, int *err) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= npts) return;
  const int ll = G.ll;
  int idx[3];
  for (int c = 0; c < 3; ++c) {
    idx[c] = (int)ceil((pts[3 * (size_t)q + c] - G.xmin[c]) / G.csize[ll]) - 1;
    if (idx[c] < 0 || idx[c] >= G.ncl[ll][c]) {
      atomicMin(err, q);
      return;
    }
  }
  for (int lv = 1; lv <= ll; ++lv) {
    const int sh = ll - lv;
    uint8_t *f = flags + G.lev_off[lv] + key_of(G, lv, idx[0] >> sh, idx[1] >> sh, idx[2] >> sh);
    if (*f & FL_LEAF) {
      *f = *f | FL_PTS;  // every writer stores the same value
      return;
    }
  }
}

// Numbers of the active cells and of the leaves before each cell in one scan of
// their flags: two 32-bit counts in one word.
struct FlagCounts {
  __host__ __device__ uint64_t operator()(uint8_t f) const {
    return ((f & FL_ACTIVE) ? 1ull : 0ull) | ((f & FL_LEAF) ? 1ull << 32 : 0ull);
  }
};
struct SplitCounts {
  __host__ __device__ thrust::tuple<uint32_t, uint32_t> operator()(uint64_t v) const {
    return thrust::make_tuple((uint32_t)v, (uint32_t)(v >> 32));
  }
};

__global__ void k_compact(TreeGeom G, uint32_t ntot, const uint8_t *__restrict__ flags,
                          const uint32_t *__restrict__ cidx,
                          const uint32_t *__restrict__ lidx,
                          const uint32_t *__restrict__ cstart, uint32_t *__restrict__ act_key,
                          uint8_t *__restrict__ act_lev, uint32_t *__restrict__ leaf_ci,
                          uint32_t *__restrict__ srcix) {
  uint32_t c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ntot) return;
  uint8_t f = flags[c];
  if (!(f & FL_ACTIVE)) {
    srcix[c] = ~0u;
    return;
  }
  int l = 1;
  while (l < G.ll && c >= G.lev_off[l + 1]) ++l;
  uint32_t ci = cidx[c];
  const uint32_t key = c - G.lev_off[l];
  // M2L sources: an empty active cell has a = 0
  srcix[c] = cell_hi(G, cstart, l, key) > cell_lo(G, cstart, l, key) ? ci : ~0u;
  act_key[ci] = c - G.lev_off[l];
  act_lev[ci] = (uint8_t)l;
  if (f & FL_LEAF) leaf_ci[lidx[c]] = ci;
}

// per-level active offsets (scan values at level boundaries) + totals
__global__ void k_level_counts(TreeGeom G, const uint32_t *__restrict__ cidx,
                               const uint32_t *__restrict__ lidx, int64_t *__restrict__ out) {
  int l = threadIdx.x + 1;
  if (l <= G.ll + 1) out[l] = cidx[G.lev_off[l]];
  if (threadIdx.x == 0) out[0] = lidx[G.lev_off[G.ll + 1]];
}

// Coefficient m of a cell's multipole (rows m >= nm: the padding of the scaled
// copy) into A and, for the cells that are M2L sources, scaled by 1/(n! h^|n|),
// into ahat as [cell][component][rs].
__device__ __forceinline__ void put_multipole(const FmmDev &d, uint32_t ci, int l, int m,
                                              const double *v) {
  if (m < d.nm) {
    double *a = d.A + (size_t)ci * 3 * d.nm + 3 * m;
    for (int c = 0; c < 3; ++c) a[c] = v[c];
  }
  if (d.ahat && ci >= d.ahat_c0) {
    double f = 0.0;
    if (m < d.nm) {
      int i, j, k;
      mono_exp(m, i, j, k);
      const double hi = 1.0 / d.G.csize[l];
      f = d.inv_fact[m];
      for (int q = 0; q < i + j + k; ++q) f *= hi;
    }
    double *o = d.ahat + (size_t)(ci - d.ahat_c0) * 3 * d.ahat_rs + m;
    for (int c = 0; c < 3; ++c) o[c * d.ahat_rs] = f * v[c];
  }
}

// P2M (leaf_M_multipole, mod_multipole.f90:224-251): one warp per leaf, the
// leaf's particles in chunks of 32: lane t forms the powers of particle t's
// offsets into the warp's shared memory (rows of 33 words: the lanes of a
// product read different rows), then the lanes take the output coefficients m
// and sum the chunk's products in particle order.  (Powers formed per
// coefficient and particle: 31 us for 3,000 particles, 381 us for 1,100,000,
// and 4 and 170 us for the scaled copy; 10 and 208 us together.)
#define P2M_W 4
#define P2M_LD 33
__global__ void __launch_bounds__(P2M_W * 32) k_p2m(FmmDev d) {
  extern __shared__ __align__(16) double p2m_sm[];
  const int w = threadIdx.x >> 5, lane = threadIdx.x & 31, np = d.p + 1;
  const uint32_t leaf = blockIdx.x * P2M_W + w;
  if (leaf >= d.n_leaves) return;  // warp-uniform
  const uint32_t ci = d.leaf_ci[leaf];
  const int l = d.act_lev[ci];
  const uint32_t key = d.act_key[ci];
  const uint32_t lo = cell_lo(d.G, d.cstart, l, key), hi = cell_hi(d.G, d.cstart, l, key);
  if (hi == lo) return;  // empty leaf: a = 0 (block zeroed before the pass)
  int i, j, k;
  cart_of_key(d.G, l, key, i, j, k);
  double c[3];
  cell_center(d.G, l, i, j, k, c);
  const size_t n = d.n;
  double *pw = p2m_sm + (size_t)w * (3 * np + 3) * P2M_LD;  // [axis][power][t], alpha[3][t]
  double *al = pw + 3 * np * P2M_LD;
  const int rs = d.ahat ? d.ahat_rs : d.nm;
  for (int m0 = 0; m0 < rs; m0 += 32) {
    const int m = m0 + lane;
    int mi = 0, mj = 0, mk = 0;
    if (m < d.nm) mono_exp(m, mi, mj, mk);
    const double *px = pw + mi * P2M_LD, *py = pw + (np + mj) * P2M_LD,
                 *pz = pw + (2 * np + mk) * P2M_LD;
    double v[3] = {0.0, 0.0, 0.0};
    for (uint32_t s0 = lo; s0 < hi; s0 += 32) {
      const int cnt = min((int)(hi - s0), 32);
      if (m0 == 0 || hi - lo > 32) {  // (one chunk: its powers stay for every m0)
        __syncwarp();
        if (lane < cnt) {
          const uint32_t s = s0 + lane;
          for (int x = 0; x < 3; ++x) {
            const double dx = d.P[x * n + s] - c[x];
            double q = 1.0;
            for (int e = 0; e < np; ++e, q *= dx) pw[(x * np + e) * P2M_LD + lane] = q;
            al[x * P2M_LD + lane] = d.P[(3 + x) * n + s];
          }
        }
        __syncwarp();
      }
      if (m < d.nm)
#pragma unroll 4
        for (int t = 0; t < cnt; ++t) {
          const double pr = px[t] * py[t] * pz[t];
          v[0] += pr * al[t];
          v[1] += pr * al[P2M_LD + t];
          v[2] += pr * al[2 * P2M_LD + t];
        }
    }
    if (m < rs) put_multipole(d, ci, l, m, v);
  }
}

// ------------------------------------------------ M2M / L2L from tables
// The child-parent displacement is (+-delta, +-delta, +-delta), delta = half
// the child's cell size, with the signs given by the child's octant.  So the
// weights of M2M_multipole (mod_multipole.f90:256-278)
//   a_par(m) += sum_{s <= m} C(m,s) d^(m-s) a_child(s)
// and of L2L_multipole (:360-384)
//   b_child(m) += sum_{s >= m, |s| <= p} C(s,m) d^(s-m) b_par(s)
// are per level the same up to the sign chi_q(ch) = (-1)^(popcount of q and the
// octant bits that are clear), q the parities of the exponents m - s along the
// axes.  The signs are a Walsh-Hadamard transform over the 8 children, so a
// weight acts once per parent instead of once per child:
//   M2M  a_par(m)   = sum_s w(m,s) H_q(m,s)(s),  H_q(s) = sum_ch chi_q(ch) a_ch(s)
//   L2L  b_ch(m)   += sum_q chi_q(ch) T_q(m),    T_q(m) = sum_{s of parity q} w(m,s) b_par(s)
// The host lists, per output m, the terms (w, position of the source value).
struct ShiftTerm {
  double w;
  int at;  // M2M: q (3 nm) + 3 s; L2L: 3 s
  int q;
};

// y_q = sum_ch chi_q(ch) x_ch, in place (index bits are octant / parity bits)
__device__ __forceinline__ void wht_up(double (&x)[8]) {
#pragma unroll
  for (int b = 1; b < 8; b *= 2)
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (!(i & b)) {
        const double u = x[i], v = x[i | b];
        x[i] = u + v;
        x[i | b] = v - u;
      }
}
// y_ch = sum_q chi_q(ch) x_q, in place
__device__ __forceinline__ void wht_down(double (&x)[8]) {
#pragma unroll
  for (int b = 1; b < 8; b *= 2)
#pragma unroll
    for (int i = 0; i < 8; ++i)
      if (!(i & b)) {
        const double u = x[i], v = x[i | b];
        x[i] = u - v;
        x[i | b] = u + v;
      }
}

#define SH_T 128
#define SH_W (SH_T / 32)
// M2M into the active branch cells of level l: one warp per parent; terms and
// offsets staged in shared memory, the children's transforms H in the warp's
// own, lanes over the output coefficient m.  (Every weight applied to each
// child: 22 us a level at least and 472 us for 1,100,000 particles; 6 and 122 us.)
__global__ void __launch_bounds__(SH_T) k_m2m_t(FmmDev d, int l, uint32_t act_lo, uint32_t na,
                                                const ShiftTerm *terms, const int *off, int nterm) {
  extern __shared__ __align__(16) unsigned char shm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int w3 = 3 * d.nm;
  ShiftTerm *st = (ShiftTerm *)shm;
  double *H = (double *)(st + nterm) + (size_t)warp * 8 * w3;  // [q][3 nm]
  int *so = (int *)((double *)(st + nterm) + (size_t)SH_W * 8 * w3);
  for (int e = threadIdx.x; e < nterm; e += SH_T) st[e] = terms[e];
  for (int e = threadIdx.x; e <= d.nm; e += SH_T) so[e] = off[e];
  __syncthreads();
  for (uint32_t c = blockIdx.x * SH_W + warp; c < na; c += gridDim.x * SH_W) {
    const uint32_t ci = act_lo + c;
    const uint32_t key = d.act_key[ci];
    if (!(d.flags[d.G.lev_off[l] + key] & FL_BRANCH)) continue;
    uint32_t cc[8];
#pragma unroll
    for (int ch = 0; ch < 8; ++ch) cc[ch] = d.cidx[d.G.lev_off[l + 1] + 8u * key + (uint32_t)ch];
    __syncwarp();
    for (int e = lane; e < w3; e += 32) {
      double x[8];
#pragma unroll
      for (int ch = 0; ch < 8; ++ch) x[ch] = d.A[(size_t)cc[ch] * w3 + e];
      wht_up(x);
#pragma unroll
      for (int q = 0; q < 8; ++q) H[q * w3 + e] = x[q];
    }
    __syncwarp();
    const int rs = d.ahat ? d.ahat_rs : d.nm;
    for (int m = lane; m < rs; m += 32) {
      double acc[3] = {0, 0, 0};
      if (m < d.nm) {
        const int t1 = so[m + 1];
#pragma unroll 4
        for (int t = so[m]; t < t1; ++t) {
          const ShiftTerm tm = st[t];
          const double *h = H + tm.at;
          acc[0] = fma(tm.w, h[0], acc[0]);
          acc[1] = fma(tm.w, h[1], acc[1]);
          acc[2] = fma(tm.w, h[2], acc[2]);
        }
      }
      put_multipole(d, ci, l, m, acc);
    }
  }
}

// L2L into the active cells of level l (>= 2) from their parents: one warp per
// parent (an active branch cell of level l - 1) and expansion (b with |s| <= p,
// and, with stretching, g with |s| <= p+1), lanes over the output coefficient
// m: the parity sums T_q from the terms (sorted by q), their transform to the
// 8 children, added to the children that are active.  (Every term added to
// each child's sum: 27 us a level at least and 626 us for 1,100,000 particles; 9
// and 328 us.)
__global__ void __launch_bounds__(SH_T) k_l2l_t(FmmDev d, int l, uint32_t act_lo, uint32_t na,
                                                const ShiftTerm *tb, const int *ob, int ntb,
                                                const ShiftTerm *tg, const int *og, int ntg) {
  extern __shared__ __align__(16) unsigned char shm[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const bool isg = blockIdx.y == 1;
  const int nm = isg ? d.nm1 : d.nm, nt = isg ? ntg : ntb, w3 = 3 * nm;
  const ShiftTerm *tt = isg ? tg : tb;
  const int *oo = isg ? og : ob;
  double *E = isg ? d.Gx : d.B;
  ShiftTerm *st = (ShiftTerm *)shm;
  double *sp = (double *)(st + nt) + (size_t)warp * w3;  // parent's expansion
  int *so = (int *)((double *)(st + nt) + (size_t)SH_W * w3);
  for (int e = threadIdx.x; e < nt; e += SH_T) st[e] = tt[e];
  for (int e = threadIdx.x; e <= 8 * nm; e += SH_T) so[e] = oo[e];
  __syncthreads();
  // act_lo / na: the active cells of level l - 1 (the candidate parents)
  for (uint32_t c = blockIdx.x * SH_W + warp; c < na; c += gridDim.x * SH_W) {
    const uint32_t pc = act_lo + c;
    const uint32_t key = d.act_key[pc];
    if (!(d.flags[d.G.lev_off[l - 1] + key] & FL_BRANCH)) continue;
    uint32_t cc[8];
    unsigned live = 0;
#pragma unroll
    for (int ch = 0; ch < 8; ++ch) {
      const uint32_t ck = 8u * key + (uint32_t)ch;
      if (d.flags[d.G.lev_off[l] + ck] & FL_ACTIVE) live |= 1u << ch;
      cc[ch] = d.cidx[d.G.lev_off[l] + ck];
    }
    if (!live) continue;
    __syncwarp();
    for (int e = lane; e < w3; e += 32) sp[e] = E[(size_t)pc * w3 + e];
    __syncwarp();
    for (int m = lane; m < nm; m += 32) {
      // (the children's values are fetched while the sums are formed)
      double T[3][8], old[8][3];
#pragma unroll
      for (int ch = 0; ch < 8; ++ch)
        if ((live >> ch) & 1u) {
          const double *b = E + (size_t)cc[ch] * w3 + 3 * m;
          old[ch][0] = b[0], old[ch][1] = b[1], old[ch][2] = b[2];
        }
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        double a0 = 0.0, a1 = 0.0, a2 = 0.0;
        const int t1 = so[8 * m + q + 1];
#pragma unroll 2
        for (int t = so[8 * m + q]; t < t1; ++t) {
          const ShiftTerm tm = st[t];
          const double *v = sp + tm.at;
          a0 = fma(tm.w, v[0], a0);
          a1 = fma(tm.w, v[1], a1);
          a2 = fma(tm.w, v[2], a2);
        }
        T[0][q] = a0, T[1][q] = a1, T[2][q] = a2;
      }
      wht_down(T[0]);
      wht_down(T[1]);
      wht_down(T[2]);
#pragma unroll
      for (int ch = 0; ch < 8; ++ch)
        if ((live >> ch) & 1u) {
          double *b = E + (size_t)cc[ch] * w3 + 3 * m;
          b[0] = old[ch][0] + T[0][ch];
          b[1] = old[ch][1] + T[1][ch];
          b[2] = old[ch][2] + T[2][ch];
        }
    }
  }
}

static double binom_h(int n, int k) {
  double r = 1.0;
  for (int q = 1; q <= k; ++q) r = r * (double)(n - k + q) / (double)q;
  return r;
}

// term lists of one shift: up = false: s <= m (M2M, deg <= p), offsets per m;
// up = true: s >= m with |s| <= q (L2L of a degree-q expansion), sorted by
// parity class, offsets per (m, class)
static void shift_terms(int nout, int q, bool up, double delta, std::vector<ShiftTerm> &t,
                        std::vector<int> &off) {
  t.clear();
  off.assign(1, 0);
  const int w3 = 3 * n_mon(q);
  for (int m = 0; m < nout; ++m) {
    int mi, mj, mk;
    mono_exp(m, mi, mj, mk);
    std::vector<ShiftTerm> cls[8];
    for (int s = 0; s < n_mon(q); ++s) {
      int si, sj, sk;
      mono_exp(s, si, sj, sk);
      int ex, ey, ez;
      double w;
      if (!up) {
        if (si > mi || sj > mj || sk > mk) continue;
        ex = mi - si;
        ey = mj - sj;
        ez = mk - sk;
        w = binom_h(mi, si) * binom_h(mj, sj) * binom_h(mk, sk);
      } else {
        if (si < mi || sj < mj || sk < mk) continue;
        ex = si - mi;
        ey = sj - mj;
        ez = sk - mk;
        w = binom_h(si, mi) * binom_h(sj, mj) * binom_h(sk, mk);
      }
      double dp = 1.0;
      for (int e = 0; e < ex + ey + ez; ++e) dp *= delta;
      ShiftTerm x;
      x.w = w * dp;
      x.q = (ex & 1) | (ey & 1) << 1 | (ez & 1) << 2;
      x.at = 3 * s + (up ? 0 : x.q * w3);
      cls[up ? x.q : 0].push_back(x);
    }
    for (int c = 0; c < (up ? 8 : 1); ++c) {
      t.insert(t.end(), cls[c].begin(), cls[c].end());
      off.push_back((int)t.size());
    }
  }
}

// per level l: [0] M2M into level l, [1] L2L b into level l, [2] L2L g
static int build_shift_tables(dust_octree *o) {
  std::vector<char> blob;
  auto put = [&](const void *p, size_t n) {
    size_t at = (blob.size() + 15) / 16 * 16;
    blob.resize(at + n);
    memcpy(blob.data() + at, p, n);
    return at;
  };
  std::vector<ShiftTerm> t;
  std::vector<int> off;
  size_t at_t[DUST_MAXLEV + 1][3], at_o[DUST_MAXLEV + 1][3];
  for (int l = 1; l <= o->G.ll; ++l)
    for (int k = 0; k < 3; ++k) {
      o->shift_n[l][k] = 0;
      at_t[l][k] = at_o[l][k] = 0;
      if (k == 0 && l >= o->G.ll) continue;
      if (k > 0 && l < 2) continue;
      if (k == 0)
        shift_terms(o->nm, o->p, false, 0.5 * o->G.csize[l + 1], t, off);
      else if (k == 1)
        shift_terms(o->nm, o->p, true, 0.5 * o->G.csize[l], t, off);
      else
        shift_terms(o->nm1, o->p + 1, true, 0.5 * o->G.csize[l], t, off);
      o->shift_n[l][k] = (int)t.size();
      at_t[l][k] = put(t.data(), t.size() * sizeof(ShiftTerm));
      at_o[l][k] = put(off.data(), off.size() * sizeof(int));
    }
  DUST_TRY(devbuf_grow(o->shift, blob.size() + 16));
  DUST_CUDA(cudaMemcpy(o->shift.p, blob.data(), blob.size(), cudaMemcpyHostToDevice));
  for (int l = 1; l <= o->G.ll; ++l)
    for (int k = 0; k < 3; ++k) {
      o->shift_t[l][k] = (const char *)o->shift.p + at_t[l][k];
      o->shift_o[l][k] = (const char *)o->shift.p + at_o[l][k];
    }
  return DUST_OK;
}

static unsigned shift_grid(int64_t na) {
  int64_t w = (na + SH_T / 32 - 1) / (SH_T / 32);
  return (unsigned)std::max<int64_t>(1, std::min<int64_t>(w, 148 * 16));
}

// M2L of the level-1 cells: every pair of cells that are not adjacent.  Adds
//   g(m') = (-1)^|m'| / m'! sum_n Dhat(m'+n) x ahat(n),  ahat(n) = a(n)/n!,
// |m'| <= p+1 (|m'| <= p without stretching), into the cell's g and (|m'| <= p)
// b.  A CTA per target; a warp takes 32 outputs of every nslot-th source, and
// the parts are added in slot order.  The level has at most a few dozen cells:
// what counts is the chain of a source's table reads.  (All outputs of one
// source after the other by two warps: 345 us for a level of 72 cells; 54 us.)
#define M1_T 512
__global__ void __launch_bounds__(M1_T) k_m2l_1(FmmDev d, uint32_t act_lo) {
  __shared__ double s_p[M1_T][3];
  const uint32_t ci = act_lo + blockIdx.x;
  const uint32_t key = d.act_key[ci];
  // an empty target cell is a leaf without particles: its local expansion
  // is evaluated only when points were sorted into it (and it has no
  // children to pass it to)
  if (cell_hi(d.G, d.cstart, 1, key) == cell_lo(d.G, d.cstart, 1, key) &&
      !(d.flags[d.G.lev_off[1] + key] & FL_PTS))
    return;
  int i, j, k;
  cart_of_key(d.G, 1, key, i, j, k);
  const int nm = d.nm, nout = d.use_vs ? d.nm1 : d.nm;
  const int Lx = d.kdlen[1][0], Ly = d.kdlen[1][1], Lz = d.kdlen[1][2];
  const uint32_t lo1 = d.G.lev_off[1];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ng = (nout + 31) / 32, nslot = (M1_T / 32) / ng;  // ng <= 7
  const int slot = warp / ng, mo = 32 * (warp % ng) + lane;
  double acc[3] = {0, 0, 0};
  int seen = 0;
  for (uint32_t q0 = 0; q0 < d.G.ncell[1] && slot < nslot; q0 += 32) {
    const uint32_t sk = q0 + lane;
    int src = 0, tab = 0;
    bool on = sk < d.G.ncell[1];
    if (on) {
      int si, sj, sk_;
      cart_of_key(d.G, 1, sk, si, sj, sk_);
      on = !(abs(si - i) <= 1 && abs(sj - j) <= 1 && abs(sk_ - k) <= 1) &&
           (d.flags[lo1 + sk] & FL_ACTIVE) &&
           cell_hi(d.G, d.cstart, 1, sk) != cell_lo(d.G, d.cstart, 1, sk);
      if (on) {
        src = (int)d.cidx[lo1 + sk];
        tab = (si - i + Lx) + (2 * Lx + 1) * ((sj - j + Ly) + (2 * Ly + 1) * (sk_ - k + Lz));
      }
    }
    for (unsigned ml = __ballot_sync(~0u, on); ml; ml &= ml - 1, ++seen) {
      const int from = __ffs(ml) - 1;
      const int s1 = __shfl_sync(~0u, src, from), t1 = __shfl_sync(~0u, tab, from);
      if (seen % nslot != slot || mo >= nout) continue;
      const double *a = d.A + (size_t)s1 * 3 * nm;
      const double *D = d.dtab[1] + (size_t)t1 * d.nD * 3;
#pragma unroll 5
      for (int nn = 0; nn < nm; ++nn) {
        const int qd = d.idxsum[(size_t)nn * d.nm1 + mo];
        const double Dx = __ldg(D + 3 * qd), Dy = __ldg(D + 3 * qd + 1), Dz = __ldg(D + 3 * qd + 2);
        const double f = d.inv_fact[nn];
        const double ax = a[3 * nn] * f, ay = a[3 * nn + 1] * f, az = a[3 * nn + 2] * f;
        acc[0] += Dy * az - Dz * ay;
        acc[1] += Dz * ax - Dx * az;
        acc[2] += Dx * ay - Dy * ax;
      }
    }
  }
  for (int e = 0; e < 3; ++e) s_p[threadIdx.x][e] = acc[e];
  __syncthreads();
  if (slot > 0 || mo >= nout) return;
  for (int s = 1; s < nslot; ++s)
    for (int e = 0; e < 3; ++e) acc[e] += s_p[32 * s * ng + threadIdx.x][e];
  int oi, oj, ok;
  mono_exp(mo, oi, oj, ok);
  const double sc = (((oi + oj + ok) & 1) ? -1.0 : 1.0) * d.inv_fact[mo];
  if (d.use_vs) {
    double *g = d.Gx + (size_t)ci * 3 * d.nm1;
    for (int e = 0; e < 3; ++e) g[3 * mo + e] += sc * acc[e];
  }
  if (mo < nm) {
    double *b = d.B + (size_t)ci * 3 * nm;
    for (int e = 0; e < 3; ++e) b[3 * mo + e] += sc * acc[e];
  }
}

// ------------------------------------------------------------- L2P + P2P
// One source q (strength a) acting on target p (strength ta): the reference's
// compute_vel, compute_stretch, compute_rotu and compute_diffusion of source q
// (mod_vortpart.f90:139-336), 4*pi factors applied by the caller.  With d = p - q,
// rho^2 = d^2 + s^2, s the source's r_v, the pair's terms are
//   velocity      -d x a / rho^3
//   stretching    x / rho^3 - 3 (d.x) d / rho^5, x = ta x a
//   rotational    a (3 s^2/rho^2 - 1) / rho^3 + 3 (d.a) d / rho^5
//   diffusion     17.5 s^-2 (s/rho)^9 (a - ta)
// (d^2 = rho^2 - s^2, 1 + d^2/s^2 = rho^2/s^2): one reciprocal root serves all
// four (v: without the sign): 63 FP64 operations a pair where term by term took
// 78 (110,000 particles: 1.22 -> 0.92 ms).  q[7] = 17.5 / s.
// (ta x taken out of the sum too, 56 operations: three times the FP32 error
// of the stretching, whose terms cancel in x where strengths are parallel.)
template <typename V>
struct P2PSums {
  V v[3], s[3], r[3], f[3];
};
template <bool VS, bool DF, bool VD>
__device__ __forceinline__ void p2p_pair(const double *tp, const double *ta, const double (&q)[8],
                                         bool self, P2PSums<double> &A) {
  const double d[3] = {tp[0] - q[0], tp[1] - q[1], tp[2] - q[2]};
  const double *a = q + 3, s2 = q[6];
  const double r = rsqrt_r(fma(d[0], d[0], fma(d[1], d[1], fma(d[2], d[2], s2))));
  const double inv = self ? 0.0 : r, i2 = inv * inv, i3 = i2 * inv, rt2 = s2 * i2;
  const double c[3] = {d[1] * a[2] - d[2] * a[1], d[2] * a[0] - d[0] * a[2],
                       d[0] * a[1] - d[1] * a[0]};
#pragma unroll
  for (int e = 0; e < 3; ++e) A.v[e] = fma(i3, c[e], A.v[e]);
  if (VS) {
    const double k3 = 3.0 * i3, i5 = k3 * i2;
    const double x[3] = {ta[1] * a[2] - ta[2] * a[1], ta[2] * a[0] - ta[0] * a[2],
                         ta[0] * a[1] - ta[1] * a[0]};
    const double t = i5 * -fma(d[0], x[0], fma(d[1], x[1], d[2] * x[2]));
#pragma unroll
    for (int e = 0; e < 3; ++e) A.s[e] = fma(i3, x[e], fma(t, d[e], A.s[e]));
    if (DF) {
      const double u = i5 * fma(d[0], a[0], fma(d[1], a[1], d[2] * a[2]));
      const double g = fma(k3, rt2, -i3);
#pragma unroll
      for (int e = 0; e < 3; ++e) A.r[e] = fma(g, a[e], fma(u, d[e], A.r[e]));
    }
  }
  if (VD) {
    const double rt4 = rt2 * rt2, w = (q[7] * inv) * (rt4 * rt4);
#pragma unroll
    for (int e = 0; e < 3; ++e) A.f[e] = fma(w, a[e] - ta[e], A.f[e]);
  }
}
// FP32 form of two sources at a time in packed operations, on coordinates
// relative to the leaf centre.  Each output gets one addition a pair, and the
// diffusion its own reciprocal root (from 1 / s^2 = q[7]; its ninth power of
// s / rho would carry the other's error): the sums' errors against 64 bits are
// those of the term-by-term form (0.97 to 0.99 of them over 16 sets of 37 to 2,500
// particles; 1,100,000 particles: 4.59 -> 3.7 ms).
template <bool VS, bool DF, bool VD>
__device__ __forceinline__ void p2p_pair2_f(const float *tp, const float *ta, const float2 (&q)[8],
                                            bool self0, bool self1, P2PSums<float2> &A) {
  auto two = [](float x) { return make_float2(x, x); };
  auto neg = [](float2 x) { return make_float2(-x.x, -x.y); };
  float2 d[3], m[3];  // d and -d
#pragma unroll
  for (int e = 0; e < 3; ++e) {
    m[e] = __fadd2_rn(q[e], two(-tp[e]));
    d[e] = neg(m[e]);
  }
  const float2 *a = q + 3, s2 = q[6];
  const float2 r2 = __ffma2_rn(m[0], m[0], __ffma2_rn(m[1], m[1], __fmul2_rn(m[2], m[2])));
  const float2 rho2 = __fadd2_rn(r2, s2);
  const float2 inv = make_float2(self0 ? 0.f : rsqrtf(rho2.x), self1 ? 0.f : rsqrtf(rho2.y));
  const float2 i2 = __fmul2_rn(inv, inv), i3 = __fmul2_rn(i2, inv);
  const float2 c[3] = {__ffma2_rn(d[1], a[2], __fmul2_rn(m[2], a[1])),
                       __ffma2_rn(d[2], a[0], __fmul2_rn(m[0], a[2])),
                       __ffma2_rn(d[0], a[1], __fmul2_rn(m[1], a[0]))};
#pragma unroll
  for (int e = 0; e < 3; ++e) A.v[e] = __ffma2_rn(i3, c[e], A.v[e]);
  if (VS) {
    const float2 i5 = __fmul2_rn(__fmul2_rn(i3, two(3.0f)), i2);
    const float2 x[3] = {
        __ffma2_rn(two(ta[1]), a[2], __fmul2_rn(two(-ta[2]), a[1])),
        __ffma2_rn(two(ta[2]), a[0], __fmul2_rn(two(-ta[0]), a[2])),
        __ffma2_rn(two(ta[0]), a[1], __fmul2_rn(two(-ta[1]), a[0]))};
    const float2 t = __fmul2_rn(
        i5, __ffma2_rn(m[0], x[0], __ffma2_rn(m[1], x[1], __fmul2_rn(m[2], x[2]))));
#pragma unroll
    for (int e = 0; e < 3; ++e)
      A.s[e] = __fadd2_rn(A.s[e], __ffma2_rn(i3, x[e], __fmul2_rn(t, d[e])));
    if (DF) {
      const float2 u = __ffma2_rn(d[0], a[0], __ffma2_rn(d[1], a[1], __fmul2_rn(d[2], a[2])));
      const float2 k = __fadd2_rn(i3, i3);
#pragma unroll
      for (int e = 0; e < 3; ++e)
        A.r[e] = __fadd2_rn(
            A.r[e], __ffma2_rn(k, a[e],
                               __fmul2_rn(i5, __ffma2_rn(d[e], u, __fmul2_rn(neg(r2), a[e])))));
    }
  }
  if (VD) {
    const float2 t = __ffma2_rn(r2, q[7], two(1.0f));
    const float2 rt = make_float2(self0 ? 0.f : rsqrtf(t.x), self1 ? 0.f : rsqrtf(t.y));
    const float2 rt2 = __fmul2_rn(rt, rt), rt4 = __fmul2_rn(rt2, rt2),
                 w = __fmul2_rn(q[7], __fmul2_rn(__fmul2_rn(rt4, rt4), rt));
#pragma unroll
    for (int e = 0; e < 3; ++e)
      A.f[e] = __ffma2_rn(w, __fadd2_rn(a[e], two(-ta[e])), A.f[e]);
  }
}

// L2P + P2P, one warp per leaf or, where a leaf's near field is large, per
// share of it.  Leaves hold a few particles (6 on average in the 2M-particle
// full step), so a CTA per leaf would leave most lanes idle.  The warp lists
// the leaf's near field as particle ranges (the 26 active same-level
// neighbours, the coarser leaf neighbours of every level above -- leaf_neigh,
// mod_octree.f90:964-988 -- and the leaf itself, at most 26 * DUST_MAXLEV + 1
// ranges), then takes its targets 32 at a time: lanes are split into
// G = 32 / cnt groups of cnt lanes (one lane per target), lane (tl, grp)
// accumulates target tl over the sources u = grp mod G of each 32-source tile
// staged in the warp's own shared memory, and group 0 adds the other groups'
// sums from shared memory.  A source is found from its position in the
// concatenated ranges by a search over the range prefix sums (walked forward
// tile by tile).
//   FP64: pairs by p2p_pair on absolute coordinates, summed in FP64.
//   FP32C (F32): pairs by p2p_pair2_f on coordinates relative to the leaf
//   centre (differences formed in FP64, rounded once), FP32 partial sums of
//   up to 128 sources folded into FP64.
// L2P (mod_octree.f90:1171-1212) is FP64 in both.
//
// A coarse leaf beside a fine cluster has the whole cluster as its near field
// (its same-level neighbours are branches): tens of thousands of sources for
// one warp, a chain that outlasted the rest of the grid (110k ring particles,
// FP64: 11.0 ms for 120M pairs, 1.3 ms cut; 1.1M FP32C: SMs idle for 44 % of
// 9.2 ms, 4.6 ms cut).  So k_p2p_split first counts every leaf's sources and cuts the leaves of more
// than `it` pair iterations per 32 targets into items of (32 targets, at most
// it * G sources), which the grid's first CTAs work off; items add to
// the outputs atomically, the first one of a target also its L2P.
#define P2W_TILE 32
#define P2W_MAXR (26 * DUST_MAXLEV + 4)
#define P2W_NV 8  // staged per source: x y z, alpha x y z, s^2 and, with
                  // s = r_v, 17.5 / s (FP64) or 1 / s^2 (FP32)
#define P2W_LQ 4  // levels whose near-field loads are issued together
#define P2W_XB (148 * 16)  // CTAs for the items: the resident ones
#define P2W_CAP (1u << 18) // items (4 MB)

struct P2PItems {
  uint8_t *split;    // per leaf: its work is in the items
  uint4 *item;       // leaf, first target, sources [z, w) of the concatenated ranges
  unsigned long long *count;  // [0] items, [1] next item
  uint32_t cap;
  int it;            // pair iterations of an item
};

// the near-field ranges of P2W_LQ levels from lev0 up for this lane's
// neighbour: flags and ranges are loaded without branches (predicated on the
// neighbour lying in the box), so the loads of all levels are in flight
// together rather than one dependent chain per level
__device__ __forceinline__ void p2p_ranges(const FmmDev &d, int l, int ci, int cj, int ck,
                                           int lev0, int lane, uint32_t (&a0)[P2W_LQ],
                                           uint32_t (&len)[P2W_LQ]) {
  uint32_t a1[P2W_LQ];
  bool ok[P2W_LQ], want[P2W_LQ];
  const int di = lane % 3 - 1, dj = (lane / 3) % 3 - 1, dk = lane / 9 - 1;
#pragma unroll
  for (int q = 0; q < P2W_LQ; ++q) {
    const int lev = lev0 - q, sh = l - lev;
    const int ai = (ci >> sh) + di, aj = (cj >> sh) + dj, ak = (ck >> sh) + dk;
    ok[q] = lev >= 1 && lane < 27 && lane != 13 && cart_in(d.G, lev, ai, aj, ak);
    const uint32_t nk = ok[q] ? key_of(d.G, lev, ai, aj, ak) : 0u;
    const uint8_t f = ok[q] ? d.flags[d.G.lev_off[lev] + nk] : (uint8_t)0;
    a0[q] = ok[q] ? cell_lo(d.G, d.cstart, lev, nk) : 0u;
    a1[q] = ok[q] ? cell_hi(d.G, d.cstart, lev, nk) : 0u;
    want[q] = (lev == l) ? (f & FL_ACTIVE) != 0 : (f & FL_LEAF) != 0;
  }
#pragma unroll
  for (int q = 0; q < P2W_LQ; ++q) len[q] = ok[q] && want[q] ? a1[q] - a0[q] : 0u;
}

// one warp per leaf: the number of its sources; cuts a large leaf into items
// (a leaf that no longer fits the list stays whole) and zeroes its outputs
__global__ void __launch_bounds__(256) k_p2p_split(FmmDev d, P2PItems w) {
  const int lane = threadIdx.x & 31;
  const uint32_t leaf = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (leaf >= d.n_leaves) return;
  const uint32_t ci = d.leaf_ci[leaf];
  const int l = d.act_lev[ci];
  const uint32_t key = d.act_key[ci];
  int i, j, k;
  cart_of_key(d.G, l, key, i, j, k);
  const uint32_t lo = cell_lo(d.G, d.cstart, l, key), hi = cell_hi(d.G, d.cstart, l, key);
  const uint32_t nt = hi - lo;
  uint32_t S = 0;
  if (nt > 0)
    for (int lev0 = l; lev0 >= 1; lev0 -= P2W_LQ) {
      uint32_t a0[P2W_LQ], len[P2W_LQ];
      p2p_ranges(d, l, i, j, k, lev0, lane, a0, len);
      for (int q = 0; q < P2W_LQ; ++q) S += len[q];
    }
  S = __reduce_add_sync(0xffffffffu, S) + nt;
  if (lane == 0 && nt > 0 && d.counters)
    atomicAdd((unsigned long long *)d.counters + 1, (unsigned long long)nt * (S - 1));
  bool split = false;
  if (nt > 0) {
    const P2PCut c = p2p_cut(nt, S, (uint32_t)w.it, w.cap);
    if (c.ni > 1 && c.ni <= w.cap) {  // (else whole, and nothing of the list taken)
      unsigned long long at = 0;
      if (lane == 0) at = atomicAdd(w.count, (unsigned long long)c.ni);
      at = __shfl_sync(0xffffffffu, at, 0);
      split = at + c.ni <= w.cap;
      for (uint32_t e = lane; e < c.ni; e += 32) {
        uint32_t tb, s0, s1;
        p2p_item(c, S, e, tb, s0, s1);
        // (an item past the list's end is never read: the count is clamped)
        if (at + e < w.cap)
          w.item[at + e] = split ? make_uint4(leaf, tb, s0, s1) : make_uint4(leaf, 0, 0, 0);
      }
    }
    if (split)
      for (uint32_t t = lane; t < nt; t += 32)
        for (int e = 0; e < 9; ++e) d.out[(size_t)e * d.n + lo + t] = 0.0;
  }
  if (lane == 0) w.split[leaf] = split;
}

template <bool VS, bool DF, bool VD, bool TV, bool F32>
__device__ __forceinline__ void p2p_share(const FmmDev &d, uint32_t leaf, int tb, int te,
                                          uint32_t s_lo, uint32_t s_hi, bool split) {
  using R = typename std::conditional<F32, float, double>::type;
  __shared__ __align__(16) R s_src[P2W_NV][P2W_TILE];
  __shared__ __align__(8) uint32_t s_sid[P2W_TILE];
  __shared__ uint32_t rlo[P2W_MAXR];
  __shared__ uint32_t rcum[P2W_MAXR + 1];
  __shared__ double s_acc[12][32];
  const int lane = threadIdx.x & 31;
  const uint32_t ci = d.leaf_ci[leaf];
  const int l = d.act_lev[ci];
  const uint32_t key = d.act_key[ci];
  int ci_, cj, ck;
  cart_of_key(d.G, l, key, ci_, cj, ck);
  double cc[3];
  cell_center(d.G, l, ci_, cj, ck, cc);
  const uint32_t lo = cell_lo(d.G, d.cstart, l, key), hi = cell_hi(d.G, d.cstart, l, key);
  if (hi == lo) return;
  // near-field source ranges: same level first, then coarser levels, the leaf
  // itself last; rcum their positions in the concatenation
  int nr = 0;
  uint32_t S = 0;
  for (int lev0 = l; lev0 >= 1; lev0 -= P2W_LQ) {
    uint32_t a0q[P2W_LQ], len[P2W_LQ];
    p2p_ranges(d, l, ci_, cj, ck, lev0, lane, a0q, len);
#pragma unroll
    for (int q = 0; q < P2W_LQ; ++q) {
      const unsigned msk = __ballot_sync(0xffffffffu, len[q] > 0);
      if (!msk) continue;
      uint32_t run = len[q];  // inclusive scan over the lanes
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += v;
      }
      const int pos = nr + __popc(msk & ((1u << lane) - 1u));
      // 26 per level and l <= DUST_MAXLEV levels: the list cannot overflow
      if (len[q] > 0 && pos < P2W_MAXR - 1) {
        rlo[pos] = a0q[q];
        rcum[pos] = S + run - len[q];
      }
      S += __shfl_sync(0xffffffffu, run, 31);
      nr = min(nr + __popc(msk), P2W_MAXR - 1);
    }
  }
  if (lane == 0) {
    rlo[nr] = lo;
    rcum[nr] = S;
    rcum[nr + 1] = S + (hi - lo);
  }
  ++nr;
  S += hi - lo;
  __syncwarp();
  s_hi = min(s_hi, S);
  const size_t n = d.n;
  const int nt = (int)(hi - lo), nm = d.nm, nm1 = d.nm1;
  const double k4pi = 1.0 / (4.0 * DUST_PI);
  const double *bl = d.B + (size_t)ci * 3 * nm, *gl = d.Gx + (size_t)ci * 3 * nm1;
  // L2P of one target (FP64): velocity and the gradient of the local field
  // (the monomials m0, m0 + ms, ... only: the caller splits the sum)
  auto l2p = [&](uint32_t ti, int m0, int ms, double *lv, double *g) {
    const double x = d.P[ti] - cc[0], y = d.P[n + ti] - cc[1], z = d.P[2 * n + ti] - cc[2];
    double px[DUST_MAXP + 1], py[DUST_MAXP + 1], pz[DUST_MAXP + 1];
    px[0] = py[0] = pz[0] = 1.0;
#pragma unroll
    for (int e = 1; e <= DUST_MAXP; ++e) {
      px[e] = px[e - 1] * x;
      py[e] = py[e - 1] * y;
      pz[e] = pz[e - 1] * z;
    }
    for (int e = 0; e < 3; ++e) lv[e] = 0.0;
    for (int e = 0; e < 9; ++e) g[e] = 0.0;
    for (int m = m0; m < nm; m += ms) {
      int mi, mj, mk;
      mono_exp(m, mi, mj, mk);
      const double pr = px[mi] * py[mj] * pz[mk];
      for (int e = 0; e < 3; ++e) lv[e] += __ldg(bl + 3 * m + e) * pr;
      if (VS) {
        const double *g0 = gl + 3 * mono_idx(mi + 1, mj, mk), *g1 = gl + 3 * mono_idx(mi, mj + 1, mk),
                     *g2 = gl + 3 * mono_idx(mi, mj, mk + 1);
        const double f0 = (mi + 1) * pr, f1 = (mj + 1) * pr, f2 = (mk + 1) * pr;
        for (int e = 0; e < 3; ++e) {
          g[0 + 3 * e] += f0 * __ldg(g0 + e);
          g[1 + 3 * e] += f1 * __ldg(g1 + e);
          g[2 + 3 * e] += f2 * __ldg(g2 + e);
        }
      }
    }
  };
  double ave_ros = 0.0;
  if (TV) {
    // leaf average of |sym(grad)|^2 from the local expansion (:1214-1230)
    double part = 0.0;
    for (int t = lane; t < nt; t += 32) {
      double lv[3], g[9];
      l2p(lo + t, 0, 1, lv, g);
      for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) {
          const double sy = 0.5 * (g[a + 3 * b] + g[b + 3 * a]);
          part += sy * sy;
        }
    }
    for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
    ave_ros = part / (double)nt;
  }
  R *fs = &s_src[0][0];
  double *acc = &s_acc[0][lane];  // this lane's 12 FP64 sums, stride 32
  for (int t0 = tb; t0 < min(nt, te); t0 += 32) {
    // G groups of cnt lanes (one lane per target) split the sources; lanes
    // beyond G * cnt idle
    const int cnt = min(32, nt - t0);
    const int TPR = cnt, G = 32 / TPR, tl = lane % TPR, grp = lane / TPR;
    const bool act = grp < G;
    const uint32_t ti = lo + t0 + (act ? tl : 0);
    R tp[3], ta[3];
    for (int q = 0; q < 3; ++q) {
      tp[q] = F32 ? (R)(d.P[(size_t)q * n + ti] - cc[q]) : (R)d.P[(size_t)q * n + ti];
      ta[q] = (R)d.P[(size_t)(3 + q) * n + ti];
    }
    // FP64 sums: in registers (FP64 pairs) or in shared memory (FP32C,
    // which keeps its registers for the FP32 partial sums)
    P2PSums<double> A;
    P2PSums<float2> B;
    auto clear_f = [&]() {
      for (int e = 0; e < 3; ++e)
        B.v[e] = B.s[e] = B.r[e] = B.f[e] = make_float2(0.f, 0.f);
    };
    for (int e = 0; e < 3; ++e) A.v[e] = A.s[e] = A.r[e] = A.f[e] = 0.0;
    clear_f();
    if (F32)
      for (int e = 0; e < 12; ++e) acc[32 * e] = 0.0;
    // adds the four outputs of a pair's sums to acc
    auto put = [&](const double *v, const double *ss, const double *r, const double *f) {
      for (int e = 0; e < 3; ++e) {
        acc[32 * e] -= v[e];
        if (VS) acc[32 * (3 + e)] += ss[e];
        if (VS && DF) acc[32 * (6 + e)] += r[e];
        if (VD) acc[32 * (9 + e)] += (F32 ? 17.5 : 1.0) * f[e];
      }
    };
    int since = 0;
    // the sources of the next tile are loaded into registers while the
    // current tile is evaluated; each lane's range index only moves forward
    // (source v = s0 + lane grows by the tile size)
    int ra = 0;
    double pf[7];
    uint32_t psid = 0;
    bool pv = false;
    auto fetch = [&](uint32_t v) {
      pv = v < s_hi;
      if (pv) {
        while (ra + 1 < nr && rcum[ra + 1] <= v) ++ra;  // last r with rcum[r] <= v
        psid = rlo[ra] + (v - rcum[ra]);
#pragma unroll
        for (int q = 0; q < 7; ++q) pf[q] = d.P[(size_t)q * n + psid];
      }
    };
    fetch(s_lo + lane);
    for (uint32_t s0 = s_lo; s0 < s_hi; s0 += P2W_TILE) {
      __syncwarp();
      // (beyond the last source: no strength, kv = 0)
      R st8[8] = {(R)0, (R)0, (R)0, (R)0, (R)0, (R)0, (R)1, (R)0};
      if (pv) {
        for (int q = 0; q < 3; ++q) st8[q] = F32 ? (R)(pf[q] - cc[q]) : (R)pf[q];
        for (int q = 3; q < 6; ++q) st8[q] = (R)pf[q];
        const R rv = (R)pf[6];
        st8[6] = rv * rv;
        if (VD) {
          // (a core of zero diffuses nothing, and the particle itself is among the
          // sources, with inv = 0)
          const R k = F32 ? (R)1 / st8[6] : (R)17.5 / fabs(rv);
          st8[7] = isinf(k) ? (R)0 : k;
        }
      }
      s_sid[lane] = psid;
#pragma unroll
      for (int q = 0; q < 8; ++q) fs[q * P2W_TILE + lane] = st8[q];
      __syncwarp();
      fetch(s0 + P2W_TILE + lane);
      const int m = (int)min((uint32_t)P2W_TILE, s_hi - s0);
      if (act)
#pragma unroll 1
        for (int u = 2 * grp; u < m; u += 2 * G) {
          const uint2 id = *(const uint2 *)&s_sid[u];
          if constexpr (F32) {
            float2 q[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) q[e] = *(const float2 *)&fs[e * P2W_TILE + u];
            p2p_pair2_f<VS, DF, VD>(tp, ta, q, id.x == ti, id.y == ti, B);
          } else {
            double q0[8], q1[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) {
              const double2 x = *(const double2 *)&fs[e * P2W_TILE + u];
              q0[e] = x.x;
              q1[e] = x.y;
            }
            p2p_pair<VS, DF, VD>(tp, ta, q0, id.x == ti, A);
            p2p_pair<VS, DF, VD>(tp, ta, q1, id.y == ti, A);
          }
        }
      if (F32 && (++since == 4 || s0 + P2W_TILE >= s_hi)) {
        // FP32 partial sums of up to 128 sources folded into FP64
        since = 0;
        double v[3], ss[3], r[3], f[3];
        for (int e = 0; e < 3; ++e) {
          v[e] = (double)B.v[e].x + (double)B.v[e].y;
          ss[e] = (double)B.s[e].x + (double)B.s[e].y;
          r[e] = (double)B.r[e].x + (double)B.r[e].y;
          f[e] = (double)B.f[e].x + (double)B.f[e].y;
        }
        put(v, ss, r, f);
        clear_f();
      }
    }
    // combine the groups of each target (group 0's lane sums the others'
    // shared-memory sums)
    if (!F32) {
      for (int e = 0; e < 12; ++e) acc[32 * e] = 0.0;
      put(A.v, A.s, A.r, A.f);
    }
    __syncwarp();
    double Q[12];
    for (int e = 0; e < 12; ++e) {
      Q[e] = acc[32 * e];
      if (grp == 0)
        for (int g = 1; g < G; ++g) Q[e] += acc[32 * e + g * TPR];
    }
    __syncwarp();
    // L2P (FP64) split over the groups: lane (tl, grp) sums the monomials
    // grp, grp + G, ... of its target; group 0 adds the other groups' parts
    // (with the first sources of the target only)
    double lv[3] = {0, 0, 0}, g[9] = {0, 0, 0, 0, 0, 0, 0, 0, 0};
    if (act && s_lo == 0) {
      l2p(ti, grp, G, lv, g);
      for (int e = 0; e < 3; ++e) acc[32 * e] = lv[e];
      for (int e = 0; e < 9; ++e) acc[32 * (3 + e)] = g[e];
    }
    __syncwarp();
    if (act && grp == 0) {
      for (int q = 1; q < G && s_lo == 0; ++q) {
        for (int e = 0; e < 3; ++e) lv[e] += acc[32 * e + q * TPR];
        for (int e = 0; e < 9; ++e) g[e] += acc[32 * (3 + e) + q * TPR];
      }
      const double tad[3] = {d.P[3 * n + ti], d.P[4 * n + ti], d.P[5 * n + ti]};
      double ls[3] = {0, 0, 0}, lr[3] = {0, 0, 0};
      if (VS) {
        for (int e = 0; e < 3; ++e) ls[e] = tad[0] * g[e] + tad[1] * g[e + 3] + tad[2] * g[e + 6];
        if (DF) {
          lr[0] = g[1 + 6] - g[2 + 3];
          lr[1] = g[2 + 0] - g[0 + 6];
          lr[2] = g[0 + 3] - g[1 + 0];
        }
      }
      double nu = d.nu_inf;
      if (TV) {
        const double rv = d.P[6 * n + ti];
        nu += (0.11 * rv) * (0.11 * rv) * sqrt(2.0 * ave_ros);
      }
      for (int e = 0; e < 3; ++e) {
        const double o0 = lv[e] + Q[e] * k4pi, o2 = lr[e] + Q[6 + e] * k4pi,
                     o1 = ls[e] + Q[3 + e] * k4pi + (VD ? Q[9 + e] * nu : 0.0);
        double *o = d.out + ti;
        if (split) {
          atomicAdd(o + (size_t)e * n, o0);
          if (VS || VD) atomicAdd(o + (size_t)(3 + e) * n, o1);
          if (DF) atomicAdd(o + (size_t)(6 + e) * n, o2);
        } else {
          o[(size_t)e * n] = o0;
          o[(size_t)(3 + e) * n] = o1;
          o[(size_t)(6 + e) * n] = o2;
        }
      }
    }
    __syncwarp();  // acc is reused by the next 32 targets
  }
}

template <bool VS, bool DF, bool VD, bool TV, bool F32>
__global__ void __launch_bounds__(32, 16) k_p2p_w(FmmDev d, P2PItems w) {
  uint32_t leaf, tb = 0, te = 0xffffffffu >> 1, s_lo = 0, s_hi = 0xffffffffu;
  const bool items = blockIdx.x < P2W_XB;
  if (!items) {
    leaf = blockIdx.x - P2W_XB;
    if (w.split[leaf]) return;
  }
  do {
    if (items) {
      unsigned long long i = 0;
      if (threadIdx.x == 0) i = atomicAdd(w.count + 1, 1ull);
      i = __shfl_sync(0xffffffffu, i, 0);
      if (i >= min(w.count[0], (unsigned long long)w.cap)) return;
      const uint4 it = w.item[i];
      leaf = it.x, tb = it.y, te = it.y + 1, s_lo = it.z, s_hi = it.w;
      if (s_hi == 0) continue;  // of a leaf that did not fit the list
      __syncwarp();
    }
    p2p_share<VS, DF, VD, TV, F32>(d, leaf, (int)tb, (int)te, s_lo, s_hi, items);
  } while (items);
}

// ======================================================== host orchestration
static inline unsigned nblk(size_t n, int t) { return (unsigned)((n + t - 1) / t); }

static void fill_dev(dust_octree *o, FmmDev &d, int n) {
  memset(&d, 0, sizeof(d));
  d.G = o->G;
  d.n = (uint32_t)n;
  d.p = o->p;
  d.nm = o->nm;
  d.nm1 = o->nm1;
  d.nD = o->nD;
  d.use_vs = o->prm.vortstretch != 0;
  d.use_df = o->prm.divergence_filtering != 0;
  d.use_vd = o->prm.diffusion != 0;
  d.nu_inf = o->prm.nu_inf;
  for (int c = 0; c < 3; ++c) d.u_inf[c] = o->prm.u_inf[c];
  for (int l = 0; l <= DUST_MAXLEV; ++l) {
    d.dtab[l] = (const double *)o->dtab[l].p;
    for (int c = 0; c < 3; ++c) d.kdlen[l][c] = o->kdlen[l][c];
  }
  d.idxsum = (const uint16_t *)o->idxsum.p;
  // 1/m! of the multi-index m, for every monomial up to degree p+1
  for (int m = 0; m < o->nm1 && m < 224; ++m) {
    int i, j, k;
    mono_exp(m, i, j, k);
    double fi = 1, fj = 1, fk = 1;
    for (int q = 2; q <= i; ++q) fi *= q;
    for (int q = 2; q <= j; ++q) fj *= q;
    for (int q = 2; q <= k; ++q) fk *= q;
    d.inv_fact[m] = 1.0 / (fi * fj * fk);
  }
}

// Builds the tree of n device-resident particles and evaluates the FMM; the
// outputs stay in o->outs (sorted order) for the element pass.
int fmm_prepare_device(dust_octree *o, int n, const double *cen, const double *dir,
                       const double *mag, const double *rv, int n_pts, const double *pts,
                       cudaStream_t st) {
  TreeGeom &G = o->G;
  o->last_stream = st;
  const int ll = G.ll;
  const uint32_t nfine = G.ncell[ll];
  const uint32_t ntot = (uint32_t)o->ncell_tot;
  size_t N = (size_t)std::max(n, 1);
  DUST_TRY(grow(o->keys, N * 4));
  DUST_TRY(grow(o->keys_s, N * 4));
  DUST_TRY(grow(o->vals, N * 4));
  DUST_TRY(grow(o->perm, N * 4));
  DUST_TRY(grow(o->cnt, (size_t)(nfine + 1) * 4));
  DUST_TRY(grow(o->cstart, (size_t)(nfine + 1) * 4));
  DUST_TRY(grow(o->part, N * 7 * 8));
  DUST_TRY(grow(o->flags, (size_t)ntot + 1));
  DUST_TRY(grow(o->cidx, (size_t)(ntot + 1) * 4));
  DUST_TRY(grow(o->lidx, (size_t)(ntot + 1) * 4));
  DUST_TRY(grow(o->srcix, (size_t)(ntot + 1) * 4));
  DUST_TRY(grow(o->outs, N * 12 * 8));
  uint32_t *keys = (uint32_t *)o->keys.p, *keys_s = (uint32_t *)o->keys_s.p;
  uint32_t *vals = (uint32_t *)o->vals.p, *perm = (uint32_t *)o->perm.p;
  uint32_t *cnt = (uint32_t *)o->cnt.p, *cstart = (uint32_t *)o->cstart.p;
  uint8_t *flags = (uint8_t *)o->flags.p;
  uint32_t *cidx = (uint32_t *)o->cidx.p, *lidx = (uint32_t *)o->lidx.p;
  int64_t *small = (int64_t *)o->small.p;
  int *err = (int *)(small + 40);

  o->kev_m2l = false;
  if (o->timing) cudaEventRecord(o->ev[0], st);
  DUST_CUDA(cudaMemsetAsync(cnt, 0, (size_t)(nfine + 1) * 4, st));
  // the first particle and the first point out of the box (small + 40 and + 41)
  const int big[3] = {0x7fffffff, 0, 0x7fffffff};
  DUST_CUDA(cudaMemcpyAsync(err, big, sizeof(big), cudaMemcpyHostToDevice, st));
  if (n > 0) k_bin<<<nblk(n, 256), 256, 0, st>>>(n, cen, G, keys, vals, cnt, err);
  // radix sort (stable) by finest key; bits needed for the finest key
  int bits = 1;
  while (bits < 32 && (1ull << bits) < (uint64_t)nfine) ++bits;
  size_t tb1 = 0, tb2 = 0, tb3 = 0;
  cub::DeviceRadixSort::SortPairs(nullptr, tb1, keys, keys_s, vals, perm, n, 0, bits, st);
  cub::DeviceScan::ExclusiveSum(nullptr, tb2, cnt, cstart, (int)nfine + 1, st);
  auto fin = thrust::make_transform_iterator((const uint8_t *)flags, FlagCounts());
  auto fout = thrust::make_transform_output_iterator(
      thrust::make_zip_iterator(thrust::make_tuple(cidx, lidx)), SplitCounts());
  cub::DeviceScan::ExclusiveSum(nullptr, tb3, fin, fout, (int)ntot + 1, st);
  size_t tb = std::max(tb1, std::max(tb2, tb3));
  DUST_TRY(grow(o->cub_tmp, tb));
  if (n > 0) {
    DUST_CUDA(cub::DeviceRadixSort::SortPairs(o->cub_tmp.p, tb, keys, keys_s, vals, perm, n,
                                              0, bits, st));
  }
  DUST_CUDA(cub::DeviceScan::ExclusiveSum(o->cub_tmp.p, tb, cnt, cstart, (int)nfine + 1, st));
  double *P = (double *)o->part.p;
  if (n > 0) k_gather<<<nblk(n, 256), 256, 0, st>>>(n, perm, cen, dir, mag, rv, P);
  // leaf rule
  for (int lb = ll, first = 1; first || lb > 1; first = 0) {
    const int lt = std::max(1, lb - 3);
    k_flags<<<nblk(G.ncell[lb], FLG_C), FLG_T, 0, st>>>(G, lb, lt, first != 0, cstart,
                                                       o->prm.min_octree_part, flags);
    lb = lt;
  }
  int *perr = (int *)(small + 41);
  if (n_pts > 0) k_mark_points<<<nblk(n_pts, 128), 128, 0, st>>>(G, n_pts, pts, flags, perr);
  DUST_CUDA(cub::DeviceScan::ExclusiveSum(o->cub_tmp.p, tb, fin, fout, (int)ntot + 1, st));
  k_level_counts<<<1, 32, 0, st>>>(G, cidx, lidx, small);
  int64_t hsmall[64];
  DUST_CUDA(cudaMemcpyAsync(hsmall, small, sizeof(hsmall), cudaMemcpyDeviceToHost, st));
  DUST_CUDA(cudaStreamSynchronize(st));
  int herr, hperr;
  memcpy(&herr, &hsmall[40], sizeof(int));
  memcpy(&hperr, &hsmall[41], sizeof(int));
  o->near_seen = (unsigned long long)hsmall[52];  // of the evaluation before
  if (hsmall[50]) {  // of the previous evaluation: a bounded wait of its M2L gave up
    DUST_CUDA(cudaMemsetAsync(small + 48, 0, 4 * sizeof(int64_t), st));
    dust_set_last_error("a wait in the previous M2L gave up", __FILE__, __LINE__);
    return DUST_ERR_TIMEOUT;
  }
  if (herr != 0x7fffffff) {
    o->bad_particle = herr;
    return DUST_ERR_OUT_OF_BOX;
  }
  if (hperr != 0x7fffffff) {
    dust_set_last_error("an evaluation point lies outside the octree box", __FILE__, __LINE__);
    return DUST_ERR_OUT_OF_BOX;
  }
  o->n_leaves = hsmall[0];
  for (int l = 1; l <= ll + 1; ++l) o->act_off[l] = hsmall[l];
  o->n_active = o->act_off[ll + 1];
  const int64_t nact = o->n_active;
  DUST_TRY(grow(o->act_key, (size_t)std::max<int64_t>(nact, 1) * 4));
  DUST_TRY(grow(o->act_lev, (size_t)std::max<int64_t>(nact, 1)));
  DUST_TRY(grow(o->leaf_ci, (size_t)std::max<int64_t>(o->n_leaves, 1) * 4));
  size_t nmp = (size_t)3 * (2 * o->nm + o->nm1);
  DUST_TRY(grow(o->mp, (size_t)std::max<int64_t>(nact, 1) * nmp * 8));
  k_compact<<<nblk(ntot, 256), 256, 0, st>>>(G, ntot, flags, cidx, lidx, cstart,
                                             (uint32_t *)o->act_key.p, (uint8_t *)o->act_lev.p,
                                             (uint32_t *)o->leaf_ci.p, (uint32_t *)o->srcix.p);
  FmmDev d;
  fill_dev(o, d, n);
  d.cstart = cstart;
  d.perm = perm;
  d.P = P;
  d.flags = flags;
  d.cidx = cidx;
  d.act_key = (const uint32_t *)o->act_key.p;
  d.act_lev = (const uint8_t *)o->act_lev.p;
  d.leaf_ci = (const uint32_t *)o->leaf_ci.p;
  d.n_leaves = (uint32_t)o->n_leaves;
  double *mp = (double *)o->mp.p;
  d.A = mp;
  d.B = mp + (size_t)nact * 3 * o->nm;
  d.Gx = mp + (size_t)nact * 3 * 2 * o->nm;
  d.out = (double *)o->outs.p;
  o->dev = d;
  if (o->timing) cudaEventRecord(o->ev[1], st);
  // upward pass
  DUST_CUDA(cudaMemsetAsync(d.A, 0, (size_t)nact * 3 * (2 * o->nm + o->nm1) * 8, st));
  d.counters = (int64_t *)(small + 48);
  DUST_CUDA(cudaMemsetAsync(d.counters, 0, 4 * sizeof(int64_t), st));
  o->dev = d;
  DUST_TRY(m2l_prepare(o, d, st));
  o->dev = d;
  if (o->n_leaves > 0) {
    const size_t shm = (size_t)P2M_W * (3 * (o->p + 1) + 3) * P2M_LD * 8;
    k_p2m<<<(unsigned)((o->n_leaves + P2M_W - 1) / P2M_W), P2M_W * 32, shm, st>>>(d);
  }
  for (int l = ll - 1; l >= 1; --l) {
    int64_t na = o->act_off[l + 1] - o->act_off[l];
    if (na > 0) {
      const int nt = o->shift_n[l][0];
      const size_t shm = (size_t)SH_W * 8 * 3 * o->nm * 8 + (size_t)nt * sizeof(ShiftTerm) +
                         (size_t)(o->nm + 1) * 4;
      if (shm > 48 * 1024)
        DUST_CUDA(cudaFuncSetAttribute(k_m2m_t, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)shm));
      k_m2m_t<<<shift_grid(na), SH_T, shm, st>>>(d, l, (uint32_t)o->act_off[l], (uint32_t)na,
                                                  (const ShiftTerm *)o->shift_t[l][0],
                                                  (const int *)o->shift_o[l][0], nt);
    }
  }
  if (o->timing) cudaEventRecord(o->ev[2], st);
  // downward pass: M2L of every level (level 1 per target, levels >= 2 in
  // one batched launch), then L2L level by level adds the parents' final
  // local expansions (mod_octree.f90:1074-1125 in another, equivalent order:
  // both are sums of the same terms)
  {
    int64_t na1 = o->act_off[2 <= ll ? 2 : ll + 1] - o->act_off[1];
    if (na1 > 0)
      k_m2l_1<<<(unsigned)na1, M1_T, 0, st>>>(d, (uint32_t)o->act_off[1]);
  }
  DUST_TRY(m2l_all_levels(o, d, st));
  for (int l = 2; l <= ll; ++l) {
    int64_t na = o->act_off[l + 1] - o->act_off[l];
    if (na <= 0) continue;
    const int ntb = o->shift_n[l][1], ntg = d.use_vs ? o->shift_n[l][2] : 0;
    const int nmx = ntg > 0 ? o->nm1 : o->nm;
    const size_t shm = (size_t)SH_W * 3 * nmx * 8 + (size_t)std::max(ntb, ntg) * sizeof(ShiftTerm) +
                       (size_t)(8 * nmx + 1) * 4;
    if (shm > 48 * 1024)
      DUST_CUDA(cudaFuncSetAttribute(k_l2l_t, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                     (int)shm));
    const int64_t npar = o->act_off[l] - o->act_off[l - 1];
    k_l2l_t<<<dim3(shift_grid(npar), ntg > 0 ? 2 : 1), SH_T, shm, st>>>(
        d, l, (uint32_t)o->act_off[l - 1], (uint32_t)npar, (const ShiftTerm *)o->shift_t[l][1],
        (const int *)o->shift_o[l][1], ntb, (const ShiftTerm *)o->shift_t[l][2],
        (const int *)o->shift_o[l][2], ntg);
  }
  if (o->timing) cudaEventRecord(o->ev[3], st);
  o->dev = d;
  o->prepared_n = n;
  o->prepared_pts = n_pts;
  DUST_CUDA(cudaGetLastError());
  return DUST_OK;
}

// leaves: L2P + P2P of the particles with the prepared tree and expansions
int fmm_near_device(dust_octree *o, cudaStream_t st) {
  FmmDev &d = o->dev;
  o->last_stream = st;
  if (o->timing) cudaEventRecord(o->ev[10], st);
  if (o->n_leaves > 0) {
    bool vs = d.use_vs, df = d.use_df, vd = d.use_vd, tv = o->prm.turbulent_viscosity != 0;
    const bool f32 = o->prm.precision == DUST_PREC_FP32C;
    // an item's iterations: short ones where the leaves alone would not fill
    // the resident warps twice, since then the longest item is the time
    // (3,000 particles: 57 us with 64, 90 with 128, 139 with 256); else long
    // enough that listing the ranges again for every item costs little (110k:
    // 1.28 ms with 256, 1.36 with 512, 1.47 with 1024)
    const bool small = o->n_leaves < 2 * P2W_XB;
    P2PItems w;
    w.it = small ? 64 : 256;
    w.cap = P2W_CAP;
    DUST_TRY(grow(o->p2p_work, 256 + (size_t)P2W_CAP * sizeof(uint4) + (size_t)o->n_leaves));
    w.count = (unsigned long long *)o->p2p_work.p;
    w.item = (uint4 *)((char *)o->p2p_work.p + 256);
    w.split = (uint8_t *)(w.item + P2W_CAP);
    DUST_CUDA(cudaMemsetAsync(w.count, 0, 16, st));
    k_p2p_split<<<nblk(o->n_leaves, 8), 256, 0, st>>>(d, w);
    const unsigned grid = (unsigned)(P2W_XB + o->n_leaves);
#define LAUNCH_P2P(A, B, C, D)                                                   \
  do {                                                                         \
    if (f32)                                                                   \
      k_p2p_w<A, B, C, D, true><<<grid, 32, 0, st>>>(d, w);                    \
    else                                                                       \
      k_p2p_w<A, B, C, D, false><<<grid, 32, 0, st>>>(d, w);                   \
  } while (0)
    if (vs && df && vd && !tv) LAUNCH_P2P(true, true, true, false);
    else if (vs && df && vd && tv) LAUNCH_P2P(true, true, true, true);
    else if (vs && df && !vd) LAUNCH_P2P(true, true, false, false);
    else if (vs && !df && vd && !tv) LAUNCH_P2P(true, false, true, false);
    else if (vs && !df && vd && tv) LAUNCH_P2P(true, false, true, true);
    else if (vs && !df && !vd) LAUNCH_P2P(true, false, false, false);
    else if (!vs && vd && !tv) LAUNCH_P2P(false, false, true, false);
    else if (!vs && vd && tv) LAUNCH_P2P(false, false, true, true);
    else LAUNCH_P2P(false, false, false, false);
#undef LAUNCH_P2P
  }
  if (o->timing) cudaEventRecord(o->ev[4], st);
  DUST_CUDA(cudaGetLastError());
  return DUST_OK;
}

int fmm_run_device(dust_octree *o, int n, const double *cen, const double *dir,
                   const double *mag, const double *rv, cudaStream_t st) {
  DUST_TRY(fmm_prepare_device(o, n, cen, dir, mag, rv, 0, nullptr, st));
  return fmm_near_device(o, st);
}

// ----------------------------------------------- particles -> points (FMM)
// apply_multipole_panels (mod_octree.f90:1433-1508) on the GPU: one thread
// per point.  The point is binned into the finest cell as sort_particles
// bins panel centres (:776-799) and takes the leaf above that cell (the
// leaves partition the box); its velocity is the leaf's local expansion
// (FP64 L2P of b) plus the particles of the leaf's 26 active same-level
// neighbours, of its coarser leaf neighbours (leaf_neigh) and of the leaf
// itself, summed in FP64 with the particle kernel of compute_vel
// (mod_vortpart.f90:139-155).  A point outside the octree box sets the
// error word (the reference stops there).
__global__ void k_points_fmm(FmmDev d, int npts, const double *__restrict__ pts,
                             double *__restrict__ uv, int *err) {
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= npts) return;
  const TreeGeom &G = d.G;
  const int ll = G.ll;
  const size_t n = d.n;
  const double pos[3] = {pts[3 * (size_t)q], pts[3 * (size_t)q + 1], pts[3 * (size_t)q + 2]};
  int idx[3];
  for (int c = 0; c < 3; ++c) {
    idx[c] = (int)ceil((pos[c] - G.xmin[c]) / G.csize[ll]) - 1;
    if (idx[c] < 0 || idx[c] >= G.ncl[ll][c]) {
      atomicMin(err, q);
      for (int e = 0; e < 3; ++e) uv[3 * (size_t)q + e] = 0.0;
      return;
    }
  }
  int l = 0, ci = 0, cj = 0, ck = 0;
  uint32_t key = 0;
  for (int lv = 1; lv <= ll; ++lv) {
    const int sh = ll - lv;
    const int a = idx[0] >> sh, b = idx[1] >> sh, c = idx[2] >> sh;
    const uint32_t k = key_of(G, lv, a, b, c);
    if (d.flags[G.lev_off[lv] + k] & FL_LEAF) {
      l = lv, ci = a, cj = b, ck = c, key = k;
      break;
    }
  }
  double v[3] = {0.0, 0.0, 0.0};
  if (l > 0) {
    const uint32_t cell = d.cidx[G.lev_off[l] + key];
    double cc[3];
    cell_center(G, l, ci, cj, ck, cc);
    const double x = pos[0] - cc[0], y = pos[1] - cc[1], z = pos[2] - cc[2];
    const double *bl = d.B + (size_t)cell * 3 * d.nm;
    for (int m = 0; m < d.nm; ++m) {
      int mi, mj, mk;
      mono_exp(m, mi, mj, mk);
      double pr = 1.0;
      for (int e = 0; e < mi; ++e) pr *= x;
      for (int e = 0; e < mj; ++e) pr *= y;
      for (int e = 0; e < mk; ++e) pr *= z;
      for (int e = 0; e < 3; ++e) v[e] += bl[3 * m + e] * pr;
    }
    const double k4pi = 1.0 / (4.0 * DUST_PI);
    auto range = [&](uint32_t lo, uint32_t hi) {
      for (uint32_t t = lo; t < hi; ++t) {
        const double dx = pos[0] - d.P[t], dy = pos[1] - d.P[n + t], dz = pos[2] - d.P[2 * n + t];
        const double ax = d.P[3 * n + t], ay = d.P[4 * n + t], az = d.P[5 * n + t],
                     s = d.P[6 * n + t];
        const double dn = sqrt(dx * dx + dy * dy + dz * dz + s * s);
        const double c = -1.0 / (dn * dn * dn) * k4pi;
        v[0] += c * (dy * az - dz * ay);
        v[1] += c * (dz * ax - dx * az);
        v[2] += c * (dx * ay - dy * ax);
      }
    };
    for (int lev = l; lev >= 1; --lev) {
      const int sh = l - lev;
      const int ai = ci >> sh, aj = cj >> sh, ak = ck >> sh;
      for (int kk = -1; kk <= 1; ++kk)
        for (int jj = -1; jj <= 1; ++jj)
          for (int ii = -1; ii <= 1; ++ii) {
            if (ii == 0 && jj == 0 && kk == 0) continue;
            if (!cart_in(G, lev, ai + ii, aj + jj, ak + kk)) continue;
            const uint32_t nk = key_of(G, lev, ai + ii, aj + jj, ak + kk);
            const uint8_t f = d.flags[G.lev_off[lev] + nk];
            if (lev == l ? !(f & FL_ACTIVE) : !(f & FL_LEAF)) continue;
            range(cell_lo(G, d.cstart, lev, nk), cell_hi(G, d.cstart, lev, nk));
          }
    }
    range(cell_lo(G, d.cstart, l, key), cell_hi(G, d.cstart, l, key));
  }
  for (int e = 0; e < 3; ++e) uv[3 * (size_t)q + e] = v[e];
}

void points_lines_add(int npts, const double *pts, const ElemDev &lines, double *uv,
                      cudaStream_t st);

int fmm_points_uvort_device(dust_octree *o, const ElemDev &lines, double *uv, cudaStream_t st) {
  const int n_pts = o->prepared_pts;
  if (o->prepared_n < 0) return DUST_ERR_BAD_ARG;
  if (n_pts <= 0) return DUST_OK;
  const double *pts = (const double *)o->h_pts.p;
  int *err = (int *)((int64_t *)o->small.p + 42);
  const int big = 0x7fffffff;
  DUST_CUDA(cudaMemcpyAsync(err, &big, sizeof(int), cudaMemcpyHostToDevice, st));
  k_points_fmm<<<nblk(n_pts, 128), 128, 0, st>>>(o->dev, n_pts, pts, uv, err);
  if (lines.nline > 0) points_lines_add(n_pts, pts, lines, uv, st);
  int herr = big;
  DUST_CUDA(cudaMemcpyAsync(&herr, err, sizeof(int), cudaMemcpyDeviceToHost, st));
  DUST_CUDA(cudaStreamSynchronize(st));
  if (herr != big) {
    dust_set_last_error("a point lies outside the octree box", __FILE__, __LINE__);
    return DUST_ERR_OUT_OF_BOX;
  }
  return DUST_OK;
}

int fmm_finish_device(dust_octree *o, int n, const ElemDev &e, double *vel, double *str,
                      double *rot, cudaStream_t st) {
  if (n > 0)
    DUST_TRY(elem_output_device(o->dev, e, o->ffbuf, o->near_buf, o->near_limit, o->near_seen,
                                (unsigned long long *)o->small.p + 52, o->prm.precision, vel, str,
                                rot, st, o->timing ? &o->ev[8] : nullptr, &o->kev_far));
  if (o->timing) cudaEventRecord(o->ev[5], st);
  DUST_CUDA(cudaGetLastError());
  return DUST_OK;
}

int fmm_collect_stats(dust_octree *o, int n, int64_t n_elem) {
  dust_fmm_stats &s = o->stats;
  memset(&s, 0, sizeof(s));
  cudaStreamSynchronize(o->last_stream);
  int status = DUST_OK;
  if (o->dev.counters) {
    int64_t c[4] = {0, 0, 0, 0};
    cudaMemcpy(c, o->dev.counters, sizeof(c), cudaMemcpyDeviceToHost);
    s.n_m2l_pairs = c[0];
    s.n_p2p_pairs = c[1];
    if (c[2]) status = DUST_ERR_TIMEOUT;  // a bounded wait of the M2L gave up
  }
  s.n_particles = n;
  s.n_leaves = o->n_leaves;
  s.n_active_cells = o->n_active;
  s.n_levels = o->G.ll;
  s.n_elem_pairs = (int64_t)n * n_elem;
  if (o->timing) {
    cudaEventSynchronize(o->ev[5]);
    cudaEventElapsedTime(&s.ms_tree, o->ev[0], o->ev[1]);
    cudaEventElapsedTime(&s.ms_upward, o->ev[1], o->ev[2]);
    cudaEventElapsedTime(&s.ms_m2l, o->ev[2], o->ev[3]);
    cudaEventElapsedTime(&s.ms_p2p, o->ev[10], o->ev[4]);
    cudaEventElapsedTime(&s.ms_elems, o->ev[4], o->ev[5]);
    float t_pre = 0.f, t_post = 0.f;
    cudaEventElapsedTime(&t_pre, o->ev[0], o->ev[3]);
    cudaEventElapsedTime(&t_post, o->ev[10], o->ev[5]);
    s.ms_total = t_pre + t_post;
    if (o->kev_m2l) cudaEventElapsedTime(&s.ms_m2l_kernel, o->ev[6], o->ev[7]);
    if (o->kev_far) cudaEventElapsedTime(&s.ms_elem_far, o->ev[8], o->ev[9]);
  }
  return status;
}
