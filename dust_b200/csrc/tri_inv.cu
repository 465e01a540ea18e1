// tri_inv.cu -- triangular solves by blocks whose inverses are kept.
//
// The unpivoted LU (lu_np.cu) leaves the inverse triangles of its 64 x 64
// diagonal blocks.  lu_inv_build merges them into the inverses of TI_B x TI_B
// diagonal blocks of L and U, doubling the size level by level,
//   [L11 0; L21 L22]^-1 = [L11^-1 0; -L22^-1 (L21 L11^-1) L22^-1]
// (and the mirror image for U), every pair of a level in one launch.  A solve
// is then, per block, a product with the inverse and an update of the rows
// not yet solved: 2 n / TI_B dependent launches instead of a chain over n / 64
// blocks (one cooperative kernel with a grid barrier per block, 20 us each) or
// over every row (the library's trsv).  n = 16,384, 64 right-hand sides, FP32:
// 10.3 -> 2.8 ms per solve (L and U), 0.4 ms to build the inverses; one
// right-hand side FP64: n = 3,001 1.83 -> 0.08 ms, 6,954 1.04 -> 0.2 ms, 12,000
// 1.72 -> 0.7 ms, 400 56 -> 12 us.
#include <algorithm>
#include <vector>

#include "lu.cuh"

// A product with the inverse of a triangular block T leaves a residual of up to
// cond(T) = || |T^-1| |T| ||_inf times a substitution's.  Certified factors
// (multipliers below 1) do not bound it: multipliers of -0.1 alone make it grow like
// 1.1^512.  So lu_inv_build measures it, and above TI_COND a solve takes the
// 64 x 64 inverses that the factorisation itself used (or the caller
// substitutes).  Panels' systems have 1.1 to 6 (ellipsoids, rotor and fuselage,
// their Schur complements), where both ways have the same backward errors; at 700
// a solve by the large blocks has ten times the substitution's, at 2e4 a hundred
// times.  An FP32 solve is refined, and a sweep gains digits as long as
// cond(T) 6e-8 is small.  (A system above the limit, n = 3,001 with 16 right-hand
// sides: 4.1 ms with the small blocks, 8.4 with the library's substitution.)
#define TI_B 512
#define TI_T 64   // tile edge of the products
#define TI_K 32   // inner dimension staged at once
#define TI_NT 256
template <typename T>
constexpr float TI_COND = sizeof(T) == 8 ? 64.f : 1e4f;

static inline int ti_blocks(int n) { return (n + TI_B - 1) / TI_B; }

// ------------------------------------------------------------ 64 x 64 products
// acc (4 x TN per thread, rows 4 ty .., columns TN tx ..) += A(:, k0 .. k1) B(k0 ..
// k1, :) of column-major operands; mr / nc valid rows and columns.  The next
// slice is loaded into registers while this one is multiplied.  Bound by shared
// memory if it is read word by word (eight reads, half of them in two-way
// conflicts, for 16 products: a quarter of the FP32 rate), so operands are read
// and B's slice is stored as vectors of four.
template <typename T, int TN>
struct TiSmem {
  alignas(16) T a[TI_K][TI_T + 4];
  alignas(16) T b[TI_K][16 * TN + 4];
};
__device__ __forceinline__ void ti_ld(const float *s, float (&v)[4]) {
  const float4 x = *(const float4 *)s;
  v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
}
__device__ __forceinline__ void ti_ld(const double *s, double (&v)[4]) {
  const double2 x = *(const double2 *)s, y = *(const double2 *)(s + 2);
  v[0] = x.x, v[1] = x.y, v[2] = y.x, v[3] = y.y;
}
__device__ __forceinline__ void ti_ld(const float *s, float (&v)[2]) {
  const float2 x = *(const float2 *)s;
  v[0] = x.x, v[1] = x.y;
}
__device__ __forceinline__ void ti_ld(const double *s, double (&v)[2]) {
  const double2 x = *(const double2 *)s;
  v[0] = x.x, v[1] = x.y;
}
template <typename T>
__device__ __forceinline__ void ti_ld(const T *s, T (&v)[1]) {
  v[0] = *s;
}
__device__ __forceinline__ void ti_st(float *s, const float *v) {
  *(float4 *)s = make_float4(v[0], v[1], v[2], v[3]);
}
__device__ __forceinline__ void ti_st(double *s, const double *v) {
  *(double2 *)s = make_double2(v[0], v[1]);
  *(double2 *)(s + 2) = make_double2(v[2], v[3]);
}

template <typename T, int TN>
__device__ __forceinline__ void ti_mm(TiSmem<T, TN> &s, const T *A, int lda, int mr, const T *B,
                                      int ldb, int nc, int k0, int k1, T (&acc)[4][TN]) {
  // B: a thread takes four columns of one k (TN = 1: half of the threads)
  constexpr int NA = TI_K * TI_T / TI_NT, NG = (4 * TN + 7) / 8;
  const int tid = threadIdx.x, ty = tid / 16, tx = tid % 16;
  const int ar = tid % TI_T, ak = tid / TI_T, bk = tid % TI_K, bc = 4 * (tid / TI_K);
  T av[NA], bv[NG][4];
  auto fetch = [&](int k) {
#pragma unroll
    for (int q = 0; q < NA; ++q) {
      const int kk = k + ak + q * (TI_NT / TI_T);
      av[q] = (ar < mr && kk < k1) ? A[(size_t)ar + (size_t)kk * lda] : (T)0;
    }
#pragma unroll
    for (int q = 0; q < NG; ++q)
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        const int c = bc + 32 * q + v;
        bv[q][v] = (c < nc && c < 16 * TN && k + bk < k1)
                       ? B[(size_t)(k + bk) + (size_t)c * ldb]
                       : (T)0;
      }
  };
  fetch(k0);
  for (int k = k0; k < k1; k += TI_K) {
    __syncthreads();
#pragma unroll
    for (int q = 0; q < NA; ++q) s.a[ak + q * (TI_NT / TI_T)][ar] = av[q];
#pragma unroll
    for (int q = 0; q < NG; ++q)
      if (bc + 32 * q < 16 * TN) ti_st(&s.b[bk][bc + 32 * q], bv[q]);
    __syncthreads();
    if (k + TI_K < k1) fetch(k + TI_K);
#pragma unroll 8
    for (int p = 0; p < TI_K; ++p) {
      T x[4], y[TN];
      ti_ld(&s.a[p][4 * ty], x);
      ti_ld(&s.b[p][TN * tx], y);
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < TN; ++v) acc[u][v] = fma(x[u], y[v], acc[u][v]);
    }
  }
}

// ------------------------------------------------------------ inverse blocks
// block i: Linv then Uinv, TI_B x TI_B each, zero outside their triangles
template <typename T>
__device__ __host__ __forceinline__ T *ti_linv(T *inv, int i) {
  return inv + (size_t)2 * TI_B * TI_B * i;
}

// the 64 x 64 inverses onto the diagonals, zeros elsewhere
template <typename T>
__global__ void k_ti_init(int n, const T *np, T *inv) {
  const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  const size_t per = (size_t)TI_B * TI_B;
  if (e >= 2 * per * (size_t)((n + TI_B - 1) / TI_B)) return;
  const int i = (int)(e / (2 * per)), up = (int)(e / per) & 1;
  const int r = (int)(e % TI_B), c = (int)(e / TI_B % TI_B);
  T v = (T)0;
  if (r / 64 == c / 64 && i * TI_B + r < n && i * TI_B + c < n) {
    const T *b = np + (size_t)2 * 4096 * (i * (TI_B / 64) + r / 64) + (up ? 4096 : 0);
    const int rr = r % 64, cc = c % 64;
    if (up ? rr <= cc : rr >= cc) v = b[rr + 64 * cc];
  }
  inv[e] = v;
}

// one phase of level s: blockIdx.y = pair (s rows and s more), blockIdx.z = 0
// for L, 1 for U, blockIdx.x = 64 x 64 tile of the s x s product.
//   phase 0: T = L21 L11^-1          T = U12 U22^-1
//   phase 1: X21 = -L22^-1 T         X12 = -U11^-1 T
template <typename T>
__global__ void __launch_bounds__(TI_NT) k_ti_merge(int n, int s, int phase, const T *A, int lda,
                                                    T *inv, T *tmp) {
  __shared__ TiSmem<T, 4> sm;
  const int per = TI_B / (2 * s), blk = blockIdx.y / per, a = (blockIdx.y % per) * 2 * s;
  const int up = blockIdx.z, nt = s / TI_T, r0 = blockIdx.x % nt * TI_T,
            c0 = blockIdx.x / nt * TI_T;
  const int k = blk * TI_B;
  if (k + a + s >= n) return;  // the pair's second half is empty
  T *I = ti_linv(inv, blk) + (up ? (size_t)TI_B * TI_B : 0);
  T *X = tmp + ((size_t)blockIdx.y * 2 + up) * s * s;
  T *I1 = I + a + (size_t)a * TI_B, *I2 = I + (a + s) + (size_t)(a + s) * TI_B;
  const int n2 = min(s, n - k - a - s);  // rows of the second half
  T acc[4][4] = {};
  if (phase == 0) {
    const T *M = up ? A + (size_t)(k + a) + (size_t)(k + a + s) * lda
                    : A + (size_t)(k + a + s) + (size_t)(k + a) * lda;
    const T *W = up ? I2 : I1;
    const int m = up ? s : n2, kk = up ? n2 : s;
    // (columns of a lower W start at their own row, of an upper one end there)
    ti_mm<T, 4>(sm, M + r0, lda, m - r0, W + (size_t)c0 * TI_B, TI_B, TI_T, up ? 0 : c0,
                up ? min(kk, c0 + TI_T) : kk, acc);
  } else {
    const T *W = up ? I1 : I2;
    ti_mm<T, 4>(sm, W + r0, TI_B, TI_T, X + (size_t)c0 * s, s, TI_T, up ? r0 : 0,
                up ? s : r0 + TI_T, acc);
  }
  T *out = phase == 0 ? X : (up ? I + a + (size_t)(a + s) * TI_B : I + (a + s) + (size_t)a * TI_B);
  const int ldo = phase == 0 ? s : TI_B;
  const int ty = threadIdx.x / 16, tx = threadIdx.x % 16;
#pragma unroll
  for (int v = 0; v < 4; ++v)
#pragma unroll
    for (int u = 0; u < 4; ++u)
      out[(size_t)(r0 + 4 * ty + u) + (size_t)(c0 + 4 * tx + v) * ldo] =
          phase == 0 ? acc[u][v] : -acc[u][v];
}

// cond(T) of every block (blockIdx.y) of L (blockIdx.z = 0) and U (1): a CTA
// takes 32 rows (lanes), its 8 warps the columns, 16 loads in flight per thread.
// Phase 0 writes w = |T| 1, phase 1 the largest (|T^-1| w)_r (float bits, infinity
// where it is no number).
template <typename T>
__global__ void __launch_bounds__(TI_NT) k_ti_cond(int n, int phase, const T *A, int lda, T *inv,
                                                   double *w, unsigned *bits) {
  __shared__ double s_s[TI_NT / 32][32];
  const int lane = threadIdx.x & 31, g = threadIdx.x >> 5, r = 32 * blockIdx.x + lane;
  const int k = TI_B * blockIdx.y, m = min(TI_B, n - k), up = blockIdx.z;
  w += (size_t)(2 * blockIdx.y + up) * TI_B;
  const T *M = phase == 0 ? A + (size_t)k + (size_t)k * lda
                          : ti_linv(inv, blockIdx.y) + (up ? (size_t)TI_B * TI_B : 0);
  const size_t ld = phase == 0 ? lda : TI_B;
  double s = 0.0;
  for (int c0 = g; c0 < m; c0 += 16 * (TI_NT / 32)) {
    double v[16];
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const int c = c0 + q * (TI_NT / 32);
      // (L's diagonal: 1)
      const bool in = r < m && c < m && (up ? c >= r : c < r);
      v[q] = in ? fabs((double)M[r + c * ld]) : (c == r ? 1.0 : 0.0);
    }
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const int c = c0 + q * (TI_NT / 32);
      if (c < m) s += phase == 0 ? v[q] : v[q] * w[c];
    }
  }
  s_s[g][lane] = s;
  __syncthreads();
  if (g > 0) return;
  for (int q = 1; q < TI_NT / 32; ++q) s += s_s[q][lane];
  if (phase == 0) {
    if (r < m) w[r] = s;
    return;
  }
  float f = s <= 3.0e38 ? (float)s : INFINITY;
  for (int o = 16; o > 0; o >>= 1) f = fmaxf(f, __shfl_xor_sync(~0u, f, o));
  if (lane == 0) atomicMax(bits, __float_as_uint(f));
}

template <typename T>
int lu_inv_build(cudaStream_t st, LuWork &w, int n, const T *A, int lda) {
  w.inv_n = 0;
  w.inv_ok = false;
  if (n <= 0) return DUST_OK;
  const int nb = ti_blocks(n);
  const size_t per = (size_t)2 * TI_B * TI_B * nb;
  // (the largest level's temporaries: s^2 for L and U of every pair, s = TI_B / 2)
  DUST_TRY(devbuf_grow(w.inv, (per + per / 4) * sizeof(T)));
  T *inv = (T *)w.inv.p, *tmp = inv + per;
  const T *np = (const T *)((const char *)w.np.p + 256);
  unsigned *bits = (unsigned *)w.np.p + 1;
  DUST_CUDA(cudaMemsetAsync(bits, 0, sizeof(unsigned), st));
  k_ti_init<T><<<(unsigned)((per + 255) / 256), 256, 0, st>>>(n, np, inv);
  for (int s = 64; s < TI_B && s < n; s *= 2)
    for (int ph = 0; ph < 2; ++ph)
      k_ti_merge<T><<<dim3((s / TI_T) * (s / TI_T), nb * (TI_B / (2 * s)), 2), TI_NT, 0, st>>>(
          n, s, ph, A, lda, inv, tmp);
  for (int ph = 0; ph < 2; ++ph)  // (tmp: the merges are done with it)
    k_ti_cond<T><<<dim3((std::min(TI_B, n) + 31) / 32, nb, 2), TI_NT, 0, st>>>(
        n, ph, A, lda, inv, (double *)tmp, bits);
  DUST_CUDA(cudaGetLastError());
  float cond = INFINITY;
  DUST_CUDA(cudaMemcpyAsync(&cond, bits, sizeof(float), cudaMemcpyDeviceToHost, st));
  DUST_CUDA(cudaStreamSynchronize(st));
  w.inv_n = n;
  w.inv_ok = cond <= TI_COND<T>;
  return DUST_OK;
}

// ------------------------------------------------------------ block solves
// Where few tiles would leave SMs idle, the inner dimension of a product is
// shared among CTAs: each writes its partial tile, and the last one to arrive
// (a counter per tile, no waiting) adds them in the shares' order, so that a
// solve repeated on the same data gives the same bits.
#define TI_PART 320  // most tiles x shares with more than one share

template <typename T>
struct TiPart {
  T *part;       // [tile x share][4096]
  int *arrived;  // per tile, zero between launches
};

__device__ __forceinline__ bool ti_last(int *arrived, int shares) {
  __shared__ int s_last;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0) s_last = atomicAdd(arrived, 1) == shares - 1;
  __syncthreads();
  if (s_last) {
    __threadfence();
    if (threadIdx.x == 0) *arrived = 0;
  }
  return s_last;
}

// C (m x nr) += alpha A (m x k) B (k x nr), 64-row tiles, blockIdx.y a tile of
// 16 TN right-hand sides, blockIdx.z a share of k.  TRI: A is a block's
// inverse, lower (1) or upper (2) triangular.
template <typename T, int TN, int TRI>
__global__ void __launch_bounds__(TI_NT) k_ti_gemm(int m, int nr, int k, T alpha, const T *A,
                                                   int lda, const T *B, int ldb, T *C, int ldc,
                                                   int kshare, TiPart<T> P) {
  __shared__ TiSmem<T, TN> sm;
  const int r0 = blockIdx.x * TI_T, c0 = blockIdx.y * 16 * TN;
  int k0 = blockIdx.z * kshare, k1 = min(k, k0 + kshare);
  if (TRI == 1) k1 = min(k1, r0 + TI_T);
  if (TRI == 2) k0 = max(k0, r0);
  const int tid = threadIdx.x, ty = tid / 16, tx = tid % 16, Z = gridDim.z;
  T acc[4][TN] = {}, old[4][TN];
  // C's values, all loads in flight together and, without shares, under the
  // product (added one after the other they took longer than the product)
  auto fetch_c = [&]() {
#pragma unroll
    for (int v = 0; v < TN; ++v)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r = r0 + 4 * ty + u, c = c0 + TN * tx + v;
        old[u][v] = (r < m && c < nr) ? C[(size_t)r + (size_t)c * ldc] : (T)0;
      }
  };
  if (Z == 1) fetch_c();
  if (k0 < k1)
    ti_mm<T, TN>(sm, A + r0, lda, m - r0, B + (size_t)c0 * ldb, ldb, nr - c0, k0, k1, acc);
  if (Z > 1) {
    const int tile = blockIdx.x + gridDim.x * blockIdx.y;
    T *mine = P.part + ((size_t)tile * Z + blockIdx.z) * 4096 + tid;
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < TN; ++v) __stcg(mine + TI_NT * (TN * u + v), acc[u][v]);
    if (!ti_last(P.arrived + tile, Z)) return;
    fetch_c();
    const T *all = P.part + (size_t)tile * Z * 4096 + tid;
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < TN; ++v) acc[u][v] = __ldcg(all + TI_NT * (TN * u + v));
#pragma unroll 2
    for (int z = 1; z < Z; ++z)
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < TN; ++v)
          acc[u][v] += __ldcg(all + (size_t)z * 4096 + TI_NT * (TN * u + v));
  }
#pragma unroll
  for (int v = 0; v < TN; ++v)
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int r = r0 + 4 * ty + u, c = c0 + TN * tx + v;
      if (r < m && c < nr) C[(size_t)r + (size_t)c * ldc] = old[u][v] + alpha * acc[u][v];
    }
}

// the same for one right-hand side: 32 rows (lanes) per CTA, the columns of a
// share among its 8 warps, 16 loads in flight per thread
template <typename T, int TRI>
__global__ void __launch_bounds__(TI_NT) k_ti_gemv(int m, int k, T alpha, const T *A, int lda,
                                                   const T *x, T *y, int kshare, TiPart<T> P) {
  __shared__ T s_x[TI_B], s_y[TI_NT / 32][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, r0 = blockIdx.x * 32, r = r0 + lane;
  int k0 = blockIdx.y * kshare, k1 = min(k, k0 + kshare);
  if (TRI == 1) k1 = min(k1, r0 + 32);
  if (TRI == 2) k0 = max(k0, r0);
  for (int c = threadIdx.x; c < k1 - k0; c += TI_NT) s_x[c] = x[k0 + c];
  __syncthreads();
  T s = (T)0;
  const T *a = A + (size_t)r + (size_t)k0 * lda;
  if (r < m)
    for (int c = w; c < k1 - k0; c += 16 * (TI_NT / 32)) {
      T v[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const int cc = c + q * (TI_NT / 32);
        v[q] = cc < k1 - k0 ? a[(size_t)cc * lda] : (T)0;
      }
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const int cc = c + q * (TI_NT / 32);
        if (cc < k1 - k0) s = fma(v[q], s_x[cc], s);
      }
    }
  s_y[w][lane] = s;
  __syncthreads();
  if (w == 0)
#pragma unroll
    for (int q = 1; q < TI_NT / 32; ++q) s += s_y[q][lane];
  const int Z = gridDim.y;
  if (Z > 1) {
    T *all = P.part + (size_t)blockIdx.x * Z * 32 + lane;
    if (w == 0) __stcg(all + blockIdx.y * 32, s);
    if (!ti_last(P.arrived + blockIdx.x, Z)) return;
    if (w == 0) {
      s = __ldcg(all);
      for (int z = 1; z < Z; ++z) s += __ldcg(all + z * 32);
    }
  }
  if (w == 0 && r < m) y[r] += alpha * s;
}

template <typename T, int TRI>
static void ti_mul(cudaStream_t st, const TiPart<T> &P, int m, int nr, int k, T alpha, const T *A,
                   int lda, const T *B, int ldb, T *C, int ldc) {
  if (m <= 0 || nr <= 0 || k <= 0) return;
  // shares of k until two CTAs per SM are busy, of whole slices
  auto share = [&](int tiles, int unit) {
    const int want = std::max(1, 2 * 148 / std::max(tiles, 1));
    return std::max(unit, ((k + want - 1) / want + unit - 1) / unit * unit);
  };
  if (nr == 1) {
    const int bx = (m + 31) / 32, ks = share(bx, 128);
    k_ti_gemv<T, TRI><<<dim3(bx, (k + ks - 1) / ks), TI_NT, 0, st>>>(m, k, alpha, A, lda, B, C, ks,
                                                                    P);
    return;
  }
  const int bx = (m + TI_T - 1) / TI_T, tn = nr <= 16 ? 1 : nr <= 32 ? 2 : 4;
  const int by = (nr + 16 * tn - 1) / (16 * tn), ks = share(bx * by, 64);
  const dim3 g(bx, by, (k + ks - 1) / ks);
  if (tn == 1)
    k_ti_gemm<T, 1, TRI><<<g, TI_NT, 0, st>>>(m, nr, k, alpha, A, lda, B, ldb, C, ldc, ks, P);
  else if (tn == 2)
    k_ti_gemm<T, 2, TRI><<<g, TI_NT, 0, st>>>(m, nr, k, alpha, A, lda, B, ldb, C, ldc, ks, P);
  else
    k_ti_gemm<T, 4, TRI><<<g, TI_NT, 0, st>>>(m, nr, k, alpha, A, lda, B, ldb, C, ldc, ks, P);
}

template <typename T>
int lu_solve_blocks(cudaStream_t st, DevBuf &work, int n, int nrhs, const T *A, int lda, T *B,
                    int ldb, const LuWork &w1, const LuWork *w2) {
  if (n <= 0 || nrhs <= 0) return DUST_OK;
  struct Blk {
    int k, s, ld;          // first row, rows, stride of the inverses
    const T *linv, *uinv;
  };
  std::vector<Blk> bl;
  auto add = [&](const LuWork &w, int base) {
    const int ld = w.inv_ok ? TI_B : 64;
    const T *inv = w.inv_ok ? (const T *)w.inv.p : (const T *)((const char *)w.np.p + 256);
    for (int k = 0; k < w.inv_n; k += ld, inv += 2 * ld * ld)
      bl.push_back({base + k, std::min(ld, w.inv_n - k), ld, inv, inv + ld * ld});
    return base + w.inv_n;
  };
  int end = add(w1, 0);
  if (w2) end = add(*w2, end);
  if (end != n) return DUST_ERR_BAD_ARG;
  const size_t xb = ((size_t)n * nrhs * sizeof(T) + 255) / 256 * 256;
  const size_t pb = nrhs == 1 ? 0 : (size_t)TI_PART * 4096 * sizeof(T);
  // (one right-hand side: tiles x shares of 32 values, counters per 32 rows)
  const size_t tiles = std::max<size_t>(TI_PART, (size_t)n / 32 + 1);
  const size_t gb = nrhs == 1 ? (size_t)TI_PART * 32 * sizeof(T) : 0;
  DUST_TRY(devbuf_grow(work, xb + pb + gb + tiles * sizeof(int)));
  T *X = (T *)work.p;
  TiPart<T> P;
  P.part = (T *)((char *)work.p + xb);
  P.arrived = (int *)((char *)work.p + xb + pb + gb);
  DUST_CUDA(cudaMemsetAsync(P.arrived, 0, tiles * sizeof(int), st));
  // L Y = B: Y into X, the rest of B updated; then U X = Y into B
  DUST_CUDA(cudaMemsetAsync(X, 0, (size_t)n * nrhs * sizeof(T), st));
  for (const Blk &b : bl) {
    ti_mul<T, 1>(st, P, b.s, nrhs, b.s, (T)1, b.linv, b.ld, B + b.k, ldb, X + b.k, n);
    const int r = b.k + b.s;
    ti_mul<T, 0>(st, P, n - r, nrhs, b.s, (T)-1, A + (size_t)r + (size_t)b.k * lda, lda, X + b.k, n,
                 B + r, ldb);
  }
  DUST_CUDA(cudaMemset2DAsync(B, (size_t)ldb * sizeof(T), 0, (size_t)n * sizeof(T), nrhs, st));
  for (size_t q = bl.size(); q-- > 0;) {
    const Blk &b = bl[q];
    ti_mul<T, 2>(st, P, b.s, nrhs, b.s, (T)1, b.uinv, b.ld, X + b.k, n, B + b.k, ldb);
    ti_mul<T, 0>(st, P, b.k, nrhs, b.s, (T)-1, A + (size_t)b.k * lda, lda, B + b.k, ldb, X, n);
  }
  DUST_CUDA(cudaGetLastError());
  return DUST_OK;
}

int lu_trsm_blocks(cublasHandle_t cb, cudaStream_t st, LuWork &w, int n, const double *A, int lda,
                   int m, double *B, double *C, int ldbc) {
  if (n <= 0 || m <= 0) return DUST_OK;
  if (w.inv_n != n || !w.inv_ok || cublasSetStream(cb, st) != CUBLAS_STATUS_SUCCESS)
    return DUST_ERR_BAD_ARG;
  DUST_TRY(devbuf_grow(w.np_x, (size_t)TI_B * m * 8));
  double *X = (double *)w.np_x.p;
  const double one = 1.0, mone = -1.0, zero = 0.0;
  auto gemm = [&](int mm, int nn, int kk, const double *alpha, const double *a, int la,
                  const double *b, int lb, const double *beta, double *c, int lc) -> int {
    if (mm <= 0 || nn <= 0 || kk <= 0) return DUST_OK;
    return cublasDgemm(cb, CUBLAS_OP_N, CUBLAS_OP_N, mm, nn, kk, alpha, a, la, b, lb, beta, c,
                       lc) == CUBLAS_STATUS_SUCCESS
               ? DUST_OK
               : DUST_ERR_CUDA;
  };
  for (int k = 0; k < n; k += TI_B) {
    const int s = std::min(TI_B, n - k), r = k + s;
    const double *li = ti_linv((const double *)w.inv.p, k / TI_B), *ui = li + (size_t)TI_B * TI_B;
    // rows k .. of B: X = Linv B, then the rows below
    DUST_TRY(gemm(s, m, s, &one, li, TI_B, B + k, ldbc, &zero, X, s));
    DUST_CUDA(cudaMemcpy2DAsync(B + k, (size_t)ldbc * 8, X, (size_t)s * 8, (size_t)s * 8, m,
                                cudaMemcpyDeviceToDevice, st));
    DUST_TRY(gemm(n - r, m, s, &mone, A + (size_t)r + (size_t)k * lda, lda, X, s, &one, B + r,
                  ldbc));
    // columns k .. of C: X = C Uinv, then the columns to the right
    DUST_TRY(gemm(m, s, s, &one, C + (size_t)k * ldbc, ldbc, ui, TI_B, &zero, X, m));
    DUST_CUDA(cudaMemcpy2DAsync(C + (size_t)k * ldbc, (size_t)ldbc * 8, X, (size_t)m * 8,
                                (size_t)m * 8, s, cudaMemcpyDeviceToDevice, st));
    DUST_TRY(gemm(m, n - r, s, &mone, X, m, A + (size_t)k + (size_t)r * lda, lda, &one,
                  C + (size_t)r * ldbc, ldbc));
  }
  return DUST_OK;
}

template int lu_inv_build<double>(cudaStream_t, LuWork &, int, const double *, int);
template int lu_inv_build<float>(cudaStream_t, LuWork &, int, const float *, int);
template int lu_solve_blocks<double>(cudaStream_t, DevBuf &, int, int, const double *, int,
                                     double *, int, const LuWork &, const LuWork *);
template int lu_solve_blocks<float>(cudaStream_t, DevBuf &, int, int, const float *, int, float *,
                                    int, const LuWork &, const LuWork *);
