// lu_np.cu -- blocked LU without row interchanges, certified against partial
// pivoting (FP64 and FP32), column-major.
//
// Partial pivoting (LAPACK dgetrf, src/linsys/mod_linsys.f90:230-246,
// :470-474) interchanges rows at column j only when some |a(i,j)|, i > j,
// exceeds the diagonal |a(j,j)| at that point of the elimination.  With no
// interchange the multipliers are l(i,j) = a(i,j) / a(j,j), so the
// factorisation computed without pivoting is partial pivoting's own
// whenever every |l(i,j)| < 1.  The surface-panel influence matrices of this
// solver are of that kind (doublet self-influence 2 pi on the diagonal,
// off-diagonal row sums of about 2 pi on a closed body; dgetrf makes no
// interchange on them).  Without the per-column pivot search the panel
// needs no column-by-column barrier across the matrix and the whole
// factorisation is blocks and GEMMs:
//
//   for each outer panel of NP_NBO columns, for each block column k (NP_NB
//   wide) in it:
//     k_np_diag   one CTA: unpivoted LU of the diagonal block in registers,
//                 its inverse triangles Linv (unit lower) and Uinv (upper) in
//                 the same elimination, max |l| of the block;
//     k_np_panel  L21 = A21 Uinv (row tiles, down to n) and U12 = Linv A12
//                 (column tiles, inside the outer panel), max |l| of L21;
//     k_np_inner  update of the outer panel's own columns;
//   then k_np_cols, the outer panel's U12 right of it, and the trailing update
//   A22 -= L21 U12 of inner dimension NP_NBO (tcgen05 TF32 GEMM for FP32, DGEMM
//   for FP64), which streams the trailing matrix a quarter as often as
//   NP_NB-wide steps.
//
// A panel is a chain of small kernels with one CTA at its core (four times 24 us
// and more), the update fills the chip: the next panel's columns are
// updated first and the panel factored on a second stream of high priority
// under the update of the other columns.  Systems of up to two panels have
// nothing to overlap and stay on the caller's stream.  n = 3,001 in
// FP64: 4.54 -> 3.52 ms with the solve; n = 16,384 in FP32: 47.2 -> 42.0 ms.
//
// The largest |l| is kept as float bits (monotone for non-negative values)
// with atomicMax.  The caller accepts the factors when it is below
// 1 - margin (a margin well above the rounding of the computed multipliers,
// so partial pivoting on the same values would also have kept every
// diagonal); otherwise, and on a zero diagonal, it restores A and runs the
// pivoted factorisation.  ipiv is the identity.
#include <algorithm>
#include <atomic>
#include <cstring>
#include <type_traits>

#include "elements.cuh"
#include "lu.cuh"

#define CUBLAS_CHECK(x)                                                   \
  do {                                                                    \
    if ((x) != CUBLAS_STATUS_SUCCESS) {                                   \
      dust_set_last_error("cuBLAS call failed", __FILE__, __LINE__);      \
      return DUST_ERR_CUDA;                                               \
    }                                                                     \
  } while (0)

#define NP_NB 64
#define NP_NBO 256  // outer panel width (a multiple of NP_NB)
#define NP_T 256

__device__ __forceinline__ void np_note_lmax(unsigned *bits, float v) {
  atomicMax(bits, __float_as_uint(v));
}

// reciprocal pivots: FP64 from the refined approximation (elements.cuh), whose
// chain of dependent operations is a third of a division's
__device__ __forceinline__ double np_rcp(double x) {
  return near_range(fabs(x)) ? rcp_r(x) : 1.0 / x;
}

// Diagonal block: LU and both inverse triangles in one block elimination, in
// FP64 for either element type.  Warp i holds rows 8 i .. 8 i + 7 of W as eight
// 8 x 8 accumulators of the FP64 tensor instruction, W = A at first.  A step
// takes four pivots Q = 4 q .. 4 q + 3.  The warp that holds their rows R = W(Q,:)
// factors W(Q,Q) = L_d U_d, inverts both triangles and leaves R' = L_d^-1 R in
// shared memory; after the step's one barrier every warp forms f = W(:,Q) U_d^-1
// of its rows, and with one instruction per tile
//   rows below Q:  f is L; W(r,c) -= f R'_c for every c outside Q (right of Q
//                  the elimination, left of it the row operations of Linv),
//                  W(r,Q) = -f L_d^-1;
//   rows above Q:  W(r,Q) = f, Uinv's columns; W(r,c) -= f R'_c right of Q;
//   rows Q:        R' is U right of Q and Linv's rows left of it;
//                  W(Q,c) = -U_d^-1 R'_c right of Q, W(Q,Q) the two inverses.
// At the end W holds Linv below the diagonal and Uinv on and above it.  Bound by
// the chain of a step: one warp's rows through shared memory, four dependent
// reciprocals, R', barrier, f, the products.  (Rows and columns Q through shared
// memory to a 4 x 4 piece per thread, every thread factoring the pivot block:
// 160 FP64 instructions a warp and step instead of about 50, 37 us in FP64 and
// 20 us in FP32 per block; 24 us in either now, 28 us beside an update.)
#define NPD_T 256
__device__ __forceinline__ void np_ld4(const double *s, double &a, double &b, double &c,
                                       double &d) {
  const double2 x = *(const double2 *)s, y = *(const double2 *)(s + 2);
  a = x.x, b = x.y, c = y.x, d = y.y;
}
__device__ __forceinline__ void np_ld4(const float *s, float &a, float &b, float &c, float &d) {
  const float4 x = *(const float4 *)s;
  a = x.x, b = x.y, c = x.z, d = x.w;
}
__device__ __forceinline__ void np_st4(double *s, double a, double b, double c, double d) {
  *(double2 *)s = make_double2(a, b);
  *(double2 *)(s + 2) = make_double2(c, d);
}
__device__ __forceinline__ void np_st4(float *s, float a, float b, float c, float d) {
  *(float4 *)s = make_float4(a, b, c, d);
}

__device__ __forceinline__ void np_dmma(double &c0, double &c1, double a, double b) {
  asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
      : "+d"(c0), "+d"(c1)
      : "d"(a), "d"(b));
}
#define NPD_LD (NP_NB + 4)  // the four rows of a B operand in different banks

template <typename T>
__global__ void __launch_bounds__(NPD_T) k_np_diag(T *A, int lda, int k, int jb, T *Linv,
                                                   T *Uinv, unsigned *lmax_bits) {
  __shared__ __align__(16) double s_rp[NP_NB][NPD_LD];  // R' of every step, L_d below its diagonal
  __shared__ __align__(16) double s_raw[4][NP_NB];
  __shared__ __align__(16) double s_iu[2][4][4], s_il[2][4][4];
  const int i = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  T *Ab = A + (size_t)k + (size_t)k * lda;
  double w[8][2];
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int r = 8 * i + g, c = 8 * j + 2 * t + e;
      w[j][e] = (r < jb && c < jb) ? (double)Ab[(size_t)r + (size_t)c * lda] : (r == c ? 1.0 : 0.0);
    }
  if (threadIdx.x < 8) s_il[threadIdx.x & 1][0][threadIdx.x >> 1] = threadIdx.x < 2 ? 1.0 : 0.0;
  float lm = 0.f;
  // the pivot rows of step q, by the warp that holds them
  auto pivots = [&](int q) {
    if ((lane >> 4) == (q & 1)) {
#pragma unroll
      for (int j = 0; j < 8; ++j)
        *(double2 *)&s_raw[g & 3][8 * j + 2 * t] = make_double2(w[j][0], w[j][1]);
    }
    __syncwarp();
    double D[4][4], x[2][4], iu[4][4], il[4][4];
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      np_ld4(&s_raw[u][4 * q], D[u][0], D[u][1], D[u][2], D[u][3]);
      x[0][u] = s_raw[u][lane];
      x[1][u] = s_raw[u][lane + 32];
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      iu[j][j] = np_rcp(D[j][j]);
#pragma unroll
      for (int r = j + 1; r < 4; ++r) {
        D[r][j] *= iu[j][j];
#pragma unroll
        for (int c = j + 1; c < 4; ++c) D[r][c] = fma(-D[r][j], D[j][c], D[r][c]);
        x[0][r] = fma(-D[r][j], x[0][j], x[0][r]);
        x[1][r] = fma(-D[r][j], x[1][j], x[1][r]);
      }
    }
#pragma unroll
    for (int c = 1; c < 4; ++c)
#pragma unroll
      for (int r = c - 1; r >= 0; --r) {
        double y = D[r][c] * iu[c][c];
#pragma unroll
        for (int p = r + 1; p < c; ++p) y = fma(D[r][p], iu[p][c], y);
        iu[r][c] = -y * iu[r][r];
        iu[c][r] = 0.0;
      }
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      il[c][c] = 1.0;
#pragma unroll
      for (int r = c + 1; r < 4; ++r) {
        double y = D[r][c];
#pragma unroll
        for (int p = c + 1; p < r; ++p) y = fma(D[r][p], il[p][c], y);
        il[r][c] = -y;
        il[c][r] = 0.0;
      }
    }
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      s_rp[4 * q + u][lane] = x[0][u];
      s_rp[4 * q + u][lane + 32] = x[1][u];
    }
    if (lane == 0) {
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        np_st4(s_iu[q & 1][u], iu[u][0], iu[u][1], iu[u][2], iu[u][3]);
        if (u > 0) np_st4(s_il[q & 1][u], il[u][0], il[u][1], il[u][2], il[u][3]);
      }
    }
    __syncwarp();
    if (lane == 0) {  // L_d, read at the end only
#pragma unroll
      for (int u = 1; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < u; ++v) s_rp[4 * q + u][4 * q + v] = D[u][v];
    }
  };
  const int nq = (jb + 3) / 4;  // (pivots beyond jb meet the identity and change nothing)
  if (i == 0) pivots(0);
#pragma unroll 1
  for (int q = 0; q < nq; ++q) {
    __syncthreads();
    const int iq = q >> 1, h = q & 1;
    const double(*siu)[4] = s_iu[h], (*sil)[4] = s_il[h];
    // the rows' values in columns Q, from the accumulators' layout
    double v0 = w[0][0], v1 = w[0][1];
#pragma unroll
    for (int j = 1; j < 8; ++j)
      if (j == iq) v0 = w[j][0], v1 = w[j][1];
    const int from = (lane & ~3) + 2 * h;
    const double c0 = __shfl_sync(~0u, v0, from), c1 = __shfl_sync(~0u, v1, from),
                 c2 = __shfl_sync(~0u, v0, from + 1), c3 = __shfl_sync(~0u, v1, from + 1);
    const double f = fma(c0, siu[0][t], c1 * siu[1][t]) + fma(c2, siu[2][t], c3 * siu[3][t]);
    const bool rq = i == iq && (lane >> 4) == h;        // a pivot row
    const bool lower = i > iq || (i == iq && h == 0);   // the warp has rows below Q
    const double a = -(rq ? siu[g & 3][t] : f);
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      if (j < iq && !lower) continue;  // left of Q, no rows below it
      double b = s_rp[4 * q + t][8 * j + g], d0 = w[j][0], d1 = w[j][1];
      if (j == iq) {
        if ((g >> 2) == h)
          b = lower ? sil[t][g & 3] : (t == (g & 3) ? -1.0 : 0.0);
        else if (h == 1 && !lower)
          b = 0.0;
        if ((t >> 1) == h) d0 = d1 = 0.0;
      }
      if (rq && j >= iq) d0 = d1 = 0.0;
      np_dmma(d0, d1, a, b);
      w[j][0] = d0;
      w[j][1] = d1;
    }
    if (q + 1 < nq && i == (q + 1) >> 1) pivots(q + 1);
    // (what the next pivots do not wait for)
    if (lower && !rq) {
      const int r = 8 * i + g, c = 4 * q + t;
      if (r < jb && c < jb) Ab[(size_t)r + (size_t)c * lda] = (T)f;
      lm = fmaxf(lm, fabsf((float)f));
    }
    if (rq) {
      // Linv's rows left of Q and the inverses of the pivot block
#pragma unroll
      for (int j = 0; j < 8; ++j)
        if (j < iq || (j == iq && h == 1 && t < 2)) {
          w[j][0] = s_rp[4 * q + (g & 3)][8 * j + 2 * t];
          w[j][1] = s_rp[4 * q + (g & 3)][8 * j + 2 * t + 1];
        } else if (j == iq && (t >> 1) == h) {
          const int r = g & 3, c = (2 * t) & 3;
          w[j][0] = r > c ? sil[r][c] : siu[r][c];
          w[j][1] = r > c + 1 ? sil[r][c + 1] : siu[r][c + 1];
        }
    }
  }
  __syncthreads();
  for (int e = threadIdx.x; e < NP_NB * NP_NB; e += NPD_T) {
    const int r = e % NP_NB, c = e / NP_NB;
    if (r >= jb || c >= jb || c < (r & ~3)) continue;
    const T o = (T)s_rp[r][c];
    Ab[(size_t)r + (size_t)c * lda] = o;
    if (r > c) lm = fmaxf(lm, fabsf((float)o));
    if (r == c && o == (T)0) lm = INFINITY;  // a zero pivot
  }
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int e = 0; e < 2; ++e) {
      const int r = 8 * i + g, c = 8 * j + 2 * t + e;
      if (r < jb && c < jb) {
        Linv[r + (size_t)c * NP_NB] = r > c ? (T)w[j][e] : (r == c ? (T)1 : (T)0);
        Uinv[r + (size_t)c * NP_NB] = r <= c ? (T)w[j][e] : (T)0;
      }
    }
  for (int o = 16; o > 0; o >>= 1) lm = fmaxf(lm, __shfl_xor_sync(0xffffffffu, lm, o));
  if (lane == 0) np_note_lmax(lmax_bits, lm);
}

// 64 x 64 x 64 products of the panel kernels: acc = or -= L X with both operands
// in shared memory by columns, L[p][r] (ld 64) and X[c][p] (ld 65); thread
// (ty, tx) owns rows 4 ty .. and columns tx, tx + 16, ..: a warp's reads of L are
// vectors at two places, those of X 16 columns of one row, without conflicts
// (columns 4 tx ..: four-way).
#define NP_XLD (NP_NB + 1)
template <bool MINUS, typename T>
__device__ __forceinline__ void np_tile(T (&acc)[4][4], const T *L, const T *X, int ty, int tx) {
#pragma unroll 4
  for (int p = 0; p < NP_NB; ++p) {
    T l[4], x[4];
    np_ld4(L + p * NP_NB + 4 * ty, l[0], l[1], l[2], l[3]);
#pragma unroll
    for (int v = 0; v < 4; ++v) x[v] = X[(tx + 16 * v) * NP_XLD + p];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v) acc[u][v] = fma(MINUS ? -l[u] : l[u], x[v], acc[u][v]);
  }
}
// a tile (nr x nc of it, zeros beyond) to a thread's registers, all loads in
// flight together, and from there to shared memory with rows of ld words
template <typename T>
__device__ __forceinline__ void np_fetch(T (&v)[16], const T *G, int ld, int nr, int nc) {
  const int r = threadIdx.x % NP_NB, c0 = threadIdx.x / NP_NB;
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    const int c = c0 + 4 * q;
    v[q] = (r < nr && c < nc) ? G[r + (size_t)c * ld] : (T)0;
  }
}
template <typename T>
__device__ __forceinline__ void np_put(T *S, const T (&v)[16], int ld) {
  const int r = threadIdx.x % NP_NB, c0 = threadIdx.x / NP_NB;
#pragma unroll
  for (int q = 0; q < 16; ++q) S[(c0 + 4 * q) * ld + r] = v[q];
}
// the result through shared memory (X[c][p]'s place) back to A, coalesced
template <typename T>
__device__ __forceinline__ void np_keep(T *X, const T (&acc)[4][4], int ty, int tx) {
#pragma unroll
  for (int v = 0; v < 4; ++v)
#pragma unroll
    for (int u = 0; u < 4; ++u) X[(tx + 16 * v) * NP_XLD + 4 * ty + u] = acc[u][v];
}
template <typename T>
__device__ __forceinline__ void np_write(T *G, int ld, const T *X, int nr, int nc) {
  const int r = threadIdx.x % NP_NB, c0 = threadIdx.x / NP_NB;
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    const int c = c0 + 4 * q;
    if (r < nr && c < nc) G[r + (size_t)c * ld] = X[c * NP_XLD + r];
  }
}
#define NP_TILE(T) ((NP_NB * NP_NB + NP_NB * NP_XLD) * (int)sizeof(T))

// 64 x 64 tiles of the panel: blocks [0, nrb) take 64 rows of A21 (rows
// below the block, to n) and write A21 Uinv over them; blocks [nrb, nrb + ncb)
// take 64 columns of A12 (rows of the block, columns [cbeg, cend)) and write
// Linv A12.
template <typename T>
__global__ void __launch_bounds__(NP_T) k_np_panel(T *A, int lda, int n, int k, int jb,
                                                   const T *Linv, const T *Uinv, int nrb,
                                                   int cbeg, int cend, unsigned *lmax_bits) {
  extern __shared__ __align__(16) unsigned char np_sm[];
  T *L = (T *)np_sm, *X = L + NP_NB * NP_NB;
  const bool rows = (int)blockIdx.x < nrb;
  const int b = rows ? blockIdx.x : blockIdx.x - nrb;
  const int r0 = rows ? k + jb + NP_NB * b : k;      // first row of the tile in A
  const int c0 = rows ? k : cbeg + NP_NB * b;        // first column of the tile in A
  const int nr = rows ? min(NP_NB, n - r0) : jb;
  const int nc = rows ? jb : min(NP_NB, cend - c0);
  T *At = A + (size_t)r0 + (size_t)c0 * lda;
  {
    T av[16], wv[16];
    np_fetch(av, At, lda, nr, nc);
    np_fetch(wv, rows ? Uinv : Linv, NP_NB, jb, jb);
    np_put(L, rows ? av : wv, NP_NB);
    np_put(X, rows ? wv : av, NP_XLD);
  }
  __syncthreads();
  const int ty = threadIdx.x / 16, tx = threadIdx.x % 16;
  T acc[4][4] = {};
  np_tile<false>(acc, L, X, ty, tx);
  __syncthreads();
  np_keep(X, acc, ty, tx);
  __syncthreads();
  np_write(At, lda, X, nr, nc);
  if (rows) {
    float lm = 0.f;  // (rows and columns beyond the tile are zero)
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v) lm = fmaxf(lm, (float)fabs((double)acc[u][v]));
    for (int o = 16; o > 0; o >>= 1) lm = fmaxf(lm, __shfl_xor_sync(0xffffffffu, lm, o));
    if ((threadIdx.x & 31) == 0) np_note_lmax(lmax_bits, lm);
  }
}

// The outer panel's own update after block k: A(r, c) -= L21 U12 for the 64 x 64
// tile blockIdx of the rows below the block and the panel's columns [c0, cend).
template <typename T>
__global__ void __launch_bounds__(NP_T) k_np_inner(T *A, int lda, int n, int k, int cend) {
  extern __shared__ __align__(16) unsigned char np_sm[];
  T *L = (T *)np_sm, *X = L + NP_NB * NP_NB;
  const int r0 = k + NP_NB + NP_NB * blockIdx.x, c0 = k + NP_NB + NP_NB * blockIdx.y;
  const int nr = min(NP_NB, n - r0), nc = min(NP_NB, cend - c0);
  T *At = A + (size_t)r0 + (size_t)c0 * lda;
  const int ty = threadIdx.x / 16, tx = threadIdx.x % 16;
  T acc[4][4];
  {
    T av[16], wv[16];
    np_fetch(av, A + (size_t)r0 + (size_t)k * lda, lda, nr, NP_NB);
    np_fetch(wv, A + (size_t)k + (size_t)c0 * lda, lda, NP_NB, nc);
#pragma unroll
    for (int v = 0; v < 4; ++v)
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const int r = 4 * ty + u, c = tx + 16 * v;
        acc[u][v] = (r < nr && c < nc) ? At[r + (size_t)c * lda] : (T)0;
      }
    np_put(L, av, NP_NB);
    np_put(X, wv, NP_XLD);
  }
  __syncthreads();
  np_tile<true>(acc, L, X, ty, tx);
  __syncthreads();
  np_keep(X, acc, ty, tx);
  __syncthreads();
  np_write(At, lda, X, nr, nc);
}

// U12 of an outer panel (columns K .. Ke, whole blocks) for NC columns of the
// trailing matrix per CTA: forward substitution over the panel's blocks,
//   X_b = Linv_b (A_b - sum_{j < b} L_bj X_j),
// products by the FP64 tensor instruction (a warp: 8 rows, all NC columns), the
// X_j staying in shared memory, the next operand and the next block's values
// fetched under a product.  It stands between a panel and everything after it,
// so NC is small: 16, or 32 from two waves of SMs on.  (A launch per block and
// per update between them: 10 and 8 us each, seven in all; 64 columns and 4 x 4
// per thread: 56 us in FP64, 40 us in FP32.  17 us for 2,700 columns, 40 for
// 12,000; 64 columns there: 74, 16: 44.)
#define NPC_LD (NP_NB + 4)  // words: the reads of a half warp in different banks
template <typename T, int NC>
__global__ void __launch_bounds__(NP_T) k_np_cols(T *A, int lda, int n, int K, int Ke,
                                                  const T *inv0) {
  extern __shared__ __align__(16) unsigned char np_sm[];
  double *L = (double *)np_sm, *X = L + NP_NB * NPC_LD;  // X: a tile per block, by columns
  const int i = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int c0 = Ke + NC * blockIdx.x, nb = (Ke - K) / NP_NB, r = 8 * i + g;
  const size_t tri = (size_t)NP_NB * NP_NB;
  T op[16], nx[NC / 8][2];
  auto block = [&](int b) {
#pragma unroll
    for (int j = 0; j < NC / 8; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = c0 + 8 * j + 2 * t + e;
        nx[j][e] = c < n ? A[(size_t)(K + NP_NB * b + r) + (size_t)c * lda] : (T)0;
      }
  };
  np_fetch(op, inv0 + 2 * tri * (size_t)(K / NP_NB), NP_NB, NP_NB, NP_NB);
  block(0);
  for (int b = 0; b < nb; ++b) {
    double *Xb = X + (size_t)b * NC * NPC_LD;
    double acc[NC / 8][2];
#pragma unroll
    for (int j = 0; j < NC / 8; ++j) acc[j][0] = (double)nx[j][0], acc[j][1] = (double)nx[j][1];
    if (b + 1 < nb) block(b + 1);
    for (int jb = 0; jb <= b; ++jb) {
      // op: L_b,jb, at the end Linv_b; the next one: L_b,jb+1, Linv_b or L_b+1,0
      __syncthreads();
      {
        const int lr = threadIdx.x % NP_NB, lc = threadIdx.x / NP_NB;
#pragma unroll
        for (int q = 0; q < 16; ++q) L[(lc + 4 * q) * NPC_LD + lr] = (double)op[q];
      }
      if (jb == b) {
#pragma unroll
        for (int j = 0; j < NC / 8; ++j)
#pragma unroll
          for (int e = 0; e < 2; ++e) Xb[(8 * j + 2 * t + e) * NPC_LD + r] = acc[j][e];
      }
      __syncthreads();
      const int jn = jb < b ? jb + 1 : 0, bn = jb < b ? b : b + 1;
      if (bn < nb) {
        if (jn < bn)
          np_fetch(op, A + (size_t)(K + NP_NB * bn) + (size_t)(K + NP_NB * jn) * lda, lda, NP_NB,
                   NP_NB);
        else
          np_fetch(op, inv0 + 2 * tri * (size_t)(K / NP_NB + bn), NP_NB, NP_NB, NP_NB);
      }
      const double sign = jb < b ? -1.0 : 1.0, *Xj = X + (size_t)jb * NC * NPC_LD;
      if (jb == b) {
#pragma unroll
        for (int j = 0; j < NC / 8; ++j) acc[j][0] = acc[j][1] = 0.0;
      }
#pragma unroll 4
      for (int p = 0; p < NP_NB; p += 4) {
        const double a = sign * L[(p + t) * NPC_LD + r];
#pragma unroll
        for (int j = 0; j < NC / 8; ++j)
          np_dmma(acc[j][0], acc[j][1], a, Xj[(8 * j + g) * NPC_LD + p + t]);
      }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < NC / 8; ++j)
#pragma unroll
      for (int e = 0; e < 2; ++e) {
        const int c = 8 * j + 2 * t + e;
        Xb[c * NPC_LD + r] = acc[j][e];
        if (c0 + c < n)
          A[(size_t)(K + NP_NB * b + r) + (size_t)(c0 + c) * lda] = (T)acc[j][e];
      }
  }
}
template <typename T, int NC>
static void np_cols(cudaStream_t st, T *A, int lda, int n, int K, int Ke, const T *inv0) {
  const int smem = (NP_NB + NP_NBO / NP_NB * NC) * NPC_LD * 8;
  static std::atomic<bool> attr{false};  // per instance
  if (!attr) {
    cudaFuncSetAttribute(k_np_cols<T, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    attr = true;
  }
  k_np_cols<T, NC><<<(n - Ke + NC - 1) / NC, NP_T, smem, st>>>(A, lda, n, K, Ke, inv0);
}

__global__ void k_np_ipiv(int n, int *ipiv) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) ipiv[i] = i + 1;
}

static cublasStatus_t np_gemm_minus(cublasHandle_t h, int m, int n, int k, const double *A,
                                    int lda, const double *B, int ldb, double *C, int ldc) {
  const double one = 1.0, mone = -1.0;
  return cublasDgemm(h, CUBLAS_OP_N, CUBLAS_OP_N, m, n, k, &mone, A, lda, B, ldb, &one, C, ldc);
}

int gemm_tf32_minus(cudaStream_t st, int m, int n, int k, const float *A, int lda,
                    const float *B, int ldb, float *C, int ldc);

__global__ void k_np_iota(int n, int *v) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) v[i] = i;
}

static cublasStatus_t np_gemm_minus(cublasHandle_t h, int m, int n, int k, const float *A,
                                    int lda, const float *B, int ldb, float *C, int ldc) {
  const float one = 1.f, mone = -1.f;
  return cublasSgemm(h, CUBLAS_OP_N, CUBLAS_OP_N, m, n, k, &mone, A, lda, B, ldb, &one, C, ldc);
}

template <typename T>
int lu_getrf_nopiv(cublasHandle_t cb, cudaStream_t st, LuWork &w, int n, T *A, int lda,
                   int *ipiv, int gemm_update, int *perm, float *lmax) {
  *lmax = 0.f;
  w.inv_n = 0;
  w.inv_ok = false;
  if (n <= 0) return DUST_OK;
  // inverse triangles of every diagonal block are kept (Linv then Uinv per
  // block) for lu_inv_build
  const size_t tri = (size_t)NP_NB * NP_NB;
  const int nblk_ = (n + NP_NB - 1) / NP_NB;
  DUST_TRY(devbuf_grow(w.np, 256 + 2 * tri * sizeof(T) * (size_t)nblk_));
  unsigned *bits = (unsigned *)w.np.p;
  T *inv0 = (T *)((char *)w.np.p + 256);
  DUST_CUDA(cudaMemsetAsync(bits, 0, sizeof(unsigned), st));
  const int smp = NP_TILE(T);
  static std::atomic<bool> attr{false};  // per element type
  if (!attr) {
    DUST_CUDA(cudaFuncSetAttribute(k_np_panel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smp));
    DUST_CUDA(cudaFuncSetAttribute(k_np_inner<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smp));
    attr = true;
  }
  if (n > 2 * NP_NBO) DUST_TRY(w.side.make());
  CUBLAS_CHECK(cublasSetStream(cb, st));
  // C -= A B (m x nn, inner kk) on the tensor cores (FP32) or DGEMM
  auto update = [&](int m, int nn, int kk, const T *Am, const T *Bm, T *Cm) -> int {
    if (m <= 0 || nn <= 0 || kk <= 0) return DUST_OK;
    if (sizeof(T) == 4 && gemm_update == 1)
      return gemm_tf32_minus(st, m, nn, kk, (const float *)Am, lda, (const float *)Bm, lda,
                             (float *)Cm, lda);
    CUBLAS_CHECK(np_gemm_minus(cb, m, nn, kk, Am, lda, Bm, lda, Cm, lda));
    return DUST_OK;
  };
  auto at = [&](int r, int c) { return A + r + (size_t)c * lda; };
  // two levels: an outer panel of NP_NBO columns is factored in NP_NB steps that
  // update only the panel's own columns
  auto panel = [&](int K, cudaStream_t s) {
    const int Ke = std::min(K + NP_NBO, n);
    for (int k = K; k < Ke; k += NP_NB) {
      const int jb = std::min(NP_NB, n - k), m2 = n - k - jb, wc = Ke - k - jb;
      T *Linv = inv0 + 2 * tri * (size_t)(k / NP_NB), *Uinv = Linv + tri;
      k_np_diag<T><<<1, NPD_T, 0, s>>>(A, lda, k, jb, Linv, Uinv, bits);
      const int nrb = (m2 + NP_NB - 1) / NP_NB, ncb = (wc + NP_NB - 1) / NP_NB;
      if (nrb + ncb > 0)
        k_np_panel<T><<<nrb + ncb, NP_T, smp, s>>>(A, lda, n, k, jb, Linv, Uinv, nrb, k + jb, Ke,
                                                    bits);
      if (nrb > 0 && ncb > 0) k_np_inner<T><<<dim3(nrb, ncb), NP_T, smp, s>>>(A, lda, n, k, Ke);
    }
  };
  // Then the panel's U12 right of it and the trailing update, the next panel's
  // columns first: that panel, a chain of small kernels, is factored on a second
  // stream under the update of the rest.
  panel(0, st);
  for (int K = 0; K + NP_NBO < n; K += NP_NBO) {
    const int Ke = K + NP_NBO, Kn = std::min(Ke + NP_NBO, n);
    if (n - Ke >= 148 * 64)
      np_cols<T, 32>(st, A, lda, n, K, Ke, inv0);
    else
      np_cols<T, 16>(st, A, lda, n, K, Ke, inv0);
    DUST_TRY(update(n - Ke, Kn - Ke, NP_NBO, at(Ke, K), at(K, Ke), at(Ke, Ke)));
    if (Kn == n) {
      panel(Ke, st);
      break;
    }
    DUST_CUDA(cudaEventRecord(w.side.go, st));
    DUST_CUDA(cudaStreamWaitEvent(w.side.st, w.side.go, 0));
    panel(Ke, w.side.st);
    DUST_CUDA(cudaEventRecord(w.side.done, w.side.st));
    const int s = update(n - Ke, n - Kn, NP_NBO, at(Ke, K), at(K, Kn), at(Ke, Kn));
    DUST_CUDA(cudaStreamWaitEvent(st, w.side.done, 0));  // joined whatever s is
    DUST_TRY(s);
  }
  if (ipiv) k_np_ipiv<<<(n + 255) / 256, 256, 0, st>>>(n, ipiv);
  if (perm) k_np_iota<<<(n + 255) / 256, 256, 0, st>>>(n, perm);
  DUST_CUDA(cudaGetLastError());
  unsigned hb = 0;
  DUST_CUDA(cudaMemcpyAsync(&hb, bits, sizeof(unsigned), cudaMemcpyDeviceToHost, st));
  DUST_CUDA(cudaStreamSynchronize(st));
  unsigned tmp = hb;
  memcpy(lmax, &tmp, sizeof(float));
  return DUST_OK;
}

template int lu_getrf_nopiv<double>(cublasHandle_t, cudaStream_t, LuWork &, int, double *, int,
                                    int *, int, int *, float *);
template int lu_getrf_nopiv<float>(cublasHandle_t, cudaStream_t, LuWork &, int, float *, int,
                                   int *, int, int *, float *);
