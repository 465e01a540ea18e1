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
//                 (column tiles, inside the outer panel), 64 x 64
//                 register-tiled products, max |l| of L21;
//     update      of the outer panel's own columns;
//   then the outer panel's U12 right of it (forward substitution over its
//   blocks with Linv) and the trailing update A22 -= L21 U12 of inner
//   dimension NP_NBO (tcgen05 TF32 GEMM for FP32, DGEMM for FP64), which
//   streams the trailing matrix a quarter as often as NP_NB-wide steps.
//
// The largest |l| is kept as float bits (monotone for non-negative values)
// with atomicMax.  The caller accepts the factors when it is below
// 1 - margin (a margin well above the rounding of the computed multipliers,
// so partial pivoting on the same values would also have kept every
// diagonal); otherwise, and on a zero diagonal, it restores A and runs the
// pivoted factorisation.  ipiv is the identity.
#include <algorithm>
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
#define NP_LD (NP_NB + 1)

__device__ __forceinline__ void np_note_lmax(unsigned *bits, float v) {
  atomicMax(bits, __float_as_uint(v));
}

// reciprocal pivots: FP64 from the refined approximation (elements.cuh), whose
// chain of dependent operations is a third of a division's
__device__ __forceinline__ double np_rcp(double x) {
  return near_range(fabs(x)) ? rcp_r(x) : 1.0 / x;
}
__device__ __forceinline__ float np_rcp(float x) { return 1.0f / x; }

// Diagonal block: LU and both inverse triangles in one block elimination.
// Thread (ty, tx) holds the 4 x 4 piece of rows 4 ty .. and columns 4 tx .. of
// W in registers, W = A at first.  A step takes four pivots Q = 4 q .. 4 q + 3:
// rows R = W(Q,:) and columns C = W(:,Q) come through shared memory (two
// buffers, so one barrier a step), every thread factors the 4 x 4 pivot block
// W(Q,Q) = L_d U_d and inverts its triangles itself, and with R' = L_d^-1 R and
// f = C U_d^-1
//   rows below Q:  f is L; W(r,c) -= f R'_c for every c outside Q (right of Q
//                  the elimination, left of it the row operations of Linv),
//                  W(r,Q) = -f L_d^-1;
//   rows above Q:  W(r,Q) = f, Uinv's columns; W(r,c) -= f R'_c right of Q;
//   rows Q:        R' is U right of Q and Linv's rows left of it;
//                  W(Q,c) = -U_d^-1 R'_c right of Q, W(Q,Q) the two inverses.
// L and U leave for global memory as the steps produce them; at the end W
// holds Linv below the diagonal and Uinv on and above it.  Bound by a step's
// chain (barrier, shared memory, reciprocals, products): four pivots a step
// (one: 57 us in FP64), the pivot block factored by every thread (by its owner
// ahead of the step: 41 us), a warp on two column stripes so that one warp
// walks the columns-Q branch (on two row stripes: 39 us).  It replaces a
// column per thread, unrolled, and two dependent substitutions, whose code did
// not stay in the instruction caches: FP32 47 -> 20 us, FP64 54 -> 37 us per
// block (one CTA).
#define NPD_T 256
template <typename T>
__global__ void __launch_bounds__(NPD_T) k_np_diag(T *A, int lda, int k, int jb, T *Linv,
                                                   T *Uinv, unsigned *lmax_bits) {
  __shared__ __align__(16) T s_row[2][4][NP_NB], s_col[2][4][NP_NB];
  const int tid = threadIdx.x, tx = tid / 16, ty = tid % 16;
  T *Ab = A + (size_t)k + (size_t)k * lda;
  T w[4][4];
#pragma unroll
  for (int v = 0; v < 4; ++v)
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int r = 4 * ty + u, c = 4 * tx + v;
      w[u][v] = (r < jb && c < jb) ? Ab[(size_t)r + (size_t)c * lda] : (r == c ? (T)1 : (T)0);
    }
  float lm = 0.f;
  // (pivots beyond jb meet the identity and change nothing)
#pragma unroll 1
  for (int q = 0; 4 * q < jb; ++q) {
    const int b = q & 1;
    if (ty == q) {
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) s_row[b][u][4 * tx + v] = w[u][v];
    }
    if (tx == q) {
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) s_col[b][v][4 * ty + u] = w[u][v];
    }
    __syncthreads();
    T D[4][4], R[4][4], f[4][4], iu[4][4], il[4][4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        D[u][v] = s_row[b][u][4 * q + v];
        R[u][v] = s_row[b][u][4 * tx + v];
        f[u][v] = s_col[b][v][4 * ty + u];
      }
    // D = L_d U_d in place; iu = U_d^-1, il = L_d^-1 (strictly lower part)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      iu[j][j] = np_rcp(D[j][j]);
#pragma unroll
      for (int r = j + 1; r < 4; ++r) {
        D[r][j] *= iu[j][j];
#pragma unroll
        for (int c = j + 1; c < 4; ++c) D[r][c] = fma(-D[r][j], D[j][c], D[r][c]);
      }
    }
#pragma unroll
    for (int c = 1; c < 4; ++c)
#pragma unroll
      for (int r = c - 1; r >= 0; --r) {
        T x = D[r][c] * iu[c][c];
#pragma unroll
        for (int p = r + 1; p < c; ++p) x = fma(D[r][p], iu[p][c], x);
        iu[r][c] = -x * iu[r][r];
      }
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
      for (int r = c + 1; r < 4; ++r) {
        T x = D[r][c];
#pragma unroll
        for (int p = c + 1; p < r; ++p) x = fma(D[r][p], il[p][c], x);
        il[r][c] = -x;
      }
    // R' = L_d^-1 R and f = C U_d^-1
#pragma unroll
    for (int v = 0; v < 4; ++v)
#pragma unroll
      for (int r = 1; r < 4; ++r)
#pragma unroll
        for (int p = 0; p < r; ++p) R[r][v] = fma(-D[r][p], R[p][v], R[r][v]);
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int c = 3; c >= 0; --c) {
        T x = f[u][c] * iu[c][c];
#pragma unroll
        for (int p = 0; p < c; ++p) x = fma(f[u][p], iu[p][c], x);
        f[u][c] = ty == q ? (u <= c ? iu[u][c] : (T)0) : x;
      }
    const bool right = tx > q, below = ty > q;
    if (tx != q) {
      if (ty == q) {
        // U right of the pivots, Linv's rows left of them
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int v = 0; v < 4; ++v) {
            if (right && 4 * tx + v < jb)
              Ab[(size_t)(4 * q + u) + (size_t)(4 * tx + v) * lda] = R[u][v];
            w[u][v] = right ? (T)0 : R[u][v];
          }
      }
      if (below || right) {
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
          for (int u = 0; u < 4; ++u)
#pragma unroll
            for (int v = 0; v < 4; ++v) w[u][v] = fma(-f[u][p], R[p][v], w[u][v]);
      }
    } else {
#pragma unroll
      for (int u = 0; u < 4; ++u)
#pragma unroll
        for (int v = 0; v < 4; ++v) {
          const int r = 4 * ty + u, c = 4 * q + v;
          T x = f[u][v];
          if (below) {
#pragma unroll
            for (int p = v + 1; p < 4; ++p) x = fma(f[u][p], il[p][v], x);
            x = -x;
          }
          if (ty == q && u > v) x = il[u][v];
          w[u][v] = x;
          if (r < jb && c < jb && (below || ty == q)) {
            const T o = below ? f[u][v] : D[u][v];
            Ab[(size_t)r + (size_t)c * lda] = o;
            if (r > c) lm = fmaxf(lm, fabsf((float)o));
            if (r == c && o == (T)0) lm = INFINITY;  // a zero pivot
          }
        }
    }
  }
  for (int o = 16; o > 0; o >>= 1) lm = fmaxf(lm, __shfl_xor_sync(0xffffffffu, lm, o));
  if ((tid & 31) == 0) np_note_lmax(lmax_bits, lm);
#pragma unroll
  for (int v = 0; v < 4; ++v)
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int r = 4 * ty + u, c = 4 * tx + v;
      if (r < jb && c < jb) {
        Linv[r + (size_t)c * NP_NB] = r > c ? w[u][v] : (r == c ? (T)1 : (T)0);
        Uinv[r + (size_t)c * NP_NB] = r <= c ? w[u][v] : (T)0;
      }
    }
}

// 64 x 64 tiles of the panel: blocks [0, nrb) take 64 rows of A21 (rows
// below the block, to n) and write A21 Uinv over them; blocks [nrb, nrb + ncb)
// take 64 columns of A12 (rows of the block, columns [cbeg, cend)) and write
// Linv A12.  Each thread computes a 4 x 4 piece of the tile from the two
// shared operands (the tile and the inverse triangle).
template <typename T>
__global__ void __launch_bounds__(NP_T) k_np_panel(T *A, int lda, int n, int k, int jb,
                                                   const T *Linv, const T *Uinv, int nrb,
                                                   int cbeg, int cend, unsigned *lmax_bits) {
  extern __shared__ __align__(16) unsigned char np_sm[];
  T *x = (T *)np_sm;            // 64 x 64 operand tile, [row][col], ld NP_LD
  T *w = x + NP_NB * NP_LD;     // 64 x 64 inverse, [row][col], ld NP_LD
  const int tid = threadIdx.x;
  const bool rows = (int)blockIdx.x < nrb;
  const int b = rows ? blockIdx.x : blockIdx.x - nrb;
  const int r0 = rows ? k + jb + NP_NB * b : k;      // first row of the tile in A
  const int c0 = rows ? k : cbeg + NP_NB * b;        // first column of the tile in A
  const int nr = rows ? min(NP_NB, n - r0) : jb;
  const int nc = rows ? jb : min(NP_NB, cend - c0);
  const T *W = rows ? Uinv : Linv;
  {
    // all of a thread's loads in flight together
    constexpr int M = NP_NB * NP_NB / NP_T;
    const int r = tid % NP_NB, cq = tid / NP_NB;
    T xv[M], wv[M];
#pragma unroll
    for (int q = 0; q < M; ++q) {
      const int c = cq + q * (NP_T / NP_NB);
      xv[q] = (r < nr && c < nc) ? A[(size_t)(r0 + r) + (size_t)(c0 + c) * lda] : (T)0;
      wv[q] = (r < jb && c < jb) ? W[r + (size_t)c * NP_NB] : (T)0;
    }
#pragma unroll
    for (int q = 0; q < M; ++q) {
      const int c = cq + q * (NP_T / NP_NB);
      x[r * NP_LD + c] = xv[q];
      w[r * NP_LD + c] = wv[q];
    }
  }
  __syncthreads();
  // out = x w (rows) or w x (columns); thread (ty, tx) owns rows 4 ty .. and
  // columns 4 tx ..
  const int ty = tid / 16, tx = tid % 16;
  T acc[4][4];
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) acc[u][v] = (T)0;
  const T *L = rows ? x : w, *R = rows ? w : x;
#pragma unroll 4
  for (int p = 0; p < NP_NB; ++p) {
    T lv[4], rv[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) lv[u] = L[(4 * ty + u) * NP_LD + p];
#pragma unroll
    for (int v = 0; v < 4; ++v) rv[v] = R[p * NP_LD + 4 * tx + v];
#pragma unroll
    for (int u = 0; u < 4; ++u)
#pragma unroll
      for (int v = 0; v < 4; ++v) acc[u][v] = fma(lv[u], rv[v], acc[u][v]);
  }
  // through shared memory back to A, coalesced along the columns
  __syncthreads();
  float lm = 0.f;
#pragma unroll
  for (int u = 0; u < 4; ++u)
#pragma unroll
    for (int v = 0; v < 4; ++v) {
      const int r = 4 * ty + u, c = 4 * tx + v;
      x[r * NP_LD + c] = acc[u][v];
      if (rows && r < nr && c < nc) lm = fmaxf(lm, (float)fabs((double)acc[u][v]));
    }
  __syncthreads();
  for (int e = tid; e < NP_NB * NP_NB; e += NP_T) {
    const int r = e % NP_NB, c = e / NP_NB;
    if (r < nr && c < nc) A[(size_t)(r0 + r) + (size_t)(c0 + c) * lda] = x[r * NP_LD + c];
  }
  if (rows) {
    for (int o = 16; o > 0; o >>= 1) lm = fmaxf(lm, __shfl_xor_sync(0xffffffffu, lm, o));
    if ((tid & 31) == 0) np_note_lmax(lmax_bits, lm);
  }
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
  if (n <= 0) return DUST_OK;
  // inverse triangles of every diagonal block are kept (Linv then Uinv per
  // block) for lu_inv_build
  const size_t tri = (size_t)NP_NB * NP_NB;
  const int nblk_ = (n + NP_NB - 1) / NP_NB;
  DUST_TRY(devbuf_grow(w.np, 256 + 2 * tri * sizeof(T) * (size_t)nblk_));
  unsigned *bits = (unsigned *)w.np.p;
  T *inv0 = (T *)((char *)w.np.p + 256);
  DUST_CUDA(cudaMemsetAsync(bits, 0, sizeof(unsigned), st));
  const int smp = 2 * NP_NB * NP_LD * (int)sizeof(T);
  static bool attr = false;  // per element type
  if (!attr) {
    DUST_CUDA(cudaFuncSetAttribute(k_np_panel<T>, cudaFuncAttributeMaxDynamicSharedMemorySize, smp));
    attr = true;
  }
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
  // two levels: outer panels of NP_NBO columns factored in NP_NB steps that
  // update only the panel's own columns; then the panel's U12 (its unit lower
  // block's forward substitution, with the kept inverse triangles) and one
  // trailing update of inner dimension NP_NBO
  for (int K = 0; K < n; K += NP_NBO) {
    const int Ke = std::min(K + NP_NBO, n);
    for (int k = K; k < Ke; k += NP_NB) {
      const int jb = std::min(NP_NB, n - k), m2 = n - k - jb, wc = Ke - k - jb;
      T *Linv = inv0 + 2 * tri * (size_t)(k / NP_NB), *Uinv = Linv + tri;
      k_np_diag<T><<<1, NPD_T, 0, st>>>(A, lda, k, jb, Linv, Uinv, bits);
      const int nrb = (m2 + NP_NB - 1) / NP_NB, ncb = (wc + NP_NB - 1) / NP_NB;
      if (nrb + ncb > 0)
        k_np_panel<T><<<nrb + ncb, NP_T, smp, st>>>(A, lda, n, k, jb, Linv, Uinv, nrb, k + jb,
                                                     Ke, bits);
      DUST_TRY(update(m2, wc, jb, at(k + jb, k), at(k, k + jb), at(k + jb, k + jb)));
    }
    if (Ke < n) {
      const int ncb = (n - Ke + NP_NB - 1) / NP_NB;
      for (int k = K; k < Ke; k += NP_NB) {
        const T *Linv = inv0 + 2 * tri * (size_t)(k / NP_NB);
        k_np_panel<T><<<ncb, NP_T, smp, st>>>(A, lda, n, k, NP_NB, Linv, Linv, 0, Ke, n, bits);
        DUST_TRY(update(Ke - k - NP_NB, n - Ke, NP_NB, at(k + NP_NB, k), at(k, Ke),
                        at(k + NP_NB, Ke)));
      }
      DUST_TRY(update(n - Ke, n - Ke, Ke - K, at(Ke, K), at(K, Ke), at(Ke, Ke)));
    }
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
