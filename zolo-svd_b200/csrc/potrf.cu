// Leaf kernels of the recursive Cholesky / triangular solves (FP64).
// The recursion (linalg.cpp) turns all O(n^3) work into DMMA GEMMs; these
// kernels factor the nb x nb diagonal blocks (nb <= 64) in shared memory and
// also return each block's inverse, which the triangular solves use at their
// leaves (so no separate inversion pass is needed).
//
// A leaf is one CTA, bound by the chain of its 64 pivots, not by arithmetic.  The chain runs in
// one warp on 16 x 16 diagonal blocks held in registers, which returns the block's factor and
// inverse together (about 220 clocks a pivot: a shuffle, a reciprocal, an exchange of the row, FMAs); the rest of the
// block column is then a product with that inverse and the trailing update and the merging of
// the inverses are products too, on the FP64 tensor path by all eight warps.  Measured:
// 53 -> 18 us for the 64 x 64 factor and inverse (one barrier per pivot and element-wise updates in
// shared memory before), 22 -> 5 us for the inverses of given factors.
#include "common.cuh"
#include "kernels.h"

namespace zolo {

namespace {

constexpr int LEAF = 64;
constexpr int LB = 16;        // diagonal block of the register factorization
constexpr int LDS = LEAF + 4; // = 4 mod 16: conflict-free fragment loads
constexpr int PT = 256;

// One 16 x 8 tile C (rows i0, columns j0 of s, ld LDS) = beta C + alpha A B with A 16 x K at a
// (a[i + k LDS]) and B K x 8: b[k + j LDS], or b[j + k LDS] when TB; by one warp, K a multiple of 8.
template <bool TB>
ZDEV void tile_mma(double (&c)[4], const double* a, const double* b, int K) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll 4
  for (int k = 0; k < K; k += 8) {
    double af[4], bf[2];
    af[0] = a[g + (k + t) * LDS];
    af[1] = a[g + 8 + (k + t) * LDS];
    af[2] = a[g + (k + t + 4) * LDS];
    af[3] = a[g + 8 + (k + t + 4) * LDS];
    bf[0] = TB ? b[g + (k + t) * LDS] : b[k + t + g * LDS];
    bf[1] = TB ? b[g + (k + t + 4) * LDS] : b[k + t + 4 + g * LDS];
    dmma_16x8x8(c, af, bf);
  }
}
ZDEV void tile_store(double* s, const double (&c)[4], double alpha) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  s[g + (2 * t) * LDS] = alpha * c[0];
  s[g + (2 * t + 1) * LDS] = alpha * c[1];
  s[g + 8 + (2 * t) * LDS] = alpha * c[2];
  s[g + 8 + (2 * t + 1) * LDS] = alpha * c[3];
}
ZDEV void tile_sub(double* s, const double (&c)[4]) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  s[g + (2 * t) * LDS] -= c[0];
  s[g + (2 * t + 1) * LDS] -= c[1];
  s[g + 8 + (2 * t) * LDS] -= c[2];
  s[g + 8 + (2 * t + 1) * LDS] -= c[3];
}

// Cholesky factor and its inverse of the 16 x 16 block at (k0, k0) by one warp: Gaussian elimination on
// the rows of [A | I], lane r the row r of A (both triangles), lane 16 + r the row r of I; L is the
// eliminated columns over sqrt(d_j), L^{-1} the transformed identity's rows over sqrt(d_r).  The pivot
// rows go round through shared memory (piv, 2 x 2 x 16) while the pivot's reciprocal is formed.
// Returns the first pivot (1-based) that is not positive, 0 if none.
ZDEV int factor_block(double* a, double* x, int k0, double* piv) {
  const int lane = threadIdx.x & 31, r = lane & 15, h = lane >> 4;
  double row[LB];
#pragma unroll
  for (int j = 0; j < LB; ++j)
    row[j] = h ? (j == r ? 1.0 : 0.0) : a[k0 + max(r, j) + (k0 + min(r, j)) * LDS];
  int bad = 0;
#pragma unroll
  for (int k = 0; k < LB; ++k) {
    const double d = __shfl_sync(0xffffffffu, row[k], k);
    const double ark = __shfl_sync(0xffffffffu, row[k], r);
    double2* pv = reinterpret_cast<double2*>(piv + (k & 1) * 2 * LB + h * LB);
    if (r == k) {
#pragma unroll
      for (int j = 0; j < LB; j += 2) pv[j / 2] = make_double2(row[j], row[j + 1]);
    }
    __syncwarp();
    const bool ok = d > 0.0;
    if (!ok && bad == 0) bad = k + 1;
    // 1/d as rsqrt(d)^2: the division's own chain is 150 clocks longer (400 against 220 a step)
    const double q = rsqrt(ok ? d : 1.0);
    const double m = (r > k && ok) ? -(ark * q) * q : 0.0;
    const double ma = h ? 0.0 : m, mx = h ? m : 0.0;  // A's columns past k, the identity's up to k
#pragma unroll
    for (int j = 0; j < LB; j += 2) {
      const double2 pk = pv[j / 2];
      row[j] = fma(j > k ? ma : mx, pk.x, row[j]);
      row[j + 1] = fma(j + 1 > k ? ma : mx, pk.y, row[j + 1]);
    }
  }
  double dr = 1.0;  // pivot of this lane's row
#pragma unroll
  for (int j = 0; j < LB; ++j) {
    const double d = __shfl_sync(0xffffffffu, row[j], j);
    if (j == r) dr = d;
  }
  const double sd = dr > 0.0 ? sqrt(dr) : 1.0, rs = 1.0 / sd;
#pragma unroll
  for (int j = 0; j < LB; ++j) {
    const double rj = __shfl_sync(0xffffffffu, rs, j);
    if (h) x[k0 + r + (k0 + j) * LDS] = j <= r ? row[j] * rs : 0.0;
    else a[k0 + r + (k0 + j) * LDS] = j < r ? row[j] * rj : (j == r ? sd : 0.0);
  }
  return bad;
}

// Inverse of the 16 x 16 lower-triangular block at (k0, k0) of a by one warp (lanes 0 .. 15: a row each).
ZDEV void invert_block(const double* a, double* x, int k0) {
  const int lane = threadIdx.x & 31, r = lane & 15;
  double row[LB], l[LB];
#pragma unroll
  for (int j = 0; j < LB; ++j) {
    l[j] = a[k0 + r + (k0 + j) * LDS];
    row[j] = j == r ? 1.0 : 0.0;
  }
  double dr = 1.0;
#pragma unroll
  for (int j = 0; j < LB; ++j)
    if (j == r) dr = l[j];
  const double rs = 1.0 / dr;
#pragma unroll
  for (int k = 0; k < LB; ++k) {
    if (r == k) {
#pragma unroll
      for (int j = 0; j <= k; ++j) row[j] *= rs;
    }
    const double m = r > k ? l[k] : 0.0;
#pragma unroll
    for (int j = 0; j <= k; ++j) row[j] = fma(-m, __shfl_sync(0xffffffffu, row[j], k), row[j]);
  }
  if (lane < 16) {
#pragma unroll
    for (int j = 0; j < LB; ++j) x[k0 + r + (k0 + j) * LDS] = j <= r ? row[j] : 0.0;
  }
}

// x = l^{-1} from the inverses of its 16 x 16 diagonal blocks: X21 = -X22 (L21 X11) for pairs of 16, then
// of 32.  The products L21 X11 go through l's upper triangle (not part of the factor).  All 8 warps.
ZDEV void merge_inverse(double* l, double* x) {
  const int warp = threadIdx.x >> 5;
#pragma unroll
  for (int half = LB; half < LEAF; half *= 2) {
    const int rt = half / 16, ct = half / 8, per = rt * ct;  // 16 x 8 tiles of one pair's X21
    const int pairs = LEAF / (2 * half);
    for (int u = warp; u < pairs * per; u += PT / 32) {
      const int o = (u / per) * 2 * half, ti = (u % per) / ct * 16, tj = (u % per) % ct * 8;
      double c[4] = {0.0, 0.0, 0.0, 0.0};
      tile_mma<false>(c, l + o + half + ti + o * LDS, x + o + (o + tj) * LDS, half);
      tile_store(l + o + ti + (o + half + tj) * LDS, c, 1.0);
    }
    __syncthreads();
    for (int u = warp; u < pairs * per; u += PT / 32) {
      const int o = (u / per) * 2 * half, ti = (u % per) / ct * 16, tj = (u % per) % ct * 8;
      double c[4] = {0.0, 0.0, 0.0, 0.0};
      tile_mma<false>(c, x + o + half + ti + (o + half) * LDS, l + o + (o + half + tj) * LDS, half);
      tile_store(x + o + half + ti + (o + tj) * LDS, c, -1.0);
    }
    __syncthreads();
  }
}

// The leaf in shared memory: lower triangle of the nb x nb block, the identity beyond nb.
ZDEV void load_leaf(int nb, const double* A, int64_t lda, double* a, double* x) {
  constexpr int NE = LEAF * LEAF / PT;
  double v[NE];  // every load in flight before the first store
#pragma unroll
  for (int q = 0; q < NE; ++q) {
    const int e = threadIdx.x + q * PT, i = e & (LEAF - 1), j = e >> 6;
    v[q] = (i < nb && j <= i) ? A[i + j * lda] : (i == j ? 1.0 : 0.0);
  }
#pragma unroll
  for (int q = 0; q < NE; ++q) {
    const int e = threadIdx.x + q * PT, i = e & (LEAF - 1), j = e >> 6;
    a[i + j * LDS] = v[q];
    x[i + j * LDS] = 0.0;
  }
  __syncthreads();
}

// Factor of the leaf in a (all warps; identity beyond nb) and the inverses of its 16 x 16 diagonal
// blocks in x, ones on x's diagonal past the eliminated blocks.
ZDEV void factor_leaf(int nb, double* a, double* x, double* piv, int* info, int info_offset) {
  const int warp = threadIdx.x >> 5;
  const int n16 = (nb + LB - 1) / LB * LB;  // identity blocks past nb need no elimination
  for (int k0 = 0; k0 < n16; k0 += LB) {
    if (warp == 0) {
      const int bad = factor_block(a, x, k0, piv);
      if (bad && threadIdx.x == 0 && info && k0 + bad <= nb)  // LAPACK INFO = first non-positive pivot
        atomicCAS(info, 0, info_offset + k0 + bad);
    }
    __syncthreads();
    const int rows = (n16 - k0 - LB) / 16;  // 16-row tiles below
    if (warp < rows) {
      // L21 = A21 L11^{-T}, a warp per 16 rows (it reads all of them before it writes)
      double* p = a + k0 + LB + 16 * warp + k0 * LDS;
      double c0[4] = {0.0, 0.0, 0.0, 0.0}, c1[4] = {0.0, 0.0, 0.0, 0.0};
      tile_mma<true>(c0, p, x + k0 + k0 * LDS, LB);
      tile_mma<true>(c1, p, x + k0 + 8 + k0 * LDS, LB);
      __syncwarp();
      tile_store(p, c0, 1.0);
      tile_store(p + 8 * LDS, c1, 1.0);
    }
    __syncthreads();
    // A22 -= L21 L21^T on the 16 x 8 tiles meeting the lower triangle
    for (int u = warp; u < rows * (rows + 1); u += PT / 32) {
      int ti = 0, r = u;
      while (r >= 2 * ti + 2) {
        r -= 2 * ti + 2;
        ++ti;
      }
      const double* pi = a + k0 + LB + 16 * ti + k0 * LDS;
      const double* pj = a + k0 + LB + 8 * r + k0 * LDS;
      double c[4] = {0.0, 0.0, 0.0, 0.0};
      tile_mma<true>(c, pi, pj, LB);
      tile_sub(a + k0 + LB + 16 * ti + (k0 + LB + 8 * r) * LDS, c);
    }
    __syncthreads();
  }
  for (int i = n16 + threadIdx.x; i < LEAF; i += PT) x[i + i * LDS] = 1.0;
  __syncthreads();
}

__global__ void __launch_bounds__(PT) potrf_leaf_kernel(int nb, double* A, int64_t lda, int64_t strideA, int* info,
                                                        int info_offset, double* Dinv, int64_t ldd, int64_t strideD) {
  extern __shared__ double sm[];
  double* a = sm;
  double* x = sm + LEAF * LDS;
  double* Ab = A + blockIdx.x * strideA;
  __shared__ __align__(16) double piv[4 * LB];
  dependency_wait();
  load_leaf(nb, Ab, lda, a, x);
  factor_leaf(nb, a, x, piv, info ? info + blockIdx.x : nullptr, info_offset);
  for (int e = threadIdx.x; e < LEAF * LEAF; e += PT) {
    const int i = e & (LEAF - 1), j = e >> 6;
    if (i < nb && j <= i) Ab[i + j * lda] = a[i + j * LDS];
  }
  release_dependents();
  if (!Dinv) return;
  __syncthreads();  // the factor is read: the merge uses its upper triangle
  merge_inverse(a, x);
  double* Db = Dinv + blockIdx.x * strideD;
  for (int e = threadIdx.x; e < LEAF * LEAF; e += PT) {
    const int i = e & (LEAF - 1), j = e >> 6;
    if (i < nb && j < nb) Db[i + j * ldd] = x[i + j * LDS];
  }
}

// Y = L^{-1} of the Cholesky factor of a block of 64 < nb <= 128 rows, one CTA: two leaves with
// their inverses, L21 = A21 X11^T, A22 - L21 L21^T, X21 = -X22 (L21 X11), all in shared memory.  As two
// leaf launches and four products of 64 x 64 tiles on a few SMs it was 57 us; the chain of 128 pivots
// and the products are 41 us here (QDWH n = 1024 9.23 -> 9.05 ms).  The factor is not written back.
__global__ void __launch_bounds__(PT) potrf_inv_pair_kernel(int nb, const double* A, int64_t lda, int64_t strideA,
                                                            int* info, int info_offset, double* Y, int64_t ldy,
                                                            int64_t strideY) {
  extern __shared__ double sm[];
  constexpr int BLK = LEAF * LDS;
  double *a11 = sm, *x11 = sm + BLK, *a21 = sm + 2 * BLK, *a22 = sm + 3 * BLK, *x22 = sm + 4 * BLK, *l21 = sm + 5 * BLK;
  __shared__ __align__(16) double piv[4 * LB];
  const double* Ab = A + blockIdx.x * strideA;
  int* inf = info ? info + blockIdx.x : nullptr;
  const int warp = threadIdx.x >> 5, nb2 = nb - LEAF;
  dependency_wait();
  {
    constexpr int NE = LEAF * LEAF / PT;
    double v[NE];
#pragma unroll
    for (int q = 0; q < NE; ++q) {
      const int e = threadIdx.x + q * PT, i = e & (LEAF - 1), j = e >> 6;
      v[q] = i < nb2 ? Ab[LEAF + i + j * lda] : 0.0;
    }
#pragma unroll
    for (int q = 0; q < NE; ++q) {
      const int e = threadIdx.x + q * PT;
      a21[(e & (LEAF - 1)) + (e >> 6) * LDS] = v[q];
    }
  }
  load_leaf(nb2, Ab + LEAF + LEAF * lda, lda, a22, x22);
  load_leaf(LEAF, Ab, lda, a11, x11);
  factor_leaf(LEAF, a11, x11, piv, inf, info_offset);
  merge_inverse(a11, x11);
  for (int u = warp; u < 32; u += PT / 32) {  // L21: column tile tj of X11^T needs k < 8 tj + 8
    const int ti = u & 3, tj = u >> 2;
    double c[4] = {0.0, 0.0, 0.0, 0.0};
    tile_mma<true>(c, a21 + 16 * ti, x11 + 8 * tj, 8 * tj + 8);
    tile_store(l21 + 16 * ti + 8 * tj * LDS, c, 1.0);
  }
  __syncthreads();
  for (int u = warp; u < 52; u += PT / 32) {
    double c[4] = {0.0, 0.0, 0.0, 0.0};
    if (u < 20) {  // A22 - L21 L21^T on the tiles meeting the lower triangle
      int ti = 0, r = u;
      while (r >= 2 * ti + 2) {
        r -= 2 * ti + 2;
        ++ti;
      }
      tile_mma<true>(c, l21 + 16 * ti, l21 + 8 * r, LEAF);
      tile_sub(a22 + 16 * ti + 8 * r * LDS, c);
    } else {  // L21 X11 over A21: X11's column tile starts at row 8 tj
      const int ti = (u - 20) & 3, k0 = ((u - 20) >> 2) * 8;
      tile_mma<false>(c, l21 + 16 * ti + k0 * LDS, x11 + k0 + k0 * LDS, LEAF - k0);
      tile_store(a21 + 16 * ti + k0 * LDS, c, 1.0);
    }
  }
  __syncthreads();
  factor_leaf(nb2, a22, x22, piv, inf, info_offset + LEAF);
  merge_inverse(a22, x22);
  for (int u = warp; u < 32; u += PT / 32) {
    const int ti = u & 3, tj = u >> 2;
    double c[4] = {0.0, 0.0, 0.0, 0.0};
    tile_mma<false>(c, x22 + 16 * ti, a21 + 8 * tj * LDS, 16 * ti + 16);
    tile_store(l21 + 16 * ti + 8 * tj * LDS, c, -1.0);
  }
  release_dependents();
  __syncthreads();
  double* Yb = Y + blockIdx.x * strideY;
  for (int e = threadIdx.x; e < LEAF * LEAF; e += PT) {
    const int i = e & (LEAF - 1), j = e >> 6, o = i + j * LDS;
    Yb[i + j * ldy] = x11[o];
    if (i < nb2) {
      Yb[LEAF + i + j * ldy] = l21[o];
      if (j < nb2) Yb[LEAF + i + (LEAF + j) * ldy] = x22[o];
    }
  }
}

// Inverses of the diagonal blocks of a lower-triangular n x n matrix:
// block kb (rows/cols kb*64 ..) of batch entry b goes to Dinv + b*strideD + kb*blk (ld ldd).
__global__ void __launch_bounds__(PT) trtri_blocks_kernel(int n, const double* L, int64_t ldl, int64_t strideL,
                                                          double* Dinv, int64_t ldd, int64_t blk,
                                                          int64_t strideD) {
  extern __shared__ double sm[];
  double* l = sm;
  double* x = sm + LEAF * LDS;
  const int kb = blockIdx.x, b = blockIdx.y;
  const int o = kb * LEAF;
  const int nb = min(LEAF, n - o);
  dependency_wait();
  load_leaf(nb, L + b * strideL + o + static_cast<int64_t>(o) * ldl, ldl, l, x);
  const int warp = threadIdx.x >> 5;
  if (warp < LEAF / LB) invert_block(l, x, warp * LB);
  __syncthreads();
  merge_inverse(l, x);
  double* Db = Dinv + b * strideD + kb * blk;
  for (int e = threadIdx.x; e < LEAF * LEAF; e += PT) {
    const int i = e & (LEAF - 1), j = e >> 6;
    if (i < nb && j < nb) Db[i + j * ldd] = x[i + j * LDS];
  }
}

constexpr int SMEM_BYTES = 2 * LEAF * LDS * 8;
constexpr int SMEM_PAIR = 6 * LEAF * LDS * 8;

}  // namespace

cudaError_t potrf_leaf(int nb, double* A, int64_t lda, int64_t strideA, int batch, int* info, int info_offset,
                       double* Dinv, int64_t ldd, int64_t strideD, cudaStream_t st) {
  if (nb <= 0 || batch <= 0) return cudaSuccess;
  if (nb > LEAF) return cudaErrorInvalidValue;
  static std::atomic<int> attr_set[kMaxDevices];
  const cudaError_t attr = once_per_device(attr_set, [] {
    return cudaFuncSetAttribute(potrf_leaf_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
  });
  if (attr != cudaSuccess) return attr;
  return launch_dependent(potrf_leaf_kernel, dim3(batch), dim3(PT), SMEM_BYTES, st, dim3(1), nb, A, lda, strideA, info,
                          info_offset, Dinv, ldd, strideD);
}

cudaError_t potrf_inv_pair(int nb, const double* A, int64_t lda, int64_t strideA, int batch, int* info, int info_offset,
                           double* Y, int64_t ldy, int64_t strideY, cudaStream_t st) {
  if (batch <= 0) return cudaSuccess;
  if (nb <= LEAF || nb > 2 * LEAF) return cudaErrorInvalidValue;
  static std::atomic<int> attr_set[kMaxDevices];
  const cudaError_t attr = once_per_device(attr_set, [] {
    return cudaFuncSetAttribute(potrf_inv_pair_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_PAIR);
  });
  if (attr != cudaSuccess) return attr;
  return launch_dependent(potrf_inv_pair_kernel, dim3(batch), dim3(PT), SMEM_PAIR, st, dim3(1), nb, A, lda, strideA, info,
                          info_offset, Y, ldy, strideY);
}

cudaError_t trtri_blocks(int n, const double* L, int64_t ldl, int64_t strideL, double* Dinv, int64_t ldd, int64_t blk,
                         int64_t strideD, int batch, cudaStream_t st) {
  if (n <= 0 || batch <= 0) return cudaSuccess;
  static std::atomic<int> attr_set[kMaxDevices];
  const cudaError_t attr = once_per_device(attr_set, [] {
    return cudaFuncSetAttribute(trtri_blocks_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
  });
  if (attr != cudaSuccess) return attr;
  const int nblk = (n + LEAF - 1) / LEAF;
  return launch_dependent(trtri_blocks_kernel, dim3(nblk, batch), dim3(PT), SMEM_BYTES, st, dim3(1), n, L, ldl, strideL,
                          Dinv, ldd, blk, strideD);
}

}  // namespace zolo
