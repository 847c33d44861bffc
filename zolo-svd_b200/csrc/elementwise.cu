// HBM-bound FP64 kernels: scaling/copies, the stacked [X; sqrt(c) I] form, the
// shifted Gram copy, norms, and the fused FormX2 / QDWH combine with the
// ||X_{k+1} - X_k||_F reduction.  Reductions are deterministic: per-block
// partials followed by one fixed-order block sum.
#include "common.cuh"
#include "kernels.h"

#include <algorithm>

namespace zolo {

namespace {

constexpr int TPB = 256;

inline int grid_for(int64_t work, int per_block = TPB) {
  int64_t b = (work + per_block - 1) / per_block;
  b = std::min<int64_t>(b, static_cast<int64_t>(num_sms()) * 8);
  return static_cast<int>(std::max<int64_t>(b, 1));
}

__global__ void scale_copy_kernel(int m, int n, double s, const double* src, int64_t lds,
                                  int64_t strideS, double* dst, int64_t ldd, int64_t strideD,
                                  double diag_add, const double* norm2, volatile double* host) {
  dependency_wait();
  release_dependents();
  const int b = blockIdx.y;
  const double* S = src + b * strideS;
  double* D = dst + b * strideD;
  if (norm2) {
    s = 1.0 / sqrt(*norm2);
    if (blockIdx.x == 0 && threadIdx.x == 0) {
      *host = *norm2;
      __threadfence_system();
    }
  }
  map_entries(
      m, n,
      [&](int i, int j) {
        const double v = s * S[i + j * lds];
        return i == j ? v + diag_add : v;
      },
      [&](int i, int j, double v) { D[i + j * ldd] = v; });
}

__global__ void form_stack_kernel(int m, int mpad, int n, const double* X, int64_t ldx, double* W,
                                  int64_t ldw, int64_t strideW, const double* s_vec, double s_scalar,
                                  int x_upper, int64_t strideX) {
  dependency_wait();
  release_dependents();
  const int b = blockIdx.y;
  X += b * strideX;
  double* Wb = W + b * strideW;
  const double s = s_vec ? s_vec[b] : s_scalar;
  const int rows = mpad + n;
  map_entries(
      rows, n,
      [&](int i, int j) {
        if (i < m) return (x_upper && i > j) ? 0.0 : X[i + j * ldx];
        return (i - mpad == j) ? s : 0.0;
      },
      [&](int i, int j, double v) { Wb[i + j * ldw] = v; });
}

__global__ void shift_lower_kernel(int n, const double* G, int64_t ldg, double* W,
                                   int64_t ldw, int64_t strideW, const double* c_vec) {
  dependency_wait();
  release_dependents();
  const int b = blockIdx.y;
  double* Wb = W + b * strideW;
  const double c = c_vec[b];
  for_entries(n, n, [&](int i, int j) {
    if (i < j) return;
    double v = G[i + j * ldg];
    if (i == j) v += c;
    Wb[i + j * ldw] = v;
  });
}

template <int BS>
__device__ double block_sum(double v, double* sh) {
  v = warp_sum(v);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  if (l == 0) sh[w] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x == 0) {
    for (int i = 0; i < BS / 32; ++i) r += sh[i];
  }
  __syncthreads();
  return r;
}

__global__ void frob2_kernel(int m, int n, const double* X, int64_t ldx, double* partial) {
  dependency_wait();
  release_dependents();
  __shared__ double sh[TPB / 32];
  double s = 0.0;
  map_entries(m, n, [&](int i, int j) { return X[i + j * ldx]; }, [&](int, int, double v) { s += v * v; });
  s = block_sum<TPB>(s, sh);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}

__global__ void reduce_sum_kernel(const double* partial, int count, double* out) {
  dependency_wait();
  release_dependents();
  __shared__ double sh[TPB / 32];
  double s = 0.0;
  for (int i = threadIdx.x; i < count; i += blockDim.x) s += partial[i];
  s = block_sum<TPB>(s, sh);
  if (threadIdx.x == 0) out[0] = s;
}

__global__ void colsum_abs_kernel(int m, int n, const double* X, int64_t ldx, double* colsum) {
  dependency_wait();
  release_dependents();
  __shared__ double sh[TPB / 32];
  for (int j = blockIdx.x; j < n; j += gridDim.x) {
    double s = 0.0;
    for (int i = threadIdx.x; i < m; i += blockDim.x) s += fabs(X[i + j * ldx]);
    s = block_sum<TPB>(s, sh);
    if (threadIdx.x == 0) colsum[j] = s;
  }
}

__global__ void max_kernel(const double* v, int count, double* out) {
  dependency_wait();
  release_dependents();
  __shared__ double sh[TPB];
  double s = 0.0;
  for (int i = threadIdx.x; i < count; i += blockDim.x) s = fmax(s, v[i]);
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int o = TPB / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] = fmax(sh[threadIdx.x], sh[threadIdx.x + o]);
    __syncthreads();
  }
  if (threadIdx.x == 0) out[0] = sh[0];
}

// X_new = cx*X + cz*sum_q Z_q ; partial = ||X_new - X||^2 per block.  In place on X.  X stays as it is when one
// of info[0 .. ninfo) is not zero (a select, not a branch: the loads are in flight together).
__global__ void combine_kernel(int m, int n, double* X, int64_t ldx, const double* Z,
                               int64_t ldz, int64_t strideZ, int nz, double cx, double cz,
                               const double* cz_vec, double* partial, const int* info, int ninfo) {
  dependency_wait();
  release_dependents();
  __shared__ double sh[TPB / 32];
  double s = 0.0;
  int stop = 0;
  for (int k = 0; k < ninfo; ++k) stop |= info[k];
  auto update = [&](int i, int j, double x, double z) {
    const double xn = stop ? x : cx * x + (cz_vec ? z : z * cz);
    const double d = x - xn;
    s += d * d;
    X[i + j * ldx] = xn;
  };
  if (nz == 1) {
    const double w = cz_vec ? cz_vec[0] : 1.0;
    map_entries(
        m, n, [&](int i, int j) { return make_double2(X[i + j * ldx], 0.0 + w * Z[i + j * ldz]); },
        [&](int i, int j, double2 v) { update(i, j, v.x, v.y); });
  } else {
    // several Z are already as many loads in flight
    for_entries(m, n, [&](int i, int j) {
      const double x = X[i + j * ldx];
      double z = 0.0;
      for (int q = 0; q < nz; ++q) z += (cz_vec ? cz_vec[q] : 1.0) * Z[q * strideZ + i + j * ldz];
      update(i, j, x, z);
    });
  }
  s = block_sum<TPB>(s, sh);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}

__global__ void symmetrize_kernel(int n, double* B, int64_t ldb) {
  dependency_wait();
  release_dependents();
  for_entries(n, n, [&](int i, int j) {
    if (i <= j) return;  // each pair once, by the lower element
    const double a = B[i + j * ldb], b = B[j + i * ldb];
    const double h = 0.5 * b + 0.5 * a;
    B[i + j * ldb] = h;
    B[j + i * ldb] = h;
  });
}

__global__ void transpose_kernel(int m, int n, const double* A, int64_t lda, double* B,
                                 int64_t ldb) {
  dependency_wait();
  release_dependents();
  __shared__ double tile[32][33];
  const int i0 = blockIdx.x * 32, j0 = blockIdx.y * 32;
  for (int jj = threadIdx.y; jj < 32; jj += blockDim.y) {
    const int i = i0 + threadIdx.x, j = j0 + jj;
    if (i < m && j < n) tile[jj][threadIdx.x] = A[i + static_cast<int64_t>(j) * lda];
  }
  __syncthreads();
  for (int ii = threadIdx.y; ii < 32; ii += blockDim.y) {
    const int j = j0 + threadIdx.x, i = i0 + ii;
    if (i < m && j < n) B[j + static_cast<int64_t>(i) * ldb] = tile[threadIdx.x][ii];
  }
}

// Newton-Schulz step matrix from the lower triangle of G = X^T X: G <- (3I - G)/2
// (both triangles written; only when `write`) and partial[block] = sum of (G - I)^2
// over all entries.
__global__ void ns_prepare_kernel(int n, double* G, int64_t ldg, int write, double* partial) {
  dependency_wait();
  release_dependents();
  __shared__ double sh[TPB / 32];
  double s = 0.0;
  for_entries(n, n, [&](int i, int j) {
    if (i < j) return;
    const double g = G[i + j * ldg];
    const double d = (i == j) ? g - 1.0 : g;
    s += (i == j) ? d * d : 2.0 * d * d;
    if (!write) return;
    const double v = (i == j) ? 1.5 - 0.5 * g : -0.5 * g;
    G[i + j * ldg] = v;
    if (i != j) G[j + i * ldg] = v;
  });
  s = block_sum<TPB>(s, sh);
  if (threadIdx.x == 0) partial[blockIdx.x] = s;
}

// B(j, i) = B(i, j) for i > j: the lower triangle copied to the upper one
__global__ void mirror_lower_kernel(int n, double* B, int64_t ldb) {
  dependency_wait();
  release_dependents();
  for_entries(n, n, [&](int i, int j) {
    if (i > j) B[j + static_cast<int64_t>(i) * ldb] = B[i + static_cast<int64_t>(j) * ldb];
  });
}

__global__ void copy_upper_kernel(int n, const double* A, int64_t lda, double scale, double* B,
                                  int64_t ldb) {
  dependency_wait();
  release_dependents();
  map_entries(
      n, n, [&](int i, int j) { return (i <= j) ? scale * A[i + static_cast<int64_t>(j) * lda] : 0.0; },
      [&](int i, int j, double v) { B[i + static_cast<int64_t>(j) * ldb] = v; });
}

__global__ void set_identity_kernel(int m, int n, double* Q, int64_t ldq, int64_t strideQ, double diag) {
  dependency_wait();
  release_dependents();
  double* Qb = Q + blockIdx.y * strideQ;
  for_entries(m, n, [&](int i, int j) {
    Qb[i + j * ldq] = (i == j) ? diag : 0.0;
  });
}

__global__ void add_diag_kernel(int n, double* A, int64_t lda, double d) {
  dependency_wait();
  release_dependents();
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
    A[i + i * lda] += d;
}

__device__ __forceinline__ uint64_t mix64(uint64_t z) {
  // SplitMix64 finaliser (Steele, Lea, Flood 2014)
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

__global__ void fill_random_kernel(int m, int n, double* X, int64_t ldx, uint64_t seed) {
  for_entries(m, n, [&](int i, int j) {
    const uint64_t r = mix64(seed * 0x100000001B3ull + static_cast<uint64_t>(i + static_cast<int64_t>(j) * m));
    X[i + j * ldx] = 2.0 * (static_cast<double>(r >> 11) * (1.0 / 9007199254740992.0)) - 1.0;
  });
}

__global__ void trace_kernel(int n, const double* A, int64_t lda, double* out) {
  __shared__ double sh[TPB / 32];
  double s = 0.0;
  for (int i = threadIdx.x; i < n; i += blockDim.x) s += A[i + i * lda];
  s = block_sum<TPB>(s, sh);
  if (threadIdx.x == 0) out[0] = s;
}

__global__ void gather_columns_kernel(int m, int n, const double* __restrict__ A, int64_t lda, const int* perm,
                                      double* B, int64_t ldb) {
  for_entries(m, n, [&](int i, int j) {
    B[i + j * ldb] = A[i + static_cast<int64_t>(perm[j]) * lda];
  });
}

__global__ void get_diag_kernel(int n, const double* A, int64_t lda, double* d) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) d[i] = A[i + i * lda];
}

}  // namespace

cudaError_t fill_random(int m, int n, double* X, int64_t ldx, uint64_t seed, cudaStream_t st) {
  if (m <= 0 || n <= 0) return cudaSuccess;
  fill_random_kernel<<<grid_for(static_cast<int64_t>(m) * n), TPB, 0, st>>>(m, n, X, ldx, seed);
  return cudaGetLastError();
}

cudaError_t trace(int n, const double* A, int64_t lda, double* out, cudaStream_t st) {
  trace_kernel<<<1, TPB, 0, st>>>(n, A, lda, out);
  return cudaGetLastError();
}

cudaError_t gather_columns(int m, int n, const double* A, int64_t lda, const int* perm, double* B, int64_t ldb,
                           cudaStream_t st) {
  if (m <= 0 || n <= 0) return cudaSuccess;
  gather_columns_kernel<<<grid_for(static_cast<int64_t>(m) * n), TPB, 0, st>>>(m, n, A, lda, perm, B, ldb);
  return cudaGetLastError();
}

cudaError_t get_diag(int n, const double* A, int64_t lda, double* d, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  get_diag_kernel<<<(n + TPB - 1) / TPB, TPB, 0, st>>>(n, A, lda, d);
  return cudaGetLastError();
}

cudaError_t scale_copy(int m, int n, double s, const double* src, int64_t lds, int64_t strideS, double* dst,
                       int64_t ldd, int64_t strideD, int batch, double diag_add, cudaStream_t st) {
  if (m <= 0 || n <= 0 || batch <= 0) return cudaSuccess;
  return launch_dependent(scale_copy_kernel, dim3(grid_for(static_cast<int64_t>(m) * n), batch), dim3(TPB), 0, st, dim3(1), m, n, s, src, lds, strideS, dst, ldd, strideD, diag_add, nullptr, nullptr);
}

cudaError_t scale_by_norm(int m, int n, const double* norm2, double* X, int64_t ldx, volatile double* host,
                          cudaStream_t st) {
  if (m <= 0 || n <= 0) return cudaSuccess;
  return launch_dependent(scale_copy_kernel, dim3(grid_for(static_cast<int64_t>(m) * n)), dim3(TPB), 0, st, dim3(1), m,
                          n, 0.0, X, ldx, 0, X, ldx, 0, 0.0, norm2, host);
}

cudaError_t form_stack(int m, int mpad, int n, const double* X, int64_t ldx, double* W, int64_t ldw,
                       int64_t strideW, const double* s_vec, double s_scalar, int batch, cudaStream_t st,
                       int x_upper, int64_t strideX) {
  if (n <= 0 || batch <= 0) return cudaSuccess;
  if (mpad < m) return cudaErrorInvalidValue;
  return launch_dependent(form_stack_kernel, dim3(grid_for(static_cast<int64_t>(mpad + n) * n), batch), dim3(TPB), 0, st, dim3(1), m, mpad, n, X, ldx, W, ldw, strideW, s_vec, s_scalar, x_upper, strideX);
}

cudaError_t shift_lower(int n, const double* G, int64_t ldg, double* W, int64_t ldw, int64_t strideW,
                        const double* c_vec, int batch, cudaStream_t st) {
  if (n <= 0 || batch <= 0) return cudaSuccess;
  return launch_dependent(shift_lower_kernel, dim3(grid_for(static_cast<int64_t>(n) * n), batch), dim3(TPB), 0, st, dim3(1), n, G, ldg, W, ldw, strideW, c_vec);
}

cudaError_t reduce_sum(const double* partial, int count, double* out, cudaStream_t st) {
  return launch_dependent(reduce_sum_kernel, dim3(1), dim3(TPB), 0, st, dim3(1), partial, count, out);
}

cudaError_t frob2(int m, int n, const double* X, int64_t ldx, double* partial, double* out, cudaStream_t st) {
  const int blocks = std::min(grid_for(static_cast<int64_t>(m) * n), 1024);
  cudaError_t e = launch_dependent(frob2_kernel, dim3(blocks), dim3(TPB), 0, st, dim3(1), m, n, X, ldx, partial);
  if (e != cudaSuccess) return e;
  return reduce_sum(partial, blocks, out, st);
}

cudaError_t norm1(int m, int n, const double* X, int64_t ldx, double* colsum, double* out, cudaStream_t st) {
  cudaError_t e = launch_dependent(colsum_abs_kernel, dim3(std::min(n, 4096)), dim3(TPB), 0, st, dim3(1), m, n, X, ldx, colsum);
  if (e != cudaSuccess) return e;
  return launch_dependent(max_kernel, dim3(1), dim3(TPB), 0, st, dim3(1), colsum, n, out);
}

cudaError_t combine_update(int m, int n, double* X, int64_t ldx, const double* Z, int64_t ldz, int64_t strideZ,
                           int nz, double cx, double cz, const double* cz_vec, double* partial, double* err2,
                           cudaStream_t st, const int* info, int ninfo) {
  const int blocks = std::min(grid_for(static_cast<int64_t>(m) * n), 1024);
  cudaError_t e = launch_dependent(combine_kernel, dim3(blocks), dim3(TPB), 0, st, dim3(1), m, n, X, ldx, Z, ldz, strideZ, nz, cx, cz, cz_vec, partial, info, ninfo);
  if (e != cudaSuccess) return e;
  return reduce_sum(partial, blocks, err2, st);
}

cudaError_t symmetrize(int n, double* B, int64_t ldb, cudaStream_t st) {
  return launch_dependent(symmetrize_kernel, dim3(grid_for(static_cast<int64_t>(n) * n)), dim3(TPB), 0, st, dim3(1), n, B, ldb);
}

cudaError_t transpose(int m, int n, const double* A, int64_t lda, double* B, int64_t ldb, cudaStream_t st) {
  dim3 grid((m + 31) / 32, (n + 31) / 32);
  return launch_dependent(transpose_kernel, grid, dim3(32, 8), 0, st, dim3(1), m, n, A, lda, B, ldb);
}

cudaError_t ns_prepare(int n, double* G, int64_t ldg, double* partial, double* err2, int write, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  const int blocks = static_cast<int>(std::min<int64_t>(grid_for(static_cast<int64_t>(n) * n), 1024));
  cudaError_t e = launch_dependent(ns_prepare_kernel, dim3(blocks), dim3(TPB), 0, st, dim3(1), n, G, ldg, write, partial);
  if (e != cudaSuccess) return e;
  return reduce_sum(partial, blocks, err2, st);
}

cudaError_t copy_upper(int n, const double* A, int64_t lda, double scale, double* B, int64_t ldb, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  return launch_dependent(copy_upper_kernel, dim3(grid_for(static_cast<int64_t>(n) * n)), dim3(TPB), 0, st, dim3(1), n, A, lda, scale, B, ldb);
}

cudaError_t mirror_lower(int n, double* B, int64_t ldb, cudaStream_t st) {
  if (n <= 0) return cudaSuccess;
  return launch_dependent(mirror_lower_kernel, dim3(grid_for(static_cast<int64_t>(n) * n)), dim3(TPB), 0, st, dim3(1), n, B, ldb);
}

cudaError_t set_identity(int m, int n, double* Q, int64_t ldq, int64_t strideQ, int batch, double diag,
                         cudaStream_t st) {
  if (m <= 0 || n <= 0 || batch <= 0) return cudaSuccess;
  return launch_dependent(set_identity_kernel, dim3(grid_for(static_cast<int64_t>(m) * n), batch), dim3(TPB), 0, st, dim3(1), m, n, Q, ldq, strideQ, diag);
}

cudaError_t add_diag(int n, double* A, int64_t lda, double d, cudaStream_t st) {
  return launch_dependent(add_diag_kernel, dim3(std::max(1, (n + TPB - 1) / TPB)), dim3(TPB), 0, st, dim3(1), n, A, lda, d);
}

}  // namespace zolo
