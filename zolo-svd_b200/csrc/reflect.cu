// Block reflector of one Householder panel applied in one launch:
// C <- (I - V op(T) V^T) C, V m x w unit lower trapezoidal (w <= 32), read where the QR left it.
//
// Between two panels this is on the critical path of the factorization, and as three products
// (V^T C, T, C - V P) it was four launches of 5 to 12 us each.  Here a cluster of CTAs holds
// 16 columns of C: every CTA keeps its rows of V and C in shared memory, the partial
// V^T C are summed over the cluster through distributed shared memory (each CTA sums and multiplies
// by op(T) its share of the 16 columns and sends them to all), and C - V P is written from
// shared memory, so C is read and written once.  Both products run on the FP64 tensor path;
// at w = 32 they are 8 flops per byte of C, above the 5.4 at which HBM would bound them, so small
// calls are bound by latency (7 to 8 us up to 1024 x 96, 13 at 4096 rows) and large ones by DMMA.
#include "common.cuh"
#include "kernels.h"

#include <cooperative_groups.h>

#include <algorithm>

namespace cg = cooperative_groups;

namespace zolo {

namespace {

constexpr int RW = 32;    // reflector width
constexpr int RN = 16;    // columns of C per cluster
constexpr int RT = 128;   // threads
constexpr int RP = RW + 4;     // = 4 mod 16: conflict-free fragment loads
constexpr int kMaxRows = 512;  // rows of one CTA

struct ReflArgs {
  int m, nc, w, trans;
  const double* V;
  int64_t ldv, strideV;
  const double* T;
  int64_t strideT;
  double* C;
  int64_t ldc, strideC;
  int split;
  int64_t gap;
  int rows_per, ld;  // rows of a CTA, leading dimension of its shared-memory copies
};

constexpr int smem_elems(int ld) { return (RW + RN) * ld + RT / 32 * RN * RP + RN * RP + RW * (RW + 1); }

// A16: V and C move in 16-byte pairs of rows (aligned bases, even leading dimensions, split and gap)
template <bool A16>
__global__ void __launch_bounds__(RT) reflect_kernel(ReflArgs p) {
  extern __shared__ __align__(16) double sm[];
  cg::cluster_group cluster = cg::this_cluster();
  const int CL = static_cast<int>(cluster.num_blocks()), rank = static_cast<int>(cluster.block_rank());
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
  const int b = blockIdx.y, n0 = (blockIdx.x / CL) * RN;
  const int ld = p.ld;
  double* Vs = sm;
  double* Cs = Vs + RW * ld;
  double* Pp = Cs + RN * ld;                 // by warp
  double* Pc = Pp + RT / 32 * RN * RP;       // this CTA's sum
  double* Pf = Pp + RT / 32 * RW;            // op(T) V^T C: over Pp, once every CTA has summed its own
  double* Ts = Pc + RN * RP;
  const int r0 = rank * p.rows_per;
  const int nloc = max(min(p.m, r0 + p.rows_per) - r0, 0);
  const int rpad = (p.rows_per + 15) / 16 * 16;
  const double* V = p.V + b * p.strideV;
  double* C = p.C + b * p.strideC;

  // rows r0 .. of V's and C's columns; zeros past the rows, the reflectors and the columns
  auto fetch = [&](double* dst, const double* src, int64_t lds, int cols, int valid) {
    if (A16) {
      const int per = rpad / 2;
      for (int e = tid; e < cols * per; e += RT) {
        const int c = e / per, l = (e - c * per) * 2, r = r0 + l;
        const int rows = c < valid ? min(max(nloc - l, 0), 2) : 0;
        const double* s = rows ? src + r + (r >= p.split ? p.gap : 0) + c * lds : src;
        cp_async16(dst + l + c * ld, s, rows * 8);
      }
    } else {
      for (int e = tid; e < cols * rpad; e += RT) {
        const int c = e / rpad, l = e - c * rpad, r = r0 + l;
        const bool ok = c < valid && l < nloc;
        const double* s = ok ? src + r + (r >= p.split ? p.gap : 0) + c * lds : src;
        cp_async8(dst + l + c * ld, s, ok ? 8 : 0);
      }
    }
  };
  dependency_wait();
  fetch(Vs, V, p.ldv, RW, p.w);
  fetch(Cs, C + n0 * p.ldc, p.ldc, RN, min(RN, p.nc - n0));
  cp_async_commit();
  // op(T) as Ts[i * (RW + 1) + j] = op(T)(i, j)
  const double* T = p.T + b * p.strideT;
  for (int e = tid; e < RW * RW; e += RT) {
    const int i = e & (RW - 1), j = e / RW;
    const double v = (i < p.w && j < p.w && i <= j) ? T[i + j * RW] : 0.0;
    Ts[p.trans ? j * (RW + 1) + i : i * (RW + 1) + j] = v;
  }
  cp_async_wait<0>();
  __syncthreads();
  if (r0 < RW) {
    // the unit lower trapezoid: the QR stores R in and above V's diagonal
    for (int e = tid; e < RW * RW; e += RT) {
      const int r = e & (RW - 1), i = e / RW, l = r - r0;
      if (l < 0 || l >= nloc || i >= p.w || r > i) continue;
      Vs[l + i * ld] = r == i ? 1.0 : 0.0;
    }
    __syncthreads();
  }

  // ---- V^T C over this CTA's rows, 8 rows a step, the steps dealt to the warps ----
  {
    double acc[2][2][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[i][j][q] = 0.0;
#pragma unroll 2
    for (int k = warp * 8; k < rpad; k += RT / 32 * 8) {
      double af[2][4], bf[2][2];
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const double* v = Vs + k + t + (16 * i + g) * ld;
        af[i][0] = v[0];
        af[i][1] = v[8 * ld];
        af[i][2] = v[4];
        af[i][3] = v[8 * ld + 4];
      }
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const double* c = Cs + k + t + (8 * j + g) * ld;
        bf[j][0] = c[0];
        bf[j][1] = c[4];
      }
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) dmma_16x8x8(acc[i][j], af[i], bf[j]);
    }
    double* P = Pp + warp * RN * RP;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        double* d = P + 16 * i + g + (8 * j + 2 * t) * RP;
        d[0] = acc[i][j][0];
        d[RP] = acc[i][j][1];
        d[8] = acc[i][j][2];
        d[8 + RP] = acc[i][j][3];
      }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < RN * RW / RT; ++q) {
    const int e = tid + q * RT, o = (e & (RW - 1)) + e / RW * RP;
    double s = 0.0;
#pragma unroll
    for (int u = 0; u < RT / 32; ++u) s += Pp[u * RN * RP + o];
    Pc[o] = s;
  }
  if (CL > 1) cluster.sync();
  else __syncthreads();
  // ---- this CTA's columns: summed over the cluster in rank order, times op(T), sent to all ----
  const int cols = RN / CL;  // CL is a power of two up to 16
  for (int c = rank * cols + warp; c < (rank + 1) * cols; c += RT / 32) {
    double s4[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int q = 0; q < 16; ++q)
      if (q < CL) s4[q & 3] += *cluster.map_shared_rank(Pc + lane + c * RP, q);
    double* x = Pp + warp * RW;
    x[lane] = (s4[0] + s4[1]) + (s4[2] + s4[3]);
    __syncwarp();
    double y[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for (int j = 0; j < RW; ++j) y[j & 3] = fma(Ts[lane * (RW + 1) + j], x[j], y[j & 3]);
    const double v = (y[0] + y[1]) + (y[2] + y[3]);
#pragma unroll 4
    for (int q = 0; q < CL; ++q) *cluster.map_shared_rank(Pf + lane + c * RP, (rank + q) & (CL - 1)) = v;
    __syncwarp();
  }
  if (CL > 1) cluster.sync();
  else __syncthreads();
  release_dependents();
  // ---- C - V P, 16 rows x 16 columns at a time ----
  for (int l0 = warp * 16; l0 < nloc; l0 += RT / 32 * 16) {
    double acc[2][4];
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[j][q] = 0.0;
#pragma unroll
    for (int k = 0; k < RW; k += 8) {
      double af[4];
      const double* v = Vs + l0 + g + (k + t) * ld;
      af[0] = v[0];
      af[1] = v[8];
      af[2] = v[4 * ld];
      af[3] = v[4 * ld + 8];
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        const double* q = Pf + k + t + (8 * j + g) * RP;
        const double bf[2] = {q[0], q[4]};
        dmma_16x8x8(acc[j], af, bf);
      }
    }
#pragma unroll
    for (int j = 0; j < 2; ++j)
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int l = l0 + g + (q & 2 ? 8 : 0), c = 8 * j + 2 * t + (q & 1), r = r0 + l;
        if (l < nloc && n0 + c < p.nc)
          C[r + (r >= p.split ? p.gap : 0) + (n0 + c) * p.ldc] = Cs[l + c * ld] - acc[j][q];
      }
  }
}

}  // namespace

bool reflect_applies(int m) { return m >= 1 && m <= panel_cluster_max() * kMaxRows; }

cudaError_t reflect(int m, int nc, int w, const double* V, int64_t ldv, int64_t strideV, const double* T,
                    int64_t strideT, int trans, double* C, int64_t ldc, int64_t strideC, int batch, cudaStream_t st,
                    int split, int64_t gap) {
  if (m <= 0 || nc <= 0 || w <= 0 || batch <= 0) return cudaSuccess;
  if (w > RW || !reflect_applies(m) || batch > 65535 || gap < 0) return cudaErrorInvalidValue;
  ReflArgs p;
  p.m = m;
  p.nc = nc;
  p.w = w;
  p.trans = trans;
  p.V = V;
  p.ldv = ldv;
  p.strideV = strideV;
  p.T = T;
  p.strideT = strideT;
  p.C = C;
  p.ldc = ldc;
  p.strideC = strideC;
  p.split = (split > 0 && gap > 0) ? split : m;
  p.gap = gap;
  // 64 rows a CTA while that leaves SMs idle, 128 otherwise; clusters of 16 then grow the rows
  const int64_t tiles = static_cast<int64_t>((nc + RN - 1) / RN) * batch;
  const int target = tiles * ((m + 63) / 64) <= 2 * static_cast<int64_t>(num_sms()) ? 64 : 128;
  const int maxcl = panel_cluster_max();
  int cl = 1;
  while (cl < maxcl && (m + cl - 1) / cl > target) cl *= 2;
  p.rows_per = ((m + cl - 1) / cl + 7) / 8 * 8;
  const int rpad = (p.rows_per + 15) / 16 * 16;
  p.ld = rpad + 4;  // = 4 mod 16
  const size_t smem = smem_elems(p.ld) * sizeof(double);
  auto al = [](const void* q, int64_t ld, int64_t stride) {
    return reinterpret_cast<uintptr_t>(q) % 16 == 0 && ld % 2 == 0 && stride % 2 == 0;
  };
  const bool a16 = al(V, ldv, batch > 1 ? strideV : 0) && al(C, ldc, batch > 1 ? strideC : 0) &&
                   (p.split >= m || (p.split % 2 == 0 && gap % 2 == 0));
  static std::atomic<int> attr_set[kMaxDevices];
  const cudaError_t attr = once_per_device(attr_set, [] {
    const int most = static_cast<int>(smem_elems(kMaxRows + 4) * sizeof(double));
    for (const void* f : {reinterpret_cast<const void*>(reflect_kernel<true>),
                          reinterpret_cast<const void*>(reflect_kernel<false>)}) {
      cudaError_t e = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, most);
      if (e == cudaSuccess) e = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
      if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
  });
  if (attr != cudaSuccess) return attr;
  const dim3 grid(static_cast<unsigned>(cl * ((nc + RN - 1) / RN)), batch, 1);
  return launch_dependent(a16 ? reflect_kernel<true> : reflect_kernel<false>, grid, dim3(RT), smem, st, dim3(cl), p);
}

}  // namespace zolo
