// FP64 GEMM on the sm_100a FP64 tensor path (DMMA mma.sync.m16n8k8.f64).
//
// tcgen05.mma has no FP64 kind, so the FP64 contractions of the polar
// iterations (Gram matrix, TRSM updates, Householder trailing updates,
// Q1*Q2^T) run on DMMA.  General shapes: CTA tile 64x64x16, 4 warps of 32x32, double-buffered
// cp.async, four CTAs per SM: independent CTAs cover each other's barriers and epilogues, and the
// small tile leaves less of the last wave idle (4096^3 31.2 TF/s and its lower triangle 29.4, against
// 31.0 with 64x128 tiles and 27.5 with eight warps on 64x64; V^T C of a 128-column block, 128 x 4096 x
// 4096 of four, 25 -> 28.7; the FP64 tensor pipe saturates at 37.0).  Padded shared-memory
// layouts make every fragment load a conflict-free LDS.128 (or LDS.64 for
// op(B)=B^T).  Products too small for that grid take 32x32 tiles with four warps, and a long K
// is split over the CTAs of a cluster, which reduce through distributed shared memory
// (1024 x 512 x 512: 72 -> 30 us against one launch with scratch in global memory).
//
// Index permutations (free because they are applied consistently):
//   * inside each 16-row MMA tile, logical row g <-> physical row 2g and
//     logical row g+8 <-> physical row 2g+1, so a thread's two A rows are
//     adjacent in memory;
//   * inside each 8-wide k step, logical k slot t <-> physical k 2t and slot
//     t+4 <-> 2t+1 for both operands, so a thread's two k values are adjacent.
#include "common.cuh"
#include "kernels.h"

#include <cooperative_groups.h>

#include <algorithm>

namespace cg = cooperative_groups;

namespace zolo {

namespace {

constexpr int BK = 16;
constexpr int LDA_T = BK + 4;  // sA[m][k]  (op(A) = A^T)
constexpr int LDB_N = BK + 8;  // sB[n][k]  (op(B) = B)

// CTA tile BM x BN, WM x WN warps, each warp owns (BM/WM) x (BN/WN) = MI m16 x NJ n8 MMA tiles.
template <int BM_, int BN_, int WM_, int WN_, int ST_ = 4, int MINB_ = 1>
struct Cfg {
  static constexpr int BM = BM_, BN = BN_, WM = WM_, WN = WN_, STAGES = ST_, MINB = MINB_;
  static constexpr int NT = WM * WN * 32;
  static constexpr int MI = BM / WM / 16, NJ = BN / WN / 8;
  static constexpr int LDA_N = BM + 2;  // sA[k][m]  (op(A) = A)
  static constexpr int LDB_T = BN + 2;  // sB[k][n]  (op(B) = B^T)
  static constexpr int SMEM_C = BN * (BM + 2) * 8;  // a tile of C
  __host__ __device__ static constexpr int a_elems(bool ta) { return ta ? BM * LDA_T : BK * LDA_N; }
  __host__ __device__ static constexpr int b_elems(bool tb) { return tb ? BK * LDB_T : BN * LDB_N; }
  __host__ __device__ static constexpr int smem(bool ta, bool tb) { return ST_ * (a_elems(ta) + b_elems(tb)) * 8; }
};
using CfgWide = Cfg<64, 64, 2, 2, 2, 4>;      // general: 4 CTAs / SM of 4 warps, warp tile 32x32
using CfgSkinnyM = Cfg<32, 64, 1, 8, 4, 3>;    // M <= 32 (V^T W products of the QR updates)
using CfgSmall = Cfg<64, 64, 2, 4, 2, 3>;      // K <= 64 rank-k updates and N <= 64: 3 CTAs / SM
using CfgTiny = Cfg<32, 32, 2, 2, 4, 4>;       // products too small to fill the GPU with larger tiles

struct KParams {
  GemmArgs g;
  int tiles_m, tiles_n;
  int splitk;   // slices of K, blockIdx.y
  int cluster;  // the slices that one cluster sums: all of them, or groups whose sums go to P
  double* P;    // partial sums of the groups: M x N (ld ldp) for each group and batch entry
  int64_t ldp;
  int stage_c;  // C copied to shared memory beside the first K tiles (rank-k updates)
};

// GROUPS: a kernel of its own, so that the general one's code stays as it is (with both in one, 128 x 1024 x 4096
// went from 61.5 to 69.5 us)
template <class C, bool TA, bool TB, bool V16, bool GROUPS>
__global__ void __launch_bounds__(C::NT, C::MINB) dgemm_kernel(KParams kp) {
  constexpr int NT = C::NT;
  constexpr int BM = C::BM, BN = C::BN, MI = C::MI, NJ = C::NJ;
  constexpr int LDA_N = C::LDA_N, LDB_T = C::LDB_T;
  constexpr int AE = C::a_elems(TA), BE = C::b_elems(TB);
  constexpr int STAGES = C::STAGES;
  extern __shared__ __align__(16) double smem[];
  const GemmArgs& p = kp.g;
  double* sAb = smem;
  double* sBb = smem + STAGES * AE;

  const int bz = blockIdx.z;
  const int split = blockIdx.y;
  int tm, tn;
  if (p.tri) {
    const int t = blockIdx.x;
    int r = static_cast<int>((sqrtf(8.0f * t + 1.0f) - 1.0f) * 0.5f);
    while ((r + 1) * (r + 2) / 2 <= t) ++r;
    while (r * (r + 1) / 2 > t) --r;
    tm = r;
    tn = t - r * (r + 1) / 2;
  } else {
    const int G = 8;
    const int t = blockIdx.x;
    const int group = t / (G * kp.tiles_n);
    const int first = group * G;
    const int gsz = min(kp.tiles_m - first, G);
    const int in = t - group * G * kp.tiles_n;
    tm = first + in % gsz;
    tn = in / gsz;
  }
  const int m0 = tm * BM, n0 = tn * BN;
  const int M = p.M, N = p.N;

  int kb = 0, ke = p.K;
  if (p.kfrom_n) kb = min((p.kfrom_n == 1 ? n0 : (p.kfrom_n == 2 ? m0 : max(m0, n0))) / BK * BK, ke);
  if (p.kto_m) ke = max(kb, min(ke, p.kto_m == 2 ? n0 + BN : m0 + BM));
  if (kp.splitk > 1) {
    const int span = ke - kb;
    int len = (span + kp.splitk - 1) / kp.splitk;
    len = (len + BK - 1) / BK * BK;
    const int nb = kb + split * len;
    kb = min(nb, ke);
    ke = min(nb + len, ke);
  }

  const double* A = p.A + static_cast<int64_t>(bz) * p.strideA;
  const double* B = p.B + static_cast<int64_t>(bz) * p.strideB;
  const int64_t lda = p.lda, ldb = p.ldb;
  const int tid = threadIdx.x;

  // 16-byte chunks (two FP64 values along the contiguous dimension).  V16: one
  // cp.async of 16 bytes with zero fill; otherwise two 8-byte copies.
  auto chunk = [&](double* dst, const double* base, int64_t off0, bool in0, bool in1) {
    if (V16) {
      const int bytes = in0 ? (in1 ? 16 : 8) : 0;
      cp_async16(dst, bytes ? base + off0 : base, bytes);
    } else {
      cp_async8(dst, in0 ? base + off0 : base, in0 ? 8 : 0);
      cp_async8(dst + 1, in1 ? base + off0 + 1 : base, in1 ? 8 : 0);
    }
  };
  auto load_stage = [&](int stage, int k0) {
    double* sa = sAb + stage * AE;
    double* sb = sBb + stage * BE;
    for (int c = tid; c < BM * BK / 2; c += NT) {
      if (!TA) {
        const int k = c / (BM / 2), m = (c % (BM / 2)) * 2;
        const int gm = m0 + m, gk = k0 + k;
        const bool kin = gk < ke;
        chunk(sa + k * LDA_N + m, A, gm + static_cast<int64_t>(gk) * lda, kin && gm < M, kin && gm + 1 < M);
      } else {
        const int m = c / (BK / 2), k = (c % (BK / 2)) * 2;
        const int gm = m0 + m, gk = k0 + k;
        const bool mi = gm < M;
        chunk(sa + m * LDA_T + k, A, gk + static_cast<int64_t>(gm) * lda, mi && gk < ke, mi && gk + 1 < ke);
      }
    }
    for (int c = tid; c < BN * BK / 2; c += NT) {
      if (!TB) {
        const int n = c / (BK / 2), k = (c % (BK / 2)) * 2;
        const int gn = n0 + n, gk = k0 + k;
        const bool ni = gn < N;
        chunk(sb + n * LDB_N + k, B, gk + static_cast<int64_t>(gn) * ldb, ni && gk < ke, ni && gk + 1 < ke);
      } else {
        const int k = c / (BN / 2), n = (c % (BN / 2)) * 2;
        const int gn = n0 + n, gk = k0 + k;
        const bool kin = gk < ke;
        chunk(sb + k * LDB_T + n, B, gn + static_cast<int64_t>(gk) * ldb, kin && gn < N, kin && gn + 1 < N);
      }
    }
  };

  const int warp = tid >> 5, lane = tid & 31;
  const int g = lane >> 2, t = lane & 3;
  const int wm = (warp % C::WM) * (BM / C::WM);
  const int wn = (warp / C::WM) * (BN / C::WN);

  double acc[MI][NJ][4];
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
      for (int r = 0; r < 4; ++r) acc[i][j][r] = 0.0;

  const int ktiles = (ke > kb) ? (ke - kb + BK - 1) / BK : 0;
  // Rank-k updates C += alpha A B of a short K spend as long on C as on the product: its tile is
  // copied to shared memory behind the first K tile, so that no thread waits for it.
  constexpr int LDC_S = BM + 2;
  double* sC = smem + STAGES * (AE + BE);
  const bool stage_c = kp.stage_c;
  dependency_wait();
#pragma unroll
  for (int s = 0; s < STAGES - 1; ++s) {
    if (s < ktiles) load_stage(s, kb + s * BK);
    cp_async_commit();
    if (s == 0 && stage_c) {
      const double* Cb = p.C + static_cast<int64_t>(bz) * p.strideC;
      for (int c = tid; c < BN * (BM / 2); c += NT) {
        const int n = c / (BM / 2), m = (c % (BM / 2)) * 2;
        const int gm = m0 + m, gn = n0 + n;
        const bool ni = gn < N;
        chunk(sC + n * LDC_S + m, Cb, gm + static_cast<int64_t>(gn) * p.ldc, ni && gm < M, ni && gm + 1 < M);
      }
      cp_async_commit();
    }
  }

  for (int kt = 0; kt < ktiles; ++kt) {
    if (kt == 0 && stage_c) cp_async_wait<STAGES - 1>();  // C still on its way
    else cp_async_wait<STAGES - 2>();
    __syncthreads();
    {
      const int nk = kt + STAGES - 1;
      if (nk < ktiles) load_stage(nk % STAGES, kb + nk * BK);
      cp_async_commit();
    }
    const double* sa = sAb + (kt % STAGES) * AE;
    const double* sb = sBb + (kt % STAGES) * BE;
#pragma unroll
    for (int kk = 0; kk < BK / 8; ++kk) {
      double af[MI][4];
      double bf[NJ][2];
#pragma unroll
      for (int i = 0; i < MI; ++i) {
        const int m = wm + i * 16 + 2 * g;
        if (!TA) {
          const double2 v0 = *reinterpret_cast<const double2*>(sa + (kk * 8 + 2 * t) * LDA_N + m);
          const double2 v1 = *reinterpret_cast<const double2*>(sa + (kk * 8 + 2 * t + 1) * LDA_N + m);
          af[i][0] = v0.x;
          af[i][1] = v0.y;
          af[i][2] = v1.x;
          af[i][3] = v1.y;
        } else {
          const double2 v0 = *reinterpret_cast<const double2*>(sa + m * LDA_T + kk * 8 + 2 * t);
          const double2 v1 = *reinterpret_cast<const double2*>(sa + (m + 1) * LDA_T + kk * 8 + 2 * t);
          af[i][0] = v0.x;
          af[i][2] = v0.y;
          af[i][1] = v1.x;
          af[i][3] = v1.y;
        }
      }
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int n = wn + j * 8 + g;
        if (!TB) {
          const double2 v = *reinterpret_cast<const double2*>(sb + n * LDB_N + kk * 8 + 2 * t);
          bf[j][0] = v.x;
          bf[j][1] = v.y;
        } else {
          bf[j][0] = sb[(kk * 8 + 2 * t) * LDB_T + n];
          bf[j][1] = sb[(kk * 8 + 2 * t + 1) * LDB_T + n];
        }
      }
#pragma unroll
      for (int i = 0; i < MI; ++i)
#pragma unroll
        for (int j = 0; j < NJ; ++j) dmma_16x8x8(acc[i][j], af[i], bf[j]);
    }
  }
  cp_async_wait<0>();
  release_dependents();

  // ---- epilogue ----
  if (kp.splitk > 1) {
    // the slices of a tile are one cluster, or a few: every CTA leaves its partial tile in shared memory,
    // and each then sums its share of the columns over the cluster in slice order and writes it
    // (a pass through global scratch costs a second launch, 2.5 us and its gap, so only where one
    // cluster leaves most SMs idle: splitk_reduce_kernel)
    constexpr int LDP = BM + 2;
    static_assert(BN * LDP * 8 <= C::smem(TA, TB), "partial tile fits the pipeline's buffers");
    cg::cluster_group cluster = cg::this_cluster();
    __syncthreads();
    double* P = smem;
#pragma unroll
    for (int i = 0; i < MI; ++i)
#pragma unroll
      for (int j = 0; j < NJ; ++j) {
        const int r = wm + i * 16 + 2 * g, c = wn + j * 8 + 2 * t;
#pragma unroll
        for (int h = 0; h < 2; ++h)
          *reinterpret_cast<double2*>(P + r + (c + h) * LDP) = make_double2(acc[i][j][h], acc[i][j][2 + h]);
      }
    cluster.sync();
    const double al = GROUPS ? 1.0 : p.alpha * (p.alpha_vec ? p.alpha_vec[bz] : 1.0);
    const double be = GROUPS ? 0.0 : p.beta;
    const int64_t ldc = GROUPS ? kp.ldp : p.ldc;
    double* Cb = GROUPS ? kp.P + (static_cast<int64_t>(split / kp.cluster) * p.batch + bz) * kp.ldp * N
                        : p.C + static_cast<int64_t>(bz) * p.strideC;
    const int S = GROUPS ? kp.cluster : kp.splitk, per = (BN + S - 1) / S;
    const int c0 = (GROUPS ? split % S : split) * per, c1 = min(BN, c0 + per);
    for (int e = tid; e < (c1 - c0) * (BM / 2); e += NT) {
      const int r = (e % (BM / 2)) * 2, c = c0 + e / (BM / 2);
      double s0 = 0.0, s1 = 0.0;
#pragma unroll 4
      for (int q = 0; q < S; ++q) {
        const double2 v = *reinterpret_cast<const double2*>(cluster.map_shared_rank(P, q) + r + c * LDP);
        s0 += v.x;
        s1 += v.y;
      }
      const int gr = m0 + r, gc = n0 + c;
      if (gc >= N) continue;
      double* dst = Cb + gr + static_cast<int64_t>(gc) * ldc;
      if (gr < M && (!p.tri || gr >= gc)) dst[0] = be != 0.0 ? fma(be, dst[0], al * s0) : al * s0;
      if (gr + 1 < M && (!p.tri || gr + 1 >= gc)) dst[1] = be != 0.0 ? fma(be, dst[1], al * s1) : al * s1;
    }
    cluster.sync();  // no CTA leaves while others read its partial tile
    return;
  }
  double* C_ = p.C + static_cast<int64_t>(bz) * p.strideC;
  const int64_t ldc = p.ldc;
  const double alpha = p.alpha * (p.alpha_vec ? p.alpha_vec[bz] : 1.0);
  const double beta = p.beta;
  if (stage_c) __syncthreads();
#pragma unroll
  for (int i = 0; i < MI; ++i)
#pragma unroll
    for (int j = 0; j < NJ; ++j) {
      const int r = m0 + wm + i * 16 + 2 * g;
      const int c = n0 + wn + j * 8 + 2 * t;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int cc = c + h;
        if (cc >= N || r >= M) continue;
        double* dst = C_ + r + static_cast<int64_t>(cc) * ldc;
        double v0 = alpha * acc[i][j][h];
        double v1 = alpha * acc[i][j][2 + h];
        const bool ok0 = !p.tri || r >= cc;
        const bool ok1 = (r + 1 < M) && (!p.tri || r + 1 >= cc);
        if (V16 && ok0 && ok1) {
          if (beta != 0.0) {
            const double2 o = *reinterpret_cast<const double2*>(
                stage_c ? sC + wm + i * 16 + 2 * g + (wn + j * 8 + 2 * t + h) * LDC_S : dst);
            v0 += beta * o.x;
            v1 += beta * o.y;
          }
          *reinterpret_cast<double2*>(dst) = make_double2(v0, v1);
        } else {
          const double* o = stage_c ? sC + wm + i * 16 + 2 * g + (wn + j * 8 + 2 * t + h) * LDC_S : dst;
          if (ok0) dst[0] = (beta != 0.0) ? v0 + beta * o[0] : v0;
          if (ok1) dst[1] = (beta != 0.0) ? v1 + beta * o[1] : v1;
        }
      }
    }
}

// C = beta C + alpha times the sum of the groups' partial sums, in their order
__global__ void splitk_reduce_kernel(GemmArgs p, int groups, const double* P, int64_t ldp) {
  dependency_wait();
  release_dependents();
  const int bz = blockIdx.y;
  const double alpha = p.alpha * (p.alpha_vec ? p.alpha_vec[bz] : 1.0);
  const int64_t one = ldp * p.N, group = one * p.batch;
  const double* Pb = P + bz * one;
  double* C = p.C + bz * p.strideC;
  for_entries(p.M, p.N, [&](int i, int j) {
    if (p.tri && i < j) return;
    const double* src = Pb + i + j * ldp;
    double s = 0.0;
#pragma unroll 4
    for (int q = 0; q < groups; ++q) s += src[q * group];
    double* dst = C + i + j * p.ldc;
    *dst = p.beta != 0.0 ? fma(p.beta, *dst, alpha * s) : alpha * s;
  });
}

template <class C, bool TA, bool TB, bool V16, bool GROUPS>
cudaError_t launch_g(const KParams& kp, dim3 grid, cudaStream_t st) {
  static std::atomic<int> attr_set[kMaxDevices];
  const cudaError_t attr = once_per_device(attr_set, [] {
    return cudaFuncSetAttribute(dgemm_kernel<C, TA, TB, V16, GROUPS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                C::smem(TA, TB) + C::SMEM_C);
  });
  if (attr != cudaSuccess) return attr;
  return launch_dependent(dgemm_kernel<C, TA, TB, V16, GROUPS>, grid, dim3(C::NT),
                          C::smem(TA, TB) + (kp.stage_c ? C::SMEM_C : 0), st, dim3(1, kp.cluster, 1), kp);
}

template <class C, bool TA, bool TB, bool V16>
cudaError_t launch_t(const KParams& kp, dim3 grid, cudaStream_t st) {
  return kp.cluster < kp.splitk ? launch_g<C, TA, TB, V16, true>(kp, grid, st)
                                : launch_g<C, TA, TB, V16, false>(kp, grid, st);
}

template <class C, bool V16>
cudaError_t launch_v(const KParams& kp, dim3 grid, cudaStream_t st) {
  const GemmArgs& a = kp.g;
  if (!a.transA && !a.transB) return launch_t<C, false, false, V16>(kp, grid, st);
  if (!a.transA && a.transB) return launch_t<C, false, true, V16>(kp, grid, st);
  if (a.transA && !a.transB) return launch_t<C, true, false, V16>(kp, grid, st);
  return launch_t<C, true, true, V16>(kp, grid, st);
}

template <class C>
cudaError_t launch_c(const KParams& kp, dim3 grid, bool v16, cudaStream_t st) {
  return v16 ? launch_v<C, true>(kp, grid, st) : launch_v<C, false>(kp, grid, st);
}

// tile shape: 0 = 64x64 with four warps (general), 1 = 32x64 (M <= 32), 2 = 64x64 with eight warps
// (K <= 64 or N <= 64, and short-K updates), 4 = 32x32 (too small to fill the GPU)
int pick_cfg(const GemmArgs& a) {
  // Products that leave SMs idle with 64 x 64 tiles (FP64 DMMA runs at 64 FMA a clock and SM, so a
  // tile of K = 64 alone takes 2.1 us): 32 x 32 tiles spread them wider.  Measured 64 x 64 against
  // 32 x 32: 64^3 5.8 / 3.7 us, 1024 x 128 x 128 11.3 / 7.1, 128 x 896 x 1024 (split K) 18.3 / 15.7; past
  // about 1.4e8 multiplications or one tile per SM the larger tiles' reuse wins
  // (1024 x 512 x 512 30 / 44 us, 1024 x 896 x 128 17.3 / 18.5).
  const int64_t t64 = (a.M + 63) / 64, u64 = (a.N + 63) / 64;
  const int64_t tiles64 = (a.tri ? t64 * (t64 + 1) / 2 : t64 * u64) * a.batch;
  const double work = static_cast<double>(a.M) * a.N * a.K * a.batch * (a.tri ? 0.5 : 1.0);
  if (tiles64 < num_sms() && work <= 1.4e8) return 4;
  if (a.tri) return 0;
  if (a.M <= 32) return 1;
  if (a.K <= 64 || a.N <= 64) return 2;
  // C += A B updates with K <= 256 (the 128-column block reflector updates of the QR):
  // eight warps, three CTAs per SM, C staged in shared memory (8192 x 8064 x 128: 25.9 TF/s, 22.5 when C
  // was loaded into the accumulators first, 24.7 with four warps)
  if (a.K <= 256 && !a.transA && a.beta != 0.0) return 2;
  return 0;
}

void tile_dims(int cfg, int* bm, int* bn, int* per_sm) {
  if (cfg == 4) {
    *bm = CfgTiny::BM;
    *bn = CfgTiny::BN;
    *per_sm = CfgTiny::MINB;
  } else if (cfg == 1) {
    *bm = CfgSkinnyM::BM;
    *bn = CfgSkinnyM::BN;
    *per_sm = CfgSkinnyM::MINB;
  } else if (cfg == 2) {
    *bm = CfgSmall::BM;
    *bn = CfgSmall::BN;
    *per_sm = CfgSmall::MINB;
  } else {
    *bm = CfgWide::BM;
    *bn = CfgWide::BN;
    *per_sm = CfgWide::MINB;
  }
}

// Slices of K for the general tiles, 4 CTAs an SM: the time in K tiles of one CTA per SM at the full
// rate is (kt / s + 2) for every CTA of a slot, and a last wave of 1, 2, 3 or 4 CTAs an SM takes as
// long as 1.75, 2.5, 3.2 or 4 of them (28 % of the FP64 tensor rate a CTA alone reaches, 80 % three).
// Powers of two: clusters of 3, 5 or 7 leave SMs of a GPC idle (with 64 x 128 tiles, 128 x 1024 x 3072
// of six ran at 18.3, 18.4 and 24.3 TF/s in 2, 3 and 4 slices).  Measured against one slice:
// 128 x 8064 x 8192 20.1 -> 25.7, 128 x 2048 x 2048 of six 24.6 -> 27.6, 1024^3 19.7 -> 22.5, lower
// triangle of 2048^3 25.0 -> 27.6 TF/s; 2048^3 stays whole (29.7).
int split_general(int64_t ctas, int kt, int sms) {
  static const double last[5] = {0.0, 1.75, 2.5, 3.2, 4.0};
  constexpr int per_sm = CfgWide::MINB;
  static_assert(per_sm == 4, "the last wave's times are for four CTAs an SM");
  int best = 1;
  double best_t = 1e300;
  for (int s = 1; s <= 8 && s <= kt; s *= 2) {
    const int64_t n = ctas * s, wave = static_cast<int64_t>(sms) * per_sm;
    const int64_t rest = n % wave;
    const double t = ((kt + s - 1) / s + 2) * (static_cast<double>(n / wave) * per_sm + last[(rest + sms - 1) / sms]);
    if (t < best_t * (1.0 - 1e-9)) {
      best_t = t;
      best = s;
    }
  }
  return best;
}

// Split K in one cluster only when the tile grid cannot fill the GPU; pick the split (the CTAs of a portable
// cluster, 8 at most) that fills whole waves (sms * resident CTAs per SM) best, with at least 8
// K tiles per split (4 of the 32 x 32 tiles).
int choose_splitk(const GemmArgs& a, int cfg, int sms) {
  if (a.splitk >= 1) return a.splitk;
  int BM, BN, per_sm;
  tile_dims(cfg, &BM, &BN, &per_sm);
  const int tm = (a.M + BM - 1) / BM, tn = (a.N + BN - 1) / BN;
  const int64_t tiles = a.tri ? static_cast<int64_t>(tm) * (tm + 1) / 2 : static_cast<int64_t>(tm) * tn;
  const int64_t ctas = tiles * a.batch;
  const int64_t wave = static_cast<int64_t>(sms) * per_sm;
  const int kt = (a.K + BK - 1) / BK;
  if (cfg == 0) return split_general(ctas, kt, sms);
  if (ctas >= wave) return 1;
  const int smax = std::min(8, kt / (cfg == 4 ? 4 : 8));
  if (smax < 2) return 1;
  int best = 1;
  double best_eff = static_cast<double>(ctas) / wave;  // fraction of one wave used unsplit
  for (int s = 2; s <= smax; ++s) {
    const int64_t c = ctas * s;
    const int64_t waves = (c + wave - 1) / wave;
    const double eff = static_cast<double>(c) / (waves * wave);  // wave fill
    // prefer more parallelism until the first full wave, then fill
    const double score = (c < wave ? static_cast<double>(c) / wave : eff) * (waves <= 3 ? 1.0 : 0.9);
    if (score > best_eff + 1e-9) {
      best_eff = score;
      best = s;
    }
  }
  return best;
}

bool long_k(const GemmArgs& a) { return a.K > 127 * BK && a.splitk < 1 && !a.kfrom_n && !a.kto_m; }

struct Plan {
  int cfg, cluster, groups;  // tile shape, slices of K summed inside a cluster, clusters a tile
};

// A long K over few tiles: one cluster of 8 CTAs a tile leaves most SMs idle, and clusters of 8 do not fill the SMs
// evenly.  From K = 2048 (kt = 128) on and up to two tiles an SM, groups of clusters share a tile, their sums
// going through scratch in global memory: a second launch of 2 to 5 us, so only where it saves more.
// About 512 CTAs, of at least 4 K tiles (8 of the larger tiles); more for a longer K, and not a second wave of a
// few (64 x 64 tiles are resident four to an SM); clusters of 2 from 16 tiles or so on.  32 x 32 tiles serve the
// smallest outputs, 64 x 64 with four warps the rest; 32 x 64 only M <= 32 with N from 4096 on.
// Measured in one cluster (the tiles and slices of choose_splitk) against this, the chain drained between, us:
// 32 x 32 x 4096 20.6 / 10.4, 32 x 512 x 8192 41 / 23, 512 x 64 x 8192 66 / 35, 128 x 512 x 8192 105 / 56,
// 64 x 64 x 65536 242 / 33, 128 x 2048 x 8192 184 / 170, 8192 x 64 x 8192 367 / 316, 1000 x 1000 x 8192 680 / 602,
// lower triangle of 512 x 512 x 8192 144 / 103; at K = 1024 groups save nothing (32 x 32 10.3 / 10.3,
// 128 x 1024 20.6 / 22.7).
Plan plan_gemm(const GemmArgs& a, int sms) {
  Plan now{pick_cfg(a), 1, 1};
  now.cluster = choose_splitk(a, now.cfg, sms);
  if (!long_k(a)) return now;
  const int kt = (a.K + BK - 1) / BK;
  auto tiles = [&](int bm, int bn) {
    const int64_t tm = (a.M + bm - 1) / bm, tn = (a.N + bn - 1) / bn;
    return (a.tri ? tm * (tm + 1) / 2 : tm * tn) * a.batch;
  };
  const int64_t t64 = tiles(64, 64);
  int cfg = now.cfg;
  if (a.M <= 32) cfg = a.N < 4096 ? 4 : 1;
  else if (a.tri) cfg = t64 <= 10 || (t64 <= 36 && kt < 512) ? 4 : 0;
  else if (kt < 512) cfg = t64 <= 16 ? 4 : (t64 >= 48 && cfg == 2 ? 0 : cfg);
  else if (t64 >= 8) cfg = 0;
  int bm, bn, per_sm;
  tile_dims(cfg, &bm, &bn, &per_sm);
  const int64_t n = tiles(bm, bn);
  if (n > sms) {
    // split_general's slices in clusters of 2, eight of them from 200 tiles on (1000 x 1000 x 20000 1461 / 1431 us)
    const bool groups = cfg == 0 && now.cfg == 0 && !a.tri && kt >= 256 && n <= 2 * sms && now.cluster >= 4;
    return groups ? Plan{0, 2, n >= 200 ? 4 : now.cluster / 2} : now;
  }
  const bool wide = n >= 96;
  if (n >= 48) {
    if (cfg == 4) return !wide ? Plan{4, 8, 1} : (a.tri || kt < 512 ? Plan{4, 4, 1} : Plan{4, 2, 4});
    if (kt < (wide ? 256 : 512)) return cfg == 1 ? Plan{1, 4, 1} : (cfg != now.cfg ? Plan{cfg, 8, 1} : now);
    if (wide) return a.tri ? now : Plan{cfg, 2, 4};
    return n > 64 && cfg == 0 ? Plan{0, 4, 8} : Plan{cfg, 2, 8};
  }
  if (n > 16 && kt < (a.tri ? 256 : 512)) return cfg == 4 ? Plan{4, 8, 1} : now;
  if (n > 24 && cfg != 4) return Plan{cfg, 2, n <= 32 ? 16 : 8};
  const int min_kt = cfg == 4 ? 4 : 8;
  const int64_t target = cfg == 4 || kt < 1024 ? 512 : (kt < 4096 ? 1024 : 2048);
  int slices = 1;
  auto more = [&] { return slices < 128 && kt / (2 * slices) >= min_kt; };
  while (n * slices < target && more()) slices *= 2;
  if (cfg != 4 && n * slices > 528 && n * slices <= 640 && more()) slices *= 2;
  return slices <= 16 ? Plan{cfg, 2, slices / 2} : Plan{cfg, 8, slices / 8};
}

size_t scratch_elems(const GemmArgs& a, const Plan& p) {
  return p.groups > 1 ? static_cast<size_t>(p.groups) * a.batch * ((a.M + 1) / 2 * 2) * a.N : 0;
}

}  // namespace

size_t dgemm_scratch(const GemmArgs& a) {
  if (a.M <= 0 || a.N <= 0 || a.batch <= 0 || !long_k(a)) return 0;
  return scratch_elems(a, plan_gemm(a, num_sms()));
}

int num_sms() {
  static std::atomic<int> cache[kMaxDevices];
  return per_device_value(cache, [] {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms > 0 ? sms : 148;
  });
}

cudaError_t dgemm(GemmArgs a, cudaStream_t st, double* scratch) {
  if (a.M <= 0 || a.N <= 0 || a.batch <= 0) return cudaSuccess;
  if (a.tri && a.M != a.N) return cudaErrorInvalidValue;
  // 16-byte cp.async path when every tile chunk is 16-byte aligned, else 8-byte copies
  auto al = [](const void* ptr, int64_t ld) {
    return (reinterpret_cast<uintptr_t>(ptr) % 16 == 0) && (ld % 2 == 0);
  };
  auto al8 = [](const void* ptr) { return reinterpret_cast<uintptr_t>(ptr) % 8 == 0; };
  if (!al8(a.A) || !al8(a.B) || !al8(a.C)) return cudaErrorMisalignedAddress;
  const bool v16 = al(a.A, a.lda) && al(a.B, a.ldb) && al(a.C, a.ldc) &&
                   (a.batch <= 1 || ((a.strideA | a.strideB | a.strideC) & 1) == 0);
  if (rank_update_applies(a)) return rank_update(a, st);
  const int sms = num_sms();
  if (a.K <= 0) {
    // C = beta*C
    return scale_copy(a.M, a.N, a.beta, a.C, a.ldc, a.strideC, a.C, a.ldc, a.strideC, a.batch, 0.0, st);
  }
  KParams kp;
  kp.g = a;
  Plan plan = plan_gemm(a, sms);
  if (plan.groups > 1 && !scratch) plan = Plan{plan.cfg, plan.cluster, 1};
  const int cfg = plan.cfg;
  int BM, BN, per_sm;
  tile_dims(cfg, &BM, &BN, &per_sm);
  kp.tiles_m = (a.M + BM - 1) / BM;
  kp.tiles_n = (a.N + BN - 1) / BN;
  kp.splitk = plan.cluster * plan.groups;
  kp.cluster = plan.cluster;
  kp.P = scratch;
  kp.ldp = (a.M + 1) / 2 * 2;
  kp.stage_c = (kp.splitk <= 1 && a.beta != 0.0 && !a.tri && !a.kto_m && !a.alpha_vec &&
                 (a.alpha == 1.0 || a.alpha == -1.0) && (a.K <= 64 || (cfg == 2 && a.K <= 256)))
                   ? 1
                   : 0;
  const int64_t tiles = a.tri ? static_cast<int64_t>(kp.tiles_m) * (kp.tiles_m + 1) / 2
                              : static_cast<int64_t>(kp.tiles_m) * kp.tiles_n;
  if (tiles > 0x7fffffff || a.batch > 65535) return cudaErrorInvalidValue;
  dim3 grid(static_cast<unsigned>(tiles), kp.splitk, a.batch);
  const cudaError_t e = cfg == 1   ? launch_c<CfgSkinnyM>(kp, grid, v16, st)
                        : cfg == 2 ? launch_c<CfgSmall>(kp, grid, v16, st)
                        : cfg == 4 ? launch_c<CfgTiny>(kp, grid, v16, st)
                                   : launch_c<CfgWide>(kp, grid, v16, st);
  if (e != cudaSuccess || plan.groups <= 1) return e;
  const int blocks = static_cast<int>(std::min<int64_t>((static_cast<int64_t>(a.M) * a.N + 255) / 256, 4 * sms));
  return launch_dependent(splitk_reduce_kernel, dim3(blocks, a.batch), dim3(256), 0, st, dim3(1), a, plan.groups,
                          scratch, kp.ldp);
}

}  // namespace zolo
