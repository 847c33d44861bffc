// Householder panel factorisation for the blocked QR of the stacked matrix
// [X; sqrt(c) I] (mpdgeqrf.f:252-313 / PDGEQR2 semantics, LAPACK dlarfg and
// dlarft conventions) on one thread-block cluster per panel.
//
// The m x w panel (w <= 32) is split by rows over the CL CTAs of a cluster.  A panel is a chain
// of 32 dependent columns, each a reduction over all rows, so latency bounds it: up to 8192 rows
// it stays in registers (qr_panel_reg_kernel, 1.1 us a column at m = 1024 and 2 us at m = 8192;
// the shared-memory kernel below took 4.2 and 4.7 us).
//
// Larger panels run on qr_panel_kernel: each CTA keeps its rows in shared memory when they fit,
// in global memory otherwise.  Inside a CTA the
// work is column-parallel: thread (c, g) owns column c of the rows
// r = g, g+8, g+16, ... of its chunk, so every phase is a short scalar loop
// over independent rows and the row sums are 3 warp shuffles.  Column k costs
// three CTA barriers and ONE cluster barrier:
//   * gather: every CTA sums all CTAs' partials (||x_below||^2 and
//     x_below . a_c) in the same fixed order, so all CTAs derive bit-identical
//     beta / tau / v^T A; the partials were pushed into every CTA's receive
//     slots (distributed shared memory stores) before the cluster barrier, so
//     the sum reads local shared memory and the remote latency overlaps the
//     barrier;
//   * update: columns c > k apply reflector k;
//   * scale + dots: column k is scaled into v_k and the partials of column
//     k+1 are formed and published (double-buffered by column parity).
// The compact-WY factor T (dlarft) is formed once, after the last column, from
// the cluster-wide V^T V.
#include "common.cuh"
#include "kernels.h"

#include <cooperative_groups.h>

#include <algorithm>

namespace cg = cooperative_groups;

namespace zolo {

namespace {

constexpr int QW = 32;   // max panel width
constexpr int QT = 256;  // threads per CTA: 32 columns x 8 row groups
constexpr int NG = 8;    // row groups
constexpr int UB = 8;    // rows per load batch
constexpr int UC = 16;   // columns per load batch in the update
constexpr int SLOT = 1 + QW;  // s0, d[QW]
constexpr int QCL = 16;       // largest cluster
constexpr size_t SMEM_CHUNK_CAP = 190 * 1024;

struct PanelArgs {
  int m, w, rows_per, rp_ld;  // rp_ld: leading dimension of the shared-memory chunk
  double* A;
  int64_t lda, strideA;
  int split;    // logical rows >= split live `gap` rows further down in A
  int64_t gap;
  double* tau;
  int64_t strideTau;
  double* T;
  int64_t strideT;
  double* V;
  int64_t ldv, strideV;
  int* status;           // written when a wait between the CTAs timed out
  long long wait_limit;  // clock cycles of such a wait
};

ZDEV double group_sum8(double v) {
  v += __shfl_xor_sync(0xffffffffu, v, 1);
  v += __shfl_xor_sync(0xffffffffu, v, 2);
  v += __shfl_xor_sync(0xffffffffu, v, 4);
  return v;
}

struct PanelShared {
  double recv[2][QCL][SLOT];  // partials of every CTA (by rank), double-buffered by column parity
  double rowkr[2][QW];        // the pivot row of the next column, from the CTA holding it
  double sum[SLOT];
  double rowk[QW];
  double colk[QW];
  double tauv[QW];
  double G[QW * QW];   // this CTA's partial V^T V (upper triangle)
  double Gs[QW * QW];  // rank 0: cluster sum of G
  double T[QW * QW];
};

template <bool SMEM>
__global__ void __launch_bounds__(QT) qr_panel_kernel(PanelArgs p) {
  cg::cluster_group cluster = cg::this_cluster();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  PanelShared& S = *reinterpret_cast<PanelShared*>(smem_raw);
  double* chunk = reinterpret_cast<double*>(smem_raw + ((sizeof(PanelShared) + 15) / 16) * 16);

  const int rank = static_cast<int>(cluster.block_rank());
  const int CL = static_cast<int>(cluster.num_blocks());
  const int b = blockIdx.y;
  const int m = p.m, w = p.w;
  double* A = p.A + b * p.strideA;
  double* V = p.V + b * p.strideV;
  const int64_t lda = p.lda, ldv = p.ldv;
  const int r0 = rank * p.rows_per;
  const int r1 = min(m, r0 + p.rows_per);
  const int nloc = max(r1 - r0, 0);
  const int tid = threadIdx.x, lane = tid & 31;
  const int col = (tid >> 5) * 4 + (lane >> 3);  // column owned by this thread
  const int grp = lane & 7;                      // row group: local rows grp, grp+8, ...
  const int rp = p.rp_ld;

  // physical row of A holding logical row r
  auto prow = [&](int r) -> int64_t { return r + (r >= p.split ? p.gap : 0); };
  auto at = [&](int rl, int c) -> double& {
    if (SMEM) return chunk[c * rp + rl];
    return A[prow(r0 + rl) + c * lda];
  };
  // first local row >= global row `from` that belongs to this thread's group
  auto first_row = [&](int from) {
    int rl = max(from - r0, 0);
    rl += (grp - rl % NG + NG) % NG;
    return rl;
  };
  // sum over this thread's rows (from rl0) of a(r, x) * a(r, col): batches of UB rows whose
  // loads are all issued first, four independent partial sums
  auto dot_rows = [&](int rl0, int x) {
    double s4[4] = {0.0, 0.0, 0.0, 0.0};
    for (int rl = rl0; rl < nloc; rl += NG * UB) {
      double xa[UB], xb[UB];
#pragma unroll
      for (int u = 0; u < UB; ++u) {
        const int r = rl + u * NG;
        xa[u] = (r < nloc) ? at(r, x) : 0.0;
        xb[u] = (r < nloc) ? at(r, col) : 0.0;
      }
#pragma unroll
      for (int u = 0; u < UB; ++u) s4[u & 3] += xa[u] * xb[u];
    }
    return (s4[0] + s4[1]) + (s4[2] + s4[3]);
  };

  if (SMEM) {
    const int tot = w * nloc;
    for (int e = tid; e < tot; e += QT) {
      const int c = e / nloc, rl = e - c * nloc;
      chunk[c * rp + rl] = A[prow(r0 + rl) + c * lda];
    }
  }
  __syncthreads();

  // partials into slot `slot` of receive buffer `bf` of every CTA of the cluster, the pivot
  // row entry c likewise (stores to distributed shared memory, visible after the barrier)
  auto publish = [&](int bf, int slot, double v) {
    for (int q = 0; q < CL; ++q) *cluster.map_shared_rank(&S.recv[bf][rank][slot], q) = v;
  };
  auto publish_pivot = [&](int bf, int c, double v) {
    for (int q = 0; q < CL; ++q) *cluster.map_shared_rank(&S.rowkr[bf][c], q) = v;
  };

  // ---- partials of column 0 ----
  {
    double acc = 0.0, pv = 0.0;
    bool has_pv = false;
    if (col < w) {
      acc = dot_rows(first_row(1), 0);  // col 0: ||x_below||^2
      if (r0 == 0 && grp == 0 && nloc > 0) {  // pivot row 0
        pv = at(0, col);
        has_pv = true;
      }
    }
    acc = group_sum8(acc);
    if (grp == 0 && col < w) publish(0, col == 0 ? 0 : 1 + col, acc);
    if (has_pv) publish_pivot(0, col, pv);
  }
  cluster.sync();

  for (int k = 0; k < w; ++k) {
    const int buf = k & 1;
    // ---- gather: thread i < SLOT sums entry i over all CTAs in rank order (the same order
    // everywhere) from this CTA's receive slots ----
    if (tid < SLOT) {
      double s = 0.0;
      for (int q = 0; q < CL; ++q) s += S.recv[buf][q][tid];
      S.sum[tid] = s;
    } else if (tid < SLOT + w) {
      const int c = tid - SLOT;
      S.rowk[c] = S.rowkr[buf][c];
    }
    __syncthreads();

    // ---- reflector k (dlarfg), computed redundantly and identically by every thread ----
    const double s0 = S.sum[0];
    const double alpha = S.rowk[k];
    double beta, tau, scal;
    if (s0 == 0.0) {
      tau = 0.0;
      beta = alpha;
      scal = 0.0;
    } else {
      beta = -copysign(sqrt(alpha * alpha + s0), alpha);
      tau = (beta - alpha) / beta;
      scal = 1.0 / (alpha - beta);
    }
    if (tid < w) S.colk[tid] = (tid > k) ? S.rowk[tid] + scal * S.sum[1 + tid] : 0.0;  // v^T a_c
    if (tid == 0) {
      S.tauv[k] = tau;
      if (rank == 0) p.tau[b * p.strideTau + k] = tau;
    }
    __syncthreads();

    // ---- update: a(r,c) -= tau * v_r * (v^T a_c) for c > k, rows r >= k ----
    // each thread owns whole rows and loads a batch of UC columns before storing any
    // (a store may alias the next loads of the same array, so batching is explicit)
    for (int rl = max(k - r0, 0) + tid; rl < nloc; rl += QT) {
      const double tv = tau * ((r0 + rl == k) ? 1.0 : at(rl, k) * scal);
      for (int c0 = k + 1; c0 < w; c0 += UC) {
        double xc[UC];
#pragma unroll
        for (int u = 0; u < UC; ++u)
          if (c0 + u < w) xc[u] = at(rl, c0 + u);
#pragma unroll
        for (int u = 0; u < UC; ++u)
          if (c0 + u < w) at(rl, c0 + u) = xc[u] - tv * S.colk[c0 + u];
      }
    }
    __syncthreads();

    // ---- scale column k into v_k (all threads); partials of column k+1 (column threads) ----
    const int nk = k + 1;
    for (int base = tid; base < nloc; base += QT * UB) {
      double x[UB];
#pragma unroll
      for (int u = 0; u < UB; ++u) {
        const int rl = base + u * QT;
        if (rl < nloc && r0 + rl > k) x[u] = at(rl, k);
      }
#pragma unroll
      for (int u = 0; u < UB; ++u) {
        const int rl = base + u * QT;
        if (rl >= nloc) continue;
        const int r = r0 + rl;
        double v;
        if (r < k) {
          v = 0.0;
        } else if (r == k) {
          at(rl, k) = beta;
          v = 1.0;
        } else {
          v = x[u] * scal;
          at(rl, k) = v;
        }
        V[r + k * ldv] = v;
      }
    }
    double acc = 0.0, pv = 0.0;
    bool has_pv = false;
    if (nk < w && col >= nk && col < w) {
      acc = dot_rows(first_row(nk + 1), nk);
      const int lr = nk - r0;  // pivot row of column k+1, if this CTA holds it
      if (lr >= 0 && lr < nloc && grp == lr % NG) {
        pv = at(lr, col);
        has_pv = true;
      }
    }
    acc = group_sum8(acc);
    // the other buffer: no CTA reads it before every CTA has passed this column's barrier
    if (nk < w && grp == 0 && col >= nk && col < w) publish(buf ^ 1, col == nk ? 0 : 1 + col, acc);
    if (has_pv) publish_pivot(buf ^ 1, col, pv);
    cluster.sync();
  }

  // ---- V^T V of this CTA's rows on the FP64 tensor path: warp q takes rows q, q+8k8 ...
  // V(r,i) = a(r,i) below the diagonal, 1 on it, 0 above; the 32 x 32 partials of the 8
  // warps are summed through shared memory into G ----
  {
    const int warp = tid >> 5;
    const int gq = lane >> 2, tq = lane & 3;
    auto vval = [&](int rl, int i) -> double {
      const int r = r0 + rl;
      if (rl >= nloc || i >= w || r < i) return 0.0;
      return (r == i) ? 1.0 : at(rl, i);
    };
    double accg[2][4][4];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
      for (int bb = 0; bb < 4; ++bb)
#pragma unroll
        for (int r = 0; r < 4; ++r) accg[a][bb][r] = 0.0;
    // k8 steps of rows: step s covers local rows 8s .. 8s+7; warp q does steps q, q+8, ...
    for (int st = warp; st * 8 < nloc; st += QT / 32) {
      const int rb = st * 8;
      double af[2][4], bf[4][2];
#pragma unroll
      for (int a = 0; a < 2; ++a) {  // A = V^T: rows i, k = local row
        const int i0 = a * 16 + gq;
        af[a][0] = vval(rb + tq, i0);
        af[a][1] = vval(rb + tq, i0 + 8);
        af[a][2] = vval(rb + tq + 4, i0);
        af[a][3] = vval(rb + tq + 4, i0 + 8);
      }
#pragma unroll
      for (int bb = 0; bb < 4; ++bb) {  // B = V: k = local row, n = j
        const int j0 = bb * 8 + gq;
        bf[bb][0] = vval(rb + tq, j0);
        bf[bb][1] = vval(rb + tq + 4, j0);
      }
#pragma unroll
      for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int bb = 0; bb < 4; ++bb) dmma_16x8x8(accg[a][bb], af[a], bf[bb]);
    }
    for (int e = tid; e < QW * QW; e += QT) S.G[e] = 0.0;
    __syncthreads();
    // warps add their partials one after another: a fixed summation order, so the
    // panel (and everything downstream) is bitwise reproducible run to run
    for (int wq = 0; wq < QT / 32; ++wq) {
      if (warp == wq) {
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
          for (int bb = 0; bb < 4; ++bb) {
            const int i = a * 16 + gq, j = bb * 8 + 2 * tq;
            S.G[i + j * QW] += accg[a][bb][0];
            S.G[i + (j + 1) * QW] += accg[a][bb][1];
            S.G[i + 8 + j * QW] += accg[a][bb][2];
            S.G[i + 8 + (j + 1) * QW] += accg[a][bb][3];
          }
      }
      __syncthreads();
    }
  }
  if (SMEM) {
    const int tot = w * nloc;
    for (int e = tid; e < tot; e += QT) {
      const int c = e / nloc, rl = e - c * nloc;
      A[prow(r0 + rl) + c * lda] = chunk[c * rp + rl];
    }
  }
  cluster.sync();
  if (rank == 0) {
    // T(k,k) = tau_k, T(0:k,k) = -tau_k T(0:k,0:k) V(:,0:k)^T v_k  (dlarft, forward, columnwise)
    for (int e = tid; e < QW * QW; e += QT) {
      double gq[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) gq[q] = (q < CL) ? cluster.map_shared_rank(S.G, q)[e] : 0.0;
      double g = 0.0;
#pragma unroll
      for (int q = 0; q < 16; ++q) g += gq[q];
      S.Gs[e] = g;
      S.T[e] = 0.0;
    }
    __syncthreads();
    for (int k = 0; k < w; ++k) {
      const double tk = S.tauv[k];
      if (tid < k) {
        double tv = 0.0;
        for (int j = tid; j < k; ++j) tv += S.T[tid + j * QW] * S.Gs[j + k * QW];
        S.T[tid + k * QW] = -tk * tv;
      } else if (tid == k) {
        S.T[k + k * QW] = tk;
      }
      __syncthreads();
    }
    double* T = p.T + b * p.strideT;
    for (int e = tid; e < QW * QW; e += QT) T[e] = S.T[e];
  }
  cluster.sync();  // no CTA leaves while others may still read its shared memory
}

// ---- register-resident panel ----
// The panel of a cluster's CTA lives in registers: warp q holds 8 RN consecutive local rows;
// thread (g = lane / 4, t = lane % 4) the rows g, g + 8, ... of them and the columns
// 2t + (j & 1) + 8 (j >> 1), j = 0 .. 7.  Column k costs one pass over the registers, two CTA
// barriers and one exchange between the CTAs:
//   * x, the entries of column k below the pivot, comes from the owning lane of each quad by a
//     shuffle; p_c = sum_r x_r a_rc for ALL 32 columns is reduced over the warp by seven
//     shuffles (8 values over 8 lanes, halved at every stage) and over the warps by warp 0, which
//     sends the CTA's sums into every CTA's receive slots (st.async on the receiver's mbarrier:
//     no fence or cluster barrier on the path);
//   * warp 0 of every CTA waits for the slots and sums them in rank order (bit-identical
//     everywhere): p_k = ||x||^2 gives beta, tau and scal (dlarfg), p_c for c > k the update's
//     v^T a_c = a_kc + scal p_c, and p_c for c < k the dlarft product v_c^T v_k = v_kc + scal p_c
//     (sent to the last CTA only, whose warp 1 forms T column by column while warp 0 waits);
//   * update a_rc += x_r (v^T a_c) / beta (tau scal = -1/beta; the pivot row is x = alpha - beta).
// Measured per column at m = 1024 (8 CTAs of 4 warps): dots and shuffles 330 clocks, the exchange
// 570, norm and reciprocals 330, update 280.  With cluster barriers instead of the mbarrier
// sends the exchange took 1050, and a barrier with release semantics alone is 420.
template <int NW>
struct RegShared {
  double recv[2][QCL][QW];  // sums of every CTA (by rank), double-buffered by column parity
  double prow_in[2][QW];    // pivot row k, from the CTA holding it
  double part[NW][QW];      // this CTA's sums by warp
  double prow[QW];          // pivot row k if this CTA holds it
  double w[QW];             // (v^T a_c) / beta for c > k, 0 otherwise
  double sc[4];             // scal, beta, alpha - beta
  double Z[2][QW];          // Z[k & 1][c] = v_c^T v_k, c < k
  double tau[QW];
  double T[QW][QW];         // T[j][i] = T(i, j)
  unsigned long long bar[2];
  uint32_t peer[QCL];  // shared-window addresses of this struct in the other CTAs, own CTA first
  int abort;  // 1 + the column at which this CTA's wait ran out, 0 = none
};

ZDEV uint32_t cluster_addr(const void* p, int rank) {
  uint32_t l = static_cast<uint32_t>(__cvta_generic_to_shared(p)), r;
  asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(l), "r"(rank));
  return r;
}
// 8 bytes into another CTA's shared memory, counted by its mbarrier
ZDEV void cluster_send(uint32_t addr, double v, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f64 [%0], %1, [%2];" ::"r"(addr), "d"(v),
               "r"(bar)
               : "memory");
}
ZDEV void cluster_sync_all() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
constexpr long long kPanelTimeoutCycles = 2000000000LL;  // about a second
// Wait of one warp on its CTA's mbarrier phase for at most `limit` clock cycles (below zero: it has run
// out whatever comes); a last look follows the limit, for a GPU that was switched away meanwhile.
ZDEV bool panel_wait(uint32_t bar, uint32_t parity, long long limit) {
  const long long t0 = clock64();
  bool late = false;
  while (true) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok && limit >= 0) return true;
    if (late) return false;
    late = clock64() - t0 > limit;
  }
}

// This lane's value into the same place of every CTA's struct (only the last CTA's unless `all`),
// counted by that CTA's barrier.  Destinations are staggered by rank, so that the CTAs do not send
// to one CTA at the same time, and their addresses come from a table: mapa per destination
// made the 16 sends 1900 clocks, the table 400.
template <class Sh>
ZDEV void panel_send(Sh& S, const void* slot, const void* bar, double v, bool all, int rank, int CL) {
  const uint32_t so = static_cast<uint32_t>(static_cast<const char*>(slot) - reinterpret_cast<const char*>(&S));
  const uint32_t bo = static_cast<uint32_t>(static_cast<const char*>(bar) - reinterpret_cast<const char*>(&S));
  const int ql = CL - 1 - rank;  // table index of the last CTA
#pragma unroll
  for (int q4 = 0; q4 < QCL; q4 += 4) {
    if (q4 < CL) {
      const uint4 b = *reinterpret_cast<const uint4*>(&S.peer[q4]);
      const uint32_t base[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
      for (int u = 0; u < 4; ++u)
        if (q4 + u < CL && (all || q4 + u == ql)) cluster_send(base[u] + so, v, base[u] + bo);
    }
  }
}

// This CTA's sums of column k: columns c >= k to every CTA, c < k to the last one only (the pivot row
// goes by itself), and what column k will bring to this CTA armed on its barrier; one warp.
template <class Sh>
ZDEV void panel_send_sums(Sh& S, uint32_t bar, int k, int buf, double sum, int rank, int CL) {
  const int lane = threadIdx.x & 31;
  if (lane == 0) {
    const int bytes = (rank == CL - 1 ? QW : QW - k) * 8 * CL + QW * 8;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
  }
  panel_send(S, &S.recv[buf][rank][lane], &S.bar[buf], sum, lane >= k, rank, CL);
}

// Column k of T by one warp (dlarft, forward, columnwise): T(k,k) = tau_k,
// T(i,k) = -tau_k sum_{i <= j < k} T(i,j) v_j^T v_k; lane i forms row i.
ZDEV void panel_t_column(double (*T)[QW], const double* z, double tau, int k) {
  const int lane = threadIdx.x & 31;
  double s[4] = {0.0, 0.0, 0.0, 0.0};
  int j = 0;
  for (; j + 4 <= k; j += 4) {
#pragma unroll
    for (int u = 0; u < 4; ++u) s[u] = fma(T[j + u][lane], z[j + u], s[u]);
  }
  for (; j < k; ++j) s[0] = fma(T[j][lane], z[j], s[0]);
  const double v = -tau * ((s[0] + s[1]) + (s[2] + s[3]));
  T[k][lane] = lane == k ? tau : (lane < k ? v : 0.0);
}

// Factors the panel held in a[][] (local rows lr(i) = 8 RN warp + g + 8 i, global row r0 + lr; rows
// at or past nloc hold zeros).  On return (all warps past a CTA barrier) S.tau is complete in
// every CTA and S.T in the last one.  False after a timed-out wait.
template <int NW, int RN>
ZDEV bool panel_factor(double (&a)[RN][8], RegShared<NW>& S, int w, int r0, int nloc, int rank, int CL,
                       long long wait_limit) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int rbase = r0 + warp * 8 * RN + g;  // global row of a[0]
  // the column whose warp sum ends in this lane after the halving stages
  const int jr = ((lane & 16) ? 4 : 0) + ((lane & 8) ? 2 : 0) + ((lane & 4) ? 1 : 0);
  const int cr = 2 * t + (jr & 1) + 8 * (jr >> 1);
  const bool h4 = lane & 16, h3 = lane & 8, h2 = lane & 4;
  const bool last = rank == CL - 1;
  const uint32_t bar0 = static_cast<uint32_t>(__cvta_generic_to_shared(&S.bar[0]));
#pragma unroll
  for (int grp = 0; grp < 4; ++grp) {
#pragma unroll 1
    for (int tt = 0; tt < 4; ++tt) {
#pragma unroll
      for (int par = 0; par < 2; ++par) {
        const int k = 8 * grp + 2 * tt + par;
        if (k >= w) goto done;
        const int jk = 2 * grp + par;
        constexpr int kParity[2] = {0, 1};
        const int buf = kParity[par];
        double x[RN];
#pragma unroll
        for (int i = 0; i < RN; ++i) {
          const double v = __shfl_sync(0xffffffffu, a[i][jk], (lane & ~3) | tt);
          x[i] = (rbase + 8 * i > k) ? v : 0.0;
        }
        const int kl = k - r0;
        const bool owner = kl >= 0 && kl < nloc;
        if (owner && kl / (8 * RN) == warp) {
#pragma unroll
          for (int i = 0; i < RN; ++i)
            if (rbase + 8 * i == k) {
#pragma unroll
              for (int j = 0; j < 8; j += 2)
                *reinterpret_cast<double2*>(&S.prow[2 * t + 4 * j]) = make_double2(a[i][j], a[i][j + 1]);
            }
        }
        double p[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          p[j] = x[0] * a[0][j];
#pragma unroll
          for (int i = 1; i < RN; ++i) p[j] = fma(x[i], a[i][j], p[j]);
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const double keep = h4 ? p[j + 4] : p[j], send = h4 ? p[j] : p[j + 4];
          p[j] = keep + __shfl_xor_sync(0xffffffffu, send, 16);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          const double keep = h3 ? p[j + 2] : p[j], send = h3 ? p[j] : p[j + 2];
          p[j] = keep + __shfl_xor_sync(0xffffffffu, send, 8);
        }
        {
          const double keep = h2 ? p[1] : p[0], send = h2 ? p[0] : p[1];
          S.part[warp][cr] = keep + __shfl_xor_sync(0xffffffffu, send, 4);
        }
        __syncthreads();
        if (warp == 0) {
          double s4[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
          for (int q = 0; q < NW; ++q) s4[q & 3] += S.part[q][lane];
          double sum = (s4[0] + s4[1]) + (s4[2] + s4[3]), pr;
          if (CL > 1) {
            const uint32_t bar = bar0 + 8 * buf;
            panel_send_sums(S, bar, k, buf, sum, rank, CL);
            if (!panel_wait(bar, (k >> 1) & 1, wait_limit)) S.abort = k + 1;
#pragma unroll
            for (int q = 0; q < 4; ++q) s4[q] = 0.0;
#pragma unroll
            for (int q = 0; q < QCL; ++q)
              if (q < CL) s4[q & 3] += S.recv[buf][q][lane];
            sum = (s4[0] + s4[1]) + (s4[2] + s4[3]);
            pr = S.prow_in[buf][lane];
          } else {
            pr = S.prow[lane];
          }
          const double s0 = __shfl_sync(0xffffffffu, sum, k);
          const double alpha = __shfl_sync(0xffffffffu, pr, k);
          double beta = alpha, tau = 0.0, rb = 0.0, rz = 0.0, half = 1.0;
          if (s0 != 0.0) {
            // norm and its reciprocal from one rsqrt (norm corrected by a Newton step)
            const double n2 = fma(alpha, alpha, s0), r = rsqrt(n2);
            double nrm = n2 * r;
            nrm = fma(0.5 * r, fma(-nrm, nrm, n2), nrm);
            beta = -copysign(nrm, alpha);
            rb = -copysign(r, alpha);
            // 1/(alpha - beta), its magnitude |alpha| + norm >= norm, as rsqrt of its square: a division's
            // chain is 150 clocks longer.  Of half of it where the square of up to twice the norm may
            // pass the largest number (n2 >= 2^1021); a branch to a division there cost 36 clocks.
            half = __double2hiint(n2) >= 0x7fc00000 ? 0.5 : 1.0;
            const double z = fma(half, nrm, half * fabs(alpha));
            rz = copysign(rsqrt(z * z), alpha);
            tau = (beta - alpha) * rb;
          }
          const double vta = fma(rz, half * sum, pr);
          S.w[lane] = lane > k ? vta * rb : 0.0;
          S.Z[buf][lane] = vta;
          if (lane == 0) {
            S.sc[0] = half * rz;
            S.sc[1] = beta;
            S.sc[2] = alpha - beta;
            S.tau[k] = tau;
          }
        } else if (warp == 1) {
          if (CL > 1 && owner) {
            const double pr = S.prow[lane];
            panel_send(S, &S.prow_in[buf][lane], &S.bar[buf], pr, true, rank, CL);
          }
          // the previous column of T, while warp 0 waits
          if (last && k > 0) panel_t_column(S.T, S.Z[buf ^ 1], S.tau[k - 1], k - 1);
        }
        __syncthreads();
        if (CL > 1 && S.abort) return false;
        const double scal = S.sc[0], beta = S.sc[1], xp = S.sc[2];
        double xu[RN];
#pragma unroll
        for (int i = 0; i < RN; ++i) xu[i] = (rbase + 8 * i == k) ? xp : x[i];
#pragma unroll
        for (int j = 2 * grp; j < 8; j += 2) {
          const double2 wj = *reinterpret_cast<const double2*>(&S.w[2 * t + 4 * j]);
#pragma unroll
          for (int i = 0; i < RN; ++i) {
            a[i][j] = fma(xu[i], wj.x, a[i][j]);
            a[i][j + 1] = fma(xu[i], wj.y, a[i][j + 1]);
          }
        }
        if (t == tt) {
#pragma unroll
          for (int i = 0; i < RN; ++i) {
            if (rbase + 8 * i > k) a[i][jk] = x[i] * scal;
            else if (rbase + 8 * i == k) a[i][jk] = beta;
          }
        }
      }
    }
  }
done:
  if (last && warp == 1) panel_t_column(S.T, S.Z[(w - 1) & 1], S.tau[w - 1], w - 1);
  return true;
}

// After a wait of this CTA ran out at column k = S.abort - 1, before it may leave (all threads): what the
// others sent to it is on its way (st.async is not ordered by the cluster barrier) and must not arrive
// in shared memory that is no longer its own.  A CTA sends column k + 1 only after all of column k
// has reached it, so the CTAs that give up stand at one column or at two neighbouring ones:
// those behind send the next column too, and every phase then completes.  A CTA that gives up before the
// last column keeps all others from finishing, so all of them come here; after the last column
// others may have left, but then nothing is missing and nothing of theirs is read.  False when the phases
// did not complete in time either.
template <int NW>
ZDEV bool panel_drain(RegShared<NW>& S, int w, int r0, int nloc, int rank, int CL) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int k = S.abort - 1;
  int top = k;
  __syncwarp();
  cluster_sync_all();  // every CTA that gave up has written its column
  if (k < w - 1) {
    cg::cluster_group cluster = cg::this_cluster();
    for (int q = 0; q < CL; ++q) top = max(top, *cluster.map_shared_rank(&S.abort, q) - 1);
  }
  bool ok = true;
  if (top > k && warp == 1 && top >= r0 && top < r0 + nloc)
    panel_send(S, &S.prow_in[top & 1][lane], &S.bar[top & 1], 0.0, true, rank, CL);
  if (warp == 0) {
    const uint32_t bar0 = static_cast<uint32_t>(__cvta_generic_to_shared(&S.bar[0]));
    if (top > k) panel_send_sums(S, bar0 + 8 * (top & 1), top, top & 1, 0.0, rank, CL);
    for (int c = max(top - 1, 0); c <= top; ++c)
      ok = panel_wait(bar0 + 8 * (c & 1), (c >> 1) & 1, kPanelTimeoutCycles) && ok;
  }
  __syncwarp();
  cluster_sync_all();  // no CTA leaves while another reads its column
  return ok;
}

template <int NW, int RN>
__global__ void __launch_bounds__(NW * 32, 1) qr_panel_reg_kernel(PanelArgs p) {
  __shared__ __align__(16) RegShared<NW> S;
  cg::cluster_group cluster = cg::this_cluster();
  const int rank = static_cast<int>(cluster.block_rank());
  const int CL = static_cast<int>(cluster.num_blocks());
  const int b = blockIdx.y, m = p.m, w = p.w;
  const int r0 = rank * p.rows_per;
  const int nloc = max(min(m, r0 + p.rows_per) - r0, 0);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  const int l0 = warp * 8 * RN + g;
  const int64_t lda = p.lda;
  // element offsets of this thread's rows (past the row gap) and first column
  double* A = p.A + b * p.strideA + r0 + l0 + 2 * t * lda;
  int64_t ro[RN];
#pragma unroll
  for (int i = 0; i < RN; ++i) ro[i] = 8 * i + (r0 + l0 + 8 * i >= p.split ? p.gap : 0);
  if (CL > 1) {
    if (threadIdx.x == 0) {
      S.abort = 0;
      for (int q = 0; q < CL; ++q) S.peer[q] = cluster_addr(&S, (rank + q) & (CL - 1));
      for (int q = 0; q < 2; ++q)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(
                         static_cast<uint32_t>(__cvta_generic_to_shared(&S.bar[q])))
                     : "memory");
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    // every CTA of the cluster runs, its barriers ready, before the first send to it
    cluster_sync_all();
  }
  dependency_wait();
  double a[RN][8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const bool in = 2 * t + (j & 1) + 8 * (j >> 1) < w;
    const double* col = A + ((j & 1) + 8 * (j >> 1)) * lda;
#pragma unroll
    for (int i = 0; i < RN; ++i) a[i][j] = (in && l0 + 8 * i < nloc) ? col[ro[i]] : 0.0;
  }
  if (!panel_factor<NW, RN>(a, S, w, r0, nloc, rank, CL, p.wait_limit)) {
    const bool drained = panel_drain(S, w, r0, nloc, rank, CL);
    if (threadIdx.x == 0 && p.status) {
      *static_cast<volatile int*>(p.status) = drained ? 911 : 912;
      __threadfence_system();
    }
    return;
  }
  release_dependents();
  double* V = p.V + b * p.strideV + r0 + l0 + 2 * t * p.ldv;
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int c = 2 * t + (j & 1) + 8 * (j >> 1);
    if (c >= w) continue;
    double* col = A + ((j & 1) + 8 * (j >> 1)) * lda;
    double* vcol = V + ((j & 1) + 8 * (j >> 1)) * p.ldv;
#pragma unroll
    for (int i = 0; i < RN; ++i) {
      if (l0 + 8 * i >= nloc) continue;
      const int r = r0 + l0 + 8 * i;
      col[ro[i]] = a[i][j];
      if (p.V) vcol[8 * i] = r > c ? a[i][j] : (r == c ? 1.0 : 0.0);
    }
  }
  if (rank == CL - 1 && warp == 1) {
    __syncwarp();
    double* T = p.T + b * p.strideT;
#pragma unroll 4
    for (int j = 0; j < QW; ++j) T[lane + j * QW] = j < w ? S.T[j][lane] : 0.0;
    if (lane < w) p.tau[b * p.strideTau + lane] = S.tau[lane];
  }
}

__global__ void extract_v_kernel(int m, int w, const double* A, int64_t lda, int64_t strideA,
                                 double* V, int64_t ldv, int64_t strideV, int split, int64_t gap) {
  dependency_wait();
  release_dependents();
  const double* Ab = A + blockIdx.y * strideA;
  double* Vb = V + blockIdx.y * strideV;
  for_entries(m, w, [&](int i, int j) {
    double v = (i > j) ? Ab[i + (i >= split ? gap : 0) + j * lda] : (i == j ? 1.0 : 0.0);
    Vb[i + j * ldv] = v;
  });
}

// T of up to four panels' block reflector from their T factors and the lower triangle of V^T V:
// T12 = -T1 (V1^T V2) T2 for pairs of 32 columns, then of 64, in one CTA's shared memory (both
// products on the FP64 tensor path).  One array holds T in its upper triangle and V^T V strictly below the
// panels' diagonal blocks.  blockIdx.x: the 128-column block of TB; the CTA writes its columns, zero
// outside its own rows.  Bound by latency: 9 us (25 with the loads in eight dependent rounds), where the
// set-up and six small products of the panel-by-panel recursion were a chain of 30 us.
constexpr int BTW = 128, BTT = 512;
constexpr int BTL = BTW + 4, BTP = 64 + 4;  // = 4 mod 16: conflict-free fragment loads
template <bool TB, int LDB>
ZDEV void bt_mma(double (&c)[4], const double* a, int lda, const double* b, int K) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
#pragma unroll 4
  for (int k = 0; k < K; k += 8) {
    double af[4], bf[2];
    af[0] = a[g + (k + t) * lda];
    af[1] = a[g + 8 + (k + t) * lda];
    af[2] = a[g + (k + t + 4) * lda];
    af[3] = a[g + 8 + (k + t + 4) * lda];
    bf[0] = TB ? b[g + (k + t) * LDB] : b[k + t + g * LDB];
    bf[1] = TB ? b[g + (k + t + 4) * LDB] : b[k + t + 4 + g * LDB];
    dmma_16x8x8(c, af, bf);
  }
}
ZDEV void bt_store(double* s, int ld, const double (&c)[4], double alpha) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
  s[g + (2 * t) * ld] = alpha * c[0];
  s[g + (2 * t + 1) * ld] = alpha * c[1];
  s[g + 8 + (2 * t) * ld] = alpha * c[2];
  s[g + 8 + (2 * t + 1) * ld] = alpha * c[3];
}

__global__ void __launch_bounds__(BTT) block_t_kernel(int jb, const double* T, int64_t strideT, const double* G,
                                                      int64_t ldg, int64_t strideG, double* TB, int64_t ldtb,
                                                      int64_t strideTB) {
  extern __shared__ __align__(16) double bt_sm[];
  double* S = bt_sm;
  double* P = bt_sm + BTW * BTL;
  const int tid = threadIdx.x, warp = tid >> 5;
  const int c0 = blockIdx.x * BTW, w = min(BTW, jb - c0);
  const double* Tb = T + blockIdx.y * strideT + static_cast<int64_t>(c0 / QW) * QW * QW;
  const double* Gb = G + blockIdx.y * strideG + c0 + c0 * ldg;
  double* Bb = TB + blockIdx.y * strideTB + c0 * ldtb;
  dependency_wait();
  {
    // the panels' T and the six blocks of V^T V below them, pairs of rows, all loads in flight together
    constexpr int NT2 = 4 * QW * QW / 2 / BTT, NG2 = 6 * QW * QW / 2 / BTT;
    double2 vt[NT2], vg[NG2];
    int og[NG2];
#pragma unroll
    for (int x = 0; x < NT2; ++x) {
      const int e = (tid + x * BTT) * 2, q = e / (QW * QW);
      vt[x] = q * QW < w ? make_double2(Tb[e], Tb[e + 1]) : make_double2(0.0, 0.0);
    }
#pragma unroll
    for (int x = 0; x < NG2; ++x) {
      const int e = (tid + x * BTT) * 2, blk = e / (QW * QW), r = e % (QW * QW);
      const int bi = blk == 0 ? 1 : (blk <= 2 ? 2 : 3), bj = blk - bi * (bi - 1) / 2;
      const int i = bi * QW + r % QW, j = bj * QW + r / QW;
      const double* src = Gb + i + j * ldg;
      og[x] = i + j * BTL;
      vg[x] = make_double2(i < w ? src[0] : 0.0, i + 1 < w ? src[1] : 0.0);
    }
#pragma unroll
    for (int x = 0; x < NT2; ++x) {
      const int e = (tid + x * BTT) * 2, q = e / (QW * QW), r = e % (QW * QW);
      *reinterpret_cast<double2*>(S + q * QW + r % QW + (q * QW + r / QW) * BTL) = vt[x];
    }
#pragma unroll
    for (int x = 0; x < NG2; ++x) *reinterpret_cast<double2*>(S + og[x]) = vg[x];
  }
  __syncthreads();
#pragma unroll
  for (int h = QW; h < BTW; h *= 2) {
    const int rt = h / 16, ct = h / 8, per = rt * ct, pairs = BTW / (2 * h);  // 16 x 8 tiles of a pair's T12
    if (w <= h) break;
    for (int u = warp; u < pairs * per; u += BTT / 32) {  // P = T1 (V2^T V1)^T, T1 upper: k from the row
      const int p = u / per, o = p * 2 * h, ti = (u % per) / ct * 16, tj = (u % per) % ct * 8;
      double c[4] = {0.0, 0.0, 0.0, 0.0};
      bt_mma<true, BTL>(c, S + o + ti + (o + ti) * BTL, BTL, S + o + h + tj + (o + ti) * BTL, h - ti);
      bt_store(P + p * h + ti + tj * BTP, BTP, c, 1.0);
    }
    __syncthreads();
    for (int u = warp; u < pairs * per; u += BTT / 32) {  // T12 = -P T2, T2 upper: k up to the column
      const int p = u / per, o = p * 2 * h, ti = (u % per) / ct * 16;
      const int cj = u >= BTT / 32 ? ct - 1 - (u % per) % ct : (u % per) % ct, tj = cj * 8;
      double c[4] = {0.0, 0.0, 0.0, 0.0};
      bt_mma<false, BTL>(c, P + p * h + ti, BTP, S + o + h + (o + h + tj) * BTL, tj + 8);
      bt_store(S + o + ti + (o + h + tj) * BTL, BTL, c, -1.0);
    }
    // V2^T V1 of these pairs is used up: T is upper triangular to the next level
    for (int e = tid; e < pairs * h * h; e += BTT) {
      const int p = e / (h * h), i = e % h, j = e / h % h;
      S[p * 2 * h + h + i + (p * 2 * h + j) * BTL] = 0.0;
    }
    __syncthreads();
  }
  release_dependents();
  // zeros below the diagonal, and beside the block when jb has more than one
  for (int j = warp; j < w; j += BTT / 32)
    for (int i = tid & 31; i < jb; i += 32) {
      const int l = i - c0;
      Bb[i + j * ldtb] = l >= 0 && l <= j ? S[l + j * BTL] : 0.0;
    }
}

// P(:,col) <- T^T P(:,col)  or  T P(:,col), T upper triangular w x w (ld QW)
__global__ void apply_t_kernel(int w, int n, const double* __restrict__ T, int64_t strideT, double* P,
                               int64_t ldp, int64_t strideP, int trans) {
  __shared__ double t[QW * QW];
  const double* Tb = T + blockIdx.y * strideT;
  double* Pb = P + blockIdx.y * strideP;
  for (int e = threadIdx.x; e < QW * QW; e += blockDim.x) t[e] = Tb[e];
  __syncthreads();
  for (int col = blockIdx.x * blockDim.x + threadIdx.x; col < n; col += gridDim.x * blockDim.x) {
    double x[QW];
#pragma unroll
    for (int i = 0; i < QW; ++i) x[i] = (i < w) ? Pb[i + col * ldp] : 0.0;
    for (int i = 0; i < w; ++i) {
      double s = 0.0;
      if (trans) {
        // (T^T x)_i = sum_{j<=i} T(j,i) x_j
#pragma unroll
        for (int j = 0; j < QW; ++j)
          if (j <= i) s += t[j + i * QW] * x[j];
      } else {
        // (T x)_i = sum_{i<=j<w} T(i,j) x_j
#pragma unroll
        for (int j = 0; j < QW; ++j)
          if (j >= i && j < w) s += t[i + j * QW] * x[j];
      }
      Pb[i + col * ldp] = s;
    }
  }
}

constexpr size_t shared_base() { return ((sizeof(PanelShared) + 15) / 16) * 16; }

template <bool SMEM>
cudaError_t set_attrs() {
  static std::atomic<int> attr_set[kMaxDevices];
  return once_per_device(attr_set, [] {
    const cudaError_t e = cudaFuncSetAttribute(qr_panel_kernel<SMEM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               static_cast<int>(shared_base() + SMEM_CHUNK_CAP + 64));
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(qr_panel_kernel<SMEM>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  });
}

template <bool SMEM>
cudaError_t launch_panel(const PanelArgs& pa, int cl, int batch, size_t smem, cudaStream_t st) {
  cudaError_t e = set_attrs<SMEM>();
  if (e != cudaSuccess) return e;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(cl, batch, 1);
  cfg.blockDim = dim3(QT, 1, 1);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr_l[1];
  attr_l[0].id = cudaLaunchAttributeClusterDimension;
  attr_l[0].val.clusterDim.x = cl;
  attr_l[0].val.clusterDim.y = 1;
  attr_l[0].val.clusterDim.z = 1;
  cfg.attrs = attr_l;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, qr_panel_kernel<SMEM>, pa);
}

template <int NW, int RN>
cudaError_t launch_reg(const PanelArgs& pa, int cl, int batch, cudaStream_t st) {
  static std::atomic<int> attr_set[kMaxDevices];
  const cudaError_t e = once_per_device(attr_set, [] {
    return cudaFuncSetAttribute(qr_panel_reg_kernel<NW, RN>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
  });
  if (e != cudaSuccess) return e;
  return launch_dependent(qr_panel_reg_kernel<NW, RN>, dim3(cl, batch, 1), dim3(NW * 32), 0, st, dim3(cl), pa);
}

// 16-CTA clusters are non-portable: use them only if the device can place one
// with the largest shared-memory footprint; otherwise the portable 8.
int max_cluster() {
  static std::atomic<int> cache[kMaxDevices];
  return per_device_value(cache, [] {
    int mc = 8;
    if (set_attrs<true>() == cudaSuccess) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(16, 1, 1);
      cfg.blockDim = dim3(QT, 1, 1);
      cfg.dynamicSmemBytes = shared_base() + SMEM_CHUNK_CAP;
      cudaLaunchAttribute a[1];
      a[0].id = cudaLaunchAttributeClusterDimension;
      a[0].val.clusterDim.x = 16;
      a[0].val.clusterDim.y = 1;
      a[0].val.clusterDim.z = 1;
      cfg.attrs = a;
      cfg.numAttrs = 1;
      int n = 0;
      if (cudaOccupancyMaxActiveClusters(&n, qr_panel_kernel<true>, &cfg) == cudaSuccess && n > 0) mc = 16;
    }
    cudaGetLastError();
    return mc;
  });
}

// Cluster size and warps per CTA (32 rows each) of the register-resident panel; false when the
// rows do not fit (m > 8192 with clusters of 16).  The cheapest configuration by the measured
// times of one 32-column panel alone on the GPU: a CTA of 4 / 8 / 16 warps 26 / 30 / 45 us, and
// the exchange 7 us more with clusters of 2 or 4, 10 us with 8, 16.5 us with 16 (m = 512: 33 us on
// 4 CTAs of 4 warps against 47 us on one of 16; m = 8192: 63 us on 16 x 16).  A batch that does
// not fit the GPU at once pays per wave: its members then take fewer, larger CTAs.
bool reg_config(int m, int batch, int maxcl, int* cl, int* nw) {
  double best = 1e300;
  for (int n : {4, 8, 16}) {
    const double t_cta = n == 4 ? 26.0 : (n == 8 ? 30.0 : 45.0);
    const int per_sm = n == 4 ? 2 : 1;
    for (int c = 1; c <= maxcl; c *= 2) {
      if (static_cast<int64_t>(c) * n * 32 < m) continue;
      const double t = t_cta + (c == 1 ? 0.0 : (c <= 4 ? 7.0 : (c == 8 ? 10.0 : 16.5)));
      const double waves = static_cast<double>(c) * batch / (static_cast<double>(num_sms()) * per_sm);
      const double cost = t * std::max(1.0, waves);
      if (cost < best) {
        best = cost;
        *cl = c;
        *nw = n;
      }
    }
  }
  return best < 1e300;
}

}  // namespace

int panel_cluster_max() { return max_cluster(); }

int qr_panel_config(int m, int w) {
  const int maxcl = max_cluster();
  int cl = 1, nw = 0;
  if (reg_config(m, 1, maxcl, &cl, &nw)) return cl;
  cl = 1;
  while (cl < maxcl && (static_cast<size_t>(((m + cl - 1) / cl + 7) / 16 * 16 + 8) * w * 8 > SMEM_CHUNK_CAP ||
                        (m + cl - 1) / cl > 512))
    cl *= 2;
  const size_t chunk = static_cast<size_t>(((m + cl - 1) / cl + 7) / 16 * 16 + 8) * w * 8;
  return chunk <= SMEM_CHUNK_CAP ? cl : -cl;
}

cudaError_t qr_panel(int m, int w, double* A, int64_t lda, int64_t strideA, double* tau, int64_t strideTau,
                     double* T, int64_t strideT, double* Vexp, int64_t ldv, int64_t strideV, int batch,
                     cudaStream_t st, int split, int64_t gap, int* status, long long wait_limit) {
  if (m <= 0 || w <= 0 || batch <= 0) return cudaSuccess;
  if (w > QW || m < w || gap < 0 || (gap > 0 && split < w)) return cudaErrorInvalidValue;
  const int maxcl = max_cluster();
  // smallest cluster whose per-CTA row chunk fits in shared memory, with at most ~512 rows per CTA
  int cl = 1;
  while (cl < maxcl && (static_cast<size_t>(((m + cl - 1) / cl + 7) / 16 * 16 + 8) * w * 8 > SMEM_CHUNK_CAP ||
                        (m + cl - 1) / cl > 512))
    cl *= 2;
  PanelArgs pa;
  pa.m = m;
  pa.w = w;
  pa.rows_per = (m + cl - 1) / cl;
  pa.rp_ld = (pa.rows_per + 7) / 16 * 16 + 8;  // = 8 mod 16: conflict-free half-warp access
  pa.A = A;
  pa.lda = lda;
  pa.strideA = strideA;
  pa.split = (split > 0 && gap > 0) ? split : m;
  pa.gap = gap;
  pa.tau = tau;
  pa.strideTau = strideTau;
  pa.T = T;
  pa.strideT = strideT;
  pa.V = Vexp;
  pa.ldv = ldv;
  pa.strideV = strideV;
  pa.status = status;
  pa.wait_limit = wait_limit == 0 ? kPanelTimeoutCycles : wait_limit;
  int rcl = 0, rnw = 0;
  if (reg_config(m, batch, maxcl, &rcl, &rnw)) {
    pa.rows_per = (m + rcl - 1) / rcl;
    switch (rnw) {
      case 4: return launch_reg<4, 4>(pa, rcl, batch, st);
      case 8: return launch_reg<8, 4>(pa, rcl, batch, st);
      default: return launch_reg<16, 4>(pa, rcl, batch, st);
    }
  }
  if (!Vexp) return cudaErrorInvalidValue;  // the panels below always write V
  const size_t chunk = static_cast<size_t>(pa.rp_ld) * w * 8;
  if (chunk <= SMEM_CHUNK_CAP) return launch_panel<true>(pa, cl, batch, shared_base() + chunk, st);
  return launch_panel<false>(pa, cl, batch, shared_base(), st);
}

cudaError_t extract_v(int m, int w, const double* A, int64_t lda, int64_t strideA, double* V, int64_t ldv,
                      int64_t strideV, int batch, cudaStream_t st, int split, int64_t gap) {
  if (m <= 0 || w <= 0 || batch <= 0) return cudaSuccess;
  if (gap < 0 || (gap > 0 && split < w)) return cudaErrorInvalidValue;
  if (!(split > 0 && gap > 0)) split = m;
  int blocks = static_cast<int>(std::min<int64_t>((static_cast<int64_t>(m) * w + 255) / 256, 2048));
  return launch_dependent(extract_v_kernel, dim3(blocks, batch), dim3(256), 0, st, dim3(1), m, w, A, lda, strideA, V, ldv, strideV, split, gap);
}

cudaError_t block_t_merge(int jb, const double* T, int64_t strideT, const double* G, int64_t ldg, int64_t strideG,
                          double* TB, int64_t ldtb, int64_t strideTB, int batch, cudaStream_t st) {
  if (jb <= 0 || batch <= 0) return cudaSuccess;
  constexpr int smem = (BTW * BTL + 64 * BTP) * 8;
  static std::atomic<int> attr_set[kMaxDevices];
  const cudaError_t attr = once_per_device(attr_set, [] {
    return cudaFuncSetAttribute(block_t_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  });
  if (attr != cudaSuccess) return attr;
  return launch_dependent(block_t_kernel, dim3((jb + BTW - 1) / BTW, batch), dim3(BTT), smem, st, dim3(1), jb, T,
                          strideT, G, ldg, strideG, TB, ldtb, strideTB);
}

cudaError_t apply_t(int w, int n, const double* T, int64_t strideT, double* P, int64_t ldp, int64_t strideP,
                    int trans, int batch, cudaStream_t st) {
  if (n <= 0 || w <= 0 || batch <= 0) return cudaSuccess;
  if (w > QW) return cudaErrorInvalidValue;
  int blocks = std::max(1, std::min((n + 127) / 128, 1024));
  apply_t_kernel<<<dim3(blocks, batch), 128, 0, st>>>(w, n, T, strideT, P, ldp, strideP, trans);
  return cudaGetLastError();
}

}  // namespace zolo
