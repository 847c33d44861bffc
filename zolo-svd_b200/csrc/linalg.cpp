// Recursive Cholesky / triangular solves and the blocked structured Householder
// QR, expressed as DMMA GEMMs plus small leaf kernels.  See linalg.h.
#include "linalg.h"

#include <algorithm>
#include <string>

namespace zolo {

namespace {
constexpr int NB = kLeaf;  // leaf of the Cholesky / TRSM recursion
constexpr int PW = 32;     // Householder panel width
constexpr int QB = 128;    // Householder block: four panels, one rank-128 trailing update
constexpr int QA = 512;    // reflector block of ormqr under the INT8-emulated GEMM: K = 512 updates

int split_point(int n) {
  int n1 = ((n / 2) + NB - 1) / NB * NB;
  if (n1 >= n) n1 = n - NB;
  if (n1 <= 0) n1 = n / 2;
  return n1;
}
// Algorithmic flops of a product: lower triangle only (tri); k >= output column (kfrom_n); the
// triangular operand's zero k range skipped (kfrom_n / kto_m).
double algo_flops(int M, int N, int K, int tri, int kfrom_n, int kto_m) {
  double f = (tri ? 1.0 : 2.0) * M * static_cast<double>(N) * K;
  if (kfrom_n == 2) {
    // row i uses k >= i, over its lower-triangle (tri) or all N columns
    f = 0.0;
    for (int i = 0; i < std::min(M, K); ++i) f += 2.0 * (tri ? std::min(i + 1, N) : N) * (K - i);
  } else if (kfrom_n == 3) {
    // entry (i, j) uses k >= max(i, j) (no tri)
    f = 0.0;
    for (int i = 0; i < std::min(M, K); ++i) {
      const double jn = std::min(i + 1, N);  // columns j <= i: K - i each
      const double jm = std::max(0, std::min(N, K) - i - 1);  // columns i < j < K: K - j each
      f += 2.0 * (jn * (K - i) + jm * (K - i - 1) - jm * (jm - 1.0) / 2.0);
    }
  } else if (kfrom_n) {
    const double nn = std::min(N, K);
    f = 2.0 * M * (static_cast<double>(N) * K - nn * (nn - 1.0) / 2.0 - (N - nn) * static_cast<double>(K));
  }
  if (kto_m == 2) {
    // column j uses k <= j: sum over columns of min(K, j + 1)
    const double nn = std::min(N, K);
    f = 2.0 * M * (nn * (nn + 1.0) / 2.0 + (N - nn) * static_cast<double>(K));
  } else if (kto_m) {
    // row i uses k <= i: sum over rows of min(K, i + 1)
    const double mm = std::min(M, K);
    f = 2.0 * N * (mm * (mm + 1.0) / 2.0 + (M - mm) * static_cast<double>(K));
  }
  return f;
}
}  // namespace

namespace {
// Products the INT8-emulated GEMM takes while an OzScope is active: long enough K for its
// tile pipeline and at least two waves of 128 x 64 output tiles on the GPU (measured against
// the DMMA GEMM on square products: equal at n = 1024, one wave; 1.7x at n = 2048, 3.5 waves;
// 2.3x at n = 4096).
constexpr int kOzMinK = 256;
bool oz_eligible(int M, int N, int K, int batch, int tri) {
  if (K < kOzMinK || M <= 0 || N <= 0) return false;
  const int64_t tm = (M + 127) / 128, tn = (N + 63) / 64;
  int64_t tiles = tm * tn;
  if (tri) {
    tiles = 0;
    for (int64_t i = 0; i < tm; ++i) tiles += std::min<int64_t>(tn, 2 * i + 2);
  }
  return tiles * batch >= 2 * static_cast<int64_t>(num_sms());
}
}  // namespace

void gemm(Context& c, int transA, int transB, int M, int N, int K, double alpha, Mat A, Mat B, double beta, Mat C,
          int batch, const double* alpha_vec, int tri, int kfrom_n, cudaStream_t st, int kto_m) {
  if (c.oz_active && !alpha_vec && oz_eligible(M, N, K, batch, tri)) {
    ozgemm(c, transA, transB, M, N, K, alpha, A, B, beta, C, batch, c.oz_active, tri, kfrom_n, st, kto_m);
    return;
  }
  GemmArgs a;
  a.M = M;
  a.N = N;
  a.K = K;
  a.transA = transA;
  a.transB = transB;
  a.A = A.p;
  a.lda = A.ld;
  a.strideA = A.stride;
  a.B = B.p;
  a.ldb = B.ld;
  a.strideB = B.stride;
  a.C = C.p;
  a.ldc = C.ld;
  a.strideC = C.stride;
  a.alpha = alpha;
  a.beta = beta;
  a.alpha_vec = alpha_vec;
  a.batch = batch;
  a.tri = tri;
  a.kfrom_n = kfrom_n;
  a.kto_m = kto_m;
  cudaStream_t s = st ? st : c.stream();
  Profiler::Rec rec;
  const int cls = tri ? 6 : (M <= 32 ? 3 : (N <= 64 ? 4 : (K <= 64 ? 5 : (K <= 256 ? 8 : 0))));
  if (c.prof.on) {
    const double f = algo_flops(M, N, K, tri, kfrom_n, kto_m);
    c.prof.begin(cls, f * batch, s, &rec);
  }
  const size_t need = dgemm_scratch(a);
  // one buffer a stream: the products of a stream follow one another
  double* scratch = need ? c.buf(s == c.stream() ? "gemm_k" : "gemm_k_side", need) : nullptr;
  ck(dgemm(a, s, scratch));
  if (c.prof.on) c.prof.end(rec, s);
  c.stats.launches += need ? 2 : 1;
}

void ozgemm(Context& c, int transA, int transB, int M, int N, int K, double alpha, Mat A, Mat B, double beta, Mat C,
            int batch, int slices, int tri, int kfrom_n, cudaStream_t st, int kto_m) {
  GemmArgs a;
  a.M = M;
  a.N = N;
  a.K = K;
  a.transA = transA;
  a.transB = transB;
  a.A = A.p;
  a.lda = A.ld;
  a.strideA = A.stride;
  a.B = B.p;
  a.ldb = B.ld;
  a.strideB = B.stride;
  a.C = C.p;
  a.ldc = C.ld;
  a.strideC = C.stride;
  a.alpha = alpha;
  a.beta = beta;
  a.batch = batch;
  a.tri = tri;
  a.kfrom_n = kfrom_n;
  a.kto_m = kto_m;
  if (!ozgemm_k_ok(slices, K)) {
    // exact INT32 accumulation bounds K: run K in chunks, accumulating into C (the
    // triangular k-skips refer to the whole K range and are dropped; zeros stay zeros)
    const int kc = 16384;
    for (int k0 = 0; k0 < K; k0 += kc) {
      const int kk = std::min(kc, K - k0);
      const Mat Ak{A.p + (transA ? k0 : static_cast<int64_t>(k0) * A.ld), A.ld, A.stride};
      const Mat Bk{B.p + (transB ? static_cast<int64_t>(k0) * B.ld : k0), B.ld, B.stride};
      ozgemm(c, transA, transB, M, N, kk, alpha, Ak, Bk, k0 == 0 ? beta : 1.0, C, batch, slices, tri, 0, st, 0);
    }
    return;
  }
  cudaStream_t s = st ? st : c.stream();
  const bool side = s == c.side_stream() && s != c.stream();
  const std::string pre = side ? "ozs_" : "oz_";
  OzWorkSizes sz;
  ozgemm_work_bytes(a, slices, &sz);
  OzWork w;
  w.sliceA = reinterpret_cast<int8_t*>(c.buf(pre + "sa", (sz.slice_a + 7) / 8));
  w.sliceB = reinterpret_cast<int8_t*>(c.buf(pre + "sb", (sz.slice_b + 7) / 8));
  unsigned long long* rows =
      reinterpret_cast<unsigned long long*>(c.buf(pre + "rows", (sz.rows_a + sz.rows_b) * 3 / 2 + 2));
  w.maxA = rows;
  w.maxB = rows + sz.rows_a;
  w.expA = reinterpret_cast<int*>(rows + sz.rows_a + sz.rows_b);
  w.expB = w.expA + sz.rows_a;
  w.status = c.oz_status_word();
  // profiled: class 9 from the start to the kernel's launch (splitting), class 7 the kernel
  Profiler::Rec split_rec, rec;
  const bool profile = c.prof.on && M > 0 && N > 0 && K > 0 && batch > 0;  // the kernel runs
  if (profile) {
    c.prof.begin(9, 0.0, s, &split_rec);
    rec.a = c.prof.take();
    rec.b = c.prof.take();
    rec.cls = 7;
    rec.flops = algo_flops(M, N, K, tri, kfrom_n, kto_m) * batch;
    w.before_kernel = split_rec.b;
    w.before_kernel2 = rec.a;
  }
  ck(zolo::ozgemm(a, slices, w, s, num_sms()));
  if (profile) {
    c.prof.recs.push_back(split_rec);
    c.prof.end(rec, s);
  }
  c.stats.launches += 3;
}

int oz_status(Context& c) {
  int* d = c.oz_status_word();
  int v = 0;
  ck(cudaMemcpyAsync(&v, d, sizeof(int), cudaMemcpyDeviceToHost, c.stream()));
  ck(cudaStreamSynchronize(c.stream()));
  if (v) ck(cudaMemsetAsync(d, 0, sizeof(int), c.stream()));
  return v;
}

static void potrf_rec(Context& c, int n, Mat A, int batch, int* dinfo, int off, DiagInv D) {
  if (n <= NB) {
    Profiler::Rec rec;
    if (c.prof.on) c.prof.begin(2, static_cast<double>(n) * n * n / 3.0 * batch, c.stream(), &rec);
    ck(potrf_leaf(n, A.p, A.ld, A.stride, batch, dinfo, off, D.block(off / NB), NB, D.stride, c.stream()));
    if (c.prof.on) c.prof.end(rec, c.stream());
    c.stats.launches++;
    return;
  }
  const int n1 = split_point(n), n2 = n - n1;
  potrf_rec(c, n1, A, batch, dinfo, off, D);
  // A21 <- A21 L11^{-T}  (out of place through a scratch copy)
  const int64_t ldt = (n2 + 1) / 2 * 2;
  Mat tmp{c.buf("potrf_tmp", static_cast<size_t>(ldt) * n1 * batch), ldt, ldt * n1};
  ck(scale_copy(n2, n1, 1.0, A.at(n1, 0).p, A.ld, A.stride, tmp.p, tmp.ld, tmp.stride, batch, 0.0, c.stream()));
  c.stats.launches++;
  trsm_rlt(c, n2, n1, A, tmp, A.at(n1, 0), batch, D, off / NB);
  // A22 -= A21 A21^T (lower)
  gemm(c, 0, 1, n2, n2, n1, -1.0, A.at(n1, 0), A.at(n1, 0), 1.0, A.at(n1, n1), batch, nullptr, 1, 0);
  potrf_rec(c, n2, A.at(n1, n1), batch, dinfo, off + n1, D);
}

void potrf(Context& c, int n, Mat A, int batch, int* dinfo, DiagInv D) {
  // size the scratch of the largest recursion level first (no growth mid-recursion)
  if (n > NB) {
    const int n1 = split_point(n), n2 = n - n1;
    c.buf("potrf_tmp", static_cast<size_t>((n2 + 1) / 2 * 2) * n1 * batch);
  }
  potrf_rec(c, n, A, batch, dinfo, 0, D);
}

// Scratch of a node's n2 x n1 block (even leading dimension), and the most that any split of n rows
// takes: even(n2) n1 <= (n2 + 1) n1 with n1 + n2 = n.
static Mat block21(double* p, int n1, int n2) {
  const int64_t ld = (n2 + 1) / 2 * 2;
  return Mat{p, ld, ld * n1};
}
constexpr int kPairBatch = 16;
static size_t block21_elems(int n) { return static_cast<size_t>(n / 2 + 1) * (n / 2 + 1); }

// Cholesky and the inverse of its factor together: with Y11 = L11^{-1} from the first half,
// L21 = A21 Y11^T is one GEMM (no recursive triangular solve) into Tmp, A21 <- L21 Y11, then
// A22 -= L21 L21^T, the second half, and Y21 = -Y22 A21.  n^3/3 + n^3/3 flops, as Cholesky plus
// triangular inverse, in four launches a node; only Y is complete at the end.
static void potrf_inv_rec(Context& c, int n, Mat A, Mat Y, int batch, int* dinfo, int off, double* tmp) {
  if (n <= NB) {
    Profiler::Rec rec;
    if (c.prof.on) c.prof.begin(2, static_cast<double>(n) * n * n / 3.0 * batch, c.stream(), &rec);
    ck(potrf_leaf(n, A.p, A.ld, A.stride, batch, dinfo, off, Y.p, Y.ld, Y.stride, c.stream()));
    if (c.prof.on) c.prof.end(rec, c.stream());
    c.stats.launches++;
    return;
  }
  // one CTA a member for two leaves, with most of an SM's shared memory: not where a batch keeps the
  // SMs busy
  const bool pair = batch <= kPairBatch;
  if (pair && n <= 2 * NB) {
    Profiler::Rec rec;
    if (c.prof.on) c.prof.begin(2, 2.0 * n * n * n / 3.0 * batch, c.stream(), &rec);
    ck(potrf_inv_pair(n, A.p, A.ld, A.stride, batch, dinfo, off, Y.p, Y.ld, Y.stride, c.stream()));
    if (c.prof.on) c.prof.end(rec, c.stream());
    c.stats.launches++;
    return;
  }
  const int n1 = pair ? (n / 2 + 2 * NB - 1) / (2 * NB) * (2 * NB) : split_point(n), n2 = n - n1;
  potrf_inv_rec(c, n1, A, Y, batch, dinfo, off, tmp);
  const Mat Tmp = block21(tmp, n1, n2);
  // Y11^T is upper triangular (k up to the column), Y11 lower (k from the column)
  gemm(c, 0, 1, n2, n1, n1, 1.0, A.at(n1, 0), Y, 0.0, Tmp, batch, nullptr, 0, 0, nullptr, 2);
  gemm(c, 0, 0, n2, n1, n1, 1.0, Tmp, Y, 0.0, A.at(n1, 0), batch, nullptr, 0, 1);
  gemm(c, 0, 1, n2, n2, n1, -1.0, Tmp, Tmp, 1.0, A.at(n1, n1), batch, nullptr, 1, 0);
  potrf_inv_rec(c, n2, A.at(n1, n1), Y.at(n1, n1), batch, dinfo, off + n1, tmp);
  // Y22 lower: k up to the row
  gemm(c, 0, 0, n2, n1, n2, -1.0, Y.at(n1, n1), A.at(n1, 0), 0.0, Y.at(n1, 0), batch, nullptr, 0, 0, nullptr, 1);
}

void potrf_inv(Context& c, int n, Mat A, Mat Y, int batch, int* dinfo) {
  ck(set_identity(n, n, Y.p, Y.ld, Y.stride, batch, 0.0, c.stream()));  // zero upper triangle
  c.stats.launches++;
  potrf_inv_rec(c, n, A, Y, batch, dinfo, 0, c.buf("potrf_inv_tmp", block21_elems(n) * batch));
}

void diag_inverses(Context& c, int n, Mat L, int batch, DiagInv D) {
  ck(trtri_blocks(n, L.p, L.ld, L.stride, D.p, NB, NB * NB, static_cast<int64_t>(nblocks(n)) * NB * NB, batch,
                  c.stream()));
  c.stats.launches++;
}

void trsm_rlt(Context& c, int m, int n, Mat L, Mat X, Mat Y, int batch, DiagInv D, int k0) {
  if (n <= NB) {
    Mat li{D.block(k0), NB, D.stride};
    gemm(c, 0, 1, m, n, n, 1.0, X, li, 0.0, Y, batch);
    return;
  }
  const int n1 = split_point(n), n2 = n - n1;
  trsm_rlt(c, m, n1, L, X, Y, batch, D, k0);
  gemm(c, 0, 1, m, n2, n1, -1.0, Y, L.at(n1, 0), 1.0, X.at(0, n1), batch);
  trsm_rlt(c, m, n2, L.at(n1, n1), X.at(0, n1), Y.at(0, n1), batch, D, k0 + n1 / NB);
}

void trsm_rln(Context& c, int m, int n, Mat L, Mat X, Mat Y, int batch, DiagInv D, int k0) {
  if (n <= NB) {
    Mat li{D.block(k0), NB, D.stride};
    gemm(c, 0, 0, m, n, n, 1.0, X, li, 0.0, Y, batch);
    return;
  }
  const int n1 = split_point(n), n2 = n - n1;
  trsm_rln(c, m, n2, L.at(n1, n1), X.at(0, n1), Y.at(0, n1), batch, D, k0 + n1 / NB);
  gemm(c, 0, 0, m, n1, n2, -1.0, Y.at(0, n1), L.at(n1, 0), 1.0, X, batch);
  trsm_rln(c, m, n1, L, X, Y, batch, D, k0);
}

// Level by level from the inverses of the 64 x 64 diagonal blocks: at block size s the blocks
// below the diagonal of all pairs of one matrix are two launches (batched over the pairs; a
// batch of matrices takes the pairs one after another), where the recursion by nodes took two a
// pair: 8 products instead of 30 in the chain at n = 1024.
void trtri_lower(Context& c, int n, Mat L, Mat Y, int batch) {
  ck(set_identity(n, n, Y.p, Y.ld, Y.stride, batch, 0.0, c.stream()));  // zero upper triangle
  ck(trtri_blocks(n, L.p, L.ld, L.stride, Y.p, Y.ld, NB * (Y.ld + 1), Y.stride, batch, c.stream()));
  c.stats.launches += 2;
  if (n <= NB) return;
  double* tmp = c.buf("trtri_tmp", block21_elems(n) * batch);
  // Y21 = -Y22 (L21 Y11) of `count` pairs from row o on, s + t rows each
  auto pairs = [&](int o, int s, int t, int count) {
    auto view = [&](Mat m, int i, int j) {
      m = m.at(o + i, o + j);
      if (count > 1) m.stride = 2 * s * (m.ld + 1);
      return m;
    };
    const int nb = count > 1 ? count : batch;
    const Mat P = block21(tmp, s, t);
    gemm(c, 0, 0, t, s, s, 1.0, view(L, s, 0), view(Y, 0, 0), 0.0, P, nb, nullptr, 0, 1);
    gemm(c, 0, 0, t, s, t, -1.0, view(Y, s, s), P, 0.0, view(Y, s, 0), nb, nullptr, 0, 0, nullptr, 1);
  };
  for (int s = NB; s < n; s *= 2) {
    const int full = n / (2 * s), rest = n - full * 2 * s;
    if (batch == 1 && full > 1) pairs(0, s, s, full);
    else
      for (int q = 0; q < full; ++q) pairs(q * 2 * s, s, s, 1);
    if (rest > s) pairs(full * 2 * s, s, rest - s, 1);
  }
}

// Rows of panel j (columns j .. j + jb - 1) in the mtot x n matrix: `mp`
// logical rows, of which the first `split` start at row j and the rest follow
// after `gap` skipped rows (gap = 0: one window).
struct PanelRows {
  int mp, split;
  int64_t gap;
};

static inline PanelRows panel_rows(int mtot, int m_top, bool top_tri, int j, int jb) {
  const int hi = m_top >= 0 ? std::min(mtot, m_top + j + jb) : mtot;
  if (!top_tri || m_top < 0 || m_top <= j + jb) return PanelRows{hi - j, hi - j, 0};
  return PanelRows{jb + (hi - m_top), jb, static_cast<int64_t>(m_top) - j - jb};
}

// P = V^T B over the panel rows (B starts at the panel's first row; V holds the rows packed)
static void panel_vt_b(Context& c, const PanelRows& R, int jb, int ncols, Mat V, Mat B, Mat P, int batch,
                       cudaStream_t st = nullptr) {
  gemm(c, 1, 0, jb, ncols, R.split, 1.0, V, B, 0.0, P, batch, nullptr, 0, 0, st);
  if (R.split < R.mp)
    gemm(c, 1, 0, jb, ncols, R.mp - R.split, 1.0, V.at(R.split, 0), B.at(static_cast<int>(R.split + R.gap), 0),
         1.0, P, batch, nullptr, 0, 0, st);
}

// B -= V P over the panel rows
static void panel_b_minus_vp(Context& c, const PanelRows& R, int jb, int ncols, Mat V, Mat P, Mat B, int batch,
                             cudaStream_t st = nullptr) {
  gemm(c, 0, 0, R.split, ncols, jb, -1.0, V, P, 1.0, B, batch, nullptr, 0, 0, st);
  if (R.split < R.mp)
    gemm(c, 0, 0, R.mp - R.split, ncols, jb, -1.0, V.at(R.split, 0), P, 1.0,
         B.at(static_cast<int>(R.split + R.gap), 0), batch, nullptr, 0, 0, st);
}

// T_B (jb x jb upper) of the block reflector I - V_B T_B V_B^T = H_1 H_2 ... of the block's
// 32-column panels (the compact WY form of LAPACK DLARFT, by pairs of panels): with the panels' T on the
// diagonal, T12 = -T1 (V1^T V2) T2, up to 128 columns in one launch, wider pairs by products.
// VB: the block's explicit V, mp packed rows.  T: the first panel's T (32 x 32 per panel).
static void block_t(Context& c, int jb, Mat VB, int mp, const double* T, int64_t strideT, Mat TB, int batch) {
  const int ldg = (std::max(jb, 2) + 1) / 2 * 2;
  Mat G{c.buf("qr_bg", static_cast<size_t>(ldg) * ldg * batch), ldg, static_cast<int64_t>(ldg) * ldg};
  // lower triangle of V_B^T V_B: its transpose gives the blocks above the diagonal
  gemm(c, 1, 0, jb, jb, mp, 1.0, VB, VB, 0.0, G, batch, nullptr, 1, 0);
  ck(block_t_merge(jb, T, strideT, G.p, G.ld, G.stride, TB.p, TB.ld, TB.stride, batch, c.stream()));
  c.stats.launches++;
  if (jb <= QB) return;
  Mat Tmp{c.buf("qr_btmp", static_cast<size_t>(ldg) * ldg * batch), ldg, static_cast<int64_t>(ldg) * ldg};
  for (int s = QB; s < jb; s *= 2)
    for (int o = 0; o + s < jb; o += 2 * s) {
      const int w = std::min(s, jb - o - s);
      // T1 upper (k from the row), T2 upper (k up to the column)
      gemm(c, 0, 1, s, w, s, 1.0, TB.at(o, o), G.at(o + s, o), 0.0, Tmp, batch, nullptr, 0, 2);
      gemm(c, 0, 0, s, w, w, -1.0, Tmp, TB.at(o + s, o + s), 0.0, TB.at(o, o + s), batch, nullptr, 0, 0, nullptr, 2);
    }
}

// C <- (I - V op(T) V^T) C over the panel's rows, V the panel at Vp in the factored matrix and C the
// columns at Cp (both at the panel's first row), one launch.
static void apply_panel(Context& c, const PanelRows& R, int jb, int ncols, Mat Vp, const double* T, int64_t strideT,
                        int trans, Mat Cp, int batch, cudaStream_t st) {
  Profiler::Rec rec;
  if (c.prof.on) c.prof.begin(5, 4.0 * R.mp * static_cast<double>(ncols) * jb * batch, st, &rec);
  ck(reflect(R.mp, ncols, jb, Vp.p, Vp.ld, Vp.stride, T, strideT, trans, Cp.p, Cp.ld, Cp.stride, batch, st, R.split,
             R.gap));
  if (c.prof.on) c.prof.end(rec, st);
  c.stats.launches++;
}

// Factorizations that apply every panel to all remaining columns at once (apply_panel) instead of
// in 128-column blocks: while the trailing update fits beside the next panel the blocks' T factors
// and products only lengthen the chain.  Measured, panelwise against blocks: QR of 1024 x 1024
// 1.52 / 1.67 ms, 2048 x 2048 3.71 / 4.04, 4096 x 2048 7.6 / 5.7; forming Q, where nothing hides the
// update, 512 x 512 0.147 / 0.157, 1024 x 1024 0.42 / 0.38, 2048 x 1024 0.86 / 0.55.  Batches of equal members form Q
// panel by panel up to 1.5e6 entries of their stacks: whole batched solves with 6e5 to 1.4e6 entries
// took 1 to 6 % less than in blocks for members of 64^2 to 160^2 and 300 x 100 (72 of 100^2 1.77 / 1.85 ms, 28 of
// 160^2 1.87 / 1.93) and the same within 1 % for 250^2, 400^2 and 600 x 150, which lose up to 2 % at 4e6.
static bool panelwise(int mtot, int n, int batch, bool qr) {
  const double one = static_cast<double>(mtot) * n, all = one * batch;
  return reflect_applies(mtot) && (qr ? all <= 4.5e6 : one <= 5e5 && all <= 1.5e6);
}

static void factor_panel(Context& c, int mtot, int n, int m_top, bool top_tri, int j, Mat W, double* tau, double* T,
                         int64_t strideT, Mat Vp, int batch, cudaStream_t st) {
  const int jb = std::min(PW, n - j);
  const PanelRows R = panel_rows(mtot, m_top, top_tri, j, jb);
  Profiler::Rec rec;
  if (c.prof.on) c.prof.begin(1, 2.0 * R.mp * static_cast<double>(jb) * jb * batch, st, &rec);
  ck(qr_panel(R.mp, jb, W.at(j, j).p, W.ld, W.stride, tau + j, n, T + (j / PW) * PW * PW, strideT, Vp.p, Vp.ld,
              Vp.stride, batch, st, R.split, R.gap, c.fault_word(), c.panel_wait));
  if (c.prof.on) c.prof.end(rec, st);
  c.stats.launches++;
}

// Householder QR panel by panel.  The chain (a panel, its reflector on the next panel's columns, the
// next panel) runs on the high-priority side stream alone, so that no step of it waits for another
// stream's event; the main stream updates the columns further right beside the next panel.
static bool geqrf_panelwise(Context& c, int mtot, int n, int m_top, Mat W, double* tau, double* T, int64_t strideT,
                            int batch, bool top_tri, const std::function<bool()>& keep_on) {
  cudaStream_t ms = c.stream(), ss = c.side_stream();
  const Mat none{nullptr, 0, 0};
  if (n <= 2 * PW) ss = ms;  // nothing to update beside a panel
  if (ss != ms) {
    ck(cudaEventRecord(c.event(0), ms));
    ck(cudaStreamWaitEvent(ss, c.event(0), 0));
  }
  bool rest = false;  // an update of the main stream that the next step on the side stream needs
  bool whole = true;
  for (int j = 0; j < n; j += PW) {
    factor_panel(c, mtot, n, m_top, top_tri, j, W, tau, T, strideT, none, batch, ss);
    const int nc = n - j - PW, jn = std::min(PW, nc);
    if (nc <= 0) break;
    if (j == 0 && keep_on && !keep_on()) {
      whole = false;
      break;
    }
    const PanelRows R = panel_rows(mtot, m_top, top_tri, j, PW);
    const double* Tj = T + (j / PW) * PW * PW;
    if (nc > jn) ck(cudaEventRecord(c.event(0), ss));
    if (rest) ck(cudaStreamWaitEvent(ss, c.event(1), 0));
    apply_panel(c, R, PW, jn, W.at(j, j), Tj, strideT, 1, W.at(j, j + PW), batch, ss);
    rest = nc > jn;
    if (rest) {
      ck(cudaStreamWaitEvent(ms, c.event(0), 0));
      apply_panel(c, R, PW, nc - jn, W.at(j, j), Tj, strideT, 1, W.at(j, j + PW + jn), batch, ms);
      ck(cudaEventRecord(c.event(1), ms));
    }
  }
  if (ss != ms) {
    ck(cudaEventRecord(c.event(0), ss));
    ck(cudaStreamWaitEvent(ms, c.event(0), 0));
  }
  return whole;
}

// Householder QR in 128-column blocks of four 32-column panels.  Inside a block each panel
// updates only the block's remaining columns (rank-32); the trailing columns take one
// rank-128 update per block, C -= V_B (T_B^T (V_B^T C)), whose GEMMs have K = rows and
// K = 128.  Look-ahead: the next block's columns are updated first, then the next block is
// factored on the side stream while the main stream updates the rest.
bool geqrf(Context& c, int mtot, int n, int m_top, Mat W, double* tau, double* T, int batch, bool top_tri,
           const std::function<bool()>& keep_on) {
  const int npan = (n + PW - 1) / PW;
  const int64_t ldv = (mtot + 1) / 2 * 2;
  const int64_t strideT = static_cast<int64_t>(npan) * PW * PW;
  if (panelwise(mtot, n, batch, true))
    return geqrf_panelwise(c, mtot, n, m_top, W, tau, T, strideT, batch, top_tri, keep_on);
  Mat Vp{c.buf("qr_v2", static_cast<size_t>(ldv) * PW * batch), ldv, ldv * PW};
  Mat Pp{c.buf("qr_p", static_cast<size_t>(PW) * QB * batch), PW, static_cast<int64_t>(PW) * QB};
  Mat VB{c.buf("qr_vb", static_cast<size_t>(ldv) * QB * batch), ldv, ldv * QB};
  Mat TB{c.buf("qr_tb", static_cast<size_t>(QB) * QB * batch), QB, static_cast<int64_t>(QB) * QB};
  Mat WB{c.buf("qr_wb", static_cast<size_t>(QB) * n * batch), QB, static_cast<int64_t>(QB) * n};
  Mat PB{c.buf("qr_pb", static_cast<size_t>(QB) * n * batch), QB, static_cast<int64_t>(QB) * n};
  cudaStream_t ms = c.stream(), ss = c.side_stream();
  auto factor_block = [&](int J, cudaStream_t st) {
    const int jend = std::min(n, J + QB);
    for (int j = J; j < jend; j += PW) {
      const int jb = std::min(PW, n - j);
      const int pj = j / PW;
      const PanelRows R = panel_rows(mtot, m_top, top_tri, j, jb);
      const int nc = jend - j - jb;
      // the panel on the block's other columns in one launch, 8 us where three products take 35 at
      // least; a large batch is past latency, and the products' 10 TF/s beat its 4.6
      const bool one = reflect_applies(R.mp) && static_cast<double>(R.mp) * nc * batch <= 1.2e6;
      factor_panel(c, mtot, n, m_top, top_tri, j, W, tau, T, strideT, one ? Mat{nullptr, 0, 0} : Vp, batch, st);
      if (j == 0 && n > PW && keep_on && !keep_on()) return false;
      if (nc <= 0) continue;
      if (one) {
        apply_panel(c, R, jb, nc, W.at(j, j), T + pj * PW * PW, strideT, 1, W.at(j, j + jb), batch, st);
        continue;
      }
      panel_vt_b(c, R, jb, nc, Vp, W.at(j, j + jb), Pp, batch, st);
      ck(apply_t(jb, nc, T + pj * PW * PW, strideT, Pp.p, Pp.ld, Pp.stride, 1, batch, st));
      c.stats.launches++;
      panel_b_minus_vp(c, R, jb, nc, Vp, Pp, W.at(j, j + jb), batch, st);
    }
    return true;
  };
  if (!factor_block(0, ms)) return false;
  for (int J = 0; J < n; J += QB) {
    const int jbB = std::min(QB, n - J);
    const int nc = n - J - jbB;
    if (nc <= 0) break;
    const PanelRows R = panel_rows(mtot, m_top, top_tri, J, jbB);
    ck(extract_v(R.mp, jbB, W.at(J, J).p, W.ld, W.stride, VB.p, VB.ld, VB.stride, batch, ms, R.split, R.gap));
    c.stats.launches++;
    block_t(c, jbB, VB, R.mp, T + (J / PW) * PW * PW, strideT, TB, batch);
    panel_vt_b(c, R, jbB, nc, VB, W.at(J, J + jbB), WB, batch, ms);
    // P = T_B^T (V_B^T C): T_B^T is lower triangular (k up to the row)
    gemm(c, 1, 0, jbB, nc, jbB, 1.0, TB, WB, 0.0, PB, batch, nullptr, 0, 0, ms, 1);
    const int jn = std::min(QB, nc);
    panel_b_minus_vp(c, R, jbB, jn, VB, PB, W.at(J, J + jbB), batch, ms);
    if (nc > jn) {
      ck(cudaEventRecord(c.event(0), ms));
      ck(cudaStreamWaitEvent(ss, c.event(0), 0));
      factor_block(J + jbB, ss);
      ck(cudaEventRecord(c.event(1), ss));
      panel_b_minus_vp(c, R, jbB, nc - jn, VB, PB.at(0, jn), W.at(J, J + jbB + jn), batch, ms);
      ck(cudaStreamWaitEvent(ms, c.event(1), 0));
    } else {
      factor_block(J + jbB, ms);
    }
  }
  return true;
}

// Q = H_1 ... H_k applied to the identity, one 128-column block reflector at a time from the
// last block: Q(rows, J:nq) -= V_B (T_B (V_B^T Q(rows, J:nq))).  Columns left of J are still
// identity columns with their one above the block's rows, so V_B^T leaves them zero.
// C <- H_1 ... H_n C (the Q of geqrf applied from the left), one block reflector of `width`
// columns (a multiple of 32) at a time from the last: C(rows, cols) -= V_B (T_B (V_B^T
// C(rows, cols))), T_B merged from the 32-column panels' T (block_t).  Width 128 gives K = 128
// updates on the DMMA update tiles; 512 gives K = 512 products, which the INT8-emulated GEMM
// takes (K >= 256), for about 1 % more flops in the T product; on DMMA both widths measure
// the same.  from_diag: C starts as the identity, so block J touches columns J .. ncols-1 only
// (left of J they are identity columns with their one above the block's rows, which V_B^T
// leaves zero).
static void apply_q_blocks(Context& c, int mtot, int n, int m_top, Mat W, const double* T, Mat C, int ncols,
                           bool from_diag, int batch, bool top_tri, int width) {
  const int npan = (n + PW - 1) / PW;
  const int64_t ldv = (mtot + 1) / 2 * 2;
  const int64_t strideT = static_cast<int64_t>(npan) * PW * PW;
  if (width == QB && panelwise(mtot, ncols, batch, false)) {
    for (int j = (npan - 1) * PW; j >= 0; j -= PW) {
      const int jb = std::min(PW, n - j), c0 = from_diag ? j : 0;
      apply_panel(c, panel_rows(mtot, m_top, top_tri, j, jb), jb, ncols - c0, W.at(j, j), T + (j / PW) * PW * PW,
                  strideT, 0, C.at(j, c0), batch, c.stream());
    }
    return;
  }
  const int bw = std::min(width, (n + PW - 1) / PW * PW);
  Mat VB{c.buf("qr_vb", static_cast<size_t>(ldv) * bw * batch), ldv, ldv * bw};
  Mat TB{c.buf("qr_tb", static_cast<size_t>(bw) * bw * batch), bw, static_cast<int64_t>(bw) * bw};
  Mat WB{c.buf("qr_wb", static_cast<size_t>(bw) * ncols * batch), bw, static_cast<int64_t>(bw) * ncols};
  Mat PB{c.buf("qr_pb", static_cast<size_t>(bw) * ncols * batch), bw, static_cast<int64_t>(bw) * ncols};
  const int nblk = (n + bw - 1) / bw;
  for (int b = nblk - 1; b >= 0; --b) {
    const int J = b * bw;
    const int jbB = std::min(bw, n - J);
    const PanelRows R = panel_rows(mtot, m_top, top_tri, J, jbB);
    const int c0 = from_diag ? J : 0;
    const int nc = ncols - c0;
    ck(extract_v(R.mp, jbB, W.at(J, J).p, W.ld, W.stride, VB.p, VB.ld, VB.stride, batch, c.stream(), R.split,
                 R.gap));
    c.stats.launches++;
    block_t(c, jbB, VB, R.mp, T + (J / PW) * PW * PW, strideT, TB, batch);
    panel_vt_b(c, R, jbB, nc, VB, C.at(J, c0), WB, batch);
    // P = T_B (V_B^T C): T_B is upper triangular (k from the row)
    gemm(c, 0, 0, jbB, nc, jbB, 1.0, TB, WB, 0.0, PB, batch, nullptr, 0, 2);
    panel_b_minus_vp(c, R, jbB, nc, VB, PB, C.at(J, c0), batch);
  }
}

void orgqr(Context& c, int mtot, int n, int m_top, Mat W, const double* T, Mat Q, int batch, int nq, bool top_tri) {
  if (nq < n) nq = n;
  ck(set_identity(mtot, nq, Q.p, Q.ld, Q.stride, batch, 1.0, c.stream()));
  c.stats.launches++;
  apply_q_blocks(c, mtot, n, m_top, W, T, Q, nq, true, batch, top_tri, QB);
}

void ormqr_left(Context& c, int mtot, int n, int m_top, Mat W, const double* T, Mat C, int ncols, int batch,
                bool top_tri) {
  if (ncols <= 0) return;
  apply_q_blocks(c, mtot, n, m_top, W, T, C, ncols, false, batch, top_tri, c.oz_active ? QA : QB);
}

}  // namespace zolo
