// C-ABI entry points of the LU path: LUDecomposition::{new, solve, det, ...},
// Matrix::{det, solve, inverse, is_non_singular} and Matrix * Matrix.
//
// FAST arithmetic: lu_fast_enqueue below. EXACT arithmetic: blocked right-looking LU
// (panel width W, default 64), for each panel [j0, j1 = j0 + jb):
//   panel  : pivots + L21/U11 of the panel, on one cluster in halves of 32 columns up to 4096 rows
//            (panel_cluster64.cu), else by the cooperative kernel (lu_panel.cu)
//   laswp  : the panel's row swaps on the other columns (lu.rs:140-145)
//   trsm   : U12 = L11^{-1} A12 for rows [j0, j1)
//   gemm   : S22 += L21 * U12
// S holds, for every not-yet-finished element, the partial sum
// of lu.rs:124-126 over the k already processed, so each element's sum is
// formed in the reference's order and subtracted once (lu.rs:128).
#include <algorithm>
#include <cstring>
#include <vector>

#include "la_internal.cuh"

namespace {

size_t pad4(size_t x) { return (x + 3) & ~size_t(3); }
bool aligned16(const void* p, size_t ld) {
  return (reinterpret_cast<uintptr_t>(p) % 16 == 0) && (ld % 2 == 0);
}

struct DevBuf {
  la_ctx ctx;
  void* p = nullptr;
  explicit DevBuf(la_ctx c) : ctx(c) {}
  ~DevBuf() { la_device_free(ctx, p); }
  la_status alloc(size_t bytes) { return la_device_alloc(ctx, &p, bytes); }
  bool try_alloc(size_t bytes) { return la_device_try_alloc(ctx, &p, bytes); }
  double* d() { return static_cast<double*>(p); }
};

// Phase timing for LA_OPT_PROFILE: a pair of events (from the context's pool)
// around each phase instance on the stream it runs on; the per-category sums
// are device time, so a panel overlapped with the trailing update is counted
// in full in both categories.
struct PhaseTimer {
  la_ctx ctx;
  bool on;
  size_t used = 0;
  struct Span { size_t b, e; int cat; };
  std::vector<Span> spans;
  explicit PhaseTimer(la_ctx c) : ctx(c), on(c->profile != 0) {}
  size_t record(cudaStream_t s) {
    if (used == ctx->event_pool.size()) {
      cudaEvent_t e;
      if (cudaEventCreate(&e) != cudaSuccess) { on = false; return 0; }
      ctx->event_pool.push_back(e);
    }
    cudaEventRecord(ctx->event_pool[used], s);
    return used++;
  }
  size_t begin(cudaStream_t s) { return on ? record(s) : 0; }
  void end(cudaStream_t s, size_t b, int cat) {
    if (!on) return;
    size_t e = record(s);
    if (on) spans.push_back({b, e, cat});
  }
  void finish() {
    for (int i = 0; i < 5; i++) ctx->phase_ms[i] = 0;
    if (!on) return;
    for (auto& sp : spans) {
      cudaEventSynchronize(ctx->event_pool[sp.e]);
      float ms = 0;
      cudaEventElapsedTime(&ms, ctx->event_pool[sp.b], ctx->event_pool[sp.e]);
      ctx->phase_ms[sp.cat] += ms;
    }
  }
};

enum { PH_PANEL = 0, PH_SWAP = 1, PH_TRSM = 2, PH_GEMM = 3, PH_OTHER = 4 };

// Shared memory that keeps trailing-update GEMM CTAs at two per SM, leaving an
// SM room for one CTA of the concurrent panel kernel.
constexpr size_t GEMM_SMEM_WITH_PANEL = 78 * 1024;

// FAST factorization of h->d_lu in place. Blocks of LU_BASE = 64 columns are factored in panels of at
// most 32:
//   panel : cluster kernel (panel_cluster64.cu); beyond 8192 rows the cooperative one (lu_panel.cu), on
//           all 64 columns
//   swaps of the panel on all other columns
//   inner : triangular solve and FMA update of the block's remaining columns (32 x 32, K = 32)
// and a wider block is its left half, that half's triangular solve and update of the right half,
// and the right half. After a block come its triangular solve and its update A22 -= L21 U12 on all
// columns right of it. Updates run on the tensor cores by exact splitting (gemm_split.cu), whose
// cost is the epilogue's per element of C, about the same for K = 64 and K = 256; so blocks are
// wide where there are many rows (lu_block), and 64 columns where the launches of the wider
// blocks' inner steps would cost more than they save. Every launch is a dependent one, so that only
// their execution adds up. Measured, factor + solve with 16 right-hand sides at n = 8192: 53.5 ms
// (64-column blocks throughout: 69.3 ms in the same build but for the guard of the split products;
// FP64 FMA updates beside a cooperative panel: 328 ms).
//
// Every element's operations depend on the blocks' columns and on the 128 x 64 tile grid that
// starts at each update's corner alone, so the allocation-free entry point, which updates in
// pieces of whole tiles, gives the same bits.
constexpr int LU_BASE = 64;
constexpr int LU_MAX_BLOCK = 256;
constexpr int SPLIT_MIN_MN = 64 * 64;  // smaller updates: one FMA launch is no slower than three

// Block width for R remaining rows.
int lu_block(int R) { return R > 3072 ? 256 : R > 1024 ? 128 : LU_BASE; }

// Workspace of the split products (digits of both operands) that a product may ask for.
constexpr size_t SPLIT_WS_MAX = (size_t)4 << 30;

// C (M x N) -= A B as a split product, in pieces of whole tiles that the workspace takes.
la_status split_update(la_ctx ctx, int M, int N, int K, const double* A, size_t lda, const double* B,
                       size_t ldb, double* C, size_t ldc, void* ws, size_t ws_bytes) {
  int rb = M, cb = N;
  auto half = [](int x, int q) { return std::max(q, ((x + 1) / 2 + q - 1) / q * q); };
  while (gemm_split_ws(rb, cb, K, false) > ws_bytes && (rb > 128 || cb > 64)) {
    if (rb > 128 && rb >= cb) rb = half(rb, 128);
    else if (cb > 64) cb = half(cb, 64);
    else rb = half(rb, 128);
  }
  la_status s = LA_OK;
  for (int r = 0; r < M && s == LA_OK; r += rb)
    for (int c = 0; c < N && s == LA_OK; c += cb)
      s = launch_gemm_split(ctx, ctx->stream, -1, std::min(rb, M - r), std::min(cb, N - c), K,
                            A + (size_t)r * lda, lda, B + c, ldb, false, C + (size_t)r * ldc + c, ldc,
                            false, ws, ws_bytes);
  return s;
}

// X <- U^-1 L^-1 X for many right-hand sides: blocks of up to SOLVE_BASE rows by the wavefront kernel,
// and between them split products, recursively, so that most terms are in few products of large K.
// What bounds the wavefront here is the FP64 pipe (n^2 nrhs FMAs at two per clock and SM: 1.7 ms of
// 2.4 at n = nrhs = 1000); the products do theirs on the tensor cores, with one rounding each.
// `id`: X is the identity on entry; row r of L^-1 ends at column r, so the forward half leaves the
// columns beyond out. (Against the permuted identity every column's zeros and single entries sent most
// tiles to the FMA chains: 4.89 ms for the inverse of order 1000 instead of 3.84.)
constexpr int SOLVE_BASE = 256;  // 128: 4.02 ms
// Inverses, ms, wavefront and blocked: n = 500 1.64, 1.67; 600 2.10, 2.19; 700 2.65, 2.55; 800 3.28,
// 2.92; 1000 4.98, 3.82; 2500 42.3, 14.7.
constexpr size_t INVERSE_BLOCKED_N = 672;
constexpr size_t SOLVE_BLOCKED_N = 512;
constexpr int SOLVE_UNEVEN = 1;  // of up to 31 sampled rows: a few scattered ones reach most tiles
struct BlockedSolve {
  la_ctx ctx;
  const double* A;
  size_t ld;
  double* X;
  size_t ldx;
  int nrhs;
  bool id;
  void* ws;
  size_t ws_bytes;

  static int middle(int r0, int r1) { return r0 + ((r1 - r0 + 1) / 2 + 63) / 64 * 64; }
  // The first nc columns of X[r0:r1] -= A[r0:r1, k0:k1] X[k0:k1].
  la_status update(int r0, int r1, int k0, int k1, int nc) {
    if (nc <= 0) return LA_OK;
    const double* a = A + (size_t)r0 * ld + k0;
    const double* x = X + (size_t)k0 * ldx;
    const la_status s = split_update(ctx, r1 - r0, nc, k1 - k0, a, ld, x, ldx, X + (size_t)r0 * ldx, ldx,
                                     ws, ws_bytes);
    if (s != LA_UNSUPPORTED) return s;
    return launch_gemm(ctx, GM_FMA_SUB, r1 - r0, nc, k1 - k0, a, ld, x, ldx, X + (size_t)r0 * ldx, ldx);
  }
  la_status block(bool upper, int r0, int r1, int nc) {
    return launch_tri_wave(ctx, false, upper, upper, A + (size_t)r0 * ld + r0, ld, X + (size_t)r0 * ldx,
                           ldx, r1 - r0, nc);
  }
  la_status lower(int r0, int r1) {
    if (r1 - r0 <= SOLVE_BASE) return block(false, r0, r1, id ? r1 : nrhs);
    const int mid = middle(r0, r1);
    LA_TRY(lower(r0, mid));
    if (!id) {
      LA_TRY(update(mid, r1, r0, mid, nrhs));
      return lower(mid, r1);
    }
    // The last 64 columns end in as many rows: their terms are an FMA product of K = 64. (Elements of
    // few terms do not fit the split product, and one such tile is a chain of all K: 590 us at K = 512.)
    const int c = mid - 64;
    LA_TRY(update(mid, r1, r0, mid, c));
    LA_TRY(launch_gemm_narrow(ctx, GM_FMA_SUB, r1 - mid, 64, 64, A + (size_t)mid * ld + c, ld,
                              X + (size_t)c * ldx + c, ldx, X + (size_t)mid * ldx + c, ldx));
    return lower(mid, r1);
  }
  la_status upper(int r0, int r1) {
    if (r1 - r0 <= SOLVE_BASE) return block(true, r0, r1, nrhs);
    const int mid = middle(r0, r1);
    LA_TRY(upper(mid, r1));
    LA_TRY(update(r0, mid, mid, r1, nrhs));
    return upper(r0, mid);
  }
};

struct FastLu {
  la_ctx ctx;
  double* A;
  size_t ld;
  int m, n, W;
  int* ipiv;
  void* ws;
  size_t ws_bytes;
  unsigned bar_base = 0;
  PhaseTimer t;

  FastLu(la_ctx c, la_lu h)
      : ctx(c), A(h->d_lu), ld(h->ld), m((int)h->m), n((int)h->n), W(std::min(32, c->panel_width)),
        ipiv(h->d_ipiv), ws(c->split_ws), ws_bytes(c->split_ws_bytes), t(c) {}

  double* at(int r, int c) { return A + (size_t)r * ld + c; }

  // C[r0:r1, c0:c1] -= A[r0:r1, k0:k1] A[k0:k1, c0:c1], in pieces of whole tiles that the
  // workspace takes.
  la_status update(int r0, int r1, int k0, int k1, int c0, int c1) {
    const int M = r1 - r0, N = c1 - c0, K = k1 - k0;
    if (M <= 0 || N <= 0) return LA_OK;
    if (ws && K >= 32 && (size_t)M * N >= SPLIT_MIN_MN) {
      const la_status s = split_update(ctx, M, N, K, at(r0, k0), ld, at(k0, c0), ld, at(r0, c0), ld, ws,
                                       ws_bytes);
      if (s != LA_UNSUPPORTED) return s;
    }
    if (N <= 64 && K <= 64)
      return launch_gemm_narrow(ctx, GM_FMA_SUB, M, N, K, at(r0, k0), ld, at(k0, c0), ld, at(r0, c0), ld);
    return launch_gemm(ctx, GM_FMA_SUB, M, N, K, at(r0, k0), ld, at(k0, c0), ld, at(r0, c0), ld);
  }

  // X = L11^-1 X, L11 the unit lower block of rows [r0, r1), X columns [c0, c1).
  la_status solve(int r0, int r1, int c0, int c1) {
    if (c1 <= c0) return LA_OK;
    if (r1 - r0 <= LU_BASE) return launch_trsm_rowpanel(ctx, false, A, nullptr, ld, r0, r1 - r0, c0, c1);
    const int mid = r0 + ((r1 - r0 + 1) / 2 + LU_BASE - 1) / LU_BASE * LU_BASE;
    LA_TRY(solve(r0, mid, c0, c1));
    LA_TRY(update(mid, r1, r0, mid, c0, c1));
    return solve(mid, r1, c0, c1);
  }

  // Columns [b0, b1), rows [b0, m).
  la_status factor(int b0, int b1) {
    if (b1 - b0 > LU_BASE) {
      const int mid = b0 + ((b1 - b0 + 1) / 2 + LU_BASE - 1) / LU_BASE * LU_BASE;
      LA_TRY(factor(b0, mid));
      size_t b = t.begin(ctx->stream);
      LA_TRY(solve(b0, mid, mid, b1));
      LA_TRY(update(mid, m, b0, mid, mid, b1));
      t.end(ctx->stream, b, PH_OTHER);
      return factor(mid, b1);
    }
    for (int j0 = b0, jb; j0 < b1; j0 += jb) {
      // The cooperative kernel takes the block in one piece (in halves, with the swaps, triangle and
      // update between them, 50000 x 64 took 845 us instead of 769, 9000 x 33 290 instead of 262).
      const bool cluster = ctx->cluster_panels && (ctx->panel_ctas == 0 || ctx->split_ws) &&
                           m - j0 <= PANEL64_ROWS;
      jb = std::min(cluster ? W : ctx->panel_width, b1 - j0);
      const int j1 = j0 + jb;
      size_t b = t.begin(ctx->stream);
      la_status s = LA_UNSUPPORTED;
      if (cluster)
        s = launch_panel_cluster64(ctx, ctx->stream, A, nullptr, ld, m, j0, jb, ipiv);
      if (s == LA_UNSUPPORTED)
        s = launch_panel(ctx, ctx->stream, false, A, nullptr, ld, m, j0, jb, ipiv, &bar_base);
      LA_TRY(s);
      t.end(ctx->stream, b, PH_PANEL);
      b = t.begin(ctx->stream);
      LA_TRY(launch_laswp(ctx, false, A, nullptr, ld, 0, n, j0, jb));
      t.end(ctx->stream, b, PH_SWAP);
      if (j1 < b1) {
        b = t.begin(ctx->stream);
        LA_TRY(solve(j0, j1, j1, b1));
        if (j1 < m)
          LA_TRY(launch_gemm_narrow(ctx, GM_FMA_SUB, m - j1, b1 - j1, jb, at(j1, j0), ld, at(j0, j1),
                                    ld, at(j1, j1), ld));
        t.end(ctx->stream, b, PH_OTHER);
      }
    }
    return LA_OK;
  }
};

la_status lu_fast_enqueue(la_ctx ctx, la_lu h, int* d_flags, int* d_uneven) {
  FastLu f(ctx, h);
  const int m = f.m, n = f.n, kmin = std::min(m, n);
  cudaStream_t st = ctx->stream;
  LA_CUDA(ctx, cudaMemsetAsync(ctx->d_bar, 0, sizeof(unsigned), st));
  // Digits of one update, kept for the whole factorization. Without memory for them the updates are
  // FMA products.
  DevBuf own(ctx);
  if (!f.ws && m > LU_BASE && n > LU_BASE) {
    const int nb = std::min(lu_block(m), kmin);
    f.ws_bytes = gemm_split_ws(m, n, nb, false);
    if (own.try_alloc(f.ws_bytes)) f.ws = own.p;
  }
  struct PdlScope {
    la_ctx c;
    ~PdlScope() { c->pdl_now = false; }
  } scope{ctx};
  ctx->pdl_now = ctx->pdl != 0 && !f.t.on;
  for (int b0 = 0; b0 < kmin;) {
    const int b1 = std::min(b0 + lu_block(m - b0), kmin);
    LA_TRY(f.factor(b0, b1));
    if (b1 < n) {
      size_t b = f.t.begin(st);
      LA_TRY(f.solve(b0, b1, b1, n));
      f.t.end(st, b, PH_TRSM);
      b = f.t.begin(st);
      LA_TRY(f.update(b1, m, b0, b1, b1, n));
      f.t.end(st, b, PH_GEMM);
    }
    b0 = b1;
  }
  ctx->pdl_now = false;
  size_t b = f.t.begin(st);
  LA_TRY(launch_lu_finish(ctx, h, d_flags, d_uneven));
  f.t.end(st, b, PH_OTHER);
  if (f.t.on) {
    LA_CUDA(ctx, cudaStreamSynchronize(st));
    f.t.finish();
  } else {
    for (int i = 0; i < 5; i++) ctx->phase_ms[i] = 0;
  }
  return LA_OK;
}

// EXACT factorization of h->d_lu in place.
//
// With lookahead (default), after panel p's row swaps and triangular update,
// the columns of panel p+1 get their trailing update first; panel p+1 is then
// factored on the high-priority side stream while the rest of panel p's
// trailing update runs on the main stream. The two touch disjoint columns:
// panel p+1 owns columns [j1, j2) of rows >= j1, the rest of the update writes
// columns >= j2 and reads L21 (columns < j1) and U12 (rows < j1).
}  // namespace

la_status lu_factor_enqueue(la_ctx ctx, la_lu h, int* d_flags, int* d_uneven) {
  if (h->arith != LA_ARITH_EXACT) return lu_fast_enqueue(ctx, h, d_flags, d_uneven);
  const int m = (int)h->m, n = (int)h->n;
  const size_t ld = h->ld;
  const int kmin = std::min(m, n);
  const int W = ctx->panel_width;
  const bool look = ctx->lookahead != 0;
  cudaStream_t ms = ctx->stream, ss = ctx->side_stream;
  double* A = h->d_lu;
  DevBuf S(ctx);
  LA_TRY(S.alloc((size_t)m * ld * sizeof(double)));
  LA_CUDA(ctx, cudaMemsetAsync(S.p, 0, (size_t)m * ld * sizeof(double), ms));
  LA_CUDA(ctx, cudaMemsetAsync(ctx->d_bar, 0, sizeof(unsigned), ms));
  unsigned bar_base = 0;
  PhaseTimer t(ctx);
  auto trailing = [&](int j0, int jb, int c0, int c1, size_t min_smem) -> la_status {
    // rows [j0+jb, m), columns [c0, c1)
    const int j1 = j0 + jb;
    if (j1 >= m || c1 <= c0) return LA_OK;
    size_t b = t.begin(ms);
    la_status st = launch_gemm(ctx, GM_EXACT_ADD, m - j1, c1 - c0, jb, A + (size_t)j1 * ld + j0, ld,
                               A + (size_t)j0 * ld + c0, ld, S.d() + (size_t)j1 * ld + c0, ld, min_smem);
    t.end(ms, b, PH_GEMM);
    return st;
  };

  // Panel [j0, j0 + jb) on stream s: in halves of 32 columns on one cluster, the swaps of each half
  // and the first half's triangular solve and carry on the panel's other columns between them (lists
  // 0 and 1 keep the halves' row moves for the other columns); where that cannot be, the cooperative
  // kernel in one piece. n = 1000: 69 us per half, 375 us for the cooperative 64 columns; the whole
  // factorization 8.2 -> 4.9 ms.
  int lists = 1;
  auto panel_kernels = [&](cudaStream_t s, int j0, int jb) -> la_status {
    const int h0 = std::min(jb, 32), jm = j0 + h0;
    ctx->swap_list = 0;
    la_status st = LA_UNSUPPORTED;
    if (ctx->cluster_panels && ctx->panel_ctas == 0)
      st = launch_panel_cluster64(ctx, s, A, S.d(), ld, m, j0, h0, h->d_ipiv);
    lists = 1;
    if (st == LA_UNSUPPORTED)
      return launch_panel(ctx, s, true, A, S.d(), ld, m, j0, jb, h->d_ipiv, &bar_base);
    LA_TRY(st);
    if (h0 == jb) return LA_OK;
    LA_TRY(launch_laswp(ctx, true, A, S.d(), ld, j0, j0 + jb, j0, h0));
    LA_TRY(launch_trsm_rowpanel(ctx, true, A, S.d(), ld, j0, h0, jm, j0 + jb));
    if (jm < m)
      LA_TRY(launch_gemm_narrow(ctx, GM_EXACT_ADD, m - jm, jb - h0, h0, A + (size_t)jm * ld + j0, ld,
                                A + (size_t)j0 * ld + jm, ld, S.d() + (size_t)jm * ld + jm, ld));
    ctx->swap_list = 1;
    LA_TRY(launch_panel_cluster64(ctx, s, A, S.d(), ld, m, jm, jb - h0, h->d_ipiv));
    lists = 2;
    return launch_laswp(ctx, true, A, S.d(), ld, j0, j0 + jb, jm, jb - h0);
  };
  auto panel = [&](cudaStream_t s, int j0, int jb) -> la_status {
    cudaStream_t saved = ctx->stream;
    ctx->stream = s;
    size_t b = t.begin(s);
    ctx->pdl_now = ctx->pdl != 0 && !t.on;
    const la_status st = panel_kernels(s, j0, jb);
    ctx->pdl_now = false;
    ctx->swap_list = 0;
    t.end(s, b, PH_PANEL);
    ctx->stream = saved;
    return st;
  };
  LA_TRY(panel(ms, 0, std::min(W, kmin)));
  for (int j0 = 0; j0 < kmin; j0 += W) {
    const int jb = std::min(W, kmin - j0);
    const int j1 = j0 + jb;
    size_t b = t.begin(ms);
    la_status sw = LA_OK;
    for (int l = 0; l < lists && sw == LA_OK; l++) {
      ctx->swap_list = l;
      sw = launch_laswp(ctx, true, A, S.d(), ld, 0, n, j0, jb);
    }
    ctx->swap_list = 0;
    LA_TRY(sw);
    t.end(ms, b, PH_SWAP);
    if (j1 < n) {
      b = t.begin(ms);
      LA_TRY(launch_trsm_rowpanel(ctx, true, A, S.d(), ld, j0, jb, j1, n));
      t.end(ms, b, PH_TRSM);
    }
    if (j1 >= kmin) break;  // no next panel
    const int jbn = std::min(W, kmin - j1);
    if (look) {
      LA_TRY(trailing(j0, jb, j1, j1 + jbn, 0));
      LA_CUDA(ctx, cudaEventRecord(ctx->ev_fork, ms));
      LA_CUDA(ctx, cudaStreamWaitEvent(ss, ctx->ev_fork, 0));
      LA_TRY(panel(ss, j1, jbn));
      LA_CUDA(ctx, cudaEventRecord(ctx->ev_join, ss));
      LA_TRY(trailing(j0, jb, j1 + jbn, n, GEMM_SMEM_WITH_PANEL));
      LA_CUDA(ctx, cudaStreamWaitEvent(ms, ctx->ev_join, 0));
    } else {
      LA_TRY(trailing(j0, jb, j1, n, 0));
      LA_TRY(panel(ms, j1, jbn));
    }
  }
  // m < n: the columns right of the last panel got their triangular update above.
  size_t b = t.begin(ms);
  LA_TRY(launch_lu_finish(ctx, h, d_flags, d_uneven));
  t.end(ms, b, PH_OTHER);
  if (t.on) {
    LA_CUDA(ctx, cudaStreamSynchronize(ms));
    t.finish();
  } else {
    for (int i = 0; i < 5; i++) ctx->phase_ms[i] = 0;
  }
  return LA_OK;
}

namespace {

la_status lu_factor(la_ctx ctx, la_lu h) {
  int* d_flags = reinterpret_cast<int*>(ctx->d_small);
  const bool look = h->arith == LA_ARITH_FAST && h->m == h->n && h->n >= SOLVE_BLOCKED_N;
  LA_TRY(lu_factor_enqueue(ctx, h, d_flags, look ? d_flags + 2 : nullptr));
  int* flags = static_cast<int*>(ctx->h_pinned);
  LA_CUDA(ctx, cudaMemcpyAsync(flags, d_flags, 3 * sizeof(int), cudaMemcpyDeviceToHost,
                               ctx->stream));
  LA_TRY(la_sync_and_check(ctx, "lu factorization"));
  h->pospivsign = flags[0];
  h->zero_diag = flags[1];
  if (look) h->uneven = flags[2];
  return LA_OK;
}

la_status lu_alloc(la_ctx ctx, size_t m, size_t n, la_lu* out) {
  if (m == 0 || n == 0) return LA_BADSHAPE;  // Matrix::new asserts (mod.rs:209)
  if (m > (size_t)INT32_MAX / 2 || n > (size_t)INT32_MAX / 2) return LA_UNSUPPORTED;
  la_lu h = new (std::nothrow) la_lu_handle();
  if (!h) return LA_NOMEM;
  h->ctx = ctx;
  h->m = m;
  h->n = n;
  h->ld = pad4(n);
  h->arith = ctx->arith;
  void* p = nullptr;
  la_status s = la_device_alloc(ctx, &p, m * h->ld * sizeof(double));
  if (s != LA_OK) { delete h; return s; }
  h->d_lu = static_cast<double*>(p);
  s = la_device_alloc(ctx, &p, std::min(m, n) * sizeof(int));
  if (s != LA_OK) { la_lu_free(h); return s; }
  h->d_ipiv = static_cast<int*>(p);
  s = la_device_alloc(ctx, &p, m * sizeof(uint64_t));
  if (s != LA_OK) { la_lu_free(h); return s; }
  h->d_piv = static_cast<uint64_t*>(p);
  *out = h;
  return LA_OK;
}

// is_non_singular (lu.rs:174-182) from the factorization's zero flag: a zero
// among U's first min(m,n) diagonal entries returns false first; with m < n the
// reference's index j*n+j leaves its data at j = m, which panics.
la_status lu_non_singular(la_lu h, int* out) {
  if (h->zero_diag) { *out = 0; return LA_OK; }
  if (h->m < h->n) return LA_BADSHAPE;
  *out = 1;
  return LA_OK;
}

// X (m x nrhs, pitch ldx) holds B(piv,:) on entry and the solution on exit
// (lu.rs:256-275; the loops run over the first n rows).
la_status lu_solve_inplace(la_ctx ctx, la_lu h, double* X, size_t ldx, int nrhs) {
  const int n = (int)h->n;
  // Where the blocked solve is the faster one. Device solve, us, wavefront and blocked: n = 512: 512
  // right-hand sides 439, 429; 1000: 751, 594. n = 1000: 256: 766, 922; 512: 1321, 959; 1000: 2466, 1299.
  // n = 2500: 192: 2835, 2922; 256: 3643, 2958. n = 6000: 64: 5497, 6553; 128: 10042, 6915; 1000: 74520,
  // 9991. Backward errors 4 to 10 times smaller. Without memory for the digits: the wavefront.
  // Where U's rows lie unevenly the products' tiles are FMA chains, and the blocked solve pays from 800000
  // on. Columns over 16 powers of ten: n = 512: 1000: 754, 728; n = 1000: 500: 1293, 1376; 1000: 2468, 1989;
  // n = 4096: 128: 4885, 6006; 256: 9182, 7316. Banded: n = 512: 1000: 754, 823; 1500: 1083, 1042; n = 1000:
  // 500: 1292, 1506; 1000: 2471, 2156; n = 6000: 128: 10071, 11817; 256: 19407, 12227.
  const long long elements = (long long)n * nrhs;
  if (h->arith == LA_ARITH_FAST && ctx->solve_wave > 0 && !ctx->split_ws && n >= (int)SOLVE_BLOCKED_N &&
      nrhs >= 64 && elements >= (h->uneven <= SOLVE_UNEVEN ? 500000 : 800000)) {
    const int half = BlockedSolve::middle(0, n);
    DevBuf ws(ctx);
    const size_t bytes = gemm_split_ws(half, nrhs, half, false);
    if (bytes <= SPLIT_WS_MAX && ws.try_alloc(bytes)) {
      BlockedSolve s{ctx, h->d_lu, h->ld, X, ldx, nrhs, false, ws.p, bytes};
      LA_TRY(s.lower(0, n));
      return s.upper(0, n);
    }
  }
  return launch_lu_solve(ctx, h->arith == LA_ARITH_EXACT, h->d_lu, h->ld, X, ldx, n, nrhs);
}

la_status check_ctx(la_ctx ctx) {
  if (!ctx) return LA_INVALID;
  cudaError_t e = cudaSetDevice(ctx->device);
  if (e != cudaSuccess) return la_cuda_fail(ctx, e, "cudaSetDevice");
  return LA_OK;
}

// Device solve shared by the host and device entry points: d_b (pitch ldb) ->
// d_x (pitch ldx); both may be unaligned, an aligned work buffer is used.
la_status solve_device_common(la_lu h, const double* d_b, size_t ldb, size_t brows, size_t nrhs,
                              double* d_x, size_t ldx) {
  la_ctx ctx = h->ctx;
  if (brows != h->m) return LA_BADSHAPE;  // lu.rs:240
  if (nrhs == 0) return LA_BADSHAPE;      // Matrix::new asserts cols > 0
  int ns = 0;
  LA_TRY(lu_non_singular(h, &ns));        // lu.rs:241
  if (!ns) return LA_SINGULAR;
  const size_t ldw = pad4(nrhs);
  DevBuf Xw(ctx);
  LA_TRY(Xw.alloc(h->m * ldw * sizeof(double)));
  LA_TRY(launch_permute_rows(ctx, h->d_piv, d_b, ldb, Xw.d(), ldw, (int)h->m, (int)nrhs));
  LA_TRY(lu_solve_inplace(ctx, h, Xw.d(), ldw, (int)nrhs));
  LA_CUDA(ctx, cudaMemcpy2DAsync(d_x, ldx * sizeof(double), Xw.d(), ldw * sizeof(double),
                                 nrhs * sizeof(double), h->m, cudaMemcpyDeviceToDevice,
                                 ctx->stream));
  return LA_OK;
}

la_status gemm_device_common(la_ctx ctx, const double* d_a, size_t lda, const double* d_b,
                             size_t ldb, double* d_c, size_t ldc, size_t m, size_t k, size_t n) {
  const int mode = ctx->arith == LA_ARITH_EXACT ? GM_EXACT_ZERO : GM_FMA_ZERO;
  if (mode == GM_FMA_ZERO && n > 16 && k >= 32) {
    // On the tensor cores from 32 k and 17 columns on: one FMA tile of 64 x 64 x 32 keeps an SM busy
    // for 33 us, while the split product's three launches of one tile take about 15 us in all
    // (8192^3: 24.0 ms against 876 ms). In slabs of K whose digits fit the workspace and whose sums fit
    // the product's integers (2 x 1048736 x 17: 61 ms, as one FMA tile 1048).
    const size_t kc = std::min<size_t>(
        SPLIT_MAX_K, std::max<size_t>(128, SPLIT_WS_MAX / (16 * (m + n)) / 128 * 128));
    DevBuf ws(ctx);
    const size_t bytes = gemm_split_ws((int)m, (int)n, (int)std::min(k, kc), false);
    if (bytes <= 2 * SPLIT_WS_MAX && ws.try_alloc(bytes)) {
      la_status s = LA_OK;
      for (size_t k0 = 0; k0 < k && s == LA_OK; k0 += kc)
        s = launch_gemm_split(ctx, ctx->stream, k0 ? 1 : 0, (int)m, (int)n,
                              (int)std::min(kc, k - k0), d_a + k0, lda, d_b + k0 * ldb, ldb, false,
                              d_c, ldc, false, ws.p, bytes);
      if (s != LA_UNSUPPORTED) return s;
    }
  }
  DevBuf a2(ctx), b2(ctx), c2(ctx);
  const double* A = d_a;
  const double* B = d_b;
  double* C = d_c;
  size_t la = lda, lb = ldb, lc = ldc;
  if (!aligned16(d_a, lda)) {
    la = pad4(k);
    LA_TRY(a2.alloc(m * la * sizeof(double)));
    LA_CUDA(ctx, cudaMemcpy2DAsync(a2.p, la * 8, d_a, lda * 8, k * 8, m, cudaMemcpyDeviceToDevice,
                                   ctx->stream));
    A = a2.d();
  }
  if (!aligned16(d_b, ldb)) {
    lb = pad4(n);
    LA_TRY(b2.alloc(k * lb * sizeof(double)));
    LA_CUDA(ctx, cudaMemcpy2DAsync(b2.p, lb * 8, d_b, ldb * 8, n * 8, k, cudaMemcpyDeviceToDevice,
                                   ctx->stream));
    B = b2.d();
  }
  if (!aligned16(d_c, ldc)) {
    lc = pad4(n);
    LA_TRY(c2.alloc(m * lc * sizeof(double)));
    C = c2.d();
  }
  LA_TRY(launch_gemm(ctx, mode, (int)m, (int)n, (int)k, A, la, B, lb, C, lc));
  if (C != d_c)
    LA_CUDA(ctx, cudaMemcpy2DAsync(d_c, ldc * 8, C, lc * 8, n * 8, m, cudaMemcpyDeviceToDevice,
                                   ctx->stream));
  return LA_OK;
}

la_status fetch(la_ctx ctx, void* host, const void* dev, size_t bytes) {
  LA_CUDA(ctx, cudaMemcpyAsync(host, dev, bytes, cudaMemcpyDeviceToHost, ctx->stream));
  return la_sync_and_check(ctx, "readback");
}

}  // namespace

extern "C" {

la_status la_lu_new(la_ctx ctx, const double* a, size_t m, size_t n, la_lu* out) {
  LA_TRY(check_ctx(ctx));
  if (!a || !out) return LA_INVALID;
  *out = nullptr;
  la_lu h = nullptr;
  LA_TRY(lu_alloc(ctx, m, n, &h));
  la_status s = LA_OK;
  s = la_copy_to_device(ctx, h->d_lu, h->ld, a, m, n);
  if (s == LA_OK) s = lu_factor(ctx, h);
  if (s != LA_OK) { la_lu_free(h); return s; }
  *out = h;
  return LA_OK;
}

la_status la_lu_new_device(la_ctx ctx, const double* d_a, size_t lda, size_t m, size_t n,
                           la_lu* out) {
  LA_TRY(check_ctx(ctx));
  if (!d_a || !out || lda < n) return LA_INVALID;
  *out = nullptr;
  la_lu h = nullptr;
  LA_TRY(lu_alloc(ctx, m, n, &h));
  la_status s = LA_OK;
  cudaError_t e = cudaMemcpy2DAsync(h->d_lu, h->ld * sizeof(double), d_a, lda * sizeof(double),
                                    n * sizeof(double), m, cudaMemcpyDeviceToDevice, ctx->stream);
  if (e != cudaSuccess) s = la_cuda_fail(ctx, e, "copy A on device");
  if (s == LA_OK) s = lu_factor(ctx, h);
  if (s != LA_OK) { la_lu_free(h); return s; }
  *out = h;
  return LA_OK;
}

void la_lu_free(la_lu h) {
  if (!h) return;
  la_ctx ctx = h->ctx;
  cudaSetDevice(ctx->device);
  la_device_free(ctx, h->d_lu);
  la_device_free(ctx, h->d_lu32);
  la_device_free(ctx, h->d_dinv);
  la_device_free(ctx, h->d_dinvf);
  la_device_free(ctx, h->d_ipiv);
  la_device_free(ctx, h->d_piv);
  delete h;
}

la_status la_lu_shape(la_lu h, size_t* m, size_t* n) {
  if (!h) return LA_INVALID;
  if (m) *m = h->m;
  if (n) *n = h->n;
  return LA_OK;
}

la_status la_lu_is_non_singular(la_lu h, int* out) {
  if (!h || !out) return LA_INVALID;
  return lu_non_singular(h, out);
}

la_status la_lu_det(la_lu h, double* out) {
  if (!h || !out) return LA_INVALID;
  la_ctx ctx = h->ctx;
  LA_TRY(check_ctx(ctx));
  if (h->m != h->n) return LA_BADSHAPE;  // lu.rs:225
  LA_TRY(launch_det(ctx, h->d_lu, h->ld, (int)h->n, h->pospivsign, ctx->d_small + 2));
  double* hp = static_cast<double*>(ctx->h_pinned);
  LA_TRY(fetch(ctx, hp, ctx->d_small + 2, sizeof(double)));
  *out = hp[0];
  return LA_OK;
}

la_status la_lu_get_piv(la_lu h, uint64_t* piv, int* pospivsign) {
  if (!h) return LA_INVALID;
  if (pospivsign) *pospivsign = h->pospivsign;
  if (piv) {
    LA_TRY(check_ctx(h->ctx));
    LA_TRY(fetch(h->ctx, piv, h->d_piv, h->m * sizeof(uint64_t)));
  }
  return LA_OK;
}

static la_status get_unpacked(la_lu h, int which, double* out) {
  if (!h || !out) return LA_INVALID;
  la_ctx ctx = h->ctx;
  LA_TRY(check_ctx(ctx));
  const size_t kmin = std::min(h->m, h->n);
  size_t rows = which == 0 ? h->m : which == 1 ? kmin : h->m;
  size_t cols = which == 0 ? kmin : which == 1 ? h->n : which == 2 ? h->m : h->n;
  DevBuf tmp(ctx);
  LA_TRY(tmp.alloc(rows * cols * sizeof(double)));
  LA_TRY(launch_unpack(ctx, which, h->d_lu, h->ld, (int)h->m, (int)h->n, h->d_piv, tmp.d()));
  return fetch(ctx, out, tmp.p, rows * cols * sizeof(double));
}

la_status la_lu_get_l(la_lu h, double* out) { return get_unpacked(h, 0, out); }
la_status la_lu_get_u(la_lu h, double* out) { return get_unpacked(h, 1, out); }
la_status la_lu_get_p(la_lu h, double* out) { return get_unpacked(h, 2, out); }
la_status la_lu_get_packed(la_lu h, double* out) { return get_unpacked(h, 3, out); }

const double* la_lu_device_data(la_lu h, size_t* ld) {
  if (!h) return nullptr;
  if (ld) *ld = h->ld;
  return h->d_lu;
}

la_status la_lu_solve(la_lu h, const double* b, size_t brows, size_t nrhs, double* x) {
  if (!h || !b || !x) return LA_INVALID;
  la_ctx ctx = h->ctx;
  LA_TRY(check_ctx(ctx));
  if (brows != h->m) return LA_BADSHAPE;
  if (nrhs == 0) return LA_BADSHAPE;
  int ns = 0;
  LA_TRY(lu_non_singular(h, &ns));
  if (!ns) return LA_SINGULAR;
  const size_t ldw = pad4(nrhs);
  DevBuf Bd(ctx), Xw(ctx);
  LA_TRY(Bd.alloc(h->m * nrhs * sizeof(double)));
  LA_TRY(Xw.alloc(h->m * ldw * sizeof(double)));
  LA_CUDA(ctx, cudaMemcpyAsync(Bd.p, b, h->m * nrhs * sizeof(double), cudaMemcpyHostToDevice,
                               ctx->stream));
  LA_TRY(launch_permute_rows(ctx, h->d_piv, Bd.d(), nrhs, Xw.d(), ldw, (int)h->m, (int)nrhs));
  LA_TRY(lu_solve_inplace(ctx, h, Xw.d(), ldw, (int)nrhs));
  LA_TRY(la_copy_to_host(ctx, x, Xw.d(), ldw, h->m, nrhs));
  return la_sync_and_check(ctx, "lu solve");
}

la_status la_lu_solve_device(la_lu h, const double* d_b, size_t ldb, size_t brows, size_t nrhs,
                             double* d_x, size_t ldx) {
  if (!h || !d_b || !d_x || ldb < nrhs || ldx < nrhs) return LA_INVALID;
  LA_TRY(check_ctx(h->ctx));
  return solve_device_common(h, d_b, ldb, brows, nrhs, d_x, ldx);
}

la_status la_matrix_det(la_ctx ctx, const double* a, size_t m, size_t n, double* out) {
  if (!a || !out) return LA_INVALID;
  if (m != n) return LA_BADSHAPE;  // mod.rs:1026
  la_lu h = nullptr;
  LA_TRY(la_lu_new(ctx, a, m, n, &h));
  la_status s = la_lu_det(h, out);
  la_lu_free(h);
  return s;
}

la_status la_matrix_solve(la_ctx ctx, const double* a, size_t m, size_t n, const double* b,
                          size_t brows, size_t nrhs, double* x) {
  if (!a || !b || !x) return LA_INVALID;
  la_lu h = nullptr;
  LA_TRY(la_lu_new(ctx, a, m, n, &h));
  la_status s = la_lu_solve(h, b, brows, nrhs, x);
  la_lu_free(h);
  return s;
}

la_status la_matrix_inverse(la_ctx ctx, const double* a, size_t m, size_t n, double* out) {
  if (!a || !out) return LA_INVALID;
  if (m != n) return LA_BADSHAPE;  // mod.rs:1035
  la_lu h = nullptr;
  LA_TRY(la_lu_new(ctx, a, m, n, &h));
  la_status s = LA_OK;
  int ns = 0;
  s = lu_non_singular(h, &ns);
  if (s == LA_OK && !ns) s = LA_SINGULAR;
  if (s == LA_OK) {
    const size_t ldw = pad4(n);
    DevBuf Xw(ctx);
    s = Xw.alloc(n * ldw * sizeof(double));
    // U^-1 L^-1 by blocks, then the columns in their order: A^-1 = (LU)^-1 P.
    DevBuf ws(ctx);
    const double* inv = Xw.d();
    if (s == LA_OK && h->arith == LA_ARITH_FAST && ctx->solve_wave > 0 && n >= INVERSE_BLOCKED_N) {
      const int half = BlockedSolve::middle(0, (int)n);
      const size_t bytes = std::max(gemm_split_ws(half, (int)n, half, false), n * ldw * sizeof(double));
      if (bytes <= SPLIT_WS_MAX && ws.try_alloc(bytes)) {
        BlockedSolve b{ctx, h->d_lu, h->ld, Xw.d(), ldw, (int)n, true, ws.p, bytes};
        s = launch_identity_permuted(ctx, nullptr, Xw.d(), ldw, (int)n);
        if (s == LA_OK) s = b.lower(0, (int)n);
        if (s == LA_OK) s = b.upper(0, (int)n);
        if (s == LA_OK) s = launch_permute_cols(ctx, h->d_piv, Xw.d(), ws.d(), ldw, (int)n);
        inv = ws.d();
      }
    }
    if (inv == Xw.d()) {
      if (s == LA_OK) s = launch_identity_permuted(ctx, h->d_piv, Xw.d(), ldw, (int)n);
      if (s == LA_OK) s = lu_solve_inplace(ctx, h, Xw.d(), ldw, (int)n);
    }
    if (s == LA_OK) s = la_copy_to_host(ctx, out, inv, ldw, n, n);
    if (s == LA_OK) s = la_sync_and_check(ctx, "inverse");
  }
  la_lu_free(h);
  return s;
}

la_status la_matrix_is_non_singular(la_ctx ctx, const double* a, size_t m, size_t n, int* out) {
  if (!a || !out) return LA_INVALID;
  if (m != n) return LA_BADSHAPE;  // mod.rs:1045
  la_lu h = nullptr;
  LA_TRY(la_lu_new(ctx, a, m, n, &h));
  la_status s = lu_non_singular(h, out);
  la_lu_free(h);
  return s;
}

la_status la_matrix_mul(la_ctx ctx, const double* a, size_t m, size_t k, const double* b,
                        size_t brows, size_t n, double* c) {
  LA_TRY(check_ctx(ctx));
  if (!a || !b || !c) return LA_INVALID;
  if (m == 0 || k == 0 || brows == 0 || n == 0) return LA_BADSHAPE;
  if (k != brows) return LA_BADSHAPE;  // mod.rs:961
  if (m > INT32_MAX || n > INT32_MAX || k > INT32_MAX) return LA_UNSUPPORTED;
  const size_t la = pad4(k), lb = pad4(n), lc = pad4(n);
  DevBuf A(ctx), B(ctx), C(ctx);
  LA_TRY(A.alloc(m * la * sizeof(double)));
  LA_TRY(B.alloc(k * lb * sizeof(double)));
  LA_TRY(C.alloc(m * lc * sizeof(double)));
  LA_TRY(la_copy_to_device(ctx, A.d(), la, a, m, k));
  LA_TRY(la_copy_to_device(ctx, B.d(), lb, b, k, n));
  LA_TRY(gemm_device_common(ctx, A.d(), la, B.d(), lb, C.d(), lc, m, k, n));
  LA_TRY(la_copy_to_host(ctx, c, C.d(), lc, m, n));
  return la_sync_and_check(ctx, "matrix mul");
}

la_status la_matrix_mmul(la_ctx ctx, const double* a, size_t m, size_t k, const double* b,
                         size_t brows, size_t n, double* dst, size_t dst_rows, size_t dst_cols) {
  if (k != brows) return LA_BADSHAPE;                    // mmatrix.rs:83
  if (dst_rows != m || dst_cols != n) return LA_BADSHAPE;  // mmatrix.rs:84-85
  return la_matrix_mul(ctx, a, m, k, b, brows, n, dst);
}

la_status la_matrix_mul_device(la_ctx ctx, const double* d_a, size_t lda, const double* d_b,
                               size_t ldb, double* d_c, size_t ldc, size_t m, size_t k, size_t n) {
  LA_TRY(check_ctx(ctx));
  if (!d_a || !d_b || !d_c || lda < k || ldb < n || ldc < n) return LA_INVALID;
  if (m == 0 || k == 0 || n == 0) return LA_BADSHAPE;
  if (m > INT32_MAX || n > INT32_MAX || k > INT32_MAX) return LA_UNSUPPORTED;
  return gemm_device_common(ctx, d_a, lda, d_b, ldb, d_c, ldc, m, k, n);
}

}  // extern "C"
