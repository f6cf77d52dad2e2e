// Cholesky decomposition of a symmetric positive definite matrix
// (CholeskyDecomposition, src/decomp/cholesky.rs:56-145): A = L L'.
//
// The reference computes L one row at a time (cholesky.rs:64-107): for row j
// and k < j, L[j][k] = (A[j][k] - s) / L[k][k] with s the sum of
// L[k][i] L[j][i] over i < k, added in ascending i; the diagonal
// L[j][j] = sqrt(A[j][j] - d) with d the sum of L[j][k]^2 in ascending k. It
// returns None for a non-square matrix, at the first pair with
// A[k][j] != A[j][k], or at the first d <= 0.
//
// Here the same values come from blocked right-looking forms (no pivoting, so every panel step is
// known in advance). chol_sym_check_kernel first compares every strictly lower entry with its
// upper twin (the reference's '!=', so NaN fails), before anything is written.
//
// FAST (chol_fast_factor): panels of 32 columns. chol_panel32_kernel factors the 32 x 32 diagonal
// block in every CTA (a 64 x 64 block would keep one SM's FP64 pipe busy for 22 us; 32 x 32 takes 3)
// and solves the rows below; blocks of 64, 128 and 256 columns are a left half, its update of the
// right half's columns, and the right half; the trailing update A22 -= L21 L21' covers the tiles at
// or below the diagonal. Updates with K >= 64 run on the tensor cores by exact splitting
// (gemm_split.cu; L21 is split once, as both operands), the K = 32 ones by FMA.
//
// EXACT: 64-column panels, chol_diag_kernel on one CTA, chol_panel_kernel for the rows below (a
// thread per row), and the trailing update over row strips, each only up to its own diagonal. It
// keeps, per element, the running sum s in a second array S, adds products unfused in ascending i
// (the GEMM's EXACT_ADD mode, then the panel kernels) and forms (A - s) / L[k][k] and sqrt(A - d)
// exactly as the reference does, so L is bit-identical to it.
// A None result is reported after the whole factorization: the reference stops
// at the first failing row, and every such row fails here too.
#include "la_internal.cuh"

struct la_chol_handle {
  la_ctx ctx = nullptr;
  size_t n = 0, ld = 0;
  double* d_l = nullptr;   // L, n x n with pitch ld, zeros above the diagonal
  double* d_lt = nullptr;  // L' (built on the first FAST solve)
  int arith = LA_ARITH_FAST;
};

namespace {

constexpr int CHW = 64;   // panel width
constexpr int CHP = CHW + 1;
constexpr int PANEL_T = 64;  // two warps per CTA: rows spread over more SMs

size_t pad4c(size_t x) { return (x + 3) & ~size_t(3); }

struct Buf {
  la_ctx ctx;
  void* p = nullptr;
  explicit Buf(la_ctx c) : ctx(c) {}
  ~Buf() { la_device_free(ctx, p); }
  la_status alloc(size_t bytes) { return la_device_alloc(ctx, &p, bytes); }
  bool try_alloc(size_t bytes) { return la_device_try_alloc(ctx, &p, bytes); }
  double* d() { return static_cast<double*>(p); }
};

// flags[0] |= 1 when some strictly lower entry differs from its upper twin
// (cholesky.rs:89-91). One 32 x 32 tile pair per CTA, lower tiles only.
__global__ void chol_sym_check_kernel(const double* __restrict__ A, size_t ld, int n, int* flags) {
  __shared__ double t[32][33];
  const int bi = blockIdx.y, bj = blockIdx.x;
  if (bj > bi) return;
  const int tx = threadIdx.x, ty = threadIdx.y;  // 32 x 8
  // t[c][r] = A[bj*32 + r][bi*32 + c]: the upper twin tile, transposed
  for (int r = ty; r < 32; r += 8) {
    const int gr = bj * 32 + r, gc = bi * 32 + tx;
    t[tx][r] = (gr < n && gc < n) ? A[(size_t)gr * ld + gc] : 0.0;
  }
  __syncthreads();
  int bad = 0;
  for (int r = ty; r < 32; r += 8) {
    const int gr = bi * 32 + r, gc = bj * 32 + tx;
    if (gr < n && gc < n && gr > gc && A[(size_t)gr * ld + gc] != t[r][tx]) bad = 1;
  }
  if (__syncthreads_or(bad) && tx == 0 && ty == 0) atomicOr(flags, 1);
}

// Diagonal block [j0, j0 + jb)^2 on one CTA (lower part, diagonal included).
// flags[1] |= 1 at a non-positive d (cholesky.rs:97-100; NaN is not <= 0).
__global__ void __launch_bounds__(256)
chol_diag_kernel(double* L, double* S, size_t ld, int j0, int jb, int* flags) {
  extern __shared__ __align__(16) double chd_raw[];
  double(*a)[CHP] = reinterpret_cast<double(*)[CHP]>(chd_raw);
  double(*s)[CHP] = reinterpret_cast<double(*)[CHP]>(chd_raw + CHW * CHP);
  const int tid = threadIdx.x;
  for (int idx = tid; idx < jb * jb; idx += 256) {
    const int r = idx / jb, c = idx % jb;
    if (c <= r) {
      a[r][c] = L[(size_t)(j0 + r) * ld + j0 + c];
      s[r][c] = S[(size_t)(j0 + r) * ld + j0 + c];
    }
  }
  __syncthreads();
  for (int k = 0; k < jb; k++) {
    if (tid == 0) {
      const double d = __dsub_rn(a[k][k], s[k][k]);  // :96
      if (d <= 0.0) atomicOr(flags + 1, 1);
      a[k][k] = sqrt(d);  // :101
    }
    __syncthreads();
    const double dk = a[k][k];
    for (int r = k + 1 + tid; r < jb; r += 256)
      a[r][k] = __dsub_rn(a[r][k], s[r][k]) / dk;  // :82
    __syncthreads();
    const int m = jb - k - 1;
    for (int idx = tid; idx < m * m; idx += 256) {
      const int r = k + 1 + idx / m, c = k + 1 + idx % m;
      if (c > r) continue;
      s[r][c] = __dadd_rn(s[r][c], __dmul_rn(a[r][k], a[c][k]));  // :78, :86
    }
    __syncthreads();
  }
  for (int idx = tid; idx < jb * jb; idx += 256) {
    const int r = idx / jb, c = idx % jb;
    if (c <= r) L[(size_t)(j0 + r) * ld + j0 + c] = a[r][c];
  }
}

// FAST panel: columns [j0, j0 + jb), jb <= 32, of rows [j0, n). Every CTA factors the diagonal block
// (written to diag by CTA 0: other CTAs may still be reading the original, so it goes to L after
// everything else), then solves its own rows below it.
//   Diagonal block (warps 0-3): lane = row, warp w the columns c = w mod 4 in registers, so that all
//   four FP64 pipes take part. Column k is scaled by 1/sqrt(d) in its warp and passed on through
//   shared memory; the square roots themselves are taken at the end, all at once. The chain of 32
//   reciprocal square roots (a dozen dependent FP64 instructions each) bounds the kernel.
//   Rows (warps 4-7, 32 rows): 4 neighbouring lanes per row, lane q the columns c = q mod 4; x_k goes
//   to the other three by a shuffle. An FMA instruction takes a sub-partition 64 clocks however few
//   lanes it has, so a thread per row would need 496 x 64 clocks where this needs a quarter. They
//   take column k while warps 0-3 work on column k + 1. Further rows of the CTA follow on all 8 warps.
constexpr int CB = 32;
constexpr int CB_T = 256;

// One step of 4 lanes per row: v *= 1/L[k][k] in the lane of column k, then the columns after it.
__device__ __forceinline__ void row_step(double (&v)[CB / 4], int k, int q, int lane,
                                         const double (&dg)[CB][CB + 1], double rd) {
  if (q == k % 4) v[k / 4] *= rd;
  const double x = __shfl_sync(0xffffffffu, v[k / 4], lane / 4 * 4 + k % 4);
#pragma unroll
  for (int i = k / 4; i < CB / 4; i++)
    if (4 * i + 3 > k && q + 4 * i > k) v[i] = fma(-x, dg[k][(q + 4 * i) % CB], v[i]);
}

__global__ void __launch_bounds__(CB_T)
chol_panel32_kernel(double* L, size_t ld, int j0, int jb, int n, int rpc, double* diag,
                    int* flags) {
  la_pdl_wait();
  la_pdl_trigger();
  __shared__ double dg[CB][CB + 1];  // the factored block, column by column: dg[k][r] = L[r][k]
  __shared__ double rdg[CB], dd[CB];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, q = lane & 3;
  constexpr int NV = CB / 4;
  const int rb = j0 + CB + blockIdx.x * rpc, re = min(n, rb + rpc);
  double v[NV];
  const int r1 = rb + (tid - CB_T / 2) / 4;  // warps 4-7: this thread's row
  double* row = L + (size_t)(warp >= 4 && r1 < re ? r1 : j0) * ld + j0 + q;
  if (warp < 4) {
    const double* src = L + (size_t)(j0 + lane) * ld + j0 + warp;
#pragma unroll
    for (int i = 0; i < NV; i++)
      v[i] = lane < jb && warp + 4 * i <= lane ? src[4 * i] : 0.0;
  } else {
#pragma unroll
    for (int i = 0; i < NV; i++) v[i] = r1 < re ? row[4 * i] : 0.0;
  }
#pragma unroll
  for (int k = 0; k < CB; k++) {
    if (k >= jb) break;
    if (warp == k % 4) {
      const double d = __shfl_sync(0xffffffffu, v[k / 4], k);
      const double rq = rsqrt(d);
      v[k / 4] *= rq;
      dg[k][lane] = v[k / 4];
      if (lane == k) {
        rdg[k] = rq;
        dd[k] = d;
      }
    }
    __syncthreads();
    if (warp < 4) {
      const double l = dg[k][lane];
#pragma unroll
      for (int i = k / 4; i < NV; i++)
        if (4 * i + 3 > k && warp + 4 * i > k) v[i] = fma(-l, dg[k][(warp + 4 * i) % CB], v[i]);
    } else {
      row_step(v, k, q, lane, dg, rdg[k]);
    }
  }
  if (warp >= 4) {
    if (r1 < re)
#pragma unroll
      for (int i = 0; i < NV; i++) row[4 * i] = v[i];
  } else if (blockIdx.x == 0) {
    if (warp == 0 && lane < jb) {
      if (dd[lane] <= 0.0) atomicOr(flags + 1, 1);  // cholesky.rs:97-100
      diag[lane * (CB + 1)] = sqrt(dd[lane]);
    }
    for (int idx = tid; idx < CB * CB; idx += CB_T / 2)
      if (idx / CB != idx % CB) diag[idx] = dg[idx % CB][idx / CB];  // [r][k]
  }
  for (int r0 = rb + CB; r0 < re; r0 += CB_T / 4) {
    const int r = r0 + tid / 4;
    row = L + (size_t)(r < re ? r : j0) * ld + j0 + q;
#pragma unroll
    for (int i = 0; i < NV; i++) v[i] = r < re ? row[4 * i] : 0.0;
#pragma unroll
    for (int k = 0; k < CB; k++) row_step(v, k, q, lane, dg, rdg[k]);
    if (r < re)
#pragma unroll
      for (int i = 0; i < NV; i++) row[4 * i] = v[i];
  }
}

// C[r][c] -= sum_k L[r][j0 + k] L[c0 + c][j0 + k], k < 32, for rows [c0, n) and columns [c0, c0 + 32)
// (the second half of a 64-column block): 16 rows per CTA, thread (column, 2 rows).
constexpr int CU_T = 256, CU_R = 16;
__global__ void __launch_bounds__(CU_T)
chol_update32_kernel(double* L, size_t ld, int j0, int c0, int nc, int n) {
  la_pdl_wait();
  la_pdl_trigger();
  __shared__ double bt[CB][CB + 1], at[CB][CU_R + 1];
  const int tid = threadIdx.x, c = tid & 31, g = tid >> 5;
  const int rb = c0 + blockIdx.x * CU_R;
  for (int idx = tid; idx < CB * CB; idx += CU_T) {
    const int r = idx / CB, k = idx % CB;
    bt[k][r] = r < nc ? L[(size_t)(c0 + r) * ld + j0 + k] : 0.0;
  }
  for (int idx = tid; idx < CU_R * CB; idx += CU_T) {
    const int r = idx / CB, k = idx % CB;
    at[k][r] = rb + r < n ? L[(size_t)(rb + r) * ld + j0 + k] : 0.0;
  }
  const int r0 = rb + g, r1 = rb + g + 8;
  const bool in = c < nc;
  double a0 = in && r0 < n ? L[(size_t)r0 * ld + c0 + c] : 0.0;
  double a1 = in && r1 < n ? L[(size_t)r1 * ld + c0 + c] : 0.0;
  __syncthreads();
#pragma unroll 8
  for (int k = 0; k < CB; k++) {
    a0 = fma(-at[k][g], bt[k][c], a0);
    a1 = fma(-at[k][g + 8], bt[k][c], a1);
  }
  if (in && r0 < n) L[(size_t)r0 * ld + c0 + c] = a0;
  if (in && r1 < n) L[(size_t)r1 * ld + c0 + c] = a1;
}

// EXACT rows [r0, n) of the panel's columns [j0, j0 + 64): one thread per row, the row's sums s in
// registers, the finished diagonal block broadcast from shared memory. Only a full-width panel has
// rows below it (a narrower one is the last), so the width is fixed.
__global__ void __launch_bounds__(PANEL_T)
chol_panel_kernel(double* L, const double* S, size_t ld, int j0, int r0, int n) {
  __shared__ double dg[CHW][CHP];
  for (int idx = threadIdx.x; idx < CHW * CHW; idx += PANEL_T) {
    const int r = idx / CHW, c = idx % CHW;
    if (c <= r) dg[r][c] = L[(size_t)(j0 + r) * ld + j0 + c];
  }
  __syncthreads();
  const int r = r0 + blockIdx.x * PANEL_T + threadIdx.x;
  if (r >= n) return;
  double* row = L + (size_t)r * ld + j0;
  double v[CHW];
#pragma unroll
  for (int c = 0; c < CHW; c++) v[c] = S[(size_t)r * ld + j0 + c];
#pragma unroll
  for (int k = 0; k < CHW; k++) {
    const double x = __dsub_rn(row[k], v[k]) / dg[k][k];  // :82
    row[k] = x;
#pragma unroll
    for (int c = k + 1; c < CHW; c++) v[c] = __dadd_rn(v[c], __dmul_rn(x, dg[c][k]));
  }
}

// T[k][c] = L[r0 + c][j0 + k]: the panel's rows below the diagonal block,
// transposed, as the GEMM's K x N operand.
__global__ void chol_transpose_kernel(const double* __restrict__ L, size_t ld, int j0, int jb,
                                      int r0, int ncols, double* T, size_t ldt) {
  __shared__ double t[32][33];
  const int c0 = blockIdx.x * 32, k0 = blockIdx.y * 32;
  const int tx = threadIdx.x, ty = threadIdx.y;
  for (int i = ty; i < 32; i += 8) {
    const int c = c0 + i, k = k0 + tx;
    t[i][tx] = (c < ncols && k < jb) ? L[(size_t)(r0 + c) * ld + j0 + k] : 0.0;
  }
  __syncthreads();
  for (int i = ty; i < 32; i += 8) {
    const int k = k0 + i, c = c0 + tx;
    if (k < jb && c < ncols) T[(size_t)k * ldt + c] = t[tx][i];
  }
}

// L[r][c] = 0 for c > r (cholesky.rs:104-106); in FAST the 32 x 32 diagonal blocks from diag.
__global__ void chol_zero_upper_kernel(double* L, size_t ld, int n, const double* diag) {
  la_pdl_wait();
  const int bi = blockIdx.y, bj = blockIdx.x;
  if (bj < bi) return;
  if (diag && bi == bj) {
    for (int r = threadIdx.y; r < 32 && bi * 32 + r < n; r += 8) {
      const int c = threadIdx.x;
      if (bi * 32 + c < n)
        L[(size_t)(bi * 32 + r) * ld + bi * 32 + c] = c <= r ? diag[bi * 1024 + r * 32 + c] : 0.0;
    }
    return;
  }
  for (int r = bi * 32 + threadIdx.y; r < min(n, bi * 32 + 32); r += 8) {
    const int c = bj * 32 + threadIdx.x;
    if (c < n && c > r) L[(size_t)r * ld + c] = 0.0;
  }
}

// L' X = Y with the reference's term order (cholesky.rs:133-141): row k takes
// x_i l_ik for i = k+1 .. n-1 ascending, unfused, then divides by l_kk. Each
// row waits for its nearest neighbour first, so the order admits no
// wavefront; one thread per right-hand side runs the whole sweep (EXACT only).
__global__ void chol_back_exact_kernel(const double* __restrict__ L, size_t ld, double* X,
                                       size_t ldx, int n, int nrhs) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= nrhs) return;
  for (int k = n - 1; k >= 0; k--) {
    double s = X[(size_t)k * ldx + j];
    for (int i = k + 1; i < n; i++)
      s = __dsub_rn(s, __dmul_rn(X[(size_t)i * ldx + j], L[(size_t)i * ld + k]));
    X[(size_t)k * ldx + j] = s / L[(size_t)k * ld + k];
  }
}

cudaError_t configure_chol() {
  static la_device_once once;
  return once.run([](int) {
    return cudaFuncSetAttribute(chol_diag_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)(2 * CHW * CHP * sizeof(double)));
  });
}

la_status chol_check_ctx(la_ctx ctx) {
  if (!ctx) return LA_INVALID;
  cudaError_t e = cudaSetDevice(ctx->device);
  if (e != cudaSuccess) return la_cuda_fail(ctx, e, "cudaSetDevice");
  return LA_OK;
}

// FAST factorization of h->d_l (see the head of the file). Block widths as in the LU: an update's
// cost is the split product's epilogue, so wide blocks where there are many rows. n = 4099 with 5
// right-hand sides: 7.6 ms, of them 2.7 in the panels, 1.9 in the split products and 1.8 in the
// solves (64-column panels with FP64 FMA updates beside them: 31.9 ms).
struct FastChol {
  la_ctx ctx;
  double* L;
  size_t ld;
  int n;
  double* diag;
  int* flags;
  void* ws;
  size_t ws_bytes;
  Buf T;  // a panel transposed, where the split product cannot be used

  double* at(int r, int c) { return L + (size_t)r * ld + c; }

  // Rows [c0, n), columns [c0, c1), -= L[.., k0:k1] L[c0:c1, k0:k1]'; lower: only at or below the
  // diagonal (c1 = n then).
  la_status update(int k0, int k1, int c0, int c1, bool lower) {
    const int M = n - c0, N = c1 - c0, K = k1 - k0;
    if (M <= 0 || N <= 0) return LA_OK;
    if (N <= CB && K == CB) {
      const cudaError_t e = la_launch(ctx, chol_update32_kernel, dim3((M + CU_R - 1) / CU_R),
                                      dim3(CU_T), 0, ctx->stream, L, ld, k0, c0, N, n);
      if (e != cudaSuccess) return la_cuda_fail(ctx, e, "chol_update32_kernel launch");
      ctx->launches++;
      return la_check_launch(ctx, "chol_update32_kernel");
    }
    if (ws) {
      const la_status s = launch_gemm_split(ctx, ctx->stream, -1, M, N, K, at(c0, k0), ld,
                                            at(c0, k0), ld, true, at(c0, c0), ld, lower, ws, ws_bytes);
      if (s != LA_UNSUPPORTED) return s;
    }
    // by FMA, in steps of the transposed panel's 64 k
    const size_t ldt = pad4c((size_t)n);
    if (!T.p) LA_TRY(T.alloc((size_t)CHW * ldt * sizeof(double)));
    for (int k = k0; k < k1; k += CHW) {
      const int kb = std::min(CHW, k1 - k);
      chol_transpose_kernel<<<dim3((N + 31) / 32, (kb + 31) / 32), dim3(32, 8), 0, ctx->stream>>>(
          L, ld, k, kb, c0, N, T.d(), ldt);
      ctx->launches++;
      LA_TRY(la_check_launch(ctx, "chol_transpose_kernel"));
      la_status s = LA_UNSUPPORTED;
      if (lower) s = launch_gemm_lower(ctx, M, kb, at(c0, k), ld, T.d(), ldt, at(c0, c0), ld);
      if (s == LA_UNSUPPORTED)
        s = launch_gemm(ctx, GM_FMA_SUB, M, N, kb, at(c0, k), ld, T.d(), ldt, at(c0, c0), ld);
      LA_TRY(s);
    }
    return LA_OK;
  }

  la_status factor(int b0, int b1) {
    if (b1 - b0 > CB) {
      const int mid = b0 + ((b1 - b0 + 1) / 2 + CB - 1) / CB * CB;
      LA_TRY(factor(b0, mid));
      LA_TRY(update(b0, mid, mid, b1, false));
      return factor(mid, b1);
    }
    const int rows = n - b1;
    // 32 rows per CTA while there are SMs for them (each CTA factors the diagonal block itself), then
    // 64 more per pass
    const int per = (rows + ctx->sm_count - 1) / ctx->sm_count;
    const int rpc = CB + (std::max(0, per - CB) + 63) / 64 * 64;
    const cudaError_t e =
        la_launch(ctx, chol_panel32_kernel, dim3(std::max(1, (rows + rpc - 1) / rpc)), dim3(CB_T), 0,
                  ctx->stream, L, ld, b0, b1 - b0, n, rpc, diag + (size_t)(b0 / CB) * CB * CB, flags);
    if (e != cudaSuccess) return la_cuda_fail(ctx, e, "chol_panel32_kernel launch");
    ctx->launches++;
    return la_check_launch(ctx, "chol_panel32_kernel");
  }
};

int chol_block(int R) { return R > 2048 ? 256 : R > 768 ? 128 : 64; }

la_status chol_fast_factor(la_ctx ctx, la_chol h, int* d_flags) {
  const int n = (int)h->n;
  Buf diag(ctx), ws(ctx);
  LA_TRY(diag.alloc((size_t)(n + CB - 1) / CB * CB * CB * sizeof(double)));
  FastChol f{ctx, h->d_l, h->ld, n, diag.d(), d_flags, nullptr, 0, Buf(ctx)};
  if (n > CHW) {
    f.ws_bytes = gemm_split_ws(n, n, std::min(chol_block(n), n), true);
    if (ws.try_alloc(f.ws_bytes)) f.ws = ws.p;
  }
  struct PdlScope {
    la_ctx c;
    ~PdlScope() { c->pdl_now = false; }
  } scope{ctx};
  ctx->pdl_now = ctx->pdl != 0;
  for (int b0 = 0; b0 < n;) {
    const int b1 = std::min(b0 + chol_block(n - b0), n);
    LA_TRY(f.factor(b0, b1));
    LA_TRY(f.update(b0, b1, b1, n, true));
    b0 = b1;
  }
  const int nt = (n + 31) / 32;
  const cudaError_t e = la_launch(ctx, chol_zero_upper_kernel, dim3(nt, nt), dim3(32, 8), 0,
                                  ctx->stream, h->d_l, h->ld, n, (const double*)diag.d());
  if (e != cudaSuccess) return la_cuda_fail(ctx, e, "chol_zero_upper_kernel launch");
  ctx->launches++;
  return la_check_launch(ctx, "chol_zero_upper_kernel");
}

// EXACT factorization of h->d_l in place.
la_status chol_exact_factor(la_ctx ctx, la_chol h, int* d_flags) {
  const int n = (int)h->n;
  const size_t ld = h->ld;
  double* L = h->d_l;
  cudaStream_t st = ctx->stream;
  LA_CUDA(ctx, configure_chol());
  Buf S(ctx), T0(ctx), T1(ctx);
  LA_TRY(S.alloc((size_t)n * ld * sizeof(double)));
  LA_CUDA(ctx, cudaMemsetAsync(S.p, 0, (size_t)n * ld * sizeof(double), st));
  // Transposed panels (the GEMM's K x N operand), two so that panel k + 1 can
  // be transposed while panel k's update still reads its own.
  const size_t ldt = pad4c((size_t)n);
  if (n > CHW) {
    LA_TRY(T0.alloc((size_t)CHW * ldt * sizeof(double)));
    LA_TRY(T1.alloc((size_t)CHW * ldt * sizeof(double)));
  }
  double* Tbuf[2] = {T0.d(), T1.d()};
  const size_t dsm = 2 * CHW * CHP * sizeof(double);
  const bool look = ctx->lookahead != 0 && ctx->side_stream != nullptr;

  // Diagonal block, rows below and transpose of panel [j0, j0 + jb) on stream s.
  auto panel = [&](int j0, int jb, double* T, cudaStream_t s) -> la_status {
    const int j1 = j0 + jb;
    chol_diag_kernel<<<1, 256, dsm, s>>>(L, S.d(), ld, j0, jb, d_flags);
    ctx->launches++;
    LA_TRY(la_check_launch(ctx, "chol_diag_kernel"));
    if (j1 >= n) return LA_OK;
    const int rows = n - j1;
    const int pg = (rows + PANEL_T - 1) / PANEL_T;
    chol_panel_kernel<<<pg, PANEL_T, 0, s>>>(L, S.d(), ld, j0, j1, n);
    ctx->launches++;
    LA_TRY(la_check_launch(ctx, "chol_panel_kernel"));
    chol_transpose_kernel<<<dim3((rows + 31) / 32, (jb + 31) / 32), dim3(32, 8), 0, s>>>(
        L, ld, j0, jb, j1, rows, T, ldt);
    ctx->launches++;
    return la_check_launch(ctx, "chol_transpose_kernel");
  };
  // S22 += L21 L21' of panel [j0, j0 + jb) on rows and columns >= c0 (lower part), in up to 8 row
  // strips [a, b) that each stop at their own diagonal block.
  auto update = [&](int j0, int jb, const double* T, int c0) -> la_status {
    const int j1 = j0 + jb, rows = n - c0;
    if (rows <= 0) return LA_OK;
    const int nstrip = std::max(1, std::min(8, rows / 512));
    const int hs = ((rows + nstrip - 1) / nstrip + CHW - 1) / CHW * CHW;
    for (int a = c0; a < n; a += hs) {
      const int b = std::min(n, a + hs);
      LA_TRY(launch_gemm(ctx, GM_EXACT_ADD, b - a, b - c0, jb, L + (size_t)a * ld + j0, ld,
                         T + (c0 - j1), ldt, S.d() + (size_t)a * ld + c0, ld));
    }
    return LA_OK;
  };
  // The next panel's columns [j1, j2) of rows >= j1 (a plain GEMM).
  auto update_next = [&](int j0, int jb, const double* T, int j1, int j2) -> la_status {
    return launch_gemm(ctx, GM_EXACT_ADD, n - j1, j2 - j1, jb, L + (size_t)j1 * ld + j0, ld, T, ldt,
                       S.d() + (size_t)j1 * ld + j1, ld);
  };

  // Lookahead: panel k's update of panel k + 1's columns first, then panel k + 1 on the
  // high-priority side stream while the rest of panel k's update runs (rows and columns >= j2).
  // They touch disjoint data: panel k + 1 owns columns [j1, j2) of rows >= j1, and the rest of the
  // update reads panel k's finished columns and its transposed copy.
  LA_TRY(panel(0, std::min(CHW, n), Tbuf[0], st));
  for (int j0 = 0, k = 0; j0 < n; j0 += CHW, k++) {
    const int jb = std::min(CHW, n - j0), j1 = j0 + jb;
    if (j1 >= n) break;
    const int jbn = std::min(CHW, n - j1), j2 = j1 + jbn;
    double* Tk = Tbuf[k & 1];
    double* Tn = Tbuf[(k + 1) & 1];
    if (look && j2 < n) {
      LA_TRY(update_next(j0, jb, Tk, j1, j2));
      LA_CUDA(ctx, cudaEventRecord(ctx->ev_fork, st));
      LA_CUDA(ctx, cudaStreamWaitEvent(ctx->side_stream, ctx->ev_fork, 0));
      LA_TRY(panel(j1, jbn, Tn, ctx->side_stream));
      LA_CUDA(ctx, cudaEventRecord(ctx->ev_join, ctx->side_stream));
      LA_TRY(update(j0, jb, Tk, j2));
      LA_CUDA(ctx, cudaStreamWaitEvent(st, ctx->ev_join, 0));
    } else {
      LA_TRY(update(j0, jb, Tk, j1));
      LA_TRY(panel(j1, jbn, Tn, st));
    }
  }
  const int nt = (n + 31) / 32;
  chol_zero_upper_kernel<<<dim3(nt, nt), dim3(32, 8), 0, st>>>(L, ld, n, nullptr);
  ctx->launches++;
  return la_check_launch(ctx, "chol_zero_upper_kernel");
}

// Factors h->d_l (a copy of A) in place; *none = the reference's None.
la_status chol_factor(la_ctx ctx, la_chol h, int* none) {
  const int n = (int)h->n;
  cudaStream_t st = ctx->stream;
  int* d_flags = reinterpret_cast<int*>(ctx->d_small);
  LA_CUDA(ctx, cudaMemsetAsync(d_flags, 0, 2 * sizeof(int), st));
  const int nt = (n + 31) / 32;
  chol_sym_check_kernel<<<dim3(nt, nt), dim3(32, 8), 0, st>>>(h->d_l, h->ld, n, d_flags);
  ctx->launches++;
  LA_TRY(la_check_launch(ctx, "chol_sym_check_kernel"));
  LA_TRY(h->arith == LA_ARITH_EXACT ? chol_exact_factor(ctx, h, d_flags)
                                    : chol_fast_factor(ctx, h, d_flags));
  int* flags = static_cast<int*>(ctx->h_pinned);
  LA_CUDA(ctx, cudaMemcpyAsync(flags, d_flags, 2 * sizeof(int), cudaMemcpyDeviceToHost, st));
  LA_TRY(la_sync_and_check(ctx, "cholesky factorization"));
  *none = (flags[0] | flags[1]) != 0;
  return LA_OK;
}

la_status chol_alloc(la_ctx ctx, size_t n, la_chol* out) {
  if (n > (size_t)INT32_MAX / 2) return LA_UNSUPPORTED;
  la_chol h = new (std::nothrow) la_chol_handle();
  if (!h) return LA_NOMEM;
  h->ctx = ctx;
  h->n = n;
  h->ld = pad4c(n);
  h->arith = ctx->arith;
  void* p = nullptr;
  la_status s = la_device_alloc(ctx, &p, n * h->ld * sizeof(double));
  if (s != LA_OK) { delete h; return s; }
  h->d_l = static_cast<double*>(p);
  *out = h;
  return LA_OK;
}

la_status chol_new_common(la_ctx ctx, la_chol h, la_chol* out) {
  int none = 0;
  la_status s = chol_factor(ctx, h, &none);
  if (s == LA_OK && none) s = LA_SINGULAR;
  if (s != LA_OK) {
    la_chol_free(h);
    return s;
  }
  *out = h;
  return LA_OK;
}

la_status chol_solve_device_common(la_chol h, const double* d_b, size_t ldb, size_t brows,
                                   size_t nrhs, double* d_x, size_t ldx) {
  la_ctx ctx = h->ctx;
  if (brows != h->n) return LA_BADSHAPE;  // cholesky.rs:118
  if (nrhs == 0) return LA_BADSHAPE;      // Matrix::new asserts cols > 0
  const int n = (int)h->n;
  const bool exact = h->arith == LA_ARITH_EXACT;
  cudaStream_t st = ctx->stream;
  const size_t ldw = pad4c(nrhs);
  Buf X(ctx);
  LA_TRY(X.alloc(h->n * ldw * sizeof(double)));
  LA_CUDA(ctx, cudaMemcpy2DAsync(X.p, ldw * sizeof(double), d_b, ldb * sizeof(double),
                                 nrhs * sizeof(double), h->n, cudaMemcpyDeviceToDevice, st));
  // L Y = B (cholesky.rs:123-131): ascending terms, then the division
  LA_TRY(launch_tri_wave(ctx, exact, false, true, h->d_l, h->ld, X.d(), ldw, n, (int)nrhs));
  if (exact) {
    chol_back_exact_kernel<<<((int)nrhs + 127) / 128, 128, 0, st>>>(h->d_l, h->ld, X.d(), ldw, n,
                                                                   (int)nrhs);
    ctx->launches++;
    LA_TRY(la_check_launch(ctx, "chol_back_exact_kernel"));
  } else {
    // L' X = Y on the transposed copy (rows of L' contiguous), any term order
    if (!h->d_lt) {
      void* p = nullptr;
      LA_TRY(la_device_alloc(ctx, &p, h->n * h->ld * sizeof(double)));
      h->d_lt = static_cast<double*>(p);
      const int nt = (n + 31) / 32;
      chol_transpose_kernel<<<dim3(nt, nt), dim3(32, 8), 0, st>>>(h->d_l, h->ld, 0, n, 0, n,
                                                                  h->d_lt, h->ld);
      ctx->launches++;
      LA_TRY(la_check_launch(ctx, "chol_transpose_kernel"));
    }
    LA_TRY(launch_tri_wave(ctx, false, true, true, h->d_lt, h->ld, X.d(), ldw, n, (int)nrhs));
  }
  LA_CUDA(ctx, cudaMemcpy2DAsync(d_x, ldx * sizeof(double), X.p, ldw * sizeof(double),
                                 nrhs * sizeof(double), h->n, cudaMemcpyDeviceToDevice, st));
  return LA_OK;
}

}  // namespace

// ---- C ABI -----------------------------------------------------------------

la_status la_chol_new(la_ctx ctx, const double* a, size_t m, size_t n, la_chol* out) {
  LA_TRY(chol_check_ctx(ctx));
  if (!a || !out) return LA_INVALID;
  *out = nullptr;
  if (m == 0 || n == 0) return LA_BADSHAPE;  // Matrix::new asserts (mod.rs:209)
  if (m != n) return LA_SINGULAR;           // cholesky.rs:57-59: None
  la_chol h = nullptr;
  LA_TRY(chol_alloc(ctx, n, &h));
  const la_status s = la_copy_to_device(ctx, h->d_l, h->ld, a, n, n);
  if (s != LA_OK) {
    la_chol_free(h);
    return s;
  }
  return chol_new_common(ctx, h, out);
}

la_status la_chol_new_device(la_ctx ctx, const double* d_a, size_t lda, size_t n, la_chol* out) {
  LA_TRY(chol_check_ctx(ctx));
  if (!d_a || !out || lda < n) return LA_INVALID;
  *out = nullptr;
  if (n == 0) return LA_BADSHAPE;
  la_chol h = nullptr;
  LA_TRY(chol_alloc(ctx, n, &h));
  cudaError_t e = cudaMemcpy2DAsync(h->d_l, h->ld * sizeof(double), d_a, lda * sizeof(double),
                                    n * sizeof(double), n, cudaMemcpyDeviceToDevice, ctx->stream);
  if (e != cudaSuccess) {
    la_chol_free(h);
    return la_cuda_fail(ctx, e, "copy A on device");
  }
  return chol_new_common(ctx, h, out);
}

void la_chol_free(la_chol h) {
  if (!h) return;
  cudaSetDevice(h->ctx->device);
  la_device_free(h->ctx, h->d_l);
  la_device_free(h->ctx, h->d_lt);
  delete h;
}

la_status la_chol_n(la_chol h, size_t* n) {
  if (!h || !n) return LA_INVALID;
  *n = h->n;
  return LA_OK;
}

la_status la_chol_get_l(la_chol h, double* out) {
  if (!h || !out) return LA_INVALID;
  la_ctx ctx = h->ctx;
  LA_TRY(chol_check_ctx(ctx));
  LA_TRY(la_copy_to_host(ctx, out, h->d_l, h->ld, h->n, h->n));
  return la_sync_and_check(ctx, "la_chol_get_l");
}

la_status la_chol_solve(la_chol h, const double* b, size_t brows, size_t nrhs, double* x) {
  if (!h || !b || !x) return LA_INVALID;
  la_ctx ctx = h->ctx;
  LA_TRY(chol_check_ctx(ctx));
  if (brows != h->n || nrhs == 0) return LA_BADSHAPE;
  Buf B(ctx);
  LA_TRY(B.alloc(brows * nrhs * sizeof(double)));
  LA_CUDA(ctx, cudaMemcpyAsync(B.p, b, brows * nrhs * sizeof(double), cudaMemcpyHostToDevice,
                               ctx->stream));
  LA_TRY(chol_solve_device_common(h, B.d(), nrhs, brows, nrhs, B.d(), nrhs));
  LA_CUDA(ctx, cudaMemcpyAsync(x, B.p, brows * nrhs * sizeof(double), cudaMemcpyDeviceToHost,
                               ctx->stream));
  return la_sync_and_check(ctx, "la_chol_solve");
}

la_status la_chol_solve_device(la_chol h, const double* d_b, size_t ldb, size_t brows,
                               size_t nrhs, double* d_x, size_t ldx) {
  if (!h || !d_b || !d_x || ldb < nrhs || ldx < nrhs) return LA_INVALID;
  LA_TRY(chol_check_ctx(h->ctx));
  return chol_solve_device_common(h, d_b, ldb, brows, nrhs, d_x, ldx);
}
