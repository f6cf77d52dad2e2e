// Row swaps, triangular updates and the small kernels around the blocked LU.
#include "la_internal.cuh"

namespace {

// ---- row swaps outside the panel (lu.rs:140-145 for the other columns) ----
// Applies the composed moves of one panel (dest <- src) to columns
// [c_begin, c_end) of one matrix. All sources are read into shared memory
// before any destination is written, so the moves act as one permutation.
constexpr int SW_COLS = 32;

// The context's error word (nonzero after a device wait gave up). The kernels
// that apply a panel's row interchanges return at entry when it is set: a
// panel that gave up left no valid interchanges behind.
__device__ __forceinline__ bool aborted(const int* err) {
  return err != nullptr && *reinterpret_cast<const volatile int*>(err) != 0;
}

template <typename T>
__global__ void __launch_bounds__(256)
laswp_kernel(T* M0, T* M1, T* M2, size_t ld, int b0, int e0, int b1, int e1,
             int b2, int e2, const int* __restrict__ swaps, const int* err) {
  la_pdl_wait();
  la_pdl_trigger();
  __shared__ T tmp[2 * MAX_PANEL_W][SW_COLS];
  __shared__ int s_abort;
  if (threadIdx.x == 0) s_abort = aborted(err);
  __syncthreads();
  if (s_abort) return;
  const int cnt = swaps[0];
  if (cnt == 0) return;
  const int* dst = swaps + 1;
  const int* src = swaps + 1 + 2 * MAX_PANEL_W;
  // blockIdx.y selects the segment.
  T* M;
  int cb, ce;
  if (blockIdx.y == 0) { M = M0; cb = b0; ce = e0; }
  else if (blockIdx.y == 1) { M = M1; cb = b1; ce = e1; }
  else { M = M2; cb = b2; ce = e2; }
  if (M == nullptr) return;
  const int c = cb + blockIdx.x * SW_COLS + (threadIdx.x % SW_COLS);
  if (cb + (int)blockIdx.x * SW_COLS >= ce) return;
  const int ty = threadIdx.x / SW_COLS;  // 0..7
  const bool ok = c < ce;
  for (int q = ty; q < cnt; q += 8)
    if (ok) tmp[q][threadIdx.x % SW_COLS] = M[(size_t)src[q] * ld + c];
  __syncthreads();
  for (int q = ty; q < cnt; q += 8)
    if (ok) M[(size_t)dst[q] * ld + c] = tmp[q][threadIdx.x % SW_COLS];
}

// The moves of `lists` panels, one list after the other, on columns [c0, c1), whose swaps were
// deferred to the end of their block: a list's sources are all in registers before its first
// destination is written. Lists go through L2 one after the other, about a microsecond each; one
// thread per column replaying the interchanges themselves took 141 us for 256 of them (n = 16384,
// every pivot off the diagonal), each a dependent round trip. (In the FP64 LU, whose chain leaves
// nothing to run beside it, deferring the swaps this way measured 2 to 3 % slower.)
template <typename T>
__global__ void __launch_bounds__(256)
laswp_lists_kernel(T* A, size_t ld, const int* __restrict__ swaps, int lists, int c0, int c1,
                   const int* err) {
  la_pdl_wait();
  la_pdl_trigger();
  constexpr int G = 256 / SW_COLS, PER = 2 * MAX_PANEL_W / G;  // move groups, moves per thread
  const int c = c0 + blockIdx.x * SW_COLS + threadIdx.x % SW_COLS;
  const int g = threadIdx.x / SW_COLS;
  // every list's length at once; lists without moves cost nothing then
  __shared__ int s_cnt[SWAP_LISTS];
  if ((int)threadIdx.x < lists) s_cnt[threadIdx.x] = aborted(err) ? 0 : swaps[threadIdx.x * SWAP_STRIDE];
  __syncthreads();
  const bool ok = c < c1;
  for (int s = 0; s < lists; s++, swaps += SWAP_STRIDE) {
    const int cnt = s_cnt[s];
    if (cnt == 0) continue;
    T v[PER];
#pragma unroll
    for (int i = 0; i < PER; i++)
      if (ok && g + i * G < cnt) v[i] = A[(size_t)swaps[1 + 2 * MAX_PANEL_W + g + i * G] * ld + c];
    __syncthreads();
#pragma unroll
    for (int i = 0; i < PER; i++)
      if (ok && g + i * G < cnt) A[(size_t)swaps[1 + g + i * G] * ld + c] = v[i];
    __syncthreads();
  }
}

// ---- row-panel triangular update: U12 = L11^{-1} A12 ----------------------
// Rows [j0, j0 + jb) of columns [c_begin, c_end). Row k is finished, then every row i > k of the block
// takes its k-th term, i.e. each element receives its terms in ascending k, like lu.rs:124-128.
//
// FP64 form, jb <= 64: 8 columns per CTA. With two FP64 FMAs per clock an SM needs 16 clocks
// for one warp's FMA, so the 64 x 64 triangle costs 0.5 us a column and the strip's width sets the
// latency: CTAs of 32 columns took 49 us however few columns there were. Row k is final when step k
// starts; the rows below take its term, neighbouring items (row, column) on neighbouring threads, so
// that no lane idles but in the last warp.
// EXACT: the running sums s from S, row k formed as a - s at its step, terms added unfused.
constexpr int TC8 = 8;
constexpr int TC8_T = 256;
template <bool EXACT>
__global__ void __launch_bounds__(TC8_T)
trsm_cols8_kernel(double* A, const double* S, size_t ld, int j0, int jb, int c_begin, int c_end) {
  la_pdl_wait();
  la_pdl_trigger();
  __shared__ double L[MAX_PANEL_W][MAX_PANEL_W + 1];
  __shared__ double x[MAX_PANEL_W][TC8], xs[EXACT ? MAX_PANEL_W : 1][TC8];
  const int tid = threadIdx.x, col = tid % TC8, r0 = tid / TC8;  // r0 0..31
  const int c = c_begin + blockIdx.x * TC8 + col;
  const bool ok = c < c_end;
  constexpr int PER = MAX_PANEL_W * MAX_PANEL_W / TC8_T;
  double l[PER];  // all loads in flight together
#pragma unroll
  for (int q = 0; q < PER; q++) {
    const int i = (tid + q * TC8_T) / MAX_PANEL_W, k = tid % MAX_PANEL_W;
    l[q] = i < jb && k < i ? A[(size_t)(j0 + i) * ld + j0 + k] : 0.0;
  }
#pragma unroll
  for (int q = 0; q < PER; q++) L[(tid + q * TC8_T) / MAX_PANEL_W][tid % MAX_PANEL_W] = l[q];
  for (int i = r0; i < jb; i += TC8_T / TC8) {
    x[i][col] = ok ? A[(size_t)(j0 + i) * ld + c] : 0.0;
    if (EXACT) xs[i][col] = ok ? S[(size_t)(j0 + i) * ld + c] : 0.0;
  }
  __syncthreads();
  if (EXACT) {
    if (r0 == 0) x[0][col] = __dsub_rn(x[0][col], xs[0][col]);
    __syncthreads();
  }
  for (int k = 0; k + 1 < jb; k++) {
    const double u = x[k][col];
    for (int i = k + 1 + r0; i < jb; i += TC8_T / TC8) {
      if (EXACT) {
        const double s = __dadd_rn(xs[i][col], __dmul_rn(L[i][k], u));
        xs[i][col] = s;
        if (i == k + 1) x[i][col] = __dsub_rn(x[i][col], s);  // its last term
      } else {
        x[i][col] = fma(-L[i][k], u, x[i][col]);
      }
    }
    __syncthreads();
  }
  if (ok)
    for (int i = r0; i < jb; i += TC8_T / TC8) A[(size_t)(j0 + i) * ld + c] = x[i][col];
}

// FP32 form for the mixed LU's 32-row blocks (jb <= 32, FMA): one thread per
// column holds the column's jb values in registers and applies the terms in
// ascending k, with the unit-lower block broadcast from shared memory. No
// barrier inside the sweep: at FP32 rates the barriers, not the FMAs, were the
// cost of the 32-step sweep.
constexpr int TRR_W = 32;
constexpr int TRR_T = 128;
__global__ void __launch_bounds__(TRR_T)
trsm_rowpanel_reg_kernel(float* A, size_t ld, int j0, int jb, int c_begin, int c_end) {
  la_pdl_wait();
  la_pdl_trigger();
  __shared__ float L[TRR_W][TRR_W + 1];
  for (int idx = threadIdx.x; idx < jb * jb; idx += TRR_T) {
    const int i = idx / jb, k = idx % jb;
    L[i][k] = A[(size_t)(j0 + i) * ld + j0 + k];
  }
  __syncthreads();
  const int c = c_begin + blockIdx.x * TRR_T + threadIdx.x;
  if (c >= c_end) return;
  float x[TRR_W];
#pragma unroll
  for (int i = 0; i < TRR_W; i++) x[i] = i < jb ? A[(size_t)(j0 + i) * ld + c] : 0.f;
#pragma unroll
  for (int k = 0; k < TRR_W; k++) {
    if (k >= jb) break;
    const float xk = x[k];
#pragma unroll
    for (int i = k + 1; i < TRR_W; i++)
      if (i < jb) x[i] = fmaf(-L[i][k], xk, x[i]);
  }
#pragma unroll
  for (int i = 0; i < TRR_W; i++)
    if (i < jb) A[(size_t)(j0 + i) * ld + c] = x[i];
}

// ---- the mixed LU's outer-panel triangular update: X = L11^-1 X ----------------------
// Rows [j0, j0 + jbo) (jbo <= 256) of columns [c_begin, c_end), L11 the unit
// lower jbo x jbo block of A at (j0, j0). One CTA per 32 columns keeps its
// jbo x 32 block of X in shared memory. Per 32-row block of L11: the block's
// rows and everything below it in its 32 columns are staged in shared memory;
// warp 0 solves the diagonal block (lane = column, the 32 values in registers,
// no barrier inside); then the 256 threads subtract the block's contribution
// from the rows below (8 threads per row, 4 columns each, 32-deep dot products
// from shared memory). One launch instead of a row-panel solve and a GEMM per
// 32 rows.
constexpr int TB_R = 256, TB_C = 32;
constexpr size_t TB_SMEM = (size_t)2 * TB_R * (TB_C + 1) * sizeof(float);
__global__ void __launch_bounds__(256)
trsm_block_kernel(float* A, size_t ld, int j0, int jbo, int c_begin, int c_end) {
  la_pdl_wait();
  la_pdl_trigger();
  extern __shared__ __align__(16) float tb_sm[];
  float(*X)[TB_C + 1] = reinterpret_cast<float(*)[TB_C + 1]>(tb_sm);
  float(*Lb)[TB_C + 1] = reinterpret_cast<float(*)[TB_C + 1]>(tb_sm + TB_R * (TB_C + 1));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int cb = c_begin + blockIdx.x * TB_C;
  for (int idx = tid; idx < jbo * TB_C; idx += 256) {
    const int r = idx / TB_C, c = idx % TB_C;
    X[r][c] = cb + c < c_end ? A[(size_t)(j0 + r) * ld + cb + c] : 0.f;
  }
  for (int kb = 0; kb < jbo; kb += TB_C) {
    const int bw = min(TB_C, jbo - kb);
    // L11 rows [kb, jbo) of columns [kb, kb + bw)
    for (int idx = tid; idx < (jbo - kb) * TB_C; idx += 256) {
      const int r = idx / TB_C, k = idx % TB_C;
      Lb[r][k] = k < bw ? A[(size_t)(j0 + kb + r) * ld + j0 + kb + k] : 0.f;
    }
    __syncthreads();
    if (warp == 0) {
      float x[TB_C];
#pragma unroll
      for (int i = 0; i < TB_C; i++) x[i] = i < bw ? X[kb + i][lane] : 0.f;
#pragma unroll
      for (int k = 0; k < TB_C; k++) {
        if (k >= bw) break;
        const float xk = x[k];
#pragma unroll
        for (int i = k + 1; i < TB_C; i++) x[i] = fmaf(-Lb[i][k], xk, x[i]);
      }
#pragma unroll
      for (int i = 0; i < TB_C; i++)
        if (i < bw) X[kb + i][lane] = x[i];
    }
    __syncthreads();
    const int rows = jbo - kb - bw;
    for (int e = tid; e < rows * 8; e += 256) {
      const int r = e >> 3, c4 = (e & 7) * 4, i = kb + bw + r;
      float a0 = X[i][c4], a1 = X[i][c4 + 1], a2 = X[i][c4 + 2], a3 = X[i][c4 + 3];
      for (int k = 0; k < bw; k++) {
        const float l = Lb[bw + r][k];
        a0 = fmaf(-l, X[kb + k][c4], a0);
        a1 = fmaf(-l, X[kb + k][c4 + 1], a1);
        a2 = fmaf(-l, X[kb + k][c4 + 2], a2);
        a3 = fmaf(-l, X[kb + k][c4 + 3], a3);
      }
      X[i][c4] = a0;
      X[i][c4 + 1] = a1;
      X[i][c4 + 2] = a2;
      X[i][c4 + 3] = a3;
    }
    __syncthreads();
  }
  for (int idx = tid; idx < jbo * TB_C; idx += 256) {
    const int r = idx / TB_C, c = idx % TB_C;
    if (cb + c < c_end) A[(size_t)(j0 + r) * ld + cb + c] = X[r][c];
  }
}

// ---- after the factorization: permutation vector, sign, zero diagonal ------
// The swap list (LAPACK ipiv form) is replayed in order on a permutation
// vector (lu.rs:147-149), the sign flips once per real swap (lu.rs:151), and
// U's diagonal is scanned for an exact zero (lu.rs:177).
// Whether the entries [c0, c1) of a row lie unevenly: one of their quarters has hardly any (1 in 32)
// within 2^-5 of the row's largest, as where they fall off along the row (columns or rows of very
// different size) or the matrix is banded. Whole warp.
__device__ bool uneven_row(const double* row, int c0, int c1) {
  const int lane = threadIdx.x & 31;
  auto exp_of = [&](int c) { return (int)(__double_as_longlong(row[c]) >> 52) & 0x7ff; };
  int top = 0;
#pragma unroll 8
  for (int c = c0 + lane; c < c1; c += 32) top = max(top, exp_of(c));
  top = __reduce_max_sync(0xffffffffu, top);
  bool uneven = false;
  for (int q = 0; q < 4; q++) {
    const int a = c0 + (int)((long long)(c1 - c0) * q / 4), b = c0 + (int)((long long)(c1 - c0) * (q + 1) / 4);
    int large = 0;
#pragma unroll 8
    for (int c = a + lane; c < b; c += 32) large += exp_of(c) >= top - 4;
    uneven |= __reduce_add_sync(0xffffffffu, large) * 32 < b - a;
  }
  return uneven;
}

// uneven (may be null): how many of LU_SAMPLES rows of U lie unevenly, for the choice of the solve. Each
// warp without a part in the replay looks at one meanwhile. (L's rows need no look: where they are uneven
// the blocked forward half is still the faster one.)
constexpr int LU_SAMPLES = 31;
constexpr int LU_FINISH_T = 32 * (LU_SAMPLES + 1);
constexpr int LU_SAMPLE_MIN = 256;  // entries of a row that is looked at
template <typename T>
__global__ void lu_finish_kernel(const int* __restrict__ ipiv, uint64_t* piv, int m, int kmin,
                                 const T* LU, size_t ld, int* flags, int* uneven, int smem_rows,
                                 const int* err) {
  extern __shared__ int sperm[];  // permutation in shared memory when m fits
  __shared__ int zero, s_abort, s_uneven;
  if (threadIdx.x == 0) s_abort = aborted(err);
  __syncthreads();
  if (s_abort) return;  // the host reports the error; flags and piv are not used
  if (threadIdx.x == 0) zero = s_uneven = 0;
  const bool in_smem = m <= smem_rows;
  if (in_smem) {
    for (int i = threadIdx.x; i < m; i += blockDim.x) sperm[i] = i;
  } else {
    for (int i = threadIdx.x; i < m; i += blockDim.x) piv[i] = (uint64_t)i;
  }
  __syncthreads();
  for (int j = threadIdx.x; j < kmin; j += blockDim.x)
    if (LU[(size_t)j * ld + j] == T(0)) atomicOr(&zero, 1);
  // One warp replays: 32 interchanges are loaded at once, ahead of the chain
  // (two shared-memory accesses per interchange; with the load in it, n = 1000
  // took 55 us).
  if (threadIdx.x < 32) {
    int swaps = 0;
    int next = (int)threadIdx.x < kmin ? ipiv[threadIdx.x] : 0;
    for (int j0 = 0; j0 < kmin; j0 += 32) {
      const int mine = next, cnt = min(32, kmin - j0);
      if (j0 + 32 + (int)threadIdx.x < kmin) next = ipiv[j0 + 32 + threadIdx.x];
      swaps += __popc(__ballot_sync(0xffffffffu, (int)threadIdx.x < cnt && mine != j0 + (int)threadIdx.x));
      for (int i = 0; i < cnt; i++) {
        const int j = j0 + i, p = __shfl_sync(0xffffffffu, mine, i);
        if (threadIdx.x != 0 || p == j) continue;
        if (in_smem) {
          const int t = sperm[p];
          sperm[p] = sperm[j];
          sperm[j] = t;
        } else {
          const uint64_t t = piv[p];
          piv[p] = piv[j];
          piv[j] = t;
        }
      }
    }
    if (threadIdx.x == 0) flags[0] = !(swaps & 1);
  } else if constexpr (sizeof(T) == 8) {
    if (uneven) {  // a square matrix
      const int i = (int)((2ll * (threadIdx.x / 32) - 1) * m / (2 * LU_SAMPLES));
      if (m - 1 - i >= LU_SAMPLE_MIN && uneven_row(LU + (size_t)i * ld, i + 1, m) && threadIdx.x % 32 == 0)
        atomicAdd(&s_uneven, 1);
    }
  }
  __syncthreads();
  if (in_smem)
    for (int i = threadIdx.x; i < m; i += blockDim.x) piv[i] = (uint64_t)sperm[i];
  if (threadIdx.x == 0) {
    flags[1] = zero;
    if (uneven) *uneven = s_uneven;
  }
}

// X = B(piv, :) (lu.rs:245-254).
__global__ void permute_rows_kernel(const uint64_t* __restrict__ piv, const double* __restrict__ B,
                                    size_t ldb, double* __restrict__ X, size_t ldx, int m,
                                    int nrhs) {
  size_t total = (size_t)m * nrhs;
  for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
       idx += (size_t)gridDim.x * blockDim.x) {
    int i = (int)(idx / nrhs), j = (int)(idx % nrhs);
    X[(size_t)i * ldx + j] = B[(size_t)piv[i] * ldb + j];
  }
}

// Y(:, piv[c]) = X(:, c), one row per CTA: written in any order, but within a row of L2 lines.
__global__ void permute_cols_kernel(const uint64_t* __restrict__ piv, const double* __restrict__ X,
                                    double* __restrict__ Y, size_t ld, int n) {
  const size_t r = (size_t)blockIdx.x * ld;
  for (int c = threadIdx.x; c < n; c += blockDim.x) Y[r + piv[c]] = X[r + c];
}

// X = I(piv, :) for inverse (mod.rs:1036 solves against Matrix::id); I without piv.
__global__ void identity_permuted_kernel(const uint64_t* __restrict__ piv, double* X, size_t ldx,
                                         int m) {
  size_t total = (size_t)m * m;
  for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
       idx += (size_t)gridDim.x * blockDim.x) {
    int i = (int)(idx / m), j = (int)(idx % m);
    X[(size_t)i * ldx + j] = ((piv ? piv[i] : (uint64_t)i) == (uint64_t)j) ? 1.0 : 0.0;
  }
}

// det (lu.rs:224-232): one thread multiplies U's diagonal in ascending order,
// the reference's exact sequence of roundings. The diagonal comes through
// shared memory, a thread to each entry: n dependent products bound it (64
// clocks each), where n loads in one thread's path took 48 us at n = 512.
constexpr int DET_T = 256, DET_CHUNK = 1024;
__global__ void __launch_bounds__(DET_T)
det_kernel(const double* LU, size_t ld, int n, int pospivsign, double* out) {
  __shared__ double diag[DET_CHUNK];
  double d = pospivsign ? 1.0 : -1.0;
  for (int j0 = 0; j0 < n; j0 += DET_CHUNK) {
    const int cnt = min(DET_CHUNK, n - j0);
    for (int i = threadIdx.x; i < cnt; i += DET_T) diag[i] = LU[(size_t)(j0 + i) * ld + j0 + i];
    __syncthreads();
    if (threadIdx.x == 0) {
#pragma unroll 8
      for (int i = 0; i < cnt; i++) d = d * diag[i];
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) out[0] = d;
}

// get_l (which 0, lu.rs:184-202), get_u (1, :204-215), get_p (2, :217-220),
// packed copy (3).
__global__ void unpack_kernel(int which, const double* LU, size_t ld, int m, int n,
                              const uint64_t* piv, double* out) {
  const int kmin = m < n ? m : n;
  int rows, cols;
  if (which == 0) { rows = m; cols = kmin; }
  else if (which == 1) { rows = kmin; cols = n; }
  else if (which == 2) { rows = m; cols = m; }
  else { rows = m; cols = n; }
  size_t total = (size_t)rows * cols;
  for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
       idx += (size_t)gridDim.x * blockDim.x) {
    int i = (int)(idx / cols), j = (int)(idx % cols);
    double v;
    if (which == 0) v = i > j ? LU[(size_t)i * ld + j] : (i == j ? 1.0 : 0.0);
    else if (which == 1) v = i <= j ? LU[(size_t)i * ld + j] : 0.0;
    else if (which == 2) v = (piv[i] == (uint64_t)j) ? 1.0 : 0.0;
    else v = LU[(size_t)i * ld + j];
    out[idx] = v;
  }
}

__global__ void copy2d_kernel(const double* __restrict__ src, size_t lds, double* __restrict__ dst,
                              size_t ldd, int rows, int cols) {
  size_t total = (size_t)rows * cols;
  for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < total;
       idx += (size_t)gridDim.x * blockDim.x) {
    int i = (int)(idx / cols), j = (int)(idx % cols);
    dst[(size_t)i * ldd + j] = src[(size_t)i * lds + j];
  }
}

int grid_for(la_ctx ctx, size_t total) {
  size_t g = (total + 255) / 256;
  size_t cap = (size_t)ctx->sm_count * 8;
  return (int)std::max<size_t>(1, std::min(g, cap));
}

}  // namespace

template <typename T>
la_status launch_laswp_t(la_ctx ctx, cudaStream_t stream, bool exact, T* A, T* S, size_t ld,
                         int c0, int c1, int j0, int jb) {
  const int j1 = j0 + jb;
  const int left = j0 - c0, right = c1 - j1;
  const int gx = std::max((left + SW_COLS - 1) / SW_COLS, (right + SW_COLS - 1) / SW_COLS);
  if (gx <= 0) return LA_OK;
  dim3 grid(gx, exact ? 3 : 2);
  const cudaError_t e = la_launch(ctx, laswp_kernel<T>, grid, dim3(256), 0, stream, A, A,
                                  exact ? S : nullptr, ld, c0, j0, j1, c1, j1, c1,
                                  (const int*)ctx->swaps(), (const int*)ctx->d_err);
  if (e != cudaSuccess) return la_cuda_fail(ctx, e, "laswp_kernel launch");
  ctx->launches++;
  return la_check_launch(ctx, "laswp_kernel");
}

la_status launch_laswp(la_ctx ctx, bool exact, double* A, double* S, size_t ld, int c0, int c1,
                       int j0, int jb) {
  return launch_laswp_t<double>(ctx, ctx->stream, exact, A, S, ld, c0, c1, j0, jb);
}
la_status launch_laswp_f32(la_ctx ctx, float* A, size_t ld, int c0, int c1, int j0, int jb) {
  return launch_laswp_t<float>(ctx, ctx->stream, false, A, nullptr, ld, c0, c1, j0, jb);
}
la_status launch_laswp_lists_f32(la_ctx ctx, float* A, size_t ld, int first, int lists, int c0,
                                 int c1) {
  if (c1 <= c0 || lists <= 0) return LA_OK;
  const cudaError_t e =
      la_launch(ctx, laswp_lists_kernel<float>, dim3((c1 - c0 + SW_COLS - 1) / SW_COLS), dim3(256), 0,
                ctx->stream, A, ld, (const int*)(ctx->d_swaps + first * SWAP_STRIDE), lists, c0, c1,
                (const int*)ctx->d_err);
  if (e != cudaSuccess) return la_cuda_fail(ctx, e, "laswp_lists_kernel launch");
  ctx->launches++;
  return la_check_launch(ctx, "laswp_lists_kernel");
}
la_status launch_trsm_block_f32(la_ctx ctx, float* A, size_t ld, int j0, int jbo, int c_begin,
                                int c_end) {
  if (c_end <= c_begin || jbo <= 0) return LA_OK;
  if (jbo > TB_R) return LA_INVALID;
  static la_device_once once;
  LA_CUDA(ctx, once.run([](int) {
            return cudaFuncSetAttribute(trsm_block_kernel,
                                        cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)TB_SMEM);
          }));
  const cudaError_t e = la_launch(ctx, trsm_block_kernel, dim3((c_end - c_begin + TB_C - 1) / TB_C),
                                  dim3(256), TB_SMEM, ctx->stream, A, ld, j0, jbo, c_begin, c_end);
  if (e != cudaSuccess) return la_cuda_fail(ctx, e, "trsm_block_kernel launch");
  ctx->launches++;
  return la_check_launch(ctx, "trsm_block_kernel");
}

la_status launch_trsm_rowpanel(la_ctx ctx, bool exact, double* A, double* S, size_t ld, int j0,
                               int jb, int c_begin, int c_end) {
  if (c_end <= c_begin) return LA_OK;
  const cudaError_t e =
      la_launch(ctx, exact ? trsm_cols8_kernel<true> : trsm_cols8_kernel<false>,
                dim3((c_end - c_begin + TC8 - 1) / TC8), dim3(TC8_T), 0, ctx->stream, A,
                (const double*)S, ld, j0, jb, c_begin, c_end);
  if (e != cudaSuccess) return la_cuda_fail(ctx, e, "trsm_cols8_kernel launch");
  ctx->launches++;
  return la_check_launch(ctx, "trsm_cols8_kernel");
}
la_status launch_trsm_rowpanel_f32(la_ctx ctx, float* A, size_t ld, int j0, int jb, int c_begin,
                                   int c_end) {
  if (c_end <= c_begin) return LA_OK;
  if (jb > TRR_W) return LA_INVALID;
  const int grid = (c_end - c_begin + TRR_T - 1) / TRR_T;
  const cudaError_t e = la_launch(ctx, trsm_rowpanel_reg_kernel, dim3(grid), dim3(TRR_T), 0,
                                  ctx->stream, A, ld, j0, jb, c_begin, c_end);
  if (e != cudaSuccess) return la_cuda_fail(ctx, e, "trsm_rowpanel_reg_kernel launch");
  ctx->launches++;
  return la_check_launch(ctx, "trsm_rowpanel_reg_kernel");
}

la_status launch_lu_finish(la_ctx ctx, la_lu h, int* d_flags, int* d_uneven) {
  const int kmin = (int)std::min(h->m, h->n);
  const int smem_rows = 50000;  // 200 KB of int32 (opt-in); larger m replays in global memory
  static la_device_once configured;
  cudaError_t ce = configured.run([&](int) {
    cudaError_t e = cudaFuncSetAttribute(lu_finish_kernel<double>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         smem_rows * (int)sizeof(int));
    if (e == cudaSuccess)
      e = cudaFuncSetAttribute(lu_finish_kernel<float>,
                               cudaFuncAttributeMaxDynamicSharedMemorySize,
                               smem_rows * (int)sizeof(int));
    return e;
  });
  if (ce != cudaSuccess) return la_cuda_fail(ctx, ce, "cudaFuncSetAttribute(lu_finish)");
  const size_t smem = (size_t)std::min((int)h->m, smem_rows) * sizeof(int);
  if (h->d_lu32)
    lu_finish_kernel<float><<<1, LU_FINISH_T, smem, ctx->stream>>>(h->d_ipiv, h->d_piv, (int)h->m, kmin,
                                                            h->d_lu32, h->ld32, d_flags, nullptr,
                                                            smem_rows, ctx->d_err);
  else
    lu_finish_kernel<double><<<1, LU_FINISH_T, smem, ctx->stream>>>(h->d_ipiv, h->d_piv, (int)h->m, kmin,
                                                             h->d_lu, h->ld, d_flags, d_uneven,
                                                             smem_rows, ctx->d_err);
  ctx->launches++;
  return la_check_launch(ctx, "lu_finish_kernel");
}

la_status launch_permute_rows(la_ctx ctx, const uint64_t* d_piv, const double* B, size_t ldb,
                              double* X, size_t ldx, int m, int nrhs) {
  permute_rows_kernel<<<grid_for(ctx, (size_t)m * nrhs), 256, 0, ctx->stream>>>(d_piv, B, ldb, X,
                                                                               ldx, m, nrhs);
  ctx->launches++;
  return la_check_launch(ctx, "permute_rows_kernel");
}

la_status launch_identity_permuted(la_ctx ctx, const uint64_t* d_piv, double* X, size_t ldx,
                                   int m) {
  identity_permuted_kernel<<<grid_for(ctx, (size_t)m * m), 256, 0, ctx->stream>>>(d_piv, X, ldx,
                                                                                  m);
  ctx->launches++;
  return la_check_launch(ctx, "identity_permuted_kernel");
}

la_status launch_permute_cols(la_ctx ctx, const uint64_t* d_piv, const double* X, double* Y, size_t ld,
                              int n) {
  permute_cols_kernel<<<n, 256, 0, ctx->stream>>>(d_piv, X, Y, ld, n);
  ctx->launches++;
  return la_check_launch(ctx, "permute_cols_kernel");
}

la_status launch_det(la_ctx ctx, const double* LU, size_t ld, int n, int pospivsign,
                     double* d_out) {
  det_kernel<<<1, DET_T, 0, ctx->stream>>>(LU, ld, n, pospivsign, d_out);
  ctx->launches++;
  return la_check_launch(ctx, "det_kernel");
}

la_status launch_unpack(la_ctx ctx, int which, const double* LU, size_t ld, int m, int n,
                        const uint64_t* d_piv, double* out) {
  size_t total = (size_t)std::max(m, n) * std::max(m, n);
  unpack_kernel<<<grid_for(ctx, total), 256, 0, ctx->stream>>>(which, LU, ld, m, n, d_piv, out);
  ctx->launches++;
  return la_check_launch(ctx, "unpack_kernel");
}

la_status launch_copy2d(la_ctx ctx, const double* src, size_t lds, double* dst, size_t ldd,
                        int rows, int cols) {
  copy2d_kernel<<<grid_for(ctx, (size_t)rows * cols), 256, 0, ctx->stream>>>(src, lds, dst, ldd,
                                                                             rows, cols);
  ctx->launches++;
  return la_check_launch(ctx, "copy2d_kernel");
}
