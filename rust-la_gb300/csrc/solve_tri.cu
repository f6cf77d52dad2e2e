// Triangular solves of LUDecomposition::solve (src/decomp/lu.rs:256-275).
//
// Three schedules that apply every term in the same order, so their results are
// bit-identical:
//
// Wavefront (more right-hand sides than the chain takes). One persistent launch per triangle. The rows are cut
// into 32-row blocks and the right-hand sides into groups of 4 columns; a work
// item is (row block, column group), taken by CTAs from an atomic ticket in
// dependency order (forward: top block first; backward: bottom block first),
// so every item a CTA waits for belongs to a CTA that is already running. The
// item's 4 warps hold one column each, lane = row, in registers. For every
// finished block k (in the reference's order) it loads the 32 x 32 tile of
// L (or U) against k into shared memory (prefetched in registers a step
// ahead, since it does not depend on k being finished), waits until the
// column group's progress counter says block k is solved (acquire loads,
// bounded), reads x_k and applies the 32 terms; then it solves its diagonal
// block lane by lane with shuffles, stores x and publishes (release). The
// critical path per block is one tile application and one 32-step diagonal
// solve; the rest of the update work fills the other SMs.
//
// Chain (more than 32 rows, up to CHAIN_MAX_NRHS right-hand sides). The wavefront with 128 rows of
// one column per item; see solve_chain_kernel.
//
// Block steps. One launch per 16-row block step: for the finished block
// [k0, k1),
//   tile 0    : rows of the next block [k1, k2): take the terms of block
//               [k0, k1), then solve the diagonal block (16 sequential steps)
//   tiles 1.. : rows [k2, n): take the terms of block [k0, k1)
// Backward (U, lu.rs:266-275) mirrors it from the bottom, with the division by
// u_kk when a row becomes final. grid.y splits the right-hand sides into
// 32-column chunks. Used for more than 4 * SOLVE_WAVE_MAX_GROUPS right-hand
// sides or when the wavefront is switched off.
//
// Order of the terms of row i (every schedule): forward (unit L, lu.rs:257-263)
// ascending k; backward (U, lu.rs:266-275) descending k, then the division by
// u_ii. EXACT applies each term as x_i = x_i - x_k * l_ik without fusion and
// divides; FAST uses FMA and multiplies by the reciprocal of u_ii (quot).
#include "la_internal.cuh"

namespace {

constexpr int SB = 16;    // block rows of the solve
constexpr int RT = 32;    // rows per update tile
constexpr int CT = 32;    // right-hand-side columns per CTA
constexpr int ST = 256;   // threads

template <bool EXACT, typename T>
__device__ __forceinline__ T apply(T x, T xk, T l) {
  if constexpr (EXACT) return __dsub_rn(x, __dmul_rn(xk, l));
  else return fma(-xk, l, x);
}

// A row's value over its diagonal entry d once its terms are in. EXACT: the
// division of the reference (lu.rs:272, cholesky.rs:127-139). FAST: the
// product with r = RN(1/d), taken before the row's turn, so no division sits
// on the solve's sequential chain (FP64 division is a long instruction
// sequence on this GPU's FP64 pipe); one extra rounding per row, far inside
// the FAST mode's backward-error bound. Both schedules use it, so their
// results stay bit-identical.
template <bool EXACT, typename T>
__device__ __forceinline__ T quot(T v, T d, T r) {
  if constexpr (EXACT) return v / d;
  else return v * r;
}

// UPPER = false: forward with unit L; UPPER = true: backward with U.
// kb_prev = size of the finished block at [k0, k0 + kb_prev) (0: no finished
// block, only solve the block that starts at `next0`).
template <typename T, bool EXACT, bool UPPER>
__global__ void __launch_bounds__(ST)
solve_step_kernel(const T* __restrict__ LU, size_t ld, T* __restrict__ X, size_t ldx,
                  int n, int nrhs, int k0, int kb_prev, int next0, int nextb) {
  __shared__ T xk[SB][CT];        // finished block's solution rows
  __shared__ T lt[RT][SB + 1];    // L/U entries of this tile against the finished block
  __shared__ T dg[SB][SB + 1];    // diagonal block (tile 0)
  __shared__ T xt[RT][CT];        // this tile's rows of X
  const int c0 = blockIdx.y * CT;
  const int tx = threadIdx.x % CT, ty = threadIdx.x / CT;  // ty 0..7
  const int col = c0 + tx;
  const bool colok = col < nrhs;
  const int tile = blockIdx.x;

  // Rows of this tile.
  int r0, rn;
  if (tile == 0) {
    r0 = next0;
    rn = nextb;
  } else if (!UPPER) {
    const int rest0 = next0 + nextb;
    r0 = rest0 + (tile - 1) * RT;
    rn = min(RT, n - r0);
  } else {
    // backward: rest rows are [0, next0), taken from the top
    r0 = (tile - 1) * RT;
    rn = min(RT, next0 - r0);
  }
  if (rn <= 0) return;

  if (kb_prev > 0) {
    for (int i = ty; i < kb_prev; i += ST / CT)
      xk[i][tx] = colok ? X[(size_t)(k0 + i) * ldx + col] : T(0);
    for (int idx = threadIdx.x; idx < rn * kb_prev; idx += ST) {
      const int i = idx / kb_prev, k = idx % kb_prev;
      lt[i][k] = LU[(size_t)(r0 + i) * ld + k0 + k];
    }
  }
  for (int i = ty; i < rn; i += ST / CT) xt[i][tx] = colok ? X[(size_t)(r0 + i) * ldx + col] : T(0);
  if (tile == 0) {
    for (int idx = threadIdx.x; idx < rn * rn; idx += ST) {
      const int i = idx / rn, k = idx % rn;
      dg[i][k] = LU[(size_t)(r0 + i) * ld + r0 + k];
    }
  }
  __syncthreads();

  // Terms of the finished block.
  if (kb_prev > 0) {
    for (int i = ty; i < rn; i += ST / CT) {
      T x = xt[i][tx];
      if (!UPPER) {
        for (int k = 0; k < kb_prev; k++) x = apply<EXACT, T>(x, xk[k][tx], lt[i][k]);
      } else {
        for (int k = kb_prev - 1; k >= 0; k--) x = apply<EXACT, T>(x, xk[k][tx], lt[i][k]);
      }
      xt[i][tx] = x;
    }
  }

  if (tile == 0) {
    __syncthreads();
    if (!UPPER) {
      for (int k = 0; k < rn; k++) {
        const T v = xt[k][tx];
        for (int i = ty; i < rn; i += ST / CT)
          if (i > k) xt[i][tx] = apply<EXACT, T>(xt[i][tx], v, dg[i][k]);
        __syncthreads();
      }
    } else {
      for (int k = rn - 1; k >= 0; k--) {
        if (ty == (k % (ST / CT))) xt[k][tx] = quot<EXACT>(xt[k][tx], dg[k][k], T(1) / dg[k][k]);
        __syncthreads();
        const T v = xt[k][tx];
        for (int i = ty; i < k; i += ST / CT) xt[i][tx] = apply<EXACT, T>(xt[i][tx], v, dg[i][k]);
        __syncthreads();
      }
    }
  }
  __syncthreads();
  if (colok)
    for (int i = ty; i < rn; i += ST / CT) X[(size_t)(r0 + i) * ldx + col] = xt[i][tx];
}

template <typename T, bool EXACT, bool UPPER>
la_status launch_step(la_ctx ctx, const T* LU, size_t ld, T* X, size_t ldx, int n,
                      int nrhs, int k0, int kb_prev, int next0, int nextb) {
  int rest;
  if (!UPPER) rest = n - (next0 + nextb);
  else rest = next0;
  if (kb_prev == 0) rest = 0;
  dim3 grid(1 + (rest + RT - 1) / RT, (nrhs + CT - 1) / CT);
  solve_step_kernel<T, EXACT, UPPER><<<grid, ST, 0, ctx->stream>>>(LU, ld, X, ldx, n, nrhs, k0,
                                                                   kb_prev, next0, nextb);
  ctx->launches++;
  return la_check_launch(ctx, "solve_step_kernel");
}

template <typename T, bool EXACT>
la_status solve_all(la_ctx ctx, const T* LU, size_t ld, T* X, size_t ldx, int n, int nrhs) {
  // Forward: block 0 alone, then one step per finished block.
  const int nb = (n + SB - 1) / SB;
  LA_TRY((launch_step<T, EXACT, false>(ctx, LU, ld, X, ldx, n, nrhs, 0, 0, 0, std::min(SB, n))));
  for (int b = 0; b + 1 < nb; b++) {
    const int k0 = b * SB, kb = std::min(SB, n - k0);
    const int nx0 = k0 + kb, nxb = std::min(SB, n - nx0);
    LA_TRY((launch_step<T, EXACT, false>(ctx, LU, ld, X, ldx, n, nrhs, k0, kb, nx0, nxb)));
  }
  // Backward: last block alone, then upward.
  const int last0 = (nb - 1) * SB;
  LA_TRY((launch_step<T, EXACT, true>(ctx, LU, ld, X, ldx, n, nrhs, 0, 0, last0, n - last0)));
  for (int b = nb - 1; b > 0; b--) {
    const int k0 = b * SB, kb = std::min(SB, n - k0);
    const int nx0 = (b - 1) * SB;
    LA_TRY((launch_step<T, EXACT, true>(ctx, LU, ld, X, ldx, n, nrhs, k0, kb, nx0, SB)));
  }
  return LA_OK;
}


// ---------------------------------------------------------------------------
// Wavefront schedule.

constexpr int WB = 32;                 // rows per block (one lane each)
constexpr int WC = 4;                  // right-hand-side columns per item (one warp each)
constexpr int WT = WB * WC;            // threads
constexpr int WPRE = WB * WB / WT;     // tile elements each thread prefetches
constexpr unsigned long long WAVE_WAIT_NS = 2000000000ull;

__device__ __forceinline__ unsigned long long wave_time() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
__device__ __forceinline__ int wave_ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void wave_st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

// All 32 lanes of a warp wait until *p >= need; every lane's own acquire load
// saw the value, so each lane's later loads see the publisher's stores.
// Returns the smallest value the lanes saw, or -1 after an error elsewhere or
// 2 s without progress (then the error word holds DERR_TRSV_TIMEOUT).
__device__ __forceinline__ int wave_wait(const int* p, int need, int* err) {
  const unsigned full = 0xffffffffu;
  unsigned long long t0 = 0;
  unsigned spins = 0;
  for (;;) {
    const int v = wave_ld_acquire(p);
    if (__all_sync(full, v >= need)) return __reduce_min_sync(full, v);
    if ((++spins & 63u) == 0) {
      int bad = 0;
      if ((threadIdx.x & 31) == 0) {
        if (*reinterpret_cast<volatile int*>(err) != 0) {
          bad = 1;
        } else {
          const unsigned long long now = wave_time();
          if (t0 == 0) t0 = now;
          else if (now - t0 > WAVE_WAIT_NS) {
            atomicCAS(err, 0, (int)DERR_TRSV_TIMEOUT);
            bad = 1;
          }
        }
      }
      if (__shfl_sync(full, bad, 0)) return -1;
    }
  }
}

// Tile s of an item: s < q are the finished blocks in the reference's order,
// s = q the diagonal block. Both are rows [r0, r0 + sb) against the columns
// of block kb = UPPER ? nb - 1 - s : s.
template <typename T>
__device__ __forceinline__ void wave_fetch_tile(const T* __restrict__ LU, size_t ld, int n, int r0,
                                                int sb, int kb, T (&pre)[WPRE]) {
  const int k0 = kb * WB, kbs = min(WB, n - k0);
#pragma unroll
  for (int j = 0; j < WPRE; j++) {
    const int idx = threadIdx.x + WT * j;
    const int r = idx / WB, k = idx % WB;
    pre[j] = (r < sb && k < kbs) ? __ldg(LU + (size_t)(r0 + r) * ld + k0 + k) : T(0);
  }
}

// DIVL: the lower triangle has a non-unit diagonal (a Cholesky factor): each
// row's value is divided by it once its terms are applied.
template <typename T, bool EXACT, bool UPPER, bool DIVL = false>
__global__ void __launch_bounds__(WT)
solve_wave_kernel(const T* __restrict__ LU, size_t ld, T* X, size_t ldx, int n, int nrhs,
                  int nb, int groups, int* ticket, int* prog, int* err) {
  __shared__ T ls[2][WB][WB + 1];
  __shared__ int s_item;
  const unsigned full = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  const int items = nb * groups;
  for (;;) {
    if (tid == 0) s_item = atomicAdd(ticket, 1);
    __syncthreads();
    const int t = s_item;
    if (t >= items) return;
    const int q = t / groups, g = t - q * groups;
    const int b = UPPER ? nb - 1 - q : q;
    const int r0 = b * WB, sb = min(WB, n - r0);
    const int col = g * WC + w;
    const bool colok = col < nrhs;  // warp-uniform
    int* pg = prog + g;

    T x = (lane < sb && colok) ? __ldcg(X + (size_t)(r0 + lane) * ldx + col) : T(0);
    T pre[WPRE];
    wave_fetch_tile<T>(LU, ld, n, r0, sb, UPPER ? nb - 1 : 0, pre);
    int known = 0;       // blocks of this column group known to be solved
    bool fail = false;   // warp-uniform
    T xn = T(0);         // x of the next finished block, when already fetched
    bool have_xn = false;
    for (int s = 0; s <= q; s++) {
      const int buf = s & 1;
      const int kb = UPPER ? nb - 1 - s : s;
      const int kbs = min(WB, n - kb * WB);
#pragma unroll
      for (int j = 0; j < WPRE; j++) {
        const int idx = tid + WT * j;
        ls[buf][idx / WB][idx % WB] = pre[j];
      }
      T xc = T(0);
      if (s < q && colok && !fail) {
        if (have_xn) {
          xc = xn;
        } else {
          if (known < s + 1) {
            const int v = wave_wait(pg, s + 1, err);
            if (v < 0) fail = true;
            else known = v;
          }
          if (!fail && lane < kbs) xc = __ldcg(X + (size_t)(kb * WB + lane) * ldx + col);
        }
      }
      if (s < q) wave_fetch_tile<T>(LU, ld, n, r0, sb, UPPER ? nb - 2 - s : s + 1, pre);
      have_xn = false;
      if (s + 1 < q && colok && !fail && known >= s + 2) {
        const int kn = UPPER ? nb - 2 - s : s + 1;
        xn = (lane < min(WB, n - kn * WB)) ? __ldcg(X + (size_t)(kn * WB + lane) * ldx + col)
                                           : T(0);
        have_xn = true;
      }
      __syncthreads();
      if (!colok || fail) continue;
      const T(*tile)[WB + 1] = ls[buf];
      if (s < q) {
        if (kbs == WB) {
          if (!UPPER) {
#pragma unroll
            for (int k = 0; k < WB; k++) x = apply<EXACT, T>(x, __shfl_sync(full, xc, k), tile[lane][k]);
          } else {
#pragma unroll
            for (int k = WB - 1; k >= 0; k--)
              x = apply<EXACT, T>(x, __shfl_sync(full, xc, k), tile[lane][k]);
          }
        } else {
          if (!UPPER) {
            for (int k = 0; k < kbs; k++) x = apply<EXACT, T>(x, __shfl_sync(full, xc, k), tile[lane][k]);
          } else {
            for (int k = kbs - 1; k >= 0; k--)
              x = apply<EXACT, T>(x, __shfl_sync(full, xc, k), tile[lane][k]);
          }
        }
      } else if (!UPPER && !DIVL) {
        for (int k = 0; k < sb; k++) {
          const T xk = __shfl_sync(full, x, k);
          if (lane > k) x = apply<EXACT, T>(x, xk, tile[lane][k]);
        }
      } else {
        // FAST: lane l takes the reciprocal of its row's diagonal entry once,
        // off the chain; EXACT divides on the chain as the reference does.
        const T rcp = (!EXACT && lane < sb) ? T(1) / tile[lane][lane] : T(1);
        if (!UPPER) {
          // as in the backward case: every lane divides row k's value in lockstep
          for (int k = 0; k < sb; k++) {
            const T xk = quot<EXACT>(__shfl_sync(full, x, k), tile[k][k], __shfl_sync(full, rcp, k));
            if (lane == k) x = xk;
            else if (lane > k) x = apply<EXACT, T>(x, xk, tile[lane][k]);
          }
        } else {
          // Every lane takes row k's undivided value and divides it by u_kk in
          // lockstep (the same operands give the same quotient in every lane),
          // so the division is not a divergent branch on the chain.
          for (int k = sb - 1; k >= 0; k--) {
            const T xk = quot<EXACT>(__shfl_sync(full, x, k), tile[k][k], __shfl_sync(full, rcp, k));
            if (lane == k) x = xk;
            else if (lane < k) x = apply<EXACT, T>(x, xk, tile[lane][k]);
          }
        }
      }
    }
    if (colok && !fail && lane < sb) X[(size_t)(r0 + lane) * ldx + col] = x;
    __threadfence();
    if (__syncthreads_or(fail ? 1 : 0)) return;
    if (tid == 0) wave_st_release(pg, q + 1);
  }
}

// ---------------------------------------------------------------------------
// The wavefront for few right-hand sides: an item is 128 rows of one column, one warp to each of its
// four 32-row blocks, in the order of the solve.
//
// What bounds a solve with few columns is the chain through all n rows: per row a shuffle and one FP64
// FMA (64 clocks of a sub-partition for a warp, whatever its active lanes). With one block per item
// every 32 rows also paid a hand-over through L2 (store, fence, release, poll, load: 2500 clocks) and,
// after it, the whole tile against the block before (2000). Here three of four hand-overs are through
// shared memory, eight rows at a time, so a warp has taken all but the last eight terms when the warp
// before it is done. Each warp stays on its own sub-partition, so that the chain has a pipe to itself.
//   * Every element takes its terms in the same order by the same operations: the same bits as the
//     other two schedules.
//   * A solved value is its own flag: xs holds a NaN that no computation here gives until it is
//     written (a value with these very bits is handed on as the default NaN).
//   * Tiles come by cp.async, one ahead, row-major with 16 bytes of padding: reading 16 bytes of its
//     row per lane is free of bank conflicts.
// Both triangles (us, one block per item and now): n = 512 213, 159; 1000 389, 278; 4096 1521, 1030;
// 8192 3107, 2067.
constexpr int CB = 4;                          // blocks of WB rows per item
template <typename T>
struct ChainTile {
  static constexpr int VN = 16 / (int)sizeof(T);
  static constexpr int P = WB + VN;            // pitch
  static constexpr size_t SMEM = (size_t)CB * 2 * WB * P * sizeof(T);
};
template <typename T>
__device__ __forceinline__ bool unset(T v) {
  if constexpr (sizeof(T) == 8) return __double_as_longlong(v) == -1ll;
  else return __float_as_int(v) == -1;
}
template <typename T>
__device__ __forceinline__ T unset_value() {
  if constexpr (sizeof(T) == 8) return __longlong_as_double(-1ll);
  else return __int_as_float(-1);
}
template <typename T>
__device__ __forceinline__ T settable(T v) {
  if constexpr (sizeof(T) == 8) return unset(v) ? __longlong_as_double(0x7ff8000000000000ll) : v;
  else return unset(v) ? __int_as_float(0x7fc00000) : v;
}
// Blocks of the column known to be solved, in order: counter w of the four counts its block of each
// item. As wave_wait, until that is at least `need`; -1 after an error or without progress. The lanes
// acquire different counters and then read rows released under all four, which takes a __syncwarp: a
// reduction orders no memory.
__device__ __forceinline__ int chain_wait(const int* p, int need, int* err) {
  const unsigned full = 0xffffffffu;
  const int w = threadIdx.x & (CB - 1);
  unsigned long long t0 = 0;
  for (unsigned spins = 1;; spins++) {
    const int done = __reduce_min_sync(full, CB * wave_ld_acquire(p + w) + w);
    if (done >= need) {
      __syncwarp();
      return done;
    }
    if ((spins & 63u) == 0) {
      int bad = 0;
      if ((threadIdx.x & 31) == 0) {
        if (*reinterpret_cast<volatile int*>(err) != 0) {
          bad = 1;
        } else {
          const unsigned long long now = wave_time();
          if (t0 == 0) t0 = now;
          else if (now - t0 > WAVE_WAIT_NS) {
            atomicCAS(err, 0, (int)DERR_TRSV_TIMEOUT);
            bad = 1;
          }
        }
      }
      if (__shfl_sync(full, bad, 0)) return -1;
    }
  }
}
// The tile of rows [r0, r0 + sb) against columns [k0, k0 + kbs) to shared memory, zeros around it; 16
// bytes per copy, or one element where rows are not 16-byte aligned.
template <typename T>
__device__ __forceinline__ void chain_fetch(T* tile, const T* __restrict__ LU, size_t ld, int r0, int sb,
                                            int k0, int kbs, bool vec) {
  constexpr int VN = ChainTile<T>::VN, P = ChainTile<T>::P;
  const int lane = threadIdx.x & 31;
  if (vec) {
    constexpr int PER = WB / VN;  // copies per row
#pragma unroll
    for (int j = 0; j < PER; j++) {
      const int idx = lane + 32 * j, r = idx / PER, k = idx % PER * VN;
      const int have = r < sb ? max(0, min(VN, kbs - k)) : 0;
      const T* src = have ? LU + (size_t)(r0 + r) * ld + k0 + k : LU;
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(
                       (unsigned)__cvta_generic_to_shared(tile + r * P + k)),
                   "l"(src), "r"(have * (int)sizeof(T)));
    }
  } else {
    for (int r = 0; r < WB; r++) {
      const int have = r < sb && lane < kbs;
      const T* src = have ? LU + (size_t)(r0 + r) * ld + k0 + lane : LU;
      asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;" ::"r"(
                       (unsigned)__cvta_generic_to_shared(tile + r * P + lane)),
                   "l"(src), "n"(sizeof(T)), "r"(have ? (int)sizeof(T) : 0));
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
}
// Entries [k, k + VN) of the lane's row.
template <typename T>
__device__ __forceinline__ void chain_row(T (&l)[ChainTile<T>::VN], const T* row, int k) {
  const int4 v = *reinterpret_cast<const int4*>(row + k);
  memcpy(l, &v, 16);
}

template <typename T, bool EXACT, bool UPPER, bool DIVL>
__global__ void __launch_bounds__(CB * 32)
solve_chain_kernel(const T* __restrict__ LU, size_t ld, T* X, size_t ldx, int n, int nrhs, int nb,
                   bool vec, int* ticket, int* prog, int* err) {
  constexpr int VN = ChainTile<T>::VN, P = ChainTile<T>::P;
  extern __shared__ __align__(16) char chain_smem[];
  __shared__ T xs_[CB * WB];
  __shared__ int s_item, s_fail_;
  volatile T* const xs = xs_;
  volatile int* const s_fail = &s_fail_;
  const unsigned full = 0xffffffffu;
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
  T* const tiles = reinterpret_cast<T*>(chain_smem) + (size_t)w * 2 * WB * P;
  const int items = (nb + CB - 1) / CB * nrhs;
  for (;;) {
    if (tid == 0) {
      s_item = atomicAdd(ticket, 1);
      s_fail_ = 0;
    }
    xs[tid] = unset_value<T>();
    __syncthreads();
    const int t = s_item;
    if (t >= items) return;
    const int q = t / nrhs, col = t - q * nrhs, o = CB * q + w;
    int* const pg = prog + CB * col;
    bool fail = false;  // warp-uniform
    if (o < nb) {
      const int b = UPPER ? nb - 1 - o : o;
      const int r0 = b * WB, sb = min(WB, n - r0);
      auto fetch = [&](int s) {
        const int k0 = (UPPER ? nb - 1 - s : s) * WB;
        chain_fetch<T>(tiles + (s & 1) * WB * P, LU, ld, r0, sb, k0, min(WB, n - k0), vec);
      };
      T x = lane < sb ? __ldcg(X + (size_t)(r0 + lane) * ldx + col) : T(0);
      T xn = T(0);
      bool have_xn = false;
      int known = 0;
      fetch(0);
      for (int s = 0; s <= o && !fail; s++) {
        const int kb = UPPER ? nb - 1 - s : s;
        const int kbs = min(WB, n - kb * WB);
        if (s < o) {
          fetch(s + 1);
          asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
          asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncwarp();
        const T* const row = tiles + (s & 1) * WB * P + lane * P;
        T l[VN];
        if (s < CB * q) {
          T xc = xn;
          if (!have_xn) {
            if (known < s + 1) {
              known = chain_wait(pg, s + 1, err);
              if (known < 0) {
                fail = true;
                break;
              }
            }
            xc = lane < kbs ? __ldcg(X + (size_t)(kb * WB + lane) * ldx + col) : T(0);
          }
          have_xn = s + 1 < CB * q && known >= s + 2;
          if (have_xn) {
            const int kn = UPPER ? kb - 1 : kb + 1;
            xn = lane < min(WB, n - kn * WB) ? __ldcg(X + (size_t)(kn * WB + lane) * ldx + col) : T(0);
          }
#pragma unroll
          for (int i = 0; i < WB; i += VN) {
            const int k0 = UPPER ? WB - VN - i : i;
            chain_row<T>(l, row, k0);
#pragma unroll
            for (int j = 0; j < VN; j++) {
              const int e = UPPER ? VN - 1 - j : j;
              const T xk = __shfl_sync(full, xc, k0 + e);
              if (k0 + e < kbs) x = apply<EXACT, T>(x, xk, l[e]);
            }
          }
        } else if (s < o) {
          // the warps before this one, eight rows at a time
#pragma unroll 1
          for (int i = 0; i < WB; i += 8) {
            const int k0 = UPPER ? WB - 8 - i : i;
            T xc;
            for (unsigned spins = 1;; spins++) {
              xc = xs[(s & (CB - 1)) * WB + k0 + (lane & 7)];
              if (__all_sync(full, !unset(xc))) break;
              if ((spins & 63u) == 0 && __any_sync(full, *s_fail)) {
                fail = true;
                break;
              }
            }
            if (fail) break;
#pragma unroll
            for (int h = 0; h < 8; h += VN) {
              const int kh = k0 + (UPPER ? 8 - VN - h : h);
              chain_row<T>(l, row, kh);
#pragma unroll
              for (int j = 0; j < VN; j++) {
                const int e = UPPER ? VN - 1 - j : j;
                const T xk = __shfl_sync(full, xc, (kh + e) & 7);
                if (kh + e < kbs) x = apply<EXACT, T>(x, xk, l[e]);
              }
            }
          }
        } else {
          // FAST: the reciprocals off the chain; EXACT divides on it (see solve_wave_kernel).
          constexpr bool DIV = UPPER || DIVL;
          const T dd = DIV && lane < sb ? row[lane] : T(1);
          const T rcp = DIV && !EXACT ? T(1) / dd : T(1);
#pragma unroll
          for (int i = 0; i < WB; i += VN) {
            const int k0 = UPPER ? WB - VN - i : i;
            chain_row<T>(l, row, k0);
#pragma unroll
            for (int j = 0; j < VN; j++) {
              const int k = k0 + (UPPER ? VN - 1 - j : j);
              if (k < sb) {  // uniform
                if (DIV) {
                  const T v = quot<EXACT>(x, dd, rcp);  // every lane's, row k's is taken
                  if (lane == k) x = v;
                }
                const T xk = __shfl_sync(full, x, k);
                if (UPPER ? lane < k : lane > k) x = apply<EXACT, T>(x, xk, l[k - k0]);
              }
              if (k % 8 == (UPPER ? 0 : 7) && lane / 8 == k / 8) xs[w * WB + lane] = settable(x);
            }
          }
        }
        __syncwarp();
      }
      if (!fail) {
        if (lane < sb) X[(size_t)(r0 + lane) * ldx + col] = x;
        __threadfence();
        __syncwarp();
        if (lane == 0) wave_st_release(pg + w, q + 1);
      } else if (lane == 0) {
        *s_fail = 1;
      }
      asm volatile("cp.async.wait_group 0;" ::: "memory");
    }
    if (__syncthreads_or(fail ? 1 : 0)) return;
  }
}

// Right-hand sides up to which the chain's items are one column each; above, four columns per item
// share each tile's load and the FP64 pipes are busy anyway. Both triangles, us, four columns and one:
// n = 8192: 16 right-hand sides 4053, 3412; 24: 4731, 4593; 32: 5609, 5839. n = 4096: 24: 1912, 1471;
// 64: 2842, 2980. A single block has nothing to hand on, and the chain's body, unrolled over the block with
// its divisions, is read from memory for one pass: whole calls at n = 24, us, four columns and one: EXACT
// 53, 66; FAST 44, 44.
constexpr int CHAIN_MAX_NRHS = 24;
bool chained(int n, int nrhs) { return nrhs <= CHAIN_MAX_NRHS && n > WB; }

// One triangle by solve_chain_kernel; ticket and prog (CB counters per right-hand side) are zero.
template <typename T, bool EXACT, bool UPPER, bool DIVL>
la_status chain(la_ctx ctx, const T* LU, size_t ld, T* X, size_t ldx, int n, int nrhs, int* ticket,
                int* prog) {
  static_assert(2 * CB * CHAIN_MAX_NRHS <= 2 * SOLVE_WAVE_MAX_GROUPS, "progress counters");
  const auto kernel = solve_chain_kernel<T, EXACT, UPPER, DIVL>;
  const size_t smem = ChainTile<T>::SMEM;
  static la_device_once configured;
  LA_CUDA(ctx, configured.run([&](int) {
    return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  }));
  const int nb = (n + WB - 1) / WB;
  const long long items = (long long)((nb + CB - 1) / CB) * nrhs;
  const int cps = ctx->solve_wave > 0 ? ctx->solve_wave : 2;
  const int grid = (int)std::min<long long>(items, (long long)cps * ctx->sm_count);
  const bool vec = ld % ChainTile<T>::VN == 0 && reinterpret_cast<uintptr_t>(LU) % 16 == 0;
  kernel<<<grid, CB * 32, smem, ctx->stream>>>(LU, ld, X, ldx, n, nrhs, nb, vec, ticket, prog, ctx->d_err);
  ctx->launches++;
  return la_check_launch(ctx, "solve_chain_kernel");
}

template <typename T, bool EXACT>
la_status solve_wave(la_ctx ctx, const T* LU, size_t ld, T* X, size_t ldx, int n, int nrhs) {
  const int nb = (n + WB - 1) / WB;
  int* tickets = ctx->d_solve_sync;
  if (chained(n, nrhs)) {
    const size_t counters = CB * (size_t)nrhs;  // of a triangle
    LA_CUDA(ctx, cudaMemsetAsync(tickets, 0, (2 + 2 * counters) * sizeof(int), ctx->stream));
    LA_TRY((chain<T, EXACT, false, false>(ctx, LU, ld, X, ldx, n, nrhs, tickets, tickets + 2)));
    return chain<T, EXACT, true, false>(ctx, LU, ld, X, ldx, n, nrhs, tickets + 1, tickets + 2 + counters);
  }
  const int groups = (nrhs + WC - 1) / WC;
  int* prog_l = tickets + 2;
  int* prog_u = prog_l + groups;
  LA_CUDA(ctx, cudaMemsetAsync(tickets, 0, (2 + 2 * (size_t)groups) * sizeof(int), ctx->stream));
  const long long items = (long long)nb * groups;
  const int grid = (int)std::min<long long>(items, (long long)ctx->solve_wave * ctx->sm_count);
  solve_wave_kernel<T, EXACT, false><<<grid, WT, 0, ctx->stream>>>(
      LU, ld, X, ldx, n, nrhs, nb, groups, tickets, prog_l, ctx->d_err);
  ctx->launches++;
  LA_TRY(la_check_launch(ctx, "solve_wave_kernel"));
  solve_wave_kernel<T, EXACT, true><<<grid, WT, 0, ctx->stream>>>(
      LU, ld, X, ldx, n, nrhs, nb, groups, tickets + 1, prog_u, ctx->d_err);
  ctx->launches++;
  return la_check_launch(ctx, "solve_wave_kernel");
}

// One triangle with the wavefront kernel, right-hand sides in chunks of at
// most 4 * SOLVE_WAVE_MAX_GROUPS columns.
template <bool EXACT, bool UPPER, bool DIVL>
la_status tri_wave(la_ctx ctx, const double* T, size_t ld, double* X, size_t ldx, int n,
                   int nrhs) {
  if (chained(n, nrhs)) {
    int* const sync = ctx->d_solve_sync;
    LA_CUDA(ctx, cudaMemsetAsync(sync, 0, (2 + CB * (size_t)nrhs) * sizeof(int), ctx->stream));
    return chain<double, EXACT, UPPER, DIVL>(ctx, T, ld, X, ldx, n, nrhs, sync, sync + 2);
  }
  const int nb = (n + WB - 1) / WB;
  const int per = WC * SOLVE_WAVE_MAX_GROUPS;
  for (int c0 = 0; c0 < nrhs; c0 += per) {
    const int nr = std::min(per, nrhs - c0);
    const int groups = (nr + WC - 1) / WC;
    int* tickets = ctx->d_solve_sync;
    int* prog = tickets + 2;
    LA_CUDA(ctx, cudaMemsetAsync(tickets, 0, (2 + (size_t)groups) * sizeof(int), ctx->stream));
    const long long items = (long long)nb * groups;
    const int cps = ctx->solve_wave > 0 ? ctx->solve_wave : 2;
    const int grid = (int)std::min<long long>(items, (long long)cps * ctx->sm_count);
    solve_wave_kernel<double, EXACT, UPPER, DIVL><<<grid, WT, 0, ctx->stream>>>(
        T, ld, X + c0, ldx, n, nr, nb, groups, tickets, prog, ctx->d_err);
    ctx->launches++;
    LA_TRY(la_check_launch(ctx, "solve_wave_kernel"));
  }
  return LA_OK;
}

template <typename T, bool EXACT>
la_status solve_any(la_ctx ctx, const T* LU, size_t ld, T* X, size_t ldx, int n, int nrhs) {
  if (ctx->solve_wave > 0 && ctx->d_solve_sync && ctx->sm_count > 0 &&
      (nrhs + WC - 1) / WC <= SOLVE_WAVE_MAX_GROUPS)
    return solve_wave<T, EXACT>(ctx, LU, ld, X, ldx, n, nrhs);
  return solve_all<T, EXACT>(ctx, LU, ld, X, ldx, n, nrhs);
}

}  // namespace

// X (>= n rows, pitch ldx) holds B(piv,:) on entry and the solution of the top
// n rows on exit; rows n.. are untouched (the reference's loops stop at n).
la_status launch_lu_solve(la_ctx ctx, bool exact, const double* LU, size_t ld, double* X,
                          size_t ldx, int n, int nrhs) {
  if (n <= 0 || nrhs <= 0) return LA_OK;
  return exact ? solve_any<double, true>(ctx, LU, ld, X, ldx, n, nrhs)
               : solve_any<double, false>(ctx, LU, ld, X, ldx, n, nrhs);
}

// FP32 factors and right-hand sides (the correction solves of iterative refinement).
la_status launch_lu_solve_f32(la_ctx ctx, const float* LU, size_t ld, float* X, size_t ldx, int n,
                              int nrhs) {
  if (n <= 0 || nrhs <= 0) return LA_OK;
  return solve_any<float, false>(ctx, LU, ld, X, ldx, n, nrhs);
}

// One triangle of a solve by the wavefront kernel: lower (unit diagonal, or
// divide = true for a non-unit one) or upper (always divides). The Cholesky
// solves use it (cholesky.rs:123-141).
la_status launch_tri_wave(la_ctx ctx, bool exact, bool upper, bool divide, const double* T,
                          size_t ld, double* X, size_t ldx, int n, int nrhs) {
  if (n <= 0 || nrhs <= 0) return LA_OK;
  if (!ctx->d_solve_sync || ctx->sm_count <= 0) return LA_UNSUPPORTED;
  if (upper)
    return exact ? tri_wave<true, true, false>(ctx, T, ld, X, ldx, n, nrhs)
                 : tri_wave<false, true, false>(ctx, T, ld, X, ldx, n, nrhs);
  if (divide)
    return exact ? tri_wave<true, false, true>(ctx, T, ld, X, ldx, n, nrhs)
                 : tri_wave<false, false, true>(ctx, T, ld, X, ldx, n, nrhs);
  return exact ? tri_wave<true, false, false>(ctx, T, ld, X, ldx, n, nrhs)
               : tri_wave<false, false, false>(ctx, T, ld, X, ldx, n, nrhs);
}
