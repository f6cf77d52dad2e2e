// FP64 panel factorization on one thread-block cluster: columns
// [j0, j0 + jb), jb <= 32, over rows [j0, m), with partial pivoting by the reference's
// rule (src/decomp/lu.rs:132-160: the first row of maximal |v|, a NaN below the
// diagonal never chosen, one on it never displaced).
//
// What bounds it. Every column needs one exchange over all rows (the pivot and its
// row), and the rank-1 updates need FP64 FMAs, two per clock and SM. The cooperative
// kernel of lu_panel.cu exchanges through global memory at 5 to 11 us per column; here
// up to 16 CTAs of one cluster exchange through distributed shared memory.
//
//   * Q threads per row (neighbouring lanes), thread q with the columns k = q mod Q, in
//     registers for the whole panel, with the row's current position; a pivot exchange
//     swaps two positions and no data. A warp's FMA takes its sub-partition 64 clocks,
//     however few of its lanes are active, so Q spreads few rows over the SM's four
//     pipes: 4 up to 64 rows per CTA, 2 up to 128, else 1. The register window rotates
//     by one slot every Q columns, so that every register index is static.
//   * An element takes its updates in ascending k by FMA and its multiplier as
//     v * (1 / pivot), exactly the operations of lu_panel.cu's FAST form: the two
//     kernels give the same bits.
//   * EXACT keeps, per element, the original a and the running sum s of l_ik u_kj (unfused,
//     ascending k, lu.rs:124-126), forms a - s when a column or a pivot row is reached, and
//     divides by the pivot: the operations of lu_panel.cu's EXACT form.
//   * Column c's updates are split: column c + 1 first, then the candidates of c + 1
//     are found and pushed, and the other columns take their update while the push
//     travels. A candidate row is therefore published one update behind, together
//     with its multiplier, and the pushing warp applies the missing update (one FMA
//     per lane).
//   * Every warp finds the CTA's best candidate for itself and pushes it (row and key,
//     st.async) into the receive slots of some CTAs of the cluster; a warp without rows
//     meanwhile divides (the candidate's reciprocal) and pushes that, so that no CTA
//     divides on its way from the winner to the next candidates. The bytes complete on
//     the receiver's mbarrier. Three slots: a CTA pushes column c + 3 only after it has
//     every push of c + 2, which each CTA sends after its last use of column c's row.
//
// Measured, 32 columns (R rows, us): R = 24 36, 512 49, 2048 63, 4096 84, 8192 138. With one row
// per thread at every R, a division in every thread and 128-row CTAs it was 53, 90, 86, 110 and
// 170; the exchange itself is hidden, and what remains per column is about 550 clocks to
// find and publish the candidate, 650 to push it, 250 to pick the winner, 350 to scale and
// form the next column, and the update (64 clocks per FMA and warp of a sub-partition:
// from 512 rows per CTA on it is half of the time).
// EXACT, 24 to 1000 rows: 69 on average, against 188 for 32 columns of the cooperative kernel.
//
// Waits are bounded (2 s or LA_OPT_WAIT_LIMIT_US): a thread whose wait gives up
// records DERR_PANEL_TIMEOUT, waits for nothing more and pushes nothing more, but
// takes part in every barrier to the end; nothing is written then.
#include "la_internal.cuh"
#include "swap_compose.cuh"

namespace {

constexpr int PW = 32;                       // panel width
constexpr int PMAXC = 16;                    // CTAs of a cluster
constexpr uint32_t PUSH_BYTES = PW * 8 + 16 + 8;  // row; key and position; reciprocal
constexpr unsigned long long WAIT_NS = 2000000000ull;

__device__ __forceinline__ uint32_t sm_addr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ uint32_t peer_addr(const void* local, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(sm_addr(local)), "r"(rank));
  return r;
}
__device__ __forceinline__ void cluster_barrier() {
  asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" :::
                   "memory");
}
__device__ __forceinline__ unsigned long long now_ns() {
  unsigned long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}
__device__ bool wait_pushes(uint64_t* bar, uint32_t parity, int* err, unsigned long long limit) {
  const uint32_t a = sm_addr(bar);
  unsigned long long t0 = 0;
  for (unsigned i = 0;; i++) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(a), "r"(parity)
        : "memory");
    if (done) return true;
    if ((i & 63u) == 63u) {
      if (*reinterpret_cast<volatile int*>(err) != 0) return false;
      const unsigned long long now = now_ns();
      if (t0 == 0) t0 = now;
      else if (now - t0 > limit) {
        atomicCAS(err, 0, (int)DERR_PANEL_TIMEOUT);
        return false;
      }
    }
  }
}

// bits(|v|) + 1 orders like |v|; NaN below the diagonal loses to everything, NaN on it wins.
__device__ __forceinline__ unsigned long long key_of(double v, bool diag) {
  const unsigned long long a = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
  if (a > 0x7ff0000000000000ull) return diag ? ~0ull : 0ull;
  return a + 1ull;
}
// The best (largest key, then lowest position) of the lanes with pos >= 0: returns its lane, -1
// without one. One 32-bit warp reduction where the key's high word decides, else three.
__device__ __forceinline__ int warp_best(unsigned long long key, int pos) {
  const bool in = pos >= 0;
  const unsigned hi = in ? (unsigned)(key >> 32) : 0u;
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  bool e = in && hi == mh;
  unsigned who = __ballot_sync(0xffffffffu, e);
  if (who & (who - 1)) {
    const unsigned ml = __reduce_max_sync(0xffffffffu, e ? (unsigned)key : 0u);
    e = e && (unsigned)key == ml;
    const unsigned mp = __reduce_min_sync(0xffffffffu, e ? (unsigned)pos : 0xffffffffu);
    who = __ballot_sync(0xffffffffu, e && (unsigned)pos == mp);
  }
  return who ? __ffs(who) - 1 : -1;
}

struct Panel64Args {
  double* A;
  const double* S;  // EXACT: the running sums
  size_t ld;
  int m, j0, jb, rpc, vec, stall;
  int* ipiv;
  int* swaps;
  int* err;
  unsigned long long wait_ns;
};

struct __align__(16) PushSlot {
  double row[PW];
  unsigned long long key;
  int pos, pad;
  double rcp, pad2;
};

// FAST: v is the element, v - l u; EXACT: v is its running sum, v + l u.
template <bool EXACT>
__device__ __forceinline__ double term(double v, double l, double u) {
  return EXACT ? __dadd_rn(v, __dmul_rn(l, u)) : fma(-l, u, v);
}
// v[i] = term(v[i], l, u[Q i]) for 1 <= i < n. A switch into the unrolled sequence: an FMA that a
// predicate switches off takes the FP64 pipe as long as any other.
template <int Q, int NV, bool EXACT>
__device__ __forceinline__ void update_tail(double (&v)[NV], double l, const double* u, int n) {
#define LA_U(i) \
  case (i) + 1: \
    if ((i) < NV) v[(i) % NV] = term<EXACT>(v[(i) % NV], l, u[Q * (i)]); \
    [[fallthrough]];
  switch (n) {
    LA_U(31) LA_U(30) LA_U(29) LA_U(28) LA_U(27) LA_U(26) LA_U(25) LA_U(24)
    LA_U(23) LA_U(22) LA_U(21) LA_U(20) LA_U(19) LA_U(18) LA_U(17) LA_U(16)
    LA_U(15) LA_U(14) LA_U(13) LA_U(12) LA_U(11) LA_U(10) LA_U(9) LA_U(8)
    LA_U(7) LA_U(6) LA_U(5) LA_U(4) LA_U(3) LA_U(2) LA_U(1)
    default: break;
  }
#undef LA_U
}

// T threads with rows and one more warp, for the reciprocals.
template <int T, int Q, bool EXACT>
__global__ void __launch_bounds__(T + 32, 1) panel_cluster64_kernel(const Panel64Args p) {
  constexpr int NW = T / 32;
  constexpr int NV = PW / Q;  // values per thread: columns q, q + Q, ...
  __shared__ PushSlot recv[3][PMAXC];
  constexpr int NS = EXACT ? NV : 1;
  __shared__ double wrow[2][NW][PW], wsum[EXACT ? 2 : 1][NW][EXACT ? PW : 1];
  __shared__ double wl[2][NW];  // the published row's multiplier of the previous column
  __shared__ unsigned long long wkey[2][NW];
  __shared__ int wpos[2][NW];
  __shared__ __align__(8) uint64_t rbar[3];
  __shared__ int s_atp[SWAP_SLOTS], s_atr[SWAP_SLOTS];

  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int g = (int)rank, C = (int)gridDim.x;  // one cluster per launch
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int jb = p.jb;
  const int row0 = p.j0 + g * p.rpc;
  const int nrows = max(0, min(p.rpc, p.m - row0));

  if (tid < 3)
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sm_addr(&rbar[tid])));
  if (tid == 0) asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");

  // Before the wait for the kernel ahead: every CTA's receive barriers are initialised before any
  // push.
  cluster_barrier();
  la_pdl_wait();
  la_pdl_trigger();
  bool live = *reinterpret_cast<volatile int*>(p.err) == 0;
  double v[NV], sm[NS];  // EXACT: a and s
  const int q = lane % Q, lr = tid / Q;
  int pos = tid < T && lr < nrows ? row0 + lr : -1;
  {
    const double* src = p.A + (size_t)(pos >= 0 ? pos : p.j0) * p.ld + p.j0;
    if (Q == 1 && p.vec && jb == PW) {
#pragma unroll
      for (int k = 0; k < NV; k += 2) {
        const double2 t = pos >= 0 ? *reinterpret_cast<const double2*>(src + k) : make_double2(0, 0);
        v[k] = t.x;
        v[k + 1] = t.y;
      }
    } else {
#pragma unroll
      for (int i = 0; i < NV; i++) v[i] = pos >= 0 && q + Q * i < jb ? src[q + Q * i] : 0.0;
    }
    if (EXACT) {
      const double* ssrc = p.S + (size_t)(pos >= 0 ? pos : p.j0) * p.ld + p.j0;
#pragma unroll
      for (int i = 0; i < NS; i++) sm[i] = pos >= 0 && q + Q * i < jb ? ssrc[q + Q * i] : 0.0;
    }
  }

  // This warp's first target: its receive slots and barriers. The last warp sends the reciprocals,
  // a lane to each CTA.
  const uint32_t to0 = (uint32_t)(warp < NW ? warp : lane) % (uint32_t)C;
  const uint32_t dst0 = peer_addr(&recv[0][g], to0), bar0 = peer_addr(&rbar[0], to0);

  int na = 0;                     // the last warp of CTA 0: slots of the composed interchanges
  bool act = false;               // this row took part in the previous column's update,
  double lp = 0.0;                // with this multiplier
  const double* uprev = nullptr;  // and this pivot row
  for (int cb = 0; cb < jb; cb += Q) {
    // one copy of the body (four of them outgrew the instruction cache: 2750 against 2200 clocks
    // per column with 32 rows per CTA)
#pragma unroll 1
    for (int s = 0; s < Q; s++) {  // column c = cb + s: slot 0 of the threads q == s
      const int c = cb + s;
      if (c >= jb) break;
      const int j = p.j0 + c, par = c & 1, slot = c % 3;
      // this warp's candidate of column c, its row one update behind
      if (warp < NW) {
        const bool mine = q == s && pos >= j;
        const unsigned long long key = key_of(EXACT ? __dsub_rn(v[0], sm[0]) : v[0], pos == j);
        const int src = warp_best(key, mine ? pos : -1);
        if (src >= 0 && lane / Q == src / Q) {
          double* dst = wrow[par][warp] + cb + q;
#pragma unroll
          for (int i = 0; i < NV; i++)
            if (cb + Q * i < jb) dst[Q * i] = v[i];
          if (EXACT) {
            double* sdst = wsum[par % (EXACT ? 2 : 1)][warp] + cb + q;
#pragma unroll
            for (int i = 0; i < NS; i++)
              if (cb + Q * i < jb) sdst[Q * i] = sm[i];
          }
          if (lane == src) {
            wl[par][warp] = lp;
            wkey[par][warp] = key;
            wpos[par][warp] = pos;
          }
        }
        if (src < 0 && lane == 0) {
          wkey[par][warp] = 0ull;
          wpos[par][warp] = -1;
        }
      }
      __syncthreads();
      // the CTA's best, its row with the previous column's update, to the cluster
      const unsigned long long wk = lane < NW ? wkey[par][lane % NW] : 0ull;
      const int wp = lane < NW ? wpos[par][lane % NW] : -1;
      const int w = warp_best(wk, wp);
      if (live && warp < NW) {
        double t = 0.0;
        if (w >= 0 && lane >= c) {
          t = wrow[par][w][lane];
          if (EXACT) {
            double sl = wsum[par % (EXACT ? 2 : 1)][w][lane % (EXACT ? PW : 1)];
            if (c > 0 && lane > c) sl = term<true>(sl, wl[par][w], uprev[lane]);
            t = __dsub_rn(t, sl);
          } else if (c > 0 && lane > c) {
            t = term<false>(t, wl[par][w], uprev[lane]);
          }
        }
        for (int to = warp; to < C; to += NW) {
          uint32_t bar = bar0 + slot * 8, dst = dst0 + slot * (uint32_t)sizeof(recv[0]);
          if (to != warp) {
            bar = peer_addr(&rbar[slot], (uint32_t)to);
            dst = peer_addr(&recv[slot][g], (uint32_t)to);
          }
          asm volatile(
              "st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(
                  dst + (uint32_t)lane * 8),
              "l"(__double_as_longlong(t)), "r"(bar)
              : "memory");
          if (lane == (w >= 0 ? w : 0))
            asm volatile(
                "st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, "
                "%4}, [%5];" ::"r"(dst + (uint32_t)offsetof(PushSlot, key)),
                "r"((unsigned)wk), "r"((unsigned)(wk >> 32)), "r"(w >= 0 ? wp : -1), "r"(0), "r"(bar)
                : "memory");
        }
      } else if (live) {
        const double rcp = EXACT ? 1.0 : 1.0 / (w >= 0 ? wrow[par][w][c] : 1.0);
        if (lane < C)
          asm volatile(
              "st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(
                  dst0 + slot * (uint32_t)sizeof(recv[0]) + (uint32_t)offsetof(PushSlot, rcp)),
              "l"(__double_as_longlong(rcp)), "r"(bar0 + slot * 8)
              : "memory");
        if (lane == 0)
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                           sm_addr(&rbar[slot])),
                       "r"((uint32_t)(C + p.stall) * PUSH_BYTES)
                       : "memory");
      }
      // the previous column's update of the columns after c, while the pushes travel
      if (act) {
        const double* u = uprev + cb + q;
        const int nt = (jb - cb + Q - 1) / Q;  // slots with cb + Q i < jb
        if (EXACT) {
          if (Q > 1 && s < Q - 1 && q > s) sm[0] = term<true>(sm[0], lp, u[0]);
          update_tail<Q, NS, true>(sm, lp, u, nt);
        } else {
          if (Q > 1 && s < Q - 1 && q > s) v[0] = term<false>(v[0], lp, u[0]);
          update_tail<Q, NV, false>(v, lp, u, nt);
        }
      }
      if (live) live = wait_pushes(&rbar[slot], (uint32_t)((c / 3) & 1), p.err, p.wait_ns);
      live = __all_sync(0xffffffffu, live);
      // the winner and its row
      const PushSlot& mine = recv[slot][lane % PMAXC];
      const int cpos = lane < C && live ? mine.pos : -1;
      const int src = warp_best(mine.key, cpos);
      // a failed wait: no use is made of what follows
      const int piv = src >= 0 ? __shfl_sync(0xffffffffu, cpos, src) : j;
      const PushSlot& win = recv[slot][src >= 0 ? src : 0];
      const double* u = win.row;
      act = false;
      if (pos == piv) {
        pos = j;  // the pivot row keeps its values
      } else {
        if (pos == j) pos = piv;  // the displaced row takes its place
        act = pos > j;
      }
      // the multiplier, from the row's thread of column c to its others; a zero pivot (key 1)
      // leaves the column as it is
      if (EXACT) {
        if (act && q == s) {
          const double x = __dsub_rn(v[0], sm[0]);
          v[0] = win.key != 1ull ? x / u[c] : x;
          sm[0] = 0.0;
        }
      } else if (act && q == s && win.key != 1ull) {
        v[0] = v[0] * win.rcp;
      }
      lp = Q == 1 ? v[0] : __shfl_sync(0xffffffffu, v[0], lane / Q * Q + s);
      if (act && c + 1 < jb) {
        double(&x)[EXACT ? NS : NV] = [&]() -> double(&)[EXACT ? NS : NV] {
          if constexpr (EXACT) return sm;
          else return v;
        }();
        if (s + 1 < Q) {
          if (q == s + 1) x[0] = term<EXACT>(x[0], lp, u[c + 1]);
        } else if (q == 0) {
          x[1] = term<EXACT>(x[1], lp, u[c + 1]);
        }
      }
      uprev = u;
      if (g == 0 && warp == NW) {
        if (lane == 0) p.ipiv[j] = piv;
        compose_step(j, piv, na, s_atp, s_atr, lane);
      }
    }
    const double t = v[0];
#pragma unroll
    for (int i = 0; i < NV - 1; i++) v[i] = v[i + 1];
    v[NV - 1] = t;
    if (EXACT) {
      const double ts = sm[0];
#pragma unroll
      for (int i = 0; i < NS - 1; i++) sm[i] = sm[i + 1];
      sm[NS - 1] = ts;
    }
  }
  const bool ok = __syncthreads_and(live ? 1 : 0) != 0;
  cluster_barrier();  // no CTA leaves while pushes into its shared memory may be in flight
  if (!ok) return;
  // one rotation per Q columns so far; NV bring every value back to its column
  for (int r = (jb + Q - 1) / Q; r < NV; r++) {
    const double t = v[0];
#pragma unroll
    for (int i = 0; i < NV - 1; i++) v[i] = v[i + 1];
    v[NV - 1] = t;
    if (EXACT) {
      const double ts = sm[0];
#pragma unroll
      for (int i = 0; i < NS - 1; i++) sm[i] = sm[i + 1];
      sm[NS - 1] = ts;
    }
  }
  if (EXACT)
#pragma unroll
    for (int i = 0; i < NS; i++) v[i] = __dsub_rn(v[i], sm[i]);
  if (pos >= 0) {
    double* dst = p.A + (size_t)pos * p.ld + p.j0;
    if (Q == 1 && p.vec && jb == PW) {
#pragma unroll
      for (int k = 0; k < NV; k += 2)
        *reinterpret_cast<double2*>(dst + k) = make_double2(v[k], v[k + 1]);
    } else {
#pragma unroll
      for (int i = 0; i < NV; i++)
        if (q + Q * i < jb) dst[q + Q * i] = v[i];
    }
  }
  if (g == 0 && warp == NW) compose_emit(na, p.swaps, s_atp, s_atr, lane);
}

// CTAs per cluster: LA_UNSUPPORTED (nothing launched) where such a cluster cannot be resident.
template <int T, int Q, bool EXACT>
la_status launch_t(la_ctx ctx, cudaStream_t st, int C, const Panel64Args& a) {
  static unsigned ok_for[LA_MAX_DEVICES];  // bit C: a cluster of C CTAs can be resident
  static la_device_once once;
  const int dev = la_current_device();
  if (dev < 0 || dev >= LA_MAX_DEVICES) return LA_UNSUPPORTED;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = C;
  at[0].val.clusterDim.y = 1;
  at[0].val.clusterDim.z = 1;
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(C);
  cfg.blockDim = dim3(T + 32);
  cfg.stream = st;
  cfg.attrs = at;
  once.run([](int d) {
    ok_for[d] = 0;
    if (cudaFuncSetAttribute(panel_cluster64_kernel<T, Q, EXACT>,
                             cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess)
      for (int c = 1; c <= PMAXC; c *= 2) {
        cudaLaunchAttribute ca;
        ca.id = cudaLaunchAttributeClusterDimension;
        ca.val.clusterDim.x = c;
        ca.val.clusterDim.y = 1;
        ca.val.clusterDim.z = 1;
        cudaLaunchConfig_t q = {};
        q.gridDim = dim3(c);
        q.blockDim = dim3(T + 32);
        q.attrs = &ca;
        q.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, panel_cluster64_kernel<T, Q, EXACT>, &q) == cudaSuccess && n > 0)
          ok_for[d] |= 1u << c;
      }
    cudaGetLastError();
    return cudaSuccess;
  });
  if (!(ok_for[dev] >> C & 1u)) return LA_UNSUPPORTED;
  cfg.numAttrs = ctx->pdl_now ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, panel_cluster64_kernel<T, Q, EXACT>, a);
  if (e != cudaSuccess) return la_cuda_fail(ctx, e, "cudaLaunchKernelEx(panel_cluster64)");
  ctx->launches++;
  return LA_OK;
}

}  // namespace

// Returns LA_UNSUPPORTED (nothing launched) when the panel does not fit one cluster: more than 32
// columns, 8192 rows or (EXACT, with twice the registers per element) 4096, or no such cluster on
// this device; the cooperative kernel takes it then. S: the running sums of EXACT, else null.
la_status launch_panel_cluster64(la_ctx ctx, cudaStream_t st, double* A, const double* S, size_t ld,
                                 int m, int j0, int jb, int* d_ipiv) {
  const int R = m - j0;
  if (R <= 0 || jb <= 0) return LA_OK;
  static_assert(PANEL64_ROWS == PMAXC * 512, "rows of the largest CTA");
  if (jb > PW || R > PANEL64_ROWS / (S ? 2 : 1)) return LA_UNSUPPORTED;
  // 32 rows per CTA until the cluster is full (R = 256: 51 us, with 128 rows per CTA 82)
  int C = 1;
  while (C < PMAXC && R > C * 32) C *= 2;
  Panel64Args a;
  a.A = A;
  a.S = S;
  a.ld = ld;
  a.m = m;
  a.j0 = j0;
  a.jb = jb;
  a.rpc = (R + C - 1) / C;
  a.vec = ld % 2 == 0 && j0 % 2 == 0 && reinterpret_cast<uintptr_t>(A) % 16 == 0 ? 1 : 0;
  a.stall = 0;
  if (ctx->inject_panel_stall > 0 && --ctx->inject_panel_stall == 0) a.stall = 1;
  a.ipiv = d_ipiv;
  a.swaps = ctx->swaps();
  a.err = ctx->d_err;
  a.wait_ns = ctx->wait_limit_us > 0 ? (unsigned long long)ctx->wait_limit_us * 1000ull : WAIT_NS;
  if (S) {
    if (a.rpc <= 64) return launch_t<256, 4, true>(ctx, st, C, a);
    if (a.rpc <= 128) return launch_t<256, 2, true>(ctx, st, C, a);
    return launch_t<512, 2, true>(ctx, st, C, a);
  }
  if (a.rpc <= 64) return launch_t<256, 4, false>(ctx, st, C, a);
  if (a.rpc <= 128) return launch_t<256, 2, false>(ctx, st, C, a);
  if (a.rpc <= 256) return launch_t<256, 1, false>(ctx, st, C, a);
  return launch_t<512, 1, false>(ctx, st, C, a);
}
