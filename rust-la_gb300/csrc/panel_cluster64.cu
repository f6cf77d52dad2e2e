// FP64 panel factorization (FAST arithmetic) on one thread-block cluster: columns
// [j0, j0 + jb), jb <= 32, over rows [j0, m), with partial pivoting by the reference's
// rule (src/decomp/lu.rs:132-160: the first row of maximal |v|, a NaN below the
// diagonal never chosen, one on it never displaced).
//
// What bounds it. Every column needs one exchange over all rows (the pivot and its
// row), and the rank-1 updates need FP64 FMAs, two per clock and SM. The cooperative
// kernel of lu_panel.cu exchanges through global memory at 5 to 11 us per column; here
// up to 16 CTAs of one cluster exchange through distributed shared memory.
//
//   * One row per thread, its 32 values in registers for the whole panel, with the
//     row's current position; a pivot exchange swaps two positions and no data. The
//     register window rotates by one slot per column, so that the current column is
//     slot 0 and every register index is static.
//   * An element takes its updates in ascending k by FMA and its multiplier as
//     v * (1 / pivot), exactly the operations of lu_panel.cu's FAST form: the two
//     kernels give the same bits.
//   * Column c's updates are split: column c + 1 first, then the candidates of c + 1
//     are found and pushed, and the other columns take their update while the push
//     travels. A candidate row is therefore published one update behind, together
//     with its multiplier, and the pushing warp applies the missing update (one FMA
//     per lane).
//   * Every warp finds the CTA's best candidate for itself and pushes it (row and key,
//     272 bytes, st.async) into the receive slot of one CTA of the cluster; the bytes
//     complete on the receiver's mbarrier. Three slots: a CTA pushes column c + 3 only
//     after it has every push of c + 2, which each CTA sends after its last use of
//     column c's row.
//
// Waits are bounded (2 s or LA_OPT_WAIT_LIMIT_US): a thread whose wait gives up
// records DERR_PANEL_TIMEOUT, waits for nothing more and pushes nothing more, but
// takes part in every barrier to the end; nothing is written then.
#include "la_internal.cuh"
#include "swap_compose.cuh"

namespace {

constexpr int PW = 32;                       // panel width
constexpr int PMAXC = 16;                    // CTAs of a cluster
constexpr uint32_t PUSH_BYTES = PW * 8 + 16;  // row, key, position
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
// The best (largest key, then lowest position) of the lanes with pos >= 0; src is its lane, -1
// without one. Three 32-bit warp reductions.
__device__ __forceinline__ int warp_best(unsigned long long key, int pos, unsigned long long& bk,
                                         int& bp) {
  const bool in = pos >= 0;
  const unsigned hi = in ? (unsigned)(key >> 32) : 0u;
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const bool e1 = in && hi == mh;
  const unsigned ml = __reduce_max_sync(0xffffffffu, e1 ? (unsigned)key : 0u);
  const bool e2 = e1 && (unsigned)key == ml;
  const unsigned mp = __reduce_min_sync(0xffffffffu, e2 ? (unsigned)pos : 0xffffffffu);
  bk = (unsigned long long)mh << 32 | ml;
  bp = (int)mp;
  const unsigned who = __ballot_sync(0xffffffffu, e2 && (unsigned)pos == mp);
  return who ? __ffs(who) - 1 : -1;
}

struct Panel64Args {
  double* A;
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
};

template <int T>
__global__ void __launch_bounds__(T, 1) panel_cluster64_kernel(const Panel64Args p) {
  la_pdl_wait();
  la_pdl_trigger();
  constexpr int NW = T / 32;
  __shared__ PushSlot recv[3][PMAXC];
  __shared__ double wrow[2][NW][PW];
  __shared__ double wl[2][NW];  // the published row's multiplier of the previous column
  __shared__ unsigned long long wkey[2][NW];
  __shared__ int wpos[2][NW];
  __shared__ __align__(8) uint64_t rbar[3];
  __shared__ int s_pivs[PW];
  __shared__ int s_atp[SWAP_SLOTS], s_atr[SWAP_SLOTS];

  uint32_t rank;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
  const int g = (int)rank, C = (int)gridDim.x;  // one cluster per launch
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int jb = p.jb;
  const int row0 = p.j0 + g * p.rpc;
  const int nrows = max(0, min(p.rpc, p.m - row0));
  bool live = *reinterpret_cast<volatile int*>(p.err) == 0;

  if (tid < 3)
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(sm_addr(&rbar[tid])));
  if (tid == 0) asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");

  double v[PW];
  int pos = tid < nrows ? row0 + tid : -1;
  {
    const double* src = p.A + (size_t)(pos >= 0 ? pos : p.j0) * p.ld + p.j0;
    if (p.vec && jb == PW) {
#pragma unroll
      for (int k = 0; k < PW; k += 2) {
        const double2 t = pos >= 0 ? *reinterpret_cast<const double2*>(src + k) : make_double2(0, 0);
        v[k] = t.x;
        v[k + 1] = t.y;
      }
    } else {
#pragma unroll
      for (int k = 0; k < PW; k++) v[k] = pos >= 0 && k < jb ? src[k] : 0.0;
    }
  }
  cluster_barrier();  // every CTA's receive barriers are initialised before any push

  bool act = false;                // this row took part in the previous column's update
  const double* uprev = nullptr;   // the previous column's pivot row
  for (int c = 0; c < jb; c++) {
    const int j = p.j0 + c, par = c & 1, slot = c % 3;
    // candidates of column c (slot 0 holds it, every update applied)
    {
      unsigned long long bk;
      int bp;
      const int src =
          warp_best(key_of(v[0], pos == j), pos >= j ? pos : -1, bk, bp);
      if (src == lane) {
        double* dst = wrow[par][warp] + c;
#pragma unroll
        for (int q = 0; q < PW; q += 4)
          if (c + q < jb)
#pragma unroll
            for (int i = q; i < q + 4; i++)
              if (c + i < PW) dst[i] = v[i];
        wl[par][warp] = c > 0 ? v[PW - 1] : 0.0;
      }
      if (lane == 0) {
        wkey[par][warp] = bk;
        wpos[par][warp] = src >= 0 ? bp : -1;
      }
    }
    __syncthreads();
    // the CTA's best, and its row with the previous column's update, to the cluster
    {
      unsigned long long bk;
      int bp;
      const int w = warp_best(lane < NW ? wkey[par][lane % NW] : 0ull,
                              lane < NW ? wpos[par][lane % NW] : -1, bk, bp);
      if (live) {
        double t = 0.0;
        if (w >= 0 && lane >= c) {
          t = wrow[par][w][lane];
          if (c > 0 && lane > c) t = fma(-wl[par][w], uprev[lane], t);
        }
        for (int to = warp; to < C; to += NW) {
          const uint32_t bar = peer_addr(&rbar[slot], (uint32_t)to);
          asm volatile(
              "st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(
                  peer_addr(&recv[slot][g].row[lane], (uint32_t)to)),
              "l"(__double_as_longlong(t)), "r"(bar)
              : "memory");
          if (lane == 0)
            asm volatile(
                "st.async.shared::cluster.mbarrier::complete_tx::bytes.v4.b32 [%0], {%1, %2, %3, "
                "%4}, [%5];" ::"r"(peer_addr(&recv[slot][g].key, (uint32_t)to)),
                "r"((unsigned)bk), "r"((unsigned)(bk >> 32)), "r"(w >= 0 ? bp : -1), "r"(0), "r"(bar)
                : "memory");
        }
        if (tid == 0)
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                           sm_addr(&rbar[slot])),
                       "r"((uint32_t)(C + p.stall) * PUSH_BYTES)
                       : "memory");
      }
    }
    // the previous column's update of the columns after c, while the pushes travel
    if (act) {
      const double l = -v[PW - 1];
#pragma unroll
      for (int q = 0; q < PW; q += 4)
        if (c + q < jb)
#pragma unroll
          for (int i = q; i < q + 4; i++)
            if (i > 0 && c + i < PW) v[i] = fma(l, uprev[c + i], v[i]);
    }
    if (live) live = wait_pushes(&rbar[slot], (uint32_t)((c / 3) & 1), p.err, p.wait_ns);
    live = __all_sync(0xffffffffu, live);
    // the winner and its row
    unsigned long long bk;
    int piv;
    const int src = warp_best(lane < C ? recv[slot][lane % PMAXC].key : 0ull,
                              lane < C && live ? recv[slot][lane % PMAXC].pos : -1, bk, piv);
    const double* u = recv[slot][src >= 0 ? src : 0].row;
    if (!live || src < 0) piv = j;  // a failed wait: no use is made of what follows
    const double d = u[c];
    const double l = d != 0.0 ? v[0] * (1.0 / d) : v[0];
    act = false;
    if (pos == piv) {
      pos = j;  // the pivot row keeps its values
    } else {
      if (pos == j) pos = piv;  // the displaced row takes its place
      act = pos > j;
    }
    if (act) {
      v[0] = l;
      if (c + 1 < jb) v[1] = fma(-l, u[c + 1], v[1]);
    }
    uprev = u;
    const double t = v[0];
#pragma unroll
    for (int k = 0; k < PW - 1; k++) v[k] = v[k + 1];
    v[PW - 1] = t;
    if (g == 0 && tid == 0) {
      p.ipiv[j] = piv;
      s_pivs[c] = piv;
    }
  }
  const bool ok = __syncthreads_and(live ? 1 : 0) != 0;
  cluster_barrier();  // no CTA leaves while pushes into its shared memory may be in flight
  if (!ok) return;
  // jb rotations so far; 32 bring every value back to its column
  for (int r = jb; r < PW; r++) {
    const double t = v[0];
#pragma unroll
    for (int k = 0; k < PW - 1; k++) v[k] = v[k + 1];
    v[PW - 1] = t;
  }
  if (pos >= 0) {
    double* dst = p.A + (size_t)pos * p.ld + p.j0;
    if (p.vec && jb == PW) {
#pragma unroll
      for (int k = 0; k < PW; k += 2)
        *reinterpret_cast<double2*>(dst + k) = make_double2(v[k], v[k + 1]);
    } else {
#pragma unroll
      for (int k = 0; k < PW; k++)
        if (k < jb) dst[k] = v[k];
    }
  }
  if (g == 0 && warp == 0)
    compose_swaps_warp(s_pivs, jb, p.j0, false, nullptr, p.swaps, s_atp, s_atr, lane);
}

// CTAs per cluster: LA_UNSUPPORTED (nothing launched) where such a cluster cannot be resident.
template <int T>
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
  cfg.blockDim = dim3(T);
  cfg.stream = st;
  cfg.attrs = at;
  once.run([](int d) {
    ok_for[d] = 0;
    if (cudaFuncSetAttribute(panel_cluster64_kernel<T>,
                             cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess)
      for (int c = 1; c <= PMAXC; c *= 2) {
        cudaLaunchAttribute ca;
        ca.id = cudaLaunchAttributeClusterDimension;
        ca.val.clusterDim.x = c;
        ca.val.clusterDim.y = 1;
        ca.val.clusterDim.z = 1;
        cudaLaunchConfig_t q = {};
        q.gridDim = dim3(c);
        q.blockDim = dim3(T);
        q.attrs = &ca;
        q.numAttrs = 1;
        int n = 0;
        if (cudaOccupancyMaxActiveClusters(&n, panel_cluster64_kernel<T>, &q) == cudaSuccess && n > 0)
          ok_for[d] |= 1u << c;
      }
    cudaGetLastError();
    return cudaSuccess;
  });
  if (!(ok_for[dev] >> C & 1u)) return LA_UNSUPPORTED;
  cfg.numAttrs = ctx->pdl_now ? 2 : 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, panel_cluster64_kernel<T>, a);
  if (e != cudaSuccess) return la_cuda_fail(ctx, e, "cudaLaunchKernelEx(panel_cluster64)");
  ctx->launches++;
  return LA_OK;
}

}  // namespace

// Returns LA_UNSUPPORTED (nothing launched) when the panel does not fit one cluster: more than 32
// columns or 8192 rows, or no such cluster on this device; the cooperative kernel takes it then.
la_status launch_panel_cluster64(la_ctx ctx, cudaStream_t st, double* A, size_t ld, int m, int j0,
                                 int jb, int* d_ipiv) {
  const int R = m - j0;
  if (R <= 0 || jb <= 0) return LA_OK;
  if (jb > PW || R > PMAXC * 512) return LA_UNSUPPORTED;
  // 128 rows per CTA until the cluster is full: the FMAs of 128 rows take about as long as an
  // exchange.
  int C = 1;
  while (C < PMAXC && R > C * 128) C *= 2;
  Panel64Args a;
  a.A = A;
  a.ld = ld;
  a.m = m;
  a.j0 = j0;
  a.jb = jb;
  a.rpc = (R + C - 1) / C;
  a.vec = ld % 2 == 0 && j0 % 2 == 0 && reinterpret_cast<uintptr_t>(A) % 16 == 0 ? 1 : 0;
  a.stall = 0;
  if (ctx->inject_panel_stall > 0 && --ctx->inject_panel_stall == 0) a.stall = 1;
  a.ipiv = d_ipiv;
  a.swaps = ctx->d_swaps;
  a.err = ctx->d_err;
  a.wait_ns = ctx->wait_limit_us > 0 ? (unsigned long long)ctx->wait_limit_us * 1000ull : WAIT_NS;
  if (a.rpc <= 128) return launch_t<128>(ctx, st, C, a);
  if (a.rpc <= 256) return launch_t<256>(ctx, st, C, a);
  return launch_t<512>(ctx, st, C, a);
}
