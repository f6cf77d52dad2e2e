// FP64 products on the tensor cores by exact splitting.
//
//   C (M x N, f64) = A B,  C -= A B  or  C += A B,  A M x K, B K x N, row-major
//
// GB300 issues about two FP64 FMAs per clock and SM, so a 64 x 64 x 64 FP64 tile
// keeps an SM busy for 66 us and an 8192^3 product the whole chip for 876 ms. Its
// FP16 tensor rate is some 1500 times higher. This file computes the same product
// from FP16 digits (the error-free splitting of Ozaki, Ogita, Oishi and Rump, 2012):
//
//   1. Row i of A is scaled by 2^-ea_i (|a_ik| < 2^ea_i), column j of B by 2^-eb_j,
//      and each value becomes a 64-bit fixed-point number cut into SL = 8 signed
//      digits of 8 bits, d_s in [-128, 128], each exact in FP16:
//        a_ik = 2^ea_i sum_s d_s 2^(-7-8s)  with an error below 2^(ea_i - 64)
//      (none at all for entries within 2^10 of the row's largest).
//   2. tcgen05.mma adds the products of digits s of A and t of B, s + t = g, of up to
//      128 k in the FP32 accumulator g. Every addend is a whole number and every sum
//      at most 8 * 128 * 2^14 = 2^24, so the accumulators are exact. The 28 products
//      with s + t > 7 are below 2^-64 of the scale and left out.
//   3. The epilogue adds the eight accumulators with their weights in two 64-bit
//      integers, over all k, and rounds the sum to a double once.
//
// So an element has one rounding where an FMA chain has K, plus an error of about
// sqrt(K) 2^-64 2^(ea_i + eb_j) from the digits left out.
//
// Which tiles take this path. That last error is relative to the row's and the
// column's largest entries, an FMA chain's to sum_k |a_ik b_kj|. The split kernels
// count, per row and per column, the entries within 2^-5 of the scale; a tile whose
// smallest row count and smallest column count add up to more than 5/4 K has at least
// K/4 k where both are large, so sum |a b| >= K/4 2^-10 2^(ea+eb), and for K >= 48 the
// error left out is below the chain's own (about 0.2 2^-53 sum |a b| for terms of
// random signs). Every other tile (outliers, graded or sparse rows, values that are
// not finite or beyond 2^+-400) goes on a list that fma_tiles_kernel, launched right
// after, works off with FMA chains in ascending k, 64 x 64 tiles as in gemm_f64.cu (it
// ends at once where the list is empty). The decision is made on the device.
//
// Measured on 8192^3 (A and B N(0,1)): 27.9 ms against 876.6 ms by FMA, 36 x 2 x 8192^3 FP16
// operations in all, 1.42 PFLOP/s; rms error against quadruple precision 5 to 17 times smaller than
// the FMA chain's (K = 64 to 2049). What bounds it: the MMAs of 128 k (9.2k clocks at the
// tensor peak) and reading the accumulators after them (about 5k clocks), one after the other, since
// a tile's accumulators fill the tensor memory. For K = 64 (8192 x 8192, 0.40 ms) the integer
// instructions of the rounding bound it (ALU pipe 59 % busy, tensor pipe 26 %, DRAM 16 %).
//
// Layout. 128 x 64 output tiles, one persistent CTA per SM: the eight accumulators of
// a tile fill its 512 tensor-memory columns. Digits are K-major FP16, [digit][row][k];
// one 3-D TMA box brings 32 k of all 8 digits of the tile's rows of A (64 KB) and one
// those of B (32 KB), 64-byte swizzle, two stages. Neighbouring digits of B lie next
// to each other in shared memory and neighbouring accumulators in tensor memory, so
// one tcgen05.mma with N = 256 multiplies a digit of A with four digits of B: 12
// instructions per 16 k instead of 36, and the operands' shared-memory reads stay
// below 128 bytes per clock (N = 64 would need 192).
//   warps 0-15 : epilogue, 32 rows x 16 columns each
//   warp 16    : TMA producer, warp 17 : MMA issuer
// Every wait is bounded as in tma_util.cuh; a CTA that gives up drains its copies and
// MMAs, frees its tensor memory and leaves C's remaining tiles as they are.
#include <cuda.h>

#include "la_internal.cuh"
#include "tma_util.cuh"

namespace {

constexpr int SL = 8;                 // digits per value
constexpr int PM = 128, PN = 64;      // output tile
constexpr int PK = 32;                // k per stage
constexpr int CHUNK_STAGES = 4;       // stages per exact accumulation (128 k)
constexpr int NST = 2;                // stages in shared memory
constexpr uint32_t PA_BYTES = SL * PM * PK * 2;  // 64 KB
constexpr uint32_t PB_BYTES = SL * PN * PK * 2;  // 32 KB
constexpr uint32_t PST_BYTES = PA_BYTES + PB_BYTES;
constexpr int EPI_WARPS = 16;
constexpr int EPI_T = EPI_WARPS * 32;
constexpr int SPLIT_T = EPI_T + 64;
constexpr uint32_t EPI_BYTES = EPI_WARPS * 32 * 8 * 8;  // 32 KB: per warp 32 rows x 8 columns
constexpr size_t SPLIT_SMEM = (size_t)NST * PST_BYTES + EPI_BYTES + 1024;
constexpr int EXP_LIMIT = 400;        // |ea|, |eb| the digits are used for
constexpr int LARGE_BITS = 4;         // "large": exponent within 4 of the largest (2^-5 of the scale)
constexpr int CNT_BAD = -(1 << 29);   // count of a row the digits cannot represent
constexpr int FT = 64, FK = 16;       // FMA tiles: 64 x 64 in slabs of 16 k
constexpr int FMA_T = 256, FMA_PER_SM = 3;

using la_tma::mbar_init;
using la_tma::smem_u32;

__device__ __forceinline__ bool sw_wait(uint64_t* bar, uint32_t parity, int* err) {
  return la_tma::mbar_wait(bar, parity, err, (int)DERR_GEMM_TIMEOUT);
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int x, int y, int z,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes"
      " [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(z), "r"(smem_u32(bar))
      : "memory");
}
// K-major operand in shared memory, 64-byte swizzle: 8-row groups 512 bytes apart.
__device__ __forceinline__ uint64_t sdesc64(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (uint64_t)1 << 16 | (uint64_t)(512u >> 4) << 32 |
         (uint64_t)1 << 46 | (uint64_t)4 << 61;
}
// kind::f16 with FP16 operands and FP32 accumulators, M = 128.
__device__ __forceinline__ constexpr uint32_t idesc_f16(int n) {
  return (1u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(PM >> 4) << 24);
}
__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc,
                                        uint32_t acc) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile(
      "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
          smem_u32(bar))
      : "memory");
}
// Two columns of an accumulator. The wait takes the registers, so that nothing that uses them
// moves above it.
__device__ __forceinline__ void tmem_ld2(uint32_t addr, uint32_t (&r)[2]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];"
               : "=r"(r[0]), "=r"(r[1])
               : "r"(addr));
}
__device__ __forceinline__ void tmem_wait(uint32_t (&r)[SL][2]) {
#define LA_R2(g) "+r"(r[g][0]), "+r"(r[g][1])
  asm volatile("tcgen05.wait::ld.sync.aligned;"
               : LA_R2(0), LA_R2(1), LA_R2(2), LA_R2(3), LA_R2(4), LA_R2(5), LA_R2(6), LA_R2(7)::
                   "memory");
#undef LA_R2
}

// ---- splitting -------------------------------------------------------------------------------

// Fixed-point form of v at scale 2^ea: round(v 2^(63 - ea)), |v| < 2^ea, with the exponent
// arithmetic on the bits (FP64 instructions cost 64 times an integer one here). top = ea - 1 +
// 1023, the biased exponent of the row's largest entry.
__device__ __forceinline__ long long to_fixed(double v, int top) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v);
  const int e = (int)(b >> 52) & 0x7ff;
  unsigned long long m = e ? ((b & 0xfffffffffffffull) | 0x10000000000000ull) : 0ull;
  const int sh = 10 - (top - e);  // denormals are far below 2^(ea - 64) wherever top is admitted
  if (sh >= 0) m <<= sh;
  else if (sh > -55) m = (m + (1ull << (-sh - 1))) >> -sh;
  else m = 0;
  return (long long)b < 0 ? -(long long)m : (long long)m;
}

// The 8 digits of two fixed-point values as FP16 pairs, digit s of both in out[s].
__device__ __forceinline__ void to_digits(long long x0, long long x1, __half2 (&out)[SL]) {
  constexpr unsigned long long MASK = 0x00ffffffffffffffull, HALF = 0x0080808080808080ull;
  const unsigned long long l0 = ((unsigned long long)x0 & MASK) + HALF;
  const unsigned long long l1 = ((unsigned long long)x1 & MASK) + HALF;
  const int t0 = (int)(x0 >> 56) + (int)(l0 >> 56), t1 = (int)(x1 >> 56) + (int)(l1 >> 56);
  out[0] = __halves2half2(__int2half_rn(t0), __int2half_rn(t1));
  const unsigned h0 = (unsigned)(l0 >> 32), h1 = (unsigned)(l1 >> 32);
  const unsigned w0 = (unsigned)l0, w1 = (unsigned)l1;
  const __half2 bias = __halves2half2(__ushort_as_half(0x6480), __ushort_as_half(0x6480));  // 1152
  // digit s is byte 7 - s of the low 56 bits, less 128: both values' bytes b as the halves
  // 1024 + b, less 1024 + 128
#pragma unroll
  for (int s = 1; s < SL; s++) {
    const int byte = 7 - s;
    const unsigned p = __byte_perm(byte >= 4 ? h0 : w0, byte >= 4 ? h1 : w1,
                                   (byte & 3) | (4 + (byte & 3)) << 4);
    const unsigned two = __byte_perm(p, 0x64u, 0x4140);
    __half2 v;
    memcpy(&v, &two, 4);
    out[s] = __hsub2(v, bias);
  }
}

__device__ __forceinline__ int top_of(int maxexp, bool& bad) {
  // maxexp: largest biased exponent of a row or column; 0 where it holds zeros (or denormals,
  // which bad reports)
  bad = maxexp != 0 && (maxexp < 1023 - EXP_LIMIT || maxexp >= 1023 + EXP_LIMIT);
  return bad || maxexp == 0 ? 1023 : maxexp;
}
__device__ __forceinline__ int exp_bits(double v) {
  return (int)((unsigned long long)__double_as_longlong(v) >> 52) & 0x7ff;
}
__device__ __forceinline__ bool is_denormal(double v) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull;
  return b != 0 && b < 0x0010000000000000ull;
}

// Rows of X (R x K, pitch ldx) into digits [SL][R][kp], exps[R] (ea) and cnt[R] (large entries).
// One warp per row, two neighbouring k per lane: a slice's row is written 128 bytes at a time. The
// row is read twice, the second time from L1 or L2 where K is a panel's width.
__global__ void __launch_bounds__(256)
split_rows_kernel(const double* __restrict__ X, size_t ldx, int R, int K, int kp,
                  __half* __restrict__ dig, int* __restrict__ exps, int* __restrict__ cnt,
                  int* nlist) {
  la_pdl_wait();
  la_pdl_trigger();
  if (nlist && blockIdx.x == 0 && threadIdx.x == 0) *nlist = 0;
  const int lane = threadIdx.x & 31;
  const int r = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (r >= R) return;
  const double* x = X + (size_t)r * ldx;
  int me = 0;
  bool den = false;
  for (int k = lane; k < K; k += 32) {
    const double v = x[k];
    me = max(me, exp_bits(v));
    den |= is_denormal(v);
  }
  me = __reduce_max_sync(0xffffffffu, me);
  den = __any_sync(0xffffffffu, den);
  bool bad;
  const int top = top_of(me, bad);
  bad |= me == 0 && den;
  int large = 0;
  const size_t ss = (size_t)R * kp;
  __half* d = dig + (size_t)r * kp;
  for (int k = 2 * lane; k < K; k += 64) {
    const double v0 = x[k], v1 = k + 1 < K ? x[k + 1] : 0.0;
    large += (exp_bits(v0) >= top - LARGE_BITS) + (k + 1 < K && exp_bits(v1) >= top - LARGE_BITS);
    __half2 q[SL];
    to_digits(bad ? 0 : to_fixed(v0, top), bad ? 0 : to_fixed(v1, top), q);
#pragma unroll
    for (int s = 0; s < SL; s++) *reinterpret_cast<__half2*>(d + s * ss + k) = q[s];
  }
  large = __reduce_add_sync(0xffffffffu, large);
  if (lane == 0) {
    exps[r] = top + 1 - 1023;
    cnt[r] = bad ? CNT_BAD : me == 0 ? K : large;
  }
}

// Largest biased exponent of each column of X (K x N) over k [blockIdx.y * kper, ...), and a
// denormal's presence as bit 11, into maxexp (zeroed before).
__global__ void __launch_bounds__(256)
col_exp_kernel(const double* __restrict__ X, size_t ldx, int K, int N, int kper,
               int* __restrict__ maxexp) {
  const int c = blockIdx.x * 32 + (threadIdx.x & 31), ty = threadIdx.x >> 5;
  const int k0 = blockIdx.y * kper, k1 = min(K, k0 + kper);
  if (c >= N) return;
  int me = 0, den = 0;
  for (int k = k0 + ty; k < k1; k += 8) {
    const double v = X[(size_t)k * ldx + c];
    me = max(me, exp_bits(v));
    den |= is_denormal(v);
  }
  if (me) atomicMax(maxexp + c, me);
  if (den) atomicOr(maxexp + N + c, 1);
}

// Columns of X (K x N, pitch ldx), k [blockIdx.y * kper, ...), into digits [SL][N][kp]. 32 columns
// per CTA: 64 k at a time go through shared memory, so that global rows are read 256 bytes at a
// time and a digit's k are written 128 bytes at a time. ALL: the CTA sees every k of its columns
// and finds their exponents itself; else they come from col_exp_kernel and counts are added up.
template <bool ALL>
__global__ void __launch_bounds__(256)
split_cols_kernel(const double* __restrict__ X, size_t ldx, int K, int N, int kp, int kper,
                  const int* __restrict__ maxexp, __half* __restrict__ dig,
                  int* __restrict__ exps, int* __restrict__ cnt) {
  la_pdl_wait();
  la_pdl_trigger();
  __shared__ double tile[64][33];
  __shared__ int s_me[32], s_den[32];
  const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
  const int c0 = blockIdx.x * 32, c = c0 + tx;
  const int kb = ALL ? 0 : blockIdx.y * kper, ke = ALL ? K : min(K, kb + kper);
  if (ALL) {
    if (tid < 32) { s_me[tid] = 0; s_den[tid] = 0; }
    __syncthreads();
    int me = 0, den = 0;
    if (c < N)
      for (int k = ty; k < K; k += 8) {
        const double v = X[(size_t)k * ldx + c];
        me = max(me, exp_bits(v));
        den |= is_denormal(v);
      }
    if (me) atomicMax(&s_me[tx], me);
    if (den) atomicOr(&s_den[tx], 1);
  } else if (tid < 32) {
    s_me[tid] = c < N ? maxexp[c] : 0;
    s_den[tid] = c < N ? maxexp[N + c] : 0;
  }
  __syncthreads();
  const size_t ss = (size_t)N * kp;
  int large[4] = {0, 0, 0, 0};
  for (int k0 = kb; k0 < ke; k0 += 64) {
#pragma unroll
    for (int i = 0; i < 8; i++) {
      const int k = k0 + ty + 8 * i;
      tile[ty + 8 * i][tx] = c < N && k < ke ? X[(size_t)k * ldx + c] : 0.0;
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; i++) {  // warp ty takes columns ty, ty + 8, ...; lane = 2 k
      const int n = ty + 8 * i, k = k0 + 2 * tx;
      if (c0 + n < N && k < ke) {
        bool bad;
        const int top = top_of(s_me[n], bad);
        bad |= s_me[n] == 0 && s_den[n];
        const double v0 = tile[2 * tx][n], v1 = tile[2 * tx + 1][n];
        large[i] += (exp_bits(v0) >= top - LARGE_BITS) + (exp_bits(v1) >= top - LARGE_BITS);
        __half2 q[SL];
        to_digits(bad ? 0 : to_fixed(v0, top), bad ? 0 : to_fixed(v1, top), q);
        __half* d = dig + (size_t)(c0 + n) * kp + k;
#pragma unroll
        for (int s = 0; s < SL; s++) *reinterpret_cast<__half2*>(d + s * ss) = q[s];
      }
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const int n = ty + 8 * i;
    const int l = __reduce_add_sync(0xffffffffu, large[i]);
    if (tx == 0 && c0 + n < N) {
      bool bad;
      const int top = top_of(s_me[n], bad);
      bad |= s_me[n] == 0 && s_den[n];
      if (ALL || blockIdx.y == 0) exps[c0 + n] = top + 1 - 1023;
      const int v = bad ? CNT_BAD : s_me[n] == 0 ? ke - kb : l;
      if (ALL) cnt[c0 + n] = v;
      else if (bad) atomicMin(cnt + c0 + n, CNT_BAD / 2);
      else atomicAdd(cnt + c0 + n, v);
    }
  }
}

// ---- the product -----------------------------------------------------------------------------

struct SplitArgs {
  int M, N, K, tri, tiles_m, tiles_n, tiles;
  const double* A;   // the operands themselves, for the FMA tiles
  size_t lda;
  const double* B;
  size_t ldb;
  int b_rows;        // B given as N x K rows (B' of the product)
  double* C;
  size_t ldc;
  const int *ea, *ca, *eb, *cb;
  int* list;         // [0] count, then the tiles left to fma_tiles_kernel
  int* err;
};

// Tile t as (row tile, column tile). Full grid: groups of 8 row tiles walk the columns together,
// so that the tiles in flight share their operands in L2. Lower triangle: the tiles with a column
// at or left of their last row, 2 (r + 1) of them in row tile r.
__device__ __forceinline__ void tile_at(const SplitArgs& p, int t, int& tm, int& tn) {
  if (p.tri) {
    int r = (int)((sqrtf(4.f * (float)t + 1.f) - 1.f) * 0.5f);
    while ((r + 1) * (r + 2) <= t) r++;
    while (r * (r + 1) > t) r--;
    tm = r;
    tn = t - r * (r + 1);
    return;
  }
  const int per = 8 * p.tiles_n, g = t / per, r = t - g * per;
  const int rows = min(8, p.tiles_m - g * 8);
  tm = g * 8 + r % rows;
  tn = r / rows;
}

// Whether the tile's digits hold what its products need (see the head of the file). Whole warp.
__device__ __forceinline__ bool tile_fits(const SplitArgs& p, int tm, int tn, int lane) {
  int a = 1 << 29, b = 1 << 29;
#pragma unroll
  for (int i = 0; i < PM / 32; i++) {
    const int r = tm * PM + i * 32 + lane;
    if (r < p.M) a = min(a, __ldg(p.ca + r));
  }
#pragma unroll
  for (int i = 0; i < PN / 32; i++) {
    const int c = tn * PN + i * 32 + lane;
    if (c < p.N) b = min(b, __ldg(p.cb + c));
  }
  a = __reduce_min_sync(0xffffffffu, a);
  b = __reduce_min_sync(0xffffffffu, b);
  return 4 * ((long long)a + b) > 5 * (long long)p.K;
}

// (hi 2^32 + lo) 2^(sc - 70) rounded to nearest (ties away from zero), by integer instructions
// without branches. The sum is below 2^95; the exponent limits keep the result a normal number.
__device__ __forceinline__ double round_sum(long long hi, long long lo, int sc) {
  const long long p = hi + (lo >> 32);  // the sum's upper 64 bits, above 32 in w
  const long long sg = p >> 63;
  const unsigned s32 = (unsigned)sg;
  unsigned w = ((unsigned)lo ^ s32) - s32;
  unsigned long long m = (unsigned long long)(p ^ sg) + (w == 0u ? (s32 & 1u) : 0u);
  const bool low = m == 0;
  m = low ? (unsigned long long)w : m;
  w = low ? 0u : w;
  const int z = __clzll((long long)m);
  const unsigned long long n = (m << z) | (((unsigned long long)w << 32) >> (64 - z));
  const unsigned long long mant = (n >> 11) + ((n >> 10) & 1u);  // 53 bits, the first one set
  const int e = (low ? 63 : 95) - z + sc - 70 + 1022;
  const unsigned long long bits = ((unsigned long long)(unsigned)e << 52) + mant;
  return __longlong_as_double((long long)(n == 0 ? 0ull : bits | (unsigned long long)sg << 63));
}

// MODE -1: C -= A B, 0: C = A B, 1: C += A B.
template <int MODE>
__global__ void __launch_bounds__(SPLIT_T, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb,
                  const __grid_constant__ SplitArgs p) {
  la_pdl_wait();
  la_pdl_trigger();
  extern __shared__ __align__(1024) unsigned char split_raw[];
  __shared__ __align__(8) uint64_t full[NST], empty[NST], acc_full, acc_empty, last;
  __shared__ uint32_t tmem_holder;
  __shared__ volatile int s_fail;
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(split_raw) + 1023) & ~uintptr_t(1023));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nst = (p.K + PK - 1) / PK;                           // stages per tile
  const int nchunk = (nst + CHUNK_STAGES - 1) / CHUNK_STAGES;

  if (tid == 0) {
    for (int s = 0; s < NST; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(&acc_full, 1);
    mbar_init(&acc_empty, EPI_WARPS);
    mbar_init(&last, 1);
    s_fail = 0;
    la_tma::mbar_init_fence();
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(
        smem_u32(&tmem_holder)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = tmem_holder;

  if (warp == EPI_WARPS) {  // TMA producer
    int n = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < p.tiles && ok; t += gridDim.x) {
      int tm, tn;
      tile_at(p, t, tm, tn);
      if (!tile_fits(p, tm, tn, lane)) continue;
      if (lane == 0)
        for (int s = 0; s < nst; s++, n++) {
          const int b = n % NST;
          if (n >= NST && !sw_wait(&empty[b], (uint32_t)((n / NST - 1) & 1), p.err)) {
            s_fail = 1;
            ok = false;
            break;
          }
          unsigned char* st = smem + b * PST_BYTES;
          la_tma::mbar_expect_tx(&full[b], PST_BYTES);
          tma_load_3d(st, &ta, s * PK, tm * PM, 0, &full[b]);
          tma_load_3d(st + PA_BYTES, &tb, s * PK, tn * PN, 0, &full[b]);
        }
      ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
    }
    if (lane == 0 && !ok)  // this CTA's copies still in flight
      for (int k = max(0, n - NST); k < n; k++)
        la_tma::mbar_drain(&full[k % NST], (uint32_t)((k / NST) & 1));
  } else if (warp == EPI_WARPS + 1) {  // MMA issuer
    int n = 0, chunk = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < p.tiles && ok; t += gridDim.x) {
      int tm, tn;
      tile_at(p, t, tm, tn);
      if (!tile_fits(p, tm, tn, lane)) continue;
      if (lane == 0)
        for (int s = 0; s < nst && ok; s++, n++) {
          const int b = n % NST;
          if (s % CHUNK_STAGES == 0 && chunk > 0 &&
              !sw_wait(&acc_empty, (uint32_t)((chunk - 1) & 1), p.err))
            ok = false;
          if (ok && !sw_wait(&full[b], (uint32_t)((n / NST) & 1), p.err)) ok = false;
          if (!ok) {
            s_fail = 1;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;");
          const uint32_t sa = smem_u32(smem + b * PST_BYTES), sb = sa + PA_BYTES;
#pragma unroll
          for (int k = 0; k < PK / 16; k++) {
            const uint32_t acc = s % CHUNK_STAGES == 0 && k == 0 ? 0u : 1u;
#pragma unroll
            for (int d = 0; d < SL; d++) {  // digit d of A with digits [0, 8 - d) of B
              const uint64_t ad = sdesc64(sa + d * (PM * PK * 2) + k * 32);
              const int n0 = SL - d < 4 ? SL - d : 4, n1 = SL - d - n0;
              mma_f16(tmem + d * PN, ad, sdesc64(sb + k * 32), idesc_f16(n0 * PN),
                      d == 0 ? acc : 1u);
              if (n1 > 0)
                mma_f16(tmem + (d + 4) * PN, ad, sdesc64(sb + 4 * (PN * PK * 2) + k * 32),
                        idesc_f16(n1 * PN), d == 0 ? acc : 1u);
            }
          }
          tc_commit(&empty[b]);
          if (s % CHUNK_STAGES == CHUNK_STAGES - 1 || s == nst - 1) {
            tc_commit(&acc_full);
            chunk++;
          }
        }
      ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
    }
    if (lane == 0 && !ok) {  // MMAs still in flight
      tc_commit(&last);
      la_tma::mbar_drain(&last, 0);
    }
  } else {  // epilogue
    const int row = (warp & 3) * 32 + lane;       // this thread's accumulator row
    const int col = (warp >> 2) * 16;             // its warp's first column
    const uint32_t tbase = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)col;
    double* wbuf = reinterpret_cast<double*>(smem + NST * PST_BYTES) + warp * (32 * 8);
    int chunk = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < p.tiles && ok; t += gridDim.x) {
      int tm, tn;
      tile_at(p, t, tm, tn);
      if (!tile_fits(p, tm, tn, lane)) {
        if (tid == 0) p.list[1 + atomicAdd(p.list, 1)] = t;
        continue;
      }
      const int m0 = tm * PM, n0 = tn * PN;
      const int sr = m0 + row < p.M ? __ldg(p.ea + m0 + row) : 0;
      const int sc = n0 + col + (lane & 15) < p.N ? __ldg(p.eb + n0 + col + (lane & 15)) : 0;
      long long hi[16], lo[16];
#pragma unroll
      for (int j = 0; j < 16; j++) hi[j] = lo[j] = 0;
      for (int c = 0; c < nchunk; c++, chunk++) {
        // warp-uniform: every lane waits on the same phase
        ok = __all_sync(0xffffffffu, sw_wait(&acc_full, (uint32_t)(chunk & 1), p.err));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
        for (int j = 0; j < 16; j += 2) {
          uint32_t r[SL][2];
#pragma unroll
          for (int g = 0; g < SL; g++) tmem_ld2(tbase + g * PN + j, r[g]);
          tmem_wait(r);
#pragma unroll
          for (int i = 0; i < 2; i++) {
            int d[SL];
#pragma unroll
            for (int g = 0; g < SL; g++) d[g] = __float2int_rn(__uint_as_float(r[g][i]));
            const int h0 = d[0] * 256 + d[1], h1 = d[2] * 256 + d[3];  // below 2^31
            hi[j + i] += (long long)h0 * 65536 + h1;
            lo[j + i] += (long long)d[4] * 16777216 + (long long)d[5] * 65536 +
                         (long long)d[6] * 256 + d[7];
          }
        }
        asm volatile("tcgen05.fence::before_thread_sync;");
        if (lane == 0) mbar_arrive(&acc_empty);
      }
      if (!ok) break;
      // 8 columns at a time through shared memory: each lane rounds its row, then the warp reads
      // and writes C in 64-byte pieces of rows.
      const int cc = lane & 7;
#pragma unroll
      for (int g = 0; g < 2; g++) {
        const int c = n0 + col + g * 8 + cc;
        double old[8];
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const int gr = m0 + (warp & 3) * 32 + 4 * i + (lane >> 3);
          if (MODE != 0) old[i] = gr < p.M && c < p.N ? p.C[(size_t)gr * p.ldc + c] : 0.0;
        }
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const int eb = __shfl_sync(0xffffffffu, sc, g * 8 + j);
          wbuf[lane * 8 + (j ^ ((lane >> 1) & 7))] =
              round_sum(hi[g * 8 + j], lo[g * 8 + j], sr + eb);
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const int r = 4 * i + (lane >> 3), gr = m0 + (warp & 3) * 32 + r;
          const double v = wbuf[r * 8 + (cc ^ ((r >> 1) & 7))];
          if (gr < p.M && c < p.N)
            p.C[(size_t)gr * p.ldc + c] = MODE == 0 ? v : MODE < 0 ? old[i] - v : old[i] + v;
        }
        __syncwarp();
      }
    }
    if (!ok) s_fail = 1;
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
}

// The listed tiles by FMA chains in ascending k, in halves of 64 x 64: thread (tx, ty) owns rows
// ty + 16 i and columns tx + 16 j. The next slab's values wait in registers while the present one
// is used; the FP64 pipe (two FMAs per clock) hides the rest.
template <int MODE>
__global__ void __launch_bounds__(FMA_T, FMA_PER_SM)
fma_tiles_kernel(const __grid_constant__ SplitArgs p) {
  la_pdl_wait();
  la_pdl_trigger();
  __shared__ double as[2][FK][FT], bs[2][FK][FT];
  if (*reinterpret_cast<volatile int*>(p.err) != 0) return;
  const int items = 2 * *reinterpret_cast<volatile int*>(p.list);
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  for (int it = blockIdx.x; it < items; it += gridDim.x) {
    int tm, tn;
    tile_at(p, p.list[1 + it / 2], tm, tn);
    const int m0 = tm * PM + (it & 1) * FT, n0 = tn * PN;
    double acc[4][4], ra[4], rb[4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int r = m0 + ty + 16 * i, c = n0 + tx + 16 * j;
        acc[i][j] = MODE != 0 && r < p.M && c < p.N ? p.C[(size_t)r * p.ldc + c] : 0.0;
      }
    auto fetch = [&](int k0) {
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int e = tid + q * FMA_T;
        const int r = e / FK, k = e % FK;
        ra[q] = m0 + r < p.M && k0 + k < p.K ? p.A[(size_t)(m0 + r) * p.lda + k0 + k] : 0.0;
        if (p.b_rows)
          rb[q] = n0 + r < p.N && k0 + k < p.K ? p.B[(size_t)(n0 + r) * p.ldb + k0 + k] : 0.0;
        else
          rb[q] = n0 + e % FT < p.N && k0 + e / FT < p.K
                      ? p.B[(size_t)(k0 + e / FT) * p.ldb + n0 + e % FT] : 0.0;
      }
    };
    fetch(0);
    for (int k0 = 0, b = 0; k0 < p.K; k0 += FK, b ^= 1) {
#pragma unroll
      for (int q = 0; q < 4; q++) {
        const int e = tid + q * FMA_T;
        as[b][e % FK][(e / FK) ^ (e % FK)] = ra[q];
        const int k = p.b_rows ? e % FK : e / FT, c = p.b_rows ? e / FK : e % FT;
        bs[b][k][c ^ k] = rb[q];
      }
      __syncthreads();  // the other buffer's readers of two slabs ago are done, too
      if (k0 + FK < p.K) fetch(k0 + FK);
      const int kn = min(FK, p.K - k0);
#pragma unroll 4
      for (int k = 0; k < kn; k++) {
        double a[4], v[4];
#pragma unroll
        for (int i = 0; i < 4; i++) a[i] = as[b][k][(ty + 16 * i) ^ k];
#pragma unroll
        for (int j = 0; j < 4; j++) v[j] = bs[b][k][(tx + 16 * j) ^ k];
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
          for (int j = 0; j < 4; j++) acc[i][j] = fma(MODE < 0 ? -a[i] : a[i], v[j], acc[i][j]);
      }
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int r = m0 + ty + 16 * i, c = n0 + tx + 16 * j;
        if (r < p.M && c < p.N) p.C[(size_t)r * p.ldc + c] = acc[i][j];
      }
  }
}

size_t up(size_t x, size_t a) { return (x + a - 1) / a * a; }

// Digits [SL][rows][kp] of `rows` rows of K values.
bool encode_digits(la_ctx ctx, CUtensorMap* map, const void* base, int rows, int K, int kp,
                   uint32_t box_rows) {
  la_tma::EncodeTiledFn enc = la_tma::get_encoder(ctx);
  if (!enc) return false;
  cuuint64_t dims[3] = {(cuuint64_t)K, (cuuint64_t)rows, (cuuint64_t)SL};
  cuuint64_t strides[2] = {(cuuint64_t)kp * 2, (cuuint64_t)kp * 2 * rows};
  cuuint32_t box[3] = {(cuuint32_t)PK, box_rows, (cuuint32_t)SL};
  cuuint32_t estr[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<void*>(base), dims, strides, box,
             estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
             CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

template <int MODE>
la_status launch_product(la_ctx ctx, cudaStream_t st, const CUtensorMap& ta, const CUtensorMap& tb,
                         const SplitArgs& p) {
  static la_device_once configured;
  cudaError_t e = configured.run([](int) {
    return cudaFuncSetAttribute(gemm_split_kernel<MODE>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SPLIT_SMEM);
  });
  if (e != cudaSuccess) return la_cuda_fail(ctx, e, "cudaFuncSetAttribute(gemm_split)");
  e = la_launch(ctx, gemm_split_kernel<MODE>, dim3(std::min(p.tiles, ctx->sm_count)),
                dim3(SPLIT_T), SPLIT_SMEM, st, ta, tb, p);
  if (e != cudaSuccess) return la_cuda_fail(ctx, e, "gemm_split_kernel launch");
  const int halves = (int)std::min<long long>(2ll * p.tiles, (long long)FMA_PER_SM * ctx->sm_count);
  e = la_launch(ctx, fma_tiles_kernel<MODE>, dim3(halves), dim3(FMA_T), 0, st, p);
  if (e != cudaSuccess) return la_cuda_fail(ctx, e, "fma_tiles_kernel launch");
  ctx->launches += 2;
  return la_check_launch(ctx, "gemm_split_kernel");
}

// One side's digits, exponents and counts in the workspace.
struct Side {
  __half* dig;
  int *exps, *cnt, *me;
  static size_t bytes(size_t rows, size_t kp) {
    return up(rows * kp * 2 * SL, 256) + up(rows * 4 * 4, 256);
  }
  Side(char* base, size_t rows, size_t kp) {
    dig = reinterpret_cast<__half*>(base);
    exps = reinterpret_cast<int*>(base + up(rows * kp * 2 * SL, 256));
    cnt = exps + rows;
    me = cnt + rows;  // [2][rows]
  }
};

constexpr int COLS_ALL_K = 512;  // columns of up to this many k are split by one CTA per 32

la_status split_rows(la_ctx ctx, cudaStream_t st, const double* X, size_t ldx, int R, int K, int kp,
                     const Side& s, int* nlist) {
  const cudaError_t e = la_launch(ctx, split_rows_kernel, dim3((R + 7) / 8), dim3(256), 0, st, X,
                                  ldx, R, K, kp, s.dig, s.exps, s.cnt, nlist);
  if (e != cudaSuccess) return la_cuda_fail(ctx, e, "split_rows_kernel launch");
  ctx->launches++;
  return la_check_launch(ctx, "split_rows_kernel");
}

la_status split_cols(la_ctx ctx, cudaStream_t st, const double* X, size_t ldx, int K, int N, int kp,
                     const Side& s) {
  cudaError_t e;
  if (K <= COLS_ALL_K) {
    e = la_launch(ctx, split_cols_kernel<true>, dim3((N + 31) / 32), dim3(256), 0, st, X, ldx, K, N,
                  kp, K, (const int*)nullptr, s.dig, s.exps, s.cnt);
  } else {
    const int kper = 256, gy = (K + kper - 1) / kper;
    LA_CUDA(ctx, cudaMemsetAsync(s.cnt, 0, (size_t)N * 3 * sizeof(int), st));  // cnt and me
    col_exp_kernel<<<dim3((N + 31) / 32, gy), 256, 0, st>>>(X, ldx, K, N, kper, s.me);
    ctx->launches++;
    split_cols_kernel<false><<<dim3((N + 31) / 32, gy), 256, 0, st>>>(
        X, ldx, K, N, kp, kper, s.me, s.dig, s.exps, s.cnt);
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) return la_cuda_fail(ctx, e, "split_cols_kernel launch");
  ctx->launches++;
  return la_check_launch(ctx, "split_cols_kernel");
}

}  // namespace

size_t gemm_split_ws(int M, int N, int K, bool same) {
  const size_t kp = up(K, 8), tiles = up(M, PM) / PM * (up(N, PN) / PN + 2);
  return Side::bytes(M, kp) + (same ? 0 : Side::bytes(N, kp)) + up((tiles + 1) * 4, 256);
}

la_status launch_gemm_split(la_ctx ctx, cudaStream_t st, int mode, int M, int N, int K,
                            const double* A, size_t lda, const double* B, size_t ldb, bool b_rows,
                            double* C, size_t ldc, bool tri, void* ws, size_t ws_bytes) {
  if (M <= 0 || N <= 0) return LA_OK;
  if (K <= 0 || K > (1 << 20) || (tri && M != N)) return LA_UNSUPPORTED;
  const bool same = b_rows && A == B && lda == ldb && M == N;
  const int kp = (int)up(K, 8);
  if (!ws || ws_bytes < gemm_split_ws(M, N, K, same)) return LA_UNSUPPORTED;
  char* base = static_cast<char*>(ws);
  const Side sa(base, M, kp);
  const Side sb = same ? sa : Side(base + Side::bytes(M, kp), N, kp);
  int* list = reinterpret_cast<int*>(base + Side::bytes(M, kp) + (same ? 0 : Side::bytes(N, kp)));
  CUtensorMap ta, tb;
  if (!encode_digits(ctx, &ta, sa.dig, M, K, kp, PM) ||
      !encode_digits(ctx, &tb, sb.dig, N, K, kp, PN))
    return LA_UNSUPPORTED;
  SplitArgs p;
  p.M = M;
  p.N = N;
  p.K = K;
  p.tri = tri ? 1 : 0;
  p.tiles_m = (M + PM - 1) / PM;
  p.tiles_n = (N + PN - 1) / PN;
  const long long lower = (long long)p.tiles_m * (p.tiles_m + 1);
  const long long tiles = tri ? lower : (long long)p.tiles_m * p.tiles_n;
  if (tiles > (1 << 24)) return LA_UNSUPPORTED;
  p.tiles = (int)tiles;
  p.A = A;
  p.lda = lda;
  p.B = B;
  p.ldb = ldb;
  p.b_rows = b_rows ? 1 : 0;
  p.C = C;
  p.ldc = ldc;
  p.ea = sa.exps;
  p.ca = sa.cnt;
  p.eb = sb.exps;
  p.cb = sb.cnt;
  p.list = list;
  p.err = ctx->d_err;
  LA_TRY(split_rows(ctx, st, A, lda, M, K, kp, sa, list));
  if (!same) {
    if (b_rows) LA_TRY(split_rows(ctx, st, B, ldb, N, K, kp, sb, nullptr));
    else LA_TRY(split_cols(ctx, st, B, ldb, K, N, kp, sb));
  }
  if (mode < 0) return launch_product<-1>(ctx, st, ta, tb, p);
  if (mode == 0) return launch_product<0>(ctx, st, ta, tb, p);
  return launch_product<1>(ctx, st, ta, tb, p);
}
