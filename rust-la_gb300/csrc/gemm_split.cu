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
// Which tiles take this path. That last error is relative to the row's and the column's largest
// entries, an FMA chain's to sum_k |a_ik b_kj|: about 0.2 2^-53 of it for terms of random signs.
// So a tile is computed this way where for every element, in units of 2^(ea_i + eb_j),
//     sum_k |a_ik b_kj| >= 2^-8.9 sqrt(K),
// where the error left out is no larger than the chain's. guard_kernel decides it per tile, in two
// steps. The split kernels count, per row and column, the entries within 2^-5 of the scale; if the
// smallest row count and the smallest column count exceed K by 2^1.1 sqrt(K) together, that many k have
// both entries large, and the sum is at least 2^1.1 sqrt(K) 2^-10. Else the sums are formed from the
// leading two digits by mma.sync (a few microseconds, where the FMA tile of K = 256 takes 1 ms; as
// FP32 FMAs they took 65 us for K = 700, a tenth of the FMA tiles that may follow). Every other
// tile (graded or sparse operands, values that are not finite or beyond 2^+-400) goes on a list that
// the epilogue warps work off at the end of the product (fma_tiles), with FMA chains in ascending k,
// in pieces small enough that every SM has some. Where all tiles are on the list (graded along k), us,
// by the FMA kernels of gemm_f64.cu alone, with 64 x 64 pieces here, and now: 100 x 64 x 100 88, 115,
// 57; 64 x 1936 x 436 1967, 2209, 333; 2048^3 14253, 15371, 14265; 4096^3 109.8 ms, 118.5, 113.3 (the
// sums that reject the tiles are 2 % of it).
//
// Measured on 8192^3 (A and B N(0,1)): 24.0 ms against 876.6 ms by FMA, 36 x 2 x 8192^3 FP16
// operations in all, 1.65 PFLOP/s; rms error against quadruple precision 5 to 17 times smaller than
// the FMA chain's (K = 64 to 2049). What bounds it: the MMAs of 128 k (9.2k clocks at the tensor
// peak) and the part of reading the accumulators (about 5k clocks per 128 k) that does not overlap
// them. The tile's accumulators fill the tensor memory, so they are handed over in two halves: 0-3
// while 4-7 are still being computed, and 4-7 while the next k's 0-3 are (28.0 ms in one piece).
// For K = 64 (8192 x 8192 in 0.37 ms) the epilogue's integer instructions bound it.
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
constexpr float GUARD = 0.0021f;      // 2^-8.9
constexpr int CNT_BAD = -(1 << 29);   // count of a row the digits cannot represent
constexpr int FR = 64, FC = 16, FK = 32;  // FMA pieces: up to 64 rows, 16 columns, slabs of 32 k

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
// Four columns of four accumulators. The wait takes the registers, so that nothing that uses them
// moves above it.
constexpr int HG = SL / 2;  // accumulators per half
__device__ __forceinline__ void tmem_ld4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr));
}
__device__ __forceinline__ void tmem_wait(uint32_t (&r)[HG][4]) {
#define LA_R4(g) "+r"(r[g][0]), "+r"(r[g][1]), "+r"(r[g][2]), "+r"(r[g][3])
  asm volatile("tcgen05.wait::ld.sync.aligned;" : LA_R4(0), LA_R4(1), LA_R4(2), LA_R4(3)::"memory");
#undef LA_R4
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

// A chain of products of the same kind (the blocks of a QR) counts in *misses how many in a row left
// nearly all of their tiles to the FMA chains. Of such a row only the products after 0, 1, 4, 16, ...
// misses form digits and look at the tiles, the others put every tile on the list at once. QR
// factorizations of 2500 x 1501, ms, digits and sums in every block, and now: entries N(0,1) exp(4 N(0,1))
// 23.06, 21.48; banded 20.33, 18.99; 2 % of the entries not zero, even from the second block on, 17.93,
// 17.74; N(0,1) 13.24, 13.28. The word is loaded ahead of a kernel's operands and looked at after them.
__device__ __forceinline__ int load_misses(const int* misses) {
  return misses ? *reinterpret_cast<const volatile int*>(misses) : 0;
}
__device__ __forceinline__ bool skips_digits(int n) { return (n & (n - 1)) != 0 || (n & 0xAAAAAAAA) != 0; }

// Rows of X (R x K, pitch ldx) into digits [SL][R][kp], exps[R] (ea) and cnt[R] (large entries).
// One warp per row, two neighbouring k per lane: a slice's row is written 128 bytes at a time. The
// row is read twice, the second time from L1 or L2 where K is a panel's width.
__device__ __forceinline__ void split_rows(int block, const double* __restrict__ X, size_t ldx,
                                           int R, int K, int kp, __half* __restrict__ dig,
                                           int* __restrict__ exps, int* __restrict__ cnt, int misses) {
  const int lane = threadIdx.x & 31;
  const int r = block * 8 + (threadIdx.x >> 5);
  if (r >= R) return;
  const double* x = X + (size_t)r * ldx;
  int me = 0;
  bool den = false;
  for (int k = lane; k < K; k += 32) {
    const double v = x[k];
    me = max(me, exp_bits(v));
    den |= is_denormal(v);
  }
  if (skips_digits(misses)) return;
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

// Largest biased exponent of each column of X (K x N) over k [yblock * kper, ...), and a denormal's
// presence as a flag, into maxexp (zeroed before).
__device__ __forceinline__ void col_exps(int block, int yblock, const double* __restrict__ X,
                                         size_t ldx, int K, int N, int kper,
                                         int* __restrict__ maxexp) {
  const int c = block * 32 + (threadIdx.x & 31), ty = threadIdx.x >> 5;
  const int k0 = yblock * kper, k1 = min(K, k0 + kper);
  if (c >= N) return;
  int me = 0, den = 0;
#pragma unroll 8
  for (int k = k0 + ty; k < k1; k += 8) {
    const double v = X[(size_t)k * ldx + c];
    me = max(me, exp_bits(v));
    den |= is_denormal(v);
  }
  if (me) atomicMax(maxexp + c, me);
  if (den) atomicOr(maxexp + N + c, 1);
}

// Columns of X (K x N, pitch ldx), k [yblock * kper, ...), into digits [SL][N][kp]. 32 columns
// per CTA: 64 k at a time go through shared memory, so that global rows are read 256 bytes at a
// time and a digit's k are written 128 bytes at a time. ALL: the CTA sees every k of its columns
// and finds their exponents itself; else they come from col_exps and counts are added up.
template <bool ALL>
__device__ __forceinline__ void split_cols(int block, int yblock, const double* __restrict__ X,
                                           size_t ldx, int K, int N, int kp, int kper,
                                           const int* __restrict__ maxexp,
                                           __half* __restrict__ dig, int* __restrict__ exps,
                                           int* __restrict__ cnt, int misses) {
  __shared__ double tile[64][33];
  __shared__ int s_me[32], s_den[32];
  const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
  const int c0 = block * 32, c = c0 + tx;
  const int kb = ALL ? 0 : yblock * kper, ke = ALL ? K : min(K, kb + kper);
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
  if (skips_digits(misses)) return;
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
      if (ALL || yblock == 0) exps[c0 + n] = top + 1 - 1023;
      const int v = bad ? CNT_BAD : s_me[n] == 0 ? ke - kb : l;
      if (ALL) cnt[c0 + n] = v;
      else if (bad) atomicMin(cnt + c0 + n, CNT_BAD / 2);
      else atomicAdd(cnt + c0 + n, v);
    }
  }
}

// Rows of A and columns of B in one launch: the first ra CTAs take 8 rows of A each, the others 8
// rows of B' (b_rows), 32 columns of B, or (kper > 0: the columns are split afterwards, in pieces of
// K) the exponents of 32 columns over one piece. list[0] is zeroed for the guard and b.cnt for the
// pieces.
struct SplitSide {
  const double* X;
  size_t ldx;
  int n;
  __half* dig;
  int *exps, *cnt;
};
__global__ void __launch_bounds__(256)
split_kernel(const SplitSide a, const SplitSide b, int K, int kp, int ra, int b_rows, int kper,
             int* list, int* maxexp, const int* misses) {
  la_pdl_wait();
  la_pdl_trigger();
  const int block = blockIdx.x;
  if (block == 0 && threadIdx.x == 0) *list = 0;
  const int n = load_misses(misses);
  if (kper)
    for (int i = block * 256 + threadIdx.x; i < b.n; i += gridDim.x * 256) b.cnt[i] = 0;
  if (block < ra) {
    split_rows(block, a.X, a.ldx, a.n, K, kp, a.dig, a.exps, a.cnt, n);
  } else if (b_rows) {
    split_rows(block - ra, b.X, b.ldx, b.n, K, kp, b.dig, b.exps, b.cnt, n);
  } else if (kper) {
    const int gx = (b.n + 31) / 32;
    if (skips_digits(n)) return;
    col_exps((block - ra) % gx, (block - ra) / gx, b.X, b.ldx, K, b.n, kper, maxexp);
  } else {
    split_cols<true>(block - ra, 0, b.X, b.ldx, K, b.n, kp, K, nullptr, b.dig, b.exps, b.cnt, n);
  }
}
__global__ void __launch_bounds__(256)
split_cols_part_kernel(const SplitSide b, int K, int kp, int kper, const int* __restrict__ maxexp,
                       const int* misses) {
  la_pdl_wait();
  la_pdl_trigger();
  split_cols<false>(blockIdx.x, blockIdx.y, b.X, b.ldx, K, b.n, kp, kper, maxexp, b.dig, b.exps,
                    b.cnt, load_misses(misses));
}

// ---- the product -----------------------------------------------------------------------------

struct SplitArgs {
  int M, N, K, tri, tiles_m, tiles_n, tiles, prefetch, per_cta;
  int splits, kper;  // K in `splits` pieces of kper (a multiple of 128), piece z into C + z czs
  size_t czs;
  const double* A;   // the operands themselves, for the FMA tiles
  size_t lda;
  const double* B;
  size_t ldb;
  int b_rows;        // B given as N x K rows (B' of the product)
  double* C;
  size_t ldc;
  const int *ea, *ca, *eb, *cb;
  const __half *da, *db;  // the digits [SL][rows][kp]
  int kp, joint;     // joint: terms of 2^-10 that make the guard's sum
  int* fits;         // per tile: 1 where the digits hold what it needs
  int* list;         // [0] count, then the tiles left to fma_tiles
  int* misses;       // see skips_digits; may be null
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

// Leading two digits of 8 neighbouring k of a row, as |a| in units of 2^ea, FP16 (11 bits are plenty
// for a sum that decides within a factor).
__device__ __forceinline__ uint4 abs8(const __half* d, size_t ss, int k, int K, int kp, bool in) {
  uint4 x = make_uint4(0u, 0u, 0u, 0u), y = x;
  if (in && k < kp) {  // rows are kp values, a multiple of 8
    x = *reinterpret_cast<const uint4*>(d + k);
    y = *reinterpret_cast<const uint4*>(d + ss + k);
  }
  const __half2 c0 = __float2half2_rn(0.0078125f), c1 = __float2half2_rn(3.0517578125e-5f);
  __half2* xs = reinterpret_cast<__half2*>(&x);
  const __half2* ys = reinterpret_cast<const __half2*>(&y);
#pragma unroll
  for (int i = 0; i < 4; i++) {
    xs[i] = __habs2(__hfma2(xs[i], c0, __hmul2(ys[i], c1)));
    // what lies between K and kp is not set
    if (k + 2 * i >= K) xs[i] = __float2half2_rn(0.f);
    else if (k + 2 * i + 1 >= K) xs[i] = __halves2half2(__low2half(xs[i]), __ushort_as_half(0));
  }
  return x;
}
__device__ __forceinline__ void mma_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2,
                                          uint32_t a3, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// fits[tile] (see the head of the file), and the list of the others. A warp per tile compares the
// counts; the tiles they do not decide are summed by the whole CTA, one after the other.
// The sums are a chain of loads through L2. Where K is long, SETS = 2 sets of 8 warps take every second
// slab of k each, two slabs' loads in flight (7 tiles of K = 1936: 177 us with one set, 76 with two); for
// short ones, of a few slabs, one set leaves room for two CTAs per SM.
constexpr int GUARD_W = 8;  // warps of a set, tiles of a CTA at most
constexpr int GUARD_LONG_K = 1024;
template <int SETS>
__global__ void __launch_bounds__(SETS * GUARD_W * 32)
guard_kernel(const __grid_constant__ SplitArgs p) {
  la_pdl_wait();
  la_pdl_trigger();
  __shared__ int s_sum[GUARD_W];
  __shared__ float s_acc[SETS > 1 ? 32 : 1][GUARD_W * 32];  // the second set's sums
  const int tid = threadIdx.x, lane = tid & 31, set = tid / (GUARD_W * 32), warp = tid / 32 % GUARD_W;
  const int misses = load_misses(p.misses);
  if (set == 0) {
    const int t = blockIdx.x * p.per_cta + warp;
    int sum = 0;
    if (warp < p.per_cta && t < p.tiles) {
      int tm, tn;
      tile_at(p, t, tm, tn);
      int a = 1 << 29, b = 1 << 29;
#pragma unroll
      for (int i = 0; i < PM / 32; i++) {
        const int r = tm * PM + i * 32 + lane;
        if (r < p.M) a = min(a, p.ca[r]);
      }
#pragma unroll
      for (int i = 0; i < PN / 32; i++) {
        const int c = tn * PN + i * 32 + lane;
        if (c < p.N) b = min(b, p.cb[c]);
      }
      if (skips_digits(misses)) a = b = CNT_BAD;
      a = __reduce_min_sync(0xffffffffu, a);
      b = __reduce_min_sync(0xffffffffu, b);
      const bool fit = (long long)a + b >= (long long)p.K + p.joint;
      sum = !fit && a >= 0 && b >= 0;
      if (lane == 0 && !sum) {
        p.fits[t] = fit ? 1 : 0;
        if (!fit) p.list[1 + atomicAdd(p.list, 1)] = t;
      }
    }
    if (lane == 0) s_sum[warp] = sum;
  }
  __syncthreads();
  for (int w = 0; w < GUARD_W; w++) {
    if (!s_sum[w]) continue;
    const int t = blockIdx.x * p.per_cta + w;
    int tm, tn;
    tile_at(p, t, tm, tn);
    // sum_k |a_ik| |b_kj| in units of 2^(ea + eb), every element of the tile: warp w the rows
    // 32 (w / 2).. and columns 32 (w % 2)... Each thread takes 8 neighbouring k of its rows at a time
    // for two mma.sync; which k an operand register holds does not matter to the sum as long as A
    // and B agree.
    const int g = lane >> 2, kq = (lane & 3) * 8;
    const int row0 = tm * PM + warp / 2 * 32 + g, col0 = tn * PN + warp % 2 * 32 + g;
    const size_t sa = (size_t)p.M * p.kp, sb = (size_t)p.N * p.kp;
    float acc[2][4][4] = {};
#pragma unroll SETS
    for (int k0 = 32 * set; k0 < p.K; k0 += 32 * SETS) {
      uint4 a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; i++) {
        a[i] = abs8(p.da + (size_t)(row0 + 8 * i) * p.kp, sa, k0 + kq, p.K, p.kp, row0 + 8 * i < p.M);
        b[i] = abs8(p.db + (size_t)(col0 + 8 * i) * p.kp, sb, k0 + kq, p.K, p.kp, col0 + 8 * i < p.N);
      }
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) {
          mma_16816(acc[i][j], a[2 * i].x, a[2 * i + 1].x, a[2 * i].y, a[2 * i + 1].y, b[j].x, b[j].y);
          mma_16816(acc[i][j], a[2 * i].z, a[2 * i + 1].z, a[2 * i].w, a[2 * i + 1].w, b[j].z, b[j].w);
        }
    }
    float* const other = &s_acc[0][tid % (GUARD_W * 32)];
    if (SETS > 1) {
      if (set != 0)
#pragma unroll
        for (int i = 0; i < 32; i++) other[i * GUARD_W * 32] = acc[i / 16][i / 4 % 4][i % 4];
      __syncthreads();
    }
    const float need = GUARD * sqrtf((float)p.K);
    bool ok = true;
    if (set == 0)
#pragma unroll
      for (int i = 0; i < 32; i++) {
        const int r = row0 + i / 16 * 16 + i % 4 / 2 * 8;
        const int c = col0 - g + i / 4 % 4 * 8 + 2 * (lane & 3) + i % 2;
        const float v = acc[i / 16][i / 4 % 4][i % 4] + (SETS > 1 ? other[i * GUARD_W * 32] : 0.f);
        if (r < p.M && c < p.N) ok = ok && v >= need;
      }
    const bool fit = __syncthreads_and(ok ? 1 : 0) != 0;
    if (tid == 0) {
      p.fits[t] = fit ? 1 : 0;
      if (!fit) p.list[1 + atomicAdd(p.list, 1)] = t;
    }
  }
}

// A signed 96-bit integer, least significant word first.
struct Sum96 {
  unsigned x0, x1, x2;
};
__device__ __forceinline__ Sum96 sum96(long long hi, long long lo) {  // hi 2^32 + lo
  const long long u = hi + (lo >> 32);
  return {(unsigned)lo, (unsigned)u, (unsigned)(u >> 32)};
}
// a 2^(sc - 70) rounded to nearest (ties away from zero), by integer instructions without
// branches; the exponent limits keep the result a normal number. (The ALU pipe, not the tensor
// pipe, bounds products of K = 64: every instruction here counts.)
__device__ __forceinline__ double round_sum(Sum96 a, int sc) {
  const bool neg = (int)a.x2 < 0;
  if (neg)
    asm("sub.cc.u32 %0, 0, %0;\n\tsubc.cc.u32 %1, 0, %1;\n\tsubc.u32 %2, 0, %2;"
        : "+r"(a.x0), "+r"(a.x1), "+r"(a.x2));
  // the first word that is not zero leads (a sum below 2^32 is moved up two words, which takes
  // another look below)
  const bool s1 = a.x2 == 0u;
  unsigned hi = s1 ? a.x1 : a.x2, mi = s1 ? a.x0 : a.x1, lo = s1 ? 0u : a.x0;
  int e = s1 ? 63 : 95;
  if (hi == 0u) {  // rare: below 2^-38 of the scale
    hi = mi;
    mi = 0u;
    e = 31;
  }
  const int z = __clz((int)hi);
  const unsigned nh = __funnelshift_l(mi, hi, z), nl = __funnelshift_l(lo, mi, z);
  const unsigned ml = __funnelshift_r(nl, nh, 11), up = nl >> 10 & 1u;
  const unsigned mh = (nh >> 11) + ((unsigned)(e - z + sc - 70 + 1022) << 20);
  unsigned rl, rh;
  asm("add.cc.u32 %0, %2, %3;\n\taddc.u32 %1, %4, 0;" : "=r"(rl), "=r"(rh) : "r"(ml), "r"(up), "r"(mh));
  rh = neg ? rh | 0x80000000u : rh;
  return hi == 0u ? 0.0 : __hiloint2double((int)rh, (int)rl);
}

// The listed tiles by FMA chains in ascending k, in pieces of 16 NI rows and 16 columns. Each of four
// groups of four epilogue warps takes pieces of its own, with its own barrier and buffers: one warp per
// sub-partition with 2 NI chains per thread keeps the FP64 pipe (two FMAs per clock and SM) busy by
// itself, and while one group fetches or waits the others have the pipe. Slabs come by 8-byte cp.async
// (any alignment), one ahead, into the stages' shared memory: nothing is in flight there any more.
constexpr int FG_T = 128;                      // threads of a group
constexpr int FSLAB = FK * (FR + FC);          // doubles of a slab: A [k][row ^ k], B [k][column ^ k]
static_assert((size_t)(EPI_T / FG_T) * 2 * FSLAB * 8 <= (size_t)NST * PST_BYTES, "slabs in the stages");

// Set where a wait of an epilogue warp gave up.
__device__ __forceinline__ volatile int& gave_up() {
  __shared__ volatile int flag;
  return flag;
}
// The group's barrier; whether `ok` holds in all of its threads.
__device__ __forceinline__ bool group_all(int g, bool ok) {
  unsigned r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n"
      " barrier.cta.red.and.aligned.pred q, %2, %3, p;\n selp.u32 %0, 1, 0, q;\n}\n"
      : "=r"(r)
      : "r"(ok ? 1u : 0u), "r"(1 + g), "n"(FG_T)
      : "memory");
  return r != 0;
}
__device__ __forceinline__ void group_sync(int g) {
  asm volatile("barrier.cta.sync.aligned %0, %1;" ::"r"(1 + g), "n"(FG_T) : "memory");
}
__device__ __forceinline__ void fetch8(double* dst, const double* src, bool in) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(smem_u32(dst)), "l"(src),
               "r"(in ? 8 : 0)
               : "memory");
}
// Pieces of the first tile, which is the largest: row pieces of 16 NI, column pieces.
__device__ __forceinline__ int piece_rows(const SplitArgs& p, int R) { return (min(PM, p.M) + R - 1) / R; }
__device__ __forceinline__ int piece_cols(const SplitArgs& p) { return (min(PN, p.N) + FC - 1) / FC; }

template <int MODE, int NI>
__device__ __forceinline__ void fma_pieces(const SplitArgs& p, double* smem, int tid, int count) {
  const int g = tid / FG_T, t = tid % FG_T, tx = t & 7, ty = t >> 3;
  double* const buf = smem + g * 2 * FSLAB;
  const int hn = piece_cols(p), per = piece_rows(p, 16 * NI) * hn;
  const int items = count * p.splits * per;
  for (int it = g * gridDim.x + blockIdx.x; it < items; it += EPI_T / FG_T * gridDim.x) {
    const int q = it % per, z = it / per % p.splits;
    int tm, tn;
    tile_at(p, p.list[1 + it / (per * p.splits)], tm, tn);
    const int m0 = tm * PM + q / hn * 16 * NI, n0 = tn * PN + q % hn * FC;
    if (m0 >= p.M || n0 >= p.N) continue;
    const int kb = z * p.kper, ke = min(p.K, kb + p.kper);
    double* const C = p.C + z * p.czs;
    auto fetch = [&](int k0, double* slab) {
#pragma unroll 4
      for (int j = 0; j < 4 * NI; j++) {
        const int k = t % FK, r = t / FK + j * (FG_T / FK);
        const bool in = m0 + r < p.M && k0 + k < ke;
        fetch8(slab + k * FR + (r ^ k), in ? p.A + (size_t)(m0 + r) * p.lda + k0 + k : p.A, in);
      }
      double* const b = slab + FK * FR;
#pragma unroll
      for (int j = 0; j < FK * FC / FG_T; j++) {
        const int e = t + j * FG_T;
        const int k = p.b_rows ? e % FK : e / FC, c = p.b_rows ? e / FK : e % FC;
        const bool in = n0 + c < p.N && k0 + k < ke;
        const size_t at = p.b_rows ? (size_t)(n0 + c) * p.ldb + k0 + k : (size_t)(k0 + k) * p.ldb + n0 + c;
        fetch8(b + k * FC + (c ^ (k % FC)), in ? p.B + at : p.B, in);
      }
      asm volatile("cp.async.commit_group;" ::: "memory");
    };
    group_sync(g);  // the buffers' last readers are done
    fetch(kb, buf);
    double acc[NI][2];
#pragma unroll
    for (int i = 0; i < NI; i++)
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const int r = m0 + ty + 16 * i, c = n0 + tx + 8 * j;
        acc[i][j] = MODE != 0 && r < p.M && c < p.N ? C[(size_t)r * p.ldc + c] : 0.0;
      }
    for (int k0 = kb, b = 0; k0 < ke; k0 += FK, b ^= 1) {
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      group_sync(g);  // the slab is there, and the other buffer's readers are done
      if (k0 + FK < ke) fetch(k0 + FK, buf + (b ^ 1) * FSLAB);
      const double *as = buf + b * FSLAB, *bs = as + FK * FR;
      const int kn = min(FK, ke - k0);
#pragma unroll 4
      for (int k = 0; k < kn; k++) {
        double a[NI], v[2];
#pragma unroll
        for (int i = 0; i < NI; i++) a[i] = as[k * FR + ((ty + 16 * i) ^ k)];
#pragma unroll
        for (int j = 0; j < 2; j++) v[j] = bs[k * FC + ((tx + 8 * j) ^ (k % FC))];
#pragma unroll
        for (int i = 0; i < NI; i++)
#pragma unroll
          for (int j = 0; j < 2; j++) acc[i][j] = fma(MODE < 0 ? -a[i] : a[i], v[j], acc[i][j]);
      }
    }
#pragma unroll
    for (int i = 0; i < NI; i++)
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const int r = m0 + ty + 16 * i, c = n0 + tx + 8 * j;
        if (r < p.M && c < p.N) C[(size_t)r * p.ldc + c] = acc[i][j];
      }
  }
}

// The pieces are as high as the number of them allows: the most loaded SM decides (R rows of 16 columns
// take it 8 R clocks per k), and a lower piece loads more per FMA.
template <int MODE>
__device__ __noinline__ void fma_tiles(const SplitArgs& p, double* epi, int tid) {
  double* const smem = epi - NST * PST_BYTES / sizeof(double);
  const int count = *reinterpret_cast<volatile int*>(p.list);
  if (!group_all(tid / FG_T, gave_up() == 0)) return;
  const long long n = (long long)count * p.splits * piece_cols(p);
  auto cost = [&](int R) {
    return ((n * piece_rows(p, R) + gridDim.x - 1) / (int)gridDim.x) * (R + 2);
  };
  const long long c64 = cost(64), c32 = cost(32), c16 = cost(16);
  if (c64 <= c32 && c64 <= c16) fma_pieces<MODE, 4>(p, smem, tid, count);
  else if (c32 <= c16) fma_pieces<MODE, 2>(p, smem, tid, count);
  else fma_pieces<MODE, 1>(p, smem, tid, count);
}

// MODE -1: C -= A B, 0: C = A B, 1: C += A B.
template <int MODE>
__global__ void __launch_bounds__(SPLIT_T, 1)
gemm_split_kernel(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb,
                  const __grid_constant__ SplitArgs p) {
  la_pdl_wait();
  la_pdl_trigger();
  extern __shared__ __align__(1024) unsigned char split_raw[];
  __shared__ __align__(8) uint64_t full[NST], empty[NST], acc_full[2], acc_empty[2], last;
  __shared__ uint32_t tmem_holder;
  unsigned char* smem = reinterpret_cast<unsigned char*>(
      (reinterpret_cast<uintptr_t>(split_raw) + 1023) & ~uintptr_t(1023));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int total = p.tiles * p.splits;
  // The grid has a CTA for every FMA piece of small products; without FMA tiles they are done here.
  if (blockIdx.x >= total && *reinterpret_cast<volatile int*>(p.list) == 0) return;
  // Item t: tile t % tiles of piece t / tiles, whose stages are s0, s0 + 1, ... (nst of them).
  auto item = [&](int t, int& tile, int& z, int& s0) {
    z = t / p.tiles;
    tile = t - z * p.tiles;
    s0 = z * (p.kper / PK);
    return (min(p.kper, p.K - z * p.kper) + PK - 1) / PK;
  };

  if (tid == 0) {
    for (int s = 0; s < NST; s++) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int h = 0; h < 2; h++) {
      mbar_init(&acc_full[h], 1);
      mbar_init(&acc_empty[h], EPI_WARPS);
    }
    mbar_init(&last, 1);
    gave_up() = 0;
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
    for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
      int tile, z, s0, tm, tn;
      const int nst = item(t, tile, z, s0);
      if (!__ldg(p.fits + tile)) continue;
      tile_at(p, tile, tm, tn);
      // C's tile into L2 (its rows are 512 bytes; the epilogue's loads would wait for DRAM)
      if (p.prefetch)
        for (int q = lane; q < PM * 4; q += 32) {
          const int r = tm * PM + q / 4, c = tn * PN + q % 4 * 16;
          if (r < p.M && c < p.N)
            asm volatile("prefetch.global.L2 [%0];" ::"l"(p.C + (size_t)r * p.ldc + c));
        }
      if (lane == 0)
        for (int s = 0; s < nst; s++, n++) {
          const int b = n % NST;
          if (n >= NST && !sw_wait(&empty[b], (uint32_t)((n / NST - 1) & 1), p.err)) {
            ok = false;
            break;
          }
          unsigned char* st = smem + b * PST_BYTES;
          la_tma::mbar_expect_tx(&full[b], PST_BYTES);
          tma_load_3d(st, &ta, (s0 + s) * PK, tm * PM, 0, &full[b]);
          tma_load_3d(st + PA_BYTES, &tb, (s0 + s) * PK, tn * PN, 0, &full[b]);
        }
      ok = __shfl_sync(0xffffffffu, (int)ok, 0) != 0;
    }
    if (lane == 0 && !ok)  // this CTA's copies still in flight
      for (int k = max(0, n - NST); k < n; k++)
        la_tma::mbar_drain(&full[k % NST], (uint32_t)((k / NST) & 1));
  } else if (warp == EPI_WARPS + 1) {  // MMA issuer
    int n = 0, chunk = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
      int tile, z, s0;
      const int nst = item(t, tile, z, s0);
      if (!__ldg(p.fits + tile)) continue;
      if (lane == 0)
        for (int s = 0; s < nst && ok; s++, n++) {
          const int b = n % NST;
          const bool first = s % CHUNK_STAGES == 0;
          const bool end = s % CHUNK_STAGES == CHUNK_STAGES - 1 || s == nst - 1;
          if (!sw_wait(&full[b], (uint32_t)((n / NST) & 1), p.err)) ok = false;
          const uint32_t sa = smem_u32(smem + b * PST_BYTES), sb = sa + PA_BYTES;
          // accumulators 0-3, then 4-7: digit d of A with the digits t of B, d + t in the half
#pragma unroll
          for (int h = 0; h < 2; h++) {
            if (ok && first && chunk > 0 &&
                !sw_wait(&acc_empty[h], (uint32_t)((chunk - 1) & 1), p.err))
              ok = false;
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
            for (int k = 0; k < PK / 16; k++)
#pragma unroll
              for (int d = 0; d < (h ? SL : HG); d++) {
                const int t0 = h ? (d < HG ? HG - d : 0) : 0;
                const int t1 = h ? SL - d : HG - d;
                mma_f16(tmem + (d + t0) * PN, sdesc64(sa + d * (PM * PK * 2) + k * 32),
                        sdesc64(sb + t0 * (PN * PK * 2) + k * 32), idesc_f16((t1 - t0) * PN),
                        d == 0 && first && k == 0 ? 0u : 1u);
              }
            if (end) tc_commit(&acc_full[h]);
          }
          if (!ok) break;
          tc_commit(&empty[b]);
          if (end) chunk++;
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
    // A miss: fifteen of sixteen tiles (the others cost less as FMA chains than the look at all of them).
    // While the first accumulators are on their way.
    if (p.misses && blockIdx.x == 0 && tid == EPI_T - 1) {
      const long long left = *reinterpret_cast<volatile int*>(p.list);
      *p.misses = left * 16 >= (long long)p.tiles * 15 ? *p.misses + 1 : 0;
    }
    int chunk = 0;
    bool ok = true;
    for (int t = blockIdx.x; t < total && ok; t += gridDim.x) {
      int tile, z, s0, tm, tn;
      const int nchunk = (item(t, tile, z, s0) + CHUNK_STAGES - 1) / CHUNK_STAGES;
      if (!__ldg(p.fits + tile)) continue;
      tile_at(p, tile, tm, tn);
      double* C = p.C + z * p.czs;
      const int m0 = tm * PM, n0 = tn * PN;
      const int sr = m0 + row < p.M ? __ldg(p.ea + m0 + row) : 0;
      const int sc = n0 + col + (lane & 15) < p.N ? __ldg(p.eb + n0 + col + (lane & 15)) : 0;
      long long hi[16], lo[16];  // d[0..3] 2^(24 - 8 g), d[4..7] 2^(56 - 8 g)
#pragma unroll
      for (int j = 0; j < 16; j++) hi[j] = lo[j] = 0;
      for (int c = 0; c < nchunk && ok; c++, chunk++) {
#pragma unroll
        for (int h = 0; h < 2; h++) {
          // warp-uniform: every lane waits on the same phase
          ok = ok && __all_sync(0xffffffffu, sw_wait(&acc_full[h], (uint32_t)(chunk & 1), p.err));
          if (!ok) break;
          asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
          for (int j = 0; j < 16; j += 4) {
            uint32_t r[HG][4];
#pragma unroll
            for (int g = 0; g < HG; g++) tmem_ld4(tbase + (h * HG + g) * PN + j, r[g]);
            tmem_wait(r);
#pragma unroll
            for (int i = 0; i < 4; i++) {
              int d[HG];
#pragma unroll
              for (int g = 0; g < HG; g++) d[g] = __float2int_rn(__uint_as_float(r[g][i]));
              if (h == 0)  // d[0] 256 + d[1] and d[2] 256 + d[3] are below 2^31
                hi[j + i] += (long long)(d[0] * 256 + d[1]) * 65536 + (d[2] * 256 + d[3]);
              else
                lo[j + i] += (long long)d[0] * 16777216 + (long long)d[1] * 65536 +
                             (long long)d[2] * 256 + d[3];
            }
          }
          asm volatile("tcgen05.fence::before_thread_sync;");
          if (lane == 0) mbar_arrive(&acc_empty[h]);
        }
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
          if (MODE != 0) old[i] = gr < p.M && c < p.N ? C[(size_t)gr * p.ldc + c] : 0.0;
        }
#pragma unroll
        for (int j = 0; j < 8; j++) {
          const int eb = __shfl_sync(0xffffffffu, sc, g * 8 + j);
          wbuf[lane * 8 + (j ^ ((lane >> 1) & 7))] =
              round_sum(sum96(hi[g * 8 + j], lo[g * 8 + j]), sr + eb);
        }
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 8; i++) {
          const int r = 4 * i + (lane >> 3), gr = m0 + (warp & 3) * 32 + r;
          const double v = wbuf[r * 8 + (cc ^ ((r >> 1) & 7))];
          if (gr < p.M && c < p.N)
            C[(size_t)gr * p.ldc + c] = MODE == 0 ? v : MODE < 0 ? old[i] - v : old[i] + v;
        }
        __syncwarp();
      }
    }
    if (!ok) gave_up() = 1;
    // Every epilogue warp comes here, whatever its waits gave, and the list is the same for all. A warp
    // whose waits all ended has seen the last of the CTA's MMAs complete, and with them its copies.
    __syncwarp();
    if (*reinterpret_cast<volatile int*>(p.list) != 0)
      fma_tiles<MODE>(p, reinterpret_cast<double*>(smem + NST * PST_BYTES), tid);
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tmem));
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
  const bool lng = p.K >= GUARD_LONG_K;
  e = la_launch(ctx, lng ? guard_kernel<2> : guard_kernel<1>, dim3((p.tiles + p.per_cta - 1) / p.per_cta),
                dim3((lng ? 2 : 1) * GUARD_W * 32), 0, st, p);
  if (e != cudaSuccess) return la_cuda_fail(ctx, e, "guard_kernel launch");
  // CTAs beyond the tiles are for the FMA pieces (up to 32 of a tile) and leave at once without any. In
  // the factorizations, chains of dependent launches, each of them also keeps the kernels around this one
  // from being placed early: Cholesky of order 4099 (K <= 256) 7.70 ms with 32 CTAs at least, 7.74 with 64,
  // 8.27 with 120, 9.5 with all 152; QR of order 1000 (K = rows) 6.35 ms with 32, 6.37 with 112, 6.48 with
  // 128, 6.67 with all, and 9.04, 8.20, 8.13, 8.18 where the pieces are needed.
  const int items = p.tiles * p.splits;
  const int most = !ctx->pdl_now ? ctx->sm_count : p.K <= 256 ? 32 : std::max(32, ctx->sm_count - 40);
  const int grid = std::min(std::max(2 * items, std::min(32 * items, most)), ctx->sm_count);
  e = la_launch(ctx, gemm_split_kernel<MODE>, dim3(grid), dim3(SPLIT_T), SPLIT_SMEM, st, ta, tb, p);
  if (e != cudaSuccess) return la_cuda_fail(ctx, e, "gemm_split_kernel launch");
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

la_status launch_splits(la_ctx ctx, cudaStream_t st, const SplitSide& a, const SplitSide& b, bool same,
                        bool b_rows, int K, int kp, int* maxexp, int* list, const int* misses) {
  const int ra = (a.n + 7) / 8;
  const bool parts = !same && !b_rows && K > COLS_ALL_K;
  const int kper = parts ? 256 : 0, pieces = parts ? (K + kper - 1) / kper : 1;
  const int gx = (b.n + 31) / 32;
  const int rb = same ? 0 : b_rows ? (b.n + 7) / 8 : gx * pieces;
  if (parts) LA_CUDA(ctx, cudaMemsetAsync(maxexp, 0, (size_t)b.n * 2 * sizeof(int), st));
  cudaError_t e = la_launch(ctx, split_kernel, dim3(ra + rb), dim3(256), 0, st, a, b, K, kp, ra,
                            b_rows ? 1 : 0, kper, list, maxexp, misses);
  if (e != cudaSuccess) return la_cuda_fail(ctx, e, "split_kernel launch");
  ctx->launches++;
  if (parts) {
    e = la_launch(ctx, split_cols_part_kernel, dim3(gx, pieces), dim3(256), 0, st, b, K, kp, kper,
                  (const int*)maxexp, misses);
    if (e != cudaSuccess) return la_cuda_fail(ctx, e, "split_cols_part_kernel launch");
    ctx->launches++;
  }
  return la_check_launch(ctx, "split_kernel");
}

}  // namespace

size_t gemm_split_ws(int M, int N, int K, bool same) {
  const size_t kp = up(K, 8), tiles = up(M, PM) / PM * (up(N, PN) / PN + 2);
  return Side::bytes(M, kp) + (same ? 0 : Side::bytes(N, kp)) + up((2 * tiles + 1) * 4, 256);
}

la_status launch_gemm_split(la_ctx ctx, cudaStream_t st, int mode, int M, int N, int K,
                            const double* A, size_t lda, const double* B, size_t ldb, bool b_rows,
                            double* C, size_t ldc, bool tri, void* ws, size_t ws_bytes, int splits,
                            int kper, size_t czs, int* misses) {
  if (M <= 0 || N <= 0) return LA_OK;
  if (K <= 0 || K > SPLIT_MAX_K || (tri && M != N)) return LA_UNSUPPORTED;
  if (splits > 1 && (mode != 0 || kper % (CHUNK_STAGES * PK) || (long long)(splits - 1) * kper >= K ||
                     (long long)splits * kper < K))
    return LA_UNSUPPORTED;
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
  if (tiles * splits > (1 << 24)) return LA_UNSUPPORTED;
  p.splits = splits;
  p.kper = splits > 1 ? kper : (int)up(K, PK);
  p.czs = czs;
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
  p.prefetch = mode != 0;
  // tiles per CTA of the guard: one while that leaves SMs free, up to eight
  p.per_cta = std::min(GUARD_W, 1 + p.tiles / (4 * ctx->sm_count));
  p.da = sa.dig;
  p.db = sb.dig;
  p.kp = kp;
  p.joint = (int)std::ceil(1024.0 * GUARD * std::sqrt((double)K));
  p.list = list;
  p.fits = list + 1 + p.tiles;
  p.misses = misses;
  p.err = ctx->d_err;
  const SplitSide xa{A, lda, M, sa.dig, sa.exps, sa.cnt}, xb{B, ldb, N, sb.dig, sb.exps, sb.cnt};
  LA_TRY(launch_splits(ctx, st, xa, xb, same, b_rows, K, kp, sb.me, list, misses));
  if (mode < 0) return launch_product<-1>(ctx, st, ta, tb, p);
  if (mode == 0) return launch_product<0>(ctx, st, ta, tb, p);
  return launch_product<1>(ctx, st, ta, tb, p);
}
