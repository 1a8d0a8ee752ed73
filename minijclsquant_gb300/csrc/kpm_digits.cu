// kpm_digits.cu -- FP64 contractions of vector tables on the tensor cores, by exact digit
// products.
//
//   kpm_table_gram: mu[n][m] (+)= sum_i conj(U[n][i]) W[m][i]      (tables [M][n] complex128)
//   kpm_table_mix:  Q[k][i] = sum_m C[k][m] T[m][i]                (C real [M][M])
//
// GB300 multiplies FP64 at 1/64 of its FP32 rate, on the tensor cores too, so these two
// GEMMs were 86 % of a conductivity gradient.  Here every operand is cut, per row (or column) and
// block of kBlockK elements, into kDigits signed digits of 7 bits of a fixed-point number scaled
// by the block's largest exponent:
//
//   x = 2^(E - 1077) sum_s d_s 128^(7 - s),   |d_s| <= 64,  55 bits below 2^(E - 1022) > |x|
//
// (an element keeps all 53 bits of its mantissa down to a quarter of the block's power of two,
// and an absolute error of 2^-56 of it below).  Plane s holds d_s 2^(-7 s), exact in bf16, so a
// product of planes s and t carries its weight, and the sums of the products of equal weight,
//
//   D_d = sum_{s + t = d} sum_k a_{s,k} b_{t,k},   d < kDigits,
//
// stay below 2^12 * 8 * 512 = 2^24 units of that weight: every FP32 accumulation in TMEM is exact.
// The 36 digit pairs with s + t < 8 are 36 MMAs.  The seven pairs with s + t = 8, up to 2^-53 of the block
// maxima, are added to D_7's accumulator, whose last bits they round (2^-61).  (Mixes of 24 to 256 orders, rms
// error in units of 2^-53 sum |a b|: FP64 products 0.9 to 1.5, 36 pairs 0.9 to 2.7, 43 pairs 0.2 to 0.3.)
// The pairs beyond are worth 2^-60.  The eight
// sums are joined as one 64-bit integer and added in FP64, one rounding per 512 products (an
// FP64 GEMM rounds at every product).  (Error-free splitting of matrix products: K. Ozaki,
// T. Ogita, S. Oishi, S. M. Rump, Numer. Algorithms 59 (2012) 95.)
//
// A digit product errs by up to 2^-55 of the block's maxima, an FP64 product by 2^-53 of itself.  Where
// large elements of one operand meet small ones of the other, the first can be the larger, so a
// ninth plane holds |x| / 2^(E - 1022) rounded down (bf16), one more MMA a step sums
// T = sum_k |a_k b_k| from it, and an output whose blocks do not add up to
//
//   sum_blocks max|a| max|b| (T - [T > 0] / 4) >= 0        (max: the blocks' powers of two)
//
// is formed again as FP64 products (as is one whose scales leave 2^-900 .. 2^900).  So every output keeps the error bound of an FP64 dot product,
// K 2^-53 sum |a b|.  Of the tables of random vectors no gram output is; of their mixes none to a few in
// a hundred, at few orders the more.  Products with a zero factor are exact and do not count.
//
// The digit planes are written to the call's workspace by a slicing pass over a chunk of the tables that
// fits L2 (its planes are read back from there), and the GEMM kernel streams them through TMA.
// A non-finite element makes the outputs of its row (column) NaN.
//
// What bounds it: the MMAs.  A CTA's tile is 128 x 64 (eight accumulators of 64 columns fill
// TMEM), where the shared-memory reads of A (4 KB per MMA of K = 16) take longer than the
// multiplications.  Measured at 131,072 sites and 256 orders (K = 262,144 reals): 5.0 ms for a
// gram and 3.1 ms for a mix, slicing included, where the FP64 library GEMMs take 63.8 and 31.4 (36 pairs and no
// magnitudes: 3.4 and 2.4); a gradient of two vectors 45 ms instead of 295.  At the smallest sizes (a few
// hundred sites, a few dozen orders) both are a few launches, so there is no second path.
#include <cuda_bf16.h>

#include <algorithm>
#include <type_traits>

#include "kpm_async.cuh"
#include "kpm_internal.cuh"
#include "kpm_tc.cuh"

namespace kpm {
namespace {

constexpr int kDigits = 8;          // digits of 7 bits
constexpr int kPlanes = kDigits + 1;  // and the magnitudes
constexpr int kBlockK = 512;        // elements of one exponent block = one exact accumulation
constexpr int kStageK = 32;         // elements of K per shared-memory stage (64 bytes of bf16)
constexpr int kTM = 128, kTN = 64;  // output tile
constexpr uint32_t kPlaneA = kTM * kStageK * 2;                    // 8 KB
constexpr uint32_t kPlaneB = kTN * kStageK * 2;                    // 4 KB
constexpr uint32_t kStage = kDigits * (kPlaneA + kPlaneB);         // 96 KB: 32 columns of all digits, or 256 of the magnitudes
constexpr int kStages = 2;
constexpr uint32_t kSmem = kStages * kStage + 1024;
constexpr int kEpiWarps = 8;                                       // two per TMEM lane quarter
constexpr int kThreads = 32 * (kEpiWarps + 2);                     // + TMA producer, MMA issuer
constexpr int kEpiCols = kTN / 2;
static_assert(kDigits * 4096LL * kBlockK <= (1 << 24), "every accumulation is exact");
static_assert(kDigits * kTN == 512, "the accumulators fill TMEM");
static_assert(kEpiCols == 32, "a mask word a thread");

// kind::f16, A = B = bf16, D = FP32, both K-major
constexpr uint32_t idesc_bf16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc,
                                        bool accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
      "l"(a_desc), "l"(b_desc), "r"(idesc), "r"((uint32_t)accumulate)
      : "memory");
}

__device__ __forceinline__ void tma_load_3d(void* dst, const CUtensorMap* map, int c0, int c1, int c2, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], "
      "[%5];" ::"r"(smem_addr(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(c0), "r"(c1), "r"(c2), "r"(smem_addr(bar))
      : "memory");
}

__device__ __forceinline__ void tmem_ld8_nowait(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr)
               : "memory");
}

// ---- slicing ---------------------------------------------------------------------------------
// Biased exponent of |x| (subnormals count as exponent 1, 2047 for Inf and NaN).
__device__ __forceinline__ int exponent_of(double x) {
  const int e = (__double2hiint(x) >> 20) & 0x7ff;
  return e > 1 ? e : 1;
}

// Biased digit fields of x for block exponent E: field s is d_s + 64 at bit 7 (7 - s), the top
// one (0 .. 128) unmasked.
__device__ __forceinline__ uint64_t digit_fields(double x, int E) {
  constexpr uint64_t kBias = 64ull * 0x0002040810204081ull;  // 64 (1 + 128 + ... + 128^7)
  const uint32_t hi = (uint32_t)__double2hiint(x), lo = (uint32_t)__double2loint(x);
  const int e = (hi >> 20) & 0x7ff;
  const uint64_t m = ((uint64_t)((hi & 0xfffffu) | (e ? 0x100000u : 0u)) << 32) | lo;
  const int sh = E - (e > 1 ? e : 1) - 2;  // >= -2
  uint64_t X;
  if (sh <= 0)
    X = m << (-sh);
  else
    X = sh < 56 ? (m + (1ull << (sh - 1))) >> sh : 0ull;  // round to nearest
  return (hi >> 31) ? kBias - X : kBias + X;
}

// Digit s of two elements as a pair of bf16 d 2^(-7 s) (128 + field is exact, times the weight minus
// 192 of them).
__device__ __forceinline__ uint32_t digit_pair(uint64_t f0, uint64_t f1, int s) {
  const uint32_t u0 = s == 0 ? (uint32_t)(f0 >> 49) : (uint32_t)(f0 >> (7 * (7 - s))) & 127u;
  const uint32_t u1 = s == 0 ? (uint32_t)(f1 >> 49) : (uint32_t)(f1 >> (7 * (7 - s))) & 127u;
  const uint32_t p = 0x43004300u + (u0 | (u1 << 16));
  const float w = __int_as_float((127 - 7 * s) << 23);
  const __nv_bfloat162 h = __hfma2(*reinterpret_cast<const __nv_bfloat162*>(&p), __floats2bfloat162_rn(w, w),
                                   __floats2bfloat162_rn(-192.f * w, -192.f * w));
  return *reinterpret_cast<const uint32_t*>(&h);
}

// |x| 2^(1022 - E) as bf16 bits, rounded down; not below 2^-31 for a nonzero x, so that a sum of
// products is zero only where every product is.
__device__ __forceinline__ uint32_t magnitude(double x, int E) {
  const uint32_t hi = (uint32_t)__double2hiint(x) & 0x7fffffffu;
  if ((hi | (uint32_t)__double2loint(x)) == 0u) return 0u;
  const int f = (int)(hi >> 20) - E + 126;
  return f < 96 ? 96u << 7 : ((uint32_t)f << 7) | ((hi >> 13) & 127u);
}
__device__ __forceinline__ uint32_t magnitude_pair(double x0, double x1, int E) {
  return magnitude(x0, E) | (magnitude(x1, E) << 16);
}

// The power of two of a block's sums (2^(E - 1077), and for the two operands together 2^49 of the
// joined sum's last digit and the 2^12 that the epilogue takes back), NaN for a block that holds a non-finite element.
__device__ __forceinline__ double block_scale(int emax, int E, int shift) {
  if (emax == 2047) return __longlong_as_double(0x7ff8000000000000ll);
  return __longlong_as_double((long long)(E - shift) << 52);
}

// Block exponents below this are raised to it, so every scale is a normal number.
constexpr int kMinE = 64;

struct SliceRows {
  const double* src;  // [rows][ld]
  int64_t ld;
  int64_t k0, kvalid;  // first column of the chunk; columns of the source from there on
  int rows, nkb;       // blocks of kBlockK in the chunk
  int64_t plane, kc;   // elements of one plane, of one plane row
  __nv_bfloat16* out;  // planes [kPlanes][plane]; row r at r * kc
  int64_t swap_off;    // > 0: also rows with every pair (x, y) as (-y, x), this many elements further
  double* scale;       // [rows][nkb]
  int scale_swap;      // > 0: the scales again this many entries further
  int shift;
};

// One warp per (row, block): 16 elements a lane, two runs of eight.
__global__ void __launch_bounds__(256) slice_rows_kernel(const SliceRows p) {
  const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (w >= (int64_t)p.rows * p.nkb) return;
  const int row = (int)(w / p.nkb), kb = (int)(w % p.nkb);
  const double* src = p.src + (int64_t)row * p.ld + p.k0;
  double x[2][8];
  int emax = 1;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int64_t k = (int64_t)kb * kBlockK + h * 256 + lane * 8;
#pragma unroll
    for (int i = 0; i < 8; i += 2) {
      double2 v = make_double2(0.0, 0.0);
      if (k + i + 1 < p.kvalid)
        v = __ldg(reinterpret_cast<const double2*>(src + k + i));
      else if (k + i < p.kvalid)
        v.x = __ldg(src + k + i);
      x[h][i] = v.x;
      x[h][i + 1] = v.y;
      emax = max(emax, max(exponent_of(v.x), exponent_of(v.y)));
    }
  }
  emax = __reduce_max_sync(0xffffffffu, emax);
  const int E = max(emax, kMinE);
  if (lane == 0) {
    const double s = block_scale(emax, E, p.shift);
    p.scale[(int64_t)row * p.nkb + kb] = s;
    if (p.scale_swap > 0) p.scale[p.scale_swap + (int64_t)row * p.nkb + kb] = s;
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int64_t k = (int64_t)kb * kBlockK + h * 256 + lane * 8;
    if (k >= p.kc) continue;
    uint64_t f[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) f[i] = digit_fields(emax == 2047 ? 0.0 : x[h][i], E);
    __nv_bfloat16* out = p.out + (int64_t)row * p.kc + k;
#pragma unroll
    for (int s = 0; s < kDigits; ++s) {
      uint4 q;
      q.x = digit_pair(f[0], f[1], s);
      q.y = digit_pair(f[2], f[3], s);
      q.z = digit_pair(f[4], f[5], s);
      q.w = digit_pair(f[6], f[7], s);
      *reinterpret_cast<uint4*>(out + s * p.plane) = q;
      if (p.swap_off > 0) {
        auto sw = [](uint32_t v) { return ((v >> 16) ^ 0x8000u) | (v << 16); };
        *reinterpret_cast<uint4*>(out + s * p.plane + p.swap_off) = make_uint4(sw(q.x), sw(q.y), sw(q.z), sw(q.w));
      }
    }
    const uint4 q = make_uint4(magnitude_pair(x[h][0], x[h][1], E), magnitude_pair(x[h][2], x[h][3], E),
                               magnitude_pair(x[h][4], x[h][5], E), magnitude_pair(x[h][6], x[h][7], E));
    *reinterpret_cast<uint4*>(out + kDigits * p.plane) = q;
    if (p.swap_off > 0) {
      auto sw = [](uint32_t v) { return (v >> 16) | (v << 16); };
      *reinterpret_cast<uint4*>(out + kDigits * p.plane + p.swap_off) = make_uint4(sw(q.x), sw(q.y), sw(q.z), sw(q.w));
    }
  }
}

struct SliceCols {
  const double* src;  // [M][ld]: column j of the chunk is src[m * ld + j]
  int64_t ld;
  int M, nkb;
  int64_t cols;       // columns of the chunk
  int64_t plane, kp;  // elements of one plane, of one plane row (K padded)
  __nv_bfloat16* out;  // planes [kPlanes][cols][kp]
  double* scale;      // [cols][nkb]
};

// 64 columns and one block of kBlockK orders per CTA: a pass for the columns' largest
// exponents, then 16 orders of one column a thread (whole 32-byte sectors of the planes).
__global__ void __launch_bounds__(256) slice_cols_kernel(const SliceCols p) {
  __shared__ int se[4][64];
  const int c = threadIdx.x & 63, grp = threadIdx.x >> 6;
  const int64_t j = (int64_t)blockIdx.x * 64 + c;
  const int kb = blockIdx.y;
  const int m0 = kb * kBlockK, m1 = min(p.M, m0 + kBlockK);
  const bool in = j < p.cols;
  int emax = 1;
  if (in)
    for (int m = m0 + grp; m < m1; m += 4) emax = max(emax, exponent_of(__ldg(p.src + (int64_t)m * p.ld + j)));
  se[grp][c] = emax;
  __syncthreads();
  emax = max(max(se[0][c], se[1][c]), max(se[2][c], se[3][c]));
  const int E = max(emax, kMinE);
  if (!in) return;
  if (grp == 0) p.scale[j * p.nkb + kb] = block_scale(emax, E, 24);
  const int mp = (int)min((int64_t)m0 + kBlockK, p.kp);  // the padded end of this block
  for (int m = m0 + 16 * grp; m < mp; m += 64) {
    uint64_t f[16];
    uint32_t g[8];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const double x = (m + i < m1 && emax != 2047) ? __ldg(p.src + (int64_t)(m + i) * p.ld + j) : 0.0;
      f[i] = digit_fields(x, E);
      const uint32_t a = magnitude(x, E);
      g[i / 2] = i & 1 ? g[i / 2] | (a << 16) : a;
    }
    __nv_bfloat16* out = p.out + j * p.kp + m;
#pragma unroll
    for (int s = 0; s < kDigits; ++s) {
      uint4 q[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        q[h].x = digit_pair(f[8 * h + 0], f[8 * h + 1], s);
        q[h].y = digit_pair(f[8 * h + 2], f[8 * h + 3], s);
        q[h].z = digit_pair(f[8 * h + 4], f[8 * h + 5], s);
        q[h].w = digit_pair(f[8 * h + 6], f[8 * h + 7], s);
      }
      uint4* o = reinterpret_cast<uint4*>(out + s * p.plane);
      o[0] = q[0];
      o[1] = q[1];
    }
    uint4* o = reinterpret_cast<uint4*>(out + kDigits * p.plane);
    o[0] = make_uint4(g[0], g[1], g[2], g[3]);
    o[1] = make_uint4(g[4], g[5], g[6], g[7]);
  }
}

// ---- the product -----------------------------------------------------------------------------
struct DigitGemm {
  int rows_a, rows_b;  // valid rows of the operands (output rows, columns)
  int mt;              // row tiles; tile index = column tile * mt + row tile
  int nkb, blocks;     // exponent blocks of a row of scales, and those of this K
  int kp;              // elements of K (a multiple of kStageK)
  const double* sa;    // [rows_a][nkb]
  const double* sb;    // [rows_b][nkb]
  double* out;         // element (row, col) at out + split * split_stride + row * ldo + col
  float* guard;        // likewise sum_blocks scale (T - [T > 0] kLeast) of the magnitudes; or, where null,
  uint32_t* mask;      // [rows_a][mask_ld] words of the outputs where that sum is negative
  int mask_ld;
  int64_t ldo, split_stride;
  int accumulate;
  int* err;
  // Budget of every wait in SM clock cycles.  Test hook (kpm_table_test_timeout): kWithholdStage arms the
  // first stage and issues no copy for it; an epilogue warp's index makes that warp's first wait run out.
  long long wait_budget;
  int test;
};
enum { kNoTest = -1, kWithholdStage = -2 };

// What the magnitudes' product demands of a block: T >= kLeast max|a| max|b|.
constexpr float kLeast = 0.25f;
// The sum over blocks runs in FP32 (FP64 instructions would take longer than the products): in units of
// the CTA's largest blocks of the row and the column, each block's share of that not below kLeastShare
// (2^-60: there only negative terms count, so the sum is never too large).
constexpr int kShareBits = 60;
__device__ __forceinline__ int scale_field(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }
__device__ __forceinline__ float block_share(int field, int top) {
  return __int_as_float((127 + max(field - top, -kShareBits)) << 23);
}
// Whether the digits can form the products of two blocks: exponents of both scales and of their product
// within 2^+-900 (kNone: a non-finite element).
constexpr int kNone = 2047, kLow = 1023 - 900, kHigh = 1023 + 900;

// The digits' products of a CTA's blocks, then the magnitudes' product of the same blocks (8 steps of K in
// a stage, the first accumulator).  As a launch of its own the second took 57 us a chunk, most of it the start
// and the end of its CTAs; behind the first it takes 18.
__global__ void __launch_bounds__(kThreads, 1)
    digit_gemm_kernel(const DigitGemm p, const __grid_constant__ CUtensorMap map_a,
                      const __grid_constant__ CUtensorMap map_b) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full[kStages], empty[kStages], tfull, tfree;
  __shared__ uint32_t tmem_slot;
  __shared__ double ssb[kTN];
  __shared__ int scol[kTN], stop[kTN];  // the columns' scale fields of a block, the largest of the CTA
  __shared__ int dead_flag;  // a wait of the epilogue ran out

  const int row0 = (blockIdx.x % p.mt) * kTM, col0 = (blockIdx.x / p.mt) * kTN;
  const int kb0 = (int)((int64_t)blockIdx.y * p.blocks / gridDim.y),
            kb1 = (int)((int64_t)(blockIdx.y + 1) * p.blocks / gridDim.y);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(&tfull, 1);
    mbar_init(&tfree, kEpiWarps);
    fence_mbar_init();
    dead_flag = 0;
  }
  if (warp == 0) {
    tmem_alloc(&tmem_slot, 512);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  auto steps_of = [&](int kb) { return (min(p.kp, (kb + 1) * kBlockK) - kb * kBlockK) / kStageK; };
  // planes (or steps, of the magnitudes) in stage ks of a block
  auto parts_of = [&](bool mag, int kb, int ks) { return mag ? min(kDigits, steps_of(kb) - ks * kDigits) : kDigits; };
  auto stages_of = [&](bool mag, int kb) { return mag ? (steps_of(kb) + kDigits - 1) / kDigits : steps_of(kb); };

  if (warp == kEpiWarps) {  // producer
    if (lane == 0) {
      int issued = 0;
      bool ok = true;
      for (int pass = 0; pass < 2; ++pass)
        for (int kb = kb0; kb < kb1 && ok; ++kb)
          for (int ks = 0; ks < stages_of(pass, kb) && ok; ++ks) {
            const int st = issued % kStages;
            if (issued >= kStages) ok = mbar_wait_bounded(&empty[st], (uint32_t)((issued / kStages - 1) & 1), p.wait_budget);
            if (!ok) break;
            const int parts = parts_of(pass, kb, ks);
            mbar_arrive_expect_tx(&full[st], (uint32_t)parts * (kPlaneA + kPlaneB));
            unsigned char* a = smem + (size_t)st * kStage;
            unsigned char* b = a + kDigits * kPlaneA;
            const bool withhold = p.test == kWithholdStage && issued == 0;
            for (int s = 0; s < parts && !withhold; ++s) {
              const int k = kb * kBlockK + (pass ? ks * kDigits + s : ks) * kStageK, plane = pass ? kDigits : s;
              tma_load_3d(a + s * kPlaneA, &map_a, k, row0, plane, &full[st]);
              tma_load_3d(b + s * kPlaneB, &map_b, k, col0, plane, &full[st]);
            }
            ++issued;
          }
      if (!ok) atomicExch(p.err, KPM_ERR_TIMEOUT);
      for (int q = max(0, issued - kStages); q < issued; ++q)  // nothing is in flight when the CTA leaves
        (void)mbar_wait_bounded(&full[q % kStages], (uint32_t)((q / kStages) & 1), p.wait_budget);
    }
  } else if (warp == kEpiWarps + 1) {  // MMA issuer
    if (lane == 0) {
      const uint32_t idesc = idesc_bf16(kTM, kTN);
      const uint32_t base = smem_addr(smem);
      auto desc = [](uint32_t addr) { return smem_desc(addr, 16, 512) | ((uint64_t)4 << 61); };
      int it = 0, blk = 0;
      bool ok = true;
      for (int pass = 0; pass < 2; ++pass)
        for (int kb = kb0; kb < kb1 && ok; ++kb, ++blk) {
          if (blk > 0) ok = mbar_wait_bounded(&tfree, (uint32_t)((blk - 1) & 1), p.wait_budget);
          tc_fence_after();
          const int ns = stages_of(pass, kb);
          for (int ks = 0; ks < ns && ok; ++ks) {
            const int st = it % kStages;
            ok = mbar_wait_bounded(&full[st], (uint32_t)((it / kStages) & 1), p.wait_budget);
            if (!ok) break;
            tc_fence_after();
            const uint32_t a0 = base + (uint32_t)st * kStage, b0 = a0 + kDigits * kPlaneA;
            if (pass == 0) {
#pragma unroll 1
              for (int j = 0; j < kStageK / 16; ++j)
#pragma unroll
                for (int s = 0; s < kDigits; ++s)
#pragma unroll
                  for (int t = 0; t < (s == 0 ? kDigits : kDigits + 1 - s); ++t)
                    mma_f16(tmem + (uint32_t)((s + t < kDigits ? s + t : kDigits - 1) * kTN),
                            desc(a0 + s * kPlaneA + j * 32), desc(b0 + t * kPlaneB + j * 32), idesc,
                            s > 0 || j > 0 || ks > 0);
            } else {
              const int parts = parts_of(true, kb, ks);
#pragma unroll 1
              for (int s = 0; s < parts; ++s)
                for (int j = 0; j < kStageK / 16; ++j)
                  mma_f16(tmem, desc(a0 + s * kPlaneA + j * 32), desc(b0 + s * kPlaneB + j * 32), idesc,
                          s > 0 || j > 0 || ks > 0);
            }
            mma_commit(&empty[st]);
            ++it;
          }
          if (ok) mma_commit(&tfull);
        }
      if (!ok) atomicExch(p.err, KPM_ERR_TIMEOUT);
      // every MMA issued is finished before the accumulators are released, also when the epilogue left early
      if (it > 0)
        (void)mbar_wait_bounded(&empty[(it - 1) % kStages], (uint32_t)(((it - 1) / kStages) & 1), p.wait_budget);
    }
  } else {  // epilogue: thread = output row 32 q + lane, half of the columns
    const int q = warp & 3, cb = (warp >> 2) * kEpiCols;
    const int row = row0 + 32 * q + lane;
    const int srow = min(row, p.rows_a - 1);
    const uint32_t t0 = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)cb;
    const int col = threadIdx.x;  // of this thread's entry of ssb, scol, stop
    const double* scale_b = p.sb + (int64_t)min(col0 + col, p.rows_b - 1) * p.nkb;
    const double* scale_a = p.sa + (int64_t)srow * p.nkb;
    // One warp's wait may run out while another's completes in time.  The outcome is shared at the
    // barrier that ends the block, so that all warps leave the loop together: a warp that went on
    // alone would wait at the next barrier for ever.
    bool dead = false;
    int blk = 0;
    auto begin_block = [&]() -> bool {
      named_sync(32 * kEpiWarps);
      bool ok = mbar_wait_bounded(&tfull, (uint32_t)(blk & 1), p.wait_budget);
      ok = __all_sync(0xffffffffu, ok && p.test != warp);
      if (!ok && lane == 0) {
        atomicExch(p.err, KPM_ERR_TIMEOUT);
        *static_cast<volatile int*>(&dead_flag) = 1;
      }
      if (ok) tc_fence_after();
      return ok;
    };
    auto end_block = [&]() {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(&tfree);
      named_sync(32 * kEpiWarps);  // ssb and scol are rewritten for the next block
      dead = *static_cast<volatile int*>(&dead_flag) != 0;  // the next write to it lies behind the next block's barrier
      ++blk;
    };
    const int64_t at = (int64_t)blockIdx.y * p.split_stride + (int64_t)row * p.ldo + col0 + cb;
    {
      double acc[kEpiCols];
#pragma unroll
      for (int c = 0; c < kEpiCols; ++c) acc[c] = 0.0;
      for (int kb = kb0; kb < kb1 && !dead; ++kb) {
        // a block of 2^l products has joined sums below 2^(61 + l) (1 + 2^-5): the l - 1 bits that do
        // not fit 63 are rounded off (the pairs left out are worth more than that)
        const int len = min(p.kp, (kb + 1) * kBlockK) - kb * kBlockK;  // 32 .. 512
        const int sh = 31 - __clz(len - 1);                            // ceil(log2 len) - 1
        const double sa = __ldg(scale_a + kb) * __longlong_as_double((long long)(1011 + sh) << 52);
        if (col < kTN) ssb[col] = __ldg(scale_b + kb);
        if (begin_block()) {
#pragma unroll
          for (int g = 0; g < kEpiCols / 8; ++g) {
            uint32_t r[kDigits][8];
#pragma unroll
            for (int d = 0; d < kDigits; ++d) tmem_ld8_nowait(t0 + (uint32_t)(d * kTN + g * 8), r[d]);
            tmem_wait_ld();
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              long long hi = 0, lo = 0;  // sum_d D_d 128^(3 - d), sum_d D_{4 + d} 128^(3 - d): below 2^46
#pragma unroll
              for (int d = 0; d < 4; ++d) {
                hi = hi * 128 + __float2int_rn(__uint_as_float(r[d][c]) * (float)(1 << 7 * d));
                lo = lo * 128 + __float2int_rn(__uint_as_float(r[4 + d][c]) * (float)(1ll << 7 * (4 + d)));
              }
              const double D = (double)(hi * (1ll << (28 - sh)) + ((lo + (1ll << (sh - 1))) >> sh));  // joined / 2^sh
              acc[8 * g + c] = fma(D * sa, ssb[cb + 8 * g + c], acc[8 * g + c]);
            }
          }
        }
        end_block();
      }
      if (!dead && row < p.rows_a) {
        double* out = p.out + at;
#pragma unroll
        for (int c = 0; c < kEpiCols; c += 2) {
          if (col0 + cb + c + 1 < p.rows_b) {
            double2 v = make_double2(acc[c], acc[c + 1]);
            double2* o = reinterpret_cast<double2*>(out + c);
            if (p.accumulate) {
              const double2 old = *o;
              v.x += old.x;
              v.y += old.y;
            }
            *o = v;
          } else if (col0 + cb + c < p.rows_b) {
            out[c] = acc[c] + (p.accumulate ? out[c] : 0.0);
          }
        }
      }
    }
    {
      float acc[kEpiCols];
#pragma unroll
      for (int c = 0; c < kEpiCols; ++c) acc[c] = 0.f;
      auto top_of = [&](const double* scale) {
        int top = 1;
        for (int kb = kb0; kb < kb1; ++kb) {
          const int f = scale_field(__ldg(scale + kb));
          if (f != kNone) top = max(top, f);
        }
        return top;
      };
      const int top = top_of(scale_a);
      if (col < kTN) stop[col] = top_of(scale_b);
      for (int kb = kb0; kb < kb1 && !dead; ++kb) {
        const int fa = scale_field(__ldg(scale_a + kb));
        if (col < kTN) scol[col] = scale_field(__ldg(scale_b + kb));
        if (begin_block()) {
          const float wa = block_share(fa, top);
#pragma unroll
          for (int g = 0; g < kEpiCols / 8; ++g) {
            uint32_t r[8];
            tmem_ld8_nowait(t0 + (uint32_t)(g * 8), r);
            tmem_wait_ld();
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              const int fb = scol[cb + 8 * g + c], low = fb - stop[cb + 8 * g + c];
              const float T = __uint_as_float(r[c]), w = wa * block_share(low, 0);
              float x = T > 0.f ? T - kLeast : 0.f;
              if (x > 0.f && min(fa - top, low) <= -kShareBits) x = 0.f;
              const int lo = min(min(fa, fb), fa + fb - 1023), hi = max(max(fa, fb), fa + fb - 1023);
              if (T > 0.f && (lo < kLow || hi > kHigh)) x = -__int_as_float(0x7f800000);
              if (max(fa, fb) == kNone) x = __int_as_float(0x7fffffff);  // NaN: the digits give it
              acc[8 * g + c] = fmaf(x, w, acc[8 * g + c]);
            }
          }
        }
        end_block();
      }
      if (!dead && row < p.rows_a) {
        uint32_t bits = 0;
#pragma unroll
        for (int c = 0; c < kEpiCols; ++c) bits |= acc[c] < 0.f ? 1u << c : 0u;
        if (p.guard) {
#pragma unroll
          for (int c = 0; c < kEpiCols; ++c)
            if (col0 + cb + c < p.rows_b) {
              // in units that all CTAs share; where FP32 does not reach, a negative sum decides alone
              const int k = top + stop[cb + c] - 2 * 1023;
              float v = acc[c];
              if (k >= -100 && k <= 100)
                v *= __int_as_float((127 + k) << 23);
              else if (v != 0.f)
                v = v < 0.f ? -__int_as_float(0x7f800000) : v > 0.f ? 0.f : v;
              float* o = p.guard + at + c;
              *o = v + (p.accumulate ? *o : 0.f);
            }
        } else {
          p.mask[(int64_t)row * p.mask_ld + (col0 + cb) / 32] = bits;
        }
      }
    }
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

// mu[n][m] = (accumulate ? mu : 0) + sum over splits, Re from rows n, Im from rows na + n; rows of mu ldm apart.
__global__ void gram_reduce_kernel(const double* __restrict__ part, int splits, int na, int nb, int ldo, int64_t ldm,
                                   int accumulate, double2* __restrict__ mu) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= na * nb) return;
  const int n = idx / nb, m = idx % nb;
  double re = 0.0, im = 0.0;
  for (int s = 0; s < splits; ++s) {
    const double* q = part + (int64_t)s * 2 * na * ldo;
    re += q[(int64_t)n * ldo + m];
    im += q[(int64_t)(na + n) * ldo + m];
  }
  double2* out = mu + (int64_t)n * ldm + m;
  double2 o = make_double2(re, im);
  if (accumulate) {
    o.x += out->x;
    o.y += out->y;
  }
  *out = o;
}

// Outputs of a gram whose magnitudes ask for it, as FP64 products of the tables: their partial sums are
// replaced.  32 outputs of a row at a time, a CTA for each that is formed again.
struct GramRepair {
  const double2* U;
  const double2* W;
  int64_t n;
  int na, nb;          // rows of U and of W
  const float* guard;  // [splits][2 na][ldo]
  double* part;
  int splits, ldo;
};

__global__ void __launch_bounds__(256) gram_repair_kernel(const GramRepair p) {
  __shared__ double red[8];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int words = (p.nb + 31) / 32;
  const int64_t stride = 2 * (int64_t)p.na * p.ldo;
  for (int64_t w = blockIdx.x; w < 2 * (int64_t)p.na * words; w += gridDim.x) {
    const int row = (int)(w / words), m0 = (int)(w % words) * 32;
    float g = 0.f;
    if (m0 + lane < p.nb)
      for (int s = 0; s < p.splits; ++s) g += p.guard[s * stride + (int64_t)row * p.ldo + m0 + lane];
    for (unsigned bits = __ballot_sync(0xffffffffu, g < 0.f); bits; bits &= bits - 1) {  // the same in every warp
      const int m = m0 + __ffs(bits) - 1;
      const bool im = row >= p.na;
      const double2* u = p.U + (int64_t)(im ? row - p.na : row) * p.n;
      const double2* x = p.W + (int64_t)m * p.n;
      double sum = 0.0;
      for (int64_t i = threadIdx.x; i < p.n; i += 256) {
        const double2 a = __ldg(u + i), b = __ldg(x + i);
        sum = im ? fma(a.x, b.y, fma(-a.y, b.x, sum)) : fma(a.x, b.x, fma(a.y, b.y, sum));
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
      if (lane == 0) red[warp] = sum;
      __syncthreads();
      if (threadIdx.x < p.splits) {
        double t = 0.0;
        for (int k = 0; k < 8; ++k) t += red[k];
        p.part[threadIdx.x * stride + (int64_t)row * p.ldo + m] = threadIdx.x == 0 ? t : 0.0;
      }
      __syncthreads();
    }
  }
}

// The same for a chunk of nc columns and some rows of a mix: mask [rows][ld] words.
__global__ void __launch_bounds__(256) mix_repair_kernel(const uint32_t* __restrict__ mask, int ld, int64_t nc,
                                                         int rows, int M,
                                                         const double* __restrict__ C, const double* __restrict__ T,
                                                         int64_t cols, double* __restrict__ Q) {
  const int lane = threadIdx.x & 31;
  // a warp's 32 words lie as far apart as there are warps: outputs to form again come in clusters (51 orders,
  // 118,592 sites, a row's words together 480 us a chunk, spread 85)
  const int64_t total = (int64_t)rows * ld, warps = (int64_t)gridDim.x * 8;
  for (int64_t w0 = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); w0 < total; w0 += warps * 32) {
    const uint32_t mine = w0 + lane * warps < total ? mask[w0 + lane * warps] : 0u;
    for (unsigned any = __ballot_sync(0xffffffffu, mine != 0u); any; any &= any - 1) {
      const int l = __ffs(any) - 1;
      const int64_t w = w0 + l * warps;
      const int row = (int)(w / ld);
      const double* c = C + (int64_t)row * M;
      for (uint32_t bits = __shfl_sync(0xffffffffu, mine, l); bits;) {
        // up to four outputs at a time, the lanes shared out among them
        const int left = __popc(bits), lg = left == 1 ? 5 : left == 2 ? 4 : 3;
        const int grp = lane >> lg, sub = lane & ((1 << lg) - 1);
        uint32_t b = bits;
        for (int i = 0; i < grp; ++i) b &= b - 1;
        for (int i = 0; i < 4; ++i) bits &= bits - 1;
        const int64_t j = (w % ld) * 32 + __ffs(b) - 1;
        const bool own = b != 0u && j < nc;  // past the last column the planes are whatever the workspace held
        double sum = 0.0;
        for (int m0 = 0; m0 < M; m0 += 8 << lg) {  // eight terms a lane in flight
          double x[8], y[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            const int m = m0 + (i << lg) + sub;
            const bool in = own && m < M;
            x[i] = in ? __ldg(c + m) : 0.0;
            y[i] = in ? __ldg(T + (int64_t)m * cols + j) : 0.0;
          }
#pragma unroll
          for (int i = 0; i < 8; ++i)
            if (m0 + (i << lg) < M) sum = fma(x[i], y[i], sum);
        }
        for (int o = 1 << (lg - 1); o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        if (own && sub == 0) Q[(int64_t)row * cols + j] = sum;
      }
    }
  }
}

// Planes [kPlanes][rows][k] of bf16 as a 3-D map; a box is one plane's 32 x box_rows piece in the
// 64-byte-swizzled layout.  Rows past the end read as zero digits.
bool plane_map(CUtensorMap* m, const __nv_bfloat16* base, int64_t k, int64_t rows, int box_rows) {
  const EncodeTiledFn enc = encode_tiled();
  if (!enc) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)k, (cuuint64_t)rows, (cuuint64_t)kPlanes};
  const cuuint64_t strides[2] = {(cuuint64_t)k * 2, (cuuint64_t)(k * rows) * 2};
  const cuuint32_t box[3] = {(cuuint32_t)kStageK, (cuuint32_t)box_rows, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<__nv_bfloat16*>(base), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int64_t round_up(int64_t x, int64_t m) { return (x + m - 1) / m * m; }

void launch_slice_rows(const SliceRows& p, cudaStream_t s) {
  const int64_t warps = (int64_t)p.rows * p.nkb;
  slice_rows_kernel<<<(unsigned)((warps + 7) / 8), 256, 0, s>>>(p);
}

// Planes of one chunk may take this much: they stay in L2 between the slicing pass and the product.
constexpr int64_t kPlaneBytes = 96ll << 20;

// The workspace of one call, from the caller: the tables' calls of a handle may be under way on several
// streams or in recorded graphs, so nothing of theirs is kept in the handle.  Offsets are multiples of
// kWorkAlign.
constexpr size_t kWorkAlign = 256;
struct WorkLayout {
  size_t bytes = 0;
  size_t take(size_t b) {
    const size_t o = bytes;
    bytes += (b + kWorkAlign - 1) / kWorkAlign * kWorkAlign;
    return o;
  }
};

// A call of many orders is cut: grams into blocks of kGramRows rows of U and of W, mixes into rows of C
// whose planes take kMixBytes, columns likewise, so that the workspace stays below 3 GB.
constexpr int kGramRows = 4096;
constexpr int64_t kMixBytes = 1ll << 30;

struct GramPlan {
  int rows;    // of U and of W in a block, at most
  int64_t kc;  // columns (reals) of a chunk
  int nkb, splits, ldo;
  size_t pa, pb, sa, sb, part, guard, bytes;
};

GramPlan gram_plan(const kpm_ell_s* h, int M) {
  GramPlan g{};
  const int64_t K = 2 * h->n;  // reals of a table row
  g.rows = std::min(M, kGramRows);
  // chunk of K: planes of U, its swapped form and W
  g.kc = kPlaneBytes / (kDigits * 3 * 2 * (int64_t)g.rows) / kBlockK * kBlockK;
  g.kc = std::max<int64_t>(4 * kBlockK, std::min<int64_t>(g.kc, 65536));
  g.kc = std::min(g.kc, round_up(K, kStageK));
  g.nkb = (int)((g.kc + kBlockK - 1) / kBlockK);
  const int tiles = (2 * g.rows + kTM - 1) / kTM * ((g.rows + kTN - 1) / kTN);
  g.splits = std::max(1, std::min(g.nkb, h->sm_count / tiles));
  g.ldo = (int)round_up(g.rows, 2);
  WorkLayout w;
  g.pa = w.take((size_t)kPlanes * 2 * g.rows * g.kc * sizeof(__nv_bfloat16));
  g.pb = w.take((size_t)kPlanes * g.rows * g.kc * sizeof(__nv_bfloat16));
  g.sa = w.take((size_t)2 * g.rows * g.nkb * sizeof(double));
  g.sb = w.take((size_t)g.rows * g.nkb * sizeof(double));
  g.part = w.take((size_t)g.splits * 2 * g.rows * g.ldo * sizeof(double));
  g.guard = w.take((size_t)g.splits * 2 * g.rows * g.ldo * sizeof(float));
  g.bytes = w.bytes;
  return g;
}

struct MixPlan {
  int rows;        // of C in a block, at most
  int64_t kp, nc;  // padded K; columns (reals) of a chunk
  int nkb;
  size_t pa, pb, cpad, sa, sb, mask, bytes;
};

MixPlan mix_plan(const kpm_ell_s* h, int M) {
  MixPlan g{};
  g.kp = round_up(M, 64);
  g.nkb = (int)((g.kp + kBlockK - 1) / kBlockK);
  const int64_t most = std::max<int64_t>(1, kMixBytes / (kPlanes * 2 * g.kp) / kTM) * kTM;  // rows or columns
  g.rows = (int)std::min<int64_t>(M, most);
  // chunk of columns: whole waves of one CTA per SM, planes within the L2 budget
  const int64_t wave = std::max<int64_t>(1, h->sm_count / ((g.rows + kTM - 1) / kTM)) * kTN;
  g.nc = std::max<int64_t>(1, kPlaneBytes / (kDigits * 2 * g.kp) / wave) * wave;
  g.nc = std::min({g.nc, round_up(2 * h->n, kTN), most});
  WorkLayout w;
  g.pb = w.take((size_t)kPlanes * g.nc * g.kp * sizeof(__nv_bfloat16));
  g.pa = w.take((size_t)kPlanes * g.rows * g.kp * sizeof(__nv_bfloat16));
  g.cpad = w.take((size_t)g.rows * g.kp * sizeof(double));
  g.sa = w.take((size_t)g.rows * g.nkb * sizeof(double));
  g.sb = w.take((size_t)g.nc * g.nkb * sizeof(double));
  g.mask = w.take((size_t)g.rows * (round_up(g.nc, kTN) / 32) * sizeof(uint32_t));
  g.bytes = w.bytes;
  return g;
}

template <typename T>
T* at(void* work, size_t offset) {
  return reinterpret_cast<T*>(static_cast<char*>(work) + offset);
}

// Rows n0 .. n0 + na of U against rows m0 .. m0 + nb of W.
int gram_block(kpm_ell_s* h, const GramPlan& t, int M, const double* U, const double* W, int n0, int na, int m0, int nb,
               int accumulate, double* mu, void* work, cudaStream_t s) {
  const int64_t K = 2 * h->n, plane_a = 2 * (int64_t)na * t.kc, plane_b = (int64_t)nb * t.kc;
  __nv_bfloat16 *pa = at<__nv_bfloat16>(work, t.pa), *pb = at<__nv_bfloat16>(work, t.pb);
  double *sa = at<double>(work, t.sa), *sb = at<double>(work, t.sb), *part = at<double>(work, t.part);
  float* guard = at<float>(work, t.guard);
  CUtensorMap ma, mb;
  if (!plane_map(&ma, pa, t.kc, 2 * na, kTM) || !plane_map(&mb, pb, t.kc, nb, kTN)) return KPM_ERR_UNSUPPORTED;
  const double *u = U + (int64_t)n0 * K, *w = W + (int64_t)m0 * K;
  const int mt = (2 * na + kTM - 1) / kTM, nt = (nb + kTN - 1) / kTN;
  for (int64_t k0 = 0; k0 < K; k0 += t.kc) {
    const int64_t kv = std::min(t.kc, K - k0), kp = round_up(kv, kStageK);
    SliceRows a{};
    a.src = u;
    a.ld = K;
    a.k0 = k0;
    a.kvalid = kv;
    a.rows = na;
    a.nkb = t.nkb;
    a.plane = plane_a;
    a.kc = t.kc;
    a.out = pa;
    a.swap_off = (int64_t)na * t.kc;
    a.scale = sa;
    a.scale_swap = na * t.nkb;
    a.shift = 23;
    SliceRows b = a;
    b.src = w;
    b.rows = nb;
    b.plane = plane_b;
    b.out = pb;
    b.swap_off = 0;
    b.scale = sb;
    b.scale_swap = 0;
    b.shift = 24;
    launch_slice_rows(a, s);
    launch_slice_rows(b, s);
    DigitGemm g{};
    g.rows_a = 2 * na;
    g.rows_b = nb;
    g.mt = mt;
    g.nkb = t.nkb;
    g.blocks = (int)((kp + kBlockK - 1) / kBlockK);
    g.kp = (int)kp;
    g.sa = sa;
    g.sb = sb;
    g.out = part;
    g.ldo = t.ldo;
    g.split_stride = 2 * (int64_t)na * t.ldo;
    g.accumulate = k0 > 0;
    g.err = h->err_flag;
    g.wait_budget = kWaitBudgetCycles;
    g.test = kNoTest;
    g.guard = guard;
    digit_gemm_kernel<<<dim3(mt * nt, t.splits), kThreads, kSmem, s>>>(g, ma, mb);
    KPM_CUDA_TRY(cudaGetLastError());
  }
  GramRepair r{};
  r.U = reinterpret_cast<const double2*>(u);
  r.W = reinterpret_cast<const double2*>(w);
  r.n = h->n;
  r.na = na;
  r.nb = nb;
  r.guard = guard;
  r.part = part;
  r.splits = t.splits;
  r.ldo = t.ldo;
  gram_repair_kernel<<<(int)std::min<int64_t>(2 * (int64_t)na * ((nb + 31) / 32), 8 * h->sm_count), 256, 0, s>>>(r);
  KPM_CUDA_TRY(cudaGetLastError());
  gram_reduce_kernel<<<(na * nb + 255) / 256, 256, 0, s>>>(part, t.splits, na, nb, t.ldo, M, accumulate ? 1 : 0,
                                                           reinterpret_cast<double2*>(mu) + (int64_t)n0 * M + m0);
  return check_cuda(cudaGetLastError());
}

int gram(kpm_ell_s* h, int M, const double* U, const double* W, int accumulate, double* mu, void* work, cudaStream_t s) {
  KPM_TRY(allow_smem(digit_gemm_kernel, kSmem));
  const GramPlan t = gram_plan(h, M);
  for (int n0 = 0; n0 < M; n0 += t.rows)
    for (int m0 = 0; m0 < M; m0 += t.rows)
      KPM_TRY(gram_block(h, t, M, U, W, n0, std::min(t.rows, M - n0), m0, std::min(t.rows, M - m0), accumulate, mu, work, s));
  return KPM_OK;
}

// Rows r0 .. r0 + rows of C and of Q.
int mix_block(kpm_ell_s* h, const MixPlan& t, int M, const double* C, const double* T, double* Q, int r0, int rows,
              void* work, cudaStream_t s) {
  const int64_t cols = 2 * h->n, plane_a = (int64_t)rows * t.kp, plane_b = t.nc * t.kp;
  const int mt = (rows + kTM - 1) / kTM;
  const double* c = C + (int64_t)r0 * M;
  double* q = Q + (int64_t)r0 * cols;
  __nv_bfloat16 *pa = at<__nv_bfloat16>(work, t.pa), *pb = at<__nv_bfloat16>(work, t.pb);
  double *cpad = at<double>(work, t.cpad), *sa = at<double>(work, t.sa), *sb = at<double>(work, t.sb);
  uint32_t* mask = at<uint32_t>(work, t.mask);
  CUtensorMap ma, mb;
  if (!plane_map(&ma, pa, t.kp, rows, kTM) || !plane_map(&mb, pb, t.kp, t.nc, kTN)) return KPM_ERR_UNSUPPORTED;
  // C's rows: an odd M would leave them 8-byte aligned, so they are copied to an even pitch
  const double* csrc = c;
  int64_t cld = M;
  if ((M & 1) || (reinterpret_cast<uintptr_t>(c) & 15)) {
    KPM_CUDA_TRY(cudaMemcpy2DAsync(cpad, (size_t)t.kp * sizeof(double), c, (size_t)M * sizeof(double),
                                   (size_t)M * sizeof(double), rows, cudaMemcpyDeviceToDevice, s));
    csrc = cpad;
    cld = t.kp;
  }
  SliceRows a{};
  a.src = csrc;
  a.ld = cld;
  a.kvalid = M;
  a.rows = rows;
  a.nkb = t.nkb;
  a.plane = plane_a;
  a.kc = t.kp;
  a.out = pa;
  a.scale = sa;
  a.shift = 23;
  launch_slice_rows(a, s);
  for (int64_t j0 = 0; j0 < cols; j0 += t.nc) {
    const int64_t nc = std::min(t.nc, cols - j0);
    SliceCols b{};
    b.src = T + j0;
    b.ld = cols;
    b.M = M;
    b.nkb = t.nkb;
    b.cols = nc;
    b.plane = plane_b;
    b.kp = t.kp;
    b.out = pb;
    b.scale = sb;
    slice_cols_kernel<<<dim3((unsigned)((nc + 63) / 64), t.nkb), 256, 0, s>>>(b);
    DigitGemm g{};
    g.rows_a = rows;
    g.rows_b = (int)nc;
    g.mt = mt;
    g.nkb = t.nkb;
    g.blocks = (int)((t.kp + kBlockK - 1) / kBlockK);
    g.kp = (int)t.kp;
    g.sa = sa;
    g.sb = sb;
    g.out = q + j0;
    g.ldo = cols;
    g.err = h->err_flag;
    g.wait_budget = kWaitBudgetCycles;
    g.test = kNoTest;
    g.mask = mask;
    g.mask_ld = (int)(round_up(nc, kTN) / 32);
    digit_gemm_kernel<<<dim3((unsigned)(mt * ((nc + kTN - 1) / kTN)), 1), kThreads, kSmem, s>>>(g, ma, mb);
    KPM_CUDA_TRY(cudaGetLastError());
    mix_repair_kernel<<<(int)std::min<int64_t>(((int64_t)rows * g.mask_ld + 255) / 256, 8 * h->sm_count), 256, 0, s>>>(
        mask, g.mask_ld, nc, rows, M, c, T + j0, cols, q + j0);
    KPM_CUDA_TRY(cudaGetLastError());
  }
  return KPM_OK;
}

int mix(kpm_ell_s* h, int M, const double* C, const double* T, double* Q, void* work, cudaStream_t s) {
  KPM_TRY(allow_smem(digit_gemm_kernel, kSmem));
  const MixPlan t = mix_plan(h, M);
  for (int r0 = 0; r0 < M; r0 += t.rows)
    KPM_TRY(mix_block(h, t, M, C, T, Q, r0, std::min(t.rows, M - r0), work, s));
  return KPM_OK;
}

constexpr int kMaxOrders = 1 << 17;  // a moment matrix of 275 GB

bool misaligned(const void* a, const void* b) { return (reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15; }

// A call without a workspace takes one from the stream's memory pool for its own length.
template <typename F>
int with_work(kpm_ell_s* h, int M, cudaStream_t s, F call) {
  void* work = nullptr;
  KPM_TRY(check_cuda(cudaMallocAsync(&work, kpm_table_work_bytes(h, M), s)));
  const int st = call(work);
  const int fr = check_cuda(cudaFreeAsync(work, s));
  return st != KPM_OK ? st : fr;
}

}  // namespace
}  // namespace kpm

using namespace kpm;

extern "C" {

int64_t kpm_table_work_bytes(const kpm_ell* h, int M) {
  if (!h || M < 1 || M > kMaxOrders) return 0;
  return (int64_t)std::max(gram_plan(h, M).bytes, mix_plan(h, M).bytes);
}

int kpm_table_gram_work(kpm_ell* h, int M, const double* U, const double* W, int accumulate, double* mu, void* work,
                        int64_t work_bytes, void* stream) {
  if (!h || !U || !W || !mu || !work || M < 1 || misaligned(U, W)) return KPM_ERR_INVALID_ARG;
  if (M > kMaxOrders) return KPM_ERR_UNSUPPORTED;
  if (work_bytes < kpm_table_work_bytes(h, M) || reinterpret_cast<uintptr_t>(work) % kWorkAlign) return KPM_ERR_INVALID_ARG;
  return gram(h, M, U, W, accumulate, mu, work, reinterpret_cast<cudaStream_t>(stream));
}

int kpm_table_gram(kpm_ell* h, int M, const double* U, const double* W, int accumulate, double* mu, void* stream) {
  if (!h || !U || !W || !mu || M < 1 || misaligned(U, W)) return KPM_ERR_INVALID_ARG;
  if (M > kMaxOrders) return KPM_ERR_UNSUPPORTED;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  return with_work(h, M, s, [&](void* work) { return gram(h, M, U, W, accumulate, mu, work, s); });
}

int kpm_table_mix_work(kpm_ell* h, int M, const double* C, const double* T, double* Q, void* work, int64_t work_bytes,
                       void* stream) {
  if (!h || !C || !T || !Q || !work || M < 1 || misaligned(T, Q)) return KPM_ERR_INVALID_ARG;
  if (M > kMaxOrders) return KPM_ERR_UNSUPPORTED;
  if (work_bytes < kpm_table_work_bytes(h, M) || reinterpret_cast<uintptr_t>(work) % kWorkAlign) return KPM_ERR_INVALID_ARG;
  return mix(h, M, C, T, Q, work, reinterpret_cast<cudaStream_t>(stream));
}

int kpm_table_mix(kpm_ell* h, int M, const double* C, const double* T, double* Q, void* stream) {
  if (!h || !C || !T || !Q || M < 1 || misaligned(T, Q)) return KPM_ERR_INVALID_ARG;
  if (M > kMaxOrders) return KPM_ERR_UNSUPPORTED;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  return with_work(h, M, s, [&](void* work) { return mix(h, M, C, T, Q, work, s); });
}

int kpm_table_test_timeout(kpm_ell* h, int64_t budget_cycles, int warp, void* stream) {
  if (!h || budget_cycles < 1000 || budget_cycles > kWaitBudgetCycles || warp >= kEpiWarps) return KPM_ERR_INVALID_ARG;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  KPM_TRY(allow_smem(digit_gemm_kernel, kSmem));
  // one tile of zeros, four blocks of K
  const int64_t k = 4 * kBlockK;
  const size_t planes = (size_t)kPlanes * (kTM + kTN) * k * sizeof(__nv_bfloat16);
  const size_t scales = (size_t)(kTM + kTN) * 4 * sizeof(double), out = (size_t)2 * kTM * kTN * sizeof(double);
  DevBuf scratch;
  KPM_TRY(ensure(scratch, planes + scales + out));
  KPM_CUDA_TRY(cudaMemsetAsync(scratch.p, 0, planes + scales + out, s));
  KPM_CUDA_TRY(cudaMemsetAsync(h->err_flag, 0, sizeof(int), s));
  __nv_bfloat16* pa = static_cast<__nv_bfloat16*>(scratch.p);
  __nv_bfloat16* pb = pa + (size_t)kPlanes * kTM * k;
  double* sa = reinterpret_cast<double*>(pb + (size_t)kPlanes * kTN * k);
  CUtensorMap ma, mb;
  if (!plane_map(&ma, pa, k, kTM, kTM) || !plane_map(&mb, pb, k, kTN, kTN)) return KPM_ERR_UNSUPPORTED;
  DigitGemm g{};
  g.rows_a = kTM;
  g.rows_b = kTN;
  g.mt = 1;
  g.nkb = g.blocks = 4;
  g.kp = (int)k;
  g.sa = sa;
  g.sb = sa + kTM * 4;
  g.out = sa + (kTM + kTN) * 4;
  g.guard = reinterpret_cast<float*>(g.out + kTM * kTN);
  g.ldo = kTN;
  g.err = h->err_flag;
  g.wait_budget = budget_cycles;
  g.test = warp < 0 ? (int)kWithholdStage : warp;
  digit_gemm_kernel<<<1, kThreads, kSmem, s>>>(g, ma, mb);
  KPM_CUDA_TRY(cudaGetLastError());
  const int st = kpm_ell_check(h, stream);  // synchronises
  release(scratch);
  return st;
}

}  // extern "C"
