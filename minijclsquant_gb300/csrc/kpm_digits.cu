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
// and an absolute error of 2^-56 of it below).  Digits are exact in fp16, a product of two is at
// most 2^12, and the sums of the products of equal weight 128^-(s + t),
//
//   D_d = sum_{s + t = d} sum_k a_{s,k} b_{t,k},   d < kDigits,
//
// stay below 2^12 * 8 * 512 = 2^24: every FP32 accumulation in TMEM is exact.  The 36 digit
// pairs with s + t < 8 are 36 MMAs; the pairs left out are worth 2^-56 of the block maxima.  The eight
// sums are joined as one 64-bit integer and added in FP64, one rounding per 512 products (an
// FP64 GEMM rounds at every product).  (Error-free splitting of matrix products: K. Ozaki,
// T. Ogita, S. Oishi, S. M. Rump, Numer. Algorithms 59 (2012) 95.)
//
// The digit planes are written to the call's workspace by a slicing pass over a chunk of the tables that
// fits L2 (its planes are read back from there), and the GEMM kernel streams them through TMA.
// A non-finite element makes the outputs of its row (column) NaN.
//
// What bounds it: the MMAs.  A CTA's tile is 128 x 64 (eight accumulators of 64 columns fill
// TMEM), where the shared-memory reads of A (4 KB per MMA of K = 16) take longer than the
// multiplications.  Measured at 131,072 sites and 256 orders (K = 262,144 reals): 3.4 ms for a
// gram and 2.4 ms for a mix, slicing included, where the FP64 library GEMMs took 63.7 and 31.4;
// a gradient of two vectors 58 ms instead of 295.  At the smallest sizes (a few hundred sites,
// a few dozen orders) both are a few launches, so there is no second path.
#include <cuda_fp16.h>

#include <algorithm>

#include "kpm_async.cuh"
#include "kpm_internal.cuh"
#include "kpm_tc.cuh"

namespace kpm {
namespace {

constexpr int kDigits = 8;          // digits of 7 bits
constexpr int kBlockK = 512;        // elements of one exponent block = one exact accumulation
constexpr int kStageK = 32;         // elements of K per shared-memory stage (64 bytes of fp16)
constexpr int kTM = 128, kTN = 64;  // output tile
constexpr uint32_t kPlaneA = kTM * kStageK * 2;                    // 8 KB
constexpr uint32_t kPlaneB = kTN * kStageK * 2;                    // 4 KB
constexpr uint32_t kStage = kDigits * (kPlaneA + kPlaneB);         // 96 KB
constexpr int kStages = 2;
constexpr uint32_t kSmem = kStages * kStage + 1024;
constexpr int kEpiWarps = 8;                                       // two per TMEM lane quarter
constexpr int kThreads = 32 * (kEpiWarps + 2);                     // + TMA producer, MMA issuer
constexpr int kEpiCols = kTN / 2;
static_assert(kDigits * 4096LL * kBlockK <= (1 << 24), "every accumulation is exact");
static_assert(kDigits * kTN == 512, "the accumulators fill TMEM");

// kind::f16, A = B = fp16, D = FP32, both K-major
constexpr uint32_t idesc_f16(int M, int N) {
  return (1u << 4) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
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

// Digit s of two elements as a pair of fp16 (1024 + field is exact, minus 1088).
__device__ __forceinline__ uint32_t digit_pair(uint64_t f0, uint64_t f1, int s) {
  const uint32_t u0 = s == 0 ? (uint32_t)(f0 >> 49) : (uint32_t)(f0 >> (7 * (7 - s))) & 127u;
  const uint32_t u1 = s == 0 ? (uint32_t)(f1 >> 49) : (uint32_t)(f1 >> (7 * (7 - s))) & 127u;
  const uint32_t p = 0x64006400u + (u0 | (u1 << 16));
  const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&p), __floats2half2_rn(1088.f, 1088.f));
  return *reinterpret_cast<const uint32_t*>(&h);
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
  __half* out;         // planes [kDigits][plane]; row r at r * kc
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
    __half* out = p.out + (int64_t)row * p.kc + k;
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
  }
}

struct SliceCols {
  const double* src;  // [M][ld]: column j of the chunk is src[m * ld + j]
  int64_t ld;
  int M, nkb;
  int64_t cols;       // columns of the chunk
  int64_t plane, kp;  // elements of one plane, of one plane row (K padded)
  __half* out;        // planes [kDigits][cols][kp]
  double* scale;      // [cols][nkb]
};

// 64 columns and one block of kBlockK orders per CTA: a pass for the columns' largest
// exponents, then 16 orders of one column a thread (whole 32-byte sectors of the planes).
__global__ void __launch_bounds__(256) slice_cols_kernel(const SliceCols p) {
  __shared__ int se[4][64];
  const int c = threadIdx.x & 63, g = threadIdx.x >> 6;
  const int64_t j = (int64_t)blockIdx.x * 64 + c;
  const int kb = blockIdx.y;
  const int m0 = kb * kBlockK, m1 = min(p.M, m0 + kBlockK);
  const bool in = j < p.cols;
  int emax = 1;
  if (in)
    for (int m = m0 + g; m < m1; m += 4) emax = max(emax, exponent_of(__ldg(p.src + (int64_t)m * p.ld + j)));
  se[g][c] = emax;
  __syncthreads();
  emax = max(max(se[0][c], se[1][c]), max(se[2][c], se[3][c]));
  const int E = max(emax, kMinE);
  if (!in) return;
  if (g == 0) p.scale[j * p.nkb + kb] = block_scale(emax, E, 24);
  const int mp = (int)min((int64_t)m0 + kBlockK, p.kp);  // the padded end of this block
  for (int m = m0 + 16 * g; m < mp; m += 64) {
    uint64_t f[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const double x = (m + i < m1 && emax != 2047) ? __ldg(p.src + (int64_t)(m + i) * p.ld + j) : 0.0;
      f[i] = digit_fields(x, E);
    }
    __half* out = p.out + j * p.kp + m;
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
  int64_t ldo, split_stride;
  int accumulate;
  int* err;
  // Budget of every wait in SM clock cycles.  Test hook (kpm_table_test_timeout): kWithholdStage arms the
  // first stage and issues no copy for it; an epilogue warp's index makes that warp's first wait run out.
  long long wait_budget;
  int test;
};
enum { kNoTest = -1, kWithholdStage = -2 };

__global__ void __launch_bounds__(kThreads, 1)
    digit_gemm_kernel(const DigitGemm p, const __grid_constant__ CUtensorMap map_a,
                      const __grid_constant__ CUtensorMap map_b) {
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
  __shared__ __align__(8) uint64_t full[kStages], empty[kStages], tfull, tfree;
  __shared__ uint32_t tmem_slot;
  __shared__ double ssb[kTN];
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
  auto stages_of = [&](int kb) { return (min(p.kp, (kb + 1) * kBlockK) - kb * kBlockK) / kStageK; };

  if (warp == kEpiWarps) {  // producer
    if (lane == 0) {
      int issued = 0;
      bool ok = true;
      for (int kb = kb0; kb < kb1 && ok; ++kb)
        for (int ks = 0; ks < stages_of(kb) && ok; ++ks) {
          const int st = issued % kStages;
          if (issued >= kStages) ok = mbar_wait_bounded(&empty[st], (uint32_t)((issued / kStages - 1) & 1), p.wait_budget);
          if (!ok) break;
          mbar_arrive_expect_tx(&full[st], kStage);
          unsigned char* a = smem + (size_t)st * kStage;
          unsigned char* b = a + kDigits * kPlaneA;
          const int k = kb * kBlockK + ks * kStageK;
          const bool withhold = p.test == kWithholdStage && issued == 0;
          for (int s = 0; s < kDigits && !withhold; ++s) {
            tma_load_3d(a + s * kPlaneA, &map_a, k, row0, s, &full[st]);
            tma_load_3d(b + s * kPlaneB, &map_b, k, col0, s, &full[st]);
          }
          ++issued;
        }
      if (!ok) atomicExch(p.err, KPM_ERR_TIMEOUT);
      for (int q = max(0, issued - kStages); q < issued; ++q)  // nothing is in flight when the CTA leaves
        (void)mbar_wait_bounded(&full[q % kStages], (uint32_t)((q / kStages) & 1), p.wait_budget);
    }
  } else if (warp == kEpiWarps + 1) {  // MMA issuer
    if (lane == 0) {
      const uint32_t idesc = idesc_f16(kTM, kTN);
      const uint32_t base = smem_addr(smem);
      int it = 0, done = 0;
      bool ok = true;
      for (int kb = kb0; kb < kb1 && ok; ++kb) {
        if (kb > kb0) ok = mbar_wait_bounded(&tfree, (uint32_t)((kb - kb0 - 1) & 1), p.wait_budget);
        tc_fence_after();
        const int ns = stages_of(kb);
        for (int ks = 0; ks < ns && ok; ++ks, ++it) {
          const int st = it % kStages;
          ok = mbar_wait_bounded(&full[st], (uint32_t)((it / kStages) & 1), p.wait_budget);
          if (!ok) break;
          tc_fence_after();
          const uint32_t a0 = base + (uint32_t)st * kStage, b0 = a0 + kDigits * kPlaneA;
#pragma unroll 1
          for (int j = 0; j < kStageK / 16; ++j)
#pragma unroll
            for (int s = 0; s < kDigits; ++s)
#pragma unroll
              for (int t = 0; t < kDigits - s; ++t)
                mma_f16(tmem + (uint32_t)((s + t) * kTN),
                        smem_desc(a0 + s * kPlaneA + j * 32, 16, 512) | ((uint64_t)4 << 61),
                        smem_desc(b0 + t * kPlaneB + j * 32, 16, 512) | ((uint64_t)4 << 61), idesc,
                        s > 0 || j > 0 || ks > 0);
          mma_commit(&empty[st]);
          ++done;
        }
        if (ok) mma_commit(&tfull);
      }
      if (!ok) atomicExch(p.err, KPM_ERR_TIMEOUT);
      // every MMA issued is finished before the accumulators are released, also when the epilogue left early
      if (done > 0)
        (void)mbar_wait_bounded(&empty[(done - 1) % kStages], (uint32_t)(((done - 1) / kStages) & 1), p.wait_budget);
    }
  } else {  // epilogue: thread = output row 32 q + lane, half of the columns
    const int q = warp & 3, cb = (warp >> 2) * kEpiCols;
    const int row = row0 + 32 * q + lane;
    const int srow = min(row, p.rows_a - 1);
    double acc[kEpiCols];
#pragma unroll
    for (int c = 0; c < kEpiCols; ++c) acc[c] = 0.0;
    // One warp's wait may run out while another's completes in time.  The outcome is shared at the
    // barrier that ends the block, so that all warps leave the loop together: a warp that went on
    // alone would wait at the next barrier for ever.
    bool dead = false;
    for (int kb = kb0; kb < kb1 && !dead; ++kb) {
      // a block of 2^l products has joined sums below 2^(61 + l) (1 + 2^-5): the l - 1 bits that do
      // not fit 63 are rounded off (the pairs left out are worth more than that)
      const int len = min(p.kp, (kb + 1) * kBlockK) - kb * kBlockK;  // 32 .. 512
      const int sh = 31 - __clz(len - 1);                            // ceil(log2 len) - 1
      const double sa = __ldg(p.sa + (int64_t)srow * p.nkb + kb) * __longlong_as_double((long long)(1011 + sh) << 52);
      if (threadIdx.x < kTN) ssb[threadIdx.x] = __ldg(p.sb + (int64_t)min(col0 + (int)threadIdx.x, p.rows_b - 1) * p.nkb + kb);
      named_sync(32 * kEpiWarps);
      bool ok = mbar_wait_bounded(&tfull, (uint32_t)((kb - kb0) & 1), p.wait_budget);
      ok = __all_sync(0xffffffffu, ok && p.test != warp);
      if (!ok && lane == 0) {
        atomicExch(p.err, KPM_ERR_TIMEOUT);
        *static_cast<volatile int*>(&dead_flag) = 1;
      }
      if (ok) {
        tc_fence_after();
        const uint32_t t0 = tmem + ((uint32_t)(32 * q) << 16) + (uint32_t)cb;
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
              hi = hi * 128 + __float2int_rn(__uint_as_float(r[d][c]));
              lo = lo * 128 + __float2int_rn(__uint_as_float(r[4 + d][c]));
            }
            const double D = (double)(hi * (1ll << (28 - sh)) + ((lo + (1ll << (sh - 1))) >> sh));  // joined / 2^sh
            acc[8 * g + c] = fma(D * sa, ssb[cb + 8 * g + c], acc[8 * g + c]);
          }
        }
        tc_fence_before();
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(&tfree);
      named_sync(32 * kEpiWarps);  // ssb is rewritten for the next block
      dead = *static_cast<volatile int*>(&dead_flag) != 0;  // the next write to it lies behind the next block's barrier
    }
    if (!dead && row < p.rows_a) {
      double* out = p.out + (int64_t)blockIdx.y * p.split_stride + (int64_t)row * p.ldo + col0 + cb;
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
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

// mu[n][m] = (accumulate ? mu : 0) + sum over splits, Re from rows n, Im from rows M + n.
__global__ void gram_reduce_kernel(const double* __restrict__ part, int splits, int M, int ldo, int accumulate,
                                   double2* __restrict__ mu) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= M * M) return;
  const int n = idx / M, m = idx % M;
  double re = 0.0, im = 0.0;
  for (int s = 0; s < splits; ++s) {
    const double* q = part + (int64_t)s * 2 * M * ldo;
    re += q[(int64_t)n * ldo + m];
    im += q[(int64_t)(M + n) * ldo + m];
  }
  double2 o = make_double2(re, im);
  if (accumulate) {
    o.x += mu[idx].x;
    o.y += mu[idx].y;
  }
  mu[idx] = o;
}

// Planes [kDigits][rows][k] of fp16 as a 3-D map; a box is one plane's 32 x box_rows piece in the
// 64-byte-swizzled layout.  Rows past the end read as zero digits.
bool plane_map(CUtensorMap* m, const __half* base, int64_t k, int64_t rows, int box_rows) {
  const EncodeTiledFn enc = encode_tiled();
  if (!enc) return false;
  const cuuint64_t dims[3] = {(cuuint64_t)k, (cuuint64_t)rows, (cuuint64_t)kDigits};
  const cuuint64_t strides[2] = {(cuuint64_t)k * 2, (cuuint64_t)(k * rows) * 2};
  const cuuint32_t box[3] = {(cuuint32_t)kStageK, (cuuint32_t)box_rows, 1};
  const cuuint32_t estr[3] = {1, 1, 1};
  return enc(m, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 3, const_cast<__half*>(base), dims, strides, box, estr,
             CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

int64_t round_up(int64_t x, int64_t m) { return (x + m - 1) / m * m; }

int gemm_attr() {
  static const cudaError_t e =
      cudaFuncSetAttribute(digit_gemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmem);
  return check_cuda(e);
}

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

struct GramPlan {
  int64_t kc;  // columns (reals) of a chunk
  int nkb, mt, nt, splits, ldo;
  int64_t plane_a, plane_b;
  size_t pa, pb, sa, sb, part, bytes;
};

GramPlan gram_plan(const kpm_ell_s* h, int M) {
  GramPlan g{};
  const int64_t K = 2 * h->n;  // reals of a table row
  // chunk of K: planes of U, its swapped form and W
  g.kc = kPlaneBytes / (kDigits * 3 * 2 * (int64_t)M) / kBlockK * kBlockK;
  g.kc = std::max<int64_t>(4 * kBlockK, std::min<int64_t>(g.kc, 65536));
  g.kc = std::min(g.kc, round_up(K, kStageK));
  g.nkb = (int)((g.kc + kBlockK - 1) / kBlockK);
  g.mt = (2 * M + kTM - 1) / kTM;
  g.nt = (M + kTN - 1) / kTN;
  g.splits = std::max(1, std::min(g.nkb, h->sm_count / (g.mt * g.nt)));
  g.ldo = (int)round_up(M, 2);
  g.plane_a = 2 * (int64_t)M * g.kc;
  g.plane_b = (int64_t)M * g.kc;
  WorkLayout w;
  g.pa = w.take((size_t)kDigits * g.plane_a * sizeof(__half));
  g.pb = w.take((size_t)kDigits * g.plane_b * sizeof(__half));
  g.sa = w.take((size_t)2 * M * g.nkb * sizeof(double));
  g.sb = w.take((size_t)M * g.nkb * sizeof(double));
  g.part = w.take((size_t)g.splits * 2 * M * g.ldo * sizeof(double));
  g.bytes = w.bytes;
  return g;
}

struct MixPlan {
  int64_t kp, nc;  // padded K; columns (reals) of a chunk
  int nkb, mt;
  int64_t plane_a, plane_b;
  size_t pa, pb, cpad, sa, sb, bytes;
};

MixPlan mix_plan(const kpm_ell_s* h, int M) {
  MixPlan g{};
  g.kp = round_up(M, 64);
  g.nkb = (int)((g.kp + kBlockK - 1) / kBlockK);
  g.mt = (M + kTM - 1) / kTM;
  // chunk of columns: whole waves of one CTA per SM, planes within the L2 budget
  const int64_t wave = std::max<int64_t>(1, h->sm_count / g.mt) * kTN;
  g.nc = std::max<int64_t>(1, kPlaneBytes / (kDigits * 2 * g.kp) / wave) * wave;
  g.nc = std::min(g.nc, round_up(2 * h->n, kTN));
  g.plane_a = (int64_t)M * g.kp;
  g.plane_b = g.nc * g.kp;
  WorkLayout w;
  g.pb = w.take((size_t)kDigits * g.plane_b * sizeof(__half));
  g.pa = w.take((size_t)kDigits * g.plane_a * sizeof(__half));
  g.cpad = w.take((size_t)M * g.kp * sizeof(double));
  g.sa = w.take((size_t)M * g.nkb * sizeof(double));
  g.sb = w.take((size_t)g.nc * g.nkb * sizeof(double));
  g.bytes = w.bytes;
  return g;
}

template <typename T>
T* at(void* work, size_t offset) {
  return reinterpret_cast<T*>(static_cast<char*>(work) + offset);
}

int gram(kpm_ell_s* h, int M, const double* U, const double* W, int accumulate, double* mu, void* work, cudaStream_t s) {
  KPM_TRY(gemm_attr());
  const GramPlan t = gram_plan(h, M);
  const int64_t K = 2 * h->n;
  __half *pa = at<__half>(work, t.pa), *pb = at<__half>(work, t.pb);
  double *sa = at<double>(work, t.sa), *sb = at<double>(work, t.sb), *part = at<double>(work, t.part);
  CUtensorMap ma, mb;
  if (!plane_map(&ma, pa, t.kc, 2 * M, kTM) || !plane_map(&mb, pb, t.kc, M, kTN)) return KPM_ERR_UNSUPPORTED;
  for (int64_t k0 = 0; k0 < K; k0 += t.kc) {
    const int64_t kv = std::min(t.kc, K - k0), kp = round_up(kv, kStageK);
    SliceRows a{};
    a.src = U;
    a.ld = K;
    a.k0 = k0;
    a.kvalid = kv;
    a.rows = M;
    a.nkb = t.nkb;
    a.plane = t.plane_a;
    a.kc = t.kc;
    a.out = pa;
    a.swap_off = t.plane_b;
    a.scale = sa;
    a.scale_swap = M * t.nkb;
    a.shift = 23;
    SliceRows b = a;
    b.src = W;
    b.plane = t.plane_b;
    b.out = pb;
    b.swap_off = 0;
    b.scale = sb;
    b.scale_swap = 0;
    b.shift = 24;
    launch_slice_rows(a, s);
    launch_slice_rows(b, s);
    DigitGemm g{};
    g.rows_a = 2 * M;
    g.rows_b = M;
    g.mt = t.mt;
    g.nkb = t.nkb;
    g.blocks = (int)((kp + kBlockK - 1) / kBlockK);
    g.kp = (int)kp;
    g.sa = sa;
    g.sb = sb;
    g.out = part;
    g.ldo = t.ldo;
    g.split_stride = 2 * (int64_t)M * t.ldo;
    g.accumulate = k0 > 0;
    g.err = h->err_flag;
    g.wait_budget = kWaitBudgetCycles;
    g.test = kNoTest;
    digit_gemm_kernel<<<dim3(t.mt * t.nt, t.splits), kThreads, kSmem, s>>>(g, ma, mb);
    KPM_CUDA_TRY(cudaGetLastError());
  }
  gram_reduce_kernel<<<(M * M + 255) / 256, 256, 0, s>>>(part, t.splits, M, t.ldo, accumulate ? 1 : 0,
                                                         reinterpret_cast<double2*>(mu));
  return check_cuda(cudaGetLastError());
}

int mix(kpm_ell_s* h, int M, const double* C, const double* T, double* Q, void* work, cudaStream_t s) {
  KPM_TRY(gemm_attr());
  const MixPlan t = mix_plan(h, M);
  const int64_t cols = 2 * h->n;
  __half *pa = at<__half>(work, t.pa), *pb = at<__half>(work, t.pb);
  double *cpad = at<double>(work, t.cpad), *sa = at<double>(work, t.sa), *sb = at<double>(work, t.sb);
  CUtensorMap ma, mb;
  if (!plane_map(&ma, pa, t.kp, M, kTM) || !plane_map(&mb, pb, t.kp, t.nc, kTN)) return KPM_ERR_UNSUPPORTED;
  // C's rows: an odd M would leave them 8-byte aligned, so they are copied to an even pitch
  const double* csrc = C;
  int64_t cld = M;
  if ((M & 1) || (reinterpret_cast<uintptr_t>(C) & 15)) {
    KPM_CUDA_TRY(cudaMemcpy2DAsync(cpad, (size_t)t.kp * sizeof(double), C, (size_t)M * sizeof(double),
                                   (size_t)M * sizeof(double), M, cudaMemcpyDeviceToDevice, s));
    csrc = cpad;
    cld = t.kp;
  }
  SliceRows a{};
  a.src = csrc;
  a.ld = cld;
  a.kvalid = M;
  a.rows = M;
  a.nkb = t.nkb;
  a.plane = t.plane_a;
  a.kc = t.kp;
  a.out = pa;
  a.scale = sa;
  a.shift = 23;
  launch_slice_rows(a, s);
  for (int64_t j0 = 0; j0 < cols; j0 += t.nc) {
    const int64_t c = std::min(t.nc, cols - j0);
    SliceCols b{};
    b.src = T + j0;
    b.ld = cols;
    b.M = M;
    b.nkb = t.nkb;
    b.cols = c;
    b.plane = t.plane_b;
    b.kp = t.kp;
    b.out = pb;
    b.scale = sb;
    slice_cols_kernel<<<dim3((unsigned)((c + 63) / 64), t.nkb), 256, 0, s>>>(b);
    DigitGemm g{};
    g.rows_a = M;
    g.rows_b = (int)c;
    g.mt = t.mt;
    g.nkb = t.nkb;
    g.blocks = (int)((t.kp + kBlockK - 1) / kBlockK);
    g.kp = (int)t.kp;
    g.sa = sa;
    g.sb = sb;
    g.out = Q + j0;
    g.ldo = cols;
    g.err = h->err_flag;
    g.wait_budget = kWaitBudgetCycles;
    g.test = kNoTest;
    digit_gemm_kernel<<<dim3((unsigned)(t.mt * ((c + kTN - 1) / kTN)), 1), kThreads, kSmem, s>>>(g, ma, mb);
    KPM_CUDA_TRY(cudaGetLastError());
  }
  return KPM_OK;
}

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
  if (!h || M < 1 || M > 16384) return 0;
  return (int64_t)std::max(gram_plan(h, M).bytes, mix_plan(h, M).bytes);
}

int kpm_table_gram_work(kpm_ell* h, int M, const double* U, const double* W, int accumulate, double* mu, void* work,
                        int64_t work_bytes, void* stream) {
  if (!h || !U || !W || !mu || !work || M < 1 || misaligned(U, W)) return KPM_ERR_INVALID_ARG;
  if (M > 16384) return KPM_ERR_UNSUPPORTED;
  if (work_bytes < kpm_table_work_bytes(h, M) || reinterpret_cast<uintptr_t>(work) % kWorkAlign) return KPM_ERR_INVALID_ARG;
  return gram(h, M, U, W, accumulate, mu, work, reinterpret_cast<cudaStream_t>(stream));
}

int kpm_table_gram(kpm_ell* h, int M, const double* U, const double* W, int accumulate, double* mu, void* stream) {
  if (!h || !U || !W || !mu || M < 1 || misaligned(U, W)) return KPM_ERR_INVALID_ARG;
  if (M > 16384) return KPM_ERR_UNSUPPORTED;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  return with_work(h, M, s, [&](void* work) { return gram(h, M, U, W, accumulate, mu, work, s); });
}

int kpm_table_mix_work(kpm_ell* h, int M, const double* C, const double* T, double* Q, void* work, int64_t work_bytes,
                       void* stream) {
  if (!h || !C || !T || !Q || !work || M < 1 || misaligned(T, Q)) return KPM_ERR_INVALID_ARG;
  if (M > 16384) return KPM_ERR_UNSUPPORTED;
  if (work_bytes < kpm_table_work_bytes(h, M) || reinterpret_cast<uintptr_t>(work) % kWorkAlign) return KPM_ERR_INVALID_ARG;
  return mix(h, M, C, T, Q, work, reinterpret_cast<cudaStream_t>(stream));
}

int kpm_table_mix(kpm_ell* h, int M, const double* C, const double* T, double* Q, void* stream) {
  if (!h || !C || !T || !Q || M < 1 || misaligned(T, Q)) return KPM_ERR_INVALID_ARG;
  if (M > 16384) return KPM_ERR_UNSUPPORTED;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  return with_work(h, M, s, [&](void* work) { return mix(h, M, C, T, Q, work, s); });
}

int kpm_table_test_timeout(kpm_ell* h, int64_t budget_cycles, int warp, void* stream) {
  if (!h || budget_cycles < 1000 || budget_cycles > kWaitBudgetCycles || warp >= kEpiWarps) return KPM_ERR_INVALID_ARG;
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  KPM_TRY(gemm_attr());
  // one tile of zeros, four blocks of K
  const int64_t k = 4 * kBlockK;
  const size_t planes = (size_t)kDigits * (kTM + kTN) * k * sizeof(__half);
  const size_t scales = (size_t)(kTM + kTN) * 4 * sizeof(double), out = (size_t)kTM * kTN * sizeof(double);
  DevBuf scratch;
  KPM_TRY(ensure(scratch, planes + scales + out));
  KPM_CUDA_TRY(cudaMemsetAsync(scratch.p, 0, planes + scales + out, s));
  KPM_CUDA_TRY(cudaMemsetAsync(h->err_flag, 0, sizeof(int), s));
  __half* pa = static_cast<__half*>(scratch.p);
  __half* pb = pa + (size_t)kDigits * kTM * k;
  double* sa = reinterpret_cast<double*>(pb + (size_t)kDigits * kTN * k);
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
