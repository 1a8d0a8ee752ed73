// kpm_resident.cu -- a whole moment recursion of a small operator as one cooperative launch.
//
// An operator whose rows fit the SMs' shared memory runs M orders of
//   T_0 = v,  T_1 = H T_0,  T_m = 2H T_{m-1} - T_{m-2},  mu_m = <v_l | T_m>
// without leaving the chip: every CTA keeps its rows' columns and values, its entries of the last
// two T, and its entries of the left vectors in shared memory for the whole recursion.  Only T_m
// itself is exchanged, through two vector sets in L2 that the neighbour gathers read.
//
// As step launches such a recursion is bound by latency: launch, column -> gather chain, moment
// reduction, one after the other (4.4 us an order at 8,192 sites and 4 vectors, of which the
// arithmetic is 0.4).  Here an order costs the gathers, the row's FMAs and one grid-wide
// exchange; everything else is off that path:
//   * kCompute threads advance the rows; kMoment threads form the moments of the order just
//     finished from shared memory while the others wait for the exchange and gather the next.
//   * the exchange has no counter: every CTA publishes the order it has finished in a word of
//     its own, and its threads poll one word each of the CTAs that it gathers from or that gather
//     from it (of all of them once, at the start).
// An order takes 2.0 us at a thousand sites and 2.6 at 8,192 sites and 4 vectors (4.4 us before).
//
// The recursion's arithmetic is that of the step kernels (bit-identical T_m); moments are FP64
// products for complex128, and for complex64 float products of one row, added in FP64.
// Sums are in a fixed order: repeated calls are bit-identical.
//
// Every wait on another CTA is bounded by clock cycles; one that runs out records
// KPM_ERR_TIMEOUT, and the CTA then runs its barriers to the end without computing; its moments become NaN.
#include <algorithm>

#include "kpm_cheb.cuh"

namespace kpm {
namespace {

constexpr int kCompute = 512, kMoment = 128;
constexpr int kResThreads = kCompute + kMoment;

constexpr int kMaxGrid = 256, kMaskWords = kMaxGrid / 32;
// Published orders lie a cache line apart: words of several CTAs in one line cost 2.4-2.9 us an
// exchange between 152 CTAs, 1.1 us like this (a counter that all CTAs add to: 1.2-1.3).
constexpr int kFlagStride = 32;
constexpr size_t kFlagInts = (size_t)kMaxGrid * (kFlagStride + kMaskWords);  // published orders, then masks

constexpr size_t kMaxSmem = 216 * 1024;
// Items (rows x vectors) of a CTA.  At least kMinItems: fewer, larger CTAs have fewer peers to wait
// for, and a few dozen items do not fill one (24 x 22 cells, us per 256 orders: 16 items 531, 64
// 512-547, 256 596).  At most: complex128 orders are bound by the FP64 pipe, where the step
// kernels' float-float products win from 3,300 items on (us per 256 orders, resident against
// steps: 8,192 sites R = 4 667 : 1112; 104k R = 1 1049 : 2230; 131k R = 4 (3,450 items) 3981 : 4360;
// 65k R = 8 (3,450) 3938 : 3927; 77k R = 8 (4,042) 4694 : 4298).  complex64 (8,192
// sites R = 4 505 : 1299): the step kernels add two to eight rows of a thread in float, this form
// every row in FP64, so its moments differ from theirs by about 1e-9 of their norm (also below the limit,
// where KPM_STEP_KERNEL or profiling asks for the steps).  Up to 80,000 items the steps that timings
// used to pick gave each thread one row and so the same sums; larger operators keep the steps' sums.
constexpr int64_t kMinItems = 64, kMaxItems64 = 3500, kMaxTotal32 = 80000;

struct Resident {
  const void* val;  // 2H values [L][ld]
  const int32_t* col;
  int64_t ld, n;
  int L, rows, M;      // rows of one CTA
  const double2* v_r;  // [R][n] of this group
  const double2* v_l;  // null: v_r
  int both;            // a second moment set <v_r | T_m>
  void* ta;            // two vector sets [n][R]
  void* tb;
  int* flags;          // [kMaxGrid][kFlagStride] orders finished (zero at launch), then [grid][kMaskWords]
  double2* part;       // [M][sets][grid][R]
  int* err;
  // limit of every wait in SM clock cycles; test hook (kpm_ell_test_withhold): from this order on CTA 0
  // publishes nothing (-1: it does)
  long long wait_budget;
  int withhold;
};

__device__ __forceinline__ void bar_sync(int id, int threads) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int threads) {
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(threads) : "memory");
}
__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int* p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}

__device__ __forceinline__ int* order_word(int* flags, int cta) { return flags + cta * kFlagStride; }

__device__ __forceinline__ bool withheld(int order, int m) { return order >= 0 && m >= order && blockIdx.x == 0; }

// Wait (bounded) until CTA `cta` has published order m; a wait that runs out sets *dead.
__device__ __forceinline__ void await_order(int* flags, int cta, int m, int* dead, int* err, long long budget) {
  const int* f = order_word(flags, cta);
  if (ld_acquire(f) > m) return;
  const long long t0 = clock64();
  while (ld_acquire(f) <= m)
    if (clock64() - t0 > budget) {
      atomicExch(err, KPM_ERR_TIMEOUT);
      *dead = 1;
      return;
    }
}

// Shared memory of one CTA, in this order: values, T (even), T (odd), left vectors, second left
// vectors, columns.
template <typename T, bool REAL>
__host__ __device__ constexpr size_t resident_smem(int L, int rows, int R, bool left2) {
  using MV = typename MatV<T, REAL>::type;
  using Raw = typename RawT<T, 1>::type;
  return (((size_t)L * rows * sizeof(MV) + 15) & ~(size_t)15) + (size_t)(left2 ? 4 : 3) * rows * R * sizeof(Raw) +
         (size_t)L * rows * sizeof(int32_t);
}

enum { kBarCompute = 1, kBarReady = 2, kBarFree = 4, kBarMoment = 6 };

template <typename T, bool REAL, int R>
__global__ void __launch_bounds__(kResThreads, 1) resident_kernel(const Resident p) {
  using Raw = typename RawT<T, 1>::type;
  using MV = typename MatV<T, REAL>::type;
  constexpr bool F32 = std::is_same<T, float>::value;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ double2 red[2][2][kMoment / 32][R];
  __shared__ int dead_flag;
  __shared__ unsigned need[kMaskWords];  // CTAs this one gathers from
  __shared__ int peer[kMaxGrid];         // CTAs it waits for: those, and those that gather from it
  __shared__ int npeers;

  const int L = p.L, rows = p.rows;
  const int64_t row0 = (int64_t)blockIdx.x * rows;
  const int mine = (int)max((int64_t)0, min((int64_t)rows, p.n - row0));
  const int items = mine * R;
  const int tid = threadIdx.x;
  const bool two = p.both != 0;
  MV* sval = reinterpret_cast<MV*>(smem);
  Raw* const sT0 = reinterpret_cast<Raw*>(smem + (((size_t)L * rows * sizeof(MV) + 15) & ~(size_t)15));
  auto sT = [&](int b) { return sT0 + b * rows * R; };
  Raw* sl = sT0 + 2 * rows * R;
  Raw* sl2 = two ? sl + rows * R : sl;
  int32_t* scol = reinterpret_cast<int32_t*>(sl2 + rows * R);
  if (tid == 0) dead_flag = npeers = 0;
  if (tid < kMaskWords) need[tid] = 0;
  __syncthreads();
  for (int e = tid; e < L * mine; e += kResThreads) {
    const int s = e / mine, r = e - s * mine;
    sval[s * rows + r] = static_cast<const MV*>(p.val)[(int64_t)s * p.ld + row0 + r];
    const int c = p.col[(int64_t)s * p.ld + row0 + r];
    const int o = c / rows;
    scol[s * rows + r] = c;
    if (!(need[o >> 5] >> (o & 31) & 1u)) atomicOr(&need[o >> 5], 1u << (o & 31));
  }
  auto buf = [&](int b) { return static_cast<Raw*>(b ? p.tb : p.ta); };
  auto load = [&](const double2* v, int it) {
    const double2 z = v[(int64_t)(it % R) * p.n + row0 + it / R];
    Cx<T, 1> c;
    c.re[0] = (T)z.x;
    c.im[0] = (T)z.y;
    return pack(c);
  };
  for (int it = tid; it < items; it += kResThreads) {
    const Raw z = load(p.v_r, it);
    sT0[it] = z;
    buf(0)[row0 * R + it] = z;
    sl[it] = p.v_l ? load(p.v_l, it) : z;
    if (two) sl2[it] = z;
  }
  __syncthreads();
  unsigned* masks = reinterpret_cast<unsigned*>(p.flags + kMaxGrid * kFlagStride);
  if (tid < kMaskWords) masks[blockIdx.x * kMaskWords + tid] = need[tid];

  if (tid < kCompute) {
    bool dead = false;
    // publish order m and wait until the peers (or all CTAs) have published it
    auto exchange = [&](int m, bool all) {
      bar_sync(kBarCompute, kCompute);  // T_m is written, the peer list complete
      if (tid == 0 && !withheld(p.withhold, m)) st_release(order_word(p.flags, blockIdx.x), m + 1);
      const int count = all ? (int)gridDim.x : npeers;
      if (tid < count) await_order(p.flags, all ? tid : peer[tid], m, &dead_flag, p.err, p.wait_budget);
      bar_sync(kBarCompute, kCompute);
      dead = *static_cast<volatile int*>(&dead_flag) != 0;
    };
    bar_arrive(kBarReady, kResThreads);
    if (p.M > 1) {
      exchange(0, true);
      // whom to wait for from now on.  A CTA may overwrite T_{m-2} with T_m when those that gather
      // from it have finished order m - 1, so both directions count.
      if (tid < (int)gridDim.x && tid != (int)blockIdx.x) {
        const unsigned theirs = __ldcg(masks + tid * kMaskWords + (blockIdx.x >> 5)) >> (blockIdx.x & 31);
        if (((need[tid >> 5] >> (tid & 31)) | theirs) & 1u) peer[atomicAdd(&npeers, 1)] = tid;
      }
    }
    for (int m = 1; m < p.M; ++m) {
      const int b = m & 1;
      if (m >= 2) bar_sync(kBarFree + b, kResThreads);  // T_{m-2}'s moments are done
      if (!dead) {
        const Raw* src = buf(b ^ 1);
        Raw* st = sT(b);
        Raw* dst = buf(b) + row0 * R;
        auto gather = [&](int it, int s, Cx<T, 1> (&x)[4]) {
          const int r = it / R, sub = it % R;
#pragma unroll
          for (int u = 0; u < 4; ++u)
            if (s + u < L) unpack(__ldcg(src + (int64_t)scol[(s + u) * rows + r] * R + sub), x[u]);
        };
        auto row = [&](int it, Cx<T, 1> (&x)[4]) {  // x: the first four slots' entries
          const int r = it / R;
          typename AccOf<T, 1>::type acc;
          Cx<T, 1> old;
          unpack(st[it], old);
          for (int s = 0; s < L; s += 4) {
            if (s > 0) gather(it, s, x);
            if (s == 0) {
              if (m == 1)
                mul_first(acc, sval[r], x[0]);
              else
                madd_first_neg(acc, sval[r], x[0], old);
            } else {
              madd(acc, sval[s * rows + r], x[0]);
            }
#pragma unroll
            for (int u = 1; u < 4; ++u)
              if (s + u < L) madd(acc, sval[(s + u) * rows + r], x[u]);
          }
          Cx<T, 1> t = finish(acc);
          if (m == 1) {
            t.re[0] *= T(0.5);
            t.im[0] *= T(0.5);
          }
          const Raw z = pack(t);
          st[it] = z;
          __stcg(dst + it, z);
        };
        Cx<T, 1> x[4];
        if constexpr (F32) {
          for (int it = tid; it < items; it += kCompute) {
            gather(it, 0, x);
            row(it, x);
          }
        } else {
          // FP64: the next item's gathers are in flight while this one's row is computed (the warps
          // run in step, so without it the FMA pipe idles for every gather: 10 % of an order at
          // 2,000 items a CTA).  Float rows are short and lose to the longer loop.
          Cx<T, 1> y[4];
          if (tid < items) gather(tid, 0, x);
          for (int it = tid; it < items; it += 2 * kCompute) {
            if (it + kCompute < items) gather(it + kCompute, 0, y);
            row(it, x);
            if (it + 2 * kCompute < items) gather(it + 2 * kCompute, 0, x);
            if (it + kCompute < items) row(it + kCompute, y);
          }
        }
      }
      bar_arrive(kBarReady + b, kResThreads);
      if (m + 1 < p.M && !dead) exchange(m, false);
    }
  } else {
    const int t = tid - kCompute, warp = t >> 5, lane = t & 31;
    const int sets = two ? 2 : 1;
    for (int m = 0; m < p.M; ++m) {
      const int b = m & 1;
      bar_sync(kBarReady + b, kResThreads);
      const Raw* st = sT(b);
      double re[2] = {0.0, 0.0}, im[2] = {0.0, 0.0};
      auto dot = [&](int k, const Raw* left, const Cx<T, 1>& x, int it) {
        Cx<T, 1> l;
        unpack(left[it], l);
        if constexpr (F32) {
          T fr = T(0), fi = T(0);
          cdot_acc(fr, fi, l.re[0], l.im[0], x.re[0], x.im[0]);
          re[k] += (double)fr;
          im[k] += (double)fi;
        } else {
          cdot_acc(re[k], im[k], l.re[0], l.im[0], x.re[0], x.im[0]);
        }
      };
      for (int it = t; it < items; it += kMoment) {  // kMoment is a multiple of R: one vector per thread
        Cx<T, 1> x;
        unpack(st[it], x);
        dot(0, sl, x, it);
        if (two) dot(1, sl2, x, it);
      }
      if (m + 2 < p.M) bar_arrive(kBarFree + b, kResThreads);
      for (int k = 0; k < sets; ++k) {
#pragma unroll
        for (int off = R; off < 32; off <<= 1) {
          re[k] += __shfl_xor_sync(0xffffffffu, re[k], off);
          im[k] += __shfl_xor_sync(0xffffffffu, im[k], off);
        }
        if (lane < R) red[b][k][warp][lane] = make_double2(re[k], im[k]);
      }
      bar_sync(kBarMoment, kMoment);  // red is double buffered: the next order's writes go to the other half
      if (t < sets * R) {
        const int k = t / R, sub = t % R;
        double2 s = make_double2(0.0, 0.0);
#pragma unroll
        for (int w = 0; w < kMoment / 32; ++w) {
          s.x += red[b][k][w][sub].x;
          s.y += red[b][k][w][sub].y;
        }
        if (*static_cast<volatile int*>(&dead_flag) != 0)  // no moment is made of what was left in shared memory
          s = make_double2(__longlong_as_double(0x7ff8000000000000ll), __longlong_as_double(0x7ff8000000000000ll));
        p.part[(((int64_t)m * sets + k) * gridDim.x + blockIdx.x) * R + sub] = s;
      }
    }
  }
}

// ---- vector tables (kpm_cheb_table, kpm_cheb_clenshaw_table) of one vector --------------------
// The same scheme with every order kept: row m of the table is both the result and what the next
// order gathers, so nothing is overwritten and a CTA waits only for those it reads from.  The second
// operator's product needs no exchange of its own: S T_{m-1} follows the publication of T_m, and
// S z_k is formed before the wait for lambda_{k+1}, both in the time the exchange takes.  As
// launches an order of 131,072 rows and four slots cost 8.2 us (table) and 12.3 us (with S, or Clenshaw),
// here 4.4 and 6.3-7.2 (imaginary S; complex 8.0-9.0), against 2.6 and 4.7 of FP64 products (imaginary S).
//
// A CTA whose S values are all imaginary (V = -i H o dx of a real H) multiplies by the imaginary part
// alone, half the FMAs; a row that comes out infinite or NaN is formed again with the zero parts.
// The arithmetic is table_step_kernel's otherwise, operation for operation.
struct ResidentTable {
  const void* vh;
  const int32_t* ch;
  int Lh;
  const void* vs;  // null: no second operator (the sources z are added as they are)
  const int32_t* cs;
  int Ls;
  int64_t ld, n;
  int rows, M;
  const double2* z;  // Clenshaw: the sources
  double2* tab;      // T rows, or lambda rows
  double2* stab;     // table: S T rows
  int* flags;
  int* err;
  long long wait_budget;  // as in Resident
  int withhold;
};

static_assert(kTableFlagInts >= (size_t)(1 + kMaxGrid) * kFlagStride, "");
constexpr int kTabItems = 3;  // rows of a thread, at most
constexpr int64_t kMaxTabRows = (int64_t)kTabItems * kCompute;

// Shared memory of one CTA: its entries of the last two rows, S values, H values, columns of H and S.
template <bool RS>
__host__ __device__ constexpr size_t table_hval(int Ls, int rows) {  // real S values may end off a 16-byte line
  return (size_t)rows * 2 * sizeof(double2) +
         (((size_t)Ls * rows * sizeof(typename MatV<double, RS>::type) + 15) & ~(size_t)15);
}
template <bool RH, bool RS>
__host__ __device__ constexpr size_t table_smem(int Lh, int Ls, int rows) {
  return table_hval<RS>(Ls, rows) + (size_t)rows * (Lh * (sizeof(typename MatV<double, RH>::type) + 4) + Ls * 4);
}

__device__ __forceinline__ void table_fma(double2& acc, double h, double2 x) {
  acc.x = fma(h, x.x, acc.x);
  acc.y = fma(h, x.y, acc.y);
}
__device__ __forceinline__ void table_fma(double2& acc, double2 h, double2 x) {
  acc.x = fma(h.x, x.x, fma(-h.y, x.y, acc.x));
  acc.y = fma(h.x, x.y, fma(h.y, x.x, acc.y));
}
__device__ __forceinline__ bool table_finite(double2 a) {
  return (__double2hiint(a.x) & 0x7ff00000) != 0x7ff00000 && (__double2hiint(a.y) & 0x7ff00000) != 0x7ff00000;
}
// acc += i h x
__device__ __forceinline__ void table_fma_imag(double2& acc, double h, double2 x) {
  acc.x = fma(-h, x.y, acc.x);
  acc.y = fma(h, x.x, acc.y);
}

// sum_s val[s][r] x[col[s][r]] of a row from shared memory, gathers in groups of four
template <typename MV, bool COH>
__device__ __forceinline__ double2 table_sum(const MV* val, const int32_t* col, int L, int rows, int r,
                                             const double2* x, bool imag) {
  double2 acc = make_double2(0.0, 0.0);
  for (int s = 0; s < L; s += 4) {
    double2 q[4];
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (s + u < L) {
        const double2* a = x + col[(s + u) * rows + r];
        q[u] = COH ? __ldcg(a) : __ldg(a);  // rows that other CTAs write during the launch come from L2
      }
#pragma unroll
    for (int u = 0; u < 4; ++u)
      if (s + u < L) {
        const MV h = val[(s + u) * rows + r];
        if constexpr (sizeof(MV) == sizeof(double2)) {
          if (imag)
            table_fma_imag(acc, h.y, q[u]);
          else
            table_fma(acc, h, q[u]);
        } else {
          table_fma(acc, h, q[u]);
        }
      }
  }
  return acc;
}

template <typename MV, bool COH>
__device__ __forceinline__ double2 table_row(const MV* val, const int32_t* col, int L, int rows, int r,
                                             const double2* x, bool imag) {
  const double2 a = table_sum<MV, COH>(val, col, L, rows, r, x, imag);
  if (sizeof(MV) == sizeof(double2) && imag && !table_finite(a))
    return table_sum<MV, COH>(val, col, L, rows, r, x, false);
  return a;
}

template <bool RH, bool RS, bool CLEN>
__global__ void __launch_bounds__(kCompute, 1) resident_table_kernel(const ResidentTable p) {
  using MH = typename MatV<double, RH>::type;
  using MS = typename MatV<double, RS>::type;
  extern __shared__ __align__(16) unsigned char smem[];
  __shared__ int dead_flag, npeers, real_parts;
  __shared__ unsigned need[kMaskWords];
  __shared__ int peer[kMaxGrid];
  const int rows = p.rows, Lh = p.Lh, Ls = p.vs ? p.Ls : 0, tid = threadIdx.x;
  const int64_t row0 = (int64_t)blockIdx.x * rows;
  const int mine = (int)max((int64_t)0, min((int64_t)rows, p.n - row0));
  double2* own = reinterpret_cast<double2*>(smem);  // this CTA's entries of the last two rows, by parity
  MS* sval = reinterpret_cast<MS*>(own + 2 * rows);
  MH* hval = reinterpret_cast<MH*>(smem + table_hval<RS>(Ls, rows));
  int32_t* hcol = reinterpret_cast<int32_t*>(hval + Lh * rows);
  int32_t* scol = hcol + Lh * rows;
  if (tid == 0) dead_flag = npeers = real_parts = 0;
  if (tid < kMaskWords) need[tid] = 0;
  __syncthreads();
  auto needs = [&](int c) {
    const int o = c / rows;
    if (!(need[o >> 5] >> (o & 31) & 1u)) atomicOr(&need[o >> 5], 1u << (o & 31));
  };
  for (int e = tid; e < Lh * mine; e += kCompute) {
    const int s = e / mine, r = e - s * mine;
    hval[s * rows + r] = static_cast<const MH*>(p.vh)[(int64_t)s * p.ld + row0 + r];
    hcol[s * rows + r] = p.ch[(int64_t)s * p.ld + row0 + r];
    needs(hcol[s * rows + r]);
  }
  for (int e = tid; e < Ls * mine; e += kCompute) {
    const int s = e / mine, r = e - s * mine;
    const MS v = static_cast<const MS*>(p.vs)[(int64_t)s * p.ld + row0 + r];
    sval[s * rows + r] = v;
    scol[s * rows + r] = p.cs[(int64_t)s * p.ld + row0 + r];
    if constexpr (!RS) {
      if (v.x != 0.0) real_parts = 1;
    }
    if (!CLEN) needs(scol[s * rows + r]);  // S gathers the table's rows; the sources z are inputs
  }
  __syncthreads();
  if (tid < (int)gridDim.x && tid != (int)blockIdx.x && (need[tid >> 5] >> (tid & 31) & 1u)) peer[atomicAdd(&npeers, 1)] = tid;
  const bool imag = !RS && real_parts == 0;
  __syncthreads();
  bool dead = false;
  auto publish = [&](int m) {  // this CTA's rows of step m are written
    __syncthreads();
    if (tid == 0 && !withheld(p.withhold, m)) st_release(order_word(p.flags, blockIdx.x), m + 1);
  };
  auto await = [&](int m) {
    if (tid < npeers) await_order(p.flags, peer[tid], m, &dead_flag, p.err, p.wait_budget);
    __syncthreads();
    dead = *static_cast<volatile int*>(&dead_flag) != 0;
  };
  if constexpr (!CLEN) {
    for (int r = tid; r < mine; r += kCompute) own[r] = __ldcg(p.tab + row0 + r);  // T_0
    auto s_rows = [&](int m) {  // S T_m
      const double2* x = p.tab + (int64_t)m * p.n;
      for (int r = tid; r < mine; r += kCompute) {
        const double2 a = table_row<MS, true>(sval, scol, Ls, rows, r, x, imag);
        p.stab[(int64_t)m * p.n + row0 + r] = make_double2(0.5 * a.x, 0.5 * a.y);
      }
    };
    for (int m = 1; m < p.M && !dead; ++m) {
      if (m > 1) {
        await(m - 1);
        if (dead) break;
      }
      const double2* x = p.tab + (int64_t)(m - 1) * p.n;
      double2* o = own + (m & 1) * rows;
      const double fh = m == 1 ? 0.5 : 1.0;
      for (int r = tid; r < mine; r += kCompute) {
        const double2 a = table_row<MH, true>(hval, hcol, Lh, rows, r, x, false);
        double2 t = make_double2(fh * a.x, fh * a.y);
        if (m > 1) {
          const double2 q = o[r];
          t.x = fma(-1.0, q.x, t.x);
          t.y = fma(-1.0, q.y, t.y);
        }
        o[r] = t;
        __stcg(p.tab + (int64_t)m * p.n + row0 + r, t);
      }
      publish(m);
      if (p.vs) s_rows(m - 1);
    }
    if (p.vs && !dead) {
      if (p.M > 1) await(p.M - 1);
      if (!dead) s_rows(p.M - 1);
    }
  } else {
    for (int k = p.M - 1; k >= 0 && !dead; --k) {
      const int t = p.M - 1 - k;
      double2 src[kTabItems];
#pragma unroll
      for (int i = 0; i < kTabItems; ++i) {
        const int r = tid + i * kCompute;
        if (r < mine)
          src[i] = p.vs ? table_row<MS, false>(sval, scol, Ls, rows, r, p.z + (int64_t)k * p.n, imag)
                        : __ldg(p.z + (int64_t)k * p.n + row0 + r);
      }
      if (t > 0) {
        await(t - 1);
        if (dead) break;
      }
      const double2* x = p.tab + (int64_t)(k + 1) * p.n;
      double2* o = own + (t & 1) * rows;
      const double fh = k == 0 ? 0.5 : 1.0;
#pragma unroll
      for (int i = 0; i < kTabItems; ++i) {
        const int r = tid + i * kCompute;
        if (r < mine) {
          double2 l = make_double2(0.0, 0.0);
          if (t > 0) {
            const double2 a = table_row<MH, true>(hval, hcol, Lh, rows, r, x, false);
            l = make_double2(fh * a.x, fh * a.y);
          }
          if (p.vs) {
            l.x = fma(0.5, src[i].x, l.x);
            l.y = fma(0.5, src[i].y, l.y);
          }
          if (t > 1) {
            const double2 q = o[r];
            l.x = fma(-1.0, q.x, l.x);
            l.y = fma(-1.0, q.y, l.y);
          }
          if (!p.vs) {
            l.x += src[i].x;
            l.y += src[i].y;
          }
          o[r] = l;
          __stcg(p.tab + (int64_t)k * p.n + row0 + r, l);
        }
      }
      publish(t);
    }
  }
}

// KPM_ERR_UNSUPPORTED where the CTAs do not all fit at once (a context with fewer SMs than the device):
// the step launches serve the call then.
int launch_together(const void* kernel, int grid, int block, void** args, size_t smem, cudaStream_t s) {
  const cudaError_t e = cudaLaunchCooperativeKernel(kernel, dim3(grid), dim3(block), args, smem, s);
  const int st = check_cuda(e);
  return e == cudaErrorCooperativeLaunchTooLarge ? KPM_ERR_UNSUPPORTED : st;
}

template <bool RH, bool RS, bool CLEN>
int launch_table(ResidentTable& p, int sms, cudaStream_t s) {
  const int64_t want = (p.n + kMinItems - 1) / kMinItems;
  int64_t g = std::max<int64_t>(1, std::min<int64_t>(want, std::min(sms, kMaxGrid)));
  const int64_t per = (p.n + g - 1) / g;
  if (per > kMaxTabRows) return KPM_ERR_UNSUPPORTED;
  p.rows = (int)per;
  const int grid = (int)((p.n + per - 1) / per);
  const size_t smem = table_smem<RH, RS>(p.Lh, p.vs ? p.Ls : 0, p.rows);
  if (smem > kMaxSmem) return KPM_ERR_UNSUPPORTED;
  KPM_TRY(allow_smem(resident_table_kernel<RH, RS, CLEN>, kMaxSmem));
  KPM_CUDA_TRY(cudaMemsetAsync(p.flags, 0, (size_t)grid * kFlagStride * sizeof(int), s));
  void* args[] = {&p};
  return launch_together((const void*)resident_table_kernel<RH, RS, CLEN>, grid, kCompute, args, smem, s);
}

// Rows per CTA, grid and shared memory of one launch; KPM_ERR_UNSUPPORTED when it would not fit or
// not pay.
template <typename T, bool REAL, int R>
int resident_shape(const Resident& p, int sm_count, int* rows, int* grid, size_t* smem) {
  const int64_t want = (p.n * R + kMinItems - 1) / kMinItems;
  int64_t g = std::max<int64_t>(1, std::min<int64_t>(want, std::min(sm_count, kMaxGrid)));
  const int64_t per = (p.n + g - 1) / g;
  if (sizeof(T) == 8 ? per * R > kMaxItems64 : p.n * R > kMaxTotal32) return KPM_ERR_UNSUPPORTED;
  *rows = (int)per;
  *grid = (int)((p.n + per - 1) / per);
  *smem = resident_smem<T, REAL>(p.L, *rows, R, p.both != 0);
  return *smem > kMaxSmem ? KPM_ERR_UNSUPPORTED : KPM_OK;
}

template <typename T, bool REAL, int R>
int launch_resident(Resident& p, int sm_count, bool launch, int* grid, cudaStream_t s) {
  size_t smem = 0;
  KPM_TRY((resident_shape<T, REAL, R>(p, sm_count, &p.rows, grid, &smem)));
  if (!launch) return KPM_OK;
  KPM_TRY(allow_smem(resident_kernel<T, REAL, R>, kMaxSmem));
  KPM_CUDA_TRY(cudaMemsetAsync(p.flags, 0, (size_t)*grid * kFlagStride * sizeof(int), s));
  void* args[] = {&p};
  return launch_together((const void*)resident_kernel<T, REAL, R>, *grid, kResThreads, args, smem, s);
}

template <typename T, bool REAL>
int dispatch_r(int R, Resident& p, int sms, bool launch, int* grid, cudaStream_t s) {
  switch (R) {
    case 1: return launch_resident<T, REAL, 1>(p, sms, launch, grid, s);
    case 2: return launch_resident<T, REAL, 2>(p, sms, launch, grid, s);
    case 4: return launch_resident<T, REAL, 4>(p, sms, launch, grid, s);
    case 8: return launch_resident<T, REAL, 8>(p, sms, launch, grid, s);
    default: return KPM_ERR_UNSUPPORTED;
  }
}

int dispatch(bool f32, bool real, int R, Resident& p, int sms, bool launch, int* grid, cudaStream_t s) {
  if (f32) return real ? dispatch_r<float, true>(R, p, sms, launch, grid, s) : dispatch_r<float, false>(R, p, sms, launch, grid, s);
  return real ? dispatch_r<double, true>(R, p, sms, launch, grid, s) : dispatch_r<double, false>(R, p, sms, launch, grid, s);
}

}  // namespace

// The grid of a launch and the handle's buffers for it; KPM_ERR_UNSUPPORTED when it would not fit.
static int resident_buffers(kpm_ell_s* h, bool f32, int Rg, Resident& p, int* grid) {
  KPM_TRY(dispatch(f32, h->is_real != 0, Rg, p, h->sm_count, false, grid, nullptr));
  const size_t pb = (size_t)p.M * (p.both ? 2 : 1) * *grid * Rg * sizeof(double2);
  if (p.M > 65535 || pb > ((size_t)256 << 20)) return KPM_ERR_UNSUPPORTED;
  const size_t vb = (size_t)h->n_pad * Rg * (f32 ? sizeof(float2) : sizeof(double2));
  Workspace& ws = h->ws;
  KPM_TRY(ensure(ws.ta, vb));
  KPM_TRY(ensure(ws.tb, vb));
  KPM_TRY(ensure(ws.part, pb));
  return ensure(ws.flags, kFlagInts * sizeof(int));
}

int resident_reserve(kpm_ell_s* h, bool f32, int Rg, int M) {
  Resident p{};
  p.n = h->n;
  p.L = h->L;
  p.M = M;
  for (p.both = 0; p.both < 2; ++p.both) {
    int grid = 0;
    const int st = resident_buffers(h, f32, Rg, p, &grid);
    if (st != KPM_OK && st != KPM_ERR_UNSUPPORTED) return st;
  }
  return KPM_OK;
}

// Moments of one group of Rg vectors (rows r0 ..), or KPM_ERR_UNSUPPORTED with nothing launched
// when the operator's rows do not fit the SMs' shared memory, or its CTAs the context.
int moments_group_resident(kpm_ell_s* h, bool f32, int R, int r0, int Rg, int M, const double* v_r, const double* v_l,
                           double* mu, double* mu_rr, cudaStream_t s) {
  Resident p{};
  p.val = f32 ? h->val32 : h->val64;
  p.col = h->col;
  p.ld = h->n_pad;
  p.n = h->n;
  p.L = h->L;
  p.M = M;
  p.v_r = reinterpret_cast<const double2*>(v_r) + (int64_t)r0 * h->n;
  p.v_l = v_l ? reinterpret_cast<const double2*>(v_l) + (int64_t)r0 * h->n : nullptr;
  p.both = mu_rr ? 1 : 0;
  p.err = h->err_flag;
  p.wait_budget = h->test_budget > 0 ? h->test_budget : kWaitBudgetCycles;
  p.withhold = h->test_order;
  const int sets = mu_rr ? 2 : 1;
  int grid = 0;
  // Partial sums of all orders take up to 256 MB, the step launches' 128 orders a few: without the memory
  // those serve the call.
  const int st = resident_buffers(h, f32, Rg, p, &grid);
  if (st != KPM_OK) return st == KPM_ERR_OOM ? KPM_ERR_UNSUPPORTED : st;
  Workspace& ws = h->ws;
  p.ta = ws.ta.p;
  p.tb = ws.tb.p;
  p.part = static_cast<double2*>(ws.part.p);
  p.flags = static_cast<int*>(ws.flags.p);
  KPM_TRY(dispatch(f32, h->is_real != 0, Rg, p, h->sm_count, true, &grid, s));
  ++h->one_launch[0];
  double* outs[2] = {mu, mu_rr};
  return reduce_partials(p.part, M, sets, grid, Rg, outs, R, r0, M, 0, s);
}

// A table of T_m (and S T_m), or of the Clenshaw rows (z given), of one vector; row 0 of tab holds T_0.
// KPM_ERR_UNSUPPORTED, nothing launched, when the rows do not fit the SMs' shared memory.
int table_resident(kpm_ell_s* h, kpm_ell_s* s_op, int M, const double2* z, double2* tab, double2* stab, cudaStream_t s) {
  ResidentTable p{};
  p.vh = h->val64;
  p.ch = h->col;
  p.Lh = h->L;
  p.vs = s_op ? s_op->val64 : nullptr;
  p.cs = s_op ? s_op->col : nullptr;
  p.Ls = s_op ? s_op->L : 0;
  p.ld = h->n_pad;
  p.n = h->n;
  p.M = M;
  p.z = z;
  p.tab = tab;
  p.stab = stab;
  p.err = h->err_flag;
  p.wait_budget = h->test_budget > 0 ? h->test_budget : kWaitBudgetCycles;
  p.withhold = h->test_order;
  if ((h->n + h->sm_count - 1) / h->sm_count > kMaxTabRows) return KPM_ERR_UNSUPPORTED;
  // The step launches need no scratch, so tables of one handle may be under way on several streams, or in
  // captured graphs replayed later; here they share the handle's words.  Launches on another stream than the
  // last wait for it, those of another thread take their turn, and a captured call takes the step launches.
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  KPM_CUDA_TRY(cudaStreamIsCapturing(s, &cap));
  if (cap != cudaStreamCaptureStatusNone) return KPM_ERR_UNSUPPORTED;
  std::lock_guard<std::mutex> turn(h->tab_mu);
  if (!h->tab_done) KPM_CUDA_TRY(cudaEventCreateWithFlags(&h->tab_done, cudaEventDisableTiming));
  KPM_CUDA_TRY(cudaStreamWaitEvent(s, h->tab_done, 0));
  p.flags = h->err_flag + kFlagStride;
  const bool rh = h->is_real != 0, rs = !s_op || s_op->is_real != 0;
  const int sms = h->sm_count;
  int st;
  if (z)
    st = rh ? (rs ? launch_table<true, true, true>(p, sms, s) : launch_table<true, false, true>(p, sms, s))
            : (rs ? launch_table<false, true, true>(p, sms, s) : launch_table<false, false, true>(p, sms, s));
  else
    st = rh ? (rs ? launch_table<true, true, false>(p, sms, s) : launch_table<true, false, false>(p, sms, s))
            : (rs ? launch_table<false, true, false>(p, sms, s) : launch_table<false, false, false>(p, sms, s));
  if (st != KPM_OK) return st;
  ++h->one_launch[1];
  return check_cuda(cudaEventRecord(h->tab_done, s));
}

}  // namespace kpm
