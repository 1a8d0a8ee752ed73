// kpm_kubo_step.cu -- one recursion step of the Kubo-Greenwood right rows with the
// velocity product fused in:
//
//   T_{m+1} = 2H T_m - T_{m-1}   (in place over T_{m-1})   and   B_m = V T_m,
//
// in complex64 with the split-float operator values and compensated accumulation of
// the step kernels.  V = H o d (modifier_velocity, jclsquant/modifiers.py:56-79) has
// H's sparsity, so when the two ELL column arrays are equal the gathers of T_m at
// the columns serve both products: one pass over the columns and over T_m instead
// of a recursion step plus a separate V T_m launch (the kpm_mu_nm right-row loop).
//
// Staging is that of cheb_next_ws_kernel: a producer warp issues 1-D bulk copies of
// the tile's column slabs, H value slabs, V value slabs and T_{m-1} into one of
// kWsStages shared-memory stages (full / empty mbarriers, every wait bounded); the
// compute warps gather T_m, accumulate both products and store T_{m+1} and B_m.
//
// V = -i H o d of a real H has no real parts: its values are then read as imaginary splits alone
// (8 bytes a slot for 16) and half of V's products fall away.  The sums are the same bit for bit.
// 1024 x 1024 cells, four vectors: 108.7 -> 98.7 us a step, of 503 -> 436 MB; neither HBM (64 us) nor the
// packed FP32 pipe (about 50) bounds it, but the gathers of 16 compute warps an SM, which registers limit.
#include "kpm_ws.cuh"

namespace kpm {

namespace {

// acc += i h x, h a split float: the general product without its zero terms
template <int VPT>
__device__ __forceinline__ void madd_imag(CxC<VPT>& acc, float2 h, const Cx<float, VPT>& x) {
  const f32x2 b = pair2(-h.x, h.x), nb = pair2(h.x, -h.x), bl = pair2(-h.y, h.y);
#pragma unroll
  for (int k = 0; k < VPT; ++k) {
    const f32x2 w = pair2(x.im[k], x.re[k]);
    two_prod_add(acc.hi[k], acc.lo[k], b, nb, w);
    acc.lo[k] = fma2(bl, w, acc.lo[k]);
  }
}
template <int VPT>
__device__ __forceinline__ void madd_v(CxC<VPT>& acc, float4 h, const Cx<float, VPT>& x) { madd(acc, h, x); }
template <int VPT>
__device__ __forceinline__ void madd_v(CxC<VPT>& acc, float2 h, const Cx<float, VPT>& x) { madd_imag(acc, h, x); }

// The same row with the zero real parts, for rows that come out infinite or NaN.
template <int TPR, int VPT, typename Raw>
__device__ __noinline__ Cx<float, VPT> imag_in_full(const float2* v, const int32_t* col, int tile, int L,
                                                    const Raw* x0) {
  CxC<VPT> acc;
#pragma unroll
  for (int q = 0; q < VPT; ++q) acc.hi[q] = acc.lo[q] = pair2(0.f, 0.f);
  for (int s = 0; s < L; ++s) {
    const float2 w = v[s * tile];
    Cx<float, VPT> x;
    unpack(__ldg(x0 + (int64_t)col[s * tile] * TPR), x);
    madd(acc, make_float4(0.f, w.x, 0.f, w.y), x);
  }
  return finish(acc);
}

// vim: the imaginary splits of V alone, used when *mixed is zero (no V value has a real part); null: not formed.
template <bool REAL, int TPR, int VPT>
__global__ void __launch_bounds__(kWsThreads, 2)
    kubo_step_kernel(const StepParams p, const float4* __restrict__ vval, const float2* __restrict__ vim,
                     const int* __restrict__ mixed, void* bout) {
  using T = float;
  using Raw = typename RawT<T, VPT>::type;
  using MV = typename MatV<T, REAL>::type;
  constexpr int RPB = kBlock / TPR;
  constexpr int TILE = RPB;
  constexpr int kWarps = kBlock / 32;

  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ __align__(8) uint64_t full[kWsStages];
  __shared__ __align__(8) uint64_t empty[kWsStages];

  const int L = p.L;
  const bool imag = vim && *mixed == 0;
  const uint32_t vv_size = imag ? (uint32_t)sizeof(float2) : (uint32_t)sizeof(float4);
  const uint32_t col_b = (uint32_t)align16((size_t)L * TILE * 4);
  const uint32_t val_b = (uint32_t)align16((size_t)L * TILE * sizeof(MV));
  const uint32_t vv_b = (uint32_t)align16((size_t)L * TILE * sizeof(float4));
  const uint32_t vec_b = (uint32_t)(TILE * TPR * sizeof(Raw));
  const uint32_t stage_b = col_b + val_b + vv_b + vec_b;
  const int ntiles = (int)(p.n_pad / TILE);
  const int my_count = ((int)blockIdx.x < ntiles) ? (ntiles - 1 - (int)blockIdx.x) / (int)gridDim.x + 1 : 0;
  auto tile_of = [&](int k) -> int64_t { return (int64_t)blockIdx.x + (int64_t)k * gridDim.x; };

  if (threadIdx.x == 0) {
#pragma unroll
    for (int s = 0; s < kWsStages; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], kWarps);
    }
    fence_mbar_init();
  }
  __syncthreads();

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (warp == kWarps) {  // producer
    if (my_count > 0) {
      const uint64_t pol = l2_evict_first_policy();
      // job j of a tile, one per lane: column, H and V slabs, T_{m-1}
      auto job = [&](int j) {
        TileLane t;
        if (j < L) {
          t.src = reinterpret_cast<const unsigned char*>(p.col + (int64_t)j * p.ld);
          t.row_bytes = 4;
          t.dst = (uint32_t)j * TILE * 4;
        } else if (j < 2 * L) {
          t.src = static_cast<const unsigned char*>(p.val) + (int64_t)(j - L) * p.ld * sizeof(MV);
          t.row_bytes = (uint32_t)sizeof(MV);
          t.dst = col_b + (uint32_t)(j - L) * TILE * (uint32_t)sizeof(MV);
        } else if (j < 3 * L) {
          t.src = (imag ? reinterpret_cast<const unsigned char*>(vim) : reinterpret_cast<const unsigned char*>(vval)) +
                  (int64_t)(j - 2 * L) * p.ld * vv_size;
          t.row_bytes = vv_size;
          t.dst = col_b + val_b + (uint32_t)(j - 2 * L) * TILE * vv_size;
        } else if (j == 3 * L) {
          t.src = static_cast<const unsigned char*>(p.tout);
          t.row_bytes = (uint32_t)(TPR * sizeof(Raw));
          t.dst = col_b + val_b + vv_b;
        }
        t.bytes = t.row_bytes * TILE;
        return t;
      };
      const TileLane mine = job(lane);
      const uint32_t tx = (uint32_t)L * TILE * (4 + (uint32_t)sizeof(MV) + vv_size) + vec_b;
      int issued = 0;
      for (int k = 0; k < my_count; ++k) {
        const int st = k % kWsStages;
        bool ok = true;  // one lane polls: 32 of them slowed the FP64-bound steps
        if (lane == 0 && k >= kWsStages) ok = mbar_wait_bounded(&empty[st], (uint32_t)(((k / kWsStages) - 1) & 1));
        if (!__all_sync(0xffffffffu, ok)) {
          if (lane == 0) atomicExch(p.err, KPM_ERR_TIMEOUT);
          break;
        }
        fence_proxy_async_shared();
        unsigned char* stage = smem + (size_t)st * stage_b;
        const int64_t row0 = tile_of(k) * TILE;
        if (lane == 0) mbar_arrive_expect_tx(&full[st], tx);
        __syncwarp();
        issue_lane(mine, stage, &full[st], row0, pol);
        for (int j = lane + 32; j < 3 * L + 1; j += 32) issue_lane(job(j), stage, &full[st], row0, pol);
        issued = k + 1;
      }
      // copies of the last stages may still be landing: wait for them before leaving
      for (int q = issued > kWsStages ? issued - kWsStages : 0; q < issued; ++q)
        (void)mbar_wait_bounded(&full[q % kWsStages], (uint32_t)((q / kWsStages) & 1));
    }
    return;
  }

  const Raw* __restrict__ tcur = static_cast<const Raw*>(p.tcur);
  Raw* tout = static_cast<Raw*>(p.tout);
  Raw* bo = static_cast<Raw*>(bout);
  const int sub = threadIdx.x % TPR;
  const int rl = threadIdx.x / TPR;
  // V: float4 splits, or the imaginary ones (one branch around the loop: inside it both forms' values
  // are live at once and 112 bytes of them spill; like this 20 to 34)
  auto compute = [&](auto vtype) {
    using V = decltype(vtype);
    bool dead = false;
    for (int k = 0; k < my_count; ++k) {
      const int st = k % kWsStages;
      bool ok = !dead && mbar_wait_bounded(&full[st], (uint32_t)((k / kWsStages) & 1));
      ok = __all_sync(0xffffffffu, ok);
      if (!ok && !dead) {
        if (lane == 0) atomicExch(p.err, KPM_ERR_TIMEOUT);
        dead = true;
      }
      if (!ok) continue;
      const unsigned char* base = smem + (size_t)st * stage_b;
      const int32_t* scol = reinterpret_cast<const int32_t*>(base);
      const MV* sval = reinterpret_cast<const MV*>(base + col_b);
      const unsigned char* svv = base + col_b + val_b;
      const Raw* sold = reinterpret_cast<const Raw*>(base + col_b + val_b + vv_b);
      CxC<VPT> acc, vacc;
      const V* sv = reinterpret_cast<const V*>(svv);
      for (int s = 0; s < L; s += 4) {
        int c[4];
        MV h[4];
        V w[4];
        Cx<T, VPT> x[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (s + j < L) {
            c[j] = scol[(s + j) * TILE + rl];
            h[j] = sval[(s + j) * TILE + rl];
            w[j] = sv[(s + j) * TILE + rl];
          }
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (s + j < L) unpack(__ldg(tcur + (int64_t)c[j] * TPR + sub), x[j]);
        if (s == 0) {
          Cx<T, VPT> o;
          unpack(sold[rl * TPR + sub], o);
          madd_first_neg(acc, h[0], x[0], o);
#pragma unroll
          for (int q = 0; q < VPT; ++q) vacc.hi[q] = vacc.lo[q] = pair2(0.f, 0.f);
        } else {
          madd(acc, h[0], x[0]);
        }
        madd_v(vacc, w[0], x[0]);
#pragma unroll
        for (int j = 1; j < 4; ++j)
          if (s + j < L) {
            madd(acc, h[j], x[j]);
            madd_v(vacc, w[j], x[j]);
          }
      }
      Cx<T, VPT> vb = finish(vacc);  // (2V) T_m: the stored values are doubled
      if constexpr (std::is_same<V, float2>::value) {
        bool bad = false;
#pragma unroll
        for (int q = 0; q < VPT; ++q) bad |= !isfinite(vb.re[q]) || !isfinite(vb.im[q]);
        if (bad) vb = imag_in_full<TPR, VPT>(sv + rl, scol + rl, TILE, L, tcur + sub);
      }
      // the stage is no longer read: hand it back to the producer
      __syncwarp();
      if (lane == 0) mbar_arrive(&empty[st]);
      const int64_t vi = (tile_of(k) * TILE + rl) * TPR + sub;
      tout[vi] = pack(finish(acc));
#pragma unroll
      for (int q = 0; q < VPT; ++q) {
        vb.re[q] *= 0.5f;
        vb.im[q] *= 0.5f;
      }
      bo[vi] = pack(vb);
    }
  };
  if (imag)
    compute(float2{});
  else
    compute(float4{});
}

// vim = the imaginary splits of vval; *mixed becomes 1 when a value has a real part
__global__ void __launch_bounds__(256) kubo_imag_kernel(const float4* __restrict__ vval, int64_t count,
                                                        float2* __restrict__ vim, int* mixed) {
  bool real = false;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (int64_t)gridDim.x * blockDim.x) {
    const float4 v = __ldcs(vval + i);
    real |= v.x != 0.f || v.z != 0.f;
    vim[i] = make_float2(v.y, v.w);
  }
  if (real) *mixed = 1;
}

template <bool REAL, int TPR, int VPT>
size_t kubo_stage_bytes(int L) {
  using MV = typename MatV<float, REAL>::type;
  constexpr int TILE = kBlock / TPR;
  return align16((size_t)L * TILE * 4) + align16((size_t)L * TILE * sizeof(MV)) +
         align16((size_t)L * TILE * sizeof(float4)) + (size_t)TILE * TPR * sizeof(typename RawT<float, VPT>::type);
}

template <bool REAL, int TPR, int VPT>
bool kubo_smem_attr(size_t smem) {
  static size_t configured = 0;
  if (smem <= configured) return true;
  if (cudaFuncSetAttribute(kubo_step_kernel<REAL, TPR, VPT>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)smem) != cudaSuccess) {
    (void)cudaGetLastError();
    return false;
  }
  configured = smem;
  return true;
}

template <bool REAL, int R>
int kubo_go(const StepParams& p, const KuboV& v, void* bout, int sm_count, cudaStream_t s, bool launch) {
  constexpr int VPT = R >= 2 ? 2 : 1;
  constexpr int TPR = R / VPT;
  const size_t smem = kWsStages * kubo_stage_bytes<REAL, TPR, VPT>(p.L);
  if (smem > 200 * 1024 || !kubo_smem_attr<REAL, TPR, VPT>(smem)) return KPM_ERR_UNSUPPORTED;
  int occ = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, kubo_step_kernel<REAL, TPR, VPT>, kWsThreads, smem) !=
          cudaSuccess ||
      occ < 1) {
    (void)cudaGetLastError();
    return KPM_ERR_UNSUPPORTED;
  }
  if (!launch) return KPM_OK;
  const int64_t ntiles = p.n_pad / (kBlock / TPR);
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(ntiles, (int64_t)occ * sm_count));
  kubo_step_kernel<REAL, TPR, VPT><<<grid, kWsThreads, smem, s>>>(p, static_cast<const float4*>(v.val), v.im, v.mixed, bout);
  return check_cuda(cudaGetLastError());
}

}  // namespace

int kubo_imag(const void* vval, int64_t count, void* buf, KuboV* v, cudaStream_t s) {
  int* mixed = static_cast<int*>(buf);
  float2* im = reinterpret_cast<float2*>(static_cast<unsigned char*>(buf) + kKuboImagHead);
  KPM_CUDA_TRY(cudaMemsetAsync(mixed, 0, sizeof(int), s));
  kubo_imag_kernel<<<(int)std::min<int64_t>((count + 255) / 256, 4096), 256, 0, s>>>(static_cast<const float4*>(vval),
                                                                                    count, im, mixed);
  KPM_CUDA_TRY(cudaGetLastError());
  v->im = im;
  v->mixed = mixed;
  return KPM_OK;
}

// The fused step for R vectors (1, 2 or 4); launch == false only checks that it fits.
int kubo_step(bool real_h, int R, const StepParams& p, const KuboV& v, void* bout, int sm_count, cudaStream_t s,
              bool launch) {
  switch (R) {
    case 1: return real_h ? kubo_go<true, 1>(p, v, bout, sm_count, s, launch)
                          : kubo_go<false, 1>(p, v, bout, sm_count, s, launch);
    case 2: return real_h ? kubo_go<true, 2>(p, v, bout, sm_count, s, launch)
                          : kubo_go<false, 2>(p, v, bout, sm_count, s, launch);
    case 4: return real_h ? kubo_go<true, 4>(p, v, bout, sm_count, s, launch)
                          : kubo_go<false, 4>(p, v, bout, sm_count, s, launch);
    default: return KPM_ERR_UNSUPPORTED;
  }
}

}  // namespace kpm
