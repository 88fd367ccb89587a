// FP32 ax_helm for lx = 8, HBM-bound, fed by bulk copies (TMA).
//
// The FP32 operator streams (2 + 6 + c) * 4 bytes per local DOF and does
// ~57 FMA per DOF, well under the FP32 roof, so its speed is the HBM stream.
// A block walks groups of two consecutive elements.  For every group one
// thread issues cp.async.bulk copies of the group's u, G11..G33 (and h1 /
// h2*B / z) -- 4 KB contiguous per array -- into shared memory and arms an
// mbarrier with the byte count.  Four blocks per SM: while one contracts, the
// copies of the others are in flight.  Compute is the same column mapping as
// the generic kernel (thread (i,j) owns the column over k; r/s contractions
// read the staged tile, t on registers).  w is stored straight to global
// memory (coalesced 128-byte rows).  Every mbarrier wait is bounded: on
// timeout the kernel raises a flag, drains its own copies (bounded) and
// returns, so it can never hang the GPU.
//
// One block per SM with three stages of four elements hid its copies but not
// its barriers, with 8 warps on the SM: with the direction update a Poisson
// solve at 43M nodes took 96.9 ms, four blocks of two elements take 89.8, one
// stage of four elements in two blocks 90.6, two stages of two elements in two
// blocks 94.0, ten blocks of one element (at 96 registers) 98.4.  Without the
// direction update, 4096 elements with the preconditioner: 87 -> 78 us; 512
// elements, which no longer fit in one block per SM: 28.9 -> 29.7.
#include "common.cuh"
#include "reduce.cuh"

namespace ntg {

namespace tma {

constexpr int LX = 8, LX2 = 64, LX3 = 512;
constexpr int EPB = 2;                       // elements per group
constexpr int NT = LX2 * EPB;                // 128 threads
constexpr int kBlocks = 4;                   // per SM
constexpr int ARR_BYTES = EPB * LX3 * 4;     // 4 KB per array per group
constexpr unsigned kSpinLimit = 1u << 26;    // bounded waits (seconds)

__device__ __forceinline__ unsigned smem_u32(const void* p) {
  return static_cast<unsigned>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, unsigned bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(dst)),
      "l"(src), "r"(bytes), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void fence_proxy_async() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void fence_mbar_init() { asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory"); }

template <int NARR>
constexpr int smem_bytes() {
  return (NARR + 2) * ARR_BYTES + 64;
}

struct F32Params {
  float d[LX * LX];
};

// Arrays in stage order: 0 u, 1..6 G11 G12 G13 G22 G23 G33, then h1, hB, z.
// DIR: u is p, updated first (AxDir): z is staged beside it, y goes through
// registers, loaded before the wait for the stage.  So p is read once for its
// update and its product; an update kernel of its own took 20 B per node, here
// it adds 16, and an iteration has a launch less.
template <bool H1ARR, bool H2, bool DOT, bool DIR>
__global__ void __launch_bounds__(NT, kBlocks)
    k_ax_helm_f32_tma(float* __restrict__ w, const float* __restrict__ u, const float* __restrict__ g11,
                      const float* __restrict__ g12, const float* __restrict__ g13, const float* __restrict__ g22,
                      const float* __restrict__ g23, const float* __restrict__ g33, const float* __restrict__ h1,
                      float h1c, const float* __restrict__ hB, int64_t nelv, const __grid_constant__ F32Params Dp,
                      double* __restrict__ part, Scalars* sc, int* __restrict__ err, AxDir dir) {
  constexpr int NARR = 7 + (H1ARR ? 1 : 0) + (H2 ? 1 : 0) + (DIR ? 1 : 0);
  dependent_start();
  if (DOT && sc->done) return;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  float* stage = reinterpret_cast<float*>(smem_raw);
  float* s_r = reinterpret_cast<float*>(smem_raw + NARR * ARR_BYTES);
  float* s_s = s_r + EPB * LX3;
  uint64_t* bar = reinterpret_cast<uint64_t*>(s_s + EPB * LX3);

  const int tid = threadIdx.x;
  const int le = tid >> 6;
  const int ij = tid & 63;
  const int i = ij & 7, j = ij >> 3;
  const int64_t ngroups = (nelv + EPB - 1) / EPB;
  const float* srcs[10] = {DIR ? dir.p : u, g11, g12, g13, g22, g23, g33, H1ARR ? h1 : nullptr, H2 ? hB : nullptr,
                           DIR ? dir.z : nullptr};
  const float alpha = DIR ? (float)sc->alpha : 0.f, beta = DIR ? (float)sc->beta : 0.f;

  if (tid == 0) {
    mbar_init(bar, 1);
    fence_mbar_init();
  }
  __syncthreads();

  auto issue = [&](int64_t grp) {
    const int64_t e0 = grp * EPB;
    const int nvalid = (int)((nelv - e0) < EPB ? (nelv - e0) : EPB);
    const unsigned bytes = (unsigned)nvalid * LX3 * 4;
    fence_proxy_async();
    mbar_expect_tx(bar, bytes * NARR);
    int a = 0;
#pragma unroll
    for (int q = 0; q < 10; ++q) {
      if (q == 7 && !H1ARR) continue;
      if (q == 8 && !H2) continue;
      if (q == 9 && !DIR) continue;
      bulk_g2s(stage + (size_t)a * (ARR_BYTES / 4), srcs[q] + e0 * LX3, bytes, bar);
      ++a;
    }
  };

  // my groups: blockIdx.x, blockIdx.x + gridDim.x, ...
  const int64_t my_first = blockIdx.x;
  const int64_t stride = gridDim.x;
  int64_t nmine = my_first < ngroups ? (ngroups - 1 - my_first) / stride + 1 : 0;
  if (tid == 0 && nmine > 0) issue(my_first);
  float Dri[LX], Dsj[LX], DTi[LX], DTj[LX];
#pragma unroll
  for (int l = 0; l < LX; ++l) {
    Dri[l] = Dp.d[i * LX + l];
    Dsj[l] = Dp.d[j * LX + l];
    DTi[l] = Dp.d[l * LX + i];
    DTj[l] = Dp.d[l * LX + j];
  }
  float dot = 0.f;
  bool failed = false;
  unsigned fail_parity = 0;
  for (int64_t t = 0; t < nmine; ++t) {
    const unsigned parity = (unsigned)(t & 1);
    const int64_t grp = my_first + t * stride;
    const int64_t e = grp * EPB + le;
    const bool active = e < nelv;
    float yv[LX];
    if (DIR && active && dir.mode == 0) {
#pragma unroll
      for (int k = 0; k < LX; ++k) yv[k] = dir.y[e * LX3 + ij + k * LX2];
    }
    unsigned spins = 0;
    while (!mbar_try_wait(bar, parity)) {
      if (++spins > kSpinLimit) {
        failed = true;
        break;
      }
    }
    if (__syncthreads_or(failed)) {
      failed = true;
      fail_parity = parity;
      break;
    }
    float* st = stage;
    float* su = st + le * LX3;
    const float* sg11 = st + 1 * (ARR_BYTES / 4) + le * LX3;
    const float* sg12 = st + 2 * (ARR_BYTES / 4) + le * LX3;
    const float* sg13 = st + 3 * (ARR_BYTES / 4) + le * LX3;
    const float* sg22 = st + 4 * (ARR_BYTES / 4) + le * LX3;
    const float* sg23 = st + 5 * (ARR_BYTES / 4) + le * LX3;
    const float* sg33 = st + 6 * (ARR_BYTES / 4) + le * LX3;
    const float* sh1 = st + 7 * (ARR_BYTES / 4) + le * LX3;
    const float* shB = st + (H1ARR ? 8 : 7) * (ARR_BYTES / 4) + le * LX3;
    float* mr = s_r + le * LX3;
    float* ms = s_s + le * LX3;
    float ureg[LX], wt[LX];
    if (active) {
#pragma unroll
      for (int k = 0; k < LX; ++k) ureg[k] = su[ij + k * LX2];
    }
    if (DIR) {
      const float* sz = st + (NARR - 1) * (ARR_BYTES / 4) + le * LX3;
      if (active) {
#pragma unroll
        for (int k = 0; k < LX; ++k) {
          const int q = ij + k * LX2;
          if (dir.mode == 0) dir.y[e * LX3 + q] = yv[k] + alpha * ureg[k];
          ureg[k] = dir.mode == 1 ? sz[q] : sz[q] + beta * ureg[k];
          dir.p[e * LX3 + q] = ureg[k];
          su[q] = ureg[k];
        }
      }
      __syncthreads();
    }
    if (active) {
#pragma unroll
      for (int k = 0; k < LX; ++k) {
        float ur = 0.f, us = 0.f, ut = 0.f;
        const float4* row = reinterpret_cast<const float4*>(su + k * LX2 + j * LX);
        const float4 r0 = row[0], r1 = row[1];
        ur = fmaf(Dri[0], r0.x, ur); ur = fmaf(Dri[1], r0.y, ur); ur = fmaf(Dri[2], r0.z, ur);
        ur = fmaf(Dri[3], r0.w, ur); ur = fmaf(Dri[4], r1.x, ur); ur = fmaf(Dri[5], r1.y, ur);
        ur = fmaf(Dri[6], r1.z, ur); ur = fmaf(Dri[7], r1.w, ur);
#pragma unroll
        for (int l = 0; l < LX; ++l) {
          us = fmaf(Dsj[l], su[k * LX2 + l * LX + i], us);
          ut = fmaf(Dp.d[k * LX + l], ureg[l], ut);
        }
        const int q = ij + k * LX2;
        const float a11 = sg11[q], a12 = sg12[q], a13 = sg13[q], a22 = sg22[q], a23 = sg23[q], a33 = sg33[q];
        const float hh = H1ARR ? sh1[q] : h1c;
        mr[q] = hh * (a11 * ur + a12 * us + a13 * ut);
        ms[q] = hh * (a12 * ur + a22 * us + a23 * ut);
        wt[k] = hh * (a13 * ur + a23 * us + a33 * ut);
      }
    }
    __syncthreads();
    if (active) {
      float* wout = w + e * LX3;
#pragma unroll
      for (int k = 0; k < LX; ++k) {
        float acc = 0.f;
        const float4* rrow = reinterpret_cast<const float4*>(mr + k * LX2 + j * LX);
        const float4 r0 = rrow[0], r1 = rrow[1];
        acc = fmaf(DTi[0], r0.x, acc); acc = fmaf(DTi[1], r0.y, acc); acc = fmaf(DTi[2], r0.z, acc);
        acc = fmaf(DTi[3], r0.w, acc); acc = fmaf(DTi[4], r1.x, acc); acc = fmaf(DTi[5], r1.y, acc);
        acc = fmaf(DTi[6], r1.z, acc); acc = fmaf(DTi[7], r1.w, acc);
#pragma unroll
        for (int l = 0; l < LX; ++l) {
          acc = fmaf(DTj[l], ms[k * LX2 + l * LX + i], acc);
          acc = fmaf(Dp.d[l * LX + k], wt[l], acc);
        }
        const int q = ij + k * LX2;
        if (H2) acc = fmaf(shB[q], ureg[k], acc);
        wout[q] = acc;
        if (DOT) dot = fmaf(ureg[k], acc, dot);
      }
    }
    __syncthreads();  // the stage and s_r/s_s are free again
    if (tid == 0 && t + 1 < nmine) issue(my_first + (t + 1) * stride);
  }
  if (failed) {
    if (tid == 0) {
      atomicExch(err, 1);
      // drain: the failed group's copies were issued; wait (bounded) for them
      // before leaving
      unsigned spins = 0;
      while (spins < kSpinLimit && !mbar_try_wait(bar, fail_parity)) ++spins;
    }
    __syncthreads();
    if (DOT && tid == 0) {
      sc->status = NTG_ERR_CUDA;
      sc->done = 1;
    }
    return;
  }
  if (DOT) {
    double v[1] = {(double)dot};
    grid_reduce<1>(v, part, sc, FinPap());
  }
}

template <bool H1ARR, bool H2, bool DOT, bool DIR>
static int launch_variant(ntg_plan* p, float* w, const float* u, const float* const* g, const float* h1, float h1c,
                          const float* hB, Scalars* sc, const AxDir* dir, cudaStream_t s) {
  constexpr int NARR = 7 + (H1ARR ? 1 : 0) + (H2 ? 1 : 0) + (DIR ? 1 : 0);
  constexpr int SMEM = smem_bytes<NARR>();
  static bool attr_done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  auto kern = k_ax_helm_f32_tma<H1ARR, H2, DOT, DIR>;
  if (dev >= 0 && dev < 64 && !attr_done[dev]) {
    NTG_CUDA_TRY(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
    attr_done[dev] = true;
  }
  F32Params Dp;
  for (int q = 0; q < LX * LX; ++q) Dp.d[q] = p->Df[q];
  const int64_t ngroups = (p->nelv + EPB - 1) / EPB;
  int grid = num_sms() * kBlocks;
  if (ngroups < grid) grid = (int)ngroups;
  return launch_dependent(p, kern, grid, NT, SMEM, s, w, u, g[0], g[1], g[2], g[3], g[4], g[5], h1, h1c, hB, p->nelv, Dp,
                          p->red_part, sc, p->dev_err, dir ? *dir : AxDir{});
}

}  // namespace tma

static bool aligned16(const void* q) { return q == nullptr || (reinterpret_cast<uintptr_t>(q) & 15u) == 0; }

int ax_f32_tma_launch(ntg_plan* p, float* w, const float* u, const float* const* g, const float* h1, float h1c,
                      const float* hB, Scalars* sc, const AxDir* dir, cudaStream_t s) {
  if (p->lx != 8 || !p->dev_err) return NTG_ERR_UNSUPPORTED;
  // a bulk copy must start on a 16-byte boundary: every element group starts
  // at a multiple of 2 KB from the array base, so the bases decide
  const void* ptrs[12] = {w, u, g[0], g[1], g[2], g[3], g[4], g[5], h1, hB, dir ? dir->p : nullptr,
                          dir ? dir->z : nullptr};
  for (const void* q : ptrs)
    if (!aligned16(q)) return NTG_ERR_UNSUPPORTED;
  const bool h1a = h1 != nullptr, h2 = hB != nullptr, dot = sc != nullptr;
#define NTG_TMA_CASE(A, B, C, E)                                    \
  if (h1a == A && h2 == B && dot == C && (dir != nullptr) == E)     \
    return tma::launch_variant<A, B, C, E>(p, w, u, g, h1, h1c, hB, sc, dir, s);
  NTG_TMA_CASE(false, false, false, false)
  NTG_TMA_CASE(false, true, false, false)
  NTG_TMA_CASE(true, false, false, false)
  NTG_TMA_CASE(true, true, false, false)
  NTG_TMA_CASE(false, false, true, false)
  NTG_TMA_CASE(false, true, true, false)
  NTG_TMA_CASE(true, false, true, false)
  NTG_TMA_CASE(true, true, true, false)
  NTG_TMA_CASE(false, false, true, true)
  NTG_TMA_CASE(false, true, true, true)
  NTG_TMA_CASE(true, false, true, true)
  NTG_TMA_CASE(true, true, true, true)
#undef NTG_TMA_CASE
  return NTG_ERR_UNSUPPORTED;
}

}  // namespace ntg

using namespace ntg;

// Select the FP32 Ax path of a plan: 1 = bulk-copy pipeline (lx = 8), 0 =
// the generic kernel.
extern "C" int ntg_plan_set_ax_path(ntg_plan* plan, int use_tma) {
  clear_error();
  NTG_CHECK_ARG(plan, "ntg_plan_set_ax_path: null plan");
  plan->use_tma = use_tma ? 1 : 0;
  return NTG_OK;
}

// Select the gather-scatter kernel: 1 = by multiplicity class (default),
// 0 = one thread per shared group.  Both give bit-identical results.
extern "C" int ntg_plan_set_gs_path(ntg_plan* plan, int by_class) {
  clear_error();
  NTG_CHECK_ARG(plan, "ntg_plan_set_gs_path: null plan");
  plan->gs_classes = by_class ? 1 : 0;
  return NTG_OK;
}

// 1 if a bounded wait of a kernel of this plan ran out (the flag is cleared).
extern "C" int ntg_plan_check_error(ntg_plan* plan, int* flag) {
  clear_error();
  NTG_CHECK_ARG(plan && flag, "ntg_plan_check_error: null argument");
  int h = 0;
  NTG_CUDA_TRY(cudaMemcpyAsync(&h, plan->dev_err, sizeof(int), cudaMemcpyDeviceToHost, plan->stream));
  NTG_CUDA_TRY(cudaStreamSynchronize(plan->stream));
  if (h) NTG_CUDA_TRY(cudaMemsetAsync(plan->dev_err, 0, sizeof(int), plan->stream));
  *flag = h;
  return NTG_OK;
}
