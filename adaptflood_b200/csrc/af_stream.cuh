// af_stream.cuh -- the time loop of a grid in HBM, many steps in one launch.
//
// The strips of af_step.cuh, one cooperative launch for a call's steps, or as
// many as take some 8 ms: one block per SM, 16 warps, each marching its strips as k_step's
// one-warp blocks do, and between steps the exchange of af_exchange.cuh instead
// of a kernel boundary.  A boundary costs its own launch, the last block's fold
// (a chain of dependent loads and atomics, the rain look-up among them) and
// every block's prologue, some 9 us a step together; the exchange 2.5.
//
// The state a step writes with ordinary stores is read by the next step's bulk
// copies (the async proxy) on other SMs: every thread fences its stores for
// that proxy before the block's barrier, warp 0 fences at GPU scope before it
// posts and after it has collected, and every thread fences for the proxy again
// before it issues copies.
#pragma once

#include "af_exchange.cuh"

namespace af {

__device__ inline void fence_proxy_async_global() {
  asm volatile("fence.proxy.async.global;" ::: "memory");
}

template <typename T>
__host__ __device__ constexpr size_t stream_smem() {
  return (size_t)kLoopWarps * kStages * 4 * RowWin<T>::bytes + 128;  // and alignment
}

template <typename T, bool kTma>
__global__ void __launch_bounds__(32 * kLoopWarps, 1)
    k_stream(const __grid_constant__ StepParams p, const __grid_constant__ LoopParams lp,
             const __grid_constant__ CUtensorMap fields) {
  using Ring = unsigned char[kStages][4][RowWin<T>::bytes];
  extern __shared__ unsigned char s_raw[];
  __shared__ __align__(8) uint64_t s_bar[kLoopWarps][kStages];
  __shared__ LoopShared<T> S;
  Ring* const rings =
      reinterpret_cast<Ring*>(s_raw + (128u - (smem_u32(s_raw) & 127u)) % 128u);
  SimCtl* ctl = p.ctl;
  const int tid = threadIdx.x, lane = tid & 31;
  const int warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int nb = gridDim.x, b = blockIdx.x;
  const int par0 = ctl->parity;
  const unsigned tag0 = *lp.tag;
  long long n = 0;
  const bool go = loop_goes(ctl, lp);
  if (tid == 0) start_clock(p, lp, S);
  uint64_t* const bar = s_bar[warp];
  if (lane == 0) {
    for (int s = 0; s < kStages; s++) mbar_init(&bar[s], 1);
    fence_mbar_init();
  }
  __syncthreads();
  RingPos pos{0u};
  const int ntiles = p.nsx * p.nsy;
  bool failed = false;
#pragma unroll 1
  while (go) {
    LaneAcc<T> acc{T(-FLT_MAX), 0.0, 0.0};
    bool ok = true;
    {
      const StepScal<T> sc = S.sc;
      for (int tile = warp * nb + b; tile < ntiles && ok; tile += kLoopWarps * nb) {
        const int sx = tile % p.nsx, sy = tile / p.nsx;
        if constexpr (sizeof(T) == 8)
          ok = run_strip64<kTma>(p, sc, sx, sy, rings[warp], bar, pos, acc, &fields);
        else
          ok = run_strip<T, true, kTma>(p, sc, sx, sy, rings[warp], bar, pos, acc, &fields);
      }
      if (!ok && lane == 0) S.fail = 1;
      hand_in(S, warp, acc.m_cell, acc.v, acc.a, sc.mass);
    }
    fence_proxy_async_global();
    __syncthreads();
    if (warp == 0) step_clock<T, true>(p, lp, S, tag0 + (unsigned)n, n);
    __syncthreads();
    n++;
    if (S.fail) {
      failed = true;
      break;
    }
    if (S.done) break;
    fence_proxy_async_global();
  }
  if (failed && tid == 0) atomicExch(&ctl->status, 2);
  if (b == 0 && tid == 0) stop_clock(p, lp, S, par0, tag0, n);
}

}  // namespace af
