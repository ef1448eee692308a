// af_exchange.cuh -- what the blocks of a whole-loop launch tell each other
// after a step, and the clock they keep alike.
//
// A cooperative launch runs many steps (af_resident.cuh: the state in shared
// memory; af_stream.cuh: in HBM).  After a step every block needs Hmax of all
// of them for the next dt; everything else of the clock (time, rain rate, loop
// decisions) each block derives from it by itself, with the same operations.
//
// Every 8 bytes that cross blocks carry 4 bytes of data and the step's tag, so
// a reader polls the data itself and no flag stands between a step's last store
// and its first use (an 8-byte aligned access is not torn).  Buffers alternate
// between two copies: a block writes step n+2's only after it has read every
// block's Hmax of step n+1, which each sends after it has read step n's.  Every
// wait is bounded; a block that gives up flags the control block and leaves,
// and so then do the others.
#pragma once

#include <type_traits>

#include "af_step.cuh"

namespace af {

constexpr int kLoopWarps = 16;  // warps of a block: one block per SM

struct LoopParams {
  void* slot;     // [2][to][from] Hmax words, see post_max
  double* part;   // [2][blocks][2] volume and area at mass-report steps
  unsigned* tag;  // first unused tag
  // The first launch of a call (more = 0) has the call's limits, those after it
  // find them in the control block.  A launch ends after `slice` steps at most.
  double t_stop;
  long long max_steps;
  int slice;
  int more;
};

__device__ inline uint4 ld_relaxed(const uint4* p) {
  uint4 v;
  asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p)
               : "memory");
  return v;
}
__device__ inline void st_relaxed(uint4* p, uint4 v) {
  asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(v.x), "r"(v.y),
               "r"(v.z), "r"(v.w)
               : "memory");
}

// Largest of a warp's ordered 64-bit images (ord_encode).
__device__ __forceinline__ unsigned long long warp_max_ord(unsigned long long v) {
  const unsigned hi = (unsigned)(v >> 32);
  const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
  const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? (unsigned)v : 0u);
  return ((unsigned long long)mh << 32) | ml;
}

__device__ inline float cell_update(float h, float qw, float qe, float qn, float qs, bool rain,
                                    const StepScal<float>& sc) {
  // The operations of update_cells<float>, one cell in a pair.
  const float2 a = __ffma2_rn(f2(qe, qs), f2(-1.0f, -1.0f), f2(qw, qn));
  const float2 d = __fadd2_rn(f2(a.x, 0.0f), f2(a.y, 0.0f));
  const float2 inc = __ffma2_rn(f2(sc.dt_dA, 0.0f), d, f2(rain ? sc.rain_depth : 0.0f, 0.0f));
  return fmaxf(__fadd2_rn(f2(h, 0.0f), inc).x, 0.0f);
}
__device__ inline double cell_update(double h, double qw, double qe, double qn, double qs,
                                     bool rain, const StepScal<double>& sc) {
  return update_cell(h, qw, qe, qn, qs, rain, sc.rain_depth, sc.dtT, sc.dAT, sc.ph);
}

// Hmax of all blocks: each writes its own (the depth's ordered image with the
// step's tag beside every 4 bytes) into every block's row and polls only its
// own row, one warp per block.  Cycles per exchange of 148 blocks by itself:
// 2900 with 8-byte words (FP32), 3700 with 16-byte words (FP64); all polling
// one shared row 5800, two rounds in groups of 13 4100; an atomic maximum with
// a counted arrival 3000, but 5000 in the loop, where its release also waits
// for the halo stores.
__device__ inline unsigned ord32(float x) {
  const unsigned u = __float_as_uint(x);
  return u & 0x80000000u ? ~u : u | 0x80000000u;
}
__device__ inline float ord32_value(unsigned u) {
  return __uint_as_float(u & 0x80000000u ? u & 0x7fffffffu : ~u);
}
struct MaxF32 {
  using Bits = unsigned;
  using Word = uint2;
  __device__ static Bits of(float m) { return ord32(m); }
  __device__ static double value(Bits b) { return (double)ord32_value(b); }
  __device__ static Bits warp(Bits b) { return __reduce_max_sync(0xffffffffu, b); }
  __device__ static void put(Word* p, Bits b, unsigned tag) {
    asm volatile("st.relaxed.gpu.global.v2.u32 [%0], {%1, %2};" ::"l"(p), "r"(b), "r"(tag)
                 : "memory");
  }
  __device__ static bool get(const Word* p, Bits& b, unsigned tag) {
    unsigned t;
    asm volatile("ld.relaxed.gpu.global.v2.u32 {%0, %1}, [%2];" : "=r"(b), "=r"(t) : "l"(p)
                 : "memory");
    return t == tag;
  }
};
struct MaxF64 {
  using Bits = unsigned long long;
  using Word = uint4;
  __device__ static Bits of(double m) { return ord_encode(m); }
  __device__ static double value(Bits b) { return ord_decode(b); }
  __device__ static Bits warp(Bits b) { return warp_max_ord(b); }
  __device__ static void put(Word* p, Bits b, unsigned tag) {
    st_relaxed(p, make_uint4((unsigned)b, tag, (unsigned)(b >> 32), tag));
  }
  __device__ static bool get(const Word* p, Bits& b, unsigned tag) {
    const uint4 x = ld_relaxed(p);
    b = ((Bits)x.z << 32) | x.x;
    return (x.y == tag) & (x.w == tag);
  }
};
template <typename T>
using MaxOf = typename std::conditional<sizeof(T) == 8, MaxF64, MaxF32>::type;

template <typename M>
__device__ __forceinline__ void post_max(void* slot, int nb, int buf, int b, unsigned tag,
                                         typename M::Bits v) {
  typename M::Word* const to = static_cast<typename M::Word*>(slot) + (size_t)buf * nb * nb + b;
  for (int k = threadIdx.x & 31; k < nb; k += 32) M::put(to + (size_t)k * nb, v, tag);
}
// False when a wait ran out.
template <typename M>
__device__ __forceinline__ bool collect_max(void* slot, int nb, int buf, int b, unsigned tag,
                                            typename M::Bits& v) {
  constexpr int K = 5;  // loads in flight per lane: one round on up to 160 blocks
  const typename M::Word* const row =
      static_cast<const typename M::Word*>(slot) + ((size_t)buf * nb + b) * nb;
  const int lane = threadIdx.x & 31;
  typename M::Bits m = 0;
  bool ok = true;
  for (int k0 = lane; k0 - lane < nb; k0 += 32 * K) {
    typename M::Bits x[K];
    bool all = false;
    for (int w = 0; w < (int)kRingWaitLimit && !all; w++) {
      all = true;
#pragma unroll
      for (int u = 0; u < K; u++) all &= M::get(row + min(k0 + 32 * u, nb - 1), x[u], tag);
    }
    ok &= all;
#pragma unroll
    for (int u = 0; u < K; u++) m = x[u] > m ? x[u] : m;
  }
  v = M::warp(m);
  return __all_sync(0xffffffffu, ok);
}

// What warp 0 carries from step to step, in shared memory so that it takes no
// registers of the step.
struct Clock {
  double t, dt_last, hmax, rate, next_mass;
  double t_stop;   // the call's
  int most;        // steps of this launch
  double r_t0, r_t1, r_v0, r_v1;  // the rain series' segment of the last look-up
  int status, mass_count;
};

// A block's shared words of the loop.
template <typename T>
struct LoopShared {
  StepScal<T> sc;  // the step's constants; rewritten by warp 0 between steps
  Clock clock;
  typename MaxOf<T>::Bits max[kLoopWarps];
  double v[kLoopWarps], a[kLoopWarps];
  int done, fail;
  int par0;       // the parity and first tag of this launch
  unsigned tag0;
};

// Whether there is a step to take, the same in every block and thread.
__device__ inline bool loop_goes(const SimCtl* ctl, const LoopParams& lp) {
  return ctl->status == 0 && (lp.more ? !ctl->done : ctl->t < lp.t_stop && lp.max_steps > 0);
}

// The loop's start from the control block, the same in every block (one
// thread).
template <typename T>
__device__ inline void start_clock(const StepParams& p, const LoopParams& lp, LoopShared<T>& S) {
  const SimCtl* ctl = p.ctl;
  Clock& k = S.clock;
  k.t_stop = lp.more ? ctl->t_stop : lp.t_stop;
  const long long left = lp.more ? ctl->step_stop - ctl->step : lp.max_steps;
  k.most = left < lp.slice ? (int)left : lp.slice;
  k.t = ctl->t;
  k.dt_last = ctl->dt_last;
  k.hmax = ctl->hmax;
  k.rate = ctl->rain_rate;
  k.next_mass = ctl->next_mass;
  k.r_t0 = k.r_v0 = k.r_v1 = 0.0;
  k.r_t1 = -1.0;
  k.status = ctl->status;
  k.mass_count = ctl->mass_count;
  fill_scalars(p, k.t, step_dt(p, k.hmax), k.rate, k.next_mass, ctl->parity, S.sc);
  S.done = !loop_goes(ctl, lp);
  S.fail = 0;
  S.par0 = ctl->parity;
  S.tag0 = *lp.tag;
}

// One warp's share of the step: its largest valid depth (-FLT_MAX: none) and,
// at mass-report steps, its volume and area.
template <typename T>
__device__ __forceinline__ void hand_in(LoopShared<T>& S, int warp, T m, double v, double a,
                                        bool mass) {
  const typename MaxOf<T>::Bits mo = MaxOf<T>::warp(MaxOf<T>::of(m));
  if (mass) {
    v = warp_sum(v);
    a = warp_sum(a);
  }
  if ((threadIdx.x & 31) == 0) {
    S.max[warp] = mo;
    S.v[warp] = v;
    S.a[warp] = a;
  }
}

// Warp 0 of every block, after the whole block's step n (tag `tag`): Hmax of
// all blocks, then the next step's time, dt and constants.  kState: the state
// went to global memory, so it must be there before the word that says so.
template <typename T, bool kState, typename N>
__device__ __forceinline__ void step_clock(const StepParams& p, const LoopParams& lp,
                                           LoopShared<T>& S, unsigned tag, N n) {
  using M = MaxOf<T>;
  constexpr int NW = kLoopWarps;
  const int lane = threadIdx.x & 31, nb = gridDim.x, b = blockIdx.x, buf = (int)(n & 1);
  const StepScal<T>& sc = S.sc;
  Clock& ck = S.clock;
  const bool mass = sc.mass;
  const typename M::Bits bm = M::warp(lane < NW ? S.max[lane] : 0);
  if (mass) {
    if (lane == 0) {
      double sv = 0.0, sa = 0.0;
      for (int w = 0; w < NW; w++) {
        sv += S.v[w];
        sa += S.a[w];
      }
      lp.part[(size_t)(buf * nb + b) * 2] = sv;
      lp.part[(size_t)(buf * nb + b) * 2 + 1] = sa;
      __threadfence();
    }
    __syncwarp();
  }
  // The limits, read before this block posts: block 0 rewrites them only after it
  // has every block's word.  The streamed FP64 loop has them from the control
  // block: with two more words of the clock the compiler gives its row loop other
  // registers, 5 % slower (8192^2 1590 -> 1665 us a step).  In the other loops the
  // loads cost (resident FP32 317x203 4.02 -> 4.18 us, streamed 2500x1801 31.2 ->
  // 31.4).
  double t_stop;
  long long most;
  if constexpr (kState && sizeof(T) == 8) {
    t_stop = lp.more ? p.ctl->t_stop : lp.t_stop;
    most = lp.more ? p.ctl->step_stop - p.ctl->step : lp.max_steps;
  } else {
    t_stop = ck.t_stop;
    most = ck.most;
  }
  // The new state, written by the whole block, before the word that says so.
  if (kState) __threadfence();
  post_max<M>(lp.slot, nb, buf, b, tag, bm);
  // Time and rain rate while the others' Hmax is on its way.
  const double t = sc.t + sc.dt;
  double rate = 0.0;
  if (p.n_rain > 0) {
    const double t0 = ck.r_t0, t1 = ck.r_t1;
    if (t0 <= t && t < t1) {  // still in the segment: interp_series' own expression
      const double v0 = ck.r_v0;
      rate = v0 + (t - t0) / (t1 - t0) * (ck.r_v1 - v0);
    } else {
      const int k = rain_segment(p, t);
      rate = interp_series(p.rain_times, p.rain_rates, p.n_rain, 0.0, t, p.rain_sorted != 0);
      __syncwarp();
      if (lane == 0) {
        ck.r_t1 = -1.0;
        if (k >= 0) {
          ck.r_t0 = p.rain_times[k];
          ck.r_t1 = p.rain_times[k + 1];
          ck.r_v0 = p.rain_rates[k];
          ck.r_v1 = p.rain_rates[k + 1];
        }
      }
    }
  }
  typename M::Bits gm;
  const bool ok = collect_max<M>(lp.slot, nb, buf, b, tag, gm);
  if (kState) __threadfence();
  const double gd = M::value(gm);
  // The bookkeeping of fold_step, in every block alike.
  const double hmax = gd > -(double)FLT_MAX ? gd : -DBL_MAX;
  double next_mass = ck.next_mass;
  int mass_count = ck.mass_count;
  if (mass) {
    if (b == 0 && mass_count < p.ctl->mass_cap) {
      __threadfence();
      const double* part = lp.part + (size_t)buf * nb * 2;
      double s = 0.0, cs = 0.0, ar = 0.0;
      for (int k = lane; k < nb; k += 32) {
        kahan_add(s, cs, __ldcg(&part[2 * k]));
        ar += __ldcg(&part[2 * k + 1]);
      }
      double S = 0.0, C = 0.0, A = 0.0;
      for (int l = 0; l < 32; l++) {
        kahan_add(S, C, __shfl_sync(0xffffffffu, s, l));
        C += __shfl_sync(0xffffffffu, cs, l);
        A += __shfl_sync(0xffffffffu, ar, l);
      }
      if (lane == 0) {
        p.mass_series[3 * mass_count] = t;
        p.mass_series[3 * mass_count + 1] = S + C;
        p.mass_series[3 * mass_count + 2] = A;
      }
      mass_count++;
    }
    next_mass += p.mass_int;
  }
  const double dt_last = sc.dt;
  const bool bad = !(dt_last > 0.0) || !(t < 1.0e300) || !(hmax == hmax);
  const int status = !ok ? 2 : bad ? 1 : 0;
  const bool done = status != 0 || !(t < t_stop) || n + 1 >= lp.slice || n + 1 >= most;
  __syncwarp();
  if (lane == 0) {
    if (!done) {
      fill_step(p, t, step_dt(p, hmax), rate, next_mass, sc.parity ^ 1, S.sc);
    }
    if (!ok) S.fail = 1;
    S.done = done;
    ck.t = t;
    ck.dt_last = dt_last;
    ck.hmax = hmax;
    ck.rate = rate;
    ck.next_mass = next_mass;
    ck.status = status;
    ck.mass_count = mass_count;
  }
}

// The control block after the launch (one thread of block 0), n steps on.
template <typename T, typename N>
__device__ inline void stop_clock(const StepParams& p, const LoopParams& lp,
                                  const LoopShared<T>& S, int par0, unsigned tag0, N n) {
  SimCtl* ctl = p.ctl;
  const Clock& k = S.clock;
  const long long limit = 0x3FFFFFFFFFFFFFFFLL;
  if (!lp.more) {
    ctl->t_stop = lp.t_stop;
    ctl->step_stop = lp.max_steps > limit - ctl->step ? limit : ctl->step + lp.max_steps;
  }
  ctl->arrive = 0u;
  if (n > 0) {
    ctl->step += n;
    ctl->t = k.t;
    ctl->hmax = k.hmax;
    ctl->dt_last = k.dt_last;
    ctl->rain_rate = k.rate;
    ctl->next_mass = k.next_mass;
    ctl->mass_count = k.mass_count;
    ctl->parity = par0 ^ (int)(n & 1);
    if (k.status != 0) atomicMax(&ctl->status, k.status);
    *lp.tag = tag0 + (unsigned)n + 16u;
  }
  // A block that gave up in the last step may say so later than this; the next
  // launch then takes no step and ends the call.
  ctl->done = *(volatile int*)&ctl->status != 0 || !(ctl->t < ctl->t_stop) ||
              ctl->step >= ctl->step_stop;
}

}  // namespace af
