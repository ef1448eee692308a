// af_resident.cuh -- the time loop of a small grid, many steps in one launch,
// its state held on chip.
//
// A step of a small grid costs a kernel boundary, a prologue of dependent
// loads and one trip to L2 per row, not bandwidth: 64 k cells took 11.4 us a
// step and 0.8 M cells 20 us, against 0.3 and 3.4 us of HBM time.  Here one
// cooperative launch runs a call's steps (8 ms of them): block b of (at most) one
// per SM keeps a band of rows in shared memory and exchanges with the others
// only its first and last rows' new H and Qx and its Hmax.
//
// Work.  A warp marches 32 columns down some rows, as the strip kernels do but
// without halo lanes: the left neighbours come from shared memory, and the
// faces on the strip's east side, for all its rows at once (a lane each),
// share one evaluation with the faces above its first row.  The same face
// law, edge law and update functions as the strip kernels, in the same order,
// so results are the same bit for bit.
#pragma once

#include "af_exchange.cuh"

namespace af {

struct ResidentParams {
  const int* row_off;       // special cells by row (CSR over rows, sorted by column)
  const SpecCell* row_spec;
  uint4* halo;              // [2][blocks][2][W][halo_words]
  int nr_max;               // rows of the tallest band
  int gy;                   // row groups a band is cut into (at most 32 rows each)
  LoopParams loop;
};

// Nanoseconds that the warps beside warp 0 are late past the march's barrier.  A
// test build sets it, so that what they read there is read after warp 0 has
// gone on to the next step.
#ifndef AF_LATE_NS
#define AF_LATE_NS 0
#endif
constexpr unsigned kLateNs = AF_LATE_NS;

template <typename T>
struct ResidentShape;
template <>
struct ResidentShape<float> {
  static constexpr int threads = 512;
  static constexpr int halo_words = 1;  // uint4 per column: {H, tag, Qx, tag}
};
template <>
struct ResidentShape<double> {
  static constexpr int threads = 512;
  static constexpr int halo_words = 2;  // {H lo, tag, H hi, tag}, the same of Qx
};

// Dynamic shared memory of a band of nr rows of nx cells: two copies of H and
// of Qx and one of Z over nr + 2 rows, two of Qy over nr + 1, per 32 cells the
// special cells' mask and first entry, and the list of marches (gy row groups
// per strip).
template <typename T>
__host__ __device__ inline size_t resident_smem(int nx, int nr, int gy) {
  const size_t W = (size_t)nx + 1, nsx = (nx + 31) / 32;
  return (W * (size_t)(7 * nr + 12) + 4) * sizeof(T) + 16 + nsx * (16 * (size_t)gy + 8 * (size_t)nr);
}

// Rows the busiest of a block's warps marches when a band of nr rows is cut
// into g groups: every group costs about one and a half more than its rows (its
// first loads and the faces above and beside it).
inline double resident_cost(int nx, int nr, int warps, int g) {
  const int nsx = (nx + 31) / 32;
  return (double)((nsx * g + warps - 1) / warps) * ((nr + g - 1) / g + 1.5);
}
// The number of groups that costs least; a group has at most 32 rows.
inline int resident_groups(int nx, int nr, int warps) {
  int best = (nr + 31) / 32;
  for (int g = best + 1; g <= nr; g++)
    if (resident_cost(nx, nr, warps, g) < resident_cost(nx, nr, warps, best)) best = g;
  return best;
}

__device__ inline void halo_put(uint4* at, float h, float q, unsigned tag) {
  st_relaxed(at, make_uint4(__float_as_uint(h), tag, __float_as_uint(q), tag));
}
__device__ inline void halo_put(uint4* at, double h, double q, unsigned tag) {
  st_relaxed(at, make_uint4((unsigned)__double2loint(h), tag, (unsigned)__double2hiint(h), tag));
  st_relaxed(at + 1, make_uint4((unsigned)__double2loint(q), tag, (unsigned)__double2hiint(q), tag));
}
__device__ inline bool halo_get(const uint4* at, float& h, float& q, unsigned tag) {
  const uint4 v = ld_relaxed(at);
  h = __uint_as_float(v.x);
  q = __uint_as_float(v.z);
  return (v.y == tag) & (v.w == tag);
}
__device__ inline bool halo_get(const uint4* at, double& h, double& q, unsigned tag) {
  const uint4 v = ld_relaxed(at), w = ld_relaxed(at + 1);
  h = __hiloint2double((int)v.z, (int)v.x);
  q = __hiloint2double((int)w.z, (int)w.x);
  return (v.y == tag) & (v.w == tag) & (w.y == tag) & (w.w == tag);
}

// Two faces by the interior law; face k lies between cells (z0k, h0k) and
// (z1k, h1k).  Discharges are the stored ones (FP64 forms Qold here).
template <typename T>
struct FaceIn {
  T z0, h0, z1, h1, q0, qa, qb, qc, qd;
};
__device__ __forceinline__ void two_faces(const FaceIn<float>& a, const FaceIn<float>& b,
                                          float /*dxinv*/, bool ea, bool eb,
                                          const Phys<float>& ph, float& qa, float& qb) {
  bool any = false;
  const float2 q = flux2<true>(f2(a.z0, b.z0), f2(a.h0, b.h0), f2(a.z1, b.z1), f2(a.h1, b.h1),
                               f2(a.q0, b.q0), f2(a.qa, b.qa), f2(a.qb, b.qb), f2(a.qc, b.qc),
                               f2(a.qd, b.qd), true, ph, any);
  qa = ea ? q.x : 0.0f;
  qb = eb ? q.y : 0.0f;
}
__device__ __forceinline__ void two_faces(const FaceIn<double>& a, const FaceIn<double>& b,
                                          double dxinv, bool ea, bool eb, const Phys<double>& ph,
                                          double& qa, double& qb) {
  const double ya0 = a.z0 + a.h0, ya1 = a.z1 + a.h1, yb0 = b.z0 + b.h0, yb1 = b.z1 + b.h1;
  const double ha = gminT(gmaxT(ya0, ya1) - gmaxT(a.z0, a.z1), ph.max_hflow);
  const double hb = gminT(gmaxT(yb0, yb1) - gmaxT(b.z0, b.z1), ph.max_hflow);
  const bool wa = ea & (a.z0 != ph.nodata) & (a.z1 != ph.nodata) & (ha > ph.depth_thresh);
  const bool wb = eb & (b.z0 != ph.nodata) & (b.z1 != ph.nodata) & (hb > ph.depth_thresh);
  qa = 0.0;
  qb = 0.0;
  if (!__any_sync(0xffffffffu, wa | wb | !ph.fast)) return;
  const double a0 = a.q0 * dxinv, aa = a.qa * dxinv, ab = a.qb * dxinv, ac = a.qc * dxinv,
               ad = a.qd * dxinv;
  const double b0 = b.q0 * dxinv, ba = b.qa * dxinv, bb = b.qb * dxinv, bc = b.qc * dxinv,
               bd = b.qd * dxinv;
  const double ma = (aa + ab + ac + ad) / 4.0, mb = (ba + bb + bc + bd) / 4.0;
  bool xa, xb;
  const double fa =
      face_fast(ya0 - ya1, ha, a0 * a0 + ma * ma, a0 + 0.0, ph.dx, ph.rh, ph.rl, ph.gdt, ph.fn, xa);
  const double fb =
      face_fast(yb0 - yb1, hb, b0 * b0 + mb * mb, b0 + 0.0, ph.dx, ph.rh, ph.rl, ph.gdt, ph.fn, xb);
  qa = wa ? fa : 0.0;
  qb = wb ? fb : 0.0;
  if (__any_sync(0xffffffffu, (xa & wa) | (xb & wb) | !ph.fast)) {
    qa = face_any64(a.z0, a.h0, a.z1, a.h1, a0, aa, ab, ac, ad, ea, ph.fast, ph.dx, ph.rh, ph.rl,
                    ph.gdt, ph.fn, ph.depth_thresh, ph.max_hflow, ph.nodata);
    qb = face_any64(b.z0, b.h0, b.z1, b.h1, b0, ba, bb, bc, bd, eb, ph.fast, ph.dx, ph.rh, ph.rl,
                    ph.gdt, ph.fn, ph.depth_thresh, ph.max_hflow, ph.nodata);
  }
}

// Edge faces, out of line (a few lanes a step).
static __device__ __noinline__ float edge_out(float h, float z, float sign, float g, float dx,
                                              float nodata) {
  return out_free(h, z, sign, g, dx, nodata);
}
static __device__ __noinline__ float edge_west(float h0, float z0, float h1, float z1, float g,
                                               float dx, float nodata) {
  return west_free(h0, z0, h1, z1, g, dx, nodata);
}
__device__ inline double edge_out(double h, double z, double sign, double g, double dx,
                                  double nodata) {
  return out_free64(h, z, sign, g, dx, nodata);
}
__device__ inline double edge_west(double h0, double z0, double h1, double z1, double g, double dx,
                                   double nodata) {
  return west_free64(h0, z0, h1, z1, g, dx, nodata);
}

// Special cells.  What their sources and boundaries are worth at a step's time
// is worked out while the blocks exchange (the time is known then, dt is not
// yet) and kept in shared memory, for bands of up to these many of each; in
// the march it would hold up the band, and with it every other, by the few
// thousand cycles of a hydrograph's look-up.  Larger bands look up as they go.
constexpr int kBandSpecials = 128;
constexpr int kBandSources = 256;

// interpolate_bc_value of source s / boundary q at t (see apply_sources and
// bc_depth).
static __device__ __noinline__ double source_value(const StepParams& p, int s, double t) {
  if (p.src_type[s] == AF_BC_QFIX) return p.src_value[s];
  const int o = p.src_off[s];
  return interp_series(p.src_times + o, p.src_vals + o, p.src_off[s + 1] - o, p.src_value[s], t,
                       p.src_sorted[s] != 0);
}
template <typename T>
static __device__ __noinline__ T boundary_depth(const StepParams& p, int q, double t) {
  return bc_depth<T>(q,
                     SeriesTable{p.bc_type, p.bc_value, p.bc_off, p.bc_times, p.bc_vals,
                                 p.bc_sorted},
                     t);
}
// One source's volume into a cell (apply_sources, src/main.cpp:253-259).
template <typename T>
__device__ inline T add_source(T h, double v, double dx, double dA, double dt) {
  const double ps = v * dx * dt / dA;
  h = h + T(ps);
  if (h < T(0)) h = T(0);
  return h;
}
// A special cell's new depth: its sources, the update, its boundary depth.  `e`
// is its entry; src (by source) and bc its band's values, or null.
template <typename T>
static __device__ __noinline__ T special_cell(const StepParams& p, const StepScal<T>& sc,
                                              const SpecCell* e, const double* src, const T* bc,
                                              T h, T qw, T qe, T qn, T qs, bool rain) {
  for (int s = e->s0; s < e->s1; s++)
    h = add_source(h, src ? src[s] : source_value(p, s, sc.t), p.dx, p.dA, sc.dt);
  h = cell_update(h, qw, qe, qn, qs, rain, sc);
  if (e->bc >= 0) h = bc ? *bc : boundary_depth<T>(p, e->bc, sc.t);
  return h;
}

template <typename T>
__global__ void __launch_bounds__(ResidentShape<T>::threads, 1)
    k_resident(const __grid_constant__ StepParams p, const __grid_constant__ ResidentParams rp) {
  constexpr int NT = ResidentShape<T>::threads, NW = NT / 32;
  constexpr int HW = ResidentShape<T>::halo_words;
  extern __shared__ __align__(16) unsigned char s_mem[];
  static_assert(NW == kLoopWarps, "one warp, one hand-in");
  __shared__ LoopShared<T> S;
  __shared__ int s_nseg;
  __shared__ double s_src[kBandSources];  // the band's sources' values at the step's time
  __shared__ T s_bc[kBandSpecials];       // and its special cells' boundary depths
  __shared__ SpecCell s_spec[kBandSpecials];
  SimCtl* ctl = p.ctl;
  int lane;  // read once: not recomputed from the thread index in the loop
  asm volatile("mov.u32 %0, %%laneid;" : "=r"(lane));
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
  const int nb = gridDim.x, b = blockIdx.x;
  const int nx = p.nx, ny = p.ny, P = p.P, W = nx + 1;
  // Band of rows: the first ny % nb bands have one row more.
  const int base = ny / nb, more = ny % nb;
  const int r0 = b * base + min(b, more);
  const int nr = base + (b < more ? 1 : 0);
  // Local row l of H, Z and Qx is grid row r0 - 1 + l, of Qy the faces north
  // of grid row r0 + l.  A row's last column (nx) is H's, Z's and Qy's next
  // row's left neighbour of column 0, never used.
  const int nH = (rp.nr_max + 2) * W, nY = (rp.nr_max + 1) * W;
  T* const H0 = reinterpret_cast<T*>(s_mem) + 1;
  T* const Z = H0 + 2 * nH;
  T* const X0 = Z + nH;
  T* const Y0 = X0 + 2 * nH + 1;
  const int nsx = (nx + 31) / 32;
  int4* const segs = reinterpret_cast<int4*>(
      s_mem + ((((size_t)W * (7 * rp.nr_max + 12) + 4) * sizeof(T) + 15) & ~(size_t)15));
  uint2* const at32 = reinterpret_cast<uint2*>(segs + nsx * rp.gy);  // {mask, first entry}

  // ---- the loop's start, the same in every block
  const double t_start = ctl->t;
  int n = 0;  // steps of this launch
  if (tid == 0) {
    start_clock(p, rp.loop, S);
    // The band's marches: strip, first and last row.
    int q = 0;
    for (int gi = 0; gi < rp.gy; gi++) {
      const int ra = nr * gi / rp.gy, rb = nr * (gi + 1) / rp.gy;
      for (int x = 0; x < nsx && ra < rb; x++) segs[q++] = make_int4(x, ra, rb, 0);
    }
    s_nseg = q;
  }
  __syncthreads();
  // The band's special cells and (consecutive, as cells are) their sources.
  const int e0 = rp.row_off[r0], ne = rp.row_off[r0 + nr] - e0;
  const int src0 = ne > 0 ? rp.row_spec[e0].s0 : 0;
  const int nsrc = ne > 0 ? rp.row_spec[e0 + ne - 1].s1 - src0 : 0;
  const bool cached = ne <= kBandSpecials && nsrc <= kBandSources;
  auto band_values = [&](double at) {
    for (int k = tid; k < nsrc; k += NT) s_src[k] = source_value(p, src0 + k, at);
    for (int e = tid; e < ne; e += NT) {
      const int q = rp.row_spec[e0 + e].bc;
      if (q >= 0) s_bc[e] = boundary_depth<T>(p, q, at);
    }
  };
  if (!S.done) {
    const int par0 = S.par0;
    const T* gH = static_cast<const T*>(p.H[par0]);
    const T* gZ = static_cast<const T*>(p.DEM);
    const T* gX = static_cast<const T*>(p.Qx[par0]);
    const T* gY = static_cast<const T*>(p.Qy[par0]);
    for (int l = warp; l < nr + 2; l += NW) {
      const int r = r0 - 1 + l;
      const bool in = r >= 0 && r < ny;
      for (int i = lane - 1; i <= nx; i += 32) {
        const long long g = (long long)r * P + i;
        const bool cell = in && i >= 0 && i < nx;
        if (i < nx) {
          H0[l * W + i] = cell ? gH[g] : T(0);
          H0[nH + l * W + i] = T(0);
          Z[l * W + i] = cell ? gZ[g] : T(0);
        }
        if (i >= 0) {
          X0[l * W + i] = in ? gX[g] : T(0);
          X0[nH + l * W + i] = T(0);
        }
        if (l <= nr && i < nx) {
          Y0[l * W + i] = i >= 0 ? gY[g + P] : T(0);
          Y0[nY + l * W + i] = T(0);
        }
      }
    }
    for (int k = tid; k < nr * nsx; k += NT) {
      const int r = r0 + k / nsx, c0 = k % nsx * 32;
      int lo = rp.row_off[r], hi = rp.row_off[r + 1];  // first entry at or past column c0
      const int end = hi;
      while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (rp.row_spec[mid].col < c0) lo = mid + 1;
        else hi = mid;
      }
      unsigned m = 0u;
      for (int e = lo; e < end && rp.row_spec[e].col < c0 + 32; e++)
        m |= 1u << (rp.row_spec[e].col - c0);
      at32[k] = make_uint2(m, (unsigned)lo);
    }
    if (cached) {
      for (int e = tid; e < ne; e += NT) s_spec[e] = rp.row_spec[e0 + e];
      band_values(t_start);
    }
  }
  __syncthreads();

  const int nseg = s_nseg;
  bool failed = false;
#pragma unroll 1
  while (!S.done) {
    const unsigned tag = S.tag0 + (unsigned)n;
    const int buf = (n & 1);
    const StepScal<T>& sc = S.sc;  // warp 0 rewrites it past the march's barrier
    const T* const H = H0 + buf * nH;
    T* const Hn = H0 + (buf ^ 1) * nH;
    const T* const X = X0 + buf * nH;
    T* const Xn = X0 + (buf ^ 1) * nH;
    const T* const Y = Y0 + buf * nY;
    T* const Yn = Y0 + (buf ^ 1) * nY;
    const Phys<T> ph = sc.ph;
    const T dxinv = sc.dxinvT;
    const bool mass = sc.mass, rain_on = sc.rain_on;
    uint4* const my_halo = rp.halo + ((size_t)(buf * nb + b) * 2) * W * HW;
    T m = T(-FLT_MAX);
    double v = 0.0, a = 0.0;
#pragma unroll 1
    for (int seg = warp; seg < nseg; seg += NW) {
      const int4 sg = segs[seg];
      const int sx = sg.x, ra = sg.y, rb = sg.z;
      const int c = sx * 32 + lane;
      const int cc = min(c, nx - 1);
      const bool own = c < nx, east = c == nx - 1;
      // Faces above row ra (their own columns), and on the strip's east side
      // of row ra + lane.
      int k = (ra + 1) * W + cc, g = ra * W + cc;
      T h = H[k], z = Z[k], x0 = X[k], x1 = X[k + 1], y0 = Y[g];
      T qn, qE;
      {
        const int ce = min(sx * 32 + 32, nx - 1);
        const int re = min(ra + lane, rb - 1);
        const int ke = (re + 1) * W + ce, ge = re * W + ce;
        two_faces(FaceIn<T>{Z[ke - 1], H[ke - 1], Z[ke], H[ke], X[ke], Y[ge - 1], Y[ge],
                            Y[ge + W - 1], Y[ge + W]},
                  FaceIn<T>{Z[k - W], H[k - W], z, h, y0, X[k - W], X[k + 1 - W], x0, x1}, dxinv,
                  sx < nsx - 1, r0 + ra > 0, ph, qE, qn);
      }
      if (r0 + ra == 0) qn = p.nf ? edge_out(h, z, T(-1), ph.g, ph.dx, ph.nodata) : T(0);
      if (ra == 0 && own) Yn[g] = qn;  // further down the group above stores it
      T hW = H[k - 1], zW = Z[k - 1], yW = Y[g - 1];
      const bool full = sx > 0 && sx < nsx - 1;  // no edge column, every lane owns a cell
#pragma unroll 1
      for (int r = ra; r < rb; r++) {
        const T hN = H[k + W], zN = Z[k + W], x0N = X[k + W], x1N = X[k + W + 1];
        const T hNW = H[k + W - 1], zNW = Z[k + W - 1];
        const T s0 = Y[g + W], sW = Y[g + W - 1];
        const unsigned specials = at32[r * nsx + sx].x;
        const bool south = r0 + r + 1 < ny;
        T qw, qs;
        two_faces(FaceIn<T>{zW, hW, z, h, x0, yW, y0, sW, s0},
                  FaceIn<T>{z, h, zN, hN, s0, x0, x1, x0N, x1N}, dxinv, true, south, ph, qw, qs);
        T qe = __shfl_down_sync(0xffffffffu, qw, 1);
        const T qEr = __shfl_sync(0xffffffffu, qE, r - ra);
        if (lane == 31) qe = qEr;
        const bool valid = z != ph.nodata;
        T hn;
        if (full & south & (specials == 0u)) {
          hn = cell_update(h, qw, qe, qn, qs, rain_on && valid, sc);
        } else {
          if (!south) qs = p.sf ? edge_out(h, z, T(1), ph.g, ph.dx, ph.nodata) : T(0);
          if (sx == 0) {
            if (lane == 0)
              qw = p.wf ? edge_west(h, z, H[k + 1], Z[k + 1], ph.g, ph.dx, ph.nodata) : T(0);
          }
          if (east) {
            qe = p.ef ? edge_out(h, z, T(1), ph.g, ph.dx, ph.nodata) : T(0);
            Xn[k + 1] = qe;
            if ((r == 0) & (b > 0)) halo_put(my_halo + (size_t)nx * HW, T(0), qe, tag);
            if ((r == nr - 1) & (b < nb - 1))
              halo_put(my_halo + (size_t)(W + nx) * HW, T(0), qe, tag);
          }
          hn = cell_update(h, qw, qe, qn, qs, rain_on && valid, sc);
          if ((specials >> lane) & 1u) {
            const int e = (int)at32[r * nsx + sx].y + __popc(specials & ((1u << lane) - 1u));
            hn = cached ? special_cell<T>(p, sc, &s_spec[e - e0], s_src - src0, &s_bc[e - e0], h, qw,
                                          qe, qn, qs, rain_on && valid)
                        : special_cell<T>(p, sc, &rp.row_spec[e], nullptr, nullptr, h, qw, qe, qn,
                                          qs, rain_on && valid);
          }
        }
        if (own) {
          Hn[k] = hn;
          Xn[k] = qw;
          Yn[g + W] = qs;
          if (valid) m = hn > m ? hn : m;  // a NaN never wins
        }
        if ((r == 0) | (r == nr - 1) | mass) {
          if (own) {
            if ((r == 0) & (b > 0)) halo_put(my_halo + (size_t)c * HW, hn, qw, tag);
            if ((r == nr - 1) & (b < nb - 1))
              halo_put(my_halo + (size_t)(W + c) * HW, hn, qw, tag);
            if (mass) {
              const double hv = (double)hn;
              v += hv * p.dA;
              if (hv > 0.01) a += p.dA;
            }
          }
        }
        k += W;
        g += W;
        h = hN;
        z = zN;
        hW = hNW;
        zW = zNW;
        x0 = x0N;
        x1 = x1N;
        y0 = s0;
        yW = sW;
        qn = qs;
      }
    }
    hand_in(S, warp, m, v, a, mass);
    // The next step's time, read before the barrier: past it warp 0 rewrites sc.
    const double at = sc.t + sc.dt;
    __syncthreads();
    if (warp == 0) {
      step_clock<T, false>(p, rp.loop, S, tag, n);
    } else {
      if constexpr (kLateNs > 0) __nanosleep(kLateNs);
      if (cached && ne > 0) {
        for (int k = tid - 32; k < nsrc; k += NT - 32) s_src[k] = source_value(p, src0 + k, at);
        for (int e = tid - 32; e < ne; e += NT - 32)
          if (s_spec[e].bc >= 0) s_bc[e] = boundary_depth<T>(p, s_spec[e].bc, at);
      }
      // ---- the neighbours' rows
      const uint4* const above = rp.halo + ((size_t)(buf * nb + b - 1) * 2 + 1) * W * HW;
      const uint4* const below = rp.halo + ((size_t)(buf * nb + b + 1) * 2) * W * HW;
      bool ok = true;
      constexpr int K = 4;  // columns in flight per thread
      for (int k0 = tid - 32; k0 < 2 * W; k0 += K * (NT - 32)) {
        T hh[K], qq[K];
        bool got[K], want[K];
#pragma unroll
        for (int u = 0; u < K; u++) {
          const int k = k0 + u * (NT - 32);
          want[u] = k < W ? b > 0 : (k < 2 * W && b < nb - 1);
          got[u] = !want[u];
          hh[u] = qq[u] = T(0);
        }
        for (int w = 0; w < (int)kRingWaitLimit && !(got[0] & got[1] & got[2] & got[3]); w++) {
#pragma unroll
          for (int u = 0; u < K; u++) {
            const int k = k0 + u * (NT - 32);
            if (!got[u])
              got[u] = halo_get(k < W ? above + (size_t)k * HW : below + (size_t)(k - W) * HW,
                                hh[u], qq[u], tag);
          }
        }
#pragma unroll
        for (int u = 0; u < K; u++) {
          const int k = k0 + u * (NT - 32);
          ok &= got[u];
          if (want[u]) {
            const int l = k < W ? 0 : nr + 1, i = k < W ? k : k - W;
            if (i < nx) Hn[l * W + i] = hh[u];
            Xn[l * W + i] = qq[u];
          }
        }
      }
      if (!ok) S.fail = 1;
    }
    __syncthreads();
    n++;
    if (S.fail) {
      failed = true;
      break;
    }
  }

  // ---- the state back to its planes, and the control block
  if (failed && tid == 0) atomicExch(&ctl->status, 2);
  const int par = S.par0 ^ (n & 1);
  if (!failed && n > 0) {
    const int buf = (n & 1);
    T* gH = static_cast<T*>(p.H[par]);
    T* gX = static_cast<T*>(p.Qx[par]);
    T* gY = static_cast<T*>(p.Qy[par]);
    for (int l = warp; l < nr + (b == nb - 1 ? 1 : 0); l += NW) {
      const long long g = (long long)(r0 + l) * P;
      for (int i = lane; i <= nx; i += 32) {
        if (l < nr) {
          if (i < nx) gH[g + i] = H0[buf * nH + (l + 1) * W + i];
          gX[g + i] = X0[buf * nH + (l + 1) * W + i];
        }
        if (i < nx) gY[g + i] = Y0[buf * nY + l * W + i];
      }
    }
  }
  if (b == 0 && tid == 0) stop_clock(p, rp.loop, S, S.par0, S.tag0, n);
}

}  // namespace af
