// Reference order (the in-place lexicographic sweep of central_diff5,
// src/solver.cc:112-224 of the reference) as a pipeline of tiles.
// This translation unit is compiled with -fmad=false; the few explicit FMAs
// below have an exact product, so every value rounds as the reference's.
//
// In lexicographic order every read at offset -1 / -2 sees this sweep's value
// and every read at +1 / +2 the previous one.  Columns of constant (y, z) are
// grouped in tiles of kTileY x kTileZ; at its step t a tile updates the voxel
// x = t - ly - lz of each of its columns, so a -1 / -2 neighbour inside the
// tile was updated one / two steps before, and its values lie in a ring of
// shared memory.  Tiles take tickets in the order of pm_wave.h and wait only for
// values of the tiles below them in y and z, whose tickets are smaller and so
// running or done: no co-residency is needed.  Those values are handed over in
// an exchange copy of the fields, filled with kEmpty before the sweep: a tile
// writes its outer columns' values there as it goes, and the next one polls
// until they differ from kEmpty.  No flag and no fence is involved, since the
// value itself is what arrives.  A tile reads old values of the tiles above it
// with plain loads, and their owners overwrite them with plain stores; no fence
// orders the two.  What does is that the stored value is computed from a value
// of the exchange which the reading tile computed from the old one: every old
// value an update uses enters the velocity or pressure handed to the column it
// came from, directly or through that column's neighbour.  A load that returned
// the later store would depend on itself.  Programs may not produce such values
// under PTX's memory model (its no-thin-air rule), and an SM does not issue a
// store before the loads its data comes from have returned; but the plain
// accesses are a race by the letter of that model, so this rests on the data
// dependence and not on synchronisation.  Every wait is bounded; when one runs out the sweep finishes without
// waiting and the host finds the error flag.
//
// What bounds it: GB300's FP64 pipe takes 64 clocks per instruction of a warp
// whatever its active lanes (measured: 63.9, 76 with a warp on each of an SM's
// four), and an update is a chain of such instructions: the time of a sweep is
// about (nx + ny + nz) steps of one update.  So a voxel's velocity components
// are three lanes of a warp (19 FP64 instructions; one lane per voxel has about
// 85 with the case branches and the divisions), and its pressure (8) is a lane
// of another warp, which runs while the velocities of the next step are under
// way: they need it only near the end.  Three velocity warps of eight columns
// and the pressure warp put one warp on each FP64 pipe.  Old values are loaded
// two steps ahead.  Three warps ask for the neighbour tiles' velocities up to
// two steps ahead in turn (one warp in step with the others takes 1.9 us a step
// of 132 tiles instead of 1.3), one for their pressures.  Progress flags behind
// a fence instead of the exchange cost 620 clocks a step: the fence holds up
// the tile's loads.
// A 48x48x64 pore takes 0.19 ms a sweep, against 1.38 ms with one grid-wide
// barrier per hyperplane and a voxel per lane.
#include <atomic>

#include "pm_internal.h"
#include "pm_stencil.cuh"
#include "pm_wave.h"

namespace pm {

namespace {

constexpr int kTileY = 4, kTileZ = 6;  // columns of a tile, 8 a velocity warp
constexpr int kRingY = kTileY + 2, kRingZ = kTileZ + 2;
constexpr int kSlot = kRingZ * kRingY * 4;  // u, v, w, p of every column of a step
// warps: velocities (0 ..), pressures, neighbours' pressures and velocities
constexpr int kPressure = kTileY * kTileZ / 8, kFetchP = kPressure + 1, kFetchV = kPressure + 2;
constexpr int kFetchers = 3;
constexpr int kWaveThreads = 32 * (kFetchV + kFetchers);
constexpr int kBelow = kTileY + kTileZ;             // columns next to the tile
constexpr int kFetched = 2 * kBelow * 3;            // velocities fetched a step
constexpr int kFetchLane = (kFetched + 31) / 32;
static_assert(kTileY * kTileZ % 8 == 0 && kTileY * kTileZ <= 32 && kBelow <= 32, "");
constexpr int kWavePolls = 1 << 22;  // seconds, against a sweep of microseconds
constexpr unsigned long long kEmpty = ~0ull;         // a NaN no operation returns
constexpr unsigned long long kOtherNaN = ~0ull << 51;

std::atomic<int> g_wave_fail{0};

__device__ __forceinline__ unsigned long long ld_exchange(const double* p) {
  unsigned long long v;
  asm volatile("ld.relaxed.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void st_exchange(double* p, double v) {
  unsigned long long b = (unsigned long long)__double_as_longlong(v);
  if (b == kEmpty) b = kOtherNaN;
  asm volatile("st.relaxed.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(b) : "memory");
}

// The pressures of a step are in the ring: the pressure warp and the one that
// fetches the neighbours' arrive, the velocity warps wait before they read them.
constexpr int kPressureCount = 32 * (kPressure + 2);
__device__ __forceinline__ void pressure_arrive() {
  asm volatile("bar.arrive 1, %0;" ::"n"(kPressureCount) : "memory");
}
__device__ __forceinline__ void pressure_wait() {
  asm volatile("bar.sync 1, %0;" ::"n"(kPressureCount) : "memory");
}

// Coefficients of the wall stencils (get_2nd_derivation, src/solver.cc:57-91)
// per case: of the centre, of the exact product (1 or 2) and of the last one;
// and the cases of a code byte, four bits an axis (solid and halo codes, whose
// results are dropped, as interior ones).
__device__ __forceinline__ void fill_tables(double (*tab)[4], unsigned short* cases) {
  const int cs = threadIdx.x;
  if (cs < 8) {
    tab[cs][0] = cs == 1 ? -8.0 : (cs <= 3 ? -16.0 / 3.0 : (cs <= 5 ? -5.0 : -2.0));
    tab[cs][1] = cs <= 5 ? 2.0 : 1.0;
    tab[cs][2] = cs <= 3 ? 8.0 / 3.0 : (cs <= 5 ? -(1.0 / 5.0) : 1.0);
    tab[cs][3] = 0.0;
  }
  for (int c = threadIdx.x; c < 256; c += blockDim.x) {
    int cx, cy, cz;
    decode_cases(c >= 1 && c <= 216 ? c : 216, cx, cy, cz);
    cases[c] = (unsigned short)(cx | cy << 4 | cz << 8);
  }
}

// A case and its coefficients.
struct CaseLane {
  int cs;
  double cm, ca, cb;
};

__device__ __forceinline__ CaseLane case_lane(int cs, const double (*tab)[4]) {
  return {cs, tab[cs][0], tab[cs][1], tab[cs][2]};
}

// d2_exact in one form for all cases, so that lanes of different cases run
// together: (A-term + first) + second, the products rounded as there.  Terms a
// case does not have are -0.0, which leaves every sum (and its sign) as it is.
__device__ __forceinline__ double d2_lane(const CaseLane& k, double ll, double l, double m,
                                          double r, double rr) {
  const int cs = k.cs;
  const double A = cs <= 3 ? -0.0 : (cs == 4 ? r : l);
  const double B = cs == 4 ? rr : (cs == 5 ? ll : (cs == 3 ? l : r));
  const double M = k.cm * m;
  double P = k.cb * B;
  if (cs == 1) P = -0.0;
  const double first = cs == 5 ? P : M, second = cs == 5 ? M : P;
  return __fma_rn(k.ca, A, first) + second;  // ca is 1 or 2: exact product
}

template <int SOLVER>
__device__ __forceinline__ double velocity_lane(double c, double visc, double pm, double pc,
                                                bool lsolid) {
  const double dp = lsolid ? 0. : -pm + pc;
  if (SOLVER == 3) return (1.0 - kOmega) * c + kOmega * (-dp + visc) * kDt;
  const double v = c + (-dp + visc) * kDt;
  return lsolid ? 0.0 : v;
}

// X: the exchange copy of the fields (same layout); ticket: all ones before
// the first block; err: set when a wait ran out.
template <int SOLVER>
__global__ void __launch_bounds__(kWaveThreads)
    k_wave(Fields<double> f, Fields<double> X, const uint8_t* codes, Grid g, int tiles_y,
           int tiles_z, int* ticket, int* err, int polls) {
  __shared__ double ring[4][kSlot];
  __shared__ double tab[8][4];
  __shared__ unsigned short cases[256];
  __shared__ int sh_tile[2];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0)
    wave_tile(atomicAdd(ticket, 1) + 1, tiles_y, tiles_z, sh_tile[0], sh_tile[1]);
  fill_tables(tab, cases);
  for (int i = threadIdx.x; i < 4 * kSlot; i += blockDim.x) (&ring[0][0])[i] = 0.0;
  __syncthreads();
  const int tY = sh_tile[0], tZ = sh_tile[1];
  const int y0 = tY * kTileY, z0 = tZ * kTileZ;
  const int ncy = min(kTileY, g.ny - y0), ncz = min(kTileZ, g.nz - z0);
  const int t_last = g.nx - 1 + ncy - 1 + ncz - 1;
  const long long px = g.px64, pl = g.pl64;
  // In main step t (a barrier ends each) the velocities of step t, the
  // pressures of step t - 1 and the neighbours' values of step t are made.
  // Steps -2 and -1 of a column bring its low x halo into the ring.

  if (warp < kPressure) {
    // ---- velocities: lane = 4 * column + component, the fourth idle
    const int k = lane & 3, c8 = 8 * warp + (lane >> 2), ly = c8 % kTileY, lz = c8 / kTileY;
    const bool col = k < 3 && ly < ncy && lz < ncz;
    const int y = col ? y0 + ly : y0, z = col ? z0 + lz : z0;
    double* F = k == 0 ? f.u : k == 1 ? f.v : f.w;
    const long long row = (long long)(z + 2) * pl + (long long)(y + 2) * px + 2;
    double* out = (k == 0 ? X.u : k == 1 ? X.v : X.w) + row;
    const bool hand = col && (ly >= kTileY - 2 || lz >= kTileZ - 2);
    const uint8_t* crow = codes + (long long)(z + 2) * g.plc + (long long)(y + 2) * g.pxc + 2;
    // strides of the component's axes in the fields and in the ring
    const long long s0 = k == 1 ? px : k == 2 ? pl : 1;
    const long long s1 = k == 0 ? px : k == 1 ? pl : 1;
    const long long s2 = k == 0 ? pl : k == 2 ? px : 1;
    const int d0 = k == 1 ? 4 : k == 2 ? 4 * kRingY : 0;
    const int d1 = k == 0 ? 4 : k == 1 ? 4 * kRingY : 0;
    const int d2 = k == 0 ? 4 * kRingY : k == 2 ? 4 : 0;
    const int o = ((lz + 2) * kRingY + ly + 2) * 4 + k;
    // bits of the component's own axis and of the next two in `cases`
    const int b0 = 4 * (k % 3), b1 = 4 * ((k + 1) % 3), b2 = 4 * ((k + 2) % 3);
    struct Old {
      double c, pc, r0, r1, rr1, r2, rr2;
      int code;
    };
    // old values of step t: nobody writes them before that step
    auto load = [&](int t) {
      const int xl = min(max(t - ly - lz, -2), g.nx - 1);
      const double* a = F + row + xl;
      Old v;
      v.code = crow[xl];
      v.c = a[0];
      v.pc = f.p[row + xl];
      v.r0 = a[s0];
      v.r1 = a[s1];
      v.rr1 = a[2 * s1];
      v.r2 = a[s2];
      v.rr2 = a[2 * s2];
      return v;
    };
    // what step t needs of its code
    struct Prep {
      CaseLane k1, k2;
      bool lsolid, upd, any;
    };
    auto prepare = [&](int t, const Old& v) {
      const int x = t - ly - lz;
      const unsigned cs = cases[v.code];
      Prep p;
      p.k1 = case_lane((cs >> b1) & 7, tab);
      p.k2 = case_lane((cs >> b2) & 7, tab);
      p.lsolid = left_solid((cs >> b0) & 7);
      p.upd = col && x >= 0 && x < g.nx && v.code != 0;
      p.any = __any_sync(0xffffffffu, p.upd);
      return p;
    };
    Prep prep;
    // step t on cur; loads step t + 2 into ahead, prepares step t + 1 (next)
    auto step = [&](int t, const Old& cur, const Old& next, Old& ahead) {
      const int x = t - ly - lz;
      const Prep p = prep;
      double v = cur.c;
      if (p.any) {
        const double* r1 = ring[(t + 3) & 3] + o;  // step t - 1
        const double* r2 = ring[(t + 2) & 3] + o;  // step t - 2
        const double l0 = r1[-d0], l1 = r1[-d1], l2 = r1[-d2];
        const double ll1 = r2[-2 * d1], ll2 = r2[-2 * d2];
        const double e1 = d2_lane(p.k1, ll1, l1, cur.c, cur.r1, cur.rr1);
        const double e2 = d2_lane(p.k2, ll2, l2, cur.c, cur.r2, cur.rr2);
        const double along = __fma_rn(-2.0, cur.c, l0) + cur.r0;
        const double visc_re = along + e1 + e2;
        double visc = div_re_step(visc_re);
        ahead = load(t + 2);
        prep = prepare(t + 1, next);
        if (p.upd && !div_re_holds(visc_re)) visc = div_re_general(visc_re);
        pressure_wait();
        const double vn = velocity_lane<SOLVER>(cur.c, visc, r1[3 - k - d0], cur.pc, p.lsolid);
        if (p.upd) {
          v = vn;
          F[row + x] = v;
        }
      } else {
        ahead = load(t + 2);
        prep = prepare(t + 1, next);
        pressure_wait();
      }
      if (k < 3) ring[t & 3][o] = v;  // (t + 4) & 3 == t & 3 for t = -2, -1
      if (hand && x >= 0 && x < g.nx) st_exchange(out + x, v);
      __syncthreads();
    };
    // loads two steps ahead, in three register sets the steps use in turn
    Old o0 = load(-2), o1 = load(-1), o2;
    prep = prepare(-2, o0);
    for (int t = -2;; t += 3) {
      step(t, o0, o1, o2);
      if (t > t_last) break;
      step(t + 1, o1, o2, o0);
      if (t + 1 > t_last) break;
      step(t + 2, o2, o0, o1);
      if (t + 2 > t_last) break;
    }
  } else if (warp == kPressure) {
    // ---- pressures of the step before, a lane per column
    const int ly = lane % kTileY, lz = lane / kTileY;
    const bool col = lz < kTileZ && ly < ncy && lz < ncz;
    const int y = col ? y0 + ly : y0, z = col ? z0 + lz : z0;
    const long long row = (long long)(z + 2) * pl + (long long)(y + 2) * px + 2;
    const bool hand = col && (ly >= kTileY - 2 || lz >= kTileZ - 2);
    const uint8_t* crow = codes + (long long)(z + 2) * g.plc + (long long)(y + 2) * g.pxc + 2;
    const int o = ((min(lz, kTileZ - 1) + 2) * kRingY + ly + 2) * 4;
    struct Old {
      double p, ub, vb, wb, ua, va, wa;
      int code;
    };
    auto load = [&](int t) {
      const int xl = min(max(t - ly - lz, -2), g.nx - 1);
      const long long a = row + xl;
      Old v;
      v.code = crow[xl];
      v.p = f.p[a];
      v.ub = f.u[a + 1];
      v.vb = f.v[a + px];
      v.wb = f.w[a + pl];
      if (SOLVER == 1) {
        v.ua = f.u[a];
        v.va = f.v[a];
        v.wa = f.w[a];
      }
      return v;
    };
    auto step = [&](int t, const Old& cur, Old& ahead) {
      const int x = t - ly - lz;
      const bool upd = col && x >= 0 && x < g.nx && cur.code != 0;
      double* r = ring[t & 3] + o;
      double v = cur.p;
      if (__any_sync(0xffffffffu, upd)) {
        // the divergence: plus-side value minus the new (solver 1: old) one
        const double ua = SOLVER == 1 ? cur.ua : r[0];
        const double va = SOLVER == 1 ? cur.va : r[1];
        const double wa = SOLVER == 1 ? cur.wa : r[2];
        const double v_sum = (cur.wb - wa + cur.vb - va + cur.ub - ua);
        const double pn = cur.p - kC2 * v_sum * kDt;
        if (upd) {
          v = pn;
          f.p[row + x] = v;
        }
      }
      if (lz < kTileZ) r[3] = v;
      pressure_arrive();
      if (hand && x >= 0 && x < g.nx) st_exchange(X.p + row + x, v);
      ahead = load(t + 3);
      __syncthreads();
    };
    Old o0 = load(-2), o1 = load(-1), o2 = load(0);
    pressure_arrive();  // nothing precedes step -2
    __syncthreads();
    for (int t = -2;; t += 3) {
      step(t, o0, o0);
      if (t >= t_last) break;
      step(t + 1, o1, o1);
      if (t + 1 >= t_last) break;
      step(t + 2, o2, o2);
      if (t + 2 >= t_last) break;
    }
  } else if (warp == kFetchP) {
    // ---- the neighbours' pressures of the step before: one column below each
    // of the tile's in y and in z, from the exchange or (at a face) the halo
    const bool below_y = lane < kTileZ;
    const int ly = below_y ? -1 : min(lane - kTileZ, kTileY - 1), lz = below_y ? lane : -1;
    const bool used = lane < kBelow && ly < ncy && lz < ncz;
    const bool poll = below_y ? tY > 0 : tZ > 0;
    const double* src = (poll ? X.p : f.p) +
                        (used ? (long long)(z0 + lz + 2) * pl + (long long)(y0 + ly + 2) * px + 2
                              : 0);
    const int dst = ((lz + 2) * kRingY + ly + 2) * 4 + 3;
    unsigned long long v = kEmpty;
    for (int m = -2; m <= t_last + 1; ++m) {
      int x = m - 1 - ly - lz;
      bool need = m > -2 && used && x >= 0 && x < g.nx;
      for (int i = 1; __any_sync(0xffffffffu, need && poll && v == kEmpty); ++i) {
        if (i > polls) {
          if (lane == 0) atomicExch(err, 1);
          polls = 0;
          break;
        }
        if (need) v = ld_exchange(src + x);
      }
      if (need) ring[(m + 3) & 3][dst] = __longlong_as_double((long long)v);
      pressure_arrive();
      ++x;  // ask for the next one ahead of time
      if (used && x >= 0 && x < g.nx) v = ld_exchange(src + x);
      __syncthreads();
    }
  } else {
    // ---- the neighbours' velocities: two columns below each of the tile's.
    // Each of the fetching warps takes every third step and asks for its values
    // up to two steps ahead.
    const double* src[kFetchLane];
    int dst[kFetchLane], shift[kFetchLane];
    bool poll[kFetchLane], used[kFetchLane];
    for (int j = 0; j < kFetchLane; ++j) {
      const int i = lane + 32 * j, c = i < kFetched ? i / 3 : 0, k = i < kFetched ? i % 3 : 0;
      const bool below_y = c < 2 * kTileZ;
      const int ly = below_y ? -1 - (c & 1) : (c - 2 * kTileZ) >> 1;
      const int lz = below_y ? c >> 1 : -1 - (c & 1);
      used[j] = i < kFetched && ly < ncy && lz < ncz;
      poll[j] = below_y ? tY > 0 : tZ > 0;
      const int y = used[j] ? y0 + ly : y0, z = used[j] ? z0 + lz : z0;
      const Fields<double>& S = poll[j] ? X : f;
      src[j] = (k == 0 ? S.u : k == 1 ? S.v : S.w) + (long long)(z + 2) * pl +
               (long long)(y + 2) * px + 2;
      dst[j] = used[j] ? ((lz + 2) * kRingY + ly + 2) * 4 + k : 0;
      shift[j] = ly + lz;
    }
    unsigned long long v[kFetchLane];
    auto needs = [&](int t, int j) {
      const int x = t - shift[j];
      return used[j] && x >= 0 && x < g.nx;
    };
    auto ask = [&](int t) {
      for (int j = 0; j < kFetchLane; ++j)
        if (needs(t, j)) v[j] = ld_exchange(src[j] + (t - shift[j]));
    };
    auto missing = [&](int t) {
      bool miss = false;
      for (int j = 0; j < kFetchLane; ++j) miss |= needs(t, j) && poll[j] && v[j] == kEmpty;
      return __any_sync(0xffffffffu, miss) != 0;
    };
    int t = -2 + warp - kFetchV;  // the next step of this warp
    if (t < 0) ask(t);
    for (int m = -2; m <= t_last + 1; ++m) {
      if (t == m + 2) {
        ask(t);
      } else if (t == m + 1) {
        if (missing(t)) ask(t);
      } else {
        for (int i = 1; missing(t); ++i) {
          if (i > polls) {  // tell the host, and wait no more
            if (lane == 0) atomicExch(err, 1);
            polls = 0;
            break;
          }
          ask(t);
        }
        for (int j = 0; j < kFetchLane; ++j)
          if (needs(t, j)) ring[t & 3][dst[j]] = __longlong_as_double((long long)v[j]);
        t += kFetchers;
      }
      __syncthreads();
    }
  }
}

}  // namespace

void wave_debug_fail(int on) { g_wave_fail.store(on ? 1 : 0); }

cudaError_t launch_wave(Fields<double> f, const uint8_t* codes, const Grid& g, int solver,
                        double* exchange, int* err, cudaStream_t st) {
  const int ty = (g.ny + kTileY - 1) / kTileY, tz = (g.nz + kTileZ - 1) / kTileZ;
  // exchange: 4 alloc64 doubles as the fields', whose first word no field uses
  static_assert(kXoff64 > 0, "room for the ticket before the first field");
  cudaError_t e = cudaMemsetAsync(exchange, 0xff, 4 * sizeof(double) * (size_t)g.alloc64, st);
  if (e != cudaSuccess) return e;
  double* b = exchange + kXoff64;
  const Fields<double> X = {b, b + g.alloc64, b + 2 * g.alloc64, b + 3 * g.alloc64};
  auto* k = solver == 1 ? k_wave<1> : solver == 2 ? k_wave<2> : k_wave<3>;
  k<<<ty * tz, kWaveThreads, 0, st>>>(f, X, codes, g, ty, tz, (int*)exchange, err,
                                      g_wave_fail.load() ? 1 : kWavePolls);
  count_launches(1);
  if ((e = cudaGetLastError()) != cudaSuccess) return e;
  if ((e = launch_halo64(f, g, st)) != cudaSuccess) return e;
  return launch_reapply64(f.p, codes, g, st);
}

}  // namespace pm
