// Device functions of the compact correction store (pm_compact.cu): shared
// by the single-problem kernels and the batched kernels of the server, so a
// sample computes the same values alone and in a batch.
#pragma once

#include "pm_stencil.cuh"

namespace pm {

// Wrap a neighbour coordinate q = c + d (d in -2..2) on an axis of length n.
// The padded store's halo cell at q holds a copy of the interior voxel one
// period away when that voxel exists (periodic axis, q -+ n inside [0, n)),
// and 0 otherwise (wall axes, and the outer halo cell of an axis of length 1);
// ok becomes false where the padded store holds 0.
__device__ __forceinline__ int wrap(int q, int n, int per, bool& ok) {
  if (q < 0) {
    ok = ok && per && q + n >= 0;
    return q + n;
  }
  if (q >= n) {
    ok = ok && per && q - n < n;
    return q - n;
  }
  return q;
}

// Fluid flags from a neighbourhood case (1 = solid in the reference's
// geometry): left fluid for cases 3, 5, 6; right fluid for 2, 4, 6; the
// second left is used (and fluid) in case 5, the second right in case 4.
__device__ __forceinline__ bool left_fluid(int c) { return c == 3 || c == 5 || c == 6; }
__device__ __forceinline__ bool right_fluid(int c) { return c == 2 || c == 4 || c == 6; }

// The sweep of list position i reads its correction and six neighbour
// positions, two per axis, chosen by the axis' neighbourhood case when the
// compact store is set up:
//   case 1 (both sides solid)         L = zero slot, R = zero slot
//   case 2 (l solid, r fluid, rr solid)  L = zero slot, R = r
//   case 3 (ll solid, l fluid, r solid)  L = l,         R = zero slot
//   case 4 (l solid, r and rr fluid)  L = rr,        R = r
//   case 5 (ll and l fluid, r solid)  L = l,         R = ll
//   case 6 (both sides fluid)         L = l,         R = r
// (a neighbour that is fluid in the geometry but has no stored value -- a
// wall-face halo, the outer halo of an axis of length 1 -- is the zero slot
// too).  The zero slot is position nlist of every correction buffer, which
// holds 0 forever.  In a case-4 or case-5 axis one side is solid, so its slot
// carries the second neighbour the wall stencil needs: six slots cover all
// twelve stencil points.
struct CompactSlots {
  int4 a;  // x L, x R, y L, y R
  int2 b;  // z L, z R
};

// Per-voxel metadata (32 bits): the three neighbourhood cases (3 bits each,
// x in bits 0-2), two plane flags and which +-1 neighbours are fluid.
constexpr unsigned kMetaZFirst = 1u << 9;   // first interior plane: -z pressure reads 0
constexpr unsigned kMetaZLast = 1u << 10;   // last interior plane: own pressure reads 0
constexpr int kMetaFluidShift = 11;         // bits 11 + 2 axis (+1): -side (+side) fluid

__device__ __forceinline__ unsigned make_meta(int cx, int cy, int cz, bool zfirst, bool zlast);

__device__ __forceinline__ unsigned make_meta(int cx, int cy, int cz, bool zfirst, bool zlast) {
  unsigned m = (unsigned)cx | ((unsigned)cy << 3) | ((unsigned)cz << 6);
  if (zfirst) m |= kMetaZFirst;
  if (zlast) m |= kMetaZLast;
  const int c[3] = {cx, cy, cz};
  for (int a = 0; a < 3; ++a) {
    if (left_fluid(c[a])) m |= 1u << (kMetaFluidShift + 2 * a);
    if (right_fluid(c[a])) m |= 1u << (kMetaFluidShift + 2 * a + 1);
  }
  return m;
}

// Packed record of a list position (kernel 13 and the server's sweeps): 16
// bytes instead of the 28 of slots and metadata.  Per axis the positions of the
// two points (F, S) its neighbourhood case uses, as offsets from the position
// itself (a value of its own, in z the offset of the zero slot, where there is
// none):
//   case     1  2  3  4  5  6
//   F        -  -  l  r  l  l
//   S        -  r  -  rr ll r
// x offsets take 14 bits each (a row's fluid voxels), y offsets 16, z offsets
// 28 (the whole list: a periodic z face); bits 0-10 of the first word are the
// cases and the plane flags of the metadata.  A position whose y offsets do
// not fit (a periodic y face of a plane of more than 32,767 fluid voxels) has
// kRecEscape set and its absolute y positions in a table of their own.
constexpr unsigned kRecMeta = 0x7ffu;
constexpr unsigned kRecEscape = 1u << 11;
constexpr int kNoneX = -(1 << 13), kNoneY = -(1 << 15);

__host__ __device__ __forceinline__ bool records_fit(const Grid& g, long long nlist) {
  return g.nx < (1 << 13) && nlist < (1LL << 27) - 1;
}

struct Neighbours {  // list positions of F, S per axis
  int x0, x1, y0, y1, z0, z1;
};

// The points F, S from the slots L, R (see CompactSlots).
__device__ __forceinline__ Neighbours neighbours_of(unsigned meta, const CompactSlots& sl) {
  int s[6] = {sl.a.x, sl.a.y, sl.a.z, sl.a.w, sl.b.x, sl.b.y};
  for (int ax = 0; ax < 3; ++ax)
    if (((meta >> (3 * ax)) & 7u) == 4u) {  // (rr, r) -> (r, rr)
      const int t = s[2 * ax];
      s[2 * ax] = s[2 * ax + 1];
      s[2 * ax + 1] = t;
    }
  return {s[0], s[1], s[2], s[3], s[4], s[5]};
}

__device__ __forceinline__ uint4 pack_record(unsigned meta, const Neighbours& n, int q,
                                             int nlist) {
  const int x0 = n.x0 == nlist ? kNoneX : n.x0 - q, x1 = n.x1 == nlist ? kNoneX : n.x1 - q;
  int y0 = n.y0 == nlist ? kNoneY : n.y0 - q, y1 = n.y1 == nlist ? kNoneY : n.y1 - q;
  const int z0 = n.z0 - q, z1 = n.z1 - q;
  auto fits = [&](int pos, int d) { return pos == nlist || (d > kNoneY && d <= 32767); };
  unsigned m = meta & kRecMeta;
  if (!fits(n.y0, y0) || !fits(n.y1, y1)) {
    m |= kRecEscape;
    y0 = y1 = 0;
  }
  uint4 r;
  r.x = m | ((unsigned)(z1 >> 8) & 0xfffffu) << 12;
  r.y = ((unsigned)x0 & 0x3fffu) | ((unsigned)x1 & 0x3fffu) << 14 | ((unsigned)z1 & 0xfu) << 28;
  r.z = ((unsigned)y0 & 0xffffu) | (unsigned)y1 << 16;
  r.w = (unsigned)z0 << 4 | (((unsigned)z1 >> 4) & 0xfu);
  return r;
}

__device__ __forceinline__ Neighbours unpack_record(const uint4& r, int q, int nlist) {
  const int x0 = (int)(r.y << 18) >> 18, x1 = (int)(r.y << 4) >> 18;
  const int y0 = (int)(r.z << 16) >> 16, y1 = (int)r.z >> 16;
  Neighbours n;
  n.x0 = x0 == kNoneX ? nlist : q + x0;
  n.x1 = x1 == kNoneX ? nlist : q + x1;
  n.y0 = y0 == kNoneY ? nlist : q + y0;
  n.y1 = y1 == kNoneY ? nlist : q + y1;
  n.z0 = q + ((int)r.w >> 4);
  n.z1 = q + ((int)(r.x & ~0xfffu) >> 4 | (int)((r.w & 0xfu) << 4) | (int)(r.y >> 28));
  return n;
}

__device__ __forceinline__ int word_rank(uint2 w, int x) {
  return (int)w.y + __popc(w.x & ((1u << (x & 31)) - 1u));
}

__device__ __forceinline__ void interior_xyz(int lin, const Grid& g, int& x, int& y, int& z) {
  lin_to_xyz(lin, g, x, y, z);
  x -= 2;
  y -= 2;
  z -= 2;
}

// Loads of the correction and residual.  COHERENT: they were written earlier
// in the same launch by another CTA (the persistent round kernel of the
// server), so they bypass L1 (ld.global.cg); otherwise the read-only path.
template <bool COHERENT>
__device__ __forceinline__ float4 ld_corr(const float4* p) {
  return COHERENT ? __ldcg(p) : __ldg(p);
}

// e2 = L(e) + r for list position i.
template <int SOLVER, bool COHERENT = false>
__device__ __forceinline__ void inner_c_compute(const float4* __restrict__ E,
                                                float4* __restrict__ E2,
                                                const float4* __restrict__ R, int i,
                                                unsigned meta, const CompactSlots& sl) {
  const int cx = (int)(meta & 7u), cy = (int)((meta >> 3) & 7u), cz = (int)((meta >> 6) & 7u);
  auto fl = [&](int axis, int side) { return (meta >> (kMetaFluidShift + 2 * axis + side)) & 1u; };
  const float4 C = ld_corr<COHERENT>(E + i);
  const float4 XL = ld_corr<COHERENT>(E + sl.a.x), XR = ld_corr<COHERENT>(E + sl.a.y);
  const float4 YL = ld_corr<COHERENT>(E + sl.a.z), YR = ld_corr<COHERENT>(E + sl.a.w);
  const float4 ZL = ld_corr<COHERENT>(E + sl.b.x), ZR = ld_corr<COHERENT>(E + sl.b.y);
  const float4 r = ld_corr<COHERENT>(R + i);
  Stencil<float> s;
  // along-axis terms and the divergence read the true +-1 neighbours (0 where
  // solid; in cases 4 / 5 the solid side's slot holds the second neighbour);
  // the wall stencils across an axis take (ll, l, r, rr) = (R, L, R, L),
  // which case_pick resolves to exactly the points each case uses
  s.uc = C.x;
  s.uxm = fl(0, 0) ? XL.x : 0.f;
  s.uxp = fl(0, 1) ? XR.x : 0.f;
  s.uymm = YR.x; s.uym = YL.x; s.uyp = YR.x; s.uypp = YL.x;
  s.uzmm = ZR.x; s.uzm = ZL.x; s.uzp = ZR.x; s.uzpp = ZL.x;
  s.vc = C.y;
  s.vym = fl(1, 0) ? YL.y : 0.f;
  s.vyp = fl(1, 1) ? YR.y : 0.f;
  s.vxmm = XR.y; s.vxm = XL.y; s.vxp = XR.y; s.vxpp = XL.y;
  s.vzmm = ZR.y; s.vzm = ZL.y; s.vzp = ZR.y; s.vzpp = ZL.y;
  s.wc = C.z;
  s.wzm = fl(2, 0) ? ZL.z : 0.f;
  s.wzp = fl(2, 1) ? ZR.z : 0.f;
  s.wxmm = XR.z; s.wxm = XL.z; s.wxp = XR.z; s.wxpp = XL.z;
  s.wymm = YR.z; s.wym = YL.z; s.wyp = YR.z; s.wypp = YL.z;
  // a pressure difference is taken only where the -side neighbour is fluid,
  // and then its slot holds it; the plane flags carry the reapplied pressure
  // (correction 0) of the last interior plane and of the z halo below the first
  s.pc = (meta & kMetaZLast) ? 0.f : C.w;
  s.pxm = XL.w;
  s.pym = YL.w;
  s.pzm = (meta & kMetaZFirst) ? 0.f : ZL.w;
  float un, vn, wn, pn;
  update_fast_cases<float, SOLVER>(s, cx, cy, cz, un, vn, wn, pn);
  E2[i] = make_float4(un + r.x, vn + r.y, wn + r.z, pn + r.w);
}

// ---- the sweep over packed records

// One velocity component of update_fast<float>: f holds its off-centre sum.
template <int SOLVER>
__device__ __forceinline__ float velocity(float c, float f, float centre, float dp, bool zero) {
  f = fmaf(centre, c, f);
  if (SOLVER == 3) {
    const float t = fmaf(float(kDt / kRe * kOmega), f, float(1.0 - kOmega) * c);
    return fmaf(float(-kDt * kOmega), dp, t);
  }
  float t = fmaf(float(kDt / kRe), f, c);
  t = fmaf(float(-kDt), dp, t);
  return zero ? 0.f : t;
}

// Wall stencil a c + cF F + cS S of a case, and which neighbours F and S are.
struct CaseTerms {
  float a, cF, cS;
  bool s;           // S is not a second neighbour
  bool lf, rf, r4;  // left / right neighbour fluid; the right one is F
};

__device__ __forceinline__ CaseTerms case_terms(unsigned c) {
  const bool le2 = c <= 2, le3 = c <= 3, le5 = c <= 5;
  CaseTerms k;
  k.a = c == 1 ? -8.f : (le3 ? float(-16.0 / 3.0) : (le5 ? -5.f : -2.f));
  k.cF = le2 ? 0.f : (le3 ? float(8.0 / 3.0) : (le5 ? 2.f : 1.f));
  k.cS = c == 2 ? float(8.0 / 3.0) : (le3 ? 0.f : (le5 ? -0.2f : 1.f));
  k.s = c - 4u >= 2u;
  k.lf = !le2 && c != 4;
  k.rf = !(c & 1u);
  k.r4 = c == 4;
  return k;
}

// The update of update_fast<float> from the centre and the points F, S of each
// axis, its terms in the same order (a missing point is a zero, as is its
// term), so every kernel gives the same values (a zero may differ in sign).
template <int SOLVER>
__device__ __forceinline__ float4 update_records(unsigned meta, const float4& C, const float4& XF,
                                                 const float4& XS, const float4& YF,
                                                 const float4& YS, const float4& ZF,
                                                 const float4& ZS, const float4& r) {
  const CaseTerms kx = case_terms(meta & 7u), ky = case_terms((meta >> 3) & 7u),
                  kz = case_terms((meta >> 6) & 7u);
  const float pc = (meta & kMetaZLast) ? 0.f : C.w;
  const float zfw = (meta & kMetaZFirst) ? 0.f : ZF.w;
  auto along = [](const CaseTerms& k, float f, float s) { return f + (k.s ? s : 0.f); };
  auto right = [](const CaseTerms& k, float f, float s) {
    return k.rf ? (k.r4 ? f : s) : 0.f;
  };
  float f = along(kx, XF.x, XS.x);
  f = fmaf(ky.cF, YF.x, f);
  f = fmaf(ky.cS, YS.x, f);
  f = fmaf(kz.cF, ZF.x, f);
  f = fmaf(kz.cS, ZS.x, f);
  const float un =
      velocity<SOLVER>(C.x, f, -2.f + ky.a + kz.a, kx.lf ? pc - XF.w : 0.f, !kx.lf);
  f = along(ky, YF.y, YS.y);
  f = fmaf(kx.cF, XF.y, f);
  f = fmaf(kx.cS, XS.y, f);
  f = fmaf(kz.cF, ZF.y, f);
  f = fmaf(kz.cS, ZS.y, f);
  const float vn =
      velocity<SOLVER>(C.y, f, -2.f + kx.a + kz.a, ky.lf ? pc - YF.w : 0.f, !ky.lf);
  f = along(kz, ZF.z, ZS.z);
  f = fmaf(kx.cF, XF.z, f);
  f = fmaf(kx.cS, XS.z, f);
  f = fmaf(ky.cF, YF.z, f);
  f = fmaf(ky.cS, YS.z, f);
  const float wn =
      velocity<SOLVER>(C.z, f, -2.f + kx.a + ky.a, kz.lf ? pc - zfw : 0.f, !kz.lf);
  const float div = ((right(kz, ZF.z, ZS.z) - wn) + (right(ky, YF.y, YS.y) - vn)) +
                    (right(kx, XF.x, XS.x) - un);
  const float pn = fmaf(float(-kC2 * kDt), div, pc);
  return make_float4(un + r.x, vn + r.y, wn + r.z, pn + r.w);
}

// Loads of values an earlier launch wrote, possibly while this one was already
// resident (programmatic launch): not the read-only path.  COHERENT: written in
// this launch by other CTAs, so past L1.
template <bool COHERENT>
__device__ __forceinline__ float4 ld_value(const float4* p) {
  float4 v;
  if (COHERENT)
    asm volatile("ld.global.cg.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "l"(p));
  else
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "l"(p));
  return v;
}

// Loads of what a sweep reads once (residuals, records): past L1, and the first
// to leave L2, so that the correction, which the next sweep reads again, stays.
__device__ __forceinline__ unsigned long long stream_policy() {
  unsigned long long p;
  asm("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
  return p;
}

__device__ __forceinline__ float4 ld_stream(const float4* p) {
  float4 v;
  asm volatile("ld.global.L1::no_allocate.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "l"(p), "l"(stream_policy()));
  return v;
}

// Overlapped sweeps load records before they wait for the launch before them:
// between the packing and such a sweep on its stream there has to be a
// synchronisation or a plain launch.  Then the read-only path is safe too.
__device__ __forceinline__ uint4 ld_record(const uint4* p) {
  uint4 v;
  asm("ld.global.nc.L1::no_allocate.L2::cache_hint.v4.u32 {%0, %1, %2, %3}, [%4], %5;"
      : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
      : "l"(p), "l"(stream_policy()));
  return v;
}

// e2 = L(e) + r at list position q, record rc.
template <int SOLVER, bool COHERENT = false>
__device__ __forceinline__ void inner_r_voxel(const float4* E, float4* E2, const float4* R,
                                              const uint4& rc, const int2* ya, int q, int nlist) {
  Neighbours n = unpack_record(rc, q, nlist);
  if (rc.x & kRecEscape) {
    const int2 y = __ldg(ya + q);
    n.y0 = y.x;
    n.y1 = y.y;
  }
  const float4 C = ld_value<COHERENT>(E + q);
  const float4 XF = ld_value<COHERENT>(E + n.x0), XS = ld_value<COHERENT>(E + n.x1);
  const float4 YF = ld_value<COHERENT>(E + n.y0), YS = ld_value<COHERENT>(E + n.y1);
  const float4 ZF = ld_value<COHERENT>(E + n.z0), ZS = ld_value<COHERENT>(E + n.z1);
  const float4 r = ld_stream(R + q);
  E2[q] = update_records<SOLVER>(rc.x, C, XF, XS, YF, YS, ZF, ZS, r);
}

// One voxel of the batched kernels.
template <int SOLVER, bool COHERENT = false>
__device__ __forceinline__ void inner_c_voxel(const float4* __restrict__ E,
                                              float4* __restrict__ E2,
                                              const float4* __restrict__ R,
                                              const unsigned* __restrict__ meta,
                                              const int4* __restrict__ sa,
                                              const int2* __restrict__ sb, int i) {
  CompactSlots sl;
  sl.a = __ldg(sa + i);
  sl.b = __ldg(sb + i);
  inner_c_compute<SOLVER, COHERENT>(E, E2, R, i, __ldg(meta + i), sl);
}

// r = F(x) - x in FP64 from the padded state (as dc_residual_voxel), stored
// at list position q, and e1 = r.  centre: the block's table, for the whole
// stencil (null: reduced loads).
template <int SOLVER>
__device__ __forceinline__ void residual_c_voxel(const Fields<double>& X, float4* R, float4* E,
                                                 const uint8_t* codes, const Grid& g, int q,
                                                 int lin, const double* centre = nullptr) {
  int x, y, z;
  lin_to_xyz(lin, g, x, y, z);
  const int code = codes[((long long)z * g.NY + y) * g.pxc + x];
  const long long c = (long long)z * g.pl64 + (long long)y * g.px64 + x;
  Own64 o;
  double un, vn, wn, pn;
  if (centre) update64_whole<SOLVER, 0>(X, X, c, x, y, z, g, code, centre, o, un, vn, wn, pn);
  else update64<SOLVER, 0, kLdNc>(X, X, c, x, y, z, g, code, nullptr, o, un, vn, wn, pn);
  const double pstored = (z == g.NZ - 3) ? __ldg(X.p + c) : o.p;
  const float4 rv = make_float4((float)(un - o.u), (float)(vn - o.v), (float)(wn - o.w),
                                (float)(pn - pstored));
  R[q] = rv;
  E[q] = rv;
}

// x += e at a fluid voxel and at the periodic halo copies the padded form
// keeps of it (the z copies that land on the planes holding reapplied
// pressure take no pressure correction), as dc_correct_voxel.
__device__ __forceinline__ void correct_c_voxel(const Fields<double>& X, float4 e, const Grid& g,
                                                int lin) {
  int x, y, z;
  lin_to_xyz(lin, g, x, y, z);
  auto add = [&](int xx, int yy, int zz, bool pz) {
    const long long c = (long long)zz * g.pl64 + (long long)yy * g.px64 + xx;
    X.u[c] += (double)e.x;
    X.v[c] += (double)e.y;
    X.w[c] += (double)e.z;
    X.p[c] += pz ? 0.0 : (double)e.w;
  };
  add(x, y, z, false);
  if (g.per[0]) {
    if (x < 4) add(x + g.nx, y, z, false);
    if (x >= g.nx) add(x - g.nx, y, z, false);
  }
  if (g.per[1]) {
    if (y < 4) add(x, y + g.ny, z, false);
    if (y >= g.ny) add(x, y - g.ny, z, false);
  }
  if (g.per[2]) {
    if (z < 4) add(x, y, z + g.nz, z == 2);
    if (z >= g.nz) add(x, y, z - g.nz, z == g.nz + 1);
  }
}

}  // namespace pm
