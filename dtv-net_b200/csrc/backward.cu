// Voxel-driven FDK-weighted backprojector: every view in one launch, each
// voxel accumulated in registers and written once.
//
// Follows Standard/plug/kernel/backwardKernel.cu:22-53 (+ helper_geometry.h:
// 26-42) and Beijing/plug/kernel/backwardKernel.cu:18-45: per voxel and view,
// the detector coordinate of the voxel's projection is sampled bilinearly
// (border value 0) and weighted by bp_scale * (SDD/L)^power. The reference ran
// one launch per view (or per 21 views), read-modify-writing the whole volume
// each time (backwardKernel.cu:50,101-103). Here the view loop is inside the
// kernel; the projective map of each view (FP64-derived, see geometry.cu)
// gives the detector coordinates with one reciprocal per voxel-view (one per
// column and view on z-affine orbits).
#include <algorithm>
#include <type_traits>
#include <vector>
#include <string.h>

#include "common.cuh"

namespace dtv {

struct BPParams {
  int nx, ny, nz, nu, nv, n_views;
  int power;
  int extent;
  float scale;
  int64_t view_recs;  // records of one view
  int warp;           // columns of a warp and a quad (DTV_TUNE_BP_WARP)
  int cull;           // blocks skip the views whose detector they miss
};

constexpr int kBPTile = 16;  // columns per block edge
// Views whose 3x4 maps travel in one launch's parameters: read through the
// constant cache, they leave the L1 pipe to the sinogram records.
constexpr int kBPParamViews = 640;
struct BPMaps {
  float m[kBPParamViews][12];
};
static_assert(sizeof(BPMaps) <= 31 * 1024, "kernel parameter space");
constexpr int kBPThreads = kBPTile * kBPTile;
// voxels per thread along z (16 measured 3 % slower through the texture unit and
// 10 - 20 % through records: fewer resident warps); of volumes of up to kFlat slices
// kZCFlat, so that a thread does not project slices that are not there (231x152x1 x 32
// views of 389 x 3, records: 16.9 -> 10.8 us; 512x512x1 x 360 views, texture: 704 -> 294);
// of four slices not where blocks look for their views first, twice then (75x78x4 x 176
// modules: 17 us, 21)
constexpr int kZC = 8, kZCFlat = 2, kFlat = 4;

// Where a bilinear detector sample comes from.
// kTex: the texture unit (a layered FP32 texture, 8-bit weights), one fetch.
// kRec: one 16-byte record through L1, FP32 weights. Record (U, V) of a view
// (padded by kPad zeros on each side) holds its cell's bilinear polynomial
// s(au, av) = A + au B + av C + au av D in the order (A, C, B, D): A = s(U, V),
// B = s(U+1, V) - A, C = s(U, V+1) - A, D the mixed difference.
// kBoth: both, two sums per voxel (the correction pass of a texture plan
// against an exact one).
// kWide: kRec on detectors with more rows or columns than kIntMagicMost, cells by floorf
// (a kernel of its own: as a branch it cost the record kernels 7 %).
enum BPMode { kRec = 0, kTex = 1, kBoth = 2, kWide = 3 };

// Where a block's sums go: out = base + sum (out = sum when base is NULL; base
// may be out). kBoth: out takes the record sum E, and
// diff = diff_base + (E - T) with T the texture sum.
struct BPOut {
  float* out;
  const float* base;
  float* diff;
  const float* diff_base;
};

// Where a view's 3x4 map comes from: the launch parameters (one chunk of
// views) or the plan's device table.
struct ParamMaps {
  const BPMaps* m;
  __device__ __forceinline__ const float* row(int jn) const { return m->m[jn]; }
};
struct TableMaps {
  const BPView* v;  // first view of the chunk
  __device__ __forceinline__ const float* row(int jn) const { return v[jn].m; }
};

// The cells of two coordinates (t = floor + kIntMagic) and the fractions in them.
struct Frac2 {
  f32x2_t t, a;
};
__device__ __forceinline__ Frac2 frac2(f32x2_t v) {
  Frac2 r;
  r.t = add2_rm(v, splat2(kIntMagic));
  r.a = sub2(v, sub2(r.t, splat2(kIntMagic)));
  return r;
}
// The record's bilinear sample; au2 = (au, au).
__device__ __forceinline__ float bilinear(const float4 r, f32x2_t au2, float av) {
  float p, q;  // (A + au B, C + au D)
  unpack2(fma2(au2, f32x2(r.z, r.w), f32x2(r.x, r.y)), p, q);
  return fmaf(av, q, p);
}

// The first record of column u's cell in a view, as an address biased so that
// adding (float bits of floor(v) + kIntMagic) * row bytes gives row floor(v).
__device__ __forceinline__ unsigned long long cell_base(const char* view, unsigned int tu_bits,
                                                        unsigned int row_bytes) {
  const long long iu = (int)(tu_bits - kIntMagicBits) + kPad;
  return (unsigned long long)view + (unsigned long long)(iu * 16) +
         (unsigned long long)row_bytes * kPad - (unsigned long long)kIntMagicBits * row_bytes;
}
__device__ __forceinline__ float4 cell_at(unsigned long long base, unsigned int tv_bits,
                                          unsigned int row_bytes) {
  return __ldg(reinterpret_cast<const float4*>(base + (unsigned long long)tv_bits * row_bytes));
}

// The sample at (u, v) of a view, cell by floorf and 64-bit index.
__device__ __forceinline__ float sample_wide(const char* view, float u, float v, float mu, float mv) {
  u = fminf(fmaxf(u, -2.f), mu);
  v = fminf(fmaxf(v, -2.f), mv);
  const float fu = floorf(u), fv = floorf(v);
  const long long row = (long long)mu + 2 * kPad;
  const float4 r = __ldg(reinterpret_cast<const float4*>(view) + ((long long)fv + kPad) * row +
                         (long long)fu + kPad);
  return bilinear(r, splat2(u - fu), v - fv);
}

// Whether view map w can see any voxel of the box [i0, i1] x [j0, j1] x
// [k0, k1]: false only if all eight corners lie in front of the source and
// project beyond one edge of the detector by more than a pixel past the last
// sample that reaches it (the box then projects into their convex hull, and
// every one of its samples is exactly zero).
__host__ __device__ __forceinline__ bool box_seen(const float* w, float i0, float i1, float j0, float j1,
                                         float k0, float k1, float nu, float nv) {
  float umin = 3.4e38f, umax = -3.4e38f, vmin = 3.4e38f, vmax = -3.4e38f, hmin = 3.4e38f;
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const float x = (c & 1) ? i1 : i0, y = (c & 2) ? j1 : j0, z = (c & 4) ? k1 : k0;
    const float h = fmaf(w[8], x, fmaf(w[9], y, fmaf(w[10], z, w[11])));
    const float u = fmaf(w[0], x, fmaf(w[1], y, fmaf(w[2], z, w[3]))) / h;
    const float v = fmaf(w[4], x, fmaf(w[5], y, fmaf(w[6], z, w[7]))) / h;
    hmin = fminf(hmin, h);
    umin = fminf(umin, u); umax = fmaxf(umax, u);
    vmin = fminf(vmin, v); vmax = fmaxf(vmax, v);
  }
  return !(hmin > 1e-3f && (umax < -2.f || umin > nu + 1.f || vmax < -2.f || vmin > nv + 1.f));
}

// One block's columns: column tile `tile`, z-chunk `zc` of ZC voxels, views
// n0 .. n0 + n_chunk - 1. S == 1: a tile is 16 x 16 columns. S > 1 (volumes
// too small to fill the GPU otherwise): the block's S groups of 256 / S threads
// own the same tile of (64 / (2 S)) x 8 columns and each takes one of S equal
// runs of the views; their sums are added through shared memory in the order
// of the runs, so the result is deterministic.
//
// kZAff: every view's u and h are independent of z (a detector parallel to the
// rotation axis, as in the circular orbits), so per column and view the kernel
// computes u, 1/h and the weight once and marches v. Voxels go in pairs along
// z through packed FP32. A thread's z-run projects to a monotone run of v (and
// u), so two end tests replace per-voxel bounds: wholly on the detector runs
// unchecked, wholly beside it is skipped (its samples are zeros), and only
// runs across an edge clamp each voxel.
//
// Bound: through the texture unit its fetch rate (256^3 x 64 views of 384^2:
// 0.84 ms; 1.03 ms before a column's views beside the detector were skipped,
// 16 % of that scan's column-views). Through records the L1 lines of a warp's
// load (6.5 per load, 2 clocks each where they miss) and their latency: 1.62 ms
// from four scalar loads, 1.22 ms from records with conversions, 0.90 ms now.
// The records could also reproduce the texture filter (its weights are
// alpha beta to 1/256 exactly), but at 1.06 - 1.11 ms they lose to it.
template <int S>
struct BPShape {
  static constexpr int kGroup = kBPThreads / S;           // threads, one column each
  static constexpr int kH = S == 1 ? kBPTile : 8;         // tile rows (y)
  static constexpr int kW = kGroup / kH;                  // tile columns (x)
};

template <int kMode, bool kZAff, int S, bool kCull, int ZC, class Maps>
__device__ __forceinline__ void bp_columns(const BPParams& bp, const Maps& maps, int n0, int n_chunk,
                                           const float4* __restrict__ recs, cudaTextureObject_t tex,
                                           const BPOut& dst, int tile, int zc) {
  static_assert(ZC % 2 == 0, "voxels go in pairs");
  using Shape = BPShape<S>;
  const int tiles_x = (bp.nx + Shape::kW - 1) / Shape::kW;
  const int t = (int)threadIdx.x;
  const int group = S > 1 ? t / Shape::kGroup : 0;
  // this thread's column in the tile: quads (4 consecutive lanes) of 2 x 2
  // columns, a warp of 8 quads covers 4 x 8 columns, or with S == 1 as
  // DTV_TUNE_BP_WARP says: 16 x 2, 8 x 4 or 4 x 8 of row quads, 8 x 4 of squares
  const int q = (t >> 2) & 7, qi = t & 1, qj = (t >> 1) & 1, wp = (t % Shape::kGroup) >> 5;
  int li = ((q & 1) << 1 | qi) | ((wp & (Shape::kW / 4 - 1)) << 2);
  int lj = ((q >> 1) << 1 | qj) | (S == 1 ? (wp >> 2) << 3 : 0);
  if constexpr (S == 1) {
    if (bp.warp == 3) {
      li = ((q & 3) << 1 | qi) | ((wp & 1) << 3);
      lj = ((q >> 2) << 1 | qj) | ((wp >> 1) << 2);
    } else if (bp.warp == 2) {
      li = (t & 3) | (((t >> 5) & 3) << 2);
      lj = ((t >> 2) & 7) | ((t >> 7) << 3);
    } else if (bp.warp == 1) {
      li = (t & 7) | (((t >> 5) & 1) << 3);
      lj = ((t >> 3) & 3) | ((t >> 6) << 2);
    } else if (bp.warp == 0) {
      li = t & 15;
      lj = t >> 4;
    }
  }
  const int ti = (tile % tiles_x) * Shape::kW, tj = (tile / tiles_x) * Shape::kH;
  const int i = ti + li, j = tj + lj;
  const int k0 = zc * ZC;
  const bool valid = i < bp.nx && j < bp.ny;
  // kCull: the views some voxel of the block can be seen in, one bit each
  __shared__ unsigned int seen[kCull ? kBPParamViews / 32 : 1];
  if constexpr (kCull) {
    for (int jb = 0; jb < n_chunk; jb += kBPThreads) {
      const int jn = jb + t;
      const bool s = jn < n_chunk &&
                     box_seen(maps.row(jn), (float)ti, (float)(ti + Shape::kW - 1), (float)tj,
                              (float)(tj + Shape::kH - 1), (float)k0, (float)(k0 + ZC - 1),
                              (float)bp.nu, (float)bp.nv);
      const unsigned int m = __ballot_sync(0xffffffffu, s);
      if ((t & 31) == 0 && jn < n_chunk) seen[jn >> 5] = m;
    }
    __syncthreads();
  }
  if (!valid && S == 1) return;  // the groups of a split block meet at a barrier below
  // this thread's views: all of the chunk, or its group's run of them
  const int hv = (n_chunk + S - 1) / S;
  const int jn0 = min(group * hv, n_chunk);
  const int jn1 = valid ? min(jn0 + hv, n_chunk) : jn0;
  float acc[ZC], act[kMode == kBoth ? ZC : 1];
#pragma unroll
  for (int z = 0; z < ZC; ++z) acc[z] = 0.f;
#pragma unroll
  for (int z = 0; z < (kMode == kBoth ? ZC : 1); ++z) act[z] = 0.f;
  const float fi = (float)i, fj = (float)j;
  const float mu = (float)bp.nu, mv = (float)bp.nv;
  const unsigned int row_bytes = (unsigned int)(bp.nu + 2 * kPad) * 16u;
  const float kf0 = (float)k0;
  // the next view at or after jn that the block can be seen in
  auto next_seen = [&](int jn) {
    if constexpr (kCull) {
      while (jn < jn1) {
        const unsigned int m = seen[jn >> 5] >> (jn & 31);
        if (m) return jn + __ffs((int)m) - 1;
        jn = (jn | 31) + 1;
      }
    }
    return jn;
  };
  for (int jn = next_seen(jn0); jn < jn1; jn = next_seen(jn + 1)) {
    const float* w = maps.row(jn);
    const float m0 = w[0], m1 = w[1], m2 = w[2], m3 = w[3];
    const float m4 = w[4], m5 = w[5], m6 = w[6], m7 = w[7];
    const float m8 = w[8], m9 = w[9], m10 = w[10], m11 = w[11];
    const float bu = fmaf(m0, fi, fmaf(m1, fj, m3));
    const float bv = fmaf(m4, fi, fmaf(m5, fj, m7));
    const float bh = fmaf(m8, fi, fmaf(m9, fj, m11));
    const char* view = reinterpret_cast<const char*>(recs + (int64_t)(n0 + jn) * bp.view_recs);
    if constexpr (kZAff) {
      const float rh = __frcp_rn(bh);
      // v from the absolute slice index: the same bits for every z-chunking.
      // Coordinates are rounded explicitly (no contraction into FMAs), so
      // every kernel instance samples a voxel-view at the same position.
      const float u = __fmul_rn(bu, rh), vb = __fmul_rn(bv, rh), dv = __fmul_rn(m6, rh);
      float wgt = bp.scale;
      if (bp.power == 2) wgt *= rh * rh;
      else if (bp.power == 1) wgt *= rh;
      if (bp.extent) {
        const float tu = __fadd_rn(u, 0.5f);
        if (tu < -1.f || tu > bp.nx + 1.f) continue;
      }
      const float va = fmaf(kf0, dv, vb), ve = fmaf(kf0 + (float)(ZC - 1), dv, vb);
      const float vlo = fminf(va, ve), vhi = fmaxf(va, ve);
      // zero samples only (a non-finite weight still goes through below)
      if ((u < -1.f || u >= mu || vhi < -1.f || vlo >= mv) && fabsf(wgt) < 3.4e38f) continue;
      const float tu = __fadd_rn(u, 0.5f);  // texture coordinate (texel centres at i + 1/2)
      const Frac2 fu = frac2(splat2(fminf(fmaxf(u, -2.f), mu)));
      float tu_f, dummy;
      unpack2(fu.t, tu_f, dummy);
      const unsigned long long base = cell_base(view, __float_as_uint(tu_f), row_bytes);
      const bool inside = vlo >= -1.f && vhi < mv && u >= -1.f && u < mu && !bp.extent && kMode != kWide;
      if (kMode == kTex || inside) {
#pragma unroll
        for (int z = 0; z < ZC; z += 2) {
          const f32x2_t v2 =
              fma2(f32x2(kf0 + (float)z, kf0 + (float)(z + 1)), splat2(dv), splat2(vb));
          float v[2], w2[2] = {wgt, wgt};
          unpack2(v2, v[0], v[1]);
          if constexpr (kMode == kTex || kMode == kBoth) {
#pragma unroll
            for (int y = 0; y < 2; ++y) {
              const float tv = __fadd_rn(v[y], 0.5f);
              if (bp.extent && (tv < -1.f || tv > bp.ny + 1.f)) w2[y] = 0.f;
              float& a = kMode == kBoth ? act[kMode == kBoth ? z + y : 0] : acc[z + y];
              a = fmaf(tex2DLayered<float>(tex, tu, tv, n0 + jn), w2[y], a);
            }
          }
          if constexpr (kMode != kTex) {
            const Frac2 fv = frac2(v2);
            float t[2], av[2];
            unpack2(fv.t, t[0], t[1]);
            unpack2(fv.a, av[0], av[1]);
#pragma unroll
            for (int y = 0; y < 2; ++y)
              acc[z + y] = fmaf(bilinear(cell_at(base, __float_as_uint(t[y]), row_bytes), fu.a, av[y]),
                                wgt, acc[z + y]);
          }
        }
      } else {
#pragma unroll
        for (int z = 0; z < ZC; ++z) {
          const float v = fmaf(kf0 + (float)z, dv, vb);
          const float tv = __fadd_rn(v, 0.5f);
          float wz = wgt;
          if (bp.extent && (tv < -1.f || tv > bp.ny + 1.f)) wz = 0.f;
          const Frac2 fv = frac2(splat2(fminf(fmaxf(v, -2.f), mv)));
          float t0, av;
          unpack2(fv.t, t0, dummy);
          unpack2(fv.a, av, dummy);
          const float val = kMode == kWide
                                ? sample_wide(view, u, v, mu, mv)
                                : bilinear(cell_at(base, __float_as_uint(t0), row_bytes), fu.a, av);
          acc[z] = fmaf(val, wz, acc[z]);
          if constexpr (kMode == kBoth)
            act[z] = fmaf(tex2DLayered<float>(tex, tu, tv, n0 + jn), wz, act[z]);
        }
      }
    } else {
      // u, v, h of two voxels at slices (ka, kb); any h, zero included, where checked
      // (only then: 2 % of a tilted scan's time otherwise)
      struct UVH {
        f32x2_t u, v, rh;
        float ha, hb;
      };
      auto project = [&](float ka, float kb, auto any) {
        constexpr bool kAny = decltype(any)::value;
        const f32x2_t kk = f32x2(ka, kb);
        UVH p;
        unpack2(fma2(splat2(m10), kk, splat2(bh)), p.ha, p.hb);
        p.rh = f32x2(rcp_newton<kAny>(p.ha), rcp_newton<kAny>(p.hb));
        p.u = mul2(fma2(splat2(m2), kk, splat2(bu)), p.rh);
        p.v = mul2(fma2(splat2(m6), kk, splat2(bv)), p.rh);
        return p;
      };
      bool inside, beside;
      {
        const UVH p = project(kf0, kf0 + (float)(ZC - 1), std::false_type{});
        float ua, ub, va, ve;
        unpack2(p.u, ua, ub);
        unpack2(p.v, va, ve);
        const bool front = p.ha > 0.f && p.hb > 0.f;
        const float ulo = fminf(ua, ub), uhi = fmaxf(ua, ub), vlo = fminf(va, ve),
                    vhi = fmaxf(va, ve);
        // u and v are monotone along the run up to rounding, hence the margin
        beside = front && (uhi < -1.02f || ulo > mu + 0.02f || vhi < -1.02f || vlo > mv + 0.02f);
        inside = front && ulo >= -1.f && uhi < mu && vlo >= -1.f && vhi < mv;
        inside = inside && kMode != kWide;
        if (bp.extent)
          inside = inside && __fadd_rn(uhi, 0.5f) <= bp.nx + 1.f && __fadd_rn(vhi, 0.5f) <= bp.ny + 1.f;
      }
      if (beside) continue;
      const unsigned long long vbase =
          cell_base(view, kIntMagicBits, row_bytes) - (unsigned long long)kIntMagicBits * 16u;
      auto step = [&](int z, auto check) {
        constexpr bool checked = decltype(check)::value;
        const UVH p = project(kf0 + (float)z, kf0 + (float)(z + 1), check);
        f32x2_t wg = splat2(bp.scale);
        if (bp.power == 2) wg = mul2(wg, mul2(p.rh, p.rh));
        else if (bp.power == 1) wg = mul2(wg, p.rh);
        float w0, w1, u0 = 0.f, u1 = 0.f, v0 = 0.f, v1 = 0.f;
        unpack2(wg, w0, w1);
        f32x2_t uu = p.u, vv = p.v;
        if (checked) {
          unpack2(uu, u0, u1);
          unpack2(vv, v0, v1);
          if (bp.extent) {
            auto out = [&](float u, float v) {
              const float tu = __fadd_rn(u, 0.5f), tv = __fadd_rn(v, 0.5f);
              return tu < -1.f || tu > bp.nx + 1.f || tv < -1.f || tv > bp.ny + 1.f;
            };
            if (out(u0, v0)) w0 = 0.f;
            if (out(u1, v1)) w1 = 0.f;
          }
          uu = f32x2(fminf(fmaxf(u0, -2.f), mu), fminf(fmaxf(u1, -2.f), mu));
          vv = f32x2(fminf(fmaxf(v0, -2.f), mv), fminf(fmaxf(v1, -2.f), mv));
        }
        if constexpr (kMode == kTex || kMode == kBoth) {
          unpack2(p.u, u0, u1);
          unpack2(p.v, v0, v1);
          const float uy[2] = {u0, u1}, vy[2] = {v0, v1};
#pragma unroll
          for (int y = 0; y < 2; ++y) {
            float& a = kMode == kBoth ? act[kMode == kBoth ? z + y : 0] : acc[z + y];
            a = fmaf(tex2DLayered<float>(tex, __fadd_rn(uy[y], 0.5f), __fadd_rn(vy[y], 0.5f), n0 + jn),
                     y ? w1 : w0, a);
          }
        }
        if constexpr (kMode != kTex) {
          const Frac2 fu = frac2(uu), fv = frac2(vv);
          float tu[2], tv[2], au[2], av[2];
          unpack2(fu.t, tu[0], tu[1]);
          unpack2(fv.t, tv[0], tv[1]);
          unpack2(fu.a, au[0], au[1]);
          unpack2(fv.a, av[0], av[1]);
#pragma unroll
          for (int y = 0; y < 2; ++y) {
            float val;
            if (checked && kMode == kWide)
              val = sample_wide(view, y ? u1 : u0, y ? v1 : v0, mu, mv);
            else
              val = bilinear(cell_at(vbase + (unsigned long long)__float_as_uint(tu[y]) * 16u,
                                     __float_as_uint(tv[y]), row_bytes),
                             splat2(au[y]), av[y]);
            acc[z + y] = fmaf(val, y ? w1 : w0, acc[z + y]);
          }
        }
      };
      if (inside) {
#pragma unroll
        for (int z = 0; z < ZC; z += 2) step(z, std::false_type{});
      } else {
#pragma unroll
        for (int z = 0; z < ZC; z += 2) step(z, std::true_type{});
      }
    }
  }
  if constexpr (S > 1) {
    // groups 1 .. S-1 hand their sums to group 0, which adds them in order
    // (dynamic shared memory, given only to split launches)
    extern __shared__ float red[];
    constexpr int kPer = (kMode == kBoth ? 2 : 1) * ZC;
    const int lt = t % Shape::kGroup;
    if (group > 0) {
      float* r = red + (group - 1) * kPer * Shape::kGroup + lt;
#pragma unroll
      for (int z = 0; z < ZC; ++z) {
        r[z * Shape::kGroup] = acc[z];
        if constexpr (kMode == kBoth) r[(ZC + z) * Shape::kGroup] = act[z];
      }
    }
    __syncthreads();
    if (group > 0 || !valid) return;
#pragma unroll
    for (int g = 0; g < S - 1; ++g) {
      const float* r = red + g * kPer * Shape::kGroup + lt;
#pragma unroll
      for (int z = 0; z < ZC; ++z) {
        acc[z] = acc[z] + r[z * Shape::kGroup];
        if constexpr (kMode == kBoth) act[z] = act[z] + r[(ZC + z) * Shape::kGroup];
      }
    }
  }
  const int64_t plane = (int64_t)bp.nx * bp.ny;
  const int64_t col = (int64_t)j * bp.nx + i;
#pragma unroll
  for (int z = 0; z < ZC; ++z) {
    const int k = k0 + z;
    if (k < bp.nz) {
      const int64_t e = col + k * plane;
      dst.out[e] = dst.base ? dst.base[e] + acc[z] : acc[z];
      if constexpr (kMode == kBoth) {
        const float d = acc[z] - act[z];
        dst.diff[e] = dst.diff_base ? dst.diff_base[e] + d : d;
      }
    }
  }
}

// Unsplit record kernels are held to 48 registers for five blocks per SM: their
// loads' latency is the bound (256^3 x 64 views: 0.97 -> 0.90 ms).
template <int kMode, bool kZAff, int S, bool kCull, int ZC>
__global__ void __launch_bounds__(kBPThreads, kMode == kRec && kZAff && S == 1 ? 5 : 1) bp_kernel(BPParams bp, const __grid_constant__ BPMaps maps,
                                                        int n0, int n_chunk,
                                                        const float4* __restrict__ recs,
                                                        cudaTextureObject_t tex, BPOut dst) {
  bp_columns<kMode, kZAff, S, kCull, ZC>(bp, ParamMaps{&maps}, n0, n_chunk, recs, tex, dst,
                                         (int)blockIdx.x, (int)blockIdx.y);
}

// Writes the records of a sinogram's views: record (U, V) of a view from
// the four detector values (u, v) = (U - 2 .. U - 1, V - 2 .. V - 1), zero
// outside the view. Only records that reach the view (U in [1, nu+1], V in
// [1, nv+1]) are written; the rest keep the plan's initial zeros. A warp owns
// 32 columns of kSinoRows records: each row of the view is loaded once and its
// right neighbours come from the next lane, so the pass is bound by its
// 16-byte writes.
constexpr int kSinoRows = 8;
__global__ void __launch_bounds__(256) stage_sino_kernel(const float* __restrict__ in,
                                                         float4* __restrict__ out, int nu, int nv,
                                                         int64_t warps) {
  const int lane = threadIdx.x & 31;
  const int64_t job = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
  if (job >= warps) return;
  const int tu = (nu + 1 + 31) / 32, tv = (nv + 1 + kSinoRows - 1) / kSinoRows;
  const int bu = (int)(job % tu);
  const int64_t r = job / tu;
  const int V0 = (int)(r % tv) * kSinoRows + 1;
  const int64_t n = r / tv;
  const int u = bu * 32 + lane - 1;  // detector column of record U = u + kPad
  const float* s = in + n * nu * nv;
  auto row = [&](int v, float& a, float& d) {  // s(u, v) and its difference to the right
    const bool vin = v >= 0 && v < nv;
    a = vin && u >= 0 && u < nu ? __ldg(s + (int64_t)v * nu + u) : 0.f;
    float right = __shfl_down_sync(0xffffffffu, a, 1);
    if (lane == 31) right = vin && u + 1 < nu ? __ldg(s + (int64_t)v * nu + u + 1) : 0.f;
    d = right - a;
  };
  float a[kSinoRows + 1], d[kSinoRows + 1];
#pragma unroll
  for (int k = 0; k <= kSinoRows; ++k) row(V0 - kPad + k, a[k], d[k]);
  const int pu = nu + 2 * kPad;
  float4* o = out + n * (int64_t)pu * (nv + 2 * kPad) + (int64_t)V0 * pu + u + kPad;
  if (u > nu - 1) return;
#pragma unroll
  for (int k = 0; k < kSinoRows; ++k)
    if (V0 + k <= nv + 1)
      o[(int64_t)k * pu] = make_float4(a[k], a[k + 1] - a[k], d[k], d[k + 1] - d[k]);
}

// The sinogram into its layered array, by surface writes: 3.9 MB (64^3 x 60 views)
// 2.8 us, 37.7 MB 14.5 us, against 8.0 and 39.5 us for the 3-D copy.
__global__ void __launch_bounds__(256) stage_sino_tex_kernel(const float* __restrict__ in,
                                                             cudaSurfaceObject_t surf, int nu,
                                                             int nv) {
  const int u = blockIdx.x * 32 + (threadIdx.x & 31);
  const int v0 = blockIdx.y * 32 + (threadIdx.x >> 5);
  const int n = blockIdx.z;
  if (u >= nu) return;
  const float* s = in + (int64_t)n * nu * nv + u;
  float x[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) x[k] = v0 + 8 * k < nv ? __ldg(s + (int64_t)(v0 + 8 * k) * nu) : 0.f;
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (v0 + 8 * k < nv) surf2DLayeredwrite(x[k], surf, u * 4, v0 + 8 * k, n);
}

// View groups per block: the least S of 1, 2, 4, 8 that gives the grid three
// blocks per SM (8 voxels per thread throughout). A property of the plan's
// geometry alone, so every launch of the plan sums its views in the same order.
// 64^3 x 60 views, records: S = 1 47 us, 2 and 4 35 us, 8 37 us; 128^3 x 48
// views: 126, 122, 128, 143 us.
constexpr int64_t kBPWantBlocks = 3 * 148;
constexpr int kBPSplits = 8;

static int bp_tiles(const GeomParams& gp, int S) {
  const int h = S == 1 ? kBPTile : 8, w = kBPThreads / S / h;
  return ((gp.nx + w - 1) / w) * ((gp.ny + h - 1) / h);
}
static int bp_split(const GeomParams& gp) {
  int S = 1;
  while (S < kBPSplits && 2 * S <= gp.n_views &&
         (int64_t)bp_tiles(gp, S) * ((gp.nz + kZC - 1) / kZC) < kBPWantBlocks)
    S *= 2;
  return S;
}
static size_t bp_smem(int mode, int S, int zc) {
  return (size_t)(S - 1) * (mode == kBoth ? 2 : 1) * zc * (kBPThreads / S) * sizeof(float);
}

struct BPLaunch {
  dim3 grid;
  int S, zc;
  cudaStream_t st;
};

template <int kMode, bool kZAff, bool kCull, int ZC>
static void launch_bp_shape(const BPLaunch& l, const BPParams& bp, const BPMaps& maps, int n0,
                            int cnt, const float4* recs, cudaTextureObject_t tex,
                            const BPOut& dst) {
  const auto kernel = l.S == 8   ? bp_kernel<kMode, kZAff, 8, kCull, ZC>
                      : l.S == 4 ? bp_kernel<kMode, kZAff, 4, kCull, ZC>
                      : l.S == 2 ? bp_kernel<kMode, kZAff, 2, kCull, ZC>
                                 : bp_kernel<kMode, kZAff, 1, kCull, ZC>;
  kernel<<<l.grid, kBPThreads, bp_smem(kMode, l.S, ZC), l.st>>>(bp, maps, n0, cnt, recs, tex, dst);
}

template <int kMode, bool kZAff, bool kCull>
static void launch_bp_chunk(const BPLaunch& l, const BPParams& bp, const BPMaps& maps, int n0,
                            int cnt, const float4* recs, cudaTextureObject_t tex,
                            const BPOut& dst) {
  if constexpr (kMode != kBoth) {
    if (l.zc == kZCFlat) {
      launch_bp_shape<kMode, kZAff, kCull, kZCFlat>(l, bp, maps, n0, cnt, recs, tex, dst);
      return;
    }
  }
  launch_bp_shape<kMode, kZAff, kCull, kZC>(l, bp, maps, n0, cnt, recs, tex, dst);
}

template <int kMode>
static void launch_bp_mode(const BPLaunch& l, bool zaff, const BPParams& bp, const BPMaps& maps,
                           int n0, int cnt, const float4* recs, cudaTextureObject_t tex,
                           const BPOut& dst) {
  if (bp.cull) {
    if (zaff) launch_bp_chunk<kMode, true, true>(l, bp, maps, n0, cnt, recs, tex, dst);
    else launch_bp_chunk<kMode, false, true>(l, bp, maps, n0, cnt, recs, tex, dst);
  } else {
    if (zaff) launch_bp_chunk<kMode, true, false>(l, bp, maps, n0, cnt, recs, tex, dst);
    else launch_bp_chunk<kMode, false, false>(l, bp, maps, n0, cnt, recs, tex, dst);
  }
}

static void launch_bp(int mode, const BPLaunch& l, bool zaff, const BPParams& bp,
                      const BPMaps& maps, int n0, int cnt, const float4* recs,
                      cudaTextureObject_t tex, const BPOut& dst) {
  if (mode == kWide && zaff)
    bp_kernel<kWide, true, 1, false, kZC><<<l.grid, kBPThreads, 0, l.st>>>(bp, maps, n0, cnt, recs, tex, dst);
  else if (mode == kWide)
    bp_kernel<kWide, false, 1, false, kZC><<<l.grid, kBPThreads, 0, l.st>>>(bp, maps, n0, cnt, recs, tex, dst);
  else if (mode == kTex) launch_bp_mode<kTex>(l, zaff, bp, maps, n0, cnt, recs, tex, dst);
  else if (mode == kBoth) launch_bp_mode<kBoth>(l, zaff, bp, maps, n0, cnt, recs, tex, dst);
  else launch_bp_mode<kRec>(l, zaff, bp, maps, n0, cnt, recs, tex, dst);
}

static BPParams plan_bp_params(const Plan* p) {
  const GeomParams& gp = p->gp;
  BPParams bp;
  bp.nx = gp.nx; bp.ny = gp.ny; bp.nz = gp.nz;
  bp.nu = gp.nu; bp.nv = gp.nv; bp.n_views = gp.n_views;
  bp.power = gp.bp_power;
  bp.extent = gp.bp_extent;
  bp.scale = (float)gp.bp_scale;
  bp.view_recs = (int64_t)(gp.nu + 2 * kPad) * (gp.nv + 2 * kPad);
  bp.warp = p->bp_warp;
  bp.cull = p->bp_cull;
  return bp;
}

// Copies one batch item's sinogram into the plan's layered texture.
static int stage_sino_tex(Plan* p, const float* sino, cudaStream_t st) {
  const GeomParams& gp = p->gp;
  const dim3 grid((gp.nu + 31) / 32, (gp.nv + 31) / 32, gp.n_views);
  stage_sino_tex_kernel<<<grid, 256, 0, st>>>(sino, p->sino_surf, gp.nu, gp.nv);
  note_launch();
  DTV_LAUNCH_CHECK();
  return DTV_OK;
}

// Writes the records of `views` views.
static int stage_sino_rec(Plan* p, const float* sino, int views, cudaStream_t st) {
  const GeomParams& gp = p->gp;
  const int64_t warps = (int64_t)((gp.nu + 1 + 31) / 32) *
                        ((gp.nv + 1 + kSinoRows - 1) / kSinoRows) * views;
  const int64_t blocks = (warps + 7) / 8;
  DTV_CHECK(blocks < 2147483647LL, "sinogram too large for one staging launch");
  stage_sino_kernel<<<(unsigned)blocks, 256, 0, st>>>(sino, p->d_sino_rec, gp.nu, gp.nv, warps);
  note_launch();
  DTV_LAUNCH_CHECK();
  return DTV_OK;
}

// Whether most (block, view) pairs miss the detector, over a sample of the
// plan's blocks and views: then the blocks look for the views they meet first.
// Of many-module scans, whose modules each see a slice of the fan, most pairs
// go; where few do the test costs more than it saves (a circular scan whose
// detector misses the volume's corners: 0.84 -> 0.86 ms through the texture
// unit, 151x163x97 through records 118 -> 133 us), and a thread's own end tests skip
// its views beside the detector anyway.
int bp_cull_rule(const Plan* p) {
  const GeomParams& gp = p->gp;
  int missed = 0, total = 0;
  const int vs = std::max(1, gp.n_views / 48);
  for (int n = 0; n < gp.n_views; n += vs)
    for (int c = 0; c < 18; ++c) {
      // blocks at 1/6, 3/6, 5/6 of x and y and 1/4, 3/4 of z
      const int n3[3] = {gp.nx, gp.ny, gp.nz}, e[3] = {kBPTile, kBPTile, kZC};
      const int at[3] = {2 * (c % 3) + 1, 2 * (c / 3 % 3) + 1, 2 * (c / 9) + 1};
      float lo[3], hi[3];
      for (int a = 0; a < 3; ++a) {
        const int b = (int)((int64_t)n3[a] * at[a] / (a == 2 ? 4 : 6)) / e[a];
        lo[a] = (float)(b * e[a]);
        hi[a] = (float)(b * e[a] + e[a] - 1);
      }
      missed += !box_seen(p->h_bpv[n].m, lo[0], hi[0], lo[1], hi[1], lo[2], hi[2], (float)gp.nu,
                          (float)gp.nv);
      ++total;
    }
  return missed * 2 >= total ? 1 : 0;
}

// The views in chunks of kBPParamViews (their maps travel in the launch parameters), and
// where records are sampled in runs of as many views as the records of plan `rec` hold,
// each staged from `sino` first; later chunks add onto the first one's result.
static int bp_view_chunks(const Plan* p, int mode, Plan* rec, const float* sino, BPOut dst,
                          cudaStream_t st) {
  const GeomParams& gp = p->gp;
  const BPParams bp = plan_bp_params(p);
  const cudaTextureObject_t tex = p->sino_tex ? p->sino_tex[0] : 0;
  if (mode == kRec && std::max(gp.nu, gp.nv) + 2 * kPad > kIntMagicMost) mode = kWide;
  const int S = mode == kWide ? 1 : bp_split(gp);
  // (the view split stays that of kZC, for the many-plan launches' sums)
  const bool flat = gp.nz <= (bp.cull ? kFlat - 1 : kFlat);
  const int zc = flat && (mode == kRec || mode == kTex) ? kZCFlat : kZC;
  const BPLaunch l{dim3(bp_tiles(gp, S), (gp.nz + zc - 1) / zc), S, zc, st};
  const int run = mode == kTex ? gp.n_views : rec->sino_rec_views;
  BPMaps maps;
  for (int r0 = 0; r0 < gp.n_views; r0 += run) {
    const int r1 = std::min(r0 + run, gp.n_views);
    const float4* recs = nullptr;  // as if of view 0
    if (mode != kTex) {
      const int rc = stage_sino_rec(rec, sino + (int64_t)r0 * gp.nu * gp.nv, r1 - r0, st);
      if (rc) return rc;
      recs = rec->d_sino_rec - r0 * bp.view_recs;
    }
    for (int n0 = r0; n0 < r1; n0 += kBPParamViews) {
      const int cnt = std::min(kBPParamViews, r1 - n0);
      for (int j = 0; j < cnt; ++j) memcpy(maps.m[j], p->h_bpv[n0 + j].m, sizeof(maps.m[j]));
      if (n0 > 0) {
        dst.base = dst.out;
        dst.diff_base = dst.diff;  // (kBoth only)
      }
      launch_bp(mode, l, p->bp_zaffine != 0, bp, maps, n0, cnt, recs, tex, dst);
      note_launch();
      DTV_LAUNCH_CHECK();
    }
  }
  return DTV_OK;
}

int backward_impl(Plan* p, const float* sino, int batch, const float* base, float* out,
                  cudaStream_t st) {
  const GeomParams& gp = p->gp;
  const int64_t per_item = (int64_t)gp.nu * gp.nv * gp.n_views;
  const int64_t vox = (int64_t)gp.nx * gp.ny * gp.nz;
  for (int b = 0; b < batch; ++b) {
    const float* s = sino + b * per_item;
    int rc = p->sino_tex ? stage_sino_tex(p, s, st) : DTV_OK;
    if (rc) return rc;
    rc = bp_view_chunks(p, p->sino_tex ? kTex : kRec, p, s,
                        BPOut{out + b * vox, base ? base + b * vox : nullptr, nullptr, nullptr}, st);
    if (rc) return rc;
  }
  return DTV_OK;
}

// The correction pass of a texture plan `fast` against an exact plan `exact`
// of the same geometry: out = BP_exact(sino), e_b = out - BP_fast(sino), one
// launch reading both plans' staged copies of the sinogram.
int backward_refresh_impl(Plan* fast, Plan* exact, const float* sino, int batch, float* out,
                          float* e_b, cudaStream_t st) {
  const GeomParams& gp = fast->gp;
  const int64_t per_item = (int64_t)gp.nu * gp.nv * gp.n_views;
  const int64_t vox = (int64_t)gp.nx * gp.ny * gp.nz;
  for (int b = 0; b < batch; ++b) {
    const float* s = sino + b * per_item;
    // beyond a layered texture's views the fast plan samples records too: no difference
    const bool both = fast->sino_tex != nullptr;
    int rc = both ? stage_sino_tex(fast, s, st) : DTV_OK;
    if (rc) return rc;
    const BPOut dst{out + b * vox, nullptr, both ? e_b + b * vox : nullptr, nullptr};
    rc = bp_view_chunks(fast, both ? kBoth : kRec, exact, s, dst, st);
    if (rc) return rc;
    if (!both) DTV_CUDA_TRY(cudaMemsetAsync(e_b + b * vox, 0, vox * sizeof(float), st));
  }
  return DTV_OK;
}

// ---- several plans' backprojections in one launch ---------------------------------------
// A flat grid over every plan's (column tile, z-chunk) blocks; a block finds
// its plan by the blocks' prefix offsets (kernel parameters, read uniformly).
// The plans' maps travel in the launch parameters too, up to kBPManyViews
// views per launch, so they are read through the constant cache as in the
// single-plan launch. A plan with more views than that reads its maps from its
// device table. Texture plans only; each item's sinogram is first copied into
// its plan's layered array.
constexpr int kBPManyViews = 560;
struct BPManyItem {
  BPParams bp;
  const BPView* views;  // device table (used when map0 < 0)
  cudaTextureObject_t tex;
  float* out;
  int tiles;
  int block0;
  int zaffine;
  int map0;  // first row of this plan's maps in BPMany::m, or -1
};
struct BPMany {
  BPManyItem it[kManyItems];
  int count;
  float m[kBPManyViews][12];
};
static_assert(sizeof(BPMany) <= 31 * 1024, "kernel parameter space");

// Rows of maps in a launch's parameters.
struct RowMaps {
  const float (*r)[12];
  __device__ __forceinline__ const float* row(int jn) const { return r[jn]; }
};

// Every item of one launch has the same S.
template <int S>
__global__ void __launch_bounds__(kBPThreads) bp_many_kernel(const __grid_constant__ BPMany m,
                                                             int accumulate) {
  int k = 0;
  while (k + 1 < m.count && (int)blockIdx.x >= m.it[k + 1].block0) ++k;
  const BPManyItem& it = m.it[k];
  const int local = (int)blockIdx.x - it.block0;
  const int tile = local % it.tiles, zc = local / it.tiles;
  const BPOut dst{it.out, accumulate ? it.out : nullptr, nullptr, nullptr};
  const int nv = it.bp.n_views;
  if (it.map0 >= 0) {
    const RowMaps rows{m.m + it.map0};
    if (it.zaffine) bp_columns<kTex, true, S, false, kZC>(it.bp, rows, 0, nv, nullptr, it.tex, dst, tile, zc);
    else bp_columns<kTex, false, S, false, kZC>(it.bp, rows, 0, nv, nullptr, it.tex, dst, tile, zc);
  } else {
    const TableMaps rows{it.views};
    if (it.zaffine) bp_columns<kTex, true, S, false, kZC>(it.bp, rows, 0, nv, nullptr, it.tex, dst, tile, zc);
    else bp_columns<kTex, false, S, false, kZC>(it.bp, rows, 0, nv, nullptr, it.tex, dst, tile, zc);
  }
}

int backward_many_impl(Plan* const* plans, const float* const* sinos, float* const* outs, int count,
                       int accumulate, cudaStream_t st) {
  BPMany m;
  // plans of one view split share launches
  std::vector<int> ord;
  for (int S = 1; S <= kBPSplits; S *= 2)
    for (int k = 0; k < count; ++k)
      if (bp_split(plans[k]->gp) == S) ord.push_back(k);
  int c0 = 0;
  while (c0 < count) {
    // this launch's plans: up to kManyItems of one split kind, whose maps fit
    // the parameters (a plan with more views than fit at all takes its maps
    // from its table)
    const int S = bp_split(plans[ord[c0]]->gp);
    int cnt = 0, rows = 0;
    while (c0 + cnt < count && cnt < kManyItems) {
      const GeomParams& g = plans[ord[c0 + cnt]]->gp;
      if (bp_split(g) != S) break;
      const int nv = g.n_views;
      if (nv <= kBPManyViews && rows + nv > kBPManyViews) break;
      if (nv <= kBPManyViews) rows += nv;
      ++cnt;
    }
    int64_t blocks = 0;
    int row = 0;
    for (int k = 0; k < cnt; ++k) {
      Plan* p = plans[ord[c0 + k]];
      const GeomParams& gp = p->gp;
      const int rc = stage_sino_tex(p, sinos[ord[c0 + k]], st);
      if (rc) return rc;
      BPManyItem& it = m.it[k];
      it.bp = plan_bp_params(p);
      it.views = p->d_bpv;
      it.tex = p->sino_tex[0];
      it.out = outs[ord[c0 + k]];
      it.tiles = bp_tiles(gp, S);
      it.block0 = (int)blocks;
      it.zaffine = p->bp_zaffine;
      it.map0 = -1;
      if (gp.n_views <= kBPManyViews) {
        it.map0 = row;
        for (int j = 0; j < gp.n_views; ++j) memcpy(m.m[row + j], p->h_bpv[j].m, sizeof(m.m[0]));
        row += gp.n_views;
      }
      blocks += (int64_t)it.tiles * ((gp.nz + kZC - 1) / kZC);
    }
    DTV_CHECK(blocks < 2147483647LL, "too many blocks for one launch");
    m.count = cnt;
    const unsigned nb = (unsigned)blocks;
    const size_t sm = bp_smem(kTex, S, kZC);
    if (S == 8) bp_many_kernel<8><<<nb, kBPThreads, sm, st>>>(m, accumulate);
    else if (S == 4) bp_many_kernel<4><<<nb, kBPThreads, sm, st>>>(m, accumulate);
    else if (S == 2) bp_many_kernel<2><<<nb, kBPThreads, sm, st>>>(m, accumulate);
    else bp_many_kernel<1><<<nb, kBPThreads, sm, st>>>(m, accumulate);
    note_launch();
    DTV_LAUNCH_CHECK();
    c0 += cnt;
  }
  return DTV_OK;
}

}  // namespace dtv
