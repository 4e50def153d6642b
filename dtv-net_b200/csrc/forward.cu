// Ray-driven cone-beam forward projector (all views and batch items in one
// launch) and its exact transpose.
//
// Follows Standard/plug/kernel/forwardKernel.cu:22-86 and
// Beijing/plug/kernel/forwardKernel.cu:17-76: a thread per detector pixel sums
// trilinear samples (border value 0) of the volume at a uniform spacing along
// the source-to-pixel ray and scales the sum. Differences of design:
//   - one launch covers every view and batch item (the reference launched per
//     view after a host sync, forwardKernel.cu:134-136);
//   - the per-ray set-up (ray direction, phase rule, sample range) runs in FP64
//     and the sample loop visits only samples that can touch the volume (the
//     reference marched the whole +-n/2 +-3 world interval, :45-80; skipped
//     samples contribute exactly 0);
//   - the volume is sampled either from a zero-padded staged copy with
//     software trilinear weights in FP32 (exact adjoint available), or through
//     a texture object (hardware filtering, as the reference).
#include <algorithm>
#include <type_traits>
#include <vector>
#include <string.h>

#include "ray.cuh"

namespace dtv {

// ---- samplers --------------------------------------------------------------------------
// The FP16-staged software plans: eight loads from the padded volume.
struct SoftSampler {
  const __half* vol;  // padded volume of this batch item
  int px, pxy;   // padded pitches
  float mx, my, mz;  // clamp maxima (n along each axis)
  __device__ __forceinline__ float operator()(float x, float y, float z) const {
    const float fx = floorf(x), fy = floorf(y), fz = floorf(z);
    const float ax = x - fx, ay = y - fy, az = z - fz;
    const int ix = (int)fminf(fmaxf(fx, -2.f), mx) + kPad;
    const int iy = (int)fminf(fmaxf(fy, -2.f), my) + kPad;
    const int iz = (int)fminf(fmaxf(fz, -2.f), mz) + kPad;
    const __half* b = vol + (iz * pxy + iy * px + ix);
    const float v000 = load_as_float(b, 0), v001 = load_as_float(b, 1);
    const float v010 = load_as_float(b, px), v011 = load_as_float(b, px + 1);
    const float v100 = load_as_float(b, pxy), v101 = load_as_float(b, pxy + 1);
    const float v110 = load_as_float(b, pxy + px), v111 = load_as_float(b, pxy + px + 1);
    const float c00 = fmaf(ax, v001 - v000, v000), c01 = fmaf(ax, v011 - v010, v010);
    const float c10 = fmaf(ax, v101 - v100, v100), c11 = fmaf(ax, v111 - v110, v110);
    const float c0 = fmaf(ay, c01 - c00, c00), c1 = fmaf(ay, c11 - c10, c10);
    return fmaf(az, c1 - c0, c0);
  }
};

// Trilinear samples with FP32 weights from the plan's record copy of the
// volume, z fastest: record (x, y, z) = the bilinear polynomial of the x/y cell
// in plane z, f(ax, ay) = A + ax B + ay C + ax ay D as (A, C, B, D), over the
// grid padded by kPad zero records on every side. A sample loads the two
// adjacent records of planes z and z+1 and interpolates between them.
//
// Why this layout: a 16-byte warp load costs one L1 clock per 128-byte line it
// touches (four at least), and the rays of a warp that share a detector column
// pass through one (x, y) column at neighbouring z. With the lanes of a half
// warp along v they read consecutive records: 5.0 lines per load, against 11.2
// with x fastest and lanes along u. 256^3 x 64 views of 384^2: 6.33 -> 3.28 ms,
// 2.4 G samples, 84 % of the L1 data clocks busy (32 bytes per sample are 8
// clocks per 32 samples at best).
//
// Floors come from rounding-down adds (kIntMagic), whose bits then address the
// record with one 64-bit multiply-add per axis; two samples go through packed
// FP32.

// kFar: a row of records spans 4 GB or more (its pitch needs 64 bits), or an axis has
// 2^22 voxels or more (kIntMagic's sums then round to more than 1): floors by floorf.
template <bool kFar>
struct RecSampler {
  using Pitch = typename std::conditional<kFar, unsigned long long, unsigned int>::type;
  unsigned long long base;  // record (0, 0, 0), biased by the magic bits on each axis (not far)
  Pitch py;                 // bytes from y to y + 1
  unsigned int px;          // bytes from x to x + 1
  float nx, ny, nz;

  __device__ __forceinline__ RecSampler(const RayParams& rp, const float4* rec) {
    px = (unsigned int)(rp.nz + 2 * kPad) * 16u;
    py = (Pitch)px * (Pitch)(rp.nx + 2 * kPad);
    const unsigned long long step = (unsigned long long)py + px + 16u;
    base = (unsigned long long)rec + (unsigned long long)kPad * step -
           (kFar ? 0ull : (unsigned long long)kIntMagicBits * step);
    nx = (float)rp.nx; ny = (float)rp.ny; nz = (float)rp.nz;
  }
  // floors plus kIntMagic (far: floors) in t, fractions in a
  __device__ __forceinline__ float at(float tx, float ty, float tz, float ax, float ay,
                                      float az) const {
    const auto index = [](float t) {
      return kFar ? (unsigned long long)(long long)t : (unsigned long long)__float_as_uint(t);
    };
    const float4* r =
        reinterpret_cast<const float4*>(base + index(ty) * py + index(tx) * px + index(tz) * 16u);
    const float4 lo = __ldg(r), hi = __ldg(r + 1);
    const float s0 = fmaf(ay, fmaf(ax, lo.w, lo.y), fmaf(ax, lo.z, lo.x));
    const float s1 = fmaf(ay, fmaf(ax, hi.w, hi.y), fmaf(ax, hi.z, hi.x));
    return fmaf(az, s1 - s0, s0);
  }
  __device__ __forceinline__ float one(float x, float y, float z) const {
    if constexpr (kFar) {
      const float fx = floorf(x), fy = floorf(y), fz = floorf(z);
      return at(fx, fy, fz, x - fx, y - fy, z - fz);
    }
    const float tx = __fadd_rd(x, kIntMagic), ty = __fadd_rd(y, kIntMagic),
                tz = __fadd_rd(z, kIntMagic);
    return at(tx, ty, tz, x - (tx - kIntMagic), y - (ty - kIntMagic), z - (tz - kIntMagic));
  }
  __device__ __forceinline__ void two(f32x2_t x, f32x2_t y, f32x2_t z, float (&s)[2]) const {
    if constexpr (kFar) {
      float xs[2], ys[2], zs[2];
      unpack2(x, xs[0], xs[1]);
      unpack2(y, ys[0], ys[1]);
      unpack2(z, zs[0], zs[1]);
#pragma unroll
      for (int j = 0; j < 2; ++j) s[j] = one(xs[j], ys[j], zs[j]);
      return;
    }
    const f32x2_t m = splat2(kIntMagic);
    const f32x2_t tx = add2_rm(x, m), ty = add2_rm(y, m), tz = add2_rm(z, m);
    float t[3][2], a[3][2];
    unpack2(tx, t[0][0], t[0][1]);
    unpack2(ty, t[1][0], t[1][1]);
    unpack2(tz, t[2][0], t[2][1]);
    unpack2(sub2(x, sub2(tx, m)), a[0][0], a[0][1]);
    unpack2(sub2(y, sub2(ty, m)), a[1][0], a[1][1]);
    unpack2(sub2(z, sub2(tz, m)), a[2][0], a[2][1]);
#pragma unroll
    for (int j = 0; j < 2; ++j) s[j] = at(t[0][j], t[1][j], t[2][j], a[0][j], a[1][j], a[2][j]);
  }
  // Whether (x, y, z) has its cell's records in the padded grid.
  __device__ __forceinline__ bool holds(float x, float y, float z) const {
    return x >= -2.f && x < nx + 1.f && y >= -2.f && y < ny + 1.f && z >= -2.f && z < nz + 1.f;
  }
  // The sum of a ray's samples, in the order of ray_sum. Positions are monotone
  // along the ray, so the two ends tell whether every sample's records exist
  // (the set-up keeps samples within one step of (-1, n)); a ray of which that
  // is not known, NaN included, tests each sample: one outside (-1, n) is zero.
  __device__ __forceinline__ float sum(const RaySetup& rs) const {
    float a0 = 0.f, a1 = 0.f;
    const float ke = (float)(rs.count - 1);
    if (holds(rs.p0[0], rs.p0[1], rs.p0[2]) &&
        holds(fmaf(ke, rs.dp[0], rs.p0[0]), fmaf(ke, rs.dp[1], rs.p0[1]),
              fmaf(ke, rs.dp[2], rs.p0[2]))) {
      int k = 0;
      f32x2_t kk = f32x2(0.f, 1.f);
      const f32x2_t two2 = splat2(2.f);
      for (; k + 3 < rs.count; k += 4) {
        float s[2][2];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          two(fma2(kk, splat2(rs.dp[0]), splat2(rs.p0[0])),
              fma2(kk, splat2(rs.dp[1]), splat2(rs.p0[1])),
              fma2(kk, splat2(rs.dp[2]), splat2(rs.p0[2])), s[j]);
          kk = add2(kk, two2);
        }
        a0 += s[0][0];
        a1 += s[0][1];
        a0 += s[1][0];
        a1 += s[1][1];
      }
      for (; k < rs.count; ++k) {
        const float kf = (float)k;
        a0 += one(fmaf(kf, rs.dp[0], rs.p0[0]), fmaf(kf, rs.dp[1], rs.p0[1]),
                  fmaf(kf, rs.dp[2], rs.p0[2]));
      }
    } else {
      for (int k = 0; k < rs.count; ++k) {
        const float kf = (float)k;
        const float x = fmaf(kf, rs.dp[0], rs.p0[0]), y = fmaf(kf, rs.dp[1], rs.p0[1]),
                    z = fmaf(kf, rs.dp[2], rs.p0[2]);
        if (x >= -1.f && x < nx && y >= -1.f && y < ny && z >= -1.f && z < nz) a0 += one(x, y, z);
      }
    }
    return a0 + a1;
  }
};

// Texture coordinates: the ray set-up already added the 1/2 texel offset.
struct TexSampler {
  cudaTextureObject_t tex;
  __device__ __forceinline__ float operator()(float x, float y, float z) const {
    return tex3D<float>(tex, x, y, z);
  }
};


// Ray tiles {log2 tu, log2 tv, log2 wu}: a block projects tu x tv detector
// pixels of one view (tu * tv = 256), a warp wu x (32 / wu) of them. The shape
// decides how compact each warp's texture footprint is.
static const int kRayTiles[kNumRayTiles][3] = {{4, 4, 3}, {4, 4, 4}, {5, 3, 5}, {4, 4, 2},
                                               {5, 3, 3}, {3, 5, 3}, {6, 2, 5}, {3, 5, 2}};

// The (ray tile, view) of this block of a (tiles, views) grid. View-major:
// the grid's own order. Band-major (rp.band tile rows per band): blocks in
// launch order take every view of one band of tiles before the next band, so
// the blocks resident at any time sample one slab of the volume.
__device__ __forceinline__ void block_tile_view(const RayParams& rp, int& tile, int& n) {
  if (rp.band <= 0) {
    tile = (int)blockIdx.x;
    n = (int)blockIdx.y;
    return;
  }
  const int tiles = (int)gridDim.x;
  const int tiles_u = (rp.nu + (1 << rp.ltu) - 1) >> rp.ltu;
  const int64_t per_band = (int64_t)tiles_u * rp.band;
  const int64_t lin = (int64_t)blockIdx.y * tiles + blockIdx.x;
  const int64_t band = lin / (per_band * rp.n_views);
  const int64_t r = lin - band * per_band * rp.n_views;
  const int64_t in_band = min(per_band, (int64_t)tiles - band * per_band);  // last band: shorter
  n = (int)(r / in_band);
  tile = (int)(band * per_band + (r - (int64_t)n * in_band));
}

__device__ __forceinline__ void tile_pixel(const RayParams& rp, int& u, int& v, int& n) {
  const int t = threadIdx.x, w = t >> 5, l = t & 31;
  const int tiles_u = (rp.nu + (1 << rp.ltu) - 1) >> rp.ltu;
  int tile;
  block_tile_view(rp, tile, n);
  const int tu = tile % tiles_u, tv = tile / tiles_u;
  const int lwpr = rp.ltu - rp.lwu;  // log2 warps per tile row
  u = (tu << rp.ltu) + ((w & ((1 << lwpr) - 1)) << rp.lwu) + (l & ((1 << rp.lwu) - 1));
  v = (tv << rp.ltv) + ((w >> lwpr) << (5 - rp.lwu)) + (l >> rp.lwu);
}

// The pixel of this thread with a warp's lanes along v first (record samplers:
// consecutive lanes then read consecutive records of one column), 2^lwu columns.
__device__ __forceinline__ void tile_pixel_v(const RayParams& rp, int lwu, int& u, int& v, int& n) {
  const int t = threadIdx.x, w = t >> 5, l = t & 31;
  const int tiles_u = (rp.nu + (1 << rp.ltu) - 1) >> rp.ltu;
  int tile;
  block_tile_view(rp, tile, n);
  const int tu = tile % tiles_u, tv = tile / tiles_u;
  const int lwpr = rp.ltu - lwu, lwv = 5 - lwu;
  u = (tu << rp.ltu) + ((w & ((1 << lwpr) - 1)) << lwu) + (l >> lwv);
  v = (tv << rp.ltv) + ((w >> lwpr) << lwv) + (l & ((1 << lwv) - 1));
}

__global__ void __launch_bounds__(kFPThreads) fp_soft_kernel(RayParams rp, const FPView* __restrict__ views,
                                                             const __half* __restrict__ vpad,
                                                             int64_t pad_elems, FPOut o) {
  int u, v, n;
  tile_pixel(rp, u, v, n);
  const int b = blockIdx.z;
  float res = 0.f;
  const bool live = u < rp.nu && v < rp.nv;
  if (live) {
    const RaySetup rs = setup_ray(rp, views[n], u, v);
    SoftSampler smp;
    smp.vol = vpad + b * pad_elems;
    smp.px = rp.nx + 2 * kPad;
    smp.pxy = smp.px * (rp.ny + 2 * kPad);
    smp.mx = (float)rp.nx; smp.my = (float)rp.ny; smp.mz = (float)rp.nz;
    const float val = rs.count > 0 ? ray_sum(smp, rs) * rp.scale : 0.f;
    fp_store(rp, o, n, b, u, v, val, res);
  }
  if (o.abs_sum) block_add_double((double)fabsf(res), o.abs_sum);
}

// Four blocks per SM: with the bound the compiler uses the 64 registers they
// leave it (56 without: 3.71 -> 3.48 ms at 256^3 x 64 views, in warps of 4 x 8); five or six blocks
// spill (3.67, 4.29 ms).
template <bool kFar>
__global__ void __launch_bounds__(kFPThreads, 4) fp_rec_kernel(RayParams rp,
                                                            const FPView* __restrict__ views,
                                                            const float4* __restrict__ recs,
                                                            int64_t pad_elems, FPOut o) {
  int u, v, n;
  tile_pixel_v(rp, rp.lwu, u, v, n);
  const int b = blockIdx.z;
  float res = 0.f;
  if (u < rp.nu && v < rp.nv) {
    const RaySetup rs = setup_ray(rp, views[n], u, v);
    const RecSampler<kFar> smp(rp, recs + b * pad_elems);
    const float val = rs.count > 0 ? smp.sum(rs) * rp.scale : 0.f;
    fp_store(rp, o, n, b, u, v, val, res);
  }
  if (o.abs_sum) block_add_double((double)fabsf(res), o.abs_sum);
}

__global__ void __launch_bounds__(kFPThreads) fp_tex_kernel(RayParams rp, const FPView* __restrict__ views,
                                                            const cudaTextureObject_t* texs, FPOut o) {
  int u, v, n;
  tile_pixel(rp, u, v, n);
  const int b = blockIdx.z;
  float res = 0.f;
  if (u < rp.nu && v < rp.nv) {
    const RaySetup rs = setup_ray(rp, views[n], u, v, 0.5f, 0.5f);
    TexSampler smp{texs[b]};
    const float val = rs.count > 0 ? ray_sum(smp, rs) * rp.scale : 0.f;
    fp_store(rp, o, n, b, u, v, val, res);
  }
  if (o.abs_sum) block_add_double((double)fabsf(res), o.abs_sum);
}

__global__ void __launch_bounds__(kFPThreads) fp_pair_kernel(RayParams rp, const FPView* __restrict__ views,
                                                             const cudaTextureObject_t* texs,
                                                             FPOut o) {
  int u, v, n;
  tile_pixel(rp, u, v, n);
  const int b = blockIdx.z;
  float res = 0.f;
  if (u < rp.nu && v < rp.nv) {
    const RaySetup rs = setup_ray(rp, views[n], u, v, 0.5f, 0.f);
    PairSampler smp{texs[b], (float)(rp.nz + 2)};
    const float val = rs.count > 0 ? ray_sum(smp, rs) * rp.scale : 0.f;
    fp_store(rp, o, n, b, u, v, val, res);
  }
  if (o.abs_sum) block_add_double((double)fabsf(res), o.abs_sum);
}

// The correction pass of a PDHG reconstruction whose texture-filtered z-pair
// operator A (8-bit weights) is corrected by the exact-weight one E: per ray
//   g_eff = g + (A f - E f),  w = (w + sigma (E f - g)) / (1 + sigma),
//   abs_sum += |E f - g|.
// Each sum has the bits of fp_pair_kernel / fp_rec_kernel for the ray. The
// texture unit wants a quad's lanes on one layer (along u), the records want
// lanes along v: a thread sums one ray of its block's tile through each, in each
// one's order, and the record sums change hands in shared memory.
struct RefreshOut {
  const float* g;
  float* w;
  float* g_eff;
  float sigma;
  double* abs_sum;
};

template <bool kFar>
__global__ void __launch_bounds__(kFPThreads, 4) fp_refresh_kernel(RayParams rp,
                                                                const FPView* __restrict__ views,
                                                                const cudaTextureObject_t* texs,
                                                                const float4* __restrict__ recs,
                                                                int64_t pad_elems, int rec_lwu,
                                                                RefreshOut o) {
  __shared__ float sums[288];  // of the tile's rays, rows padded by one
  int u, v, n, ue, ve;
  tile_pixel(rp, u, v, n);
  tile_pixel_v(rp, rec_lwu, ue, ve, n);
  const int b = blockIdx.z;
  float sf = 0.f, se = 0.f;
  if (u < rp.nu && v < rp.nv) {
    const RaySetup rs = setup_ray(rp, views[n], u, v, 0.5f, 0.f);  // texture coordinates
    const PairSampler fast{texs[b], (float)(rp.nz + 2)};
    if (rs.count > 0) sf = ray_sum(fast, rs);
  }
  if (ue < rp.nu && ve < rp.nv) {
    const RaySetup rs = setup_ray(rp, views[n], ue, ve);  // voxel index coordinates
    const RecSampler<kFar> exact(rp, recs + b * pad_elems);
    if (rs.count > 0) se = exact.sum(rs);
  }
  const int mu = (1 << rp.ltu) - 1, mv = (1 << rp.ltv) - 1;
  sums[(ve & mv) * (mu + 2) + (ue & mu)] = se;
  __syncthreads();
  se = sums[(v & mv) * (mu + 2) + (u & mu)];
  float res = 0.f;
  if (u < rp.nu && v < rp.nv) {
    const float a = sf * rp.scale, e = se * rp.scale;
    const int64_t idx = ((int64_t)b * rp.n_views + n) * rp.nu * rp.nv + (int64_t)v * rp.nu + u;
    const float gi = o.g[idx];
    res = e - gi;
    o.g_eff[idx] = gi + (a - e);
    o.w[idx] = (o.w[idx] + o.sigma * res) / (1.f + o.sigma);
  }
  if (o.abs_sum) block_add_double((double)fabsf(res), o.abs_sum);
}

// Writes the z-pair layers of one volume: layer L = (f[L-2], f[L-1]), zero
// outside [0, nz), to the layered texture and, when `lin` is set, to the
// linear [nz+3][ny][pitch] copy. A thread owns one (x, y) column and a run of
// `layers` layers (grid z), so the whole volume is in flight at once.

template <class Tin>
__global__ void __launch_bounds__(256) stage_pairs_kernel(const Tin* __restrict__ in,
                                                          cudaSurfaceObject_t surf,
                                                          unsigned int* __restrict__ lin, int pitch,
                                                          int64_t lin_plane, int nx, int ny,
                                                          int nz, int layers) {
  const int x = blockIdx.x * 32 + (threadIdx.x & 31);
  const int y = blockIdx.y * 8 + (threadIdx.x >> 5);
  if (x >= nx || y >= ny) return;
  const int L0 = blockIdx.z * layers;
  const int L1 = min(L0 + layers, nz + 3);
  const int64_t plane = (int64_t)nx * ny;
  const Tin* col = in + (int64_t)y * nx + x;
  auto member = [&](int z) {
    return (z >= 0 && z < nz) ? __float2half_rn(load_as_float(col, z * plane))
                              : __float2half_rn(0.f);
  };
  __half prev = member(L0 - 2);  // f[L-2]
#pragma unroll 4
  for (int L = L0; L < L1; ++L) {
    const __half cur = member(L - 1);  // the new member f[L-1]
    const unsigned int bits = (unsigned int)__half_as_ushort(prev) |
                              ((unsigned int)__half_as_ushort(cur) << 16);
    if (surf) surf2DLayeredwrite(bits, surf, x * 4, y, L);
    if (lin) lin[(int64_t)L * lin_plane + (int64_t)y * pitch + x] = bits;
    prev = cur;
  }
}

// ---- staging -------------------------------------------------------------------------
template <class Tin>
__global__ void stage_pad_kernel(const Tin* __restrict__ in, __half* __restrict__ out, int nx,
                                 int ny, int nz, int64_t pad_elems) {
  const int64_t vol = (int64_t)nx * ny * nz;
  const int b = blockIdx.y;
  const int px = nx + 2 * kPad, pxy = px * (ny + 2 * kPad);
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < vol;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(i % nx);
    const int64_t r = i / nx;
    const int y = (int)(r % ny), z = (int)(r / ny);
    const float val = load_as_float(in + b * vol, i);
    store_from_float(out + b * pad_elems, (int64_t)(z + kPad) * pxy + (y + kPad) * px + x + kPad,
                     val);
  }
}

template <class Tin, class Tout>
__global__ void stage_surface_kernel(const Tin* __restrict__ in, cudaSurfaceObject_t surf, int nx,
                                     int ny, int nz) {
  const int64_t vol = (int64_t)nx * ny * nz;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < vol;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(i % nx);
    const int64_t r = i / nx;
    const int y = (int)(r % ny), z = (int)(r / ny);
    if constexpr (sizeof(Tout) == 4) {
      surf3Dwrite(load_as_float(in, i), surf, x * 4, y, z);
    } else {  // half texels are written through their bit pattern
      surf3Dwrite(__half_as_ushort(__float2half_rn(load_as_float(in, i))), surf, x * 2, y, z);
    }
  }
}

static int grid_for(int64_t n, int threads = 256) {
  int64_t b = (n + threads - 1) / threads;
  return (int)std::min<int64_t>(b, 148 * 16);
}

// Writes the records of the volumes (z fastest, see RecSampler): records that
// reach the volume only, x and y in [-1, n-1], z in [0, nz-1]; the others keep
// the plan's initial zeros. A block transposes a tile of 32 x 4 x 32 records
// through shared memory: x runs along the lanes when it reads the volume, z
// when it writes the records. All loads of a thread are in flight together, and
// a column's values serve the records on both sides of it, so that the pass is
// bound by its 16-byte writes: 256^3 62 us (load by load and four shared loads per
// record: 93), 128^3 8.9 (14.6), 24x20x12 2.3 (6.1). kRound: the exact plans'
// FP16-rounded volume.
constexpr int kRecX = 32, kRecY = 4, kRecZ = 32;
template <class Tin, bool kRound>
__global__ void __launch_bounds__(256) stage_rec_kernel(const Tin* __restrict__ in,
                                                        float4* __restrict__ rec, int nx, int ny,
                                                        int nz, int xtiles, int ytiles,
                                                        int64_t pad_elems) {
  __shared__ float s[kRecY + 1][kRecX + 1][kRecZ + 1];
  const int b = blockIdx.y, row = (int)blockIdx.x / xtiles;
  const int x0 = (int)blockIdx.x % xtiles * kRecX - 1, y0 = row % ytiles * kRecY - 1,
            z0 = row / ytiles * kRecZ;
  const Tin* vol = in + (int64_t)b * nx * ny * nz;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  // rows (y, z) of the tile, 33 values from x0: a warp takes four of each y, and its
  // first four lanes their last values; all loads before the first store
  const int64_t zrow = (int64_t)nx * ny;
  float v[kRecY + 1][4], e[kRecY + 1];
#pragma unroll
  for (int yy = 0; yy <= kRecY; ++yy) {
    const int y = y0 + yy;
    const bool yin = y >= 0 && y < ny;
    auto at = [&](int x, int z) {
      float f = yin && z < nz && x >= 0 && x < nx ? load_as_float(vol + z * zrow + (int64_t)y * nx, x) : 0.f;
      if constexpr (kRound) f = __half2float(__float2half_rn(f));
      return f;
    };
#pragma unroll
    for (int j = 0; j < 4; ++j) v[yy][j] = at(x0 + lane, z0 + w + 8 * j);
    e[yy] = lane < 4 ? at(x0 + kRecX, z0 + w + 8 * lane) : 0.f;
  }
#pragma unroll
  for (int yy = 0; yy <= kRecY; ++yy) {
#pragma unroll
    for (int j = 0; j < 4; ++j) s[yy][lane][w + 8 * j] = v[yy][j];
    if (lane < 4) s[yy][kRecX][w + 8 * lane] = e[yy];
  }
  __syncthreads();
  const int z = z0 + lane;
  if (z >= nz) return;
  const int64_t pz = nz + 2 * kPad, py = pz * (nx + 2 * kPad);
  // four columns of x per warp, from one to the next
  float f0[kRecY + 1], f1[kRecY + 1];
#pragma unroll
  for (int yy = 0; yy <= kRecY; ++yy) f0[yy] = s[yy][w * 4][lane];
  float4* out = rec + b * pad_elems + (y0 + kPad) * py + (x0 + w * 4 + kPad) * pz + z + kPad;
#pragma unroll
  for (int k = 0; k < 4; ++k, out += pz) {
    if (x0 + w * 4 + k >= nx) return;
#pragma unroll
    for (int yy = 0; yy <= kRecY; ++yy) f1[yy] = s[yy][w * 4 + k + 1][lane];
#pragma unroll
    for (int yy = 0; yy < kRecY; ++yy) {
      const float B = f1[yy] - f0[yy];
      if (y0 + yy < ny)
        out[yy * py] = make_float4(f0[yy], f0[yy + 1] - f0[yy], B, (f1[yy + 1] - f0[yy + 1]) - B);
    }
#pragma unroll
    for (int yy = 0; yy <= kRecY; ++yy) f0[yy] = f1[yy];
  }
}

template <class Tin, bool kRound>
static int stage_volume_rec(Plan* p, const Tin* vol, int batch, cudaStream_t st) {
  const GeomParams& g = p->gp;
  const int64_t vox = (int64_t)g.nx * g.ny * g.nz;
  // a flat grid of tiles: an axis may have more of them than a grid's y or z holds
  const int xtiles = (g.nx + 1 + kRecX - 1) / kRecX, ytiles = (g.ny + 1 + kRecY - 1) / kRecY;
  const unsigned tiles = (unsigned)xtiles * ytiles * ((g.nz + kRecZ - 1) / kRecZ);
  for (int b = 0; b < batch; b += 65535) {
    const dim3 grid(tiles, std::min(65535, batch - b));
    stage_rec_kernel<Tin, kRound><<<grid, 256, 0, st>>>(vol + b * vox, p->d_vol_rec + b * p->pad_elems,
                                                        g.nx, g.ny, g.nz, xtiles, ytiles, p->pad_elems);
    note_launch();
    DTV_LAUNCH_CHECK();
  }
  return DTV_OK;
}

template <class Tin>
static int stage_volume_soft(Plan* p, const Tin* vol, int batch, cudaStream_t st) {
  const GeomParams& g = p->gp;
  const int64_t vox = (int64_t)g.nx * g.ny * g.nz;
  dim3 grid(grid_for(vox), batch);
  if (p->flags & DTV_PLAN_PAIRS_EXACT) return stage_volume_rec<Tin, true>(p, vol, batch, st);
  if (p->d_vol_rec) return stage_volume_rec<Tin, false>(p, vol, batch, st);
  stage_pad_kernel<Tin><<<grid, 256, 0, st>>>(vol, (__half*)p->d_vol_pad, g.nx, g.ny, g.nz,
                                              p->pad_elems); note_launch();
  DTV_LAUNCH_CHECK();
  return DTV_OK;
}

template <class Tin>
static int stage_volume_tex(Plan* p, const Tin* vol, int batch, cudaStream_t st) {
  const GeomParams& g = p->gp;
  const int64_t vox = (int64_t)g.nx * g.ny * g.nz;
  for (int b = 0; b < batch; ++b) {
    const cudaSurfaceObject_t surf = p->vol_surf[b];
    if (p->stage_dtype == DTV_F16) {
      stage_surface_kernel<Tin, __half><<<grid_for(vox), 256, 0, st>>>(vol + b * vox, surf, g.nx,
                                                                        g.ny, g.nz); note_launch();
    } else {
      stage_surface_kernel<Tin, float><<<grid_for(vox), 256, 0, st>>>(vol + b * vox, surf, g.nx,
                                                                       g.ny, g.nz); note_launch();
    }
    DTV_LAUNCH_CHECK();
  }
  return DTV_OK;
}

template <class Tin>
static int stage_volume_pairs(Plan* p, const Tin* vol, int batch, cudaStream_t st) {
  const GeomParams& g = p->gp;
  const int64_t vox = (int64_t)g.nx * g.ny * g.nz;
  // 16 layers per thread, fewer where that grid has under four blocks per SM
  // (64^3: 5.7 us with 16, 2.3 with 2)
  const int64_t cols = (int64_t)((g.nx + 31) / 32) * ((g.ny + 7) / 8);
  int layers = 16;
  while (layers > 2 && cols * ((g.nz + 3 + layers - 1) / layers) < 4 * 148) layers /= 2;
  dim3 grid((g.nx + 31) / 32, (g.ny + 7) / 8, (g.nz + 3 + layers - 1) / layers);
  for (int b = 0; b < batch; ++b) {
    unsigned int* lin =
        p->d_pair_lin ? p->d_pair_lin + (int64_t)b * p->pair_pitch * g.ny * (g.nz + 3) : nullptr;
    stage_pairs_kernel<Tin><<<grid, 256, 0, st>>>(vol + b * vox, p->pair_surf[b], lin, p->pair_pitch,
                                                  (int64_t)p->pair_pitch * g.ny, g.nx, g.ny, g.nz,
                                                  layers); note_launch();
    DTV_LAUNCH_CHECK();
  }
  return DTV_OK;
}

// Writes batch items 0 .. batch-1 of vol into the plan's staged copy.
static int stage_volume(Plan* p, const void* vol, int vol_dtype, int batch, cudaStream_t st) {
  int rc;
  const bool tex = (p->flags & DTV_PLAN_TEX) != 0;
  const bool pairs = (p->flags & DTV_PLAN_TEX_PAIRS) != 0;
  switch (vol_dtype) {
    case DTV_F32:
      rc = pairs ? stage_volume_pairs(p, (const float*)vol, batch, st)
                 : tex ? stage_volume_tex(p, (const float*)vol, batch, st)
                       : stage_volume_soft(p, (const float*)vol, batch, st);
      break;
    case DTV_F16:
      rc = pairs ? stage_volume_pairs(p, (const __half*)vol, batch, st)
                 : tex ? stage_volume_tex(p, (const __half*)vol, batch, st)
                       : stage_volume_soft(p, (const __half*)vol, batch, st);
      break;
    default:
      rc = pairs ? stage_volume_pairs(p, (const __nv_bfloat16*)vol, batch, st)
                 : tex ? stage_volume_tex(p, (const __nv_bfloat16*)vol, batch, st)
                       : stage_volume_soft(p, (const __nv_bfloat16*)vol, batch, st);
      break;
  }
  return rc;
}

// RecSampler's kFar.
static bool rec_far(const GeomParams& g) {
  return (int64_t)(g.nx + 2 * kPad) * (g.nz + 2 * kPad) * 16 >= (1LL << 32) ||
         std::max(g.nx, std::max(g.ny, g.nz)) + 2 * kPad > kIntMagicMost;
}

// The ray tile of a launch that samples records, {log2 tu, log2 tv, log2 wu}: warps of
// two columns of 16 pixels. A half warp's rays pass one (x, y) column and read its records
// once; lower warps touch more 128-byte lines and one of 32 needs blocks of 32 rows, which
// cross more of the volume at a time. 256^3 x 64 views of 384^2: 2 x 16 3.28 ms, 4 x 8
// 3.49, 1 x 32 3.45, 8 x 4 4.07, 16 x 2 5.90; 151x163x97 x 45 views of 231x149: 0.366,
// 0.387, 0.357 (1 x 32). Of detectors of up to four rows a warp and a block take no more
// rows than there are: 512x512 x 360 views of 768 x 1 2106 -> 587 us, 200x180x3 x 60 views
// of 256 x 3 70 -> 42. From five rows idle lanes can cost less than lower warps do
// (96x96x64 x 45 views of 120 x 8: 31 us in 2 x 16, 41 in 4 x 8).
static void rec_tile(int nv, int (&t)[3]) {
  const int l = nv > 4 ? 4 : nv > 2 ? 2 : nv > 1 ? 1 : 0;
  t[0] = 8 - l;
  t[1] = l;
  t[2] = 5 - l;
}

// `records`: the launch samples records (tile 0, the default, then stands for rec_tile).
static RayParams plan_ray_params(const Plan* p, bool records) {
  RayParams rp = make_ray_params(p->gp);
  int own[3];
  rec_tile(p->gp.nv, own);
  const int* t = records && p->fp_ray_tile == 0 ? own : kRayTiles[p->fp_ray_tile];
  rp.ltu = t[0];
  rp.ltv = t[1];
  rp.lwu = t[2];
  rp.band = p->fp_band;
  return rp;
}

int forward_impl(Plan* p, const void* vol, int vol_dtype, int batch, float* out, int epilogue,
                 const float* g, float sigma, double* abs_sum, cudaStream_t st) {
  const GeomParams& gp = p->gp;
  const bool tex = (p->flags & DTV_PLAN_TEX) != 0;
  const bool pairs = (p->flags & DTV_PLAN_TEX_PAIRS) != 0;
  int rc = stage_volume(p, vol, vol_dtype, batch, st);
  if (rc) return rc;
  const RayParams rp = plan_ray_params(p, p->d_vol_rec != nullptr);
  FPOut o{out, g, sigma, abs_sum, epilogue};
  const int tiles = ((gp.nu + (1 << rp.ltu) - 1) >> rp.ltu) * ((gp.nv + (1 << rp.ltv) - 1) >> rp.ltv);
  dim3 grid(tiles, gp.n_views, batch);
  if (p->flags & DTV_PLAN_TMA) {
    return fp_tma_launch(p, rp, o, batch, st);
  } else if (pairs) {
    fp_pair_kernel<<<grid, kFPThreads, 0, st>>>(rp, p->d_fpv, p->pair_tex_dev, o); note_launch();
  } else if (tex) {
    fp_tex_kernel<<<grid, kFPThreads, 0, st>>>(rp, p->d_fpv, p->vol_tex_dev, o); note_launch();
  } else if (p->d_vol_rec) {
    if (rec_far(gp))
      fp_rec_kernel<true><<<grid, kFPThreads, 0, st>>>(rp, p->d_fpv, p->d_vol_rec, p->pad_elems, o);
    else
      fp_rec_kernel<false><<<grid, kFPThreads, 0, st>>>(rp, p->d_fpv, p->d_vol_rec, p->pad_elems, o);
    note_launch();
  } else {
    fp_soft_kernel<<<grid, kFPThreads, 0, st>>>(rp, p->d_fpv, (const __half*)p->d_vol_pad,
                                                p->pad_elems, o); note_launch();
  }
  DTV_LAUNCH_CHECK();
  return DTV_OK;
}

// The correction pass (fp_refresh_kernel) of a DTV_PLAN_TEX_PAIRS plan `fast`
// and a DTV_PLAN_PAIRS_EXACT plan `exact` of the same geometry: each stages
// the volume into its own copy, one launch projects through both.
int forward_refresh_impl(Plan* fast, Plan* exact, const void* vol, int vol_dtype, int batch,
                         const float* g, float sigma, float* w, float* g_eff, double* abs_sum,
                         cudaStream_t st) {
  const GeomParams& gp = fast->gp;
  int rc = stage_volume(fast, vol, vol_dtype, batch, st);
  if (rc) return rc;
  rc = stage_volume(exact, vol, vol_dtype, batch, st);
  if (rc) return rc;
  RayParams rp = plan_ray_params(fast, false);
  // the record order's columns per warp: two where the tile has 16 rows, as many as the
  // tile takes for detectors of few rows (rec_tile)
  int own[3];
  rec_tile(gp.nv, own);
  const int rec_lwu = std::min(rp.ltu, std::max(own[2], 5 - rp.ltv));
  // band-major plans march bands of one tile row here: with the exact
  // sampler's records beside the z-pairs, the narrower slab keeps more of both
  // in L2 (5.66 ms against 5.74 ms with the plan's 4 rows at 256^3 x 64 views)
  if (rp.band > 0) rp.band = 1;
  const int tiles = ((gp.nu + (1 << rp.ltu) - 1) >> rp.ltu) * ((gp.nv + (1 << rp.ltv) - 1) >> rp.ltv);
  dim3 grid(tiles, gp.n_views, batch);
  const RefreshOut o{g, w, g_eff, sigma, abs_sum};
  if (rec_far(gp))
    fp_refresh_kernel<true><<<grid, kFPThreads, 0, st>>>(rp, fast->d_fpv, fast->pair_tex_dev,
                                                         exact->d_vol_rec, exact->pad_elems, rec_lwu, o);
  else
    fp_refresh_kernel<false><<<grid, kFPThreads, 0, st>>>(rp, fast->d_fpv, fast->pair_tex_dev,
                                                          exact->d_vol_rec, exact->pad_elems, rec_lwu, o);
  note_launch();
  DTV_LAUNCH_CHECK();
  return DTV_OK;
}

// ---- several plans' forward projections in one launch -----------------------------------
// A flat grid over every plan's (view, 16x16-ray tile) blocks, heaviest plans
// first; a block finds its plan by the blocks' prefix offsets (kernel
// parameters, read uniformly) and runs the z-pair sampler of fp_pair_kernel,
// so each ray's sum is the same computation as a single-plan launch.
struct FPManyItem {
  RayParams rp;
  const FPView* views;
  cudaTextureObject_t tex;
  FPOut o;
  int tiles_u, tiles;
  int block0;
};
struct FPMany {
  FPManyItem it[kManyItems];
  int count;
};
static_assert(sizeof(FPMany) <= 31 * 1024, "kernel parameter space");

__global__ void __launch_bounds__(kFPThreads) fp_pair_many_kernel(const __grid_constant__ FPMany m) {
  int k = 0;
  while (k + 1 < m.count && (int)blockIdx.x >= m.it[k + 1].block0) ++k;
  const FPManyItem& it = m.it[k];
  const int local = (int)blockIdx.x - it.block0;
  const int n = local / it.tiles, tile = local % it.tiles;
  const int t = threadIdx.x, w = t >> 5, l = t & 31;
  const int u = (tile % it.tiles_u) * 16 + (w & 1) * 8 + (l & 7);
  const int v = (tile / it.tiles_u) * 16 + (w >> 1) * 4 + (l >> 3);
  const RayParams& rp = it.rp;
  if (u < rp.nu && v < rp.nv) {
    const RaySetup rs = setup_ray(rp, it.views[n], u, v, 0.5f, 0.f);
    PairSampler smp{it.tex, (float)(rp.nz + 2)};
    const float val = rs.count > 0 ? ray_sum(smp, rs) * rp.scale : 0.f;
    float res;
    fp_store(rp, it.o, n, 0, u, v, val, res);
  }
}

int forward_many_impl(Plan* const* plans, const void* const* vols, int vol_dtype, float* const* outs,
                      int count, int epilogue, const float* const* gs, float sigma,
                      cudaStream_t st) {
  for (int k = 0; k < count; ++k) {
    Plan* p = plans[k];
    int rc;
    switch (vol_dtype) {
      case DTV_F32: rc = stage_volume_pairs(p, (const float*)vols[k], 1, st); break;
      case DTV_F16: rc = stage_volume_pairs(p, (const __half*)vols[k], 1, st); break;
      default: rc = stage_volume_pairs(p, (const __nv_bfloat16*)vols[k], 1, st); break;
    }
    if (rc) return rc;
  }
  // heaviest first (rays x volume edge), so the longest blocks start earliest
  std::vector<int> order(count);
  for (int k = 0; k < count; ++k) order[k] = k;
  auto work = [&](int k) {
    const GeomParams& g = plans[k]->gp;
    return (double)g.n_views * g.nu * g.nv * std::max(g.nx, std::max(g.ny, g.nz));
  };
  std::stable_sort(order.begin(), order.end(), [&](int a, int b) { return work(a) > work(b); });
  FPMany m;
  for (int c0 = 0; c0 < count; c0 += kManyItems) {
    const int cnt = std::min(kManyItems, count - c0);
    int64_t blocks = 0;
    for (int j = 0; j < cnt; ++j) {
      const int k = order[c0 + j];
      Plan* p = plans[k];
      const GeomParams& gp = p->gp;
      FPManyItem& it = m.it[j];
      it.rp = make_ray_params(gp);
      it.views = p->d_fpv;
      it.tex = p->pair_tex[0];
      it.o = FPOut{outs[k], gs ? gs[k] : nullptr, sigma, nullptr, epilogue};
      it.tiles_u = (gp.nu + 15) / 16;
      it.tiles = it.tiles_u * ((gp.nv + 15) / 16);
      it.block0 = (int)blocks;
      blocks += (int64_t)it.tiles * gp.n_views;
    }
    DTV_CHECK(blocks < 2147483647LL, "too many blocks for one launch");
    m.count = cnt;
    fp_pair_many_kernel<<<(unsigned)blocks, kFPThreads, 0, st>>>(m);
    note_launch();
    DTV_LAUNCH_CHECK();
  }
  return DTV_OK;
}

// ---- exact transpose of the soft forward projector -------------------------------------
// A^T y scatters every forward sample's value y_r * scale * w_tap onto its 8
// trilinear taps. Instead of 8 global atomics per sample, the volume is cut
// into kAB^3 bricks: one block owns a brick (plus a one-voxel halo) in shared
// memory and, for every view, visits the rays that can reach it -- the
// detector rectangle onto which the brick's box projects, through the view's
// projective map -- rebuilding each ray with the forward projector's own
// set-up and scattering only the samples whose base voxel floor(p) lies in the
// brick (the first brick along an axis also takes base -1, whose upper taps
// are inside). Every contributing sample belongs to exactly one brick, so the
// sum is the exact transpose; each brick then adds its tile to the output once.
// Ray table: rays[2*r] = (p0, count), rays[2*r+1] = (dp, 0) for ray r = (n*nv + v)*nu + u.
__global__ void ray_table_kernel(RayParams rp, const FPView* __restrict__ views,
                                 float4* __restrict__ rays) {
  const int64_t total = (int64_t)rp.n_views * rp.nu * rp.nv;
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < total;
       r += (int64_t)gridDim.x * blockDim.x) {
    const int u = (int)(r % rp.nu);
    const int64_t q = r / rp.nu;
    const int v = (int)(q % rp.nv), n = (int)(q / rp.nv);
    const RaySetup rs = setup_ray(rp, views[n], u, v);
    const int c = rs.count > 0 ? rs.count : 0;
    rays[2 * r] = make_float4(c ? rs.p0[0] : 0.f, c ? rs.p0[1] : 0.f, c ? rs.p0[2] : 0.f,
                              __int_as_float(c));
    rays[2 * r + 1] = make_float4(c ? rs.dp[0] : 0.f, c ? rs.dp[1] : 0.f, c ? rs.dp[2] : 0.f, 0.f);
  }
}

int build_ray_table(Plan* p, cudaStream_t st) {
  RayParams rp = make_ray_params(p->gp);
  const int64_t total = (int64_t)rp.n_views * rp.nu * rp.nv;
  ray_table_kernel<<<grid_for(total), 256, 0, st>>>(rp, p->d_fpv, p->d_rays); note_launch();
  DTV_LAUNCH_CHECK();
  return DTV_OK;
}

constexpr int kAB = 16;         // brick edge (voxels)
constexpr int kAT = kAB + 2;    // tile edge: voxels lo-1 .. lo+kAB
constexpr int kAdjThreads = 256;

template <bool kTable>
__global__ void __launch_bounds__(kAdjThreads) adjoint_brick_kernel(
    RayParams rp, const FPView* __restrict__ views, const BPView* __restrict__ pviews,
    const float4* __restrict__ rays, const float* __restrict__ sino, float* __restrict__ out) {
  __shared__ float tile[kAT * kAT * kAT];
  const int nbx = (rp.nx + kAB - 1) / kAB, nby = (rp.ny + kAB - 1) / kAB;
  const int bid = blockIdx.x;
  const int lo[3] = {(bid % nbx) * kAB, ((bid / nbx) % nby) * kAB, (bid / (nbx * nby)) * kAB};
  const int n3[3] = {rp.nx, rp.ny, rp.nz};
  const int b = blockIdx.y;
  for (int i = threadIdx.x; i < kAT * kAT * kAT; i += blockDim.x) tile[i] = 0.f;
  // base voxels owned by this brick: [blo, bhi] per axis
  float blo[3], bhi[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    blo[c] = lo[c] == 0 ? -1.f : (float)lo[c];
    bhi[c] = (float)(min(lo[c] + kAB, n3[c]) - 1);
  }
  __syncthreads();
  const int64_t per_view = (int64_t)rp.nu * rp.nv;
  const float* sb = sino + (int64_t)b * rp.n_views * per_view;
  for (int n = 0; n < rp.n_views; ++n) {
    // detector rectangle of the box [blo, bhi + 1] through view n
    const float* m = pviews[n].m;
    float umin = 3.4e38f, umax = -3.4e38f, vmin = 3.4e38f, vmax = -3.4e38f;
#pragma unroll
    for (int cr = 0; cr < 8; ++cr) {
      const float x = (cr & 1) ? bhi[0] + 1.f : blo[0];
      const float y = (cr & 2) ? bhi[1] + 1.f : blo[1];
      const float z = (cr & 4) ? bhi[2] + 1.f : blo[2];
      const float h = fmaf(m[8], x, fmaf(m[9], y, fmaf(m[10], z, m[11])));
      const float u = fmaf(m[0], x, fmaf(m[1], y, fmaf(m[2], z, m[3]))) / h;
      const float v = fmaf(m[4], x, fmaf(m[5], y, fmaf(m[6], z, m[7]))) / h;
      umin = fminf(umin, u); umax = fmaxf(umax, u);
      vmin = fminf(vmin, v); vmax = fmaxf(vmax, v);
    }
    const int u0 = max(0, (int)fmaxf(floorf(umin) - 1.f, -1.f));
    const int u1 = min(rp.nu - 1, (int)fminf(ceilf(umax) + 1.f, (float)rp.nu));
    const int v0 = max(0, (int)fmaxf(floorf(vmin) - 1.f, -1.f));
    const int v1 = min(rp.nv - 1, (int)fminf(ceilf(vmax) + 1.f, (float)rp.nv));
    if (u0 > u1 || v0 > v1) continue;
    const int w = u1 - u0 + 1;
    const int cnt = w * (v1 - v0 + 1);
    const float* sv = sb + n * per_view;
    for (int r = threadIdx.x; r < cnt; r += blockDim.x) {  // one ray per thread
      const int u = u0 + r % w, v = v0 + r / w;
      const float y = __ldg(sv + (int64_t)v * rp.nu + u) * rp.scale;
      if (y == 0.f) continue;
      RaySetup rs;
      if constexpr (kTable) {
        const int64_t r2 = 2 * (((int64_t)n * rp.nv + v) * rp.nu + u);
        const float4 a = __ldg(rays + r2), d = __ldg(rays + r2 + 1);
        rs.p0[0] = a.x; rs.p0[1] = a.y; rs.p0[2] = a.z;
        rs.count = __float_as_int(a.w);
        rs.dp[0] = d.x; rs.dp[1] = d.y; rs.dp[2] = d.z;
      } else {
        rs = setup_ray(rp, views[n], u, v);
      }
      if (rs.count <= 0) continue;
      // samples that can have their base in this brick (one-sample margin)
      float kl = 0.f, kh = (float)rs.count;
      bool miss = false;
#pragma unroll
      for (int c = 0; c < 3; ++c) {
        if (rs.dp[c] != 0.f) {
          const float ka = (blo[c] - 1.f - rs.p0[c]) / rs.dp[c];
          const float kb = (bhi[c] + 2.f - rs.p0[c]) / rs.dp[c];
          kl = fmaxf(kl, fminf(ka, kb));
          kh = fminf(kh, fmaxf(ka, kb));
        } else if (rs.p0[c] < blo[c] - 1.f || rs.p0[c] >= bhi[c] + 2.f) {
          miss = true;
        }
      }
      if (miss || !(kh >= kl)) continue;
      const int k0 = max(0, (int)floorf(kl) - 1);
      const int k1 = min(rs.count, (int)ceilf(kh) + 1);
      for (int k = k0; k < k1; ++k) {
        const float kf = (float)k;  // positions exactly as the forward projector forms them
        const float x = fmaf(kf, rs.dp[0], rs.p0[0]), yy = fmaf(kf, rs.dp[1], rs.p0[1]),
                    z = fmaf(kf, rs.dp[2], rs.p0[2]);
        const float fx = floorf(x), fy = floorf(yy), fz = floorf(z);
        if (fx < blo[0] || fx > bhi[0] || fy < blo[1] || fy > bhi[1] || fz < blo[2] ||
            fz > bhi[2])
          continue;
        const float ax = x - fx, ay = yy - fy, az = z - fz;
        const int tx = (int)fx - lo[0] + 1, ty = (int)fy - lo[1] + 1, tz = (int)fz - lo[2] + 1;
        float* t = tile + (tz * kAT + ty) * kAT + tx;
        const float wz1 = az * y, wz0 = y - wz1;
        const float w00 = wz0 - ay * wz0, w01 = ay * wz0, w10 = wz1 - ay * wz1, w11 = ay * wz1;
        atomicAdd(t, w00 - ax * w00);
        atomicAdd(t + 1, ax * w00);
        atomicAdd(t + kAT, w01 - ax * w01);
        atomicAdd(t + kAT + 1, ax * w01);
        atomicAdd(t + kAT * kAT, w10 - ax * w10);
        atomicAdd(t + kAT * kAT + 1, ax * w10);
        atomicAdd(t + kAT * kAT + kAT, w11 - ax * w11);
        atomicAdd(t + kAT * kAT + kAT + 1, ax * w11);
      }
    }
  }
  __syncthreads();
  float* ob = out + (int64_t)b * rp.nx * rp.ny * rp.nz;
  for (int i = threadIdx.x; i < kAT * kAT * kAT; i += blockDim.x) {
    const float val = tile[i];
    if (val == 0.f) continue;
    const int tx = i % kAT, ty = (i / kAT) % kAT, tz = i / (kAT * kAT);
    const int gx = lo[0] - 1 + tx, gy = lo[1] - 1 + ty, gz = lo[2] - 1 + tz;
    if (gx < 0 || gy < 0 || gz < 0 || gx >= rp.nx || gy >= rp.ny || gz >= rp.nz) continue;
    atomicAdd(ob + ((int64_t)gz * rp.ny + gy) * rp.nx + gx, val);
  }
}

// ---- the same transpose with vector atomics into cell records ---------------------------
// Record (ix, iy, z) holds the four contributions of a trilinear cell to the
// voxels (ix, iy, z), (ix+1, iy, z), (ix, iy+1, z), (ix+1, iy+1, z), z fastest
// over the grid padded by kPad on every side (the padded grid of RecSampler,
// so every sample's records exist). A sample of base cell (ix, iy, iz) adds its
// bilinear weights times (1 - az) to record (ix, iy, iz) and times az to record
// (ix, iy, iz+1): two 16-byte vector reductions into L2 instead of eight
// scalar atomics. A gather pass then sums each voxel's four record entries.
//
// The L2 takes reductions by the 32-byte sector, and lanes of one record one
// after the other: two reductions per sample bounded the scatter (2.61 ms for
// 2 x 128^3 x 48 views of 192^2, 18.2 ms for 256^3 x 64 views of 384^2).
// So the lanes of a warp run along v (one column of rays, whose samples of one
// step fall into one (x, y) column at neighbouring z) and merge before they
// reduce: lanes of one base record add up in the run's first lane, and a run's
// upper-plane sums join the next run where that is the next record. With 1.3
// rays per voxel along v, 64 reductions of 32 samples become 25 on consecutive
// records: 1.29 and 9.5 ms, bound by instruction issue (117 per 32 samples, 91 %).
//
// A thread takes NB batch items through the same samples: the positions, records
// and runs are theirs alike (2 x 128^3: 1.32 -> 1.17 ms; adjoint_impl says when).
//
// Five blocks per SM: the bound gives the compiler a few registers more than it took
// (47 against 43; 256^3 9.45 -> 8.98 ms, 128^3 0.697 -> 0.680); six spill (9.48).
//
// kSlab: this launch takes the samples whose base y-cell is in [yb0, yb1).
template <bool kSlab, int NB>
__global__ void __launch_bounds__(256, 5) adjoint_cells_kernel(RayParams rp,
                                                            const FPView* __restrict__ views,
                                                            const float4* __restrict__ rays,
                                                            const float* __restrict__ sino,
                                                            float4* __restrict__ cells,
                                                            int64_t pad_elems, int yb0, int yb1) {
  constexpr unsigned int kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31;
  int u, v, n;
  tile_pixel_v(rp, rp.lwu, u, v, n);
  // z grows with the lane: a detector whose rows run down takes them reversed
  const int wv = 32 >> rp.lwu;
  if (views[n].v[2] < 0.0) v += wv - 1 - 2 * (lane & (wv - 1));
  const int b = (int)blockIdx.z * NB;
  const int64_t per_view = (int64_t)rp.nu * rp.nv, per_item = rp.n_views * per_view;
  const int64_t ray = n * per_view + (int64_t)v * rp.nu + u;
  float val[NB];
#pragma unroll
  for (int i = 0; i < NB; ++i) val[i] = 0.f;
  float4 a = make_float4(0.f, 0.f, 0.f, 0.f), c = a;
  int k0 = 0, k1 = 0;
  const float lo = (float)yb0, hi = (float)yb1;
  const float fnx = (float)rp.nx, fny = (float)rp.ny, fnz = (float)rp.nz;
  bool safe = true;
  if (u < rp.nu && v < rp.nv) {
    bool zero = true;
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      val[i] = __ldg(sino + (b + i) * per_item + ray) * rp.scale;
      zero = zero && val[i] == 0.f;
    }
    if (!zero) {
      a = __ldg(rays + 2 * ray);
      c = __ldg(rays + 2 * ray + 1);
      k1 = __float_as_int(a.w);
      // the k range of the slab from the ray's (monotone) y, widened by one
      if (kSlab && c.y != 0.f) {
        const float inv = 1.f / c.y;
        const float ka = (lo - a.y) * inv, kb = (hi - a.y) * inv;
        const float cnt = (float)k1;  // clamp in float: the estimates may be huge
        k0 = (int)fminf(fmaxf(floorf(fminf(ka, kb)) - 1.f, 0.f), cnt);
        k1 = (int)fminf(fmaxf(ceilf(fmaxf(ka, kb)) + 1.f, 0.f), cnt);
      }
      // positions are monotone: the ends tell whether every record exists; else
      // a sample outside (-1, n), whose forward taps read zeros, is left out
      auto holds = [&](float k) {
        const float x = fmaf(k, c.x, a.x), y = fmaf(k, c.y, a.y), z = fmaf(k, c.z, a.z);
        return x >= -2.f && x < fnx + 1.f && y >= -2.f && y < fny + 1.f && z >= -2.f &&
               z < fnz + 1.f;
      };
      safe = k0 < k1 && holds((float)k0) && holds((float)(k1 - 1));
    }
  }
  const bool any = k0 < k1;
  const int kmin = __reduce_min_sync(kAll, any ? k0 : 0x7fffffff);
  const int kmax = __reduce_max_sync(kAll, any ? k1 : 0);
  const unsigned int pz = (unsigned int)rp.nz + 2 * kPad, pxz = pz * (unsigned int)(rp.nx + 2 * kPad);
  // record (0, 0, 0), biased by the magic bits (modulo 2^32; indices stay below 2^31)
  const unsigned int origin = kPad * (pxz + pz + 1) - kIntMagicBits * (pxz + pz + 1);
  float4* cb = cells + b * pad_elems;
  const bool checked = !__all_sync(kAll, safe || !any);
  const unsigned int len = (unsigned int)(any ? k1 - k0 : 0);
  unsigned int j = (unsigned int)(kmin - k0);  // samples into this ray (wraps below its first)
  float kf = (float)kmin;
  for (int k = kmin; k < kmax; ++k, ++j, kf += 1.f) {
    const float x = fmaf(kf, c.x, a.x), y = fmaf(kf, c.y, a.y), z = fmaf(kf, c.z, a.z);
    const float tx = __fadd_rd(x, kIntMagic), ty = __fadd_rd(y, kIntMagic),
                tz = __fadd_rd(z, kIntMagic);
    const float fy = ty - kIntMagic;
    bool live = j < len;
    if (kSlab) live = live && fy >= lo && fy < hi;
    if (checked)
      live = live && (safe || (x >= -1.f && x < fnx && y >= -1.f && y < fny && z >= -1.f && z < fnz));
    // idle lanes take markers that equal and adjoin no record
    const unsigned int rec = live ? __float_as_uint(ty) * pxz + __float_as_uint(tx) * pz +
                                        __float_as_uint(tz) + origin
                                  : 0xffffff00u + 2u * lane;
    const float ax = x - (tx - kIntMagic), ay = y - fy, az = z - (tz - kIntMagic);
    const unsigned int prec = __shfl_up_sync(kAll, rec, 1);
    const bool first = lane == 0 || prec != rec;
    const unsigned int firsts = __ballot_sync(kAll, first);
    // the last lane of a run of one record
    const bool last = lane == 31 || ((firsts >> lane >> 1) & 1);
    // a run's upper plane joins the next run's lower one where that is the same record
    const bool take = first && lane > 0 && prec + 1 == rec;
    const unsigned int joins = __ballot_sync(kAll, take);
    const bool red_a = live && first, red_b = live && last && !((joins >> lane >> 1) & 1);
    float4* r = cb + rec;
#pragma unroll
    for (int i = 0; i < NB; ++i) {
      const float w1 = val[i] * az, w0 = val[i] - w1;
      const float q0 = w0 * ay, p0 = w0 - q0, q1 = w1 * ay, p1 = w1 - q1;
      float A[4], B[4];
      A[1] = p0 * ax; A[0] = p0 - A[1]; A[3] = q0 * ax; A[2] = q0 - A[3];
      B[1] = p1 * ax; B[0] = p1 - B[1]; B[3] = q1 * ax; B[2] = q1 - B[3];
      // runs: A sums into the run's first lane, B into its last
      unsigned int rest = ~firsts;
      if (rest) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float da = __shfl_down_sync(kAll, A[e], 1), db = __shfl_up_sync(kAll, B[e], 1);
          if (!last) A[e] += da;
          if (!first) B[e] += db;
        }
        rest &= rest << 1;  // runs longer than two
        for (int o = 2; rest; o <<= 1) {
          const unsigned int reach = (1u << o) - 1;  // lanes (l, l + o] start no run
          const bool down = lane + o < 32 && ((firsts >> lane >> 1) & reach) == 0;
          const bool up = lane >= o && ((firsts >> (lane - o + 1)) & reach) == 0;
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const float da = __shfl_down_sync(kAll, A[e], o), db = __shfl_up_sync(kAll, B[e], o);
            if (down) A[e] += da;
            if (up) B[e] += db;
          }
          rest &= rest << o;
        }
      }
      if (joins) {
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          const float d = __shfl_up_sync(kAll, B[e], 1);
          if (take) A[e] += d;
        }
      }
      if (red_a) atomicAdd(r + i * pad_elems, make_float4(A[0], A[1], A[2], A[3]));
      if (red_b) atomicAdd(r + i * pad_elems + 1, make_float4(B[0], B[1], B[2], B[3]));
    }
  }
}

// Each voxel's four record entries, summed. A warp owns 32 slices of one row
// and marches x, reading records along z; the sums go through shared memory so
// that the volume is written along x.
__global__ void __launch_bounds__(256) adjoint_gather_kernel(const float4* __restrict__ cells,
                                                             float* __restrict__ out, int nx,
                                                             int ny, int nz, int xtiles, int ytiles,
                                                             int64_t pad_elems) {
  __shared__ float s[8][32][33];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int b = blockIdx.y, row = (int)blockIdx.x / xtiles;
  const int x0 = (int)blockIdx.x % xtiles * 32, z0 = row / ytiles * 32;
  const int y = row % ytiles * 8 + w;
  const int z = z0 + lane;
  const int64_t pz = nz + 2 * kPad, px = nx + 2 * kPad;
  const int xs = min(32, nx - x0);
  if (y < ny && z < nz) {
    // record (x - 1, y) and (x - 1, y - 1), then march
    const float4* r = cells + b * pad_elems + ((int64_t)(y + kPad) * px + x0 - 1 + kPad) * pz + z + kPad;
    const float4* q = r - px * pz;
    float4 r0 = __ldg(r), q0 = __ldg(q);
    for (int x = 0; x < xs; ++x) {
      const float4 r1 = __ldg(r + (x + 1) * pz), q1 = __ldg(q + (x + 1) * pz);
      s[w][lane][x] = r1.x + r0.y + q1.z + q0.w;
      r0 = r1;
      q0 = q1;
    }
  }
  __syncwarp();
  if (y >= ny || lane >= xs) return;
  float* o = out + ((int64_t)b * nz * ny + y) * nx + x0 + lane;
  for (int k = 0; k < min(32, nz - z0); ++k) o[(int64_t)(z0 + k) * ny * nx] = s[w][k][lane];
}

// ---- the same without merging ------------------------------------------------------------
// For calls that have nothing to merge or too few rays to hide a warp's shuffles: records
// x fastest over the cells that reach the volume (x and y from -1, z in it), threads in
// the rays' own order, along u, so that a warp's reductions of neighbouring rays meet in
// the L2's sectors. Cells by floorf: any axis length. Shared memory that it does not use
// holds it to three blocks per SM: more reductions in flight contend for records (128^3,
// 0.3 detector rows per voxel: 253 us with three blocks, 258 with four, 283 with six;
// 512x512x1, 768 x 1: 545, 574, 604).
constexpr int kScatterSmem = 70 * 1024;
__global__ void __launch_bounds__(256) adjoint_scatter_kernel(float scale, const float4* __restrict__ rays,
                                                              const float* __restrict__ sino,
                                                              float4* __restrict__ cells, int64_t per_item,
                                                              int batch, int nx, int ny, int nz, int zb0,
                                                              int zb1) {
  const int64_t cplane = (int64_t)(nx + 1) * (ny + 1);
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < per_item * batch;
       r += (int64_t)gridDim.x * blockDim.x) {
    const float val = __ldg(sino + r) * scale;
    if (val == 0.f) continue;
    const int64_t b = r / per_item, ray = r - b * per_item;
    const float4 a = __ldg(rays + 2 * ray), c = __ldg(rays + 2 * ray + 1);
    float4* cb = cells + b * cplane * nz;
    // the k range of the slab [zb0, zb1) from the ray's (monotone) z, widened by one
    const int count = __float_as_int(a.w);
    int k0 = 0, k1 = count;
    if (c.z != 0.f) {
      const float inv = 1.f / c.z, ka = ((float)zb0 - a.z) * inv, kb = ((float)zb1 - a.z) * inv;
      const float n = (float)count;  // clamp in float: the estimates may be huge
      k0 = (int)fminf(fmaxf(floorf(fminf(ka, kb)) - 1.f, 0.f), n);
      k1 = (int)fminf(fmaxf(ceilf(fmaxf(ka, kb)) + 1.f, 0.f), n);
    }
    for (int k = k0; k < k1; ++k) {
      const float kf = (float)k;
      const float x = fmaf(kf, c.x, a.x), y = fmaf(kf, c.y, a.y), z = fmaf(kf, c.z, a.z);
      const float fx = floorf(x), fy = floorf(y), fz = floorf(z);
      const int ix = (int)fx, iy = (int)fy, iz = (int)fz;
      if (iz < zb0 || iz >= zb1 || ix < -1 || ix >= nx || iy < -1 || iy >= ny) continue;
      const float ax = x - fx, ay = y - fy, az = z - fz, bx = 1.f - ax, by = 1.f - ay;
      float4* cell = cb + (int64_t)(iy + 1) * (nx + 1) + ix + 1;
      if (iz >= 0) {
        const float w = val * (1.f - az);
        atomicAdd(cell + iz * cplane, make_float4(w * bx * by, w * ax * by, w * bx * ay, w * ax * ay));
      }
      if (iz + 1 < nz) {
        const float w = val * az;
        atomicAdd(cell + (iz + 1) * cplane,
                  make_float4(w * bx * by, w * ax * by, w * bx * ay, w * ax * ay));
      }
    }
  }
}

__global__ void __launch_bounds__(256) adjoint_scatter_gather_kernel(const float4* __restrict__ cells,
                                                                     float* __restrict__ out, int nx, int ny,
                                                                     int64_t total) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total;
       i += (int64_t)gridDim.x * blockDim.x) {
    const int x = (int)(i % nx);
    const int64_t q = i / nx, z = q / ny;  // z over the whole batch
    const int y = (int)(q - z * ny);
    const float4* r = cells + ((z * (ny + 1) + y + 1) * (nx + 1) + x + 1);  // cell (x, y)
    out[i] = __ldg(&r->x) + __ldg(&r[-1].y) + __ldg(&r[-(nx + 1)].z) + __ldg(&r[-(nx + 1) - 1].w);
  }
}

static int adjoint_scatter(Plan* p, const float* sino, int batch, float* out, cudaStream_t st) {
  const GeomParams& gp = p->gp;
  const int64_t cplane = (int64_t)(gp.nx + 1) * (gp.ny + 1);
  DTV_CUDA_TRY(cudaMemsetAsync(p->d_cells, 0, cplane * gp.nz * batch * sizeof(float4), st));
  const int64_t rays = (int64_t)gp.n_views * gp.nu * gp.nv;
  const int grid = (int)std::min<int64_t>((rays * batch + 255) / 256, 148LL * 64);
  // z-slabs whose records (at most 72 MB over the batch) stay in L2; cells from z = -1
  const int slab = (int)std::max<int64_t>(1, (72LL << 20) / (cplane * (int64_t)sizeof(float4) * batch));
  DTV_CUDA_TRY(cudaFuncSetAttribute(adjoint_scatter_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    kScatterSmem));
  for (int zb0 = -1; zb0 < gp.nz; zb0 += slab) {
    adjoint_scatter_kernel<<<grid, 256, kScatterSmem, st>>>((float)gp.scale, p->d_rays, sino, p->d_cells, rays, batch,
                                                 gp.nx, gp.ny, gp.nz, zb0, std::min(zb0 + slab, gp.nz));
    note_launch();
    DTV_LAUNCH_CHECK();
  }
  const int64_t total = (int64_t)gp.nx * gp.ny * gp.nz * batch;
  adjoint_scatter_gather_kernel<<<(int)std::min<int64_t>((total + 255) / 256, 148LL * 32), 256, 0, st>>>(
      p->d_cells, out, gp.nx, gp.ny, total);
  note_launch();
  DTV_LAUNCH_CHECK();
  return DTV_OK;
}

// Detector rows per voxel along z, seen from the volume's centre, over a sample of views.
float adjoint_rows(const Plan* p) {
  const GeomParams& gp = p->gp;
  const double x = 0.5 * (gp.nx - 1), y = 0.5 * (gp.ny - 1), z = 0.5 * (gp.nz - 1);
  double sum = 0.0;
  int n = 0;
  for (int i = 0; i < gp.n_views; i += std::max(1, gp.n_views / 48), ++n) {
    const float* m = p->h_bpv[i].m;
    const double h = m[8] * x + m[9] * y + m[10] * z + m[11];
    const double v = m[4] * x + m[5] * y + m[6] * z + m[7];
    const double d = fabs((m[6] * h - m[10] * v) / (h * h));
    if (d < 1e6) sum += d;  // (NaN and infinity of a source plane through the centre left out)
  }
  return (float)(sum / n);
}

int adjoint_impl(Plan* p, const float* sino, int batch, float* out, cudaStream_t st) {
  const GeomParams& gp = p->gp;
  RayParams rp = make_ray_params(gp);
  const int64_t vox = (int64_t)gp.nx * gp.ny * gp.nz;
  if (p->adjoint_method == 1 && p->d_cells) {
    // Merging pays from about half a detector row per voxel on, where the rows fill a
    // warp's eight lanes, and with enough warps to hide its shuffles: below 3500 (a call
    // of 1300 at 40^3, 1.2 rows per voxel: 25.0 us without, 28.0 with; 2600: 36.6, 34.3;
    // 5400 at 64^3: 84, 60), on few rows (512x512 x 360 views of 768 x 1: 545, 2288) or
    // sparse ones (0.3 per voxel, 96^3: 95, 145; 128^3: 257, 310; 0.46: 1180, 1152) the
    // plain scatter is the faster one. Axes beyond kIntMagicMost have it too.
    const int64_t warps = (int64_t)gp.n_views * gp.nu * gp.nv / 32;
    const bool wide = std::max(gp.nx, std::max(gp.ny, gp.nz)) + 2 * kPad > kIntMagicMost;
    if (p->adjoint_rows < 0.4f || gp.nv < 5 || warps * batch < 3500 || wide)
      return adjoint_scatter(p, sino, batch, out, st);
    // Two items per thread where many rays share records: 2 x 96^3, 1.2 rows per voxel,
    // 18600 warps: 287 us, 304 singly; 0.9: 267, 248; 2 x 64^3, 1.2, 5400 warps: 94, 89.
    const bool pairs = p->adjoint_rows >= 1.1f && warps >= 9000;
    DTV_CUDA_TRY(cudaMemsetAsync(p->d_cells, 0, p->pad_elems * batch * sizeof(float4), st));
    // warps of 4 x 8 rays: 128^3 x 48 views 0.68 ms (1 x 32: 0.73, 2 x 16: 0.69;
    // 97x113x61 x 33 views: 271, 334, 291 us)
    rp.ltu = kRayTiles[3][0];
    rp.ltv = kRayTiles[3][1];
    rp.lwu = kRayTiles[3][2];
    const int tiles = ((gp.nu + (1 << rp.ltu) - 1) >> rp.ltu) * ((gp.nv + (1 << rp.ltv) - 1) >> rp.ltv);
    // y-slabs of base cells whose records (at most 160 MB over the batch) stay
    // in L2 while their samples scatter; cells run over [-2, ny]. 256^3 x 64
    // views of 384^2: 9.51 ms (slabs of 72 MB 9.80, none 10.63)
    const int64_t row_bytes = (int64_t)(gp.nx + 2 * kPad) * (gp.nz + 2 * kPad) * sizeof(float4) * batch;
    const int64_t rows = std::max<int64_t>(1, (160LL << 20) / row_bytes);
    const int slabs = (int)((gp.ny + 3 + rows - 1) / rows);
    const int slab = (gp.ny + 3 + slabs - 1) / slabs;
    const int64_t per_view = (int64_t)gp.nu * gp.nv, per_item = gp.n_views * per_view;
    for (int yb = -2; yb <= gp.ny; yb += slab) {
      const int ye = std::min(yb + slab, gp.ny + 1);
      for (int v0 = 0; v0 < gp.n_views; v0 += 65535) {  // views in the grid's y
        const int nv = std::min(65535, gp.n_views - v0);
        auto scatter = [&](auto kernel, int first, int z) {  // items from `first`
          kernel<<<dim3(tiles, nv, z), 256, 0, st>>>(
              rp, p->d_fpv + v0, p->d_rays + 2 * v0 * per_view, sino + v0 * per_view + first * per_item,
              p->d_cells + first * p->pad_elems, p->pad_elems, yb, ye);
          note_launch();
          DTV_LAUNCH_CHECK();
          return (int)DTV_OK;
        };
        const int two = pairs ? batch / 2 : 0;
        int rc = DTV_OK;
        if (two > 0)
          rc = scatter(slabs > 1 ? adjoint_cells_kernel<true, 2> : adjoint_cells_kernel<false, 2>, 0, two);
        if (!rc && batch > 2 * two)
          rc = scatter(slabs > 1 ? adjoint_cells_kernel<true, 1> : adjoint_cells_kernel<false, 1>, 2 * two,
                       batch - 2 * two);
        if (rc) return rc;
      }
    }
    const int xtiles = (gp.nx + 31) / 32, ytiles = (gp.ny + 7) / 8;
    const unsigned gtiles = (unsigned)xtiles * ytiles * ((gp.nz + 31) / 32);
    for (int b = 0; b < batch; b += 65535) {
      const dim3 grid(gtiles, std::min(65535, batch - b));
      adjoint_gather_kernel<<<grid, 256, 0, st>>>(p->d_cells + b * p->pad_elems, out + b * vox,
                                                  gp.nx, gp.ny, gp.nz, xtiles, ytiles, p->pad_elems);
      note_launch();
      DTV_LAUNCH_CHECK();
    }
    return DTV_OK;
  }
  const int bricks = ((gp.nx + kAB - 1) / kAB) * ((gp.ny + kAB - 1) / kAB) *
                     ((gp.nz + kAB - 1) / kAB);
  DTV_CUDA_TRY(cudaMemsetAsync(out, 0, vox * batch * sizeof(float), st));
  if (p->d_rays) {
    adjoint_brick_kernel<true><<<dim3(bricks, batch), kAdjThreads, 0, st>>>(
        rp, p->d_fpv, p->d_bpv, p->d_rays, sino, out); note_launch();
  } else {
    adjoint_brick_kernel<false><<<dim3(bricks, batch), kAdjThreads, 0, st>>>(
        rp, p->d_fpv, p->d_bpv, nullptr, sino, out); note_launch();
  }
  DTV_LAUNCH_CHECK();
  return DTV_OK;
}

}  // namespace dtv
