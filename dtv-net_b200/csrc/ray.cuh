// Ray set-up shared by the forward projectors: the phase rules of the
// reference's ray marchers restated on the unified per-view geometry, the
// projector output epilogues and the per-ray sample loop.
#pragma once

#include "common.cuh"

namespace dtv {

struct RayParams {
  int nx, ny, nz, nu, nv, n_views;
  int phase;
  double voxel[3];
  double step, inv_step;
  float scale;
  // ray tile of a block (tu x tv pixels) and of a warp (wu x wv = 32), log2
  int ltu, ltv, lwu;
  int band;  // tile rows per band of the band-major block order; 0: view-major
};

inline RayParams make_ray_params(const GeomParams& gp) {
  RayParams r;
  r.nx = gp.nx; r.ny = gp.ny; r.nz = gp.nz;
  r.nu = gp.nu; r.nv = gp.nv; r.n_views = gp.n_views;
  r.phase = gp.phase;
  for (int c = 0; c < 3; ++c) r.voxel[c] = gp.voxel[c];
  r.step = gp.step;
  r.inv_step = 1.0 / gp.step;
  r.scale = (float)gp.scale;
  r.ltu = 4; r.ltv = 4; r.lwu = 3;
  r.band = 0;
  return r;
}

// Per-ray set-up: the first sample position and step (index space) and the
// number of samples that can be non-zero.
struct RaySetup {
  float p0[3];
  float dp[3];
  int count;
};

// 1 / x in FP64: the hardware's approximation (about 20 bits) refined by two
// Newton steps r + r (1 - x r).
__device__ __forceinline__ double rcp64(double x) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  r = __fma_rn(r, __fma_rn(-x, r, 1.0), r);
  return __fma_rn(r, __fma_rn(-x, r, 1.0), r);
}
// x / d from q = 1 / d: the quotient corrected by its remainder (Markstein 1990).
__device__ __forceinline__ double div64(double x, double d, double q) {
  const double t = __dmul_rn(x, q);
  return __fma_rn(__fma_rn(-t, d, x), q, t);
}

// `sxy` / `sz` are added to the start position's x,y / z (1/2 where the
// sampler takes texture coordinates, whose texel centres sit at i + 1/2).
//
// Short rays spend as much on this as on their samples: with twelve divisions
// and an indexed axis in local memory it was some 800 of a warp's 1900
// instructions at 64^3 x 60 views (z-pair texture, 81 us; now 74 us and 1600,
// 78 % of the texture unit's rate). One reciprocal q = 1/d per axis serves its four
// quotients, and the sign of d says which of an axis's two planes comes first.
// The chord, whose length in steps is rounded up, keeps divisions' rounding: a
// ray along an axis crosses a whole number of steps. Every step rounds
// explicitly, so that all kernels set a ray up to the same bits.
__device__ __forceinline__ RaySetup setup_ray(const RayParams& rp, const FPView& f, int u, int v,
                                              float sxy = 0.f, float sz = 0.f) {
  RaySetup rs;
  double r[3], rw[3], d[3], q[3], A[3];
  const double du = (double)u, dv = (double)v;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    r[c] = __fma_rn(dv, f.v[c], __fma_rn(du, f.u[c], f.d0ms[c]));
    rw[c] = __dmul_rn(r[c], rp.voxel[c]);
  }
  const double inv = rsqrt(__fma_rn(rw[2], rw[2], __fma_rn(rw[1], rw[1], __dmul_rn(rw[0], rw[0]))));
  const int n3[3] = {rp.nx, rp.ny, rp.nz};
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    d[c] = __dmul_rn(r[c], inv);  // index units per world unit of alpha
    q[c] = rcp64(d[c]);
    A[c] = -__dmul_rn(f.s[c], q[c]);
  }
  double a0, ktot;
  if (rp.phase == DTV_PHASE_BOX) {
    double lo = -1e300, hi = 1e300;
    bool miss = false;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double e = n3[c] - 0.5;
      if (d[c] == 0.0) {
        miss = miss || f.s[c] < -0.5 || f.s[c] > e;
      } else {
        const bool up = d[c] > 0.0;
        lo = fmax(lo, div64(__dadd_rn(up ? -0.5 : e, -f.s[c]), d[c], q[c]));
        hi = fmin(hi, div64(__dadd_rn(up ? e : -0.5, -f.s[c]), d[c], q[c]));
      }
    }
    if (miss || !(hi > lo)) {
      rs.count = 0;
      return rs;
    }
    ktot = ceil(div64(__dadd_rn(hi, -lo), rp.step, rp.inv_step));
    a0 = __fma_rn(0.5, rp.step, lo);
  } else {
    // the dominant axis of the world direction
    const double wx = fabs(rw[0]), wy = fabs(rw[1]), wz = fabs(rw[2]);
    int ax;
    if (rp.phase == DTV_PHASE_STANDARD) {
      ax = wx >= wy ? 0 : 1;  // Standard forwardKernel.cu:45
    } else {                  // Beijing forwardKernel.cu:40-58
      const double dom = fmax(wx, fmax(wz, wy));
      ax = wx == dom ? 0 : (wy == dom ? 1 : 2);
    }
    // bounds +-n/2 in WORLD units against the world source (the reference's
    // alpha range, forwardKernel.cu:46-58)
    const double e = 0.5 * (ax == 0 ? rp.nx : (ax == 1 ? rp.ny : rp.nz));
    const double sw = ax == 0 ? f.sw[0] : (ax == 1 ? f.sw[1] : f.sw[2]);
    const double dw = __dmul_rn(ax == 0 ? rw[0] : (ax == 1 ? rw[1] : rw[2]), inv);
    const double qw = rcp64(dw);
    const double t0 = __dmul_rn(__dadd_rn(-e, -sw), qw), t1 = __dmul_rn(__dadd_rn(e, -sw), qw);
    const double lo = __dadd_rn(fmin(t0, t1), -3.0), hi = __dadd_rn(fmax(t0, t1), 3.0);
    a0 = lo;
    ktot = ceil(__dmul_rn(__dadd_rn(hi, -lo), rp.inv_step));
  }
  // clip k to samples whose position lies in (-1, n) on every axis
  double alo = a0, ahi = 1e300;
  bool out = false;
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    const double n = n3[c];
    if (fabs(d[c]) * rp.step < 1e-12) {
      const double base = __fma_rn(a0, d[c], f.s[c]);
      out = out || base <= -1.0 || base >= n;
    } else {
      const bool up = d[c] > 0.0;
      alo = fmax(alo, __fma_rn(up ? -1.0 : n, q[c], A[c]));
      ahi = fmin(ahi, __fma_rn(up ? n : -1.0, q[c], A[c]));
    }
  }
  const double kb = floor(__dmul_rn(__dadd_rn(alo, -a0), rp.inv_step));
  const double ke = fmin(ceil(__dmul_rn(__dadd_rn(ahi, -a0), rp.inv_step)) + 1.0, ktot);
  if (out || !(ke > kb)) {
    rs.count = 0;
    return rs;
  }
  rs.count = (int)(ke - kb);
  const double ab = __fma_rn(kb, rp.step, a0);
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    rs.p0[c] = (float)__dadd_rn(__fma_rn(ab, d[c], f.s[c]), (double)(c < 2 ? sxy : sz));
    rs.dp[c] = (float)__dmul_rn(d[c], rp.step);
  }
  return rs;
}

struct FPOut {
  float* out;
  const float* g;
  float sigma;
  double* abs_sum;
  int epilogue;
};

constexpr int kFPThreads = 256;

__device__ __forceinline__ void block_add_double(double val, double* dst) {
  __shared__ double red[kFPThreads / 32];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) val += __shfl_xor_sync(0xffffffffu, val, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = val;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int i = 0; i < kFPThreads / 32; ++i) s += red[i];
    if (s != 0.0) atomicAdd(dst, s);
  }
}

template <class Sampler>
__device__ __forceinline__ float ray_sum(const Sampler& smp, const RaySetup& rs) {
  float a0 = 0.f, a1 = 0.f;
  int k = 0;
  float kb = 0.f;  // (float)k, advanced by exact integer additions
  for (; k + 3 < rs.count; k += 4, kb += 4.f) {
    float s[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float kf = kb + (float)j;
      s[j] = smp(fmaf(kf, rs.dp[0], rs.p0[0]), fmaf(kf, rs.dp[1], rs.p0[1]),
                 fmaf(kf, rs.dp[2], rs.p0[2]));
    }
    a0 += s[0];
    a1 += s[1];
    a0 += s[2];
    a1 += s[3];
  }
  for (; k < rs.count; ++k) {
    const float kf = (float)k;
    a0 += smp(fmaf(kf, rs.dp[0], rs.p0[0]), fmaf(kf, rs.dp[1], rs.p0[1]),
              fmaf(kf, rs.dp[2], rs.p0[2]));
  }
  return a0 + a1;
}

// z-pair sampler through the texture unit: layer L of the half2 layered
// texture holds (f[L-2], f[L-1]). x, y arrive as texture coordinates (shifted
// by 1/2), z as a voxel index.
struct PairSampler {
  cudaTextureObject_t tex;
  float lmax;  // nz + 2, the last layer
  __device__ __forceinline__ float operator()(float x, float y, float z) const {
    const float fz = floorf(z);
    const float w = z - fz;
    const float L = fminf(fmaxf(fz + 2.f, 0.f), lmax);
    const float2 a = tex2DLayered<float2>(tex, x, y, (int)L);
    return fmaf(w, a.y - a.x, a.x);
  }
};

__device__ __forceinline__ void fp_store(const RayParams& rp, const FPOut& o, int n, int b, int u,
                                         int v, float val, float& res) {
  const int64_t idx = ((int64_t)b * rp.n_views + n) * rp.nu * rp.nv + (int64_t)v * rp.nu + u;
  if (o.epilogue == DTV_EPI_STORE) {
    o.out[idx] = val;
    res = val;
  } else {
    res = val - o.g[idx];
    if (o.epilogue == DTV_EPI_RESIDUAL) o.out[idx] = res;
    else o.out[idx] = (o.out[idx] + o.sigma * res) / (1.f + o.sigma);
  }
}

// Shared-memory staged z-pair forward projector (forward_tma.cu).
int fp_tma_launch(Plan* p, const RayParams& rp, const FPOut& o, int batch, cudaStream_t st);

}  // namespace dtv
