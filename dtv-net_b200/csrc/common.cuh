// Internal definitions shared by the library's translation units.
#pragma once

#include <cuda_runtime.h>
#include <cuda_fp16.h>
#include <cuda_bf16.h>
#include <stdint.h>

#include <string>

#include "dtv_b200.h"

namespace dtv {

// ---- error reporting -------------------------------------------------------------
// Host-side count of kernel launches issued by the library (dtv_launch_count).
void note_launch();
void set_error(const char* fmt, ...);
int fail(int code, const char* fmt, ...);

#define DTV_CUDA_TRY(expr)                                                             \
  do {                                                                                 \
    cudaError_t _e = (expr);                                                           \
    if (_e != cudaSuccess)                                                             \
      return ::dtv::fail(DTV_ERR_CUDA, "%s failed: %s (%s:%d)", #expr,                 \
                         cudaGetErrorString(_e), __FILE__, __LINE__);                  \
  } while (0)

#define DTV_CHECK(cond, ...)                                                           \
  do {                                                                                 \
    if (!(cond)) return ::dtv::fail(DTV_ERR_INVALID, __VA_ARGS__);                     \
  } while (0)

// Launch-error check right after a kernel launch.
#define DTV_LAUNCH_CHECK()                                                             \
  do {                                                                                 \
    cudaError_t _e = cudaGetLastError();                                               \
    if (_e != cudaSuccess)                                                             \
      return ::dtv::fail(DTV_ERR_CUDA, "kernel launch failed: %s (%s:%d)",             \
                         cudaGetErrorString(_e), __FILE__, __LINE__);                  \
  } while (0)

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// ---- storage types -------------------------------------------------------------------
__device__ __forceinline__ float load_as_float(const float* p, int64_t i) { return __ldg(p + i); }
__device__ __forceinline__ float load_as_float(const __half* p, int64_t i) {
  return __half2float(p[i]);
}
__device__ __forceinline__ float load_as_float(const __nv_bfloat16* p, int64_t i) {
  return __bfloat162float(p[i]);
}
__device__ __forceinline__ void store_from_float(float* p, int64_t i, float v) { p[i] = v; }
__device__ __forceinline__ void store_from_float(__half* p, int64_t i, float v) {
  p[i] = __float2half_rn(v);
}
__device__ __forceinline__ void store_from_float(__nv_bfloat16* p, int64_t i, float v) {
  p[i] = __float2bfloat16_rn(v);
}

// The half2 held in a 32-bit word (low half first, as surface and linear
// z-pair copies store it).
__device__ __forceinline__ __half2 u32_as_half2(unsigned int w) {
  return __halves2half2(__ushort_as_half((unsigned short)(w & 0xFFFFu)),
                        __ushort_as_half((unsigned short)(w >> 16)));
}

// Packed FP32 pairs (Blackwell's two-lane FP32 arithmetic); each lane rounds as
// the scalar instruction does.
using f32x2_t = unsigned long long;
__device__ __forceinline__ f32x2_t f32x2(float lo, float hi) {
  f32x2_t r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ f32x2_t splat2(float v) { return f32x2(v, v); }
__device__ __forceinline__ void unpack2(f32x2_t v, float& lo, float& hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f32x2_t add2(f32x2_t a, f32x2_t b) {
  f32x2_t r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2_t add2_rm(f32x2_t a, f32x2_t b) {  // rounding down
  f32x2_t r;
  asm("add.rm.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2_t sub2(f32x2_t a, f32x2_t b) {
  f32x2_t r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2_t mul2(f32x2_t a, f32x2_t b) {
  f32x2_t r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ f32x2_t fma2(f32x2_t a, f32x2_t b, f32x2_t c) {
  f32x2_t r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// Adding 1.5 * 2^23 leaves an integer in the sum's low bits; with rounding down
// the sum is the floor. The float to integer conversions this replaces run at
// a quarter rate.
constexpr float kIntMagic = 12582912.f;
constexpr unsigned int kIntMagicBits = 0x4B400000u;
constexpr int kIntMagicMost = 1 << 22;  // beyond it the sums' steps are more than 1

// 1 / x by one Newton step r + r (1 - x r) on the approximate reciprocal. kAny: x may
// be zero or infinite, where 1 - x r is no remainder and r, infinite or zero, stands.
template <bool kAny>
__device__ __forceinline__ float rcp_newton(float x) {
  float r;
  asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
  const float e = fmaf(-x, r, 1.f);
  return kAny && !(fabsf(e) < 1.f) ? r : fmaf(r, e, r);
}

inline int dtype_size(int dt) { return dt == DTV_F32 ? 4 : 2; }
inline bool dtype_ok(int dt) { return dt == DTV_F32 || dt == DTV_F16 || dt == DTV_BF16; }

// ---- per-view tables (built in FP64 on the host) ------------------------------------
// Forward projector, index space (voxel (i,j,k) centred at (i,j,k)):
//   ray to pixel (u,v): r = d0ms + u*U + v*V   (d0ms = pixel(0,0) centre - source)
//   source S (index) and Sw (world) for the phase rule.
struct FPView {
  double s[3];     // source, index coordinates
  double sw[3];    // source, world coordinates
  double d0ms[3];  // pixel (0,0) centre minus source, index coordinates
  double u[3];     // one pixel step along u, index coordinates
  double v[3];     // one pixel step along v, index coordinates
  double pad;
};
static_assert(sizeof(FPView) == 128, "FPView layout");

// Backprojector: projective map from voxel index (i,j,k,1):
//   h = m[8..11].x, u = m[0..3].x / h, v = m[4..7].x / h (pixel-index coordinates),
//   weight = bp_scale * h^-power, with h = L / SDD (distances along the normal).
struct BPView {
  float m[12];
  float pad[4];
};
static_assert(sizeof(BPView) == 64, "BPView layout");

struct GeomParams {
  int nx, ny, nz, nu, nv, n_views;
  int phase;
  int bp_power;
  int bp_extent;
  double voxel[3];
  double vol_offset[3];
  double det_offset[2];
  double step, scale, bp_scale;
};

// Host helpers (geometry.cu)
int build_tables(const dtv_geometry* g, GeomParams* gp, FPView* fpv, BPView* bpv);
int validate_geometry(const dtv_geometry* g);
double count_fp_samples(const GeomParams& gp, const FPView* fpv);

// ---- plans -----------------------------------------------------------------------------
struct Plan {
  int device;
  int flags;
  int max_batch;
  GeomParams gp;
  FPView* d_fpv;  // device
  BPView* d_bpv;  // device
  BPView* h_bpv;  // host copy (the backprojector passes the maps as launch parameters)
  // FP16-staged soft plans: zero-padded volumes (border kPad) of max_batch items
  void* d_vol_pad;
  // FP32 soft and exact plans: 16-byte records of the x/y cells, z fastest, over
  // the same padded grid (forward.cu RecSampler), read instead of d_vol_pad
  float4* d_vol_rec;
  int stage_dtype;    // DTV_F32 or DTV_F16
  int64_t pad_elems;  // elements of one padded volume
  // backprojector: the sinogram of one batch item as 16-byte records (one
  // bilinear detector cell each) or, texture plans, a layered array
  float4* d_sino_rec;
  int sino_rec_views;  // views that d_sino_rec holds
  cudaArray_t* sino_arrays;
  cudaTextureObject_t* sino_tex;
  cudaSurfaceObject_t sino_surf;
  int bp_cull;  // its blocks look for the views they meet first
  // texture sampler (DTV_PLAN_TEX): one 3-D array per batch item
  cudaArray_t* vol_arrays;
  cudaTextureObject_t* vol_tex;      // host copy
  cudaTextureObject_t* vol_tex_dev;  // device copy (kernel argument)
  cudaSurfaceObject_t* vol_surf;     // staging writes into vol_arrays
  // z-pair sampler (DTV_PLAN_TEX_PAIRS): one layered half2 array per batch item
  cudaArray_t* pair_arrays;
  cudaTextureObject_t* pair_tex;
  cudaSurfaceObject_t* pair_surf;
  cudaTextureObject_t* pair_tex_dev;
  int fp_ray_tile;           // DTV_TUNE_FP_RAY_TILE
  int fp_band;               // DTV_TUNE_FP_BAND
  int bp_warp;               // DTV_TUNE_BP_WARP
  // shared-memory staged forward projector (DTV_PLAN_TMA): the z pairs as a
  // linear [batch][nz+3][ny][pair_pitch] u32 array and its two tensor maps
  // (boxes for chunks along x and along y)
  unsigned int* d_pair_lin;
  int pair_pitch;
  int fp_tex_share;          // DTV_TUNE_FP_TEX_SHARE
  alignas(64) unsigned char tmap[2][128];
  int* d_status;             // device error bits
  int bp_zaffine;            // every view's u and h are independent of z
  // adjoint ray table (DTV_PLAN_ADJOINT): per view and pixel, (p0, count) and (dp, 0)
  float4* d_rays;
  // adjoint cell records (DTV_PLAN_ADJOINT): float4, room for the padded grid of d_vol_rec per
  // batch item
  float4* d_cells;
  int adjoint_method;  // DTV_TUNE_ADJOINT
  float adjoint_rows;  // detector rows per voxel (adjoint_impl's choice of scatter)
  double fp_samples;  // per volume, < 0 until computed
  uint64_t geom_key;  // hash of the geometry and its per-view tables
};

constexpr int kNumRayTiles = 8;  // forward-projector ray tiles (DTV_TUNE_FP_RAY_TILE)
// default forward block order (DTV_TUNE_FP_BAND): bands of kDefaultBand tile
// rows for staged volumes above kBandAboveBytes, view by view below
constexpr int kDefaultBand = 4;
// most bytes of a plan's sinogram records (plan.cu)
constexpr int64_t kSinoRecBytes = 4LL << 30;
constexpr double kBandAboveBytes = 32.0 * (1 << 20);
constexpr int kPad = 2;  // zero border of the staged volume

// kernels entry points used across units
int forward_impl(Plan* p, const void* vol, int vol_dtype, int batch, float* out, int epilogue,
                 const float* g, float sigma, double* abs_sum, cudaStream_t st);
// out = base + BP(sino); base NULL: out = BP(sino) (base may be out)
int backward_impl(Plan* p, const float* sino, int batch, const float* base, float* out,
                  cudaStream_t st);
// the correction passes of a texture-filtered plan against an exact one
int forward_refresh_impl(Plan* fast, Plan* exact, const void* vol, int vol_dtype, int batch,
                         const float* g, float sigma, float* w, float* g_eff, double* abs_sum,
                         cudaStream_t st);
int backward_refresh_impl(Plan* fast, Plan* exact, const float* sino, int batch, float* out,
                          float* e_b, cudaStream_t st);
int bp_cull_rule(const Plan* p);
float adjoint_rows(const Plan* p);
int adjoint_impl(Plan* p, const float* sino, int batch, float* out, cudaStream_t st);
int encode_pair_maps(Plan* p);
// several plans' projections in one launch (forward.cu, backward.cu)
constexpr int kManyItems = 24;  // plans per launch; more run in further launches
int forward_many_impl(Plan* const* plans, const void* const* vols, int vol_dtype, float* const* outs,
                      int count, int epilogue, const float* const* gs, float sigma,
                      cudaStream_t st);
int backward_many_impl(Plan* const* plans, const float* const* sinos, float* const* outs, int count,
                       int accumulate, cudaStream_t st);
int build_ray_table(Plan* p, cudaStream_t st);

}  // namespace dtv
