// FBP detector-row filter: cosine weighting followed by the spatial Ram-Lak
// ramp, one fused pass over the sinogram.
//
// Follows model/ConeBeamLayers/Standard/StandardGeometry.py:51-93 (and the
// Beijing variant BeijingGeometry.py:57-84): the residual is multiplied by
//   cos(i, j) = SDD / sqrt(SDD^2 + (i - mid_i)^2 + (j - mid_j)^2)
// over each view's rows i and columns j, then every detector row of length W
// is cross-correlated with the W+1-tap kernel k[t], t = 0..W, centred at
// m = floor(W/2): k[m] = 1/8, k[t] = 0 for even t - m != 0, and
// k[t] = -1/(2 pi^2 (t-m)^2) for odd t - m, with W/2 zero columns of padding on
// each side (torch conv2d, padding (0, W/2)). W must be even (for odd W the
// reference's output row is one column short and its reshape fails).
//
// Design: an output of even index meets only odd columns and the other way
// round (but for the centre tap), so a row is two sequences, x[2m+1] and x[2m],
// each filtered by the symmetric odd taps into the other's outputs. A thread
// owns kOut consecutive outputs of both parities, one in each lane of packed
// FP32, and slides two register windows over the sequences, left and right of
// its outputs: per tap it loads one new pair on each side and the tap, for kOut
// packed adds and FMAs. Taps run from the farthest in, so that the small terms
// add up first. (One output per thread needed 2.5 shared loads per tap, which
// bounded it: 6144 rows of 1680 columns, 1.21 ms; now 0.36 ms, bound by
// the FP32 pipe at 60 % of its rate. 24576 rows of 384: 0.26 -> 0.16 ms.) The weighted sequences sit in shared memory between their
// zero paddings, one pair of skew per kOut, so that lanes kOut apart read
// different banks. The taps are built once per block in FP64 and rounded to
// FP32 as the reference's float32 kernel array holds them. The transpose (for
// autograd) applies the same symmetric correlation first and the cosine weight
// after.
#include <algorithm>
#include <atomic>
#include <type_traits>

#include "common.cuh"

namespace dtv {

constexpr int kFiltThreads = 256;
constexpr int kFiltMaxWidth = 8192;
constexpr int64_t kFiltSmall = 10000;  // threads (filt_small)
// outputs of each parity per thread: 8, or 2 for calls with few rows (filt_small)

// Shared layout: the taps (one set per block), then per row a padded sequence
// of pairs; slot lead + m holds (x[2m+1], x[2m+2]), so that both parities'
// outputs m meet slots lead + m + j and lead + m - 1 - j.
struct FiltShape {
  int n;        // outputs per parity (width / 2)
  int groups;   // threads per row
  int taps;     // odd taps, rounded up to kOut (the extra ones are zero)
  int lead;     // slot of m = 0, a multiple of kOut
  int seq;      // skewed slots per row
  int rows;     // rows per block
  int threads;  // per block
};
template <int kOut>
__host__ __device__ constexpr int filt_skew(int i) { return i + i / kOut; }
// the skewed offset of slot d from one at a multiple of kOut
template <int kOut>
__host__ __device__ constexpr int filt_off(int d) {
  return d >= 0 ? d + d / kOut : d - (-d + kOut - 1) / kOut;
}
// Rows per block: what 256 threads hold, less where the grid would have fewer
// than four blocks per SM.
template <int kOut>
static FiltShape filt_shape(int width, int64_t rows) {
  FiltShape f;
  f.n = width / 2;
  f.groups = (f.n + kOut - 1) / kOut;
  f.taps = ((width / 2 + 1) / 2 + kOut - 1) / kOut * kOut;
  f.lead = f.taps + kOut;
  // the right window reaches taps + kOut beyond the last output's slot
  f.seq = filt_skew<kOut>(f.lead + f.groups * kOut + f.taps + kOut) + 1;
  f.rows = (int)std::max<int64_t>(1, std::min<int64_t>(kFiltThreads / f.groups, rows / (4 * 148)));
  f.rows = std::min(f.rows, 16);
  f.threads = std::min(kFiltThreads, (f.groups * f.rows + 31) / 32 * 32);
  return f;
}
static size_t filt_smem(const FiltShape& f) {
  return sizeof(float) * ((size_t)f.taps + 2 * (size_t)f.seq * f.rows);
}

// At most 72 registers: rows of 1680 columns then have four blocks of 224 threads per
// SM (unbounded the compiler takes 80; 6144 x 1680: 411 us, with the bound 362).
template <int kOut>
__global__ void __maxnreg__(72) fbp_filter_kernel(const float* __restrict__ in,
                                                                  float* __restrict__ out, int64_t rows,
                                                                  int rows_per_view, int width,
                                                                  FiltShape f, float sdd, float mid_i,
                                                                  float mid_j, int adjoint) {
  extern __shared__ float sm[];
  float* taps = sm;
  f32x2_t* seqs = reinterpret_cast<f32x2_t*>(sm + f.taps);  // f.taps is a multiple of kOut
  const int64_t r0 = (int64_t)blockIdx.x * f.rows;
  const int nr = (int)min((int64_t)f.rows, rows - r0);
  auto row_term = [&](int64_t r) {  // sdd^2 + (i - mid_i)^2
    const float fi = (float)(r % rows_per_view) - mid_i;
    return sdd * sdd + fi * fi;
  };
  auto cosine = [&](float row, int c) {
    const float fj = (float)c - mid_j;
    return sdd / sqrtf(row + fj * fj);
  };
  for (int i = threadIdx.x; i < f.seq * nr; i += blockDim.x) seqs[i] = 0;
  const int used = (width / 2 + 1) / 2;
  for (int e = threadIdx.x; e < f.taps; e += blockDim.x) {
    const double d = 2.0 * e + 1.0;
    taps[e] = e < used ? (float)(-0.5 / (3.141592653589793 * 3.141592653589793 * d * d)) : 0.f;
  }
  __syncthreads();
  for (int rr = 0; rr < nr; ++rr) {
    float* s = reinterpret_cast<float*>(seqs + rr * f.seq);
    const float row = row_term(r0 + rr);
    for (int c = threadIdx.x; c < width; c += blockDim.x) {
      float x = __ldg(in + (r0 + rr) * width + c);
      if (!adjoint) x *= cosine(row, c);
      s[2 * filt_skew<kOut>(f.lead + ((c - 1) >> 1)) + ((c - 1) & 1)] = x;
    }
  }
  __syncthreads();
  for (int job = threadIdx.x; job < f.groups * nr; job += blockDim.x) {
    const int g = job % f.groups, rr = job / f.groups;
    const int m0 = g * kOut;
    const f32x2_t* mid = seqs + rr * f.seq + filt_skew<kOut>(f.lead + m0);
    const f32x2_t* right = mid + filt_skew<kOut>(f.taps - kOut);
    const f32x2_t* left = mid - filt_skew<kOut>(f.taps - kOut);
    // windows of the last tap, slot of offset o at o mod kOut: right offsets
    // taps - 1 + e, left offsets -taps + e
    f32x2_t acc[kOut], rw[kOut], lw[kOut];
#pragma unroll
    for (int e = 0; e < kOut; ++e) {
      acc[e] = 0;
      rw[(e + kOut - 1) % kOut] = right[filt_off<kOut>(kOut - 1 + e)];
      lw[(e + 1) % kOut] = left[filt_off<kOut>(e - kOut)];
    }
    // kOut taps from j; those beyond the last of the width (kLast) meet columns whose
    // infinities or NaN do not belong to the sum
    auto group = [&](int j, auto last) {
      constexpr bool kLast = decltype(last)::value;
#pragma unroll
      for (int q = kOut - 1; q >= 0; --q) {
        const f32x2_t t = splat2(taps[j + q]);
        if (!kLast || j + q < used) {
#pragma unroll
          for (int e = 0; e < kOut; ++e)
            acc[e] = fma2(t, add2(rw[(e + q) % kOut], lw[(e - q + kOut) % kOut]), acc[e]);
        }
        rw[(q + kOut - 1) % kOut] = right[filt_off<kOut>(q - 1)];
        lw[(kOut - q) % kOut] = left[filt_off<kOut>(kOut - 1 - q)];
      }
      right -= kOut + 1;
      left += kOut + 1;
    };
    group(f.taps - kOut, std::true_type{});
    for (int j = f.taps - 2 * kOut; j >= 0; j -= kOut) group(j, std::false_type{});
    const int64_t r = r0 + rr;
    const float row = adjoint ? row_term(r) : 0.f;
#pragma unroll
    for (int e = 0; e < kOut; ++e) {
      if (m0 + e >= f.n) break;
      // the centre tap: x[2m] and x[2m+1]
      float y0, y1, c0, c1, unused;
      unpack2(acc[e], y0, y1);
      unpack2(mid[filt_off<kOut>(e - 1)], unused, c0);
      unpack2(mid[filt_off<kOut>(e)], c1, unused);
      y0 = fmaf(0.125f, c0, y0);
      y1 = fmaf(0.125f, c1, y1);
      const int u = 2 * (m0 + e);
      if (adjoint) {
        y0 *= cosine(row, u);
        y1 *= cosine(row, u + 1);
      }
      out[r * width + u] = y0;
      out[r * width + u + 1] = y1;
    }
  }
}

// Whether the threads of eight outputs per parity leave most of the GPU idle: each sums
// over half the row one tap after the other, so more threads of two finish earlier, as
// long as they fit the GPU about once and a row one block. 40 rows of 250: 6.2 us with
// eight, 4.1 with two; 600 of 250 7.2, 5.1; 40 of 1000 12.9, 8.7; 600 of 1000 23.7, 30.1;
// 40 of 1680 16.8, 20.1.
static bool filt_small(int width, int64_t rows) {
  return width <= 1024 && (width / 2 + 7) / 8 * rows < kFiltSmall;
}

template <int kOut>
static int filt_launch(const float* in, float* out, int64_t rows, int32_t rows_per_view, int32_t width,
                       float sdd, float mid_i, float mid_j, int32_t adjoint, cudaStream_t st) {
  const FiltShape f = filt_shape<kOut>(width, rows);
  const size_t smem = filt_smem(f);
  if (smem > 48 * 1024) {
    // per-device function attribute, raised once to the widest row's need
    static std::atomic<unsigned long long> raised{0};
    int dev = 0;
    DTV_CUDA_TRY(cudaGetDevice(&dev));
    const unsigned long long bit = 1ull << (dev & 63);
    if (!(raised.load() & bit)) {
      DTV_CUDA_TRY(cudaFuncSetAttribute(fbp_filter_kernel<kOut>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                        (int)filt_smem(filt_shape<kOut>(kFiltMaxWidth, 1))));
      raised |= bit;
    }
  }
  fbp_filter_kernel<kOut><<<(unsigned)((rows + f.rows - 1) / f.rows), f.threads, smem, st>>>(
      in, out, rows, rows_per_view, width, f, sdd, mid_i, mid_j, adjoint ? 1 : 0);
  note_launch();
  DTV_LAUNCH_CHECK();
  return DTV_OK;
}

}  // namespace dtv

using namespace dtv;

extern "C" int dtv_fbp_filter(const float* in, float* out, int64_t rows, int32_t rows_per_view,
                              int32_t width, float sdd, float mid_i, float mid_j, int32_t adjoint,
                              void* stream) {
  DTV_CHECK(in && out, "NULL argument");
  DTV_CHECK(in != out, "the filter cannot run in place");
  DTV_CHECK(rows > 0 && rows_per_view > 0 && rows % rows_per_view == 0,
            "rows must be a positive multiple of rows_per_view");
  DTV_CHECK(rows <= 2147483647LL, "too many rows");
  DTV_CHECK(width >= 2 && width % 2 == 0 && width <= kFiltMaxWidth,
            "row width must be even and in [2, %d]", kFiltMaxWidth);
  DTV_CHECK(sdd > 0.f, "sdd must be positive");
  if (filt_small(width, rows))
    return filt_launch<2>(in, out, rows, rows_per_view, width, sdd, mid_i, mid_j, adjoint, as_stream(stream));
  return filt_launch<8>(in, out, rows, rows_per_view, width, sdd, mid_i, mid_j, adjoint, as_stream(stream));
}
