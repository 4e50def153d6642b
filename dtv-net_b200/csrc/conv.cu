// The unrolled networks' convolution block in BF16, forward and backward:
// Conv3d(1, F) - ReLU - Conv3d(F, F) - ReLU - Conv3d(F, 1), 3x3x3 kernels, zero
// padding (the shape of model/PDHG/RegularizationLayers/CNN.py:4-18), F = 16 or 32.
// Activations are channels-last, [batch, z, y, x, F]. Each convolution sums in
// FP32 and is rounded to BF16, then the BF16 bias is added and rounded again: the
// roundings that autocast makes around a library convolution.
// Measured at 2 x 128^3, F = 32: 0.42 ms (0.06 + 0.22 + 0.12 and the weights), where
// three library convolutions with their layout conversions, bias additions and ReLUs
// took 4.1 ms; F = 16: 0.28 ms. Backward, all gradients: 1.06 ms, the library's 8.4.
// Gradients are rounded to BF16 where autocast's are: the data gradients after each
// convolution, the weight and bias gradients once summed. Sums are FP32 in an order
// fixed by the sizes and the number of SMs.
#include <cuda.h>
#include <cuda_bf16.h>

#include "common.cuh"

namespace dtv {
namespace {

typedef __nv_bfloat16 bf16;

struct ConvDims {
  int X, Y, Z, B;
};
struct ConvW {  // a weight tensor [out, in, z, y, x] in elements
  const bf16* w;
  long long s[5];
};

__device__ __forceinline__ uint32_t conv_smem(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ float round_bf16(float v) { return __bfloat162float(__float2bfloat16_rn(v)); }
// relu(bf16(bf16(sum) + bias)) of two channels; NaN stays NaN
__device__ __forceinline__ unsigned conv_act(float lo, float hi, __nv_bfloat162 bias) {
  const __nv_bfloat162 v =
      __hmax2_nan(__hadd2(__floats2bfloat162_rn(lo, hi), bias), __nv_bfloat162(0.f, 0.f));
  return *reinterpret_cast<const unsigned*>(&v);
}
// bf16(sum) of two channels where the activations of the forward pass are positive (or NaN)
__device__ __forceinline__ unsigned conv_masked(float lo, float hi, unsigned act) {
  const __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162*>(&act);
  return *reinterpret_cast<const unsigned*>(&v) & ~__hle2_mask(h, __nv_bfloat162(0.f, 0.f));
}
// D[16 x 8] += A[16 x 16] B[16 x 8], BF16 in, FP32 out
__device__ __forceinline__ void warp_mma(float (&d)[4], unsigned a0, unsigned a1, unsigned a2, unsigned a3,
                                         unsigned b0, unsigned b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, "
      "{%8, %9}, {%0, %1, %2, %3};"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// ---- F = 16, 32 middle convolution on the tensor cores -----------------------------------
// A block marches down z over a column of 8 x 16 voxels (the 128 rows of a tile).
// Each input plane is loaded once by TMA with its y halo, in three copies shifted
// by -1, 0, 1 in x; a shift in y is then an offset of whole 8-row swizzle atoms, so
// the nine (x, y) taps read their operands from the copies in place. The three z
// taps of an (x, y) tap stand side by side in the B operand: one instruction of
// 3F columns adds an input plane's share to the three output planes around it,
// which lie side by side in a ring of kRing accumulators in tensor memory. Reading
// A once for three planes is what makes the step arithmetic-bound: with F columns
// an instruction waits on its 4 KB of A. 2 x 128^3, F = 32: 0.223 ms, 1.04 PFLOP/s
// (F = 16: 0.120); the library's kernel 1.03 ms. On the way: 0.63 ms while one thread
// built each descriptor, 0.30 with them precomputed, 0.28 with the whole warp in the
// loop and one lane elected per instruction. Not faster: one unswizzled copy of a
// plane addressed at odd offsets (cp.async, a third of the loads; 0.30), two
// accumulators per plane (0.32).
// Two columns at a time, each with a warp that loads, one that issues and four that
// write finished planes: the issue of a plane's instructions and its waits take longer
// than the tensor core takes for them.
constexpr int kCX = 8, kCY = 16;   // column: rows of 8 voxels, one swizzle atom each
constexpr int kPipes = 2;          // columns a block works on
constexpr int kRing = 8;           // accumulators of a column
constexpr int kStages = 3;         // input planes in flight of a column
constexpr int kMidThreads = kPipes * (64 + 128);
constexpr unsigned kConvWaitLimit = 1u << 20;  // polls of one wait

template <int F>
struct Mid {
  static constexpr int kRow = F * 2;                        // bytes of a voxel
  static constexpr int kCopy = kCX * (kCY + 2) * kRow;      // a shifted copy of a plane
  static constexpr int kStage = 3 * kCopy;
  static constexpr int kTap = 3 * F * kRow;                 // B operand of an (x, y) tap
  static constexpr int kWeights = 9 * kTap;
  static constexpr int kFirst = (kWeights + 1023) / 1024 * 1024;  // of the stages
  static constexpr int kSmem = 1024 + kFirst + kPipes * kStages * kStage;
  static constexpr int kCols = kPipes * F * kRing;          // tensor-memory columns
  static constexpr unsigned long long kLayout = F == 32 ? 4ull : 6ull;  // 64- / 32-byte swizzle
};

struct MidWork {
  int tx, ty, nzc, zc;  // columns along x, y; z chunks and their length
  long long items;
};

__device__ __forceinline__ bool conv_wait(uint32_t bar, uint32_t parity) {
  for (unsigned i = 0; i < kConvWaitLimit; ++i) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}
__device__ __forceinline__ void conv_arrive(uint32_t bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void conv_expect(uint32_t bar, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
               : "memory");
}
// all matrix instructions issued so far arrive on bar when they are done
__device__ __forceinline__ void conv_commit(uint32_t bar, uint32_t elected) {
  asm volatile(
      "{\n .reg .pred e;\n setp.ne.u32 e, %1, 0;\n"
      " @e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(bar),
      "r"(elected)
      : "memory");
}
// one lane of the warp, the same at each call
__device__ __forceinline__ uint32_t conv_elect() {
  uint32_t e;
  asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xffffffff;\n selp.u32 %0, 1, 0, p;\n}\n" : "=r"(e));
  return e;
}
// the whole warp waits
__device__ __forceinline__ bool conv_wait_all(uint32_t bar, uint32_t parity) {
  return __all_sync(0xffffffffu, conv_wait(bar, parity));
}
// K-major operand descriptor, 8-row atoms one after another
template <int F>
__device__ __forceinline__ unsigned long long conv_desc(uint32_t addr) {
  return (unsigned long long)((addr >> 4) & 0x3fffu) | (1ull << 16) |
         ((unsigned long long)(8 * Mid<F>::kRow / 16) << 32) | (1ull << 46) |
         (Mid<F>::kLayout << 61);
}
// D[128 x n] (+)= A[128 x 16] B[n x 16]^T, BF16 in, FP32 out
__device__ __forceinline__ uint32_t conv_idesc(int n) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | (8u << 24);
}
__device__ __forceinline__ void conv_mma(uint32_t d, unsigned long long a, unsigned long long b,
                                         uint32_t idesc, bool add, uint32_t elected) {
  asm volatile(
      "{\n .reg .pred p, e;\n setp.ne.u32 p, %4, 0;\n setp.ne.u32 e, %5, 0;\n"
      " @e tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)add), "r"(elected)
      : "memory");
}

// descriptor offsets of step k = (tap, 16 input channels) from the first step's
template <int F>
__device__ constexpr unsigned mid_a(int k) {
  const int t = k / (F / 16), c = k % (F / 16);
  return (t % 3 * Mid<F>::kCopy + t / 3 * 8 * Mid<F>::kRow + 32 * c) / 16;
}
template <int F>
__device__ constexpr unsigned mid_b(int k) {
  return (k / (F / 16) * Mid<F>::kTap + 32 * (k % (F / 16))) / 16;
}

// 16 columns of this warp's lanes
__device__ __forceinline__ void tmem_load16(uint32_t* r, uint32_t addr) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, "
      "%13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]),
        "=r"(r[15])
      : "r"(addr));
}

struct MidItem {
  int x0, y0, z0, z1, b;
};
__device__ __forceinline__ MidItem mid_item(const ConvDims& d, const MidWork& w, long long i) {
  MidItem r;
  r.x0 = (int)(i % w.tx) * kCX;
  i /= w.tx;
  r.y0 = (int)(i % w.ty) * kCY;
  i /= w.ty;
  r.z0 = (int)(i % w.nzc) * w.zc;
  r.b = (int)(i / w.nzc);
  r.z1 = min(d.Z, r.z0 + w.zc);
  return r;
}

// kMask: the data gradient, with flipped weights: no bias, zero where `act` (the
// forward pass's output of the ReLU below) is zero. Otherwise `act` is unused.
template <int F, bool kMask>
__global__ void __launch_bounds__(kMidThreads, 1)
    conv_mid_kernel(const __grid_constant__ CUtensorMap map, const unsigned char* __restrict__ wimg,
                    const bf16* __restrict__ bias, const bf16* __restrict__ act, bf16* __restrict__ out,
                    ConvDims d, MidWork wk, int* status) {
  typedef Mid<F> M;
  extern __shared__ unsigned char conv_dyn[];
  __shared__ __align__(8) unsigned long long bars[kPipes * (2 * kStages + 2 * kRing + 1) + 1];
  __shared__ uint32_t tmem_slot;
  const uint32_t base = (conv_smem(conv_dyn) + 1023u) & ~1023u;
  // (the shuffle tells the compiler that a warp's number is the same in all its lanes)
  const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
  const int pipe = warp < 2 * kPipes ? warp >> 1 : (warp - 2 * kPipes) >> 2;
  const uint32_t wsm = base, stages = base + M::kFirst + pipe * kStages * M::kStage;
  const uint32_t wbar = conv_smem(bars), bar0 = wbar + 8 + pipe * 8 * (2 * kStages + 2 * kRing + 1);
  const uint32_t full = bar0, empty = full + 8 * kStages, acc_full = empty + 8 * kStages,
                 acc_empty = acc_full + 8 * kRing, drain = acc_empty + 8 * kRing;
  if (threadIdx.x == 0) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(wbar) : "memory");
  if (warp < 2 * kPipes && (threadIdx.x & 63) == 0) {
    for (int i = 0; i < kStages; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full + 8 * i) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(empty + 8 * i) : "memory");
    }
    for (int i = 0; i < kRing; ++i) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(acc_full + 8 * i) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 4;" ::"r"(acc_empty + 8 * i) : "memory");
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(drain) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     conv_smem(&tmem_slot)),
                 "r"(M::kCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot + pipe * F * kRing;
  const long long first = (long long)blockIdx.x * kPipes + pipe, step = (long long)gridDim.x * kPipes;
  bool ok = true;

  if (warp < 2 * kPipes && !(warp & 1)) {  // loads
    if (lane == 0) {
      if (pipe == 0) {
        conv_expect(wbar, M::kWeights);
        asm volatile(
            "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(wsm),
            "l"(wimg), "r"(M::kWeights), "r"(wbar)
            : "memory");
      }
      long long n = 0;  // planes loaded
      for (long long i = first; ok && i < wk.items; i += step) {
        const MidItem it = mid_item(d, wk, i);
        for (int zi = it.z0 - 1; zi <= it.z1; ++zi, ++n) {
          const int s = (int)(n % kStages);
          if (n >= kStages && !(ok = conv_wait(empty + 8 * s, (uint32_t)((n / kStages - 1) & 1)))) break;
          conv_expect(full + 8 * s, M::kStage);
#pragma unroll
          for (int c = 0; c < 3; ++c)
            asm volatile(
                "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
                " [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(stages + s * M::kStage + c * M::kCopy),
                "l"(&map), "r"(0), "r"(it.x0 + c - 1), "r"(it.y0 - 1), "r"(zi), "r"(it.b),
                "r"(full + 8 * s)
                : "memory");
        }
      }
      // the last copies land before the block can end
      for (long long k = n > kStages ? n - kStages : 0; k < n; ++k)
        ok &= conv_wait(full + 8 * (int)(k % kStages), (uint32_t)((k / kStages) & 1));
    }
  } else if (warp < 2 * kPipes) {  // matrix instructions
    const uint32_t e1 = conv_elect();
    ok = conv_wait_all(wbar, 0);
    long long n = 0, g = 0;  // input planes, output planes so far
    for (long long i = first; ok && i < wk.items; i += step) {
      const MidItem it = mid_item(d, wk, i);
      for (int zi = it.z0 - 1; zi <= it.z1; ++zi, ++n) {
        const int s = (int)(n % kStages);
        const int lo = max(it.z0, zi - 1), hi = min(it.z1 - 1, zi + 1);
        if (hi == zi + 1) {  // a plane begins: its accumulator is drained
          const long long u = g + (hi - it.z0);
          if (u >= kRing &&
              !(ok = conv_wait_all(acc_empty + 8 * (int)(u % kRing), (uint32_t)((u / kRing - 1) & 1))))
            break;
        }
        if (!(ok = conv_wait_all(full + 8 * s, (uint32_t)((n / kStages) & 1)))) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const unsigned long long ad = conv_desc<F>(stages + s * M::kStage);
        const unsigned long long bd = conv_desc<F>(wsm + (lo - zi + 1) * F * M::kRow);
        constexpr unsigned kB = F * M::kRow / 16;  // one plane's rows of B
        const int slot = (int)((g + (lo - it.z0)) % kRing), n1 = min(hi - lo + 1, kRing - slot),
                  n2 = hi - lo + 1 - n1;
        const uint32_t d1 = tmem + slot * F;
        // the first step one plane at a time: the plane that begins is overwritten
        for (int j = 0; j < n1 + n2; ++j)
          conv_mma(j < n1 ? d1 + j * F : tmem + (j - n1) * F, ad, bd + j * kB, conv_idesc(F),
                   lo + j != zi + 1, e1);
        const uint32_t i1 = conv_idesc(n1 * F), i2 = conv_idesc(n2 * F);
        if (n2 == 0) {
#pragma unroll
          for (int k = 1; k < 9 * (F / 16); ++k)
            conv_mma(d1, ad + mid_a<F>(k), bd + mid_b<F>(k), i1, true, e1);
        } else {  // the planes wrap round the ring
#pragma unroll
          for (int k = 1; k < 9 * (F / 16); ++k) {
            conv_mma(d1, ad + mid_a<F>(k), bd + mid_b<F>(k), i1, true, e1);
            conv_mma(tmem, ad + mid_a<F>(k), bd + mid_b<F>(k) + n1 * kB, i2, true, e1);
          }
        }
        conv_commit(empty + 8 * s, e1);
        if (zi - 1 >= it.z0) conv_commit(acc_full + 8 * (int)((g + (zi - 1 - it.z0)) % kRing), e1);
      }
      g += it.z1 - it.z0;
    }
    conv_commit(drain, e1);  // nothing in flight when the tensor memory is given back
    ok &= conv_wait_all(drain, 0);
  } else {  // finished planes
    const int q = warp & 3;  // the quarter of the lanes this warp may read
    __nv_bfloat162 bs[F / 2];
#pragma unroll
    for (int c = 0; c < F / 2; ++c)
      if (!kMask) bs[c] = __nv_bfloat162(bias[2 * c], bias[2 * c + 1]);
    long long g = 0;
    for (long long i = first; ok && i < wk.items; i += step) {
      const MidItem it = mid_item(d, wk, i);
      const int x = it.x0 + (lane & 7), y = it.y0 + q * 4 + (lane >> 3);
      const bool in = x < d.X && y < d.Y;
      for (int z = it.z0; z < it.z1; ++z, ++g) {
        const int slot = (int)(g % kRing);
        const long long vox = ((((long long)it.b * d.Z + z) * d.Y + y) * d.X + x) * F;
        uint4 m[F / 8];
        if (kMask) {
#pragma unroll
          for (int c = 0; c < F / 8; ++c)
            m[c] = in ? __ldg(reinterpret_cast<const uint4*>(act + vox) + c) : make_uint4(0u, 0u, 0u, 0u);
        }
        ok = __all_sync(0xffffffffu, conv_wait(acc_full + 8 * slot, (uint32_t)((g / kRing) & 1)));
        if (!ok) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        uint32_t r[F];
#pragma unroll
        for (int c = 0; c < F; c += 16)
          tmem_load16(r + c, tmem + ((uint32_t)(q * 32) << 16) + slot * F + c);
        asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncwarp();
        if (lane == 0) conv_arrive(acc_empty + 8 * slot);
        if (in) {
          uint4* o = reinterpret_cast<uint4*>(out + vox);
#pragma unroll
          for (int c = 0; c < F; c += 8) {
            unsigned p[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
              p[j] = kMask ? conv_masked(__uint_as_float(r[c + 2 * j]), __uint_as_float(r[c + 2 * j + 1]),
                                         (&m[c / 8].x)[j])
                           : conv_act(__uint_as_float(r[c + 2 * j]), __uint_as_float(r[c + 2 * j + 1]),
                                      bs[c / 2 + j]);
            o[c / 8] = make_uint4(p[0], p[1], p[2], p[3]);
          }
        }
      }
    }
  }
  __syncwarp();
  if (!ok) *status = 1;
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_slot), "r"(M::kCols));
}

// The weights as the three kernels read them: the B operands of the middle one's nine
// (x, y) taps in their swizzled shared-memory layout (rows (output plane zi - 1, zi,
// zi + 1; output channel), input channels along K), and the fragments of the first and
// the last one's B operands, lane by lane.
template <int F>
struct ConvWs {
  static constexpr int kIn = Mid<F>::kWeights;     // bytes before the first one's fragments
  static constexpr int kInWords = F / 2;           // per lane
  static constexpr int kOut = kIn + 32 * kInWords * 4;
  static constexpr int kOutWords = F / 2;
  // 16 bytes: a wait ran out; the last, the middle one's weight gradient is not finite
  static constexpr int kStatus = kOut + 32 * kOutWords * 4;
};

__device__ __forceinline__ bf16 conv_weight(const ConvW& w, int co, int ci, int kz, int ky, int kx) {
  return w.w[co * w.s[0] + ci * w.s[1] + kz * w.s[2] + ky * w.s[3] + kx * w.s[4]];
}

template <int F>
__global__ void conv_weights_kernel(ConvW w1, ConvW w2, ConvW w3, unsigned char* ws) {
  typedef ConvWs<F> W;
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i == 0) *reinterpret_cast<int4*>(ws + W::kStatus) = make_int4(0, 0, 0, 0);
  if (i < 27 * F * F) {
    const int ci = i % F, n = (i / F) % (3 * F), t = i / (3 * F * F);
    const int sw = F == 32 ? (n >> 1) & 3 : (n >> 2) & 1;
    reinterpret_cast<bf16*>(ws)[(t * Mid<F>::kTap + n * Mid<F>::kRow + (((ci >> 3) ^ sw) << 4)) / 2 + (ci & 7)] =
        conv_weight(w2, n % F, ci, 2 - n / F, t / 3, t % 3);
    return;
  }
  i -= 27 * F * F;
  // element e of word j of a lane: column n = lane / 4, k pair lane % 4
  if (i < 32 * W::kInWords * 2) {
    const int e = i & 1, j = (i >> 1) % W::kInWords, lane = (i >> 1) / W::kInWords;
    const int half = j & 1, ks = (j >> 1) & 1, t = j >> 2, n = lane >> 2, q = lane & 3;
    const int tap = ks * 16 + 2 * q + 8 * half + e, c = F / 4 * (n >> 1) + 2 * t + (n & 1);
    reinterpret_cast<bf16*>(ws + W::kIn)[i] =
        tap < 27 ? conv_weight(w1, c, 0, tap / 9, tap / 3 % 3, tap % 3) : __float2bfloat16_rn(0.f);
    return;
  }
  i -= 32 * W::kInWords * 2;
  if (i < 32 * W::kOutWords * 2) {
    const int e = i & 1, j = (i >> 1) % W::kOutWords, lane = (i >> 1) / W::kOutWords;
    const int half = j & 1, ks = (j >> 1) % (F / 16), t = (j >> 1) / (F / 16), n = lane >> 2, q = lane & 3;
    const int tap = 8 * t + n, c = F / 4 * q + 4 * ks + 2 * half + e;
    reinterpret_cast<bf16*>(ws + W::kOut)[i] =
        tap < 27 ? conv_weight(w3, 0, c, tap / 9, tap / 3 % 3, tap % 3) : __float2bfloat16_rn(0.f);
  }
}
template <int F>
constexpr int conv_weight_items() { return 27 * F * F + 32 * F * 2; }

// F / 2 consecutive words of a lane
template <int F>
__device__ __forceinline__ void load_frags(unsigned (&r)[F / 2], const unsigned char* p, int lane) {
  const uint4* q = reinterpret_cast<const uint4*>(p) + lane * (F / 8);
#pragma unroll
  for (int i = 0; i < F / 8; ++i) {
    const uint4 v = q[i];
    r[4 * i] = v.x; r[4 * i + 1] = v.y; r[4 * i + 2] = v.z; r[4 * i + 3] = v.w;
  }
}
// F / 4 channels of a voxel: 8 or 16 bytes
template <int F>
struct Quarter {
  unsigned w[F / 8];
};
template <int F>
__device__ __forceinline__ Quarter<F> load_quarter(const bf16* p) {
  Quarter<F> r;
  if (F == 32) {
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(p));
    r.w[0] = v.x; r.w[1] = v.y; r.w[F / 16] = v.z; r.w[F / 8 - 1] = v.w;
  } else {
    const uint2 v = __ldg(reinterpret_cast<const uint2*>(p));
    r.w[0] = v.x; r.w[1] = v.y;
  }
  return r;
}
template <int F>
__device__ __forceinline__ void store_quarter(bf16* p, const Quarter<F>& r) {
  if (F == 32)
    *reinterpret_cast<uint4*>(p) = make_uint4(r.w[0], r.w[1], r.w[F / 16], r.w[F / 8 - 1]);
  else
    *reinterpret_cast<uint2*>(p) = make_uint2(r.w[0], r.w[1]);
}

// ---- first convolution: one channel to F ----------------------------------------------
// 27 taps padded to K = 32 and F columns: eight small matrix instructions per 16
// voxels of a row leave the kernel to its writes of 2 F bytes per voxel (27 F FP32
// multiply-adds per voxel took 0.26 ms at 2 x 128^3, this 0.060). The columns are permuted so
// that a lane ends with F / 4 adjacent channels. A warp takes a row of 16 voxels and
// walks along z.
constexpr int kInX = 16, kInY = 8, kInZ = 16;

// kMask: the data gradient of the last convolution, as in conv_mid_kernel; `sums`
// takes the block's sum of each channel.
template <int F, bool kMask>
__global__ void __launch_bounds__(256) conv_in_kernel(const bf16* __restrict__ x,
                                                      const unsigned char* __restrict__ wf,
                                                      const bf16* __restrict__ bias,
                                                      const bf16* __restrict__ act,
                                                      bf16* __restrict__ out, ConvDims d,
                                                      float* __restrict__ sums) {
  constexpr int kPX = kInX + 2, kNT = F / 8;
  __shared__ float part[kMask ? 8 * F : 1];
  __shared__ unsigned short in[(kInZ + 2) * (kInY + 2) * kPX];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = lane >> 2, q = lane & 3;
  unsigned w[F / 2];
  load_frags<F>(w, wf, lane);
  __nv_bfloat162 bs[kNT];
#pragma unroll
  for (int t = 0; t < kNT; ++t) {
    const int c = F / 4 * q + 2 * t;
    if (!kMask) bs[t] = __nv_bfloat162(bias[c], bias[c + 1]);
  }
  const int tx = (d.X + kInX - 1) / kInX, ty = (d.Y + kInY - 1) / kInY, tz = (d.Z + kInZ - 1) / kInZ;
  long long id = blockIdx.x;
  const int x0 = (int)(id % tx) * kInX;
  id /= tx;
  const int y0 = (int)(id % ty) * kInY;
  id /= ty;
  const int z0 = (int)(id % tz) * kInZ, b = (int)(id / tz);
  const unsigned short* xs = reinterpret_cast<const unsigned short*>(x) + (long long)b * d.Z * d.Y * d.X;
  for (int i = threadIdx.x; i < (kInZ + 2) * (kInY + 2) * kPX; i += 256) {
    const int ix = i % kPX, iy = i / kPX % (kInY + 2), iz = i / (kPX * (kInY + 2));
    const int gx = x0 + ix - 1, gy = y0 + iy - 1, gz = z0 + iz - 1;
    in[i] = gx >= 0 && gx < d.X && gy >= 0 && gy < d.Y && gz >= 0 && gz < d.Z
                ? xs[((long long)gz * d.Y + gy) * d.X + gx]
                : (unsigned short)0;
  }
  // this lane's taps, 2 per word; the last word's beyond 26 are padding, zero on both
  // sides (an infinite voxel times a zero weight would be NaN)
  const unsigned keep = q == 0 ? 0xffffffffu : q == 1 ? 0xffffu : 0u;
  int off[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    const int tap = min((j >> 2) * 16 + 2 * q + (j >> 1 & 1) * 8 + (j & 1), 26);
    off[j] = (tap / 9 * (kInY + 2) + tap / 3 % 3) * kPX + tap % 3 + warp * kPX + row;
  }
  __syncthreads();
  const int gy = y0 + warp;
  const bool in0 = x0 + row < d.X, in1 = x0 + row + 8 < d.X;
  long long vox = ((((long long)b * d.Z + z0) * d.Y + gy) * d.X + x0 + row) * F + F / 4 * q;
  const int nz = gy < d.Y ? min(kInZ, d.Z - z0) : 0;
  float2 sum[kNT];
#pragma unroll
  for (int t = 0; t < kNT; ++t) sum[t] = make_float2(0.f, 0.f);
  for (int k = 0; k < nz; ++k, vox += (long long)d.Y * d.X * F) {
    Quarter<F> m0{}, m1{};
    if (kMask) {
      if (in0) m0 = load_quarter<F>(act + vox);
      if (in1) m1 = load_quarter<F>(act + vox + 8 * F);
    }
    const unsigned short* s = in + k * (kInY + 2) * kPX;
    unsigned a[2][4];
#pragma unroll
    for (int ks = 0; ks < 2; ++ks)
#pragma unroll
      for (int j = 0; j < 4; ++j) {  // (row, row + 8) x (low, high half of k)
        const unsigned short* r = s + (j & 1) * 8;
        const int u = ks * 4 + (j >> 1) * 2;
        a[ks][j] = (unsigned)r[off[u]] | (unsigned)r[off[u + 1]] << 16;
        if (u == 6) a[ks][j] &= keep;
      }
    Quarter<F> r0, r1;
#pragma unroll
    for (int t = 0; t < kNT; ++t) {
      float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
      for (int ks = 0; ks < 2; ++ks)
        warp_mma(acc, a[ks][0], a[ks][1], a[ks][2], a[ks][3], w[(t * 2 + ks) * 2], w[(t * 2 + ks) * 2 + 1]);
      r0.w[t] = kMask ? conv_masked(acc[0], acc[1], m0.w[t]) : conv_act(acc[0], acc[1], bs[t]);
      r1.w[t] = kMask ? conv_masked(acc[2], acc[3], m1.w[t]) : conv_act(acc[2], acc[3], bs[t]);
      if (kMask) {
        sum[t].x += __uint_as_float(r0.w[t] << 16) + __uint_as_float(r1.w[t] << 16);
        sum[t].y += __uint_as_float(r0.w[t] & 0xffff0000u) + __uint_as_float(r1.w[t] & 0xffff0000u);
      }
    }
    if (in0) store_quarter<F>(out + vox, r0);
    if (in1) store_quarter<F>(out + vox + 8 * F, r1);
  }
  if (kMask) {
#pragma unroll
    for (int t = 0; t < kNT; ++t)
#pragma unroll
      for (int o = 4; o < 32; o *= 2) {
        sum[t].x += __shfl_xor_sync(0xffffffffu, sum[t].x, o);
        sum[t].y += __shfl_xor_sync(0xffffffffu, sum[t].y, o);
      }
    if (row == 0)
#pragma unroll
      for (int t = 0; t < kNT; ++t) {
        part[warp * F + F / 4 * q + 2 * t] = sum[t].x;
        part[warp * F + F / 4 * q + 2 * t + 1] = sum[t].y;
      }
    __syncthreads();
    if (threadIdx.x < F) {
      float v = 0.f;
#pragma unroll
      for (int i = 0; i < 8; ++i) v += part[i * F + threadIdx.x];
      sums[(long long)blockIdx.x * F + threadIdx.x] = v;
    }
  }
}

// ---- last convolution: F channels to one ----------------------------------------------
// Read once: the 27 products of a voxel's F channels with the taps' weights are a
// matrix product of K = F and 32 columns; each output then adds 27 of them from
// shared memory. A block walks down z over 16 x 16 outputs, with the products of one
// plane's 18 x 18 voxels in shared memory (two planes, written and read in turn), its
// next plane's voxels on their way in registers, and three outputs in progress.
// 2 x 128^3, F = 32: 0.124 ms (0.38 with FP32 multiply-adds from a BF16 tile).
constexpr int kOutT = 16, kOutM = (kOutT + 2) * (kOutT + 2);  // kOutM = 4 mod 16: no bank conflicts
constexpr int kOutTiles = (kOutM + 15) / 16, kOutPerWarp = (kOutTiles + 7) / 8;
constexpr int kOutSmem = 2 * 27 * kOutM * 4;

template <int F>
__global__ void __launch_bounds__(256) conv_out_kernel(const bf16* __restrict__ h,
                                                       const unsigned char* __restrict__ wf,
                                                       const bf16* __restrict__ bias,
                                                       bf16* __restrict__ out, ConvDims d, int zc,
                                                       const int* status) {
  constexpr int kKS = F / 16;
  extern __shared__ __align__(16) unsigned char conv_dyn[];
  float* prod = reinterpret_cast<float*>(conv_dyn);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, row = lane >> 2, q = lane & 3;
  unsigned w[F / 2];
  load_frags<F>(w, wf, lane);
  const int tx = (d.X + kOutT - 1) / kOutT, ty = (d.Y + kOutT - 1) / kOutT, tz = (d.Z + zc - 1) / zc;
  long long id = blockIdx.x;
  const int x0 = (int)(id % tx) * kOutT;
  id /= tx;
  const int y0 = (int)(id % ty) * kOutT;
  id /= ty;
  const int z0 = (int)(id % tz) * zc, z1 = min(d.Z, z0 + zc), b = (int)(id / tz);
  const long long plane = (long long)d.X * d.Y;
  const bf16* hb = h + (long long)b * d.Z * plane * F + F / 4 * q;
  // this lane's voxels of a plane, -1 outside the volume
  int off[kOutPerWarp][2];
#pragma unroll
  for (int i = 0; i < kOutPerWarp; ++i)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int m = (warp + 8 * i) * 16 + row + 8 * j;
      const int gx = x0 + m % (kOutT + 2) - 1, gy = y0 + m / (kOutT + 2) - 1;
      off[i][j] = m < kOutM && gx >= 0 && gx < d.X && gy >= 0 && gy < d.Y ? gy * d.X + gx : -1;
    }
  Quarter<F> a[kOutPerWarp][2];
  const auto fetch = [&](int z) {
#pragma unroll
    for (int i = 0; i < kOutPerWarp; ++i)
#pragma unroll
      for (int j = 0; j < 2; ++j) {
        if (off[i][j] >= 0 && z >= 0 && z < d.Z) {
          a[i][j] = load_quarter<F>(hb + (z * plane + off[i][j]) * F);
        } else {
#pragma unroll
          for (int c = 0; c < F / 8; ++c) a[i][j].w[c] = 0u;
        }
      }
  };
  fetch(z0 - 1);
  const int lx = threadIdx.x % kOutT, ly = threadIdx.x / kOutT;
  const int gx = x0 + lx, gy = y0 + ly;
  const bool in = gx < d.X && gy < d.Y, bad = *status != 0;  // a wait of the middle one ran out
  const float bs = bias ? __bfloat162float(bias[0]) : 0.f;  // none for the data gradient
  bf16* o = out + (long long)b * d.Z * plane + (long long)gy * d.X + gx;
  float s0 = 0.f, s1 = 0.f;  // outputs z - 1 and z
  for (int z = z0 - 1; z <= z1; ++z) {
    float* p = prod + ((z - z0 + 1) & 1) * 27 * kOutM;
#pragma unroll
    for (int i = 0; i < kOutPerWarp; ++i) {
      const int m = (warp + 8 * i) * 16 + row;
      if (warp + 8 * i < kOutTiles) {
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          float acc[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
          for (int ks = 0; ks < kKS; ++ks)
            warp_mma(acc, a[i][0].w[2 * ks], a[i][1].w[2 * ks], a[i][0].w[2 * ks + 1],
                     a[i][1].w[2 * ks + 1], w[(t * kKS + ks) * 2], w[(t * kKS + ks) * 2 + 1]);
          const int tap = 8 * t + 2 * q;
          if (tap < 27) {
            float* r = p + tap * kOutM + m;
            if (m < kOutM) r[0] = acc[0];
            if (m + 8 < kOutM) r[8] = acc[2];
            if (tap + 1 < 27) {
              if (m < kOutM) r[kOutM] = acc[1];
              if (m + 8 < kOutM) r[kOutM + 8] = acc[3];
            }
          }
        }
      }
    }
    if (z < z1) fetch(z + 1);
    __syncthreads();
    float t[3] = {0.f, 0.f, 0.f};
    const float* r = p + ly * (kOutT + 2) + lx;
#pragma unroll
    for (int kz = 0; kz < 3; ++kz)
#pragma unroll
      for (int k = 0; k < 9; ++k)
        t[kz] += r[(kz * 9 + k) * kOutM + k / 3 * (kOutT + 2) + k % 3];
    const float done = s0 + t[2];  // output z - 1
    s0 = s1 + t[1];
    s1 = t[0];
    if (in && z - 1 >= z0)
      o[(z - 1) * plane] = __float2bfloat16_rn(bad ? __int_as_float(0x7fffffff) : round_bf16(done) + bs);
  }
}

// ---- weight gradients -------------------------------------------------------------------
// Of the first or the last convolution: sum over voxels of s[v + tap - 1] T[v][c], a
// one-channel and an F-channel tensor; tap 27 stands for the sum of T alone. 32 rows
// of taps, F columns, voxels along K: eight small matrix instructions per 16 voxels,
// so that the kernel takes little more than the time of reading T (2 x 128^3, F = 32:
// 0.090 ms; the library's 0.47-0.70; 0.134 with the two blocks per SM that its 92
// registers allowed unbounded). The columns are permuted so that a lane loads
// F / 8 adjacent channels. Each block leaves its sums in `part`.
template <int F>
__global__ void __launch_bounds__(256, 3) wgrad_edge_kernel(const bf16* __restrict__ s_in,
                                                         const bf16* __restrict__ T, ConvDims d,
                                                         long long tiles, float* __restrict__ part) {
  constexpr int kPX = kInX + 2, kNT = F / 8, kCells = (kInZ + 2) * (kInY + 2) * kPX;
  __shared__ unsigned short in[kCells];
  __shared__ float red[32 * F];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, q = lane & 3;
  int off[4];  // this lane's taps: rows g, g + 8, g + 16, g + 24
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    const int tap = min(g + 8 * j, 26);
    off[j] = (tap / 9 * (kInY + 2) + tap / 3 % 3) * kPX + tap % 3 + warp * kPX + 2 * q;
  }
  const int tap3 = g + 24;
  float acc[2][kNT][4];
#pragma unroll
  for (int i = 0; i < 2; ++i)
#pragma unroll
    for (int t = 0; t < kNT; ++t)
#pragma unroll
      for (int e = 0; e < 4; ++e) acc[i][t][e] = 0.f;
  const int tx = (d.X + kInX - 1) / kInX, ty = (d.Y + kInY - 1) / kInY, tz = (d.Z + kInZ - 1) / kInZ;
  for (long long tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
    long long id = tile;
    const int x0 = (int)(id % tx) * kInX;
    id /= tx;
    const int y0 = (int)(id % ty) * kInY;
    id /= ty;
    const int z0 = (int)(id % tz) * kInZ, b = (int)(id / tz);
    const unsigned short* xs =
        reinterpret_cast<const unsigned short*>(s_in) + (long long)b * d.Z * d.Y * d.X;
    __syncthreads();
    for (int i = threadIdx.x; i < kCells; i += 256) {
      const int ix = i % kPX, iy = i / kPX % (kInY + 2), iz = i / (kPX * (kInY + 2));
      const int gx = x0 + ix - 1, gy = y0 + iy - 1, gz = z0 + iz - 1;
      in[i] = gx >= 0 && gx < d.X && gy >= 0 && gy < d.Y && gz >= 0 && gz < d.Z
                  ? xs[((long long)gz * d.Y + gy) * d.X + gx]
                  : (unsigned short)0;
    }
    __syncthreads();
    const int gy = y0 + warp, nz = gy < d.Y ? min(kInZ, d.Z - z0) : 0;
    unsigned have[2];  // this lane's voxels inside the volume
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int x = x0 + 2 * q + 8 * j;
      have[j] = (x < d.X ? 0xffffu : 0u) | (x + 1 < d.X ? 0xffff0000u : 0u);
    }
    const bf16* tp = T + ((((long long)b * d.Z + z0) * d.Y + gy) * d.X + x0) * F + F / 8 * g;
    for (int k = 0; k < nz; ++k, tp += (long long)d.Y * d.X * F) {
      unsigned v[4][F / 16];  // voxels 2q, 2q + 1, 2q + 8, 2q + 9
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int x = 2 * q + (j & 1) + (j >> 1) * 8;
#pragma unroll
        for (int c = 0; c < F / 16; ++c) v[j][c] = 0u;
        if (x0 + x < d.X) {
          if (F == 32) {
            const uint2 u = __ldg(reinterpret_cast<const uint2*>(tp + x * F));
            v[j][0] = u.x;
            v[j][F / 16 - 1] = u.y;
          } else {
            v[j][0] = __ldg(reinterpret_cast<const unsigned*>(tp + x * F));
          }
        }
      }
      const unsigned short* s = in + k * (kInY + 2) * kPX;
      unsigned a[2][4];
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {  // (tap, tap + 8) x (voxels 2q.., 2q + 8..)
          const unsigned short* r = s + off[2 * i + (j & 1)] + (j >> 1) * 8;
          a[i][j] = ((unsigned)r[0] | (unsigned)r[1] << 16) & have[j >> 1];
        }
      if (tap3 == 27) a[1][1] = a[1][3] = 0x3f803f80u;  // ones
#pragma unroll
      for (int t = 0; t < kNT; ++t) {
        const unsigned sel = t & 1 ? 0x7632u : 0x5410u;
        const unsigned b0 = __byte_perm(v[0][t / 2], v[1][t / 2], sel);
        const unsigned b1 = __byte_perm(v[2][t / 2], v[3][t / 2], sel);
#pragma unroll
        for (int i = 0; i < 2; ++i) warp_mma(acc[i][t], a[i][0], a[i][1], a[i][2], a[i][3], b0, b1);
      }
    }
  }
  // warp by warp, in order
  for (int w = 0; w < 8; ++w) {
    __syncthreads();
    if (warp == w)
#pragma unroll
      for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int t = 0; t < kNT; ++t)
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int c = F / 8 * (2 * q + (e & 1)) + t;  // column 2q + (e & 1) of tile t
            float& r = red[(16 * i + g + 8 * (e >> 1)) * F + c];
            r = w == 0 ? acc[i][t][e] : r + acc[i][t][e];
          }
  }
  __syncthreads();
  for (int i = threadIdx.x; i < 28 * F; i += 256) part[(long long)blockIdx.x * 28 * F + i] = red[i];
}

// Of the middle convolution, dW[co][ci][k] = sum_v g[v][co] h[v + k - 1][ci], on the
// tensor cores with the voxels of a plane along K: A = h with rows (y tap, ci), read
// in place at row offsets of the y halo (the rows of a fourth tap and on are
// ignored), B = g with columns (x tap, co) from three copies shifted in x, one set of
// columns in tensor memory per z tap. The sums stay in tensor memory over all the
// columns a block marches through; each block leaves its own in `part`.
// 2 x 128^3, F = 32: 0.288 ms (the library's 1.4), 0.81 PFLOP/s of wanted products;
// loading through cp.async without the copies of g in global reads took 0.54 ms.
template <int F>
struct Wgrad {
  static constexpr int kRow = F * 2;
  static constexpr int kA = kCX * (kCY + 128 / F - 1) * kRow;  // a plane of h, y halo, ignored rows
  static constexpr int kALoad = kCX * (kCY + 2) * kRow;
  static constexpr int kCopy = kCX * kCY * kRow, kB = 3 * kCopy;  // a plane of g, three times
  static constexpr int kAStages = 6, kBStages = 3;
  static constexpr int kSmem = 1024 + kAStages * kA + kBStages * kB;
  static constexpr int kCols = 9 * F, kAlloc = F == 32 ? 512 : 256;
};

template <int F>
__device__ __forceinline__ unsigned long long wgrad_desc(uint32_t addr, int mn_stride) {
  return (unsigned long long)((addr >> 4) & 0x3fffu) | ((unsigned long long)(mn_stride / 16) << 16) |
         ((unsigned long long)(8 * Mid<F>::kRow / 16) << 32) | (1ull << 46) | (Mid<F>::kLayout << 61);
}

template <int F>
__global__ void __launch_bounds__(192, 1)
    wgrad_mid_kernel(const __grid_constant__ CUtensorMap hmap, const __grid_constant__ CUtensorMap gmap,
                     ConvDims d, MidWork wk, float* __restrict__ part, int* status) {
  typedef Wgrad<F> W;
  extern __shared__ unsigned char conv_dyn[];
  __shared__ __align__(8) unsigned long long bars[2 * (W::kAStages + W::kBStages) + 1];
  __shared__ uint32_t tmem_slot;
  const uint32_t sa = (conv_smem(conv_dyn) + 1023u) & ~1023u, sb = sa + W::kAStages * W::kA;
  const uint32_t a_full = conv_smem(bars), a_empty = a_full + 8 * W::kAStages,
                 b_full = a_empty + 8 * W::kAStages, b_empty = b_full + 8 * W::kBStages,
                 done = b_empty + 8 * W::kBStages;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  if (threadIdx.x == 0) {
    for (int i = 0; i < 2 * (W::kAStages + W::kBStages) + 1; ++i)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(a_full + 8 * i) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     conv_smem(&tmem_slot)),
                 "r"(W::kAlloc)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_slot;
  bool ok = true;

  if (warp == 0 && lane == 0) {  // loads: per z a plane of g and the plane of h above it
    long long na = 0, nb = 0;
    for (long long i = blockIdx.x; ok && i < wk.items; i += gridDim.x) {
      const MidItem it = mid_item(d, wk, i);
      for (int zi = it.z0 - 1; ok && zi <= it.z1; ++zi, ++na) {
        const int s = (int)(na % W::kAStages);
        if (na >= W::kAStages && !(ok = conv_wait(a_empty + 8 * s, (uint32_t)((na / W::kAStages - 1) & 1))))
          break;
        conv_expect(a_full + 8 * s, W::kALoad);
        asm volatile(
            "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
            " [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(sa + s * W::kA),
            "l"(&hmap), "r"(0), "r"(it.x0), "r"(it.y0 - 1), "r"(zi), "r"(it.b), "r"(a_full + 8 * s)
            : "memory");
        const int z = zi - 1;
        if (z < it.z0) continue;
        const int t = (int)(nb % W::kBStages);
        if (nb >= W::kBStages && !(ok = conv_wait(b_empty + 8 * t, (uint32_t)((nb / W::kBStages - 1) & 1)))) {
          ++na;
          break;
        }
        conv_expect(b_full + 8 * t, W::kB);
#pragma unroll
        for (int c = 0; c < 3; ++c)
          asm volatile(
              "cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes"
              " [%0], [%1, {%2, %3, %4, %5, %6}], [%7];" ::"r"(sb + t * W::kB + c * W::kCopy),
              "l"(&gmap), "r"(0), "r"(it.x0 + 1 - c), "r"(it.y0), "r"(z), "r"(it.b), "r"(b_full + 8 * t)
              : "memory");
        ++nb;
      }
    }
    // the last copies land before the block can end
    for (long long k = na > W::kAStages ? na - W::kAStages : 0; k < na; ++k)
      ok &= conv_wait(a_full + 8 * (int)(k % W::kAStages), (uint32_t)((k / W::kAStages) & 1));
    for (long long k = nb > W::kBStages ? nb - W::kBStages : 0; k < nb; ++k)
      ok &= conv_wait(b_full + 8 * (int)(k % W::kBStages), (uint32_t)((k / W::kBStages) & 1));
  } else if (warp == 1) {  // matrix instructions
    const uint32_t e1 = conv_elect();
    const uint32_t idesc = conv_idesc(3 * F) | (1u << 15) | (1u << 16);  // both operands MN-major
    long long na = 0, nb = 0;  // plane z - 1 of h, plane z of g
    for (long long i = blockIdx.x; ok && i < wk.items; i += gridDim.x) {
      const MidItem it = mid_item(d, wk, i);
      for (int z = it.z0; ok && z < it.z1; ++z, ++na, ++nb) {
        for (int k = z == it.z0 ? 0 : 2; ok && k < 3; ++k)
          ok = conv_wait_all(a_full + 8 * (int)((na + k) % W::kAStages), (uint32_t)(((na + k) / W::kAStages) & 1));
        const int t = (int)(nb % W::kBStages);
        if (!ok || !(ok = conv_wait_all(b_full + 8 * t, (uint32_t)((nb / W::kBStages) & 1)))) break;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        const unsigned long long bd = wgrad_desc<F>(sb + t * W::kB, W::kCopy);
        unsigned long long ad[3];
#pragma unroll
        for (int kz = 0; kz < 3; ++kz)
          ad[kz] = wgrad_desc<F>(sa + (int)((na + kz) % W::kAStages) * W::kA, 8 * W::kRow);
        // 16 voxels, two rows of the column, at a time; the z taps in turn, since an
        // instruction waits for the last one on its accumulator
#pragma unroll
        for (int k = 0; k < 8; ++k)
#pragma unroll
          for (int kz = 0; kz < 3; ++kz)
            conv_mma(tmem + kz * 3 * F, ad[kz] + k * W::kRow, bd + k * W::kRow, idesc, nb > 0 || k > 0, e1);
        conv_commit(b_empty + 8 * t, e1);
        conv_commit(a_empty + 8 * (int)(na % W::kAStages), e1);
        if (z == it.z1 - 1) {  // the item's last two planes of h
          conv_commit(a_empty + 8 * (int)((na + 1) % W::kAStages), e1);
          conv_commit(a_empty + 8 * (int)((na + 2) % W::kAStages), e1);
        }
      }
      na += 2;
    }
    conv_commit(done, e1);
    ok &= conv_wait_all(done, 0);
  }
  __syncwarp();
  // every warp sees the sums complete; readers of tensor memory are warps 2-5
  ok = __all_sync(0xffffffffu, ok);
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp >= 2) {
    const int q = warp & 3;
    for (int c = 0; c < W::kCols; c += 16) {
      uint32_t r[16];
      tmem_load16(r, tmem + ((uint32_t)(q * 32) << 16) + c);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (q * 32 + lane < 3 * F) {
#pragma unroll
        for (int j = 0; j < 16; ++j)
          part[((long long)blockIdx.x * W::kCols + c + j) * (3 * F) + q * 32 + lane] = __uint_as_float(r[j]);
      }
    }
  }
  if (!ok) *status = 1;
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (warp == 1)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(W::kAlloc));
}

// A weight gradient voxel by voxel, dW[co][ci][k] = sum_v g[v][co] h[v + k - 1][ci] with
// h zero beyond the volume. The kernels above also multiply zeros in the place of
// gradients beyond it with activations inside, and the last convolution's leaves the
// zeros beyond h out: the same sums, but not where a factor is infinite or NaN. An
// infinity or NaN anywhere shows in the centre tap, whose pairs all lie inside; only
// then (`odd`) does this kernel do its work, on the FP32 pipe, and its sums replace
// theirs. One tap and one run of rows per block. 2 x 128^3, F = 32: all gradients 1.05
// -> 1.06 ms with nothing to do, 44 ms with an infinite voxel.
template <int F, int G>
__global__ void __launch_bounds__(256) wgrad_plain_kernel(const bf16* __restrict__ g, const bf16* __restrict__ h,
                                                          ConvDims d, float* __restrict__ part,
                                                          const int* odd) {
  constexpr int kOuts = F * G, kPer = kOuts >= 256 ? kOuts / 256 : 1;  // outputs, of a thread
  constexpr int kSub = kOuts >= 256 ? 1 : 256 / kOuts;                 // threads of an output
  __shared__ float red[256];
  if (!*odd) return;
  const int tap = blockIdx.x, t = threadIdx.x, ci = t % F, co = t / F % G, sub = t / kOuts;
  const int dz = tap / 9 - 1, dy = tap / 3 % 3 - 1, dx = tap % 3 - 1;
  const long long rows = (long long)d.B * d.Z * d.Y;
  float acc[kPer];
#pragma unroll
  for (int j = 0; j < kPer; ++j) acc[j] = 0.f;
  for (long long r = rows * blockIdx.y / gridDim.y; r < rows * (blockIdx.y + 1) / gridDim.y; ++r) {
    const int y = (int)(r % d.Y) + dy, z = (int)(r / d.Y % d.Z) + dz;
    const bool in = y >= 0 && y < d.Y && z >= 0 && z < d.Z;
    const bf16* gr = g + r * d.X * G + co;
    const bf16* hr = h + (r + (long long)dz * d.Y + dy) * d.X * F + ci;
    for (int x = sub; x < d.X; x += kSub) {
      const bool ok = in && x + dx >= 0 && x + dx < d.X;
      const float hv = ok ? __bfloat162float(hr[(long long)(x + dx) * F]) : 0.f;
#pragma unroll
      for (int j = 0; j < kPer; ++j)
        acc[j] = fmaf(__bfloat162float(gr[(long long)x * G + j * (256 / F)]), hv, acc[j]);
    }
  }
  float* p = part + ((long long)blockIdx.y * 27 + tap) * kOuts + ci;
  if (kSub == 1) {
#pragma unroll
    for (int j = 0; j < kPer; ++j) p[(co + j * (256 / F)) * F] = acc[j];
    return;
  }
  red[t] = acc[0];
  __syncthreads();
  if (t >= kOuts) return;
#pragma unroll
  for (int i = 1; i < kSub; ++i) acc[0] += red[t + i * kOuts];
  p[co * F] = acc[0];
}

// Adds the blocks' sums, element by element in a fixed order, and writes them to a
// weight gradient [out, in, z, y, x] or a bias gradient in BF16. kind 0: rows of F
// sums to a bias. 1, 2: rows [28][F] of wgrad_edge_kernel, to a weight whose one
// channel is the input (1; tap 27 to the bias) or the output (2: the taps run
// backwards). 3: rows [9 F][3 F] of wgrad_mid_kernel. 2 and 3 note in `odd` a
// centre tap that is not finite.
struct ConvGrad {
  bf16* w;
  bf16* b;
  long long s[5];
};
template <int F>
__global__ void __launch_bounds__(1024) conv_sum_kernel(const float* __restrict__ part, int n, int width,
                                                        int kind, ConvGrad out, const int* status,
                                                        int* odd) {
  __shared__ float red[32][33];
  const int e = blockIdx.x * 32 + threadIdx.x;
  float v = 0.f;
  if (e < width)
    for (int i = threadIdx.y; i < n; i += 32) v += part[(long long)i * width + e];
  red[threadIdx.y][threadIdx.x] = v;
  __syncthreads();
  if (threadIdx.y != 0 || e >= width) return;
  v = 0.f;
#pragma unroll
  for (int i = 0; i < 32; ++i) v += red[i][threadIdx.x];
  const bf16 r = __float2bfloat16_rn(*status ? __int_as_float(0x7fffffff) : v);
  if (kind == 0) {
    out.b[e] = r;
  } else if (kind == 3) {
    const int col = e / (3 * F), m = e % (3 * F);
    const int kz = col / (3 * F), kx = col / F % 3, co = col % F, ky = m / F, ci = m % F;
    if (kz == 1 && ky == 1 && kx == 1 && !isfinite(v)) *odd = 1;
    out.w[co * out.s[0] + ci * out.s[1] + kz * out.s[2] + ky * out.s[3] + kx * out.s[4]] = r;
  } else {
    int tap = e / F;
    const int c = e % F;
    if (kind == 2 && tap == 13 && !isfinite(v)) *odd = 1;
    if (tap == 27) {
      if (kind == 1 && out.b) out.b[c] = r;
      return;
    }
    if (!out.w) return;
    if (kind == 2) tap = 26 - tap;
    out.w[c * out.s[kind - 1] + tap / 9 * out.s[2] + tap / 3 % 3 * out.s[3] + tap % 3 * out.s[4]] = r;
  }
}

// The sums of wgrad_plain_kernel's n runs of rows, [27][G][F] each.
template <int F, int G>
__global__ void __launch_bounds__(256) plain_sum_kernel(const float* __restrict__ part, int n, ConvGrad out,
                                                        const int* status, const int* odd) {
  const int e = blockIdx.x * 256 + threadIdx.x;
  if (!*odd || e >= 27 * F * G) return;
  float v = 0.f;
  for (int i = 0; i < n; ++i) v += part[(long long)i * 27 * F * G + e];
  const int tap = e / (F * G), co = e % (F * G) / F, ci = e % F;
  out.w[co * out.s[0] + ci * out.s[1] + tap / 9 * out.s[2] + tap / 3 % 3 * out.s[3] + tap % 3 * out.s[4]] =
      __float2bfloat16_rn(*status ? __int_as_float(0x7fffffff) : v);
}

typedef CUresult (*ConvEncodeFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                 const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                 const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                 CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

ConvEncodeFn conv_encoder() {
  static const ConvEncodeFn enc = [] {
    void* ptr = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &ptr, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      ptr = nullptr;
    return reinterpret_cast<ConvEncodeFn>(ptr);
  }();
  return enc;
}

// planes of a channels-last tensor in boxes of kCX x rows voxels
template <int F>
int conv_map(CUtensorMap* map, const bf16* p, const ConvDims& d, int rows) {
  const ConvEncodeFn enc = conv_encoder();
  if (!enc) return fail(DTV_ERR_CUDA, "cuTensorMapEncodeTiled is not available");
  const cuuint64_t row = Mid<F>::kRow;
  const cuuint64_t dims[5] = {(cuuint64_t)F, (cuuint64_t)d.X, (cuuint64_t)d.Y, (cuuint64_t)d.Z,
                              (cuuint64_t)d.B};
  const cuuint64_t strides[4] = {row, row * d.X, row * d.X * d.Y, row * d.X * d.Y * d.Z};
  const cuuint32_t box[5] = {F, kCX, (cuuint32_t)rows, 1, 1}, es[5] = {1, 1, 1, 1, 1};
  const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 5, const_cast<bf16*>(p), dims, strides, box,
                         es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                         F == 32 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_32B,
                         CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return fail(DTV_ERR_CUDA, "cuTensorMapEncodeTiled failed (%d)", (int)r);
  return DTV_OK;
}

long long conv_tiles(const ConvDims& d, int x, int y, int z) {
  return (long long)((d.X + x - 1) / x) * ((d.Y + y - 1) / y) * ((d.Z + z - 1) / z) * d.B;
}

int conv_sms(int* sms) {
  int dev = 0;
  DTV_CUDA_TRY(cudaGetDevice(&dev));
  DTV_CUDA_TRY(cudaDeviceGetAttribute(sms, cudaDevAttrMultiProcessorCount, dev));
  return DTV_OK;
}

// z chunks: a chunk pays two halo planes; the length with the fewest planes in the
// longest block
MidWork mid_work(const ConvDims& d, int sms) {
  MidWork wk{};
  wk.tx = (d.X + kCX - 1) / kCX;
  wk.ty = (d.Y + kCY - 1) / kCY;
  long long best = -1;
  for (int c = 1; c <= d.Z && c <= 64; ++c) {
    const int len = (d.Z + c - 1) / c, chunks = (d.Z + len - 1) / len;
    const long long items = (long long)wk.tx * wk.ty * d.B * chunks;
    const long long cost = (items + sms - 1) / sms * (len + 2);
    if (best < 0 || cost < best) {
      best = cost;
      wk.zc = len;
      wk.nzc = chunks;
      wk.items = items;
    }
  }
  return wk;
}

template <int F>
int launch_weights(const ConvW& w1, const ConvW& w2, const ConvW& w3, unsigned char* ws, cudaStream_t st) {
  conv_weights_kernel<F><<<(conv_weight_items<F>() + 255) / 256, 256, 0, st>>>(w1, w2, w3, ws);
  note_launch();
  DTV_LAUNCH_CHECK();
  return DTV_OK;
}

template <int F, bool kMask>
int launch_in(const bf16* x, const unsigned char* ws, const bf16* bias, const bf16* act, bf16* out,
              const ConvDims& d, float* sums, cudaStream_t st) {
  const long long n = conv_tiles(d, kInX, kInY, kInZ);
  DTV_CHECK(n < (1ll << 31), "volume too large");
  conv_in_kernel<F, kMask><<<(unsigned)n, 256, 0, st>>>(x, ws + ConvWs<F>::kIn, bias, act, out, d, sums);
  note_launch();
  DTV_LAUNCH_CHECK();
  return DTV_OK;
}

template <int F, bool kMask>
int launch_mid(const bf16* in, unsigned char* ws, const bf16* bias, const bf16* act, bf16* out,
               const ConvDims& d, int sms, cudaStream_t st) {
  CUtensorMap map;
  if (const int rc = conv_map<F>(&map, in, d, kCY + 2)) return rc;
  DTV_CUDA_TRY(cudaFuncSetAttribute(conv_mid_kernel<F, kMask>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    Mid<F>::kSmem));
  const MidWork wk = mid_work(d, sms * kPipes);
  conv_mid_kernel<F, kMask><<<(unsigned)std::min<long long>((wk.items + kPipes - 1) / kPipes, sms), kMidThreads, Mid<F>::kSmem, st>>>(
      map, ws, bias, act, out, d, wk, reinterpret_cast<int*>(ws + ConvWs<F>::kStatus));
  note_launch();
  DTV_LAUNCH_CHECK();
  return DTV_OK;
}

template <int F>
int launch_out(const bf16* h, unsigned char* ws, const bf16* bias, bf16* out, const ConvDims& d, int sms,
               cudaStream_t st) {
  DTV_CUDA_TRY(cudaFuncSetAttribute(conv_out_kernel<F>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    kOutSmem));
  // z chunks: four blocks or so for each of the three places of an SM
  const long long columns = conv_tiles(d, kOutT, kOutT, d.Z);
  const int zc = (int)std::max<long long>(4, std::min<long long>(32, d.Z * columns / (sms * 12)));
  const long long n = conv_tiles(d, kOutT, kOutT, zc);
  DTV_CHECK(n < (1ll << 31), "volume too large");
  conv_out_kernel<F><<<(unsigned)n, 256, kOutSmem, st>>>(h, ws + ConvWs<F>::kOut, bias, out, d, zc,
                                                         reinterpret_cast<int*>(ws + ConvWs<F>::kStatus));
  note_launch();
  DTV_LAUNCH_CHECK();
  return DTV_OK;
}

template <int F>
int conv_block(const bf16* x, const ConvW* w, const bf16* const* bias, bf16* h1, bf16* h2, bf16* y,
               unsigned char* ws, const ConvDims& d, cudaStream_t st) {
  int sms = 0, rc = conv_sms(&sms);
  if (!rc) rc = launch_weights<F>(w[0], w[1], w[2], ws, st);
  if (!rc) rc = launch_in<F, false>(x, ws, bias[0], nullptr, h1, d, nullptr, st);
  if (!rc) rc = launch_mid<F, false>(h1, ws, bias[1], nullptr, h2, d, sms, st);
  if (!rc) rc = launch_out<F>(h2, ws, bias[2], y, d, sms, st);
  return rc;
}

// blocks of the one-channel weight gradients: three fit an SM
int edge_blocks(const ConvDims& d, int sms) {
  return (int)std::min<long long>(conv_tiles(d, kInX, kInY, kInZ), 3LL * sms);
}

// bytes of the blocks' sums, shared by the kernels that leave some
template <int F>
long long conv_sum_bytes(const ConvDims& d, int sms) {
  const long long mid = std::min<long long>(mid_work(d, sms).items, sms) * 27 * F * F;
  return 4 * std::max(std::max(mid, (long long)edge_blocks(d, sms) * 28 * F),
                      conv_tiles(d, kInX, kInY, kInZ) * F);
}

template <int F>
int launch_sum(const float* part, long long n, int width, int kind, const ConvGrad& g, const int* status,
               int* odd, cudaStream_t st) {
  conv_sum_kernel<F><<<(width + 31) / 32, dim3(32, 32), 0, st>>>(part, (int)n, width, kind, g, status, odd);
  note_launch();
  DTV_LAUNCH_CHECK();
  return DTV_OK;
}

// The weight gradient of g and h again, voxel by voxel, if `odd` says so (`part` holds
// the sums of n blocks of it). 22 x 27 blocks are four per SM.
template <int F, int G>
int launch_plain(const bf16* g, const bf16* h, const ConvDims& d, float* part, long long n, const ConvGrad& out,
                 const int* status, const int* odd, cudaStream_t st) {
  n = std::min(n, 22ll);
  wgrad_plain_kernel<F, G><<<dim3(27, (unsigned)n), 256, 0, st>>>(g, h, d, part, odd);
  note_launch();
  DTV_LAUNCH_CHECK();
  plain_sum_kernel<F, G><<<(27 * F * G + 255) / 256, 256, 0, st>>>(part, (int)n, out, status, odd);
  note_launch();
  DTV_LAUNCH_CHECK();
  return DTV_OK;
}

template <int F>
int launch_edge_grad(const bf16* s, const bf16* T, const ConvDims& d, int sms, float* part, int kind,
                     const ConvGrad& g, int* status, int* odd, cudaStream_t st) {
  const int n = edge_blocks(d, sms);
  wgrad_edge_kernel<F><<<n, 256, 0, st>>>(s, T, d, conv_tiles(d, kInX, kInY, kInZ), part);
  note_launch();
  DTV_LAUNCH_CHECK();
  const int rc = launch_sum<F>(part, n, 28 * F, kind, g, status, odd, st);
  return rc || kind != 2 ? rc : launch_plain<F, 1>(s, T, d, part, n, g, status, odd, st);
}

// the kernel of the data gradient: taps backwards, in and out swapped
ConvW conv_flip(const ConvW& w) {
  return ConvW{w.w + 2 * (w.s[2] + w.s[3] + w.s[4]), {w.s[1], w.s[0], -w.s[2], -w.s[3], -w.s[4]}};
}

template <int F>
int conv_block_backward(const bf16* gy, const bf16* x, const ConvW* w, const bf16* h1, const bf16* h2,
                        bf16* g1, bf16* g2, bf16* gx, const ConvGrad* g, unsigned char* ws,
                        const ConvDims& d, cudaStream_t st) {
  typedef Wgrad<F> W;
  int sms = 0, rc = conv_sms(&sms);
  if (rc) return rc;
  int* status = reinterpret_cast<int*>(ws + ConvWs<F>::kStatus);
  float* part = reinterpret_cast<float*>(ws + ConvWs<F>::kStatus + 16);
  rc = launch_weights<F>(conv_flip(w[2]), conv_flip(w[1]), conv_flip(w[0]), ws, st);
  if (!rc && g[2].w) rc = launch_edge_grad<F>(gy, h2, d, sms, part, 2, g[2], status, status + 1, st);
  if (rc || !g2) return rc;
  rc = launch_in<F, true>(gy, ws, nullptr, h2, g2, d, part, st);
  if (!rc && g[1].b)
    rc = launch_sum<F>(part, conv_tiles(d, kInX, kInY, kInZ), F, 0, g[1], status, nullptr, st);
  if (!rc && g[1].w) {
    CUtensorMap hmap, gmap;
    rc = conv_map<F>(&hmap, h1, d, kCY + 2);
    if (!rc) rc = conv_map<F>(&gmap, g2, d, kCY);
    if (rc) return rc;
    DTV_CUDA_TRY(cudaFuncSetAttribute(wgrad_mid_kernel<F>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      W::kSmem));
    const MidWork wk = mid_work(d, sms);
    const long long n = std::min<long long>(wk.items, sms);
    wgrad_mid_kernel<F><<<(unsigned)n, 192, W::kSmem, st>>>(hmap, gmap, d, wk, part, status);
    note_launch();
    DTV_LAUNCH_CHECK();
    rc = launch_sum<F>(part, n, 27 * F * F, 3, g[1], status, status + 2, st);
    if (!rc) rc = launch_plain<F, F>(g2, h1, d, part, n, g[1], status, status + 2, st);
  }
  if (rc || !g1) return rc;
  rc = launch_mid<F, true>(g2, ws, nullptr, h1, g1, d, sms, st);
  if (!rc && (g[0].w || g[0].b)) rc = launch_edge_grad<F>(x, g1, d, sms, part, 1, g[0], status, nullptr, st);
  if (!rc && gx) rc = launch_out<F>(g1, ws, nullptr, gx, d, sms, st);
  return rc;
}

}  // namespace
}  // namespace dtv

using namespace dtv;

int64_t dtv_conv_block_workspace_bytes(int32_t features) {
  return (int64_t)27 * features * features * 2 + 32 * features * 4 + 16;
}

int dtv_conv_block(const void* x, const void* const weights[3], const int64_t strides[15],
                   const void* const biases[3], void* h1, void* h2, void* y, const int32_t size[3],
                   int32_t batch, int32_t features, void* workspace, void* stream) {
  DTV_CHECK(x && weights && strides && biases && h1 && h2 && y && size && workspace, "NULL argument");
  DTV_CHECK(size[0] > 0 && size[1] > 0 && size[2] > 0 && batch > 0, "empty volume");
  DTV_CHECK((int64_t)size[0] * size[1] < (1ll << 31), "plane of 2^31 voxels or more");
  DTV_CHECK(features == 16 || features == 32, "features must be 16 or 32");
  ConvW w[3];
  const bf16* bias[3];
  for (int i = 0; i < 3; ++i) {
    DTV_CHECK(weights[i] && biases[i], "NULL argument");
    w[i].w = static_cast<const bf16*>(weights[i]);
    for (int k = 0; k < 5; ++k) w[i].s[k] = strides[5 * i + k];
    bias[i] = static_cast<const bf16*>(biases[i]);
  }
  DTV_CHECK(((uintptr_t)h1 | (uintptr_t)h2 | (uintptr_t)workspace) % 16 == 0, "buffers must be 16-byte aligned");
  const ConvDims d{size[0], size[1], size[2], batch};
  return (features == 32 ? conv_block<32> : conv_block<16>)(
      static_cast<const bf16*>(x), w, bias, static_cast<bf16*>(h1), static_cast<bf16*>(h2),
      static_cast<bf16*>(y), static_cast<unsigned char*>(workspace), d, static_cast<cudaStream_t>(stream));
}

int64_t dtv_conv_block_backward_workspace_bytes(const int32_t size[3], int32_t batch, int32_t features) {
  if (!size || size[0] <= 0 || size[1] <= 0 || size[2] <= 0 || batch <= 0 || (features != 16 && features != 32))
    return 0;
  int sms = 0;
  if (conv_sms(&sms)) return 0;
  const ConvDims d{size[0], size[1], size[2], batch};
  return dtv_conv_block_workspace_bytes(features) +
         (features == 32 ? conv_sum_bytes<32>(d, sms) : conv_sum_bytes<16>(d, sms));
}

int dtv_conv_block_backward(const void* gy, const void* x, const void* const weights[3],
                            const int64_t strides[15], const void* h1, const void* h2, void* g1, void* g2,
                            void* gx, void* const grad_weights[3], const int64_t grad_strides[15],
                            void* const grad_biases[3], const int32_t size[3], int32_t batch,
                            int32_t features, void* workspace, void* stream) {
  DTV_CHECK(gy && x && weights && strides && h1 && h2 && grad_weights && grad_strides && grad_biases &&
                size && workspace, "NULL argument");
  DTV_CHECK(size[0] > 0 && size[1] > 0 && size[2] > 0 && batch > 0, "empty volume");
  DTV_CHECK((int64_t)size[0] * size[1] < (1ll << 31), "plane of 2^31 voxels or more");
  DTV_CHECK(features == 16 || features == 32, "features must be 16 or 32");
  ConvW w[3];
  ConvGrad g[3];
  for (int i = 0; i < 3; ++i) {
    DTV_CHECK(weights[i], "NULL argument");
    w[i].w = static_cast<const bf16*>(weights[i]);
    g[i].w = static_cast<bf16*>(grad_weights[i]);
    g[i].b = static_cast<bf16*>(grad_biases[i]);
    for (int k = 0; k < 5; ++k) {
      w[i].s[k] = strides[5 * i + k];
      g[i].s[k] = grad_strides[5 * i + k];
    }
  }
  DTV_CHECK(!g[2].b, "the last bias's gradient is the sum of gy");
  DTV_CHECK(g2 || !(g1 || g[1].w || g[1].b), "g2 is needed");
  DTV_CHECK(g1 || !(gx || g[0].w || g[0].b), "g1 is needed");
  DTV_CHECK(((uintptr_t)h1 | (uintptr_t)h2 | (uintptr_t)g1 | (uintptr_t)g2 | (uintptr_t)workspace) % 16 == 0,
            "buffers must be 16-byte aligned");
  const ConvDims d{size[0], size[1], size[2], batch};
  return (features == 32 ? conv_block_backward<32> : conv_block_backward<16>)(
      static_cast<const bf16*>(gy), static_cast<const bf16*>(x), w, static_cast<const bf16*>(h1),
      static_cast<const bf16*>(h2), static_cast<bf16*>(g1), static_cast<bf16*>(g2), static_cast<bf16*>(gx),
      g, static_cast<unsigned char*>(workspace), d, static_cast<cudaStream_t>(stream));
}
