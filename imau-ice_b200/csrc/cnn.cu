// cnn.cu -- the learned warm start of the DIVA solve (include/diva_cnn.h): a small
// encoder-decoder network on the a-grid, trained on solutions of this solver, whose
// prediction sets u_vav_cx / v_vav_cy before the viscosity iteration starts.
//
// Every 3x3 convolution is an implicit GEMM on the 5th-generation tensor cores:
//   forward  D[pixel][cout] = sum_(tap,cin)  X[pixel+tap][cin]     W[tap][cout][cin]
//   dgrad    D[pixel][cin]  = sum_(tap,cout) dZ[pixel-tap][cout]   W[tap][cout][cin]
//   wgrad    D[cout][cin]   = sum_pixel      dZ[pixel][cout]       X[pixel+tap][cin]
// (dZ: the gradient of a layer's output masked by its ReLU; the kernel that writes a
// gradient masks it, so every later reader takes it as it stands).  A persistent CTA
// copies an image tile with its one-pixel halo into shared memory once (cp.async, zeros
// outside the image), in the no-swizzle core-matrix layout -- 16-byte chunks of 8
// channels, consecutive pixels 16 bytes apart, one plane per chunk -- so that a tap is a
// shifted start address of the same tile: no operand is gathered twice.  One elected
// thread issues the tcgen05.mma instructions (K = 16 each) with FP32 accumulators in
// tensor memory and commits them to an mbarrier; the epilogue reads them back with
// tcgen05.ld.  The weight gradient takes the same pixel-major tiles as MN-major operands
// and keeps the sums of all its taps in tensor memory over every tile of the CTA; the
// CTAs' sums are added in a fixed order afterwards, so training is deterministic.
//
// Pooling, the 1x1 head with the masked squared-error loss, and Adam are elementwise or
// reduction kernels on CUDA cores; upsampling + concatenation happens in the loads of
// the convolutions that read it.  Every mbarrier wait is bounded; on time-out the kernel
// raises the network's error flag and frees its tensor memory, and the host returns
// DIVA_TIMEOUT.
#include <cuda_bf16.h>
#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <vector>
#include "cnn_tiles.hpp"
#include "ctx.hpp"
#include "../../include/diva_cnn.h"

namespace diva {
namespace cnn {

using bf16 = __nv_bfloat16;

constexpr int kInC = 16;            // input channels (8 used)
constexpr double kVelScale = 10.0;  // m/yr; outputs are asinh(u / kVelScale)
constexpr long kSpin = 1L << 22;    // mbarrier polls before a wait gives up

// ---------------------------------------------------------------------------
// PTX wrappers (sm_100a)
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* b, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity) {
  for (long it = 0; it < kSpin; ++it) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(done)
        : "r"(smem_u32(b)), "r"(parity)
        : "memory");
    if (done) return true;
  }
  return false;
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_alloc(uint32_t* dst, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)),
               "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tc_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
// D[tmem] (+)= A[smem] * B[smem]^T, both K-major; acc = 0 overwrites D
__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc)
      : "memory");
}
__device__ __forceinline__ void tc_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
                   smem_u32(bar))
               : "memory");
}
// 16 consecutive FP32 columns of this thread's lane
__device__ __forceinline__ void tc_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
      "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int q = 0; q < 16; ++q) v[q] = __uint_as_float(r[q]);
}

// Shared-memory matrix descriptor, no swizzle: start, leading (K) and stride (8-row)
// byte offsets in 16-byte units, descriptor version 1 (bit 46).
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// A descriptor whose start address lies `off` 16-byte units further on (the addresses of a
// CTA's shared memory stay below the 14-bit field's end).  One thread issues all MMAs, so
// their rate is that of its instructions: forming each descriptor from scratch took longer
// than the MMA itself at these tile sizes.
__device__ __forceinline__ uint64_t sdesc_at(uint64_t d, uint32_t off) {
  return (d & 0xFFFFFFFF00000000ull) | (uint64_t)((uint32_t)d + off);
}
// Instruction descriptor, kind::f16: D FP32 (bits 4-5 = 1), A and B BF16 (bits 7-9,
// 10-12 = 1), both K-major, N >> 3 at bit 17, M >> 4 at bit 24.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

template <int N>
__host__ __device__ constexpr int tmem_cols() {
  return N <= 32 ? 32 : N <= 64 ? 64 : N <= 128 ? 128 : N <= 256 ? 256 : 512;
}

// zero the lanes of v whose BF16 gate value is not > 0 (ReLU derivative)
__device__ __forceinline__ uint4 relu_gate(uint4 v, uint4 g) {
  uint32_t* pv = &v.x;
  const uint32_t* pg = &g.x;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    uint32_t m = 0;
    if ((int16_t)(pg[q] & 0xFFFFu) > 0) m |= 0x0000FFFFu;
    if ((int16_t)(pg[q] >> 16) > 0) m |= 0xFFFF0000u;
    pv[q] &= m;
  }
  return v;
}

__device__ __forceinline__ unsigned char* align128(unsigned char* p) {
  return reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(p) + 127) & ~uintptr_t(127));
}
// 16 bytes global -> shared without registers; zeros when !in (src is then not read)
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool in) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The input of a 3x3 layer: one tensor [n][H][W][C], or the concatenation of a tensor at half
// the resolution (lo, its first C1 channels, read at (y/2, x/2)) and one at the full (x).
struct Input {
  const bf16 *x, *lo;
  int c1;   // channels from lo (0: none)
};
constexpr int kConvThreads = 256;

// Stage `rows` image rows from y0 (possibly -1) and `cols` pixels from x0 (possibly -1) of the
// C-channel input of image b: pixel (r, xx), chunk c8 at dst + r rpitch + c8 cpitch + 16 xx
// bytes, zeros outside the image.  A thread keeps its (pixel, chunk) positions of a row and
// walks down the rows with two additions per copy; recomputing every chunk's address from
// scratch made the copies' instructions the bound of the tiles.
template <int C>
__device__ __forceinline__ void stage_rows(uint32_t dst, int rpitch, int cpitch, const Input& in, int H, int W, int b,
                                           int y0, int rows, int x0, int cols) {
  constexpr int C8 = C / 8;
  for (int e = threadIdx.x; e < cols * C8; e += kConvThreads) {
    const int c8 = e % C8, xx = e / C8, x = x0 + xx;
    const bool xin = x >= 0 && x < W, low = c8 * 8 < in.c1;
    const int xc = xin ? x : 0;
    const char* src;   // row 0 of the image
    int stride;        // bytes per row
    if (low) {
      src = reinterpret_cast<const char*>(in.lo + ((long)b * (H / 2) * (W / 2) + xc / 2) * in.c1 + c8 * 8);
      stride = (W / 2) * in.c1 * 2;
    } else {
      src = reinterpret_cast<const char*>(in.x + ((long)b * H * W + xc) * (C - in.c1) + c8 * 8 - in.c1);
      stride = W * (C - in.c1) * 2;
    }
    uint32_t d = dst + c8 * cpitch + xx * 16;
    const int sh = low ? 1 : 0;
#pragma unroll 4
    for (int r = 0; r < rows; ++r, d += rpitch) {
      const int y = y0 + r;
      const bool ok = xin && y >= 0 && y < H;
      cp16(d, src + (ok ? (long)(y >> sh) * stride : 0), ok);
    }
  }
}

// ---------------------------------------------------------------------------
// forward / dgrad 3x3 convolution
// ---------------------------------------------------------------------------
// A tile is TH x TW output pixels; its input, with the halo, is staged as (TH+2) rows of
// P = TW + 2 pixels, row after row.  An accumulator block is 128 consecutive positions of
// that pitch-P order (row m of D = position 128 blk + m), so that tap (ty, tx) of every
// position is the same tile ty P + tx pixels further on: the two halo columns of a row
// are computed as well and dropped (2 of P), instead of staging each tap's operand anew.
struct ConvArgs {
  Input in;          // forward input, or (dgrad) dZ of the layer
  const bf16* w;     // forward: W [9][COUT][CIN]; dgrad: W^T [9][CIN][COUT]
  const float* bias; // forward: [COUT]
  const bf16* mask;  // dgrad: the tensor whose ReLU masks the result, or null
  bf16* y;           // [n][H][W][NO]
  int n, H, W;
  int* err;
  ConvTile t;
};

// Bound by the rate at which the tensor core takes K = 16 MMAs from unswizzled operands (about
// 100 cycles each) and by the tile copies.  On 8 samples of 561 x 321 the 32 -> 32 layer takes
// 92 us, the 64 -> 32 one 170 us (2 x 93 MB and 4 x 93 MB in and out); a kernel that gathered
// its 128-pixel operand per tap, nine copies of the input through L2 with a barrier each, took
// 274 and 892 us.
template <int KC, int NO, bool DGRAD>
__global__ void __launch_bounds__(kConvThreads) k_conv3x3(ConvArgs a) {
  static_assert(KC % 16 == 0 && NO % 32 == 0 && NO <= 128, "tile shape");
  constexpr int C8 = KC / 8, NB = conv_blocks(KC, NO);
  constexpr int WL = conv_wplane(KC, NO), WT = C8 * WL;
  constexpr int NCOL = tmem_cols<NB * NO>();
  constexpr uint32_t IDESC = idesc_bf16(128, NO);
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bar;
  __shared__ uint32_t taddr_s;
  __shared__ __align__(16) float sbias[NO];
  unsigned char* Ws = align128(smem_raw);
  unsigned char* Xs = Ws + conv_wbytes(KC, NO);
  const uint32_t ws = smem_u32(Ws), xs = smem_u32(Xs);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int H = a.H, W = a.W, P = a.t.P, npx = a.t.npx;

  if (tid == 0) {
    mbar_init(&bar, 1);
    fence_mbar_init();
  }
  if (warp == 0) tc_alloc(&taddr_s, NCOL);
  if (!DGRAD && tid < NO) sbias[tid] = a.bias[tid];
  // the weights of all taps, once per CTA: B(n, k) of tap t at t WT + (k/8) WL + 16 n
  for (int i = tid; i < 9 * NO * C8; i += kConvThreads) {
    const int c8 = i % C8, r = i / C8;   // r = t NO + n
    cp16(ws + (r / NO) * WT + c8 * WL + (r % NO) * 16, a.w + (long)r * KC + c8 * 8, true);
  }
  auto origin = [&](int tile, int& b, int& y0, int& x0) {
    const int c = tile % a.t.ncol, q = tile / a.t.ncol;
    x0 = c * a.t.TW;
    y0 = (q % a.t.nrow) * a.t.TH;
    b = q / a.t.nrow;
  };
  auto stage = [&](int tile) {
    int b, y0, x0;
    origin(tile, b, y0, x0);
    stage_rows<KC>(xs, P * 16, npx * 16, a.in, H, W, b, y0 - 1, a.t.TH + 2, x0 - 1, P);
  };
  int tile = blockIdx.x;
  if (tile < a.t.ntile) stage(tile);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = taddr_s;
  bool ok = true;
  uint32_t phase = 0;
  for (; tile < a.t.ntile; tile += gridDim.x) {
    cp_wait_all();
    fence_async_smem();
    tc_fence_before();   // the previous tile's accumulator reads before this tile's MMAs
    __syncthreads();
    if (tid == 0) {
      tc_fence_after();
      const uint64_t da0 = sdesc(xs, npx * 16, 128), db0 = sdesc(ws, WL, 128);
#pragma unroll 1
      for (int blk = 0; blk < NB; ++blk) {
        const uint32_t d = tmem + blk * NO;
        uint32_t ao = blk * 128 + (DGRAD ? 2 * P + 2 : 0), bo = 0;   // dgrad: the taps mirrored
#pragma unroll 1
        for (int ty = 0; ty < 3; ++ty) {
#pragma unroll
          for (int tx = 0; tx < 3; ++tx)
#pragma unroll
            for (int k = 0; k < KC / 16; ++k)
              tc_mma(d, sdesc_at(da0, ao + 2 * k * npx + (DGRAD ? -tx : tx)),
                     sdesc_at(db0, bo + (tx * WT + 2 * k * WL) / 16), IDESC, (ty > 0 || tx > 0 || k > 0) ? 1u : 0u);
          ao += DGRAD ? -P : P;
          bo += 3 * WT / 16;
        }
      }
      tc_commit(&bar);
    }
    ok = mbar_wait(&bar, phase) && ok;
    phase ^= 1;
    tc_fence_after();
    ok = __syncthreads_and(ok);
    if (!ok) break;
    int b, y0, x0;
    origin(tile, b, y0, x0);
    if (tile + (int)gridDim.x < a.t.ntile) stage(tile + gridDim.x);   // overlaps the epilogue
    // warps 4g..4g+3 read block g (two blocks) or column half g (one block)
    const int g = warp >> 2, blk = NB == 2 ? g : 0;
    constexpr int NC = NB == 2 ? NO : NO / 2;
    const int c0 = NB == 2 ? 0 : g * NC;
    const int pos = blk * 128 + (warp & 3) * 32 + lane, py = pos / P, px = pos % P;
    const bool pin = py < a.t.TH && px < a.t.TW && y0 + py < H && x0 + px < W;
    const long out = (((long)b * H + y0 + py) * W + x0 + px) * NO + c0;
#pragma unroll
    for (int n0 = 0; n0 < NC; n0 += 16) {
      float v[16];
      tc_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(blk * NO + c0 + n0), v);
      if (pin) {
        __align__(16) bf16 o[16];
#pragma unroll
        for (int q4 = 0; q4 < 4; ++q4) {
          float4 b4 = make_float4(0.f, 0.f, 0.f, 0.f);
          if (!DGRAD) b4 = *reinterpret_cast<const float4*>(sbias + c0 + n0 + 4 * q4);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            float f = v[4 * q4 + q];
            if (!DGRAD) f = fmaxf(f + (&b4.x)[q], 0.0f);
            o[4 * q4 + q] = __float2bfloat16_rn(f);
          }
        }
        uint4 o0 = reinterpret_cast<const uint4*>(o)[0], o1 = reinterpret_cast<const uint4*>(o)[1];
        if (DGRAD && a.mask) {
          const uint4* m = reinterpret_cast<const uint4*>(a.mask + out + n0);
          o0 = relu_gate(o0, m[0]);
          o1 = relu_gate(o1, m[1]);
        }
        uint4* dst = reinterpret_cast<uint4*>(a.y + out + n0);
        dst[0] = o0;
        dst[1] = o1;
      }
    }
  }
  if (!ok && tid == 0) atomicExch(a.err, 1);
  cp_wait_all();
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tc_dealloc(tmem, NCOL);
  }
}

// ---------------------------------------------------------------------------
// wgrad: every tap's D[cout][cin] over the pixels of the CTA's tiles, and the bias gradient
// ---------------------------------------------------------------------------
// A tile is TH rows of X (TW + 2 pixels, halo columns included) and the TH + 2 rows of dZ
// (TW pixels) that they meet.  K runs over 16 pixels of a row; both operands are MN-major
// (8 channels contiguous), a tap's column shift is a start address one pixel further on.
// dZ is staged [row][8-channel chunk][pixel], so the 16 chunk groups of a 128-row A operand
// run on into the following dZ rows: one MMA forms 128 / COUT vertical taps at once
// (COUT = 32: all three, the last 32 rows of D unused; 64: two and one; 128: one each).
struct WgradArgs {
  Input in;          // the layer's input
  const bf16* dz;    // masked gradient of the layer's output [n][H][W][CO]
  float* part;       // [nsplit][9 CO CI + CO]
  int n, H, W;
  int* err;
  WgradTile t;
};
// A CTA (blockIdx.y) takes one set of vertical taps of the layer and one horizontal tap; the
// slices of the pixels (blockIdx.x) are as many as keep the chains short (wgrad_tile).
template <int CO>
__host__ __device__ constexpr int wgrad_sets() {
  return CO == 32 ? 1 : CO == 64 ? 2 : 3;
}

// Bound by the copies of its tiles and the MMA issue of its CTAs (about 3000 and 2700 cycles a
// tile).  436 us for the 32 -> 32 layer on 8 samples of 561 x 321 with its bias
// gradient; one tap per CTA, with both operands transposed by 2-byte shared-memory stores, took
// 958 us and 1 to 2 ms for the bias in a kernel of its own.
template <int CI, int CO>
__global__ void __launch_bounds__(kConvThreads) k_conv3x3_wgrad(WgradArgs a) {
  static_assert(CI % 16 == 0 && CI <= 128 && (CO == 32 || CO == 64 || CO == 128), "tile shape");
  constexpr int O8 = CO / 8, NT = 128 / CO;   // NT: vertical taps per MMA
  constexpr int NCOL = tmem_cols<CI>();
  constexpr uint32_t IDESC = idesc_bf16(128, CI) | (1u << 15) | (1u << 16);   // A and B MN-major
  extern __shared__ unsigned char smem_raw[];
  __shared__ __align__(8) uint64_t bar[2];
  __shared__ uint32_t taddr_s;
  __shared__ float bsum[kConvThreads];
  const int TW = a.t.TW, TH = a.t.TH, zp = a.t.zp, xp = a.t.xp, XW = TW + 2;
  unsigned char* sm = align128(smem_raw);
  const int xoff = (TH + 2) * O8 * zp * 16;   // X after dZ in each buffer
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int H = a.H, W = a.W, set = blockIdx.y / 3, dx = blockIdx.y % 3;

  if (tid == 0) {
    mbar_init(&bar[0], 1);
    mbar_init(&bar[1], 1);
    fence_mbar_init();
  }
  if (warp == 0) tc_alloc(&taddr_s, NCOL);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = taddr_s;
  auto stage = [&](int tile, int buf) {
    const uint32_t zs = smem_u32(sm + buf * a.t.buf), xs = zs + xoff;
    const int c = tile % a.t.ncol, q = tile / a.t.ncol;
    const int x0 = c * TW, y0 = (q % a.t.nrow) * TH, b = q / a.t.nrow;
    stage_rows<CO>(zs, O8 * zp * 16, zp * 16, Input{a.dz, nullptr, 0}, H, W, b, y0 - 1, TH + 2, x0, TW);
    stage_rows<CI>(xs, XW * 16, xp * 16, a.in, H, W, b, y0, TH, x0 - 1, XW);
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  bool ok = true, any = false;
  uint32_t phase[2] = {0, 0};
  float bias = 0.0f;   // channel tid % CO over the pixel slice tid / CO
  int it = 0;
  if ((int)blockIdx.x < a.t.ntile) stage(blockIdx.x, 0);
  for (int tile = blockIdx.x; tile < a.t.ntile; tile += gridDim.x, ++it) {
    const int buf = it & 1;
    const bool more = tile + (int)gridDim.x < a.t.ntile;
    if (more) {   // the next tile's copies run beside this tile's MMAs, once the last ones are done
      if (it > 0) {
        ok = mbar_wait(&bar[buf ^ 1], phase[buf ^ 1]) && ok;
        phase[buf ^ 1] ^= 1;
        __syncthreads();   // and the bias sums' reads of that buffer
      }
      stage(tile + gridDim.x, buf ^ 1);
      asm volatile("cp.async.wait_group 1;" ::: "memory");
    } else {
      cp_wait_all();
    }
    fence_async_smem();
    ok = __syncthreads_and(ok);
    if (!ok) break;
    unsigned char* Zs = sm + buf * a.t.buf;
    const uint32_t zs = smem_u32(Zs), xs = zs + xoff;
    if (tid == 0) {
      tc_fence_after();
      const uint64_t da0 = sdesc(zs + set * NT * O8 * zp * 16, 128, zp * 16), db0 = sdesc(xs + dx * 16, 128, xp * 16);
      uint32_t ao = 0, bo = 0, acc = any ? 1u : 0u;
#pragma unroll 1
      for (int r = 0; r < TH; ++r, ao += O8 * zp, bo += XW)
#pragma unroll 1
        for (int x = 0; x < TW; x += 16, acc = 1u) tc_mma(tmem, sdesc_at(da0, ao + x), sdesc_at(db0, bo + x), IDESC, acc);
      tc_commit(&bar[buf]);
    }
    any = true;
    if (blockIdx.y == 0) {   // the bias gradient: the tile's own rows of dZ (zeros outside the image)
      const int co = tid % CO;
      const unsigned char* z = Zs + (O8 + co / 8) * zp * 16 + (co % 8) * 2;
      for (int r = 0; r < TH; ++r, z += O8 * zp * 16)
        for (int xx = tid / CO; xx < TW; xx += kConvThreads / CO)
          bias += __bfloat162float(*reinterpret_cast<const bf16*>(z + xx * 16));
    }
  }
  // the last one or two tiles' MMAs
  if (ok && it > 1) ok = mbar_wait(&bar[it & 1], phase[it & 1]);
  if (ok && it > 0) ok = mbar_wait(&bar[(it - 1) & 1], phase[(it - 1) & 1]) && ok;
  tc_fence_after();
  cp_wait_all();
  ok = __syncthreads_and(ok);
  float* dst = a.part + (long)blockIdx.x * (9 * CO * CI + CO);
  if (ok) {
    // row r of D: vertical tap (r / CO) of its set, cout r % CO; the dZ row above the X row
    // (index 0) is the tap dy = +1
    const int r = (warp & 3) * 32 + lane, g = warp >> 2;
#pragma unroll 1
    for (int n0 = g * 16; n0 < CI; n0 += 32) {
      float v[16];
      if (any) {
        tc_ld16(tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)n0, v);
      } else {
#pragma unroll
        for (int k = 0; k < 16; ++k) v[k] = 0.0f;
      }
      const int dyi = set * NT + r / CO;
      if (dyi < 3) {
        float4* o = reinterpret_cast<float4*>(dst + ((long)(3 * (2 - dyi) + dx) * CO + r % CO) * CI + n0);
#pragma unroll
        for (int k = 0; k < 4; ++k) o[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
      }
    }
    if (blockIdx.y == 0) {
      bsum[tid] = bias;
      __syncthreads();
      if (tid < CO) {
        float s = 0.0f;
        for (int k = tid; k < kConvThreads; k += CO) s += bsum[k];
        dst[9 * CO * CI + tid] = s;
      }
    }
  } else if (tid == 0) {
    atomicExch(a.err, 1);
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tc_dealloc(tmem, NCOL);
  }
}

// ---------------------------------------------------------------------------
// reductions, elementwise layers, head + loss, Adam
// ---------------------------------------------------------------------------
// out[c] = sum over r of part[r][c] in a fixed order: 8 threads per column take every eighth
// row, their sums are added in turn (deterministic)
__global__ void __launch_bounds__(256) k_sum_rows(const float* part, int nrows, int ncols, float* out) {
  __shared__ float sh[8][32];
  const int c = blockIdx.x * 32 + threadIdx.x;
  float s = 0.0f;
  if (c < ncols) {
#pragma unroll 8
    for (int r = threadIdx.y; r < nrows; r += 8) s += part[(long)r * ncols + c];
  }
  sh[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && c < ncols) {
    for (int k = 1; k < 8; ++k) s += sh[k][threadIdx.x];
    out[c] = s;
  }
}
// out[0] = sum of part[0..n) by one block, in a fixed order
__global__ void __launch_bounds__(1024) k_sum_all(const float* part, int n, float* out) {
  __shared__ float sh[32];
  float s = 0.0f;
  for (int i = threadIdx.x; i < n; i += 1024) s += part[i];
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    s = sh[threadIdx.x];
    for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
    if (threadIdx.x == 0) out[0] = s;
  }
}

// 2x2 average pool, 8 channels per thread
__global__ void k_pool(const bf16* x, bf16* y, int n, int H, int W, int C) {
  const int H2 = H / 2, W2 = W / 2, C8 = C / 8;
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long)n * H2 * W2 * C8) return;
  const int c8 = (int)(i % C8);
  long q = i / C8;
  const int X = (int)(q % W2);
  q /= W2;
  const int Y = (int)(q % H2), b = (int)(q / H2);
  float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
  for (int d = 0; d < 4; ++d) {
    const long src = (((long)b * H + 2 * Y + (d >> 1)) * W + 2 * X + (d & 1)) * C + c8 * 8;
    const uint4 v = *reinterpret_cast<const uint4*>(x + src);
    const bf16* e = reinterpret_cast<const bf16*>(&v);
#pragma unroll
    for (int k = 0; k < 8; ++k) s[k] += __bfloat162float(e[k]);
  }
  __align__(16) bf16 o[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) o[k] = __float2bfloat16_rn(0.25f * s[k]);
  *reinterpret_cast<uint4*>(y + (((long)b * H2 + Y) * W2 + X) * C + c8 * 8) = *reinterpret_cast<uint4*>(o);
}

// g_hi = (g_hi + 0.25 g_lo) masked by the ReLU of act: the adjoint of the 2x2 average pool
// added to the gradient from the skip connection, which completes that tensor's gradient
__global__ void k_pool_bwd_add(const bf16* glo, const bf16* act, bf16* ghi, int n, int H, int W, int C) {
  const int C8 = C / 8;
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (long)n * H * W * C8) return;
  const int c8 = (int)(i % C8);
  long q = i / C8;
  const int x = (int)(q % W);
  q /= W;
  const int y = (int)(q % H), b = (int)(q / H);
  const long dst = (((long)b * H + y) * W + x) * C + c8 * 8;
  const long src = (((long)b * (H / 2) + y / 2) * (W / 2) + x / 2) * C + c8 * 8;
  uint4 vh = *reinterpret_cast<const uint4*>(ghi + dst);
  const uint4 vl = *reinterpret_cast<const uint4*>(glo + src);
  bf16* eh = reinterpret_cast<bf16*>(&vh);
  const bf16* el = reinterpret_cast<const bf16*>(&vl);
#pragma unroll
  for (int k = 0; k < 8; ++k) eh[k] = __float2bfloat16_rn(__bfloat162float(eh[k]) + 0.25f * __bfloat162float(el[k]));
  *reinterpret_cast<uint4*>(ghi + dst) = relu_gate(vh, *reinterpret_cast<const uint4*>(act + dst));
}

// adjoint of the upsampling + concatenation [lo (nearest x2), skip]: g_lo = sum of the 4
// children, masked by the ReLU of alo; g_skip = its slice (written, not yet masked)
__global__ void k_upcat_bwd(const bf16* gout, const bf16* alo, bf16* glo, bf16* gskip, int n, int H, int W, int C1, int C2) {
  const int C = C1 + C2;
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long nlo = (long)n * (H / 2) * (W / 2) * (C1 / 8);
  const long nsk = (long)n * H * W * (C2 / 8);
  if (i < nlo) {
    const int c8 = (int)(i % (C1 / 8));
    long q = i / (C1 / 8);
    const int X = (int)(q % (W / 2));
    q /= (W / 2);
    const int Y = (int)(q % (H / 2)), b = (int)(q / (H / 2));
    float s[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int d = 0; d < 4; ++d) {
      const uint4 v = *reinterpret_cast<const uint4*>(
          gout + (((long)b * H + 2 * Y + (d >> 1)) * W + 2 * X + (d & 1)) * C + c8 * 8);
      const bf16* e = reinterpret_cast<const bf16*>(&v);
#pragma unroll
      for (int k = 0; k < 8; ++k) s[k] += __bfloat162float(e[k]);
    }
    __align__(16) bf16 o[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) o[k] = __float2bfloat16_rn(s[k]);
    const long dst = (((long)b * (H / 2) + Y) * (W / 2) + X) * C1 + c8 * 8;
    *reinterpret_cast<uint4*>(glo + dst) =
        relu_gate(*reinterpret_cast<uint4*>(o), *reinterpret_cast<const uint4*>(alo + dst));
  } else if (i < nlo + nsk) {
    const long r = i - nlo;
    const int c8 = (int)(r % (C2 / 8));
    const long pix = r / (C2 / 8);
    *reinterpret_cast<uint4*>(gskip + pix * C2 + c8 * 8) =
        *reinterpret_cast<const uint4*>(gout + pix * C + C1 + c8 * 8);
  }
}

// The 1x1 head (FP32 weights, BF16 input): out[o] = sum_c W[o][c] d1[c] + b[o] for the
// kOut state channels.  With targets: the masked squared error (per-block partial sums
// into part[block]), dL/d(out) into dout (FP32, for the weight gradient) and dL/d(d1)
// (BF16).  Channel validity: 0 and 2 on cx points (x < nx-1, y < ny), 1 and 3 on cy
// points (y < ny-1, x < nx), 4 .. 4+nz-1 on a points, the rest never.
constexpr int kHeadC = 32;
constexpr int kOut = 20;
constexpr int kMaxNzOut = kOut - 4;
__device__ __forceinline__ bool out_valid(int o, int x, int y, int nx, int ny, int nz) {
  if (o == 0 || o == 2) return x < nx - 1 && y < ny;
  if (o == 1 || o == 3) return y < ny - 1 && x < nx;
  return o < 4 + nz && x < nx && y < ny;
}
struct LossWeights {
  float w[kOut];
};

// One thread per pixel.  The weights are read from shared memory four at a time (a broadcast:
// every thread needs the same ones); read from global memory, one load per multiply-add made
// the load unit the bound (326 us for 8 training samples of 561 x 321, whose tensors cross
// HBM in 65 us).  With targets, gd1 is masked by the ReLU of d1.  out and tgt may be a caller's
// buffers at any float's address: four floats at a time where both lie on 16 bytes (WIDE), else
// one by one.
template <bool WIDE>
__global__ void __launch_bounds__(128) k_head(const bf16* d1, const float* wh, const float* bh, float* out,
                                              const float* tgt, float* dout, bf16* gd1, float* part, int n, int H,
                                              int W, int ny, int nx, int nz, float inv_count, LossWeights lw) {
  __shared__ float red[4];
  __shared__ __align__(16) float sw[kOut * kHeadC];
  __shared__ float sb[kOut];
  for (int i = threadIdx.x; i < kOut * kHeadC; i += 128) sw[i] = wh[i];
  if (threadIdx.x < kOut) sb[threadIdx.x] = bh[threadIdx.x];
  __syncthreads();
  const long p = (long)blockIdx.x * blockDim.x + threadIdx.x;
  const long npix = (long)n * H * W;
  float se = 0.0f;
  if (p < npix) {
    float f[kHeadC];
#pragma unroll
    for (int c8 = 0; c8 < kHeadC / 8; ++c8) {
      const uint4 v = *reinterpret_cast<const uint4*>(d1 + p * kHeadC + c8 * 8);
      const bf16* e = reinterpret_cast<const bf16*>(&v);
#pragma unroll
      for (int k = 0; k < 8; ++k) f[c8 * 8 + k] = __bfloat162float(e[k]);
    }
    float gd[kHeadC];
#pragma unroll
    for (int c = 0; c < kHeadC; ++c) gd[c] = 0.0f;
    const int x = (int)(p % W), y = (int)((p / W) % H);
#pragma unroll
    for (int j4 = 0; j4 < kOut; j4 += 4) {
      float4 t4 = make_float4(0.f, 0.f, 0.f, 0.f), o4, g4;
      if (tgt) {
        const float* t = tgt + p * kOut + j4;
        t4 = WIDE ? *reinterpret_cast<const float4*>(t) : make_float4(t[0], t[1], t[2], t[3]);
      }
#pragma unroll
      for (int jj = 0; jj < 4; ++jj) {
        const int j = j4 + jj;
        const float4* w4 = reinterpret_cast<const float4*>(sw + j * kHeadC);
        float s = sb[j];
#pragma unroll
        for (int c4 = 0; c4 < kHeadC / 4; ++c4) {
          const float4 w = w4[c4];
          s = fmaf(w.x, f[4 * c4], s);
          s = fmaf(w.y, f[4 * c4 + 1], s);
          s = fmaf(w.z, f[4 * c4 + 2], s);
          s = fmaf(w.w, f[4 * c4 + 3], s);
        }
        (&o4.x)[jj] = s;
        if (tgt) {
          const float e = out_valid(j, x, y, nx, ny, nz) ? s - (&t4.x)[jj] : 0.0f;
          const float g = 2.0f * lw.w[j] * e * inv_count;
          se += lw.w[j] * e * e;
          (&g4.x)[jj] = g;
#pragma unroll
          for (int c4 = 0; c4 < kHeadC / 4; ++c4) {
            const float4 w = w4[c4];
            gd[4 * c4] = fmaf(g, w.x, gd[4 * c4]);
            gd[4 * c4 + 1] = fmaf(g, w.y, gd[4 * c4 + 1]);
            gd[4 * c4 + 2] = fmaf(g, w.z, gd[4 * c4 + 2]);
            gd[4 * c4 + 3] = fmaf(g, w.w, gd[4 * c4 + 3]);
          }
        }
      }
      if (out) {
        float* o = out + p * kOut + j4;
        if (WIDE) *reinterpret_cast<float4*>(o) = o4;
        else o[0] = o4.x, o[1] = o4.y, o[2] = o4.z, o[3] = o4.w;
      }
      if (tgt) *reinterpret_cast<float4*>(dout + p * kOut + j4) = g4;
    }
    if (tgt) {
      __align__(16) bf16 gb[kHeadC];
#pragma unroll
      for (int c = 0; c < kHeadC; ++c) gb[c] = __float2bfloat16_rn(f[c] > 0.0f ? gd[c] : 0.0f);
#pragma unroll
      for (int c8 = 0; c8 < kHeadC / 8; ++c8)
        *reinterpret_cast<uint4*>(gd1 + p * kHeadC + c8 * 8) = reinterpret_cast<const uint4*>(gb)[c8];
    }
  }
  if (!tgt) return;
  for (int o = 16; o > 0; o >>= 1) se += __shfl_down_sync(0xffffffffu, se, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = se;
  __syncthreads();
  if (threadIdx.x == 0) part[blockIdx.x] = ((red[0] + red[1]) + red[2]) + red[3];
}

// per-block partial sums of the head's gradient, out[o][c] = sum_p dout[p][o] d1[p][c], then
// the bias gradient out[kOut kHeadC + o] = sum_p dout[p][o], all in FP32.  A block stages
// kHwChunk pixels in shared memory; a thread owns a 4 x 4 tile of (o, c) over every fourth
// pixel (two 16-byte reads for 16 multiply-adds; one output per thread took 1223 us on 8
// samples of 561 x 321), and the four slices are added in turn at the end.
constexpr int kHeadGrad = kOut * kHeadC + kOut;
constexpr int kHwChunk = 64, kHwTiles = (kOut / 4) * (kHeadC / 4), kHwThreads = 4 * kHwTiles;
__global__ void __launch_bounds__(kHwThreads) k_head_wgrad(const float* dout, const bf16* d1, long npix, int nblk,
                                                           float* part) {
  __shared__ __align__(16) float sd[kHwChunk * kOut];
  __shared__ __align__(16) float sf[kHwChunk * kHeadC];
  const int t = threadIdx.x, tile = t % kHwTiles, slice = t / kHwTiles;
  const int o0 = tile % (kOut / 4) * 4, c0 = tile / (kOut / 4) * 4;
  const long per = (npix + nblk - 1) / nblk;
  const long p0 = blockIdx.x * per, p1 = p0 + per < npix ? p0 + per : npix;
  float acc[4][4] = {}, bs[4] = {};
  for (long p = p0; p < p1; p += kHwChunk) {
    const int m = (int)(p1 - p < kHwChunk ? p1 - p : kHwChunk);
    __syncthreads();
    for (int i = t; i < kHwChunk * kOut / 4; i += kHwThreads)
      reinterpret_cast<float4*>(sd)[i] = i < m * (kOut / 4) ? reinterpret_cast<const float4*>(dout + p * kOut)[i]
                                                            : make_float4(0.f, 0.f, 0.f, 0.f);
    for (int i = t; i < kHwChunk * kHeadC / 8; i += kHwThreads) {
      uint4 v = make_uint4(0u, 0u, 0u, 0u);
      if (i < m * (kHeadC / 8)) v = reinterpret_cast<const uint4*>(d1 + p * kHeadC)[i];
      const bf16* e = reinterpret_cast<const bf16*>(&v);
#pragma unroll
      for (int k = 0; k < 8; ++k) sf[i * 8 + k] = __bfloat162float(e[k]);
    }
    __syncthreads();
#pragma unroll 4
    for (int q = slice; q < kHwChunk; q += 4) {
      const float4 d = *reinterpret_cast<const float4*>(sd + q * kOut + o0);
      const float4 f = *reinterpret_cast<const float4*>(sf + q * kHeadC + c0);
      const float dv[4] = {d.x, d.y, d.z, d.w}, fv[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        bs[i] += dv[i];
#pragma unroll
        for (int k = 0; k < 4; ++k) acc[i][k] = fmaf(dv[i], fv[k], acc[i][k]);
      }
    }
  }
  float* dst = part + (long)blockIdx.x * kHeadGrad;
  __shared__ float red[4][kHeadGrad];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
#pragma unroll
    for (int k = 0; k < 4; ++k) red[slice][(o0 + i) * kHeadC + c0 + k] = acc[i][k];
    if (c0 == 0) red[slice][kOut * kHeadC + o0 + i] = bs[i];
  }
  __syncthreads();
  for (int i = t; i < kHeadGrad; i += kHwThreads) dst[i] = ((red[0][i] + red[1][i]) + red[2][i]) + red[3][i];
}

__global__ void k_adam(float* w, const float* g, float* m, float* v, bf16* wb, long n, float lr, float c1,
                       float c2) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = 0.9f * m[i] + 0.1f * gi;
  const float vi = 0.999f * v[i] + 0.001f * gi * gi;
  m[i] = mi;
  v[i] = vi;
  const float wi = w[i] - lr * (mi / c1) / (sqrtf(vi / c2) + 1e-8f);
  w[i] = wi;
  wb[i] = __float2bfloat16_rn(wi);
}

__global__ void k_to_bf16(const float* w, bf16* wb, long n) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) wb[i] = __float2bfloat16_rn(w[i]);
}

// W^T[t][ci][co] = bf16(W[t][co][ci]) of one 3x3 layer: the dgrad operand
__global__ void k_transpose_w(const float* w, bf16* wt, int cin, int cout) {
  const long i = (long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= 9L * cin * cout) return;
  const int co = (int)(i % cout);
  const long r = i / cout;
  const int ci = (int)(r % cin), t = (int)(r / cin);
  wt[i] = __float2bfloat16_rn(w[((long)t * cout + co) * cin + ci]);
}

// ---------------------------------------------------------------------------
// the context's fields <-> network tensors
// ---------------------------------------------------------------------------
struct FieldPtrs {
  const double *Hi, *Hb, *dx, *dy, *A, *beta;
  const int *sheet, *shelf;
};

__global__ void k_features(Dims d, FieldPtrs f, bf16* feat, int Hp, int Wp) {
  const int y = blockIdx.x * blockDim.x + threadIdx.x;  // j
  const int x = blockIdx.y * blockDim.y + threadIdx.y;  // i
  if (y >= Hp || x >= Wp) return;
  __align__(16) bf16 o[kInC];
#pragma unroll
  for (int c = 0; c < kInC; ++c) o[c] = __float2bfloat16_rn(0.0f);
  if (y < d.ny && x < d.nx) {
    const long long q = d.at(y, x);
    o[0] = __float2bfloat16_rn((float)(f.Hi[q] / 1000.0));
    o[1] = __float2bfloat16_rn((float)(f.Hb[q] / 1000.0));
    o[2] = __float2bfloat16_rn((float)(f.dx[q] * 100.0));
    o[3] = __float2bfloat16_rn((float)(f.dy[q] * 100.0));
    o[4] = __float2bfloat16_rn((float)(log10(fmax(f.A[q], 1e-30)) + 17.0));
    o[5] = __float2bfloat16_rn((float)(log10(fmax(f.beta[q], 1e-30)) - 4.0));
    o[6] = __float2bfloat16_rn((float)f.sheet[q]);
    o[7] = __float2bfloat16_rn((float)f.shelf[q]);
  }
  uint4* dst = reinterpret_cast<uint4*>(feat + ((long)y * Wp + x) * kInC);
  dst[0] = reinterpret_cast<const uint4*>(o)[0];
  dst[1] = reinterpret_cast<const uint4*>(o)[1];
}

struct StatePtrs {
  double *ucx, *vcy, *tbx, *tby, *visc;
};
constexpr double kTauScale = 1000.0;  // Pa; outputs 2, 3 are asinh(taub / kTauScale)
constexpr double kViscShift = 8.0;    // outputs 4.. are log10(visc_eff) - kViscShift

__global__ void k_targets(Dims d, StatePtrs s, float* tgt, int Hp, int Wp) {
  const int y = blockIdx.x * blockDim.x + threadIdx.x;
  const int x = blockIdx.y * blockDim.y + threadIdx.y;
  if (y >= Hp || x >= Wp) return;
  float t[kOut];
#pragma unroll
  for (int o = 0; o < kOut; ++o) t[o] = 0.0f;
  if (y < d.ny && x < d.nx - 1) {
    t[0] = (float)asinh(s.ucx[d.at(y, x)] / kVelScale);
    t[2] = (float)asinh(s.tbx[d.at(y, x)] / kTauScale);
  }
  if (y < d.ny - 1 && x < d.nx) {
    t[1] = (float)asinh(s.vcy[d.at(y, x)] / kVelScale);
    t[3] = (float)asinh(s.tby[d.at(y, x)] / kTauScale);
  }
  if (y < d.ny && x < d.nx)
    for (int k = 0; k < d.nz && k < kMaxNzOut; ++k)
      t[4 + k] = (float)(log10(fmax(s.visc[k * d.plane + d.at(y, x)], 1e-30)) - kViscShift);
#pragma unroll
  for (int o = 0; o < kOut; ++o) tgt[((long)y * Wp + x) * kOut + o] = t[o];
}

// an output clamped to [-lim, lim]; a non-finite one becomes 0
__device__ __forceinline__ double clamp_out(float v, double lim) {
  const double x = (double)v;
  return x == x ? fmax(-lim, fmin(lim, x)) : 0.0;
}

// the predicted state into the context's fields, within physical bounds (velocities
// within the solver's DIVA_vel_max, |taub| <= 1e7 Pa, viscosity in [1e3, 1e18]) so that
// a poorly trained network cannot hand the solve an overflow; velocities_only: u, v
__global__ void k_apply(Dims d, const float* pred, StatePtrs s, int Wp, int velocities_only, double vmax) {
  const int y = blockIdx.x * blockDim.x + threadIdx.x;
  const int x = blockIdx.y * blockDim.y + threadIdx.y;
  if (y >= d.ny || x >= d.nx) return;
  const float* q = pred + ((long)y * Wp + x) * kOut;
  const double ulim = asinh(vmax / kVelScale), tlim = asinh(1e7 / kTauScale);
  if (x < d.nx - 1) s.ucx[d.at(y, x)] = kVelScale * sinh(clamp_out(q[0], ulim));
  if (y < d.ny - 1) s.vcy[d.at(y, x)] = kVelScale * sinh(clamp_out(q[1], ulim));
  if (velocities_only) return;
  if (x < d.nx - 1) s.tbx[d.at(y, x)] = kTauScale * sinh(clamp_out(q[2], tlim));
  if (y < d.ny - 1) s.tby[d.at(y, x)] = kTauScale * sinh(clamp_out(q[3], tlim));
  for (int k = 0; k < d.nz; ++k) {
    const double l = fmax(3.0 - kViscShift, fmin(18.0 - kViscShift, clamp_out(q[4 + k], 1e30)));
    s.visc[k * d.plane + d.at(y, x)] = pow(10.0, l + kViscShift);
  }
}

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// CTAs of a persistent kernel that fit on the GPU: by its shared memory (228 KB per SM, 1 KB of
// it per CTA) and by tensor memory (512 columns per SM)
int resident_ctas(int smem, int ncols) {
  const int by_smem = 228 * 1024 / (smem + 1024 + 2048), by_tmem = 512 / ncols;
  const int k = std::min(std::min(by_smem, by_tmem), 8);
  return kSMs * std::max(k, 1);
}

template <int KC, int NO, bool DG>
int launch_conv(ConvArgs a, cudaStream_t st) {
  constexpr int NB = conv_blocks(KC, NO);
  a.t = conv_tile(a.n, a.H, a.W, KC, NO);
  const int smem = conv_smem(KC, NO, a.t.npx);
  const int grid = std::min(a.t.ntile, resident_ctas(smem, tmem_cols<NB * NO>()));
  k_conv3x3<KC, NO, DG><<<grid, kConvThreads, smem, st>>>(a);
  return DIVA_OK;
}

template <int CI, int CO>
int launch_wgrad(WgradArgs a, long part_floats, int* nsplit, cudaStream_t st) {
  constexpr int NCOL = tmem_cols<CI>();
  a.t = wgrad_tile(a.n, a.H, a.W, CI, CO);
  int smem = 2 * a.t.buf + 128;
  // no more CTAs on an SM than its tensor memory serves
  smem = std::max(smem, 227 * 1024 / (512 / NCOL + 1));
  if (wgrad_part_floats(a.t, CI, CO) > part_floats) return DIVA_BAD_INPUT;
  *nsplit = a.t.slices;
  k_conv3x3_wgrad<CI, CO><<<dim3(a.t.slices, 3 * wgrad_sets<CO>()), kConvThreads, smem, st>>>(a);
  return DIVA_OK;
}

// the channel counts there are kernels for: (read, written) of a forward layer and of an input
// gradient, (cin, cout) of a weight gradient
#define FOR_FWD(X) X(16, 32) X(32, 32) X(32, 64) X(64, 64) X(64, 128) X(128, 64) X(64, 32)
#define FOR_DGRAD(X) X(32, 32) X(32, 64) X(64, 128) X(128, 64) X(64, 64) X(64, 32)
#define FOR_WGRAD(X) X(16, 32) X(32, 32) X(32, 64) X(64, 64) X(64, 128) X(128, 64) X(64, 32)

int conv_fwd(int cin, int cout, const ConvArgs& a, cudaStream_t st) {
#define FWD(KC, NO) \
  if (cin == KC && cout == NO) return launch_conv<KC, NO, false>(a, st);
  FOR_FWD(FWD)
#undef FWD
  return DIVA_UNSUPPORTED;
}
int conv_dgrad(int cin, int cout, const ConvArgs& a, cudaStream_t st) {
#define DGR(KC, NO) \
  if (cout == KC && cin == NO) return launch_conv<KC, NO, true>(a, st);
  FOR_DGRAD(DGR)
#undef DGR
  return DIVA_UNSUPPORTED;
}
int conv_wgrad(int cin, int cout, const WgradArgs& a, long part_floats, int* nsplit, cudaStream_t st) {
#define WGR(CI, CO) \
  if (cin == CI && cout == CO) return launch_wgrad<CI, CO>(a, part_floats, nsplit, st);
  FOR_WGRAD(WGR)
#undef WGR
  return DIVA_UNSUPPORTED;
}
// The current device's limit of every kernel's dynamic shared memory, the same for every network
// and never lowered: the limit belongs to the kernel, so a launch's own size set as the limit
// would refuse a larger one that another thread's network is about to make.
bool allow_shared_memory() {
  bool ok = true;
  auto allow = [&](const void* kernel) {
    ok = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kDynSmemMax) == cudaSuccess && ok;
  };
#define ALLOW(KC, NO) allow((const void*)k_conv3x3<KC, NO, false>);
  FOR_FWD(ALLOW)
#undef ALLOW
#define ALLOW(KC, NO) allow((const void*)k_conv3x3<KC, NO, true>);
  FOR_DGRAD(ALLOW)
#undef ALLOW
#define ALLOW(CI, CO) allow((const void*)k_conv3x3_wgrad<CI, CO>);
  FOR_WGRAD(ALLOW)
#undef ALLOW
  return ok;
}

// tensors of the network (index, level, channels)
enum T { T_IN, T_A1, T_E1, T_P1, T_A2, T_E2, T_P2, T_B1, T_B2, T_U2, T_C2, T_D2, T_U1, T_C1, T_D1, T_N };
constexpr int kTLevel[T_N] = {0, 0, 0, 1, 1, 1, 2, 2, 2, 1, 1, 1, 0, 0, 0};
constexpr int kTChan[T_N] = {16, 32, 32, 32, 64, 64, 64, 128, 64, 128, 64, 32, 64, 32, 32};

struct Layer {
  int cin, cout, in, out;
  long woff, boff;
};
constexpr int kNL = 10;
constexpr int kLayerDef[kNL][4] = {{16, 32, T_IN, T_A1}, {32, 32, T_A1, T_E1}, {32, 64, T_P1, T_A2},
                                   {64, 64, T_A2, T_E2}, {64, 128, T_P2, T_B1}, {128, 64, T_B1, T_B2},
                                   {128, 64, T_U2, T_C2}, {64, 32, T_C2, T_D2}, {64, 32, T_U1, T_C1},
                                   {32, 32, T_C1, T_D1}};

uint64_t splitmix(uint64_t& s) {
  uint64_t z = (s += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}
double unit(uint64_t& s) { return ((splitmix(s) >> 11) + 0.5) * (1.0 / 9007199254740992.0); }

}  // namespace cnn
}  // namespace diva

using namespace diva;
using namespace diva::cnn;

struct diva_cnn {
  int ny = 0, nx = 0, nz = 0, Hp = 0, Wp = 0, batch = 0, capacity = 0, nsamples = 0;
  Layer L[kNL];
  long head_w = 0, head_b = 0, nw = 0;
  cudaStream_t stream = nullptr;
  void* arena = nullptr;
  float *w = nullptr, *g = nullptr, *m = nullptr, *v = nullptr;
  bf16* wb = nullptr;
  bf16* wbt = nullptr;   // per-layer transposed BF16 weights (dgrad)
  bf16* act[T_N] = {};
  bf16* grad[T_N] = {};
  float *out = nullptr, *tgt = nullptr, *dout = nullptr, *part = nullptr, *loss = nullptr, *loss_hist = nullptr;
  long part_floats = 0;
  bf16* ds_feat = nullptr;
  float* ds_tgt = nullptr;
  int* err = nullptr;
  long adam_t = 0;
  LossWeights lw{};

  // valid output entries of n samples (the loss is their mean squared error)
  long valid(int n) const {
    return (long)n * (2L * ny * (nx - 1) + 2L * (ny - 1) * nx + (long)nz * ny * nx);
  }
  int lvH(int l) const { return Hp >> l; }
  int lvW(int l) const { return Wp >> l; }
  long tsize(int t) const { return (long)lvH(kTLevel[t]) * lvW(kTLevel[t]) * kTChan[t]; }
};

namespace {

#define CK(x)                                              \
  do {                                                     \
    if ((x) != cudaSuccess) return DIVA_CUDA_ERROR;        \
  } while (0)
#define RET(x)                                             \
  do {                                                     \
    const int _st = (x);                                   \
    if (_st != DIVA_OK) return _st;                        \
  } while (0)

inline unsigned nblk(long n, int b) { return (unsigned)((n + b - 1) / b); }
constexpr int kHeadBlocks = 592;   // four per SM

// the input of layer l: a stored tensor, or the concatenation [lo (upsampled), skip]
Input layer_input(const diva_cnn_t* N, int l, const bf16* in) {
  const int t = N->L[l].in;
  if (t == T_U1) return Input{N->act[T_E1], N->act[T_D2], kTChan[T_D2]};
  if (t == T_U2) return Input{N->act[T_E2], N->act[T_B2], kTChan[T_B2]};
  return Input{t == T_IN ? in : N->act[t], nullptr, 0};
}

// of a caller's buffer (a misaligned access is a fault on the GPU)
bool aligned(const void* p, size_t bytes) { return reinterpret_cast<uintptr_t>(p) % bytes == 0; }

int forward(diva_cnn_t* N, const bf16* in, float* out, int n, cudaStream_t st) {
  auto conv = [&](int l) {
    const Layer& ly = N->L[l];
    const int lv = kTLevel[ly.out];
    ConvArgs a{layer_input(N, l, in), N->wb + ly.woff, N->w + ly.boff, nullptr, N->act[ly.out], n, N->lvH(lv),
               N->lvW(lv), N->err, {}};
    return conv_fwd(ly.cin, ly.cout, a, st);
  };
  auto pool = [&](int src, int dst) {
    const int lv = kTLevel[src];
    const long cnt = (long)n * (N->lvH(lv) / 2) * (N->lvW(lv) / 2) * (kTChan[src] / 8);
    k_pool<<<nblk(cnt, 256), 256, 0, st>>>(N->act[src], N->act[dst], n, N->lvH(lv), N->lvW(lv), kTChan[src]);
  };
  RET(conv(0));
  RET(conv(1));
  pool(T_E1, T_P1);
  RET(conv(2));
  RET(conv(3));
  pool(T_E2, T_P2);
  RET(conv(4));
  RET(conv(5));
  RET(conv(6));
  RET(conv(7));
  RET(conv(8));
  RET(conv(9));
  if (out) {
    const long npix = (long)n * N->Hp * N->Wp;
    const auto head = aligned(out, 16) ? k_head<true> : k_head<false>;
    head<<<nblk(npix, 128), 128, 0, st>>>(N->act[T_D1], N->w + N->head_w, N->w + N->head_b, out, nullptr,
                                            nullptr, nullptr, nullptr, n, N->Hp, N->Wp, N->ny, N->nx, N->nz, 0.0f,
                                            N->lw);
  }
  CK(cudaGetLastError());
  return DIVA_OK;
}

// gradient of the batch loss into N->g, the batch's squared-error sum into *loss_dst
int backward(diva_cnn_t* N, const bf16* in, const float* tgt, int n, cudaStream_t st, float* loss_dst) {
  const long npix0 = (long)n * N->Hp * N->Wp;
  const unsigned hb = nblk(npix0, 128);
  if ((long)hb > N->part_floats - 128 || (long)kHeadBlocks * kHeadGrad > N->part_floats - 128) return DIVA_BAD_INPUT;
  auto sum_rows = [&](int rows, long cols, float* dst) {
    k_sum_rows<<<nblk(cols, 32), dim3(32, 8), 0, st>>>(N->part, rows, (int)cols, dst);
  };
  const auto head = aligned(tgt, 16) ? k_head<true> : k_head<false>;
  head<<<hb, 128, 0, st>>>(N->act[T_D1], N->w + N->head_w, N->w + N->head_b, nullptr, tgt, N->dout,
                             N->grad[T_D1], N->part, n, N->Hp, N->Wp, N->ny, N->nx, N->nz,
                             1.0f / (float)N->valid(n), N->lw);
  k_sum_all<<<1, 1024, 0, st>>>(N->part, (int)hb, loss_dst);
  k_head_wgrad<<<kHeadBlocks, kHwThreads, 0, st>>>(N->dout, N->act[T_D1], npix0, kHeadBlocks, N->part);
  sum_rows(kHeadBlocks, kHeadGrad, N->g + N->head_w);

  auto layer_bwd = [&](int l, bool dgrad) -> int {
    const Layer& ly = N->L[l];
    const int lv = kTLevel[ly.out];
    const int H = N->lvH(lv), W = N->lvW(lv);
    int ns = 0;
    WgradArgs wa{layer_input(N, l, in), N->grad[ly.out], N->part, n, H, W, N->err, {}};
    RET(conv_wgrad(ly.cin, ly.cout, wa, N->part_floats - 128, &ns, st));
    sum_rows(ns, 9L * ly.cout * ly.cin + ly.cout, N->g + ly.woff);   // the bias follows the weights
    if (dgrad) {
      // a tensor that one convolution writes and one reads has its whole gradient here: masked;
      // pooled and concatenated ones pass through the adjoints below
      const bool whole = ly.in == T_A1 || ly.in == T_A2 || ly.in == T_B1 || ly.in == T_C1 || ly.in == T_C2;
      ConvArgs a{Input{N->grad[ly.out], nullptr, 0}, N->wbt + ly.woff, nullptr, whole ? N->act[ly.in] : nullptr,
                 N->grad[ly.in], n, H, W, N->err, {}};
      RET(conv_dgrad(ly.cin, ly.cout, a, st));
    }
    return DIVA_OK;
  };
  auto upcat_bwd = [&](int dst, int lo, int skip) {
    const int lv = kTLevel[dst];
    const int H = N->lvH(lv), W = N->lvW(lv);
    const long cnt = (long)n * (H / 2) * (W / 2) * (kTChan[lo] / 8) + (long)n * H * W * (kTChan[skip] / 8);
    k_upcat_bwd<<<nblk(cnt, 256), 256, 0, st>>>(N->grad[dst], N->act[lo], N->grad[lo], N->grad[skip], n, H, W,
                                                kTChan[lo], kTChan[skip]);
  };
  auto pool_bwd = [&](int lo, int hi) {
    const int lv = kTLevel[hi];
    const long cnt = (long)n * N->lvH(lv) * N->lvW(lv) * (kTChan[hi] / 8);
    k_pool_bwd_add<<<nblk(cnt, 256), 256, 0, st>>>(N->grad[lo], N->act[hi], N->grad[hi], n, N->lvH(lv), N->lvW(lv),
                                                   kTChan[hi]);
  };
  RET(layer_bwd(9, true));   // d1b -> g_c1
  RET(layer_bwd(8, true));   // d1a -> g_u1
  upcat_bwd(T_U1, T_D2, T_E1);
  RET(layer_bwd(7, true));   // d2b -> g_c2
  RET(layer_bwd(6, true));   // d2a -> g_u2
  upcat_bwd(T_U2, T_B2, T_E2);
  RET(layer_bwd(5, true));   // bb -> g_b1
  RET(layer_bwd(4, true));   // ba -> g_p2
  pool_bwd(T_P2, T_E2);
  RET(layer_bwd(3, true));   // e2b -> g_a2
  RET(layer_bwd(2, true));   // e2a -> g_p1
  pool_bwd(T_P1, T_E1);
  RET(layer_bwd(1, true));   // e1b -> g_a1
  RET(layer_bwd(0, false));  // e1a
  CK(cudaGetLastError());
  return DIVA_OK;
}

void transpose_weights(diva_cnn_t* N, cudaStream_t st) {
  for (int l = 0; l < kNL; ++l) {
    const Layer& ly = N->L[l];
    k_transpose_w<<<nblk(9L * ly.cin * ly.cout, 256), 256, 0, st>>>(N->w + ly.woff, N->wbt + ly.woff, ly.cin,
                                                                    ly.cout);
  }
}

int adam(diva_cnn_t* N, float lr, cudaStream_t st) {
  N->adam_t += 1;
  const float c1 = 1.0f - powf(0.9f, (float)N->adam_t), c2 = 1.0f - powf(0.999f, (float)N->adam_t);
  k_adam<<<nblk(N->nw, 256), 256, 0, st>>>(N->w, N->g, N->m, N->v, N->wb, N->nw, lr, c1, c2);
  transpose_weights(N, st);
  CK(cudaGetLastError());
  return DIVA_OK;
}

int check_err(diva_cnn_t* N) {
  int e = 0;
  CK(cudaMemcpy(&e, N->err, sizeof(int), cudaMemcpyDeviceToHost));
  if (e) {
    CK(cudaMemset(N->err, 0, sizeof(int)));
    return DIVA_TIMEOUT;
  }
  return DIVA_OK;
}

FieldPtrs field_ptrs(const Ctx* c) {
  return FieldPtrs{c->D(DIVA_F_HI_A),     c->D(DIVA_F_HB_A),       c->D(DIVA_F_DHS_DX_A),
                   c->D(DIVA_F_DHS_DY_A), c->D(DIVA_F_A_FLOW_VAV_A), c->D(DIVA_F_BETA_SQ_A),
                   static_cast<const int*>(c->f[DIVA_F_MASK_SHEET_A]),
                   static_cast<const int*>(c->f[DIVA_F_MASK_SHELF_A])};
}

StatePtrs state_ptrs(Ctx* c) {
  return StatePtrs{c->D(DIVA_F_U_VAV_CX), c->D(DIVA_F_V_VAV_CY), c->D(DIVA_F_TAUB_CX), c->D(DIVA_F_TAUB_CY),
                   c->D(DIVA_F_VISC_EFF_3D_A)};
}

dim3 img_grid(int Hp, int Wp) { return dim3((Hp + kBX - 1) / kBX, (Wp + kBY - 1) / kBY); }

}  // namespace

extern "C" {

int32_t diva_cnn_create(diva_cnn_t** out, int32_t ny, int32_t nx, int32_t nz, int32_t batch, int32_t capacity,
                        uint64_t seed) {
  if (!out || ny < 2 || nx < 2 || nz < 2 || batch < 1 || capacity < 0) return DIVA_BAD_INPUT;
  *out = nullptr;
  if (nz > kMaxNzOut) return DIVA_UNSUPPORTED;
  diva_cnn_t* N = new (std::nothrow) diva_cnn_t();
  if (!N) return DIVA_CUDA_ERROR;
  N->ny = ny;
  N->nx = nx;
  N->nz = nz;
  N->Hp = (ny + 3) / 4 * 4;
  N->Wp = (nx + 3) / 4 * 4;
  N->batch = batch;
  N->capacity = capacity;
  for (int o = 0; o < kOut; ++o) N->lw.w[o] = 1.0f;
  long off = 0;
  for (int l = 0; l < kNL; ++l) {
    Layer& ly = N->L[l];
    ly.cin = kLayerDef[l][0];
    ly.cout = kLayerDef[l][1];
    ly.in = kLayerDef[l][2];
    ly.out = kLayerDef[l][3];
    ly.woff = off;
    off += 9L * ly.cin * ly.cout;
    ly.boff = off;
    off += ly.cout;
  }
  N->head_w = off;
  off += (long)kOut * kHeadC;
  N->head_b = off;
  off += kOut;
  N->nw = off;

  // weight-gradient sums of the slices of any layer and minibatch size; head sums
  long part = 0;
  for (int b = 1; b <= batch; ++b)
    for (const Layer& ly : N->L) {
      const int lv = kTLevel[ly.out];
      const WgradTile t = wgrad_tile(b, N->lvH(lv), N->lvW(lv), ly.cin, ly.cout);
      part = std::max(part, wgrad_part_floats(t, ly.cin, ly.cout));
    }
  const long hb = (long)nblk((long)batch * N->Hp * N->Wp, 128);
  if (hb > part) part = hb;
  if ((long)kHeadBlocks * kHeadGrad > part) part = (long)kHeadBlocks * kHeadGrad;
  N->part_floats = part + 128;

  const long img = (long)N->Hp * N->Wp;
  size_t bytes = 0;
  auto carve = [&](size_t b) {
    const size_t o = bytes;
    bytes += (b + 255) / 256 * 256;
    return o;
  };
  const size_t o_w = carve(N->nw * 4), o_g = carve(N->nw * 4), o_m = carve(N->nw * 4), o_v = carve(N->nw * 4);
  const size_t o_wb = carve(N->nw * 2), o_wbt = carve(N->nw * 2);
  size_t o_act[T_N], o_grad[T_N];
  for (int t = 0; t < T_N; ++t) {
    // the concatenated tensors are never stored: the convolutions read their two parts
    o_act[t] = (t == T_U1 || t == T_U2) ? 0 : carve((size_t)batch * N->tsize(t) * 2);
    o_grad[t] = t == T_IN ? 0 : carve((size_t)batch * N->tsize(t) * 2);
  }
  const size_t o_out = carve((size_t)batch * img * kOut * 4), o_tgt = carve((size_t)batch * img * kOut * 4);
  const size_t o_dout = carve((size_t)batch * img * kOut * 4);
  const size_t o_part = carve(N->part_floats * 4), o_loss = carve(256), o_err = carve(256);
  const size_t o_lh = carve((size_t)(capacity + 1) * 4);
  const size_t o_dsf = carve((size_t)capacity * img * kInC * 2), o_dst = carve((size_t)capacity * img * kOut * 4);
  if (cudaMalloc(&N->arena, bytes) != cudaSuccess) {
    delete N;
    return DIVA_CUDA_ERROR;
  }
  char* base = static_cast<char*>(N->arena);
  N->w = reinterpret_cast<float*>(base + o_w);
  N->g = reinterpret_cast<float*>(base + o_g);
  N->m = reinterpret_cast<float*>(base + o_m);
  N->v = reinterpret_cast<float*>(base + o_v);
  N->wb = reinterpret_cast<bf16*>(base + o_wb);
  N->wbt = reinterpret_cast<bf16*>(base + o_wbt);
  for (int t = 0; t < T_N; ++t) {
    N->act[t] = (t == T_U1 || t == T_U2) ? nullptr : reinterpret_cast<bf16*>(base + o_act[t]);
    N->grad[t] = t == T_IN ? nullptr : reinterpret_cast<bf16*>(base + o_grad[t]);
  }
  N->out = reinterpret_cast<float*>(base + o_out);
  N->tgt = reinterpret_cast<float*>(base + o_tgt);
  N->dout = reinterpret_cast<float*>(base + o_dout);
  N->part = reinterpret_cast<float*>(base + o_part);
  N->loss = reinterpret_cast<float*>(base + o_loss);
  N->err = reinterpret_cast<int*>(base + o_err);
  N->loss_hist = reinterpret_cast<float*>(base + o_lh);
  N->ds_feat = reinterpret_cast<bf16*>(base + o_dsf);
  N->ds_tgt = reinterpret_cast<float*>(base + o_dst);
  if (cudaStreamCreateWithFlags(&N->stream, cudaStreamNonBlocking) != cudaSuccess || !allow_shared_memory() ||
      cudaMemset(N->arena, 0, bytes) != cudaSuccess) {
    diva_cnn_destroy(N);
    return DIVA_CUDA_ERROR;
  }
  // He-normal weights from the seed, zero biases
  std::vector<float> h(N->nw, 0.0f);
  uint64_t s = seed;
  auto normal = [&]() {
    const double u1 = unit(s), u2 = unit(s);
    return std::sqrt(-2.0 * std::log(u1)) * std::cos(2.0 * kPi * u2);
  };
  for (int l = 0; l < kNL; ++l) {
    const double sd = std::sqrt(2.0 / (9.0 * N->L[l].cin));
    for (long i = 0; i < 9L * N->L[l].cin * N->L[l].cout; ++i) h[N->L[l].woff + i] = (float)(sd * normal());
  }
  for (int i = 0; i < kOut * kHeadC; ++i) h[N->head_w + i] = (float)(std::sqrt(1.0 / kHeadC) * normal());
  const int st = diva_cnn_weights(N, h.data(), N->nw, 1);
  if (st != DIVA_OK) {
    diva_cnn_destroy(N);
    return st;
  }
  *out = N;
  return DIVA_OK;
}

int32_t diva_cnn_destroy(diva_cnn_t* N) {
  if (!N) return DIVA_BAD_INPUT;
  if (N->stream) cudaStreamSynchronize(N->stream);
  if (N->arena) cudaFree(N->arena);
  if (N->stream) cudaStreamDestroy(N->stream);
  delete N;
  return DIVA_OK;
}

int32_t diva_cnn_num_weights(const diva_cnn_t* N, int64_t* n) {
  if (!N || !n) return DIVA_BAD_INPUT;
  *n = N->nw;
  return DIVA_OK;
}

int32_t diva_cnn_padded_shape(const diva_cnn_t* N, int32_t* Hp, int32_t* Wp) {
  if (!N || !Hp || !Wp) return DIVA_BAD_INPUT;
  *Hp = N->Hp;
  *Wp = N->Wp;
  return DIVA_OK;
}

int32_t diva_cnn_num_samples(const diva_cnn_t* N, int32_t* n) {
  if (!N || !n) return DIVA_BAD_INPUT;
  *n = N->nsamples;
  return DIVA_OK;
}

int32_t diva_cnn_weights(diva_cnn_t* N, float* host, int64_t n, int32_t direction) {
  if (!N || !host || n != N->nw || (direction != 0 && direction != 1)) return DIVA_BAD_INPUT;
  CK(cudaStreamSynchronize(N->stream));
  if (direction == 0) {
    CK(cudaMemcpy(host, N->w, n * 4, cudaMemcpyDeviceToHost));
    return DIVA_OK;
  }
  CK(cudaMemcpy(N->w, host, n * 4, cudaMemcpyHostToDevice));
  CK(cudaMemset(N->m, 0, n * 4));
  CK(cudaMemset(N->v, 0, n * 4));
  N->adam_t = 0;
  k_to_bf16<<<nblk(n, 256), 256, 0, N->stream>>>(N->w, N->wb, n);
  transpose_weights(N, N->stream);
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(N->stream));
  return DIVA_OK;
}

int32_t diva_cnn_grads(diva_cnn_t* N, float* host, int64_t n) {
  if (!N || !host || n != N->nw) return DIVA_BAD_INPUT;
  CK(cudaStreamSynchronize(N->stream));
  CK(cudaMemcpy(host, N->g, n * 4, cudaMemcpyDeviceToHost));
  return DIVA_OK;
}

int32_t diva_cnn_set_loss_weights(diva_cnn_t* N, const float* w, int32_t n) {
  if (!N || !w || n != kOut) return DIVA_BAD_INPUT;
  for (int o = 0; o < kOut; ++o)
    if (!(w[o] >= 0.0f) || std::isinf(w[o])) return DIVA_BAD_INPUT;
  CK(cudaStreamSynchronize(N->stream));
  for (int o = 0; o < kOut; ++o) N->lw.w[o] = w[o];
  return DIVA_OK;
}

int32_t diva_cnn_add_sample(diva_cnn_t* N, diva_ctx_t* ctx) {
  if (!N || !ctx) return DIVA_BAD_INPUT;
  Ctx* c = &ctx->c;
  if (c->d.ny != N->ny || c->d.nx != N->nx || c->d.nz != N->nz || N->nsamples >= N->capacity)
    return DIVA_BAD_INPUT;
  const long img = (long)N->Hp * N->Wp;
  const int k = N->nsamples;
  k_features<<<img_grid(N->Hp, N->Wp), block2d(), 0, c->stream>>>(c->d, field_ptrs(c), N->ds_feat + k * img * kInC,
                                                                   N->Hp, N->Wp);
  k_targets<<<img_grid(N->Hp, N->Wp), block2d(), 0, c->stream>>>(c->d, state_ptrs(c), N->ds_tgt + k * img * kOut,
                                                                  N->Hp, N->Wp);
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(c->stream));
  N->nsamples += 1;
  return DIVA_OK;
}

int32_t diva_cnn_predict(diva_cnn_t* N, diva_ctx_t* ctx, int32_t complete_sweeps) {
  if (!N || !ctx || complete_sweeps < 0 || complete_sweeps > 10000) return DIVA_BAD_INPUT;
  Ctx* c = &ctx->c;
  if (c->d.ny != N->ny || c->d.nx != N->nx || c->d.nz != N->nz) return DIVA_BAD_INPUT;
  CK(cudaStreamSynchronize(N->stream));
  k_features<<<img_grid(N->Hp, N->Wp), block2d(), 0, c->stream>>>(c->d, field_ptrs(c), N->act[T_IN], N->Hp,
                                                                   N->Wp);
  RET(forward(N, N->act[T_IN], N->out, 1, c->stream));
  k_apply<<<img_grid(N->ny, N->nx), block2d(), 0, c->stream>>>(c->d, N->out, state_ptrs(c), N->Wp,
                                                                complete_sweeps > 0, c->c.DIVA_vel_max);
  // the context's launch count includes the network's kernels run on its stream: features,
  // 10 convolutions, 2 pools, the head and the state write
  c->launches += 15;
  CK(cudaGetLastError());
  CK(cudaStreamSynchronize(c->stream));
  RET(check_err(N));
  return complete_sweeps > 0 ? diva_complete_state(ctx, complete_sweeps) : DIVA_OK;
}

int32_t diva_cnn_forward(diva_cnn_t* N, const void* feat, float* out, int32_t n) {
  if (!N || !feat || !out || n < 1 || n > N->batch) return DIVA_BAD_INPUT;
  if (!aligned(feat, 16) || !aligned(out, sizeof(float))) return DIVA_BAD_INPUT;
  RET(forward(N, static_cast<const bf16*>(feat), out, n, N->stream));
  CK(cudaStreamSynchronize(N->stream));
  return check_err(N);
}

int32_t diva_cnn_train_step(diva_cnn_t* N, const void* feat, const float* tgt, int32_t n, float lr, float* loss) {
  if (!N || !feat || !tgt || n < 1 || n > N->batch || !(lr >= 0.0f)) return DIVA_BAD_INPUT;
  if (!aligned(feat, 16) || !aligned(tgt, sizeof(float))) return DIVA_BAD_INPUT;
  const bf16* in = static_cast<const bf16*>(feat);
  RET(forward(N, in, nullptr, n, N->stream));
  RET(backward(N, in, tgt, n, N->stream, N->loss));
  float l = 0.0f;
  CK(cudaMemcpyAsync(&l, N->loss, 4, cudaMemcpyDeviceToHost, N->stream));
  RET(adam(N, lr, N->stream));
  CK(cudaStreamSynchronize(N->stream));
  if (loss) *loss = l / (float)N->valid(n);
  return check_err(N);
}

int32_t diva_cnn_train(diva_cnn_t* N, int32_t epochs, float lr, uint64_t seed, float* loss) {
  if (!N || epochs < 0 || !(lr >= 0.0f) || N->nsamples < 1) return DIVA_BAD_INPUT;
  const long img = (long)N->Hp * N->Wp;
  std::vector<int> order(N->nsamples);
  for (int i = 0; i < N->nsamples; ++i) order[i] = i;
  uint64_t s = seed;
  std::vector<float> batch_loss;
  double last = 0.0;
  for (int e = 0; e < epochs; ++e) {
    for (int i = N->nsamples - 1; i > 0; --i) {
      const int j = (int)(splitmix(s) % (uint64_t)(i + 1));
      const int t = order[i];
      order[i] = order[j];
      order[j] = t;
    }
    const int nb = (N->nsamples + N->batch - 1) / N->batch;
    batch_loss.assign(nb, 0.0f);
    for (int b = 0; b < nb; ++b) {
      const int n = std::min(N->batch, N->nsamples - b * N->batch);
      for (int k = 0; k < n; ++k) {
        const int smp = order[b * N->batch + k];
        CK(cudaMemcpyAsync(N->act[T_IN] + k * img * kInC, N->ds_feat + smp * img * kInC, img * kInC * 2,
                           cudaMemcpyDeviceToDevice, N->stream));
        CK(cudaMemcpyAsync(N->tgt + k * img * kOut, N->ds_tgt + smp * img * kOut, img * kOut * 4,
                           cudaMemcpyDeviceToDevice, N->stream));
      }
      RET(forward(N, N->act[T_IN], nullptr, n, N->stream));
      RET(backward(N, N->act[T_IN], N->tgt, n, N->stream, N->loss_hist + b));
      RET(adam(N, lr, N->stream));
    }
    CK(cudaMemcpyAsync(batch_loss.data(), N->loss_hist, nb * 4, cudaMemcpyDeviceToHost, N->stream));
    CK(cudaStreamSynchronize(N->stream));
    RET(check_err(N));
    double sum = 0.0;
    for (int b = 0; b < nb; ++b) sum += batch_loss[b];
    last = sum / (double)N->valid(N->nsamples);
    if (!(last == last) || std::isinf(last)) {   // diverged: the weights are no longer usable
      if (loss) *loss = (float)last;
      return DIVA_NAN_DETECTED;
    }
  }
  if (loss) *loss = (float)last;
  return DIVA_OK;
}

}  // extern "C"
