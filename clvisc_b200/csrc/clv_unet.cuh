// Kernels of the learned surrogate: a U-Net on (N, H, W, C) BF16 activations
// with FP32 accumulation.
//
// conv3x3_tma_kernel and conv3x3_tc_kernel (the default path) are implicit
// GEMMs on the 5th-generation tensor cores (tcgen05.mma, accumulator in tensor
// memory), described at the kernels; conv3x3_kernel is the same GEMM on
// mma.sync m16n8k16 (BF16 in, FP32 accumulate), kept as a selectable variant: rows are output pixels, columns output
// channels, the reduction runs over (tap, input channel) in chunks of 32,
// staged through shared memory with cp.async double buffering (zero fill at
// the image border). Its epilogue adds the bias and applies GELU, writes the
// pre-activation for the backward pass, and can scale by GELU'(gate) (the
// backward of a preceding GELU). The input gradient of a 3x3 convolution is
// the same kernel on the output gradient with the taps flipped and the
// channel roles swapped (weights packed by unet_pack_weights).
//
// wgrad3x3_kernel is the weight gradient, a GEMM over pixels:
// dW[(tap, ci)][co] = sum_p x[p + tap][ci] g[p][co], split over pixel ranges
// into FP32 partials that reduce_partials_kernel adds in a fixed order.
//
// Activations may be channel slices of a wider buffer (the U-Net's
// concatenations): element (p, c) of a slice is ptr[p * stride + offset + c].
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <type_traits>
#include <stdint.h>

#include "clv_launch.cuh"

namespace clv {
namespace unet {

typedef __nv_bfloat16 bf16;

// GELU(z) = z Phi(z) (exact form, with the error function) and its derivative
__device__ __forceinline__ float gelu_f(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_grad(float z) {
  return 0.5f * (1.0f + erff(z * 0.70710678118654752f)) + z * 0.39894228040143268f * expf(-0.5f * z * z);
}

struct ConvArgs {
  const bf16* in;
  int in_cs, in_co;  // input channel stride and offset
  const bf16* w;     // [9][Cin][Cout]
  const float* bias;  // Cout, or null
  bf16* out;
  int out_cs, out_co;
  bf16* pre;  // pre-activation [P][Cout], or null
  const bf16* gate;  // scale by gelu_grad(gate[p][c]) (stride gate_cs, offset gate_co), or null
  int gate_cs, gate_co;
  int N, H, W, Cin, Cout;
  int gelu;  // apply GELU to the output
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return (uint32_t)__cvta_generic_to_shared(p);
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src, bool valid) {
  const int n = valid ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(smem_u32(dst)), "l"(src), "r"(n));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

__device__ __forceinline__ void ldsm_x4(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(smem_u32(p)));
}
__device__ __forceinline__ void ldsm_x4_t(uint32_t& r0, uint32_t& r1, uint32_t& r2, uint32_t& r3, const void* p) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
               : "=r"(r0), "=r"(r1), "=r"(r2), "=r"(r3)
               : "r"(smem_u32(p)));
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, "
      "{%0,%1,%2,%3};\n"
      : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// ------------------------------------------------------------ conv 3x3
// block: 128 pixels x BN channels, 256 threads; BN = 64: warps 4 x 2 of
// 32 x 32; BN = 32: warps 8 x 1 of 16 x 32. K chunk 32 = (tap, 32 channels).
constexpr int CONV_BM = 128, CONV_BK = 32, A_LD = CONV_BK + 8;

template <int BN> __global__ void __launch_bounds__(256) conv3x3_kernel(ConvArgs a) {
  after_previous();
  constexpr int B_LD = BN + 8;
  constexpr int WARPS_M = BN == 64 ? 4 : 8;
  constexpr int WM = CONV_BM / WARPS_M;  // 32 or 16
  constexpr int MI = WM / 16;            // m16 tiles per warp
  __shared__ __align__(16) bf16 sA[2][CONV_BM][A_LD];
  __shared__ __align__(16) bf16 sB[2][CONV_BK][B_LD];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp % WARPS_M, wn = warp / WARPS_M;
  const long long P = (long long)a.N * a.H * a.W;
  const long long m0 = (long long)blockIdx.x * CONV_BM;
  const int n0 = blockIdx.y * BN;
  const int kchunks = 9 * (a.Cin / CONV_BK);
  // this thread's A rows: r = tid / 2, vectors (tid % 2) * 2 + {0, 1}
  const int ar = tid >> 1, av0 = (tid & 1) * 2;
  const long long ap = m0 + ar;
  int an = 0, ah = 0, aw = 0;
  if (ap < P) {
    an = (int)(ap / ((long long)a.H * a.W));
    const int rem = (int)(ap % ((long long)a.H * a.W));
    ah = rem / a.W;
    aw = rem % a.W;
  }
  auto load = [&](int chunk, int buf) {
    const int tap = chunk / (a.Cin / CONV_BK), c0 = (chunk % (a.Cin / CONV_BK)) * CONV_BK;
    const int dy = tap / 3 - 1, dx = tap % 3 - 1;
    const int hh = ah + dy, ww = aw + dx;
    const bool ok = ap < P && hh >= 0 && hh < a.H && ww >= 0 && ww < a.W;
    const bf16* src = ok ? a.in + ((long long)(an * a.H + hh) * a.W + ww) * a.in_cs + a.in_co + c0 : a.in;
#pragma unroll
    for (int v = 0; v < 2; v++) cp_async16(&sA[buf][ar][(av0 + v) * 8], ok ? src + (av0 + v) * 8 : a.in, ok);
    constexpr int BV = BN / 8;  // vectors per B row
    if (tid < CONV_BK * BV) {
      const int br = tid / BV, bv = tid % BV;
      const int col = n0 + bv * 8;
      const bool okb = col < a.Cout;
      const bf16* bsrc = okb ? a.w + ((long long)(tap * a.Cin + c0 + br)) * a.Cout + col : a.w;
      cp_async16(&sB[buf][br][bv * 8], bsrc, okb);
    }
    cp_async_commit();
  };
  float acc[MI][4][4];
#pragma unroll
  for (int i = 0; i < MI; i++)
#pragma unroll
    for (int j = 0; j < 4; j++)
#pragma unroll
      for (int q = 0; q < 4; q++) acc[i][j][q] = 0.0f;
  load(0, 0);
  for (int ch = 0; ch < kchunks; ch++) {
    const int buf = ch & 1;
    if (ch + 1 < kchunks) {
      load(ch + 1, buf ^ 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
#pragma unroll
    for (int ks = 0; ks < CONV_BK; ks += 16) {
      uint32_t af[MI][4];
#pragma unroll
      for (int i = 0; i < MI; i++)
        ldsm_x4(af[i][0], af[i][1], af[i][2], af[i][3], &sA[buf][wm * WM + i * 16 + (lane & 15)][ks + (lane >> 4) * 8]);
      uint32_t bfr[4][2];
#pragma unroll
      for (int jj = 0; jj < 2; jj++) {
        uint32_t r0, r1, r2, r3;
        ldsm_x4_t(r0, r1, r2, r3, &sB[buf][ks + (lane & 15)][wn * 32 + jj * 16 + (lane >> 4) * 8]);
        bfr[2 * jj][0] = r0;
        bfr[2 * jj][1] = r1;
        bfr[2 * jj + 1][0] = r2;
        bfr[2 * jj + 1][1] = r3;
      }
#pragma unroll
      for (int i = 0; i < MI; i++)
#pragma unroll
        for (int j = 0; j < 4; j++) mma_bf16(acc[i][j], af[i], bfr[j][0], bfr[j][1]);
    }
    __syncthreads();
  }
  // epilogue
  const int g = lane >> 2, t4 = lane & 3;
#pragma unroll
  for (int i = 0; i < MI; i++)
#pragma unroll
    for (int h2 = 0; h2 < 2; h2++) {
      const long long p = m0 + wm * WM + i * 16 + g + h2 * 8;
      if (p >= P) continue;
#pragma unroll
      for (int j = 0; j < 4; j++) {
        const int c = n0 + wn * 32 + j * 8 + t4 * 2;
        if (c >= a.Cout) continue;
        float v0 = acc[i][j][h2 * 2], v1 = acc[i][j][h2 * 2 + 1];
        if (a.bias) {
          v0 += a.bias[c];
          v1 += a.bias[c + 1];
        }
        if (a.gate) {
          const __nv_bfloat162 gz = *reinterpret_cast<const __nv_bfloat162*>(a.gate + p * a.gate_cs + a.gate_co + c);
          v0 *= gelu_grad(__bfloat162float(gz.x));
          v1 *= gelu_grad(__bfloat162float(gz.y));
        }
        if (a.pre)
          *reinterpret_cast<__nv_bfloat162*>(a.pre + p * a.Cout + c) = __floats2bfloat162_rn(v0, v1);
        if (a.gelu) {
          v0 = gelu_f(v0);
          v1 = gelu_f(v1);
        }
        *reinterpret_cast<__nv_bfloat162*>(a.out + p * a.out_cs + a.out_co + c) = __floats2bfloat162_rn(v0, v1);
      }
    }
}

// ------------------------------------------------- conv 3x3, tcgen05 path
// The same implicit GEMM on the 5th-generation tensor cores, for images that
// do not tile into 128-pixel blocks (conv3x3_tma_kernel takes the others). A
// CTA of 128 threads owns 128 output pixels x BN output channels; the FP32
// accumulator (128 lanes x BN columns) lives in tensor memory. Per K chunk of
// 32 (one tap, 32 input channels) the threads stage, with cp.async into a ring
// of TC_STAGES buffers TC_AHEAD chunks ahead, the A tile (pixels x channels,
// K-major 8x16-byte core matrices, zero fill at the image border) and the B
// tile (weights rows of [tap][Cin][Cout], MN-major core matrices); one thread
// issues two tcgen05.mma (M 128, N BN, K 16, BF16 in, FP32 accumulate) and
// commits them to the stage's mbarrier; a stage is refilled once the MMAs
// that read it are done. The epilogue reads the accumulator with tcgen05.ld
// (warp w: lanes 32w..32w+31, one pixel a thread) and applies the same bias /
// gate / GELU as conv3x3_kernel. Every mbarrier wait is bounded; a wait that
// runs out counts in g_tc_timeouts and the kernel stops issuing, waits
// (bounded) for the MMAs it issued and frees its tensor memory.
#ifndef CLV_TC_STAGES
#define CLV_TC_STAGES 4
#endif
#ifndef CLV_TC_AHEAD
#define CLV_TC_AHEAD 2
#endif
constexpr int TC_BM = 128, TC_BK = 32, TC_STAGES = CLV_TC_STAGES, TC_AHEAD = CLV_TC_AHEAD;
static_assert(TC_AHEAD >= 1 && TC_AHEAD < TC_STAGES, "pipeline depth");

__device__ int g_tc_timeouts;  // bounded waits that ran out (read by clv_unet_timeouts)

// shared-memory matrix descriptor: byte offsets lbo (leading-dimension
// stride) and sbo (stride-dimension stride), descriptor version 1 (sm_100),
// layout 0 (no swizzle) or 4 (64-byte swizzle)
__device__ __forceinline__ uint64_t tc_smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo, uint32_t layout = 0) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46) | ((uint64_t)layout << 61);
}
// instruction descriptor of kind::f16: BF16 A and B, FP32 D, A K-major,
// B MN-major, M x N
__host__ __device__ constexpr uint32_t tc_idesc(int M, int N) {
  return (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}
__device__ __forceinline__ bool tc_wait(uint32_t bar, uint32_t parity) {
  for (int i = 0; i < (1 << 22); i++) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.b32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
__device__ __forceinline__ void tc_mma(uint32_t dtm, uint64_t da, uint64_t db, uint32_t idesc, uint32_t accum) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(dtm),
      "l"(da), "l"(db), "r"(idesc), "r"(accum));
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }

// the epilogue of one pixel (thread) over 8 accumulator columns starting at
// output channel c0: bias, gate, pre-activation, GELU, BF16 store
__device__ __forceinline__ void tc_epilogue8(const ConvArgs& a, long long p, int c0, const uint32_t (&v)[8]) {
  // 16-byte accesses when every row of 8 channels starts 16-byte aligned
  const bool vec = c0 + 8 <= a.Cout && ((a.out_cs | a.out_co) & 7) == 0 &&
                   ((reinterpret_cast<uintptr_t>(a.out) | reinterpret_cast<uintptr_t>(a.pre) |
                     reinterpret_cast<uintptr_t>(a.gate)) & 15) == 0 &&
                   (!a.gate || ((a.gate_cs | a.gate_co) & 7) == 0);
  if (vec) {
    float f[8];
#pragma unroll
    for (int jj = 0; jj < 8; jj++) f[jj] = __uint_as_float(v[jj]);
    if (a.bias)
#pragma unroll
      for (int jj = 0; jj < 8; jj++) f[jj] += a.bias[c0 + jj];
    if (a.gate) {
      const uint4 g4 = *reinterpret_cast<const uint4*>(a.gate + p * a.gate_cs + a.gate_co + c0);
      const __nv_bfloat162* gz = reinterpret_cast<const __nv_bfloat162*>(&g4);
#pragma unroll
      for (int jj = 0; jj < 4; jj++) {
        f[2 * jj] *= gelu_grad(__bfloat162float(gz[jj].x));
        f[2 * jj + 1] *= gelu_grad(__bfloat162float(gz[jj].y));
      }
    }
    uint4 o;
    __nv_bfloat162* ob = reinterpret_cast<__nv_bfloat162*>(&o);
    if (a.pre) {
#pragma unroll
      for (int jj = 0; jj < 4; jj++) ob[jj] = __floats2bfloat162_rn(f[2 * jj], f[2 * jj + 1]);
      *reinterpret_cast<uint4*>(a.pre + p * a.Cout + c0) = o;
    }
    if (a.gelu)
#pragma unroll
      for (int jj = 0; jj < 8; jj++) f[jj] = gelu_f(f[jj]);
#pragma unroll
    for (int jj = 0; jj < 4; jj++) ob[jj] = __floats2bfloat162_rn(f[2 * jj], f[2 * jj + 1]);
    *reinterpret_cast<uint4*>(a.out + p * a.out_cs + a.out_co + c0) = o;
    return;
  }
#pragma unroll
  for (int jj = 0; jj < 8; jj += 2) {
    const int c = c0 + jj;
    if (c >= a.Cout) continue;
    float v0 = __uint_as_float(v[jj]), v1 = __uint_as_float(v[jj + 1]);
    if (a.bias) {
      v0 += a.bias[c];
      v1 += a.bias[c + 1];
    }
    if (a.gate) {
      const __nv_bfloat162 gz = *reinterpret_cast<const __nv_bfloat162*>(a.gate + p * a.gate_cs + a.gate_co + c);
      v0 *= gelu_grad(__bfloat162float(gz.x));
      v1 *= gelu_grad(__bfloat162float(gz.y));
    }
    if (a.pre) *reinterpret_cast<__nv_bfloat162*>(a.pre + p * a.Cout + c) = __floats2bfloat162_rn(v0, v1);
    if (a.gelu) {
      v0 = gelu_f(v0);
      v1 = gelu_f(v1);
    }
    *reinterpret_cast<__nv_bfloat162*>(a.out + p * a.out_cs + a.out_co + c) = __floats2bfloat162_rn(v0, v1);
  }
}
__device__ __forceinline__ void tc_ld8(uint32_t taddr, uint32_t (&v)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];\n"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
}

template <int BN> struct TcSmem {
  bf16 A[TC_STAGES][TC_BM * TC_BK];
  bf16 B[TC_STAGES][BN * TC_BK];
  uint64_t bar[TC_STAGES];
  uint32_t tmem;
};

template <int BN> __global__ void __launch_bounds__(128) conv3x3_tc_kernel(ConvArgs a) {
  after_previous();
  static_assert(BN == 32 || BN == 64 || BN == 128, "BN");
  constexpr int TCOLS = BN;                    // tensor-memory columns (a power of two >= 32)
  constexpr uint32_t LBO_A = TC_BM / 8 * 128;  // A: K-adjacent core matrices (8 channels apart)
  constexpr uint32_t LBO_B = BN / 8 * 128;     // B: K-adjacent core matrices (8 rows apart)
  constexpr uint32_t IDESC = tc_idesc(TC_BM, BN);
  extern __shared__ __align__(1024) unsigned char tc_raw[];
  TcSmem<BN>& s = *reinterpret_cast<TcSmem<BN>*>(tc_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const long long P = (long long)a.N * a.H * a.W;
  const long long m0 = (long long)blockIdx.x * TC_BM;
  const int n0 = blockIdx.y * BN;
  const int cpt = a.Cin / TC_BK;  // K chunks per tap
  const int kchunks = 9 * cpt;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s.tmem)),
                 "r"(TCOLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  if (tid == 0) {
#pragma unroll
    for (int st = 0; st < TC_STAGES; st++)
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&s.bar[st])) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s.tmem;

  // this thread's A row (pixel m0 + tid)
  const long long ap = m0 + tid;
  int an = 0, ah = 0, aw = 0;
  if (ap < P) {
    an = (int)(ap / ((long long)a.H * a.W));
    const int rem = (int)(ap % ((long long)a.H * a.W));
    ah = rem / a.W;
    aw = rem % a.W;
  }
  auto load = [&](int chunk, int st) {
    const int tap = chunk / cpt, c0 = (chunk % cpt) * TC_BK;
    const int hh = ah + tap / 3 - 1, ww = aw + tap % 3 - 1;
    const bool ok = ap < P && hh >= 0 && hh < a.H && ww >= 0 && ww < a.W;
    const bf16* src = ok ? a.in + ((long long)(an * a.H + hh) * a.W + ww) * a.in_cs + a.in_co + c0 : a.in;
    unsigned char* A = reinterpret_cast<unsigned char*>(s.A[st]);
#pragma unroll
    for (int v = 0; v < TC_BK / 8; v++)  // core matrix (row group tid/8, channel group v), row tid%8
      cp_async16(A + v * LBO_A + (tid >> 3) * 128 + (tid & 7) * 16, ok ? src + v * 8 : a.in, ok);
    unsigned char* B = reinterpret_cast<unsigned char*>(s.B[st]);
#pragma unroll
    for (int q = tid; q < BN * TC_BK / 8; q += 128) {  // weight row kk, output channels ng*8 .. ng*8+7
      const int kk = q / (BN / 8), ng = q % (BN / 8);
      const int col = n0 + ng * 8;
      const bool okb = col < a.Cout;
      const bf16* bsrc = okb ? a.w + ((long long)(tap * a.Cin + c0 + kk)) * a.Cout + col : a.w;
      cp_async16(B + (kk >> 3) * LBO_B + ng * 128 + (kk & 7) * 16, bsrc, okb);
    }
  };

  bool live = true;  // no bounded wait has run out
#pragma unroll
  for (int c = 0; c < TC_AHEAD; c++) {
    if (c < kchunks) load(c, c);
    cp_async_commit();
  }
  for (int ch = 0; ch < kchunks; ch++) {
    const int st = ch % TC_STAGES;
    const int nxt = ch + TC_AHEAD;
    if (nxt < kchunks) {
      // the stage of chunk nxt was last read by the MMAs of chunk old
      const int old = nxt - TC_STAGES;
      if (old >= 0 && live && !tc_wait(smem_u32(&s.bar[old % TC_STAGES]), (old / TC_STAGES) & 1)) {
        live = false;
        atomicAdd(&g_tc_timeouts, 1);
      }
      if (live) load(nxt, nxt % TC_STAGES);
    }
    cp_async_commit();
    cp_async_wait<TC_AHEAD>();  // chunk ch has landed
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    __syncthreads();
    if (tid == 0 && live) {
      tc_fence_after();
      const uint32_t sa = smem_u32(s.A[st]), sb = smem_u32(s.B[st]);
#pragma unroll
      for (int kh = 0; kh < TC_BK / 16; kh++)
        tc_mma(tmem, tc_smem_desc(sa + kh * 2 * LBO_A, LBO_A, 128), tc_smem_desc(sb + kh * 2 * LBO_B, LBO_B, 128),
               IDESC, (ch > 0 || kh > 0) ? 1u : 0u);
      tc_commit(smem_u32(&s.bar[st]));
    }
  }
  cp_async_wait<0>();
  // the last chunk's commit completes when every MMA of the tile has
  const int last = kchunks - 1;
  bool ready = tc_wait(smem_u32(&s.bar[last % TC_STAGES]), (last / TC_STAGES) & 1);
  if (!ready) atomicAdd(&g_tc_timeouts, 1);
  tc_fence_after();
  live = live && ready;
  live = __syncthreads_and(live);

  if (live) {
    const long long p = m0 + warp * 32 + lane;
    const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
#pragma unroll 1
    for (int c8 = 0; c8 < BN / 8; c8++) {
      uint32_t v[8];
      tc_ld8(trow + c8 * 8, v);
      if (p < P) tc_epilogue8(a, p, n0 + c8 * 8, v);
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TCOLS));
  }
}

// ------------------------------------------ conv 3x3, TMA + tcgen05 path
// For images that tile evenly into blocks of 128 pixels (W divides 128 and H
// is a multiple of 128 / W, or W is a multiple of 128). Persistent and warp
// specialised: a CTA of 6 warps takes tiles (a (128 / bw) x bw pixel block of
// one image, BN output channels) blockIdx.x, blockIdx.x + gridDim.x, ...
//   * warp 0 (one thread) loads each K chunk (one tap, 32 input channels)
//     with the tensor memory accelerator into a ring of TC_STAGES stages, the
//     image border as TMA's zero fill. With SW (the default), one box of
//     [32 channels, bw, 128 / bw, 1] of the activation tensor at the tap's
//     offset lands as the K-major operand in the 64-byte swizzled layout
//     (128 pixel rows of 64 bytes; 8-row atoms 512 bytes apart) and BN / 32
//     boxes of [32 output channels, 32 rows] of the weights as the MN-major
//     operand in the same swizzle; without SW, boxes 16 bytes wide fill the
//     no-swizzle core-matrix layouts (four [8, bw, 128 / bw, 1] activation
//     boxes, BN / 8 [8, 32] weight boxes);
//   * warp 1 (one thread) issues the chunk's two tcgen05.mma (M 128, N BN,
//     K 16) into one of two tensor-memory accumulators, commits them to the
//     stage's empty barrier and, after a tile's last chunk, to the
//     accumulator's full barrier;
//   * warps 2-5 drain a full accumulator (warp w: lanes 32 (w % 4) ..,
//     one pixel a thread) through the bias / gate / GELU epilogue while the
//     next tile accumulates in the other one, then free it.
// Every wait is bounded (g_tc_timeouts); a role whose wait runs out stops.
// Threads: a producer warp, an issuer warp, four epilogue warps and, with two or
// more weight boxes a chunk, a second producer warp for those (one thread issues
// a load every 150 to 200 cycles, which was the pace of the wide tiles).
__host__ __device__ constexpr int tma_threads(int BN) { return BN >= 64 ? 224 : 192; }

template <int BN> struct TmaSmem {
  bf16 A[TC_STAGES][TC_BM * TC_BK];
  bf16 B[TC_STAGES][BN * TC_BK];
  uint64_t full[TC_STAGES], empty[TC_STAGES], acc_full[2], acc_empty[2];
  uint32_t tmem;
};

__device__ __forceinline__ void tma_load4(uint32_t dst, const void* map, int c0, int c1, int c2, int c3, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];\n" ::"r"(
          dst),
      "l"(map), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(bar)
      : "memory");
}
__device__ __forceinline__ void tma_load2(uint32_t dst, const void* map, int c0, int c1, uint32_t bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n" ::"r"(dst),
      "l"(map), "r"(c0), "r"(c1), "r"(bar)
      : "memory");
}

template <int BN, bool SW>
__global__ void __launch_bounds__(tma_threads(BN))
    conv3x3_tma_kernel(const __grid_constant__ CUtensorMap ta, const __grid_constant__ CUtensorMap tb, ConvArgs a, int bw) {
  after_previous();
  static_assert(BN == 32 || BN == 64 || BN == 128, "BN");
  constexpr int TCOLS = 2 * BN;  // two accumulators
  constexpr bool WIDE = tma_threads(BN) == 224;
  constexpr uint32_t A_BYTES = TC_BM * TC_BK * 2, B_BYTES = BN * TC_BK * 2;
  // no swizzle: A 8-channel groups (LBO) 2048 B apart, 8-row groups (SBO) 128 B; B 8-row groups (LBO) 128 B,
  // 8-channel groups (SBO) 512 B. 64-byte swizzle: A 8-row atoms (SBO) 512 B apart, K step of 16 channels
  // +32 B; B 32-channel groups (LBO) 2048 B apart, 8-row atoms (SBO) 512 B, K step of 16 rows +1024 B
  constexpr uint32_t LAYOUT = SW ? 4u : 0u;
  constexpr uint32_t LBO_A = SW ? 16 : TC_BM * 16, SBO_A = SW ? 512 : 128;
  constexpr uint32_t LBO_B = SW ? 2048 : 128, SBO_B = SW ? 512 : TC_BK * 16;
  constexpr uint32_t KSTEP_A = SW ? 32 : 2 * TC_BM * 16, KSTEP_B = SW ? 1024 : 2 * 128;
  constexpr uint32_t IDESC = tc_idesc(TC_BM, BN);
  extern __shared__ __align__(1024) unsigned char tma_raw[];
  TmaSmem<BN>& s = *reinterpret_cast<TmaSmem<BN>*>(tma_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int bh = TC_BM / bw;
  const int tiles_w = a.W / bw, tiles_h = a.H / bh;
  const int ntn = a.Cout / BN;
  const long long ntiles = (long long)a.N * tiles_h * tiles_w * ntn;
  const int cpt = a.Cin / TC_BK, kchunks = 9 * cpt;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s.tmem)),
                 "r"(TCOLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  if (tid == 32) {
#pragma unroll
    for (int st = 0; st < TC_STAGES; st++) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(&s.full[st])), "r"(WIDE ? 2 : 1)
                   : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&s.empty[st])) : "memory");
    }
#pragma unroll
    for (int q = 0; q < 2; q++) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&s.acc_full[q])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 128;\n" ::"r"(smem_u32(&s.acc_empty[q])) : "memory");
    }
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s.tmem;

  // tile q -> (image, pixel block, output-channel block); channel blocks of
  // one pixel block are consecutive, so they share its activations in L2
  auto tile = [&](long long q, int& img, int& h0, int& w0, int& n0) {
    n0 = (int)(q % ntn) * BN;
    q /= ntn;
    w0 = (int)(q % tiles_w) * bw;
    q /= tiles_w;
    h0 = (int)(q % tiles_h) * bh;
    img = (int)(q / tiles_h);
  };

  // the loads of one thread: the activations (ACT), the weights (WGT) or both
  auto produce = [&](auto act, auto wgt) {
    constexpr bool ACT = decltype(act)::value, WGT = decltype(wgt)::value;
    // counters in place of divisions: this one thread's instructions, one
    // after the other, are the pace of a tile with few of them in flight
    long long it = 0;
    int st = 0;
    uint32_t round = 0;  // it / TC_STAGES
    bool ok = true;
    for (long long q = blockIdx.x; q < ntiles && ok; q += gridDim.x) {
      int img, h0, w0, n0;
      tile(q, img, h0, w0, n0);
      int row = 0;  // tap Cin + c0 of the weights
      for (int tap = 0; tap < 9 && ok; tap++) {
        const int wt = w0 + tap % 3 - 1, ht = h0 + tap / 3 - 1;
        for (int c0 = 0; c0 < a.Cin; c0 += TC_BK, row += TC_BK, it++) {
          if (round && !tc_wait(smem_u32(&s.empty[st]), (round - 1) & 1)) {
            ok = false;
            atomicAdd(&g_tc_timeouts, 1);
            break;
          }
          const uint32_t fb = smem_u32(&s.full[st]);
          asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(fb),
                       "r"((ACT ? A_BYTES : 0u) + (WGT ? B_BYTES : 0u))
                       : "memory");
          const uint32_t sa = smem_u32(s.A[st]), sb = smem_u32(s.B[st]);
          if constexpr (ACT) {
            if (SW) {
              tma_load4(sa, &ta, a.in_co + c0, wt, ht, img, fb);
            } else {
#pragma unroll
              for (int g = 0; g < TC_BK / 8; g++)
                tma_load4(sa + g * TC_BM * 16, &ta, a.in_co + c0 + 8 * g, wt, ht, img, fb);
            }
          }
          if constexpr (WGT) {
            if (SW) {
#pragma unroll
              for (int ng = 0; ng < BN / 32; ng++) tma_load2(sb + ng * 2048, &tb, n0 + 32 * ng, row, fb);
            } else {
#pragma unroll
              for (int ng = 0; ng < BN / 8; ng++) tma_load2(sb + ng * TC_BK * 16, &tb, n0 + 8 * ng, row, fb);
            }
          }
          if (++st == TC_STAGES) st = 0, round++;
        }
      }
    }
    // the loads in flight land before the CTA can exit
    for (long long c = it - 1; c >= 0 && c >= it - TC_STAGES; c--)
      tc_wait(smem_u32(&s.full[c % TC_STAGES]), (uint32_t)((c / TC_STAGES) & 1));
  };
  if (warp == 0) {
    if (lane == 0) produce(std::true_type(), std::integral_constant<bool, !WIDE>());
  } else if (WIDE && warp == 6) {
    if (lane == 0) produce(std::false_type(), std::true_type());
  } else if (warp == 1) {
    if (lane == 0) {  // MMA issuer
      int t = 0, st = 0;
      uint32_t round = 0;
      bool ok = true;
      for (long long q = blockIdx.x; q < ntiles && ok; q += gridDim.x, t++) {
        const int acc = t & 1;
        if (t >= 2 && !tc_wait(smem_u32(&s.acc_empty[acc]), (uint32_t)(((t >> 1) - 1) & 1))) {
          ok = false;
          atomicAdd(&g_tc_timeouts, 1);
          break;
        }
        tc_fence_after();
        const uint32_t dtm = tmem + acc * BN;
        for (int ch = 0; ch < kchunks; ch++) {
          if (!tc_wait(smem_u32(&s.full[st]), round & 1)) {
            ok = false;
            atomicAdd(&g_tc_timeouts, 1);
            break;
          }
          tc_fence_after();
          const uint32_t sa = smem_u32(s.A[st]), sb = smem_u32(s.B[st]);
#pragma unroll
          for (int kh = 0; kh < TC_BK / 16; kh++)
            tc_mma(dtm, tc_smem_desc(sa + kh * KSTEP_A, LBO_A, SBO_A, LAYOUT),
                   tc_smem_desc(sb + kh * KSTEP_B, LBO_B, SBO_B, LAYOUT), IDESC, (ch > 0 || kh > 0) ? 1u : 0u);
          tc_commit(smem_u32(&s.empty[st]));
          if (++st == TC_STAGES) st = 0, round++;
        }
        if (ok) tc_commit(smem_u32(&s.acc_full[acc]));
      }
    }
  } else {  // epilogue warps 2-5
    const int quarter = warp & 3;  // tensor-memory lanes 32 quarter .. 32 quarter + 31
    const int r = quarter * 32 + lane;
    int t = 0;
    for (long long q = blockIdx.x; q < ntiles; q += gridDim.x, t++) {
      const int acc = t & 1;
      const bool ok = __all_sync(0xffffffffu, tc_wait(smem_u32(&s.acc_full[acc]), (uint32_t)((t >> 1) & 1)));
      if (!ok) {
        if (lane == 0) atomicAdd(&g_tc_timeouts, 1);
        break;
      }
      tc_fence_after();
      int img, h0, w0, n0;
      tile(q, img, h0, w0, n0);
      const long long p = ((long long)img * a.H + h0 + r / bw) * a.W + w0 + r % bw;
      const uint32_t trow = tmem + ((uint32_t)(quarter * 32) << 16) + acc * BN;
#pragma unroll 1
      for (int c8 = 0; c8 < BN / 8; c8++) {
        uint32_t v[8];
        tc_ld8(trow + c8 * 8, v);
        tc_epilogue8(a, p, n0 + c8 * 8, v);
      }
      tc_fence_before();
      asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(&s.acc_empty[acc])) : "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(TCOLS));
  }
}

// ------------------------------------------------------------ wgrad 3x3
struct WgradArgs {
  const bf16* x;  // layer input slice
  int x_cs, x_co;
  const bf16* g;  // gradient wrt the pre-activation [P][Cout]
  float* part;    // [S][9 Cin][Cout]
  int N, H, W, Cin, Cout;
  long long pix_per_split;
};
constexpr int WG_BM = 64, WG_BN = 64, WG_BK = 32, WG_LD = 64 + 8;

// grid (ceil(9 Cin / 64), ceil(Cout / 64), S); warps 2 (m) x 4 (n) of 32 x 16
__global__ void __launch_bounds__(256) wgrad3x3_kernel(WgradArgs a) {
  after_previous();
  __shared__ __align__(16) bf16 sA[2][WG_BK][WG_LD];  // [pixel][(tap, ci)]
  __shared__ __align__(16) bf16 sB[2][WG_BK][WG_LD];  // [pixel][co]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int wm = warp & 1, wn = warp >> 1;
  const int M = 9 * a.Cin;
  const int mb = blockIdx.x * WG_BM, nb = blockIdx.y * WG_BN;
  const long long P = (long long)a.N * a.H * a.W;
  const long long p_lo = (long long)blockIdx.z * a.pix_per_split;
  const long long p_hi = p_lo + a.pix_per_split < P ? p_lo + a.pix_per_split : P;
  // this thread loads pixel row r = tid / 8 and vector v = tid % 8 of both tiles
  const int r = tid >> 3, v = tid & 7;
  const int m_v = mb + v * 8;  // 8 consecutive (tap, ci) rows: one tap, as Cin % 8 == 0
  const int tap = m_v < M ? m_v / a.Cin : 0, ci0 = m_v < M ? m_v % a.Cin : 0;
  const int dy = tap / 3 - 1, dx = tap % 3 - 1;
  auto load = [&](long long k0, int buf) {
    const long long p = k0 + r;
    bool okp = p < p_hi;
    int n = 0, h = 0, w = 0;
    if (okp) {
      n = (int)(p / ((long long)a.H * a.W));
      const int rem = (int)(p % ((long long)a.H * a.W));
      h = rem / a.W;
      w = rem % a.W;
    }
    const int hh = h + dy, ww = w + dx;
    const bool oka = okp && m_v < M && hh >= 0 && hh < a.H && ww >= 0 && ww < a.W;
    cp_async16(&sA[buf][r][v * 8],
               oka ? a.x + ((long long)(n * a.H + hh) * a.W + ww) * a.x_cs + a.x_co + ci0 : a.x, oka);
    const int co = nb + v * 8;
    const bool okb = okp && co < a.Cout;
    cp_async16(&sB[buf][r][v * 8], okb ? a.g + p * a.Cout + co : a.g, okb);
    cp_async_commit();
  };
  float acc[2][2][4];
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
      for (int q = 0; q < 4; q++) acc[i][j][q] = 0.0f;
  const long long nk = (p_hi - p_lo + WG_BK - 1) / WG_BK;
  if (nk > 0) load(p_lo, 0);
  for (long long kc = 0; kc < nk; kc++) {
    const int buf = (int)(kc & 1);
    if (kc + 1 < nk) {
      load(p_lo + (kc + 1) * WG_BK, buf ^ 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
#pragma unroll
    for (int ks = 0; ks < WG_BK; ks += 16) {
      uint32_t af[2][4];
#pragma unroll
      for (int i = 0; i < 2; i++) {
        // A (m x k) from sA[k][m]: rows k, transposed loads
        const int k = ks + (lane & 7) + ((lane >> 4) << 3);
        const int m = wm * 32 + i * 16 + ((lane >> 3) & 1) * 8;
        ldsm_x4_t(af[i][0], af[i][1], af[i][2], af[i][3], &sA[buf][k][m]);
      }
      uint32_t r0, r1, r2, r3;
      ldsm_x4_t(r0, r1, r2, r3, &sB[buf][ks + (lane & 15)][wn * 16 + (lane >> 4) * 8]);
#pragma unroll
      for (int i = 0; i < 2; i++) {
        mma_bf16(acc[i][0], af[i], r0, r1);
        mma_bf16(acc[i][1], af[i], r2, r3);
      }
    }
    __syncthreads();
  }
  const int g = lane >> 2, t4 = lane & 3;
  float* out = a.part + (long long)blockIdx.z * M * a.Cout;
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int h2 = 0; h2 < 2; h2++) {
      const int m = mb + wm * 32 + i * 16 + g + h2 * 8;
      if (m >= M) continue;
#pragma unroll
      for (int j = 0; j < 2; j++) {
        const int c = nb + wn * 16 + j * 8 + t4 * 2;
        if (c >= a.Cout) continue;
        out[(long long)m * a.Cout + c] = acc[i][j][h2 * 2];
        out[(long long)m * a.Cout + c + 1] = acc[i][j][h2 * 2 + 1];
      }
    }
}

// out[i] (+)= sum_s part[s][i], in s order
// ------------------------------------------ wgrad 3x3, TMA + tcgen05 path
// (the default path; wgrad3x3_kernel takes images that do not tile and the
// mma.sync paths.) The weight gradient on the
// 5th-generation tensor cores, for images whose pixels tile into blocks of 32
// (bw = min(W, 64) columns x 64 / bw rows):
// D[(tap, ci)][co] = sum over pixels p of x[p + tap][ci] g[p][co], the rows
// r = tap * Cin + ci of the [9 Cin][Cout] result in tiles of M = 128 (four
// 32-channel groups, each a [32 channels, bw, 64 / bw, 1] box of x shifted by
// its tap, the image border as zero fill), N = up to 128 output channels
// ([32, bw, 64 / bw, 1] boxes of g), K = 64-pixel blocks; both operands are
// MN-major in the 64-byte swizzled layout. A CTA of 128 threads takes one
// (row tile, channel tile) and a contiguous range of pixel blocks (split K):
// threads 0, 64 and 96 load with TMA into WGT_STAGES stages, thread 32 issues the
// tcgen05.mma and commits each stage back, and all four warps write the
// accumulator (one row a thread) as an FP32 partial [split][9 Cin][Cout] that
// reduce_partials_kernel adds in a fixed order.
constexpr int WGT_BM = 128, WGT_BN = 128, WGT_BK = 64, WGT_STAGES = 3;

struct WgTmaSmem {
  bf16 A[WGT_STAGES][WGT_BM * WGT_BK];
  bf16 B[WGT_STAGES][WGT_BN * WGT_BK];
  uint64_t full[WGT_STAGES], empty[WGT_STAGES], done;
  uint32_t tmem;
};

__global__ void __launch_bounds__(128)
    wgrad3x3_tma_kernel(const __grid_constant__ CUtensorMap tg, const __grid_constant__ CUtensorMap tx, WgradArgs a,
                        int bw, int chunks_per_split) {
  after_previous();
  // MN-major, 64-byte swizzle: 32-channel groups (one box each) WGT_BK x 64 B apart, 8-row atoms 512 B,
  // K step of 16 pixel rows 1024 B
  constexpr uint32_t LBO = WGT_BK * 64, SBO = 512, KSTEP = 1024, LAYOUT = 4;
  extern __shared__ __align__(1024) unsigned char wgt_raw[];
  WgTmaSmem& s = *reinterpret_cast<WgTmaSmem*>(wgt_raw);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rows = 9 * a.Cin;
  const int mblocks = (rows + WGT_BM - 1) / WGT_BM;
  const int m0 = (blockIdx.x % mblocks) * WGT_BM, co0 = (blockIdx.x / mblocks) * WGT_BN;
  const int nn = min(WGT_BN, a.Cout - co0);        // a multiple of 32
  const int groups = min(4, (rows - m0) / 32);     // 32-row groups with data
  const int split = blockIdx.y;
  const int bh = WGT_BK / bw;
  const int per_row = a.W / bw, per_img = per_row * (a.H / bh);
  const long long nchunks = (long long)a.N * per_img;
  const long long c0 = (long long)split * chunks_per_split;
  const long long c1 = min(nchunks, c0 + chunks_per_split);
  const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 15) | (1u << 16) | ((uint32_t)(nn >> 3) << 17) |
                         ((uint32_t)(WGT_BM >> 4) << 24);

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&s.tmem)),
                 "r"(WGT_BN));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
  }
  if (tid == 32) {
#pragma unroll
    for (int st = 0; st < WGT_STAGES; st++) {
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 3;\n" ::"r"(smem_u32(&s.full[st])) : "memory");
      asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&s.empty[st])) : "memory");
    }
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(&s.done)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = s.tmem;

  // Three TMA producers: warp 0 the first two row groups, warp 2 the other two,
  // warp 3 the gradients. One thread issues a load every 150 to 200 cycles, so
  // the four to eight boxes of a pixel block from one thread took longer than
  // its MMAs and loads.
  if (lane == 0 && warp != 1) {
    const int b0 = warp == 0 ? 0 : 2, nbox = warp == 3 ? nn / 32 : max(0, min(2, groups - b0));
    int gc[2], gw[2], gh[2];  // rows m0 + 32 (b0 + i) ..: one tap, 32 input channels
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const int r0 = m0 + 32 * (b0 + i), tap = r0 / a.Cin;
      gc[i] = a.x_co + r0 % a.Cin;
      gw[i] = tap % 3 - 1;
      gh[i] = tap / 3 - 1;
    }
    int img = (int)(c0 / per_img), q = (int)(c0 % per_img), h0 = (q / per_row) * bh, w0 = (q % per_row) * bw;
    long long it = 0;
    int st = 0;
    uint32_t round = 0;  // it / WGT_STAGES
    for (long long c = c0; c < c1; c++, it++) {
      if (round && !tc_wait(smem_u32(&s.empty[st]), (round - 1) & 1)) {
        atomicAdd(&g_tc_timeouts, 1);
        break;
      }
      const uint32_t fb = smem_u32(&s.full[st]);
      asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(fb),
                   "r"((uint32_t)(nbox * 32) * WGT_BK * 2)
                   : "memory");
      const uint32_t sa = smem_u32(s.A[st]), sb = smem_u32(s.B[st]);
      if (warp == 3) {
        for (int ng = 0; ng < nbox; ng++) tma_load4(sb + ng * LBO, &tg, co0 + 32 * ng, w0, h0, img, fb);
      } else {
#pragma unroll
        for (int i = 0; i < 2; i++)
          if (i < nbox) tma_load4(sa + (b0 + i) * LBO, &tx, gc[i], w0 + gw[i], h0 + gh[i], img, fb);
      }
      w0 += bw;  // the next pixel block
      if (w0 == a.W) {
        w0 = 0;
        h0 += bh;
        if (h0 == a.H) h0 = 0, img++;
      }
      if (++st == WGT_STAGES) st = 0, round++;
    }
    // the loads in flight land before the CTA can exit
    for (long long c = it - 1; c >= 0 && c >= it - WGT_STAGES; c--)
      tc_wait(smem_u32(&s.full[c % WGT_STAGES]), (uint32_t)((c / WGT_STAGES) & 1));
  } else if (tid == 32) {  // MMA issuer
    int st = 0;
    uint32_t round = 0;
    bool ok = true;
    for (long long c = c0; c < c1; c++) {
      if (!tc_wait(smem_u32(&s.full[st]), round & 1)) {
        ok = false;
        atomicAdd(&g_tc_timeouts, 1);
        break;
      }
      tc_fence_after();
      const uint32_t sa = smem_u32(s.A[st]), sb = smem_u32(s.B[st]);
#pragma unroll
      for (int kh = 0; kh < WGT_BK / 16; kh++)
        tc_mma(tmem, tc_smem_desc(sa + kh * KSTEP, LBO, SBO, LAYOUT), tc_smem_desc(sb + kh * KSTEP, LBO, SBO, LAYOUT),
               idesc, (c > c0 || kh > 0) ? 1u : 0u);
      tc_commit(smem_u32(&s.empty[st]));
      if (++st == WGT_STAGES) st = 0, round++;
    }
    if (ok && c1 > c0) tc_commit(smem_u32(&s.done));
  }
  // The other lanes of the warps wait here, not on the barrier: a try_wait
  // suspends the whole warp for a time, the producer's or the issuer's lane with
  // it (2.3 us a pixel block, whatever its size, in place of 0.6).
  __syncwarp();
  bool ready = c1 > c0 ? tc_wait(smem_u32(&s.done), 0) : true;
  tc_fence_after();
  ready = __syncthreads_and(ready);
  if (!ready && tid == 0) atomicAdd(&g_tc_timeouts, 1);
  if (ready) {
    const int r = m0 + warp * 32 + lane;  // (tap, ci) row of this thread
    const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
    float* out = a.part + ((long long)split * rows + r) * a.Cout + co0;
#pragma unroll 1
    for (int c8 = 0; c8 < nn / 8; c8++) {
      uint32_t v[8];
      tc_ld8(trow + c8 * 8, v);
      if (r < rows) {
        float4 lo, hi;
        const bool any = c1 > c0;
        lo.x = any ? __uint_as_float(v[0]) : 0.0f;
        lo.y = any ? __uint_as_float(v[1]) : 0.0f;
        lo.z = any ? __uint_as_float(v[2]) : 0.0f;
        lo.w = any ? __uint_as_float(v[3]) : 0.0f;
        hi.x = any ? __uint_as_float(v[4]) : 0.0f;
        hi.y = any ? __uint_as_float(v[5]) : 0.0f;
        hi.z = any ? __uint_as_float(v[6]) : 0.0f;
        hi.w = any ? __uint_as_float(v[7]) : 0.0f;
        *reinterpret_cast<float4*>(out + c8 * 8) = lo;
        *reinterpret_cast<float4*>(out + c8 * 8 + 4) = hi;
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(WGT_BN));
  }
}

// out[i] (+)= the sum over S partials of part[k][i], in order, a thread an output
__global__ void __launch_bounds__(256) reduce_partials_kernel(const float* part, int S, long long n, float* out,
                                                              int accumulate) {
  after_previous();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  float s = 0.0f;
#pragma unroll 8
  for (int k = 0; k < S; k++) s += part[(long long)k * n + i];
  out[i] = accumulate ? out[i] + s : s;
}
// The same sums (the same order) for few outputs: the weight gradients of the
// small layers and every bias have 32 to a few thousand, and a thread an output
// was one chain of S dependent reads on a nearly empty chip (20 us a launch, 29
// launches a training step). A block takes 32 outputs: its 32 warps bring
// the partials to shared memory, one adds them.
constexpr int RED_ROWS = 320;  // partials at most (the callers have up to 296)
__global__ void __launch_bounds__(1024) reduce_few_kernel(const float* part, int S, long long n, float* out,
                                                          int accumulate) {
  after_previous();
  __shared__ float sh[RED_ROWS][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const long long i = (long long)blockIdx.x * 32 + lane;
  float v[RED_ROWS / 32];
#pragma unroll
  for (int q = 0; q < RED_ROWS / 32; q++)
    v[q] = i < n && w + 32 * q < S ? part[(long long)(w + 32 * q) * n + i] : 0.0f;
#pragma unroll
  for (int q = 0; q < RED_ROWS / 32; q++) sh[w + 32 * q][lane] = v[q];
  __syncthreads();
  if (w != 0 || i >= n) return;
  float s = 0.0f;
#pragma unroll 16
  for (int k = 0; k < S; k++) s += sh[k][lane];
  out[i] = accumulate ? out[i] + s : s;
}
inline void reduce_partials(const float* part, int S, long long n, float* out, int accumulate, cudaStream_t s) {
  if (n < 65536 && S <= RED_ROWS) clv::launch_early(reduce_few_kernel, (unsigned int)((n + 31) / 32), 1024, 0, s, part, S, n, out,
                        accumulate);
  else clv::launch_early(reduce_partials_kernel, (unsigned int)((n + 255) / 256), 256, 0, s, part, S, n, out,
                        accumulate);
}

// Eight neighbouring channels (16 bytes) a thread for the layers below where
// C, the strides and the offsets are multiples of 8 and the pointers 16-byte
// aligned (vec8_ok); else one channel a thread. They move 30 to 100 MB a launch
// at the first level, and with one 2-byte element and two 64-bit divisions a
// thread they ran at a tenth of the memory's rate (32 images of 128 x 128, a
// training step's upsampling 323 us, now 27; skip gradients 240, now 73; first
// layer 216, now 53).
struct Vec8 {
  float v[8];
};
__device__ __forceinline__ Vec8 load8(const bf16* p) {
  const uint4 u = *reinterpret_cast<const uint4*>(p);
  const unsigned int w[4] = {u.x, u.y, u.z, u.w};
  Vec8 r;
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const __nv_bfloat162 h = *reinterpret_cast<const __nv_bfloat162*>(&w[i]);
    r.v[2 * i] = __low2float(h);
    r.v[2 * i + 1] = __high2float(h);
  }
  return r;
}
__device__ __forceinline__ void store8(bf16* p, const Vec8& r) {
  unsigned int w[4];
#pragma unroll
  for (int i = 0; i < 4; i++) {
    const __nv_bfloat162 h = __halves2bfloat162(__float2bfloat16_rn(r.v[2 * i]), __float2bfloat16_rn(r.v[2 * i + 1]));
    w[i] = *reinterpret_cast<const unsigned int*>(&h);
  }
  *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
}
inline bool vec8_ok(const void* p, int cs, int co) {
  return (reinterpret_cast<uintptr_t>(p) % 16) == 0 && cs % 8 == 0 && co % 8 == 0;
}

// column sums of g[P][C] (bias gradient): block b sums rows [b*rows, ...) into part[b][C]
__global__ void colsum_kernel(const bf16* g, int g_cs, long long P, int C, long long rows, float* part) {
  after_previous();
  const long long p0 = (long long)blockIdx.x * rows;
  const long long p1 = p0 + rows < P ? p0 + rows : P;
  for (int c = threadIdx.x; c < C; c += blockDim.x) {
    float s = 0.0f;
    for (long long p = p0; p < p1; p++) s += __bfloat162float(g[p * g_cs + c]);
    part[(long long)blockIdx.x * C + c] = s;
  }
}
// Sums over the pixels of a block, each output by one thread in pixel order
// (the order of colsum_kernel, wgrad_first_kernel and head_wgrad_kernel: the
// same bits). The chain of one output is short work (a few cycles a pixel);
// what those kernels waited for was a global load in every link of it. Here
// threads 256 .. 511 of a block bring the next tile of rows to shared memory
// (16 bytes a load, NV a thread) while the first 256 add up the present one.
// 32 images of 128 x 128, 32 channels: the first layer's weight gradient 1015 to
// 89 us, the head's 408 to 44, a bias gradient 110 to 18.
template <int NV> struct RowTile {
  static constexpr int NE = 256 * NV * 8;       // elements
  static constexpr int RMAX = 64 * NV;          // rows at most
  static __device__ __forceinline__ int rows(int C) { return min(NE / C, RMAX); }
  // rows p .. of g (up to p1) to dst[row][C]; q: the thread's number, 0 .. 255
  static __device__ __forceinline__ void load(const bf16* g, long long g_cs, long long p, long long p1, int C, int q,
                                              bf16* dst) {
    const int tx = C / 8, n = (int)min((long long)rows(C), p1 - p) * tx;
    uint4 v[NV];
#pragma unroll
    for (int i = 0; i < NV; i++) {
      const int k = q + 256 * i;
      if (k < n) v[i] = *reinterpret_cast<const uint4*>(g + (p + k / tx) * g_cs + 8 * (k % tx));
    }
#pragma unroll
    for (int i = 0; i < NV; i++) {
      const int k = q + 256 * i;
      if (k < n) *reinterpret_cast<uint4*>(dst + 8 * k) = v[i];
    }
  }
};
__global__ void __launch_bounds__(512) colsum8_kernel(const bf16* g, int g_cs, long long P, int C, long long rows,
                                                      float* part) {
  after_previous();
  typedef RowTile<4> T;
  __shared__ __align__(16) bf16 sh[2][T::NE];
  const int t = threadIdx.x, R = T::rows(C);
  const long long p0 = (long long)blockIdx.x * rows, p1 = p0 + rows < P ? p0 + rows : P;
  float s = 0.0f;
  if (t >= 256 && p0 < p1) T::load(g, g_cs, p0, p1, C, t - 256, sh[0]);
  int b = 0;
  for (long long p = p0; p < p1; p += R, b ^= 1) {
    __syncthreads();  // tile b is here, and the one before it has been read
    if (t >= 256) {
      if (p + R < p1) T::load(g, g_cs, p + R, p1, C, t - 256, sh[b ^ 1]);
    } else if (t < C) {
      const int n = (int)min((long long)R, p1 - p);
      const bf16* v = sh[b] + t;
#pragma unroll 16
      for (int r = 0; r < n; r++) s += __bfloat162float(v[r * C]);
    }
  }
  if (t < C) part[(long long)blockIdx.x * C + t] = s;
}

// --------------------------------------------------- small layers (CUDA cores)
// first layer: 1 input channel (FP32 image) -> C channels, bias, GELU
__global__ void conv_first_kernel(const float* x, const float* w /*[9][C]*/, const float* bias, int N, int H, int W,
                                  int C, bf16* pre, bf16* out, int out_cs, int out_co) {
  after_previous();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const long long P = (long long)N * H * W;
  if (t >= P * C) return;
  const long long p = t / C;
  const int c = (int)(t % C);
  const int n = (int)(p / ((long long)H * W)), rem = (int)(p % ((long long)H * W)), h = rem / W, wq = rem % W;
  float s = bias[c];
  for (int tap = 0; tap < 9; tap++) {
    const int hh = h + tap / 3 - 1, ww = wq + tap % 3 - 1;
    if (hh < 0 || hh >= H || ww < 0 || ww >= W) continue;
    s += x[((long long)n * H + hh) * W + ww] * w[tap * C + c];
  }
  pre[p * C + c] = __float2bfloat16_rn(s);
  out[p * out_cs + out_co + c] = __float2bfloat16_rn(gelu_f(s));
}
// its weight gradient: part[b][tap][c] = sum over pixel block b of x[p + tap] g[p][c]
__global__ void wgrad_first_kernel(const float* x, const bf16* g, int N, int H, int W, int C, long long rows,
                                   float* part) {
  after_previous();
  const long long P = (long long)N * H * W;
  const long long p0 = (long long)blockIdx.x * rows, p1 = p0 + rows < P ? p0 + rows : P;
  for (int q = threadIdx.x; q < 9 * C; q += blockDim.x) {
    const int tap = q / C, c = q % C;
    float s = 0.0f;
    for (long long p = p0; p < p1; p++) {
      const int n = (int)(p / ((long long)H * W)), rem = (int)(p % ((long long)H * W));
      const int hh = rem / W + tap / 3 - 1, ww = rem % W + tap % 3 - 1;
      if (hh < 0 || hh >= H || ww < 0 || ww >= W) continue;
      s += x[((long long)n * H + hh) * W + ww] * __bfloat162float(g[p * C + c]);
    }
    part[(long long)blockIdx.x * 9 * C + q] = s;
  }
}

// both with 8 channels a thread: the nine inputs of a pixel are read once for
// eight outputs; per output the same products in the same order
__global__ void __launch_bounds__(256) conv_first8_kernel(const float* x, const float* w, const float* bias, int N,
                                                          int H, int W, int C, bf16* pre, bf16* out, int out_cs,
                                                          int out_co) {
  after_previous();
  const unsigned int t = blockIdx.x * 256u + threadIdx.x, cg = (unsigned int)C / 8u;
  const unsigned int p = t / cg, c = 8u * (t % cg);
  if (p >= (unsigned int)(N * H * W)) return;
  const int wq = (int)(p % (unsigned int)W), hn = (int)(p / (unsigned int)W), h = hn % H;
  Vec8 s;
#pragma unroll
  for (int i = 0; i < 8; i++) s.v[i] = bias[c + i];
#pragma unroll
  for (int tap = 0; tap < 9; tap++) {
    const int hh = h + tap / 3 - 1, ww = wq + tap % 3 - 1;
    if (hh < 0 || hh >= H || ww < 0 || ww >= W) continue;
    const float xv = x[(long long)(hn - h + hh) * W + ww];
#pragma unroll
    for (int i = 0; i < 8; i++) s.v[i] += xv * __ldg(w + tap * C + c + i);
  }
  store8(pre + (long long)p * C + c, s);
#pragma unroll
  for (int i = 0; i < 8; i++) s.v[i] = gelu_f(s.v[i]);
  store8(out + (long long)p * out_cs + out_co + c, s);
}
// wgrad_first_kernel's sums with the tiles of RowTile: a thread has one channel
// and one row of taps (3 C <= 256). The pixels are consecutive, so a tap's
// inputs are too: x[p + dr W + ds].
__global__ void __launch_bounds__(512) wgrad_first8_kernel(const float* x, const bf16* g, int N, int H, int W, int C,
                                                           long long rows, float* part) {
  after_previous();
  typedef RowTile<2> T;
  __shared__ __align__(16) bf16 sh[2][T::NE];
  __shared__ __align__(16) float xs[2][3][T::RMAX + 4];  // x[p - 1 + dr W + i]
  const int t = threadIdx.x, R = T::rows(C);
  const long long P = (long long)N * H * W;
  const long long p0 = (long long)blockIdx.x * rows, p1 = p0 + rows < P ? p0 + rows : P;
  auto load = [&](long long p, int b) {
    constexpr int NX = T::RMAX + 2, NQ = (3 * NX + 255) / 256;
    float v[NQ];
#pragma unroll
    for (int u = 0; u < NQ; u++) {
      const int q = t - 256 + 256 * u, d = q / NX, i = q - d * NX;
      const long long k = p - 1 + (long long)(d - 1) * W + i;
      v[u] = d < 3 && k >= 0 && k < P ? x[k] : 0.0f;
    }
    T::load(g, C, p, p1, C, t - 256, sh[b]);
#pragma unroll
    for (int u = 0; u < NQ; u++) {
      const int q = t - 256 + 256 * u, d = q / NX;
      if (d < 3) xs[b][d][q - d * NX] = v[u];
    }
  };
  float s[3] = {};
  const int tr = t / C, c = t - tr * C;  // the thread's row of taps and channel (t < 3 C)
  if (t >= 256 && p0 < p1) load(p0, 0);
  int h = (int)(p0 / W % H), w = (int)(p0 % W), b = 0;
  for (long long p = p0; p < p1; p += R, b ^= 1) {
    __syncthreads();
    if (t >= 256) {
      if (p + R < p1) load(p + R, b ^ 1);
    } else if (t < 3 * C) {
      const int n = (int)min((long long)R, p1 - p);
      const bf16* gv = sh[b] + c;
      const float* xr = xs[b][tr];
      for (int r = 0; r < n; r += 4) {
        if (r + 8 <= n && w >= 1 && w + 8 < W && h + tr >= 1 && h + tr <= H) {  // eight pixels with all taps inside
          const float4 a = *reinterpret_cast<const float4*>(xr + r), e = *reinterpret_cast<const float4*>(xr + r + 4);
          const float2 f = *reinterpret_cast<const float2*>(xr + r + 8);
          const float v[10] = {a.x, a.y, a.z, a.w, e.x, e.y, e.z, e.w, f.x, f.y};
          float gj[8];
#pragma unroll
          for (int j = 0; j < 8; j++) gj[j] = __bfloat162float(gv[(r + j) * C]);
#pragma unroll
          for (int j = 0; j < 8; j++)
#pragma unroll
            for (int d = 0; d < 3; d++) s[d] += v[j + d] * gj[j];
          w += 8;
          r += 4;
          continue;
        }
        for (int j = 0; j < 4 && r + j < n; j++) {
          const float gj = __bfloat162float(gv[(r + j) * C]);
          if (h + tr >= 1 && h + tr <= H)
#pragma unroll
            for (int d = 0; d < 3; d++)
              if (w + d >= 1 && w + d <= W) s[d] += xr[r + j + d] * gj;
          if (++w == W) {
            w = 0;
            if (++h == H) h = 0;
          }
        }
      }
    }
  }
  if (t < 3 * C)
#pragma unroll
    for (int d = 0; d < 3; d++) part[((long long)blockIdx.x * 9 + tr * 3 + d) * C + c] = s[d];
}

// head: 1x1 convolution C -> K (FP32 out)
__global__ void head_fwd_kernel(const bf16* y, int y_cs, int y_co, const float* w /*[C][K]*/, const float* b,
                                long long P, int C, int K, float* out) {
  after_previous();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= P * K) return;
  const long long p = t / K;
  const int k = (int)(t % K);
  float s = b[k];
  for (int c = 0; c < C; c++) s += __bfloat162float(y[p * y_cs + y_co + c]) * w[c * K + k];
  out[t] = s;
}
// the same (K <= 8, C <= 256) with a thread a pixel, which reads its channels
// once, 16 bytes at a time, for all outputs; per output the same order
constexpr int HEAD_C = 256;
__global__ void __launch_bounds__(256) head_fwd8_kernel(const bf16* y, int y_cs, int y_co, const float* w,
                                                        const float* b, long long P, int C, int K, float* out) {
  after_previous();
  __shared__ __align__(16) float sw[HEAD_C][8];
  for (int i = threadIdx.x; i < C * 8; i += 256) sw[i / 8][i % 8] = i % 8 < K ? w[i / 8 * K + i % 8] : 0.0f;
  __syncthreads();
  const long long p = (long long)blockIdx.x * 256 + threadIdx.x;
  if (p >= P) return;
  float s[8];
#pragma unroll
  for (int k = 0; k < 8; k++) s[k] = k < K ? b[k] : 0.0f;
  for (int c0 = 0; c0 < C; c0 += 8) {
    const Vec8 v = load8(y + p * y_cs + y_co + c0);
#pragma unroll
    for (int i = 0; i < 8; i++)
#pragma unroll
      for (int k = 0; k < 8; k++) s[k] += v.v[i] * sw[c0 + i][k];
  }
#pragma unroll
  for (int k = 0; k < 8; k++)
    if (k < K) out[p * K + k] = s[k];
}
// head backward to its input, times GELU'(z): gy[p][c] = gelu'(z[p][c]) sum_k g[p][k] w[c][k]
__global__ void head_dgrad_kernel(const float* g, const float* w, const bf16* z, long long P, int C, int K, bf16* gz) {
  after_previous();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= P * C) return;
  const long long p = t / C;
  const int c = (int)(t % C);
  float s = 0.0f;
  for (int k = 0; k < K; k++) s += g[p * K + k] * w[c * K + k];
  gz[t] = __float2bfloat16_rn(s * gelu_grad(__bfloat162float(z[t])));
}
// head weight and bias gradients: part[b][c][k] and part[b][C][k] over pixel block b
__global__ void head_wgrad_kernel(const bf16* y, int y_cs, int y_co, const float* g, long long P, int C, int K,
                                  long long rows, float* part) {
  after_previous();
  const long long p0 = (long long)blockIdx.x * rows, p1 = p0 + rows < P ? p0 + rows : P;
  for (int q = threadIdx.x; q < (C + 1) * K; q += blockDim.x) {
    const int c = q / K, k = q % K;
    float s = 0.0f;
    for (long long p = p0; p < p1; p++)
      s += (c < C ? __bfloat162float(y[p * y_cs + y_co + c]) : 1.0f) * g[p * K + k];
    part[(long long)blockIdx.x * (C + 1) * K + q] = s;
  }
}

// head backward with 8 channels a thread (K <= 8); per output the same order
__global__ void __launch_bounds__(256) head_dgrad8_kernel(const float* g, const float* w, const bf16* z, long long P,
                                                          int C, int K, bf16* gz) {
  after_previous();
  const unsigned int t = blockIdx.x * 256u + threadIdx.x, cg = (unsigned int)C / 8u;
  const unsigned int p = t / cg, c = 8u * (t % cg);
  if (p >= (unsigned int)P) return;
  Vec8 s = {};
#pragma unroll
  for (int k = 0; k < 8; k++) {
    if (k >= K) break;
    const float gk = g[(long long)p * K + k];
#pragma unroll
    for (int i = 0; i < 8; i++) s.v[i] += gk * __ldg(w + (c + i) * K + k);
  }
  const Vec8 zv = load8(z + (long long)p * C + c);
#pragma unroll
  for (int i = 0; i < 8; i++) s.v[i] = s.v[i] * gelu_grad(zv.v[i]);
  store8(gz + (long long)p * C + c, s);
}
// head_wgrad_kernel's sums with the tiles of RowTile: a thread has one channel
// and three outputs, the next K threads one bias each (C ceil(K/3) + K <= 256,
// K <= 8)
__global__ void __launch_bounds__(512) head_wgrad8_kernel(const bf16* y, int y_cs, int y_co, const float* g,
                                                          long long P, int C, int K, long long rows, float* part) {
  after_previous();
  typedef RowTile<2> T;
  __shared__ __align__(16) bf16 sh[2][T::NE];
  __shared__ __align__(16) float gs[2][9][T::RMAX];  // g[p + r][k] at [k][r]
  const int t = threadIdx.x, R = T::rows(C), ng = (K + 2) / 3;
  const long long p0 = (long long)blockIdx.x * rows, p1 = p0 + rows < P ? p0 + rows : P;
  auto load = [&](long long p, int b) {
    constexpr int NQ = T::RMAX * 8 / 256;
    const int n = (int)min((long long)R, p1 - p) * K;
    float v[NQ];
#pragma unroll
    for (int u = 0; u < NQ; u++) {
      const int q = t - 256 + 256 * u;
      if (q < n) v[u] = g[p * K + q];
    }
    T::load(y + y_co, y_cs, p, p1, C, t - 256, sh[b]);
#pragma unroll
    for (int u = 0; u < NQ; u++) {
      const int q = t - 256 + 256 * u;
      if (q < n) gs[b][q % K][q / K] = v[u];
    }
  };
  float s[3] = {};
  const int kg = t / C, c = t - kg * C;
  const int kb = t - C * ng;  // the bias of threads C ng .. C ng + K - 1
  if (t >= 256 && p0 < p1) load(p0, 0);
  int b = 0;
  for (long long p = p0; p < p1; p += R, b ^= 1) {
    __syncthreads();
    const int n = (int)min((long long)R, p1 - p);
    if (t >= 256) {
      if (p + R < p1) load(p + R, b ^ 1);
    } else if (kb < 0) {
      const bf16* yv = sh[b] + c;
      const float* gk = gs[b][3 * kg];  // rows K .. 8 are not read for an output that counts
      int r = 0;
      for (; r + 4 <= n; r += 4) {
        float v[3][4];
#pragma unroll
        for (int d = 0; d < 3; d++) {
          const float4 a = *reinterpret_cast<const float4*>(gk + d * T::RMAX + r);
          v[d][0] = a.x, v[d][1] = a.y, v[d][2] = a.z, v[d][3] = a.w;
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
          const float yj = __bfloat162float(yv[(r + j) * C]);
#pragma unroll
          for (int d = 0; d < 3; d++) s[d] += yj * v[d][j];
        }
      }
      for (; r < n; r++) {
        const float yj = __bfloat162float(yv[r * C]);
#pragma unroll
        for (int d = 0; d < 3; d++) s[d] += yj * gk[d * T::RMAX + r];
      }
    } else if (kb < K) {
#pragma unroll 16
      for (int r = 0; r < n; r++) s[0] += gs[b][kb][r];
    }
  }
  float* out = part + (long long)blockIdx.x * (C + 1) * K;
  if (kb < 0) {
#pragma unroll
    for (int d = 0; d < 3; d++)
      if (3 * kg + d < K) out[c * K + 3 * kg + d] = s[d];
  } else if (kb < K) {
    out[C * K + kb] = s[0];
  }
}

// 2x2 average pooling of a channel slice
__global__ void pool_kernel(const bf16* x, int x_cs, int x_co, int N, int H, int W, int C, bf16* out) {
  after_previous();
  const int Ho = H / 2, Wo = W / 2;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)N * Ho * Wo * C) return;
  const int c = (int)(t % C);
  const long long q = t / C;
  const int n = (int)(q / ((long long)Ho * Wo)), rem = (int)(q % ((long long)Ho * Wo)), h = rem / Wo, w = rem % Wo;
  float s = 0.0f;
  for (int d = 0; d < 4; d++) {
    const long long p = ((long long)n * H + 2 * h + d / 2) * W + 2 * w + d % 2;
    s += __bfloat162float(x[p * x_cs + x_co + c]);
  }
  out[t] = __float2bfloat16_rn(0.25f * s);
}
// nearest 2x upsampling into a channel slice
__global__ void up_kernel(const bf16* x, int N, int H, int W, int C, bf16* out, int out_cs, int out_co) {
  after_previous();
  const int Ho = 2 * H, Wo = 2 * W;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)N * Ho * Wo * C) return;
  const int c = (int)(t % C);
  const long long q = t / C;
  const int n = (int)(q / ((long long)Ho * Wo)), rem = (int)(q % ((long long)Ho * Wo)), h = rem / Wo, w = rem % Wo;
  out[q * out_cs + out_co + c] = x[(((long long)n * H + h / 2) * W + w / 2) * C + c];
}
// gradient of an encoder output used twice (skip slice of the concatenation
// and input of the pooling): gz = (gcat[p][co + c] + gpool[p/2][c] / 4) gelu'(z)
__global__ void skip_grad_kernel(const bf16* gcat, int gcat_cs, int gcat_co, const bf16* gpool, const bf16* z, int N,
                                 int H, int W, int C, bf16* gz) {
  after_previous();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)N * H * W * C) return;
  const int c = (int)(t % C);
  const long long p = t / C;
  const int n = (int)(p / ((long long)H * W)), rem = (int)(p % ((long long)H * W)), h = rem / W, w = rem % W;
  float s = __bfloat162float(gcat[p * gcat_cs + gcat_co + c]);
  if (gpool) s += 0.25f * __bfloat162float(gpool[(((long long)n * (H / 2) + h / 2) * (W / 2) + w / 2) * C + c]);
  gz[t] = __float2bfloat16_rn(s * gelu_grad(__bfloat162float(z[t])));
}
// upsampling backward (sum of the 4 children of a channel slice) times gelu'(z)
__global__ void up_grad_kernel(const bf16* gcat, int gcat_cs, int gcat_co, const bf16* z, int N, int H, int W, int C,
                               bf16* gz) {
  after_previous();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (long long)N * H * W * C) return;
  const int c = (int)(t % C);
  const long long q = t / C;
  const int n = (int)(q / ((long long)H * W)), rem = (int)(q % ((long long)H * W)), h = rem / W, w = rem % W;
  float s = 0.0f;
  for (int d = 0; d < 4; d++) {
    const long long p = ((long long)n * 2 * H + 2 * h + d / 2) * (2 * W) + 2 * w + d % 2;
    s += __bfloat162float(gcat[p * gcat_cs + gcat_co + c]);
  }
  gz[t] = __float2bfloat16_rn(s * gelu_grad(__bfloat162float(z[t])));
}

// pooling, upsampling and their gradients with 8 channels a thread; each output
// is the one-channel kernels' expression
__global__ void __launch_bounds__(256) pool8_kernel(const bf16* x, int x_cs, int x_co, int N, int H, int W, int C,
                                                    bf16* out) {
  after_previous();
  const unsigned int t = blockIdx.x * 256u + threadIdx.x, cg = (unsigned int)C / 8u, Ho = H / 2, Wo = W / 2;
  const unsigned int q = t / cg, c = 8u * (t % cg);
  if (q >= N * Ho * Wo) return;
  const unsigned int w = q % Wo, hn = q / Wo, h = hn % Ho, n = hn / Ho;
  Vec8 s = {};
#pragma unroll
  for (int d = 0; d < 4; d++) {
    const long long p = ((long long)n * H + 2 * h + d / 2) * W + 2 * w + d % 2;
    const Vec8 v = load8(x + p * x_cs + x_co + c);
#pragma unroll
    for (int i = 0; i < 8; i++) s.v[i] += v.v[i];
  }
#pragma unroll
  for (int i = 0; i < 8; i++) s.v[i] = 0.25f * s.v[i];
  store8(out + (long long)q * C + c, s);
}
__global__ void __launch_bounds__(256) up8_kernel(const bf16* x, int N, int H, int W, int C, bf16* out, int out_cs,
                                                  int out_co) {
  after_previous();
  const unsigned int t = blockIdx.x * 256u + threadIdx.x, cg = (unsigned int)C / 8u;
  const unsigned int q = t / cg, c = 8u * (t % cg);
  if (q >= (unsigned int)(N * H * W)) return;  // an input pixel: read once, written four times
  const unsigned int w = q % (unsigned int)W, hn = q / (unsigned int)W, h = hn % (unsigned int)H, n = hn / (unsigned int)H;
  const uint4 v = *reinterpret_cast<const uint4*>(x + (long long)q * C + c);
#pragma unroll
  for (int d = 0; d < 4; d++) {
    const long long p = ((long long)n * 2 * H + 2 * h + d / 2) * (2 * W) + 2 * w + d % 2;
    *reinterpret_cast<uint4*>(out + p * out_cs + out_co + c) = v;
  }
}
__global__ void __launch_bounds__(256) skip_grad8_kernel(const bf16* gcat, int gcat_cs, int gcat_co, const bf16* gpool,
                                                         const bf16* z, int N, int H, int W, int C, bf16* gz) {
  after_previous();
  const unsigned int t = blockIdx.x * 256u + threadIdx.x, cg = (unsigned int)C / 8u;
  const unsigned int p = t / cg, c = 8u * (t % cg);
  if (p >= (unsigned int)(N * H * W)) return;
  const unsigned int w = p % (unsigned int)W, hn = p / (unsigned int)W, h = hn % (unsigned int)H, n = hn / (unsigned int)H;
  Vec8 s = load8(gcat + (long long)p * gcat_cs + gcat_co + c);
  if (gpool) {
    const Vec8 v = load8(gpool + (((long long)n * (H / 2) + h / 2) * (W / 2) + w / 2) * C + c);
#pragma unroll
    for (int i = 0; i < 8; i++) s.v[i] += 0.25f * v.v[i];
  }
  const Vec8 zv = load8(z + (long long)p * C + c);
#pragma unroll
  for (int i = 0; i < 8; i++) s.v[i] = s.v[i] * gelu_grad(zv.v[i]);
  store8(gz + (long long)p * C + c, s);
}
__global__ void __launch_bounds__(256) up_grad8_kernel(const bf16* gcat, int gcat_cs, int gcat_co, const bf16* z, int N,
                                                       int H, int W, int C, bf16* gz) {
  after_previous();
  const unsigned int t = blockIdx.x * 256u + threadIdx.x, cg = (unsigned int)C / 8u;
  const unsigned int q = t / cg, c = 8u * (t % cg);
  if (q >= (unsigned int)(N * H * W)) return;
  const unsigned int w = q % (unsigned int)W, hn = q / (unsigned int)W, h = hn % (unsigned int)H, n = hn / (unsigned int)H;
  Vec8 s = {};
#pragma unroll
  for (int d = 0; d < 4; d++) {
    const long long p = ((long long)n * 2 * H + 2 * h + d / 2) * (2 * W) + 2 * w + d % 2;
    const Vec8 v = load8(gcat + p * gcat_cs + gcat_co + c);
#pragma unroll
    for (int i = 0; i < 8; i++) s.v[i] += v.v[i];
  }
  const Vec8 zv = load8(z + (long long)q * C + c);
#pragma unroll
  for (int i = 0; i < 8; i++) s.v[i] = s.v[i] * gelu_grad(zv.v[i]);
  store8(gz + (long long)q * C + c, s);
}

// weighted squared error: loss partials per block, gradient dL/dout
__global__ void mse_kernel(const float* out, const float* target, const float* wch, long long P, int K, float scale,
                           float* grad, float* part) {
  after_previous();
  __shared__ float sh[256];
  const long long t0 = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  float s = 0.0f;
  for (long long t = t0; t < P * K; t += (long long)gridDim.x * blockDim.x) {
    const int k = (int)(t % K);
    const float d = out[t] - target[t];
    s += wch[k] * d * d;
    grad[t] = 2.0f * wch[k] * d * scale;
  }
  sh[threadIdx.x] = s;
  __syncthreads();
  for (int o = blockDim.x / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) part[blockIdx.x] = sh[0] * scale;
}

// Adam on FP32 master weights (Kingma and Ba, 2015), bias-corrected step size given
__global__ void adam_kernel(float* w, const float* g, float* m, float* v, long long n, float lr_t, float b1, float b2,
                            float eps) {
  after_previous();
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.0f - b1) * gi;
  const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  w[i] -= lr_t * mi / (sqrtf(vi) + eps);
}

// BF16 weights of a 3x3 layer from FP32 [9][Cin][Cout]: w (same layout) and,
// for the input gradient, wt[tap][co][ci] = w[8 - tap][ci][co]
__global__ void pack_weights_kernel(const float* wf, int Cin, int Cout, bf16* w, bf16* wt) {
  after_previous();
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= 9LL * Cin * Cout) return;
  const int co = (int)(t % Cout);
  const long long q = t / Cout;
  const int ci = (int)(q % Cin), tap = (int)(q / Cin);
  const bf16 b = __float2bfloat16_rn(wf[t]);
  w[t] = b;
  wt[((long long)(8 - tap) * Cout + co) * Cin + ci] = b;
}

}  // namespace unet
}  // namespace clv
