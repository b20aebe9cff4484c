// Forward pass of the learned proposal's network in one kernel: a CTA takes 128 candidates
// through all four layers, the activations staying in shared memory and TMEM.
//
// Layer by layer through HBM, 100,000 candidates of six cameras took 587 us: 244 us to turn
// the f32 inputs into padded bf16 rows, three GEMMs of about 100 us that wrote and re-read
// the activations, 43 us for the head.  Here the inputs are read once (296 MB, 45 us at the
// measured copy rate) and 1.6 MB of results written; what bounds it is the issue of the
// 98,304 erf evaluations of a tile (about 14 us a tile, 5.3 tiles an SM), so two CTAs share
// an SM, one loading and multiplying while the other is in an epilogue.
//
// Shared memory (112 KB a CTA): R = 48 KB, H = 64 KB.
//   layer 1: K slices of 64: A (128 x 64 bf16, written by all threads from the f32 or bf16
//            input rows) and W1 (256 x 64, TMA) in two stages, R and the first 48 KB of H;
//   layers 2, 3: A = the activations in H (four 128 x 64 slabs), W2 / W3 in 16 KB pieces
//            (128 x 64, TMA) through three slots in R, loaded ahead of the epilogues;
//   head: the third activations in H, one warp a row, summed as head_fwd_kernel does.
// All operand tiles are K-major with the 128-byte swizzle.  The accumulator (128 x 256 f32)
// takes 256 TMEM columns.  Warp 0 lane 0 issues the MMAs, warp 1 lane 0 the TMA loads; every
// wait is bounded and reports through *err, after which the CTA still runs to its end.
#include <cuda.h>
#include <cudaTypedefs.h>

#include "olpt_ctx.cuh"
#include "olpt_gemm.h"
#include "olpt_mlp.h"
#include "olpt_umma.cuh"

namespace olpt {
namespace {

constexpr int kRows = 128, kThreads = 256;
constexpr uint32_t kABytes = kRows * 64 * 2, kB1Bytes = kMlpHid * 64 * 2, kPiece = 128 * 64 * 2;
constexpr uint32_t kR = kABytes + kB1Bytes, kH = kRows * kMlpHid * 2;
constexpr uint32_t kBars = 16;
constexpr size_t kSmem = kR + kH + kBars * 8 + 16;
constexpr int kPieces = 16;  // of W2 and W3: K slice q / 2 % 4, output half q % 2

struct FusedArgs {
  const void* x;  // f32 rows of `in`, or bf16 rows of in_pad
  int64_t n;
  int in, in_pad;
  const float *b1, *b2, *b3, *w4, *b4;
  float* o;
  int* err;
};

// byte offset of 16-byte chunk c of row r in a 128-byte-swizzled tile of 64-element rows
__device__ __forceinline__ uint32_t swz(int r, int c) {
  return (uint32_t)r * 128u + (uint32_t)((c ^ (r & 7)) << 4);
}

__device__ __forceinline__ void fence_async_smem() {
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

template <bool F32>
__global__ void __launch_bounds__(kThreads, 2)
    mlp_fused_kernel(const __grid_constant__ CUtensorMap tm1, const __grid_constant__ CUtensorMap tm2,
                     const __grid_constant__ CUtensorMap tm3, FusedArgs g) {
  using namespace umma;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint8_t* R = smem;
  uint8_t* H = smem + kR;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kR + kH);
  uint64_t *full1 = bars, *empty1 = bars + 2, *full2 = bars + 4, *empty2 = bars + 7;
  uint64_t* done = bars + 10;  // one per layer
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + kBars);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t row0 = (int64_t)blockIdx.x * kRows;
  const int rows = (int)min((int64_t)kRows, g.n - row0);
  const int slices = g.in_pad / 64;
  const bool mma_thread = tid == 0, tma_thread = tid == 32;

  if (smem_u32(smem) & 1023u) {  // the swizzle needs it; the same in every thread
    if (tid == 0) atomicOr(g.err, 64);
    return;
  }
  if (tid == 0) {
    for (int i = 0; i < 13; ++i) mbar_init(bars + i, 1);
    fence_barrier_init();
  }
  __syncwarp();
  if (warp == 0) tmem_alloc(tmem_slot, kMlpHid);
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
  const uint32_t tmem = *tmem_slot;
  auto stage = [&](int s) { return s ? H : R; };  // layer-1 stage: A, then W1
  auto wait = [&](uint64_t* bar, uint32_t parity, int code) {
    if (!mbar_wait(bar, parity)) atomicOr(g.err, code);
  };

  // ---- layer 1: the input rows, 64 columns at a time, through registers
  constexpr int kReg = F32 ? 32 : 4;
  float xr[F32 ? kReg : 1];
  uint4 xq[F32 ? 1 : kReg];
  auto fetch = [&](int s) {
    if constexpr (F32) {
      // warp w: rows w, w + 8, ..; lane: columns lane and lane + 32 of the slice
      const float* x = static_cast<const float*>(g.x);
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const int r = warp + 8 * q;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c = 64 * s + 32 * h + lane;
          xr[2 * q + h] = r < rows && c < g.in ? __ldg(x + (row0 + r) * g.in + c) : 0.0f;
        }
      }
    } else {
      const uint4* x = static_cast<const uint4*>(g.x);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int r = (tid >> 3) + 32 * q, c = tid & 7;
        xq[q] = r < rows ? __ldg(x + (row0 + r) * (g.in_pad / 8) + 8 * s + c)
                         : make_uint4(0, 0, 0, 0);
      }
    }
  };
  auto store = [&](uint8_t* A) {
    if constexpr (F32) {
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const int r = warp + 8 * q;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          const int c = 32 * h + lane;
          *reinterpret_cast<__nv_bfloat16*>(A + swz(r, c >> 3) + 2 * (c & 7)) =
              __float2bfloat16_rn(xr[2 * q + h]);
        }
      }
    } else {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        *reinterpret_cast<uint4*>(A + swz((tid >> 3) + 32 * q, tid & 7)) = xq[q];
    }
  };
  auto load_w1 = [&](int s) {
    uint64_t* bar = &full1[s & 1];
    mbar_arrive_expect_tx(bar, kB1Bytes);
    tma_load_2d(stage(s & 1) + kABytes, &tm1, bar, s * 64, 0);
  };
  auto load_piece = [&](int q) {
    const int slot = q % 3;
    mbar_arrive_expect_tx(&full2[slot], kPiece);
    tma_load_2d(R + slot * kPiece, q < 8 ? &tm2 : &tm3, &full2[slot], (q >> 1 & 3) * 64,
                (q & 1) * 128);
  };
  if (tma_thread) load_w1(0);
  fetch(0);
  for (int s = 0; s < slices; ++s) {
    // stage s & 1 was last read by the MMAs of slice s - 2
    if (s >= 2) wait(&empty1[s & 1], (uint32_t)(s / 2 - 1) & 1u, 1);
    store(stage(s & 1));
    if (s + 1 < slices) fetch(s + 1);
    fence_async_smem();
    __syncthreads();
    if (mma_thread) {
      wait(&full1[s & 1], (uint32_t)(s / 2) & 1u, 2);
      fence_after_sync();
      const uint64_t ad = sw128_desc(smem_u32(stage(s & 1)));
      const uint64_t bd = sw128_desc(smem_u32(stage(s & 1) + kABytes));
#pragma unroll
      for (int k = 0; k < 4; ++k)
        mma_bf16(tmem, ad + 2 * k, bd + 2 * k, idesc_bf16(kRows, kMlpHid), s > 0 || k > 0);
      mma_commit(&empty1[s & 1]);
      if (s == slices - 1) mma_commit(&done[0]);
    }
    if (tma_thread && s + 1 < slices) {
      if (s >= 1) wait(&empty1[(s + 1) & 1], (uint32_t)((s + 1) / 2 - 1) & 1u, 4);
      load_w1(s + 1);
    }
  }

  // ---- layers 1 .. 3: bias, GELU, bf16 activations into H; the next layer's MMAs
  const int quarter = warp & 3, half = warp >> 2;
  const int row = quarter * 32 + lane;
  int q_next = 0;  // tma_thread: next weight piece
#pragma unroll 1
  for (int layer = 0; layer < 3; ++layer) {
    wait(&done[layer], 0, 8);
    fence_after_sync();
    if (tma_thread && layer == 0)  // R is free: weights load while the epilogue runs
      for (; q_next < 3; ++q_next) load_piece(q_next);
    __syncwarp();
    const float* bias = layer == 0 ? g.b1 : layer == 1 ? g.b2 : g.b3;
#pragma unroll 1
    for (int c = half * 128; c < half * 128 + 128; c += 16) {
      float v[16];
      tmem_ld16(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c, v);
      uint32_t w[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const float a = gelu_f(v[2 * k] + __ldg(bias + c + 2 * k));
        const float b = gelu_f(v[2 * k + 1] + __ldg(bias + c + 2 * k + 1));
        const __nv_bfloat162 p = __floats2bfloat162_rn(a, b);
        w[k] = *reinterpret_cast<const uint32_t*>(&p);
      }
      uint8_t* slab = H + (c >> 6) * kABytes;
      const int ch = (c & 63) >> 3;
      *reinterpret_cast<uint4*>(slab + swz(row, ch)) = make_uint4(w[0], w[1], w[2], w[3]);
      *reinterpret_cast<uint4*>(slab + swz(row, ch + 1)) = make_uint4(w[4], w[5], w[6], w[7]);
    }
    fence_async_smem();
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    if (layer == 2) break;
    if (mma_thread) {
      for (int q = 8 * layer; q < 8 * layer + 8; ++q) {
        const int slot = q % 3;
        wait(&full2[slot], (uint32_t)(q / 3) & 1u, 16);
        fence_after_sync();
        const uint64_t ad = sw128_desc(smem_u32(H + (q >> 1 & 3) * kABytes));
        const uint64_t bd = sw128_desc(smem_u32(R + slot * kPiece));
#pragma unroll
        for (int k = 0; k < 4; ++k)
          mma_bf16(tmem + (q & 1) * 128, ad + 2 * k, bd + 2 * k, idesc_bf16(kRows, 128),
                   (q >> 1 & 3) > 0 || k > 0);
        mma_commit(&empty2[slot]);
      }
      mma_commit(&done[layer + 1]);
    }
    if (tma_thread)
      for (const int end = layer == 0 ? 11 : kPieces; q_next < end; ++q_next) {
        wait(&empty2[q_next % 3], (uint32_t)(q_next / 3 - 1) & 1u, 32);
        load_piece(q_next);
      }
    __syncwarp();
  }

  // ---- head: one warp a row
  {
    float w4[kMlpOut][8];
#pragma unroll
    for (int j = 0; j < kMlpOut; ++j)
#pragma unroll
      for (int m = 0; m < 8; ++m) w4[j][m] = __ldg(g.w4 + j * kMlpHid + lane + 32 * m);
    const float b4 = lane < kMlpOut ? g.b4[lane] : 0.0f;
    for (int r = warp; r < rows; r += 8) {
      float acc[kMlpOut] = {0, 0, 0, 0};
#pragma unroll
      for (int m = 0; m < 8; ++m) {
        const int c = lane + 32 * m;
        const float h = __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(
            H + (c >> 6) * kABytes + swz(r, (c & 63) >> 3) + 2 * (c & 7)));
#pragma unroll
        for (int j = 0; j < kMlpOut; ++j) acc[j] += h * w4[j][m];
      }
#pragma unroll
      for (int j = 0; j < kMlpOut; ++j)
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc[j] += __shfl_xor_sync(0xffffffffu, acc[j], o);
      const float v = lane == 0 ? acc[0] : lane == 1 ? acc[1] : lane == 2 ? acc[2] : acc[3];
      if (lane < kMlpOut) g.o[(row0 + r) * kMlpOut + lane] = v + b4;
    }
  }
  __syncwarp();
  fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, kMlpHid);
}

CUtensorMap weight_map(const __nv_bfloat16* w, int cols, int box_rows) {
  CUtensorMap m;
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)kMlpHid};
  const cuuint64_t strides[1] = {(cuuint64_t)cols * 2};
  const cuuint32_t box[2] = {64, (cuuint32_t)box_rows};
  const cuuint32_t estr[2] = {1, 1};
  const CUresult r = tensor_map_encoder()(
      &m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (void*)w, dims, strides, box, estr,
      CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
      CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  OLPT_REQUIRE(r == CUDA_SUCCESS, OLPT_ERR_CUDA,
               "cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
  return m;
}

template <bool F32>
void launch(MlpWork& W, const FusedArgs& g, cudaStream_t s) {
  const CUtensorMap t1 = weight_map(W.wb1.as<__nv_bfloat16>(), W.dims.in_pad, kMlpHid);
  const CUtensorMap t2 = weight_map(W.wb2.as<__nv_bfloat16>(), kMlpHid, 128);
  const CUtensorMap t3 = weight_map(W.wb3.as<__nv_bfloat16>(), kMlpHid, 128);
  OLPT_CUDA(cudaFuncSetAttribute(mlp_fused_kernel<F32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)kSmem));
  const unsigned grid = (unsigned)((g.n + kRows - 1) / kRows);
  mlp_fused_kernel<F32><<<OLPT_G(grid), kThreads, kSmem, s>>>(t1, t2, t3, g);
  OLPT_CUDA(cudaGetLastError());
}

}  // namespace

void mlp_fused_forward(olpt_ctx* ctx, const float* x_f32, const __nv_bfloat16* x, int64_t n,
                       float* o) {
  MlpWork& W = ctx->mlp;
  const MlpDims& D = W.dims;
  const float* M = W.master.as<float>();
  FusedArgs g{};
  g.x = x_f32 ? (const void*)x_f32 : (const void*)x;
  g.n = n;
  g.in = D.in;
  g.in_pad = D.in_pad;
  g.b1 = M + D.off_b1;
  g.b2 = M + D.off_b2;
  g.b3 = M + D.off_b3;
  g.w4 = M + D.off_w4;
  g.b4 = M + D.off_b4;
  g.o = o;
  g.err = W.err.as<int>();
  if (x_f32)
    launch<true>(W, g, ctx->stream);
  else
    launch<false>(W, g, ctx->stream);
}

}  // namespace olpt
