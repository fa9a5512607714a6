// Learned flux closure: an edge-local MLP 24 -> 64 -> 64 -> 2 (GELU) whose two hidden
// layers run on the 5th-generation tensor cores (tcgen05.mma, BF16 operands in shared
// memory, FP32 accumulators in tensor memory), for inference and for training.
//
// There is no closure in the reference; the closure is this library's addition. The MLP reads
// 24 normalized features of an edge and returns two corrections (to the edge mass flux and
// to the edge momentum tendency).
//
// A CTA = 4 warps = 128 threads; a tile = 128 edges, thread t owns row t (TMEM lane t).
// Shared-memory operands use the no-swizzle "core matrix" layout (8 rows x 16 bytes, rows
// 16 bytes apart). A buffer tiled as
//     offset(r, c) = (c / 8) * CHUNK + (r / 8) * 128 + (r % 8) * 16 + (c % 8) * 2
// is a K-major operand with rows r along M/N and columns c along K (SBO = 128, LBO =
// CHUNK), and the same bytes are an MN-major operand with c along M/N and r along K
// (SBO = CHUNK, LBO = 128). Forward GEMMs use the first view, backward GEMMs the second,
// so no operand is ever transposed in memory.
//
// Inference (k_mlp_forward): a persistent grid, several CTAs per SM, 64 TMEM columns each.
//   Z1 = X W1^T + b1   M=128 N=64 K=32  (A = XH[:, 0:32]: X and ones; B = W1 and b1 K-major)
//   H1 = gelu(Z1) -> bf16 -> XH[:, 0:64]  (over X: MMA 1 has finished reading it)
//   Z2 = H1 W2^T + b2  M=128 N=64 K=80  (same TMEM columns: Z1 has been read)
//   H2 = gelu(Z2) -> bf16 -> XH[:, 0:64]
//   Y  = H2 W3^T + b3  M=128 N=16 K=64  (two columns used)
// Training (k_mlp_train): forward, backward and weight gradients of one tile per step, every
// product with a weight or over the rows on the tensor cores:
//   Z1 = X W1^T + b1, H1 = gelu(Z1), gelu'(Z1) -> TMEM (over Z1)
//   Z2 = H1 W2^T + b2, H2 = gelu(Z2), gelu'(Z2) in registers
//   Y  = H2 W3^T (+ b3);  dY = 2 (Y - target) / n, as three BF16 terms each (exact: 24 bits)
//   P  = dY W3           M=128 N=64 K=16   (A = dY K-major, B = W3 transposed)
//   dH2 = P * gelu'(Z2) -> DD[:, 0:64]
//   G  = dH2 W2          M=128 N=64 K=64   (A = DD[:, 0:64] K-major, B = W2 MN-major)
//   dH1 = G * gelu'(Z1) -> DD[:, 64:128]
//   DW += DD^T [H1 | X | 1]  M=128 N=96 K=128 (A = DD MN-major, B = HX MN-major): rows 0..63 x
//         cols 0..63 = dW2, rows 64..127 x cols 64..87 = dW1, column 88 the biases
//   DW3 += [H2 | .]^T dY     M=128 N=16 K=128 (rows 0..63 used)
//   Tensor memory: Z1 then gelu'(Z1) at 0, Z2 then P then G at 64, DW at 128..224, Y at 224, DW3
//   at 240 (256 columns, two CTAs per SM).
// Every tanh is evaluated once, gelu' being kept from the forward pass. What bounds a tile is the
// latency of its seven barrier and tensor-core round trips, two CTAs an SM hiding one another's; at
// the end every CTA adds its sums to the same 5890 addresses. Measured, the kernel alone, back to
// back: 10.3 us for 1000 rows (8 CTAs of one tile), 14.6 for 18944 (148 of one), 22.5 for 37888 (296 of
// one) and 23.5 for 65536 (296, most of two): past one tile's chain the time goes with the CTAs that
// add their sums, hardly with the tiles. A step of 65536 rows (sums cleared, kernel, loss read back,
// Adam) takes 44 us by wall clock from C and 55 from Python; it took 95 to 104 with dW3, the output layer and
// the biases on the CUDA cores and every tanh evaluated twice.
//
// GELU is the tanh form of Hendrycks and Gimpel (2016), gelu(x) = x/2 (1 + tanh(sqrt(2/pi)
// (x + 0.044715 x^3))), with tanh on the special-function unit (tanh.approx.f32); it is the
// network's activation in training and inference alike, and the oracle's.
//
// Every tensor-core wait is bounded in time. A wait that gives up marks the CTA; at the next
// CTA-wide barrier every thread sees the mark and the CTA leaves its tile loop, waits (again
// bounded) for a tensor-core operation it committed and has not seen finish, frees its tensor
// memory and reports TRISK_ERR_TIMEOUT through a status word the host reads.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstddef>
#include <cstring>
#include <memory>

#include "closure_mlp.cuh"
#include "model.hpp"

namespace trisk {
namespace closure {

// Inference: Y (n x 2) = MLP(X) over a persistent grid. expire_tile >= 0 names a tile whose
// first tensor-core operation is not issued, so its bounded wait runs out (the test of the
// give-up path); -1 in normal use.
__global__ void __launch_bounds__(TILE) k_mlp_forward(const __nv_bfloat16* __restrict__ X, int64_t n,
                                                      const ParamsBF16* __restrict__ wbf,
                                                      const Params* __restrict__ p, float* __restrict__ Y,
                                                      Status* status, int64_t expire_tile) {
  extern __shared__ __align__(1024) unsigned char smem[];
  __shared__ __align__(16) InferStatic st;
  const int t = threadIdx.x;
  const int64_t ntiles = (n + TILE - 1) / TILE;
  if ((int64_t)blockIdx.x >= ntiles) return;
  const InferSmem S(smem);
  const uint32_t tmem = infer_setup(S, st, wbf, p);
  MmaWaits waits(smem_u32(S.mbar), &st.abort);
  // row t of tile `tile` (24 features as three 16-byte loads; zeros past the last row)
  auto load_row = [&](int64_t tile, uint4 (&q)[3]) {
    q[0] = q[1] = q[2] = make_uint4(0, 0, 0, 0);
    const int64_t row = tile * TILE + t;
    if (tile < ntiles && row < n) {
      const uint4* src = reinterpret_cast<const uint4*>(X + row * NIN);
      q[0] = __ldcs(src);
      q[1] = __ldcs(src + 1);
      q[2] = __ldcs(src + 2);
    }
  };
  uint4 xq[3];
  load_row(blockIdx.x, xq);
  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int64_t row = tile * TILE + t;
    infer_put_row(S, xq);
    load_row(tile + gridDim.x, xq);  // the next tile's row, in flight during this tile
    float y0, y1;
    if (!infer_tile(S, st, tmem, waits, tile != expire_tile, y0, y1)) break;
    if (row < n) __stcs(reinterpret_cast<float2*>(Y + row * NOUT), make_float2(y0, y1));
  }
  infer_finish(waits, tmem, status);
}

// Training accumulates the gradients of the mean squared error (1/n) sum_rows sum_k
// (y_k - t_k)^2 into grad (FP32, zeroed by the caller) and the squared-error sum into *loss.
// Columns 88..90 of HX (the first padding columns of the input chunk) hold 1 for valid rows: they
// carry b1 into Z1 (and, as a chunk of their own, b2 into Z2), and through the weight-gradient
// MMA column 88 returns the bias gradients: DW[j][88] = db2[j], DW[64 + i][88] = db1[i].
constexpr int ONES_COL = 64 + NIN;
constexpr uint32_t TRAIN_DW = 128, TRAIN_Y = 224, TRAIN_DW3 = 240;

__global__ void __launch_bounds__(TILE, 2) k_mlp_train(const __nv_bfloat16* __restrict__ X, int64_t n,
                                                       const ParamsBF16* __restrict__ wbf,
                                                       const Params* __restrict__ p,
                                                       const float* __restrict__ target, Params* __restrict__ grad,
                                                       float* loss, float inv_n, Status* status) {
  extern __shared__ __align__(1024) unsigned char smem[];
  unsigned char* HX = smem;
  unsigned char* H2 = HX + HX_BYTES;  // directly before DD: dW3's operand reaches into it (unused rows)
  unsigned char* DD = H2 + H2_BYTES;
  unsigned char* DY = DD + DD_BYTES;
  unsigned char* W1s = DY + DY_BYTES;
  unsigned char* W2s = W1s + W1_BYTES;
  unsigned char* B2s = W2s + W2_BYTES;
  unsigned char* W3s = B2s + B2_BYTES;
  unsigned char* W3t = W3s + W3_BYTES;  // 64 units x 16: W3 of output 0 three times, of output 1 three times
  uint64_t* mbar = reinterpret_cast<uint64_t*>(W3t + 2 * W_CHUNK);
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(W3t + 2 * W_CHUNK + 16);
  __shared__ float sb3[NOUT];
  __shared__ int s_abort;

  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  const int64_t ntiles = (n + TILE - 1) / TILE;
  if ((int64_t)blockIdx.x >= ntiles) return;

  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(TRAIN_TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (t == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(mbar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    s_abort = 0;
  }
  load_weights(W1s, W2s, B2s, W3s, wbf, p, t);
  if (t < NH) {
    const uint16_t* w3 = reinterpret_cast<const uint16_t*>(wbf->W3);
    const uint32_t a = w3[t], b = w3[NH + t];
    *reinterpret_cast<uint4*>(W3t + tile_off(t, 0, W_CHUNK)) = make_uint4(a | (a << 16), a | (b << 16), b | (b << 16), 0);
    *reinterpret_cast<uint4*>(W3t + tile_off(t, 8, W_CHUNK)) = make_uint4(0, 0, 0, 0);
  }
  *reinterpret_cast<uint4*>(DY + tile_off(t, 8, HX_CHUNK)) = make_uint4(0, 0, 0, 0);
  if (t < NOUT) sb3[t] = p->b3[t];
  fence_async_smem();
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = *tmem_slot;
  const uint32_t lane_base = tmem + ((uint32_t)(warp * 32) << 16);
  const uint32_t hx = smem_u32(HX), h2 = smem_u32(H2), dd = smem_u32(DD), dy = smem_u32(DY), w1 = smem_u32(W1s),
                 w2 = smem_u32(W2s), b2 = smem_u32(B2s), w3 = smem_u32(W3s), w3t = smem_u32(W3t);
  const uint32_t ID = idesc_bf16(128, 64, 0, 0), ID_G = idesc_bf16(128, 64, 0, 1), ID_DW = idesc_bf16(128, 96, 1, 1),
                 ID_Y = idesc_bf16(128, 16, 0, 0), ID_DW3 = idesc_bf16(128, 16, 1, 1);
  MmaWaits waits(smem_u32(mbar), &s_abort);
  bool first = true;
  float loss_local = 0.0f, gb3[NOUT] = {0.0f, 0.0f};
  auto sync_for_mma = [&]() {  // shared-memory writes -> visible to the tensor core
    fence_async_smem();
    fence_before();
    __syncthreads();
    fence_after();
  };
  auto put32 = [&](unsigned char* base, int c0, const uint32_t* q) {  // 32 BF16 columns of row t
#pragma unroll
    for (int k = 0; k < 4; ++k)
      *reinterpret_cast<uint4*>(base + tile_off(t, c0 + 8 * k, HX_CHUNK)) =
          make_uint4(q[4 * k], q[4 * k + 1], q[4 * k + 2], q[4 * k + 3]);
  };

  for (int64_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const int64_t row = tile * TILE + t;
    const bool valid = row < n;
    float2 want = make_float2(0.0f, 0.0f);
    {  // X -> HX[:, 64:88], the ones of a valid row
      uint4 q[3] = {make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0), make_uint4(0, 0, 0, 0)};
      if (valid) {
        const uint4* src = reinterpret_cast<const uint4*>(X + row * NIN);
        q[0] = src[0];
        q[1] = src[1];
        q[2] = src[2];
        want = make_float2(target[row * NOUT], target[row * NOUT + 1]);
      }
#pragma unroll
      for (int c = 0; c < 3; ++c) *reinterpret_cast<uint4*>(HX + tile_off(t, 64 + 8 * c, HX_CHUNK)) = q[c];
      *reinterpret_cast<uint4*>(HX + tile_off(t, ONES_COL, HX_CHUNK)) = valid ? three_ones() : make_uint4(0, 0, 0, 0);
    }
    sync_for_mma();
    if (waits.aborted()) break;
    if (t == 0) {  // Z1 = X W1^T + b1
#pragma unroll
      for (int kk = 0; kk < 2; ++kk)
        mma_bf16(tmem, sdesc(hx + (8 + 2 * kk) * HX_CHUNK, HX_CHUNK, 128), sdesc(w1 + 2 * kk * W_CHUNK, W_CHUNK, 128),
                 ID, kk);
      mma_commit(waits.mb);
    }
    waits.wait(true);
#pragma unroll
    for (int c = 0; c < 2; ++c) {  // H1 -> HX[:, 0:64], gelu'(Z1) over Z1
      float v[32];
      uint32_t q[16];
      tmem_ld32(lane_base + 32 * c, v);
#pragma unroll
      for (int k = 0; k < 16; ++k) {
        F2 g;
        q[k] = bf16x2(gelu2_of_half(pack2(v[2 * k], v[2 * k + 1]), g));
        unpack2(g, v[2 * k], v[2 * k + 1]);
      }
      put32(HX, 32 * c, q);
      tmem_st32(lane_base + 32 * c, v);
    }
    sync_for_mma();
    if (waits.aborted()) break;
    if (t == 0) {  // Z2 = H1 W2^T + b2
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
        mma_bf16(tmem + 64, sdesc(hx + 2 * kk * HX_CHUNK, HX_CHUNK, 128), sdesc(w2 + 2 * kk * W_CHUNK, W_CHUNK, 128), ID,
                 kk);
      // the ones, and W1's first chunk against zeros
      mma_bf16(tmem + 64, sdesc(hx + 11 * HX_CHUNK, w1 - (hx + 11 * HX_CHUNK), 128), sdesc(b2, W_CHUNK, 128), ID, 1);
      mma_commit(waits.mb);
    }
    waits.wait(true);
    F2 grad2[NH / 2];
#pragma unroll
    for (int c = 0; c < 2; ++c) {  // H2, gelu'(Z2)
      float v[32];
      uint32_t q[16];
      tmem_ld32(lane_base + 64 + 32 * c, v);
#pragma unroll
      for (int k = 0; k < 16; ++k) q[k] = bf16x2(gelu2_of_half(pack2(v[2 * k], v[2 * k + 1]), grad2[16 * c + k]));
      put32(H2, 32 * c, q);
    }
    sync_for_mma();
    if (waits.aborted()) break;
    if (t == 0) {  // Y = H2 W3^T
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
        mma_bf16(tmem + TRAIN_Y, sdesc(h2 + 2 * kk * HX_CHUNK, HX_CHUNK, 128),
                 sdesc(w3 + 2 * kk * W3_CHUNK, W3_CHUNK, 128), ID_Y, kk);
      mma_commit(waits.mb);
    }
    waits.wait(true);
    {
      float y0, y1;
      tmem_ld2(lane_base + TRAIN_Y, y0, y1);
      const float e0 = valid ? y0 + sb3[0] - want.x : 0.0f, e1 = valid ? y1 + sb3[1] - want.y : 0.0f;
      loss_local += e0 * e0;
      loss_local += e1 * e1;
      const float d0 = 2.0f * e0 * inv_n, d1 = 2.0f * e1 * inv_n;
      gb3[0] += d0;
      gb3[1] += d1;
      const uint4 a = split_bf16(d0), b = split_bf16(d1);  // columns 0..2 and 3..5
      *reinterpret_cast<uint4*>(DY + tile_off(t, 0, HX_CHUNK)) =
          make_uint4(a.x, a.y | (b.x << 16), (b.x >> 16) | (b.y << 16), 0);
    }
    sync_for_mma();
    if (waits.aborted()) break;
    if (t == 0) {  // P = dY W3 (over Z2) and DW3 += [H2 | .]^T dY
      mma_bf16(tmem + 64, sdesc(dy, HX_CHUNK, 128), sdesc(w3t, W_CHUNK, 128), ID, 0);
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)
        mma_bf16(tmem + TRAIN_DW3, sdesc(h2 + 2 * kk * 128, 128, HX_CHUNK), sdesc(dy + 2 * kk * 128, 128, HX_CHUNK),
                 ID_DW3, (first && kk == 0) ? 0 : 1);
      mma_commit(waits.mb);
    }
    waits.wait(true);
#pragma unroll
    for (int c = 0; c < 2; ++c) {  // dH2 = P * gelu'(Z2) -> DD[:, 0:64]
      float v[32];
      uint32_t q[16];
      tmem_ld32(lane_base + 64 + 32 * c, v);
#pragma unroll
      for (int k = 0; k < 16; ++k) q[k] = bf16x2(mul2(pack2(v[2 * k], v[2 * k + 1]), grad2[16 * c + k]));
      put32(DD, 32 * c, q);
    }
    sync_for_mma();
    if (waits.aborted()) break;
    if (t == 0) {  // G / 2 = dH2 W2 / 2 (over P; W2s holds W2 / 2)
#pragma unroll
      for (int kk = 0; kk < 4; ++kk)
        mma_bf16(tmem + 64, sdesc(dd + 2 * kk * HX_CHUNK, HX_CHUNK, 128), sdesc(w2 + 2 * kk * 128, 128, W_CHUNK), ID_G,
                 kk);
      mma_commit(waits.mb);
    }
    waits.wait(true);
#pragma unroll
    for (int c = 0; c < 4; ++c) {  // dH1 = G * gelu'(Z1) -> DD[:, 64:128]
      float v[16], g[16];
      uint32_t q[8];
      tmem_ld16(lane_base + 64 + 16 * c, v);
      tmem_ld16(lane_base + 16 * c, g);
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const F2 G = pack2(v[2 * k], v[2 * k + 1]);
        q[k] = bf16x2(mul2(add2(G, G), pack2(g[2 * k], g[2 * k + 1])));
      }
      *reinterpret_cast<uint4*>(DD + tile_off(t, 64 + 16 * c, HX_CHUNK)) = make_uint4(q[0], q[1], q[2], q[3]);
      *reinterpret_cast<uint4*>(DD + tile_off(t, 72 + 16 * c, HX_CHUNK)) = make_uint4(q[4], q[5], q[6], q[7]);
    }
    sync_for_mma();
    if (waits.aborted()) break;
    if (t == 0) {  // DW += DD^T [H1 | X | 1]
#pragma unroll
      for (int kk = 0; kk < 8; ++kk)
        mma_bf16(tmem + TRAIN_DW, sdesc(dd + 2 * kk * 128, 128, HX_CHUNK), sdesc(hx + 2 * kk * 128, 128, HX_CHUNK), ID_DW,
                 (first && kk == 0) ? 0 : 1);
      mma_commit(waits.mb);
    }
    first = false;
    waits.wait(true);
    fence_before();
    __syncthreads();  // the next tile rewrites HX, DD and dY
    fence_after();
    if (waits.aborted()) break;
  }

  waits.drain();
  auto add16 = [](float* to, const float* v) {
#pragma unroll
    for (int k = 0; k < 16; k += 4)
      atomicAdd(reinterpret_cast<float4*>(to + k), make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]));
  };
  if (!waits.aborted() && !first) {  // row t of DW: dW2 and db2 (t < 64) or dW1 and db1
    float v[16], u[16];
    tmem_ld16(lane_base + TRAIN_DW + 80, v);  // columns 80..95: inputs 16..23, then the ones
    if (t < NH) {
      atomicAdd(&grad->b2[t], v[ONES_COL - 80]);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        tmem_ld16(lane_base + TRAIN_DW + 16 * c, u);
        add16(&grad->W2[t * NH + 16 * c], u);
      }
      tmem_ld16(lane_base + TRAIN_DW3, u);  // dW3[o][t]: the sums over dY's three terms
      atomicAdd(&grad->W3[t], u[0] + (u[1] + u[2]));
      atomicAdd(&grad->W3[NH + t], u[3] + (u[4] + u[5]));
    } else {
      float* w = &grad->W1[(t - NH) * NIN];
      atomicAdd(&grad->b1[t - NH], v[ONES_COL - 80]);
      tmem_ld16(lane_base + TRAIN_DW + 64, u);
      add16(w, u);
#pragma unroll
      for (int k = 0; k < 8; k += 4)
        atomicAdd(reinterpret_cast<float4*>(w + 16 + k), make_float4(v[k], v[k + 1], v[k + 2], v[k + 3]));
    }
  }
  float l = loss_local;
#pragma unroll
  for (int s = 16; s > 0; s >>= 1) {
    l += __shfl_xor_sync(0xffffffffu, l, s);
    gb3[0] += __shfl_xor_sync(0xffffffffu, gb3[0], s);
    gb3[1] += __shfl_xor_sync(0xffffffffu, gb3[1], s);
  }
  if (lane == 0) {
    atomicAdd(loss, l);
    if (!waits.aborted()) {
      atomicAdd(&grad->b3[0], gb3[0]);
      atomicAdd(&grad->b3[1], gb3[1]);
    }
  }
  if (waits.aborted() && t == 0) atomicExch(&status->error, 1);
  fence_before();
  __syncthreads();
  fence_after();
  if (warp == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TRAIN_TMEM_COLS)
                 : "memory");
}

// parameter i's BF16 copy
__device__ __forceinline__ void refresh_bf16(ParamsBF16* wbf, int i, float x) {
  const __nv_bfloat16 b = __float2bfloat16_rn(x);
  constexpr int oW2 = offsetof(Params, W2) / 4, ob2 = offsetof(Params, b2) / 4, oW3 = offsetof(Params, W3) / 4;
  if (i < NH * NIN)
    wbf->W1[i / NIN * KIN + i % NIN] = b;
  else if (i >= oW2 && i < ob2)
    wbf->W2[i - oW2] = b;
  else if (i >= oW3 && i < oW3 + NOUT * NH)
    wbf->W3[i - oW3] = b;
}

// Adam on the FP32 master parameters; refreshes the BF16 copies.
__global__ void k_adam(Params* p, const Params* g, Params* m, Params* v, ParamsBF16* wbf, float lr, float beta1,
                       float beta2, float eps, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= NPARAM) return;
  float* P = reinterpret_cast<float*>(p);
  const float* G = reinterpret_cast<const float*>(g);
  float* Mm = reinterpret_cast<float*>(m);
  float* Vv = reinterpret_cast<float*>(v);
  const float gi = G[i];
  const float mi = beta1 * Mm[i] + (1 - beta1) * gi;
  const float vi = beta2 * Vv[i] + (1 - beta2) * gi * gi;
  Mm[i] = mi;
  Vv[i] = vi;
  P[i] -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  refresh_bf16(wbf, i, P[i]);
}

__global__ void k_refresh_bf16(const Params* p, ParamsBF16* wbf) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < NPARAM) refresh_bf16(wbf, i, reinterpret_cast<const float*>(p)[i]);
}

// A training step's sums, in one allocation: cleared and read back in one operation each.
struct LossStatus {
  float loss;  // squared errors
  Status status;
};
struct Sums {
  Params g;  // gradients
  LossStatus end;
};

}  // namespace closure
}  // namespace trisk

using namespace trisk;
using namespace trisk::closure;

// The closure works on the legacy default stream, so it is ordered with the caller's
// default-stream work on the feature and target arrays it reads.
struct TriskClosure {
  int device = 0;
  cudaStream_t stream = cudaStreamLegacy;
  Params* p = nullptr;
  Sums* sums = nullptr;
  Params *g = nullptr, *m = nullptr, *v = nullptr;  // g: sums->g
  ParamsBF16* wbf = nullptr;
  float* loss = nullptr;     // &sums->end.loss
  Status* status = nullptr;  // &sums->end.status
  int64_t adam_step = 0;
  int64_t launches = 0;
  int sms = 0;              // the device's SM count (persistent grids)
  int forward_per_sm = 1;   // resident inference CTAs per SM (the grid's multiple of the SMs)
  int64_t expire_tile = -1;  // test of the bounded wait: see trisk_closure_expire_wait_once
  ~TriskClosure() {
    int prev = -1;
    cudaGetDevice(&prev);
    cudaSetDevice(device);
    cudaStreamSynchronize(stream);
    for (void* q : {(void*)p, (void*)sums, (void*)m, (void*)v, (void*)wbf})
      if (q) cudaFree(q);
    if (prev >= 0) cudaSetDevice(prev);
  }
};

namespace {

TriskClosure* checked_c(TriskClosure* c) {
  if (!c) throw Error(TRISK_ERR_ARGUMENT, "closure is NULL");
  return c;
}

// Waits for the closure's work; the loss of the last gradients call; throws if a wait gave up.
float check_status(TriskClosure& c) {
  LossStatus r{};
  CUDA_CHECK(cudaMemcpyAsync(&r, &c.sums->end, sizeof(r), cudaMemcpyDeviceToHost, c.stream));
  CUDA_CHECK(cudaStreamSynchronize(c.stream));
  if (r.status.error) {
    CUDA_CHECK(cudaMemset(c.status, 0, sizeof(Status)));
    throw Error(TRISK_ERR_TIMEOUT, "a bounded tensor-core wait in the closure MLP gave up");
  }
  return r.loss;
}

// persistent grids: every resident CTA of the device, or one per tile when there are fewer
int mlp_grid(const TriskClosure& c, int64_t n, int per_sm) {
  const int64_t tiles = (n + TILE - 1) / TILE;
  return (int)std::max<int64_t>(1, std::min<int64_t>(tiles, (int64_t)c.sms * per_sm));
}

void launch_forward(TriskClosure& c, const __nv_bfloat16* X, int64_t n, float* Y, cudaStream_t stream) {
  if (n == 0) return;
  const int64_t expire = c.expire_tile;
  c.expire_tile = -1;
  k_mlp_forward<<<mlp_grid(c, n, c.forward_per_sm), TILE, FWD_SMEM_BYTES, stream>>>(X, n, c.wbf, c.p, Y, c.status,
                                                                                     expire);
  CUDA_CHECK(cudaGetLastError());
  c.launches++;
}

void launch_train(TriskClosure& c, const __nv_bfloat16* X, int64_t n, const float* target, float inv_n) {
  if (n == 0) return;
  k_mlp_train<<<mlp_grid(c, n, 2), TILE, SMEM_BYTES, c.stream>>>(X, n, c.wbf, c.p, target, c.g, c.loss, inv_n,
                                                                 c.status);
  CUDA_CHECK(cudaGetLastError());
  c.launches++;
}

}  // namespace

namespace trisk {

namespace closure {

void closure_device_params(TriskClosure* c, const ParamsBF16** wbf, const Params** p, Status** status) {
  *wbf = c->wbf;
  *p = c->p;
  *status = c->status;
}

int infer_ctas_per_sm(const void* kernel, int device) {
  // all of the unified L1/shared storage as shared memory, so that several CTAs fit an SM
  CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, FWD_SMEM_BYTES));
  CUDA_CHECK(cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout,
                                  cudaSharedmemCarveoutMaxShared));
  // From the kernel's resources: shared memory (dynamic, static and the per-CTA reservation),
  // registers (allocated per warp in units of 256), threads, and tensor memory (512 columns).
  // The runtime's occupancy query reports one CTA for these kernels, which would leave most of
  // each SM idle, so it is not used.
  cudaFuncAttributes fa{};
  CUDA_CHECK(cudaFuncGetAttributes(&fa, kernel));
  int smem_sm = 0, reserved = 0, regs_sm = 0, threads_sm = 0;
  CUDA_CHECK(cudaDeviceGetAttribute(&smem_sm, cudaDevAttrMaxSharedMemoryPerMultiprocessor, device));
  CUDA_CHECK(cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, device));
  CUDA_CHECK(cudaDeviceGetAttribute(&regs_sm, cudaDevAttrMaxRegistersPerMultiprocessor, device));
  CUDA_CHECK(cudaDeviceGetAttribute(&threads_sm, cudaDevAttrMaxThreadsPerMultiProcessor, device));
  const int by_smem = smem_sm / (FWD_SMEM_BYTES + (int)fa.sharedSizeBytes + reserved);
  const int warp_regs = ((fa.numRegs * 32 + 255) / 256) * 256;
  const int by_regs = regs_sm / std::max(1, warp_regs * (TILE / 32));
  const int by_threads = threads_sm / TILE;
  const int per_sm = std::min(std::min(by_smem, by_regs), std::min(by_threads, 512 / (int)FWD_TMEM_COLS));
  return std::max(1, per_sm);
}

}  // namespace closure

void closure_forward_on(TriskClosure* c, const void* X, int64_t n, float* Y, cudaStream_t stream) {
  launch_forward(*c, static_cast<const __nv_bfloat16*>(X), n, Y, stream);
}

void closure_check(TriskClosure* c) { check_status(*c); }

int closure_device(const TriskClosure* c) { return c->device; }

}  // namespace trisk

extern "C" {

int trisk_closure_create(int32_t device, const float* params, TriskClosure** out) {
  TRISK_API_BEGIN
  if (!out) throw Error(TRISK_ERR_ARGUMENT, "NULL argument");
  *out = nullptr;
  auto c = std::make_unique<TriskClosure>();
  c->device = device;
  DeviceGuard guard(device);
  CUDA_CHECK(cudaMalloc(&c->p, sizeof(Params)));
  CUDA_CHECK(cudaMalloc(&c->sums, sizeof(Sums)));
  c->g = &c->sums->g;
  c->loss = &c->sums->end.loss;
  c->status = &c->sums->end.status;
  CUDA_CHECK(cudaMalloc(&c->m, sizeof(Params)));
  CUDA_CHECK(cudaMalloc(&c->v, sizeof(Params)));
  CUDA_CHECK(cudaMalloc(&c->wbf, sizeof(ParamsBF16)));
  CUDA_CHECK(cudaMemset(c->m, 0, sizeof(Params)));
  CUDA_CHECK(cudaMemset(c->v, 0, sizeof(Params)));
  CUDA_CHECK(cudaMemset(c->sums, 0, sizeof(Sums)));
  CUDA_CHECK(cudaMemset(c->wbf, 0, sizeof(ParamsBF16)));  // W1's padding
  if (params) CUDA_CHECK(cudaMemcpy(c->p, params, sizeof(Params), cudaMemcpyHostToDevice));
  else CUDA_CHECK(cudaMemset(c->p, 0, sizeof(Params)));
  k_refresh_bf16<<<(NPARAM + 255) / 256, 256, 0, c->stream>>>(c->p, c->wbf);
  CUDA_CHECK(cudaGetLastError());
  CUDA_CHECK(cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES));
  CUDA_CHECK(cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributePreferredSharedMemoryCarveout,
                                  cudaSharedmemCarveoutMaxShared));
  int sms = 0;
  CUDA_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
  c->sms = sms;
  c->forward_per_sm = infer_ctas_per_sm(reinterpret_cast<const void*>(k_mlp_forward), device);
  CUDA_CHECK(cudaStreamSynchronize(c->stream));
  *out = c.release();
  TRISK_API_END
}

void trisk_closure_destroy(TriskClosure* c) { delete c; }

int32_t trisk_closure_param_count(void) { return NPARAM; }

int trisk_closure_get_params(TriskClosure* closure, float* params) {
  TRISK_API_BEGIN
  TriskClosure& c = *checked_c(closure);
  if (!params) throw Error(TRISK_ERR_ARGUMENT, "NULL argument");
  DeviceGuard guard(c.device);
  CUDA_CHECK(cudaMemcpyAsync(params, c.p, sizeof(Params), cudaMemcpyDeviceToHost, c.stream));
  CUDA_CHECK(cudaStreamSynchronize(c.stream));
  TRISK_API_END
}

int trisk_closure_set_params(TriskClosure* closure, const float* params) {
  TRISK_API_BEGIN
  TriskClosure& c = *checked_c(closure);
  if (!params) throw Error(TRISK_ERR_ARGUMENT, "NULL argument");
  DeviceGuard guard(c.device);
  CUDA_CHECK(cudaMemcpyAsync(c.p, params, sizeof(Params), cudaMemcpyHostToDevice, c.stream));
  k_refresh_bf16<<<(NPARAM + 255) / 256, 256, 0, c.stream>>>(c.p, c.wbf);
  CUDA_CHECK(cudaGetLastError());
  CUDA_CHECK(cudaStreamSynchronize(c.stream));
  TRISK_API_END
}

// Y (n x 2, FP32) = MLP(X) for X (n x 24, BF16), all device pointers.
int trisk_closure_forward(TriskClosure* closure, const void* X, int64_t n, float* Y) {
  TRISK_API_BEGIN
  TriskClosure& c = *checked_c(closure);
  if (!X || !Y || n < 0) throw Error(TRISK_ERR_ARGUMENT, "bad argument");
  DeviceGuard guard(c.device);
  launch_forward(c, static_cast<const __nv_bfloat16*>(X), n, Y, c.stream);
  check_status(c);
  TRISK_API_END
}

// Gradients (FP32, same layout as the parameters) of the mean squared error over the batch
// and the loss; grads may be NULL (then kept on the device for trisk_closure_adam).
int trisk_closure_gradients(TriskClosure* closure, const void* X, const float* target, int64_t n, float* grads,
                            float* loss) {
  TRISK_API_BEGIN
  TriskClosure& c = *checked_c(closure);
  if (!X || !target || n <= 0) throw Error(TRISK_ERR_ARGUMENT, "bad argument");
  DeviceGuard guard(c.device);
  CUDA_CHECK(cudaMemsetAsync(c.sums, 0, offsetof(Sums, end) + offsetof(LossStatus, status), c.stream));  // the status stays until it is read
  launch_train(c, static_cast<const __nv_bfloat16*>(X), n, target, 1.0f / (float)n);
  if (grads) CUDA_CHECK(cudaMemcpyAsync(grads, c.g, sizeof(Params), cudaMemcpyDeviceToHost, c.stream));
  const float l = check_status(c);
  if (loss) *loss = l / (float)n;
  TRISK_API_END
}

// One Adam step with the gradients left by the last trisk_closure_gradients call.
int trisk_closure_adam(TriskClosure* closure, float lr, float beta1, float beta2, float eps) {
  TRISK_API_BEGIN
  TriskClosure& c = *checked_c(closure);
  DeviceGuard guard(c.device);
  c.adam_step++;
  const float c1 = 1.0f - powf(beta1, (float)c.adam_step), c2 = 1.0f - powf(beta2, (float)c.adam_step);
  k_adam<<<(NPARAM + 255) / 256, 256, 0, c.stream>>>(c.p, c.g, c.m, c.v, c.wbf, lr, beta1, beta2, eps, c1, c2);
  CUDA_CHECK(cudaGetLastError());
  c.launches++;
  TRISK_API_END
}

int trisk_closure_synchronize(TriskClosure* closure) {
  TRISK_API_BEGIN
  TriskClosure& c = *checked_c(closure);
  DeviceGuard guard(c.device);
  check_status(c);
  TRISK_API_END
}

// Launch shape of the inference kernel: CTAs per SM of its persistent grid, and SMs.
int trisk_closure_info(TriskClosure* closure, int32_t* forward_ctas_per_sm, int32_t* sms) {
  TRISK_API_BEGIN
  TriskClosure& c = *checked_c(closure);
  if (forward_ctas_per_sm) *forward_ctas_per_sm = c.forward_per_sm;
  if (sms) *sms = c.sms;
  TRISK_API_END
}

// Test of the bounded tensor-core wait: the next inference launch of this closure leaves the
// first tensor-core operation of `tile` un-issued, so that tile's wait runs out (after half a
// second) and the call reports TRISK_ERR_TIMEOUT; later calls are unaffected.
int trisk_closure_expire_wait_once(TriskClosure* closure, int64_t tile) {
  TRISK_API_BEGIN
  TriskClosure& c = *checked_c(closure);
  if (tile < 0) throw Error(TRISK_ERR_ARGUMENT, "tile must be >= 0");
  c.expire_tile = tile;
  TRISK_API_END
}

int trisk_closure_stream(TriskClosure* closure, void** stream) {
  TRISK_API_BEGIN
  TriskClosure& c = *checked_c(closure);
  if (!stream) throw Error(TRISK_ERR_ARGUMENT, "NULL argument");
  *stream = (void*)c.stream;
  TRISK_API_END
}

}  // extern "C"
