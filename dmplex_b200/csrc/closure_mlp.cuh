// Device side of the closure network shared by its own kernels (closure.cu) and the fused
// feature + network + correction kernel of the ensembles (ensemble.cu): the tcgen05 helpers,
// the no-swizzle operand layout, the bounded waits, GELU, and the inference of one 128-row
// tile whose inputs are in shared memory. The layout, the tensor-memory use and the waits
// are described at the top of closure.cu.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <memory>

#include "model.hpp"

struct TriskClosure;

namespace trisk {
namespace closure {

constexpr int NIN = 24, KIN = 32, NH = 64, NOUT = 2, TILE = 128;
constexpr int HX_CHUNK = TILE * 16;  // 2048 B: one 8-column chunk of a 128-row tile
constexpr int W_CHUNK = NH * 16;     // 1024 B: one 8-column chunk of a 64-row weight
constexpr int HX_BYTES = 12 * HX_CHUNK;  // 96 columns: H1 (0..63) | X (64..95)
constexpr int DD_BYTES = 16 * HX_CHUNK;  // 128 columns: dH2 (0..63) | dH1 (64..127)
constexpr int W1_BYTES = 4 * W_CHUNK;    // 64 x 32
constexpr int W2_BYTES = 8 * W_CHUNK;    // 64 x 64
constexpr uint32_t TRAIN_TMEM_COLS = 256;  // two CTAs per SM share its 512 columns
// Inference: a chunk of ones, XH (X, then H1, then H2: 8 chunks), W1, W2, b2, W3 and the barrier, 64
// TMEM columns; six CTAs fit an SM's shared memory, and eight x 64 columns fit its TMEM, so no CTA
// ever waits in tcgen05.alloc.
constexpr int XH_BYTES = 8 * HX_CHUNK;
constexpr int B2_BYTES = 2 * W_CHUNK;  // 64 x 16
constexpr int W3_CHUNK = 16 * 16;      // one 8-column chunk of the 16-row (two used) output weight
constexpr int W3_BYTES = 8 * W3_CHUNK;
constexpr int FWD_SMEM_BYTES = HX_CHUNK + XH_BYTES + W1_BYTES + W2_BYTES + B2_BYTES + W3_BYTES + 64;
constexpr uint32_t FWD_TMEM_COLS = 64;
static_assert(FWD_SMEM_BYTES * 6 <= 220 * 1024, "six inference CTAs per SM");
// Training: HX, H2 (8 chunks), DD, dY (2 chunks), W1, W2, b2, W3 in both orders and the barrier.
constexpr int H2_BYTES = 8 * HX_CHUNK, DY_BYTES = 2 * HX_CHUNK;
constexpr int SMEM_BYTES =
    HX_BYTES + H2_BYTES + DD_BYTES + DY_BYTES + W1_BYTES + W2_BYTES + B2_BYTES + W3_BYTES + 2 * W_CHUNK + 64;
static_assert(SMEM_BYTES * 2 <= 220 * 1024, "two training CTAs per SM");
// A bounded tensor-core wait gives up after this long (the operations take microseconds).
constexpr long long MBAR_WAIT_NS = 500000000LL;

// FP32 master parameters and their BF16 tensor-core copies (one contiguous block each).
struct Params {
  float W1[NH * NIN], b1[NH], W2[NH * NH], b2[NH], W3[NOUT * NH], b3[NOUT];
};
constexpr int NPARAM = sizeof(Params) / sizeof(float);
struct ParamsBF16 {
  __nv_bfloat16 W1[NH * KIN];  // padded to 32 inputs
  __nv_bfloat16 W2[NH * NH];
  __nv_bfloat16 W3[NOUT * NH];
};

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// no-swizzle shared-memory matrix descriptor (sm100 layout: version 1 at bit 46)
__device__ __forceinline__ uint64_t sdesc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | (1ull << 46);
}

// instruction descriptor of kind::f16 with BF16 operands and an FP32 accumulator
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N, int a_mn, int b_mn) {
  return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)a_mn << 15) | ((uint32_t)b_mn << 16) |
         ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, int accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}\n" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}

__device__ __forceinline__ void mma_commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
               : "memory");
}

__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ long long global_ns() {
  long long t;
  asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
  return t;
}

// Waits for the completion of the mbarrier phase of parity `phase`, for at most MBAR_WAIT_NS
// and at most MBAR_WAIT_TRIES polls (a backstop that the clock always beats: a poll takes more
// than a nanosecond); false if it gave up.
constexpr uint32_t MBAR_WAIT_TRIES = 1u << 31;
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t phase) {
  long long start = 0;
  for (uint32_t i = 0; i < MBAR_WAIT_TRIES; ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(mbar), "r"(phase)
        : "memory");
    if (done) return true;
    if ((i & 255) == 0) {
      const long long now = global_ns();
      if (i == 0) start = now;
      else if (now - start > MBAR_WAIT_NS) return false;
    }
  }
  return false;
}

// 16 consecutive FP32 columns of this thread's TMEM lane
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int k = 0; k < 16; ++k) v[k] = __uint_as_float(r[k]);
}

// 32 consecutive columns
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
      "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int k = 0; k < 32; ++k) v[k] = __uint_as_float(r[k]);
}
// 32 consecutive columns of this thread's lane written (complete on return)
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const float* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,"
      "%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
      "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]), "f"(v[9]),
      "f"(v[10]), "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15]), "f"(v[16]), "f"(v[17]), "f"(v[18]),
      "f"(v[19]), "f"(v[20]), "f"(v[21]), "f"(v[22]), "f"(v[23]), "f"(v[24]), "f"(v[25]), "f"(v[26]), "f"(v[27]),
      "f"(v[28]), "f"(v[29]), "f"(v[30]), "f"(v[31])
      : "memory");
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}
// two
__device__ __forceinline__ void tmem_ld2(uint32_t taddr, float& a, float& b) {
  uint32_t r[2];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x2.b32 {%0,%1}, [%2];" : "=r"(r[0]), "=r"(r[1]) : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
  a = __uint_as_float(r[0]);
  b = __uint_as_float(r[1]);
}

__device__ __forceinline__ float tanh_approx(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
// gelu(x) = x/2 (1 + tanh(u)), u = sqrt(2/pi) (x + 0.044715 x^3) (Hendrycks and Gimpel 2016)
constexpr float GELU_C0 = 0.7978845608028654f;   // sqrt(2/pi)
constexpr float GELU_C1 = 0.035677408136300125f;  // 0.044715 sqrt(2/pi)
// Two FP32 values at once (Blackwell's packed instructions, each half rounded as the scalar one):
// half the issue slots, which the epilogues of the network run out of.
struct F2 {
  unsigned long long v;
};
__device__ __forceinline__ F2 pack2(float a, float b) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b));
  return r;
}
__device__ __forceinline__ void unpack2(F2 x, float& a, float& b) {
  asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v));
}
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
  return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
  return r;
}
__device__ __forceinline__ F2 tanh2(F2 x) {
  float a, b;
  unpack2(x, a, b);
  return pack2(tanh_approx(a), tanh_approx(b));
}
// gelu(2h) of both halves: x/2 is h itself, and u = x (C0 + C1 x^2) = h (2 C0 + 8 C1 h^2), scaled by
// powers of two throughout. The caller halves the weights and biases that form x (exact in
// binary), which saves the multiplication by 1/2.
__device__ __forceinline__ F2 gelu2_of_half(F2 h) {
  const F2 u = mul2(h, fma2(pack2(8.0f * GELU_C1, 8.0f * GELU_C1), mul2(h, h), pack2(2.0f * GELU_C0, 2.0f * GELU_C0)));
  return fma2(h, tanh2(u), h);
}
// gelu(2h) and its derivative at 2h, of both halves: with x = 2h and t = tanh(u),
// d gelu / dx = (1 + t)/2 + h (1 - t^2) du/dx, du/dx = C0 + 3 C1 x^2 = C0 + 12 C1 h^2
__device__ __forceinline__ F2 gelu2_of_half(F2 h, F2& grad) {
  const F2 s = mul2(h, h);
  const F2 t = tanh2(mul2(h, fma2(pack2(8.0f * GELU_C1, 8.0f * GELU_C1), s, pack2(2.0f * GELU_C0, 2.0f * GELU_C0))));
  const F2 one_t2 = fma2(F2{t.v ^ 0x8000000080000000ull}, t, pack2(1.0f, 1.0f));
  const F2 du = fma2(pack2(12.0f * GELU_C1, 12.0f * GELU_C1), s, pack2(GELU_C0, GELU_C0));
  grad = fma2(mul2(h, one_t2), du, fma2(pack2(0.5f, 0.5f), t, pack2(0.5f, 0.5f)));
  return fma2(h, t, h);
}
// the two halves rounded to BF16 (low half first)
__device__ __forceinline__ uint32_t bf16x2(F2 x) {
  float a, b;
  unpack2(x, a, b);
  const __nv_bfloat162 p = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const uint32_t*>(&p);
}
__device__ __forceinline__ uint32_t tile_off(int r, int c, int chunk) {
  return (uint32_t)((c >> 3) * chunk + (r >> 3) * 128 + (r & 7) * 16 + (c & 7) * 2);
}

struct Status {
  int error;  // 1: a bounded tensor-core wait gave up
};

// 8 BF16 values halved (exact in binary)
__device__ __forceinline__ uint4 half_bf16x8(const __nv_bfloat16* p) {
  uint4 q = *reinterpret_cast<const uint4*>(p);
  __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&q);
  const __nv_bfloat162 half = __float2bfloat162_rn(0.5f);
#pragma unroll
  for (int k = 0; k < 4; ++k) h[k] = __hmul2(h[k], half);
  return q;
}
// x as the sum of three BF16 values (3 x 8 significant bits: exact), in columns 0..2 of a chunk row.
// A finite x that would round to infinity takes the largest BF16 value first; an infinite x is its
// first term alone (infinity less infinity would be NaN).
__device__ __forceinline__ uint4 split_bf16(float x) {
  __nv_bfloat16 hi = __float2bfloat16_rn(x);
  if (isinf(__bfloat162float(hi))) hi = __float2bfloat16_rz(x);
  const float r1 = isinf(x) ? 0.0f : x - __bfloat162float(hi);
  const __nv_bfloat16 mid = __float2bfloat16_rn(r1);
  const __nv_bfloat16 lo = __float2bfloat16_rn(r1 - __bfloat162float(mid));
  const uint32_t h = *reinterpret_cast<const uint16_t*>(&hi), m = *reinterpret_cast<const uint16_t*>(&mid),
                 l = *reinterpret_cast<const uint16_t*>(&lo);
  return make_uint4(h | (m << 16), l, 0u, 0u);
}
// columns 0..2 of a chunk row = 1: what split_bf16's three terms are multiplied with
__device__ __forceinline__ uint4 three_ones() { return make_uint4(0x3F803F80u, 0x3F80u, 0u, 0u); }

// The network's weights as K-major B operands: W1 with b1 in its padding, W2 and b2, all halved as
// gelu2_of_half takes them, and W3 (16 rows, two used).
__device__ __forceinline__ void load_weights(unsigned char* W1s, unsigned char* W2s, unsigned char* B2s,
                                             unsigned char* W3s, const ParamsBF16* __restrict__ wbf,
                                             const Params* __restrict__ p, int t) {
  const uint4 zero = make_uint4(0, 0, 0, 0);
  for (int idx = t; idx < NH * 4; idx += TILE) {
    const int r = idx >> 2, c = idx & 3;
    *reinterpret_cast<uint4*>(W1s + tile_off(r, 8 * c, W_CHUNK)) =
        c < 3 ? half_bf16x8(wbf->W1 + r * KIN + 8 * c) : split_bf16(0.5f * p->b1[r]);
  }
  for (int idx = t; idx < NH * 8; idx += TILE) {
    const int r = idx >> 3, c0 = (idx & 7) * 8;
    *reinterpret_cast<uint4*>(W2s + tile_off(r, c0, W_CHUNK)) = half_bf16x8(wbf->W2 + r * NH + c0);
  }
  {
    const int r = t >> 1, c = t & 1;  // 64 rows x 2 chunks
    *reinterpret_cast<uint4*>(B2s + tile_off(r, 8 * c, W_CHUNK)) = c == 0 ? split_bf16(0.5f * p->b2[r]) : zero;
  }
  {
    const int r = t >> 3, c = t & 7;  // 16 rows x 8 chunks
    *reinterpret_cast<uint4*>(W3s + tile_off(r, 8 * c, W3_CHUNK)) =
        r < NOUT ? *reinterpret_cast<const uint4*>(wbf->W3 + r * NH + 8 * c) : zero;
  }
}

// The bounded tensor-core waits of a CTA. wait() records a give-up in the CTA's shared abort
// word; every thread reads that word only right after a CTA-wide barrier, so all threads
// leave the tile loop together. `last` and `issued` (the parity of the last wait and whether
// an operation was committed to it) are the same in every thread.
struct MmaWaits {
  uint32_t mb;
  volatile int* abort;
  uint32_t phase = 0, last = 0;
  bool issued = false;
  __device__ MmaWaits(uint32_t mbar, int* abort_word) : mb(mbar), abort(abort_word) {}
  __device__ __forceinline__ void wait(bool committed) {
    last = phase;
    if (!mbar_wait(mb, phase)) *abort = 1;
    phase ^= 1;
    issued = committed;
    fence_after();
  }
  __device__ __forceinline__ bool aborted() const { return *abort != 0; }
  // after an abort: wait (bounded) for the committed operation whose completion was not seen,
  // so that the tensor memory it writes is no longer in use when it is freed
  __device__ __forceinline__ void drain() {
    if (*abort && issued) mbar_wait(mb, last);
  }
};

// ---- inference of one tile ------------------------------------------------------------
// A CTA of TILE threads with FWD_SMEM_BYTES of dynamic shared memory and FWD_TMEM_COLS
// tensor-memory columns. Everything a row needs of the weights reaches it through the tensor
// cores. A value read from shared memory for every row costs the shared-memory pipe a clock a
// warp however few bytes it is: biases and output weights, 256 values a row, kept that pipe
// 65 % busy and the tanh unit at 64 %. So a bias is three BF16 terms (exact) against columns of
// ones (b1 in X's padding, b2 in one more K step), and the output layer is a third MMA on H2.
struct InferSmem {
  unsigned char* ones;  // the second chunk of its K step is W1's first, against zeros
  unsigned char* XH;
  unsigned char* W1s;
  unsigned char* W2s;
  unsigned char* B2s;
  unsigned char* W3s;
  uint64_t* mbar;
  uint32_t* tmem_slot;
  __device__ explicit InferSmem(unsigned char* smem)
      : ones(smem), XH(ones + HX_CHUNK), W1s(XH + XH_BYTES), W2s(W1s + W1_BYTES), B2s(W2s + W2_BYTES),
        W3s(B2s + B2_BYTES), mbar(reinterpret_cast<uint64_t*>(W3s + W3_BYTES)),
        tmem_slot(reinterpret_cast<uint32_t*>(W3s + W3_BYTES + 16)) {}
};
struct InferStatic {
  float b3[NOUT];
  int abort;
};

// Tensor memory, the mbarrier and the weights; returns the CTA's TMEM base address.
__device__ __forceinline__ uint32_t infer_setup(const InferSmem& S, InferStatic& st, const ParamsBF16* wbf,
                                                const Params* p) {
  const int t = threadIdx.x, warp = t >> 5;
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(S.tmem_slot)),
                 "r"(FWD_TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  if (t == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(S.mbar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    st.abort = 0;
  }
  *reinterpret_cast<uint4*>(S.ones + tile_off(t, 0, HX_CHUNK)) = three_ones();
  load_weights(S.W1s, S.W2s, S.B2s, S.W3s, wbf, p, t);
  if (t < NOUT) st.b3[t] = p->b3[t];
  fence_async_smem();
  fence_before();
  __syncthreads();
  fence_after();
  return *S.tmem_slot;
}

// Row t of the tile's features (24 BF16 values as three 16-byte chunks) into XH chunks 0..2, and
// the ones of b1's columns into chunk 3.
__device__ __forceinline__ void infer_put_row(const InferSmem& S, const uint4 (&q)[3]) {
  const int t = threadIdx.x;
#pragma unroll
  for (int c = 0; c < 3; ++c) *reinterpret_cast<uint4*>(S.XH + tile_off(t, 8 * c, HX_CHUNK)) = q[c];
  *reinterpret_cast<uint4*>(S.XH + tile_off(t, 24, HX_CHUNK)) = three_ones();
}

// bf16(gelu(2 Z)) of this thread's row of Z (64 TMEM columns) into XH's row
__device__ __forceinline__ void infer_activate(const InferSmem& S, uint32_t lane_base) {
  const int t = threadIdx.x;
#pragma unroll
  for (int c = 0; c < 2; ++c) {
    float v[32];
    tmem_ld32(lane_base + 32 * c, v);
#pragma unroll
    for (int q = 0; q < 4; ++q) {  // 8 columns, one 16-byte store
      uint32_t h[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) h[k] = bf16x2(gelu2_of_half(pack2(v[8 * q + 2 * k], v[8 * q + 2 * k + 1])));
      *reinterpret_cast<uint4*>(S.XH + tile_off(t, 32 * c + 8 * q, HX_CHUNK)) = make_uint4(h[0], h[1], h[2], h[3]);
    }
  }
}

// The network on the tile in XH (all threads call it after writing their rows): this thread's
// two outputs; false if the CTA has given up a wait (then every thread returns false). With
// issue = false the first tensor-core operation is left out (the bounded wait's test). What
// bounds it is the special-function unit (128 tanh a row at 16 a clock: 1024 clocks a tile; 67 %
// busy by ncu) and the latency of three barrier and tensor-core round trips a tile behind it.
// Measured on 3.9 M rows: 253 us with scalar epilogues and shared-memory biases, 205 us with
// packed ones, 194 us in this form.
__device__ __forceinline__ bool infer_tile(const InferSmem& S, const InferStatic& st, uint32_t tmem, MmaWaits& waits,
                                           bool issue, float& y0, float& y1) {
  const int t = threadIdx.x, warp = t >> 5;
  const uint32_t lane_base = tmem + ((uint32_t)(warp * 32) << 16);
  const uint32_t xh = smem_u32(S.XH), w1 = smem_u32(S.W1s), w2 = smem_u32(S.W2s);
  const uint32_t ID = idesc_bf16(128, 64, 0, 0);
  auto sync_for_mma = [&]() {  // shared-memory writes -> visible to the tensor core
    fence_async_smem();
    fence_before();
    __syncthreads();
    fence_after();
  };
  sync_for_mma();
  if (waits.aborted()) return false;
  if (t == 0 && issue) {  // Z1 = X W1^T + b1
#pragma unroll
    for (int kk = 0; kk < 2; ++kk)
      mma_bf16(tmem, sdesc(xh + 2 * kk * HX_CHUNK, HX_CHUNK, 128), sdesc(w1 + 2 * kk * W_CHUNK, W_CHUNK, 128), ID, kk);
    mma_commit(waits.mb);
  }
  waits.wait(issue);
  infer_activate(S, lane_base);  // H1 (MMA 1 has read X)
  sync_for_mma();                // also: every thread has read Z1, which Z2 overwrites
  if (waits.aborted()) return false;
  if (t == 0) {  // Z2 = H1 W2^T + b2
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
      mma_bf16(tmem, sdesc(xh + 2 * kk * HX_CHUNK, HX_CHUNK, 128), sdesc(w2 + 2 * kk * W_CHUNK, W_CHUNK, 128), ID, kk);
    mma_bf16(tmem, sdesc(smem_u32(S.ones), w1 - smem_u32(S.ones), 128), sdesc(smem_u32(S.B2s), W_CHUNK, 128), ID, 1);
    mma_commit(waits.mb);
  }
  waits.wait(true);
  infer_activate(S, lane_base);  // H2 (MMA 2 has read H1)
  sync_for_mma();
  if (waits.aborted()) return false;
  if (t == 0) {  // Y = H2 W3^T
    const uint32_t w3 = smem_u32(S.W3s);
#pragma unroll
    for (int kk = 0; kk < 4; ++kk)
      mma_bf16(tmem, sdesc(xh + 2 * kk * HX_CHUNK, HX_CHUNK, 128), sdesc(w3 + 2 * kk * W3_CHUNK, W3_CHUNK, 128),
               idesc_bf16(128, 16, 0, 0), kk);
    mma_commit(waits.mb);
  }
  waits.wait(true);
  tmem_ld2(lane_base, y0, y1);
  y0 += st.b3[0];
  y1 += st.b3[1];
  fence_before();
  __syncthreads();  // the next tile rewrites XH, and its MMA 1 overwrites Y
  fence_after();
  return !waits.aborted();
}

// After the tile loop: the drain of a given-up wait, the status, the TMEM free.
__device__ __forceinline__ void infer_finish(MmaWaits& waits, uint32_t tmem, Status* status) {
  waits.drain();
  if (waits.aborted() && threadIdx.x == 0) atomicExch(&status->error, 1);
  fence_before();
  __syncthreads();
  fence_after();
  if ((threadIdx.x >> 5) == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(FWD_TMEM_COLS)
                 : "memory");
}

// Host side, defined in closure.cu. The network's device parameters and status word, for
// kernels that run it inline.
void closure_device_params(TriskClosure* c, const ParamsBF16** wbf, const Params** p, Status** status);
// Resident CTAs per SM of an inference-shaped kernel (TILE threads, FWD_SMEM_BYTES of dynamic
// shared memory, FWD_TMEM_COLS tensor-memory columns), from its shared memory, registers and
// threads; sets the kernel's shared-memory attributes on the current device first.
int infer_ctas_per_sm(const void* kernel, int device);

}  // namespace closure
}  // namespace trisk
