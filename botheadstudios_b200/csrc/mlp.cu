// Learned smoothing-length MLP on the tensor cores: 8 → 64 → 64 → 1 with GELU, BF16 operands and FP32
// accumulation. Inference (the in-step proposal and the standalone forward) and training both run on tcgen05:
// M = 128 × N = 64 tcgen05.mma tiles issued by one thread, operands in shared memory in the canonical
// no-swizzle K-major layout, accumulators in tensor memory (see the inference and training sections). Training
// computes the weight gradients as tcgen05 GEMMs over a tile's 128 samples; Adam updates an FP32 master copy.
#include <cstdint>
#include <cstring>
#include <map>
#include <mutex>
#include <thread>
#include <vector>

#include "../../include/sph_b200.h"
#include "mlp.cuh"

namespace sphb {

namespace {

constexpr int ROWS = 128;
// Largest proposed change of log h: an outlier proposal stays within reach of the fallback's Newton steps
// (±20 % each, inside the list skin around the proposal).
constexpr float kMaxStep = 0.03f;

__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.0f + erff(z * 0.70710678118654752f)); }

// ---- feature definition (the solver's state at the start of the step's drift) ---------------------------
__device__ __forceinline__ void features(int t, const State& st, const float* __restrict__ rho,
                                         const unsigned* __restrict__ cnt, const float4* __restrict__ acc,
                                         const float4* __restrict__ fdata, const float* __restrict__ divv,
                                         const Eos* __restrict__ eos, const Seg* __restrict__ segs,
                                         const DevParams* __restrict__ P, const MlpFeatureArgs& fa,
                                         float f[MLP_IN]) {
  const float4 p = st.pos_h[t];
  const float m = st.mass[t];
  const float r = fmaxf(rho[t], 1.0e-30f);
  const unsigned mat = st.mat[t];
  const float rho0 = eos[mat].rho0, e_iv = eos[mat].e_iv;
  const float heq = fa.eta * cbrtf(m / r);
  const float dt = (float)segs[st.seg[t]].dt;
  const float4 a = acc[t];
  const float c = fmaxf(fdata[t].w, P->sig_floor);  // the Courant signal's floor keeps c² > 0
  f[0] = logf(p.w / heq);                                                      // log h relative to h(rho)
  f[1] = logf(r / rho0);                                                       // log rho / rho0
  f[2] = divv[t] * dt;                                                         // div v over the step
  f[3] = (float)cnt[t] / fa.n_target;                                          // neighbours / target
  f[4] = log1pf(sqrtf(a.x * a.x + a.y * a.y + a.z * a.z) * p.w / (c * c));     // |a| h / c²
  f[5] = (float)mat;                                                           // material
  f[6] = log1pf(fmaxf(st.vel_u[t].w, 0.0f) / e_iv);                            // u / E_iv
  f[7] = P->progress;                                                          // step fraction
}

// ---- inference on the 5th-generation tensor cores (tcgen05) ---------------------------------------------
// A CTA of 128 threads holds 128 rows. Each thread writes its row of x' (layer 1) or of a1 (layer 2) into
// shared memory in the canonical no-swizzle K-major layout (8-row × 16-byte core matrices; core matrices
// adjacent along K are 128 B apart, 8-row groups K·16 B apart); one thread issues tcgen05.mma (BF16 × BF16 →
// FP32, M = 128, N = 64, K = 16 per instruction) with the weights as the K-major B operand, and commits to an
// mbarrier. The accumulators live in tensor memory: row r of D is TMEM lane r, so after the barrier every
// thread reads its own row (tcgen05.ld 32x32b) and applies bias, GELU and the next layer's input rounding,
// and the 64 → 1 output layer is a per-thread dot product. Every barrier wait is bounded: on a timeout the
// CTA stops issuing, raises an error flag, waits (bounded) for what it issued and frees its tensor memory.
constexpr int TC_COLS = 128;            // TMEM columns per CTA: D1 [0, 64), D2 [64, 128)
constexpr int TC_SMEM = 56 * 1024;      // dynamic shared memory per CTA: at most 4 CTAs (4 × 128 of 512 columns)
constexpr unsigned kTcSpin = 1u << 16;  // barrier polls before giving up
constexpr uint32_t kTcIdesc = (1u << 4)            // D: FP32
                              | (1u << 7)          // A: BF16
                              | (1u << 10)         // B: BF16 (A and B K-major: bits 15, 16 clear)
                              | ((64u >> 3) << 17) // N = 64
                              | ((128u >> 4) << 24);  // M = 128

struct TcSmem {
  __nv_bfloat16 a1[ROWS * 16];      // x' rows (K = 16, inputs 8..15 zero)
  __nv_bfloat16 a2[ROWS * MLP_H];   // a1 rows (K = 64)
  __nv_bfloat16 w1[MLP_H * 16];     // W1ᵀ [out][in] (K = 16)
  __nv_bfloat16 w2[MLP_H * MLP_H];  // W2ᵀ [out][in] (K = 64)
  float b1[MLP_H], b2[MLP_H], w3[MLP_H];
  unsigned long long mbar;
  unsigned tmem;
  int ok;
};
static_assert(sizeof(TcSmem) <= TC_SMEM, "tcgen05 tile fits its shared memory");

// element offset of (row r, k) in a K-major no-swizzle operand with K columns
__device__ __forceinline__ int cm(int r, int k, int K) { return (r >> 3) * (K * 8) + (k >> 3) * 64 + (r & 7) * 8 + (k & 7); }
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
// shared-memory matrix descriptor: start, leading (K) and stride (8-row) byte offsets, sm100 version bits, no swizzle
__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
__device__ __forceinline__ void tc_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t acc) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
               :: "r"(d), "l"(a), "l"(b), "r"(kTcIdesc), "r"(acc) : "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" :: "r"(mbar) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity) {
  for (unsigned i = 0; i < kTcSpin; ++i) {
    uint32_t done;
    asm volatile("{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(done) : "r"(mbar), "r"(parity) : "memory");
    if (done) return true;
  }
  return false;
}
// 16 consecutive FP32 columns of this warp's 32 TMEM lanes (one per thread)
__device__ __forceinline__ void tc_ld16(uint32_t taddr, float v[16]) {
  uint32_t r[16];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                 "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
               : "r"(taddr));
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void tc_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ uint4 pack8(const float f[8]) {
  __nv_bfloat162 h[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) h[i] = __floats2bfloat162_rn(f[2 * i], f[2 * i + 1]);
  return *reinterpret_cast<uint4*>(h);
}

// A weight matrix into shared memory: the packed form has the operand layout already.
__device__ __forceinline__ void copy_operand(__nv_bfloat16* dst, const __nv_bfloat16* __restrict__ src, int count, int threads) {
  for (int i = threadIdx.x; i < count / 8; i += threads)
    reinterpret_cast<uint4*>(dst)[i] = reinterpret_cast<const uint4*>(src)[i];
}

// CTA set-up: tensor memory, the barrier, the weights.
__device__ void tc_setup(TcSmem& S, const MlpPacked* __restrict__ W) {
  copy_operand(S.w1, W->w1t, MLP_H * 16, ROWS);
  copy_operand(S.w2, W->w2t, MLP_H * MLP_H, ROWS);
  for (int i = threadIdx.x; i < MLP_H; i += ROWS) {
    S.b1[i] = W->b1[i];
    S.b2[i] = W->b2[i];
    S.w3[i] = W->w3[i];
  }
  if (threadIdx.x == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&S.mbar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    S.ok = 1;
  }
  if (threadIdx.x < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(smem_u32(&S.tmem)), "r"(TC_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
}

// One 128-row tile: this thread's normalised inputs in, its y (before b3) out (NaN after a barrier timeout).
__device__ float tc_tile(TcSmem& S, const float xq[MLP_IN], uint32_t& phase) {
  const int r = threadIdx.x, w = r >> 5;
  const uint32_t mbar = smem_u32(&S.mbar);
  const uint32_t trow = S.tmem + ((uint32_t)(w * 32) << 16);
  const float zero8[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  *reinterpret_cast<uint4*>(S.a1 + cm(r, 0, 16)) = pack8(xq);
  *reinterpret_cast<uint4*>(S.a1 + cm(r, 8, 16)) = pack8(zero8);
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (!S.ok) return __int_as_float(0x7fc00000);
  if (r == 0) {
    tc_mma(S.tmem, umma_desc(smem_u32(S.a1), 128, 256), umma_desc(smem_u32(S.w1), 128, 256), 0u);
    tc_commit(mbar);
  }
  // on a timeout `phase` keeps the parity of the commit still outstanding, for the tear-down to wait on
  bool got = mbar_wait(mbar, phase);
  if (!__syncthreads_and(got)) {
    if (r == 0) S.ok = 0;
    return __int_as_float(0x7fc00000);
  }
  phase ^= 1u;
  tc_fence_after();
  // layer 1 → GELU → a1 (bf16) row
  float z[64];
#pragma unroll
  for (int c = 0; c < 4; ++c) tc_ld16(trow + 16 * c, z + 16 * c);
  tc_wait_ld();
#pragma unroll
  for (int kb = 0; kb < 8; ++kb) {
    float h[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) h[i] = gelu(z[8 * kb + i] + S.b1[8 * kb + i]);
    *reinterpret_cast<uint4*>(S.a2 + cm(r, 8 * kb, 64)) = pack8(h);
  }
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (r == 0) {
#pragma unroll
    for (int kt = 0; kt < 4; ++kt)
      tc_mma(S.tmem + 64, umma_desc(smem_u32(S.a2) + 256 * kt, 128, 1024), umma_desc(smem_u32(S.w2) + 256 * kt, 128, 1024),
             kt > 0 ? 1u : 0u);
    tc_commit(mbar);
  }
  got = mbar_wait(mbar, phase);
  if (!__syncthreads_and(got)) {
    if (r == 0) S.ok = 0;
    return __int_as_float(0x7fc00000);
  }
  phase ^= 1u;
  tc_fence_after();
#pragma unroll
  for (int c = 0; c < 4; ++c) tc_ld16(trow + 64 + 16 * c, z + 16 * c);
  tc_wait_ld();
  float y = 0.0f;
#pragma unroll
  for (int j = 0; j < MLP_H; ++j) y += gelu(z[j] + S.b2[j]) * S.w3[j];
  tc_fence_before();
  return y;
}

// CTA tear-down: after a timeout, wait (bounded) for the last commit; then free the tensor memory.
__device__ bool tc_teardown(TcSmem& S, uint32_t phase) {
  const bool failed = !S.ok;
  if (failed) mbar_wait(smem_u32(&S.mbar), phase);  // what was issued before the timeout, if anything
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (threadIdx.x < 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(S.tmem), "r"(TC_COLS) : "memory");
  return !failed;
}

__device__ __forceinline__ void normalise(const float f[MLP_IN], const MlpPacked* W, float xq[MLP_IN]) {
#pragma unroll
  for (int k = 0; k < MLP_IN; ++k) xq[k] = (f[k] - W->xm[k]) * W->xs[k];
}

__global__ void __launch_bounds__(ROWS) k_mlp_propose(int n, State st, const float* __restrict__ rho,
                                                     const unsigned* __restrict__ cnt,
                                                     const float4* __restrict__ acc,
                                                     const float4* __restrict__ fdata,
                                                     const float* __restrict__ divv, const Eos* __restrict__ eos,
                                                     const Seg* __restrict__ segs, DevParams* __restrict__ P,
                                                     MlpFeatureArgs fa, const MlpPacked* __restrict__ W,
                                                     float* __restrict__ rec, float* __restrict__ dh, int apply) {
  extern __shared__ __align__(1024) unsigned char tc_raw[];
  TcSmem& S = *reinterpret_cast<TcSmem*>(tc_raw);
  tc_setup(S, W);
  const float b3 = W->b3, ym = W->ym, ys = W->ys;
  uint32_t phase = 0;
  const int r = threadIdx.x;
  for (int base = blockIdx.x * ROWS; base < n; base += gridDim.x * ROWS) {
    const int t = base + r;
    float f[MLP_IN] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, xq[MLP_IN];
    if (t < n) features(t, st, rho, cnt, acc, fdata, divv, eos, segs, P, fa, f);
    normalise(f, W, xq);
    const float y = tc_tile(S, xq, phase);
    if (t < n) {
      // the network gives log(h_next / h(rho)); the step from the current h subtracts log(h / h(rho)) = f[0],
      // so a residual left by the previous solve is corrected whatever the network learned
      const float d = (y + b3) * ys + ym - f[0];
      const float dc = d == d ? fminf(fmaxf(d, -kMaxStep), kMaxStep) : 0.0f;  // no proposal from a NaN
      if (apply) st.pos_h[t].w = st.pos_h[t].w * expf(dc);
      if (rec) {
        const unsigned id = st.id[t];
#pragma unroll
        for (int k = 0; k < MLP_IN; ++k) rec[(size_t)id * MLP_IN + k] = f[k];
        dh[id] = d;
      }
    }
  }
  if (!tc_teardown(S, phase) && threadIdx.x == 0) atomicOr(&P->flags, kFlagTensorTimeout);
}

__global__ void __launch_bounds__(ROWS) k_mlp_forward(const MlpPacked* __restrict__ W, const float* __restrict__ x,
                                                     int n, float* __restrict__ out, unsigned* __restrict__ err) {
  extern __shared__ __align__(1024) unsigned char tc_raw[];
  TcSmem& S = *reinterpret_cast<TcSmem*>(tc_raw);
  tc_setup(S, W);
  uint32_t phase = 0;
  const int r = threadIdx.x;
  for (int base = blockIdx.x * ROWS; base < n; base += gridDim.x * ROWS) {
    const int t = base + r;
    float f[MLP_IN] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, xq[MLP_IN];
    if (t < n)
#pragma unroll
      for (int k = 0; k < MLP_IN; ++k) f[k] = x[(size_t)t * MLP_IN + k];
    normalise(f, W, xq);
    const float y = tc_tile(S, xq, phase);
    if (t < n) out[t] = (y + W->b3) * W->ys + W->ym;
  }
  if (!tc_teardown(S, phase) && threadIdx.x == 0) atomicOr(err, 1u);
}

// ---- training on tcgen05: forward + backward, 128 samples at a time --------------------------------------------
// The same tiles as inference (M = 128 × N = 64, BF16 × BF16 → FP32 in tensor memory, one issuing thread, bounded
// mbarrier waits), five MMA groups per tile: the two forward layers (D1 = x'·W1ᵀ, D2 = a1·W2ᵀ), then da1 = dz2·W2 (D3)
// together with dW2 += a1ᵀ·dz2 (D4), then dW1 += x'ᵀ·dz1 (D5). The weight gradients contract over the tile's 128
// samples: their operands are the row-major activations read as M-major (the transpose bits of the instruction), so
// nothing is stored twice. Their M (64 inputs of layer 2, 16 padded inputs of layer 1) is padded to the instruction's
// 128 rows, whose extra rows read whatever follows in shared memory and are never used.
// Bound by the chain of a tile: five MMA groups and, between them, the GELU of 64 columns a row. So a tile has 512
// threads, four to a row: a thread takes 16 columns of its row of each accumulator, evaluates GELU and its derivative
// from one erf and one exp, and keeps what the backward pass needs in registers (with one thread to a row, its values
// in shared memory and 4.8k atomic adds a tile, a minibatch of 4,096 took 77.6 µs, and 10 µs more for the optimizer and
// the packing; this takes 16.9 and 5.7). Weight gradients stay in tensor
// memory and bias gradients in registers over a CTA's tiles; the CTA writes them once, and the optimizer adds the
// CTAs' shares in their order, so a training run is repeatable.
constexpr int TT_THREADS = 512, TT_CG = TT_THREADS / ROWS, TT_COL = MLP_H / TT_CG;  // 4 column groups of 16
constexpr int TT_COLS = 512;  // TMEM columns: D1 [0, 64), D2 [64, 128), D3 [128, 192), D4 [192, 256), D5 [256, 320)
constexpr uint32_t kTcIdescT = kTcIdesc | (1u << 15) | (1u << 16);  // A and B M-/N-major
constexpr int MLP_PART = MLP_TRAIN + 1;  // a CTA's share: the gradient, then the summed squared error

struct TrainTcSmem {
  __nv_bfloat16 xa[ROWS * 16];       // x' [row][k], K = 16
  __nv_bfloat16 ha[ROWS * MLP_H];    // a1 [row][i], then dz1 [row][i]
  __nv_bfloat16 dza[ROWS * MLP_H];   // dz2 [row][out]
  __nv_bfloat16 w1[MLP_H * 16];      // W1ᵀ [out][k] (B of layer 1)
  __nv_bfloat16 w2t[MLP_H * MLP_H];  // W2ᵀ [out][i] (B of layer 2)
  __nv_bfloat16 w2b[MLP_H * MLP_H];  // W2 [i][out] (B of da1 = dz2 W2: N = i, K = out)
  float b1[MLP_H], b2[MLP_H], w3[MLP_H];
  float y[TT_CG][ROWS];              // the column groups' shares of each row's output
  float tn[ROWS];                    // normalised targets
  float col[4][3][MLP_H];            // the row quarters' column sums: W3, b2, b1 gradients
  float row[4][2];                   // ... and their sums of dy and of the squared error
  unsigned long long mbar;
  unsigned tmem;
  int ok;
};

__device__ __forceinline__ void tc_mma_t(uint32_t d, uint64_t a, uint64_t b, uint32_t acc) {
  asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
               "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
               :: "r"(d), "l"(a), "l"(b), "r"(kTcIdescT), "r"(acc) : "memory");
}

// Issue (thread 0) the MMAs of `fn`, commit to the barrier, wait (bounded) for them; false on a timeout.
template <typename F>
__device__ bool tt_run(TrainTcSmem& S, uint32_t& phase, F fn) {
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (!S.ok) return false;
  const uint32_t mbar = smem_u32(&S.mbar);
  if (threadIdx.x == 0) {
    fn();
    tc_commit(mbar);
  }
  const bool got = mbar_wait(mbar, phase);
  if (!__syncthreads_and(got)) {
    if (threadIdx.x == 0) S.ok = 0;
    return false;
  }
  phase ^= 1u;
  tc_fence_after();
  return true;
}

// GELU and its derivative from one erf and one exp.
__device__ __forceinline__ void gelu_both(float z, float& g, float& d) {
  const float c = 0.5f * (1.0f + erff(z * 0.70710678118654752f));
  g = z * c;
  d = c + z * expf(-0.5f * z * z) * 0.39894228040143268f;
}

// This thread's 16 columns of its row, as BF16, into an operand of 64 columns.
__device__ __forceinline__ void tt_store(__nv_bfloat16* op, int r, int c0, const float v[TT_COL]) {
  *reinterpret_cast<uint4*>(op + cm(r, c0, MLP_H)) = pack8(v);
  *reinterpret_cast<uint4*>(op + cm(r, c0 + 8, MLP_H)) = pack8(v + 8);
}

__global__ void __launch_bounds__(TT_THREADS) k_mlp_train_tc(const MlpPacked* __restrict__ W, const float* __restrict__ x,
                                                            const float* __restrict__ tgt, const unsigned* __restrict__ idx,
                                                            int m, float denom, float* __restrict__ part,
                                                            unsigned* __restrict__ err) {
  extern __shared__ __align__(1024) unsigned char tt_raw[];
  TrainTcSmem& S = *reinterpret_cast<TrainTcSmem*>(tt_raw);
  const int tid = threadIdx.x, lane = tid & 31, quarter = (tid >> 5) & 3, r = quarter * 32 + lane;
  const int cg = tid / ROWS, c0 = cg * TT_COL;
  cudaTriggerProgrammaticLaunchCompletion();  // the optimizer's blocks may take their places and wait
  if (tid == 0) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" :: "r"(smem_u32(&S.mbar)) : "memory");
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    S.ok = 1;
  }
  if (tid < 32) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                 :: "r"(smem_u32(&S.tmem)), "r"(TT_COLS) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // the first tile's row (the samples do not depend on the previous step), then the previous step's weights
  float f[MLP_IN] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}, traw = 0.0f;
  const auto sample = [&](int s) {
    const unsigned j = idx[s];
    *reinterpret_cast<float4*>(f) = reinterpret_cast<const float4*>(x)[2 * (size_t)j];
    *reinterpret_cast<float4*>(f + 4) = reinterpret_cast<const float4*>(x)[2 * (size_t)j + 1];
    traw = tgt[j];
  };
  if (cg == 0 && (int)(blockIdx.x * ROWS) + r < m) sample((int)(blockIdx.x * ROWS) + r);
  cudaGridDependencySynchronize();
  copy_operand(S.w1, W->w1t, MLP_H * 16, TT_THREADS);
  copy_operand(S.w2t, W->w2t, MLP_H * MLP_H, TT_THREADS);
  copy_operand(S.w2b, W->w2, MLP_H * MLP_H, TT_THREADS);
  if (tid < MLP_H) {
    S.b1[tid] = W->b1[tid];
    S.b2[tid] = W->b2[tid];
    S.w3[tid] = W->w3[tid];
  }
  const float b3 = W->b3;
  const uint32_t xa = smem_u32(S.xa), ha = smem_u32(S.ha), w1 = smem_u32(S.w1), w2t = smem_u32(S.w2t);
  const uint32_t w2b = smem_u32(S.w2b), dza = smem_u32(S.dza);
  const float zero8[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  float gw3[TT_COL], gb2[TT_COL], gb1[TT_COL], sdy = 0.0f, se2 = 0.0f;
#pragma unroll
  for (int j = 0; j < TT_COL; ++j) gw3[j] = gb2[j] = gb1[j] = 0.0f;
  uint32_t phase = 0, more = 0;
  bool ok = true;
  for (int base = blockIdx.x * ROWS; base < m && ok; base += gridDim.x * ROWS, more = 1u) {
    const bool valid = base + r < m;  // rows past m carry dy = 0 and add nothing
    if (cg == 0) {
      float xq[MLP_IN];
      normalise(f, W, xq);
      *reinterpret_cast<uint4*>(S.xa + cm(r, 0, 16)) = pack8(xq);
      *reinterpret_cast<uint4*>(S.xa + cm(r, 8, 16)) = pack8(zero8);
      S.tn[r] = valid ? (traw - W->ym) / W->ys : 0.0f;
      const int next = base + (int)gridDim.x * ROWS + r;
      if (next < m) sample(next);
    }
    // ---- layer 1: z1 = x'·W1ᵀ + b1, a1 = GELU(z1) ------------------------------------------------------------
    ok = tt_run(S, phase, [&] { tc_mma(S.tmem, umma_desc(xa, 128, 256), umma_desc(w1, 128, 256), 0u); });
    if (!ok) break;
    const uint32_t trow = S.tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0;
    float v[TT_COL], d1[TT_COL], a[TT_COL];
    tc_ld16(trow, v);
    tc_wait_ld();
#pragma unroll
    for (int j = 0; j < TT_COL; ++j) gelu_both(v[j] + S.b1[c0 + j], a[j], d1[j]);
    tt_store(S.ha, r, c0, a);
    // ---- layer 2 and the output: y = Σ GELU(z2)·w3 + b3, dy, dz2 = dy·w3·GELU'(z2) ----------------------------
    ok = tt_run(S, phase, [&] {
      for (int kt = 0; kt < 4; ++kt)
        tc_mma(S.tmem + 64, umma_desc(ha + 256 * kt, 128, 1024), umma_desc(w2t + 256 * kt, 128, 1024), kt > 0 ? 1u : 0u);
    });
    if (!ok) break;
    tc_ld16(trow + 64, v);
    tc_wait_ld();
    float y = 0.0f;
#pragma unroll
    for (int j = 0; j < TT_COL; ++j) {
      float g;
      gelu_both(v[j] + S.b2[c0 + j], a[j], g);
      y += a[j] * S.w3[c0 + j];
      v[j] = g;
    }
    S.y[cg][r] = y;
    __syncthreads();
    y = 0.0f;
#pragma unroll
    for (int k = 0; k < TT_CG; ++k) y += S.y[k][r];
    const float e = valid ? (y + b3 - S.tn[r]) : 0.0f;
    const float dy = 2.0f * e / denom;
    if (cg == 0) {
      sdy += dy;
      se2 += e * e;
    }
#pragma unroll
    for (int j = 0; j < TT_COL; ++j) {
      gw3[j] += dy * a[j];
      v[j] = dy * S.w3[c0 + j] * v[j];
      gb2[j] += v[j];
    }
    tt_store(S.dza, r, c0, v);
    // ---- da1 = dz2·W2 (D3) and dW2 += a1ᵀ·dz2 (D4, rows 0..63) ------------------------------------------------
    ok = tt_run(S, phase, [&] {
      for (int kt = 0; kt < 4; ++kt)
        tc_mma(S.tmem + 128, umma_desc(dza + 256 * kt, 128, 1024), umma_desc(w2b + 256 * kt, 128, 1024), kt > 0 ? 1u : 0u);
      for (int kt = 0; kt < 8; ++kt)  // 16 samples: two 8-sample blocks 1,024 B apart, 8 columns 128 B apart
        tc_mma_t(S.tmem + 192, umma_desc(ha + 2048 * kt, 1024, 128), umma_desc(dza + 2048 * kt, 1024, 128), kt > 0 ? 1u : more);
    });
    if (!ok) break;
    tc_ld16(trow + 128, v);
    tc_wait_ld();
#pragma unroll
    for (int j = 0; j < TT_COL; ++j) {
      v[j] *= d1[j];
      gb1[j] += v[j];
    }
    tt_store(S.ha, r, c0, v);  // a1 is done with
    // ---- dW1 += x'ᵀ·dz1 (D5, rows k < 8) -----------------------------------------------------------------------
    ok = tt_run(S, phase, [&] {
      for (int kt = 0; kt < 8; ++kt)
        tc_mma_t(S.tmem + 256, umma_desc(xa + 512 * kt, 256, 128), umma_desc(ha + 2048 * kt, 1024, 128), kt > 0 ? 1u : more);
    });
  }
  // ---- the CTA's share of the gradient -------------------------------------------------------------------------
  float* out = part + (size_t)blockIdx.x * MLP_PART;
  if (ok) {
#pragma unroll
    for (int j = 0; j < TT_COL; ++j) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        gw3[j] += __shfl_xor_sync(SPH_FULL_MASK, gw3[j], o);
        gb2[j] += __shfl_xor_sync(SPH_FULL_MASK, gb2[j], o);
        gb1[j] += __shfl_xor_sync(SPH_FULL_MASK, gb1[j], o);
      }
      if (lane == j) {
        S.col[quarter][0][c0 + j] = gw3[j];
        S.col[quarter][1][c0 + j] = gb2[j];
        S.col[quarter][2][c0 + j] = gb1[j];
      }
    }
    if (cg == 0) {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        sdy += __shfl_xor_sync(SPH_FULL_MASK, sdy, o);
        se2 += __shfl_xor_sync(SPH_FULL_MASK, se2, o);
      }
      if (lane == 0) {
        S.row[quarter][0] = sdy;
        S.row[quarter][1] = se2;
      }
    }
    const uint32_t trow = S.tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0;
    float v[TT_COL];
    if (quarter < 2) {
      tc_ld16(trow + 192, v);
      tc_wait_ld();
#pragma unroll
      for (int j = 0; j < TT_COL; ++j) out[MLP_W2 + r * MLP_H + c0 + j] = v[j];
    }
    if (quarter == 0) {
      tc_ld16(trow + 256, v);
      tc_wait_ld();
      if (r < MLP_IN)
#pragma unroll
        for (int j = 0; j < TT_COL; ++j) out[MLP_W1 + r * MLP_H + c0 + j] = v[j];
    }
    __syncthreads();
    if (tid < 3 * MLP_H) {
      const int k = tid / MLP_H, c = tid % MLP_H;
      out[(k == 0 ? MLP_W3 : k == 1 ? MLP_B2 : MLP_B1) + c] = S.col[0][k][c] + S.col[1][k][c] + S.col[2][k][c] + S.col[3][k][c];
    } else if (tid < 3 * MLP_H + 2) {
      const int k = tid - 3 * MLP_H;
      out[k == 0 ? MLP_B3 : MLP_TRAIN] = S.row[0][k] + S.row[1][k] + S.row[2][k] + S.row[3][k];
    }
  }
  // ---- tear-down: after a timeout wait (bounded) for what was issued, then free the tensor memory -------------
  if (!ok) mbar_wait(smem_u32(&S.mbar), phase);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (tid < 32)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" :: "r"(S.tmem), "r"(TT_COLS) : "memory");
  if (!ok && tid == 0) atomicOr(err, 1u);
}

// Trainable parameter i as the kernels read it (BF16 matrices in the operand layout).
__device__ __forceinline__ void pack_param(int i, float p, MlpPacked* __restrict__ o) {
  if (i < MLP_B1) {
    o->w1t[cm(i % MLP_H, i / MLP_H, 16)] = __float2bfloat16_rn(p);
  } else if (i < MLP_W2) {
    o->b1[i - MLP_B1] = p;
  } else if (i < MLP_B2) {
    const int in = (i - MLP_W2) / MLP_H, out = (i - MLP_W2) % MLP_H;
    const __nv_bfloat16 b = __float2bfloat16_rn(p);
    o->w2t[cm(out, in, MLP_H)] = b;
    o->w2[cm(in, out, MLP_H)] = b;
  } else if (i < MLP_W3) {
    o->b2[i - MLP_B2] = p;
  } else if (i < MLP_B3) {
    o->w3[i - MLP_W3] = __bfloat162float(__float2bfloat16_rn(p));
  } else {
    o->b3 = p;
  }
}

__global__ void k_mlp_pack(const float* __restrict__ P, MlpPacked* __restrict__ o) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < MLP_TRAIN) pack_param(i, P[i], o);
  if (i < MLP_H * 8) o->w1t[cm(i / 8, 8 + i % 8, 16)] = __float2bfloat16_rn(0.0f);  // inputs 8..15
  if (i < MLP_IN) {
    o->xm[i] = P[MLP_XM + i];
    o->xs[i] = P[MLP_XS + i];
  }
  if (i == 0) {
    o->ym = P[MLP_YM];
    o->ys = P[MLP_YS];
  }
}

// The CTAs' shares of value i, in their order.
__device__ __forceinline__ float part_sum(const float* __restrict__ part, int ctas, int i) {
  float g = 0.0f;
#pragma unroll 16
  for (int k = 0; k < ctas; ++k) g += part[(size_t)k * MLP_PART + i];
  return g;
}

__global__ void k_mlp_reduce(const float* __restrict__ part, int ctas, float* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < MLP_PART) out[i] = part_sum(part, ctas, i);
}

// Adam, the loss of the minibatch, and the packed weights of the next one.
__global__ void k_mlp_adam(float* __restrict__ p, const float* __restrict__ part, int ctas, float* __restrict__ m,
                           float* __restrict__ v, MlpPacked* __restrict__ w, float* __restrict__ loss, float lr,
                           float b1, float b2, float eps, float wd, float c1, float c2) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  cudaGridDependencySynchronize();            // the minibatch's shares
  cudaTriggerProgrammaticLaunchCompletion();  // the next minibatch may gather its samples
  if (i >= MLP_PART) return;
  const float g = part_sum(part, ctas, i);
  if (i == MLP_TRAIN) {
    *loss += g;
    return;
  }
  float q = p[i];
  const float gi = g + wd * q;
  const float mi = b1 * m[i] + (1.0f - b1) * gi;
  const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  q -= lr * (mi / c1) / (sqrtf(vi / c2) + eps);
  p[i] = q;
  pack_param(i, q, w);
}

int propose_grid() {  // 4 blocks per SM of the current device
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return sms * 4;
}

}  // namespace

int launch_mlp_pack(const float* params, MlpPacked* out, cudaStream_t s) {
  k_mlp_pack<<<(MLP_TRAIN + 127) / 128, 128, 0, s>>>(params, out);
  return 1;
}

int launch_mlp_propose(const Dev& d, const MlpPacked* w, const MlpFeatureArgs& fa, const float* divv, float* rec,
                       float* dh, bool apply, cudaStream_t s) {
  static SmemLimit attr;
  smem_limit(k_mlp_propose, TC_SMEM, attr);
  const int tiles = (d.n + ROWS - 1) / ROWS;
  const int cap = propose_grid();
  const int grid = tiles < cap ? tiles : cap;
  k_mlp_propose<<<grid, ROWS, TC_SMEM, s>>>(d.n, d.s(), d.rho, d.nbr_cnt, d.acc, d.fdata, divv, d.eos, d.segs, d.P, fa,
                                      w, rec, dh, apply ? 1 : 0);
  return 1;
}

int launch_mlp_forward(const MlpPacked* w, const float* x, int n, float* out, unsigned* err, cudaStream_t s) {
  static SmemLimit attr;
  smem_limit(k_mlp_forward, TC_SMEM, attr);
  const int tiles = (n + ROWS - 1) / ROWS;
  const int cap = propose_grid();
  const int grid = tiles < cap ? tiles : cap;
  k_mlp_forward<<<grid, ROWS, TC_SMEM, s>>>(w, x, n, out, err);
  return 1;
}

// A launch whose set-up overlaps the previous kernel of the stream (it waits for it in cudaGridDependencySynchronize).
template <typename... P, typename... A>
static void launch_overlapped(void (*kernel)(P...), int grid, int block, size_t smem, cudaStream_t s, A... args) {
  cudaLaunchConfig_t cfg{};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3((unsigned)block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute a[1];
  a[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  a[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = a;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, P(args)...);
}

int mlp_train_ctas(int m) {
  const int tiles = (m + ROWS - 1) / ROWS, sms = propose_grid() / 4;
  return tiles < sms ? tiles : sms;
}

size_t mlp_part_floats(int m) { return (size_t)mlp_train_ctas(m) * MLP_PART; }

int launch_mlp_train_batch(const MlpPacked* w, const float* x, const float* t, const unsigned* idx, int m,
                           float denom, float* part, unsigned* err, cudaStream_t s) {
  static SmemLimit attr;
  smem_limit(k_mlp_train_tc, (int)sizeof(TrainTcSmem), attr);
  launch_overlapped(k_mlp_train_tc, mlp_train_ctas(m), TT_THREADS, sizeof(TrainTcSmem), s, w, x, t, idx, m, denom, part,
                    err);
  return 1;
}

int launch_mlp_reduce(const float* part, int m, float* grad_loss, cudaStream_t s) {
  k_mlp_reduce<<<(MLP_PART + 127) / 128, 128, 0, s>>>(part, mlp_train_ctas(m), grad_loss);
  return 1;
}

int launch_mlp_adam(float* params, const float* part, int batch, float* m, float* v, MlpPacked* w, float* loss, int step,
                    float lr, float b1, float b2, float eps, float wd, cudaStream_t s) {
  const float c1 = 1.0f - powf(b1, (float)step), c2 = 1.0f - powf(b2, (float)step);
  launch_overlapped(k_mlp_adam, (MLP_PART + 127) / 128, 128, 0, s, params, part, mlp_train_ctas(batch), m, v, w, loss, lr,
                    b1, b2, eps, wd, c1, c2);
  return 1;
}

}  // namespace sphb

// ---- the network on its own (host arrays, blocking, the calling thread's current device) ------------------
using namespace sphb;

namespace {

// The calls below allocate from a pool of their own for each device context, which keeps up to 64 MB of what they free for
// the next call and gives the rest back (cudaMalloc and cudaFree of a call's buffers took 0.4-0.7 ms of a 2 ms epoch of
// 100,000 samples, and milliseconds on a busy host). A pool ends with its context: after a cudaDeviceReset the next call
// makes another. Stream order on the default stream makes it safe between threads.
constexpr unsigned long long kPoolKeeps = 64ull << 20;

cudaError_t call_pool(cudaMemPool_t* pool) {
  static std::mutex mu;
  static std::map<unsigned long long, cudaMemPool_t> pools;  // by the context's id
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess && current_ctx_id() == 0) e = cudaFree(nullptr);  // the device's context, if there is none yet
  if (e != cudaSuccess) return e;
  const unsigned long long id = current_ctx_id();
  if (id == 0) return cudaDeviceGetDefaultMemPool(pool, dev);  // nothing to remember a pool under
  std::lock_guard<std::mutex> lock(mu);
  cudaMemPool_t& p = pools[id];
  if (!p) {
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    e = cudaMemPoolCreate(&p, &props);
    unsigned long long keep = kPoolKeeps;
    if (e == cudaSuccess) e = cudaMemPoolSetAttribute(p, cudaMemPoolAttrReleaseThreshold, &keep);
    if (e != cudaSuccess) {
      if (p) cudaMemPoolDestroy(p);
      pools.erase(id);
      return e;
    }
  }
  *pool = p;
  return cudaSuccess;
}

// The device buffers of one call, in one allocation.
struct DevBuf {
  size_t bytes = 0;
  char* base = nullptr;
  template <typename T>
  size_t add(size_t count) {
    const size_t at = bytes;
    bytes += (count * sizeof(T) + 255) / 256 * 256;
    return at;
  }
  cudaError_t alloc() {
    cudaMemPool_t pool;
    const cudaError_t e = call_pool(&pool);
    return e != cudaSuccess ? e : cudaMallocFromPoolAsync(reinterpret_cast<void**>(&base), bytes, pool, 0);
  }
  template <typename T>
  T* at(size_t o) const { return reinterpret_cast<T*>(base + o); }
  ~DevBuf() {
    if (base) cudaFreeAsync(base, 0);
  }
};

sph_status status_of(cudaError_t e) {
  if (e == cudaSuccess) return SPH_OK;
  return e == cudaErrorMemoryAllocation ? SPH_ERR_OOM : SPH_ERR_CUDA;
}

uint64_t splitmix(uint64_t& s) {
  uint64_t z = (s += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

}  // namespace

extern "C" {

sph_status sph_mlp_forward(const float* params, const float* x, uint32_t n, float* out) {
  if (!params || (!x && n) || (!out && n)) return SPH_ERR_INVALID;
  if (n == 0) return SPH_OK;
  DevBuf b;
  const size_t o_p = b.add<float>(MLP_TOTAL), o_w = b.add<MlpPacked>(1), o_x = b.add<float>((size_t)n * MLP_IN),
               o_y = b.add<float>(n), o_f = b.add<unsigned>(1);
  cudaError_t e = b.alloc();
  if (e != cudaSuccess) return status_of(e);
  float *dp = b.at<float>(o_p), *dx = b.at<float>(o_x), *dy = b.at<float>(o_y);
  MlpPacked* w = b.at<MlpPacked>(o_w);
  unsigned* flag = b.at<unsigned>(o_f);
  e = cudaMemcpy(dp, params, MLP_TOTAL * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dx, x, (size_t)n * MLP_IN * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(flag, 0, sizeof(unsigned));
  if (e != cudaSuccess) return status_of(e);
  launch_mlp_pack(dp, w, 0);
  launch_mlp_forward(w, dx, (int)n, dy, flag, 0);
  e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpy(out, dy, (size_t)n * sizeof(float), cudaMemcpyDeviceToHost);
  unsigned timeout = 0;
  if (e == cudaSuccess) e = cudaMemcpy(&timeout, flag, sizeof(unsigned), cudaMemcpyDeviceToHost);
  if (e == cudaSuccess && timeout) return SPH_ERR_TIMEOUT;
  return status_of(e);
}

sph_status sph_mlp_grad(const float* params, const float* x, const float* t, uint32_t n, float* grad, float* loss) {
  if (!params || !x || !t || !grad || !loss || n == 0) return SPH_ERR_INVALID;
  DevBuf b;
  const size_t o_p = b.add<float>(MLP_TOTAL), o_w = b.add<MlpPacked>(1), o_x = b.add<float>((size_t)n * MLP_IN),
               o_t = b.add<float>(n), o_i = b.add<unsigned>(n), o_part = b.add<float>(mlp_part_floats((int)n)),
               o_g = b.add<float>(MLP_TRAIN + 1), o_f = b.add<unsigned>(1);
  cudaError_t e = b.alloc();
  if (e != cudaSuccess) return status_of(e);
  float *dp = b.at<float>(o_p), *dx = b.at<float>(o_x), *dt = b.at<float>(o_t), *part = b.at<float>(o_part),
        *dg = b.at<float>(o_g);  // gradient, then the summed squared error
  MlpPacked* w = b.at<MlpPacked>(o_w);
  unsigned *idx = b.at<unsigned>(o_i), *flag = b.at<unsigned>(o_f);
  std::vector<unsigned> id(n);
  for (uint32_t i = 0; i < n; ++i) id[i] = i;
  e = cudaMemcpy(dp, params, MLP_TOTAL * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dx, x, (size_t)n * MLP_IN * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dt, t, (size_t)n * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(idx, id.data(), (size_t)n * sizeof(unsigned), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(flag, 0, sizeof(unsigned));
  if (e != cudaSuccess) return status_of(e);
  launch_mlp_pack(dp, w, 0);
  launch_mlp_train_batch(w, dx, dt, idx, (int)n, (float)n, part, flag, 0);
  launch_mlp_reduce(part, (int)n, dg, 0);
  e = cudaGetLastError();
  std::vector<float> h(MLP_TRAIN + 1);
  if (e == cudaSuccess) e = cudaMemcpy(h.data(), dg, h.size() * sizeof(float), cudaMemcpyDeviceToHost);
  unsigned timeout = 0;
  if (e == cudaSuccess) e = cudaMemcpy(&timeout, flag, sizeof(unsigned), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return status_of(e);
  if (timeout) return SPH_ERR_TIMEOUT;
  std::memcpy(grad, h.data(), MLP_TRAIN * sizeof(float));
  *loss = h[MLP_TRAIN] / (float)n;
  return SPH_OK;
}

sph_status sph_mlp_train(float* params, const float* x, const float* t, uint32_t n, const sph_mlp_train_cfg* cfg,
                         float* loss_per_epoch) {
  if (!params || !x || !t || !cfg || n == 0 || cfg->batch == 0 || !(cfg->lr > 0.0f)) return SPH_ERR_INVALID;
  std::vector<unsigned> perm(n);
  uint64_t rs = cfg->seed * 0x2545F4914F6CDD1Dull + 1;
  const auto shuffle = [&] {  // Fisher-Yates: a chain of n swaps, about as long as the copies and the steps it overlaps
    for (uint32_t i = n - 1; i > 0; --i) std::swap(perm[i], perm[splitmix(rs) % (i + 1)]);
  };
  for (uint32_t i = 0; i < n; ++i) perm[i] = i;
  std::thread first;  // the first epoch's order, while the inputs go to the device
  if (cfg->epochs) {
    try {
      first = std::thread(shuffle);
    } catch (...) {  // no thread to be had
      shuffle();
    }
  }
  struct Join {
    std::thread& t;
    ~Join() {
      if (t.joinable()) t.join();
    }
  } join{first};
  DevBuf b;
  const int most = (int)(n < cfg->batch ? n : cfg->batch);
  const size_t o_p = b.add<float>(MLP_TOTAL), o_w = b.add<MlpPacked>(1), o_x = b.add<float>((size_t)n * MLP_IN),
               o_t = b.add<float>(n), o_i = b.add<unsigned>(n), o_part = b.add<float>(mlp_part_floats(most)),
               o_m = b.add<float>(MLP_TRAIN), o_v = b.add<float>(MLP_TRAIN), o_l = b.add<float>(1), o_f = b.add<unsigned>(1);
  cudaError_t e = b.alloc();
  if (e != cudaSuccess) return status_of(e);
  float *dp = b.at<float>(o_p), *dx = b.at<float>(o_x), *dt = b.at<float>(o_t), *part = b.at<float>(o_part),
        *dm = b.at<float>(o_m), *dv = b.at<float>(o_v), *dl = b.at<float>(o_l);
  MlpPacked* w = b.at<MlpPacked>(o_w);
  unsigned *idx = b.at<unsigned>(o_i), *flag = b.at<unsigned>(o_f);
  e = cudaMemcpy(dp, params, MLP_TOTAL * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dx, x, (size_t)n * MLP_IN * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemcpy(dt, t, (size_t)n * sizeof(float), cudaMemcpyHostToDevice);
  if (e == cudaSuccess) e = cudaMemset(dm, 0, MLP_TRAIN * sizeof(float));
  if (e == cudaSuccess) e = cudaMemset(dv, 0, MLP_TRAIN * sizeof(float));
  if (e == cudaSuccess) e = cudaMemset(flag, 0, sizeof(unsigned));
  if (e != cudaSuccess) return status_of(e);
  const float b1 = cfg->beta1 > 0.0f ? cfg->beta1 : 0.9f, b2 = cfg->beta2 > 0.0f ? cfg->beta2 : 0.999f;
  const float eps = cfg->eps > 0.0f ? cfg->eps : 1.0e-8f;
  int step = 0;
  launch_mlp_pack(dp, w, 0);
  for (uint32_t ep = 0; ep < cfg->epochs; ++ep) {
    if (first.joinable()) first.join();
    e = cudaMemcpy(idx, perm.data(), (size_t)n * sizeof(unsigned), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemset(dl, 0, sizeof(float));
    if (e != cudaSuccess) return status_of(e);
    for (uint32_t off = 0; off < n; off += cfg->batch) {
      const uint32_t m = n - off < cfg->batch ? n - off : cfg->batch;
      launch_mlp_train_batch(w, dx, dt, idx + off, (int)m, (float)m, part, flag, 0);
      launch_mlp_adam(dp, part, (int)m, dm, dv, w, dl, ++step, cfg->lr, b1, b2, eps, cfg->weight_decay, 0);
    }
    if (ep + 1 < cfg->epochs) shuffle();  // the next epoch's order, while the device works on this one
    float l = 0.0f;
    unsigned timeout = 0;
    e = cudaMemcpy(&l, dl, sizeof(float), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(&timeout, flag, sizeof(unsigned), cudaMemcpyDeviceToHost);
    if (e != cudaSuccess) return status_of(e);
    if (timeout) return SPH_ERR_TIMEOUT;
    if (loss_per_epoch) loss_per_epoch[ep] = l / (float)n;
  }
  e = cudaMemcpy(params, dp, MLP_TRAIN * sizeof(float), cudaMemcpyDeviceToHost);
  return status_of(e);
}

}  // extern "C"
