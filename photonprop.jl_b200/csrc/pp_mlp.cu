// Learned surrogate: MLP 4 -> 128 -> 128 -> 128 -> 5 with GELU, on sm_100a.
//
// A tile is 128 rows (queries).
// The 128 x 128 layers run on the 5th-generation tensor cores: one thread
// issues eight tcgen05.mma (M = N = 128, K = 16, BF16 inputs, FP32
// accumulation in tensor memory) per layer, commits them to an mbarrier, and
// every warp reads its 32 rows back with tcgen05.ld; bias, GELU and the BF16
// conversion of the next layer's operand are fused into that read-back.
//
// Operand tiles live in shared memory in the no-swizzle K-major canonical
// layout: 8-row x 16-byte core matrices, core matrices along K 128 bytes apart
// (leading byte offset), 8-row groups 2048 bytes apart (stride byte offset).
//
// Training: one fused kernel per 128-row tile (forward, masked-MSE loss and
// backward, see train_kernel), then an Adam kernel that updates the FP32
// master weights and their BF16 tensor-core copies.
//
// Every mbarrier wait is bounded (iteration and clock limits); on expiry the
// kernel sets an error flag, stops issuing work and frees its tensor memory.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <string>
#include <vector>

#include "pp_internal.h"
#include "pp_special.cuh"

namespace mlp {

constexpr int H = 128, IN = 4, OUT = 5, TILE = 128, THREADS = 128;
// flat FP32 parameter vector
constexpr int OFF_W1 = 0, OFF_B1 = OFF_W1 + H * IN, OFF_W2 = OFF_B1 + H, OFF_B2 = OFF_W2 + H * H,
              OFF_W3 = OFF_B2 + H, OFF_B3 = OFF_W3 + H * H, OFF_W4 = OFF_B3 + H, OFF_B4 = OFF_W4 + OUT * H,
              N_PARAMS = OFF_B4 + OUT;
constexpr int TILE_BYTES = TILE * H * 2;  // one BF16 128 x 128 operand tile

// element offset of (row, k) in a 128-column K-major canonical tile
__host__ __device__ __forceinline__ int tc_offset(int row, int k) {
  return (((row >> 3) * 16 + (k >> 3)) << 6) + ((row & 7) << 3) + (k & 7);
}

// Training's GELU and its derivative, from one (accurate) tanh.
__device__ __forceinline__ void gelu_both(float z, float& h, float& g) {
  const float u = 0.7978845608028654f * fmaf(0.044715f * z, z * z, z);
  const float t = tanhf(u);
  h = 0.5f * z * (1.f + t);
  const float du = 0.7978845608028654f * fmaf(3.f * 0.044715f, z * z, 1.f);
  g = 0.5f * (1.f + t) + 0.5f * z * (1.f - t * t) * du;
}
// Twice the inference GELU with the MUFU tanh (tanh.approx.f32, relative
// error below 2^-10, under the BF16 rounding that follows it), in four FP32
// operations: u = z (k + k c z^2), 2 GELU = z (1 + t).  The factor 1/2 is
// folded into the next layer's weights (exact: a power of two commutes with
// the BF16 rounding of both the weights and the activations).  Two activations
// at once with sm_100's packed FP32 instructions: half the FP32 issue slots of
// the epilogue.
__device__ __forceinline__ float2 gelu2_fast2(float2 z) {
  constexpr float k0 = 0.7978845608028654f, k1 = 0.7978845608028654f * 0.044715f;
  const float2 k = __ffma2_rn(__fmul2_rn(z, z), make_float2(k1, k1), make_float2(k0, k0));
  const float2 u = __fmul2_rn(z, k);
  float2 t;
  asm("tanh.approx.f32 %0, %1;" : "=f"(t.x) : "f"(u.x));
  asm("tanh.approx.f32 %0, %1;" : "=f"(t.y) : "f"(u.y));
  return __ffma2_rn(z, t, z);
}
__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }

__device__ __forceinline__ uint32_t smem_u32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

// UMMA shared-memory descriptor: no swizzle, K-major, version 1.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((addr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}
// Instruction descriptor: D = F32, A = B = BF16, both K-major, N = 128, M = 128.
constexpr uint32_t kIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((128u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ void mma_commit(uint32_t mbar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar)
               : "memory");
}
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void mbar_init(uint32_t mbar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(mbar) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
// Bounded wait for the given phase parity: about 2^22 polls and ~4e9 cycles.
__device__ __forceinline__ bool mbar_wait(uint32_t mbar, uint32_t parity) {
  const long long t0 = clock64();
  for (int i = 0; i < (1 << 22); ++i) {
    uint32_t done;
    asm volatile(
        "{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.b32 %0, 1, 0, p;\n\t}\n"
        : "=r"(done)
        : "r"(mbar), "r"(parity)
        : "memory");
    if (done) return true;
    if (clock64() - t0 > 4000000000ll) break;
  }
  return false;
}

// Bulk copy of global to shared memory, completing on the mbarrier (its one arrival).
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint32_t mbar) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(mbar), "r"(bytes) : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(mbar)
               : "memory");
}

// 32 FP32 accumulator columns [col, col+32) of this thread's row.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]),
        "=r"(r[23]), "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]),
        "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// Tensor-memory allocation of COLS columns by warp 0; the address lands in *slot.
template <int COLS>
__device__ __forceinline__ void tmem_alloc(uint32_t* slot) {
  if ((threadIdx.x >> 5) == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "n"(COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
}
template <int COLS>
__device__ __forceinline__ void tmem_free(uint32_t taddr) {
  if ((threadIdx.x >> 5) == 0)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "n"(COLS));
}

// Writes 8 consecutive columns [k8*8, k8*8+8) of `row` (FP32 values, rounded
// to BF16) into a canonical tile with one 16-byte store.
__device__ __forceinline__ void store8(__nv_bfloat16* tile, int row, int k8, const float* v) {
  __align__(16) __nv_bfloat162 p[4];
#pragma unroll
  for (int i = 0; i < 4; ++i) p[i] = __floats2bfloat162_rn(v[2 * i], v[2 * i + 1]);
  *reinterpret_cast<int4*>(tile + tc_offset(row, k8 * 8)) = *reinterpret_cast<int4*>(p);
}

// element offset of (row, k) in a K-major canonical tile of 16 columns
__host__ __device__ __forceinline__ int tc16_offset(int row, int k) {
  return (((row >> 3) * 2 + (k >> 3)) << 6) + ((row & 7) << 3) + (k & 7);
}
// Instruction descriptor for N = 16 (the padded output layer).
constexpr uint32_t kIdescN16 = (1u << 4) | (1u << 7) | (1u << 10) | ((16u >> 3) << 17) | ((128u >> 4) << 24);
__device__ __forceinline__ void mma_idesc(uint32_t tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, {%5, %6, %7, %8}, p;\n\t}\n" ::"r"(tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(acc), "r"(0u), "r"(0u), "r"(0u), "r"(0u));
}
// 16 FP32 accumulator columns [col, col+16) of this thread's row.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

// ---------------------------------------------------------------------------
// Device parameter block.
struct DevParams {
  const float* p;        // FP32 master parameters (N_PARAMS)
  const __nv_bfloat16* w2tc;  // W2, W3 as canonical tiles (rows = out, columns = in): the B operand of
  const __nv_bfloat16* w3tc;  // h W^T read K-major, and of dz W read MN-major
  const __nv_bfloat16* w2h;   // W2 / 2, W3 / 2: inference B operands (they take 2 GELU)
  const __nv_bfloat16* w3h;
  const __nv_bfloat16* w1tc;  // W1 as the B operand of x W1^T: 128 rows x K 16 (4 used, then b1 in two)
  const __nv_bfloat16* w4tc;  // W4 / 2 as the B operand of h W4^T: 16 rows (5 used) x K 128
  const float* norm;     // x_mean[4], x_std[4], y_mean[5], y_std[5]
  int* error;
};

// Cooperative copy of a 32 KB canonical tile from global to shared memory.
__device__ __forceinline__ void load_tile(__nv_bfloat16* dst, const __nv_bfloat16* src) {
  const int4* s = reinterpret_cast<const int4*>(src);
  int4* d = reinterpret_cast<int4*>(dst);
  for (int i = threadIdx.x; i < TILE_BYTES / 16; i += blockDim.x) d[i] = s[i];
}

// ---------------------------------------------------------------------------
// Inference: persistent over 128-row tiles.  x [n][4] raw features; out
// [5][n] (structure of arrays): raw = the de-standardised network outputs
// (ln(mu/N), logit w, ln a1, ln a2, ln theta); physical = (mu, w, a1, a2, theta).
//
// One CTA per SM with kGroups independent groups of 128 threads (four
// warps, one query row per thread).  The groups share the BF16 weight tiles
// of layers 2 and 3 in shared memory; each owns an activation tile, an
// mbarrier and 128 of the CTA's TMEM columns, and walks its own sequence of
// row tiles with group-local named barriers.  While one group's MMAs run on
// the tensor cores the others run their GELU epilogues on the FP32 and MUFU
// pipes, and sixteen warps per SM keep those pipes busy.  The biases of the
// hidden layers are added by the tensor cores and the GELU's factor 1/2 sits
// in the next layer's weights, so an activation costs four FP32 operations,
// one tanh and half a BF16 pack.
constexpr int kGroups = 4, INFER_THREADS = kGroups * THREADS;

__device__ __forceinline__ void group_sync(int g) {
  asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "r"(THREADS) : "memory");
}
// Group barrier that also ANDs a flag over the group's threads, so that every
// thread of the group takes the same branch after a bounded wait.
__device__ __forceinline__ bool group_all(int g, bool v) {
  uint32_t r;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\tbar.red.and.pred q, %2, %3, p;\n\t"
      "selp.u32 %0, 1, 0, q;\n\t}\n"
      : "=r"(r)
      : "r"((uint32_t)v), "r"(g + 1), "r"(THREADS)
      : "memory");
  return r != 0;
}

// The group's MMAs of one layer; kind 1: x (128 x 16) W1^T, one MMA (the
// bias rides in K columns 4 and 5: x has ones there, W1 the bias split into
// BF16 hi and lo); kind 2: h (128 x 128) W^T, eight MMAs, then a ninth,
// ones (128 x 16) times the bias tile, that adds the bias in the
// accumulator; kind 4: h W4^T with N = 16.  The epilogues then read z with
// its bias and spend no FP32 add on it.
__device__ __forceinline__ bool group_layer(int kind, const __nv_bfloat16* a, const __nv_bfloat16* b, uint32_t tmem,
                                            uint32_t mbar, uint32_t& parity, int g, int gt,
                                            const __nv_bfloat16* ones = nullptr,
                                            const __nv_bfloat16* bias = nullptr) {
  fence_async_smem();
  tc_fence_before();
  group_sync(g);
  tc_fence_after();
  if (gt == 0) {
    const uint32_t sa = smem_u32(a), sb = smem_u32(b);
    if (kind == 1) {
      mma_idesc(tmem, smem_desc(sa, 128, 256), smem_desc(sb, 128, 256), kIdesc, 0u);
    } else {
      const uint32_t idesc = kind == 4 ? kIdescN16 : kIdesc;
#pragma unroll
      for (int k = 0; k < 8; ++k)
        mma_idesc(tmem, smem_desc(sa + k * 256, 128, 2048), smem_desc(sb + k * 256, 128, 2048), idesc, k > 0);
      if (kind == 2)  // + 1 (bias hi, bias lo): the layer's bias, one more K = 16 step
        mma_idesc(tmem, smem_desc(smem_u32(ones), 128, 256), smem_desc(smem_u32(bias), 128, 256), kIdesc, 1u);
    }
    mma_commit(mbar);
  }
  const bool ok = group_all(g, mbar_wait(mbar, parity));
  parity ^= 1u;
  tc_fence_after();
  return ok;
}

__global__ void __launch_bounds__(INFER_THREADS, 1) infer_kernel(DevParams P, const float* __restrict__ x,
                                                                float* __restrict__ out, int64_t n, int physical) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __nv_bfloat16* w2 = reinterpret_cast<__nv_bfloat16*>(smem_raw);
  __nv_bfloat16* w3 = w2 + TILE * H;
  __nv_bfloat16* w1t = w3 + TILE * H;   // 128 x 16: W1 in K 0..3, b1 (hi, lo) in K 4, 5
  __nv_bfloat16* w4t = w1t + H * 16;    // 16 x 128
  __nv_bfloat16* b2t = w4t + 16 * H;    // 128 x 16: b2 (hi, lo) in K 0, 1
  __nv_bfloat16* b3t = b2t + H * 16;
  __nv_bfloat16* ones = b3t + H * 16;   // 128 x 16: 1 in K 0, 1
  __nv_bfloat16* acts = ones + TILE * 16;  // kGroups activation tiles (the x tile is the first 4 KB of one)
  float* b4 = reinterpret_cast<float*>(acts + kGroups * TILE * H);
  float* nrm = b4 + 8;
  uint64_t* mbars = reinterpret_cast<uint64_t*>(nrm + 24);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(mbars + kGroups + 2);

  const int t = threadIdx.x;
  const int g = t >> 7, gt = t & (THREADS - 1);  // group, thread (= row) within the group
  // the weight tiles (W1, W4, b2, b3 contiguous, then W2 and W3), as bulk
  // copies that the first tile's layers wait for
  const uint32_t mb_narrow = smem_u32(mbars + kGroups), mb_wide = smem_u32(mbars + kGroups + 1);
  if (t == 0) {
    for (int i = 0; i < kGroups + 2; ++i) mbar_init(smem_u32(mbars + i));
    bulk_load(w1t, P.w1tc, 4 * H * 16 * 2, mb_narrow);
    bulk_load(w2, P.w2h, 2 * TILE_BYTES, mb_wide);
  }
  for (int i = t; i < TILE * 16 / 8; i += INFER_THREADS) {  // the ones tile, 8 columns per 16-byte word
    const int row = i >> 1, k8 = i & 1;
    const uint32_t one2 = 0x3F803F80u;  // two BF16 ones
    *reinterpret_cast<int4*>(ones + tc16_offset(row, k8 * 8)) =
        k8 == 0 ? make_int4((int)one2, 0, 0, 0) : make_int4(0, 0, 0, 0);
  }
  if (t < OUT) b4[t] = P.p[OFF_B4 + t];
  if (t < 18) nrm[t] = P.norm[t];
  if (t < IN) nrm[18 + t] = 1.f / P.norm[4 + t];  // feature scales as reciprocals: no division per row
  tmem_alloc<512>(tslot);  // 128 columns per group
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tslot;
  const uint32_t tmem = tmem_base + (uint32_t)(g * 128);           // the group's columns
  const uint32_t taddr = tmem + ((uint32_t)(gt & ~31) << 16);      // this warp's 32 lanes
  __nv_bfloat16* act = acts + g * TILE * H;
  const uint32_t mb = smem_u32(mbars + g);
  uint32_t parity = 0;
  bool ok = true;

  // whole rounds of the grid take neighbouring tiles to a block's groups; what
  // is left goes to the blocks first and to their groups second, so that a few
  // thousand queries have an SM per tile (3001 queries: four tiles on each of
  // six SMs 16.6 us, one tile on each of 24 SMs 10.2 us per call; whole rounds
  // in that order: 1 % slower at 6e5 to 1.7e6 queries)
  const int64_t tile_step = (int64_t)gridDim.x * kGroups, whole = n / TILE / tile_step * tile_step;
  const int64_t last = whole + blockIdx.x + (int64_t)g * gridDim.x;
  const int64_t tile0 = whole > 0 ? (int64_t)blockIdx.x * kGroups + g : last;
  // the row's features, loaded one tile ahead so that the global loads
  // overlap the previous tile's layers
  float xr[IN];
  {
    const int64_t row0 = tile0 * TILE + gt;
#pragma unroll
    for (int j = 0; j < IN; ++j) xr[j] = row0 < n ? x[row0 * IN + j] : nrm[j];
  }
  if (tile0 * TILE < n) ok = group_all(g, mbar_wait(mb_narrow, 0));
  bool wide = false;  // W2 and W3 are here
  int64_t next;
  for (int64_t tile = tile0; ok && tile * TILE < n; tile = next) {
    // from the last round on the step leads past the end
    next = tile + tile_step;
    if (tile < whole && next >= whole) next = last;
    const int64_t row = tile * TILE + gt;
    const bool valid = row < n;
    float xn[8];
    float lnN = 0.f;
#pragma unroll
    for (int j = 0; j < IN; ++j) {
      const float raw = xr[j];
      if (j == 2) lnN = raw * 2.302585092994046f;
      xn[j] = (raw - nrm[j]) * nrm[18 + j];
    }
    {
      const int64_t nrow = next * TILE + gt;
#pragma unroll
      for (int j = 0; j < IN; ++j) xr[j] = nrow < n ? x[nrow * IN + j] : nrm[j];
    }
    xn[IN] = 1.f;  // times the bias columns of W1
    xn[IN + 1] = 1.f;
#pragma unroll
    for (int j = IN + 2; j < 8; ++j) xn[j] = 0.f;
    // layer 1 (tensor cores, K = 4 padded to 16): the row's x in the x tile
    {
      __align__(16) __nv_bfloat162 p[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) p[i] = __floats2bfloat162_rn(xn[2 * i], xn[2 * i + 1]);
      *reinterpret_cast<int4*>(act + tc16_offset(gt, 0)) = *reinterpret_cast<int4*>(p);
      *reinterpret_cast<int4*>(act + tc16_offset(gt, 8)) = make_int4(0, 0, 0, 0);
    }
    ok = group_layer(1, act, w1t, tmem, mb, parity, g, gt);
    if (!ok) break;
    for (int c = 0; c < 4; ++c) {
      float v[32];
      tmem_ld32(taddr + c * 32, v);
#pragma unroll
      for (int i = 0; i < 32; i += 2) {
        const float2 r = gelu2_fast2(make_float2(v[i], v[i + 1]));
        v[i] = r.x;
        v[i + 1] = r.y;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) store8(act, gt, c * 4 + q, v + q * 8);
    }
    // layer 2
    if (!wide) {
      ok = group_all(g, mbar_wait(mb_wide, 0));
      if (!ok) break;
      wide = true;
    }
    ok = group_layer(2, act, w2, tmem, mb, parity, g, gt, ones, b2t);
    if (!ok) break;
    for (int c = 0; c < 4; ++c) {
      float v[32];
      tmem_ld32(taddr + c * 32, v);
#pragma unroll
      for (int i = 0; i < 32; i += 2) {
        const float2 r = gelu2_fast2(make_float2(v[i], v[i + 1]));
        v[i] = r.x;
        v[i + 1] = r.y;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) store8(act, gt, c * 4 + q, v + q * 8);
    }
    // layer 3
    ok = group_layer(2, act, w3, tmem, mb, parity, g, gt, ones, b3t);
    if (!ok) break;
    for (int c = 0; c < 4; ++c) {
      float v[32];
      tmem_ld32(taddr + c * 32, v);
#pragma unroll
      for (int i = 0; i < 32; i += 2) {
        const float2 r = gelu2_fast2(make_float2(v[i], v[i + 1]));
        v[i] = r.x;
        v[i + 1] = r.y;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) store8(act, gt, c * 4 + q, v + q * 8);
    }
    // layer 4 (tensor cores, N = 5 padded to 16)
    ok = group_layer(4, act, w4t, tmem, mb, parity, g, gt);
    if (!ok) break;
    float y[16];
    tmem_ld16(taddr, y);
    if (valid) {
#pragma unroll
      for (int j = 0; j < OUT; ++j) {
        float o = fmaf(y[j] + b4[j], nrm[13 + j], nrm[8 + j]);
        if (physical) {
          if (j == 0) o = expf(o + lnN);
          else if (j == 1) o = 1.f / (1.f + expf(-o));
          else o = expf(o);
        }
        out[(int64_t)j * n + row] = o;
      }
    }
  }
  if (!ok && gt == 0) {
    atomicExch(P.error, 1);
    mbar_wait(mb_narrow, 0);  // the block's copies in flight
    mbar_wait(mb_wide, 0);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  tmem_free<512>(tmem_base);
}

// ---------------------------------------------------------------------------
// Training.  count_kernel zeroes the gradients and the loss and sums the mask
// in FP64 (kCountBlocks partial sums, added in one order by every reader);
// train_kernel adds a tile's gradients; adam_kernel applies them.
constexpr int kCountBlocks = 32;
// What a step brings back: the gradients, the loss sum, the error flag, the mask sums (doubles).
constexpr int kPartAt = (N_PARAMS + 3) & ~1, kBack = kPartAt + 2 * kCountBlocks;

__global__ void __launch_bounds__(256) count_kernel(const float* __restrict__ mask, int64_t count,
                                                    float* __restrict__ grad, double* __restrict__ part) {
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int64_t first = (int64_t)blockIdx.x * blockDim.x + threadIdx.x, stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = first; i < N_PARAMS + 1; i += stride) grad[i] = 0.f;  // and the loss
  double s = 0.0;
  for (int64_t i = first; i < count; i += stride) s += (double)mask[i];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  __shared__ double warp[8];
  if ((threadIdx.x & 31u) == 0) warp[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < 8; ++w) t += warp[w];
    part[blockIdx.x] = t;
  }
}

// FP32 columns [0, 32) to this thread's row of tensor memory.
__device__ __forceinline__ void tmem_st32(uint32_t taddr, const float* v) {
  asm volatile(
      "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,"
      "%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(taddr),
      "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]), "f"(v[9]),
      "f"(v[10]), "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15]), "f"(v[16]), "f"(v[17]), "f"(v[18]),
      "f"(v[19]), "f"(v[20]), "f"(v[21]), "f"(v[22]), "f"(v[23]), "f"(v[24]), "f"(v[25]), "f"(v[26]), "f"(v[27]),
      "f"(v[28]), "f"(v[29]), "f"(v[30]), "f"(v[31]));
  asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

// Sums of 32 values over the 32 lanes of a warp: lane l returns the sum of
// v[l] (31 shuffles: each halving step keeps one half of the values and adds
// the partner's).
__device__ __forceinline__ float warp_column_sum(float* v) {
  const unsigned lane = threadIdx.x & 31u;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool upper = lane & o;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const float keep = upper ? v[i + o] : v[i], give = upper ? v[i] : v[i + o];
      v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
    }
  }
  return v[0];
}

// Adds a 512-byte row of FP32 in shared memory to global memory.
__device__ __forceinline__ void bulk_add_row(float* dst, const void* src) {
  asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.f32 [%0], [%1], 512;" ::"l"(dst),
               "r"(smem_u32(src))
               : "memory");
}

// The k-th 16 of K of an operand tile: read K-major, or as MN-major (neighbouring
// 8-column groups 128 B apart, 8-row groups, K then, 2048 B).
__device__ __forceinline__ uint64_t kmaj(const __nv_bfloat16* tile, int k) {
  return smem_desc(smem_u32(tile) + k * 256, 128, 2048);
}
__device__ __forceinline__ uint64_t mn(const __nv_bfloat16* tile, int k) {
  return smem_desc(smem_u32(tile) + k * 4096, 2048, 128);
}
// A and B both MN-major (bits 15 and 16), or B alone.
constexpr uint32_t kIdescMnMn = kIdesc | (1u << 15) | (1u << 16), kIdescKMn = kIdesc | (1u << 16);

// One CTA of 512 threads per 128-row tile.  xn [n][4] standardised features,
// yt [n][5] standardised targets, mask [n][5]; grad (N_PARAMS, then the loss
// sum) accumulated with atomics; loss += sum of mask * (y - t)^2.
//
// Warp w holds the tile's rows 32 (w mod 4) .. + 31 (its tensor-memory lanes),
// one per lane, and columns 32 (w / 4) .. + 31 of every layer.  Nothing goes
// through global memory between layers: the activations h1, h2 stay in shared
// memory as BF16 operand tiles, and the GELU derivatives of all three layers,
// computed in the forward pass from the same tanh, in tensor memory (three
// quarters of it; the fourth holds weight gradients, and a layer's quarter
// takes its dh once its derivative is read).  An operand tile has 8 x 8 core
// matrices, so one tile serves as a K-major operand in the forward pass and
// MN-major in the backward pass (dW = dz^T h, dh = dz W): nothing is
// transposed.  Bias gradients are warp column sums, the weight gradients go
// from tensor memory through padded shared rows to global memory as bulk
// additions of 512 bytes.
//
// What bounds it: three dependent layers forward and three back on one SM,
// with 96 accurate tanh per thread (4096 rows are 32 CTAs).  Before, one warp
// per 32 rows walked 128 columns with all activations in global memory and
// every thread adding its bias gradients to the same addresses: 950-1080 us
// for 4096 rows (32 tiles), now 36 us.
constexpr int TRAIN_THREADS = 512;
constexpr int kGradPitch = 528;  // bytes of a staged gradient row: 16-byte lanes of 8 rows fall on different banks

__global__ void __launch_bounds__(TRAIN_THREADS, 1) train_kernel(DevParams P, const float* __restrict__ xn,
                                                                const float* __restrict__ yt,
                                                                const float* __restrict__ mask, int64_t n,
                                                                const double* part, float* grad) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  // W2 H1 W3 H2 DZ3 DZ2, 32 KB each; reused as they fall free:
  unsigned char* const base = smem_raw;
  __nv_bfloat16* w2 = reinterpret_cast<__nv_bfloat16*>(base);
  __nv_bfloat16* h1 = reinterpret_cast<__nv_bfloat16*>(base + TILE_BYTES);
  __nv_bfloat16* w3 = reinterpret_cast<__nv_bfloat16*>(base + 2 * TILE_BYTES);
  __nv_bfloat16* h2 = reinterpret_cast<__nv_bfloat16*>(base + 3 * TILE_BYTES);
  __nv_bfloat16* dz3 = reinterpret_cast<__nv_bfloat16*>(base + 4 * TILE_BYTES);
  __nv_bfloat16* dz2 = reinterpret_cast<__nv_bfloat16*>(base + 5 * TILE_BYTES);
  unsigned char* const h3s = base + 5 * TILE_BYTES;         // h3, BF16 rows, until dz2
  unsigned char* const gw3 = base + 2 * TILE_BYTES + 2048;  // dW3 rows, once w3, h2 and dz3 are free
  unsigned char* const gw2 = base;                          // dW2 rows, once w2 and h1 are free (to 2 KB into w3)
  unsigned char* const dz1s = base + 4 * TILE_BYTES;        // dz1, FP32 rows, once dz3 and dz2 are free: 64 KB
  static_assert(2048 + TILE * kGradPitch <= 3 * TILE_BYTES && TILE * kGradPitch <= 2 * TILE_BYTES + 2048,
                "staged gradients fit the tiles they replace");
  float* w1 = reinterpret_cast<float*>(base + 6 * TILE_BYTES);  // [128][4]
  float* w4 = w1 + H * IN;                                      // [128][8], 5 used
  float* dys = w4 + H * 8;                                      // [128][8], 5 used
  float* xs = dys + TILE * 8;                                   // [128][4], BF16-rounded
  float* b123 = xs + TILE * IN;                                 // [3][128]
  uint64_t* mbar = reinterpret_cast<uint64_t*>(b123 + 3 * H);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(mbar + 1);

  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const int r = (warp & 3) * 32 + lane, c0 = (warp >> 2) * 32;  // this thread's row and first column
  const int64_t row = (int64_t)blockIdx.x * TILE + r;
  const bool valid = row < n;
  load_tile(w2, P.w2tc);
  load_tile(w3, P.w3tc);
  for (int i = t; i < H * IN; i += TRAIN_THREADS) w1[i] = bf16r(P.p[OFF_W1 + i]);
  for (int i = t; i < OUT * H; i += TRAIN_THREADS) w4[(i % H) * 8 + i / H] = bf16r(P.p[OFF_W4 + i]);
  if (t < H) {
    b123[t] = P.p[OFF_B1 + t];
    b123[H + t] = P.p[OFF_B2 + t];
    b123[2 * H + t] = P.p[OFF_B3 + t];
  }
  float x[IN];
#pragma unroll
  for (int j = 0; j < IN; ++j) x[j] = valid ? bf16r(xn[row * IN + j]) : 0.f;
  if (c0 == 0) *reinterpret_cast<float4*>(xs + r * IN) = make_float4(x[0], x[1], x[2], x[3]);
  if (t == 0) mbar_init(smem_u32(mbar));
  tmem_alloc<512>(tslot);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tm = *tslot;  // g1 [0, 128), g2 / dh1 [128, 256), g3 / dh2 [256, 384), dW [384, 512)
  const uint32_t ta = tm + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)c0;  // this thread's lanes and columns
  const uint32_t mb = smem_u32(mbar);
  uint32_t parity = 0;
  bool ok = true;
  // every thread's shared-memory writes and tensor-memory reads before the MMAs that thread 0 issues next
  auto handover = [&]() {
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
  };
  auto finished = [&]() {  // the MMAs committed last, or a wait that expired, for all threads alike
    const bool w = mbar_wait(mb, parity);
    parity ^= 1u;
    ok = __syncthreads_and(w);
    tc_fence_after();
    return ok;
  };
  // one layer's activations: z (this thread's 32 columns) to h and, in place, g
  auto activate = [&](float* z, float* h) {
#pragma unroll
    for (int i = 0; i < 32; ++i) gelu_both(z[i], h[i], z[i]);
  };
  auto store_tile = [&](__nv_bfloat16* tile, const float* v) {
#pragma unroll
    for (int q = 0; q < 4; ++q) store8(tile, r, c0 / 8 + q, v + q * 8);
  };

  // ---- forward
  {
    float z[32], h[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) {
      const float4 w = *reinterpret_cast<const float4*>(w1 + (c0 + i) * IN);
      z[i] = fmaf(w.w, x[3], fmaf(w.z, x[2], fmaf(w.y, x[1], fmaf(w.x, x[0], b123[c0 + i]))));
    }
    activate(z, h);
    tmem_st32(ta, z);
    store_tile(h1, h);
  }
  handover();
  if (t == 0) {
    for (int k = 0; k < 8; ++k) mma_idesc(tm + 128, kmaj(h1, k), kmaj(w2, k), kIdesc, k > 0);
    mma_commit(mb);
  }
  if (finished()) {
    float z[32], h[32];
    tmem_ld32(ta + 128, z);
#pragma unroll
    for (int i = 0; i < 32; ++i) z[i] += b123[H + c0 + i];
    activate(z, h);
    tmem_st32(ta + 128, z);
    store_tile(h2, h);
    handover();
    if (t == 0) {
      for (int k = 0; k < 8; ++k) mma_idesc(tm + 256, kmaj(h2, k), kmaj(w3, k), kIdesc, k > 0);
      mma_commit(mb);
    }
  }
  // BF16 rows of h3, the 16-byte words of a row permuted by its low bits (no bank conflicts by row or by column)
  auto h3_at = [&](int rr, int word) { return h3s + rr * 256 + ((word ^ (rr & 7)) << 4); };
  if (ok && finished()) {
    float z[32], h[32];
    tmem_ld32(ta + 256, z);
#pragma unroll
    for (int i = 0; i < 32; ++i) z[i] += b123[2 * H + c0 + i];
    activate(z, h);
    tmem_st32(ta + 256, z);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      __align__(16) __nv_bfloat162 b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) b[i] = __floats2bfloat162_rn(h[q * 8 + 2 * i], h[q * 8 + 2 * i + 1]);
      *reinterpret_cast<int4*>(h3_at(r, c0 / 8 + q)) = *reinterpret_cast<int4*>(b);
    }
    __syncthreads();
    // ---- output layer, loss and output gradient: one row per thread of the first four warps
    asm volatile("griddepcontrol.wait;" ::: "memory");  // count_kernel: mask sum, zeroed gradients
    double cnt = 0.0;
    for (int i = 0; i < kCountBlocks; ++i) cnt += part[i];
    const float inv_count = cnt > 0.0 ? (float)(1.0 / cnt) : 0.f;
    if (t < TILE) {
      float y[OUT];
#pragma unroll
      for (int j = 0; j < OUT; ++j) y[j] = P.p[OFF_B4 + j];
      for (int q = 0; q < 16; ++q) {
        const int4 b = *reinterpret_cast<const int4*>(h3_at(r, q));
        const __nv_bfloat162* hb = reinterpret_cast<const __nv_bfloat162*>(&b);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const float hv = i & 1 ? __high2float(hb[i / 2]) : __low2float(hb[i / 2]);
          const float4 w = *reinterpret_cast<const float4*>(w4 + (q * 8 + i) * 8);
          y[0] = fmaf(w.x, hv, y[0]);
          y[1] = fmaf(w.y, hv, y[1]);
          y[2] = fmaf(w.z, hv, y[2]);
          y[3] = fmaf(w.w, hv, y[3]);
          y[4] = fmaf(w4[(q * 8 + i) * 8 + 4], hv, y[4]);
        }
      }
      float lsum = 0.f;
#pragma unroll
      for (int j = 0; j < OUT; ++j) {
        const float m = valid ? mask[row * OUT + j] : 0.f;
        const float e = valid ? y[j] - yt[row * OUT + j] : 0.f;
        lsum += m * e * e;
        dys[r * 8 + j] = 2.f * m * e * inv_count;
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) lsum += __shfl_xor_sync(0xffffffffu, lsum, o);
      if (lane == 0) atomicAdd(grad + N_PARAMS, lsum);
    }
    __syncthreads();
    // dW4, db4: feature f over a quarter of the rows
    {
      const int f = t & (H - 1), r0 = (t >> 7) * 32;
      float acc[OUT] = {0.f, 0.f, 0.f, 0.f, 0.f}, s = 0.f;
#pragma unroll 4
      for (int rr = r0; rr < r0 + 32; ++rr) {
        const float hv = __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(h3_at(rr, f >> 3) + (f & 7) * 2));
        const float4 d = *reinterpret_cast<const float4*>(dys + rr * 8);
        const float d4 = dys[rr * 8 + 4];
        acc[0] = fmaf(d.x, hv, acc[0]);
        acc[1] = fmaf(d.y, hv, acc[1]);
        acc[2] = fmaf(d.z, hv, acc[2]);
        acc[3] = fmaf(d.w, hv, acc[3]);
        acc[4] = fmaf(d4, hv, acc[4]);
        if (f < OUT) s += dys[rr * 8 + f];
      }
#pragma unroll
      for (int j = 0; j < OUT; ++j) atomicAdd(grad + OFF_W4 + j * H + f, acc[j]);
      if (f < OUT) atomicAdd(grad + OFF_B4 + f, s);
    }
    // ---- backward: dz3 = (dy W4) * g3
    {
      float g[32];
      tmem_ld32(ta + 256, g);
      const float4 d = *reinterpret_cast<const float4*>(dys + r * 8);
      const float d4 = dys[r * 8 + 4];
#pragma unroll
      for (int i = 0; i < 32; ++i) {
        const float4 w = *reinterpret_cast<const float4*>(w4 + (c0 + i) * 8);
        float dh = fmaf(d.x, w.x, 0.f);
        dh = fmaf(d.y, w.y, dh);
        dh = fmaf(d.z, w.z, dh);
        dh = fmaf(d.w, w.w, dh);
        dh = fmaf(d4, w4[(c0 + i) * 8 + 4], dh);
        g[i] = valid ? dh * g[i] : 0.f;
      }
      store_tile(dz3, g);
      atomicAdd(grad + OFF_B3 + c0 + lane, warp_column_sum(g));
    }
    handover();
    if (t == 0) {  // dW3 = dz3^T h2 and dh2 = dz3 W3
      for (int k = 0; k < 8; ++k) mma_idesc(tm + 256, kmaj(dz3, k), mn(w3, k), kIdescKMn, k > 0);
      for (int k = 0; k < 8; ++k) mma_idesc(tm + 384, mn(dz3, k), mn(h2, k), kIdescMnMn, k > 0);
      mma_commit(mb);
    }
  }
  if (ok && finished()) {
    {
      float v[32], g[32];
      tmem_ld32(ta + 256, v);
      tmem_ld32(ta + 128, g);
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = valid ? v[i] * g[i] : 0.f;
      store_tile(dz2, v);
      atomicAdd(grad + OFF_B2 + c0 + lane, warp_column_sum(v));
      tmem_ld32(ta + 384, v);
#pragma unroll
      for (int q = 0; q < 8; ++q)
        *reinterpret_cast<float4*>(gw3 + r * kGradPitch + (c0 + 4 * q) * 4) =
            make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
    }
    handover();
    if (t == 0) {  // dh1 = dz2 W2 and dW2 = dz2^T h1
      for (int k = 0; k < 8; ++k) mma_idesc(tm + 128, kmaj(dz2, k), mn(w2, k), kIdescKMn, k > 0);
      for (int k = 0; k < 8; ++k) mma_idesc(tm + 384, mn(dz2, k), mn(h1, k), kIdescMnMn, k > 0);
      mma_commit(mb);
    }
    if (t >= TRAIN_THREADS - TILE) {
      const int o = t - (TRAIN_THREADS - TILE);
      bulk_add_row(grad + OFF_W3 + o * H, gw3 + o * kGradPitch);
      asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // dz1 and dW2 are staged over it next
    }
    if (finished()) {
      float v[32], g[32];
      tmem_ld32(ta + 128, v);
      tmem_ld32(ta, g);
#pragma unroll
      for (int q = 0; q < 8; ++q) {  // dz1 rows, their 16-byte words permuted like those of h3
        float d[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) d[i] = valid ? v[4 * q + i] * g[4 * q + i] : 0.f;
        *reinterpret_cast<float4*>(dz1s + r * 512 + (((c0 / 4 + q) ^ (r & 7)) << 4)) =
            make_float4(d[0], d[1], d[2], d[3]);
      }
      tmem_ld32(ta + 384, v);
#pragma unroll
      for (int q = 0; q < 8; ++q)
        *reinterpret_cast<float4*>(gw2 + r * kGradPitch + (c0 + 4 * q) * 4) =
            make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
      handover();
      if (t >= TRAIN_THREADS - TILE) {
        const int o = t - (TRAIN_THREADS - TILE);
        bulk_add_row(grad + OFF_W2 + o * H, gw2 + o * kGradPitch);
        asm volatile("cp.async.bulk.commit_group;" ::: "memory");
      }
      // dW1, db1: feature f over a quarter of the rows
      const int f = t & (H - 1), r0 = (t >> 7) * 32;
      float a0 = 0.f, a1 = 0.f, a2 = 0.f, a3 = 0.f, s = 0.f;
#pragma unroll 4
      for (int rr = r0; rr < r0 + 32; ++rr) {
        const float d = *reinterpret_cast<const float*>(dz1s + rr * 512 + (((f >> 2) ^ (rr & 7)) << 4) + (f & 3) * 4);
        const float4 xr = *reinterpret_cast<const float4*>(xs + rr * IN);
        a0 = fmaf(d, xr.x, a0);
        a1 = fmaf(d, xr.y, a1);
        a2 = fmaf(d, xr.z, a2);
        a3 = fmaf(d, xr.w, a3);
        s += d;
      }
      atomicAdd(grad + OFF_W1 + f * IN + 0, a0);
      atomicAdd(grad + OFF_W1 + f * IN + 1, a1);
      atomicAdd(grad + OFF_W1 + f * IN + 2, a2);
      atomicAdd(grad + OFF_W1 + f * IN + 3, a3);
      atomicAdd(grad + OFF_B1 + f, s);
    }
    if (t >= TRAIN_THREADS - TILE) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  }
  if (!ok && t == 0) atomicExch(P.error, 1);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  tmem_free<512>(tm);
}

// The BF16 copies of the master parameters that the tensor cores read.
struct Copies {
  __nv_bfloat16 *w2tc, *w3tc, *w2h, *w3h, *w1tc, *w4tc, *b2t, *b3t;
};

// Writes the copies of parameter i, of value v (the tiles' padding is zeroed
// once, at creation).
__device__ __forceinline__ void write_copies(const Copies& C, int i, float v) {
  auto split = [&](__nv_bfloat16* tile, int o, int k) {  // a bias as two BF16 columns, hi + lo = b to about 2^-16 relative
    const __nv_bfloat16 hi = __float2bfloat16_rn(v);
    tile[tc16_offset(o, k)] = hi;
    tile[tc16_offset(o, k + 1)] = __float2bfloat16_rn(v - __bfloat162float(hi));
  };
  if (i < OFF_B1) {
    C.w1tc[tc16_offset(i / IN, i % IN)] = __float2bfloat16_rn(v);
  } else if (i < OFF_W2) {
    split(C.w1tc, i - OFF_B1, IN);
  } else if (i < OFF_B2) {
    const int at = tc_offset((i - OFF_W2) / H, (i - OFF_W2) % H);
    C.w2tc[at] = __float2bfloat16_rn(v);
    C.w2h[at] = __float2bfloat16_rn(0.5f * v);
  } else if (i < OFF_W3) {
    split(C.b2t, i - OFF_B2, 0);
  } else if (i < OFF_B3) {
    const int at = tc_offset((i - OFF_W3) / H, (i - OFF_W3) % H);
    C.w3tc[at] = __float2bfloat16_rn(v);
    C.w3h[at] = __float2bfloat16_rn(0.5f * v);
  } else if (i < OFF_W4) {
    split(C.b3t, i - OFF_B3, 0);
  } else if (i < OFF_B4) {
    C.w4tc[tc_offset((i - OFF_W4) / H, (i - OFF_W4) % H)] = __float2bfloat16_rn(0.5f * v);
  }
}

// Adam on the FP32 master parameters, and their BF16 copies.
__global__ void __launch_bounds__(256) adam_kernel(float* __restrict__ p, const float* g,
                                                   float* __restrict__ m, float* __restrict__ v, const Copies C,
                                                   float lr, float b1, float b2, float eps, float c1, float c2) {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= N_PARAMS) return;
  const float gi = g[i];
  const float mi = b1 * m[i] + (1.f - b1) * gi;
  const float vi = b2 * v[i] + (1.f - b2) * gi * gi;
  m[i] = mi;
  v[i] = vi;
  const float w = p[i] - lr * (mi * c1) / (sqrtf(vi * c2) + eps);
  p[i] = w;
  write_copies(C, i, w);
}

__global__ void __launch_bounds__(256) prepare_kernel(const float* __restrict__ p, const Copies C) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < N_PARAMS) write_copies(C, i, p[i]);
}

// One 128 x 128 x 128 GEMM with the descriptors that training uses, a and b
// BF16 row-major, c FP32: layout 0 a b^T (a layer), 1 a b (dh = dz W), 2 a^T b
// (dW = dz^T h).
__global__ void __launch_bounds__(THREADS, 1) gemm_test_kernel(int layout, const __nv_bfloat16* __restrict__ a,
                                                              const __nv_bfloat16* __restrict__ b,
                                                              float* __restrict__ c, int* error) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  __nv_bfloat16* ta = reinterpret_cast<__nv_bfloat16*>(smem_raw);
  __nv_bfloat16* tb = ta + TILE * H;
  uint64_t* mbar = reinterpret_cast<uint64_t*>(tb + TILE * H);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(mbar + 1);
  const int t = threadIdx.x;
  for (int k = 0; k < H; ++k) {
    ta[tc_offset(t, k)] = a[t * H + k];
    tb[tc_offset(t, k)] = b[t * H + k];
  }
  if (t == 0) mbar_init(smem_u32(mbar));
  tmem_alloc<128>(tslot);
  fence_async_smem();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;
  if (t == 0) {
    for (int k = 0; k < 8; ++k) {
      if (layout == 0) mma_idesc(tmem, kmaj(ta, k), kmaj(tb, k), kIdesc, k > 0);
      if (layout == 1) mma_idesc(tmem, kmaj(ta, k), mn(tb, k), kIdescKMn, k > 0);
      if (layout == 2) mma_idesc(tmem, mn(ta, k), mn(tb, k), kIdescMnMn, k > 0);
    }
    mma_commit(smem_u32(mbar));
  }
  const bool ok = __syncthreads_and(mbar_wait(smem_u32(mbar), 0));
  tc_fence_after();
  if (ok) {
    for (int q = 0; q < 4; ++q) {
      float v[32];
      tmem_ld32(tmem + ((uint32_t)(t & ~31) << 16) + q * 32, v);
      for (int i = 0; i < 32; ++i) c[t * H + q * 32 + i] = v[i];
    }
  } else if (t == 0) {
    atomicExch(error, 1);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  tmem_free<128>(tmem);
}

// ---------------------------------------------------------------------------
// Two-component Gamma mixture w G(a1, theta) + (1 - w) G(a2, theta) fitted by
// weighted EM to each pair's arrival-time histogram, as a function of the
// time residual t - t_shift (bins with a positive residual only; the reference
// fits a single Gamma to the time residual, src/modelling.jl:52-79).
// M step: theta = sum of weight x time / sum_k a_k S0_k, then psi(a_k) =
// SL_k / S0_k - ln theta solved by Newton, three times.  Output per pair: w,
// a1 <= a2, theta, mean log-likelihood per weight; NaNs when the histogram is
// empty.
//
// A warp fits up to 16 pairs together.  Their filled bins (weight, log time)
// are gathered once into the warp's part of shared memory.  E step: the warp
// walks one pair's bins after the other, two per lane at a time; the two
// densities share t / theta, so their ratio takes one exponential, and the
// log-likelihood one logarithm more, in the last iteration only.  M step: one
// lane per (pair, component).  Bins that do not fit (a first pair of more than
// kMixEntries filled bins) are read from the histogram again each time.
//
// Bound by FP64 latency and issue.  With one pair per warp, every lane did the
// same 48 digamma and trigamma evaluations per iteration: 20,000 pairs of 1000
// bins (60 iterations) took 36.1 ms.  Shared M steps: 3.76 ms.  The table-driven
// exponential and a reciprocal without branches, so that two bins overlap;
// no sum for the times, whose total is known; Newton from the last evaluation
// (one a solve, or none): 2.62 ms.  A pair taken only when there is room for
// it: 2.53 ms; the histogram loaded four rows ahead: 2.33 ms (issue 55 % of
// active cycles, FP64 pipe 36 %).  16 warps of 896 bins: 20 of 704 (96
// registers) took 12 % longer, 24 of 592 17 %.  Pairs beyond shared memory gain
// less, and still gain: every bin of 3000 filled, 200, 2000 and 20,000 pairs
// 6.9, 9.3 and 67.4 ms with one pair per warp, 2.6, 3.1 and 27.5 now; of 10,000,
// 200 and 2000 pairs 17.9 and 25.8, now 9.2 and 14.7.
constexpr int kMixWarps = 16, kMixEntries = 896, kMixPairs = 16;
constexpr size_t kMixSmem = (size_t)kMixWarps * kMixEntries * sizeof(double2);

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// psi(a) = y, a >= 1e-3, by Newton from the last point that psi was evaluated
// at (where its step is far off: from Minka's initial value).  psi is concave,
// so from the second step on the iterates rise to the root; their error is
// squared by each step, so a step of 1e-8 leaves none that FP64 holds, and a
// right side that moved by less takes no evaluation.  All lanes of the warp call.
struct Psi {
  double at, f, rf1;  // psi and 1 / psi' at `at`
  __device__ void eval(double x) {
    double f1;
    at = x;
    ppsf::psi_both(x, f, f1);
    rf1 = 1.0 / f1;
  }
};
__device__ __forceinline__ double inv_digamma(double y, Psi& P, bool active) {
#pragma unroll 1
  for (int i = 0;; ++i) {
    const double a = P.at;
    double n = a - (P.f - y) * P.rf1;
    if (i == 0 && !(n > 0.5 * a && n < 2.0 * a)) n = y >= -2.22 ? exp(y) + 0.5 : -1.0 / (y + 0.5772156649015329);
    n = n < 1e-3 ? 1e-3 : n;
    const bool moving = active && fabs(n - a) > 1e-8 * a;
    if (i == 24 || !__any_sync(0xffffffffu, moving)) return n;
    if (moving) P.eval(n);
  }
}

__global__ void __launch_bounds__(kMixWarps * 32, 1) gamma_fit_kernel(const double* __restrict__ hist, int64_t n, int bins,
                                                                     float t0, float bw,
                                                                     const float* __restrict__ tshift,
                                                                     float* __restrict__ out, int iters) {
  extern __shared__ double2 mix_smem[];
  constexpr unsigned kAll = 0xffffffffu;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double2* const entry = mix_smem + (size_t)warp * kMixEntries;  // the filled bins: weight, log time
  // the block's pairs are blockIdx.x + i gridDim.x; its warps take them from a
  // counter, at most a warp's share of what is left at a time
  __shared__ unsigned taken;
  if (threadIdx.x == 0) taken = 0;
  __syncthreads();
  const ppsf::WarpTables T = ppsf::warp_tables();
  const int64_t mine = (n - blockIdx.x + gridDim.x - 1) / gridDim.x;
  auto take = [&]() {
    unsigned i = 0;
    if (lane == 0) i = atomicAdd(&taken, 1u);
    return (int64_t)__shfl_sync(kAll, i, 0);
  };
  int64_t next = take();
  while (next < mine) {
    const int share = (int)min((int64_t)kMixPairs, (mine - next + kMixWarps - 1) / kMixWarps);
    bool held = true;  // `next` is not fitted yet
    // this lane's pair (lane / 2) and component (lane % 2; 0 is the one with the smaller start value)
    int64_t pair = -1;
    int first = 0, count = 0, rest = bins;  // entries in shared memory; bins from `rest` on are read again
    double s0 = 0, st = 0, a = 1, w = 0.5, th = 1;  // sums of the weights and of weight x time
    int used = 0, m = 0;
    for (; m < share; ++m) {
      if (!held) next = take();
      held = true;
      if (next >= mine) break;
      const int64_t row = blockIdx.x + next * gridDim.x;
      const double* h = hist + row * bins;
      const double ts = tshift[row];
      double p0 = 0, p1 = 0, p2 = 0;
      int k = 0, b0 = 0, stop = bins;
      auto ahead = [&](unsigned b) { return b < (unsigned)bins ? h[b] : 0.0; };
      double h1 = ahead(lane), h2 = ahead(32 + lane), h3 = ahead(64 + lane), h4 = ahead(96 + lane);
      for (; b0 < bins; b0 += 32) {
        const int b = b0 + lane;
        const double hb = h1, t = t0 + (b + 0.5) * bw - ts;
        h1 = h2;
        h2 = h3;
        h3 = h4;
        h4 = ahead(b + 128u);
        const bool in = t > 0 && hb > 0;
        const unsigned ball = __ballot_sync(kAll, in);
        if (!ball) continue;
        if (in) {
          p0 += hb;
          p1 += hb * t;
          p2 += hb * t * t;
        }
        if (stop < bins || used + k + __popc(ball) > kMixEntries) {
          stop = min(stop, b0);
          if (m > 0) break;  // the pair opens the next round
          continue;
        }
        if (in) {
          entry[used + k + __popc(ball & ((1u << lane) - 1u))] = make_double2(hb, log(t));
        }
        k += __popc(ball);
      }
      if (m > 0 && stop < bins) break;
      p0 = warp_sum(p0);
      p1 = warp_sum(p1);
      p2 = warp_sum(p2);
      if ((lane >> 1) == m) {
        pair = row;
        first = used;
        count = k;
        rest = stop;
        s0 = p0;
        st = p1;
        const double mean = p1 / p0, v = fmax(p2 / p0 - mean * mean, 1e-6 * mean * mean + 1e-12);
        const double a0 = fmax(mean * mean / v, 0.05);
        a = (lane & 1) ? 2.0 * a0 : fmax(0.5 * a0, 0.02);
        th = v / mean;
      }
      used += k;
      held = false;
    }
    __syncwarp();
    const bool live = pair >= 0 && s0 > 0;
    if (!live) a = th = 1.0;  // harmless values for the lanes without a fit
    Psi P;
    P.eval(a);
    double ll = 0, lth = log(th);
#pragma unroll 1
    for (int it = 0; it < iters; ++it) {
      const double c = log((lane & 1) ? 1.0 - w : w) - a * lth - lgamma(a);
      const double cd = c - __shfl_xor_sync(kAll, c, 1), ad = a - __shfl_xor_sync(kAll, a, 1);
      double S0 = 0, SL = 0;  // this lane's component
#pragma unroll 1
      for (int p = 0; p < m; ++p) {
        // log ratio of component 1's density to component 2's: da lt + dc (even lanes hold component 1)
        const double dc = __shfl_sync(kAll, cd, 2 * p), da = __shfl_sync(kAll, ad, 2 * p);
        const int f0 = __shfl_sync(kAll, first, 2 * p), k = __shfl_sync(kAll, count, 2 * p);
        const int stop = __shfl_sync(kAll, rest, 2 * p);
        double q0 = 0, q2 = 0, r0 = 0, r2 = 0;
        auto add = [&](auto... h_lt) {  // all lanes
          constexpr int Q = sizeof...(h_lt);
          const double2 in[Q] = {h_lt...};
          double d[Q], e[Q];
          bool far = false;  // beyond the table's range
#pragma unroll
          for (int q = 0; q < Q; ++q) {
            d[q] = fma(da, in[q].y, dc);
            e[q] = ppsf::exp_tab(-fabs(d[q]), T);
            far = far || (__double2hiint(d[q]) & 0x7fffffff) >= 0x40862000;
          }
          if (__any_sync(kAll, far)) {
#pragma unroll
            for (int q = 0; q < Q; ++q) e[q] = exp(-fabs(d[q]));
          }
#pragma unroll
          for (int q = 0; q < Q; ++q) {
            const double v = ppsf::reciprocal_1_2(1.0 + e[q]);
            const double f = d[q] > 0 ? v : e[q] * v;  // component 1's share
            // 1 - f, which is 0 once component 2 falls below the rounding of 1:
            // its parameters then stay as they are
            const double x = in[q].x * f, y = in[q].x * (1.0 - f);
            q0 += x;
            q2 = fma(x, in[q].y, q2);
            r0 += y;
            r2 = fma(y, in[q].y, r2);
          }
        };
        const double2 none = make_double2(0.0, 0.0);
        int i = lane;
#pragma unroll 1
        for (; i - lane + 32 < k; i += 64) add(entry[f0 + i], i + 32 < k ? entry[f0 + i + 32] : none);
        if (i - lane < k) add(i < k ? entry[f0 + i] : none);
        if (stop < bins) {  // what did not fit
          const int64_t row = __shfl_sync(kAll, pair, 2 * p);
          const double* h = hist + row * bins;
          const double ts = tshift[row];
#pragma unroll 1
          for (int b0 = stop; b0 < bins; b0 += 32) {
            const int b = b0 + lane;
            const double hb = b < bins ? h[b] : 0.0, t = t0 + (b + 0.5) * bw - ts;
            add(t > 0 && hb > 0 ? make_double2(hb, log(t)) : none);
          }
        }
        // even lanes sum component 1, odd lanes component 2
        const bool odd = lane & 1;
        double u0 = odd ? r0 : q0, u2 = odd ? r2 : q2;
        u0 += __shfl_xor_sync(kAll, odd ? q0 : r0, 1);
        u2 += __shfl_xor_sync(kAll, odd ? q2 : r2, 1);
#pragma unroll
        for (int o = 2; o < 32; o <<= 1) {
          u0 += __shfl_xor_sync(kAll, u0, o);
          u2 += __shfl_xor_sync(kAll, u2, o);
        }
        if ((lane >> 1) == p) {
          S0 = u0;
          SL = u2;
        }
      }
      if (it == iters - 1) {  // the log-likelihood, of the parameters that this iteration began with
#pragma unroll 1
        for (int p = 0; p < m; ++p) {
          const double dc = __shfl_sync(kAll, cd, 2 * p), da = __shfl_sync(kAll, ad, 2 * p);
          const double c2 = __shfl_sync(kAll, c, 2 * p + 1), a2 = __shfl_sync(kAll, a, 2 * p + 1);
          const int f0 = __shfl_sync(kAll, first, 2 * p), k = __shfl_sync(kAll, count, 2 * p);
          const int stop = __shfl_sync(kAll, rest, 2 * p);
          double L = 0;
          auto add = [&](double hb, double lt) {
            const double d = fma(da, lt, dc);
            L += hb * (fma(a2 - 1.0, lt, c2) + fmax(d, 0.0) + log1p(exp(-fabs(d))));
          };
#pragma unroll 1
          for (int i = f0 + lane; i < f0 + k; i += 32) add(entry[i].x, entry[i].y);
          if (stop < bins) {
            const int64_t row = __shfl_sync(kAll, pair, 2 * p);
            const double* h = hist + row * bins;
            const double ts = tshift[row];
#pragma unroll 1
            for (int b = stop + lane; b < bins; b += 32) {
              const double hb = h[b], t = t0 + (b + 0.5) * bw - ts;
              if (t > 0 && hb > 0) add(hb, log(t));
            }
          }
          L = warp_sum(L);
          if ((lane >> 1) == p) ll = (L - st / th) / s0;
        }
      }
      const double o0 = __shfl_xor_sync(kAll, S0, 1);
      const double wa = (lane & 1) ? o0 : S0, wb = (lane & 1) ? S0 : o0;
      if (live) w = fmin(fmax(wa / (wa + wb), 1e-4), 1 - 1e-4);
      const bool solve = live && S0 > 0;
#pragma unroll 1
      for (int j = 0; j < 3; ++j) {
        const double v = a * S0, vt = v + __shfl_xor_sync(kAll, v, 1);
        if (live) th = st / vt;
        lth = log(th);
        const double y = solve ? SL / S0 - lth : 0.0;
        const double an = inv_digamma(y, P, solve);
        if (solve) a = an;
      }
    }
    const double oa = __shfl_xor_sync(kAll, a, 1);
    if (pair >= 0 && !(lane & 1)) {
      float* o = out + pair * 5;
      // order the components, by the shapes as they are returned: where the two
      // have met but for rounding (1 % of pairs with a few filled bins), the order stays
      const bool swap = (float)a > (float)oa;
      const float nan = __int_as_float(0x7fc00000);
      o[0] = live ? (float)(swap ? 1 - w : w) : nan;
      o[1] = live ? (float)(swap ? oa : a) : nan;
      o[2] = live ? (float)(swap ? a : oa) : nan;
      o[3] = live ? (float)th : nan;
      o[4] = live ? (float)ll : nan;
    }
    __syncwarp();
    if (!held) next = take();
  }
}

constexpr size_t kInferSmem = (2 + kGroups) * TILE_BYTES + 5 * H * 16 * 2 + (8 + 24) * 4 + 8 * (kGroups + 2) + 16;
constexpr size_t kTrainSmem = 6 * TILE_BYTES + (H * IN + H * 8 + TILE * 8 + TILE * IN + 3 * H) * 4 + 16;
constexpr size_t kTestSmem = 2 * TILE_BYTES + 32;

}  // namespace mlp

// ---------------------------------------------------------------------------
// Host side.
struct pp_mlp {
  int device = 0;
  int sm_count = 0;
  std::mutex mu;
  float* d_params = nullptr;  // N_PARAMS
  float* d_grad = nullptr;  // kBack words: gradients, loss sum, error flag, mask sums
  float* d_m = nullptr;
  float* d_v = nullptr;
  __nv_bfloat16* d_tc = nullptr;  // 4 tiles of 128 x 128, then 4 of 128 x 16
  float* d_norm = nullptr;        // 18 (+ pad)
  int64_t step = 0;
  std::string err;
};

namespace {
struct Guard {
  int prev = -1;
  explicit Guard(int d) {
    cudaGetDevice(&prev);
    if (prev != d) cudaSetDevice(d);
  }
  ~Guard() {
    if (prev >= 0) cudaSetDevice(prev);
  }
};

mlp::DevParams dev_params(pp_mlp* m) {
  mlp::DevParams P;
  P.p = m->d_params;
  P.w2tc = m->d_tc;
  P.w3tc = m->d_tc + mlp::TILE * mlp::H;
  P.w2h = m->d_tc + 2 * mlp::TILE * mlp::H;
  P.w3h = m->d_tc + 3 * mlp::TILE * mlp::H;
  P.w1tc = m->d_tc + 4 * mlp::TILE * mlp::H;
  P.w4tc = P.w1tc + mlp::H * 16;
  P.norm = m->d_norm;
  P.error = reinterpret_cast<int*>(m->d_grad + mlp::N_PARAMS + 1);
  return P;
}

mlp::Copies copies(pp_mlp* m) {
  __nv_bfloat16* t = m->d_tc;
  constexpr int T = mlp::TILE * mlp::H, S = mlp::H * 16;
  return mlp::Copies{t, t + T, t + 2 * T, t + 3 * T, t + 4 * T, t + 4 * T + S, t + 4 * T + 2 * S, t + 4 * T + 3 * S};
}
constexpr int kParamBlocks = (mlp::N_PARAMS + 255) / 256;

cudaError_t prepare(pp_mlp* m, cudaStream_t s) {
  mlp::prepare_kernel<<<kParamBlocks, 256, 0, s>>>(m->d_params, copies(m));
  pp::count_launches(1);
  return cudaGetLastError();
}

pp_status fail(pp_mlp* m, pp_status s, const std::string& msg) {
  m->err = msg;
  return s;
}
}  // namespace

extern "C" {

pp_status pp_mlp_create(int device, uint64_t seed, pp_mlp** out) {
  if (!out) return PP_ERR_ARG;
  *out = nullptr;
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || device < 0 || device >= ndev) {
    cudaGetLastError();
    return PP_ERR_ARG;
  }
  pp_mlp* m = new pp_mlp();
  m->device = device;
  Guard g(device);
  cudaDeviceProp prop;
  cudaGetDeviceProperties(&prop, device);
  m->sm_count = prop.multiProcessorCount;
  cudaError_t e;
  constexpr size_t kTcBytes = 4 * mlp::TILE_BYTES + 4 * mlp::H * 16 * 2;
  if ((e = cudaMalloc(&m->d_params, mlp::N_PARAMS * 4)) || (e = cudaMalloc(&m->d_grad, mlp::kBack * 4)) ||
      (e = cudaMalloc(&m->d_m, mlp::N_PARAMS * 4)) || (e = cudaMalloc(&m->d_v, mlp::N_PARAMS * 4)) ||
      (e = cudaMalloc(&m->d_tc, kTcBytes)) || (e = cudaMalloc(&m->d_norm, 32 * 4))) {
    cudaGetLastError();
    for (void* b : {(void*)m->d_params, (void*)m->d_grad, (void*)m->d_m, (void*)m->d_v, (void*)m->d_tc,
                    (void*)m->d_norm})
      if (b) cudaFree(b);
    delete m;
    return e == cudaErrorMemoryAllocation ? PP_ERR_OOM : PP_ERR_CUDA;
  }
  // Glorot-uniform weights, zero biases, from a splitmix64 stream of `seed`
  std::vector<float> p(mlp::N_PARAMS, 0.f);
  uint64_t st = seed;
  auto next = [&]() {
    uint64_t z = (st += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return (double)(z >> 11) * (1.0 / 9007199254740992.0);
  };
  auto fill = [&](int off, int fan_out, int fan_in) {
    const double a = std::sqrt(6.0 / (fan_in + fan_out));
    for (int i = 0; i < fan_out * fan_in; ++i) p[off + i] = (float)((2.0 * next() - 1.0) * a);
  };
  fill(mlp::OFF_W1, mlp::H, mlp::IN);
  fill(mlp::OFF_W2, mlp::H, mlp::H);
  fill(mlp::OFF_W3, mlp::H, mlp::H);
  fill(mlp::OFF_W4, mlp::OUT, mlp::H);
  float norm[32] = {0};
  for (int j = 0; j < 4; ++j) norm[4 + j] = 1.f;
  for (int j = 0; j < 5; ++j) norm[13 + j] = 1.f;
  if ((e = cudaMemcpy(m->d_params, p.data(), mlp::N_PARAMS * 4, cudaMemcpyHostToDevice)) ||
      (e = cudaMemset(m->d_grad, 0, mlp::kBack * 4)) || (e = cudaMemset(m->d_m, 0, mlp::N_PARAMS * 4)) ||
      (e = cudaMemset(m->d_v, 0, mlp::N_PARAMS * 4)) || (e = cudaMemcpy(m->d_norm, norm, 128, cudaMemcpyHostToDevice)) ||
      (e = cudaMemset(m->d_tc, 0, kTcBytes)) || (e = prepare(m, nullptr)) || (e = cudaDeviceSynchronize())) {
    cudaGetLastError();
    pp_mlp_destroy(m);
    return PP_ERR_CUDA;
  }
  cudaFuncSetAttribute(mlp::infer_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mlp::kInferSmem);
  cudaFuncSetAttribute(mlp::train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mlp::kTrainSmem);
  cudaFuncSetAttribute(mlp::gemm_test_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mlp::kTestSmem);
  *out = m;
  return PP_OK;
}

void pp_mlp_destroy(pp_mlp* m) {
  if (!m) return;
  Guard g(m->device);
  cudaDeviceSynchronize();
  for (void* p : {(void*)m->d_params, (void*)m->d_grad, (void*)m->d_m, (void*)m->d_v, (void*)m->d_tc,
                  (void*)m->d_norm})
    if (p) cudaFree(p);
  delete m;
}

const char* pp_mlp_last_error(const pp_mlp* m) { return m ? m->err.c_str() : ""; }

int32_t pp_mlp_num_params(void) { return mlp::N_PARAMS; }

pp_status pp_mlp_get_params(pp_mlp* m, float* out) {
  if (!m || !out) return PP_ERR_ARG;
  std::lock_guard<std::mutex> lk(m->mu);
  Guard g(m->device);
  return cudaMemcpy(out, m->d_params, mlp::N_PARAMS * 4, cudaMemcpyDeviceToHost) ? PP_ERR_CUDA : PP_OK;
}

pp_status pp_mlp_set_params(pp_mlp* m, const float* in) {
  if (!m || !in) return PP_ERR_ARG;
  std::lock_guard<std::mutex> lk(m->mu);
  Guard g(m->device);
  if (cudaMemcpy(m->d_params, in, mlp::N_PARAMS * 4, cudaMemcpyHostToDevice) || prepare(m, nullptr) ||
      cudaDeviceSynchronize())
    return fail(m, PP_ERR_CUDA, "pp_mlp_set_params");
  return PP_OK;
}

pp_status pp_mlp_set_normalization(pp_mlp* m, const float* x_mean, const float* x_std, const float* y_mean,
                                   const float* y_std) {
  if (!m || !x_mean || !x_std || !y_mean || !y_std) return PP_ERR_ARG;
  float norm[32] = {0};
  for (int j = 0; j < 4; ++j) {
    norm[j] = x_mean[j];
    norm[4 + j] = x_std[j] > 0.f ? x_std[j] : 1.f;
  }
  for (int j = 0; j < 5; ++j) {
    norm[8 + j] = y_mean[j];
    norm[13 + j] = y_std[j] > 0.f ? y_std[j] : 1.f;
  }
  std::lock_guard<std::mutex> lk(m->mu);
  Guard g(m->device);
  return cudaMemcpy(m->d_norm, norm, 128, cudaMemcpyHostToDevice) ? PP_ERR_CUDA : PP_OK;
}

pp_status pp_mlp_get_normalization(pp_mlp* m, float* out18) {
  if (!m || !out18) return PP_ERR_ARG;
  std::lock_guard<std::mutex> lk(m->mu);
  Guard g(m->device);
  return cudaMemcpy(out18, m->d_norm, 18 * 4, cudaMemcpyDeviceToHost) ? PP_ERR_CUDA : PP_OK;
}

pp_status pp_mlp_forward(pp_mlp* m, const float* d_x, float* d_out, int64_t n, int32_t physical, void* stream) {
  pp::Range range_("pp_mlp_forward");
  if (!m || n < 0 || (n > 0 && (!d_x || !d_out))) return PP_ERR_ARG;
  if (n == 0) return PP_OK;
  std::lock_guard<std::mutex> lk(m->mu);
  Guard g(m->device);
  const int64_t tiles = (n + mlp::TILE - 1) / mlp::TILE;
  const int grid = (int)std::min<int64_t>(tiles, (int64_t)m->sm_count);
  mlp::infer_kernel<<<grid, mlp::INFER_THREADS, mlp::kInferSmem, static_cast<cudaStream_t>(stream)>>>(
      dev_params(m), d_x, d_out, n, physical);
  pp::count_launches(1);
  const cudaError_t e = cudaGetLastError();
  return e ? fail(m, PP_ERR_CUDA, std::string("pp_mlp_forward: ") + cudaGetErrorString(e)) : PP_OK;
}

// One Adam step on a batch (or, with lr = 0 and grad_out, the raw gradients).
pp_status pp_mlp_train_step(pp_mlp* m, const float* d_xn, const float* d_yt, const float* d_mask, int64_t n,
                            float lr, float* loss_out, float* grad_out) {
  pp::Range range_("pp_mlp_train_step");
  if (!m || n <= 0 || !d_xn || !d_yt || !d_mask) return PP_ERR_ARG;
  std::lock_guard<std::mutex> lk(m->mu);
  Guard g(m->device);
  cudaError_t e;
  const int64_t tiles = (n + mlp::TILE - 1) / mlp::TILE;
  if (tiles > INT32_MAX) return fail(m, PP_ERR_ARG, "pp_mlp_train_step: too many rows");
  double* part = reinterpret_cast<double*>(m->d_grad + mlp::kPartAt);
  mlp::count_kernel<<<mlp::kCountBlocks, 256>>>(d_mask, n * mlp::OUT, m->d_grad, part);
  pp::count_launches(1);
  if ((e = cudaGetLastError()) ||
      (e = pp::launch_dependent(mlp::train_kernel, (int)tiles, mlp::TRAIN_THREADS, mlp::kTrainSmem, nullptr,
                                dev_params(m), d_xn, d_yt, d_mask, n, part, m->d_grad)))
    return fail(m, PP_ERR_CUDA, std::string("train: ") + cudaGetErrorString(e));
  if (lr > 0.f) {
    m->step += 1;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = (float)(1.0 / (1.0 - std::pow((double)b1, (double)m->step)));
    const float c2 = (float)(1.0 / (1.0 - std::pow((double)b2, (double)m->step)));
    if ((e = pp::launch_dependent(mlp::adam_kernel, kParamBlocks, 256, 0, nullptr, m->d_params, m->d_grad, m->d_m,
                                  m->d_v, copies(m), lr, b1, b2, 1e-8f, c1, c2)))
      return fail(m, PP_ERR_CUDA, std::string("adam: ") + cudaGetErrorString(e));
  }
  float back[mlp::kBack - mlp::N_PARAMS];  // loss sum, error flag, mask sums
  if ((grad_out && (e = cudaMemcpyAsync(grad_out, m->d_grad, mlp::N_PARAMS * 4, cudaMemcpyDeviceToHost, nullptr))) ||
      (e = cudaMemcpyAsync(back, m->d_grad + mlp::N_PARAMS, sizeof back, cudaMemcpyDeviceToHost, nullptr)) ||
      (e = cudaStreamSynchronize(nullptr)))
    return fail(m, PP_ERR_CUDA, std::string("train: ") + cudaGetErrorString(e));
  int errflag;
  std::memcpy(&errflag, back + 1, 4);
  if (errflag) return fail(m, PP_ERR_TIMEOUT, "tensor-core wait expired");
  double sums[mlp::kCountBlocks], cnt = 0.0;
  std::memcpy(sums, back + (mlp::kPartAt - mlp::N_PARAMS), sizeof sums);
  for (double v : sums) cnt += v;
  if (loss_out) *loss_out = (float)(back[0] * (cnt > 0.0 ? (float)(1.0 / cnt) : 0.f));
  return PP_OK;
}

pp_status pp_mlp_gemm_selftest(int device, const uint16_t* a_bf16, const uint16_t* b_bf16, float* c) {
  return pp_mlp_gemm_selftest_layout(device, 0, a_bf16, b_bf16, c);
}

pp_status pp_mlp_gemm_selftest_layout(int device, int32_t layout, const uint16_t* a_bf16, const uint16_t* b_bf16,
                                      float* c) {
  if (!a_bf16 || !b_bf16 || !c || layout < 0 || layout > 2) return PP_ERR_ARG;
  Guard g(device);
  void *da = nullptr, *db = nullptr, *dc = nullptr, *de = nullptr;
  cudaError_t e;
  if ((e = cudaMalloc(&da, 128 * 128 * 2)) || (e = cudaMalloc(&db, 128 * 128 * 2)) ||
      (e = cudaMalloc(&dc, 128 * 128 * 4)) || (e = cudaMalloc(&de, 16))) {
    cudaGetLastError();
    for (void* b : {da, db, dc, de})
      if (b) cudaFree(b);
    return e == cudaErrorMemoryAllocation ? PP_ERR_OOM : PP_ERR_CUDA;
  }
  cudaFuncSetAttribute(mlp::gemm_test_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mlp::kTestSmem);
  int flag = 0;
  cudaMemcpy(da, a_bf16, 128 * 128 * 2, cudaMemcpyHostToDevice);
  cudaMemcpy(db, b_bf16, 128 * 128 * 2, cudaMemcpyHostToDevice);
  cudaMemset(de, 0, 16);
  mlp::gemm_test_kernel<<<1, mlp::THREADS, mlp::kTestSmem>>>(layout, static_cast<const __nv_bfloat16*>(da),
                                                             static_cast<const __nv_bfloat16*>(db),
                                                             static_cast<float*>(dc), static_cast<int*>(de));
  pp::count_launches(1);
  e = cudaGetLastError();
  if (!e) e = cudaMemcpy(c, dc, 128 * 128 * 4, cudaMemcpyDeviceToHost);
  if (!e) e = cudaMemcpy(&flag, de, 4, cudaMemcpyDeviceToHost);
  cudaFree(da);
  cudaFree(db);
  cudaFree(dc);
  cudaFree(de);
  if (e) return PP_ERR_CUDA;
  return flag ? PP_ERR_TIMEOUT : PP_OK;
}

}  // extern "C"

extern "C" pp_status pp_gamma_mixture_fit(const double* d_hist, int64_t n, int32_t bins, float t0, float bin_width,
                                          const float* d_tshift, float* d_out, int32_t iters, void* stream) {
  if (n < 0 || bins <= 0 || !(bin_width > 0.f) || iters < 1 || (n > 0 && (!d_hist || !d_tshift || !d_out)))
    return PP_ERR_ARG;
  if (n == 0) return PP_OK;
  int dev = 0, sms = 0;
  if (cudaGetDevice(&dev) || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) ||
      cudaFuncSetAttribute(mlp::gamma_fit_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)mlp::kMixSmem))
    return PP_ERR_CUDA;
  const int grid = (int)std::min<int64_t>(n, sms);
  mlp::gamma_fit_kernel<<<grid, mlp::kMixWarps * 32, mlp::kMixSmem, static_cast<cudaStream_t>(stream)>>>(
      d_hist, n, bins, t0, bin_width, d_tshift, d_out, iters);
  pp::count_launches(1);
  return cudaGetLastError() ? PP_ERR_CUDA : PP_OK;
}
