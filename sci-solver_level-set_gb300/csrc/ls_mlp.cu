// ls_mlp.cu -- the learned warm start: a 128-128-128-128-1 ReLU MLP on the
// 5th-generation tensor cores (tcgen05.mma, BF16 operands in shared memory,
// FP32 accumulators in tensor memory), with forward, backward and Adam
// kernels for training on the GPU and a feature kernel that builds the
// network input of a vertex from its 1-ring.
//
// Network (per sample, all layers 128 wide):
//   a0 = bf16(x)                                  x: 32 padded 1-ring slots x
//                                                 (dx, dy, dz, phi) / h
//   z_l = a_l W_l^T (fp32 accumulate) + b_l,      l = 1, 2, 3, W_l [out][in] bf16
//   a_l = bf16(relu(z_l))
//   y   = sum_j a_3[j] w4[j] + b4                 (fp32)
// Loss: 1/(2n) sum (y - t)^2.  Backward in the same precisions:
//   dy = (y - t)/n;  g_w4 = sum dy a_3;  g_b4 = sum dy
//   d_3 = bf16(dy w4 * [a_3 > 0])
//   g_W_l = d_l^T a_{l-1} (fp32 accumulate);  g_b_l = sum_samples d_l
//   d_{l-1} = bf16((d_l W_l) * [a_{l-1} > 0])
//
// One CTA of 256 threads handles a tile of 128 samples.  Operand tiles use
// the no-swizzle K-major core-matrix layout of the tensor core: element
// (row r, k) of a 128 x 128 BF16 tile sits at byte
//   (r / 8) * 2048 + (k / 8) * 128 + (r % 8) * 16 + (k % 8) * 2,
// i.e. 8 x 16-byte core matrices, 128 bytes apart along K (leading byte
// offset) and 2048 bytes apart along M/N (stride byte offset).  One MMA
// (M = N = 128, K = 16) covers two core matrices along K; the K loop
// advances both descriptors by 256 bytes.  The accumulator (M = 128) keeps
// row r in tensor-memory lane r, column n in column n; warp w of the CTA
// reads lanes 32 (w % 4) .. +31 with tcgen05.ld, warps 0-3 the columns below
// 64, warps 4-7 the others.
// The same bytes are the MN-major operand of the transposed product: its
// core matrices hold 8 K rows of 8 contiguous M/N elements, 128 bytes apart
// along M/N and 2048 along K, so the leading and stride offsets swap, the K
// loop advances by 4096 bytes and the instruction descriptor's transpose bit
// is set.  The weight gradients d^T a and the back-propagation d W therefore
// read the tiles of d, a and W that the forward pass uses; nothing is
// transposed.
//
// Every wait on an mbarrier is bounded (about one second of clock cycles);
// on expiry the kernel records the error, waits (bounded) for its MMAs,
// frees its tensor memory and returns.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "ls_mlp.h"

namespace lsgb {
namespace mlp {

namespace {

constexpr int F = 128;        // features = hidden width
constexpr int TILE = 128;     // samples per tile
constexpr int THREADS = 256;  // of the network kernels' CTAs
constexpr int TILE_BYTES = TILE * F * 2;   // one BF16 operand tile (32 KB)
constexpr uint32_t LBO = 128, SBO = 2048;  // core-matrix strides (bytes)
// kind::f16 instruction descriptor: D fp32 (bits 4-5 = 1), A bf16 (bits
// 7-9 = 1), B bf16 (bits 10-12 = 1), A and B K-major, N >> 3 at bits 17-22,
// M >> 4 at bits 24-28
constexpr uint32_t IDESC = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(F >> 3) << 17) |
                           ((uint32_t)(TILE >> 4) << 24);
constexpr uint32_t IDESC_TA = 1u << 15, IDESC_TB = 1u << 16;  // A, B MN-major
constexpr long long WAIT_CYCLES = 2000000000LL;  // ~1 s at 2 GHz

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ uint32_t tile_off(int r, int k) {
  return (uint32_t)((r >> 3) * SBO + (k >> 3) * LBO + (r & 7) * 16 + (k & 7) * 2);
}

// shared-memory matrix descriptor, no swizzle (layout type 0), version 1;
// mn: the tile read as an MN-major operand
__device__ __forceinline__ uint64_t make_desc(uint32_t saddr, bool mn) {
  uint64_t d = 0;
  d |= (uint64_t)((saddr >> 4) & 0x3FFFu);
  d |= (uint64_t)(((mn ? SBO : LBO) >> 4) & 0x3FFFu) << 16;
  d |= (uint64_t)(((mn ? LBO : SBO) >> 4) & 0x3FFFu) << 32;
  d |= (uint64_t)1 << 46;
  return d;
}

__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t ncols) {
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(slot)), "r"(ncols)
               : "memory");
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_async_smem() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

__device__ __forceinline__ void mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, int accumulate) {
  asm volatile(
      "{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
               : "memory");
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// bounded wait for the phase with the given parity to complete
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) {
  const long long t0 = clock64();
  while (true) {
    uint32_t ok = 0;
    asm volatile(
        "{\n.reg .pred p;\nmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\nselp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
    if (clock64() - t0 > WAIT_CYCLES) return false;
  }
}

// 32 consecutive accumulator columns of this warp's 32 lanes
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float* v) {
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
      "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
        "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
        "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
        "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr)
      : "memory");
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// rows [s0, s0 + 128) of a [n][128] BF16 global matrix -> a tile (zeros past
// n), by all threads: a warp takes 8 rows x 4 chunks of 16 bytes at a time,
// whole 64-byte pieces of the rows, and its stores fall on all banks
__device__ __forceinline__ void load_rows(uint8_t* tile, const __nv_bfloat16* X, int s0, int n) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int rl = lane & 7, cl = lane >> 3;
#pragma unroll
  for (int k = 0; k < 64 / (THREADS / 32); ++k) {
    const int i = warp + k * (THREADS / 32);  // 16 row groups x 4 chunk groups
    const int r = (i >> 2) * 8 + rl, c = ((i & 3) * 4 + cl) * 8;
    const uint4 v = s0 + r < n ? __ldg(reinterpret_cast<const uint4*>(X + (size_t)(s0 + r) * F + c)) : make_uint4(0, 0, 0, 0);
    *reinterpret_cast<uint4*>(tile + tile_off(r, c)) = v;
  }
}

// 8 floats -> 8 BF16 (round to nearest even) in one 16-byte chunk
__device__ __forceinline__ uint4 pack8(const float* v) {
  uint4 o;
  __nv_bfloat162 p0 = __floats2bfloat162_rn(v[0], v[1]);
  __nv_bfloat162 p1 = __floats2bfloat162_rn(v[2], v[3]);
  __nv_bfloat162 p2 = __floats2bfloat162_rn(v[4], v[5]);
  __nv_bfloat162 p3 = __floats2bfloat162_rn(v[6], v[7]);
  o.x = *reinterpret_cast<uint32_t*>(&p0);
  o.y = *reinterpret_cast<uint32_t*>(&p1);
  o.z = *reinterpret_cast<uint32_t*>(&p2);
  o.w = *reinterpret_cast<uint32_t*>(&p3);
  return o;
}

__device__ __forceinline__ float bf16r(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }


}  // namespace

// ---------------------------------------------------------------------------
// Weight copy for the tensor cores: BF16 tiles in the operand layout above
// (tile_off; rows = output feature, K = input feature), so that one bulk
// asynchronous copy of 32 KB stages a layer's weights.
__device__ __forceinline__ void store_weight(__nv_bfloat16* Wt, int i, float p) {
  const int l = i / (F * F), o = (i / F) % F, in = i % F;
  Wt[(size_t)l * F * F + tile_off(o, in) / 2] = __float2bfloat16_rn(p);
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("{\n.reg .b64 st;\nmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n}" ::"r"(smem_u32(bar)),
               "r"(bytes)
               : "memory");
}

// one tile (32 KB, 16-byte aligned at both ends) from global into shared
// memory, completing on bar
__device__ __forceinline__ void bulk_tile(uint8_t* dst, const __nv_bfloat16* src, uint64_t* bar) {
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_u32(dst)),
               "l"(__cvta_generic_to_global(src)), "r"((uint32_t)TILE_BYTES), "r"(smem_u32(bar))
               : "memory");
}

// MMAs of one 128 x 128 x 128 product that add to the accumulator when acc
// is set (thread 0 only); ta, tb: the tile is read as an MN-major operand
__device__ __forceinline__ void mma_tile(uint32_t tmem_d, const uint8_t* a, bool ta, const uint8_t* b, bool tb, bool acc) {
  const uint32_t sa = smem_u32(a), sb = smem_u32(b);
  const uint32_t ka = ta ? 2 * SBO : 2 * LBO, kb = tb ? 2 * SBO : 2 * LBO;
  const uint32_t idesc = IDESC | (ta ? IDESC_TA : 0u) | (tb ? IDESC_TB : 0u);
#pragma unroll
  for (int ks = 0; ks < F / 16; ++ks)
    mma(tmem_d, make_desc(sa + ks * ka, ta), make_desc(sb + ks * kb, tb), idesc, (acc || ks > 0) ? 1 : 0);
}

struct SmemW {
  uint64_t bar;    // MMA completion
  uint64_t bar_w;  // weight tiles staged
  uint32_t tmem;
  int fail;
};

// The half of a layer's epilogue that belongs to this thread: its sample
// row's 64 columns (from column 64 * (warp / 4)) of bf16(relu(z + b)) to tile
// `out` (when given), their values added up with the weights w4 in column
// order (last layer).  The two halves of a row's sum are one chain: the lower
// columns' partial sum goes through s_out to the upper ones' thread.
__device__ __forceinline__ float layer_epilogue(uint32_t tz, const float* s_b, uint8_t* out, const float* s_w4,
                                                float* s_out) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int r = (warp & 3) * 32 + lane, c0 = (warp >> 2) * 64;
  float v[64];
  tmem_ld32(tz + ((uint32_t)((warp & 3) * 32) << 16) + c0, v);
  tmem_ld32(tz + ((uint32_t)((warp & 3) * 32) << 16) + c0 + 32, v + 32);
#pragma unroll
  for (int j = 0; j < 64; ++j) v[j] = bf16r(fmaxf(v[j] + s_b[c0 + j], 0.f));
  if (out) {
#pragma unroll
    for (int q = 0; q < 8; ++q) *reinterpret_cast<uint4*>(out + tile_off(r, c0 + q * 8)) = pack8(v + q * 8);
  }
  float sum = 0.f;
  if (s_w4) {
    if (warp < 4) {
#pragma unroll
      for (int j = 0; j < 64; ++j) sum += v[j] * s_w4[j];
      s_out[r] = sum;
    }
    __syncthreads();
    if (warp >= 4) {
      sum = s_out[r];
#pragma unroll
      for (int j = 0; j < 64; ++j) sum += v[j] * s_w4[64 + j];
    }
  }
  return sum;  // complete in warps 4-7
}

// ---------------------------------------------------------------------------
// Forward.  X [n][128] BF16 rows; Wt the three weight tiles; P4 = [b (3 x
// 128) | w4 (128) | b4] fp32; y [n].  n_dev (optional) overrides n from
// device memory (a device-side sample count).  Each CTA stages the weights
// once (three bulk copies) and then runs the sample tiles blockIdx.x,
// blockIdx.x + gridDim.x, ... through the three layers.
__global__ void __launch_bounds__(THREADS, 1)
    k_mlp_fwd(const __nv_bfloat16* __restrict__ X, int n, const int* n_dev, const __nv_bfloat16* __restrict__ Wt,
              const float* __restrict__ P4, float* __restrict__ y, int* err) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* act = base;                       // activation tile (A operand)
  uint8_t* wt = base + TILE_BYTES;           // 3 weight tiles (B operands)
  float* s_b = reinterpret_cast<float*>(base + 4 * TILE_BYTES);  // [3][128] biases
  float* s_w4 = s_b + 3 * F;                                      // [128]
  float* s_out = s_w4 + F;                                        // [128]
  SmemW* sm = reinterpret_cast<SmemW*>(s_out + F);
  const int tid = threadIdx.x, warp = tid >> 5;
  if (n_dev) n = *n_dev;
  const int ntiles = (n + TILE - 1) / TILE;
  if ((int)blockIdx.x >= ntiles) return;  // whole CTA exits before any tensor-core work
  if (tid == 0) {
    mbar_init(&sm->bar, 1);
    mbar_init(&sm->bar_w, 1);
    sm->fail = 0;
    mbar_expect_tx(&sm->bar_w, 3 * TILE_BYTES);
    for (int l = 0; l < 3; ++l) bulk_tile(wt + l * TILE_BYTES, Wt + (size_t)l * F * F, &sm->bar_w);
  }
  for (int i = tid; i < 4 * F; i += THREADS) s_b[i] = __ldg(P4 + i);  // b and w4
  __syncwarp();
  if (warp == 0) tmem_alloc(&sm->tmem, 128);
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tmem = sm->tmem;
  uint32_t phase = 0;
  bool ok = true, weights = false, mma_pending = false;
  for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
    const int s0 = tile * TILE;
    load_rows(act, X, s0, n);
    fence_async_smem();
    fence_before();
    __syncthreads();
    fence_after();
    if (!weights) {
      ok = __syncthreads_and(mbar_wait(&sm->bar_w, 0)) != 0;
      weights = ok;
      if (!ok) break;
    }
    float out = 0.f;
    for (int l = 0; l < 3 && ok; ++l) {
      if (tid == 0) {
        mma_tile(tmem, act, false, wt + l * TILE_BYTES, false, false);
        mma_commit(&sm->bar);
      }
      mma_pending = true;
      ok = __syncthreads_and(mbar_wait(&sm->bar, phase)) != 0;
      if (!ok) break;
      mma_pending = false;
      phase ^= 1;
      fence_after();
      out = layer_epilogue(tmem, s_b + l * F, l < 2 ? act : nullptr, l == 2 ? s_w4 : nullptr, s_out);
      fence_before();
      fence_async_smem();
      __syncthreads();
      fence_after();
    }
    if (ok && tid >= TILE && s0 + tid - TILE < n) y[s0 + tid - TILE] = out + __ldg(P4 + 4 * F);
  }
  if (!ok) {
    sm->fail = 1;
    if (err) atomicExch(err, 1);
    // drain (bounded): the weight copies and the MMAs in flight before TMEM goes
    if (!weights) mbar_wait(&sm->bar_w, 0);
    if (mma_pending) mbar_wait(&sm->bar, phase);
  }
  fence_before();
  __syncthreads();
  fence_after();
  if (warp == 0) tmem_dealloc(tmem, 128);
}

// Column sums of a tile in sample order (the order is part of the result:
// Adam turns the last bit of a small gradient into a step).  Thread c < 128
// sums column c.  Eight columns share 16 bytes, and the four such groups of
// a warp lie on the same banks for one sample, so group g runs g samples
// behind: the four read different rows of the core matrices, without
// conflicts.
__device__ __forceinline__ float column_sum(const uint8_t* tile) {
  const int c = threadIdx.x & (TILE - 1), lag = (threadIdx.x & 31) >> 3;
  float sum = 0.f;
#pragma unroll 8
  for (int k = 0; k < TILE + 3; ++k) {
    const int r = k - lag;
    if (r >= 0 && r < TILE) sum += __bfloat162float(*reinterpret_cast<const __nv_bfloat16*>(tile + tile_off(r, c)));
  }
  return sum;
}

// Weighted column sums sum_s w_s tile[s][c] of a tile's halves h of 64
// samples (w in shared memory) to s_part[h][c]: the samples of each 32 add up
// as a butterfly does (16 apart, then 8, 4, 2, 1), and the two 32s of a half.
// Thread (h, j, q) has the samples 64 h + 8 i + q of the columns 8 j .. 8 j + 7.
__device__ __forceinline__ void weighted_column_sums(const uint8_t* tile, const float* w, float* s_part) {
  const int q = threadIdx.x & 7, j = (threadIdx.x >> 3) & 15, h = threadIdx.x >> 7;
  float a[2][8];
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    float v[4][8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int r = 64 * h + 32 * g + 8 * i + q;
      const uint4 raw = *reinterpret_cast<const uint4*>(tile + tile_off(r, 8 * j));
      const __nv_bfloat16* hb = reinterpret_cast<const __nv_bfloat16*>(&raw);
#pragma unroll
      for (int k = 0; k < 8; ++k) v[i][k] = __fmul_rn(w[r], __bfloat162float(hb[k]));
    }
#pragma unroll
    for (int k = 0; k < 8; ++k) a[g][k] = (v[0][k] + v[2][k]) + (v[1][k] + v[3][k]);
#pragma unroll
    for (int o = 4; o > 0; o >>= 1)
#pragma unroll
      for (int k = 0; k < 8; ++k) a[g][k] += __shfl_xor_sync(0xffffffffu, a[g][k], o);
  }
  if (q == 0)
#pragma unroll
    for (int k = 0; k < 8; ++k) s_part[h * F + 8 * j + k] = a[0][k] + a[1][k];
}

// ---------------------------------------------------------------------------
// Gradients: forward and backward of a batch in one kernel.  Each CTA runs
// the sample tiles blockIdx.x, blockIdx.x + gridDim.x, ...  A tile's
// activations stay in shared memory (X, a_1, a_2; a_3 takes W_1's place,
// which is staged again for the next tile, and the deltas d_3, d_2, d_1 take
// a_3's), and the transposed products read the same tiles as MN-major
// operands.  The three weight gradients accumulate in tensor memory across
// the CTA's tiles (gW_l in columns [128 l, 128 l + 128); z and dH of the
// current layer in [384, 512)); the bias, w4 and b4 gradients and the loss
// accumulate in shared memory and registers.  At the end the CTA writes its
// sums as row blockIdx.x of Gp [gridDim.x][NG_STRIDE], laid out as G =
// [gW (3x128x128) | gb (3x128) | gw4 (128) | gb4 (1) | loss (1)]; the rows
// are added in a fixed order (no atomics in global memory, the same gradient
// bits on every run).
// Bound by the chain of a tile (six products with their epilogues): at 8,192
// samples 64 CTAs have one tile each, 24.5 us.  The separate forward (19.5
// us) and backward (70.7 us: explicit 2-byte transposes of d and a, 640
// shuffles for gw4, 2-byte loads of the activations) took 90 us for such a
// batch; this kernel with rows of Gp in parameter order 30 us.
// A row's weight gradients lie as the accumulators are read out, four columns
// of 128 rows at a time (whole 512-byte stores of a warp).
constexpr int NG_ROW = 3 * F * F + 3 * F + F + 1 + 1;
// The element of G's order at place j of a row.
__device__ __forceinline__ int grad_element(int j) {
  if (j >= 3 * F * F) return j;
  const int l = j / (F * F), c = (j / (4 * F)) % (F / 4), r = (j / 4) % F;
  return (l * F + r) * F + c * 4 + j % 4;
}
// rows of Gp start on 16-byte boundaries (the weight gradients are stored as
// float4)
constexpr int NG_STRIDE = (NG_ROW + 3) & ~3;

__global__ void __launch_bounds__(THREADS, 1)
    k_mlp_grad(const __nv_bfloat16* __restrict__ X, int n, const __nv_bfloat16* __restrict__ Wt,
               const float* __restrict__ P4, const float* __restrict__ t, float inv_n, float* __restrict__ Gp, int* err) {
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint8_t* tD = base;                       // W_1, then a_3, then the deltas
  uint8_t* tW2 = base + TILE_BYTES;
  uint8_t* tW3 = base + 2 * TILE_BYTES;
  uint8_t* tX = base + 3 * TILE_BYTES;
  uint8_t* tA1 = base + 4 * TILE_BYTES;
  uint8_t* tA2 = base + 5 * TILE_BYTES;
  float* s_b = reinterpret_cast<float*>(base + 6 * TILE_BYTES);  // [3][128] biases
  float* s_w4 = s_b + 3 * F;                                      // [128]
  float* s_out = s_w4 + F;                                        // [128]
  float* s_dy = s_out + F;                                        // [128]
  float* s_g = s_dy + F;         // [4][128] gradient sums gb_1, gb_2, gb_3, gw4, each entry one thread's
  float* s_part = s_g + 4 * F;   // [2][128] the tile's gw4 by halves
  float* s_red = s_part + 2 * F;  // [2][4] per-warp gb4 and loss
  SmemW* sm = reinterpret_cast<SmemW*>(s_red + 8);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int ntiles = (n + TILE - 1) / TILE;
  if ((int)blockIdx.x >= ntiles) return;
  if (tid == 0) {
    mbar_init(&sm->bar, 1);
    mbar_init(&sm->bar_w, 1);
    sm->fail = 0;
    mbar_expect_tx(&sm->bar_w, 3 * TILE_BYTES);
    bulk_tile(tD, Wt, &sm->bar_w);
    bulk_tile(tW2, Wt + (size_t)F * F, &sm->bar_w);
    bulk_tile(tW3, Wt + (size_t)2 * F * F, &sm->bar_w);
  }
  for (int i = tid; i < 4 * F; i += THREADS) s_b[i] = __ldg(P4 + i);  // b and w4
  for (int i = tid; i < 4 * F; i += THREADS) s_g[i] = 0.f;
  __syncwarp();
  if (warp == 0) tmem_alloc(&sm->tmem, 512);
  fence_before();
  __syncthreads();
  fence_after();
  const uint32_t tm = sm->tmem, tz = tm + 384;
  const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
  const int r = (warp & 3) * 32 + lane;  // sample row of this thread
  const int c0 = (warp >> 2) * 64;       // and its first column
  const float b4 = __ldg(P4 + 4 * F);
  float gb4_acc = 0.f, loss_acc = 0.f;  // warps 4-7
  uint32_t phase = 0, phase_w = 0;
  bool ok = true, w_pending = true, mma_pending = false, first = true;
  // one group of MMAs issued by thread 0, waited for by all
  auto finish = [&]() {
    mma_pending = true;
    ok = __syncthreads_and(mbar_wait(&sm->bar, phase)) != 0;
    if (ok) {
      mma_pending = false;
      phase ^= 1;
      fence_after();
    }
    return ok;
  };
  // generic writes to the tiles, before the tensor cores (or a bulk copy) use them
  auto publish = [&]() {
    fence_async_smem();
    fence_before();
    __syncthreads();
    fence_after();
  };
  for (int tile = blockIdx.x; tile < ntiles && ok; tile += gridDim.x) {
    const int s0 = tile * TILE;
    if (!first && tid == 0) {
      // (the deltas' last product is done and the barrier after it passed)
      mbar_expect_tx(&sm->bar_w, TILE_BYTES);
      bulk_tile(tD, Wt, &sm->bar_w);
    }
    w_pending = true;
    const bool valid = s0 + r < n;
    const float tv = warp >= 4 && valid ? __ldg(t + s0 + r) : 0.f;
    load_rows(tX, X, s0, n);
    publish();
    ok = __syncthreads_and(mbar_wait(&sm->bar_w, phase_w)) != 0;
    if (!ok) break;
    w_pending = false;
    phase_w ^= 1;
    // forward
    float out = 0.f;
    for (int l = 0; l < 3; ++l) {
      if (tid == 0) {
        mma_tile(tz, l == 0 ? tX : l == 1 ? tA1 : tA2, false, l == 0 ? tD : l == 1 ? tW2 : tW3, false, false);
        mma_commit(&sm->bar);
      }
      if (!finish()) break;
      out = layer_epilogue(tz, s_b + l * F, l == 0 ? tA1 : l == 1 ? tA2 : tD, l == 2 ? s_w4 : nullptr, s_out);
      if (l < 2) publish();
    }
    if (!ok) break;
    // output layer
    if (warp >= 4) {
      float dy = 0.f;
      if (valid) {
        const float e = (out + b4) - tv;
        dy = e * inv_n;
        loss_acc += 0.5f * e * e * inv_n;
      }
      gb4_acc += dy;
      s_dy[r] = dy;
    }
    __syncthreads();
    weighted_column_sums(tD, s_dy, s_part);
    __syncthreads();
    if (tid < F) s_g[3 * F + tid] += s_part[tid] + s_part[F + tid];  // gw4
    // d_3 = bf16(dy w4 [a_3 > 0]) over a_3
    {
      const float dy = s_dy[r];
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        uint4* p = reinterpret_cast<uint4*>(tD + tile_off(r, c0 + q * 8));
        const uint4 raw = *p;
        const __nv_bfloat16* hb = reinterpret_cast<const __nv_bfloat16*>(&raw);
        float dv[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) dv[k] = __bfloat162float(hb[k]) > 0.f ? dy * s_w4[c0 + q * 8 + k] : 0.f;
        *p = pack8(dv);
      }
    }
    publish();
    for (int l = 2; l >= 0; --l) {
      const uint8_t* below = l == 2 ? tA2 : l == 1 ? tA1 : tX;  // a_l, the layer's input
      if (tid == 0) {
        mma_tile(tm + l * 128, tD, true, below, true, !first);                            // gW_l (+)= d^T a_l
        if (l > 0) mma_tile(tz, tD, false, l == 2 ? tW3 : tW2, true, false);  // dH = d W
        mma_commit(&sm->bar);
      }
      if (tid < F) s_g[l * F + tid] += column_sum(tD);  // gb_l, while the tensor cores read the same tile
      if (!finish()) break;
      if (l > 0) {
        // the next delta, bf16(dH [a_l > 0])
        float v[64];
        tmem_ld32(tz + lanes + c0, v);
        tmem_ld32(tz + lanes + c0 + 32, v + 32);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const uint4 raw = *reinterpret_cast<const uint4*>(below + tile_off(r, c0 + q * 8));
          const __nv_bfloat16* hb = reinterpret_cast<const __nv_bfloat16*>(&raw);
#pragma unroll
          for (int k = 0; k < 8; ++k) v[q * 8 + k] = __bfloat162float(hb[k]) > 0.f ? v[q * 8 + k] : 0.f;
          *reinterpret_cast<uint4*>(tD + tile_off(r, c0 + q * 8)) = pack8(v + q * 8);
        }
        publish();
      }
    }
    if (!ok) break;
    publish();  // before the next tile's copies land over this one's
    first = false;
  }
  if (ok) {
    float* row = Gp + (size_t)blockIdx.x * NG_STRIDE;
    // weight gradients: row r's 64 columns of each gW_l from tensor memory
    for (int l = 0; l < 3; ++l)
      for (int c = 0; c < 64; c += 32) {
        float v[32];
        tmem_ld32(tm + lanes + l * 128 + c0 + c, v);
        float4* dst = reinterpret_cast<float4*>(row) + (size_t)(l * (F / 4) + (c0 + c) / 4) * F + r;
#pragma unroll
        for (int q = 0; q < 8; ++q) dst[q * F] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
      }
    for (int o = 16; o > 0; o >>= 1) {
      gb4_acc += __shfl_xor_sync(0xffffffffu, gb4_acc, o);
      loss_acc += __shfl_xor_sync(0xffffffffu, loss_acc, o);
    }
    if (lane == 0 && warp >= 4) {
      s_red[warp - 4] = gb4_acc;
      s_red[warp] = loss_acc;
    }
    __syncthreads();
    // gb and gw4
    for (int i = tid; i < 4 * F; i += THREADS) row[3 * F * F + i] = s_g[i];
    if (tid == 0) {
      row[3 * F * F + 4 * F] = (s_red[0] + s_red[1]) + (s_red[2] + s_red[3]);
      row[3 * F * F + 4 * F + 1] = (s_red[4] + s_red[5]) + (s_red[6] + s_red[7]);
    }
  } else {
    sm->fail = 1;
    if (err) atomicExch(err, 1);
    // drain (bounded) before the tensor memory goes
    if (w_pending) mbar_wait(&sm->bar_w, phase_w);
    if (mma_pending) mbar_wait(&sm->bar, phase);
  }
  fence_before();
  __syncthreads();
  fence_after();
  if (warp == 0) tmem_dealloc(tm, 512);
}

// Sum of place i of the rows of Gp, in row order.
__device__ __forceinline__ float row_sum(const float* __restrict__ Gp, int rows, int i) {
  float sum = 0.f;
  int r = 0;
  for (; r + 8 <= rows; r += 8) {
    float v[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) v[k] = __ldg(Gp + (size_t)(r + k) * NG_STRIDE + i);
#pragma unroll
    for (int k = 0; k < 8; ++k) sum += v[k];
  }
  for (; r < rows; ++r) sum += __ldg(Gp + (size_t)r * NG_STRIDE + i);
  return sum;
}

// G[i] = sum over the rows of Gp (fixed order).
__global__ void k_mlp_reduce(const float* __restrict__ Gp, int rows, float* __restrict__ G) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < NG_ROW; i += gridDim.x * blockDim.x)
    G[grad_element(i)] = row_sum(Gp, rows, i);
}

// ---------------------------------------------------------------------------
// Gradient reduction and Adam in one pass: each thread adds up its
// parameter's rows of Gp (fixed order) and steps the fp32 master parameter P
// = [W (3x128x128) | b (3x128) | w4 | b4], refreshing the BF16 weight tiles;
// the batch's loss is added to *loss_acc (the epoch's sum on the device).
__global__ void k_adam(float* __restrict__ P, const float* __restrict__ Gp, int rows, float* __restrict__ M1,
                       float* __restrict__ M2, int np, float lr, float b1, float b2, float eps, float c1, float c2,
                       __nv_bfloat16* __restrict__ Wt, float* __restrict__ loss_acc) {
  const int j = blockIdx.x * blockDim.x + threadIdx.x;
  if (j >= NG_ROW) return;
  const float g = row_sum(Gp, rows, j);
  const int i = grad_element(j);
  if (i >= np) {
    *loss_acc += g;
    return;
  }
  const float m = b1 * M1[i] + (1.f - b1) * g;
  const float v = b2 * M2[i] + (1.f - b2) * g * g;
  M1[i] = m;
  M2[i] = v;
  const float p = P[i] - lr * (m * c1) / (sqrtf(v * c2) + eps);
  P[i] = p;
  if (i < 3 * F * F) store_weight(Wt, i, p);
}

__global__ void k_pack_weights(const float* __restrict__ P, __nv_bfloat16* __restrict__ Wt) {
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 3 * F * F; i += gridDim.x * blockDim.x)
    store_weight(Wt, i, P[i]);
}

// BF16 copies of fp32 values, four per thread at a time; vec: both arrays
// start on a boundary of four values.  `in` may be the caller's host array
// where the GPU can read it: the conversion then costs the transfer alone.
__global__ void k_to_bf16(const float* __restrict__ in, size_t n, int vec, __nv_bfloat16* __restrict__ out) {
  const size_t stride = (size_t)gridDim.x * blockDim.x;
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; 4 * i < n; i += stride) {
    if (vec && 4 * i + 4 <= n) {
      const float4 v = *reinterpret_cast<const float4*>(in + 4 * i);
      __nv_bfloat162 p[2] = {__floats2bfloat162_rn(v.x, v.y), __floats2bfloat162_rn(v.z, v.w)};
      *reinterpret_cast<uint2*>(out + 4 * i) = *reinterpret_cast<uint2*>(p);
    } else {
      float v[4];
      for (int k = 0; k < 4; ++k) v[k] = 4 * i + k < n ? in[4 * i + k] : 0.f;
      for (int k = 0; k < 4; ++k)
        if (4 * i + k < n) out[4 * i + k] = __float2bfloat16_rn(v[k]);
    }
  }
}

// ---------------------------------------------------------------------------
// Features of the vertices in vlist (product vertex ids): slot 0 = the vertex
// itself (0, 0, 0, phi / h), slots 1..31 = its first 31 1-ring neighbours
// (ascending id) as (dx, dy, dz, phi) / h, zeros beyond the ring.  h is
// 1 / inv_h, or 1 / vinv_h[v] per vertex when given (batches of meshes of
// different resolution).
__global__ void k_features(int nlist, const int* __restrict__ vlist, const int* __restrict__ nlist_dev,
                           const int* __restrict__ adj_off, const int* __restrict__ adj, const float* __restrict__ xyz,
                           int nv, const float* __restrict__ phi, float inv_h, const float* __restrict__ vinv_h,
                           __nv_bfloat16* __restrict__ Xo) {
  if (nlist_dev) nlist = *nlist_dev;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < nlist; i += gridDim.x * blockDim.x) {
    const int v = vlist[i];
    if (vinv_h) inv_h = vinv_h[v];
    const float x0 = xyz[v], y0 = xyz[nv + v], z0 = xyz[2 * (size_t)nv + v];
    const int a = adj_off[v], e = adj_off[v + 1];
    __nv_bfloat16* dst = Xo + (size_t)i * F;
    for (int slot = 0; slot < 32; ++slot) {
      float f[4] = {0.f, 0.f, 0.f, 0.f};
      if (slot == 0) {
        f[3] = phi[v] * inv_h;
      } else if (a + slot - 1 < e) {
        const int u = adj[a + slot - 1];
        f[0] = (xyz[u] - x0) * inv_h;
        f[1] = (xyz[nv + u] - y0) * inv_h;
        f[2] = (xyz[2 * (size_t)nv + u] - z0) * inv_h;
        f[3] = phi[u] * inv_h;
      }
      __nv_bfloat162 p0 = __floats2bfloat162_rn(f[0], f[1]);
      __nv_bfloat162 p1 = __floats2bfloat162_rn(f[2], f[3]);
      uint2 o;
      o.x = *reinterpret_cast<uint32_t*>(&p0);
      o.y = *reinterpret_cast<uint32_t*>(&p1);
      *reinterpret_cast<uint2*>(dst + slot * 4) = o;
    }
  }
}

// Training pairs: rows i < *n of X / t with a finite target are appended to
// the pair buffer (capacity cap; overflow is counted, not written).
__global__ void k_append_pairs(const __nv_bfloat16* __restrict__ X, const float* __restrict__ t, const int* n_dev,
                               __nv_bfloat16* __restrict__ PX, float* __restrict__ PT,
                               unsigned long long* count, long long cap) {
  const int n = *n_dev;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float v = t[i];
    if (!isfinite(v)) continue;
    const unsigned long long pos = atomicAdd(count, 1ull);
    if ((long long)pos >= cap) continue;
    const uint4* src = reinterpret_cast<const uint4*>(X + (size_t)i * F);
    uint4* dst = reinterpret_cast<uint4*>(PX + (size_t)pos * F);
#pragma unroll 4
    for (int j = 0; j < F / 8; ++j) dst[j] = src[j];
    PT[pos] = v;
  }
}

// rows perm[i] of (X, t) -> row i of (Xo, to)
__global__ void k_gather_pairs(const __nv_bfloat16* __restrict__ X, const float* __restrict__ t,
                               const int* __restrict__ perm, long long n, __nv_bfloat16* __restrict__ Xo,
                               float* __restrict__ to) {
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const long long j = perm[i];
    const uint4* src = reinterpret_cast<const uint4*>(X + (size_t)j * F);
    uint4* dst = reinterpret_cast<uint4*>(Xo + (size_t)i * F);
#pragma unroll 4
    for (int q = 0; q < F / 8; ++q) dst[q] = src[q];
    to[i] = t[j];
  }
}

// ---------------------------------------------------------------------------
// Host side.

namespace {
constexpr int NP = 3 * F * F + 3 * F + F + 1;  // master parameters
constexpr int NG = NP + 1;                      // gradients + loss
static_assert(NG == NG_ROW, "gradient row layout");
size_t fwd_smem() { return 4 * (size_t)TILE_BYTES + 5 * F * sizeof(float) + 1024 + 64; }
size_t grad_smem() { return 6 * (size_t)TILE_BYTES + (12 * F + 8) * sizeof(float) + 1024 + 64; }
size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }
}  // namespace

#define MLP_TRY(expr, what)                                                     \
  do {                                                                          \
    cudaError_t _e = (expr);                                                    \
    if (_e != cudaSuccess) return std::string(what) + ": " + cudaGetErrorString(_e); \
  } while (0)

Net::~Net() {
  if (ws_) cudaFree(ws_);
  if (h_end_) cudaFreeHost(h_end_);
  for (void* p : allocs_) cudaFree(p);
  if (PX_) cudaFree(PX_);
  if (PT_) cudaFree(PT_);
  if (pair_count_) cudaFree(pair_count_);
  for (cudaEvent_t e : uploaded_)
    if (e) cudaEventDestroy(e);
  if (upload_) cudaStreamDestroy(upload_);
  if (stream_) cudaStreamDestroy(stream_);
}

std::string Net::init(unsigned long long seed) {
  MLP_TRY(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking), "stream");
  MLP_TRY(cudaStreamCreateWithFlags(&upload_, cudaStreamNonBlocking), "stream");
  for (cudaEvent_t& e : uploaded_) MLP_TRY(cudaEventCreateWithFlags(&e, cudaEventDisableTiming), "event");
  auto alloc = [&](void** p, size_t bytes) -> cudaError_t {
    cudaError_t e = cudaMalloc(p, bytes);
    if (e == cudaSuccess) allocs_.push_back(*p);
    return e;
  };
  MLP_TRY(alloc((void**)&P_, sizeof(float) * NP), "alloc");
  MLP_TRY(alloc((void**)&G_, sizeof(float) * NG), "alloc");
  MLP_TRY(alloc((void**)&M1_, sizeof(float) * NP), "alloc");
  MLP_TRY(alloc((void**)&M2_, sizeof(float) * NP), "alloc");
  MLP_TRY(alloc((void**)&Wb_, sizeof(__nv_bfloat16) * 3 * F * F), "alloc");
  // the error word, then the epoch's loss: read together
  MLP_TRY(alloc((void**)&err_, 2 * sizeof(int)), "alloc");
  loss_acc_ = reinterpret_cast<float*>(err_ + 1);
  MLP_TRY(cudaMallocHost((void**)&h_end_, 2 * sizeof(int)), "pinned");
  {
    int dev = 0;
    MLP_TRY(cudaGetDevice(&dev), "device");
    MLP_TRY(cudaDeviceGetAttribute(&sms_, cudaDevAttrMultiProcessorCount, dev), "device");
    if (sms_ < 1) sms_ = 1;
  }
  set_host_staging(false);
  // one partial-gradient row per backward CTA (at most one CTA per SM)
  MLP_TRY(alloc((void**)&Gp_, sizeof(float) * (size_t)NG_STRIDE * sms_), "alloc");
  MLP_TRY(cudaMemsetAsync(M1_, 0, sizeof(float) * NP, stream_), "memset");
  MLP_TRY(cudaMemsetAsync(M2_, 0, sizeof(float) * NP, stream_), "memset");
  MLP_TRY(cudaMemsetAsync(err_, 0, sizeof(int), stream_), "memset");
  MLP_TRY(cudaFuncSetAttribute(k_mlp_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)fwd_smem()), "attr");
  MLP_TRY(cudaFuncSetAttribute(k_mlp_grad, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)grad_smem()), "attr");
  // He-uniform initialisation of the weights, zero biases
  std::mt19937_64 rng(seed);
  std::vector<float> p(NP, 0.f);
  const float lim = std::sqrt(6.f / F);
  std::uniform_real_distribution<float> U(-lim, lim);
  for (int i = 0; i < 3 * F * F; ++i) p[i] = U(rng);
  std::uniform_real_distribution<float> U4(-std::sqrt(3.f / F), std::sqrt(3.f / F));
  for (int i = 0; i < F; ++i) p[3 * F * F + 3 * F + i] = U4(rng);
  return set_params(p.data());
}

// Host rows through a device copy (on), or read by the GPU where they are if
// it can access pageable memory.
std::string Net::set_host_staging(bool on) {
  int dev = 0;
  pageable_ = 0;
  if (on) return "";
  MLP_TRY(cudaGetDevice(&dev), "device");
  if (cudaDeviceGetAttribute(&pageable_, cudaDevAttrPageableMemoryAccess, dev) != cudaSuccess) pageable_ = 0;
  return "";
}

std::string Net::set_params(const float* host) {
  MLP_TRY(cudaMemcpyAsync(P_, host, sizeof(float) * NP, cudaMemcpyHostToDevice, stream_), "h2d");
  k_pack_weights<<<96, 256, 0, stream_>>>(P_, Wb_);
  MLP_TRY(cudaGetLastError(), "pack");
  MLP_TRY(cudaMemsetAsync(M1_, 0, sizeof(float) * NP, stream_), "memset");
  MLP_TRY(cudaMemsetAsync(M2_, 0, sizeof(float) * NP, stream_), "memset");
  step_ = 0;
  MLP_TRY(cudaStreamSynchronize(stream_), "sync");
  return "";
}

std::string Net::get_params(float* host) {
  MLP_TRY(cudaMemcpyAsync(host, P_, sizeof(float) * NP, cudaMemcpyDeviceToHost, stream_), "d2h");
  MLP_TRY(cudaStreamSynchronize(stream_), "sync");
  return "";
}

int Net::num_params() { return NP; }

// Waits for the stream; the error word and, when given, the epoch's loss.
std::string Net::finish(float* loss) {
  MLP_TRY(cudaMemcpyAsync(h_end_, err_, 2 * sizeof(int), cudaMemcpyDeviceToHost, stream_), "d2h");
  MLP_TRY(cudaStreamSynchronize(stream_), "sync");
  if (loss) std::memcpy(loss, h_end_ + 1, sizeof(float));
  if (h_end_[0]) {
    cudaMemsetAsync(err_, 0, sizeof(int), stream_);
    return "tensor-core wait timed out";
  }
  return "";
}

// Workspace of the host-buffer entry points: grown to the largest call, kept
// up to kWorkspaceKeep bytes (trim, with the stream idle).
char* Net::workspace(size_t bytes) {
  if (bytes > ws_bytes_) {
    if (ws_) cudaFree(ws_);
    ws_ = nullptr;
    ws_bytes_ = 0;
    if (cudaMalloc((void**)&ws_, bytes) != cudaSuccess) {
      cudaGetLastError();
      ws_ = nullptr;
      return nullptr;
    }
    ws_bytes_ = bytes;
  }
  return ws_;
}
std::string Net::trim(std::string r) {
  if (ws_bytes_ > kWorkspaceKeep) {
    cudaStreamSynchronize(stream_);
    cudaFree(ws_);
    ws_ = nullptr;
    ws_bytes_ = 0;
  }
  return r;
}
size_t Net::staging_bytes(size_t n) const { return pageable_ ? 0 : align256(n * F * sizeof(float)); }

// Host rows -> BF16 on the device, through the GPU's own access to the
// caller's array where it has it, otherwise through `staging`.
std::string Net::upload_rows(const float* Xh, size_t n, __nv_bfloat16* X, char* staging, cudaStream_t st) {
  const float* src = Xh;
  if (!pageable_) {
    MLP_TRY(cudaMemcpyAsync(staging, Xh, sizeof(float) * n * F, cudaMemcpyHostToDevice, st), "h2d");
    src = reinterpret_cast<const float*>(staging);
  }
  const size_t quads = (n * F + 3) / 4;
  const int grid = (int)std::min<size_t>((quads + 255) / 256, (size_t)sms_ * 8);
  k_to_bf16<<<grid, 256, 0, st>>>(src, n * F, (reinterpret_cast<uintptr_t>(src) & 15) == 0, X);
  MLP_TRY(cudaGetLastError(), "conversion");
  return "";
}

std::string Net::forward_dev(const __nv_bfloat16* X, int n, const int* n_dev, int max_n, float* y, cudaStream_t st) {
  // one CTA per SM at most, each over several sample tiles (the weights are
  // staged once per CTA)
  const int tiles = (max_n + TILE - 1) / TILE;
  const int grid = tiles < sms_ ? tiles : sms_;
  if (grid <= 0) return "";
  k_mlp_fwd<<<grid, THREADS, fwd_smem(), st>>>(X, n, n_dev, Wb_, P_ + 3 * F * F, y, err_);
  MLP_TRY(cudaGetLastError(), "mlp forward");
  return "";
}

std::string Net::gradient_rows(const __nv_bfloat16* X, int n, const float* t, int* rows) {
  const int tiles = (n + TILE - 1) / TILE;
  *rows = tiles < sms_ ? tiles : sms_;
  if (*rows <= 0) return "";
  k_mlp_grad<<<*rows, THREADS, grad_smem(), stream_>>>(X, n, Wb_, P_ + 3 * F * F, t, 1.f / n, Gp_, err_);
  MLP_TRY(cudaGetLastError(), "mlp gradients");
  return "";
}

std::string Net::predict(const float* Xh, int n, float* yh) {
  if (n <= 0) return "";
  const size_t bx = align256(sizeof(__nv_bfloat16) * (size_t)n * F), by = align256(sizeof(float) * (size_t)n);
  char* w = workspace(bx + by + staging_bytes(n));
  if (!w) return "alloc";
  __nv_bfloat16* X = reinterpret_cast<__nv_bfloat16*>(w);
  float* y = reinterpret_cast<float*>(w + bx);
  std::string r = upload_rows(Xh, n, X, w + bx + by, stream_);
  if (r.empty()) r = forward_dev(X, n, nullptr, n, y, stream_);
  if (r.empty()) {
    cudaError_t e = cudaMemcpyAsync(yh, y, sizeof(float) * n, cudaMemcpyDeviceToHost, stream_);
    if (e != cudaSuccess) r = std::string("d2h: ") + cudaGetErrorString(e);
  }
  const std::string f = finish(nullptr);
  return trim(r.empty() ? f : r);
}

std::string Net::gradients(const float* Xh, const float* th, int n, float* gh, float* loss) {
  if (n <= 0) return "empty batch";
  const size_t bx = align256(sizeof(__nv_bfloat16) * (size_t)n * F), bt = align256(sizeof(float) * (size_t)n);
  char* w = workspace(bx + bt + staging_bytes(n));
  if (!w) return "alloc";
  __nv_bfloat16* X = reinterpret_cast<__nv_bfloat16*>(w);
  float* t = reinterpret_cast<float*>(w + bx);
  auto body = [&]() -> std::string {
    std::string r = upload_rows(Xh, n, X, w + bx + bt, stream_);
    if (!r.empty()) return r;
    MLP_TRY(cudaMemcpyAsync(t, th, sizeof(float) * n, cudaMemcpyHostToDevice, stream_), "h2d");
    int rows = 0;
    r = gradient_rows(X, n, t, &rows);
    if (!r.empty()) return r;
    k_mlp_reduce<<<(NG + 255) / 256, 256, 0, stream_>>>(Gp_, rows, G_);
    MLP_TRY(cudaGetLastError(), "mlp gradient reduction");
    MLP_TRY(cudaMemcpyAsync(gh, G_, sizeof(float) * NP, cudaMemcpyDeviceToHost, stream_), "d2h");
    MLP_TRY(cudaMemcpyAsync(loss_acc_, G_ + NP, sizeof(float), cudaMemcpyDeviceToDevice, stream_), "loss");
    return "";
  };
  std::string r = body();
  float l = 0.f;
  const std::string f = finish(&l);
  if (loss) *loss = l;
  return trim(r.empty() ? f : r);
}

std::string Net::train(const float* Xh, const float* th, int n, int epochs, int batch, float lr, float* last_loss) {
  if (n <= 0 || batch <= 0 || epochs <= 0) return "empty training set";
  const size_t bx = align256(sizeof(__nv_bfloat16) * (size_t)n * F), bt = align256(sizeof(float) * (size_t)n);
  char* w = workspace(bx + bt + staging_bytes(n));
  if (!w) return "alloc";
  __nv_bfloat16* X = reinterpret_cast<__nv_bfloat16*>(w);
  float* t = reinterpret_cast<float*>(w + bx);
  // The rows arrive in up to kUploads pieces of whole batches on a stream of
  // their own, the first epoch's batches wait for theirs: the transfer (150 us
  // for 25.6 MB) runs behind the training of the pieces before.
  const size_t batches = ((size_t)n + batch - 1) / batch;
  const size_t per = (batches + kUploads - 1) / kUploads * (size_t)batch;  // rows of a piece
  auto body = [&]() -> std::string {
    MLP_TRY(cudaMemcpyAsync(t, th, sizeof(float) * (size_t)n, cudaMemcpyHostToDevice, stream_), "h2d");
    int piece = 0;
    for (size_t r0 = 0; r0 < (size_t)n; r0 += per, ++piece) {
      const size_t rows = std::min(per, (size_t)n - r0);
      std::string r = upload_rows(Xh + r0 * F, rows, X + r0 * F, w + bx + bt + (pageable_ ? 0 : r0 * F * sizeof(float)),
                                  upload_);
      if (!r.empty()) return r;
      MLP_TRY(cudaEventRecord(uploaded_[piece], upload_), "event");
    }
    return train_device(X, t, n, epochs, batch, lr, last_loss, per);
  };
  std::string r = body();
  cudaStreamSynchronize(upload_);
  cudaStreamSynchronize(stream_);
  return trim(r);
}

std::string Net::train_device(const __nv_bfloat16* X, const float* t, int n, int epochs, int batch, float lr,
                              float* last_loss, size_t piece_rows) {
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  float loss_sum = 0.f;
  int loss_cnt = 0;
  for (int ep = 0; ep < epochs; ++ep) {
    // the batches' losses add up on the device; one read per epoch
    MLP_TRY(cudaMemsetAsync(loss_acc_, 0, sizeof(float), stream_), "memset");
    loss_cnt = 0;
    for (int s0 = 0; s0 < n; s0 += batch) {
      const int m = (n - s0) < batch ? (n - s0) : batch;
      if (piece_rows && ep == 0 && (size_t)s0 % piece_rows == 0)
        MLP_TRY(cudaStreamWaitEvent(stream_, uploaded_[(size_t)s0 / piece_rows], 0), "wait");
      int rows = 0;
      std::string r = gradient_rows(X + (size_t)s0 * F, m, t + s0, &rows);
      if (!r.empty()) return r;
      ++step_;
      const float c1 = 1.f / (1.f - std::pow(b1, (float)step_));
      const float c2 = 1.f / (1.f - std::pow(b2, (float)step_));
      k_adam<<<(NG + 127) / 128, 128, 0, stream_>>>(P_, Gp_, rows, M1_, M2_, NP, lr, b1, b2, eps, c1, c2, Wb_,
                                                    loss_acc_);
      MLP_TRY(cudaGetLastError(), "adam");
      ++loss_cnt;
    }
    std::string r = finish(&loss_sum);
    if (!r.empty()) return r;
  }
  if (last_loss) *last_loss = loss_cnt ? loss_sum / loss_cnt : 0.f;
  return "";
}

std::string Net::reserve_pairs(long long cap) {
  if (cap <= pair_cap_) return "";
  __nv_bfloat16* px = nullptr;
  float* pt = nullptr;
  MLP_TRY(cudaMalloc(&px, sizeof(__nv_bfloat16) * (size_t)cap * F), "alloc pairs");
  cudaError_t e = cudaMalloc(&pt, sizeof(float) * (size_t)cap);
  if (e != cudaSuccess) {
    cudaFree(px);
    return std::string("alloc pairs: ") + cudaGetErrorString(e);
  }
  if (!pair_count_) MLP_TRY(cudaMalloc(&pair_count_, sizeof(unsigned long long)), "alloc");
  long long have = 0;
  if (PX_) {
    have = num_pairs();
    if (have > 0) {
      cudaMemcpyAsync(px, PX_, sizeof(__nv_bfloat16) * (size_t)have * F, cudaMemcpyDeviceToDevice, stream_);
      cudaMemcpyAsync(pt, PT_, sizeof(float) * (size_t)have, cudaMemcpyDeviceToDevice, stream_);
    }
    cudaStreamSynchronize(stream_);
    cudaFree(PX_);
    cudaFree(PT_);
  }
  PX_ = px;
  PT_ = pt;
  pair_cap_ = cap;
  unsigned long long h = (unsigned long long)have;
  MLP_TRY(cudaMemcpyAsync(pair_count_, &h, sizeof(h), cudaMemcpyHostToDevice, stream_), "h2d");
  MLP_TRY(cudaStreamSynchronize(stream_), "sync");
  return "";
}

long long Net::num_pairs() {
  if (!pair_count_) return 0;
  unsigned long long h = 0;
  cudaMemcpyAsync(&h, pair_count_, sizeof(h), cudaMemcpyDeviceToHost, stream_);
  cudaStreamSynchronize(stream_);
  return (long long)(h < (unsigned long long)pair_cap_ ? h : (unsigned long long)pair_cap_);
}

std::string Net::clear_pairs() {
  if (pair_count_) MLP_TRY(cudaMemsetAsync(pair_count_, 0, sizeof(unsigned long long), stream_), "memset");
  MLP_TRY(cudaStreamSynchronize(stream_), "sync");
  return "";
}

std::string Net::append_pairs(const __nv_bfloat16* X, const float* t, const int* n_dev, int max_n, cudaStream_t st,
                              long long* added) {
  if (added) *added = 0;
  if (!PX_) {
    std::string r = reserve_pairs(1LL << 22);
    if (!r.empty()) return r;
  }
  const long long before = num_pairs();
  // the solver's stream produced X and t: order this stream after it
  cudaEvent_t ev;
  MLP_TRY(cudaEventCreateWithFlags(&ev, cudaEventDisableTiming), "event");
  cudaEventRecord(ev, st);
  cudaStreamWaitEvent(stream_, ev, 0);
  cudaEventDestroy(ev);
  const int grid = (max_n + 255) / 256 < 4096 ? (max_n + 255) / 256 : 4096;
  k_append_pairs<<<grid > 0 ? grid : 1, 256, 0, stream_>>>(X, t, n_dev, PX_, PT_, pair_count_, pair_cap_);
  MLP_TRY(cudaGetLastError(), "append pairs");
  MLP_TRY(cudaStreamSynchronize(stream_), "sync");
  if (added) *added = num_pairs() - before;
  return "";
}

std::string Net::eval_pairs(long long first, long long count, float* abs_err) {
  const long long n = num_pairs();
  if (first < 0 || count < 0 || first + count > n) return "pair range outside the buffer";
  if (count == 0) return "";
  if (count > 0x7fffffffLL) return "too many pairs";
  float* y = nullptr;
  MLP_TRY(cudaMalloc(&y, sizeof(float) * (size_t)count), "alloc");
  std::string r = forward_dev(PX_ + (size_t)first * F, (int)count, nullptr, (int)count, y, stream_);
  std::vector<float> yh((size_t)count), th((size_t)count);
  if (r.empty() &&
      (cudaMemcpyAsync(yh.data(), y, sizeof(float) * (size_t)count, cudaMemcpyDeviceToHost, stream_) != cudaSuccess ||
       cudaMemcpyAsync(th.data(), PT_ + first, sizeof(float) * (size_t)count, cudaMemcpyDeviceToHost, stream_) !=
           cudaSuccess))
    r = "d2h";
  cudaStreamSynchronize(stream_);
  cudaFree(y);
  if (!r.empty()) return r;
  for (long long i = 0; i < count; ++i) abs_err[i] = std::fabs(yh[(size_t)i] - th[(size_t)i]);
  return finish(nullptr);
}

std::string Net::train_pairs(int epochs, int batch, float lr, unsigned long long seed, float* last_loss) {
  const long long n = num_pairs();
  if (n <= 0) return "no training pairs";
  if (n > 0x7fffffffLL) return "too many pairs";
  // one shuffle of the pairs, then epochs of sequential batches
  std::vector<int> perm((size_t)n);
  for (long long i = 0; i < n; ++i) perm[(size_t)i] = (int)i;
  std::mt19937_64 rng(seed);
  std::shuffle(perm.begin(), perm.end(), rng);
  std::vector<void*> tmp;
  auto fin = [&](const std::string& r) {
    cudaStreamSynchronize(stream_);
    for (void* p : tmp) cudaFree(p);
    return r;
  };
  int* dperm = nullptr;
  __nv_bfloat16* Xs = nullptr;
  float* ts = nullptr;
  if (cudaMalloc(&dperm, sizeof(int) * (size_t)n) != cudaSuccess) return fin("alloc");
  tmp.push_back(dperm);
  if (cudaMalloc(&Xs, sizeof(__nv_bfloat16) * (size_t)n * F) != cudaSuccess) return fin("alloc");
  tmp.push_back(Xs);
  if (cudaMalloc(&ts, sizeof(float) * (size_t)n) != cudaSuccess) return fin("alloc");
  tmp.push_back(ts);
  cudaMemcpyAsync(dperm, perm.data(), sizeof(int) * (size_t)n, cudaMemcpyHostToDevice, stream_);
  k_gather_pairs<<<4096, 256, 0, stream_>>>(PX_, PT_, dperm, n, Xs, ts);
  if (cudaGetLastError() != cudaSuccess) return fin("gather pairs");
  return fin(train_device(Xs, ts, (int)n, epochs, batch, lr, last_loss, 0));
}

}  // namespace mlp
}  // namespace lsgb
