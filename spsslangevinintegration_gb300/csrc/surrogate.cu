// Learned surrogate: the 5 -> 128 -> 128 -> 128 -> 4 GELU network of
// spss_surrogate.h, trained and evaluated by hand-written tcgen05 kernels.
//
// Tensor-core scheme (one CTA = 128 rows of a batch, 16 warps):
//   * operands live in shared memory in the K-major, no-swizzle canonical
//     layout: core matrices of 8 rows x 16 bytes (8 BF16), adjacent along K at
//     128 bytes (leading byte offset), row groups at K/8 * 128 bytes (stride
//     byte offset); the weight copies and the input tiles are kept in that
//     layout in global memory, so a tile or a set of weights is one bulk copy;
//   * one thread issues tcgen05.mma.cta_group::1.kind::f16 (BF16 x BF16 ->
//     FP32, M = 128, N = 128 or 16, K = 16 per instruction) into tensor memory
//     and commits to an mbarrier (bounded wait);
//   * after the wait every thread reads 32 columns of a row of the accumulator
//     with tcgen05.ld (warp w: lanes 32 (w mod 4) .. + 31, columns 32 (w / 4) ..
//     + 31), applies bias and GELU in FP32 and writes the BF16 activation into
//     shared memory as the next layer's A operand.
// Training: one kernel runs forward, loss, dZ_l = dA_l * GELU'(Z_l) with
// dA_{l-1} = dZ_l W_l, and dW_l = dZ_l^T A_{l-1} for its 128 rows.  The weight
// gradients read the same row-major tiles as MN-major operands (a core matrix
// of 8 rows x 8 columns serves either way; only the strides change names), so
// nothing is transposed.  Partial gradients are summed over CTAs in a fixed
// order; Adam on FP32 master weights.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <new>
#include <random>
#include <vector>

#include "spss_internal.cuh"
#include "spss_surrogate.h"

namespace spss
{
namespace mlp
{

constexpr int IN = SPSS_MLP_INPUTS, H = SPSS_MLP_HIDDEN, OUT = SPSS_MLP_OUTPUTS;
constexpr int INP = 16, OUTP = 16;  // input and output widths padded to the MMA granularity
constexpr int TR = 128;             // rows per CTA (MMA M)
constexpr int NP = SPSS_MLP_PARAMS;
constexpr int oW1 = 0, ob1 = oW1 + H * IN, oW2 = ob1 + H, ob2 = oW2 + H * H, oW3 = ob2 + H, ob3 = oW3 + H * H,
              oW4 = ob3 + H, ob4 = oW4 + OUT * H, oEnd = ob4 + OUT;
static_assert(oEnd == NP, "parameter count");
constexpr long long kWaitCycles = 1ll << 31;  // about one second at the SM clock
constexpr int kMaxPartials = 2 * 152;         // CTAs of the training kernel

typedef __nv_bfloat16 bf16;

// ---------------------------------------------------------------- tcgen05

__device__ __forceinline__ uint32_t smem_addr(const void *p)
{
  return (uint32_t) __cvta_generic_to_shared(p);
}

// Byte offset of element (r, k) of a K-major operand with K columns.
__device__ __forceinline__ uint32_t canon(int r, int k, int K)
{
  return (uint32_t) ((r >> 3) * (K >> 3) * 128 + (k >> 3) * 128 + (r & 7) * 16 + (k & 7) * 2);
}

// Shared-memory matrix descriptor: start address, leading and stride byte
// offsets (16-byte units), descriptor version 1, no swizzle.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr, uint32_t lbo, uint32_t sbo)
{
  return (uint64_t) ((addr >> 4) & 0x3FFFu) | ((uint64_t) ((lbo >> 4) & 0x3FFFu) << 16) |
         ((uint64_t) ((sbo >> 4) & 0x3FFFu) << 32) | ((uint64_t) 1 << 46);
}

// Instruction descriptor of kind::f16: FP32 accumulator, BF16 A and B, both
// K-major (or, `mn`, both MN-major), N >> 3 and M >> 4.
__device__ __forceinline__ constexpr uint32_t instr_desc(int M, int N, bool mn = false)
{
  return (1u << 4) | (1u << 7) | (1u << 10) | (mn ? (1u << 15) | (1u << 16) : 0u) | ((uint32_t) (N >> 3) << 17) |
         ((uint32_t) (M >> 4) << 24);
}

// An operand in shared memory: `lbo` and `sbo` of its descriptor, and the bytes
// from one K = 16 step to the next.  K-major: the tile is [rows of M or N][K
// columns]; MN-major: the same layout read as [K rows][columns of M or N].
struct Operand
{
  uint32_t addr, lbo, sbo, step;
};

__device__ __forceinline__ Operand k_major(const void *p, int K)
{
  return Operand{smem_addr(p), 128u, (uint32_t) (K >> 3) * 128u, 256u};
}

__device__ __forceinline__ Operand mn_major(const void *p, int columns)
{
  const uint32_t group = (uint32_t) (columns >> 3) * 128u;  // eight rows
  return Operand{smem_addr(p), group, 128u, 2u * group};
}

// D[128 x N] (+)= A B, K = 16 * steps.
__device__ __forceinline__ void mma_issue(uint32_t tmem, Operand a, Operand b, int steps, uint32_t idesc, bool accumulate)
{
  for (int kk = 0; kk < steps; ++kk)
  {
    const uint64_t ad = smem_desc(a.addr + kk * a.step, a.lbo, a.sbo);
    const uint64_t bd = smem_desc(b.addr + kk * b.step, b.lbo, b.sbo);
    const uint32_t acc = (accumulate || kk > 0) ? 1u : 0u;
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(
            tmem),
        "l"(ad), "l"(bd), "r"(idesc), "r"(acc));
  }
}

__device__ __forceinline__ void mma_commit(const unsigned long long *mbar)
{
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(mbar))
               : "memory");
}

__device__ __forceinline__ uint32_t wait_phase(const unsigned long long *mbar, uint32_t phase)
{
  uint32_t done = 0;
  const long long t0 = clock64();
  while (!done && clock64() - t0 < kWaitCycles)
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(done)
                 : "r"(smem_addr(mbar)), "r"(phase)
                 : "memory");
  return done;
}

__device__ __forceinline__ void fence_before_sync()
{
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
}

__device__ __forceinline__ void fence_after_sync()
{
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
}

// Operands written by threads become visible to the tensor cores, then a barrier.
__device__ __forceinline__ void publish_operands()
{
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  fence_before_sync();
  __syncthreads();
  fence_after_sync();
}

// 32 (16, 8) consecutive accumulator columns of this thread's row.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, float v[32])
{
  uint32_t r[32];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,"
      "%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
        "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
        "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]);
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float v[16])
{
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < 16; ++j) v[j] = __uint_as_float(r[j]);
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, float v[8])
{
  uint32_t r[8];
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int j = 0; j < 8; ++j) v[j] = __uint_as_float(r[j]);
}

// Tensor memory columns (a power of two), by one warp.
__device__ __forceinline__ void tmem_alloc(uint32_t *dst, uint32_t columns)
{
  asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(dst)), "r"(columns));
  asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}

__device__ __forceinline__ void tmem_dealloc(uint32_t tmem, uint32_t columns)
{
  asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(columns));
}

// Bulk copy global -> shared (both 16-byte aligned), completing on the mbarrier.
__device__ __forceinline__ void bulk_copy(void *dst, const void *src, uint32_t bytes, const unsigned long long *mbar)
{
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                   smem_addr(dst)),
               "l"(src), "r"(bytes), "r"(smem_addr(mbar))
               : "memory");
}

__device__ __forceinline__ void expect_bytes(const unsigned long long *mbar, uint32_t bytes)
{
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(mbar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ void mbar_init(unsigned long long *mbar)
{
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(mbar)));
  asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

// Eight consecutive columns c8 .. c8 + 7 of row r of a K-major operand.
__device__ __forceinline__ void put8(unsigned char *dst, int r, int c8, int K, const float v[8])
{
  __nv_bfloat162 h[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) h[j] = __floats2bfloat162_rn(v[2 * j], v[2 * j + 1]);
  *reinterpret_cast<uint4 *>(dst + canon(r, c8, K)) = *reinterpret_cast<const uint4 *>(h);
}

// GELU (exact, erf form) and its derivative.
__device__ __forceinline__ float gelu(float x)
{
  return 0.5f * x * (1.0f + erff(x * 0.70710678118654752f));
}

__device__ __forceinline__ void gelu_both(float x, float &g, float &dg)
{
  const float e = 1.0f + erff(x * 0.70710678118654752f);
  g = 0.5f * x * e;
  dg = 0.5f * e + x * 0.39894228040143268f * expf(-0.5f * x * x);
}

// BF16 weights in the canonical layout: forward B operands W1 [128][16], W2, W3
// [128][128], W4 [16][128]; backward B operands (transposes) W4t [128][16], W3t,
// W2t.  Offsets in elements.
constexpr int kF1 = 0, kF2 = kF1 + H * INP, kF3 = kF2 + H * H, kF4 = kF3 + H * H, kForward = kF4 + OUTP * H;
constexpr int kB4 = 0, kB3 = kB4 + H * OUTP, kB2 = kB3 + H * H, kBackward = kB2 + H * H;

struct Weights
{
  const float *p;        // FP32 master parameters (flat order)
  const bf16 *fwd, *bwd;
};

constexpr int kThreads = 512;
constexpr int kTileX = TR * INP * 2;  // bytes of an input tile
constexpr int kTileA = TR * H * 2;    // bytes of an activation tile
constexpr int kFwdSmem = kTileX + kTileA + kForward * 2;                                   // 108 KiB: two CTAs an SM
constexpr int kTrainSmem = kTileX + 4 * kTileA + TR * OUTP * 2 + kForward * 2;             // 208 KiB

// Accumulator columns c .. c + 7 of this thread's row plus their biases.
__device__ __forceinline__ void biased8(uint32_t trow, const float *b, int c, float v[8])
{
  const float4 b0 = __ldg(reinterpret_cast<const float4 *>(b + c)), b1 = __ldg(reinterpret_cast<const float4 *>(b + c + 4));
  tmem_ld8(trow + c, v);
  v[0] += b0.x;
  v[1] += b0.y;
  v[2] += b0.z;
  v[3] += b0.w;
  v[4] += b1.x;
  v[5] += b1.y;
  v[6] += b1.z;
  v[7] += b1.w;
}

// ---------------------------------------------------------------- forward

// Network outputs y [n][4] of the input tiles x (128 rows of BF16 [16] each, in
// the canonical layout; rows beyond n zero).  A CTA keeps the weights and takes
// tiles blockIdx.x, blockIdx.x + gridDim.x, ...  Bound by the GELUs (25 million
// at 65,536 rows, some 35 instructions each): with one thread a row and the
// weights staged by the threads for every tile 70 us there, now 37.
__global__ void __launch_bounds__(kThreads, 2) mlp_forward_kernel(Weights W, const bf16 *__restrict__ x, int n,
                                                                  float *__restrict__ y, int *status)
{
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char *sX = smem;
  unsigned char *sA = sX + kTileX;
  const bf16 *sW = reinterpret_cast<const bf16 *>(sA + kTileA);
  __shared__ __align__(8) unsigned long long mload, mmath;
  __shared__ uint32_t tmem_base;
  const int tid = threadIdx.x, warp = tid >> 5;
  const int tiles = (n + TR - 1) / TR;
  const int r = 32 * (warp & 3) + (tid & 31), c0 = 32 * (warp >> 2);
  if (warp == 0) tmem_alloc(&tmem_base, 128);
  if (tid == 0)
  {
    mbar_init(&mload);
    mbar_init(&mmath);
    expect_bytes(&mload, kForward * 2 + kTileX);
    bulk_copy((void *) sW, W.fwd, kForward * 2, &mload);
    bulk_copy(sX, x + (long) blockIdx.x * TR * INP, kTileX, &mload);
  }
  publish_operands();
  const uint32_t tmem = tmem_base;
  const uint32_t trow = tmem + ((uint32_t) (32 * (warp & 3)) << 16);
  uint32_t phase = 0, lphase = 0;
  bool ok = true;
  for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x)
  {
    ok = __syncthreads_and(wait_phase(&mload, lphase));
    if (!ok) break;
    lphase ^= 1u;
    for (int l = 0; l < 4 && ok; ++l)
    {
      if (tid == 0)
      {
        const bf16 *w = sW + (l == 0 ? kF1 : (l == 1 ? kF2 : (l == 2 ? kF3 : kF4)));
        const int K = l == 0 ? INP : H;
        mma_issue(tmem, k_major(l == 0 ? sX : sA, K), k_major(w, K), K / 16, instr_desc(TR, l == 3 ? OUTP : H), false);
        mma_commit(&mmath);
      }
      ok = __syncthreads_and(wait_phase(&mmath, phase));
      if (!ok) break;
      phase ^= 1u;
      fence_after_sync();
      if (l < 3)
      {
        if (l == 0 && tid == 0 && tile + (int) gridDim.x < tiles)
        {
          // the input tile has been read: fetch the next one
          expect_bytes(&mload, kTileX);
          bulk_copy(sX, x + (long) (tile + gridDim.x) * TR * INP, kTileX, &mload);
        }
        const float *b = W.p + (l == 0 ? ob1 : (l == 1 ? ob2 : ob3));
#pragma unroll 1
        for (int c = c0; c < c0 + 32; c += 8)
        {
          float v[8];
          biased8(trow, b, c, v);
#pragma unroll
          for (int j = 0; j < 8; ++j) v[j] = gelu(v[j]);
          put8(sA, r, c, H, v);
        }
        publish_operands();
      } else
      {
        const int row = tile * TR + r;
        if (warp < 4)
        {
          float v[16];
          tmem_ld16(trow, v);
          const float *b = W.p + ob4;
          if (row < n)
            *reinterpret_cast<float4 *>(y + (long) row * OUT) =
                make_float4(v[0] + __ldg(b), v[1] + __ldg(b + 1), v[2] + __ldg(b + 2), v[3] + __ldg(b + 3));
        }
        fence_before_sync();
        __syncthreads();  // the accumulator has been read
        fence_after_sync();
      }
    }
  }
  if (!ok)
  {
    // a copy or an accumulator did not complete in time: report and give what
    // is in flight a second bounded wait before the memory is released
    if (tid == 0) atomicOr(status, 1);
    wait_phase(&mload, lphase);
    wait_phase(&mmath, phase);
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 128);
}

// ---------------------------------------------------------------- training

struct Partials
{
  float *w[4];  // [cta][128][kin] per layer (layer 4: rows 0 .. 3)
  float *b[4];  // [cta][128]
};

// Sum over the 128 rows of column m of a tile with K columns, added to `s` in
// row order.
__device__ __forceinline__ float add_column(const unsigned char *tile, int m, int K, float s)
{
#pragma unroll 16
  for (int k = 0; k < TR; ++k) s += __bfloat162float(*reinterpret_cast<const bf16 *>(tile + canon(k, m, K)));
  return s;
}

// Loss and gradient partials of the rows of tiles blockIdx.x, blockIdx.x +
// gridDim.x, ... of a batch: forward, dZ4 = 2 w (y - t) / n_batch, dZ3, dZ2, dZ1
// and the weight gradients, each accumulated in its own tensor-memory columns.
// `dgelu`: scratch, 3 * 32 * 512 floats a CTA (GELU' of a thread's own
// elements, written and read back by the same thread).
// A minibatch of 1,024 rows is eight CTAs, each a chain of eleven MMA-epilogue
// stages, so latency is all there is: with a kernel each for forward, backward
// and the four weight gradients, one thread a row and the gradients' operands
// transposed by 2-byte stores, 69 + 89 + 4 * 16.5 us; this one 34 us.
__global__ void __launch_bounds__(kThreads, 1) mlp_train_kernel(Weights W, const bf16 *__restrict__ x,
                                                                const float *__restrict__ t, float4 wl, float scale,
                                                                int n, float *__restrict__ dgelu, Partials out,
                                                                float *__restrict__ loss_partial, int *status)
{
  extern __shared__ __align__(128) unsigned char smem[];
  unsigned char *sX = smem;
  unsigned char *sA1 = sX + kTileX;
  unsigned char *sA2 = sA1 + kTileA;  // later dZ1
  unsigned char *sA3 = sA2 + kTileA;  // later dZ2
  unsigned char *sD = sA3 + kTileA;   // dZ3
  unsigned char *sZ4 = sD + kTileA;   // dZ4 [128][16]
  const bf16 *sW = reinterpret_cast<const bf16 *>(sZ4 + TR * OUTP * 2);
  __shared__ __align__(8) unsigned long long mload, mmath;
  __shared__ uint32_t tmem_base;
  __shared__ float red[4];
  const int tid = threadIdx.x, warp = tid >> 5;
  const int tiles = (n + TR - 1) / TR;
  const int r = 32 * (warp & 3) + (tid & 31), c0 = 32 * (warp >> 2);
  // tensor-memory columns: the chain's accumulator and the weight gradients
  constexpr uint32_t kChain = 0, kG2 = 128, kG3 = 256, kG4 = 384, kG1 = 416;
  if (warp == 0) tmem_alloc(&tmem_base, 512);
  if (tid == 0)
  {
    mbar_init(&mload);
    mbar_init(&mmath);
  }
  publish_operands();
  const uint32_t tmem = tmem_base;
  const uint32_t trow = tmem + ((uint32_t) (32 * (warp & 3)) << 16);
  uint32_t phase = 0, lphase = 0;
  bool ok = true, any = false;
  float db[4] = {0.f, 0.f, 0.f, 0.f};  // bias gradients of column tid (tid < 128)
  float *const dg = dgelu + (long) blockIdx.x * 3 * 32 * kThreads + tid;
  auto done = [&]() -> bool {  // every thread: the committed MMAs are complete
    const bool all = __syncthreads_and(wait_phase(&mmath, phase));
    phase ^= all ? 1u : 0u;
    fence_after_sync();
    return all;
  };
  auto loaded = [&]() -> bool {
    const bool all = __syncthreads_and(wait_phase(&mload, lphase));
    lphase ^= all ? 1u : 0u;
    return all;
  };
  for (int tile = blockIdx.x; tile < tiles && ok; tile += gridDim.x)
  {
    const int row = tile * TR + r;
    const bool live = row < n;
    if (tid == 0)
    {
      expect_bytes(&mload, kForward * 2 + kTileX);
      bulk_copy(sX, x + (long) tile * TR * INP, kTileX, &mload);
      bulk_copy((void *) sW, W.fwd, kForward * 2, &mload);
    }
    if (!(ok = loaded())) break;
    // forward
    for (int l = 0; l < 3 && ok; ++l)
    {
      unsigned char *in = l == 0 ? sX : (l == 1 ? sA1 : sA2), *to = l == 0 ? sA1 : (l == 1 ? sA2 : sA3);
      if (tid == 0)
      {
        const int K = l == 0 ? INP : H;
        mma_issue(tmem + kChain, k_major(in, K), k_major(sW + (l == 0 ? kF1 : (l == 1 ? kF2 : kF3)), K), K / 16,
                  instr_desc(TR, H), false);
        mma_commit(&mmath);
      }
      if (!(ok = done())) break;
      const float *b = W.p + (l == 0 ? ob1 : (l == 1 ? ob2 : ob3));
#pragma unroll 1
      for (int c = 0; c < 32; c += 8)
      {
        float v[8];
        biased8(trow + kChain, b, c0 + c, v);
#pragma unroll
        for (int j = 0; j < 8; ++j)
        {
          float g, d;
          gelu_both(v[j], g, d);
          v[j] = g;
          dg[(l * 32 + c + j) * kThreads] = d;
        }
        put8(to, r, c0 + c, H, v);
      }
      publish_operands();
    }
    if (!ok) break;
    // output layer and loss
    if (tid == 0)
    {
      mma_issue(tmem + kChain, k_major(sA3, H), k_major(sW + kF4, H), H / 16, instr_desc(TR, OUTP), false);
      mma_commit(&mmath);
    }
    if (!(ok = done())) break;
    if (tid == 0)
    {
      // the forward weights have been read: the backward ones take their place
      expect_bytes(&mload, kBackward * 2);
      bulk_copy((void *) sW, W.bwd, kBackward * 2, &mload);
    }
    if (warp < 4)
    {
      float v[16], g[16], loss = 0.0f;
      tmem_ld16(trow + kChain, v);
      const float w4[4] = {wl.x, wl.y, wl.z, wl.w};
      float4 target = make_float4(0.f, 0.f, 0.f, 0.f);
      if (live) target = *reinterpret_cast<const float4 *>(t + (long) row * OUT);
      const float tt[4] = {target.x, target.y, target.z, target.w};
#pragma unroll
      for (int o = 0; o < 16; ++o) g[o] = 0.0f;
      if (live)
#pragma unroll
        for (int o = 0; o < OUT; ++o)
        {
          const float d = v[o] + __ldg(W.p + ob4 + o) - tt[o];
          loss += w4[o] * d * d;
          g[o] = 2.0f * w4[o] * d * scale;
        }
      put8(sZ4, r, 0, OUTP, g);
      put8(sZ4, r, 8, OUTP, g + 8);
      for (int off = 16; off > 0; off >>= 1) loss += __shfl_xor_sync(0xffffffffu, loss, off);
      if ((tid & 31) == 0) red[warp] = loss;
    }
    publish_operands();
    if (tid == 0) loss_partial[tile] = red[0] + red[1] + red[2] + red[3];
    if (!(ok = loaded())) break;
    // dA_l = dZ_{l+1} W_{l+1} for hidden layers 3, 2, 1, each followed by the
    // weight gradient that its input completes; MMAs run in order, so the wait
    // for the next chain product also covers that gradient, whose operands may
    // be overwritten from then on
    for (int l = 2; l >= 0 && ok; --l)
    {
      unsigned char *dz = l == 2 ? sZ4 : (l == 1 ? sD : sA3), *to = l == 2 ? sD : (l == 1 ? sA3 : sA2);
      if (tid == 0)
      {
        const int K = l == 2 ? OUTP : H;
        mma_issue(tmem + kChain, k_major(dz, K), k_major(sW + (l == 2 ? kB4 : (l == 1 ? kB3 : kB2)), K), K / 16,
                  instr_desc(TR, H), false);
        mma_commit(&mmath);
        if (l == 2)  // dW4^T = A3^T dZ4
          mma_issue(tmem + kG4, mn_major(sA3, H), mn_major(sZ4, OUTP), TR / 16, instr_desc(TR, OUTP, true), any);
        else  // dW3 = dZ3^T A2, dW2 = dZ2^T A1
          mma_issue(tmem + (l == 1 ? kG3 : kG2), mn_major(dz, H), mn_major(l == 1 ? sA2 : sA1, H), TR / 16,
                    instr_desc(TR, H, true), any);
      }
      float d[32], v[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) d[j] = dg[(l * 32 + j) * kThreads];
      if (l == 2)
      {
        if (tid < OUTP) db[3] = add_column(sZ4, tid, OUTP, db[3]);
      } else if (tid < H)
      {
        db[l + 1] = add_column(dz, tid, H, db[l + 1]);
      }
      if (!(ok = done())) break;
      tmem_ld32(trow + kChain + c0, v);
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = live ? v[j] * d[j] : 0.0f;
#pragma unroll
      for (int j = 0; j < 32; j += 8) put8(to, r, c0 + j, H, v + j);
      publish_operands();
    }
    if (!ok) break;
    if (tid == 0)  // dW1 = dZ1^T X
    {
      mma_issue(tmem + kG1, mn_major(sA2, H), mn_major(sX, INP), TR / 16, instr_desc(TR, INP, true), any);
      mma_commit(&mmath);
    }
    if (tid < H) db[0] = add_column(sA2, tid, H, db[0]);
    if (!(ok = done())) break;
    any = true;
  }
  const long cta = blockIdx.x;
  if (ok)
  {
    float v[32], g[16];
#pragma unroll
    for (int l = 1; l < 3; ++l)
    {
      tmem_ld32(trow + (l == 1 ? kG2 : kG3) + c0, v);
      float *o = out.w[l] + (cta * TR + r) * H + c0;
#pragma unroll
      for (int j = 0; j < 32; j += 4) *reinterpret_cast<float4 *>(o + j) = make_float4(v[j], v[j + 1], v[j + 2], v[j + 3]);
    }
    if (warp < 4)
    {
      tmem_ld16(trow + kG1, g);
      float *o = out.w[0] + (cta * TR + r) * INP;
#pragma unroll
      for (int j = 0; j < 16; j += 4) *reinterpret_cast<float4 *>(o + j) = make_float4(g[j], g[j + 1], g[j + 2], g[j + 3]);
      tmem_ld16(trow + kG4, g);
#pragma unroll
      for (int j = 0; j < OUT; ++j) out.w[3][(cta * TR + j) * H + r] = g[j];
    }
    if (tid < H)
#pragma unroll
      for (int l = 0; l < 4; ++l) out.b[l][cta * TR + tid] = db[l];
  } else
  {
    // report, and give what is in flight a second bounded wait before the
    // memory is released; the gradient of this batch is zero
    if (tid == 0) atomicOr(status, 1);
    wait_phase(&mload, lphase);
    wait_phase(&mmath, phase);
    for (int l = 0; l < 4; ++l)
    {
      const int kin = l == 0 ? INP : H;
      for (int i = tid; i < TR * kin; i += kThreads) out.w[l][cta * TR * kin + i] = 0.0f;
      if (tid < H) out.b[l][cta * TR + tid] = 0.0f;
    }
  }
  fence_before_sync();
  __syncthreads();
  if (warp == 0) tmem_dealloc(tmem, 512);
}

// ---------------------------------------------------------------- optimiser

struct Grads
{
  const float *pw[4], *pb[4];  // partials of the four layers
  int parts[4];                // partial count per layer
};

struct Adam
{
  float *p, *m1, *m2;
  bf16 *fwd, *bwd;
  float lr, c1, c2;  // learning rate, 1 - beta1^t, 1 - beta2^t
};

// Layer, row and column of flat parameter i (col -1: bias).
__device__ __forceinline__ void locate(int i, int &layer, int &m, int &c)
{
  if (i < ob1)
  {
    layer = 0;
    m = i / IN;
    c = i - m * IN;
  } else if (i < oW2)
  {
    layer = 0;
    m = i - ob1;
    c = -1;
  } else if (i < ob2)
  {
    layer = 1;
    m = (i - oW2) / H;
    c = (i - oW2) - m * H;
  } else if (i < oW3)
  {
    layer = 1;
    m = i - ob2;
    c = -1;
  } else if (i < ob3)
  {
    layer = 2;
    m = (i - oW3) / H;
    c = (i - oW3) - m * H;
  } else if (i < oW4)
  {
    layer = 2;
    m = i - ob3;
    c = -1;
  } else if (i < ob4)
  {
    layer = 3;
    m = (i - oW4) / H;
    c = (i - oW4) - m * H;
  } else
  {
    layer = 3;
    m = i - ob4;
    c = -1;
  }
}

// Sum the partial gradients (fixed order), optionally take an Adam step, and
// refresh the BF16 operand copies of every weight.
__global__ void mlp_update_kernel(Adam A, Grads G, int update, float *__restrict__ grad_out)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= NP) return;
  int layer, m, c;
  locate(i, layer, m, c);
  const int kin = layer == 0 ? INP : H;
  float g = 0.0f;
  for (int q = 0; q < G.parts[layer]; ++q)
    g += c >= 0 ? G.pw[layer][((long) q * TR + m) * kin + c] : G.pb[layer][(long) q * TR + m];
  if (grad_out) grad_out[i] = g;
  float p = A.p[i];
  if (update)
  {
    const float m1 = 0.9f * A.m1[i] + 0.1f * g;
    const float m2 = 0.999f * A.m2[i] + 0.001f * g * g;
    A.m1[i] = m1;
    A.m2[i] = m2;
    p -= A.lr * (m1 / A.c1) / (sqrtf(m2 / A.c2) + 1e-8f);
    A.p[i] = p;
  }
  if (c < 0) return;
  const bf16 h = __float2bfloat16_rn(p);
  switch (layer)
  {
    case 0: A.fwd[kF1 + canon(m, c, INP) / 2] = h; break;
    case 1:
      A.fwd[kF2 + canon(m, c, H) / 2] = h;
      A.bwd[kB2 + canon(c, m, H) / 2] = h;
      break;
    case 2:
      A.fwd[kF3 + canon(m, c, H) / 2] = h;
      A.bwd[kB3 + canon(c, m, H) / 2] = h;
      break;
    default:
      A.fwd[kF4 + canon(m, c, H) / 2] = h;
      A.bwd[kB4 + canon(c, m, OUTP) / 2] = h;
      break;
  }
}

// FP32 inputs [n][5] -> tiles of 128 rows of BF16 [16] in the canonical layout
// (zero columns, and zero rows up to the end of the last tile), optionally
// gathered through a permutation; targets [n][4] gathered alongside.
__global__ void mlp_pack_kernel(const float *__restrict__ x, const float *__restrict__ t, const int *__restrict__ perm,
                                long n, bf16 *__restrict__ xb, float *__restrict__ tout)
{
  const long i = (long) blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (n + TR - 1) / TR * TR) return;
  bf16 v[INP];
  const long s = i < n ? (perm ? perm[i] : i) : 0;
#pragma unroll
  for (int k = 0; k < INP; ++k) v[k] = __float2bfloat16_rn(k < IN && i < n ? x[s * IN + k] : 0.0f);
  unsigned char *tile = reinterpret_cast<unsigned char *>(xb) + (i / TR) * kTileX;
  const int r = (int) (i % TR);
  *reinterpret_cast<uint4 *>(tile + canon(r, 0, INP)) = *reinterpret_cast<const uint4 *>(v);
  *reinterpret_cast<uint4 *>(tile + canon(r, 8, INP)) = *reinterpret_cast<const uint4 *>(v + 8);
  if (t && tout && i < n)
    for (int o = 0; o < OUT; ++o) tout[i * OUT + o] = t[s * OUT + o];
}

}  // namespace mlp
}  // namespace spss

using namespace spss;
using namespace spss::mlp;

struct spss_mlp
{
  cudaStream_t stream = nullptr;
  DeviceArray<float> p, m1, m2, grad;
  DeviceArray<bf16> fwd, bwd;
  // resident training set and its shuffled copy
  DeviceArray<float> x_raw, t_raw, t_shuf;
  DeviceArray<bf16> x_shuf;
  DeviceArray<int> perm;
  long n_data = 0;
  // batch workspace
  DeviceArray<bf16> xb;
  DeviceArray<float> xin, tin, y, dgelu, pw[4], pb[4], loss_partial;
  DeviceArray<int> status;
  long step = 0;
  unsigned long long launches = 0;
};

namespace
{

long padded(long rows)
{
  return (rows + TR - 1) / TR * TR;
}

Weights weights(spss_mlp *m)
{
  return Weights{m->p.ptr, m->fwd.ptr, m->bwd.ptr};
}

int check_status(spss_mlp *m)
{
  int st = 0;
  SPSS_CUDA_TRY(cudaMemcpyAsync(&st, m->status.ptr, sizeof(int), cudaMemcpyDeviceToHost, m->stream));
  SPSS_CUDA_TRY(cudaStreamSynchronize(m->stream));
  return st ? SPSS_ERR_CUDA : SPSS_OK;
}

int forward_rows(spss_mlp *m, const bf16 *xb, long rows, float *y)
{
  const int blocks = (int) std::min<long>(padded(rows) / TR, 2 * 152);
  mlp_forward_kernel<<<blocks, kThreads, kFwdSmem, m->stream>>>(weights(m), xb, (int) rows, y, m->status.ptr);
  ++m->launches;
  return check_launch("mlp_forward_kernel");
}

// Gradient of a batch (input tiles xb, targets tin): partials, then the update
// kernel (with or without an Adam step); a loss partial per tile.
int train_rows(spss_mlp *m, const bf16 *xb, const float *tin, long rows, const float w[4], float lr, int update,
               float *grad_out, float *loss_partial)
{
  const int parts = (int) std::min<long>(padded(rows) / TR, kMaxPartials);
  const float4 wl = make_float4(w[0], w[1], w[2], w[3]);
  SPSS_TRY(m->dgelu.reserve((size_t) parts * 3 * 32 * kThreads));
  Partials out;
  Grads G;
  for (int l = 0; l < 4; ++l)
  {
    out.w[l] = m->pw[l].ptr;
    out.b[l] = m->pb[l].ptr;
    G.pw[l] = m->pw[l].ptr;
    G.pb[l] = m->pb[l].ptr;
    G.parts[l] = parts;
  }
  mlp_train_kernel<<<parts, kThreads, kTrainSmem, m->stream>>>(weights(m), xb, tin, wl, 1.0f / (float) rows, (int) rows,
                                                               m->dgelu.ptr, out, loss_partial, m->status.ptr);
  ++m->launches;
  SPSS_TRY(check_launch("mlp_train_kernel"));
  Adam A;
  A.p = m->p.ptr;
  A.m1 = m->m1.ptr;
  A.m2 = m->m2.ptr;
  A.fwd = m->fwd.ptr;
  A.bwd = m->bwd.ptr;
  A.lr = 0.0f;
  A.c1 = A.c2 = 1.0f;
  if (update)
  {
    m->step += 1;
    A.lr = lr;
    A.c1 = (float) (1.0 - std::pow(0.9, (double) m->step));
    A.c2 = (float) (1.0 - std::pow(0.999, (double) m->step));
  }
  mlp_update_kernel<<<(NP + 255) / 256, 256, 0, m->stream>>>(A, G, update, grad_out);
  return check_launch("mlp_update_kernel");
}

// BF16 operand copies from the master parameters.
int refresh_copies(spss_mlp *m)
{
  Grads G;
  for (int l = 0; l < 4; ++l)
  {
    G.pw[l] = nullptr;
    G.pb[l] = nullptr;
    G.parts[l] = 0;
  }
  Adam A;
  std::memset(&A, 0, sizeof(A));
  A.p = m->p.ptr;
  A.fwd = m->fwd.ptr;
  A.bwd = m->bwd.ptr;
  A.c1 = A.c2 = 1.0f;
  mlp_update_kernel<<<(NP + 255) / 256, 256, 0, m->stream>>>(A, G, 0, nullptr);
  return check_launch("mlp_update_kernel");
}

int upload_batch(spss_mlp *m, const float *x, const float *t, long n)
{
  SPSS_TRY(m->xb.reserve((size_t) padded(n) * INP));
  SPSS_TRY(m->xin.reserve((size_t) n * IN));
  SPSS_CUDA_TRY(cudaMemcpyAsync(m->xin.ptr, x, sizeof(float) * n * IN, cudaMemcpyHostToDevice, m->stream));
  if (t)
  {
    SPSS_TRY(m->tin.reserve((size_t) n * OUT));
    SPSS_CUDA_TRY(cudaMemcpyAsync(m->tin.ptr, t, sizeof(float) * n * OUT, cudaMemcpyHostToDevice, m->stream));
  }
  mlp_pack_kernel<<<(int) ((padded(n) + 255) / 256), 256, 0, m->stream>>>(m->xin.ptr, nullptr, nullptr, n, m->xb.ptr,
                                                                          nullptr);
  return check_launch("mlp_pack_kernel");
}

}  // namespace

extern "C" {

int spss_mlp_create(unsigned long long seed, spss_mlp **out)
{
  if (!out) return SPSS_ERR_INVALID_ARGUMENT;
  *out = nullptr;
  spss_mlp *m = new (std::nothrow) spss_mlp();
  if (!m) return SPSS_ERR_OUT_OF_MEMORY;
  int rc = SPSS_OK;
  auto fail = [&](int code) {
    spss_mlp_destroy(m);
    return code;
  };
  if (cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess)
  {
    cudaGetLastError();
    return fail(SPSS_ERR_CUDA);
  }
  if ((rc = m->p.reserve(NP)) || (rc = m->m1.reserve(NP)) || (rc = m->m2.reserve(NP)) || (rc = m->grad.reserve(NP)) ||
      (rc = m->fwd.reserve(kForward)) || (rc = m->bwd.reserve(kBackward)) || (rc = m->status.reserve(1)))
    return fail(rc);
  for (int l = 0; l < 4; ++l)
  {
    const int kin = l == 0 ? INP : H;
    if ((rc = m->pw[l].reserve((size_t) kMaxPartials * TR * kin)) || (rc = m->pb[l].reserve((size_t) kMaxPartials * TR)))
      return fail(rc);
  }
  if (cudaFuncSetAttribute(mlp_forward_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kFwdSmem) != cudaSuccess ||
      cudaFuncSetAttribute(mlp_train_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kTrainSmem) != cudaSuccess)
  {
    cudaGetLastError();
    return fail(SPSS_ERR_CUDA);
  }
  // padding of the operand copies stays zero
  cudaMemsetAsync(m->fwd.ptr, 0, sizeof(bf16) * kForward, m->stream);
  cudaMemsetAsync(m->bwd.ptr, 0, sizeof(bf16) * kBackward, m->stream);
  cudaMemsetAsync(m->m1.ptr, 0, sizeof(float) * NP, m->stream);
  cudaMemsetAsync(m->m2.ptr, 0, sizeof(float) * NP, m->stream);
  cudaMemsetAsync(m->status.ptr, 0, sizeof(int), m->stream);
  std::vector<float> h(NP, 0.0f);
  std::mt19937_64 gen(seed);
  auto fill = [&](int off, int count, int fan_in) {
    std::uniform_real_distribution<float> U(-1.0f / std::sqrt((float) fan_in), 1.0f / std::sqrt((float) fan_in));
    for (int i = 0; i < count; ++i) h[off + i] = U(gen);
  };
  fill(oW1, H * IN, IN);
  fill(oW2, H * H, H);
  fill(oW3, H * H, H);
  fill(oW4, OUT * H, H);
  *out = m;
  rc = spss_mlp_set_params(m, h.data(), NP);
  if (rc != SPSS_OK)
  {
    *out = nullptr;
    return fail(rc);
  }
  return SPSS_OK;
}

int spss_mlp_destroy(spss_mlp *m)
{
  if (!m) return SPSS_ERR_INVALID_ARGUMENT;
  if (m->stream) cudaStreamSynchronize(m->stream);
  m->p.release();
  m->m1.release();
  m->m2.release();
  m->grad.release();
  m->fwd.release();
  m->bwd.release();
  m->x_raw.release();
  m->t_raw.release();
  m->t_shuf.release();
  m->x_shuf.release();
  m->perm.release();
  m->xb.release();
  m->xin.release();
  m->tin.release();
  m->y.release();
  m->dgelu.release();
  m->loss_partial.release();
  m->status.release();
  for (int l = 0; l < 4; ++l)
  {
    m->pw[l].release();
    m->pb[l].release();
  }
  if (m->stream) cudaStreamDestroy(m->stream);
  cudaGetLastError();
  delete m;
  return SPSS_OK;
}

int spss_mlp_set_params(spss_mlp *m, const float *params, long len)
{
  if (!m || !params) return SPSS_ERR_INVALID_ARGUMENT;
  if (len != NP) return SPSS_ERR_SIZE;
  SPSS_CUDA_TRY(cudaMemcpyAsync(m->p.ptr, params, sizeof(float) * NP, cudaMemcpyHostToDevice, m->stream));
  SPSS_CUDA_TRY(cudaMemsetAsync(m->m1.ptr, 0, sizeof(float) * NP, m->stream));
  SPSS_CUDA_TRY(cudaMemsetAsync(m->m2.ptr, 0, sizeof(float) * NP, m->stream));
  m->step = 0;
  SPSS_TRY(refresh_copies(m));
  SPSS_CUDA_TRY(cudaStreamSynchronize(m->stream));
  return SPSS_OK;
}

int spss_mlp_get_params(spss_mlp *m, float *params, long len)
{
  if (!m || !params) return SPSS_ERR_INVALID_ARGUMENT;
  if (len != NP) return SPSS_ERR_SIZE;
  SPSS_CUDA_TRY(cudaMemcpyAsync(params, m->p.ptr, sizeof(float) * NP, cudaMemcpyDeviceToHost, m->stream));
  SPSS_CUDA_TRY(cudaStreamSynchronize(m->stream));
  return SPSS_OK;
}

int spss_mlp_forward(spss_mlp *m, const float *x, long n, float *y)
{
  if (!m || !x || !y || n <= 0) return SPSS_ERR_INVALID_ARGUMENT;
  if (n > 0x7fffff00L) return SPSS_ERR_SIZE;
  SPSS_TRY(m->y.reserve((size_t) n * OUT));
  SPSS_TRY(upload_batch(m, x, nullptr, n));
  SPSS_TRY(forward_rows(m, m->xb.ptr, n, m->y.ptr));
  SPSS_CUDA_TRY(cudaMemcpyAsync(y, m->y.ptr, sizeof(float) * n * OUT, cudaMemcpyDeviceToHost, m->stream));
  return check_status(m);
}

int spss_mlp_gradient(spss_mlp *m, const float *x, const float *t, const float *w, long n, float *grad, double *loss)
{
  if (!m || !x || !t || !grad || n <= 0) return SPSS_ERR_INVALID_ARGUMENT;
  if (n > 0x7fffff00L) return SPSS_ERR_SIZE;
  const float ones[4] = {1.0f, 1.0f, 1.0f, 1.0f};
  float wl[4];
  std::memcpy(wl, w ? w : ones, 4 * sizeof(float));
  SPSS_TRY(m->loss_partial.reserve((size_t) padded(n) / TR));
  SPSS_TRY(upload_batch(m, x, t, n));
  SPSS_TRY(train_rows(m, m->xb.ptr, m->tin.ptr, n, wl, 0.0f, 0, m->grad.ptr, m->loss_partial.ptr));
  SPSS_CUDA_TRY(cudaMemcpyAsync(grad, m->grad.ptr, sizeof(float) * NP, cudaMemcpyDeviceToHost, m->stream));
  const int blocks = (int) ((n + TR - 1) / TR);
  std::vector<float> lp(blocks);
  SPSS_CUDA_TRY(cudaMemcpyAsync(lp.data(), m->loss_partial.ptr, sizeof(float) * blocks, cudaMemcpyDeviceToHost,
                                m->stream));
  SPSS_TRY(check_status(m));
  if (loss)
  {
    double s = 0.0;
    for (float v : lp) s += v;
    *loss = s / (double) n;
  }
  return SPSS_OK;
}

int spss_mlp_set_data(spss_mlp *m, const float *x, const float *t, long n)
{
  if (!m || !x || !t || n <= 0) return SPSS_ERR_INVALID_ARGUMENT;
  if (n > 0x7fffff00L) return SPSS_ERR_SIZE;
  SPSS_TRY(m->x_raw.reserve((size_t) n * IN));
  SPSS_TRY(m->t_raw.reserve((size_t) n * OUT));
  SPSS_TRY(m->x_shuf.reserve((size_t) padded(n) * INP));
  SPSS_TRY(m->t_shuf.reserve((size_t) padded(n) * OUT));
  SPSS_TRY(m->perm.reserve((size_t) n));
  SPSS_CUDA_TRY(cudaMemcpyAsync(m->x_raw.ptr, x, sizeof(float) * n * IN, cudaMemcpyHostToDevice, m->stream));
  SPSS_CUDA_TRY(cudaMemcpyAsync(m->t_raw.ptr, t, sizeof(float) * n * OUT, cudaMemcpyHostToDevice, m->stream));
  SPSS_CUDA_TRY(cudaStreamSynchronize(m->stream));
  m->n_data = n;
  return SPSS_OK;
}

int spss_mlp_train(spss_mlp *m, int epochs, int batch, float lr, const float *w, unsigned long long shuffle_seed,
                   float *loss_per_epoch)
{
  if (!m || epochs < 0 || batch < TR || batch % TR || !(lr > 0.0f)) return SPSS_ERR_INVALID_ARGUMENT;
  if (m->n_data <= 0) return SPSS_ERR_INVALID_ARGUMENT;
  const long n = m->n_data;
  float wl[4] = {1.0f, 1.0f, 1.0f, 1.0f};
  if (w) std::memcpy(wl, w, 4 * sizeof(float));
  std::vector<int> perm((size_t) n);
  const long nb = (n + batch - 1) / batch, tiles = padded(n) / TR;
  SPSS_TRY(m->loss_partial.reserve((size_t) tiles));
  std::vector<float> lp((size_t) tiles);
  for (int e = 0; e < epochs; ++e)
  {
    for (long i = 0; i < n; ++i) perm[i] = (int) i;
    std::mt19937_64 gen(shuffle_seed + (unsigned long long) e);
    std::shuffle(perm.begin(), perm.end(), gen);
    SPSS_CUDA_TRY(cudaMemcpyAsync(m->perm.ptr, perm.data(), sizeof(int) * n, cudaMemcpyHostToDevice, m->stream));
    mlp_pack_kernel<<<(int) ((padded(n) + 255) / 256), 256, 0, m->stream>>>(m->x_raw.ptr, m->t_raw.ptr, m->perm.ptr, n,
                                                                            m->x_shuf.ptr, m->t_shuf.ptr);
    SPSS_TRY(check_launch("mlp_pack_kernel"));
    // the minibatches are runs of whole tiles of the shuffled set, read in
    // place; their losses are read once, after the epoch
    for (long b = 0; b < nb; ++b)
    {
      const long r0 = b * batch, rows = std::min<long>(batch, n - r0);
      SPSS_TRY(train_rows(m, m->x_shuf.ptr + r0 * INP, m->t_shuf.ptr + r0 * OUT, rows, wl, lr, 1, nullptr,
                          m->loss_partial.ptr + r0 / TR));
    }
    SPSS_CUDA_TRY(cudaMemcpyAsync(lp.data(), m->loss_partial.ptr, sizeof(float) * tiles, cudaMemcpyDeviceToHost,
                                  m->stream));
    SPSS_CUDA_TRY(cudaStreamSynchronize(m->stream));
    double epoch_loss = 0.0;
    for (long b = 0; b < nb; ++b)
    {
      const long r0 = b * batch, rows = std::min<long>(batch, n - r0);
      double s = 0.0;
      for (long q = r0 / TR; q < (r0 + rows + TR - 1) / TR; ++q) s += lp[q];
      epoch_loss += s / (double) rows;
    }
    if (loss_per_epoch) loss_per_epoch[e] = (float) (epoch_loss / (double) nb);
  }
  return check_status(m);
}

int spss_mlp_kernel_launches(spss_mlp *m, unsigned long long *count)
{
  if (!m || !count) return SPSS_ERR_INVALID_ARGUMENT;
  *count = m->launches;
  return SPSS_OK;
}

}  // extern "C"
