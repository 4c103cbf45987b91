// Internal declarations shared by the translation units of libspss_gpu.so.
#pragma once

#include <cuda_runtime.h>
#include <limits.h>
#include <stdint.h>

#include <cmath>
#include <vector>

#include "spss_gpu.h"

namespace spss
{

// ------------------------------------------------------------------ errors

struct Status
{
  int code = SPSS_OK;
};

#define SPSS_CUDA_TRY(expr)                                  \
  do                                                         \
  {                                                          \
    cudaError_t _e = (expr);                                 \
    if (_e != cudaSuccess)                                   \
    {                                                        \
      ::spss::record_cuda_error(_e, #expr, __FILE__, __LINE__); \
      return SPSS_ERR_CUDA;                                  \
    }                                                        \
  } while (0)

#define SPSS_TRY(expr)          \
  do                            \
  {                             \
    int _rc = (expr);           \
    if (_rc != SPSS_OK) return _rc; \
  } while (0)

void record_cuda_error(cudaError_t e, const char *what, const char *file, int line);
int check_launch(const char *what);

// Programmatic dependent launch along a chain of kernels: cell-list steps, the
// control launch and the download behind a step, FP64 steps on lists and the
// stages of an all-pairs RK4 step.  Every kernel that may be launched with the
// programmatic attribute begins with pdl_enter(): it waits until the kernel
// before it in the stream has completed and its writes are visible (without the
// attribute the instruction does nothing).  No kernel triggers its dependents
// early: with the trigger at the start of every CTA a chain of seventeen kernels
// at N = 4,194,304 ran about 2 % slower (0.6095 -> 0.6204 ms) and without it it
// gained (0.6059 ms; N = 65,536: 0.0475 -> 0.0437 ms).
__device__ __forceinline__ void pdl_enter()
{
  asm volatile("griddepcontrol.wait;" ::: "memory");
}

// A kernel launch, with the programmatic-serialization attribute when `chained`
// (the kernel must begin with pdl_enter()).
template<typename... Params, typename... Args>
inline cudaError_t launch_chained(bool chained, void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem,
                                  cudaStream_t stream, Args... args)
{
  cudaLaunchAttribute attr;
  attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr.val.programmaticStreamSerializationAllowed = 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = chained ? &attr : nullptr;
  cfg.numAttrs = chained ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}

// ------------------------------------------------------------------ host memory

// Maps the pages of a caller's result array by one system call in place of a
// fault on each as the copy reaches it (a new 3.1 MB array: 380 -> 231 us for
// the whole call; pages that are there already: within the noise).  Contents
// stay as they are, and where the system refuses, the faults come as before.
void prefault(void *p, size_t bytes);

// ------------------------------------------------------------------ device memory

template<class T>
struct DeviceArray
{
  T *ptr = nullptr;
  size_t count = 0;
  int reserve(size_t n)
  {
    if (n <= count && ptr) return SPSS_OK;
    release();
    if (n == 0) n = 1;
    cudaError_t e = cudaMalloc((void **) &ptr, n * sizeof(T));
    if (e != cudaSuccess)
    {
      ptr = nullptr;
      count = 0;
      cudaGetLastError();
      return SPSS_ERR_OUT_OF_MEMORY;
    }
    count = n;
    return SPSS_OK;
  }
  void release()
  {
    if (ptr) cudaFree(ptr);
    ptr = nullptr;
    count = 0;
  }
  size_t bytes() const { return count * sizeof(T); }
};

// ------------------------------------------------------------------ Philox

// Philox4x32-10 (Salmon, Moraes, Dror & Shaw, "Parallel random numbers: as
// easy as 1, 2, 3", SC'11).  Counter = (particle, step lo, step hi,
// replica << 8 | block), key = seed.
struct Philox
{
  __host__ __device__ static inline uint4 generate(uint4 c, uint2 k)
  {
#pragma unroll
    for (int r = 0; r < 10; ++r)
    {
      const uint64_t p0 = (uint64_t) 0xD2511F53u * c.x;
      const uint64_t p1 = (uint64_t) 0xCD9E8D57u * c.z;
      const uint32_t hi0 = (uint32_t) (p0 >> 32), lo0 = (uint32_t) p0;
      const uint32_t hi1 = (uint32_t) (p1 >> 32), lo1 = (uint32_t) p1;
      c = make_uint4(hi1 ^ c.y ^ k.x, lo1, hi0 ^ c.w ^ k.y, lo0);
      k.x += 0x9E3779B9u;
      k.y += 0xBB67AE85u;
    }
    return c;
  }
};

// The ten round keys of a seed (the Weyl sequence of Philox4x32-10).
__host__ __device__ inline void philox_round_keys(uint64_t seed, uint32_t kx[10], uint32_t ky[10])
{
  uint32_t a = (uint32_t) seed, b = (uint32_t) (seed >> 32);
  for (int r = 0; r < 10; ++r)
  {
    kx[r] = a;
    ky[r] = b;
    a += 0x9E3779B9u;
    b += 0xBB67AE85u;
  }
}

// Philox4x32-10 with the round keys given (equal to Philox::generate with
// the seed they come from), so a kernel takes them from its parameters
// instead of recomputing the key schedule per draw.
__device__ __forceinline__ uint4 philox_keyed(uint4 c, const uint32_t kx[10], const uint32_t ky[10])
{
#pragma unroll
  for (int r = 0; r < 10; ++r)
  {
    const uint64_t p0 = (uint64_t) 0xD2511F53u * c.x;
    const uint64_t p1 = (uint64_t) 0xCD9E8D57u * c.z;
    const uint32_t hi0 = (uint32_t) (p0 >> 32), lo0 = (uint32_t) p0;
    const uint32_t hi1 = (uint32_t) (p1 >> 32), lo1 = (uint32_t) p1;
    c = make_uint4(hi1 ^ c.y ^ kx[r], lo1, hi0 ^ c.w ^ ky[r], lo0);
  }
  return c;
}

struct NoiseKey
{
  uint64_t seed;
  uint32_t replica;
  uint64_t step;
};

__device__ __forceinline__ uint4 philox_block(const NoiseKey &nk, uint32_t particle, uint32_t block)
{
  uint4 c = make_uint4(particle, (uint32_t) nk.step, (uint32_t) (nk.step >> 32), (nk.replica << 8) | block);
  return Philox::generate(c, make_uint2((uint32_t) nk.seed, (uint32_t) (nk.seed >> 32)));
}

// ------------------------------------------------------------------ FP64 functions
//
// GB300 has one FP64 instruction for about 69 FP32 ones, and the FP64 kernels
// are bound by their count: the general-purpose functions spend about 40
// (sin), 30 (log) and 15 (sqrt) of them.  Table-driven evaluation (the method
// of P. T. P. Tang, "Table-driven implementation of the logarithm function in
// IEEE floating-point arithmetic", ACM TOMS 16, 1990, and of his sine of the
// same kind) needs 15 for a sine, 17 with the cosine, 13 for the logarithm and
// 8 for the square root.  Sine and cosine carry at most 1.5 units of 2^-53 (and 2
// ulp where one of them is small beside a multiple of pi / 2), the normals a few
// units of 2^-53 of their radius (tests/test_gpu_f64_functions.py,
// tests/test_gpu_f64_quarter_turns.py).

constexpr int kTrigTable = 256;      // cos and sin of 2 pi k / 256
constexpr int kLogFirst = 88, kLogLast = 184;  // j / 128 covers [sqrt(1/2), sqrt(2)] with room
constexpr int kTableEntries = kTrigTable + (kLogLast - kLogFirst + 1);  // then the first kTrigTable in units of 2^-59

// 1.5 * 2^52: adding it rounds to an integer, which then stands in the low word.
#define SPSS_ROUND_MAGIC 6755399441055744.0

// sin r and cos r - 1 for 0 <= |r| <= 2 pi / 256 by Taylor polynomials
// (remainders below 1e-20 and 4e-18).
__device__ __forceinline__ void sincos_rest(double r, double &sr, double &cm)
{
  const double p = r * r;
  sr = fma(r * p, fma(p, fma(p, -1.0 / 5040.0, 1.0 / 120.0), -1.0 / 6.0), r);
  cm = p * fma(p, fma(p, -1.0 / 720.0, 1.0 / 24.0), -0.5);
}

// sin and cos of 2 pi k / 256 + r by the angle sum.
__device__ __forceinline__ void sincos_at(const double2 *__restrict__ table, int k, double r, double &s, double &c)
{
  const double2 T = __ldg(table + (k & (kTrigTable - 1)));
  double sr, cm;
  sincos_rest(r, sr, cm);
  s = fma(T.x, sr, fma(T.y, cm, T.y));
  c = fma(-T.y, sr, fma(T.x, cm, T.x));
}

// |x| below 2^20 is reduced by hand (k < 2^26 keeps its products with the upper
// two parts of pi / 128, 26 bits each, exact); beyond it, for infinities and
// for NaN the CUDA functions.
__device__ __forceinline__ bool reducible(double x)
{
  return (__double2hiint(x) & 0x7fffffff) < 0x41300000;
}

// x = k pi / 128 + r, |r| <= pi / 256: the first two products and differences
// are exact, the third rounds once, and the parts' sum is pi / 128 to 2^-116, so
// r is off by half an ulp of itself and k 2^-116.
__device__ __forceinline__ void reduce_turn(double x, int &k, double &r)
{
  const double t = fma(x, 40.743665431525205957, SPSS_ROUND_MAGIC);  // 128 / pi
  k = __double2loint(t);
  const double kd = t - SPSS_ROUND_MAGIC;
  r = fma(kd, -0x1.921fb58p-6, x);
  r = fma(kd, 0x1.dde974p-33, r);
  r = fma(kd, -0x1.1a62633145c07p-60, r);
}

// Whether sine or cosine is a remainder so small (below 2^-30, next to a multiple
// of pi / 2 other than 0) that the error of the reduction shows in it.
__device__ __forceinline__ bool near_quarter(int k, double r)
{
  return (k & 63) == 0 && k != 0 && (__double2hiint(r) & 0x7fffffff) < 0x3e100000;
}

// Within 1.5 units of 2^-53 of sine and cosine, and within 2 ulp of the one
// that is small next to a multiple of pi / 2.
__device__ __forceinline__ void fast_sincos(const double2 *__restrict__ table, double x, double &s, double &c)
{
  int k = 0;
  double r = 0.0;
  const bool mine = reducible(x);
  if (mine) reduce_turn(x, k, r);
  if (!mine || near_quarter(k, r))
  {
    sincos(x, &s, &c);
    return;
  }
  sincos_at(table, k, r, s, c);
}

// log((a + 0.5) 2^-32) for a 32-bit a: the mantissa m in [sqrt(1/2), sqrt(2)),
// c = j / 128 the nearest table point (c = 1 around 1, where the result is
// small), log(m / c) by its series to r^7 (|r| <= 1 / 180).
__device__ __forceinline__ double log_uniform(const double2 *__restrict__ table, uint32_t a)
{
  const double u = __hiloint2double(0x43300000, (int) a) - 4503599627370495.5;  // a + 0.5, exact
  int hi = __double2hiint(u);
  const int shift = (hi - 0x3fe6a09f) >> 20;  // 0x3fe6a09f: sqrt(1/2), rounded up
  hi -= shift << 20;
  const double m = __hiloint2double(hi, __double2loint(u));
  const float mf = __uint_as_float((((uint32_t) hi - 0x38000000u) << 3));  // the leading 21 bits
  const int j = __float2int_rn(mf * 128.0f);
  const double2 T = __ldg(table + kTrigTable + (j - kLogFirst));  // 128 / j (rounded), minus the log of that
  const double r = fma(m, T.x, -1.0);
  double q = fma(r, 1.0 / 7.0, -1.0 / 6.0);
  q = fma(r, q, 1.0 / 5.0);
  q = fma(r, q, -1.0 / 4.0);
  q = fma(r, q, 1.0 / 3.0);
  q = fma(r, q, -0.5);
  const double e = __hiloint2double(0x43300000, (shift - 32) ^ 0x80000000) - 4503601774854144.0;  // (double) (shift - 32)
  return fma(e, 0.693147180559945309417, T.y) + fma(r * r, q, r);
}

// Square root of a positive double in the range of float normals: the FP32
// reciprocal square root and one third-order step.
__device__ __forceinline__ double sqrt_positive(double v)
{
  const double y = (double) rsqrtf((float) v);
  const double g = v * y;
  const double e = fma(-g, y, 1.0);
  return fma(g * e, fma(e, 0.375, 0.5), g);
}

// cos and sin of x, and in fixed point, units of 2^-59: what is added to the
// table's point is below 2^-6, so the fixed-point pair is right to some 2^-60
// (2^-58 at most) where the doubles are to 2^-53.  A phase that is not reduced by hand
// (beyond 2^20, infinite, NaN) has none: the lowest value.
__device__ __forceinline__ void directions(const double2 *__restrict__ table, double x, double2 &cs, longlong2 &turn)
{
  if (!reducible(x))
  {
    sincos(x, &cs.y, &cs.x);
    turn = make_longlong2(LLONG_MIN, LLONG_MIN);
    return;
  }
  int k;
  double r, sr, cm;
  reduce_turn(x, k, r);
  const double2 T = __ldg(table + (k & (kTrigTable - 1)));
  const longlong2 F = __ldg(reinterpret_cast<const longlong2 *>(table + kTableEntries) + (k & (kTrigTable - 1)));
  sincos_rest(r, sr, cm);
  const double dc = fma(T.x, cm, -(T.y * sr)), ds = fma(T.x, sr, T.y * cm);
  cs = make_double2(T.x + dc, T.y + ds);
  if (near_quarter(k, r)) sincos(x, &cs.y, &cs.x);
  turn = make_longlong2(F.x + __double2ll_rn(dc * 576460752303423488.0), F.y + __double2ll_rn(ds * 576460752303423488.0));
}

// The tables of the functions above: cos, sin of 2 pi k / 256, then 128 / j and
// -log(128 / j as rounded), then the first in units of 2^-59.
int make_f64_tables(DeviceArray<double2> &table, cudaStream_t stream);

// Box-Muller on two 32-bit uniforms in (0, 1): FP64 variant for the
// reference-arithmetic path, FP32 variant for the fast path.
__device__ __forceinline__ void box_muller_f64(const double2 *__restrict__ table, uint32_t a, uint32_t b, double &z0,
                                               double &z1)
{
  const double r = sqrt_positive(-2.0 * log_uniform(table, a));
  // angle 2 pi (b + 0.5) 2^-32: the 256th of a turn and the rest
  const double rest = __hiloint2double(0x43300000, (int) (b & 0xffffffu)) - 4503599627370495.5;  // + 0.5, exact
  double s, c;
  sincos_at(table, (int) (b >> 24), rest * 1.46291807926715968e-9, s, c);  // 2 pi / 2^32
  z0 = r * c;
  z1 = r * s;
}

// The angle is uniform on (-pi, pi) and goes through the hardware sine and
// cosine (absolute error below 2^-21 there); the radius uses the hardware
// logarithm (absolute error below 2^-21.4 on [0.5, 2], where u1 lies unless the
// radius exceeds 1.18, and 3 ulp beyond): the radius r is off by at most about
// 2^-21.4 / r, more than 1 % relative only for r < 6e-3, which a fraction 2e-5
// of the draws reach, far beneath any statistical resolution of the runs.
// spss_noise evaluates the same function, so replayed noise is bit-identical.
// Rounding is spelled out (__fmul_rn, __fadd_rn) so every inlined copy of this
// function produces the same bits.
__device__ __forceinline__ void box_muller_f32(uint32_t a, uint32_t b, float &z0, float &z1)
{
  const float u1 = __fmul_rn(__fadd_rn((float) (a >> 8), 0.5f), 5.9604644775390625e-8f);
  const float theta = __fmul_rn(__fadd_rn(__fmul_rn((float) (b >> 8), 5.9604644775390625e-8f), -0.49999997f),
                                6.2831853f);
  const float r = sqrtf(__fmul_rn(-2.0f, __logf(u1)));
  float s, c;
  __sincosf(theta, &s, &c);
  z0 = __fmul_rn(r, c);
  z1 = __fmul_rn(r, s);
}

// Six normals from one Philox block (128 bits), for the steps that need six
// (second-order SRK): three Box-Muller pairs with 24-bit radius uniforms (the
// top 24 bits of words 0..2) and 16-bit angle uniforms (the two halves of
// word 3, and the low bytes of words 0 and 1).  A 16-bit angle is resolved to
// 1e-4 rad; the radius keeps the tails of the 24-bit draws above.
__device__ __forceinline__ void box_muller6_f32(const uint4 &u, float z[6])
{
  const uint32_t a[3] = {u.x >> 8, u.y >> 8, u.z >> 8};
  const uint32_t b[3] = {u.w & 0xffffu, u.w >> 16, (u.x & 0xffu) | ((u.y & 0xffu) << 8)};
#pragma unroll
  for (int k = 0; k < 3; ++k)
  {
    const float u1 = __fmul_rn(__fadd_rn((float) a[k], 0.5f), 5.9604644775390625e-8f);
    const float theta = __fmul_rn(__fadd_rn(__fmul_rn(__fadd_rn((float) b[k], 0.5f), 1.52587890625e-5f), -0.5f),
                                  6.2831853f);
    const float r = sqrtf(__fmul_rn(-2.0f, __logf(u1)));
    float s, c;
    __sincosf(theta, &s, &c);
    z[2 * k] = __fmul_rn(r, c);
    z[2 * k + 1] = __fmul_rn(r, s);
  }
}

__device__ __forceinline__ void normals4_f32(const NoiseKey &nk, uint32_t particle, uint32_t block, float z[4])
{
  const uint4 u = philox_block(nk, particle, block);
  box_muller_f32(u.x, u.y, z[0], z[1]);
  box_muller_f32(u.z, u.w, z[2], z[3]);
}

// The first `pairs` Box-Muller pairs of a block of four uniforms.
template<int PAIRS>
__device__ __forceinline__ void normals_f64(const double2 *__restrict__ table, const NoiseKey &nk, uint32_t particle,
                                            uint32_t block, double *z)
{
  const uint4 u = philox_block(nk, particle, block);
  box_muller_f64(table, u.x, u.y, z[0], z[1]);
  if (PAIRS > 1) box_muller_f64(table, u.z, u.w, z[2], z[3]);
}

// ------------------------------------------------------------------ reductions

// Sums of four values over a warp: lane l gets that of value l >> 3.  The first
// two exchanges halve what a lane carries, so six additions an FP64 warp sum
// costs, not 20 (16 cycles each: the chip has two FP64 lanes an SM).
__device__ __forceinline__ double warp_sum4(const double a[4])
{
  const int lane = threadIdx.x & 31;
  const bool up = lane & 16, odd = lane & 8;
  const double k0 = (up ? a[2] : a[0]) + __shfl_xor_sync(0xffffffffu, up ? a[0] : a[2], 16);
  const double k1 = (up ? a[3] : a[1]) + __shfl_xor_sync(0xffffffffu, up ? a[1] : a[3], 16);
  double k = (odd ? k1 : k0) + __shfl_xor_sync(0xffffffffu, odd ? k0 : k1, 8);
#pragma unroll
  for (int off = 4; off > 0; off >>= 1) k += __shfl_xor_sync(0xffffffffu, k, off);
  return k;
}

// Sums of four values over a block of 256 threads, `mine` as warp_sum4 returns
// it: lane l of warp 0 gets that of value l >> 3.
__device__ __forceinline__ double block_sum4(double mine)
{
  __shared__ double sh[4][8];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  if ((lane & 7) == 0) sh[lane >> 3][wid] = mine;
  __syncthreads();
  double k = 0.0;
  if (wid == 0)
  {
    k = sh[lane >> 3][lane & 7];
#pragma unroll
    for (int off = 4; off > 0; off >>= 1) k += __shfl_xor_sync(0xffffffffu, k, off);
  }
  __syncthreads();
  return k;
}

// Sums of `nparts` partials of four values each, in a fixed order, by one
// block of 256 threads: lane l of warp 0 gets that of value l >> 3.
__device__ __forceinline__ double block_sum_partials4(const double *__restrict__ partials, int nparts)
{
  double t[4] = {0.0, 0.0, 0.0, 0.0};
  for (int b = threadIdx.x; b < nparts; b += 256)
  {
    // __ldcg: the partials may have been written by other blocks of the same launch
    const double2 lo = __ldcg(reinterpret_cast<const double2 *>(partials + 4 * (long) b));
    const double2 hi = __ldcg(reinterpret_cast<const double2 *>(partials + 4 * (long) b + 2));
    t[0] += lo.x;
    t[1] += lo.y;
    t[2] += hi.x;
    t[3] += hi.y;
  }
  return block_sum4(warp_sum4(t));
}

// The same with all four sums in thread 0.
__device__ __forceinline__ void block_sum_partials(const double *__restrict__ partials, int nparts, double t[4])
{
  const double k = block_sum_partials4(partials, nparts);
  if (threadIdx.x < 32)
#pragma unroll
    for (int c = 0; c < 4; ++c) t[c] = __shfl_sync(0xffffffffu, k, 8 * c);
}

// {|R|, arg R, |R_v|, arg R_v} from the sums of cos phi, sin phi, v_x/|v|, v_y/|v|.
__host__ __device__ __forceinline__ void order_from_sums(const double t[4], double n, int model, double *out)
{
  const double re = t[0] / n, im = t[1] / n;
  out[0] = sqrt(re * re + im * im);
  out[1] = atan2(im, re);
  if (model == 2)
  {
    const double vre = t[2] / n, vim = t[3] / n;
    out[2] = sqrt(vre * vre + vim * vim);
    out[3] = atan2(vim, vre);
  } else
  {
    out[2] = out[0];
    out[3] = out[1];
  }
}

// The reference's observer wraps of a frame value, computed in double on the
// float value and rounded back (BinaryObserverFirstOrder.cpp:112-117,
// PeriodicBoundaryConditions.cpp:137-145): `x -= floor(x * 1) * 1` and
// `phi -= floor(phi / 2 pi) * 2 pi`.
__device__ __forceinline__ float frame_wrap_position(float v)
{
  const double d = (double) v;
  return __double2float_rn(__dsub_rn(d, floor(d)));
}

__device__ __forceinline__ float frame_wrap_phase(float v)
{
  const double two_pi = 6.283185307179586;
  const double d = (double) v;
  return __double2float_rn(__dsub_rn(d, __dmul_rn(floor(__ddiv_rn(d, two_pi)), two_pi)));
}

inline int normals_per_particle(int model, int stepper)
{
  if (stepper == SPSS_STEPPER_RK4) return 0;
  if (stepper == SPSS_STEPPER_STOCHASTIC_EULER) return model == 1 ? 1 : 3;
  return model == 1 ? 2 : 6;
}

// Control words of a GB300-path context, on the device (fast_path.cu).
struct FastControl
{
  unsigned long long step;  // Philox step counter of the next stochastic step
  double acc;               // accumulated displacement of system 0 (FP64)
  int parity;               // current rec/aux buffer
  int order_parity;         // current vel/pid buffer (they change places only when the slots are re-sorted)
  int rebuild;              // lists (and slot order) rebuilt before the next evaluation
  int cells_fresh;          // the last step left what the next one begins with: cell ids and counts of the
                            // current slots (cell lists), the field of the current state (global field)
  int overflow;             // largest Verlet count seen beyond capacity (0: none)
  int rebuilds;             // number of rebuilds performed
  int error;                // bit 0: displacement too large for the fixed-point increment; bit 3: the
                            // device launch of the rebuild graph was refused
  int uses_verlet;
  unsigned ticket;          // blocks of the running reduction that are done (its last block puts it back to 0)
  int triggered;            // the last step's displacement trigger fired (its rebuild may already be done)
  long long sample_every;   // order-parameter samples after steps that are multiples of this (0: none)
  long long sample_from;    // ... and not before this step
};

// Exclusive prefix sum of `n` int32 counts into offsets[0..n] (offsets[n] =
// total): block sums, then every block adds the sums before its own and scans
// its tile (two launches, one for a single tile).  `zero` clears the counts on
// the way; `ctrl` (not null): the launch also begins a cell-list step
// (begin_cell_step).
struct Scanner
{
  std::vector<DeviceArray<int>> levels;
  int prepare(int n);  // buffers for n counts
  int run(int *in, int *out, int n, cudaStream_t stream, unsigned long long &launches, bool chained = false,
          bool zero = false, FastControl *ctrl = nullptr);
  int run_level(int *in, int *out, int n, size_t level, cudaStream_t stream, unsigned long long &launches, bool chained,
                bool zero, FastControl *ctrl);
  void release()
  {
    for (auto &l : levels) l.release();
    levels.clear();
  }
};

// Stable cell binning: cell id per element -> CSR offsets and members that list
// each cell's elements in ascending element order (the push_back order of the
// reference's linked_list_, ParticleSystemFirstOrder.cpp:285-288).
struct BinRows
{
  const float2 *pos = nullptr;
  const longlong2 *turns = nullptr;
  float2 *pos_out = nullptr;
  longlong2 *turns_out = nullptr;
};

struct Binner
{
  DeviceArray<int> count, offsets, slot, members;
  Scanner scanner;
  int ncell = 0;
  // buffers for n elements and ncell cells; newly allocated counts are zero
  int prepare(int n, int ncell, cudaStream_t stream);
  // From the counts and each element's arrival number in its cell (slot, both
  // left by the caller's kernel, counts zero before it): offsets, and members
  // in arrival order; the counts are zero again.
  int place(const int *cell_of, int n, cudaStream_t stream, unsigned long long &launches, bool chained = false,
            FastControl *ctrl = nullptr);
  // the same with members in ascending order, and (outputs not null) what a scan
  // of the cells reads of each member, in members' order
  int finish(const int *cell_of, int n, cudaStream_t stream, unsigned long long &launches, bool chained,
             const BinRows &rows);
  // all of it
  int run(const int *cell_of, int n, int ncell, cudaStream_t stream, unsigned long long &launches);
  void release()
  {
    count.release();
    offsets.release();
    slot.release();
    members.release();
    scanner.release();
  }
};

// ------------------------------------------------------------------ contexts

struct F64Path;
struct FastPath;

}  // namespace spss

struct spss_ctx
{
  spss_params p{};  // a batch: the first system's parameters, n = all particles
  std::vector<spss_params> systems;  // a batch: every system (empty for one system)
  int s = 4;
  cudaStream_t stream = nullptr;      // where work is issued
  cudaStream_t own_stream = nullptr;  // created with the context; graph capture runs here
  // CUDA-event timing of the pair-and-update kernel (spss_set_timing)
  int timing = 0;
  double timing_ms = 0.0;
  unsigned long long timing_count = 0;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr;
  unsigned long long launches = 0;
  unsigned long long step_counter = 0;
  int higher_order = 0;
  // Verlet bookkeeping (CalculateMaxDisplacement), kept on the host in FP64.
  double accumulated_displacement = 0.0;
  int should_update_lists = 1;
  int uses_verlet_list = 0;
  unsigned long long list_builds = 0;  // Verlet / cell list builds so far (FP64 path; the fast path counts on the device)
  double r_min = 0.0, r_max = 0.0;
  int nc = 1, nc_verlet = 1;
  // host registration of the caller's array for spss_step_host
  void *registered_host = nullptr;
  size_t registered_bytes = 0;
  double *registered_device = nullptr;  // device view of the registered array (mapped pinned memory)
  bool registered_here = false;         // registered by this context (else the caller's page-locked memory)
  spss::F64Path *f64 = nullptr;
  spss::FastPath *fast = nullptr;
  // AveragingObserver accumulator (FP64, AoS) and its count
  spss::DeviceArray<double> average;
  int average_count = 0;
  // AoS staging buffers for host-array entry points
  spss::DeviceArray<double> scratch_a, scratch_b, scratch_c;
  // trajectory frames (spss_frame_async) on their way to memory the GPU cannot address
  spss::DeviceArray<float> frame;
};

namespace spss
{
// F64 (reference arithmetic) path, f64_path.cu
int f64_create(spss_ctx *ctx);
void f64_destroy(spss_ctx *ctx);
int f64_set_state(spss_ctx *ctx, const double *d_aos);
int f64_get_state(spss_ctx *ctx, double *d_aos);
int f64_evaluate(spss_ctx *ctx, int variant, const double *d_state, const double *d_kprev, double *d_knext,
                 double k_coef, double dt);
int f64_step(spss_ctx *ctx, int stepper, double t, double dt);
int f64_steps(spss_ctx *ctx, int stepper, double t0, double dt, int nsteps);
int f64_noise(spss_ctx *ctx, int stepper, unsigned long long step, double *d_out);
int f64_max_displacement(spss_ctx *ctx, const double *d_td, double *max2_out);
int f64_complementary_force(spss_ctx *ctx, double *d_out);
int f64_set_natural_frequencies(spss_ctx *ctx, const double *d_freqs);
int f64_lists(spss_ctx *ctx, int **pll, int **cell_off, int **cell_mem, int *ncell, int **vl_off, int **vl_ent,
              long *vl_total);
int f64_apply_pbc(spss_ctx *ctx);
int f64_state_ptr(spss_ctx *ctx, const double **d_aos);

// Fast (GB300) path, fast_path.cu
int fast_create(spss_ctx *ctx);
void fast_destroy(spss_ctx *ctx);
int fast_rebuild_count(spss_ctx *ctx, unsigned long long *count);
int fast_set_state(spss_ctx *ctx, const double *d_aos);
int fast_get_state(spss_ctx *ctx, double *d_aos);
int fast_evaluate(spss_ctx *ctx, int variant, const double *d_state, const double *d_kprev, double *d_knext,
                  double k_coef, double dt);
int fast_step_state(spss_ctx *ctx, int stepper, double dt, double *io);
int fast_step(spss_ctx *ctx, int stepper, double t, double dt);
int fast_steps(spss_ctx *ctx, int stepper, double t0, double dt, int nsteps);
int fast_noise(spss_ctx *ctx, int stepper, unsigned long long step, double *d_out);
int fast_set_natural_frequencies(spss_ctx *ctx, const double *d_freqs);
int fast_complementary_force(spss_ctx *ctx, double *d_out);
int fast_apply_pbc(spss_ctx *ctx);

int fast_set_tiling(spss_ctx *ctx, int tile_cells, int persistent);
int fast_get_tiling(spss_ctx *ctx, int *tile_cells, int *persistent);
int fast_set_device_rebuild(spss_ctx *ctx, int enabled);
int fast_autotune(spss_ctx *ctx, int stepper, double dt, int steps, double *best_ms);
int fast_system_order_parameters(spss_ctx *ctx, double *h_out);
int fast_batch_run(spss_ctx *ctx, int stepper, double dt, long nsteps, long sample_every, long sample_from);
int fast_batch_stats(spss_ctx *ctx, double *h_out);
int fast_batch_reset_stats(spss_ctx *ctx);
int fast_order_parameters(spss_ctx *ctx, double *out4);
int fast_frame(spss_ctx *ctx, int wrap, float *d_out);
int fast_num_systems(const spss_ctx *ctx);
int fast_system_first(const spss_ctx *ctx, int r);

// Shared helpers, spss_gpu.cu
int order_parameters_aos(spss_ctx *ctx, const double *d_aos, double out[4]);
int host_calculate_max_displacement(spss_ctx *ctx, double max2);
int variant_for(const spss_ctx *ctx, int variant);
int variant_for_params(const spss_params &p, int variant);
// List geometry of a system: r_min = rho, r_max (Verlet cutoff), the cell grid
// of the linked list and of the Verlet rebuild.
void derive_lists(const spss_params &p, double &r_min, double &r_max, int &nc, int &nc_verlet);
}  // namespace spss
