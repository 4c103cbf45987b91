// GB300 fast path: fixed-point positions, FP32 pair and stage arithmetic,
// fused pair sums + stochastic stepper update + Philox noise.
//
// Representation (slot order; slots are re-sorted by cell at every rebuild):
//   rec[2][n]  uint4 {x_hi, y_hi, cos phi, sin phi}: the record a neighbour
//              gathers; double-buffered, a step reads rec[parity] (neighbours
//              see the previous state) and writes rec[parity ^ 1]
//   aux[2][n]  uint4 {x_lo, y_lo, phase, omega}, double-buffered with rec
//   vel[n]     float2 {v_x, v_y} (second-order model), updated in place
//   pid[n]     original particle index (noise counter, output order); inv[n]
//              its inverse
//   img[n], turns[n]  box crossings and 2*pi turns of the phase, indexed by
//              original index (they change rarely, so the slot re-sort of a
//              rebuild does not move them)
// x = img + (x_hi * 2^32 + x_lo) * 2^-64 (unit box), phase = 2*pi*(turns + phase * 2^-32).
//
// The owner of a particle evaluates cos and sin of its phase once per step and
// stores them in its record, so a pair costs no transcendental:
// sum_j sin(phi_j - phi_i) = cos phi_i sum_j sin phi_j - sin phi_i sum_j cos phi_j.
//
// FP64 appears only where the result must not depend on FP32 rounding: the
// exact cutoff decision inside a guard band around r = rho (a few pairs per
// step), the accumulated Verlet displacement and the upload/download
// conversions.  GB300 runs FP64 at about 1/70 of its FP32 rate.
//
// Reference semantics mirrored: ParticleSystemFirstOrder.cpp / ParticleSystemFirstOrderPtr.cpp
// (pair sums, isolated particles keep zero torque derivative in SE/SRK),
// ParticleSystemSecondOrder.cpp, StochasticEulerStepper.hpp:33-51,
// StochasticEulerStepperPtr.hpp:40-73, StochasticRungeKuttaStepperPtr.hpp:40-76,
// CalculateMaxDisplacement ParticleSystemFirstOrder.cpp:670-696.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <map>
#include <tuple>
#include <utility>

#include "spss_internal.cuh"

namespace spss
{

constexpr int kTB = 256;

// Per-system Verlet trigger state (CalculateMaxDisplacement of each system).
struct SysControl
{
  double acc;              // accumulated displacement (FP64)
  unsigned int max2_bits;  // max |dr|^2 of the step, FP32 bits (non-negative floats order as ints)
  int rebuild;             // this system's lists are rebuilt before the next step (per-system rebuilds)
};

// FastControl::rebuild: no rebuild, every system, or the systems whose own
// trigger fired (SysControl::rebuild; batches of Verlet-list systems).
enum
{
  REBUILD_NONE = 0,
  REBUILD_ALL = 1,
  REBUILD_FLAGGED = 2
};

// One independent system of a context (a context holds one or a batch of
// them; each is the reference's particle system on its own unit box).  Its
// particles are the slots [first, first + n) in every slot order, its cells
// the global cells [cell0, cell0 + nc^2).
struct SysParams
{
  int n, first, nc, cell0;
  int index, replica;
  float v0, xi, xi_r, xi_phi, sigma, ca, sa, rho2_f;
  float band_f, rmax2_f, b_r, b_phi;
  double rho2_d, half_skin;
};

enum Kind
{
  KIND_ALL_PAIRS = 0,
  KIND_GLOBAL = 3,  // global polar order field (first order): no lists, slot = original index
  KIND_CELLS = 1,
  KIND_VERLET = 2
};

// Launch parameters: context-wide fields, plus the fields of one system
// (nc .. replica), which kernels that work on several systems overwrite from
// the system table (with_system).
struct FastParams
{
  int n, nc, cap, model;      // n: slots of the whole context
  int always_rebuild, nsys;
  int first, sub_n;
  int cell0, selective;       // selective: per-system rebuilds (batches of Verlet-list systems)
  float v0, xi, xi_r, xi_phi, sigma, ca, sa;
  float rho2_f, band_f;
  double rho2_d;
  float dt, sqdt, half_dt2, half_dt15, inv_sqrt3, b_r, b_phi;
  uint64_t seed;
  uint32_t replica;
  uint32_t kx[10], ky[10];  // Philox round keys of `seed`, the same for every particle
};

struct FastBuffers
{
  uint4 *rec0, *rec1;
  uint4 *aux0, *aux1;
  float2 *vel, *vel_tmp;  // the current buffer and the other one (buffers_now)
  unsigned *pid, *pid_tmp, *inv;
  int2 *img;   // box crossings, by original index
  int *turns;  // 2 pi turns of the phase, by original index
  int *cell_of, *cell_sorted;
  const int *cell_off;
  int *cell_off_w;  // the same offsets, for the kernel that writes a system's
  const int *order;            // slots in cell order, arrival order inside a cell
  int *cell_count, *cell_slot; // counts of the next binning, and each slot's arrival number
  short *vl;
  int *vl_cnt;
  float *nu;             // natural frequencies (global field), slot = original index
  float *field;          // Z = <e^{i phi}>, W = <omega e^{i phi}> and derived values (global field)
  double *field_partial; // block partials of the field sums
  const SysParams *sys;  // system table
  const int *sys_of;     // system of each slot (equivalently of each original index)
  SysControl *sysctl;
  FastControl *ctrl;
};

// The kernel's view of the buffers with vel and pid the current ones.
__device__ __forceinline__ void buffers_now(FastBuffers &B, int order_parity)
{
  if (!order_parity) return;
  float2 *v = B.vel;
  B.vel = B.vel_tmp;
  B.vel_tmp = v;
  unsigned *p = B.pid;
  B.pid = B.pid_tmp;
  B.pid_tmp = p;
}

// How a step graph does the list rebuild: under a conditional node at the
// start of the step (GRAPH_CONDITIONAL), tail-launched as a device graph by the
// control kernel when the trigger fires (GRAPH_DEVICE), unconditionally at the
// start of every step (GRAPH_ALWAYS: cell lists, and batches of small systems,
// whose rebuild kernels leave at once when nothing is due), or not at all (GRAPH_NONE:
// kinds without lists or trigger).  Rebuilds requested from the host run
// before the first graph step in the last three forms.
enum
{
  GRAPH_CONDITIONAL = 0,
  GRAPH_DEVICE = 1,
  GRAPH_ALWAYS = 2,
  GRAPH_NONE = 3
};

// Device copy of the stepping state, for restoring it after trial steps.
struct Snapshot
{
  DeviceArray<uint4> rec[2], aux[2];
  DeviceArray<float2> vel[2];
  DeviceArray<unsigned> pid[2], inv;
  DeviceArray<int2> img;
  DeviceArray<int> turns;
  DeviceArray<SysControl> sysctl;
  DeviceArray<FastControl> ctrl;
  void release()
  {
    for (int b = 0; b < 2; ++b)
    {
      rec[b].release();
      aux[b].release();
      vel[b].release();
      pid[b].release();
    }
    inv.release();
    img.release();
    turns.release();
    sysctl.release();
    ctrl.release();
  }
};

// FP64 sums of one chunk of a system: cos phi, sin phi, v_x/|v|, v_y/|v|.
struct __align__(16) OrderSums
{
  double c, s, vx, vy;
};

struct GraphEntry
{
  cudaGraphExec_t exec = nullptr;
  cudaGraph_t graph = nullptr;
  // the rebuild as a device-launchable graph, tail-launched by the step's
  // control kernel when the trigger fires (null: the step graph holds the
  // rebuild under a conditional node instead)
  cudaGraphExec_t rebuild_exec = nullptr;
  cudaGraph_t rebuild_graph = nullptr;
  int per_step = 0;     // kernels of the unconditional part
  int per_rebuild = 0;  // kernels of the rebuild
  int form = 0;         // GRAPH_* below
  void release()
  {
    if (exec) cudaGraphExecDestroy(exec);
    if (graph) cudaGraphDestroy(graph);
    if (rebuild_exec) cudaGraphExecDestroy(rebuild_exec);
    if (rebuild_graph) cudaGraphDestroy(rebuild_graph);
    *this = GraphEntry();
  }
};

struct FastPath
{
  DeviceArray<uint4> rec[2], aux[2];
  DeviceArray<float2> vel, vel_tmp;
  DeviceArray<unsigned> pid, pid_tmp, inv;
  DeviceArray<int2> img;
  DeviceArray<int> turns, cell_of, cell_sorted, vl_cnt;
  DeviceArray<short> vl;
  DeviceArray<SysParams> sys;
  DeviceArray<int> sys_of;
  DeviceArray<SysControl> sysctl;
  DeviceArray<float> nu;
  DeviceArray<float> field;
  DeviceArray<double> field_partial;
  // order parameters of the whole context (fast_order_parameters)
  DeviceArray<double2> turn_table;     // unit vectors of the phase's bit groups, made at first use
  DeviceArray<double> observe_partial;
  double *h_order = nullptr;           // pinned: the four sums, written by the reduction's last block
  std::vector<SysParams> h_sys;
  int nsys = 1;
  int total_cells = 1;
  int tile_cells = 32;  // spss_set_tiling: reported back, no kernel depends on them
  int persistent = 0;
  Binner binner;
  FastControl *ctrl = nullptr;    // device
  FastControl *h_ctrl = nullptr;  // pinned mirror
  int kind = KIND_CELLS;
  // Verlet bookkeeping without lists: a Verlet-list context whose radius
  // leaves fewer than three cells per side evaluates all pairs every step and
  // keeps the displacement trigger (uses_verlet_list, accumulated displacement).
  bool trigger_only = false;
  int cap = 0;
  bool small_systems = false;  // a batch of Verlet-list systems that one CTA each rebuilds
  bool have_state = false;
  bool perm_valid = false;
  std::map<std::tuple<int, double, int>, GraphEntry> graphs;  // (stepper, dt, with sampling)
  bool device_rebuild = true;  // rebuilds tail-launched as device graphs (cleared if this device refuses)
  // per-system order parameters and their time averages
  DeviceArray<OrderSums> order_partial;
  DeviceArray<int2> order_items;   // (system, first slot) of every chunk, systems in order
  DeviceArray<int> order_first;    // first chunk of every system, nsys + 1 entries
  DeviceArray<double> order_out, stats;
  int order_chunks = 1;  // chunks of all systems
  int order_grid = 1;
  Snapshot snap;
};

// ---------------------------------------------------------------- helpers

__device__ __forceinline__ uint64_t join64(uint32_t hi, uint32_t lo)
{
  return ((uint64_t) hi << 32) | lo;
}

// The launch parameters with the fields of system S.
__device__ __forceinline__ FastParams with_system(const FastParams &P, const SysParams &S)
{
  FastParams Q = P;
  Q.nc = S.nc;
  Q.first = S.first;
  Q.sub_n = S.n;
  Q.cell0 = S.cell0;
  Q.v0 = S.v0;
  Q.xi = S.xi;
  Q.xi_r = S.xi_r;
  Q.xi_phi = S.xi_phi;
  Q.sigma = S.sigma;
  Q.ca = S.ca;
  Q.sa = S.sa;
  Q.rho2_f = S.rho2_f;
  Q.band_f = S.band_f;
  Q.b_r = S.b_r;
  Q.b_phi = S.b_phi;
  Q.rho2_d = S.rho2_d;
  Q.replica = (uint32_t) S.replica;
  return Q;
}

// round-toward-zero f * 2^64 as a signed integer, exact for the 24-bit
// mantissa; |f| < 0.5 (one step never moves a particle half a box).
__device__ __forceinline__ long long fix64_of(float f, int &err)
{
  if (!(fabsf(f) < 0.5f))
  {
    err = 1;
    return 0;
  }
  return __float2ll_rz(__fmul_rn(f, 18446744073709551616.0f));  // exact scaling by 2^64, then truncation
}

// X += dX on the periodic unit box; `carry` receives the box crossing (-1, 0, 1).
__device__ __forceinline__ uint64_t advance(uint64_t X, long long dX, int &carry)
{
  const uint64_t Y = X + (uint64_t) dX;
  carry = (dX > 0 && Y < X) ? 1 : ((dX < 0 && Y > X) ? -1 : 0);
  return Y;
}

__device__ __forceinline__ uint32_t advance_phase(uint32_t P, float dphi, int &carry, int &err)
{
  // 2^32 / (2 pi)
  const float q = dphi * 683565275.5764316f;
  carry = 0;
  if (!(fabsf(q) < 2.1e9f))
  {
    err = 1;
    return P;
  }
  const int d = __float2int_rn(q);
  const uint32_t R = P + (uint32_t) d;
  carry = (d > 0 && R < P) ? 1 : ((d < 0 && R > P) ? -1 : 0);
  return R;
}

// sin and cos of the fixed-point phase P (one turn = 2^32).  The nearest
// quarter turn comes exactly from the top bits; the remainder is the angle
// theta = 2 pi r 2^-32 in [-pi/4, pi/4), where sin and cos are an odd degree-7
// and an even degree-8 polynomial in theta (coefficients fitted by weighted
// least squares on Chebyshev nodes of theta^2, rounded to float).  The
// result is within 1e-7 of the exact sin and cos of the phase over all 2^32
// phases (the rounding of theta to float is the larger part); the quarter-turn
// rotation is exact.  Rounding is spelled out so every copy gives the same bits.
__device__ __forceinline__ void phase_sincos(uint32_t P, float &s, float &c)
{
  const uint32_t qd = (P + 0x20000000u) >> 30;  // nearest quarter turn (mod 4)
  const int r = (int) (P - (qd << 30));         // [-2^29, 2^29)
  const float th = __fmul_rn((float) r, 1.4629180792671596e-9f);  // 2 pi / 2^32
  const float t2 = __fmul_rn(th, th);
  const float ps = fmaf(th, __fmul_rn(t2, fmaf(t2, fmaf(t2, -1.9520212663337588e-4f, 8.332204073667526e-3f),
                                               -0.16666655242443085f)),
                        th);
  const float pc = fmaf(t2, fmaf(t2, fmaf(t2, fmaf(t2, 2.4394103093072772e-5f, -1.3886808883398771e-3f),
                                          4.166662320494652e-2f),
                                 -0.5f),
                        1.0f);
  // rotate by qd quarter turns: (sin, cos) = (ps, pc), (pc, -ps), (-ps, -pc), (-pc, ps)
  const float a = (qd & 1u) ? pc : ps;
  const float b = (qd & 1u) ? ps : pc;
  s = (qd & 2u) ? -a : a;
  c = ((qd + 1u) & 2u) ? -b : b;
}

__device__ __forceinline__ int cell_of_fix(uint64_t X, uint64_t Y, int nc)
{
  const int cx = (int) __umul64hi(X, (uint64_t) nc);
  const int cy = (int) __umul64hi(Y, (uint64_t) nc);
  return cy * nc + cx;
}

__device__ __forceinline__ int wrap_cell(int c, int nc)
{
  return c < 0 ? nc - 1 : (c >= nc ? 0 : c);
}

struct Acc
{
  float ss, sc, ws, wc;
  int card;
};

// A candidate pair is decided by its FP32 distance from the 32-bit high words
// (exact minimum image by integer subtraction); inside the guard band the FP64
// distance of the full 64-bit positions decides, so the neighbour set is the
// FP64 one for these positions.
__device__ __forceinline__ bool exact_within(uint32_t xh, uint32_t yh, uint32_t xl, uint32_t yl, uint64_t Xi,
                                             uint64_t Yi, double rho2)
{
  const double ex = (double) (long long) (join64(xh, xl) - Xi) * 5.421010862427522e-20;
  const double ey = (double) (long long) (join64(yh, yl) - Yi) * 5.421010862427522e-20;
  return __dadd_rn(__dmul_rn(ex, ex), __dmul_rn(ey, ey)) <= rho2;
}

__device__ __forceinline__ void accumulate(Acc &a, const uint4 &rj, float wj)
{
  const float cj = __uint_as_float(rj.z), sj = __uint_as_float(rj.w);
  a.sc += cj;
  a.ss += sj;
  a.wc = fmaf(wj, cj, a.wc);
  a.ws = fmaf(wj, sj, a.ws);
  a.card += 1;
}

// ---------------------------------------------------------------- conversions

// A block's contiguous AoS rows move between global (possibly host) memory
// and shared memory in 16-byte pieces when the array allows it, so that reads
// and writes over the host link are whole coalesced lines.
__device__ __forceinline__ void rows_to_shared(const double *__restrict__ g, double *sh, int count)
{
  if (((uintptr_t) g & 15) == 0)
  {
    const double2 *g2 = reinterpret_cast<const double2 *>(g);
    double2 *s2 = reinterpret_cast<double2 *>(sh);
    for (int i = threadIdx.x; i < count / 2; i += blockDim.x) s2[i] = g2[i];
    if ((count & 1) && threadIdx.x == 0) sh[count - 1] = g[count - 1];
  } else
  {
    for (int i = threadIdx.x; i < count; i += blockDim.x) sh[i] = g[i];
  }
}

__device__ __forceinline__ void rows_from_shared(double *__restrict__ g, const double *sh, int count)
{
  if (((uintptr_t) g & 15) == 0)
  {
    double2 *g2 = reinterpret_cast<double2 *>(g);
    const double2 *s2 = reinterpret_cast<const double2 *>(sh);
    for (int i = threadIdx.x; i < count / 2; i += blockDim.x) g2[i] = s2[i];
    if ((count & 1) && threadIdx.x == 0) g[count - 1] = sh[count - 1];
  } else
  {
    for (int i = threadIdx.x; i < count; i += blockDim.x) g[i] = sh[i];
  }
}

// A block's rows of floats to global (possibly host) memory, 16 bytes at a time
// where the array allows it.
__device__ __forceinline__ void rows_from_shared(float *__restrict__ g, const float *sh, int count)
{
  int done = 0;
  if (((uintptr_t) g & 15) == 0)
  {
    float4 *g4 = reinterpret_cast<float4 *>(g);
    const float4 *s4 = reinterpret_cast<const float4 *>(sh);
    for (int i = threadIdx.x; i < count / 4; i += blockDim.x) g4[i] = s4[i];
    done = count & ~3;
  }
  for (int i = done + threadIdx.x; i < count; i += blockDim.x) g[i] = sh[i];
}

// Upload from reference AoS, one thread per original index p (its block's
// rows read as one coalesced chunk), scattered to the particle's slot inv[p]
// (identity when no slot order exists yet).
__global__ void fast_upload_kernel(const double *__restrict__ x, int n, int s, int model, int perm_valid,
                                   FastBuffers B)
{
  extern __shared__ double rows[];
  const int p0 = blockIdx.x * blockDim.x;
  const int count = min((int) blockDim.x, n - p0) * s;
  rows_to_shared(x + (long) s * p0, rows, count);
  __syncthreads();
  const int p = p0 + threadIdx.x;
  if (p >= n) return;
  if (p == 0) B.ctrl->cells_fresh = 0;  // new positions: nothing of the last step's holds for them
  const int par = B.ctrl->parity;
  buffers_now(B, B.ctrl->order_parity);
  unsigned q = (unsigned) p;
  if (perm_valid)
  {
    q = B.inv[p];
  } else
  {
    B.pid[p] = (unsigned) p;
    B.inv[p] = (unsigned) p;
  }
  const double *st = rows + s * threadIdx.x;
  int2 im;
  uint64_t X, Y;
  {
    const double fx = floor(st[0]), fy = floor(st[1]);
    im = make_int2((int) fx, (int) fy);
    const double rx = st[0] - fx, ry = st[1] - fy;
    X = (rx * 18446744073709551616.0 >= 18446744073709551615.0) ? ~0ull : __double2ull_rz(rx * 18446744073709551616.0);
    Y = (ry * 18446744073709551616.0 >= 18446744073709551615.0) ? ~0ull : __double2ull_rz(ry * 18446744073709551616.0);
  }
  const int ip = model == 1 ? 2 : 4;
  const double t = st[ip] * 0.15915494309189535;  // phi / (2 pi)
  const double ft = floor(t);
  const double fr = (t - ft) * 4294967296.0;
  const uint32_t ph = fr >= 4294967295.0 ? 0xffffffffu : (uint32_t) fr;
  const float w = (float) st[ip + 1];
  float sp, cp;
  phase_sincos(ph, sp, cp);
  (par ? B.rec1 : B.rec0)[q] = make_uint4((uint32_t) (X >> 32), (uint32_t) (Y >> 32), __float_as_uint(cp),
                                          __float_as_uint(sp));
  (par ? B.aux1 : B.aux0)[q] = make_uint4((uint32_t) X, (uint32_t) Y, ph, __float_as_uint(w));
  B.img[p] = im;
  B.turns[p] = (int) ft;
  if (model == 2) B.vel[q] = make_float2((float) st[2], (float) st[3]);
}

// Download to reference AoS, one thread per original index: gathers the slot
// inv[p]; the block's rows are written as one coalesced chunk.
// `host_ctrl` (the step of a host array): the control block goes to its pinned
// mirror with it, and a step that failed leaves `x` as it was.
__global__ void fast_download_kernel(double *__restrict__ x, int n, int s, int model, FastBuffers B,
                                     FastControl *__restrict__ host_ctrl)
{
  pdl_enter();
  extern __shared__ double rows[];
  if (host_ctrl)
  {
    if (blockIdx.x == 0 && threadIdx.x == 0) *host_ctrl = *B.ctrl;
    if (B.ctrl->error) return;
  }
  const int p0 = blockIdx.x * blockDim.x;
  const int count = min((int) blockDim.x, n - p0) * s;
  const int p = p0 + threadIdx.x;
  if (p < n)
  {
    const int par = B.ctrl->parity;
    buffers_now(B, B.ctrl->order_parity);
    const unsigned q = B.inv[p];
    const uint4 r = (par ? B.rec1 : B.rec0)[q];
    const uint4 a = (par ? B.aux1 : B.aux0)[q];
    const int2 im = B.img[p];
    double *st = rows + s * threadIdx.x;
    st[0] = (double) im.x + (double) join64(r.x, a.x) * 5.421010862427522e-20;
    st[1] = (double) im.y + (double) join64(r.y, a.y) * 5.421010862427522e-20;
    const int ip = model == 1 ? 2 : 4;
    st[ip] = 6.283185307179586 * ((double) B.turns[p] + (double) a.z * 2.3283064365386963e-10);
    st[ip + 1] = (double) __uint_as_float(a.w);
    if (model == 2)
    {
      const float2 v = B.vel[q];
      st[2] = v.x;
      st[3] = v.y;
    }
  }
  __syncthreads();
  rows_from_shared(x + (long) s * p0, rows, count);
}

// Trajectory frame: the float conversion of the downloaded state (and, WRAP,
// the observers' wraps), one thread per original index, without the FP64 copy
// of the state in between; `out` may be host memory, which the rows then reach
// over the host link as whole lines.  N = 4,194,304 to page-locked memory:
// FP64 download, frame kernel and copy took 0.79 ms, this takes 0.535, of
// which the link needs 0.52 (100.7 MB).
template<bool WRAP>
__global__ void __launch_bounds__(256) fast_frame_kernel(float *__restrict__ out, int n, int s, int model, FastBuffers B)
{
  extern __shared__ __align__(16) float frame_rows[];
  const int p0 = blockIdx.x * blockDim.x;
  const int count = min((int) blockDim.x, n - p0) * s;
  const int p = p0 + threadIdx.x;
  if (p < n)
  {
    const int par = B.ctrl->parity;
    buffers_now(B, B.ctrl->order_parity);
    const unsigned q = B.inv[p];
    const uint4 r = (par ? B.rec1 : B.rec0)[q];
    const uint4 a = (par ? B.aux1 : B.aux0)[q];
    const int2 im = B.img[p];
    const int turns = B.turns[p];
    float *st = frame_rows + s * threadIdx.x;
    // the expressions of fast_download_kernel
    float x = __double2float_rn((double) im.x + (double) join64(r.x, a.x) * 5.421010862427522e-20);
    float y = __double2float_rn((double) im.y + (double) join64(r.y, a.y) * 5.421010862427522e-20);
    float ph = __double2float_rn(6.283185307179586 * ((double) turns + (double) a.z * 2.3283064365386963e-10));
    if (WRAP)
    {
      x = frame_wrap_position(x);
      y = frame_wrap_position(y);
      ph = frame_wrap_phase(ph);
    }
    st[0] = x;
    st[1] = y;
    const int ip = model == 1 ? 2 : 4;
    st[ip] = ph;
    st[ip + 1] = __uint_as_float(a.w);
    if (model == 2)
    {
      const float2 v = B.vel[q];
      st[2] = v.x;
      st[3] = v.y;
    }
  }
  __syncthreads();
  rows_from_shared(out + (long) s * p0, frame_rows, count);
}

// ---------------------------------------------------------------- rebuild

// Whether this rebuild covers system `sys`: every system, or those whose own
// trigger fired.  A system left out keeps its slots, cells and
// lists exactly as its last rebuild made them.
__device__ __forceinline__ bool rebuilds_system(const FastBuffers &B, int sys)
{
  return B.ctrl->rebuild != REBUILD_FLAGGED || B.sysctl[sys].rebuild;
}

// Cell id of every slot, and its arrival number in the cell (the binning's
// count, in the same pass).
__global__ void fast_cells_kernel(FastParams P, FastBuffers B)
{
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= P.n) return;
  int c;
  if (!rebuilds_system(B, B.sys_of[q]))
  {
    // sorted by cell since its last rebuild: the stable counting sort leaves it in place
    c = B.cell_sorted[q];
  } else
  {
    const int par = B.ctrl->parity;
    const uint4 r = (par ? B.rec1 : B.rec0)[q];
    const uint4 a = (par ? B.aux1 : B.aux0)[q];
    const SysParams *S = B.sys + B.sys_of[q];
    c = S->cell0 + cell_of_fix(join64(r.x, a.x), join64(r.y, a.y), S->nc);
  }
  B.cell_of[q] = c;
  B.cell_slot[q] = atomicAdd(B.cell_count + c, 1);
}

// The slots in cell order: the particle at place m of the binning's members
// (arrival order inside its cell) moves to the place its old slot has among the
// cell's, ascending: a rank among a handful of members, so the members need
// no sorting pass of their own.  Writes the other rec/aux and vel/pid buffers.
// STEP: part of a cell-list step, whose scan already exchanged vel and pid.
template<bool STEP>
__global__ void fast_permute_kernel(FastParams P, FastBuffers B)
{
  pdl_enter();
  const int m = blockIdx.x * blockDim.x + threadIdx.x;
  if (m >= P.n) return;
  if (!STEP && !rebuilds_system(B, B.sys_of[m])) return;  // its order is the identity
  const int par = B.ctrl->parity;
  buffers_now(B, B.ctrl->order_parity ^ (STEP ? 1 : 0));
  const int src = B.order[m];
  const int c = B.cell_of[src];
  const int b = B.cell_off[c], e = B.cell_off[c + 1];
  int q = b;
  for (int k = b; k < e; ++k) q += B.order[k] < src;
  (par ? B.rec0 : B.rec1)[q] = (par ? B.rec1 : B.rec0)[src];
  (par ? B.aux0 : B.aux1)[q] = (par ? B.aux1 : B.aux0)[src];
  const unsigned p = B.pid[src];
  B.pid_tmp[q] = p;
  B.inv[p] = (unsigned) q;
  if (P.model == 2) B.vel_tmp[q] = B.vel[src];
  B.cell_sorted[q] = c;
}

// A rebuild of every system leaves the permuted particles in the other buffers
// (their parities flip); a rebuild of the flagged systems copies theirs back, so
// the systems left out keep theirs where they are.
__global__ void fast_copyback_kernel(FastParams P, FastBuffers B)
{
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= P.n || B.ctrl->rebuild != REBUILD_FLAGGED) return;
  if (!rebuilds_system(B, B.sys_of[q])) return;
  const int par = B.ctrl->parity;
  buffers_now(B, B.ctrl->order_parity);
  (par ? B.rec1 : B.rec0)[q] = (par ? B.rec0 : B.rec1)[q];
  (par ? B.aux1 : B.aux0)[q] = (par ? B.aux0 : B.aux1)[q];
  B.pid[q] = B.pid_tmp[q];
  if (P.model == 2) B.vel[q] = B.vel_tmp[q];
}

// The permuted particles are current: a rebuild of every system flips the
// buffer parities (the flagged-system form copied its particles back).  One
// thread; runs before the list build, which reads them.
__global__ void fast_after_permute_kernel(FastControl *ctrl, int permuted)
{
  if (permuted && ctrl->rebuild != REBUILD_FLAGGED)
  {
    ctrl->parity ^= 1;
    ctrl->order_parity ^= 1;
  }
  ctrl->cells_fresh = 0;  // the slots moved
}

// Lists are now current.  The flags are cleared only here, after the list
// kernel, so that it rebuilds the lists of the flagged systems alone.  One block.
__global__ void fast_after_rebuild_kernel(FastControl *ctrl, SysControl *sysctl, int nsys)
{
  for (int r = threadIdx.x; r < nsys; r += blockDim.x) sysctl[r].rebuild = 0;
  if (threadIdx.x == 0)
  {
    ctrl->rebuild = REBUILD_NONE;
    ctrl->rebuilds += 1;
  }
}

// ---------------------------------------------------------------- step

// One candidate slot j of particle q, with the decision above.
template<bool OMEGA>
__device__ __forceinline__ void exact_candidate(const uint4 *__restrict__ rec, const uint4 *__restrict__ aux, int j,
                                                const uint4 &ri, uint64_t Xi, uint64_t Yi, float rho2, float band,
                                                double rho2_d, Acc &a)
{
  const uint4 rj = __ldg(rec + j), aj = __ldg(aux + j);
  const float dx = (float) (int) (rj.x - ri.x), dy = (float) (int) (rj.y - ri.y);
  const float d2 = fmaf(dx, dx, dy * dy);
  bool in = d2 <= rho2;
  if (fabsf(d2 - rho2) <= band) in = exact_within(rj.x, rj.y, aj.x, aj.y, Xi, Yi, rho2_d);
  if (in) accumulate(a, rj, OMEGA ? __uint_as_float(aj.w) : 0.0f);
}

// Neighbour sums of slot q (in cell c of an nc x nc grid with offsets coff) from
// the stencil of its cell, candidate by candidate: the cell-list step's and the
// Verlet walk's rare cases.
template<bool OMEGA>
__device__ __noinline__ void stencil_sums_exact(const uint4 *__restrict__ rec, const uint4 *__restrict__ aux,
                                                const int *__restrict__ coff, int c, int nc, int q, float rho2,
                                                float band, double rho2_d, Acc *out)
{
  const uint4 ri = rec[q], ai = aux[q];
  const uint64_t Xi = join64(ri.x, ai.x), Yi = join64(ri.y, ai.y);
  const int cy = c / nc, cx = c - cy * nc;
  Acc a{0.f, 0.f, 0.f, 0.f, 0};
  // stencil in the reference's order (-1,-1),(0,-1),(1,-1),(-1,0),... (ParticleSystemFirstOrder.cpp:47-52)
  for (int sy = -1; sy <= 1; ++sy)
  {
    const int jy = wrap_cell(cy + sy, nc);
    for (int sx = -1; sx <= 1; ++sx)
    {
      const int jc = jy * nc + wrap_cell(cx + sx, nc);
      const int e = coff[jc + 1];
      for (int j = coff[jc]; j < e; ++j)
        if (j != q) exact_candidate<OMEGA>(rec, aux, j, ri, Xi, Yi, rho2, band, rho2_d, a);
    }
  }
  *out = a;
}

// Exactly the normals the stepper consumes, in the reference's draw order.
template<int MODEL, int STEPPER>
__device__ __forceinline__ void draw_noise(const FastParams &P, unsigned long long step, unsigned p, float z[6])
{
  constexpr int kNeed = MODEL == 1 ? (STEPPER == 1 ? 1 : 2) : (STEPPER == 1 ? 3 : 6);
  p -= (unsigned) P.first;  // index of the particle within its system
  // philox_block(seed, replica, step; p, block 0) with the round keys from the parameters
  const uint4 u = philox_keyed(make_uint4(p, (uint32_t) step, (uint32_t) (step >> 32), P.replica << 8), P.kx, P.ky);
  if (kNeed > 4)
  {
    box_muller6_f32(u, z);  // six normals from the one block
    return;
  }
  box_muller_f32(u.x, u.y, z[0], z[1]);
  if (kNeed > 2) box_muller_f32(u.z, u.w, z[2], z[3]);
}

// Torque derivative f_w and (SRK) complementary force C from the neighbour
// sums.  Every rounding step is spelled out (fmaf, __fmul_rn, __fadd_rn): the
// compiler cannot contract or reassociate, so each instantiation (one system
// or a batch) rounds identically.
template<int STEPPER>
__device__ __forceinline__ void sums_forces(const FastParams &P, const Acc &a, float cphi, float sphi, float wi,
                                            float &f_w, float &C)
{
  // sum sin(phi_j - phi_i - alpha) and sum (omega_j - omega_i) cos(phi_j - phi_i - alpha)
  f_w = 0.0f;  // SE/SRK zero-fill the derivative: an isolated particle keeps 0
  C = 0.0f;
  if (a.card > 0)
  {
    const float inv = 1.0f / (float) a.card;
    const float S = fmaf(cphi, a.ss, -__fmul_rn(sphi, a.sc));  // sum sin(phi_j - phi_i)
    const float K = fmaf(cphi, a.sc, __fmul_rn(sphi, a.ss));   // sum cos(phi_j - phi_i)
    f_w = fmaf(-P.xi_phi, wi, __fmul_rn(__fmul_rn(P.sigma, fmaf(P.ca, S, -__fmul_rn(P.sa, K))), inv));
    if (STEPPER == 2)
    {
      const float WS = fmaf(cphi, a.ws, -__fmul_rn(sphi, a.wc));  // sum omega_j sin(phi_j - phi_i)
      const float WK = fmaf(cphi, a.wc, __fmul_rn(sphi, a.ws));   // sum omega_j cos(phi_j - phi_i)
      C = __fmul_rn(__fmul_rn(P.sigma, inv), __fsub_rn(fmaf(P.ca, WK, __fmul_rn(P.sa, WS)),
                                                       __fmul_rn(wi, fmaf(P.ca, K, __fmul_rn(P.sa, S)))));
    }
  }
}

template<int MODEL, int STEPPER, bool CELLS = false>
__device__ __forceinline__ float advance_particle(const FastParams &P, const FastBuffers &B, int q, const uint4 &ri,
                                                  const uint4 &ai, float2 v, float f_w, float C, const float z[6],
                                                  uint4 &rnew, uint4 &anew, int &err);

// Derivative from the neighbour sums, SE or SRK update in fixed point, new
// record.  Returns |dr|^2 of the step.
template<int MODEL, int STEPPER, bool CELLS = false>
__device__ __forceinline__ float update_particle(const FastParams &P, const FastBuffers &B, int q, const uint4 &ri,
                                                 const uint4 &ai, float2 v, const Acc &a, const float z[6],
                                                 uint4 *rout, uint4 *aout, int &err)
{
  float f_w, C;
  sums_forces<STEPPER>(P, a, __uint_as_float(ri.z), __uint_as_float(ri.w), __uint_as_float(ai.w), f_w, C);
  uint4 rnew, anew;
  const float d2 = advance_particle<MODEL, STEPPER, CELLS>(P, B, q, ri, ai, v, f_w, C, z, rnew, anew, err);
  rout[q] = rnew;
  aout[q] = anew;
  return d2;
}

// SE or SRK update in fixed point from the forces, new record.  Returns
// |dr|^2 of the step.  CELLS (cell-list steps): the new position's cell is
// counted for the next step's binning, which then needs no pass for it.
template<int MODEL, int STEPPER, bool CELLS>
__device__ __forceinline__ float advance_particle(const FastParams &P, const FastBuffers &B, int q, const uint4 &ri,
                                                  const uint4 &ai, float2 v, float f_w, float C, const float z[6],
                                                  uint4 &rnew, uint4 &anew, int &err)
{
  const uint64_t Xi = join64(ri.x, ai.x), Yi = join64(ri.y, ai.y);
  const float cphi = __uint_as_float(ri.z), sphi = __uint_as_float(ri.w);
  const float wi = __uint_as_float(ai.w);
  const float dt = P.dt;
  float ddx, ddy, dphi, dw;
  if (MODEL == 1)
  {
    const float fx = __fmul_rn(P.v0, cphi), fy = __fmul_rn(P.v0, sphi), fp = wi;
    if (STEPPER == 1)
    {
      // StochasticEulerStepperPtr.hpp:58-66
      ddx = __fmul_rn(fx, dt);
      ddy = __fmul_rn(fy, dt);
      dphi = __fmul_rn(fp, dt);
      dw = fmaf(f_w, dt, __fmul_rn(P.b_phi, __fmul_rn(P.sqdt, z[0])));
    } else
    {
      // StochasticRungeKuttaStepperPtr.hpp:54-70
      const float dW = __fmul_rn(z[0], P.sqdt);
      const float dZ = __fmul_rn(P.half_dt15, fmaf(P.inv_sqrt3, z[1], z[0]));
      ddx = fmaf(fx, dt, -__fmul_rn(__fmul_rn(fp, fy), P.half_dt2));
      ddy = fmaf(fy, dt, __fmul_rn(__fmul_rn(fp, fx), P.half_dt2));
      dphi = fmaf(fp, dt, fmaf(f_w, P.half_dt2, __fmul_rn(P.b_phi, dZ)));
      dw = fmaf(f_w, dt, fmaf(fmaf(-P.xi, f_w, C), P.half_dt2, __fmul_rn(P.b_phi, fmaf(-P.xi, dZ, dW))));
    }
  } else
  {
    const float fvx = fmaf(-P.xi_r, v.x, __fmul_rn(P.v0, cphi));
    const float fvy = fmaf(-P.xi_r, v.y, __fmul_rn(P.v0, sphi));
    float dvx, dvy;
    if (STEPPER == 1)
    {
      // StochasticEulerStepper.hpp:44-50 with AddNoise (ParticleSystemSecondOrder.cpp:447-449)
      ddx = __fmul_rn(dt, v.x);
      ddy = __fmul_rn(dt, v.y);
      dvx = fmaf(dt, fvx, __fmul_rn(P.sqdt, __fmul_rn(P.b_r, z[0])));
      dvy = fmaf(dt, fvy, __fmul_rn(P.sqdt, __fmul_rn(P.b_r, z[1])));
      dphi = __fmul_rn(dt, wi);
      dw = fmaf(dt, f_w, __fmul_rn(P.sqdt, __fmul_rn(P.b_phi, z[2])));
    } else
    {
      // second-order strong order 1.5 Taylor scheme (no reference code)
      const float dWx = __fmul_rn(z[0], P.sqdt), dZx = __fmul_rn(P.half_dt15, fmaf(P.inv_sqrt3, z[1], z[0]));
      const float dWy = __fmul_rn(z[2], P.sqdt), dZy = __fmul_rn(P.half_dt15, fmaf(P.inv_sqrt3, z[3], z[2]));
      const float dWw = __fmul_rn(z[4], P.sqdt), dZw = __fmul_rn(P.half_dt15, fmaf(P.inv_sqrt3, z[5], z[4]));
      ddx = fmaf(v.x, dt, fmaf(fvx, P.half_dt2, __fmul_rn(P.b_r, dZx)));
      ddy = fmaf(v.y, dt, fmaf(fvy, P.half_dt2, __fmul_rn(P.b_r, dZy)));
      dvx = fmaf(fvx, dt, fmaf(fmaf(-P.xi_r, fvx, -__fmul_rn(__fmul_rn(P.v0, sphi), wi)), P.half_dt2,
                               __fmul_rn(P.b_r, fmaf(-P.xi_r, dZx, dWx))));
      dvy = fmaf(fvy, dt, fmaf(fmaf(-P.xi_r, fvy, __fmul_rn(__fmul_rn(P.v0, cphi), wi)), P.half_dt2,
                               __fmul_rn(P.b_r, fmaf(-P.xi_r, dZy, dWy))));
      dphi = fmaf(wi, dt, fmaf(f_w, P.half_dt2, __fmul_rn(P.b_phi, dZw)));
      dw = fmaf(f_w, dt, fmaf(fmaf(-P.xi_phi, f_w, C), P.half_dt2, __fmul_rn(P.b_phi, fmaf(-P.xi_phi, dZw, dWw))));
    }
    B.vel[q] = make_float2(__fadd_rn(v.x, dvx), __fadd_rn(v.y, dvy));
  }
  int cx, cy, ct;
  const uint64_t Xn = advance(Xi, fix64_of(ddx, err), cx);
  const uint64_t Yn = advance(Yi, fix64_of(ddy, err), cy);
  const uint32_t Pn = advance_phase(ai.z, dphi, ct, err);
  float sn, cn;
  phase_sincos(Pn, sn, cn);
  rnew = make_uint4((uint32_t) (Xn >> 32), (uint32_t) (Yn >> 32), __float_as_uint(cn), __float_as_uint(sn));
  anew = make_uint4((uint32_t) Xn, (uint32_t) Yn, Pn, __float_as_uint(__fadd_rn(wi, dw)));
  if (CELLS)
  {
    const int c = P.cell0 + cell_of_fix(Xn, Yn, P.nc);
    B.cell_of[q] = c;
    B.cell_slot[q] = atomicAdd(B.cell_count + c, 1);
  }
  // box crossings and phase turns are rare: read-modify-write only then (the
  // counts are kept by original index, so the slot re-sort never moves them)
  if (cx | cy | ct)
  {
    const unsigned p = B.pid[q];
    if (cx | cy)
    {
      const int2 im = B.img[p];
      B.img[p] = make_int2(im.x + cx, im.y + cy);
    }
    if (ct) B.turns[p] += ct;
  }
  return fmaf(ddx, ddx, __fmul_rn(ddy, ddy));
}

// max |dr|^2 of each system for its Verlet trigger: a warp whose lanes all
// belong to one system reduces first and issues one atomic, and only when it
// can raise the maximum already stored (no block barrier).
__device__ __forceinline__ void raise_max(SysControl *sc, float d2)
{
  const unsigned bits = __float_as_uint(d2);
  if (bits > *(volatile unsigned *) &sc->max2_bits) atomicMax(&sc->max2_bits, bits);
}

__device__ __forceinline__ void publish_max(FastControl *ctrl, SysControl *sysctl, int sys, float d2max, int err)
{
  const int sys0 = __shfl_sync(0xffffffffu, sys, 0);
  if (__all_sync(0xffffffffu, sys == sys0))
  {
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) d2max = fmaxf(d2max, __shfl_xor_sync(0xffffffffu, d2max, off));
    if ((threadIdx.x & 31) == 0) raise_max(sysctl + sys0, d2max);
  } else
  {
    raise_max(sysctl + sys, d2max);
  }
  err = __any_sync(0xffffffffu, err);
  if ((threadIdx.x & 31) == 0 && err) atomicOr(&ctrl->error, 1);
}

// Whether this block is the last of the launch to get here (its partials are
// written); all threads of the block get the answer.
__device__ __forceinline__ bool last_block(FastControl *ctrl)
{
  __shared__ unsigned mine;
  __threadfence();
  __syncthreads();
  if (threadIdx.x == 0)
  {
    mine = atomicAdd(&ctrl->ticket, 1u);
    if (mine == gridDim.x - 1) ctrl->ticket = 0u;
    __threadfence();
  }
  __syncthreads();
  return mine == gridDim.x - 1;
}

// After a step: advance the noise counter and the buffer parity, accumulate
// each system's displacement in FP64 and set the rebuild flag
// (CalculateMaxDisplacement, ParticleSystemFirstOrder.cpp:670-696).  With
// per-system rebuilds (`selective`) a system whose trigger fires is flagged
// and restarts its own accumulator, so each system rebuilds exactly when it
// would alone; otherwise the lists of all systems are rebuilt together and
// every accumulator restarts.  One block, all of its threads.
__device__ __forceinline__ void end_step(FastControl *ctrl, SysControl *sysctl, const SysParams *sys, int nsys,
                                         int always_rebuild, int verlet, int selective, int cells_written)
{
  __shared__ int any;
  if (threadIdx.x == 0) any = 0;
  __syncthreads();
  for (int r = threadIdx.x; r < nsys; r += blockDim.x)
  {
    const double max2 = (double) __uint_as_float(__ldcg(&sysctl[r].max2_bits));
    sysctl[r].max2_bits = 0u;
    if (verlet && !always_rebuild)
    {
      double acc = sysctl[r].acc + sqrt(max2);
      if (acc > sys[r].half_skin)
      {
        any = 1;
        if (selective)
        {
          sysctl[r].rebuild = 1;
          acc = 0.0;
        }
      }
      sysctl[r].acc = acc;
    }
  }
  __syncthreads();
  if (any && !selective)
    for (int r = threadIdx.x; r < nsys; r += blockDim.x) sysctl[r].acc = 0.0;
  __syncthreads();
  if (threadIdx.x == 0)
  {
    ctrl->step += 1;
    ctrl->parity ^= 1;
    ctrl->cells_fresh = cells_written;
    ctrl->triggered = (always_rebuild || any) ? 1 : 0;
    if (always_rebuild) ctrl->rebuild = REBUILD_ALL;
    else if (any) ctrl->rebuild = selective ? REBUILD_FLAGGED : REBUILD_ALL;
    ctrl->acc = sysctl[0].acc;
  }
}

// ---------------------------------------------------------------- all pairs
//
// A block steps 32 particles, one per lane, and its 16 warps share the scan:
// warp w takes the w-th sixteenth of the system's slots, so all lanes of a warp
// test the same candidate (one record load for the warp) and a system of a few
// thousand particles fills the chip.  The slices are summed in order, so a
// particle's sums depend on its system alone (a system of a batch has the
// bits it has by itself).  One thread per particle scanning everything left
// most SMs idle (N = 4,000: 16 blocks): 625 us, this 18 us; the
// instructions of a pair bound it from about N = 4,000 on.
constexpr int kPairWarps = 16;

// Running sums over a slice, the (cos, sin) and omega (cos, sin) pairs packed.
// The count is kept as a float (exact below 2^24, more than a slice can be
// scanned through): the integer pipe is what bounds the loop.
struct PairAcc
{
  float2 cs, w;
  float card;
};

// Both components of a packed FP32 pair in one instruction (each rounded as
// the scalar addition and fma).
__device__ __forceinline__ float2 add2(float2 a, float2 b)
{
  float2 r;
  asm("{\n .reg .b64 x, y, z;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n add.rn.f32x2 z, x, y;\n"
      " mov.b64 {%0, %1}, z;\n}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
  return r;
}

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c)
{
  float2 r;
  asm("{\n .reg .b64 x, y, z, u;\n mov.b64 x, {%2, %3};\n mov.b64 y, {%4, %5};\n mov.b64 z, {%6, %7};\n"
      " fma.rn.f32x2 u, x, y, z;\n mov.b64 {%0, %1}, u;\n}"
      : "=f"(r.x), "=f"(r.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(c.x), "f"(c.y));
  return r;
}

// U staged candidates, decided in FP32; `nearest` keeps the smallest distance
// of any d2 to rho^2, so the caller sees whether one lay inside the guard band.
// SELF: candidate `self` (an index into the staged rows) is the particle.
template<bool OMEGA, bool SELF, int U>
__device__ __forceinline__ void pair_group(const uint4 *srec, const float *sw, int k0, int self, uint32_t xi, uint32_t yi,
                                           float rho2, float &nearest, PairAcc &a)
{
  uint4 r[U];
  float w[U], d2[U];
#pragma unroll
  for (int k = 0; k < U; ++k)
  {
    r[k] = srec[k0 + k];
    w[k] = OMEGA ? sw[k0 + k] : 0.0f;
  }
#pragma unroll
  for (int k = 0; k < U; ++k)
  {
    const float dx = (float) (int) (r[k].x - xi);
    const float dy = (float) (int) (r[k].y - yi);
    d2[k] = fmaf(dx, dx, dy * dy);
    if (SELF && k0 + k == self) d2[k] = 3.0e38f;
    nearest = fminf(nearest, fabsf(d2[k] - rho2));
  }
#pragma unroll
  for (int k = 0; k < U; ++k)
    if (d2[k] <= rho2)
    {
      const float2 cs = make_float2(__uint_as_float(r[k].z), __uint_as_float(r[k].w));
      a.cs = add2(a.cs, cs);
      if (OMEGA) a.w = fma2(make_float2(w[k], w[k]), cs, a.w);
      a.card += 1.0f;
    }
}

// The same candidates again (one of them lies inside the guard band), each
// decided by exact_within where it has to be.
template<bool OMEGA>
__device__ __noinline__ void pair_batch_exact(const uint4 *srec, const float *sw,
                                              const uint4 *__restrict__ aux, int j0, int m, int q, const uint4 ri,
                                              float rho2, float band, double rho2_d, PairAcc *acc)
{
  const uint4 ai = aux[q];
  const uint64_t Xi = join64(ri.x, ai.x), Yi = join64(ri.y, ai.y);
  PairAcc a = *acc;
  for (int k = 0; k < m; ++k)
  {
    if (j0 + k == q) continue;
    const uint4 rj = srec[k];
    const float dx = (float) (int) (rj.x - ri.x), dy = (float) (int) (rj.y - ri.y);
    const float d2 = fmaf(dx, dx, dy * dy);
    bool in = d2 <= rho2;
    if (fabsf(d2 - rho2) <= band)
    {
      const uint2 l = __ldg(reinterpret_cast<const uint2 *>(&aux[j0 + k]));
      in = exact_within(rj.x, rj.y, l.x, l.y, Xi, Yi, rho2_d);
    }
    if (!in) continue;
    const float2 cs = make_float2(__uint_as_float(rj.z), __uint_as_float(rj.w));
    a.cs = add2(a.cs, cs);
    if (OMEGA) a.w = fma2(make_float2(sw[k], sw[k]), cs, a.w);
    a.card += 1.0f;
  }
  *acc = a;
}

// Candidates [j0, j1) of particle q by one warp: 32 records at a time, one per
// lane, go through the warp's own shared rows while the next 32 are on their
// way (read straight from global memory, one candidate for the whole warp at a
// time, every eighth record waited for L2: 27.0 us at N = 4,000 against
// 18.4).  A batch with a candidate inside the guard band is done again
// with the FP64 decisions (about one in 3,000), so the common path has one
// comparison a candidate: the integer pipe (differences, conversions,
// comparisons) bounds it.
template<bool OMEGA, bool SELF>
__device__ __forceinline__ void pair_slice(const uint4 *__restrict__ rec, const uint4 *__restrict__ aux, uint4 *srec,
                                           float *sw, int j0, int j1, int q, const uint4 &ri, float rho2, float band,
                                           const double *rho2_d, PairAcc &a)
{
  const int lane = threadIdx.x & 31;
  uint4 next = make_uint4(0u, 0u, 0u, 0u);
  float next_w = 0.0f;
  if (j0 + lane < j1)
  {
    next = __ldg(&rec[j0 + lane]);
    if (OMEGA) next_w = __uint_as_float(__ldg(&aux[j0 + lane].w));
  }
  for (; j0 < j1; j0 += 32)
  {
    srec[lane] = next;
    if (OMEGA) sw[lane] = next_w;
    __syncwarp();
    if (j0 + 32 + lane < j1)
    {
      next = __ldg(&rec[j0 + 32 + lane]);
      if (OMEGA) next_w = __uint_as_float(__ldg(&aux[j0 + 32 + lane].w));
    }
    const int m = min(32, j1 - j0);
    const PairAcc before = a;
    float nearest = 3.0e38f;
    int k = 0;
#pragma unroll 1
    for (; k + 8 <= m; k += 8) pair_group<OMEGA, SELF, 8>(srec, sw, k, q - j0, ri.x, ri.y, rho2, nearest, a);
#pragma unroll 1
    for (; k < m; ++k) pair_group<OMEGA, SELF, 1>(srec, sw, k, q - j0, ri.x, ri.y, rho2, nearest, a);
    if (nearest <= band)
    {
      PairAcc again = before;
      pair_batch_exact<OMEGA>(srec, sw, aux, j0, m, q, ri, rho2, band, *rho2_d, &again);
      a = again;
    }
    __syncwarp();
  }
}

template<int MODEL, int STEPPER, bool MULTI>
__global__ void __launch_bounds__(32 * kPairWarps, 2) fast_allpairs_kernel(FastParams P, FastBuffers B)
{
  __shared__ float sums[5][kPairWarps][32];
  __shared__ __align__(16) uint4 srec[kPairWarps][32];
  __shared__ float sw[kPairWarps][STEPPER == 2 ? 32 : 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int begin = 32 * blockIdx.x;
  const int q = begin + lane;
  FastControl *ctrl = B.ctrl;
  const int par = ctrl->parity;
  buffers_now(B, ctrl->order_parity);
  const uint4 *rin = par ? B.rec1 : B.rec0;
  const uint4 *ain = par ? B.aux1 : B.aux0;
  uint4 *rout = par ? B.rec0 : B.rec1;
  uint4 *aout = par ? B.aux0 : B.aux1;
  const bool live = q < P.n;
  const int qc = live ? q : P.n - 1;
  const uint4 ri = rin[qc];
  const int sys = MULTI ? B.sys_of[qc] : 0;
  // a block of a batch may hold the end of one system and the next ones: each
  // is scanned in turn by the lanes it owns
  const int sys_end = MULTI ? B.sys_of[min(begin + 31, P.n - 1)] : 0;
  PairAcc a{make_float2(0.f, 0.f), make_float2(0.f, 0.f), 0.f};
  for (int s = MULTI ? B.sys_of[begin] : 0; s <= sys_end; ++s)
  {
    const int first = MULTI ? B.sys[s].first : P.first, n = MULTI ? B.sys[s].n : P.sub_n;
    const double *rho2_d = MULTI ? &B.sys[s].rho2_d : &P.rho2_d;
    // a lane of another system takes nothing
    const float rho2 = sys != s ? -1.0f : (MULTI ? B.sys[s].rho2_f : P.rho2_f);
    const float band = sys != s ? -1.0f : (MULTI ? B.sys[s].band_f : P.band_f);
    const int j0 = first + (int) ((long long) n * warp / kPairWarps);
    const int j1 = first + (int) ((long long) n * (warp + 1) / kPairWarps);
    if (j0 < begin + 32 && j1 > begin)
      pair_slice<STEPPER == 2, true>(rin, ain, srec[warp], sw[warp], j0, j1, qc, ri, rho2, band, rho2_d, a);
    else
      pair_slice<STEPPER == 2, false>(rin, ain, srec[warp], sw[warp], j0, j1, qc, ri, rho2, band, rho2_d, a);
  }
  sums[0][warp][lane] = a.cs.x;
  sums[1][warp][lane] = a.cs.y;
  sums[2][warp][lane] = a.card;
  if (STEPPER == 2)
  {
    sums[3][warp][lane] = a.w.x;
    sums[4][warp][lane] = a.w.y;
  }
  __syncthreads();
  // warp c adds the slices of sum c in order
  if (warp < (STEPPER == 2 ? 5 : 3))
  {
    if (warp == 2)
    {
      int card = 0;
      for (int w = 0; w < kPairWarps; ++w) card += (int) sums[2][w][lane];
      sums[2][0][lane] = __int_as_float(card);
    } else
    {
      float t = sums[warp][0][lane];
      for (int w = 1; w < kPairWarps; ++w) t = __fadd_rn(t, sums[warp][w][lane]);
      sums[warp][0][lane] = t;
    }
  }
  __syncthreads();
  if (warp != 0) return;
  float d2max = 0.0f;
  int err = 0;
  if (live)
  {
    const FastParams Q = MULTI ? with_system(P, B.sys[sys]) : P;
    const float2 v = MODEL == 2 ? B.vel[q] : make_float2(0.f, 0.f);
    float z[6];
    draw_noise<MODEL, STEPPER>(Q, ctrl->step, B.pid[q], z);
    Acc t{sums[1][0][lane], sums[0][0][lane], 0.f, 0.f, __float_as_int(sums[2][0][lane])};
    if (STEPPER == 2)
    {
      t.ws = sums[4][0][lane];
      t.wc = sums[3][0][lane];
    }
    d2max = update_particle<MODEL, STEPPER>(Q, B, q, ri, ain[q], v, t, z, rout, aout, err);
  }
  publish_max(ctrl, B.sysctl, sys, d2max, err);
}

// ---------------------------------------------------------------- cell-list step
//
// One SE or SRK step of one particle per thread, neighbours from the 3 x 3
// stencil of the cells just sorted (ParticleSystemFirstOrder.cpp:231-353).  Slots
// are in cell order, so the stencil of a cell is one run of slots per row (two
// where the periodic x-wrap crosses the row's end), in the reference's order
// (ParticleSystemFirstOrder.cpp:47-52), and a warp's runs largely coincide: the
// records come through L1 without staging, and every warp has 32 particles
// whatever their density (flocking runs cluster: after 20,000 steps at N = 65,536
// cells hold up to 100 particles, where tiles of cells took 308 us a step, this
// 44).  One comparison a candidate; a particle with a candidate inside the guard
// band is summed again with the FP64 decisions.  Instructions bound it (19
// candidates a particle at density 2).  512 systems, 8,852,499 particles, SE:
// staged one-row tiles with a layout pass 905 us, staged tiles of several rows
// 446, this 392; staging a warp's stretch of records in shared memory instead of
// leaving it to L1 ran 15 % slower, two candidates at a time everywhere as fast
// here and 20 % slower in clusters, 6 resident blocks of 256 threads 3 % slower.
template<bool OMEGA>
struct CellSums
{
  float2 cs, w;
  int card;
  float nearest;  // smallest distance of a candidate's d2 to rho^2
};

// U candidates from s on (CLAMP: those at e and beyond left out) but `self`,
// decided in FP32; their loads are in flight together.
template<bool OMEGA, int U, bool CLAMP>
__device__ __forceinline__ void cell_group(const uint4 *__restrict__ rec, const uint4 *__restrict__ aux, int s, int e,
                                           int self, uint32_t xi, uint32_t yi, float rho2, CellSums<OMEGA> &a)
{
  uint4 r[U];
  float w[U], d2[U];
#pragma unroll
  for (int k = 0; k < U; ++k)
  {
    const int t = CLAMP ? min(s + k, e - 1) : s + k;
    r[k] = __ldg(rec + t);
    w[k] = OMEGA ? __uint_as_float(__ldg(&aux[t].w)) : 0.0f;
  }
#pragma unroll
  for (int k = 0; k < U; ++k)
  {
    const float dx = (float) (int) (r[k].x - xi), dy = (float) (int) (r[k].y - yi);
    d2[k] = fmaf(dx, dx, dy * dy);
    if (s + k == self || (CLAMP && s + k >= e)) d2[k] = 3.0e38f;
    a.nearest = fminf(a.nearest, fabsf(d2[k] - rho2));
  }
#pragma unroll
  for (int k = 0; k < U; ++k)
    if (d2[k] <= rho2)
    {
      const float2 c = make_float2(__uint_as_float(r[k].z), __uint_as_float(r[k].w));
      a.cs = add2(a.cs, c);
      if (OMEGA) a.w = fma2(make_float2(w[k], w[k]), c, a.w);
      a.card += 1;
    }
}

// Candidates [s, e): in fours while they last (the long runs of dense cells),
// the rest in twos.
template<bool OMEGA>
__device__ __forceinline__ void cell_run(const uint4 *__restrict__ rec, const uint4 *__restrict__ aux, int s, int e,
                                         int self, uint32_t xi, uint32_t yi, float rho2, CellSums<OMEGA> &a)
{
#pragma unroll 1
  for (; s + 4 <= e; s += 4) cell_group<OMEGA, 4, false>(rec, aux, s, e, self, xi, yi, rho2, a);
#pragma unroll 1
  for (; s < e; s += 2) cell_group<OMEGA, 2, true>(rec, aux, s, e, self, xi, yi, rho2, a);
}

constexpr int kCellThreads = 128;
constexpr int kCellBlocks = 12;  // an SM: 40 registers a thread

// `fresh`: the slots were just re-sorted (the particles stand in the other
// rec/aux buffer, the step was counted by the scan); 0: a step on the lists of
// an earlier binning.
template<int MODEL, int STEPPER, bool MULTI>
__global__ void __launch_bounds__(kCellThreads, kCellBlocks) fast_cell_step_kernel(FastParams P, FastBuffers B, int fresh)
{
  pdl_enter();
  constexpr bool OMEGA = STEPPER == 2;
  const int q = blockIdx.x * kCellThreads + threadIdx.x;
  if (q >= P.n) return;
  FastControl *ctrl = B.ctrl;
  const int par = ctrl->parity ^ fresh;
  buffers_now(B, ctrl->order_parity);
  const uint4 *rin = par ? B.rec1 : B.rec0;
  const uint4 *ain = par ? B.aux1 : B.aux0;
  uint4 *rout = par ? B.rec0 : B.rec1;
  uint4 *aout = par ? B.aux0 : B.aux1;
  const SysParams *S = MULTI ? B.sys + B.sys_of[q] : nullptr;
  const int cell0 = MULTI ? S->cell0 : P.cell0, nc = MULTI ? S->nc : P.nc;
  const float rho2 = MULTI ? S->rho2_f : P.rho2_f, band = MULTI ? S->band_f : P.band_f;
  const int c = B.cell_sorted[q] - cell0;
  const uint4 ri = rin[q];
  const int cy = c / nc, cx = c - cy * nc;
  const int *coff = B.cell_off + cell0;
  CellSums<OMEGA> a{make_float2(0.f, 0.f), make_float2(0.f, 0.f), 0, 3.0e38f};
  if (nc >= 3)
  {
    const int lo = max(cx - 1, 0), hi = min(cx + 2, nc);
    int s[3], e[3];
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
      const int row = wrap_cell(cy + k - 1, nc) * nc;
      s[k] = coff[row + lo];
      e[k] = coff[row + hi];
    }
    if (cx > 0 && cx + 1 < nc)
    {
#pragma unroll
      for (int k = 0; k < 3; ++k) cell_run<OMEGA>(rin, ain, s[k], e[k], q, ri.x, ri.y, rho2, a);
    } else
    {
      for (int k = 0; k < 3; ++k)
      {
        const int row = wrap_cell(cy + k - 1, nc) * nc;
        const int wx = row + (cx == 0 ? nc - 1 : 0);
        const int ws = coff[wx], we = coff[wx + 1];
        const int rs = coff[row + lo], re = coff[row + hi];
        if (cx == 0) cell_run<OMEGA>(rin, ain, ws, we, q, ri.x, ri.y, rho2, a);
        cell_run<OMEGA>(rin, ain, rs, re, q, ri.x, ri.y, rho2, a);
        if (cx != 0) cell_run<OMEGA>(rin, ain, ws, we, q, ri.x, ri.y, rho2, a);
      }
    }
  }
  Acc t{a.cs.y, a.cs.x, a.w.y, a.w.x, a.card};
  if (nc < 3 || a.nearest <= band)
  {
    // fewer than three cells a side (the stencil meets cells more than once), or
    // a candidate inside the guard band
    Acc again;
    stencil_sums_exact<OMEGA>(rin, ain, coff, c, nc, q, rho2, band, MULTI ? S->rho2_d : P.rho2_d, &again);
    t = again;
  }
  const uint4 ai = ain[q];
  const FastParams Q = MULTI ? with_system(P, *S) : P;
  int err = 0;
  float z[6];
  draw_noise<MODEL, STEPPER>(Q, ctrl->step - (unsigned long long) fresh, B.pid[q], z);
  update_particle<MODEL, STEPPER, true>(Q, B, q, ri, ai, MODEL == 2 ? B.vel[q] : make_float2(0.f, 0.f), t, z, rout, aout,
                                        err);
  if (err) atomicOr(&ctrl->error, 1);
}

// ---------------------------------------------------------------- Verlet lists
//
// Lists by slot, the 32 slots of a warp together: entries 4 g .. 4 g + 3 of slot
// q stand in the eight bytes at [q / 32][g][q mod 32], so a warp reads four
// entries of all its lanes as one 256-byte line and its lists are one stretch of
// memory (rows [g][q] over all slots instead: the list kernel 300 us for 238 us
// at 4.19 million particles).  An entry is the neighbour's slot offset j - q in
// 16 bits, modulo the system's size where the stencil crosses the vertical
// periodic boundary (kListWrapped in the count: one list in 70 at N = 65,536; as
// stencil scans these few took as long as the rest of the step).  A count of -1 marks a list longer than the capacity or an offset
// beyond 16 bits; the step then scans the stencil of the rebuild-time cell,
// which holds every particle the list would.
constexpr int kListWrapped = 1 << 30;

// Slot of an entry of a wrapped list: q + e back into the system's slots.
__device__ __forceinline__ int wrapped_slot(int q, int e, int first, int n)
{
  const int j = q + e;
  return j < first ? j + n : (j >= first + n ? j - n : j);
}

__device__ __forceinline__ long list_at(int cap, int q)
{
  return (long) (q >> 5) * (32L * cap) + 4 * (q & 31);
}

// Verlet list of slot q from the 3x3 stencil of the rebuild grid
// (ParticleSystemFirstOrder.cpp:536-589): pairs with r <= r_max (conservatively
// widened by the guard band; an entry beyond r_max can never come within rho
// before the next rebuild), in the reference's order.
__device__ __forceinline__ void build_list(const FastParams &P, const FastBuffers &B, const SysParams *S,
                                           const uint4 *rec, int q)
{
  const int nc = S->nc;
  const float rmax2 = S->rmax2_f;
  const int *coff = B.cell_off + S->cell0;
  const int c = B.cell_sorted[q] - S->cell0;
  const uint2 ri = *reinterpret_cast<const uint2 *>(rec + q);
  const int cy = c / nc, cx = c - cy * nc;
  short *list = B.vl + list_at(P.cap, q);
  const int n = S->n, half = n / 2;
  int cnt = 0;
  bool far = false, wrapped = false;
  auto scan = [&](int s, int e) {
    for (; s < e; s += 4)
    {
      uint2 r[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) r[k] = __ldg(reinterpret_cast<const uint2 *>(rec + min(s + k, e - 1)));
#pragma unroll
      for (int k = 0; k < 4; ++k)
      {
        const float dx = (float) (int) (r[k].x - ri.x), dy = (float) (int) (r[k].y - ri.y);
        if (s + k >= e || s + k == q || !(fmaf(dx, dx, dy * dy) <= rmax2)) continue;
        int off = s + k - q;
        if (off != (int) (short) off)
        {
          off += off > half ? -n : n;
          far |= off != (int) (short) off;
          wrapped = true;
        }
        if (cnt < P.cap) list[(cnt >> 2) * 128 + (cnt & 3)] = (short) off;
        ++cnt;
      }
    }
  };
  for (int sy = -1; sy <= 1; ++sy)
  {
    const int row = wrap_cell(cy + sy, nc) * nc;
    if (cx > 0 && cx + 1 < nc)
    {
      scan(coff[row + cx - 1], coff[row + cx + 2]);
    } else
    {
      for (int sx = -1; sx <= 1; ++sx)
      {
        const int jc = row + wrap_cell(cx + sx, nc);
        scan(coff[jc], coff[jc + 1]);
      }
    }
  }
  if (cnt > P.cap) atomicMax(&B.ctrl->overflow, cnt);
  B.vl_cnt[q] = (cnt > P.cap || far) ? -1 : (wrapped ? cnt | kListWrapped : cnt);
}

// One slot per thread.  `finish`: the launch also ends the rebuild (the batches
// of small systems, whose step graphs hold it unconditionally: it leaves at once
// when nothing is due).
constexpr int kBuildThreads = 256;

__global__ void __launch_bounds__(kBuildThreads) fast_verlet_build_kernel(FastParams P, FastBuffers B, int finish)
{
  FastControl *ctrl = B.ctrl;
  if (finish && ctrl->rebuild == REBUILD_NONE) return;
  const int q = blockIdx.x * kBuildThreads + threadIdx.x;
  if (q < P.n)
  {
    const SysParams *S = B.sys + B.sys_of[q];
    if (rebuilds_system(B, S->index)) build_list(P, B, S, ctrl->parity ? B.rec1 : B.rec0, q);
  }
  if (!finish || !last_block(ctrl)) return;
  for (int r = threadIdx.x; r < P.nsys; r += kBuildThreads) B.sysctl[r].rebuild = 0;
  if (threadIdx.x == 0)
  {
    ctrl->rebuild = REBUILD_NONE;
    ctrl->rebuilds += 1;
    ctrl->cells_fresh = 0;
  }
}

// The re-sort of one small system by one CTA: cell ids and counts, offsets,
// members, the particles through the other buffers and back (so no parity flips
// and the other systems are not touched); CTAs of systems that are not due leave
// at once, and the list kernel follows.  A batch of a thousand systems rebuilds
// some of them on most steps, and the general sequence of eleven launches over
// every slot, launched from the device, took as long as the step.  1,024
// systems of 1,024 particles, one of them or all due, take 12.6 us; a step with
// its share of rebuilds 80.5 -> 55 us, in clustered states, where some system is
// due on every step, 336 -> 160 us (the list build in this kernel: 190 us; with
// 1,024 threads: 14 us).
constexpr int kSystemThreads = 512;
constexpr int kSystemSlots = 4096;  // largest system taken
constexpr int kSystemCells = 4096;  // and cells of its grid

__global__ void __launch_bounds__(kSystemThreads) fast_system_rebuild_kernel(FastParams P, FastBuffers B)
{
  __shared__ int off[kSystemCells + 1];            // counts, then offsets within the system
  __shared__ short member[kSystemSlots], cell[kSystemSlots];
  __shared__ unsigned short arrival[kSystemSlots];
  __shared__ int warp_tot[kSystemThreads / 32];
  FastControl *ctrl = B.ctrl;
  if (ctrl->rebuild == REBUILD_NONE) return;
  const SysParams *S = B.sys + blockIdx.x;
  const bool due = rebuilds_system(B, blockIdx.x);
  if (due)
  {
    const int n = S->n, first = S->first, nc = S->nc, ncell = nc * nc, cell0 = S->cell0;
    const int par = ctrl->parity;
    buffers_now(B, ctrl->order_parity);
    uint4 *rec = par ? B.rec1 : B.rec0, *rec_to = par ? B.rec0 : B.rec1;
    uint4 *aux = par ? B.aux1 : B.aux0, *aux_to = par ? B.aux0 : B.aux1;
    for (int c = threadIdx.x; c < ncell; c += kSystemThreads) off[c] = 0;
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += kSystemThreads)
    {
      const uint4 r = rec[first + i], a = aux[first + i];
      const int c = cell_of_fix(join64(r.x, a.x), join64(r.y, a.y), nc);
      cell[i] = (short) c;
      arrival[i] = (unsigned short) atomicAdd(&off[c], 1);
    }
    __syncthreads();
    // exclusive scan of the counts: consecutive cells a thread
    {
      constexpr int kItems = kSystemCells / kSystemThreads;
      const int base = threadIdx.x * kItems, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
      int v[kItems], local = 0;
#pragma unroll
      for (int k = 0; k < kItems; ++k)
      {
        v[k] = base + k < ncell ? off[base + k] : 0;
        local += v[k];
      }
      int x = local;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1)
      {
        const int y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
      }
      if (lane == 31) warp_tot[warp] = x;
      __syncthreads();
      int excl = x - local;
      for (int w = 0; w < warp; ++w) excl += warp_tot[w];
#pragma unroll
      for (int k = 0; k < kItems; ++k)
      {
        if (base + k < ncell)
        {
          off[base + k] = excl;
          B.cell_off_w[cell0 + base + k] = first + excl;
        }
        excl += v[k];
      }
      if (threadIdx.x == 0)
      {
        off[ncell] = n;
        B.cell_off_w[cell0 + ncell] = first + n;  // the next system's first offset, or the total: the same value
      }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += kSystemThreads) member[off[cell[i]] + arrival[i]] = (short) i;
    __syncthreads();
    for (int m = threadIdx.x; m < n; m += kSystemThreads)
    {
      const int i = member[m], c = cell[i], b = off[c], e = off[c + 1];
      int q = b;
      for (int k = b; k < e; ++k) q += member[k] < i;
      const int src = first + i, to = first + q;
      rec_to[to] = rec[src];
      aux_to[to] = aux[src];
      const unsigned p = B.pid[src];
      B.pid_tmp[to] = p;
      B.inv[p] = (unsigned) to;
      if (P.model == 2) B.vel_tmp[to] = B.vel[src];
      B.cell_sorted[to] = cell0 + c;
    }
    __syncthreads();
    for (int i = threadIdx.x; i < n; i += kSystemThreads)
    {
      const int q = first + i;
      rec[q] = rec_to[q];
      aux[q] = aux_to[q];
      B.pid[q] = B.pid_tmp[q];
      if (P.model == 2) B.vel[q] = B.vel_tmp[q];
    }
  }
}

// A particle's own words, loaded from global memory at its slot.
struct OwnParticle
{
  unsigned p;  // original index (noise counter)
  uint4 r, a;  // record and aux words
  float2 v;    // velocity (second order)
};

template<int MODEL>
__device__ __forceinline__ OwnParticle load_own(const FastBuffers &B, const uint4 *rin, const uint4 *ain, int q)
{
  OwnParticle o;
  o.p = B.pid[q];
  o.r = rin[q];
  o.a = ain[q];
  o.v = MODEL == 2 ? B.vel[q] : make_float2(0.f, 0.f);
  return o;
}

// Listed neighbours again, candidate by candidate.
template<bool OMEGA>
__device__ __noinline__ void list_sums_exact(const uint4 *__restrict__ rec, const uint4 *__restrict__ aux,
                                             const short *list, int cnt, int q, int first, int n,
                                             float rho2, float band, double rho2_d, Acc *out)
{
  const uint4 ri = rec[q], ai = aux[q];
  const uint64_t Xi = join64(ri.x, ai.x), Yi = join64(ri.y, ai.y);
  Acc a{0.f, 0.f, 0.f, 0.f, 0};
  for (int m = 0; m < cnt; ++m)
    exact_candidate<OMEGA>(rec, aux, wrapped_slot(q, list[(m >> 2) * 128 + (m & 3)], first, n), ri, Xi, Yi, rho2,
                           band, rho2_d, a);
  *out = a;
}

// The listed neighbours of particle q in fours, decided in FP32; the entries of
// the next four are on their way meanwhile.
template<bool OMEGA, bool WRAPPED>
__device__ __forceinline__ void walk_list(const uint4 *__restrict__ rec, const uint4 *__restrict__ aux,
                                          const short *list, short4 next, int cnt, int q, int first, int n,
                                          uint32_t xi, uint32_t yi, float rho2, CellSums<OMEGA> &a)
{
#pragma unroll 1
  for (int m = 0; m < cnt; m += 4)
  {
    const short4 e = next;
    list += 128;
    if (m + 4 < cnt) next = *reinterpret_cast<const short4 *>(list);
    const int last = cnt - m;
    // entries past the end repeat the particle itself, which is never counted
    int j[4] = {q + e.x, last > 1 ? q + e.y : q, last > 2 ? q + e.z : q, last > 3 ? q + e.w : q};
    if (WRAPPED)
#pragma unroll
      for (int k = 0; k < 4; ++k) j[k] = wrapped_slot(j[k], 0, first, n);
    uint4 r[4];
    float w[4], d2[4];
#pragma unroll
    for (int k = 0; k < 4; ++k)
    {
      r[k] = __ldg(rec + j[k]);
      w[k] = OMEGA ? __uint_as_float(__ldg(&aux[j[k]].w)) : 0.0f;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
    {
      const float dx = (float) (int) (r[k].x - xi), dy = (float) (int) (r[k].y - yi);
      d2[k] = fmaf(dx, dx, dy * dy);
      if (k > 0 && last <= k) d2[k] = 3.0e38f;
      a.nearest = fminf(a.nearest, fabsf(d2[k] - rho2));
    }
#pragma unroll
    for (int k = 0; k < 4; ++k)
      if (d2[k] <= rho2)
      {
        const float2 c = make_float2(__uint_as_float(r[k].z), __uint_as_float(r[k].w));
        a.cs = add2(a.cs, c);
        if (OMEGA) a.w = fma2(make_float2(w[k], w[k]), c, a.w);
        a.card += 1;
      }
  }
}

constexpr int kTileThreads = 128;
constexpr int kTileBlocksSRK = 12, kTileBlocksSE = 13;  // an SM: 40 and 32 registers a thread

// SE or SRK step of a tile of 128 slots a CTA, one particle per thread, neighbours
// from its Verlet list through L1 (a warp's particles are neighbours of each other).
template<int MODEL, int STEPPER, bool MULTI>
__global__ void __launch_bounds__(kTileThreads, STEPPER == 2 ? kTileBlocksSRK : kTileBlocksSE)
    fast_tile_kernel(FastParams P, FastBuffers B)
{
  pdl_enter();
  constexpr bool OMEGA = STEPPER == 2;
  const int slot = blockIdx.x * kTileThreads + threadIdx.x;
  const int q = min(slot, P.n - 1);
  FastControl *ctrl = B.ctrl;
  const int par = ctrl->parity;
  buffers_now(B, ctrl->order_parity);
  const uint4 *rin = par ? B.rec1 : B.rec0;
  const uint4 *ain = par ? B.aux1 : B.aux0;
  uint4 *rout = par ? B.rec0 : B.rec1;
  uint4 *aout = par ? B.aux0 : B.aux1;
  const int listed = B.vl_cnt[q];
  const int cnt = listed < 0 ? listed : listed & ~kListWrapped;
  const short *list = B.vl + list_at(P.cap, q);
  const uint4 ri = rin[q];
  // the first entries of every list, before anything waits
  const short4 entries = *reinterpret_cast<const short4 *>(list);
  const int sys = MULTI ? B.sys_of[q] : 0;
  const SysParams *S = MULTI ? B.sys + sys : nullptr;
  const float rho2 = MULTI ? S->rho2_f : P.rho2_f;
  CellSums<OMEGA> a{make_float2(0.f, 0.f), make_float2(0.f, 0.f), 0, 3.0e38f};
  if (listed == cnt)
    walk_list<OMEGA, false>(rin, ain, list, entries, cnt, q, 0, 0, ri.x, ri.y, rho2, a);
  else
    walk_list<OMEGA, true>(rin, ain, list, entries, cnt, q, MULTI ? S->first : P.first, MULTI ? S->n : P.sub_n, ri.x,
                           ri.y, rho2, a);
  float d2max = 0.0f;
  int err = 0;
  if (slot < P.n)
  {
    Acc t{a.cs.y, a.cs.x, a.w.y, a.w.x, a.card};
    const float band = MULTI ? S->band_f : P.band_f;
    if (cnt < 0 || a.nearest <= band)
    {
      const double rho2_d = MULTI ? S->rho2_d : P.rho2_d;
      const int cell0 = MULTI ? S->cell0 : P.cell0, nc = MULTI ? S->nc : P.nc;
      Acc again;
      if (cnt < 0)
        stencil_sums_exact<OMEGA>(rin, ain, B.cell_off + cell0, B.cell_sorted[q] - cell0, nc, q, rho2, band, rho2_d,
                                  &again);
      else
        list_sums_exact<OMEGA>(rin, ain, list, cnt, q, MULTI ? S->first : P.first, MULTI ? S->n : P.sub_n, rho2, band,
                               rho2_d, &again);
      t = again;
    }
    const OwnParticle o = load_own<MODEL>(B, rin, ain, q);
    const FastParams Q = MULTI ? with_system(P, *S) : P;
    float z[6];
    draw_noise<MODEL, STEPPER>(Q, ctrl->step, o.p, z);
    d2max = update_particle<MODEL, STEPPER>(Q, B, q, o.r, o.a, o.v, t, z, rout, aout, err);
  }
  publish_max(ctrl, B.sysctl, sys, d2max, err);
}

// end_step as a launch of its own, resident before the step kernel ends (a step
// of 2,000 to 65,536 particles on Verlet lists 0.5 us shorter; as the last block
// of the step kernel, whose barrier and registers every block then pays for,
// 1 to 2 us longer, 25 % at 4,194,304).
// TAIL (steps run as graphs): `rebuild_exec`, the rebuild as a device graph,
// is tail-launched here when a rebuild is due, so it runs right after this
// step's graph and before the next one, and a step without a rebuild needs
// no conditional node.  A kernel that can launch a graph runs only as a node
// of a graph, so eager steps use the form without it.
template<bool TAIL>
__global__ void fast_control_kernel(FastControl *ctrl, SysControl *sysctl, const SysParams *sys, int nsys,
                                    int always_rebuild, int verlet, int selective, int cells_written,
                                    cudaGraphExec_t rebuild_exec)
{
  pdl_enter();
  end_step(ctrl, sysctl, sys, nsys, always_rebuild, verlet, selective, cells_written);
  if (threadIdx.x == 0 && TAIL && ctrl->rebuild)
    if (cudaGraphLaunch(rebuild_exec, cudaStreamGraphTailLaunch) != cudaSuccess) atomicOr(&ctrl->error, 8);
}

__global__ void fast_set_condition_kernel(const FastControl *ctrl, cudaGraphConditionalHandle handle)
{
  cudaGraphSetConditional(handle, ctrl->rebuild ? 1u : 0u);
}

__global__ void fast_noise_kernel(double *__restrict__ out, int n, int per, NoiseKey nk, const SysParams *sys,
                                  const int *sys_of)
{
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= n) return;
  const SysParams *S = sys + sys_of[p];
  nk.replica = (uint32_t) S->replica;
  const uint32_t local = (uint32_t) (p - S->first);
  float z[6];
  if (per > 4)
  {
    box_muller6_f32(philox_block(nk, local, 0), z);
  } else
  {
    normals4_f32(nk, local, 0, z);
  }
  for (int d = 0; d < per; ++d) out[(long) per * p + d] = (double) z[d];
}

// ApplyPeriodicBoundaryConditions: positions are kept wrapped; forget the box crossings.
__global__ void fast_pbc_kernel(int2 *img, int n)
{
  const int q = blockIdx.x * blockDim.x + threadIdx.x;
  if (q < n) img[q] = make_int2(0, 0);
}

// ---------------------------------------------------------------- order parameters per system
//
// Phase order |<e^{i phi}>| and, for the second-order model, the polar order
// of the velocity directions |<v/|v|>| of every system (the observers'
// reduction, BinaryObserverFirstOrder.cpp:125-142, BinaryObserverSecondOrder.cpp:121-138),
// summed in FP64 from the records of the current state.

constexpr int kOrderChunk = 2048;  // slots per partial sum
constexpr int kOrderThreads = 256;

// Whether a sample follows the step that brought the counter to `step`.
__host__ __device__ __forceinline__ bool samples_after(const FastControl *c, unsigned long long step)
{
  return c->sample_every > 0 && (long long) step >= c->sample_from && (long long) step % c->sample_every == 0;
}

__device__ __forceinline__ bool sample_now(const FastControl *c)
{
  return samples_after(c, c->step);
}

__device__ __forceinline__ double warp_sum(double v)
{
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

// The double x 2^ex of a finite float by integer instructions (a conversion takes
// the FP64 pipe); subnormal ones by way of a multiple of theirs.
__device__ __forceinline__ double widen(float x, int ex = 0)
{
  const bool small = fabsf(x) < 1.17549435e-38f;  // the smallest normal float
  const uint32_t b = __float_as_uint(small ? x * 4294967296.0f : x), m = b & 0x7fffffffu;
  const uint32_t hi = m ? (b & 0x80000000u) | ((m >> 3) + (small ? 0x36000000u : 0x38000000u) + ((uint32_t) ex << 20)) : 0u;
  return __hiloint2double((int) hi, (int) (b << 29));
}

// v / |v| in FP64, added to (sx, sy); nothing for v = 0.  The reciprocal square
// root starts from the FP32 one (relative error below 2^-22) and takes one
// third-order step, y (1 + e/2 + 3 e^2/8) with e = 1 - |v|^2 y^2, whose
// remainder 5 e^3 / 16 is below 1e-19: nine FP64 instructions against about 70
// for the square root and the two divisions (GB300 runs FP64 at 1/69 of its
// FP32 rate, so the FP64 count is what these reductions cost).
__device__ __forceinline__ void add_direction(float2 v, double &sx, double &sy)
{
  // powers of two that bring the larger component near 1: no overflow or
  // underflow of the FP32 square for any finite v
  const float big = fmaxf(fabsf(v.x), fabsf(v.y));
  if (!(big > 0.0f)) return;
  const int ex = max(-120, min(120, 127 - (int) (__float_as_uint(big) >> 23)));
  const float scale = __uint_as_float((uint32_t) (ex + 127) << 23);
  const float fx = __fmul_rn(v.x, scale), fy = __fmul_rn(v.y, scale);
  const float f2 = fmaf(fx, fx, __fmul_rn(fy, fy));
  if (!(f2 > 0.0f)) return;  // a NaN component: left out, as a comparison |v| > 0 leaves it out
  if (f2 > 3.0e38f)          // an infinite one has no direction
  {
    sx = sy = __longlong_as_double(0x7ff8000000000000ll);
    return;
  }
  const double x = widen(v.x, ex), y = widen(v.y, ex), r = widen(rsqrtf(f2));
  const double m2 = fma(x, x, y * y);
  const double e = fma(-m2 * r, r, 1.0);
  const double c = fma(r * e, fma(e, 0.375, 0.5), r);
  sx = fma(x, c, sx);
  sy = fma(y, c, sy);
}

// Sum of sines or cosines as integers, in units of 2^-24 and 2^-53 (the last bit of
// the smallest one, of a phase 2^-32 turns from a multiple of a quarter): exact,
// at a quarter of the conversion and the addition in FP64.  Up to 64 terms.
struct UnitSum
{
  int hi = 0;
  long long lo = 0;

  __device__ __forceinline__ void add(float x)
  {
    const float t = x * 16777216.0f;
    const int h = __float2int_rn(t);
    hi += h;
    lo += __float2int_rn((t - (float) h) * 536870912.0f);
  }

  __device__ __forceinline__ double value() const
  {
    return (double) (((long long) hi << 29) + lo) * 1.1102230246251565e-16;
  }
};

// partial[k] = sums over chunk k (at most kOrderChunk slots of one system);
// a small grid walks all chunks, so the gated launch that finds no sampling
// step costs a few hundred CTAs.  FP64 instructions bound it (nine a particle,
// 24 with conversions, FP64 sums of the phases' floats and a tree for each sum):
// with the finish kernel 414 -> 229 us for 8.85 million particles in 512
// systems, 84 -> 57 us for 1,024 systems of 1,024.
__global__ void __launch_bounds__(kOrderThreads) fast_order_partials_kernel(FastParams P, FastBuffers B, OrderSums *__restrict__ partial,
                                           const int2 *__restrict__ items, int nitems, int gated)
{
  if (gated && !sample_now(B.ctrl)) return;
  const uint4 *rec = B.ctrl->parity ? B.rec1 : B.rec0;
  buffers_now(B, B.ctrl->order_parity);
  for (int k = blockIdx.x; k < nitems; k += gridDim.x)
  {
    const int2 it = items[k];
    const SysParams *S = B.sys + it.x;
    const long begin = it.y;
    const long end = min((long) S->first + S->n, begin + kOrderChunk);
    double a[4] = {0.0, 0.0, 0.0, 0.0};
    UnitSum c, sn;
#pragma unroll 4
    for (long q = begin + threadIdx.x; q < end; q += kOrderThreads)
    {
      const uint4 r = rec[q];
      c.add(__uint_as_float(r.z));
      sn.add(__uint_as_float(r.w));
      if (P.model == 2) add_direction(B.vel[q], a[2], a[3]);
    }
    a[0] = c.value();
    a[1] = sn.value();
    const double sum = block_sum4(warp_sum4(a));
    if (threadIdx.x < 32 && (threadIdx.x & 7) == 0)
      reinterpret_cast<double *>(partial + k)[threadIdx.x >> 3] = sum;
  }
}

// Per system: the order parameters (R, arg, R_v, arg_v) into out4 and, after a
// sampling step, the running sums of R, R^2, R_v, R_v^2 and the sample count.
// Blocks of one warp, so the arguments' FP64 work spreads over the SMs.
__global__ void fast_order_finish_kernel(FastParams P, FastBuffers B, const OrderSums *__restrict__ partial,
                                         const int *__restrict__ first_item, double *__restrict__ out4,
                                         double *__restrict__ stats, int gated)
{
  const int r = blockIdx.x * blockDim.x + threadIdx.x;
  if (r >= P.nsys) return;
  if (gated && !sample_now(B.ctrl)) return;
  double t0 = 0.0, t1 = 0.0, t2 = 0.0, t3 = 0.0;
#pragma unroll 4
  for (int c = first_item[r]; c < first_item[r + 1]; ++c)
  {
    const OrderSums v = partial[c];
    t0 += v.c;
    t1 += v.s;
    t2 += v.vx;
    t3 += v.vy;
  }
  const double n = (double) B.sys[r].n;
  const double re = t0 / n, im = t1 / n;
  double o[4];
  o[0] = sqrt(re * re + im * im);
  o[1] = atan2(im, re);
  if (P.model == 2)
  {
    const double vre = t2 / n, vim = t3 / n;
    o[2] = sqrt(vre * vre + vim * vim);
    o[3] = atan2(vim, vre);
  } else
  {
    o[2] = o[0];
    o[3] = o[1];
  }
  for (int k = 0; k < 4; ++k) out4[4 * r + k] = o[k];
  if (gated)
  {
    double *st = stats + 5 * r;
    st[0] += o[0];
    st[1] += o[0] * o[0];
    st[2] += o[2];
    st[3] += o[2] * o[2];
    st[4] += 1.0;
  }
}

// ---------------------------------------------------------------- global polar order field
//
// EvaluateInteractionsWithGlobalPolarOrderField (ParticleSystemFirstOrderPtr.cpp:155-223):
// every particle couples to Z = <e^{i phi}> (and, for the complementary force
// of the SRK stepper, to W = <omega e^{i phi}>), both summed over the stage state
// as error-free FP32 pairs within a warp, in FP64 beyond; no lists.  The field is
// rounded to FP32, whose last bit is some 2^24 times what the pairs leave out.  (An
// omega that overflows them has failed its step: |omega| dt must stay below pi.)

constexpr int kFieldThreads = 256;  // as block_sum4 needs
constexpr int kFieldBlocks = 2 * 152;

// Error-free running sum hi + lo of floats (Knuth's TwoSum): the rounding
// error of every addition is kept in lo.
__device__ __forceinline__ void two_sum_add(float &hi, float &lo, float x)
{
  const float s = __fadd_rn(hi, x);
  const float b = __fsub_rn(s, hi);
  lo = __fadd_rn(lo, __fadd_rn(__fsub_rn(hi, __fsub_rn(s, b)), __fsub_rn(x, b)));
  hi = s;
}

// Running sums of cos phi, sin phi, omega cos phi and omega sin phi over a
// thread's particles, in FP32 with every rounding error kept (products too),
// which no FP64 sum of so few terms would better by more than 1e-14 of a term;
// FP64 takes over at the thread sums.
struct FieldSum
{
  float hi[4] = {0.f, 0.f, 0.f, 0.f}, lo[4] = {0.f, 0.f, 0.f, 0.f};

  __device__ __forceinline__ void add(float c, float sn, float w)
  {
    const float wc = __fmul_rn(w, c), ws = __fmul_rn(w, sn);
    two_sum_add(hi[0], lo[0], c);
    two_sum_add(hi[1], lo[1], sn);
    two_sum_add(hi[2], lo[2], wc);
    two_sum_add(hi[3], lo[3], ws);
    lo[2] = __fadd_rn(lo[2], fmaf(w, c, -wc));
    lo[3] = __fadd_rn(lo[3], fmaf(w, sn, -ws));
  }
};

// (hi, lo) of two such sums.
__device__ __forceinline__ void sum_add(float &hi, float &lo, float ohi, float olo)
{
  two_sum_add(hi, lo, ohi);
  lo = __fadd_rn(lo, olo);
}

// warp_sum4 of a FieldSum: the pairs are added as pairs, FP64 takes over at the
// warp's sums (conversions included 3 FP64 instructions a warp, not 32).
__device__ __forceinline__ double field_warp_sum(const FieldSum &f)
{
  const int lane = threadIdx.x & 31;
  const bool up = lane & 16, odd = lane & 8;
  float h[2], l[2];
#pragma unroll
  for (int c = 0; c < 2; ++c)
  {
    h[c] = up ? f.hi[c + 2] : f.hi[c];
    l[c] = up ? f.lo[c + 2] : f.lo[c];
    sum_add(h[c], l[c], __shfl_xor_sync(0xffffffffu, up ? f.hi[c] : f.hi[c + 2], 16),
            __shfl_xor_sync(0xffffffffu, up ? f.lo[c] : f.lo[c + 2], 16));
  }
  float hi = odd ? h[1] : h[0], lo = odd ? l[1] : l[0];
  sum_add(hi, lo, __shfl_xor_sync(0xffffffffu, odd ? h[0] : h[1], 8),
          __shfl_xor_sync(0xffffffffu, odd ? l[0] : l[1], 8));
#pragma unroll
  for (int off = 4; off > 0; off >>= 1)
    sum_add(hi, lo, __shfl_xor_sync(0xffffffffu, hi, off), __shfl_xor_sync(0xffffffffu, lo, off));
  return (double) hi + (double) lo;
}

// The launch's sums, and from them field = {Re Z, Im Z, |Z|, Re W, Im W, |W|,
// cos arg W, sin arg W} by the last block.  Returns whether this block is the
// last.
__device__ __forceinline__ bool field_finish(const FastParams &P, const FastBuffers &B, const FieldSum &f)
{
  const int lane = threadIdx.x & 31;
  const double mine = block_sum4(field_warp_sum(f));
  if (threadIdx.x < 32 && (lane & 7) == 0) B.field_partial[4 * blockIdx.x + (lane >> 3)] = mine;
  if (!last_block(B.ctrl)) return false;
  const double sum = block_sum_partials4(B.field_partial, gridDim.x);
  if (threadIdx.x >= 32) return true;
  // lanes 0, 8: Z, lanes 16, 24: W; their parts, moduli and arguments side by side
  const double part = sum / P.n, other = __shfl_xor_sync(0xffffffffu, part, 8);
  const double re = lane & 8 ? other : part, im = lane & 8 ? part : other;
  const double modulus = sqrt(re * re + im * im);
  const double dir = modulus > 0.0 ? part / modulus : (lane & 8 ? 0.0 : 1.0);  // arg 0 = 0, as std::arg
  const int at = lane >> 4;
  if ((lane & 7) == 0)
  {
    const int first = 3 * at;
    B.field[first + ((lane >> 3) & 1)] = (float) part;
    if (!(lane & 8)) B.field[first + 2] = (float) modulus;
    if (at) B.field[6 + ((lane >> 3) & 1)] = (float) dir;
  }
  return true;
}

// The field of a state that no step has left (an upload, a restored snapshot):
// the step's sums in the step's order, so a run goes on with the same bits.
__global__ void __launch_bounds__(kFieldThreads) fast_field_kernel(FastParams P, FastBuffers B)
{
  const int par = B.ctrl->parity;
  const uint4 *rec = par ? B.rec1 : B.rec0;
  const uint4 *aux = par ? B.aux1 : B.aux0;
  FieldSum f;
#pragma unroll 4
  for (int q = blockIdx.x * kFieldThreads + threadIdx.x; q < P.n; q += gridDim.x * kFieldThreads)
  {
    const uint2 cs = __ldg(reinterpret_cast<const uint2 *>(&rec[q].z));
    f.add(__uint_as_float(cs.x), __uint_as_float(cs.y), __uint_as_float(__ldg(&aux[q].w)));
  }
  field_finish(P, B, f);
}

// ---------------------------------------------------------------- order parameters of the context
//
// The observers' reduction over every particle of the context
// (BinaryObserverFirstOrder.cpp:125-142, BinaryObserverSecondOrder.cpp:121-138)
// from the 32-bit phases and the velocities, in FP64.

// e^{i 2 pi P / 2^32} = T1[P >> 21] T2[(P >> 10) & 2047] T3[P & 1023].
constexpr int kTurn1 = 2048, kTurn2 = 2048, kTurn3 = 1024, kTurnAll = kTurn1 + kTurn2 + kTurn3;
// Contexts of at least this many particles take e^{i phi} from the tables (80
// KB of shared memory a block, so at most two blocks an SM), smaller ones
// evaluate sincospi.  A whole order-parameter call, tables / sincospi: 31.3 /
// 31.9 us at 50,000 particles, 33.0 / 35.2 at 100,000, 66.6 / 105.2 at
// 1,000,000; below 50,000 the two do not differ.
constexpr int kTurnTableMin = 50000;

__global__ void fast_turn_table_kernel(double2 *__restrict__ table)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kTurnAll) return;
  double turns;  // exact: a power of two times an integer
  if (i < kTurn1) turns = (double) i / 2048.0;
  else if (i < kTurn1 + kTurn2) turns = (double) (i - kTurn1) / 4194304.0;
  else turns = (double) (i - kTurn1 - kTurn2) / 4294967296.0;
  double s, c;
  sincospi(2.0 * turns, &s, &c);
  table[i] = make_double2(c, s);
}

// FP64 instructions bound this kernel (4,194,304 particles: 8 a phase with the
// tables, 9 a velocity, 8.4 us for each of them at the measured 0.50 T/s).
// Through an FP64 copy of the state, sincos, square roots and divisions it was
// three kernels of 181 + 436 + 204 us; the whole call takes 146 us (181 with
// the velocities converted on the FP64 pipe).
template<bool TABLE>
__global__ void __launch_bounds__(256) fast_observe_kernel(FastParams P, FastBuffers B, const double2 *__restrict__ table,
                                                           double *__restrict__ partial, double *__restrict__ sums)
{
  extern __shared__ __align__(16) double2 turn[];
  if (TABLE)
  {
    for (int i = threadIdx.x; i < kTurnAll; i += blockDim.x) turn[i] = table[i];
    __syncthreads();
  }
  const uint4 *aux = B.ctrl->parity ? B.aux1 : B.aux0;
  buffers_now(B, B.ctrl->order_parity);
  double a[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll 2
  for (int q = blockIdx.x * blockDim.x + threadIdx.x; q < P.n; q += gridDim.x * blockDim.x)
  {
    const uint32_t ph = __ldg(&aux[q].z);
    const float2 v = P.model == 2 ? B.vel[q] : make_float2(0.f, 0.f);
    if (TABLE)
    {
      const double2 x = turn[ph >> 21], y = turn[kTurn1 + ((ph >> 10) & 2047u)];
      const double2 z = turn[kTurn1 + kTurn2 + (ph & 1023u)];
      const double yc = fma(y.x, z.x, -(y.y * z.y)), ys = fma(y.x, z.y, y.y * z.x);
      a[0] = fma(x.x, yc, a[0]);
      a[0] = fma(-x.y, ys, a[0]);
      a[1] = fma(x.y, yc, a[1]);
      a[1] = fma(x.x, ys, a[1]);
    } else
    {
      double sn, cs;
      sincospi((double) ph * 4.6566128730773926e-10, &sn, &cs);  // 2 / 2^32, exact
      a[0] += cs;
      a[1] += sn;
    }
    if (P.model == 2) add_direction(v, a[2], a[3]);
  }
  const int lane = threadIdx.x & 31;
  const double mine = block_sum4(warp_sum4(a));
  if (threadIdx.x < 32 && (lane & 7) == 0) partial[4 * blockIdx.x + (lane >> 3)] = mine;
  if (!last_block(B.ctrl)) return;
  const double sum = block_sum_partials4(partial, gridDim.x);
  if (threadIdx.x < 32 && (lane & 7) == 0) sums[lane >> 3] = sum;
}

// One SE or SRK step of the first-order model in the global field:
// k[3] = -xi omega + nu_i + sigma |Z| (sin(arg Z - phi) cos a - cos(arg Z - phi) sin a)
// and the complementary force as the reference computes it, whose last term
// takes sin(arg W - phi) (ParticleSystemFirstOrderPtr.cpp:213-219).
//
// A slot is its original index.  The thread that moves a particle adds its new
// direction to the sums, and the last block leaves the field for the next step
// and ends this one: one launch and one pass over the state.  A step, both
// steppers, with field, step and control kernels before and now: 20.3 -> 8.3 us
// at N = 1,000, 24.6 -> 10.3 at 100,000, 39.5 -> 18.6 to 19.7 at 999,983.
// Small sizes are the launch and the last block's FP64 chain; large ones move
// 68 bytes a particle (the buffers fit the L2: 3.6 TB/s) beside the noise and
// two sine pairs.  Two blocks an SM leave the fewest partials and room for the
// next particle's loads in registers (three to five: 2 to 6 us slower).
template<int STEPPER>
__global__ void __launch_bounds__(kFieldThreads, 2) fast_global_step_kernel(FastParams P, FastBuffers B)
{
  FastControl *ctrl = B.ctrl;
  const int par = ctrl->parity;
  const unsigned long long step = ctrl->step;
  buffers_now(B, ctrl->order_parity);
  const uint4 *rin = par ? B.rec1 : B.rec0;
  const uint4 *ain = par ? B.aux1 : B.aux0;
  uint4 *rout = par ? B.rec0 : B.rec1;
  uint4 *aout = par ? B.aux0 : B.aux1;
  const float zr = B.field[0], zi = B.field[1], az = B.field[2];
  const float wr = B.field[3], wim = B.field[4], aw = B.field[5];
  const float cw = B.field[6], sw = B.field[7];
  FieldSum sums;
  int err = 0;
  const int stride = gridDim.x * kFieldThreads;
  int q = blockIdx.x * kFieldThreads + threadIdx.x;
  uint4 rn = make_uint4(0, 0, 0, 0), an = rn;
  float nun = 0.0f;
  if (q < P.n)
  {
    rn = rin[q];
    an = ain[q];
    nun = B.nu[q];
  }
  for (; q < P.n; q += stride)
  {
    const uint4 ri = rn, ai = an;
    const float nu = nun;
    if (q + stride < P.n)
    {
      rn = rin[q + stride];
      an = ain[q + stride];
      nun = B.nu[q + stride];
    }
    float z[6];
    draw_noise<1, STEPPER>(P, step, (unsigned) q, z);
    const float cphi = __uint_as_float(ri.z), sphi = __uint_as_float(ri.w), wi = __uint_as_float(ai.w);
    const float SZ = fmaf(zi, cphi, -__fmul_rn(zr, sphi));  // |Z| sin(arg Z - phi)
    const float KZ = fmaf(zr, cphi, __fmul_rn(zi, sphi));   // |Z| cos(arg Z - phi)
    const float f_w = fmaf(-P.xi_phi, wi, __fadd_rn(nu, __fmul_rn(P.sigma, fmaf(P.ca, SZ, -__fmul_rn(P.sa, KZ)))));
    float C = 0.0f;
    if (STEPPER == 2)
    {
      const float KW = fmaf(wr, cphi, __fmul_rn(wim, sphi));   // |W| cos(arg W - phi)
      const float sWp = fmaf(sw, cphi, -__fmul_rn(cw, sphi));  // sin(arg W - phi)
      const float first = fmaf(P.ca, KW, __fmul_rn(P.sa, __fmul_rn(aw, sWp)));
      const float second = __fmul_rn(wi, fmaf(P.ca, KZ, __fmul_rn(P.sa, __fmul_rn(az, sWp))));
      C = __fmul_rn(P.sigma, __fsub_rn(first, second));
    }
    uint4 r, a;
    advance_particle<1, STEPPER>(P, B, q, ri, ai, make_float2(0.f, 0.f), f_w, C, z, r, a, err);
    rout[q] = r;
    aout[q] = a;
    sums.add(__uint_as_float(r.z), __uint_as_float(r.w), __uint_as_float(a.w));
  }
  if (__any_sync(0xffffffffu, err) && (threadIdx.x & 31) == 0) atomicOr(&ctrl->error, 1);
  if (field_finish(P, B, sums)) end_step(ctrl, B.sysctl, B.sys, 1, P.always_rebuild, 0, 0, 1);
}

__global__ void fast_set_frequencies_kernel(const double *__restrict__ freqs, int n, float *__restrict__ nu)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) nu[i] = (float) freqs[i];
}

// ---------------------------------------------------------------- host side

static int blocks_for(long n, int tb)
{
  return (int) ((n + tb - 1) / tb);
}

static bool has_cells(int kind)
{
  return kind == KIND_CELLS || kind == KIND_VERLET;
}

static FastBuffers buffers(spss_ctx *ctx)
{
  FastPath *f = ctx->fast;
  FastBuffers B;
  B.rec0 = f->rec[0].ptr;
  B.rec1 = f->rec[1].ptr;
  B.aux0 = f->aux[0].ptr;
  B.aux1 = f->aux[1].ptr;
  B.vel = f->vel.ptr;
  B.vel_tmp = f->vel_tmp.ptr;
  B.pid = f->pid.ptr;
  B.pid_tmp = f->pid_tmp.ptr;
  B.inv = f->inv.ptr;
  B.img = f->img.ptr;
  B.turns = f->turns.ptr;
  B.cell_of = f->cell_of.ptr;
  B.cell_sorted = f->cell_sorted.ptr;
  B.cell_off = f->binner.offsets.ptr;
  B.cell_off_w = f->binner.offsets.ptr;
  B.order = f->binner.members.ptr;
  B.cell_count = f->binner.count.ptr;
  B.cell_slot = f->binner.slot.ptr;
  B.vl = f->vl.ptr;
  B.vl_cnt = f->vl_cnt.ptr;
  B.sys = f->sys.ptr;
  B.sys_of = f->sys_of.ptr;
  B.sysctl = f->sysctl.ptr;
  B.nu = f->nu.ptr;
  B.field = f->field.ptr;
  B.field_partial = f->field_partial.ptr;
  B.ctrl = f->ctrl;
  return B;
}

// Table entry of one system: its parameters in the FP32 / fixed-point units
// of the kernels.
static SysParams system_params(const spss_params &p, int index, int first, int nc, int cell0, double r_min,
                               double r_max)
{
  SysParams S;
  std::memset(&S, 0, sizeof(S));
  S.n = p.n;
  S.first = first;
  S.nc = nc;
  S.cell0 = cell0;
  S.index = index;
  S.replica = (int) p.replica;
  S.v0 = (float) p.v0;
  S.xi = (float) p.xi;
  S.xi_r = (float) p.xi_r;
  // first order: the torque friction is xi; second order: xi_phi
  S.xi_phi = (float) (p.model == 1 ? p.xi : p.xi_phi);
  S.sigma = (float) p.sigma;
  S.ca = (float) std::cos(p.alpha);
  S.sa = (float) std::sin(p.alpha);
  const double rho2 = p.rho * p.rho;
  S.rho2_d = rho2;
  // FP32 pair distances are squared differences of the 32-bit position words,
  // i.e. in units of 2^-64 of the box area
  const double area = 18446744073709551616.0;
  S.rho2_f = (float) (rho2 * area);
  // A difference of the 32-bit high words is off by less than 2^-32 of the box,
  // so |d2_f - d2| <= 2 (|dx| + |dy|) 2^-32 + 2 * 2^-64 + 5 d2 2^-24 (conversions,
  // square, fma, rounding of rho2_f), with |dx| + |dy| <= 2 rho near r = rho;
  // doubled.  (A term 2^-32 in place of 2 * 2^-64 had made the band 300 times
  // wider at N = 4,194,304: 1.2 % of the particles met it every step.)
  const double word = 2.3283064365386963e-10;  // 2^-32
  S.band_f = (float) (area * 2.0 * (4.0 * p.rho * word + 2.0 * word * word + 5.0 * rho2 * 5.9604644775390625e-8));
  const double rmax2 = r_max * r_max;
  S.rmax2_f = (float) (area * (rmax2 + 2.0 * (4.0 * r_max * 2.3283064365386963e-10 + 4.0 * rmax2 * 5.9604644775390625e-8)));
  S.half_skin = 0.5 * (r_max - r_min);
  S.b_r = (float) std::sqrt(2.0 * p.D_r);
  S.b_phi = (float) std::sqrt(2.0 * p.D_phi);
  return S;
}

static FastParams params(spss_ctx *ctx, double dt)
{
  const spss_params &p = ctx->p;
  FastPath *f = ctx->fast;
  const SysParams &S = f->h_sys[0];
  FastParams P;
  std::memset(&P, 0, sizeof(P));
  P.n = p.n;
  P.cap = f->cap;
  P.model = p.model;
  P.always_rebuild = f->kind == KIND_CELLS ? 1 : 0;
  P.selective = f->nsys > 1 && f->kind == KIND_VERLET ? 1 : 0;
  P.nsys = f->nsys;
  // system 0 (kernels that serve several systems read theirs from the table)
  P.nc = S.nc;
  P.first = S.first;
  P.sub_n = S.n;
  P.cell0 = S.cell0;
  P.v0 = S.v0;
  P.xi = S.xi;
  P.xi_r = S.xi_r;
  P.xi_phi = S.xi_phi;
  P.sigma = S.sigma;
  P.ca = S.ca;
  P.sa = S.sa;
  P.rho2_f = S.rho2_f;
  P.band_f = S.band_f;
  P.rho2_d = S.rho2_d;
  P.b_r = S.b_r;
  P.b_phi = S.b_phi;
  P.dt = (float) dt;
  P.sqdt = (float) std::sqrt(dt);
  P.half_dt2 = (float) (0.5 * dt * dt);
  P.half_dt15 = (float) (0.5 * std::pow(dt, 1.5));
  P.inv_sqrt3 = (float) (1.0 / std::sqrt(3.0));
  P.seed = p.seed;
  philox_round_keys(p.seed, P.kx, P.ky);
  P.replica = (uint32_t) S.replica;
  return P;
}

int fast_create(spss_ctx *ctx)
{
  FastPath *f = new FastPath();
  ctx->fast = f;
  const spss_params &p = ctx->p;
  const int n = p.n;
  std::vector<spss_params> systems = ctx->systems;
  if (systems.empty()) systems.push_back(p);
  f->nsys = (int) systems.size();
  int kind = -1;
  double lam_max = 0.0;
  int first = 0, cell0 = 0;
  for (int r = 0; r < f->nsys; ++r)
  {
    const spss_params &q = systems[r];
    double r_min, r_max;
    int nc, nc_verlet;
    derive_lists(q, r_min, r_max, nc, nc_verlet);
    int k, grid;
    switch (variant_for_params(q, q.variant))
    {
      case SPSS_VARIANT_ALL_PAIRS:
        k = KIND_ALL_PAIRS;
        grid = 1;
        break;
      case SPSS_VARIANT_LINKED_LIST:
        k = KIND_CELLS;
        grid = nc;
        break;
      case SPSS_VARIANT_VERLET:
        // O(N^2) list build = every pair within r_max: cells no smaller than r_max.  With fewer
        // than three such cells per side (r_max > 1/3: the reference's first-order dispatch for
        // 0.25 < rho <= 0.5, ParticleSystemFirstOrder.cpp:96-111) a list holds a third of the
        // system or more and the stencil would visit cells twice: every pair is evaluated each
        // step instead, the same neighbours within rho, with the list trigger kept.
        grid = std::max(1, (int) (1.0 / r_max));
        k = grid < 3 ? KIND_ALL_PAIRS : KIND_VERLET;
        if (grid < 3)
        {
          grid = 1;
          f->trigger_only = true;
        }
        break;
      case SPSS_VARIANT_LINKED_LIST_VERLET:
        k = KIND_VERLET;
        grid = nc_verlet;
        break;
      case SPSS_VARIANT_GLOBAL_FIELD:
        // the reference's global field belongs to the first-order model; one system
        if (q.model != 1 || systems.size() != 1) return SPSS_ERR_NOT_SUPPORTED;
        k = KIND_GLOBAL;
        grid = 1;
        break;
      default:
        return SPSS_ERR_NOT_SUPPORTED;
    }
    if (kind >= 0 && k != kind) return SPSS_ERR_NOT_SUPPORTED;  // one list kind per context
    kind = k;
    if ((long) cell0 + (long) grid * grid > 0x7fffffffL) return SPSS_ERR_SIZE;
    f->h_sys.push_back(system_params(q, r, first, grid, cell0, r_min, r_max));
    first += q.n;
    cell0 += grid * grid;
    lam_max = std::max(lam_max, M_PI * r_max * r_max * q.n);
  }
  if (first != n) return SPSS_ERR_INVALID_ARGUMENT;
  f->kind = kind;
  f->total_cells = cell0;
  f->small_systems = kind == KIND_VERLET && f->nsys > 1;
  for (const SysParams &S : f->h_sys)
    if (S.n > kSystemSlots || S.nc * S.nc > kSystemCells) f->small_systems = false;
  if (kind == KIND_GLOBAL)
  {
    SPSS_TRY(f->nu.reserve((size_t) n));
    SPSS_TRY(f->field.reserve(8));
    SPSS_TRY(f->field_partial.reserve(4 * kFieldBlocks));
    SPSS_CUDA_TRY(cudaMemsetAsync(f->nu.ptr, 0, sizeof(float) * n, ctx->stream));
  }
  if (f->kind == KIND_VERLET || f->trigger_only) ctx->uses_verlet_list = 1;
  for (int b = 0; b < 2; ++b)
  {
    SPSS_TRY(f->rec[b].reserve(n));
    SPSS_TRY(f->aux[b].reserve(n));
  }
  SPSS_TRY(f->vel.reserve(n));
  SPSS_TRY(f->vel_tmp.reserve(n));
  SPSS_TRY(f->pid.reserve(n));
  SPSS_TRY(f->pid_tmp.reserve(n));
  SPSS_TRY(f->inv.reserve(n));
  SPSS_TRY(f->img.reserve(n));
  SPSS_TRY(f->turns.reserve(n));
  SPSS_TRY(f->cell_of.reserve(n));
  SPSS_TRY(f->cell_sorted.reserve(n));
  SPSS_TRY(f->vl_cnt.reserve(n));
  SPSS_TRY(f->sys.reserve((size_t) f->nsys));
  SPSS_TRY(f->sysctl.reserve((size_t) f->nsys));
  SPSS_TRY(f->sys_of.reserve((size_t) n));
  {
    std::vector<int2> items;
    std::vector<int> first_item;
    for (const SysParams &S : f->h_sys)
    {
      first_item.push_back((int) items.size());
      for (long b = 0; b < S.n; b += kOrderChunk) items.push_back(make_int2(S.index, (int) (S.first + b)));
    }
    first_item.push_back((int) items.size());
    f->order_chunks = (int) items.size();
    f->order_grid = std::min(f->order_chunks, 4 * 152);
    SPSS_TRY(f->order_partial.reserve((size_t) f->order_chunks));
    SPSS_TRY(f->order_items.reserve(items.size()));
    SPSS_TRY(f->order_first.reserve(first_item.size()));
    SPSS_CUDA_TRY(cudaMemcpyAsync(f->order_items.ptr, items.data(), sizeof(int2) * items.size(),
                                  cudaMemcpyHostToDevice, ctx->stream));
    SPSS_CUDA_TRY(cudaMemcpyAsync(f->order_first.ptr, first_item.data(), sizeof(int) * first_item.size(),
                                  cudaMemcpyHostToDevice, ctx->stream));
    SPSS_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
    SPSS_TRY(f->order_out.reserve((size_t) f->nsys * 4));
    SPSS_TRY(f->stats.reserve((size_t) f->nsys * 5));
    SPSS_CUDA_TRY(cudaMemsetAsync(f->stats.ptr, 0, sizeof(double) * 5 * f->nsys, ctx->stream));
  }
  if (f->kind == KIND_VERLET)
  {
    // mean list length: pi r_max^2 n (unit box); room for six standard deviations
    f->cap = std::max(16, ((int) std::ceil(lam_max + 6.0 * std::sqrt(lam_max) + 8.0) + 3) & ~3);
  }
  {
    std::vector<int> sys_of((size_t) n);
    for (int r = 0; r < f->nsys; ++r)
      std::fill(sys_of.begin() + f->h_sys[r].first, sys_of.begin() + f->h_sys[r].first + f->h_sys[r].n, r);
    SPSS_CUDA_TRY(cudaMemcpyAsync(f->sys_of.ptr, sys_of.data(), sizeof(int) * n, cudaMemcpyHostToDevice, ctx->stream));
    SPSS_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  }
  SPSS_CUDA_TRY(cudaMemsetAsync(f->sysctl.ptr, 0, sizeof(SysControl) * f->nsys, ctx->stream));
  SPSS_CUDA_TRY(cudaMemcpyAsync(f->sys.ptr, f->h_sys.data(), sizeof(SysParams) * f->nsys, cudaMemcpyHostToDevice,
                                ctx->stream));
  SPSS_CUDA_TRY(cudaMalloc((void **) &f->ctrl, sizeof(FastControl)));
  SPSS_CUDA_TRY(cudaMallocHost((void **) &f->h_ctrl, sizeof(FastControl)));
  std::memset(f->h_ctrl, 0, sizeof(FastControl));
  f->h_ctrl->rebuild = 1;
  f->h_ctrl->uses_verlet = f->kind == KIND_VERLET;
  SPSS_CUDA_TRY(cudaMemcpyAsync(f->ctrl, f->h_ctrl, sizeof(FastControl), cudaMemcpyHostToDevice, ctx->stream));
  SPSS_CUDA_TRY(cudaMemsetAsync(f->vel.ptr, 0, sizeof(float2) * n, ctx->stream));
  // a download before the first state gathers slot 0; empty lists until the first build, as the reference's
  SPSS_CUDA_TRY(cudaMemsetAsync(f->inv.ptr, 0, sizeof(unsigned) * n, ctx->stream));
  SPSS_CUDA_TRY(cudaMemsetAsync(f->vl_cnt.ptr, 0, sizeof(int) * n, ctx->stream));
  if (has_cells(f->kind)) SPSS_TRY(f->binner.prepare(n, f->total_cells, ctx->stream));
  if (f->kind == KIND_VERLET) SPSS_TRY(f->vl.reserve((size_t) f->cap * (((size_t) n + 31) / 32 * 32)));
  SPSS_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  return SPSS_OK;
}

void fast_destroy(spss_ctx *ctx)
{
  FastPath *f = ctx->fast;
  if (!f) return;
  for (auto &g : f->graphs) g.second.release();
  for (int b = 0; b < 2; ++b)
  {
    f->rec[b].release();
    f->aux[b].release();
  }
  f->vel.release();
  f->vel_tmp.release();
  f->pid.release();
  f->pid_tmp.release();
  f->inv.release();
  f->img.release();
  f->turns.release();
  f->cell_of.release();
  f->cell_sorted.release();
  f->vl.release();
  f->vl_cnt.release();
  f->sys.release();
  f->sys_of.release();
  f->sysctl.release();
  f->nu.release();
  f->field.release();
  f->field_partial.release();
  f->turn_table.release();
  f->observe_partial.release();
  if (f->h_order) cudaFreeHost(f->h_order);
  f->order_partial.release();
  f->order_items.release();
  f->order_first.release();
  f->order_out.release();
  f->stats.release();
  f->snap.release();
  f->binner.release();
  if (f->ctrl) cudaFree(f->ctrl);
  if (f->h_ctrl) cudaFreeHost(f->h_ctrl);
  delete f;
  ctx->fast = nullptr;
}

// Cell binning, slot re-sort and list build (Verlet lists), as one stream
// sequence; kinds without lists only clear the flag.
static int launch_rebuild(spss_ctx *ctx, const FastParams &P)
{
  FastPath *f = ctx->fast;
  const FastBuffers B = buffers(ctx);
  const int n = P.n;
  const bool lists = f->kind == KIND_VERLET;
  if (lists && f->small_systems)
  {
    fast_system_rebuild_kernel<<<f->nsys, kSystemThreads, 0, ctx->stream>>>(P, B);
    ++ctx->launches;
    SPSS_TRY(check_launch("fast_system_rebuild_kernel"));
    fast_verlet_build_kernel<<<blocks_for(n, kBuildThreads), kBuildThreads, 0, ctx->stream>>>(P, B, 1);
    ++ctx->launches;
    return check_launch("fast_verlet_build_kernel");
  }
  if (lists)
  {
    fast_cells_kernel<<<blocks_for(n, kTB), kTB, 0, ctx->stream>>>(P, B);
    ++ctx->launches;
    SPSS_TRY(check_launch("fast_cells_kernel"));
    SPSS_TRY(f->binner.place(f->cell_of.ptr, n, ctx->stream, ctx->launches));
    fast_permute_kernel<false><<<blocks_for(n, kTB), kTB, 0, ctx->stream>>>(P, B);
    ++ctx->launches;
    SPSS_TRY(check_launch("fast_permute_kernel"));
    if (P.selective)
    {
      fast_copyback_kernel<<<blocks_for(n, kTB), kTB, 0, ctx->stream>>>(P, B);
      ++ctx->launches;
      SPSS_TRY(check_launch("fast_copyback_kernel"));
    }
  }
  fast_after_permute_kernel<<<1, 1, 0, ctx->stream>>>(f->ctrl, (int) lists);
  ++ctx->launches;
  SPSS_TRY(check_launch("fast_after_permute_kernel"));
  if (lists)
  {
    fast_verlet_build_kernel<<<blocks_for(n, kBuildThreads), kBuildThreads, 0, ctx->stream>>>(P, B, 0);
    ++ctx->launches;
    SPSS_TRY(check_launch("fast_verlet_build_kernel"));
  }
  fast_after_rebuild_kernel<<<1, 256, 0, ctx->stream>>>(f->ctrl, f->sysctl.ptr, f->nsys);
  ++ctx->launches;
  return check_launch("fast_after_rebuild_kernel");
}

// Cell ids and counts of the current slots, where the last cell-list step did
// not leave them (a new state, a restored snapshot).
static int ensure_cells(spss_ctx *ctx, const FastParams &P)
{
  FastPath *f = ctx->fast;
  if (f->h_ctrl->cells_fresh) return SPSS_OK;
  SPSS_CUDA_TRY(cudaMemsetAsync(f->binner.count.ptr, 0, sizeof(int) * f->binner.count.count, ctx->stream));
  fast_cells_kernel<<<blocks_for(P.n, kTB), kTB, 0, ctx->stream>>>(P, buffers(ctx));
  ++ctx->launches;
  f->h_ctrl->cells_fresh = 1;
  return check_launch("fast_cells_kernel");
}

static int field_blocks(int n)
{
  return std::min(kFieldBlocks, blocks_for(n, kFieldThreads));
}

// The global field of the current state, where no step has left it.
static int ensure_field(spss_ctx *ctx, const FastParams &P)
{
  FastPath *f = ctx->fast;
  if (f->kind != KIND_GLOBAL || f->h_ctrl->cells_fresh) return SPSS_OK;
  fast_field_kernel<<<field_blocks(P.n), kFieldThreads, 0, ctx->stream>>>(P, buffers(ctx));
  ++ctx->launches;
  f->h_ctrl->cells_fresh = 1;
  return check_launch("fast_field_kernel");
}

template<int MODEL, int STEPPER>
static void launch_cell_steps(spss_ctx *ctx, const FastParams &P, const FastBuffers &B, int fresh, bool chained)
{
  const int blocks = blocks_for(P.n, kCellThreads);
  if (P.nsys > 1)
    launch_chained(chained, fast_cell_step_kernel<MODEL, STEPPER, true>, blocks, kCellThreads, 0, ctx->stream, P, B, fresh);
  else
    launch_chained(chained, fast_cell_step_kernel<MODEL, STEPPER, false>, blocks, kCellThreads, 0, ctx->stream, P, B, fresh);
}

static int launch_cell_kernel(spss_ctx *ctx, int stepper, const FastParams &P, int fresh, bool chained)
{
  const FastBuffers B = buffers(ctx);
  if (ctx->timing) SPSS_CUDA_TRY(cudaEventRecord(ctx->ev0, ctx->stream));
  if (ctx->p.model == 1)
  {
    if (stepper == SPSS_STEPPER_STOCHASTIC_EULER) launch_cell_steps<1, 1>(ctx, P, B, fresh, chained);
    else launch_cell_steps<1, 2>(ctx, P, B, fresh, chained);
  } else
  {
    if (stepper == SPSS_STEPPER_STOCHASTIC_EULER) launch_cell_steps<2, 1>(ctx, P, B, fresh, chained);
    else launch_cell_steps<2, 2>(ctx, P, B, fresh, chained);
  }
  ++ctx->launches;
  SPSS_TRY(check_launch("fast_cell_step_kernel"));
  if (ctx->timing) SPSS_CUDA_TRY(cudaEventRecord(ctx->ev1, ctx->stream));
  return SPSS_OK;
}

// A cell-list step from the counts the last one left: offsets (which also count
// the step), members, slot re-sort, pair sums and update.  `chained`: captured
// as a programmatic-dependent chain (each kernel begins with pdl_enter).
static int launch_cells_step(spss_ctx *ctx, int stepper, const FastParams &P, bool chained)
{
  FastPath *f = ctx->fast;
  SPSS_TRY(f->binner.place(f->cell_of.ptr, P.n, ctx->stream, ctx->launches, chained, f->ctrl));
  SPSS_CUDA_TRY(launch_chained(chained, fast_permute_kernel<true>, blocks_for(P.n, kTB), kTB, 0, ctx->stream, P,
                               buffers(ctx)));
  ++ctx->launches;
  SPSS_TRY(check_launch("fast_permute_kernel"));
  return launch_cell_kernel(ctx, stepper, P, 1, chained);
}

template<int MODEL, int STEPPER>
static void launch_tiles(spss_ctx *ctx, const FastParams &P, const FastBuffers &B, bool chained)
{
  const int blocks = blocks_for(P.n, kTileThreads);
  if (P.nsys > 1)
    launch_chained(chained, fast_tile_kernel<MODEL, STEPPER, true>, blocks, kTileThreads, 0, ctx->stream, P, B);
  else
    launch_chained(chained, fast_tile_kernel<MODEL, STEPPER, false>, blocks, kTileThreads, 0, ctx->stream, P, B);
}

template<int MODEL, int STEPPER>
static void launch_step_kind(spss_ctx *ctx, const FastParams &P, const FastBuffers &B, bool chained)
{
  if (ctx->fast->kind == KIND_GLOBAL)
  {
    if (MODEL == 1)
    {
      fast_global_step_kernel<STEPPER><<<field_blocks(P.n), kFieldThreads, 0, ctx->stream>>>(P, B);
    }
  } else if (ctx->fast->kind == KIND_ALL_PAIRS)
  {
    const int blocks = blocks_for(P.n, 32);
    if (P.nsys > 1) fast_allpairs_kernel<MODEL, STEPPER, true><<<blocks, 32 * kPairWarps, 0, ctx->stream>>>(P, B);
    else fast_allpairs_kernel<MODEL, STEPPER, false><<<blocks, 32 * kPairWarps, 0, ctx->stream>>>(P, B);
  } else
  {
    launch_tiles<MODEL, STEPPER>(ctx, P, B, chained);
  }
}

// One block: a system a thread, whose FP64 chain (square root, sum, comparison)
// is all the kernel does (1,024 systems: 9.5 us with 256 threads, 6.6 us with 1,024).
static int control_threads(int nsys)
{
  return std::min(1024, (nsys + 31) / 32 * 32);
}

static int launch_control(spss_ctx *ctx, const FastParams &P, int cells_written)
{
  FastPath *f = ctx->fast;
  SPSS_CUDA_TRY(launch_chained(true, fast_control_kernel<false>, 1, control_threads(f->nsys), 0, ctx->stream, f->ctrl,
                               f->sysctl.ptr, (const SysParams *) f->sys.ptr, f->nsys, P.always_rebuild,
                               (int) (f->kind == KIND_VERLET || f->trigger_only), P.selective, cells_written,
                               (cudaGraphExec_t) nullptr));
  ++ctx->launches;
  return check_launch("fast_control_kernel");
}

// `chained`: the launch before it in the stream is a kernel.
static int launch_step(spss_ctx *ctx, int stepper, const FastParams &P, cudaGraphExec_t rebuild_exec = nullptr,
                       bool chained = false)
{
  const FastBuffers B = buffers(ctx);
  if (ctx->timing) SPSS_CUDA_TRY(cudaEventRecord(ctx->ev0, ctx->stream));
  if (ctx->p.model == 1)
  {
    if (stepper == SPSS_STEPPER_STOCHASTIC_EULER) launch_step_kind<1, 1>(ctx, P, B, chained);
    else launch_step_kind<1, 2>(ctx, P, B, chained);
  } else
  {
    if (stepper == SPSS_STEPPER_STOCHASTIC_EULER) launch_step_kind<2, 1>(ctx, P, B, chained);
    else launch_step_kind<2, 2>(ctx, P, B, chained);
  }
  ++ctx->launches;
  SPSS_TRY(check_launch("step kernel"));
  if (ctx->timing) SPSS_CUDA_TRY(cudaEventRecord(ctx->ev1, ctx->stream));
  FastPath *f = ctx->fast;
  if (f->kind == KIND_GLOBAL) return SPSS_OK;  // its step kernel ends the step
  if (rebuild_exec)
    SPSS_CUDA_TRY(launch_chained(true, fast_control_kernel<true>, 1, control_threads(f->nsys), 0, ctx->stream, f->ctrl,
                                 f->sysctl.ptr, (const SysParams *) f->sys.ptr, f->nsys, P.always_rebuild,
                                 (int) (f->kind == KIND_VERLET || f->trigger_only), P.selective, 0, rebuild_exec));
  else
    SPSS_TRY(launch_control(ctx, P, 0));
  if (rebuild_exec) ++ctx->launches;
  return check_launch("fast_control_kernel");
}

// Order parameters of every system; `gated`: only after a sampling step, and
// then also added to the running averages.
static int launch_sampling(spss_ctx *ctx, const FastParams &P, int gated)
{
  FastPath *f = ctx->fast;
  const FastBuffers B = buffers(ctx);
  fast_order_partials_kernel<<<f->order_grid, kOrderThreads, 0, ctx->stream>>>(P, B, f->order_partial.ptr,
                                                                       f->order_items.ptr, f->order_chunks, gated);
  ++ctx->launches;
  SPSS_TRY(check_launch("fast_order_partials_kernel"));
  fast_order_finish_kernel<<<blocks_for(f->nsys, 32), 32, 0, ctx->stream>>>(
      P, B, f->order_partial.ptr, f->order_first.ptr, f->order_out.ptr, f->stats.ptr, gated);
  ++ctx->launches;
  return check_launch("fast_order_finish_kernel");
}

// The reference's should_update_lists after a step: set by the trigger until
// the next evaluation rebuilds.  A graph step performs its rebuild at once
// (tail launch), so the flag reads from the trigger of the last step as well.
static int reported_list_flag(const FastControl *c)
{
  return (c->rebuild || c->triggered) ? 1 : 0;
}

// Waits for the stream, then takes over the control block's host copy.
static int adopt_control(spss_ctx *ctx)
{
  FastPath *f = ctx->fast;
  SPSS_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  ctx->step_counter = f->h_ctrl->step;
  ctx->accumulated_displacement = f->h_ctrl->acc;
  ctx->should_update_lists = reported_list_flag(f->h_ctrl);
  if (f->h_ctrl->error & ~1) return SPSS_ERR_CUDA;  // a device launch failed
  if (f->h_ctrl->error) return SPSS_ERR_NONFINITE;
  return SPSS_OK;
}

static int sync_control(spss_ctx *ctx)
{
  FastPath *f = ctx->fast;
  SPSS_CUDA_TRY(cudaMemcpyAsync(f->h_ctrl, f->ctrl, sizeof(FastControl), cudaMemcpyDeviceToHost, ctx->stream));
  return adopt_control(ctx);
}

// The host-side step counter and list flag (spss_set_step_counter,
// spss_set_should_update_lists) win over the device copy.
static int push_host_control(spss_ctx *ctx)
{
  FastPath *f = ctx->fast;
  if (f->h_ctrl->step == ctx->step_counter && reported_list_flag(f->h_ctrl) == ctx->should_update_lists)
    return SPSS_OK;
  if (reported_list_flag(f->h_ctrl) != ctx->should_update_lists)
  {
    f->h_ctrl->rebuild = ctx->should_update_lists ? REBUILD_ALL : REBUILD_NONE;
    f->h_ctrl->triggered = 0;
  }
  f->h_ctrl->step = ctx->step_counter;
  SPSS_CUDA_TRY(cudaMemcpyAsync(f->ctrl, f->h_ctrl, sizeof(FastControl), cudaMemcpyHostToDevice, ctx->stream));
  return SPSS_OK;
}

int fast_set_state(spss_ctx *ctx, const double *d_aos)
{
  FastPath *f = ctx->fast;
  fast_upload_kernel<<<blocks_for(ctx->p.n, kTB), kTB, sizeof(double) * kTB * ctx->s, ctx->stream>>>(
      d_aos, ctx->p.n, ctx->s, ctx->p.model, f->perm_valid ? 1 : 0, buffers(ctx));
  ++ctx->launches;
  SPSS_TRY(check_launch("fast_upload_kernel"));
  f->h_ctrl->cells_fresh = 0;  // as the kernel leaves the device's
  // the last step's trigger fired and a graph step already rebuilt the lists
  // from the positions before this upload: the reference rebuilds from the
  // state it is given next, so rebuild again before the next step
  if (f->h_ctrl->triggered && !f->h_ctrl->rebuild)
  {
    f->h_ctrl->rebuild = REBUILD_ALL;
    SPSS_CUDA_TRY(cudaMemcpyAsync(&f->ctrl->rebuild, &f->h_ctrl->rebuild, sizeof(int), cudaMemcpyHostToDevice,
                                  ctx->stream));
  }
  f->perm_valid = true;
  f->have_state = true;
  return SPSS_OK;
}

static int launch_download(spss_ctx *ctx, double *d_aos, FastControl *host_ctrl)
{
  SPSS_CUDA_TRY(launch_chained(host_ctrl != nullptr, fast_download_kernel, blocks_for(ctx->p.n, kTB), kTB,
                               sizeof(double) * kTB * ctx->s, ctx->stream, d_aos, ctx->p.n, ctx->s, ctx->p.model,
                               buffers(ctx), host_ctrl));
  ++ctx->launches;
  return check_launch("fast_download_kernel");
}

int fast_get_state(spss_ctx *ctx, double *d_aos)
{
  return launch_download(ctx, d_aos, nullptr);
}

// Room for longer lists once some were too long (clusters outgrow the capacity
// estimated for the mean density, and a particle whose list did not fit scans
// its stencil every step): a quarter more than the longest seen.  The lists in
// use move as they are, and the next rebuild fills the larger ones, so no result
// depends on when this happens.  Memory is taken only while it is plentiful; a
// failed allocation leaves things as they were.
constexpr int kListCapMax = 512;

static int grow_lists(spss_ctx *ctx)
{
  FastPath *f = ctx->fast;
  if (f->kind != KIND_VERLET || f->h_ctrl->overflow <= f->cap) return SPSS_OK;
  const int cap = std::min(kListCapMax, (f->h_ctrl->overflow + f->h_ctrl->overflow / 4 + 3) & ~3);
  if (cap <= f->cap) return SPSS_OK;
  const size_t warps = ((size_t) ctx->p.n + 31) / 32, want = warps * 32 * cap;
  size_t free_bytes = 0, total_bytes = 0;
  SPSS_CUDA_TRY(cudaMemGetInfo(&free_bytes, &total_bytes));
  if (want * sizeof(short) > free_bytes / 4) return SPSS_OK;
  DeviceArray<short> larger;
  if (larger.reserve(want) != SPSS_OK) return SPSS_OK;
  const size_t pitch = 32 * sizeof(short) * cap, old_pitch = 32 * sizeof(short) * f->cap;
  SPSS_CUDA_TRY(cudaMemcpy2DAsync(larger.ptr, pitch, f->vl.ptr, old_pitch, old_pitch, warps, cudaMemcpyDeviceToDevice,
                                  ctx->stream));
  SPSS_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  f->vl.release();
  f->vl = larger;
  f->cap = cap;
  for (auto &g : f->graphs) g.second.release();
  f->graphs.clear();
  return SPSS_OK;
}

// The launches of one step by themselves (no graph).
static int launch_single_step(spss_ctx *ctx, int stepper, double dt)
{
  FastPath *f = ctx->fast;
  if (!f->have_state) return SPSS_ERR_INVALID_ARGUMENT;
  if (stepper == SPSS_STEPPER_RK4) return SPSS_ERR_NOT_SUPPORTED;
  SPSS_TRY(grow_lists(ctx));
  const FastParams P = params(ctx, dt);
  SPSS_TRY(push_host_control(ctx));
  if (f->kind == KIND_CELLS)
  {
    if (f->h_ctrl->rebuild || !f->h_ctrl->rebuilds)
    {
      SPSS_TRY(ensure_cells(ctx, P));
      SPSS_TRY(launch_cells_step(ctx, stepper, P, !ctx->timing));
    } else
    {
      // the caller asked for the lists to stay (spss_set_should_update_lists):
      // a step on the last binning (there was one), which counts the cells anew
      SPSS_CUDA_TRY(cudaMemsetAsync(f->binner.count.ptr, 0, sizeof(int) * f->binner.count.count, ctx->stream));
      SPSS_TRY(launch_cell_kernel(ctx, stepper, P, 0, false));
      SPSS_TRY(launch_control(ctx, P, 1));
    }
  } else
  {
    if (f->h_ctrl->rebuild) SPSS_TRY(launch_rebuild(ctx, P));
    SPSS_TRY(ensure_field(ctx, P));
    SPSS_TRY(launch_step(ctx, stepper, P, nullptr, !ctx->timing));
  }
  return SPSS_OK;
}

static int take_timing(spss_ctx *ctx)
{
  if (!ctx->timing) return SPSS_OK;
  float ms = 0.0f;
  SPSS_CUDA_TRY(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
  ctx->timing_ms += ms;
  ctx->timing_count += 1;
  return SPSS_OK;
}

int fast_step(spss_ctx *ctx, int stepper, double t, double dt)
{
  (void) t;
  SPSS_TRY(launch_single_step(ctx, stepper, dt));
  const int rc = sync_control(ctx);
  SPSS_TRY(take_timing(ctx));
  return rc;
}

// One step of an AoS state the GPU addresses (`io`: read, stepped, written
// back), with one wait for the stream: the download writes the control block's
// host copy as well.  With a copy and a wait of its own between step and
// download, N = 2,000: 45.4 -> 26.9 us a call on Verlet lists, 66.6 -> 44.0 on cell lists.
int fast_step_state(spss_ctx *ctx, int stepper, double dt, double *io)
{
  SPSS_TRY(fast_set_state(ctx, io));
  SPSS_TRY(launch_single_step(ctx, stepper, dt));
  SPSS_TRY(launch_download(ctx, io, ctx->fast->h_ctrl));
  const int rc = adopt_control(ctx);
  SPSS_TRY(take_timing(ctx));
  return rc;
}

static int build_graph_on(spss_ctx *ctx, int stepper, const FastParams &P, int sampling, GraphEntry &g,
                          unsigned long long launches0);

// One step as a graph (+ the gated order-parameter sample): on a rebuild
// trigger, step + control, the control kernel tail-launching the rebuild graph
// when it is due (or the conditional form, whose rebuild sits under a
// conditional node ahead of the step); with cell lists, rebuild + step +
// control; otherwise step + control.
static int build_graph(spss_ctx *ctx, int stepper, double dt, int sampling, GraphEntry &g)
{
  const FastParams P = params(ctx, dt);
  const unsigned long long launches0 = ctx->launches;
  const int timing = ctx->timing;
  cudaStream_t work = ctx->stream;
  ctx->timing = 0;
  ctx->stream = ctx->own_stream;  // capture needs a non-legacy stream
  int rc_all = build_graph_on(ctx, stepper, P, sampling, g, launches0);
  ctx->stream = work;
  ctx->timing = timing;
  return rc_all;
}

// The conditional form: set-condition kernel, IF rebuild, step and control.
static int build_graph_conditional(spss_ctx *ctx, int stepper, const FastParams &P, int sampling, GraphEntry &g,
                                   unsigned long long launches0)
{
  FastPath *f = ctx->fast;
  cudaGraph_t graph;
  SPSS_CUDA_TRY(cudaGraphCreate(&graph, 0));
  cudaGraphConditionalHandle handle;
  SPSS_CUDA_TRY(cudaGraphConditionalHandleCreate(&handle, graph, 0, cudaGraphCondAssignDefault));
  // node 1: copy the rebuild flag into the condition
  SPSS_CUDA_TRY(cudaStreamBeginCaptureToGraph(ctx->stream, graph, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed));
  fast_set_condition_kernel<<<1, 1, 0, ctx->stream>>>(f->ctrl, handle);
  ++ctx->launches;
  SPSS_CUDA_TRY(cudaStreamEndCapture(ctx->stream, &graph));
  size_t nnodes = 0;
  SPSS_CUDA_TRY(cudaGraphGetNodes(graph, nullptr, &nnodes));
  std::vector<cudaGraphNode_t> nodes(nnodes);
  SPSS_CUDA_TRY(cudaGraphGetNodes(graph, nodes.data(), &nnodes));
  cudaGraphNode_t set_node = nodes.back();
  // node 2: IF rebuild
  // the struct holds a union with deleted constructors: zeroed raw storage
  alignas(cudaGraphNodeParams) unsigned char cp_storage[sizeof(cudaGraphNodeParams)] = {};
  cudaGraphNodeParams &cp = *reinterpret_cast<cudaGraphNodeParams *>(cp_storage);
  cp.type = cudaGraphNodeTypeConditional;
  cp.conditional.handle = handle;
  cp.conditional.type = cudaGraphCondTypeIf;
  cp.conditional.size = 1;
  cudaGraphNode_t cond_node;
  SPSS_CUDA_TRY(cudaGraphAddNode(&cond_node, graph, &set_node, nullptr, 1, &cp));
  cudaGraph_t body = cp.conditional.phGraph_out[0];
  SPSS_CUDA_TRY(cudaStreamBeginCaptureToGraph(ctx->stream, body, nullptr, nullptr, 0, cudaStreamCaptureModeRelaxed));
  const unsigned long long before_body = ctx->launches;
  int rc = launch_rebuild(ctx, P);
  g.per_rebuild = (int) (ctx->launches - before_body);
  cudaGraph_t body_out = body;
  cudaError_t e = cudaStreamEndCapture(ctx->stream, &body_out);
  if (rc != SPSS_OK) return rc;
  SPSS_CUDA_TRY(e);
  // nodes 3-4: step and control
  SPSS_CUDA_TRY(cudaStreamBeginCaptureToGraph(ctx->stream, graph, &cond_node, nullptr, 1, cudaStreamCaptureModeRelaxed));
  rc = launch_step(ctx, stepper, P);
  if (rc == SPSS_OK && sampling) rc = launch_sampling(ctx, P, 1);
  e = cudaStreamEndCapture(ctx->stream, &graph);
  if (rc != SPSS_OK) return rc;
  SPSS_CUDA_TRY(e);
  SPSS_CUDA_TRY(cudaGraphInstantiate(&g.exec, graph, 0));
  g.graph = graph;
  g.per_step = (int) (ctx->launches - launches0) - g.per_rebuild;
  g.form = GRAPH_CONDITIONAL;
  ctx->launches = launches0;  // captured, not launched
  return SPSS_OK;
}

// The rebuild as a graph that the control kernel can launch on the device.
static int build_device_rebuild(spss_ctx *ctx, const FastParams &P, GraphEntry &g)
{
  cudaGraph_t rg = nullptr;
  const unsigned long long before = ctx->launches;
  SPSS_CUDA_TRY(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeRelaxed));
  const int rc = launch_rebuild(ctx, P);
  const cudaError_t e = cudaStreamEndCapture(ctx->stream, &rg);
  g.per_rebuild = (int) (ctx->launches - before);
  if (rc != SPSS_OK)
  {
    if (rg) cudaGraphDestroy(rg);
    return rc;
  }
  SPSS_CUDA_TRY(e);
  g.rebuild_graph = rg;
  SPSS_CUDA_TRY(cudaGraphInstantiate(&g.rebuild_exec, rg, cudaGraphInstantiateFlagDeviceLaunch));
  SPSS_CUDA_TRY(cudaGraphUpload(g.rebuild_exec, ctx->stream));
  SPSS_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  return SPSS_OK;
}

// One step as a graph.  Verlet lists (and the trigger of list-less Verlet
// contexts): step and control, the control kernel tail-launching the rebuild
// graph when the trigger fires, so a step without a rebuild is two kernels
// and no conditional node (a conditional node and its set-condition kernel
// cost about 12 us per step on this GB300); the conditional form where this
// device refuses device-launched graphs or spss_set_device_rebuild asks for it
// (then for the kinds without lists too).  Cell lists and batches of small
// systems: the rebuild and the step, every step.  Kinds without lists: the step
// alone.
static int build_graph_on(spss_ctx *ctx, int stepper, const FastParams &P, int sampling, GraphEntry &g,
                          unsigned long long launches0)
{
  FastPath *f = ctx->fast;
  // a batch of small systems rebuilds by one kernel, which every step launches
  const bool trigger = (f->kind == KIND_VERLET && !f->small_systems) || f->trigger_only;
  const bool always = f->kind == KIND_CELLS || f->small_systems;
  if (trigger && f->device_rebuild)
  {
    const int rc = build_device_rebuild(ctx, P, g);
    if (rc != SPSS_OK)
    {
      // this device or driver refuses device-launched graphs: conditional form
      cudaGetLastError();
      g.release();
      f->device_rebuild = false;
      ctx->launches = launches0;
    }
  }
  if (!f->device_rebuild && !always)
    return build_graph_conditional(ctx, stepper, P, sampling, g, launches0);
  const unsigned long long launches_step = ctx->launches;
  cudaGraph_t graph = nullptr;
  SPSS_CUDA_TRY(cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeRelaxed));
  int rc = SPSS_OK;
  if (f->kind == KIND_CELLS) rc = launch_cells_step(ctx, stepper, P, true);
  else if (f->small_systems) rc = launch_rebuild(ctx, P);
  if (rc == SPSS_OK && f->kind != KIND_CELLS) rc = launch_step(ctx, stepper, P, trigger ? g.rebuild_exec : nullptr);
  if (rc == SPSS_OK && sampling) rc = launch_sampling(ctx, P, 1);
  const cudaError_t e = cudaStreamEndCapture(ctx->stream, &graph);
  if (rc != SPSS_OK)
  {
    if (graph) cudaGraphDestroy(graph);
    return rc;
  }
  SPSS_CUDA_TRY(e);
  g.graph = graph;
  SPSS_CUDA_TRY(cudaGraphInstantiate(&g.exec, graph, 0));
  g.per_step = (int) (ctx->launches - launches_step);
  g.form = trigger ? GRAPH_DEVICE : (always ? GRAPH_ALWAYS : GRAPH_NONE);
  ctx->launches = launches0;  // captured, not launched
  return SPSS_OK;
}

// nsteps steps: one graph launch each.
static int run_steps(spss_ctx *ctx, int stepper, double dt, long nsteps, int sampling)
{
  FastPath *f = ctx->fast;
  if (!f->have_state) return SPSS_ERR_INVALID_ARGUMENT;
  if (stepper == SPSS_STEPPER_RK4) return SPSS_ERR_NOT_SUPPORTED;
  if (nsteps <= 0) return nsteps == 0 ? SPSS_OK : SPSS_ERR_INVALID_ARGUMENT;
  if (ctx->timing)
  {
    for (long k = 0; k < nsteps; ++k)
    {
      SPSS_TRY(fast_step(ctx, stepper, 0.0, dt));
      if (sampling) SPSS_TRY(launch_sampling(ctx, params(ctx, dt), 1));
    }
    return sampling ? sync_control(ctx) : SPSS_OK;
  }
  SPSS_TRY(grow_lists(ctx));
  SPSS_TRY(push_host_control(ctx));
  if (f->kind == KIND_CELLS) SPSS_TRY(ensure_cells(ctx, params(ctx, dt)));
  SPSS_TRY(ensure_field(ctx, params(ctx, dt)));
  // the plain step, and the step with a sample behind it for the steps that
  // take one (whose kernels check the same condition on the device)
  GraphEntry *graph[2] = {nullptr, nullptr};
  int rebuilds0 = f->h_ctrl->rebuilds;
  bool first = true;
  int per_rebuild = 0;
  for (long k = 0; k < nsteps; ++k)
  {
    const int with_sample = sampling && samples_after(f->h_ctrl, f->h_ctrl->step + (unsigned long long) k + 1) ? 1 : 0;
    if (!graph[with_sample])
    {
      const auto key = std::make_tuple(stepper, dt, with_sample);
      auto it = f->graphs.find(key);
      if (it == f->graphs.end())
      {
        GraphEntry g;
        SPSS_TRY(build_graph(ctx, stepper, dt, with_sample, g));
        it = f->graphs.emplace(key, g).first;
      }
      graph[with_sample] = &it->second;
      per_rebuild = it->second.per_rebuild;
    }
    GraphEntry &g = *graph[with_sample];
    if (first && (g.form == GRAPH_DEVICE || g.form == GRAPH_NONE) && f->h_ctrl->rebuild)
    {
      // a rebuild pending before the first step (host request, eager steps):
      // these graphs rebuild only after a step's trigger
      SPSS_TRY(launch_rebuild(ctx, params(ctx, dt)));
      rebuilds0 += 1;
    }
    first = false;
    SPSS_CUDA_TRY(cudaGraphLaunch(g.exec, ctx->stream));
    ctx->launches += (unsigned long long) g.per_step;
  }
  const int rc = sync_control(ctx);
  ctx->launches += (unsigned long long) (f->h_ctrl->rebuilds - rebuilds0) * per_rebuild;
  return rc;
}

int fast_steps(spss_ctx *ctx, int stepper, double t0, double dt, int nsteps)
{
  (void) t0;
  return run_steps(ctx, stepper, dt, nsteps, 0);
}

int fast_batch_run(spss_ctx *ctx, int stepper, double dt, long nsteps, long sample_every, long sample_from)
{
  FastPath *f = ctx->fast;
  if (sample_every < 0 || sample_from < 0) return SPSS_ERR_INVALID_ARGUMENT;
  f->h_ctrl->sample_every = sample_every;
  f->h_ctrl->sample_from = sample_from;
  SPSS_CUDA_TRY(cudaMemcpyAsync(&f->ctrl->sample_every, &f->h_ctrl->sample_every, 2 * sizeof(long long),
                                cudaMemcpyHostToDevice, ctx->stream));
  return run_steps(ctx, stepper, dt, nsteps, sample_every > 0 ? 1 : 0);
}

int fast_batch_stats(spss_ctx *ctx, double *h_out)
{
  FastPath *f = ctx->fast;
  std::vector<double> raw((size_t) 5 * f->nsys);
  SPSS_CUDA_TRY(cudaMemcpyAsync(raw.data(), f->stats.ptr, sizeof(double) * raw.size(), cudaMemcpyDeviceToHost,
                                ctx->stream));
  SPSS_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  for (int r = 0; r < f->nsys; ++r)
  {
    const double *st = &raw[5 * (size_t) r];
    const double c = st[4];
    double *o = h_out + 5 * (size_t) r;
    const double m0 = c > 0 ? st[0] / c : 0.0, m2 = c > 0 ? st[2] / c : 0.0;
    o[0] = m0;
    o[1] = c > 0 ? std::max(0.0, st[1] / c - m0 * m0) : 0.0;
    o[2] = m2;
    o[3] = c > 0 ? std::max(0.0, st[3] / c - m2 * m2) : 0.0;
    o[4] = c;
  }
  return SPSS_OK;
}

int fast_batch_reset_stats(spss_ctx *ctx)
{
  FastPath *f = ctx->fast;
  SPSS_CUDA_TRY(cudaMemsetAsync(f->stats.ptr, 0, sizeof(double) * 5 * f->nsys, ctx->stream));
  SPSS_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  return SPSS_OK;
}

int fast_system_order_parameters(spss_ctx *ctx, double *h_out)
{
  FastPath *f = ctx->fast;
  if (!f->have_state) return SPSS_ERR_INVALID_ARGUMENT;
  SPSS_TRY(launch_sampling(ctx, params(ctx, 0.0), 0));
  SPSS_CUDA_TRY(cudaMemcpyAsync(h_out, f->order_out.ptr, sizeof(double) * 4 * f->nsys, cudaMemcpyDeviceToHost,
                                ctx->stream));
  SPSS_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  return SPSS_OK;
}

// |<e^{i phi}>|, its argument and the velocity-direction pair over the context.
int fast_order_parameters(spss_ctx *ctx, double *out4)
{
  FastPath *f = ctx->fast;
  const bool table = ctx->p.n >= kTurnTableMin;
  const int blocks = std::min(2 * 152, blocks_for(ctx->p.n, 256));
  const int smem = table ? kTurnAll * (int) sizeof(double2) : 0;
  SPSS_TRY(f->observe_partial.reserve(4 * 2 * 152));
  if (!f->h_order) SPSS_CUDA_TRY(cudaMallocHost((void **) &f->h_order, 4 * sizeof(double)));
  if (table && !f->turn_table.ptr)
  {
    SPSS_TRY(f->turn_table.reserve(kTurnAll));
    SPSS_CUDA_TRY(cudaFuncSetAttribute(fast_observe_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    fast_turn_table_kernel<<<blocks_for(kTurnAll, 256), 256, 0, ctx->stream>>>(f->turn_table.ptr);
    ++ctx->launches;
    SPSS_TRY(check_launch("fast_turn_table_kernel"));
  }
  const FastParams P = params(ctx, 0.0);
  const FastBuffers B = buffers(ctx);
  if (table)
    fast_observe_kernel<true><<<blocks, 256, smem, ctx->stream>>>(P, B, f->turn_table.ptr, f->observe_partial.ptr,
                                                                  f->h_order);
  else
    fast_observe_kernel<false><<<blocks, 256, 0, ctx->stream>>>(P, B, nullptr, f->observe_partial.ptr, f->h_order);
  ++ctx->launches;
  SPSS_TRY(check_launch("fast_observe_kernel"));
  SPSS_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  // two square roots and two arguments: a chain of FP64 latencies on the device, nothing here
  order_from_sums(f->h_order, (double) ctx->p.n, ctx->p.model, out4);
  return SPSS_OK;
}

// The state as a float frame at `d_out` (device memory, or host memory the GPU addresses).
int fast_frame(spss_ctx *ctx, int wrap, float *d_out)
{
  const int smem = (int) sizeof(float) * 256 * ctx->s, blocks = blocks_for(ctx->p.n, 256);
  if (wrap)
    fast_frame_kernel<true><<<blocks, 256, smem, ctx->stream>>>(d_out, ctx->p.n, ctx->s, ctx->p.model, buffers(ctx));
  else
    fast_frame_kernel<false><<<blocks, 256, smem, ctx->stream>>>(d_out, ctx->p.n, ctx->s, ctx->p.model, buffers(ctx));
  ++ctx->launches;
  return check_launch("fast_frame_kernel");
}

int fast_rebuild_count(spss_ctx *ctx, unsigned long long *count)
{
  SPSS_TRY(sync_control(ctx));
  *count = (unsigned long long) ctx->fast->h_ctrl->rebuilds;
  return SPSS_OK;
}

int fast_num_systems(const spss_ctx *ctx)
{
  return ctx->fast ? ctx->fast->nsys : 1;
}

int fast_system_first(const spss_ctx *ctx, int r)
{
  return ctx->fast->h_sys[r].first;
}

int fast_set_tiling(spss_ctx *ctx, int tile_cells, int persistent)
{
  if (tile_cells < 1 || tile_cells > 4096 || (persistent != 0 && persistent != 1)) return SPSS_ERR_INVALID_ARGUMENT;
  FastPath *f = ctx->fast;
  if (!has_cells(f->kind))
  {
    f->persistent = persistent;
    return SPSS_OK;
  }
  f->tile_cells = tile_cells;
  f->persistent = persistent;
  // the lists are rebuilt before the next step
  f->h_ctrl->rebuild = REBUILD_ALL;
  ctx->should_update_lists = 1;
  SPSS_CUDA_TRY(cudaMemcpyAsync(&f->ctrl->rebuild, &f->h_ctrl->rebuild, sizeof(int), cudaMemcpyHostToDevice,
                                ctx->stream));
  SPSS_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  return SPSS_OK;
}

int fast_set_device_rebuild(spss_ctx *ctx, int enabled)
{
  FastPath *f = ctx->fast;
  if (f->device_rebuild == (enabled != 0)) return SPSS_OK;
  f->device_rebuild = enabled != 0;
  for (auto &g : f->graphs) g.second.release();
  f->graphs.clear();
  return SPSS_OK;
}

int fast_get_tiling(spss_ctx *ctx, int *tile_cells, int *persistent)
{
  *tile_cells = ctx->fast->tile_cells;
  *persistent = ctx->fast->persistent;
  return SPSS_OK;
}

template<class T>
static int copy_device(DeviceArray<T> &dst, const T *src, size_t count, cudaStream_t stream)
{
  SPSS_TRY(dst.reserve(count));
  SPSS_CUDA_TRY(cudaMemcpyAsync(dst.ptr, src, sizeof(T) * count, cudaMemcpyDeviceToDevice, stream));
  return SPSS_OK;
}

template<class T>
static int restore_device(T *dst, const DeviceArray<T> &src, size_t count, cudaStream_t stream)
{
  SPSS_CUDA_TRY(cudaMemcpyAsync(dst, src.ptr, sizeof(T) * count, cudaMemcpyDeviceToDevice, stream));
  return SPSS_OK;
}

static int take_snapshot(spss_ctx *ctx)
{
  FastPath *f = ctx->fast;
  Snapshot &S = f->snap;
  const size_t n = (size_t) ctx->p.n;
  cudaStream_t st = ctx->stream;
  for (int b = 0; b < 2; ++b)
  {
    SPSS_TRY(copy_device(S.rec[b], f->rec[b].ptr, n, st));
    SPSS_TRY(copy_device(S.aux[b], f->aux[b].ptr, n, st));
    SPSS_TRY(copy_device(S.vel[b], b ? f->vel_tmp.ptr : f->vel.ptr, n, st));
    SPSS_TRY(copy_device(S.pid[b], b ? f->pid_tmp.ptr : f->pid.ptr, n, st));
  }
  SPSS_TRY(copy_device(S.inv, f->inv.ptr, n, st));
  SPSS_TRY(copy_device(S.img, f->img.ptr, n, st));
  SPSS_TRY(copy_device(S.turns, f->turns.ptr, n, st));
  SPSS_TRY(copy_device(S.sysctl, f->sysctl.ptr, (size_t) f->nsys, st));
  SPSS_TRY(copy_device(S.ctrl, f->ctrl, 1, st));
  SPSS_CUDA_TRY(cudaStreamSynchronize(st));
  return SPSS_OK;
}

// Back to the snapshot; the lists are rebuilt before the next step.
static int restore_snapshot(spss_ctx *ctx)
{
  FastPath *f = ctx->fast;
  Snapshot &S = f->snap;
  const size_t n = (size_t) ctx->p.n;
  cudaStream_t st = ctx->stream;
  for (int b = 0; b < 2; ++b)
  {
    SPSS_TRY(restore_device(f->rec[b].ptr, S.rec[b], n, st));
    SPSS_TRY(restore_device(f->aux[b].ptr, S.aux[b], n, st));
    SPSS_TRY(restore_device(b ? f->vel_tmp.ptr : f->vel.ptr, S.vel[b], n, st));
    SPSS_TRY(restore_device(b ? f->pid_tmp.ptr : f->pid.ptr, S.pid[b], n, st));
  }
  SPSS_TRY(restore_device(f->inv.ptr, S.inv, n, st));
  SPSS_TRY(restore_device(f->img.ptr, S.img, n, st));
  SPSS_TRY(restore_device(f->turns.ptr, S.turns, n, st));
  SPSS_TRY(restore_device(f->sysctl.ptr, S.sysctl, (size_t) f->nsys, st));
  SPSS_CUDA_TRY(cudaMemcpyAsync(f->h_ctrl, S.ctrl.ptr, sizeof(FastControl), cudaMemcpyDeviceToHost, st));
  SPSS_CUDA_TRY(cudaStreamSynchronize(st));
  f->h_ctrl->rebuild = 1;
  f->h_ctrl->cells_fresh = 0;  // cell ids are not part of the snapshot
  SPSS_CUDA_TRY(cudaMemcpyAsync(f->ctrl, f->h_ctrl, sizeof(FastControl), cudaMemcpyHostToDevice, st));
  SPSS_CUDA_TRY(cudaStreamSynchronize(st));
  ctx->step_counter = f->h_ctrl->step;
  ctx->accumulated_displacement = f->h_ctrl->acc;
  ctx->should_update_lists = 1;
  S.release();
  return SPSS_OK;
}

// Times `steps` steps (graph launches, CUDA events) from the state the call
// finds and puts the state back as it was.  The step kernels take a particle
// per thread whatever the tiling, so there is nothing to choose between.
int fast_autotune(spss_ctx *ctx, int stepper, double dt, int steps, double *best_ms)
{
  FastPath *f = ctx->fast;
  if (!f->have_state || steps < 1) return SPSS_ERR_INVALID_ARGUMENT;
  if (stepper == SPSS_STEPPER_RK4) return SPSS_ERR_NOT_SUPPORTED;
  if (!has_cells(f->kind))
  {
    if (best_ms) *best_ms = 0.0;
    return SPSS_OK;
  }
  const int timing = ctx->timing;
  ctx->timing = 0;
  SPSS_TRY(take_snapshot(ctx));
  float ms = 0.0f;
  int rc = run_steps(ctx, stepper, dt, 2, 0);  // builds the graph, warms up
  if (rc == SPSS_OK)
  {
    cudaEventRecord(ctx->ev0, ctx->stream);
    rc = run_steps(ctx, stepper, dt, steps, 0);
    cudaEventRecord(ctx->ev1, ctx->stream);
  }
  if (rc == SPSS_OK && (cudaEventSynchronize(ctx->ev1) != cudaSuccess ||
                        cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1) != cudaSuccess))
  {
    cudaGetLastError();
    rc = SPSS_ERR_CUDA;
  }
  const int rc2 = restore_snapshot(ctx);
  ctx->timing = timing;
  if (rc != SPSS_OK) return rc;
  if (rc2 != SPSS_OK) return rc2;
  if (best_ms) *best_ms = ms / steps;
  return SPSS_OK;
}

int fast_set_natural_frequencies(spss_ctx *ctx, const double *d_freqs)
{
  FastPath *f = ctx->fast;
  if (f->kind != KIND_GLOBAL) return SPSS_ERR_NOT_SUPPORTED;  // the reference uses them in the global field only
  fast_set_frequencies_kernel<<<blocks_for(ctx->p.n, kTB), kTB, 0, ctx->stream>>>(d_freqs, ctx->p.n, f->nu.ptr);
  ++ctx->launches;
  return check_launch("fast_set_frequencies_kernel");
}

int fast_noise(spss_ctx *ctx, int stepper, unsigned long long step, double *d_out)
{
  const int per = normals_per_particle(ctx->p.model, stepper);
  if (per == 0) return SPSS_OK;
  NoiseKey nk;
  nk.seed = ctx->p.seed;
  nk.replica = ctx->p.replica;
  nk.step = step;
  fast_noise_kernel<<<blocks_for(ctx->p.n, kTB), kTB, 0, ctx->stream>>>(d_out, ctx->p.n, per, nk, ctx->fast->sys.ptr,
                                                                       ctx->fast->sys_of.ptr);
  ++ctx->launches;
  return check_launch("fast_noise_kernel");
}

int fast_evaluate(spss_ctx *, int, const double *, const double *, double *, double, double)
{
  return SPSS_ERR_NOT_SUPPORTED;
}

int fast_complementary_force(spss_ctx *, double *)
{
  return SPSS_ERR_NOT_SUPPORTED;
}

int fast_apply_pbc(spss_ctx *ctx)
{
  fast_pbc_kernel<<<blocks_for(ctx->p.n, kTB), kTB, 0, ctx->stream>>>(ctx->fast->img.ptr, ctx->p.n);
  ++ctx->launches;
  return check_launch("fast_pbc_kernel");
}

}  // namespace spss
