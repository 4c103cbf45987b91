// FP64 path: the reference's arithmetic in 64 bits on the GPU.
//
// This translation unit is compiled with --fmad=false, so the stage, distance
// and stepper expressions below round exactly like the reference built with
// -ffp-contract=off.  Cell ids, member lists (ascending) and Verlet lists (in
// push_back order) are bit-identical to the reference's; floating-point results
// differ only by the last bits of sin/cos/atan2/hypot and of the torques: where
// sums of directions are as accurate as the reference's sine a pair they are
// formed from those, elsewhere (aligned phases) pair by pair (NeighbourSums).
// Layout: AoS double[n*s], as the reference.
//
// Reference: DynamicalSystems/ParticleSystemFirstOrder.cpp, ParticleSystemFirstOrderPtr.cpp,
// ParticleSystemSecondOrder.cpp, BoundaryConfiguration/PeriodicBoundaryConditions.cpp,
// Steppers/*.
#include <algorithm>
#include <cstring>

#include "spss_internal.cuh"

namespace spss
{

struct F64Path
{
  DeviceArray<double> state, rk, k[4], td, det, caf, nat_freq, partials, scratch_state, scratch_kprev,
      scratch_knext;
  DeviceArray<int> cell_of;
  DeviceArray<float2> posf;  // stage positions wrapped into the box, float (all-pairs range pre-test)
  DeviceArray<double2> table;  // of the FP64 functions
  DeviceArray<double2> csphi;    // cos and sin of the stage phase, written with the stage
  DeviceArray<longlong2> turns;  // the same in fixed point
  // the other stage buffers of an all-pairs RK4 step, whose pair kernels
  // write the next stage's state while they read this one's
  DeviceArray<double> rk2;
  DeviceArray<float2> posf2;
  DeviceArray<float2> posf_rows;  // posf and turns in cell order (linked list)
  DeviceArray<longlong2> turns_rows;
  DeviceArray<double2> csphi2;
  DeviceArray<longlong2> turns2;
  Binner binner;
  int cells_nc = 0;  // cells per side of the last build (0: none)
  DeviceArray<int> vl_count, vl_off, vl_ent;
  long vl_total = 0;
  int vl_built = 0;
  DeviceArray<unsigned long long> max2;
  unsigned long long *h_max2 = nullptr;  // pinned
  // one RK4 step captured as a CUDA graph (f64_steps), for the dt and
  // higher-order flag it was captured with
  cudaGraph_t rk4_graph = nullptr;
  cudaGraphExec_t rk4_exec = nullptr;
  double rk4_dt = 0.0;
  int rk4_higher_order = -1;
  unsigned long long rk4_launches = 0;  // kernels in the captured step
};

struct K64
{
  int model, flavor, n, s;
  double v0, xi, xi_r, xi_phi, sigma, alpha, rho2, rmax2, ca, sa;
  const double2 *table;  // of the FP64 functions (make_f64_tables)
  int higher_order;
  float rho_excl;  // a pair whose float minimum-image distance bound exceeds this is out of range
  float rho_incl, rmax_excl, rmax_incl;  // the cutoffs less (plus) two margins
  float ca_f, sa_f;  // ca, sa
  float least;       // mean |sin(phi_j - phi_i - alpha)| from which on sums of directions are accurate enough
};

// Margin of the range pre-test, in box units: six times what the float rounding
// of the wrapped positions (6e-8 a difference), of the minimum image and of
// the squares (1e-7 together) and the FP64 differences of positions up to 2^20
// boxes away (2e-10) amount to; a position farther away has no float one
// (pretest_position).  A pair nearer to the cutoff than this is decided in
// FP64, for the whole warp's time: at N = 65,536 a margin of 2e-5 left 0.27
// such pairs a particle and the linked-list kernel took 64 us, now 44.
constexpr float kPretestMargin = 1e-6f;

static K64 make_k64(const spss_ctx *ctx)
{
  K64 k;
  const spss_params &p = ctx->p;
  k.model = p.model;
  k.flavor = p.flavor;
  k.n = p.n;
  k.s = ctx->s;
  k.v0 = p.v0;
  k.xi = p.xi;
  k.xi_r = p.xi_r;
  k.xi_phi = p.xi_phi;
  k.sigma = p.sigma;
  k.alpha = p.alpha;
  k.rho2 = p.rho * p.rho;
  k.rmax2 = ctx->r_max * ctx->r_max;
  k.ca = std::cos(p.alpha);  // host libm, as the reference's constructor
  k.sa = std::sin(p.alpha);
  k.higher_order = ctx->higher_order;
  k.table = ctx->f64->table.ptr;
  k.rho_excl = (float) (p.rho + 2.0 * kPretestMargin);
  k.rho_incl = (float) std::max(0.0, p.rho - 2.0 * kPretestMargin);
  k.rmax_excl = (float) (ctx->r_max + 2.0 * kPretestMargin);
  k.rmax_incl = (float) std::max(0.0, ctx->r_max - 2.0 * kPretestMargin);
  k.ca_f = (float) k.ca;
  k.sa_f = (float) k.sa;
  k.least = p.model == 2 && p.alpha != 0.0 ? 0.25f : 0.03125f;
  return k;
}

// ------------------------------------------------------------ PBC helpers

// ClassAEffectiveParticleDistance, unit box (PeriodicBoundaryConditions.cpp:26-38).
__device__ __forceinline__ double class_a(double d)
{
  return d - (double) (int) (d * 2.0 * 1.0) * 1.0;
}

// ClassCEffectiveParticleDistanceUnsigned, unit box (PeriodicBoundaryConditions.cpp:107-119).
__device__ __forceinline__ double class_c(double d)
{
  d = fabs(d);
  return d - (double) (int) (d * 1.0 + 0.5) * 1.0;
}

// ApplyPeriodicBoundaryConditions(x, y, ...) (PeriodicBoundaryConditions.cpp:121-125).
__device__ __forceinline__ double wrap1(double x)
{
  return x - floor(x * 1.0) * 1.0;
}

// Second-order classes wrap only positions that left the box (ParticleSystemSecondOrder.cpp:323-326).
__device__ __forceinline__ void wrap_if_outside(double &x, double &y)
{
  if (x < 0.0 || x >= 1.0 || y < 0.0 || y >= 1.0)
  {
    x = wrap1(x);
    y = wrap1(y);
  }
}

// int(x / x_size * num_subcells) (ParticleSystemFirstOrder.cpp:277-279); the
// reference's out-of-range result for a coordinate that rounds to the box
// edge is clamped to the last cell.
__device__ __forceinline__ int cell_coord(double x, int nc)
{
  int c = (int) (x / 1.0 * nc);
  return c >= nc ? nc - 1 : (c < 0 ? 0 : c);
}

// AdjustNeighboringCellToPeriodicBoundaries (ParticleSystemFirstOrder.cpp:651-668).
__device__ __forceinline__ int adjust_cell(int c, int nc)
{
  return c < 0 ? nc - 1 : (c >= nc ? 0 : c);
}

// neighboring_cells_ (ParticleSystemFirstOrder.cpp:47-52).
__constant__ int c_stencil[9][2] = {{-1, -1}, {0, -1}, {1, -1}, {-1, 0}, {0, 0}, {1, 0}, {-1, 1}, {0, 1}, {1, 1}};

__device__ __forceinline__ void pos_for_cells(const K64 &k, const double *rk, int i, double &x, double &y)
{
  x = rk[(long) k.s * i];
  y = rk[(long) k.s * i + 1];
  if (k.model == 1)
  {
    x = wrap1(x);
    y = wrap1(y);
  } else
  {
    wrap_if_outside(x, y);
  }
}

// dr^2 of one candidate pair as the given class computes it.  The
// second-order all-pairs routine uses x_j as is; its linked-list routine
// wraps x_j if it left the box (ParticleSystemSecondOrder.cpp:380-385).
template<bool WRAP_J>
__device__ __forceinline__ double pair_dr2(const K64 &k, double x_i, double y_i, double x_j, double y_j)
{
  double dx, dy;
  if (k.model == 1)
  {
    dx = class_c(x_j - x_i);
    dy = class_c(y_j - y_i);
  } else
  {
    if (WRAP_J) wrap_if_outside(x_j, y_j);
    dx = class_a(x_j - x_i);
    dy = class_a(y_j - y_i);
  }
  return dx * dx + dy * dy;
}

struct Sums
{
  double af, card, caf;

  // af and caf summed another way
  __device__ __forceinline__ void take(double2 v)
  {
    af = v.x;
    caf = v.y;
  }
};

// Sums over the neighbours of one particle: of the directions, exactly, as
// integers, and of the directions times omega_j - omega_i in FP64 (only for the
// complementary force).
//
// Every pair term is a sine or cosine of phi_j - phi_i (- alpha), so their sums
// follow from the sums of cos phi_j and sin phi_j, one evaluation a particle
// in place of one a pair: the integer pipe adds 64 bits some thirty times faster
// than the FP64 pipe.  But a direction is off by some 2^-60 whatever the term, where
// a sine is off by 2^-54 of itself.  So the sum of |sin(phi_j - phi_i - alpha)| goes
// along in FP32, and where the terms are smaller than K64::least on average
// (aligned or opposite neighbours) they are summed again pair by pair, as they
// are where a phase has no fixed-point direction.  At the line, 1/32, both ways are
// off by about the same; with alpha in the second-order model it lies at 1/4,
// because the rotation by alpha rounds at 2^-53 of the sums of sines and cosines.
struct NeighbourSums
{
  long long c = 0, s = 0;                    // of the candidates scanned together, units of 2^-59
  long long ch = 0, cl = 0, sh = 0, sl = 0;  // units of 2^-27 and 2^-59
  int n = 0, bad = 0;
  float sines = 0.0f;
  double wc = 0.0, ws = 0.0;
  unsigned long long hits = 0;  // of the first 64 candidates

  // |sin(phi_j - phi_i - alpha)|; own: own_turned of the particle
  __device__ __forceinline__ static float sine(longlong2 d, float2 own)
  {
    return fabsf(fmaf((float) (int) (d.y >> 32), own.x, -((float) (int) (d.x >> 32) * own.y)));
  }

  // A candidate's direction, zeros where it is out of range (no branch: all
  // lanes go on together).
  __device__ __forceinline__ void add(longlong2 d, float2 own)
  {
    const int hc = (int) (d.x >> 32);
    c += d.x;
    s += d.y;
    sines += sine(d, own);
    bad |= hc ^ (hc << 1);  // negative for the lowest value alone
  }

  // After a set of eight, the `at`-th (`in`: those in range); the two sums hold
  // fifteen at most.
  __device__ __forceinline__ void close(unsigned in, int at)
  {
    ch += (int) (c >> 32);
    cl += (unsigned) c;
    sh += (int) (s >> 32);
    sl += (unsigned) s;
    c = s = 0;
    n += __popc(in);
    if (at < 8) hits |= (unsigned long long) in << (8 * at);
  }
};

// cos and sin of phi_i + alpha over 2^27, from the fixed-point direction.
__device__ __forceinline__ float2 own_turned(const K64 &k, longlong2 d)
{
  const float c = (float) (int) (d.x >> 32) * 5.5511151231257827e-17f;
  const float s = (float) (int) (d.y >> 32) * 5.5511151231257827e-17f;
  return make_float2(fmaf(c, k.ca_f, -(s * k.sa_f)), fmaf(s, k.ca_f, c * k.sa_f));
}

__device__ __forceinline__ bool lacks_direction(longlong2 d)
{
  return (int) (d.x >> 32) == INT_MIN;
}

__device__ __forceinline__ bool not_finite(double v)
{
  return (__double2hiint(v) & 0x7ff00000) == 0x7ff00000;
}

// Whether the sums of directions do not do (see above), or those with omega are
// not finite: an infinite omega_j then meets its own cosine alone.
__device__ __forceinline__ bool needs_pairs(const K64 &k, const NeighbourSums &a, longlong2 own)
{
  return a.n > 0 && (a.bad < 0 || lacks_direction(own) || a.sines < k.least * (float) a.n ||
                     (k.higher_order && not_finite(a.wc + a.ws)));
}

// Pair sums: first order ParticleSystemFirstOrderPtr.cpp:404-415; second order
// ParticleSystemSecondOrder.cpp:160-161, sin(phi_j - phi_i - alpha) (its
// complementary force is the first-order term in that convention).
// own, turn: the particle's direction in FP64 and in fixed point.  The products of
// the upper words are taken without a rounding between them (Kahan's ab - cd).
__device__ __forceinline__ Sums pair_sums(const K64 &k, const NeighbourSums &a, double2 own, longlong2 turn)
{
  const double Ch = (double) a.ch, Sh = (double) a.sh, Cl = (double) a.cl, Sl = (double) a.sl;
  const double ch = (double) (int) (turn.x >> 32), sh = (double) (int) (turn.y >> 32);
  const double cl = (double) (unsigned) turn.x, sl = (double) (unsigned) turn.y;
  constexpr double u54 = 5.5511151231257827e-17, u86 = 1.2924697071141057e-26, u59 = 1.7347234759768071e-18;
  // sum of sin(phi_j - phi_i)
  const double t = Ch * sh;
  const double p = fma(fma(Sh, ch, -t) - fma(Ch, sh, -t), u54,
                       fma(fma(Sh, cl, -(Ch * sl)), u86, fma(Sl, own.x, -(Cl * own.y)) * u59));
  Sums r{p, (double) a.n, 0.0};
  if (k.alpha != 0.0)
  {
    const double v = Sh * sh;
    const double q = fma(fma(Ch, ch, v) + fma(Sh, sh, -v), u54,  // and of cos
                         fma(fma(Ch, cl, Sh * sl), u86, fma(Cl, own.x, Sl * own.y) * u59));
    r.af = p * k.ca - q * k.sa;
  }
  if (k.higher_order)
  {
    const double pw = a.ws * own.x - a.wc * own.y, qw = a.wc * own.x + a.ws * own.y;
    r.caf = qw * k.ca + pw * k.sa;
  }
  return r;
}

// A sum with what its additions rounded off (Knuth's TwoSum).
struct KeptSum
{
  double v = 0.0, e = 0.0;

  __device__ __forceinline__ void add(double x)
  {
    const double s = v + x, b = s - v;
    e += (v - (s - b)) + (x - b);
    v = s;
  }

  __device__ __forceinline__ double value() const { return e == e ? v + e : v; }  // infinite terms: no rest
};

struct PairTerms
{
  KeptSum af, caf;

  __device__ __forceinline__ double2 values() const { return make_double2(af.value(), caf.value()); }
};

// The term of one pair by its own sine and cosine, the difference of the phases
// with what its subtractions rounded off.
__device__ __forceinline__ void add_pair(const K64 &k, PairTerms &a, double phi_i, double omega_i, double phi_j,
                                         double omega_j)
{
  double d = phi_j - phi_i, e = 0.0;
  if (k.model == 2 && k.alpha != 0.0)
  {
    const double v = d - phi_j;
    e = (phi_j - (d - v)) - (phi_i + v);
    const double f = d - k.alpha, w = f - d;
    e += (d - (f - w)) - (k.alpha + w);
    d = f;
  } else if (fabs(d) > 0.0625)  // below, what is rounded off is 2^-53 of the term at most
  {
    const double v = d - phi_j;
    e = (phi_j - (d - v)) - (phi_i + v);
  }
  double s, c;
  fast_sincos(k.table, d, s, c);
  const double sd = fma(c, e, s), cd = fma(-s, e, c);
  if (k.model == 1)
  {
    a.af.add(sd * k.ca - cd * k.sa);
    if (k.higher_order) a.caf.add((omega_j - omega_i) * (cd * k.ca + sd * k.sa));
  } else
  {
    a.af.add(sd);
    if (k.higher_order) a.caf.add((omega_j - omega_i) * cd);
  }
}

// Output of one particle (ParticleSystemFirstOrder.cpp:220-226, ParticleSystemSecondOrder.cpp:166-175);
// the torque component is left untouched when the particle has no neighbour.
// In two parts: what needs the pair sums (the torque component and the
// complementary force) and what does not (c, s: cos and sin of the phase).
__device__ __forceinline__ void write_k_but_torque(const K64 &k, int i, const double *st, double *k_next, double c,
                                                   double s)
{
  double *out = k_next + (long) k.s * i;
  if (k.model == 1)
  {
    *reinterpret_cast<double2 *>(out) = make_double2(k.v0 * c, k.v0 * s);
    out[2] = st[3];
  } else
  {
    const double v_x_i = st[2], v_y_i = st[3];
    *reinterpret_cast<double2 *>(out) = make_double2(v_x_i, v_y_i);
    *reinterpret_cast<double2 *>(out + 2) = make_double2(-k.xi_r * v_x_i + k.v0 * c, -k.xi_r * v_y_i + k.v0 * s);
    out[4] = st[5];
  }
}

// own: cos and sin of the particle's phase.
__device__ __forceinline__ void write_k(const K64 &k, int i, const double *st, double2 own, Sums a, double *k_next,
                                        double *caf)
{
  write_k_but_torque(k, i, st, k_next, own.x, own.y);
  if (a.card != 0.0)
  {
    k_next[(long) k.s * i + k.s - 1] = -(k.model == 1 ? k.xi : k.xi_phi) * st[k.s - 1] + k.sigma * a.af / a.card;
    if (k.higher_order) a.caf *= k.sigma / a.card;
  }
  if (k.higher_order) caf[i] = a.caf;
}

// ------------------------------------------------------------ kernels

// The binning that a stage kernel starts (nc cells a side, 0: none).
struct StageCells
{
  int nc, *cell_of, *count, *slot;
};

// The position for the range pre-test: wrapped into the unit box, as floats.
// From 2^20 boxes on, where the rounding of an FP64 difference approaches the
// margin (and at 10^10 exceeds it), no number: every pair is then left to the
// reference's FP64 expression.
__device__ __forceinline__ float2 pretest_position(double x, double y)
{
  if (max(__double2hiint(x) & 0x7fffffff, __double2hiint(y) & 0x7fffffff) >= 0x41300000)
    return make_float2(__int_as_float(0x7fffffff), __int_as_float(0x7fffffff));
  return make_float2((float) (x - floor(x)), (float) (y - floor(y)));
}

// Cell of a stage position, and its place among the cell's members by arrival.
__device__ __forceinline__ int stage_cell(const K64 &k, const double *rk, int i, int nc)
{
  double x, y;
  pos_for_cells(k, rk, i, x, y);
  return cell_coord(y, nc) * nc + cell_coord(x, nc);
}

// rk_system_state = system_state + k_coef * dt * k_prev (ParticleSystemFirstOrder.cpp:175-184),
// and (posf not null) the stage positions wrapped into the unit box as floats
// for the range pre-test and the directions of the phases (FP64 and fixed
// point); one particle per thread.  kp null: k_prev is zero.
// det (not null): its torque components are cleared, which the derivative
// leaves as they are where a particle has no neighbour.  Cells: counted on the
// way, which as two kernels behind this one took 9 us of a step of N = 65,536.
__global__ void f64_stage_kernel(K64 k, const double *__restrict__ st, const double *__restrict__ kp,
                                 double *__restrict__ rk, float2 *__restrict__ posf, double2 *__restrict__ csphi,
                                 longlong2 *__restrict__ turns, double k_coef, double dt, double *__restrict__ det,
                                 StageCells cells)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= k.n) return;
  const double2 *s2 = reinterpret_cast<const double2 *>(st + (long) k.s * i);
  const double2 *k2 = reinterpret_cast<const double2 *>(kp + (long) k.s * i);
  double2 *r2 = reinterpret_cast<double2 *>(rk + (long) k.s * i);
  for (int q = 0; q < k.s / 2; ++q)
  {
    const double2 a = s2[q], b = kp ? k2[q] : make_double2(0.0, 0.0);
    const double2 r = make_double2(a.x + k_coef * dt * b.x, a.y + k_coef * dt * b.y);
    r2[q] = r;
    if (q == 0 && posf) posf[i] = pretest_position(r.x, r.y);
    if (q == k.s / 2 - 1 && posf)
    {
      double2 cs;
      longlong2 turn;
      directions(k.table, r.x, cs, turn);
      csphi[i] = cs;
      turns[i] = turn;
    }
  }
  if (det) det[(long) k.s * i + k.s - 1] = 0.0;
  if (cells.nc)
  {
    const int c = stage_cell(k, rk, i, cells.nc);
    cells.cell_of[i] = c;
    cells.slot[i] = atomicAdd(cells.count + c, 1);
  }
}

__global__ void f64_cell_kernel(K64 k, const double *__restrict__ rk, int nc, int *__restrict__ cell_of)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= k.n) return;
  cell_of[i] = stage_cell(k, rk, i, nc);
}

// The stage state of one particle per thread (the same expression as
// f64_stage_kernel, element by element), its position wrapped into the
// unit box as floats, for the all-pairs range pre-test, and the cos and sin
// of its phase for its own derivative (one thread per particle here, where
// the pair kernel would spend a whole warp's FP64 pipe time on one lane).
__global__ void f64_stage_posf_kernel(K64 k, const double *__restrict__ st, const double *__restrict__ kp,
                                      double *__restrict__ rk, float2 *__restrict__ posf,
                                      double2 *__restrict__ csphi, longlong2 *__restrict__ turns, double k_coef,
                                      double dt)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= k.n) return;
  const long ii = (long) k.s * i;
  for (int q = 0; q < k.s; ++q) rk[ii + q] = st[ii + q] + k_coef * dt * kp[ii + q];
  posf[i] = pretest_position(rk[ii], rk[ii + 1]);
  const double phi = rk[ii + (k.model == 1 ? 2 : 4)];
  double2 cs;
  longlong2 turn;
  directions(k.table, phi, cs, turn);
  csphi[i] = cs;
  turns[i] = turn;
}

// Where a pair stands to a cutoff by its float wrapped positions alone: 0 out of
// range, 1 in range, 2 too near the cutoff to tell.  The exact minimum image of
// the float positions is within the margin of the FP64 distance whenever the
// reference's distance function picks the minimum image: the first-order
// classes always do; the second-order one does for coordinate differences
// below 1, so a float difference within the margin of 1 is left to the FP64
// expression, and its all-pairs routine, whose x_j is not wrapped, may not use
// the answer 1.  Out of range holds for every image the reference may pick.
// `incl` and `excl` are the cutoff less and plus 2 margins.
__device__ __forceinline__ int pretest(float2 a, float2 b, float incl, float excl)
{
  const float rx = fabsf(b.x - a.x), ry = fabsf(b.y - a.y);
  const float dx = fminf(rx, 1.0f - rx), dy = fminf(ry, 1.0f - ry);
  const float lx = fmaxf(dx - kPretestMargin, 0.0f), ly = fmaxf(dy - kPretestMargin, 0.0f);
  const float ux = fabsf(dx) + kPretestMargin, uy = fabsf(dy) + kPretestMargin;
  // without branches: several pairs are tested at once
  const bool out = fmaf(lx, lx, ly * ly) > excl * excl;
  const bool sure = fmaf(ux, ux, uy * uy) < incl * incl && fmaxf(rx, ry) < 1.0f - kPretestMargin;
  return out ? 0 : (sure ? 1 : 2);
}

// What the pair kernel of an RK4 stage does after its derivative: the next
// stage rk = x + coef * dt * k_next (COMBINE: first the step's result
// x += (k1 + 2 k2 + 2 k3 + k4) dt / 6, RungeKutta4Stepper.cpp:56-59, which is
// the first stage of the next step), its wrapped float position and the cos
// and sin of its phase, the expressions of f64_stage_posf_kernel.
struct NextStage
{
  double *x;
  double coef, dt;
  double *rk;
  float2 *posf;
  double2 *csphi;
  longlong2 *turns;
  const double *k1, *k2, *k3;  // COMBINE
  double *td;
};

enum
{
  AFTER_NOTHING = 0,
  AFTER_STAGE = 1,
  AFTER_COMBINE = 2
};

// Component q of the next stage of a particle from its derivative kq (at
// `at`, its place in the state): k1, k2, k3 and x as stored there.
struct StageWords
{
  double x, k1, k2, k3;
};

template<int AFTER>
__device__ __forceinline__ StageWords load_stage(const NextStage &next, long at)
{
  if (AFTER == AFTER_COMBINE) return StageWords{next.x[at], next.k1[at], next.k2[at], next.k3[at]};
  return StageWords{AFTER == AFTER_STAGE ? next.x[at] : 0.0, 0.0, 0.0, 0.0};
}

template<int AFTER>
__device__ __forceinline__ double advance_component(const NextStage &next, long at, const StageWords &w, double kq)
{
  double r;
  if (AFTER == AFTER_COMBINE)
  {
    const double d = (w.k1 + 2.0 * w.k2 + 2.0 * w.k3 + kq) * next.dt / 6.0;
    next.td[at] = d;
    r = w.x + d;
    next.x[at] = r;
  } else
  {
    r = w.x + next.coef * next.dt * kq;
  }
  next.rk[at] = r;
  return r;
}

// The next stage but omega, whose derivative needs the pair sums, with the
// float position and the cos and sin of the phase.
template<int AFTER>
__device__ __forceinline__ void advance_but_omega(const K64 &k, int i, const double *k_next, const NextStage &next)
{
  const long ii = (long) k.s * i;
  double row[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
#pragma unroll
  for (int q = 0; q < 5; ++q)
    if (q < k.s - 1) row[q] = advance_component<AFTER>(next, ii + q, load_stage<AFTER>(next, ii + q), k_next[ii + q]);
  next.posf[i] = pretest_position(row[0], row[1]);
  double2 cs;
  longlong2 turn;
  directions(k.table, k.model == 1 ? row[2] : row[4], cs, turn);
  next.csphi[i] = cs;
  next.turns[i] = turn;
}

// All pairs (ParticleSystemFirstOrder.cpp:162-228, ParticleSystemFirstOrderPtr.cpp:225-316,
// ParticleSystemSecondOrder.cpp:116-177): eight particles a block, two warps
// scanning half the system each for one of them by the float pre-test (FP64
// within the margins of the cutoff, and for every second-order pair not
// certainly out of range).  Every lane adds up the neighbours it finds, each warp
// (for each 2,048 candidates) by their directions or, where NeighbourSums says so,
// by their sines; after the scan eight lanes finish the eight particles, while
// another warp does what does not need the sums: everything of the derivative
// and of the next stage but the torque and omega.  At N = 1,000 the block is a
// chain of latencies (an FP64 instruction's result takes 64 cycles): in a graph of
// RK4 steps an evaluation takes 9.3 us with random phases, 10.3 with all aligned
// (7.7 with directions everywhere, which aligned phases do not allow; 20.5 with a
// library sine in each lane that finds a neighbour).  Two blocks an SM, although 64
// registers a thread spill some: with one 8.7 us here, but 47 in place of 39 at N = 4,000.
constexpr int kAllParticles = 8;
constexpr int kAllWarps = 2 * kAllParticles;

// One scanning warp's sums: of directions and, pair by pair, of near terms and
// forces; the phases of a few near neighbours, whose sines are taken after the
// block meets (16 warps with one each would spend the FP64 pipe on one lane a warp),
// and of the particle.
constexpr int kNears = 8;
constexpr int kNearWarps = kAllWarps * kNears / 32;

struct WarpSums
{
  long long ch, cl, sh, sl;
  int n, nears;
  double wc, ws, near_sum, caf, phi, near[kNears];
};

__device__ __forceinline__ long long warp_add(long long v)
{
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

__device__ __forceinline__ float warp_add(float v)
{
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

__device__ __forceinline__ double warp_add(double v)
{
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  return v;
}

// sin(phi_j - phi_i - alpha), mostly of at most 1/4: the difference with what its
// subtractions rounded off, less the nearest multiple of pi, and the series to
// the eleventh power, in few steps one after the other (an FP64 instruction's
// result takes 64 cycles).
__device__ __noinline__ double near_sine(double phi_i, double phi_j, double alpha)
{
  double d = phi_j - phi_i;
  const double v = d - phi_j;
  double e = (phi_j - (d - v)) - (phi_i + v);
  if (alpha != 0.0)
  {
    const double f = d - alpha, w = f - d;
    e += (d - (f - w)) - (alpha + w);
    d = f;
  }
  double r = d;
  int odd = 0;
  if ((__double2hiint(d) & 0x7fffffff) > 0x3fd0a3d7)  // 0.26
  {
    const double t = fma(d, 0.31830988618379067, SPSS_ROUND_MAGIC);  // 1 / pi
    const double m = t - SPSS_ROUND_MAGIC;
    odd = __double2loint(t) & 1;
    r = fma(m, -0x1.921fb58p+1, d);  // pi in three parts, as pi / 128 in reduce_turn
    r = fma(m, 0x1.dde974p-26, r);
    r = fma(m, -0x1.1a62633145c07p-53, r);
    // phases without a direction have any sine, and as in near_quarter
    const int size = __double2hiint(r) & 0x7fffffff;
    if (!reducible(d) || size > 0x3fd0a3d7 || size < 0x3e100000)
    {
      double s, c;
      sincos(d, &s, &c);
      return fma(c, e, s);
    }
  }
  r += e;
  const double q = r * r;
  const double high = fma(q, -1.0 / 39916800.0, 1.0 / 362880.0), low = fma(q, 1.0 / 120.0, -1.0 / 6.0);
  const double q2 = q * q, cube = r * q;
  const double s = fma(cube, fma(q2, fma(q, high, -1.0 / 5040.0), low), r);
  return odd ? -s : s;
}

// A lane's complementary force over its pairs among the slots j0, j0 + 32, ... below
// end, each by its own cosine (a neighbour's omega is infinite).
__device__ __noinline__ double forces_by_pairs(const K64 &k, const double *rk, const float2 *posf, int i, int j0,
                                               int end)
{
  const double *st = rk + (long) k.s * i;
  PairTerms a;
  for (int j = j0; j < end; j += 32)
  {
    if (j == i) continue;
    const double *sj = rk + (long) k.s * j;
    int in = pretest(posf[i], posf[j], k.rho_incl, k.rho_excl);
    if (in == 1 && k.model == 2) in = 2;
    if (in == 2)
    {
      double x_i = st[0], y_i = st[1];
      if (k.model == 1 && k.flavor == 1)
      {
        x_i = wrap1(x_i);
        y_i = wrap1(y_i);
      }
      in = pair_dr2<false>(k, x_i, y_i, sj[0], sj[1]) <= k.rho2;
    }
    if (in) add_pair(k, a, st[k.s - 2], st[k.s - 1], sj[k.s - 2], sj[k.s - 1]);
  }
  return a.caf.value();
}

template<int AFTER>
__global__ void __launch_bounds__(32 * kAllWarps, 2) f64_allpairs_kernel(const __grid_constant__ K64 k,
                                                                      const double *__restrict__ rk,
                                                                      const float2 *__restrict__ posf,
                                                                      const double2 *__restrict__ csphi,
                                                                      const longlong2 *__restrict__ turns,
                                                                      double *__restrict__ k_next,
                                                                      double *__restrict__ caf, NextStage next)
{
  __shared__ WarpSums sums[kAllWarps];
  pdl_enter();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i0 = blockIdx.x * kAllParticles;
  const int i = i0 + (warp >> 1);
  const int ip = k.model == 1 ? 2 : 4;
  if (lane == 0) sums[warp] = WarpSums{};
  __syncwarp();
  if (i < k.n)
  {
    const double *st = rk + (long) k.s * i;
    const double phi_i = st[ip], omega_i = k.higher_order ? st[ip + 1] : 0.0;
    const longlong2 turn = turns[i];
    const float2 p_i = posf[i], own = own_turned(k, turn);
    const int half = (k.n + 1) / 2;
    const int begin = (warp & 1) ? half : 0, end = (warp & 1) ? k.n : half;
    constexpr int U = 8, kStretch = 32 * 64;  // candidates whose hits a lane remembers
    const bool one_stretch = end - begin <= kStretch;
    NeighbourSums a;
    for (int j0 = begin + lane, at = 0; j0 - lane < end; j0 += 32 * U, at = (at + 1) & 7)
    {
      float2 p[U];
      unsigned hits = 0, unsure = 0;
#pragma unroll
      for (int u = 0; u < U; ++u) p[u] = posf[min(j0 + 32 * u, k.n - 1)];
#pragma unroll
      for (int u = 0; u < U; ++u)
      {
        const int j = j0 + 32 * u;
        int in = pretest(p_i, p[u], k.rho_incl, k.rho_excl);
        if (j >= end || j == i) in = 0;
        if (in == 1 && k.model == 2) in = 2;
        if (in == 1) hits |= 1u << u;
        if (in == 2) unsure |= 1u << u;
      }
      if (unsure)
      {
        double x_i = st[0], y_i = st[1];
        if (k.model == 1 && k.flavor == 1)
        {
          x_i = wrap1(x_i);
          y_i = wrap1(y_i);
        }
        for (; unsure; unsure &= unsure - 1)
        {
          const int u = __ffs(unsure) - 1;
          const double *sj = rk + (long) k.s * (j0 + 32 * u);
          if (pair_dr2<false>(k, x_i, y_i, sj[0], sj[1]) <= k.rho2) hits |= 1u << u;
        }
      }
      if (!__any_sync(0xffffffffu, __popc(hits) > 2))
      {
        // few: one set of loads and sums for most
        for (unsigned rest = hits; rest; rest &= rest - 1) a.add(turns[j0 + 32 * (__ffs(rest) - 1)], own);
      } else
      {
        constexpr int V = 4;
#pragma unroll
        for (int v = 0; v < U; v += V)
        {
          longlong2 d[V];
#pragma unroll
          for (int u = 0; u < V; ++u) d[u] = hits & (1u << (v + u)) ? turns[j0 + 32 * (v + u)] : make_longlong2(0, 0);
#pragma unroll
          for (int u = 0; u < V; ++u) a.add(d[u], own);
        }
      }
      a.close(hits, at);
      if (k.higher_order)
      {
#pragma unroll
        for (int u = 0; u < U; ++u)
          if (hits & (1u << u))
          {
            const int j = j0 + 32 * u;
            const double2 cs = csphi[j];
            const double dw = rk[(long) k.s * j + ip + 1] - omega_i;
            a.wc = fma(dw, cs.x, a.wc);
            a.ws = fma(dw, cs.y, a.ws);
          }
      }
      if (at < 7 && j0 + 32 * U - lane < end) continue;
      // the end of a stretch: the warp's directions, or its sines one by one
      const int first = j0 - 32 * U * at, found = __reduce_add_sync(0xffffffffu, a.n);
      const float sines = warp_add(a.sines);
      const bool apart = __any_sync(0xffffffffu, a.bad < 0) || lacks_direction(turn) || sines < k.least * (float) found;
      WarpSums w{};
      if (!apart)
      {
        w.ch = warp_add(a.ch);
        w.cl = warp_add(a.cl);
        w.sh = warp_add(a.sh);
        w.sl = warp_add(a.sl);
      } else if (found > 0)
      {
        const double *phi = rk + (long) k.s * first + ip;
        if (one_stretch && found <= kNears)
        {
          for (unsigned with; (with = __ballot_sync(0xffffffffu, a.hits != 0)) != 0; w.nears += __popc(with))
          {
            if (!a.hits) continue;
            sums[warp].near[w.nears + __popc(with & ((1u << lane) - 1))] = phi[(long) k.s * 32 * (__ffsll(a.hits) - 1)];
            a.hits &= a.hits - 1;
          }
        } else
        {
          double sum = 0.0;
          for (; a.hits; a.hits &= a.hits - 1)
            sum += near_sine(phi_i, phi[(long) k.s * 32 * (__ffsll(a.hits) - 1)], k.alpha);
          w.near_sum = warp_add(sum);
        }
      }
      if (k.higher_order)
      {
        double force = 0.0;
        if (not_finite(a.wc + a.ws))
        {
          force = forces_by_pairs(k, rk, posf, i, first, min(end, first + kStretch));
          a.wc = a.ws = 0.0;
        }
        w.wc = warp_add(a.wc);
        w.ws = warp_add(a.ws);
        w.caf = warp_add(force);
      }
      if (lane == 0)
      {
        WarpSums &to = sums[warp];
        to.ch += w.ch;
        to.cl += w.cl;
        to.sh += w.sh;
        to.sl += w.sl;
        to.n += found;
        to.nears = w.nears;
        to.near_sum += w.near_sum;
        to.phi = phi_i;
        if (k.higher_order)
        {
          to.wc += w.wc;
          to.ws += w.ws;
          to.caf += w.caf;
        }
      }
      a = NeighbourSums();
    }
  }
  const int g = i0 + lane;
  // the finishing lanes' words, asked for before the block meets
  const bool finisher = warp == 0 && lane < kAllParticles && g < k.n;
  const long at = (long) k.s * (finisher ? g : min(i0, k.n - 1)) + k.s - 1;
  StageWords words{0.0, 0.0, 0.0, 0.0};
  double torque = 0.0, omega = 0.0;
  double2 own = make_double2(0.0, 0.0);
  longlong2 turn = make_longlong2(0, 0);
  if (finisher)
  {
    own = csphi[g];
    turn = turns[g];
    omega = rk[at];
    if (AFTER != AFTER_NOTHING)
    {
      words = load_stage<AFTER>(next, at);
      torque = k_next[at];  // kept where the particle has no neighbour
    }
  }
  __syncthreads();
  if (warp == kAllWarps - 1 && lane < kAllParticles && g < k.n)
  {
    const double2 cs = csphi[g];
    write_k_but_torque(k, g, rk + (long) k.s * g, k_next, cs.x, cs.y);
    if (AFTER != AFTER_NOTHING) advance_but_omega<AFTER>(k, g, k_next, next);
  }
  if (warp >= kNearWarps) return;
  // the near sines: 32 of their places for each of a few warps
  const bool more = __any_sync(0xffffffffu, lane < kAllWarps && sums[lane & (kAllWarps - 1)].nears > 0);
  if (more)
  {
    const int at = 32 * warp + lane;
    WarpSums &of = sums[at / kNears];
    if (at % kNears < of.nears) of.near[at % kNears] = near_sine(of.phi, of.near[at % kNears], k.alpha);
    asm volatile("bar.sync 1, %0;" ::"n"(32 * kNearWarps) : "memory");
  }
  if (!finisher) return;
  const WarpSums &u = sums[2 * lane], &v = sums[2 * lane + 1];
  NeighbourSums a;
  a.ch = u.ch + v.ch;
  a.cl = u.cl + v.cl;
  a.sh = u.sh + v.sh;
  a.sl = u.sl + v.sl;
  a.n = u.n + v.n;
  a.wc = u.wc + v.wc;
  a.ws = u.ws + v.ws;
  Sums r = pair_sums(k, a, own, turn);
  r.af += u.near_sum + v.near_sum;
  for (int t = 0; t < u.nears; ++t) r.af += u.near[t];
  for (int t = 0; t < v.nears; ++t) r.af += v.near[t];
  r.caf += u.caf + v.caf;
  if (r.card != 0.0)
  {
    torque = -(k.model == 1 ? k.xi : k.xi_phi) * omega + k.sigma * r.af / r.card;
    k_next[at] = torque;
    if (k.higher_order) r.caf *= k.sigma / r.card;
  }
  if (k.higher_order) caf[g] = r.caf;
  if (AFTER != AFTER_NOTHING) advance_component<AFTER>(next, at, words, torque);
}

// ------------------------------------------------------------ neighbour sums
//
// One particle per lane finds its neighbours by the float pre-test (FP64 only
// for a pair within the margins of the cutoff) and adds up their directions.
// With a sine a pair (queued, and evaluated by the whole warp) ten steps of
// N = 65,536 took 815 us, and 2,160 once clusters had formed; by sums of
// directions 825 and 1,520, with the linked list's positions and directions
// copied into cell order by the sort (one load, contiguous, before a test in
// place of two) 700 and 1,150, and without branches around the sums (the few
// lanes that need sines included) another 5 % less.
constexpr int kScan = 8;          // candidates a lane looks at together (their loads are in flight at once)
constexpr int kPairThreads = 32;  // one warp a block: 20,011 particles in blocks of 64 left SMs with 3 blocks beside SMs with 2

// Read-only views of what the pair kernels need of every particle.
struct PairInputs
{
  const double *rk;
  const float2 *posf;
  const double2 *csphi;
  const longlong2 *turns;
  const float2 *posf_rows;  // posf and turns in cell order (linked list)
  const longlong2 *turns_rows;
};

// Candidates list[m .. m + kScan) (below e) of the lane's particle: those in
// range are added to its sums.  ROWS: a stretch of the cell list, whose
// positions and directions stand in its order, so a lane waits for one load
// before it tests (the member's index only where it needs more of it); `self`
// is the particle's place there.  Else entries of a Verlet list, `self` the
// particle.
template<bool ROWS>
__device__ __forceinline__ void scan_candidates(const K64 &k, const PairInputs &in, const int *__restrict__ list,
                                                int m, int e, int at, int self, float2 p_i, double x_i, double y_i,
                                                double omega_i, float2 own, NeighbourSums &a)
{
  int j[kScan];
  float2 p[kScan];
  longlong2 d[kScan];
  unsigned hits = 0;
#pragma unroll
  for (int u = 0; u < kScan; ++u) j[u] = m + u < e ? (ROWS ? m + u : __ldg(list + m + u)) : self;
#pragma unroll
  for (int u = 0; u < kScan; ++u) p[u] = __ldg((ROWS ? in.posf_rows : in.posf) + j[u]);
#pragma unroll
  for (int u = 0; u < kScan; ++u)
  {
    int hit = j[u] == self ? 0 : pretest(p_i, p[u], k.rho_incl, k.rho_excl);
    if (hit == 2)
    {
      const double *sj = in.rk + (long) k.s * (ROWS ? __ldg(list + j[u]) : j[u]);
      hit = pair_dr2<true>(k, x_i, y_i, sj[0], sj[1]) <= k.rho2;
    }
    d[u] = hit ? __ldg((ROWS ? in.turns_rows : in.turns) + j[u]) : make_longlong2(0, 0);
    if (hit) hits |= 1u << u;
  }
#pragma unroll
  for (int u = 0; u < kScan; ++u) a.add(d[u], own);
  a.close(hits, at);
  if (k.higher_order)
  {
    // sums of a few terms first: a long list's additions then round less
    double wc = 0.0, ws = 0.0;
#pragma unroll
    for (int u = 0; u < kScan; ++u)
      if (hits & (1u << u))
      {
        const int o = ROWS ? __ldg(list + j[u]) : j[u];
        const double2 cs = __ldg(in.csphi + o);
        const double dw = __ldg(in.rk + (long) k.s * o + k.s - 1) - omega_i;
        wc = fma(dw, cs.x, wc);
        ws = fma(dw, cs.y, ws);
      }
    a.wc += wc;
    a.ws += ws;
  }
}

// The candidates of one such set again, those in range by their own sines: known
// from the first scan (`hits`) or, beyond its first 64, tested again.
template<bool ROWS>
__device__ __forceinline__ void candidate_terms(const K64 &k, const PairInputs &in, const int *__restrict__ list, int m,
                                                int e, int at, unsigned long long hits, int i, double x_i, double y_i,
                                                const double *st, PairTerms &a)
{
  unsigned set = at < 8 ? (unsigned) (hits >> (8 * at)) & 255u : (1u << min(e - m, kScan)) - 1u;
  for (; set; set &= set - 1)
  {
    const int o = list[m + __ffs(set) - 1];
    const double *sj = in.rk + (long) k.s * o;
    if (at >= 8)
    {
      int hit = o == i ? 0 : pretest(in.posf[i], in.posf[o], k.rho_incl, k.rho_excl);
      if (hit == 2) hit = pair_dr2<true>(k, x_i, y_i, sj[0], sj[1]) <= k.rho2;
      if (!hit) continue;
    }
    add_pair(k, a, st[k.s - 2], st[k.s - 1], sj[k.s - 2], sj[k.s - 1]);
  }
}

// The stencil of a cell as runs of the cell list, in the reference's order: a
// row of three cells away from the grid's edge is one run, cells at the edge
// are runs of their own.  `c` counts the stencil's cells done.
__device__ __forceinline__ void next_run(int cx, int cy, int nc, const int *__restrict__ off, int &c, int &m, int &e)
{
  const int row = adjust_cell(cy + c_stencil[c][1], nc) * nc;
  if (cx > 0 && cx + 1 < nc)
  {
    m = off[row + cx - 1];
    e = off[row + cx + 2];
    c += 3;
    return;
  }
  const int jc = row + adjust_cell(cx + c_stencil[c][0], nc);
  m = off[jc];
  e = off[jc + 1];
  ++c;
}

// The pair sums of one particle pair by pair, in the reference's order: from the
// cell list, and from its Verlet list.
__device__ __noinline__ double2 linked_list_terms(const K64 &k, const PairInputs &in, int nc, const int *off,
                                               const int *mem, int t, unsigned long long hits)
{
  const int i = mem[t];
  double x_i, y_i;
  pos_for_cells(k, in.rk, i, x_i, y_i);
  const int cx = cell_coord(x_i, nc), cy = cell_coord(y_i, nc);
  PairTerms a;
  int at = 0;
  for (int c = 0; c < 9;)
  {
    int m, e;
    next_run(cx, cy, nc, off, c, m, e);
    for (; m < e; m += kScan, ++at)
      candidate_terms<true>(k, in, mem, m, e, at, hits, i, x_i, y_i, in.rk + (long) k.s * i, a);
  }
  return a.values();
}

__device__ __noinline__ double2 verlet_terms(const K64 &k, const PairInputs &in, const int *vl_off, const int *vl_ent,
                                          int i, unsigned long long hits)
{
  const double *st = in.rk + (long) k.s * i;
  double x_i = st[0], y_i = st[1];
  if (k.model == 2) wrap_if_outside(x_i, y_i);
  PairTerms a;
  const int e = vl_off[i + 1];
  int at = 0;
  for (int m = vl_off[i]; m < e; m += kScan, ++at)
    candidate_terms<false>(k, in, vl_ent, m, e, at, hits, i, x_i, y_i, st, a);
  return a.values();
}

// Linked list (ParticleSystemFirstOrder.cpp:231-353, ParticleSystemSecondOrder.cpp:276-409).
// Particles are taken in cell order, so a warp's lanes scan neighbouring cells.
__global__ void __launch_bounds__(kPairThreads) f64_linked_list_kernel(const __grid_constant__ K64 k,
                                                                       const __grid_constant__ PairInputs in, int nc,
                                                                       const int *__restrict__ off,
                                                                       const int *__restrict__ mem,
                                                                       double *__restrict__ k_next,
                                                                       double *__restrict__ caf)
{
  pdl_enter();
  const int t = blockIdx.x * kPairThreads + threadIdx.x;
  if (t >= k.n) return;
  const int i = mem[t];
  const double *st = in.rk + (long) k.s * i;
  double x_i, y_i;
  pos_for_cells(k, in.rk, i, x_i, y_i);
  const double omega_i = st[k.s - 1];
  const float2 p_i = in.posf[i];
  const int cx = cell_coord(x_i, nc), cy = cell_coord(y_i, nc);
  const longlong2 turn = in.turns[i];
  const float2 own_f = own_turned(k, turn);
  NeighbourSums a;
  int at = 0;
  for (int c = 0; c < 9;)
  {
    int m, e;
    next_run(cx, cy, nc, off, c, m, e);
    for (; m < e; m += kScan, ++at) scan_candidates<true>(k, in, mem, m, e, at, t, p_i, x_i, y_i, omega_i, own_f, a);
  }
  const double2 own = in.csphi[i];
  Sums r = pair_sums(k, a, own, turn);
  if (needs_pairs(k, a, turn)) r.take(linked_list_terms(k, in, nc, off, mem, t, a.hits));
  write_k(k, i, st, own, r, k_next, caf);
}

// Verlet list from the cell list (ParticleSystemFirstOrder.cpp:536-589): first
// pass counts, second pass fills in the reference's push_back order.  Almost
// every pair is decided by the float pre-test (N = 20,011: 97 + 83 us with the
// FP64 distance for every candidate, 22 + 24 us with it).
template<bool FILL>
__global__ void f64_verlet_cells_kernel(K64 k, const double *__restrict__ rk, const float2 *__restrict__ posf, int nc,
                                        const int *__restrict__ off, const int *__restrict__ mem,
                                        int *__restrict__ count, const int *__restrict__ vl_off,
                                        int *__restrict__ vl_ent)
{
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= k.n) return;
  const int i = mem[t];
  double x_i, y_i;
  pos_for_cells(k, rk, i, x_i, y_i);
  const float2 p_i = posf[i];
  const int cx = cell_coord(x_i, nc), cy = cell_coord(y_i, nc);
  int cnt = 0;
  const int base = FILL ? vl_off[i] : 0;
  for (int c = 0; c < 9;)
  {
    int m, e;
    next_run(cx, cy, nc, off, c, m, e);
    for (; m < e; m += kScan)
    {
      int j[kScan];
      float2 p[kScan];
#pragma unroll
      for (int u = 0; u < kScan; ++u) j[u] = m + u < e ? __ldg(mem + m + u) : i;
#pragma unroll
      for (int u = 0; u < kScan; ++u) p[u] = __ldg(posf + j[u]);
#pragma unroll
      for (int u = 0; u < kScan; ++u)
      {
        int in = j[u] == i ? 0 : pretest(p_i, p[u], k.rmax_incl, k.rmax_excl);
        if (in == 2)
        {
          const double *sj = rk + (long) k.s * j[u];
          in = pair_dr2<true>(k, x_i, y_i, sj[0], sj[1]) <= k.rmax2;
        }
        if (in)
        {
          if (FILL) vl_ent[base + cnt] = j[u];
          ++cnt;
        }
      }
    }
  }
  if (!FILL) count[i] = cnt;
}

// Verlet list by an O(N^2) scan (ParticleSystemFirstOrder.cpp:376-422).
template<bool FILL>
__global__ void f64_verlet_all_kernel(K64 k, const double *__restrict__ rk, int *__restrict__ count,
                                      const int *__restrict__ vl_off, int *__restrict__ vl_ent)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= k.n) return;
  double x_i = rk[(long) k.s * i], y_i = rk[(long) k.s * i + 1];
  if (k.model == 2) wrap_if_outside(x_i, y_i);
  int cnt = 0;
  const int base = FILL ? vl_off[i] : 0;
  for (int j = 0; j < k.n; ++j)
  {
    if (j == i) continue;
    if (pair_dr2<true>(k, x_i, y_i, rk[(long) k.s * j], rk[(long) k.s * j + 1]) <= k.rmax2)
    {
      if (FILL) vl_ent[base + cnt] = j;
      ++cnt;
    }
  }
  if (!FILL) count[i] = cnt;
}

// Pair loop over the Verlet list (ParticleSystemFirstOrder.cpp:594-648, ParticleSystemFirstOrderPtr.cpp:861-930).
// `order` (not null): particles in the cell order of the last build, so a
// warp's lanes read neighbouring particles.
__global__ void __launch_bounds__(kPairThreads) f64_verlet_pairs_kernel(const __grid_constant__ K64 k,
                                                                        const __grid_constant__ PairInputs in,
                                                                        const int *__restrict__ order,
                                                                        const int *__restrict__ vl_off,
                                                                        const int *__restrict__ vl_ent,
                                                                        double *__restrict__ k_next,
                                                                        double *__restrict__ caf)
{
  pdl_enter();
  const int t = blockIdx.x * kPairThreads + threadIdx.x;
  if (t >= k.n) return;
  const int i = order ? order[t] : t;
  const double *st = in.rk + (long) k.s * i;
  double x_i = st[0], y_i = st[1];
  if (k.model == 2) wrap_if_outside(x_i, y_i);
  const double omega_i = st[k.s - 1];
  const float2 p_i = in.posf[i];
  const longlong2 turn = in.turns[i];
  const float2 own_f = own_turned(k, turn);
  NeighbourSums a;
  const int e = vl_off[i + 1];
  int at = 0;
  for (int m = vl_off[i]; m < e; m += kScan, ++at)
    scan_candidates<false>(k, in, vl_ent, m, e, at, i, p_i, x_i, y_i, omega_i, own_f, a);
  const double2 own = in.csphi[i];
  Sums r = pair_sums(k, a, own, turn);
  if (needs_pairs(k, a, turn)) r.take(verlet_terms(k, in, vl_off, vl_ent, i, a.hits));
  write_k(k, i, st, own, r, k_next, caf);
}

// Global polar order field, first order (ParticleSystemFirstOrder.cpp:122-159,
// ParticleSystemFirstOrderPtr.cpp:155-223): block partial sums, then one block
// adds them in a fixed order.
__global__ void f64_field_partials_kernel(K64 k, const double *__restrict__ rk, double *__restrict__ partials)
{
  __shared__ double sh[4][256];
  double acc[4] = {0.0, 0.0, 0.0, 0.0};
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < k.n; i += gridDim.x * blockDim.x)
  {
    const double phi = rk[(long) k.s * i + 2], om = rk[(long) k.s * i + 3];
    const double c = cos(phi), s = sin(phi);
    acc[0] += c;
    acc[1] += s;
    acc[2] += om * c;
    acc[3] += om * s;
  }
  for (int q = 0; q < 4; ++q) sh[q][threadIdx.x] = acc[q];
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1)
  {
    if ((int) threadIdx.x < w)
      for (int q = 0; q < 4; ++q) sh[q][threadIdx.x] += sh[q][threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0)
    for (int q = 0; q < 4; ++q) partials[4 * blockIdx.x + q] = sh[q][0];
}

__global__ void f64_field_apply_kernel(K64 k, const double *__restrict__ rk, const double *__restrict__ partials,
                                       int nparts, const double *__restrict__ nat_freq, double *__restrict__ k_next,
                                       double *__restrict__ caf)
{
  double tot[4] = {0.0, 0.0, 0.0, 0.0};
  for (int b = 0; b < nparts; ++b)
    for (int q = 0; q < 4; ++q) tot[q] += partials[4 * b + q];
  const double pre = tot[0] / k.n, pim = tot[1] / k.n, wre = tot[2] / k.n, wim = tot[3] / k.n;
  const double pabs = hypot(pre, pim), parg = atan2(pim, pre);
  const double wabs = hypot(wre, wim), warg = atan2(wim, wre);
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= k.n) return;
  const long ii = (long) k.s * i;
  const double phi_i = rk[ii + 2], omega_i = rk[ii + 3];
  k_next[ii] = k.v0 * cos(phi_i);
  k_next[ii + 1] = k.v0 * sin(phi_i);
  k_next[ii + 2] = omega_i;
  k_next[ii + 3] = -k.xi * omega_i + nat_freq[i]
      + k.sigma * pabs * (sin(parg - phi_i) * k.ca - cos(parg - phi_i) * k.sa);
  if (k.flavor == 1 && k.higher_order)
  {
    // the last sine uses arg(weighted field) as ParticleSystemFirstOrderPtr.cpp:219 does
    caf[i] = k.sigma * (wabs * (cos(warg - phi_i) * k.ca + sin(warg - phi_i) * k.sa)
        - omega_i * pabs * (cos(parg - phi_i) * k.ca + sin(warg - phi_i) * k.sa));
  }
}

// ------------------------------------------------------------ steppers

// RK4 combine (RungeKutta4Stepper.cpp:56-59): td = (k1 + 2 k2 + 2 k3 + k4) dt / 6; x += td.
__global__ void f64_rk4_combine_kernel(double *__restrict__ x, const double *__restrict__ k1,
                                       const double *__restrict__ k2, const double *__restrict__ k3,
                                       const double *__restrict__ k4, double *__restrict__ td, long len, double dt)
{
  const long q = (long) blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= len) return;
  const double d = (k1[q] + 2.0 * k2[q] + 2.0 * k3[q] + k4[q]) * dt / 6.0;
  td[q] = d;
  x[q] += d;
}

// Where a stepper leaves the largest squared displacement of its step for the
// Verlet trigger (ParticleSystemFirstOrder.cpp:672-684): `host` is page-locked,
// `max2` and `ticket` are zero between launches.  max2 null: not asked for.
struct MaxOut
{
  unsigned long long *max2, *host;
  unsigned *ticket;
};

// Non-negative doubles order like their bit patterns; NaN counts as 0.  All
// threads of all blocks; the last block hands the maximum to the host (a kernel
// over the displacements, a copy and two clears, as it was, took 6 us a step).
__device__ __forceinline__ void publish_max2(const MaxOut &m, double2 d)
{
  if (!m.max2) return;
  const double d2 = d.x * d.x + d.y * d.y;
  unsigned long long v = d2 > 0.0 ? (unsigned long long) __double_as_longlong(d2) : 0ull;
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v = max(v, __shfl_xor_sync(0xffffffffu, v, off));
  if ((threadIdx.x & 31) == 0 && v > *(volatile unsigned long long *) m.max2) atomicMax(m.max2, v);
  __threadfence();
  __syncthreads();
  if (threadIdx.x != 0 || atomicAdd(m.ticket, 1u) != gridDim.x - 1) return;
  __threadfence();
  *m.ticket = 0u;
  *m.host = atomicExch(m.max2, 0ull);
}

// Second-order stochastic Euler (StochasticEulerStepper.hpp:33-51 with
// ParticleSystemSecondOrder::AddNoise, ParticleSystemSecondOrder.cpp:439-451).
__device__ __forceinline__ double2 se2_particle(int i, double *__restrict__ x, const double *__restrict__ det,
                                                double *__restrict__ td, double dt, double sqrt_dt,
                                                double intensity_r, double intensity_phi, NoiseKey nk,
                                                const double2 *__restrict__ table)
{
  const uint4 u = philox_block(nk, (uint32_t) i, 0);
  // without translational noise (intensity_r = 0) its two normals multiply 0
  double z[4] = {0.0, 0.0, 0.0, 0.0};
  if (intensity_r != 0.0) box_muller_f64(table, u.x, u.y, z[0], z[1]);
  box_muller_f64(table, u.z, u.w, z[2], z[3]);
  double2 *t2 = reinterpret_cast<double2 *>(td + 6L * i);
  double2 *x2 = reinterpret_cast<double2 *>(x + 6L * i);
  const double2 *d2 = reinterpret_cast<const double2 *>(det + 6L * i);
  const double2 dr = d2[0], dv = d2[1], dp = d2[2];
  const double2 tr = make_double2(dt * dr.x, dt * dr.y);
  const double2 tv = make_double2(dt * dv.x + sqrt_dt * (intensity_r * z[0]), dt * dv.y + sqrt_dt * (intensity_r * z[1]));
  const double2 tp = make_double2(dt * dp.x, dt * dp.y + sqrt_dt * (intensity_phi * z[2]));
  t2[0] = tr;
  t2[1] = tv;
  t2[2] = tp;
  const double2 a = x2[0], b = x2[1], c = x2[2];
  x2[0] = make_double2(a.x + tr.x, a.y + tr.y);
  x2[1] = make_double2(b.x + tv.x, b.y + tv.y);
  x2[2] = make_double2(c.x + tp.x, c.y + tp.y);
  return tr;
}

__global__ void f64_se2_kernel(double *__restrict__ x, const double *__restrict__ det, double *__restrict__ td,
                               int n, double dt, double sqrt_dt, double intensity_r, double intensity_phi,
                               NoiseKey nk, const double2 *__restrict__ table, MaxOut m)
{
  pdl_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double2 moved = make_double2(0.0, 0.0);
  if (i < n) moved = se2_particle(i, x, det, td, dt, sqrt_dt, intensity_r, intensity_phi, nk, table);
  publish_max2(m, moved);
}

// First-order stochastic Euler (StochasticEulerStepperPtr.hpp:40-73).
__device__ __forceinline__ double2 se1_particle(int i, double *__restrict__ x, const double *__restrict__ d,
                                                double *__restrict__ td, double dt, double sqrt_dt,
                                                double intensity_phi, NoiseKey nk,
                                                const double2 *__restrict__ table)
{
  double z[2];
  normals_f64<1>(table, nk, (uint32_t) i, 0, z);
  const double delta_W_phi = sqrt_dt * z[0];
  const long ii = 4L * i;
  td[ii] = d[ii] * dt;
  td[ii + 1] = d[ii + 1] * dt;
  td[ii + 2] = d[ii + 2] * dt;
  td[ii + 3] = d[ii + 3] * dt + intensity_phi * delta_W_phi;
  for (int s = 0; s < 4; ++s) x[ii + s] += td[ii + s];
  return make_double2(td[ii], td[ii + 1]);
}

__global__ void f64_se1_kernel(double *__restrict__ x, const double *__restrict__ d, double *__restrict__ td,
                               int n, double dt, double sqrt_dt, double intensity_phi, NoiseKey nk,
                               const double2 *__restrict__ table, MaxOut m)
{
  pdl_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double2 moved = make_double2(0.0, 0.0);
  if (i < n) moved = se1_particle(i, x, d, td, dt, sqrt_dt, intensity_phi, nk, table);
  publish_max2(m, moved);
}

// First-order strong order 1.5 Taylor scheme (StochasticRungeKuttaStepperPtr.hpp:40-76).
__device__ __forceinline__ double2 srk1_particle(int i, double *__restrict__ x, const double *__restrict__ d,
                                                 const double *__restrict__ caf, double *__restrict__ td,
                                                 double dt, double sqrt_dt, double dt15, double inv_sqrt3,
                                                 double sqrt_2noise, double friction, NoiseKey nk,
                                                 const double2 *__restrict__ table)
{
  double z[2];
  normals_f64<1>(table, nk, (uint32_t) i, 0, z);
  const double U_1 = z[0], U_2 = z[1];
  const double delta_W_i = U_1 * sqrt_dt;
  const double delta_Z_i = 0.5 * dt15 * (U_1 + inv_sqrt3 * U_2);
  const long ii = 4L * i;
  td[ii] = d[ii] * dt - 0.5 * d[ii + 2] * d[ii + 1] * dt * dt;
  td[ii + 1] = d[ii + 1] * dt + 0.5 * d[ii + 2] * d[ii] * dt * dt;
  td[ii + 2] = d[ii + 2] * dt + 0.5 * d[ii + 3] * dt * dt + sqrt_2noise * delta_Z_i;
  td[ii + 3] = d[ii + 3] * dt + 0.5 * (caf[i] - friction * d[ii + 3]) * dt * dt
      + sqrt_2noise * (delta_W_i - friction * delta_Z_i);
  for (int s = 0; s < 4; ++s) x[ii + s] += td[ii + s];
  return make_double2(td[ii], td[ii + 1]);
}

__global__ void f64_srk1_kernel(double *__restrict__ x, const double *__restrict__ d,
                                const double *__restrict__ caf, double *__restrict__ td, int n, double dt,
                                double sqrt_dt, double dt15, double inv_sqrt3, double sqrt_2noise, double friction,
                                NoiseKey nk, const double2 *__restrict__ table, MaxOut m)
{
  pdl_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double2 moved = make_double2(0.0, 0.0);
  if (i < n) moved = srk1_particle(i, x, d, caf, td, dt, sqrt_dt, dt15, inv_sqrt3, sqrt_2noise, friction, nk, table);
  publish_max2(m, moved);
}

// Second-order strong order 1.5 Taylor scheme (no reference code): the
// first-order scheme's construction applied to the second-order drift with
// additive noise on v_x, v_y (b_r) and omega (b_phi); see spss_oracle.c.
__device__ __forceinline__ double2 srk2_particle(int i, double *__restrict__ x, const double *__restrict__ d,
                                                 const double *__restrict__ caf, double *__restrict__ td,
                                                 double dt, double sqdt, double dt15, double inv_sqrt3, double b_r,
                                                 double b_phi, double xi_r, double xi_phi, double v0, NoiseKey nk,
                                                 const double2 *__restrict__ table)
{
  double u[6] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
  if (b_r != 0.0) normals_f64<2>(table, nk, (uint32_t) i, 0, u);  // b_r = 0 multiplies them
  normals_f64<1>(table, nk, (uint32_t) i, 1, u + 4);
  const double dWx = u[0] * sqdt, dZx = 0.5 * dt15 * (u[0] + inv_sqrt3 * u[1]);
  const double dWy = u[2] * sqdt, dZy = 0.5 * dt15 * (u[2] + inv_sqrt3 * u[3]);
  const double dWw = u[4] * sqdt, dZw = 0.5 * dt15 * (u[4] + inv_sqrt3 * u[5]);
  const long ii = 6L * i;
  double cphi, sphi;
  fast_sincos(table, x[ii + 4], sphi, cphi);
  td[ii] = d[ii] * dt + 0.5 * d[ii + 2] * dt * dt + b_r * dZx;
  td[ii + 1] = d[ii + 1] * dt + 0.5 * d[ii + 3] * dt * dt + b_r * dZy;
  td[ii + 2] = d[ii + 2] * dt + 0.5 * (-xi_r * d[ii + 2] - v0 * sphi * d[ii + 4]) * dt * dt + b_r * (dWx - xi_r * dZx);
  td[ii + 3] = d[ii + 3] * dt + 0.5 * (-xi_r * d[ii + 3] + v0 * cphi * d[ii + 4]) * dt * dt + b_r * (dWy - xi_r * dZy);
  td[ii + 4] = d[ii + 4] * dt + 0.5 * d[ii + 5] * dt * dt + b_phi * dZw;
  td[ii + 5] = d[ii + 5] * dt + 0.5 * (caf[i] - xi_phi * d[ii + 5]) * dt * dt + b_phi * (dWw - xi_phi * dZw);
  for (int s = 0; s < 6; ++s) x[ii + s] += td[ii + s];
  return make_double2(td[ii], td[ii + 1]);
}

__global__ void f64_srk2_kernel(double *__restrict__ x, const double *__restrict__ d,
                                const double *__restrict__ caf, double *__restrict__ td, int n, double dt,
                                double sqdt, double dt15, double inv_sqrt3, double b_r, double b_phi, double xi_r,
                                double xi_phi, double v0, NoiseKey nk, const double2 *__restrict__ table,
                                MaxOut m)
{
  pdl_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  double2 moved = make_double2(0.0, 0.0);
  if (i < n) moved = srk2_particle(i, x, d, caf, td, dt, sqdt, dt15, inv_sqrt3, b_r, b_phi, xi_r, xi_phi, v0, nk,
                               table);
  publish_max2(m, moved);
}

// max_i (dx^2 + dy^2) of a displacement array (ParticleSystemFirstOrder.cpp:672-684);
// non-negative doubles order like their bit patterns.
__global__ void f64_max2_kernel(const double *__restrict__ td, int n, int s, unsigned long long *__restrict__ out)
{
  __shared__ double sh[256];
  double m = 0.0;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
  {
    const double dx = td[(long) s * i], dy = td[(long) s * i + 1];
    const double d2 = dx * dx + dy * dy;
    if (m < d2) m = d2;
  }
  sh[threadIdx.x] = m;
  __syncthreads();
  for (int w = blockDim.x / 2; w > 0; w >>= 1)
  {
    if ((int) threadIdx.x < w && sh[threadIdx.x] < sh[threadIdx.x + w]) sh[threadIdx.x] = sh[threadIdx.x + w];
    __syncthreads();
  }
  if (threadIdx.x == 0) atomicMax(out, (unsigned long long) __double_as_longlong(sh[0]));
}

__global__ void f64_noise_kernel(double *__restrict__ out, int n, int per, NoiseKey nk,
                                 const double2 *__restrict__ table)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  double u[6];
  normals_f64<2>(table, nk, (uint32_t) i, 0, u);
  if (per > 4) normals_f64<1>(table, nk, (uint32_t) i, 1, u + 4);
  for (int d = 0; d < per; ++d) out[(long) per * i + d] = u[d];
}

// ApplyPeriodicBoundaryConditions(system_state) (PeriodicBoundaryConditions.cpp:127-135).
__global__ void f64_pbc_kernel(double *__restrict__ x, int n, int s)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const long ii = (long) s * i;
  x[ii] -= floor(x[ii] * 1.0) * 1.0;
  x[ii + 1] -= floor(x[ii + 1] * 1.0) * 1.0;
}

// ------------------------------------------------------------ host side

static inline int blocks_for(long n, int tb)
{
  return (int) ((n + tb - 1) / tb);
}

int f64_create(spss_ctx *ctx)
{
  F64Path *f = new F64Path();
  ctx->f64 = f;
  const long len = (long) ctx->p.n * ctx->s;
  SPSS_TRY(f->state.reserve(len));
  SPSS_TRY(f->rk.reserve(len));
  for (auto &kb : f->k) SPSS_TRY(kb.reserve(len));
  SPSS_TRY(f->td.reserve(len));
  SPSS_TRY(f->det.reserve(len));
  SPSS_TRY(f->caf.reserve(ctx->p.n));
  SPSS_TRY(f->nat_freq.reserve(ctx->p.n));
  SPSS_TRY(f->cell_of.reserve(ctx->p.n));
  SPSS_TRY(f->posf.reserve(ctx->p.n));
  SPSS_TRY(f->csphi.reserve(ctx->p.n));
  SPSS_TRY(f->turns.reserve(ctx->p.n));
  SPSS_TRY(f->vl_count.reserve(ctx->p.n));
  SPSS_TRY(f->vl_off.reserve(ctx->p.n + 1));
  SPSS_TRY(f->max2.reserve(3));  // of an array of displacements; a stepper's, and its count of finished blocks
  SPSS_CUDA_TRY(cudaMemsetAsync(f->max2.ptr, 0, 3 * sizeof(unsigned long long), ctx->stream));
  SPSS_TRY(f->partials.reserve(4 * 1024));
  SPSS_TRY(make_f64_tables(f->table, ctx->stream));
  SPSS_CUDA_TRY(cudaMallocHost((void **) &f->h_max2, sizeof(unsigned long long)));
  SPSS_CUDA_TRY(cudaMemsetAsync(f->state.ptr, 0, sizeof(double) * len, ctx->stream));
  for (auto &kb : f->k) SPSS_CUDA_TRY(cudaMemsetAsync(kb.ptr, 0, sizeof(double) * len, ctx->stream));
  SPSS_CUDA_TRY(cudaMemsetAsync(f->caf.ptr, 0, sizeof(double) * ctx->p.n, ctx->stream));
  // empty lists until the first build, as the reference's
  SPSS_CUDA_TRY(cudaMemsetAsync(f->vl_off.ptr, 0, sizeof(int) * (ctx->p.n + 1), ctx->stream));
  SPSS_CUDA_TRY(cudaMemsetAsync(f->nat_freq.ptr, 0, sizeof(double) * ctx->p.n, ctx->stream));
  return SPSS_OK;
}

void f64_destroy(spss_ctx *ctx)
{
  F64Path *f = ctx->f64;
  if (!f) return;
  f->state.release();
  f->rk.release();
  for (auto &kb : f->k) kb.release();
  f->td.release();
  f->det.release();
  f->caf.release();
  f->nat_freq.release();
  f->partials.release();
  f->scratch_state.release();
  f->scratch_kprev.release();
  f->scratch_knext.release();
  f->cell_of.release();
  f->posf.release();
  f->csphi.release();
  f->turns.release();
  f->posf_rows.release();
  f->turns_rows.release();
  f->table.release();
  f->rk2.release();
  f->posf2.release();
  f->csphi2.release();
  f->turns2.release();
  if (f->rk4_exec) cudaGraphExecDestroy(f->rk4_exec);
  if (f->rk4_graph) cudaGraphDestroy(f->rk4_graph);
  f->binner.release();
  f->vl_count.release();
  f->vl_off.release();
  f->vl_ent.release();
  f->max2.release();
  if (f->h_max2) cudaFreeHost(f->h_max2);
  delete f;
  ctx->f64 = nullptr;
}

int f64_set_state(spss_ctx *ctx, const double *d_aos)
{
  const long len = (long) ctx->p.n * ctx->s;
  SPSS_CUDA_TRY(cudaMemcpyAsync(ctx->f64->state.ptr, d_aos, sizeof(double) * len, cudaMemcpyDefault,
                                ctx->stream));
  return SPSS_OK;
}

int f64_get_state(spss_ctx *ctx, double *d_aos)
{
  const long len = (long) ctx->p.n * ctx->s;
  SPSS_CUDA_TRY(cudaMemcpyAsync(d_aos, ctx->f64->state.ptr, sizeof(double) * len, cudaMemcpyDefault,
                                ctx->stream));
  return SPSS_OK;
}

int f64_state_ptr(spss_ctx *ctx, const double **d_aos)
{
  *d_aos = ctx->f64->state.ptr;
  return SPSS_OK;
}

static int build_cells(spss_ctx *ctx, const K64 &k, int nc)
{
  F64Path *f = ctx->f64;
  const int tb = 256;
  f64_cell_kernel<<<blocks_for(k.n, tb), tb, 0, ctx->stream>>>(k, f->rk.ptr, nc, f->cell_of.ptr);
  ++ctx->launches;
  SPSS_TRY(check_launch("f64_cell_kernel"));
  SPSS_TRY(f->binner.run(f->cell_of.ptr, k.n, nc * nc, ctx->stream, ctx->launches));
  f->cells_nc = nc;
  return SPSS_OK;
}

static int build_verlet(spss_ctx *ctx, const K64 &k, bool from_cells)
{
  F64Path *f = ctx->f64;
  const int tb = 128;
  if (from_cells)
  {
    SPSS_TRY(build_cells(ctx, k, ctx->nc_verlet));
    f64_verlet_cells_kernel<false><<<blocks_for(k.n, tb), tb, 0, ctx->stream>>>(
        k, f->rk.ptr, f->posf.ptr, ctx->nc_verlet, f->binner.offsets.ptr, f->binner.members.ptr, f->vl_count.ptr, nullptr,
        nullptr);
  } else
  {
    f64_verlet_all_kernel<false><<<blocks_for(k.n, tb), tb, 0, ctx->stream>>>(k, f->rk.ptr, f->vl_count.ptr,
                                                                               nullptr, nullptr);
  }
  ++ctx->launches;
  SPSS_TRY(check_launch("f64_verlet_count"));
  SPSS_TRY(f->binner.scanner.run(f->vl_count.ptr, f->vl_off.ptr, k.n, ctx->stream, ctx->launches));
  int total = 0;
  SPSS_CUDA_TRY(cudaMemcpyAsync(&total, f->vl_off.ptr + k.n, sizeof(int), cudaMemcpyDeviceToHost, ctx->stream));
  SPSS_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  SPSS_TRY(f->vl_ent.reserve(total > 0 ? total : 1));
  if (from_cells)
  {
    f64_verlet_cells_kernel<true><<<blocks_for(k.n, tb), tb, 0, ctx->stream>>>(
        k, f->rk.ptr, f->posf.ptr, ctx->nc_verlet, f->binner.offsets.ptr, f->binner.members.ptr, nullptr, f->vl_off.ptr,
        f->vl_ent.ptr);
  } else
  {
    f64_verlet_all_kernel<true><<<blocks_for(k.n, tb), tb, 0, ctx->stream>>>(k, f->rk.ptr, nullptr, f->vl_off.ptr,
                                                                              f->vl_ent.ptr);
  }
  ++ctx->launches;
  SPSS_TRY(check_launch("f64_verlet_fill"));
  f->vl_total = total;
  f->vl_built = 1;
  return SPSS_OK;
}

// `det` (not null): cleared as a derivative whose torque components nothing adds to.
static int evaluate(spss_ctx *ctx, int variant, const double *d_state, const double *d_kprev, double *d_knext,
                    double k_coef, double dt, double *det)
{
  F64Path *f = ctx->f64;
  variant = variant_for(ctx, variant);
  if (variant < SPSS_VARIANT_ALL_PAIRS || variant > SPSS_VARIANT_GLOBAL_FIELD) return SPSS_ERR_INVALID_ARGUMENT;
  if (variant == SPSS_VARIANT_GLOBAL_FIELD && ctx->p.model != 1) return SPSS_ERR_NOT_SUPPORTED;
  const K64 k = make_k64(ctx);
  const int tb = 256;
  if (variant == SPSS_VARIANT_ALL_PAIRS)
    f64_stage_posf_kernel<<<blocks_for(k.n, tb), tb, 0, ctx->stream>>>(k, d_state, d_kprev, f->rk.ptr, f->posf.ptr,
                                                                       f->csphi.ptr, f->turns.ptr, k_coef, dt);
  else
  {
    StageCells cells{0, nullptr, nullptr, nullptr};
    if (variant == SPSS_VARIANT_LINKED_LIST)
    {
      SPSS_TRY(f->binner.prepare(k.n, ctx->nc * ctx->nc, ctx->stream));
      SPSS_TRY(f->posf_rows.reserve(k.n));
      SPSS_TRY(f->turns_rows.reserve(k.n));
      cells = StageCells{ctx->nc, f->cell_of.ptr, f->binner.count.ptr, f->binner.slot.ptr};
    }
    f64_stage_kernel<<<blocks_for(k.n, tb), tb, 0, ctx->stream>>>(
        k, d_state, d_kprev, f->rk.ptr, variant == SPSS_VARIANT_GLOBAL_FIELD ? nullptr : f->posf.ptr, f->csphi.ptr,
        f->turns.ptr, k_coef, dt, det, cells);
  }
  ++ctx->launches;
  SPSS_TRY(check_launch("f64_stage_kernel"));
  const PairInputs in{f->rk.ptr,    f->posf.ptr,      f->csphi.ptr,
                      f->turns.ptr, f->posf_rows.ptr, f->turns_rows.ptr};
  // the pair kernels write every complementary force
  if (k.higher_order && variant == SPSS_VARIANT_GLOBAL_FIELD) SPSS_CUDA_TRY(cudaMemsetAsync(f->caf.ptr, 0, sizeof(double) * k.n, ctx->stream));
  switch (variant)
  {
    case SPSS_VARIANT_ALL_PAIRS:
      f64_allpairs_kernel<AFTER_NOTHING><<<blocks_for(k.n, kAllParticles), 32 * kAllWarps, 0, ctx->stream>>>(
          k, f->rk.ptr, f->posf.ptr, f->csphi.ptr, f->turns.ptr, d_knext, f->caf.ptr, NextStage{});
      ++ctx->launches;
      return check_launch("f64_allpairs_kernel");
    case SPSS_VARIANT_LINKED_LIST:
      SPSS_TRY(f->binner.finish(f->cell_of.ptr, k.n, ctx->stream, ctx->launches, true,
                                BinRows{f->posf.ptr, f->turns.ptr, f->posf_rows.ptr, f->turns_rows.ptr}));
      f->cells_nc = ctx->nc;
      SPSS_CUDA_TRY(launch_chained(true, f64_linked_list_kernel, blocks_for(k.n, kPairThreads), kPairThreads, 0,
                                   ctx->stream, k, in, ctx->nc, (const int *) f->binner.offsets.ptr,
                                   (const int *) f->binner.members.ptr, d_knext, f->caf.ptr));
      ++ctx->launches;
      return check_launch("f64_linked_list_kernel");
    case SPSS_VARIANT_VERLET:
    case SPSS_VARIANT_LINKED_LIST_VERLET:
    {
      const bool build = ctx->should_update_lists;
      if (build)
      {
        SPSS_TRY(build_verlet(ctx, k, variant == SPSS_VARIANT_LINKED_LIST_VERLET));
        ctx->should_update_lists = 0;
        ++ctx->list_builds;
      }
      ctx->uses_verlet_list = 1;
      SPSS_CUDA_TRY(launch_chained(!build, f64_verlet_pairs_kernel, blocks_for(k.n, kPairThreads), kPairThreads, 0,
                                   ctx->stream, k, in, (const int *) (f->cells_nc ? f->binner.members.ptr : nullptr),
                                   (const int *) f->vl_off.ptr, (const int *) f->vl_ent.ptr, d_knext, f->caf.ptr));
      ++ctx->launches;
      return check_launch("f64_verlet_pairs_kernel");
    }
    case SPSS_VARIANT_GLOBAL_FIELD:
    {
      const int nparts = std::min(1024, blocks_for(k.n, 256));
      f64_field_partials_kernel<<<nparts, 256, 0, ctx->stream>>>(k, f->rk.ptr, f->partials.ptr);
      ++ctx->launches;
      SPSS_TRY(check_launch("f64_field_partials_kernel"));
      f64_field_apply_kernel<<<blocks_for(k.n, 256), 256, 0, ctx->stream>>>(k, f->rk.ptr, f->partials.ptr, nparts,
                                                                            f->nat_freq.ptr, d_knext, f->caf.ptr);
      ++ctx->launches;
      return check_launch("f64_field_apply_kernel");
    }
  }
  return SPSS_ERR_INVALID_ARGUMENT;
}

int f64_evaluate(spss_ctx *ctx, int variant, const double *d_state, const double *d_kprev, double *d_knext,
                 double k_coef, double dt)
{
  return evaluate(ctx, variant, d_state, d_kprev, d_knext, k_coef, dt, nullptr);
}

int f64_max_displacement(spss_ctx *ctx, const double *d_td, double *max2_out)
{
  F64Path *f = ctx->f64;
  SPSS_CUDA_TRY(cudaMemsetAsync(f->max2.ptr, 0, sizeof(unsigned long long), ctx->stream));
  const int nb = std::min(1024, blocks_for(ctx->p.n, 256));
  f64_max2_kernel<<<nb, 256, 0, ctx->stream>>>(d_td, ctx->p.n, ctx->s, f->max2.ptr);
  ++ctx->launches;
  SPSS_TRY(check_launch("f64_max2_kernel"));
  SPSS_CUDA_TRY(cudaMemcpyAsync(f->h_max2, f->max2.ptr, sizeof(unsigned long long), cudaMemcpyDeviceToHost,
                                ctx->stream));
  SPSS_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
  unsigned long long bits = *f->h_max2;
  std::memcpy(max2_out, &bits, sizeof(double));
  return SPSS_OK;
}

static NoiseKey noise_key(const spss_ctx *ctx, unsigned long long step)
{
  NoiseKey nk;
  nk.seed = ctx->p.seed;
  nk.replica = ctx->p.replica;
  nk.step = step;
  return nk;
}

// The four evaluations of an all-pairs RK4 step whose first stage stands in the
// first stage buffers; the last one leaves the next step's first stage there.
static int allpairs_rk4_stages(spss_ctx *ctx, const K64 &k, double dt, bool chained)
{
  F64Path *f = ctx->f64;
  double *rk[2] = {f->rk.ptr, f->rk2.ptr};
  float2 *pf[2] = {f->posf.ptr, f->posf2.ptr};
  double2 *cs[2] = {f->csphi.ptr, f->csphi2.ptr};
  longlong2 *ts[2] = {f->turns.ptr, f->turns2.ptr};
  const double coef[4] = {0.5, 0.5, 1.0, 0.0};
  for (int e = 0; e < 4; ++e)
  {
    const int a = e & 1, b = a ^ 1;
    const NextStage next{f->state.ptr, coef[e],     dt,          rk[b],       pf[b],
                         cs[b],        ts[b],       f->k[0].ptr, f->k[1].ptr, f->k[2].ptr, f->td.ptr};
    const int blocks = blocks_for(k.n, kAllParticles), threads = 32 * kAllWarps;
    const double *in = rk[a];
    const float2 *pin = pf[a];
    const double2 *cin = cs[a];
    const longlong2 *tin = ts[a];
    if (e < 3)
      SPSS_CUDA_TRY(launch_chained(chained && e > 0, f64_allpairs_kernel<AFTER_STAGE>, blocks, threads, 0, ctx->stream,
                                   k, in, pin, cin, tin, f->k[e].ptr, f->caf.ptr, next));
    else
      SPSS_CUDA_TRY(launch_chained(chained, f64_allpairs_kernel<AFTER_COMBINE>, blocks, threads, 0, ctx->stream, k, in,
                                   pin, cin, tin, f->k[e].ptr, f->caf.ptr, next));
    ++ctx->launches;
    SPSS_TRY(check_launch("f64_allpairs_kernel"));
  }
  return SPSS_OK;
}

int f64_step(spss_ctx *ctx, int stepper, double t, double dt)
{
  (void) t;
  F64Path *f = ctx->f64;
  const int n = ctx->p.n, s = ctx->s;
  const long len = (long) n * s;
  const int variant = ctx->p.variant;
  const int tb = 256;
  if (stepper == SPSS_STEPPER_RK4 && variant_for(ctx, variant) == SPSS_VARIANT_ALL_PAIRS && !ctx->higher_order)
  {
    // the first stage, then four all-pairs evaluations, each also writing the
    // next stage (x + 0.5 dt k1, x + 0.5 dt k2, x + dt k3, and the step's
    // result, which is the next step's first stage) into the other stage
    // buffers
    const K64 k = make_k64(ctx);
    SPSS_TRY(f->rk2.reserve(len));
    SPSS_TRY(f->posf2.reserve(n));
    SPSS_TRY(f->csphi2.reserve(n));
    SPSS_TRY(f->turns2.reserve(n));
    f64_stage_posf_kernel<<<blocks_for(n, tb), tb, 0, ctx->stream>>>(k, f->state.ptr, f->k[0].ptr, f->rk.ptr,
                                                                     f->posf.ptr, f->csphi.ptr, f->turns.ptr, 0.0,
                                                                     dt);
    ++ctx->launches;
    SPSS_TRY(check_launch("f64_stage_posf_kernel"));
    SPSS_TRY(allpairs_rk4_stages(ctx, k, dt, false));
  } else if (stepper == SPSS_STEPPER_RK4)
  {
    double *x = f->state.ptr;
    SPSS_TRY(f64_evaluate(ctx, variant, x, f->k[0].ptr, f->k[0].ptr, 0.0, dt));
    SPSS_TRY(f64_evaluate(ctx, variant, x, f->k[0].ptr, f->k[1].ptr, 0.5, dt));
    SPSS_TRY(f64_evaluate(ctx, variant, x, f->k[1].ptr, f->k[2].ptr, 0.5, dt));
    SPSS_TRY(f64_evaluate(ctx, variant, x, f->k[2].ptr, f->k[3].ptr, 1.0, dt));
    f64_rk4_combine_kernel<<<blocks_for(len, tb), tb, 0, ctx->stream>>>(x, f->k[0].ptr, f->k[1].ptr, f->k[2].ptr,
                                                                        f->k[3].ptr, f->td.ptr, len, dt);
    ++ctx->launches;
    SPSS_TRY(check_launch("f64_rk4_combine_kernel"));
  } else
  {
    const NoiseKey nk = noise_key(ctx, ctx->step_counter);
    if (variant_for(ctx, variant) == SPSS_VARIANT_ALL_PAIRS)
      SPSS_CUDA_TRY(cudaMemsetAsync(f->det.ptr, 0, sizeof(double) * len, ctx->stream));
    if (stepper == SPSS_STEPPER_STOCHASTIC_RUNGE_KUTTA) ctx->higher_order = 1;
    if (variant_for(ctx, variant) == SPSS_VARIANT_ALL_PAIRS)
      SPSS_TRY(evaluate(ctx, variant, f->state.ptr, f->det.ptr, f->det.ptr, 0.0, dt, nullptr));
    else
      SPSS_TRY(evaluate(ctx, variant, f->state.ptr, nullptr, f->det.ptr, 0.0, dt, f->det.ptr));
    const double sqrt_dt = std::sqrt(dt), dt15 = std::pow(dt, 1.5), inv_sqrt3 = 1.0 / std::sqrt(3.0);
    const double b_r = std::sqrt(2.0 * ctx->p.D_r), b_phi = std::sqrt(2.0 * ctx->p.D_phi);
    const double *det = f->det.ptr, *caf = f->caf.ptr;
    const double2 *table = f->table.ptr;
    const int blocks = blocks_for(n, tb);
    MaxOut m{nullptr, nullptr, nullptr};
    if (ctx->uses_verlet_list) m = MaxOut{f->max2.ptr + 1, f->h_max2, reinterpret_cast<unsigned *>(f->max2.ptr + 2)};
    if (stepper == SPSS_STEPPER_STOCHASTIC_EULER)
    {
      if (ctx->p.model == 2)
        SPSS_CUDA_TRY(launch_chained(true, f64_se2_kernel, blocks, tb, 0, ctx->stream, f->state.ptr, det, f->td.ptr, n,
                                     dt, sqrt_dt, b_r, b_phi, nk, table, m));
      else
        SPSS_CUDA_TRY(launch_chained(true, f64_se1_kernel, blocks, tb, 0, ctx->stream, f->state.ptr, det, f->td.ptr, n,
                                     dt, sqrt_dt, b_phi, nk, table, m));
    } else if (stepper == SPSS_STEPPER_STOCHASTIC_RUNGE_KUTTA)
    {
      if (ctx->p.model == 1)
        SPSS_CUDA_TRY(launch_chained(true, f64_srk1_kernel, blocks, tb, 0, ctx->stream, f->state.ptr, det, caf,
                                     f->td.ptr, n, dt, sqrt_dt, dt15, inv_sqrt3, b_phi, ctx->p.xi, nk, table, m));
      else
        SPSS_CUDA_TRY(launch_chained(true, f64_srk2_kernel, blocks, tb, 0, ctx->stream, f->state.ptr, det, caf,
                                     f->td.ptr, n, dt, sqrt_dt, dt15, inv_sqrt3, b_r, b_phi, ctx->p.xi_r,
                                     ctx->p.xi_phi, ctx->p.v0, nk, table, m));
    } else
    {
      return SPSS_ERR_INVALID_ARGUMENT;
    }
    ++ctx->launches;
    SPSS_TRY(check_launch("f64 stepper kernel"));
    ++ctx->step_counter;
  }
  if (ctx->uses_verlet_list)
  {
    double max2 = 0.0;
    if (stepper == SPSS_STEPPER_RK4)
    {
      SPSS_TRY(f64_max_displacement(ctx, f->td.ptr, &max2));
    } else
    {
      SPSS_CUDA_TRY(cudaStreamSynchronize(ctx->stream));
      std::memcpy(&max2, f->h_max2, sizeof(double));
    }
    SPSS_TRY(host_calculate_max_displacement(ctx, max2));
  }
  return SPSS_OK;
}

// nsteps RK4 steps: one step runs as it is (sizing every buffer), the rest
// replay that step captured as a CUDA graph — RK4 draws no noise and, without
// a Verlet list, needs no host decision between steps.  The state is
// identical to nsteps single steps.  Other steppers and Verlet contexts step
// one by one.
int f64_steps(spss_ctx *ctx, int stepper, double t0, double dt, int nsteps)
{
  F64Path *f = ctx->f64;
  double t = t0;
  const bool graphable = stepper == SPSS_STEPPER_RK4 && !ctx->uses_verlet_list &&
                         variant_for(ctx, ctx->p.variant) != SPSS_VARIANT_VERLET &&
                         variant_for(ctx, ctx->p.variant) != SPSS_VARIANT_LINKED_LIST_VERLET;
  if (!graphable || nsteps < 3)
  {
    for (int k = 0; k < nsteps; ++k)
    {
      t += dt;
      SPSS_TRY(f64_step(ctx, stepper, t, dt));
    }
    return SPSS_OK;
  }
  t += dt;
  SPSS_TRY(f64_step(ctx, stepper, t, dt));
  const bool stages_only = variant_for(ctx, ctx->p.variant) == SPSS_VARIANT_ALL_PAIRS && !ctx->higher_order;
  if (!f->rk4_exec || f->rk4_dt != dt || f->rk4_higher_order != ctx->higher_order)
  {
    if (f->rk4_exec) cudaGraphExecDestroy(f->rk4_exec);
    if (f->rk4_graph) cudaGraphDestroy(f->rk4_graph);
    f->rk4_exec = nullptr;
    f->rk4_graph = nullptr;
    cudaStream_t work = ctx->stream;
    ctx->stream = ctx->own_stream;  // capture needs a non-legacy stream
    const unsigned long long launches0 = ctx->launches;
    SPSS_CUDA_TRY(cudaStreamSynchronize(work));
    int rc = SPSS_OK;
    if (cudaStreamBeginCapture(ctx->stream, cudaStreamCaptureModeThreadLocal) != cudaSuccess) rc = SPSS_ERR_CUDA;
    // an all-pairs step leaves the next step's first stage behind: without the stage kernel
    if (rc == SPSS_OK)
      rc = stages_only ? allpairs_rk4_stages(ctx, make_k64(ctx), dt, true) : f64_step(ctx, stepper, t + dt, dt);
    cudaGraph_t g = nullptr;
    const cudaError_t e = cudaStreamEndCapture(ctx->stream, &g);
    ctx->stream = work;
    f->rk4_launches = ctx->launches - launches0;
    ctx->launches = launches0;
    if (rc == SPSS_OK && e != cudaSuccess) rc = SPSS_ERR_CUDA;
    if (rc == SPSS_OK && cudaGraphInstantiate(&f->rk4_exec, g, 0) != cudaSuccess) rc = SPSS_ERR_CUDA;
    if (rc != SPSS_OK)
    {
      cudaGetLastError();
      if (g) cudaGraphDestroy(g);
      f->rk4_exec = nullptr;
      return rc;
    }
    f->rk4_graph = g;
    f->rk4_dt = dt;
    f->rk4_higher_order = ctx->higher_order;
  }
  for (int k = 1; k < nsteps; ++k) SPSS_CUDA_TRY(cudaGraphLaunch(f->rk4_exec, ctx->stream));
  ctx->launches += f->rk4_launches * (unsigned long long) (nsteps - 1);
  return SPSS_OK;
}

int f64_noise(spss_ctx *ctx, int stepper, unsigned long long step, double *d_out)
{
  const int per = normals_per_particle(ctx->p.model, stepper);
  if (per == 0) return SPSS_OK;
  f64_noise_kernel<<<blocks_for(ctx->p.n, 256), 256, 0, ctx->stream>>>(d_out, ctx->p.n, per, noise_key(ctx, step),
                                                                     ctx->f64->table.ptr);
  ++ctx->launches;
  return check_launch("f64_noise_kernel");
}

int f64_complementary_force(spss_ctx *ctx, double *d_out)
{
  SPSS_CUDA_TRY(cudaMemcpyAsync(d_out, ctx->f64->caf.ptr, sizeof(double) * ctx->p.n, cudaMemcpyDeviceToDevice,
                                ctx->stream));
  return SPSS_OK;
}

int f64_set_natural_frequencies(spss_ctx *ctx, const double *d_freqs)
{
  SPSS_CUDA_TRY(cudaMemcpyAsync(ctx->f64->nat_freq.ptr, d_freqs, sizeof(double) * ctx->p.n,
                                cudaMemcpyDeviceToDevice, ctx->stream));
  return SPSS_OK;
}

int f64_lists(spss_ctx *ctx, int **pll, int **cell_off, int **cell_mem, int *ncell, int **vl_off, int **vl_ent,
              long *vl_total)
{
  F64Path *f = ctx->f64;
  *pll = f->cells_nc ? f->cell_of.ptr : nullptr;
  *cell_off = f->cells_nc ? f->binner.offsets.ptr : nullptr;
  *cell_mem = f->cells_nc ? f->binner.members.ptr : nullptr;
  *ncell = f->cells_nc * f->cells_nc;
  *vl_off = f->vl_built ? f->vl_off.ptr : nullptr;
  *vl_ent = f->vl_built ? f->vl_ent.ptr : nullptr;
  *vl_total = f->vl_built ? f->vl_total : 0;
  return SPSS_OK;
}

int f64_apply_pbc(spss_ctx *ctx)
{
  f64_pbc_kernel<<<blocks_for(ctx->p.n, 256), 256, 0, ctx->stream>>>(ctx->f64->state.ptr, ctx->p.n, ctx->s);
  ++ctx->launches;
  return check_launch("f64_pbc_kernel");
}

}  // namespace spss
