// Shared device utilities: prefix sum, stable cell binning, error recording.
#include <sys/mman.h>
#include <unistd.h>
#include <climits>
#include <cmath>
#include <cstdio>
#include <cstring>

#include "spss_internal.cuh"

namespace spss
{

void prefault(void *p, size_t bytes)
{
#ifdef __linux__
  const uintptr_t page = (uintptr_t) sysconf(_SC_PAGESIZE);
  const uintptr_t first = (uintptr_t) p & ~(page - 1), end = ((uintptr_t) p + bytes + page - 1) & ~(page - 1);
  constexpr int kPopulateWrite = 23;  // MADV_POPULATE_WRITE, Linux 5.14
  if (bytes >= 2 * page) madvise((void *) first, end - first, kPopulateWrite);
#endif
}

static thread_local char g_last_error[512];

void record_cuda_error(cudaError_t e, const char *what, const char *file, int line)
{
  std::snprintf(g_last_error, sizeof(g_last_error), "%s: %s (%s:%d)", cudaGetErrorString(e), what, file, line);
}

int check_launch(const char *what)
{
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess)
  {
    record_cuda_error(e, what, __FILE__, __LINE__);
    return SPSS_ERR_CUDA;
  }
  return SPSS_OK;
}

const char *last_error_text()
{
  return g_last_error;
}

// ------------------------------------------------------------------ tables of the FP64 functions

__global__ void f64_tables_kernel(double2 *__restrict__ table)
{
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kTableEntries) return;
  if (i < kTrigTable)
  {
    double s, c;
    sincospi((double) i / 128.0, &s, &c);
    table[i] = make_double2(c, s);
    return;
  }
  const int j = i - kTrigTable + kLogFirst;
  const double inv = 128.0 / (double) j;
  // -log(inv) of the rounded inv, from the exact j / 128: log(j / 128) - log1p(delta), inv = (1 + delta) 128 / j
  const double delta = fma(inv, (double) j / 128.0, -1.0);
  table[i] = make_double2(inv, log((double) j / 128.0) - delta);
}

// cos and sin of 2 pi k / 256 in units of 2^-59, from the first eighth of a turn.
struct FixedTable
{
  longlong2 at[kTrigTable];

  FixedTable()
  {
    constexpr int quarter = kTrigTable / 4, eighth = kTrigTable / 8;
    const long double angle = 3.14159265358979323846264338327950288L / 128.0L, unit = 576460752303423488.0L;
    long long c[quarter + 1];  // cosines of the first quarter
    for (int k = 0; k <= eighth; ++k)
    {
      c[k] = std::llroundl(std::cos(angle * k) * unit);
      c[quarter - k] = std::llroundl(std::sin(angle * k) * unit);
    }
    auto cosine = [&](int k) {
      k &= kTrigTable - 1;
      if (k > 2 * quarter) k = kTrigTable - k;
      return k <= quarter ? c[k] : -c[2 * quarter - k];
    };
    for (int k = 0; k < kTrigTable; ++k) at[k] = make_longlong2(cosine(k), cosine(k - quarter));
  }
};

int make_f64_tables(DeviceArray<double2> &table, cudaStream_t stream)
{
  static const FixedTable fixed;  // constants, the same for every context
  SPSS_TRY(table.reserve(kTableEntries + kTrigTable));
  f64_tables_kernel<<<(kTableEntries + 127) / 128, 128, 0, stream>>>(table.ptr);
  SPSS_TRY(check_launch("f64_tables_kernel"));
  SPSS_CUDA_TRY(cudaMemcpyAsync(table.ptr + kTableEntries, fixed.at, sizeof(fixed.at), cudaMemcpyHostToDevice, stream));
  return SPSS_OK;
}

// ------------------------------------------------------------------ scan

constexpr int kScanThreads = 256;
constexpr int kScanItems = 16;
constexpr int kScanTile = kScanThreads * kScanItems;
// Up to this many tiles every tile adds the sums before its own (its share of
// at most 32 KiB of L2 reads); beyond it the sums are scanned first.
constexpr int kScanDirect = 8192;

__device__ __forceinline__ int block_sum(int v, int *warp_tot)
{
#pragma unroll
  for (int off = 16; off > 0; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
  if ((threadIdx.x & 31) == 0) warp_tot[threadIdx.x >> 5] = v;
  __syncthreads();
  int t = 0;
#pragma unroll
  for (int w = 0; w < kScanThreads / 32; ++w) t += warp_tot[w];
  __syncthreads();
  return t;
}

__device__ __forceinline__ void load_items(const int *__restrict__ in, int base, int n, int v[kScanItems])
{
  if (base + kScanItems <= n)
  {
#pragma unroll
    for (int q = 0; q < kScanItems; q += 4) *reinterpret_cast<int4 *>(v + q) = *reinterpret_cast<const int4 *>(in + base + q);
    return;
  }
#pragma unroll
  for (int q = 0; q < kScanItems; ++q) v[q] = base + q < n ? in[base + q] : 0;
}

__global__ void __launch_bounds__(kScanThreads) scan_sums_kernel(const int *__restrict__ in, int *__restrict__ sums, int n)
{
  __shared__ int warp_tot[kScanThreads / 32];
  int v[kScanItems], local = 0;
  load_items(in, blockIdx.x * kScanTile + threadIdx.x * kScanItems, n, v);
#pragma unroll
  for (int q = 0; q < kScanItems; ++q) local += v[q];
  const int t = block_sum(local, warp_tot);
  if (threadIdx.x == 0) sums[blockIdx.x] = t;
}

// A cell-list step begins: its re-sort exchanges the vel/pid buffers, its
// update takes the noise of the step counted here (step - 1), and the next
// step's cell ids and counts come from it.  What a control kernel after the
// step would do, without the launch; nothing else in the launch reads these.
__device__ __forceinline__ void begin_cell_step(FastControl *c)
{
  c->step += 1;
  c->order_parity ^= 1;
  c->rebuilds += 1;
  c->cells_fresh = 1;
  c->rebuild = 1;
  c->triggered = 1;
}

// Exclusive scan of one tile per block, after the sum of the tiles before it:
// `sums` of the tiles (`scanned`: their exclusive prefix), null for one tile.
__global__ void __launch_bounds__(kScanThreads) scan_tile_kernel(int *__restrict__ in, int *__restrict__ out,
                                                                 const int *__restrict__ sums, int n, int scanned,
                                                                 int zero, FastControl *ctrl)
{
  __shared__ int warp_tot[kScanThreads / 32];
  pdl_enter();
  if (ctrl && blockIdx.x == 0 && threadIdx.x == 0) begin_cell_step(ctrl);
  const int base = blockIdx.x * kScanTile + threadIdx.x * kScanItems;
  int v[kScanItems];
  load_items(in, base, n, v);
  int before = 0;
  if (sums)
  {
    if (scanned)
    {
      before = sums[blockIdx.x];
    } else
    {
      for (int k = threadIdx.x; k < (int) blockIdx.x; k += kScanThreads) before += sums[k];
      before = block_sum(before, warp_tot);
    }
  }
  int local = 0;
#pragma unroll
  for (int q = 0; q < kScanItems; ++q) local += v[q];
  // inclusive scan of the per-thread totals across the block
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int x = local;
#pragma unroll
  for (int off = 1; off < 32; off <<= 1)
  {
    const int y = __shfl_up_sync(0xffffffffu, x, off);
    if (lane >= off) x += y;
  }
  if (lane == 31) warp_tot[warp] = x;
  __syncthreads();
  int excl = before + x - local;
#pragma unroll
  for (int w = 0; w < kScanThreads / 32; ++w) excl += w < warp ? warp_tot[w] : 0;
  int o[kScanItems];
#pragma unroll
  for (int q = 0; q < kScanItems; ++q)
  {
    o[q] = excl;
    excl += v[q];
  }
  if (base + kScanItems <= n)
  {
#pragma unroll
    for (int q = 0; q < kScanItems; q += 4)
    {
      *reinterpret_cast<int4 *>(out + base + q) = *reinterpret_cast<const int4 *>(o + q);
      if (zero) *reinterpret_cast<int4 *>(in + base + q) = make_int4(0, 0, 0, 0);
    }
  } else
  {
#pragma unroll
    for (int q = 0; q < kScanItems; ++q)
      if (base + q < n)
      {
        out[base + q] = o[q];
        if (zero) in[base + q] = 0;
      }
  }
  if (blockIdx.x == gridDim.x - 1 && threadIdx.x == kScanThreads - 1) out[n] = excl;
}

int Scanner::run(int *in, int *out, int n, cudaStream_t stream, unsigned long long &launches, bool chained, bool zero,
                 FastControl *ctrl)
{
  return run_level(in, out, n, 0, stream, launches, chained, zero, ctrl);
}

int Scanner::prepare(int n)
{
  for (size_t level = 0; n > kScanTile; ++level)
  {
    n = (n + kScanTile - 1) / kScanTile;
    if (levels.size() < 2 * (level + 1)) levels.resize(2 * (level + 1));
    SPSS_TRY(levels[2 * level].reserve(n));
    SPSS_TRY(levels[2 * level + 1].reserve(n + 1));
  }
  return SPSS_OK;
}

int Scanner::run_level(int *in, int *out, int n, size_t level, cudaStream_t stream, unsigned long long &launches,
                       bool chained, bool zero, FastControl *ctrl)
{
  if (n <= 0)
  {
    SPSS_CUDA_TRY(cudaMemsetAsync(out, 0, sizeof(int), stream));
    return SPSS_OK;
  }
  const int nblocks = (n + kScanTile - 1) / kScanTile;
  const int *sums = nullptr;
  int scanned = 0;
  if (nblocks > 1)
  {
    if (levels.size() < 2 * (level + 1)) levels.resize(2 * (level + 1));
    SPSS_TRY(levels[2 * level].reserve(nblocks));
    SPSS_TRY(levels[2 * level + 1].reserve(nblocks + 1));
    int *s = levels[2 * level].ptr, *off = levels[2 * level + 1].ptr;  // device pointers stay valid if `levels` grows
    scan_sums_kernel<<<nblocks, kScanThreads, 0, stream>>>(in, s, n);
    ++launches;
    SPSS_TRY(check_launch("scan_sums_kernel"));
    sums = s;
    if (nblocks > kScanDirect)
    {
      SPSS_TRY(run_level(s, off, nblocks, level + 1, stream, launches, chained, false, nullptr));
      sums = off;
      scanned = 1;
    }
  }
  // the first launch of a chain is an ordinary one
  SPSS_CUDA_TRY(launch_chained(chained && nblocks > 1, scan_tile_kernel, nblocks, kScanThreads, 0, stream, in, out, sums, n, scanned,
                               (int) zero, ctrl));
  ++launches;
  return check_launch("scan_tile_kernel");
}

// ------------------------------------------------------------------ binning

__global__ void bin_count_kernel(const int *__restrict__ cell_of, int n, int *__restrict__ count,
                                 int *__restrict__ slot)
{
  pdl_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) slot[i] = atomicAdd(&count[cell_of[i]], 1);
}

__global__ void bin_scatter_kernel(const int *__restrict__ cell_of, const int *__restrict__ slot,
                                   const int *__restrict__ offsets, int n, int *__restrict__ members)
{
  pdl_enter();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) members[offsets[cell_of[i]] + slot[i]] = i;
}

// Members of one cell into ascending order (cells hold a handful of particles):
// up to kSortRegs members are sorted in registers by an odd-even transposition
// network (all loads issued together, one store each), larger cells by an
// insertion sort in place.
constexpr int kSortRegs = 8;

__device__ __forceinline__ void write_row(const BinRows &rows, int at, int member)
{
  if (!rows.pos_out) return;
  rows.pos_out[at] = __ldg(rows.pos + member);
  rows.turns_out[at] = __ldg(rows.turns + member);
}

__global__ void bin_sort_kernel(const int *__restrict__ offsets, int ncell, int *__restrict__ members, BinRows rows)
{
  pdl_enter();
  const int c = blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= ncell) return;
  const int b = offsets[c], e = offsets[c + 1];
  const int m = e - b;
  if (m <= 1)
  {
    if (m == 1) write_row(rows, b, members[b]);
    return;
  }
  if (m <= kSortRegs)
  {
    int v[kSortRegs];
#pragma unroll
    for (int k = 0; k < kSortRegs; ++k) v[k] = k < m ? members[b + k] : INT_MAX;
#pragma unroll
    for (int r = 0; r < kSortRegs; ++r)
#pragma unroll
      for (int k = r & 1; k + 1 < kSortRegs; k += 2)
      {
        const int lo = min(v[k], v[k + 1]), hi = max(v[k], v[k + 1]);
        v[k] = lo;
        v[k + 1] = hi;
      }
#pragma unroll
    for (int k = 0; k < kSortRegs; ++k)
      if (k < m)
      {
        members[b + k] = v[k];
        write_row(rows, b + k, v[k]);
      }
    return;
  }
  for (int q = b + 1; q < e; ++q)
  {
    const int v = members[q];
    int r = q - 1;
    while (r >= b && members[r] > v)
    {
      members[r + 1] = members[r];
      --r;
    }
    members[r + 1] = v;
  }
  for (int q = b; q < e; ++q) write_row(rows, q, members[q]);
}

int Binner::prepare(int n, int ncell_in, cudaStream_t stream)
{
  ncell = ncell_in;
  const int *had = count.ptr;
  const size_t held = count.count;
  SPSS_TRY(count.reserve(ncell));
  SPSS_TRY(offsets.reserve(ncell + 1));
  SPSS_TRY(slot.reserve(n));
  SPSS_TRY(members.reserve(n));
  SPSS_TRY(scanner.prepare(ncell));  // nothing is allocated while a step is captured
  if (count.ptr != had || count.count != held) SPSS_CUDA_TRY(cudaMemsetAsync(count.ptr, 0, sizeof(int) * count.count, stream));
  return SPSS_OK;
}

int Binner::place(const int *cell_of, int n, cudaStream_t stream, unsigned long long &launches, bool chained,
                  FastControl *ctrl)
{
  const int tb = 256;
  SPSS_TRY(scanner.run(count.ptr, offsets.ptr, ncell, stream, launches, chained, true, ctrl));
  SPSS_CUDA_TRY(launch_chained(chained, bin_scatter_kernel, (n + tb - 1) / tb, tb, 0, stream, cell_of,
                               (const int *) slot.ptr, (const int *) offsets.ptr, n, members.ptr));
  ++launches;
  return check_launch("bin_scatter_kernel");
}

// From the counts to the sorted members.
int Binner::finish(const int *cell_of, int n, cudaStream_t stream, unsigned long long &launches, bool chained,
                   const BinRows &rows)
{
  const int tb = 256;
  SPSS_TRY(place(cell_of, n, stream, launches, chained));
  SPSS_CUDA_TRY(launch_chained(chained, bin_sort_kernel, (ncell + tb - 1) / tb, tb, 0, stream,
                               (const int *) offsets.ptr, ncell, members.ptr, rows));
  ++launches;
  return check_launch("bin_sort_kernel");
}

int Binner::run(const int *cell_of, int n, int ncell_in, cudaStream_t stream, unsigned long long &launches)
{
  SPSS_TRY(prepare(n, ncell_in, stream));
  const int tb = 256;
  bin_count_kernel<<<(n + tb - 1) / tb, tb, 0, stream>>>(cell_of, n, count.ptr, slot.ptr);
  ++launches;
  SPSS_TRY(check_launch("bin_count_kernel"));
  return finish(cell_of, n, stream, launches, false, BinRows{});
}

}  // namespace spss
