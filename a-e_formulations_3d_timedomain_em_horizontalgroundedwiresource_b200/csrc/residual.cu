// Residual norms of a block of solutions of a sparse system, on the device:
//   norms[2j] = ||b_j - A x_j||_2,  norms[2j + 1] = ||b_j||_2   for j < ncols.
//
// Two deterministic passes.  Pass 1 (kResBlocks CTAs of 256 threads): tiles of 256 CSR
// rows, one row per thread.  The tile's entries are staged in shared memory (read from
// device memory once for all columns, in order), then every thread forms its row's
// residual for KC columns at a time; neighbouring rows of a mesh's matrix have
// neighbouring columns, so a warp's reads of x nearly coalesce and stay in L1.  Each CTA
// adds the squares up per column and writes its partial sums to scratch[cta][j][2].
// Pass 2 (a warp per sum) adds the kResBlocks partials.  The row -> thread assignment and
// every summation order are fixed, so repeated calls on the same data give bit-identical
// norms.  (A warp per row, all lanes gathering and reducing one column after another,
// was 4,125 us for 270,400 rows of 27 entries and 32 columns, 225 MB; this is 230 us, bound by
// the reads of x through L1 and L2.)
//
// A tile of more entries than fit goes in 2 to 32 parts, in each of which as many threads
// share a row; a part that still does not fit, and a row that would keep a thread longer
// than the rest of its tile, goes a warp per row.  Where there are fewer tiles than CTAs the
// parts and then the columns are spread over them.  (us for 1 / 32 columns, cold L2: a warp
// per row, then a thread per row whatever its length, then this: 33 entries a row, 65 x 65 x
// 64 rows 310 / 4,904, 128 / 534, 71 / 339; 300 entries, 20,000 rows 83 / 570, 251 / 1,099,
// 58 / 271; 500 dense rows 48 / 175, 343 / 1,367, 22 / 38; 50,000 short rows and a dense one
// 499 / 6,764, 7,762 / 71,474, 200 / 3,256.  Staging 34 entries a row instead leaves the
// reads of x less L1: 255 where 28 have 230 us in the first case.)
#include <cuda.h>
#include <cuda_runtime.h>

#include <map>
#include <mutex>

#include "../../include/tdem.h"
#include "residual.h"

namespace tdem {
namespace {

constexpr int kThreads = 256;         // rows of a tile
constexpr int kWarps = kThreads / 32;
constexpr int kPerThread = 28;        // entries of a row, on average, up to which one thread takes it
constexpr int kLongRow = 128;         // most of a row's entries that one thread takes
constexpr int kStaged = kPerThread * kThreads;  // entries that fit the staging buffers
constexpr size_t kStageBytes = kStaged * (sizeof(double) + sizeof(int));

// Sums of v[0..N) over the warp, N a power of two up to 32: lane l returns the total of
// v[l mod N].  Each round halves the values a lane holds, handing its partner the other
// half; the order of the additions is fixed by the lanes alone.
template <int N>
__device__ __forceinline__ double warp_totals(double (&v)[N], int lane) {
  int bit = N / 2;
#pragma unroll
  for (int h = N / 2; h >= 1; h /= 2, bit /= 2) {
    const bool up = (lane & bit) != 0;
#pragma unroll
    for (int e = 0; e < h; ++e) {
      const double mine = up ? v[h + e] : v[e], other = up ? v[e] : v[h + e];
      v[e] = mine + __shfl_xor_sync(0xffffffffu, other, bit);
    }
  }
  double t = v[0];
#pragma unroll
  for (int o = N; o < 32; o *= 2) t += __shfl_xor_sync(0xffffffffu, t, o);
  return t;
}

// The sums of a warp: squares of the residuals and of the right-hand sides per column.
using WarpSums = double (*)[2];

// Row i by a warp, KC columns (from c_first in steps of c_step) at a time, B of a lane's
// entries on their way at once.
template <int KC>
__device__ __noinline__ void warp_row(int64_t i, int lane, const int64_t* __restrict__ rowptr,
                                      const int* __restrict__ col, const double* __restrict__ val,
                                      const double* __restrict__ x, const double* __restrict__ b, int64_t ld, int ncols,
                                      int c_first, int c_step, WarpSums red) {
  constexpr int B = KC >= 8 ? 2 : (KC >= 4 ? 4 : 8);
  const int64_t p0 = rowptr[i], p1 = rowptr[i + 1];
  __syncwarp();  // other lanes may have added to the same sums
  for (int c0 = c_first; c0 < ncols; c0 += c_step) {
    const bool mine = lane < KC && c0 + lane < ncols;
    const double bi = mine ? __ldg(b + i + (int64_t)(c0 + lane) * ld) : 0.0;
    const double* xc = x + (int64_t)c0 * ld;
    double acc[KC];
#pragma unroll
    for (int e = 0; e < KC; ++e) acc[e] = 0.0;
    auto entries = [&](int64_t q, bool whole) {
      double v[B], xv[B][KC];
      int64_t j[B];
#pragma unroll
      for (int u = 0; u < B; ++u) {
        const bool in = whole || q + 32 * u < p1;
        v[u] = in ? __ldg(val + q + 32 * u) : 0.0;
        j[u] = in ? __ldg(col + q + 32 * u) : -1;
      }
#pragma unroll
      for (int u = 0; u < B; ++u)
#pragma unroll
        for (int e = 0; e < KC; ++e)
          xv[u][e] = (whole || j[u] >= 0) && c0 + e < ncols ? __ldg(xc + j[u] + (int64_t)e * ld) : 0.0;
#pragma unroll
      for (int u = 0; u < B; ++u)
#pragma unroll
        for (int e = 0; e < KC; ++e) acc[e] = fma(v[u], xv[u][e], acc[e]);
    };
    int64_t q = p0 + lane;
    for (; q + 32 * (B - 1) < p1; q += 32 * B) entries(q, true);
    if (q < p1) entries(q, false);
    const double r = bi - warp_totals<KC>(acc, lane);
    if (mine) {
      red[c0 + lane][0] += r * r;
      red[c0 + lane][1] += bi * bi;
    }
  }
  __syncwarp();
}

// The rows of a staged tile, entries [p0, p1) of the staging buffers the calling thread's;
// SPLIT: g threads (a power of two up to 32) share a row, each with p0 at its first entry.
template <int KC, bool SPLIT>
__device__ __forceinline__ void staged_rows(const double* vs, const int* cs, int p0, int p1, int g, bool own,
                                            int64_t row, const double* __restrict__ x, const double* __restrict__ b,
                                            int64_t ld, int ncols, int c_first, int c_step, int lane, WarpSums red) {
  const bool first = own && (!SPLIT || (lane & (g - 1)) == 0);
  for (int c0 = c_first; c0 < ncols; c0 += c_step) {
    double acc[KC], bi[KC];
#pragma unroll
    for (int e = 0; e < KC; ++e) {
      acc[e] = 0.0;
      bi[e] = first && c0 + e < ncols ? __ldg(b + row + (int64_t)(c0 + e) * ld) : 0.0;
    }
    const double* xc = x + (int64_t)c0 * ld;
#pragma unroll 4
    for (int q = p0; q < p1; q += SPLIT ? g : 1) {
      const double v = vs[q];
      const int64_t j = cs[q];
#pragma unroll
      for (int e = 0; e < KC; ++e)
        if (c0 + e < ncols) acc[e] = fma(v, __ldg(xc + j + (int64_t)e * ld), acc[e]);
    }
    if (SPLIT)
      for (int o = 1; o < g; o *= 2)
#pragma unroll
        for (int e = 0; e < KC; ++e) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
    double sq[2 * KC];  // squares of the residuals, then of the right-hand sides
#pragma unroll
    for (int e = 0; e < KC; ++e) {
      const double r = first ? bi[e] - acc[e] : 0.0;
      sq[e] = r * r;
      sq[KC + e] = bi[e] * bi[e];
    }
    const double tot = warp_totals<2 * KC>(sq, lane);
    if (lane < 2 * KC && c0 + lane % KC < ncols) red[c0 + lane % KC][lane / KC] += tot;
  }
}

template <int KC>
__global__ void __launch_bounds__(kThreads)
k_residual_partial(int64_t n, const int64_t* __restrict__ rowptr, const int* __restrict__ col,
                   const double* __restrict__ val, const double* __restrict__ x, const double* __restrict__ b,
                   int64_t ld, int ncols, double* __restrict__ partial) {
  extern __shared__ __align__(16) unsigned char sm[];
  double* vs = reinterpret_cast<double*>(sm);
  int* cs = reinterpret_cast<int*>(sm + kStaged * sizeof(double));
  __shared__ double red[kWarps][kResMaxCols][2];
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  for (int q = t; q < kWarps * kResMaxCols * 2; q += kThreads) (&red[0][0][0])[q] = 0.0;
  // (with fewer tiles than CTAs a tile has `share` of them: for its parts, and from there
  // on for its columns)
  const int64_t tiles = (n + kThreads - 1) / kThreads;
  const int few = (int)min(max(tiles, (int64_t)1), (int64_t)gridDim.x);
  const int share = gridDim.x / few, member = blockIdx.x / few;
  for (int64_t tile = blockIdx.x % few; tile < tiles && member < share; tile += gridDim.x) {
    // parts of the tile, and threads per row: one, or so many that a part should fit
    const int64_t t0 = tile * kThreads, entries = rowptr[min(n, t0 + kThreads)] - rowptr[t0];
    const int rows = (int)min((int64_t)kThreads, n - t0);
    int g = 1;
    while (g < 32 && entries > (int64_t)kPerThread * rows * g) g *= 2;
    const int chunks = (ncols + KC - 1) / KC, sets = max(1, min(chunks, share / g)), set = min(member / g, sets);
    const bool many = share > g;
    const int c_first = (many ? set : 0) * KC, c_step = sets * KC;
    for (int part = !many ? member : (set < sets ? member % g : g); part < g; part += min(g, share)) {
      const int64_t r0 = t0 + part * (kThreads / g), r1 = min(n, r0 + kThreads / g), row = r0 + t / g;
      if (r0 >= n) break;
      const int64_t first = rowptr[r0], last = rowptr[r1];
      const bool live = row < n;
      const int64_t p0 = live ? rowptr[row] : 0, p1 = live ? rowptr[row + 1] : 0;
      __syncthreads();
      if (last - first > kStaged) {
        for (int64_t i = r0 + warp; i < r1; i += kWarps)
          warp_row<KC>(i, lane, rowptr, col, val, x, b, ld, ncols, c_first, c_step, red[warp]);
        continue;
      }
      for (int q = t; q < (int)(last - first); q += kThreads) {
        vs[q] = __ldg(val + first + q);
        cs[q] = __ldg(col + first + q);
      }
      __syncthreads();
      const bool longer = p1 - p0 > (int64_t)kLongRow * g, own = live && !longer;
      for (unsigned todo = __ballot_sync(0xffffffffu, longer && t % g == 0); todo; todo &= todo - 1)
        warp_row<KC>(r0 + (32 * warp + __ffs(todo) - 1) / g, lane, rowptr, col, val, x, b, ld, ncols, c_first, c_step,
                     red[warp]);
      const int s0 = own ? (int)(p0 - first) : 0, s1 = own ? (int)(p1 - first) : 0;  // (none: no entries)
      if (g == 1)
        staged_rows<KC, false>(vs, cs, s0, s1, 1, own, row, x, b, ld, ncols, c_first, c_step, lane, red[warp]);
      else
        staged_rows<KC, true>(vs, cs, s0 + t % g, s1, g, own, row, x, b, ld, ncols, c_first, c_step, lane,
                               red[warp]);
    }
  }
  __syncthreads();
  for (int q = t; q < 2 * ncols; q += kThreads) {
    const int j = q >> 1, c = q & 1;
    double s = 0.0;
    for (int w = 0; w < kWarps; ++w) s += red[w][j][c];
    partial[((int64_t)blockIdx.x * kResMaxCols + j) * 2 + c] = s;
  }
}

// One warp per sum: lane l adds the partials of CTAs l, l + 32, ..., then the lanes.
__global__ void k_residual_final(int ncols, const double* __restrict__ partial, double* __restrict__ norms) {
  const int q = (int)((blockIdx.x * blockDim.x + threadIdx.x) >> 5), lane = threadIdx.x & 31;
  if (q >= 2 * ncols) return;
  double s = 0.0;
  for (int blk = lane; blk < kResBlocks; blk += 32) s += partial[(int64_t)blk * kResMaxCols * 2 + q];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (lane == 0) norms[q] = sqrt(s);
}

template <int KC>
cudaError_t launch_partial(int64_t n, const int64_t* rowptr, const int* col, const double* val, const double* x,
                           const double* b, int64_t ld, int ncols, double* scratch, cudaStream_t s) {
  // per device and cheap; the kernel would not launch without it
  const cudaError_t e =
      cudaFuncSetAttribute(k_residual_partial<KC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kStageBytes);
  if (e != cudaSuccess) return e;
  k_residual_partial<KC><<<kResBlocks, kThreads, kStageBytes, s>>>(n, rowptr, col, val, x, b, ld, ncols, scratch);
  return cudaGetLastError();
}

}  // namespace

const char* check_residual_args(int64_t n, const int64_t* rowptr, const int* col, const double* val,
                                const double* x, const double* b, int64_t ld, int ncols, const double* norms) {
  if (n < 0) return "n must be non-negative";
  if (ncols < 1 || ncols > kResMaxCols) return "ncols must be in [1, 64]";
  if (ld < n) return "ld must be at least n";
  if (!rowptr || !norms || (n > 0 && (!col || !val || !x || !b))) return "null pointer";
  return nullptr;
}

cudaError_t launch_residual_norms(int64_t n, const int64_t* rowptr, const int* col, const double* val,
                                  const double* x, const double* b, int64_t ld, int ncols, double* norms,
                                  double* scratch, cudaStream_t s) {
  const cudaError_t e = ncols >= 8   ? launch_partial<8>(n, rowptr, col, val, x, b, ld, ncols, scratch, s)
                        : ncols >= 3 ? launch_partial<4>(n, rowptr, col, val, x, b, ld, ncols, scratch, s)
                        : ncols == 2 ? launch_partial<2>(n, rowptr, col, val, x, b, ld, ncols, scratch, s)
                                     : launch_partial<1>(n, rowptr, col, val, x, b, ld, ncols, scratch, s);
  if (e != cudaSuccess) return e;
  k_residual_final<<<(2 * ncols + 7) / 8, 256, 0, s>>>(ncols, scratch, norms);
  return cudaGetLastError();
}

}  // namespace tdem

namespace {

// Makes `device` current for the lifetime of the guard and restores the caller's.
struct DeviceGuard {
  int prev = -1;
  cudaError_t err = cudaSuccess;
  explicit DeviceGuard(int device) {
    err = cudaGetDevice(&prev);
    if (err == cudaSuccess && prev != device) err = cudaSetDevice(device);
  }
  ~DeviceGuard() {
    int cur = -1;
    if (prev >= 0 && cudaGetDevice(&cur) == cudaSuccess && cur != prev) cudaSetDevice(prev);
  }
};

// Memory pool of the scratch on one device: the device's default pool gives its memory
// back at every synchronisation (its release threshold is 0, and it is the process's to
// set), so a call after one paid a millisecond for 303 KB.  This one keeps up to 64 MB,
// which is its smallest piece of device memory (2 to 32 MB) at one call at a time; what
// calls overlapping on several streams or threads take beyond that goes back.  One per
// context: after a cudaDeviceReset the old context's pool is gone with it, and the new
// context's number finds none.
constexpr uint64_t kResPoolKeeps = 64ull << 20;

cudaError_t alloc_scratch(int device, double** p, cudaStream_t s) {
  static std::mutex mu;
  static std::map<unsigned long long, cudaMemPool_t> pools;
  static const auto entry = [](const char* name) -> void* {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    return cudaGetDriverEntryPoint(name, &fn, cudaEnableDefault, &q) == cudaSuccess &&
                   q == cudaDriverEntryPointSuccess
               ? fn
               : nullptr;
  };
  static const auto current = reinterpret_cast<CUresult (*)(CUcontext*)>(entry("cuCtxGetCurrent"));
  static const auto number = reinterpret_cast<CUresult (*)(CUcontext, unsigned long long*)>(entry("cuCtxGetId"));
  cudaMemPool_t pool = nullptr;
  CUcontext ctx = nullptr;
  unsigned long long id = 0;
  // a captured call keeps to the plain node it always was
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  const bool plain = cudaStreamIsCapturing(s, &cap) == cudaSuccess && cap == cudaStreamCaptureStatusNone;
  if (plain && current && number && current(&ctx) == CUDA_SUCCESS && ctx &&
      number(ctx, &id) == CUDA_SUCCESS) {
    std::lock_guard<std::mutex> lk(mu);
    cudaMemPool_t& kept = pools[id];
    if (!kept) {
      cudaMemPoolProps props = {};
      props.allocType = cudaMemAllocationTypePinned;
      props.location.type = cudaMemLocationTypeDevice;
      props.location.id = device;
      uint64_t keep = kResPoolKeeps;
      if (cudaMemPoolCreate(&kept, &props) != cudaSuccess)
        kept = nullptr;
      else
        cudaMemPoolSetAttribute(kept, cudaMemPoolAttrReleaseThreshold, &keep);
    }
    pool = kept;
  }
  if (!pool) {
    if (plain) cudaGetLastError();
    return cudaMallocAsync((void**)p, tdem::kResScratchBytes, s);
  }
  return cudaMallocFromPoolAsync((void**)p, tdem::kResScratchBytes, pool, s);
}

}  // namespace

extern "C" tdem_status tdem_residual_norms(int device, int64_t n, const int64_t* rowptr, const int* col,
                                           const double* val, const double* x, const double* b, int64_t ld,
                                           int ncols, double* norms, void* stream) {
  if (tdem::check_residual_args(n, rowptr, col, val, x, b, ld, ncols, norms)) return TDEM_ERR_ARGUMENT;
  DeviceGuard g(device);
  if (g.err != cudaSuccess) return TDEM_ERR_CUDA;
  cudaStream_t s = (cudaStream_t)stream;
  double* scratch = nullptr;
  if (alloc_scratch(device, &scratch, s) != cudaSuccess) return TDEM_ERR_CUDA;
  const cudaError_t e = tdem::launch_residual_norms(n, rowptr, col, val, x, b, ld, ncols, norms, scratch, s);
  const cudaError_t f = cudaFreeAsync(scratch, s);
  return (e == cudaSuccess && f == cudaSuccess) ? TDEM_OK : TDEM_ERR_CUDA;
}

// ---------------------------------------------------------------------------
// Allocation-free variant: the scratch is a file-scope device array of fixed
// size (kResScratchBytes = 303,104 bytes: 296 CTAs x 64 columns x 2 sums), so a
// call makes no device allocation.  Its device address is looked up on every
// call (cudaGetSymbolAddress, with the call's device current): cheap once the
// module is loaded, and never stale, also after a caller's cudaDeviceReset.  The
// first call on a device may load the module and should happen before any stream
// capture.  The scratch needs no initial value (pass 1 writes every entry pass 2
// reads).  Calls whose executions overlap on one device share the scratch and
// race: order them on one stream or synchronise between them.
// ---------------------------------------------------------------------------
namespace {

__device__ __align__(256) double g_res_scratch[tdem::kResBlocks * tdem::kResMaxCols * 2];

constexpr int kMaxDevices = 64;

// Device address of g_res_scratch on the current device (nullptr on failure).
double* scratch_address() {
  void* p = nullptr;
  if (cudaGetSymbolAddress(&p, g_res_scratch) != cudaSuccess) return nullptr;
  return static_cast<double*>(p);
}

}  // namespace

extern "C" tdem_status tdem_residual_norms_noalloc(int device, int64_t n, const int64_t* rowptr, const int* col,
                                                   const double* val, const double* x, const double* b, int64_t ld,
                                                   int ncols, double* norms, void* stream) {
  if (tdem::check_residual_args(n, rowptr, col, val, x, b, ld, ncols, norms)) return TDEM_ERR_ARGUMENT;
  if (device < 0 || device >= kMaxDevices) return TDEM_ERR_ARGUMENT;
  DeviceGuard g(device);
  if (g.err != cudaSuccess) return TDEM_ERR_CUDA;
  double* scratch = scratch_address();
  if (!scratch) return TDEM_ERR_CUDA;
  const cudaError_t e =
      tdem::launch_residual_norms(n, rowptr, col, val, x, b, ld, ncols, norms, scratch, (cudaStream_t)stream);
  return e == cudaSuccess ? TDEM_OK : TDEM_ERR_CUDA;
}
