// ibm_residual_noalloc: r = b - A x and the norms ||r||_2, ||b||_2 for one
// 7-point operator, with no device allocation at all.
//
// Who needs this: callers that cannot call cudaMalloc. Typical ones hand all
// free device memory to their own pool allocator at start-up (so a foreign
// cudaMalloc fails or fragments their pool), run under a fixed device-memory
// budget where an out-of-memory error mid-run is not acceptable, or cannot
// accept the device-wide synchronisation that cudaFree implies. Every other
// entry point of this library works through a context, and creating a context
// allocates; this one needs none.
//
// Its only scratch is the file-scope array below: per-block partial sums of the
// two norms and the counter that elects the block finishing the reduction.
// The array lives in the library's module and is held on every device that
// loads the library until the process exits. Its address in the current
// context is looked up with cudaGetSymbolAddress on every call made outside
// stream capture, so a device reset or another context made current on the
// device is followed; a call made while its stream is being captured reuses
// the address found by the last uncaptured call on that device. In host code
// the array's name is only a stand-in for the symbol, never a device address.
#include <algorithm>
#include <cmath>
#include <mutex>

#include "ibm_common.cuh"

namespace ibm {
namespace {

constexpr long kNaMaxRows = IBM_NOALLOC_MAX_ROWS;
constexpr int kNaMaxTiles = (int)(kNaMaxRows / kTile);
constexpr int kNaMaxDevices = 64;
static_assert(kNaMaxRows % kTile == 0, "the row limit is a whole number of tiles");

struct NoAllocScratch {
  double part[2 * kNaMaxTiles];  // per block: sum r^2, sum b^2
  unsigned ticket;               // blocks finished; cleared before every launch
};

}  // namespace

// 2 * 32768 doubles + the counter: 512 KiB + 256 B per device.
static __device__ __align__(256) NoAllocScratch g_noalloc_scratch;

namespace {

// A warp takes 32 rows at a time and keeps kNaStages such chunks on their way.
constexpr int kNaStages = 3;
constexpr int kNaBlocksPerSm = 2;
constexpr int kNaChunk = 32 * 7;  // coefficients of a chunk

template <int BYTES>
__device__ __forceinline__ void copy_async(double *smem, const double *g) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem);
  if constexpr (BYTES == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(g) : "memory");
  else asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(d), "l"(g) : "memory");
}

// The rows' coefficients lie row by row (56 bytes each): read by the thread of
// each row they are seven 8-byte loads 56 bytes apart across the lanes, which
// touch the same 14 lines seven times. So a warp copies the rows of its next
// chunks to shared memory as they lie, 16 bytes a lane (8 when vals is aligned
// to 8 only), while it sums the present one; a row's values are then 14 words
// apart between neighbouring lanes, which no two lanes of a half-warp have in
// one bank. Warps run free of each other, so that one's FP64 work (10
// operations a row, 75 us at 512x96x96) covers another's loads (57 us at the
// copy bandwidth). A call at that size took 125 us and takes 94; with one copy
// of a whole tile per block and a barrier it took 156, since blocks then load
// and compute in step.
//
// The norms' sums count beside ten operations a row: with four blocks an SM and
// a butterfly of both sums in every warp, a call on 131072 rows (one chunk a
// warp) spent as much FP64 issue there as on its rows, 16.5 us in a graph. With
// two blocks an SM, twice the chunks a warp, and the sums by two warps of a block
// it takes 12.4, as a block per 1024 rows did; 1M rows 28.4 (31.7; 35.0 so).
//
// The stencil is evaluated in the same order as the context path's operator
// apply (centre, -x, +x, -y, +y, -z, +z, one fma each), so r is bitwise equal
// to b - ibm_apply_operator(x). The norms are summed in a fixed order (chunks
// of a warp, lanes, warps, blocks), so the result does not depend on which
// block finishes last.
__global__ void __launch_bounds__(kThreads, kNaBlocksPerSm)
    k_residual_noalloc(const double *__restrict__ vals, Box bx, int aligned16, const double *__restrict__ x,
                       const double *__restrict__ b, double *__restrict__ r, double *__restrict__ norms,
                       NoAllocScratch *sc) {
  __shared__ __align__(16) double rows[kWarps][kNaStages][kNaChunk];
  __shared__ double srr[kWarps], sbb[kWarps];
  __shared__ int last;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nx = bx.nx, ny = bx.ny, nz = bx.nz;
  const long n = bx.n, sy = nx, sz = (long)nx * ny;
  const int chunks = (int)((n + 31) / 32), step = gridDim.x * kWarps;
  // copies chunk c (none past the end); every call commits one group
  auto fetch = [&](int c, int stage) {
    if (c < chunks) {
      const double *src = vals + (long)c * kNaChunk;
      double *dst = rows[warp][stage];
      const int count = (int)(n - 32l * c < 32 ? (n - 32l * c) * 7 : kNaChunk);
      if (aligned16) {
        for (int e = 2 * lane; e < count; e += 64) {
          if (e + 1 < count) copy_async<16>(dst + e, src + e);
          else copy_async<8>(dst + e, src + e);
        }
      } else {
        for (int e = lane; e < count; e += 32) copy_async<8>(dst + e, src + e);
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };
  int c = blockIdx.x * kWarps + warp;
#pragma unroll
  for (int q = 0; q < kNaStages - 1; ++q) fetch(c + q * step, q);
  double rr = 0.0, bb = 0.0;
  for (int stage = 0; c < chunks; c += step) {
    const long row = 32l * c + lane;
    const bool in = row < n;
    int i = 0, j = 0, k = 0;
    if (in) box_ijk(row, bx, i, j, k);
    const double x0 = in ? x[row] : 0.0, xw = in && i > 0 ? x[row - 1] : 0.0, xe = in && i < nx - 1 ? x[row + 1] : 0.0,
                 xs = in && j > 0 ? x[row - sy] : 0.0, xn = in && j < ny - 1 ? x[row + sy] : 0.0,
                 xb = in && k > 0 ? x[row - sz] : 0.0, xt = in && k < nz - 1 ? x[row + sz] : 0.0;
    const double bv = in ? b[row] : 0.0;
    asm volatile("cp.async.wait_group %0;" ::"n"(kNaStages - 2) : "memory");
    __syncwarp();  // every lane's copies are in, and the stage refilled next has been read by all
    int next = stage + kNaStages - 1;
    if (next >= kNaStages) next -= kNaStages;
    fetch(c + (kNaStages - 1) * step, next);
    if (in) {
      const double *v = rows[warp][stage] + 7 * lane;
      double acc = 0.0;
      acc = fma(v[0], x0, acc);
      acc = fma(v[1], xw, acc);
      acc = fma(v[2], xe, acc);
      acc = fma(v[3], xs, acc);
      acc = fma(v[4], xn, acc);
      acc = fma(v[5], xb, acc);
      acc = fma(v[6], xt, acc);
      const double rv = bv - acc;
      r[row] = rv;
      rr = fma(rv, rv, rr);
      bb = fma(bv, bv, bb);
    }
    if (++stage == kNaStages) stage = 0;
  }
  // the block's sums by two warps, each lane first the eight warps' values of
  // its place: 26 warp-wide FP64 instructions a block, not 80
  double(*const sums)[kThreads] = reinterpret_cast<double(*)[kThreads]>(&rows[0][0][0]);
  __syncthreads();  // every warp has read its rows
  sums[0][threadIdx.x] = rr;
  sums[1][threadIdx.x] = bb;
  __syncthreads();
  if (warp < 2) {
    double a = 0.0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) a += sums[warp][32 * w + lane];
    a = warp_sum(a);
    if (lane == 0) sc->part[2 * blockIdx.x + warp] = a;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    last = atomicAdd(&sc->ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double a = 0.0, e = 0.0;
  for (int q = threadIdx.x; q < (int)gridDim.x; q += kThreads) {
    a += __ldcg(&sc->part[2 * q]);
    e += __ldcg(&sc->part[2 * q + 1]);
  }
  a = warp_sum(a);
  e = warp_sum(e);
  __syncthreads();
  if (lane == 0) {
    srr[warp] = a;
    sbb[warp] = e;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    double ta = 0.0, te = 0.0;
    for (int w = 0; w < kWarps; ++w) {
      ta += srr[w];
      te += sbb[w];
    }
    norms[0] = sqrt(ta);
    norms[1] = sqrt(te);
    sc->ticket = 0;
  }
}

std::mutex g_na_mutex;
NoAllocScratch *g_na_ptr[kNaMaxDevices] = {};

// The scratch address in the current context. Outside capture it is looked
// up again (cheap, and correct after cudaDeviceReset or with a non-primary
// context current); during capture the last address found on the device is
// used, since the lookup itself may load the module and is not a stream
// operation that capture records.
cudaError_t scratch_on_device(int dev, bool capturing, NoAllocScratch **out) {
  std::lock_guard<std::mutex> lock(g_na_mutex);
  if (!capturing || !g_na_ptr[dev]) {
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) return e;
    g_na_ptr[dev] = (NoAllocScratch *)p;
  }
  *out = g_na_ptr[dev];
  return cudaSuccess;
}

// [a, a + na) and [b, b + nb) share a byte.
bool overlaps(const void *a, size_t na, const void *b, size_t nb) {
  const char *pa = (const char *)a, *pb = (const char *)b;
  return pa < pb + nb && pb < pa + na;
}

bool on_device(const void *p, int dev) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (a.type == cudaMemoryTypeManaged) return true;
  return a.type == cudaMemoryTypeDevice && a.device == dev;
}

}  // namespace
}  // namespace ibm

extern "C" int ibm_residual_noalloc(const double *vals, int nx, int ny, int nz, const double *x, const double *b,
                                    double *r, double *norms, void *stream) {
  using namespace ibm;
  if (!vals || !x || !b || !r || !norms || nx <= 0 || ny <= 0 || nz <= 0) return IBM_ERR_ARG;
  const long n = (long)nx * ny * nz;
  if (n > kNaMaxRows) return IBM_ERR_TOO_LARGE;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return IBM_ERR_CUDA;
  if (dev < 0 || dev >= kNaMaxDevices) return IBM_ERR_UNSUPPORTED;
  // r and norms are written while other blocks still read x and b (each row
  // reads its six neighbours): an output sharing memory with an input races.
  const size_t vb = (size_t)n * sizeof(double), nb = 2 * sizeof(double);
  if (overlaps(r, vb, x, vb) || overlaps(r, vb, b, vb) || overlaps(r, vb, vals, 7 * vb) ||
      overlaps(norms, nb, x, vb) || overlaps(norms, nb, b, vb) || overlaps(norms, nb, r, vb) ||
      overlaps(norms, nb, vals, 7 * vb))
    return IBM_ERR_ARG;
  for (const void *p : {(const void *)vals, (const void *)x, (const void *)b, (const void *)r, (const void *)norms})
    if (!on_device(p, dev)) return IBM_ERR_ARG;
  cudaStream_t st = (cudaStream_t)stream;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(st, &cs) != cudaSuccess) return IBM_ERR_CUDA;
  NoAllocScratch *sc = nullptr;
  if (scratch_on_device(dev, cs != cudaStreamCaptureStatusNone, &sc) != cudaSuccess) return IBM_ERR_CUDA;
  if (cudaMemsetAsync(&sc->ticket, 0, sizeof(unsigned), st) != cudaSuccess) return IBM_ERR_CUDA;
  int sms = 0;
  if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return IBM_ERR_CUDA;
  // one chunk per warp up to one resident wave; 152 x 2 blocks are within the scratch's tiles on any device
  const long blocks = (n + 32 * kWarps - 1) / (32 * kWarps);
  const int grid = (int)std::min({blocks, (long)sms * kNaBlocksPerSm, (long)kNaMaxTiles});
  k_residual_noalloc<<<grid, kThreads, 0, st>>>(vals, make_box(nx, ny, nz),
                                                reinterpret_cast<uintptr_t>(vals) % 16 == 0, x, b, r, norms, sc);
  return cudaGetLastError() == cudaSuccess ? IBM_OK : IBM_ERR_CUDA;
}
