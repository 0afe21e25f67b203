// Allocation-free variant of the dead-cell sweep (lbm_absorb_dead_cells_noalloc,
// declared in include/lbm_b200.h).
//
// Some callers cannot allocate device memory at the point where they need the
// sweep: an engine that hands out all device memory from its own fixed pool and
// forbids allocation elsewhere, a host process whose allocator is owned by
// another runtime, or a loop that must not pay the device-wide synchronisation a
// cudaMalloc / cudaFree can cost.  This entry point works on device arrays the
// caller already owns and keeps its own scratch -- the per-chunk counts, the
// totals and the scan-ordered cell lists of the compaction -- in one fixed,
// file-scope device array.  It calls no allocator, host or device.
//
// Limit: the search box (the union of the spheres' bounding boxes, clamped to
// the interior) may hold at most NOALLOC_MAX_BOX = 2^20 cells, e.g. one sphere
// of radius up to ~49 cells.  Every GPU that loads the library holds the array
// (about 8.4 MB) until the process exits.
//
// Set-up: the first call on each device, with that device current, looks up
// the array's device address (cudaGetSymbolAddress, which also loads this
// module onto the device).  Make that first call before any stream capture.
//
// Sharing: all calls on a device use the same array, which keeps the last
// call's contents.  Everything a call reads there it has written first (the
// plan, the counts of the chunks in use, the totals and the list entries below
// the totals), so nothing needs clearing between calls.  Calls whose kernels
// overlap on the GPU (different streams, or several host threads) race on the
// array and must be serialised by the caller.
#include <stdarg.h>
#include <stdio.h>
#include <string.h>

#include <mutex>

#include "lbm_kernels.cuh"
#include "lbm_state.h"

using namespace lbm;

namespace {

constexpr int COMPACT_THREADS = 256;

// Count fresh (FLUID, was SOLID) and dead (SOLID, was FLUID) cells per chunk
// of the box's linear (scan) order.
__global__ void k_compact_count(const uint8_t *tag, const uint8_t *tagPrev, int nx, int ny,
                                const Plan *__restrict__ P, int2 *counts) {
  __shared__ int sf[COMPACT_THREADS / 32], sd[COMPACT_THREADS / 32];
  const Box bx = P->U;
  const long long total = P->ucells;
  const int nchunks = P->nchunks;
  // CTAs stride over the chunks (block-uniform trip count)
  for (int c = blockIdx.x; c < nchunks; c += gridDim.x) {
    const long long base = (long long)c * COMPACT_CHUNK;
    int nf = 0, nd = 0;
    for (int j = threadIdx.x; j < COMPACT_CHUNK; j += blockDim.x) {
      long long l = base + j;
      if (l >= total) break;
      int x, y, z;
      box_cell(bx, l, x, y, z);
      long long i = cell_index(x, y, z, nx, ny);
      uint8_t t = tag[i], p = tagPrev[i];
      nf += (t == TAG_FLUID && p == TAG_SOLID);
      nd += (t == TAG_SOLID && p == TAG_FLUID);
    }
    for (int o = 16; o > 0; o >>= 1) {
      nf += __shfl_xor_sync(0xffffffffu, nf, o);
      nd += __shfl_xor_sync(0xffffffffu, nd, o);
    }
    if ((threadIdx.x & 31) == 0) {
      sf[threadIdx.x >> 5] = nf;
      sd[threadIdx.x >> 5] = nd;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      int a = 0, b = 0;
      for (int w = 0; w < (int)(blockDim.x >> 5); w++) {
        a += sf[w];
        b += sd[w];
      }
      counts[c] = make_int2(a, b);
    }
    __syncthreads();  // sf / sd are rewritten for the next chunk
  }
}

// Exclusive scan of the per-chunk counts (single CTA, sequential per thread).
__global__ void k_compact_scan(int2 *counts, const Plan *__restrict__ P, int *totals) {
  __shared__ int2 part[1024];
  const int nchunks = P->nchunks;
  int per = (nchunks + blockDim.x - 1) / blockDim.x;
  int b0 = threadIdx.x * per, b1 = min(b0 + per, nchunks);
  int2 sum = make_int2(0, 0);
  for (int b = b0; b < b1; b++) {
    sum.x += counts[b].x;
    sum.y += counts[b].y;
  }
  part[threadIdx.x] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    int2 run = make_int2(0, 0);
    for (int t = 0; t < (int)blockDim.x; t++) {
      int2 v = part[t];
      part[t] = run;
      run.x += v.x;
      run.y += v.y;
    }
    totals[0] = run.x;
    totals[1] = run.y;
  }
  __syncthreads();
  int2 run = part[threadIdx.x];
  for (int b = b0; b < b1; b++) {
    int2 v = counts[b];
    counts[b] = run;
    run.x += v.x;
    run.y += v.y;
  }
}

// Emit the fresh / dead cell indices in scan order.
__global__ void k_compact_emit(const uint8_t *tag, const uint8_t *tagPrev, int nx, int ny,
                               const Plan *__restrict__ P, const int2 *offsets, int *fresh, int *dead, int cap) {
  __shared__ int wf[COMPACT_THREADS / 32], wd[COMPACT_THREADS / 32];
  __shared__ int runF, runD;
  const Box bx = P->U;
  const long long total = P->ucells;
  const int nchunks = P->nchunks;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
  // CTAs stride over the chunks (block-uniform trip count); the inner loop
  // ends on a barrier, so runF / runD are free to be reset for the next chunk
  for (int c = blockIdx.x; c < nchunks; c += gridDim.x) {
    const long long base = (long long)c * COMPACT_CHUNK;
    if (threadIdx.x == 0) {
      runF = offsets[c].x;
      runD = offsets[c].y;
    }
    __syncthreads();
    for (int j0 = 0; j0 < COMPACT_CHUNK; j0 += blockDim.x) {
      long long l = base + j0 + threadIdx.x;
      bool isF = false, isD = false;
      long long i = 0;
      if (l < total && j0 + (int)threadIdx.x < COMPACT_CHUNK) {
        int x, y, z;
        box_cell(bx, l, x, y, z);
        i = cell_index(x, y, z, nx, ny);
        uint8_t t = tag[i], p = tagPrev[i];
        isF = (t == TAG_FLUID && p == TAG_SOLID);
        isD = (t == TAG_SOLID && p == TAG_FLUID);
      }
      unsigned bf = __ballot_sync(0xffffffffu, isF), bd = __ballot_sync(0xffffffffu, isD);
      if (lane == 0) {
        wf[warp] = __popc(bf);
        wd[warp] = __popc(bd);
      }
      __syncthreads();
      int offF = runF, offD = runD;
      for (int w = 0; w < warp; w++) {
        offF += wf[w];
        offD += wd[w];
      }
      unsigned below = (1u << lane) - 1u;
      if (isF) {
        int pos = offF + __popc(bf & below);
        if (pos < cap) fresh[pos] = (int)i;
      }
      if (isD) {
        int pos = offD + __popc(bd & below);
        if (pos < cap) dead[pos] = (int)i;
      }
      __syncthreads();
      if (threadIdx.x == 0) {
        int a = 0, b = 0;
        for (int w = 0; w < nw; w++) {
          a += wf[w];
          b += wd[w];
        }
        runF += a;
        runD += b;
      }
      __syncthreads();
    }
  }
}

constexpr long long NOALLOC_MAX_BOX = 1LL << 20;  // cells of the search box
constexpr int NOALLOC_MAX_CHUNKS = (int)(NOALLOC_MAX_BOX / COMPACT_CHUNK);
constexpr int NOALLOC_MAX_DEVICES = 64;

struct NoAllocScratch {
  Plan plan;
  int totals[2];
  int2 counts[NOALLOC_MAX_CHUNKS];
  int fresh[NOALLOC_MAX_BOX];
  int dead[NOALLOC_MAX_BOX];
};

std::mutex g_mu;
NoAllocScratch *g_scratch[NOALLOC_MAX_DEVICES] = {nullptr};

int fail(char *err, size_t errlen, int code, const char *fmt, ...) {
  if (err && errlen > 0) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(err, errlen, fmt, ap);
    va_end(ap);
  }
  return code;
}

__global__ void k_noalloc_set_plan(Plan *dst, const __grid_constant__ Plan src) {
  if (blockIdx.x == 0 && threadIdx.x == 0) *dst = src;
}

bool on_device(const void *p) {
  cudaPointerAttributes at;
  if (!p || cudaPointerGetAttributes(&at, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return at.type == cudaMemoryTypeDevice || at.type == cudaMemoryTypeManaged;
}

}  // namespace

// The scratch.  In host code this name only identifies the array for
// cudaGetSymbolAddress; it is not a device address.
static __device__ __align__(256) unsigned char lbm_noalloc_scratch[sizeof(NoAllocScratch)];

extern "C" int lbm_absorb_dead_cells_noalloc(int nx, int ny, int nz, double rhoL, double rhoG,
                                             const uint8_t *tag, const uint8_t *tagPrev,
                                             const float *phi, const float *ux, const float *uy,
                                             const float *uz, const lbm_sphere *spheres,
                                             int nspheres, double *out, void *stream, char *err,
                                             size_t errlen) {
  if (err && errlen > 0) err[0] = '\0';
  if (nx < 3 || ny < 3 || nz < 3 || (long long)nx * ny * nz >= (1LL << 31))
    return fail(err, errlen, LBM_ERR_ARG, "grid %d x %d x %d out of range", nx, ny, nz);
  if (nspheres < 0 || nspheres > LBM_MAX_SPHERES)
    return fail(err, errlen, LBM_ERR_ARG, "nspheres %d outside [0, %d]", nspheres, LBM_MAX_SPHERES);
  if (nspheres == 0) return LBM_OK;
  if (!spheres) return fail(err, errlen, LBM_ERR_ARG, "spheres is NULL");

  // search box: dead cells are SOLID, so they lie inside the spheres' boxes
  Plan P;
  memset(&P, 0, sizeof(P));
  Box U{{1, 1, 1}, {0, 0, 0}};
  P.ss.nsph = nspheres;
  for (int b = 0; b < nspheres; b++) {
    SphereDesc &d = P.ss.sph[b];
    d.cx = spheres[b].cx;
    d.cy = spheres[b].cy;
    d.cz = spheres[b].cz;
    d.r = spheres[b].r;
    d.vx = spheres[b].vx;
    d.vy = spheres[b].vy;
    d.vz = spheres[b].vz;
    d.wx = spheres[b].wx;
    d.wy = spheres[b].wy;
    d.wz = spheres[b].wz;
    U = box_union(U, sphere_box(d.cx, d.cy, d.cz, d.r, nx, ny, nz));
  }
  const long long cells = box_cells(U);
  if (cells > NOALLOC_MAX_BOX)
    return fail(err, errlen, LBM_ERR_CAPACITY,
                "the spheres' search box holds %lld cells; this entry point handles at most %lld "
                "(use lbm_absorb_dead_cells for larger spheres)",
                cells, NOALLOC_MAX_BOX);
  if (cells == 0) {
    // no interior cell can be SOLID: the impulse is zero
    if (!on_device(out)) return fail(err, errlen, LBM_ERR_ARG, "out must be a device pointer");
    cudaError_t e = cudaMemsetAsync(out, 0, (size_t)nspheres * 6 * sizeof(double), (cudaStream_t)stream);
    if (e != cudaSuccess) return fail(err, errlen, LBM_ERR_CUDA, "cudaMemsetAsync: %s", cudaGetErrorString(e));
    return LBM_OK;
  }
  const void *dptrs[] = {tag, tagPrev, phi, ux, uy, uz, out};
  for (const void *p : dptrs)
    if (!on_device(p))
      return fail(err, errlen, LBM_ERR_ARG, "tag, tagPrev, phi, ux, uy, uz and out must be device pointers");
  P.U = U;
  P.ucells = cells;
  P.nchunks = (int)((cells + COMPACT_CHUNK - 1) / COMPACT_CHUNK);

  // set-up, once per device, with that device current
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= NOALLOC_MAX_DEVICES)
    return fail(err, errlen, LBM_ERR_CUDA, "no usable current CUDA device");
  NoAllocScratch *S = nullptr;
  {
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_scratch[dev]) {
      void *p = nullptr;
      e = cudaGetSymbolAddress(&p, lbm_noalloc_scratch);
      if (e != cudaSuccess || !p) {
        cudaGetLastError();
        return fail(err, errlen, LBM_ERR_CUDA, "cudaGetSymbolAddress: %s", cudaGetErrorString(e));
      }
      g_scratch[dev] = (NoAllocScratch *)p;
    }
    S = g_scratch[dev];
  }

  cudaStream_t s = (cudaStream_t)stream;
  const unsigned grid = (unsigned)P.nchunks;  // 1 .. NOALLOC_MAX_CHUNKS
  k_noalloc_set_plan<<<1, 1, 0, s>>>(&S->plan, P);
  k_compact_count<<<grid, COMPACT_THREADS, 0, s>>>(tag, tagPrev, nx, ny, &S->plan, S->counts);
  k_compact_scan<<<1, 1024, 0, s>>>(S->counts, &S->plan, S->totals);
  k_compact_emit<<<grid, COMPACT_THREADS, 0, s>>>(tag, tagPrev, nx, ny, &S->plan, S->counts, S->fresh,
                                                   S->dead, (int)NOALLOC_MAX_BOX);
  k_absorb_dead<float><<<nspheres, DEAD_THREADS, 0, s>>>(phi, ux, uy, uz, nx, ny, S->dead, S->totals,
                                                          (int)NOALLOC_MAX_BOX, rhoL, rhoG,
                                                          &S->plan.ss, out);
  e = cudaGetLastError();
  if (e != cudaSuccess) return fail(err, errlen, LBM_ERR_CUDA, "launch: %s", cudaGetErrorString(e));
  return LBM_OK;
}
