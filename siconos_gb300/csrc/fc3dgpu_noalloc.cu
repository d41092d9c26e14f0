// fc3d_compute_error on a problem that is already in device memory, with no
// device allocation at all: the variant of the solver's error evaluation
// (u = q + W r and the natural-map residual, reduced over all contacts)
// whose scratch -- per-chunk partial sums and a completion ticket -- lives in
// a fixed file-scope device array instead of buffers owned by a context.
//
// Callers that cannot let a library allocate: applications that hand all
// device memory to their own pool (a cudaMalloc or cudaFree would synchronise
// the device and stall their other streams in the middle of a time step, or
// fail because the pool has taken the memory).
//
// The reduction order is fixed by the chunking (chunk_of(nc) contacts per
// chunk, chunks summed in index order), so the result does not depend on the
// grid.
//
// What bounds it: the FP64 unit (a warp instruction in 64 cycles per SM
// quarter: 9 fused multiply-adds a block of W against 72 bytes, 21 us of
// arithmetic against 13 us of HBM time for 94,400 contacts), and below some
// 20,000 contacts one row's chain of them.  So three threads share a row, one
// component each (a third of the chain, and their loads of a block and stores
// of the velocity are contiguous), then one thread a contact forms the
// natural map from shared memory; chunks are small, so that few contacts
// still reach every SM and the last round is short; and the completion
// tickets rotate instead of being cleared by a copy operation before every
// launch.  21.2 -> 9.0 us at 16 contacts, 33.6 -> 16.9 at 23,200, 76.2 -> 41.3 at
// 94,400, 210 -> 147 at 320,400 (back to back on the device).
#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include <mutex>

#include "fc3dgpu.h"
#include "fc3dgpu_local64.cuh"

extern "C" void fc3dgpu_set_error(const char* fmt, ...);

namespace fc3dgpu {
namespace noalloc {

// Contacts per chunk: 64, which spreads few contacts over the SMs, or 256 where 64
// would make more chunks than the last block sums quickly (and, beyond 2^20
// contacts, than the scratch holds).  us a call with 64 and 256: 480 contacts 12.4
// and 24.6, 40,935 24.6 and 39.0, 94,400 43.1 and 53.3, 320,400 151.6 and 149.6,
// 509,600 238 and 222, 968,352 444 and 390.
constexpr int SMALL_CHUNK = 64, LARGE_CHUNK = 256;
constexpr int SMALL_MAX = 1 << 18;  // contacts
static int chunk_of(int nc) { return nc <= SMALL_MAX ? SMALL_CHUNK : LARGE_CHUNK; }
constexpr int MAX_CHUNKS = FC3DGPU_NOALLOC_MAX_CONTACTS / LARGE_CHUNK;
static_assert(MAX_CHUNKS * LARGE_CHUNK == FC3DGPU_NOALLOC_MAX_CONTACTS, "limit must be a multiple of the chunk");
static_assert(SMALL_MAX / SMALL_CHUNK <= MAX_CHUNKS, "the scratch holds the small chunks");
// 3 partial sums per chunk, then one 256-byte line of SLOTS completion slots
// (ticket, bad-input flag).  A call takes the next slot; a launch that
// completes leaves its slot at zero and clears the one half a turn ahead, so
// what an interrupted launch leaves is gone before its slot's turn comes again.
// A call that is captured keeps its slot in every replay: there a copy
// operation clears the slot before each launch.
constexpr int SLOTS = 16;
constexpr int SCRATCH_DOUBLES = 3 * MAX_CHUNKS + 32;
static_assert(SCRATCH_DOUBLES * 8 == FC3DGPU_NOALLOC_SCRATCH_BYTES, "header states the scratch size");

static __device__ __align__(256) double g_scratch[SCRATCH_DOUBLES];

// Sums of three values over the first CH threads of the block (the others
// pass nothing), warps in order; every thread gets them.
template <int CH>
__device__ __forceinline__ void block_sum3(double v[3], double (*sh)[3]) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (threadIdx.x < CH) {
#pragma unroll
    for (int k = 0; k < 3; k++) {
      double x = v[k];
#pragma unroll
      for (int o = 16; o >= 1; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
      if (lane == 0) sh[w][k] = x;
    }
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < 3; k++) {
    double s = sh[0][k];
#pragma unroll
    for (int i = 1; i < CH / 32; i++) s += sh[i][k];
    v[k] = s;
  }
}

// Rows are read in the caller's block-CSR order (the diagonal block at its
// own position), as SBM_gemv_3x3 does (SparseBlockMatrix.c:360-419).  A row
// pointer or column index out of range is not followed: the error becomes
// NaN.
template <int CH>
__global__ void __launch_bounds__(3 * CH) k_error_noalloc(int nc, long long nnz, const int64_t* __restrict__ rowptr,
                                                          const int64_t* __restrict__ colidx,
                                                          const double* __restrict__ blocks,
                                                          const double* __restrict__ q, const double* __restrict__ mu,
                                                          const double* __restrict__ r, double norm_q,
                                                          double* __restrict__ velocity, double* __restrict__ error,
                                                          double* __restrict__ scratch, int slot) {
  __shared__ double su[3 * CH], sr[3 * CH];
  __shared__ double sh[CH / 32][3];
  __shared__ int last;
  double* part = scratch;
  unsigned* slots = reinterpret_cast<unsigned*>(scratch + 3 * MAX_CHUNKS);
  unsigned *ticket = slots + 2 * slot, *bad = ticket + 1;
  const int nchunks = (nc + CH - 1) / CH;
  int badl = 0;
  const int t = threadIdx.x, comp = t % 3;
  for (int ch = blockIdx.x; ch < nchunks; ch += gridDim.x) {
    const size_t x0 = (size_t)3 * ch * CH + t;  // the thread's entry of the vectors
    const int i = ch * CH + t / 3;
    if (i < nc) {
      double u = q[x0];
      const long long b0 = rowptr[i], b1 = rowptr[i + 1];
      if (b0 < 0 || b1 < b0 || b1 > nnz) {
        badl = 1;
      } else {
        // blocks four at a time: their columns, then their values and
        // reactions, are requested together; a column out of range (-1, as
        // behind the row's end) is left out and flags the input
        constexpr int U = 4;
        for (long long b = b0; b < b1; b += U) {
          long long j[U];
          double wv[U][3], rv[U][3];
#pragma unroll
          for (int k = 0; k < U; k++) {
            j[k] = b + k < b1 ? __ldg(&colidx[b + k]) : -1;
            if (j[k] < 0 || j[k] >= nc) {
              if (b + k < b1) badl = 1;
              j[k] = -1;
            }
          }
#pragma unroll
          for (int k = 0; k < U; k++)
#pragma unroll
            for (int e = 0; e < 3; e++) {
              wv[k][e] = b + k < b1 ? __ldg(&blocks[9 * (b + k) + 3 * e + comp]) : 0.0;
              rv[k][e] = b + k < b1 ? __ldg(&r[3 * (j[k] < 0 ? 0 : j[k]) + e]) : 0.0;
            }
#pragma unroll
          for (int k = 0; k < U; k++)
            if (j[k] >= 0)
#pragma unroll
              for (int e = 0; e < 3; e++) u = fma(wv[k][e], rv[k][e], u);
        }
      }
      su[t] = u;
      sr[t] = r[x0];
      if (velocity) velocity[x0] = u;
    }
    __syncthreads();
    double v[3] = {0.0, 0.0, 0.0};
    const int i1 = ch * CH + t;
    if (t < CH && i1 < nc) {
      const double uu[3] = {su[3 * t], su[3 * t + 1], su[3 * t + 2]}, rr[3] = {sr[3 * t], sr[3 * t + 1], sr[3 * t + 2]};
      v[0] = unitary_error2<double>(rr, uu, mu[i1]);
      v[1] = fma(uu[2], uu[2], fma(uu[1], uu[1], uu[0] * uu[0]));
      v[2] = fma(rr[2], rr[2], fma(rr[1], rr[1], rr[0] * rr[0]));
    }
    block_sum3<CH>(v, sh);
    if (t == 0) {
      part[3 * ch] = v[0];
      part[3 * ch + 1] = v[1];
      part[3 * ch + 2] = v[2];
    }
    __syncthreads();  // sh and the vectors are free for the next chunk
  }
  if (__syncthreads_or(badl) && t == 0) atomicOr(bad, 1u);
  // the last block to finish sums the chunk partials in chunk order
  if (t == 0) {
    __threadfence();
    last = atomicAdd(ticket, 1u) == gridDim.x - 1;
  }
  __syncthreads();
  if (!last) return;
  __threadfence();
  double v[3] = {0.0, 0.0, 0.0};
  if (t < CH) {
#pragma unroll 4
    for (int ch = t; ch < nchunks; ch += CH) {
      v[0] += __ldcg(&part[3 * ch]);
      v[1] += __ldcg(&part[3 * ch + 1]);
      v[2] += __ldcg(&part[3 * ch + 2]);
    }
  }
  block_sum3<CH>(v, sh);
  if (t == 0) {
    double e = ie_sqrt(v[0]);
    const double scal = fmax(norm_q, fmax(ie_sqrt(v[2]), ie_sqrt(v[1])));
    if (fabs(scal) > DBL_EPSILON) e = ie_div(e, scal);
    *error = atomicOr(bad, 0u) ? __longlong_as_double(0x7ff8000000000000LL) : e;
    *ticket = 0u;
    *bad = 0u;
    const int ahead = (slot + SLOTS / 2) % SLOTS;
    slots[2 * ahead] = 0u;
    slots[2 * ahead + 1] = 0u;
  }
}

// Address of g_scratch and SM count per device, looked up at the first call
// with that device current.  The address belongs to the CUDA context that was
// current then (the device's primary context, unless the caller made another
// driver context current): the entry is keyed by that context and looked up
// again when another context is current, e.g. after cudaDeviceReset.
constexpr int MAX_DEVICES = 64;
std::mutex g_mutex;
struct Entry {
  void* ctx;
  double* addr;
  int sms;
  unsigned calls;
};
Entry g_entry[MAX_DEVICES];
typedef int (*CtxGetCurrent)(void**);  // cuCtxGetCurrent, through the runtime
CtxGetCurrent g_ctx_current = nullptr;

static void* current_context() {
  void* ctx = nullptr;
  if (g_ctx_current && g_ctx_current(&ctx) != 0) ctx = nullptr;
  return ctx;
}

int setup(int dev, double** addr, int* sms, int* slot) {
  std::lock_guard<std::mutex> lock(g_mutex);
  if (!g_ctx_current) {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess || !fn) {
      cudaGetLastError();
      fc3dgpu_set_error("fc3dgpu_compute_error_device: cuCtxGetCurrent is not available");
      return NUMERICS_ERR_NOT_IMPLEMENTED;
    }
    g_ctx_current = reinterpret_cast<CtxGetCurrent>(fn);
  }
  Entry& en = g_entry[dev];
  void* ctx = current_context();
  if (!en.addr || !ctx || ctx != en.ctx) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_scratch);
    if (e != cudaSuccess || !p) {
      cudaGetLastError();
      fc3dgpu_set_error("fc3dgpu_compute_error_device: cudaGetSymbolAddress on device %d: %s", dev,
                        cudaGetErrorString(e));
      return NUMERICS_ERR_UNKNOWN;
    }
    int n = 0;
    e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
    if (e != cudaSuccess || n <= 0) {
      cudaGetLastError();
      fc3dgpu_set_error("fc3dgpu_compute_error_device: SM count of device %d: %s", dev, cudaGetErrorString(e));
      return NUMERICS_ERR_UNKNOWN;
    }
    en.ctx = current_context();  // the look-up made the primary context current if none was
    en.sms = n;
    en.addr = static_cast<double*>(p);
  }
  *addr = en.addr;
  *sms = en.sms;
  *slot = (int)(en.calls++ % SLOTS);
  return 0;
}

// Memory a kernel on device dev may read or write through p as given: device
// memory of that device (memory of another device is refused, since peer
// access may be off), managed memory, or mapped pinned host memory whose
// device address is p itself.
bool device_accessible(const void* p, int dev) {
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  switch (at.type) {
    case cudaMemoryTypeDevice: return at.device == dev;
    case cudaMemoryTypeManaged: return true;
    case cudaMemoryTypeHost: return at.devicePointer == p;
    default: return false;
  }
}

}  // namespace noalloc
}  // namespace fc3dgpu

extern "C" int fc3dgpu_compute_error_device(int nc, int64_t nnz, const int64_t* rowptr, const int64_t* colidx,
                                            const double* blocks, const double* q, const double* mu,
                                            const double* reaction, double norm_q, double* velocity, double* error,
                                            void* stream) {
  using namespace fc3dgpu::noalloc;
  if (nc < 0 || nnz < 0) {
    fc3dgpu_set_error("fc3dgpu_compute_error_device: negative size (nc = %d, nnz = %lld)", nc, (long long)nnz);
    return NUMERICS_ERR_INVALID_ARGUMENT;
  }
  if (nc > FC3DGPU_NOALLOC_MAX_CONTACTS) {
    fc3dgpu_set_error(
        "fc3dgpu_compute_error_device: %d contacts exceed the limit of %d (FC3DGPU_NOALLOC_MAX_CONTACTS); use "
        "fc3dgpu_ctx_compute_error",
        nc, FC3DGPU_NOALLOC_MAX_CONTACTS);
    return NUMERICS_ERR_INVALID_ARGUMENT;
  }
  if (!error || !rowptr || (nc > 0 && (!q || !mu || !reaction)) || (nnz > 0 && (!colidx || !blocks))) {
    fc3dgpu_set_error("fc3dgpu_compute_error_device: null pointer");
    return NUMERICS_ERR_NULL_POINTER;
  }
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) {
    cudaGetLastError();
    fc3dgpu_set_error("fc3dgpu_compute_error_device: no current CUDA device (%s)", cudaGetErrorString(e));
    return NUMERICS_ERR_NOT_IMPLEMENTED;
  }
  if (dev < 0 || dev >= MAX_DEVICES) {
    fc3dgpu_set_error("fc3dgpu_compute_error_device: device %d beyond %d", dev, MAX_DEVICES);
    return NUMERICS_ERR_INVALID_ARGUMENT;
  }
  const void* ptrs[] = {rowptr, colidx, blocks, q, mu, reaction, velocity, error};
  for (const void* p : ptrs)
    if (p && !device_accessible(p, dev)) {
      fc3dgpu_set_error("fc3dgpu_compute_error_device: %p is not memory device %d can access", p, dev);
      return NUMERICS_ERR_INVALID_ARGUMENT;
    }
  double* scratch = nullptr;
  int sms = 0, slot = 0;
  int rc = setup(dev, &scratch, &sms, &slot);
  if (rc) return rc;
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  if (cudaStreamIsCapturing(s, &capture) != cudaSuccess) cudaGetLastError();  // the launch reports it
  if (capture == cudaStreamCaptureStatusActive) {
    e = cudaMemsetAsync(scratch + 3 * MAX_CHUNKS + slot, 0, 2 * sizeof(unsigned), s);
    if (e != cudaSuccess) {
      fc3dgpu_set_error("fc3dgpu_compute_error_device: %s", cudaGetErrorString(e));
      return NUMERICS_ERR_UNKNOWN;
    }
  }
  auto launch = [&](auto kernel, int chunk, int per_sm) {
    const int nchunks = (nc + chunk - 1) / chunk;
    int grid = per_sm * sms;
    if (grid > nchunks) grid = nchunks;
    if (grid < 1) grid = 1;
    kernel<<<grid, 3 * chunk, 0, s>>>(nc, (long long)nnz, rowptr, colidx, blocks, q, mu, reaction, norm_q, velocity,
                                      error, scratch, slot);
    return cudaGetLastError();
  };
  e = chunk_of(nc) == SMALL_CHUNK ? launch(k_error_noalloc<SMALL_CHUNK>, SMALL_CHUNK, 8)
                                  : launch(k_error_noalloc<LARGE_CHUNK>, LARGE_CHUNK, 2);
  if (e != cudaSuccess) {
    fc3dgpu_set_error("fc3dgpu_compute_error_device: %s", cudaGetErrorString(e));
    return NUMERICS_ERR_UNKNOWN;
  }
  return 0;
}
