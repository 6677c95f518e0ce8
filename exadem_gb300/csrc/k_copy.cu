// k_copy.cu -- several device-to-device copies or fills in one launch.
//
// The particle set is 31 arrays and the list 13: one cudaMemcpyAsync each cost 2 to 3
// us on the stream, 60 to 100 us for a read-back or a restore of any size up to some
// 10,000 particles.  One launch takes a table of them, a row of blocks per entry;
// large copies run at the memory's rate as before (four 16-byte loads in flight a
// thread).
#include <cuda.h>  // types of the driver's range query (no symbol of it is linked)

#include <algorithm>

#include "../../include/dem_selftest.h"
#include "dem_ctx.cuh"

namespace dem {
namespace {
constexpr int CP_THREADS = 256;

template <class T>
__device__ __forceinline__ void copy_words(T* __restrict__ d, const T* __restrict__ s, uint64_t n, uint64_t t,
                                           uint64_t stride) {
  uint64_t k = t;
  for (; k + 3 * stride < n; k += 4 * stride) {
    const T a = s[k], b = s[k + stride], c = s[k + 2 * stride], e = s[k + 3 * stride];
    d[k] = a;
    d[k + stride] = b;
    d[k + 2 * stride] = c;
    d[k + 3 * stride] = e;
  }
  for (; k < n; k += stride) d[k] = s[k];
}

__global__ void __launch_bounds__(CP_THREADS) k_copies(const __grid_constant__ CopyTab t) {
  const int e = blockIdx.y;
  const uint64_t bytes = t.bytes[e];
  char* const d = static_cast<char*>(t.dst[e]);
  const char* const s = static_cast<const char*>(t.src[e]);
  const uint64_t tid = (uint64_t)blockIdx.x * CP_THREADS + threadIdx.x, stride = (uint64_t)gridDim.x * CP_THREADS;
  if (!s) {
    uint64_t* const w = reinterpret_cast<uint64_t*>(d);  // fills are of whole, aligned doubles
    for (uint64_t k = tid; k < bytes / 8; k += stride) w[k] = t.fill[e];
    return;
  }
  // the widest word both addresses are aligned to
  const uint64_t al = (uint64_t)d | (uint64_t)s;
  uint64_t done = 0;
  if ((al & 15u) == 0) {
    copy_words(reinterpret_cast<uint4*>(d), reinterpret_cast<const uint4*>(s), bytes / 16, tid, stride);
    done = bytes / 16 * 16;
  } else if ((al & 7u) == 0) {
    copy_words(reinterpret_cast<uint2*>(d), reinterpret_cast<const uint2*>(s), bytes / 8, tid, stride);
    done = bytes / 8 * 8;
  } else if ((al & 3u) == 0) {
    copy_words(reinterpret_cast<uint32_t*>(d), reinterpret_cast<const uint32_t*>(s), bytes / 4, tid, stride);
    done = bytes / 4 * 4;
  }
  copy_words(d + done, s + done, bytes - done, tid, stride);
}

// the largest positive radius: positive doubles order like their bits; zero, negative
// and NaN radii do not count
__global__ void k_radius_max(const double* __restrict__ r, uint64_t n, unsigned long long* out) {
  unsigned long long m = 0;
  for (uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; k < n; k += (uint64_t)gridDim.x * blockDim.x) {
    const long long u = __double_as_longlong(r[k]);
    if (u > 0 && u <= 0x7ff0000000000000ll && (unsigned long long)u > m) m = (unsigned long long)u;
  }
  for (int o = 16; o; o >>= 1) {
    const unsigned long long q = __shfl_xor_sync(0xffffffffu, m, o);
    m = q > m ? q : m;
  }
  if ((threadIdx.x & 31) == 0 && m) atomicMax(out, m);
}
}  // namespace

int launch_copies(dem_ctx* c, const CopyTab& t) {
  if (!t.n) return DEM_OK;
  uint64_t most = 0;
  for (int e = 0; e < t.n; e++) most = std::max(most, t.bytes[e]);
  const uint64_t want = most / (CP_THREADS * 64) + 1, cap = std::max(1, c->num_sms * 16 / t.n);
  k_copies<<<dim3((unsigned)std::min(want, cap), (unsigned)t.n), CP_THREADS, 0, c->stream>>>(t);
  DEM_CUDA_TRY(c, cudaGetLastError());
  return DEM_OK;
}

int launch_radius_max(dem_ctx* c, const double* radius, uint64_t n, double* out) {
  *out = 0.0;
  if (!n) return DEM_OK;
  unsigned long long* const slot = c->d_scalars + SC_RADMAX;
  DEM_CUDA_TRY(c, cudaMemsetAsync(slot, 0, sizeof(*slot), c->stream));
  k_radius_max<<<std::min<unsigned>(grid_for(n, 256), (unsigned)c->num_sms * 4u), 256, 0, c->stream>>>(radius, n, slot);
  DEM_CUDA_TRY(c, cudaGetLastError());
  DEM_CUDA_TRY(c, cudaMemcpyAsync(c->h_scalars, slot, sizeof(*slot), cudaMemcpyDeviceToHost, c->stream));
  DEM_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  static_assert(sizeof(double) == sizeof(unsigned long long), "bits");
  __builtin_memcpy(out, c->h_scalars, sizeof(double));
  return DEM_OK;
}

// A copy of more bytes than the allocation holds is an error of cudaMemcpyAsync, which
// looks the range up; a kernel would run past it.  So only what is known to lie inside
// one allocation of the device goes through k_copies.
bool device_memory(int device, const void* p, uint64_t bytes) {
  cudaPointerAttributes at;
  if (cudaPointerGetAttributes(&at, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  if (at.type != cudaMemoryTypeDevice || at.device != device) return false;
  using Range = CUresult(CUDAAPI*)(CUdeviceptr*, size_t*, CUdeviceptr);
  static const Range range = [] {
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult found;
    if (cudaGetDriverEntryPointByVersion("cuMemGetAddressRange", &fn, 12000, cudaEnableDefault, &found) != cudaSuccess ||
        found != cudaDriverEntryPointSuccess) {
      cudaGetLastError();
      fn = nullptr;
    }
    return reinterpret_cast<Range>(fn);
  }();
  CUdeviceptr base = 0;
  size_t size = 0;
  const CUdeviceptr first = reinterpret_cast<CUdeviceptr>(p);
  if (!range || range(&base, &size, first) != CUDA_SUCCESS) return false;
  return first >= base && bytes <= size && first - base <= size - bytes;
}
}  // namespace dem

extern "C" int dem_selftest_copy_range(const void* p, uint64_t bytes, int* inside) {
  if (!p || !inside) return DEM_ERR_INVALID_ARG;
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess) return DEM_ERR_CUDA;
  *inside = dem::device_memory(device, p, bytes) ? 1 : 0;
  return DEM_OK;
}
