// noalloc.cu -- level time step of a device-resident level state, computed
// without allocating any memory.
//
// Some callers cannot call cudaMalloc at all: a solver embedded in another
// code's memory pool (every byte on the device owned by that pool), a process
// that must not allocate after start-up, or a stream in the middle of work that
// an allocation would serialise.  emma_hydro_level_dt_noalloc serves them: the
// caller passes the level state already on the device and receives dt; the
// reduction's scratch is a fixed array inside this library.
//
// Scratch: g_dt_scratch, a file-scope __device__ array of kMaxBlocks + 2 64-bit slots
// (128 KiB + 16 B) that every GPU which loads the library holds until the process exits.
// Slot b < kMaxBlocks receives the maximum signal speed of block b, slot kMaxBlocks the
// maximum over the blocks; every one of these that a call reads is written earlier in the
// same call.  The last slot counts a call's finished blocks, above the call's own
// number: calls are numbered from 1, a block first raises the slot to its call's number
// with no block counted, so it counts from zero whatever any call before it left there, one
// that never ran, failed or overlapped another.  Calls whose kernels overlap on the GPU
// (different streams, or several host threads) share the array and race: serialise them
// on one stream.
//
// Host code only ever uses the array's device address, obtained once per device
// with cudaGetSymbolAddress on the first call made while that device is
// current; that first call must therefore not be made during a stream capture.
// The address is cached for the life of the device's primary context: after a
// cudaDeviceReset (which unloads this library's module) call
// emma_hydro_noalloc_forget() before the next call, so that the address is
// looked up again in the new context.  The per-device cache slots are atomic, so
// host threads may make first calls concurrently.
//
// Built with -fmad=false: the signal speed rounds exactly as the reference's
// L_comptstep_hydro (src/advanceamr.c:122-135) and emma_hydro_comptstep do.
#include <cuda_runtime.h>
#include <atomic>
#include <cmath>
#include <cstdio>
#include <cstring>
#include "emma_hydro.h"

namespace {

constexpr int kThreads = 256;
constexpr int kMaxBlocks = 16384;
constexpr int kCountBits = 20;  // of the counting slot; the call's number above them
constexpr long long kMaxCells = 2048LL * kMaxBlocks;  // 33,554,432 cells (a 256^3 level is 16,777,216)
constexpr int kMaxDevices = 64;
static_assert(kMaxBlocks < (1 << kCountBits), "the blocks of a call in the counting slot's low bits");

static __device__ __align__(256) unsigned long long g_dt_scratch[kMaxBlocks + 2];

std::atomic<unsigned long long *> g_scratch_addr[kMaxDevices];  // zero-initialised (static storage)
std::atomic<unsigned long long> g_calls[kMaxDevices];
std::atomic<int> g_sms[kMaxDevices];

__device__ __forceinline__ double block_max(double m) {
  __shared__ double part[kThreads / 32];
  for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = m;
  __syncthreads();
  m = (threadIdx.x < kThreads / 32) ? part[threadIdx.x] : 0.;
  if (threadIdx.x < 32)
    for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  return m;
}

// max over the cells of |v| + sqrt(gamma p / rho) -> scratch[kMaxBlocks]; W = 5 planes of
// n8 cells.  One launch: each block leaves its maximum, the last to finish takes the
// maximum over them.  A second launch for that cost as much as the whole reduction of a
// small level (32^3: 30.6 us a call with two launches, 19.9 with one, most of it the
// read-back).  Small levels take one cell a thread (latency; 128^3 32.9 -> 29.8 us), large
// ones eight at a time (256^3 130 -> 127 us, 5.3 TB/s with the call's fixed cost).
__global__ void __launch_bounds__(kThreads) dt_kernel(const double *__restrict__ W, long long n8, int per_thread,
                                                      unsigned long long call, unsigned long long *scratch) {
  unsigned long long *count = scratch + kMaxBlocks + 1;
  if (threadIdx.x == 0) atomicMax(count, call << kCountBits);  // here, beside the loads
  double m = 0.;
  const long long base = (long long)blockIdx.x * kThreads * per_thread + threadIdx.x;
  auto cell = [&](long long i) {
    const double d = W[i], u = W[n8 + i], v = W[2 * n8 + i], w = W[3 * n8 + i], p = W[4 * n8 + i];
    const double va = sqrt(u * u + v * v + w * w);
    const double aa = sqrt((5. / 3.) * p / d);
    m = fmax(m, va + aa);  // fmax drops NaN like the reference's FMAX
  };
  if (per_thread % 8 == 0 && base - threadIdx.x + (long long)per_thread * kThreads <= n8) {
    for (int j = 0; j < per_thread; j += 8)
#pragma unroll
      for (int i = 0; i < 8; i++) cell(base + (long long)(j + i) * kThreads);
  } else {
    for (int j = 0; j < per_thread; j++)
      if (base + (long long)j * kThreads < n8) cell(base + (long long)j * kThreads);
  }
  m = block_max(m);
  __shared__ bool last;
  if (threadIdx.x == 0) {
    scratch[blockIdx.x] = (unsigned long long)__double_as_longlong(m);
    __threadfence();
    last = atomicAdd(count, 1ULL) == (call << kCountBits) + gridDim.x - 1;
  }
  __syncthreads();  // also: block_max's shared memory is free again
  if (!last) return;
  __threadfence();
  m = 0.;
  for (int b = threadIdx.x; b < gridDim.x; b += kThreads) m = fmax(m, __longlong_as_double((long long)__ldcg(scratch + b)));
  m = block_max(m);
  if (threadIdx.x == 0) scratch[kMaxBlocks] = (unsigned long long)__double_as_longlong(m);
}

}  // namespace

extern "C" int emma_hydro_level_dt_noalloc(const double *d_state, long long ncells, int level, double cfl,
                                           void *stream, double *dt_out) {
  if (d_state == nullptr || dt_out == nullptr || ncells < 0 || level < 1 || level > 40) {
    std::fputs("emma_hydro_level_dt_noalloc: null pointer, negative size or level out of range\n", stderr);
    return EMMA_ST_ARG;
  }
  if (ncells > kMaxCells) {
    std::fputs("emma_hydro_level_dt_noalloc: more than 33554432 cells, beyond the fixed scratch of this entry\n",
               stderr);
    return EMMA_ST_ARG;
  }
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return EMMA_ST_CUDA;
  unsigned long long *scratch = g_scratch_addr[dev].load(std::memory_order_acquire);
  if (scratch == nullptr) {
    void *p = nullptr;
    if (cudaGetSymbolAddress(&p, g_dt_scratch) != cudaSuccess || p == nullptr) return EMMA_ST_CUDA;
    scratch = static_cast<unsigned long long *>(p);
    int sms = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return EMMA_ST_CUDA;
    g_sms[dev].store(sms, std::memory_order_relaxed);
    g_scratch_addr[dev].store(scratch, std::memory_order_release);
  }
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  double smax = 0.;
  if (ncells > 0) {
    // enough cells a thread to keep to 8 blocks an SM, a power of two up to 8; beyond 4096
    // blocks 16, or the counting of the blocks shows
    const long long resident = 8LL * kThreads * g_sms[dev].load(std::memory_order_relaxed);
    int per = 1;
    while (per < 8 && ncells > resident * per) per *= 2;
    if (ncells > (long long)kThreads * per * 4096) per = 16;
    const int nblocks = (int)((ncells + (long long)kThreads * per - 1) / ((long long)kThreads * per));
    dt_kernel<<<nblocks, kThreads, 0, s>>>(d_state, ncells, per, g_calls[dev].fetch_add(1u) + 1u, scratch);
    if (cudaGetLastError() != cudaSuccess) return EMMA_ST_CUDA;
    unsigned long long bits = 0;
    if (cudaMemcpyAsync(&bits, scratch + kMaxBlocks, sizeof(bits), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess) {
      cudaGetLastError();  // a call refused here (a stream under capture) is not the next call's error
      return EMMA_ST_CUDA;
    }
    std::memcpy(&smax, &bits, sizeof(smax));
  }
  // L_comptstep_hydro's final step (src/advanceamr.c:135)
  double dt = 1e9;
  const double dxcur = std::pow(0.5, level);
  if (smax > 0.) dt = std::fmin(dxcur * cfl / (smax * 3.), dt);
  *dt_out = dt;
  return 0;
}

extern "C" void emma_hydro_noalloc_forget(void) {
  for (int d = 0; d < kMaxDevices; d++) g_scratch_addr[d].store(nullptr, std::memory_order_release);
}
