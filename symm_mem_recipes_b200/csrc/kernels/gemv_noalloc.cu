// Allocation-free C entry point of the rank-local GEMV (see gemv_noalloc.h).  The global memory that the
// kernel needs besides its operands, the 32-byte Status record its bounded waits
// report into, lives in this array (at offset 64).  The K splits of a tile meet in
// shared memory, so nothing else is kept in global memory between or during calls.
#include <cuda_runtime.h>
#include <stdio.h>

#include <exception>
#include <mutex>

#include "gemv_local.h"
#include "gemv_noalloc.h"

namespace {

static __device__ __align__(256) unsigned char g_gemv_noalloc_scratch[SMR_GEMV_NOALLOC_SCRATCH_BYTES];

constexpr int kMaxDevices = 64;
std::mutex g_noalloc_mu;
unsigned char* g_noalloc_base[kMaxDevices] = {};   // device address of the array, per device
int g_noalloc_sms[kMaxDevices] = {};
constexpr size_t kNoallocStatusOffset = 64;

int noalloc_fail(int code, char* err, int err_len, const char* what, const char* detail = "") {
  if (err != nullptr && err_len > 0) snprintf(err, (size_t)err_len, "smr_gemv_bf16_noalloc: %s%s", what, detail);
  return code;
}

}  // namespace

extern "C" int smr_gemv_bf16_noalloc(const void* x, const void* w, void* out, int batch, int K, int N,
                                     void* stream_ptr, char* err, int err_len) {
  using namespace smr;
  if (batch < 1 || batch > SMR_GEMV_NOALLOC_MAX_BATCH)
    return noalloc_fail(1, err, err_len, "batch must be between 1 and 16");
  if (N < 8 || N > SMR_GEMV_NOALLOC_MAX_N || N % 8 != 0)
    return noalloc_fail(1, err, err_len, "N must be a multiple of 8 and at most 8192 (the limit of this entry point)");
  if (K < 8 || K % 8 != 0) return noalloc_fail(1, err, err_len, "K must be a positive multiple of 8");
  if (x == nullptr || w == nullptr || out == nullptr || ((uintptr_t)x | (uintptr_t)w | (uintptr_t)out) % 16 != 0)
    return noalloc_fail(2, err, err_len, "x, w and out must be non-null and 16-byte aligned");
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);

  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return noalloc_fail(3, err, err_len, "cudaGetDevice: ", cudaGetErrorString(e));
  if (dev < 0 || dev >= kMaxDevices) return noalloc_fail(3, err, err_len, "device ordinal out of range");
  unsigned char* base;
  int sms;
  {
    // Once per device, with that device current: the array's name is only a
    // host-side handle; the kernel needs the address the symbol has on THIS GPU.
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    if (g_noalloc_base[dev] == nullptr) {
      void* p = nullptr;
      e = cudaGetSymbolAddress(&p, g_gemv_noalloc_scratch);
      if (e != cudaSuccess) return noalloc_fail(3, err, err_len, "cudaGetSymbolAddress: ", cudaGetErrorString(e));
      int n = 0;
      e = cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
      if (e != cudaSuccess) return noalloc_fail(3, err, err_len, "cudaDeviceGetAttribute: ", cudaGetErrorString(e));
      g_noalloc_sms[dev] = n;
      g_noalloc_base[dev] = static_cast<unsigned char*>(p);
    }
    base = g_noalloc_base[dev];
    sms = g_noalloc_sms[dev];
  }

  GemvLocalArgs args{};
  args.x = x; args.w = w; args.out = out;
  args.batch = batch; args.K = K; args.N = N;
  args.num_sms = sms;
  args.timeout_ns = 2000000000ull;
  args.status = reinterpret_cast<Status*>(base + kNoallocStatusOffset);
  int rc = 0;
  try {
    rc = launch_gemv_local(args, stream);
  } catch (const std::exception& ex) {
    return noalloc_fail(3, err, err_len, "CUDA driver: ", ex.what());
  }
  if (rc != 0) return noalloc_fail(3, err, err_len, "kernel launch: ", cudaGetErrorString((cudaError_t)rc));
  return 0;
}

extern "C" int smr_gemv_bf16_noalloc_status(void* stream_ptr, unsigned int record[6], char* err, int err_len) {
  using namespace smr;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) return noalloc_fail(3, err, err_len, "cudaGetDevice: ", cudaGetErrorString(e));
  if (dev < 0 || dev >= kMaxDevices) return noalloc_fail(3, err, err_len, "device ordinal out of range");
  unsigned char* base;
  {
    std::lock_guard<std::mutex> lock(g_noalloc_mu);
    base = g_noalloc_base[dev];
  }
  if (record != nullptr)
    for (int i = 0; i < 6; ++i) record[i] = 0u;
  if (base == nullptr) return 0;                 // no call on this device yet: nothing can have failed
  cudaStream_t stream = static_cast<cudaStream_t>(stream_ptr);
  e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) return noalloc_fail(3, err, err_len, "cudaStreamSynchronize: ", cudaGetErrorString(e));
  Status st{};
  e = cudaMemcpy(&st, base + kNoallocStatusOffset, sizeof(Status), cudaMemcpyDeviceToHost);
  if (e != cudaSuccess) return noalloc_fail(3, err, err_len, "cudaMemcpy(status): ", cudaGetErrorString(e));
  if (record != nullptr) {
    record[0] = st.code; record[1] = st.rank; record[2] = st.block;
    record[3] = st.peer; record[4] = st.where; record[5] = st.aux;
  }
  if (st.code == kOk) return 0;
  e = cudaMemsetAsync(base + kNoallocStatusOffset, 0, sizeof(Status), stream);    // reported once
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream);                        // before a call on any other stream
  if (e != cudaSuccess) return noalloc_fail(3, err, err_len, "clear of the status: ", cudaGetErrorString(e));
  return noalloc_fail(4, err, err_len, "a wait inside an earlier call ran out after 2 s (the CTAs of the kernel were "
                                       "not all resident at once?); that call left `out` unwritten");
}
