// Host-side odds and ends of the native library: last-error string, version, device query.
#include <cuda_runtime.h>
#include <stdarg.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>
#include <memory>
#include <mutex>
#include <new>
#include <vector>
#include "psgd_common.cuh"

static thread_local char g_last_error[1024] = "";

void psgd_set_error(const char* fmt, ...) {
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(g_last_error, sizeof(g_last_error), fmt, ap);
  va_end(ap);
}

PSGD_API const char* psgd_last_error() { return g_last_error; }

PSGD_API int psgd_version() { return 100; }

// Fills sm_count / major / minor of the CURRENT device. Returns a CUDA error code.
PSGD_API int psgd_device_info(int* sm_count, int* cc_major, int* cc_minor, int* max_smem_optin) {
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) { psgd_set_error("cudaGetDevice: %s", cudaGetErrorString(e)); return (int)e; }
  cudaDeviceProp prop;
  e = cudaGetDeviceProperties(&prop, dev);
  if (e != cudaSuccess) { psgd_set_error("cudaGetDeviceProperties: %s", cudaGetErrorString(e)); return (int)e; }
  *sm_count = prop.multiProcessorCount;
  *cc_major = prop.major;
  *cc_minor = prop.minor;
  *max_smem_optin = (int)prop.sharedMemPerBlockOptin;
  return 0;
}

// Which recording (CUDA-graph capture) `stream` is part of: an id of its own for every capture of the
// process, 0 when the stream is not being recorded. Returns a CUDA error code.
PSGD_API int psgd_capture_id(cudaStream_t stream, unsigned long long* id) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  *id = 0;
  const cudaError_t e = cudaStreamGetCaptureInfo_v2(stream, &status, id, nullptr, nullptr, nullptr);
  if (e != cudaSuccess) { psgd_set_error("cudaStreamGetCaptureInfo: %s", cudaGetErrorString(e)); return (int)e; }
  if (status == cudaStreamCaptureStatusNone) *id = 0;
  return 0;
}

// Exchanges the calling thread's capture mode (see cudaThreadExchangeStreamCaptureMode): *mode goes in, the
// previous one comes out. In the relaxed mode (2) a thread that is recording one stream may allocate
// memory and wait for others. Returns a CUDA error code.
PSGD_API int psgd_capture_mode(int* mode) {
  cudaStreamCaptureMode m = (cudaStreamCaptureMode)*mode;
  const cudaError_t e = cudaThreadExchangeStreamCaptureMode(&m);
  if (e != cudaSuccess) { psgd_set_error("cudaThreadExchangeStreamCaptureMode: %s", cudaGetErrorString(e)); return (int)e; }
  *mode = (int)m;
  return 0;
}

// Returns once everything put on `stream` so far is done. Returns a CUDA error code.
PSGD_API int psgd_stream_wait(cudaStream_t stream) {
  const cudaError_t e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) { psgd_set_error("cudaStreamSynchronize: %s", cudaGetErrorString(e)); return (int)e; }
  return 0;
}

// ---- launches written down and made again ---------------------------------------------------------
// An eager step repeats the launches of the step before it with the same arguments. Each through its own entry point and a foreign
// function call with some fifteen converted arguments took 4.3 us of the host; one call that makes them all takes half.
struct PsgdTape {
  struct Launch {
    const void* kernel;
    int grid, block, early, cluster;
    size_t smem;
    std::vector<std::unique_ptr<max_align_t[]>> held;   // copies of the arguments
    std::vector<void*> args;
  };
  std::vector<Launch> launches;
  bool complete = true;
};
thread_local PsgdTape* psgd_tape_now = nullptr;

void psgd_tape_add(const void* kernel, int grid, int block, size_t smem, int early, int cluster, int count, const void* const* args,
                   const size_t* sizes) {
  PsgdTape& tape = *psgd_tape_now;
  try {
    PsgdTape::Launch l = {kernel, grid, block, early, cluster, smem, {}, {}};
    for (int i = 0; i < count; ++i) {
      l.held.emplace_back(new max_align_t[sizes[i] / sizeof(max_align_t) + 1]);
      memcpy(l.held.back().get(), args[i], sizes[i]);
      l.args.push_back(l.held.back().get());
    }
    tape.launches.push_back(std::move(l));
  } catch (const std::bad_alloc&) {   // the launch itself has been made: the callers of the library get no exception from it
    tape.complete = false;
  }
}

// Writes down the launches that this thread makes through psgd_launch from here to psgd_tape_end, which returns their number; -1
// if there was no memory for all of them. Null if there is none at all.
PSGD_API void* psgd_tape_begin() { return psgd_tape_now = new (std::nothrow) PsgdTape; }
PSGD_API int psgd_tape_end() {
  const PsgdTape* tape = psgd_tape_now;
  psgd_tape_now = nullptr;
  return tape && tape->complete ? (int)tape->launches.size() : -1;
}
PSGD_API void psgd_tape_free(void* tape) {
  if (tape == psgd_tape_now) psgd_tape_now = nullptr;   // (dropped while it is being written)
  delete (PsgdTape*)tape;
}
// Makes them again, on `stream`. Returns a CUDA error code.
PSGD_API int psgd_tape_replay(const void* tape, cudaStream_t stream) {
  for (const PsgdTape::Launch& l : ((const PsgdTape*)tape)->launches) {
    cudaLaunchConfig_t cfg;
    cudaLaunchAttribute attrs[2];
    psgd_launch_config(cfg, attrs, l.grid, l.block, l.smem, stream, l.early, l.cluster);
    PSGD_CUDA_OK(cudaLaunchKernelExC(&cfg, l.kernel, const_cast<void**>(l.args.data())));
  }
  return 0;
}

// ---- what lives as long as a recorded graph --------------------------------------------------
// The caller numbers what a graph refers to and asks from time to time which numbers are free again. The
// destructor of a user object may run on a thread of the driver and may call nothing of CUDA, so it only
// notes the number. The list is never destroyed: graphs may go after the static objects of the process.
struct Finished {
  std::mutex lock;
  std::vector<long long> numbers;
};
static Finished& finished() {
  static Finished* f = new Finished;
  return *f;
}
static void CUDART_CB note_finished(void* number) {
  Finished& f = finished();
  std::lock_guard<std::mutex> hold(f.lock);
  f.numbers.push_back((long long)(intptr_t)number);
}

// Notes `number` as finished once the graph that `stream` is being recorded into, and every executable
// instance of it, are destroyed. Returns a CUDA error code (-1: the stream is not being recorded).
PSGD_API int psgd_graph_retain(long long number, cudaStream_t stream) {
  cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
  cudaGraph_t graph = nullptr;
  cudaError_t e = cudaStreamGetCaptureInfo_v2(stream, &status, nullptr, &graph, nullptr, nullptr);
  if (e == cudaSuccess && (status != cudaStreamCaptureStatusActive || graph == nullptr)) {
    psgd_set_error("psgd_graph_retain: the stream is not being recorded");
    return -1;
  }
  cudaUserObject_t object = nullptr;
  if (e == cudaSuccess) e = cudaUserObjectCreate(&object, (void*)(intptr_t)number, note_finished, 1, cudaUserObjectNoDestructorSync);
  if (e == cudaSuccess) {
    e = cudaGraphRetainUserObject(graph, object, 1, cudaGraphUserObjectMove);
    if (e != cudaSuccess) cudaUserObjectRelease(object, 1);
  }
  if (e != cudaSuccess) { psgd_set_error("psgd_graph_retain: %s", cudaGetErrorString(e)); return (int)e; }
  return 0;
}

// Up to `most` finished numbers, each handed out once; returns how many.
PSGD_API int psgd_graph_released(long long* numbers, int most) {
  Finished& f = finished();
  std::lock_guard<std::mutex> hold(f.lock);
  int n = 0;
  while (n < most && !f.numbers.empty()) {
    numbers[n++] = f.numbers.back();
    f.numbers.pop_back();
  }
  return n;
}

#ifdef PSGD_BOUNDS_CHECK
extern "C" int psgd_bounds_read_products(int* out, int reset);
extern "C" int psgd_bounds_read_finalize(int* out, int reset);
extern "C" int psgd_bounds_read_orth(int* out, int reset);
extern "C" int psgd_bounds_read_panel(int* out, int reset);
// Debug build only. out[0..23]: the status blocks of the product, decompression / flat and
// orthonormalisation translation units (8 ints each: violations, kernel id of the first, what,
// value lo / hi, limit lo / hi, unused); the panel kernel's stands in the second place when that
// is empty. Returns the total number of violations, or -1 on error.
PSGD_API int psgd_bounds_status(int* out, int reset) {
  int panel[8];
  if (psgd_bounds_read_products(out, reset) != 0 || psgd_bounds_read_finalize(out + 8, reset) != 0 ||
      psgd_bounds_read_orth(out + 16, reset) != 0 || psgd_bounds_read_panel(panel, reset) != 0) {
    psgd_set_error("psgd_bounds_status: reading a status block failed");
    return -1;
  }
  const int total = out[0] + out[8] + out[16] + panel[0];
  if (out[8] == 0) memcpy(out + 8, panel, sizeof(panel));
  return total;
}
#endif
