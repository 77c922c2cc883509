// Per-device context: error word, scratch buffers, status helpers.
#include <atomic>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

#include "lepic_internal.cuh"

namespace lepic {

namespace {
std::mutex g_mu;
std::map<int, Ctx> g_ctx;
struct Buf {
  void *p = nullptr;
  size_t bytes = 0;
};
std::map<std::pair<int, std::string>, Buf> g_scratch;
thread_local int g_last_cuda_error = 0;
constexpr unsigned BARRIERS = 64, BARRIER_WORDS = 32;   // a 128-byte line each
std::atomic<unsigned> g_barrier{0};
}  // namespace

int cuda_status(cudaError_t e, const char *what) {
  g_last_cuda_error = (int)e;
  fprintf(stderr, "lepic_gpu: CUDA error %d (%s) in %s\n", (int)e, cudaGetErrorString(e), what);
  return LEPIC_ERR_CUDA;
}

Ctx &ctx() {
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(g_mu);
  Ctx &c = g_ctx[dev];
  if (c.device < 0) {
    c.device = dev;
    cudaGetDeviceProperties(&c.prop, dev);
    c.sms = c.prop.multiProcessorCount;
    cudaMalloc(&c.d_err, 2 * sizeof(int));
    cudaMemset(c.d_err, 0, 2 * sizeof(int));
    cudaMallocHost(&c.h_err, 2 * sizeof(int));
    c.h_err[0] = c.h_err[1] = 0;
    if (cudaMalloc(&c.d_barrier, BARRIERS * BARRIER_WORDS * sizeof(unsigned)) == cudaSuccess)
      cudaMemset(c.d_barrier, 0, BARRIERS * BARRIER_WORDS * sizeof(unsigned));
    else
      c.d_barrier = nullptr;
    cudaStreamSynchronize(nullptr);   // a first launch on any stream finds them cleared
  }
  return c;
}

GridBarrier grid_barrier(unsigned rounds) {
  Ctx &c = ctx();
  return {c.d_barrier ? c.d_barrier + (g_barrier++ % BARRIERS) * BARRIER_WORDS : nullptr, rounds};
}

void *scratch(const char *name, size_t bytes) {
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(g_mu);
  Buf &b = g_scratch[{dev, std::string(name)}];
  if (b.bytes < bytes) {
    if (b.p) cudaFree(b.p);
    b.p = nullptr;
    b.bytes = 0;
    size_t want = bytes + bytes / 8 + 256;
    if (cudaMalloc(&b.p, want) != cudaSuccess) {
      b.p = nullptr;
      return nullptr;
    }
    b.bytes = want;
  }
  return b.p;
}

void scratch_drop(const char *prefix) {
  int dev = 0;
  cudaGetDevice(&dev);
  std::lock_guard<std::mutex> lk(g_mu);
  for (auto &kv : g_scratch) {
    if (kv.first.first != dev || kv.first.second.compare(0, strlen(prefix), prefix) != 0) continue;
    if (kv.second.p) cudaFree(kv.second.p);   // (waits for the kernels that use it)
    kv.second = Buf{};
  }
}

namespace {
struct ResultBlock {
  double *p = nullptr;
  bool tried = false;
  ~ResultBlock() {
    if (p) cudaFreeHost(p);
  }
};
}  // namespace

double *result_block() {
  static thread_local ResultBlock b;
  if (!b.tried) {
    b.tried = true;
    if (cudaHostAlloc((void **)&b.p, RESULT_WORDS * sizeof(double), cudaHostAllocPortable | cudaHostAllocMapped) !=
        cudaSuccess) {
      b.p = nullptr;
      cudaGetLastError();
    }
  }
  return b.p;
}

// Synchronise the stream, read and clear the device error word.
int check_err(cudaStream_t s) {
  Ctx &c = ctx();
  cudaError_t e = cudaMemcpyAsync(c.h_err, c.d_err, 2 * sizeof(int), cudaMemcpyDeviceToHost, s);
  if (e != cudaSuccess) return cuda_status(e, "read error word");
  e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return cuda_status(e, "stream synchronize");
  int code = c.h_err[0];
  if (code) {
    fprintf(stderr, "lepic_gpu: device status %d (detail %d)\n", code, c.h_err[1]);
    cudaMemsetAsync(c.d_err, 0, 2 * sizeof(int), s);
    cudaStreamSynchronize(s);
  }
  return code;
}

}  // namespace lepic
