// A CUDA runtime without a GPU, for tests of the solver's host code: linked
// with the library's own objects in place of libcudart. Device memory is host
// memory with a limit (fake_limit), kernels are not run but counted by name
// (fake_launches), and a copy or clear that is not inside live allocations is
// an error. Small copies (the kernels' error word) and clears are done, the
// rest are not.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

namespace {
std::map<char *, size_t> g_live;
size_t g_limit = (size_t)1 << 40, g_used = 0;
long g_mapped = 0; // allocations of 1 MB and more: each maps device memory of its own
std::map<const void *, std::string> g_names;
std::map<std::string, long> g_count;
cudaError_t g_last = cudaSuccess;
struct {
  dim3 grid, block;
  size_t shared;
  void *stream;
} g_call;

cudaError_t note(cudaError_t e)
{
  if (e != cudaSuccess)
    g_last = e;
  return e;
}

bool inside(const void *p, size_t bytes)
{
  auto it = g_live.upper_bound((char *)p);
  if (it == g_live.begin())
    return false;
  --it;
  return (char *)p + bytes <= it->first + it->second;
}

cudaError_t move(void *dst, const void *src, size_t n, cudaMemcpyKind kind)
{
  if ((kind != cudaMemcpyDeviceToHost && !inside(dst, n)) ||
      (kind != cudaMemcpyHostToDevice && !inside(src, n)) || !dst || !src)
    return note(cudaErrorInvalidValue);
  if (n <= 64)
    std::memcpy(dst, src, n);
  return cudaSuccess;
}

cudaError_t clear(void *p, int v, size_t n)
{
  if (!inside(p, n))
    return note(cudaErrorInvalidValue);
  if (n <= 64)
    std::memset(p, v, n);
  return cudaSuccess;
}
} // namespace

extern "C" {
void fake_limit(size_t bytes) { g_limit = bytes; }
size_t fake_used(void) { return g_used; }
long fake_mapped(void) { return g_mapped; }
// launches since the last reset of kernels whose mangled name contains `part`
long fake_launches(const char *part, int reset)
{
  long n = 0;
  for (auto &k : g_count)
    if (k.first.find(part) != std::string::npos)
      n += k.second;
  if (reset)
    g_count.clear();
  return n;
}
// sets the word of every live allocation of 4 bytes (a solver's error word)
void fake_raise(unsigned v)
{
  for (auto &a : g_live)
    if (a.second == sizeof(v))
      std::memcpy(a.first, &v, sizeof(v));
}

void **__cudaRegisterFatBinary(void *f) { return (void **)f; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *,
    uint3 *, dim3 *, dim3 *, int *)
{
  g_names[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t shared, void *stream)
{
  g_call = { grid, block, shared, stream };
  return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *shared, void *stream)
{
  *grid = g_call.grid;
  *block = g_call.block;
  *shared = g_call.shared;
  *(void **)stream = g_call.stream;
  return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 grid, dim3, void **, size_t, cudaStream_t)
{
  if (!grid.x || grid.y > 65535 || grid.z > 65535)
    return note(cudaErrorInvalidConfiguration);
  ++g_count[g_names[f]];
  return cudaSuccess;
}

cudaError_t cudaMalloc(void **p, size_t n)
{
  *p = nullptr;
  if (n > g_limit || g_used > g_limit - n)
    return note(cudaErrorMemoryAllocation);
  *p = std::calloc(1, n ? n : 1);
  g_live[(char *)*p] = n;
  g_used += n;
  g_mapped += n >= (size_t)1 << 20;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p)
{
  if (!p)
    return cudaSuccess;
  auto it = g_live.find((char *)p);
  if (it == g_live.end())
    return note(cudaErrorInvalidValue);
  g_used -= it->second;
  g_live.erase(it);
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t *free_bytes, size_t *total)
{
  *total = g_limit;
  *free_bytes = g_limit > g_used ? g_limit - g_used : 0;
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k)
{
  return move(d, s, n, k);
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind k, cudaStream_t)
{
  return move(d, s, n, k);
}
cudaError_t cudaMemset(void *p, int v, size_t n) { return clear(p, v, n); }
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { return clear(p, v, n); }

cudaError_t cudaGetLastError(void)
{
  const cudaError_t e = g_last;
  g_last = cudaSuccess;
  return e;
}
const char *cudaGetErrorString(cudaError_t e)
{
  return e == cudaErrorMemoryAllocation ? "out of memory" : "an error of the fake runtime";
}
cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int)
{
  *v = a == cudaDevAttrMultiProcessorCount ? 148
      : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448 : 10;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int *a, int *b) { return *a = *b = 0, cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *) { return *p = nullptr, cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *)
{
  a->type = cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaHostRegister(void *, size_t, unsigned) { return cudaSuccess; }
cudaError_t cudaHostUnregister(void *) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned)
{
  return *s = (cudaStream_t)1, cudaSuccess;
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int)
{
  return *s = (cudaStream_t)1, cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return *e = (cudaEvent_t)1, cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned)
{
  return *e = (cudaEvent_t)1, cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *t, cudaEvent_t, cudaEvent_t) { return *t = 0, cudaSuccess; }
}
