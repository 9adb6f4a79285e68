// A device of limited memory for the tests: preloaded, it counts what the
// process holds from cudaMalloc and refuses (as a full device does) what would
// take it past a limit.
#include <dlfcn.h>

#include <cstddef>
#include <mutex>
#include <unordered_map>

namespace {
std::mutex g_mutex;
std::unordered_map<void *, size_t> g_held;
size_t g_live = 0, g_limit = (size_t)-1;
long g_refused = 0, g_refuse_in = 0;
// (the runtime is loaded later, and not into the global scope)
template <typename F>
F next(const char *name) {
  return reinterpret_cast<F>(dlsym(dlopen("libcudart.so.13", RTLD_LAZY), name));
}
}  // namespace

extern "C" int cudaMalloc(void **p, size_t bytes) {
  static const auto real = next<int (*)(void **, size_t)>("cudaMalloc");
  std::lock_guard<std::mutex> lock(g_mutex);
  const bool turn = g_refuse_in > 0 && --g_refuse_in == 0;
  if (turn || bytes > g_limit || g_live > g_limit - bytes) {
    ++g_refused;
    *p = nullptr;
    return 2;  // cudaErrorMemoryAllocation
  }
  const int e = real(p, bytes);
  if (e == 0) {
    g_held[*p] = bytes;
    g_live += bytes;
  }
  return e;
}

extern "C" int cudaFree(void *p) {
  static const auto real = next<int (*)(void *)>("cudaFree");
  std::lock_guard<std::mutex> lock(g_mutex);
  const auto it = g_held.find(p);
  if (it != g_held.end()) {
    g_live -= it->second;
    g_held.erase(it);
  }
  return real(p);
}

extern "C" size_t malloc_limit_live() { return g_live; }
extern "C" long malloc_limit_refused() { return g_refused; }
// refuse the k-th call from here (1: the next) and no other; 0: none
extern "C" void malloc_limit_refuse(long k) { g_refuse_in = k; }
extern "C" void malloc_limit_set(size_t bytes) { g_limit = bytes; }
