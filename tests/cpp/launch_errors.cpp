// Stands in for the CUDA driver library of one test process: every call goes to
// the real one (path in REAL_LIBCUDA), except that kernel launches return an error
// of their own, without reaching it, while fail_launches(1) is in force.
#include <dlfcn.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>

namespace {
int failing = 0;
using Launch = int (*)(void*, void*, void*, void*);
using LaunchLong = int (*)(void*, unsigned, unsigned, unsigned, unsigned, unsigned, unsigned, unsigned, void*, void**, void**);
Launch real_ex = nullptr, real_ex_ptsz = nullptr;
LaunchLong real_long = nullptr, real_long_ptsz = nullptr;
constexpr int kLaunchOutOfResources = 701;

int launch_ex(void* a, void* b, void* c, void* d) { return failing ? kLaunchOutOfResources : real_ex(a, b, c, d); }
int launch_ex_ptsz(void* a, void* b, void* c, void* d) { return failing ? kLaunchOutOfResources : real_ex_ptsz(a, b, c, d); }
int launch_long(void* f, unsigned a, unsigned b, unsigned c, unsigned d, unsigned e, unsigned g, unsigned h, void* s,
                void** p, void** q) {
  return failing ? kLaunchOutOfResources : real_long(f, a, b, c, d, e, g, h, s, p, q);
}
int launch_long_ptsz(void* f, unsigned a, unsigned b, unsigned c, unsigned d, unsigned e, unsigned g, unsigned h, void* s,
                     void** p, void** q) {
  return failing ? kLaunchOutOfResources : real_long_ptsz(f, a, b, c, d, e, g, h, s, p, q);
}

void* driver() {
  static void* lib = dlopen(std::getenv("REAL_LIBCUDA"), RTLD_NOW | RTLD_LOCAL);
  return lib;
}
template <class F> F real(const char* name) { return reinterpret_cast<F>(dlsym(driver(), name)); }

// The per-thread default stream's variants are other functions under the same name.
constexpr uint64_t kPerThread = 2;
void stand_in(const char* name, uint64_t flags, void** fn) {
  const bool ptsz = flags & kPerThread;
  if (!fn || !*fn) return;
  if (!std::strcmp(name, "cuLaunchKernelEx")) {
    (ptsz ? real_ex_ptsz : real_ex) = reinterpret_cast<Launch>(*fn);
    *fn = reinterpret_cast<void*>(ptsz ? launch_ex_ptsz : launch_ex);
  } else if (!std::strcmp(name, "cuLaunchKernel")) {
    (ptsz ? real_long_ptsz : real_long) = reinterpret_cast<LaunchLong>(*fn);
    *fn = reinterpret_cast<void*>(ptsz ? launch_long_ptsz : launch_long);
  }
}
}  // namespace

extern "C" {
void fail_launches(int on) { failing = on; }

int cuGetProcAddress_v2(const char* name, void** fn, int version, uint64_t flags, void* status);
int cuGetProcAddress(const char* name, void** fn, int version, uint64_t flags) {
  const int r = real<int (*)(const char*, void**, int, uint64_t)>("cuGetProcAddress")(name, fn, version, flags);
  if (!std::strcmp(name, "cuGetProcAddress") && fn && *fn)
    *fn = version >= 12000 ? reinterpret_cast<void*>(cuGetProcAddress_v2) : reinterpret_cast<void*>(cuGetProcAddress);
  else stand_in(name, flags, fn);
  return r;
}
int cuGetProcAddress_v2(const char* name, void** fn, int version, uint64_t flags, void* status) {
  const int r = real<int (*)(const char*, void**, int, uint64_t, void*)>("cuGetProcAddress_v2")(name, fn, version, flags, status);
  if (!std::strcmp(name, "cuGetProcAddress") && fn && *fn)
    *fn = version >= 12000 ? reinterpret_cast<void*>(cuGetProcAddress_v2) : reinterpret_cast<void*>(cuGetProcAddress);
  else stand_in(name, flags, fn);
  return r;
}
int cuDriverGetVersion(int* v) { return real<int (*)(int*)>("cuDriverGetVersion")(v); }
int cuInit(unsigned f) { return real<int (*)(unsigned)>("cuInit")(f); }
int cuDeviceGet(int* d, int i) { return real<int (*)(int*, int)>("cuDeviceGet")(d, i); }
int cuGetExportTable(const void** t, const void* id) {
  return real<int (*)(const void**, const void*)>("cuGetExportTable")(t, id);
}
}
