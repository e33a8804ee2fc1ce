// A stand-in for the CUDA runtime on the host, linked with the library's own
// objects: device memory is host memory, copies and clears are done, kernels
// are noted and not run.  Tests use it to make a call fail at a chosen place
// and to count what is launched, without a GPU.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>
#include <vector>

namespace {
struct Dim3 { unsigned x, y, z; };
struct Config { Dim3 grid, block; size_t smem; void* stream; };
struct LaunchConfig { Dim3 grid, block; size_t smem; void* stream; void* attrs; unsigned n; };

std::map<const void*, std::string> names;  // host stub -> kernel
std::vector<Config> configs;
std::set<void*> live;
std::vector<std::string> launched;
std::vector<std::string>* capture = nullptr;  // the graph being captured
std::map<std::string, std::vector<void*>> pointers;  // kernel -> its last pointer arguments
std::string fail_kernel;
long fail_in = 0, alloc_fail_in = 0, bad_frees = 0;
int last = 0;
std::vector<int> words;  // what the next 4-byte reads return
std::string text;

int set(int e) { if (e) last = e; return e; }

int launch(const void* f, void** args) {
  const std::string& name = names[f];
  if (!fail_kernel.empty() && name.find(fail_kernel) != std::string::npos && --fail_in == 0)
    return set(719);
  (capture ? *capture : launched).push_back(name);
  if (name.find("k_sorted_keys") != std::string::npos) {
    std::vector<void*>& p = pointers["k_sorted_keys"];
    p.assign(9, nullptr);
    for (int k = 0; k < 9; ++k)
      if (k != 4) std::memcpy(&p[k], args[k], sizeof(void*));
  }
  return 0;
}
int copy(void* d, const void* s, size_t n, int kind) {
  if (kind == 2 && n == 4 && !words.empty()) {
    std::memcpy(d, &words.front(), 4);
    words.erase(words.begin());
  } else {
    std::memmove(d, s, n);
  }
  return 0;
}
int alloc(void** p, size_t n) {
  *p = nullptr;
  if (alloc_fail_in && --alloc_fail_in == 0) return set(2);
  *p = std::calloc(n, 1);
  live.insert(*p);
  return 0;
}
int release(void* p) {
  if (!p) return 0;
  if (!live.erase(p)) ++bad_frees;
  else std::free(p);
  return 0;
}
int handle(void** p) { *p = std::malloc(8); return 0; }
}  // namespace

extern "C" {
// ------------------------------------------------------------ for the tests
void fake_reset() {
  launched.clear();
  fail_kernel.clear();
  fail_in = alloc_fail_in = bad_frees = 0;
  last = 0;
  words.clear();
}
void fake_fail_launch(const char* kernel, long nth) { fail_kernel = kernel; fail_in = nth; }
void fake_fail_alloc(long nth) { alloc_fail_in = nth; }
void fake_next_word(int v) { words.push_back(v); }
long fake_launches() { return (long)launched.size(); }
long fake_bad_frees() { return bad_frees; }
void* fake_pointer(const char* kernel, int arg) { return pointers[kernel].at(arg); }
const char* fake_names() {
  text.clear();
  for (const std::string& n : launched) text += n + "\n";
  return text.c_str();
}

// ------------------------------------------------------------- the runtime
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*,
                            void*, void*, int*) {
  names[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(Dim3 g, Dim3 b, size_t smem, void* stream) {
  configs.push_back({g, b, smem, stream});
  return 0;
}
int __cudaPopCallConfiguration(Dim3* g, Dim3* b, size_t* smem, void* stream) {
  const Config c = configs.back();
  configs.pop_back();
  *g = c.grid;
  *b = c.block;
  *smem = c.smem;
  *(void**)stream = c.stream;
  return 0;
}
int cudaLaunchKernel(const void* f, Dim3, Dim3, void** args, size_t, void*) {
  return launch(f, args);
}
int cudaLaunchKernelExC(const LaunchConfig*, const void* f, void** args) { return launch(f, args); }
int cudaMalloc(void** p, size_t n) { return alloc(p, n); }
int cudaMallocAsync(void** p, size_t n, void*) { return alloc(p, n); }
int cudaHostAlloc(void** p, size_t n, unsigned) { return alloc(p, n); }
int cudaFree(void* p) { return release(p); }
int cudaFreeAsync(void* p, void*) { return release(p); }
int cudaFreeHost(void* p) { return release(p); }
int cudaMemcpy(void* d, const void* s, size_t n, int kind) { return copy(d, s, n, kind); }
int cudaMemcpyAsync(void* d, const void* s, size_t n, int kind, void*) {
  return capture ? 0 : copy(d, s, n, kind);
}
int cudaMemset(void* p, int v, size_t n) { std::memset(p, v, n); return 0; }
int cudaMemsetAsync(void* p, int v, size_t n, void*) {
  if (!capture) std::memset(p, v, n);
  return 0;
}
int cudaGetSymbolAddress(void** p, const void*) {
  static void* area = std::calloc(32 << 20, 1);
  *p = area;
  return 0;
}
int cudaGetLastError() { const int e = last; last = 0; return e; }
const char* cudaGetErrorString(int e) { return e == 2 ? "out of memory" : "a failure made up"; }
int cudaGetDevice(int* d) { *d = 0; return 0; }
int cudaDeviceGetAttribute(int* v, int, int) { *v = 148; return 0; }
int cudaDeviceSynchronize() { return 0; }
int cudaFuncSetAttribute(const void*, int, int) { return 0; }
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* b, const void*, int, size_t,
                                                           unsigned) {
  *b = 4;
  return 0;
}
int cudaOccupancyMaxActiveClusters(int* c, const void*, const void*) { *c = 1; return 0; }
int cudaEventCreate(void** e) { return handle(e); }
int cudaEventCreateWithFlags(void** e, unsigned) { return handle(e); }
int cudaEventDestroy(void* e) { std::free(e); return 0; }
int cudaEventElapsedTime(float* ms, void*, void*) { *ms = 1.f; return 0; }
int cudaEventRecord(void*, void*) { return 0; }
int cudaEventRecordWithFlags(void*, void*, unsigned) { return 0; }
int cudaEventSynchronize(void*) { return 0; }
int cudaStreamCreateWithFlags(void** s, unsigned) { return handle(s); }
int cudaStreamDestroy(void* s) { std::free(s); return 0; }
int cudaStreamSynchronize(void*) { return 0; }
int cudaStreamWaitEvent(void*, void*, unsigned) { return 0; }
int cudaStreamBeginCapture(void*, int) { capture = new std::vector<std::string>(); return 0; }
int cudaStreamEndCapture(void*, void** g) {
  *g = capture;
  capture = nullptr;
  return 0;
}
int cudaGraphInstantiate(void** x, void* g, unsigned long long) {
  *x = new std::vector<std::string>(*(std::vector<std::string>*)g);
  return 0;
}
int cudaGraphDestroy(void* g) { delete (std::vector<std::string>*)g; return 0; }
int cudaGraphExecDestroy(void* x) { delete (std::vector<std::string>*)x; return 0; }
int cudaGraphLaunch(void* x, void*) {
  for (const std::string& n : *(std::vector<std::string>*)x) launched.push_back(n);
  return 0;
}
}
