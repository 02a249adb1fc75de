// A CUDA runtime for host tests, put in front of the real one with LD_PRELOAD: allocations are addresses that nothing
// touches, launches are counted and their kernels named, and the n-th allocation or launch from now can be made to fail.  It
// needs no GPU and no CUDA headers.
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <map>
#include <string>

namespace {
std::atomic<long> g_fail_in{0};             // 1: the next allocation fails; 0: none does
std::atomic<long> g_launches{0};
std::atomic<long> g_fail_launch_in{0};      // as g_fail_in, of launches
std::map<const void*, std::string> g_names;      // of the registered kernels
unsigned g_grid = 0;                        // blocks of the last launch in x
std::string g_launched;                     // kernels launched since fake_launched(), one name a line
std::map<void*, void*> g_recorded;          // event -> the stream it was last recorded on
std::map<void*, bool> g_forked;             // stream of the library's -> something has waited for it since it waited
std::map<void*, long> g_unfinished;         // fills and copies to the device that nothing has waited for, by stream
uintptr_t g_next = uintptr_t(1) << 44;
int encode(...) { return 0; }
void* const kOwnStream = reinterpret_cast<void*>(uintptr_t(0x1000));
int launch(const void* kernel) {
  if (g_fail_launch_in > 0 && --g_fail_launch_in == 0) return 2;
  ++g_launches;
  g_launched += g_names[kernel] + "\n";
  return 0;
}
}  // namespace

extern "C" {

void fake_fail_allocation(long in) { g_fail_in = in; }
long fake_allocations_left() { return g_fail_in; }
long fake_launches() { return g_launches; }
void fake_fail_launch(long in) { g_fail_launch_in = in; }
long fake_launch_failures_left() { return g_fail_launch_in; }
const char* fake_launched() {
  static std::string last;
  last.swap(g_launched);
  g_launched.clear();
  return last.c_str();
}
long fake_grid() { return g_grid; }
// 1: the library's own stream waited for another, which has not waited for it since
long fake_forked() { return g_forked[kOwnStream]; }
long fake_unfinished() {
  long sum = 0;
  for (const auto& stream : g_unfinished) sum += stream.second;
  return sum;
}

int cudaMalloc(void** p, size_t bytes) {
  if (g_fail_in > 0 && --g_fail_in == 0) return 2;         // cudaErrorMemoryAllocation
  *p = reinterpret_cast<void*>(g_next);
  g_next += (bytes + 511) / 512 * 512 + 512;
  return 0;
}
int cudaFree(void*) { return 0; }
// cudaMemset and a cudaMemcpy to the device return before the device has done them
int cudaMemset(void*, int, size_t) { ++g_unfinished[nullptr]; return 0; }
int cudaMemsetAsync(void*, int, size_t, void* stream) { ++g_unfinished[stream]; return 0; }
int cudaMemcpy(void*, const void*, size_t, int kind) { if (kind == 1) ++g_unfinished[nullptr]; return 0; }
int cudaMemcpyAsync(void*, const void*, size_t, int, void* stream) { ++g_unfinished[stream]; return 0; }
int cudaDeviceSynchronize() { g_unfinished.clear(); return 0; }
int cudaStreamSynchronize(void* stream) { g_unfinished.erase(stream); return 0; }

int cudaGetDevice(int* device) { *device = 0; return 0; }
int cudaDeviceGetAttribute(int* value, int, int) { *value = 148; return 0; }      // asked for the number of SMs only
int cudaGetLastError() { return 0; }
int cudaFuncSetAttribute(const void*, int, int) { return 0; }
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*, void*, void*, int*) { g_names[host] = name; }
int cudaOccupancyMaxActiveClusters(int* clusters, const void*, const void* config) {      // gridDim.x is one cluster's blocks
  *clusters = 148 / int(*static_cast<const unsigned*>(config));
  return 0;
}
int cudaLaunchKernelExC(const void* config, const void* kernel, void**) {      // it begins with gridDim.x
  g_grid = *static_cast<const unsigned*>(config);
  return launch(kernel);
}
struct Dim3 { unsigned x, y, z; };
int cudaLaunchKernel(const void* kernel, Dim3, Dim3, void**, size_t, void*) { return launch(kernel); }
int cudaGetDriverEntryPoint(const char*, void** entry, unsigned long long, int* result) {
  *entry = reinterpret_cast<void*>(&encode);
  if (result) *result = 0;
  return 0;
}
int cudaStreamCreateWithFlags(void** stream, unsigned) { *stream = kOwnStream; return 0; }
int cudaStreamDestroy(void*) { return 0; }
int cudaStreamWaitEvent(void* stream, void* event, unsigned) {
  if (stream == kOwnStream) g_forked[stream] = true;
  else g_forked[g_recorded[event]] = false;
  return 0;
}
int cudaEventCreateWithFlags(void** event, unsigned) {
  static uintptr_t next = 0x2000;
  *event = reinterpret_cast<void*>(next += 8);
  return 0;
}
int cudaEventDestroy(void*) { return 0; }
int cudaEventRecord(void* event, void* stream) { g_recorded[event] = stream; return 0; }

}  // extern "C"
