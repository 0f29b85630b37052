// A stand-in for the CUDA runtime, for tests of the library's host side without
// a GPU: the objects of libhowmhd.so are linked against this file instead of
// cudart.  Nothing runs on a device and no byte is copied; what is checked and
// counted is what the host asks for: launches (kernel, device, grid, dynamic
// shared memory against the kernel's limit on that device, 48 KB unless raised),
// captures, graphs and their replays.  A call can be made to fail by name.
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

namespace {

struct Dim { unsigned x, y, z; };
enum { kOk = 0, kInvalidValue = 1, kNotFound = 500, kUnknown = 999 };

std::mutex mu;
std::map<const void*, std::string> names;                 // host stub -> kernel's name
std::map<std::pair<int, const void*>, int> smem_limit;    // (device, kernel) -> bytes
std::map<std::string, long> calls;                        // counted calls by name
std::map<std::string, int> failing;                       // calls that fail, and with what
std::vector<std::string> log_;                            // launches
uintptr_t next_address = uintptr_t(1) << 40;
int devices = 1;
int watched = -1;                                         // offset into the first argument (fake_watch)
thread_local int device = 0, last_error = kOk;
thread_local bool capturing = false;
thread_local struct { Dim grid, block; size_t smem; void* stream; } pushed;

int done(int e) {
    if (e != kOk) last_error = e;
    return e;
}
int enter(const char* name) {
    std::lock_guard<std::mutex> l(mu);
    ++calls[name];
    const auto f = failing.find(name);
    return done(f == failing.end() ? int(kOk) : f->second);
}
int accept_tensor_map(...) { return 0; }   // stands for cuTensorMapEncodeTiled

}  // namespace

extern "C" {

// ---- what the tests call
void fake_reset(int ndevices) {
    std::lock_guard<std::mutex> l(mu);
    calls.clear(); failing.clear(); log_.clear();
    devices = ndevices;
    watched = -1;
    device = 0;
    last_error = kOk;
}
void fake_fail(const char* name, int error) {
    std::lock_guard<std::mutex> l(mu);
    if (error) failing[name] = error; else failing.erase(name);
}
long fake_calls(const char* name) { std::lock_guard<std::mutex> l(mu); return calls[name]; }
// from here on launches of the sweeps note the int at this offset of their first argument
void fake_watch(int offset) { watched = offset; }
// the launches since the last call, a line each: captured, device, grid, block, dynamic shared memory, the
// watched int, kernel
const char* fake_launches() {
    static std::string out;
    std::lock_guard<std::mutex> l(mu);
    out.clear();
    for (const auto& s : log_) out += s + "\n";
    log_.clear();
    return out.c_str();
}
int fake_set_device(int d) { device = d; return 0; }

// ---- the runtime
void** __cudaRegisterFatBinary(void*) { static void* h = nullptr; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*, void*, void*, int*) {
    std::lock_guard<std::mutex> l(mu);
    names[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(Dim g, Dim b, size_t smem, void* stream) {
    pushed = {g, b, smem, stream};
    return 0;
}
int __cudaPopCallConfiguration(Dim* g, Dim* b, size_t* smem, void** stream) {
    *g = pushed.grid; *b = pushed.block; *smem = pushed.smem; *stream = pushed.stream;
    return 0;
}
int cudaLaunchKernel(const void* f, Dim g, Dim b, void** args, size_t smem, void*) {
    const int e = enter(capturing ? "captured launch" : "cudaLaunchKernel");
    if (e) return e;
    std::lock_guard<std::mutex> l(mu);
    const auto lim = smem_limit.find({device, f});
    if (smem > size_t(lim == smem_limit.end() ? 49152 : lim->second)) return done(kInvalidValue);
    char line[160];
    const std::string& name = names[f];
    int seen = 0;
    if (watched >= 0 && name.find("k_sweep") != std::string::npos)
        std::memcpy(&seen, static_cast<char*>(args[0]) + watched, sizeof(int));
    std::snprintf(line, sizeof(line), "%d %d %u,%u,%u %u,%u,%u %zu %d ", int(capturing), device, g.x, g.y, g.z, b.x, b.y,
                  b.z, smem, seen);
    log_.push_back(line + name);
    return kOk;
}
int cudaFuncSetAttribute(const void* f, int attr, int value) {
    const int e = enter("cudaFuncSetAttribute");
    if (e) return e;
    std::lock_guard<std::mutex> l(mu);
    if (attr == 8) smem_limit[{device, f}] = value;   // cudaFuncAttributeMaxDynamicSharedMemorySize
    return kOk;
}
int cudaGetLastError() { const int e = last_error; last_error = kOk; return e; }
int cudaPeekAtLastError() { return last_error; }
const char* cudaGetErrorName(int) { return "fake error"; }
const char* cudaGetErrorString(int) { return "fake error"; }
int cudaGetDeviceCount(int* n) { *n = devices; return enter("cudaGetDeviceCount"); }
int cudaGetDevice(int* d) { *d = device; return kOk; }
int cudaSetDevice(int d) {
    if (d < 0 || d >= devices) return done(101);
    device = d;
    return kOk;
}
int cudaDeviceReset() {   // the current device's function attributes go with its context
    std::lock_guard<std::mutex> l(mu);
    for (auto it = smem_limit.begin(); it != smem_limit.end();)
        it = it->first.first == device ? smem_limit.erase(it) : std::next(it);
    return kOk;
}
int cudaDeviceGetAttribute(int* v, int attr, int d) {
    *v = attr == 16 ? (d == 0 ? 148 : 100) : 0;   // cudaDevAttrMultiProcessorCount: another one on other devices
    return enter("cudaDeviceGetAttribute");
}
int cudaDeviceCanAccessPeer(int* ok, int, int) { *ok = 1; return kOk; }
int cudaDeviceEnablePeerAccess(int, unsigned) { return kOk; }
int cudaGetDriverEntryPoint(const char*, void** f, unsigned long long, int* q) {
    *f = reinterpret_cast<void*>(&accept_tensor_map);
    *q = 0;
    return kOk;
}
int cudaGetSymbolAddress(void** p, const void*) { *p = reinterpret_cast<void*>(uintptr_t(1) << 39); return kOk; }
int cudaMalloc(void** p, size_t n) {
    const int e = enter("cudaMalloc");
    if (e) return e;
    std::lock_guard<std::mutex> l(mu);
    *p = reinterpret_cast<void*>(next_address);
    next_address += (n + 4095) / 4096 * 4096;
    return kOk;
}
int cudaFree(void*) { return kOk; }
int cudaHostAlloc(void** p, size_t n, unsigned) { *p = std::calloc(1, n); return kOk; }
int cudaMallocHost(void** p, size_t n) { *p = std::calloc(1, n); return kOk; }
int cudaFreeHost(void* p) { std::free(p); return kOk; }
int cudaMemcpy(void*, const void*, size_t, int) { return enter("cudaMemcpy"); }
int cudaMemcpyAsync(void*, const void*, size_t, int, void*) { return enter("cudaMemcpyAsync"); }
int cudaMemcpyPeerAsync(void*, int, const void*, int, size_t, void*) { return enter("cudaMemcpyPeerAsync"); }
int cudaMemset(void*, int, size_t) { return kOk; }
int cudaMemsetAsync(void*, int, size_t, void*) { return kOk; }
int cudaEventCreate(void** e) { *e = std::malloc(1); return kOk; }
int cudaEventCreateWithFlags(void** e, unsigned) { *e = std::malloc(1); return kOk; }
int cudaEventDestroy(void* e) { std::free(e); return kOk; }
int cudaEventRecord(void*, void*) { return kOk; }
int cudaEventSynchronize(void*) { return kOk; }
int cudaEventElapsedTime(float* ms, void*, void*) { *ms = 1.0f; return kOk; }
int cudaStreamCreateWithFlags(void** s, unsigned) { *s = std::malloc(1); return kOk; }
int cudaStreamDestroy(void* s) { std::free(s); return kOk; }
int cudaStreamSynchronize(void*) { return kOk; }
int cudaStreamWaitEvent(void*, void*, unsigned) { return kOk; }
int cudaStreamBeginCapture(void*, int) {
    const int e = enter("cudaStreamBeginCapture");
    if (!e) capturing = true;
    return e;
}
int cudaStreamEndCapture(void*, void** graph) {
    capturing = false;
    const int e = enter("cudaStreamEndCapture");
    *graph = e ? nullptr : std::malloc(1);
    return e;
}
int cudaGraphInstantiate(void** exec, void*, unsigned long long) {
    const int e = enter("cudaGraphInstantiate");
    if (!e) *exec = std::malloc(1);
    return e;
}
int cudaGraphDestroy(void* g) { std::free(g); return kOk; }
int cudaGraphExecDestroy(void* g) { std::free(g); enter("cudaGraphExecDestroy"); return kOk; }
int cudaGraphLaunch(void*, void*) { return enter("cudaGraphLaunch"); }

}  // extern "C"
