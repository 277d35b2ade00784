// fake_cudart.cpp - a stand-in for libcudart.so.12 on machines without a GPU: two devices whose memory
// is the host's, streams that run at once, kernels that are checked and not run. It keeps what belongs
// to a device in the real runtime (a kernel's dynamic shared-memory limit, memory, constants, events)
// per device, takes it away on cudaDeviceReset, and answers the use of what was taken away with an
// error, so that the library's host side can be tested for several devices and across resets.
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <set>
#include <string>
#include <utility>
#include <vector>

extern "C" {

typedef int Err;  // cudaError_t
enum { OK = 0, BAD_VALUE = 1, NO_MEMORY = 2, BAD_HANDLE = 400, NOT_FOUND = 500 };
struct Dim3 { unsigned x, y, z; };
struct Event { int dev; unsigned long long ctx; };

static std::mutex mu;
static thread_local int curDev = 0;
static thread_local Err lastErr = OK;
static unsigned long long ctxId[2] = {1, 2}, nextCtx = 3;
static std::map<std::pair<int, const void *>, size_t> smemLimit;  // (device, kernel)
static std::map<const void *, std::string> kernelName;
static std::map<std::pair<int, const void *>, std::vector<char>> symbols;  // (device, variable): as last uploaded
static std::set<Event *> events;
static std::map<std::string, int> calls;
static std::vector<std::string> launches;

static Err fail(Err e) { if (e != OK) { lastErr = e; } return e; }
static void count(const char *what) { std::lock_guard<std::mutex> lk(mu); calls[what]++; }

// ---- for the tests
int fake_calls(const char *what) { std::lock_guard<std::mutex> lk(mu); return calls[what]; }
int fake_events_alive() { std::lock_guard<std::mutex> lk(mu); return (int)events.size(); }
// The launched kernels since the last call, one per line: device, name, dynamic shared memory, blocks, threads.
const char *fake_launches()
{
   static std::string s;
   std::lock_guard<std::mutex> lk(mu);
   s.clear();
   for (const std::string &l : launches) { s += l + "\n"; }
   launches.clear();
   return s.c_str();
}

// ---- registration and launch
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, void *, void *, void *, void *, int *)
{
   kernelName[host] = name;
}
static thread_local struct { Dim3 g, b; size_t smem; void *s; } config;
unsigned __cudaPushCallConfiguration(Dim3 g, Dim3 b, size_t smem, void *s) { config = {g, b, smem, s}; return 0; }
Err __cudaPopCallConfiguration(Dim3 *g, Dim3 *b, size_t *smem, void **s)
{
   *g = config.g; *b = config.b; *smem = config.smem; *s = config.s;
   return OK;
}
static size_t limitOf(const void *f)
{
   auto it = smemLimit.find({curDev, f});
   return it == smemLimit.end() ? 48 * 1024 : it->second;
}
// The first argument of the last batch kernel launched (tasks, chunks, number of chunks, counter).
static unsigned char batchArgs[32];
const void *fake_batch_args() { return batchArgs; }
Err cudaLaunchKernel(const void *f, Dim3 g, Dim3 b, void **args, size_t smem, void *)
{
   std::lock_guard<std::mutex> lk(mu);
   if (kernelName[f].find("Batch") != std::string::npos) { memcpy(batchArgs, args[0], sizeof(batchArgs)); }
   if (smem > limitOf(f) || g.x == 0 || b.x == 0 || b.x > 1024) { return fail(BAD_VALUE); }
   launches.push_back(std::to_string(curDev) + " " + kernelName[f] + " " + std::to_string(smem) + " " +
                      std::to_string(g.x) + " " + std::to_string(b.x));
   return OK;
}
Err cudaFuncSetAttribute(const void *f, int attr, int v)
{
   if (attr != 8 || v < 0 || v > 232448) { return fail(BAD_VALUE); }  // 8: the dynamic shared-memory limit
   std::lock_guard<std::mutex> lk(mu);
   smemLimit[{curDev, f}] = (size_t)v;
   return OK;
}
Err cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int, size_t smem, unsigned)
{
   std::lock_guard<std::mutex> lk(mu);
   if (smem > limitOf(f)) { *n = 0; return OK; }
   *n = smem > 0 ? (int)(232448 / (smem + 1024)) : 8;
   return OK;
}

// ---- devices and errors
Err cudaGetDevice(int *d) { *d = curDev; return OK; }
Err cudaSetDevice(int d) { if (d < 0 || d > 1) { return fail(BAD_VALUE); } curDev = d; return OK; }
Err cudaGetDeviceCount(int *n) { *n = 2; return OK; }
Err cudaDeviceGetAttribute(int *v, int attr, int) { *v = attr == 16 ? 148 : 0; return OK; }  // 16: multiprocessors
Err cudaDeviceReset()
{
   std::lock_guard<std::mutex> lk(mu);
   ctxId[curDev] = nextCtx++;
   for (auto it = smemLimit.begin(); it != smemLimit.end();) { it = it->first.first == curDev ? smemLimit.erase(it) : std::next(it); }
   for (auto it = symbols.begin(); it != symbols.end();) { it = it->first.first == curDev ? symbols.erase(it) : std::next(it); }
   for (auto it = events.begin(); it != events.end();) { it = (*it)->dev == curDev ? events.erase(it) : std::next(it); }
   return OK;
}
Err cudaGetLastError() { const Err e = lastErr; lastErr = OK; return e; }
const char *cudaGetErrorName(Err) { return "fake"; }
const char *cudaGetErrorString(Err) { return "fake error"; }
static int fakeCtxGetId(void *, unsigned long long *id) { *id = ctxId[curDev]; return 0; }
static int fakeEncode() { return 0; }
Err cudaGetDriverEntryPointByVersion(const char *name, void **p, unsigned, unsigned long long, int *q)
{
   *p = !strcmp(name, "cuCtxGetId") ? (void *)fakeCtxGetId : !strcmp(name, "cuTensorMapEncodeTiled") ? (void *)fakeEncode : nullptr;
   *q = *p ? 0 : 1;
   return *p ? OK : fail(NOT_FOUND);
}

// ---- memory (the host's; freed memory is left alone, a reset device's too)
Err cudaMalloc(void **p, size_t n) { *p = calloc(1, n ? n : 1); return *p ? OK : fail(NO_MEMORY); }
Err cudaMallocHost(void **p, size_t n) { return cudaMalloc(p, n); }
Err cudaHostAlloc(void **p, size_t n, unsigned) { return cudaMalloc(p, n); }
Err cudaFree(void *) { return OK; }
Err cudaFreeHost(void *) { return OK; }
Err cudaMemcpy(void *d, const void *s, size_t n, int) { memcpy(d, s, n); return OK; }
Err cudaMemcpyAsync(void *d, const void *s, size_t n, int, void *) { memcpy(d, s, n); return OK; }
Err cudaMemset(void *d, int v, size_t n) { memset(d, v, n); return OK; }
Err cudaMemsetAsync(void *d, int v, size_t n, void *) { memset(d, v, n); return OK; }
Err cudaMemcpyToSymbol(const void *sym, const void *s, size_t n, size_t, int)
{
   count("cudaMemcpyToSymbol");
   std::lock_guard<std::mutex> lk(mu);
   symbols[{curDev, sym}].assign((const char *)s, (const char *)s + n);
   return OK;
}
Err cudaMemcpyFromSymbol(void *d, const void *sym, size_t n, size_t, int)
{
   std::lock_guard<std::mutex> lk(mu);
   std::vector<char> v = symbols[{curDev, sym}];
   v.resize(n, 0);
   memcpy(d, v.data(), n);
   return OK;
}
Err cudaGetSymbolAddress(void **p, const void *) { static char buf[1 << 26]; *p = buf; return OK; }

// ---- streams, events, graphs
Err cudaStreamCreateWithFlags(void **s, unsigned) { *s = calloc(1, 8); return OK; }
Err cudaStreamDestroy(void *) { return OK; }
Err cudaStreamSynchronize(void *) { return OK; }
Err cudaStreamWaitEvent(void *, void *, unsigned) { return OK; }
Err cudaStreamBeginCapture(void *, int) { return OK; }
Err cudaStreamEndCapture(void *, void **g) { *g = calloc(1, 8); return OK; }
Err cudaGraphInstantiate(void **e, void *, unsigned long long) { *e = calloc(1, 8); return OK; }
Err cudaGraphLaunch(void *, void *) { return OK; }
Err cudaGraphDestroy(void *) { return OK; }
Err cudaGraphExecDestroy(void *) { return OK; }
Err cudaEventCreateWithFlags(void **e, unsigned)
{
   count("cudaEventCreate");
   std::lock_guard<std::mutex> lk(mu);
   Event *v = new Event{curDev, ctxId[curDev]};
   events.insert(v);
   *e = v;
   return OK;
}
Err cudaEventCreate(void **e) { return cudaEventCreateWithFlags(e, 0); }
// (a handle that is not alive: counted, as the real runtime may answer with a crash)
static Err useEvent(void *e, bool here)
{
   std::lock_guard<std::mutex> lk(mu);
   if (!events.count((Event *)e)) { calls["dead event"]++; return fail(BAD_HANDLE); }
   return here && ((Event *)e)->dev != curDev ? fail(BAD_HANDLE) : OK;
}
Err cudaEventRecord(void *e, void *) { return useEvent(e, true); }
Err cudaEventQuery(void *e) { return useEvent(e, false); }
Err cudaEventSynchronize(void *e) { return useEvent(e, false); }
Err cudaEventElapsedTime(float *ms, void *a, void *b) { *ms = 0.25f; const Err e = useEvent(a, false); return e != OK ? e : useEvent(b, false); }
Err cudaEventDestroy(void *e)
{
   if (useEvent(e, false) != OK) { return BAD_HANDLE; }
   std::lock_guard<std::mutex> lk(mu);
   events.erase((Event *)e);
   return OK;
}

}  // extern "C"
