// A CUDA runtime without a device, preloaded in front of the real one by
// test_host_calls.py: memory is host memory, copies run at once, kernels do
// nothing.  What it keeps is what the engine's host code is checked for:
// work queued and not yet waited for, streams being captured, graphs alive,
// and calls made to fail.  Capture follows the runtime's rules: a stream
// joins by waiting for an event recorded in the capture, a failing call
// invalidates the capture until the stream that began it ends it, and waits
// on a capturing stream are refused.
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>

namespace {

constexpr int kOk = 0, kFail = 2, kCaptureUnsupported = 900, kCaptureInvalidated = 901, kNotCapturing = 400;

struct Graph {
  int nodes = 0;
};
struct Stream {
  Graph *capture = nullptr;  // the graph it is captured into
  bool origin = false;
};
struct Event {
  Graph *capture = nullptr;
};

int last_error = kOk;
long long pending = 0, captures = 0, live_graphs = 0, live_execs = 0, instantiated = 0, waits = 0;
bool capture_failed = false;
std::set<Stream *> streams;
struct Fail {
  int after;       // calls of that name that still succeed
  bool recording;  // of those in a recording, or of all
};
std::map<std::string, Fail> fail_after;
long long patch_at = -1;  // bytes from the end of the next copy to the host
int patch_value = 0;

// whether this call, part of a recording or not, is the one to fail
bool fails(const char *name, bool recording)
{
  auto it = fail_after.find(name);
  if (it == fail_after.end() || (it->second.recording && !recording) || it->second.after-- > 0) return false;
  fail_after.erase(it);
  return true;
}
int note(int rc)
{
  if (rc) last_error = rc;
  return rc;
}
// one operation on a stream: a node of its graph, or pending work
int queue(const char *name, void *s)
{
  Stream *st = static_cast<Stream *>(s);
  if (fails(name, st && st->capture)) {
    capture_failed = true;
    return note(kFail);
  }
  if (st && st->capture)
    st->capture->nodes++;
  else
    pending++;
  return kOk;
}

}  // namespace

extern "C" {

// what the tests read and set: after `after` more calls of that name (in recordings, or all), one fails
void fake_fail(const char *name, int after, int recording) { fail_after[name] = Fail{after, recording != 0}; }
int fake_failed(const char *name) { return !fail_after.count(name); }
// an int of the next copy to the host, that far from its end, reads `value`
void fake_patch(long long from_end, int value) { patch_at = from_end, patch_value = value; }
long long fake_pending() { return pending; }
long long fake_capturing()
{
  long long n = 0;
  for (Stream *s : streams) n += s->capture != nullptr;
  return n;
}
long long fake_graphs() { return live_graphs; }
long long fake_execs() { return live_execs; }
long long fake_instantiated() { return instantiated; }
long long fake_waits() { return waits; }

int cudaGetDevice(int *d) { return *d = 0, kOk; }
int cudaSetDevice(int) { return kOk; }
int cudaDeviceGetAttribute(int *v, int, int) { return *v = 148, kOk; }
int cudaDeviceGetStreamPriorityRange(int *lo, int *hi) { return *lo = 0, *hi = -5, kOk; }
const char *cudaGetErrorString(int e) { return e == kOk ? "no error" : e == kFail ? "made to fail" : "capture error"; }
int cudaGetLastError()
{
  const int e = last_error;
  last_error = kOk;
  return e;
}
int cudaGetDriverEntryPoint(const char *, void **f, unsigned long long, void *) { return *f = nullptr, kOk; }
int cudaGetSymbolAddress(void **p, const void *) { return *p = nullptr, kFail; }
int cudaFuncSetAttribute(const void *, int, int) { return kOk; }
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) { return *n = 2, kOk; }

int cudaMalloc(void **p, size_t n)
{
  if (fails("cudaMalloc", false)) return note(kFail);
  return *p = calloc(n ? n : 1, 1), kOk;
}
int cudaFree(void *p) { return free(p), kOk; }
int cudaHostAlloc(void **p, size_t n, unsigned) { return *p = calloc(n ? n : 1, 1), kOk; }
int cudaFreeHost(void *p) { return free(p), kOk; }
int cudaMemcpy(void *d, const void *s, size_t n, int) { return memmove(d, s, n), kOk; }
int cudaMemset(void *d, int v, size_t n) { return memset(d, v, n), kOk; }
int cudaMemcpyAsync(void *d, const void *s, size_t n, int kind, void *st)
{
  const int rc = queue("cudaMemcpyAsync", st);
  if (rc || (st && static_cast<Stream *>(st)->capture)) return rc;
  memmove(d, s, n);
  if (kind == 2 && patch_at >= 0 && patch_at <= (long long) n) {  // device to host
    memcpy(static_cast<char *>(d) + n - patch_at, &patch_value, sizeof patch_value);
    patch_at = -1;
  }
  return rc;
}
int cudaMemsetAsync(void *d, int v, size_t n, void *st)
{
  const int rc = queue("cudaMemsetAsync", st);
  if (!rc && !(st && static_cast<Stream *>(st)->capture)) memset(d, v, n);
  return rc;
}

int cudaStreamCreateWithPriority(void **s, unsigned, int)
{
  Stream *st = new Stream;
  streams.insert(st);
  return *s = st, kOk;
}
int cudaStreamDestroy(void *s)
{
  streams.erase(static_cast<Stream *>(s));
  delete static_cast<Stream *>(s);
  return kOk;
}
int cudaStreamSynchronize(void *s)
{
  if (static_cast<Stream *>(s)->capture) return note(kCaptureUnsupported);
  pending = 0;  // the engine waits for its first stream, which the others have joined
  waits++;
  return kOk;
}
int cudaEventCreateWithFlags(void **e, unsigned) { return *e = new Event, kOk; }
int cudaEventCreate(void **e) { return *e = new Event, kOk; }
int cudaEventDestroy(void *e) { return delete static_cast<Event *>(e), kOk; }
int cudaEventElapsedTime(float *ms, void *, void *) { return *ms = 0.0027f, kOk; }  // two events side by side
int cudaEventRecord(void *e, void *s)
{
  Stream *st = static_cast<Stream *>(s);
  if (fails("cudaEventRecord", st->capture)) {
    capture_failed = true;
    return note(kFail);
  }
  static_cast<Event *>(e)->capture = st->capture;
  return kOk;
}
int cudaStreamWaitEvent(void *s, void *e, unsigned)
{
  Stream *st = static_cast<Stream *>(s);
  if (Graph *g = static_cast<Event *>(e)->capture) {
    if (st->capture && st->capture != g) return note(kCaptureUnsupported);
    st->capture = g;
  }
  return kOk;
}

int cudaStreamBeginCapture(void *s, int)
{
  Stream *st = static_cast<Stream *>(s);
  if (st->capture) return note(kCaptureUnsupported);
  st->capture = new Graph;
  st->origin = true;
  capture_failed = false;
  captures++;
  return kOk;
}
int cudaStreamEndCapture(void *s, void **g)
{
  Stream *st = static_cast<Stream *>(s);
  *g = nullptr;
  if (!st->capture || !st->origin) return note(kNotCapturing);
  Graph *graph = st->capture;
  st->origin = false;
  for (Stream *q : streams)
    if (q->capture == graph) q->capture = nullptr;
  if (capture_failed) {
    delete graph;
    return note(kCaptureInvalidated);
  }
  live_graphs++;
  return *g = graph, kOk;
}
int cudaGraphDestroy(void *g)
{
  live_graphs--;
  delete static_cast<Graph *>(g);
  return kOk;
}
int cudaGraphGetNodes(void *, void **, size_t *n) { return *n = 0, kOk; }
int cudaGraphNodeGetType(void *, int *t) { return *t = 0, kOk; }
int cudaGraphKernelNodeGetParams(void *, void *) { return kOk; }
int cudaGraphKernelNodeSetAttribute(void *, int, const void *) { return kOk; }
int cudaGraphInstantiate(void **x, void *, unsigned long long)
{
  if (fails("cudaGraphInstantiate", true)) return note(kFail);
  live_execs++;
  instantiated++;
  return *x = new int, kOk;
}
int cudaGraphExecDestroy(void *x)
{
  live_execs--;
  delete static_cast<int *>(x);
  return kOk;
}
int cudaGraphLaunch(void *, void *s) { return queue("cudaGraphLaunch", s); }

// launches: <<<...>>> pushes its stream, the kernel's stub pops it
static void *pushed;
unsigned __cudaPushCallConfiguration(unsigned long long, unsigned, unsigned long long, unsigned, size_t, void *s)
{
  pushed = s;
  return 0;
}
int __cudaPopCallConfiguration(void *, void *, size_t *shared, void **s)
{
  *shared = 0;
  return *s = pushed, kOk;
}
struct Dim3 {
  unsigned x, y, z;
};
int cudaLaunchKernel(const void *, Dim3, Dim3, void **, size_t, void *s) { return queue("cudaLaunchKernel", s); }
int cudaLaunchKernelExC(const void *cfg, const void *, void **)
{
  // cudaLaunchConfig_t: grid, block (12 bytes each), shared bytes, stream
  void *s;
  memcpy(&s, static_cast<const char *>(cfg) + 32, sizeof s);
  return queue("cudaLaunchKernel", s);
}
static void *module;
void **__cudaRegisterFatBinary(void *) { return &module; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, void *, void *, void *, void *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
}
