// A CUDA runtime that runs nothing: loaded in front of the real one, it keeps
// "device" memory on the host, carries out copies at once and writes one line
// per call that touches a stream to stderr:
//   default <call>            work on the default stream
//   stream <s> <call or kernel>
//   wait <s> | wait all       the host waited for a stream, or for the device
// A test reads the order from it, with no GPU.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

extern "C" {

struct dim3 {
  unsigned x, y, z;
};
struct launch_config {
  dim3 grid, block;
  size_t smem;
  void *stream;
};
typedef int status;

static long next_handle = 1;
static std::map<const void *, std::string> names;
static launch_config pushed;

static void *handle() { return (void *)(next_handle++ << 4); }
static void on(void *s, const char *what) {
  if (s) fprintf(stderr, "stream %ld %s\n", (long)s >> 4, what);
  else fprintf(stderr, "default %s\n", what);
}

// programs
void **__cudaRegisterFatBinary(void *) { return (void **)handle(); }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *fun, char *, const char *name, int, void *, void *, void *, void *,
                            int *) {
  names[fun] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
status __cudaGetKernel(const void **k, const void *fun) {
  *k = fun;
  return 0;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void *stream) {
  pushed = launch_config{g, b, smem, stream};
  return 0;
}
status __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void **stream) {
  *g = pushed.grid;
  *b = pushed.block;
  *smem = pushed.smem;
  *stream = pushed.stream;
  return 0;
}
status __cudaLaunchKernel(const void *k, dim3, dim3, void **, size_t, void *stream) {
  on(stream, names[k].c_str());
  return 0;
}
status cudaLaunchKernelExC(const launch_config *c, const void *k, void **) {
  on(c->stream, names[k].c_str());
  return 0;
}
status cudaFuncSetAttribute(const void *, int, int) { return 0; }
status cudaOccupancyMaxActiveClusters(int *n, const void *, const launch_config *) {
  *n = 1;
  return 0;
}

// memory
status cudaMalloc(void **p, size_t n) {
  *p = calloc(1, n ? n : 1);
  return *p ? 0 : 2;
}
status cudaFree(void *p) {
  if (p) fprintf(stderr, "wait all\n");  // freeing waits for the device
  free(p);
  return 0;
}
status cudaHostAlloc(void **p, size_t n, unsigned) {
  *p = calloc(1, n ? n : 1);
  return *p ? 0 : 2;
}
status cudaMallocHost(void **p, size_t n) { return cudaHostAlloc(p, n, 0); }
status cudaFreeHost(void *p) {
  free(p);
  return 0;
}
status cudaHostRegister(void *, size_t, unsigned) { return 0; }
status cudaHostUnregister(void *) { return 0; }
status cudaGetSymbolAddress(void **p, const void *) { return cudaMalloc(p, 1 << 24); }
status cudaMemcpy(void *d, const void *s, size_t n, int) {
  memcpy(d, s, n);
  on(nullptr, "cudaMemcpy");
  return 0;
}
status cudaMemcpyAsync(void *d, const void *s, size_t n, int, void *stream) {
  memcpy(d, s, n);
  on(stream, "cudaMemcpyAsync");
  return 0;
}
status cudaMemset(void *d, int v, size_t n) {
  memset(d, v, n);
  on(nullptr, "cudaMemset");
  return 0;
}
status cudaMemsetAsync(void *d, int v, size_t n, void *stream) {
  memset(d, v, n);
  on(stream, "cudaMemsetAsync");
  return 0;
}

// streams, events, graphs
status cudaStreamCreateWithFlags(void **s, unsigned) {
  *s = handle();
  return 0;
}
status cudaStreamDestroy(void *) { return 0; }
status cudaStreamSynchronize(void *s) {
  fprintf(stderr, "wait %ld\n", (long)s >> 4);
  return 0;
}
status cudaDeviceSynchronize() {
  fprintf(stderr, "wait all\n");
  return 0;
}
status cudaStreamWaitEvent(void *, void *, unsigned) { return 0; }
status cudaStreamBeginCapture(void *, int) { return 0; }
status cudaStreamEndCapture(void *, void **g) {
  *g = handle();
  return 0;
}
status cudaGraphInstantiate(void **x, void *, unsigned long long) {
  *x = handle();
  return 0;
}
status cudaGraphDestroy(void *) { return 0; }
status cudaGraphExecDestroy(void *) { return 0; }
status cudaGraphLaunch(void *, void *s) {
  on(s, "cudaGraphLaunch");
  return 0;
}
status cudaEventCreate(void **e) {
  *e = handle();
  return 0;
}
status cudaEventCreateWithFlags(void **e, unsigned) { return cudaEventCreate(e); }
status cudaEventDestroy(void *) { return 0; }
status cudaEventRecord(void *, void *) { return 0; }
status cudaEventSynchronize(void *) { return 0; }
status cudaEventElapsedTime(float *ms, void *, void *) {
  *ms = 1.0f;
  return 0;
}

status cudaSetDevice(int) { return 0; }
status cudaGetDevice(int *d) {
  *d = 0;
  return 0;
}
status cudaGetLastError() { return 0; }
const char *cudaGetErrorString(status) { return "error"; }
}
