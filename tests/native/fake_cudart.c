/* A CUDA runtime without a GPU for libwrfgpu.so, loaded ahead of the real one:
 * memory is host memory, copies are copies, streams and events are nothing,
 * and a launch runs no kernel but is refused, as the runtime refuses it, when
 * it asks for more dynamic shared memory than its kernel has been allowed on
 * the current device (48 KB until cudaFuncSetAttribute says otherwise).
 * Devices are numbers, chosen by fake_set_device. */
#include <stddef.h>
#include <stdlib.h>
#include <string.h>

typedef struct { unsigned x, y, z; } Dim3;
enum { OK = 0, INVALID = 1, NDEV = 4, NKERNEL = 512, DEFAULT_BYTES = 49152 };

static int device, last, launches, refused, lowered, nkernel;
static struct { const void* f; int bytes[NDEV]; } kernel[NKERNEL];

void fake_set_device(int d) { device = d; }
int fake_launches(void) { return launches; }
int fake_refused(void) { return refused; }
int fake_lowered(void) { return lowered; } /* allowances set below an earlier one */

static int* allowance(const void* f) {
  int q = 0;
  while (q < nkernel && kernel[q].f != f) ++q;
  if (q == NKERNEL) abort();
  if (q == nkernel) {
    kernel[nkernel++].f = f;
    for (int d = 0; d < NDEV; ++d) kernel[q].bytes[d] = DEFAULT_BYTES;
  }
  return &kernel[q].bytes[device];
}
int cudaFuncSetAttribute(const void* f, int attr, int value) {
  if (attr != 8) return OK; /* cudaFuncAttributeMaxDynamicSharedMemorySize */
  int* a = allowance(f);
  if (value < *a && *a != DEFAULT_BYTES) ++lowered;
  *a = value;
  return OK;
}
int __cudaGetKernel(const void** k, const void* f) { *k = f; return OK; }
int __cudaLaunchKernel(const void* k, Dim3 grid, Dim3 block, void** args, size_t smem, void* stream) {
  (void)args; (void)stream;
  ++launches;
  if (!grid.x || !grid.y || !grid.z || block.x * block.y * block.z > 1024u || smem > (size_t)*allowance(k)) {
    ++refused;
    return last = INVALID;
  }
  return OK;
}
int cudaGetLastError(void) { const int e = last; last = OK; return e; }

static struct { Dim3 grid, block; size_t smem; void* stream; } pushed;
unsigned __cudaPushCallConfiguration(Dim3 grid, Dim3 block, size_t smem, void* stream) {
  pushed.grid = grid; pushed.block = block; pushed.smem = smem; pushed.stream = stream;
  return 0;
}
int __cudaPopCallConfiguration(Dim3* grid, Dim3* block, size_t* smem, void* stream) {
  *grid = pushed.grid; *block = pushed.block; *smem = pushed.smem; *(void**)stream = pushed.stream;
  return OK;
}
static void* handle = &handle;
void** __cudaRegisterFatBinary(void* b) { (void)b; return &handle; }
void __cudaRegisterFatBinaryEnd(void** h) { (void)h; }
void __cudaUnregisterFatBinary(void** h) { (void)h; }
void __cudaRegisterFunction(void) {}
void __cudaRegisterVar(void) {}

int cudaMalloc(void** p, size_t n) { *p = calloc(n, 1); return *p ? OK : 2; }
int cudaFree(void* p) { free(p); return OK; }
int cudaMemcpy(void* d, const void* s, size_t n, int kind) { (void)kind; memcpy(d, s, n); return OK; }
int cudaMemcpyAsync(void* d, const void* s, size_t n, int kind, void* st) { (void)st; return cudaMemcpy(d, s, n, kind); }
int cudaMemset(void* d, int v, size_t n) { memset(d, v, n); return OK; }
int cudaMemsetAsync(void* d, int v, size_t n, void* st) { (void)st; return cudaMemset(d, v, n); }
int cudaStreamCreateWithFlags(void** s, unsigned f) { (void)f; *s = &handle; return OK; }
int cudaStreamDestroy(void* s) { (void)s; return OK; }
int cudaStreamSynchronize(void* s) { (void)s; return OK; }
int cudaStreamWaitEvent(void* s, void* e, unsigned f) { (void)s; (void)e; (void)f; return OK; }
int cudaDeviceSynchronize(void) { return OK; }
int cudaEventCreate(void** e) { *e = &handle; return OK; }
int cudaEventCreateWithFlags(void** e, unsigned f) { (void)f; *e = &handle; return OK; }
int cudaEventDestroy(void* e) { (void)e; return OK; }
int cudaEventRecord(void* e, void* s) { (void)e; (void)s; return OK; }
int cudaEventSynchronize(void* e) { (void)e; return OK; }
static int encode(void) { return OK; } /* a tensor map nobody reads */
int cudaGetDriverEntryPointByVersion(const char* name, void** fn, unsigned v, unsigned long long flags, int* status) {
  (void)name; (void)v; (void)flags;
  *fn = (void*)encode;
  *status = 0;
  return OK;
}
