/* A CUDA runtime for host-path tests, preloaded before libcudart: device memory
 * is host memory, kernels do nothing, and calls of interest are counted.  A
 * library run on it takes the host's path through its entry points (what it
 * allocates, captures and launches, and how it handles a call that fails)
 * without a GPU; fields keep the values the host copied in.
 *
 *   fake_count(name)     calls so far of "HostAlloc", "HostRegister", "Instantiate",
 *                        "GraphLaunch", "Launch" (outside a capture), "Capture" (within one)
 *   fake_fail_launch(n)  the n-th launch from now fails (0: none)
 *
 * Only the arguments that matter are declared: the rest stay in registers or on
 * the caller's stack. */
#include <stddef.h>
#include <stdlib.h>
#include <string.h>

enum { OK = 0, INVALID_CONFIGURATION = 9 };
static long n_hostalloc, n_register, n_instantiate, n_graphlaunch, n_launch, n_capture, fail_at;
static int capturing, last_error;
static char some[16], fatbin[16];
static double symbol[1 << 16];

long fake_count(const char *what) {
    if (!strcmp(what, "HostAlloc")) return n_hostalloc;
    if (!strcmp(what, "HostRegister")) return n_register;
    if (!strcmp(what, "Instantiate")) return n_instantiate;
    if (!strcmp(what, "GraphLaunch")) return n_graphlaunch;
    if (!strcmp(what, "Launch")) return n_launch;
    if (!strcmp(what, "Capture")) return n_capture;
    return -1;
}
void fake_fail_launch(long n) { fail_at = n; }

static int launch(void) {
    if (capturing) ++n_capture; else ++n_launch;
    if (fail_at > 0 && --fail_at == 0) return last_error = INVALID_CONFIGURATION;
    return OK;
}
int cudaLaunchKernel(void) { return launch(); }
int cudaLaunchKernelExC(void) { return launch(); }

void **__cudaRegisterFatBinary(void) { return (void **)fatbin; }
void __cudaRegisterFatBinaryEnd(void) {}
void __cudaUnregisterFatBinary(void) {}
void __cudaRegisterFunction(void) {}
void __cudaRegisterVar(void) {}
unsigned __cudaPushCallConfiguration(void) { return 0; }
int __cudaPopCallConfiguration(unsigned *grid, unsigned *block, size_t *smem, void **stream) {
    for (int d = 0; d < 3; ++d) grid[d] = block[d] = 1;
    *smem = 0;
    *stream = NULL;
    return OK;
}

int cudaMalloc(void **p, size_t n) { *p = calloc(1, n); return *p ? OK : 2; }
int cudaFree(void *p) { free(p); return OK; }
int cudaHostAlloc(void **p, size_t n) { ++n_hostalloc; *p = calloc(1, n); return *p ? OK : 2; }
int cudaFreeHost(void *p) { free(p); return OK; }
int cudaHostRegister(void) { ++n_register; return OK; }
int cudaHostUnregister(void) { return OK; }
int cudaMemcpy(void *d, const void *s, size_t n) { memcpy(d, s, n); return OK; }
int cudaMemcpyAsync(void *d, const void *s, size_t n) { memcpy(d, s, n); return OK; }
int cudaMemset(void *p, int v, size_t n) { memset(p, v, n); return OK; }
int cudaMemsetAsync(void *p, int v, size_t n) { memset(p, v, n); return OK; }
int cudaMemGetInfo(size_t *f, size_t *t) { *f = *t = (size_t)1 << 36; return OK; }

int cudaGetDevice(int *d) { *d = 0; return OK; }
int cudaDeviceGetAttribute(int *v) { *v = 148; return OK; }
int cudaDeviceSynchronize(void) { return OK; }
int cudaFuncSetAttribute(void) { return OK; }
int cudaGetSymbolAddress(void **p) { *p = symbol; return OK; }
static int entry(void) { return OK; }
int cudaGetDriverEntryPoint(const char *name, void **f, unsigned long long flags, int *result) {
    *f = (void *)entry;
    *result = 0;
    return OK;
}
const char *cudaGetErrorString(int e) { return e == OK ? "no error" : "error of the fake runtime"; }
int cudaGetLastError(void) { const int e = last_error; last_error = OK; return e; }
int cudaPeekAtLastError(void) { return last_error; }

int cudaStreamCreateWithFlags(void **s) { *s = some; return OK; }
int cudaStreamDestroy(void) { return OK; }
int cudaStreamSynchronize(void) { return OK; }
int cudaStreamWaitEvent(void) { return OK; }
int cudaEventCreate(void **e) { *e = some; return OK; }
int cudaEventCreateWithFlags(void **e) { *e = some; return OK; }
int cudaEventDestroy(void) { return OK; }
int cudaEventRecord(void) { return OK; }
int cudaEventSynchronize(void) { return OK; }
int cudaEventElapsedTime(float *ms) { *ms = 1.0f; return OK; }

int cudaStreamBeginCapture(void) { capturing = 1; return OK; }
int cudaStreamEndCapture(void *s, void **g) { capturing = 0; *g = some; return OK; }
int cudaGraphInstantiate(void **x) { ++n_instantiate; *x = some; return OK; }
int cudaGraphLaunch(void) { ++n_graphlaunch; return OK; }
int cudaGraphDestroy(void) { return OK; }
int cudaGraphExecDestroy(void) { return OK; }
