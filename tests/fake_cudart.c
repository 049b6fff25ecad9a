/* A CUDA runtime without a device, as far as the launchers of this package use it: it knows how much dynamic shared memory each
   kernel was allowed on each device and refuses a launch that asks for more, as the real one does. */
#include <stddef.h>
#include <string.h>

enum { DEVICES = 128, KERNELS = 4096, OK = 0, INVALID = 1 };
static int device_now, last_error;
static const void* kernels[KERNELS];
static int n_kernels, allowed[KERNELS][DEVICES], early_at[KERNELS];
static void* handle;
int fake_launches, fake_last_grid, fake_last_early, fake_attribute_calls;

struct config { unsigned gx, gy, gz, bx, by, bz; size_t smem; void* stream; void* attrs; unsigned n; };

static int place(const void* f) {
    for (int i = 0; i < n_kernels; ++i) if (kernels[i] == f) return i;
    kernels[n_kernels] = f;
    return n_kernels++;
}
void fake_set_device(int d) { device_now = d; }
/* a device with an odd number holds half as many multiprocessors */
static int sms(int d) { return d % 2 ? 74 : 148; }

int cudaGetDevice(int* d) { *d = device_now; return OK; }
int cudaDeviceGetAttribute(int* v, int what, int d) { *v = what == 16 ? sms(d) : 0; return OK; }
int cudaGetLastError(void) { int e = last_error; last_error = OK; return e; }
int cudaFuncSetAttribute(const void* f, int what, int v) {
    ++fake_attribute_calls;
    if (v > 227 * 1024) return INVALID;
    if (what == 8) allowed[place(f)][device_now] = v;
    return OK;
}
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void* f, int threads, size_t smem, unsigned flags) {
    (void)f; (void)threads; (void)flags;
    *n = smem ? (int)(227 * 1024 / smem) : 16;
    return OK;
}
int cudaLaunchKernelExC(const struct config* c, const void* f, void** args) {
    const int most = allowed[place(f)][device_now];
    if (c->smem > (size_t)(most > 48 * 1024 ? most : 48 * 1024)) return last_error = INVALID;
    ++fake_launches;
    fake_last_grid = (int)c->gx;
    fake_last_early = *(int*)args[early_at[place(f)]];
    return OK;
}
int cudaLaunchKernel(const void* f, unsigned gx, unsigned gy, unsigned gz, unsigned bx, unsigned by, unsigned bz, void** a, size_t s, void* st) {
    (void)f; (void)gx; (void)gy; (void)gz; (void)bx; (void)by; (void)bz; (void)a; (void)s; (void)st;
    return INVALID;
}
void** __cudaRegisterFatBinary(void* p) { (void)p; return &handle; }
void __cudaRegisterFatBinaryEnd(void** h) { (void)h; }
void __cudaUnregisterFatBinary(void** h) { (void)h; }
void __cudaRegisterFunction(void** h, const char* host, char* dev, const char* name, int lim, void* a, void* b, void* c, void* d, int* e) {
    early_at[place(host)] = strstr(name, "wide") ? 12 : 14;      /* the last argument of the plain product's kernels */
    (void)h; (void)dev; (void)lim; (void)a; (void)b; (void)c; (void)d; (void)e;
}
int __cudaPopCallConfiguration(void* g, void* b, size_t* s, void* st) { (void)g; (void)b; (void)s; (void)st; return INVALID; }
unsigned __cudaPushCallConfiguration(void) { return 1; }
