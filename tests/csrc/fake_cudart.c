/* Test-only stand-in for the CUDA runtime on a machine without a GPU: memory is host memory, copies are made, launches do
 * nothing. fake_fail_next_wait(): at the first stream synchronisation after the next launch that kernel is taken to have given
 * up a bounded wait, so the error word of every page-locked scratch block (64 KB, the last word but one) is set.
 * fake_no_scratch(1): no such block can be had, and the runtime's last error says so until it is asked for. */
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#define SCRATCH_BYTES 65536
#define BLOCKS 64
static uint64_t* blocks[BLOCKS];
static int fail_next, launched, allocated, freed, no_scratch, last_error, synchronised;
static unsigned device_flags;

void fake_fail_next_wait(void) { fail_next = 1; launched = 0; }
void fake_no_scratch(int on) { no_scratch = on; }
void fake_device_flags(unsigned flags) { device_flags = flags; }
int fake_synchronised(void) { return synchronised; }
int fake_scratch_allocated(void) { return allocated; }
int fake_scratch_freed(void) { return freed; }

static int get(void** p, size_t n) {
    *p = NULL;
    return posix_memalign(p, 256, n ? n : 1) == 0 ? (memset(*p, 0, n), 0) : 2;
}
int cudaHostAlloc(void** p, size_t n, unsigned flags) {
    if (no_scratch && n == SCRATCH_BYTES) return *p = NULL, last_error = 2;
    int rc = get(p, n);
    if (rc == 0 && n == SCRATCH_BYTES)
        for (int i = 0; i < BLOCKS; i++)
            if (!blocks[i]) {
                blocks[i] = *p;
                allocated++;
                break;
            }
    return rc;
}
int cudaFreeHost(void* p) {
    for (int i = 0; i < BLOCKS; i++)
        if (p && blocks[i] == p) {
            blocks[i] = NULL;
            freed++;
        }
    free(p);
    return 0;
}
int cudaStreamSynchronize_ptsz(void* st) {
    synchronised++;
    for (int i = 0; fail_next && launched && i < BLOCKS; i++)
        if (blocks[i]) blocks[i][SCRATCH_BYTES / 8 - 2] = 1;
    if (launched) fail_next = 0;
    return 0;
}
int cudaMallocHost(void** p, size_t n) { return get(p, n); }
int cudaMalloc(void** p, size_t n) { return get(p, n); }
int cudaMallocAsync_ptsz(void** p, size_t n, void* st) { return get(p, n); }
int cudaFree(void* p) { free(p); return 0; }
int cudaFreeAsync_ptsz(void* p, void* st) { free(p); return 0; }
int cudaMemcpyAsync_ptsz(void* d, const void* s, size_t n, int kind, void* st) { memcpy(d, s, n); return 0; }
int cudaMemsetAsync_ptsz(void* d, int v, size_t n, void* st) { memset(d, v, n); return 0; }
int cudaLaunchKernel_ptsz(void) { launched = 1; return 0; }
int cudaLaunchKernelExC_ptsz(void) { launched = 1; return 0; }
int cudaFuncSetAttribute(void) { return 0; }
int cudaGetDeviceFlags(unsigned* f) { *f = device_flags; return 0; }
int cudaGetDevice(int* d) { *d = 0; return 0; }
int cudaSetDevice(int d) { return 0; }
int cudaGetDeviceCount(int* n) { *n = 1; return 0; }
int cudaGetDeviceProperties_v2(void* p, int d) { return 0; }
int cudaDeviceGetAttribute(int* v, int attr, int d) { *v = 148; return 0; }
int cudaDeviceGetDefaultMemPool(void** p, int d) { *p = NULL; return 0; }
int cudaMemPoolSetAttribute(void) { return 0; }
int cudaMemGetInfo(size_t* f, size_t* t) { *f = *t = (size_t)1 << 34; return 0; }
int cudaDeviceSynchronize(void) { return 0; }
int cudaGetLastError(void) {
    int rc = last_error;
    last_error = 0;
    return rc;
}
int cudaPeekAtLastError(void) { return 0; }
int cudaEventCreate(void** e) { *e = NULL; return 0; }
int cudaEventCreateWithFlags(void** e, unsigned f) { *e = NULL; return 0; }
int cudaEventDestroy(void* e) { return 0; }
int cudaEventElapsedTime(float* ms, void* a, void* b) { *ms = 0; return 0; }
int cudaEventQuery(void* e) { return 0; }
int cudaEventRecord_ptsz(void* e, void* st) { return 0; }
int cudaEventSynchronize(void* e) { return 0; }
void** __cudaRegisterFatBinary(void* f) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void** h) {}
void __cudaUnregisterFatBinary(void** h) {}
void __cudaRegisterFunction(void) {}
void __cudaRegisterVar(void) {}
unsigned __cudaPushCallConfiguration(void) { return 0; }
int __cudaPopCallConfiguration(void* grid, void* block, size_t* smem, void** st) { *smem = 0; *st = NULL; return 0; }
