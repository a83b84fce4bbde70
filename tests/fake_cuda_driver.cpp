// The library's host code (libcuopus.cu) on a CUDA runtime made here, with two
// devices and no GPU: threads that reach it without a common lock, under
// ThreadSanitizer (tests/test_host_threads.py).  Exit status 0 when the launches
// are the ones that each device and size ask for; a data race makes it 66.
#include <atomic>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <thread>

#include <cuda_runtime.h>

#include "../include/cuopus.h"

// of kernels.cuh, which belongs to the kernel's translation units
namespace cuo {
cudaError_t decode_kernel_occupancy(int block, int width, int *blocks_per_sm);
cudaError_t resample_into(const int16_t *in, long long avail, long long n_out, float *out, cudaStream_t st);
}

static thread_local int t_dev = 0;
static thread_local dim3 t_grid, t_block;
static std::atomic<int> g_occupancy_calls{0};
static std::atomic<unsigned> g_grid[2];

enum { RS_BLOCKS = 5 };   // resampler blocks an SM on long inputs
static int sms_of(int dev) { return 148 - 16 * dev; }

extern "C" {
cudaError_t cudaGetDevice(int *d) { *d = t_dev; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int dev) { *v = sms_of(dev); return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaMalloc(void **p, size_t) { *p = malloc(256); return cudaSuccess; }
cudaError_t cudaFree(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpyToSymbolAsync(const void *, const void *, size_t, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s) { *s = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { *e = nullptr; return cudaSuccess; }
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t, void *) { t_grid = g; t_block = b; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *s, void *st)
{
    *g = t_grid;
    *b = t_block;
    *s = 0;
    *(void **)st = nullptr;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *, dim3 g, dim3, void **, size_t, cudaStream_t)
{
    g_grid[t_dev] = g.x;
    return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
}

cudaError_t cuo::decode_kernel_occupancy(int, int, int *per_sm)
{
    g_occupancy_calls++;
    *per_sm = 4;
    return cudaSuccess;
}

int main()
{
    const long long n = 40000000;
    int16_t in = 0;
    float out = 0;
    std::atomic<int> failed{0};
    // a float server's thread, on device 0, and a program's own calls on device 1
    std::thread server([&] {
        t_dev = 0;
        for (int i = 0; i < 100; i++)
            if (cuo::resample_into(&in, 3 * n, n, &out, nullptr) != cudaSuccess) failed++;
    });
    std::thread calls([&] {
        t_dev = 1;
        cuopus_release_workspaces();
        for (int i = 0; i < 100; i++)
            if (cuopus_warmup(nullptr, 0) || cuopus_resample48to16(&in, 3 * n, n, &out, nullptr, nullptr, 0)) failed++;
    });
    server.join();
    calls.join();
    for (int d = 0; d < 2; d++) {
        const unsigned want = sms_of(d) * RS_BLOCKS;
        if (g_grid[d] != want) printf("device %d: grid %u, not %u\n", d, g_grid[d].load(), want), failed++;
    }
    // one set of occupancies: the decoder ran on device 1 only
    if (g_occupancy_calls != 24) printf("%d occupancy queries, not 24\n", g_occupancy_calls.load()), failed++;
    // the form of the resampler: tiles of 768 outputs until four blocks an SM have one of 2304
    t_dev = 0;
    for (const long long tiles : {3ll * 148, 4ll * 148 - 1, 4ll * 148}) {
        const long long outs = 2304 * tiles;
        if (cuopus_resample48to16(&in, 3 * outs, outs, &out, nullptr, nullptr, 0)) failed++;
        const unsigned want = tiles < 4 * 148 ? 5 * 148 : (unsigned)tiles;
        if (g_grid[0] != want) printf("%lld outputs: grid %u, not %u\n", outs, g_grid[0].load(), want), failed++;
    }
    return failed ? 1 : 0;
}
