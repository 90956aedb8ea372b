// The built launch code (objects of gol_kernels.cu and gol_local.cu) over a CUDA runtime that only keeps accounts: every device has
// its own shared-memory limit per kernel (48 KB until raised there), and a
// launch above it fails, as on a GPU. Nothing is executed.
#include <cstdio>
#include <cstring>
#include <map>
#include <utility>

#include "gol_b200.h"
#include "../stencil-optimalizations_b200/csrc/gol_internal.h"

namespace {
constexpr size_t kDefaultLimit = 48 << 10, kOptin = 227 << 10;
int current = 0, launches = 0, set_calls = 0;
size_t largest = 0;   // dynamic shared memory of the launches
std::map<std::pair<int, const void*>, size_t> limit;

cudaError_t launch(const void* f, size_t smem) {
    auto it = limit.find({current, f});
    if (smem > (it == limit.end() ? kDefaultLimit : it->second)) return cudaErrorInvalidValue;
    if (smem > largest) largest = smem;
    ++launches;
    return cudaSuccess;
}
size_t pushed_smem = 0;
} // namespace

extern "C" {
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t smem, cudaStream_t) { pushed_smem = smem; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
    *g = dim3(1);
    *b = dim3(1);
    *smem = pushed_smem;
    *static_cast<cudaStream_t*>(s) = nullptr;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t smem, cudaStream_t) { return launch(f, smem); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) { return launch(f, c->dynamicSmemBytes); }
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3, dim3, void**, size_t smem, cudaStream_t) { return launch(f, smem); }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
    ++set_calls;
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) limit[{current, f}] = (size_t)v;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { *d = current; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { current = d; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrCooperativeLaunch ? 1 : (int)kOptin;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) { *s = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaPeekAtLastError() { return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMalloc(void**, size_t) { return cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void*) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t*) { return cudaErrorMemoryAllocation; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float*, cudaEvent_t, cudaEvent_t) { return cudaErrorMemoryAllocation; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
}

#define CHECK(c)                                                             \
    do {                                                                     \
        if (!(c)) {                                                          \
            std::printf("%s:%d: %s (device %d)\n", __FILE__, __LINE__, #c, current); \
            return 1;                                                        \
        }                                                                    \
    } while (0)

int main() {
    using namespace golb200;
    alignas(16) static uint32_t a[4], b[4];   // (never read or written)
    // One-generation passes: a row's CTAs have no warp past its end.
    for (int lanes : {1, 31, 32, 33, 64, 65, 96, 97, 128, 160, 224, 256, 257}) {
        RowsPlan p;
        CHECK(plan_rows(4 * lanes, 1000, 1, 0, 0, 148, &p) && p.once && p.threads <= 64);
        CHECK(p.nslices * p.threads == (lanes + 31) / 32 * 32);
    }
    for (int round = 0; round < 2; ++round) {
        for (int dev = 0; dev < 3; ++dev) {
            current = dev;
            const int calls = set_calls;
            RowsPlan p;
            // the row-pair pipeline, rows as they are and interleaved
            largest = 0;
            CHECK(plan_rows(512, 16384, 4, 0, 0, 148, &p) && p.pair);
            CHECK(launch_rows_pass(a, b, 512, 16384, 4, p, nullptr) == cudaSuccess);
            CHECK(launch_rows_pass(a, b, 512, 16384, 4, p, nullptr, 0, true) == cudaSuccess);
            CHECK(largest > kDefaultLimit);
            // a K-stage pass deep enough to need more than the default
            largest = 0;
            CHECK(plan_rows(512, 4096, 16, 0, 1, 148, &p) && !p.pair && !p.block);
            CHECK(launch_rows_pass(a, b, 512, 4096, 16, p, nullptr) == cudaSuccess);
            CHECK(largest > kDefaultLimit);
            // the change-tracking pass's dense form
            largest = 0;
            LocalPlan lp;
            CHECK(plan_local_tiles(512, 4096, 8, 0, 2, 148, 0, &lp) && !lp.block);
            CHECK(launch_local_pass(a, b, 512, 4096, 8, lp, LocalState{}, 0, nullptr) == cudaSuccess);
            CHECK(largest > kDefaultLimit);
            CHECK(round == 0 || set_calls == calls);   // raised once per device
        }
    }
    std::puts("ok");
    return 0;
}
