// gol_engine.cu over a CUDA runtime made of host memory, in which chosen calls
// fail. A pass adds one to every word (of the grid as it is: interleaved words
// stand for themselves XOR kInter), so a fetched word tells the generations it
// has seen and whether it came out interleaved.
//
//   engine_fake_cuda instantiate   the chunk graph cannot be instantiated
//   engine_fake_cuda launch        the second chunk cannot be launched
//   engine_fake_cuda restore       the grid cannot be restored afterwards
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <vector>

#include "gol_b200.h"
#include "../stencil-optimalizations_b200/csrc/gol_internal.h"

namespace {

constexpr uint32_t kInter = 0xA5A5A5A5u;
bool fail_instantiate = false, fail_restore = false;
int graph_launches_left = -1;   // < 0: no limit
bool capturing = false;
std::vector<std::function<void()>> captured, graph;

void enqueue(std::function<void()> f) {
    if (capturing)
        captured.push_back(std::move(f));
    else
        f();
}

} // namespace

extern "C" {
cudaError_t cudaMalloc(void** p, size_t n) { return (*p = std::malloc(n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorName(cudaError_t) { return "fake"; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = reinterpret_cast<cudaStream_t>(8); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { capturing = true; captured.clear(); return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    capturing = false;
    *g = reinterpret_cast<cudaGraph_t>(8);
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
    if (fail_instantiate) return cudaErrorMemoryAllocation;
    graph = captured;
    *x = reinterpret_cast<cudaGraphExec_t>(8);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) {
    if (graph_launches_left == 0) return cudaErrorLaunchOutOfResources;
    if (graph_launches_left > 0) --graph_launches_left;
    for (auto& f : graph) f();
    return cudaSuccess;
}
}

namespace golb200 {

int device_sm_count(int) { return 148; }
int best_depth(int, int, int) { return 4; }
bool plan_rows(int, int, int, int, int, int, RowsPlan* p, bool) {
    *p = RowsPlan{};
    p->wpl = 4;
    p->pair = true;
    return true;
}
cudaError_t launch_rows_pass(const uint32_t* src, uint32_t* dst, int W, int Y, int, const RowsPlan&,
                             cudaStream_t, int, bool interleaved) {
    enqueue([=] {
        const uint32_t x = interleaved ? kInter : 0u;
        for (int i = 0; i < W * Y; ++i) dst[i] = ((src[i] ^ x) + 1u) ^ x;
    });
    return cudaSuccess;
}
cudaError_t launch_interleave(uint32_t* grid, int W, int Y, bool back, cudaStream_t) {
    if (back && fail_restore) return cudaErrorLaunchFailure;
    enqueue([=] { for (int i = 0; i < W * Y; ++i) grid[i] ^= kInter; });
    return cudaSuccess;
}
void host_copy(void* d, const void* s, size_t n, bool) { std::memcpy(d, s, n); }

// never reached by a dense run
bool plan_resident(int, int, int, int, ResidentPlan*) { std::abort(); }
cudaError_t launch_resident(const uint32_t*, uint32_t*, int, int, long long, const ResidentPlan&,
                            unsigned long long*, int*, int*, cudaStream_t, long long) { std::abort(); }
bool plan_local_tiles(int, int, int, int, int, int, int, LocalPlan*) { std::abort(); }
cudaError_t launch_local_pass(const uint32_t*, uint32_t*, int, int, int, const LocalPlan&,
                              const LocalState&, int, cudaStream_t) { std::abort(); }
cudaError_t reset_local(const LocalPlan&, const LocalState&, int, bool, cudaStream_t) { std::abort(); }

} // namespace golb200

#define CHECK(c)                                                             \
    do {                                                                     \
        if (!(c)) {                                                          \
            std::printf("%s:%d: %s\n", __FILE__, __LINE__, #c);              \
            return 1;                                                        \
        }                                                                    \
    } while (0)

int main(int argc, char** argv) {
    const char* what = argc > 1 ? argv[1] : "";
    constexpr int kWords = 4 * 8;
    std::vector<uint32_t> in(kWords), out(kWords);
    for (int i = 0; i < kWords; ++i) in[i] = 1000u * (uint32_t)i;
    gol_config cfg;
    gol_config_init(&cfg, 128, 8);
    gol_engine* e = nullptr;
    CHECK(gol_create(&e, &cfg) == GOL_OK);
    CHECK(gol_set_input_words(e, in.data(), 128, 8, 32) == GOL_OK);
    CHECK(gol_init(e) == GOL_OK);
    uint32_t seen = 0;   // passes that the grid has seen
    if (!std::strcmp(what, "instantiate")) {
        fail_instantiate = true;
        CHECK(gol_run(e, 4 * 50) == GOL_E_CUDA);
        CHECK(gol_performed(e) == 0);
        fail_instantiate = false;
    } else if (!std::strcmp(what, "launch")) {
        graph_launches_left = 1;
        CHECK(gol_run(e, 4 * 50) == GOL_E_CUDA);
        CHECK(gol_performed(e) == 4 * 16);
        seen = 16;
        graph_launches_left = -1;
    } else if (!std::strcmp(what, "restore")) {
        fail_restore = true;
        CHECK(gol_run(e, 4 * 50) == GOL_E_CUDA);
        // the grid is lost: nothing hands out its words
        CHECK(gol_device_grid(e) == nullptr);
        CHECK(gol_run(e, 4) == GOL_E_STATE);
        CHECK(gol_finalize(e) == GOL_E_STATE);
        CHECK(gol_fetch_words(e, out.data(), 32) == GOL_E_STATE);
        fail_restore = false;
        CHECK(gol_set_input_words(e, in.data(), 128, 8, 32) == GOL_OK);
        CHECK(gol_init(e) == GOL_OK);
    } else {
        return 2;
    }
    CHECK(gol_run(e, 4 * 50) == GOL_OK);   // and the engine goes on
    CHECK(gol_finalize(e) == GOL_OK);
    CHECK(gol_fetch_words(e, out.data(), 32) == GOL_OK);
    for (int i = 0; i < kWords; ++i) CHECK(out[i] == in[i] + seen + 50u);
    gol_destroy(e);
    std::puts("ok");
    return 0;
}
