// The runtime's host side against a CUDA runtime that lives on the CPU (no GPU): device memory is host
// memory, and what is enqueued on a stream runs when that stream is waited for, not before.  A wait can
// call back first, as another thread would run meanwhile.  Prints "ok <name>" or "FAILED <name>" per check.
//
// Built by tests/test_host_runtime.py from this file and the runtime's sources.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <thread>
#include <vector>

#include "ml_pipeline.hpp"
#include "ml_runtime.hpp"

using namespace mlg;

namespace {
std::map<cudaStream_t, std::vector<std::function<void()>>> g_queue;
std::function<void(cudaStream_t)> g_on_wait;  // called once, at the next wait
int g_failed = 0;
void run(cudaStream_t s) {
    auto work = std::move(g_queue[s]);
    g_queue[s].clear();
    for (auto& f : work) f();
}
void check(const char* name, bool ok) {
    printf("%s %s\n", ok ? "ok" : "FAILED", name);
    g_failed += !ok;
}
}  // namespace

extern "C" {
cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "error"; }
cudaError_t cudaMalloc(void** p, size_t n) { return *p = aligned_alloc(256, (n + 255) / 256 * 256), cudaSuccess; }
cudaError_t cudaFree(void* p) { return free(p), cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return *p = malloc(n), cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return free(p), cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    static uintptr_t next = 0;
    return *s = (cudaStream_t)(++next), cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    if (auto f = std::move(g_on_wait)) {
        g_on_wait = nullptr;
        f(s);
    }
    run(s);
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c) { return *c = cudaStreamCaptureStatusNone, cudaSuccess; }
cudaError_t cudaDeviceSynchronize() {
    for (auto& q : g_queue) run(q.first);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    g_queue[st].push_back([=] { memcpy(d, s, n); });
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
    g_queue[st].push_back([=] { memset(d, v, n); });
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {  // every caller's buffer is pageable
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 0, cudaSuccess; }
}

namespace {
constexpr int64_t kRows = 100'000;

ml_column host_column(int dtype, const void* data) {
    ml_column c{};
    c.dtype = dtype;
    c.encoding = ML_ENC_PLAIN;
    c.location = ML_LOC_HOST;
    c.len = kRows;
    c.data = data;
    return c;
}
bool all(const DevColumn& c, int32_t v) {
    for (int64_t i = 0; i < kRows; i++)
        if (((const int32_t*)c.dptr())[i] != v) return false;
    return true;
}

// Pageable columns that grow: the second needs a larger staging block while the first one's copy still
// reads the old block, and another thread uploads its own column just then.
void staging_grows() {
    Ctx ctx(0, 0, 0);
    const cudaStream_t a = ctx.new_stream(), b = ctx.new_stream();
    std::vector<int32_t> ones(kRows, 1), twos(kRows, 2);
    std::vector<double> wide(kRows, 0.5);
    Staging sa(&ctx), sb(&ctx);
    std::unique_ptr<DevColumn> mine, other, second;
    mine = stage_column(&ctx, host_column(ML_TYPE_INT32, ones.data()), kRows, a, sa, nullptr);
    g_on_wait = [&](cudaStream_t) { other = stage_column(&ctx, host_column(ML_TYPE_INT32, twos.data()), kRows, b, sb, nullptr); };
    second = stage_column(&ctx, host_column(ML_TYPE_FLOAT64, wide.data()), kRows, a, sa, nullptr);
    cudaDeviceSynchronize();
    check("a block that a copy reads is not handed out when its owner takes a larger one", all(*mine, 1) && other && all(*other, 2));
}

// A staging buffer that goes away before its stream is waited for.
void staging_dies() {
    Ctx ctx(0, 0, 0);
    const cudaStream_t a = ctx.new_stream(), b = ctx.new_stream();
    std::vector<int32_t> ones(kRows, 1), twos(kRows, 2);
    std::unique_ptr<DevColumn> mine, other;
    {
        Staging sa(&ctx);
        mine = stage_column(&ctx, host_column(ML_TYPE_INT32, ones.data()), kRows, a, sa, nullptr);
    }
    Staging sb(&ctx);
    other = stage_column(&ctx, host_column(ML_TYPE_INT32, twos.data()), kRows, b, sb, nullptr);
    cudaDeviceSynchronize();
    check("a block that a copy reads is not handed out when its owner goes", all(*mine, 1) && all(*other, 2));
}

// An allocation that the budget refuses while work on buffers that the error gives back is still in flight.
void errors_wait() {
    Ctx ctx(0, 64 << 20, 0);
    const cudaStream_t a = ctx.new_stream(), b = ctx.new_stream();
    bool refused = false;
    try {
        const StreamScope outer(a);
        const StreamScope scope(b);
        DevBuf mine(&ctx, 1 << 20, nullptr);
        cudaMemsetAsync(mine.get(), 1, 1 << 20, a);
        Reservation res(&ctx, "Test");
        DevBuf large(&ctx, 128 << 20, &res);
    } catch (const MlError& e) {
        refused = e.code == ML_ERR_BUDGET;
    }
    DevBuf other(&ctx, 1 << 20, nullptr);  // the next caller's, perhaps the same memory
    memset(other.get(), 2, 1 << 20);
    cudaDeviceSynchronize();
    bool kept = true;
    for (size_t i = 0; i < 1 << 20; i++) kept = kept && other.get<uint8_t>()[i] == 2;
    check("an error waits for the work on the buffers it gives back", refused && kept);
}
}  // namespace

int main() {
    staging_grows();
    staging_dies();
    errors_wait();
    return g_failed ? 1 : 0;
}
