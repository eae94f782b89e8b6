// fake_cuda.cpp — a CUDA runtime and kernel launchers that run nothing, linked
// with the library's host sources by test_host_runtime.py: device memory with a
// settable limit, launches that can be made to fail, and the order in which
// streams, events and host waits put the launches.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <vector>

#include "kernels.h"
#include "powmod_kernels.h"
#include "word.h"

namespace {

using Clock = std::map<const void*, long>;  // launches per stream that are known to be done

struct State {
    std::mutex mu;
    size_t limit = SIZE_MAX, used = 0;
    std::map<void*, size_t> sizes;
    Clock host, heads, mark;  // waited for; issued; issued before the mark
    std::map<const void*, Clock> streams;
    long fail_at = -1;       // launches until one fails
    bool marked = false;
    int unordered = 0;       // launches after the mark not ordered after all before it
    long word = 0, fp64 = 0;
    bool coarse = false;  // the lengths the last product was offered
    std::vector<const void*> copied;  // both ends of every copy since the last question
    cudaError_t last = cudaSuccess;
};
State& S() {
    static State s;
    return s;
}
void join(Clock& a, const Clock& b) {
    for (const auto& kv : b) a[kv.first] = std::max(a[kv.first], kv.second);
}
struct Event {
    Clock c;
};

// kind: 0 neither, 1 word product, 2 FP64 passes
cudaError_t launched(cudaStream_t st, int kind) {
    State& s = S();
    std::lock_guard<std::mutex> lk(s.mu);
    if (s.fail_at >= 0 && s.fail_at-- == 0) return cudaErrorLaunchOutOfResources;
    Clock& c = s.streams[st];
    join(c, s.host);
    if (s.marked)
        for (const auto& kv : s.mark)
            if (c[kv.first] < kv.second) {
                s.unordered++;
                break;
            }
    c[st] = ++s.heads[st];
    if (kind) (kind == 1 ? s.word : s.fp64)++;
    return cudaSuccess;
}

cudaError_t take(void** p, size_t n) {
    State& s = S();
    std::lock_guard<std::mutex> lk(s.mu);
    if (s.used + n > s.limit) return s.last = cudaErrorMemoryAllocation;
    *p = std::aligned_alloc(256, (n + 255) / 256 * 256);
    s.used += n;
    s.sizes[*p] = n;
    return cudaSuccess;
}
cudaError_t give(void* p) {
    if (!p) return cudaSuccess;
    State& s = S();
    std::lock_guard<std::mutex> lk(s.mu);
    s.used -= s.sizes[p];
    s.sizes.erase(p);
    std::free(p);
    return cudaSuccess;
}
cudaError_t handle(void** p) {
    *p = std::malloc(16);
    return cudaSuccess;
}

}  // namespace

extern "C" {

// ---- the tests' side
void fake_limit(size_t free_bytes) { S().limit = free_bytes == SIZE_MAX ? SIZE_MAX : S().used + free_bytes; }
size_t fake_used() { return S().used; }
void fake_fail_at(long n) { S().fail_at = n; }
void fake_mark() {
    S().mark = S().heads;
    S().marked = true;
    S().unordered = 0;
}
int fake_unordered() { return S().unordered; }
void fake_counts(long* word, long* fp64) {
    *word = S().word;
    *fp64 = S().fp64;
    S().word = S().fp64 = 0;
}
int fake_coarse() { return S().coarse; }
// how many of the pointers a copy started at, since the last call
int fake_copied(const void* const* p, int n) {
    int k = 0;
    for (int i = 0; i < n; i++) k += std::count(S().copied.begin(), S().copied.end(), p[i]) > 0;
    S().copied.clear();
    return k;
}

// ---- runtime
cudaError_t cudaMalloc(void** p, size_t n) { return take(p, n); }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return take(p, n); }
cudaError_t cudaFree(void* p) { return give(p); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return give(p); }
cudaError_t cudaMallocHost(void** p, size_t n) {
    *p = std::aligned_alloc(256, (n + 255) / 256 * 256);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMallocHost(p, n); }
cudaError_t cudaFreeHost(void* p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    {
        std::lock_guard<std::mutex> lk(S().mu);
        S().copied.insert(S().copied.end(), {d, s});
    }
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t) { return cudaMemcpy(d, s, n, k); }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
    std::memset(a, 0, sizeof *a);
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* p, unsigned) { return handle((void**)p); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t st) {
    State& s = S();
    std::lock_guard<std::mutex> lk(s.mu);
    join(s.host, s.streams[st]);
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
    std::lock_guard<std::mutex> lk(S().mu);
    S().host = S().heads;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = (cudaEvent_t) new Event;
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) {
    std::lock_guard<std::mutex> lk(S().mu);
    ((Event*)e)->c = S().streams[st];
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    std::lock_guard<std::mutex> lk(S().mu);
    join(S().host, ((Event*)e)->c);
    return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 0;
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t e, unsigned) {
    std::lock_guard<std::mutex> lk(S().mu);
    join(S().streams[st], ((Event*)e)->c);
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c) {
    *c = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { return handle((void**)g); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) { return handle((void**)x); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaLaunchHostFunc(cudaStream_t, cudaHostFn_t fn, void* p) {
    fn(p);
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = S().last;
    S().last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetDeviceCount(int* n) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) {
    std::memset(p, 0, sizeof *p);
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
    *v = 148;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t*, int) { return cudaErrorNotSupported; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** p, unsigned long long, cudaDriverEntryPointQueryResult*) {
    *p = nullptr;
    return cudaErrorNotSupported;
}

}  // extern "C"

// ---- kernel launchers
namespace nbg {

cudaError_t kernels_init(double, double) { return cudaSuccess; }
int kernels_smem_optin() { return 227 * 1024; }
cudaError_t kernels_take_faults(unsigned* n) {
    *n = 0;
    return cudaSuccess;
}
cudaError_t kernels_binary_version(int* v) {
    *v = 100;
    return cudaSuccess;
}
cudaError_t launch_jobs(int, const DProd*, const DPlan*, const JobSrc&, int64_t, size_t, int, cudaStream_t st, bool) {
    return launched(st, 2);
}
cudaError_t launch_qcount(const DProd*, const Job*, const QLaunch*, int, int64_t, uint32_t*, cudaStream_t) { return cudaSuccess; }
cudaError_t queue_grid(size_t, int* g) {
    *g = 148;
    return cudaSuccess;
}
cudaError_t launch_queue(const DProd*, const DPlan*, const Job*, const QLaunch*, int, QState*, uint32_t*, const uint32_t*,
                         size_t, int, int, cudaStream_t) {
    return cudaSuccess;
}
cudaError_t launch_expand(const ExpandEntry*, int, Job*, int64_t, cudaStream_t st) { return launched(st, 0); }
cudaError_t launch_twiddle(double*, int, int64_t, int64_t, const double*, const double*, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_pack(double*, int64_t, const uint64_t*, int64_t, int, int64_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_pointwise(double*, const double*, int64_t, int, cudaStream_t) { return cudaSuccess; }
cudaError_t launch_topbits(const DProd* p, int64_t n, int64_t* bits, cudaStream_t st) {
    for (int64_t k = 0; k < n; k++) {
        bits[2 * k] = 64 * p[k].m;
        bits[2 * k + 1] = 64 * p[k].n;
    }
    return launched(st, 0);
}

// the real lengths, without their splits into passes
bool word_shape(int64_t nconv, WordShape& s, bool coarse) {
    S().coarse = coarse;
    int64_t best = INT64_MAX;
    auto take = [&](int odd, int k, int set) {
        const int64_t N = (int64_t)odd << k;
        if (N < nconv || N >= best) return;
        best = N;
        const bool small = k <= 11 && WPR * N <= 16 * 1024;
        const int lm = small || k < 12 ? k : 12;
        s = WordShape{(int32_t)N, odd, k - lm, 0, lm, small, set};
    };
    for (int odd : {1, 3, 5, 7})
        for (int k = 6; k <= WORD_MAX_LOG2 && ((int64_t)odd << k) <= 7 << 19; k++) take(odd, k, 0);
    for (int k = 22; k <= 25; k++) take(1, k, 2);
    for (int k = 21; k <= 23; k++) take(3, k, 1);
    return best != INT64_MAX;
}
cudaError_t word_init() { return cudaSuccess; }
cudaError_t launch_word(int kind, int, const DProd*, const WSeg*, int, const int32_t*, int64_t, cudaStream_t st) {
    return launched(st, kind == JK_WCARRY ? 0 : 1);  // carries between tiles: of either
}
cudaError_t launch_word_one(int, int, const DProd&, int64_t, cudaStream_t st) { return launched(st, 1); }
int64_t word_ctas(int, const WordShape&, int, int64_t) { return 1; }
size_t word_table_bytes(int set, int odd, int L) { return sizeof(uint64_t) * ((size_t)word_np(set) * odd << L); }
cudaError_t word_build_tables(int, int, int, void*, void*, cudaStream_t) { return cudaSuccess; }
void word_scales(const WordShape&, uint32_t* out) { std::memset(out, 0, sizeof(uint32_t) * WPR_MAX); }
cudaError_t pm_chain_init() { return cudaSuccess; }

}  // namespace nbg
