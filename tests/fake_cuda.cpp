// A CUDA runtime without a device, for CPU tests of the library's host code (es_abi.cu, es_cascade.cu
// and es_mitm.cu linked against this file in place of libcudart and of the scan kernels' dispatch).
//
// Work on a stream runs as late as the runtime's rules allow: an operation waits in its stream's queue
// until the host synchronises that stream, and no stream runs because of another one (the library's
// streams are non-blocking ones).  So a kernel whose input was written on another stream, without
// the host waiting for that stream in between, finds memory that was never written (0xcd).  A launch
// looks, when its stream runs, at what it was given and counts what is wrong:
//   fake_faults()   launches while writes wait on the legacy default stream, work counters that are
//                   not zero, shared memory above what the kernel may use
//   fake_launches() launches that ran; fake_tables(), fake_layout() the inner
//                   tables and the layout of the last scan
//   fake_fail_alloc(n)  the library's n-th host allocation from now on throws std::bad_alloc (0: none);
//                   returns how far an earlier request still was from failing (0: it has failed)
//   (device allocations of 32 GB and more are refused)
//   fake_live()     device and pinned allocations that have not been freed
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <new>
#include <string>
#include <vector>

#include "../include/es_gb300.h"
#include "../erdos-selfridge_gb300/csrc/es_internal.h"

namespace {
std::map<cudaStream_t, std::vector<std::function<void()>>> queues;
int faults = 0, launches = 0, live = 0, tables = 0, layouts = 0;
thread_local long fail_in = 0;
thread_local int inside = 0;   // in this file: its own allocations neither count nor fail
struct Inside {
    Inside() { ++inside; }
    ~Inside() { --inside; }
};
uintptr_t next_handle = 16;

void run(cudaStream_t s) {
    const Inside here;
    auto q = std::move(queues[s]);
    queues[s].clear();
    for (auto& f : q) f();
}
template <class F>
void put(cudaStream_t s, const F& f) {
    const Inside here;
    queues[s].push_back(f);
}

cudaError_t copy(void* dst, const void* src, size_t n, cudaMemcpyKind kind, cudaStream_t s) {
    const Inside here;
    if (kind == cudaMemcpyHostToDevice) {   // the host buffer is read now, the device written later
        std::vector<unsigned char> b((const unsigned char*)src, (const unsigned char*)src + n);
        put(s, [=] { memcpy(dst, b.data(), n); });
    } else {
        put(s, [=] { memcpy(dst, src, n); });
    }
    return cudaSuccess;
}
// What a launch on stream s finds, apart from its arguments.
void launched(cudaStream_t s) {
    const Inside here;
    if (s != nullptr && !queues[nullptr].empty()) ++faults;
    ++launches;
}
}  // namespace

extern "C" {
int fake_faults() { return faults; }
int fake_launches() { return launches; }
int fake_live() { return live; }
int fake_tables() { return tables; }
int fake_layout() { return layouts; }
long fake_fail_alloc(long n) { const long left = fail_in; fail_in = n; return left; }
void fake_drain() { for (auto& q : queues) run(q.first); }

cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrComputeCapabilityMajor ? 10 : a == cudaDevAttrComputeCapabilityMinor ? 3
       : a == cudaDevAttrMultiProcessorCount ? 152 : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448 : 0;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) { memset(p, 0, sizeof *p); return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) {
    *p = n < 32ull << 30 ? aligned_alloc(256, (n + 511) / 256 * 256) : nullptr;
    if (*p && n <= (64u << 20)) memset(*p, 0xcd, n);
    live += *p != nullptr;
    return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFree(void* p) { live -= p != nullptr; free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned f) {
    if (f != cudaStreamNonBlocking) ++faults;
    *s = (cudaStream_t)(next_handle += 16);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { run(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { run(s); return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) { *s = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)(next_handle += 16); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { for (auto& q : queues) if (q.first) run(q.first); return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
    static unsigned char scratch[1 << 17];
    *p = scratch;
    return cudaSuccess;
}
// Pageable copies to the device return when the host buffer has been read: after what waits on the
// stream, before the device memory is written.
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) {
    run(nullptr);
    copy(d, s, n, k, nullptr);
    if (k != cudaMemcpyHostToDevice) run(nullptr);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) { return copy(d, s, n, k, st); }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t s) {
    put(s, [=] { memset(d, v, n); });
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { return cudaMemsetAsync(d, v, n, nullptr); }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }

// kernel launches by <<< >>> (the MITM kernel: 16 KB of static shared memory, no opt-in to more than
// 48 KB): noted, not run
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t smem, struct CUstream_st* s) {
    if (smem + 16384u > 49152u) ++faults;
    launched(s);
    return 1;
}
cudaError_t __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return cudaErrorNotSupported; }
cudaError_t __cudaGetKernel(cudaKernel_t*, const void*) { return cudaErrorNotSupported; }
cudaError_t __cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t) { return cudaErrorNotSupported; }
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
}

// ---- the scan kernels' dispatch ----------------------------------------------------------------
int es_scan_prepare(int) { return 0; }
int es_scan_occupancy(int, int, uint32_t, uint32_t, int threads, int smem, int* n) {
    *n = threads <= 640 && smem <= 231424 ? 1 : 0;
    return 0;
}
int es_launch_scan(const EsLaunch& L, int layout, int, uint32_t, int, void* stream) {
    cudaStream_t s = (cudaStream_t)stream;
    launched(s);
    tables = (int)L.mask_filters;
    layouts = layout;
    EsLaunch l = L;
    if (!l.items) put(s, [=] {
        if (!l.surv && l.surv_cap) ++faults;   // records would go to a null pointer
        if (*l.unit_counter != 0 || *l.ctas_done != 0) ++faults;
        // the plan's header and tables are there
        const EsInst& I = *l.item0.inst;
        if (I.n_filters > ES_MAX_ENTRIES || I.small_bytes == 0 || I.r0 == 0 || I.r0 > 65535) { ++faults; return; }
        if (I.small != l.small || (layout == ES_LAYOUT_PROD && I.tab_words != l.tab_words)) ++faults;
        if (l.item0.list)
            for (uint64_t i = l.item0.o_begin; i < l.item0.o_end; ++i) if (l.item0.list[i] >= I.n_outer) { ++faults; break; }
    });
    return 0;
}
int es_launch_min(const es_survivor*, const unsigned long long*, uint64_t, const EsItem*, uint32_t, const unsigned long long*,
                  unsigned long long*, void* stream) {
    launched((cudaStream_t)stream);
    return 0;
}
int es_launch_int_peak(unsigned long long*, int, int, int, int, void*) { return 0; }

// ---- host allocations that fail on request ------------------------------------------------------
static bool fails() { return !inside && fail_in > 0 && --fail_in == 0; }
void* operator new(size_t n) {
    void* p = fails() ? nullptr : malloc(n ? n : 1);
    if (!p) throw std::bad_alloc();
    return p;
}
void* operator new(size_t n, const std::nothrow_t&) noexcept { return fails() ? nullptr : malloc(n ? n : 1); }
void operator delete(void* p) noexcept { free(p); }
void operator delete(void* p, size_t) noexcept { free(p); }
void operator delete(void* p, const std::nothrow_t&) noexcept { free(p); }
