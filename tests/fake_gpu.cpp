// The CUDA runtime calls and kernel launchers that renderer.cpp uses, over host memory: device buffers are
// heap blocks, copies are memcpy, launches do nothing. fake_fail makes a call fail, fake_calls counts it;
// fake_null_launches counts launches that were handed a null buffer which their kernel reads or writes.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

#include "encode.cuh"
#include "kernels.cuh"

namespace {
std::mutex g_mutex;
std::map<std::string, int> g_calls, g_failFrom;
std::map<const void*, size_t> g_locked, g_live;
std::atomic<int> g_nullLaunches{0};

cudaError_t called(const char* name, cudaError_t failure = cudaErrorMemoryAllocation) {
    std::lock_guard<std::mutex> lock(g_mutex);
    const int n = ++g_calls[name];
    const auto f = g_failFrom.find(name);
    return f != g_failFrom.end() && (f->second < 0 ? n >= -f->second : n == f->second) ? failure : cudaSuccess;
}
template <class... P>
cudaError_t launched(P... buffers) {
    if ((... || (buffers == nullptr))) ++g_nullLaunches;
    return cudaSuccess;
}
char g_scratch[64];
}  // namespace

extern "C" {
// the nth call of `name` from now on fails (0: none does; -n: the nth and all after it)
void fake_fail(const char* name, int nth) {
    std::lock_guard<std::mutex> lock(g_mutex);
    if (nth) g_failFrom[name] = nth > 0 ? g_calls[name] + nth : nth - g_calls[name];
    else g_failFrom.erase(name);
}
int fake_calls(const char* name) {
    std::lock_guard<std::mutex> lock(g_mutex);
    return g_calls[name];
}
int fake_null_launches() { return g_nullLaunches.exchange(0); }  // since the last call
size_t fake_live_bytes() {  // of device memory
    std::lock_guard<std::mutex> lock(g_mutex);
    size_t sum = 0;
    for (const auto& [p, n] : g_live) sum += n;
    return sum;
}
// host memory that counts as page-locked
void fake_page_locked(const void* p, size_t bytes) {
    std::lock_guard<std::mutex> lock(g_mutex);
    if (bytes) g_locked[p] = bytes;
    else g_locked.erase(p);
}

extern const uint32_t gsr_logf_fixups[1], gsr_logf_bucket_start[2];
extern const uint32_t gsr_logf_fixup_count, gsr_logf_bucket_count, gsr_logf_fixup_base, gsr_logf_fixup_last;
const uint32_t gsr_logf_fixups[1] = {0}, gsr_logf_bucket_start[2] = {0, 0};
const uint32_t gsr_logf_fixup_count = 0, gsr_logf_bucket_count = 1, gsr_logf_fixup_base = 0, gsr_logf_fixup_last = 0;

cudaError_t cudaMalloc(void** p, size_t n) {
    const cudaError_t e = called("cudaMalloc");
    if (e != cudaSuccess) return e;
    *p = std::aligned_alloc(256, (n + 255) / 256 * 256);
    std::lock_guard<std::mutex> lock(g_mutex);
    g_live[*p] = n;
    return e;
}
cudaError_t cudaFree(void* p) {
    {
        std::lock_guard<std::mutex> lock(g_mutex);
        g_live.erase(p);
    }
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    const cudaError_t e = called("cudaHostAlloc");
    if (e == cudaSuccess) *p = std::malloc(n);
    return e;
}
cudaError_t cudaFreeHost(void* p) { called("cudaFreeHost"); std::free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    const cudaError_t e = called("cudaMemcpy", cudaErrorUnknown);
    if (e == cudaSuccess) std::memcpy(d, s, n);
    return e;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    const cudaError_t e = called("cudaMemcpyAsync", cudaErrorUnknown);
    if (e == cudaSuccess) std::memcpy(d, s, n);
    return e;
}
cudaError_t cudaMemcpy2D(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind) {
    for (size_t r = 0; r < h; ++r) std::memcpy(static_cast<char*>(d) + r * dp, static_cast<const char*>(s) + r * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { std::memset(p, v, n); return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    std::lock_guard<std::mutex> lock(g_mutex);
    std::memset(a, 0, sizeof(*a));
    a->type = cudaMemoryTypeUnregistered;
    for (const auto& [base, bytes] : g_locked)
        if (p >= base && p < static_cast<const char*>(base) + bytes) a->type = cudaMemoryTypeHost;
    return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPoint(const char*, void** p, unsigned long long, cudaDriverEntryPointQueryResult*) {
    *p = nullptr;
    return cudaErrorNotSupported;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = reinterpret_cast<cudaStream_t>(g_scratch);
    return called("cudaStreamCreateWithFlags");
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) { *s = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return cudaErrorNotSupported; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = reinterpret_cast<cudaEvent_t>(g_scratch);
    return called("cudaEventCreateWithFlags");
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventRecordWithFlags(cudaEvent_t, cudaStream_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
}

namespace gsr {
cudaError_t launchFrameBegin(DeviceControl* ctl, uint32_t, uint32_t, uint32_t* ranges, uint32_t rangeWords, SortPlan*, uint32_t,
                             cudaStream_t, SortPlan*, uint32_t* clear, uint32_t clearCount, uint4* clear4, uint32_t clear4Count) {
    return launched(ctl, rangeWords ? static_cast<void*>(ranges) : ctl, clearCount ? static_cast<void*>(clear) : ctl,
                    clear4Count ? static_cast<void*>(clear4) : ctl);
}
uint32_t rowPartitionTile(uint64_t) { return kRowPartTile; }
cudaError_t launchFront(const FrontArgs& a, uint32_t, uint32_t, cudaStream_t) {
    return launched(static_cast<void*>(a.offsets), static_cast<void*>(a.tileCounts), static_cast<void*>(a.keys), static_cast<void*>(a.scanStatus));
}
cudaError_t launchFrontBinningKeys(const FrontArgs& a, uint32_t, uint32_t, cudaStream_t) {
    return launched(static_cast<void*>(a.depthKeys[0]), static_cast<void*>(a.hints), static_cast<void*>(a.spanRows),
                    static_cast<void*>(a.tileCounts), a.rowRecords ? static_cast<void*>(a.rowHist) : a.ctl,
                    a.rowRecords ? static_cast<void*>(a.spill) : a.ctl);
}
cudaError_t launchFrontBinningEmit(const FrontArgs& a, cudaStream_t) {
    return launched(static_cast<void*>(a.offsets), static_cast<void*>(a.keys), static_cast<void*>(a.scanStatus));
}
cudaError_t launchRowPartition(const FrontArgs& a, cudaStream_t) {
    return launched(static_cast<void*>(a.rowStatus), static_cast<void*>(a.rowPlan), static_cast<void*>(a.rowEntries),
                    static_cast<void*>(a.spill));
}
cudaError_t launchRowTiles(const FrontArgs& a, uint32_t, cudaStream_t) {
    return launched(static_cast<void*>(a.rowPlan), static_cast<void*>(a.list), static_cast<void*>(a.ranges));
}
cudaError_t launchDecodeColoursTc(const FrontArgs&, uint32_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launchSort(const SortArgs& a, uint32_t, cudaStream_t) {
    return launched(static_cast<void*>(a.status), static_cast<void*>(a.keys[0]), static_cast<void*>(a.keys[1]));
}
bool depthSortInCluster(uint32_t, uint32_t) { return true; }
cudaError_t launchDepthSortCluster(const SortArgs& a, cudaStream_t) { return launched(static_cast<void*>(a.keys[0])); }
cudaError_t launchRanges(const RenderArgs& a, uint32_t, cudaStream_t) { return launched(static_cast<void*>(a.ranges)); }
cudaError_t launchRender(const RenderArgs& a, cudaStream_t) { return launched(a.image, static_cast<void*>(a.ranges)); }
cudaError_t launchLogfTable(float*, LogfFixups, cudaStream_t) { return cudaSuccess; }
cudaError_t launchScan(const uint32_t*, const uint32_t*, uint32_t*, uint32_t*, uint32_t, uint32_t, uint64_t*, DeviceControl*,
                       cudaStream_t, uint32_t, uint32_t, const ScanGather*) { return cudaSuccess; }
cudaError_t launchShDecode(const SceneArgs&, uint32_t, uint32_t, uint32_t, int, float*, uint8_t*, cudaStream_t) { return cudaSuccess; }
cudaError_t launchPackTrain(const float*, void*, cudaStream_t) { return cudaSuccess; }
cudaError_t launchColorTrainStep(const float*, const uint8_t*, uint32_t, uint32_t, uint32_t, uint32_t, float*, float*, float*,
                                 float*, void*, uint32_t, uint32_t*, float, float*, uint32_t, uint32_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launchPackDecoder(const float*, DecoderWeights*, cudaStream_t) { return cudaSuccess; }
uint32_t colorTrainBatchMultiple() { return 256; }
cudaError_t launchColorEncode(const float*, const float*, uint4*, DecoderWeights*, uint32_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launchColorGate(const float*, const uint8_t*, uint32_t, uint32_t, const DecoderWeights*, uint4*, float, uint32_t*,
                            uint32_t*, cudaStream_t) { return cudaSuccess; }
cudaError_t staticScanScratch(void** base) { *base = g_scratch; return cudaSuccess; }
cudaError_t loadScanKernel() { return cudaSuccess; }
cudaError_t loadFrameBeginKernel() { return cudaSuccess; }
cudaError_t launchPack64(const uint32_t*, const uint32_t*, uint64_t*, uint32_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launchUnpack64(const uint64_t*, uint32_t*, uint32_t*, uint32_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launchSetEntries(DeviceControl*, uint32_t, cudaStream_t) { return cudaSuccess; }
cudaError_t launchEncodeDegrees(const EncodeArgs&, uint8_t*, uint32_t*, cudaStream_t) { return cudaSuccess; }
cudaError_t launchEncodeRecords(const EncodeArgs&, const uint8_t*, const uint32_t*, cudaStream_t) { return cudaSuccess; }
cudaError_t launchCodebookPoints(const EncodeArgs&, const uint8_t*, float*, cudaStream_t) { return cudaSuccess; }
cudaError_t launchCodebookGather(const float*, uint32_t, const uint32_t*, uint32_t, float*, cudaStream_t) { return cudaSuccess; }
cudaError_t launchNearestCentroid(const float*, uint32_t, uint32_t, const float*, const float*, uint32_t, uint32_t*, float*, cudaStream_t) { return cudaSuccess; }
}  // namespace gsr
