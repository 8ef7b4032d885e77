// A CUDA runtime without a device, for tests of the library's host code: device
// memory is host memory whose allocations are tracked and can be made to
// fail, kernels are lines in a log, and a launch on memory that is not
// allocated is logged as "bad" instead of being run. Linked with the library's
// C++ sources (tests/test_host_memory.py).
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <initializer_list>
#include <map>
#include <string>
#include <utility>

#include "../include/photon_cuda.h"
#include "../photon_tracer_b200/csrc/batch.h"
#include "../photon_tracer_b200/csrc/kernels.h"
#include "../photon_tracer_b200/csrc/unet.h"
#include "../photon_tracer_b200/csrc/wavefront.h"

namespace {

std::map<const char*, size_t> g_live;  // allocation -> bytes
std::string g_log;
long g_fail_after = -1;  // allocations that still succeed; -1: all
size_t g_fail_above = ~size_t(0), g_budget = ~size_t(0);
bool g_falling_times = false;
cudaStream_t g_capturing = nullptr;
bool g_tensor_cores = true;
long g_next = 0, g_finished = 0;
cudaError_t g_last = cudaSuccess;  // what cudaGetLastError has not been asked for yet
std::map<cudaEvent_t, long> g_recorded;

void log(const std::string& line) { g_log += line + "\n"; }
std::string hex(const void* p) {
    char b[32];
    std::snprintf(b, sizeof b, "%p", p);
    return b;
}
cudaError_t allocate(void** p, size_t bytes) {
    *p = nullptr;
    size_t used = 0;
    for (const auto& a : g_live) used += a.second;
    if (g_fail_after == 0 || bytes > g_fail_above || used + bytes > g_budget)
        return g_last = cudaErrorMemoryAllocation;
    if (g_fail_after > 0) --g_fail_after;
    *p = std::malloc(bytes ? bytes : 1);
    g_live[static_cast<const char*>(*p)] = bytes;
    return cudaSuccess;
}
// Whether [p, p + bytes) lies in one allocation.
bool live(const void* p, size_t bytes) {
    auto it = g_live.upper_bound(static_cast<const char*>(p));
    if (it == g_live.begin()) return false;
    --it;
    return static_cast<const char*>(p) + bytes <= it->first + it->second;
}
struct Use {
    const void* p;
    size_t bytes;
};
// Reports, as the library's launches do, whatever error is pending.
cudaError_t launch(const std::string& what, std::initializer_list<Use> uses) {
    if (g_last != cudaSuccess) return std::exchange(g_last, cudaSuccess);
    for (const Use& u : uses)
        if (u.bytes && !live(u.p, u.bytes)) {
            log("bad " + what);
            return cudaSuccess;
        }
    log(what);
    return cudaSuccess;
}

}  // namespace

extern "C" {

// ---- the test's side ----
void fake_clear() { g_log.clear(); }
const char* fake_log() { return g_log.c_str(); }
void fake_fail_after(long n) { g_fail_after = n; }
void fake_finish() { ++g_finished; }  // all work so far is done
void fake_fail_above(size_t bytes) { g_fail_above = bytes; }
void fake_budget(size_t bytes) { g_budget = bytes; }
void fake_falling_times(int on) { g_falling_times = on != 0; }
void fake_tensor_cores(int on) { g_tensor_cores = on != 0; }
void fake_capture(void* stream) { g_capturing = static_cast<cudaStream_t>(stream); }
size_t fake_live_bytes() {
    size_t n = 0;
    for (const auto& a : g_live) n += a.second;
    return n;
}

// ---- the runtime ----
cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrComputeCapabilityMajor ? 10 : a == cudaDevAttrMultiProcessorCount ? 148 : 1;
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) { return std::memset(a, 0, sizeof *a), cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "a fake's error"; }
cudaError_t cudaGetLastError() { return std::exchange(g_last, cudaSuccess); }
cudaError_t cudaDeviceSynchronize() { return log("wait device"), cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) { return log("malloc " + std::to_string(n)), allocate(p, n); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return *p = std::malloc(n), cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return std::free(p), cudaSuccess; }
cudaError_t cudaFree(void* p) {
    if (!p) return cudaSuccess;
    log("free");
    g_live.erase(static_cast<const char*>(p));
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return std::memcpy(d, s, n), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    return std::memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) { return std::memset(d, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
    if (!live(d, n)) return log("bad memset"), cudaSuccess;
    return std::memset(d, v, n), cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    return *s = reinterpret_cast<cudaStream_t>(0x1000 + 16 * ++g_next), cudaSuccess;
}
cudaError_t cudaStreamGetId(cudaStream_t s, unsigned long long* id) {
    return *id = reinterpret_cast<unsigned long long>(s), cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return log("wait stream"), cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* c) {
    *c = g_capturing && s == g_capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) { return g_capturing = s, cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    g_capturing = nullptr;
    return *g = reinterpret_cast<cudaGraph_t>(1), log("captured"), cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
    return *e = reinterpret_cast<cudaGraphExec_t>(1), cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return log("graph destroy"), cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return log("graph launch"), cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    return *e = reinterpret_cast<cudaEvent_t>(0x100000 + 16 * ++g_next), cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return g_recorded.erase(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t) { return g_recorded[e] = g_finished, cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t e) {  // pending until the test lets the device finish
    const auto it = g_recorded.find(e);
    return it != g_recorded.end() && it->second == g_finished ? g_last = cudaErrorNotReady : cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t, unsigned) {
    return log("stream waits " + hex(s)), cudaSuccess;
}
cudaError_t cudaPeekAtLastError() { return g_last; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = g_falling_times ? 1.0f / float(++g_next) : 1.0f;
    return log("timed"), cudaSuccess;
}

pt_status pt_accumulate_pass(const float*, size_t, double, double*, void*) { return PT_OK; }

}  // extern "C"

// ---- the library's kernels ----
namespace {
cudaError_t kernel(const char* name) { return launch(name, {}); }
}  // namespace

cudaError_t pt_build_qnodes(const float4* nodes, float4* q, uint32_t n, cudaStream_t) {
    return launch("build_qnodes", {{nodes, n * size_t(128)}, {q, n * size_t(128)}});
}
cudaError_t pt_launch_megakernel(const PtSceneDev&, const PtRenderParams& p, const PtLaunchShape&, cudaStream_t st) {
    return launch("megakernel " + hex(st) + " work " + hex(p.work), {{p.work, 4}});
}
int pt_megakernel_blocks_per_sm(const PtSceneDev&, int, bool, bool, bool) { return 4; }
size_t pt_sample_bytes(const PtRenderParams& p) { return size_t(p.width) * p.rows * (p.aux ? 36 : 12); }
cudaError_t pt_launch_samples(const PtSceneDev&, const PtRenderParams& p, int, int count, float* buffer, int,
                              int& blocks_per_sm, cudaStream_t st) {
    if (!blocks_per_sm) {
        log("blocks worked out");
        blocks_per_sm = 5;
    }
    return launch("samples " + hex(st) + " work " + hex(p.work) + " buffer " + hex(buffer),
                  {{p.work, 4}, {buffer, pt_sample_bytes(p) * size_t(count)}});
}
cudaError_t pt_launch_trace_closest(const PtSceneDev& S, const float*, size_t n, float, float, void*, int sms,
                                    cudaStream_t) {
    return kernel(pt_rays_stream(S, n, false, sms) ? "closest stream" : "closest lock-step");
}
cudaError_t pt_launch_trace_any(const PtSceneDev& S, const float*, size_t n, float, float, uint8_t*, int sms,
                                cudaStream_t) {
    return kernel(pt_rays_stream(S, n, true, sms) ? "any stream" : "any lock-step");
}
cudaError_t pt_launch_trace_count(const PtSceneDev&, const float*, size_t, float, float, unsigned long long*,
                                  cudaStream_t) {
    return kernel("count");
}
cudaError_t pt_launch_primary_depth(const PtSceneDev&, const PtCamDev&, int, int, float*, cudaStream_t) {
    return kernel("depth");
}
cudaError_t pt_launch_mean_of_sum(const double*, size_t, double, float*, cudaStream_t) { return kernel("mean"); }
size_t pt_wavefront_bytes(uint32_t slots) { return size_t(slots) * 64; }
cudaError_t pt_launch_wavefront(const PtSceneDev&, const PtRenderParams&, void*, uint32_t, int, cudaStream_t,
                                uint32_t*) {
    return kernel("wavefront");
}
cudaError_t pt_launch_batch(const PtSceneDev&, const PtBatchLaunch&, int threads, int, cudaStream_t) {
    return kernel(("batch " + std::to_string(threads)).c_str());
}
cudaError_t pt_launch_batch_stream(const PtSceneDev&, const PtBatchStream& b, int, cudaStream_t) {
    return launch("batch stream", {{b.samples, 12 * size_t(b.items)}, {b.segments, b.n_segments * sizeof(PtBatchSegment)}});
}

namespace unet {
namespace {
size_t px(const ConvShape& s) { return size_t(s.B) * s.H * s.W; }
}  // namespace
cudaError_t conv_fwd(const ConvShape& s, const void* in, bool in_f32, const __nv_bfloat16*, const float*, bool,
                     void* out, bool out_f32, int stride, int, cudaStream_t) {
    return launch("conv", {{in, px(s) * s.Cin * (in_f32 ? 4 : 2)}, {out, px(s) * stride * (out_f32 ? 4 : 2)}});
}
cudaError_t conv_fwd_tc(const ConvShape& s, const __nv_bfloat16* in, const __nv_bfloat16*, const float*, bool,
                        const ConvOut& o, bool out_f32, unsigned int*, cudaStream_t) {
    if (!g_tensor_cores) return cudaErrorNotSupported;
    return launch("conv tc", {{in, px(s) * s.Cin * 2},
                              {o.out, o.out ? px(s) * o.stride * (out_f32 ? 4 : 2) : 0},
                              {o.out2, o.out2 ? px(s) * o.stride2 * (o.up2 ? 8 : 2) : 0},
                              {o.pool, o.pool ? px(s) / 4 * s.Cout * 2 : 0},
                              {o.mask, o.mask ? px(s) * s.Cout * 2 : 0}});
}
cudaError_t conv_wgrad(const ConvShape& s, const __nv_bfloat16* in, const float* g, float*, float*, cudaStream_t) {
    return launch("wgrad", {{in, px(s) * s.Cin * 2}, {g, px(s) * s.Cout * 4}});
}
cudaError_t conv_wgrad_tc(const ConvShape& s, const __nv_bfloat16* in, const __nv_bfloat16* g, float*, unsigned int*,
                          cudaStream_t) {
    if (!g_tensor_cores) return cudaErrorNotSupported;
    return launch("wgrad tc", {{in, px(s) * s.Cin * 2}, {g, px(s) * s.Cout * 2}});
}
cudaError_t flip_transpose_all(const FlipLayers&, const __nv_bfloat16*, __nv_bfloat16*, cudaStream_t) {
    return kernel("flip all");
}
cudaError_t relu_grad(long n, const __nv_bfloat16* y, float* g, cudaStream_t) {
    return launch("relu_grad", {{y, size_t(n) * 2}, {g, size_t(n) * 4}});
}
cudaError_t pool_fwd(int B, int H, int W, int C, const __nv_bfloat16* in, __nv_bfloat16* out, cudaStream_t) {
    const size_t n = size_t(B) * H * W * C * 2;
    return launch("pool", {{in, n}, {out, n / 4}});
}
cudaError_t pool_bwd(int B, int H, int W, int C, const __nv_bfloat16*, const __nv_bfloat16*, const float* gout,
                     float* gin, cudaStream_t) {
    const size_t n = size_t(B) * H * W * C * 4;
    return launch("pool_bwd", {{gout, n / 4}, {gin, n}});
}
cudaError_t up_fwd(int B, int h, int w, int C, const __nv_bfloat16* in, __nv_bfloat16* out, int stride, int,
                   cudaStream_t) {
    const size_t n = size_t(B) * h * w;
    return launch("up", {{in, n * C * 2}, {out, n * 4 * stride * 2}});
}
cudaError_t up_bwd(int B, int h, int w, int C, const float* gout, int stride, int, float* gin, cudaStream_t) {
    const size_t n = size_t(B) * h * w;
    return launch("up_bwd", {{gout, n * 4 * stride * 4}, {gin, n * C * 4}});
}
cudaError_t copy_channels(long n, int C, const __nv_bfloat16* src, __nv_bfloat16* dst, int stride, int, cudaStream_t) {
    return launch("copy", {{src, size_t(n) * C * 2}, {dst, size_t(n) * stride * 2}});
}
cudaError_t add_channels(long n, int C, const float* src, int stride, int, float* dst, cudaStream_t) {
    return launch("add", {{src, size_t(n) * stride * 4}, {dst, size_t(n) * C * 4}});
}
cudaError_t make_input(long n, const float*, __nv_bfloat16* dst, int stride, cudaStream_t) {
    return launch("input", {{dst, size_t(n) * stride * 2}});
}
cudaError_t frame_input(int, int, int Wp, int Hp, const float*, const float*, const float*, __nv_bfloat16* dst,
                        int stride, cudaStream_t) {
    return launch("input", {{dst, size_t(Wp) * Hp * stride * 2}});
}
cudaError_t frame_output(int, int H, int Wp, int stride, const float* pred, float*, cudaStream_t) {
    return launch("output", {{pred, size_t(Wp) * H * stride * 4}});
}
cudaError_t make_output(long n, int stride, const float* pred, float*, cudaStream_t) {
    return launch("output", {{pred, size_t(n) * stride * 4}});
}
cudaError_t l1_loss(long n, int stride, const float* pred, const float*, float* grad, float*, cudaStream_t) {
    return launch("l1_loss", {{pred, size_t(n) * stride * 4}, {grad, size_t(n) * stride * 4}});
}
cudaError_t l1_back(long n, const float* pred, const float*, float4* g4, __nv_bfloat16* g16, float*, float*,
                    cudaStream_t) {
    return launch("l1_back", {{pred, size_t(n) * 64}, {g4, size_t(n) * 16}, {g16, size_t(n) * 32}});
}
cudaError_t last_back(int B, int H, int W, const float4* g4, const __nv_bfloat16*, const __nv_bfloat16* y,
                      __nv_bfloat16* g16, float*, cudaStream_t) {
    const size_t n = size_t(B) * H * W;
    return launch("last_back", {{g4, n * 16}, {y, n * 64}, {g16, n * 64}});
}
cudaError_t up_back(int B, int h, int w, int C, const float* gcat, int stride, const __nv_bfloat16* y,
                    __nv_bfloat16* g16, float*, cudaStream_t) {
    const size_t n = size_t(B) * h * w;
    return launch("up_back", {{gcat, n * 4 * stride * 4}, {y, n * C * 2}, {g16, n * C * 2}});
}
cudaError_t skip_back(int B, int H, int W, int C, const float* gcat, int stride, int, const __nv_bfloat16* y,
                      const __nv_bfloat16* pooled, const float* gpool, __nv_bfloat16* g16, float*, cudaStream_t) {
    const size_t n = size_t(B) * H * W;
    return launch("skip_back", {{gcat, n * stride * 4}, {y, n * C * 2}, {pooled, n / 4 * C * 2}, {gpool, n / 4 * C * 4},
                                {g16, n * C * 2}});
}
cudaError_t adam(long, float*, const float*, float*, float*, __nv_bfloat16*, float, int, cudaStream_t) {
    return kernel("adam");
}
cudaError_t f32_to_bf16(long, const float*, __nv_bfloat16*, cudaStream_t) { return kernel("f32_to_bf16"); }
}  // namespace unet
