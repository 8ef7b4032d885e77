// Edge-avoiding a-trous denoiser on the GPU: the filter of
// include/denoise.hpp:55-139 (demodulate by albedo, five 5x5 B3-spline passes
// with taps 1, 2, 4, 8, 16 apart, weights from normals, albedo and the
// variance-scaled luminance difference, variance filtered along). Each pass
// reads a 5x5 neighbourhood of the previous pass's lighting, so the passes
// are separate launches ping-ponging two scratch buffers.
#include <cuda_runtime.h>

#include <cstdint>
#include <string>

#include "../../include/photon_cuda.h"
#include "pt_host.hpp"

namespace {

__device__ __forceinline__ float lum(float r, float g, float b) { return 0.2126f * r + 0.7152f * g + 0.0722f * b; }

// Lighting and variance of a pixel, one 16-byte word in the scratch; ALIGNED
// is whether the caller's scratch allows 16-byte accesses.
template <bool ALIGNED>
__device__ __forceinline__ float4 load_lv(const float* lv, size_t p) {
    if (ALIGNED) return reinterpret_cast<const float4*>(lv)[p];
    return make_float4(lv[4 * p], lv[4 * p + 1], lv[4 * p + 2], lv[4 * p + 3]);
}
template <bool ALIGNED>
__device__ __forceinline__ void store_lv(float* lv, size_t p, float4 v) {
    if (ALIGNED) {
        reinterpret_cast<float4*>(lv)[p] = v;
    } else {
        lv[4 * p] = v.x;
        lv[4 * p + 1] = v.y;
        lv[4 * p + 2] = v.z;
        lv[4 * p + 3] = v.w;
    }
}

template <bool ALIGNED>
__global__ void prepare(int n, const float* __restrict__ color, const float* __restrict__ albedo,
                        const float* __restrict__ normal, const float* __restrict__ variance, float* __restrict__ lv,
                        float* __restrict__ nrm) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const size_t q = 3 * size_t(p);
    const float a0 = albedo[q], a1 = albedo[q + 1], a2 = albedo[q + 2];
    const float a = fmaxf(lum(a0, a1, a2), 0.01f);
    store_lv<ALIGNED>(lv, p, make_float4(color[q] / fmaxf(a0, 0.01f), color[q + 1] / fmaxf(a1, 0.01f),
                                         color[q + 2] / fmaxf(a2, 0.01f), fmaxf(variance[p], 0.0f) / (a * a)));
    const float* s = normal + q;
    const float len = sqrtf(s[0] * s[0] + s[1] * s[1] + s[2] * s[2]);
    for (int c = 0; c < 3; ++c) nrm[q + c] = len > 1e-6f ? s[c] / len : 0;
}

// One pass. A block takes 32 x 8 pixels of one phase in y and PH adjacent
// phases in x of the step x step lattice (32 / PH lattice columns, 8 rows), so
// that for every step its taps are a dense 5x5 stencil of the pixels it stages
// in shared memory: 1.7 to 2.3 loads per pixel instead of 25 of ten scalars
// each, of PH neighbouring pixels at a time (PH = 1 throughout: the pass of
// step 16 at 239 us, from half-used sectors). A staged pixel is three 16-byte
// words (48 bytes apart, free of bank conflicts) with its luminance and its
// kind -- 0 surface, 1 sky (zero normal), 2 outside the image -- worked out
// once: taps of another kind than the centre are skipped. What bounds it is
// the arithmetic of the taps (65 instructions each, an exponential among
// them; issue slots 89% busy) and their shared-memory reads. 1920x1080:
// 183 -> 134..143 us per pass, the filter 0.96 -> 0.70 ms.
constexpr int kTX = 32, kTY = 8, kHY = kTY + 4;
template <int PH, bool ALIGNED, bool LAST>
__global__ void __launch_bounds__(kTX* kTY) atrous_pass(
    int w, int h, int step, int blocks_x, const float* __restrict__ albedo, const float* __restrict__ nrm,
    const float* __restrict__ lv, float* __restrict__ lv_next, float* __restrict__ out) {
    constexpr int LX = kTX / PH, HX = (LX + 4) * PH;  // lattice columns; staged pixels per row
    __shared__ float4 tile[HX * kHY][3];              // (light, variance) (normal, luminance) (albedo, kind)
    const int bx = int(blockIdx.x % unsigned(blocks_x)), by = int(blockIdx.x / unsigned(blocks_x));
    const int groups = step / PH;  // groups of PH phases in x
    const int px = bx % groups * PH, py = by % step, lx0 = bx / groups * LX, ly0 = by / step * kTY;
    const int tid = threadIdx.y * kTX + threadIdx.x;
    for (int i = tid; i < HX * kHY; i += kTX * kTY) {
        const int c = i % HX;
        const long x = px + c % PH + long(lx0 + c / PH - 2) * step, y = py + long(ly0 + i / HX - 2) * step;
        float4 a = make_float4(0, 0, 0, 0), b = a, k = make_float4(0, 0, 0, 2);
        if (x >= 0 && y >= 0 && x < w && y < h) {
            const size_t q = size_t(y) * w + x;
            a = load_lv<ALIGNED>(lv, q);
            b = make_float4(nrm[3 * q], nrm[3 * q + 1], nrm[3 * q + 2], lum(a.x, a.y, a.z));
            k = make_float4(albedo[3 * q], albedo[3 * q + 1], albedo[3 * q + 2],
                            b.x == 0 && b.y == 0 && b.z == 0 ? 1.0f : 0.0f);
        }
        tile[i][0] = a;
        tile[i][1] = b;
        tile[i][2] = k;
    }
    __syncthreads();
    const int ph = threadIdx.x % PH, lx = threadIdx.x / PH;
    const long xl = px + ph + long(lx0 + lx) * step, yl = py + long(ly0 + int(threadIdx.y)) * step;
    if (xl >= w || yl >= h) return;
    const int x = int(xl), y = int(yl);
    const size_t p = size_t(y) * w + x;
    const float4* centre = tile[(threadIdx.y + 2) * HX + threadIdx.x + 2 * PH];
    const float4 np = centre[1], ap = centre[2];
    const bool p_sky = ap.w == 1.0f;
    const float lp = np.w;
    float v = 0, vw = 0;
#pragma unroll
    for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
        for (int dx = -1; dx <= 1; ++dx) {
            const int qx = x + dx, qy = y + dy;
            if (qx < 0 || qy < 0 || qx >= w || qy >= h) continue;
            const float k = (dx ? 0.5f : 1) * (dy ? 0.5f : 1);
            v += k * lv[4 * (size_t(qy) * w + qx) + 3];
            vw += k;
        }
    const float scale = 1 / (4.0f * sqrtf(v / vw) + 1e-4f);
    float s0 = 0, s1 = 0, s2 = 0, sum_w = 0, sum_var = 0;
    const float kernel[3] = {3.0f / 8, 1.0f / 4, 1.0f / 16};
#pragma unroll 1
    for (int dy = -2; dy <= 2; ++dy) {
        const float ky = dy == 0 ? kernel[0] : dy * dy == 1 ? kernel[1] : kernel[2];
        const float4* row = tile[(int(threadIdx.y) + 2 + dy) * HX + threadIdx.x];
#pragma unroll
        for (int dx = -2; dx <= 2; ++dx) {
            const float4 lq = row[3 * PH * (dx + 2)], nq = row[3 * PH * (dx + 2) + 1],
                         aq = row[3 * PH * (dx + 2) + 2];
            if (aq.w != ap.w) continue;
            float weight = kernel[dx < 0 ? -dx : dx] * ky;
            if (!p_sky) {
                float nd = fmaxf(np.x * nq.x + np.y * nq.y + np.z * nq.z, 0.0f);
                for (int k = 0; k < 6; ++k) nd *= nd;
                weight *= nd;
            }
            const float da0 = ap.x - aq.x, da1 = ap.y - aq.y, da2 = ap.z - aq.z;
            weight *= expf(-(da0 * da0 + da1 * da1 + da2 * da2) * (1 / 0.01f) - fabsf(lp - nq.w) * scale);
            s0 += weight * lq.x;
            s1 += weight * lq.y;
            s2 += weight * lq.z;
            sum_w += weight;
            sum_var += weight * weight * lq.w;
        }
    }
    const float4 r = make_float4(s0 / sum_w, s1 / sum_w, s2 / sum_w, sum_var / (sum_w * sum_w));
    if (LAST) {  // modulate by the albedo again
        out[3 * p] = r.x * fmaxf(ap.x, 0.01f);
        out[3 * p + 1] = r.y * fmaxf(ap.y, 0.01f);
        out[3 * p + 2] = r.z * fmaxf(ap.z, 0.01f);
    } else {
        store_lv<ALIGNED>(lv_next, p, r);
    }
}

struct Pixel {
    float4 lv;
    float n0, n1, n2, a0, a1, a2, l;  // normal, albedo, luminance
    bool sky;
};
template <bool ALIGNED>
__device__ __forceinline__ Pixel load_pixel(const float* __restrict__ lv, const float* __restrict__ nrm,
                                            const float* __restrict__ albedo, size_t q) {
    Pixel p;
    p.lv = load_lv<ALIGNED>(lv, q);
    p.l = lum(p.lv.x, p.lv.y, p.lv.z);
    p.n0 = nrm[3 * q];
    p.n1 = nrm[3 * q + 1];
    p.n2 = nrm[3 * q + 2];
    p.a0 = albedo[3 * q];
    p.a1 = albedo[3 * q + 1];
    p.a2 = albedo[3 * q + 2];
    p.sky = p.n0 == 0 && p.n1 == 0 && p.n2 == 0;
    return p;
}

// The same pass with a thread per pixel in image order, reading its taps where
// they are: for strips, which fill few of a tile's lattice columns or rows (the
// filter in tiles throughout, then as launch_pass chooses: 16x20000 287 ->
// 153 us, 20000x2 85 -> 46, 48x20000 503 -> 427).
template <bool ALIGNED, bool LAST>
__global__ void __launch_bounds__(128) atrous_direct(
    int w, int h, int step, const float* __restrict__ albedo, const float* __restrict__ nrm,
    const float* __restrict__ lv, float* __restrict__ lv_next, float* __restrict__ out) {
    const unsigned p = blockIdx.x * 128u + threadIdx.x;
    if (p >= unsigned(w) * unsigned(h)) return;
    const int y = int(p / unsigned(w)), x = int(p - unsigned(y) * unsigned(w));
    const Pixel c = load_pixel<ALIGNED>(lv, nrm, albedo, p);
    float v = 0, vw = 0;
#pragma unroll
    for (int dy = -1; dy <= 1; ++dy)
#pragma unroll
        for (int dx = -1; dx <= 1; ++dx) {
            const int qx = x + dx, qy = y + dy;
            if (qx < 0 || qy < 0 || qx >= w || qy >= h) continue;
            const float k = (dx ? 0.5f : 1) * (dy ? 0.5f : 1);
            v += k * lv[4 * (size_t(qy) * w + qx) + 3];
            vw += k;
        }
    const float scale = 1 / (4.0f * sqrtf(v / vw) + 1e-4f);
    float s0 = 0, s1 = 0, s2 = 0, sum_w = 0, sum_var = 0;
    const float kernel[3] = {3.0f / 8, 1.0f / 4, 1.0f / 16};
#pragma unroll 1
    for (int dy = -2; dy <= 2; ++dy) {
        const long qy = y + long(dy) * step;
        if (qy < 0 || qy >= h) continue;
        const float ky = dy == 0 ? kernel[0] : dy * dy == 1 ? kernel[1] : kernel[2];
#pragma unroll
        for (int dx = -2; dx <= 2; ++dx) {
            const long qx = x + long(dx) * step;
            if (qx < 0 || qx >= w) continue;
            const Pixel q = load_pixel<ALIGNED>(lv, nrm, albedo, size_t(qy) * w + qx);
            if (q.sky != c.sky) continue;
            float weight = kernel[dx < 0 ? -dx : dx] * ky;
            if (!c.sky) {
                float nd = fmaxf(c.n0 * q.n0 + c.n1 * q.n1 + c.n2 * q.n2, 0.0f);
                for (int k = 0; k < 6; ++k) nd *= nd;
                weight *= nd;
            }
            const float da0 = c.a0 - q.a0, da1 = c.a1 - q.a1, da2 = c.a2 - q.a2;
            weight *= expf(-(da0 * da0 + da1 * da1 + da2 * da2) * (1 / 0.01f) - fabsf(c.l - q.l) * scale);
            s0 += weight * q.lv.x;
            s1 += weight * q.lv.y;
            s2 += weight * q.lv.z;
            sum_w += weight;
            sum_var += weight * weight * q.lv.w;
        }
    }
    const float4 r = make_float4(s0 / sum_w, s1 / sum_w, s2 / sum_w, sum_var / (sum_w * sum_w));
    if (LAST) {
        out[3 * size_t(p)] = r.x * fmaxf(c.a0, 0.01f);
        out[3 * size_t(p) + 1] = r.y * fmaxf(c.a1, 0.01f);
        out[3 * size_t(p) + 2] = r.z * fmaxf(c.a2, 0.01f);
    } else {
        store_lv<ALIGNED>(lv_next, p, r);
    }
}

template <bool ALIGNED>
__global__ void finish(int n, const float* __restrict__ lv, const float* albedo, float* out) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= n) return;
    const float4 l = load_lv<ALIGNED>(lv, p);
    const float r[3] = {l.x, l.y, l.z};
    for (int c = 0; c < 3; ++c) {
        const size_t at = 3 * size_t(p) + c;
        out[at] = r[c] * fmaxf(albedo[at], 0.01f);
    }
}

template <int PH, bool ALIGNED, bool LAST>
void launch_pass(int w, int h, int step, const float* albedo, const float* nrm, const float* lv, float* lv_next,
                 float* out, cudaStream_t stream) {
    const int lw = (w + step - 1) / step, lh = (h + step - 1) / step, columns = kTX / PH;
    const int tx = (lw + columns - 1) / columns, ty = (lh + kTY - 1) / kTY;
    const int bx = tx * (step / PH);
    const unsigned blocks = unsigned(bx) * unsigned(ty * step);
    // Tiles cost two thirds of a direct pass when full (1920x1080: 138 us, 183),
    // so they lose where less than two thirds of their pixels are in the image --
    // unless they are too few to fill the GPU (eight to an SM), where a pass
    // takes as long as one tile or one pixel, and the tile's loads go out at once
    // (64x36, the filter: 54 us, 82).
    const bool filled = 3 * (long(lw) * lh) >= 2 * (long(tx) * columns * ty * kTY);
    if (!filled && blocks > 148u * 8u)
        atrous_direct<ALIGNED, LAST><<<unsigned((long(w) * h + 127) / 128), 128, 0, stream>>>(w, h, step, albedo, nrm, lv,
                                                                                              lv_next, out);
    else
        atrous_pass<PH, ALIGNED, LAST><<<blocks, dim3(kTX, kTY), 0, stream>>>(w, h, step, bx, albedo, nrm, lv, lv_next,
                                                                              out);
}

template <bool ALIGNED>
void run_atrous(int w, int h, const float* color, const float* albedo, const float* normal, const float* variance,
                float* out, float* scratch, cudaStream_t stream) {
    const int n = w * h;
    // A caller may filter into its albedo buffer: the last pass, which reads
    // neighbours' albedo, must then not write there.
    // Nor where the caller reuses the scratch for the image: that pass still
    // reads lighting and normals there.
    auto meets_out = [&](const float* p, size_t floats) {
        return reinterpret_cast<uintptr_t>(out) < reinterpret_cast<uintptr_t>(p + floats) &&
               reinterpret_cast<uintptr_t>(p) < reinterpret_cast<uintptr_t>(out + 3 * size_t(n));
    };
    const bool in_albedo = meets_out(albedo, 3 * size_t(n)), in_scratch = meets_out(scratch, 11 * size_t(n));
    float* lv = scratch;
    float* lv_next = lv + 4 * size_t(n);
    float* nrm = lv_next + 4 * size_t(n);
    prepare<ALIGNED><<<(n + 255) / 256, 256, 0, stream>>>(n, color, albedo, normal, variance, lv, nrm);
    launch_pass<1, ALIGNED, false>(w, h, 1, albedo, nrm, lv, lv_next, nullptr, stream);
    launch_pass<2, ALIGNED, false>(w, h, 2, albedo, nrm, lv_next, lv, nullptr, stream);
    launch_pass<4, ALIGNED, false>(w, h, 4, albedo, nrm, lv, lv_next, nullptr, stream);
    launch_pass<4, ALIGNED, false>(w, h, 8, albedo, nrm, lv_next, lv, nullptr, stream);
    if (in_albedo || in_scratch) {
        launch_pass<4, ALIGNED, false>(w, h, 16, albedo, nrm, lv, lv_next, nullptr, stream);
        // beside lv_next, in a part of the scratch that is free by now and that out does not meet
        float* image = !in_scratch ? out : meets_out(lv, 4 * size_t(n)) ? nrm : lv;
        finish<ALIGNED><<<(n + 255) / 256, 256, 0, stream>>>(n, lv_next, albedo, image);
        if (in_scratch) cudaMemcpyAsync(out, image, 12 * size_t(n), cudaMemcpyDeviceToDevice, stream);
    } else {
        launch_pass<4, ALIGNED, true>(w, h, 16, albedo, nrm, lv, nullptr, out, stream);
    }
}

pt_status cuda_status(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return PT_OK;
    cudaGetLastError();  // reported now, not by the next call's launch check
    return pt::fail(e == cudaErrorMemoryAllocation ? PT_ERR_OUT_OF_MEMORY : PT_ERR_CUDA,
                    std::string(what) + ": " + cudaGetErrorString(e));
}

}  // namespace

extern "C" {

size_t pt_denoise_atrous_scratch_floats(int width, int height) {
    if (width <= 0 || height <= 0) return 0;
    return 11 * size_t(width) * size_t(height);
}

pt_status pt_denoise_atrous_device(int w, int h, const float* color, const float* albedo, const float* normal,
                                   const float* variance, float* out, float* scratch, void* stream_) {
    pt::clear_error();
    if (w <= 0 || h <= 0) return pt::fail(PT_ERR_INVALID_ARG, "pt_denoise_atrous_device: bad size");
    if (!color || !albedo || !normal || !variance || !out || !scratch)
        return pt::fail(PT_ERR_INVALID_ARG, "pt_denoise_atrous_device: null pointer");
    if (size_t(w) * h > (size_t(1) << 30)) return pt::fail(PT_ERR_INVALID_ARG, "pt_denoise_atrous_device: too large");
    cudaStream_t stream = static_cast<cudaStream_t>(stream_);
    if (reinterpret_cast<uintptr_t>(scratch) % 16 == 0)
        run_atrous<true>(w, h, color, albedo, normal, variance, out, scratch, stream);
    else
        run_atrous<false>(w, h, color, albedo, normal, variance, out, scratch, stream);
    return cuda_status(cudaGetLastError(), "pt_denoise_atrous_device");
}

pt_status pt_denoise_atrous(int w, int h, const float* color, const float* albedo, const float* normal,
                            const float* variance, float* out) {
    pt::clear_error();
    if (w <= 0 || h <= 0) return pt::fail(PT_ERR_INVALID_ARG, "pt_denoise_atrous: bad size");
    if (!color || !albedo || !normal || !variance || !out)
        return pt::fail(PT_ERR_INVALID_ARG, "pt_denoise_atrous: null pointer");
    const size_t n = size_t(w) * h;
    float* d = nullptr;
    const size_t floats = 3 * n * 4 + n + pt_denoise_atrous_scratch_floats(w, h);
    if (pt_status st = cuda_status(cudaMalloc(&d, floats * sizeof(float)), "pt_denoise_atrous: allocation")) return st;
    float *dc = d, *da = dc + 3 * n, *dn = da + 3 * n, *dv = dn + 3 * n, *dout = dv + n, *ds = dout + 3 * n;
    cudaError_t e = cudaMemcpy(dc, color, 3 * n * 4, cudaMemcpyHostToDevice);
    if (!e) e = cudaMemcpy(da, albedo, 3 * n * 4, cudaMemcpyHostToDevice);
    if (!e) e = cudaMemcpy(dn, normal, 3 * n * 4, cudaMemcpyHostToDevice);
    if (!e) e = cudaMemcpy(dv, variance, n * 4, cudaMemcpyHostToDevice);
    pt_status st = cuda_status(e, "pt_denoise_atrous: copy");
    if (st == PT_OK) st = pt_denoise_atrous_device(w, h, dc, da, dn, dv, dout, ds, nullptr);
    if (st == PT_OK) st = cuda_status(cudaMemcpy(out, dout, 3 * n * 4, cudaMemcpyDeviceToHost), "pt_denoise_atrous: copy back");
    cudaFree(d);
    return st;
}

}  // extern "C"

// ---- the filter without any allocation ------------------------------------------------------
// Some callers of this library cannot call cudaMalloc: a host application that
// owns all device memory through its own pool and does not let plugins
// allocate, or a per-frame loop where an allocation -- which can synchronise
// the device and can fail under memory pressure -- is not allowed. For them
// pt_denoise_atrous_device_noalloc runs the same filter with its scratch in
// the array below, a fixed part of the library's device image: every GPU that
// loads the library holds these 11.5 MB until the process exits, and frames
// are limited to PT_ATROUS_NOALLOC_MAX_PIXELS pixels.
//
// Host code must not hand g_atrous_scratch to a kernel: here its name is only
// a host-side stand-in. The device address is looked up once per CUDA context,
// with that context current, by the first call in it (cudaGetSymbolAddress), so
// the first call on each device -- and the first after a cudaDeviceReset, which
// makes a new context where the module may load elsewhere -- should come
// before any stream capture. Every call
// uses the same array and leaves the last call's data in it; the filter writes
// every scratch value before reading it, so nothing needs clearing, but two
// calls whose work overlaps on the GPU (different streams, or different host
// threads on one device) race on the array and corrupt each other's output.
static __device__ __align__(256) float g_atrous_scratch[11 * size_t(PT_ATROUS_NOALLOC_MAX_PIXELS)];

#include <cuda.h>

#include <map>
#include <mutex>

namespace {
std::mutex g_scratch_lock;
// CUDA context id -> device address of g_atrous_scratch in that context. Keyed
// by context, not device ordinal: after a device reset the module is loaded
// again into a new context (a new id) and its address is looked up again.
std::map<unsigned long long, float*> g_scratch_addr;

// The id of the calling thread's current context (cuCtxGetId, CUDA 12), or 0
// when none is current yet. The driver calls are reached through the runtime's
// entry-point lookup, so the library needs no link against libcuda.
unsigned long long current_context_id() {
    using GetCurrent = CUresult (*)(CUcontext*);
    using GetId = CUresult (*)(CUcontext, unsigned long long*);
    static GetCurrent get_current = nullptr;
    static GetId get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_current = reinterpret_cast<GetCurrent>(p);
        p = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = reinterpret_cast<GetId>(p);
    });
    CUcontext ctx = nullptr;
    unsigned long long id = 0;
    if (!get_current || !get_id || get_current(&ctx) != CUDA_SUCCESS || !ctx || get_id(ctx, &id) != CUDA_SUCCESS)
        return 0;
    return id;
}
}  // namespace

extern "C" pt_status pt_denoise_atrous_device_noalloc(int w, int h, const float* color, const float* albedo,
                                                      const float* normal, const float* variance, float* out,
                                                      void* stream) {
    pt::clear_error();
    if (w <= 0 || h <= 0) return pt::fail(PT_ERR_INVALID_ARG, "pt_denoise_atrous_device_noalloc: bad size");
    if (size_t(w) * size_t(h) > size_t(PT_ATROUS_NOALLOC_MAX_PIXELS))
        return pt::fail(PT_ERR_INVALID_ARG,
                        "pt_denoise_atrous_device_noalloc: " + std::to_string(w) + "x" + std::to_string(h) +
                            " is more than the " + std::to_string(PT_ATROUS_NOALLOC_MAX_PIXELS) +
                            " pixels its built-in scratch holds; use pt_denoise_atrous_device with your own scratch");
    if (!color || !albedo || !normal || !variance || !out)
        return pt::fail(PT_ERR_INVALID_ARG, "pt_denoise_atrous_device_noalloc: null pointer");
    float* scratch = nullptr;
    {
        std::lock_guard<std::mutex> lock(g_scratch_lock);
        const unsigned long long ctx = current_context_id();
        auto it = ctx ? g_scratch_addr.find(ctx) : g_scratch_addr.end();
        if (it == g_scratch_addr.end()) {
            // Looking the symbol up also makes the device's primary context
            // current when no runtime call has yet on this thread.
            void* p = nullptr;
            if (pt_status st = cuda_status(cudaGetSymbolAddress(&p, g_atrous_scratch),
                                           "pt_denoise_atrous_device_noalloc: scratch address"))
                return st;
            scratch = static_cast<float*>(p);
            if (const unsigned long long now = current_context_id()) g_scratch_addr[now] = scratch;
        } else {
            scratch = it->second;
        }
    }
    return pt_denoise_atrous_device(w, h, color, albedo, normal, variance, out, scratch, stream);
}
