// Persistent-thread megakernel path tracer: the lock-step form, and the frames
// and sums of the streaming form (stream_mega.cuh), which renders whatever
// api.cpp's streams() sends there.
//
// The lock-step form. The CPU renderer gives each thread a whole scanline, taken from an atomic
// row counter (src/main.cpp:137-158), and runs samples_per_pixel paths per
// pixel one after another (include/renderer.hpp:366-409). Here each LANE owns
// a pixel, runs its samples one path after another (so the per-pixel sums
// are formed in the same order as the reference's), and advances one bounce
// (or, for scenes without instances, one ray query) per loop trip; when its pixel is finished it takes the next from a global
// counter, warp-aggregated (one atomicAdd per warp per refill). Pixels are
// numbered by 8x4 tiles so a warp's first pixels are neighbours and their
// primary rays coherent. Work per warp is therefore balanced at path
// granularity and no lane waits for another lane's pixel.
#include "kernels.h"
#include "path.cuh"
#include "stream_mega.cuh"

using namespace ptd;

namespace {

constexpr int kTileW = 8, kTileH = 4;

// Resident 128-thread blocks per SM the register allocation targets (5: at
// most 96 registers; +6.6% on the 1024x1024 room frame and +8% on the
// 10,000-instance frame against 3 and 4, which the compiler met with 116-128
// registers; 6 lost).
#ifndef PT_MEGA_MIN_BLOCKS
#define PT_MEGA_MIN_BLOCKS 5
#endif

// The pixel coordinates, sample number and running sum of each lane in
// shared memory instead of registers (they change once per path): 170 -> 100
// bytes of spills in the flat-scene form, room frame +0.8%, images identical.
#ifndef PT_MEGA_SMEM_STATE
#define PT_MEGA_SMEM_STATE 1
#endif

// The path state of each lane in shared memory too, in the flat-scene form:
// no spills left there, room frame +1.0%, random spheres +3.7%; the instanced
// form lost 3% with it and keeps registers (the RNG state moved as well
// gained nothing more).
#ifndef PT_MEGA_SMEM_PATH
#define PT_MEGA_SMEM_PATH 1
#endif

// Scenes without instances trace one query per loop trip (a path ray or a
// shadow ray) through one traversal call site: lanes on shadow rays traverse
// alongside lanes on path rays instead of after them. Same images; +28.6% on
// the 1920x1080x16 random-spheres frame (2,797 -> 3,597 Mrays/s), the room
// frame within 0.5%, and at four blocks per SM 7% slower.
#ifndef PT_MEGA_ONE_QUERY
#define PT_MEGA_ONE_QUERY 1
#endif

// Traversal-stack entries per lane in shared memory (the rest in its local
// array). Measured on the 1024x1024 room frame, the 1080p random-spheres
// frame and the 10,000-instance frame (identical images): 0 is fastest; 2, 4
// and 8 entries lost 1-3%, 1-5% and 1-6% (the kernel already keeps 15 KB of
// path state per block in shared memory; a stack on top leaves the SM's L1
// data cache 60 KB smaller for node and primitive fetches), 16 lost 14%.
// The wavefront stages and ray-query kernels, with no other shared state,
// gain from it and use PT_SH_STACK.
#ifndef PT_MEGA_SH_STACK
#define PT_MEGA_SH_STACK 0
#endif

// A second flat-scene form whose stack has 8-byte entries (PackedStack,
// PT_TREES_FLAT8), launched for flat scenes whose leaves fit them
// (PtSceneDev::stack_pack8) and whose nodes and leaf slots take more than
// PT_MEGA_PACK_MIN_KIB: the deep local array is 768 instead of 1,536 bytes
// per lane, and its hot entries take half the L1 lines. Measured on one
// B200 with identical images (Mrays/s, 16-byte -> 8-byte): room frames with
// the icosphere at 1,290 / 5,130 / 20,490 / 81,930 triangles (1024x1024,
// 16 spp; about 0.1, 0.4, 1.8, 7 MB of nodes and slots) 3,191 -> 3,325 /
// 2,921 -> 3,030 / 2,737 -> 2,827 / 2,586 -> 2,661 (+4.2 / +3.7 / +3.3 /
// +2.9%), the 64-spp bench frame 2,608 -> 2,684; the 1080p random spheres
// (488 spheres, about 44 KB) 4,210 -> 4,191 and 4,222 -> 4,165 in two runs
// (-0.5 / -1.3%: the packing instructions without an L1 gain), hence the
// threshold between the two. Shared-memory entries on top
// (PT_MEGA_SH_STACK8 = 4, 8, 12: 4, 8, 12 KB per block) lost 4-6% on the
// room and random-spheres frames.
#ifndef PT_MEGA_PACK_STACK
#define PT_MEGA_PACK_STACK 1
#endif
#ifndef PT_MEGA_PACK_MIN_KIB
#define PT_MEGA_PACK_MIN_KIB 64
#endif
#ifndef PT_MEGA_SH_STACK8
#define PT_MEGA_SH_STACK8 0
#endif


// EXT: the extended light sampling of PT_FLAG_NEE_EXTENDED (production
// streams only); false compiles exactly the reference's estimator.
template <bool AUX, bool SNAP, int TREES, bool TEX, bool EXT>
__global__ void __launch_bounds__(128, PT_MEGA_MIN_BLOCKS) megakernel(PtSceneDev S, PtRenderParams P, uint32_t tiles_x,
                                                  uint32_t total_items) {
    PT_FORM_STACK(stack, TREES, 128, PT_MEGA_SH_STACK, PT_MEGA_SH_STACK8);
    // With the extended light sampling, SMALL but for the large flat scenes and
    // textures (640x360, us, SMALL and FULL: room of 81,920 triangles, 8 samples
    // 5,240, 4,960; textured room with guides, 1 sample 1,171, 1,086; but 488
    // spheres, 8 samples 1,900, 2,550, the emissive meshes 4,700, 5,770).
    constexpr int CODE = !EXT ? CODE_LOOP : TEX || TREES == PT_TREES_FLAT8 ? CODE_FULL : CODE_SMALL;
    // the traversal form the queries compile (PT_TREES_FLAT8 is the flat one
    // with the other stack)
    constexpr int QT = TREES == PT_TREES_FLAT8 ? int(PT_TREES_FLAT) : TREES;
    const int lane = threadIdx.x & 31;
    const Cam cam = {mk(P.cam.origin[0], P.cam.origin[1], P.cam.origin[2]),
                     mk(P.cam.llc[0], P.cam.llc[1], P.cam.llc[2]),
                     mk(P.cam.horizontal[0], P.cam.horizontal[1], P.cam.horizontal[2]),
                     mk(P.cam.vertical[0], P.cam.vertical[1], P.cam.vertical[2])};
    const float scale = 1.0f / float(P.spp);
    const float wm1 = float(P.width - 1), hm1 = float(P.height - 1);

    unsigned long long rays = 0;
    bool exhausted = false, has_pixel = false, in_path = false;
#if PT_MEGA_SMEM_STATE
    // The pixel, its sample number and its running sum change once per
    // path: they live in shared memory, leaving registers to the traversal.
    __shared__ int s_pix[3][128];
    __shared__ V s_acc[128];
    int& pi = s_pix[0][threadIdx.x];
    int& pj = s_pix[1][threadIdx.x];
    int& s = s_pix[2][threadIdx.x];
    V& acc = s_acc[threadIdx.x];
    pi = pj = s = 0;
    acc = mk(0, 0, 0);
    V acc_albedo = mk(0, 0, 0), acc_normal = mk(0, 0, 0);
#else
    int pi = 0, pj = 0, s = 0;
    V acc = mk(0, 0, 0), acc_albedo = mk(0, 0, 0), acc_normal = mk(0, 0, 0);
#endif
    float lum2 = 0;
    // Flat-scene form: the path (ray, throughput, radiance, bounce) in shared
    // memory too, read into registers where a query or shading needs it.
    constexpr bool SMEM_PATH = PT_MEGA_SMEM_PATH && QT == PT_TREES_FLAT;
    __shared__ Path s_path[SMEM_PATH ? 128 : 1];
    Path local_path;
    Path& path = SMEM_PATH ? s_path[threadIdx.x] : local_path;
    First first = {mk(0, 0, 0), mk(0, 0, 0)};
    Sampler smp;
    Rng rng;
    bool overflow = false;
    // Single-query form: the pending shadow ray (origin, direction, t_max,
    // unblocked value) of each lane, kept in shared memory between trips.
    constexpr bool ONE_QUERY = PT_MEGA_ONE_QUERY && QT == PT_TREES_FLAT;
    __shared__ float pend[10][ONE_QUERY ? 128 : 1];
    bool shadow_pending = false, done_after_shadow = false;

    while (true) {
        // Refill lanes without a pixel.
        const bool need = !has_pixel && !exhausted;
        const unsigned want = __ballot_sync(0xffffffffu, need);
        if (want) {
            const int leader = __ffs(want) - 1;
            uint32_t base = 0;
            if (lane == leader) base = atomicAdd(P.work, uint32_t(__popc(want)));
            base = __shfl_sync(0xffffffffu, base, leader);
            if (need) {
                const uint32_t item = base + __popc(want & ((1u << lane) - 1u));
                if (item >= total_items) {
                    exhausted = true;
                } else {
                    const uint32_t tile = item >> 5, l = item & 31u;
                    pi = int((tile % tiles_x) * kTileW + (l & 7u));
                    pj = P.row0 + int((tile / tiles_x) * kTileH + (l >> 3));
                    if (pi < P.width && pj < P.row0 + P.rows) {
                        has_pixel = true;
                        s = 0;
                        in_path = false;
                        acc = acc_albedo = acc_normal = mk(0, 0, 0);
                        lum2 = 0;
                    }
                }
            }
        }
        if (__all_sync(0xffffffffu, exhausted)) break;
        if (!has_pixel) continue;

        if (!in_path) {
            if (P.depth <= 0 || P.spp <= 0) {
                s = P.spp;  // nothing to trace: every sample is black
            } else {
                // render_row_impl's sample loop body (:379-385)
                const uint32_t idx = uint32_t(P.first_sample + s);
                smp.begin(P.seed, pi, pj, idx);
                float du, dv;
                smp.sample_2d(0, rng, du, dv);
                const float u = (float(pi) + du) / wm1;
                const float v = (float(pj) + dv) / hm1;
                path.o = cam.origin;
                path.d = cam.llc + cam.horizontal * u + cam.vertical * v - cam.origin;
                path.tp = mk(1, 1, 1);
                path.rad = mk(0, 0, 0);
                path.bounce = 0;
                path.sampled = false;
                path.mis_pdf = 0;
                first = {mk(0, 0, 0), mk(0, 0, 0)};
                if (SNAP) {
                    const uint64_t* st = P.states + 4 * ((size_t(pj) * P.width + pi) * P.spp + s);
                    rng.s0 = st[0];
                    rng.s1 = st[1];
                    rng.s2 = st[2];
                    rng.s3 = st[3];
                } else {
                    rng.seed(sample_stream_seed(P.seed, pi, pj, idx));
                }
                in_path = true;
            }
        }

        if constexpr (ONE_QUERY) {
            if (in_path && query_trip<AUX, TEX, EXT, CODE>(S, path, P.depth, smp, rng, first, pend, shadow_pending,
                                                done_after_shadow, stack, rays, overflow)) {
                acc = acc + path.rad;
                if (AUX) {
                    acc_albedo = acc_albedo + first.albedo;
                    acc_normal = acc_normal + first.normal;
                    const float l = luminance(path.rad);
                    lum2 += l * l;
                }
                in_path = false;
                ++s;
            }
        } else if (in_path) {
            // One iteration of ray_color's bounce loop.
            ++rays;
            smp.set_bounce(path.bounce);
            float t = 1000.0f;
            Hit h;
            Counts cnt;
            Rec rec;
            bool ok = closest<false, QT>(S, path.o, path.d, 0.001f, t, h, stack, cnt);
            if (!ok) {
                overflow = true;
                h.kind = PT_HIT_NONE;
            }
            const bool hit = h.kind != PT_HIT_NONE;
            if (hit) fill<TEX, EXT>(S, h, path.o, path.d, t, rec);
            bool nee;
            Shadow sh;
            const int step = shade<AUX, TEX, EXT, CODE>(S, path, hit, rec, P.depth, smp, rng, first, nee, sh, rays);
            if (nee) {
                bool ovf = false;
                if (!occluded<false, QT>(S, sh.o, sh.d, 0.001f, sh.t_max, stack, cnt, &ovf))
                    path.rad = path.rad + sh.value;
                overflow |= ovf;
            }
            if (step == STEP_DONE) {
                acc = acc + path.rad;
                if (AUX) {
                    acc_albedo = acc_albedo + first.albedo;
                    acc_normal = acc_normal + first.normal;
                    const float l = luminance(path.rad);
                    lum2 += l * l;
                }
                in_path = false;
                ++s;
            }
        }

        if (s >= P.spp) {
            const int row = P.flip ? (P.height - 1 - pj) : (pj - P.row0);
            const size_t px = size_t(row) * P.width + pi;
            P.out[3 * px + 0] = acc.x * scale;
            P.out[3 * px + 1] = acc.y * scale;
            P.out[3 * px + 2] = acc.z * scale;
            if (AUX) {
                float* a = P.aux + 7 * px;
                a[0] = acc_albedo.x * scale;
                a[1] = acc_albedo.y * scale;
                a[2] = acc_albedo.z * scale;
                a[3] = acc_normal.x * scale;
                a[4] = acc_normal.y * scale;
                a[5] = acc_normal.z * scale;
                a[6] = lum2 * scale;
            }
            has_pixel = false;
        }
    }

    // Ray count: warp sum, one atomic per warp.
    unsigned long long total = rays;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) total += __shfl_down_sync(0xffffffffu, total, off);
    if (lane == 0 && P.rays) atomicAdd(P.rays, total);
    if (__any_sync(0xffffffffu, overflow) && lane == 0) atomicOr(S.status, PT_DEV_ERR_STACK);
}

// ---- the streaming form (stream_mega.cuh) over one frame -----------------------------------------
// `per_pixel` samples of every pixel from sample `first` on, item = pixel *
// per_pixel + sample, so that neighbouring items are samples of one pixel.
// Pixels are numbered by tiles of 8 x 4, rows of a short image by runs of 32.
struct PtSampleLaunch {
    uint32_t items, pixels, per_pixel, first, tiles_x;
    int tile_w, tile_h;
    int contexts;   // paths a warp keeps in flight
    float* samples; // radiance of each sample, 3 floats at sample * pixels + pixel
    float* guides;  // first hit's albedo and normal, 6 floats, with auxiliary outputs
};

__device__ __forceinline__ void sample_pixel(const PtSampleLaunch& L, const PtRenderParams& P, uint32_t pixel, int& pi,
                                             int& pj) {
    const uint32_t tile = pixel >> 5, l = pixel & 31u;
    const uint32_t ty = tile / L.tiles_x;
    const uint32_t sh = L.tile_w == 32 ? 5u : 3u;
    pi = int((tile - ty * L.tiles_x) << sh) + int(l & (uint32_t(L.tile_w) - 1u));
    pj = P.row0 + int(ty) * L.tile_h + int(l >> sh);
}

template <bool SNAP>
struct OneFrame {
    static constexpr bool kManyScenes = false;
    PtSceneDev S;
    PtRenderParams P;
    PtSampleLaunch L;
    __device__ __forceinline__ const PtSceneDev& scene(uint32_t) const { return S; }
    __device__ __forceinline__ int depth(uint32_t) const { return P.depth; }
    __device__ __forceinline__ uint32_t items() const { return L.items; }
    __device__ __forceinline__ int contexts() const { return L.contexts; }
    __device__ __forceinline__ unsigned int* work() const { return P.work; }
    __device__ __forceinline__ unsigned long long* rays() const { return P.rays; }
    __device__ __forceinline__ unsigned int* status() const { return S.status; }
    __device__ __forceinline__ float* samples() const { return L.samples; }
    __device__ __forceinline__ float* guides() const { return L.guides; }
    __device__ __forceinline__ void started() const {}
    // False for an item of a tile past the image's edge.
    __device__ __forceinline__ bool locate(uint32_t item, SampleAt& a) const {
        const uint32_t pixel = item / L.per_pixel, s = item - pixel * L.per_pixel;
        sample_pixel(L, P, pixel, a.i, a.j);
        a.sample = uint32_t(P.first_sample) + L.first + s;
        a.place = s * L.pixels + pixel;
        a.scene = 0;
        return a.i < P.width && a.j < P.row0 + P.rows;
    }
    __device__ __forceinline__ uint64_t seed(const SampleAt&) const { return P.seed; }
    __device__ __forceinline__ void ray(const SampleAt& a, float du, float dv, V& o, V& d) const {
        const float u = (float(a.i) + du) / float(P.width - 1);
        const float v = (float(a.j) + dv) / float(P.height - 1);
        o = mk(P.cam.origin[0], P.cam.origin[1], P.cam.origin[2]);
        d = mk(P.cam.llc[0], P.cam.llc[1], P.cam.llc[2]) +
            mk(P.cam.horizontal[0], P.cam.horizontal[1], P.cam.horizontal[2]) * u +
            mk(P.cam.vertical[0], P.cam.vertical[1], P.cam.vertical[2]) * v - o;
    }
    __device__ __forceinline__ void start(const SampleAt& a, Rng& rng) const {
        if (SNAP) {
            const uint64_t* st =
                P.states + 4 * ((size_t(a.j) * P.width + a.i) * P.spp + (a.sample - uint32_t(P.first_sample)));
            rng.s0 = st[0];
            rng.s1 = st[1];
            rng.s2 = st[2];
            rng.s3 = st[3];
        } else {
            rng.seed(sample_stream_seed(P.seed, a.i, a.j, a.sample));
        }
    }
};

// Adds one launch's samples to the pixels' running sums in sample order -- the
// order, and so the rounding, of a pixel's samples rendered one after another
// -- and scales them after the last one.
template <bool AUX>
__global__ void __launch_bounds__(256) sum_samples(PtRenderParams P, PtSampleLaunch L) {
    const uint32_t pixel = blockIdx.x * blockDim.x + threadIdx.x;
    if (pixel >= L.pixels) return;
    int pi, pj;
    sample_pixel(L, P, pixel, pi, pj);
    if (pi >= P.width || pj >= P.row0 + P.rows) return;
    const int row = P.flip ? (P.height - 1 - pj) : (pj - P.row0);
    const size_t px = size_t(row) * P.width + pi;
    float* out = P.out + 3 * px;
    float* aux = AUX ? P.aux + 7 * px : nullptr;
    float a[7] = {0, 0, 0, 0, 0, 0, 0};
    V acc = mk(0, 0, 0);
    if (L.first) {
        acc = mk(out[0], out[1], out[2]);
        if (AUX)
            for (int i = 0; i < 7; ++i) a[i] = aux[i];
    }
    for (uint32_t s = 0; s < L.per_pixel; ++s) {
        const size_t at = size_t(s) * L.pixels + pixel;
        const float* r = L.samples + 3 * at;
        const V rad = mk(r[0], r[1], r[2]);
        acc = acc + rad;
        if (AUX) {
            const float* g = L.guides + 6 * at;
            for (int i = 0; i < 6; ++i) a[i] = a[i] + g[i];
            const float l = luminance(rad);
            a[6] += l * l;
        }
    }
    const float scale = L.first + L.per_pixel >= uint32_t(P.spp) ? 1.0f / float(P.spp) : 1.0f;
    out[0] = acc.x * scale;
    out[1] = acc.y * scale;
    out[2] = acc.z * scale;
    if (AUX)
        for (int i = 0; i < 7; ++i) aux[i] = a[i] * scale;
}

template <bool AUX, bool SNAP, bool INST, bool TEX, bool EXT>
cudaError_t launch_s(const PtSceneDev& S, const PtRenderParams& p, PtSampleLaunch L, int sms, int& blocks_per_sm,
                     cudaStream_t stream) {
    if (!blocks_per_sm)
        blocks_per_sm = pt_resident_blocks(
            reinterpret_cast<const void*>(megakernel_stream<AUX, INST, TEX, EXT, OneFrame<SNAP>>), 128, 0);
    const uint32_t warps = uint32_t(sms * blocks_per_sm) * 4u;
    L.contexts = int((L.items + warps - 1) / warps);
    megakernel_stream<AUX, INST, TEX, EXT, OneFrame<SNAP>><<<sms * blocks_per_sm, 128, 0, stream>>>({S, p, L});
    sum_samples<AUX><<<(L.pixels + 255) / 256, 256, 0, stream>>>(p, L);
    return cudaGetLastError();
}

template <bool INST, bool TEX>
cudaError_t launch_stream(const PtSceneDev& S, const PtRenderParams& p, const PtSampleLaunch& L, int sms,
                          int& per_sm, cudaStream_t stream) {
    const bool aux = p.aux != nullptr, snap = p.rng_mode == 1;
    if (p.nee_ext)  // production streams only (the host refuses it with snapshots)
        return aux ? launch_s<true, false, INST, TEX, true>(S, p, L, sms, per_sm, stream)
                   : launch_s<false, false, INST, TEX, true>(S, p, L, sms, per_sm, stream);
    if (aux)
        return snap ? launch_s<true, true, INST, TEX, false>(S, p, L, sms, per_sm, stream)
                    : launch_s<true, false, INST, TEX, false>(S, p, L, sms, per_sm, stream);
    return snap ? launch_s<false, true, INST, TEX, false>(S, p, L, sms, per_sm, stream)
                : launch_s<false, false, INST, TEX, false>(S, p, L, sms, per_sm, stream);
}

template <bool AUX, bool SNAP, int TREES, bool TEX, bool EXT>
cudaError_t launch(const PtSceneDev& S, const PtRenderParams& p, const PtLaunchShape& shape, cudaStream_t stream) {
    const uint32_t tiles_x = uint32_t((p.width + kTileW - 1) / kTileW);
    const uint32_t tiles_y = uint32_t((p.rows + kTileH - 1) / kTileH);
    const uint32_t total = tiles_x * tiles_y * 32u;
    megakernel<AUX, SNAP, TREES, TEX, EXT><<<shape.blocks, shape.threads, 0, stream>>>(S, p, tiles_x, total);
    return cudaGetLastError();
}

template <int TREES, bool TEX>
cudaError_t launch_form(const PtSceneDev& S, const PtRenderParams& p, const PtLaunchShape& shape,
                        cudaStream_t stream) {
    const bool aux = p.aux != nullptr, snap = p.rng_mode == 1;
    if (p.nee_ext)  // production streams only (the host refuses it with snapshots)
        return aux ? launch<true, false, TREES, TEX, true>(S, p, shape, stream)
                   : launch<false, false, TREES, TEX, true>(S, p, shape, stream);
    if (aux)
        return snap ? launch<true, true, TREES, TEX, false>(S, p, shape, stream)
                    : launch<true, false, TREES, TEX, false>(S, p, shape, stream);
    return snap ? launch<false, true, TREES, TEX, false>(S, p, shape, stream)
                : launch<false, false, TREES, TEX, false>(S, p, shape, stream);
}

template <int TREES, bool TEX>
int occupancy(int threads, bool aux, bool snap, bool ext) {
    const void* fn = ext ? (aux ? reinterpret_cast<const void*>(megakernel<true, false, TREES, TEX, true>)
                                : reinterpret_cast<const void*>(megakernel<false, false, TREES, TEX, true>))
                   : aux ? (snap ? reinterpret_cast<const void*>(megakernel<true, true, TREES, TEX, false>)
                                 : reinterpret_cast<const void*>(megakernel<true, false, TREES, TEX, false>))
                         : (snap ? reinterpret_cast<const void*>(megakernel<false, true, TREES, TEX, false>)
                                 : reinterpret_cast<const void*>(megakernel<false, false, TREES, TEX, false>));
    return pt_resident_blocks(fn, threads, 0);
}

// The single-loop traversal for scenes with instances, one loop per tree
// otherwise; texture code only in the kernels for scenes with textures; for
// large flat scenes without textures whose leaves fit them, 8-byte stack
// entries.
bool one_loop(const PtSceneDev& S) { return S.use_bvh && S.inst_root != PT_NONE; }
bool flat_only(const PtSceneDev& S) { return S.inst_root == PT_NONE && S.n_instances == 0; }
bool flat8(const PtSceneDev& S) {
    return PT_MEGA_PACK_STACK && S.use_bvh && S.stack_pack8 && S.tree_kib > PT_MEGA_PACK_MIN_KIB;
}

}  // namespace

cudaError_t pt_launch_megakernel(const PtSceneDev& S, const PtRenderParams& p, const PtLaunchShape& shape,
                                 cudaStream_t stream) {
    if (S.has_textures)
        return one_loop(S)   ? launch_form<PT_TREES_ONE, true>(S, p, shape, stream)
               : flat_only(S) ? launch_form<PT_TREES_FLAT, true>(S, p, shape, stream)
                              : launch_form<PT_TREES_EACH, true>(S, p, shape, stream);
    if (one_loop(S)) return launch_form<PT_TREES_ONE, false>(S, p, shape, stream);
    if (!flat_only(S)) return launch_form<PT_TREES_EACH, false>(S, p, shape, stream);
    return flat8(S) ? launch_form<PT_TREES_FLAT8, false>(S, p, shape, stream)
                    : launch_form<PT_TREES_FLAT, false>(S, p, shape, stream);
}

int pt_megakernel_blocks_per_sm(const PtSceneDev& S, int threads, bool aux, bool snapshot, bool ext) {
    if (S.has_textures)
        return one_loop(S)   ? occupancy<PT_TREES_ONE, true>(threads, aux, snapshot, ext)
               : flat_only(S) ? occupancy<PT_TREES_FLAT, true>(threads, aux, snapshot, ext)
                              : occupancy<PT_TREES_EACH, true>(threads, aux, snapshot, ext);
    if (one_loop(S)) return occupancy<PT_TREES_ONE, false>(threads, aux, snapshot, ext);
    if (!flat_only(S)) return occupancy<PT_TREES_EACH, false>(threads, aux, snapshot, ext);
    return flat8(S) ? occupancy<PT_TREES_FLAT8, false>(threads, aux, snapshot, ext)
                    : occupancy<PT_TREES_FLAT, false>(threads, aux, snapshot, ext);
}

size_t pt_sample_bytes(const PtRenderParams& p) {
    const int tile_h = p.rows >= 4 ? 4 : 1, tile_w = 32 / tile_h;
    const size_t tiles = size_t((p.width + tile_w - 1) / tile_w) * size_t((p.rows + tile_h - 1) / tile_h);
    return tiles * 32 * (p.aux ? 36 : 12);
}

cudaError_t pt_launch_samples(const PtSceneDev& S, const PtRenderParams& p, int first, int count, float* buffer, int sms,
                              int& per_sm, cudaStream_t stream) {
    PtSampleLaunch L{};
    L.tile_h = p.rows >= 4 ? 4 : 1;
    L.tile_w = 32 / L.tile_h;
    L.tiles_x = uint32_t((p.width + L.tile_w - 1) / L.tile_w);
    L.pixels = 32u * L.tiles_x * uint32_t((p.rows + L.tile_h - 1) / L.tile_h);
    L.per_pixel = uint32_t(count);
    L.first = uint32_t(first);
    L.items = L.pixels * L.per_pixel;
    L.samples = buffer;
    L.guides = p.aux ? buffer + 3 * size_t(L.items) : nullptr;
    const bool flat = flat_only(S);
    if (S.has_textures)
        return flat ? launch_stream<false, true>(S, p, L, sms, per_sm, stream) : launch_stream<true, true>(S, p, L, sms, per_sm, stream);
    return flat ? launch_stream<false, false>(S, p, L, sms, per_sm, stream) : launch_stream<true, false>(S, p, L, sms, per_sm, stream);
}
