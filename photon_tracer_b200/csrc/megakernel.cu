// Persistent-thread megakernel path tracer.
//
// The CPU renderer gives each thread a whole scanline, taken from an atomic
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
#include "stream.cuh"

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
            if (in_path && query_trip<AUX, TEX, EXT>(S, path, P.depth, smp, rng, first, pend, shadow_pending,
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
            const int step = shade<AUX, TEX, EXT>(S, path, hit, rec, P.depth, smp, rng, first, nee, sh, rays);
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

// ---- the streaming form ----------------------------------------------------------------------
// The lock-step form above is bound by divergence: a room-frame query takes
// 250 warp instructions at 6.6 threads each, because a warp walks until its
// longest ray is done (4.7 nodes on average, 22 for the longest of 32) and
// then shades the lanes that happen to hold a path ray. Here a warp keeps up
// to 64 paths (contexts) in shared memory and works in phases:
//   shade  32 contexts whose ray was traced, with all lanes busy; ended
//          samples are written out and their contexts take the next sample;
//   hand   lanes whose walk is done give their context back and take the
//          next ray (a shadow ray's context goes straight on to its path ray);
//   walk   node and leaf steps (stream.cuh), while enough lanes stand at them.
// 64 contexts are 32 walking and 32 waiting, so that lanes run out of rays just
// when 32 contexts are ready to shade (48: 10% slower, 40: 20%). It takes 140
// warp instructions per query at 16.7 threads. What bounds it now: latency of
// node fetches (L1 hits 78%, long-scoreboard 3.0 of 10 stall cycles per
// issue) and instruction fetch (65 KB of code, 2.2 of 10).
//
// A work item is one sample, not one pixel, so that a small frame fills the
// GPU and a large one ends without a tail of whole pixels; each sample's
// radiance goes to a buffer that sum_samples adds up in sample order, which
// rounds as one pixel's samples rendered in turn. Images are the lock-step
// form's bit for bit. Measured on one B200, lock-step -> streaming: 1024x1024
// room, 64 samples 145.0 -> 95.8 ms; 960x540, 16 samples of 10,000 instances
// 64.3 -> 37.1 ms; 400x225, 16 samples of random spheres 1.86 -> 1.22 ms; one
// such row of 400 pixels 0.71 -> 0.16 ms.
//
// Five resident blocks per SM (96 registers; 4: room 13% slower), four for
// the forms with more live state, auxiliary outputs (1080p room, 4 samples:
// 10.0 ms, 5 blocks 11.1) and extended light sampling (8.5 ms, 5 blocks 8.9).
// Fetch and node thresholds are flat optima (4..12, 8..12: within 2%).
constexpr int kContexts = 64, kShade = 32, kFetch = 8, kNodes = 12, kStreamBlocks = 5;

// A path's state between the phases, in shared memory: word `field` of
// context c is ctx[field][c].
enum : int {
    C_O = 0,       // origin of the next ray, 3
    C_D = 3,       // direction of the path's next ray, 3
    C_SD = 6,      // shadow ray's direction, 3; else the hit's t, u, v
    C_ST = 9,      // shadow ray's t_max; else the hit's kind
    C_SV = 10,     // light sample if unblocked, 3; else the hit's index, instance
    C_TP = 13,     // throughput, 3
    C_RAD = 16,    // radiance, 3
    C_FLAGS = 19,  // bounce in bits 0-15, and the CF_ bits
    C_RNG = 20,    // 8
    C_SEED = 28,   // the sampler's pixel seed
    C_INDEX = 29,  // the sampler's index: the sample's number
    C_ITEM = 30,   // the sample's place in the launch
    C_MIS = 31     // EXT
};
enum : uint32_t { CF_BOUNCE = 0xffffu, CF_SAMPLED = 1u << 16, CF_SHADOW = 1u << 17, CF_ENDED = 1u << 18, CF_LIVE = 1u << 19 };

// One launch over samples: `per_pixel` samples of every pixel from sample
// `first` on, item = pixel * per_pixel + sample, so that neighbouring items
// are samples of one pixel. Pixels are numbered by tiles of tile_w x tile_h.
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

template <bool AUX, bool SNAP, bool INST, bool TEX, bool EXT>
__global__ void __launch_bounds__(128, AUX || EXT ? kStreamBlocks - 1 : kStreamBlocks)
    megakernel_stream(PtSceneDev S, PtRenderParams P, PtSampleLaunch L) {
    constexpr int C = kContexts, FIELDS = EXT ? 32 : 31;
    PT_WORD_STACK(stack, 128, 0);
    constexpr unsigned ALL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    __shared__ uint32_t s_ctx[4][FIELDS][C];
    __shared__ uint8_t s_ray_q[4][64], s_shade_q[4][64];
    uint32_t(&ctx)[FIELDS][C] = s_ctx[threadIdx.x >> 5];
    uint8_t* const ray_q = s_ray_q[threadIdx.x >> 5];
    uint8_t* const shade_q = s_shade_q[threadIdx.x >> 5];
    auto getf = [&](int f, int c) { return __uint_as_float(ctx[f][c]); };
    auto setf = [&](int f, int c, float x) { ctx[f][c] = __float_as_uint(x); };
    auto getv = [&](int f, int c) { return mk(getf(f, c), getf(f + 1, c), getf(f + 2, c)); };
    auto setv = [&](int f, int c, V x) {
        setf(f, c, x.x);
        setf(f + 1, c, x.y);
        setf(f + 2, c, x.z);
    };

    const int contexts = min(L.contexts, C);
    for (int c = lane; c < contexts; c += 32) {
        ctx[C_FLAGS][c] = CF_ENDED;
        shade_q[c] = uint8_t(c);
    }
    __syncwarp();
    // queue heads and lengths, the same in every lane
    int ray_h = 0, ray_n = 0, shade_h = 0, shade_n = contexts;
    unsigned long long rays = 0;
    bool overflow = false, shadow = false;
    int state = WALK_DONE, c = -1;  // c: the context this lane walks for
    Walk<INST> w;
    w.top = 0;
    w.h.kind = PT_HIT_NONE;

    while (true) {
        const unsigned walking = __ballot_sync(ALL, state != WALK_DONE);
        if (shade_n >= kShade || (shade_n > 0 && ray_n == 0 && shade_n >= __popc(walking))) {
            // Shade up to 32 contexts.
            const int m = min(32, shade_n);
            const bool act = lane < m;
            const int k = act ? shade_q[(shade_h + lane) & 63] : 0;
            shade_h += m;
            shade_n -= m;
            uint32_t flags = act ? ctx[C_FLAGS][k] : 0u;
            bool ended = act && (flags & CF_ENDED), push = false;
            Rng rng;
            Sampler smp;
            if (act && !ended) {
                Path path;
                path.o = getv(C_O, k);
                path.d = getv(C_D, k);
                path.tp = getv(C_TP, k);
                path.rad = getv(C_RAD, k);
                path.bounce = int(flags & CF_BOUNCE);
                path.sampled = (flags & CF_SAMPLED) != 0;
                if (EXT) path.mis_pdf = getf(C_MIS, k);
                uint64_t r[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) r[i] = ctx[C_RNG + 2 * i][k] | (uint64_t(ctx[C_RNG + 2 * i + 1][k]) << 32);
                rng.s0 = r[0];
                rng.s1 = r[1];
                rng.s2 = r[2];
                rng.s3 = r[3];
                smp.pixel_seed = ctx[C_SEED][k];
                smp.index = ctx[C_INDEX][k];
                smp.set_bounce(path.bounce);
                Hit h;
                h.kind = ctx[C_ST][k];
                h.index = ctx[C_SV][k];
                h.inst = INST ? ctx[C_SV + 1][k] : 0u;
                h.u = getf(C_SD + 1, k);
                h.v = getf(C_SD + 2, k);
                const bool hit = h.kind != PT_HIT_NONE;
                Rec rec;
                if (hit) fill<TEX, EXT>(S, h, path.o, path.d, getf(C_SD, k), rec);
                First first;
                const bool primary = AUX && path.bounce == 0;
                bool nee;
                Shadow sh;
                const bool done =
                    shade<AUX, TEX, EXT>(S, path, hit, rec, P.depth, smp, rng, first, nee, sh, rays) == STEP_DONE;
                if (primary) {  // the first hit's guides
                    float* g = L.guides + 6 * size_t(ctx[C_ITEM][k]);
                    g[0] = first.albedo.x;
                    g[1] = first.albedo.y;
                    g[2] = first.albedo.z;
                    g[3] = first.normal.x;
                    g[4] = first.normal.y;
                    g[5] = first.normal.z;
                }
                setv(C_RAD, k, path.rad);
                flags = CF_LIVE | (uint32_t(path.bounce) & CF_BOUNCE) | (path.sampled ? CF_SAMPLED : 0u);
                if (!done) {
                    setv(C_O, k, path.o);
                    setv(C_D, k, path.d);
                    setv(C_TP, k, path.tp);
                    if (EXT) setf(C_MIS, k, path.mis_pdf);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint64_t x = i == 0 ? rng.s0 : i == 1 ? rng.s1 : i == 2 ? rng.s2 : rng.s3;
                        ctx[C_RNG + 2 * i][k] = uint32_t(x);
                        ctx[C_RNG + 2 * i + 1][k] = uint32_t(x >> 32);
                    }
                }
                if (nee) {
                    setv(C_O, k, sh.o);
                    setv(C_SD, k, sh.d);
                    setf(C_ST, k, sh.t_max);
                    setv(C_SV, k, sh.value);
                    flags |= CF_SHADOW | (done ? CF_ENDED : 0u);
                    push = true;
                } else if (done) {
                    ended = true;
                } else {
                    push = true;
                }
            }
            if (ended && (flags & CF_LIVE)) {
                const V rad = getv(C_RAD, k);
                float* out = L.samples + 3 * size_t(ctx[C_ITEM][k]);
                out[0] = rad.x;
                out[1] = rad.y;
                out[2] = rad.z;
            }
            // Contexts whose sample ended take the next ones; those past the
            // last are dropped.
            bool need = ended, fresh = false;
            int pi = 0, pj = 0;
            uint32_t s = 0, place = 0;
            while (true) {
                const unsigned want = __ballot_sync(ALL, need);
                if (!want) break;
                const int leader = __ffs(want) - 1;
                uint32_t base = 0;
                if (lane == leader) base = atomicAdd(P.work, uint32_t(__popc(want)));
                base = __shfl_sync(ALL, base, leader);
                if (need) {
                    const uint32_t item = base + __popc(want & ((1u << lane) - 1u));
                    if (item >= L.items) {
                        need = false;
                    } else {
                        const uint32_t pixel = item / L.per_pixel;
                        s = item - pixel * L.per_pixel;
                        place = s * L.pixels + pixel;
                        sample_pixel(L, P, pixel, pi, pj);
                        if (pi < P.width && pj < P.row0 + P.rows) {
                            need = false;
                            fresh = true;
                        }
                    }
                }
            }
            if (fresh) {
                // render_row_impl's sample loop body (:379-385)
                const uint32_t idx = uint32_t(P.first_sample) + L.first + s;
                smp.begin(P.seed, pi, pj, idx);
                float du, dv;
                smp.sample_2d(0, rng, du, dv);
                const float u = (float(pi) + du) / float(P.width - 1);
                const float v = (float(pj) + dv) / float(P.height - 1);
                const V org = mk(P.cam.origin[0], P.cam.origin[1], P.cam.origin[2]);
                setv(C_O, k, org);
                setv(C_D, k,
                     mk(P.cam.llc[0], P.cam.llc[1], P.cam.llc[2]) +
                         mk(P.cam.horizontal[0], P.cam.horizontal[1], P.cam.horizontal[2]) * u +
                         mk(P.cam.vertical[0], P.cam.vertical[1], P.cam.vertical[2]) * v - org);
                setv(C_TP, k, mk(1, 1, 1));
                setv(C_RAD, k, mk(0, 0, 0));
                if (EXT) setf(C_MIS, k, 0);
                if (SNAP) {
                    const uint64_t* st = P.states + 4 * ((size_t(pj) * P.width + pi) * P.spp + L.first + s);
                    rng.s0 = st[0];
                    rng.s1 = st[1];
                    rng.s2 = st[2];
                    rng.s3 = st[3];
                } else {
                    rng.seed(sample_stream_seed(P.seed, pi, pj, idx));
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint64_t x = i == 0 ? rng.s0 : i == 1 ? rng.s1 : i == 2 ? rng.s2 : rng.s3;
                    ctx[C_RNG + 2 * i][k] = uint32_t(x);
                    ctx[C_RNG + 2 * i + 1][k] = uint32_t(x >> 32);
                }
                ctx[C_SEED][k] = smp.pixel_seed;
                ctx[C_INDEX][k] = idx;
                ctx[C_ITEM][k] = place;
                flags = CF_LIVE;
                push = true;
            }
            if (push) ctx[C_FLAGS][k] = flags;
            const unsigned pushed = __ballot_sync(ALL, push);
            if (push) ray_q[(ray_h + ray_n + __popc(pushed & ((1u << lane) - 1u))) & 63] = uint8_t(k);
            ray_n += __popc(pushed);
            __syncwarp();
        }

        // Lanes whose walk is done hand over their context and take the next.
        {
            const unsigned done = __ballot_sync(ALL, state == WALK_DONE);
            const unsigned full = __ballot_sync(ALL, state == WALK_DONE && c >= 0);
            if (done == ALL && !full && ray_n == 0 && shade_n == 0) break;
            if ((full | (ray_n ? done : 0u)) && (__popc(full | (ray_n ? done : 0u)) >= kFetch || done == ALL)) {
                bool go = false, hand = false;
                if (state == WALK_DONE && c >= 0) {
                    if (shadow) {
                        if (w.h.kind == PT_HIT_NONE) setv(C_RAD, c, getv(C_RAD, c) + getv(C_SV, c));
                        const uint32_t flags = ctx[C_FLAGS][c] & ~CF_SHADOW;
                        ctx[C_FLAGS][c] = flags;
                        hand = (flags & CF_ENDED) != 0;
                        go = !hand;
                    } else {
                        setf(C_SD, c, w.t_max);
                        setf(C_SD + 1, c, w.h.u);
                        setf(C_SD + 2, c, w.h.v);
                        ctx[C_ST][c] = w.h.kind;
                        ctx[C_SV][c] = w.h.index;
                        if (INST) ctx[C_SV + 1][c] = w.h.inst;
                        hand = true;
                    }
                }
                const unsigned handed = __ballot_sync(ALL, hand);
                if (hand) {
                    shade_q[(shade_h + shade_n + __popc(handed & ((1u << lane) - 1u))) & 63] = uint8_t(c);
                    c = -1;
                }
                shade_n += __popc(handed);
                const unsigned take = __ballot_sync(ALL, state == WALK_DONE && c < 0);
                if (state == WALK_DONE && c < 0) {
                    const int i = __popc(take & ((1u << lane) - 1u));
                    if (i < ray_n) {
                        c = ray_q[(ray_h + i) & 63];
                        go = true;
                    }
                }
                const int got = min(ray_n, __popc(take));
                ray_h += got;
                ray_n -= got;
                __syncwarp();
                if (go) {
                    shadow = (ctx[C_FLAGS][c] & CF_SHADOW) != 0;
                    if (!shadow) ++rays;
                    state = w.begin(S, getv(C_O, c), getv(shadow ? C_SD : C_D, c), 0.001f,
                                    shadow ? getf(C_ST, c) : 1000.0f, shadow, stack);
                }
            }
        }

        if (shade_n >= kShade && ray_n == 0) continue;
        while (true) {
            const unsigned nodes = __ballot_sync(ALL, state == AT_NODE);
            if (!nodes) break;
            if (__popc(nodes) < kNodes) {
                const unsigned done = __ballot_sync(ALL, state == WALK_DONE && (c >= 0 || ray_n > 0));
                const unsigned leaves = __ballot_sync(ALL, state == AT_LEAF);
                if (leaves || __popc(done) >= kFetch) break;
                if (shade_n > 0 && ray_n == 0 && shade_n >= __popc(nodes)) break;
            } else if (ray_n > 0 && __popc(__ballot_sync(ALL, state == WALK_DONE)) >= kFetch) {
                break;
            }
            if (state == AT_NODE) state = w.expand(S, 0.001f, stack, overflow);
        }
        if (state == AT_LEAF) state = w.leaf(S, 0.001f, shadow, stack, overflow);
    }

    unsigned long long total = rays;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) total += __shfl_down_sync(ALL, total, off);
    if (lane == 0 && P.rays) atomicAdd(P.rays, total);
    if (__any_sync(ALL, overflow) && lane == 0) atomicOr(S.status, PT_DEV_ERR_STACK);
}

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
cudaError_t launch_s(const PtSceneDev& S, const PtRenderParams& p, PtSampleLaunch L, int sms, cudaStream_t stream) {
    static int blocks_per_sm = 0;
    int per_sm = blocks_per_sm;
    if (!per_sm)
        blocks_per_sm = per_sm = pt_resident_blocks(
            reinterpret_cast<const void*>(megakernel_stream<AUX, SNAP, INST, TEX, EXT>), 128, 0);
    const uint32_t warps = uint32_t(sms * per_sm) * 4u;
    L.contexts = int((L.items + warps - 1) / warps);
    megakernel_stream<AUX, SNAP, INST, TEX, EXT><<<sms * per_sm, 128, 0, stream>>>(S, p, L);
    sum_samples<AUX><<<(L.pixels + 255) / 256, 256, 0, stream>>>(p, L);
    return cudaGetLastError();
}

template <bool INST, bool TEX>
cudaError_t launch_stream(const PtSceneDev& S, const PtRenderParams& p, const PtSampleLaunch& L, int sms,
                          cudaStream_t stream) {
    const bool aux = p.aux != nullptr, snap = p.rng_mode == 1;
    if (p.nee_ext)  // production streams only (the host refuses it with snapshots)
        return aux ? launch_s<true, false, INST, TEX, true>(S, p, L, sms, stream)
                   : launch_s<false, false, INST, TEX, true>(S, p, L, sms, stream);
    if (aux)
        return snap ? launch_s<true, true, INST, TEX, false>(S, p, L, sms, stream)
                    : launch_s<true, false, INST, TEX, false>(S, p, L, sms, stream);
    return snap ? launch_s<false, true, INST, TEX, false>(S, p, L, sms, stream)
                : launch_s<false, false, INST, TEX, false>(S, p, L, sms, stream);
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
                              cudaStream_t stream) {
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
        return flat ? launch_stream<false, true>(S, p, L, sms, stream) : launch_stream<true, true>(S, p, L, sms, stream);
    return flat ? launch_stream<false, false>(S, p, L, sms, stream) : launch_stream<true, false>(S, p, L, sms, stream);
}
