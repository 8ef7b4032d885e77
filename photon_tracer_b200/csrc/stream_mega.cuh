// The streaming megakernel, over one frame (megakernel.cu) or a batch's
// (batch.cu).
//
// A lock-step megakernel is bound by divergence: a room-frame query takes
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
// issue) and instruction fetch (65 KB of code, 2.2 of 10: 3.7 KB more cost the
// room frame 14%, so duplicates in the code count).
//
// A work item is one sample, not one pixel, so that a small frame fills the
// GPU and a large one ends without a tail of whole pixels; each sample's
// radiance goes to a buffer that a second kernel adds up in sample order, which
// rounds as one pixel's samples rendered in turn. Images are the lock-step
// form's bit for bit. Measured on one B200, lock-step -> streaming: 1024x1024
// room, 64 samples 145.0 -> 94.4 ms; 960x540, 16 samples of 10,000 instances
// 64.3 -> 35.9 ms; 400x225, 16 samples of random spheres 1.86 -> 1.22 ms; one
// such row of 400 pixels 0.71 -> 0.16 ms.
//
// Five resident blocks per SM (96 registers; 4: room 13% slower), four for
// the forms with more live state, auxiliary outputs (1080p room, 4 samples:
// 10.0 ms, 5 blocks 11.1) and extended light sampling (8.5 ms, 5 blocks 8.9; 7.1 with one copy of its draws).
// Fetch and node thresholds are flat optima (4..12, 8..12: within 2%).
#pragma once
#include "path.cuh"
#include "stream.cuh"

namespace ptd {

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
    C_SCENE = 31,  // scene number, with many scenes
    C_MIS = 32     // EXT
};
enum : uint32_t { CF_BOUNCE = 0xffffu, CF_SAMPLED = 1u << 16, CF_SHADOW = 1u << 17, CF_ENDED = 1u << 18, CF_LIVE = 1u << 19 };

// A sample's place: pixel (i, j), sample number, scene, and index in the
// buffer of samples.
struct SampleAt {
    int i, j;
    uint32_t sample, scene, place;
};

// The context a lane walks for, and its hit: in registers until the walk is
// done, or (IN_CONTEXT) a path ray's straight in its context's words. In
// registers the plain forms are faster (room frame 1%, instances 2.6%), in the
// context the forms with more live state (a batch 4.5%, guides 1.3%).
template <int C, bool INST, bool IN_CONTEXT>
struct WalkHit;

template <int C, bool INST>
struct WalkHit<C, INST, false> : HitRegs {
    uint32_t (*ctx)[C];
    int c;
    bool shadow;
    __device__ __forceinline__ void start(V o_, V d_) {
        o = o_;
        d = d_;
    }
    __device__ __forceinline__ bool is_blocked() const { return h.kind != PT_HIT_NONE; }
    __device__ __forceinline__ void keep() const {
        ctx[C_SD + 1][c] = __float_as_uint(h.u);
        ctx[C_SD + 2][c] = __float_as_uint(h.v);
        ctx[C_ST][c] = h.kind;
        ctx[C_SV][c] = h.index;
        if (INST) ctx[C_SV + 1][c] = h.inst;
    }
};

template <int C, bool INST>
struct WalkHit<C, INST, true> {
    uint32_t (*ctx)[C];
    int c;
    bool shadow, blocked;
    __device__ __forceinline__ V get(int f) const {
        return mk(__uint_as_float(ctx[f][c]), __uint_as_float(ctx[f + 1][c]), __uint_as_float(ctx[f + 2][c]));
    }
    __device__ __forceinline__ void start(V, V) {}
    __device__ __forceinline__ bool is_blocked() const { return blocked; }
    __device__ __forceinline__ void keep() const {}
    __device__ __forceinline__ void world(V& wo, V& wd) const {
        wo = get(C_O);
        wd = get(shadow ? C_SD : C_D);
    }
    __device__ __forceinline__ void clear(uint32_t kind, uint32_t index) {
        blocked = kind != PT_HIT_NONE;
        if (!shadow) {
            set(kind, index, 0);
            set_uv(0, 0);
        }
    }
    __device__ __forceinline__ void set(uint32_t kind, uint32_t index, uint32_t inst) {
        blocked = true;
        if (shadow) return;
        ctx[C_ST][c] = kind;
        ctx[C_SV][c] = index;
        if (INST) ctx[C_SV + 1][c] = inst;
    }
    __device__ __forceinline__ void set_uv(float u, float v) {
        if (shadow) return;
        ctx[C_SD + 1][c] = __float_as_uint(u);
        ctx[C_SD + 2][c] = __float_as_uint(v);
    }
    __device__ __forceinline__ void drop() {
        blocked = false;
        if (!shadow) ctx[C_ST][c] = PT_HIT_NONE;
    }
};

// Frame: what is rendered -- its items, scenes, cameras and buffers.
template <bool AUX, bool INST, bool TEX, bool EXT, class Frame>
__global__ void __launch_bounds__(128, AUX || EXT ? kStreamBlocks - 1 : kStreamBlocks)
    megakernel_stream(const __grid_constant__ Frame F) {
    constexpr int C = kContexts, FIELDS = EXT ? 33 : Frame::kManyScenes ? 32 : 31;
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

    const int contexts = min(F.contexts(), C);
    F.started();
    auto scene_of = [&](int c) -> uint32_t { return Frame::kManyScenes ? ctx[C_SCENE][c] : 0u; };
    for (int c = lane; c < contexts; c += 32) {
        ctx[C_FLAGS][c] = CF_ENDED;
        shade_q[c] = uint8_t(c);
    }
    __syncwarp();
    // queue heads and lengths, the same in every lane
    int ray_h = 0, ray_n = 0, shade_h = 0, shade_n = contexts;
    uint32_t rays = 0;
    bool overflow = false;
    int state = WALK_DONE;
    WalkHit<C, INST, AUX || EXT || Frame::kManyScenes> hit;
    hit.ctx = ctx;
    hit.shadow = false;
    int& c = hit.c;  // the context this lane walks for
    c = -1;
    uint32_t walk_scene = 0;
    Walk<INST> w;
    w.top = 0;

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
                const bool found = h.kind != PT_HIT_NONE;
                Rec rec;
                const uint32_t sc = scene_of(k);
                const PtSceneDev& S = F.scene(sc);
                if (found) fill<TEX, EXT>(S, h, path.o, path.d, getf(C_SD, k), rec);
                First first;
                const bool primary = AUX && path.bounce == 0;
                bool nee;
                Shadow sh;
                unsigned long long shadow_rays = 0;
                const bool done = shade<AUX, TEX, EXT>(S, path, found, rec, F.depth(sc), smp, rng, first, nee, sh,
                                                       shadow_rays) == STEP_DONE;
                rays += uint32_t(shadow_rays);
                if (primary) {  // the first hit's guides
                    float* g = F.guides() + 6 * size_t(ctx[C_ITEM][k]);
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
                float* out = F.samples() + 3 * size_t(ctx[C_ITEM][k]);
                out[0] = rad.x;
                out[1] = rad.y;
                out[2] = rad.z;
            }
            // Contexts whose sample ended take the next ones; those past the
            // last are dropped.
            bool need = ended, fresh = false;
            SampleAt at = {0, 0, 0, 0, 0};
            while (true) {
                const unsigned want = __ballot_sync(ALL, need);
                if (!want) break;
                const int leader = __ffs(want) - 1;
                uint32_t base = 0;
                if (lane == leader) base = atomicAdd(F.work(), uint32_t(__popc(want)));
                base = __shfl_sync(ALL, base, leader);
                if (need) {
                    const uint32_t item = base + __popc(want & ((1u << lane) - 1u));
                    if (item >= F.items()) {
                        need = false;
                    } else if (F.locate(item, at)) {
                        need = false;
                        fresh = true;
                    }
                }
            }
            if (fresh) {
                // render_row_impl's sample loop body (:379-385)
                smp.begin(F.seed(at), at.i, at.j, at.sample);
                float du, dv;
                smp.sample_2d(0, rng, du, dv);
                V o, d;
                F.ray(at, du, dv, o, d);
                setv(C_O, k, o);
                setv(C_D, k, d);
                setv(C_TP, k, mk(1, 1, 1));
                setv(C_RAD, k, mk(0, 0, 0));
                if (EXT) setf(C_MIS, k, 0);
                F.start(at, rng);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint64_t x = i == 0 ? rng.s0 : i == 1 ? rng.s1 : i == 2 ? rng.s2 : rng.s3;
                    ctx[C_RNG + 2 * i][k] = uint32_t(x);
                    ctx[C_RNG + 2 * i + 1][k] = uint32_t(x >> 32);
                }
                ctx[C_SEED][k] = smp.pixel_seed;
                ctx[C_INDEX][k] = at.sample;
                ctx[C_ITEM][k] = at.place;
                if (Frame::kManyScenes) ctx[C_SCENE][k] = at.scene;
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
                    if (hit.shadow) {
                        if (!hit.is_blocked()) setv(C_RAD, c, getv(C_RAD, c) + getv(C_SV, c));
                        const uint32_t flags = ctx[C_FLAGS][c] & ~CF_SHADOW;
                        ctx[C_FLAGS][c] = flags;
                        hand = (flags & CF_ENDED) != 0;
                        go = !hand;
                    } else {
                        setf(C_SD, c, w.t_max);
                        hit.keep();
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
                    const bool shadow = (ctx[C_FLAGS][c] & CF_SHADOW) != 0;
                    const V d = getv(shadow ? C_SD : C_D, c);
                    const float t = shadow ? getf(C_ST, c) : 1000.0f;
                    hit.shadow = shadow;
                    if (!shadow) ++rays;
                    walk_scene = scene_of(c);
                    const V o = getv(C_O, c);
                    hit.start(o, d);
                    state = w.begin(F.scene(walk_scene), o, d, 0.001f, t, shadow, stack, hit);
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
            if (state == AT_NODE) state = w.expand(F.scene(walk_scene), 0.001f, stack, hit, overflow);
        }
        if (state == AT_LEAF) state = w.leaf(F.scene(walk_scene), 0.001f, hit.shadow, stack, hit, overflow);
    }

    unsigned long long total = rays;
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) total += __shfl_down_sync(ALL, total, off);
    if (lane == 0 && F.rays()) atomicAdd(F.rays(), total);
    if (__any_sync(ALL, overflow) && lane == 0) atomicOr(F.status(), PT_DEV_ERR_STACK);
}

}  // namespace ptd
