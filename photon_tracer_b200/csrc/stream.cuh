// Streaming tree walks: each lane walks one ray, and the lanes of a warp meet
// at the phases of the walk instead of waiting for the warp's longest ray.
//
// What bounds a lock-step walk (`traverse`, `walk` in tracer.cuh) here is
// divergence: the rays of a warp need 3 nodes at the median, 13 at the 90th
// percentile (random rays in the room scene), and a warp works on until its
// longest ray is done, so an instruction serves 5-7 of 32 lanes. Here a lane
// is in one state at a time -- at a node, at a leaf, at an instance to enter,
// done -- and the caller's loop runs a phase when enough lanes stand at it;
// lanes that are done get their next ray while the others walk on.
//
// Every ray visits the nodes and primitives that the lock-step walks visit, in
// the same order, with the same float operations: hits are the same bit for
// bit.
#pragma once
#include "tracer.cuh"

namespace ptd {

// Stack words (the seventh plane of PtSceneDev::qnodes): an interior child is
// its node index (bit 31 clear). A leaf sets bit 31, bit 30 when it holds a
// sphere, bit 29 when its entries are instances, its count in bits 25-28 and
// its first slot in bits 0-24; the word with bits 29, 30 and 31 set returns
// to the world ray.
enum : uint32_t {
    PT_Q_LEAF = 0x80000000u,
    PT_Q_SPHERE = 0x40000000u,
    PT_Q_INST = 0x20000000u,
    PT_Q_WORLD = 0xe0000000u,
    PT_Q_COUNT = 0x1e000000u,
    PT_Q_FIRST = 0x01ffffffu
};
__device__ __forceinline__ uint32_t q_count(uint32_t w) { return (w & PT_Q_COUNT) >> 25; }

// A lane's state between the phases.
enum WalkState : int { WALK_DONE = 0, AT_NODE = 1, AT_LEAF = 2 };

// The traversal stack in 8-byte entries: the first SH of each lane in shared
// memory ([depth][thread]), deeper ones in a local array. The ray-query
// kernel keeps 8 in shared memory (none: 2% slower); the megakernel, whose
// paths fill shared memory, none.
constexpr int kWalkStack = 8;

template <int SH, int NT>
struct WordStack {
    uint32_t base;  // shared-window address of this thread's entry 0
    uint2* deep;    // entries SH and up
    __device__ __forceinline__ void put(int i, uint32_t w, float t) {
        if (SH > 0 && i < SH)
            asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(base + uint32_t(i) * (8u * NT)), "r"(w),
                         "r"(__float_as_uint(t)));
        else
            deep[i - SH] = make_uint2(w, __float_as_uint(t));
    }
    __device__ __forceinline__ void get(int i, uint32_t& w, float& t) const {
        uint32_t b;
        if (SH > 0 && i < SH) {
            asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(w), "=r"(b) : "r"(base + uint32_t(i) * (8u * NT)));
        } else {
            const uint2 q = deep[i - SH];
            w = q.x;
            b = q.y;
        }
        t = __uint_as_float(b);
    }
};
#define PT_WORD_STACK(name, NT, SH)                                                                     \
    __shared__ uint2 name##_s[(SH) > 0 ? (SH) * (NT) : 1];                                                \
    uint2 name##_deep[PT_STACK_MAX - (SH)];                                                               \
    ::ptd::WordStack<(SH), (NT)> name{                                                                    \
        static_cast<uint32_t>(__cvta_generic_to_shared(&name##_s[0])) + threadIdx.x * 8u, name##_deep}

// Where a walk leaves its nearest hit and finds its world-space ray. In
// registers, for ray queries:
struct HitRegs {
    Hit h;
    V o, d;  // the ray in world space
    __device__ __forceinline__ void world(V& wo, V& wd) const {
        wo = o;
        wd = d;
    }
    __device__ __forceinline__ void clear(uint32_t kind, uint32_t index) { h = {kind, index, 0, 0, 0}; }
    __device__ __forceinline__ void set(uint32_t kind, uint32_t index, uint32_t inst) {
        h.kind = kind;
        h.index = index;
        h.inst = inst;
    }
    __device__ __forceinline__ void set_uv(float u, float v) {
        h.u = u;
        h.v = v;
    }
    __device__ __forceinline__ void drop() { h.kind = PT_HIT_NONE; }
};

// One ray's walk. INST: the scene has instances.
template <bool INST>
struct Walk {
    V o, d;
    float ix, iy, iz;
    bool fast;
    int nx, ny, nz;  // float4 index of each axis' near plane (lo: 0-2, hi: 3-5)
    float t_max;
    int top;
    uint32_t cur;
    uint32_t cur_inst;
    bool in_mesh;

    __device__ __forceinline__ void set(const PtSceneDev& S, V o_, V d_, float t_min) {
        o = o_;
        d = d_;
        ix = 1.0f / d.x;
        iy = 1.0f / d.y;
        iz = 1.0f / d.z;
        fast = S.ordered_boxes && finite_nonzero(ix) && finite_nonzero(iy) && finite_nonzero(iz) && finite_f(o.x) &&
               finite_f(o.y) && finite_f(o.z) && t_min == t_min;
        nx = fast && ix < 0 ? 3 : 0;
        ny = fast && iy < 0 ? 4 : 1;
        nz = fast && iz < 0 ? 5 : 2;
    }

    // The next entry that is not behind t_max becomes cur.
    template <class Stack, class Out>
    __device__ __forceinline__ int pop(const PtSceneDev& S, float t_min, Stack& stack, const Out& out) {
        while (top > 0) {
            float t;
            stack.get(--top, cur, t);
            if (t >= t_max) continue;
            if (INST && cur == PT_Q_WORLD) {
                V wo, wd;
                out.world(wo, wd);
                set(S, wo, wd, t_min);
                in_mesh = false;
                continue;
            }
            return (cur & PT_Q_LEAF) ? AT_LEAF : AT_NODE;
        }
        return WALK_DONE;
    }

    // Large spheres, then the root of the tree; WALK_DONE when nothing is left to walk.
    template <class Stack, class Out>
    __device__ __forceinline__ int begin(const PtSceneDev& S, V o_, V d_, float t_min, float t_max_, bool any,
                                         Stack& stack, Out& hit) {
        t_max = t_max_;
        top = 0;
        uint32_t kind = PT_HIT_NONE, index = 0;
#pragma unroll 1
        for (uint32_t i = 0; i < S.n_large; ++i)
            if (sphere_hit_double(__ldg(S.large + i), o_, d_, t_min, t_max)) {
                kind = PT_HIT_LARGE;
                index = i;
                if (any) break;
            }
        hit.clear(kind, index);
        if (any && kind != PT_HIT_NONE) return WALK_DONE;
        set(S, o_, d_, t_min);
        if (INST) {
            in_mesh = false;
            cur_inst = 0;
            if (S.inst_root != PT_NONE) stack.put(top++, S.inst_root, t_min);
        }
        if (S.flat_root != PT_NONE) stack.put(top++, S.flat_root, t_min);
        return pop(S, t_min, stack, hit);
    }

    // Slab-tests node cur's four children against [t_min, t_max] and pushes
    // the ones hit, farthest first (bvh.hpp:72-103), then pops. The walk
    // ends, with the overflow flag set, if the stack would overflow.
    template <class Stack, class Out>
    __device__ __forceinline__ int expand(const PtSceneDev& S, float t_min, Stack& stack, Out& out, bool& overflow) {
        const float4* nd = S.qnodes + 8 * size_t(cur);
        const float4 lox = __ldg(nd + nx), loy = __ldg(nd + ny), loz = __ldg(nd + nz);
        const float4 hix = __ldg(nd + (3 - nx)), hiy = __ldg(nd + (5 - ny)), hiz = __ldg(nd + (7 - nz));
        const uint4 words = __ldg(reinterpret_cast<const uint4*>(nd + 6));
        float X0[4], X1[4], Y0[4], Y1[4], Z0[4], Z1[4];
        {
            const float2 ox = make_float2(o.x, o.x), oy = make_float2(o.y, o.y), oz = make_float2(o.z, o.z);
            const float2 vx = make_float2(ix, ix), vy = make_float2(iy, iy), vz = make_float2(iz, iz);
#define PT_PAIR(ARR, V4, O2, I2)                                       \
    {                                                                  \
        const float2 a = sub_mul2(make_float2(V4.x, V4.y), O2, I2);    \
        const float2 b = sub_mul2(make_float2(V4.z, V4.w), O2, I2);    \
        ARR[0] = a.x; ARR[1] = a.y; ARR[2] = b.x; ARR[3] = b.y;        \
    }
            PT_PAIR(X0, lox, ox, vx)
            PT_PAIR(X1, hix, ox, vx)
            PT_PAIR(Y0, loy, oy, vy)
            PT_PAIR(Y1, hiy, oy, vy)
            PT_PAIR(Z0, loz, oz, vz)
            PT_PAIR(Z1, hiz, oz, vz)
#undef PT_PAIR
        }
        float tn[4];
        int mask = 0;
        if (fast && t_max == t_max) {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float n_ = fmaxf(fmaxf(X0[c], Y0[c]), fmaxf(Z0[c], t_min));
                const float f_ = fminf(fminf(X1[c], Y1[c]), fminf(Z1[c], t_max));
                tn[c] = n_;
                mask |= (n_ <= f_) ? (1 << c) : 0;
            }
        } else {
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float n_ = sse_max(sse_max(sse_min(X0[c], X1[c]), sse_min(Y0[c], Y1[c])),
                                         sse_max(sse_min(Z0[c], Z1[c]), t_min));
                const float f_ = sse_min(sse_min(sse_max(X0[c], X1[c]), sse_max(Y0[c], Y1[c])),
                                         sse_min(sse_max(Z0[c], Z1[c]), t_max));
                tn[c] = n_;
                mask |= (n_ <= f_) ? (1 << c) : 0;
            }
        }
        if (mask) {
            const int n = __popc(mask);
            if (top + n > PT_STACK_MAX) {
                overflow = true;
                out.drop();
                return WALK_DONE;
            }
            const uint32_t ws[4] = {words.x, words.y, words.z, words.w};
            int rank[4];
            child_ranks(tn, mask, rank);
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (mask & (1 << c)) stack.put(top + rank[c], ws[c], tn[c]);
            top += n;
        }
        return pop(S, t_min, stack, out);
    }

    // The leaf cur: its primitives in order, or its first instance entered.
    template <class Stack, class Out>
    __device__ __forceinline__ int leaf(const PtSceneDev& S, float t_min, bool any, Stack& stack, Out& out,
                                        bool& overflow) {
        const uint32_t first = cur & PT_Q_FIRST, n = q_count(cur);
        if (INST && (cur & PT_Q_INST)) {
            // hit_instance (include/geometry.hpp:212-229): the rest of the
            // leaf and the return to the world ray wait on the stack, unpruned.
            if (top + 3 > PT_STACK_MAX) {
                overflow = true;
                out.drop();
                return WALK_DONE;
            }
            const float4* is = S.islots + 4 * size_t(first);
            const float4 rows[3] = {__ldg(is), __ldg(is + 1), __ldg(is + 2)};
            const uint4 meta = __ldg(reinterpret_cast<const uint4*>(is + 3));
            const float never = -__int_as_float(0x7f800000);
            if (n > 1) stack.put(top++, PT_Q_LEAF | PT_Q_INST | ((n - 1) << 25) | (first + 1), never);
            stack.put(top++, PT_Q_WORLD, never);
            V wo, wd;
            out.world(wo, wd);
            set(S, aff_point(rows, wo), aff_vector(rows, wd), t_min);
            cur_inst = meta.y;
            in_mesh = true;
            if (t_min >= t_max) return pop(S, t_min, stack, out);
            cur = meta.x;
            return AT_NODE;
        }
        const bool spheres = (cur & PT_Q_SPHERE) != 0;
#pragma unroll 1
        for (uint32_t q = first; q < first + n; ++q) {
            const float4* sl = S.slots + 3 * size_t(q);
            const float4 a = __ldg(sl), b = __ldg(sl + 1), c = __ldg(sl + 2);
            const uint32_t in = INST && in_mesh ? cur_inst : 0u;
            bool hit;
            if (spheres && (fbits(c.y) & PT_SLOT_SPHERE)) {
                hit = sphere_hit(a, o, d, t_min, t_max);
                if (hit) out.set(PT_HIT_SPHERE, q, in);
            } else {
                float u, v;
                hit = tri_hit(a, b, c, o, d, t_min, t_max, u, v);
                if (hit) {
                    out.set(INST && in_mesh ? PT_HIT_INSTANCE : PT_HIT_TRIANGLE, q, in);
                    out.set_uv(u, v);
                }
            }
            if (hit && any) return WALK_DONE;
        }
        return pop(S, t_min, stack, out);
    }
};

}  // namespace ptd
