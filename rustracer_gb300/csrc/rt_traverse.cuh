// BVH traversal of the wavefront's persistent warps (gather.wgsl:66-88, common.wgsl:78-100).
//
// Every lane of a warp walks its own ray through the tree, one record (four or two child boxes) per
// step.  A record fetch tests the children's boxes with the reference's slab test (gather.wgsl:71-75:
// (bmin - ro) / d, te <= ta && ta > 0 && te < t); hit internal children are visited nearest entry
// first, the others pushed.  Hit leaves are not tested by the lane that met them: they go into the
// warp's leaf list, which the warp tests together before it goes on, four lanes per leaf, one triangle
// per lane.  The tree is the reference's, so the closest hit is the reference's.
//
// Triangles hit at exactly equal t resolve to the lowest prim slot: leaves hold consecutive slot ranges
// with the left child's below the right's (bvh.rs:159-219), so the reference's left-first walk, where
// the first strictly smaller t wins, meets the lowest slot first.  The best hit of a lane's ray is one
// 64-bit word, t's bits above the prim slot (t is positive, so the words order as (t, slot) pairs), and a
// test that hits lowers it with an atomic minimum, whatever order a step's tests come in.
//
// A leaf is tested only if its box is entered before the nearest hit so far, and a hit's computed distance
// can lie before its own leaf's box: by rounding, or by far more on a sliver.  So which leaves have been
// tested when a box is looked at can decide between two overlapping surfaces.  Every ray's leaves are
// therefore tested before its next record, and the result is its own: it does not depend on which rays share
// the warp or on the launch.  (Waiting until eight leaves are listed keeps more lanes busy, 1080p frame of the
// 1.31M-triangle room 18.28 against 18.42 ms, but leaves a walk unaware of a hit for a record or two.)
#pragma once
#include "rt_kernels.h"

namespace rtd {

// Stack entries per lane: the oldest kTopStack in shared memory, the ones above them (a few rays get
// there) in local memory.  11 let 7 blocks of 128 threads share an SM with 28 KB of L1 left; 8 measure
// 2% slower, 14 0.5%, 16 (6 blocks) 9%.
constexpr uint32_t kTopStack = 11, kMaxStack = 64;
// Leaves a step can meet: up to 4 per lane.
constexpr uint32_t kLeafCap = 4 * 32;

// A warp's shared state.
struct __align__(16) WarpTrav {
    // The lanes' rays, read by the lanes that test their leaves; .w: halves of the scene's tri_ord.
    float4 ro[32], rd[32];
    // The next rays of the warp's queue segment, copied in ahead of need: origin, direction (.w: job
    // index), reciprocal direction (.w: ray id).
    float4 next_ro[32], next_rd[32], next_inv[32];
    uint32_t next_queue[32];  // path slots of the rays after those
    uint32_t n_ext, n;        // the work list: closest-hit rays, then occlusion rays up to n
    uint32_t item, seg_end;   // the warp's segment of the work list: first item not read ahead, end
    uint32_t items, first;    // entries in next_queue, the first one's item
    uint32_t at, ready;       // rays [at, ready) of the copied ones are unclaimed
    uint32_t coming;          // rays being copied
    unsigned long long best[32];  // t bits << 32 | prim slot
    float limit[32];              // occlusion rays that look for the closest hit: hits below it count
    uint2 leaf[kLeafCap];         // the step's leaves: first prim slot, count << 5 | owner lane
};

__device__ __forceinline__ unsigned long long hit_word(float t, uint32_t prim) {
    return ((unsigned long long)__float_as_uint(t) << 32) | prim;
}
__device__ __forceinline__ float hit_t(unsigned long long w) { return __uint_as_float((uint32_t)(w >> 32)); }

// 16 bytes from global to shared memory without a register in between; cp_async_wait waits for all the
// thread's copies.
__device__ __forceinline__ void cp_async16(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async4(void *dst, const void *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// The scene's tri_ord carried by a ray of WarpTrav.
__device__ __forceinline__ const float4 *ray_triangles(float4 ro, float4 rd) {
    return reinterpret_cast<const float4 *>(((unsigned long long)__float_as_uint(rd.w) << 32) |
                                            (unsigned long long)__float_as_uint(ro.w));
}

// Moller-Trumbore (common.wgsl:78-100) with the edges precomputed, without a branch; 0 for a miss (hits
// count above kEps).
__device__ __forceinline__ float hit_distance(f3 ro, f3 rd, float4 v0, float4 e1, float4 e2) {
    const f3 h3 = cross(rd, xyz(e2));
    const float a = dot(xyz(e1), h3);
    const float f = 1.0f / a;
    const f3 sv = ro - xyz(v0);
    const float u = f * dot(sv, h3);
    const f3 q = cross(sv, xyz(e1));
    const float v = f * dot(rd, q);
    const float t = f * dot(xyz(e2), q);
    return fabsf(a) < 1e-7f || u < 0.0f || u > 1.0f || v < 0.0f || u + v > 1.0f ? 0.0f : t;
}

// Tests the triangles of listed leaves [first, first + n), n <= 8: lane l takes triangles l % 4,
// l % 4 + 4, ... of leaf l / 4, against the ray of the lane that met it.
// tris: the scene's leaf-ordered triangles (kMulti: each ray's own, from its record).
template <bool kMulti>
__device__ __forceinline__ void test_leaves(WarpTrav &w, uint32_t first, uint32_t n, const float4 *tris) {
    const uint32_t lane = threadIdx.x & 31u, e = lane >> 2;
    if (e >= n) return;
    const uint2 leaf = w.leaf[first + e];
    const uint32_t ref = leaf.x, o = leaf.y & 31u, cnt = leaf.y >> 5;
    const float4 r0 = w.ro[o], r1 = w.rd[o];
    if (kMulti) tris = ray_triangles(r0, r1);
    const f3 ro = xyz(r0), rd = xyz(r1);
    for (uint32_t k = lane & 3u; k < cnt; k += 4u) {
        const float4 *tp = tris + 3ull * (ref + k);
        const float4 v0 = __ldg(tp), e1 = __ldg(tp + 1), e2 = __ldg(tp + 2);
        const float t = hit_distance(ro, rd, v0, e1, e2);
        if (t > kEps) atomicMin(&w.best[o], hit_word(t, ref + k));
    }
}

// Two floats of a packed pair, and the pairs' IEEE sum and product (each half rounded as the scalar
// operation rounds it).
using f32x2 = unsigned long long;
__device__ __forceinline__ f32x2 pack2(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(f32x2 v, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// One ray's walk, kept by its lane.
struct TravLane {
    f32x2 minus_ro[3], inv[3];  // -origin and 1 / direction, each component in both halves
    float t;                // closest hit folded in so far (occlusion rays: the limit until then)
    float te;               // entry distance of the record visited next
    uint32_t node;          // record visited next
    uint32_t sp;            // stack entries in use
    const float4 *records;  // the traversal layout of the ray's scene
    uint32_t cap;           // stack entries the scene may use
};

// The lane's stack of pending records with their entry distances: top[i * kBlock] for i < kTopStack
// (lane-interleaved shared memory), then deep[] (local memory).
template <int kBlock>
__device__ __forceinline__ void trav_push(TravLane &st, uint2 *top, uint2 *deep, uint32_t ref, float te) {
    const uint2 e = make_uint2(ref, __float_as_uint(te));
    if (st.sp < kTopStack) top[st.sp * kBlock] = e;
    else if (st.sp < st.cap) deep[st.sp - kTopStack] = e;
    else return;
    st.sp += 1u;
}
// Moves to the nearest pending record the ray still reaches, unless the current one is; false when none
// is left.  A record entered at or beyond t holds no box entered below it.
template <int kBlock>
__device__ __forceinline__ bool trav_settle(TravLane &st, const uint2 *top, const uint2 *deep) {
    while (!(st.te < st.t)) {
        if (st.sp == 0u) return false;
        st.sp -= 1u;
        uint2 e;
        if (st.sp < kTopStack) e = top[st.sp * kBlock];
        else e = deep[st.sp - kTopStack];
        st.node = e.x;
        st.te = __uint_as_float(e.y);
    }
    return true;
}

// The treelet of a block: the first `count` four-wide records of the scene whose records start at `src`,
// staged in shared memory.
struct Treelet {
    const float4 *smem, *src;
    uint32_t count;
};

// One step of every lane of a warp: `visiting` lanes test the child boxes of their record, list the hit
// leaves in w (`leaves` of them) and move on to the next record (visiting ends when none is left).
// records: the scene's (kMulti: each ray's own, st.records).  tests: the lane's listed triangles are
// added.  Every lane calls it.
//
// A child is 32 bytes, one load: four-wide (min.x, max.x, min.y, max.y), (min.z, max.z, ref, count), so
// that both planes of an axis go through one packed subtraction and one packed product; two-wide
// (min, ref), (max, count).
template <bool kWide, int kTree, int kBlock, bool kMulti>
__device__ __forceinline__ void trav_step(TravLane &st, uint2 *top, uint2 *deep, bool &visiting, WarpTrav &w,
                                          uint32_t &leaves, const Treelet &tree, const float4 *records,
                                          uint32_t &tests) {
    constexpr int K = kWide ? 4 : 2;
    if (kMulti) records = st.records;
    const float kNone = __int_as_float(0x7F800000);
    float key[K];
    uint32_t ref[K], cnt[K];
#pragma unroll
    for (int c = 0; c < K; ++c) cnt[c] = 0u;
    if (visiting) {
        float4 q[2 * K];
        if (kTree > 0 && records == tree.src && st.node < tree.count) {
#pragma unroll
            for (int i = 0; i < 2 * K; ++i) q[i] = tree.smem[2u * K * st.node + i];
        } else {
            // In the children's order on every lane: it decides between children entered at the same distance.  (An
            // order that differs from lane to lane spreads the loads over more of L1's banks: 1080p frame of the
            // 1.31M-triangle room 17.84 against 18.28 ms.  But then the one of two overlapping surfaces that a ray
            // hits depends on its lane.)
            const float4 *np = records + (size_t)(2 * K) * st.node;
#pragma unroll
            for (int i = 0; i < K; ++i) ldg32(np + 2 * i, q[2 * i], q[2 * i + 1]);
        }
#pragma unroll
        for (int c = 0; c < K; ++c) {
            const float4 u = q[2 * c], v = q[2 * c + 1];
            const f32x2 x = kWide ? pack2(u.x, u.y) : pack2(u.x, v.x);
            const f32x2 y = kWide ? pack2(u.z, u.w) : pack2(u.y, v.y);
            const f32x2 z = kWide ? pack2(v.x, v.y) : pack2(u.z, v.z);
            ref[c] = __float_as_uint(kWide ? v.z : u.w);
            const uint32_t n = __float_as_uint(v.w);
            float x0, x1, y0, y1, z0, z1;
            unpack2(mul2(add2(x, st.minus_ro[0]), st.inv[0]), x0, x1);
            unpack2(mul2(add2(y, st.minus_ro[1]), st.inv[1]), y0, y1);
            unpack2(mul2(add2(z, st.minus_ro[2]), st.inv[2]), z0, z1);
            const float te = fmax3f(fminf(x0, x1), fminf(y0, y1), fminf(z0, z1));
            const float tx = fmin3f(fmaxf(x0, x1), fmaxf(y0, y1), fmaxf(z0, z1));
            // (an empty place holds a NaN box, which no ray hits)
            const bool hit = te <= tx && tx > 0.0f && te < st.t;
            cnt[c] = hit ? n : 0u;
            key[c] = hit && n == 0u ? te : kNone;  // +inf: not a pending child
        }
    }
    uint32_t anyl = cnt[0];
#pragma unroll
    for (int c = 1; c < K; ++c) anyl |= cnt[c];
    if (__any_sync(0xFFFFFFFFu, anyl != 0u))
#pragma unroll
    for (int c = 0; c < K; ++c) {
        const uint32_t m = __ballot_sync(0xFFFFFFFFu, cnt[c] != 0u);
        if (cnt[c] != 0u) {
            w.leaf[leaves + __popc(m & lanemask_lt())] =
                make_uint2(ref[c], cnt[c] << 5 | (threadIdx.x & 31u));
            tests += cnt[c];
        }
        leaves += __popc(m);
    }
    if (visiting) {
        auto cswap = [&](int i, int j) {
            if (key[j] < key[i]) {
                const float tk = key[i];
                key[i] = key[j];
                key[j] = tk;
                const uint32_t tr = ref[i];
                ref[i] = ref[j];
                ref[j] = tr;
            }
        };
        // Near-first order of the hit internal children (four: a fixed five-exchange network; pushing the
        // farther ones unsorted visits more records, trace 9% slower).
        cswap(0, 1);
        if (kWide) {
            cswap(2, 3);
            cswap(0, 2);
            cswap(1, 3);
            cswap(1, 2);
        }
        st.node = ref[0];
        st.te = key[0];
        if (key[1] < kNone) {
            if (st.sp + (K - 1) <= kTopStack) {
                uint2 *e = top + st.sp * kBlock;
#pragma unroll
                for (int i = K - 1; i >= 1; --i) {
                    const bool on = key[i] < kNone;
                    if (on) *e = make_uint2(ref[i], __float_as_uint(key[i]));
                    e += on ? kBlock : 0;
                    st.sp += on ? 1u : 0u;
                }
            } else {
#pragma unroll
                for (int i = K - 1; i >= 1; --i)
                    if (key[i] < kNone) trav_push<kBlock>(st, top, deep, ref[i], key[i]);
            }
        }
        visiting = trav_settle<kBlock>(st, top, deep);
    }
}

// A lane and its ray: idle, or walking until it visits no more records.
struct LaneWalk {
    TravLane st;
    bool busy, visiting;
    bool any_hit;  // an occlusion ray that may stop at its first hit below st.t
    bool found;    // a hit below the starting st.t
};

// Gives the lane a ray to walk from the root (r.st.t, records and cap and r.any_hit are set): origin o,
// direction d, the scene's triangles.
__device__ __forceinline__ void walk_begin(LaneWalk &r, WarpTrav &w, f3 o, f3 d, f3 inv, const float4 *tris) {
    const uint32_t lane = threadIdx.x & 31u;
    const unsigned long long tp = (unsigned long long)tris;
    w.ro[lane] = make_float4(o.x, o.y, o.z, __uint_as_float((uint32_t)tp));
    w.rd[lane] = make_float4(d.x, d.y, d.z, __uint_as_float((uint32_t)(tp >> 32)));
    w.best[lane] = hit_word(r.st.t, 0u);
    r.st.minus_ro[0] = pack2(-o.x, -o.x);
    r.st.minus_ro[1] = pack2(-o.y, -o.y);
    r.st.minus_ro[2] = pack2(-o.z, -o.z);
    r.st.inv[0] = pack2(inv.x, inv.x);
    r.st.inv[1] = pack2(inv.y, inv.y);
    r.st.inv[2] = pack2(inv.z, inv.z);
    r.st.node = 0u;
    r.st.te = -kInf;
    r.st.sp = 0u;
    r.found = false;
    r.busy = true;
}

// Up to max_steps records for every lane of a warp (fewer once `few` or less lanes still walk), with the
// tests of their leaves.  visits and tests (kCount) count the lane's records and triangles.
template <bool kWide, int kTree, int kBlock, bool kMulti, bool kCount>
__device__ __forceinline__ void walk_records(LaneWalk &r, WarpTrav &w, uint2 *top, uint2 *deep, const Treelet &tree,
                                             const float4 *records, const float4 *tris, uint32_t max_steps, int few,
                                             uint32_t &visits, uint32_t &tests) {
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t k = 0;;) {
        uint32_t leaves = 0u, n = 0u;
        if (kCount && r.visiting) visits += 1u;
        trav_step<kWide, kTree, kBlock, kMulti>(r.st, top, deep, r.visiting, w, leaves, tree, records, n);
        if (kCount) tests += n;
        if (leaves != 0u) {
            __syncwarp();
            for (uint32_t g = 0u; g < leaves; g += 8u) test_leaves<kMulti>(w, g, min(8u, leaves - g), tris);
            __syncwarp();
            if (r.busy) {
                const float t = hit_t(w.best[lane]);
                if (t < r.st.t) {
                    r.found = true;
                    if (r.any_hit) r.visiting = false;
                }
                r.st.t = t;
                if (r.visiting) r.visiting = trav_settle<kBlock>(r.st, top, deep);
            }
        }
        if (++k >= max_steps || __popc(__ballot_sync(0xFFFFFFFFu, r.visiting)) <= few) break;
    }
}

// Dynamic shared memory of a traversal block: the lane-interleaved stack tops, one WarpTrav per warp, then
// the treelet (four-wide launches with a treelet).
inline size_t trav_smem_bytes(uint32_t block_threads, bool tree) {
    return (size_t)kTopStack * block_threads * sizeof(uint2) + (block_threads / 32u) * sizeof(WarpTrav) +
           (tree ? (size_t)kTreeletRecords * 8u * sizeof(float4) : 0u);
}

}  // namespace rtd
