// The gather pass as a wavefront: rustracer-renderer/shaders/gather.wgsl:258-594 split into kernels that
// each run one uniform piece of code over a compacted queue of paths.
//
//   generate   camera ray of sample 0 for every pixel (gather.wgsl:262-297); fills queue 0
//   extend     closest hit of every queued path (gather.wgsl:300)
//   shade      one loop body of gather.wgsl:299-537 per queued path: hit shading, emission, debug
//              views, dielectric / metallic-roughness lobes, the light sample of NEE
//              (gather.wgsl:152-206, its shadow ray deferred to `shadow`), photon lookup, next
//              direction, Russian roulette; a finished sample starts the pixel's next sample in the
//              same slot; continuing paths are appended to the next queue (warp ballot + one atomic)
//   shadow     occlusion of each deferred NEE ray; a visible light adds its contribution
//   finalize   sigma clamp and the frame / moments / gbuffer writes (gather.wgsl:548-593)
//
// extend and shadow run as one persistent traversal launch (`wf_trace_kernel`): the occlusion rays of
// iteration i-1 ride with the closest-hit rays of iteration i, which need only shade(i-1) too.  The
// photon pass uses the same kernel for its closest-hit rays.
//
// One path slot per pixel: a pixel's samples run one after the other in its slot, with one RNG
// stream, exactly as the reference's per-pixel loop.  Every pixel receives its contributions in the
// reference's order except that a bounce's NEE term lands after that bounce's other terms; floating
// point addition order is the only difference (an ulp).  The host launches spp * max_bounces
// iterations; a path extends at most once per iteration, so that bounds every pixel's segments.
#include <cstring>

#include "rt_paths.cuh"

namespace rtd {

__global__ void __launch_bounds__(256) triangle_terms_kernel(float4 *__restrict__ tris, uint64_t n) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= n) return;
    float4 *p = tris + 8ull * i;
    const f3 v0 = xyz(p[0]), v1 = xyz(p[1]), v2 = xyz(p[2]), e1 = v1 - v0, e2 = v2 - v0, gn = triangle_normal(v0, v1, v2);
    const float d00 = dot(e1, e1), d01 = dot(e1, e2), d11 = dot(e2, e2);
    p[0].w = gn.x;
    p[1].w = gn.y;
    p[2].w = gn.z;
    p[3].w = d00;
    p[4].w = d01;
    p[5].w = d11;
    p[7].w = d00 * d11 - d01 * d01;
}

cudaError_t launch_triangle_terms(float4 *tris, uint64_t n, cudaStream_t st) {
    triangle_terms_kernel<<<(unsigned)((n + 255u) / 256u), 256, 0, st>>>(tris, n);
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------------------------
// generate: 8 x 4 pixel tiles, one per warp, so the first queue is tile-coherent.  One launch over
// every job's tiles (job j's start at its tile0).
// ------------------------------------------------------------------------------------------------
template <bool kMulti>
__global__ void __launch_bounds__(128) wf_generate_kernel(const __grid_constant__ WaveJob p, uint32_t n_tiles) {
    grid_launch_dependents();
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint32_t gtile = blockIdx.x * 4u + warp;
    if (gtile >= n_tiles) return;  // whole warps: warp_append below is warp-uniform
    const uint32_t jid = job_of<kMulti>(p, gtile, [](const DevJob &j) { return j.tile0; });
    const DevJob &job = job_at<kMulti>(p, jid);
    const uint32_t W = job.ip.width, H = job.ip.height;
    const uint32_t tiles_x = (W + 7u) / 8u;
    const uint32_t tile = gtile - job.tile0;
    const uint32_t tx = tile % tiles_x, ty = tile / tiles_x;
    const uint32_t px = tx * 8u + (lane & 7u), py = ty * 4u + (lane >> 3);
    const bool active = px < W && py < H;
    const uint32_t slot = job.base + py * W + px;
    if (active) start_slot(p, job, jid, px, py, slot);
    warp_append(active, slot, p.queue[0], p.counts + 0);
}

// ------------------------------------------------------------------------------------------------
// shade: one bounce of gather.wgsl's loop body per queued path.  kPhotons / kDebug compile the photon
// lookup and the debug views in; the host picks the variant that covers every job of the launch
// (a job without photons or debug view takes the same path through either variant), so frames
// without them run a smaller kernel.
//
// Each round a block takes 128 queue entries and orders them by what the hit needs -- a miss, a
// dielectric, a Lambertian or emissive surface, a metal -- before shading, so a warp runs mostly one
// of the loop body's branches (neighbouring paths hit triangles of unrelated materials).  Only the
// order in which paths are shaded changes: each path's operations are its own, so images are the
// same bit for bit.  Surviving paths, their shadow rays and photon-lookup requests are queued in the
// paths' original order (which keeps neighbouring pixels together for the traversal).
// ------------------------------------------------------------------------------------------------
constexpr uint32_t kShadeKeys = 5;  // miss, dielectric, Lambertian / emissive, metal, no entry

// The entry's order key; for a hit also its triangle and material word, read from the hit prim
// slot's record (the traversal stores the slot: `orig` = the triangle's index, `word` = key | material
// << 2, filled at scene upload).
template <bool kMulti>
__device__ __forceinline__ uint32_t shade_key(const WaveJob &p, const uint32_t *q, uint32_t i, uint32_t n,
                                              uint32_t &slot, uint32_t &orig, uint32_t &word, float &t) {
    t = kInf;
    slot = 0u;
    orig = 0u;
    word = 0u;
    if (i >= n) return 4u;
    slot = q[i];
    const float2 h = p.hit[slot];
    t = h.x;
    if (h.x >= kInf) return 0u;
    const float4 *tris = kMulti ? p.jobs[__float_as_uint(p.thr[slot].w)].scene.tri_ord : p.job0.scene.tri_ord;
    const float4 *rec = tris + 3ull * __float_as_uint(h.y);
    orig = __float_as_uint(__ldg(rec).w);
    word = __float_as_uint(__ldg(rec + 1).w);
    return word & 3u;
}

// kBlocks: resident blocks per SM the register allocation aims at (4: ~123 registers; 5: 96
// registers with 62 bytes of spills; 6: 80 registers, 100 to 200 bytes of spills, the default: the extra
// warps hide the kernel's dependent loads), chosen per launch by the tuning's shade_blocks.  Bound by divergence
// (16 of 32 lanes), those loads and a long body (10% of a warp's cycles wait for instructions).  1080p room frame
// with the job in the launch: 19.17 ms with 5 blocks, 18.14 with 6, 18.68 with 7; with the state prefetched to L1
// while the entries are ordered, blocks of 64, 256 or 384, or the texture fetch out of line: the same to 2% slower.
template <bool kPhotons, bool kDebug, bool kMulti, int kBlocks>
__global__ void __launch_bounds__(128, kBlocks) wf_shade_kernel(const __grid_constant__ WaveJob p, uint32_t iter,
                                                               uint32_t most) {
    __shared__ uint32_t s_count[4][kShadeKeys];  // entries per warp and key
    __shared__ uint32_t s_order[128];
    __shared__ uint8_t s_emit[128];   // by original position: 1 survives, 2 shadow ray, 4 photon lookup
    __shared__ uint32_t s_spos[128];  // by original position: shadow record index
    __shared__ uint32_t s_ppos[128];  // by original position: photon-lookup record index
    __shared__ uint32_t s_orig[128], s_word[128];
    __shared__ float2 s_own[128];  // by shading position: the hit's triangle and material word
    grid_dependency_wait();
    grid_launch_dependents();
    const uint32_t n = p.counts[4 * iter];
    if (n <= most) return;  // the launch before this one ran these paths to their end
    const uint32_t *q = p.queue[iter & 1u];
    uint32_t *q_next = p.queue[(iter + 1u) & 1u];
    uint32_t *n_next = p.counts + 4 * (iter + 1u);
    uint32_t *n_shadow = p.counts + 4 * iter + 1u;
    uint32_t *n_photon = p.counts + 4 * iter + 3u;
    const uint32_t stride = gridDim.x * blockDim.x;
    const uint32_t rounds = (n + stride - 1u) / stride;
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;

    for (uint32_t r = 0; r < rounds; ++r) {
        // The block's entries ranked by key, stable (warp-major, then lane order within a key).
        const uint32_t round_base = r * stride + blockIdx.x * blockDim.x;
        const uint32_t i_own = round_base + threadIdx.x;
        uint32_t slot_own, orig_own, word_own;
        float t_own;
        const uint32_t key = shade_key<kMulti>(p, q, i_own, n, slot_own, orig_own, word_own, t_own);
        uint32_t same = 0;
#pragma unroll
        for (uint32_t k = 0; k < kShadeKeys; ++k) {
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, key == k);
            if (lane == k) s_count[warp][k] = __popc(m);
            if (key == k) same = __popc(m & lanemask_lt());
        }
        __syncthreads();
        uint32_t pos = same;
#pragma unroll
        for (uint32_t k = 0; k < kShadeKeys; ++k)
#pragma unroll
            for (uint32_t w = 0; w < 4; ++w)
                if (k < key || (k == key && w < warp)) pos += s_count[w][k];
        s_order[pos] = i_own;
        s_own[pos] = make_float2(__uint_as_float(slot_own), t_own);
        s_orig[pos] = orig_own;
        s_word[pos] = word_own;
        __syncthreads();
        const uint32_t i = s_order[threadIdx.x];
        const bool valid = i < n;
        ShadeOut out;
        uint32_t slot = 0;
        if (valid) {
            const float2 own = s_own[threadIdx.x];
            slot = __float_as_uint(own.x);
            out = shade_path<kPhotons, kDebug, kMulti>(p, slot, own.y, s_orig[threadIdx.x], s_word[threadIdx.x] >> 2, false);
        }
        // Queue positions by original order: each thread appends for the entry it keyed, then the
        // thread that shaded it writes its records there.
        const uint32_t li = i - round_base;
        s_emit[li] = (out.keep ? 1u : 0u) | (out.shadow ? 2u : 0u) | ((kPhotons && out.photon) ? 4u : 0u);
        __syncthreads();
        {
            const uint32_t e = s_emit[threadIdx.x];
            warp_append((e & 1u) != 0u, slot_own, q_next, n_next);
            const uint32_t ms = __ballot_sync(0xFFFFFFFFu, (e & 2u) != 0u);
            if (ms) {
                const uint32_t leader = __ffs(ms) - 1u;
                uint32_t base = 0;
                if (lane == leader) base = atomicAdd(n_shadow, (uint32_t)__popc(ms));
                base = __shfl_sync(0xFFFFFFFFu, base, leader);
                if (e & 2u) s_spos[threadIdx.x] = base + __popc(ms & lanemask_lt());
            }
            if (kPhotons) {
                const uint32_t mp = __ballot_sync(0xFFFFFFFFu, (e & 4u) != 0u);
                if (mp) {
                    const uint32_t leader = __ffs(mp) - 1u;
                    uint32_t base = 0;
                    if (lane == leader) base = atomicAdd(n_photon, (uint32_t)__popc(mp));
                    base = __shfl_sync(0xFFFFFFFFu, base, leader);
                    if (e & 4u) s_ppos[threadIdx.x] = base + __popc(mp & lanemask_lt());
                }
            }
        }
        __syncthreads();
        // NEE shadow ray (deferred) and the photon-map lookup request.
        if (out.shadow) {
            float4 *rec = p.shadow + 2ull * s_spos[li];
            rec[0] = make_float4(out.sh_o.x, out.sh_o.y, out.sh_o.z, out.sh_max);
            rec[1] = make_float4(out.sh_d.x, out.sh_d.y, out.sh_d.z, __uint_as_float(slot));
        }
        if (kPhotons && out.photon) {
            float4 *rec = p.preq + 3ull * s_ppos[li];
            const uint32_t jid = kMulti ? __float_as_uint(p.thr[slot].w) : 0u;
            rec[0] = make_float4(out.ph_hp.x, out.ph_hp.y, out.ph_hp.z, __uint_as_float(slot));
            rec[1] = make_float4(out.ph_n.x, out.ph_n.y, out.ph_n.z, __uint_as_float(out.ph_sidx));
            rec[2] = make_float4(out.ph_td.x, out.ph_td.y, out.ph_td.z, __uint_as_float(jid));
        }
    }
}

// ------------------------------------------------------------------------------------------------
// photon: the photon-map lookup of the diffuse bounces shade recorded (gather.wgsl:473-514), one
// request per thread.  A separate pass keeps the shade kernel's registers (and its occupancy) off the
// divergent cell loops.  Runs after shade(iter) and before the occlusion rays of iter, so a pixel's
// terms arrive in the order the inline lookup added them.
// ------------------------------------------------------------------------------------------------
template <bool kMulti>
__global__ void __launch_bounds__(128) wf_photon_kernel(const __grid_constant__ WaveJob p, uint32_t iter) {
    grid_dependency_wait();
    grid_launch_dependents();
    const uint32_t n = p.counts[4 * iter + 3];
    constexpr uint32_t kRunsA = 10;
    __shared__ uint2 s_runs[4][kRunsA * 32];
    uint2 rest[kLookupCells - kRunsA];
    __shared__ uint32_t s_hits[4][kHitList * 32];
    const LookupRuns<kRunsA> runs{s_runs[threadIdx.x >> 5] + (threadIdx.x & 31u), rest};
    uint32_t *hit_list = s_hits[threadIdx.x >> 5] + (threadIdx.x & 31u);
    const uint32_t lane = threadIdx.x & 31u;
    for (uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x - lane; i0 < n; i0 += gridDim.x * blockDim.x) {
        const uint32_t i = i0 + lane, lanes = __ballot_sync(0xFFFFFFFFu, i < n);
        if (i < n) {
            const float4 r0 = p.preq[3ull * i], r1 = p.preq[3ull * i + 1], r2 = p.preq[3ull * i + 2];
            photon_lookup(p, job_at<kMulti>(p, __float_as_uint(r2.w)), __float_as_uint(r0.w), __float_as_uint(r1.w), xyz(r0),
                          xyz(r1), xyz(r2), lanes, runs, hit_list);
        }
    }
}

// ------------------------------------------------------------------------------------------------
// trace: the deferred NEE occlusion rays of iteration `shd_iter` (gather.wgsl:91-103; a visible light marks its
// slot's NEE term) and the closest-hit rays of iteration `ext_iter` in one persistent launch (either may be
// kNoIter).  Both depend only on the shade pass before them and touch disjoint state (shadow records and NEE
// words / path rays and hits), so one launch carries
// them with one tail instead of two.  Closest-hit rays come first in the work list: the longer rays
// start early and the shorter occlusion rays fill the end.
constexpr uint32_t kNoIter = 0xFFFFFFFFu;
constexpr uint32_t kOcclusion = 0x80000000u;  // ray id: path slot, and whether it is the slot's occlusion ray

// Each lane of a warp walks its own ray, `steps` records at a time; then finished lanes write their
// result and take new rays.  The warp is bound by instruction issue and by the latency of its record
// fetches together, so the step is kept short and the registers few: 7 blocks of 128 threads per SM
// (72 registers; 64 registers for 8 blocks spill in the step and measure 4% slower, 80 for 6 blocks 4%),
// the ray feed in shared memory, no branch in the triangle test.  Config-2 frame (28.5 M closest-hit and
// 24.8 M occlusion rays): 12.8 ms against 16.1 ms for the kernel this one replaced, which laid a step's
// triangles out over the warp with a scan and read rays when a lane ran out; 11% fewer records visited
// (pending records entered beyond the hit are dropped unread).
//
// kCount: the profiling variant, which also counts the records each kind of ray visits and its leaf
// triangle tests into p.work (one atomic per warp at exit); the same rays and results otherwise.
// kTree (four-wide only): the block first stages the top kTree records of job 0's tree in shared
// memory (after the stacks and the WarpTravs), and lanes on that scene read them from there.
// kMulti: the launch's jobs may be on different scenes (each ray carries its own); otherwise the scene
// comes with the launch, which saves four registers and the job table's loads for every ray.
// kCut: scenes of the launch may have cut-out materials.  Without them every occlusion ray may stop at its
// first hit, and the call of the alpha rule with its spills goes.
template <int kBlock, bool kWide, bool kCount, int kTree, bool kMulti, bool kCut>
__global__ void __launch_bounds__(kBlock, 896 / kBlock) wf_trace_kernel(const __grid_constant__ WaveParams p, uint32_t ext_iter,
                                                          uint32_t shd_iter, uint32_t chunk, uint32_t steps) {
    extern __shared__ __align__(16) unsigned char trav_smem[];
    const uint32_t lane = threadIdx.x & 31u;
    uint2 *top = reinterpret_cast<uint2 *>(trav_smem) + threadIdx.x;
    uint2 deep[kMaxStack - kTopStack];
    WarpTrav *warps = reinterpret_cast<WarpTrav *>(trav_smem + sizeof(uint2) * kTopStack * kBlock);
    WarpTrav &w = warps[threadIdx.x >> 5];
    grid_dependency_wait();
    grid_launch_dependents();
    Treelet tree{nullptr, nullptr, 0u};
    if (kTree > 0) {
        float4 *t = reinterpret_cast<float4 *>(warps + kBlock / 32);
        const DevScene &s0 = p.jobs[0].scene;
        tree.smem = t;
        tree.src = s0.wnodes;
        tree.count = s0.wnode_count < (uint32_t)kTree ? s0.wnode_count : (uint32_t)kTree;
        for (uint32_t i = threadIdx.x; i < 8u * tree.count; i += kBlock) t[i] = __ldg(tree.src + i);
        __syncthreads();
    }
    {
        const uint32_t n_ext = ext_iter != kNoIter ? p.counts[4 * ext_iter] : 0u;
        const uint32_t n_shd = shd_iter != kNoIter ? p.counts[4 * shd_iter + 1] : 0u;
        if (lane == 0u) {
            w.n_ext = n_ext;
            w.n = n_ext + n_shd;
        }
    }
    const uint32_t *q = p.queue[ext_iter & 1u];
    // Row ext_iter's cursor; the closing launch (no closest-hit rays) takes row shd_iter + 1's, which
    // no other launch uses.  Entry [3] of a row counts shade's photon-lookup requests.
    uint32_t *fetch = p.counts + 4 * (ext_iter != kNoIter ? ext_iter : shd_iter + 1u) + 2;

    // The work list is dealt out in segments of `chunk` items: the first by warp number, the later ones
    // by one atomic each, issued a segment ahead.  The entries of the next 32 rays are copied to shared
    // memory ahead of need, and so are the rays themselves, while the warp walks.
    uint32_t after = (blockIdx.x * (kBlock / 32) + (threadIdx.x >> 5)) * chunk;  // lane 0: the next segment
    auto read_ahead = [&]() {
        const uint32_t n = w.n, n_ext = w.n_ext;
        uint32_t item = w.item, end = w.seg_end, items = 0u;
        if (item >= end) {
            item = __shfl_sync(0xFFFFFFFFu, after, 0);
            end = min(item + chunk, n);
            if (item < n && lane == 0u) after = gridDim.x * (kBlock / 32) * chunk + atomicAdd(fetch, chunk);
        }
        if (item < end) {
            items = min(32u, end - item);
            if (lane < items) {
                if (item + lane < n_ext) cp_async4(&w.next_queue[lane], q + item + lane);
                else cp_async4(&w.next_queue[lane], &p.shadow[2ull * (item + lane - n_ext) + 1].w);  // its slot
            }
        }
        __syncwarp();
        if (lane == 0u) {
            w.item = item + items;
            w.seg_end = end;
            w.items = items;
            w.first = item;
        }
    };
    // Starts the copy of the next rays (all the copied ones are claimed) and reads on.
    auto request = [&]() {
        const uint32_t items = w.items;
        if (lane < items) {
            const uint32_t slot = w.next_queue[lane], item = w.first + lane, n_ext = w.n_ext;
            const bool occ = item >= n_ext;
            const float4 *rec = p.shadow + 2ull * (item - n_ext);
            cp_async16(&w.next_ro[lane], occ ? rec : p.ro + slot);
            cp_async16(&w.next_rd[lane], occ ? rec + 1 : p.rd + slot);
            w.next_inv[lane].w = __uint_as_float(occ ? slot | kOcclusion : slot);
            if (kMulti) cp_async4(&w.next_inv[lane].x, &p.thr[slot].w);
        }
        __syncwarp();
        if (lane == 0u) w.coming = items;
        if (items != 0u) read_ahead();
        __syncwarp();
    };
    if (lane == 0u) w.item = w.seg_end = w.at = w.ready = 0u;
    __syncwarp();
    read_ahead();
    cp_async_wait();
    __syncwarp();
    request();

    LaneWalk r;
    r.busy = r.visiting = r.any_hit = false;
    r.st.sp = 0u;
    uint32_t id = 0u;
    uint32_t work[4] = {0u, 0u, 0u, 0u};  // kCount: records closest / occlusion, tests closest / occlusion
    // Records between refills (low 16 bits), fewer once `few` or less lanes still walk.
    const uint32_t max_steps = steps & 0xFFFFu;
    const int few = (int)(steps >> 16);
    for (;;) {
        // Idle lanes take the next rays.
        const uint32_t idle = __ballot_sync(0xFFFFFFFFu, !r.busy);
        if (idle != 0u) {
            uint32_t at = w.at, ready = w.ready;
            const uint32_t coming = w.coming;
            if (at == ready && coming != 0u) {
                cp_async_wait();
                if (lane < coming) {
                    const f3 inv = mk3(1.0f, 1.0f, 1.0f) / xyz(w.next_rd[lane]);
                    const float4 x = w.next_inv[lane];
                    w.next_inv[lane] = make_float4(inv.x, inv.y, inv.z, x.w);
                    if (kMulti) w.next_rd[lane].w = x.x;
                }
                at = 0u;
                ready = coming;
                __syncwarp();
                if (lane == 0u) {
                    w.ready = coming;
                    w.coming = 0u;
                }
            }
            const uint32_t avail = ready - at;
            if (avail == 0u) {
                if (idle == 0xFFFFFFFFu) break;
            } else {
                const uint32_t rank = __popc(idle & lanemask_lt());
                if (!r.busy && rank < avail) {
                    const float4 o = w.next_ro[at + rank], d = w.next_rd[at + rank], v = w.next_inv[at + rank];
                    id = __float_as_uint(v.w);
                    const bool occ = (id & kOcclusion) != 0u;
                    const float4 *tris = p.tris0;
                    uint32_t any = p.any_hit0, empty = p.empty0;
                    r.st.records = p.records0;
                    r.st.cap = kMaxStack;
                    if (kMulti) {
                        const DevScene &sc = p.jobs[__float_as_uint(d.w)].scene;
                        r.st.records = kWide ? sc.wnodes : sc.cnodes;
                        r.st.cap = kWide ? kMaxStack : sc.stack_cap;
                        tris = sc.tri_ord;
                        any = sc.any_hit_shadows;
                        empty = sc.cnode_count == 0u;
                    }
                    // An occlusion ray asks for hits below the limit: any one without cut-out materials, the
                    // closest with them (the reference's closest-hit-then-alpha rule).  The closest is looked for
                    // without a limit: a sliver's computed distance can lie far before its box, whose entry may be
                    // beyond the limit then (a search up to 1.001 of it is no faster: cut-out foliage 1.41 ms
                    // against 1.40).
                    r.any_hit = occ && (!kCut || any != 0u);
                    r.st.t = occ ? o.w - 0.001f : kInf;
                    if (kCut && occ && !r.any_hit) {
                        w.limit[lane] = r.st.t;
                        r.st.t = kInf;
                    }
                    walk_begin(r, w, xyz(o), xyz(d), xyz(v), tris);
                    // No triangle counts below kEps, so a limit at or below it (or a NaN) is never met: the
                    // ray ends as it starts, and so does any ray of an empty scene.
                    r.visiting = empty == 0u && r.st.t > kEps;
                }
                at += min((uint32_t)__popc(idle), avail);
                __syncwarp();
                if (lane == 0u) w.at = at;
                __syncwarp();  // (every lane reads it and w.ready next time round)
                if (at == ready) request();
            }
        }
        uint32_t visits = 0u, tests = 0u;
        walk_records<kWide, kTree, kBlock, kMulti, kCount>(r, w, top, deep, tree, p.records0, p.tris0, max_steps, few,
                                                           visits, tests);
        if (kCount) {
            work[(id & kOcclusion) ? 1 : 0] += visits;
            work[(id & kOcclusion) ? 3 : 2] += tests;
        }
        if (r.busy && !r.visiting) {
            const uint32_t slot = id & ~kOcclusion;
            const bool occ = (id & kOcclusion) != 0u;
            bool lit = !r.found && r.st.t == r.st.t;  // (a NaN limit counts as occluded)
            if (!r.any_hit) {
                const unsigned long long hit = w.best[lane];
                if (kCut && occ)
                    lit = cut_out_lit(p.jobs[__float_as_uint(p.thr[slot].w)].scene, w.ro[lane], w.rd[lane], w.limit[lane],
                                      hit);
                else  // the hit's prim slot
                    p.hit[slot] = make_float2(hit_t(hit), __uint_as_float((uint32_t)hit));
            }
            if (occ && lit) atomicOr(reinterpret_cast<uint32_t *>(&p.nee[slot].w), kNeeLit);
            r.busy = false;
        }
    }
    if (kCount && p.work) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            uint32_t v = work[i];
#pragma unroll
            for (uint32_t d = 16u; d > 0u; d >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, d);
            if (lane == 0u) atomicAdd(p.work + i, (unsigned long long)v);
        }
    }
}

// ------------------------------------------------------------------------------------------------
// finalize: one launch over every job's slots.
// ------------------------------------------------------------------------------------------------
template <bool kMulti>
__global__ void __launch_bounds__(256) wf_finalize_kernel(const __grid_constant__ WaveJob p, uint32_t n_slots) {
    grid_dependency_wait();
    grid_launch_dependents();
    const uint32_t slot = blockIdx.x * blockDim.x + threadIdx.x;
    if (slot >= n_slots) return;
    finalize_slot(p, job_at<kMulti>(p, job_of<kMulti>(p, slot, [](const DevJob &j) { return j.base; })), slot);
}

// Segments (paths queued per iteration) and shadow rays of the pass, added to the 64-bit counters.
__global__ void wf_count_kernel(const __grid_constant__ WaveParams p, uint32_t iters) {
    grid_dependency_wait();
    if (!p.counters) return;
    unsigned long long seg = 0, shd = 0;
    for (uint32_t i = threadIdx.x; i < iters; i += 32u) {
        seg += p.counts[4 * i];
        shd += p.counts[4 * i + 1];
    }
#pragma unroll
    for (uint32_t d = 16u; d > 0u; d >>= 1) {
        seg += __shfl_xor_sync(0xFFFFFFFFu, seg, d);
        shd += __shfl_xor_sync(0xFFFFFFFFu, shd, d);
    }
    if (threadIdx.x == 0u) {
        p.counters[0] += seg;
        p.counters[1] += shd;
    }
}

// ------------------------------------------------------------------------------------------------
// Host launcher: the gather pass of one frame of every job.
// ------------------------------------------------------------------------------------------------
WaveTuning default_tuning() { return WaveTuning{128u, 7u, 32u, 3u, 32u, 0u, 6u, 0u}; }

bool normalize_tuning(WaveTuning &t, uint32_t stack_need) {
    const WaveTuning in = t;
    if (t.block_threads != 64u && t.block_threads != 128u && t.block_threads != 256u) t.block_threads = 128u;
    const uint32_t max_blocks = 2048u / t.block_threads;  // resident threads per SM
    t.blocks_per_sm = t.blocks_per_sm < 1u ? 1u : (t.blocks_per_sm > max_blocks ? max_blocks : t.blocks_per_sm);
    t.chunk = t.chunk < 32u ? 32u : (t.chunk > 1024u ? 1024u : (t.chunk + 31u) / 32u * 32u);
    t.steps = t.steps < 1u ? 1u : (t.steps > 64u ? 64u : t.steps);
    t.refill_idle = t.refill_idle > 31u ? 31u : t.refill_idle;
    const uint32_t need = stack_need > t.stack_entries ? stack_need : t.stack_entries;
    t.stack_entries = need <= 32u ? 32u : (need <= 48u ? 48u : 64u);
    t.treelet = t.treelet ? kTreeletRecords : 0u;
    t.shade_blocks = t.shade_blocks >= 4u && t.shade_blocks <= 6u ? t.shade_blocks : 6u;
    return std::memcmp(&in, &t, sizeof(t)) == 0;
}

namespace {

using TraceKernel = void (*)(const WaveParams, uint32_t, uint32_t, uint32_t, uint32_t);

// wf_trace_kernel's `steps`.
uint32_t trace_steps(const WaveTuning &t) { return t.steps | (t.refill_idle ? 32u - t.refill_idle : 0u) << 16; }

// multi: the jobs may be on different scenes; cut: some may have cut-out materials.  The two-wide, counting
// and treelet variants are compiled for both only, which covers the rest.
template <int kBlock>
TraceKernel trace_kernel_of(bool wide, bool count, bool tree, bool multi, bool cut) {
    constexpr int kT = (int)kTreeletRecords;
    if (!wide)
        return count ? wf_trace_kernel<kBlock, false, true, 0, true, true>
                     : wf_trace_kernel<kBlock, false, false, 0, true, true>;
    if (tree)
        return count ? wf_trace_kernel<kBlock, true, true, kT, true, true>
                     : wf_trace_kernel<kBlock, true, false, kT, true, true>;
    if (count) return wf_trace_kernel<kBlock, true, true, 0, true, true>;
    if (multi)
        return cut ? wf_trace_kernel<kBlock, true, false, 0, true, true> : wf_trace_kernel<kBlock, true, false, 0, true, false>;
    return cut ? wf_trace_kernel<kBlock, true, false, 0, false, true> : wf_trace_kernel<kBlock, true, false, 0, false, false>;
}

TraceKernel trace_kernel(const WaveTuning &t, bool wide, bool count, bool multi, bool cut) {
    const bool tree = wide && t.treelet != 0u;
    if (t.block_threads == 64u) return trace_kernel_of<64>(wide, count, tree, multi, cut);
    if (t.block_threads == 256u) return trace_kernel_of<256>(wide, count, tree, multi, cut);
    return trace_kernel_of<128>(wide, count, tree, multi, cut);
}

}  // namespace

void prepare_wavefront_kernels() {
    // Blocks above 48 KB of dynamic shared memory need the opt-in; set it for every variant.
    for (uint32_t block : {64u, 128u, 256u})
        for (int v = 0; v < 32; ++v) {
            const bool wide = (v & 1) != 0, count = (v & 2) != 0, multi = (v & 4) != 0, tree = wide && (v & 8) != 0;
            const bool cut = (v & 16) != 0;
            WaveTuning t = default_tuning();
            t.block_threads = block;
            t.treelet = tree ? kTreeletRecords : 0u;
            cudaFuncSetAttribute(reinterpret_cast<const void *>(trace_kernel(t, wide, count, multi, cut)),
                                 cudaFuncAttributeMaxDynamicSharedMemorySize, (int)trav_smem_bytes(block, tree));
        }
    prepare_paths_kernels();
}

namespace {
void set_scene0(WaveParams &p, const DevScene &scene, bool wide) {
    p.records0 = wide ? scene.wnodes : scene.cnodes;
    p.tris0 = scene.tri_ord;
    p.any_hit0 = scene.any_hit_shadows;
    p.empty0 = scene.cnode_count == 0u ? 1u : 0u;
}
}  // namespace

bool one_job_reads_table(const JobShape &shape, const WaveTuning &tune, bool profiled) {
    WaveTuning t = tune;
    normalize_tuning(t, 0u);
    return profiled || shape.wide == 0u || shape.debug != 0u || shape.scene->any_hit_shadows == 0u || t.treelet != 0u ||
           t.shade_blocks != 6u;
}
bool photon_pass_reads_table(const DevScene &scene, const WaveTuning &tune) {
    return scene.wnodes == nullptr || tune.treelet != 0u;
}

cudaError_t launch_extend(const WaveParams &params, uint32_t iter, uint64_t max_items, const DevScene &scene, int num_sms,
                          const WaveTuning &tune, cudaStream_t st) {
    const bool wide = scene.wnodes != nullptr;
    WaveParams p = params;
    set_scene0(p, scene, wide);
    WaveTuning t = tune;
    normalize_tuning(t, wide ? scene.wide_stack : scene.stack_cap);
    const uint64_t blocks_needed = (max_items + t.block_threads - 1u) / t.block_threads;
    const uint64_t persistent = (uint64_t)num_sms * t.blocks_per_sm;
    const uint32_t grid = (uint32_t)(blocks_needed < persistent ? (blocks_needed ? blocks_needed : 1u) : persistent);
    return launch_dependent(trace_kernel(t, wide, false, false, false), grid, t.block_threads,
                            trav_smem_bytes(t.block_threads, wide && t.treelet), st, p, iter, kNoIter, t.chunk,
                            trace_steps(t));
}

cudaError_t launch_wavefront(const WaveParams &params, const JobShape *jobs, uint32_t n_jobs, uint32_t iters, int num_sms,
                             const WaveTuning &tune, cudaStream_t st, WaveProfile *prof) {
    cudaError_t e;
    WaveJob p;
    std::memset(&p, 0, sizeof(p));
    static_cast<WaveParams &>(p) = params;
    uint64_t slots = 0;
    uint32_t stack_need = 0, wide_need = 0;
    bool wide = n_jobs > 0;  // four-wide records when every job's scene has them
    bool cut = false, few_records = true;
    uint64_t tiles = 0;
    for (uint32_t j = 0; j < n_jobs; ++j) {
        tiles += ((jobs[j].width + 7u) / 8u) * ((jobs[j].height + 3u) / 4u);
        slots += jobs[j].npix;
        stack_need = jobs[j].stack_cap > stack_need ? jobs[j].stack_cap : stack_need;
        wide_need = jobs[j].wide_stack > wide_need ? jobs[j].wide_stack : wide_need;
        wide = wide && jobs[j].wide != 0u;
        cut = cut || jobs[j].scene->any_hit_shadows == 0u;
        few_records = few_records && jobs[j].scene->wnode_count <= 64u;
    }
    if (n_jobs == 1u) set_scene0(p, *jobs[0].scene, wide);
    const bool one = n_jobs == 1u && jobs[0].job != nullptr;  // the launches carry the job
    if (one) p.job0 = *jobs[0].job;
    bool photons = false, debug = false;
    for (uint32_t j = 0; j < n_jobs; ++j) {
        photons = photons || jobs[j].photons != 0u;
        debug = debug || jobs[j].debug != 0u;
    }
    // Few pixels: the whole pass in one launch (paths_limit), with trees of a few dozen records, whose walks hardly
    // differ, up to 8/5 as many: Cornell box at 400 x 311, 1 and 4 spp, 155 and 526 us against 178 and 578, 20 leaf
    // cards 91 and 237 against 138 and 389; above that, at 512 x 300, the Cornell box 181 and 612 against 184 and 590.
    // Few paths left: the rest of them in one launch, tried at every third iteration, with photon maps (which end
    // most paths at once) at every second.  Gather without the tries over gather with them, rooms of 20k and 328k
    // triangles and the Cornell box, 1 to 4 spp, then with a photon map: 420 x 300 1.06 .. 1.20, 1.07 .. 1.67;
    // 640 x 360 1.00 .. 1.13, 1.05 .. 1.55; 800 x 600 0.99 .. 1.03, 1.00 .. 1.33; 1080p 0.99 .. 1.01, 1.00 .. 1.10.
    // (An idle try costs 2.5 us; the 0.99s are frames of one sample, whose paths are never few.)  With a limit of
    // half as many paths 1080p room frames measure 17.99 against 17.83 ms, with twice as many 17.98.
    // Both need the four-wide records, no debug view and no per-launch profile.
    const uint32_t most = wide && !debug && !prof && !p.work ? paths_limit(num_sms) : 0u;
    const uint32_t whole = few_records ? most + most / 5u * 3u : most;
    if (iters && slots <= whole) return launch_paths_frame(p, (uint32_t)tiles, iters, !one, photons, num_sms, st);
    if ((e = cudaMemsetAsync(p.counts, 0, sizeof(uint32_t) * 4 * (size_t)(iters + 1), st)) != cudaSuccess) return e;
    if (tiles)
        (one ? wf_generate_kernel<false> : wf_generate_kernel<true>)<<<(unsigned)((tiles + 3u) / 4u), 128, 0, st>>>(
            p, (uint32_t)tiles);
    WaveTuning t = tune;
    normalize_tuning(t, wide ? wide_need : stack_need);
    const TraceKernel trc = trace_kernel(t, wide, p.work != nullptr, n_jobs > 1u, cut);
    const size_t smem = trav_smem_bytes(t.block_threads, wide && t.treelet);
    // A launch carries up to one path per slot plus one occlusion ray per slot.
    const uint64_t blocks_needed = (2u * slots + t.block_threads - 1u) / t.block_threads;
    const uint64_t persistent = (uint64_t)num_sms * t.blocks_per_sm;
    const uint32_t grid = (uint32_t)(blocks_needed < persistent ? blocks_needed : persistent);
    const uint64_t shade_needed = (slots + 127u) / 128u, shade_cap = (uint64_t)num_sms * 2u * t.shade_blocks;
    const uint32_t shade_grid = (uint32_t)(shade_needed < shade_cap ? shade_needed : shade_cap);
    const uint64_t photon_cap = (uint64_t)num_sms * 16u;
    const uint32_t photon_grid = (uint32_t)(shade_needed < photon_cap ? shade_needed : photon_cap);
    // extend(0), shade(0), then per iteration one trace launch with the occlusion rays of the
    // iteration before and the closest-hit rays of this one, then its shade; the last occlusion rays
    // close the pass.
    void (*shade)(const WaveJob, uint32_t, uint32_t);
    if (one && !debug && t.shade_blocks == 6u)
        shade = photons ? wf_shade_kernel<true, false, false, 6> : wf_shade_kernel<false, false, false, 6>;
    else if (t.shade_blocks == 6u)
        shade = photons ? (debug ? wf_shade_kernel<true, true, true, 6> : wf_shade_kernel<true, false, true, 6>)
                        : (debug ? wf_shade_kernel<false, true, true, 6> : wf_shade_kernel<false, false, true, 6>);
    else if (t.shade_blocks == 5u)
        shade = photons ? (debug ? wf_shade_kernel<true, true, true, 5> : wf_shade_kernel<true, false, true, 5>)
                        : (debug ? wf_shade_kernel<false, true, true, 5> : wf_shade_kernel<false, false, true, 5>);
    else
        shade = photons ? (debug ? wf_shade_kernel<true, true, true, 4> : wf_shade_kernel<true, false, true, 4>)
                        : (debug ? wf_shade_kernel<false, true, true, 4> : wf_shade_kernel<false, false, true, 4>);
    // In a small pass each launch's blocks are scheduled while the one before drains.  In a large one that keeps
    // traversal and shade on the same SMs and with them the traversal's split of L1 for both.  Gather without it
    // over gather with it, rooms of 20k and 328k triangles and the Cornell box at 1 and 3 spp, then with a photon
    // map: 480 x 270 1.02 .. 1.17, 1.06 .. 1.24; 640 x 360, just below the line, 0.99 .. 1.11, 1.04 .. 1.19;
    // 800 x 600 1.00 .. 1.03, 1.03 .. 1.12; 1280 x 720 0.96 .. 0.99, 1.00 .. 1.06; config 2 0.95.  So the line is on
    // the safe side: the two are even near twice as many slots, and later with a photon map.
    const bool early = slots <= (uint64_t)num_sms * 1536u;
    uint32_t n_trc = 0, n_shd = 0, n_pho = 0;
    // Events of the profiled pass around one launch (never inside a captured graph: prof is null there).
    auto mark = [&](cudaEvent_t *ev, uint32_t i, int side) {
        if (prof && ev) cudaEventRecord(ev[2 * i + side], st);
    };
    for (uint32_t it = 0; it < iters; ++it) {
        mark(prof ? prof->trace_ev : nullptr, n_trc, 0);
        if ((e = launch_dependent_if(early, trc, grid, t.block_threads, smem, st, static_cast<const WaveParams &>(p), it, it ? it - 1u : kNoIter, t.chunk,
                                  trace_steps(t))) != cudaSuccess)
            return e;
        mark(prof ? prof->trace_ev : nullptr, n_trc++, 1);
        mark(prof ? prof->shade_ev : nullptr, n_shd, 0);
        uint32_t rest = 0u;
        if (most && it && (photons ? it % 2u == 1u && iters - it >= 2u : it % 3u == 0u && iters - it >= 3u)) {
            rest = most;
            if ((e = launch_paths_rest(p, it, rest, iters - it, !one, photons, early, num_sms, st)) != cudaSuccess) return e;
        }
        if ((e = launch_dependent_if(early, shade, shade_grid, 128u, 0, st, p, it, rest)) != cudaSuccess) return e;
        mark(prof ? prof->shade_ev : nullptr, n_shd++, 1);
        if (photons) {
            mark(prof ? prof->photon_ev : nullptr, n_pho, 0);
            if ((e = launch_dependent_if(early, one ? wf_photon_kernel<false> : wf_photon_kernel<true>, photon_grid, 128u, 0, st, p, it)) != cudaSuccess) return e;
            mark(prof ? prof->photon_ev : nullptr, n_pho++, 1);
        }
    }
    if (iters) {
        mark(prof ? prof->trace_ev : nullptr, n_trc, 0);
        if ((e = launch_dependent_if(early, trc, grid, t.block_threads, smem, st, static_cast<const WaveParams &>(p), kNoIter, iters - 1u, t.chunk, trace_steps(t))) !=
            cudaSuccess)
            return e;
        mark(prof ? prof->trace_ev : nullptr, n_trc++, 1);
    }
    if (prof) {
        prof->trace_launches = n_trc;
        prof->shade_launches = n_shd;
        prof->photon_launches = n_pho;
    }
    if (slots && (e = launch_dependent_if(early, one ? wf_finalize_kernel<false> : wf_finalize_kernel<true>, (unsigned)((slots + 255u) / 256u), 256u, 0, st, p,
                                       (uint32_t)slots)) != cudaSuccess)
        return e;
    return launch_dependent_if(early, wf_count_kernel, 1u, 32u, 0, st, static_cast<const WaveParams &>(p), iters);
}

}  // namespace rtd
