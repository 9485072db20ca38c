// The gather pass of few paths in one launch (gather.wgsl:91-593).  A warp takes up to 32 paths and runs
// extend, shade, photon lookup and shadow for all of them until the last sample of the last pixel has ended,
// with the wavefront's traversal (the occlusion rays of a step ride with the closest-hit rays of the next one,
// taken by whichever lanes are idle) and its per-path steps in the same order, so the images are the same
// bit for bit.  Two uses:
//
//   a frame of few pixels as a whole, generate and finalize included;
//   the end of a larger frame: a launch in front of a shade pass that returns at once while more than `most`
//   paths are queued and otherwise runs all that is left of them.
//
// What bounds few paths in the wavefront is its chain of launches, each of them one dependent load after the
// other for a fraction of a warp per scheduler: the Cornell box at 256 x 256, 5 segments deep, took 15
// launches and 188 us.  Here a warp waits for its own loads only.  It is bound by the fetch and the latency of one
// path's instructions (16 warps per SM, issue 45% of cycles): 118 us for that frame, 40% of it waits for instructions,
// before the warps of a block shaded together, 95 with that, 84 since idle lanes look for work after every
// record.  With more paths than the SMs hold at once the compacted queues win: lanes whose path has ended idle
// here until the warp's last one ends.
#include "rt_paths.cuh"

namespace rtd {

namespace {
constexpr int kPathsBlock = 256, kPathsBlocksPerSm = 2;  // 128 registers
// Paths per warp when they are too few for 32 each: below this a warp's idle lanes gain nothing (measured at
// 64 x 64: 2, 4 and 8 alike, 16 10% slower, 32 28%).
constexpr uint32_t kPathsShare = 4;
}  // namespace

template <bool kMulti, bool kPhotons, bool kWhole>
__global__ void __launch_bounds__(kPathsBlock, kPathsBlocksPerSm) wf_paths_kernel(const __grid_constant__ WaveJob p,
                                                                                  uint32_t iter, uint32_t most,
                                                                                  uint32_t steps) {
    extern __shared__ __align__(16) unsigned char trav_smem[];
    grid_dependency_wait();
    grid_launch_dependents();
    // kWhole: `most` pixel positions, 8 x 4 tiles as in generate; otherwise the paths queued for `iter`.  steps: the
    // shade steps a path may take, the wavefront's iterations (a path's 16-bit sample and segment numbers wrap around
    // before 65,537 samples or segments are done, so they alone would not end it).
    const uint32_t n = kWhole ? most : p.counts[4 * iter];
    if (!kWhole && n > most) return;
    const uint32_t lane = threadIdx.x & 31u;
    uint2 *top = reinterpret_cast<uint2 *>(trav_smem) + threadIdx.x;
    uint2 deep[kMaxStack - kTopStack];
    WarpTrav &w = reinterpret_cast<WarpTrav *>(trav_smem + sizeof(uint2) * kTopStack * kPathsBlock)[threadIdx.x >> 5];
    // Between walks the warp's traversal state holds the photon lookups' runs and hits.
    constexpr uint32_t kRunsA = 4;
    uint2 rest[kLookupCells - kRunsA];
    const LookupRuns<kRunsA> runs{reinterpret_cast<uint2 *>(&w) + lane, rest};
    uint32_t *hit_list = reinterpret_cast<uint32_t *>(runs.a - lane + 32u * kRunsA) + lane;
    static_assert(sizeof(WarpTrav) >= 32 * (kRunsA * sizeof(uint2) + kHitList * sizeof(uint32_t)), "lookup state");
    // A step is some 3,000 instructions without a loop, which the warps of a scheduler would each fetch at another
    // place (40% of their cycles), so a block's warps start each shade step together: 16 Cornell frames of
    // 256 x 256 2.07 -> 1.71 ms (blocks of four warps 1.79, of sixteen 1.73).  With photon maps too: gather of a whole
    // Cornell frame at 300 x 240, 1 / 4 spp, 0.067 / 0.217 ms against 0.082 / 0.333 with each warp on its own, a
    // 20k-triangle room 0.250 / 0.967 against 0.279 / 1.137; the last paths of 640 x 360 0.494 / 1.899 against
    // 0.515 / 1.989 in the room, 0.197 / 0.650 against 0.195 / 0.643 in the Cornell box.
    const Treelet tree{nullptr, nullptr, 0u};
    LaneWalk r;
    r.busy = r.visiting = r.any_hit = false;
    r.st.sp = 0u;
    uint32_t segments = 0u, shadow_rays = 0u;
    // Few paths are spread over all warps.
    const uint32_t warps = gridDim.x * (kPathsBlock / 32);
    const uint32_t share = min(32u, max(kPathsShare, (n + warps - 1u) / warps));
    for (uint32_t first = 0u; first < n; first += share * warps) {  // (the same rounds for a block's warps)
        const uint32_t base = first + share * (blockIdx.x * (kPathsBlock / 32) + (threadIdx.x >> 5));
        bool alive = lane < share && base + lane < n;
        uint32_t slot = 0u, jid = 0u;
        if (kWhole) {
            const uint32_t at = min(base + lane, n - 1u), gtile = at >> 5;
            jid = job_of<kMulti>(p, gtile, [](const DevJob &j) { return j.tile0; });
            const DevJob &job = job_at<kMulti>(p, jid);
            const uint32_t W = job.ip.width, tiles_x = (W + 7u) / 8u, tile = gtile - job.tile0;
            const uint32_t px = tile % tiles_x * 8u + (at & 7u), py = tile / tiles_x * 4u + (at >> 3 & 3u);
            alive = alive && px < W && py < job.ip.height;
            slot = job.base + py * W + px;
            if (alive) start_slot(p, job, jid, px, py, slot);
        } else if (alive) {
            slot = p.queue[iter & 1u][base + lane];
            if (kMulti) jid = __float_as_uint(p.thr[slot].w);
        }
        const bool mine = alive;
        bool lookup = false;  // a photon lookup waits in the slot's record of preq
        const DevJob &job = job_at<kMulti>(p, jid);
        const DevScene &sc = job.scene;
        auto look_up = [&]() {
            const uint32_t lanes = __ballot_sync(0xFFFFFFFFu, lookup);
            if (lookup) {
                const float4 *req = p.preq + 3ull * slot;
                const float4 r0 = req[0], r1 = req[1], r2 = req[2];
                photon_lookup(p, job, slot, __float_as_uint(r0.w), xyz(r0), xyz(r1), xyz(r2), lanes, runs, hit_list);
                lookup = false;
            }
            __syncwarp();
        };
        const float4 *records = kMulti ? sc.wnodes : p.records0, *tris = kMulti ? sc.tri_ord : p.tris0;
        const bool empty = kMulti ? sc.cnode_count == 0u : p.empty0 != 0u;
        const bool any = kMulti ? sc.any_hit_shadows != 0u : p.any_hit0 != 0u;
        ShadeOut out;
        out.sh_o = out.sh_d = mk3(0.0f, 0.0f, 0.0f);
        out.sh_max = 0.0f;
        uint32_t left = steps;
        for (bool traced = !kWhole;; traced = false) {
            float hit_dist = kInf;
            uint32_t hit_slot = 0u;
            bool lit = false;
            if (traced) {  // the wavefront has traced the queued paths and the shadow rays before them
                if (alive) {
                    const float2 h = p.hit[slot];
                    hit_dist = h.x;
                    hit_slot = __float_as_uint(h.y);
                }
            } else {
                // The occlusion rays of the last shade step, packed for whichever lane takes them; the
                // direction's .w: the lane that waits for the answer.
                const uint32_t occ_mask = __ballot_sync(0xFFFFFFFFu, out.shadow), n_occ = __popc(occ_mask);
                if (out.shadow) {
                    const uint32_t k = __popc(occ_mask & lanemask_lt());
                    w.next_ro[k] = make_float4(out.sh_o.x, out.sh_o.y, out.sh_o.z, out.sh_max);
                    w.next_rd[k] = make_float4(out.sh_d.x, out.sh_d.y, out.sh_d.z, __uint_as_float(lane));
                    if (kMulti) w.next_queue[k] = jid;
                    shadow_rays += 1u;
                }
                if (lane == 0u) w.coming = 0u;  // the answers: lanes whose light is visible
                __syncwarp();
                uint32_t at = 0u, owner = lane, occ_job = 0u;
                bool occ = false;
                if (alive) {
                    const float4 o = p.ro[slot], d = p.rd[slot];
                    r.st.records = records;
                    r.st.cap = kMaxStack;
                    r.any_hit = false;
                    r.st.t = kInf;
                    walk_begin(r, w, xyz(o), xyz(d), mk3(1.0f, 1.0f, 1.0f) / xyz(d), tris);
                    r.visiting = !empty;
                    segments += 1u;
                }
                for (;;) {
                    const uint32_t idle = __ballot_sync(0xFFFFFFFFu, !r.busy);
                    if (idle == 0xFFFFFFFFu && at == n_occ) break;
                    if (idle != 0u && at != n_occ) {
                        const uint32_t k = at + __popc(idle & lanemask_lt());
                        if (!r.busy && k < n_occ) {
                            const float4 o = w.next_ro[k], d = w.next_rd[k];
                            owner = __float_as_uint(d.w);
                            occ = true;
                            const float4 *otris = tris;
                            bool oany = any;
                            r.st.records = records;
                            r.st.cap = kMaxStack;
                            if (kMulti) {
                                occ_job = w.next_queue[k];
                                const DevScene &os = p.jobs[occ_job].scene;
                                r.st.records = os.wnodes;
                                otris = os.tri_ord;
                                oany = os.any_hit_shadows != 0u;
                            }
                            // (see wf_trace_kernel)
                            r.any_hit = oany;
                            r.st.t = o.w - 0.001f;
                            if (!oany) {
                                w.limit[lane] = r.st.t;
                                r.st.t = kInf;
                            }
                            walk_begin(r, w, xyz(o), xyz(d), mk3(1.0f, 1.0f, 1.0f) / xyz(d), otris);
                            r.visiting = r.st.t > kEps;
                        }
                        at = min(at + (uint32_t)__popc(idle), n_occ);
                    }
                    uint32_t visits = 0u, tests = 0u;
                    // (a refill costs little here: three records between them 1.73 ms for the 16 frames, two 1.66,
                    // one 1.57)
                    walk_records<true, 0, kPathsBlock, kMulti, false>(r, w, top, deep, tree, p.records0, p.tris0, 1u, 0,
                                                                      visits, tests);
                    if (r.busy && !r.visiting) {
                        bool clear = !r.found && r.st.t == r.st.t;  // (a NaN limit counts as occluded)
                        if (!r.any_hit) {
                            const unsigned long long hit = w.best[lane];
                            if (occ) {
                                clear = cut_out_lit(job_at<kMulti>(p, occ_job).scene, w.ro[lane], w.rd[lane], w.limit[lane], hit);
                            } else {
                                hit_dist = hit_t(hit);
                                hit_slot = (uint32_t)hit;
                            }
                        }
                        if (occ && clear) atomicOr(&w.coming, 1u << owner);
                        r.busy = false;
                    }
                }
                __syncwarp();
                lit = (w.coming >> lane & 1u) != 0u;
                __syncwarp();
            }
            if (!alive) {
                // an ended path's last term is finalize's to add
                if (lit) p.nee[slot].w = __uint_as_float(__float_as_uint(p.nee[slot].w) | kNeeLit);
                out.shadow = false;
            }
            if (!__syncthreads_or(alive)) break;
            if (alive) {
                uint32_t prim = 0u, word = 0u;
                if (hit_dist < kInf) {
                    prim = __float_as_uint(__ldg(tris + 3ull * hit_slot).w);
                    word = __float_as_uint(__ldg(tris + 3ull * hit_slot + 1).w);
                }
                out = shade_path<kPhotons, false, kMulti>(p, slot, hit_dist, prim, word >> 2, lit);
                if (kPhotons && out.photon) {
                    float4 *req = p.preq + 3ull * slot;
                    req[0] = make_float4(out.ph_hp.x, out.ph_hp.y, out.ph_hp.z, __uint_as_float(out.ph_sidx));
                    req[1] = make_float4(out.ph_n.x, out.ph_n.y, out.ph_n.z, 0.0f);
                    req[2] = make_float4(out.ph_td.x, out.ph_td.y, out.ph_td.z, 0.0f);
                    lookup = true;
                }
                alive = out.keep && left > 1u;
            }
            left -= 1u;
            // A lookup's term comes before the next one added to its slot: the lookups wait until a lane that
            // has one goes on, or the block's paths have all ended, and run together
            // (640 x 360 with a photon map, four frames: 2.15 ms with each lookup right after its shade step).
            if (kPhotons && __any_sync(0xFFFFFFFFu, lookup && alive)) look_up();
        }
        if (kPhotons) look_up();
        if (kWhole && mine) finalize_slot(p, job, slot);
    }
    segments = __reduce_add_sync(0xFFFFFFFFu, segments);
    shadow_rays = __reduce_add_sync(0xFFFFFFFFu, shadow_rays);
    if (lane == 0u && p.counters && (segments | shadow_rays) != 0u) {
        atomicAdd(p.counters, (unsigned long long)segments);
        atomicAdd(p.counters + 1, (unsigned long long)shadow_rays);
    }
}

namespace {
using PathsKernel = void (*)(const WaveJob, uint32_t, uint32_t, uint32_t);
template <bool kWhole>
PathsKernel paths_kernel(bool multi, bool photons) {
    if (multi) return photons ? wf_paths_kernel<true, true, kWhole> : wf_paths_kernel<true, false, kWhole>;
    return photons ? wf_paths_kernel<false, true, kWhole> : wf_paths_kernel<false, false, kWhole>;
}
}  // namespace

void prepare_paths_kernels() {
    for (int v = 0; v < 4; ++v) {
        const int bytes = (int)trav_smem_bytes(kPathsBlock, false);
        cudaFuncSetAttribute(reinterpret_cast<const void *>(paths_kernel<true>((v & 1) != 0, (v & 2) != 0)),
                             cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
        cudaFuncSetAttribute(reinterpret_cast<const void *>(paths_kernel<false>((v & 1) != 0, (v & 2) != 0)),
                             cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    }
}

// As many paths as the SMs hold threads of the kernel.  Measured against the wavefront (gather, ms, 1 and 4 spp):
// 304 x 250 in a 20k-triangle room 0.28 / 0.99 against 0.38 / 1.17, in a 328k-triangle room 0.46 / 1.59 against
// 0.60 / 1.70, cut-out foliage 0.19 / 0.64 against 0.28 / 0.85; above the limit, 352 x 280, 0.40 / 1.45 against
// 0.39 / 1.31 and 0.63 / 2.20 against 0.64 / 1.97 in the rooms.  (With photon maps it still gains there: 0.29 / 1.16
// against 0.37 / 1.33, up to 480 x 270.)
uint32_t paths_limit(int num_sms) { return (uint32_t)num_sms * kPathsBlocksPerSm * kPathsBlock; }

cudaError_t launch_paths_frame(const WaveJob &p, uint32_t tiles, uint32_t steps, bool multi, bool photons, int num_sms,
                               cudaStream_t st) {
    const uint32_t blocks = (uint32_t)num_sms * kPathsBlocksPerSm;
    paths_kernel<true>(multi, photons)<<<blocks, kPathsBlock, trav_smem_bytes(kPathsBlock, false), st>>>(p, 0u, 32u * tiles,
                                                                                                        steps);
    return cudaGetLastError();
}

cudaError_t launch_paths_rest(const WaveJob &p, uint32_t iter, uint32_t most, uint32_t steps, bool multi, bool photons,
                              bool early, int num_sms, cudaStream_t st) {
    const uint32_t blocks = (uint32_t)num_sms * kPathsBlocksPerSm;
    return launch_dependent_if(early, paths_kernel<false>(multi, photons), blocks, kPathsBlock,
                               trav_smem_bytes(kPathsBlock, false), st, p, iter, most, steps);
}

}  // namespace rtd
