// One path of the gather pass (gather.wgsl:91-593), step by step: what the wavefront's kernels
// (k_wavefront.cu) each run for one queued path and the one-launch form (k_paths.cu) runs in a loop.
#pragma once
#include "rt_kernels.h"
#include "rt_traverse.cuh"

namespace rtd {

__device__ __forceinline__ float luma(f3 c) { return dot(c, mk3(0.2126f, 0.7152f, 0.0722f)); }

struct Accum {
    f3 col;
    float lum_sum, lum2_sum;
    float sl[8];
};
// The words of a slot's accumulator one shade step can change: every term it adds belongs to the
// sample it started with.  That sample's luminance sum lies beside the colour and the two luminance moments
// and goes to the list of the samples' sums when the sample ends, so a step reads and writes 32 bytes of the
// accumulator, not 64: batch of twelve 8.51 -> 8.43 ms, 256 x 256 frame
// 192 -> 187 us.
struct PathAcc {
    f3 col;
    float lum_sum, lum2_sum, sl;
};
// The NEE term of a path's last bounce waits in its slot (p.nee: the contribution and a word) until its
// occlusion ray has been traced: kNeeLit is set if the light is visible, and the slot's next shade (or
// finalize) adds the term first of all.  The word's low bits: the sample it belongs to, and whether only
// its luminance counts (photon debug).
constexpr uint32_t kNeePending = 0x20000u, kNeeLumaOnly = 0x10000u, kNeeLit = 0x80000000u;

__device__ __forceinline__ void add_radiance(PathAcc &a, f3 c) {
    a.col = a.col + c;
    float l = luma(c);
    a.lum_sum += l;
    a.lum2_sum += l * l;
    a.sl += l;
}
// One radiance term (or only its luminance) of an ended sample added straight into a slot's accumulator in
// memory: colour, the two luminance moments and the sample's luminance sum, as every path step adds them.
__device__ __forceinline__ void acc_add_term(const WaveParams &p, uint32_t slot, uint32_t s, f3 c, bool luma_only) {
    float4 *a = p.acc + 4 * (size_t)slot;
    float4 a0 = a[0];
    float *lum2 = reinterpret_cast<float *>(a + 1);
    const float l = luma(c);
    if (!luma_only) {
        a0.x = a0.x + c.x;
        a0.y = a0.y + c.y;
        a0.z = a0.z + c.z;
    }
    a0.w += l;
    a[0] = a0;
    *lum2 += l * l;
    if (s < 8u) reinterpret_cast<float *>(a + 2)[s] += l;
}
// A lit NEE term added to a slot's accumulator, whose words for sample s0 are in A.
__device__ __forceinline__ void add_nee(const float4 &nee, float4 *acc, uint32_t s0, PathAcc &A) {
    const uint32_t word = __float_as_uint(nee.w), s = word & 0xFFFFu;
    const f3 c = xyz(nee);
    const float l = luma(c);
    if (!(word & kNeeLumaOnly)) A.col = A.col + c;
    A.lum_sum += l;
    A.lum2_sum += l * l;
    if (s == s0) A.sl += l;
    else if (s < 8u) reinterpret_cast<float *>(acc + 2)[s] += l;  // the sample that ended with this term
}
__device__ __forceinline__ Accum load_acc(const WaveParams &p, uint32_t pix) {
    const float4 a = p.acc[4 * (size_t)pix], b = p.acc[4 * (size_t)pix + 1], c = p.acc[4 * (size_t)pix + 2],
                 d = p.acc[4 * (size_t)pix + 3];
    Accum A;
    A.col = mk3(a.x, a.y, a.z);
    A.lum_sum = a.w;
    A.lum2_sum = b.x;
    A.sl[0] = c.x; A.sl[1] = c.y; A.sl[2] = c.z; A.sl[3] = c.w;
    A.sl[4] = d.x; A.sl[5] = d.y; A.sl[6] = d.z; A.sl[7] = d.w;
    return A;
}

__device__ __forceinline__ f3 sky_color(f3 dir, f3 zenith, f3 horizon, float intensity) {
    float t = clampf(dir.y * 0.5f + 0.5f, 0.0f, 1.0f);
    return mix3(horizon, zenith, sqrtf(t)) * intensity;  // pow(t, 0.5) for t in [0, 1]
}
__device__ __forceinline__ float smith_g1(float nd, float a) {
    float k = a * 0.5f;
    return nd / (nd * (1.0f - k) + k);
}
__device__ __forceinline__ f3 spec_ggx(f3 wo, f3 n, f3 wi, float a, f3 f0) {
    float ndl = dot(n, wi);
    float ndv = dot(n, wo);
    if (ndl <= 0.0f || ndv <= 0.0f) return mk3(0.0f, 0.0f, 0.0f);
    f3 h = normalize(wo + wi);
    float ndh = fmaxf(dot(n, h), 0.0f);
    float a2 = a * a;
    float dd = ndh * ndh * (a2 - 1.0f) + 1.0f;
    float D = a2 / (kPi * dd * dd);
    f3 F = fresnel_schlick(fmaxf(dot(wo, h), 0.0f), f0);
    return F * (D * smith_g1(ndl, a) * smith_g1(ndv, a) / (4.0f * ndl * ndv));
}
// What the two lobes' direction samples have in common: the frame around n, the two random numbers, one's
// square root (r; w: the square root of its complement) and the other's angle.
struct DirSample {
    f3 t, b;
    float r, w, sp, cp;
};
__device__ __forceinline__ DirSample dir_sample(f3 n, bool spec, Rng &rng) {
    DirSample d;
    const f3 up = fabsf(n.y) < 0.999f ? mk3(0.0f, 1.0f, 0.0f) : mk3(1.0f, 0.0f, 0.0f);
    d.t = normalize(cross(up, n));
    d.b = cross(n, d.t);
    const float u1 = rng_f32(rng), u2 = rng_f32(rng);
    d.r = sqrtf(spec ? u1 : u2);
    d.w = sqrtf(1.0f - (spec ? u1 : u2));
    sincos_fixed(2.0f * kPi * (spec ? u2 : u1), d.sp, d.cp);
    return d;
}
__device__ __forceinline__ f3 sample_spec_dir(f3 rd, f3 n, float a, const DirSample &d) {
    const f3 bt = d.t, bb = d.b;
    f3 mrd = -rd;
    f3 v = mk3(dot(bt, mrd), dot(bb, mrd), dot(n, mrd));
    f3 vh = normalize(mk3(a * v.x, a * v.y, fmaxf(v.z, 1e-4f)));
    float l2 = vh.x * vh.x + vh.y * vh.y;
    f3 t1 = l2 > 0.0f ? mk3(-vh.y, vh.x, 0.0f) * (1.0f / sqrtf(l2)) : mk3(1.0f, 0.0f, 0.0f);
    f3 t2 = cross(vh, t1);
    float x = d.r * d.cp;
    float y = d.r * d.sp;
    float s = 0.5f * (1.0f + vh.z);
    float yy = (1.0f - s) * sqrtf(fmaxf(0.0f, 1.0f - x * x)) + s * y;
    f3 hh = x * t1 + yy * t2 + sqrtf(fmaxf(0.0f, 1.0f - x * x - yy * yy)) * vh;
    f3 hn = normalize(hh);
    f3 m = bt * hn.x + bb * hn.y + n * hn.z;
    f3 out = reflect(rd, m);
    return dot(out, n) > 0.0f ? out : reflect(rd, n);
}

// The light sample of direct_light (gather.wgsl:152-206) up to its shadow query.  `occlude` is set
// when the sample needs the shadow ray (origin o, direction ld, max_dist); e is the unoccluded value.
struct LightSample {
    f3 e, wi, o;
    float max_dist;
    bool occlude;
};
__device__ __forceinline__ LightSample light_sample(const DevJob &job, f3 hp, f3 sn, Rng &rng) {
    const DevScene &s = job.scene;
    const uint32_t n = s.light_count;
    const f3 zero = mk3(0.0f, 0.0f, 0.0f);
    LightSample ls{zero, sn, zero, 0.0f, false};
    if (n == 0u) return ls;
    uint32_t li = f2u_sat(rng_f32(rng) * (float)n);
    li = li < n ? li : n - 1u;
    const Light l = load_light(s, li);
    const float fn = (float)n;
    if (l.kind == 0u) {
        f3 to = l.data - hp;
        float r2 = dot(to, to);
        float r = sqrtf(r2);
        f3 ld = to / r;
        ls.wi = ld;
        if (dot(sn, ld) <= 0.0f) return ls;
        f3 pl = mk3(job.ip.point_light_emission[0], job.ip.point_light_emission[1], job.ip.point_light_emission[2]);
        ls.e = l.color * l.intensity * pl * fmaxf(dot(sn, ld), 0.0f) / (r2 + 0.01f) * fn;
        ls.o = hp + sn * 0.01f;
        ls.max_dist = r - 0.001f;
        ls.occlude = true;
    } else if (l.kind == 1u) {
        f3 ld = normalize(l.data);
        float ndl = dot(sn, ld);
        ls.wi = ld;
        if (ndl <= 0.0f) return ls;
        ls.e = l.color * l.intensity * ndl * fn;
        ls.o = hp + sn * 0.01f;
        ls.max_dist = 1e30f;
        ls.occlude = true;
    } else if (l.kind == 2u) {
        TriFull tri = load_tri(s, f2u_sat(l.data.x));
        Mat mat = load_mat(s, tri.material_id);
        float u1 = rng_f32(rng);
        float u2 = rng_f32(rng);
        float su = sqrtf(u1);
        float u = 1.0f - su;
        float v = u2 * su;
        float w = 1.0f - u - v;
        f3 lp = tri.v0 * w + tri.v1 * u + tri.v2 * v;
        float uvx = tri.uv0x * w + tri.uv1x * u + tri.uv2x * v;
        float uvy = tri.uv0y * w + tri.uv1y * u + tri.uv2y * v;
        f3 le = l.color;
        if (mat.tex_emissive != RT_TEX_NONE) {
            float4 t = tex_sample(s.tex[RT_TEX_EMISSIVE], uvx, uvy, (int32_t)mat.tex_emissive);
            le = le * mk3(t.x, t.y, t.z);
        }
        le = le * mk3(job.ip.light_emission[0], job.ip.light_emission[1], job.ip.light_emission[2]);
        f3 to = lp - hp;
        float r2 = dot(to, to);
        float r = sqrtf(r2);
        f3 ld = to / r;
        ls.wi = ld;
        float ndl = dot(sn, ld);
        if (ndl <= 0.0f) return ls;
        float ndl_l = dot(tri.gn, -ld);
        if (ndl_l <= 0.0f) return ls;
        float area = 0.5f * len3(cross(tri.v1 - tri.v0, tri.v2 - tri.v0));
        ls.e = le * l.intensity * ndl * ndl_l * area * fn / (r2 + 0.01f);
        ls.o = hp + sn * 0.01f;
        ls.max_dist = r - 0.001f;
        ls.occlude = true;
    }
    return ls;
}

__device__ __forceinline__ int32_t clampi(int32_t x, int32_t lo, int32_t hi) { return x < lo ? lo : (x > hi ? hi : x); }

// The camera ray of the pixel's next sample (gather.wgsl:292-297).
__device__ __forceinline__ void camera_ray(const DevJob &job, uint32_t px, uint32_t py, Rng &rng, f3 &ro, f3 &rd) {
    const rt_camera_uniform &cam = job.cam;
    float jx = rng_f32(rng) - 0.5f;
    float jy = rng_f32(rng) - 0.5f;
    float ux = ((float)px + jx) * cam.inv_half_res[0] - 1.0f;
    float uy = 1.0f - ((float)py + jy) * cam.inv_half_res[1];
    ro = mk3(cam.position[0], cam.position[1], cam.position[2]);
    rd = normalize(mk3(cam.forward[0], cam.forward[1], cam.forward[2]) +
                   mk3(cam.right[0], cam.right[1], cam.right[2]) * ux + mk3(cam.up[0], cam.up[1], cam.up[2]) * uy);
}

__device__ __forceinline__ uint32_t pack_sb(uint32_t s, uint32_t b) { return (s & 0xFFFFu) | (b << 16); }

// The last job whose first index (`first` of DevJob: base slot or first tile) is at or below i; jobs
// are laid out in order, so their first indices ascend.
template <bool kMulti, typename First>
__device__ __forceinline__ uint32_t job_of(const WaveParams &p, uint32_t i, First first) {
    if (!kMulti) return 0u;
    uint32_t lo = 0u, hi = p.n_jobs;
    while (hi - lo > 1u) {
        const uint32_t mid = (lo + hi) >> 1;
        if (first(p.jobs[mid]) <= i) lo = mid;
        else hi = mid;
    }
    return lo;
}

// The pixel's slot with the camera ray of its first sample (gather.wgsl:262-297) and nothing accumulated.
__device__ __forceinline__ void start_slot(const WaveParams &p, const DevJob &job, uint32_t jid, uint32_t px, uint32_t py,
                                           uint32_t slot) {
    uint32_t base_seed = slot - job.base + job.ip.frame * 2654435761u;
    Rng rng = rng_init(base_seed * 1664525u + 1013904223u);
    f3 ro, rd;
    camera_ray(job, px, py, rng, ro, rd);
    p.ro[slot] = make_float4(ro.x, ro.y, ro.z, __uint_as_float(rng.state));
    p.rd[slot] = make_float4(rd.x, rd.y, rd.z, __uint_as_float(pack_sb(0u, 0u)));
    p.thr[slot] = make_float4(1.0f, 1.0f, 1.0f, __uint_as_float(jid));
    const float4 z = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    p.acc[4 * (size_t)slot] = z;
    p.acc[4 * (size_t)slot + 1] = make_float4(0.0f, 1e30f, 0.0f, 0.0f);
    p.nrm[slot] = make_float4(0.0f, 1.0f, 0.0f, 0.0f);
    p.nee[slot] = z;
}

// What one shade step of a path leaves to do: its occlusion ray and photon-map lookup, and whether the slot
// goes on (the path's next segment or the pixel's next sample; ray and state are in the slot).
struct ShadeOut {
    bool keep = false, shadow = false, photon = false;
    f3 sh_o, sh_d;  // occlusion ray, up to sh_max
    float sh_max;
    f3 ph_hp, ph_n, ph_td;  // lookup: hit point, shading normal, throughput x diffuse weight
    uint32_t ph_sidx;
};

// One loop body of gather.wgsl:299-537 for the path in `slot`, whose ray hit triangle `prim` at hit_t (a miss:
// kInf); hmat: the hit's material, known before its triangle, or kNoMat.  lit: the light of the slot's
// pending NEE term is visible (also if its word says so).
template <bool kPhotons, bool kDebug, bool kMulti>
__device__ __forceinline__ ShadeOut shade_path(const WaveJob &p, uint32_t slot, float hit_t, uint32_t prim,
                                               uint32_t hmat, bool lit) {
    ShadeOut out;
    out.sh_o = out.sh_d = out.ph_hp = out.ph_n = out.ph_td = mk3(0.0f, 0.0f, 0.0f);
    out.sh_max = 0.0f;
    out.ph_sidx = 0u;
    const float4 o4 = p.ro[slot], d4 = p.rd[slot], t4 = p.thr[slot];
    const uint32_t jid = __float_as_uint(t4.w);
    const DevJob &job = job_at<kMulti>(p, jid);
    const DevScene &s = job.scene;
    const rt_image_params &ip = job.ip;
    const uint32_t W = ip.width;
    const uint32_t spp = job.spp;
    const uint32_t debug_view = ip._pad[0];
    const float env_intensity = s.env_intensity;
    const f3 env_color = mk3(s.env_color[0], s.env_color[1], s.env_color[2]);
    const f3 env_horizon = mk3(s.env_horizon[0], s.env_horizon[1], s.env_horizon[2]);
    const uint32_t pix = slot - job.base;
    f3 ro = xyz(o4), rd = xyz(d4), thr = xyz(t4);
    Rng rng{__float_as_uint(o4.w)};
    const uint32_t sb = __float_as_uint(d4.w);
    uint32_t sidx = sb & 0xFFFFu, b = sb >> 16;
    float4 *acc = p.acc + 4 * (size_t)slot;
    const uint32_t sidx0 = sidx;
    const float4 acc0 = acc[0], nee = p.nee[slot];
    float4 acc1 = acc[1];  // .x = lum2_sum, .y = first_depth, .z = this sample's luminance sum
    PathAcc A{xyz(acc0), acc0.w, acc1.x, acc1.z};
    const uint32_t nee_word = __float_as_uint(nee.w);
    if (lit || (nee_word & kNeeLit)) add_nee(nee, acc, sidx0, A);
    bool first_hit = false;  // this step found a nearer first hit (normal and depth change)
    float4 nrm = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    bool alive = true;  // the sample continues with another segment

    if (hit_t >= kInf) {
        if (b > 0u) add_radiance(A, thr * sky_color(rd, env_color, env_horizon, env_intensity));
        alive = false;
    } else {
        const TriFull tr = load_tri(s, prim);
        Mat mat;
        if (hmat != kNoMat) mat = load_mat(s, hmat);
        else mat = load_mat(s, tr.material_id);
        const f3 hp = ro + rd * hit_t;
        const Bary bb = barycentric(tr, ro, rd, hit_t);
        const float uvx = bb.uvx, uvy = bb.uvy;
        bool done_step = false;  // a `continue` of the reference loop

        if ((mat.flags & RT_MAT_FLAG_ALPHA_CUTOUT) != 0u && mat.tex_albedo != RT_TEX_NONE &&
            tex_sample(s.tex[RT_TEX_ALBEDO], uvx, uvy, (int32_t)mat.tex_albedo).w < 0.5f) {
            ro = hp + rd * 0.002f;
            done_step = true;
        }
        if (!done_step) {
            const f3 gn = tr.gn;
            const bool ff = dot(rd, gn) < 0.0f;
            const f3 sn_geom = smooth_normal(tr, bb, gn);
            const f3 sn = ff ? sn_geom : -sn_geom;
            f3 shn = sn;
            if (mat.tex_normal != RT_TEX_NONE) {
                float4 t = tex_sample(s.tex[RT_TEX_NORMAL], uvx, uvy, (int32_t)mat.tex_normal);
                f3 nm = mk3(t.x, t.y, t.z) * 2.0f - mk3(1.0f, 1.0f, 1.0f);
                f3 ft, fb;
                tangent_frame(tr, sn, ft, fb);
                shn = normalize(ft * nm.x + fb * nm.y + sn * nm.z);
            }
            if (b == 0u && hit_t < acc1.y) {
                nrm = make_float4(sn.x, sn.y, sn.z, 0.0f);
                first_hit = true;
                acc1.y = hit_t;
            }
            f3 albedo = mat.albedo;
            float rough = mat.roughness, metal = mat.metallic;
            if (mat.tex_albedo != RT_TEX_NONE) {
                float4 t = tex_sample(s.tex[RT_TEX_ALBEDO], uvx, uvy, (int32_t)mat.tex_albedo);
                albedo = mat.albedo * mk3(t.x, t.y, t.z);
            }
            if (mat.tex_mr != RT_TEX_NONE) {
                float4 mr = tex_sample(s.tex[RT_TEX_MR], uvx, uvy, (int32_t)mat.tex_mr);
                rough = clampf(mat.roughness * mr.y, 0.0f, 1.0f);
                metal = clampf(mat.metallic * mr.z, 0.0f, 1.0f);
            }
            f3 emis = mat.emissive;
            if (mat.tex_emissive != RT_TEX_NONE) {
                float4 t = tex_sample(s.tex[RT_TEX_EMISSIVE], uvx, uvy, (int32_t)mat.tex_emissive);
                emis = mat.emissive * mk3(t.x, t.y, t.z);
            }
            add_radiance(A, thr * emis);

            bool stop = false;
            if (kDebug && debug_view != 0u) {  // gather.wgsl:359-419
                const f3 half = mk3(0.5f, 0.5f, 0.5f);
                stop = true;
                switch (debug_view) {
                    case 1: A.col = mk3(uvx, uvy, 0.0f); break;
                    case 2: A.col = sn * 0.5f + half; break;
                    case 3: A.col = shn * 0.5f + half; break;
                    case 4: A.col = gn * 0.5f + half; break;
                    case 5: A.col = emis; break;
                    case 8:
                    case 9: {
                        float pu = (float)(pix % W) / (float)ip.width, pv = (float)(pix / W) / (float)ip.height;
                        float4 t =
                            tex_sample(s.tex[debug_view == 8 ? RT_TEX_EMISSIVE : RT_TEX_ALBEDO], pu, pv, 0);
                        A.col = mk3(t.x, t.y, t.z);
                        break;
                    }
                    case 11: {
                        float4 t = tex_sample(s.tex[RT_TEX_EMISSIVE], uvx, uvy, 0);
                        A.col = mk3(t.x, t.y, t.z);
                        break;
                    }
                    case 12: A.col = mat.emissive; break;
                    case 13: A.col = mk3((float)mat.tex_emissive / 65535.0f, 0.0f, 0.0f); break;
                    case 17: A.col = mk3(uvx - floorf(uvx), uvy - floorf(uvy), 0.0f); break;
                    case 18: {
                        float4 t = tex_sample(s.tex[RT_TEX_ALBEDO], uvx, uvy, (int32_t)mat.tex_albedo);
                        A.col = mk3(t.x, t.y, t.z);
                        break;
                    }
                    case 19:
                    case 20: {
                        f3 ft, fb;
                        tangent_frame(tr, sn, ft, fb);
                        A.col = (debug_view == 19 ? ft : fb) * 0.5f + half;
                        break;
                    }
                    case 21: A.col = hp; break;
                    default: stop = false; break;
                }
            }
            if (stop) {
                alive = false;
            } else if (mat.kind == 2u) {  // dielectric (gather.wgsl:421-436)
                float qd = (mat.ior - 1.0f) / (mat.ior + 1.0f);
                float f0s = qd * qd;
                float ct = fabsf(dot(rd, shn));
                float fr = fresnel_schlick(ct, mk3(f0s, f0s, f0s)).x;
                if (rng_f32(rng) < fr) {
                    rd = reflect(rd, shn);
                    ro = hp + shn * 0.001f;
                } else {
                    float eta = ff ? 1.0f / mat.ior : mat.ior;
                    rd = refract(rd, shn, eta);
                    ro = hp - shn * 0.001f;
                    thr = thr * mat.albedo;
                }
            } else {  // metallic-roughness (gather.wgsl:439-537)
                f3 f0 = mk3(0.04f * (1.0f - metal) + albedo.x * metal, 0.04f * (1.0f - metal) + albedo.y * metal,
                            0.04f * (1.0f - metal) + albedo.z * metal);
                f3 wo = -rd;
                float a = fmaxf(rough * rough, 1e-3f);
                f3 fr = fresnel_schlick(fabsf(dot(rd, shn)), f0);
                f3 diffuse_weight = (1.0f - metal) * albedo;
                float sp = max3(fr);
                float dp = max3(diffuse_weight);
                float ratio = sp / (sp + dp);
                float spec_prob = clampf(sp + dp <= 0.0f ? 0.5f : ratio, 0.001f, 0.999f);
                bool do_spec = rng_f32(rng) < spec_prob;
                f3 dscale = diffuse_weight / (1.0f - spec_prob);

                LightSample ls = light_sample(job, hp, shn, rng);
                // (What both lobes compute alike stands outside the branches: most warps have paths of both.)
                f3 lobe = dscale;
                if (!do_spec) {
                    if (env_intensity > 0.0f)
                        add_radiance(A, thr * dscale * sky_color(shn, env_color, env_horizon, env_intensity));
                    add_radiance(A, thr * albedo * ip.ambient);
                } else {
                    lobe = spec_ggx(wo, shn, ls.wi, a, f0);
                }
                const f3 c_nee = thr * lobe * ls.e / (do_spec ? spec_prob : kPi);
                bool nee_luma_only = false;
                if (kPhotons && ip.use_photons == 1u && !do_spec) {  // gather.wgsl:473-514
                    // The lookup runs in wf_photon_kernel right after this pass; its term
                    // lands before this bounce's NEE term, as here.  Photon debug mode
                    // overwrites the colour after the lookup and keeps only the luminance of
                    // the NEE term, whatever the lookup finds.
                    out.photon = true;
                    out.ph_hp = hp;
                    out.ph_n = shn;
                    out.ph_td = thr * dscale;
                    out.ph_sidx = sidx;
                    if (ip.photon_debug == 1u) nee_luma_only = true;
                }
                if (ls.occlude && (c_nee.x != 0.0f || c_nee.y != 0.0f || c_nee.z != 0.0f)) {
                    out.shadow = true;
                    out.sh_o = ls.o;
                    out.sh_d = ls.wi;
                    out.sh_max = ls.max_dist;
                    p.nee[slot] = make_float4(c_nee.x, c_nee.y, c_nee.z,
                                              __uint_as_float((sidx & 0xFFFFu) | kNeePending |
                                                              (nee_luma_only ? kNeeLumaOnly : 0u)));
                }
                const DirSample ds = dir_sample(shn, do_spec, rng);
                ro = hp + shn * 0.001f;
                if (do_spec) {
                    rd = sample_spec_dir(rd, shn, a, ds);
                    f3 h = normalize(wo + rd);
                    float ndl = fmaxf(dot(shn, rd), 0.0f);
                    thr = thr * fresnel_schlick(fmaxf(dot(wo, h), 0.0f), f0) * smith_g1(ndl, a) / spec_prob;
                } else {
                    rd = ds.t * (ds.cp * ds.w) + shn * ds.r + ds.b * (ds.sp * ds.w);
                    thr = thr * dscale;
                    if (kPhotons && ip.use_photons == 1u) alive = false;
                }
                if (alive) {
                    float pr = max3(thr);
                    if (pr <= 0.0f || rng_f32(rng) > pr) alive = false;
                    else thr = thr / pr;
                }
            }
        }
    }
    // for-loop step: the segment index advances; the sample ends after max_bounces segments.
    b += 1u;
    if (alive && b >= job.max_bounces) alive = false;
    if (!alive) {
        sidx += 1u;
        if (sidx < spp) {
            camera_ray(job, pix % W, pix / W, rng, ro, rd);
            thr = mk3(1.0f, 1.0f, 1.0f);
            b = 0u;
            out.keep = true;
        }
    } else {
        out.keep = true;
    }
    if (!out.shadow && nee_word != 0u) p.nee[slot].w = 0.0f;
    if (out.keep) {
        p.ro[slot] = make_float4(ro.x, ro.y, ro.z, __uint_as_float(rng.state));
        p.rd[slot] = make_float4(rd.x, rd.y, rd.z, __uint_as_float(pack_sb(sidx, b)));
        p.thr[slot] = make_float4(thr.x, thr.y, thr.z, __uint_as_float(jid));
    }
    const bool ended = sidx != sidx0;
    acc[0] = make_float4(A.col.x, A.col.y, A.col.z, A.lum_sum);
    acc[1] = make_float4(A.lum2_sum, acc1.y, ended ? 0.0f : A.sl, 0.0f);
    if (ended && sidx0 < 8u) reinterpret_cast<float *>(acc + 2)[sidx0] = A.sl;
    if (first_hit) p.nrm[slot] = nrm;
    return out;
}

// The photons a lookup may examine, as runs of the sorted array: at most one run per cell of the 27, hardly ever
// more than one per row of three.  A lane keeps run i at a[32 i] in shared memory for i < kRunsA, the others in b
// (local memory).  Its list of hits that wait to be added: entry i at [32 i].
constexpr uint32_t kLookupCells = 27u, kHitList = 24u, kMaxHits = 64u;
template <uint32_t kRunsA>
struct LookupRuns {
    uint2 *a, *b;
    __device__ __forceinline__ uint2 &operator[](uint32_t i) const { return i < kRunsA ? a[32u * i] : b[i - kRunsA]; }
};

// Squared distance along one axis from x to the photons of cell c: none lie nearer than its faces, less
// `margin` for the rounding in the key; those below the grid are kept in cell 0, and those beyond it in the
// cells of the next row or plane, a grid's width away.
__device__ __forceinline__ float cell_distance2(float x, float grid_min, float cell, int32_t c, float margin) {
    const float lo = grid_min + (float)c * cell;
    const float d = fmaxf(c == 0 ? 0.0f : lo - x, x - (lo + cell)) - margin;
    return d > 0.0f ? d * d : 0.0f;
}

// The photon-map lookup (gather.wgsl:473-514) of sample sidx of the path in `slot`: hit point hp, shading normal
// shn, throughput x diffuse weight td.  lanes: the lanes of the warp that call it together.
//
// The reference examines the 27 cells around the hit point in order (dz, then dy, then dx), at most 384
// photons, and adds the first 64 within the radius.  First the photons to test are laid out as runs: cells
// farther than the radius only use up the budget, neighbouring cells of a row merge.  With radius = cell / 2
// on a surface, four of its nine occupied cells remain.  Then the runs are tested as one flat loop over
// groups of eight photons, so a thread moves to its next run by itself.  Bound by the latency of the photon
// loads and by lanes that wait for the warp's longest lookup (11 of 32 active), so hits only go into a list of the
// lane; the warp adds them, four loaded at a time, when a list is nearly full.  1920 x 1080 at 4 spp, 2^20 photons
// in 128^3 cells, 3.19 ms of lookups per frame with every cell tested and a hit's loads between the tests, 2.38
// with the runs, 1.79 with groups of eight.  Relight and frame, then a batch of twelve: 4.67 and 9.30 ms with the
// 27 runs in shared memory, 4.51 and 9.15 with ten (its rest is L1) and positions loaded in pairs, 4.38 and 8.53
// with the lists (16 long: 4.40 and 8.55; eight hits at a time 4.60 and 8.62, two 4.62 and 9.05).
template <typename Runs>
__device__ __forceinline__ void photon_lookup(const WaveParams &p, const DevJob &job, uint32_t slot, uint32_t sidx, f3 hp,
                                              f3 shn, f3 td, uint32_t lanes, const Runs &runs, uint32_t *hit_list) {
    const rt_image_params &ip = job.ip;
    const rt_grid_params &gp = job.gp;
    const float radius = fabsf(ip.photon_radius), r2max = radius * radius, cell = gp.cell_size;  // (only its square counts)
    const int32_t bx = f2i_sat((hp.x - gp.room_min_x) / cell);
    const int32_t by = f2i_sat((hp.y - gp.room_min_y) / cell);
    const int32_t bz = f2i_sat((hp.z - gp.room_min_z) / cell);
    const int32_t gx = (int32_t)gp.grid_x, gy = (int32_t)gp.grid_y, gz = (int32_t)gp.grid_z;
    uint32_t n_runs = 0u;
    if (job.sorted_count != 0u) {
        // Cells may be passed over when a hit point this near the grid is farther than the radius from every
        // photon that some other row's or plane's overflow put among theirs.
        const float wide = (float)min(gx, min(gy, gz)) - 2.0f;
        const bool pass = bx >= -1 && by >= -1 && bz >= -1 && bx <= gx && by <= gy && bz <= gz && wide * cell > radius * 1.01f;
        const float far2 = pass ? r2max * (1.0f + 0x1p-18f) : __int_as_float(0x7F800000);
        const float margin = 0x1p-19f * (fabsf(gp.room_min_x) + fabsf(gp.room_min_y) + fabsf(gp.room_min_z) +
                                         (float)max(gx, max(gy, gz)) * cell);
        int32_t cx[3], cy[3], cz[3];
        float dx2[3], dy2[3], dz2[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            cx[d] = clampi((int32_t)((uint32_t)bx + (uint32_t)(d - 1)), 0, gx - 1);
            cy[d] = clampi((int32_t)((uint32_t)by + (uint32_t)(d - 1)), 0, gy - 1);
            cz[d] = clampi((int32_t)((uint32_t)bz + (uint32_t)(d - 1)), 0, gz - 1);
            dx2[d] = cell_distance2(hp.x, gp.room_min_x, cell, cx[d], margin);
            dy2[d] = cell_distance2(hp.y, gp.room_min_y, cell, cy[d], margin);
            dz2[d] = cell_distance2(hp.z, gp.room_min_z, cell, cz[d], margin);
        }
        uint32_t budget = 384u;
        uint2 run = make_uint2(0u, 0u);
#pragma unroll
        for (int z = 0; z < 3; ++z) {
#pragma unroll
            for (int y = 0; y < 3; ++y) {
                const uint2 *row = job.grid_meta + ((uint32_t)cy[y] * gp.grid_x + (uint32_t)cz[z] * gp.grid_x * gp.grid_y);
                const float row2 = dy2[y] + dz2[z];
#pragma unroll
                for (int x = 0; x < 3; ++x) {
                    const uint2 m = __ldg(row + cx[x]);
                    const uint32_t take = min(m.y, budget);
                    budget -= take;
                    if (take != 0u && !(row2 + dx2[x] > far2)) {
                        if (run.x + run.y == m.x && run.y != 0u) {
                            run.y += take;
                        } else {
                            if (run.y != 0u) runs[n_runs++] = run;
                            run = make_uint2(m.x, take);
                        }
                    }
                }
            }
        }
        if (run.y != 0u) runs[n_runs++] = run;
    }
    // Photon indices are u32 and clamped to the last sorted photon (the backend's rule for an
    // out-of-range index; the grid's ranges never leave the array).
    const uint32_t last = (uint32_t)job.sorted_count - 1u;
    const float4 *posv = job.sorted_pos;
    f3 ph_sum = mk3(0.0f, 0.0f, 0.0f);
    uint32_t ph_hits = 0u, waiting = 0u;  // hits added, hits in the lane's list
    auto add_hits = [&]() {
        for (uint32_t k = 0u; k < waiting; k += 4u) {
            float4 pw[4], inc[4];
#pragma unroll
            for (uint32_t j = 0; j < 4u; ++j) {
                const float4 *ph = job.sorted_photons + 4ull * hit_list[32u * min(k + j, waiting - 1u)];
                pw[j] = __ldg(ph + 1);
                inc[j] = __ldg(ph + 2);
            }
#pragma unroll
            for (uint32_t j = 0; j < 4u; ++j)
                if (k + j < waiting) ph_sum = ph_sum + xyz(pw[j]) * fmaxf(dot(shn, -xyz(inc[j])), 0.0f);
        }
        ph_hits += waiting;
        waiting = 0u;
    };
    bool more = n_runs != 0u;
    uint2 m = more ? runs[0] : make_uint2(0u, 0u);
    uint32_t ri = 1u;
    while (__any_sync(lanes, more)) {
        if (more) {
            // A group of up to eight photons: the four pairs of positions that hold the first are loaded together.
            float4 pos[8];
            const uint32_t first = m.x & ~1u, skip = m.x & 1u;
#pragma unroll
            for (uint32_t j = 0; j < 8u; j += 2u) ldg32(posv + min(first + j, last & ~1u), pos[j], pos[j + 1]);
            const uint32_t group = min(m.y, 8u - skip);
            uint32_t hits = 0u;
#pragma unroll
            for (uint32_t j = 0; j < 8u; ++j) {
                const f3 dd = xyz(pos[j]) - hp;
                const float d2 = dot(dd, dd);
                if (d2 < r2max) hits |= 1u << j;
            }
            hits &= ((1u << group) - 1u) << skip;
#pragma unroll
            for (uint32_t j = 0; j < 8u; ++j)
                if (hits >> j & 1u) hit_list[32u * waiting++] = min(first + j, last);
            m.x += group;
            m.y -= group;
            if (ph_hits + waiting >= kMaxHits) {
                waiting = kMaxHits - ph_hits;
                more = false;
            } else if (m.y == 0u) {
                more = ri < n_runs;
                if (more) m = runs[ri++];
            }
        }
        if (__any_sync(lanes, waiting > kHitList - 8u)) add_hits();
    }
    add_hits();
    if (ph_hits > 0u)
        acc_add_term(p, slot, sidx, td * ph_sum * ip.photon_scale / (kPi * (float)ph_hits * ip.photon_radius * ip.photon_radius),
                     false);
    if (ip.photon_debug == 1u) {
        const float density = fminf((float)ph_hits / 64.0f, 1.0f);
        const f3 col = mk3(1.0f - density, density, 0.0f) * 2.0f;
        float4 *a = p.acc + 4 * (size_t)slot;
        a[0] = make_float4(col.x, col.y, col.z, a[0].w);
    }
}

// Whether the light of an occlusion ray in a scene with cut-out materials is visible (gather.wgsl:91-103):
// its closest hit (hit_word) lies at or beyond the limit, or is cut away there by its texture's alpha.  Out of
// line: few scenes need it, and its registers would weigh on the traversal.
static __device__ __noinline__ bool cut_out_lit(const DevScene &s, float4 ro, float4 rd, float limit,
                                         unsigned long long hit) {
    const float t = hit_t(hit);
    if (t >= limit) return true;  // (not for a NaN limit, which counts as occluded)
    const TriFull bt = load_tri(s, t < kInf ? __float_as_uint(__ldg(s.tri_ord + 3ull * (uint32_t)hit).w) : 0u);
    const Mat bm = load_mat(s, bt.material_id);
    if ((bm.flags & RT_MAT_FLAG_ALPHA_CUTOUT) == 0u || bm.tex_albedo == RT_TEX_NONE) return false;
    const Bary b = barycentric(bt, xyz(ro), xyz(rd), t);
    return tex_sample(s.tex[RT_TEX_ALBEDO], b.uvx, b.uvy, (int32_t)bm.tex_albedo).w < 0.5f;
}

// The pixel in `slot`: the last NEE term, the firefly sigma clamp and the frame outputs (gather.wgsl:548-593).
__device__ __forceinline__ void finalize_slot(const WaveParams &p, const DevJob &job, uint32_t slot) {
    const uint32_t pix = slot - job.base;
    if (pix >= job.npix) return;
    const uint32_t spp = job.spp;
    Accum A = load_acc(p, slot);
    const float4 nee = p.nee[slot];
    if (__float_as_uint(nee.w) & kNeeLit) {  // the last bounce's term
        const uint32_t word = __float_as_uint(nee.w), s = word & 0xFFFFu;
        const float l = luma(xyz(nee));
        if (!(word & kNeeLumaOnly)) A.col = A.col + xyz(nee);
        A.lum_sum += l;
        A.lum2_sum += l * l;
#pragma unroll
        for (uint32_t i = 0; i < 8u; ++i)
            if (i == s) A.sl[i] += l;
    }
    const float first_depth = p.acc[4 * (size_t)slot + 1].y;
    const float4 nrm = p.nrm[slot];
    if (spp <= 8u) {
        float *sl = A.sl;
        for (uint32_t i = 1; i < spp; ++i) {
            float key = sl[i];
            uint32_t j = i;
            while (j > 0u && sl[j - 1u] > key) {
                sl[j] = sl[j - 1u];
                j -= 1u;
            }
            sl[j] = key;
        }
        float median = (sl[(spp - 1u) / 2u] + sl[spp / 2u]) * 0.5f;
        uint32_t half = spp / 2u > 1u ? spp / 2u : 1u;
        float spread = 0.0f;
        for (uint32_t i = 0; i < half; ++i) {
            float dd = sl[i] - median;
            spread += dd * dd;
        }
        float sigma = fmaxf(sqrtf(spread / (float)half), 0.25f * median + 1e-5f);
        float thresh = median + 3.0f * sigma;
        float cl = 0.0f, cl2 = 0.0f;
        for (uint32_t i = 0; i < spp; ++i) {
            float lc = fminf(sl[i], thresh);
            cl += lc;
            cl2 += lc * lc;
        }
        A.col = A.col * (cl / fmaxf(A.lum_sum, 1e-10f));
        A.lum_sum = cl;
        A.lum2_sum = cl2;
    }
    f3 col = vmin(A.col / (float)spp, mk3(10.0f, 10.0f, 10.0f));
    job.frame[pix] = make_float4(col.x, col.y, col.z, 1.0f);
    job.moments[pix] = make_float4(fminf(A.lum_sum / (float)spp, 10.0f), fminf(A.lum2_sum / (float)spp, 100.0f), 0.0f, 0.0f);
    job.gbuffer[pix] = make_float4(nrm.x, nrm.y, nrm.z, first_depth);
}

}  // namespace rtd
