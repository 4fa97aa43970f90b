// One path between its vertices: the records and requests of a render, camera
// samples, hits, emitter sampling, and the vertex functions (emitter hit,
// Russian roulette, next-event estimation, BSDF sampling) that the wavefront
// kernels (render.cu) and the resident kernel (resident.cu) share.
#pragma once

#include "device.cuh"
#include "guide.cuh"
#include "internal.h"

namespace dl {

enum PathFlags { PF_CAMERA = 1, PF_PREV_DIFFUSE = 2, PF_ENDED = 4 };

struct __align__(32) RayRec {
    float4 o;   // origin, tmin
    float4 d;   // direction, tmax
};
struct __align__(32) PathRec {
    float4 tp;  // throughput.rgb, eta
    float4 L;   // radiance.rgb, pdf of the last BSDF sample
};
struct __align__(32) MetaRec {
    int4 m;     // depth, flags, path index lo, path index hi
    uint4 rng;  // pcg32 state lo/hi, inc lo/hi
};
struct __align__(32) HitRec {
    float4 h;   // t, u, v, leaf-order triangle (int bits; -1 = miss)
    float4 pad;
};
static_assert(sizeof(RayRec) == 32 && sizeof(PathRec) == 32 && sizeof(MetaRec) == 32 && sizeof(HitRec) == 32,
              "path records are one 32-byte sector each");
// A slot's four records share one 128-byte line: the ray and its hit in one
// half, the path state in the other.  Slots are visited in queue order, i.e.
// at random; a random 32-byte read costs a whole DRAM burst, so records read
// together are kept inside one.
struct __align__(128) SlotRec {
    RayRec ray;
    HitRec hit;
    PathRec path;
    MetaRec meta;
};
static_assert(sizeof(SlotRec) == 128, "one 128-byte line per slot");
constexpr size_t kSlotBytes = 4 * 32 + 8 + 3 * 16 + 4 * (2 + kNumMaterialTypes + 1);  // records, pos, shadow, queues

constexpr int kMissQueue = kNumMaterialTypes;  // queue index of rays that hit nothing

// One render request: a scene and its render options.  A single render has
// one request, carried in the kernel parameters; a batch has a table of them
// in device memory and every path carries its request's index (in the path
// flags, in the ray records' w slot).
struct DevRequest {
    DevScene sc;
    unsigned long long pid_first;  // the request's first path index in the current pass
    int spp_offset;                // sample index of its first sample in the pass
    int max_depth;
    int rr_depth;
    unsigned int flags;
    unsigned long long seed_mix;
};
constexpr int kReqShift = 8;  // path flags: request index << kReqShift | PathFlags

// Guided renders: per slot, the training records of the path's two most
// recent guided vertices with the throughput after each (a: older, b: newer;
// record index in w, -1 for none).  Radiance the path gathers later is
// credited to them divided by that throughput: the estimate of the radiance
// arriving along the direction sampled there.
struct __align__(32) GuideRec {
    float4 a;
    float4 b;
};

struct RenderParams {
    DevRequest r0;                 // the request of a single render
    int capacity;                  // path slots (queue and record arrays hold this many entries)
    const DevRequest* reqs;        // batch: request table (pid_first ascending)
    int num_reqs;
    SlotRec* rec;    // per slot: ray, hit, path state
    float2* pos;     // film position of the camera sample (Li mode only)
    int* ext_q[2];
    int* mat_q[kNumMaterialTypes + 1];  // per material type, then the miss queue
    float4* sh_o;
    float4* sh_d;
    float4* sh_c;    // contribution.rgb, target: slot >= 0 (live path) or -1 - path index (ended path)
    RenderCounters* cnt;
    float4* samples; // radiance.rgb + presence flag per path index of this chunk
    int mode;        // 0: film, 1: Li of explicit paths
    const int* xys;
    float* li_L;
    float* li_pos;
    unsigned long long total;  // resident kernel: paths of the pass
    // guided renders
    int guided;
    GuideNet gnet;
    GuideRec* grec;
    GuideRecord* grecords;
    int grecord_cap;
};

template <bool kMulti>
__device__ __forceinline__ const DevRequest& request(const RenderParams& P, int rid) {
    if (kMulti) return P.reqs[rid];
    return P.r0;
}

// Bounds-checked build (compiled with -DDL_CHECKS): before each access whose
// index comes from a queue, a counter or a record -- path slots, queue
// positions, path indices, BVH nodes and triangles -- the index is checked
// against its array; a violation sets kErrBounds in the render's error word
// and the access is skipped.  Without DL_CHECKS the checks compile to
// nothing.
constexpr unsigned kErrBounds = 4u;
#ifdef DL_CHECKS
__device__ __forceinline__ bool in_bounds(bool ok, unsigned int* err) {
    if (!ok) atomicOr(err, kErrBounds);
    return ok;
}
#define DL_IN_BOUNDS(cond, err) in_bounds((cond), (err))
#else
#define DL_IN_BOUNDS(cond, err) true
#endif
constexpr const char* kBoundsMessage = "bounds check failed: a queue, slot, path, node or triangle index "
                                        "outside its array (bounds-checked build)";
__device__ __forceinline__ bool slot_ok(const RenderParams& P, int slot) {
    return DL_IN_BOUNDS(slot >= 0 && slot < P.capacity, &P.cnt->err);
}

// Request of batch path `pid`: the last request whose first path is <= pid.
__device__ __forceinline__ int find_request(const RenderParams& P, unsigned long long pid) {
    int lo = 0, hi = P.num_reqs;
    while (hi - lo > 1) {
        int mid = (lo + hi) >> 1;
        if (P.reqs[mid].pid_first <= pid) lo = mid; else hi = mid;
    }
    return lo;
}

// ------------------------------------------------------------ warp helpers
__device__ __forceinline__ int lane_id() { return threadIdx.x & 31; }

// All 32 lanes call this with their predicate; returns the lane's slot in the
// queue (or -1).  One atomic per warp.
__device__ __forceinline__ int warp_push(int* counter, bool pred) {
    unsigned mask = __ballot_sync(0xffffffffu, pred);
    if (mask == 0) return -1;
    int leader = __ffs(mask) - 1;
    int base = 0;
    if (lane_id() == leader) base = atomicAdd(counter, __popc(mask));
    base = __shfl_sync(0xffffffffu, base, leader);
    return pred ? base + __popc(mask & ((1u << lane_id()) - 1u)) : -1;
}
__device__ __forceinline__ unsigned long long warp_claim(unsigned long long* counter, bool pred) {
    unsigned mask = __ballot_sync(0xffffffffu, pred);
    if (mask == 0) return ~0ull;
    int leader = __ffs(mask) - 1;
    unsigned long long base = 0;
    if (lane_id() == leader) base = atomicAdd(counter, (unsigned long long)__popc(mask));
    base = __shfl_sync(0xffffffffu, base, leader);
    return pred ? base + (unsigned long long)__popc(mask & ((1u << lane_id()) - 1u)) : ~0ull;
}

__device__ __forceinline__ unsigned long long warp_claim_u32(unsigned int* counter, bool pred) {
    unsigned mask = __ballot_sync(0xffffffffu, pred);
    if (mask == 0) return ~0ull;
    int leader = __ffs(mask) - 1;
    unsigned base = 0;
    if (lane_id() == leader) base = atomicAdd(counter, (unsigned)__popc(mask));
    base = __shfl_sync(0xffffffffu, base, leader);
    return pred ? (unsigned long long)base + __popc(mask & ((1u << lane_id()) - 1u)) : ~0ull;
}

__device__ __forceinline__ Pcg32 load_rng(const uint4& r) {
    Pcg32 g;
    g.state = ((uint64_t)r.y << 32) | r.x;
    g.inc = ((uint64_t)r.w << 32) | r.z;
    return g;
}
__device__ __forceinline__ uint4 store_rng(const Pcg32& g) {
    return make_uint4((uint32_t)g.state, (uint32_t)(g.state >> 32), (uint32_t)g.inc, (uint32_t)(g.inc >> 32));
}
__device__ __forceinline__ unsigned long long path_index(const int4& m) {
    return (unsigned long long)(unsigned)m.z | ((unsigned long long)(unsigned)m.w << 32);
}

// A path between two vertices.
struct PathState {
    float3 tp;              // throughput
    float eta;
    float3 L;               // radiance gathered so far
    float prev_pdf;         // pdf of the last BSDF sample
    Pcg32 g;
    int depth;
    int flags;              // request index << kReqShift | PathFlags
    unsigned long long pid;
};

// Path `pid` of request `rid`: camera sample (film position `ps`) and ray
// (cpu_renderer.cpp:36-44).  kPass: a single render's first sample index is
// among the pass values on the device (the wavefront's captured graph), else
// in the request.
template <bool kMulti, bool kPass>
__device__ __forceinline__ void camera_path(const RenderParams& P, unsigned long long pid, int rid, PathState& S,
                                            float2& ps, float3& o, float3& d, float& tmax) {
    const DevRequest& R = request<kMulti>(P, rid);
    const DevCamera& cam = R.sc.cam;
    int x, y, s;
    if (P.mode == 1) {
        x = P.xys[3 * pid];
        y = P.xys[3 * pid + 1];
        s = P.xys[3 * pid + 2];
    } else {
        unsigned long long local = pid - R.pid_first;
        unsigned long long npix = (unsigned long long)cam.w * cam.h;
        if ((local | npix) < 0x100000000ull) {  // 32-bit division where it fits
            const unsigned l32 = (unsigned)local, n32 = (unsigned)npix, pix = l32 % n32;
            s = (int)(l32 / n32);
            x = (int)(pix % (unsigned)cam.w);
            y = (int)(pix / (unsigned)cam.w);
        } else {
            unsigned long long pix = local % npix;
            s = (int)(local / npix);
            x = (int)(pix % cam.w);
            y = (int)(pix / cam.w);
        }
        s += kMulti || !kPass ? R.spp_offset : P.cnt->pass_spp_offset;
    }
    seed_path(S.g, R.seed_mix, cam.w, cam.h, x, y, s);
    ps = S.g.next2d();
    ps.x = __fadd_rn((float)x, ps.x);
    ps.y = __fadd_rn((float)y, ps.y);
    (void)S.g.next2d();  // aperture sample: drawn, unused by the "virtual" camera
    camera_ray(cam, ps, o, d, tmax);
    S.tp = f3(1.f, 1.f, 1.f);
    S.eta = 1.f;
    S.L = f3(0.f, 0.f, 0.f);
    S.prev_pdf = 0.f;
    S.depth = 0;
    S.flags = PF_CAMERA | (rid << kReqShift);
    S.pid = pid;
}

// Start path `pid` in `slot`.  Ray records carry the request index in o.w
// (every render ray starts at tmin = kRayEps).  The path record of a camera
// ray (PF_CAMERA) is not written: throughput 1, no radiance yet.
template <bool kMulti>
__device__ void start_path(const RenderParams& P, int slot, unsigned long long pid) {
    if (!slot_ok(P, slot) || !DL_IN_BOUNDS(pid < P.cnt->pass_total, &P.cnt->err)) return;
    const int rid = kMulti ? find_request(P, pid) : 0;
    PathState S;
    float2 ps;
    float3 o, d;
    float tmax;
    camera_path<kMulti, true>(P, pid, rid, S, ps, o, d, tmax);
    RayRec r;
    r.o = make_float4(o.x, o.y, o.z, __int_as_float(rid));
    r.d = make_float4(d.x, d.y, d.z, tmax);
    P.rec[slot].ray = r;
    MetaRec mr;
    mr.m = make_int4(S.depth, S.flags, (int)(pid & 0xffffffffu), (int)(pid >> 32));
    mr.rng = store_rng(S.g);
    P.rec[slot].meta = mr;
    if (P.mode == 1) P.pos[slot] = ps;
    if (P.guided) {
        GuideRec gr;
        gr.a = make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
        gr.b = gr.a;
        P.grec[slot] = gr;
    }
}

// The path record of a camera ray.
__device__ __forceinline__ PathRec camera_record() {
    PathRec r;
    r.tp = make_float4(1.f, 1.f, 1.f, 1.f);
    r.L = make_float4(0.f, 0.f, 0.f, 0.f);
    return r;
}

// Radiance of ended path `pid` (slot `slot`): into the sample buffer at its
// path index (the film kernel gathers it), or as its Li.
__device__ __forceinline__ void store_sample(const RenderParams& P, unsigned long long pid, float3 L, int slot) {
    if (!slot_ok(P, slot) || !DL_IN_BOUNDS(pid < P.cnt->pass_total, &P.cnt->err)) return;
    if (P.mode == 1) {
        P.li_L[3 * pid] = L.x;
        P.li_L[3 * pid + 1] = L.y;
        P.li_L[3 * pid + 2] = L.z;
        float2 ps = P.pos[slot];
        P.li_pos[2 * pid] = ps.x;
        P.li_pos[2 * pid + 1] = ps.y;
    } else {
        P.samples[pid] = make_float4(L.x, L.y, L.z, 1.f);
    }
}

// A shadow ray of an ended path was unoccluded: add its contribution to the
// stored sample.  One shadow ray per path at a time, so no atomics.
__device__ __forceinline__ void add_to_sample(const RenderParams& P, unsigned long long pid, float4 c) {
    if (!DL_IN_BOUNDS(pid < P.cnt->pass_total, &P.cnt->err)) return;
    if (P.mode == 1) {
        P.li_L[3 * pid] = __fadd_rn(P.li_L[3 * pid], c.x);
        P.li_L[3 * pid + 1] = __fadd_rn(P.li_L[3 * pid + 1], c.y);
        P.li_L[3 * pid + 2] = __fadd_rn(P.li_L[3 * pid + 2], c.z);
    } else {
        float4 s = P.samples[pid];
        P.samples[pid] = make_float4(__fadd_rn(s.x, c.x), __fadd_rn(s.y, c.y), __fadd_rn(s.z, c.z), s.w);
    }
}

// Radiance `c` reached the path: credit it to the training records of its
// guided vertices (the newer one too if `both`), divided by the throughput
// after each vertex (mean over the channels it is non-zero in).
__device__ __forceinline__ void credit_one(const RenderParams& P, float4 t, float3 c) {
    int idx = __float_as_int(t.w);
    if (idx < 0) return;
    float s = 0.f;
    int k = 0;
    if (t.x > 0.f) { s += c.x / t.x; k++; }
    if (t.y > 0.f) { s += c.y / t.y; k++; }
    if (t.z > 0.f) { s += c.z / t.z; k++; }
    if (k > 0 && isfinite(s)) static_cast<GuideRecord*>(P.cnt->pass_recs)[idx].L += s / (float)k;
}
__device__ __forceinline__ void credit(const RenderParams& P, const GuideRec& gr, float3 c, bool both) {
    credit_one(P, gr.a, c);
    if (both) credit_one(P, gr.b, c);
}

// Claim new path indices for the lanes in `want`, start them; returns true
// for lanes that now hold a fresh camera ray.
template <bool kMulti>
__device__ __forceinline__ bool regenerate(const RenderParams& P, int slot, bool want) {
    unsigned long long pid = warp_claim(&P.cnt->next_path, want);
    bool ok = want && pid < P.cnt->pass_total;
    if (ok) start_path<kMulti>(P, slot, pid);
    return ok;
}

struct HitInfo {
    float3 p;
    Frame sh;
    int mesh;
};

__device__ __forceinline__ HitInfo hit_info(const DevScene& sc, int tri, float u, float v) {
    HitInfo h;
    const float4* tp = sc.tris + 3 * tri;
    float3 p0 = xyz(__ldg(tp)), p1 = xyz(__ldg(tp + 1)), p2 = xyz(__ldg(tp + 2));
    float b0 = __fsub_rn(__fsub_rn(1.f, u), v);
    h.p = add(add(scale(p0, b0), scale(p1, u)), scale(p2, v));
    int4 vi = __ldg(sc.tri_vidx + tri);
    h.mesh = vi.w;
    if (sc.meshes[vi.w].has_normals) {
        float3 n0 = xyz(__ldg(sc.normals + vi.x)), n1 = xyz(__ldg(sc.normals + vi.y));
        float3 n2 = normalize(xyz(__ldg(sc.normals + vi.z)));
        // only the third term normalised (src/tracer/accel/octree.cpp:202-206)
        h.sh = make_frame(add(add(scale(n0, b0), scale(n1, u)), scale(n2, v)));
    } else {
        h.sh = make_frame(normalize(cross(sub(p1, p0), sub(p2, p0))));
    }
    return h;
}

// Mesh::samplePosition over an area light's triangles (mesh.cpp:222-244,
// DiscretePDF::sampleReuse dpdf.h:131-136).
__device__ __forceinline__ void sample_area(const DevScene& sc, const DevLight& L, float2 s, float3& p,
                                            float3& n) {
    const float* cdf = sc.emit_cdf + L.cdf_begin;
    int cnt = L.tri_count;
    // lower_bound over cdf[0..cnt]
    int lo = 0, hi = cnt + 1;
    while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (__ldg(cdf + mid) < s.x) lo = mid + 1; else hi = mid;
    }
    int f = max(lo - 1, 0);
    f = min(f, cnt - 1);
    float c0 = __ldg(cdf + f), c1 = __ldg(cdf + f + 1);
    s.x = __fdiv_rn(__fsub_rn(s.x, c0), __fsub_rn(c1, c0));
    const float4* et = sc.emit_tris + 6 * (L.tri_begin + f);
    float3 p0 = xyz(__ldg(et)), p1 = xyz(__ldg(et + 1)), p2 = xyz(__ldg(et + 2));
    float3 b = square_to_uniform_triangle(s);
    p = add(add(scale(p0, b.x), scale(p1, b.y)), scale(p2, b.z));
    if (L.has_normals) {
        float3 n0 = xyz(__ldg(et + 3)), n1 = xyz(__ldg(et + 4)), n2 = xyz(__ldg(et + 5));
        n = add(add(scale(n0, b.x), scale(n1, b.y)), scale(n2, b.z));
    } else {
        n = cross(sub(p1, p0), sub(p2, p1));
    }
    n = normalize(n);
}

// The emitter that the NEE sample's first number picks, that number rescaled
// to [0, 1) for reuse: uniformly (scene.cpp:148-163), or, with
// DL_RENDER_POWER_LIGHT_PICK, through the power alias table (slot from the
// number, alias coin from its fraction).
__device__ __forceinline__ int pick_light(const DevRequest& R, float& sx) {
    const DevScene& sc = R.sc;
    const int N = sc.num_lights;
    if (!(R.flags & DL_RENDER_POWER_LIGHT_PICK)) {
        if (N <= 1) return 0;
        int idx = min((int)__fmul_rn(sx, (float)N), N - 1);
        sx = __fsub_rn(__fmul_rn(sx, (float)N), (float)idx);
        return idx;
    }
    float u = __fmul_rn(sx, (float)N);
    int i = min((int)u, N - 1);
    float coin = fminf(__fsub_rn(u, (float)i), 0.99999994f);
    float4 a = __ldg(sc.light_pick + i);
    if (coin < a.x) {
        sx = __fdiv_rn(coin, a.x);
        return i;
    }
    sx = __fdiv_rn(__fsub_rn(coin, a.x), __fsub_rn(1.f, a.x));
    return __float_as_int(a.y);
}

// pdf of direction sample `pdf` of emitter `l` times its pick probability
// (pdfEmitterDirection, scene.cpp:171-179).
__device__ __forceinline__ float with_pick_pdf(const DevRequest& R, int l, float pdf) {
    if (R.flags & DL_RENDER_POWER_LIGHT_PICK) return __fmul_rn(pdf, __ldg(R.sc.light_pick + l).z);
    return R.sc.num_lights != 1 ? __fdiv_rn(pdf, (float)R.sc.num_lights) : pdf;
}

// Three fresh numbers for an envmap NEE sample, drawn after the NEE 2D sample.
__device__ __forceinline__ float3 env_xi(Pcg32& g) {
    float3 xi;
    xi.x = g.next_float();
    xi.y = g.next_float();
    xi.z = g.next_float();
    return xi;
}

// Scene::sampleEmitterDirection without the visibility test (the caller
// traces the shadow ray).  Returns the unoccluded spectrum.  An envmap pick
// draws three more numbers from `g`.
__device__ __forceinline__ float3 sample_emitter(const DevRequest& R, float3 its_p, float3 sh_n, float2 s,
                                                 Pcg32& g, float3& d, float& dist, float& pdf, bool& delta) {
    const DevScene& sc = R.sc;
    int N = sc.num_lights;
    float3 zero = f3(0.f, 0.f, 0.f);
    delta = false;
    pdf = 0.f;
    dist = 0.f;
    d = zero;
    if (N == 0) return zero;
    const int idx = pick_light(R, s.x);
    const DevLight& L = sc.lights[idx];
    float3 spec;
    if (L.type == LIGHT_AREA) {
        float3 lp, ln;
        sample_area(sc, L, s, lp, ln);
        float3 vec = sub(lp, its_p);
        d = normalize(vec);
        dist = length(vec);
        float dp = fmaxf(dot(ln, neg(d)), 0.f);
        float pw = dp != 0.f ? __fdiv_rn(__fmul_rn(__fmul_rn(L.pA, dist), dist), dp) : 0.f;
        pdf = pw;
        spec = pw != 0.f ? divs(scale(ld3(L.radiance), fmaxf(dot(sh_n, d), 0.f)), pw) : zero;
    } else if (L.type == LIGHT_POINT) {
        float3 vec = sub(ld3(L.position), its_p);
        d = normalize(vec);
        dist = length(vec);
        pdf = 1.f;
        delta = true;
        float inv = __fdiv_rn(1.0f, dist);
        if (R.flags & DL_RENDER_FIX_POINT_LIGHT) {
            float c = fmaxf(dot(sh_n, d), 0.f);
            spec = c > 0.f ? scale(scale(scale(ld3(L.radiance), c), inv), inv) : zero;
        } else {
            spec = scale(scale(ld3(L.radiance), inv), inv);
        }
    } else if (L.type == LIGHT_ENVMAP) {
        spec = env_sample(sc, sh_n, env_xi(g), d, pdf);
        dist = 1e16f;  // envmap.h:67
    } else {
        spec = zero;
    }
    if (R.flags & DL_RENDER_POWER_LIGHT_PICK) {
        const float pl = __ldg(sc.light_pick + idx).z;
        spec = divs(spec, pl);
        pdf = __fmul_rn(pdf, pl);
    } else if (N > 1) {
        spec = scale(spec, (float)N);
        pdf = __fmul_rn(pdf, __fdiv_rn(1.f, (float)N));
    }
    return spec;
}

// traversal state: ray finished (below every leaf reference: scenes hold
// fewer than 2^27 triangles)
constexpr int kDone = INT_MIN;

// The envmap's radiance along a ray that hit nothing (miss.cu:11-49): camera
// rays see it if "visual", else the background colour; later rays weight it
// by MIS against the BSDF pdf after a diffuse bounce (`on_light` gets that
// contribution).  Only for scenes with an envmap, and not for the normals
// integrator, which returns 0 on a miss (normal.cpp:13-14).
template <typename F>
__device__ __forceinline__ void add_miss(const DevRequest& R, float3 dir, PathState& S, F&& on_light) {
    const DevScene& sc = R.sc;
    if (S.flags & PF_CAMERA) {
        S.L = add(S.L, sc.env_visual ? env_lookup_dir(sc, dir) : ld3(sc.env_bg));
        return;
    }
    float3 le = env_lookup_dir(sc, dir);
    float w = 1.f;
    if (S.flags & PF_PREV_DIFFUSE) {
        float ep = env_pdf(sc, dir);
        ep = with_pick_pdf(R, sc.env_light, ep);
        w = mis_weight(S.prev_pdf, ep);
    }
    float3 c = mul(scale(S.tp, w), le);
    S.L = add(S.L, c);
    on_light(c);
}

// The BSDF functions of device.cuh for material type T, or for `type` where
// T is kAnyType (one copy of the code around them serves every type; `type`
// is the same for all lanes of a warp).
constexpr int kAnyType = -1;
template <int T>
__device__ __forceinline__ float3 eval_of(int type, const DevMaterial& m, const BRec& r) {
    if (T != kAnyType) return bsdf_eval<T>(m, r);
    switch (type) {
        case MAT_DIFFUSE: return bsdf_eval<MAT_DIFFUSE>(m, r);
        case MAT_MICROFACET: return bsdf_eval<MAT_MICROFACET>(m, r);
        case MAT_ANISO_GGX: return bsdf_eval<MAT_ANISO_GGX>(m, r);
        default: return f3(0.f, 0.f, 0.f);
    }
}
template <int T>
__device__ __forceinline__ float pdf_of(int type, const DevMaterial& m, const BRec& r) {
    if (T != kAnyType) return bsdf_pdf<T>(m, r);
    switch (type) {
        case MAT_DIFFUSE: return bsdf_pdf<MAT_DIFFUSE>(m, r);
        case MAT_MICROFACET: return bsdf_pdf<MAT_MICROFACET>(m, r);
        case MAT_ANISO_GGX: return bsdf_pdf<MAT_ANISO_GGX>(m, r);
        default: return 0.f;
    }
}
template <int T>
__device__ __forceinline__ float3 sample_of(int type, const DevMaterial& m, BRec& r, float2 s, float lobe) {
    if (T != kAnyType) return bsdf_sample<T>(m, r, s, lobe);
    switch (type) {
        case MAT_DIFFUSE: return bsdf_sample<MAT_DIFFUSE>(m, r, s, lobe);
        case MAT_MIRROR: return bsdf_sample<MAT_MIRROR>(m, r, s, lobe);
        case MAT_DIELECTRIC: return bsdf_sample<MAT_DIELECTRIC>(m, r, s, lobe);
        case MAT_MICROFACET: return bsdf_sample<MAT_MICROFACET>(m, r, s, lobe);
        default: return bsdf_sample<MAT_ANISO_GGX>(m, r, s, lobe);
    }
}

// A path's arrival at a hit (triangle `tri`, barycentrics u, v; ray from
// `ray_o` along `dir`) on a material of type T (kAnyType: `type`): emitter hit + MIS
// (path.cpp:72-84) or first-hit emission (27-29), Russian roulette (89-97)
// and the depth limit.  Returns whether the path ends here.  `on_light` gets
// the radiance an emitter hit adds after the first vertex.
template <int T, typename F>
__device__ __forceinline__ bool enter_vertex(const DevRequest& R, int type, int tri, float u, float v, float3 ray_o, float3 dir,
                                             PathState& S, HitInfo& h, float2& tuv, float3& s_tan, F&& on_light) {
    const int Y = T == kAnyType ? type : T;
    const DevScene& sc = R.sc;
    bool done = false;
    h = hit_info(sc, tri, u, v);
    if (Y == MAT_DIFFUSE || Y == MAT_ANISO_GGX) {
        const DevMaterial& mt = sc.materials[sc.meshes[h.mesh].material];
        if (mt.has_tex) {
            tuv = hit_texcoord(sc, tri, u, v);
            // world-space normal / tangent maps (shader_common.h:62-64,
            // 104-107): normalize(2 rgb - 1) replaces the shading normal
            if (Y == MAT_ANISO_GGX && mt.tex[TEX_NORMAL] >= 0) {
                const float3 c = tex_lookup(sc, mt.tex[TEX_NORMAL], tuv);
                h.sh.n = normalize(f3(__fsub_rn(__fmul_rn(c.x, 2.f), 1.f), __fsub_rn(__fmul_rn(c.y, 2.f), 1.f),
                                      __fsub_rn(__fmul_rn(c.z, 2.f), 1.f)));
            }
            if (Y == MAT_ANISO_GGX && mt.tex[TEX_TANGENT] >= 0) {
                const float3 c = tex_lookup(sc, mt.tex[TEX_TANGENT], tuv);
                s_tan = normalize(f3(__fsub_rn(__fmul_rn(c.x, 2.f), 1.f), __fsub_rn(__fmul_rn(c.y, 2.f), 1.f),
                                     __fsub_rn(__fmul_rn(c.z, 2.f), 1.f)));
            }
        }
    }
    int light = sc.meshes[h.mesh].light;
    if (R.flags & DL_RENDER_NORMALS) {
        // the normals integrator (normal.cpp:10-20): |shading normal|
        // of the first hit, and the path ends
        S.L = f3(fabsf(h.sh.n.x), fabsf(h.sh.n.y), fabsf(h.sh.n.z));
        done = true;
    } else if (S.flags & PF_CAMERA) {
        if (light >= 0 && dot(h.sh.n, neg(dir)) > 0.f) S.L = add(S.L, mul(S.tp, ld3(sc.lights[light].radiance)));
        S.depth = 0;
    } else {
        if (light >= 0) {
            const DevLight& Lt = sc.lights[light];
            float3 le = dot(h.sh.n, neg(dir)) > 0.f ? ld3(Lt.radiance) : f3(0.f, 0.f, 0.f);
            float3 vec = sub(h.p, ray_o);
            float3 dd = normalize(vec);
            float dist = length(vec);
            float dp = fmaxf(dot(h.sh.n, neg(dd)), 0.f);
            float ep = dp != 0.f ? __fdiv_rn(__fmul_rn(__fmul_rn(Lt.pA, dist), dist), dp) : 0.f;
            ep = with_pick_pdf(R, light, ep);
            float w = (S.flags & PF_PREV_DIFFUSE) ? mis_weight(S.prev_pdf, ep) : 1.f;
            float3 c = mul(scale(S.tp, w), le);
            S.L = add(S.L, c);
            on_light(c);
        }
        if (S.depth > R.rr_depth) {
            float pq = fminf(maxc(scale(scale(S.tp, S.eta), S.eta)), 0.99f);
            if (S.g.next_float() > pq) done = true;
            else S.tp = divs(S.tp, pq);
        }
        S.depth += 1;
    }
    return done || (R.max_depth > 0 && S.depth >= R.max_depth);
}

// What a vertex sends out: the next-event estimate of its light sample (a
// shadow ray along `ld` over `ldist`, if `emit`) and the next direction.
struct Scatter {
    bool emit;
    float3 c, ld;      // contribution of the light sample, its direction
    float ldist;
    float3 nd;         // next direction
};

// Next-event estimation (path.cpp:36-56) and BSDF sampling (60-69) at a hit
// on a material of type T (kAnyType: `type`).  Mirror and dielectric still draw the NEE sample
// (their eval and pdf are zero: no contribution, no shadow ray).  kGuided,
// `use_guide`: the next direction by one-sample MIS between the decoded lobes
// at `lob` (probability `alpha`) and the BSDF, NEE weighted by the combined
// pdf.  Returns whether the path ends (every later contribution is zero).
template <int T, bool kGuided>
__device__ __forceinline__ bool scatter_vertex(const DevRequest& R, int type, int rid, const HitInfo& h, float3 dir, float2 tuv,
                                               float3 s_tan, bool use_guide, const float* lob, float alpha,
                                               PathState& S, Scatter& out) {
    const int Y = T == kAnyType ? type : T;
    const DevScene& sc = R.sc;
    DevMaterial m = sc.materials[sc.meshes[h.mesh].material];
    if ((Y == MAT_DIFFUSE || Y == MAT_ANISO_GGX) && m.has_tex) {
        // texture lookups replace the constants (diffuse.cu:15-20,
        // aniso_ggx.cu:19-35)
        if (m.tex[TEX_ALBEDO] >= 0) {
            const float3 a = tex_lookup(sc, m.tex[TEX_ALBEDO], tuv);
            m.albedo[0] = a.x;
            m.albedo[1] = a.y;
            m.albedo[2] = a.z;
        }
        if (Y == MAT_ANISO_GGX && m.tex[TEX_SPECULAR] >= 0) {
            const float3 a = tex_lookup(sc, m.tex[TEX_SPECULAR], tuv);
            m.specular[0] = a.x;
            m.specular[1] = a.y;
            m.specular[2] = a.z;
        }
        if (Y == MAT_ANISO_GGX && m.tex[TEX_ALPHA] >= 0) {
            const float3 a = tex_lookup(sc, m.tex[TEX_ALPHA], tuv);
            m.ax = a.x;
            m.ay = a.y;
        }
    }
    Frame fr = Y == MAT_ANISO_GGX ? make_onb_t(normalize(h.sh.n), s_tan) : h.sh;
    float3 wi = to_local(fr, neg(normalize(dir)));
    if (Y == MAT_ANISO_GGX) wi = normalize(wi);
    float2 s_nee = S.g.next2d();
    out.emit = false;
    out.c = f3(0.f, 0.f, 0.f);
    out.ld = out.c;
    out.ldist = 0.f;
    if (Y == MAT_MIRROR || Y == MAT_DIELECTRIC) {
        // no NEE contribution, but an envmap pick still draws its numbers
        float sx = s_nee.x;
        if (sc.env_light >= 0 && sc.num_lights > 0 && pick_light(R, sx) == sc.env_light) (void)env_xi(S.g);
    } else {
        float lpdf;
        bool delta;
        float3 espec = sample_emitter(R, h.p, h.sh.n, s_nee, S.g, out.ld, out.ldist, lpdf, delta);
        if (__fadd_rn(__fadd_rn(espec.x, espec.y), espec.z) > 0.f && lpdf > 0.f) {
            BRec q1;
            q1.wi = wi;
            q1.wo = to_local(fr, out.ld);
            q1.measure = M_SOLID;
            q1.eta = 1.f;
            float3 bv = eval_of<T>(Y, m, q1);
            float bp = pdf_of<T>(Y, m, q1);
            if (kGuided && use_guide) bp = alpha * stored_mixture_pdf(lob, out.ld) + (1.f - alpha) * bp;
            float w = (delta && (R.flags & DL_RENDER_FIX_POINT_LIGHT)) ? 1.f : mis_weight(lpdf, bp);
            out.c = mul(mul(scale(S.tp, w), bv), espec);
            out.emit = out.c.x != 0.f || out.c.y != 0.f || out.c.z != 0.f;
        }
    }
    BRec q2;
    q2.wi = wi;
    q2.wo = f3(0.f, 0.f, 0.f);
    q2.eta = 1.f;
    q2.measure = M_UNKNOWN;
    if (kGuided && use_guide) {
        // one-sample MIS between the learned mixture and the BSDF
        float3 fcos_over_p;
        if (S.g.next_float() < alpha) {
            float u0 = S.g.next_float();
            out.nd = stored_mixture_sample(lob, u0, S.g.next2d());
            q2.wo = to_local(fr, out.nd);
            q2.measure = M_SOLID;
            float3 fv = eval_of<T>(Y, m, q2);
            float pb = pdf_of<T>(Y, m, q2);
            S.prev_pdf = alpha * stored_mixture_pdf(lob, out.nd) + (1.f - alpha) * pb;
            fcos_over_p = S.prev_pdf > 0.f ? scale(fv, fmaxf(q2.wo.z, 0.f) / S.prev_pdf) : f3(0.f, 0.f, 0.f);
        } else {
            const float2 s2 = S.g.next2d();
            const float lobe = Y == MAT_ANISO_GGX ? S.g.next_float() : 0.f;
            float3 wgt = sample_of<T>(Y, m, q2, s2, lobe);
            float pb = pdf_of<T>(Y, m, q2);
            out.nd = to_world(fr, q2.wo);
            if (Y == MAT_ANISO_GGX) out.nd = normalize(out.nd);
            S.prev_pdf = alpha * stored_mixture_pdf(lob, out.nd) + (1.f - alpha) * pb;
            fcos_over_p = S.prev_pdf > 0.f ? scale(wgt, pb / S.prev_pdf) : f3(0.f, 0.f, 0.f);
        }
        S.tp = mul(S.tp, fcos_over_p);
    } else {
        const float2 s2 = S.g.next2d();
        const float lobe = Y == MAT_ANISO_GGX ? S.g.next_float() : 0.f;
        float3 f = sample_of<T>(Y, m, q2, s2, lobe);
        S.tp = mul(S.tp, f);
        S.eta = __fmul_rn(S.eta, q2.eta);
        S.prev_pdf = pdf_of<T>(Y, m, q2);
        out.nd = to_world(fr, q2.wo);
        if (Y == MAT_ANISO_GGX) out.nd = normalize(out.nd);
    }
    S.flags = (rid << kReqShift) | (is_diffuse(Y) ? PF_PREV_DIFFUSE : 0);
    return S.tp.x == 0.f && S.tp.y == 0.f && S.tp.z == 0.f;
}

// Passes of at most kResidentMaxPaths paths run as one launch of the resident
// kernel (resident.cu), the first kResidentFewPaths in its shape for few
// paths.  Above, the wavefront's fuller kernels win on most scenes (device ms,
// resident | wavefront, finished as below: Cornell 1.05 M 1.18 | 1.18, 1.57 M
// 1.70 | 1.57, 2.0 M 2.15 | 1.89; sky 1.0 M 0.86 | 0.82, 1.6 M 1.20 | 1.07;
// textured Cornell 1.0 M 1.37 | 1.42, 1.3 M 1.75 | 1.66, 2.0 M 2.50 | 2.14;
// window-lit room 1.04 M 2.15 | 2.30, 1.56 M 3.10 | 2.86; MIS plates 0.9 M 0.75
// | 0.90, 1.8 M 1.39 | 1.36), later on others (batch scene 1.6 M 1.77 | 1.99,
// 2.0 M 2.20 | 2.32; material spheres 2.1 M 1.31 | 1.58).
constexpr unsigned long long kResidentMaxPaths = 3ull << 19, kResidentFewPaths = 7ull << 15;
constexpr unsigned kErrRounds = 8u;  // error-word bit: the resident kernel gave up (a wait or a path's vertices ran out)

// One pass of P.total paths as one launch on `st`; P.cnt reset before.
void resident_launch(dl_context* ctx, const RenderParams& P, bool multi, cudaStream_t st);

// A wavefront pass whose paths have all been started is finished by the
// resident kernel once at most kTailPaths are left (counted after every graph
// launch, of 8 iterations in the figures): long paths -- through glass, unbounded -- kept hundreds of almost
// empty iterations of 50 us going.  Device ms with the wavefront to the end |
// the rest at 2^14 | 2^17 | 2^20 paths: unbounded sky 1024x768 8 spp 18.4 |
// 5.4 | 5.5 | 5.5, material spheres 800x600 8 spp 13.8 | 6.1 | 5.9 | 5.9,
// reference spheres 640x480 16 spp 17.3 | 4.8 | 4.9 | 4.9, textured box
// 1024x768 8 spp 5.7 | 5.6 | 5.1 | 5.1; depth 12, room 960x540 16 spp 10.9 |
// 10.9 | 10.6 | 10.6.
constexpr int kTailPaths = 1 << 17;
// The `n` paths of extension queue 0 to their ends, as one launch on `st`;
// their shadow rays have been traced.
void resident_finish(dl_context* ctx, const RenderParams& P, int n, bool multi, cudaStream_t st);

}  // namespace dl
