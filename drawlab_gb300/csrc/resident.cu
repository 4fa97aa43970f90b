// A pass of few paths in one launch: the wavefront's path slots and queues
// held in shared memory, block by block.
//
// A wavefront iteration (render.cu) costs 24 us with no path in it and 35-55 us
// with a few -- eight kernels, two joins, the longest search -- and keeps its
// paths in DRAM.
// Here each block owns some hundred slots and takes paths of the pass until
// none are left.  Its warps work through queues in shared memory without
// block-wide barriers: a warp takes 32 hits on one material (or 32 ended
// paths, whose slots start the next camera paths) when a queue holds that
// many; else it traces rays, extension and shadow rays alike, lanes taking
// the next ray as theirs finish; else it takes what there is.  The functions
// that draw, intersect and shade are the wavefront's (path.cuh), every path
// adds its terms in the same order, so images are bit-equal.
//
// What bounds it: the chain of dependent searches and vertices while there
// are fewer paths than threads (about 10 us a vertex; Cornell 256x256 1 spp:
// issue slots 37 % used, 15 of 64 warps), then issue slots (16 spp: 52 %;
// instruction fetch is the largest stall, 3.3-4.0 cycles per issue, since a
// warp runs a vertex alone where the wavefront's kernels run it in step) and
// half-idle warps (14-17 of 32 lanes).  Hence one copy of the vertex code for
// all materials (`type` is the same for all lanes of a warp) and helpers as
// functions: with five inlined copies the code was 285 KB, now 100 KB, and the
// instruction cache misses cost the sky scene 1.6x.
//
// Two shapes.  Few paths: 256 threads with up to 128 registers, no spills:
// the shortest chain.  More: 384 threads at 80 registers, 24 warps an SM (28
// at 72 registers spilled twice as much: Cornell 256x256 16 spp 1.18 ms
// against 1.22, sky 517x389 2 spp 0.53 | 0.55, 400k reference-sphere paths
// 2.30 | 2.45; the batch scene 512x512 4 spp 1.25 | 1.23, the room 480x270 16
// spp 4.00 | 3.98).  Their slots are as many as leave the L1 cache 60 KB of
// the SM's 256 (two blocks in 196 KB of shared memory): with 640 slots it had
// 28 KB, with 480 too few paths are in flight (Cornell 16 spp 1.24 | 1.29
// (640) | 1.30 ms, textured box 333x251 16 spp 1.77 | 1.82 | 1.86).  Up to 256
// paths a block there is a small shape with 256 slots (L1 156 KB): 60k
// reference-sphere paths 1.94 ms against 1.99, batch scene 256x256 1 spp 0.31
// against 0.33; with more paths to take it is slower (Cornell 256x256 4 spp
// 0.47 against 0.42).
// Where the shapes cross (device ms, small | large): Cornell 256x256 2 spp
// 0.25 | 0.26, 3 spp 0.34 | 0.31, 4 spp 0.43 | 0.38; sky 517x389 1 spp 0.39 |
// 0.41; textured box 2 spp 0.41 | 0.42, 3 spp 0.50 | 0.51; batch scene 3 spp
// 0.48 | 0.47, 4 spp 0.55 | 0.53; room 2 spp 0.81 | 0.74.  Against the
// wavefront: Cornell 64x64 1 spp 0.12 | 0.54 (wavefront), 256x256 1 spp 0.20 |
// 0.58, 16 spp 1.18 | 1.39; sky 1 spp 0.39 | 0.94; material spheres 1080p 1
// spp 1.31 | 2.1, 64 spp 66 | 58.
#include <algorithm>

#define DL_SHARED_FN __noinline__
#include "path.cuh"

namespace dl {

constexpr int kResStack = 4;                 // top traversal-stack entries of a thread in shared memory
// Vertices of one path, as many as the wavefront's host loop allows
// iterations: what bounds the kernel's work, whatever the number of paths.
#ifndef DL_MAX_VERTICES   // (tests set a small one)
#define DL_MAX_VERTICES 1000000
#endif
constexpr int kResMaxVertices = DL_MAX_VERTICES;
constexpr int kResMaxSpins = 1 << 22;        // polls of one wait (each about 0.1 us)
constexpr uint32_t kShadowTask = 0x8000u, kFreeEntry = 0x8000u, kNoEntry = 0xffffu;
constexpr int kEndedQueue = kNumMaterialTypes;  // misses, and kFreeEntry | slot for empty slots

// A queue of slots that any warp of the block appends to and takes from.
// `tail` counts the entries announced, `head` the ones taken; an entry is
// kNoEntry until its value has been written, and again once it was read.
// N: at least the entries that can be outstanding.
template <int N>
struct alignas(8) Ring {
    uint32_t head, tail;
    uint16_t entry[N];
};

// A block's paths and queues.  The arrays are indexed by slot (consecutive
// words for consecutive slots: no bank conflicts where a warp holds
// neighbouring slots).
template <int kThreads, int kSlots>
struct ResidentSmem {
    static constexpr int kBlockThreads = kThreads, kBlockSlots = kSlots;
    float o[3][kSlots], d[3][kSlots], tmax[kSlots];        // ray
    float tp[3][kSlots], eta[kSlots], L[3][kSlots], pdf[kSlots];
    uint32_t rng[4][kSlots];
    int depth[kSlots], flags[kSlots];
    uint32_t pid[kSlots];
    float hu[kSlots], hv[kSlots];
    int hit[kSlots];                               // triangle | queue << 27
    int pending[kSlots];                           // rays of the path still to be traced
    float sd[3][kSlots], sdist[kSlots], sc[3][kSlots];     // shadow ray from o, its contribution
    int stack[kResStack][kThreads];
    Ring<2 * kSlots> rays;                         // slot, or kShadowTask | slot
    Ring<kSlots> queue[kNumMaterialTypes + 1];     // hits by material type; ended paths
    int live;                                      // slots in use
    int abort;                                     // a wait ran out: leave
};

__device__ __forceinline__ uint32_t ld_shared(const uint32_t* p) { return *(const volatile uint32_t*)p; }
__device__ __forceinline__ int ld_shared(const int* p) { return *(const volatile int*)p; }
__device__ __forceinline__ void st_shared(int* p, int v) { *(volatile int*)p = v; }

// Waits (bounded) until an entry is (or is not) kNoEntry: the other side has
// announced it and is about to read (write) it.  Returns its value.
__device__ __forceinline__ uint32_t ring_wait(volatile uint16_t* e, bool empty, int* abort, uint32_t& err) {
    uint32_t v = *e;
    for (int k = 0; (v == kNoEntry) != empty; k++) {
        if (k == kResMaxSpins || ld_shared(abort)) {
            err |= kErrRounds;
            st_shared(abort, 1);
            return kNoEntry;
        }
        __nanosleep(20);
        v = *e;
    }
    return v;
}

// `pred` lanes append `v`.  Whatever they wrote to the slot before is visible
// to the lane that takes the entry.
template <int N>
__device__ __forceinline__ void ring_push(Ring<N>& r, bool pred, uint32_t v, int* abort, uint32_t& err) {
    const unsigned mask = __ballot_sync(0xffffffffu, pred);
    if (mask == 0) return;
    uint32_t base = 0;
    __threadfence_block();
    if (lane_id() == __ffs(mask) - 1) base = atomicAdd(&r.tail, (uint32_t)__popc(mask));
    base = __shfl_sync(0xffffffffu, base, __ffs(mask) - 1);
    if (pred) {
        volatile uint16_t* e = &r.entry[(base + __popc(mask & ((1u << lane_id()) - 1u))) % N];
        (void)ring_wait(e, true, abort, err);   // (the entry N pushes ago has been read)
        *e = (uint16_t)v;
    }
}
// The same for one lane of a diverged warp.
template <int N>
__device__ __forceinline__ void ring_push_lane(Ring<N>& r, uint32_t v, int* abort, uint32_t& err) {
    __threadfence_block();
    volatile uint16_t* e = &r.entry[atomicAdd(&r.tail, 1u) % N];
    (void)ring_wait(e, true, abort, err);
    *e = (uint16_t)v;
}
// Whether entries are there to take (all lanes; one load).
template <int N>
__device__ __forceinline__ bool ring_some(const Ring<N>& r) {
    const unsigned long long v = *reinterpret_cast<const volatile unsigned long long*>(&r.head);
    return __any_sync(0xffffffffu, (uint32_t)v != (uint32_t)(v >> 32)) != 0;
}
// Takes up to `want` entries: returns how many, `base` the first (the same in
// all lanes).
template <int N>
__device__ __forceinline__ int ring_claim(Ring<N>& r, int want, uint32_t& base) {
    int n = 0;
    uint32_t h = 0;
    if (lane_id() == 0) {
        h = ld_shared(&r.head);
        for (;;) {  // (ends: each failed exchange is another warp's claim)
            n = max(0, min(want, (int)(ld_shared(&r.tail) - h)));
            if (n == 0) break;
            const uint32_t seen = atomicCAS(&r.head, h, h + (uint32_t)n);
            if (seen == h) break;
            h = seen;
        }
    }
    base = __shfl_sync(0xffffffffu, h, 0);
    return __shfl_sync(0xffffffffu, n, 0);
}
// Entry `at` of a claimed range.  (In the bounds-checked build one that names
// no slot of the block ends the block's work.)
template <class Sm, int N>
__device__ __forceinline__ uint32_t ring_take(const RenderParams& P, Sm& sm, Ring<N>& r, uint32_t at, uint32_t& err) {
    volatile uint16_t* e = &r.entry[at % N];
    const uint32_t v = ring_wait(e, false, &sm.abort, err);
    *e = (uint16_t)kNoEntry;
    __threadfence_block();
    if (!DL_IN_BOUNDS(v == kNoEntry || (int)(v & ~kFreeEntry) < Sm::kBlockSlots, &P.cnt->err)) {
        st_shared(&sm.abort, 1);
        return kNoEntry;
    }
    return v;
}

// Radiance of an ended path into the sample buffer, or as its Li with the
// camera sample's film position (its stream's first 2D draw).
template <bool kMulti>
__device__ __forceinline__ void resident_store(const RenderParams& P, uint32_t pid, float3 L) {
    if (!DL_IN_BOUNDS(pid < P.total, &P.cnt->err)) return;
    if (P.mode == 1) {
        const size_t i = pid;
        P.li_L[3 * i] = L.x;
        P.li_L[3 * i + 1] = L.y;
        P.li_L[3 * i + 2] = L.z;
        const int x = P.xys[3 * i], y = P.xys[3 * i + 1], s = P.xys[3 * i + 2];
        const DevRequest& R = request<kMulti>(P, 0);
        Pcg32 g;
        seed_path(g, R.seed_mix, R.sc.cam.w, R.sc.cam.h, x, y, s);
        const float2 ps = g.next2d();
        P.li_pos[2 * i] = __fadd_rn((float)x, ps.x);
        P.li_pos[2 * i + 1] = __fadd_rn((float)y, ps.y);
    } else {
        P.samples[pid] = make_float4(L.x, L.y, L.z, 1.f);
    }
}

// A ray of the path in `slot` is done: the last one hands the path on to the
// queue of its hit, or ends it.
template <bool kMulti, class Sm>
__device__ __forceinline__ void ray_done(const RenderParams& P, Sm& sm, int slot, uint32_t& err) {
    __threadfence_block();
    if (atomicSub(&sm.pending[slot], 1) != 1) return;
    __threadfence_block();
    if (sm.flags[slot] & PF_ENDED) {
        resident_store<kMulti>(P, sm.pid[slot], f3(sm.L[0][slot], sm.L[1][slot], sm.L[2][slot]));
        ring_push_lane(sm.queue[kEndedQueue], kFreeEntry | (uint32_t)slot, &sm.abort, err);
    } else {
        const int q = sm.hit[slot] >> 27;
        if (DL_IN_BOUNDS(q >= 0 && q <= kEndedQueue, &P.cnt->err))
            ring_push_lane(sm.queue[q], (uint32_t)slot, &sm.abort, err);
        else
            st_shared(&sm.abort, 1);
    }
}

// Rays of the block, closest hits and shadow rays alike, until none are left
// to take: a lane whose ray finishes takes the next one.
template <bool kMulti, class Sm>
__device__ __forceinline__ void resident_trace(const RenderParams& P, Sm& sm, uint32_t& err, unsigned& n_ext,
                                               unsigned& n_shadow) {
    constexpr int kThreads = Sm::kBlockThreads;
    // Few paths: idle lanes look whether there is a ray before they claim one
    // (a claim of nothing cost a lone ray a fifth of its search: 60k
    // reference-sphere paths 1.94 -> 1.87 ms).  With many there mostly is:
    // Cornell 256x256 16 spp 1.225 -> 1.253 ms with the look.
    constexpr bool kLookFirst = kThreads <= 256;
    const int lane = lane_id();
    bool has = false, any = false;
    int slot = 0, node = kDone, sp = 0, hit_tri = -1, hit_mat = 0;
    float3 o = f3(0.f, 0.f, 0.f), d = o;
    float tmax = 0.f, hu = 0.f, hv = 0.f;
    RayBox rb;
    rb.idir = o;
    rb.ood = o;
    int stack[kStackSize - kResStack];
    int* const my_stack = &sm.stack[0][threadIdx.x];
    auto push = [&](int v) {
        if (sp < kResStack) my_stack[sp * kThreads] = v;
        else stack[sp - kResStack] = v;
        sp++;
    };
    auto pop = [&]() -> int {
        --sp;
        return sp < kResStack ? my_stack[sp * kThreads] : stack[sp - kResStack];
    };
    const float4* nodes = P.r0.sc.nodes;
    const float4* tris = P.r0.sc.tris;
    int ntris = P.r0.sc.num_tris;
#ifdef DL_CHECKS
    int nnodes = P.r0.sc.num_nodes;
#endif
    for (;;) {
        const unsigned m = __ballot_sync(0xffffffffu, !has);
        const bool look = m && (!kLookFirst || ring_some(sm.rays));
        if (look) {
            uint32_t base;
            const int n = ring_claim(sm.rays, __popc(m), base);
            const int i = __popc(m & ((1u << lane) - 1u));
            if (!has && i < n) {
                const uint32_t task = ring_take(P, sm, sm.rays, base + i, err);
                if (task != kNoEntry) {
                    any = (task & kShadowTask) != 0;
                    slot = (int)(task & ~kShadowTask);
                    o = f3(sm.o[0][slot], sm.o[1][slot], sm.o[2][slot]);
                    if (any) {
                        d = f3(sm.sd[0][slot], sm.sd[1][slot], sm.sd[2][slot]);
                        tmax = sm.sdist[slot];
                        n_shadow++;
                    } else {
                        d = f3(sm.d[0][slot], sm.d[1][slot], sm.d[2][slot]);
                        tmax = sm.tmax[slot];
                        n_ext++;
                    }
                    if (kMulti) {
                        const DevScene& rs = P.reqs[sm.flags[slot] >> kReqShift].sc;
                        nodes = rs.nodes;
                        tris = rs.tris;
                        ntris = rs.num_tris;
#ifdef DL_CHECKS
                        nnodes = rs.num_nodes;
#endif
                    }
                    rb = make_raybox(o, d);
                    node = ntris > 0 ? 0 : kDone;
                    sp = 0;
                    hit_tri = -1;
                    has = true;
                }
            }
        }
        if ((look || !kLookFirst ? __ballot_sync(0xffffffffu, has) : ~m) == 0) break;
        bool finished = false;
        if (has) {
            while (node >= 0) {
#ifdef DL_CHECKS
                if (!DL_IN_BOUNDS(node < nnodes, &P.cnt->err)) {
                    node = kDone;
                    break;
                }
#endif
                const float4* np = nodes + 4 * node;
                float4 a, b, c, dd;
                ld_nc_256(np, a, b);
                ld_nc_256(np + 2, c, dd);
                const int2 ch = make_int2(__float_as_int(dd.x), __float_as_int(dd.y));
                bool h0, h1;
                float t0, t1;
                box2(rb, kRayEps, tmax, a, b, c, h0, h1, t0, t1);
                if (h0 && h1) {
                    int near = ch.x, far = ch.y;
                    if (t1 < t0) { near = ch.y; far = ch.x; }
#ifdef DL_CHECKS
                    if (sp < kStackSize) push(far); else err |= 1u;
#else
                    push(far);
#endif
                    node = near;
                } else if (h0) {
                    node = ch.x;
                } else if (h1) {
                    node = ch.y;
                } else {
                    node = sp > 0 ? pop() : kDone;
                }
            }
            finished = node == kDone;
            if (!finished) {
                const int ref = ~node;
                int first = ref >> 4, count = (ref & 15) + 1;
                if (!DL_IN_BOUNDS(first >= 0 && first + count <= ntris, &P.cnt->err)) count = 0;
                for (int k = 0; k < count; k++) {
                    const float4* tp = tris + 3 * (first + k);
                    const float4 p0 = __ldg(tp), p1 = __ldg(tp + 1), p2 = __ldg(tp + 2);
                    float t, u, v;
                    if (intersect_tri(xyz(p0), xyz(p1), xyz(p2), o, d, kRayEps, tmax, t, u, v)) {
                        hit_tri = first + k;
                        if (any) break;
                        tmax = t;
                        hu = u;
                        hv = v;
                        hit_mat = __float_as_int(p1.w);
                    }
                }
                if (any && hit_tri >= 0) {
                    finished = true;
                } else {
                    node = sp > 0 ? pop() : kDone;
                    finished = node == kDone;
                }
            }
            if (finished) {
                has = false;
                if (any) {
                    if (hit_tri < 0) {  // unoccluded: add the NEE contribution
                        sm.L[0][slot] = __fadd_rn(sm.L[0][slot], sm.sc[0][slot]);
                        sm.L[1][slot] = __fadd_rn(sm.L[1][slot], sm.sc[1][slot]);
                        sm.L[2][slot] = __fadd_rn(sm.L[2][slot], sm.sc[2][slot]);
                    }
                } else if (hit_tri >= 0) {
                    sm.hu[slot] = hu;
                    sm.hv[slot] = hv;
                    sm.hit[slot] = hit_tri | (hit_mat << 27);
                } else {
                    sm.hit[slot] = kEndedQueue << 27;
                }
                ray_done<kMulti>(P, sm, slot, err);
            }
        }
    }
}

// One vertex of the path in `slot` (lanes with `active`): its hit on a
// material of `type`.  The rays it sends out join the next round's, the slot
// of a path that ends without a shadow ray is free then.
template <bool kMulti, class Sm>
__device__ __forceinline__ void resident_shade(const RenderParams& P, Sm& sm, int type, int slot, bool active,
                                               uint32_t& err) {
    bool done = false, emit = false;
    if (active) {
        PathState S;
        S.tp = f3(sm.tp[0][slot], sm.tp[1][slot], sm.tp[2][slot]);
        S.eta = sm.eta[slot];
        S.L = f3(sm.L[0][slot], sm.L[1][slot], sm.L[2][slot]);
        S.prev_pdf = sm.pdf[slot];
        S.g = load_rng(make_uint4(sm.rng[0][slot], sm.rng[1][slot], sm.rng[2][slot], sm.rng[3][slot]));
        S.depth = sm.depth[slot];
        S.flags = sm.flags[slot];
        S.pid = sm.pid[slot];
        if (S.depth >= kResMaxVertices) {   // give up, all warps of the block
            err |= kErrRounds;
            st_shared(&sm.abort, 1);
        }
        const int rid = S.flags >> kReqShift;
        const DevRequest& R = request<kMulti>(P, rid);
        const float3 dir = f3(sm.d[0][slot], sm.d[1][slot], sm.d[2][slot]);
        const float3 ray_o = f3(sm.o[0][slot], sm.o[1][slot], sm.o[2][slot]);
        int tri = sm.hit[slot] & ((1 << 27) - 1);
        if (!DL_IN_BOUNDS(tri >= 0 && tri < R.sc.num_tris, &P.cnt->err)) tri = 0;
        HitInfo h;
        float2 tuv = make_float2(0.f, 0.f);
        float3 s_tan = f3(0.f, 0.f, 0.f);
        Scatter sc;
        sc.emit = false;
        done = enter_vertex<kAnyType>(R, type, tri, sm.hu[slot], sm.hv[slot], ray_o, dir, S, h, tuv, s_tan, [](float3) {});
        if (!done) done = scatter_vertex<kAnyType, false>(R, type, rid, h, dir, tuv, s_tan, false, nullptr, 0.f, S, sc);
        emit = sc.emit;
        if (done && !emit) {
            resident_store<kMulti>(P, (uint32_t)S.pid, S.L);
        } else {
            sm.L[0][slot] = S.L.x;
            sm.L[1][slot] = S.L.y;
            sm.L[2][slot] = S.L.z;
            sm.o[0][slot] = h.p.x;
            sm.o[1][slot] = h.p.y;
            sm.o[2][slot] = h.p.z;
            sm.flags[slot] = S.flags | (done ? PF_ENDED : 0);
            sm.pending[slot] = (emit ? 1 : 0) + (done ? 0 : 1);
            if (emit) {
                sm.sd[0][slot] = sc.ld.x;
                sm.sd[1][slot] = sc.ld.y;
                sm.sd[2][slot] = sc.ld.z;
                sm.sdist[slot] = __fsub_rn(sc.ldist, kRayEps);
                sm.sc[0][slot] = sc.c.x;
                sm.sc[1][slot] = sc.c.y;
                sm.sc[2][slot] = sc.c.z;
            }
            if (!done) {
                sm.d[0][slot] = sc.nd.x;
                sm.d[1][slot] = sc.nd.y;
                sm.d[2][slot] = sc.nd.z;
                sm.tmax[slot] = __int_as_float(0x7f800000);
                sm.tp[0][slot] = S.tp.x;
                sm.tp[1][slot] = S.tp.y;
                sm.tp[2][slot] = S.tp.z;
                sm.eta[slot] = S.eta;
                sm.pdf[slot] = S.prev_pdf;
                const uint4 r = store_rng(S.g);
                sm.rng[0][slot] = r.x;
                sm.rng[1][slot] = r.y;
                sm.depth[slot] = S.depth;
            }
        }
    }
    ring_push(sm.rays, active && !done, (uint32_t)slot, &sm.abort, err);
    ring_push(sm.rays, emit, kShadowTask | (uint32_t)slot, &sm.abort, err);
    ring_push(sm.queue[kEndedQueue], active && done && !emit, kFreeEntry | (uint32_t)slot, &sm.abort, err);
}

// Misses (the envmap's radiance, the sample stored) and free slots: each
// lane's slot starts the next path of the pass, 32 consecutive ones a warp;
// kTail: it takes the next of the `tail` paths that the wavefront left.
template <bool kMulti, bool kTail, class Sm>
__device__ __forceinline__ void resident_restart(const RenderParams& P, Sm& sm, uint32_t entry, bool active,
                                                 unsigned tail, uint32_t& err) {
    const int slot = (int)(entry & ~kFreeEntry);
    if (active && !(entry & kFreeEntry)) {
        PathState S;
        S.flags = sm.flags[slot];
        S.L = f3(sm.L[0][slot], sm.L[1][slot], sm.L[2][slot]);
        const DevRequest& R = request<kMulti>(P, S.flags >> kReqShift);
        if (R.sc.env_light >= 0 && !(R.flags & DL_RENDER_NORMALS)) {
            S.tp = f3(sm.tp[0][slot], sm.tp[1][slot], sm.tp[2][slot]);
            S.prev_pdf = sm.pdf[slot];
            add_miss(R, f3(sm.d[0][slot], sm.d[1][slot], sm.d[2][slot]), S, [](float3) {});
        }
        resident_store<kMulti>(P, sm.pid[slot], S.L);
    }
    const unsigned long long pid = kTail ? warp_claim_u32(&P.cnt->tail_next, active) : warp_claim(&P.cnt->next_path, active);
    bool start = active && pid < (kTail ? tail : P.total);
    if (kTail && start) {
        const int from = DL_IN_BOUNDS(pid < (unsigned)P.capacity, &P.cnt->err) ? P.ext_q[0][pid] : -1;
        if (from >= 0 && slot_ok(P, from)) {
            const RayRec r = P.rec[from].ray;
            const MetaRec mr = P.rec[from].meta;
            const PathRec pr = mr.m.y & PF_CAMERA ? camera_record() : P.rec[from].path;
            sm.o[0][slot] = r.o.x;
            sm.o[1][slot] = r.o.y;
            sm.o[2][slot] = r.o.z;
            sm.d[0][slot] = r.d.x;
            sm.d[1][slot] = r.d.y;
            sm.d[2][slot] = r.d.z;
            sm.tmax[slot] = r.d.w;
            sm.tp[0][slot] = pr.tp.x;
            sm.tp[1][slot] = pr.tp.y;
            sm.tp[2][slot] = pr.tp.z;
            sm.eta[slot] = pr.tp.w;
            sm.L[0][slot] = pr.L.x;
            sm.L[1][slot] = pr.L.y;
            sm.L[2][slot] = pr.L.z;
            sm.pdf[slot] = pr.L.w;
            sm.rng[0][slot] = mr.rng.x;
            sm.rng[1][slot] = mr.rng.y;
            sm.rng[2][slot] = mr.rng.z;
            sm.rng[3][slot] = mr.rng.w;
            sm.depth[slot] = mr.m.x;
            sm.flags[slot] = mr.m.y;
            sm.pid[slot] = (uint32_t)mr.m.z;
            sm.pending[slot] = 1;
        } else {
            start = false;
        }
    } else if (start) {
        const int rid = kMulti ? find_request(P, pid) : 0;
        PathState S;
        float2 ps;
        float3 o, d;
        float tmax;
        camera_path<kMulti, false>(P, pid, rid, S, ps, o, d, tmax);
        sm.o[0][slot] = o.x;
        sm.o[1][slot] = o.y;
        sm.o[2][slot] = o.z;
        sm.d[0][slot] = d.x;
        sm.d[1][slot] = d.y;
        sm.d[2][slot] = d.z;
        sm.tmax[slot] = tmax;
        for (int k = 0; k < 3; k++) {
            sm.tp[k][slot] = 1.f;
            sm.L[k][slot] = 0.f;
        }
        sm.eta[slot] = 1.f;
        sm.pdf[slot] = 0.f;
        const uint4 r = store_rng(S.g);
        sm.rng[0][slot] = r.x;
        sm.rng[1][slot] = r.y;
        sm.rng[2][slot] = r.z;
        sm.rng[3][slot] = r.w;
        sm.depth[slot] = 0;
        sm.flags[slot] = S.flags;
        sm.pid[slot] = (uint32_t)S.pid;
        sm.pending[slot] = 1;
    }
    ring_push(sm.rays, start, (uint32_t)slot, &sm.abort, err);
    const int lost = __popc(__ballot_sync(0xffffffffu, active && !start));
    if (lost && lane_id() == 0) atomicSub(&sm.live, lost);
}

// `slots`: path slots each block uses (a multiple of 32, at most kSlots).
template <bool kMulti, bool kTail, int kThreads, int kSlots, int kBlocks>
__global__ void __launch_bounds__(kThreads, kBlocks) k_resident(RenderParams P, int slots, unsigned tail) {
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    auto& sm = *reinterpret_cast<ResidentSmem<kThreads, kSlots>*>(dyn_smem);
    const int lane = lane_id();
    // at first every slot is free
    for (int i = threadIdx.x; i < 2 * kSlots; i += kThreads) sm.rays.entry[i] = (uint16_t)kNoEntry;
    for (int t = 0; t <= kNumMaterialTypes; t++)
        for (int i = threadIdx.x; i < kSlots; i += kThreads)
            sm.queue[t].entry[i] = (uint16_t)(t == kEndedQueue && i < slots ? kFreeEntry | i : kNoEntry);
    if (threadIdx.x == 0) {
        sm.rays.head = sm.rays.tail = 0;
        for (int t = 0; t <= kNumMaterialTypes; t++) {
            sm.queue[t].head = 0;
            sm.queue[t].tail = t == kEndedQueue ? slots : 0;
        }
        sm.live = slots;
        sm.abort = 0;
    }
    __syncthreads();
    uint32_t err = 0;
    unsigned n_ext = 0, n_shadow = 0;
    int idle = 0;
    for (;;) {
        // the fullest queue, and the rays
        int most = 0, rays = 0;
        if (lane <= kNumMaterialTypes)
            most = (int)(ld_shared(&sm.queue[lane].tail) - ld_shared(&sm.queue[lane].head)) << 3 | lane;
        else if (lane == 31)
            rays = (int)(ld_shared(&sm.rays.tail) - ld_shared(&sm.rays.head));
        rays = __shfl_sync(0xffffffffu, rays, 31);
        most = __reduce_max_sync(0xffffffffu, most);
        const int best = most & 7;
        most >>= 3;
        if (most < 32 && rays > 0) {
            resident_trace<kMulti>(P, sm, err, n_ext, n_shadow);
            idle = 0;
        } else if (most > 0) {
            uint32_t base;
            const int n = ring_claim(sm.queue[best], 32, base);
            if (n > 0) {
                const uint32_t e = lane < n ? ring_take(P, sm, sm.queue[best], base + lane, err) : kNoEntry;
                const bool active = e != kNoEntry;
                if (best == kEndedQueue) resident_restart<kMulti, kTail>(P, sm, e, active, tail, err);
                else resident_shade<kMulti>(P, sm, best, active ? (int)e : 0, active, err);
                idle = 0;
            }
        } else {
            // nothing to do: the pass has no more paths, or other warps hold
            // them.  A warp may leave: those that hold rays or paths go on by
            // themselves.
            // The warp leaves as one: its lanes may read different counts, as
            // other warps end paths meanwhile.
            if (__any_sync(0xffffffffu, ld_shared(&sm.live) == 0 || ++idle > kResMaxSpins)) break;
            __nanosleep(100);
        }
        if (__any_sync(0xffffffffu, ld_shared(&sm.abort))) break;
    }
    __syncthreads();
    if (sm.live != 0) err |= kErrRounds;  // paths left behind
    n_ext = __reduce_add_sync(0xffffffffu, n_ext);
    n_shadow = __reduce_add_sync(0xffffffffu, n_shadow);
    if (lane == 0) {
        atomicAdd(&P.cnt->stat_ext, (unsigned long long)n_ext);
        atomicAdd(&P.cnt->stat_shadow, (unsigned long long)n_shadow);
    }
    if (err) atomicOr(&P.cnt->err, err);
}

static int resident_sms(const dl_context* ctx) { return ctx->num_sms > 0 ? ctx->num_sms : 152; }

// One shape of the kernel (`index`: 0 .. 3), its blocks per SM found when the
// context first launches it.  kTail: `total` paths that the wavefront left.
template <bool kMulti, bool kTail, int kThreads, int kSlots, int kBlocks>
static void launch_shape(dl_context* ctx, int index, const RenderParams& P, unsigned long long total,
                         cudaStream_t st) {
    auto* fn = k_resident<kMulti, kTail, kThreads, kSlots, kBlocks>;
    constexpr size_t smem = sizeof(ResidentSmem<kThreads, kSlots>);
    static_assert(kSlots % 32 == 0 && kSlots < (int)kFreeEntry && kBlocks * (smem + 1024) <= 228 * 1024, "shared memory");
    int& per_sm = ctx->resident_per_sm[2 * index + (kMulti ? 1 : 0)];
    if (per_sm == 0) {
        DL_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        int n = 0;
        DL_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, fn, kThreads, smem));
        per_sm = std::max(1, n);
    }
    const int64_t blocks = (int64_t)resident_sms(ctx) * per_sm;
    // few paths: spread over all blocks, whole warps of them
    const int64_t share = (int64_t)((total + blocks - 1) / blocks);
    const int slots = (int)std::min<int64_t>(kSlots, (share + 31) / 32 * 32);
    const int grid = (int)std::min<int64_t>(blocks, (int64_t)((total + slots - 1) / slots));
    fn<<<grid, kThreads, smem, st>>>(P, slots, kTail ? (unsigned)total : 0u);
    DL_CUDA(cudaGetLastError());
}

void resident_launch(dl_context* ctx, const RenderParams& P, bool multi, cudaStream_t st) {
    // (the shapes cross at about 0.2 M paths, the slots at 256 a block: see the top)
    if (P.total <= kResidentFewPaths) {
        if (P.total <= 2ull * resident_sms(ctx) * 256) {
            if (multi) launch_shape<true, false, 256, 256, 2>(ctx, 0, P, P.total, st);
            else launch_shape<false, false, 256, 256, 2>(ctx, 0, P, P.total, st);
        } else {
            if (multi) launch_shape<true, false, 256, 576, 2>(ctx, 1, P, P.total, st);
            else launch_shape<false, false, 256, 576, 2>(ctx, 1, P, P.total, st);
        }
    } else {
        if (multi) launch_shape<true, false, 384, 608, 2>(ctx, 2, P, P.total, st);
        else launch_shape<false, false, 384, 608, 2>(ctx, 2, P, P.total, st);
    }
}

void resident_finish(dl_context* ctx, const RenderParams& P, int n, bool multi, cudaStream_t st) {
    if (multi) launch_shape<true, true, 256, 576, 2>(ctx, 3, P, (unsigned long long)n, st);
    else launch_shape<false, true, 256, 576, 2>(ctx, 3, P, (unsigned long long)n, st);
}

}  // namespace dl
