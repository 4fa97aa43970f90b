// Wavefront path tracer (sm_103a).
//
// The reference runs one path per thread/loop iteration (CPU:
// PathIntegrator::Li, src/tracer/integrator/path.cpp:13-100; OptiX:
// __raygen__path, src/optix/cuda/integrator/path.cu:28-97).  Here a fixed
// pool of path slots advances one segment per iteration through:
//
//   extend    persistent closest-hit traversal of queue E[p]; lanes whose ray
//             finishes fetch the next one (per-lane replacement); each hit
//             joins the queue of its material type, misses the miss queue
//   shadow    same, any hit, for last iteration's NEE rays: the contribution
//             goes to the path (or, if the path has ended, to its sample)
//   miss      paths whose ray missed: store the sample, start a new camera
//             path in the slot                                     -> E[q]
//   material  one kernel per BSDF type (diffuse, mirror, dielectric,
//             Beckmann microfacet, GGX): emitter hit + MIS, Russian roulette,
//             NEE (emits a shadow ray), BSDF sampling (emits the next ray);
//             a path that ends stores its sample and its slot starts a new
//             camera path                                          -> E[q], S
//   film      after the last path: gather every sample into the film
//
// Path state lives in 32-byte records (ray, path, meta+rng, hit), each read
// and written whole: a full DRAM sector, no read-modify-write of partial
// sectors.  Queues are compacted with warp ballots: one atomic per warp, or
// per 32 entries where a warp stages them in shared memory; the hot counters
// sit in separate 128-byte lines.  A batch of iterations is captured as a CUDA
// graph, replayed, and updated in place for other frames.  Passes of few paths
// run in one launch instead (resident.cu).  Every path (x, y, s) owns a pcg32
// stream and draws its numbers in the reference's order (pixel 2D, aperture
// 2D, then per bounce NEE 2D, BSDF 2D, RR 1D), so each path reproduces the
// oracle's path of the same (x, y, s).
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <climits>
#include <cmath>
#include <cstring>

#include "device.cuh"
#include "guide.cuh"
#include "guide_tc.cuh"
#include "internal.h"
#include "path.cuh"
#include "scene.h"

namespace dl {

// ---------------------------------------------------------------- kernels
// First camera paths of a pass: slot i starts path i (no claiming needed),
// and the extension queue lists the started slots in order.
template <bool kMulti>
__global__ void k_init(RenderParams P, int capacity) {
    const unsigned long long total = P.cnt->pass_total;
    int n = (int)min((unsigned long long)capacity, total);
    if (!DL_IN_BOUNDS(capacity <= P.capacity, &P.cnt->err)) n = 0;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        P.cnt->next_path = (unsigned long long)n;
        P.cnt->ext[0] = n;
    }
    for (int slot = blockIdx.x * blockDim.x + threadIdx.x; slot < n; slot += gridDim.x * blockDim.x) {
        start_path<kMulti>(P, slot, (unsigned long long)slot);
        P.ext_q[0][slot] = slot;
    }
}

// Persistent traversal over a ray queue.  Each lane holds one ray's
// traversal state (node, stack); a lane whose ray finishes takes the next ray
// of the queue, so lanes do not idle while the warp's longest ray finishes.
// A warp reserves queue entries kFetchChunk at a time (one atomic per chunk)
// and hands them to its lanes as they free up.
//   kAny = false: closest hit of extension rays E[p] (slots) -> hit[slot], and
//                 the slot joins the queue of its hit's material type (or the
//                 miss queue).  Each warp stages those entries per destination
//                 in shared memory and appends them 32 at a time: one atomic
//                 and one coalesced 128-byte store per 32 entries.
//   kAny = true:  any hit of shadow rays S (queue positions); unoccluded ones
//                 add their contribution to the path or the ended path's sample
constexpr unsigned kFetchChunk = 64;
constexpr int kTraverseWarps = 4;  // 128 threads
constexpr int kStage = 64;         // staged entries per warp and destination (flushed at 32)
// Fewer lanes than this in the descent loop leave it for the leaf phase.  On
// the 1080p material-sphere frame (64 spp) 0 / 4 / 6 / 8 / 12 took 59.0 / 57.4 /
// 57.1 / 57.0 / 56.9 ms (extension 29.7 -> 27.9), on the MIS plates (64 spp)
// 31.5 / 31.2 / 31.2 / 31.1 / 31.0, in the window-lit room 11.6 / 11.1 / 11.1 /
// 11.0 / 11.1.  A vote per step for an exact count cost what it gained; a
// quarter of the warp's rays instead of 8 lanes: plates 31.4.
constexpr int kDescendLanes = 8;
constexpr int kSmemStack = 8;      // top traversal-stack entries per thread kept in shared memory

template <bool kCount, bool kAny, bool kMulti>
__global__ void __launch_bounds__(128) k_traverse(RenderParams P, int p) {
    const int q = p ^ 1;
    int n = kAny ? P.cnt->shadow[p] : P.cnt->ext[p];
    if (!DL_IN_BOUNDS(n >= 0 && n <= P.capacity, &P.cnt->err)) n = 0;
    unsigned int* work = kAny ? &P.cnt->work_sh : &P.cnt->work_ext;
    constexpr int kDests = kAny ? 1 : kNumMaterialTypes + 1;
    __shared__ int s_qbuf[kTraverseWarps][kDests][kStage];
    __shared__ int s_qcnt[kTraverseWarps][kDests];
    const int warp = threadIdx.x >> 5, lane = lane_id();
    const unsigned lt = (1u << lane) - 1u;
    if (lane < kDests) s_qcnt[warp][lane] = 0;
    __syncwarp();
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (!kAny) {
            // this iteration's output queues start empty
            P.cnt->ext[q] = 0;
            P.cnt->shadow[q] = 0;
            P.cnt->stat_ext += (unsigned long long)n;
        } else {
            // next iteration's material queues start empty (the extension
            // traversal, which may run concurrently, appends to mat[p])
            for (int k = 0; k <= kNumMaterialTypes; k++) P.cnt->mat[q][k].n = 0;
            P.cnt->stat_shadow += (unsigned long long)n;
        }
    }
    uint32_t err = 0, nn = 0, nt = 0;
    bool has = false, exhausted = false;
    int idx = 0, slot = 0, node = kDone, sp = 0, hit_tri = -1, hit_mat = 0;
    float3 o = f3(0.f, 0.f, 0.f), d = o;
    float tmin = 0.f, tmax = 0.f, ht = 0.f, hu = 0.f, hv = 0.f;
    RayBox rb;
    rb.idir = o;
    rb.ood = o;
    // traversal stack: the first kSmemStack entries in shared memory, laid out
    // [depth][thread] so that lanes at different depths hit different banks;
    // deeper entries in local memory
    __shared__ int s_stack[kSmemStack][kTraverseWarps * 32];
    int stack[kStackSize - kSmemStack];
    int* const my_stack = &s_stack[0][threadIdx.x];
    auto push = [&](int v) {
        if (sp < kSmemStack) my_stack[sp * kTraverseWarps * 32] = v;
        else stack[sp - kSmemStack] = v;
        sp++;
    };
    auto pop = [&]() -> int {
        --sp;
        return sp < kSmemStack ? my_stack[sp * kTraverseWarps * 32] : stack[sp - kSmemStack];
    };
    int rid = 0;  // the ray's request
    const float4* nodes = P.r0.sc.nodes;
    const float4* tris = P.r0.sc.tris;
    int ntris = P.r0.sc.num_tris;
    unsigned c_next = 0, c_end = 0;  // the warp's reserved queue entries [c_next, c_end)
    for (;;) {
        bool need = !has && !exhausted;
        unsigned m = __ballot_sync(0xffffffffu, need);
        if (m) {
            const unsigned k = __popc(m), rank = __popc(m & lt), avail = c_end - c_next;
            unsigned mine;
            if (k > avail) {  // warp-uniform: reserve the next chunk
                unsigned base = 0;
                if (lane == 0) base = atomicAdd(work, kFetchChunk);
                base = __shfl_sync(0xffffffffu, base, 0);
                mine = rank < avail ? c_next + rank : base + (rank - avail);
                c_next = base + (k - avail);
                c_end = base + kFetchChunk;
            } else {
                mine = c_next + rank;
                c_next += k;
            }
            if (need) {
                idx = (int)min(mine, (unsigned)n);
                if (mine < (unsigned)n) {
                    float4 ro = make_float4(0.f, 0.f, 0.f, 0.f), rd = make_float4(0.f, 0.f, 0.f, -1.f);
                    if (kAny) {
                        ro = P.sh_o[idx];
                        rd = P.sh_d[idx];
                    } else {
                        slot = P.ext_q[p][idx];
                        if (slot_ok(P, slot)) {
                            RayRec r = P.rec[slot].ray;
                            ro = r.o;
                            rd = r.d;
                        }
                    }
                    o = xyz(ro);
                    d = xyz(rd);
                    tmin = kRayEps;
                    tmax = rd.w;
                    if (kMulti) {
                        rid = __float_as_int(ro.w);
                        const DevScene& rs = P.reqs[rid].sc;
                        nodes = rs.nodes;
                        tris = rs.tris;
                        ntris = rs.num_tris;
                    }
                    rb = make_raybox(o, d);
                    node = ntris > 0 ? 0 : kDone;
                    sp = 0;
                    hit_tri = -1;
                    has = true;
                } else {
                    exhausted = true;
                }
            }
        }
        const unsigned with = __ballot_sync(0xffffffffu, has);
        if (with == 0) break;
        const int leave = __popc(with) > kDescendLanes ? kDescendLanes : 0;
        bool finished = false;
        int dest = 0;
        if (has) {
            // descend inner nodes until a leaf (or the end of the traversal)
            while (node >= 0) {
#ifdef DL_CHECKS
                const int num_nodes = kMulti ? P.reqs[rid].sc.num_nodes : P.r0.sc.num_nodes;
                if (!DL_IN_BOUNDS(node < num_nodes, &P.cnt->err)) {
                    node = kDone;
                    break;
                }
#endif
                const float4* np = nodes + 4 * node;
                float4 a, b, c, dd;
                ld_nc_256(np, a, b);        // a node is two 32-byte halves
                ld_nc_256(np + 2, c, dd);
                const int2 ch = make_int2(__float_as_int(dd.x), __float_as_int(dd.y));
                if (kCount) nn++;
                bool h0, h1;
                float t0, t1;
                box2(rb, tmin, tmax, a, b, c, h0, h1, t0, t1);
                if (h0 && h1) {   // (both slots always hold a child: see bvh.h)
                    int near = ch.x, far = ch.y;
                    if (t1 < t0) { near = ch.y; far = ch.x; }
#ifdef DL_CHECKS
                    if (sp < kStackSize) push(far); else err |= 1u;
#else
                    push(far);   // depth <= kStackSize + 1: checked when the scene is built
#endif
                    node = near;
                } else if (h0) {
                    node = ch.x;
                } else if (h1) {
                    node = ch.y;
                } else {
                    node = sp > 0 ? pop() : kDone;
                }
                // the last lanes to descend would keep those that wait at a
                // leaf idle: they go on next round
                if (__popc(__activemask()) < leave) break;
            }
            finished = node == kDone;
            if (!finished && node < 0) {
                // leaf: test its triangles (the reference's Moller-Trumbore)
                int ref = ~node;
                int first = ref >> 4, count = (ref & 15) + 1;
                if (!DL_IN_BOUNDS(first >= 0 && first + count <= ntris, &P.cnt->err)) count = 0;
                bool any = false;
                for (int k = 0; k < count; k++) {
                    const float4* tp = tris + 3 * (first + k);
                    float4 p0 = __ldg(tp), p1 = __ldg(tp + 1), p2 = __ldg(tp + 2);
                    if (kCount) nt++;
                    float t, u, v;
                    if (intersect_tri(xyz(p0), xyz(p1), xyz(p2), o, d, tmin, tmax, t, u, v)) {
                        if (kAny) {
                            any = true;
                            break;
                        }
                        tmax = t;
                        ht = t;
                        hu = u;
                        hv = v;
                        hit_tri = first + k;
                        hit_mat = __float_as_int(p1.w);  // material type of the triangle's mesh
                    }
                }
                if (kAny && any) {
                    finished = true;
                    hit_tri = 0;
                } else {
                    node = sp > 0 ? pop() : kDone;
                    finished = node == kDone;
                }
            }
            if (finished) {
                if (kAny) {
                    if (hit_tri < 0) {  // unoccluded: add the NEE contribution
                        float4 c = P.sh_c[idx];
                        int target = __float_as_int(c.w);
                        if (target >= 0) {
                            if (slot_ok(P, target)) {
                                PathRec pr = P.rec[target].path;
                                pr.L = make_float4(__fadd_rn(pr.L.x, c.x), __fadd_rn(pr.L.y, c.y),
                                                   __fadd_rn(pr.L.z, c.z), pr.L.w);
                                P.rec[target].path = pr;
                                // NEE at the newest guided vertex feeds the record before it
                                if (P.guided) credit(P, P.grec[target], xyz(c), false);
                            }
                        } else {
                            add_to_sample(P, (unsigned long long)(unsigned)(-1 - target), c);
                        }
                    }
                } else {
                    HitRec hr;
                    hr.pad = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (hit_tri >= 0) {
                        hr.h = make_float4(ht, hu, hv, __int_as_float(hit_tri));
                        dest = hit_mat;
                    } else {
                        hr.h = make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
                        dest = kMissQueue;
                    }
                    if (slot_ok(P, slot)) P.rec[slot].hit = hr;
                }
                has = false;
            }
        }
        if (!kAny) {
            unsigned fm = __ballot_sync(0xffffffffu, finished);
            while (fm) {  // warp-uniform loop over the destinations present
                const int dd = __shfl_sync(0xffffffffu, dest, __ffs(fm) - 1);
                const unsigned g = __ballot_sync(0xffffffffu, finished && dest == dd);
                fm &= ~g;
                int* buf = s_qbuf[warp][dd];
                int c = s_qcnt[warp][dd];
                if ((g >> lane) & 1u) buf[c + __popc(g & lt)] = slot;
                c += __popc(g);
                __syncwarp();
                if (c >= 32) {
                    int base = 0;
                    if (lane == 0) base = atomicAdd(&P.cnt->mat[p][dd].n, 32);
                    base = __shfl_sync(0xffffffffu, base, 0);
                    if (DL_IN_BOUNDS(base + 32 <= P.capacity, &P.cnt->err)) P.mat_q[dd][base + lane] = buf[lane];
                    const int rest = c - 32;
                    const int v = lane < rest ? buf[32 + lane] : 0;
                    __syncwarp();
                    if (lane < rest) buf[lane] = v;
                    c = rest;
                }
                __syncwarp();
                if (lane == 0) s_qcnt[warp][dd] = c;
                __syncwarp();
            }
        }
    }
    if (!kAny) {  // flush the staged remainders
        for (int dd = 0; dd < kDests; dd++) {
            const int c = s_qcnt[warp][dd];
            if (c == 0) continue;
            int base = 0;
            if (lane == 0) base = atomicAdd(&P.cnt->mat[p][dd].n, c);
            base = __shfl_sync(0xffffffffu, base, 0);
            if (lane < c && DL_IN_BOUNDS(base + c <= P.capacity, &P.cnt->err))
                P.mat_q[dd][base + lane] = s_qbuf[warp][dd][lane];
        }
    }
    if (err) atomicOr(&P.cnt->err, err);
    if (kCount) {
        if (kAny) {
            atomicAdd(&P.cnt->stat_nodes_sh, (unsigned long long)nn);
            atomicAdd(&P.cnt->stat_tris_sh, (unsigned long long)nt);
        } else {
            atomicAdd(&P.cnt->stat_nodes_ext, (unsigned long long)nn);
            atomicAdd(&P.cnt->stat_tris_ext, (unsigned long long)nt);
        }
    }
}

// Rays that hit nothing (path.cpp:23-25, 85-87): with an envmap, add its
// radiance first.  Store the sample, then start new camera paths in the
// freed slots.
template <bool kMulti, int kThreads>
__global__ void __launch_bounds__(kThreads) k_miss(RenderParams P, int p) {
    const int q = p ^ 1;
    if (blockIdx.x == 0 && threadIdx.x == 0) {  // next iteration's traversal cursors (both traversals are done)
        P.cnt->work_ext = 0;
        P.cnt->work_sh = 0;
    }
    int n = P.cnt->mat[p][kMissQueue].n;
    if (!DL_IN_BOUNDS(n >= 0 && n <= P.capacity, &P.cnt->err)) n = 0;
    // Every queued miss starts a new path in its slot.  A warp's entries over
    // the whole launch are known (i0 = w0 + j * stride, all lanes but the
    // last round's tail), so it claims their path indices, and queue
    // positions for the ones the pass still has, with one atomic each; the
    // started paths are a prefix of the warp's entries.
    const int stride = gridDim.x * blockDim.x;
    const int w0 = (blockIdx.x * blockDim.x + threadIdx.x) & ~31;
    int count = 0;
    for (int i0 = w0; i0 < n; i0 += stride) count += min(32, n - i0);
    const unsigned long long total = P.cnt->pass_total;
    unsigned long long pid0 = 0;
    int e0 = 0;
    if (lane_id() == 0 && count > 0) {
        pid0 = atomicAdd(&P.cnt->next_path, (unsigned long long)count);
        const int starts = pid0 < total ? (int)min((unsigned long long)count, total - pid0) : 0;
        if (starts > 0) e0 = atomicAdd(&P.cnt->ext[q], starts);
    }
    pid0 = __shfl_sync(0xffffffffu, pid0, 0);
    e0 = __shfl_sync(0xffffffffu, e0, 0);
    int done_before = 0;  // the warp's entries in earlier rounds
    for (int i0 = w0; i0 < n; i0 += stride) {
        int i = i0 + lane_id();
        bool active = i < n;
        int slot = active ? P.mat_q[kMissQueue][i] : 0;
        if (active && !slot_ok(P, slot)) active = false;
        if (active) {
            int4 m = P.rec[slot].meta.m;
            PathRec pr = camera_record();
            if (!(m.y & PF_CAMERA)) pr = P.rec[slot].path;
            const DevRequest& R = request<kMulti>(P, m.y >> kReqShift);
            const DevScene& sc = R.sc;
            PathState S;
            S.tp = f3(pr.tp.x, pr.tp.y, pr.tp.z);
            S.L = f3(pr.L.x, pr.L.y, pr.L.z);
            S.prev_pdf = pr.L.w;
            S.flags = m.y;
            if (sc.env_light >= 0 && !(R.flags & DL_RENDER_NORMALS))
                add_miss(R, xyz(P.rec[slot].ray.d), S, [&](float3 c) {
                    if (P.guided) credit(P, P.grec[slot], c, true);
                });
            store_sample(P, path_index(m), S.L, slot);
        }
        const int r = done_before + lane_id();
        const unsigned long long pid = pid0 + (unsigned long long)r;
        if (active && pid < total) {
            start_path<kMulti>(P, slot, pid);
            if (DL_IN_BOUNDS(e0 + r < P.capacity, &P.cnt->err)) P.ext_q[q][e0 + r] = slot;
        }
        done_before += min(32, n - i0);
    }
}

// One BSDF type, the whole rest of the path iteration for hits on it
// (enter_vertex, scatter_vertex).  A path that ends here stores its sample
// and its slot starts a new camera path at once; a shadow ray it emitted on
// the way adds to the stored sample when traced.
//
// kGuided (diffuse, Beckmann, GGX in a guided render): blocks of two
// warpgroups; each warpgroup takes 128 queued hits at a time and evaluates
// the guiding network for them on the tensor cores (guide_tc.cuh:
// tcgen05.mma, accumulators in tensor memory);
// each path samples its next direction by one-sample MIS between the learned
// vMF mixture (probability `fraction`) and the BSDF, weighting by
// f cos / (fraction q + (1 - fraction) p_bsdf); NEE's MIS weight uses the
// same combined pdf.  The vertex becomes a training record.
constexpr size_t kGuidedSmem = sizeof(GuideTcSmem);

// A warp's 32 slot records on their way to shared memory: eight lanes fetch
// one 128-byte line each, four lines an instruction, and chunk c of lane l's
// record lands at chunk c ^ (l & 7) of line l (no bank conflicts when each
// lane reads its own record).
__device__ __forceinline__ void fetch_slots(const SlotRec* rec, int slot, float4* line) {
    const int lane = lane_id(), c = lane & 7;
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const int l = 4 * j + (lane >> 3);
        const int s = __shfl_sync(0xffffffffu, slot, l);
        if (s >= 0)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::
                         "r"((uint32_t)__cvta_generic_to_shared(line + 8 * l + (c ^ (l & 7)))),
                         "l"(reinterpret_cast<const float4*>(rec + s) + c) : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}
__device__ __forceinline__ float4 fetched(const float4* line, int c) {
    const int l = lane_id();
    return line[8 * l + (c ^ (l & 7))];
}

// Threads per SM of the plain kernels (80 registers each).  The records of a
// warp's next 32 entries travel to shared memory while it shades the present
// ones; loaded where they were used, DRAM latency left the kernels at 40 % of
// the issue slots (shading, serialised, before -> with 768 | 896 | 1024
// threads: material spheres 11.5 -> 10.5 | 11.6 | 12.0 ms, MIS plates 64 spp
// 11.7 -> 10.4 | 10.8 | 9.5, Cornell 512x512 32 spp 2.9 -> 2.6 | 2.9 | 3.0,
// window-lit room 4.4 -> 3.9 | 4.2 | 3.9; the smaller register budgets spill
// in the GGX kernel).
constexpr int kMaterialThreads = 768;

template <int T, bool kMulti, bool kGuided, int kThreads>
__global__ void __launch_bounds__(kGuided ? kTcThreads : kThreads, kGuided ? 2 : kMaterialThreads / kThreads)
    k_material(RenderParams P, int p) {
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    // the warps' next records (not in the guided kernels, whose shared memory
    // holds the network)
    __shared__ __align__(128) float4 s_line[kGuided ? 1 : kThreads / 32][kGuided ? 1 : 8 * 32];
    const int q = p ^ 1;
    const int lane = lane_id();
    int n = P.cnt->mat[p][T].n;
    if (!DL_IN_BOUNDS(n >= 0 && n <= P.capacity, &P.cnt->err)) n = 0;
    // guided: each warpgroup walks whole 128-row tiles (every thread takes
    // part in the network's warpgroup-wide steps); otherwise each warp walks
    // 32 rows
    constexpr int kSpan = kGuided ? kTcRows : 32;
    // training-record bookkeeping: guided kernels, and mirror / dielectric
    // hits of a guided render (the other types then run their guided kernel)
    constexpr bool kMayGuide = kGuided || (!kMulti && (T == MAT_MIRROR || T == MAT_DIELECTRIC));
    const bool guided = kMayGuide && P.guided;
    uint32_t mma_phase = 0;
    bool net_ok = false;
    if (kGuided) {
        if ((int)blockIdx.x * kTcThreads >= n) return;
        net_ok = guide_tc_begin(*reinterpret_cast<GuideTcSmem*>(dyn_smem), P.gnet.image, &P.cnt->err);
    }
    const int first = (blockIdx.x * blockDim.x + threadIdx.x) & ~(kSpan - 1), stride = gridDim.x * blockDim.x;
    // queue entry i's slot, -1 past the queue's end
    auto queued = [&](int i) {
        const int s = i < n ? P.mat_q[T][i] : -1;
        return s < 0 || slot_ok(P, s) ? s : -1;
    };
    float4* const line = s_line[kGuided ? 0 : threadIdx.x >> 5];
    int next = kGuided ? -1 : queued(first + lane), after = kGuided ? -1 : queued(first + stride + lane);
    if (!kGuided && first < n) fetch_slots(P.rec, next, line);
    for (int i0 = first; i0 < n; i0 += stride) {
        int slot = kGuided ? queued(i0 + tc_row()) : next;
        const bool active = slot >= 0;
        if (!active) slot = 0;
        bool cont = false, emit = false, done = false;
        float4 sh_o = make_float4(0.f, 0.f, 0.f, 0.f), sh_d = sh_o, sh_c = sh_o;
        // ---- phase 1: emitter hit, Russian roulette, depth limit
        PathState S;
        HitInfo h;
        GuideRec gr;
        float2 tuv = make_float2(0.f, 0.f);  // texture coordinates (textured materials)
        float3 s_tan = f3(0.f, 0.f, 0.f);    // aniso_ggx: shading tangent from a tangent map
        float3 dir = f3(0.f, 0.f, 0.f);
        int rid = 0;
        S.tp = dir;
        S.pid = 0;
        S.depth = 0;
        float4 hit;
        RayRec ray;
        PathRec pr;
        MetaRec mr;
        if (kGuided) {
            if (active) {
                hit = P.rec[slot].hit.h;
                ray = P.rec[slot].ray;
                pr = P.rec[slot].path;
                mr = P.rec[slot].meta;
            }
        } else {
            // this round's records have arrived; the next round's travel
            // while this one is computed
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            __syncwarp();
            ray.o = fetched(line, 0);
            ray.d = fetched(line, 1);
            hit = fetched(line, 2);
            pr.tp = fetched(line, 4);
            pr.L = fetched(line, 5);
            const float4 m0 = fetched(line, 6), m1 = fetched(line, 7);
            mr.m = make_int4(__float_as_int(m0.x), __float_as_int(m0.y), __float_as_int(m0.z), __float_as_int(m0.w));
            mr.rng = make_uint4(__float_as_uint(m1.x), __float_as_uint(m1.y), __float_as_uint(m1.z),
                                __float_as_uint(m1.w));
            __syncwarp();
            next = after;
            if (i0 + stride < n) fetch_slots(P.rec, next, line);
            after = queued(i0 + 2 * stride + lane);
        }
        if (active) {
            if (guided) gr = P.grec[slot];
            if (mr.m.y & PF_CAMERA) pr = camera_record();
            S.g = load_rng(mr.rng);
            S.pid = path_index(mr.m);
            S.tp = f3(pr.tp.x, pr.tp.y, pr.tp.z);
            S.eta = pr.tp.w;
            S.L = f3(pr.L.x, pr.L.y, pr.L.z);
            S.prev_pdf = pr.L.w;
            S.depth = mr.m.x;
            S.flags = mr.m.y;
            dir = xyz(ray.d);
            rid = S.flags >> kReqShift;
            const DevRequest& R = request<kMulti>(P, rid);
            if (!DL_IN_BOUNDS(__float_as_int(hit.w) >= 0 && __float_as_int(hit.w) < R.sc.num_tris, &P.cnt->err))
                hit.w = __int_as_float(0);
            done = enter_vertex<T>(R, T, __float_as_int(hit.w), hit.y, hit.z, xyz(ray.o), dir, S, h, tuv, s_tan,
                                   [&](float3 c) {
                                       if (guided) credit(P, gr, c, true);
                                   });
        }
        // ---- phase 2 (guided): the network on the block's 128 shading points
        const bool sampling = active && !done;
        bool use_guide = kGuided && sampling && S.depth < P.gnet.max_depth;
        float in6[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
        float* lob = nullptr;
        if (kGuided) {
            GuideTcSmem& Sm = *reinterpret_cast<GuideTcSmem*>(dyn_smem);
            const int grp = tc_group();
            lob = tc_out_row(Sm, grp, tc_row());
            if (use_guide) guide_input(request<kMulti>(P, rid).sc, h.p, normalize(h.sh.n), in6);
            // (also the barrier after which the previous tile's lobes are dead)
            if (wg_or(grp, use_guide) && net_ok) {
                encode_row_tc(in6, Sm.act[grp], tc_row());
                net_ok = guide_tc_forward(Sm, grp, mma_phase, &P.cnt->err);
            }
            if (!net_ok) use_guide = false;  // a wait ran out: sample the BSDF alone
            if (use_guide) decode_lobes_inplace(lob);
        }
        // ---- phase 3: NEE and the next direction
        bool record = false, rotate = false;
        float3 nd = f3(0.f, 0.f, 0.f);
        if (active) {
            int target = slot;
            if (!done) {
                Scatter sc;
                done = scatter_vertex<T, kGuided>(request<kMulti>(P, rid), T, rid, h, dir, tuv, s_tan, use_guide, lob,
                                                  use_guide ? P.gnet.fraction : 0.f, S, sc);
                nd = sc.nd;
                emit = sc.emit;
                if (!done) {
                    RayRec nr;
                    nr.o = make_float4(h.p.x, h.p.y, h.p.z, __int_as_float(rid));
                    nr.d = make_float4(nd.x, nd.y, nd.z, __int_as_float(0x7f800000));
                    P.rec[slot].ray = nr;
                    cont = true;
                    rotate = use_guide && P.grecords != nullptr;
                    record = rotate && (uint32_t)(splitmix64(S.pid * 64ull + (unsigned long long)S.depth) >> 40) <
                                           P.cnt->pass_keep;
                }
                if (emit) {
                    if (done) target = -1 - (int)S.pid;  // lands in the stored sample
                    sh_o = make_float4(h.p.x, h.p.y, h.p.z, __int_as_float(rid));
                    sh_d = make_float4(sc.ld.x, sc.ld.y, sc.ld.z, __fsub_rn(sc.ldist, kRayEps));
                    sh_c = make_float4(sc.c.x, sc.c.y, sc.c.z, __int_as_float(target));
                }
            }
            if (done) {
                store_sample(P, S.pid, S.L, slot);
            } else {
                PathRec npr;
                npr.tp = make_float4(S.tp.x, S.tp.y, S.tp.z, S.eta);
                npr.L = make_float4(S.L.x, S.L.y, S.L.z, S.prev_pdf);
                P.rec[slot].path = npr;
                MetaRec nmr;
                nmr.m = make_int4(S.depth, S.flags, (int)(S.pid & 0xffffffffu), (int)(S.pid >> 32));
                nmr.rng = store_rng(S.g);
                P.rec[slot].meta = nmr;
            }
        }
        // ---- phase 4 (guided): training record of the vertex (a hashed
        // subset of the guided vertices, spread over the whole pass)
        if (kGuided) {
            unsigned long long ri = warp_claim_u32(&P.cnt->guide_next, record);
            if (rotate) {
                int idx = record && ri < (unsigned long long)P.grecord_cap ? (int)ri : -1;
                if (idx >= 0) {
                    GuideRecord rc;
                    for (int k = 0; k < 6; k++) rc.in[k] = in6[k];
                    rc.w[0] = nd.x;
                    rc.w[1] = nd.y;
                    rc.w[2] = nd.z;
                    rc.pdf = S.prev_pdf;
                    rc.L = 0.f;
                    rc.pad = 0.f;
                    static_cast<GuideRecord*>(P.cnt->pass_recs)[idx] = rc;
                }
                GuideRec ngr;
                ngr.a = gr.b;
                ngr.b = make_float4(S.tp.x, S.tp.y, S.tp.z, __int_as_float(idx));
                P.grec[slot] = ngr;
            }
        }
        int sp = warp_push(&P.cnt->shadow[q], emit);
        if (emit && DL_IN_BOUNDS(sp < P.capacity, &P.cnt->err)) {
            P.sh_o[sp] = sh_o;
            P.sh_d[sp] = sh_d;
            P.sh_c[sp] = sh_c;
        }
        bool fresh = regenerate<kMulti>(P, slot, done);
        bool push = cont || fresh;
        int e = warp_push(&P.cnt->ext[q], push);
        if (push && DL_IN_BOUNDS(e < P.capacity, &P.cnt->err)) P.ext_q[q][e] = slot;
    }
    if (kGuided) guide_tc_end(*reinterpret_cast<GuideTcSmem*>(dyn_smem), mma_phase);
}

// Film accumulation as a gather (the reference splats each sample with
// ImageBlock::put, src/core/bitmap/block.cpp:81-113).  One block of 256
// threads owns a tile of kTile x kTile film pixels; per sample index it
// stages the samples of the (kTile + 4)^2 image pixels around it (radiance
// from the sample buffer, film position recomputed from the path's pcg32
// stream: its first 2D draw) in shared memory together with their 5 x and 5 y
// filter weights (the reference's table lookup).  Each thread then owns
// kFilmRows film pixels of one column and sums the weighted samples of their
// 5x5 neighbourhoods; a staged sample's radiance and x weight are read once
// for all of them.  Every pixel sums in a fixed order (sample index, then
// row, then column): no atomics, bit-reproducible films.  Samples the film
// rejects (NaN, Inf or negative: ImageBlock::put block.cpp:82-88) get zero
// weight and are counted.
//
// The next sample's radiances are loaded while the present one is summed.
// Two tile sizes: 32 (four rows a thread) moves the fewest bytes and
// instructions a pixel, 16 (one row a thread) has four times the blocks and a
// shorter chain a sample, for frames whose tiles of 32 leave the chip idle.
//
// Bound by issue slots and the width of shared memory (57 % and 65 % of their
// peaks at 1080p with tiles of 32).  A cell's geometry is the thread's, not
// found again for every sample; weights are taken without bounds tests (those
// of film pixels outside the tile are never read) and without integer
// conversions; and what the sums read together is one vector.  That is 31 %
// fewer instructions than a plane per value and a test per weight: film of 16
// samples 1080p 0.73 -> 0.63 ms, 517x389 0.130 -> 0.085, 256x256 0.062 ->
// 0.039 (launches alone).  Tiles of 32 at two blocks an SM: at three the 80
// registers spill (1080p frame 3.93 ms against 3.87).
constexpr int kFilmApron = 2, kFilmThreads = 256;
constexpr int kFilmTaps = 2 * kFilmApron + 1;  // 5 film pixels per axis around a sample
template <int kTile>
struct FilmTile {
    static constexpr int kRegion = kTile + 2 * kFilmApron, kCells = kRegion * kRegion;
    static constexpr int kRows = kTile * kTile / kFilmThreads;                       // film pixels of a thread
    // staging: a thread's cells are in one region column, kStride rows apart
    static constexpr int kStride = kFilmThreads / kRegion, kOwn = (kRegion + kStride - 1) / kStride;
    // staged per cell: r, g, b, 5 y weights, 5 x weights
    static constexpr size_t kSmem = (3 + 2 * kFilmTaps) * sizeof(float) * kCells;
    // A cell's {r, g, b, y weight 4} is one vector; y weights 0..3 are two
    // vectors where a thread with four rows takes several of them, else
    // planes of words (a word of a vector costs the vector's bandwidth).
    static constexpr bool kPairs = kRows > 1;
};

struct FilmParams {
    float4* film;
    const float4* samples;
    unsigned long long* invalid;
    int w, h, cols, rows, border;
    float lookup;
    float table[33];
    int nspp;             // samples per pixel in the sample buffer
    int s_first;          // sample index of the buffer's first sample
    unsigned long long seed_mix;
    int accumulate;       // add to the film instead of overwriting it
};

template <int kTile>
__global__ void __launch_bounds__(kFilmThreads, kTile == 32 ? 2 : 4)
    k_film_gather(FilmParams F) {
    using Tile = FilmTile<kTile>;
    constexpr int kRows = Tile::kRows, kCells = Tile::kCells, kRegion = Tile::kRegion;
    extern __shared__ __align__(16) unsigned char dyn_smem[];
    float4* const s_v = reinterpret_cast<float4*>(dyn_smem);
    float* const s_wy = reinterpret_cast<float*>(s_v + kCells);   // [4][kCells], or [2][kCells] pairs
    float* const s_wx = s_wy + 4 * kCells;                        // [kFilmTaps][kCells]
    __shared__ float s_table[33];
    __shared__ unsigned int s_invalid;
    const int tx = threadIdx.x % kTile, ty = threadIdx.x / kTile;  // column, group of kRows rows
    const int X0 = blockIdx.x * kTile, Y0 = blockIdx.y * kTile;
    const int X = X0 + tx, Yb = Y0 + kRows * ty;
    const int IX0 = X0 - F.border - kFilmApron, IY0 = Y0 - F.border - kFilmApron;
    const size_t npix = (size_t)F.w * F.h;
    if (threadIdx.x < 33) s_table[threadIdx.x] = F.table[threadIdx.x];
    if (threadIdx.x == 0) s_invalid = 0;
    // the thread's cells: column rx of the region, rows ry0, ry0 + kStride, ...
    const int rx = threadIdx.x % kRegion, ry0 = threadIdx.x / kRegion;
    const int sx = IX0 + rx;
    const bool stages = ry0 < Tile::kStride;
    const bool inside = stages && sx >= 0 && sx < F.w;
    const float fcol = (float)(X0 + rx);
    // their samples of index k (w = 0 outside the image)
    float4 L[Tile::kOwn];
    auto load = [&](int k) {
#pragma unroll
        for (int j = 0; j < Tile::kOwn; j++) {
            const int ry = ry0 + j * Tile::kStride, sy = IY0 + ry;
            L[j] = make_float4(0.f, 0.f, 0.f, 0.f);
            if (inside && ry < kRegion && sy >= 0 && sy < F.h)
                L[j] = F.samples[(size_t)k * npix + (size_t)sy * F.w + sx];
        }
    };
    // the filter's weight at distance |c - p|: entry min(int(distance x lookup),
    // 32) of the table (the truncation by an addition that rounds towards
    // zero: conversions run at a quarter of the rate); entry 32 is 0
    auto weight = [&](float c, float p) {
        const float v = fminf(__fmul_rn(fabsf(__fsub_rn(c, p)), F.lookup), 32.f);
        return s_table[__float_as_int(__fadd_rz(v, 8388608.f)) - 0x4b000000];
    };
    load(0);
    __syncthreads();
    float ar[kRows], ag[kRows], ab[kRows], aw[kRows];
#pragma unroll
    for (int j = 0; j < kRows; j++) ar[j] = ag[j] = ab[j] = aw[j] = 0.f;
    for (int k = 0; k < F.nspp; k++) {
#pragma unroll
        for (int j = 0; j < Tile::kOwn; j++) {
            const int ry = ry0 + j * Tile::kStride;
            if (!stages || ry >= kRegion) break;
            const int e = ry * kRegion + rx, sy = IY0 + ry;
            const bool ok = L[j].w != 0.f && L[j].x >= 0.f && L[j].y >= 0.f && L[j].z >= 0.f && isfinite(L[j].x) &&
                            isfinite(L[j].y) && isfinite(L[j].z);
            // each sample is counted by the tile that owns its pixel
            if (!ok && L[j].w != 0.f && rx >= kFilmApron && rx < kFilmApron + kTile && ry >= kFilmApron &&
                ry < kFilmApron + kTile)
                atomicAdd(&s_invalid, 1u);
            float px = -1e6f, py = -1e6f;   // (weight 0 everywhere)
            if (ok) {
                Pcg32 g;
                seed_path(g, F.seed_mix, F.w, F.h, sx, sy, F.s_first + k);
                float2 ps = g.next2d();
                float fx = __fadd_rn((float)sx, ps.x), fy = __fadd_rn((float)sy, ps.y);
                px = __fsub_rn(__fsub_rn(fx, 0.5f), (float)(-F.border));
                py = __fsub_rn(__fsub_rn(fy, 0.5f), (float)(-F.border));
            }
            // weights of this sample for film columns X0 + rx - d and rows
            // Y0 + ry - d (those outside the film or the tile are not used)
            const float frow = (float)(Y0 + ry);
            float wy[kFilmTaps];
#pragma unroll
            for (int d = 0; d < kFilmTaps; d++) {
                s_wx[d * kCells + e] = weight(__fsub_rn(fcol, (float)d), px);
                wy[d] = weight(__fsub_rn(frow, (float)d), py);
            }
            s_v[e] = make_float4(ok ? L[j].x : 0.f, ok ? L[j].y : 0.f, ok ? L[j].z : 0.f, wy[4]);
            if (Tile::kPairs) {
                reinterpret_cast<float2*>(s_wy)[e] = make_float2(wy[0], wy[1]);
                reinterpret_cast<float2*>(s_wy)[kCells + e] = make_float2(wy[2], wy[3]);
            } else {
#pragma unroll
                for (int d = 0; d < 4; d++) s_wy[d * kCells + e] = wy[d];
            }
        }
        __syncthreads();
        if (k + 1 < F.nspp) load(k + 1);
        // region rows kRows*ty + r reach this thread's pixel j when
        // dy = r - j is a filter tap; per pixel the order is dy, then dx
#pragma unroll
        for (int r = 0; r < kRows + kFilmTaps - 1; r++) {
            const int lo = r < kRows ? 0 : r - kRows + 1, hi = r < kFilmTaps ? r : kFilmTaps - 1;  // taps in use
#pragma unroll
            for (int dx = 0; dx < kFilmTaps; dx++) {
                const int c = (kRows * ty + r) * kRegion + tx + dx;
                const float wx = s_wx[dx * kCells + c];
                const float4 v = s_v[c];
                float wy[kFilmTaps];
                wy[4] = v.w;
                if (Tile::kPairs) {
#pragma unroll
                    for (int q = 0; q < 2; q++)
                        if (lo <= 2 * q + 1 && hi >= 2 * q) {
                            const float2 y = reinterpret_cast<const float2*>(s_wy)[q * kCells + c];
                            wy[2 * q] = y.x;
                            wy[2 * q + 1] = y.y;
                        }
                } else if (lo < 4) {
                    wy[lo] = s_wy[lo * kCells + c];
                }
                const float R = __fmul_rn(v.x, wx), G = __fmul_rn(v.y, wx), B = __fmul_rn(v.z, wx);
#pragma unroll
                for (int j = 0; j < kRows; j++) {
                    const int dy = r - j;
                    if (dy < 0 || dy >= kFilmTaps) continue;
                    ar[j] = __fmaf_rn(R, wy[dy], ar[j]);
                    ag[j] = __fmaf_rn(G, wy[dy], ag[j]);
                    ab[j] = __fmaf_rn(B, wy[dy], ab[j]);
                    aw[j] = __fmaf_rn(wx, wy[dy], aw[j]);
                }
            }
        }
        __syncthreads();
    }
    if (threadIdx.x == 0 && s_invalid) atomicAdd(F.invalid, (unsigned long long)s_invalid);
    if (X >= F.cols) return;
#pragma unroll
    for (int j = 0; j < kRows; j++) {
        const int Y = Yb + j;
        if (Y >= F.rows) break;
        float4* o = F.film + (size_t)Y * F.cols + X;
        if (F.accumulate) {
            float4 c = *o;
            *o = make_float4(__fadd_rn(c.x, ar[j]), __fadd_rn(c.y, ag[j]), __fadd_rn(c.z, ab[j]),
                             __fadd_rn(c.w, aw[j]));
        } else {
            *o = make_float4(ar[j], ag[j], ab[j], aw[j]);
        }
    }
}

template <int kTile>
static void launch_film(const FilmParams& F, cudaStream_t st) {
    const dim3 grid((F.cols + kTile - 1) / kTile, (F.rows + kTile - 1) / kTile);
    k_film_gather<kTile><<<grid, kFilmThreads, FilmTile<kTile>::kSmem, st>>>(F);
    DL_CUDA(cudaGetLastError());
}

// The gather of F's samples, on tiles of 32 when there are three for every
// four SMs: fewer leave the chip idle longer than the smaller tiles' wider
// margins cost.  Whole renders of an empty scene, device ms (tiles of 16 | of
// 32): 64x64 64 spp 0.134 | 0.255; 256x256 16 spp 0.097 | 0.119 (81 tiles of
// 32 on 152 SMs); 360x270 16 spp 0.130 | 0.132 (108); 400x300 16 spp 0.156 |
// 0.144 (130); 517x389 16 spp 0.53 | 0.51; 1280x720 16 spp 1.85 | 1.73.
static void film_gather(const FilmParams& F, int sms, cudaStream_t st) {
    const int64_t tiles = (int64_t)((F.cols + 31) / 32) * ((F.rows + 31) / 32);
    if (4 * tiles >= 3 * (int64_t)sms) launch_film<32>(F, st);
    else launch_film<16>(F, st);
}

// Per device, once per context: kernels whose shared memory exceeds the
// default 48 KB limit.
void render_setup_device() {
    DL_CUDA(cudaFuncSetAttribute(k_film_gather<32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)FilmTile<32>::kSmem));
}

// film -> rgb (ImageBlock::toBitmap, block.cpp:58-66)
__global__ void k_resolve(const float4* film, int cols, int border, int w, int h, float* rgb) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= w * h) return;
    int x = i % w, y = i / w;
    float4 c = film[(size_t)(y + border) * cols + (x + border)];
    float r = 0.f, g = 0.f, b = 0.f;
    if (c.w != 0.f) {
        r = __fdiv_rn(c.x, c.w);
        g = __fdiv_rn(c.y, c.w);
        b = __fdiv_rn(c.z, c.w);
    }
    rgb[3 * (size_t)i] = r;
    rgb[3 * (size_t)i + 1] = g;
    rgb[3 * (size_t)i + 2] = b;
}

// ------------------------------------------------------------------- host
void RenderBuffers::ensure(int64_t cap) {
    if (cap <= capacity) return;
    size_t c = (size_t)cap;
    rec.ensure(128 * c);
    pos.ensure(8 * c);
    for (DevBuf* b : {&sh_o, &sh_d, &sh_c}) b->ensure(16 * c);
    for (DevBuf* b : {&ext_q[0], &ext_q[1]}) b->ensure(4 * c);
    for (int k = 0; k <= kNumMaterialTypes; k++) mat_q[k].ensure(4 * c);
    counters.ensure(sizeof(RenderCounters));
    invalid.ensure(sizeof(unsigned long long));
    host_counters.ensure(sizeof(RenderCounters) + sizeof(unsigned long long));
    capacity = cap;
}

size_t RenderBuffers::device_bytes() const {
    size_t s = rec.bytes + pos.bytes + ext_q[0].bytes + ext_q[1].bytes +
               sh_o.bytes + sh_d.bytes + sh_c.bytes + counters.bytes + film.bytes + rgb.bytes + samples.bytes;
    for (int k = 0; k <= kNumMaterialTypes; k++) s += mat_q[k].bytes;
    return s;
}

constexpr int kKernelsPerIteration = 8;

// The material kernel of type T: guided (the network's tiles and weights in
// dynamic shared memory, as many blocks as fit at once) for the non-delta
// BSDFs of a guided render.
template <int T, bool kMulti>
static void launch_material(const RenderParams& P, int p, cudaStream_t st, int wb, int th) {
    constexpr bool kCanGuide = !kMulti && T != MAT_MIRROR && T != MAT_DIELECTRIC;
    if (kCanGuide && P.guided)
        k_material<T, false, true, kTcThreads><<<P.gnet.blocks, kTcThreads, kGuidedSmem, st>>>(P, p);
    else if (th > 128)  // compiled for 256-thread blocks
        k_material<T, kMulti, false, 256><<<wb, th, 0, st>>>(P, p);
    else
        k_material<T, kMulti, false, 128><<<wb, th, 0, st>>>(P, p);
}

template <bool kMulti>
static void launch_miss(const RenderParams& P, int p, cudaStream_t st, int wb, int th) {
    if (th > 128)
        k_miss<kMulti, 256><<<wb, th, 0, st>>>(P, p);
    else
        k_miss<kMulti, 128><<<wb, th, 0, st>>>(P, p);
}

// Launches one wavefront iteration (8 kernels) with the context's launch
// shape.  `ev`, when given, holds 8 events bracketing extend, shadow, the
// material kernels, miss (kernels then run one after another).  Otherwise,
// with `fj` given, independent kernels run concurrently on the context's
// side streams: the extension traversal (this iteration's rays: reads their
// ray records, writes hit records) beside the shadow traversal (the previous
// iteration's NEE rays: adds to path records), then the miss kernel beside
// the five material kernels (disjoint slots and queues), joined before the
// next iteration.
template <bool kMulti>
static void launch_iteration(const RenderParams& P, int p, cudaStream_t st, int sms, const TuneParams& tp,
                             bool count, cudaEvent_t* ev, const dl_context* fj) {
    const int tb = sms * tp.trav_ctas_per_sm, wb = sms * tp.shade_ctas_per_sm, th = 128, sth = tp.shade_threads;
    if (!ev && fj) {
        cudaEventRecord(fj->fork_ev, st);
        cudaStreamWaitEvent(fj->aux[0], fj->fork_ev, 0);
        if (count) {
            k_traverse<true, false, kMulti><<<tb, th, 0, st>>>(P, p);
            k_traverse<true, true, kMulti><<<tb, th, 0, fj->aux[0]>>>(P, p);
        } else {
            k_traverse<false, false, kMulti><<<tb, th, 0, st>>>(P, p);
            k_traverse<false, true, kMulti><<<tb, th, 0, fj->aux[0]>>>(P, p);
        }
        cudaEventRecord(fj->join_ev[0], fj->aux[0]);
        cudaStreamWaitEvent(st, fj->join_ev[0], 0);
    } else {
        if (ev) cudaEventRecord(ev[0], st);
        if (count) k_traverse<true, false, kMulti><<<tb, th, 0, st>>>(P, p);
        else k_traverse<false, false, kMulti><<<tb, th, 0, st>>>(P, p);
        if (ev) { cudaEventRecord(ev[1], st); cudaEventRecord(ev[2], st); }
        if (count) k_traverse<true, true, kMulti><<<tb, th, 0, st>>>(P, p);
        else k_traverse<false, true, kMulti><<<tb, th, 0, st>>>(P, p);
        if (ev) { cudaEventRecord(ev[3], st); cudaEventRecord(ev[4], st); }
    }
    if (!ev && fj) {
        cudaEventRecord(fj->fork_ev, st);
        for (int i = 0; i < dl_context::kAux; i++) cudaStreamWaitEvent(fj->aux[i], fj->fork_ev, 0);
        launch_miss<kMulti>(P, p, st, wb, sth);
        launch_material<MAT_DIFFUSE, kMulti>(P, p, fj->aux[0], wb, sth);
        launch_material<MAT_MIRROR, kMulti>(P, p, fj->aux[1], wb, sth);
        launch_material<MAT_DIELECTRIC, kMulti>(P, p, fj->aux[2], wb, sth);
        launch_material<MAT_MICROFACET, kMulti>(P, p, fj->aux[3], wb, sth);
        launch_material<MAT_ANISO_GGX, kMulti>(P, p, fj->aux[4], wb, sth);
        for (int i = 0; i < dl_context::kAux; i++) {
            cudaEventRecord(fj->join_ev[i], fj->aux[i]);
            cudaStreamWaitEvent(st, fj->join_ev[i], 0);
        }
    } else {
        launch_material<MAT_DIFFUSE, kMulti>(P, p, st, wb, sth);
        launch_material<MAT_MIRROR, kMulti>(P, p, st, wb, sth);
        launch_material<MAT_DIELECTRIC, kMulti>(P, p, st, wb, sth);
        launch_material<MAT_MICROFACET, kMulti>(P, p, st, wb, sth);
        launch_material<MAT_ANISO_GGX, kMulti>(P, p, st, wb, sth);
        if (ev) { cudaEventRecord(ev[5], st); cudaEventRecord(ev[6], st); }
        launch_miss<kMulti>(P, p, st, wb, sth);
    }
    if (ev) cudaEventRecord(ev[7], st);
}

static void bind_pool(RenderParams& P, const RenderBuffers& B) {
    P.capacity = (int)B.capacity;
    P.rec = B.rec.as<SlotRec>();
    P.pos = B.pos.as<float2>();
    P.ext_q[0] = B.ext_q[0].as<int>();
    P.ext_q[1] = B.ext_q[1].as<int>();
    for (int k = 0; k <= kNumMaterialTypes; k++) P.mat_q[k] = B.mat_q[k].as<int>();
    P.sh_o = B.sh_o.as<float4>();
    P.sh_d = B.sh_d.as<float4>();
    P.sh_c = B.sh_c.as<float4>();
    P.cnt = B.counters.as<RenderCounters>();
}

void filter_setup(int filter, float& radius, int& border, float& lookup, float* table) {
    const int RES = 32;
    radius = filter == DL_FILTER_BOX ? 0.5f : 2.0f;
    border = (int)std::ceil(radius - 0.5f);
    for (int i = 0; i < RES; ++i) {
        float pos = (radius * i) / RES;
        if (filter == DL_FILTER_BOX) {
            table[i] = 1.0f;
        } else {
            const float stddev = 0.5f;
            float alpha = -1.0f / (2.0f * stddev * stddev);
            table[i] = std::max(0.0f, std::exp(alpha * pos * pos) - std::exp(alpha * radius * radius));
        }
    }
    table[RES] = 0.0f;
    lookup = RES / radius;
}

int64_t film_floats(int w, int h, int filter) {
    int b = filter == DL_FILTER_BOX ? 0 : 2;
    return (int64_t)(w + 2 * b) * (h + 2 * b) * 4;
}

static DevRequest make_request(dl_scene* S, const dl_render_opts& o) {
    DevRequest R;
    std::memset(&R, 0, sizeof(R));
    R.sc = S->dev;
    R.pid_first = 0;
    R.spp_offset = o.spp_offset;
    R.max_depth = o.max_depth;
    R.rr_depth = o.rr_depth;
    R.flags = o.flags;
    R.seed_mix = splitmix64(o.seed);
    return R;
}

// The values that change from pass to pass live in the device counters (set
// after their reset), not in the kernel parameters: one captured graph serves
// every pass and frame.
struct PassValues {
    unsigned long long total;
    int spp_offset;
    unsigned keep;
    void* recs;
};
static_assert(sizeof(PassValues) == 24, "pass values layout");

static void check_render_error(unsigned int err) {
    if (err & kErrBounds) throw Error(DL_ERR_QUEUE_OVERFLOW, kBoundsMessage);
    if (err & kErrTensorWait) throw Error(DL_ERR_TIMEOUT, "tensor-core wait timed out in a guided kernel");
    if (err & kErrRounds) throw Error(DL_ERR_TIMEOUT, "render did not converge");
    if (err) throw Error(DL_ERR_QUEUE_OVERFLOW, "traversal stack overflow");
}

// Wavefront loop over the paths [0, total) of one pass, until every path and
// every shadow ray has finished.  Adds the pass's counters into `acc` and
// per-kernel times into kms.  `multi`: paths of a request table.
static void run_wavefront(dl_context* ctx, RenderParams& P, int64_t cap, bool multi, bool count_traversal,
                          double* kms, int64_t& launches, int64_t& iters, RenderCounters& acc,
                          unsigned long long total, int spp_offset, unsigned keep, bool tail, void* recs = nullptr) {
    cudaStream_t st = ctx->stream;
    RenderBuffers& B = ctx->render;
    const TuneParams tp = ctx->tune;
    const int batch = graph_iterations(tp, tail);
    DL_CUDA(cudaMemsetAsync(P.cnt, 0, sizeof(RenderCounters), st));
    B.host_pass.ensure(sizeof(PassValues));
    PassValues* pv = B.host_pass.as<PassValues>();
    pv->total = total;
    pv->spp_offset = spp_offset;
    pv->keep = keep;
    pv->recs = recs;
    DL_CUDA(cudaMemcpyAsync(&P.cnt->pass_total, pv, sizeof(PassValues), cudaMemcpyHostToDevice, st));
    const int sms = ctx->num_sms > 0 ? ctx->num_sms : 152;
    const bool timing = ctx->kernel_timing;
    const bool use_graph = !timing && !count_traversal;
    if (timing && (int)ctx->timing_events.size() < 8 * batch) {
        size_t have = ctx->timing_events.size();
        ctx->timing_events.resize(8 * batch);
        for (size_t k = have; k < ctx->timing_events.size(); k++) DL_CUDA(cudaEventCreate(&ctx->timing_events[k]));
    }
    auto iteration = [&](int k, bool count, cudaEvent_t* ev) {
        if (multi) launch_iteration<true>(P, k & 1, st, sms, tp, count, ev, ctx);
        else launch_iteration<false>(P, k & 1, st, sms, tp, count, ev, ctx);
    };
    if (use_graph) {
        std::vector<unsigned char> key(sizeof(P) + sizeof(int) + sizeof(cudaStream_t) + sizeof(TuneParams) + 2);
        unsigned char* kp = key.data();
        std::memcpy(kp, &P, sizeof(P));
        kp += sizeof(P);
        std::memcpy(kp, &sms, sizeof(int));
        kp += sizeof(int);
        std::memcpy(kp, &st, sizeof(cudaStream_t));
        kp += sizeof(cudaStream_t);
        std::memcpy(kp, &tp, sizeof(TuneParams));
        kp += sizeof(TuneParams);
        *kp++ = multi ? 1 : 0;
        *kp = (unsigned char)batch;
        if (!ctx->graph_exec || key != ctx->graph_key) {
            cudaGraph_t g = nullptr;
            DL_CUDA(cudaStreamBeginCapture(st, cudaStreamCaptureModeThreadLocal));
            for (int k = 0; k < batch; k++) iteration(k, false, nullptr);
            DL_CUDA(cudaStreamEndCapture(st, &g));
            // another frame of the same launches: the new parameters go into
            // the graph there is (instantiating one took 0.4 of the 0.5 ms
            // that a new frame cost)
            cudaGraphExecUpdateResultInfo info;
            cudaError_t e = ctx->graph_exec ? cudaGraphExecUpdate(ctx->graph_exec, g, &info) : cudaErrorGraphExecUpdateFailure;
            if (e != cudaSuccess) {
                (void)cudaGetLastError();
                if (ctx->graph_exec) cudaGraphExecDestroy(ctx->graph_exec);
                ctx->graph_exec = nullptr;
                e = cudaGraphInstantiate(&ctx->graph_exec, g, 0);
            }
            cudaGraphDestroy(g);
            if (e != cudaSuccess) {
                ctx->graph_exec = nullptr;
                throw Error(DL_ERR_CUDA, std::string("cudaGraphInstantiate: ") + cudaGetErrorString(e));
            }
            ctx->graph_key = key;
        }
    }
    if (multi) k_init<true><<<sms * 16, 128, 0, st>>>(P, (int)cap);
    else k_init<false><<<sms * 16, 128, 0, st>>>(P, (int)cap);
    launches += 1;
    RenderCounters* hc = B.host_counters.as<RenderCounters>();
    for (;;) {
        if (use_graph) {
            DL_CUDA(cudaGraphLaunch(ctx->graph_exec, st));
        } else {
            for (int k = 0; k < batch; k++)
                iteration(k, count_traversal, timing ? &ctx->timing_events[8 * k] : nullptr);
        }
        iters += batch;
        launches += batch * kKernelsPerIteration;
        DL_CUDA(cudaGetLastError());
        DL_CUDA(cudaMemcpyAsync(hc, P.cnt, sizeof(RenderCounters), cudaMemcpyDeviceToHost, st));
        DL_CUDA(cudaStreamSynchronize(st));
        if (timing) {
            for (int k = 0; k < batch; k++)
                for (int j = 0; j < 4; j++) {
                    float ms = 0.f;
                    DL_CUDA(cudaEventElapsedTime(&ms, ctx->timing_events[8 * k + 2 * j],
                                                 ctx->timing_events[8 * k + 2 * j + 1]));
                    kms[j] += ms;
                }
        }
        check_render_error(hc->err);
        if (hc->ext[0] == 0 && hc->shadow[0] == 0 && hc->next_path >= total) break;
        if (tail && hc->next_path >= total && hc->ext[0] <= kTailPaths) {
            // few paths left: their shadow rays, then the rest in one launch
            RenderParams R = P;
            R.total = total;
            const int blocks = sms * tp.trav_ctas_per_sm;
            if (multi) k_traverse<false, true, true><<<blocks, 128, 0, st>>>(R, 0);
            else k_traverse<false, true, false><<<blocks, 128, 0, st>>>(R, 0);
            launches += 1;
            if (hc->ext[0] > 0) {
                resident_finish(ctx, R, hc->ext[0], multi, st);
                launches += 1;
            }
            DL_CUDA(cudaGetLastError());
            DL_CUDA(cudaMemcpyAsync(hc, P.cnt, sizeof(RenderCounters), cudaMemcpyDeviceToHost, st));
            DL_CUDA(cudaStreamSynchronize(st));
            check_render_error(hc->err);
            break;
        }
        if (iters > 1000000) throw Error(DL_ERR_TIMEOUT, "render did not converge");
    }
    acc.stat_camera += std::min<unsigned long long>(hc->next_path, total);
    acc.stat_ext += hc->stat_ext;
    acc.stat_shadow += hc->stat_shadow;
    acc.stat_nodes_ext += hc->stat_nodes_ext;
    acc.stat_tris_ext += hc->stat_tris_ext;
    acc.stat_nodes_sh += hc->stat_nodes_sh;
    acc.stat_tris_sh += hc->stat_tris_sh;
}

// Whether the resident kernel may take over a wavefront pass's last paths: no
// pool size asked for, and no need for the wavefront's separate kernels (their
// times or traversal counts).
static bool may_finish(const dl_context* ctx, int64_t pool, bool count_traversal) {
    return pool == 0 && !count_traversal && !ctx->kernel_timing;
}
// Whether it runs a whole pass of `total` paths: few, and not to tune the
// wavefront's launch shape, which it has no use for.
static bool use_resident(const dl_context* ctx, int64_t pool, unsigned long long total, bool count_traversal) {
    return total <= kResidentMaxPaths && may_finish(ctx, pool, count_traversal) && !ctx->tuning;
}

// Budget of the per-path sample buffer; larger frames render in passes of
// whole samples per pixel.
constexpr size_t kSampleBufferBytes = (size_t)4 << 30;

static FilmParams film_params(const DevCamera& cam, const DevRequest& R, int filter, float* d_film,
                              const float4* samples, unsigned long long* invalid) {
    FilmParams F;
    std::memset(&F, 0, sizeof(F));
    float radius;
    filter_setup(filter, radius, F.border, F.lookup, F.table);
    F.film = reinterpret_cast<float4*>(d_film);
    F.samples = samples;
    F.invalid = invalid;
    F.w = cam.w;
    F.h = cam.h;
    F.cols = cam.w + 2 * F.border;
    F.rows = cam.h + 2 * F.border;
    F.seed_mix = R.seed_mix;
    return F;
}

// The end of a render, in two halves around the caller's results: reads the
// counters of a resident pass (`resident`), or the count of invalid samples,
// and marks the end of the render's time; then, after one wait, checks the
// error word of a resident pass and adds its counters.
static void end_render(dl_context* ctx, bool resident, const RenderParams& P, const void* d_invalid,
                       const std::function<void()>& results, RenderCounters& acc) {
    cudaStream_t st = ctx->stream;
    RenderCounters* hc = ctx->render.host_counters.as<RenderCounters>();
    unsigned long long* hinv = reinterpret_cast<unsigned long long*>(hc + 1);
    *hinv = 0;
    if (resident) DL_CUDA(cudaMemcpyAsync(hc, P.cnt, sizeof(RenderCounters), cudaMemcpyDeviceToHost, st));
    else if (d_invalid) DL_CUDA(cudaMemcpyAsync(hinv, d_invalid, sizeof(*hinv), cudaMemcpyDeviceToHost, st));
    DL_CUDA(cudaEventRecord(ctx->ev1, st));
    if (results) results();
    DL_CUDA(cudaStreamSynchronize(st));
    if (resident) {
        check_render_error(hc->err);
        acc.stat_camera += P.total;
        acc.stat_ext += hc->stat_ext;
        acc.stat_shadow += hc->stat_shadow;
        *hinv = hc->stat_invalid;
    }
    acc.stat_invalid = *hinv;
}

static void finish_stats(dl_context* ctx, const RenderCounters& acc, unsigned long long invalid, int64_t iters,
                         int64_t launches, const double* kms) {
    float ms = 0.f;
    DL_CUDA(cudaEventElapsedTime(&ms, ctx->ev0, ctx->ev1));
    ctx->stats.camera_rays = (int64_t)acc.stat_camera;
    ctx->stats.extension_rays = (int64_t)acc.stat_ext;
    ctx->stats.shadow_rays = (int64_t)acc.stat_shadow;
    ctx->stats.invalid_samples = (int64_t)invalid;
    ctx->stats.iterations = iters;
    ctx->stats.render_ms = ms;
    ctx->stats.extend_ms = kms[0];
    ctx->stats.shadow_ms = kms[1];
    ctx->stats.shade_ms = kms[2];
    ctx->stats.retire_ms = kms[3];
    ctx->stats.kernel_launches = launches;
}

static int64_t pool_capacity(dl_context* ctx, int64_t requested, unsigned long long paths) {
    int64_t cap = requested > 0 ? requested : ctx->tune.paths_in_flight;
    cap = std::min<int64_t>(cap, (int64_t)std::max<unsigned long long>(paths, 1ull));
    return ((cap + 31) / 32) * 32;
}

// Runs one render.  mode 0: the film (d_film) receives every sample through
// the gather kernel; mode 1: Li of li_n explicit paths (d_xys -> d_L, d_pos).
void render_run(dl_scene* S, const dl_render_opts& o, float* d_film, int64_t li_n, const int* d_xys,
                float* d_L, float* d_pos, bool count_traversal, RenderCounters* out_counters,
                const std::function<void()>& results) {
    dl_context* ctx = S->ctx;
    cudaStream_t st = ctx->stream;
    const DevCamera& cam = S->dev.cam;
    RenderParams P;
    std::memset(&P, 0, sizeof(P));
    P.r0 = make_request(S, o);
    P.mode = li_n > 0 ? 1 : 0;
    const unsigned long long npix = (unsigned long long)cam.w * cam.h;
    const int spp = std::max(o.spp, 1);
    int chunk_spp = P.mode == 1 ? 1 : (int)std::max<size_t>(1, std::min<size_t>(spp, kSampleBufferBytes / (npix * 16)));
    unsigned long long chunk_total = P.mode == 1 ? (unsigned long long)li_n : npix * (unsigned long long)chunk_spp;
    const bool resident = use_resident(ctx, o.max_paths_in_flight, chunk_total, count_traversal);
    const int64_t cap = resident ? 32 : pool_capacity(ctx, o.max_paths_in_flight, chunk_total);
    RenderBuffers& B = ctx->render;
    B.ensure(cap);
    bind_pool(P, B);
    P.xys = d_xys;
    P.li_L = d_L;
    P.li_pos = d_pos;
    if (P.mode == 0) {
        B.samples.ensure((size_t)chunk_total * 16);
        P.samples = B.samples.as<float4>();
    }
    double kms[4] = {0, 0, 0, 0};
    int64_t launches = 0, iters = 0;
    RenderCounters acc;
    std::memset(&acc, 0, sizeof(acc));
    DL_CUDA(cudaEventRecord(ctx->ev0, st));
    FilmParams F;
    if (P.mode == 0) {
        // (a resident pass counts invalid samples among its counters)
        F = film_params(cam, P.r0, o.filter, d_film, P.samples,
                        resident ? &P.cnt->stat_invalid : B.invalid.as<unsigned long long>());
        if (!resident) DL_CUDA(cudaMemsetAsync(F.invalid, 0, sizeof(unsigned long long), st));
    }
    if (resident) {   // (a whole render: its samples fit the buffer)
        P.total = chunk_total;
        DL_CUDA(cudaMemsetAsync(P.cnt, 0, sizeof(RenderCounters), st));
        resident_launch(ctx, P, false, st);
        launches = iters = 1;
    }
    if (P.mode == 1) {
        if (!resident)
            run_wavefront(ctx, P, cap, false, count_traversal, kms, launches, iters, acc, (unsigned long long)li_n, 0,
                          1u << 24, may_finish(ctx, o.max_paths_in_flight, count_traversal));
    } else {
        for (int s0 = 0; s0 < spp; s0 += chunk_spp) {
            int ns = std::min(chunk_spp, spp - s0);
            if (!resident)
                run_wavefront(ctx, P, cap, false, count_traversal, kms, launches, iters, acc,
                              npix * (unsigned long long)ns, o.spp_offset + s0, 1u << 24,
                              may_finish(ctx, o.max_paths_in_flight, count_traversal));
            F.nspp = ns;
            F.s_first = o.spp_offset + s0;
            F.accumulate = s0 > 0;
            film_gather(F, ctx->num_sms, st);
            launches += 1;
        }
    }
    end_render(ctx, resident, P, P.mode == 0 ? F.invalid : nullptr, results, acc);
    finish_stats(ctx, acc, acc.stat_invalid, iters, launches, kms);
    if (out_counters) *out_counters = acc;
}

// Guided progressive render: passes of 1, 1, 2, 4, ... samples per pixel
// (the last takes the rest; all in one with a frozen network).  During a pass every guided vertex writes a
// training record; after the pass (train) the records feed steps_per_pass
// Adam steps on consecutive batches, and the next pass samples with the
// updated network.  All passes add to one film: each sample is an unbiased
// estimate whichever network drew it.
// Blocks of a guided material launch: as many as are resident at once (each
// loads the weights once and walks tiles), from the SM's registers and
// shared memory.  A context's first call raises the kernels' dynamic
// shared-memory limit (before any graph capture).
template <int T>
static int guided_resident_blocks() {
    auto* fn = k_material<T, false, true, kTcThreads>;
    DL_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kGuidedSmem));
    DL_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributePreferredSharedMemoryCarveout, 100));
    int dev = 0;
    DL_CUDA(cudaGetDevice(&dev));
    cudaDeviceProp prop;
    DL_CUDA(cudaGetDeviceProperties(&prop, dev));
    cudaFuncAttributes fa;
    DL_CUDA(cudaFuncGetAttributes(&fa, fn));
    const int regs_per_warp = ((fa.numRegs + 7) / 8) * 8 * 32;
    const int by_regs = prop.regsPerMultiprocessor / std::max(1, regs_per_warp * (kTcThreads / 32));
    const size_t smem = kGuidedSmem + fa.sharedSizeBytes + prop.reservedSharedMemPerBlock;
    const int by_smem = (int)(prop.sharedMemPerMultiprocessor / smem);
    return std::max(1, std::min(by_regs, by_smem));
}
static int guided_blocks(dl_context* ctx) {
    if (ctx->guided_per_sm == 0)
        ctx->guided_per_sm = std::min(std::min(guided_resident_blocks<MAT_DIFFUSE>(),
                                               guided_resident_blocks<MAT_MICROFACET>()),
                                      guided_resident_blocks<MAT_ANISO_GGX>());
    return ctx->num_sms * ctx->guided_per_sm;
}

void render_guided(dl_scene* S, const dl_render_opts& o, dl_guide* G, float* d_film, bool train) {
    dl_context* ctx = S->ctx;
    cudaStream_t st = ctx->stream;
    const DevCamera& cam = S->dev.cam;
    RenderParams P;
    std::memset(&P, 0, sizeof(P));
    P.r0 = make_request(S, o);
    P.mode = 0;
    const unsigned long long npix = (unsigned long long)cam.w * cam.h;
    const int spp = std::max(o.spp, 1);
    const int chunk_spp = (int)std::max<size_t>(1, std::min<size_t>(spp, kSampleBufferBytes / (npix * 16)));
    const int64_t cap = pool_capacity(ctx, o.max_paths_in_flight, npix * (unsigned long long)chunk_spp);
    RenderBuffers& B = ctx->render;
    B.ensure(cap);
    B.grec.ensure((size_t)cap * 32);
    bind_pool(P, B);
    B.samples.ensure((size_t)npix * chunk_spp * 16);
    P.samples = B.samples.as<float4>();
    P.guided = 1;
    P.gnet.image = G->image.ptr;
    P.gnet.blocks = guided_blocks(ctx);
    P.gnet.fraction = G->cfg.guide_fraction;
    P.gnet.max_depth = G->cfg.max_guided_depth;
    P.grec = B.grec.as<GuideRec>();
    const int64_t rec_cap = std::min<int64_t>((int64_t)G->cfg.batch * std::max(1, G->cfg.steps_per_pass), 1 << 23);
    GuideRecord* rec_half[2] = {nullptr, nullptr};
    if (train) {
        // a training step takes at most ceil(rec_cap / steps) records
        guide_reserve(G, (rec_cap + std::max(1, G->cfg.steps_per_pass) - 1) / std::max(1, G->cfg.steps_per_pass));
        // two halves: pass k writes half k % 2 while the training stream
        // learns from the other half (the previous pass)
        G->pass_recs.ensure(2 * (size_t)rec_cap * sizeof(GuideRecord));
        rec_half[0] = G->pass_recs.as<GuideRecord>();
        rec_half[1] = rec_half[0] + rec_cap;
        P.grecords = rec_half[0];  // non-null: the kernels write records
        P.grecord_cap = (int)rec_cap;
    }
    double kms[4] = {0, 0, 0, 0};
    int64_t launches = 0, iters = 0, records = 0;
    float train_ms = 0.f;
    RenderCounters acc;
    std::memset(&acc, 0, sizeof(acc));
    DL_CUDA(cudaEventRecord(ctx->ev0, st));
    FilmParams F = film_params(cam, P.r0, o.filter, d_film, P.samples, B.invalid.as<unsigned long long>());
    DL_CUDA(cudaMemsetAsync(F.invalid, 0, sizeof(unsigned long long), st));
    RenderCounters* hc = B.host_counters.as<RenderCounters>();
    int done = 0;
    bool trained[2] = {false, false};
    double guided_per_sample = 2.0 * (double)npix;  // guided vertices per sample per pixel: first guess
    cudaStream_t ts = G->train_stream;
    for (int pass = 0; done < spp; pass++) {
        // passes grow while the network learns between them; a frozen one
        // needs no more passes than the sample buffer (16 spp at 480x270:
        // five passes of 16 iterations each took 11.8 ms, one takes 5.2)
        int ns = std::min(train ? std::min(pass == 0 ? 1 : (1 << (pass - 1)), spp - done) : spp - done, chunk_spp);
        // keep about rec_cap of the pass's guided vertices, spread over it
        const double expect = guided_per_sample * ns;
        const double frac = std::min(1.0, 0.9 * (double)rec_cap / std::max(expect, 1.0));
        const unsigned keep = (unsigned)std::max(1.0, frac * (double)(1u << 24));
        const int half = pass & 1;
        // the half this pass writes must be free of the training that read it
        if (train && trained[half]) DL_CUDA(cudaStreamWaitEvent(st, G->train_done[half], 0));
        run_wavefront(ctx, P, cap, false, false, kms, launches, iters, acc, npix * (unsigned long long)ns,
                      o.spp_offset + done, keep, false, rec_half[half]);
        const int64_t claimed = train ? (int64_t)hc->guide_next : 0;
        const int64_t nrec = std::min<int64_t>(claimed, rec_cap);
        if (train && claimed > 0)
            guided_per_sample = (double)claimed / ((double)keep / (double)(1u << 24)) / ns;
        F.nspp = ns;
        F.s_first = o.spp_offset + done;
        F.accumulate = done > 0;
        film_gather(F, ctx->num_sms, st);
        launches += 1;
        done += ns;
        const int steps = G->cfg.steps_per_pass;
        if (train && nrec >= 16 * (int64_t)std::max(1, steps) && done < spp) {
            // Adam steps on this pass's records, on the training stream: the
            // next pass renders meanwhile with the network as it changes (its
            // kernels sample and evaluate the same lobes, so every sample
            // stays unbiased).  Step k trains on records k, k + steps, ...:
            // every step sees the whole image.
            DL_CUDA(cudaEventRecord(G->pass_done[half], st));
            DL_CUDA(cudaStreamWaitEvent(ts, G->pass_done[half], 0));
            DL_CUDA(cudaEventRecord(G->t0, ts));
            for (int k = 0; k < steps; k++) {
                const int64_t cnt = (nrec - k + steps - 1) / steps;
                guide_step(G, rec_half[half] + k, cnt, steps, ts);
            }
            DL_CUDA(cudaEventRecord(G->t1, ts));
            DL_CUDA(cudaEventRecord(G->train_done[half], ts));
            trained[half] = true;
        }
        records += nrec;
    }
    if (train && (trained[0] || trained[1])) {
        // the render ends when its last training round has ended
        DL_CUDA(cudaEventRecord(G->pass_done[0], ts));
        DL_CUDA(cudaStreamWaitEvent(st, G->pass_done[0], 0));
        DL_CUDA(cudaStreamSynchronize(ts));
        DL_CUDA(cudaEventElapsedTime(&train_ms, G->t0, G->t1));  // the last round's device time
    }
    end_render(ctx, false, P, F.invalid, nullptr, acc);
    finish_stats(ctx, acc, acc.stat_invalid, iters, launches, kms);
    ctx->stats.guide_records = records;
    ctx->stats.guide_train_ms = train_ms;
}

// Batch of requests in one wavefront: every pass renders, for each request
// with samples left, its next slice of samples per pixel; all requests' paths
// share the path pool and the material queues (each path carries its
// request), and after the pass one gather per request adds the slice to its
// film.  Slices are sized so a pass fits the sample buffer.
void render_batch(dl_context* ctx, const BatchItem* items, int n, bool count_traversal,
                  const std::function<void()>& results) {
    cudaStream_t st = ctx->stream;
    RenderBuffers& B = ctx->render;
    std::vector<int> done(n, 0);
    unsigned long long all = 0;
    for (int r = 0; r < n; r++)
        all += (unsigned long long)items[r].cam.w * items[r].cam.h * items[r].opts.spp;
    const unsigned long long budget = kSampleBufferBytes / 16;
    // slice of request r per pass: its share of the budget, at least one sample
    std::vector<int> slice(n);
    unsigned long long max_pass = 0;
    for (int r = 0; r < n; r++) {
        const unsigned long long npix = (unsigned long long)items[r].cam.w * items[r].cam.h;
        double share = all <= budget ? 1.0 : (double)budget / (double)all;
        slice[r] = std::max(1, std::min(items[r].opts.spp, (int)(items[r].opts.spp * share)));
        max_pass += npix * (unsigned long long)slice[r];
    }
    int64_t requested = 0;
    for (int r = 0; r < n; r++) requested = std::max<int64_t>(requested, items[r].opts.max_paths_in_flight);
    const bool resident = use_resident(ctx, requested, max_pass, count_traversal);
    const int64_t cap = resident ? 32 : pool_capacity(ctx, requested, max_pass);
    B.ensure(cap);
    B.samples.ensure((size_t)std::max<unsigned long long>(max_pass, 1) * 16);
    B.requests.ensure(sizeof(DevRequest) * (size_t)std::max(n, 1));
    B.host_requests.ensure(sizeof(DevRequest) * (size_t)std::max(n, 1));
    DevRequest* hreq = B.host_requests.as<DevRequest>();
    RenderParams P;
    std::memset(&P, 0, sizeof(P));
    bind_pool(P, B);
    P.mode = 0;
    P.samples = B.samples.as<float4>();
    P.reqs = B.requests.as<DevRequest>();
    // (a resident pass counts invalid samples among its counters)
    unsigned long long* d_invalid = resident ? &P.cnt->stat_invalid : B.invalid.as<unsigned long long>();
    double kms[4] = {0, 0, 0, 0};
    int64_t launches = 0, iters = 0;
    RenderCounters acc;
    std::memset(&acc, 0, sizeof(acc));
    DL_CUDA(cudaEventRecord(ctx->ev0, st));
    if (!resident) DL_CUDA(cudaMemsetAsync(d_invalid, 0, sizeof(unsigned long long), st));
    std::vector<int> active(n), ns(n);
    for (;;) {
        int na = 0;
        unsigned long long first = 0;
        for (int r = 0; r < n; r++) {
            if (done[r] >= items[r].opts.spp) continue;
            const unsigned long long npix = (unsigned long long)items[r].cam.w * items[r].cam.h;
            ns[na] = std::min(slice[r], items[r].opts.spp - done[r]);
            DevRequest R = make_request(items[r].scene, items[r].opts);
            R.sc.cam = items[r].cam;
            R.pid_first = first;
            R.spp_offset = items[r].opts.spp_offset + done[r];
            hreq[na] = R;
            active[na] = r;
            first += npix * (unsigned long long)ns[na];
            na++;
        }
        if (na == 0) break;
        // the pass's request table; the copy is ordered before the pass's kernels
        DL_CUDA(cudaMemcpyAsync(B.requests.ptr, hreq, sizeof(DevRequest) * na, cudaMemcpyHostToDevice, st));
        P.num_reqs = na;
        if (resident) {   // (one pass: every request's samples fit the buffer)
            P.total = first;
            DL_CUDA(cudaMemsetAsync(P.cnt, 0, sizeof(RenderCounters), st));
            resident_launch(ctx, P, true, st);
            launches = iters = 1;
        } else {
            run_wavefront(ctx, P, cap, true, count_traversal, kms, launches, iters, acc, first, 0, 1u << 24,
                          may_finish(ctx, requested, count_traversal));
        }
        for (int a = 0; a < na; a++) {
            const int r = active[a];
            const DevCamera& cam = items[r].cam;
            FilmParams F = film_params(cam, hreq[a], items[r].opts.filter, items[r].d_film,
                                       P.samples + hreq[a].pid_first, d_invalid);
            F.nspp = ns[a];
            F.s_first = hreq[a].spp_offset;
            F.accumulate = done[r] > 0;
            film_gather(F, ctx->num_sms, st);
            launches += 1;
            done[r] += ns[a];
        }
        // (host_requests is rewritten next pass, after the wavefront's wait)
        if (resident) break;
    }
    end_render(ctx, resident, P, d_invalid, results, acc);
    finish_stats(ctx, acc, acc.stat_invalid, iters, launches, kms);
}

// Li of explicit paths with every piece of path state in caller-provided
// device memory (`pool`, laid out below) and no allocation of any kind: no
// cudaMalloc, no pinned staging (the counters are read back into a stack
// copy), no graph.  Used by the allocation-free entry point.
constexpr size_t kCounterBytes = (sizeof(RenderCounters) + 255) / 256 * 256;
size_t fixed_pool_bytes(int64_t slots) { return kSlotBytes * (size_t)slots + kCounterBytes; }

// Failures throw dl::Error with the status and message that run_wavefront
// gives for the same condition.
void render_li_fixed(dl_scene* S, const dl_render_opts& o, void* pool, int64_t slots, int64_t li_n,
                     const int* d_xys, float* d_L, float* d_pos) {
    dl_context* ctx = S->ctx;
    cudaStream_t st = ctx->stream;
    RenderParams P;
    std::memset(&P, 0, sizeof(P));
    P.r0 = make_request(S, o);
    P.mode = 1;
    P.capacity = (int)slots;
    size_t c = (size_t)slots;
    char* b = static_cast<char*>(pool);
    P.cnt = reinterpret_cast<RenderCounters*>(b);
    b += kCounterBytes;
    P.rec = reinterpret_cast<SlotRec*>(b); b += 128 * c;
    float4** f4[] = {&P.sh_o, &P.sh_d, &P.sh_c};
    for (float4** f : f4) {
        *f = reinterpret_cast<float4*>(b);
        b += 16 * c;
    }
    P.pos = reinterpret_cast<float2*>(b); b += 8 * c;
    int** iq[] = {&P.ext_q[0], &P.ext_q[1], &P.mat_q[0], &P.mat_q[1], &P.mat_q[2], &P.mat_q[3], &P.mat_q[4],
                  &P.mat_q[5]};
    for (int** q : iq) {
        *q = reinterpret_cast<int*>(b);
        b += 4 * c;
    }
    P.xys = d_xys;
    P.li_L = d_L;
    P.li_pos = d_pos;
    int64_t cap = std::min<int64_t>(slots, ((li_n + 31) / 32) * 32);
    const int sms = ctx->num_sms > 0 ? ctx->num_sms : 152;
    DL_CUDA(cudaMemsetAsync(P.cnt, 0, sizeof(RenderCounters), st));
    // pass values from the stack (a pageable copy: staged before it returns)
    PassValues pv;
    pv.total = (unsigned long long)li_n;
    pv.spp_offset = 0;
    pv.keep = 1u << 24;
    pv.recs = nullptr;
    DL_CUDA(cudaMemcpyAsync(&P.cnt->pass_total, &pv, sizeof(pv), cudaMemcpyHostToDevice, st));
    k_init<false><<<sms * 16, 128, 0, st>>>(P, (int)cap);
    RenderCounters hc;
    int64_t iters = 0;
    const TuneParams tp;  // default launch shape
    for (;;) {
        for (int k = 0; k < kGraphIterations; k++)
            launch_iteration<false>(P, k & 1, st, sms, tp, false, nullptr, nullptr);
        iters += kGraphIterations;
        DL_CUDA(cudaGetLastError());
        DL_CUDA(cudaMemcpyAsync(&hc, P.cnt, sizeof(RenderCounters), cudaMemcpyDeviceToHost, st));
        DL_CUDA(cudaStreamSynchronize(st));
        if (hc.err & kErrBounds) throw Error(DL_ERR_QUEUE_OVERFLOW, kBoundsMessage);
        if (hc.err & kErrTensorWait) throw Error(DL_ERR_TIMEOUT, "tensor-core wait timed out in a guided kernel");
        if (hc.err) throw Error(DL_ERR_QUEUE_OVERFLOW, "traversal stack overflow");
        if (hc.ext[0] == 0 && hc.shadow[0] == 0 && hc.next_path >= (unsigned long long)li_n) break;
        if (iters > 1000000) throw Error(DL_ERR_TIMEOUT, "render did not converge");
    }
}

void resolve_film(dl_scene* S, const float* d_film, int filter, float* d_rgb) {
    resolve_film_cam(S->dev.cam, S->ctx->stream, d_film, filter, d_rgb);
}

void resolve_film_cam(const DevCamera& cam, cudaStream_t st, const float* d_film, int filter, float* d_rgb) {
    int b = filter == DL_FILTER_BOX ? 0 : 2;
    int n = cam.w * cam.h;
    k_resolve<<<(n + 255) / 256, 256, 0, st>>>(reinterpret_cast<const float4*>(d_film),
                                                         cam.w + 2 * b, b, cam.w, cam.h, d_rgb);
    DL_CUDA(cudaGetLastError());
}

}  // namespace dl

namespace dl {

// ------------------------------------------------- rays through k_traverse
// Ray batches through the renderer's own traversal kernels, the exact
// template instances a single-scene render launches (k_traverse<false,
// false, false> for closest hits, k_traverse<false, true, false> for shadow
// rays) with the context's launch shape, so that ray-level parity tests
// exercise the kernels dl_render runs.  Each ray gets a path slot: its ray
// record (closest hit) or its shadow-queue entry with a unit contribution
// aimed at sample i (any hit), in queue order 0..n-1.

__global__ void k_wavefront_rays_setup(RenderParams P, const float4* __restrict__ rays, int n, int any) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float4 o = rays[2 * i], d = rays[2 * i + 1];
        if (any) {
            P.sh_o[i] = make_float4(o.x, o.y, o.z, __int_as_float(0));
            P.sh_d[i] = d;
            P.sh_c[i] = make_float4(1.f, 1.f, 1.f, __int_as_float(-1 - i));
            P.li_L[3 * i] = 0.f;
            P.li_L[3 * i + 1] = 0.f;
            P.li_L[3 * i + 2] = 0.f;
        } else {
            RayRec r;
            r.o = make_float4(o.x, o.y, o.z, __int_as_float(0));
            r.d = d;
            P.rec[i].ray = r;
            P.ext_q[0][i] = i;
        }
    }
}

// hits (n x float4: t, u, v, original triangle id bits, -1 = miss) from the
// hit records; occluded flags from the delivered unit contributions.
__global__ void k_wavefront_rays_out(RenderParams P, int n, int any, float4* __restrict__ hits,
                                     uint8_t* __restrict__ occ) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (any) {
            occ[i] = P.li_L[3 * i] == 0.f ? 1 : 0;
        } else {
            const float4 h = P.rec[i].hit.h;
            const int tri = __float_as_int(h.w);
            const int prim = tri >= 0 ? __float_as_int(__ldg(P.r0.sc.tris + 3 * tri).w) : -1;
            hits[i] = make_float4(tri >= 0 ? h.x : 0.f, tri >= 0 ? h.y : 0.f, tri >= 0 ? h.z : 0.f,
                                  __int_as_float(prim));
        }
    }
}

size_t wavefront_rays_bytes(int64_t n) {
    return kCounterBytes + 128 * (size_t)n + 3 * 16 * (size_t)n + 12 * (size_t)n +
           4 * (size_t)n * (2 + kNumMaterialTypes + 1);
}

// d_rays: n x 8 floats (o, tmin, d, tmax) with tmin = kRayEps for every ray
// (the renderer's constant ray start); `work` holds wavefront_rays_bytes(n).
void trace_wavefront_launch(dl_scene* S, bool any, const float* d_rays, int64_t n, float* d_hits, uint8_t* d_occ,
                            void* work) {
    dl_context* ctx = S->ctx;
    cudaStream_t st = ctx->stream;
    if (n == 0) return;
    RenderParams P;
    std::memset(&P, 0, sizeof(P));
    dl_render_opts o;
    std::memset(&o, 0, sizeof(o));
    P.r0 = make_request(S, o);
    P.mode = 1;
    P.capacity = (int)n;
    char* b = static_cast<char*>(work);
    P.cnt = reinterpret_cast<RenderCounters*>(b);
    b += kCounterBytes;
    P.rec = reinterpret_cast<SlotRec*>(b);
    b += 128 * (size_t)n;
    float4** f4[] = {&P.sh_o, &P.sh_d, &P.sh_c};
    for (float4** f : f4) {
        *f = reinterpret_cast<float4*>(b);
        b += 16 * (size_t)n;
    }
    P.li_L = reinterpret_cast<float*>(b);
    b += 12 * (size_t)n;
    int** iq[] = {&P.ext_q[0], &P.ext_q[1], &P.mat_q[0], &P.mat_q[1], &P.mat_q[2], &P.mat_q[3], &P.mat_q[4],
                  &P.mat_q[5]};
    for (int** q : iq) {
        *q = reinterpret_cast<int*>(b);
        b += 4 * (size_t)n;
    }
    DL_CUDA(cudaMemsetAsync(P.cnt, 0, sizeof(RenderCounters), st));
    const int ni = (int)n;
    const unsigned long long total = (unsigned long long)n;  // path indices of the shadow targets: 0..n-1
    DL_CUDA(cudaMemcpyAsync(any ? &P.cnt->shadow[0] : &P.cnt->ext[0], &ni, sizeof(int), cudaMemcpyHostToDevice, st));
    DL_CUDA(cudaMemcpyAsync(&P.cnt->pass_total, &total, sizeof(total), cudaMemcpyHostToDevice, st));
    const int sms = ctx->num_sms > 0 ? ctx->num_sms : 152;
    const int g = (int)std::min<int64_t>((n + 127) / 128, (int64_t)sms * 16);
    k_wavefront_rays_setup<<<g, 128, 0, st>>>(P, reinterpret_cast<const float4*>(d_rays), ni, any ? 1 : 0);
    const int tb = sms * ctx->tune.trav_ctas_per_sm;
    if (any) k_traverse<false, true, false><<<tb, 128, 0, st>>>(P, 0);
    else k_traverse<false, false, false><<<tb, 128, 0, st>>>(P, 0);
    k_wavefront_rays_out<<<g, 128, 0, st>>>(P, ni, any ? 1 : 0, reinterpret_cast<float4*>(d_hits), d_occ);
    DL_CUDA(cudaGetLastError());
    unsigned int err = 0;
    DL_CUDA(cudaMemcpyAsync(&err, &P.cnt->err, sizeof(err), cudaMemcpyDeviceToHost, st));
    DL_CUDA(cudaStreamSynchronize(st));
    if (err & kErrBounds) throw Error(DL_ERR_QUEUE_OVERFLOW, kBoundsMessage);
    if (err) throw Error(DL_ERR_QUEUE_OVERFLOW, "traversal stack overflow");
}

}  // namespace dl

namespace dl {

// ------------------------------------------------------- emitter queries
// Scene::sampleEmitterDirection without the visibility test, at given
// points, normals and 2D samples, by the device function the material
// kernels run (an envmap pick draws its three numbers from a pcg32 seeded
// with the query index); `light` receives the picked emitter.
__global__ void __launch_bounds__(128) k_emitter_query(DevRequest R, int n, const float* __restrict__ pts,
                                                        const float* __restrict__ nrm, const float* __restrict__ smp,
                                                        float* __restrict__ out, int* __restrict__ light) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float3 p = f3(pts[3 * i], pts[3 * i + 1], pts[3 * i + 2]);
        const float3 nn = f3(nrm[3 * i], nrm[3 * i + 1], nrm[3 * i + 2]);
        const float2 s = make_float2(smp[2 * i], smp[2 * i + 1]);
        float sx = s.x;
        light[i] = R.sc.num_lights > 0 ? pick_light(R, sx) : -1;
        Pcg32 g;
        g.seed((unsigned long long)i, 7ull);
        float3 d;
        float dist, pdf;
        bool delta;
        const float3 spec = sample_emitter(R, p, nn, s, g, d, dist, pdf, delta);
        float* o = out + 8 * (size_t)i;
        o[0] = d.x;
        o[1] = d.y;
        o[2] = d.z;
        o[3] = dist;
        o[4] = pdf;
        o[5] = spec.x;
        o[6] = spec.y;
        o[7] = spec.z;
    }
}

void emitter_query(dl_scene* S, uint32_t flags, int64_t n, const float* pts, const float* nrm, const float* smp,
                   float* d, float* dist, float* pdf, float* spec, int32_t* light) {
    if (n == 0) return;
    dl_context* ctx = S->ctx;
    cudaStream_t st = ctx->stream;
    dl_render_opts o;
    std::memset(&o, 0, sizeof(o));
    o.flags = flags;
    const DevRequest R = make_request(S, o);
    const size_t f = sizeof(float) * (size_t)n;
    DevBuf buf;
    buf.ensure(f * (3 + 3 + 2 + 8 + 1));
    float* d_pts = buf.as<float>();
    float* d_nrm = d_pts + 3 * n;
    float* d_smp = d_nrm + 3 * n;
    float* d_out = d_smp + 2 * n;
    int* d_light = reinterpret_cast<int*>(d_out + 8 * n);
    DL_CUDA(cudaMemcpyAsync(d_pts, pts, 3 * f, cudaMemcpyHostToDevice, st));
    DL_CUDA(cudaMemcpyAsync(d_nrm, nrm, 3 * f, cudaMemcpyHostToDevice, st));
    DL_CUDA(cudaMemcpyAsync(d_smp, smp, 2 * f, cudaMemcpyHostToDevice, st));
    const int sms = ctx->num_sms > 0 ? ctx->num_sms : 152;
    const int g = (int)std::max<int64_t>(1, std::min<int64_t>((n + 127) / 128, (int64_t)sms * 8));
    k_emitter_query<<<g, 128, 0, st>>>(R, (int)n, d_pts, d_nrm, d_smp, d_out, d_light);
    DL_CUDA(cudaGetLastError());
    std::vector<float> h((size_t)n * 8);
    DL_CUDA(cudaMemcpyAsync(h.data(), d_out, 8 * f, cudaMemcpyDeviceToHost, st));
    DL_CUDA(cudaMemcpyAsync(light, d_light, f, cudaMemcpyDeviceToHost, st));
    DL_CUDA(cudaStreamSynchronize(st));
    for (int64_t i = 0; i < n; i++) {
        const float* q = &h[8 * (size_t)i];
        for (int k = 0; k < 3; k++) {
            d[3 * i + k] = q[k];
            spec[3 * i + k] = q[5 + k];
        }
        dist[i] = q[3];
        pdf[i] = q[4];
    }
}

}  // namespace dl
