// Ray-batch traversal kernels behind dl_trace_closest / dl_trace_any
// (the reference's Accel::rayIntersect, include/tracer/accel.h:52, over the
// OCTree of src/tracer/accel/octree.cpp:53-133).
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>

#include "device.cuh"
#include "internal.h"
#include "scene.h"

namespace dl {

constexpr int kRayThreads = 128;
constexpr int kRayStack = 8;      // top traversal-stack entries of a thread in shared memory
constexpr int kRayDone = INT_MIN; // traversal state: ray finished (below every leaf reference)

// One word of scratch for the errors, one for the rays handed out.
struct RayScratch {
    unsigned int err;
    unsigned int pad;
    unsigned long long next;
};

// rays: n x 8 floats (ox, oy, oz, tmin, dx, dy, dz, tmax) as 2 float4.
// kAny = false: out is n x float4 (t, u, v, original triangle id bits; -1 =
// miss); kAny = true: n bytes, 1 = occluded.
//
// A warp takes 32 rays at a time and hands them to its lanes as they free up;
// each lane descends to a leaf, then tests the leaf's triangles.  Bounded by
// the latency of dependent node fetches while the rays are no more than the
// resident threads (one thread a ray), then by the L1's wavefronts, as the
// renderer's traversal.  Material-sphere scene, whole calls on host arrays used
// before | on new ones, against one thread a ray, copies and hits split on the
// host: dl_trace_closest of 1000 rays 73 -> 62 us | 118 -> 93, 20,000 136 -> 76
// | 195 -> 110, 200,003 568 -> 131 | 742 -> 211, 2 M 4.97 -> 0.57 ms | 6.20 ->
// 1.43; dl_trace_any of 200,003 139 -> 102 us | 255 -> 141, 2 M 669 -> 399 |
// 758 -> 475.
template <bool kAny>
__global__ void __launch_bounds__(kRayThreads) k_trace_rays(DevScene sc, const float4* __restrict__ rays, int64_t n,
                                                             void* __restrict__ out, RayScratch* scratch) {
    __shared__ int s_stack[kRayStack][kRayThreads];
    int stack[kStackSize - kRayStack];
    int* const my_stack = &s_stack[0][threadIdx.x];
    const int lane = threadIdx.x & 31;
    uint32_t err = 0;
    bool has = false, exhausted = false;
    int64_t idx = 0;
    int node = kRayDone, sp = 0, hit = -1;
    float3 o = f3(0.f, 0.f, 0.f), d = o;
    float tmin = 0.f, tmax = 0.f, ht = 0.f, hu = 0.f, hv = 0.f;
    RayBox rb;
    rb.idir = o;
    rb.ood = o;
    auto push = [&](int v) {
        if (sp < kRayStack) my_stack[sp * kRayThreads] = v;
        else stack[sp - kRayStack] = v;
        sp++;
    };
    auto pop = [&]() -> int {
        --sp;
        return sp < kRayStack ? my_stack[sp * kRayThreads] : stack[sp - kRayStack];
    };
    int64_t c_next = 0, c_end = 0;  // the warp's rays not yet handed out
    for (;;) {
        const bool need = !has && !exhausted;
        const unsigned m = __ballot_sync(0xffffffffu, need);
        if (m) {
            const int k = __popc(m), rank = __popc(m & ((1u << lane) - 1u)), avail = (int)(c_end - c_next);
            int64_t mine;
            if (k > avail) {
                unsigned long long base = 0;
                if (lane == 0) base = atomicAdd(&scratch->next, 32ull);
                base = __shfl_sync(0xffffffffu, base, 0);
                mine = rank < avail ? c_next + rank : (int64_t)base + (rank - avail);
                c_next = (int64_t)base + (k - avail);
                c_end = (int64_t)base + 32;
            } else {
                mine = c_next + rank;
                c_next += k;
            }
            if (need) {
                if (mine < n) {
                    idx = mine;
                    const float4 ro = __ldg(rays + 2 * idx), rd = __ldg(rays + 2 * idx + 1);
                    o = xyz(ro);
                    d = xyz(rd);
                    tmin = ro.w;
                    tmax = rd.w;
                    rb = make_raybox(o, d);
                    node = sc.num_tris > 0 ? 0 : kRayDone;
                    sp = 0;
                    hit = -1;
                    has = true;
                } else {
                    exhausted = true;
                }
            }
        }
        if (__ballot_sync(0xffffffffu, has) == 0) break;
        if (has) {
            while (node >= 0) {
#ifdef DL_CHECKS
                if (node >= sc.num_nodes) {  // bounds-checked build: bit 4 of the error word
                    err |= 4u;
                    node = kRayDone;
                    break;
                }
#endif
                const float4* np = sc.nodes + 4 * node;
                float4 a, b, c, dd;
                ld_nc_256(np, a, b);
                ld_nc_256(np + 2, c, dd);
                const int2 ch = make_int2(__float_as_int(dd.x), __float_as_int(dd.y));
                bool h0, h1;
                float t0, t1;
                box2(rb, tmin, tmax, a, b, c, h0, h1, t0, t1);
                if (h0 && h1) {   // (both slots always hold a child: see bvh.h)
                    int near = ch.x, far = ch.y;
                    if (t1 < t0) { near = ch.y; far = ch.x; }
                    if (sp < kStackSize) push(far); else err |= 1u;
                    node = near;
                } else if (h0) {
                    node = ch.x;
                } else if (h1) {
                    node = ch.y;
                } else {
                    node = sp > 0 ? pop() : kRayDone;
                }
            }
            if (node != kRayDone) {
                const int ref = ~node;
                const int first = ref >> 4;
                int count = (ref & 15) + 1;
#ifdef DL_CHECKS
                if (first < 0 || first + count > sc.num_tris) {
                    err |= 4u;
                    count = 0;
                }
#endif
                for (int k = 0; k < count; k++) {
                    const float4* tp = sc.tris + 3 * (first + k);
                    const float4 p0 = __ldg(tp), p1 = __ldg(tp + 1), p2 = __ldg(tp + 2);
                    float t, u, v;
                    if (intersect_tri(xyz(p0), xyz(p1), xyz(p2), o, d, tmin, tmax, t, u, v)) {
                        hit = __float_as_int(p0.w);  // the triangle's original id
                        if (kAny) break;
                        tmax = t;
                        ht = t;
                        hu = u;
                        hv = v;
                    }
                }
                node = (kAny && hit >= 0) || sp == 0 ? kRayDone : pop();
            }
            if (node == kRayDone) {
                if (kAny)
                    static_cast<uint8_t*>(out)[idx] = hit >= 0 ? 1 : 0;
                else
                    static_cast<float4*>(out)[idx] =
                        hit >= 0 ? make_float4(ht, hu, hv, __int_as_float(hit))
                                 : make_float4(0.f, 0.f, 0.f, __int_as_float(-1));
                has = false;
            }
        }
    }
    if (err) atomicOr(&scratch->err, err);
}

// hits (n x float4) into the caller's four arrays: each warp writes 32
// consecutive values of an array (split on the host, 200,003 hits took 420 us).
// A caller that wants one of them may give one array for several: t, u, v and
// prim (as bits, one type throughout) are stored in this order.
__global__ void __launch_bounds__(256) k_split_hits(const float4* __restrict__ hits, int64_t n, float* prim, float* t,
                                                     float* u, float* v) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const float4 h = hits[i];
        t[i] = h.x;
        u[i] = h.y;
        v[i] = h.z;
        prim[i] = h.w;
    }
}

__global__ void __launch_bounds__(256) k_copy_bytes(const uint8_t* __restrict__ from, int64_t n, uint8_t* to) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        to[i] = from[i];
}

static int ray_grid(const dl_context* ctx, int64_t n, int threads, int per_sm) {
    return (int)std::max<int64_t>(1, std::min<int64_t>((n + threads - 1) / threads, (int64_t)ctx->num_sms * per_sm));
}

template <bool kAny>
static void launch_rays(dl_scene* S, const float* d_rays, int64_t n, void* d_out, void* scratch) {
    cudaStream_t st = S->ctx->stream;
    DL_CUDA(cudaMemsetAsync(scratch, 0, sizeof(RayScratch), st));
    if (n == 0) return;
    k_trace_rays<kAny><<<ray_grid(S->ctx, n, kRayThreads, 16), kRayThreads, 0, st>>>(
        S->dev, reinterpret_cast<const float4*>(d_rays), n, d_out, static_cast<RayScratch*>(scratch));
    DL_CUDA(cudaGetLastError());
}

// Launches on the context stream; `scratch` (16 bytes) holds the error word
// first.
void trace_closest_launch(dl_scene* S, const float* d_rays, int64_t n, float* d_hits, void* scratch) {
    launch_rays<false>(S, d_rays, n, d_hits, scratch);
}
void trace_any_launch(dl_scene* S, const float* d_rays, int64_t n, uint8_t* d_occ, void* scratch) {
    launch_rays<true>(S, d_rays, n, d_occ, scratch);
}

void split_hits_launch(const dl_context* ctx, const float* d_hits, int64_t n, int32_t* prim, float* t, float* u,
                       float* v) {
    k_split_hits<<<ray_grid(ctx, n, 256, 8), 256, 0, ctx->stream>>>(reinterpret_cast<const float4*>(d_hits), n,
                                                                   reinterpret_cast<float*>(prim), t, u, v);
    DL_CUDA(cudaGetLastError());
}
void copy_bytes_launch(const dl_context* ctx, const uint8_t* from, int64_t n, uint8_t* to) {
    k_copy_bytes<<<ray_grid(ctx, n, 256, 8), 256, 0, ctx->stream>>>(from, n, to);
    DL_CUDA(cudaGetLastError());
}

}  // namespace dl
