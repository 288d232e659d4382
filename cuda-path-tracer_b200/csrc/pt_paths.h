// pt_paths.h — one persistent kernel that carries paths from their first camera ray to their last
// bounce: the four-wide walk with its node and leaf phases (persistent_walk4_spec), and between
// rounds of it the shading of the lanes whose walk has ended.
//
// A wavefront renderer runs extend, shade and shadow as kernels over queues, so every bounce of the
// whole image waits for the slowest ray of the bounce before (a third of an extend launch's time at
// 300,000 rays), and the last few paths need a kernel of their own, whose warps wait for their
// slowest lane at every bounce.  Here a lane whose walk has ended waits only until fewer than
// kPathsActive lanes of its warp still walk; then the lanes that have ended shade together and walk
// on: the shadow ray of the bounce first, then the extension ray.
//
// Samples of one pixel must run in order (they consume the pixel's PCG stream), and a pixel behind
// glass takes many times the average: all pixels therefore advance together, a sample at a time.
// Work item k is one sample of pixel k mod pixels.  A lane that draws an item adds one to the pixel's
// claim count; if the count was zero it runs the sample, otherwise the lane that is running the pixel
// finds the claim when its sample ends and runs the next sample itself.  No lane waits for another,
// and a heavy pixel runs without a break from the first pass on.
//
// What it measured (kernel time, 1M triangles, bounce limit 8, 16 spp; wavefront and pair tail before):
// 960x600 15.1 -> 9.5 ms, 1920x1080 30.4 -> 27.1; 65,000 triangles at 960x600 5.4 -> 2.9.  Where it loses, inside rooms
// and on large images, pt_forms.h says.
// Lanes that shade together cost one pass through 60 KB of shading code whether 8 or 28 of them do, so
// a warp waits until fewer than kPathsActive still walk (time with 2, 5, 8 and 16 over that with 4: 1M triangles
// 960x600 1.01, 1.00, 1.04, 1.12, 1920x1080 1.07, 0.99, 0.99, 1.05; 65,000 at 960x600 0.95, 1.04, 1.09, 1.12; six-job
// batch 0.98, 1.01, 1.04, 1.06).  Five blocks of 128 per SM, since records became the lanes' own and stay in L1, although
// 96 registers then spill (bytes stored and loaded per thread: render_paths_kernel 56 and 52, batch_paths 100 and 92,
// frame_kernel 190 and 196): with four, which spill 48 in frame_kernel alone, 1920x1080 takes 10 % longer, the batch 5,
// 960x600 2, and 640x400 13 % less; with six 960x600 takes 7 % longer, 640x400 17, the batch 8.  Shading 32 at a time
// from rings of 64 paths per warp filled the lanes better (8.2 ms until the items ran out, records in the pixels' slots)
// but doubled the time a heavy pixel waits for each bounce (12.6 ms in all).
#pragma once

#include "pt_forms.h"
#include "pt_wavefront.h"

#ifdef __CUDACC__
namespace ptb {

constexpr int kProbeBlock = 8;        // few paths to a warp: a probe lasts as long as its slowest warp
// Camera path `i` of the probe of a view (pt_forms.h): how many surfaces other than lights it meets in two walks,
// every one of them taken as diffuse.
__device__ inline uint32_t probe_path(const DeviceScene &scene, const pt_camera &camera, int32_t root, int32_t i) {
    Pcg rng;
    rng.seed(1, uint64_t(i));
    PathState s;
    camera_path(camera, kProbeSide, kProbeSide, i, rng, s);
    uint32_t met = 0;
    for (; met < 2; met++) {
        const pt_ray r = path_ray(s);
        HitInfo h;
        uint32_t boxes = 0, prims = 0;
        int error = 0;
        if (!traverse4_rt(scene, r, 0.001f, FLT_MAX, kTieLastLeaf, false, h, boxes, prims, error, root) || error) break;
        Surface o;
        surface_hit(scene, r, h, o);
        if (scene.materials[o.material].type == PT_LIGHT) break;
        const f3 in = mk(r.direction), d = cosine_direction(dot(o.normal, in) > 0 ? -o.normal : o.normal, rng);
        s.ox = o.p.x; s.oy = o.p.y; s.oz = o.p.z;
        s.dx = d.x; s.dy = d.y; s.dz = d.z;
    }
    return met;
}

constexpr int kPathsBlock = 128, kPathsBlocksPerSm = 5;   // 96 registers, with spills (see above)
constexpr int kPathsActive = 4;   // lanes of a warp still walking below which the others shade

// The lane's next ray: path and shadow records begin with origin and (shadow) tmax, then the direction.
template <class Path, class Shadow>
__device__ inline void lane_ray(const Path &path, const Shadow &shadow_ray, bool shadow, pt_ray &r, float &tmax) {
    const float4 *rec = shadow ? reinterpret_cast<const float4 *>(&shadow_ray) : reinterpret_cast<const float4 *>(&path);
    const float4 o = rec[0], d = rec[1];
    r.origin = pt_vec3{o.x, o.y, o.z};
    r.direction = pt_vec3{d.x, d.y, d.z};
    if (shadow) tmax = o.w;
}

// What a shaded bounce asks for next.
struct NextWalk {
    bool live = false;          // the sample goes on with the path's extension ray
    bool shadow = false;        // after its shadow ray
};

// Ops, the lane's path (its records are the lane's own; only the pixel's stream and sum outlive a sample):
//   bool claim(item, root)          starts work item `item` if this lane is to run it
//   bool again()                    the sample has ended: start the pixel's next claimed one
//   void shade(hit, next)           one bounce
//   void ray(shadow, r, tmax)       the path's extension or shadow ray
//   void unblocked()                its pending shadow contribution counts
//   void hand_over()                leaves the path, its extension ray not yet walked, to a later kernel
// All lanes of the warp call this together; the block provides kSharedStack4 * blockDim.x int2 of
// dynamic shared memory.
template <class Ops>
__device__ inline void persistent_paths4(const DeviceScene &s, Ops &ops, unsigned long long items, unsigned long long *next,
                                         int tie, unsigned long long &rays, int32_t *error_flag) {
    extern __shared__ int32_t shared_stack[];
    int2 *my_stack = reinterpret_cast<int2 *>(shared_stack) + threadIdx.x;
    const int stride = blockDim.x;
    int2 spill[kStack4 - kSharedStack4];
    const unsigned full = 0xffffffffu;
    const unsigned lane = threadIdx.x & 31;
    constexpr int32_t kNone = kEmptyChild;
    constexpr float tmin = 0.001f;
    bool path = false;              // the lane runs a sample
    bool walking = false, any = false, drained = false, error = false;
    int32_t root = 0;
    pt_ray r{};
    RayBox4 rb{};
    float dl = 0, limit = 0;
    HitInfo hit;
    hit.slot = -1; hit.t = 0; hit.u = 0; hit.v = 0;
    uint32_t boxes = 0, prims = 0;
    int32_t cur = kNone, leaf = kNone, leaf2 = kNone;
    int sp = 0;
    auto pop = [&]() -> int32_t {
        while (sp > 0) {
            sp--;
            int2 e = sp < kSharedStack4 ? my_stack[sp * stride] : spill[sp - kSharedStack4];
            if (__int_as_float(e.y) < limit) return e.x;
        }
        return kNone;
    };
    for (;;) {
        // ---- lanes whose walk has ended go on with their path
        if (path && !walking) {
            if (error) *error_flag = 1;
            if (any) {
                if (!error && hit.slot < 0) ops.unblocked();
                any = false;
            } else {
                PathHit h;
                h.t = hit.t; h.u = hit.u; h.v = hit.v; h.slot = error ? -2 : hit.slot;
                NextWalk n;
                ops.shade(h, n);
                any = n.shadow;
                if (!n.live && !ops.again()) path = false;
            }
        }
        // ---- lanes without a path draw work items
        while (!drained && __any_sync(full, !path)) {
            const unsigned m = __ballot_sync(full, !path);
            const int leader = __ffs(m) - 1;
            unsigned long long base = 0;
            if ((int)lane == leader) base = atomicAdd(next, (unsigned long long)__popc(m));
            base = __shfl_sync(full, base, leader);
            if (!path) {
                const unsigned long long k = base + __popc(m & ((1u << lane) - 1u));
                path = k < items && ops.claim(k, root);
                any = false;
            }
            if (base + __popc(m) >= items) drained = true;
        }
        // ---- with no items left, paths go to the tail kernel at their next extension ray
        if (drained && path && !walking && !any) { ops.hand_over(); path = false; }
        if (path && !walking) {
            float tmax = FLT_MAX;
            ops.ray(any, r, tmax);
            rays++;   // each query counts once, as trace_color counts it (transport.h:177)
            rb = ray_box4(r);
            dl = length(mk(r.direction));
            limit = tmax;
            hit.slot = -1; hit.t = 0; hit.u = 0; hit.v = 0;
            sp = 0; error = false;
            cur = (s.empty || s.node_count == 0 || root < 0) ? kNone : root;
            leaf = kNone; leaf2 = kNone;
            walking = true;
        }
        const int live = __popc(__ballot_sync(full, walking));
        if (!live) break;
        // with no items left, few lanes do not wait for each other
        const int threshold = drained ? max(1, live / 2) : kPathsActive;
        for (;;) {
            bool end = false;
            // ---- node phase (see persistent_walk4_spec)
            for (;;) {
                bool need_pop = false;
                if (walking && cur >= 0 && cur != kNone && !error) {
                    int32_t ref[4];
                    float dist[4];
                    int hits = node4_children(s, cur, rb, tmin, limit, ref, dist, boxes);
                    if (hits) {
                        if (sp + hits - 1 > kStack4) { error = true; cur = kNone; leaf = kNone; leaf2 = kNone; }
                        else {
#pragma unroll
                            for (int k = 3; k >= 1; k--) {
                                if (k < hits) {
                                    int2 e = make_int2(ref[k], __float_as_int(dist[k]));
                                    if (sp < kSharedStack4) my_stack[sp * stride] = e; else spill[sp - kSharedStack4] = e;
                                    sp++;
                                }
                            }
                            cur = ref[0];
                        }
                    } else {
                        need_pop = true;
                    }
                }
                if (walking && cur < 0) {
                    if (leaf == kNone) { leaf = cur; need_pop = true; }
                    else if (leaf2 == kNone) { leaf2 = cur; need_pop = true; }
                }
                if (need_pop) cur = pop();
                const bool searching = walking && leaf == kNone && cur != kNone;
                const unsigned sm = __ballot_sync(full, searching);
                if (!sm) break;
                if (__popc(sm) < 4 && __any_sync(full, walking && leaf != kNone)) break;
            }
            // ---- leaf phase
            if (walking && leaf != kNone) {
                const int32_t v1 = ~leaf, f1 = v1 >> 3, c1 = (v1 & 7) + 1;
                int32_t f2 = 0, c2 = 0;
                if (leaf2 != kNone) { const int32_t v2 = ~leaf2; f2 = v2 >> 3; c2 = (v2 & 7) + 1; }
                for (int32_t j = 0; j < c1 + c2; j++) {
                    const int32_t at = j < c1 ? f1 + j : f2 + (j - c1);
                    if (test_leaf_rt(s, at, r, dl, tmin, limit, tie, any, hit, prims) && any) { end = true; break; }
                }
                leaf = kNone; leaf2 = kNone;
            }
            if (walking && (end || error || (leaf == kNone && cur == kNone))) walking = false;
            if (__popc(__ballot_sync(full, walking)) < threshold) break;
        }
    }
}

} // namespace ptb
#endif
