// pt_small.h — walks of scenes with at most kSmallLeaves primitives, held whole in shared memory.
//
// On a tree of a few nodes a warp of unrelated rays visits every node anyway, a few lanes at a
// time: the lanes' tree walks diverge at each step (10 of 32 lanes busy on the 23-primitive
// Cornell box).  Here all lanes of a warp test the same leaf box in the same instruction, reading
// it from shared memory as a broadcast; each lane keeps the boxes it passed as bits of one 32-bit
// word (hence the limit of 32 leaves) and then tests only those primitives, a handful of rounds
// for the whole warp.  The box test is the two-wide walk's (box_hit, the reference's arithmetic):
// boxes nest and the slab arithmetic is monotone, so a leaf whose box passes has ancestors whose
// boxes pass, and the primitives tested are those the tree walk reaches.
#pragma once

#include "pt_traverse.h"

#ifdef __CUDACC__
namespace ptb {

struct SmallScene {                    // in shared memory
    float4 xy[kSmallLeaves];           // box: min x, min y, max x, max y
    float2 z[kSmallLeaves];            // min z, max z
    float4 record[kSmallLeaves][3];    // TriRecord, or SphereRecord in the first two
    int32_t slot[kSmallLeaves];
};

// Fills `sh` with the block's threads; the boxes are widened by `pad` on every side.
__device__ inline void small_load(const DeviceScene &s, SmallScene &sh, float pad) {
    for (int k = threadIdx.x; k < s.small_count; k += blockDim.x) {
        const SmallLeaf leaf = s.small[k];
        sh.xy[k] = make_float4(leaf.lo[0] - pad, leaf.lo[1] - pad, leaf.hi[0] + pad, leaf.hi[1] + pad);
        sh.z[k] = make_float2(leaf.lo[2] - pad, leaf.hi[2] + pad);
        sh.slot[k] = leaf.slot;
        if (leaf.slot < s.tri_slots) {
            const float4 *p = reinterpret_cast<const float4 *>(&s.tris[leaf.slot]);
            for (int j = 0; j < 3; j++) sh.record[k][j] = p[j];
        } else {
            const float4 *p = reinterpret_cast<const float4 *>(&s.spheres[leaf.slot - s.tri_slots]);
            for (int j = 0; j < 2; j++) sh.record[k][j] = p[j];
        }
    }
    __syncthreads();
}

// Closest hit (any = false) or any hit of one ray per lane; true when something was hit.
__device__ __forceinline__ bool small_walk(const DeviceScene &s, const SmallScene &sh, const pt_ray &r, float tmin, float tmax,
                                           int tie, bool any, HitInfo &hit) {
    hit.slot = -1; hit.t = 0; hit.u = 0; hit.v = 0;
    const RayBox rb = ray_box(r);
    const f2x oxy = f2x_make(-rb.ox, -rb.oy), ozz = f2x_make(-rb.oz, -rb.oz);   // a - b and a + (-b) round alike
    const f2x ixy = f2x_make(rb.ix, rb.iy), izz = f2x_make(rb.iz, rb.iz);
    uint32_t passed = 0;
#pragma unroll 4
    for (int k = 0; k < s.small_count; k++) {
        const float4 b = sh.xy[k];
        const float2 z = sh.z[k];
        float ax, ay, az, bx, by, bz;
        f2x_split(f2x_mul(f2x_add(f2x_make(rb.nx ? b.z : b.x, rb.ny ? b.w : b.y), oxy), ixy), ax, ay);
        f2x_split(f2x_mul(f2x_add(f2x_make(rb.nx ? b.x : b.z, rb.ny ? b.y : b.w), oxy), ixy), bx, by);
        f2x_split(f2x_mul(f2x_add(f2x_make(rb.nz ? z.y : z.x, rb.nz ? z.x : z.y), ozz), izz), az, bz);
        const float lo = fmaxf(max3(tmin, ax, ay), az), hi = fminf(min3(tmax, bx, by), bz);
        if (hi > lo) passed |= 1u << k;
    }
    const float dl = length(mk(r.direction));
    float limit = tmax;
    // leaves are in slot order, triangles before spheres: one loop for each kind, so lanes testing
    // different kinds do not alternate
    const int tri_leaves = s.tri_slots < s.small_count ? s.tri_slots : s.small_count;
    const uint32_t tri_mask = tri_leaves < 32 ? (1u << tri_leaves) - 1u : 0xffffffffu;
    uint32_t left = dl > 0 ? passed & tri_mask : 0;   // !(direction_length > 0), flat_intersect.h:14
    while (left) {
        const int k = __ffs(left) - 1;
        left &= left - 1;
        const float4 a = sh.record[k][0], b = sh.record[k][1], c = sh.record[k][2];
        TriRecord tr;
        tr.v0x = a.x; tr.v0y = a.y; tr.v0z = a.z; tr.eps = a.w;
        tr.e1x = b.x; tr.e1y = b.y; tr.e1z = b.z;
        tr.e2x = c.x; tr.e2y = c.y; tr.e2z = c.z;
        float t, u, v;
        if (tri_hit(tr, r, dl, tmin, limit, t, u, v) && accept_hit(s, sh.slot[k], t, u, v, tie, any, limit, hit) && any) return true;
    }
    left = passed & ~tri_mask;
    while (left) {
        const int k = __ffs(left) - 1;
        left &= left - 1;
        const float4 a = sh.record[k][0];
        SphereRecord sp;
        sp.cx = a.x; sp.cy = a.y; sp.cz = a.z; sp.radius = a.w;
        float t;
        if (sphere_hit(sp, r, tmin, limit, t) && accept_hit(s, sh.slot[k], t, 0.0f, 0.0f, tie, any, limit, hit) && any) return true;
    }
    return hit.slot >= 0;
}

} // namespace ptb
#endif
