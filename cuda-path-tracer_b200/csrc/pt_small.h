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

// The boxes are stored once per sign pattern of the ray direction, entered planes first: a lane then
// needs no selects (6 of 20 instructions a box), and the eight patterns of a leaf are 128
// consecutive bytes, so lanes of any mix of patterns read them without bank conflicts (Cornell
// render 2.00 -> 1.87 ms).
struct SmallScene {                    // in shared memory
    ulonglong2 xy[kSmallLeaves][8];    // (near x, near y), (far x, far y) as packed floats
    unsigned long long z[kSmallLeaves][8];   // (near z, far z)
    float4 record[kSmallLeaves][3];    // TriRecord, or SphereRecord in the first two
    int32_t slot[kSmallLeaves];
};

// Fills `sh` with the block's threads; the boxes are widened by `pad` on every side.
__device__ inline void small_load(const DeviceScene &s, SmallScene &sh, float pad) {
    for (int j = threadIdx.x; j < 8 * s.small_count; j += blockDim.x) {
        const SmallLeaf leaf = s.small[j >> 3];
        const float lo[3] = {leaf.lo[0] - pad, leaf.lo[1] - pad, leaf.lo[2] - pad};
        const float hi[3] = {leaf.hi[0] + pad, leaf.hi[1] + pad, leaf.hi[2] + pad};
        const bool nx = j & 1, ny = j & 2, nz = j & 4;
        sh.xy[j >> 3][j & 7] = make_ulonglong2(f2x_make(nx ? hi[0] : lo[0], ny ? hi[1] : lo[1]),
                                               f2x_make(nx ? lo[0] : hi[0], ny ? lo[1] : hi[1]));
        sh.z[j >> 3][j & 7] = f2x_make(nz ? hi[2] : lo[2], nz ? lo[2] : hi[2]);
    }
    for (int k = threadIdx.x; k < s.small_count; k += blockDim.x) {
        const SmallLeaf leaf = s.small[k];
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

// Closest hit (any = false) or any hit of one ray per lane; true when something was hit.  kFar (queries, whose rays
// may start anywhere): the boxes are widened by the rounding of the slab arithmetic as well, eight units in the
// last place of the origin's largest coordinate (2^-21), since far from the scene two planes of a box, padded or
// not, round to the same distance and neighbouring axes to distances in the wrong order.  The primitives' own
// tests decide, so a box too wide costs time only.
template <bool kFar>
__device__ __forceinline__ bool small_walk(const DeviceScene &s, const SmallScene &sh, const pt_ray &r, float tmin, float tmax,
                                           int tie, bool any, HitInfo &hit) {
    hit.slot = -1; hit.t = 0; hit.u = 0; hit.v = 0;
    const RayBox rb = ray_box(r);
    const f2x oxy = f2x_make(-rb.ox, -rb.oy), ozz = f2x_make(-rb.oz, -rb.oz);   // a - b and a + (-b) round alike
    const f2x ixy = f2x_make(rb.ix, rb.iy), izz = f2x_make(rb.iz, rb.iz);
    const int pattern = (rb.nx ? 1 : 0) | (rb.ny ? 2 : 0) | (rb.nz ? 4 : 0);
    f2x out_xy = 0, in_xy = 0, out_in_z = 0;             // how much earlier a ray enters and later it leaves (kFar)
    if constexpr (kFar) {
        const float pad = fmaxf(fmaxf(fabsf(rb.ox), fabsf(rb.oy)), fabsf(rb.oz)) * 0x1p-21f;
        auto reach = [&](float inverse) { return fabsf(inverse) <= FLT_MAX ? pad * fabsf(inverse) : 0.0f; };   // 0: parallel to the slab
        const float x = reach(rb.ix), y = reach(rb.iy), z = reach(rb.iz);
        out_xy = f2x_make(-x, -y); in_xy = f2x_make(x, y); out_in_z = f2x_make(-z, z);
    }
    uint32_t passed = 0;
#pragma unroll 4
    for (int k = 0; k < s.small_count; k++) {
        const ulonglong2 xy = sh.xy[k][pattern];
        float ax, ay, az, bx, by, bz;
        if constexpr (kFar) {
            f2x_split(f2x_fma(f2x_add(xy.x, oxy), ixy, out_xy), ax, ay);
            f2x_split(f2x_fma(f2x_add(xy.y, oxy), ixy, in_xy), bx, by);
            f2x_split(f2x_fma(f2x_add(sh.z[k][pattern], ozz), izz, out_in_z), az, bz);
        } else {
            f2x_split(f2x_mul(f2x_add(xy.x, oxy), ixy), ax, ay);
            f2x_split(f2x_mul(f2x_add(xy.y, oxy), ixy), bx, by);
            f2x_split(f2x_mul(f2x_add(sh.z[k][pattern], ozz), izz), az, bz);
        }
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
