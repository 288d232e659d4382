// pt_shade.h — per-bounce shading of the MIS path tracer (device), same arithmetic as the
// reference's trace_color pieces so a path makes the same decisions and sums the same floats.
//
//   textures         src/renderer/transport.h:87-111
//   scatter          src/renderer/transport.h:113-155
//   light sampling   src/renderer/light_sampling.h:10-73
//   emitter lookup   binary search over the cumulative-area table (scene_lights)
#pragma once

#include <cmath>
#include "pt_traverse.h"

namespace ptb {

// trace_image: nearest texel, V flipped, clamped (transport.h:87-101)
__device__ inline f3 trace_image(const DeviceScene &scene, const pt_texture &tex, float u, float v) {
    u = fminf(1.0f, fmaxf(0.0f, u));
    v = fminf(1.0f, fmaxf(0.0f, v));
    int i = u * tex.width;
    int j = (1 - v) * tex.height - 0.001;
    if (i < 0) i = 0;
    if (j < 0) j = 0;
    if (i > tex.width - 1) i = tex.width - 1;
    if (j > tex.height - 1) j = tex.height - 1;
    size_t offset = size_t(tex.byte_offset) + 3 * size_t(i) + 3 * size_t(tex.width) * size_t(j);
    float red = int(scene.pixels[offset]) / 255.0;
    float green = int(scene.pixels[offset + 1]) / 255.0;
    float blue = int(scene.pixels[offset + 2]) / 255.0;
    return mk(red, green, blue);
}

__device__ inline f3 trace_texture(const DeviceScene &scene, int32_t id, float u, float v) {
    const pt_texture &tex = scene.textures[id];
    if (tex.type == PT_TEX_CONSTANT) return mk(tex.color);
    if (tex.type == PT_TEX_IMAGE) return trace_image(scene, tex, u, v);
    u = u * tex.scale.x + tex.offset.x;
    v = v * tex.scale.y + tex.offset.y;
    if (!tex.clamp) { u -= floor(u); v -= floor(v); }
    return mk(tex.color) * trace_image(scene, scene.textures[tex.image_id], u, v);
}

__device__ inline f3 trace_reflect(f3 v, f3 n) { return v - 2 * dot(v, n) * n; }

// mis_weight: power heuristic, scaled before squaring (light_sampling.h:10-16)
__device__ inline float mis_weight(float a, float b) {
    float scale = fmaxf(a, b);
    if (!(scale > 0)) return 0;
    a /= scale; b /= scale;
    return a * a / (a * a + b * b);
}

// cosine_direction (light_sampling.h:18-25)
__device__ inline f3 cosine_direction(f3 normal, Pcg &random) {
    float u = random.uniform(), v = random.uniform();
    float radius = sqrtf(u), angle = 2 * float(M_PI) * v;
    f3 helper = fabsf(normal.x) > 0.9f ? mk(0, 1, 0) : mk(1, 0, 0);
    f3 tangent = unit(cross(helper, normal));
    f3 bitangent = cross(normal, tangent);
    return radius * cosf(angle) * tangent + radius * sinf(angle) * bitangent + sqrtf(1 - u) * normal;
}

// The winning hit as shading uses it: finalize_hit's position and normal (flat_intersect.h:27-42,
// 53-64) with the triangle's normal read from its 16-byte record, the texture coordinates left for
// surface_texture, which most hits never need (with the emitters' records: Cornell render 3.06 -> 2.27
// ms, six-job batch 14.0 -> 13.7, cached 1080p frame 12.0 -> 11.7; sphere hits no longer take an
// atan2f, an asinf and two double divisions for coordinates a constant colour ignores).
struct Surface {
    f3 p, normal;
    float u, v;                 // barycentric (triangles)
    int32_t slot, material;
};

__device__ inline void surface_hit(const DeviceScene &s, const pt_ray &r, const HitInfo &h, Surface &o) {
    o.u = h.u; o.v = h.v; o.slot = h.slot;
    o.p = mk(r.origin) + h.t * mk(r.direction);
    if (h.slot < s.tri_slots) {
        const float4 a = __ldg(reinterpret_cast<const float4 *>(&s.shade_tris[h.slot]));
        const f3 outward = mk(a.x, a.y, a.z);
        o.normal = outward;
        o.material = __float_as_int(a.w);
        if (o.material < 0) {   // smooth face
            o.material = ~o.material;
            const pt_triangle &face = s.triangles[s.tris[h.slot].id];
            f3 interpolated = (1 - h.u - h.v) * mk(face.n0) + h.u * mk(face.n1) + h.v * mk(face.n2);
            float length_squared = sqlen(interpolated);
            if (length_squared > 0 && finite(length_squared)) {
                f3 normal = unit(interpolated);
                if (dot(normal, outward) < 0) normal = -normal;
                if (dot(normal, outward) == 0) normal = outward;
                o.normal = normal;
            }
        }
    } else {
        const SphereRecord &sr = s.spheres[h.slot - s.tri_slots];
        o.normal = (o.p - mk(sr.cx, sr.cy, sr.cz)) / sr.radius;
        o.material = s.sphere_src[sr.id].material_id;
    }
}

// Texture coordinates of a hit, and the texture there.  Rarer code like this (textures other than constant colours, glass, the
// debug views) is long: kernels that carry paths through all their bounces keep it out of line (kWhole), the others
// inline, since a kernel that calls anything keeps registers for it (shade_kernel with the calls and without: a
// room of 1,280 triangles at 960x600, 16 spp, 36.1 and 34.2 ms; 64 triangles at 1920x1080 7.11 and 6.69; the Cornell box
// in render_small_kernel, 960x600, 11.5 and 11.9).
static __device__ __forceinline__ f3 surface_texel_inline(const DeviceScene &s, int32_t id, int32_t slot, float u, float v, f3 normal) {
    if (slot < s.tri_slots) {
        const pt_triangle &face = s.triangles[s.tris[slot].id];
        f3 uv = (1 - u - v) * mk(face.uv0) + u * mk(face.uv1) + v * mk(face.uv2);
        u = uv.x; v = uv.y;
    } else {
        sphere_uv(normal, u, v);
    }
    return trace_texture(s, id, u, v);
}
static __device__ __noinline__ f3 surface_texel(const DeviceScene &s, int32_t id, int32_t slot, float u, float v, f3 normal) {
    return surface_texel_inline(s, id, slot, u, v, normal);
}
template <bool kWhole> __device__ inline f3 surface_texture(const DeviceScene &s, int32_t id, const Surface &o) {
    const pt_texture &tex = s.textures[id];
    if (tex.type == PT_TEX_CONSTANT) return mk(tex.color);
    if constexpr (kWhole) return surface_texel(s, id, o.slot, o.u, o.v, o.normal);
    else return surface_texel_inline(s, id, o.slot, o.u, o.v, o.normal);
}

// A sampled emitter point; `u`, `v` are the two uniform draws it came from.
struct LightSample { f3 point, normal; float u, v; int32_t index, material; };

// sample_light: area-weighted emitter choice, uniform point on it (light_sampling.h:27-54)
__device__ inline LightSample sample_light(const DeviceScene &scene, Pcg &random) {
    float choice = random.uniform() * scene.light_area;
    int low = 0, high = scene.light_count - 1;
    while (low < high) {
        int middle = low + (high - low) / 2;
        if (choice < scene.lights[middle].cumulative_area) high = middle;
        else low = middle + 1;
    }
    const float4 *rec = reinterpret_cast<const float4 *>(&scene.shade_lights[low]);
    const float4 p0 = __ldg(rec), p1 = __ldg(rec + 1);
    LightSample result;
    result.u = random.uniform(); result.v = random.uniform();
    result.index = low;
    result.material = __float_as_int(p1.w);
    if (__float_as_int(p0.w) == PT_TRIANGLE) {
        const float4 p2 = __ldg(rec + 2), n = __ldg(rec + 3);
        float root = sqrtf(result.u), a = 1 - root, b = root * (1 - result.v), c = root * result.v;
        result.point = a * mk(p0.x, p0.y, p0.z) + b * mk(p1.x, p1.y, p1.z) + c * mk(p2.x, p2.y, p2.z);
        result.normal = mk(n.x, n.y, n.z);
    } else {
        float z = 1 - 2 * result.u, radius = sqrtf(fmaxf(0, 1 - z * z)), angle = 2 * float(M_PI) * result.v;
        result.normal = mk(radius * cosf(angle), z, radius * sinf(angle));
        result.point = mk(p0.x, p0.y, p0.z) + fabsf(p1.x) * result.normal;
        if (p1.x < 0) result.normal = -result.normal;
    }
    return result;
}

// The emitter's texture at the sampled point.
static __device__ __forceinline__ f3 light_texel_inline(const DeviceScene &s, int32_t id, int32_t index, float u, float v, f3 normal) {
    const pt_light &light = s.lights[index];
    if (light.type == PT_TRIANGLE) {
        const pt_triangle &t = s.triangles[light.primitive];
        float root = sqrtf(u), a = 1 - root, b = root * (1 - v), c = root * v;
        f3 uv = a * mk(t.uv0) + b * mk(t.uv1) + c * mk(t.uv2);
        u = uv.x; v = uv.y;
    } else {
        sphere_uv(normal, u, v);
    }
    return trace_texture(s, id, u, v);
}
static __device__ __noinline__ f3 light_texel(const DeviceScene &s, int32_t id, int32_t index, float u, float v, f3 normal) {
    return light_texel_inline(s, id, index, u, v, normal);
}
template <bool kWhole> __device__ inline f3 light_emission(const DeviceScene &s, const LightSample &l) {
    const int32_t id = s.materials[l.material].texture_id;
    const pt_texture &tex = s.textures[id];
    if (tex.type == PT_TEX_CONSTANT) return mk(tex.color);
    if constexpr (kWhole) return light_texel(s, id, l.index, l.u, l.v, l.normal);
    else return light_texel_inline(s, id, l.index, l.u, l.v, l.normal);
}

// light_direction_pdf (light_sampling.h:56-65)
__device__ inline float light_direction_pdf(float area, f3 from, f3 point, f3 normal) {
    f3 delta = point - from;
    float distance_squared = sqlen(delta);
    if (!(area > 0) || !(distance_squared > 0)) return 0;
    float cosine = fabsf(dot(normal, delta)) / sqrtf(distance_squared);
    if (!(cosine > 0)) return 0;
    float pdf = distance_squared / (cosine * area);
    return finite(pdf) ? pdf : 0;
}

// hit_light_pdf (light_sampling.h:67-73); a triangle's edges are those of its walk record
__device__ inline float hit_light_pdf(const DeviceScene &scene, f3 from, const Surface &hit) {
    f3 normal = hit.normal;
    if (hit.slot < scene.tri_slots) {
        TriRecord t;
        load_tri(scene, hit.slot, t);
        normal = unit(cross(mk(t.e1x, t.e1y, t.e1z), mk(t.e2x, t.e2y, t.e2z)));
    }
    return light_direction_pdf(scene.light_area, from, hit.p, normal);
}

// Schlick's pow(1 - cosine, 5) in double, as the reference's C++ promotes it
static __device__ __noinline__ double schlick_pow_call(float cosine) { return pow(1 - cosine, 5); }
template <bool kWhole> __device__ inline double schlick_pow(float cosine) {
    if constexpr (kWhole) return schlick_pow_call(cosine);
    else return pow(1 - cosine, 5);
}

// trace_scatter (transport.h:115-155)
template <bool kWhole>
__device__ inline bool trace_scatter(const DeviceScene &scene, const pt_material &mat, f3 in_dir,
                                     const Surface &rec, Pcg &random, f3 &attenuation, f3 &out_dir) {
    f3 p = rec.p, n = rec.normal;
    if (mat.type == PT_DIFFUSE) {
        f3 target = p + n + sample_ball(random);
        out_dir = target - p;
        attenuation = surface_texture<kWhole>(scene, mat.texture_id, rec);
        return true;
    }
    if (mat.type == PT_METAL) {
        f3 reflected = trace_reflect(unit(in_dir), n);
        f3 ball = sample_ball(random);
        out_dir = reflected + mat.fuzz * ball;
        attenuation = mk(mat.albedo);
        return dot(out_dir, n) > 0;
    }
    if (mat.type == PT_GLASS) {
        f3 outward, refracted = mk(0, 0, 0);
        f3 reflected = trace_reflect(in_dir, n);
        float ratio, cosine;
        if (dot(in_dir, n) > 0) {
            outward = -n; ratio = mat.ref_idx;
            cosine = mat.ref_idx * dot(in_dir, n) / length(in_dir);
        } else {
            outward = n; ratio = 1.0f / mat.ref_idx;
            cosine = -dot(in_dir, n) / length(in_dir);
        }
        f3 uv = unit(in_dir);
        float dt = dot(uv, outward);
        float discriminant = 1.0f - ratio * ratio * (1 - dt * dt);
        float probability = 1;
        if (discriminant > 0) {
            refracted = ratio * (uv - outward * dt) - outward * sqrt(discriminant);
            float r0 = (1 - mat.ref_idx) / (1 + mat.ref_idx);
            r0 *= r0;
            probability = r0 + (1 - r0) * schlick_pow<kWhole>(cosine);
        }
        if (random.uniform() < probability) out_dir = reflected;
        else out_dir = refracted;
        attenuation = mk(1, 1, 1);
        return true;
    }
    return false;
}

// id_color (transport.h:164-167)
__device__ inline f3 id_color(int id) {
    uint32_t bits = (uint32_t(id) + 1u) * 2654435761u;
    return mk((bits & 255) / 255.0f, ((bits >> 8) & 255) / 255.0f, ((bits >> 16) & 255) / 255.0f);
}

} // namespace ptb
