// st_render.cu — the per-frame kernels: screen-space bounds, ray-direction rows, the trace+shade
// megakernel and the QCAA resolve.
#include <cstdio>
#include "st_trace.cuh"
#include "st_kernels.h"

namespace st {

// Records of 64 bytes are read with two 256-bit loads (a warp's lanes read unrelated records, so
// every load instruction costs a tag look-up per lane: four 128-bit loads made the traces 1 to 3 %
// slower).  Cache hints: node pairs are marked to stay in L1 (evict_last; the top of every BLAS is
// read by every ray that enters an instance), triangle records to leave first (evict_first; a
// triangle is tested by the few neighbouring rays that reach its leaf; the 128-byte record of the
// winning triangle is read once per hit).  Hints change no value read.
__device__ __forceinline__ NodePair load_pair(const NodePair *p) {
    NodePair r;
    const float *f = reinterpret_cast<const float *>(p);
    asm("ld.global.nc.L1::evict_last.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(r.a.x), "=f"(r.a.y), "=f"(r.a.z), "=f"(r.a.w), "=f"(r.b.x), "=f"(r.b.y), "=f"(r.b.z), "=f"(r.b.w) : "l"(f));
    float d[4];
    asm("ld.global.nc.L1::evict_last.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(r.c.x), "=f"(r.c.y), "=f"(r.c.z), "=f"(r.c.w), "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "l"(f + 8));
    r.d = make_uint4(__float_as_uint(d[0]), __float_as_uint(d[1]), __float_as_uint(d[2]), __float_as_uint(d[3]));
    return r;
}
__device__ __forceinline__ TriHot load_tri(const TriHot *p) {
    TriHot T;
    const float *f = reinterpret_cast<const float *>(p);
    asm("ld.global.nc.L1::evict_first.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(T.p.x), "=f"(T.p.y), "=f"(T.p.z), "=f"(T.p.w), "=f"(T.q.x), "=f"(T.q.y), "=f"(T.q.z), "=f"(T.q.w) : "l"(f));
    asm("ld.global.nc.L1::evict_first.v8.f32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=f"(T.r.x), "=f"(T.r.y), "=f"(T.r.z), "=f"(T.r.w), "=f"(T.s.x), "=f"(T.s.y), "=f"(T.s.z), "=f"(T.s.w) : "l"(f + 8));
    return T;
}

// The closest hit's full record (hitPrimitives' copy of the winner's RayHit and its final step,
// primitives.h:63-108), rebuilt after a walk that found t.best: the winner's hit test runs again on
// the same object-space ray (to_object and the offset as in the candidate loop), which gives the
// record the candidate loop saw bit for bit; then the barycentric interpolation of mesh normals and
// uvs, the primitive id, the world normal, distance, cone width and area.
template <bool CNT, int SHS>
__device__ __forceinline__ void finalize_hit(TState<CNT, SHS> &t, const SceneDev &S, const RayD &ray, float cone_angle) {
    Hit closest = {};       // every field is written below: the last hit's record is not live through a walk
    const u32t hid = t.best.prim;
    const PrimDev HP = S.prims[hid];
    const unsigned flags = prim_flags(HP), type = prim_type(HP);
    v3 lo, ld;
    to_object(ray.origin, ray.direction, HP, lo, ld);
    lo = vsfma(ld, kTraceOffset, lo);
    switch (type) {
        case PrimitiveType_Quad: hit_quad(closest, lo, ld, flags); break;
        case PrimitiveType_Box: hit_box(closest, lo, ld, flags); break;
        case PrimitiveType_Sphere: hit_sphere(closest, lo, ld, flags); break;
        case PrimitiveType_Tetrahedron: hit_tetra(closest, lo, ld, flags); break;
        default: {                                              // PrimitiveType_Mesh
            const MeshDev &M = S.meshes[__float_as_uint(HP.scale_id.w)];
            const u32t tri = t.best.tri;
            const TriHot T = S.tri_hot[M.tri_offset + tri];
            const v3 pos = V(T.p.x, T.p.y, T.p.z);
            hit_plane(pos, V(T.p.w, T.q.x, T.q.y), lo, ld, closest);
            const float m[9] = {T.q.z, T.q.w, T.r.x, T.r.y, T.r.z, T.r.w, T.s.x, T.s.y, T.s.z};
            const v3 UV = vmat3(closest.position - pos, m);
            closest.u = UV.x;
            closest.v = UV.y;
            Triangle TF;
            {
                const float4 *f = reinterpret_cast<const float4 *>(S.tri_full + M.tri_offset + tri);
                float4 *o = reinterpret_cast<float4 *>(&TF);
#pragma unroll
                for (int k = 0; k < 8; k++)
                    asm("ld.global.nc.L1::evict_first.v4.f32 {%0,%1,%2,%3}, [%4];"
                        : "=f"(o[k].x), "=f"(o[k].y), "=f"(o[k].z), "=f"(o[k].w) : "l"(f + k));
            }
            closest.area = TF.area_of_parallelogram;
            closest.uv_area = TF.area_of_uv;
            if (M.normals_count | M.uvs_count) {
                float u = closest.u, v = closest.v;
                float w = 1 - u - v;
                if (M.uvs_count) {
                    closest.u = TF.uvs[2].x * u + (TF.uvs[1].x * v + TF.uvs[0].x * w);
                    closest.v = TF.uvs[2].y * u + (TF.uvs[1].y * v + TF.uvs[0].y * w);
                }
                if (M.normals_count) {
                    const vec3 *vn = TF.vertex_normals;
                    closest.normal.x = vn[2].x * u + (vn[1].x * v + vn[0].x * w);
                    closest.normal.y = vn[2].y * u + (vn[1].y * v + vn[0].y * w);
                    closest.normal.z = vn[2].z * u + (vn[1].z * v + vn[0].z * w);
                    closest.normal = norm(closest.normal);
                }
            }
        } break;
    }
    closest.position = t.best.position;
    closest.distance_squared = t.best.distance_squared;
    closest.object_type = type;
    closest.material_id = prim_material(HP);
    closest.object_id = hid;
    closest.normal = norm(dir_to_world(closest.normal, HP));
    closest.distance = t.best.distance;
    closest.cone_width = 2.0f * cone_angle * closest.distance;
    v3 rs = qrot(V(HP.scale_id.x, HP.scale_id.y, HP.scale_id.z), prim_rot(HP));
    closest.area *= dot(one_minus(closest.normal), rs);
    t.closest = closest;
}

// ---- traceScene shaders/trace.h:8, hitPrimitives primitives.h:9 and traceMesh mesh.h:38 --------------
// One loop walks both levels.  A lane is either in the TLAS or, between enter_mesh and leave_mesh, in
// the BLAS of one instance; both kinds of node are the same step on the same registers (node array,
// reciprocal direction, scaled origin, limit), so that lanes of a warp that are in different
// instances, or some in the TLAS, step together instead of waiting for one another's BLAS walk.  What
// the TLAS level needs after the instance (its leaf queue, its next pair, its ray) is kept in the
// stack's frame meanwhile.  (With the BLAS walk nested in the candidate loop, as in the reference, a
// warp waited at every candidate for the longest BLAS walk among its lanes, and the outer walk's
// state was spilled around the inner one: 1080p mesh frames 3.28-4.07 ms against 2.91-3.74, the
// moving scene 1.32-1.57 against 0.92-1.09.  Leaving the node loop early by a warp vote once half
// or a quarter of the lanes wait cost more in votes than it saved; keeping each pending pair's entry
// distance on the stack to drop those beyond the closest hit saved as many steps as the wider stack
// cost.)  Each lane's own sequence of tests is the reference's:
// the leaves met at a node (left, then right) are tested before the walk moves on, the nearer child
// is entered first, and candidates are tested in leaf order.
// with ssb != null it serves primary rays (the screen-space cull); all_prims: every primitive in
// leaf-id order without the root box (the primary-ray path of scenes with few primitives,
// raytracer.h:100, and picking).
// A winner updates t.best: the world distance (as hitPrimitives' final step leaves it,
// primitives.h:105), its square, the world position and which primitive and triangle it is; the rest
// of hitPrimitives' record is finalize_hit's.
template <bool CNT, int SHS>
__device__ __forceinline__ bool trace_scene(TState<CNT, SHS> &t, const SceneDev &S, const RayD &ray, bool any_hit,
                                            const int4 *ssb, int x, int y, bool all_prims) {
    Best &best = t.best;
    Slabs slabs = prepare(ray.origin, ray.direction);
    v3 lo = ray.origin, ld = ray.direction;            // the object-space ray while in a mesh
    if (!all_prims) {
        t.count(C_AABB);
        if (!hit_box_slabs(S.tlas_root_aabb, slabs, best.distance)) return false;
    }
    const NodePair *nodes = S.tlas_pairs;
    // the leaf queue: items [q0, q0_end) of the leaf being tested, then the q1_count items from q1
    u32t q0 = 0, q0_end = 0, q1 = 0, q1_count = 0, pair = kNoPair;
    if (all_prims || S.tlas_root_count) q0_end = S.n_prims;
    else pair = (S.tlas_root_first - 1) >> 1;
    u32t sp = 0, base = 0;                             // base: the stack's first entry of this level
    float limit = best.distance;                       // the walk's closest hit at this level
    bool in_mesh = false, found = false;
    u32t tri_base = 0;
    for (;;) {
        // inner nodes until this lane has leaves queued ("while-while": lanes of a warp walk nodes
        // together and test leaves together)
        while (q0 == q0_end && pair != kNoPair) {
            const NodePair P = load_pair(nodes + pair);
            t.count(C_AABB, 2);
            float ldist, rdist;
            bool lgo, rgo;
            hit_pair(P, slabs, S.neg_zero, limit, lgo, rgo, ldist, rdist);
            if (lgo && P.d.y) { q0 = P.d.x; q0_end = P.d.x + P.d.y; lgo = false; }
            if (rgo && P.d.w) {
                if (q0 != q0_end) { q1 = P.d.z; q1_count = P.d.w; }
                else { q0 = P.d.z; q0_end = P.d.z + P.d.w; }
                rgo = false;
            }
            if (lgo && rgo) {
                const bool swap = !any_hit && ldist > rdist;
                if (sp - base >= (u32t)kStack) {       // the queued leaves still run, then the level ends
                    t.status |= S_STACK_OVERFLOW;
                    pair = kNoPair;
                    sp = base;
                    continue;
                }
                t.push(sp++, swap ? P.d.x : P.d.z);
                pair = swap ? P.d.z : P.d.x;
            } else if (lgo | rgo) {
                pair = lgo ? P.d.x : P.d.z;
            } else {
                pair = sp != base ? t.at(--sp) : kNoPair;
            }
        }
        bool leave = false;
        if (in_mesh) {
            // hitTriangles (mesh.h:5) over the queued leaves: an accepted triangle (in front of the
            // closest so far, inside by its tangent-space UV) becomes the closest
            leave = q0 == q0_end;
            while (q0 != q0_end) {
                const TriHot T = load_tri(S.tri_hot + tri_base + q0);
                t.count(C_TRI);
                const v3 pos = V(T.p.x, T.p.y, T.p.z), nrm = V(T.p.w, T.q.x, T.q.y);
                Hit hit;
                if (hit_plane(pos, nrm, lo, ld, hit) && hit.distance < limit) {
                    const float m[9] = {T.q.z, T.q.w, T.r.x, T.r.y, T.r.z, T.r.w, T.s.x, T.s.y, T.s.z};
                    const v3 UV = vmat3(hit.position - pos, m);
                    if (!(UV.x < 0 || UV.y < 0 || (UV.x + UV.y) > 1)) {
                        limit = hit.distance;
                        t.mesh_tri = q0;
                        if (any_hit) { leave = true; break; }
                    }
                }
                if (++q0 == q0_end && q1_count) {
                    q0 = q1;
                    q0_end = q1 + q1_count;
                    q1_count = 0;
                }
            }
        }
        if (in_mesh) {
            if (!leave) continue;
            // leave the instance: its ray's hit, if any, is a candidate (hitPrimitives after traceMesh)
            sp = base;
            const u32t pid = t.at(sp - 1), tri = t.mesh_tri;
            in_mesh = false;
            if (tri != kNoTriangle) {
                // the accepted triangle's object-space hit point, recomputed exactly as it was
                // computed above (same triangle, same ray, same operations)
                const PrimDev Pm = S.prims[pid];
                const float4 tp = __ldg(reinterpret_cast<const float4 *>(S.tri_hot + tri_base + tri));
                const float4 tq = __ldg(reinterpret_cast<const float4 *>(S.tri_hot + tri_base + tri) + 1);
                Hit h;
                hit_plane(V(tp.x, tp.y, tp.z), V(tp.w, tq.x, tq.y), lo, ld, h);
                const v3 pos = pos_to_world(h.position, Pm);
                const float dsq = sqlen(pos - ray.origin);
                if (dsq < best.distance_squared) {
                    best.distance_squared = dsq;
                    best.distance = sqrtf(dsq);
                    best.position = pos;
                    best.prim = pid;
                    best.tri = tri;
                    found = true;
                    if (any_hit) return true;
                }
            }
            pair = t.at(sp - 2);
            q0 = t.at(sp - 3);
            q0_end = t.at(sp - 4);
            q1 = t.at(sp - 5);
            q1_count = t.at(sp - 6);
            sp -= kFrame;
            base = 0;
            nodes = S.tlas_pairs;
            limit = best.distance;
            slabs = prepare(ray.origin, ray.direction);
            if (q0 == q0_end && q1_count) {
                q0 = q1;
                q0_end = q1 + q1_count;
                q1_count = 0;
            }
        }
        // candidates of the queued TLAS leaves, up to the next instance whose BLAS is to be walked
        if (q0 == q0_end && pair == kNoPair) break;
        while (q0 != q0_end) {
            t.count(C_LEAF);
            const u32t pid = __ldg(S.tlas_leaf_ids + q0);
            q0++;
            bool cull = false;
            if (ssb) {      // primary rays: IS_VISIBLE and the screen-space rect, folded into one rect per view
                const int4 b = __ldg(ssb + pid);
                cull = x < b.x || x >= b.z || y < b.y || y >= b.w;
            }
            if (!cull) {
                const PrimDev P = S.prims[pid];
                const unsigned flags = prim_flags(P);
                if (!any_hit || (flags & IS_SHADOWING)) {
                    t.count(C_PRIM);
                    to_object(ray.origin, ray.direction, P, lo, ld);
                    lo = vsfma(ld, kTraceOffset, lo);
                    const unsigned type = prim_type(P);
                    if (type == PrimitiveType_Mesh) {
                        const MeshDev &M = S.meshes[__float_as_uint(P.scale_id.w)];
                        const Slabs ms = prepare(lo, ld);
                        const float md = best.distance == INFINITY ? INFINITY : len(pos_to_object(best.position, P) - lo);
                        t.count(C_MESH);
                        t.count(C_AABB);
                        // md is NaN where the instance has a zero scale and something was hit before:
                        // nothing of it can be nearer (without the test such a ray walked the mesh, up
                        // to 2.3 times the triangles of frames with one primitive in three flat)
                        if (md >= 0 && hit_box_slabs(M.aabb, ms, md)) {
                            t.push(sp, q1_count);
                            t.push(sp + 1, q1);
                            t.push(sp + 2, q0_end);
                            t.push(sp + 3, q0);
                            t.push(sp + 4, pair);
                            t.push(sp + 5, pid);
                            sp += kFrame;
                            base = sp;
                            in_mesh = true;
                            slabs = ms;
                            limit = md;
                            t.mesh_tri = kNoTriangle;
                            tri_base = M.tri_offset;
                            nodes = S.mesh_pairs + M.pair_offset;
                            q0 = q0_end = q1_count = 0;
                            pair = kNoPair;
                            if (M.root_count) q0_end = M.triangle_count;
                            else pair = (M.root_first - 1) >> 1;
                            break;
                        }
                    } else {
                        Hit hit;
                        bool cur = false;
                        switch (type) {
                            case PrimitiveType_Quad: cur = hit_quad(hit, lo, ld, flags); break;
                            case PrimitiveType_Box: cur = hit_box(hit, lo, ld, flags); break;
                            case PrimitiveType_Sphere: cur = hit_sphere(hit, lo, ld, flags); break;
                            case PrimitiveType_Tetrahedron: cur = hit_tetra(hit, lo, ld, flags); break;
                        }
                        if (cur) {
                            const v3 pos = pos_to_world(hit.position, P);
                            const float dsq = sqlen(pos - ray.origin);
                            if (dsq < best.distance_squared) {
                                best.distance_squared = dsq;
                                limit = best.distance = sqrtf(dsq);
                                best.position = pos;
                                best.prim = pid;
                                best.tri = 0;
                                found = true;
                                if (any_hit) return true;
                            }
                        }
                    }
                }
            }
            if (q0 == q0_end && q1_count) {
                q0 = q1;
                q0_end = q1 + q1_count;
                q1_count = 0;
            }
        }
    }
    return found;
}

// ---- closest_hit/surface.h, lights.h ------------------------------------------------------------
template <bool CNT, int SHS>
__device__ v3 shade_from_lights(TState<CNT, SHS> &t, const SceneDev &S, Shaded &s, RayD &ray, v3 color) {   // surface.h:9
    // The reference writes each light into trace->closest_hit (:14-17) and the shadow ray's walk
    // reads it there (the occluder must be nearer than the light) or overwrites it with an
    // occluder: the walk's record t.best plays that part, and closest_hit's position and distances
    // are left as the last light's walk left them, because the emissive-quad test reads them (:55).
    Best &b = t.best;
    for (u32t i = 0; i < S.n_lights; i++) {
        const Light &light = S.lights[i];
        b.position = from(light.position_or_direction);
        s.light_direction = b.position - s.position;
        b.distance_squared = sqlen(s.light_direction);
        b.distance = sqrtf(b.distance_squared);
        s.light_direction = vscale(s.light_direction, 1.0f / b.distance);
        float NdotL = dot(s.normal, s.light_direction);
        if (NdotL <= 0) continue;
        float li = light.intensity / b.distance_squared;
        ray.origin = s.position;
        ray.direction = s.light_direction;
        t.count(C_SHADOW);
        if (trace_scene(t, S, ray, true, nullptr, 0, 0, false)) continue;       // inShadow trace.h:85
        color = vvfma(shade_point(s, NdotL), vscale(from(light.color), li), color);
    }
    if (S.n_lights) {
        t.closest.position = b.position;
        t.closest.distance_squared = b.distance_squared;
        t.closest.distance = b.distance;
    }
    return color;
}

template <bool CNT, int SHS>
__device__ bool shade_from_emissive_quads(TState<CNT, SHS> &t, const SceneDev &S, Shaded &s, RayD &ray, v3 &color) {  // surface.h:37
    Hit hit;                                    // the reference's trace->current_hit, scratch here
    bool found = false;
    for (u32t e = 0; e < S.n_emissive; e++) {
        const u32t qi = S.emissive_quads[e];
        const PrimDev Q = S.prims[qi];
        const Primitive &quad = S.prims_raw[qi];
        const Material &em = S.materials[prim_material(Q)];
        v3 Ro, Rd;
        to_object(s.viewing_origin, s.viewing_direction, Q, Ro, Rd);
        if (hit_quad(hit, Ro, Rd, prim_flags(Q))) {
            hit.position = pos_to_world(hit.position, Q);
            hit.distance_squared = sqlen(hit.position - s.viewing_origin);
            if (hit.distance_squared < t.closest.distance_squared) {
                hit.object_id = qi;
                hit.object_type = PrimitiveType_Quad;
                hit.material_id = prim_material(Q);
                t.closest = hit;
                found = true;
            }
        }
        v3 qn = qrot(V(0, 1, 0), prim_rot(Q));
        v3 qpos = V(Q.pos_bits.x, Q.pos_bits.y, Q.pos_bits.z);
        s.light_direction = ray.direction = qpos - s.position;
        if (dot(qn, s.light_direction) >= 0) continue;
        v3 quad_vertices[4];
        float ei = dot(s.normal, area_light_vector(quad, s.position, quad_vertices));
        if (ei > 0) {
            bool skip = true;
            for (int j = 0; j < 4; j++)
                if (dot(s.normal, quad_vertices[j] - s.position) >= 0) { skip = false; break; }
            if (skip) continue;
            float shaded_light = 1;
            if (qi != s.prim_index) {
                for (u32t k = 0; k < S.n_occluders; k++) {
                    const u32t oi = S.occluders[k];
                    const PrimDev O = S.prims[oi];
                    if (oi == qi || dot(qn, V(O.pos_bits.x, O.pos_bits.y, O.pos_bits.z) - qpos) <= 0) continue;
                    v3 oRo, oRd;
                    to_object(s.position, s.light_direction, O, oRo, oRd);
                    oRo = vsfma(oRd, kTraceOffset, oRo);
                    float d = 1;
                    if (prim_type(O) == PrimitiveType_Sphere) {
                        if (hit_sphere(hit, oRo, oRd, prim_flags(O)))
                            d -= (1.0f - sqrtf(hit.distance_squared)) / (hit.distance * ei * 3);
                    } else {
                        if (hit_quad(hit, oRo, oRd, prim_flags(O))) {
                            hit.position.y = 0;
                            hit.position.x = hit.position.x < 0 ? -hit.position.x : hit.position.x;
                            hit.position.z = hit.position.z < 0 ? -hit.position.z : hit.position.z;
                            if (hit.position.x > hit.position.z) {
                                hit.position.y = hit.position.z;
                                hit.position.z = hit.position.x;
                                hit.position.x = hit.position.y;
                                hit.position.y = 0;
                            }
                            d -= (1.0f - hit.position.z) / (hit.distance * ei);
                        }
                    }
                    if (d < shaded_light) shaded_light = d;
                }
            }
            if (shaded_light > 0) {
                float NdotL = dot01(s.normal, s.light_direction);
                if (NdotL) color = vvfma(shade_point(s, NdotL), vscale(from(em.emission), ei * shaded_light), color);
            }
        }
    }
    if (found) t.closest.distance = sqrtf(t.closest.distance_squared);
    return found;
}

__device__ __forceinline__ float volume_density(const SphereHitD &h) {   // lights.h:7
    float t1 = h.t_near > 0 ? h.t_near : 0;
    float t2 = h.t_far < h.furthest ? h.t_far : h.furthest;
    return (h.c * t1 - h.b * t1 * t1 + t1 * t1 * t1 / 3.0f - (
            h.c * t2 - h.b * t2 * t2 + t2 * t2 * t2 / 3.0f)) * (3.0f / 4.0f);
}
template <bool CNT, int SHS>
__device__ bool shade_lights(TState<CNT, SHS> &t, const SceneDev &S, v3 Ro, v3 Rd, float max_distance, v3 &color) {  // lights.h:17
    bool hit_light = false;
    SphereHitD &sh = t.sphere;
    sh.closest_distance = INFINITY;
    for (u32t i = 0; i < S.n_lights; i++) {
        const Light &light = S.lights[i];
        float size = light.intensity * (1.0f / 16.0f);
        float oor = 8.0f / size;
        sh.furthest = max_distance * oor;
        if (hit_sphere_simple(Ro, Rd, from(light.position_or_direction), oor, sh)) {
            float distance = sh.t_far - size * 8;
            float density = powf(volume_density(sh), 8) * 8;
            if (distance < sh.closest_distance) sh.closest_distance = distance;
            color = vsfma(from(light.color), density, color);
            hit_light = true;
        }
    }
    return hit_light;
}

template <bool CNT, int SHS>
__device__ __forceinline__ void apply_textures(TState<CNT, SHS> &t, const SceneDev &S, Shaded &s, Hit &hit, const Material &M,
                                               float &dv, bool first) {
    const float u = hit.u * M.uv_repeat.x, v = hit.v * M.uv_repeat.y;
    hit.uv_area /= M.uv_repeat.x / M.uv_repeat.y;
    const float du = duv_ray_cone(hit.NdotV, hit.cone_width, hit.area, hit.uv_area);
    if (first) dv = du;             // surface.h:162 sets u and v; the bounce path (:230) only u
    if (M.use & ALBEDO_MAP) s.albedo = sample_texture(t, S, M.texture_ids[0], u, v, du, dv);
    if ((M.use & NORMAL_MAP) && M.texture_count > 1) {
        q4 rot = normal_rotation(sample_normal(t, S, M.texture_ids[1], u, v, du, dv));
        hit.normal = qrot(hit.normal, rot);
    }
}

// ---- the frame kernels -----------------------------------------------------------------------
// computeSSB render/SSB.h:5 for one primitive; the result is folded with IS_VISIBLE into one rect
// (an invisible primitive gets an empty rect) so that the primary-ray cull is a single test.
__device__ bool compute_ssb(int4 &b, v3 pos, float r, float fl, const ViewDev &v) {
    b.x = v.grid_w + 1; b.z = v.grid_w + 1; b.y = v.grid_h + 1; b.w = v.grid_h + 1;
    if (pos.z <= -r) return false;
    float x = pos.x, y = pos.y, z = pos.z, left, right, top, bottom, factor;
    if (z <= r) {
        float h = fabsf(z) / fl;
        top = y + r;
        bottom = y - r;
        if (h < bottom || top < -h) return false;
        float w = h * v.width_over_height;
        right = x + r;
        left = x - r;
        if (w < left || right < -w) return false;
        b.x = -w < left ? (int)(uint16_t)(v.f_width * (left + w) / (2 * w)) : 0;
        b.z = right < w ? (int)(uint16_t)(v.f_width * (right + w) / (2 * w)) : (int)v.grid_w;
        b.y = top < h ? (int)(uint16_t)(v.f_height * (h - top) / (2 * h)) : 0;
        b.w = -h < bottom ? (int)(uint16_t)(v.f_height * (h - bottom) / (2 * h)) : (int)v.grid_h;
        return true;
    }
    float den = z * z - r * r;
    factor = fl / den;
    float yz = y * z;
    float sqr = y * y + den;
    sqr = r * sqrtf(sqr);
    bottom = factor * (yz - sqr);
    top = factor * (yz + sqr);
    if (bottom < 1 && top > -1) {
        factor *= v.height_over_width;
        float xz = x * z;
        sqr = r * sqrtf(x * x + den);
        left = factor * (xz - sqr);
        right = factor * (xz + sqr);
        if (left < 1 && right > -1) {
            bottom = bottom > -1 ? bottom : -1; bottom += 1;
            top = top < 1 ? top : 1; top += 1;
            left = left > -1 ? left : -1; left += 1;
            right = right < 1 ? right : 1; right += 1;
            top = 2 - top;
            bottom = 2 - bottom;
            b.x = (int)(uint16_t)(v.h_width * left);
            b.z = (int)(uint16_t)(v.h_width * right);
            b.w = (int)(uint16_t)(v.h_height * bottom);
            b.y = (int)(uint16_t)(v.h_height * top);
            return true;
        }
    }
    return false;
}

// updatePrimitiveSSB render/SSB.h:137 for primitive i of one view
__device__ __forceinline__ int4 ssb_of(const SceneDev &S, const ViewDev &v, u32t i) {
    const Primitive p = S.prims_raw[i];
    v3 view = vmat3(from(p.position) - v.cam_pos, v.cam_rot_matrix_inv);
    float radius;
    v3 sc = from(p.scale);
    switch (p.type) {
        case PrimitiveType_Quad: case PrimitiveType_Box: radius = len(sc); break;
        case PrimitiveType_Tetrahedron: { float m = sc.x; if (sc.y > m) m = sc.y; if (sc.z > m) m = sc.z; radius = m * kSqrt2; } break;
        case PrimitiveType_Sphere: { float m = sc.x; if (sc.y > m) m = sc.y; if (sc.z > m) m = sc.z; radius = m; } break;
        case PrimitiveType_Mesh: {
            const MeshDev &M = S.meshes[p.id];
            float mn = len(vmul(sc, V(M.mesh_aabb[0], M.mesh_aabb[1], M.mesh_aabb[2])));
            float mx = len(vmul(sc, V(M.mesh_aabb[3], M.mesh_aabb[4], M.mesh_aabb[5])));
            radius = mx > mn ? mx : mn;
        } break;
        default: {
            // updatePrimitiveSSB returns without touching other types: keep the uploaded values
            const bool vis = p.flags & IS_VISIBLE;
            return vis ? make_int4(p.screen_bounds.min.x, p.screen_bounds.min.y, p.screen_bounds.max.x, p.screen_bounds.max.y)
                       : make_int4(1, 1, 0, 0);
        }
    }
    int4 b;
    bool vis = compute_ssb(b, view, radius, v.focal_length, v);
    return vis ? b : make_int4(1, 1, 0, 0);
}

// The reference walks each row of the QCAA grid by repeated addition (raytracer.h:156-170):
// row y starts at start + down added y times, pixel x at that plus right added x times.  That
// sequence is kept exactly: one thread per row walks it and stores every kSegment-th value
// ("segment starts", 3 MB at 1080p instead of a 25 MB direction table); the trace kernel adds
// `right` the remaining x % kSegment times itself.  The starts are stored segment-major (segment k
// of every row, row after row), so that the threads of a warp, one per row, write one contiguous
// run per segment, and a warp tile's four rows read 48 contiguous bytes.
__device__ __forceinline__ void row_segments_one(const ViewDev &v, float *seg, u32t row) {
    v3 cur = v.pp_start;
#pragma unroll 8
    for (u32t y = 0; y < row; y++) cur = cur + v.pp_down;
    const u32t nseg = (v.grid_w + kSegment - 1) / kSegment;
    for (u32t k = 0; k < nseg; k++) {
        float *out = seg + ((size_t)k * v.grid_h + row) * 3;
        out[0] = cur.x;
        out[1] = cur.y;
        out[2] = cur.z;
        for (int i = 0; i < kSegment; i++) cur = cur + v.pp_right;
    }
}
// What a frame's trace reads of its view: the first row_blocks blocks make the row-segment starts (a
// chain of additions as long as the frame's sides, whatever the parallelism), the others the
// primitives' screen bounds beside them; one launch, since each of the two is shorter than a launch.
constexpr u32t kSetupThreads = 64;
__device__ __forceinline__ void setup_one(const SceneDev &S, const ViewDev &v, int4 *ssb, float *seg, u32t block, u32t row_blocks) {
    if (block < row_blocks) {
        const u32t row = block * kSetupThreads + threadIdx.x;
        if (row < v.grid_h) row_segments_one(v, seg, row);
    } else {
        const u32t i = (block - row_blocks) * kSetupThreads + threadIdx.x;
        if (i < S.n_prims) ssb[i] = ssb_of(S, v, i);
    }
}
__global__ void frame_setup_kernel(SceneDev S, ViewDev v, int4 *ssb, float *seg, u32t row_blocks) {
    setup_one(S, v, ssb, seg, blockIdx.x, row_blocks);
}

__device__ __forceinline__ v3 grid_direction(const ViewDev &v, const float *seg, u32t x, u32t y) {
    const float *s = seg + ((size_t)(x / kSegment) * v.grid_h + y) * 3;
    v3 cur = V(__ldg(s), __ldg(s + 1), __ldg(s + 2));
    for (u32t i = 0; i < x % kSegment; i++) cur = cur + v.pp_right;
    return cur;
}

// What a path carries from one trace to the next: shadeSurface's state across its bounce loop
// (surface.h:146-239) and what rayTrace keeps of the primary hit.
struct Path {
    v3 color, throughput;
    float dv;                       // the ray-cone footprint the primary hit leaves (surface.h:162)
    float max_distance;             // the lights' glow limit
    float closest_distance, z;      // the primary hit's distance and depth
    u32t bounces;                   // shadeSurface's `depth`
    bool lights_shaded, hit_found;
};

// The primary ray of grid point (x, y), and the path and walk state rayTrace starts with.
template <bool CNT, int SHS>
__device__ __forceinline__ void start_path(TState<CNT, SHS> &t, const ViewDev &v, const float *dirs, u32t x, u32t y,
                                           RayD &ray) {
    t.closest.distance = t.closest.distance_squared = INFINITY;
    t.closest.cone_width = 0;
    t.best.distance = t.best.distance_squared = INFINITY;
    ray.origin = v.cam_pos;
    ray.direction = norm(grid_direction(v, dirs, x, y));
    t.count(C_PRIMARY);
}
__device__ __forceinline__ void start_path(Path &p, u32t depth) {
    p.color = splat(0);
    p.throughput = splat(1);
    p.dv = p.max_distance = 0;
    p.closest_distance = p.z = INFINITY;
    p.bounces = depth;
    p.lights_shaded = p.hit_found = false;
}

// The steps of rayTrace and shadeSurface (surface.h:146) from one trace to the next: what the ray
// that was just traced found (t.best, when `found`) is shaded into the path.  True: the path goes on
// with the bounce ray left in `ray`, its walk state reset; false: the path is done.
template <bool CNT, int SHS>
__device__ __forceinline__ bool shade_step(TState<CNT, SHS> &t, const SceneDev &S, const ViewDev &v, RayD &ray, Path &p,
                                           bool primary, bool found) {
    Hit &hit = t.closest;
    if (found) finalize_hit(t, S, ray, primary ? v.cone_angle : 0.0f);
    Shaded s;
    const Material *M;
    if (primary) {                                          // rayTrace after the hit test (raytracer.h:89)
        p.hit_found = found;
        p.closest_distance = found ? hit.distance : INFINITY;
        if (!found) return false;
        p.z = qrot(hit.position - v.cam_pos, v.cam_rot_inv).z;
        if (v.mode != RenderMode_Beauty) {
            switch (v.mode) {
                case RenderMode_Depth: p.color = splat(4 / hit.distance); break;
                case RenderMode_Normals: {
                    const Material &NM = S.materials[hit.material_id];
                    if (NM.texture_count > 1 && (NM.use & NORMAL_MAP)) {
                        float u = hit.u * NM.uv_repeat.x, vv = hit.v * NM.uv_repeat.y;
                        hit.uv_area /= NM.uv_repeat.x / NM.uv_repeat.y;
                        float ndu = duv_ray_cone(hit.NdotV, hit.cone_width, hit.area, hit.uv_area);
                        q4 rot = normal_rotation(sample_normal(t, S, NM.texture_ids[1], u, vv, ndu, 0.0f));
                        hit.normal = qrot(hit.normal, rot);
                    }
                    p.color = V(0.5f * (hit.normal.x + 1), 0.5f * (hit.normal.y + 1), 0.5f * (hit.normal.z + 1));
                } break;
                case RenderMode_UVs: p.color = V(0.5f * hit.u, 0.5f * hit.v, 0.5f); break;
            }
            return false;
        }
        // shadeSurface (surface.h:146) up to its bounce loop
        M = S.materials + hit.material_id;
        t.count(C_SHADE);
        if (M->is & EMISSIVE) {
            if (!hit.from_behind) p.color = from(M->emission);
            return false;
        }
        s.albedo = from(M->albedo);
        if (M->use && M->texture_count) apply_textures(t, S, s, hit, *M, p.dv, true);
        p.max_distance = hit.distance;
    } else {                                                // traceRay returned (surface.h:214-239)
        if (!found) return false;
        t.count(C_SHADE);
        M = S.materials + hit.material_id;
        s.albedo = from(M->albedo);
        if (M->use && M->texture_count) apply_textures(t, S, s, hit, *M, p.dv, false);
        if (hit.object_type == PrimitiveType_Quad && (M->is & EMISSIVE)) {
            p.color = hit.from_behind ? splat(0) : from(M->emission);
            return false;
        }
        if (M->brdf != BRDF_CookTorrance) p.throughput = vmul(p.throughput, from(M->reflectivity));
    }
    s.viewing_origin = ray.origin;
    s.viewing_direction = ray.direction;
    s.prim_index = hit.object_id;
    s.material = M;
    // one iteration of shadeSurface's bounce loop
    if (!p.bounces) return false;
    s.position = ray.origin = hit.position;
    s.normal = hit.from_behind ? neg(hit.normal) : hit.normal;
    const float ior = hit.from_behind ? M->n2_over_n1 : M->n1_over_n2;
    const bool is_ref = (M->is & REFLECTIVE) || (M->is & REFRACTIVE);
    float NdotRd = 0;
    s.reflected_direction = splat(0);
    if (is_ref || M->brdf == BRDF_Phong) {
        NdotRd = -clamp01(-dot(s.normal, s.viewing_direction));      // invDotVec3 common.h:97
        s.reflected_direction = vsfma(s.normal, -2.0f * NdotRd, s.viewing_direction);  // reflectWithDot :101
    }
    v3 cur = is_ref ? splat(0) : from(S.ambient);
    if (S.lights) cur = shade_from_lights(t, S, s, ray, cur);
    if (S.n_emissive)
        if (shade_from_emissive_quads(t, S, s, ray, cur)) p.max_distance = hit.distance;
    p.color = vvfma(cur, p.throughput, p.color);
    if (S.lights && shade_lights(t, S, s.viewing_origin, s.viewing_direction, p.max_distance, p.color))
        p.lights_shaded = true;
    if (!(is_ref && --p.bounces)) return false;
    if (M->is & REFLECTIVE) ray.direction = s.reflected_direction;
    else {                                                         // refract common.h:105
        v3 Vv = s.viewing_direction, N = s.normal;
        float c = ior * ior * (1 - (NdotRd * NdotRd));
        if (c > 1) ray.direction = splat(0);
        else {
            Vv = vscale(Vv, ior);
            Vv = vsfma(N, ior * -NdotRd - sqrtf(1 - c), Vv);
            ray.direction = norm(Vv);
        }
        if (ray.direction.x == 0 && ray.direction.y == 0 && ray.direction.z == 0)
            ray.direction = s.reflected_direction;
    }
    t.count(C_BOUNCE);
    t.closest.distance = t.closest.distance_squared = INFINITY;           // traceRay trace.h:89
    t.best.distance = t.best.distance_squared = INFINITY;
    return true;
}

// The end of rayTrace for a path that is done: the last glow, the tone map, and the FloatPixel the
// reference's setPixel leaves after beginDrawing's clear (viewport.h:88): hit -> (color, 1, z), miss
// -> (black, 0, +inf).
template <bool CNT, int SHS>
__device__ __forceinline__ void finish_path(TState<CNT, SHS> &t, const SceneDev &S, const ViewDev &v, const float *dirs,
                                            u32t x, u32t y, Path &p, FloatPixel *out) {
    if (v.mode == RenderMode_Beauty && S.lights && !p.lights_shaded) {
        const v3 Rd = norm(grid_direction(v, dirs, x, y));
        if (shade_lights(t, S, v.cam_pos, Rd, p.closest_distance, p.color)) {
            p.hit_found = true;
            p.z = t.sphere.closest_distance;
        }
    }
    v3 color = p.color;
    float4 c01;
    double depth;
    if (p.hit_found) {
        if (v.mode == RenderMode_Beauty) {
            color.x = tone_mapped(color.x);
            color.y = tone_mapped(color.y);
            color.z = tone_mapped(color.z);
        }
        color = vscale(color, 255.0f);
        color = vmul(color, color);
        c01 = make_float4(color.x, color.y, color.z, 1.0f);
        depth = (double)p.z;
    } else {
        c01 = make_float4(0, 0, 0, 0);
        depth = (double)INFINITY;
    }
    // streaming stores: the grid is written once and read back by a copy or the resolve, so its
    // lines go first from L2 rather than the scene's nodes (0.5 % off the 1080p mesh frame)
    float2 *o = reinterpret_cast<float2 *>(out + (size_t)y * v.grid_w + x);
    __stcs(o, make_float2(c01.x, c01.y));
    __stcs(o + 1, make_float2(c01.z, c01.w));
    __stcs(reinterpret_cast<double *>(o) + 2, depth);
}

// rayTrace render/raytracer.h:81 for one QCAA grid point.
// park (optional): at each bounce, a warp whose lanes still tracing number fewer than
// park->threshold parks those lanes' paths in the queue (returns false: the point is not finished,
// nothing is written); resume (optional): a parked path, continued from its bounce ray.  A path
// runs the same steps whether it is parked or not, so the outputs and counters do not change.
template <bool CNT, int SHS>
__device__ __forceinline__ bool trace_point(TState<CNT, SHS> &t, const SceneDev &S, const ViewDev &v, const int4 *ssb,
                                            const float *dirs, u32t x, u32t y, FloatPixel *out, u32t *prim_ids,
                                            const ParkQueue *park = nullptr,
                                            u32t view_index = 0, const ParkedRay *resume = nullptr) {
    RayD ray;
    Path p;
    bool primary = true;
    if (resume) {                                           // a parked path, at its bounce ray
        const ParkedRay &P = *resume;
        t.closest.distance = t.closest.distance_squared = INFINITY;
        t.best.distance = t.best.distance_squared = INFINITY;
        ray.origin = V(P.origin_r.x, P.origin_r.y, P.origin_r.z);
        ray.direction = V(P.direction_g.x, P.direction_g.y, P.direction_g.z);
        p.color = V(P.origin_r.w, P.direction_g.w, P.throughput_b.w);
        p.throughput = V(P.throughput_b.x, P.throughput_b.y, P.throughput_b.z);
        p.dv = P.carry.x;
        p.max_distance = P.carry.y;
        p.closest_distance = P.carry.z;
        p.z = P.carry.w;
        p.bounces = P.where.w >> 2;
        p.lights_shaded = (P.where.w >> 1) & 1u;
        p.hit_found = P.where.w & 1u;
        primary = false;
    } else {
        start_path(t, v, dirs, x, y, ray);
        start_path(p, v.depth);
    }
    // The primary ray and every bounce ray of shadeSurface's loop share this one trace site, so the
    // kernel carries one inlined copy of the walk for both (shadow rays keep theirs).
    for (;;) {
        const bool found = trace_scene(t, S, ray, false, primary ? ssb : nullptr, (int)x, (int)y,
                                       primary && !v.primary_tlas);
        if (primary && prim_ids) __stcs(prim_ids + (size_t)y * v.grid_w + x, found ? t.best.prim : 0xFFFFFFFFu);
        const bool more = shade_step(t, S, v, ray, p, primary, found);
        primary = false;
        if (!more) break;
        if (park && park->threshold) {
            // warp-vote compaction: the lanes at this bounce are the warp's lanes still tracing
            const unsigned mask = __activemask();
            const u32t n = __popc(mask);
            if (n < park->threshold) {
                const u32t lane = threadIdx.x & 31, leader = __ffs(mask) - 1;
                u32t base = 0;
                if (lane == leader) base = atomicAdd(park->reserved, n);
                base = __shfl_sync(mask, base, leader);
                const u32t slot = base + __popc(mask & ((1u << lane) - 1u));
                if (base + n <= park->capacity) {
                    ParkedRay &P = park->rays[slot];
                    P.origin_r = make_float4(ray.origin.x, ray.origin.y, ray.origin.z, p.color.x);
                    P.direction_g = make_float4(ray.direction.x, ray.direction.y, ray.direction.z, p.color.y);
                    P.throughput_b = make_float4(p.throughput.x, p.throughput.y, p.throughput.z, p.color.z);
                    P.carry = make_float4(p.dv, p.max_distance, p.closest_distance, p.z);
                    P.where = make_uint4(x, y, view_index,
                                         (p.bounces << 2) | ((u32t)p.lights_shaded << 1) | (u32t)p.hit_found);
                    return false;
                }
                // the queue is full: these paths go on here; slots of the refused range that lie
                // inside the queue are marked empty for the drain
                if (slot < park->capacity) park->rays[slot].where = make_uint4(0, 0, kEmptySlot, 0);
            }
        }
    }
    finish_path(t, S, v, dirs, x, y, p, out);
    return true;
}

template <bool CNT, int SHS>
__device__ __forceinline__ void flush_counters(TState<CNT, SHS> &t, unsigned *status, unsigned long long *counters) {
    // one flag only, so a plain store, which may go to page-locked host memory
    if (t.status) *static_cast<volatile unsigned *>(status) = t.status;
    if (CNT) {
        const u32t lane = threadIdx.x & 31;
        for (int k = 0; k < C_COUNT; k++) {
            unsigned long long s = t.cnt[k];
            for (int off = 16; off; off >>= 1) s += __shfl_down_sync(0xFFFFFFFFu, s, off);
            if (lane == 0 && s) atomicAdd(counters + k, s);
        }
    }
}

// Resident 128-thread blocks per SM the register allocation must allow: seven (72 registers).  Over
// three seeds each of the 1080p and 1001x563 mesh scenes, the moving scene and the 16-primitive scene
// the traces sum to 14.97 ms at seven, 15.21 at eight, 15.46 at nine, 15.30 at six, 15.68 at five:
// fewer registers spill more, more registers leave too few warps to cover the node loads.  Frames
// whose grid is copied to the host while they are traced and batches have the same optimum.
#ifndef ST_TRACE_MIN_BLOCKS
#define ST_TRACE_MIN_BLOCKS 7
#endif
#define ST_TRACE_BOUNDS __launch_bounds__(128, ST_TRACE_MIN_BLOCKS)
template <bool CNT>
__global__ void ST_TRACE_BOUNDS trace_kernel(SceneDev S, ViewDev v, const int4 *ssb, const float *dirs, FloatPixel *out,
                                             u32t *prim_ids, unsigned *status, unsigned long long *counters,
                                             u32t bx_first, bool from_middle) {
    const u32t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // A block covers 8x16 grid points: four 8x4 warp tiles stacked vertically.  Blocks start in launch
    // order, down the columns, so this decides which part of the frame is in flight at once, and which
    // is left when the others are done.  A frame of one launch over a scene in which no material reflects
    // or refracts starts in the middle of both sides and goes outwards: what the camera looks at is there
    // more often than not, and the margins, mostly background, fill the end (moving scene of 4096
    // primitives at 1280x720, three seeds: 1.01 to 0.97 ms against columns from the left; at 640x480 and
    // 1920x1080 within 1 %).  The same primitives in a ring round the view's axis, or all at its left
    // margin, take the same either way (within 1 %), as do depth and normals frames of scenes with mirrors,
    // which stay in column order.  Where paths bounce, the end belongs to a few long ones, wherever they
    // are: from the middle took 2 % more over six seeds of the mesh scenes, and starting the tiles first
    // that meet a reflecting or refracting primitive's screen bounds 2 % less with 6 to 10 % more for one
    // seed.  Launches beside one another (strips, batches) fill each
    // other's ends and stay in column order (served burst 2 % slower from the middle).
    u32t bx = blockIdx.y, by = blockIdx.x;
    if (from_middle) {
        bx = bx & 1 ? gridDim.y / 2 - 1 - bx / 2 : gridDim.y / 2 + bx / 2;
        by = by & 1 ? gridDim.x / 2 - 1 - by / 2 : gridDim.x / 2 + by / 2;
    }
    const u32t x = (bx + bx_first) * 8 + (lane & 7);
    const u32t y = by * 16 + warp * 4 + (lane >> 3);
    TState<CNT, 0> t;
    t.status = 0;
    if (CNT) for (int k = 0; k < C_COUNT; k++) t.cnt[k] = 0;
    if (x < v.grid_w && y < v.grid_h) trace_point(t, S, v, ssb, dirs, x, y, out, prim_ids);
    flush_counters(t, status, counters);
}

// ---- picking: manipulateSelection viewport/manipulation.h:55-123 ---------------------------------
// The ray of setRayFromCoords (shaders/common.h:170) through pixel (x, y), hitPrimitives over the TLAS
// leaf list with the visibility cull at (x, y), then every light's glow sphere (radius intensity/128,
// hitSphereSimple sphere.h:44); out (page-locked host memory): found, type, id, position, distance,
// camera-space z.  The cull is the block's, 256 leaf places at a time; what passes, a few, is tested by
// the first thread in leaf order.  (By one thread after a launch for the screen bounds, and with the
// result copied back, a pick took 34 us of 16 primitives and 1.08 ms of 4096, against 18 and 0.40.)
constexpr u32t kPickThreads = 256;
__global__ void __launch_bounds__(kPickThreads) pick_kernel(SceneDev S, ViewDev v, int x, int y, PickDev *out) {
    __shared__ u32t places[kPickThreads], sums[kPickThreads / 32];
    const u32t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int cx = (int)(uint16_t)x, cy = (int)(uint16_t)y;
    TState<false> t;
    t.status = 0;
    t.closest.distance = t.closest.distance_squared = INFINITY;       // MAX_DISTANCE base.h:164
    t.closest.cone_width = 0;
    t.best.distance = t.best.distance_squared = INFINITY;
    RayD ray;
    ray.origin = v.cam_pos;
    ray.direction = norm(vsfma(v.pp_down, (float)y, vsfma(v.pp_right, (float)x, v.pp_start)));
    bool found = false;
    for (u32t first = 0; first < S.n_prims; first += kPickThreads) {
        const u32t i = first + tid;
        bool seen = false;
        if (i < S.n_prims) {
            const int4 b = ssb_of(S, v, S.tlas_leaf_ids[i]);
            seen = cx >= b.x && cx < b.z && cy >= b.y && cy < b.w;
        }
        const unsigned mask = __ballot_sync(0xFFFFFFFFu, seen);
        if (lane == 0) sums[warp] = __popc(mask);
        __syncthreads();
        u32t at = __popc(mask & ((1u << lane) - 1u)), count = 0;
        for (u32t w = 0; w < kPickThreads / 32; w++) {
            if (w < warp) at += sums[w];
            count += sums[w];
        }
        if (seen) places[at] = i;
        __syncthreads();
        if (tid == 0) {
            SceneDev one = S;             // the leaf list from the candidate's place, one long
            one.n_prims = 1;
            for (u32t k = 0; k < count; k++) {
                one.tlas_leaf_ids = S.tlas_leaf_ids + places[k];
                found |= trace_scene(t, one, ray, false, nullptr, 0, 0, true);
            }
        }
        __syncthreads();
    }
    if (tid) return;
    if (found) finalize_hit(t, S, ray, 0.0f);
    Hit &hit = t.closest;
    for (u32t i = 0; S.lights && i < S.n_lights; i++) {
        const Light &L = S.lights[i];
        const float radius = L.intensity * (1.0f / (8.0f * 16.0f));
        t.sphere.furthest = hit.distance / radius;
        if (hit_sphere_simple(ray.origin, ray.direction, from(L.position_or_direction), 1.0f / radius, t.sphere)) {
            hit.distance = t.sphere.t_near * radius;
            hit.position = vsfma(ray.direction, hit.distance, ray.origin);
            hit.object_type = PrimitiveType_Light;
            hit.object_id = i;
            found = true;
        }
    }
    PickDev r;
    r.found = found;
    r.object_type = found ? hit.object_type : 0;
    r.object_id = found ? hit.object_id : 0;
    r.position[0] = found ? hit.position.x : 0;
    r.position[1] = found ? hit.position.y : 0;
    r.position[2] = found ? hit.position.z : 0;
    r.distance = found ? hit.distance : 0;
    r.object_distance = found ? vmat3(hit.position - ray.origin, v.cam_rot_matrix_inv).z : 0;
    *out = r;
}

// ---- batched views: one persistent launch over the tiles of many views ------------------------
// Every view is cut into tiles of tile_w x tile_h grid points (one warp per tile), and the tiles
// into groups of four that cover about 8x16 grid points (the per-frame kernel's block), numbered
// down the view's columns of groups.  A block takes `chunk` groups at a time from one global
// counter, its four warps one tile of each, so a block traces one compact region as the
// per-frame kernel's blocks do, views of different sizes, scenes and bounce counts share the
// launch, and no block idles while work is left.  (Measured on 64 views: warps taking tiles on
// their own 45.4 ms, groups numbered along the rows 43.0 ms.)
template <bool CNT, int TW, int TH, int SHS>
__global__ void ST_TRACE_BOUNDS batch_kernel(const BatchView *views, u32t n_views, u32t total_tiles, u32t chunk,
                                                    u32t *tile_counter, unsigned *status, unsigned long long *counters,
                                                    ParkQueue park) {
    static_assert(TW * TH == 32, "one warp per tile");
    constexpr u32t GW = group_tiles_w(TW), GH = 4 / GW;
    const u32t lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    __shared__ u32t stack_columns[SHS > 0 ? 2 * SHS * kTraceBlock : 1];
    __shared__ u32t block_first;
    TState<CNT, SHS> t;
    t.sh = stack_columns + threadIdx.x;
    t.status = 0;
    if (CNT) for (int k = 0; k < C_COUNT; k++) t.cnt[k] = 0;
    u32t vi = 0;       // a block's groups come in increasing order, so its view index only grows
    for (;;) {
        if (threadIdx.x == 0) block_first = atomicAdd(tile_counter, 4 * chunk);
        __syncthreads();
        const u32t first = block_first;
        __syncthreads();
        if (first >= total_tiles) break;
        const u32t last = min(first + 4 * chunk, total_tiles);
        for (u32t tile = first + warp; tile < last; tile += 4) {
            while (vi + 1 < n_views && views[vi + 1].tile_begin <= tile) vi++;
            const BatchView &B = views[vi];
            const u32t local = tile - B.tile_begin;
            const u32t group = local >> 2, q = local & 3;
            const u32t tx = (group / B.groups_y) * GW + q % GW, ty = (group % B.groups_y) * GH + q / GW;
            const u32t x = tx * TW + (lane % TW), y = ty * TH + (lane / TW);
            if (x < B.view.grid_w && y < B.view.grid_h)
                trace_point(t, B.scene, B.view, B.ssb, B.dirs, x, y, B.out, B.prim_ids, &park, vi);
        }
    }
    flush_counters(t, status, counters);
}

// The paths batch_kernel parked, continued from their bounce rays to the end and written to their
// views' outputs: a persistent grid whose warps take 32 queue slots at a time.
template <bool CNT, int SHS>
__global__ void ST_TRACE_BOUNDS drain_kernel(const BatchView *views, ParkQueue park, unsigned *status,
                                                    unsigned long long *counters) {
    const u32t lane = threadIdx.x & 31;
    __shared__ u32t stack_columns[SHS > 0 ? 2 * SHS * kTraceBlock : 1];
    TState<CNT, SHS> t;
    t.sh = stack_columns + threadIdx.x;
    t.status = 0;
    if (CNT) for (int k = 0; k < C_COUNT; k++) t.cnt[k] = 0;
    const u32t n = min(*park.reserved, park.capacity);
    u32t drained = 0;
    for (;;) {
        u32t first = 0;
        if (lane == 0) first = atomicAdd(park.taken, 32u);
        first = __shfl_sync(0xFFFFFFFFu, first, 0);
        if (first >= n) break;
        const u32t i = first + lane;
        if (i < n) {
            const ParkedRay P = park.rays[i];
            if (P.where.z != kEmptySlot) {
                const BatchView &B = views[P.where.z];
                trace_point(t, B.scene, B.view, B.ssb, B.dirs, P.where.x, P.where.y, B.out, nullptr, nullptr, 0, &P);
                drained++;
            }
        }
    }
    for (int off = 16; off; off >>= 1) drained += __shfl_down_sync(0xFFFFFFFFu, drained, off);
    if (lane == 0 && drained) atomicAdd(park.drained, drained);
    flush_counters(t, status, counters);
}

// drawViewportToWindowContent viewport/viewport.h:12 (QCAA branch): the 2x2 corners' colour times
// opacity, averaged, square-rooted in double, truncated to u8; all-infinite corners -> background.
__device__ __forceinline__ void resolve_one(const FloatPixel *in, u32t grid_w, u32t width, uint32_t *out, u32t x, u32t y) {
    const FloatPixel TL = in[(size_t)y * grid_w + x], TR = in[(size_t)y * grid_w + x + 1];
    const FloatPixel BL = in[(size_t)(y + 1) * grid_w + x], BR = in[(size_t)(y + 1) * grid_w + x + 1];
    uint32_t px;
    if (BL.depth == INFINITY && BR.depth == INFINITY && TL.depth == INFINITY && TR.depth == INFINITY) {
        px = 0xFF000000u;
    } else {
        v3 c = vscale(vsfma(from(TL.color), TL.opacity, vsfma(from(TR.color), TR.opacity,
                      vsfma(from(BL.color), BL.opacity, vscale(from(BR.color), BR.opacity)))), 0.25f);
        unsigned R = (unsigned char)(c.x > (255 * 255) ? 255.0 : sqrt((double)c.x));
        unsigned G = (unsigned char)(c.y > (255 * 255) ? 255.0 : sqrt((double)c.y));
        unsigned B = (unsigned char)(c.z > (255 * 255) ? 255.0 : sqrt((double)c.z));
        px = B | (G << 8) | (R << 16) | 0xFF000000u;
    }
    out[(size_t)y * width + x] = px;
}
// Pixel columns [x0, x1) of the frame (pixel x reads grid columns x and x + 1), one thread per
// pixel along the rows of the range, so that a narrow range leaves no block mostly idle.
__global__ void resolve_kernel(const FloatPixel *in, u32t grid_w, u32t width, u32t height, uint32_t *out, u32t x0,
                               u32t x1) {
    const u32t n = x1 - x0;
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const u32t y = (u32t)(i / n), x = x0 + (u32t)(i % n);
    if (y < height) resolve_one(in, grid_w, width, out, x, y);
}

// ---- a batch's per-view set-up and resolve, driven by the view table (one launch each) ----------
__global__ void batch_setup_kernel(const BatchTable T, u32t n_views, u32t row_blocks) {
    const u32t vi = blockIdx.y;
    if (vi >= n_views) return;
    const BatchView &B = T.v[vi];
    setup_one(B.scene, B.view, const_cast<int4 *>(B.ssb), const_cast<float *>(B.dirs), blockIdx.x, row_blocks);
}
__global__ void batch_resolve_kernel(const BatchTable T, u32t n_views) {
    const u32t vi = blockIdx.z, x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y;
    if (vi >= n_views) return;
    const BatchView &B = T.v[vi];
    if (B.out_u8 && x + 1 < B.view.grid_w && y + 1 < B.view.grid_h)
        resolve_one(B.out, B.view.grid_w, B.view.grid_w - 1, B.out_u8, x, y);
}

// ---- launchers -------------------------------------------------------------------------------
void launch_frame_setup(const SceneDev &S, const ViewDev &v, int4 *ssb, float *dirs, cudaStream_t st) {
    const u32t rows = (v.grid_h + kSetupThreads - 1) / kSetupThreads;
    frame_setup_kernel<<<rows + (S.n_prims + kSetupThreads - 1) / kSetupThreads, kSetupThreads, 0, st>>>(S, v, ssb, dirs, rows);
}
void launch_trace(const SceneDev &S, const ViewDev &v, const int4 *ssb, const float *dirs, FloatPixel *out,
                  u32t *prim_ids, unsigned *status, unsigned long long *counters, bool count, cudaStream_t st,
                  bool from_middle, u32t bx_first, u32t bx_count) {
    const u32t bw = (v.grid_w + 7) / 8, bh = (v.grid_h + 15) / 16;
    if (bx_first >= bw) return;
    if (!bx_count || bx_first + bx_count > bw) bx_count = bw - bx_first;
    const dim3 grid(bh, bx_count);
    if (count) trace_kernel<true><<<grid, 128, 0, st>>>(S, v, ssb, dirs, out, prim_ids, status, counters, bx_first, from_middle);
    else trace_kernel<false><<<grid, 128, 0, st>>>(S, v, ssb, dirs, out, prim_ids, status, counters, bx_first, from_middle);
}
int launch_batch(const BatchView *views, u32t n_views, u32t total_tiles, int variant, u32t chunk, u32t grid_blocks,
                 u32t *tile_counter, unsigned *status, unsigned long long *counters, bool count, cudaStream_t st,
                 const ParkQueue &park) {
#define ST_BATCH(TW, TH, SHS) (count ? (batch_kernel<true, TW, TH, SHS><<<grid_blocks, 128, 0, st>>>(views, n_views, total_tiles, chunk, tile_counter, status, counters, park), 0) \
                                     : (batch_kernel<false, TW, TH, SHS><<<grid_blocks, 128, 0, st>>>(views, n_views, total_tiles, chunk, tile_counter, status, counters, park), 0))
#define ST_BATCH_STACKS(TW, TH) (variant_stack(variant) ? ST_BATCH(TW, TH, kSharedStackEntries) : ST_BATCH(TW, TH, 0))
    if (variant < 0 || variant >= BATCH_VARIANTS) return -1;
    switch (variant_tile(variant)) {
        case TILE_8x4: return ST_BATCH_STACKS(8, 4);
        case TILE_16x2: return ST_BATCH_STACKS(16, 2);
        case TILE_32x1: return ST_BATCH_STACKS(32, 1);
        case TILE_4x8: return ST_BATCH_STACKS(4, 8);
    }
#undef ST_BATCH_STACKS
#undef ST_BATCH
    return -1;
}
int launch_drain(const BatchView *views, const ParkQueue &park, int variant, u32t grid_blocks, unsigned *status,
                 unsigned long long *counters, bool count, cudaStream_t st) {
    if (variant < 0 || variant >= BATCH_VARIANTS) return -1;
    const bool shared_stacks = variant_stack(variant) != 0;
    if (count) {
        if (shared_stacks) drain_kernel<true, kSharedStackEntries><<<grid_blocks, 128, 0, st>>>(views, park, status, counters);
        else drain_kernel<true, 0><<<grid_blocks, 128, 0, st>>>(views, park, status, counters);
    } else {
        if (shared_stacks) drain_kernel<false, kSharedStackEntries><<<grid_blocks, 128, 0, st>>>(views, park, status, counters);
        else drain_kernel<false, 0><<<grid_blocks, 128, 0, st>>>(views, park, status, counters);
    }
    return 0;
}
int batch_blocks_per_sm(int variant) {
    int n = 0;
#define ST_OCC(TW, TH) (variant_stack(variant) \
        ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, batch_kernel<false, TW, TH, kSharedStackEntries>, 128, 0) \
        : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, batch_kernel<false, TW, TH, 0>, 128, 0))
    switch (variant_tile(variant)) {
        case TILE_16x2: ST_OCC(16, 2); break;
        case TILE_32x1: ST_OCC(32, 1); break;
        case TILE_4x8: ST_OCC(4, 8); break;
        default: ST_OCC(8, 4); break;
    }
#undef ST_OCC
    return n > 0 ? n : 1;
}
void tile_dims(int variant, u32t &tw, u32t &th) {
    switch (variant_tile(variant)) {
        case TILE_16x2: tw = 16; th = 2; return;
        case TILE_32x1: tw = 32; th = 1; return;
        case TILE_4x8: tw = 4; th = 8; return;
        default: tw = 8; th = 4; return;
    }
}
void launch_pick(const SceneDev &S, const ViewDev &v, int x, int y, PickDev *out, cudaStream_t st) {
    pick_kernel<<<1, kPickThreads, 0, st>>>(S, v, x, y, out);
}
void launch_batch_setup(const BatchTable &T, u32t n_views, u32t max_prims, u32t max_rows, cudaStream_t st) {
    const u32t rows = (max_rows + kSetupThreads - 1) / kSetupThreads;
    batch_setup_kernel<<<dim3(rows + (max_prims + kSetupThreads - 1) / kSetupThreads, n_views), kSetupThreads, 0, st>>>(T, n_views, rows);
}
void launch_batch_resolve(const BatchTable &T, u32t n_views, u32t max_width, u32t max_height, cudaStream_t st) {
    batch_resolve_kernel<<<dim3((max_width + 127) / 128, max_height, n_views), 128, 0, st>>>(T, n_views);
}
void launch_resolve(const FloatPixel *in, u32t grid_w, u32t width, u32t height, uint32_t *out, cudaStream_t st,
                    u32t x0, u32t x1) {
    if (x1 > width) x1 = width;
    if (x0 >= x1 || !height) return;
    const size_t pixels = (size_t)(x1 - x0) * height;
    resolve_kernel<<<(unsigned)((pixels + 255) / 256), 256, 0, st>>>(in, grid_w, width, height, out, x0, x1);
}

}  // namespace st
