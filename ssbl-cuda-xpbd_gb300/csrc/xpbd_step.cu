// Per-vertex kernels of one XPBD substep: prediction, the fused constraint /
// contact pass, bends per colour, and the position pack for downloads.
//
// The reference launches one kernel per stage over every vertex or
// constraint (native/src/ssbl_xpbd_cuda_abi41.cu:9165-9376): integrate, pins,
// springs (float atomics into pos), pins, analytic contacts, SDF contacts,
// pins, velocity.  Pins, analytic contacts, SDF contacts and the velocity
// update only read and write the vertex they act on, so this library runs
// them as stages of one per-vertex kernel.  Stretch (and the once-per-frame
// tethers) become a gather over a vertex->constraint CSR that reads a
// snapshot of the positions (ping-pong buffer) and sums the corrections of
// the incident constraints in constraint order: the same snapshot-Jacobi
// update as the reference's atomics, without float atomics, and therefore
// deterministic.
#include "xpbd_constraint.cuh"
#include <algorithm>
#include <initializer_list>

#include "xpbd_cluster.cuh"
#include "xpbd_contact.cuh"
#include "xpbd_fields.cuh"
#include "xpbd_solver.cuh"

namespace xg {

namespace {

struct VState {
    F3 p, prev, vel;
    float w;  // effective inverse mass
};

// Weighted pin projection of one vertex (abi41.cu:3466-3509).  Pins are
// stored per vertex (weight -1 = no pin; a vertex listed twice keeps its last
// entry) and the relaxation 1 - (1 - s)^(1/(I+1)) is precomputed on the host.
__device__ __forceinline__ void pin_apply(float weight, F3 target, float relax, float inv_mass, float dt, VState* s) {
    if (!isfinite(weight) || weight < 0.05f) return;
    if (weight >= 0.75f || inv_mass <= 0.0f) {
        s->p = target;
        s->prev = target;
        s->vel = F3{0.0f, 0.0f, 0.0f};
        return;
    }
    if (relax <= 0.0f) return;
    const F3 corrected = s->p + (target - s->p) * relax;
    const F3 damped = s->vel * fmaxf(1.0f - relax, 0.0f);
    s->p = corrected;
    s->prev = corrected - damped * fmaxf(dt, kEps);
    s->vel = damped;
}

__device__ void pin_stage(const View& v, int i, float inv_mass, float dt, VState* s) {
    const float weight = __ldg(&v.pin_weight[i]);
    if (!isfinite(weight) || weight < 0.05f) return;
    pin_apply(weight, f3(ld4(&v.pin_target[i])), __ldg(&v.pin_relax[i]), inv_mass, dt, s);
}

// Ground plane (z up), sphere and wall (abi41.cu:3511-3590).
__device__ void analytic_stage(const Params& P, unsigned long long* counts, float inv_mass, float dt, VState* s) {
    if (inv_mass <= 0.0f) return;
    F3 p = s->p;
    F3 vel = s->vel;
    bool contacted = false;
    const float margin = fmaxf(P.margin, 0.0f);
    const float sdt = fmaxf(dt, kEps);
    if (P.use_ground && p.z < P.ground_height + margin) {
        const float target_z = P.ground_height + margin;
        const float pen = target_z - p.z;
        const F3 n{0.0f, 0.0f, 1.0f};
        const float inward = fmaxf(-dot3(vel, n), 0.0f);
        p.z = target_z;
        contact_response(P, counts, n, inward + pen / sdt, &vel);
        contacted = true;
    }
    if (P.use_sphere && P.sphere_radius > 0.0f) {
        const F3 c{P.sphere_center[0], P.sphere_center[1], P.sphere_center[2]};
        const F3 d = p - c;
        const float dist = sqrtf(fmaxf(dot3(d, d), kEps));
        const float target = P.sphere_radius + margin;
        if (dist < target) {
            const F3 n = dist > kEps ? d * (1.0f / dist) : F3{0.0f, 0.0f, 1.0f};
            const float pen = target - dist;
            const float inward = fmaxf(-dot3(vel, n), 0.0f);
            p = c + n * target;
            contact_response(P, counts, n, inward + pen / sdt, &vel);
            contacted = true;
        }
    }
    if (P.use_wall) {
        const F3 o{P.wall_origin[0], P.wall_origin[1], P.wall_origin[2]};
        F3 n{P.wall_normal[0], P.wall_normal[1], P.wall_normal[2]};
        const float nlen = sqrtf(fmaxf(dot3(n, n), kEps));
        n = n * (1.0f / nlen);
        const float gap = dot3(p - o, n);
        if (gap < margin) {
            const float pen = margin - gap;
            const float inward = fmaxf(-dot3(vel, n), 0.0f);
            p = p + n * (margin - gap);
            contact_response(P, counts, n, inward + pen / sdt, &vel);
            contacted = true;
        }
    }
    s->p = p;
    if (contacted) {
        s->vel = vel;
        s->prev = p - vel * sdt;
    }
}

__device__ __forceinline__ int sdf_index(const Params& P, int x, int y, int z) {
    return (z * P.sdf_dim[1] + y) * P.sdf_dim[0] + x;
}

__device__ __forceinline__ float lerpf(float a, float b, float t) { return a + (b - a) * t; }

__device__ float sdf_trilinear(const Params& P, const float* sdf, float gx, float gy, float gz) {
    const int x0 = min(max((int)floorf(gx), 0), P.sdf_dim[0] - 1);
    const int y0 = min(max((int)floorf(gy), 0), P.sdf_dim[1] - 1);
    const int z0 = min(max((int)floorf(gz), 0), P.sdf_dim[2] - 1);
    const int x1 = min(x0 + 1, P.sdf_dim[0] - 1);
    const int y1 = min(y0 + 1, P.sdf_dim[1] - 1);
    const int z1 = min(z0 + 1, P.sdf_dim[2] - 1);
    const float tx = gx - (float)x0, ty = gy - (float)y0, tz = gz - (float)z0;
    const float c000 = __ldg(&sdf[sdf_index(P, x0, y0, z0)]);
    const float c100 = __ldg(&sdf[sdf_index(P, x1, y0, z0)]);
    const float c010 = __ldg(&sdf[sdf_index(P, x0, y1, z0)]);
    const float c110 = __ldg(&sdf[sdf_index(P, x1, y1, z0)]);
    const float c001 = __ldg(&sdf[sdf_index(P, x0, y0, z1)]);
    const float c101 = __ldg(&sdf[sdf_index(P, x1, y0, z1)]);
    const float c011 = __ldg(&sdf[sdf_index(P, x0, y1, z1)]);
    const float c111 = __ldg(&sdf[sdf_index(P, x1, y1, z1)]);
    const float c0 = lerpf(lerpf(c000, c100, tx), lerpf(c010, c110, tx), ty);
    const float c1 = lerpf(lerpf(c001, c101, tx), lerpf(c011, c111, tx), ty);
    return lerpf(c0, c1, tz);
}

// Trilinear sample inside the grid, false outside (abi41.cu:1645-1691).
__device__ bool sdf_sample(const Params& P, const float* sdf, F3 p, float* out) {
    if (P.sdf_dim[0] < 2 || P.sdf_dim[1] < 2 || P.sdf_dim[2] < 2 || P.sdf_voxel <= 0.0f) return false;
    const float inv = 1.0f / P.sdf_voxel;
    const float gx = (p.x - P.sdf_origin[0]) * inv;
    const float gy = (p.y - P.sdf_origin[1]) * inv;
    const float gz = (p.z - P.sdf_origin[2]) * inv;
    if (gx < 0.0f || gy < 0.0f || gz < 0.0f || gx > (float)(P.sdf_dim[0] - 1) || gy > (float)(P.sdf_dim[1] - 1) ||
        gz > (float)(P.sdf_dim[2] - 1))
        return false;
    *out = sdf_trilinear(P, sdf, gx, gy, gz);
    return isfinite(*out);
}

// Sample with the point clamped into the grid (abi41.cu:1693-1723).
__device__ float sdf_sample_clamped(const Params& P, const float* sdf, F3 p) {
    const float inv = 1.0f / fmaxf(P.sdf_voxel, kEps);
    const float gx = fminf(fmaxf((p.x - P.sdf_origin[0]) * inv, 0.0f), (float)(P.sdf_dim[0] - 1));
    const float gy = fminf(fmaxf((p.y - P.sdf_origin[1]) * inv, 0.0f), (float)(P.sdf_dim[1] - 1));
    const float gz = fminf(fmaxf((p.z - P.sdf_origin[2]) * inv, 0.0f), (float)(P.sdf_dim[2] - 1));
    return sdf_trilinear(P, sdf, gx, gy, gz);
}

// Normal of the nearest static triangle, used when the SDF gradient vanishes
// (abi41.cu:1749-1769).
__device__ F3 nearest_static_normal(const Params& P, const float4* tris, F3 p) {
    F3 best{0.0f, 0.0f, 1.0f};
    float best_sq = 3.402823466e+38f;
    for (int t = 0; t < P.static_tri_count; ++t) {
        const F3 a = f3(ld4(&tris[t * 3 + 0])), b = f3(ld4(&tris[t * 3 + 1])), c = f3(ld4(&tris[t * 3 + 2]));
        const F3 d = p - closest_on_triangle(p, a, b, c);
        const float dsq = dot3(d, d);
        if (dsq < best_sq) {
            best_sq = dsq;
            best = dsq > kEps * kEps ? normalize_or(d, best) : normalize_or(cross3(b - a, c - a), best);
        }
    }
    return normalize_or(best, F3{0.0f, 0.0f, 1.0f});
}

// Central-difference SDF gradient (abi41.cu:1771-1785).
__device__ F3 sdf_normal(const Params& P, const float* sdf, const float4* tris, F3 p) {
    const float h = fmaxf(P.sdf_voxel, 1.0e-5f);
    const float dx = sdf_sample_clamped(P, sdf, p + F3{h, 0.0f, 0.0f}) - sdf_sample_clamped(P, sdf, p + F3{-h, 0.0f, 0.0f});
    const float dy = sdf_sample_clamped(P, sdf, p + F3{0.0f, h, 0.0f}) - sdf_sample_clamped(P, sdf, p + F3{0.0f, -h, 0.0f});
    const float dz = sdf_sample_clamped(P, sdf, p + F3{0.0f, 0.0f, h}) - sdf_sample_clamped(P, sdf, p + F3{0.0f, 0.0f, -h});
    const F3 n{dx, dy, dz};
    const float lsq = dot3(n, n);
    if (!isfinite(lsq) || lsq <= 1.0e-12f) return nearest_static_normal(P, tris, p);
    return n * (1.0f / sqrtf(lsq));
}

// Static SDF contact (abi41.cu:1831-1867).
__device__ void sdf_stage(const View& v, const Params& P, float inv_mass, float dt, VState* s) {
    if (inv_mass <= 0.0f || !P.sdf_ready) return;
    const float margin = fmaxf(P.margin, 0.0f);
    if (margin <= 0.0f) return;
    float d = 0.0f;
    if (!sdf_sample(P, P.sdf, s->p, &d) || d >= margin) return;
    const F3 n = sdf_normal(P, P.sdf, P.static_tris, s->p);
    if (!finite3(n)) return;
    const float pen = margin - d;
    if (!isfinite(pen) || pen <= 0.0f) return;
    const F3 corrected = s->p + n * pen;
    F3 vel = s->vel;
    const float inward = fmaxf(-dot3(vel, n), 0.0f);
    contact_response(P, v.counts, n, inward + pen / fmaxf(dt, kEps), &vel);
    s->p = corrected;
    s->vel = vel;
    s->prev = corrected - vel * fmaxf(dt, kEps);
    count1(v.counts, kCntStaticSdfContacts);
}

// v = v + feedback(measured - v) with the aligned-feedback clamp
// (abi41.cu:5846-5884); the arithmetic is velocity_update.
__device__ void velocity_stage(const Params& P, float dt, VState* s) {
    s->vel = velocity_update(s->p, s->prev, s->vel, s->w, P.thickness, dt);
}

// Stretch constraint of edge (i, j) seen from one of its endpoints
// (abi41.cu:1927-1980): the correction is computed in the edge's own
// orientation so both endpoints get bit-identical values.
__device__ __forceinline__ void spring_term(unsigned long long* counts, float alpha, float4 pi, float4 pj, float rest,
                                            bool self_is_j, F3* dp, F3* dprev) {
    F3 corr;
    float c;
    bool clamped;
    if (!stretch_correction(pi, pj, rest, alpha, &corr, &c, &clamped)) return;
    if (clamped && !self_is_j) count1(counts, kCntHardFallbacks);
    const float wi = pi.w, wj = pj.w;
    const float wself = self_is_j ? wj : wi;
    if (wself > 0.0f) {
        const F3 d = self_is_j ? corr * wj : corr * (-wi);
        *dp = *dp + d;
        if (c > 0.0f) *dprev = *dprev + d * 0.08f;
    }
}

// Long-range tether (anchor i, dynamic j) seen from one endpoint
// (abi41.cu:2710-2803).
__device__ __forceinline__ void tether_term(const Params& P, unsigned long long* counts, float dt, float4 pi4, float4 pj4,
                                            float rest, bool self_is_j, bool by_dynamic, F3* dp, F3* dprev) {
    const bool counter = self_is_j == by_dynamic;  // count once per tether
    const float wi = pi4.w, wj = pj4.w;
    const float weight = wi + wj;
    if (!isfinite(weight) || weight <= 0.0f) {
        if (counter) count1(counts, kCntTackGuards);
        return;
    }
    const F3 pi = f3(pi4), pj = f3(pj4);
    if (!finite3(pi) || !finite3(pj)) {
        if (counter) count1(counts, kCntTackGuards);
        return;
    }
    F3 dx = pj - pi;
    const float len_sq = len_sq_xyz(dx);
    if (!isfinite(len_sq) || len_sq <= 1.0e-10f || !isfinite(rest) || rest <= kEps) {
        if (counter) count1(counts, kCntTackGuards);
        return;
    }
    const float inv_len = 1.0f / sqrtf(len_sq);
    const float len = len_sq * inv_len;
    const float stretch = len - rest;
    if (!isfinite(stretch) || stretch <= 0.0f) return;
    dx = dx * inv_len;
    const float base_c = fmaxf(P.lra_compliance, 1.0e-12f);
    const float stiff = (1.0f / base_c) * 500000.0f;
    const float alpha = (base_c / 500000.0f) / fmaxf(dt * dt, kEps);
    const float sw = stiff / fmaxf(stiff + 500000.0f, 1.0f);
    const float dlambda = -stretch / fmaxf(weight + alpha, kEps);
    F3 corr = dx * (0.35f * sw * dlambda);
    if (!finite3(corr)) {
        if (counter) count1(counts, kCntTackGuards);
        return;
    }
    const float corr_len = len3(corr);
    const float max_corr = fmaxf(5.0e-4f, fminf(fmaxf(rest, P.thickness) * 0.20f, 0.035f));
    if (!isfinite(corr_len) || corr_len <= 0.0f) return;
    if (corr_len > max_corr) {
        corr = corr * (max_corr / fmaxf(corr_len, kEps));
        if (counter) count1(counts, kCntTackGuards);
    }
    const bool has_th = P.thickness > 0.0f;
    const float cap = has_th ? 0.0025f : 0.012f;
    const float rest_limit = fmaxf(rest, 0.0f) * (has_th ? 0.02f : 0.08f);
    const float th_limit = has_th ? P.thickness * 0.12f : cap;
    const float applied = fmaxf(5.0e-4f, fminf(fminf(rest_limit, th_limit), cap));
    if (self_is_j) {
        if (wj > 0.0f) {
            const F3 d = limit_delta(corr * (wj / fmaxf(weight, kEps)), applied);
            *dp = *dp + d;
            *dprev = *dprev + d * 0.32f;
        }
    } else if (wi > 0.0f) {
        const F3 d = limit_delta(corr * (-wi / fmaxf(weight, kEps)), applied);
        *dp = *dp + d;
        *dprev = *dprev + d * 0.32f;
    }
    if (counter) count1(counts, kCntLraTacks);
}

// Bend distance constraint between the two wing-opposite vertices, shared by
// the per-colour kernel and the Jacobi gather used when no colours are given
// (abi41.cu:2805-2884 and 2886-2970).  Returns false when the constraint is
// skipped; `guard` is set when the reference would count a guard.
__device__ __forceinline__ bool bend_correction(const Params& P, float dt, float4 pi4, float4 pj4, float rest, F3* corr_out,
                                                bool* guard) {
    bool clamped;
    return bend_correction_k(pi4, pj4, rest, P.bend_compliance, P.thickness, dt, corr_out, guard, &clamped);
}

__device__ __forceinline__ void bend_term(const Params& P, unsigned long long* counts, float dt, float4 pi, float4 pj,
                                          float rest, bool self_is_j, F3* dp, F3* dprev) {
    F3 corr;
    bool guard;
    const bool applied = bend_correction(P, dt, pi, pj, rest, &corr, &guard);
    if (!self_is_j) {
        if (guard) count1(counts, kCntBendingGuards);
        if (applied) count1(counts, kCntBendingWings);
    }
    if (!applied) return;
    const float wself = self_is_j ? pj.w : pi.w;
    if (wself > 0.0f) {
        const F3 d = self_is_j ? corr * pj.w : corr * (-pi.w);
        *dp = *dp + d;
        *dprev = *dprev + d * 0.06f;
    }
}

// Area-weighted normal of a vertex from its incident triangles in the
// snapshot positions (abi41.cu:1213-1261; 1/sqrt in IEEE arithmetic).
__device__ bool vertex_normal(const View& v, int i, F3* out) {
    if (!v.vt_off) return false;
    const int begin = __ldg(&v.vt_off[i]), end = __ldg(&v.vt_off[i + 1]);
    if (end <= begin) return false;
    F3 acc{0.0f, 0.0f, 0.0f};
    for (int k = begin; k < end; ++k) {
        const int t = __ldg(&v.vt_tri[k]);
        if (t < 0 || t >= v.nT) continue;
        const int4 tr = __ldg(&v.tris[t]);
        if (tr.x < 0 || tr.y < 0 || tr.z < 0 || tr.x >= v.nV || tr.y >= v.nV || tr.z >= v.nV) continue;
        const F3 p0 = f3(v.pos_in[tr.x]), p1 = f3(v.pos_in[tr.y]), p2 = f3(v.pos_in[tr.z]);
        const F3 n = cross3(p1 - p0, p2 - p0);
        const float l2 = dot3(n, n);
        if (!isfinite(l2) || l2 <= 1.0e-10f) continue;
        acc = acc + n * (1.0f / sqrtf(l2));
    }
    const float a2 = dot3(acc, acc);
    if (!isfinite(a2) || a2 <= 1.0e-10f) return false;
    *out = acc * (1.0f / sqrtf(a2));
    return true;
}

// The prediction of a free vertex without force fields or volume pressure.
__device__ __forceinline__ void predict_free(const Params& P, float dt, VState* s) {
    const F3 accel = F3{P.gravity[0], P.gravity[1], P.gravity[2]} + F3{0.0f, 0.0f, 0.0f};
    F3 vel = s->vel + accel * dt;
    vel = vel * P.damping;
    s->vel = vel;
    s->p = s->p + vel * dt;
}

// Integrate (abi41.cu:1869-1925): gravity, volume pressure along the vertex
// normal, force fields, damping, pressure speed trims; fixed vertices return
// to rest.  Reads the snapshot `pos_in` and writes `pos` (the same buffer
// unless vertex normals are gathered).
__device__ __forceinline__ void predict_item(const View& v, int i) {
    const Params& P = params_v(v, i);
    const float4 p4 = v.pos_in[i];
    if (!P.active) {
        if (v.pos != v.pos_in) v.pos[i] = p4;
        return;
    }
    const float dt = P.sub_dt;
    const float inv_mass = __ldg(&v.inv_mass[i]);
    VState s;
    s.w = p4.w;
    s.prev = f3(p4);
    if (!(p4.w > 0.0f)) {
        s.vel = F3{0.0f, 0.0f, 0.0f};
        s.p = f3(ld4(&v.rest[i]));
    } else {
        F3 normal{0.0f, 0.0f, 0.0f};
        const bool has_normal = P.needs_normal && vertex_normal(v, i, &normal);
        F3 accel = F3{P.gravity[0], P.gravity[1], P.gravity[2]} + F3{0.0f, 0.0f, 0.0f};
        const bool pressure = P.pressure_on && has_normal;
        const float area = pressure ? __ldg(&v.p_area[i]) : 0.0f;
        if (pressure && isfinite(area) && area > 0.0f)
            accel = accel + normal * (P.pressure_strength * P.pressure_accel_scale * area * inv_mass);
        if (P.field_count > 0) {
            F3 fa{0.0f, 0.0f, 0.0f};
            const F3 vel0 = f3(v.vel[i]);
            const int n = min(P.field_count, kMaxFields);
            for (int k = 0; k < n; ++k) fa = fa + field_accel(P.fields[k], f3(p4), vel0, normal, has_normal);
            accel = accel + cap_field_accel(fa);
        }
        F3 vel = f3(v.vel[i]) + accel * dt;
        vel = vel * P.damping;
        if (pressure) {
            const float rest = __ldg(&v.p_rest[i]);
            if (isfinite(rest) && rest > kEps && isfinite(dt) && dt > kEps) {
                const float pa = fmaxf(P.pressure_strength, 0.0f) * fmaxf(P.pressure_accel_scale, 0.0f) * fmaxf(area, 0.0f) *
                                 fmaxf(inv_mass, 0.0f);
                const float max_delta = fmaxf(rest * fmaxf(P.pressure_impulse_rest_scale, 0.0f), 1.0e-7f);
                const float delta = pa * dt * dt;
                if (isfinite(delta) && delta > max_delta) vel = vel - normal * ((delta - max_delta) / dt);
                const float vrest = fmaxf(rest, fmaxf(P.pressure_velocity_length_scale, 0.0f));
                const float max_out = fmaxf(vrest * fmaxf(P.pressure_velocity_rest_scale, 0.0f) / dt, 1.0e-6f);
                const float out = dot3(vel, normal);
                if (isfinite(out) && out > max_out) vel = vel - normal * (out - max_out);
            }
        }
        s.vel = vel;
        s.p = f3(p4) + vel * dt;
    }
    pin_stage(v, i, inv_mass, dt, &s);
    v.pos[i] = f4(s.p, s.w);
    v.prev[i] = f4(s.prev, 0.0f);
    v.vel[i] = f4(s.vel, 0.0f);
}

__global__ void __launch_bounds__(kThreads) k_predict(View v) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < v.nV) predict_item(v, i);
}

// Average of a vertex's accumulated self-collision pushes, clamped to 0.35 r,
// applied with a 0.55 prev shift; the accumulators are cleared for the next
// pass (abi41.cu:4953-4988).
__device__ __forceinline__ void apply_pushes(const View& v, const Params& P, int i, float inv_mass, VState* s) {
    const Acc4 a = v.acc[i];
    if (a.w == 0) return;  // every push adds a weight: nothing accumulated, the row is still zero
    v.acc[i] = Acc4{0, 0, 0, 0};
    if (!(inv_mass > 0.0f) || a.w <= 0) return;
    F3 avg = F3{from_fix(a.x), from_fix(a.y), from_fix(a.z)} * (1.0f / (float)a.w);
    const float max_delta = fmaxf(P.self_radius * 0.35f, 1.0e-4f);
    const float dl = len3(avg);
    if (dl > max_delta) avg = avg * (max_delta / dl);
    s->p = s->p + avg;
    s->prev = s->prev + avg * 0.55f;
    const float al = len3(avg);
    if (al > 0.0f) atomicMax(v.max_delta_bits, __float_as_uint(al));
}

// The stages of a pass after its gather, and the vertex's rows.
__device__ __forceinline__ void finish_vertex(const View& v, const Params& P, int i, unsigned flags, float inv_mass, float dt, VState* st) {
    VState& s = *st;
    if (flags & kPassApply) apply_pushes(v, P, i, inv_mass, &s);
    if (flags & kPassPin) pin_stage(v, i, inv_mass, dt, &s);
    if (flags & kPassAnalytic) analytic_stage(P, v.counts, inv_mass, dt, &s);
    if (flags & kPassSdf) sdf_stage(v, P, inv_mass, dt, &s);
    // final pin polish when this cloth ran a contact stage in this iteration
    // (analytic colliders, SDF, or any last iteration; abi41.cu:9360-9369)
    if ((flags & kPassPinPolish) &&
        (v.last_it || P.use_ground || P.use_wall || P.use_sphere || P.sdf_ready))
        pin_stage(v, i, inv_mass, dt, &s);
    if (flags & kPassVelocity) velocity_stage(P, dt, &s);
    if (flags & kPassPredict) {
        // the next substep's prediction (predict_item without vertex normals)
        s.prev = s.p;
        if (!(s.w > 0.0f)) {
            s.vel = F3{0.0f, 0.0f, 0.0f};
            s.p = f3(ld4(&v.rest[i]));
        } else {
            predict_free(P, dt, &s);
        }
        pin_stage(v, i, inv_mass, dt, &s);
    }
    v.pos[i] = f4(s.p, s.w);
    v.prev[i] = f4(s.prev, 0.0f);
    v.vel[i] = f4(s.vel, 0.0f);
}


__device__ __forceinline__ void vertex_pass_item(const View& v, int i, unsigned flags) {
    const Params& P = params_v(v, i);
    const float dt = P.sub_dt;
    const float4 p4 = v.pos_in[i];
    if (!P.active) {
        if (v.pos != v.pos_in) v.pos[i] = p4;  // keep the ping-pong buffers in step
        return;
    }
    VState s;
    s.w = p4.w;
    s.p = f3(p4);
    s.prev = f3(v.prev[i]);
    s.vel = f3(v.vel[i]);
    const float inv_mass = __ldg(&v.inv_mass[i]);
    // a cloth with the CG stretch solve has no spring gather (in a batch the
    // pass still carries its vertices to the other buffer)
    const unsigned gather = flags & (P.pcg_on ? (kPassTether | kPassBend) : (kPassSpring | kPassTether | kPassBend));
    if (gather) {
        const int kind = (gather & kPassSpring) ? 0 : ((gather & kPassTether) ? 1 : 2);
        const int* off = kind == 0 ? v.sp_off : (kind == 1 ? v.te_off : v.bj_off);
        const int2* ent = kind == 0 ? v.sp_ent : (kind == 1 ? v.te_ent : v.bj_ent);
        // Where every tether's dynamic end is free, that end counts the
        // tether and a fixed vertex skips its own: it gets nothing from them,
        // and the anchor of a whole cloth has one to every free vertex (a
        // 1,000-entry walk by one thread, 0.1 ms per frame of a 32 x 32 cloth).
        const bool skip = kind == 1 && v.te_free && !(p4.w > 0.0f);
        const int begin = __ldg(&off[i]), end = skip ? begin : __ldg(&off[i + 1]);
        const float alpha = stretch_alpha(P.stretch_compliance, dt);
        F3 dp = s.p, dprev = s.prev;
        for (int k = begin; k < end; ++k) {
            const int2 e = __ldg(&ent[k]);
            const bool self_is_j = (e.x & kSideBit) != 0;
            const float4 q4 = v.pos_in[e.x & 0x7fffffff];
            const float rest = __int_as_float(e.y);
            const float4 pi = self_is_j ? q4 : p4;
            const float4 pj = self_is_j ? p4 : q4;
            if (kind == 0)
                spring_term(v.counts, alpha, pi, pj, rest, self_is_j, &dp, &dprev);
            else if (kind == 1)
                tether_term(P, v.counts, dt, pi, pj, rest, self_is_j, v.te_free != 0, &dp, &dprev);
            else
                bend_term(P, v.counts, dt, pi, pj, rest, self_is_j, &dp, &dprev);
        }
        s.p = dp;
        s.prev = dprev;
    }
    finish_vertex(v, P, i, flags, inv_mass, dt, &s);
}

// A launch that was allowed to start before the one before it on the stream
// ended (launch_carved, chained) waits here until that one has ended and its
// writes are visible; any other launch passes at once.  Every thread of such a
// kernel calls it, so that no launch ends before those ahead of it have.
__device__ __forceinline__ void wait_for_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// The same pass with L lanes per vertex (32 / L vertices per warp) for the
// stretch gather: lane u takes entries u, u + L, ... and the vertex's first
// lane adds the corrections in entry order, so the sums are those of
// vertex_pass_item.  A thread per vertex walks its six or so entries one after
// another, each a load and a chain of a root and two quotients, while a cloth
// of a few ten thousand vertices leaves most of the chip's warps unused (180 x
// 180, launched, with the host calls: 235 us per frame with one lane, 154 with
// two).
template <int L>
__global__ void __launch_bounds__(kThreads) k_vertex_pass_lanes(View v, unsigned flags) {
    const long long g = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const int i = (int)(g / L), sub = (int)(g % L);
    bool work = i < v.nV;
    // before the wait: what no kernel of the frame writes, parameters and
    // constraints
    const Params* P = nullptr;
    int k = 0, end = 0, active = 0;
    float dt = 0.0f, alpha = 0.0f;
    if (work) {
        P = &params_v(v, i);
        active = P->active;
        dt = P->sub_dt;
        alpha = stretch_alpha(P->stretch_compliance, dt);
        if (active && !P->pcg_on) {
            k = __ldg(&v.sp_off[i]);
            end = __ldg(&v.sp_off[i + 1]);
        }
    }
    const int rounds = (__reduce_max_sync(0xffffffffu, end - k) + L - 1) / L;
    k += sub;
    int2 next = k < end ? __ldg(&v.sp_ent[k]) : make_int2(0, 0);
    wait_for_previous();
    float4 p4 = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    VState s{F3{0.0f, 0.0f, 0.0f}, F3{0.0f, 0.0f, 0.0f}, F3{0.0f, 0.0f, 0.0f}, 0.0f};
    if (work) {
        p4 = v.pos_in[i];
        if (!active) {
            if (sub == 0 && v.pos != v.pos_in) v.pos[i] = p4;  // keep the ping-pong buffers in step
            work = false;
        }
    }
    if (work) {
        s.w = p4.w;
        s.p = f3(p4);
        if (sub == 0) {
            s.prev = f3(v.prev[i]);
            s.vel = f3(v.vel[i]);
        }
    }
    for (int n = 0; n < rounds; ++n, k += L) {
        F3 d{0.0f, 0.0f, 0.0f};
        int use = 0;  // bit 0 a correction, bit 1 a stretched edge
        const int2 e = next;
        if (k + L < end) next = __ldg(&v.sp_ent[k + L]);
        if (k < end) {
            const bool self_is_j = (e.x & kSideBit) != 0;
            const float4 q4 = v.pos_in[e.x & 0x7fffffff];
            F3 corr;
            float c;
            bool clamped;
            if (stretch_correction(self_is_j ? q4 : p4, self_is_j ? p4 : q4, __int_as_float(e.y), alpha, &corr, &c, &clamped)) {
                if (clamped && !self_is_j) count1(v.counts, kCntHardFallbacks);
                if (p4.w > 0.0f) {
                    d = self_is_j ? corr * p4.w : corr * (-p4.w);
                    use = c > 0.0f ? 3 : 1;
                }
            }
        }
#pragma unroll
        for (int u = 0; u < L; ++u) {
            // (only the first lane's sums count: its own correction needs no exchange)
            const F3 du = u == 0 ? d
                                 : F3{__shfl_down_sync(0xffffffffu, d.x, u, L), __shfl_down_sync(0xffffffffu, d.y, u, L),
                                      __shfl_down_sync(0xffffffffu, d.z, u, L)};
            const int uu = u == 0 ? use : __shfl_down_sync(0xffffffffu, use, u, L);
            if (uu & 1) s.p = s.p + du;
            if (uu & 2) s.prev = s.prev + du * 0.08f;
        }
    }
    if (work && sub == 0) finish_vertex(v, *P, i, flags, __ldg(&v.inv_mass[i]), dt, &s);
}

// Six 256-thread blocks per SM (40 registers): the gathers are latency
// bound, and the extra resident warps outweigh the spills (batch256 stretch
// passes 2.05 -> 1.85 ms per frame; five blocks 1.98).
__global__ void __launch_bounds__(kThreads, 6) k_vertex_pass(View v, unsigned flags) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < v.nV) vertex_pass_item(v, i, flags);
}

// Bend constraints of one colour, applied in place: no two bends of a colour
// share a vertex (abi41.cu:2886-2970).
__device__ __forceinline__ void bend_pair(const View& v, int2 pr, float rest) {
    const int i = pr.x, j = pr.y;
    if (i < 0 || j < 0 || i >= v.nV || j >= v.nV || i == j) {
        count1(v.counts, kCntBendingGuards);
        return;
    }
    const Params& P = params_v(v, i);
    if (!P.active) return;
    const float dt = P.sub_dt;
    const float4 pi4 = v.pos[i], pj4 = v.pos[j];
    F3 corr;
    bool guard;
    const bool applied = bend_correction(P, dt, pi4, pj4, rest, &corr, &guard);
    if (guard) count1(v.counts, kCntBendingGuards);
    if (!applied) return;
    if (pi4.w > 0.0f) {
        const F3 d = corr * (-pi4.w);
        v.pos[i] = f4(f3(pi4) + d, pi4.w);
        v.prev[i] = f4(f3(v.prev[i]) + d * 0.06f, 0.0f);
    }
    if (pj4.w > 0.0f) {
        const F3 d = corr * pj4.w;
        v.pos[j] = f4(f3(pj4) + d, pj4.w);
        v.prev[j] = f4(f3(v.prev[j]) + d * 0.06f, 0.0f);
    }
    count1(v.counts, kCntBendingWings);
}

__device__ __forceinline__ void bend_item(const View& v, int b) {
    if (b < 0 || b >= v.nB) {
        count1(v.counts, kCntBendingGuards);
        return;
    }
    bend_pair(v, __ldg(&v.bends[b]), __ldg(&v.bend_rest[b]));
}

__global__ void __launch_bounds__(kThreads) k_bend_color(View v, int start, int count) {
    const int local = blockIdx.x * blockDim.x + threadIdx.x, b = start + local;
    const bool listed = local < count && b >= 0 && b < v.nB;
    const int2 pr = listed ? __ldg(&v.bends[b]) : make_int2(-1, -1);
    const float rest = listed ? __ldg(&v.bend_rest[b]) : 0.0f;
    wait_for_previous();
    if (local < count) bend_pair(v, pr, rest);
}

__global__ void k_copy_pos(float4* dst, const float4* src, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) dst[i] = src[i];
}

// Row of vertex i in a transfer of [lo, ...): its place in the caller's order
// of the cloths, or in the range.
__device__ __forceinline__ size_t transfer_row(const View& v, int i, int lo, bool external) {
    if (!external) return (size_t)(i - lo);
    const Params& P = params_v(v, i);
    return (size_t)(P.ext_vstart + (i - P.vstart));
}

__global__ void k_pack_positions(View v, float* dst, const float4* src, int lo, int n, bool external) {
    // a thread per float: the rows may lie in host memory, which takes whole
    // sectors better than three passes of strided words
    const long long at = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (at >= 3ll * n) return;
    const int i = lo + (int)(at / 3), c = (int)(at % 3);
    dst[3 * transfer_row(v, i, lo, external) + c] = reinterpret_cast<const float*>(src + i)[c];
}

__global__ void k_unpack_positions(View v, float4* pos, float4* prev, const float* src, const float4* rest, int lo, int n,
                                   bool external) {
    const int at = blockIdx.x * blockDim.x + threadIdx.x;
    if (at >= n) return;
    const float* s = src + 3 * transfer_row(v, lo + at, lo, external);
    const float4 p = make_float4(s[0], s[1], s[2], rest[lo + at].w);
    pos[lo + at] = p;
    prev[lo + at] = p;
}

// Back to rest, with the diagnostic counters at zero.
__global__ void k_reset_state(float4* pos, float4* prev, float4* vel, const float4* rest, int n, unsigned long long* counts) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (blockIdx.x == 0)
        for (int k = threadIdx.x; k < kCntSlots; k += blockDim.x) counts[k] = 0;
    if (i >= n) return;
    const float4 p = rest[i];
    pos[i] = p;
    prev[i] = p;
    vel[i] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
}

// Scatter of changed pin entries (vertices whose pin was set or cleared).
__global__ void k_pin_scatter(const int* idx, const float4* target, const float* weight, const float* relax, int n,
                              float4* pin_target, float* pin_weight, float* pin_relax, int nV) {
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= n) return;
    const int i = idx[k];
    if (i < 0 || i >= nV) return;
    pin_target[i] = target[k];
    pin_weight[i] = weight[k];
    pin_relax[i] = relax[k];
}

// A few pin changes (an animated garment moves a handful of pins per frame):
// as kernel arguments they need no staging copy at all.
__global__ void __launch_bounds__(kPinBatch) k_pin_batch(const __grid_constant__ PinBatch b, int n, float4* pin_target,
                                                         float* pin_weight, float* pin_relax, int nV) {
    const int k = threadIdx.x;
    if (k >= n) return;
    const int i = b.idx[k];
    if (i < 0 || i >= nV) return;
    pin_target[i] = b.target[k];
    pin_weight[i] = b.weight[k];
    pin_relax[i] = b.relax[k];
}

inline int blocks_for(int n) { return (n + kThreads - 1) / kThreads; }

}  // namespace

// The per-vertex passes are latency bound (gathers of neighbours): by default
// 128-thread blocks spread a 10k-vertex cloth over twice as many SMs.
// One block per cloth; the cloth's positions (both ping-pong buffers),
// previous positions and velocities live in shared memory for the whole
// frame, so the neighbour gathers and the per-vertex stages touch no global
// memory for state.  Every operation of the recorded frame sweeps the cloth's
// items with the block's threads, then the block synchronises.  The state
// pointers of the View are offset by the cloth's first vertex, so the item
// functions index them with global vertex indices as in the launched form.
__global__ void __launch_bounds__(1024) k_frame_fused(View base, const FrameOp* ops, int nops, float4* buf0,
                                                       const int2* bend_ranges, int K) {
    extern __shared__ float4 sm[];
    const int k = blockIdx.x;
    if (k >= K) return;
    const Params& P = base.P[k];
    const int v0 = P.vstart, n = P.V, v1 = P.vstart + P.V;
    const int cap = (int)(blockDim.x);  // vertices per state array in shared memory
    float4* s0 = sm;
    float4* s1 = sm + cap;
    float4* sprev = sm + 2 * cap;
    float4* svel = sm + 3 * cap;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        s0[i] = buf0[v0 + i];
        sprev[i] = base.prev[v0 + i];
        svel[i] = base.vel[v0 + i];
    }
    __syncthreads();
    View v = base;
    v.prev = sprev - v0;
    v.vel = svel - v0;
    float4* b0 = s0 - v0;
    float4* b1 = s1 - v0;
    for (int o = 0; o < nops; ++o) {
        const FrameOp op = ops[o];
        v.pos_in = op.in_buf ? b1 : b0;
        v.pos = op.out_buf ? b1 : b0;
        v.substep = op.substep;
        v.last_it = op.last_it;
        if (op.kind == 0) {
            for (int i = v0 + (int)threadIdx.x; i < v1; i += blockDim.x) predict_item(v, i);
        } else if (op.kind == 1) {
            for (int i = v0 + (int)threadIdx.x; i < v1; i += blockDim.x) vertex_pass_item(v, i, op.flags);
        } else if (op.kind == 2) {
            const int2 r = bend_ranges[op.color * K + k];
            for (int b = r.x + (int)threadIdx.x; b < r.x + r.y; b += blockDim.x) bend_item(v, b);
        } else {
            for (int i = v0 + (int)threadIdx.x; i < v1; i += blockDim.x) v.pos[i] = v.pos_in[i];
        }
        __syncthreads();
    }
    // a frame ends with its result in buffer 0
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        buf0[v0 + i] = s0[i];
        base.prev[v0 + i] = sprev[i];
        base.vel[v0 + i] = svel[i];
    }
}

// Cluster form of the fused frame: a thread-block cluster of C CTAs (C SMs)
// per cloth.  Each CTA holds a full copy of the cloth's state in its shared
// memory and computes the vertex operations for its slice of the vertices;
// after each operation it writes its slice of the arrays the operation wrote
// into the other CTAs' copies (distributed shared memory), then the cluster
// synchronises.  Bend colours are computed by every CTA on its own copy
// (identical work, identical results), so their scattered writes need no
// exchange.  Within an operation the incoming copies touch only other
// slices of the arrays being written (gathers read the other buffer; the
// previous positions and velocities are read for the own vertex only).
namespace cgx = cooperative_groups;

__global__ void __launch_bounds__(256) k_frame_cluster(View base, const FrameOp* ops, int nops, float4* buf0,
                                                        const int2* bend_ranges, int K, int cap) {
    extern __shared__ float4 sm[];
    cgx::cluster_group cluster = cgx::this_cluster();
    const int C = (int)cluster.num_blocks();
    const int r = (int)cluster.block_rank();
    const int k = (int)(blockIdx.x / C);
    if (k >= K) return;  // uniform over the cluster
    const Params& P = base.P[k];
    const int v0 = P.vstart, n = P.V;
    const int chunk = (n + C - 1) / C;
    const int lo = min(r * chunk, n), hi = min(lo + chunk, n);
    float4* s0 = sm;
    float4* s1 = sm + cap;
    float4* sprev = sm + 2 * cap;
    float4* svel = sm + 3 * cap;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        s0[i] = buf0[v0 + i];
        sprev[i] = base.prev[v0 + i];
        svel[i] = base.vel[v0 + i];
    }
    cluster.sync();  // every copy is complete before any CTA writes into another
    View v = base;
    v.prev = sprev - v0;
    v.vel = svel - v0;
    float4* b0 = s0 - v0;
    float4* b1 = s1 - v0;
    for (int o = 0; o < nops; ++o) {
        const FrameOp op = ops[o];
        v.pos_in = op.in_buf ? b1 : b0;
        v.pos = op.out_buf ? b1 : b0;
        v.substep = op.substep;
        v.last_it = op.last_it;
        if (op.kind == 2) {
            // every CTA applies the colour to its copy; one of them counts
            View bv = v;
            if (r != 0) bv.counts = nullptr;
            const int2 rg = bend_ranges[op.color * K + k];
            for (int b = rg.x + (int)threadIdx.x; b < rg.x + rg.y; b += blockDim.x) bend_item(bv, b);
        } else {
            for (int i = v0 + lo + (int)threadIdx.x; i < v0 + hi; i += blockDim.x) {
                if (op.kind == 0)
                    predict_item(v, i);
                else if (op.kind == 1)
                    vertex_pass_item(v, i, op.flags);
                else
                    v.pos[i] = v.pos_in[i];
            }
            __syncthreads();
            // the own slice of the written arrays into every other copy
            const int out = op.out_buf ? 1 : 0;
            const bool state = op.kind != 3;
            for (int q = 1; q < C; ++q) {
                const int dst = (r + q) % C;
                float4* rem = cluster.map_shared_rank(sm, dst);
                for (int i = lo + (int)threadIdx.x; i < hi; i += blockDim.x) {
                    rem[out * cap + i] = sm[out * cap + i];
                    if (state) {
                        rem[2 * cap + i] = sprev[i];
                        rem[3 * cap + i] = svel[i];
                    }
                }
            }
        }
        cluster.sync();
    }
    for (int i = lo + (int)threadIdx.x; i < hi; i += blockDim.x) {
        buf0[v0 + i] = s0[i];
        base.prev[v0 + i] = sprev[i];
        base.vel[v0 + i] = svel[i];
    }
}

// The fused frame with an edge per thread, by a cluster of C CTAs per cloth
// (plain shared memory for one).  k_frame_fused is bound by instruction issue:
// its one SM computes every edge's correction at both ends (5.0 us per
// operation of a 32 x 32 cloth, 285 issue cycles per warp of edges).  Here a
// CTA computes each edge of its vertices once into shared memory and a vertex
// adds its edges' corrections in its entry order, which is the launched form's
// sum; C CTAs divide the work, and only the edges between two CTAs are
// computed twice.  A vertex's state stays in its thread's registers, positions
// are published by turns in two buffers, so an operation costs one cluster
// barrier.  Counters are kept per thread and added at the end: a barrier would
// wait for atomics in flight.  Per frame with the host calls, k_frame_fused or
// launched kernels -> this form: 8 x 8 144 -> 61 us, 32 x 32 216 -> 86,
// 64 x 64 248 -> 119, 110 x 110 258 -> 174; 150 cloths of 20 x 20 156 -> 72.
constexpr unsigned kEdgeFixed = 1u, kEdgeMine = 2u, kEdgeAddr = ~7u;

template <int T, bool kOne>
__global__ void __launch_bounds__(T, T == 384 ? 2 : 1) k_frame_edges(View v, FramePlan f, const FrameOp* ops, int first, int last, float4* buf0,
                                                      const int2* bend_ranges, int K) {
    extern __shared__ float4 sm[];
    __shared__ unsigned long long s_counter;
    __shared__ int s_lost;
    __shared__ Params sP;
    const cgx::cluster_group cluster = cgx::this_cluster();
    const int C = kOne ? 1 : (int)cluster.num_blocks(), rank = kOne ? 0 : (int)cluster.block_rank();
    const int cloth = (int)(blockIdx.x / C);
    for (int k = threadIdx.x; k < (int)(sizeof(Params) / 4); k += blockDim.x)
        reinterpret_cast<unsigned*>(&sP)[k] = reinterpret_cast<const unsigned*>(&v.P[cloth])[k];
    if (threadIdx.x == 0) {
        ClusterBarrier::init(&s_counter, C);
        ClusterBarrier::init_fence();
        s_lost = 0;
    }
    __syncthreads();
    const Params& P = sP;
    if (!P.active) return;        // uniform over the cluster: the state stays as it is
    if (!kOne) cluster.sync();    // every CTA's counter is set before the first arrival
    ClusterBarrier bar{smem_addr(&s_counter), 0u, C, false};
    const int chunk = f.chunk;
    float4* rows = sm;            // positions by turns in two buffers, previous positions
    float4* result = rows + 3 * chunk;
    uint4* edge = reinterpret_cast<uint4*>(result + f.edge_rows);
    int* ent = reinterpret_cast<int*>(edge + f.edge_rows);
    const ClusterMap<kOne> map(smem_addr(rows), chunk, rank);
    const float dt = P.sub_dt;
    const int v0 = P.vstart, V = P.V;
    const int* off = f.off + (size_t)cloth * C + rank;
    const int edge0 = off[0], edges = off[1] - edge0;
    const float alpha = stretch_alpha(P.stretch_compliance, dt);
    for (int e = threadIdx.x; e < edges; e += blockDim.x) {
        const int id = __ldg(&f.edge[edge0 + e]);
        const int2 p = __ldg(&v.edges[id]);
        const float weight = buf0[p.x].w + buf0[p.y].w;
        const unsigned flags = (weight <= 0.0f ? kEdgeFixed : 0u) |
                               (p.x - v0 >= rank * chunk && p.x - v0 < (rank + 1) * chunk ? kEdgeMine : 0u);
        edge[e] = make_uint4(map.addr(p.x - v0) | flags, map.addr(p.y - v0), __float_as_uint(__ldg(&v.edge_rest[id])),
                             __float_as_uint(weight + alpha));
    }
    const int t = (int)threadIdx.x, l = rank * chunk + t;
    const bool mine = t < chunk && l < V;
    const int i = v0 + l;
    VState s{F3{0.0f, 0.0f, 0.0f}, F3{0.0f, 0.0f, 0.0f}, F3{0.0f, 0.0f, 0.0f}, 0.0f};
    int begin = 0, end = 0;
    float inv_mass = 0.0f, pin_weight = -1.0f, pin_relax = 0.0f;
    F3 pin_target{0.0f, 0.0f, 0.0f};
    if (mine) {
        const float4 p4 = buf0[i];
        s = VState{f3(p4), f3(v.prev[i]), f3(v.vel[i]), p4.w};
        const int row0 = __ldg(&v.sp_off[v0 + rank * chunk]);
        begin = __ldg(&v.sp_off[i]) - row0;
        end = __ldg(&v.sp_off[i + 1]) - row0;
        inv_mass = __ldg(&v.inv_mass[i]);
        pin_weight = __ldg(&v.pin_weight[i]);
        pin_relax = __ldg(&v.pin_relax[i]);
        pin_target = f3(ld4(&v.pin_target[i]));
        for (int k = begin; k < end; ++k) ent[k] = __ldg(&f.ent[row0 + k]);
    }
    unsigned clamps = 0, wings = 0, guards = 0;
    int turn = 0;
    bool bending = false;  // the state is in the rows, a bend colour in progress
    for (int o = first; o < last; ++o) {
        const FrameOp op = ops[o];
        if (op.kind == 2) {
            // one bend colour in place (bend_item)
            if (!bending) {
                if (mine) {
                    rows[turn * chunk + t] = f4(s.p, s.w);
                    rows[2 * chunk + t] = f4(s.prev, 0.0f);
                }
                bar.sync();
                bending = true;
            }
            const unsigned at = 16u * (unsigned)(turn * chunk), prev_at = 16u * (unsigned)(2 * chunk);
            const int2 r = __ldg(&bend_ranges[op.color * K + cloth]);
            for (int b = r.x + rank * (int)blockDim.x + t; b < r.x + r.y; b += C * (int)blockDim.x) {
                const int2 pr = __ldg(&v.bends[b]);
                if (pr.x < 0 || pr.y < 0 || pr.x >= v.nV || pr.y >= v.nV || pr.x == pr.y) {
                    ++guards;
                    continue;
                }
                const unsigned ai = map.addr(pr.x - v0), aj = map.addr(pr.y - v0);
                const float4 pi4 = ld_cluster<kOne>(ai + at), pj4 = ld_cluster<kOne>(aj + at);
                F3 corr;
                bool guard;
                const bool applied = bend_correction(P, dt, pi4, pj4, __ldg(&v.bend_rest[b]), &corr, &guard);
                if (guard) ++guards;
                if (!applied) continue;
                if (pi4.w > 0.0f) {
                    const F3 d = corr * (-pi4.w);
                    st_cluster<kOne>(ai + at, f4(f3(pi4) + d, pi4.w));
                    st_cluster<kOne>(ai + prev_at, f4(f3(ld_cluster<kOne>(ai + prev_at)) + d * 0.06f, 0.0f));
                }
                if (pj4.w > 0.0f) {
                    const F3 d = corr * pj4.w;
                    st_cluster<kOne>(aj + at, f4(f3(pj4) + d, pj4.w));
                    st_cluster<kOne>(aj + prev_at, f4(f3(ld_cluster<kOne>(aj + prev_at)) + d * 0.06f, 0.0f));
                }
                ++wings;
            }
            bar.sync();
            continue;
        }
        if (bending) {
            if (mine) {
                s.p = f3(rows[turn * chunk + t]);
                s.prev = f3(rows[2 * chunk + t]);
            }
            turn ^= 1;
            bending = false;
        }
        if (op.kind == 0) {
            if (mine) {
                s.prev = s.p;
                if (!(s.w > 0.0f)) {
                    s.vel = F3{0.0f, 0.0f, 0.0f};
                    s.p = f3(ld4(&v.rest[i]));
                } else {
                    predict_free(P, dt, &s);
                }
                pin_apply(pin_weight, pin_target, pin_relax, inv_mass, dt, &s);
            }
            continue;
        }
        if (op.kind != 1) continue;  // a buffer copy: the state is in registers
        const unsigned gather = op.flags & (kPassSpring | kPassTether | kPassBend);
        if (gather) {
            const unsigned at = 16u * (unsigned)(turn * chunk);
            if (mine) rows[turn * chunk + t] = f4(s.p, s.w);
            turn ^= 1;
            bar.sync();
            if (gather & kPassSpring) {
                for (int e = t; e < edges; e += (int)blockDim.x) {
                    const uint4 c = edge[e];
                    if (c.x & kEdgeFixed) continue;  // neither end moves, nobody reads the result
                    F3 corr;
                    float cc;
                    bool clamped;
                    stretch_step(f3(ld_cluster<kOne>((c.x & kEdgeAddr) + at)), f3(ld_cluster<kOne>(c.y + at)), __uint_as_float(c.z),
                                 __uint_as_float(c.w), &corr, &cc, &clamped);
                    if (clamped && (c.x & kEdgeMine)) ++clamps;
                    result[e] = f4(corr, cc > 0.0f ? 1.0f : 0.0f);
                }
                __syncthreads();
                if (mine && s.w > 0.0f)
                    for (int k = begin; k < end; ++k) {
                        const int e = ent[k];
                        const float4 r = result[e & 0x7fffffff];
                        const F3 d = f3(r) * (e < 0 ? s.w : -s.w);
                        s.p = s.p + d;
                        if (r.w != 0.0f) s.prev = s.prev + d * 0.08f;
                    }
            } else if (mine) {
                const bool tether = (gather & kPassTether) != 0;
                const int* goff = tether ? v.te_off : v.bj_off;
                const int2* gent = tether ? v.te_ent : v.bj_ent;
                const float4 p4 = f4(s.p, s.w);
                const int g0 = __ldg(&goff[i]), g1 = tether && v.te_free && !(s.w > 0.0f) ? g0 : __ldg(&goff[i + 1]);
                for (int k = g0; k < g1; ++k) {
                    const int2 e = __ldg(&gent[k]);
                    const bool self_is_j = (e.x & kSideBit) != 0;
                    const float4 q4 = ld_cluster<kOne>(map.addr((e.x & 0x7fffffff) - v0) + at);
                    const float4 pi = self_is_j ? q4 : p4, pj = self_is_j ? p4 : q4;
                    if (tether)
                        tether_term(P, v.counts, dt, pi, pj, __int_as_float(e.y), self_is_j, v.te_free != 0, &s.p, &s.prev);
                    else
                        bend_term(P, v.counts, dt, pi, pj, __int_as_float(e.y), self_is_j, &s.p, &s.prev);
                }
            }
        }
        if (!mine) continue;
        if (op.flags & kPassPin) pin_apply(pin_weight, pin_target, pin_relax, inv_mass, dt, &s);
        if (op.flags & kPassAnalytic) analytic_stage(P, v.counts, inv_mass, dt, &s);
        if (op.flags & kPassSdf) sdf_stage(v, P, inv_mass, dt, &s);
        if ((op.flags & kPassPinPolish) && (op.last_it || P.use_ground || P.use_wall || P.use_sphere || P.sdf_ready))
            pin_apply(pin_weight, pin_target, pin_relax, inv_mass, dt, &s);
        if (op.flags & kPassVelocity) velocity_stage(P, dt, &s);
    }
    clamps = __reduce_add_sync(0xffffffffu, clamps);
    wings = __reduce_add_sync(0xffffffffu, wings);
    guards = __reduce_add_sync(0xffffffffu, guards);
    if ((t & 31) == 0) {
        count_add(v.counts, kCntHardFallbacks, clamps);
        count_add(v.counts, kCntBendingWings, wings);
        count_add(v.counts, kCntBendingGuards, guards);
    }
    if (bar.end(&s_lost)) {  // the state stays as it was
        if (t == 0) *v.lost = 1;
        return;
    }
    if (mine) {
        buf0[i] = f4(s.p, s.w);
        v.prev[i] = f4(s.prev, 0.0f);
        v.vel[i] = f4(s.vel, 0.0f);
    }
}

namespace {

using FrameKernel = void (*)(View, FramePlan, const FrameOp*, int, int, float4*, const int2*, int);
struct FrameShape {
    FrameKernel run;
    int threads;
};
FrameShape frame_kernel(const FramePlan& f) {
    if (f.ctas == 1) return f.chunk <= 512 ? FrameShape{k_frame_edges<512, true>, 512} : FrameShape{k_frame_edges<1024, true>, 1024};
    // 129 to 288 vertices per CTA: two rounds over the edges by 512 threads or
    // three by 384, of which an SM holds two blocks.  Us per frame of one cloth
    // and of 64 handles stepped at once: 48 x 48 100 and 850, 98 and 475; 64 x
    // 64 99 and 847, 100 and 502.  Up to 128 one round of 512 counts for more
    // (40 x 40 76 and 655, 94 and 466), and so do two of 512 above (72 x 72
    // 104 and 905, 123 and 629).
    if (f.chunk > 128 && f.chunk <= 288) return FrameShape{k_frame_edges<384, false>, 384};
    return f.chunk <= 512 ? FrameShape{k_frame_edges<512, false>, 512} : FrameShape{k_frame_edges<768, false>, 768};
}
size_t frame_smem(const FramePlan& f) { return 3 * 16 * (size_t)f.chunk + 32 * (size_t)f.edge_rows + 4 * (size_t)f.ent_rows; }
constexpr int kFrameSmem = 220 * 1024;

}  // namespace

bool frame_shape(int K, int max_v, FramePlan* f) {
    f->ctas = 0;
    if (K < 1 || max_v < 1) return false;
    // as many CTAs per cloth as keep every cloth resident at once (of 16-CTA
    // clusters, one per processing cluster), with at least 128 vertices each,
    // past 256 vertices: the barriers between CTAs cost a small cloth more than
    // they save.  Us per frame with the host calls at 64, 128 and 256 vertices
    // per CTA: 144 vertices 81, 80, 65; 256 85, 84, 76; 576 84, 83, 96; 1,024
    // 86, 86, 100.
    // Past 768 vertices per CTA the launched passes are no slower (30 cloths
    // of up to 64 x 64: 235 us launched, 232 here).
    auto shape = [&](int c) {
        f->ctas = c;
        f->chunk = std::max((max_v + 32 * c - 1) / (32 * c), 1) * 32;
    };
    int c = 1;
    while (c < 16 && max_v > 256 && c * 128 < max_v && 2 * c * (long long)K <= 152) {
        shape(2 * c);
        if (f->chunk <= 768 && cluster_fit(frame_kernel(*f).run, f->ctas, frame_kernel(*f).threads, kFrameSmem, kFrameSmem) < K) break;
        c *= 2;
    }
    shape(c);
    if (f->chunk > (c == 1 ? 1024 : 768)) f->ctas = 0;
    return f->ctas > 0;
}

bool frame_fits(int K, FramePlan* f) {
    const FrameShape k = frame_kernel(*f);
    const size_t smem = frame_smem(*f);
    if (smem > (size_t)kFrameSmem || cluster_fit(k.run, f->ctas, k.threads, kFrameSmem, kFrameSmem) < 1) return false;
    auto warps = [](int n) { return (n + 31) / 32 * 32; };
    f->threads = std::min(k.threads, warps(std::max(f->chunk, f->edge_rows)));
    // More cloths than SMs: the shape with the fewest waves of resident
    // clusters, from an edge per thread down to a thread per vertex with more
    // rounds over the edges; of equal ones the most threads.  Us per frame
    // with 512 threads for each cloth, k_frame_fused and so: 1,000 cloths of
    // 8 x 8 294, 153, 74; 600 of 16 x 16 231, 194, 142; 160 of 8 x 8 87, 123,
    // 48.
    auto waves = [&](int threads) {
        const int fit = std::max(cluster_fit(k.run, f->ctas, threads, smem, kFrameSmem), 1);
        return (K + fit - 1) / fit;
    };
    if ((long long)K * f->ctas > 152) {
        int best = waves(f->threads);
        for (int rounds = 2, t = f->threads; best > 1 && t > f->chunk; ++rounds) {
            t = std::max(f->chunk, warps((f->edge_rows + rounds - 1) / rounds));
            const int w = waves(t);
            if (w < best) {
                best = w;
                f->threads = t;
            }
        }
    }
    return true;
}

cudaError_t launch_frame_edges(const View& v, const FramePlan& f, const FrameOp* ops, int first, int last, float4* buf0,
                               const int2* bend_ranges, int K, cudaStream_t s) {
    const FrameShape k = frame_kernel(f);
    return cluster_launch(k.run, K, f.ctas, f.threads, frame_smem(f), s, v, f, ops, first, last, buf0, bend_ranges, K);
}

// cluster > 1: one cluster of that many CTAs per cloth (block threads each)
void launch_frame_cluster(const View& v, const FrameOp* ops, int nops, float4* buf0, const int2* bend_ranges, int K, int cap,
                          int cluster, int block, cudaStream_t s) {
    static bool configured = false;
    if (!configured) {
        cudaFuncSetAttribute(k_frame_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * 1024 * (int)sizeof(float4));
        configured = true;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(K * cluster), 1, 1);
    cfg.blockDim = dim3((unsigned)block, 1, 1);
    cfg.dynamicSmemBytes = (size_t)4 * cap * sizeof(float4);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = (unsigned)cluster;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (K > 0) cudaLaunchKernelEx(&cfg, k_frame_cluster, v, ops, nops, buf0, bend_ranges, K, cap);
}

void launch_frame_fused(const View& v, const FrameOp* ops, int nops, float4* buf0, float4* buf1, const int2* bend_ranges,
                        int K, int block, cudaStream_t s) {
    (void)buf1;
    static bool configured = false;
    if (!configured) {
        cudaFuncSetAttribute(k_frame_fused, cudaFuncAttributeMaxDynamicSharedMemorySize, 4 * 1024 * (int)sizeof(float4));
        configured = true;
    }
    const size_t smem = (size_t)4 * block * sizeof(float4);
    if (K > 0) k_frame_fused<<<K, block, smem, s>>>(v, ops, nops, buf0, bend_ranges, K);
}

// The share of L1 that the launched passes prefer as a kernel property (-1: the
// driver's choice): no solver changes it.
extern "C" __attribute__((visibility("default"))) int xpbd_gb300_pass_carveout(void) {
    int share = -2;
    for (const void* k : {(const void*)k_predict, (const void*)k_vertex_pass, (const void*)k_vertex_pass_lanes<2>,
                          (const void*)k_bend_color, (const void*)k_copy_pos}) {
        cudaFuncAttributes a;
        if (cudaFuncGetAttributes(&a, k) != cudaSuccess || (share != -2 && a.preferredShmemCarveout != share)) return -2;
        share = a.preferredShmemCarveout;
    }
    return share;
}

void launch_predict(const View& v, int V, cudaStream_t s) {
    const int b = tune_of(v.tune, kTuneVertexBlock);
    if (V > 0) launch_carved(k_predict, grid_for(V, b), b, s, v.carve, false, v);
}

// Lanes per vertex of a stretch pass over V vertices: more shorten the pass,
// but a vertex's remaining stages take a warp's slot for each, which a GPU
// shared with other solvers feels.  Us per frame of a plain cloth (launched
// passes, with the host calls) with 1, 2, 4, 8 lanes: 1,600 vertices 214, 135,
// 125, 118; 4,096 210, 136, 127, 120; 8,100 223, 147, 137, 132; 12,544 233, 150,
// 138, 139; 32,400 235, 154, 167, 208.  Of handles stepped at once, 64 of 4,096
// vertices 462, 445, 685, 1,069; 32 of 8,100 395, 399, 633, 994; 16 of 12,544
// 340, 301, 477, 738; 16 of 32,400 609, 719, 1,168, 1,819; 4 of 202,500 872,
// 1,138, 1,887, 3,023.  With volume pressure 10,000 vertices take 193 us with 4
// lanes and 195 with 2, 24 handles of them 621 and 429.  Frames with self
// collision spend little of a shared GPU on their passes and wait for them
// between longer stages, so they keep 4 lanes for longer (three fast frames of
// a folded 100 x 100 cloth with 8 lanes and with 2: 2,819 and 2,860 us; with 8
// and with 4: 2,799 and 2,813).
constexpr int kPassLanes8 = 2 << 10, kPassLanes4 = 4608, kPassLanes4Self = 12 << 10, kPassLanes2 = 128 << 10;

// A kernel that waits by itself (wait_for_previous) may start while the one
// before it drains: its launch and its first loads, of constraints and
// parameters, then overlap that one's last blocks.  Us per frame without and
// with it: 112 x 112 vertices 117 and 111, 140 x 140 125 and 117, 180 x 180 137
// and 133, 240 x 240 140 and 134, 300 x 300 198 and 188.  Not earlier still: a
// kernel that lets the next one start beside all of its blocks shares the SMs
// with them (240 x 240 153).
void launch_bend_color(const View& v, int start, int count, cudaStream_t s, bool chained) {
    const int b = tune_of(v.tune, kTuneVertexBlock);
    if (count > 0) launch_carved(k_bend_color, grid_for(count, b), b, s, v.carve, chained, v, start, count);
}

void launch_vertex_pass(const View& v, int V, unsigned flags, cudaStream_t s, bool chained) {
    const int b = tune_of(v.tune, kTuneVertexBlock);
    if (V <= 0) return;
    auto lanes = [&](void (*kernel)(View, unsigned), int n) {
        launch_carved(kernel, grid_for((long long)n * V, b), b, s, v.carve, chained, v, flags);
    };
    if ((flags & kPassSpring) && V <= kPassLanes8)
        lanes(k_vertex_pass_lanes<8>, 8);
    else if ((flags & kPassSpring) && V <= (v.carve >= 0 ? kPassLanes4Self : kPassLanes4))
        lanes(k_vertex_pass_lanes<4>, 4);
    else if ((flags & kPassSpring) && V <= kPassLanes2)
        lanes(k_vertex_pass_lanes<2>, 2);
    else
        launch_carved(k_vertex_pass, grid_for(V, b), b, s, v.carve, false, v, flags);
}


void launch_pin_scatter(const int* idx, const float4* target, const float* weight, const float* relax, int n,
                        float4* pin_target, float* pin_weight, float* pin_relax, int nV, cudaStream_t s) {
    if (n > 0) k_pin_scatter<<<blocks_for(n), kThreads, 0, s>>>(idx, target, weight, relax, n, pin_target, pin_weight, pin_relax, nV);
}

void launch_copy_pos(const View& v, float4* dst, const float4* src, int V, cudaStream_t s) {
    if (V > 0) launch_carved(k_copy_pos, blocks_for(V), kThreads, s, v.carve, false, dst, src, V);
}

void launch_pin_batch(const PinBatch& b, int n, float4* pin_target, float* pin_weight, float* pin_relax, int nV, cudaStream_t s) {
    if (n > 0) k_pin_batch<<<1, kPinBatch, 0, s>>>(b, std::min(n, kPinBatch), pin_target, pin_weight, pin_relax, nV);
}

void launch_pack_positions(const View& v, float* dst, const float4* src, int lo, int n, bool external, cudaStream_t s) {
    if (n > 0) k_pack_positions<<<(unsigned)((3ll * n + kThreads - 1) / kThreads), kThreads, 0, s>>>(v, dst, src, lo, n, external);
}

void launch_unpack_positions(const View& v, float4* pos, float4* prev, const float* src, const float4* rest, int lo, int n,
                             bool external, cudaStream_t s) {
    if (n > 0) k_unpack_positions<<<blocks_for(n), kThreads, 0, s>>>(v, pos, prev, src, rest, lo, n, external);
}

void launch_reset_state(float4* pos, float4* prev, float4* vel, const float4* rest, int n, unsigned long long* counts, cudaStream_t s) {
    k_reset_state<<<std::max(blocks_for(n), 1), kThreads, 0, s>>>(pos, prev, vel, rest, n, counts);
}

}  // namespace xg
