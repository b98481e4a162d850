// Hard-stretch optimisation: the block-Jacobi preconditioned CG stretch solve
// and the ratio caps / averaged polish around it (reference
// native/src/ssbl_xpbd_cuda_abi41.cu:1982-2708, 3032-3464, 7626-8027).
//
// System assembly and every per-vertex sum are gathers over the vertex ->
// edge CSR in edge order (the reference scatters with float atomics).  The CG
// dot products are reduced deterministically: a shuffle-down tree inside each
// 32-vertex warp, partials stored per warp, and the last block to finish
// (atomic ticket, no waiting) sums the partials in a fixed order -- lane l
// adds partials l, l+32, ... then a shuffle-down tree.  The device-side
// alpha / beta / status logic is the reference's (abi41.cu:3320-3464).
//
// In a batch every cloth that enables the optimisation solves its own system:
// the solve grid is the concatenation of the grids one-cloth solvers of
// those cloths would launch (a block belongs to one cloth), each cloth has
// its own partials segment, ticket and scalar slots, so its reductions, its
// alpha / beta and its status follow exactly the one-cloth sequence.
//
// Two forms run the same per-vertex arithmetic and the same sums.  The
// launched form has a kernel per step of the iteration and per cap colour
// and spreads each over the whole chip.  The cluster form
// (k_hard_cluster) gives a cloth one thread-block cluster for the whole
// solve and its caps, with a cluster barrier where the launched form has a
// kernel boundary.
#include <algorithm>

#include "xpbd_cluster.cuh"
#include "xpbd_solver.cuh"

namespace xg {

namespace cgx = cooperative_groups;

namespace {

constexpr float kStatusOk = 0.0f, kStatusBadResidual = 1.0f, kStatusZeroResidual = 2.0f, kStatusBadDad = 3.0f,
                kStatusBadAlpha = 4.0f;

inline int blocks_for(int n) { return (n + kThreads - 1) / kThreads; }

struct Sym {
    float m11, m12, m13, m22, m23, m33;
};

__device__ __forceinline__ Sym sym_load(const float4* a, int i) {
    const float4 u = a[2 * i], w = a[2 * i + 1];
    return Sym{u.x, u.y, u.z, u.w, w.x, w.y};
}
__device__ __forceinline__ void sym_store(float4* a, int i, Sym m) {
    a[2 * i] = make_float4(m.m11, m.m12, m.m13, m.m22);
    a[2 * i + 1] = make_float4(m.m23, m.m33, 0.0f, 0.0f);
}
// m * v + acc with the reference's fused chains (abi41.cu:1125-1131).
__device__ __forceinline__ F3 sym_madd(Sym m, F3 v, F3 acc) {
    return F3{fmaf(m.m13, v.z, fmaf(m.m12, v.y, fmaf(m.m11, v.x, acc.x))),
              fmaf(m.m23, v.z, fmaf(m.m22, v.y, fmaf(m.m12, v.x, acc.y))),
              fmaf(m.m33, v.z, fmaf(m.m23, v.y, fmaf(m.m13, v.x, acc.z)))};
}
__device__ __forceinline__ Sym sym_outer(F3 n, float s) {
    return Sym{n.x * n.x * s, n.x * n.y * s, n.x * n.z * s, n.y * n.y * s, n.y * n.z * s, n.z * n.z * s};
}
__device__ __forceinline__ Sym sym_add(Sym a, Sym b) {
    return Sym{a.m11 + b.m11, a.m12 + b.m12, a.m13 + b.m13, a.m22 + b.m22, a.m23 + b.m23, a.m33 + b.m33};
}
// Inverse of a symmetric 3x3 block, diagonal fallback when singular
// (abi41.cu:1158-1189).
__device__ Sym sym_inverse_or_diag(Sym m, unsigned long long* guard) {
    const float a = m.m11, b = m.m12, c = m.m13, d = m.m22, e = m.m23, f = m.m33;
    const float df_ee = fmaf(d, f, -e * e);
    const float bf_ce = fmaf(b, f, -c * e);
    const float be_cd = fmaf(b, e, -c * d);
    const float det = fmaf(c, be_cd, fmaf(-b, bf_ce, a * df_ee));
    if (isfinite(det) && fabsf(det) > 1.0e-12f) {
        const float inv = 1.0f / det;
        return Sym{df_ee * inv,
                   fmaf(c, e, -b * f) * inv,
                   be_cd * inv,
                   fmaf(a, f, -c * c) * inv,
                   fmaf(b, c, -a * e) * inv,
                   fmaf(a, d, -b * b) * inv};
    }
    if (guard) atomicAdd(guard, 1ull);
    return Sym{1.0f / fmaxf(fabsf(a), 1.0e-4f), 0.0f, 0.0f, 1.0f / fmaxf(fabsf(d), 1.0e-4f), 0.0f,
               1.0f / fmaxf(fabsf(f), 1.0e-4f)};
}

// Per-edge projection bound (abi41.cu:1070-1089).
__device__ float projection_limit(const Params& P, float rest) {
    const float base = fmaxf(1.0e-5f, fminf(fmaxf(rest, P.thickness) * 0.5f, 0.25f));
    if (P.stretch_strength < 0.95f || !isfinite(P.thickness) || P.thickness <= kEps) return base;
    const float hard = fmaxf(1.0e-5f, fminf(fmaxf(rest * 0.18f, P.thickness * 0.06f), 0.0035f));
    return fminf(base, hard);
}
// Per-iteration position write-back bound (abi41.cu:1091-1104).
__device__ float writeback_limit(const Params& P) {
    if (P.stretch_strength < 0.95f || !isfinite(P.thickness) || P.thickness <= kEps) return 0.25f;
    return fmaxf(2.5e-4f, fminf(P.thickness * 0.035f, 9.0e-4f));
}

// ---------------------------------------------------- fixed-order sums --
__device__ __forceinline__ float warp_tree(float v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// The vertex of this thread in the solve grid: the block's cloth, its local
// vertex index and its global one.
struct PcgItem {
    int cloth, local, i;
    bool valid;
};
__device__ __forceinline__ PcgItem pcg_item(const View& v, const PcgView& g) {
    const int c = __ldg(&g.blk_cloth[blockIdx.x]);
    const Params& P = v.P[c];
    const int local = (blockIdx.x - P.pcg_block0) * blockDim.x + threadIdx.x;
    return PcgItem{c, local, P.vstart + local, local < P.V};
}

// Store this warp's tree partial; the last block of the cloth to finish
// returns true in every thread of its first warp together with the cloth's
// total in `*total`.
__device__ bool reduce_partials(const PcgView& g, const Params& P, int cloth, float v, float* total) {
    __shared__ bool last;
    const float w = warp_tree(v);
    const int lane = threadIdx.x & 31;
    const int wpb = blockDim.x >> 5;
    const int gw = blockIdx.x * wpb + (threadIdx.x >> 5);
    if (lane == 0) g.partials[gw] = w;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned ticket = atomicAdd(&g.ticket[cloth], 1u);
        last = ticket == (unsigned)(P.pcg_nblocks - 1);
    }
    __syncthreads();
    if (!last || threadIdx.x >= 32) return false;
    __threadfence();
    const int nw = P.pcg_nblocks * wpb;
    const volatile float* part = g.partials + (long long)P.pcg_block0 * wpb;
    float s = 0.0f;
    for (int k = lane; k < nw; k += 32) s += part[k];
    s = warp_tree(s);
    *total = __shfl_sync(0xffffffffu, s, 0);
    if (lane == 0) g.ticket[cloth] = 0u;
    return true;
}

__device__ __forceinline__ float4 z4() { return make_float4(0.0f, 0.0f, 0.0f, 0.0f); }

// Where the polish and caps read and write positions and previous positions:
// global memory in the launched form, the cluster's shared memory in the
// cluster form.
struct GlobalState {
    float4* p;
    float4* q;
    __device__ __forceinline__ float4 pos(int i) const { return p[i]; }
    __device__ __forceinline__ float4 prev(int i) const { return q[i]; }
    __device__ __forceinline__ void set_pos(int i, float4 x) const { p[i] = x; }
    __device__ __forceinline__ void set_prev(int i, float4 x) const { q[i] = x; }
};

// ------------------------------------------------------- system build --
// Assembly gathered per vertex (abi41.cu:3085-3186) fused with the
// preconditioner / initial residual (abi41.cu:3188-3226) and the iteration
// set-up (abi41.cu:3071-3083).
// Returns the vertex's r.z; its off-diagonal blocks are handed to put(k, o).
template <class S, class Put>
__device__ __forceinline__ float build_item(const View& v, const S& st, unsigned long long* guard, const Params& P, int i, int begin,
                                            int end, Sym* diag_out, Sym* pinv, F3* r, F3* z_out, Put&& put) {
    const float4 p4 = st.pos(i);
    Sym diag{1.0f, 0.0f, 0.0f, 1.0f, 0.0f, 1.0f};
    F3 rhs{0.0f, 0.0f, 0.0f};
    const float strength = clamp01f(P.stretch_strength * 2.5f);
    auto entry = [&](int k, int2 e, float4 q4) __attribute__((always_inline)) {
        const bool self_is_j = (e.x & kSideBit) != 0;
        const float4 pi = self_is_j ? q4 : p4, pj = self_is_j ? p4 : q4;
        const float rest = __int_as_float(e.y);
        float4 off = z4();
        const float wi = pi.w, wj = pj.w, weight = wi + wj;
        const bool ai = wi > 0.0f, aj = wj > 0.0f;
        bool ok = isfinite(weight) && weight > 0.0f && isfinite(rest) && rest > kEps && finite3(f3(pi)) && finite3(f3(pj));
        F3 normal{0.0f, 0.0f, 0.0f};
        float projected = 0.0f;
        if (ok) {
            const F3 delta = f3(pj) - f3(pi);
            const float len_sq = dot3(delta, delta);
            ok = isfinite(len_sq) && len_sq > kEps;
            if (ok) {
                const float len = sqrtf(len_sq);
                const float err = len - rest;
                ok = isfinite(err) && fabsf(err) > 1.0e-6f && strength > 0.0f;
                if (ok) {
                    const float lim = projection_limit(P, rest);
                    projected = fmaxf(-lim, fminf(err * strength, lim));
                    ok = isfinite(projected) && fabsf(projected) > 1.0e-7f;
                    normal = delta * (1.0f / len);
                }
            }
        }
        if (ok) {
            const F3 desired = normal * (projected / weight);
            const float stiff = fmaxf(strength, 1.0e-3f);
            const bool mine = self_is_j ? aj : ai;
            if (mine) {
                rhs = rhs + (self_is_j ? desired * (-wj) : desired * wi);
                diag = sym_add(diag, sym_outer(normal, stiff));
            }
            if (ai && aj) off = make_float4(normal.x, normal.y, normal.z, stiff);
        }
        put(k, e.x & 0x7fffffff, off);
    };
    // three entries at a time, their loads in flight together
    for (int k = begin; k < end; k += 3) {
        int2 e[3];
        float4 q4[3];
#pragma unroll
        for (int u = 0; u < 3; ++u) e[u] = __ldg(&v.sp_ent[min(k + u, end - 1)]);
#pragma unroll
        for (int u = 0; u < 3; ++u) q4[u] = st.pos(e[u].x & 0x7fffffff);
#pragma unroll 1
        for (int u = 0; u < 3; ++u) {
            if (k + u >= end) break;
            entry(k + u, u == 0 ? e[0] : (u == 1 ? e[1] : e[2]), u == 0 ? q4[0] : (u == 1 ? q4[1] : q4[2]));
        }
    }
    *diag_out = diag;
    if (!(p4.w > 0.0f)) {
        *r = *z_out = F3{0.0f, 0.0f, 0.0f};
        *pinv = Sym{1.0f, 0.0f, 0.0f, 1.0f, 0.0f, 1.0f};
        return 0.0f;
    }
    const Sym inv = sym_inverse_or_diag(diag, guard);
    const F3 z = sym_madd(inv, rhs, F3{0.0f, 0.0f, 0.0f});
    *pinv = inv;
    *r = rhs;
    *z_out = z;
    return dot3(rhs, z);
}

__global__ void __launch_bounds__(kThreads) k_pcg_build(View v, PcgView g) {
    const PcgItem it = pcg_item(v, g);
    const Params& P = v.P[it.cloth];
    const int i = it.i;
    float rz = 0.0f;
    if (it.valid) {
        Sym diag, pinv;
        F3 r, z;
        rz = build_item(v, GlobalState{v.pos, v.prev}, g.guard, P, i, v.sp_off[i], v.sp_off[i + 1], &diag, &pinv, &r, &z,
                        [&](int k, int, float4 o) { g.offdiag[k] = o; });
        sym_store(g.diag, i, diag);
        sym_store(g.pinv, i, pinv);
        g.r[i] = f4(r, 0.0f);
        g.z[i] = f4(z, 0.0f);
        g.d[i] = f4(z, 0.0f);
    }
    float total;
    if (reduce_partials(g, P, it.cloth, rz, &total) && (threadIdx.x & 31) == 0) {
        float* R = g.red + it.cloth * kRedSlots;
        R[kRedRZ] = total;
        R[kRedInitialRZ] = total;
        R[kRedIterations] = 0.0f;
        R[kRedDAD] = 0.0f;
        R[kRedRZNext] = 0.0f;
        R[kRedStatus] = kStatusOk;
    }
}

// One off-diagonal block times a neighbour's direction.  Inactive entries
// hold a zero block (+0 entries, like the reference's cleared texels).
__device__ __forceinline__ F3 offdiag_madd(float4 o, F3 d, F3 q) {
    Sym nb{0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    if (o.w != 0.0f) {
        const Sym b = sym_outer(F3{o.x, o.y, o.z}, o.w);
        nb = Sym{-b.m11, -b.m12, -b.m13, -b.m22, -b.m23, -b.m33};
    }
    return sym_madd(nb, d, q);
}

// Device alpha and the status it implies (abi41.cu:3320-3340).
__device__ __forceinline__ float cg_alpha(float rz_old, float dad, float* status) {
    *status = kStatusOk;
    if (!isfinite(rz_old) || rz_old < 0.0f) {
        *status = kStatusBadResidual;
    } else if (rz_old <= 1.0e-14f) {
        *status = kStatusZeroResidual;
    } else if (!isfinite(dad) || dad <= 1.0e-14f) {
        *status = kStatusBadDad;
    } else {
        const float alpha = rz_old / dad;
        if (isfinite(alpha)) return alpha;
        *status = kStatusBadAlpha;
    }
    return 0.0f;
}

// Residual and position update of one free vertex; returns its r.z and the
// squared length of its move (the root is monotonic, so the largest move is
// the root of the largest square).
template <class S>
__device__ __forceinline__ float update_item(const S& st, const Params& P, int i, float4 p4, F3 di, F3 qi, float alpha,
                                             const Sym& pinv, F3* r, F3* z_out, float* moved_sq, unsigned* clamped) {
    const F3 ri = *r;
    const F3 res{fmaf(qi.x, -alpha, ri.x), fmaf(qi.y, -alpha, ri.y), fmaf(qi.z, -alpha, ri.z)};
    const F3 safe_res = finite3(res) ? res : F3{0.0f, 0.0f, 0.0f};
    const F3 z = sym_madd(pinv, safe_res, F3{0.0f, 0.0f, 0.0f});
    *r = safe_res;
    *z_out = z;
    F3 delta = di * alpha;
    const float max_delta = writeback_limit(P);
    const float sq = dot3(delta, delta);
    const float len = sq < max_delta * max_delta * 0.99999f ? 0.0f : len3(delta);  // only its being over the limit counts
    if (len > max_delta) {
        delta = delta * (max_delta / fmaxf(len, kEps));
        *clamped += 1u;
    }
    st.set_pos(i, f4(f3(p4) + delta, p4.w));
    st.set_prev(i, f4(f3(st.prev(i)) + delta * 0.08f, 0.0f));
    *moved_sq = fmaxf(dot3(delta, delta), 0.0f);
    return dot3(safe_res, z);
}

// q = A d, partial d.q (abi41.cu:3228-3267); the last block publishes dAd.
__global__ void __launch_bounds__(kThreads) k_pcg_ad(View v, PcgView g) {
    const PcgItem it = pcg_item(v, g);
    const Params& P = v.P[it.cloth];
    const int i = it.i;
    float* R = g.red + it.cloth * kRedSlots;
    const bool status_ok = R[kRedStatus] == kStatusOk;
    float dq = 0.0f;
    if (status_ok && it.valid) {
        if (!(v.pos[i].w > 0.0f)) {
            g.q[i] = z4();
        } else {
            const F3 di = f3(g.d[i]);
            F3 q = sym_madd(sym_load(g.diag, i), di, F3{0.0f, 0.0f, 0.0f});
            const int begin = v.sp_off[i], end = v.sp_off[i + 1];
            for (int k = begin; k < end; ++k) {
                const int col = __ldg(&v.sp_ent[k]).x & 0x7fffffff;
                q = offdiag_madd(g.offdiag[k], f3(g.d[col]), q);
            }
            g.q[i] = f4(q, 0.0f);
            dq = dot3(di, q);
        }
    }
    float total;
    if (reduce_partials(g, P, it.cloth, dq, &total) && (threadIdx.x & 31) == 0) R[kRedDAD] = R[kRedDAD] + total;
}

// Device alpha, solution / residual / preconditioned residual update with the
// incremental position write-back, partial r.z (abi41.cu:3320-3405).
__global__ void __launch_bounds__(kThreads) k_pcg_update(View v, PcgView g) {
    const PcgItem it = pcg_item(v, g);
    const Params& P = v.P[it.cloth];
    const int i = it.i;
    float* R = g.red + it.cloth * kRedSlots;
    float status;
    const float alpha = cg_alpha(R[kRedRZ], R[kRedDAD], &status);
    float rz = 0.0f;
    if (status == kStatusOk && it.valid) {
        const float4 p4 = v.pos[i];
        if (!(p4.w > 0.0f)) {
            g.r[i] = z4();
            g.z[i] = z4();
        } else {
            F3 r = f3(g.r[i]), z;
            float moved_sq;
            unsigned clamped = 0u;
            rz = update_item(GlobalState{v.pos, v.prev}, P, i, p4, f3(g.d[i]), f3(g.q[i]), alpha, sym_load(g.pinv, i), &r, &z, &moved_sq,
                             &clamped);
            if (clamped) count1(v.counts, kCntHardFallbacks);
            g.r[i] = f4(r, 0.0f);
            g.z[i] = f4(z, 0.0f);
            if (moved_sq > 0.0f) atomicMax(g.max_delta_bits, __float_as_uint(sqrtf(moved_sq)));
        }
    }
    if (status != kStatusOk) {
        if (it.local == 0) {
            R[kRedStatus] = status;
            if (status != kStatusZeroResidual) atomicAdd(g.guard, 1ull);
        }
        return;
    }
    float total;
    if (reduce_partials(g, P, it.cloth, rz, &total) && (threadIdx.x & 31) == 0) {
        R[kRedRZNext] = R[kRedRZNext] + total;
        R[kRedIterations] = R[kRedIterations] + 1.0f;
    }
}

// Device beta and d = z + beta d (abi41.cu:3421-3450); the last block then
// advances the scalar slots (abi41.cu:3452-3464).
__global__ void __launch_bounds__(kThreads) k_pcg_dir(View v, PcgView g) {
    const PcgItem it = pcg_item(v, g);
    const Params& P = v.P[it.cloth];
    const int i = it.i;
    float* R = g.red + it.cloth * kRedSlots;
    const float status = R[kRedStatus], rz_old = R[kRedRZ], rz_new = R[kRedRZNext];
    const bool ok = status == kStatusOk && isfinite(rz_old) && isfinite(rz_new) && rz_old > 1.0e-14f && rz_new >= 0.0f;
    const float beta = ok ? rz_new / rz_old : 0.0f;
    if (ok && isfinite(beta) && it.valid) {
        if (!(v.pos[i].w > 0.0f)) {
            g.d[i] = z4();
        } else {
            const F3 d = f3(g.d[i]), z = f3(g.z[i]);
            g.d[i] = make_float4(fmaf(d.x, beta, z.x), fmaf(d.y, beta, z.y), fmaf(d.z, beta, z.z), 0.0f);
        }
    }
    float total;
    if (reduce_partials(g, P, it.cloth, 0.0f, &total) && threadIdx.x == 0) {
        if (status == kStatusOk && isfinite(rz_new) && rz_new >= 0.0f) {
            R[kRedRZ] = rz_new;
            R[kRedDAD] = 0.0f;
            R[kRedRZNext] = 0.0f;
            R[kRedStatus] = kStatusOk;
        }
    }
}

// ------------------------------------------------------- averaged caps --
// limit_delta without its root and quotient where the squared length shows
// that the step is neither too long nor vanishing (the usual case; a chain of
// dependent roots and quotients is what a cap step's time goes into).
__device__ __forceinline__ F3 limit_step(F3 d, float max_len) {
    const float sq = dot3(d, d);
    if (sq < max_len * max_len * 0.99999f && sq > 4.0f * kEps * kEps) return d;
    return limit_delta(d, max_len);
}

// len3(a) <= 1e-20, by the root only where the square is not far above.
__device__ __forceinline__ bool length_at_most_1e20(F3 a) {
    const float sq = dot3(a, a);
    return !(sq > 1.0e-38f) && len3(a) <= 1.0e-20f;
}

// Whether an edge of squared length len_sq is certainly not longer than
// `limit`: the computed length is within a few units in the last place of
// the root, so below limit^2 by a relative 1e-5 the comparison's outcome is
// known without it (most edges of most sweeps; NaN and infinities are not
// taken here).
__device__ __forceinline__ bool surely_within(float len_sq, float limit) { return len_sq < limit * limit * 0.99999f; }

// Length up to which the averaged polish / tiny passes leave an edge alone.
__device__ __forceinline__ float averaged_target(const Params& P, bool tiny, float rest) {
    return rest * (tiny ? 1.06f : (P.stretch_strength >= 0.95f ? 1.08f : 1.18f));
}

// Edge correction shared by the averaged polish / tiny passes, seen from one
// endpoint (abi41.cu:1995-2082, 2399-2467).  Returns false when the edge
// contributes nothing to this vertex.
__device__ bool averaged_delta(const Params& P, bool tiny, float4 pi, float4 pj, F3 prev_i, F3 prev_j, float rest,
                               bool self_is_j, F3* out) {
    const float wi = pi.w, wj = pj.w, weight = wi + wj;
    if (!isfinite(weight) || weight <= 0.0f) return false;
    if (tiny) {
        if (!isfinite(rest) || rest <= kEps || rest > 7.5e-4f) return false;
        if (!finite3(f3(pi)) || !finite3(f3(pj))) return false;
    } else {
        if (!isfinite(rest) || rest <= kEps) return false;
        if (!finite3(f3(pi)) || !finite3(f3(pj)) || !finite3(prev_i) || !finite3(prev_j)) return false;
    }
    const F3 edge = f3(pj) - f3(pi);
    const float len_sq = dot3(edge, edge);
    if (!isfinite(len_sq) || len_sq <= 1.0e-14f) return false;
    const float len = sqrtf(len_sq);
    const float target = averaged_target(P, tiny, rest);
    float relax, max_delta;
    if (tiny) {
        relax = 1.0f;
        max_delta = fminf(fmaxf(rest * 3.0f, 2.5e-4f), 8.0e-4f);
    } else {
        relax = 0.90f;
        max_delta = fmaxf(5.0e-4f, fminf(fmaxf(rest * 2.0f, P.thickness * 0.25f), 0.008f));
    }
    const float excess = len - target;
    if (!isfinite(excess) || excess <= 0.0f) return false;
    const F3 corr = edge * (-relax * excess / fmaxf(weight * len, kEps));
    if (!finite3(corr) || length_at_most_1e20(corr) || (!tiny && !isfinite(dot3(corr, corr)))) return false;
    const float w = self_is_j ? wj : wi;
    if (!(w > 0.0f)) return false;
    const F3 d = limit_step(self_is_j ? corr * wj : corr * (-wi), max_delta);
    if (!finite3(d) || !(dot3(d, d) > 0.0f)) return false;
    *out = d;
    return true;
}

// Gather of the averaged corrections of a vertex's edges: sum and count.
// Vertices of cloths without the hard polish are left alone.
template <class S>
__device__ __forceinline__ float4 avg_gather_item(const View& v, const S& st, const Params& P, int i, int tiny) {
    const float4 p4 = st.pos(i);
    const F3 prev_self = f3(st.prev(i));
    F3 sum{0.0f, 0.0f, 0.0f};
    float count = 0.0f;
    const int begin = v.sp_off[i], end = v.sp_off[i + 1];
    // three edges at a time, their loads in flight together; the neighbour's
    // previous position is read only for an edge that may be too long
    for (int k = begin; k < end; k += 3) {
        int2 e[3];
        float4 q4[3];
#pragma unroll
        for (int u = 0; u < 3; ++u) e[u] = __ldg(&v.sp_ent[min(k + u, end - 1)]);
#pragma unroll
        for (int u = 0; u < 3; ++u) q4[u] = st.pos(e[u].x & 0x7fffffff);
#pragma unroll
        for (int u = 0; u < 3; ++u) {
            if (k + u >= end) continue;
            const float rest = __int_as_float(e[u].y);
            const F3 edge = f3(q4[u]) - f3(p4);  // either orientation: the squared length is the same
            if (rest > kEps && surely_within(dot3(edge, edge), averaged_target(P, tiny != 0, rest))) continue;
            const bool self_is_j = (e[u].x & kSideBit) != 0;
            const F3 prev_o = tiny ? F3{0.0f, 0.0f, 0.0f} : f3(st.prev(e[u].x & 0x7fffffff));
            F3 d;
            if (averaged_delta(P, tiny != 0, self_is_j ? q4[u] : p4, self_is_j ? p4 : q4[u], self_is_j ? prev_o : prev_self,
                               self_is_j ? prev_self : prev_o, rest, self_is_j, &d)) {
                sum = sum + d;
                count += 1.0f;
            }
        }
    }
    return f4(sum, count);
}

__global__ void __launch_bounds__(kThreads) k_avg_gather(View v, PcgView g, int tiny) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= v.nV) return;
    const Params& P = params_v(v, i);
    if (P.pcg_hard) g.avg[i] = avg_gather_item(v, GlobalState{v.pos, v.prev}, P, i, tiny);
}

// Apply the averaged corrections (abi41.cu:2084-2112, 2469-2494).
template <class S>
__device__ __forceinline__ void avg_apply_item(const View& v, const S& st, const Params& P, int i, int tiny, float4 a) {
    const float4 p4 = st.pos(i);
    if (!(p4.w > 0.0f)) return;
    const float count = a.w;
    if (!isfinite(count) || count <= 0.0f) return;
    F3 delta = F3{a.x, a.y, a.z} * (1.0f / count);
    if (!finite3(delta)) {
        count1(v.counts, kCntHardFallbacks);
        return;
    }
    const float max_delta = tiny ? fminf(fmaxf(P.thickness * 0.015f, 2.5e-4f), 9.0e-4f)
                                 : fmaxf(5.0e-4f, fminf(fmaxf(P.thickness * 0.20f, 1.0e-3f), 0.005f));
    delta = limit_step(delta, max_delta);
    if (!finite3(delta) || !(dot3(delta, delta) > 0.0f)) return;
    st.set_pos(i, f4(f3(p4) + delta, p4.w));
    st.set_prev(i, f4(f3(st.prev(i)) + delta * (tiny ? 0.24f : 0.16f), 0.0f));
}

__global__ void __launch_bounds__(kThreads) k_avg_apply(View v, PcgView g, int tiny) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= v.nV) return;
    const Params& P = params_v(v, i);
    if (P.pcg_hard) avg_apply_item(v, GlobalState{v.pos, v.prev}, P, i, tiny, g.avg[i]);
}

// ------------------------------------------------------------ ratio caps --
// One edge of a ratio cap: normal (kind 0, abi41.cu:2249-2362), tiny (1,
// 2496-2601) or extreme (2, 2603-2708).  Writes each endpoint's position
// correction d and previous-position shift pd; ok = false where that
// endpoint gets nothing.  Returns false when the edge is skipped.
__device__ __forceinline__ float cap_start_ratio(const Params& P, int kind) {
    return kind == 0 ? (P.stretch_strength >= 0.95f ? 1.12f : 1.32f) : (kind == 1 ? 1.35f : 1.24f);
}

struct CapSide {
    F3 d, pd;
    bool ok;
};

__device__ bool cap_edge(const Params& P, int kind, float rest, float4 pi4, float4 pj4, F3 qi, F3 qj, CapSide* si, CapSide* sj) {
    si->ok = sj->ok = false;
    const bool tiny = kind == 1;
    if (!isfinite(rest) || rest <= kEps) return false;
    if (tiny ? rest > 7.5e-4f : rest <= 7.5e-4f) return false;
    const float dt = P.sub_dt;
    const float wi = pi4.w, wj = pj4.w, weight = wi + wj;
    if (!isfinite(weight) || weight <= 0.0f) return false;
    const F3 pi = f3(pi4), pj = f3(pj4);
    if (!finite3(pi) || !finite3(pj) || !finite3(qi) || !finite3(qj)) return false;
    const F3 edge = pj - pi;
    const float len_sq = dot3(edge, edge);
    if (!isfinite(len_sq) || len_sq <= 1.0e-14f) return false;
    const float len = sqrtf(len_sq);
    const bool high = P.stretch_strength >= 0.95f;
    const float start_ratio = cap_start_ratio(P, kind);
    float target_ratio, max_delta, prev_sync;
    if (kind == 0) {
        target_ratio = high ? 1.04f : 1.22f;
        max_delta = fminf(fmaxf(rest * 0.60f, P.thickness * 0.10f), 0.010f);
        prev_sync = 0.08f;
    } else if (kind == 1) {
        target_ratio = 1.12f;
        max_delta = fminf(fmaxf(rest * 6.0f, 5.0e-4f), 1.5e-3f);
        prev_sync = 1.0f;
    } else {
        target_ratio = 1.10f;
        max_delta = fminf(fmaxf(rest * 1.25f, P.thickness * 0.10f), 0.006f);
        prev_sync = 0.30f;
    }
    if (!isfinite(len) || len <= rest * start_ratio) return false;
    const float excess = len - rest * target_ratio;
    if (!isfinite(excess) || excess <= 0.0f) return false;
    const F3 corr = edge * (-excess / fmaxf(weight * len, kEps));
    if (!finite3(corr) || length_at_most_1e20(corr)) return false;
    F3 pdi{0.0f, 0.0f, 0.0f}, pdj{0.0f, 0.0f, 0.0f};
    const F3 normal = edge * (1.0f / fmaxf(len, kEps));
    const float sdt = kind == 0 ? fmaxf(dt, kEps) : dt;
    if (isfinite(sdt) && sdt > kEps) {
        const float inv_dt = 1.0f / sdt;
        const F3 vi = (pi - qi) * inv_dt, vj = (pj - qj) * inv_dt;
        const float sep = dot3(vj - vi, normal);
        if (isfinite(sep) && sep > 0.0f) {
            const float trim = sep * sdt * 1.0f / weight;
            if (wi > 0.0f) pdi = pdi + normal * (-wi * trim);
            if (wj > 0.0f) pdj = pdj + normal * (wj * trim);
        }
    }
    if (wi > 0.0f) {
        const F3 d = limit_step(corr * (-wi), max_delta);
        if (finite3(d) && dot3(d, d) > 0.0f) *si = CapSide{d, pdi + d * prev_sync, true};
    }
    if (wj > 0.0f) {
        const F3 d = limit_step(corr * wj, max_delta);
        if (finite3(d) && dot3(d, d) > 0.0f) *sj = CapSide{d, pdj + d * prev_sync, true};
    }
    return true;
}

// Caps applied in place one edge colour at a time (no two edges of a colour
// share a vertex), over a caller's edge colouring.  In a batch a launch
// covers one colour of every cloth that uses its colouring; the time step is
// the cloth's substep length.
// Returns false when the edge's length shows that nothing changes.
template <class S>
__device__ __forceinline__ bool cap_item(const S& st, const Params& P, int nV, int2 ed, float rest, int kind) {
    const int i = ed.x, j = ed.y;
    if (i < 0 || j < 0 || i >= nV || j >= nV || i == j) return false;
    const float4 pi4 = st.pos(i), pj4 = st.pos(j);
    const F3 edge = f3(pj4) - f3(pi4);
    if (rest > kEps && surely_within(dot3(edge, edge), rest * cap_start_ratio(P, kind))) return false;
    const F3 qi = f3(st.prev(i)), qj = f3(st.prev(j));
    CapSide si, sj;
    if (!cap_edge(P, kind, rest, pi4, pj4, qi, qj, &si, &sj)) return true;
    if (si.ok) {
        st.set_pos(i, f4(f3(pi4) + si.d, pi4.w));
        st.set_prev(i, f4(qi + si.pd, 0.0f));
    }
    if (sj.ok) {
        st.set_pos(j, f4(f3(pj4) + sj.d, pj4.w));
        st.set_prev(j, f4(qj + sj.pd, 0.0f));
    }
    return true;
}

__global__ void __launch_bounds__(kThreads) k_cap_range(View v, int start, int count, int kind) {
    const int local = blockIdx.x * blockDim.x + threadIdx.x;
    const int s = start + local;
    if (local >= count || s < 0 || s >= v.nE) return;
    const int2 ed = __ldg(&v.edges[s]);
    if (ed.x < 0 || ed.x >= v.nV) return;
    cap_item(GlobalState{v.pos, v.prev}, params_v(v, ed.x), v.nV, ed, __ldg(&v.edge_rest[s]), kind);
}

// Caps of a cloth without a caller's colouring: the reference launches one
// kernel over every edge, each adding its corrections to both endpoints with
// float atomics (abi41.cu:7794-7801), i.e. a Jacobi pass.  Here every edge
// sees the positions and previous positions at the start of the pass and
// each vertex adds its edges' corrections in edge order (vertex -> edge CSR)
// into pos_out / prev_out; k_cap_store copies them back.
template <class S>
__device__ __forceinline__ void cap_jacobi_item(const View& v, const S& st, const Params& P, int i, int kind, float4* pos_out,
                                                float4* prev_out) {
    const float4 self4 = st.pos(i);
    const F3 self_prev = f3(st.prev(i));
    F3 p = f3(self4), q = self_prev;
    for (int k = v.sp_off[i]; k < v.sp_off[i + 1]; ++k) {
        const int2 e = __ldg(&v.sp_ent[k]);
        const bool self_is_j = (e.x & kSideBit) != 0;
        const int o = e.x & 0x7fffffff;
        const float4 o4 = st.pos(o);
        const F3 oq = f3(st.prev(o));
        CapSide si, sj;
        if (!cap_edge(P, kind, __int_as_float(e.y), self_is_j ? o4 : self4, self_is_j ? self4 : o4, self_is_j ? oq : self_prev,
                      self_is_j ? self_prev : oq, &si, &sj))
            continue;
        const CapSide& me = self_is_j ? sj : si;
        if (me.ok) {
            p = p + me.d;
            q = q + me.pd;
        }
    }
    *pos_out = f4(p, self4.w);
    *prev_out = f4(q, 0.0f);
}

__global__ void __launch_bounds__(kThreads) k_cap_jacobi(View v, int kind, float4* pos_out, float4* prev_out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= v.nV) return;
    const Params& P = params_v(v, i);
    if (P.pcg_hard && P.cap_jacobi) cap_jacobi_item(v, GlobalState{v.pos, v.prev}, P, i, kind, &pos_out[i], &prev_out[i]);
}

__global__ void __launch_bounds__(kThreads) k_cap_store(View v, const float4* pos_in, const float4* prev_in) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= v.nV) return;
    const Params& P = params_v(v, i);
    if (!P.pcg_hard || !P.cap_jacobi) return;
    v.pos[i] = pos_in[i];
    v.prev[i] = prev_in[i];
}

// -------------------------------------------------------- cluster form --
// The whole CG solve of a cloth, its averaged polish and its ratio caps by
// one thread-block cluster of C CTAs of T threads, N vertices per
// thread.  The launched form is bound by its launches: 23 per solve and one
// per cap colour and sweep (144 per substep on a 32 x 32 cloth), 2-3 us each
// for work of well under 1 us.  Per frame, launched and cluster form: 32 x 32
// with caps 4.4 -> 0.65 ms, 100 x 100 without 1.56 -> 0.66 ms.
//
// With the launches gone the steps are bound by load latency (600-800 cycles
// to L2 for every dependent gather), so the cluster's shared memory holds
// what neighbours read: each CTA its vertices' positions, previous positions,
// the two direction arrays and z, and its rows of the matrix with the
// neighbours' shared-memory addresses (rows past the space left stay in
// global memory).  A vertex keeps its diagonal block, preconditioner and
// residual in registers.
//
// A warp's partial of a dot product covers the same 32 vertices as in the
// launched form and goes to the same place of the same sum, into the shared
// memory of every CTA, so each warp computes the total itself in the launched
// form's order.  Two sets of partials alternate.  Every warp that waits for a
// sum also sends to it, zeros where it has no vertex: so a set is written
// again only when every warp that reads it has sent its partial of the sum
// between, and no warp falls a phase behind the counter it waits on.  Warps
// past the CTA's share (a smaller cloth of a batch) take no part.
//
// The direction update is folded into the next product: a neighbour's
// d = z + beta d_old is formed where it is read (the same fused step), and
// the own one is written to the other of two direction arrays, which saves
// the barrier that publishing d before the product would need.
//
// A sum's partials travel by st.async: the store and the arrival at the
// receiving CTA's counter are one trip through the cluster (about 800 cycles
// on 16 CTAs; the hardware's cluster barrier measured 1,600 with 32 warps per
// CTA, after which the partials would still have to be read).  The other
// barriers are one arrival per CTA at every CTA's counter.
constexpr int kHardSmem = 216 * 1024;
constexpr int kHardColors = 64;  // edge colours the caps keep in shared memory

// Vertex state in the cluster's shared memory: the own CTA's positions at the
// map's base, the previous positions after them.
template <bool kOne>
struct ClusterState {
    ClusterMap<kOne> map;
    int v0;
    __device__ __forceinline__ unsigned addr(int i) const { return map.addr(i - v0); }
    __device__ __forceinline__ float4 pos(int i) const { return ld_cluster<kOne>(addr(i)); }
    __device__ __forceinline__ float4 prev(int i) const { return ld_cluster<kOne>(addr(i) + 16u * map.chunk); }
    __device__ __forceinline__ void set_pos(int i, float4 x) const { st_cluster<kOne>(addr(i), x); }
    __device__ __forceinline__ void set_prev(int i, float4 x) const { st_cluster<kOne>(addr(i) + 16u * map.chunk, x); }
};

__device__ __forceinline__ F3 next_direction(F3 d, F3 z, float beta) {
    return F3{fmaf(d.x, beta, z.x), fmaf(d.y, beta, z.y), fmaf(d.z, beta, z.z)};
}

template <int T, int N, bool kOne>
__global__ void __launch_bounds__(T) k_hard_cluster(View v, PcgView g, HardPlan h, int final_caps) {
    const int kRows = h.rows;  // matrix entries kept in shared memory
    const int S = (int)blockDim.x;
    extern __shared__ float4 sm[];
    __shared__ float part[2][kHardMaxVertices / 32];
    __shared__ Params sP;
    __shared__ unsigned long long s_counter, s_sum[2];  // barrier; arrivals of the two sets of partials
    __shared__ int s_mark, s_any[2], s_lost;
    __shared__ int s_color[kHardColors + 1];  // first kept cap edge of each colour
    const cgx::cluster_group cluster = cgx::this_cluster();
    const int C = kOne ? 1 : (int)cluster.num_blocks(), rank = kOne ? 0 : (int)cluster.block_rank();
    const int cloth = __ldg(&h.cloths[blockIdx.x / C]);
    static_assert(sizeof(Params) % 4 == 0, "copied as words");
    for (int k = threadIdx.x; k < (int)(sizeof(Params) / 4); k += S)
        reinterpret_cast<unsigned*>(&sP)[k] = reinterpret_cast<const unsigned*>(&v.P[cloth])[k];
    // partials of the launched grid's warps past the cluster's stay zero (those
    // of the cluster's past the grid's are not read)
    for (int k = threadIdx.x; k < 2 * kHardMaxVertices / 32; k += S) (&part[0][0])[k] = 0.0f;
    if (threadIdx.x == 0) {
        ClusterBarrier::init(&s_counter, C);
        for (int k = 0; k < 2; ++k) ClusterBarrier::init(&s_sum[k], 1);
        ClusterBarrier::init_fence();
        s_mark = s_any[0] = s_any[1] = s_lost = 0;
    }
    __syncthreads();
    const Params& P = sP;
    if (final_caps && !P.pcg_hard) return;  // uniform over the cluster
    if (C > 1) cluster.sync();  // every CTA's counter is set before the first arrival
    ClusterBarrier bar{smem_addr(&s_counter), 0u, C, false};
    auto barrier = [&]() __attribute__((always_inline)) { bar.sync(); };
    const int lane = threadIdx.x & 31;
    const int V = P.V, v0 = P.vstart;
    // vertices per CTA: an even share in whole warps of the launched grid
    const int kChunk = max((V + 32 * C - 1) / (32 * C), 1) * 32;
    float4 *s_pos = sm, *s_prev = sm + kChunk, *s_d = sm + 2 * kChunk, *s_z = sm + 4 * kChunk;
    float4* s_off = sm + 5 * kChunk;
    unsigned* s_col = reinterpret_cast<unsigned*>(s_off + kRows);
    const int first = rank * kChunk + (int)threadIdx.x;  // local vertices first + n * S
    const ClusterState<kOne> st{ClusterMap<kOne>(smem_addr(s_pos), kChunk, rank), v0};
#pragma unroll
    for (int n = 0; n < N; ++n) {
        const int t = (int)threadIdx.x + n * S, l = rank * kChunk + t;
        if (t < kChunk && l < V) {
            s_pos[t] = v.pos[v0 + l];
            s_prev[t] = v.prev[v0 + l];
        }
    }
    barrier();
    if (!final_caps && (kOne || (int)threadIdx.x < kChunk)) {
        const int nw = P.pcg_nblocks * (kThreads / 32);  // warps of the launched grid, those past V included
        Sym diag[N], pinv[N];
        F3 r[N], q[N];
        float w[N];
        int begin[N], end[N];
        int sums = 0;
        auto total = [&](const float (&val)[N], bool publish) __attribute__((always_inline)) {
            float* mine = part[sums & 1];
            if (!kOne && threadIdx.x == 0)
                asm volatile("mbarrier.arrive.expect_tx.release.cta.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(&s_sum[sums & 1])),
                             "r"(4 * (C * kChunk / 32))
                             : "memory");
#pragma unroll
            for (int n = 0; n < N; ++n) {
                const int gw = (first + n * S) >> 5;
                const float t = __shfl_sync(0xffffffffu, warp_tree(val[n]), 0);
                const bool mine_too = (int)threadIdx.x + n * S < kChunk;
                if (kOne) {
                    if (mine_too && lane == 0) mine[gw] = t;
                } else {
                    if (publish) __syncwarp();
                    if (mine_too && lane < C) {
                        // the warp's writes that other CTAs read next go before the partial
                        if (publish) asm volatile("fence.acq_rel.cluster;" ::: "memory");
                        asm volatile("st.async.weak.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];" ::"r"(
                                         map_rank(smem_addr(&mine[gw]), lane)),
                                     "f"(t), "r"(map_rank(smem_addr(&s_sum[sums & 1]), lane))
                                     : "memory");
                    }
                }
            }
            if (kOne)
                __syncthreads();
            else
                bar.wait(smem_addr(&s_sum[sums & 1]), (sums >> 1) & 1);
            ++sums;
            float s = 0.0f;
            for (int k = lane; k < nw; k += 32) s += mine[k];
            return __shfl_sync(0xffffffffu, warp_tree(s), 0);
        };
        const int row0 = rank * kChunk < V ? v.sp_off[v0 + rank * kChunk] : 0;  // first matrix entry of this CTA
        float val[N];
#pragma unroll
        for (int n = 0; n < N; ++n) {
            const int t = (int)threadIdx.x + n * S, l = rank * kChunk + t;
            val[n] = 0.0f;
            w[n] = 0.0f;
            begin[n] = end[n] = 0;
            q[n] = F3{0.0f, 0.0f, 0.0f};
            if (t < kChunk && l < V) {
                const int i = v0 + l;
                F3 z;
                begin[n] = v.sp_off[i];
                end[n] = v.sp_off[i + 1];
                w[n] = s_pos[t].w;
                val[n] = build_item(v, st, g.guard, P, i, begin[n], end[n], &diag[n], &pinv[n], &r[n], &z, [&](int k, int other, float4 o) {
                    if (k - row0 < kRows) {
                        s_off[k - row0] = o;
                        s_col[k - row0] = st.addr(other);
                    } else {
                        g.offdiag[k] = o;
                    }
                });
                s_d[t] = s_z[t] = f4(z, 0.0f);
            }
        }
        float rz = total(val, true);
        const float initial = rz;
        float dad = 0.0f, rz_next = 0.0f, status = kStatusOk, iterations = 0.0f, beta = 0.0f;
        // written at the end: a fence would wait for them in every sum
        unsigned moved_bits = 0u, clamped = 0u;
        bool turn = false;  // the next product starts with d = z + beta d
        int from = 0;       // direction array the neighbours' d is read from
        for (int it = 0; it < 8; ++it) {
            // q = A d and d.q (k_pcg_ad)
            const unsigned d_off = (2u + from) * 16u * kChunk, z_off = 4u * 16u * kChunk;  // from a vertex's position address
#pragma unroll
            for (int n = 0; n < N; ++n) {
                const int t = (int)threadIdx.x + n * S;
                val[n] = 0.0f;
                if (t >= kChunk) continue;
                F3 d = f3(s_d[from * kChunk + t]);
                if (w[n] > 0.0f) {
                    if (turn) d = next_direction(d, f3(s_z[t]), beta);
                    q[n] = sym_madd(diag[n], d, F3{0.0f, 0.0f, 0.0f});
                    // two entries at a time: their loads are in flight together
                    for (int k = begin[n]; k < end[n]; k += 2) {
                        float4 o[2];
                        F3 od[2], oz[2];
#pragma unroll
                        for (int u = 0; u < 2; ++u) {
                            const int ku = min(k + u, end[n] - 1), e = ku - row0;
                            const unsigned a = e < kRows ? s_col[e] : st.addr(__ldg(&v.sp_ent[ku]).x & 0x7fffffff);
                            o[u] = e < kRows ? s_off[e] : g.offdiag[ku];
                            od[u] = f3(ld_cluster<kOne>(a + d_off));
                            if (turn) oz[u] = f3(ld_cluster<kOne>(a + z_off));
                        }
#pragma unroll
                        for (int u = 0; u < 2; ++u)
                            if (k + u < end[n]) q[n] = offdiag_madd(o[u], turn ? next_direction(od[u], oz[u], beta) : od[u], q[n]);
                    }
                    val[n] = dot3(d, q[n]);
                }
                if (turn) s_d[(from ^ 1) * kChunk + t] = f4(d, 0.0f);
            }
            if (turn) from ^= 1;
            dad = dad + total(val, false);
            const float alpha = cg_alpha(rz, dad, &status);
            if (status != kStatusOk) {
                // every remaining iteration finds the same status
                if (rank == 0 && threadIdx.x == 0 && status != kStatusZeroResidual) atomicAdd(g.guard, (unsigned long long)(8 - it));
                break;
            }
            // residual, preconditioned residual and positions (k_pcg_update)
#pragma unroll
            for (int n = 0; n < N; ++n) {
                const int t = (int)threadIdx.x + n * S;
                val[n] = 0.0f;
                if (w[n] > 0.0f) {
                    float moved_sq;
                    F3 z;
                    val[n] = update_item(GlobalState{s_pos, s_prev}, P, t, s_pos[t], f3(s_d[from * kChunk + t]), q[n], alpha, pinv[n],
                                         &r[n], &z, &moved_sq, &clamped);
                    s_z[t] = f4(z, 0.0f);
                    if (moved_sq > 0.0f) moved_bits = max(moved_bits, __float_as_uint(moved_sq));
                }
            }
            rz_next = rz_next + total(val, true);
            iterations += 1.0f;
            if (it + 1 == 8) break;
            // beta and the scalar slots (k_pcg_dir)
            const bool ok = isfinite(rz) && isfinite(rz_next) && rz > 1.0e-14f && rz_next >= 0.0f;
            beta = ok ? rz_next / rz : 0.0f;
            turn = ok && isfinite(beta);
            if (isfinite(rz_next) && rz_next >= 0.0f) {
                rz = rz_next;
                dad = 0.0f;
                rz_next = 0.0f;
            }
        }
        moved_bits = __reduce_max_sync(0xffffffffu, moved_bits);
        clamped = __reduce_add_sync(0xffffffffu, clamped);
        if (lane == 0 && moved_bits) atomicMax(g.max_delta_bits, __float_as_uint(sqrtf(__uint_as_float(moved_bits))));
        if (lane == 0 && clamped) count_add(v.counts, kCntHardFallbacks, clamped);
        if (rank == 0 && threadIdx.x == 0) {
            float* R = g.red + cloth * kRedSlots;
            R[kRedRZ] = rz;
            R[kRedInitialRZ] = initial;
            R[kRedIterations] = iterations;
            R[kRedDAD] = dad;
            R[kRedRZNext] = rz_next;
            R[kRedStatus] = status;
        }
    }
    if (!final_caps && P.pcg_hard) barrier();  // the polish reads every vertex
    if (P.pcg_hard) {
        int epoch = 0;
        // Whether some edge of the cloth may be longer than `ratio` rest
        // lengths.  Below that a polish or cap sweep changes nothing, so the
        // stage is left out: the usual outcome for a cloth the CG solve
        // holds, at the cost of one read of the edges.
        auto longer = [&](float ratio) __attribute__((always_inline)) {
            ++epoch;
            bool found = false;
            for (int l = rank * S + (int)threadIdx.x; l < P.E; l += C * S) {
                const int2 ed = __ldg(&v.edges[P.estart + l]);
                const float rest = __ldg(&v.edge_rest[P.estart + l]);
                if (ed.x < 0 || ed.y < 0 || ed.x >= v.nV || ed.y >= v.nV || !(rest > kEps)) continue;
                const F3 edge = f3(st.pos(ed.y)) - f3(st.pos(ed.x));
                found |= !surely_within(dot3(edge, edge), rest * ratio);
            }
            if (found) s_mark = epoch;
            return bar.sync_any(&s_mark, &s_any[epoch & 1], epoch);
        };
        // The CTA's share of every colour's edges, padded to whole rounds of
        // the block, goes to the space of the matrix rows (done with by now)
        // before the first sweep: a sweep then reads shared memory only.
        // Vertex ids take 16 bits each.
        int2* s_edge = reinterpret_cast<int2*>(s_off);
        int kept = P.cap_jacobi || h.colors > kHardColors ? -1 : 0;  // 1 kept, 0 not yet, -1 read from global memory
        // the averaged polish and cap sweeps in order, one per round: twice
        // (polish + normal caps, two times tiny polish + tiny caps) and the
        // extreme caps; after the contacts normal, extreme and tiny caps
        for (int s = 0; s < (final_caps ? 3 : 7); ++s) {
            const int kind = final_caps ? (s == 0 ? 0 : (s == 1 ? 2 : 1)) : (s == 6 ? 2 : (s % 3 > 0 ? 1 : 0));
            if (kind == 1 && !P.cap_tiny) continue;
            const bool polish = !final_caps && s < 6;
            if (!longer(polish ? (kind ? 1.06f : averaged_target(P, false, 1.0f)) : cap_start_ratio(P, kind))) continue;
            if (polish) {
                float4 a[N];
#pragma unroll
                for (int n = 0; n < N; ++n)
                    if ((int)threadIdx.x + n * S < kChunk && first + n * S < V) a[n] = avg_gather_item(v, st, P, v0 + first + n * S, kind);
                barrier();
#pragma unroll
                for (int n = 0; n < N; ++n)
                    if ((int)threadIdx.x + n * S < kChunk && first + n * S < V)
                        avg_apply_item(v, GlobalState{s_pos, s_prev}, P, (int)threadIdx.x + n * S, kind, a[n]);
                barrier();
            }
            const int passes = kind == 0 ? 2 : 3;
            if (P.cap_jacobi) {
                for (int p = 0; p < passes; ++p) {
                    float4 np[N], nq[N];
#pragma unroll
                    for (int n = 0; n < N; ++n)
                        if ((int)threadIdx.x + n * S < kChunk && first + n * S < V)
                            cap_jacobi_item(v, st, P, v0 + first + n * S, kind, &np[n], &nq[n]);
                    barrier();
#pragma unroll
                    for (int n = 0; n < N; ++n)
                        if ((int)threadIdx.x + n * S < kChunk && first + n * S < V) {
                            s_pos[threadIdx.x + n * S] = np[n];
                            s_prev[threadIdx.x + n * S] = nq[n];
                        }
                    barrier();
                }
                continue;
            }
            if (kept == 0) {
                int at = 0;
                kept = 1;
                for (int c = 0; c < h.colors; ++c) {
                    const int2 rg = __ldg(&h.ranges[c * v.K + cloth]);
                    const int rounds = (rg.y + C * S - 1) / (C * S);
                    if (threadIdx.x == 0) s_color[c] = at;
                    if ((at + rounds * S) * 8 > kRows * 20) {
                        kept = -1;
                        break;
                    }
                    for (int m = 0; m < rounds; ++m) {
                        const int l = (m * C + rank) * S + (int)threadIdx.x;
                        int2 e = make_int2(-1, 0);
                        if (l < rg.y) {
                            const int2 ed = __ldg(&h.edges[rg.x + l]);
                            if (ed.x >= 0 && ed.y >= 0 && ed.x != ed.y)
                                e = make_int2(((ed.x - v0) << 16) | (ed.y - v0), __float_as_int(__ldg(&h.rest[rg.x + l])));
                        }
                        s_edge[at + m * S + threadIdx.x] = e;
                    }
                    at += rounds * S;
                }
                if (threadIdx.x == 0) s_color[h.colors] = at;
                __syncthreads();
            }
            // colours forward, in the normal caps backward as well; a sweep
            // without a long edge leaves nothing for the sweeps after it
            const int turns = kind == 0 ? 2 * passes : passes;
            for (int p = 0; p < turns; ++p) {
                const bool back = kind == 0 && (p & 1);
                ++epoch;
                for (int k = 0; k < h.colors; ++k) {
                    const int c = back ? h.colors - 1 - k : k;
                    bool hit = false;
                    if (kept > 0) {
                        for (int m = s_color[c] + (int)threadIdx.x; m < s_color[c + 1]; m += S) {
                            const int2 e = s_edge[m];
                            if (e.x >= 0)
                                hit |= cap_item(st, P, v.nV, make_int2(v0 + (e.x >> 16), v0 + (e.x & 0xffff)), __int_as_float(e.y), kind);
                        }
                    } else {
                        const int2 rg = __ldg(&h.ranges[c * v.K + cloth]);
                        for (int l = rank * S + (int)threadIdx.x; l < rg.y; l += C * S)
                            hit |= cap_item(st, P, v.nV, __ldg(&h.edges[rg.x + l]), __ldg(&h.rest[rg.x + l]), kind);
                    }
                    if (hit) s_mark = epoch;
                    if (k + 1 < h.colors) barrier();
                }
                if (!bar.sync_any(&s_mark, &s_any[epoch & 1], epoch)) break;
            }
        }
    }
    if (bar.end(&s_lost)) {  // positions stay as they were
        if (threadIdx.x == 0) *v.lost = 1;
        return;
    }
#pragma unroll
    for (int n = 0; n < N; ++n) {
        const int t = (int)threadIdx.x + n * S, l = rank * kChunk + t;
        if (t < kChunk && l < V) {
            v.pos[v0 + l] = s_pos[t];
            v.prev[v0 + l] = s_prev[t];
        }
    }
}

}  // namespace

int pcg_blocks(int V) { return V > 0 ? blocks_for(V) : 0; }

void pcg_solve(const View& v, const PcgView& g, int blocks, cudaStream_t s, long long* launches) {
    if (blocks <= 0) return;
    const int b = blocks;
    k_pcg_build<<<b, kThreads, 0, s>>>(v, g);
    for (int it = 0; it < 8; ++it) {
        k_pcg_ad<<<b, kThreads, 0, s>>>(v, g);
        k_pcg_update<<<b, kThreads, 0, s>>>(v, g);
        *launches += 2;
        if (it + 1 < 8) {
            k_pcg_dir<<<b, kThreads, 0, s>>>(v, g);
            *launches += 1;
        }
    }
    *launches += 1;
}

namespace {

template <int T, int N, bool kOne>
int hard_fit(int c) {
    return cluster_fit(k_hard_cluster<T, N, kOne>, c, T, kHardSmem, kHardSmem);
}

template <int T, int N, bool kOne>
void hard_launch(const View& v, const PcgView& g, const HardPlan& h, bool final_caps, cudaStream_t s) {
    cluster_launch(k_hard_cluster<T, N, kOne>, h.cloth_count, h.cluster, h.threads, (size_t)5 * 16 * h.chunk + 20 * (size_t)h.rows, s, v,
                   g, h, final_caps ? 1 : 0);
}

}  // namespace

bool hard_plan(HardPlan* h, int max_v, int degree, int cloths, bool hard) {
    h->cluster = 0;
    // Past 1,280 vertices per CTA the launched form's whole-chip passes win
    // for the solve alone (us per frame, launched / cluster: 1,762 / 1,509 at
    // 19,600 vertices, 1,693 / 1,752 at 25,600); with caps the cluster form
    // does up to the vertices it can address (10,046 / 3,472 at 32,400).
    if (max_v <= 0 || max_v > (hard ? kHardMaxVertices : 1280 * kHardMaxCluster)) return false;
    // one CTA up to 1,024 vertices with caps, whose colour steps are bound by
    // their barriers (930 cycles a step against 1,900 on 16 CTAs); else as
    // many CTAs as the cluster may have (the solve of 1,024 vertices without
    // cap work: 69 us per substep on one CTA, 57 on 16)
    int c = max_v <= 1024 && hard ? 1 : kHardMaxCluster;
    while (c > 1 && (long long)c * cloths > 152) c /= 2;
    const int chunk = std::max((max_v + 32 * c - 1) / (32 * c), 1) * 32;
    const int n = chunk <= 640 ? 1 : (chunk <= 1024 ? 2 : 4);
    if (chunk > 2048 || (long long)c * cloths > 152) return false;
    // the cluster has to fit this GPU's processing clusters
    const int fit = n == 1 ? (c == 1 ? hard_fit<640, 1, true>(c) : hard_fit<640, 1, false>(c))
                           : n == 2 ? (c == 1 ? hard_fit<512, 2, true>(c) : hard_fit<512, 2, false>(c))
                                    : hard_fit<512, 4, false>(c);
    if (fit < 1) return false;
    h->cluster = c;
    h->chunk = chunk;
    h->threads = (chunk / n + 31) / 32 * 32;
    h->rows = std::min((kHardSmem - 5 * 16 * chunk) / 20, degree * chunk);
    return true;
}

void hard_cluster(const View& v, const PcgView& g, const HardPlan& h, bool final_caps, cudaStream_t s) {
    const bool one = h.cluster == 1;
    if (h.chunk <= 640 && one)
        hard_launch<640, 1, true>(v, g, h, final_caps, s);
    else if (h.chunk <= 640)
        hard_launch<640, 1, false>(v, g, h, final_caps, s);
    else if (h.chunk <= 1024 && one)
        hard_launch<512, 2, true>(v, g, h, final_caps, s);
    else if (h.chunk <= 1024)
        hard_launch<512, 2, false>(v, g, h, final_caps, s);
    else
        hard_launch<512, 4, false>(v, g, h, final_caps, s);
}

void pcg_averaged_pass(const View& v, const PcgView& g, int V, bool tiny, cudaStream_t s) {
    if (V <= 0) return;
    k_avg_gather<<<blocks_for(V), kThreads, 0, s>>>(v, g, tiny ? 1 : 0);
    k_avg_apply<<<blocks_for(V), kThreads, 0, s>>>(v, g, tiny ? 1 : 0);
}

void pcg_cap_range(const View& v, int start, int count, int kind, cudaStream_t s) {
    if (count > 0) k_cap_range<<<blocks_for(count), kThreads, 0, s>>>(v, start, count, kind);
}

void pcg_cap_jacobi(const View& v, const PcgView& g, int V, int kind, cudaStream_t s) {
    if (V <= 0) return;
    k_cap_jacobi<<<blocks_for(V), kThreads, 0, s>>>(v, kind, g.r, g.z);
    k_cap_store<<<blocks_for(V), kThreads, 0, s>>>(v, g.r, g.z);
}

}  // namespace xg
