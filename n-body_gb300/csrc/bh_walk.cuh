// Device pieces of the Barnes-Hut walks shared by their kernels (bh.cu, walk_team.cu): the force of a record
// or of a run of bodies, the decision of a record for a set of bodies from its box, the union walk of a subtree,
// and the fused integrator.
#pragma once

#include "bh.h"
#include "common.cuh"

namespace nbody {

// Float min / max through unsigned atomics on an order-preserving encoding
// (exact and order-independent, as the single-system reduction).
__device__ __forceinline__ unsigned ord_of(float f) {
    const unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float float_of(unsigned o) {
    return __uint_as_float((o & 0x80000000u) ? (o & 0x7fffffffu) : ~o);
}

// Both bodies of a lane summing the same run of bodies in one packed loop;
// side A takes part when doA, side B when doB. Per side the arithmetic and
// its rounding are those of direct_sum_range: a side that does not take part,
// or a pair it skips (m == 0 or r^2 == 0), adds dx * 0 = +0 to its sums.
// U bodies are loaded before they are summed (the order of the sums is the
// same for every U).
template <int U = 1>
__device__ __forceinline__ void direct_sum_range2(const float4 *__restrict__ pos, int64_t n, int first, int count,
                                                  float2 nx, float2 ny, float2 nz, float eps2, bool doA, bool doB,
                                                  float2 &ax, float2 &ay, float2 &az) {
    const int q0 = first < 0 ? 0 : first;
    const int q1 = first + count < n ? first + count : static_cast<int>(n);
    for (int q = q0; q < q1; q += U) {
        float4 r[U];
#pragma unroll
        for (int u = 0; u < U; ++u) r[u] = q + u < q1 ? pos[q + u] : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const float4 o = r[u];
            const float2 ex = __fadd2_rn(make_float2(o.x, o.x), nx);
            const float2 ey = __fadd2_rn(make_float2(o.y, o.y), ny);
            const float2 ez = __fadd2_rn(make_float2(o.z, o.z), nz);
            const float2 r2 = __fadd2_rn(__fadd2_rn(__fmul2_rn(ex, ex), __fmul2_rn(ey, ey)), __fmul2_rn(ez, ez));
            const float2 iv = make_float2(rsqrt_ftz(r2.x + eps2), rsqrt_ftz(r2.y + eps2));
            const float2 w = __fmul2_rn(__fmul2_rn(__fmul2_rn(make_float2(o.w, o.w), iv), iv), iv);
            const bool ua = doA && o.w > 0.f && r2.x > 0.f, ub = doB && o.w > 0.f && r2.y > 0.f;
            const float2 ws = make_float2(ua ? w.x : 0.f, ub ? w.y : 0.f);
            ax = __ffma2_rn(ex, ws, ax);
            ay = __ffma2_rn(ey, ws, ay);
            az = __ffma2_rn(ez, ws, az);
        }
    }
}

// One body summing a run of bodies, with the pair count and the potential where asked for.
__device__ __forceinline__ void direct_sum_range(const float4 *__restrict__ pos, int64_t n, int first, int count,
                                                 float4 me, float eps2, float &fx, float &fy, float &fz,
                                                 unsigned long long &n_pairs, bool count_pairs, float &phi,
                                                 bool pot) {
    const int q0 = first < 0 ? 0 : first;
    const int q1 = first + count < n ? first + count : static_cast<int>(n);
    for (int q = q0; q < q1; ++q) {
        const float4 o = pos[q];
        const float ex = __fsub_rn(o.x, me.x), ey = __fsub_rn(o.y, me.y), ez = __fsub_rn(o.z, me.z);
        const float e2 = __fadd_rn(__fadd_rn(__fmul_rn(ex, ex), __fmul_rn(ey, ey)), __fmul_rn(ez, ez));
        if (o.w > 0.f && e2 > 0.f) {
            if (count_pairs) ++n_pairs;
            const float iv = rsqrt_ftz(e2 + eps2);
            const float wq = o.w * iv * iv * iv;
            fx = fmaf(ex, wq, fx);
            fy = fmaf(ey, wq, fy);
            fz = fmaf(ez, wq, fz);
            if (pot) phi = fmaf(-o.w, iv, phi);
        }
    }
}

// Body b's new state into the caller's arrays at its caller index.
__device__ __forceinline__ void write_host(const HostOut host, const int *__restrict__ ids, int64_t b, int64_t n,
                                        float4 p, float4 v, float4 a) {
    const int d = ids ? ids[b] : static_cast<int>(b);
    if (d < 0 || d >= n) return;
    host.pos[d] = make_float4(p.x, p.y, p.z, 0.f);
    host.vel[d] = v;
    host.acc[d] = a;
    if (host.force) host.force[d] = a;
}

__device__ __forceinline__ void integrate_sorted(int64_t b, float4 p, float fx, float fy, float fz, float dt,
                                                 float4 *__restrict__ pos_out, float4 *__restrict__ vel,
                                                 float4 *__restrict__ acc, float4 *__restrict__ force_out,
                                                 const int *__restrict__ ids, int64_t n, int euler,
                                                 const HostOut &host = HostOut{}) {
    const float4 anew = make_float4(fx, fy, fz, 0.f);
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (pos_out && euler) {
        // updateParticles.glsl:44-55: v += F dt, then x += v dt.
        v = vel[b];
        v.x = __fadd_rn(v.x, __fmul_rn(fx, dt));
        v.y = __fadd_rn(v.y, __fmul_rn(fy, dt));
        v.z = __fadd_rn(v.z, __fmul_rn(fz, dt));
        p.x = __fadd_rn(p.x, __fmul_rn(v.x, dt));
        p.y = __fadd_rn(p.y, __fmul_rn(v.y, dt));
        p.z = __fadd_rn(p.z, __fmul_rn(v.z, dt));
        pos_out[b] = p;
        vel[b] = v;
        acc[b] = anew;
    } else if (pos_out) {
        // Reference integrator (include/ParticleSystem.h:52-69), no contraction.
        const float h = __fmul_rn(dt, 0.5f);
        v = vel[b];
        const float4 a = acc[b];
        v.x = __fadd_rn(v.x, __fmul_rn(a.x, h));
        v.y = __fadd_rn(v.y, __fmul_rn(a.y, h));
        v.z = __fadd_rn(v.z, __fmul_rn(a.z, h));
        p.x = __fadd_rn(p.x, __fmul_rn(v.x, dt));
        p.y = __fadd_rn(p.y, __fmul_rn(v.y, dt));
        p.z = __fadd_rn(p.z, __fmul_rn(v.z, dt));
        v.x = __fadd_rn(v.x, __fmul_rn(fx, h));
        v.y = __fadd_rn(v.y, __fmul_rn(fy, h));
        v.z = __fadd_rn(v.z, __fmul_rn(fz, h));
        pos_out[b] = p;
        vel[b] = v;
        acc[b] = anew;
    }
    if (force_out) {
        const int d = ids ? ids[b] : static_cast<int>(b);
        if (d >= 0 && d < n) force_out[d] = anew;
    }
    if (host.pos && pos_out) write_host(host, ids, b, n, p, v, anew);
}

// Two bodies per lane: a warp serves 64 consecutive sorted bodies (lane l
// holds bodies base + l and base + 32 + l), so each record load, vote and
// branch is shared by twice the bodies. The criterion and forces use packed
// f32x2 arithmetic, each lane of a pair rounded exactly as the scalar walk.
// The union walk over the records [i, iend) (the whole tree, or the subtree
// of record i) for the lane's bodies whose flags vA / vB are set, all active
// at record i: each evaluates the reference criterion on the records it has
// not covered (skip <= i); an accepted record adds its force and sets skip to
// the record's `next`; the warp descends if any lane opened the record, else
// jumps to the smallest skip. Sums go to fx, fy, fz (x: body A, y: body B).
template <bool COUNT, bool POT, bool GUARD>
__device__ __forceinline__ void union_range(const BHNode *__restrict__ nodes, const float4 *__restrict__ pos,
                                            int64_t n, int i, const int iend, const bool vA, const bool vB,
                                            const float2 nx, const float2 ny, const float2 nz, const float2 th,
                                            const float eps2, float2 &fx, float2 &fy, float2 &fz, float &phiA,
                                            float &phiB, unsigned long long &n_pairs,
                                            unsigned long long &n_visits) {
    const float2 e2 = make_float2(eps2, eps2);
    int skipA = vA ? i : iend, skipB = vB ? i : iend;
    while (i < iend) {
        const float4 cm = __ldg(&nodes[i].cm);
        const int4 meta = __ldg(&nodes[i].meta);
        const bool actA = skipA <= i, actB = skipB <= i;
        const float2 dx = __fadd2_rn(make_float2(cm.x, cm.x), nx);
        const float2 dy = __fadd2_rn(make_float2(cm.y, cm.y), ny);
        const float2 dz = __fadd2_rn(make_float2(cm.z, cm.z), nz);
        const float2 d2 = __fadd2_rn(__fadd2_rn(__fmul2_rn(dx, dx), __fmul2_rn(dy, dy)), __fmul2_rn(dz, dz));
        const float s2 = __int_as_float(meta.x);
        const float2 rhs = __fmul2_rn(th, d2);
        bool accA, accB, useA, useB;
        if (GUARD) {
            accA = actA && (s2 < 0.f || s2 < rhs.x);
            accB = actB && (s2 < 0.f || s2 < rhs.y);
            const bool self = meta.w <= 1 && cm.w > 0.f;
            useA = accA && self && d2.x > 0.f;
            useB = accB && self && d2.y > 0.f;
        } else {
            accA = actA && s2 < rhs.x;
            accB = actB && s2 < rhs.y;
            const bool self = meta.w <= 1;  // a bucket's bodies are summed one by one below
            useA = accA && self;
            useB = accB && self;
        }
        if (useA || useB) {
            if (COUNT) n_pairs += (useA ? 1u : 0u) + (useB ? 1u : 0u);
            const float2 e = __fadd2_rn(d2, e2);
            const float2 inv = make_float2(rsqrt_ftz(e.x), rsqrt_ftz(e.y));
            const float2 inv3 = __fmul2_rn(__fmul2_rn(inv, inv), inv);
            const float2 mw = __fmul2_rn(make_float2(cm.w, cm.w), inv3);
            const float2 w = make_float2(useA ? mw.x : 0.f, useB ? mw.y : 0.f);
            fx = __ffma2_rn(dx, w, fx);
            fy = __ffma2_rn(dy, w, fy);
            fz = __ffma2_rn(dz, w, fz);
            if (POT) {
                phiA = fmaf(useA ? -cm.w : 0.f, inv.x, phiA);
                phiB = fmaf(useB ? -cm.w : 0.f, inv.y, phiB);
            }
        }
        if (meta.w != 0 && meta.w != 1) {  // warp-uniform: a bucket or a terminal cell
            const int cntb = meta.w >= 2 ? meta.w : -meta.w;
            const bool doA = (meta.w >= 2 && accA) || (meta.w < 0 && actA && !accA);
            const bool doB = (meta.w >= 2 && accB) || (meta.w < 0 && actB && !accB);
            if (COUNT || POT) {
                const float4 meA = make_float4(-nx.x, -ny.x, -nz.x, 0.f), meB = make_float4(-nx.y, -ny.y, -nz.y, 0.f);
                if (doA) direct_sum_range(pos, n, meta.z, cntb, meA, eps2, fx.x, fy.x, fz.x, n_pairs, COUNT, phiA, POT);
                if (doB) direct_sum_range(pos, n, meta.z, cntb, meB, eps2, fx.y, fy.y, fz.y, n_pairs, COUNT, phiB, POT);
            } else if (doA || doB) {
                direct_sum_range2(pos, n, meta.z, cntb, nx, ny, nz, eps2, doA, doB, fx, fy, fz);
            }
        }
        const bool doneA = accA || (actA && meta.w < 0), doneB = accB || (actB && meta.w < 0);
        if (doneA) skipA = meta.y;
        if (doneB) skipB = meta.y;
        const bool open = (actA && !doneA) || (actB && !doneB);
        if (COUNT) ++n_visits;
        if (__any_sync(0xffffffffu, open)) {
            ++i;
        } else {
            const int mine = skipA < skipB ? skipA : skipB;
            const int nx2 = static_cast<int>(__reduce_min_sync(0xffffffffu, static_cast<unsigned>(mine)));
            i = nx2 > i ? nx2 : i + 1;
        }
    }
}

// Deciding for a set.
// From the box of a set of bodies, a record is
//   accepted by all  when s^2 < theta^2 * d2lo, d2lo the least squared
//                    distance to the box in the walk's own rounding (each
//                    step is monotone, so every body's d^2 >= d2lo and its
//                    product >= theta^2 * d2lo: the body accepts), or when it
//                    is a lone body (every body accepts a leaf);
//   opened by all    when it is a plain cell and s^2 >= theta^2 * d2hi, d2hi
//                    the largest squared distance in the same rounding;
//   ambiguous        otherwise (and for buckets and terminal cells that are
//                    not accepted by all), to be decided body by body.
struct SetBox {
    float lx, ly, lz, hx, hy, hz;
};

// 0: accepted by every body in the box; 1: opened by every body (a plain
// cell); 2: ambiguous.
__device__ __forceinline__ int certify(const float4 cm, const int4 meta, const SetBox &b, const float theta2) {
    if (meta.w == 1) return 0;  // a lone body: a leaf is always accepted
    if (meta.w >= 2) return 2;  // a bucket: its bodies are summed one by one in the walk
    const float s2 = __int_as_float(meta.x);
    // per axis, the least |dx| over the box (0 inside it) and the largest, both
    // rounded as the walk rounds cm - p
    const float gx = fmaxf(fmaxf(__fsub_rn(b.lx, cm.x), __fsub_rn(cm.x, b.hx)), 0.f);
    const float gy = fmaxf(fmaxf(__fsub_rn(b.ly, cm.y), __fsub_rn(cm.y, b.hy)), 0.f);
    const float gz = fmaxf(fmaxf(__fsub_rn(b.lz, cm.z), __fsub_rn(cm.z, b.hz)), 0.f);
    const float lo2 = __fadd_rn(__fadd_rn(__fmul_rn(gx, gx), __fmul_rn(gy, gy)), __fmul_rn(gz, gz));
    if (s2 < __fmul_rn(theta2, lo2)) return 0;
    if (meta.w != 0) return 2;
    const float ux = fmaxf(fabsf(__fsub_rn(cm.x, b.lx)), fabsf(__fsub_rn(b.hx, cm.x)));
    const float uy = fmaxf(fabsf(__fsub_rn(cm.y, b.ly)), fabsf(__fsub_rn(b.hy, cm.y)));
    const float uz = fmaxf(fabsf(__fsub_rn(cm.z, b.lz)), fabsf(__fsub_rn(b.hz, cm.z)));
    const float hi2 = __fadd_rn(__fadd_rn(__fmul_rn(ux, ux), __fmul_rn(uy, uy)), __fmul_rn(uz, uz));
    return s2 < __fmul_rn(theta2, hi2) ? 2 : 1;
}

// Least / largest value over the warp (exact; a NaN is passed over).
__device__ __forceinline__ float warp_min(float x) {
    float y;
    asm volatile("redux.sync.min.f32 %0, %1, 0xffffffff;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float warp_max(float x) {
    float y;
    asm volatile("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(y) : "f"(x));
    return y;
}

// Box of the bodies in masks sa / sb (exact min / max). Six float reductions
// over the warp; through the order-preserving integer image each coordinate
// took three more instructions per body and three to come back. With the
// fused d^2 of add_record: 3.24 against 3.40 ms per walk of 2^20 Plummer
// bodies (GB300).
__device__ __forceinline__ SetBox set_box(unsigned sa, unsigned sb, int lane, float4 pa, float4 pb) {
    const bool ia = (sa >> lane) & 1u, ib = (sb >> lane) & 1u;
    const float inf = __int_as_float(0x7f800000);
    SetBox b;
    b.lx = warp_min(fminf(ia ? pa.x : inf, ib ? pb.x : inf));
    b.ly = warp_min(fminf(ia ? pa.y : inf, ib ? pb.y : inf));
    b.lz = warp_min(fminf(ia ? pa.z : inf, ib ? pb.z : inf));
    b.hx = warp_max(fmaxf(ia ? pa.x : -inf, ib ? pb.x : -inf));
    b.hy = warp_max(fmaxf(ia ? pa.y : -inf, ib ? pb.y : -inf));
    b.hz = warp_max(fmaxf(ia ? pa.z : -inf, ib ? pb.z : -inf));
    return b;
}

// The record's force on each of the lane's bodies whose flag is set (the
// walk's arithmetic; GUARD keeps the explicit zero-distance and massless
// tests).
template <bool COUNT, bool POT, bool GUARD>
__device__ __forceinline__ void add_record(const float4 cm, bool useA, bool useB, const float2 nx, const float2 ny,
                                           const float2 nz, const float2 e2, float2 &fx, float2 &fy, float2 &fz,
                                           float &phiA, float &phiB, unsigned long long &n_pairs) {
    const float2 dx = __fadd2_rn(make_float2(cm.x, cm.x), nx);
    const float2 dy = __fadd2_rn(make_float2(cm.y, cm.y), ny);
    const float2 dz = __fadd2_rn(make_float2(cm.z, cm.z), nz);
    float2 ee;
    if (GUARD) {
        const float2 d2 = __fadd2_rn(__fadd2_rn(__fmul2_rn(dx, dx), __fmul2_rn(dy, dy)), __fmul2_rn(dz, dz));
        useA = useA && cm.w > 0.f && d2.x > 0.f;
        useB = useB && cm.w > 0.f && d2.y > 0.f;
        ee = __fadd2_rn(d2, e2);
    } else {  // no decision hangs on d^2 here: three fused operations instead of six
        ee = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __ffma2_rn(dx, dx, e2)));
    }
    const float2 inv = make_float2(rsqrt_ftz(ee.x), rsqrt_ftz(ee.y));
    const float2 inv3 = __fmul2_rn(__fmul2_rn(inv, inv), inv);
    const float2 mw = __fmul2_rn(make_float2(cm.w, cm.w), inv3);
    const float2 w = make_float2(useA ? mw.x : 0.f, useB ? mw.y : 0.f);
    fx = __ffma2_rn(dx, w, fx);
    fy = __ffma2_rn(dy, w, fy);
    fz = __ffma2_rn(dz, w, fz);
    if (COUNT) n_pairs += (useA ? 1u : 0u) + (useB ? 1u : 0u);
    if (POT) {
        phiA = fmaf(useA ? -cm.w : 0.f, inv.x, phiA);
        phiB = fmaf(useB ? -cm.w : 0.f, inv.y, phiB);
    }
}

}  // namespace nbody
