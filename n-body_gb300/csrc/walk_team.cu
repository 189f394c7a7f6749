// The cell walk by a team of warps: one CTA of W warps serves one set of 64
// consecutive sorted bodies (two per lane, the same bodies in every warp), for
// systems too small to fill the GPU with one warp per set.
//
// What bounds it. With one warp per set a system of n bodies has n / 64 warps,
// each a serial chain of some 300-500 cells whose children are fetched (two
// dependent loads), decided and summed: a system of 4,096 bodies keeps 64 of
// the chip's 608 schedulers busy, one warp each, for as long as the longest
// chain takes (372 us; 53 us by teams of 16).
//
// Rounds. The warps take the top 4 W cells of one shared stack, cell j of a
// round going to warp j % W. A warp decides its cells' children for their sets
// (certify), sums those accepted by all into its own sums, and leaves the
// cells opened by all and the ambiguous children in areas of its own. Between
// two barriers the opened cells go to the stack in warp order; the ambiguous
// children, which cost most and gather in few cells, are shared out evenly in
// the next round (deciding each where it turned up: 87 against 74 us for 4,096
// bodies and 8 warps). Nothing depends on which warp is faster, so the result
// is the same on every run; it depends on W, which follows from the system's
// size alone (bh_team_size), so a system gives the same bits alone and in an
// ensemble. Per body the accepted records are those of cell_walk_kernel
// (bh.cu), in another order of summation; the W sums are added in warp order.
//
// Not kept: a stack per warp, shared out anew every one to four rounds (fewer
// barriers, but uneven warps: 308 against 288 us for 65,536 bodies and 8
// warps).
#include <cuda_runtime.h>

#include <cstdlib>

#include "bh.h"
#include "bh_walk.cuh"
#include "common.cuh"
#include "launch.h"

namespace nbody {

namespace {

// Stack entries: a round pops 4 W cells and pushes some 1.2 for each; a full
// stack hands a cell to union_range.
constexpr int team_depth(int W) { return W >= 16 ? 256 : W >= 8 ? 224 : W >= 4 ? 192 : 128; }
constexpr int kTeamPush = 40;  // a warp's push area: at most 32 cells opened by all, then those its bodies differ on

template <int W>
struct TeamArea {
    static constexpr int S = team_depth(W);
    int4 stk_i[S];     // cell, mask A, mask B, box hz (float bits)
    float4 stk_lo[S];  // box: lx, ly, lz, hx
    union {
        struct {
            int4 push_i[W][kTeamPush];  // what each warp opened in this round
            float4 push_lo[W][kTeamPush];
        };
        float sums[W][3][64];  // after the last round: every warp's sums of the 64 bodies
    };
    int4 amb[2][W][32];   // ambiguous children of the last round and of this one: record, mask A, mask B
    // The accepted children of each cell of a round, packed to the front of
    // its eight places, each coordinate twice (an operand of the packed sums).
    float4 ch_xy[W][32], ch_zm[W][32];
    float stk_hy[S];      // box: hy
    float push_hy[W][kTeamPush];
    int count[W];         // entries in push (low half) and amb (high half)
};

// The force of one child (its coordinates twice) on the lane's two bodies.
template <bool COUNT, bool GUARD, bool ALL>
__device__ __forceinline__ void add_kid(const float4 xy, const float4 zm, bool useA, bool useB, const float2 nx,
                                        const float2 ny, const float2 nz, const float2 e2, float2 &fx, float2 &fy,
                                        float2 &fz, unsigned long long &n_pairs) {
    const float2 dx = __fadd2_rn(make_float2(xy.x, xy.y), nx);
    const float2 dy = __fadd2_rn(make_float2(xy.z, xy.w), ny);
    const float2 dz = __fadd2_rn(make_float2(zm.x, zm.y), nz);
    float2 ee;
    if (GUARD) {
        const float2 d2 = __fadd2_rn(__fadd2_rn(__fmul2_rn(dx, dx), __fmul2_rn(dy, dy)), __fmul2_rn(dz, dz));
        useA = useA && zm.z > 0.f && d2.x > 0.f;
        useB = useB && zm.z > 0.f && d2.y > 0.f;
        ee = __fadd2_rn(d2, e2);
    } else {  // no decision hangs on d^2 here: three fused operations instead of six
        ee = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __ffma2_rn(dx, dx, e2)));
    }
    const float2 inv = make_float2(rsqrt_ftz(ee.x), rsqrt_ftz(ee.y));
    const float2 inv3 = __fmul2_rn(__fmul2_rn(inv, inv), inv);
    float2 w = __fmul2_rn(make_float2(zm.z, zm.w), inv3);
    if (GUARD || !ALL) w = make_float2(useA ? w.x : 0.f, useB ? w.y : 0.f);
    fx = __ffma2_rn(dx, w, fx);
    fy = __ffma2_rn(dy, w, fy);
    fz = __ffma2_rn(dz, w, fz);
    if (COUNT) n_pairs += (useA ? 1u : 0u) + (useB ? 1u : 0u);
}

template <bool COUNT, bool GUARD, bool ALL>
__device__ __forceinline__ void add_kids(const float4 *xy, const float4 *zm, int cnt, bool useA, bool useB,
                                         const float2 nx, const float2 ny, const float2 nz, const float2 e2, float2 &fx,
                                         float2 &fy, float2 &fz, unsigned long long &n_pairs) {
    int j = 0;
    for (; j + 4 <= cnt; j += 4) {
#pragma unroll
        for (int u = 0; u < 4; ++u)
            add_kid<COUNT, GUARD, ALL>(xy[j + u], zm[j + u], useA, useB, nx, ny, nz, e2, fx, fy, fz, n_pairs);
    }
    for (; j < cnt; ++j) add_kid<COUNT, GUARD, ALL>(xy[j], zm[j], useA, useB, nx, ny, nz, e2, fx, fy, fz, n_pairs);
}

// Registers: 64 (32 warps per SM), and up to 98 for the largest team of a
// single system, which rarely has more than one CTA per SM anyway (4,096
// bodies: 57 against 64 us at 64 registers); 48 registers lose at every size
// (65,536 bodies, 4 warps: 405 against 302 us).
template <int W, bool COUNT, bool SEG, bool GUARD, bool HOST>
__global__ void __launch_bounds__(32 * W, W >= 16 && !SEG ? 1 : 32 / W) team_walk_kernel(
    const BHNode *__restrict__ nodes, const int *__restrict__ kids, const uint32_t *__restrict__ node_total,
    const float4 *__restrict__ pos, int64_t n, float eps2, float theta2, float dt, float4 *__restrict__ pos_out,
    float4 *__restrict__ vel, float4 *__restrict__ acc, float4 *__restrict__ force_out, const int *__restrict__ ids,
    unsigned long long *__restrict__ counters, int euler, const int4 *__restrict__ work,
    const float4 *__restrict__ params, const uint32_t *__restrict__ P, const HostOut host, int64_t first, int beside,
    unsigned *ready) {
    __shared__ __align__(16) TeamArea<W> A;
    constexpr int S = TeamArea<W>::S;
    // Beside the walk before it (bh.h): what the build wrote is seen through that
    // walk's word, or, where it cannot be seen yet, by waiting for its end.
    if (!(beside & kWalkWaitsLast) || !__syncthreads_or(threadIdx.x == 0 && load_acquire(ready) != 0u))
        wait_for_launches_before();
    if (beside & kWalkLetsNext) {
        if (!(beside & kWalkWaitsLast) && blockIdx.x == 0 && threadIdx.x == 0) store_release(ready, 1u);
        let_next_launch_begin();
    }
    unsigned long long n_pairs = 0, n_visits = 0;
    float phi = 0.f;  // no potential in this form
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int64_t base, end;
    int root, rend;
    if (SEG) {
        const int4 ww = work[blockIdx.x];
        const float4 prm = params[ww.x];
        eps2 = prm.y;
        theta2 = prm.z;
        base = ww.y;
        end = ww.w;
        root = static_cast<int>(P[ww.z]);
        rend = static_cast<int>(P[ww.w]);
    } else {
        base = (first + blockIdx.x) * 64;
        end = n;
        root = 0;
        rend = static_cast<int>(*node_total);
    }
    const bool vA = base + lane < end, vB = base + lane + 32 < end;
    const float4 meA = vA ? pos[base + lane] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 meB = vB ? pos[base + lane + 32] : make_float4(0.f, 0.f, 0.f, 0.f);
    const float2 nx = make_float2(-meA.x, -meB.x), ny = make_float2(-meA.y, -meB.y), nz = make_float2(-meA.z, -meB.z);
    const float2 th = make_float2(theta2, theta2);
    const float2 e2 = make_float2(eps2, eps2);
    float2 fx = make_float2(0.f, 0.f), fy = make_float2(0.f, 0.f), fz = make_float2(0.f, 0.f);
    int pushed = 0;  // this warp's entries of the round

    // Record k decided body by body for the bodies in (sa, sb); the bodies
    // that open a plain cell are pushed with it.
    auto decide = [&](int k, const float4 cm, const int4 meta, unsigned sa, unsigned sb) {
        const bool actA = (sa >> lane) & 1u, actB = (sb >> lane) & 1u;
        const float2 dx = __fadd2_rn(make_float2(cm.x, cm.x), nx);
        const float2 dy = __fadd2_rn(make_float2(cm.y, cm.y), ny);
        const float2 dz = __fadd2_rn(make_float2(cm.z, cm.z), nz);
        const float2 d2 = __fadd2_rn(__fadd2_rn(__fmul2_rn(dx, dx), __fmul2_rn(dy, dy)), __fmul2_rn(dz, dz));
        const float s2 = __int_as_float(meta.x);
        const float2 rhs = __fmul2_rn(th, d2);
        const bool accA = actA && ((GUARD && s2 < 0.f) || s2 < rhs.x);
        const bool accB = actB && ((GUARD && s2 < 0.f) || s2 < rhs.y);
        const bool self = meta.w <= 1 && (!GUARD || cm.w > 0.f);
        const bool useA = accA && self && (!GUARD || d2.x > 0.f);
        const bool useB = accB && self && (!GUARD || d2.y > 0.f);
        if (COUNT) ++n_visits;
        const float2 ee = __fadd2_rn(d2, e2);
        const float2 inv = make_float2(rsqrt_ftz(ee.x), rsqrt_ftz(ee.y));
        const float2 inv3 = __fmul2_rn(__fmul2_rn(inv, inv), inv);
        const float2 mw = __fmul2_rn(make_float2(cm.w, cm.w), inv3);
        const float2 w = make_float2(useA ? mw.x : 0.f, useB ? mw.y : 0.f);
        fx = __ffma2_rn(dx, w, fx);
        fy = __ffma2_rn(dy, w, fy);
        fz = __ffma2_rn(dz, w, fz);
        if (COUNT) n_pairs += (useA ? 1u : 0u) + (useB ? 1u : 0u);
        if (meta.w != 0 && meta.w != 1) {  // a bucket accepted, or a terminal cell opened: body by body
            const int cntb = meta.w >= 2 ? meta.w : -meta.w;
            const bool doA = (meta.w >= 2 && accA) || (meta.w < 0 && actA && !accA);
            const bool doB = (meta.w >= 2 && accB) || (meta.w < 0 && actB && !accB);
            if (COUNT) {
                if (doA) direct_sum_range(pos, n, meta.z, cntb, meA, eps2, fx.x, fy.x, fz.x, n_pairs, COUNT, phi, false);
                if (doB) direct_sum_range(pos, n, meta.z, cntb, meB, eps2, fx.y, fy.y, fz.y, n_pairs, COUNT, phi, false);
            } else if (__any_sync(0xffffffffu, doA || doB)) {
                direct_sum_range2<4>(pos, n, meta.z, cntb, nx, ny, nz, eps2, doA, doB, fx, fy, fz);
            }
            return;
        }
        if (meta.w != 0) return;
        const unsigned oa = __ballot_sync(0xffffffffu, actA && !accA);
        const unsigned ob = __ballot_sync(0xffffffffu, actB && !accB);
        if (!(oa | ob)) return;
        if (pushed >= kTeamPush) {  // no room: the subtree record by record
            union_range<COUNT, false, GUARD>(nodes, pos, n, k + 1, meta.y, (oa >> lane) & 1u, (ob >> lane) & 1u, nx, ny,
                                             nz, th, eps2, fx, fy, fz, phi, phi, n_pairs, n_visits);
            return;
        }
        const SetBox b = set_box(oa, ob, lane, meA, meB);
        if (lane == 0) {
            A.push_i[warp][pushed] =
                make_int4(k, static_cast<int>(oa), static_cast<int>(ob), __float_as_int(b.hz));
            A.push_lo[warp][pushed] = make_float4(b.lx, b.ly, b.lz, b.hx);
            A.push_hy[warp][pushed] = b.hy;
        }
        ++pushed;
    };

    if (warp == 0 && root < rend)
        decide(root, __ldg(&nodes[root].cm), __ldg(&nodes[root].meta), __ballot_sync(0xffffffffu, vA),
               __ballot_sync(0xffffffffu, vB));
    const int grp = lane >> 3;
    int sp = 0;         // entries left under the round's cells, then all of them: the same in every warp
    int ambiguous = 0;  // this warp's entries in amb
    for (int parity = 0;; parity ^= 1) {
        // The round's pushes onto the stack, in warp order.
        if (lane == 0) A.count[warp] = pushed | ambiguous << 16;
        __syncthreads();  // counts, push and amb areas written; the popped entries read
        int upto = lane < W ? A.count[lane] : 0;  // inclusive prefix over the warps, both halves at once
        const int own = __shfl_sync(0xffffffffu, upto, warp);
#pragma unroll
        for (int off = 1; off < W; off <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, upto, off);
            if (lane >= off) upto += u;
        }
        const int all = __shfl_sync(0xffffffffu, upto, W - 1);
        const int at = sp + ((__shfl_sync(0xffffffffu, upto, warp) - own) & 0xffff);
        for (int q = lane; q < pushed; q += 32)
            if (at + q < S) {
                A.stk_i[at + q] = A.push_i[warp][q];
                A.stk_lo[at + q] = A.push_lo[warp][q];
                A.stk_hy[at + q] = A.push_hy[warp][q];
            }
        for (int q = at < S ? S - at : 0; q < pushed; ++q) {  // no room: the subtree record by record
            const int4 t = A.push_i[warp][q];
            const int kend = __ldg(&nodes[t.x].meta).y;
            const bool actA = (static_cast<unsigned>(t.y) >> lane) & 1u, actB = (static_cast<unsigned>(t.z) >> lane) & 1u;
            union_range<COUNT, false, GUARD>(nodes, pos, n, t.x + 1, kend, actA, actB, nx, ny, nz, th, eps2, fx, fy,
                                             fz, phi, phi, n_pairs, n_visits);
        }
        const int todo = all >> 16;  // ambiguous children of the round before
        upto = lane < W ? upto >> 16 : 0x7fff;
        sp += all & 0xffff;
        sp = sp < S ? sp : S;
        __syncthreads();  // the stack is whole
        if (sp == 0 && todo == 0) break;
        const int nb = sp < 4 * W ? sp : 4 * W;
        sp -= nb;
        pushed = 0;
        ambiguous = 0;
        // Cells warp, warp + W, ... of the round.
        if (warp < nb) {
            int kid = -1, cls = 3;
            float4 cm = make_float4(0.f, 0.f, 0.f, 0.f);
            const int mine = warp + W * grp;
            if (mine < nb) {
                const int4 t = A.stk_i[sp + mine];
                kid = __ldg(&kids[8 * static_cast<int64_t>(t.x) + (lane & 7)]);
                if (kid >= 0) {
                    const float4 bl = A.stk_lo[sp + mine];
                    const float hy = A.stk_hy[sp + mine];
                    SetBox box;
                    box.lx = bl.x;
                    box.ly = bl.y;
                    box.lz = bl.z;
                    box.hx = bl.w;
                    box.hy = hy;
                    box.hz = __int_as_float(t.w);
                    cm = __ldg(&nodes[kid].cm);
                    cls = certify(cm, __ldg(&nodes[kid].meta), box, theta2);
                }
            }
            const unsigned below = (1u << lane) - 1u;
            const unsigned bAcc = __ballot_sync(0xffffffffu, cls == 0);
            if (cls == 0) {
                const int to = 8 * grp + __popc(bAcc & below & (0xffu << (8 * grp)));
                A.ch_xy[warp][to] = make_float4(cm.x, cm.x, cm.y, cm.y);
                A.ch_zm[warp][to] = make_float4(cm.z, cm.z, cm.w, cm.w);
            }
            __syncwarp();
            const unsigned bOpen = __ballot_sync(0xffffffffu, cls == 1);
            const unsigned bAmb = __ballot_sync(0xffffffffu, cls == 2);
            if (COUNT) n_visits += __popc(bAcc | bOpen | bAmb);
            // Children opened by all go on with their cell's set and box;
            // ambiguous ones are shared out in the next round.
            if (cls == 1) {
                const int to = __popc(bOpen & below);
                const int4 t = A.stk_i[sp + mine];
                A.push_i[warp][to] = make_int4(kid, t.y, t.z, t.w);
                A.push_lo[warp][to] = A.stk_lo[sp + mine];
                A.push_hy[warp][to] = A.stk_hy[sp + mine];
            } else if (cls == 2) {
                const int4 t = A.stk_i[sp + mine];
                A.amb[parity][warp][__popc(bAmb & below)] = make_int4(kid, t.y, t.z, 0);
            }
            pushed = __popc(bOpen);
            ambiguous = __popc(bAmb);
            for (int q = 0; q < 4 && warp + W * q < nb; ++q) {
                const int cnt = __popc(bAcc & (0xffu << (8 * q)));
                const int4 t = A.stk_i[sp + warp + W * q];
                const float4 *xy = &A.ch_xy[warp][8 * q], *zm = &A.ch_zm[warp][8 * q];
                const bool actA = (static_cast<unsigned>(t.y) >> lane) & 1u,
                           actB = (static_cast<unsigned>(t.z) >> lane) & 1u;
                if ((t.y & t.z) == -1)
                    add_kids<COUNT, GUARD, true>(xy, zm, cnt, true, true, nx, ny, nz, e2, fx, fy, fz, n_pairs);
                else
                    add_kids<COUNT, GUARD, false>(xy, zm, cnt, actA, actB, nx, ny, nz, e2, fx, fy, fz, n_pairs);
            }
        }
        // Ambiguous children warp, warp + W, ... of the round before.
        for (int j = warp; j < todo; j += W) {
            const int v = __popc(__ballot_sync(0xffffffffu, upto <= j));  // whose area holds it
            const int first = v ? __shfl_sync(0xffffffffu, upto, v - 1) : 0;
            const int4 t = A.amb[parity ^ 1][v][j - first];
            decide(t.x, __ldg(&nodes[t.x].cm), __ldg(&nodes[t.x].meta), static_cast<unsigned>(t.y),
                   static_cast<unsigned>(t.z));
        }
    }

    if (COUNT) {
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) n_pairs += __shfl_down_sync(0xffffffffu, n_pairs, off);
        if (lane == 0) {
            atomicAdd(&counters[0], n_pairs);
            atomicAdd(&counters[1], n_visits);
        }
    }
    // The W sums of each body, in warp order, and the integrator.
    A.sums[warp][0][lane] = fx.x;
    A.sums[warp][0][lane + 32] = fx.y;
    A.sums[warp][1][lane] = fy.x;
    A.sums[warp][1][lane + 32] = fy.y;
    A.sums[warp][2][lane] = fz.x;
    A.sums[warp][2][lane + 32] = fz.y;
    __syncthreads();
    if ((beside & kWalkWaitsLast) && blockIdx.x == gridDim.x - 1) wait_for_launches_before();
    const int t = threadIdx.x;
    if (t >= 64) return;
    float gx = 0.f, gy = 0.f, gz = 0.f;
#pragma unroll
    for (int v = 0; v < W; ++v) {
        gx += A.sums[v][0][t];
        gy += A.sums[v][1][t];
        gz += A.sums[v][2][t];
    }
    if (SEG) {
        const int4 ww = work[blockIdx.x];
        const float4 prm = params[ww.x];
        dt = prm.x;
        euler = prm.w != 0.f ? 1 : 0;
    }
    const int64_t b = base + t;
    if (b < end)
        integrate_sorted(b, pos[b], gx, gy, gz, dt, pos_out, vel, acc, force_out, ids, n, euler,
                         HOST ? host : HostOut{});
}

template <int W, bool COUNT, bool SEG, bool GUARD>
cudaError_t launch_form(const TeamWalk &a, unsigned sets, cudaStream_t st) {
    const auto launch = [&](auto kernel) {
        return launch_behind(kernel, dim3(sets), dim3(32 * W), 0, st, a.nodes, a.kids, a.node_total, a.pos, a.n, a.eps2,
                             a.theta2, a.dt, a.pos_out, a.vel, a.acc, a.force_out, a.ids, a.counters, a.euler, a.work,
                             a.params, a.P, a.host, a.first, a.beside, a.ready);
    };
    if constexpr (!SEG)
        if (a.host.pos) return launch(team_walk_kernel<W, COUNT, SEG, GUARD, true>);
    return launch(team_walk_kernel<W, COUNT, SEG, GUARD, false>);
}

template <int W>
cudaError_t launch_team(const TeamWalk &a, bool guard, unsigned sets, cudaStream_t st) {
    const bool seg = a.work != nullptr;
    if (a.counters) return seg ? launch_form<W, true, true, true>(a, sets, st) : launch_form<W, true, false, true>(a, sets, st);
    if (seg) return guard ? launch_form<W, false, true, true>(a, sets, st) : launch_form<W, false, true, false>(a, sets, st);
    return guard ? launch_form<W, false, false, true>(a, sets, st) : launch_form<W, false, false, false>(a, sets, st);
}

}  // namespace

// Walk of one Plummer system (GB300, us) with teams of 1 / 2 / 4 / 8 / 16 warps:
//     4,096 bodies   369 /  218 /  117 /   74 /   53
//    10,000          503 /  289 /  156 /   94 /   68
//    30,001          722 /  380 /  216 /  152 /  186
//    65,536          796 /  447 /  297 /  282 /  375
//   262,144         1131 / 1066 /  964 /  971 / 1481
//   524,288         1857 / 1873 / 1820 / 1889 / 2983
//       2^20        3238 / 3533 / 3530 / 3732 / 6014
// The size of a team follows from the system's size alone, so that it sums in
// the same order in an ensemble, where fewer barriers count for more (128
// ragged systems of up to 131,072 bodies: 1 warp 9.5, 4 warps 9.9, 8 warps
// 10.6, 16 warps 12.4 ms per walk; 200 systems of 20,000: 1 warp 10.3, 8 warps
// 11.7, 60 of 65,536: 1 warp 11.2, 4 warps 11.7): 4 from 32,768 on although 8 is
// level with it for one system up to 2^17, and 16 only below the sizes at which
// ensembles turn to Barnes-Hut.
// What that costs an ensemble that fills the chip: steps of 2,048 ragged systems of
// 256 to 131,072 bodies 140.0 ms by this rule, 138.1 by teams of 4 throughout, 130.8
// by one warp per set; what it buys a lone system stands in the table (one warp per
// set takes 5 to 7 times as long up to 30,001 bodies).
constexpr int64_t kMaxTeams = 458752;  // with the tails below: 393,216 bodies 1.357 by fours, 1.381 ms by one warp
int bh_team_size(int64_t n) {
    if (const char *e = std::getenv("NBODY_BH_TEAM")) {  // 1, 2, 4, 8 or 16: that team for every size
        const int v = std::atoi(e);
        if (v == 1 || v == 2 || v == 4 || v == 8 || v == 16) return v;
    }
    return n < 10240 ? 16 : n < (1 << 15) ? 8 : n <= kMaxTeams ? 4 : 1;
}

// The last sets of a large system go to a launch of their own, by teams of 8,
// that starts when the last CTAs of the others have: a set walked by one warp
// takes 1.4 ms of a 3.2 ms walk of 2^20 bodies, so the SMs ran empty for a good
// part of it. Walk of one Plummer system (GB300, ms), all sets alike / with the
// tail: 131,073 bodies .527 / .498, 262,144 .961 / .922, 393,216 1.385 / 1.357,
// 524,288 1.865 (4 warps: 1.808) / 1.686, 2^20 3.240 / 3.064, 2^21 6.115 / 5.970,
// 2^22 12.19 / 12.01; a ball of 2^20 1.491 / 1.454. Behind teams of 4, 600 or 800
// sets are level with 400; behind single warps 2,100 or 2,700 with 2,432 (16 per
// SM). Tails by teams of 4 gain nothing, by teams of 16 half as much. Not up to
// 2^17 bodies: the systems of an ensemble fill each other's ends, and teams of 8
// cost 7 % more than teams of 4 there; which set is walked how follows from n
// alone, so that a system sums in the same order in an ensemble.
constexpr int64_t kTailMinBodies = 1 << 17;
constexpr int64_t kTailSetsTeams = 400, kTailSetsOne = 2432;
int64_t bh_main_sets(int64_t n) {
    const int64_t sets = (n + 63) / 64;
    if (n <= kTailMinBodies || std::getenv("NBODY_BH_TEAM")) return sets;
    return (sets - (n <= kMaxTeams ? kTailSetsTeams : kTailSetsOne)) & ~int64_t(7);  // whole CTAs of cell_walk_kernel
}

cudaError_t bh_team_walk(const TeamWalk &a, int team, bool guard, int64_t sets, cudaStream_t st) {
    if (sets <= 0) return cudaSuccess;
    const unsigned g = static_cast<unsigned>(sets);
    switch (team) {
        case 2: return launch_team<2>(a, guard, g, st);
        case 4: return launch_team<4>(a, guard, g, st);
        case 8: return launch_team<8>(a, guard, g, st);
        case 16: return launch_team<16>(a, guard, g, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace nbody
