// Direct sum with every pair of bodies evaluated once.
//
// pp.cu evaluates every ordered pair: 12 packed FP32 operations (and two
// MUFU.RSQ) for two interactions. The separation, its square and the inverse
// cube are the same for (i, j) and (j, i), so evaluating the pair once and
// adding it to both bodies takes 16 packed operations (and two MUFU.RSQ) for
// four interactions: the FP32 pipe, which bounds the direct sum, gets 1.5
// times the interactions per instruction. At 20 operations per interaction, on
// GB300 (nominal FP32 peak 80.5 TFLOP/s): 16,384 bodies 105 -> 88 us, 61
// TFLOP/s; 131,071 bodies 6.01 -> 4.63 ms, 74 TFLOP/s. The FP32 pipe is some 74%
// busy; pp.cu reaches 85% of its own bound. Without the shuffles (a timing
// probe) 6% more would be had; the accumulations with three different operands
// cost more than their two cycles; a step needs the sixteen-fold unrolling (4:
// 66, 8: 73 TFLOP/s at 131,071) to overlap its chains.
//
// Shape. Bodies are cut into NB blocks of 1,024. A CTA of 256 threads holds one
// block, four bodies per thread, in registers, and takes j-bodies in tiles of
// 64 (TMA bulk copies into a ring, re-laid as 32 j-pairs). Block I meets itself
// (ordered pairs, as pp.cu, 16 tiles) and the blocks I + 1 .. I + NB / 2
// (cyclic), so that each pair of blocks meets once. On those tiles a warp's
// lane l takes j-pair l + s in step s (mod 32): its four bodies' sums stay in
// registers, and the pair's sums move from lane to lane with the steps, six
// shuffles for 64 packed operations, and are back at lane l's own pair after 32
// steps. The eight warps' sums of a tile are added in warp order in shared
// memory and go to a row of the block (j-row: 12 bytes per body and block).
// Measured against it at 131,071 bodies: eight bodies per thread and one CTA
// per SM 75 TFLOP/s (but 55 against 61 at 16,384, whose ranges are then too
// coarse), 512 threads 74, 384 threads 71, two bodies per thread 47.
//
// The tiles of all blocks are spread over two CTAs per SM, by weight (a tile
// of the own block costs 3/4 of another). A second kernel adds for each body
// the parts of the CTAs that held it (in the order of their ranges) and the
// j-rows that met it (in order of distance), and integrates: the same bits on
// every run.
//
// The inverse cube is formed before the mass is multiplied in. Where it could
// leave the range of FP32 although the product does not (coordinates beyond
// 2^40, softening below 2^-80 or beyond 2^83), one more operation per pair keeps
// pp.cu's order (m * inv) * inv^2.
#include <algorithm>

#include "common.cuh"
#include "kernels.h"
#include "launch.h"
#include "pp_common.cuh"

namespace nbody {

namespace {

constexpr int kSymT = 256;
constexpr int kSymK = 4;
constexpr int kSymPerSm = 2;  // CTAs (128 registers)
constexpr int kSymB = kSymT * kSymK;      // bodies per block
constexpr int kSymTile = 64;              // j-bodies per tile
constexpr int kSymTiles = kSymB / kSymTile;  // tiles per block
constexpr int kSymStages = 4;
constexpr int kSymWarps = kSymT / 32;
constexpr float kSymFar = 1099511627776.f;  // 2^40
constexpr int kSymMaxBlocks = 256;          // 2^18 bodies: 0.4 GB of j-rows
constexpr int kOwn = 3, kOther = 4;         // weight of a tile of the own block, and of another

// Block b meets p.window blocks in front of it (cyclic), and one more if it is
// among the first p.heavy: NB / 2 for each block when NB is odd; when it is
// even the pairs NB / 2 apart belong to their first block. sym_met: how many
// meet it from behind.
__host__ __device__ __forceinline__ int sym_met(const SymPlan &p, int b) {
    return p.window + (p.heavy > 0 && b >= p.heavy ? 1 : 0);
}
// Tiles, and weight, of blocks 0 .. b - 1.
__host__ __device__ __forceinline__ int sym_first(const SymPlan &p, int b) {
    return kSymTiles * (b * (1 + p.window) + (b < p.heavy ? b : p.heavy));
}
__host__ __device__ __forceinline__ int sym_light(const SymPlan &p) {
    return kOwn * kSymTiles + kOther * kSymTiles * p.window;  // weight of a block that is not heavy
}
__host__ __device__ __forceinline__ int sym_weight(const SymPlan &p, int b) {
    return sym_light(p) * b + kOther * kSymTiles * (b < p.heavy ? b : p.heavy);
}
// The block of tile x (of all blocks, one after the other).
__host__ __device__ __forceinline__ int sym_block(const SymPlan &p, int x) {
    const int q = x / kSymTiles, wide = p.heavy * (2 + p.window);
    return q < wide ? q / (2 + p.window) : p.heavy + (q - wide) / (1 + p.window);
}
// The first tile, counted within a block, at or after weight w of the block.
__host__ __device__ __forceinline__ int sym_tile_at(int w) {
    return w <= kOwn * kSymTiles ? (w + kOwn - 1) / kOwn : kSymTiles + (w - kOwn * kSymTiles + kOther - 1) / kOther;
}
struct SymSmem {
    alignas(128) float4 ring[kSymStages][kSymTile];
    // Two tiles as j-pairs {x0 x1 y0 y1} and {z0 z1 m0 m1}, each pair twice (at
    // q and q + 32), so that lane l reads pair l + s without wrapping.
    alignas(16) float4 xy[2][kSymTile], zm[2][kSymTile];
    alignas(16) float sums[2][kSymWarps][3][kSymTile];
    alignas(8) uint64_t full[kSymStages];
    int far[2];  // a tile with a coordinate beyond kSymFar
};

// One pass of the 32 steps of a tile: WIDE keeps the mass inside the cube.
template <bool GUARD, bool WIDE>
__device__ __forceinline__ void sym_tile(const float4 *__restrict__ xy, const float4 *__restrict__ zm, int next,
                                         const float2 (&nx)[kSymK], const float2 (&ny)[kSymK],
                                         const float2 (&nz)[kSymK], const float2 (&nm)[kSymK], const float2 e2,
                                         float2 (&ax)[kSymK], float2 (&ay)[kSymK], float2 (&az)[kSymK], float2 &bx,
                                         float2 &by, float2 &bz) {
#pragma unroll 16
    for (int s = 0; s < 32; ++s) {
        const float4 u = xy[s], v = zm[s];
        const float2 xj = f2(u.x, u.y), yj = f2(u.z, u.w), zj = f2(v.x, v.y), mj = f2(v.z, v.w);
#pragma unroll
        for (int r = 0; r < kSymK; ++r) {
            const float2 dx = __fadd2_rn(xj, nx[r]);
            const float2 dy = __fadd2_rn(yj, ny[r]);
            const float2 dz = __fadd2_rn(zj, nz[r]);
            const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __ffma2_rn(dx, dx, e2)));
            float2 inv = f2(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y));
            if (GUARD) {
                inv.x = r2.x > 0.f ? inv.x : 0.f;
                inv.y = r2.y > 0.f ? inv.y : 0.f;
            }
            const float2 inv2 = __fmul2_rn(inv, inv);
            float2 sj, si;
            if (WIDE) {
                sj = __fmul2_rn(__fmul2_rn(mj, inv), inv2);
                si = __fmul2_rn(__fmul2_rn(nm[r], inv), inv2);
            } else {
                const float2 inv3 = __fmul2_rn(inv, inv2);
                sj = __fmul2_rn(mj, inv3);
                si = __fmul2_rn(nm[r], inv3);
            }
            ax[r] = __ffma2_rn(dx, sj, ax[r]);
            ay[r] = __ffma2_rn(dy, sj, ay[r]);
            az[r] = __ffma2_rn(dz, sj, az[r]);
            bx = __ffma2_rn(dx, si, bx);
            by = __ffma2_rn(dy, si, by);
            bz = __ffma2_rn(dz, si, bz);
        }
        bx = f2(__shfl_sync(0xffffffffu, bx.x, next), __shfl_sync(0xffffffffu, bx.y, next));
        by = f2(__shfl_sync(0xffffffffu, by.x, next), __shfl_sync(0xffffffffu, by.y, next));
        bz = f2(__shfl_sync(0xffffffffu, bz.x, next), __shfl_sync(0xffffffffu, bz.y, next));
    }
}

template <bool GUARD>
__global__ void __launch_bounds__(kSymT, kSymPerSm)
    pp_sym_kernel(const float4 *__restrict__ pos, int64_t n, float eps2, const __grid_constant__ SymPlan p, float *__restrict__ parts,
                  float *__restrict__ rows, int *status) {
    __shared__ SymSmem S;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int range = blockIdx.x;
    const int x0 = p.begin[range], x1 = p.begin[range + 1];
    const float2 e2 = f2(eps2, eps2);
    wait_for_launches_before();
    // Tile x: block b's own tiles, then those of blocks b + 1, b + 2, ... (cyclic).
    auto tile_first = [&](int x, int b) -> int64_t {
        const int t = x - sym_first(p, b);
        int j = b + t / kSymTiles;
        if (j >= p.blocks) j -= p.blocks;
        return static_cast<int64_t>(j) * kSymB + (t % kSymTiles) * kSymTile;
    };
    auto count_of = [&](int64_t j0) -> int {
        const int64_t left = n - j0;
        return left <= 0 ? 0 : left < kSymTile ? static_cast<int>(left) : kSymTile;
    };
    // Thread 0 fetches tile x; an empty tile (past the last body) completes at once.
    int fetch_block = x0 < x1 ? sym_block(p, x0) : 0;
    auto issue = [&](int x) {
        const int stage = (x - x0) % kSymStages;
        while (x >= sym_first(p, fetch_block + 1)) ++fetch_block;
        const int64_t j0 = tile_first(x, fetch_block);
        const int cnt = count_of(j0);
        fence_proxy_async_smem();
        mbar_arrive_expect_tx(&S.full[stage], static_cast<uint32_t>(cnt) * 16u);
        if (cnt > 0) tma_bulk_g2s(&S.ring[stage][0], pos + j0, static_cast<uint32_t>(cnt) * 16u, &S.full[stage]);
    };
    if (tid == 0) {
        for (int s = 0; s < kSymStages; ++s) mbar_init(&S.full[s], 1);
        mbar_init_fence();
        for (int x = x0; x < x1 && x < x0 + kSymStages; ++x) issue(x);
    }
    float2 nx[kSymK], ny[kSymK], nz[kSymK], nm[kSymK], ax[kSymK], ay[kSymK], az[kSymK];
    int block = -1, seg = 0;
    bool far_i = false;
    // The block's bodies into registers; a place past the last body holds a
    // massless one out of the way.
    auto load_block = [&](int b) {
        bool far = false;
#pragma unroll
        for (int r = 0; r < kSymK; ++r) {
            const int64_t i = static_cast<int64_t>(b) * kSymB + tid + r * kSymT;
            const float4 q = i < n ? pos[i] : make_float4(1e18f, 1e18f, 1e18f, 0.f);
            far = far || (i < n && !(fabsf(q.x) <= kSymFar && fabsf(q.y) <= kSymFar && fabsf(q.z) <= kSymFar));
            nx[r] = f2(-q.x, -q.x);
            ny[r] = f2(-q.y, -q.y);
            nz[r] = f2(-q.z, -q.z);
            nm[r] = f2(-q.w, -q.w);
            ax[r] = ay[r] = az[r] = f2(0.f, 0.f);
        }
        far_i = __syncthreads_or(far);  // also publishes the mbarriers
        block = b;
    };
    auto store_part = [&]() {
        float *out = parts + (static_cast<int64_t>(range) * 2 + seg) * (3 * kSymB);
#pragma unroll
        for (int r = 0; r < kSymK; ++r) {
            out[tid + r * kSymT] = ax[r].x + ax[r].y;
            out[kSymB + tid + r * kSymT] = ay[r].x + ay[r].y;
            out[2 * kSymB + tid + r * kSymT] = az[r].x + az[r].y;
        }
    };
    // Waits for tile x and re-lays it (warp x % 8, one pair per lane).
    auto stage_in = [&](int x) -> bool {
        const int t = x - x0;
        const int stage = t % kSymStages;
        if (warp != t % kSymWarps) return true;
        if (!mbar_wait_bounded(&S.full[stage], static_cast<uint32_t>(t / kSymStages) & 1u, status)) return false;
        const int cnt = count_of(tile_first(x, sym_block(p, x)));
        const float4 none = make_float4(1e18f, 1e18f, 1e18f, 0.f);
        const float4 a = 2 * lane < cnt ? S.ring[stage][2 * lane] : none;
        const float4 c = 2 * lane + 1 < cnt ? S.ring[stage][2 * lane + 1] : none;
        const bool far =
            (2 * lane < cnt && !(fabsf(a.x) <= kSymFar && fabsf(a.y) <= kSymFar && fabsf(a.z) <= kSymFar)) ||
            (2 * lane + 1 < cnt && !(fabsf(c.x) <= kSymFar && fabsf(c.y) <= kSymFar && fabsf(c.z) <= kSymFar));
        const float4 xy = make_float4(a.x, c.x, a.y, c.y), zm = make_float4(a.z, c.z, a.w, c.w);
        S.xy[t & 1][lane] = xy;
        S.xy[t & 1][lane + 32] = xy;
        S.zm[t & 1][lane] = zm;
        S.zm[t & 1][lane + 32] = zm;
        const unsigned any = __ballot_sync(0xffffffffu, far);
        if (lane == 0) S.far[t & 1] = any != 0u;
        return true;
    };
    bool failed = false;
    int fail_at = x0;
    if (x0 < x1) {
        load_block(sym_block(p, x0));
        if (!__syncthreads_and(stage_in(x0))) {
            failed = true;
        } else if (tid == 0 && x0 + kSymStages < x1) {
            issue(x0 + kSymStages);
        }
    }
    const int next = (lane + 1) & 31;
    for (int x = x0; x < x1 && !failed; ++x) {
        const int buf = (x - x0) & 1;
        if (x >= sym_first(p, block + 1)) {  // at most one change of block per CTA
            if (seg > 0) {
                record_error(status, NBODY_ERR_CAPACITY);
                failed = true;
                fail_at = x + 1;
                break;
            }
            store_part();
            ++seg;
            load_block(block + 1);
        }
        const bool ok = x + 1 < x1 ? stage_in(x + 1) : true;
        const int t = x - sym_first(p, block);
        if (t < kSymTiles) {  // the block itself: ordered pairs
            const float4 *xy = S.xy[buf], *zm = S.zm[buf];
#pragma unroll 2
            for (int q = 0; q < kSymTile / 2; ++q) {
                const float4 u = xy[q], v = zm[q];
                const float2 xj = f2(u.x, u.y), yj = f2(u.z, u.w), zj = f2(v.x, v.y), mj = f2(v.z, v.w);
#pragma unroll
                for (int r = 0; r < kSymK; ++r) {
                    const float2 dx = __fadd2_rn(xj, nx[r]);
                    const float2 dy = __fadd2_rn(yj, ny[r]);
                    const float2 dz = __fadd2_rn(zj, nz[r]);
                    const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __ffma2_rn(dx, dx, e2)));
                    float2 inv = f2(rsqrt_ftz(r2.x), rsqrt_ftz(r2.y));
                    if (GUARD) {
                        inv.x = r2.x > 0.f ? inv.x : 0.f;
                        inv.y = r2.y > 0.f ? inv.y : 0.f;
                    }
                    const float2 s = __fmul2_rn(__fmul2_rn(mj, inv), __fmul2_rn(inv, inv));
                    ax[r] = __ffma2_rn(dx, s, ax[r]);
                    ay[r] = __ffma2_rn(dy, s, ay[r]);
                    az[r] = __ffma2_rn(dz, s, az[r]);
                }
            }
        } else {
            float2 bx = f2(0.f, 0.f), by = bx, bz = bx;
            if (GUARD || far_i || S.far[buf])
                sym_tile<GUARD, true>(S.xy[buf] + lane, S.zm[buf] + lane, next, nx, ny, nz, nm, e2, ax, ay, az, bx, by, bz);
            else
                sym_tile<GUARD, false>(S.xy[buf] + lane, S.zm[buf] + lane, next, nx, ny, nz, nm, e2, ax, ay, az, bx, by, bz);
            *reinterpret_cast<float2 *>(&S.sums[buf][warp][0][2 * lane]) = bx;
            *reinterpret_cast<float2 *>(&S.sums[buf][warp][1][2 * lane]) = by;
            *reinterpret_cast<float2 *>(&S.sums[buf][warp][2][2 * lane]) = bz;
        }
        if (!__syncthreads_and(ok)) {  // also: everyone is done with this tile's pairs, its sums are written
            failed = true;
            fail_at = x + 1;
            break;
        }
        if (tid == 0 && x + 1 + kSymStages < x1) issue(x + 1 + kSymStages);
        if (t >= kSymTiles && tid < 3 * kSymTile) {
            const float *q = &S.sums[buf][0][0][0] + tid;
            float sum = q[0];
#pragma unroll
            for (int w = 1; w < kSymWarps; ++w) sum += q[w * 3 * kSymTile];
            rows[(static_cast<int64_t>(block) * p.row_tiles + (t - kSymTiles)) * (3 * kSymTile) + tid] = sum;
        }
    }
    if (failed) {
        // Drain this CTA's copies still in flight before shared memory goes away.
        if (tid == 0) {
            parts[-1] = 1.f;
            for (int u = fail_at; u < x1 && u < fail_at + kSymStages; ++u)
                mbar_wait_bounded(&S.full[(u - x0) % kSymStages], static_cast<uint32_t>((u - x0) / kSymStages) & 1u,
                                  status);
        }
        __syncthreads();
        return;
    }
    if (x0 < x1) store_part();
}

// The sum of each body, one thread per body: the parts of the ranges that held
// its block, in order, then the j-rows that met it, in order of distance; then
// the integrator. A kernel of its own, over the whole chip: the last CTA of
// each block doing it in pp_sym_kernel took 15 us at 16,384 bodies. Where a CTA
// gave up (parts[-1]), its parts and rows are those of an earlier call, and
// nothing is written until the status has been reported and the word cleared.
__global__ void __launch_bounds__(kSymT) pp_sym_sum_kernel(const float4 *__restrict__ pos, int64_t n,
                                                           const __grid_constant__ SymPlan p,
                                                           const float *__restrict__ parts,
                                                           const float *__restrict__ rows,
                                                           Integrate g) {
    constexpr int kBatch = 16;
    wait_for_launches_before();
    const int to = blockIdx.x / (kSymB / kSymT), i0 = (blockIdx.x % (kSymB / kSymT)) * kSymT + threadIdx.x;
    const int64_t i = static_cast<int64_t>(to) * kSymB + i0;
    // One thread's load for the block: every warp's took 0.3 us of a step.
    const bool gave_up = threadIdx.x == 0 && parts[-1] != 0.f;
    const int first = sym_first(p, to), past = sym_first(p, to + 1);
    int lo = 0, hi = p.ctas;  // the range of the block's first tile: begin[lo] <= first < begin[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) / 2;
        if (p.begin[mid] <= first) lo = mid; else hi = mid;
    }
    float fx = 0.f, fy = 0.f, fz = 0.f;
    for (int c0 = lo; c0 < p.ctas && p.begin[c0] < past; c0 += kBatch) {
        float vx[kBatch], vy[kBatch], vz[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int c = c0 + u;
            vx[u] = vy[u] = vz[u] = 0.f;
            if (c >= p.ctas || p.begin[c] >= past || p.begin[c] >= p.begin[c + 1]) continue;
            // Its second part where it began in the block before.
            const float *in = parts + (static_cast<int64_t>(c) * 2 + (p.begin[c] < first ? 1 : 0)) * (3 * kSymB) + i0;
            vx[u] = in[0];
            vy[u] = in[kSymB];
            vz[u] = in[2 * kSymB];
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            fx += vx[u];
            fy += vy[u];
            fz += vz[u];
        }
    }
    const int met = sym_met(p, to);
    for (int k0 = 1; k0 <= met; k0 += kBatch) {
        float vx[kBatch], vy[kBatch], vz[kBatch];
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            const int k = k0 + u;
            vx[u] = vy[u] = vz[u] = 0.f;
            if (k > met) continue;
            const int from = to >= k ? to - k : to - k + p.blocks;
            const float *in = rows + (static_cast<int64_t>(from) * p.row_tiles + (k - 1) * kSymTiles + i0 / kSymTile) *
                                         (3 * kSymTile) + i0 % kSymTile;
            vx[u] = in[0];
            vy[u] = in[kSymTile];
            vz[u] = in[2 * kSymTile];
        }
#pragma unroll
        for (int u = 0; u < kBatch; ++u) {
            fx += vx[u];
            fy += vy[u];
            fz += vz[u];
        }
    }
    if (__syncthreads_or(gave_up) || i >= n) return;
    if (g.pos_out) integrate_body(i, pos[i], fx, fy, fz, g);
    else if (g.force) g.force[i] = make_float4(fx, fy, fz, 0.f);
}

}  // namespace

SymPlan pp_sym_plan(int64_t n, int sms) {
    SymPlan p;
    const int64_t blocks = (n + kSymB - 1) / kSymB;
    if (blocks > kSymMaxBlocks) return p;
    p.blocks = static_cast<int>(blocks);
    p.window = (p.blocks - 1) / 2;
    p.heavy = p.blocks % 2 == 0 ? p.blocks / 2 : 0;
    p.row_tiles = kSymTiles * (p.blocks / 2);
    // Two CTAs per SM, or as many waves of them as leave a range less than 3/4 of
    // a block's tiles, so that it meets a change of block once at most.
    p.ctas = kSymPerSm * sms;
    while (4 * p.blocks > 3 * p.ctas) p.ctas += kSymPerSm * sms;
    if (p.ctas > kSymMaxCtas) {
        p.blocks = 0;
        return p;
    }
    // Where every block can have whole ranges of its own, and the longest is no
    // longer than an even cut's (to which changes of block add), it gets them;
    // else one even cut over all blocks.
    const int total = sym_weight(p, p.blocks);
    auto weight_of = [&](int b) { return sym_weight(p, b + 1) - sym_weight(p, b); };
    int of[kSymMaxBlocks];
    int given = 0, longest = 0;
    for (int b = 0; b < p.blocks; ++b)
        given += of[b] = static_cast<int>(static_cast<int64_t>(weight_of(b)) * p.ctas / total);
    for (int b = 0; b < p.blocks && given < p.ctas; ++b, ++given) ++of[b];
    for (int b = 0; b < p.blocks; ++b)
        longest = std::max(longest, of[b] > 0 ? (weight_of(b) + kOther * of[b] - 1) / (kOther * of[b]) : total);
    const bool whole = longest <= (total + kOther * p.ctas - 1) / (kOther * p.ctas);
    int r = 0, b = 0;
    if (whole) {
        for (b = 0; b < p.blocks; ++b)
            for (int k = 0; k < of[b]; ++k) p.begin[r++] = sym_first(p, b) + sym_tile_at(weight_of(b) * k / of[b]);
    } else {
        for (int k = 0; k < p.ctas; ++k) {
            const int w = static_cast<int>(static_cast<int64_t>(total) * k / p.ctas);
            while (sym_weight(p, b + 1) <= w) ++b;
            p.begin[r++] = sym_first(p, b) + sym_tile_at(w - sym_weight(p, b));
        }
    }
    p.begin[r] = sym_first(p, p.blocks);
    p.parts_bytes = static_cast<size_t>(p.ctas) * 2 * 3 * kSymB * sizeof(float);
    p.bytes = p.parts_bytes +
              static_cast<size_t>(p.blocks) * static_cast<size_t>(p.row_tiles) * 3 * kSymTile * sizeof(float);
    return p;
}

int pp_sym_bodies_per_thread() { return kSymK; }

cudaError_t pp_sym_launch(const SymPlan &p, const float4 *pos, int64_t n, float eps2, const Integrate &g, void *scratch,
                          cudaStream_t stream, int *status) {
    float *parts = static_cast<float *>(scratch);
    float *rows = reinterpret_cast<float *>(static_cast<char *>(scratch) + p.parts_bytes);
    constexpr float lo = 8.2718061255302767e-25f /* 2^-80 */, hi = 9.6714065569170334e24f /* 2^83 */;
    if (eps2 >= lo && eps2 <= hi)
        launch_behind(pp_sym_kernel<false>, dim3(p.ctas), dim3(kSymT), 0, stream, pos, n, eps2, p, parts, rows,
                      status);
    else
        launch_behind(pp_sym_kernel<true>, dim3(p.ctas), dim3(kSymT), 0, stream, pos, n, eps2, p, parts, rows,
                      status);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    return launch_behind(pp_sym_sum_kernel, dim3(static_cast<unsigned>((n + kSymT - 1) / kSymT)), dim3(kSymT), 0, stream, pos,
                         n, p, parts, rows, g);
}

}  // namespace nbody
