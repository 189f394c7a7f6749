// Stable merge sort of (64-bit key, 32-bit value) pairs, for arrays that do not
// fill the GPU.
//
// sort.cu's radix sort takes ten launches whatever the size, each a chain of
// some 10 us in every CTA (tile number, loads, sixteen rounds of ranking,
// block scan, look-back, scatter): 105 us for 4,096 pairs and 121 us for
// 65,536. Here a CTA sorts a tile in shared memory in one launch (four or
// eight pairs per thread in registers, then merge rounds over twice as many
// threads each), and each further launch merges neighbouring runs: four or eight
// at a time by searching every pair's place (rank_merge_kernel) up to 2^18 pairs,
// two at a time above, every CTA producing 2,048 pairs from the part of two runs
// that a search along the merge path gives it (merge_pass_kernel). Taking the
// left run first where keys are equal keeps the sort stable, so the permutation
// is the radix sort's. (Merge path: Green, McColl, Bader, "GPU Merge Path", ICS 2012.) GB300, us, radix / merge: 4,096 pairs 105 / 17, 30,001
// 120 / 22, 65,536 121 / 26, 262,144 137 / 53, 2^20 212 / 121, 2^22 553 / 452.
// A tile of 2,048 pairs takes 10 us, a pass by searching 5 us up to 2^17 pairs, a
// merge pass 7 us while its launch and the chain of its searches bound it and
// 12 us of traffic at 2^20.
#include <cuda_runtime.h>

#include "common.cuh"
#include "launch.h"
#include "sort.h"

namespace nbody {

namespace {

constexpr int kMergeThreads = 256;
constexpr int kMergeItems = 8;
constexpr int kMergeOut = kMergeThreads * kMergeItems;  // pairs per CTA of a merge pass

constexpr int kRankThreads = 128;
constexpr int kRankSearches = 4;

// Places in shared memory: one left free in every 16, so that threads whose
// items lie side by side do not meet in the banks.
__device__ __forceinline__ int pad(int i) { return i + (i >> 4); }
constexpr int padded(int n) { return n + n / 16; }

// The number of A's items among the first `diag` of the merge of A and B
// (each sorted, in shared memory from a0 and b0 on); A's come first among equals.
__device__ __forceinline__ int merge_path(const uint64_t *__restrict__ k, int a0, int la, int b0, int lb, int diag) {
    int lo = diag > lb ? diag - lb : 0, hi = diag < la ? diag : la;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (k[pad(a0 + mid)] <= k[pad(b0 + diag - 1 - mid)]) lo = mid + 1; else hi = mid;
    }
    return lo;
}

// Items [diag, diag + N) of the merge of A and B into registers.
template <int N>
__device__ __forceinline__ void merge_items(const uint64_t *__restrict__ k, const uint32_t *__restrict__ v, int a,
                                            int a_end, int b, int b_end, uint64_t (&ko)[N], uint32_t (&vo)[N]) {
    uint64_t ka = a < a_end ? k[pad(a)] : ~0ull, kb = b < b_end ? k[pad(b)] : ~0ull;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const bool left = b >= b_end || (a < a_end && ka <= kb);
        const int at = left ? a : b;
        ko[i] = left ? ka : kb;
        vo[i] = v[pad(at)];
        if (left) {
            ++a;
            ka = a < a_end ? k[pad(a)] : ~0ull;
        } else {
            ++b;
            kb = b < b_end ? k[pad(b)] : ~0ull;
        }
    }
}

// One tile of T * N pairs, sorted. The pairs past the end of the
// array are filled up with the greatest key; they come last, behind any pair
// of the array with that key.
template <int T, int N>
__global__ void __launch_bounds__(T) block_sort_kernel(const uint64_t *keys_in, const uint32_t *vals_in,
                                                                   uint64_t *keys_out, uint32_t *vals_out, int64_t n) {
    constexpr int kTile = T * N;
    extern __shared__ __align__(16) unsigned char smem[];
    uint64_t *k = reinterpret_cast<uint64_t *>(smem);
    uint32_t *v = reinterpret_cast<uint32_t *>(k + padded(kTile));
    const int tid = threadIdx.x;
    wait_for_launches_before();
    const int64_t base = static_cast<int64_t>(blockIdx.x) * kTile;
    const int count = n - base < kTile ? static_cast<int>(n - base) : kTile;
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const int at = i * T + tid;
        k[pad(at)] = at < count ? keys_in[base + at] : ~0ull;
        v[pad(at)] = at < count ? vals_in[base + at] : 0u;
    }
    __syncthreads();
    uint64_t ki[N];
    uint32_t vi[N];
#pragma unroll
    for (int i = 0; i < N; ++i) {
        ki[i] = k[pad(tid * N + i)];
        vi[i] = v[pad(tid * N + i)];
    }
    // Neighbours in turn, only a greater one moving: stable.
#pragma unroll
    for (int round = 0; round < N; ++round) {
#pragma unroll
        for (int i = round & 1; i + 1 < N; i += 2) {
            const bool swap = ki[i] > ki[i + 1];
            const uint64_t tk = swap ? ki[i] : ki[i + 1];
            const uint32_t tv = swap ? vi[i] : vi[i + 1];
            ki[i] = swap ? ki[i + 1] : ki[i];
            vi[i] = swap ? vi[i + 1] : vi[i];
            ki[i + 1] = tk;
            vi[i + 1] = tv;
        }
    }
    // Runs of `width` threads' items merge in pairs, until one holds all pairs.
    for (int width = 1; width * N < count; width *= 2) {
        __syncthreads();  // the round before has been read
#pragma unroll
        for (int i = 0; i < N; ++i) {
            k[pad(tid * N + i)] = ki[i];
            v[pad(tid * N + i)] = vi[i];
        }
        __syncthreads();
        const int first = (tid & ~(2 * width - 1)) * N, len = width * N;
        const int diag = (tid & (2 * width - 1)) * N;
        const int a = merge_path(k, first, len, first + len, len, diag);
        merge_items<N>(k, v, first + a, first + len, first + len + diag - a, first + 2 * len, ki, vi);
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < N; ++i) {
        k[pad(tid * N + i)] = ki[i];
        v[pad(tid * N + i)] = vi[i];
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < N; ++i) {
        const int at = i * T + tid;
        if (at < count) {
            keys_out[base + at] = k[pad(at)];
            vals_out[base + at] = v[pad(at)];
        }
    }
}

// As merge_path on two runs in global memory, by a warp: 32 places at a time.
__device__ __forceinline__ int64_t merge_path_warp(const uint64_t *__restrict__ a, int64_t la,
                                                   const uint64_t *__restrict__ b, int64_t lb, int64_t diag, int lane) {
    int64_t lo = diag > lb ? diag - lb : 0, hi = diag < la ? diag : la;  // the answer is in [lo, hi]
    while (lo < hi) {
        const int64_t len = hi - lo;
        const int64_t step = (len + 31) / 32;
        const int64_t mid = lo + step * lane;  // A[mid] before B[diag - 1 - mid]?
        const bool before = mid < hi && a[mid] <= b[diag - 1 - mid];
        const int taken = __popc(__ballot_sync(0xffffffffu, before));  // a prefix of the lanes
        if (taken == 0) {
            hi = lo;
        } else {
            const int64_t last = lo + step * (taken - 1);  // before, and the next place, if any, is not
            hi = last + step < hi ? last + step : hi;
            lo = last + 1;
        }
    }
    return lo;
}

// Runs of `run` pairs (the last one shorter) merge in pairs into runs of 2 * run.
__global__ void __launch_bounds__(kMergeThreads) merge_pass_kernel(const uint64_t *__restrict__ keys_in,
                                                                   const uint32_t *__restrict__ vals_in,
                                                                   uint64_t *__restrict__ keys_out,
                                                                   uint32_t *__restrict__ vals_out, int64_t n,
                                                                   int64_t run) {
    __shared__ uint64_t k[padded(kMergeOut)];
    __shared__ uint32_t v[padded(kMergeOut)];
    __shared__ int64_t split[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    wait_for_launches_before();
    const int64_t o0 = static_cast<int64_t>(blockIdx.x) * kMergeOut;  // 2 * run is a multiple of kMergeOut
    const int64_t pair = o0 / (2 * run) * (2 * run);
    const int64_t la = n - pair < run ? n - pair : run;
    const int64_t lb = n - pair - la < run ? n - pair - la : run;
    const uint64_t *a = keys_in + pair, *b = a + la;
    const int64_t d0 = o0 - pair, d1 = d0 + kMergeOut < la + lb ? d0 + kMergeOut : la + lb;
    if (warp < 2) {
        const int64_t s = merge_path_warp(a, la, b, lb, warp == 0 ? d0 : d1, lane);
        if (lane == 0) split[warp] = s;
    }
    __syncthreads();
    const int64_t a0 = split[0], b0 = d0 - a0;
    const int na = static_cast<int>(split[1] - a0), total = static_cast<int>(d1 - d0), nb = total - na;
#pragma unroll
    for (int i = 0; i < kMergeItems; ++i) {
        const int at = i * kMergeThreads + tid;
        if (at < total) {
            const int64_t from = at < na ? pair + a0 + at : pair + la + b0 + (at - na);
            k[pad(at)] = keys_in[from];
            v[pad(at)] = vals_in[from];
        }
    }
    __syncthreads();
    const int diag = tid * kMergeItems < total ? tid * kMergeItems : total;
    const int ia = merge_path(k, 0, na, na, nb, diag);
    uint64_t ko[kMergeItems];
    uint32_t vo[kMergeItems];
    if (diag + kMergeItems <= total) {
        merge_items<kMergeItems>(k, v, ia, na, na + diag - ia, total, ko, vo);
        // Eight pairs side by side: whole 16-byte stores (o0 and diag are multiples of eight).
        ulonglong2 *kd = reinterpret_cast<ulonglong2 *>(keys_out + o0 + diag);
        uint4 *vd = reinterpret_cast<uint4 *>(vals_out + o0 + diag);
#pragma unroll
        for (int i = 0; i < kMergeItems / 2; ++i) kd[i] = make_ulonglong2(ko[2 * i], ko[2 * i + 1]);
#pragma unroll
        for (int i = 0; i < kMergeItems / 4; ++i) vd[i] = make_uint4(vo[4 * i], vo[4 * i + 1], vo[4 * i + 2], vo[4 * i + 3]);
    } else if (diag < total) {
        int x = ia, y = na + diag - ia;
        for (int i = diag; i < total; ++i) {
            const bool left = y >= total || (x < na && k[pad(x)] <= k[pad(y)]);
            const int at = left ? x++ : y++;
            keys_out[o0 + i] = k[pad(at)];
            vals_out[o0 + i] = v[pad(at)];
        }
    }
}

// Groups of `ways` runs (four or eight) of 2^run_bits pairs, the last ones
// shorter or missing, into one run each: a pair's place is its own place in its
// run plus what a binary search finds before it in each other run of its group
// (its equals in earlier runs included, those in later ones not: stable).
// A step of a search waits for a load, so four searches go side by side. The
// group's size is left to run time: with four or eight as a constant the same
// loop took 30 instead of 22 us for 30,001 pairs (sort of all tiles included).
__global__ void __launch_bounds__(kRankThreads) rank_merge_kernel(const uint64_t *__restrict__ keys_in,
                                                                  const uint32_t *__restrict__ vals_in,
                                                                  uint64_t *__restrict__ keys_out,
                                                                  uint32_t *__restrict__ vals_out, int n, int run_bits,
                                                                  int ways) {
    wait_for_launches_before();
    const int i = blockIdx.x * kRankThreads + threadIdx.x;
    if (i >= n) return;
    const int run = 1 << run_bits, mine = i >> run_bits, first = mine & ~(ways - 1);
    const uint64_t x = keys_in[i];
    const uint32_t v = vals_in[i];
    int to = i - (mine - first) * run;
    for (int s0 = 0; s0 < ways; s0 += kRankSearches) {
        int at[kRankSearches], end[kRankSearches];
        uint64_t bound[kRankSearches];  // the keys below it come first
#pragma unroll
        for (int j = 0; j < kRankSearches; ++j) {
            const int s = first + s0 + j;
            const bool other = s != mine && s * run < n;
            at[j] = other ? s * run : 0;
            end[j] = other ? (n - at[j] < run ? n : at[j] + run) : 0;
            to -= at[j];
            bound[j] = x;
            if (s < mine) {
                if (x == ~0ull) at[j] = end[j]; else bound[j] = x + 1;
            }
        }
        for (int step = run; step > 0; step >>= 1) {
            uint64_t k[kRankSearches];
#pragma unroll
            for (int j = 0; j < kRankSearches; ++j) k[j] = keys_in[at[j] + step <= end[j] ? at[j] + step - 1 : 0];
#pragma unroll
            for (int j = 0; j < kRankSearches; ++j) at[j] += at[j] + step <= end[j] && k[j] < bound[j] ? step : 0;
        }
#pragma unroll
        for (int j = 0; j < kRankSearches; ++j) to += at[j];
    }
    keys_out[to] = x;
    vals_out[to] = v;
}

template <int T, int N>
constexpr size_t block_smem() {
    return static_cast<size_t>(padded(T * N)) * (sizeof(uint64_t) + sizeof(uint32_t));
}

template <int T, int N>
cudaError_t prepare_block() {
    return cudaFuncSetAttribute(block_sort_kernel<T, N>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                static_cast<int>(block_smem<T, N>()));
}

// Tiles of 2,048 pairs while passes are cheaper than the larger tile's rounds
// (262,144 pairs: 53 us against 60 with 4,096 per tile; 524,288, merging in
// pairs: 86 with 2,048, 80 with 4,096, 90 with 8,192).
constexpr int64_t kSmallTiles = 1 << 18;
int64_t tile_of(int64_t n) { return n <= kSmallTiles ? 2048 : 4096; }

// Runs merged by the next pass over runs of `run` pairs. Up to 2^18 pairs a pass
// is bound by its launch and a chain of loads, not by traffic, and places found
// by searching merge four or eight runs in about the time of one pass of two:
// whole sorts of 8,192 / 30,001 / 65,536 / 131,072 / 262,144 pairs take 16.6 /
// 21.7 / 25.5 / 30.1 / 53.4 us against 23.6 / 37.9 / 45.0 / 52.8 / 61.0 in
// pairs; above, the searches' loads cost more (524,288: 97 against 77 us).
// Eight at once only for the last pass (16,384: 18.7 against 22.4 us by fours).
int merge_ways(int64_t n, int64_t run) {
    if (n > kSmallTiles) return 2;
    return n > 4 * run && n <= 8 * run ? 8 : 4;
}

}  // namespace

cudaError_t merge_sort_prepare() {
    const cudaError_t e = prepare_block<512, 4>();
    return e == cudaSuccess ? prepare_block<512, 8>() : e;
}

// The passes of two runs store 16 bytes at a time, into either pair of arrays;
// the others move single keys and values.
bool merge_sort_takes(const uint64_t *keys, const uint32_t *vals, const uint64_t *keys_alt, const uint32_t *vals_alt,
                      int64_t n) {
    if (merge_ways(n, tile_of(n)) != 2) return true;
    const uintptr_t all = reinterpret_cast<uintptr_t>(keys) | reinterpret_cast<uintptr_t>(vals) |
                          reinterpret_cast<uintptr_t>(keys_alt) | reinterpret_cast<uintptr_t>(vals_alt);
    return (all & 15u) == 0;
}

cudaError_t merge_sort_pairs(uint64_t *keys, uint32_t *vals, uint64_t *keys_alt, uint32_t *vals_alt, int64_t n,
                             cudaStream_t stream) {
    const int64_t tile = tile_of(n);
    const int passes = merge_sort_launches(n) - 1;
    // A tile may be sorted in place; the last pass ends in keys.
    uint64_t *ki = passes % 2 ? keys_alt : keys, *ko = passes % 2 ? keys : keys_alt;
    uint32_t *vi = passes % 2 ? vals_alt : vals, *vo = passes % 2 ? vals : vals_alt;
    const unsigned blocks = static_cast<unsigned>((n + tile - 1) / tile);
    cudaError_t e = tile == 2048 ? launch_behind(block_sort_kernel<512, 4>, dim3(blocks), dim3(512), block_smem<512, 4>(),
                                                 stream, keys, vals, ki, vi, n)
                                 : launch_behind(block_sort_kernel<512, 8>, dim3(blocks), dim3(512), block_smem<512, 8>(),
                                                 stream, keys, vals, ki, vi, n);
    for (int64_t run = tile; run < n && e == cudaSuccess;) {
        const int ways = merge_ways(n, run);
        if (ways == 2) {
            e = launch_behind(merge_pass_kernel, dim3(static_cast<unsigned>((n + kMergeOut - 1) / kMergeOut)),
                              dim3(kMergeThreads), 0, stream, ki, vi, ko, vo, n, run);
        } else {
            int bits = 0;
            while ((int64_t(1) << bits) < run) ++bits;
            e = launch_behind(rank_merge_kernel,
                              dim3(static_cast<unsigned>((n + kRankThreads - 1) / kRankThreads)), dim3(kRankThreads), 0,
                              stream, ki, vi, ko, vo, static_cast<int>(n), bits, ways);
        }
        run *= ways;
        uint64_t *tk = ki; ki = ko; ko = tk;
        uint32_t *tv = vi; vi = vo; vo = tv;
    }
    return e;
}

int merge_sort_launches(int64_t n) {
    int launches = 1;
    for (int64_t run = tile_of(n); run < n; run *= merge_ways(n, run)) ++launches;
    return launches;
}

}  // namespace nbody
