// Host check of the direct sum's scratch (scratch.h) over a device memory that
// refuses what goes beyond a budget; run by test_scratch.py.
#include <cstdio>
#include <map>

#include "scratch.h"

using namespace nbody;

namespace {

struct FakeDevice {
    size_t budget = 0, used = 0;
    std::map<void *, size_t> live;
    int allocs = 0, refusals = 0, clears = 0, waits = 0, frees = 0;
    char *next = reinterpret_cast<char *>(0x100000);
    cudaError_t alloc(void **p, size_t bytes) {
        ++allocs;
        if (used + bytes > budget) {
            ++refusals;
            return cudaErrorMemoryAllocation;
        }
        *p = next;
        next += bytes;
        live[*p] = bytes;
        used += bytes;
        return cudaSuccess;
    }
    cudaError_t clear(void *p, size_t bytes) {
        ++clears;
        return live.count(p) && live[p] >= bytes ? cudaSuccess : cudaErrorInvalidValue;
    }
    cudaError_t wait() {
        ++waits;
        return cudaSuccess;
    }
    void free(void *p) {
        ++frees;
        used -= live.at(p);
        live.erase(p);
    }
    int calls() const { return allocs + clears + waits + frees; }
};

constexpr size_t kMB = 1 << 20;

// n stands for a number of MB that the ordered form needs; the pair-once form ten times as many.
PPPlan fake_plan(int64_t n, bool sym) {
    PPPlan p;
    if (sym) {
        p.sym.blocks = 1;
        p.partial_bytes = 10 * n * kMB;
    } else {
        p.arrivals_bytes = 256;
        p.partial_bytes = 256 + n * kMB;
    }
    return p;
}

struct Context {
    PPScratch s;
    FakeDevice d;
    PPPlan plan;
    cudaError_t call(int64_t n) {
        const auto of = [&](bool sym) { return fake_plan(n, sym); };
        plan = pp_scratch_plan(s, of);
        return pp_scratch_ensure(s, plan, d, of);
    }
};

int line = 0;
#define CHECK(x) do { if (!(x) && !line) line = __LINE__; } while (0)

void plenty() {
    Context c;
    c.d.budget = 1000 * kMB;
    CHECK(c.call(1) == cudaSuccess && c.plan.sym.blocks == 1 && c.s.bytes == 10 * kMB + kArrivalsArea);
    const void *first = c.s.mem;
    const int calls = c.d.calls();
    CHECK(c.call(1) == cudaSuccess && c.s.mem == first && c.d.calls() == calls);
    // Grows: the old one given back after the new one is there, the stream waited for once.
    CHECK(c.call(3) == cudaSuccess && c.s.mem != first && c.d.waits == 1 && c.d.frees == 1);
    CHECK(c.d.used == c.s.bytes && c.d.live.size() == 1);
    CHECK(c.call(2) == cudaSuccess && c.d.frees == 1);
}

void pair_once_refused() {
    Context c;
    c.d.budget = 25 * kMB;
    CHECK(c.call(1) == cudaSuccess && c.plan.sym.blocks == 1);
    const void *first = c.s.mem;
    // 40 MB refused: the ordered form fits what is there; nothing moves, nobody waits.
    CHECK(c.call(4) == cudaSuccess && c.plan.sym.blocks == 0 && c.s.mem == first);
    CHECK(c.d.refusals == 1 && c.d.waits == 0 && c.d.frees == 0);
    int calls = c.d.calls();
    for (int i = 0; i < 3; ++i) CHECK(c.call(4) == cudaSuccess && c.plan.sym.blocks == 0 && c.s.mem == first);
    CHECK(c.d.calls() == calls);
    // Larger ones are not tried again; smaller ones keep the pair-once form.
    CHECK(c.call(7) == cudaSuccess && c.plan.sym.blocks == 0 && c.d.calls() == calls);
    CHECK(c.call(1) == cudaSuccess && c.plan.sym.blocks == 1 && c.d.calls() == calls && c.s.mem == first);
    // An ordered form that outgrows it: one allocation, no second refusal.
    CHECK(c.call(12) == cudaSuccess && c.plan.sym.blocks == 0 && c.s.bytes == 12 * kMB + kArrivalsArea);
    CHECK(c.d.refusals == 1 && c.d.frees == 1 && c.d.used == c.s.bytes);
}

void ordered_refused() {
    Context c;
    c.d.budget = 25 * kMB;
    CHECK(c.call(1) == cudaSuccess);
    // 18 MB beside 10 MB do not fit: the old scratch makes room.
    CHECK(c.call(18) == cudaSuccess && c.plan.sym.blocks == 0 && c.s.bytes == 18 * kMB + kArrivalsArea);
    CHECK(c.d.used == c.s.bytes && c.d.waits == 1);
    // What cannot be had at all is an error, and the next call that fits works.
    CHECK(c.call(60) == cudaErrorMemoryAllocation && c.s.mem == nullptr && c.s.bytes == 0 && c.d.used == 0);
    CHECK(c.call(5) == cudaSuccess && c.s.bytes == 5 * kMB + kArrivalsArea);
}

void counters() {
    Context c;
    c.d.budget = 1000 * kMB;
    CHECK(c.call(1) == cudaSuccess);
    const int clears = c.d.clears;
    PPPlan wide = fake_plan(1, false);  // counters beyond the common area
    wide.arrivals_bytes = 2 * kArrivalsArea;
    wide.partial_bytes = 3 * kArrivalsArea;
    const auto of = [&](bool) { return wide; };
    PPPlan p = pp_scratch_plan(c.s, of);
    CHECK(pp_scratch_ensure(c.s, p, c.d, of) == cudaSuccess && c.d.clears == clears + 1);
    CHECK(pp_scratch_ensure(c.s, p, c.d, of) == cudaSuccess && c.d.clears == clears + 1);
    CHECK(c.call(1) == cudaSuccess && c.d.clears == clears + 2);
}

void first_scratch() {
    Context c;
    c.d.budget = 25 * kMB;
    CHECK(pp_scratch_first(c.s, c.d) == cudaSuccess && c.s.mem == c.s.first && c.d.clears == 1);
    const auto small = [](bool) {
        PPPlan p;
        p.arrivals_bytes = 256;
        p.partial_bytes = 256 + 510 * 8 * 16;
        return p;
    };
    const int calls = c.d.calls();
    PPPlan p = pp_scratch_plan(c.s, small);
    CHECK(pp_scratch_ensure(c.s, p, c.d, small) == cudaSuccess && c.d.calls() == calls && c.s.mem == c.s.first);
    // A larger one beside it: no wait, nothing given back, then or when that one makes room.
    CHECK(c.call(1) == cudaSuccess && c.s.mem != c.s.first && c.d.waits == 0 && c.d.frees == 0);
    CHECK(c.call(18) == cudaSuccess && c.d.waits == 1 && c.d.frees == 1 && c.d.live.count(c.s.first) == 1);
    CHECK(c.call(60) == cudaErrorMemoryAllocation && c.s.mem == c.s.first && c.s.bytes == kFirstScratch);
    CHECK(c.d.used == kFirstScratch);
    p = pp_scratch_plan(c.s, small);
    CHECK(pp_scratch_ensure(c.s, p, c.d, small) == cudaSuccess && c.s.mem == c.s.first);
}

}  // namespace

int main() {
    first_scratch();
    plenty();
    pair_once_refused();
    ordered_refused();
    counters();
    if (line) std::printf("FAILED at line %d\n", line);
    return line ? 1 : 0;
}
