// The scratch of a context's direct sums (internal to the library).
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "kernels.h"

namespace nbody {

// Every plan's sums begin behind this much of the scratch, and its arrival
// counters (zero before and after a launch) lie within: a launch of one plan, also
// one replayed from a caller's graph, leaves the others' counters alone. Enough
// for 8M bodies.
constexpr size_t kArrivalsArea = 64 << 10;

// Scratch that a context has from the start: enough for the plans of up to 510
// bodies (eight slices of 16 bytes a body). They took one slice and no scratch
// before short slices came (pp_small_shape), so that their first call may itself
// be one that the caller captures, where nothing can be allocated. It is kept
// beside a larger one (giving it back would cost the first larger call a wait and
// a free, 12 us).
constexpr size_t kFirstScratch = kArrivalsArea + 510 * 8 * 16;

struct PPScratch {
    void *mem = nullptr;
    size_t bytes = 0;
    size_t arrivals = 0;         // bytes of arrival counters of the plan that used it last
    size_t refused = SIZE_MAX;   // a pair-once plan of this many bytes could not be had
    void *first = nullptr;       // kFirstScratch bytes, once pp_scratch_first has been called
};

// The context's first scratch.
template <class Mem>
cudaError_t pp_scratch_first(PPScratch &s, Mem &&m) {
    cudaError_t e = m.alloc(&s.first, kFirstScratch);
    if (e != cudaSuccess) return e;
    s.mem = s.first;
    s.bytes = kFirstScratch;
    s.arrivals = kArrivalsArea;
    return m.clear(s.first, kFirstScratch);
}

inline void pp_scratch_reserve(PPPlan &plan) {
    if (plan.partial_bytes == 0 || plan.arrivals_bytes >= kArrivalsArea) return;
    plan.partial_bytes += kArrivalsArea - plan.arrivals_bytes;
    plan.arrivals_bytes = kArrivalsArea;
}

// The plan for a context whose scratch is s. plan_of(allow_sym): the plan of
// these bodies, with the pair-once form or without. That form keeps every
// block's sums apart and takes much more scratch than the others (131,071
// bodies: 108 MB against 10): once it could not be had, plans as large go
// without.
template <class PlanOf>
PPPlan pp_scratch_plan(const PPScratch &s, PlanOf &&plan_of) {
    PPPlan plan = plan_of(true);
    pp_scratch_reserve(plan);
    if (plan.sym.blocks > 0 && plan.partial_bytes >= s.refused) {
        plan = plan_of(false);
        pp_scratch_reserve(plan);
    }
    return plan;
}

// Scratch for a plan from pp_scratch_plan, its arrival counters zero. m: alloc
// (device memory), clear (to zero, in the stream's order), wait (for the stream),
// free. The memory in use is given back only when the larger one is there, or
// where nothing else makes room. Where a plan's counters outgrow kArrivalsArea,
// they are cleared when the layout is not the one used last.
template <class Mem, class PlanOf>
cudaError_t pp_scratch_ensure(PPScratch &s, PPPlan &plan, Mem &&m, PlanOf &&plan_of) {
    if (plan.partial_bytes > s.bytes) {
        void *more = nullptr;
        cudaError_t e = m.alloc(&more, plan.partial_bytes);
        if (e == cudaErrorMemoryAllocation && plan.sym.blocks > 0) {
            s.refused = plan.partial_bytes;
            plan = pp_scratch_plan(s, plan_of);
            e = plan.partial_bytes > s.bytes ? m.alloc(&more, plan.partial_bytes) : cudaSuccess;
        }
        if (e == cudaErrorMemoryAllocation && s.mem != s.first) {
            if (const cudaError_t w = m.wait()) return w;
            m.free(s.mem);
            s.mem = s.first;
            s.bytes = s.first ? kFirstScratch : 0;
            s.arrivals = s.first ? kArrivalsArea : 0;
            e = m.alloc(&more, plan.partial_bytes);
        }
        if (e != cudaSuccess) return e;
        if (more) {
            e = m.clear(more, plan.partial_bytes);
            if (e == cudaSuccess && s.mem != s.first) e = m.wait();
            if (e != cudaSuccess) {
                m.free(more);
                return e;
            }
            if (s.mem != s.first) m.free(s.mem);
            s.mem = more;
            s.bytes = plan.partial_bytes;
            s.arrivals = plan.arrivals_bytes;
        }
    }
    if (plan.partial_bytes > 0 && plan.arrivals_bytes != s.arrivals) {
        if (const cudaError_t e = m.clear(s.mem, plan.arrivals_bytes)) return e;
        s.arrivals = plan.arrivals_bytes;
    }
    return cudaSuccess;
}

}  // namespace nbody
