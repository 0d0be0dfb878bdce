// One launch over many trace jobs: different fields (of one store type),
// seed sets, integrators and tolerances.  Each job's lines occupy a
// warp-aligned range [begin[j], begin[j] + n_j) of the launch's line space, so
// no warp mixes two jobs; a warp finds its job by binary search over the
// (small) begin table and traces its lines with that job's settings, both
// ways, lanes in lockstep.  Used for batched uneven solves (many fields in one
// captured graph) and by the serving loop to merge the work of concurrently
// admitted requests into one launch.
#pragma once
#include "qsl_trace.cuh"

namespace qsl {

// The lines of one job that a warp holds: the first of them, counted from the
// job's start, and how the warp shares them (trace_lines, spread_of).
struct BatchSlot {
    long long first;
    bool split;
    int spread;
};

// The lines of one warp's turn in a job whose range starts at `begin` and
// holds `room` lines; `g` is the warp's line in the launch's line space.
//
// A job whose count comes from the device (n_dev) usually fills a small part
// of its range, and the warps past it would start and exit.  When the whole
// batch runs in one launch with the GPU's idle lanes at its disposal, its
// lines go to all the job's warps: directions to pairs of warps and up to four
// lanes per line (all after the main trace of two requests of 17,000 seeds:
// 0.90 -> 0.75 ms).
template <class F>
__device__ __forceinline__ BatchSlot batch_slot(const TraceJob<F>& J, long long n, long long g, long long begin,
                                                long long room, bool whole) {
    if (J.s.n_dev && whole) {
        // the job's warps as pairs of the block; its first warp may be the
        // second of a pair
        const long long warp = (g - begin) / 32;
        const int odd = (int)(((threadIdx.x >> 5) ^ (unsigned)warp) & 1u);
        const long long usable = (room / 32 - odd) & ~1LL;
        if (splits(n, usable)) {
            int s = spread_of(n, usable);
            while (s > 1 && 2 * ((n * s + 31) / 32) > usable) s /= 2;
            if (2 * ((n * s + 31) / 32) <= usable)
                return {warp < odd ? n : ((warp - odd) >> 1) * (32 / s), true, s};
        }
    }
    return {g - begin, false, 1};
}

template <bool TWIST, class F>
__device__ __forceinline__ void batch_line(const TraceJob<F>& J, const BatchSlot& slot, long long n, long long skip,
                                           long long left, unsigned& ns) {
    F f = J.f;
    if (f.d.nx < 2 || f.d.ny < 2 || f.d.nz < 2) return;
    const int lane = threadIdx.x & 31;
    const long long line = slot.first + lane / slot.spread;
    if (slot.first >= n) return;  // past the job's lines (a whole warp, or a whole pair)
    // else lanes past the job's lines, outside the window, or between spread lines
    const int k = lane / slot.spread;
    const bool valid = lane % slot.spread == 0 && line < n && k >= skip && k < left;
    const long long i = (valid && J.order) ? (long long)__ldg(J.order + line) : line;
    const bool tw_on = TWIST && J.s.twist_on != 0;
    store_prepare(f);
    float len_lim;
    if constexpr (std::is_same<F, FieldH4B>::value || std::is_same<F, FieldH4BW>::value || std::is_same<F, FieldF4>::value ||
                  std::is_same<F, FieldH8C>::value)
        len_lim = J.lim.len_lim;
    else
        len_lim = (float)(J.prm.len_ratio * len_scale(f));
    trace_lines<false, TWIST>(
        f, J, i, valid, slot.split, LenLimit<false>{len_lim, 0.f}, [&J]() { return J.s.s_len; },
        [&J]() { return J.s.tol_coef; }, [&J]() { return v3(J.s.cross[0], J.s.cross[1], J.s.cross[2]); }, tw_on, ns);
}

// The shape of a launch of n lines of the batch: without spare lanes one
// thread per line, whatever the grid.
__host__ __device__ __forceinline__ LaunchShape batch_shape(long long n, long long warps, bool lanes_free) {
    return lanes_free ? launch_shape(n, warps) : LaunchShape{false, 1};
}

// begin[j]: first line of job j (multiples of 32, increasing); begin[njobs]:
// the total.  Each job's TraceJob sits in device memory.  Only the lines of
// the window [line_lo, line_hi) run.  The warps' lines are counted from the
// multiple of 32 at or below line_lo, whatever the window, so that every warp
// stays inside one job; lanes below line_lo have no line.  lanes_free: the
// launch may give a line several lanes (a caller that limits its blocks shares
// the GPU with other launches: then it may not).
template <bool TWIST, class F>
__device__ __forceinline__ void batch_kernel_body(const TraceJob<F>* __restrict__ jobs,
                                                  const long long* __restrict__ begin, int njobs,
                                                  unsigned long long* samples, long long line_lo,
                                                  long long line_hi, bool lanes_free) {
    long long total = __ldg(begin + njobs);
    const long long warps = (long long)gridDim.x * (kTraceThreads / 32);
    // the whole batch in this launch, with the GPU's idle lanes at its disposal
    const bool whole = lanes_free && line_lo == 0 && line_hi >= total && 32 * warps >= total;
    total = line_hi < total ? line_hi : total;
    const long long w = (long long)blockIdx.x * (kTraceThreads / 32) + (threadIdx.x >> 5);
    // lanes to spare: the directions over warp pairs, fewer lines per warp
    const long long base = line_lo & ~31LL;
    const LaunchShape shape = batch_shape(total - base, warps, lanes_free);
    const bool split = shape.split;
    const int spread = shape.spread;
    const int lines = 32 / spread;
    const long long stride = warps * lines / (split ? 2 : 1);
    unsigned ns = 0;
    unsigned long long ns_total = 0;
    for (long long g = base + (split ? w >> 1 : w) * lines; g < total; g += stride) {
        int lo = 0, hi = njobs - 1;  // last j with begin[j] <= g
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(begin + mid) <= g) lo = mid;
            else hi = mid - 1;
        }
        const TraceJob<F>& J = jobs[lo];
        const long long b = __ldg(begin + lo);
        long long n = J.s.n;
        if (J.s.n_dev) {  // count produced on the device; the range was sized by n
            const long long nd = (long long)__ldg(J.s.n_dev);
            n = nd < n ? nd : n;
        }
        const BatchSlot slot =
            split ? BatchSlot{g - b, true, spread} : batch_slot(J, n, g, b, __ldg(begin + lo + 1) - b, whole);
        batch_line<TWIST>(J, slot, n, line_lo - g, split | !slot.split ? total - g : 32, ns);
        ns_total += ns;
        ns = 0;
    }
    if (samples) {
        __syncwarp();
        unsigned long long v = ns_total;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0) atomicAdd(samples, v);
    }
}

}  // namespace qsl
