// One launch over many trace jobs: different fields (of one store type),
// seed sets, integrators and tolerances.  Each job's lines occupy a
// warp-aligned range [begin[j], begin[j] + n_j) of the launch's line space, so
// no warp mixes two jobs; a thread finds its job by binary search over the
// (small) begin table and traces one line with that job's settings, both ways,
// lanes in lockstep.  Used for batched uneven solves (many
// fields in one captured graph) and by the serving loop to merge the work of
// concurrently admitted requests into one launch.
#pragma once
#include "qsl_trace.cuh"

namespace qsl {

template <bool TWIST, class F>
__device__ __forceinline__ void batch_line(const TraceJob<F>& J, long long line, bool in_window,
                                           bool split, unsigned& ns) {
    F f = J.f;
    if (f.d.nx < 2 || f.d.ny < 2 || f.d.nz < 2) return;
    long long n = J.s.n;
    if (J.s.n_dev) {  // count produced on the device; the range was sized by n
        const long long nd = (long long)__ldg(J.s.n_dev);
        n = nd < n ? nd : n;
    }
    if (line - (threadIdx.x & 31) >= n) return;  // past the job's lines (a whole warp, or a whole pair)
    const bool valid = in_window && line < n;    // else a padding lane of the job's warp-aligned range
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
        f, J, i, valid, split, LenLimit<false>{len_lim, 0.f}, [&J]() { return J.s.s_len; }, [&J]() { return J.s.tol_coef; },
        [&J]() { return v3(J.s.cross[0], J.s.cross[1], J.s.cross[2]); }, tw_on, ns);
}

// begin[j]: first line of job j (multiples of 32, increasing); begin[njobs]:
// the total.  Each job's TraceJob sits in device memory.  Only the lines of
// the window [line_lo, line_hi) run (a multiple of 32 for line_lo keeps every
// warp inside one job).
template <bool TWIST, class F>
__device__ __forceinline__ void batch_kernel_body(const TraceJob<F>* __restrict__ jobs,
                                                  const long long* __restrict__ begin, int njobs,
                                                  unsigned long long* samples, long long line_lo,
                                                  long long line_hi) {
    long long total = __ldg(begin + njobs);
    total = line_hi < total ? line_hi : total;
    const int lane = threadIdx.x & 31;
    const long long threads = (long long)gridDim.x * blockDim.x;
    const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x - lane;
    // two threads per line: the directions over warp pairs (trace_lines)
    const bool split = 2 * (total - line_lo) <= threads;
    const long long stride = split ? threads / 2 : threads;
    unsigned ns = 0;
    unsigned long long ns_total = 0;
    for (long long g = line_lo + (split ? (t >> 6) * 32 : t); g < total; g += stride) {
        int lo = 0, hi = njobs - 1;  // last j with begin[j] <= g
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (__ldg(begin + mid) <= g) lo = mid;
            else hi = mid - 1;
        }
        batch_line<TWIST>(jobs[lo], g + lane - __ldg(begin + lo), g + lane < total, split, ns);
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
