// Kernel templates of the fast tracers and their launchers, instantiated per
// field store by one translation unit each (trace_fast_soa.cu, trace_fast_f4.cu,
// trace_fast_h4b.cu, trace_fast_h8c.cu), compiled in parallel.
#pragma once
#include "qsl_internal.h"

namespace qsl {

// MINB: minimum resident blocks per SM the register allocation must allow
// (1 = compiler's choice).  Higher values trade registers (possibly spills)
// for resident warps; the autotuner measures and picks.
template <bool TWIST, bool QUEUE, class F, int MINB>
__global__ void __launch_bounds__(kTraceBlock, MINB) k_trace_fast(const __grid_constant__ TraceJob<F> J) {
    trace_kernel_body<false, TWIST, QUEUE>(J);
}

// The static brick kernel in blocks of 256, for launches of many waves: four
// 8 x 8 seed tiles then share an SM's L1 instead of two (258 x 258 x 128 seeds
// of a 512 x 512 x 256 field 106.1 -> 103.4 ms).  Launches of a wave or two
// lose by it (258 x 514 seeds 1.14 -> 1.18 ms: a block's warps wait for its
// longest line), and below a full wave the directions split over pairs of
// warps, which the 128-thread blocks are made for.
constexpr int kWideBlock = 256;
constexpr int kWideWaves = 8;
template <bool TWIST, class F, int MINB>
__global__ void __launch_bounds__(kWideBlock, MINB* kTraceBlock / kWideBlock)
    k_trace_fast_wide(const __grid_constant__ TraceJob<F> J) {
    trace_kernel_body<false, TWIST, false>(J);
}

template <class F, int MINB>
static cudaError_t launch_fast_minb(const TraceJob<F>& J, bool twist, Schedule sched, long long n_host,
                                    cudaStream_t st) {
    const bool q = sched == SCHED_QUEUE;
    const void* k = q ? (twist ? (const void*)k_trace_fast<true, true, F, MINB>
                               : (const void*)k_trace_fast<false, true, F, MINB>)
                      : (twist ? (const void*)k_trace_fast<true, false, F, MINB>
                               : (const void*)k_trace_fast<false, false, F, MINB>);
    int grid = persistent_grid(k, kTraceBlock);
    if (!q) {
        // a device-side count (n_host is only the capacity): at most two
        // resident waves of blocks stride over the lines instead of a grid
        // over the whole capacity whose surplus blocks would each start and
        // exit
        const int waves = 2 * grid;
        if constexpr (std::is_same<F, FieldH4B>::value && MINB == 6) {
            const long long blocks = (n_host + kWideBlock - 1) / kWideBlock;
            if (grid > 0 && !J.s.n_dev && n_host >= (long long)kWideWaves * grid * kTraceBlock && blocks <= (1 << 30)) {
                if (twist) k_trace_fast_wide<true, F, MINB><<<(int)blocks, kWideBlock, 0, st>>>(J);
                else k_trace_fast_wide<false, F, MINB><<<(int)blocks, kWideBlock, 0, st>>>(J);
                return cudaGetLastError();
            }
        }
        grid = static_grid(n_host, grid);
        if (J.s.n_dev && waves > 0 && grid > waves) grid = waves;
    }
    if (grid <= 0) return cudaErrorInvalidConfiguration;
    if (q) {
        if (twist) k_trace_fast<true, true, F, MINB><<<grid, kTraceBlock, 0, st>>>(J);
        else k_trace_fast<false, true, F, MINB><<<grid, kTraceBlock, 0, st>>>(J);
    } else {
        if (twist) k_trace_fast<true, false, F, MINB><<<grid, kTraceBlock, 0, st>>>(J);
        else k_trace_fast<false, false, F, MINB><<<grid, kTraceBlock, 0, st>>>(J);
    }
    return cudaGetLastError();
}

template <class F>
static cudaError_t launch_fast(const TraceJob<F>& J, bool twist, Schedule sched, long long n_host, cudaStream_t st) {
    switch (J.occupancy) {
        case 6: return launch_fast_minb<F, 6>(J, twist, sched, n_host, st);
        case 7: return launch_fast_minb<F, 7>(J, twist, sched, n_host, st);
        case 8: return launch_fast_minb<F, 8>(J, twist, sched, n_host, st);
        case 9: return launch_fast_minb<F, 9>(J, twist, sched, n_host, st);
        case 10: return launch_fast_minb<F, 10>(J, twist, sched, n_host, st);
        default: return launch_fast_minb<F, 1>(J, twist, sched, n_host, st);
    }
}

// (held to 3 blocks per SM: 168 registers; the twist form would take ~210)
template <int GRAD, bool TWIST, class F>
__global__ void __launch_bounds__(kTraceBlock, 3) k_scott_fast(const ScottJob<F> J) {
    scott_kernel_body<false, GRAD, TWIST>(J);
}

template <class F>
static cudaError_t launch_scott(const ScottJob<F>& J, int grad, bool twist, long long n_grid, cudaStream_t st) {
    long long g = (n_grid + kTraceBlock - 1) / kTraceBlock;
    const int grid = (int)(g < 1 ? 1 : (g > (1 << 30) ? (1 << 30) : g));
    if (grad == GRAD_ANALYTIC) {
        if (twist) k_scott_fast<GRAD_ANALYTIC, true, F><<<grid, kTraceBlock, 0, st>>>(J);
        else k_scott_fast<GRAD_ANALYTIC, false, F><<<grid, kTraceBlock, 0, st>>>(J);
    } else {
        if (twist) k_scott_fast<GRAD_FD, true, F><<<grid, kTraceBlock, 0, st>>>(J);
        else k_scott_fast<GRAD_FD, false, F><<<grid, kTraceBlock, 0, st>>>(J);
    }
    return cudaGetLastError();
}

// Batched trace; MINB resident blocks per SM the register allocation must
// allow (6-10; the autotuner picks, 6 by default).
template <bool TWIST, class F, int MINB>
__global__ void __launch_bounds__(kTraceBlock, MINB) k_trace_batch(const TraceJob<F>* __restrict__ jobs,
                                                                    const long long* __restrict__ begin, int njobs,
                                                                    unsigned long long* samples, long long line_lo,
                                                                    long long line_hi, bool lanes_free) {
    batch_kernel_body<TWIST>(jobs, begin, njobs, samples, line_lo, line_hi, lanes_free);
}

template <class F, int MINB>
static void launch_batch_minb(int grid, const TraceJob<F>* jobs, const long long* begin, int njobs, bool twist,
                              unsigned long long* samples, long long line_lo, long long line_hi, bool lanes_free,
                              cudaStream_t st) {
    auto k = twist ? k_trace_batch<true, F, MINB> : k_trace_batch<false, F, MINB>;
    k<<<grid, kTraceBlock, 0, st>>>(jobs, begin, njobs, samples, line_lo, line_hi, lanes_free);
}

template <class F, int MINB>
static const void* batch_kernel_minb(bool twist) {
    return twist ? (const void*)k_trace_batch<true, F, MINB> : (const void*)k_trace_batch<false, F, MINB>;
}
template <class F>
static const void* batch_kernel(int occupancy, bool twist) {
    switch (occupancy) {
        case 7: return batch_kernel_minb<F, 7>(twist);
        case 8: return batch_kernel_minb<F, 8>(twist);
        case 9: return batch_kernel_minb<F, 9>(twist);
        case 10: return batch_kernel_minb<F, 10>(twist);
        default: return batch_kernel_minb<F, 6>(twist);
    }
}

template <class F>
static cudaError_t launch_batch(const TraceJob<F>* jobs, const long long* begin, int njobs, long long total,
                                bool twist, unsigned long long* samples, int max_blocks, long long line_lo,
                                long long line_hi, int occupancy, cudaStream_t st) {
    if (njobs <= 0 || total <= 0) return cudaSuccess;
    if (line_lo < 0) line_lo = 0;
    if (line_hi < 0 || line_hi > total) line_hi = total;
    if (line_lo >= line_hi) return cudaSuccess;
    const int resident = persistent_grid(batch_kernel<F>(occupancy, twist), kTraceBlock);
    if (resident <= 0) return cudaErrorInvalidConfiguration;
    const int grid = batch_grid(line_hi - (line_lo & ~31LL), resident, max_blocks);  // (batch_kernel_body's first line)
    const bool free = max_blocks <= 0;
    switch (occupancy) {
        case 7: launch_batch_minb<F, 7>(grid, jobs, begin, njobs, twist, samples, line_lo, line_hi, free, st); break;
        case 8: launch_batch_minb<F, 8>(grid, jobs, begin, njobs, twist, samples, line_lo, line_hi, free, st); break;
        case 9: launch_batch_minb<F, 9>(grid, jobs, begin, njobs, twist, samples, line_lo, line_hi, free, st); break;
        case 10: launch_batch_minb<F, 10>(grid, jobs, begin, njobs, twist, samples, line_lo, line_hi, free, st); break;
        default: launch_batch_minb<F, 6>(grid, jobs, begin, njobs, twist, samples, line_lo, line_hi, free, st); break;
    }
    return cudaGetLastError();
}

}  // namespace qsl
