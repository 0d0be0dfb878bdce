// Field-line polylines for plotting: the fixed-step RK4 tracer of
// fastqslpy/MagTool.py (trilerp :3-18, Bnorm :20-22, RK4_bline :24-34,
// TraceBline :36-45), which records every point of a line instead of its
// footpoints.  That module computes in float64 (its weights come from
// float32 positions minus int64 indices, so every product and sum after the
// corner gather is float64) and stores the points as float32; each thread
// here follows one line in the same operation order with IEEE float64 adds,
// multiplies, divides and square roots (this translation unit is compiled
// with -fmad=false), so the stored points agree bit for bit.
//
// Behaviour kept from that module:
//  * a position is clamped per axis before sampling: below 0 -> 1e-8, above
//    n -> n - 1e-8; corner indices past the last node repeat the last node
//    (its slices come back shorter and broadcast);
//  * the 8 corner products are summed as a contiguous (2, 2, 2) float64
//    array: ((p000+p001)+(p010+p011)) + ((p100+p101)+(p110+p111)), index
//    order [x][y][z]; |B|^2 is summed x, y, z in sequence;
//  * the loop stops when any coordinate is below 0 or above nx (the first
//    axis length bounds all three); the current point is clamped in place at
//    the first sample of each step, and that clamped point is stored and
//    advanced.
// Where that module raises (a zero field sample gives NaN, a point exactly
// on the far face slices past the array), a line here stops at the NaN and
// clamps the index to the last node.
#include "qsl_internal.h"

namespace qsl {

struct PathField {
    const float *bx, *by, *bz;
    int n[3];
};

__device__ __forceinline__ double clamp_ref(double v, int n) {
    if (v < 0.0) return 1e-8;
    if (v > (double)n) return __dsub_rn((double)n, 1e-8);
    return v;
}

// trilerp (MagTool.py:3-18) at the clamped point c
__device__ void trilerp_ref(const PathField& F, const double c[3], double b[3]) {
    long long i0[3], i1[3];
    double w[3][2];
    for (int d = 0; d < 3; ++d) {
        long long i = (long long)c[d];  // truncation; c >= 0 after the clamp (NaN converts to 0)
        i = i < 0 ? 0 : (i > F.n[d] - 1 ? F.n[d] - 1 : i);
        i0[d] = i;
        i1[d] = i + 1 > F.n[d] - 1 ? F.n[d] - 1 : i + 1;
        const double f = __dsub_rn(c[d], (double)i);
        w[d][0] = __dsub_rn(1.0, f);
        w[d][1] = f;
    }
    const long long sx = 1, sy = F.n[0], sz = (long long)F.n[0] * F.n[1];
    const float* comp[3] = {F.bx, F.by, F.bz};
    for (int q = 0; q < 3; ++q) {
        double p[8];
        for (int i = 0; i < 2; ++i)
            for (int j = 0; j < 2; ++j)
                for (int k = 0; k < 2; ++k) {
                    const long long o = (i ? i1[0] : i0[0]) * sx + (j ? i1[1] : i0[1]) * sy + (k ? i1[2] : i0[2]) * sz;
                    const double wt = __dmul_rn(__dmul_rn(w[0][i], w[1][j]), w[2][k]);
                    p[i * 4 + j * 2 + k] = __dmul_rn((double)__ldg(comp[q] + o), wt);
                }
        b[q] = __dadd_rn(__dadd_rn(__dadd_rn(p[0], p[1]), __dadd_rn(p[2], p[3])),
                         __dadd_rn(__dadd_rn(p[4], p[5]), __dadd_rn(p[6], p[7])));
    }
}

// Bnorm (MagTool.py:20-22) at v (clamped on a copy)
__device__ void bnorm_ref(const PathField& F, const double v[3], double u[3]) {
    double c[3], b[3];
    for (int d = 0; d < 3; ++d) c[d] = clamp_ref(v[d], F.n[d]);
    trilerp_ref(F, c, b);
    const double s = __dsqrt_rn(__dadd_rn(__dadd_rn(__dmul_rn(b[0], b[0]), __dmul_rn(b[1], b[1])), __dmul_rn(b[2], b[2])));
    for (int d = 0; d < 3; ++d) u[d] = __ddiv_rn(b[d], s);
}

// Output indices start, start + stride, ... of a Python range(start, stop,
// stride), and the step along them.
struct PathRun {
    long long start, stop, stride;
    double dr;
};
struct PathArgs {
    PathField F;
    const double* seeds;  // n x 3
    long long n;
    PathRun run[2];       // per grid row (a line's two directions, or one run)
    float *ox, *oy, *oz;  // n x out_len
    long long out_len;
};
__device__ __forceinline__ bool in_range(const PathRun& R, long long idx) {
    return R.stride > 0 ? idx < R.stop : idx > R.stop;
}

// RK4_bline (MagTool.py:24-34), one thread per seed and run.  A warp's FP64
// operations take this GPU's FP64 pipe (two lanes per clock and SM) the same
// time for one lane as for 32, so this form is the faster one once there are
// lines enough to fill warps on every SM (kPathRuns).  BOTH: two runs a seed;
// one run's constants then need no register (6001 lines, 600 points: 13.06
// ms, 13.28 with the run picked by the grid row).
template <bool BOTH>
__global__ void __launch_bounds__(32) k_trace_path(const __grid_constant__ PathArgs A) {
    const long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= A.n) return;
    const PathRun& R = A.run[BOTH ? blockIdx.y : 0];
    double P[3] = {A.seeds[3 * s], A.seeds[3 * s + 1], A.seeds[3 * s + 2]};
    const double bound = (double)A.F.n[0];
    float* ox = A.ox + s * A.out_len;
    float* oy = A.oy + s * A.out_len;
    float* oz = A.oz + s * A.out_len;
    const double dr = R.dr;
    for (long long idx = R.start; in_range(R, idx); idx += R.stride) {
        if (P[0] < 0.0 || P[1] < 0.0 || P[2] < 0.0 || P[0] > bound || P[1] > bound || P[2] > bound) break;
        if (isnan(P[0]) || isnan(P[1]) || isnan(P[2])) break;
        for (int d = 0; d < 3; ++d) P[d] = clamp_ref(P[d], A.F.n[d]);
        double f1[3], f2[3], f3[3], f4[3], t[3];
        bnorm_ref(A.F, P, f1);
        for (int d = 0; d < 3; ++d) t[d] = __dadd_rn(P[d], __dmul_rn(dr, f1[d]) * 0.5);
        bnorm_ref(A.F, t, f2);
        for (int d = 0; d < 3; ++d) t[d] = __dadd_rn(P[d], __dmul_rn(dr, f2[d]) * 0.5);
        bnorm_ref(A.F, t, f3);
        for (int d = 0; d < 3; ++d) t[d] = __dadd_rn(P[d], __dmul_rn(dr, f3[d]));
        bnorm_ref(A.F, t, f4);
        ox[idx] = (float)P[0];
        oy[idx] = (float)P[1];
        oz[idx] = (float)P[2];
        for (int d = 0; d < 3; ++d) {
            const double k = __dadd_rn(__dadd_rn(__dadd_rn(f1[d], 2.0 * f2[d]), 2.0 * f3[d]), f4[d]);
            P[d] = __dadd_rn(P[d], __ddiv_rn(__dmul_rn(dr, k), 6.0));
        }
    }
}

// The same line by eight lanes.  One FP64 operation takes a warp 64 cycles
// here (19 per SM with four warps on it) whether its lanes are one or 32 and
// whether it waits for the one before or not, so what counts is how many a
// step issues: about 120 here against 700 one lane to a line (and the lines
// of a plot run on 8 times the warps).  Lane c of a group holds
//   * the corner (i, j, k) = bits (4, 2, 1) of c of the sample's cell,
//   * one component of every vector (c & 3 = 0: x, 1: y, 2 and 3: z), and of
//     that axis the fraction f (c < 4) or 1 - f.
// The corner products are summed over lanes as the reference's (2, 2, 2)
// array is, over k, then j, then i, each exchange also halving the components
// a lane holds.  Comparisons, truncations and the widening of the corner
// values are done on the bits.  Square root and quotients are Newton steps
// from the hardware's reciprocal square root, rounded once from an exact
// residual (Markstein) and tested (Ziv): where the last correction, stretched
// or shrunk by 2^-20 of itself, could round otherwise, the IEEE operation is
// called.  Every operation thus rounds as the reference's own and the points
// are the same bits.  300 lines of a 160 x 144 x 96 field, 2000 points each
// way: 10.4 ms, against 36.1 one lane to a line (both directions in one
// launch; 72 in two).  Eight lanes with the library's square root, division
// and conversions: 16.5 ms.
constexpr unsigned kAll = 0xffffffffu;
__device__ __forceinline__ double pick3(double v, int base, int comp) { return __shfl_sync(kAll, v, base + comp); }

// a lane's axis of the grid
struct PathAxis {
    int n;
    double top, last, inside;  // n, n - 1, n - 1e-8
};
// v < 0 (a negative zero is not; a NaN may count as either)
__device__ __forceinline__ bool below_zero(double v) {
    return __double2hiint(v) < 0 && __double_as_longlong(v) != (long long)0x8000000000000000ull;
}
// v > b of a v not below zero and a positive b (a NaN counts as above)
__device__ __forceinline__ bool above(double v, double b) {
    return __double_as_longlong(v) > __double_as_longlong(b);
}
// clamp_ref on the lane's axis
__device__ __forceinline__ double clamp_axis(double v, const PathAxis& X) {
    return below_zero(v) ? 1e-8 : (above(v, X.top) ? X.inside : v);
}
// Cell index of v in [0, n] and that index as a double: the mantissa bits
// above the binary point (a coordinate below 2^20; else the conversion).
__device__ __forceinline__ int cell_axis(double v, const PathAxis& X, double& id) {
    const int hi = __double2hiint(v), e = ((hi >> 20) & 0x7ff) - 1023;
    int i = 0;
    id = 0.0;
    if (e >= 20) {
        const long long q = (long long)v;
        i = q < 0 ? 0 : (q > X.n - 1 ? X.n - 1 : (int)q);
        id = (double)i;
    } else if (e >= 0) {
        i = ((hi & 0xfffff) | 0x100000) >> (20 - e);
        id = __hiloint2double(hi & ~((1 << (20 - e)) - 1), 0);
    }
    if (i > X.n - 1) {
        i = X.n - 1;
        id = X.last;
    }
    return i;
}
// the float at p as a double
__device__ __forceinline__ double widen(float f) {
    const unsigned u = __float_as_uint(f), x = u & 0x7fffffffu;
    if (x - 0x00800000u >= 0x7f000000u && x != 0u) return (double)f;  // subnormal, infinite, NaN
    return __hiloint2double((int)((u & 0x80000000u) | (x ? (x >> 3) + 0x38000000u : 0u)), (int)(u << 29));
}
// y stretched (d > 0) or shrunk by about d 2^-20 of itself
__device__ __forceinline__ double nudge(double y, int d) { return __hiloint2double(__double2hiint(y) + d, __double2loint(y)); }

// a / sqrt(s), both rounded (the square root first), s a sum of squares.
__device__ __forceinline__ double over_sqrt(double a, double s) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(s));
    // g -> sqrt(s), y -> 1 / sqrt(s), relative errors ~2^-38
    double g = __dmul_rn(s, y);
    const double e = __fma_rn(-g, nudge(y, -(1 << 20)), 0.5);  // 0.5 y: one less in the exponent
    g = __fma_rn(g, e, g);
    y = __fma_rn(y, e, y);
    const double d = __fma_rn(-g, g, s), h = nudge(y, -(1 << 20));
    const double r = __fma_rn(d, nudge(h, 1), g), r2 = __fma_rn(d, nudge(h, -1), g);
    // (the remainder negated, so that a zero keeps its sign)
    const double q = __dmul_rn(a, y), m = __fma_rn(q, r, -a);
    const double u = __fma_rn(-m, nudge(y, 1), q), u2 = __fma_rn(-m, nudge(y, -1), q);
    // s in [2^-500, 2^500]: no step over- or underflows
    const int ex = (__double2hiint(s) >> 20) - 1023;
    const bool sure = (r == r2) & (u == u2) & (ex >= -500) & (ex <= 500);
    return sure ? u : __ddiv_rn(a, __dsqrt_rn(s));
}

// x / 6
__device__ __forceinline__ double sixth(double x) {
    const double y = 1.0 / 6.0;
    const double q = __dmul_rn(x, y), m = __fma_rn(-6.0, q, x);
    const double u = __fma_rn(m, nudge(y, 1), q), u2 = __fma_rn(m, nudge(y, -1), q);
    const int ex = ((__double2hiint(x) >> 20) & 0x7ff) - 1023;
    return (u == u2) & (ex >= -500) & (ex <= 500) ? u : __ddiv_rn(x, 6.0);
}

// Bnorm at the point whose component on this lane's axis is v: this lane's
// component of the unit vector.
__device__ __forceinline__ double bnorm_lanes(const PathField& F, const PathAxis& X, double v, int c, int base) {
    v = clamp_axis(v, X);
    double id;
    const int i = cell_axis(v, X, id);
    const double f = __dsub_rn(v, id);
    const double wf = c < 4 ? f : __dsub_rn(1.0, f);
    // the weight and node index of this lane's corner
    double w = 0.0;
    long long o = 0, step = 1;
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const bool hi = (c >> (2 - d)) & 1;
        const double wd = __shfl_sync(kAll, wf, base + d + (hi ? 0 : 4));
        w = d == 0 ? wd : __dmul_rn(w, wd);
        int k = __shfl_sync(kAll, i, base + d);
        if (hi && k < F.n[d] - 1) ++k;
        o += k * step;
        step *= F.n[d];
    }
    const double px = __dmul_rn(widen(__ldg(F.bx + o)), w), py = __dmul_rn(widen(__ldg(F.by + o)), w),
                 pz = __dmul_rn(widen(__ldg(F.bz + o)), w);
    // over k: even lanes keep x, odd lanes y, both z
    const bool odd = c & 1;
    double a = __dadd_rn(odd ? py : px, __shfl_xor_sync(kAll, odd ? px : py, 1));
    const double b = __dadd_rn(pz, __shfl_xor_sync(kAll, pz, 1));
    // over j: lanes with j = 0 keep theirs, the others z
    const bool up = c & 2;
    a = __dadd_rn(up ? b : a, __shfl_xor_sync(kAll, up ? a : b, 2));
    // over i
    a = __dadd_rn(a, __shfl_xor_sync(kAll, a, 4));
    const double q = __dmul_rn(a, a);
    return over_sqrt(a, __dadd_rn(__dadd_rn(pick3(q, base, 0), pick3(q, base, 1)), pick3(q, base, 2)));
}

__global__ void __launch_bounds__(32) k_trace_path_lanes(const __grid_constant__ PathArgs A) {
    const int lane = threadIdx.x, c = lane & 7, base = lane & 24;
    const long long s = (long long)blockIdx.x * 4 + (lane >> 3);
    const PathRun R = A.run[blockIdx.y];
    bool alive = s < A.n;
    const long long row = alive ? s : 0;
    const int own = c & 2 ? 2 : c & 1;
    double P = A.seeds[3 * row + own];
    PathAxis X;
    X.n = own == 0 ? A.F.n[0] : (own == 1 ? A.F.n[1] : A.F.n[2]);
    X.top = (double)X.n;
    X.last = (double)(X.n - 1);
    X.inside = __dsub_rn(X.top, 1e-8);
    const double bound = (double)A.F.n[0], dr = R.dr;
    // lanes 0-2 of a group store its points
    float* const out = (own == 0 ? A.ox : (own == 1 ? A.oy : A.oz)) + row * A.out_len;
    for (long long idx = R.start; in_range(R, idx); idx += R.stride) {
        const bool in = !below_zero(P) && ((__double_as_longlong(P) << 1) == 0 || !above(P, bound));
        // (every lane votes, whether its line still runs or not)
        const unsigned votes = (__ballot_sync(kAll, in) >> base) & 7u;
        alive = alive & (votes == 7u);
        if (__ballot_sync(kAll, alive) == 0u) break;
        P = clamp_axis(P, X);
        const double f1 = bnorm_lanes(A.F, X, P, c, base);
        // (half a product and twice a vector are exact, so the multiply-adds
        // round as the sums do)
        const double f2 = bnorm_lanes(A.F, X, __fma_rn(0.5, __dmul_rn(dr, f1), P), c, base);
        const double f3 = bnorm_lanes(A.F, X, __fma_rn(0.5, __dmul_rn(dr, f2), P), c, base);
        const double f4 = bnorm_lanes(A.F, X, __dadd_rn(P, __dmul_rn(dr, f3)), c, base);
        if (alive && c < 3) out[idx] = (float)P;
        const double k = __dadd_rn(__fma_rn(2.0, f3, __fma_rn(2.0, f2, f1)), f4);
        P = __dadd_rn(P, sixth(__dmul_rn(dr, k)));
    }
}

// Runs (lines times directions) up to which eight lanes share one.  The FP64
// pipes of all SMs are full from ~2000 runs on and the time grows with the
// runs from there, while one lane to a run takes the same time for any number
// up to a warp per pipe (~10,000 and, both ways, ~14,000): 600 points a run,
// ms, eight lanes / one: 3000 runs 4.4 / 13.1, 6000 8.4 / 13.1, 8000 11.7 /
// 13.1, 9000 12.6 / 13.1, 10,000 14.8 / 13.1, 12,000 16.8 / 13.1.
constexpr long long kPathRuns = 9000;

static cudaError_t launch_path(const PathArgs& A, int runs, cudaStream_t st) {
    const bool wide = A.n * runs <= kPathRuns;
    const dim3 grid((unsigned)(wide ? (A.n + 3) / 4 : (A.n + 31) / 32), (unsigned)runs);
    if (wide) k_trace_path_lanes<<<grid, 32, 0, st>>>(A);
    else if (runs == 1) k_trace_path<false><<<grid, 32, 0, st>>>(A);
    else k_trace_path<true><<<grid, 32, 0, st>>>(A);
    return cudaGetLastError();
}

struct SampleArgs {
    PathField F;
    const double* pts;  // n x 3
    long long n;
    int normalize;
    double* out;  // n x 3
};

__global__ void __launch_bounds__(128) k_sample_points(const SampleArgs A) {
    const long long s = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (s >= A.n) return;
    const double v[3] = {A.pts[3 * s], A.pts[3 * s + 1], A.pts[3 * s + 2]};
    double r[3];
    if (A.normalize) {
        bnorm_ref(A.F, v, r);
    } else {
        double c[3];
        for (int d = 0; d < 3; ++d) c[d] = clamp_ref(v[d], A.F.n[d]);
        trilerp_ref(A.F, c, r);
    }
    for (int d = 0; d < 3; ++d) A.out[3 * s + d] = r[d];
}

cudaError_t launch_trace_path(const float* bx, const float* by, const float* bz, int nx, int ny, int nz,
                              const double* seeds, long long n, long long start, long long stop, long long stride,
                              double dr, float* ox, float* oy, float* oz, long long out_len, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    const PathRun r{start, stop, stride, dr};
    return launch_path(PathArgs{{bx, by, bz, {nx, ny, nz}}, seeds, n, {r, r}, ox, oy, oz, out_len}, 1, st);
}

cudaError_t launch_trace_path_both(const float* bx, const float* by, const float* bz, int nx, int ny, int nz,
                                   const double* seeds, long long n, long long mid, double dr, float* ox, float* oy,
                                   float* oz, long long out_len, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    return launch_path(PathArgs{{bx, by, bz, {nx, ny, nz}},
                                seeds,
                                n,
                                {PathRun{mid, out_len, 1, dr}, PathRun{mid, 0, -1, -dr}},
                                ox, oy, oz, out_len},
                       2, st);
}

cudaError_t launch_sample_points(const float* bx, const float* by, const float* bz, int nx, int ny, int nz,
                                 const double* pts, long long n, int normalize, double* out, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    const SampleArgs A{{bx, by, bz, {nx, ny, nz}}, pts, n, normalize, out};
    k_sample_points<<<(unsigned)((n + 127) / 128), 128, 0, st>>>(A);
    return cudaGetLastError();
}

}  // namespace qsl
