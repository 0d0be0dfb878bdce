// Field-line tracer kernels (RK4 / RKF45), templated on the field store and
// the arithmetic.  Semantics per seed follow the reference's TraceAllBline
// (fastqslpy/cu/TraceBlineAdaptive.cu:429-510, fastqslpy/cu/TraceBline.cu:
// 383-464): forward trace -> end footpoint, backward trace -> start footpoint,
// B at both footpoints and at the seed, B_flag, line length, optional twist.
//
// Scheduling: a warp takes 32 lines (neighbouring seeds when the order is a
// tile order) and traces them in lockstep, each lane forward and then
// backward; the footpoints, the samples of B and the outputs follow once for
// the whole warp (trace_lines).  Where the launch has two threads per line,
// the directions go to a pair of warps instead.  Static: the warp's lines
// follow from its index; queue: a persistent grid whose warps take lines from
// a device counter, new ones for the lanes that wait when the rest of a warp
// takes too long (trace_queue), for device-side counts and for lines whose
// lengths differ by orders of magnitude.
//
// What it replaced: every lane taking its next line from the queue as its
// own ended, and doing its line's end then and there.  A warp's lanes were
// then at different points of the loop (9-13 of 32 active, instruction-fetch
// stalls at 10-15 cycles per issue in the exact kernels) and their gathers
// scattered.  Drop-in RKF45 on 201 x 203 x 4 seeds with twist 11.0 -> 4.0 ms,
// map of 256 x 512 seeds 11.0 -> 6.6 ms, RK4 on 128 x 128 seeds 5.0 -> 3.2 ms;
// fast kernels: 100 x 100 seeds in 64^3 0.366 -> 0.244 ms, a 258 x 258 x 32
// slab of 512 x 512 x 256 22.5 -> 21.4 ms.
#pragma once
#include <type_traits>
#include "qsl_field.cuh"
#include "../../include/fastqsl_gb300.h"

namespace qsl {

constexpr int kTraceThreads = 128;  // threads per block of the tracer kernels (kWideBlock in one case)

constexpr double kRefPi = 3.14159265;  // the reference's M_PI (TraceBlineAdaptive.cu:10)
// 1 / (4 pi) for the fast twist increment: one float product per step and a
// single double add, instead of the reference's double divides (the FP64
// pipe is narrow on this GPU)
constexpr float kInv4PiF = (float)(1.0 / (4.0 * kRefPi));

struct TraceOut {
    float *start_x, *start_y, *start_z;
    int* flag_start;
    float *end_x, *end_y, *end_z;
    int* flag_end;
    float *bthis_x, *bthis_y, *bthis_z;
    int* b_flag;
    float *bstart_x, *bstart_y, *bstart_z;
    float *bend_x, *bend_y, *bend_z;
    double* line_len;
    double* twist;
    int* status_start;  // optional qsl_line_status per direction
    int* status_end;
};

// Scalars the reference passes as one-element device arrays are read from
// device memory when the *_dev pointer is set, else taken by value.
struct TraceScalars {
    const float* s_len_dev;
    const float* tol_coef_dev;
    const unsigned long long* n_dev;
    const float* cross_dev;
    const bool* twist_flag_dev;
    long long n_cap;  // >= 0: lines beyond this index are never touched (array capacity)
    float s_len;
    float tol_coef;
    long long n;
    float cross[3];
    int twist_on;
};

// Step-size limits of the adaptive controller narrowed to float once on the
// host.  For a float h and a double bound H, `h > H` and `h > (float)H` clamp
// h to the same value (the only float between H and its rounding is the
// rounding itself), so the fast kernels compare in float and keep the FP64
// pipe off the per-step path.  max_steps is clamped to the int range of the
// lane's step counter.
struct StepLimits {
    float h_min, h_max, reject;
    int max_steps;
    float len_lim;  // len_ratio x (nx + ny + nz) in float, formed on the host (packed stores)
};

template <class F>
struct TraceJob {
    F f;
    const int* shape_dev;  // when set, the field dims are read from here (nx, ny, nz)
    FieldSoA cur;  // current density for the twist integral (the caller's arrays)
    F cur_store;   // or, when cur_packed, the current density in a store of F's layout
    int cur_packed;
    const float *inp_x, *inp_y, *inp_z;
    TraceOut o;
    TraceScalars s;
    qsl_trace_params prm;
    StepLimits lim;               // prm's controller limits in float (fast arithmetic)
    unsigned long long* queue;    // work counter, zero at launch; null = static
    unsigned long long* samples;  // optional: total field samples
    const unsigned* order;        // optional: line k traces seed order[k] and writes its outputs there
    int chunk;                    // most lines a warp takes from the queue at a time (QUEUE; 0 = 32)
    int occupancy;                // resident-block variant of the fast kernels (0 = default)
};

// Fehlberg 4(5) coefficients, stored to float as the reference does
// (TraceBlineAdaptive.cu:224-235).
struct Fehlberg {
    static constexpr float a21 = (float)(1. / 4.);
    static constexpr float a31 = (float)(3. / 32.), a32 = (float)(9. / 32.);
    static constexpr float a41 = (float)(1932. / 2197.), a42 = (float)(-7200. / 2197.), a43 = (float)(7296. / 2197.);
    static constexpr float a51 = (float)(439. / 216.), a52 = -8.f, a53 = (float)(3680. / 513.),
                           a54 = (float)(-845. / 4104.);
    static constexpr float a61 = (float)(-8. / 27.), a62 = 2.f, a63 = (float)(-3544. / 2565.),
                           a64 = (float)(1859. / 4104.), a65 = (float)(-11. / 40.);
    static constexpr float b1 = (float)(16. / 135.), b3 = (float)(6656. / 12825.), b4 = (float)(28561. / 56430.),
                           b5 = (float)(-9. / 50.), b6 = (float)(2. / 55.);
    static constexpr float e1 = (float)(1. / 360.), e3 = (float)(-128. / 4275.), e4 = (float)(-2197. / 75240.),
                           e5 = (float)(1. / 50.), e6 = (float)(2. / 55.);
};

// One Fehlberg step (RKF45, TraceBlineAdaptive.cu:215-254): returns the
// 5th-order increment (the reference adds it to P0 in one rounding) and the
// error estimate: its norm in exact arithmetic; in fast arithmetic its
// square, h^2 |e|^2 (the fast controller works with log2 of it, so no square
// root is taken).
// Vector as an (x, y) pair for the packed f32x2 pipe plus a scalar z.
struct PV {
    float2 xy;
    float z;
};
__device__ __forceinline__ PV pv(float3 a) { return {make_float2(a.x, a.y), a.z}; }
__device__ __forceinline__ float3 f3(PV a) { return v3(a.xy.x, a.xy.y, a.z); }
// a*x + y
__device__ __forceinline__ PV axpy(float a, PV x, PV y) {
    return {__ffma2_rn(make_float2(a, a), x.xy, y.xy), fmaf(a, x.z, y.z)};
}
__device__ __forceinline__ PV scal(float a, PV x) { return {__fmul2_rn(make_float2(a, a), x.xy), a * x.z}; }

// Fast-arithmetic Fehlberg step: the same stages on the unit field b with
// the step folded in once per stage (p + h * sum a_ij b_j), combinations on
// packed (x, y) pairs.  Differs from the reference's rounding sequence only
// in rounding.  err2: the squared error estimate h^2 |e|^2.
template <class F>
__device__ __forceinline__ float3 step_rkf45_fast(const F& f, float3 p, float h, float& err2, unsigned& ns,
                                                 float3* b_raw = nullptr) {
    using C = Fehlberg;
    const PV P = pv(p);
    // b_raw: also return B itself at p (from the same interpolation)
    const PV b1 = pv(b_raw ? sample_unit_raw(f, p, *b_raw) : sample<false>(f, p, true));
    const PV b2 = pv(sample<false>(f, f3(axpy(h * C::a21, b1, P)), true));
    PV c = axpy(C::a32, b2, scal(C::a31, b1));
    const PV b3 = pv(sample<false>(f, f3(axpy(h, c, P)), true));
    c = axpy(C::a43, b3, axpy(C::a42, b2, scal(C::a41, b1)));
    const PV b4 = pv(sample<false>(f, f3(axpy(h, c, P)), true));
    c = axpy(C::a54, b4, axpy(C::a53, b3, axpy(C::a52, b2, scal(C::a51, b1))));
    const PV b5 = pv(sample<false>(f, f3(axpy(h, c, P)), true));
    c = axpy(C::a65, b5, axpy(C::a64, b4, axpy(C::a63, b3, axpy(C::a62, b2, scal(C::a61, b1)))));
    const PV b6 = pv(sample<false>(f, f3(axpy(h, c, P)), true));
    const PV e = axpy(C::e6, b6, axpy(C::e5, b5, axpy(C::e4, b4, axpy(C::e3, b3, scal(C::e1, b1)))));
    err2 = (h * h) * fmaf(e.xy.x, e.xy.x, fmaf(e.xy.y, e.xy.y, e.z * e.z));
    ns += 6;
    return f3(scal(h, axpy(C::b6, b6, axpy(C::b5, b5, axpy(C::b4, b4, axpy(C::b3, b3, scal(C::b1, b1)))))));
}

// The fast Fehlberg step with its six stages in a rolled loop, for the
// stretched-grid stores: their sample (three axis searches, eight corner
// loads and the blend) inlined six times makes a loop body that does not fit
// the instruction cache.  The sums of the stages still to come are held in
// a shift register of five vectors: entering stage st, slot[i] is the sum
// of stage st + i (slot[0] complete); after its sample each slot takes the
// next one's sum plus this stage's term, so the shift costs no moves and
// every index is static.  Coefficients from constant memory.  The same sums
// in the same order as step_rkf45_fast except that the step multiplies each
// stage's sum (h * sum a_ij b_j) instead of being folded into a21.
struct FehlbergTab {
    float a[6][5];  // a[st][i] = A(st + 1 + i, st)
    float b[6], e[6];
};
static __constant__ FehlbergTab kFehlbergTab = {
    {{Fehlberg::a21, Fehlberg::a31, Fehlberg::a41, Fehlberg::a51, Fehlberg::a61},
     {Fehlberg::a32, Fehlberg::a42, Fehlberg::a52, Fehlberg::a62, 0.f},
     {Fehlberg::a43, Fehlberg::a53, Fehlberg::a63, 0.f, 0.f},
     {Fehlberg::a54, Fehlberg::a64, 0.f, 0.f, 0.f},
     {Fehlberg::a65, 0.f, 0.f, 0.f, 0.f},
     {0.f, 0.f, 0.f, 0.f, 0.f}},
    {Fehlberg::b1, 0.f, Fehlberg::b3, Fehlberg::b4, Fehlberg::b5, Fehlberg::b6},
    {Fehlberg::e1, 0.f, Fehlberg::e3, Fehlberg::e4, Fehlberg::e5, Fehlberg::e6}};

template <class F>
struct RolledStages : std::false_type {};
template <int M>
struct RolledStages<FieldStretchT<M>> : std::true_type {};

template <class F>
__device__ __forceinline__ float3 step_rkf45_fast_rolled(const F& f, float3 p, float h, float& err2, unsigned& ns,
                                                        float3* b_raw) {
    const PV P = pv(p);
    const PV zero = {make_float2(0.f, 0.f), 0.f};
    PV slot[5] = {zero, zero, zero, zero, zero};
    PV sol = zero, e = zero;
    // b_raw (twist kernels): the first stage's B itself, from its own
    // interpolation before the loop so that the loop holds one sample
    PV b = pv(b_raw ? sample_unit_raw(f, p, *b_raw) : sample<false>(f, p, true));
#pragma unroll 1
    for (int st = 0; st < 6; ++st) {
        if (st > 0) b = pv(sample<false>(f, f3(axpy(h, slot[0], P)), true));
#pragma unroll
        for (int i = 0; i < 4; ++i) slot[i] = axpy(kFehlbergTab.a[st][i], b, slot[i + 1]);
        slot[4] = scal(kFehlbergTab.a[st][4], b);
        sol = axpy(kFehlbergTab.b[st], b, sol);
        e = axpy(kFehlbergTab.e[st], b, e);
    }
    err2 = (h * h) * fmaf(e.xy.x, e.xy.x, fmaf(e.xy.y, e.xy.y, e.z * e.z));
    ns += 6;
    return f3(scal(h, sol));
}

// aside(st) runs at the start of stage st of an exact step: work whose results
// are not needed in the step (Lane's pending sums), placed where the stage's
// sample hides its latency.  Without any:
struct Nothing {
    __device__ __forceinline__ void operator()(int) const {}
    template <class F>
    __device__ __forceinline__ void field(const F&, int, int3, const float*, float3) const {}
};
// The unit field at p by exact arithmetic; aside.field(st, ...) is given the
// cell, its corner weights and B before the normalisation.
template <class F, class A>
__device__ __forceinline__ float3 stage_exact(const F& f, float3 p, int st, A& aside) {
    int3 cell;
    float w[8];
    cell_exact(f, p, cell, w);
    float3 c[8];
    f.corners(cell.x, cell.y, cell.z, c);
    const float3 raw = blend<true>(c, w);
    aside.field(f, st, cell, w, raw);
    return unit_exact(raw);
}
// The exact Fehlberg step: k = h b per stage, every product and sum rounded on
// its own in the reference's order (sums from the left; a stage's input is
// p plus its whole sum).  The stages are rolled as above: each stage's k adds
// its term to the sums still to come, which is that order.  (Unrolled, the
// exact samples do not fit the instruction cache: drop-in planes 18-35 %
// slower.)
template <class F, class A>
__device__ __forceinline__ float3 step_rkf45_exact(const F& f, float3 p, float h, float& err, unsigned& ns, A& aside) {
    const float3 zero = v3(0.f, 0.f, 0.f);
    float3 slot[5] = {zero, zero, zero, zero, zero};
    float3 sol = zero, e = zero;
#pragma unroll 1
    for (int st = 0; st < 6; ++st) {
        aside(st);
        const float3 k = h * stage_exact(f, st > 0 ? p + slot[0] : p, st, aside);
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            const float3 t = kFehlbergTab.a[st][i] * k;
            slot[i] = st > 0 ? (i < 4 ? slot[i + 1] + t : t) : t;
        }
        const float3 ts = kFehlbergTab.b[st] * k, te = kFehlbergTab.e[st] * k;
        sol = st > 0 ? sol + ts : ts;
        e = st > 0 ? e + te : te;
    }
    err = norm(e);
    ns += 6;
    return sol;
}

template <bool EXACT, class F, class A>
__device__ __forceinline__ float3 step_rkf45(const F& f, float3 p, float h, float& err, unsigned& ns, float3* b_raw,
                                            A& aside) {
    if constexpr (EXACT) return step_rkf45_exact(f, p, h, err, ns, aside);
    else if constexpr (RolledStages<F>::value) return step_rkf45_fast_rolled(f, p, h, err, ns, b_raw);
    else return step_rkf45_fast(f, p, h, err, ns, b_raw);
}

// (float)((1. / 6.) * (double)h) without the FP64 pipe: h times the double
// 1/6 held as two floats.
__device__ __forceinline__ float sixth_exact(float h) {
    constexpr double y = 1.0 / 6.0;
    constexpr float yh = (float)y, yl = (float)(y - (double)(float)y);
    bool sure = (fabsf(h) >= 0x1p-60f) & (fabsf(h) <= 0x1p+60f);
    const float p = h * yh;
    const float r = round_f2(F2{p, __fmaf_rn(h, yl, __fmaf_rn(h, yh, -p))}, sure);
    return sure ? r : (float)(y * (double)h);
}

// Classic RK4 on b (RK4, TraceBlineAdaptive.cu:259-267); returns the
// increment.  Exact arithmetic: the 1/6 factor as (1./6.)*h rounded once, and
// the stages rolled (one sample in the loop body; the same operations in the
// same order).
template <bool EXACT, class F, class A>
__device__ __forceinline__ float3 step_rk4(const F& f, float3 p, float h, unsigned& ns, float3* b_raw, A& aside) {
    ns += 4;
    if constexpr (EXACT) {
        float3 q = p, sum = v3(0.f, 0.f, 0.f);
#pragma unroll 1
        for (int st = 0; st < 4; ++st) {
            aside(st);
            const float3 k = stage_exact(f, q, st, aside);
            const float3 hk = h * k;
            q = p + (st < 2 ? 0.5f * hk : hk);
            sum = st == 0 ? k : (st < 3 ? sum + 2.f * k : sum + k);
        }
        return sixth_exact(h) * sum;
    } else {
        const float3 k1 = b_raw ? sample_unit_raw(f, p, *b_raw) : sample<false>(f, p, true);
        const float3 k2 = sample<false>(f, p + (h * k1) / 2.f, true);
        const float3 k3 = sample<false>(f, p + (h * k2) / 2.f, true);
        const float3 k4 = sample<false>(f, p + h * k3, true);
        return h * (1.f / 6.f) * (((k1 + 2.f * k2) + 2.f * k3) + k4);
    }
}

// RK4 in the face-normal coordinate, dx/dq = b / b_d over dq = h
// (RK4_boundary, TraceBlineAdaptive.cu:286-307), its four stages in a rolled
// loop (it runs once per line end).  4 field samples.
template <bool EXACT, class F>
__device__ __forceinline__ float3 step_rk4_normal(const F& f, float3 p, float h, int d) {
    float3 k1 = v3(0.f, 0.f, 0.f), k2 = k1, k3 = k1, k4 = k1, q = p;
#pragma unroll 1
    for (int st = 0; st < 4; ++st) {
        const float3 b = sample_outlined<EXACT>(f, q, true);
        const float3 k = b / comp(b, d);
        if (st == 0) {
            k1 = k;
            q = p + (h * k1) / 2.f;
        } else if (st == 1) {
            k2 = k;
            q = p + (h * k2) / 2.f;
        } else if (st == 2) {
            k3 = k;
            q = p + h * k3;
        } else {
            k4 = k;
        }
    }
    const float c = EXACT ? sixth_exact(h) : h * (1.f / 6.f);
    return p + c * (((k1 + 2.f * k2) + 2.f * k3) + k4);
}

// Boundary classification (checkFlag, TraceBlineAdaptive.cu:309-331).
__device__ __forceinline__ int box_flag(const Dims& n, float3 p) {
    const float X = (float)(n.nx - 1), Y = (float)(n.ny - 1), Z = (float)(n.nz - 1);
    if ((p.x >= 0.f) & (p.y > 0.f) & (p.z >= 0.f) & (p.x <= X) & (p.y <= Y) & (p.z <= Z)) return 0;
    int f = 42;
    if ((p.x < 0.f) & (p.y >= 0.f) & (p.z >= 0.f) & (p.x < X) & (p.y < Y) & (p.z < Z)) f = 1;
    if ((p.x >= 0.f) & (p.y >= 0.f) & (p.z >= 0.f) & (p.x >= X) & (p.y < Y) & (p.z < Z)) f = 2;
    if ((p.x >= 0.f) & (p.y < 0.f) & (p.z >= 0.f) & (p.x < X) & (p.y < Y) & (p.z < Z)) f = 3;
    if ((p.x >= 0.f) & (p.y >= 0.f) & (p.z >= 0.f) & (p.x < X) & (p.y >= Y) & (p.z < Z)) f = 4;
    if ((p.x >= 0.f) & (p.y >= 0.f) & (p.z < 0.f) & (p.x < X) & (p.y < Y) & (p.z < Z)) f = 5;
    if ((p.x >= 0.f) & (p.y >= 0.f) & (p.z >= 0.f) & (p.x < X) & (p.y < Y) & (p.z >= Z)) f = 6;
    return f;
}

// ---------------------------------------------------------------------------
// Per-store geometry: the box tests, the length-limit scale, the kernel-start
// set-up and the view of the twist current density on the store's grid.
// ---------------------------------------------------------------------------
template <class F>
__device__ __forceinline__ bool box_inside(const F& f, float3 p) {
    return (p.x >= 0.f) & (p.y > 0.f) & (p.z >= 0.f) & (p.x <= (float)(f.d.nx - 1)) &
           (p.y <= (float)(f.d.ny - 1)) & (p.z <= (float)(f.d.nz - 1));
}
template <class F>
__device__ __forceinline__ int box_exit(const F& f, float3 p) {
    return box_flag(f.d, p);
}
// len_lim = len_ratio * this (the node counts' sum)
template <class F>
__device__ __forceinline__ double len_scale(const F& f) {
    return (double)(f.d.nx + f.d.ny + f.d.nz);
}
template <class F>
__device__ __forceinline__ void store_prepare(F&) {}
// Whether this launch's kernel does the work: always, except for the
// drop-in's two stretched kernels (search / uniform formula), of which only
// the one matching the caller's device flag runs.
template <class F>
__device__ __forceinline__ bool store_active(const F&) { return true; }
template <int M>
__device__ __forceinline__ bool store_active(const FieldStretchT<M>& f) {
    if constexpr (M == 4 || M == 5) {
        if (f.uni_dev) return (*f.uni_dev) == (M == 4);
    }
    return true;
}
// The current density shares the traced field's grid; J.cur carries only its
// three arrays, the geometry comes from the traced store (whose dims may have
// been read from the device at kernel start).
template <class F>
__device__ __forceinline__ FieldSoA current_view(const F& f, const FieldSoA& c) {
    return FieldSoA{c.bx, c.by, c.bz, f.d};
}

// Stretched grid (checkFlag, TraceBlineAdaptiveStretch.cu:309-331): the same
// tests against the first and last node coordinates.
template <int M>
__device__ __forceinline__ bool box_inside(const FieldStretchT<M>& f, float3 p) {
    return (p.x >= f.lo.x) & (p.y > f.lo.y) & (p.z >= f.lo.z) & (p.x <= f.hi.x) & (p.y <= f.hi.y) &
           (p.z <= f.hi.z);
}
template <int M>
__device__ __forceinline__ int box_exit(const FieldStretchT<M>& f, float3 p) {
    const float3 a = f.lo, b = f.hi;
    if ((p.x >= a.x) & (p.y > a.y) & (p.z >= a.z) & (p.x <= b.x) & (p.y <= b.y) & (p.z <= b.z)) return 0;
    int r = 42;
    if ((p.x < a.x) & (p.y >= a.y) & (p.z >= a.z) & (p.x < b.x) & (p.y < b.y) & (p.z < b.z)) r = 1;
    if ((p.x >= a.x) & (p.y >= a.y) & (p.z >= a.z) & (p.x >= b.x) & (p.y < b.y) & (p.z < b.z)) r = 2;
    if ((p.x >= a.x) & (p.y < a.y) & (p.z >= a.z) & (p.x < b.x) & (p.y < b.y) & (p.z < b.z)) r = 3;
    if ((p.x >= a.x) & (p.y >= a.y) & (p.z >= a.z) & (p.x < b.x) & (p.y >= b.y) & (p.z < b.z)) r = 4;
    if ((p.x >= a.x) & (p.y >= a.y) & (p.z < a.z) & (p.x < b.x) & (p.y < b.y) & (p.z < b.z)) r = 5;
    if ((p.x >= a.x) & (p.y >= a.y) & (p.z >= a.z) & (p.x < b.x) & (p.y < b.y) & (p.z >= b.z)) r = 6;
    return r;
}
// the summed coordinate extents, in float as the reference (:337-339)
template <int M>
__device__ __forceinline__ double len_scale(const FieldStretchT<M>& f) {
    return (double)(((f.hi.x + f.hi.y) + f.hi.z) - ((f.lo.x + f.lo.y) + f.lo.z));
}
template <int M>
__device__ __forceinline__ void store_prepare(FieldStretchT<M>& f) {
    // the packed stores' constants are formed on the host (qsl_trace_stretch)
    // in this same arithmetic and stay kernel parameters
    if constexpr (M == 1 || M == 2) return;
    f.lo = v3(__ldg(f.ax), __ldg(f.ay), __ldg(f.az));
    f.hi = v3(__ldg(f.ax + f.d.nx - 1), __ldg(f.ay + f.d.ny - 1), __ldg(f.az + f.d.nz - 1));
    // per-sample constants of the cell search, formed once (the FP64 pipe
    // is narrow on this GPU)
    f.clo = v3((float)((double)f.lo.x + 1e-6), (float)((double)f.lo.y + 1e-6), (float)((double)f.lo.z + 1e-6));
    f.chi = v3((float)((double)f.hi.x - 1e-6), (float)((double)f.hi.y - 1e-6), (float)((double)f.hi.z - 1e-6));
    f.us = v3((f.hi.x - f.lo.x) / __int2float_rd(f.d.nx), (f.hi.y - f.lo.y) / __int2float_rd(f.d.ny),
              (f.hi.z - f.lo.z) / __int2float_rd(f.d.nz));
    if constexpr (M == 1) {
        // the bin width of the search tables (only picks the bin; the
        // tables' ranges absorb its rounding)
        f.sbinv = v3((float)(STRETCH_BINS_PER_CELL * (f.d.nx - 1)) / (f.hi.x - f.lo.x),
                     (float)(STRETCH_BINS_PER_CELL * (f.d.ny - 1)) / (f.hi.y - f.lo.y),
                     (float)(STRETCH_BINS_PER_CELL * (f.d.nz - 1)) / (f.hi.z - f.lo.z));
    } else if constexpr (M == 4) {
        // the uniform formula's reciprocal spacing (fast arithmetic)
        f.sbinv = v3(1.f / f.us.x, 1.f / f.us.y, 1.f / f.us.z);
    }
}
// The current density is always the caller's arrays: a view of them on the
// store's grid that finds cells the way the store does (a packed store's
// tables or formula, else the drop-in's run-time choice).
template <int M>
__device__ __forceinline__ auto current_view(const FieldStretchT<M>& f, const FieldSoA& c) {
    FieldStretchT<M == 1 ? 3 : (M == 2 ? 4 : M)> r;
    r.bx = c.bx;
    r.by = c.by;
    r.bz = c.bz;
    r.d = f.d;
    r.ax = f.ax;
    r.ay = f.ay;
    r.az = f.az;
    r.uni_dev = nullptr;
    r.lo = f.lo;
    r.hi = f.hi;
    r.clo = f.clo;
    r.chi = f.chi;
    r.us = f.us;
    r.b4 = nullptr;
    r.srec = f.srec;
    r.sbin = f.sbin;
    r.sbinv = f.sbinv;
    return r;
}

// 2^x and log2 x by the hardware approximations (ex2/lg2.approx.ftz.f32):
// the fast step controller only needs the next step size to a few digits.
__device__ __forceinline__ float ex2_approx(float x) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float lg2_approx(float x) {
    float r;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// x^y correctly rounded to float: the double-precision power narrowed once
// (its error is far below half a float ulp except within ~2^-28 of a float
// rounding boundary).  The exact kernels use it so that the step controller's
// decisions do not depend on one library's powf rounding.
__device__ __forceinline__ float pow_cr(float x, float y) { return (float)pow((double)x, (double)y); }

// The exact step controller's power, (float)pow((double)x, (double)0.2f) of
// x = (float)((double)q / 11.09), q = tol / err.  The double form, kept out
// of line, costs ~100 operations of the FP64 pipe (two lanes per clock and
// SM); the float form below replaces it wherever the rounding is certain.
static __device__ __noinline__ float step_scale_double(float q) { return pow_cr((float)((double)q / 11.09), 0.2f); }

// x: q times 1 / 11.09 held as two floats (the pair is within 2^-47 of the
// quotient).  s = x^0.2f: 5 x 0.2f is 1 + 2^-26 exactly, so s^5 = x (1 +
// 2^-26 ln x) to 2^-45; two Newton steps on s^5 from the hardware log2 / exp2
// with the fifth power as a pair of floats, the last one kept apart from s as
// its correction (the pair is within 2^-45 of the power).  round_f2 rounds
// both; where it is not sure (one in 10^4), and for x outside
// [2^-20, 2^20] (a step grown 16 times, or cut far below rejection), the
// double form decides.
__device__ __forceinline__ float step_scale_exact(float q) {
    constexpr double r = 1.0 / 11.09;
    constexpr float rh = (float)r, rl = (float)(r - (double)(float)r);
    bool sure = (q >= 0x1p-16f) & (q <= 0x1p+23f);
    F2 xq;
    xq.h = q * rh;
    xq.l = __fmaf_rn(q, rl, __fmaf_rn(q, rh, -xq.h));
    const float x = round_f2(xq, sure);
    const float l2 = lg2_approx(x);
    const float xc = x * (l2 * (float)(0.6931471805599453 * 0x1p-26));
    float ri;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(ri) : "f"(x));
    ri = 0.2f * ri;
    F2 s = {ex2_approx(0.2f * l2), 0.f};
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        s.h = s.h + s.l;
        const float s2 = s.h * s.h, s2l = __fmaf_rn(s.h, s.h, -s2);
        const float s4 = s2 * s2, s4l = __fmaf_rn(2.f * s2, s2l, __fmaf_rn(s2, s2, -s4));
        const float s5 = s4 * s.h, s5l = __fmaf_rn(s4l, s.h, __fmaf_rn(s4, s.h, -s5));
        s.l = s.h * (((x - s5) + (xc - s5l)) * ri);
    }
    const float y = round_f2(s, sure);
    return sure ? y : step_scale_double(q);
}

// The smallest float not below 0.618: a float is below it exactly when its
// double is below 0.618.
constexpr float kAcceptScale = (double)0.618f >= 0.618 ? 0.618f : 0.618f + 0x1p-24f;

// J.B / |B|^2, the twist integrand.  The fast form fixes its rounding
// sequence with explicit multiply-adds: left as plain expressions, the
// compiler is free to fuse the products in an order that depends on the code
// around them, and two kernels tracing the same line would then differ in
// the last bit.  (The exact form is compiled without fusion.)
template <bool EXACT>
__device__ __forceinline__ float twist_density(float3 j, float3 b) {
    if (EXACT) return dot(j, b) / dot(b, b);
    const float jb = fmaf(j.z, b.z, fmaf(j.y, b.y, __fmul_rn(j.x, b.x)));
    const float bb = fmaf(b.z, b.z, fmaf(b.y, b.y, __fmul_rn(b.x, b.x)));
    return jb / bb;
}

// Per-lane state of one direction of one line.  The length accumulates in
// double for exact arithmetic (as the reference does) and in Kahan-
// compensated float otherwise (FP64 adds are slow on GB300).
template <bool EXACT>
struct Lane {
    typedef typename std::conditional<EXACT, double, float>::type len_t;
    float3 p;      // current point
    float3 pc;     // Kahan compensation of p (fast arithmetic)
    float h;       // current step
    float tol;     // local error tolerance (fast arithmetic: 0.2 log2(tol / 11.09), the controller's form)
    len_t len;     // accumulated length
    float lc;      // Kahan compensation of len (fast arithmetic); a float sum of the length (exact)
    double tw;     // accumulated twist
    // exact arithmetic: the last step's length and twist integrand, not yet
    // in len and tw (lane_pending)
    float pend_dl, pend_td;
    int steps;     // accepted steps
    int rej;       // trial steps rejected in a row
    unsigned dsign;  // sign bit of the step: 0 forward, 0x80000000 backward
    float3 out;    // footpoint of this direction when finished (the point past the face before lane_foot)
    int flag;      // reference flag; bits 8.. hold the qsl_line_status when finished
};

// Lane::flag of a direction that left the box, until lane_foot classifies it
constexpr int kLaneExit = 1 << 30;

// The reference flag and the qsl_line_status of a finished direction
// (packed into Lane::flag so that the status costs no register in the loop).
__device__ __forceinline__ int lane_flag(int packed) { return packed & 0xff; }
__device__ __forceinline__ int lane_status(int packed) { return packed >> 8; }
__device__ __forceinline__ int pack_flag(int flag, int status) { return flag | (status << 8); }

template <bool EXACT>
__device__ __forceinline__ void len_add(Lane<EXACT>& L, double x_exact, float x_fast) {
    if (EXACT) {
        L.len = L.len + x_exact;
    } else {
        const float y = x_fast - L.lc;
        const float t = (float)L.len + y;
        L.lc = (t - (float)L.len) - y;
        L.len = t;
    }
}

template <bool EXACT, class F>
__device__ __forceinline__ void lane_begin(const F& f, const TraceJob<F>& J, Lane<EXACT>& L, long long line, int dir,
                                           float s_len, float tol_coef, const float3 nrm, unsigned& ns) {
    L.dsign = dir > 0 ? 0u : 0x80000000u;
    L.p = v3(__ldg(J.inp_x + line), __ldg(J.inp_y + line), __ldg(J.inp_z + line));
    L.pc = v3(0.f, 0.f, 0.f);
    L.h = s_len;
    L.len = 0;
    L.lc = 0.f;
    L.tw = 0.0;
    L.pend_dl = 0.f;
    L.pend_td = 0.f;
    L.steps = 0;
    L.rej = 0;
    L.flag = 0;
    L.out = L.p;
    L.tol = 0.f;
    if (J.prm.integrator == QSL_RKF45) {
        // tolerance law (TraceBlineAdaptive.cu:351-359)
        const float3 b0 = sample<EXACT>(f, L.p, true);
        ns += 1;
        const float bn = fabsf(dot(b0, nrm));
        float tol;
        if (J.prm.tol_law == QSL_TOL_REFERENCE) {
            if ((double)bn <= 0.05) tol = (float)(J.prm.tol / 8e3);
            else tol = (float)(J.prm.tol * (double)(EXACT ? pow_cr(bn, 1.5f) : powf(bn, 1.5f)));
        } else {
            tol = (float)J.prm.tol;
        }
        L.tol = tol * tol_coef;
        // the fast controller's power (tol / (11.09 err))^0.2 as
        // 2^(0.2 log2(tol / 11.09) - 0.1 log2(err^2)): the first term once
        if (!EXACT) L.tol = 0.2f * log2f(L.tol * (float)(1.0 / 11.09));
    }
}

// a - b on the packed f32x2 pipe
__device__ __forceinline__ float2 fsub2(float2 a, float2 b) {
    float2 d;
    asm("{\n\t"
        ".reg .b64 ra, rb, rd;\n\t"
        "mov.b64 ra, {%2, %3};\n\t"
        "mov.b64 rb, {%4, %5};\n\t"
        "sub.rn.f32x2 rd, ra, rb;\n\t"
        "mov.b64 {%0, %1}, rd;\n\t"
        "}"
        : "=f"(d.x), "=f"(d.y)
        : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return d;
}

// The length limit; near: a float below which the float sum of the length
// settles the exact arithmetic's comparison.
template <bool EXACT>
struct LenLimit {
    typename Lane<EXACT>::len_t lim;
    float near;
};
constexpr int kNearSteps = 100000;  // the float sum is then within 0.6 %

// (double)td / 4 / pi in the reference's rounding: td / 4 is exact, the
// quotient by pi comes from its reciprocal and once more from the exact
// remainder (Markstein), that correction stretched and shrunk by 2^-20 to see
// whether it could round otherwise (then the division).
constexpr double kInvPi = 1.0 / kRefPi;
__device__ __forceinline__ double over_4pi(float td, double u, double v) {
    const bool sure = (u == v) & ((fabsf(td) >= 0x1p-100f) | (td == 0.f));
    return sure ? u : (double)td / 4.0 / kRefPi;
}

// The exact twist kernels' per-step sums in double, one step behind: the
// length's and the twist's FP64 operations (64 cycles each for a warp,
// dependent on one another) run between the next step's samples instead of
// on the way to it.  The same operations in the same order.  (Twist on 201 x
// 203 x 4 seeds, curl included, 2.87 -> 2.72 ms; the length alone, in the
// kernels without the twist, gains nothing: it is added at once.)
//
// The twist integrand at the step's start point comes out of the first
// stage: B is the sample before its normalisation, and the current density is
// summed with the same corner weights (two samples less per step: 2.73 ->
// 2.43 ms on the same planes).
template <class F>
struct Pending {
    const TraceJob<F>& J;
    Lane<true>& L;
    const bool tw_on;
    double d, t, q, m, u, v;
    float td;
    __device__ __forceinline__ void field(const F& f, int st, int3 cell, const float* w, float3 raw) {
        if (st == 0 && tw_on) {
            float3 c[8];
            if (J.cur_packed) J.cur_store.corners(cell.x, cell.y, cell.z, c);
            else current_view(f, J.cur).corners(cell.x, cell.y, cell.z, c);
            td = twist_density<true>(blend<true>(c, w), raw);
        }
    }
    __device__ __forceinline__ void operator()(int st) {
        if (st == 0) {
            d = (double)L.pend_dl;
            if (tw_on) t = (double)(0.25f * L.pend_td);
        } else if (st == 1) {
            L.len = L.len + d;
            if (tw_on) q = t * kInvPi;
        } else if (st == 2) {
            if (tw_on) m = __fma_rn(q, kRefPi, -t);  // (negated: a zero keeps its sign)
        } else if (st == 3) {
            if (tw_on) {
                u = __fma_rn(-m, kInvPi * (1.0 + 0x1p-20), q);
                v = __fma_rn(-m, kInvPi * (1.0 - 0x1p-20), q);
            }
        }
    }
    __device__ __forceinline__ void done() {
        if (tw_on) {
            L.tw = L.tw + over_4pi(L.pend_td, u, v) * d;
            L.pend_td = 0.f;
        }
        L.pend_dl = 0.f;
    }
};
// The pending step's sums at once; returns its twist increment.
template <bool TWIST>
__device__ __forceinline__ double lane_flush(Lane<true>& L, bool tw_on) {
    const double d = (double)L.pend_dl;
    L.len = L.len + d;
    L.pend_dl = 0.f;
    double dtw = 0.0;
    if (TWIST && tw_on) {
        dtw = (double)L.pend_td / 4.0 / kRefPi * d;
        L.tw = L.tw + dtw;
        L.pend_td = 0.f;
    }
    return dtw;
}

// The limits checked before a trial step: true (direction finished, L.out
// and L.flag set) when the length or step limit stops it.
template <bool EXACT, bool TWIST, class F>
__device__ __forceinline__ bool lane_limits(const TraceJob<F>& J, Lane<EXACT>& L, const LenLimit<EXACT>& limit,
                                            bool tw_on) {
    const bool more_steps = EXACT ? ((long long)L.steps < J.prm.max_steps) : (L.steps < J.lim.max_steps);
    bool more_len;
    if constexpr (EXACT) {
        // the double comparison, and the wait for the last step's sum, only
        // where the float sum does not settle it
        more_len = (L.lc < limit.near) & (L.steps < kNearSteps);
        if (!(more_len & more_steps)) {
            lane_flush<TWIST>(L, tw_on);
            more_len = L.len < limit.lim;
        }
    } else {
        more_len = L.len < limit.lim;
    }
    if (!(more_len & more_steps)) {
        L.out = L.p;
        L.flag = pack_flag(0, more_len ? QSL_LINE_MAX_STEPS : QSL_LINE_MAX_LENGTH);
        return true;
    }
    return false;
}

// the signed step: h with the direction's sign bit (h x +-1 exactly)
template <bool EXACT>
__device__ __forceinline__ float lane_hd(const Lane<EXACT>& L) {
    return __int_as_float(__float_as_int(L.h) ^ (int)L.dsign);
}

// The RKF45 step controller after a trial step with error estimate err (its
// norm in exact arithmetic, h^2 |e|^2 in fast): 0 = accepted (L.h is the
// next step), 1 = rejected (L.h shrunk; try again), 2 = rejected and the
// direction finished by the reject limit.
template <bool EXACT, class F>
__device__ __forceinline__ int lane_control(const TraceJob<F>& J, Lane<EXACT>& L, float err) {
    const qsl_trace_params& pr = J.prm;
    float scale;
    if (EXACT) {
        scale = step_scale_exact(L.tol / err);
        if (scale < kAcceptScale) {
            L.h = (float)((double)L.h * pr.reject_factor);
            if (pr.max_rejects > 0 && ++L.rej >= pr.max_rejects) {
                L.out = L.p;
                L.flag = pack_flag(0, QSL_LINE_REJECT_LIMIT);
                return 2;
            }
            return 1;
        }
    } else {
        // only the next step size depends on this power: hardware
        // log2 / exp2 are accurate enough (err is h^2 |e|^2 here, L.tol
        // 0.2 log2(tol / 11.09))
        scale = ex2_approx(fmaf(-0.1f, lg2_approx(err), L.tol));
        if (scale < 0.618f) {
            L.h = L.h * J.lim.reject;
            if (pr.max_rejects > 0 && ++L.rej >= pr.max_rejects) {
                L.out = L.p;
                L.flag = pack_flag(0, QSL_LINE_REJECT_LIMIT);
                return 2;
            }
            return 1;
        }
    }
    L.rej = 0;
    float h = L.h * scale;
    // (the same clamps in float, see StepLimits)
    if (h > J.lim.h_max) h = J.lim.h_max;  // a NaN step stays NaN
    if (h < J.lim.h_min) h = J.lim.h_min;
    L.h = h;
    return 0;
}

// The accepted step's move: the position update (Kahan-compensated in fast
// arithmetic), the length, the twist increment and the inside test.  True
// when the point left the box: L.p then stays the last point inside and
// L.out is the one outside (lane_foot finds the footpoint).
template <bool EXACT, bool TWIST, class F>
__device__ __forceinline__ bool lane_move(const F& f, const TraceJob<F>& J, Lane<EXACT>& L, float3 inc,
                                          float3 b_at_p, float td, bool tw_on, unsigned& ns) {
    // the twist integrand at the step's start point, before the position
    // update (fewer values live during the current density's sample)
    if (TWIST && tw_on) {
        if (EXACT) {
            ns += 2;
        } else {
            const float3 j1 =
                J.cur_packed ? sample<false>(J.cur_store, L.p, false) : sample<false>(current_view(f, J.cur), L.p, false);
            td = twist_density<false>(j1, b_at_p);
            ns += 1;
        }
    }
    float3 p2;
    float dl;
    if (EXACT) {
        p2 = L.p + inc;
        dl = norm(L.p - p2);
    } else {
        // Kahan-compensated position update: the rounding lost in p + inc is
        // carried into the next step, so long lines of short steps do not
        // drift by accumulated float rounding.  (x, y) on the packed pipe;
        // t = p2 - p, the increment as applied, also gives the step length.
        const float2 pxy = make_float2(L.p.x, L.p.y);
        const float2 yxy = fsub2(make_float2(inc.x, inc.y), make_float2(L.pc.x, L.pc.y));
        const float yz = inc.z - L.pc.z;
        const float2 qxy = __fadd2_rn(pxy, yxy);
        const float qz = L.p.z + yz;
        const float2 txy = fsub2(qxy, pxy);
        const float tz = qz - L.p.z;
        const float2 cxy = fsub2(txy, yxy);
        L.pc = v3(cxy.x, cxy.y, tz - yz);
        p2 = v3(qxy.x, qxy.y, qz);
        dl = norm_fast(v3(txy.x, txy.y, tz));
    }
    L.steps++;
    const bool left = !box_inside(f, p2);
    if constexpr (EXACT) {
        L.lc = L.lc + dl;
        L.pend_dl = dl;
        if (TWIST && tw_on) L.pend_td = td;
        if (!TWIST && !left) lane_flush<TWIST>(L, tw_on);
        if (left) {
            const double dtw = lane_flush<TWIST>(L, tw_on);
            L.len = L.len + -(double)dl;
            if (TWIST && tw_on) L.tw = L.tw - dtw;
        }
    } else {
        double dtw = 0.0;
        len_add(L, 0.0, dl);
        if (TWIST && tw_on) {
            dtw = (double)(td * dl * kInv4PiF);
            L.tw = L.tw + dtw;
        }
        if (left) {
            len_add(L, 0.0, -dl);
            if (TWIST && tw_on) L.tw = L.tw - dtw;
        }
    }
    if (left) {
        L.out = p2;
        L.flag = kLaneExit;
        return true;
    }
    L.p = p2;
    return false;
}

// One trial step of the current direction.  Returns true when the direction
// is finished (left the box, or stopped by the length / step / reject limit).
// Reference: TraceBlineAdap, TraceBlineAdaptive.cu:361-421 and TraceBline,
// TraceBline.cu:320-373.
template <bool EXACT, bool TWIST, class F>
__device__ __forceinline__ bool lane_step(const F& f, const TraceJob<F>& J, Lane<EXACT>& L,
                                          const LenLimit<EXACT>& limit, bool tw_on, unsigned& ns) {
    if (lane_limits<EXACT, TWIST>(J, L, limit, tw_on)) return true;
    const float hd = lane_hd(L);
    float3 inc;
    // fast twist kernels: B at L.p comes out of the step's first sample
    float3 b_at_p = v3(0.f, 0.f, 0.f);
    float3* const want_b = (!EXACT && TWIST && tw_on) ? &b_at_p : nullptr;
    auto step = [&](auto& aside) {
        float err = 0.f;
        if (J.prm.integrator == QSL_RKF45) inc = step_rkf45<EXACT>(f, L.p, hd, err, ns, want_b, aside);
        else inc = step_rk4<EXACT>(f, L.p, hd, ns, want_b, aside);
        return err;
    };
    float err;
    float td = 0.f;  // exact twist kernels: the twist integrand at L.p
    if constexpr (EXACT && TWIST) {
        Pending<F> pending{J, L, tw_on, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.f};
        err = step(pending);
        pending.done();
        td = pending.td;
    } else {
        Nothing nothing;
        err = step(nothing);
    }
    if (J.prm.integrator == QSL_RKF45) {
        const int c = lane_control(J, L, err);
        if (c != 0) return c == 2;
    }
    return lane_move<EXACT, TWIST>(f, J, L, inc, b_at_p, td, tw_on, ns);
}

// The footpoint of a finished direction: the exit face of a point that left
// the box and the line's crossing of it, with the length and twist of the
// exit segment (TraceBlineAdaptive.cu:380-418).  Sets L.out and L.flag
// (reference flag and qsl_line_status).  A limit's end has both already.
template <bool EXACT, bool TWIST, class F>
__device__ __forceinline__ void lane_foot(const F& f, const TraceJob<F>& J, Lane<EXACT>& L, bool tw_on,
                                          unsigned& ns) {
    if (L.flag != kLaneExit) return;
    const float3 p2 = L.out;
    const int flag = box_exit(f, p2);
    if (flag <= 6) {
        const int d = (flag - 1) / 2;
        const float q1 = comp(L.p, d), q2 = comp(p2, d);
        float qmid = q1;
        float3 b1 = v3(0.f, 0.f, 0.f);
        const bool far = (double)fabsf(q1 - q2) > 1e-3;
        if (far) {
            qmid = (flag % 2 == 1) ? 0.f : (float)f.d.n(d);
            const float3 u1 = sample_outlined<EXACT>(f, L.p, true);
            const float3 u2 = sample_outlined<EXACT>(f, p2, true);
            ns += 2;
            if (((double)fabsf(comp(u1, d)) < 0.2) | ((double)fabsf(comp(u2, d)) < 0.2)) {
                L.out.x = (L.p.x * (q2 - qmid) + p2.x * (qmid - q1)) / (q2 - q1);
                L.out.y = (L.p.y * (q2 - qmid) + p2.y * (qmid - q1)) / (q2 - q1);
                L.out.z = (L.p.z * (q2 - qmid) + p2.z * (qmid - q1)) / (q2 - q1);
            } else {
                L.out = step_rk4_normal<EXACT>(f, L.p, qmid - q1, d);
                ns += 4;
            }
            len_add(L, (double)fabsf(qmid - q1) / (1e-4 + (double)fabsf(comp(u1, d))),
                    fabsf(qmid - q1) / (1e-4f + fabsf(comp(u1, d))));
            b1 = u1;
        } else {
            L.out = L.p;
        }
        if (TWIST && tw_on && J.prm.boundary_twist) {
            // J and (on the face already) B at the exit step's start point
            const float3 j1 = J.cur_packed ? sample_outlined<EXACT>(J.cur_store, L.p, false)
                                           : sample_outlined<EXACT>(current_view(f, J.cur), L.p, false);
            if (!far) b1 = sample_outlined<EXACT>(f, L.p, false);
            L.tw = L.tw + (double)twist_density<EXACT>(j1, b1) / 4.0 / kRefPi * (double)fabsf(qmid - q1) /
                              (1e-4 + (double)fabsf(comp(b1, d)));
        }
    }
    const bool finite = isfinite(p2.x) & isfinite(p2.y) & isfinite(p2.z);
    L.flag = pack_flag(flag, flag <= 6 ? QSL_LINE_FACE : (finite ? QSL_LINE_EDGE : QSL_LINE_NAN));
}

// The second direction of a line: from the seed again with the first step
// size and the same tolerance (it depends on the seed alone).
template <bool EXACT, class F>
__device__ __forceinline__ void lane_turn(const TraceJob<F>& J, Lane<EXACT>& L, long long line, float s_len,
                                          unsigned& ns) {
    L.dsign = 0x80000000u;
    L.p = v3(__ldg(J.inp_x + line), __ldg(J.inp_y + line), __ldg(J.inp_z + line));
    L.pc = v3(0.f, 0.f, 0.f);
    L.h = s_len;
    L.len = 0;
    L.lc = 0.f;
    L.tw = 0.0;
    L.pend_dl = 0.f;
    L.pend_td = 0.f;
    L.steps = 0;
    L.rej = 0;
    if (J.prm.integrator == QSL_RKF45) ns += 1;  // the tolerance's sample counts for both directions
}

// What a finished direction leaves behind until its warp's other lanes are
// done (lane_foot and the outputs then run once for the whole warp): an
// array per lane, one row per direction.  Indexed by the direction it lives
// in local memory, which the stepping loop does not touch.
template <bool EXACT>
struct Stash {
    float p[3], q[3];
    int code;
    float lc;
    typename Lane<EXACT>::len_t len;
    double tw;
};
// (trace_queue's rows; kept apart so that other kernels' frames stay small)
template <bool EXACT>
struct QueueStash : Stash<EXACT> {
    long long line;  // the lane's line (of S[0])
};
template <bool EXACT, bool TWIST>
__device__ __forceinline__ void stash_put(Stash<EXACT>& S, const Lane<EXACT>& L) {
    S.p[0] = L.p.x; S.p[1] = L.p.y; S.p[2] = L.p.z;
    S.q[0] = L.out.x; S.q[1] = L.out.y; S.q[2] = L.out.z;
    S.code = L.flag;
    S.lc = L.lc;
    S.len = L.len;
    if (TWIST) S.tw = L.tw;
}
template <bool EXACT, bool TWIST>
__device__ __forceinline__ void stash_get(const Stash<EXACT>& S, Lane<EXACT>& L) {
    L.p = v3(S.p[0], S.p[1], S.p[2]);
    L.out = v3(S.q[0], S.q[1], S.q[2]);
    L.flag = S.code;
    L.lc = S.lc;
    L.len = S.len;
    if (TWIST) L.tw = S.tw;
}
// the two warps of a split pair wait for each other (64 threads, a barrier
// of their own).  The barrier's number is a constant on each side: a number
// from a register reserves all sixteen for the block, and the SM then holds
// four blocks.
__device__ __forceinline__ void pair_sync() {
    static_assert(kTraceThreads == 128, "two pairs of warps per block");
    __syncwarp();
    __threadfence_block();
    if (threadIdx.x < 64) asm volatile("bar.sync 1, 64;" ::: "memory");
    else asm volatile("bar.sync 2, 64;" ::: "memory");
}

// The end of a warp's lines, for all its lanes at once: the footpoints and
// samples of B of the directions in S and the outputs.
template <bool EXACT, bool TWIST, class F, class Rows>
__device__ __forceinline__ unsigned lines_finish(const F& f, const TraceJob<F>& J, const Rows* S, long long i,
                                         bool valid, bool split, float3 nrm, bool tw_on) {
    Lane<EXACT> L;
    unsigned ns = 0;
    const TraceOut& o = J.o;
    const bool back_only = split && ((threadIdx.x >> 5) & 1);
    double len = 0.0, tw = 0.0;
    if (valid) {
        const float3 p0 = v3(__ldg(J.inp_x + i), __ldg(J.inp_y + i), __ldg(J.inp_z + i));
#pragma unroll 1
        for (int dir = back_only ? 1 : 0; dir < (split && !back_only ? 1 : 2); ++dir) {
            stash_get<EXACT, TWIST>(S[dir], L);
            const bool fwd = dir == 0;
            lane_foot<EXACT, TWIST>(f, J, L, tw_on, ns);
            const float3 foot = L.out;
            const float3 b = sample_endpoint<EXACT>(f, foot);
            ns += 1;
            // the end footpoint's arrays forward, the start's backward
            (fwd ? o.end_x : o.start_x)[i] = foot.x;
            (fwd ? o.end_y : o.start_y)[i] = foot.y;
            (fwd ? o.end_z : o.start_z)[i] = foot.z;
            (fwd ? o.flag_end : o.flag_start)[i] = lane_flag(L.flag);
            int* const st = fwd ? o.status_end : o.status_start;
            if (st) st[i] = lane_status(L.flag);
            (fwd ? o.bend_x : o.bstart_x)[i] = b.x;
            (fwd ? o.bend_y : o.bstart_y)[i] = b.y;
            (fwd ? o.bend_z : o.bstart_z)[i] = b.z;
            len = (fwd | back_only) ? (double)L.len : len + (double)L.len;
            if (TWIST && tw_on) tw = (fwd | back_only) ? L.tw : tw + L.tw;
        }
        if (!split | back_only) {
            const float3 b0 = sample_endpoint<EXACT>(f, p0);
            ns += 1;
            o.bthis_x[i] = b0.x; o.bthis_y[i] = b0.y; o.bthis_z[i] = b0.z;
            // B nearly in the seed plane (TraceBlineAdaptive.cu:498-501)
            const float bn = b0.x * nrm.x + b0.y * nrm.y + b0.z * nrm.z;
            const float bm = sqrtf(b0.x * b0.x + b0.y * b0.y + b0.z * b0.z);
            o.b_flag[i] = ((double)fabsf(bn) * 100. < (double)bm) ? 1 : 0;
        }
    }
    if (split) {
        // the backward warp's length and twist through the output arrays
        if (valid & back_only) {
            o.line_len[i] = len;
            if (TWIST && tw_on) o.twist[i] = tw;
        }
        pair_sync();
        if (valid & !back_only) {
            len = len + __ldcg(o.line_len + i);
            if (TWIST && tw_on) tw = tw + __ldcg(o.twist + i);
        }
    }
    if (valid & !back_only) {
        o.line_len[i] = len;
        if (TWIST && tw_on) o.twist[i] = tw;
    }
    return ns;
}

// One line per lane of a warp, the lanes in lockstep: seed `i` of every lane
// that has one (`valid`), forward, then backward.  A lane whose direction
// ends goes on with its next one at once but leaves the footpoint, the
// samples of B and the outputs to the end, where the whole warp does them
// together: done as each lane ends, they ran for one or two lanes at a time
// (7-9 samples per direction, 32 times over).
//
// split: warps 2k and 2k + 1 of a block hold the same 32 lines, the first
// forward and the second backward, and the pair adds the two lengths (and
// twists) up at the end.  A line's directions depend on each other in
// nothing else, and a launch that leaves the GPU's warp slots half empty
// lasts as long as its longest line.
//
// The per-line scalars come from functors so that they are re-read where
// they are used rather than held in registers through the stepping loop.
template <bool EXACT, bool TWIST, class F, class SL, class TC, class NR>
__device__ __forceinline__ void trace_lines(const F& f, const TraceJob<F>& J, long long i, bool valid,
                                            bool split, const LenLimit<EXACT>& limit, const SL& s_len_of,
                                            const TC& tol_coef_of, const NR& nrm_of, bool tw_on, unsigned& ns) {
    Lane<EXACT> L;
    Stash<EXACT> S[2];
    if (valid) {
        lane_begin<EXACT>(f, J, L, i, split && ((threadIdx.x >> 5) & 1) ? -1 : 1, s_len_of(), tol_coef_of(), nrm_of(),
                          ns);
        while (true) {
            if (!lane_step<EXACT, TWIST>(f, J, L, limit, tw_on, ns)) continue;
            stash_put<EXACT, TWIST>(S[L.dsign >> 31], L);
            if (split | (L.dsign != 0)) break;
            lane_turn(J, L, i, s_len_of(), ns);
        }
    }
    __syncwarp();
    ns += lines_finish<EXACT, TWIST>(f, J, S, i, valid, split, nrm_of(), tw_on);
}

__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

// The work-queue schedule, for more lines than the grid has lanes: a warp
// takes lines from the device counter for all its lanes, traces them in
// lockstep, and takes new ones for the lanes whose lines have ended once too
// many wait.  The ended lines' footpoints, samples of B and outputs are done
// then, for all of them at once.
//
// When it refills: a partial refill costs the coherence of a warp of
// neighbours and does the ends for a part of its lanes, so it has to be
// worth that.  A warp whose seeds are neighbours (`neighbours`: a 1 /
// kNeighbours of the box's edges summed is 2-3 cells of a 64^3 box) waits for
// its last line: their lengths are alike, and what is left of such a warp
// costs little.  Others refill at kRefillLanes idle lanes; kRefillIdle looks,
// kRefillSteps trial steps apart, summed over the idle lanes (64 steps of the
// whole warp); and idle lane steps of a 1 / (1 + kRefillShare) part of all
// since the last refill.  200,000 lines, ms, one refill per line as it ends /
// none before the last line of 32 / this: a field whose lines are 3 % ropes of
// ten times the mean length, bricks 8.0 / 9.8 / 6.8, float4 7.6 / 11.2 / 7.3,
// drop-in RKF45 480 / 146 / 137; seeds anywhere in a charge field's volume
// 3.6 / 3.5 / 3.4, 4.9 / 5.1 / 4.7, 37 / 11.5 / 9.3; its bottom plane in
// random order 1.9 / 2.2 / 1.65.  Coherent, even planes (none / refills
// whatever the seeds / this): 258 x 258 x 32 seeds on bricks in tile order
// 13.77 / 13.85 / 13.80, drop-in twist on 201 x 203 x 4 seeds 3.05 / 3.15 /
// 3.07 and 2.83 / 2.92 / 2.84.
constexpr int kRefillSteps = 8;
constexpr int kRefillLanes = 16;
constexpr unsigned kRefillIdle = 256;
constexpr unsigned kRefillShare = 2;
constexpr float kNeighbours = 64.f;
// Whether a warp's seeds are neighbours: all but a quarter of them within
// `apart`, per axis, of the lane before.
__device__ __forceinline__ bool neighbours(float3 p, bool active, float apart) {
    const float3 d = p - v3(__shfl_up_sync(0xffffffffu, p.x, 1), __shfl_up_sync(0xffffffffu, p.y, 1),
                            __shfl_up_sync(0xffffffffu, p.z, 1));
    const bool far = active & (fmaxf(fmaxf(fabsf(d.x), fabsf(d.y)), fabsf(d.z)) > apart);
    return __popc(__ballot_sync(0xffffffffu, far)) <= 8;
}
template <bool EXACT, bool TWIST, class F, class N, class SL, class TC, class NR>
__device__ __forceinline__ void trace_queue(const F& f, const TraceJob<F>& J, const N& n_of,
                                            const LenLimit<EXACT>& limit, const SL& s_len_of, const TC& tol_coef_of,
                                            const NR& nrm_of, bool tw_on, unsigned& ns) {
    Lane<EXACT> L;
    QueueStash<EXACT> S[2];
    bool active = false, ended = false;
    // (warp-uniform) the counter is past the last line; the warp's seeds are neighbours
    bool drained = false, together = false;
    while (true) {
        if (__any_sync(0xffffffffu, ended)) {
            ns += lines_finish<EXACT, TWIST>(f, J, S, S[0].line, ended, false, nrm_of(), tw_on);
            ended = false;
            // a lane's sample count nears 32 bits: hand it over (exact while
            // one line takes fewer than 5e8 trial steps)
            if (ns > (1u << 30)) {
                if (J.samples) atomicAdd(J.samples, (unsigned long long)ns);
                ns = 0;
            }
        }
        unsigned want = __ballot_sync(0xffffffffu, !active);
        const bool fresh = want == 0xffffffffu;
        while (want != 0u && !drained) {
            // no more than the idle lanes: what a warp held back for later
            // (a chunk of 256) waited while others had nothing left
            int take = __popc(want);
            if (J.chunk > 0 && take > J.chunk) take = J.chunk;
            unsigned long long base = 0;
            if ((threadIdx.x & 31) == 0) base = atomicAdd(J.queue, (unsigned long long)take);
            const long long first = (long long)__shfl_sync(0xffffffffu, base, 0), n = n_of();
            drained = first + take >= n;
            const int rank = __popc(want & lanemask_lt());
            if (!active && rank < take && first + rank < n) {
                const long long i = J.order ? (long long)__ldg(J.order + first + rank) : first + rank;
                S[0].line = i;
                lane_begin<EXACT>(f, J, L, i, 1, s_len_of(), tol_coef_of(), nrm_of(), ns);
                active = true;
            }
            want = __ballot_sync(0xffffffffu, !active);
        }
        if (!__any_sync(0xffffffffu, active)) break;
        if (fresh) together = neighbours(L.p, active, (float)len_scale(f) * (1.f / kNeighbours));
        const bool wait = drained | together;
        int idle;
        unsigned busy_steps = 0, idle_steps = 0;
        do {
            for (int k = wait ? 0x7fffffff : kRefillSteps; active && k > 0; --k) {
                if (!lane_step<EXACT, TWIST>(f, J, L, limit, tw_on, ns)) continue;
                stash_put<EXACT, TWIST>(S[L.dsign >> 31], L);
                if (L.dsign == 0) {
                    lane_turn(J, L, S[0].line, s_len_of(), ns);
                } else {
                    active = false;
                    ended = true;
                }
            }
            idle = __popc(__ballot_sync(0xffffffffu, !active));
            idle_steps += idle;
            busy_steps += 32 - idle;
        } while (idle < 32 && (wait || idle < kRefillLanes || idle_steps < kRefillIdle ||
                               kRefillShare * idle_steps < busy_steps));
    }
}

// Lanes a line takes in a launch of n lines (or capacity for as many) on
// `warps` warps, the first of them active: the launch splits the directions
// over warp pairs where it has two lanes per line, and gives every line two
// or four lanes where it has as many more.  A warp of 8 lines waits less for
// its loads (each request touches fewer 128-byte lines, which the L1 serves
// one by one) and for its longest line: 100 x 100 seeds of a 64^3 box 0.246
// ms at 1, 0.238 at 2, 0.231 at 4 and at 8; RK4 drop-in on 128 x 128 seeds
// 3.52, 3.27, 3.25, 3.28.
constexpr int kMaxSpread = 4;
__host__ __device__ __forceinline__ bool splits(long long n, long long warps) { return 2 * n <= 32 * warps; }
__host__ __device__ __forceinline__ int spread_of(long long n, long long warps) {
    int s = 1;
    while (s < kMaxSpread && splits(2 * s * n, warps)) s *= 2;
    return s;
}

// How a launch of n lines on `warps` warps shares its lanes out.
struct LaunchShape {
    bool split;
    int spread;
};
__host__ __device__ __forceinline__ LaunchShape launch_shape(long long n, long long warps) {
    const bool split = splits(n, warps);
    return {split, split ? spread_of(n, warps) : 1};
}

// A queue launch with a lane for every line and more than three quarters of its
// lanes in use takes its warps' lines from the counter, in the order in which
// the warps come: a block's four warps then hold lines from four places, where
// by index they hold neighbours, which are long together.  Below that, lines by
// index fill whole blocks, which lie evenly over the SMs.  Drop-ins on 152 x 4
// blocks, ms, from the counter / by index: 98 % of the lanes 0.87 / 0.89 and
// 1.07 / 1.10 (stretched), 1.77 / 1.79 and 1.73 / 1.75 (RKF45), 96 % 0.92 /
// 0.96 and 1.04 / 1.13, 80 % 1.74 / 1.71 and 1.67 / 1.71, 66 % 1.66 / 1.58 and
// 1.66 / 1.59, 51 % 1.61 / 1.44 and 1.58 / 1.45.
__host__ __device__ __forceinline__ bool scattered(long long n, long long warps) { return 4 * n > 3 * 32 * warps; }
// (out of line: inlined, RK4 drop-ins, which never take it, 3.46 -> 3.50 ms)
static __device__ __noinline__ unsigned queue_turn(unsigned long long* queue) {
    unsigned turn = 0;
    if ((threadIdx.x & 31) == 0) turn = (unsigned)atomicAdd(queue, 1ull);
    return __shfl_sync(0xffffffffu, turn, 0);
}

// The tracer kernel.  QUEUE = true and more lines than the grid has lanes:
// warps take lines from the device counter J.queue (trace_queue).  Else every
// warp takes 32 lines at a time and traces them in lockstep, line = global
// thread index + k * total threads (the warp's index from the counter where
// `scattered` says so); a launch whose grid has two threads per line splits
// the directions over warp pairs (trace_lines).  Lines are visited in J.order
// when it is set.  TWIST compiles the twist integral in; it runs when the runtime
// flag is set.
template <bool EXACT, bool TWIST, bool QUEUE, class F>
__device__ __forceinline__ void trace_kernel_body(const TraceJob<F>& J) {
    F f = J.f;
    // only the drop-in stores (the caller's arrays) take their shape from the
    // device; the packed stores' dims stay kernel parameters
    if constexpr (std::is_same<F, FieldSoA>::value || std::is_same<F, FieldStretch>::value ||
                  std::is_same<F, FieldStretchU>::value) {
        if (J.shape_dev) {
            f.d.nx = __ldg(J.shape_dev);
            f.d.ny = __ldg(J.shape_dev + 1);
            f.d.nz = __ldg(J.shape_dev + 2);
        }
    }
    // a grid needs two nodes per axis for a trilinear cell (uniform exit)
    if (f.d.nx < 2 || f.d.ny < 2 || f.d.nz < 2) return;
    // Loop invariants that are used once per line are re-read at each use
    // (kernel parameters or one cached load) rather than held in registers:
    // registers set how many blocks stay resident, and the gathers need
    // every resident warp to hide their latency.
    auto s_len_of = [&J]() { return J.s.s_len_dev ? __ldg(J.s.s_len_dev) : J.s.s_len; };
    auto tol_coef_of = [&J]() { return J.s.tol_coef_dev ? __ldg(J.s.tol_coef_dev) : J.s.tol_coef; };
    auto nrm_of = [&J]() {
        return J.s.cross_dev ? v3(__ldg(J.s.cross_dev), __ldg(J.s.cross_dev + 1), __ldg(J.s.cross_dev + 2))
                             : v3(J.s.cross[0], J.s.cross[1], J.s.cross[2]);
    };
    auto n_of = [&J]() {
        const long long n = J.s.n_dev ? (long long)__ldg(J.s.n_dev) : J.s.n;
        return J.s.n_cap >= 0 && n > J.s.n_cap ? (long long)J.s.n_cap : n;
    };
    const bool tw_on = TWIST && (J.s.twist_flag_dev ? *J.s.twist_flag_dev : (J.s.twist_on != 0));
    if (!store_active(f)) return;
    store_prepare(f);
    // the packed stores' dims (and the stretched stores' coordinate
    // extents) are known on the host: their length limit is a kernel
    // parameter (a register would be re-formed from the double
    // product at every step once the loop runs short of registers)
    typename Lane<EXACT>::len_t len_lim;
    if constexpr (!EXACT && (std::is_same<F, FieldH4B>::value || std::is_same<F, FieldH4BW>::value ||
                             std::is_same<F, FieldF4>::value || std::is_same<F, FieldH8C>::value ||
                             std::is_same<F, FieldStretchP>::value || std::is_same<F, FieldStretchPU>::value))
        len_lim = J.lim.len_lim;
    else
        len_lim = (typename Lane<EXACT>::len_t)(J.prm.len_ratio * len_scale(f));
    const LenLimit<EXACT> limit{len_lim, 0.9f * (float)len_lim};
    unsigned ns = 0;
    const int lane_id = threadIdx.x & 31;
    const long long warps = (long long)gridDim.x * (blockDim.x / 32);
    // (launch_shape's values: a struct of them spills in the stretched kernels)
    const bool split = splits(n_of(), warps);
    const int spread = split ? spread_of(n_of(), warps) : 1;
    const int lines = 32 / spread;  // of a warp
    if (QUEUE && n_of() > 32 * warps) {
        trace_queue<EXACT, TWIST>(f, J, n_of, limit, s_len_of, tol_coef_of, nrm_of, tw_on, ns);
    } else {
        long long line = QUEUE && scattered(n_of(), warps)
                             ? (long long)queue_turn(J.queue)
                             : (long long)blockIdx.x * (blockDim.x / 32) + (threadIdx.x >> 5);
        for (line = (split ? line >> 1 : line) * lines; line < n_of(); line += warps * lines / (split ? 2 : 1)) {
            const long long slot = line + lane_id / spread;
            const bool valid = lane_id % spread == 0 && slot < n_of();
            const long long i = (valid && J.order) ? (long long)__ldg(J.order + slot) : slot;
            trace_lines<EXACT, TWIST>(f, J, i, valid, split, limit, s_len_of, tol_coef_of, nrm_of, tw_on, ns);
            if (ns > (1u << 30)) {  // (as in trace_queue)
                if (J.samples) atomicAdd(J.samples, (unsigned long long)ns);
                ns = 0;
            }
        }
    }
    if (J.samples) {
        // one atomic per warp (blocks are whole warps; every lane gets here)
        __syncwarp();
        unsigned long long v = ns;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
        if (lane_id == 0) atomicAdd(J.samples, v);
    }
}

}  // namespace qsl
