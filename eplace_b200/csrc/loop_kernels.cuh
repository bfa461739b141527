// loop_kernels.cuh -- the per-iteration kernels of the ePlace inner loop.
//
//   scatter   cell/filler -> bin overlap areas as int64 fixed point with
//             atomics: order-independent, so the maps are bit-exact and
//             deterministic (EPlacer_2D::binNodeDensityUpdate,
//             EPlace/eplace.cpp:1029-1133)
//   prep      fixed point -> bin density for the Poisson solve, overflow tau
//             in FP64, the 1/gamma schedule (EPlace/eplace.cpp:438-500,
//             570-580)
//   wirelength  per-net bound pins + HPWL (FP64), WA / LSE exponentials and
//             per-pin gradients (PlaceCommon/objects.cpp:75-144,161-241,
//             248-437); the lambda update owed by the previous step
//             (EPlace/eplace.cpp:846-883)
//   combine   field gather (EPlace/eplace.cpp:599-674), per-object sum of its
//             pin gradients in pin order (:531-549), preconditioned direction
//             (:698-737), FP64 Lipschitz sums and the step / a_k update
//             (Optimization/optutils.hpp:20-35, nesterov.hpp:375-415)
//   update    x_{k+1} = y_k + s g_k, y_{k+1} = x_{k+1} + (a_k-1)/a_{k+1}
//             (x_{k+1}-x_k), clamp into the core (PlaceDB/placedb.cpp:253-288)
//
// Every kernel of the loop returns at once when S->done is set, so a captured
// multi-iteration graph stops doing work after the stop condition.  Each is a
// template on the working precision R (float: the engine's mixed-precision
// form, whose arithmetic follows the reference's float steps; double: the
// plain FP64 form), instantiated in a file of its own for each (loop.h).
#pragma once
#include <algorithm>
#include <cmath>
#include <vector>

#include "loop.h"
#include "scatter.cuh"

namespace ep {

namespace {

constexpr int kPinChunk = 128;  // pin gradients a warp of the combine kernel stages per round

__device__ __forceinline__ float exact_exp(float a) { return expf(a); }
__device__ __forceinline__ double exact_exp(double a) { return exp(a); }
__device__ __forceinline__ float warp_sum_r(float v) { return warp_sum_f(v); }
__device__ __forceinline__ double warp_sum_r(double v) { return warp_sum(v); }

// ---------------------------------------------------------------- scatter --
// Rectangle and contribution scale of an object: sx*sy, times the target
// density for macros (EPlace/eplace.cpp:1114-1128, evaluated left to right).
// In FP32 sx*sy is the static table's value, the same float operations.
template <typename R>
__device__ __forceinline__ RectT<R> scatter_rect(const Grid &g, vec2<R> p, float2 s, float sxy_table, uint8_t f,
                                                 R &scale) {
    const RectT<R> r = object_rect(g, p.x, p.y, (R)s.x, (R)s.y);
    if constexpr (sizeof(R) == 4)
        scale = sxy_table;
    else
        scale = mul_rn(r.sx, r.sy);
    if (f & kMacro) scale = mul_rn(scale, (R)g.td);
    return r;
}

// The objects of a warp, one a lane (valid false: none); every lane calls it.
// The filler map lies behind the node map.
template <typename R>
__device__ __forceinline__ void scatter_objects(const Grid &g, bool valid, vec2<R> p, float2 s, float sxy_table,
                                                uint8_t f, double qscale, ull *__restrict__ maps) {
    R scale;
    const RectT<R> r = scatter_rect<R>(g, p, s, sxy_table, f, scale);
    int i0, i1, j0, j1;
    bin_range<R>(g, r, i0, i1, j0, j1);
    if (!valid) i1 = i0 - 1;
    const unsigned bin = (unsigned)(i0 * g.ny + j0) + ((f & kFiller) ? (unsigned)(g.nx * g.ny) : 0u);
    scatter_by_lane<R>(g, r, scale, i0, i1, j0, j1, qscale, bin, maps);
}

// One kBig object by `count` threads of which this is the rank-th.
template <typename R>
__device__ __forceinline__ void scatter_big(const Grid &g, vec2<R> p, float2 s, float sxy_table, uint8_t f,
                                            double qscale, int rank, int count, ull *__restrict__ maps) {
    R scale;
    const RectT<R> r = scatter_rect<R>(g, p, s, sxy_table, f, scale);
    int i0, i1, j0, j1;
    bin_range<R>(g, r, i0, i1, j0, j1);
    scatter_by_group<R>(g, r, scale, i0, i1, j0, j1, qscale, rank, count,
                        maps + ((f & kFiller) ? (size_t)g.nx * g.ny : 0));
}

// Work of the object kernels: blocks [0, big_blocks) take the kBig objects (a
// block each for the first n_huge, then a warp each; they start first), the
// blocks after them a thread per object.  o = n_obj: nothing.
struct ObjectUnit {
    int o;
    int rank, count;  // this thread among the threads of the object
};
__device__ __forceinline__ ObjectUnit object_unit(const DeviceNetlist &d, int big_blocks) {
    const int b = blockIdx.x, t = threadIdx.x;
    if (b >= big_blocks) return ObjectUnit{min((int)((b - big_blocks) * blockDim.x + t), d.n_obj), 0, 1};
    if (b < d.n_huge_objs) return ObjectUnit{d.big_objs[b], t, kThreads};
    const int slot = d.n_huge_objs + (b - d.n_huge_objs) * (kThreads / 32) + (t >> 5);
    return ObjectUnit{slot < d.n_big_objs ? d.big_objs[slot] : d.n_obj, t & 31, 32};
}

template <typename R>
__global__ void __launch_bounds__(kThreads)
k_scatter(Grid g, DeviceNetlist d, int big_blocks, double qscale, ull *__restrict__ maps,
          const DevScalars *__restrict__ S) {
    const ObjectUnit u = object_unit(d, big_blocks);
    bool valid = u.o < d.n_obj;
    const uint8_t f = valid ? d.flags[u.o] : 0;
    const float2 s = valid ? d.size[u.o] : make_float2(1.f, 1.f);
    const float sxy = valid ? d.sxy[u.o] : 0.f;
    pdl_begin();
    if (S->done) return;
    const vec2<R> p = valid ? ((const vec2<R> *)d.pos)[u.o] : mk2<R>((R)g.llx, (R)g.lly);
    if (u.count == 1)
        scatter_objects<R>(g, valid && !(f & kBig), p, s, sxy, f, qscale, maps);
    else if (valid)
        scatter_big<R>(g, p, s, sxy, f, qscale, u.rank, u.count, maps);
}

// ------------------------------------------------------------------- prep --
// 1/gamma of wirelengthGradientUpdate (EPlace/eplace.cpp:475-500), in the
// reference's float sequence: 0.125f / binStep, then the tau-dependent factor.
__device__ __forceinline__ void inv_gamma(double tau_d, float sx, float sy, double &gx, double &gy) {
    float tau = (float)tau_d;
    float bx = __fdiv_rn(0.125f, sx), by = __fdiv_rn(0.125f, sy);
    if (tau > 1.0f) {
        bx = (float)((double)bx * 0.1);
        by = (float)((double)by * 0.1);
    } else if (tau < 0.1f) {
        bx = (float)((double)bx * 10.0);
        by = (float)((double)by * 10.0);
    } else {
        float t = (float)(1.0 / pow(10.0, ((double)tau - 0.1) * 20 / 9.0 - 1.0));
        bx = __fmul_rn(bx, t);
        by = __fmul_rn(by, t);
    }
    gx = bx;
    gy = by;
}

template <typename R>
__global__ void __launch_bounds__(kThreads)
k_prep(Grid g, ull *__restrict__ node_q, ull *__restrict__ filler_q, const float2 *__restrict__ stat,
       R *__restrict__ rho, uint16_t *__restrict__ rho_hi, uint16_t *__restrict__ rho_lo, float *__restrict__ node_f,
       float *__restrict__ filler_f, int zero, double inv_q, double inv_bin_area, double bin_area, double area_norm,
       double *__restrict__ partials, DevScalars *__restrict__ S) {
    pdl_begin();
    __shared__ double sh[32];
    // tested behind the first bin's loads, one round trip for both: a step at 200k
    // cells 55.6 -> 55.25 us, at 1M the same
    const int done = S->done;
    int nb = g.nx * g.ny;
    double acc[1] = {0.0};
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < nb; k += gridDim.x * blockDim.x) {
        const ull nq = node_q[k], fq = filler_q[k];
        float2 st = stat[k];  // (terminal, base)
        if (done) break;
        double node = (double)(long long)nq * inv_q;
        double fill = (double)(long long)fq * inv_q;
        // eDensity = node + base + filler + terminal (EPlace/eplace.cpp:576-577)
        double dens = (node + (double)st.y + fill + (double)st.x) * inv_bin_area;
        R d = (R)dens;
        if (rho) rho[k] = d;
        if (rho_hi) {
            // 3xBF16 operand split (FP32 path only): hi = bf16(d), lo = bf16(d - hi)
            const float df = (float)d;
            uint32_t u = __float_as_uint(df);
            uint32_t r = u + 0x7fffu + ((u >> 16) & 1u);
            uint16_t h = (uint16_t)(r >> 16);
            float hf = __uint_as_float((uint32_t)h << 16);
            float rem = df - hf;
            uint32_t u2 = __float_as_uint(rem);
            uint32_t r2 = u2 + 0x7fffu + ((u2 >> 16) & 1u);
            rho_hi[k] = h;
            rho_lo[k] = (uint16_t)(r2 >> 16);
        }
        // overflow counts nodes, terminals and base, not fillers (:438-453)
        double ov = (node + (double)st.x + (double)st.y) * inv_bin_area - (double)g.td;
        if (ov > 0.0) acc[0] += ov * bin_area;
        if (node_f) {
            node_f[k] = (float)node;
            filler_f[k] = (float)fill;
        }
        if (zero) {
            node_q[k] = 0ull;
            filler_q[k] = 0ull;
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) S->step_done = done;
    if (done) return;
    if (!grid_arrive<1>(acc, sh, partials, &S->cnt_prep, gridDim.x, blockIdx.x)) return;
    const int status = S->status;
    grid_total<1>(acc, sh, partials, &S->cnt_prep, gridDim.x);
    if (threadIdx.x == 0) {
        const double tau = acc[0] / area_norm;
        S->tau = tau;
        if (!isfinite(tau)) S->status = status | 1 << EP_ERR_NAN;
        double gx, gy;
        inv_gamma(tau, g.sx, g.sy, gx, gy);
        S->inv_gamma_x = gx;
        S->inv_gamma_y = gy;
    }
}

// ------------------------------------------------------------- wirelength --
template <typename R>
struct PinCtx {
    const int32_t *__restrict__ owner;
    const float2 *__restrict__ off;
    const vec2<R> *__restrict__ pos;
    const int32_t *__restrict__ slot;  // device pin -> object-major gradient slot (-1: terminal)
};

// Pin::calculateAbsolutePos: centre + offset.
template <typename R>
__device__ __forceinline__ vec2<R> pin_xy(const PinCtx<R> &c, int p) {
    float2 o = c.off[p];
    vec2<R> q = c.pos[c.owner[p]];
    return mk2<R>(add_rn(q.x, (R)o.x), add_rn(q.y, (R)o.y));
}

template <typename R>
struct NetSums {
    R nmx, dmx, nnx, dnx, nmy, dmy, nny, dny;
};

// Exponential terms of one pin (calcWirelengthWA_2D, objects.cpp:275-332):
// arguments <= -300 make the term zero.
template <typename R>
struct PinExp {
    R emx, enx, emy, eny;
};

template <bool EXACT, typename R>
__device__ __forceinline__ R term_exp(R a) {
    if (!(a > (R)kNegMaxExp)) return (R)0;
    return EXACT ? exact_exp(a) : fast_exp<R>(a);
}

template <bool EXACT, typename R>
__device__ __forceinline__ PinExp<R> pin_exps(vec2<R> xy, R x1, R x0, R y1, R y0, R igx, R igy) {
    PinExp<R> e;
    e.emx = term_exp<EXACT, R>(mul_rn(sub_rn(xy.x, x1), igx));
    e.enx = term_exp<EXACT, R>(mul_rn(sub_rn(x0, xy.x), igx));
    e.emy = term_exp<EXACT, R>(mul_rn(sub_rn(xy.y, y1), igy));
    e.eny = term_exp<EXACT, R>(mul_rn(sub_rn(y0, xy.y), igy));
    return e;
}

// Add one pin's terms to a running sum set (calcWirelengthWA_2D's sums).
template <typename R>
__device__ __forceinline__ void add_terms(R (&s)[8], const PinExp<R> &e, vec2<R> xy) {
    s[0] = add_rn(s[0], mul_rn(xy.x, e.emx));
    s[1] = add_rn(s[1], e.emx);
    s[2] = add_rn(s[2], mul_rn(xy.x, e.enx));
    s[3] = add_rn(s[3], e.enx);
    s[4] = add_rn(s[4], mul_rn(xy.y, e.emy));
    s[5] = add_rn(s[5], e.emy);
    s[6] = add_rn(s[6], mul_rn(xy.y, e.eny));
    s[7] = add_rn(s[7], e.eny);
}

// Per-net factors of the gradient: 1 / (sum of exponentials) of each of the
// four terms, and the weighted sums whose quotients are the weighted mean
// coordinates.  Every denominator holds the bound pin's exp(0) = 1, so it is
// >= 1.
template <typename R>
struct NetCoef {
    R rmx, nmx, rnx, nnx, rmy, nmy, rny, nny;
};

template <typename R>
__device__ __forceinline__ NetCoef<R> net_coef(const NetSums<R> &s) {
    return NetCoef<R>{rcp_rn(s.dmx), s.nmx, rcp_rn(s.dnx), s.nnx, rcp_rn(s.dmy), s.nmy, rcp_rn(s.dny), s.nny};
}

// Per-pin gradient of the WA model (objects.cpp:359-415).  The reference's
// (nd * d - dd * n) / d^2 equals e / d * (1 + (x - n / d) / gamma) for the max
// term and e / d * (1 - (x - n / d) / gamma) for the min term; this form
// subtracts the weighted mean from the coordinate before scaling, which
// avoids the cancellation of the expanded quotient (the two agree to the
// reference's own rounding).  A zero exponential (argument <= -300) gives a
// zero term as in the reference.  LSE (:423-437): e / d per term.  Every
// contraction is written out, so that each form of the pass rounds alike.
template <bool LSE, typename R>
__device__ __forceinline__ R axis_gradient(R em, R en, R x, R ig, R rm, R nm, R rn, R nn) {
    const R am = mul_rn(em, rm), an = mul_rn(en, rn);
    if (LSE) return fma_r(em, rm, -an);
    const R fm = fma_r(ig, fma_r(-nm, rm, x), (R)1), fn = fma_r(-ig, fma_r(-nn, rn, x), (R)1);
    return fma_r(am, fm, -mul_rn(an, fn));
}
template <bool LSE, typename R>
__device__ __forceinline__ vec2<R> pin_gradient(const PinExp<R> &e, vec2<R> xy, R igx, R igy, const NetCoef<R> &c) {
    return mk2<R>(axis_gradient<LSE, R>(e.emx, e.enx, xy.x, igx, c.rmx, c.nmx, c.rnx, c.nnx),
                  axis_gradient<LSE, R>(e.emy, e.eny, xy.y, igy, c.rmy, c.nmy, c.rny, c.nny));
}

template <typename R>
__device__ __forceinline__ double net_value(const NetSums<R> &s, R x1, R x0, R y1, R y0, R igx, R igy, bool lse) {
    if (lse)
        return ((double)x1 - x0 + log((double)s.dmx) / igx + log((double)s.dnx) / igx) +
               ((double)y1 - y0 + log((double)s.dmy) / igy + log((double)s.dny) / igy);
    return ((double)s.nmx / s.dmx - (double)s.nnx / s.dnx) + ((double)s.nmy / s.dmy - (double)s.nny / s.dny);
}

// lambda multiplier of updatePenaltyFactor (EPlace/eplace.cpp:849-871).
__device__ __forceinline__ double lambda_multiplier(double cur, double last) {
    double delta = cur - last;
    double m = delta < 0.0 ? 1.05 : pow(1.05, -delta / 350000.0 + 1.0);
    return fmin(fmax(m, 0.95), 1.05);
}

// The scalars that the HPWL finalisers read, loaded ahead of them.
struct HpwlScalars {
    double lambda, last_hpwl;
    int lambda_pending, lambda0_mode;
};
__device__ __forceinline__ HpwlScalars load_hpwl_scalars(const DevScalars *S) {
    return HpwlScalars{S->lambda, S->last_hpwl, S->lambda_pending, S->lambda0_mode};
}

// HPWL finaliser of the wirelength pass.
__device__ __forceinline__ void finish_wirelength(DevScalars *S, const HpwlScalars &h, double hp, double wl) {
    S->wirelength = wl;
    S->hpwl = hp;
    // atomic: the Poisson solve, running beside this pass, may raise a bit too
    if (!isfinite(hp)) atomicOr(&S->status, 1 << EP_ERR_NAN);
    if (h.lambda_pending) {
        S->lambda = h.lambda * lambda_multiplier(hp, h.last_hpwl);
        S->lambda_pending = 0;
    }
    // updatePenaltyFactor's, or penaltyFactorInitilization's lastHPWL = calcHPWL()
    if (h.lambda_pending || h.lambda0_mode) S->last_hpwl = hp;
}

// Finaliser of the HPWL-only pass (PlaceDB::calcHPWL): mode 0 stores it,
// mode 1 applies updatePenaltyFactor, mode 2 applies it only if one is owed.
__device__ __forceinline__ void finish_hpwl(DevScalars *S, const HpwlScalars &h, double hp, int mode) {
    S->hpwl_query = hp;
    if (mode == 1 || (mode == 2 && h.lambda_pending)) {
        S->lambda = h.lambda * lambda_multiplier(hp, h.last_hpwl);
        S->last_hpwl = hp;
        S->lambda_pending = 0;
    }
}

// ---- the per-net pass ---------------------------------------------------------
// On the device the nets are ordered by degree, largest first, and cut into
// tasks (degree D, first pin, nets, m), each run by one unit:
//   D >  kBlockPins: one net, a whole block (net_in_block);
//   D >  kWarpPins:  one net, a warp striding over its pins (net_in_warp);
//   D >  kThreadPins: floor(32 / D) nets on the lanes of a warp, one pin per
//       lane (nets_in_warp; s = lane * m >> 16, m = ceil(2^16 / D), exact for
//       lanes < 32), segmented shuffle reductions over the lanes;
//   D <= kThreadPins: 32 nets, a thread each (nets_by_thread): no shuffles, and
//       D position loads of a lane in flight at once.
// The long tasks start first.  The pass is bound by the latency of its
// dependent loads (pin -> owner -> centre), so the split follows the loads in
// flight: a 500-pin net on one warp was a chain of 16 rounds in each of three
// sweeps that the whole pass waited for, and one pin per lane left a warp with
// one load in flight and 450 instructions of shuffle trees.
// The sums are in the working precision as in Net::calcWirelengthWA_2D (float
// there), added in one fixed order per degree, the same in every form: the
// lane form's trees below, and for D > kWarpPins lane l adds pins l, l + 32,
// ... and an xor tree adds the lanes.  Pin gradients go to their object-major
// slots.  Within a degree the nets follow their lowest owner, so that a warp's
// centres and slots share sectors (1M cells: 84 -> 79 us).  The split of the
// work and six blocks an SM (40 registers; four in FP64) took the pass from
// 26.1 to 17.7 us at 200k cells, 112 to 75 at 1M, 17.4 to 8.6 at 30k (FP32),
// 36.9 to 26.2 at 200k (FP64), with bitwise the same gradients.  WL = false
// computes only the HPWL with the same layout and reduction tree, so both
// passes give bitwise the same HPWL.
struct NetOut {
    double hpwl, value;
};

constexpr unsigned kFull = 0xffffffffu;

// Bound pins of each aligned segment of D lanes (segment base `base`, this
// lane's index k in it); every lane of the segment gets them.  The windows
// double cyclically, which is exact for max / min.
template <typename R>
__device__ __forceinline__ void seg_bounds(R &x1, R &x0, R &y1, R &y0, int D, int base, int k) {
    for (int o = 1; o < D; o <<= 1) {
        const int j = k + o;
        const int src = base + (j < D ? j : j - D);
        x1 = max_r(x1, __shfl_sync(kFull, x1, src));
        x0 = min_r(x0, __shfl_sync(kFull, x0, src));
        y1 = max_r(y1, __shfl_sync(kFull, y1, src));
        y0 = min_r(y0, __shfl_sync(kFull, y0, src));
    }
}

// The eight exponential sums of each segment, every lane of the segment gets
// bitwise the same totals: a butterfly when D is a power of two, else a tree
// into the segment's first lane and a broadcast.
template <typename R>
__device__ __forceinline__ void seg_sums(R (&s)[8], int D, int base, int k) {
    if ((D & (D - 1)) == 0) {
        for (int o = D >> 1; o > 0; o >>= 1)
#pragma unroll
            for (int i = 0; i < 8; i++) s[i] = add_rn(s[i], __shfl_xor_sync(kFull, s[i], o));
        return;
    }
    for (int o = 1; o < D; o <<= 1) {
        const bool take = k + o < D;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const R t = __shfl_down_sync(kFull, s[i], o);
            if (take) s[i] = add_rn(s[i], t);
        }
    }
#pragma unroll
    for (int i = 0; i < 8; i++) s[i] = __shfl_sync(kFull, s[i], base);
}

template <typename R>
__device__ __forceinline__ NetSums<R> net_sums(const R (&s)[8]) {
    return NetSums<R>{s[0], s[1], s[2], s[3], s[4], s[5], s[6], s[7]};
}

// Nets of degree D <= 32 packed on the lanes of one warp.
template <bool WL, bool EXACT, bool LSE, typename R>
__device__ __forceinline__ NetOut nets_in_warp(const int4 t, int lane, const PinCtx<R> &pc, vec2<R> *__restrict__ out,
                                               R igx, R igy, int want_value) {
    const int D = t.x, p0 = t.y;
    const int seg = (lane * t.w) >> 16, base = seg * D, k = lane - base;
    const bool act = seg < t.z;
    const vec2<R> xy = act ? pin_xy<R>(pc, p0 + lane) : mk2<R>((R)0, (R)0);
    // bound pins (Net::calcBoundPin, PlaceCommon/objects.cpp:75-144)
    R x1 = xy.x, x0 = xy.x, y1 = xy.y, y0 = xy.y;
    seg_bounds<R>(x1, x0, y1, y0, D, base, k);
    NetOut r{0.0, 0.0};
    if (act && k == 0) r.hpwl = ((double)x1 - (double)x0) + ((double)y1 - (double)y0);
    if (WL) {
        const PinExp<R> e = pin_exps<EXACT, R>(xy, x1, x0, y1, y0, igx, igy);
        R s[8] = {mul_rn(xy.x, e.emx), e.emx, mul_rn(xy.x, e.enx), e.enx,
                  mul_rn(xy.y, e.emy), e.emy, mul_rn(xy.y, e.eny), e.eny};
        seg_sums<R>(s, D, base, k);
        const NetSums<R> ns = net_sums<R>(s);
        const int sl = act ? pc.slot[p0 + lane] : -1;
        if (sl >= 0) out[sl] = pin_gradient<LSE, R>(e, xy, igx, igy, net_coef<R>(ns));
        if (want_value && act && k == 0) r.value = net_value<R>(ns, x1, x0, y1, y0, igx, igy, LSE);
    }
    return r;
}

// Sum of v[0..D-1] in the order of seg_sums: halves for a power of two, else
// pairs of neighbours, level by level.
template <int D, typename R>
__device__ __forceinline__ R tree_sum(const R (&v)[D]) {
    R t[D];
#pragma unroll
    for (int k = 0; k < D; k++) t[k] = v[k];
    if constexpr ((D & (D - 1)) == 0) {
#pragma unroll
        for (int o = D >> 1; o > 0; o >>= 1)
#pragma unroll
            for (int k = 0; k < o; k++) t[k] = add_rn(t[k], t[k + o]);
    } else {
#pragma unroll
        for (int o = 1; o < D; o <<= 1)
#pragma unroll
            for (int k = 0; k + o < D; k += 2 * o) t[k] = add_rn(t[k], t[k + o]);
    }
    return t[0];
}

// One axis of a net held by a thread: coordinates x, bounds x1 and x0; the
// gradient of each pin along the axis.
template <int D, bool EXACT, bool LSE, typename R>
__device__ __forceinline__ void net_axis(const R (&x)[D], R x1, R x0, R ig, R (&grad)[D], R &nm, R &dm, R &nn, R &dn) {
    R em[D], en[D], v[D];
#pragma unroll
    for (int k = 0; k < D; k++) {
        em[k] = term_exp<EXACT, R>(mul_rn(sub_rn(x[k], x1), ig));
        en[k] = term_exp<EXACT, R>(mul_rn(sub_rn(x0, x[k]), ig));
        v[k] = mul_rn(x[k], em[k]);
    }
    nm = tree_sum<D, R>(v);
    dm = tree_sum<D, R>(em);
#pragma unroll
    for (int k = 0; k < D; k++) v[k] = mul_rn(x[k], en[k]);
    nn = tree_sum<D, R>(v);
    dn = tree_sum<D, R>(en);
    const R rm = rcp_rn(dm), rn = rcp_rn(dn);
#pragma unroll
    for (int k = 0; k < D; k++) grad[k] = axis_gradient<LSE, R>(em[k], en[k], x[k], ig, rm, nm, rn, nn);
}

// 32 nets of D <= kThreadPins pins, a thread each; one axis after the other,
// so that only one axis's exponentials are held.
template <int D, bool WL, bool EXACT, bool LSE, typename R>
__device__ __forceinline__ NetOut nets_by_thread(const int4 t, int lane, const PinCtx<R> &pc,
                                                 vec2<R> *__restrict__ out, R igx, R igy, int want_value) {
    NetOut r{0.0, 0.0};
    if (lane >= t.z) return r;
    const int p = t.y + lane * D;
    int owner[D], sl[D];
    float2 off[D];
#pragma unroll
    for (int k = 0; k < D; k++) {
        owner[k] = pc.owner[p + k];
        off[k] = pc.off[p + k];
        if (WL) sl[k] = pc.slot[p + k];
    }
    R x[D], y[D];
#pragma unroll
    for (int k = 0; k < D; k++) {
        const vec2<R> c = pc.pos[owner[k]];
        x[k] = add_rn(c.x, (R)off[k].x);
        y[k] = add_rn(c.y, (R)off[k].y);
    }
    R x1 = x[0], x0 = x[0], y1 = y[0], y0 = y[0];
#pragma unroll
    for (int k = 1; k < D; k++) {
        x1 = max_r(x1, x[k]);
        x0 = min_r(x0, x[k]);
        y1 = max_r(y1, y[k]);
        y0 = min_r(y0, y[k]);
    }
    r.hpwl = ((double)x1 - (double)x0) + ((double)y1 - (double)y0);
    if (WL) {
        NetSums<R> ns;
        R gx[D], gy[D];
        net_axis<D, EXACT, LSE, R>(x, x1, x0, igx, gx, ns.nmx, ns.dmx, ns.nnx, ns.dnx);
        net_axis<D, EXACT, LSE, R>(y, y1, y0, igy, gy, ns.nmy, ns.dmy, ns.nny, ns.dny);
#pragma unroll
        for (int k = 0; k < D; k++)
            if (sl[k] >= 0) out[sl[k]] = mk2<R>(gx[k], gy[k]);
        if (want_value) r.value = net_value<R>(ns, x1, x0, y1, y0, igx, igy, LSE);
    }
    return r;
}

// One net of kWarpPins < D <= kBlockPins pins on one warp, its pin positions
// staged in shared memory (each read back by the lane that wrote it).
template <bool WL, bool EXACT, bool LSE, typename R>
__device__ __forceinline__ NetOut net_in_warp(const int4 t, int lane, const PinCtx<R> &pc, vec2<R> *__restrict__ out,
                                              R igx, R igy, int want_value, vec2<R> *__restrict__ stage) {
    const int D = t.x, p0 = t.y;
    R x1 = (R)-3.4e38f, x0 = (R)3.4e38f, y1 = (R)-3.4e38f, y0 = (R)3.4e38f;
#pragma unroll 4
    for (int k = lane; k < D; k += 32) {
        const vec2<R> xy = pin_xy<R>(pc, p0 + k);
        if (WL) stage[k] = xy;
        x1 = max_r(x1, xy.x);
        x0 = min_r(x0, xy.x);
        y1 = max_r(y1, xy.y);
        y0 = min_r(y0, xy.y);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        x1 = max_r(x1, __shfl_xor_sync(kFull, x1, o));
        x0 = min_r(x0, __shfl_xor_sync(kFull, x0, o));
        y1 = max_r(y1, __shfl_xor_sync(kFull, y1, o));
        y0 = min_r(y0, __shfl_xor_sync(kFull, y0, o));
    }
    NetOut r{lane == 0 ? ((double)x1 - (double)x0) + ((double)y1 - (double)y0) : 0.0, 0.0};
    if (WL) {
        R s[8] = {(R)0, (R)0, (R)0, (R)0, (R)0, (R)0, (R)0, (R)0};
        for (int k = lane; k < D; k += 32) {
            const vec2<R> xy = stage[k];
            add_terms<R>(s, pin_exps<EXACT, R>(xy, x1, x0, y1, y0, igx, igy), xy);
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int i = 0; i < 8; i++) s[i] = add_rn(s[i], __shfl_xor_sync(kFull, s[i], o));
        const NetSums<R> ns = net_sums<R>(s);
        const NetCoef<R> c = net_coef<R>(ns);
        for (int k = lane; k < D; k += 32) {
            const vec2<R> xy = stage[k];
            const int sl = pc.slot[p0 + k];
            if (sl >= 0)
                out[sl] = pin_gradient<LSE, R>(pin_exps<EXACT, R>(xy, x1, x0, y1, y0, igx, igy), xy, igx, igy, c);
        }
        if (want_value && lane == 0) r.value = net_value<R>(ns, x1, x0, y1, y0, igx, igy, LSE);
    }
    return r;
}

// One net of more than kBlockPins pins on a whole block.  Its pins are taken
// kChunkPins at a time: every thread computes its pins' exponentials into
// shared memory, then warp i adds the i-th of the eight sums, lane l the pins
// l, l + 32, ... in order across the chunks, and an xor tree adds the lanes --
// net_in_warp's order.  kChunkPins keeps the FP32 pass's staging at 6 KB: at 12
// KB four blocks an SM were left under the loop's 64 KB split and the whole pass
// slowed by a fifth.  (In FP64 the warp form's positions take 12 KB anyway, for
// four blocks an SM.)  A net of more pins gathers its positions anew in each
// sweep.
template <typename R>
struct BlockStage {
    static constexpr int kChunkPins = 1024 / (int)sizeof(R);
    vec2<R> xy[kChunkPins];
    R e[4][kChunkPins];
};

template <bool WL, bool EXACT, bool LSE, typename R>
__device__ __forceinline__ NetOut net_in_block(const int4 t, const PinCtx<R> &pc, vec2<R> *__restrict__ out, R igx,
                                               R igy, int want_value, BlockStage<R> &sm, R *__restrict__ red) {
    constexpr int C = BlockStage<R>::kChunkPins, NT = kNetWarps * 32;
    static_assert(kNetWarps == 8, "a warp for each of the eight sums");
    static_assert(C % 32 == 0, "a lane's pins keep their order across the chunks");
    const int D = t.x, p0 = t.y, tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    R x1 = (R)-3.4e38f, x0 = (R)3.4e38f, y1 = (R)-3.4e38f, y0 = (R)3.4e38f;
#pragma unroll 2
    for (int k = tid; k < D; k += NT) {
        const vec2<R> xy = pin_xy<R>(pc, p0 + k);
        if (WL && k < C) sm.xy[k] = xy;
        x1 = max_r(x1, xy.x);
        x0 = min_r(x0, xy.x);
        y1 = max_r(y1, xy.y);
        y0 = min_r(y0, xy.y);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        x1 = max_r(x1, __shfl_xor_sync(kFull, x1, o));
        x0 = min_r(x0, __shfl_xor_sync(kFull, x0, o));
        y1 = max_r(y1, __shfl_xor_sync(kFull, y1, o));
        y0 = min_r(y0, __shfl_xor_sync(kFull, y0, o));
    }
    if (lane == 0) {
        red[wid] = x1;
        red[kNetWarps + wid] = x0;
        red[2 * kNetWarps + wid] = y1;
        red[3 * kNetWarps + wid] = y0;
    }
    __syncthreads();
#pragma unroll
    for (int w = 0; w < kNetWarps; w++) {
        x1 = max_r(x1, red[w]);
        x0 = min_r(x0, red[kNetWarps + w]);
        y1 = max_r(y1, red[2 * kNetWarps + w]);
        y0 = min_r(y0, red[3 * kNetWarps + w]);
    }
    NetOut r{tid == 0 ? ((double)x1 - (double)x0) + ((double)y1 - (double)y0) : 0.0, 0.0};
    if (WL) {
        R s = (R)0;
        const R *es = sm.e[wid >> 1];
        for (int c0 = 0; c0 < D; c0 += C) {  // block-uniform
            const int n = min(C, D - c0);
            if (c0 > 0) __syncthreads();  // the sums of the chunk before have read its staging
            for (int k = tid; k < n; k += NT) {
                if (c0 > 0) sm.xy[k] = pin_xy<R>(pc, p0 + c0 + k);
                const PinExp<R> e = pin_exps<EXACT, R>(sm.xy[k], x1, x0, y1, y0, igx, igy);
                sm.e[0][k] = e.emx;
                sm.e[1][k] = e.enx;
                sm.e[2][k] = e.emy;
                sm.e[3][k] = e.eny;
            }
            __syncthreads();
#pragma unroll 4
            for (int k = lane; k < n; k += 32) {
                const R e = es[k];
                s = add_rn(s, (wid & 1) ? e : mul_rn(wid < 4 ? sm.xy[k].x : sm.xy[k].y, e));
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s = add_rn(s, __shfl_xor_sync(kFull, s, o));
        if (lane == 0) red[4 * kNetWarps + wid] = s;
        __syncthreads();
        const R *tot = red + 4 * kNetWarps;
        const NetSums<R> ns{tot[0], tot[1], tot[2], tot[3], tot[4], tot[5], tot[6], tot[7]};
        const NetCoef<R> c = net_coef<R>(ns);
        for (int k = tid; k < D; k += NT) {
            const int sl = pc.slot[p0 + k];
            if (sl < 0) continue;
            const vec2<R> xy = D <= C ? sm.xy[k] : pin_xy<R>(pc, p0 + k);
            const PinExp<R> e = D <= C ? PinExp<R>{sm.e[0][k], sm.e[1][k], sm.e[2][k], sm.e[3][k]}
                                       : pin_exps<EXACT, R>(xy, x1, x0, y1, y0, igx, igy);
            out[sl] = pin_gradient<LSE, R>(e, xy, igx, igy, c);
        }
        if (want_value && tid == 0) r.value = net_value<R>(ns, x1, x0, y1, y0, igx, igy, LSE);
    }
    return r;
}

// Shared memory of the per-net pass: a block runs either one net or the tasks
// of its warps.
template <typename R>
union NetStage {
    BlockStage<R> block;
    vec2<R> warp[kNetWarps][kBlockPins];
    __device__ NetStage() {}
};

// Blocks [0, n_block): one net of more than kBlockPins pins each; the warps of
// the blocks after them take the other tasks in turn, at most kNetBlocks of
// them: as many as the SMs hold at once in FP32, where a block that ends after
// one task per warp waits for its slowest warp and its reduction three times as
// often (1M cells 75 -> 59 us, 200k 20.1 -> 17.4 on the same board).  In FP64,
// four blocks an SM, they are a wave and a half (28.7 -> 25.2), and the blocks
// of the large nets come on top in both.  The registers cost FP32 up to 128
// bytes of spills a thread, FP64 up to 432.
template <bool WL, bool EXACT, bool LSE, typename R>
__global__ void __launch_bounds__(kNetWarps * 32, sizeof(R) == 8 ? 4 : 6)
k_wl(const int4 *__restrict__ tasks, int n_block, int n_tasks, PinCtx<R> pc, vec2<R> *__restrict__ out,
     int want_value, double *__restrict__ partials, int mode, DevScalars *__restrict__ S) {
    pdl_begin();
    __shared__ double sh[64];
    __shared__ R red[5 * kNetWarps];
    __shared__ unsigned char stage_mem[WL ? sizeof(NetStage<R>) : 16] __attribute__((aligned(16)));
    NetStage<R> &stage = *reinterpret_cast<NetStage<R> *>(stage_mem);
    if (WL && S->done) return;
    const R igx = (R)S->inv_gamma_x, igy = (R)S->inv_gamma_y;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    NetOut r{0.0, 0.0};
    if ((int)blockIdx.x < n_block) {
        r = net_in_block<WL, EXACT, LSE, R>(tasks[blockIdx.x], pc, out, igx, igy, want_value, stage.block, red);
    } else {
        const int stride = ((int)gridDim.x - n_block) * kNetWarps;
        for (int w = n_block + ((int)blockIdx.x - n_block) * kNetWarps + wid; w < n_tasks; w += stride) {
            const int4 t = tasks[w];
            NetOut q{0.0, 0.0};
            static_assert(kThreadPins == 5, "the degrees below");
            if (t.x == 2)
                q = nets_by_thread<2, WL, EXACT, LSE, R>(t, lane, pc, out, igx, igy, want_value);
            else if (t.x == 3)
                q = nets_by_thread<3, WL, EXACT, LSE, R>(t, lane, pc, out, igx, igy, want_value);
            else if (t.x == 4)
                q = nets_by_thread<4, WL, EXACT, LSE, R>(t, lane, pc, out, igx, igy, want_value);
            else if (t.x == 5)
                q = nets_by_thread<5, WL, EXACT, LSE, R>(t, lane, pc, out, igx, igy, want_value);
            else if (t.x <= kWarpPins)
                q = nets_in_warp<WL, EXACT, LSE, R>(t, lane, pc, out, igx, igy, want_value);
            else
                q = net_in_warp<WL, EXACT, LSE, R>(t, lane, pc, out, igx, igy, want_value, stage.warp[wid]);
            r.hpwl += q.hpwl;
            r.value += q.value;
        }
    }
    // the smooth wirelength value rides along only when asked for
    unsigned *cnt = WL ? &S->cnt_wl : &S->cnt_hp;
    double acc[2] = {r.hpwl, r.value};
    HpwlScalars h;
    if (WL && want_value) {
        if (!grid_arrive<2>(acc, sh, partials, cnt, gridDim.x, blockIdx.x)) return;
        h = load_hpwl_scalars(S);
        grid_total<2>(acc, sh, partials, cnt, gridDim.x);
    } else {
        double a1[1] = {r.hpwl};
        if (!grid_arrive<1>(a1, sh, partials, cnt, gridDim.x, blockIdx.x)) return;
        h = load_hpwl_scalars(S);
        grid_total<1>(a1, sh, partials, cnt, gridDim.x);
        acc[0] = a1[0];
        acc[1] = 0.0;
    }
    if (threadIdx.x == 0) {
        if (WL)
            finish_wirelength(S, h, acc[0], acc[1]);
        else
            finish_hpwl(S, h, acc[0], mode);
    }
}

// ---------------------------------------------------------------- gather --
// Field gather (EPlace/eplace.cpp:599-674) in the working precision: the same
// smoothed rectangle and bin range as the scatter, the overlap in R, and the
// smoothing scale sx*sy of the object (the static FP32 table in the FP32
// path, formed in double from the size in the FP64 path).  (The scatter
// keeps the reference's exact FP64 overlap arithmetic because its maps are
// compared bit for bit; the gather is compared within tolerance.)
template <typename R>
struct FRect {
    R l, b, r, t;
};

template <typename R>
__device__ __forceinline__ FRect<R> gather_rect(const Grid &g, vec2<R> p, float2 s, uint8_t f) {
    const R hw = (R)0.5 * (R)((f & kSmoothX) ? g.sx : s.x);
    const R hh = (R)0.5 * (R)((f & kSmoothY) ? g.sy : s.y);
    return FRect<R>{p.x - hw, p.y - hh, p.x + hw, p.y + hh};
}

template <typename R>
__device__ __forceinline__ void gather_range(const Grid &g, const FRect<R> &r, int &i0, int &i1, int &j0, int &j1) {
    if constexpr (sizeof(R) == 4) {
        i0 = max(0, (int)((r.l - g.llx) * g.isx));
        i1 = min(g.nx - 1, (int)((r.r - g.llx) * g.isx));
        j0 = max(0, (int)((r.b - g.lly) * g.isy));
        j1 = min(g.ny - 1, (int)((r.t - g.lly) * g.isy));
    } else {
        i0 = max(0, (int)((r.l - (R)g.llx) / (R)g.sx));
        i1 = min(g.nx - 1, (int)((r.r - (R)g.llx) / (R)g.sx));
        j0 = max(0, (int)((r.b - (R)g.lly) / (R)g.sy));
        j1 = min(g.ny - 1, (int)((r.t - (R)g.lly) / (R)g.sy));
    }
}

template <typename R>
__device__ __forceinline__ R smoothing_scale(const Grid &g, float table, float2 s, uint8_t f) {
    if constexpr (sizeof(R) == 4) {
        return table;
    } else {
        const R sx = (f & kSmoothX) ? (R)s.x / (R)g.sx : (R)1;
        const R sy = (f & kSmoothY) ? (R)s.y / (R)g.sy : (R)1;
        return sx * sy;
    }
}

// Overlap length of [lo, hi] with bin k of an axis, 0 where they do not meet.
template <typename R>
__device__ __forceinline__ R gather_len(R base, R step, int k, R lo, R hi) {
    const R b = fma_r((R)k, step, base);
    const R len = min_r(hi, b + step) - max_r(lo, b);
    return len <= (R)0 ? (R)0 : len;
}

// acc += overlap * field; a bin that the rectangle does not meet adds nothing,
// whatever its field holds.
template <typename R>
__device__ __forceinline__ void gather_add(R &gx, R &gy, R ov, vec2<R> e) {
    if (ov == (R)0) return;
    gx = add_rn(gx, mul_rn(ov, e.x));
    gy = add_rn(gy, mul_rn(ov, e.y));
}

// Field sum of an object of at most kSmallObjectBins bins by one thread, bins
// in order (x, then y).  Rows are two at most but for objects higher than a
// bin: their overlap lengths are formed once, and the loads of two columns are
// in flight at once.
template <typename R>
__device__ __forceinline__ vec2<R> gather_small(const Grid &g, const FRect<R> &r, R sxy,
                                                const vec2<R> *__restrict__ field) {
    int i0, i1, j0, j1;
    gather_range<R>(g, r, i0, i1, j0, j1);
    R gx = (R)0, gy = (R)0;
    if (j1 < j0) return mk2<R>(gx, gy);
    if (j1 - j0 <= 1) {
        const bool two = j1 > j0;
        const R v0 = gather_len<R>((R)g.lly, (R)g.sy, j0, r.b, r.t);
        const R v1 = two ? gather_len<R>((R)g.lly, (R)g.sy, j1, r.b, r.t) : (R)0;
        const vec2<R> *row = field + (size_t)i0 * g.ny + j0;
        const vec2<R> zero = mk2<R>((R)0, (R)0);
        for (int i = i0; i <= i1; i += 2, row += 2 * g.ny) {
            const bool more = i < i1;
            const vec2<R> a0 = row[0], a1 = two ? row[1] : zero;
            const vec2<R> b0 = more ? row[g.ny] : zero, b1 = more && two ? row[g.ny + 1] : zero;
            const R ha = mul_rn(sxy, gather_len<R>((R)g.llx, (R)g.sx, i, r.l, r.r));
            const R hb = more ? mul_rn(sxy, gather_len<R>((R)g.llx, (R)g.sx, i + 1, r.l, r.r)) : (R)0;
            gather_add<R>(gx, gy, mul_rn(ha, v0), a0);
            gather_add<R>(gx, gy, mul_rn(ha, v1), a1);
            gather_add<R>(gx, gy, mul_rn(hb, v0), b0);
            gather_add<R>(gx, gy, mul_rn(hb, v1), b1);
        }
        return mk2<R>(gx, gy);
    }
    for (int i = i0; i <= i1; i++) {
        const R h = mul_rn(sxy, gather_len<R>((R)g.llx, (R)g.sx, i, r.l, r.r));
        for (int j = j0; j <= j1; j++)
            gather_add<R>(gx, gy, mul_rn(h, gather_len<R>((R)g.lly, (R)g.sy, j, r.b, r.t)),
                          field[(size_t)i * g.ny + j]);
    }
    return mk2<R>(gx, gy);
}

// Field sum of a kBig object: kBigLanes partial sums, sum v over the bins v, v +
// kBigLanes, ... in order, a tree over each 32 of them, then these in order.
// By a warp (a lane holds four of the sums) up to kWarpObjectBins bins, by the
// first kBigLanes threads of a block above.
constexpr int kBigLanes = 128;
template <typename R>
__device__ __forceinline__ void gather_strided(const Grid &g, const FRect<R> &r, R sxy, int i0, int j0, int wy, int nb,
                                               int v, const vec2<R> *__restrict__ field, R &gx, R &gy) {
#pragma unroll 4
    for (int t = v; t < nb; t += kBigLanes) {
        const int i = i0 + t / wy, j = j0 + t % wy;
        const R h = mul_rn(sxy, gather_len<R>((R)g.llx, (R)g.sx, i, r.l, r.r));
        gather_add<R>(gx, gy, mul_rn(h, gather_len<R>((R)g.lly, (R)g.sy, j, r.b, r.t)), field[(size_t)i * g.ny + j]);
    }
}

// One kBig object by a warp (block_wide false) or by a whole block; the sum in
// lane 0 of the warp, or in thread 0.
template <typename R>
__device__ __forceinline__ vec2<R> gather_big(const Grid &g, vec2<R> p, float2 size, uint8_t f, float sxy_table,
                                              const vec2<R> *__restrict__ field, bool block_wide, vec2<R> *sm) {
    const FRect<R> r = gather_rect<R>(g, p, size, f);
    const R sxy = smoothing_scale<R>(g, sxy_table, size, f);
    int i0, i1, j0, j1;
    gather_range<R>(g, r, i0, i1, j0, j1);
    const int wy = j1 - j0 + 1;
    const int nb = (i1 >= i0 && j1 >= j0) ? (i1 - i0 + 1) * wy : 0;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    R ax = (R)0, ay = (R)0;
    if (block_wide) {
        R gx = (R)0, gy = (R)0;
        if (threadIdx.x < kBigLanes) gather_strided<R>(g, r, sxy, i0, j0, wy, nb, threadIdx.x, field, gx, gy);
        gx = warp_sum_r(gx);
        gy = warp_sum_r(gy);
        if (lane == 0) sm[wid] = mk2<R>(gx, gy);
        __syncthreads();
        for (int k = 0; k < kBigLanes / 32; k++) {
            ax += sm[k].x;
            ay += sm[k].y;
        }
        __syncthreads();  // sm is used again
    } else {
#pragma unroll
        for (int k = 0; k < kBigLanes / 32; k++) {
            R gx = (R)0, gy = (R)0;
            gather_strided<R>(g, r, sxy, i0, j0, wy, nb, 32 * k + lane, field, gx, gy);
            ax += warp_sum_r(gx);
            ay += warp_sum_r(gy);
        }
    }
    return mk2<R>(ax, ay);
}

// --------------------------------------------------------------- combine --
// The scalars that the combine's finaliser reads, loaded ahead of it.
struct CombineScalars {
    double tau, step, a, bk_ratio;
    int iter, stage, max_iter, step_cap, status, step_rule, lambda0_mode;
    float target_overflow;
};
__device__ __forceinline__ CombineScalars load_combine_scalars(const DevScalars *S) {
    return CombineScalars{S->tau,      S->step,   S->a,         S->bk_ratio,     S->iter,           S->stage, S->max_iter,
                          S->step_cap, S->status, S->step_rule, S->lambda0_mode, S->target_overflow};
}

// stop_condition after a step (Optimization/nesterov.hpp:86-122): `it` steps
// taken in this stage, tau of the last gradient evaluation.
__device__ __forceinline__ int stop_after_step(const CombineScalars &c, int status, int it) {
    int stop;
    if (c.stage == EP_STAGE_MGP)
        stop = c.tau < (double)c.target_overflow || it > c.max_iter;
    else if (c.stage == EP_STAGE_FILLERONLY)
        stop = it >= 20;
    else
        stop = c.tau < (double)0.07f || it > c.max_iter;
    if (c.step_cap > 0 && it >= c.step_cap) stop = 1;
    if (status) stop = 1;
    return stop;
}

// acc: dg2, dy2, s.y, |gwl|, |gd|
__device__ __forceinline__ void finish_combine(DevScalars *S, const CombineScalars &c, const double (&acc)[5],
                                               int stepping) {
    const double dg2 = acc[0], dy2 = acc[1], sy = acc[2];
    int status = c.status;
    if (c.lambda0_mode) {
        // penaltyFactorInitilization (EPlace/eplace.cpp:812-835)
        const double lambda = acc[3] / acc[4];
        S->lambda = lambda;
        S->lambda0_mode = 0;
        if (!isfinite(lambda)) status |= 1 << EP_ERR_NAN;
    }
    if (stepping == 2) {
        // backtracking trial (opt_step_bktrk, Optimization/nesterov.hpp:351-364):
        // 1/L between the trial point and y_k; accepted when it is at
        // least BKTRK_EPS (0.95, nesterov.hpp:37; ep_limits) of the step tried
        double ns = sqrt(dy2) / sqrt(dg2);
        if (!isfinite(ns)) {
            status |= 1 << EP_ERR_NAN;
            ns = 0.0;
        }
        S->bk_accept = c.bk_ratio * c.step <= ns;
        S->step = ns;
        S->stop_pending = stop_after_step(c, status, c.iter + 1);
    } else if (stepping) {
        double step = 1.0;
        if (c.iter > 0) {
            const double lip = sqrt(dy2) / sqrt(dg2);  // 1/L
            S->lip_step = lip;
            step = lip;
            if (c.step_rule == EP_STEP_BB) {
                // BB short step s.y / y.y, else min(|s|/|y|, 1/L), which are the
                // same number (nesterov.hpp:262-274)
                const double bb = sy / dg2;
                step = bb > 0.0 ? bb : lip;
            }
        }
        if (!isfinite(step)) {
            status |= 1 << EP_ERR_NAN;
            step = 0.0;
        }
        const double an = (1.0 + sqrt(4.0 * c.a * c.a + 1.0)) / 2.0;
        S->step = step;
        S->coef = (c.a - 1.0) / an;
        S->a = an;
        S->stop_pending = stop_after_step(c, status, c.iter + 1);
    }
    if (status != c.status) S->status = status;
}

// What the combine reads of an object that no kernel writes.
struct ObjStatic {
    int o, ps, pe;
    float2 size;
    float sxy, npins, area;
    uint8_t f;
};
__device__ __forceinline__ ObjStatic load_static(const DeviceNetlist &d, int o) {
    ObjStatic s{o, 0, 0, make_float2(0.f, 0.f), 0.f, 0.f, 0.f, 0};
    if (o < d.n_obj) {
        s.f = d.flags[o];
        s.size = d.size[o];
        s.sxy = d.sxy[o];
        s.npins = d.npins[o];
        s.area = d.area[o];
        s.ps = d.obj_pin_start[o];
        s.pe = d.obj_pin_start[o + 1];
    }
    return s;
}

// The objects' field and wirelength gradients, the direction, and the sums of
// the step: a thread per object, the kBig objects in blocks of their own before
// them (object_unit).  Bound by the latency of an object's loads (netlist arrays
// -> pin gradients and field bins -> the previous step's vectors) at about half
// the warps an SM can hold.  So: the blocks loop, and load the next object's
// static arrays during this one's gather (the first one's before the wait for
// the previous grid); pin gradients and previous vectors are in flight during
// the gather; and the registers are left room, as spilling cost more than the
// warps it bought in FP32 (1M cells, blocks an SM: 2 69 us, 3 59, 4 64, 5 73; one
// object a thread at 4 blocks 96; FP64 takes three as well and spills 276 bytes
// a thread).  With the kBig objects' gather, a launch of its own
// before, us: 200k cells 18.3 + 3.1 -> 16.8, FP64 29.9 + 3.4 -> 25.5, 1M
// 88.7 + 9.1 -> 59.5.
template <typename R>
__global__ void __launch_bounds__(kThreads, 3)
k_combine(Grid g, DeviceNetlist d, const vec2<R> *__restrict__ field, const vec2<R> *__restrict__ pin_grad,
          vec2<R> *__restrict__ gout, const vec2<R> *__restrict__ g_prev, const vec2<R> *__restrict__ y_prev,
          vec2<R> *__restrict__ dump_gd, vec2<R> *__restrict__ dump_gwl, int big_blocks, int stepping,
          double *__restrict__ partials, DevScalars *__restrict__ S) {
    __shared__ double sh[32 * 5];
    __shared__ vec2<R> pin_sm[kThreads / 32][kPinChunk];
    const vec2<R> *__restrict__ pos = (const vec2<R> *)d.pos;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const ObjectUnit unit = object_unit(d, big_blocks);
    const bool big = unit.count > 1, huge = unit.count == kThreads;
    const int stride = big ? d.n_obj : ((int)gridDim.x - big_blocks) * kThreads;
    ObjStatic next = load_static(d, unit.o);
    pdl_begin();
    if (S->done) return;
    const R lam = S->lambda0_mode ? (R)0 : (R)S->lambda;
    const int iter = S->iter;
    double acc[5] = {0.0, 0.0, 0.0, 0.0, 0.0};  // dg2, dy2, s.y, |gwl|, |gd|
    do {
        const ObjStatic c = next;
        const int o = c.o;
        const uint8_t f = c.f;
        const bool valid = o < d.n_obj && (big ? unit.rank == 0 : !(f & kBig));
        // Lipschitz sums against the previous reference point: from the second
        // step on, and for every backtracking trial (stepping == 2)
        const bool lip = valid && (stepping == 2 || (stepping && iter > 0)) && (f & kInView);

        // Wirelength gradient of the object: its pins' gradients added in pin
        // order (EPlace/eplace.cpp:539-547).  The per-net pass wrote them in
        // object-major order, so the objects of a warp own one contiguous run
        // of gradient slots: the warp stages that run in shared memory with
        // coalesced loads all in flight at once (kPinChunk per round), then
        // every lane adds its own pins from there in order.  Fillers own none.
        const int wend = (int)__reduce_max_sync(kFull, valid ? (unsigned)c.pe : 0u);
        const int wbeg = min((int)__reduce_min_sync(kFull, valid ? (unsigned)c.ps : 0x7fffffffu), wend);
        vec2<R> pv[kPinChunk / 32];
#pragma unroll
        for (int u = 0; u < kPinChunk / 32; u++)
            if (wbeg + lane + 32 * u < wend) pv[u] = pin_grad[wbeg + lane + 32 * u];
        vec2<R> p = mk2<R>((R)0, (R)0), gp = p, yp = p;
        if (o < d.n_obj) p = pos[o];
        if (lip) {
            gp = g_prev[o];
            yp = y_prev[o];
        }
        next = load_static(d, o < d.n_obj - stride ? o + stride : d.n_obj);
        vec2<R> gd = mk2<R>((R)0, (R)0);
        if (big) {
            if (o < d.n_obj) gd = gather_big<R>(g, p, c.size, f, c.sxy, field, huge, pin_sm[0]);  // uniform per unit
        } else if (valid) {
            gd = gather_small<R>(g, gather_rect<R>(g, p, c.size, f), smoothing_scale<R>(g, c.sxy, c.size, f), field);
        }
        R wx = (R)0, wy = (R)0;
        vec2<R> *sm = pin_sm[wid];
        for (int base = wbeg; base < wend; base += kPinChunk) {  // warp-uniform
            const int n = min(kPinChunk, wend - base);
#pragma unroll
            for (int u = 0; u < kPinChunk / 32; u++) {
                const int t = lane + 32 * u;
                if (t < n) sm[t] = base == wbeg ? pv[u] : pin_grad[base + t];
            }
            __syncwarp();
            if (valid) {
                const int k1 = min(c.pe, base + n);
                for (int k = max(c.ps, base); k < k1; k++) {
                    const vec2<R> v = sm[k - base];
                    wx = add_rn(wx, v.x);
                    wy = add_rn(wy, v.y);
                }
            }
            __syncwarp();
        }
        if (valid) {
            // preconditioner 1/max(1, #pins + lambda*area) and direction
            R den = max_r((R)1, add_rn((R)c.npins, mul_rn(lam, (R)c.area)));
            R pre = div_rn((R)1, den);
            vec2<R> gg;
            if (f & kFiller) {
                gg.x = mul_rn(mul_rn(pre, lam), gd.x);
                gg.y = mul_rn(mul_rn(pre, lam), gd.y);
            } else {
                gg.x = mul_rn(pre, sub_rn(mul_rn(lam, gd.x), wx));
                gg.y = mul_rn(pre, sub_rn(mul_rn(lam, gd.y), wy));
            }
            gout[o] = gg;
            if (dump_gd) {
                dump_gd[o] = gd;
                dump_gwl[o] = mk2<R>(wx, wy);
            }
            if (lip) {
                double dgx = sub_rn(gg.x, gp.x), dgy = sub_rn(gg.y, gp.y);
                double dyx = sub_rn(p.x, yp.x), dyy = sub_rn(p.y, yp.y);
                acc[0] += dgx * dgx + dgy * dgy;
                acc[1] += dyx * dyx + dyy * dyy;
                acc[2] += dyx * dgx + dyy * dgy;
            }
            if (S->lambda0_mode) {
                if (!(f & kFiller)) acc[3] += fabs((double)wx) + fabs((double)wy);
                acc[4] += fabs((double)gd.x) + fabs((double)gd.y);
            }
        }
    } while (!big && __shfl_sync(kFull, next.o, 0) < d.n_obj);
    // only the sums that this call reads: the step's three, or lambda_0's two
    const bool lambda0 = S->lambda0_mode;
    CombineScalars c;
    if (stepping && !lambda0) {
        double a3[3] = {acc[0], acc[1], acc[2]};
        if (!grid_arrive<3>(a3, sh, partials, &S->cnt_comb, gridDim.x, blockIdx.x)) return;
        c = load_combine_scalars(S);
        grid_total<3>(a3, sh, partials, &S->cnt_comb, gridDim.x);
        for (int k = 0; k < 3; k++) acc[k] = a3[k];
    } else if (stepping || lambda0) {
        if (!grid_arrive<5>(acc, sh, partials, &S->cnt_comb, gridDim.x, blockIdx.x)) return;
        c = load_combine_scalars(S);
        grid_total<5>(acc, sh, partials, &S->cnt_comb, gridDim.x);
    } else {
        return;
    }
    if (threadIdx.x == 0) finish_combine(S, c, acc, stepping);
}

// ---------------------------------------------------------------- update --

// x_{k+1} = y_k + s g_k, y_{k+1} = x_{k+1} + c (x_{k+1} - x_k)
// (opt_step_vanilla, Optimization/nesterov.hpp:391-404); returns the clamped
// new position, which becomes the object's position.
template <typename R>
struct MoveInput {
    vec2<R> y, g, x;
};
template <typename R>
__device__ __forceinline__ MoveInput<R> load_move(int o, const vec2<R> *__restrict__ pos, const vec2<R> *__restrict__ x,
                                                  const vec2<R> *__restrict__ gin) {
    return MoveInput<R>{pos[o], gin[o], x[o]};
}
template <typename R>
__device__ __forceinline__ vec2<R> nesterov_move(const Grid &g, int o, R s, R c, float2 size, const MoveInput<R> &in,
                                                 vec2<R> *__restrict__ pos, vec2<R> *__restrict__ x,
                                                 vec2<R> *__restrict__ y_prev, vec2<R> *__restrict__ g_prev) {
    vec2<R> y = in.y, gg = in.g, xo = in.x;
    vec2<R> xn = mk2<R>(add_rn(y.x, mul_rn(gg.x, s)), add_rn(y.y, mul_rn(gg.y, s)));
    vec2<R> yn = mk2<R>(add_rn(xn.x, mul_rn(sub_rn(xn.x, xo.x), c)), add_rn(xn.y, mul_rn(sub_rn(xn.y, xo.y), c)));
    y_prev[o] = y;
    g_prev[o] = gg;
    x[o] = xn;
    const vec2<R> p = clamp_center<R>(g, yn, size);
    pos[o] = p;
    return p;
}

// The scalars of an update, read by one thread of the block for all of it, and
// the step's end, by the first block: iteration, stop flags and progress (host
// memory, mapped, that the host watches during a run: steps taken, kProgressDone
// once the stage has ended).  No block reads what the first one writes (`done`
// is read in the copy that the density pass left), so it need not know that the
// others have read theirs, and the stores are out while it moves its objects;
// what follows the update waits for the kernel's end.  A step (us) with the
// blocks counted and the last one ending it / with every block's count ordered
// behind its reads by a release / as here: 16^2 bins 21.5 / 22.4 / 21.5, 200k
// cells 55.2 / 57.3 / 55.0, in FP64 84.0 / 86.7 / 82.6, 1M 219 / 221 / 202.
template <typename R>
struct StepScalars {
    R step, coef;
    int stop_pending, done;
};
template <typename R>
__device__ __forceinline__ void read_step(StepScalars<R> *sh, DevScalars *S, volatile int *progress) {
    const bool ends = blockIdx.x == 0 && threadIdx.x == 0;
    int iter = 0, stage = 0;
    if (threadIdx.x == 0) {
        const StepScalars<R> v{(R)S->step, (R)S->coef, S->stop_pending, S->step_done};
        if (ends) {
            iter = S->iter;
            stage = S->stage;
        }
        *sh = v;
    }
    __syncthreads();
    if (!ends || sh->done) return;
    S->iter = ++iter;
    S->lambda_pending = 1;
    if (sh->stop_pending) {
        S->done = 1;
        if (stage == EP_STAGE_MGP) S->mgp_iterations = iter;
    }
    *progress = iter | (sh->stop_pending ? kProgressDone : 0);
}

template <typename R>
__global__ void __launch_bounds__(kThreads)
k_update(Grid g, int n, const uint8_t *__restrict__ flags, const float2 *__restrict__ size, vec2<R> *__restrict__ pos,
         vec2<R> *__restrict__ x, const vec2<R> *__restrict__ gin, vec2<R> *__restrict__ y_prev,
         vec2<R> *__restrict__ g_prev, DevScalars *__restrict__ S, int *progress) {
    __shared__ StepScalars<R> step;
    pdl_begin();
    const int o = blockIdx.x * blockDim.x + threadIdx.x;
    const bool mine = o < n && (flags[o] & kInView);
    MoveInput<R> in;
    if (mine) in = load_move<R>(o, pos, x, gin);
    read_step<R>(&step, S, progress);
    if (step.done) return;
    if (mine) nesterov_move<R>(g, o, step.step, step.coef, size[o], in, pos, x, y_prev, g_prev);
}

// The update of the captured loop, with the next evaluation's scatter fused
// in: every object is scattered at its new position right after its move
// (objects outside the stage view at their unchanged one); of a kBig object's
// threads the first moves it.  The step that ends the stage scatters nothing,
// so the maps stay clear (prep clears them after each read).
// MINB: blocks an SM that the registers have to allow.  Six hide the latency of
// a large design's atomics (40 registers, no spills); a design whose blocks are
// all resident anyway takes the instance without.
template <int MINB, typename R>
__global__ void __launch_bounds__(kThreads, MINB)
k_update_scatter(Grid g, DeviceNetlist d, int big_blocks, vec2<R> *__restrict__ pos, vec2<R> *__restrict__ x,
                 const vec2<R> *__restrict__ gin, vec2<R> *__restrict__ y_prev, vec2<R> *__restrict__ g_prev,
                 double qscale, ull *__restrict__ maps, DevScalars *__restrict__ S, int *progress) {
    __shared__ vec2<R> big_pos[kThreads / 32];
    __shared__ StepScalars<R> step;
    const ObjectUnit u = object_unit(d, big_blocks);
    const bool valid = u.o < d.n_obj;
    const uint8_t f = valid ? d.flags[u.o] : 0;
    const float2 sz = valid ? d.size[u.o] : make_float2(1.f, 1.f);
    const float sxy = valid ? d.sxy[u.o] : 0.f;
    pdl_begin();
    MoveInput<R> in;
    const bool mover = valid && (u.count == 1 ? !(f & kBig) : u.rank == 0);
    if (mover) in = load_move<R>(u.o, pos, x, gin);
    read_step<R>(&step, S, progress);
    if (step.done) return;
    const bool scatter = !step.stop_pending;
    auto move = [&] {
        return (f & kInView) ? nesterov_move<R>(g, u.o, step.step, step.coef, sz, in, pos, x, y_prev, g_prev) : in.y;
    };
    if (u.count == 1) {
        const vec2<R> p = mover ? move() : mk2<R>((R)g.llx, (R)g.lly);
        if (scatter) scatter_objects<R>(g, mover, p, sz, sxy, f, qscale, maps);
    } else {
        const int slot = u.count == kThreads ? 0 : threadIdx.x >> 5;
        if (mover) big_pos[slot] = move();
        __syncthreads();  // block-uniform: every unit of this block has several threads
        if (valid && scatter) scatter_big<R>(g, big_pos[slot], sz, sxy, f, qscale, u.rank, u.count, maps);
    }
}

// Backtracking trial move (opt_step_bktrk, Optimization/nesterov.hpp:337-349):
// from y_k (kept in ysave) x_t = y_k + step g_k, y_t = x_t + coef (x_t - x_k);
// the positions become clamp(y_t) and x_t is kept in xtrial until accepted.
template <typename R>
__global__ void __launch_bounds__(kThreads)
k_bktrk_move(Grid g, int n, const uint8_t *__restrict__ flags, const float2 *__restrict__ size,
             const vec2<R> *__restrict__ ysave, const vec2<R> *__restrict__ gin, const vec2<R> *__restrict__ x,
             vec2<R> *__restrict__ pos, vec2<R> *__restrict__ xtrial, const DevScalars *__restrict__ S) {
    pdl_begin();
    if (S->done) return;
    int o = blockIdx.x * blockDim.x + threadIdx.x;
    if (o >= n) return;
    if (!(flags[o] & kInView)) {
        xtrial[o] = x[o];
        return;
    }
    R s = (R)S->step, c = (R)S->coef;
    vec2<R> y = ysave[o], gg = gin[o], xo = x[o];
    vec2<R> xn = mk2<R>(add_rn(y.x, mul_rn(gg.x, s)), add_rn(y.y, mul_rn(gg.y, s)));
    vec2<R> yn = mk2<R>(add_rn(xn.x, mul_rn(sub_rn(xn.x, xo.x), c)), add_rn(xn.y, mul_rn(sub_rn(xn.y, xo.y), c)));
    xtrial[o] = xn;
    pos[o] = clamp_center<R>(g, yn, size[o]);
}

// EplaceNesterovOpt::init (nesterov.hpp:207-214): x_0 = current positions.
template <typename R>
__global__ void k_stage_begin(int n, const uint8_t *__restrict__ flags, const vec2<R> *__restrict__ pos,
                              vec2<R> *__restrict__ x, int step_cap, DevScalars *__restrict__ S, int *progress) {
    pdl_begin();
    for (int o = blockIdx.x * blockDim.x + threadIdx.x; o < n; o += gridDim.x * blockDim.x)
        if (flags[o] & kInView) x[o] = pos[o];
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        S->a = 1.0;
        S->iter = 0;
        S->lambda_pending = 0;
        S->stop_pending = 0;
        S->status = 0;
        double tau = S->tau;
        int stop;
        if (S->stage == EP_STAGE_MGP)
            stop = tau < (double)S->target_overflow;
        else if (S->stage == EP_STAGE_FILLERONLY)
            stop = 0;
        else
            stop = tau < (double)0.07f;
        S->done = stop;
        S->step_cap = step_cap;
        if (stop && S->stage == EP_STAGE_MGP) S->mgp_iterations = 0;
        *(volatile int *)progress = stop ? kProgressDone : 0;
    }
}

// wrap_up (nesterov.hpp:216-223): positions = main solution, clamped.
template <typename R>
__global__ void k_wrap_up(Grid g, int n, const uint8_t *__restrict__ flags, const float2 *__restrict__ size,
                          vec2<R> *__restrict__ pos, const vec2<R> *__restrict__ x) {
    pdl_begin();
    int o = blockIdx.x * blockDim.x + threadIdx.x;
    if (o < n && (flags[o] & kInView)) pos[o] = clamp_center<R>(g, x[o], size[o]);
}

}  // namespace

// ------------------------------------------------------------- launchers --
namespace {
template <typename R>
inline vec2<R> *V(void *p) {
    return static_cast<vec2<R> *>(p);
}
template <typename R>
inline const vec2<R> *V(const void *p) {
    return static_cast<const vec2<R> *>(p);
}

template <bool WL, bool EXACT, bool LSE, typename R>
void launch_nets(const KernelCtx &c, const DeviceNetlist &d, void *pin_grad, double *partials, int mode, DevScalars *S,
                 cudaStream_t st) {
    PinCtx<R> pc{d.pin_owner, d.pin_off, V<R>(d.pos), d.pin_obj_slot};
    if (d.n_net_tasks == 0) return;
    launch_kp(k_wl<WL, EXACT, LSE, R>, reduction_blocks(d, 0), kNetWarps * 32, 0, st, launch_priority(false),
              d.net_tasks, d.n_block_nets, d.n_net_tasks, pc, V<R>(pin_grad), c.want_wl_value, partials, mode, S);
}

// Blocks an SM that k_update_scatter's registers allow in a large design.
template <typename R>
constexpr int kUpdateBlocks = sizeof(R) == 8 ? 5 : 6;
}  // namespace

template <typename R>
void Loop<R>::scatter(const KernelCtx &c, const DeviceNetlist &d, ull *maps, const DevScalars *S, cudaStream_t st) {
    const int bb = big_blocks(d);
    launch_k(k_scatter<R>, bb + blocks_for(d.n_obj, kThreads), kThreads, 0, st, c.grid, d, bb, c.qscale, maps, S);
}

template <typename R>
void Loop<R>::update_scatter(const KernelCtx &c, const DeviceNetlist &d, void *pos, void *x, const void *g,
                             void *y_prev, void *g_prev, ull *maps, DevScalars *S, int *progress, cudaStream_t st) {
    const int bb = big_blocks(d);
    const int blocks = bb + blocks_for(d.n_obj, kThreads);
    launch_k(blocks <= kSms * 4 ? k_update_scatter<1, R> : k_update_scatter<kUpdateBlocks<R>, R>, blocks, kThreads, 0,
             st, c.grid, d, bb, V<R>(pos), V<R>(x), V<R>(g), V<R>(y_prev), V<R>(g_prev), c.qscale, maps, S, progress);
}

template <typename R>
void Loop<R>::prep(const KernelCtx &c, ull *node_q, ull *filler_q, const float2 *static_map, void *rho, void *rho_bf16,
                   float *node_f, float *filler_f, int zero_maps, DevScalars *S, cudaStream_t st) {
    uint16_t *hi = sizeof(R) == 4 ? (uint16_t *)rho_bf16 : nullptr;
    uint16_t *lo = hi ? hi + c.grid.nx * c.grid.ny : nullptr;
    launch_k(k_prep<R>, prep_blocks(c.grid), kThreads, 0, st, c.grid, node_q, filler_q, static_map, (R *)rho, hi, lo,
             node_f, filler_f, zero_maps, c.inv_qscale, c.inv_bin_area, c.bin_area, c.area_norm, c.part_prep, S);
}

template <typename R>
void Loop<R>::wirelength(const KernelCtx &c, const DeviceNetlist &d, void *pin_grad, DevScalars *S, cudaStream_t st) {
    if (c.exact_exp)
        c.lse ? launch_nets<true, true, true, R>(c, d, pin_grad, c.part_wl, 0, S, st)
              : launch_nets<true, true, false, R>(c, d, pin_grad, c.part_wl, 0, S, st);
    else
        c.lse ? launch_nets<true, false, true, R>(c, d, pin_grad, c.part_wl, 0, S, st)
              : launch_nets<true, false, false, R>(c, d, pin_grad, c.part_wl, 0, S, st);
}

template <typename R>
void Loop<R>::hpwl(const KernelCtx &c, const DeviceNetlist &d, int mode, DevScalars *S, cudaStream_t st) {
    launch_nets<false, false, false, R>(c, d, nullptr, c.part_hp, mode, S, st);
}

template <typename R>
void Loop<R>::combine(const KernelCtx &c, const DeviceNetlist &d, const void *field, const void *pin_grad, void *g,
                      const void *g_prev, const void *y_prev, void *dump_gd, void *dump_gwl, int stepping,
                      DevScalars *S, cudaStream_t st) {
    launch_k(k_combine<R>, reduction_blocks(d, 1), kThreads, 0, st, c.grid, d, V<R>(field), V<R>(pin_grad), V<R>(g),
             V<R>(g_prev), V<R>(y_prev), V<R>(dump_gd), V<R>(dump_gwl), big_blocks(d), stepping, c.part_comb, S);
}

template <typename R>
void Loop<R>::update(const KernelCtx &c, const DeviceNetlist &d, void *pos, void *x, const void *g, void *y_prev,
                     void *g_prev, DevScalars *S, int *progress, cudaStream_t st) {
    launch_k(k_update<R>, blocks_for(d.n_obj, kThreads), kThreads, 0, st, c.grid, d.n_obj, d.flags, d.size,
             V<R>(pos), V<R>(x), V<R>(g), V<R>(y_prev), V<R>(g_prev), S, progress);
}

template <typename R>
void Loop<R>::bktrk_move(const KernelCtx &c, const DeviceNetlist &d, const void *ysave, const void *g, const void *x,
                         void *pos, void *xtrial, const DevScalars *S, cudaStream_t st) {
    launch_k(k_bktrk_move<R>, blocks_for(d.n_obj, kThreads), kThreads, 0, st, c.grid, d.n_obj, d.flags, d.size,
             V<R>(ysave), V<R>(g), V<R>(x), V<R>(pos), V<R>(xtrial), S);
}

template <typename R>
void Loop<R>::stage_begin(const DeviceNetlist &d, const void *pos, void *x, int step_cap, DevScalars *S,
                          int *progress, cudaStream_t st) {
    launch_k(k_stage_begin<R>, std::min(blocks_for(d.n_obj, kThreads), kSms * 4), kThreads, 0, st, d.n_obj, d.flags,
             V<R>(pos), V<R>(x), step_cap, S, progress);
}

template <typename R>
void Loop<R>::wrap_up(const KernelCtx &c, const DeviceNetlist &d, void *pos, const void *x, cudaStream_t st) {
    launch_k(k_wrap_up<R>, blocks_for(d.n_obj, kThreads), kThreads, 0, st, c.grid, d.n_obj, d.flags, d.size,
             V<R>(pos), V<R>(x));
}

template <typename R>
std::vector<const void *> Loop<R>::kernels(bool exact_exp, bool lse) {
    const void *wl = exact_exp ? (lse ? (const void *)k_wl<true, true, true, R> : (const void *)k_wl<true, true, false, R>)
                               : (lse ? (const void *)k_wl<true, false, true, R> : (const void *)k_wl<true, false, false, R>);
    return {(const void *)k_scatter<R>, (const void *)k_prep<R>, wl, (const void *)k_wl<false, false, false, R>,
            (const void *)k_combine<R>, (const void *)k_update<R>, (const void *)k_update_scatter<1, R>,
            (const void *)k_update_scatter<kUpdateBlocks<R>, R>, (const void *)k_bktrk_move<R>,
            (const void *)k_stage_begin<R>, (const void *)k_wrap_up<R>};
}

}  // namespace ep
