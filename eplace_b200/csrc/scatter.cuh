// scatter.cuh -- an object's contributions to the int64 density maps
// (EPlacer_2D::binNodeDensityUpdate, EPlace/eplace.cpp:1029-1133), shared by
// the engine's scatter and ep_density_scatter_noalloc.
//
// A contribution is the overlap area (the reference's FP64 products) rounded to
// the working precision, times the object's scale, rounded to the fixed-point
// grid and added with an atomic.  The overlap is a product of one length per
// axis, so the lengths are formed once per column and row of the footprint
// instead of once per bin (a third of a bin's instructions), and the two rows
// of a cell are added by neighbouring lanes.  What bounds it then is the L2's
// rate of 64-bit adds: 9.5M in 37 us at 1M cells and fillers (42.8 before; 200k
// 10.7 -> 8.4 us, FP64 12.7 -> 10.5; ep_density_scatter_noalloc with 300k objects
// 25.3 -> 23.4 us in all, and 19.2 with its launches overlapped).
#pragma once
#include "common.cuh"

namespace ep {

// Overlap length (0 or negative, as overlap_len) of [lo, hi] with bin k of an axis.
template <typename R>
__device__ __forceinline__ double bin_overlap_len(R base, R step, int k, double lo, double hi) {
    const R b = add_rn(mul_rn((R)k, step), base), t = add_rn(b, step);
    return overlap_len((double)b, (double)t, lo, hi);
}

// Fixed-point contribution of one bin (0: the object does not meet it).
template <typename R>
__device__ __forceinline__ long long scatter_value(double len_x, double len_y, R scale, double qscale) {
    const R ovl = (R)__dmul_rn(len_x, len_y);
    return ovl == (R)0 ? 0ll : __double2ll_rn(__dmul_rn((double)mul_rn(scale, ovl), qscale));
}

template <typename R>
__device__ __forceinline__ void scatter_add(double len_x, double len_y, R scale, double qscale,
                                            unsigned long long *__restrict__ bin) {
    const long long q = scatter_value<R>(len_x, len_y, scale, qscale);
    if (q) atomicAdd(bin, (unsigned long long)q);
}

// The objects of a warp, one a lane: bins [i0, i1] x [j0, j1] each (i1 < i0: the
// lane has none), `bin` the index of bin (i0, j0) in maps.  Every lane of the
// warp calls it.  An object no higher than a bin touches two rows, neighbours
// in memory; so that both adds of a column reach the L2 as one request, lanes 2m
// and 2m + 1 add the two rows of one lane's object together, then of the
// other's.  The L2's atomic rate is what bounds the scatter.
template <typename R>
__device__ __forceinline__ void scatter_by_lane(const Grid &g, const RectT<R> &r, R scale, int i0, int i1, int j0,
                                                int j1, double qscale, unsigned bin,
                                                unsigned long long *__restrict__ maps) {
    constexpr unsigned kAll = 0xffffffffu;
    const double llx = r.llx, urx = r.urx, lly = r.lly, ury = r.ury;
    if (j1 < j0) i1 = i0 - 1;
    if (j1 - j0 > 1) {
        for (int i = i0; i <= i1; i++, bin += g.ny) {
            const double h = bin_overlap_len<R>((R)g.llx, (R)g.sx, i, llx, urx);
            for (int j = j0; j <= j1; j++)
                scatter_add<R>(h, bin_overlap_len<R>((R)g.lly, (R)g.sy, j, lly, ury), scale, qscale,
                               maps + bin + (j - j0));
        }
        i1 = i0 - 1;
    }
    const int cols = (int)__reduce_max_sync(kAll, (unsigned)max(i1 - i0 + 1, 0));
    const double v0 = bin_overlap_len<R>((R)g.lly, (R)g.sy, j0, lly, ury);
    const double v1 = j1 > j0 ? bin_overlap_len<R>((R)g.lly, (R)g.sy, j1, lly, ury) : 0.0;
    const bool odd = threadIdx.x & 1;
    for (int c = 0; c < cols; c++, bin += g.ny) {
        long long q0 = 0, q1 = 0;
        if (i0 + c <= i1) {
            const double h = bin_overlap_len<R>((R)g.llx, (R)g.sx, i0 + c, llx, urx);
            q0 = scatter_value<R>(h, v0, scale, qscale);
            q1 = scatter_value<R>(h, v1, scale, qscale);
        }
        const long long other = __shfl_xor_sync(kAll, odd ? q0 : q1, 1);
        const unsigned other_bin = __shfl_xor_sync(kAll, bin, 1) + (odd ? 1u : 0u);
        const long long mine = odd ? q1 : q0;
        const unsigned my_bin = bin + (odd ? 1u : 0u);
        // the even lane's object, then the odd lane's
        const long long qa = odd ? other : mine, qb = odd ? mine : other;
        const unsigned ba = odd ? other_bin : my_bin, bb = odd ? my_bin : other_bin;
        if (qa) atomicAdd(maps + ba, (unsigned long long)qa);
        if (qb) atomicAdd(maps + bb, (unsigned long long)qb);
    }
}

// All bins [i0, i1] x [j0, j1] of one object by `count` threads, this one the
// rank-th.
template <typename R>
__device__ __forceinline__ void scatter_by_group(const Grid &g, const RectT<R> &r, R scale, int i0, int i1, int j0,
                                                 int j1, double qscale, int rank, int count,
                                                 unsigned long long *__restrict__ map) {
    if (i1 < i0 || j1 < j0) return;
    const int wy = j1 - j0 + 1, nb = (i1 - i0 + 1) * wy;
    for (int t = rank; t < nb; t += count) {
        const int i = i0 + t / wy, j = j0 + t % wy;
        scatter_add<R>(bin_overlap_len<R>((R)g.llx, (R)g.sx, i, r.llx, r.urx),
                       bin_overlap_len<R>((R)g.lly, (R)g.sy, j, r.lly, r.ury), scale, qscale,
                       map + (size_t)i * g.ny + j);
    }
}

}  // namespace ep
