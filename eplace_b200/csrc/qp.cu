// qp.cu -- quadratic placement (QPPlacer::quadraticPlacement,
// QPlace/qplace.cpp:20-106) on the device: the initial placement ePlace
// starts from.
//
// Each outer round freezes the current centres, builds for X and for Y the
// system A x = b of the bound-pin model (QPPlacer::createSparseMatrix,
// qplace.cpp:125-272) and solves both with BiCGSTAB (identity
// preconditioner, warm start from the centres), then moves the nodes to the
// solution (clamped into the core) and recomputes the bound pins.
//
// The model, per net of p pins with bound pins found first-occurrence as
// Net::calcBoundPin does (PlaceCommon/objects.cpp:75-144): an unordered pin
// pair on different modules contributes w = (1/(p-1)) / max(d, 25) (d the
// pair's distance along the axis, MIN_DISTANCE 25, qplace.h) when, for X,
// either pin is the net's min- or max-x pin; for Y the reference tests
// "pin2 == Ymin || pin1 == Ymax || pin2 == Ymin || pin2 == Ymax" with pin1
// before pin2 in the net (qplace.cpp:206), which the engine reproduces: the
// Y system differs from the X one exactly as the reference's does.
// Movable-movable pairs add w to both diagonals, -w off the diagonal and
// -w (off_i - off_j) to b_i; a pair with a fixed pin adds w to the movable
// diagonal and w (abs_fixed - off_i) to its b.
//
// The matrices are built row by row (one thread per movable node, its pins in
// Module::modulePins order, each pin's partners in net order): a count pass,
// a prefix sum, a fill pass.  The row order of entries is fixed, and every
// dot product is an FP64 sum in a fixed tree, so the solve is bitwise
// repeatable.
#include <algorithm>

#include "engine.h"

namespace ep {

namespace {

constexpr int kQT = 256;
constexpr float kMinDistance = 25.0f;  // MIN_DISTANCE, QPlace/qplace.h

inline int qblocks(int n) { return (n + kQT - 1) / kQT; }
// The bounds pass runs on at most 8 blocks per SM and loops over its nets, so the
// finalising block adds few partials; the grid depends only on the sizes, so
// the sum is the same on every run.
constexpr int kQpMaxBlocks = 148 * 8;
// The solver's kernels: at most what the SMs hold at once.  The SpMV's need 80
// registers for that; with the 90 it would take, half of the blocks wait for a
// second wave (24 against 17 us).
constexpr int kSolveBlocks = 148 * 3;
inline int qgrid(int n) { return std::min(qblocks(n), kQpMaxBlocks); }

__device__ __forceinline__ float2 abs_pin(const float2 *__restrict__ pos, const float2 *__restrict__ off,
                                          int owner, int q) {
    const float2 c = pos[owner], o = off[q];
    return make_float2(__fadd_rn(c.x, o.x), __fadd_rn(c.y, o.y));
}

// Net::calcBoundPin: strict compares in double, the first pin at the
// extreme wins; bound = (x-min, x-max, y-min, y-max) as indices in the net.
// Nets in device order: the nets above kWarpPins pins (the head of that
// order) take a warp each -- lane l scans pins l, l + 32, ... and the lanes'
// (value, first index) pairs meet in a tree that keeps the extreme value and,
// among equal values, the lower index, which is the serial scan's answer --
// and the others a thread each.  A grid-stride loop over 32 n_big + (nnet -
// n_big) slots; the HPWL of the net (double) joins the grid sum.
struct Ext {
    double v;
    int k;
};
__device__ __forceinline__ void ext_min(Ext &a, double v, int k) {
    if (v < a.v || (v == a.v && k < a.k)) a = Ext{v, k};
}
__device__ __forceinline__ void ext_max(Ext &a, double v, int k) {
    if (v > a.v || (v == a.v && k < a.k)) a = Ext{v, k};
}

__global__ void __launch_bounds__(kQT)
k_qp_bounds(int nnet, int n_big, const int32_t *__restrict__ order, const int32_t *__restrict__ first,
            const int32_t *__restrict__ deg, const int32_t *__restrict__ owner, const float2 *__restrict__ off,
            const float2 *__restrict__ pos, int4 *__restrict__ bound, float2 *__restrict__ abspin,
            double *__restrict__ partials, unsigned *__restrict__ cnt, double *__restrict__ hpwl) {
    __shared__ double sh[32];
    double acc[1] = {0.0};
    const long long big = 32LL * n_big, slots = big + (nnet - n_big);
    const int lane = threadIdx.x & 31;
    for (long long t = blockIdx.x * (long long)blockDim.x + threadIdx.x; t < slots;
         t += (long long)gridDim.x * blockDim.x) {
        if (t < big) {  // whole warps (big is a multiple of 32, so is the stride)
            const int n = order[t >> 5], f = first[n], d = deg[n];
            Ext lx{1.79769e308, 0x7fffffff}, hx{-1.79769e308, 0x7fffffff};
            Ext ly{1.79769e308, 0x7fffffff}, hy{-1.79769e308, 0x7fffffff};
            for (int k = lane; k < d; k += 32) {
                const float2 a = abs_pin(pos, off, owner[f + k], f + k);
                abspin[f + k] = a;
                ext_min(lx, a.x, k);
                ext_max(hx, a.x, k);
                ext_min(ly, a.y, k);
                ext_max(hy, a.y, k);
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                ext_min(lx, __shfl_xor_sync(0xffffffffu, lx.v, o), __shfl_xor_sync(0xffffffffu, lx.k, o));
                ext_max(hx, __shfl_xor_sync(0xffffffffu, hx.v, o), __shfl_xor_sync(0xffffffffu, hx.k, o));
                ext_min(ly, __shfl_xor_sync(0xffffffffu, ly.v, o), __shfl_xor_sync(0xffffffffu, ly.k, o));
                ext_max(hy, __shfl_xor_sync(0xffffffffu, hy.v, o), __shfl_xor_sync(0xffffffffu, hy.k, o));
            }
            if (lane == 0) {
                bound[n] = make_int4(lx.k, hx.k, ly.k, hy.k);
                acc[0] += (hx.v - lx.v) + (hy.v - ly.v);
            }
            continue;
        }
        const int n = order[n_big + (int)(t - big)], f = first[n], d = deg[n];
        double mnx = 1.79769e308, mxx = -1.79769e308, mny = 1.79769e308, mxy = -1.79769e308;
        int4 b = make_int4(0, 0, 0, 0);
        for (int k = 0; k < d; k++) {
            const float2 a = abs_pin(pos, off, owner[f + k], f + k);
            abspin[f + k] = a;
            if ((double)a.x < mnx) { mnx = a.x; b.x = k; }
            if ((double)a.x > mxx) { mxx = a.x; b.y = k; }
            if ((double)a.y < mny) { mny = a.y; b.z = k; }
            if ((double)a.y > mxy) { mxy = a.y; b.w = k; }
        }
        bound[n] = b;
        if (d > 0) acc[0] += (mxx - mnx) + (mxy - mny);
    }
    if (!grid_arrive<1>(acc, sh, partials, cnt, gridDim.x, blockIdx.x)) return;
    grid_total<1>(acc, sh, partials, cnt, gridDim.x);
    if (threadIdx.x == 0) *hpwl = acc[0];
}

// Partners of pin a (index in its net of d pins) in the X model: every pin
// when a is a bound pin, else the two bound pins.
template <class F>
__device__ __forceinline__ void partners_x(int a, int d, int lo, int hi, F &&f) {
    if (a == lo || a == hi) {
        for (int b = 0; b < d; b++)
            if (b != a) f(b);
    } else {
        f(lo);
        if (hi != lo) f(hi);
    }
}

// Partners of pin a in the reference's Y model: the unordered pair (j < k)
// counts when k == y-min, j == y-max or k == y-max.
template <class F>
__device__ __forceinline__ void partners_y(int a, int d, int lo, int hi, F &&f) {
    if (a == hi) {
        for (int b = 0; b < d; b++)
            if (b != a) f(b);
    } else if (a == lo) {
        for (int b = 0; b < a; b++) f(b);
        if (hi > a) f(hi);
    } else {
        f(hi);
        if (lo > a && lo != hi) f(lo);
    }
}

// weightX / weightY of createSparseMatrix (qplace.cpp:172-183): float
// division, the distance held at MIN_DISTANCE from below (float_greaterorequal
// reduces to >= for float operands).
__device__ __forceinline__ float pair_weight(float c, float dist) {
    return dist >= kMinDistance ? __fdiv_rn(c, dist) : __fdiv_rn(c, kMinDistance);
}

// Pair (i, owner of pin q2) on one axis (pa, oa: pin a's coordinate and
// offset on that axis): adds the pair's weight to the diagonal sum and its
// term to the right-hand side; returns the partner node when it is movable
// (an off-diagonal entry of weight -w), -1 when it is i itself (no pair) or
// fixed (right-hand side only).
__device__ __forceinline__ int pair_terms(int i, int nn, int q2, int axis, const int32_t *__restrict__ owner,
                                          const float2 *__restrict__ abspin, const float2 *__restrict__ off, float c,
                                          float pa, float oa, float &w, double &dsum, double &bsum) {
    const int j = owner[q2];
    if (j == i) return -1;
    const float2 pb2 = abspin[q2];
    const float pb = axis ? pb2.y : pb2.x, ob = axis ? off[q2].y : off[q2].x;
    w = pair_weight(c, fabsf(__fsub_rn(pa, pb)));
    dsum += w;
    if (j < nn) {
        bsum += -(double)w * (double)__fsub_rn(oa, ob);
        return j;
    }
    bsum += (double)w * (double)__fsub_rn(pb, oa);
    return -1;
}

// The count pass's test of a pair: the partner node when it gives an
// off-diagonal entry (movable and not i itself), else -1 -- the entries
// pair_terms reports, without the weights.
__device__ __forceinline__ int pair_partner(int i, int nn, int q2, const int32_t *__restrict__ owner) {
    const int j = owner[q2];
    return j != i && j < nn ? j : -1;
}

// A pin's partner set as a range: pins [0, end) of its net but `skip`, then
// `extra` (-1: none) -- the bound pins' sets of partners_x / partners_y.
struct PartnerRange {
    int end, skip, extra;
};
__device__ __forceinline__ bool range_x(int a, int d, int lo, int hi, PartnerRange &r) {
    if (a != lo && a != hi) return false;
    r = PartnerRange{d, a, -1};
    return true;
}
__device__ __forceinline__ bool range_y(int a, int d, int lo, int hi, PartnerRange &r) {
    if (a == hi) {
        r = PartnerRange{d, a, -1};
        return true;
    }
    if (a != lo) return false;
    r = PartnerRange{a, -1, hi > a ? hi : -1};
    return true;
}
// partner sets above kLongPartners pins are taken by the whole warp (placed
// after the row's short sets; the threshold fixes the order of a row's
// entries, so the SpMV's sums)
constexpr int kLongPartners = 32;
__device__ __forceinline__ bool is_long(const PartnerRange &r) {
    return r.end - (r.skip >= 0) + (r.extra >= 0) > kLongPartners;
}

// ---- matrix layout --------------------------------------------------------------
// Entries (column, value) of one axis lie in one array.  The rows of at most
// kLongRow entries on both axes go by slices of 32 rows (a warp): entry k of
// the slice's row l is at base + 32 k + l, so a thread per row reads them with
// one coalesced load per k.  A slice is as long as its longest row, so the rows
// of each window of kQT rows (a block) are sorted by length first; the window
// is small, so that a slice's rows still lie near one another in the vectors.
// The longer rows (the bound pins of large nets) follow all slices, their
// entries contiguous, and are listed in `longs`, so that warps of their own take
// them first.  The count pass sorts its
// window and leaves the rows' places in it; one block scans the windows.
constexpr int kLongRow = 32;
constexpr int kSlices = kQT / 32;  // of a window

struct __align__(16) Window {  // totals of a window, then its first places
    int x, y;                  // entries of its slices (32 x the longest row of each)
    int n_long, long_x, long_y, pad[3];
};

struct QpLayout {
    Window *win;
    int2 *slice;  // a slice's first X and Y entry, from its window's
    int2 *slot;   // the slices' rows: (row, X entries | Y entries << 8), row -1: none
    int2 *rel;    // a row's first X and Y entry, from its window's
    int4 *longs;  // two per long row: (row, first X entry, first Y entry, X entries), (Y entries, 0, 0, 0)
};

constexpr int kScanThreads = 1024;
__global__ void __launch_bounds__(kScanThreads)
k_qp_scan(int nw, Window *__restrict__ t, int cap_x, int cap_y, QpSolve *__restrict__ S) {
    __shared__ int warp_tot[5][kScanThreads / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    // a contiguous run of windows per thread
    const int per = (nw + kScanThreads - 1) / kScanThreads, s0 = min(nw, (int)threadIdx.x * per), s1 = min(nw, s0 + per);
    int v[5] = {0, 0, 0, 0, 0};
    for (int k = s0; k < s1; k++) {
        const Window c = t[k];
        v[0] += c.x;
        v[1] += c.y;
        v[2] += c.n_long;
        v[3] += c.long_x;
        v[4] += c.long_y;
    }
    int run[5];
    long long total[5];  // past 2^31 they overflow any allocation, and the places are not used
#pragma unroll
    for (int q = 0; q < 5; q++) {
        int x = v[q];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_tot[q][w] = x;
        run[q] = x - v[q];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 5; q++) {
        total[q] = 0;
        for (int k = 0; k < kScanThreads / 32; k++) {
            if (k < w) run[q] += warp_tot[q][k];
            total[q] += warp_tot[q][k];
        }
    }
    for (int k = s0; k < s1; k++) {
        const Window c = t[k];
        t[k] = Window{run[0], run[1], run[2], (int)total[0] + run[3], (int)total[1] + run[4], {0, 0, 0}};
        run[0] += c.x;
        run[1] += c.y;
        run[2] += c.n_long;
        run[3] += c.long_x;
        run[4] += c.long_y;
    }
    if (threadIdx.x == 0) {
        S->n_long = (int)total[2];
        S->overflow = total[0] + total[3] > cap_x || total[1] + total[4] > cap_y;
    }
}

// Sort the block's rows by their length (stable, the long rows last) and leave
// their places: a counting sort over the keys 0 .. kLongRow + 1.  Every thread
// of the block calls it; lx, ly: its row's entries (rows past the last: 0, 0,
// which take slots of no row).
__device__ __forceinline__ void place_window(int i, int nn, int lx, int ly, const QpLayout &q) {
    constexpr int kKeys = kLongRow + 2;
    __shared__ int warp_key[kSlices][kKeys], first[kKeys];
    __shared__ int slice_len[2][kSlices], long_n, long_x, long_y;
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    const bool lg = max(lx, ly) > kLongRow;
    const int key = lg ? kKeys - 1 : max(lx, ly);
    for (int k = tid; k < kSlices * kKeys; k += kQT) (&warp_key[0][0])[k] = 0;
    if (tid < kSlices) slice_len[0][tid] = slice_len[1][tid] = 0;
    __syncthreads();
    const unsigned peers = __match_any_sync(0xffffffffu, key);
    const int rank = __popc(peers & ((1u << lane) - 1));
    if (rank == 0) warp_key[w][key] = __popc(peers);
    __syncthreads();
    if (tid < kKeys) {  // rows of this key in the warps before each warp
        int n = 0;
        for (int k = 0; k < kSlices; k++) {
            const int c = warp_key[k][tid];
            warp_key[k][tid] = n;
            n += c;
        }
        first[tid] = n;
    }
    __syncthreads();
    if (tid == 0) {
        int n = 0;
        for (int k = 0; k < kKeys; k++) {
            const int c = first[k];
            first[k] = n;
            n += c;
        }
        // the long rows' entries one after another, in row order
        long_n = long_x = long_y = 0;
    }
    __syncthreads();
    const int at = first[key] + warp_key[w][key] + rank, sl = at >> 5;
    if (!lg) {
        atomicMax(&slice_len[0][sl], lx);
        atomicMax(&slice_len[1][sl], ly);
    }
    // exclusive sums over the long rows of the block, warp by warp
    int px = lg ? lx : 0, py = lg ? ly : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int a = __shfl_up_sync(0xffffffffu, px, o), b = __shfl_up_sync(0xffffffffu, py, o);
        if (lane >= o) {
            px += a;
            py += b;
        }
    }
    const int nlong = __popc(__ballot_sync(0xffffffffu, lg));
    int bx = 0, by = 0;
    for (int k = 0; k < kSlices; k++) {
        __syncthreads();
        if (k == w) {
            bx = long_x;
            by = long_y;
        }
        __syncthreads();
        if (k == w && lane == 31) {
            long_x += px;
            long_y += py;
            long_n += nlong;
        }
    }
    __syncthreads();
    int ox = 0, oy = 0, tx = 0, ty = 0;
    for (int k = 0; k < kSlices; k++) {
        if (k == sl) {
            ox = tx;
            oy = ty;
        }
        tx += 32 * slice_len[0][k];
        ty += 32 * slice_len[1][k];
    }
    const size_t slot0 = (size_t)blockIdx.x * kQT;
    q.slot[slot0 + at] = make_int2(i < nn && !lg ? i : -1, lg ? 0 : lx | (ly << 8));
    if ((at & 31) == 0) q.slice[blockIdx.x * kSlices + sl] = make_int2(ox, oy);
    if (i < nn)
        q.rel[i] = lg ? make_int2(bx + px - lx, by + py - ly) : make_int2(ox + (at & 31), oy + (at & 31));
    if (tid == 0) q.win[blockIdx.x] = Window{tx, ty, long_n, long_x, long_y, {0, 0, 0}};
}

// One movable node's row of both systems: counts (FILL = false: the
// partners only, no weights) or entries, diagonal and right-hand side
// (FILL = true).  A thread per node takes its pins'
// short partner sets in pin order; then the warp takes the long ones (a bound
// pin of a large net pairs with every other pin of it), in pin order, 32
// partners at a time, entries placed by a ballot prefix so they keep the
// partner order, the sums of the pairs' terms through a fixed xor tree.
template <bool FILL>
__global__ void __launch_bounds__(kQT)
k_qp_rows(int nn, const int32_t *__restrict__ obj_pin_start, const int32_t *__restrict__ obj_pin_dev,
          const int32_t *__restrict__ pin_net, const int32_t *__restrict__ first, const int32_t *__restrict__ deg,
          const int4 *__restrict__ bound, const int32_t *__restrict__ owner, const float2 *__restrict__ off,
          const float2 *__restrict__ abspin, int32_t *__restrict__ count, QpLayout lay,
          int2 *__restrict__ ent_x, int2 *__restrict__ ent_y, float2 *__restrict__ diag,
          float2 *__restrict__ rhs, const QpSolve *__restrict__ S) {
    constexpr bool fill = FILL;
    if (fill && S->overflow) return;  // uniform: the offsets exceed the allocation, the solve reports it
    const int i = blockIdx.x * blockDim.x + threadIdx.x, lane = threadIdx.x & 31;
    const bool valid = i < nn;  // every lane stays for the warp's long sets
    int cnt[2] = {0, 0};
    double dsum[2] = {0.0, 0.0}, bsum[2] = {0.0, 0.0};
    int row0[2] = {0, 0}, step = 1;
    if (fill) {
        const Window w = lay.win[blockIdx.x];
        const bool lg = valid && max(count[i], count[nn + i]) > kLongRow;
        const int2 rel = valid ? lay.rel[i] : make_int2(0, 0);
        row0[0] = (lg ? w.long_x : w.x) + rel.x;
        row0[1] = (lg ? w.long_y : w.y) + rel.y;
        step = lg ? 1 : 32;
        // the window's long rows in row order
        __shared__ int warp_long[kSlices];
        const unsigned m = __ballot_sync(0xffffffffu, lg);
        if (lane == 0) warp_long[threadIdx.x >> 5] = __popc(m);
        __syncthreads();
        if (lg) {
            int at = w.n_long + __popc(m & ((1u << lane) - 1));
            for (int k = 0; k < (int)(threadIdx.x >> 5); k++) at += warp_long[k];
            lay.longs[2 * at] = make_int4(i, row0[0], row0[1], count[i]);
            lay.longs[2 * at + 1] = make_int4(count[nn + i], 0, 0, 0);
        }
    }
    int2 *const ent[2] = {ent_x, ent_y};
    const int k0 = valid ? obj_pin_start[i] : 0, np_i = valid ? obj_pin_start[i + 1] - k0 : 0;
    auto entry = [&](int axis, int j, float w, int at) {
        if (fill) ent[axis][row0[axis] + at * step] = make_int2(j, __float_as_int(-w));
    };
    for (int k = k0; k < k0 + np_i; k++) {
        const int q = obj_pin_dev[k], n = pin_net[q], f = first[n], d = deg[n], a = q - f;
        const int4 bd = bound[n];
        const float c = (float)(1.0 / ((double)d - 1.0));
        const float2 pa = abspin[q], oa = off[q];
        PartnerRange rx, ry;
        const bool lx = range_x(a, d, bd.x, bd.y, rx) && is_long(rx);
        const bool ly = range_y(a, d, bd.z, bd.w, ry) && is_long(ry);
        if (!lx)
            partners_x(a, d, bd.x, bd.y, [&](int b) {
                if constexpr (FILL) {
                    float w;
                    const int j = pair_terms(i, nn, f + b, 0, owner, abspin, off, c, pa.x, oa.x, w, dsum[0], bsum[0]);
                    if (j >= 0) entry(0, j, w, cnt[0]++);
                } else if (pair_partner(i, nn, f + b, owner) >= 0) {
                    cnt[0]++;
                }
            });
        if (!ly)
            partners_y(a, d, bd.z, bd.w, [&](int b) {
                if constexpr (FILL) {
                    float w;
                    const int j = pair_terms(i, nn, f + b, 1, owner, abspin, off, c, pa.y, oa.y, w, dsum[1], bsum[1]);
                    if (j >= 0) entry(1, j, w, cnt[1]++);
                } else if (pair_partner(i, nn, f + b, owner) >= 0) {
                    cnt[1]++;
                }
            });
    }
    const int steps = __reduce_max_sync(0xffffffffu, np_i);
    for (int s = 0; s < steps; s++) {
        int q = 0, f = 0, d = 0;
        PartnerRange r[2] = {{0, -1, -1}, {0, -1, -1}};
        bool lg[2] = {false, false};
        if (s < np_i) {
            q = obj_pin_dev[k0 + s];
            const int n = pin_net[q];
            f = first[n];
            d = deg[n];
            const int4 bd = bound[n];
            lg[0] = range_x(q - f, d, bd.x, bd.y, r[0]) && is_long(r[0]);
            lg[1] = range_y(q - f, d, bd.z, bd.w, r[1]) && is_long(r[1]);
        }
        for (int axis = 0; axis < 2; axis++) {
            unsigned todo = __ballot_sync(0xffffffffu, lg[axis]);
            while (todo) {  // warp-uniform
                const int src = __ffs(todo) - 1;
                todo &= todo - 1;
                const int si = __shfl_sync(0xffffffffu, i, src), sq = __shfl_sync(0xffffffffu, q, src);
                const int sf = __shfl_sync(0xffffffffu, f, src), sd = __shfl_sync(0xffffffffu, d, src);
                const int end = __shfl_sync(0xffffffffu, r[axis].end, src);
                const int skip = __shfl_sync(0xffffffffu, r[axis].skip, src);
                const int extra = __shfl_sync(0xffffffffu, r[axis].extra, src);
                const int at0 = __shfl_sync(0xffffffffu, cnt[axis], src);
                const float c = (float)(1.0 / ((double)sd - 1.0));
                const float2 pa2 = abspin[sq], oa2 = off[sq];
                const float pa = axis ? pa2.y : pa2.x, oa = axis ? oa2.y : oa2.x;
                const int row = __shfl_sync(0xffffffffu, row0[axis], src);
                const int rstep = __shfl_sync(0xffffffffu, step, src);
                double ds = 0.0, bs = 0.0;
                int added = 0;
                for (int base = 0; base < end; base += 32) {
                    const int b = base + lane;
                    float w = 0.f;
                    int j = -1;
                    if (b < end && b != skip)
                        j = FILL ? pair_terms(si, nn, sf + b, axis, owner, abspin, off, c, pa, oa, w, ds, bs)
                                 : pair_partner(si, nn, sf + b, owner);
                    const unsigned m = __ballot_sync(0xffffffffu, j >= 0);
                    if (fill && j >= 0)
                        ent[axis][row + (at0 + added + __popc(m & ((1u << lane) - 1))) * rstep] =
                            make_int2(j, __float_as_int(-w));
                    added += __popc(m);
                }
                if (extra >= 0) {
                    int j = -1;
                    float w = 0.f;
                    if (lane == 0)
                        j = FILL ? pair_terms(si, nn, sf + extra, axis, owner, abspin, off, c, pa, oa, w, ds, bs)
                                 : pair_partner(si, nn, sf + extra, owner);
                    if (fill && j >= 0) ent[axis][row + (at0 + added) * rstep] = make_int2(j, __float_as_int(-w));
                    added += __shfl_sync(0xffffffffu, j >= 0 ? 1 : 0, 0);
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    ds += __shfl_xor_sync(0xffffffffu, ds, o);
                    bs += __shfl_xor_sync(0xffffffffu, bs, o);
                }
                if (lane == src) {
                    cnt[axis] += added;
                    dsum[axis] += ds;
                    bsum[axis] += bs;
                }
            }
        }
    }
    if (!fill) place_window(i, nn, cnt[0], cnt[1], lay);
    if (!valid) return;
    if (!fill) {
        count[i] = cnt[0];
        count[nn + i] = cnt[1];
    } else {
        diag[i] = make_float2((float)dsum[0], (float)dsum[1]);
        rhs[i] = make_float2((float)bsum[0], (float)bsum[1]);
    }
}

struct QpMat {
    const int2 *ent_x, *ent_y;
    QpLayout lay;
    const float2 *diag;
    int nn;
};

// The partial sums of a row of eight lanes, in its tree's order.
__device__ __forceinline__ float tree8(const float (&a)[8]) {
    return ((a[0] + a[4]) + (a[2] + a[6])) + ((a[1] + a[5]) + (a[3] + a[7]));
}

// (A_x v.x, A_y v.y) of every row i, and emit(i, result, pre), pre = before(i)
// loaded ahead of the row: a thread per row of a slice, a warp per long row
// (emit on its first lane).  The sums keep one order per row: eight partial
// sums over the entries k, k + 8, ... in order, added by a tree (a long row: 32,
// and a tree over the lanes), the diagonal last.  Bound by the latency of
// entry -> vector element: a thread has eight of each on either axis in flight
// where a lane of eight per row had one.  Three blocks an SM: 444 blocks sum
// fewer partials than 1184.  200k rows, 1.9M entries an axis, warm, us: SpMV
// 27 -> 17, an iteration (five kernels) 80 -> 47.
template <class Before, class Emit>
__device__ __forceinline__ void spmv_rows(const QpMat &m, const float2 *__restrict__ v, const QpSolve *__restrict__ S,
                                          Before &&before, Emit &&emit) {
    const int lane = threadIdx.x & 31, nn = m.nn;
    const int windows = (nn + kQT - 1) / kQT;
    const int n_long = S->n_long, units = S->overflow ? 0 : n_long + windows * kSlices;
    const int warps = (gridDim.x * blockDim.x) >> 5;
    for (int u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < units; u += warps) {  // warp-uniform
        if (u < n_long) {
            const int4 r = m.lay.longs[2 * u];
            const int lx = r.w, ly = m.lay.longs[2 * u + 1].x, len = max(lx, ly);
            float2 pre, d, vi;
            if (lane == 0) {
                pre = before(r.x);
                d = m.diag[r.x];
                vi = v[r.x];
            }
            float ax = 0.f, ay = 0.f;
#pragma unroll 4
            for (int k = lane; k < len; k += 32) {
                if (k < lx) {
                    const int2 e = m.ent_x[r.y + k];
                    ax = fmaf(__int_as_float(e.y), v[e.x].x, ax);
                }
                if (k < ly) {
                    const int2 e = m.ent_y[r.z + k];
                    ay = fmaf(__int_as_float(e.y), v[e.x].y, ay);
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                ax += __shfl_xor_sync(0xffffffffu, ax, o);
                ay += __shfl_xor_sync(0xffffffffu, ay, o);
            }
            if (lane == 0) emit(r.x, make_float2(fmaf(d.x, vi.x, ax), fmaf(d.y, vi.y, ay)), pre);
            continue;
        }
        // the longest slices of all windows first, so that a block's warps have
        // slices of about one length
        const int q = u - n_long, slice = q % windows * kSlices + kSlices - 1 - q / windows;
        const int2 slot = m.lay.slot[(size_t)slice * 32 + lane], rel = m.lay.slice[slice];
        const int2 first = *reinterpret_cast<const int2 *>(m.lay.win + slice / kSlices);  // x, y
        const int i = slot.x, lx = slot.y & 255, ly = slot.y >> 8;
        const bool mine = i >= 0;
        const int len = __reduce_max_sync(0xffffffffu, max(lx, ly));
        const float2 zero = make_float2(0.f, 0.f);
        const float2 pre = mine ? before(i) : zero, d = mine ? m.diag[i] : zero, vi = mine ? v[i] : zero;
        const int2 *ex = m.ent_x + first.x + rel.x + lane, *ey = m.ent_y + first.y + rel.y + lane;
        float sx[8], sy[8];
#pragma unroll
        for (int k = 0; k < 8; k++) sx[k] = sy[k] = 0.f;
        for (int k0 = 0; k0 < len; k0 += 8) {
            int2 a[8], b[8];
#pragma unroll
            for (int k = 0; k < 8; k++) {
                a[k] = k0 + k < lx ? ex[(k0 + k) * 32] : make_int2(-1, 0);
                b[k] = k0 + k < ly ? ey[(k0 + k) * 32] : make_int2(-1, 0);
            }
#pragma unroll
            for (int k = 0; k < 8; k++) {
                if (a[k].x >= 0) sx[k] = fmaf(__int_as_float(a[k].y), v[a[k].x].x, sx[k]);
                if (b[k].x >= 0) sy[k] = fmaf(__int_as_float(b[k].y), v[b[k].x].y, sy[k]);
            }
        }
        if (mine) emit(i, make_float2(fmaf(d.x, vi.x, tree8(sx)), fmaf(d.y, vi.y, tree8(sy))), pre);
    }
}

// ---- BiCGSTAB on the device -----------------------------------------------------
// Eigen's BiCGSTAB (van der Vorst's method, restart when r0.r vanishes,
// identity preconditioner) for both systems at once, every scalar of the
// recurrence kept in device memory (QpSolve) and updated by the finalising
// block of the grid reduction that produces its inputs; vector kernels read
// alpha, beta and omega from there.  Per axis c:
//   head     rho_old = rho; rho = r0.r; restart when |rho| < eps^2 r0sq
//            (in the finaliser of the previous step, or of the set-up)
//   restart  (only when flagged, launched by the host when it sees the flag)
//            r = b - A x, r0 = r; rho = r0sq = |r|^2, the iteration count reset
//            at the first restart
//   dir      p = r + beta (p - omega v), beta = (rho / rho_old)(alpha / omega)
//   av       v = A p; alpha = rho / (r0.v)
//   s        s = r - alpha v
//   at       t = A s; omega = t.s / t.t (0 when t.t = 0)
//   step     x += alpha p + omega s; r = s - omega t; |r|^2, r0.r; count;
//            the axis stays active while |r|^2 > (eps |b|)^2 and the count
//            is below the limit
// An inactive axis uses alpha = beta = omega = 0 (its x and r stay), and
// every kernel returns at once when neither axis is active, so iterations
// can be enqueued ahead of the convergence test.
// Neither axis stopped, and no restart owed: the kernels of the iterations
// already enqueued wait (return at once) until the host has launched it.
__device__ __forceinline__ bool any_active(const QpSolve *S) { return S->active[0] || S->active[1]; }
__device__ __forceinline__ bool running(const QpSolve *S) { return any_active(S) && !S->restart_mask; }

// The head of an iteration (rho_old = rho; rho = r0.r; the restart test),
// run by the finaliser that ends the previous iteration (or the set-up).
__device__ __forceinline__ void qp_pre(QpSolve *S) {
    if (!any_active(S)) return;
    const double eps = 1.1920928955078125e-07, eps2 = eps * eps;
    int restart = 0;
    for (int c = 0; c < 2; c++) {
        S->rho_old[c] = S->rho[c];
        if (!S->active[c]) continue;
        S->rho[c] = S->r0r[c];
        if (fabs(S->rho[c]) < eps2 * S->r0sq[c]) restart |= 1 << c;
    }
    S->restart_mask = restart;
}

// r = b - A x, r0 = r, p = v = 0; |r|^2 and |b|^2 per system, then the
// solver's initial state.
__global__ void __launch_bounds__(kQT, kSolveBlocks / 148)
k_qp_init(int nn, QpMat m, const float2 *__restrict__ rhs, const float2 *__restrict__ x, float2 *__restrict__ r,
          float2 *__restrict__ r0, float2 *__restrict__ p, float2 *__restrict__ v, double *__restrict__ partials,
          unsigned *__restrict__ cnt, int max_it, QpSolve *__restrict__ G) {
    __shared__ double sh[4 * 32];
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    spmv_rows(m, x, G, [&](int i) { return rhs[i]; }, [&](int i, float2 ax, float2 bi) {
        const float2 ri = make_float2(bi.x - ax.x, bi.y - ax.y);
        r[i] = ri;
        r0[i] = ri;
        p[i] = make_float2(0.f, 0.f);
        v[i] = make_float2(0.f, 0.f);
        acc[0] += (double)ri.x * ri.x;
        acc[1] += (double)ri.y * ri.y;
        acc[2] += (double)bi.x * bi.x;
        acc[3] += (double)bi.y * bi.y;
    });
    if (!grid_arrive<4>(acc, sh, partials, cnt, gridDim.x, blockIdx.x)) return;
    grid_total<4>(acc, sh, partials, cnt, gridDim.x);
    if (threadIdx.x == 0) {
        QpSolve s = *G, *S = &s;
        const double eps = 1.1920928955078125e-07, eps2 = eps * eps;
        S->zero_mask = 0;
        S->restart_mask = 0;
        S->iters = 0;
        for (int c = 0; c < 2; c++) {
            S->rr[c] = acc[c];
            S->bb[c] = acc[2 + c];
            S->r0sq[c] = acc[c];
            S->r0r[c] = acc[c];
            S->rho[c] = S->alpha[c] = S->w[c] = 1.0;
            S->it[c] = 0;
            S->restarts[c] = 0;
            S->tol2[c] = eps2 * S->bb[c];
            if (S->bb[c] == 0.0) {  // x = 0 (Eigen returns at once)
                S->zero_mask |= 1 << c;
                S->rr[c] = 0.0;
                S->active[c] = 0;
            } else {
                S->active[c] = S->rr[c] > S->tol2[c] && max_it > 0;
            }
        }
        S->max_it = max_it;
        qp_pre(S);
        *G = s;
    }
}

// A zero right-hand side gives x = 0.
__global__ void k_qp_zero(int nn, const QpSolve *__restrict__ S, float2 *__restrict__ x) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nn || !S->zero_mask) return;
    if (S->zero_mask & 1) x[i].x = 0.f;
    if (S->zero_mask & 2) x[i].y = 0.f;
}



// Restart of the flagged systems: r = b - A x, r0 = r; rho = r0sq = |r|^2.
__global__ void __launch_bounds__(kQT, kSolveBlocks / 148)
k_qp_restart(int nn, QpMat m, const float2 *__restrict__ rhs, const float2 *__restrict__ x, float2 *__restrict__ r,
             float2 *__restrict__ r0, double *__restrict__ partials, unsigned *__restrict__ cnt,
             QpSolve *__restrict__ S) {
    __shared__ double sh[2 * 32];
    pdl_begin();
    const int mask = S->restart_mask;
    double acc[2] = {0.0, 0.0};
    spmv_rows(m, x, S, [&](int i) { return rhs[i]; }, [&](int i, float2 ax, float2 bi) {
        float2 ri = r[i], zi = r0[i];
        if (mask & 1) ri.x = zi.x = bi.x - ax.x;
        if (mask & 2) ri.y = zi.y = bi.y - ax.y;
        r[i] = ri;
        r0[i] = zi;
        acc[0] += (double)ri.x * ri.x;
        acc[1] += (double)ri.y * ri.y;
    });
    if (!grid_arrive<2>(acc, sh, partials, cnt, gridDim.x, blockIdx.x)) return;
    grid_total<2>(acc, sh, partials, cnt, gridDim.x);
    if (threadIdx.x == 0) {
        for (int c = 0; c < 2; c++)
            if (mask & (1 << c)) {
                S->rho[c] = S->r0sq[c] = acc[c];
                if (S->restarts[c]++ == 0) S->it[c] = 0;
            }
        S->restart_mask = 0;
    }
}

// Rows 2 k and 2 k + 1 of a vector (allocated to an even number of rows).
__device__ __forceinline__ float4 pair(const float2 *v, int k) { return reinterpret_cast<const float4 *>(v)[k]; }
__device__ __forceinline__ void set_pair(float2 *v, int k, float4 a) { reinterpret_cast<float4 *>(v)[k] = a; }

// p = r + beta (p - omega v); with a diagonal preconditioner (dinv, else
// null) also y = M^-1 p, the vector the SpMV then takes
__global__ void __launch_bounds__(kQT)
k_qp_dir(int nn, const float2 *__restrict__ r, const float2 *__restrict__ v, float2 *__restrict__ p,
         const float2 *__restrict__ dinv, float2 *__restrict__ y, const QpSolve *__restrict__ S) {
    pdl_begin();
    if (!running(S)) return;
    float b[2], w[2];
    for (int c = 0; c < 2; c++) {
        b[c] = S->active[c] ? (float)((S->rho[c] / S->rho_old[c]) * (S->alpha[c] / S->w[c])) : 0.f;
        w[c] = S->active[c] ? (float)S->w[c] : 0.f;
    }
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (nn + 1) / 2) return;
    const float4 ri = pair(r, t), vi = pair(v, t), pi = pair(p, t);
    const float4 pn = make_float4(ri.x + b[0] * (pi.x - w[0] * vi.x), ri.y + b[1] * (pi.y - w[1] * vi.y),
                                  ri.z + b[0] * (pi.z - w[0] * vi.z), ri.w + b[1] * (pi.w - w[1] * vi.w));
    set_pair(p, t, pn);
    if (dinv) {
        const float4 d = pair(dinv, t);
        set_pair(y, t, make_float4(pn.x * d.x, pn.y * d.y, pn.z * d.z, pn.w * d.w));
    }
}

// v = A p; alpha = rho / (r0.v)
__global__ void __launch_bounds__(kQT, kSolveBlocks / 148)
k_qp_av(int nn, QpMat m, const float2 *__restrict__ p, const float2 *__restrict__ r0, float2 *__restrict__ v,
        double *__restrict__ partials, unsigned *__restrict__ cnt, QpSolve *__restrict__ S) {
    __shared__ double sh[2 * 32];
    pdl_begin();
    if (!running(S)) return;
    double acc[2] = {0.0, 0.0};
    spmv_rows(m, p, S, [&](int i) { return r0[i]; }, [&](int i, float2 vi, float2 z) {
        v[i] = vi;
        acc[0] += (double)z.x * vi.x;
        acc[1] += (double)z.y * vi.y;
    });
    if (!grid_arrive<2>(acc, sh, partials, cnt, gridDim.x, blockIdx.x)) return;
    const double rho[2] = {S->rho[0], S->rho[1]};
    const int active[2] = {S->active[0], S->active[1]};
    grid_total<2>(acc, sh, partials, cnt, gridDim.x);
    if (threadIdx.x == 0)
        for (int c = 0; c < 2; c++) S->alpha[c] = active[c] ? rho[c] / acc[c] : 0.0;
}

// s = r - alpha v; with the preconditioner also z = M^-1 s
__global__ void __launch_bounds__(kQT)
k_qp_s(int nn, const float2 *__restrict__ r, const float2 *__restrict__ v, float2 *__restrict__ s,
       const float2 *__restrict__ dinv, float2 *__restrict__ z, const QpSolve *__restrict__ S) {
    pdl_begin();
    if (!running(S)) return;
    const float ax = (float)S->alpha[0], ay = (float)S->alpha[1];
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= (nn + 1) / 2) return;
    const float4 ri = pair(r, t), vi = pair(v, t);
    const float4 si = make_float4(ri.x - ax * vi.x, ri.y - ay * vi.y, ri.z - ax * vi.z, ri.w - ay * vi.w);
    set_pair(s, t, si);
    if (dinv) {
        const float4 d = pair(dinv, t);
        set_pair(z, t, make_float4(si.x * d.x, si.y * d.y, si.z * d.z, si.w * d.w));
    }
}

// t = A z (z = s, or M^-1 s); omega = t.s / t.t
__global__ void __launch_bounds__(kQT, kSolveBlocks / 148)
k_qp_at(int nn, QpMat m, const float2 *__restrict__ z, const float2 *__restrict__ s, float2 *__restrict__ t,
        double *__restrict__ partials, unsigned *__restrict__ cnt, QpSolve *__restrict__ S) {
    __shared__ double sh[4 * 32];
    pdl_begin();
    if (!running(S)) return;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    spmv_rows(m, z, S, [&](int i) { return s[i]; }, [&](int i, float2 ti, float2 si) {
        t[i] = ti;
        acc[0] += (double)ti.x * ti.x;
        acc[1] += (double)ti.y * ti.y;
        acc[2] += (double)ti.x * si.x;
        acc[3] += (double)ti.y * si.y;
    });
    if (!grid_arrive<4>(acc, sh, partials, cnt, gridDim.x, blockIdx.x)) return;
    const int active[2] = {S->active[0], S->active[1]};
    grid_total<4>(acc, sh, partials, cnt, gridDim.x);
    if (threadIdx.x == 0)
        for (int c = 0; c < 2; c++)
            if (active[c]) S->w[c] = acc[c] > 0.0 ? acc[2 + c] / acc[c] : 0.0;
}

// x += alpha y + omega z (y, z = p, s, or their preconditioned forms);
// r = s - omega t; |r|^2, r0.r; convergence per axis.
__global__ void __launch_bounds__(kQT)
k_qp_step(int nn, const float2 *__restrict__ p, const float2 *__restrict__ zs, const float2 *__restrict__ s,
          const float2 *__restrict__ t, const float2 *__restrict__ r0, float2 *__restrict__ x, float2 *__restrict__ r,
          double *__restrict__ partials, unsigned *__restrict__ cnt, QpSolve *__restrict__ S) {
    __shared__ double sh[4 * 32];
    pdl_begin();
    if (!running(S)) return;
    float a[2], w[2];
    for (int c = 0; c < 2; c++) {
        a[c] = S->active[c] ? (float)S->alpha[c] : 0.f;
        w[c] = S->active[c] ? (float)S->w[c] : 0.f;
    }
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    for (int k = blockIdx.x * blockDim.x + threadIdx.x; k < (nn + 1) / 2; k += gridDim.x * blockDim.x) {
        const float4 pi = pair(p, k), zi = pair(zs, k), si = pair(s, k), ti = pair(t, k), xi = pair(x, k), z = pair(r0, k);
        set_pair(x, k, make_float4(xi.x + a[0] * pi.x + w[0] * zi.x, xi.y + a[1] * pi.y + w[1] * zi.y,
                                   xi.z + a[0] * pi.z + w[0] * zi.z, xi.w + a[1] * pi.w + w[1] * zi.w));
        const float4 ri = make_float4(si.x - w[0] * ti.x, si.y - w[1] * ti.y, si.z - w[0] * ti.z, si.w - w[1] * ti.w);
        set_pair(r, k, ri);
        acc[0] += (double)ri.x * ri.x;
        acc[1] += (double)ri.y * ri.y;
        acc[2] += (double)z.x * ri.x;
        acc[3] += (double)z.y * ri.y;
        if (2 * k + 1 < nn) {  // the last row's pair holds no row
            acc[0] += (double)ri.z * ri.z;
            acc[1] += (double)ri.w * ri.w;
            acc[2] += (double)z.z * ri.z;
            acc[3] += (double)z.w * ri.w;
        }
    }
    if (!grid_arrive<4>(acc, sh, partials, cnt, gridDim.x, blockIdx.x)) return;
    QpSolve h = *S;  // the finaliser works on a copy
    grid_total<4>(acc, sh, partials, cnt, gridDim.x);
    if (threadIdx.x == 0) {
        h.iters++;
        for (int c = 0; c < 2; c++) {
            if (!h.active[c]) continue;
            h.rr[c] = acc[c];
            h.r0r[c] = acc[2 + c];
            h.it[c]++;
            h.active[c] = h.rr[c] > h.tol2[c] && h.it[c] < h.max_it;
        }
        qp_pre(&h);
        *S = h;
    }
}

// Node centres <-> solution vector (setModuleCenter_2D clamp on the way back).
__global__ void k_qp_to_x(int nn, const float2 *__restrict__ pos, float2 *__restrict__ x) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nn) x[i] = pos[i];
}

__global__ void k_qp_from_x(Grid g, int nn, const float2 *__restrict__ x, const float2 *__restrict__ size,
                            float2 *__restrict__ pos) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nn) pos[i] = clamp_center<float>(g, x[i], size[i]);
}

// PlaceDB::moveNodesCenterToCenter (PlaceDB/placedb.cpp:591-598).
__global__ void k_qp_center(Grid g, int nn, const float2 *__restrict__ size, float2 *__restrict__ pos) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < nn) {
        const float2 c = make_float2((float)(0.5 * ((double)g.urx + (double)g.llx)),
                                     (float)(0.5 * ((double)g.ury + (double)g.lly)));
        pos[i] = clamp_center<float>(g, c, size[i]);
    }
}

}  // namespace

void qp_bounds(const QpDev &q, const float2 *pos, double *hpwl, cudaStream_t st) {
    k_qp_bounds<<<qgrid(31 * q.n_big + q.nnet), kQT, 0, st>>>(q.nnet, q.n_big, q.net_order, q.net_first, q.net_deg,
                                                               q.owner, q.off, pos, q.bound, q.abspin, q.partials,
                                                               q.cnt, hpwl);
}

static int windows(int nn) { return qblocks(nn); }
// The layout arrays in one block of memory.
size_t qp_layout_bytes(int nn) {
    const size_t w = windows(nn);
    return w * (sizeof(Window) + kSlices * sizeof(int2) + kQT * (2 * sizeof(int2) + 2 * sizeof(int4)));
}
static QpLayout layout(const QpDev &q) {
    const size_t w = windows(q.nn);
    QpLayout l;
    l.win = static_cast<Window *>(q.layout);
    l.longs = reinterpret_cast<int4 *>(l.win + w);
    l.slot = reinterpret_cast<int2 *>(l.longs + 2 * w * kQT);
    l.rel = l.slot + w * kQT;
    l.slice = l.rel + w * kQT;
    return l;
}
// Entries an axis can need, the smaller of two bounds.  A net of d pins gives an
// axis fewer than 4 d entries (its counted pairs involve one of its two bound
// pins), and no slice is longer than kLongRow.  Or: of a pin's entries on either
// axis, the more, there are d - 1 for the at most four bound pins of its net and
// two for the others; m, their sum over a row, is at least the row's sort key and
// the length of its longer axis.  In a window a slice's length is at most every m
// of the slice after it (its long rows included, as their places in the order
// are), and the last one's at most kLongRow.  So the slices take at most the sum
// of min(m, kLongRow) over the window's rows and a slice of kLongRow; the long
// rows' own entries count at most 31 of them twice.  200k cells and 788k pins:
// 63 MB for both axes, 153 by the first bound alone.
size_t qp_entry_cap(int nn, const int32_t *deg, int nnet) {
    size_t pins = 0, most = 0;
    for (int n = 0; n < nnet; n++) {
        const size_t d = deg[n];
        pins += d;
        most += d > 4 ? 4 * (d - 1) + 2 * (d - 4) : d * (d - 1) * (d > 0);
    }
    const size_t w = windows(nn);
    return std::min(w * kQT * kLongRow + 4 * pins, w * 2 * 32 * kLongRow + most) + 16;
}

void qp_rows(const QpDev &q, int fill, cudaStream_t st) {
    (fill ? k_qp_rows<true> : k_qp_rows<false>)<<<qblocks(q.nn), kQT, 0, st>>>(
        q.nn, q.obj_pin_start, q.obj_pin_dev, q.pin_net, q.net_first, q.net_deg, q.bound, q.owner, q.off, q.abspin,
        q.count, layout(q), q.ent_x, q.ent_y, q.diag, q.rhs, q.solve);
}

void qp_scan(const QpDev &q, cudaStream_t st) {
    k_qp_scan<<<1, kScanThreads, 0, st>>>(windows(q.nn), layout(q).win, q.cap_x, q.cap_y, q.solve);
}

static QpMat mat(const QpDev &q) { return QpMat{q.ent_x, q.ent_y, layout(q), q.diag, q.nn}; }

// Grids that depend on the sizes alone, so that the dot products group alike on
// every run: the SpMV kernels' with warps to spare for the long rows of a small
// design.
static int spmv_grid(int nn) { return std::min(2 * qblocks(nn), kSolveBlocks); }

void qp_init(const QpDev &q, int max_it, cudaStream_t st) {
    k_qp_init<<<spmv_grid(q.nn), kQT, 0, st>>>(q.nn, mat(q), q.rhs, q.x, q.r, q.r0, q.p, q.v, q.partials,
                                                         q.cnt, max_it, q.solve);
    k_qp_zero<<<qblocks(q.nn), kQT, 0, st>>>(q.nn, q.solve, q.x);
}

// M^-1 of the Jacobi preconditioner: 1 / diagonal (1 where the diagonal is 0)
__global__ void k_qp_dinv(int nn, const float2 *__restrict__ diag, float2 *__restrict__ dinv) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nn) return;
    const float2 d = diag[i];
    dinv[i] = make_float2(d.x != 0.f ? 1.f / d.x : 1.f, d.y != 0.f ? 1.f / d.y : 1.f);
}

void qp_restart(const QpDev &q, cudaStream_t st) {
    launch_k(k_qp_restart, spmv_grid(q.nn), kQT, 0, st, q.nn, mat(q), q.rhs, q.x, q.r, q.r0, q.partials, q.cnt,
             q.solve);
}

void qp_iterations(const QpDev &q, int count, bool jacobi, cudaStream_t st) {
    const int b = qblocks((q.nn + 1) / 2), bm = spmv_grid(q.nn), br = std::min(b, kSolveBlocks);
    for (int k = 0; k < count; k++) {
        // programmatic serialisation: each kernel's blocks are resident and
        // waiting (pdl_begin) while the previous one drains.  Eigen's
        // preconditioned form: y = M^-1 p and z = M^-1 s go into the SpMVs and
        // the update; without a preconditioner y = p and z = s
        const float2 *dinv = jacobi ? q.dinv : nullptr;
        const float2 *y = jacobi ? q.y : q.p, *z = jacobi ? q.z : q.s;
        launch_k(k_qp_dir, b, kQT, 0, st, q.nn, q.r, q.v, q.p, dinv, q.y, q.solve);
        launch_k(k_qp_av, bm, kQT, 0, st, q.nn, mat(q), y, q.r0, q.v, q.partials, q.cnt, q.solve);
        launch_k(k_qp_s, b, kQT, 0, st, q.nn, q.r, q.v, q.s, dinv, q.z, q.solve);
        launch_k(k_qp_at, bm, kQT, 0, st, q.nn, mat(q), z, q.s, q.t, q.partials, q.cnt, q.solve);
        launch_k(k_qp_step, br, kQT, 0, st, q.nn, y, z, q.s, q.t, q.r0, q.x, q.r, q.partials, q.cnt, q.solve);
    }
}

void qp_dinv(const QpDev &q, cudaStream_t st) { k_qp_dinv<<<qblocks(q.nn), kQT, 0, st>>>(q.nn, q.diag, q.dinv); }

void qp_to_x(const QpDev &q, const float2 *pos, cudaStream_t st) {
    k_qp_to_x<<<qblocks(q.nn), kQT, 0, st>>>(q.nn, pos, q.x);
}

void qp_from_x(const QpDev &q, const Grid &g, const float2 *size, float2 *pos, cudaStream_t st) {
    k_qp_from_x<<<qblocks(q.nn), kQT, 0, st>>>(g, q.nn, q.x, size, pos);
}

void qp_center(const QpDev &q, const Grid &g, const float2 *size, float2 *pos, cudaStream_t st) {
    k_qp_center<<<qblocks(q.nn), kQT, 0, st>>>(g, q.nn, size, pos);
}

int qp_partial_blocks(int nn, int nnet) { return kQpMaxBlocks; }

}  // namespace ep
