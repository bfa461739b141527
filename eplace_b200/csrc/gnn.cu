// gnn.cu -- the learned warm start: a small message-passing network over the
// cell-net incidence that proposes the initial placement in place of the
// quadratic placement (QPPlacer::quadraticPlacement, QPlace/qplace.cpp:20-103),
// which stays the fallback and the judge.  No counterpart in the reference.
//
// Graph: the movable nodes (0..nn-1) and the terminals (nn..nn+nt-1) of an
// engine, read from the engine's device arrays (nets contiguous in device
// pin order, each object's pins through its object -> pin map); a net joins
// the nodes of its pins.  Two mean aggregations:
//   net_mean   a[n] = mean over the pins of net n of h[node(pin)]
//   node_mean  m[c] = mean over the pins of movable node c of a[net(pin)]
//                     (terminals receive nothing: m = 0)
//
// Features (kF per node, from the netlist alone, computed on the device):
// log(1 + area) / 4, log(1 + pins) / 3, terminal flag, and the node's
// coordinates (normalised to the core) after 8, 32 and 128 steps of
// pad-anchored diffusion: every movable node starts at the core centre,
// terminals sit at their own centres, and a step replaces each movable node
// by node_mean(net_mean(.)).  These are the fixed-pin distances the network
// reads: a node's diffused coordinate says how its pads pull it, at three
// ranges; d, the 128-step coordinates, is the base of the predictions.
//
// Network (hidden 64, weights stored BF16 for the forward pass, FP32
// accumulate, FP32 master weights for training):
//   h0 = relu(W0 x + b0)
//   h_l = relu(W_l [h_{l-1} ; node_mean(net_mean(h_{l-1}))] + b_l),  l = 1..3
//   q = d + 0.25 tanh(W4[0:2] h3 + b4[0:2])   the engine's quadratic placement
//   f = d + 0.25 tanh(W4[2:4] h3 + b4[2:4])   the engine's final mGP placement
// (normalised core coordinates).  Training: the mean squared error of both
// heads against the engine's own quadratic placement and final placement of
// the design, Adam; every reduction (weight gradients, loss) is a per-block
// partial summed in a fixed order, so a training step is bitwise repeatable.
// A proposal moves the movable nodes to q + alpha (f - q), mapped to the
// core: the quadratic placement's compact layout moved part of the way to
// where the optimizer ends.
#include <cuda_bf16.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <random>
#include <vector>

#include "engine.h"
#include "tc_ptx.cuh"

namespace ep {
namespace {

constexpr int kH = 64;      // hidden width
constexpr int kF = 9;       // input features
constexpr int kOut = 4;     // q (x, y), f (x, y)
constexpr int kLayers = 3;  // message-passing layers
constexpr int kDiff1 = 8, kDiff2 = 32, kDiff3 = 128;  // diffusion steps of the three coordinate features
constexpr float kCorr = 0.25f;  // bound of a head's correction, in core sizes

// Parameter layout (floats): W0[kH][kF], b0[kH], per layer W[kH][2kH], b[kH],
// then W4[kOut][kH], b4[kOut].
constexpr int kOffW0 = 0, kOffB0 = kOffW0 + kH * kF, kOffL = kOffB0 + kH;
constexpr int kLayerParams = kH * 2 * kH + kH;
constexpr int kOffW4 = kOffL + kLayers * kLayerParams, kOffB4 = kOffW4 + kOut * kH;
constexpr int kParams = kOffB4 + kOut;
inline int off_w(int l) { return kOffL + (l - 1) * kLayerParams; }
inline int off_b(int l) { return off_w(l) + kH * 2 * kH; }

constexpr int kT = 256;
inline int nblk(long long n, int t = kT) { return (int)((n + t - 1) / t); }

// Device view of the bound netlist.
struct Net {
    int nn, n_obj, N, nnet;
    const int32_t *owner, *net_first, *net_deg, *pin_net, *obj_pin_start, *obj_pin_dev;
    const int32_t *net_order;            // nets in device pin order (neighbouring nets of equal degree)
    int n_big;                           // nets above kWarpPins pins: the head of net_order
    const int32_t *pad_start, *pad_net;  // terminals' pins (training only; may be null)
    // flattened indices, built once per bound netlist (k_graph_index):
    const int4 *kinfo;        // [nnet] per net in device order: first pin, degree, 1/degree (bits), net
    const int32_t *pin_node;  // [np] node (0..N-1) of each device pin
    const int32_t *q_net;     // [pins of movable nodes] net of each pin, in object pin order
};

__device__ __forceinline__ int node_of(int o, int nn, int n_obj) { return o < nn ? o : nn + (o - n_obj); }
__device__ __forceinline__ float bf(const __nv_bfloat16 v) { return __bfloat162float(v); }

// ------------------------------------------------------------ features ----
template <typename R>
__global__ void k_init(Net g, const float *__restrict__ area, const float *__restrict__ npins,
                       const vec2<R> *__restrict__ pos, Grid gr, float *__restrict__ X, float2 *__restrict__ v,
                       float *__restrict__ inv_pins) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= g.N) return;
    float *x = X + (size_t)c * kF;
#pragma unroll
    for (int k = 0; k < kF; k++) x[k] = 0.f;
    if (c < g.nn) {
        x[0] = log1pf(area[c]) * 0.25f;
        x[1] = log1pf(npins[c]) * (1.f / 3.f);
        v[c] = make_float2(0.5f, 0.5f);
        inv_pins[c] = npins[c] > 0.f ? 1.f / npins[c] : 0.f;
    } else {
        const vec2<R> t = pos[g.n_obj + (c - g.nn)];
        x[2] = 1.f;
        v[c] = make_float2((float)(((double)t.x - gr.llx) / ((double)gr.urx - gr.llx)),
                           (float)(((double)t.y - gr.lly) / ((double)gr.ury - gr.lly)));
        inv_pins[c] = 0.f;
    }
}

__global__ void k_pad_pins(int np, Net g, int *__restrict__ cnt) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < np && g.owner[p] >= g.n_obj) atomicAdd(&cnt[g.owner[p] - g.n_obj], 1);
}

__global__ void k_pad_feature(int nt, int nn, const int *__restrict__ cnt, float *__restrict__ X) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < nt) X[(size_t)(nn + t) * kF + 1] = log1pf((float)cnt[t]) * (1.f / 3.f);
}

// The terminals' pin lists (the transposed aggregation into terminals reads
// them; training only): their starts by one block from the counts, the pins in
// any order, then each list in pin order (a block per terminal, k_pad_sort).
__global__ void __launch_bounds__(kT) k_pad_start(int nt, const int *__restrict__ cnt, int32_t *__restrict__ start,
                                                  int *__restrict__ cursor) {
    __shared__ int tot[kT / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int carry = 0;
    for (int t0 = 0; t0 < nt; t0 += kT) {
        const int t = t0 + threadIdx.x, v = t < nt ? cnt[t] : 0;
        int x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        __syncthreads();
        if (lane == 31) tot[w] = x;
        __syncthreads();
        int before = carry;
        for (int k = 0; k < kT / 32; k++) {
            if (k < w) before += tot[k];
            carry += tot[k];
        }
        if (t < nt) start[t] = cursor[t] = before + x - v;
    }
    if (threadIdx.x == 0) start[nt] = carry;
}

__global__ void k_pad_fill(int np, Net g, int *__restrict__ cursor, int32_t *__restrict__ pins) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p < np && g.owner[p] >= g.n_obj) pins[atomicAdd(&cursor[g.owner[p] - g.n_obj], 1)] = p;
}

// A list of L of the np pins: by counting the smaller pins of each while L^2 <=
// kPadScan np, else by walking all pins in order and keeping its own, so that no
// list costs more than a walk or so (a fixed macro may have 100k pins).  Measured
// for one list, counting / walking, us: 200k pins, L = 1000 58 / 95, 2000 193 /
// 104; 788k pins, 2000 193 / 341, 4000 691 / 348, 64000 410000 / 646; the same
// for 200 lists at once to a third.
constexpr int kPadScan = 10;
__global__ void __launch_bounds__(kT) k_pad_sort(Net g, int np, const int32_t *__restrict__ start,
                                                 const int32_t *__restrict__ pins, int32_t *__restrict__ nets) {
    const int b = start[blockIdx.x], e = start[blockIdx.x + 1];
    if ((long long)(e - b) * (e - b) <= (long long)kPadScan * np) {
        for (int i = b + threadIdx.x; i < e; i += kT) {
            const int p = pins[i];
            int rank = 0;
#pragma unroll 8
            for (int j = b; j < e; j++) rank += pins[j] < p;
            nets[b + rank] = g.pin_net[p];
        }
        return;
    }
    constexpr int kU = 8;  // pins of a thread in flight
    __shared__ int found[2][kU][kT / 32];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, owner = g.n_obj + blockIdx.x;
    int at = b, buf = 0;
    for (unsigned p0 = 0; p0 < (unsigned)np && at < e; p0 += kU * kT, buf ^= 1) {  // block-uniform
        unsigned m[kU];
#pragma unroll
        for (int u = 0; u < kU; u++) {
            const unsigned p = p0 + u * kT + threadIdx.x;
            m[u] = p < (unsigned)np && g.owner[p] == owner;
        }
#pragma unroll
        for (int u = 0; u < kU; u++) {
            m[u] = __ballot_sync(0xffffffffu, m[u]);
            if (lane == 0) found[buf][u][w] = __popc(m[u]);
        }
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kU; u++) {
            int before = 0, all = 0;
#pragma unroll
            for (int k = 0; k < kT / 32; k++) {
                const int c = found[buf][u][k];
                if (k < w) before += c;
                all += c;
            }
            if (m[u] >> lane & 1)
                nets[at + before + __popc(m[u] & ((1u << lane) - 1))] = g.pin_net[p0 + u * kT + threadIdx.x];
            at += all;
        }
    }
}

// Targets normalised to the core in place; terminals (c >= nn) have none.
__global__ void k_target(int N, int nn, float llx, float lly, float w, float h, float4 *__restrict__ t) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= N) return;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c < nn) {
        v = t[c];
        v = make_float4(__fdiv_rn(__fsub_rn(v.x, llx), w), __fdiv_rn(__fsub_rn(v.y, lly), h),
                        __fdiv_rn(__fsub_rn(v.z, llx), w), __fdiv_rn(__fsub_rn(v.w, lly), h));
    }
    t[c] = v;
}

__global__ void k_inv_deg(int nnet, const int32_t *__restrict__ deg, float *__restrict__ inv) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n < nnet) inv[n] = deg[n] > 0 ? 1.f / deg[n] : 0.f;
}

// The aggregations' index arrays, one level of indirection shallower than
// the engine's: kinfo[k] for the k-th net of the device order (its first
// pin, degree, 1/degree as in k_inv_deg, id), the node of every pin, and the
// net of every pin of a movable node in object pin order.  Launched with
// max(nnet, np) threads.
__global__ void k_graph_index(Net g, int np, int4 *__restrict__ kinfo, int32_t *__restrict__ pin_node,
                              int32_t *__restrict__ q_net) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t < g.nnet) {
        const int n = g.net_order[t], d = g.net_deg[n];
        kinfo[t] = make_int4(g.net_first[n], d, __float_as_int(d > 0 ? 1.f / d : 0.f), n);
    }
    if (t < np) pin_node[t] = node_of(g.owner[t], g.nn, g.n_obj);
    if (t < g.obj_pin_start[g.nn]) q_net[t] = g.pin_net[g.obj_pin_dev[t]];
}

// The nets above kWarpPins pins (the head of the device order) take a warp
// each: lane l sums pins l, l + 32, ... and a fixed xor tree adds the lanes.
// Every other net takes a thread, in device order, so a warp's nets have the
// same degree.  Launched with 32 n_big + (nnet - n_big) threads.
__global__ void k_diff_net(Net g, const float2 *__restrict__ v, float2 *__restrict__ a) {
    pdl_begin();
    const int t = blockIdx.x * blockDim.x + threadIdx.x, big = g.n_big * 32;
    if (t < big) {  // whole warps
        const int4 r = g.kinfo[t >> 5];
        const int lane = t & 31;
        float sx = 0.f, sy = 0.f;
        for (int p = r.x + lane, e = r.x + r.y; p < e; p += 32) {
            const float2 q = v[g.pin_node[p]];
            sx += q.x;
            sy += q.y;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            sx += __shfl_xor_sync(0xffffffffu, sx, o);
            sy += __shfl_xor_sync(0xffffffffu, sy, o);
        }
        const float inv = __int_as_float(r.z);
        if (lane == 0) a[r.w] = make_float2(sx * inv, sy * inv);
        return;
    }
    const int k = g.n_big + (t - big);
    if (k >= g.nnet) return;
    const int4 r = g.kinfo[k];
    float sx = 0.f, sy = 0.f;
#pragma unroll 4
    for (int p = r.x, e = r.x + r.y; p < e; p++) {
        const float2 q = v[g.pin_node[p]];
        sx += q.x;
        sy += q.y;
    }
    const float inv = __int_as_float(r.z);
    a[r.w] = make_float2(sx * inv, sy * inv);
}

__global__ void k_diff_node(Net g, const float *__restrict__ inv_pins, const float2 *__restrict__ a,
                            float2 *__restrict__ v) {
    pdl_begin();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= g.nn) return;
    const int q0 = g.obj_pin_start[c], q1 = g.obj_pin_start[c + 1];
    if (q1 == q0) return;
    float sx = 0.f, sy = 0.f;
#pragma unroll 4
    for (int q = q0; q < q1; q++) {
        const float2 t = a[g.q_net[q]];
        sx += t.x;
        sy += t.y;
    }
    v[c] = make_float2(sx * inv_pins[c], sy * inv_pins[c]);
}

__global__ void k_store_feature(int N, const float2 *__restrict__ v, float *__restrict__ X, int col) {
    pdl_begin();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= N) return;
    X[(size_t)c * kF + col] = v[c].x;
    X[(size_t)c * kF + col + 1] = v[c].y;
}

// ---- the diffusion as one launch -----------------------------------------------
// 256 dependent passes of a few microseconds: launched one by one they cost 4.2
// us each however small the design.  Here a CTA per SM keeps its share of the
// indices in shared memory for all of them -- a run of nets and a run of movable
// nodes, cut so that every CTA has about the same number of pins -- and the CTAs
// meet at a barrier in global memory after each pass (a cooperative launch, so
// they are resident together).  In a pass all threads gather their CTA's pin
// values into shared memory, every load in flight at once (the barrier's acquire
// is what makes the L1 fetch them anew), and then a thread per row (a warp per net above kWarpPins
// pins) adds them in the order of k_diff_net and k_diff_node: the same sums bit
// for bit.  Taken when the share fits (kDiffSmem); the pass-by-pass kernels above
// stay for larger designs and devices without cooperative launches.  128 steps,
// us: 2k cells 1050 -> 590, 50k 1190 -> 790, 200k 1910 -> 1400.
constexpr int kDiffThreads = 1024;
constexpr size_t kDiffSmem = 216 * 1024;

struct DiffShare {  // pins a CTA's share can have (net phase, node phase)
    int net_pins, node_pins;
};
__host__ __device__ __forceinline__ size_t diff_smem(DiffShare s) {
    const int most = max(s.net_pins, s.node_pins);
    return sizeof(float2) * ((size_t)most + most / 16 + 1) + sizeof(int32_t) * ((size_t)s.net_pins + s.node_pins);
}
// Place of pin i's value: skewed, so that the threads of a warp, whose rows start
// 2, 4, ... 32 pins apart, read different banks.
__device__ __forceinline__ int skew(int i) { return i + (i >> 4); }

// First k in [0, n) whose key(k) >= x (keys ascending), n if there is none.
template <class Key>
__device__ __forceinline__ int first_at_least(int n, int x, Key &&key) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) >> 1;
        if (key(mid) >= x)
            hi = mid;
        else
            lo = mid + 1;
    }
    return lo;
}

// All CTAs have written what they wrote before it; false when the wait gave up
// (the default limit is a second or two).
__device__ __forceinline__ bool grid_barrier(unsigned *count, unsigned target, unsigned limit) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(count) : "memory");
        unsigned left = limit, v = 0;
        while (left > 0) {
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(count) : "memory");
            if (v >= target) break;
            left--;
        }
        ok = left > 0;
    }
    __syncthreads();
    return ok != 0;
}

__device__ __forceinline__ void gather_pins(const int32_t *__restrict__ idx, int n, const float2 *src,
                                            float2 *__restrict__ val) {
#pragma unroll 8
    for (int i = threadIdx.x; i < n; i += kDiffThreads) val[skew(i)] = src[idx[i]];
    __syncthreads();
}

__global__ void __launch_bounds__(kDiffThreads, 1)
k_diffuse(Net g, int np, DiffShare share, const float *__restrict__ inv_pins, float2 *v, float2 *a,
          float *__restrict__ X, unsigned *__restrict__ count, unsigned limit, int *__restrict__ status,
          int *__restrict__ engine_status) {
    extern __shared__ __align__(16) unsigned char diff_sm[];
    float2 *val = reinterpret_cast<float2 *>(diff_sm);
    int32_t *net_idx = reinterpret_cast<int32_t *>(val + skew(max(share.net_pins, share.node_pins)) + 1);
    int32_t *node_idx = net_idx + share.net_pins;
    __shared__ int cut[4];
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, G = gridDim.x, b = blockIdx.x;
    const int nq = g.obj_pin_start[g.nn];
    if (tid < 2)  // nets [cut 0, cut 1): those whose first pin lies in this CTA's run of pins
        cut[tid] = b + tid == G ? g.nnet
                                : first_at_least(g.nnet, (int)((long long)np * (b + tid) / G), [&](int k) { return g.kinfo[k].x; });
    else if (tid < 4)  // nodes [cut 2, cut 3) likewise
        cut[tid] = b + tid - 2 == G ? g.nn
                                    : first_at_least(g.nn, (int)((long long)nq * (b + tid - 2) / G),
                                                     [&](int c) { return g.obj_pin_start[c]; });
    __syncthreads();
    const int k0 = cut[0], k1 = cut[1], c0 = cut[2], c1 = cut[3];
    const int p0 = k0 < g.nnet ? g.kinfo[k0].x : np, p1 = k1 < g.nnet ? g.kinfo[k1].x : np;
    const int q0 = g.obj_pin_start[c0], q1 = g.obj_pin_start[c1];
    for (int i = tid; i < p1 - p0; i += kDiffThreads) net_idx[i] = g.pin_node[p0 + i];
    for (int i = tid; i < q1 - q0; i += kDiffThreads) node_idx[i] = g.q_net[q0 + i];
    // the terminals' coordinates stay
    for (int c = g.nn + b * kDiffThreads + tid; c < g.N; c += G * kDiffThreads)
#pragma unroll
        for (int j = 0; j < 3; j++) {
            X[(size_t)c * kF + 3 + 2 * j] = v[c].x;
            X[(size_t)c * kF + 4 + 2 * j] = v[c].y;
        }
    const int kb = min(max(g.n_big, k0), k1);  // nets [k0, kb) of this CTA take a warp each
    // a thread's first rows, the same in every step
    constexpr int kKept = 2;
    int4 net[kKept];
    int node_s[kKept], node_e[kKept];
    float node_inv[kKept];
#pragma unroll
    for (int u = 0; u < kKept; u++) {
        const int k = kb + tid + u * kDiffThreads, c = c0 + tid + u * kDiffThreads;
        net[u] = k < k1 ? g.kinfo[k] : make_int4(0, 0, 0, 0);
        node_s[u] = c < c1 ? g.obj_pin_start[c] - q0 : 0;
        node_e[u] = c < c1 ? g.obj_pin_start[c + 1] - q0 : 0;
        node_inv[u] = c < c1 ? inv_pins[c] : 0.f;
    }
    __syncthreads();
    unsigned target = 0;
    bool ok = true;
    for (int step = 1; step <= kDiff3; step++) {
        gather_pins(net_idx, p1 - p0, v, val);
        for (int k = k0 + wid; k < kb; k += kDiffThreads / 32) {
            const int4 r = g.kinfo[k];
            float sx = 0.f, sy = 0.f;
            for (int p = r.x - p0 + lane, e = r.x - p0 + r.y; p < e; p += 32) {
                const float2 t = val[skew(p)];
                sx += t.x;
                sy += t.y;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                sx += __shfl_xor_sync(0xffffffffu, sx, o);
                sy += __shfl_xor_sync(0xffffffffu, sy, o);
            }
            const float inv = __int_as_float(r.z);
            if (lane == 0) a[r.w] = make_float2(sx * inv, sy * inv);
        }
        auto sum_net = [&](const int4 r) {
            float sx = 0.f, sy = 0.f;
#pragma unroll 4
            for (int p = r.x - p0, e = p + r.y; p < e; p++) {
                const float2 t = val[skew(p)];
                sx += t.x;
                sy += t.y;
            }
            const float inv = __int_as_float(r.z);
            a[r.w] = make_float2(sx * inv, sy * inv);
        };
#pragma unroll
        for (int u = 0; u < kKept; u++)
            if (kb + tid + u * kDiffThreads < k1) sum_net(net[u]);
        for (int k = kb + tid + kKept * kDiffThreads; k < k1; k += kDiffThreads) sum_net(g.kinfo[k]);
        ok = grid_barrier(count, target += G, limit);
        if (!ok) break;
        gather_pins(node_idx, q1 - q0, a, val);
        const int col = step == kDiff1 ? 3 : step == kDiff2 ? 5 : step == kDiff3 ? 7 : 0;
        auto sum_node = [&](int c, int s, int e, float inv) {
            float2 t = make_float2(0.5f, 0.5f);  // a node on no net stays at the centre
            if (e > s) {
                float sx = 0.f, sy = 0.f;
#pragma unroll 4
                for (int q = s; q < e; q++) {
                    const float2 w = val[skew(q)];
                    sx += w.x;
                    sy += w.y;
                }
                t = make_float2(sx * inv, sy * inv);
                v[c] = t;
            }
            if (col) {
                X[(size_t)c * kF + col] = t.x;
                X[(size_t)c * kF + col + 1] = t.y;
            }
        };
#pragma unroll
        for (int u = 0; u < kKept; u++) {
            const int c = c0 + tid + u * kDiffThreads;
            if (c < c1) sum_node(c, node_s[u], node_e[u], node_inv[u]);
        }
        for (int c = c0 + tid + kKept * kDiffThreads; c < c1; c += kDiffThreads)
            sum_node(c, g.obj_pin_start[c] - q0, g.obj_pin_start[c + 1] - q0, inv_pins[c]);
        if (step == kDiff3) break;
        ok = grid_barrier(count, target += G, limit);
        if (!ok) break;
    }
    if (!ok && tid == 0) {
        *(volatile int *)status = 1;  // mapped host memory: a plain store
        atomicOr(engine_status, 1 << EP_ERR_TIMEOUT);
    }
}

// ------------------------------------------------------ aggregations ------
// Half a warp per row, a float4 of channels per lane, and the rows of four
// pins in flight: a pin costs two dependent loads (its row's number, the row),
// and most rows have two to five pins, so a warp that summed one row pin after
// pin waited for the L2 most of the time.  A warp per row before, us: at 200k
// cells k_net_mean 52.2 -> 32.5 and k_node_mean 52.6 -> 41.4, at 50k
// k_node_mean_t 29.0 -> 15.1 and k_net_mean_t_add 16.2 -> 14.7 (18.9 with the
// row's load behind its weight's).  What bounds them now is the L2's rate (256
// bytes a pin) and, at 200k, writing the 51 MB of rows.
// The nets above kWarpPins pins take the first n_big blocks of the per-net
// passes, a block each (warp w sums pins w, w + 8, ..., with a float2 per
// lane; the 8 warp sums are added in warp order).
constexpr int kHalf = 16;  // lanes per row

// Sum of rows idx[p], idx[p + 1], ..., idx[e - 1] of h, in that order, without
// the rows from `limit` on; row i times weight[i] (Scaled).
template <bool Scaled>
__device__ __forceinline__ float4 sum_rows(const int32_t *__restrict__ idx, int p, int e, int limit,
                                           const float4 *__restrict__ h, int lane, const float *__restrict__ weight) {
    constexpr int kU = 4;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    for (; p < e; p += kU) {
        int i[kU];
        float w[kU];
        float4 t[kU];
#pragma unroll
        for (int u = 0; u < kU; u++) i[u] = p + u < e ? idx[p + u] : limit;
#pragma unroll
        for (int u = 0; u < kU; u++) {
            if (i[u] < limit) {
                t[u] = h[(size_t)i[u] * kHalf + lane];
                if (Scaled) w[u] = weight[i[u]];
            }
        }
#pragma unroll
        for (int u = 0; u < kU; u++) {
            if (i[u] < limit) {
                s.x += Scaled ? t[u].x * w[u] : t[u].x;
                s.y += Scaled ? t[u].y * w[u] : t[u].y;
                s.z += Scaled ? t[u].z * w[u] : t[u].z;
                s.w += Scaled ? t[u].w * w[u] : t[u].w;
            }
        }
    }
    return s;
}

constexpr int kBigWarps = kT / 32;
__global__ void __launch_bounds__(kT) k_net_mean(Net g, const float2 *__restrict__ h,
                                                 float2 *__restrict__ a) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if ((int)blockIdx.x < g.n_big) {
        __shared__ float2 part[kBigWarps][32];
        const int4 r = g.kinfo[blockIdx.x];
        const int n = r.w;
        float2 s = make_float2(0.f, 0.f);
        for (int p = r.x + w, e = r.x + r.y; p < e; p += kBigWarps) {
            const float2 q = h[(size_t)g.pin_node[p] * 32 + lane];
            s.x += q.x;
            s.y += q.y;
        }
        part[w][lane] = s;
        __syncthreads();
        if (w == 0) {
            float2 t = part[0][lane];
            for (int k = 1; k < kBigWarps; k++) {
                t.x += part[k][lane].x;
                t.y += part[k][lane].y;
            }
            const float inv = __int_as_float(r.z);
            a[(size_t)n * 32 + lane] = make_float2(t.x * inv, t.y * inv);
        }
        return;
    }
    const int k = g.n_big + ((int)blockIdx.x - g.n_big) * (kT / kHalf) + (int)threadIdx.x / kHalf;
    if (k >= g.nnet) return;
    const int4 r = g.kinfo[k];
    const int l = threadIdx.x & (kHalf - 1);
    const float4 s = sum_rows<false>(g.pin_node, r.x, r.x + r.y, g.N, (const float4 *)h, l, nullptr);
    const float inv = __int_as_float(r.z);
    ((float4 *)a)[(size_t)r.w * kHalf + l] = make_float4(s.x * inv, s.y * inv, s.z * inv, s.w * inv);
}

__global__ void k_node_mean(Net g, const float *__restrict__ inv_pins, const float4 *__restrict__ a,
                            float4 *__restrict__ m) {
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) / kHalf, l = threadIdx.x & (kHalf - 1);
    if (c >= g.N) return;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    if (c < g.nn) {
        const float inv = inv_pins[c];
        s = sum_rows<false>(g.q_net, g.obj_pin_start[c], g.obj_pin_start[c + 1], g.nnet, a, l, nullptr);
        s = make_float4(s.x * inv, s.y * inv, s.z * inv, s.w * inv);
    }
    m[(size_t)c * kHalf + l] = s;
}

// transpose of node_mean: da[n] = sum over the pins of n on movable nodes c of
// dm[c] / pins(c); nets above kWarpPins pins a block each, as in k_net_mean
__device__ __forceinline__ void add_scaled(float2 &s, float2 t, float w) {
    s.x += t.x * w;
    s.y += t.y * w;
}
__global__ void __launch_bounds__(kT) k_node_mean_t(Net g, const float *__restrict__ inv_pins,
                                                    const float2 *__restrict__ dm, float2 *__restrict__ da) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if ((int)blockIdx.x < g.n_big) {
        const int4 r = g.kinfo[blockIdx.x];
        float2 s = make_float2(0.f, 0.f);
#pragma unroll 4
        for (int p = r.x + w, e = r.x + r.y; p < e; p += kBigWarps) {
            const int c = g.pin_node[p];
            if (c < g.nn) add_scaled(s, dm[(size_t)c * 32 + lane], inv_pins[c]);
        }
        __shared__ float2 part[kBigWarps][32];
        part[w][lane] = s;
        __syncthreads();
        if (w != 0) return;
        for (int j = 1; j < kBigWarps; j++) {
            s.x += part[j][lane].x;
            s.y += part[j][lane].y;
        }
        da[(size_t)r.w * 32 + lane] = s;
        return;
    }
    const int k = g.n_big + ((int)blockIdx.x - g.n_big) * (kT / kHalf) + (int)threadIdx.x / kHalf;
    if (k >= g.nnet) return;
    const int4 r = g.kinfo[k];
    const int l = threadIdx.x & (kHalf - 1);
    ((float4 *)da)[(size_t)r.w * kHalf + l] = sum_rows<true>(g.pin_node, r.x, r.x + r.y, g.nn, (const float4 *)dm, l,
                                                                    inv_pins);
}

// transpose of net_mean, added: dh[c] += sum over the pins of node c of da[net] / deg(net)
__global__ void k_net_mean_t_add(Net g, const float *__restrict__ inv_deg, const float4 *__restrict__ da,
                                 float4 *__restrict__ dh) {
    const int c = (blockIdx.x * blockDim.x + threadIdx.x) / kHalf, l = threadIdx.x & (kHalf - 1);
    if (c >= g.N) return;
    const bool node = c < g.nn;
    const int32_t *start = node ? g.obj_pin_start + c : g.pad_start + (c - g.nn);
    const float4 s = sum_rows<true>(node ? g.q_net : g.pad_net, start[0], start[1], g.nnet, da, l, inv_deg);
    float4 &o = dh[(size_t)c * kHalf + l];
    float4 v = o;
    o = make_float4(v.x + s.x, v.y + s.y, v.z + s.z, v.w + s.w);
}

// ------------------------------------------------------------ dense -------
// Y[r][o] = relu(b[o] + sum_k X[r][k] W[o][k]) with X = [XA (KA cols) | XB
// (KB cols)], W the BF16 weights, read here from their FP32 transposed copy
// Wt[k][o] (k_transpose_w).  kDenseRows rows per 256-thread block: Wt and
// the block's rows (row-major, padded to K + 1) staged in shared memory;
// thread (tx, ty) accumulates rows 4 ty .. 4 ty + 3 x outputs 8 tx .. 8 tx + 7
// in registers, k in order (two 16-byte weight loads and four row loads per
// 32 FMAs, without bank conflicts), so each output is the same sum as a
// plain loop over k.
constexpr int kDenseRows = 128;
template <int KA, int KB>
__global__ void __launch_bounds__(kT) k_dense(int N, const float *__restrict__ XA, const float *__restrict__ XB,
                                              const float *__restrict__ Wt, const float *__restrict__ b,
                                              float *__restrict__ Y) {
    constexpr int K = KA + KB, XP = K + 1;
    extern __shared__ float sm[];
    float *Ws = sm;            // [K][kH]
    float *Xs = sm + K * kH;   // [kDenseRows][XP]
    for (int i = threadIdx.x; i < K * kH / 4; i += kT)
        reinterpret_cast<float4 *>(Ws)[i] = reinterpret_cast<const float4 *>(Wt)[i];
    const int r0 = blockIdx.x * kDenseRows;
    for (int i = threadIdx.x; i < kDenseRows * K; i += kT) {
        const int r = i / K, k = i - r * K, row = r0 + r;
        float v = 0.f;
        if (row < N) v = k < KA ? XA[(size_t)row * KA + k] : XB[(size_t)row * KB + (k - KA)];
        Xs[r * XP + k] = v;
    }
    __syncthreads();
    const int tx = threadIdx.x & 7, ty = threadIdx.x >> 3;
    const float4 *W4 = reinterpret_cast<const float4 *>(Ws);
    float acc[4][8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
        const float bj = b[tx * 8 + j];
#pragma unroll
        for (int i = 0; i < 4; i++) acc[i][j] = bj;
    }
#pragma unroll 4
    for (int k = 0; k < K; k++) {
        float x[4];
#pragma unroll
        for (int i = 0; i < 4; i++) x[i] = Xs[(ty * 4 + i) * XP + k];
        const float4 wa = W4[k * (kH / 4) + tx * 2], wb = W4[k * (kH / 4) + tx * 2 + 1];
        const float w[8] = {wa.x, wa.y, wa.z, wa.w, wb.x, wb.y, wb.z, wb.w};
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 8; j++) acc[i][j] = fmaf(x[i], w[j], acc[i][j]);
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int row = r0 + ty * 4 + i;
        if (row >= N) continue;
        float4 *y = reinterpret_cast<float4 *>(Y + (size_t)row * kH + tx * 8);
        y[0] = make_float4(fmaxf(acc[i][0], 0.f), fmaxf(acc[i][1], 0.f), fmaxf(acc[i][2], 0.f), fmaxf(acc[i][3], 0.f));
        y[1] = make_float4(fmaxf(acc[i][4], 0.f), fmaxf(acc[i][5], 0.f), fmaxf(acc[i][6], 0.f), fmaxf(acc[i][7], 0.f));
    }
}

// The input layer's BF16 weights as FP32, transposed to [k][o], for k_dense.
constexpr int kWtSize = kF * kH;
__global__ void k_transpose_w(const __nv_bfloat16 *__restrict__ wb, float *__restrict__ wt) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= kWtSize) return;
    const int k = i / kH, o = i % kH;
    wt[i] = bf(wb[kOffW0 + o * kF + k]);
}

// ------------------------------------------------------ dense, tcgen05 ----
// The hidden layers (K = 2 kH = 128 inputs [XA | XB], kH = 64 outputs) on
// the tensor cores: Y = relu(b + [XA | XB] W^T).  Each FP32 input is split
// into two BF16 planes, hi = bf16(x) and lo = bf16(x - hi) (hi + lo holds x
// to 2^-17 relative), and both are multiplied by the BF16 weights (exact in
// BF16) with tcgen05.mma.kind::f16, FP32 accumulators in tensor memory.  A
// persistent CTA of 256 threads (two per SM) takes 128-row tiles in turn:
//   all threads  load the tile's rows (coalesced float4), split them and
//                store both planes in shared memory in the K-major,
//                128-byte-swizzled layout of the MMA descriptors;
//   thread 0     issues 16 MMAs (2 K blocks x 4 steps of 16 x 2 planes) and
//                commits them to an mbarrier;
//   all threads  wait (bounded), read the accumulators (warp w: TMEM lanes
//                32 (w % 4) .. + 31 = tile rows, columns 32 (w / 4) .. + 31),
//                add the bias, relu, stage the tile in shared memory (over the
//                consumed planes) and store it row-major with coalesced float4
//                stores.
// The next tile's loads are in flight during a tile's MMAs and epilogue.  The
// weights (64 x 128 BF16) are staged once per CTA.  A wait that gives up sets
// its flag in *status (and EP_ERR_TIMEOUT in the engine's word); the CTA
// waits for its own MMAs (bounded) before it frees its tensor memory.
constexpr int kTcRows = 128, kTcThreads = 256, kTcKB = 2;
constexpr int kTcWBlock = kH * 128;                 // one K block of W: 64 rows x 128 B
constexpr int kTcABlock = kTcRows * 128;            // one K block of one input plane
constexpr int kTcW = kTcKB * kTcWBlock;             // 16 KB
constexpr int kTcA = 2 * kTcKB * kTcABlock;         // hi and lo planes, 64 KB
constexpr int kTcLd = kH + 4;                       // staging row stride, floats
constexpr int kTcLoads = kTcRows * 32 / kTcThreads;  // float4 loads per thread and tile
constexpr int kTcCols = 64;                         // TMEM columns
static_assert(kTcRows * kTcLd * 4 <= kTcA, "the staged tile fits over the input planes");
constexpr size_t kTcSmem = 1024 + kTcW + kTcA + 64;

// Byte offset of element k (0..63) of row r in a K-major block with the
// 128-byte swizzle: 8-row x 128-byte atoms 1024 bytes apart, the 16-byte
// chunk index XOR-ed with the row inside the atom.
__device__ __forceinline__ uint32_t sw128(int r, int k) {
    return (uint32_t)((r >> 3) * 1024 + (r & 7) * 128 + (((k >> 3) ^ (r & 7)) << 4) + (k & 7) * 2);
}

__device__ __forceinline__ uint32_t pack_bf16(uint16_t a, uint16_t b) { return (uint32_t)a | ((uint32_t)b << 16); }

__global__ void __launch_bounds__(kTcThreads, 2)
k_dense_tc(int N, const float *__restrict__ XA, const float *__restrict__ XB, const __nv_bfloat16 *__restrict__ W,
           const float *__restrict__ b, float *__restrict__ Y, int *__restrict__ status, int *__restrict__ engine_status,
           unsigned wait_limit) {
    extern __shared__ uint8_t smem_raw[];
    uint8_t *smem = (uint8_t *)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint8_t *Ws = smem, *As = smem + kTcW;
    float *stage = (float *)As;
    uint64_t *bar = (uint64_t *)(As + kTcA);
    volatile uint32_t *tmem_slot = (volatile uint32_t *)(bar + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        tc::mbar_init(bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(tc::smem_u32((const void *)tmem_slot)), "r"(kTcCols));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    // weights: row o, K block kb, 16-byte chunk j (8 BF16)
    for (int i = tid; i < kH * kTcKB * 8; i += kTcThreads) {
        const int o = i >> 4, kb = (i >> 3) & 1, j = i & 7;
        const uint4 v = *reinterpret_cast<const uint4 *>(W + (size_t)o * 2 * kH + kb * 64 + j * 8);
        *reinterpret_cast<uint4 *>(Ws + kb * kTcWBlock + sw128(o, j * 8)) = v;
    }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;
    const int ntiles = (N + kTcRows - 1) / kTcRows;
    const int kb_l = lane >> 4, k_l = (lane & 15) * 4;  // this lane's K block and first K of its float4
    const float *src = kb_l ? XB : XA;
    uint32_t phase = 0;
    bool ok = true;
    // warp w, load i: row 8 i + w of a tile (a warp reads one row: XA's 64
    // floats in lanes 0-15, XB's in lanes 16-31); rows past N (and tiles past
    // the last) read as zeros
    float4 v[kTcLoads];
    auto load_tile = [&](int t) {
#pragma unroll
        for (int i = 0; i < kTcLoads; i++) {
            const int gr = t * kTcRows + i * 8 + warp;
            v[i] = gr < N ? __ldg(reinterpret_cast<const float4 *>(src + (size_t)gr * kH + k_l))
                          : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    load_tile(blockIdx.x);
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int r0 = tile * kTcRows;
#pragma unroll
        for (int i = 0; i < kTcLoads; i++) {
            const int row = i * 8 + warp;
            uint16_t h[4], l[4];
            tc::bf16_split(v[i].x, h[0], l[0]);
            tc::bf16_split(v[i].y, h[1], l[1]);
            tc::bf16_split(v[i].z, h[2], l[2]);
            tc::bf16_split(v[i].w, h[3], l[3]);
            const uint32_t off = kb_l * kTcABlock + sw128(row, k_l);
            *reinterpret_cast<uint2 *>(As + off) = make_uint2(pack_bf16(h[0], h[1]), pack_bf16(h[2], h[3]));
            *reinterpret_cast<uint2 *>(As + kTcKB * kTcABlock + off) =
                make_uint2(pack_bf16(l[0], l[1]), pack_bf16(l[2], l[3]));
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
        if (tid == 0) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t idesc = tc::umma_idesc(kTcRows, kH);
            const uint32_t a = tc::smem_u32(As), w = tc::smem_u32(Ws);
#pragma unroll
            for (int kb = 0; kb < kTcKB; kb++)
#pragma unroll
                for (int k = 0; k < 4; k++) {
                    const uint32_t ao = kb * kTcABlock + k * 32, wo = kb * kTcWBlock + k * 32;
                    tc::umma_bf16(tmem, tc::umma_desc(a + ao), tc::umma_desc(w + wo), idesc, (kb | k) != 0);
                    tc::umma_bf16(tmem, tc::umma_desc(a + kTcKB * kTcABlock + ao), tc::umma_desc(w + wo), idesc, 1);
                }
            tc::umma_commit(bar);
        }
        load_tile(tile + gridDim.x);  // the next tile's rows in flight during the MMAs and the epilogue
        // lane 0 of each warp waits; the CTA goes on only if every warp saw
        // the commit (a uniform decision, so no barrier is left half-reached)
        int got = 1;
        if (lane == 0) {
            got = 0;
            for (unsigned it = 0; it < wait_limit; it++)
                if (tc::mbar_try_wait(bar, phase)) {
                    got = 1;
                    break;
                }
        }
        got = __shfl_sync(0xffffffffu, got, 0);
        ok = __syncthreads_and(got) != 0;
        if (!ok) break;
        phase ^= 1;
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        {
            const int q = warp & 3, ch = warp >> 2, row = q * 32 + lane;
            const uint32_t taddr = tmem + ((uint32_t)(q * 32) << 16) + (uint32_t)(ch * 32);
#pragma unroll
            for (int c0 = 0; c0 < 32; c0 += 16) {
                uint32_t r[16];
                tc::tmem_ld16(taddr + (uint32_t)c0, r);
#pragma unroll
                for (int j = 0; j < 16; j += 4) {
                    const int col = ch * 32 + c0 + j;
                    float4 o;
                    o.x = fmaxf(__uint_as_float(r[j]) + __ldg(b + col), 0.f);
                    o.y = fmaxf(__uint_as_float(r[j + 1]) + __ldg(b + col + 1), 0.f);
                    o.z = fmaxf(__uint_as_float(r[j + 2]) + __ldg(b + col + 2), 0.f);
                    o.w = fmaxf(__uint_as_float(r[j + 3]) + __ldg(b + col + 3), 0.f);
                    *reinterpret_cast<float4 *>(stage + row * kTcLd + col) = o;
                }
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
#pragma unroll
        for (int i = 0; i < kTcRows * 16 / kTcThreads; i++) {
            const int u = i * kTcThreads + tid, row = u >> 4, c4 = u & 15, gr = r0 + row;
            if (gr < N)
                *reinterpret_cast<float4 *>(Y + (size_t)gr * kH + c4 * 4) =
                    *reinterpret_cast<const float4 *>(stage + row * kTcLd + c4 * 4);
        }
        __syncthreads();  // the staged rows are read before the next tile's planes overwrite them
    }
    if (!ok && tid == 0) {
        // the MMAs of the tile in flight complete before the tensor memory is freed
        for (unsigned it = 0; it < tc::kWaitLimit && !tc::mbar_try_wait(bar, phase); it++) {
        }
        *(volatile int *)status = 1;  // mapped host memory: a plain store
        if (engine_status) atomicOr(engine_status, 1 << EP_ERR_TIMEOUT);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 0) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTcCols));
    }
}

// Launched as clusters of one CTA, like the tensor-core Poisson GEMMs.
void launch_dense_tc(int grid, cudaStream_t st, int N, const float *XA, const float *XB, const __nv_bfloat16 *W,
                     const float *b, float *Y, int *status, int *engine_status, unsigned wait_limit) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kTcThreads);
    cfg.dynamicSmemBytes = kTcSmem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k_dense_tc, N, XA, XB, W, b, Y, status, engine_status, wait_limit);
}

// ------------------------------------------------- dense, backward --------
// FP32 on the CUDA cores: gradients stay in 32 bits, and the hidden
// layers' two products (0.82 GFLOP each at 50k nodes) are 14 us of FP32 FMAs.
// One output per thread and two shared-memory reads per FMA made them 258 and
// 323 us; a thread now holds 4 x 8 outputs and reads 3 (or 5) 16-byte vectors
// per 32 FMAs, the next tile's rows in flight meanwhile.  50k nodes, us: dX
// 258 -> 28, dW 323 -> 30.
constexpr int kDxRows = 64;                       // rows of a tile
constexpr int kDwRows = 32;
constexpr int kDwBlocks = 148 * 2;                // partial weight gradients, at most
constexpr size_t kDxSmem = sizeof(float) * (kH * 2 * kH + kDxRows * kH);

__device__ __forceinline__ float4 relu_mask(float4 d, float4 y) {
    return make_float4(y.x > 0.f ? d.x : 0.f, y.y > 0.f ? d.y : 0.f, y.z > 0.f ? d.z : 0.f, y.w > 0.f ? d.w : 0.f);
}
__device__ __forceinline__ void fma4(float4 &a, float s, float4 w) {
    a.x = fmaf(s, w.x, a.x);
    a.y = fmaf(s, w.y, a.y);
    a.z = fmaf(s, w.z, a.z);
    a.w = fmaf(s, w.w, a.w);
}

// dX = (dY .* (Y > 0)) W of a hidden layer, split into dXA and dXB (kH columns
// each).  Blocks take tiles of kDxRows rows in turn, W (FP32) staged once; thread
// (tx, ty): rows 4 ty .. 4 ty + 3, columns 4 tx .. 4 tx + 3 of each half; every
// output adds o = 0 .. 63 in order.
__global__ void __launch_bounds__(kT) k_dense_dx(int N, const float *__restrict__ dY, const float *__restrict__ Y,
                                                 const __nv_bfloat16 *__restrict__ W, float *__restrict__ dXA,
                                                 float *__restrict__ dXB) {
    extern __shared__ float4 sm4[];
    float4 *Ws = sm4;                        // [kH][2 kH / 4]
    float4 *Zs = sm4 + kH * 2 * kH / 4;      // [kDxRows][kH / 4]
    for (int i = threadIdx.x; i < kH * 2 * kH / 4; i += kT) {
        const __nv_bfloat16 *w = W + 4 * i;
        Ws[i] = make_float4(bf(w[0]), bf(w[1]), bf(w[2]), bf(w[3]));
    }
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int tiles = (N + kDxRows - 1) / kDxRows;
    constexpr int kPer = kDxRows * (kH / 4) / kT;  // float4 of a tile per thread
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 d[kPer], y[kPer];
    auto load = [&](int tile) {
#pragma unroll
        for (int u = 0; u < kPer; u++) {
            const int i = threadIdx.x + u * kT, row = tile * kDxRows + (i >> 4);
            const size_t at = (size_t)row * (kH / 4) + (i & 15);
            d[u] = row < N ? reinterpret_cast<const float4 *>(dY)[at] : zero;
            y[u] = row < N ? reinterpret_cast<const float4 *>(Y)[at] : zero;
        }
    };
    load(blockIdx.x);
    for (int tile = blockIdx.x; tile < tiles; tile += gridDim.x) {
        __syncthreads();  // the tile before has been read (first: nothing)
#pragma unroll
        for (int u = 0; u < kPer; u++) Zs[threadIdx.x + u * kT] = relu_mask(d[u], y[u]);
        __syncthreads();
        load(tile + gridDim.x);
        float4 a[4], b[4];
#pragma unroll
        for (int i = 0; i < 4; i++) a[i] = b[i] = zero;
#pragma unroll 4
        for (int o4 = 0; o4 < kH / 4; o4++) {
            float z[4][4];
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float4 v = Zs[(4 * ty + i) * (kH / 4) + o4];
                z[i][0] = v.x;
                z[i][1] = v.y;
                z[i][2] = v.z;
                z[i][3] = v.w;
            }
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const float4 wa = Ws[(4 * o4 + j) * (2 * kH / 4) + tx], wb = Ws[(4 * o4 + j) * (2 * kH / 4) + 16 + tx];
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    fma4(a[i], z[i][j], wa);
                    fma4(b[i], z[i][j], wb);
                }
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int row = tile * kDxRows + 4 * ty + i;
            if (row >= N) continue;
            reinterpret_cast<float4 *>(dXA)[(size_t)row * (kH / 4) + tx] = a[i];
            reinterpret_cast<float4 *>(dXB)[(size_t)row * (kH / 4) + tx] = b[i];
        }
    }
}

// Rows [rb, re) of a block's partial weight gradient: equal runs of whole tiles.
__device__ __forceinline__ void dw_rows(int N, int &rb, int &re) {
    const int tiles = (N + kDwRows - 1) / kDwRows, per = (tiles + gridDim.x - 1) / gridDim.x;
    rb = min(N, (int)blockIdx.x * per * kDwRows);
    re = min(N, rb + per * kDwRows);
}

// Per-block partial weight gradient of a hidden layer: P[o][k] = sum_r Z[r][o]
// X[r][k] and P[kH 2kH + o] = sum_r Z[r][o] over the block's rows, Z = dY .* (Y >
// 0), X = [XA | XB].  Thread (tx, ty): outputs 4 ty .. 4 ty + 3 x columns 4 tx ..
// of each half, rows in order.
__global__ void __launch_bounds__(kT, 2) k_dw_hidden(int N, const float *__restrict__ dY, const float *__restrict__ Y,
                                                     const float *__restrict__ XA, const float *__restrict__ XB,
                                                     float *__restrict__ partial) {
    __shared__ float4 Zs[kDwRows][kH / 4], As[kDwRows][kH / 4], Bs[kDwRows][kH / 4];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    int rb, re;
    dw_rows(N, rb, re);
    constexpr int kPer = kDwRows * (kH / 4) / kT;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    float4 d[kPer], y[kPer], xa[kPer], xb[kPer];
    auto load = [&](int t0) {
#pragma unroll
        for (int u = 0; u < kPer; u++) {
            const int i = threadIdx.x + u * kT, row = t0 + (i >> 4);
            const size_t at = (size_t)row * (kH / 4) + (i & 15);
            const bool in = row < re;
            d[u] = in ? reinterpret_cast<const float4 *>(dY)[at] : zero;
            y[u] = in ? reinterpret_cast<const float4 *>(Y)[at] : zero;
            xa[u] = in ? reinterpret_cast<const float4 *>(XA)[at] : zero;
            xb[u] = in ? reinterpret_cast<const float4 *>(XB)[at] : zero;
        }
    };
    float4 a[4], b[4];
    float bias[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int i = 0; i < 4; i++) a[i] = b[i] = zero;
    load(rb);
    for (int t0 = rb; t0 < re; t0 += kDwRows) {
        __syncthreads();
#pragma unroll
        for (int u = 0; u < kPer; u++) {
            const int i = threadIdx.x + u * kT;
            (&Zs[0][0])[i] = relu_mask(d[u], y[u]);
            (&As[0][0])[i] = xa[u];
            (&Bs[0][0])[i] = xb[u];
        }
        __syncthreads();
        load(t0 + kDwRows);
#pragma unroll 8
        for (int r = 0; r < kDwRows; r++) {
            const float4 z4 = Zs[r][ty], va = As[r][tx], vb = Bs[r][tx];
            const float z[4] = {z4.x, z4.y, z4.z, z4.w};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                fma4(a[i], z[i], va);
                fma4(b[i], z[i], vb);
                bias[i] += z[i];
            }
        }
    }
    float *P = partial + (size_t)blockIdx.x * (kH * 2 * kH + kH);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        float4 *row = reinterpret_cast<float4 *>(P + (size_t)(4 * ty + i) * 2 * kH);
        row[tx] = a[i];
        row[kH / 4 + tx] = b[i];
        if (tx == 0) P[kH * 2 * kH + 4 * ty + i] = bias[i];
    }
}

// The same of the input layer (kF columns): lane o of four row groups, the
// groups' sums added in order.
__global__ void __launch_bounds__(kT) k_dw_input(int N, const float *__restrict__ dY, const float *__restrict__ Y,
                                                 const float *__restrict__ X, float *__restrict__ partial) {
    constexpr int kG = kT / kH;
    __shared__ float sums[kG][kF + 1][kH];
    const int o = threadIdx.x & (kH - 1), grp = threadIdx.x / kH;
    int rb, re;
    dw_rows(N, rb, re);
    float acc[kF + 1];
#pragma unroll
    for (int k = 0; k <= kF; k++) acc[k] = 0.f;
#pragma unroll 4
    for (int r = rb + grp; r < re; r += kG) {
        const size_t at = (size_t)r * kH + o;
        const float z = Y[at] > 0.f ? dY[at] : 0.f;
        const float *x = X + (size_t)r * kF;
#pragma unroll
        for (int k = 0; k < kF; k++) acc[k] = fmaf(z, __ldg(x + k), acc[k]);
        acc[kF] += z;
    }
#pragma unroll
    for (int k = 0; k <= kF; k++) sums[grp][k][o] = acc[k];
    __syncthreads();
    float *P = partial + (size_t)blockIdx.x * (kH * kF + kH);
    for (int i = threadIdx.x; i < kH * (kF + 1); i += kT) {
        const int oo = i & (kH - 1), k = i / kH;
        float v = sums[0][k][oo];
        for (int j = 1; j < kG; j++) v += sums[j][k][oo];
        P[k < kF ? oo * kF + k : kH * kF + oo] = v;
    }
}

// The same of the output layer: P[j][k] = sum_r dout[r][j] h[r][k], lane k of
// four row groups.
__global__ void __launch_bounds__(kT) k_dw_output(int N, const float4 *__restrict__ dout, const float *__restrict__ h,
                                                  float *__restrict__ partial) {
    constexpr int kG = kT / kH;
    __shared__ float sums[kG][kOut][kH], bsum[kG][kOut];
    const int k = threadIdx.x & (kH - 1), grp = threadIdx.x / kH;
    int rb, re;
    dw_rows(N, rb, re);
    float acc[kOut] = {0.f, 0.f, 0.f, 0.f}, b[kOut] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
    for (int r = rb + grp; r < re; r += kG) {
        const float4 d = dout[r];
        const float x = h[(size_t)r * kH + k], dd[kOut] = {d.x, d.y, d.z, d.w};
#pragma unroll
        for (int j = 0; j < kOut; j++) {
            acc[j] = fmaf(dd[j], x, acc[j]);
            b[j] += dd[j];
        }
    }
#pragma unroll
    for (int j = 0; j < kOut; j++) {
        sums[grp][j][k] = acc[j];
        if (k == 0) bsum[grp][j] = b[j];
    }
    __syncthreads();
    float *P = partial + (size_t)blockIdx.x * (kOut * kH + kOut);
    for (int i = threadIdx.x; i < kOut * kH; i += kT) {
        const int j = i / kH, kk = i & (kH - 1);
        float v = sums[0][j][kk];
        for (int q = 1; q < kG; q++) v += sums[q][j][kk];
        P[i] = v;
    }
    if (threadIdx.x < kOut) {
        float v = bsum[0][threadIdx.x];
        for (int q = 1; q < kG; q++) v += bsum[q][threadIdx.x];
        P[kOut * kH + threadIdx.x] = v;
    }
}

// grad[w_off + i] = sum over blocks of partial[blk][i] (weights), then biases.
// 32 outputs per block; thread row j adds the blocks j, j + 8, ... in order, the
// eight sums are added in order.
__global__ void __launch_bounds__(kT) k_reduce_partials(int blocks, int OK, int O, const float *__restrict__ partial,
                                                        float *__restrict__ grad, int w_off, int b_off) {
    __shared__ float part[kT / 32][32];
    const int lane = threadIdx.x & 31, j = threadIdx.x >> 5, i = blockIdx.x * 32 + lane;
    float s = 0.f;
    if (i < OK + O) {
#pragma unroll 8
        for (int b = j; b < blocks; b += kT / 32) s += partial[(size_t)b * (OK + O) + i];
    }
    part[j][lane] = s;
    __syncthreads();
    if (j != 0 || i >= OK + O) return;
    for (int k = 1; k < kT / 32; k++) s += part[k][lane];
    if (i < OK)
        grad[w_off + i] = s;
    else
        grad[b_off + (i - OK)] = s;
}

// ------------------------------------------------------------ output ------
// raw = W4 h + b4; pred = d + 0.25 tanh(raw) for both heads.
__global__ void k_output(int N, const float *__restrict__ h, const __nv_bfloat16 *__restrict__ W4,
                         const float *__restrict__ b4, const float2 *__restrict__ base, float4 *__restrict__ raw,
                         float4 *__restrict__ pred) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= N) return;
    float r[kOut];
#pragma unroll
    for (int j = 0; j < kOut; j++) r[j] = b4[j];
    const float4 *hc = reinterpret_cast<const float4 *>(h + (size_t)c * kH);
    float4 x4[kH / 4];
#pragma unroll
    for (int k4 = 0; k4 < kH / 4; k4++) x4[k4] = __ldg(hc + k4);  // the whole row in flight
#pragma unroll
    for (int k4 = 0; k4 < kH / 4; k4++) {
        const float x[4] = {x4[k4].x, x4[k4].y, x4[k4].z, x4[k4].w};
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < kOut; j++) r[j] = fmaf(x[i], bf(W4[j * kH + 4 * k4 + i]), r[j]);
    }
    raw[c] = make_float4(r[0], r[1], r[2], r[3]);
    const float2 b = base[c];
    pred[c] = make_float4(b.x + kCorr * tanhf(r[0]), b.y + kCorr * tanhf(r[1]), b.x + kCorr * tanhf(r[2]),
                          b.y + kCorr * tanhf(r[3]));
}

// Loss: the squared errors of both heads over the movable nodes, divided by
// 2 nn (per-block partials), and d loss / d raw.
__global__ void k_loss(int N, int nn, const float4 *__restrict__ raw, const float4 *__restrict__ pred,
                       const float4 *__restrict__ target, float4 *__restrict__ dout, double *__restrict__ part) {
    __shared__ double sh[kT / 32];
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    double l = 0.0;
    if (c < N) {
        float4 d = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c < nn) {
            const float4 p = pred[c], t = target[c], r = raw[c];
            const float e[4] = {p.x - t.x, p.y - t.y, p.z - t.z, p.w - t.w};
            const float rr[4] = {r.x, r.y, r.z, r.w};
            float dd[4];
            const float s = 1.f / (float)nn;  // d/dp of e^2 / (2 nn)
#pragma unroll
            for (int j = 0; j < 4; j++) {
                l += (double)e[j] * e[j];
                const float th = tanhf(rr[j]);
                dd[j] = s * e[j] * kCorr * (1.f - th * th);
            }
            d = make_float4(dd[0], dd[1], dd[2], dd[3]);
        }
        dout[c] = d;
    }
    l = warp_sum(l);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = l;
    __syncthreads();
    if (threadIdx.x == 0) {
        double s = 0.0;
        for (int w = 0; w < kT / 32; w++) s += sh[w];
        part[blockIdx.x] = s;
    }
}

// One block: thread t adds the partials t, t + kT, ... in order, then a fixed tree.
__global__ void __launch_bounds__(kT) k_sum_loss(int n, const double *__restrict__ part, int nn,
                                                 double *__restrict__ out) {
    __shared__ double sh[32];
    double s[1] = {0.0};
    for (int i = threadIdx.x; i < n; i += kT) s[0] += part[i];
    block_sum<1>(s, sh);
    if (threadIdx.x == 0) out[0] = s[0] / (2.0 * nn);
}

// dh[c][k] = sum_j dout[c][j] W4[j][k]
__global__ void k_output_dh(int N, const float4 *__restrict__ dout, const __nv_bfloat16 *__restrict__ W4,
                            float *__restrict__ dh) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (size_t)N * kH) return;
    const int c = (int)(i / kH), k = (int)(i % kH);
    const float4 d = dout[c];
    dh[i] = d.x * bf(W4[k]) + d.y * bf(W4[kH + k]) + d.z * bf(W4[2 * kH + k]) + d.w * bf(W4[3 * kH + k]);
}

// -------------------------------------------------------------- adam ------
__global__ void k_adam(int n, float *__restrict__ w, const float *__restrict__ g, float *__restrict__ m,
                       float *__restrict__ v, float lr, float c1, float c2, __nv_bfloat16 *__restrict__ wb) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float gi = g[i];
    const float mi = 0.9f * m[i] + 0.1f * gi, vi = 0.999f * v[i] + 0.001f * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float wi = w[i] - lr * (mi * c1) / (sqrtf(vi * c2) + 1e-8f);
    w[i] = wi;
    wb[i] = __float2bfloat16_rn(wi);
}

__global__ void k_to_bf16(int n, const float *__restrict__ w, __nv_bfloat16 *__restrict__ wb) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) wb[i] = __float2bfloat16_rn(w[i]);
}

// proposal: the movable nodes at q + alpha (f - q), in core units
__global__ void k_propose(int nn, const float4 *__restrict__ pred, float alpha, float llx, float lly, float w,
                          float h, float2 *__restrict__ xy) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if (c >= nn) return;
    const float4 p = pred[c];
    const float x = fminf(fmaxf(p.x + alpha * (p.z - p.x), 0.f), 1.f);
    const float y = fminf(fmaxf(p.y + alpha * (p.w - p.y), 0.f), 1.f);
    xy[c] = make_float2(llx + x * w, lly + y * h);
}

}  // namespace
}  // namespace ep

using namespace ep;

// Workspace of the network, grown to the largest netlist bound so far, and
// the netlist it currently holds features of.
struct ep_gnn {
    int device = 0;
    std::string err;
    float *w = nullptr, *grad = nullptr, *adam_m = nullptr, *adam_v = nullptr;
    __nv_bfloat16 *wb = nullptr;
    float *wt = nullptr;  // the input layer's weights as FP32 [k][o] (k_transpose_w)
    // mapped, raised by a bounded wait that gave up: [0] the tensor-core layers',
    // whose outputs every pass computes anew, [1] the diffusion's, whose are kept
    int *gave_up_h = nullptr, *gave_up_d = nullptr;
    unsigned wait_limit = tc::kWaitLimit;  // polls of those waits (ep_gnn_set_wait_limit)
    int sms = 148;
    int cooperative = 0;         // the device takes cooperative launches
    unsigned *barrier = nullptr;  // the diffusion's arrival count
    double *loss = nullptr;
    int64_t step = 0;
    cudaEvent_t used = nullptr;  // the end of the last call's work, where it returned with work
    bool pending = false;        // pending (Use)
    // bound netlist
    uint64_t uid = 0;         // 0: none
    bool pads_ready = false;  // terminal pin lists uploaded (training)
    Net net{};
    EngineGraph eg{};
    // capacities and buffers
    size_t capN = 0, capNet = 0, capT = 0, capP = 0;
    float *X = nullptr, *inv_pins = nullptr, *inv_deg = nullptr;
    float2 *v = nullptr, *netv = nullptr;
    int *padcnt = nullptr, *pad_cursor = nullptr;
    int32_t *pad_start = nullptr, *pad_net = nullptr, *pad_pins = nullptr;
    int4 *kinfo = nullptr;
    int32_t *pin_node = nullptr, *q_net = nullptr;
    float *h[kLayers + 1] = {}, *m[kLayers + 1] = {};
    float *a = nullptr, *dh = nullptr, *dx = nullptr, *dm = nullptr, *da = nullptr, *partial = nullptr;
    float4 *raw = nullptr, *pred = nullptr, *dout = nullptr, *target = nullptr;
    float2 *xy = nullptr;
    double *loss_part = nullptr;
    std::vector<void *> ws;  // workspace allocations (freed on growth)
    ep_gnn() { err.reserve(256); }
};

namespace {

#define GK(call)                                                                  \
    do {                                                                          \
        cudaError_t _e = (call);                                                  \
        if (_e != cudaSuccess) {                                                  \
            g->err = std::string(#call) + ": " + cudaGetErrorString(_e);          \
            return EP_ERR_CUDA;                                                   \
        }                                                                         \
    } while (0)

// One call's use of the network's workspace and weights, on its engine's stream.
// Engines have streams of their own and some calls return with work pending, so
// a call waits on the device for one that did, and marks its own end unless it
// has waited for its stream (synced).  Neither while the stream is being
// captured, where they may not be.
class Use {
  public:
    explicit Use(ep_gnn *g) : g_(g) {}
    Use(const Use &) = delete;
    ep_status begin(cudaStream_t st) {
        ep_gnn *const g = g_;
        if (g->pending && !capturing(st)) GK(cudaStreamWaitEvent(st, g->used));
        st_ = st;
        open_ = true;
        return EP_OK;
    }
    void synced() {
        open_ = false;
        g_->pending = false;  // what was pending came before on this stream
    }
    ~Use() {
        if (!open_ || capturing(st_)) return;
        if (cudaEventRecord(g_->used, st_) == cudaSuccess)
            g_->pending = true;
        else
            cudaStreamSynchronize(st_);
    }

  private:
    static bool capturing(cudaStream_t st) {
        cudaStreamCaptureStatus c;
        return cudaStreamIsCapturing(st, &c) == cudaSuccess && c != cudaStreamCaptureStatusNone;
    }
    ep_gnn *g_;
    cudaStream_t st_ = nullptr;
    bool open_ = false;
};

size_t smem_dense(int K) { return sizeof(float) * ((size_t)K * kH + (size_t)kDenseRows * (K + 1)); }

void set_smem_attrs() {
    static std::vector<int> done;
    int dev = 0;
    cudaGetDevice(&dev);
    if (std::find(done.begin(), done.end(), dev) != done.end()) return;
    done.push_back(dev);
    cudaFuncSetAttribute(k_dense<kF, 0>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_dense(kF));
    cudaFuncSetAttribute(k_dense_tc, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTcSmem);
    cudaFuncSetAttribute(k_diffuse, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDiffSmem);
    cudaFuncSetAttribute(k_dense_dx, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDxSmem);
}

template <typename T>
bool walloc(ep_gnn *g, T *&p, size_t n) {
    if (cudaMalloc((void **)&p, std::max<size_t>(n, 1) * sizeof(T)) != cudaSuccess) {
        p = nullptr;
        return false;
    }
    g->ws.push_back(p);
    return true;
}

// Grow the workspace to hold N nodes, nnet nets, nt terminals and np pins.
ep_status reserve(ep_gnn *g, size_t N, size_t nnet, size_t nt, size_t np) {
    if (N <= g->capN && nnet <= g->capNet && nt <= g->capT && np <= g->capP) return EP_OK;
    cudaDeviceSynchronize();
    for (void *p : g->ws) cudaFree(p);
    g->ws.clear();
    g->uid = 0;
    g->pads_ready = false;
    // a quarter of headroom on every dimension, so designs of about the same
    // size do not each grow the workspace again (a growth frees and
    // reallocates all of it)
    auto grow = [](size_t want, size_t cap) { return std::max(want + want / 4, cap); };
    N = grow(N, g->capN);
    nnet = grow(nnet, g->capNet);
    nt = grow(nt, g->capT);
    np = grow(np, g->capP);
    bool ok = walloc(g, g->X, N * kF) && walloc(g, g->inv_pins, N) && walloc(g, g->inv_deg, nnet) &&
              walloc(g, g->v, N) && walloc(g, g->netv, nnet) && walloc(g, g->padcnt, nt) &&
              walloc(g, g->pad_start, nt + 1) && walloc(g, g->pad_cursor, nt) && walloc(g, g->pad_net, np) &&
              walloc(g, g->pad_pins, np) && walloc(g, g->a, nnet * kH) && walloc(g, g->dh, N * kH) &&
              walloc(g, g->dx, N * kH) && walloc(g, g->dm, N * kH) && walloc(g, g->da, nnet * kH) &&
              walloc(g, g->partial, (size_t)kDwBlocks * (kH * 2 * kH + kH)) &&
              walloc(g, g->raw, N) && walloc(g, g->pred, N) && walloc(g, g->dout, N) && walloc(g, g->target, N) &&
              walloc(g, g->xy, N) && walloc(g, g->loss_part, nblk((long long)N)) && walloc(g, g->kinfo, nnet) &&
              walloc(g, g->pin_node, np) && walloc(g, g->q_net, np);
    for (int l = 0; l <= kLayers && ok; l++) ok = walloc(g, g->h[l], N * kH) && walloc(g, g->m[l], N * kH);
    if (!ok) {
        g->capN = g->capNet = g->capT = g->capP = 0;
        g->err = "cudaMalloc failed for the network's workspace";
        return EP_ERR_NOMEM;
    }
    g->capN = N;
    g->capNet = nnet;
    g->capT = nt;
    g->capP = np;
    return EP_OK;
}

// The diffusion as one cooperative launch; false when the design's share of a CTA
// does not fit or the device cannot, and the passes have to go one by one.
bool diffuse_at_once(ep_gnn *g, ep_status &status) {
    const EngineGraph &eg = g->eg;
    // enough pins for every CTA to be worth its place at the barrier
    const int G = std::max(1, std::min(g->sms, (eg.np + 255) / 256));
    const DiffShare share{eg.np / G + 1 + eg.max_net_pins, eg.np / G + 1 + eg.max_node_pins};
    if (!g->cooperative || diff_smem(share) > kDiffSmem) return false;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(G);
    cfg.blockDim = dim3(kDiffThreads);
    cfg.dynamicSmemBytes = diff_smem(share);
    cfg.stream = eg.st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t rc = cudaMemsetAsync(g->barrier, 0, sizeof(unsigned), eg.st);
    if (rc == cudaSuccess)
        rc = cudaLaunchKernelEx(&cfg, k_diffuse, g->net, eg.np, share, (const float *)g->inv_pins, g->v, g->netv, g->X,
                                g->barrier, g->wait_limit, g->gave_up_d + 1, eg.d_status);
    if (rc == cudaErrorCooperativeLaunchTooLarge) {  // fewer SMs than the device's are ours
        cudaGetLastError();
        return false;
    }
    if (rc != cudaSuccess) {
        g->err = std::string("diffusion launch: ") + cudaGetErrorString(rc);
        status = EP_ERR_CUDA;
    }
    return true;
}

// Bind an engine's netlist: its device arrays, the features (computed on the
// engine's stream) -- skipped when the workspace already holds them.
ep_status bind(ep_gnn *g, ep_engine *e, Use &use) {
    EngineGraph eg{};
    if (engine_graph(e, &eg)) return EP_ERR_ARG;
    if (eg.nn <= 0 || eg.nnet <= 0) {
        g->err = "the network needs movable nodes and nets";
        return EP_ERR_ARG;
    }
    if (eg.device != g->device) {
        g->err = "the engine lives on another device than the network";
        return EP_ERR_ARG;
    }
    ep_status s = use.begin(eg.st);
    if (s) return s;
    if (g->uid == eg.uid) {
        g->eg = eg;
        return EP_OK;
    }
    set_smem_attrs();
    const int N = eg.nn + eg.nt;
    s = reserve(g, N, eg.nnet, eg.nt, eg.np);
    if (s) return s;
    g->eg = eg;
    g->uid = 0;  // until the features are on their way
    g->pads_ready = false;
    Net &n = g->net;
    n.nn = eg.nn;
    n.n_obj = eg.n_obj;
    n.N = N;
    n.nnet = eg.nnet;
    n.owner = eg.d_pin_owner;
    n.net_first = eg.d_net_first;
    n.net_deg = eg.d_net_deg;
    n.pin_net = eg.d_pin_net;
    n.obj_pin_start = eg.d_obj_pin_start;
    n.obj_pin_dev = eg.d_obj_pin_dev;
    n.net_order = eg.d_net_dev_order;
    n.n_big = eg.n_big_nets;
    n.pad_start = g->pad_start;
    n.pad_net = g->pad_net;
    n.kinfo = g->kinfo;
    n.pin_node = g->pin_node;
    n.q_net = g->q_net;
    cudaStream_t st = eg.st;
    if (eg.fp64)
        k_init<double><<<nblk(N), kT, 0, st>>>(n, eg.d_area, eg.d_npins, (const double2 *)eg.d_pos, eg.grid, g->X,
                                                g->v, g->inv_pins);
    else
        k_init<float><<<nblk(N), kT, 0, st>>>(n, eg.d_area, eg.d_npins, (const float2 *)eg.d_pos, eg.grid, g->X,
                                               g->v, g->inv_pins);
    if (eg.nt > 0) {
        GK(cudaMemsetAsync(g->padcnt, 0, sizeof(int) * eg.nt, st));
        k_pad_pins<<<nblk(eg.np), kT, 0, st>>>(eg.np, n, g->padcnt);
        k_pad_feature<<<nblk(eg.nt), kT, 0, st>>>(eg.nt, eg.nn, g->padcnt, g->X);
    }
    k_inv_deg<<<nblk(eg.nnet), kT, 0, st>>>(eg.nnet, eg.d_net_deg, g->inv_deg);
    k_graph_index<<<nblk(std::max(eg.nnet, eg.np)), kT, 0, st>>>(n, eg.np, g->kinfo, g->pin_node, g->q_net);
    ep_status ds = EP_OK;
    if (!diffuse_at_once(g, ds)) {
        int col = 3;
        for (int k = 1; k <= kDiff3; k++) {
            // programmatic serialisation: the next pass's blocks wait resident
            launch_k(k_diff_net, nblk(31LL * n.n_big + eg.nnet), kT, 0, st, n, (const float2 *)g->v, g->netv);
            launch_k(k_diff_node, nblk(eg.nn), kT, 0, st, n, (const float *)g->inv_pins, (const float2 *)g->netv, g->v);
            if (k == kDiff1 || k == kDiff2 || k == kDiff3) {
                launch_k(k_store_feature, nblk(N), kT, 0, st, N, (const float2 *)g->v, g->X, col);
                col += 2;
            }
        }
    }
    if (ds) return ds;
    GK(cudaGetLastError());
    g->uid = eg.uid;
    return EP_OK;
}

// The terminals' pin lists of the bound netlist.
ep_status bind_pads(ep_gnn *g) {
    if (g->pads_ready) return EP_OK;
    const EngineGraph &eg = g->eg;
    cudaStream_t st = eg.st;
    if (eg.nt > 0) {
        k_pad_start<<<1, kT, 0, st>>>(eg.nt, g->padcnt, g->pad_start, g->pad_cursor);
        k_pad_fill<<<nblk(eg.np), kT, 0, st>>>(eg.np, g->net, g->pad_cursor, g->pad_pins);
        k_pad_sort<<<eg.nt, kT, 0, st>>>(g->net, eg.np, g->pad_start, g->pad_pins, g->pad_net);
        GK(cudaGetLastError());
    }
    g->pads_ready = true;
    return EP_OK;
}

// A wait that gave up since the last check, reported once: the diffusion's, and
// with all also the tensor-core layers'.  The features that a diffusion left
// incomplete are not kept.  Every CTA that gives up raises the flag, so it is
// cleared when the pass is over.  Called before a call enqueues anything (an
// earlier pass that was not waited for) and after it has waited for its own.
ep_status gave_up(ep_gnn *g, bool all) {
    volatile int *f = g->gave_up_h;
    if (!f[1] && !(all && f[0])) return EP_OK;
    GK(cudaEventSynchronize(g->used));
    if (f[1]) g->uid = 0;
    f[1] = 0;
    if (all) f[0] = 0;
    g->err = "a bounded wait of the network's kernels gave up";
    return EP_ERR_TIMEOUT;
}

// Forward pass on the bound netlist (activations kept for the backward pass).
ep_status forward(ep_gnn *g) {
    const Net &n = g->net;
    const int N = n.N;
    cudaStream_t st = g->eg.st;
    const float *w = g->w;
    const __nv_bfloat16 *wb = g->wb;
    const int tc_grid = std::max(1, std::min((N + kTcRows - 1) / kTcRows, 2 * g->sms));
    k_dense<kF, 0><<<nblk(N, kDenseRows), kT, smem_dense(kF), st>>>(N, g->X, nullptr, g->wt, w + kOffB0,
                                                                    g->h[0]);
    for (int l = 1; l <= kLayers; l++) {
        k_net_mean<<<n.n_big + nblk(n.nnet - n.n_big, kT / kHalf), kT, 0, st>>>(n, (const float2 *)g->h[l - 1],
                                                                                (float2 *)g->a);
        k_node_mean<<<nblk((long long)N * kHalf), kT, 0, st>>>(n, g->inv_pins, (const float4 *)g->a, (float4 *)g->m[l]);
        launch_dense_tc(tc_grid, st, N, g->h[l - 1], g->m[l], wb + off_w(l), w + off_b(l), g->h[l], g->gave_up_d,
                        g->eg.d_status, g->wait_limit);
    }
    k_output<<<nblk(N), kT, 0, st>>>(N, g->h[kLayers], wb + kOffW4, w + kOffB4, g->v, g->raw, g->pred);
    GK(cudaGetLastError());
    return EP_OK;
}

// Loss against g->target and the gradient of every parameter into g->grad.
ep_status backward(ep_gnn *g) {
    const Net &n = g->net;
    const int N = n.N;
    cudaStream_t st = g->eg.st;
    const __nv_bfloat16 *wb = g->wb;
    const int lb = nblk(N);
    k_loss<<<lb, kT, 0, st>>>(N, n.nn, g->raw, g->pred, g->target, g->dout, g->loss_part);
    k_sum_loss<<<1, kT, 0, st>>>(lb, g->loss_part, n.nn, g->loss);
    const int pb = std::min(nblk(N, kDwRows), kDwBlocks);
    auto reduce = [&](int OK, int O, int w_off, int b_off) {
        k_reduce_partials<<<nblk(OK + O, 32), kT, 0, st>>>(pb, OK, O, g->partial, g->grad, w_off, b_off);
    };
    // output layer
    k_dw_output<<<pb, kT, 0, st>>>(N, g->dout, g->h[kLayers], g->partial);
    reduce(kOut * kH, kOut, kOffW4, kOffB4);
    k_output_dh<<<nblk((long long)N * kH), kT, 0, st>>>(N, g->dout, wb + kOffW4, g->dh);
    // message-passing layers, last to first; dh holds d loss / d h_l
    float *dh = g->dh, *dx = g->dx;
    for (int l = kLayers; l >= 1; l--) {
        k_dw_hidden<<<pb, kT, 0, st>>>(N, dh, g->h[l], g->h[l - 1], g->m[l], g->partial);
        reduce(kH * 2 * kH, kH, off_w(l), off_b(l));
        // d h_{l-1} (direct part) into dx, d m_l into g->dm
        k_dense_dx<<<std::min(nblk(N, kDxRows), 148 * 2), kT, kDxSmem, st>>>(N, dh, g->h[l], wb + off_w(l), dx, g->dm);
        k_node_mean_t<<<n.n_big + nblk(n.nnet - n.n_big, kT / kHalf), kT, 0, st>>>(
            n, g->inv_pins, (const float2 *)g->dm, (float2 *)g->da);
        k_net_mean_t_add<<<nblk((long long)N * kHalf), kT, 0, st>>>(n, g->inv_deg, (const float4 *)g->da, (float4 *)dx);
        std::swap(dh, dx);
    }
    // input layer
    k_dw_input<<<pb, kT, 0, st>>>(N, dh, g->h[0], g->X, g->partial);
    reduce(kH * kF, kH, kOffW0, kOffB0);
    GK(cudaGetLastError());
    return EP_OK;
}

// Targets of the movable nodes: [nn][4] core coordinates (quadratic
// placement x, y, final x, y), normalised to the core.
ep_status upload_target(ep_gnn *g, const float *t4) {
    const Grid &gr = g->eg.grid;
    GK(cudaMemcpyAsync(g->target, t4, sizeof(float4) * g->net.nn, cudaMemcpyHostToDevice, g->eg.st));
    k_target<<<nblk(g->net.N), kT, 0, g->eg.st>>>(g->net.N, g->net.nn, gr.llx, gr.lly, gr.urx - gr.llx, gr.ury - gr.lly,
                                                 g->target);
    GK(cudaGetLastError());
    return EP_OK;
}

ep_status oom(ep_gnn *g) {
    g->err.assign("out of host memory");
    return EP_ERR_NOMEM;
}

}  // namespace

extern "C" {

int32_t ep_gnn_num_weights(void) { return kParams; }

const char *ep_gnn_last_error(const ep_gnn *g) { return g ? g->err.c_str() : "null network"; }

ep_status ep_gnn_create(int32_t device, uint64_t seed, ep_gnn **out) try {
    if (!out) return EP_ERR_ARG;
    *out = nullptr;
    ep_gnn *g = new ep_gnn();
    *out = g;
    g->device = device;
    GK(cudaSetDevice(device));
    if (cudaMalloc(&g->w, sizeof(float) * kParams) != cudaSuccess ||
        cudaMalloc(&g->grad, sizeof(float) * kParams) != cudaSuccess ||
        cudaMalloc(&g->adam_m, sizeof(float) * kParams) != cudaSuccess ||
        cudaMalloc(&g->adam_v, sizeof(float) * kParams) != cudaSuccess ||
        cudaMalloc(&g->wb, sizeof(__nv_bfloat16) * kParams) != cudaSuccess ||
        cudaMalloc(&g->wt, sizeof(float) * kWtSize) != cudaSuccess ||
        cudaMalloc(&g->loss, sizeof(double)) != cudaSuccess ||
        cudaMalloc(&g->barrier, sizeof(unsigned)) != cudaSuccess ||
        cudaEventCreateWithFlags(&g->used, cudaEventDisableTiming) != cudaSuccess ||
        cudaHostAlloc(&g->gave_up_h, 2 * sizeof(int), cudaHostAllocMapped) != cudaSuccess ||
        cudaHostGetDevicePointer(&g->gave_up_d, g->gave_up_h, 0) != cudaSuccess) {
        g->err = "cudaMalloc failed for the network's weights";
        return EP_ERR_NOMEM;
    }
    g->gave_up_h[0] = g->gave_up_h[1] = 0;
    cudaDeviceGetAttribute(&g->sms, cudaDevAttrMultiProcessorCount, device);
    cudaDeviceGetAttribute(&g->cooperative, cudaDevAttrCooperativeLaunch, device);
    // Glorot-uniform weights, zero biases; the output layer starts small so
    // the first predictions stay near the diffusion coordinates
    std::vector<float> w(kParams, 0.f);
    std::mt19937_64 rng(seed);
    auto fill = [&](int off, int rows, int cols, float gain) {
        std::uniform_real_distribution<float> u(-1.f, 1.f);
        const float a = gain * std::sqrt(6.f / (float)(rows + cols));
        for (int i = 0; i < rows * cols; i++) w[off + i] = a * u(rng);
    };
    fill(kOffW0, kH, kF, 1.f);
    for (int l = 1; l <= kLayers; l++) fill(off_w(l), kH, 2 * kH, 1.f);
    fill(kOffW4, kOut, kH, 0.1f);
    return ep_gnn_set_weights(g, w.data());
} catch (const std::bad_alloc &) {
    return EP_ERR_NOMEM;
}

void ep_gnn_destroy(ep_gnn *g) {
    if (!g) return;
    cudaDeviceSynchronize();
    for (void *p : g->ws) cudaFree(p);
    for (void *p : {(void *)g->w, (void *)g->grad, (void *)g->adam_m, (void *)g->adam_v, (void *)g->wb,
                    (void *)g->wt, (void *)g->loss, (void *)g->barrier})
        if (p) cudaFree(p);
    if (g->gave_up_h) cudaFreeHost(g->gave_up_h);
    if (g->used) cudaEventDestroy(g->used);
    delete g;
}

ep_status ep_gnn_get_weights(ep_gnn *g, float *w) {
    if (!g || !w) return EP_ERR_ARG;
    GK(cudaMemcpy(w, g->w, sizeof(float) * kParams, cudaMemcpyDeviceToHost));
    return EP_OK;
}

ep_status ep_gnn_set_weights(ep_gnn *g, const float *w) {
    if (!g || !w) return EP_ERR_ARG;
    if (g->pending) GK(cudaEventSynchronize(g->used));  // a pass that still reads the weights
    GK(cudaMemcpy(g->w, w, sizeof(float) * kParams, cudaMemcpyHostToDevice));
    GK(cudaMemset(g->adam_m, 0, sizeof(float) * kParams));
    GK(cudaMemset(g->adam_v, 0, sizeof(float) * kParams));
    k_to_bf16<<<nblk(kParams), kT>>>(kParams, g->w, g->wb);
    k_transpose_w<<<nblk(kWtSize), kT>>>(g->wb, g->wt);
    GK(cudaGetLastError());
    GK(cudaDeviceSynchronize());
    g->step = 0;
    return EP_OK;
}

ep_status ep_gnn_release(ep_gnn *g, ep_engine *e) {
    if (!g || !e) return EP_ERR_ARG;
    EngineGraph eg{};
    if (engine_graph(e, &eg)) return EP_ERR_ARG;
    if (g->uid == eg.uid) g->uid = 0;
    return EP_OK;
}

ep_status ep_gnn_features(ep_gnn *g, ep_engine *e, float *X) {
    if (!g || !e || !X) return EP_ERR_ARG;
    Use use(g);
    ep_status s = gave_up(g, false);
    if (s || (s = bind(g, e, use))) return s;
    GK(cudaMemcpyAsync(X, g->X, sizeof(float) * (size_t)g->net.N * kF, cudaMemcpyDeviceToHost, g->eg.st));
    GK(cudaStreamSynchronize(g->eg.st));
    use.synced();
    return gave_up(g, false);
}

ep_status ep_gnn_forward(ep_gnn *g, ep_engine *e, float *xy4) try {
    if (!g || !e || !xy4) return EP_ERR_ARG;
    Use use(g);
    ep_status s = gave_up(g, true);
    if (s || (s = bind(g, e, use)) || (s = forward(g))) return s;
    const int nn = g->net.nn;
    std::vector<float4> p(nn);
    GK(cudaMemcpyAsync(p.data(), g->pred, sizeof(float4) * nn, cudaMemcpyDeviceToHost, g->eg.st));
    GK(cudaStreamSynchronize(g->eg.st));
    use.synced();
    if ((s = gave_up(g, true))) return s;
    const Grid &gr = g->eg.grid;
    const float W = gr.urx - gr.llx, H = gr.ury - gr.lly;
    for (int c = 0; c < nn; c++) {
        xy4[4 * c] = gr.llx + p[c].x * W;
        xy4[4 * c + 1] = gr.lly + p[c].y * H;
        xy4[4 * c + 2] = gr.llx + p[c].z * W;
        xy4[4 * c + 3] = gr.lly + p[c].w * H;
    }
    return EP_OK;
} catch (const std::bad_alloc &) {
    return oom(g);
}

ep_status ep_gnn_loss_grad(ep_gnn *g, ep_engine *e, const float *target4, double *loss, float *grad) try {
    if (!g || !e || !target4) return EP_ERR_ARG;
    Use use(g);
    ep_status s = gave_up(g, true);
    if (s || (s = bind(g, e, use)) || (s = bind_pads(g)) || (s = upload_target(g, target4)) || (s = forward(g)) ||
        (s = backward(g)))
        return s;
    if (loss) GK(cudaMemcpyAsync(loss, g->loss, sizeof(double), cudaMemcpyDeviceToHost, g->eg.st));
    if (grad) GK(cudaMemcpyAsync(grad, g->grad, sizeof(float) * kParams, cudaMemcpyDeviceToHost, g->eg.st));
    GK(cudaStreamSynchronize(g->eg.st));
    use.synced();
    return gave_up(g, true);
} catch (const std::bad_alloc &) {
    return oom(g);
}

ep_status ep_gnn_train_step(ep_gnn *g, ep_engine *e, const float *target4, float lr, double *loss) try {
    if (!g || !e || !target4 || !(lr > 0)) return EP_ERR_ARG;
    Use use(g);
    ep_status s = gave_up(g, true);
    if (s || (s = bind(g, e, use)) || (s = bind_pads(g)) || (s = upload_target(g, target4)) || (s = forward(g)) ||
        (s = backward(g)))
        return s;
    g->step++;
    const float c1 = 1.f / (1.f - std::pow(0.9f, (float)g->step)), c2 = 1.f / (1.f - std::pow(0.999f, (float)g->step));
    k_adam<<<nblk(kParams), kT, 0, g->eg.st>>>(kParams, g->w, g->grad, g->adam_m, g->adam_v, lr, c1, c2, g->wb);
    k_transpose_w<<<nblk(kWtSize), kT, 0, g->eg.st>>>(g->wb, g->wt);
    GK(cudaGetLastError());
    if (loss) GK(cudaMemcpyAsync(loss, g->loss, sizeof(double), cudaMemcpyDeviceToHost, g->eg.st));
    GK(cudaStreamSynchronize(g->eg.st));
    use.synced();
    return gave_up(g, true);
} catch (const std::bad_alloc &) {
    return oom(g);
}

ep_status ep_gnn_set_wait_limit(ep_gnn *g, int32_t polls) {
    if (!g) return EP_ERR_ARG;
    g->wait_limit = polls < 0 ? tc::kWaitLimit : (unsigned)polls;
    return EP_OK;
}

ep_status ep_gnn_propose(ep_gnn *g, ep_engine *e, float alpha) {
    if (!g || !e || !(alpha >= 0.f) || alpha > 1.f) return EP_ERR_ARG;
    Use use(g);
    ep_status s = gave_up(g, true);
    if (s || (s = bind(g, e, use)) || (s = forward(g))) return s;
    const Grid &gr = g->eg.grid;
    k_propose<<<nblk(g->net.nn), kT, 0, g->eg.st>>>(g->net.nn, g->pred, alpha, gr.llx, gr.lly, gr.urx - gr.llx,
                                                    gr.ury - gr.lly, g->xy);
    GK(cudaGetLastError());
    if (engine_set_node_centres(e, g->xy)) {
        g->err = "setting the proposed positions failed";
        return EP_ERR_CUDA;
    }
    return EP_OK;
}

}  // extern "C"
