// fft_kernels.cuh -- the electrostatic Poisson solve of FFT_2D::doFFT
// (FFT/fft.cpp:191-284) by fast transforms: the same sums as dct.cu,
//   a   = C_nx rho C_ny^T,   P = a .* K,
//   E_x = S_nx^T diag(wx) P C_ny,   E_y = C_nx^T P diag(wy) S_ny,   phi = C_nx^T P C_ny,
// evaluated as 1-D transforms along one axis at a time, each a length-n
// complex FFT in shared memory (n a power of two), O(n^2 log n) per map
// instead of the GEMMs' O(n^3).
//
// The 1-D transforms (C_n[k][j] = cos(pi k (j+1/2) / n)):
//   DCT-II  X = C_n x     by Makhoul's permutation v = (x0, x2, .., x3, x1),
//                         V = FFT(v), X[k] = Re(V[k] e^{-i pi k / 2n});
//   DCT-III y = C_n^T X   by the inverse of that: Z[k] = (X~[k] - i X[n-k])
//                         e^{i pi k / 2n} / 2 (X~[0] = 2 X[0], X[n] = 0),
//                         z = IFFT(Z) (unnormalised), y[2j] = z[j],
//                         y[2j+1] = z[n-1-j] (z is real: Z is Hermitian);
//   sine    y = S_n^T X   = (-1)^j C_n^T b with b[0] = 0, b[k] = X[n-k]
//                         (sin(pi (n-k)(j+1/2)/n) = (-1)^j cos(pi k (j+1/2)/n)).
// Two real sequences share one complex FFT (one in the real, one in the
// imaginary part) wherever the inputs or outputs are real.
//
// Three kernels, maps x-major [nx][ny] as everywhere in the engine:
//   k_fft_rows_fwd  T[x][v]  = DCT-II of rho[x][:] along y          (2 rows per FFT)
//   k_fft_cols      per column v of T: DCT-II along x, times K, then
//                   X1[:][v] = S^T diag(wx) P[:][v] and X2[:][v] = C^T P[:][v]
//                   (2 or 4 columns per block; X1 of two columns share one
//                   complex IFFT and X2 of two another: P is dominated by its
//                   low frequencies, so an FFT carrying P beside wx P would
//                   round the small E inputs relative to |P|)
//   k_fft_rows_inv  per row x: E_x = C^T X1[x][:], E_y = S^T diag(wy) X2[x][:]
//                   (one complex IFFT), phi = C^T X2[x][:] when asked
// Twiddles, the e^{i pi k / 2n} factors and the frequency weights come from
// tables computed in double on the host, staged in shared memory by every
// block before it waits on the previous grid.  The kernels are instantiated
// per log2 n so that every loop has a fixed trip count and a thread issues
// all its loads before it uses any, and per working precision R (float for
// the engine's mixed-precision form, double for the plain FP64 form; the
// tables are rounded to R).
//
// What bounds them is the shared memory that every butterfly goes through and
// the barriers between the passes, then (from 1024^2) the L2 sectors of the
// columns.  Eight elements per thread and pass with the places spread over the
// banks took the three from 18.5 us to 13.4 (10.7 with four columns) at 512^2,
// from 54.2 to 29.5 at 1024^2 and from 196 to 112 at 2048^2 in FP32, in FP64
// from 23.0 to 17.0, 78 to 56 and 282 to 194; up to 256^2 they are launch and
// latency bound (9 us).
#pragma once
#include <algorithm>
#include <array>
#include <cmath>
#include <utility>
#include <string>
#include <vector>

#include "fft.h"

namespace ep {

namespace {

// Threads and elements of a block of the row passes and threads of the column
// pass: with eight elements per butterfly pass the block size hardly matters
// (128 to 256 threads and 512 to 1024 elements are within 1% in a whole
// Nesterov step at 136^2 to 1024^2 bins).
constexpr int kThreads = 256;
constexpr int kRowElems = 1024;

// Columns per block of the column pass.  Two columns are eight bytes of a
// row in FP32, a quarter of the sector that is fetched; four are half of it,
// but leave half the blocks.  Four where that is still more than a block per
// SM: at 1024^2 29.5 us for the three passes, 36.9 with two; at 512^2 128
// blocks of four leave the other streams' kernels fewer whole SMs, and a
// Nesterov step takes 57.1 us, with two 56.4.
template <typename R>
constexpr int col_count(int ny) {
    return sizeof(R) == 4 && ny / 4 > 148 ? 4 : 2;
}

__device__ __forceinline__ int makhoul(int j, int n) { return (j & 1) ? n - 1 - (j >> 1) : (j >> 1); }

__device__ __forceinline__ int brev(int i, int logn) { return (int)(__brev((unsigned)i) >> (32 - logn)); }

// a b + c d and a b - c d with the second product rounded by itself, and the
// complex product: the contractions are spelled out so that the transforms
// round alike however the butterflies are grouped into passes.  XY: the
// imaginary part rounds a.y b.x by itself, else a.x b.y.
template <typename R>
__device__ __forceinline__ R sum2(R a, R b, R c, R d) {
    return fma_r(a, b, mul_rn(c, d));
}
template <typename R>
__device__ __forceinline__ R dif2(R a, R b, R c, R d) {
    return fma_r(a, b, -mul_rn(c, d));
}
template <typename R>
__device__ __forceinline__ vec2<R> cmul(vec2<R> a, vec2<R> b, bool xy) {
    return mk2<R>(dif2<R>(a.x, b.x, a.y, b.y), xy ? sum2<R>(a.x, b.y, a.y, b.x) : sum2<R>(a.y, b.x, a.x, b.y));
}

// The dynamic shared memory of a kernel, as an array of R's complex type.
template <typename R>
__device__ __forceinline__ vec2<R> *smem_c() {
    extern __shared__ __align__(16) unsigned char fft_smem[];
    return reinterpret_cast<vec2<R> *>(fft_smem);
}

// Where element i of a sequence lies in shared memory.  A row of banks holds
// 16 float2 or 8 double2 elements; the index's low bits (its place in the row)
// are XORed with folds of its high bits, so that the accesses of the kernels
// below (butterflies at every stride, bit-reversed stores, spectra read
// upwards and downwards, Makhoul's order) spread over the banks.  The folds
// are the best of all sums of up to three shifts over n = 32..2048, counted
// on the kernels' own indices: the column pass of n = 1024 in FP32 takes 1.6 K
// rows of banks per block, 7.0 K in plain order with radix-4 butterflies
// (a bit-reversed store alone then puts 16 lanes on one bank).  Linear over
// XOR: place(a ^ b) = place(a) ^ place(b).
template <typename R>
__host__ __device__ constexpr int place(int i) {
    return sizeof(R) == 4 ? i ^ (((i >> 4 << 1) ^ (i >> 4) ^ (i >> 8)) & 15) : i ^ (((i >> 3) ^ (i >> 4) ^ (i >> 7)) & 7);
}

// Stages taken by the first pass over a sequence; the later ones take three.
__host__ __device__ constexpr int first_stages(int logn) {
    return logn % 3 == 0 ? 3 : (logn % 3 == 2 ? 2 : (logn > 1 ? 4 : 1));
}

// Radix-2 stages s .. s + RL - 1 on the 2^RL elements at stride 2^s from
// position pos of their group, in registers.  The stages count in pairs from
// `first`; xy is set in the second of a pair for the lower half's products.
template <bool INV, int LOGN, int RL, typename R>
__device__ __forceinline__ void butterfly(vec2<R> (&a)[1 << RL], int s, int pos, const vec2<R> *tw) {
    constexpr int first = LOGN & 1;
#pragma unroll
    for (int t = 0; t < RL; t++) {
        const int hl = 1 << t;
#pragma unroll
        for (int c = 0; c < hl; c++) {
            vec2<R> w = tw[(hl << s) - 1 + pos + (c << s)];
            if (INV) w.y = -w.y;
            const bool xy = !INV && s + t > 0 && ((s + t - first) & 1) &&
                            !(t > 0 ? (c >> (t - 1)) & 1 : (pos >> (s - 1)) & 1);
#pragma unroll
            for (int g = 0; g < (1 << RL); g += 2 * hl) {
                const vec2<R> lo = a[g + c];
                const vec2<R> x = s + t == 0 ? a[g + c + hl] : cmul<R>(a[g + c + hl], w, xy);  // stage 0: twiddle 1
                a[g + c] = mk2<R>(lo.x + x.x, lo.y + x.y);
                a[g + c + hl] = mk2<R>(lo.x - x.x, lo.y - x.y);
            }
        }
    }
}

// One pass of block_fft: stages S .. S + RL - 1 of nseq <= NSEQ sequences.
template <bool INV, int LOGN, int S, int RL, int NSEQ, int NT, typename R>
__device__ __forceinline__ void fft_pass(vec2<R> *buf, int nseq, const vec2<R> *tw) {
    constexpr int per = LOGN - RL, its = ((NSEQ << per) + NT - 1) / NT, h = 1 << S;
#pragma unroll
    for (int it = 0; it < its; it++) {
        const int j = threadIdx.x + it * NT;
        if (j >= nseq << per) break;
        const int q = j >> per, b = j & ((1 << per) - 1);
        const int pos = b & (h - 1);
        vec2<R> *o = buf + (q << LOGN);
        const int i0 = place<R>(((b >> S) << (S + RL)) + pos);
        vec2<R> a[1 << RL];
#pragma unroll
        for (int k = 0; k < (1 << RL); k++) a[k] = o[i0 ^ place<R>(k << S)];
        butterfly<INV, LOGN, RL, R>(a, S, pos, tw);
#pragma unroll
        for (int k = 0; k < (1 << RL); k++) o[i0 ^ place<R>(k << S)] = a[k];
    }
    __syncthreads();
}

// In-place decimation-in-time FFT of nseq (<= NSEQ) length-2^LOGN sequences
// in shared memory (element i of each at place(i)), input in bit-reversed
// order, output in natural order, by NT threads; FROM: the stages already
// done (0, or those of the first pass).  tw: the stage-major twiddles, in
// shared memory.  INV uses e^{+...} (unnormalised inverse).  The radix-2
// stages run three to a pass (two or four in the first, by log2 n): a thread
// loads the eight elements that they combine, applies them in registers (the
// same operations as radix-2 passes) and stores them, one barrier per pass.
// Ends with a block barrier.
template <bool INV, int LOGN, int FROM, int NSEQ, int NT, typename R>
__device__ __forceinline__ void block_fft(vec2<R> *buf, int nseq, const vec2<R> *tw) {
    if constexpr (FROM < LOGN) {
        constexpr int RL = FROM == 0 ? first_stages(LOGN) : 3;
        fft_pass<INV, LOGN, FROM, RL, NSEQ, NT, R>(buf, nseq, tw);
        block_fft<INV, LOGN, FROM + RL, NSEQ, NT, R>(buf, nseq, tw);
    }
}

// The first pass of a forward FFT of a Makhoul-permuted sequence, from memory:
// thread r < n / 2^RL combines the entries r + c n / 2^RL of the permuted
// sequence, which lie side by side in bit-reversed order.  elem(x): entry x
// of the sequence as it is in memory.
template <int LOGN, int RL, typename T, typename F>
__device__ __forceinline__ void load_group(T (&a)[1 << RL], int r, F elem) {
    constexpr int n = 1 << LOGN;
#pragma unroll
    for (int k = 0; k < (1 << RL); k++) {
        int c = 0;
#pragma unroll
        for (int t = 0; t < RL; t++) c |= ((k >> t) & 1) << (RL - 1 - t);
        const int m = (c << (LOGN - RL)) + r;
        a[k] = elem((k & 1) ? 2 * n - 1 - 2 * m : 2 * m);
    }
}
template <int LOGN, int RL, typename R>
__device__ __forceinline__ void store_group(vec2<R> *o, vec2<R> (&a)[1 << RL], int r, const vec2<R> *tw) {
    butterfly<false, LOGN, RL, R>(a, 0, 0, tw);
    const int i0 = LOGN == RL ? 0 : place<R>(brev(r, LOGN - RL ? LOGN - RL : 1) << RL);
#pragma unroll
    for (int k = 0; k < (1 << RL); k++) o[i0 ^ place<R>(k)] = a[k];
}

// The twiddles (n - 1) and the (cos, sin)(pi k / 2n) factors (n/2 + 1) of
// one axis, and its frequency weights (n, when w is given), into shared
// memory, every load of a thread issued before its first store (one memory
// round trip).  These are constant tables, so blocks stage them before
// waiting on the previous grid; the caller's barrier publishes them.
template <int LOGN, int NT, typename R>
__device__ __forceinline__ void stage_tables(vec2<R> *tw_s, vec2<R> *q_s, R *w_s, const vec2<R> *__restrict__ tw,
                                             const vec2<R> *__restrict__ q, const R *__restrict__ w) {
    constexpr int n = 1 << LOGN;
    constexpr int it_t = (n - 1 + NT - 1) / NT, it_q = (n / 2 + 1 + NT - 1) / NT, it_w = (n + NT - 1) / NT;
    vec2<R> vt[it_t], vq[it_q];
    R vw[it_w];
#pragma unroll
    for (int it = 0; it < it_t; it++) {
        const int i = threadIdx.x + it * NT;
        if (i < n - 1) vt[it] = tw[i];
    }
#pragma unroll
    for (int it = 0; it < it_q; it++) {
        const int i = threadIdx.x + it * NT;
        if (i <= n / 2) vq[it] = q[i];
    }
#pragma unroll
    for (int it = 0; it < it_w; it++) {
        const int i = threadIdx.x + it * NT;
        if (w && i < n) vw[it] = w[i];
    }
#pragma unroll
    for (int it = 0; it < it_t; it++) {
        const int i = threadIdx.x + it * NT;
        if (i < n - 1) tw_s[i] = vt[it];
    }
#pragma unroll
    for (int it = 0; it < it_q; it++) {
        const int i = threadIdx.x + it * NT;
        if (i <= n / 2) q_s[i] = vq[it];
    }
#pragma unroll
    for (int it = 0; it < it_w; it++) {
        const int i = threadIdx.x + it * NT;
        if (w && i < n) w_s[i] = vw[it];
    }
}

// Spectrum entry k (1 <= k <= n/2) of the DCT-III input X (entry n-k is its
// conjugate): (X[k] c + X[n-k] s, X[k] s - X[n-k] c) / 2.  At k = n/2 the two
// products are equal but for the tables' rounding; FIRST: the first of them is
// the one rounded by itself.
template <typename R, bool FIRST = false>
__device__ __forceinline__ vec2<R> dct3_spec(R xk, R xm, vec2<R> cs) {
    const R im = FIRST ? -dif2<R>(xm, cs.x, xk, cs.y) : dif2<R>(xk, cs.y, xm, cs.x);
    return mk2<R>((R)0.5 * sum2<R>(xk, cs.x, xm, cs.y), (R)0.5 * im);
}

// Entries k and n-k (bit-reversed positions) of the complex spectrum that
// carries DCT-III input a in its real part and b in its imaginary part.
template <typename R>
__device__ __forceinline__ void pack_spec(vec2<R> *o, int k, int m, int logn, vec2<R> sa, vec2<R> sb, bool self) {
    o[place<R>(brev(k, logn))] = mk2<R>(sa.x - sb.y, sa.y + sb.x);
    if (!self) o[place<R>(brev(m, logn))] = mk2<R>(sa.x + sb.y, sb.x - sa.y);
}

// Shared-memory bytes of the per-axis tables (twiddles, factors, weights).
template <typename R>
__host__ __device__ constexpr size_t table_bytes(int n) {
    return sizeof(vec2<R>) * ((size_t)n - 1 + n / 2 + 1) + sizeof(R) * n;
}

// Row pairs (pass 1) and rows (pass 3) per block, and threads.
template <int LOGN>
__host__ __device__ constexpr int seqs_per_block() {
    return kRowElems >> LOGN > 1 ? kRowElems >> LOGN : 1;
}
__host__ __device__ constexpr int row_threads(int logn) { return logn > 10 ? 2 * kThreads : kThreads; }
__host__ __device__ constexpr int col_threads(int logn) { return logn > 9 ? 2 * kThreads : kThreads; }

// ---- pass 1: rows along y --------------------------------------------------
template <int LOGN, typename R>
__global__ void __launch_bounds__(row_threads(LOGN))
k_fft_rows_fwd(const R *__restrict__ rho, R *__restrict__ T, int pairs, const vec2<R> *__restrict__ tw,
               const vec2<R> *__restrict__ q, const DevScalars *__restrict__ S) {
    using C = vec2<R>;
    constexpr int n = 1 << LOGN, NS = seqs_per_block<LOGN>(), NT = row_threads(LOGN);
    constexpr int RL = first_stages(LOGN), per = LOGN - RL;
    C *sm = smem_c<R>();
    C *tw_s = sm + NS * n, *q_s = tw_s + n - 1;
    stage_tables<LOGN, NT, R>(tw_s, q_s, nullptr, tw, q, nullptr);
    pdl_begin();
    if (S && S->done) return;
    const int x0 = blockIdx.x * pairs * 2;
    constexpr int li = ((NS << per) + NT - 1) / NT;
    C v[li][1 << RL];
#pragma unroll
    for (int it = 0; it < li; it++) {
        const int e = threadIdx.x + it * NT;
        if (e < (pairs << per)) {
            const R *ra = rho + (size_t)(x0 + 2 * (e >> per)) * n;
            load_group<LOGN, RL>(v[it], e & ((1 << per) - 1), [&](int y) { return mk2<R>(ra[y], ra[n + y]); });
        }
    }
    __syncthreads();  // the tables
#pragma unroll
    for (int it = 0; it < li; it++) {
        const int e = threadIdx.x + it * NT;
        if (e < (pairs << per)) store_group<LOGN, RL, R>(sm + ((e >> per) << LOGN), v[it], e & ((1 << per) - 1), tw_s);
    }
    __syncthreads();
    block_fft<false, LOGN, RL, NS, NT, R>(sm, pairs, tw_s);
    constexpr int pi_ = (NS * n / 2 + NT - 1) / NT;
#pragma unroll
    for (int it = 0; it < pi_; it++) {
        const int e = threadIdx.x + it * NT;
        if (e >= (pairs << (LOGN - 1))) break;
        const int p = e >> (LOGN - 1), k0 = e & (n / 2 - 1);
        const C *z = sm + (p << LOGN);
        R *ta = T + (size_t)(x0 + 2 * p) * n, *tb = ta + n;
        // entries k and n - k; entry 0's thread also takes n/2
        auto entry = [&](int k, C Z, C M, bool pair) {
            // V_a = (Z + conj M) / 2, V_b = (Z - conj M) / 2i
            const R ar = (R)0.5 * (Z.x + M.x), ai = (R)0.5 * (Z.y - M.y);
            const R br = (R)0.5 * (Z.y + M.y), bi = (R)-0.5 * (Z.x - M.x);
            const C cs = q_s[k];
            ta[k] = sum2<R>(ar, cs.x, ai, cs.y);
            tb[k] = sum2<R>(br, cs.x, bi, cs.y);
            if (pair) {
                ta[n - k] = dif2<R>(ar, cs.y, ai, cs.x);
                tb[n - k] = dif2<R>(br, cs.y, bi, cs.x);
            }
        };
        if (k0 == 0) entry(n / 2, z[place<R>(n / 2)], z[place<R>(n / 2)], false);
        const C Z = z[place<R>(k0)];
        entry(k0, Z, k0 ? z[place<R>(n - k0)] : Z, k0 != 0);
    }
}

// ---- pass 2: columns along x -----------------------------------------------
// COLS (2 or 4) columns per block, NT threads; column pairs
// (v0 + 2p, v0 + 2p + 1) share the forward FFT, the E-branch IFFT and the
// cosine-branch IFFT.  The spectral scale K[u][v] = kscale h_u h_v /
// (wx_u^2 + wy_v^2) (h_0 = 1/2, K[0][0] = 0) is formed here from the weight
// tables.  ColVec: COLS consecutive R values of a row, loaded as one vector.
template <typename R, int COLS>
struct ColVec;
template <>
struct ColVec<float, 2> {
    using T = float2;
};
template <>
struct ColVec<float, 4> {
    using T = float4;
};
template <>
struct ColVec<double, 2> {
    using T = double2;
};

template <int LOGN, int COLS, int NT, typename R>
__global__ void __launch_bounds__(NT)
k_fft_cols(const R *__restrict__ T, const R *__restrict__ wx, const R *__restrict__ wy, R kscale, R *__restrict__ X1,
           R *__restrict__ X2, int ny, const vec2<R> *__restrict__ tw, const vec2<R> *__restrict__ q,
           const DevScalars *__restrict__ S) {
    using C = vec2<R>;
    constexpr int n = 1 << LOGN;
    constexpr int NP = COLS / 2;
    constexpr int RL = first_stages(LOGN), per = LOGN - RL;
    using V = typename ColVec<R, COLS>::T;
    C *sm = smem_c<R>();
    C *fw = sm;  // NP packed forward sequences (columns v0 + 2p, v0 + 2p + 1)
    C *iv = sm;  // then COLS inverse sequences: E branch of each pair, then cosine branch of each pair
    C *tw_s = sm + COLS * n, *q_s = tw_s + n - 1;
    R *wx_s = (R *)(q_s + n / 2 + 1);
    stage_tables<LOGN, NT, R>(tw_s, q_s, wx_s, tw, q, wx);
    const int v0 = blockIdx.x * COLS;
    const V wvv = *reinterpret_cast<const V *>(wy + v0);
    const R *wvc = reinterpret_cast<const R *>(&wvv);
    pdl_begin();
    if (S && S->done) return;
    constexpr int li = ((1 << per) + NT - 1) / NT;
    C t[li][NP][1 << RL];
#pragma unroll
    for (int it = 0; it < li; it++) {
        const int r = threadIdx.x + it * NT;
        if (r >= (1 << per)) break;
        V raw[1 << RL];
        load_group<LOGN, RL>(raw, r, [&](int x) { return *reinterpret_cast<const V *>(T + (size_t)x * ny + v0); });
#pragma unroll
        for (int k = 0; k < (1 << RL); k++)
#pragma unroll
            for (int p = 0; p < NP; p++) {
                const R *tv = reinterpret_cast<const R *>(&raw[k]);
                t[it][p][k] = mk2<R>(tv[2 * p], tv[2 * p + 1]);
            }
    }
    __syncthreads();  // the tables
#pragma unroll
    for (int it = 0; it < li; it++) {
        const int r = threadIdx.x + it * NT;
        if (r >= (1 << per)) break;
#pragma unroll
        for (int p = 0; p < NP; p++) store_group<LOGN, RL, R>(fw + p * n, t[it][p], r, tw_s);
    }
    __syncthreads();
    block_fft<false, LOGN, RL, NP, NT, R>(fw, NP, tw_s);
    constexpr int pi_ = (NP * n / 2 + NT - 1) / NT;
    // the forward spectra into registers: the inverse sequences overwrite them
    C zk[pi_], zm[pi_];
#pragma unroll
    for (int it = 0; it < pi_; it++) {
        const int e = threadIdx.x + it * NT;
        if (e < NP * n / 2) {
            const int p = e >> (LOGN - 1), k = e & (n / 2 - 1);
            zk[it] = fw[p * n + place<R>(k)];
            zm[it] = fw[p * n + place<R>(k ? n - k : n / 2)];
        }
    }
    __syncthreads();
#pragma unroll
    for (int it = 0; it < pi_; it++) {
        const int e = threadIdx.x + it * NT;
        if (e >= NP * n / 2) break;
        const int p = e >> (LOGN - 1), k0 = e & (n / 2 - 1);
        C *oe = iv + p * n, *oc = iv + (NP + p) * n;
        // frequencies k and m = n - k of both columns; k = 0 and k = n/2 are
        // their own partners and share a thread
        auto entry = [&](auto first, int k, int m, C Z, C M, bool self) {
            constexpr bool FIRST = decltype(first)::value;
            const C cs = q_s[k];
            const R re[2] = {(R)0.5 * (Z.x + M.x), (R)0.5 * (Z.y + M.y)};
            const R im[2] = {(R)0.5 * (Z.y - M.y), (R)-0.5 * (Z.x - M.x)};
            const R wk = wx_s[k], wm = wx_s[m];
            R pk[2], pm[2];
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int v = v0 + 2 * p + h;
                const R wv = wvc[2 * p + h];
                const R cv = (v == 0 ? (R)0.5 : (R)1) * kscale;
                // DCT-II outputs k and n-k, times K
                const R kk = (k == 0) ? (v == 0 ? (R)0 : (R)0.5 * cv / (wv * wv)) : cv / fma_r(wk, wk, wv * wv);
                pk[h] = sum2<R>(re[h], cs.x, im[h], cs.y) * kk;
                pm[h] = self ? pk[h] : dif2<R>(re[h], cs.y, im[h], cs.x) * (cv / fma_r(wm, wm, wv * wv));
            }
            if (k == 0) {
                oe[0] = mk2<R>((R)0, (R)0);  // sine branch: b[0] = 0
                oc[0] = mk2<R>(pk[0], pk[1]);
                return;
            }
            // sine branch: b[k] = wx[n-k] P[n-k], b[n-k] = wx[k] P[k]
            pack_spec<R>(oe, k, m, LOGN, dct3_spec<R, FIRST>(wm * pm[0], wk * pk[0], cs),
                         dct3_spec<R, FIRST>(wm * pm[1], wk * pk[1], cs), self);
            pack_spec<R>(oc, k, m, LOGN, dct3_spec<R, FIRST>(pk[0], pm[0], cs), dct3_spec<R, FIRST>(pk[1], pm[1], cs),
                         self);
        };
        if (k0 == 0) {
            entry(std::false_type{}, 0, 0, zk[it], zk[it], true);
            // Both roundings of this one frequency are equally near its value.
            // One for all lengths would move 512^2 placements: the loop
            // amplifies a last place to 1.2e-3 (FP32, 200k cells, 16 steps), so
            // 512 keeps the one its placements have had.
            entry(std::bool_constant<LOGN == 9>{}, n / 2, n / 2, zm[it], zm[it], true);
        } else {
            entry(std::false_type{}, k0, n - k0, zk[it], zm[it], false);
        }
    }
    __syncthreads();
    block_fft<true, LOGN, 0, COLS, NT, R>(iv, COLS, tw_s);
    constexpr int oi = (n + NT - 1) / NT;
#pragma unroll
    for (int it = 0; it < oi; it++) {
        const int x = threadIdx.x + it * NT;
        if (x >= n) break;
        const int m = place<R>(makhoul(x, n));
        const R sg = (x & 1) ? (R)-1 : (R)1;
        V o1, o2;
        R *f1 = reinterpret_cast<R *>(&o1), *f2 = reinterpret_cast<R *>(&o2);
#pragma unroll
        for (int p = 0; p < NP; p++) {
            const C e = iv[p * n + m], c = iv[(NP + p) * n + m];
            f1[2 * p] = sg * e.x;
            f1[2 * p + 1] = sg * e.y;
            f2[2 * p] = c.x;
            f2[2 * p + 1] = c.y;
        }
        *reinterpret_cast<V *>(X1 + (size_t)x * ny + v0) = o1;
        *reinterpret_cast<V *>(X2 + (size_t)x * ny + v0) = o2;
    }
}

// ---- pass 3: rows along y, to the field -------------------------------------
template <typename R>
struct Quad;
template <>
struct Quad<float> {
    using T = float4;
    static __device__ __forceinline__ float4 make(float a, float b, float c, float d) { return make_float4(a, b, c, d); }
};
template <>
struct Quad<double> {
    struct T {
        double x, y, z, w;
    };
    static __device__ __forceinline__ T make(double a, double b, double c, double d) { return T{a, b, c, d}; }
};

template <int LOGN, bool PHI, typename R>
__global__ void __launch_bounds__(row_threads(LOGN))
k_fft_rows_inv(const R *__restrict__ X1, const R *__restrict__ X2, const R *__restrict__ wy, vec2<R> *__restrict__ field,
               R *__restrict__ phi, int rows, const vec2<R> *__restrict__ tw, const vec2<R> *__restrict__ q,
               const DevScalars *__restrict__ S) {
    using C = vec2<R>;
    constexpr int n = 1 << LOGN, NS = seqs_per_block<LOGN>(), NT = row_threads(LOGN);
    constexpr int nseq = PHI ? 2 : 1;  // per row: (E_x, E_y) packed, then phi
    C *sm = smem_c<R>();
    C *tw_s = sm + NS * nseq * n, *q_s = tw_s + n - 1;
    R *wy_s = (R *)(q_s + n / 2 + 1);
    stage_tables<LOGN, NT, R>(tw_s, q_s, wy_s, tw, q, wy);
    pdl_begin();
    if (S && S->done) return;
    const int x0 = blockIdx.x * rows;
    constexpr int li = (NS * n / 2 + NT - 1) / NT;
    typename Quad<R>::T v[li];  // X1[k], X1[m], X2[k], X2[m]; m = n - k, but n/2 for k = 0
#pragma unroll
    for (int it = 0; it < li; it++) {
        const int e = threadIdx.x + it * NT;
        if (e < (rows << (LOGN - 1))) {
            const int r = e >> (LOGN - 1), k = e & (n / 2 - 1);
            const int m = k ? n - k : n / 2;
            const size_t base = (size_t)(x0 + r) * n;
            v[it] = Quad<R>::make(X1[base + k], X1[base + m], X2[base + k], X2[base + m]);
        }
    }
    __syncthreads();  // the tables
#pragma unroll
    for (int it = 0; it < li; it++) {
        const int e = threadIdx.x + it * NT;
        if (e >= (rows << (LOGN - 1))) break;
        const int r = e >> (LOGN - 1), k0 = e & (n / 2 - 1);
        C *o = sm + ((r * nseq) << LOGN);
        auto entry = [&](int k, int m, R a_k, R a_m, R b_k, R b_m, bool self) {
            const C cs = q_s[k];
            // sine branch of wy X2: b[k] = wy[n-k] X2[n-k], b[n-k] = wy[k] X2[k]
            pack_spec<R>(o, k, m, LOGN, dct3_spec<R>(a_k, a_m, cs), dct3_spec<R>(wy_s[m] * b_m, wy_s[k] * b_k, cs), self);
            if (PHI) pack_spec<R>(o + n, k, m, LOGN, dct3_spec<R>(b_k, b_m, cs), mk2<R>((R)0, (R)0), self);
        };
        if (k0 == 0) {  // frequencies 0 and n/2, each its own partner
            o[0] = mk2<R>(v[it].x, (R)0);
            if (PHI) o[n] = mk2<R>(v[it].z, (R)0);
            entry(n / 2, n / 2, v[it].y, v[it].y, v[it].w, v[it].w, true);
        } else {
            entry(k0, n - k0, v[it].x, v[it].y, v[it].z, v[it].w, false);
        }
    }
    __syncthreads();
    block_fft<true, LOGN, 0, NS * nseq, NT, R>(sm, rows * nseq, tw_s);
    constexpr int oi = (NS * n + NT - 1) / NT;
#pragma unroll
    for (int it = 0; it < oi; it++) {
        const int e = threadIdx.x + it * NT;
        if (e >= (rows << LOGN)) break;
        const int r = e >> LOGN, y = e & (n - 1);
        const int m = place<R>(makhoul(y, n));
        const C *z = sm + ((r * nseq) << LOGN);
        const size_t at = (size_t)(x0 + r) * n + y;
        field[at] = mk2<R>(z[m].x, (y & 1) ? -z[m].y : z[m].y);
        if (PHI) phi[at] = z[n + m].x;
    }
}

// Kernel instances for log2 n = kMinLog .. kMaxLog, per precision.
constexpr int kLogs = kMaxLog - kMinLog + 1;
template <typename R>
struct FftFns {
    using RowsFwdFn = void (*)(const R *, R *, int, const vec2<R> *, const vec2<R> *, const DevScalars *);
    using ColsFn = void (*)(const R *, const R *, const R *, R, R *, R *, int, const vec2<R> *, const vec2<R> *,
                            const DevScalars *);
    using RowsInvFn = void (*)(const R *, const R *, const R *, vec2<R> *, R *, int, const vec2<R> *,
                               const vec2<R> *, const DevScalars *);
    template <int... L>
    static constexpr std::array<RowsFwdFn, sizeof...(L)> rows_fwd(std::integer_sequence<int, L...>) {
        return {k_fft_rows_fwd<L + kMinLog, R>...};
    }
    template <int COLS, int... L>
    static constexpr std::array<ColsFn, sizeof...(L)> cols(std::integer_sequence<int, L...>) {
        return {k_fft_cols<L + kMinLog, COLS, col_threads(L + kMinLog), R>...};
    }
    // two columns are half a sector in FP64
    static constexpr std::array<ColsFn, kLogs> cols4() {
        if constexpr (sizeof(R) == 4)
            return cols<4>(std::make_integer_sequence<int, kLogs>{});
        else
            return {};
    }
    static ColsFn cols_fn(int logn, int cols) { return cols == 2 ? kCols2[logn - kMinLog] : kCols4[logn - kMinLog]; }
    template <bool PHI, int... L>
    static constexpr std::array<RowsInvFn, sizeof...(L)> rows_inv(std::integer_sequence<int, L...>) {
        return {k_fft_rows_inv<L + kMinLog, PHI, R>...};
    }
    using LogSeq = std::make_integer_sequence<int, kLogs>;
    static const std::array<RowsFwdFn, kLogs> kRowsFwd;
    static const std::array<ColsFn, kLogs> kCols2, kCols4;
    static const std::array<RowsInvFn, kLogs> kRowsInv, kRowsInvPhi;
};
template <typename R>
const std::array<typename FftFns<R>::RowsFwdFn, kLogs> FftFns<R>::kRowsFwd = FftFns<R>::rows_fwd(LogSeq{});
template <typename R>
const std::array<typename FftFns<R>::ColsFn, kLogs> FftFns<R>::kCols2 = FftFns<R>::template cols<2>(LogSeq{});
template <typename R>
const std::array<typename FftFns<R>::ColsFn, kLogs> FftFns<R>::kCols4 = FftFns<R>::cols4();
template <typename R>
const std::array<typename FftFns<R>::RowsInvFn, kLogs> FftFns<R>::kRowsInv = FftFns<R>::template rows_inv<false>(LogSeq{});
template <typename R>
const std::array<typename FftFns<R>::RowsInvFn, kLogs> FftFns<R>::kRowsInvPhi =
    FftFns<R>::template rows_inv<true>(LogSeq{});

int seqs_per_block_rt(int logn) { return std::max(1, kRowElems >> logn); }

template <typename T>
int upload_vec(void *&dst, const std::vector<T> &src, std::string &err) {
    if (cudaMalloc(&dst, src.size() * sizeof(T)) != cudaSuccess) {
        err = "cudaMalloc failed for FFT tables";
        return EP_ERR_NOMEM;
    }
    if (cudaMemcpy(dst, src.data(), src.size() * sizeof(T), cudaMemcpyHostToDevice) != cudaSuccess) {
        err = "copy of FFT tables failed";
        return EP_ERR_CUDA;
    }
    return EP_OK;
}

template <typename R>
void tables(int n, std::vector<vec2<R>> &tw, std::vector<vec2<R>> &q) {
    const double pi = 3.14159265358979323846;
    tw.assign(n - 1, mk2<R>((R)0, (R)0));
    for (int h = 1; h < n; h <<= 1)
        for (int j = 0; j < h; j++) tw[h - 1 + j] = mk2<R>((R)cos(pi * j / h), (R)-sin(pi * j / h));
    q.assign(n / 2 + 1, mk2<R>((R)0, (R)0));
    for (int k = 0; k <= n / 2; k++) q[k] = mk2<R>((R)cos(pi * k / (2.0 * n)), (R)sin(pi * k / (2.0 * n)));
}

}  // namespace

template <typename R>
int FftPasses<R>::init(FftPlan *f, int nx, int ny, const std::vector<double> &wx, const std::vector<double> &wy,
                       std::string &err) {
    const int lx = f->lognx, ly = f->logny;
    std::vector<vec2<R>> tw, q;
    int rc;
    tables<R>(nx, tw, q);
    if ((rc = upload_vec(f->twx, tw, err)) || (rc = upload_vec(f->qx, q, err))) return rc;
    tables<R>(ny, tw, q);
    if ((rc = upload_vec(f->twy, tw, err)) || (rc = upload_vec(f->qy, q, err))) return rc;
    std::vector<R> wxr(nx), wyr(ny);
    for (int u = 0; u < nx; u++) wxr[u] = (R)wx[u];
    for (int v = 0; v < ny; v++) wyr[v] = (R)wy[v];
    if ((rc = upload_vec(f->wx, wxr, err)) || (rc = upload_vec(f->wy, wyr, err))) return rc;
    f->kscale = (double)(R)(4.0 / nx / ny);
    if (cudaMalloc(&f->T, sizeof(R) * nx * ny) != cudaSuccess ||
        cudaMalloc(&f->X, sizeof(R) * 2 * nx * ny) != cudaSuccess) {
        err = "cudaMalloc failed for FFT intermediates";
        return EP_ERR_NOMEM;
    }
    const int nsf = seqs_per_block_rt(ly);
    f->pairs_fwd = std::min(nsf, nx / 2);
    f->rows_inv = std::min(nsf, nx);
    f->cols = col_count<R>(ny);
    f->smem_rows_fwd = sizeof(vec2<R>) * (size_t)nsf * ny + table_bytes<R>(ny);
    f->smem_cols = sizeof(vec2<R>) * (size_t)f->cols * nx + table_bytes<R>(nx);
    f->smem_rows_inv = sizeof(vec2<R>) * (size_t)nsf * 2 * ny + table_bytes<R>(ny);
    using F = FftFns<R>;
    const std::pair<const void *, size_t> attr[4] = {
        {(const void *)F::kRowsFwd[ly - kMinLog], f->smem_rows_fwd},
        {(const void *)F::cols_fn(lx, f->cols), f->smem_cols},
        {(const void *)F::kRowsInv[ly - kMinLog], f->smem_rows_inv - sizeof(vec2<R>) * (size_t)nsf * ny},
        {(const void *)F::kRowsInvPhi[ly - kMinLog], f->smem_rows_inv}};
    for (auto &a : attr) {
        if (a.second > 48 * 1024 &&
            cudaFuncSetAttribute(a.first, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)a.second) != cudaSuccess) {
            err = "shared memory of the FFT Poisson kernels refused";
            return EP_ERR_UNSUPPORTED;
        }
        // the loop's split, unless this block needs more (1 KB per block is
        // reserved by the hardware)
        cudaFuncSetAttribute(a.first, cudaFuncAttributePreferredSharedMemoryCarveout,
                             carveout_percent(std::max(kLoopSmemBytes, a.second + 1024)));
    }
    return EP_OK;
}

template <typename R>
void FftPasses<R>::run(const FftPlan *f, int nx, int ny, const R *rho, vec2<R> *field, R *phi, const DevScalars *S,
                       cudaStream_t st) {
    using F = FftFns<R>;
    R *X1 = (R *)f->X, *X2 = X1 + (size_t)nx * ny;
    const int pr = launch_priority(true);
    const int ly = f->logny - kMinLog;
    launch_kp(F::kRowsFwd[ly], nx / (2 * f->pairs_fwd), row_threads(f->logny), f->smem_rows_fwd, st, pr, rho, (R *)f->T,
              f->pairs_fwd, (const vec2<R> *)f->twy, (const vec2<R> *)f->qy, S);
    launch_kp(F::cols_fn(f->lognx, f->cols), ny / f->cols, col_threads(f->lognx), f->smem_cols, st, pr, (const R *)f->T, (const R *)f->wx,
              (const R *)f->wy, (R)f->kscale, X1, X2, ny, (const vec2<R> *)f->twx, (const vec2<R> *)f->qx, S);
    const size_t phi_seqs = sizeof(vec2<R>) * (size_t)seqs_per_block_rt(f->logny) * ny;
    launch_kp(phi ? F::kRowsInvPhi[ly] : F::kRowsInv[ly], nx / f->rows_inv, row_threads(f->logny),
              phi ? f->smem_rows_inv : f->smem_rows_inv - phi_seqs, st, pr, (const R *)X1, (const R *)X2,
              (const R *)f->wy, field, phi, f->rows_inv, (const vec2<R> *)f->twy, (const vec2<R> *)f->qy, S);
}

}  // namespace ep
