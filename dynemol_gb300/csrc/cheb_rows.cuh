// Chebyshev propagation of one trajectory on an explicit Hs whose rows stay in
// shared memory for the whole launch (FP64 and DF64: up to 1,250 AOs with four columns and
// about 1,900 with two; FP32: 2,432).
//
// At these sizes an order of cheb_kernel (cheb.cu) is latency, not work: a grid
// barrier (2,750 cycles with the fastest form of it), the previous vector staged
// through shared memory (850), 23 to 31 FP64 adds per warp to sum accumulators
// over lanes (a warp instruction takes GB300's FP64 unit 76 cycles whatever it
// does) against 16 products at N = 450.  Here
//   - there is no grid barrier: every 8-byte element of v_k is published with the
//     order's tag beside it as one 16-byte word (a 128-bit access is a single copy),
//     and a reader polls the words it needs until their tags match.  Two buffers
//     suffice: a CTA writes v_{k+2} only after it has read all of v_{k+1}, which
//     every CTA wrote after it had read all of v_k;
//   - lane (s, c) of a warp owns component c of the columns j = s mod S
//     (S = 32 / C), so the word a lane polls is the operand it multiplies, and a
//     row's sum meets over S lanes instead of 32;
//   - v_{k-1}, v_{k-2} and the accumulated sum of a CTA's own rows stay in registers.
// Bound: FP64 the FP64 unit above about N = 700, the exchange (about 1,200 cycles)
// below; measured figures at launch_cheb_rows.
//
// Every wait is bounded: a CTA whose poll gives up reports ELHL_ERR_TIMEOUT and
// leaves, and the others leave when they see it.
#pragma once

#include <cuda_runtime.h>

#include "df64.cuh"
#include "elhl_internal.cuh"
#include "exchange.cuh"

namespace elhl {
namespace rows {

constexpr int kThreads = 256, kWarps = kThreads / 32;
constexpr int kBatch = 8;                      // words in flight per lane
constexpr size_t kSmemLimit = 220 * 1024;

// ---- arithmetics -------------------------------------------------------------
// Word: what a word carries; C words per column j (components, or complex columns
// in FP32).  Sum: a row's running sum of one word's products.
struct F64 {
    using H = double;
    using Sum = double;
    static constexpr int kPerColumn = 2;  // words per complex column
    static __device__ __forceinline__ Sum zero() { return 0.0; }
    static __device__ __forceinline__ void fma_(Sum &a, const H &h, unsigned long long w) {
        a = fma(h, __longlong_as_double((long long)w), a);
    }
    static __device__ __forceinline__ Sum add(const Sum &a, const Sum &b) { return a + b; }
    static __device__ __forceinline__ Sum shfl(const Sum &a, int o) { return __shfl_xor_sync(0xffffffffu, a, o); }
};
struct F32 {
    using H = float;
    using Sum = float2;
    static constexpr int kPerColumn = 1;
    static __device__ __forceinline__ Sum zero() { return make_float2(0.f, 0.f); }
    static __device__ __forceinline__ void fma_(Sum &a, const H &h, unsigned long long w) {
        a.x = fmaf(h, __uint_as_float((unsigned)w), a.x);
        a.y = fmaf(h, __uint_as_float((unsigned)(w >> 32)), a.y);
    }
    static __device__ __forceinline__ Sum add(const Sum &a, const Sum &b) { return make_float2(a.x + b.x, a.y + b.y); }
    static __device__ __forceinline__ Sum shfl(const Sum &a, int o) {
        return make_float2(__shfl_xor_sync(0xffffffffu, a.x, o), __shfl_xor_sync(0xffffffffu, a.y, o));
    }
};
struct DF64 {
    using H = float2;  // (hi, lo)
    using Sum = float2;
    static constexpr int kPerColumn = 2;
    static __device__ __forceinline__ Sum zero() { return make_float2(0.f, 0.f); }
    static __device__ __forceinline__ void fma_(Sum &a, const H &h, unsigned long long w) {
        df_fma(a.x, a.y, h.x, h.y, __uint_as_float((unsigned)w), __uint_as_float((unsigned)(w >> 32)));
    }
    static __device__ __forceinline__ Sum add(const Sum &a, const Sum &b) {
        float h = a.x, l = a.y;
        df_add(h, l, b.x, b.y);
        return make_float2(h, l);
    }
    static __device__ __forceinline__ Sum shfl(const Sum &a, int o) {
        return make_float2(__shfl_xor_sync(0xffffffffu, a.x, o), __shfl_xor_sync(0xffffffffu, a.y, o));
    }
};
__device__ __forceinline__ unsigned long long pack2(float x, float y) {
    return (unsigned long long)__float_as_uint(x) | ((unsigned long long)__float_as_uint(y) << 32);
}

// One output word (row, component or complex column) of a CTA: the recurrence
// state, held by the four lanes that sum its partials.
template <typename A> struct Out;
template <> struct Out<F64> {
    double v1 = 0.0, v2 = 0.0, acc = 0.0;
    // order 0 from the scaled input element x (re or im) and its partner
    __device__ unsigned long long start(double x, double xo, bool im, double2 c0, float) {
        v1 = x;
        acc = im ? c0.x * x + c0.y * xo : c0.x * x - c0.y * xo;
        return (unsigned long long)__double_as_longlong(x);
    }
    __device__ unsigned long long step(double y, int k) {
        const double v = k == 1 ? y : 2.0 * y - v2;
        v2 = v1;
        v1 = v;
        return (unsigned long long)__double_as_longlong(v);
    }
    __device__ void accumulate(bool im, double2 ck) {
        const double o = __shfl_xor_sync(0xffffffffu, v1, 4);  // the other part (re <-> im)
        acc += im ? ck.x * v1 + ck.y * o : ck.x * v1 - ck.y * o;
    }
};
template <> struct Out<DF64> {
    double v1 = 0.0, v2 = 0.0, acc = 0.0, exact = 0.0;
    __device__ unsigned long long round_to_pair(double v) {
        const float2 p = df_split(v);
        exact = v;
        v2 = v1;
        v1 = (double)p.x + (double)p.y;  // the recurrence goes on with the published pair
        return pack2(p.x, p.y);
    }
    __device__ unsigned long long start(double x, double xo, bool im, double2 c0, float) {
        acc = im ? c0.x * x + c0.y * xo : c0.x * x - c0.y * xo;
        return round_to_pair(x);
    }
    __device__ unsigned long long step(float2 s, int k) {
        const double y = (double)s.x + (double)s.y;
        return round_to_pair(k == 1 ? y : 2.0 * y - v2);
    }
    __device__ void accumulate(bool im, double2 ck) {
        const double o = __shfl_xor_sync(0xffffffffu, exact, 4);
        acc += im ? ck.x * exact + ck.y * o : ck.x * exact - ck.y * o;
    }
};
template <> struct Out<F32> {
    float2 v1 = make_float2(0.f, 0.f), v2 = make_float2(0.f, 0.f);
    double2 acc = make_double2(0.0, 0.0);
    float d = 0.f;  // the FP32 rounding residual of Hs's diagonal, added back before v is rounded once
    __device__ unsigned long long start(double2 x, double2 c0, float dcorr) {
        d = dcorr;
        v1 = make_float2((float)x.x, (float)x.y);
        acc = make_double2(c0.x * x.x - c0.y * x.y, c0.x * x.y + c0.y * x.x);
        return pack2(v1.x, v1.y);
    }
    __device__ unsigned long long step(float2 y, int k) {
        const float dr = __fmul_rn(d, v1.x), di = __fmul_rn(d, v1.y);
        float2 v;
        if (k == 1) {
            v = make_float2(__fadd_rn(y.x, dr), __fadd_rn(y.y, di));
        } else {
            v.x = two_sum_plus(__fmul_rn(2.f, y.x), -v2.x, __fmul_rn(2.f, dr));
            v.y = two_sum_plus(__fmul_rn(2.f, y.y), -v2.y, __fmul_rn(2.f, di));
        }
        v2 = v1;
        v1 = v;
        return pack2(v.x, v.y);
    }
    __device__ void accumulate(bool, double2 ck) {
        const double vr = (double)v1.x, vi = (double)v1.y;
        acc.x += ck.x * vr - ck.y * vi;
        acc.y += ck.x * vi + ck.y * vr;
    }
};

// columns padded to whole lane groups
template <int C> __host__ __device__ constexpr int padded(int n) { return (n + 32 / C - 1) / (32 / C) * (32 / C); }

// dynamic shared memory: the operator's rows [R][padded N], the warps' sums [2][kWarps][R C]
template <typename A, int C>
constexpr size_t smem_bytes(int n, int R) {
    return (size_t)R * padded<C>(n) * sizeof(typename A::H) + 2 * (size_t)kWarps * R * C * sizeof(typename A::Sum);
}

template <typename A, int C, int R>
__global__ void __launch_bounds__(kThreads, 1) cheb_rows_kernel(const RowsLaunch L) {
    using H = typename A::H;
    using Sum = typename A::Sum;
    constexpr int S = 32 / C;                              // columns per warp step
    constexpr int kPasses = (4 * R * C + kThreads - 1) / kThreads;
    extern __shared__ __align__(16) unsigned char dyn[];
    __shared__ int s_abort;
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int N = L.N, np = padded<C>(N), groups = np / S;
    const int r0 = blockIdx.x * R;
    H *sh = reinterpret_cast<H *>(dyn);
    Sum *part = reinterpret_cast<Sum *>(sh + (size_t)R * np);
    if (__syncthreads_or(*(volatile const int *)L.error)) return;  // an earlier launch of this call gave up
    if ((int)blockIdx.x + 1 == L.exit_cta1) return;  // test hook: the other CTAs' waits run out
    const unsigned long long limit = L.barrier_ns ? L.barrier_ns : kBarrierNs;
    if (tid == 0) s_abort = 0;
    const H *M = static_cast<const H *>(L.H);
    for (int q = tid; q < R * np; q += kThreads) {  // Hs symmetric: row i is the contiguous column i
        const int r = q / np, j = q % np;
        sh[q] = r0 + r < N && j < N ? M[(size_t)(r0 + r) * L.ld + j] : H{};
    }

    // ---- order 0: v_0 = s phi, acc = c_0 v_0
    Out<A> out[kPasses];
    const int q4 = tid & 3;
    auto word_of = [&](int p) { return (tid >> 2) + p * (kThreads / 4); };  // output word of pass p: row * C + component
#pragma unroll
    for (int p = 0; p < kPasses; ++p) {
        const int w = word_of(p), row = r0 + w / C, c = w % C;
        const bool in = w < R * C && row < N;
        const double2 c0 = L.coef[0];
        const int col = A::kPerColumn == 2 ? c >> 1 : c;
        double2 x = make_double2(0.0, 0.0);
        if (in) {
            x = L.phi[(size_t)row * L.m + col];
            if (L.scale) {
                const double sc = L.scale[col % L.P];
                x.x *= sc;
                x.y *= sc;
            }
        }
        const float d = in && L.dcorr ? L.dcorr[row] : 0.f;
        unsigned long long v;
        if constexpr (A::kPerColumn == 2)
            v = out[p].start((c & 1) ? x.y : x.x, (c & 1) ? x.x : x.y, c & 1, c0, d);
        else
            v = out[p].start(x, c0, d);
        if (in && q4 == 0) publish(L.xbuf[0] + (size_t)row * C + c, v, L.tag0);
    }
    __syncthreads();

    for (int k = 1; k <= L.K; ++k) {
        const unsigned long long want = L.tag0 + (unsigned long long)(k - 1);
        const ulonglong2 *src = (k & 1) ? L.xbuf[0] : L.xbuf[1];  // v_{k-1}
        ulonglong2 *dst = (k & 1) ? L.xbuf[1] : L.xbuf[0];
        const double2 ck = L.coef[k];
        Sum acc[R];
#pragma unroll
        for (int r = 0; r < R; ++r) acc[r] = A::zero();
        // word of (group, lane): column group * S + lane / C, component lane % C
        auto load = [&](int g, ulonglong2 (&w)[kBatch]) {
#pragma unroll
            for (int u = 0; u < kBatch; ++u) {
                const int e = (g + u * kWarps) * 32 + lane;
                w[u] = make_ulonglong2(0ull, want);
                if (e < N * C) w[u] = fetch(src + e);
            }
        };
        auto use = [&](int g, ulonglong2 (&w)[kBatch]) {
            if (!await_words(w, want, src + g * 32 + lane, kWarps * 32, L.error, limit)) s_abort = 1;
#pragma unroll
            for (int u = 0; u < kBatch; ++u) {
                const int gu = g + u * kWarps;
                if (gu < groups) {
                    const H *h = sh + (size_t)gu * S + lane / C;
#pragma unroll
                    for (int r = 0; r < R; ++r) A::fma_(acc[r], h[(size_t)r * np], w[u].x);
                }
            }
        };
        ulonglong2 wa[kBatch], wb[kBatch];
        load(warp, wa);
        for (int g = warp; g < groups; g += 2 * kBatch * kWarps) {
            load(g + kBatch * kWarps, wb);
            use(g, wa);
            if (g + kBatch * kWarps >= groups) break;
            load(g + 2 * kBatch * kWarps, wa);
            use(g + kBatch * kWarps, wb);
        }
        // a row's sum over the S lanes of a component: halve the rows a lane holds with each
        // lane bit (an odd one is summed by both), then plain sums; idx: the rows it holds
        int idx[R];
#pragma unroll
        for (int r = 0; r < R; ++r) idx[r] = r;
        int held = R;
        {
            int n = R;
#pragma unroll
            for (int o = 16; o >= C; o >>= 1) {
                const int h = (n + 1) / 2;
                const bool upper = (lane & o) != 0;
#pragma unroll
                for (int i = 0; i < R; ++i) {
                    if (i >= h) continue;
                    if (i + h < n) {
                        const Sum send = upper ? acc[i] : acc[i + h];
                        const Sum keep = upper ? acc[i + h] : acc[i];
                        acc[i] = A::add(keep, A::shfl(send, o));
                        idx[i] = upper ? idx[i + h] : idx[i];
                    } else {
                        acc[i] = A::add(acc[i], A::shfl(acc[i], o));
                    }
                }
                n = h;
            }
            held = n;
        }
        Sum *mine = part + ((size_t)(k & 1) * kWarps + warp) * R * C;
#pragma unroll
        for (int i = 0; i < R; ++i)
            if (i < held) mine[idx[i] * C + lane % C] = acc[i];
        __syncthreads();
        if (s_abort) return;
        // ---- the order's new words: four lanes per word sum the eight warps' partials
        const Sum *sums = part + (size_t)(k & 1) * kWarps * R * C;
#pragma unroll
        for (int p = 0; p < kPasses; ++p) {
            const int w = word_of(p), c = w % C, row = r0 + w / C;
            const int wc = w < R * C ? w : 0;
            Sum s = A::add(sums[(size_t)(2 * q4) * R * C + wc], sums[(size_t)(2 * q4 + 1) * R * C + wc]);
            s = A::add(s, A::shfl(s, 1));
            s = A::add(s, A::shfl(s, 2));
            const unsigned long long v = out[p].step(s, k);
            if (w < R * C && row < N && q4 == 0)
                publish(dst + (size_t)row * C + c, v, L.tag0 + (unsigned long long)k);
        }
#pragma unroll
        for (int p = 0; p < kPasses; ++p) out[p].accumulate((word_of(p) % C) & 1, ck);
    }
#pragma unroll
    for (int p = 0; p < kPasses; ++p) {
        const int w = word_of(p), row = r0 + w / C, c = w % C;
        if (w >= R * C || row >= N || q4 != 0) continue;
        if constexpr (A::kPerColumn == 2)
            reinterpret_cast<double *>(L.acc)[((size_t)row * L.m + (c >> 1)) * 2 + (c & 1)] = out[p].acc;
        else
            L.acc[(size_t)row * L.m + c] = out[p].acc;
    }
}

template <typename A, int C, int R>
cudaError_t launch(const RowsLaunch &L, cudaStream_t st) {
    auto kern = cheb_rows_kernel<A, C, R>;
    const size_t smem = smem_bytes<A, C>(L.N, R);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    RowsLaunch copy = L;
    const int grid = (L.N + R - 1) / R;
    if (copy.exit_cta1 > grid) copy.exit_cta1 = grid;
    void *args[] = {&copy};
    e = cudaLaunchCooperativeKernel((const void *)kern, dim3(grid), dim3(kThreads), args, smem, st);
    count_launch();
    return e;
}

}  // namespace rows
}  // namespace elhl
