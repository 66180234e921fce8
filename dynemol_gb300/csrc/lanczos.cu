// Spectral bounds of the Chebyshev operator by Lanczos, in FP64 on the FP64
// pipe, all k steps in one cooperative launch (no host round trip, no library
// GEMV).  The operator is
//   explicit: H~ (symmetric, both triangles stored), w = H~ q:
//             lanczos_rows_kernel (below), while its rows fit in shared memory;
//   implicit: H~ = G h G^T with G = L^-1 lower triangular and its transpose
//             Gt stored, w = G (h (G^T q)) in three column-dot phases:
//             lanczos64_kernel, which also takes the explicit operator of larger bases.
// In lanczos64_kernel every product is a set of column dot products M(:, i) . x (columns are
// contiguous in the column-major storage, so the reads coalesce): CTA c takes
// the columns i = c, c + grid, ..., one warp per column, so that every SM
// reads the same share of the matrix; x sits in shared memory when it fits.
// A product with q_j = r_{j-1} / beta_{j-1} is formed from the unnormalised
// r_{j-1} and scaled afterwards, so q_j is never written out.  The dot
// products alpha_j = w.q_j and |w|^2 are summed per CTA in a fixed order and
// then over the CTAs in CTA order: the same grid gives the same bits.
// The reference's adaptive-tau Taylor steps (ElHl_Chebyshev.f:148-268) need
// no spectral interval; the Chebyshev expansion does, and this is its source.
#include <algorithm>

#include "elhl_internal.cuh"
#include "exchange.cuh"
#include "grid_sync.cuh"

namespace elhl {
namespace {

constexpr int kLzThreads = 512, kLzWarps = kLzThreads / 32;
constexpr int kXsCap = 25600;  // x in shared memory up to 200 KB

struct LzArgs {
    int n, ld, k;
    const double *H;   // explicit H~, or h of the implicit operator
    const double *G;   // implicit: G (lower), nullptr for the explicit operator
    const double *Gt;  // implicit: G^T (upper)
    double *r;         // [4][ld] rotating unnormalised Lanczos vectors r_{j-1}
    double *t;         // [2][ld] implicit intermediates G^T q, h G^T q
    double *part;      // [2][grid] per-CTA partial sums
    double *rec;       // alpha [k], beta [k], steps used [1]
    unsigned *bar_count;  // grid barrier: two words, one 64-bit count (zero at the launch)
    int *err;
};

// Scalar work is done by one warp and broadcast through shared memory: GB300's
// FP64 pipe retires under two FMAs per clock per SM, so 512 threads repeating a
// 152-term sum or a square root would cost tens of microseconds per step.
// red: kLzWarps warp partials, then the broadcast slots.
constexpr int kRedSlots = kLzWarps + 3;

// block sum of one value per thread in a fixed order (every thread returns it)
__device__ double block_sum(double v, double *red) {
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (warp == 0) {
        double s = lane < kLzWarps ? red[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) red[kLzWarps] = s;
    }
    __syncthreads();
    const double s = red[kLzWarps];
    __syncthreads();
    return s;
}

// the sum of part[0 .. g) in a fixed order (lane-strided partial sums, then a
// shuffle tree), or its square root when root is set (then *inv = 1 / root);
// every thread returns it
__device__ double grid_sum(const double *part, int g, bool root, double *red, double *inv = nullptr) {
    const int lane = threadIdx.x % 32;
    if (threadIdx.x < 32) {
        double s = 0.0;
        for (int c = lane; c < g; c += 32) s += __ldcg(part + c);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
        if (lane == 0) {
            if (root) s = sqrt(s);
            red[kLzWarps + 1] = s;
            red[kLzWarps + 2] = root ? 1.0 / s : 0.0;
        }
    }
    __syncthreads();
    const double s = red[kLzWarps + 1];
    if (inv) *inv = red[kLzWarps + 2];
    __syncthreads();
    return s;
}

// x[l]: shared memory, or global memory written earlier in this launch by other
// CTAs (read through L2, never a possibly stale L1 line)
template <bool kGlobal>
__device__ __forceinline__ double xload(const double *x, int l) {
    if constexpr (kGlobal) return __ldcg(x + l);
    else return x[l];
}

// out[i] = scale * sum_l M(l, i) x[l] over the rows l of column i that may be
// non-zero (tri 0: all; 1: l >= i, M lower; 2: l <= i, M upper), for the columns
// of this CTA; returns this CTA's sum of out[i] * y[i] * ys (y may be null).
template <bool kGlobal>
__device__ double column_dots(const double *__restrict__ M, int ld, int n, int tri, const double *x, double *out,
                              double scale, const double *y, double ys, double *red) {
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    double mine = 0.0;
    for (int i = blockIdx.x + (int)gridDim.x * warp; i < n; i += (int)gridDim.x * kLzWarps) {
        const int lo = tri == 1 ? i : 0, hi = tri == 2 ? i + 1 : n;
        const double *col = M + (size_t)i * ld;
        double a0 = 0.0, a1 = 0.0, a2 = 0.0, a3 = 0.0;
        int l = lo + lane;
        for (; l + 96 < hi; l += 128) {
            a0 = fma(__ldcs(col + l), xload<kGlobal>(x, l), a0);
            a1 = fma(__ldcs(col + l + 32), xload<kGlobal>(x, l + 32), a1);
            a2 = fma(__ldcs(col + l + 64), xload<kGlobal>(x, l + 64), a2);
            a3 = fma(__ldcs(col + l + 96), xload<kGlobal>(x, l + 96), a3);
        }
        for (; l < hi; l += 32) a0 = fma(__ldcs(col + l), xload<kGlobal>(x, l), a0);
        double s = (a0 + a1) + (a2 + a3);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) {
            s *= scale;
            out[i] = s;
            if (y) mine = fma(s, __ldcg(y + i) * ys, mine);
        }
    }
    return block_sum(lane == 0 ? mine : 0.0, red);
}

// out <- scale * M^T x (column dots as above) with x = src staged in shared
// memory when it fits, read through L2 otherwise
__device__ double product(const double *__restrict__ M, int ld, int n, int tri, const double *src, double *out,
                          double scale, const double *y, double ys, double *xs, double *red) {
    if (n > kXsCap) return column_dots<true>(M, ld, n, tri, src, out, scale, y, ys, red);
    for (int i = threadIdx.x; i < n; i += kLzThreads) xs[i] = __ldcg(src + i);
    __syncthreads();
    const double r = column_dots<false>(M, ld, n, tri, xs, out, scale, y, ys, red);
    return r;  // block_sum's barriers keep xs until every warp is done
}

__global__ void __launch_bounds__(kLzThreads) lanczos64_kernel(const LzArgs a) {
    extern __shared__ double xs[];  // [min(n, kXsCap)], then kRedSlots reduction slots
    double *red = xs + (a.n > kXsCap ? 0 : a.n);
    const int n = a.n, ld = a.ld, k = a.k, g = gridDim.x;
    const int stride = g * kLzThreads;
    double *pa = a.part, *pb = a.part + g;
    // r_{-1}: a deterministic start with every component present; q_0 = r_{-1} / |r_{-1}|
    double acc = 0.0;
    for (int i = blockIdx.x * kLzThreads + threadIdx.x; i < n; i += stride) {
        const double v = 1.0 + 0.5 * sin(1.37 * i + 0.2);
        a.r[i] = v;
        acc = fma(v, v, acc);
    }
    acc = block_sum(acc, red);
    if (threadIdx.x == 0) pb[blockIdx.x] = acc;
    if (!grid_barrier(a.bar_count, g, a.err)) return;
    double sq = 0.0;  // q_j = r[j & 3] * sq
    grid_sum(pb, g, true, red, &sq);
    double sp = 0.0, bprev = 0.0;              // q_{j-1} = r[(j + 3) & 3] * sp
    for (int j = 0; j < k; ++j) {
        const double *rq = a.r + (size_t)(j & 3) * ld, *rp = a.r + (size_t)((j + 3) & 3) * ld;
        double *rw = a.r + (size_t)((j + 1) & 3) * ld;
        double part;
        if (!a.G) {
            part = product(a.H, ld, n, 0, rq, rw, sq, rq, sq, xs, red);
        } else {
            double *t1 = a.t, *t2 = a.t + ld;
            product(a.G, ld, n, 1, rq, t1, 1.0, nullptr, 0.0, xs, red);  // G^T r
            if (!grid_barrier(a.bar_count, g, a.err)) return;
            product(a.H, ld, n, 0, t1, t2, 1.0, nullptr, 0.0, xs, red);  // h (.)
            if (!grid_barrier(a.bar_count, g, a.err)) return;
            part = product(a.Gt, ld, n, 2, t2, rw, sq, rq, sq, xs, red);  // G (.) sq
        }
        if (threadIdx.x == 0) pa[blockIdx.x] = part;
        if (!grid_barrier(a.bar_count, g, a.err)) return;
        const double alpha = grid_sum(pa, g, false, red);
        // r_j = w - alpha q_j - beta_{j-1} q_{j-1}
        acc = 0.0;
        for (int i = blockIdx.x * kLzThreads + threadIdx.x; i < n; i += stride) {
            double x = __ldcg(rw + i) - alpha * (__ldcg(rq + i) * sq);
            if (j > 0) x -= bprev * (__ldcg(rp + i) * sp);
            rw[i] = x;
            acc = fma(x, x, acc);
        }
        acc = block_sum(acc, red);
        if (threadIdx.x == 0) pb[blockIdx.x] = acc;
        if (!grid_barrier(a.bar_count, g, a.err)) return;
        double ibeta = 0.0;
        const double beta = grid_sum(pb, g, true, red, &ibeta);
        const bool stop = !(beta > 1e-10 * (fabs(alpha) + 1.0));  // invariant subspace found
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            a.rec[j] = alpha;
            a.rec[k + j] = beta;
            if (stop) a.rec[2 * k] = j + 1;
        }
        if (stop) return;
        sp = sq;
        sq = ibeta;
        bprev = beta;
    }
}

// ---- explicit operator, every CTA with the whole vectors -----------------------
// One hand-over per step instead of two grid barriers: each CTA forms w = H~ q for
// its rows and publishes them (exchange.cuh); every CTA then reads all of w and
// carries q_j and q_{j-1} and the scalars itself, by the same operations in the same
// order, so that all agree to the bit.  p = w - beta_{j-1} q_{j-1}, alpha = p . q and
// beta^2 = |p|^2 - alpha^2 from one pass over p; a second pass sums |p - alpha q|^2 where
// that difference would cancel by more than a factor of eight (beta loses two bits at most;
// on the C/H/O systems beta^2 stays above a quarter of |p|^2, so the second pass is rare).  Bound: the FP64 unit for the products above
// about N = 700, latency below.  Twenty steps: N = 62 217 -> 75 us, N = 744 272 -> 174,
// N = 932 275 -> 193, N = 1860 379 -> 300.
constexpr int kLrThreads = 256, kLrWarps = kLrThreads / 32, kLrBatch = 4;
constexpr size_t kLrSmem = 220 * 1024;
constexpr double kLrCancel = 0.125;

struct LrArgs {
    int n, ld, k;
    const double *H;
    ulonglong2 *x;            // [2][n] exchanged words
    unsigned long long tag0;  // a value no earlier launch used, its low 32 bits zero
    double *rec;              // alpha [k], beta [k], steps used [1]
    int *err;
    unsigned long long limit;  // of the waits
    int exit_cta1;             // test hook: 1 + the CTA that leaves at once (0: none)
};

__global__ void __launch_bounds__(kLrThreads, 1) lanczos_rows_kernel(const LrArgs a) {
    extern __shared__ double dyn[];
    __shared__ double s_red[2][kLrWarps], s_sc[4];
    __shared__ int s_abort;
    if ((int)blockIdx.x + 1 == a.exit_cta1) return;  // test hook: the other CTAs' waits run out
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int n = a.n, rows = (n + gridDim.x - 1) / gridDim.x;
    const int r0 = min(n, (int)blockIdx.x * rows), nrow = min(n, r0 + rows) - r0;
    double *q = dyn, *p = dyn + n;        // q_j; q_{j-1}, overwritten by p and then by q_{j+1}
    double *sh = dyn + 2 * (size_t)n;
    if (tid == 0) s_abort = 0;
    for (int r = 0; r < nrow; ++r)
        for (int j = tid; j < n; j += kLrThreads) sh[(size_t)r * n + j] = a.H[(size_t)(r0 + r) * a.ld + j];
    // the start vector (every component present), published like a product
    for (int r = tid; r < nrow; r += kLrThreads)
        publish(a.x + r0 + r, (unsigned long long)__double_as_longlong(1.0 + 0.5 * sin(1.37 * (r0 + r) + 0.2)), a.tag0);
    for (int i = tid; i < 2 * n; i += kLrThreads) dyn[i] = 0.0;
    __syncthreads();
    double beta = 0.0;
    for (int j = -1; j < a.k; ++j) {
        const unsigned long long tag = a.tag0 + (unsigned long long)(j + 1);
        ulonglong2 *x = a.x + (size_t)((j + 1) & 1) * n;
        if (j >= 0) {
            for (int r = warp; r < nrow; r += kLrWarps) {
                const double *h = sh + (size_t)r * n;
                double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
                int l = lane;
                for (; l + 96 < n; l += 128) {
                    s0 = fma(h[l], q[l], s0);
                    s1 = fma(h[l + 32], q[l + 32], s1);
                    s2 = fma(h[l + 64], q[l + 64], s2);
                    s3 = fma(h[l + 96], q[l + 96], s3);
                }
                for (; l < n; l += 32) s0 = fma(h[l], q[l], s0);
                double s = (s0 + s1) + (s2 + s3);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                if (lane == 0) publish(x + r0 + r, (unsigned long long)__double_as_longlong(s), tag);
            }
        }
        // all of w: p = w - beta q_{j-1}; sums p . q (j >= 0) and |p|^2
        double pq = 0.0, pp = 0.0;
        for (int i0 = warp * 32; i0 < n; i0 += kLrBatch * kLrThreads) {
            ulonglong2 w[kLrBatch];
#pragma unroll
            for (int u = 0; u < kLrBatch; ++u) {
                const int i = i0 + u * kLrThreads + lane;
                w[u] = make_ulonglong2(0ull, tag);
                if (i < n) w[u] = fetch(x + i);
            }
            if (!await_words(w, tag, x + i0 + lane, kLrThreads, a.err, a.limit)) s_abort = 1;
#pragma unroll
            for (int u = 0; u < kLrBatch; ++u) {
                const int i = i0 + u * kLrThreads + lane;
                if (i0 + u * kLrThreads >= n) break;  // the same for the warp
                if (i < n) {
                    const double v = fma(-beta, p[i], __longlong_as_double((long long)w[u].x));
                    p[i] = v;
                    pq = fma(v, q[i], pq);
                    pp = fma(v, v, pp);
                }
            }
        }
        // lanes 0-15 sum p . q, lanes 16-31 |p|^2; then the eight warps' sums in warp order
        auto block_sums = [&](double x0, double x1) {
            const bool upper = lane & 16;
            double v = upper ? x1 : x0;
            v += __shfl_xor_sync(0xffffffffu, upper ? x0 : x1, 16);
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if ((lane & 15) == 0) s_red[lane >> 4][warp] = v;
            __syncthreads();
        };
        block_sums(pq, pp);
        if (s_abort) return;
        if (warp == 0) {
            double v = s_red[lane >> 4][lane & 7];
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            const double alpha = __shfl_sync(0xffffffffu, v, 0), p2 = __shfl_sync(0xffffffffu, v, 16);
            if (lane == 0) {
                const double b2 = p2 - alpha * alpha, ib = rsqrt(b2);
                s_sc[0] = alpha;
                s_sc[1] = b2 > kLrCancel * p2 ? 1.0 : 0.0;  // else |p - alpha q|^2 is summed
                s_sc[2] = b2 * ib;
                s_sc[3] = ib;
            }
        }
        __syncthreads();
        const double alpha = s_sc[0];
        if (s_sc[1] == 0.0) {
            double rr = 0.0;
            for (int i = tid; i < n; i += kLrThreads) {
                const double v = p[i] - alpha * q[i];
                rr = fma(v, v, rr);
            }
            block_sums(rr, 0.0);
            if (warp == 0) {
                double v = s_red[0][lane & 7];
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
                if (lane == 0) {
                    s_sc[2] = sqrt(v);
                    s_sc[3] = 1.0 / s_sc[2];
                }
            }
            __syncthreads();
        }
        const double ib = s_sc[3];
        beta = s_sc[2];
        if (j >= 0) {
            const bool stop = !(beta > 1e-10 * (fabs(alpha) + 1.0));  // invariant subspace found
            if (blockIdx.x == 0 && tid == 0) {
                a.rec[j] = alpha;
                a.rec[a.k + j] = beta;
                if (stop) a.rec[2 * a.k] = j + 1;
            }
            if (stop) return;
        }
        // q_{j+1} = (p - alpha q_j) / beta (the start vector: j = -1, q = 0); roles swap
        for (int i = tid; i < n; i += kLrThreads) p[i] = (p[i] - alpha * q[i]) * ib;
        double *t = q;
        q = p;
        p = t;
        if (j < 0) beta = 0.0;
        __syncthreads();
    }
}

// shared memory of a CTA: its rows of H~ and the two vectors
size_t rows_smem(int n, int sms) { return (size_t)(2 + (n + sms - 1) / sms) * n * sizeof(double); }

cudaError_t launch_rows(int n, int ld, int k, const double *H, double *x, double *rec, int *err, int sms,
                        cudaStream_t st, unsigned long long wait_ns, int exit_cta1) {
    static unsigned long long launches = 0;  // under the library's lock
    const int rows = (n + sms - 1) / sms, grid = (n + rows - 1) / rows;
    const size_t smem = rows_smem(n, sms);
    cudaError_t e = cudaFuncSetAttribute(lanczos_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    LrArgs a{n, ld, k, H, reinterpret_cast<ulonglong2 *>(x), ++launches << 32, rec, err, wait_ns ? wait_ns : kBarrierNs,
             std::min(exit_cta1, grid)};
    void *args[] = {&a};
    e = cudaLaunchCooperativeKernel((const void *)lanczos_rows_kernel, dim3(grid), dim3(kLrThreads), args, smem, st);
    count_launch();
    return e;
}

}  // namespace

cudaError_t launch_lanczos64(int n, int ld, int k, const double *H, const double *G, const double *Gt, double *r,
                             double *t, double *part, int part_cap, double *rec, unsigned *bar, int *err,
                             cudaStream_t st,
                             unsigned long long wait_ns, int exit_cta1) {
    static int grid = 0;
    if (!grid) {  // one CTA per SM, co-resident at the largest shared-memory size
        const int smem_max = (int)((kXsCap + kRedSlots) * sizeof(double));
        int dev = 0, sms = 0, per = 0;
        cudaError_t e = cudaFuncSetAttribute(lanczos64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_max);
        if (e == cudaSuccess) e = cudaGetDevice(&dev);
        if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
        if (e == cudaSuccess)
            e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, lanczos64_kernel, kLzThreads, smem_max);
        if (e != cudaSuccess) return e;
        if (per < 1) return cudaErrorInvalidConfiguration;
        grid = sms;
    }
    // explicit operator while its rows fit (N up to about 1,900; read from L2 by eight warps
    // a step at N = 3720 takes 57 us against lanczos64_kernel's 43): the words' [2][n] x 16
    // bytes lie in r's 4 x ld doubles
    if (!G && n >= 1 && k >= 1 && rows_smem(n, grid) <= kLrSmem)
        return launch_rows(n, ld, k, H, r, rec, err, grid, st, wait_ns, exit_cta1);
    const size_t smem = (size_t)(std::min(n, kXsCap) + kRedSlots) * sizeof(double);
    if (grid > part_cap || k < 1 || n < 1 || (G && !Gt)) return cudaErrorInvalidValue;
    LzArgs a{n, ld, k, H, G, Gt, r, t, part, rec, bar, err};
    void *args[] = {&a};
    cudaError_t e = cudaMemsetAsync(bar, 0, 2 * sizeof(unsigned), st);
    if (e == cudaSuccess)
        e = cudaLaunchCooperativeKernel((const void *)lanczos64_kernel, dim3(grid), dim3(kLzThreads), args, smem, st);
    count_launch();
    return e;
}

}  // namespace elhl
