// Dense Cholesky-with-inverse of one diagonal block of at most 64 rows in FP64:
// the leaves of the rebuild's recursive factorisation (S = L L^T with G = L^-1) for
// every precision, and of the drop-in's H' = S^-1 h.  Library triangular kernels
// at these sizes (cuSOLVER trtri on 256 rows, cuBLAS DTRMM/DTRSM panels) ran on a
// handful of CTAs for 65-106 us per call.
//
// The cost model is GB300's FP64 unit: one FP64 warp instruction occupies its SM
// sub-partition (SMSP) for 64-76 cycles whether 1 or 32 lanes are active, a
// dependent one waits as long.  One SM's unit alone needs 27 us for the 2 x 64^3/6
// FMAs of the factor and its inverse, and the chain of 64 pivots 22 us, so the work
// is one cluster of four CTAs:
//   CTA 0    the factor, by 8-column blocks b: F factors and inverts the 8 x 8
//            diagonal block (warp 0), P forms the panel below it, U updates what the
//            next block needs.  U runs beside the next F: warps 1-3 first update the
//            next diagonal block, on which F waits; warps 1-3 and 5-7 (not on warp
//            0's SMSP) then update the rest of the next block's columns and bring the
//            columns after that up to date with every panel so far (left-looking, so
//            that each step carries about the same work);
//            warp 4 sends the finished panel and the diagonal block's inverse to the
//            other CTAs (distributed shared memory).
//   CTAs 1-3 G = L^-1 by column blocks, right-looking: W_ij += L_ib G_bj as panel b
//            arrives, G_bj = -G_bb W_bj as the inverse of diagonal block b arrives, so
//            that only one such product remains when the factor ends.
// The pivots of F: reciprocal instead of reciprocal root in the chain (the roots of
// all eight pivots together afterwards), the eliminated column of A replaced in place
// by the inverse's, one FMA per lane and pivot for both.
// 66 us per leaf of 64 rows in one CTA, 41 us on the cluster with the pivots' elements found
// per lane in branches, 34.5 us with them in a table of offsets and L written after the loop:
// F 5,000 cycles, P 1,100-1,900, the next diagonal block 1,000, eight times.
#include "elhl_internal.cuh"
#include "grid_sync.cuh"

namespace elhl {
namespace {

constexpr int kLeafRows = 64, kThreads = 256, kCluster = 4;
constexpr int kB = 8, kBlocks = kLeafRows / kB;
constexpr int kPitch = kLeafRows + 2;      // row pitch of the factor (16-byte rows)
constexpr int kOwn = 3;                    // column blocks of G per CTA, at most
constexpr int kGPitch = kOwn * kB + 2;
constexpr int kUpdaters = 6;               // warps 1-3 and 5-7
constexpr unsigned long long kWaitNs = 2000000000ull;
// column blocks of G by CTA (balanced by their products in the last steps)
__constant__ int c_own[kCluster][kOwn] = {{-1, -1, -1}, {0, 5, -1}, {1, 4, 6}, {2, 3, 7}};

// element e of an 8 x 8 lower triangle, row by row
__device__ __forceinline__ void tri_elem(int e, int &i, int &j) {
    i = 0;
    while ((i + 1) * (i + 2) / 2 <= e) ++i;
    j = e - i * (i + 1) / 2;
}

// 1 / d by one step of Householder's third-order iteration for the root of 1 / y - d (A. S.
// Householder, The Numerical Treatment of a Single Nonlinear Equation, 1970; the geometric
// series of 1 / (1 - e)): y (1 + e + e^2), e = 1 - d y.  The start is rcp.approx.ftz.f64,
// whose result has 20 fraction bits: e is below 2^-19, so 1 - d y is exact in an FMA, the
// terms left out are below 2^-57, and the result is within 0.63 ulp of 1 / d (tested against
// exact quotients and against CUDA's division).  d and the start have to be normal; outside
// 2^-999 .. 2^998, well inside the normal range on either side, and for zero, infinities
// and NaN, the division.
__device__ __forceinline__ double reciprocal(double d) {
    const int ex = (__double2hiint(d) >> 20) & 0x7ff;
    if (ex < 24 || ex > 2020) return 1.0 / d;
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(d));
    const double e = fma(-d, y, 1.0);
    return fma(y, fma(e, e, e), y);
}

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void cluster_barrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the address of this CTA's shared variable in CTA `rank` of the cluster
__device__ __forceinline__ unsigned remote(const void *p, unsigned rank) {
    unsigned a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((unsigned)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void store_remote(unsigned a, double x, double y) {
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(x), "d"(y) : "memory");
}
// whole warp: what its lanes stored in the CTAs 1 .. 3 is visible there before *flag = 1
__device__ __forceinline__ void raise_flag(int *flag) {
    asm volatile("fence.acq_rel.cluster;" ::: "memory");
    __syncwarp();
    const unsigned lane = threadIdx.x & 31;
    if (lane >= 1 && lane < kCluster)
        asm volatile("st.release.cluster.shared::cluster.u32 [%0], %1;" ::"r"(remote(flag, lane)), "r"(1) : "memory");
}
// one thread: bounded wait for a flag of this CTA
__device__ __forceinline__ bool wait_flag(const int *flag, unsigned long long limit_ns) {
    const unsigned a = (unsigned)__cvta_generic_to_shared(flag);
    unsigned long long t0 = 0;
    for (unsigned n = 1;; ++n) {
        int v;
        asm volatile("ld.acquire.cluster.shared::cta.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
        if (v) return true;
        if ((n & 63u) == 0) {
            const unsigned long long t = globaltimer_ns();
            if (!t0) t0 = t;
            if (t - t0 > limit_ns) return false;
        }
    }
}

struct Smem {
    double A[kLeafRows * kPitch];          // CTA 0: A, then L; others: the panels of L
    double Gd[kBlocks][kB * kB];           // inverses of the diagonal blocks (zero above the diagonal)
    double G[kLeafRows * kGPitch];         // others: W, then G, of the CTA's column blocks
    // F: the block, its eliminated columns (unscaled), the pivots and their root's reciprocals
    double M[kB * kB], Lr[kB * kB], d[kB], rr[kB];
    double zero, one, dump;                // operands of F's lanes without an element, and where they write
    int flag_g[kBlocks], flag_p[kBlocks];  // others: Gd[b], panel b have arrived
    int ok;
};

// One lane's part of one pivot of F: out = m - (a u) / a_kk, with a also kept at `keep`
// (offsets in doubles from the start of Smem).
struct Step {
    short a, u, m, out, keep;
};
__device__ __forceinline__ short at(const Smem &s, const double *p) { return (short)(p - s.A); }
// The n-th element pivot k changes: a_ij (i >= j > k) and x_ij (j < k) take m = itself,
// a = a_ik, u = a_jk or x_kj; the new column x_ik takes u = 1, m = 0 and keeps a_ik.
__device__ __forceinline__ Step pivot_step(Smem &s, int k, int n) {
    const int updates = (kB * (kB - 1) - k * (k + 1)) / 2;
    if (n < updates) {
        int i = k + 1, e = n;
        while (e >= i) e -= i++;
        const int j = e < k ? e : e + 1;
        const short m = at(s, s.M + i * kB + j);
        return Step{at(s, s.M + i * kB + k), at(s, j > k ? s.M + j * kB + k : s.M + k * kB + j), m, m, at(s, &s.dump)};
    }
    const int i = k + 1 + n - updates;
    const short none = at(s, &s.dump), zero = at(s, &s.zero), c = at(s, s.M + i * kB + k);
    if (i < kB) return Step{c, at(s, &s.one), zero, c, at(s, s.Lr + i * kB + k)};
    return Step{zero, zero, zero, none, none};
}
constexpr int kTwice = 2;  // pivots with more than 32 elements (35, 33, then 30 and fewer)

// F, warp 0: the 8 x 8 block at (b0, b0) of s.A, all of its updates done: its Cholesky
// factor in place and the factor's inverse in s.Gd[b].  At pivot k, with m_i = a_ik / a_kk:
// a_ij -= m_i a_jk for i >= j > k and, for the unit lower inverse x kept where the
// columns <= k of A were, x_ij -= m_i x_kj for j < k and x_ik = -m_i: at most 35
// elements, one multiplication beside the reciprocal and one FMA after it.  A
// non-positive pivot of a real row (< nb) sets *info (the first one); nothing after it
// depends on the values.
__device__ __forceinline__ void factor_block(Smem &s, int b, int nb, int row0, const Step (&step)[kB - 1], const Step (&more)[kTwice],
                             int *info) {
    const int lane = threadIdx.x & 31, b0 = b * kB;
    double *w = s.A;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int e = lane + 32 * u;
        s.M[e] = s.A[(b0 + e / kB) * kPitch + b0 + e % kB];  // above the diagonal: not read
    }
#pragma unroll
    for (int k = 0; k < kB; ++k) {
        __syncwarp();
        const double d = s.M[k * kB + k];
        if (lane == 0) s.d[k] = d;
        if (k + 1 == kB) break;
        const Step &q = step[k < kB - 1 ? k : 0];
        const double a = w[q.a], m = w[q.m], t = a * w[q.u], inv = reciprocal(d), v = fma(-t, inv, m);
        if (k < kTwice) {
            const Step &r = more[k < kTwice ? k : 0];
            const double a2 = w[r.a], v2 = fma(-(a2 * w[r.u]), inv, w[r.m]);
            __syncwarp();
            w[r.out] = v2;
            w[r.keep] = a2;
        } else {
            __syncwarp();
        }
        w[q.out] = v;
        w[q.keep] = a;
    }
    __syncwarp();
    if (lane < kB) {
        const double d = s.d[lane];
        s.rr[lane] = rsqrt(d);
        const unsigned bad = __ballot_sync(0xffu, !(d > 0.0) && b0 + lane < nb);
        if (bad && lane == 0) atomicCAS(info, 0, row0 + b0 + __ffs(bad));
    }
    __syncwarp();
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int e = lane + 32 * u, i = e / kB, j = e % kB;
        double g = 0.0;
        if (i >= j) {
            s.A[(b0 + i) * kPitch + b0 + j] = (i > j ? s.Lr[e] : s.d[j]) * s.rr[j];
            g = i > j ? s.M[e] * s.rr[i] : s.rr[i];
        }
        s.Gd[b][e] = g;
    }
    __syncwarp();
}

// CTA 0: the factor
__device__ void factor_cta(Smem &s, double *A, int nb, int ld, int row0, int *info) {
    const int tid = threadIdx.x, warp = tid / 32, lane = tid & 31;
    const int blocks = (nb + kB - 1) / kB, end = blocks * kB;  // rows in use (padded to whole blocks)
    Step step[kB - 1], more[kTwice];
#pragma unroll
    for (int k = 0; k < kB - 1; ++k) step[k] = pivot_step(s, k, lane);
#pragma unroll
    for (int k = 0; k < kTwice; ++k) more[k] = pivot_step(s, k, 32 + lane);
    if (warp == 0) factor_block(s, 0, nb, row0, step, more, info);
    for (int b = 0; b < blocks; ++b) {
        const int b0 = b * kB, r0 = b0 + kB;
        const bool last = b + 1 == blocks;
        __syncthreads();  // F(b) and U(b - 1) done
        if (!last) {
            // P: L(i, b0 + t) = sum_{s <= t} A(i, b0 + s) Gd(t, s); a warp takes the columns t and
            // 7 - t (nine FMAs) of 32 rows, results held until every row has been read
            const int t0 = warp & 3, t1 = kB - 1 - t0, i = r0 + (warp >> 2) * 32 + lane;
            double o0 = 0.0, o1 = 0.0;
            if (i < end) {
                const double *a = s.A + i * kPitch + b0, *g0 = s.Gd[b] + t0 * kB, *g1 = s.Gd[b] + t1 * kB;
#pragma unroll
                for (int q = 0; q < kB; ++q) {
                    if (q <= t0) o0 = fma(a[q], g0[q], o0);
                    if (q <= t1) o1 = fma(a[q], g1[q], o1);
                }
            }
            __syncthreads();
            if (i < end) {
                s.A[i * kPitch + b0 + t0] = o0;
                s.A[i * kPitch + b0 + t1] = o1;
            }
            __syncthreads();
        }
        if (warp == 4) {
            // the inverse of the diagonal block, then the panel, to the CTAs 1 .. 3
            for (int c = 1; c < kCluster; ++c)
                store_remote(remote(&s.Gd[b][2 * lane], c), s.Gd[b][2 * lane], s.Gd[b][2 * lane + 1]);
            raise_flag(&s.flag_g[b]);
            for (int q = lane; q < (end - r0) * (kB / 2); q += 32) {
                const double *v = s.A + (r0 + q / (kB / 2)) * kPitch + b0 + 2 * (q % (kB / 2));
                for (int c = 1; c < kCluster; ++c) store_remote(remote(v, c), v[0], v[1]);
            }
            if (!last) raise_flag(&s.flag_p[b]);
        }
        if (last) break;
        if (warp == 0) {
            asm volatile("bar.sync 1, 128;" ::: "memory");  // the next diagonal block is up to date
            factor_block(s, b + 1, nb, row0, step, more, info);
            continue;
        }
        if (warp == 4) continue;
        if (warp < 4) {
            // the next diagonal block: 12 of its 36 elements per warp, two lanes of four FMAs each
            const int half = lane >= 12;
            int i, j;
            tri_elem((warp - 1) * 12 + lane % 12, i, j);
            const double *x = s.A + (r0 + i) * kPitch + b0 + 4 * half, *y = s.A + (r0 + j) * kPitch + b0 + 4 * half;
            double v = 0.0;
#pragma unroll
            for (int q = 0; q < 4; ++q) v = fma(x[q], y[q], v);
            v += __shfl_down_sync(0xffffffffu, v, 12);
            if (lane < 12) s.A[(r0 + i) * kPitch + r0 + j] -= v;
            asm volatile("bar.arrive 1, 128;" ::: "memory");
        }
        // the rows below it: the next block's columns with this panel (set 0), the columns after
        // those with every panel so far (set 1), in chunks of 32 elements along the rows
        const int c0 = r0 + kB, rows = end - c0, chunks = (rows * kB + 31) / 32;
        for (int q = warp < 4 ? warp - 1 : warp - 2; q < 2 * chunks; q += kUpdaters) {
            const bool ahead = q >= chunks;
            const int e = (ahead ? q - chunks : q) * 32 + lane, i = c0 + e % max(rows, 1), j = (ahead ? c0 : r0) + e / max(rows, 1);
            if (e >= rows * kB || i < j) continue;
            const int k0 = ahead ? 0 : b0;
            const double *x = s.A + i * kPitch, *y = s.A + j * kPitch;
            double v = s.A[i * kPitch + j];
#pragma unroll 8
            for (int k = k0; k < r0; ++k) v = fma(-x[k], y[k], v);
            s.A[i * kPitch + j] = v;
        }
    }
    // L, zero above the diagonal
#pragma unroll 4
    for (int e = tid; e < kLeafRows * kLeafRows; e += kThreads) {
        const int i = e % kLeafRows, j = e / kLeafRows;
        if (i < nb && j < nb) A[(size_t)j * ld + i] = i >= j ? s.A[i * kPitch + j] : 0.0;
    }
}

// CTAs 1 .. 3: the columns of G of their column blocks
__device__ void inverse_cta(Smem &s, unsigned rank, double *G, int nb, int ld, int *info,
                            unsigned long long limit_ns) {
    const int tid = threadIdx.x;
    const int blocks = (nb + kB - 1) / kB, end = blocks * kB;
    int own[kOwn];
#pragma unroll
    for (int q = 0; q < kOwn; ++q) own[q] = c_own[rank][q];
    // zero above the diagonal, and W
    for (int e = tid; e < kOwn * kB * kLeafRows; e += kThreads) {
        const int i = e % kLeafRows, c = e / kLeafRows, j = own[c / kB] * kB + c % kB;
        s.G[i * kGPitch + c] = 0.0;
        if (j >= 0 && j < nb && i < min(nb, own[c / kB] * kB)) G[(size_t)j * ld + i] = 0.0;
    }
    __syncthreads();
    for (int b = 0; b < blocks; ++b) {
        const int b0 = b * kB, r0 = b0 + kB;
        if (tid == 0) s.ok = wait_flag(&s.flag_g[b], limit_ns);
        __syncthreads();
        if (!s.ok) break;
        // row block b of G: -Gd W for the column blocks before b, Gd for b itself
        const int c = tid / kB, i = tid % kB, jb = c < kOwn * kB ? own[c / kB] : -1;
        double v = 0.0;
        if (jb >= 0 && jb < b) {
            for (int t = 0; t <= i; ++t) v = fma(-s.Gd[b][i * kB + t], s.G[(b0 + t) * kGPitch + c], v);
        } else if (jb == b) {
            v = s.Gd[b][i * kB + c % kB];
        }
        __syncthreads();  // W has been read
        if (jb >= 0 && jb <= b) {
            s.G[(b0 + i) * kGPitch + c] = v;
            const int j = jb * kB + c % kB;
            if (b0 + i < nb && j < nb) G[(size_t)j * ld + b0 + i] = v;
        }
        if (b + 1 == blocks) break;
        if (tid == 0) s.ok = wait_flag(&s.flag_p[b], limit_ns);
        __syncthreads();
        if (!s.ok) break;
        for (int e = tid; e < (end - r0) * kOwn * kB; e += kThreads) {  // W += L_b G_b, lanes along the rows
            const int r = r0 + e % (end - r0), q = e / (end - r0);
            if (own[q / kB] < 0 || own[q / kB] > b) continue;
            double w = s.G[r * kGPitch + q];
#pragma unroll
            for (int t = 0; t < kB; ++t) w = fma(s.A[r * kPitch + b0 + t], s.G[(b0 + t) * kGPitch + q], w);
            s.G[r * kGPitch + q] = w;
        }
        __syncthreads();
    }
    if (tid == 0 && !s.ok) atomicExch(info + 1, ELHL_ERR_TIMEOUT);
}

__global__ void __cluster_dims__(kCluster, 1, 1) __launch_bounds__(kThreads)
    leaf_chol_inv64_kernel(double *A, double *G, int nb, int ld, int row0, int *info, unsigned long long wait_ns,
                           bool mute) {
    extern __shared__ __align__(16) unsigned char raw[];
    Smem &s = *reinterpret_cast<Smem *>(raw);
    const unsigned rank = cluster_rank();
    const int tid = threadIdx.x;
    if (tid < kBlocks) s.flag_g[tid] = s.flag_p[tid] = 0;
    if (rank == 0) {
        constexpr int kLoads = kLeafRows * kLeafRows / kThreads;
        double v[kLoads];
#pragma unroll
        for (int q = 0; q < kLoads; ++q) {  // rows past nb: the identity
            const int e = tid + q * kThreads, i = e % kLeafRows, j = e / kLeafRows;
            v[q] = i == j ? 1.0 : 0.0;
            if (i < nb && j < nb && i >= j) v[q] = A[(size_t)j * ld + i];
        }
#pragma unroll
        for (int q = 0; q < kLoads; ++q) {
            const int e = tid + q * kThreads, i = e % kLeafRows, j = e / kLeafRows;
            s.A[i * kPitch + j] = v[q];
        }
        if (tid == 0) {
            s.zero = 0.0;
            s.one = 1.0;
        }
    }
    cluster_barrier();  // flags and A in place
    if (rank == 0 && mute) {  // test hook: no flag is raised, the other CTAs' waits run out
    } else if (rank == 0) factor_cta(s, A, nb, ld, row0, info);
    else inverse_cta(s, rank, G, nb, ld, info, wait_ns ? wait_ns : kWaitNs);
    cluster_barrier();  // no CTA leaves while its shared memory may still be written
}

__global__ void reciprocal_kernel(const double *x, double *y, double *q, int n) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    y[i] = reciprocal(x[i]);
    q[i] = 1.0 / x[i];
}

}  // namespace

int leaf_rows() { return kLeafRows; }

cudaError_t launch_reciprocal(const double *x, double *y, double *q, int n, cudaStream_t st) {
    if (n <= 0) return cudaSuccess;
    reciprocal_kernel<<<(n + 255) / 256, 256, 0, st>>>(x, y, q, n);
    count_launch();
    return cudaGetLastError();
}

cudaError_t leaf_chol_inv64(double *A, double *G, int nb, int ld, int row0, int *info, cudaStream_t st,
                            unsigned long long wait_ns, bool mute) {
    static bool attr = false;
    if (!attr) {
        cudaError_t e = cudaFuncSetAttribute(leaf_chol_inv64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)sizeof(Smem));
        if (e != cudaSuccess) return e;
        attr = true;
    }
    if (nb <= 0 || nb > kLeafRows) return cudaErrorInvalidValue;
    leaf_chol_inv64_kernel<<<kCluster, kThreads, sizeof(Smem), st>>>(A, G, nb, ld, row0, info, wait_ns, mute);
    count_launch();
    return cudaGetLastError();
}

}  // namespace elhl
