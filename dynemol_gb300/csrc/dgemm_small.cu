// FP64 products of the factorisations' smallest blocks (up to 192 rows):
//   C = alpha op(A) op(B) + beta C, flags and masking as in dgemm.cu.
// At these sizes the product is a matter of latency, not of the FP64 pipe (64^3: 0.5 us
// if every SM took part): dgemm.cu's 16 x 16 tiles of one 64^3 product are 16 CTAs whose
// warps issue 32 FMAs each on top of one another (a warp instruction occupies its SM
// sub-partition for about 70 cycles), behind a scheduler's counter, two staged k tiles
// and, for split k ranges, a second pass: 10 us.  Here a CTA forms an 8 x 4 tile, one
// output per lane, its eight warps taking every eighth k: 128 CTAs for 64^3, eight FMAs
// per warp, all operands of a warp asked for at once, no staging, no scheduler.
#include "elhl_internal.cuh"

namespace elhl {
namespace {

constexpr int kTM = 8, kTN = 4, kWarps = 8;
constexpr int kUnroll = 8;  // k values of a warp in flight

struct SmallArgs {
    int m, n, k;
    double alpha, beta;
    const double *A, *B;
    double *C;
    int lda, ldb, ldc, tri;
};

template <bool TA, bool TB>
__global__ void __launch_bounds__(32 * kWarps) dgemm_small_kernel(const SmallArgs g) {
    __shared__ double part[kWarps][32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tri = g.tri;
    const int i0 = blockIdx.x * kTM, j0 = blockIdx.y * kTN;
    if ((tri & kTriLowerC) && i0 + kTM <= j0) return;  // tile strictly above the diagonal
    const int i = i0 + lane % kTM, j = j0 + lane / kTM;
    int klo = 0, khi = g.k;
    if (tri & kTriA) khi = min(khi, i0 + kTM);   // op(A)(i, l) = A(i, l) = 0 for l > i
    if (tri & kTriAt) klo = max(klo, i0);        // op(A)(i, l) = A(l, i) = 0 for l < i
    if (tri & kTriB) klo = max(klo, j0);         // op(B)(l, j) = B(l, j) = 0 for l < j
    if (tri & kTriBt) khi = min(khi, j0 + kTN);  // op(B)(l, j) = B(j, l) = 0 for l > j
    const bool in = i < g.m && j < g.n;
    double acc = 0.0;
    for (int l0 = klo + warp; l0 < khi; l0 += kWarps * kUnroll) {
        double a[kUnroll], b[kUnroll];
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) {
            const int l = l0 + kWarps * u;
            const bool on = in && l < khi;
            const bool za = ((tri & kTriA) && l > i) || ((tri & kTriAt) && l < i);
            const bool zb = ((tri & kTriB) && l < j) || ((tri & kTriBt) && l > j);
            a[u] = on && !za ? g.A[TA ? (size_t)i * g.lda + l : (size_t)l * g.lda + i] : 0.0;
            b[u] = on && !zb ? g.B[TB ? (size_t)l * g.ldb + j : (size_t)j * g.ldb + l] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < kUnroll; ++u) acc = fma(a[u], b[u], acc);
    }
    part[warp][lane] = acc;
    __syncthreads();
    if (warp || !in) return;
    double s[kWarps];
#pragma unroll
    for (int w = 0; w < kWarps; ++w) s[w] = part[w][lane];
#pragma unroll
    for (int o = kWarps / 2; o > 0; o >>= 1)
#pragma unroll
        for (int w = 0; w < o; ++w) s[w] += s[w + o];
    double *c = g.C + (size_t)j * g.ldc + i;
    *c = g.beta == 0.0 ? g.alpha * s[0] : fma(g.alpha, s[0], g.beta * *c);
}

}  // namespace

cudaError_t dgemm_small(int m, int n, int k, double alpha, const double *A, int lda, bool transA, const double *B,
                        int ldb, bool transB, double beta, double *C, int ldc, cudaStream_t st, int tri) {
    if (m <= 0 || n <= 0) return cudaSuccess;
    const SmallArgs g{m, n, k, alpha, beta, A, B, C, lda, ldb, ldc, tri};
    const dim3 grid((m + kTM - 1) / kTM, (n + kTN - 1) / kTN);
    if (transA && transB) dgemm_small_kernel<true, true><<<grid, 32 * kWarps, 0, st>>>(g);
    else if (transA) dgemm_small_kernel<true, false><<<grid, 32 * kWarps, 0, st>>>(g);
    else if (transB) dgemm_small_kernel<false, true><<<grid, 32 * kWarps, 0, st>>>(g);
    else dgemm_small_kernel<false, false><<<grid, 32 * kWarps, 0, st>>>(g);
    count_launch();
    return cudaGetLastError();
}

}  // namespace elhl
