// Split-precision GEMM on the 5th-generation tensor cores (tcgen05) for the
// Chebyshev GEMM regime:
//
//   Y (rows x n2, FP32, row-major) = sum_t A_t (rows x K) * B_t^T,   B_t: n2 x K
//
// A is the scaled Hamiltonian Hs split in three BF16 terms (Hs = A0 + A1 + A2,
// each the BF16 rounding of what the previous terms left), B the current
// Chebyshev block split the same way.  The six products A_i B_j with i + j <= 2
// reproduce FP32 products to about 2^-24 relative (the dropped terms are below
// 2^-27).  They accumulate in FP32 in tensor memory (TMEM), where every MMA rounds
// the running sum: the result's error grows with the length of that chain (16 K-chunks
// on one chain: 2.6 times the error of 6.4).  So a chain never crosses a K-chunk of 64:
// TMEM holds two sets of accumulators that alternate chunk by chunk, and while one set
// takes the next chunk the epilogue warps add the other to FP32 sums in registers (round
// to nearest; in FP32 pairs the error is the same, and the drain 9 us longer).  A0 B0
// takes kBig accumulators of a set in turn (as many as fit, up to the chunk's four MMAs),
// the five smaller products (2^-8 and below) one more.
//
// One CTA computes a 128-row tile of Y over all n2 columns for its K range, one wave of
// CTAs for the whole product (umma_splits); Y holds one FP32 partial per CTA and element.
//   warp 0  one elected thread issues the bulk copies (cp.async.bulk) of the six K-chunks
//           (64 BF16 = 128 B per row, 128B swizzle) of a stage,
//   warp 1  allocates TMEM and one elected thread issues tcgen05.mma
//           (kind::f16, BF16 x BF16 -> FP32, M = 128, N = n2, K = 16) and
//           tcgen05.commit to release a stage and to hand over a set,
//   the other warps (n2 / 8) drain the sets with tcgen05.ld (32 lanes x 16 columns per
//           instruction; a warp owns 32 rows x 32 columns) and store Y.
// Stages of six tiles, two (n2 = 128) or three, are buffered through mbarriers.  Every
// wait is bounded (globaltimer, 2 s): on a timeout the CTA records ELHL_ERR_TIMEOUT,
// stops issuing work, waits for what it issued and frees its TMEM.
//
// The MMA warp runs its loop as one and elects a lane only around the MMAs: descriptors
// computed by a single lane cost 37 cycles per MMA (N = 4092: 21.5 us at n2 = 32, 16.4 us
// so), more than the MMA itself at n2 <= 64.
//
// What bounds it, N = 4092: at n2 = 32 and 64 the 100 MB of A from memory (16.4 and
// 19.9 us per product; 36 and 36 us in the form below); at n2 = 128 the 96 KB per chunk
// out of L2, 196 MB in all (27.6 us, 40.3 us before; the MMAs alone would take 13.3).
// Chains over a CTA's whole K range with 10 CTAs per row tile (three waves, the third
// nearly empty) were the earlier form.
#include <algorithm>

#include "df64.cuh"
#include "elhl_internal.cuh"
#include "tc_ptx.cuh"

namespace elhl {
namespace {

constexpr int kBM = 128;        // rows per CTA (MMA M)
constexpr int kBK = 64;         // K per chunk: 64 BF16 = one 128-byte swizzle row
constexpr int kSMs = 152;
constexpr int kNumPairs = 6;    // (i, j) with i + j <= 2
constexpr unsigned long long kWaitNs = 2000000000ull;

using namespace tc;

struct UmmaParams {
    const unsigned char *A, *B;  // packed operands
    int rows, K;           // Y is rows x N2; the packed operands are zero past K
    int splits;            // CTAs along K per row tile (blockIdx.y)
    float *Y;              // [splits][rows][N2] partial tiles
    int *error;
};

template <int N2>
struct UmmaShape {
    static constexpr int kStages = N2 == 128 ? 2 : 3;
    static constexpr int kDrainWarps = N2 / 8, kThreads = 64 + 32 * kDrainWarps;  // 32 rows x 32 columns per warp
    static constexpr int kSlots = 256 / N2;                         // accumulators per set (two sets: 512 columns)
    static constexpr int kBig = kSlots - 1 < 4 ? kSlots - 1 : 4;    // of A0 B0; slot kBig: the smaller products
    static constexpr size_t kATile = (size_t)kBM * kBK * 2, kBTile = (size_t)N2 * kBK * 2;
    static constexpr size_t kStageBytes = 3 * (kATile + kBTile);
};

// dynamic shared memory: [stage][3 A tiles (128 x 64)][3 B tiles (N2 x 64)], then barriers
template <int N2>
__global__ void __launch_bounds__(UmmaShape<N2>::kThreads, 1)
    umma_bf16x3_kernel(UmmaParams p) {
    using S = UmmaShape<N2>;
    constexpr int kStages = S::kStages;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    // 1024-byte alignment for the 128B-swizzled tiles
    unsigned char *smem = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~static_cast<uintptr_t>(1023));
    uint64_t *full = reinterpret_cast<uint64_t *>(smem + kStages * S::kStageBytes);
    uint64_t *empty = full + kStages;
    uint64_t *set_full = empty + kStages;   // [2] a chunk's MMAs are done
    uint64_t *set_empty = set_full + 2;     // [2] every drain warp has read the set
    uint64_t *done = set_empty + 2;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(done + 1);
    int *abort_flag = reinterpret_cast<int *>(tmem_slot + 1);

    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int row0 = blockIdx.x * kBM;
    const int nk_all = (p.K + kBK - 1) / kBK;
    const int kc0 = (int)((long long)nk_all * blockIdx.y / p.splits);
    const int nk = (int)((long long)nk_all * (blockIdx.y + 1) / p.splits) - kc0;  // K chunks of this CTA
    float *Yp = p.Y + (size_t)blockIdx.y * p.rows * N2;

    if (threadIdx.x == 0) {
        for (int s = 0; s < kStages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int s = 0; s < 2; ++s) {
            mbar_init(&set_full[s], 1);
            mbar_init(&set_empty[s], S::kDrainWarps);
        }
        mbar_init(done, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;");
    const uint32_t tmem = *tmem_slot;

    if (warp == 0 && lane == 0) {
        // ---- TMA producer
        const unsigned char *a = p.A + ((size_t)blockIdx.x * nk_all + kc0) * (3 * S::kATile);
        const unsigned char *b = p.B + (size_t)kc0 * (3 * S::kBTile);
        int issued = 0;
        for (int kc = 0; kc < nk; ++kc) {
            const int s = kc % kStages;
            if (kc >= kStages && !mbar_wait(&empty[s], ((kc / kStages) - 1) & 1, kWaitNs)) {
                atomicExch(abort_flag, 1);
                break;
            }
            if (*(volatile int *)abort_flag) break;
            unsigned char *st = smem + s * S::kStageBytes;
            mbar_expect_tx(&full[s], (unsigned)S::kStageBytes);
            for (int t = 0; t < 3; ++t) {
                bulk_load(st + t * S::kATile, a + ((size_t)kc * 3 + t) * S::kATile, (unsigned)S::kATile, &full[s]);
                bulk_load(st + 3 * S::kATile + t * S::kBTile, b + ((size_t)kc * 3 + t) * S::kBTile,
                          (unsigned)S::kBTile, &full[s]);
            }
            ++issued;
        }
        // loads still in flight land before the CTA ends: wait for every issued stage
        for (int kc = (issued > kStages ? issued - kStages : 0); kc < issued; ++kc)
            mbar_wait(&full[kc % kStages], (kc / kStages) & 1, kWaitNs);
    } else if (warp == 1) {
        // ---- MMA issuer (the warp as one, so that descriptors stay in uniform registers)
        const uint32_t idesc = idesc_bf16(kBM, N2);
        const int pa[kNumPairs] = {0, 0, 1, 0, 1, 2};
        const int pb[kNumPairs] = {0, 1, 0, 2, 1, 0};
        for (int kc = 0; kc < nk; ++kc) {
            const int s = kc % kStages, set = kc & 1;
            if (!mbar_wait_warp(&full[s], (kc / kStages) & 1, kWaitNs) ||
                (kc >= 2 && !mbar_wait_warp(&set_empty[set], ((kc >> 1) - 1) & 1, kWaitNs))) {
                if (lane == 0) atomicExch(abort_flag, 1);
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;");
            unsigned char *st = smem + s * S::kStageBytes;
            const uint32_t base = tmem + (uint32_t)(set * S::kSlots * N2);
            const uint64_t d0 = smem_desc_sw128(st);
            if (elect_one()) {
#pragma unroll
                for (int q = 0; q < kNumPairs; ++q) {
#pragma unroll
                    for (int k = 0; k < kBK / 16; ++k) {  // K = 16 per MMA: +32 bytes along the swizzled row
                        const uint64_t da = d0 + (pa[q] * S::kATile + k * 32) / 16;
                        const uint64_t db = d0 + (3 * S::kATile + pb[q] * S::kBTile + k * 32) / 16;
                        const int slot = q == 0 ? k % S::kBig : S::kBig;
                        const int accumulate = q == 0 ? k >= S::kBig : !(q == 1 && k == 0);
                        umma_bf16(base + (uint32_t)(slot * N2), da, db, idesc, accumulate);
                    }
                }
                umma_commit(&empty[s]);       // the stage is free once these MMAs have read it
                umma_commit(&set_full[set]);  // and the set complete
            }
            __syncwarp();
        }
        if (elect_one()) umma_commit(done);
    } else if (warp >= 2) {
        // ---- drain: TMEM -> FP32 sums in registers, chunk by chunk; at the end -> Y
        constexpr int kCols = 32, kLd = 16;
        const int quad = warp & 3;  // this warp may read TMEM lanes [32 quad, 32 quad + 32)
        const int col0 = (warp - 2) / 4 * kCols;
        float sum[kCols];
#pragma unroll
        for (int q = 0; q < kCols; ++q) sum[q] = 0.f;
        bool ok = true;
        for (int kc = 0; kc < nk; ++kc) {
            const int set = kc & 1;
            if (lane == 0) ok = mbar_wait(&set_full[set], (kc >> 1) & 1, kWaitNs) && !*(volatile int *)abort_flag;
            ok = __shfl_sync(0xffffffffu, ok, 0);
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;");
            const uint32_t base = tmem + (uint32_t)(set * S::kSlots * N2 + col0) + ((uint32_t)(quad * 32) << 16);
#pragma unroll
            for (int c0 = 0; c0 < kCols; c0 += kLd) {
                uint32_t r[S::kBig + 1][kLd];
#pragma unroll
                for (int a = 0; a <= S::kBig; ++a) tmem_ld16(base + (uint32_t)(a * N2 + c0), r[a]);
                tmem_wait_ld();
#pragma unroll
                for (int q = 0; q < kLd; ++q) {
                    float x = __uint_as_float(r[S::kBig][q]);  // the small products first
#pragma unroll
                    for (int a = 0; a < S::kBig; ++a) x += __uint_as_float(r[a][q]);
                    sum[c0 + q] += x;
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;");
            __syncwarp();
            if (lane == 0) mbar_arrive(&set_empty[set]);
        }
        const int row = row0 + quad * 32 + lane;
        if (ok) {
            if (row < p.rows) {
                float4 *dst = reinterpret_cast<float4 *>(Yp + (size_t)row * N2 + col0);
#pragma unroll
                for (int q = 0; q < kCols / 4; ++q)
                    dst[q] = make_float4(sum[4 * q], sum[4 * q + 1], sum[4 * q + 2], sum[4 * q + 3]);
            }
        } else if (lane == 0) {
            atomicExch(abort_flag, 1);
        }
        if (lane == 0) mbar_wait(done, 0, kWaitNs);  // no MMA in flight when the TMEM is freed
    }
    asm volatile("tcgen05.fence::before_thread_sync;");
    __syncthreads();
    if (threadIdx.x == 0 && *(volatile int *)abort_flag) atomicExch(p.error, (int)ELHL_ERR_TIMEOUT);
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
    }
}

template <int N2>
int launch_umma(const UmmaParams &p, cudaStream_t st) {
    using S = UmmaShape<N2>;
    const size_t smem = 1024 + S::kStages * S::kStageBytes + 128;
    if (cudaFuncSetAttribute(umma_bf16x3_kernel<N2>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) !=
        cudaSuccess)
        return ELHL_ERR_CUDA;
    const dim3 grid((p.rows + kBM - 1) / kBM, p.splits);
    umma_bf16x3_kernel<N2><<<grid, S::kThreads, smem, st>>>(p);
    count_launch();
    return cudaGetLastError() == cudaSuccess ? ELHL_OK : ELHL_ERR_CUDA;
}

// Packed operand: for each tile of `tile` rows and each chunk of 64 K, the three terms'
// tiles as they lie in shared memory (rows of 128 B, 16-byte piece c of row r at piece
// c ^ (r & 7): the 128B swizzle), so that a chunk is one contiguous run of memory.
// KN (4 or 8) consecutive K from k0 on of one row: x = x0 + x1 + x2 in BF16 terms, each the
// rounding of the remainder.
template <int KN>
__device__ __forceinline__ void pack_row(unsigned char *dst, int tile, int nk, int row, int k0, const float (&x)[KN]) {
    unsigned w[3][KN / 2];
#pragma unroll
    for (int q = 0; q < KN / 2; ++q) {
        unsigned short v[2][3];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const __nv_bfloat16 a = __float2bfloat16_rn(x[2 * q + u]);
            const float ra = x[2 * q + u] - __bfloat162float(a);
            const __nv_bfloat16 b = __float2bfloat16_rn(ra);
            v[u][0] = __bfloat16_as_ushort(a);
            v[u][1] = __bfloat16_as_ushort(b);
            v[u][2] = __bfloat16_as_ushort(__float2bfloat16_rn(ra - __bfloat162float(b)));
        }
#pragma unroll
        for (int s = 0; s < 3; ++s) w[s][q] = (unsigned)v[0][s] | ((unsigned)v[1][s] << 16);
    }
    const int r = row % tile, c = (k0 % kBK) / 8;
    unsigned char *d = dst + ((size_t)(row / tile) * nk + k0 / kBK) * (3 * (size_t)tile * kBK * 2) + (size_t)r * kBK * 2 +
                       (size_t)((c ^ (r & 7)) * 16 + (k0 & 4) * 2);
#pragma unroll
    for (int s = 0; s < 3; ++s) {
        unsigned char *t = d + s * (size_t)tile * kBK * 2;
        if constexpr (KN == 8) *reinterpret_cast<uint4 *>(t) = make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
        else *reinterpret_cast<uint2 *>(t) = make_uint2(w[s][0], w[s][1]);
    }
}

// A of a symmetric H in FP32 (N columns of ld rows): a row's K are a column
__global__ void pack_h_kernel(const float *__restrict__ H, int N, int ld, unsigned char *dst, int nk) {
    const int k0 = 8 * (blockIdx.x * blockDim.x + threadIdx.x), row = blockIdx.y;
    if (k0 >= nk * kBK) return;
    float x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = row < N && k0 + u < N ? H[(size_t)row * ld + k0 + u] : 0.f;
    pack_row(dst, kBM, nk, row, k0, x);
}

// B of the Chebyshev block v (n rows of n2 reals): one row of B per column of v
__global__ void pack_v_kernel(const float *__restrict__ v, int n, int n2, unsigned char *dst, int nk) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, c = t % n2, k0 = 8 * (t / n2);
    if (k0 >= nk * kBK) return;
    float x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) x[u] = k0 + u < n ? v[(size_t)(k0 + u) * n2 + c] : 0.f;
    pack_row(dst, n2, nk, c, k0, x);
}

// y = sum of the nsplit partial products (fixed order, as an FP32 triple: closer than an FP64
// sum), v_k = 2 y - v_{k-2} (v_1 = y) rounded once to FP32, acc += c_k v_k
// in FP64, and v_k packed as the next product's B (rows past n keep the zeros that
// packing v_0 left).  A thread takes kEpiRows rows of one complex column, everything it
// reads asked for before the first result: bound by the FP64 unit (eight of its
// instructions per element, 4 us at N = 4092, 64 columns).  There 9.4 us, against 7.0 + 2.8
// and a launch with the packing apart; eight rows one after another took 17.6.
constexpr int kEpiRows = 4;
__global__ void __launch_bounds__(128) umma_epilogue_kernel(const float2 *__restrict__ Y, int nsplit,
                                                            size_t split_stride, const float2 *__restrict__ vprev2,
                                                            float2 *__restrict__ vout, double2 *__restrict__ acc,
                                                            const double2 *coef, int k, int n, int m,
                                                            unsigned char *dst, int nk) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, c = t % m, r0 = kEpiRows * (t / m);
    if (r0 >= n) return;
    const int rows = min(kEpiRows, n - r0);
    double2 a[kEpiRows];
    float2 w[kEpiRows];
    float yr[kEpiRows][3], yi[kEpiRows][3];
#pragma unroll
    for (int i = 0; i < kEpiRows; ++i) {
        const size_t q = (size_t)(r0 + min(i, rows - 1)) * m + c;
        a[i] = acc[q];
        w[i] = k == 1 ? make_float2(0.f, 0.f) : vprev2[q];
        const float2 y = Y[q];
        yr[i][0] = y.x;
        yi[i][0] = y.y;
        yr[i][1] = yr[i][2] = yi[i][1] = yi[i][2] = 0.f;
    }
    const double2 ck = coef[k];
    constexpr int kAhead = 3;  // partials under way together
    for (int s0 = 1; s0 < nsplit; s0 += kAhead) {
        float2 y[kAhead][kEpiRows];
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
#pragma unroll
            for (int i = 0; i < kEpiRows; ++i)
                y[u][i] = s0 + u < nsplit ? Y[(s0 + u) * split_stride + (size_t)(r0 + min(i, rows - 1)) * m + c]
                                          : make_float2(0.f, 0.f);
#pragma unroll
        for (int u = 0; u < kAhead; ++u)
#pragma unroll
            for (int i = 0; i < kEpiRows; ++i) {
                ts_add(yr[i], y[u][i].x);
                ts_add(yi[i], y[u][i].y);
            }
    }
    float re[kEpiRows], im[kEpiRows];
#pragma unroll
    for (int i = 0; i < kEpiRows; ++i) {
        if (k > 1) {
#pragma unroll
            for (int s = 0; s < 3; ++s) {
                yr[i][s] = __fmul_rn(2.f, yr[i][s]);
                yi[i][s] = __fmul_rn(2.f, yi[i][s]);
            }
            ts_add(yr[i], -w[i].x);
            ts_add(yi[i], -w[i].y);
        }
        const float2 v = make_float2(ts_round(yr[i][0], yr[i][1], yr[i][2]), ts_round(yi[i][0], yi[i][1], yi[i][2]));
        re[i] = im[i] = 0.f;
        if (i >= rows) continue;
        re[i] = v.x;
        im[i] = v.y;
        const size_t q = (size_t)(r0 + i) * m + c;
        vout[q] = v;
        double2 s = a[i];
        s.x += ck.x * (double)v.x - ck.y * (double)v.y;
        s.y += ck.x * (double)v.y + ck.y * (double)v.x;
        acc[q] = s;
    }
    pack_row(dst, 2 * m, nk, 2 * c, r0, re);
    pack_row(dst, 2 * m, nk, 2 * c + 1, r0, im);
}

}  // namespace

int umma_supported_n2(int n2) { return n2 >= 32 && n2 <= 128 && (n2 & (n2 - 1)) == 0; }

size_t umma_a_bytes(int N) { return (size_t)((N + kBM - 1) / kBM) * ((N + kBK - 1) / kBK) * 3 * kBM * kBK * 2; }

size_t umma_b_bytes(int N, int n2) { return (size_t)((N + kBK - 1) / kBK) * 3 * n2 * kBK * 2; }

int umma_pack_h(const float *H, int N, int ld, void *dst, cudaStream_t st) {
    const int nk = (N + kBK - 1) / kBK;
    const dim3 grid((nk * (kBK / 8) + 127) / 128, (N + kBM - 1) / kBM * kBM);
    pack_h_kernel<<<grid, 128, 0, st>>>(H, N, ld, static_cast<unsigned char *>(dst), nk);
    count_launch();
    return cudaGetLastError() == cudaSuccess ? ELHL_OK : ELHL_ERR_CUDA;
}

int umma_pack_v(const float *v, int n, int n2, void *dst, cudaStream_t st) {
    const int nk = (n + kBK - 1) / kBK;
    pack_v_kernel<<<(nk * (kBK / 8) * n2 + 127) / 128, 128, 0, st>>>(v, n, n2, static_cast<unsigned char *>(dst), nk);
    count_launch();
    return cudaGetLastError() == cudaSuccess ? ELHL_OK : ELHL_ERR_CUDA;
}

int umma_epilogue(const float *Y, int nsplit, const float2 *vprev2, float2 *vout, double2 *acc, const double2 *coef, int k,
                  int n, int m, void *dst, cudaStream_t st) {
    const int threads = (n + kEpiRows - 1) / kEpiRows * m;
    umma_epilogue_kernel<<<(threads + 127) / 128, 128, 0, st>>>(reinterpret_cast<const float2 *>(Y), nsplit,
                                                                (size_t)n * m, vprev2, vout, acc, coef, k, n, m,
                                                                static_cast<unsigned char *>(dst),
                                                                (n + kBK - 1) / kBK);
    count_launch();
    return cudaGetLastError() == cudaSuccess ? ELHL_OK : ELHL_ERR_CUDA;
}

int umma_splits(int rows, int K) {
    // the K split with the shortest sequence of waves, a CTA counted as its chunks and
    // three more for its first loads and its stores
    const int tiles = (rows + kBM - 1) / kBM, nk = (K + kBK - 1) / kBK;
    int best = 1;
    long long best_cost = 0;
    for (int s = 1; s <= std::min(16, nk); ++s) {
        const long long waves = ((long long)tiles * s + kSMs - 1) / kSMs, cost = waves * ((nk + s - 1) / s + 3);
        if (s == 1 || cost < best_cost) {
            best = s;
            best_cost = cost;
        }
    }
    return best;
}

int umma_bf16x3_gemm(const void *A, const void *B, int rows, int K, int n2, int splits, float *Y, int *d_error,
                     cudaStream_t st) {
    if (!umma_supported_n2(n2) || rows <= 0 || K <= 0) return ELHL_ERR_UNSUPPORTED;
    if (splits < 1 || ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(B)) & 15)) return ELHL_ERR_BAD_ARG;
    const UmmaParams p{static_cast<const unsigned char *>(A), static_cast<const unsigned char *>(B), rows, K, splits, Y,
                       d_error};
    switch (n2) {
        case 32: return launch_umma<32>(p, st);
        case 64: return launch_umma<64>(p, st);
        default: return launch_umma<128>(p, st);
    }
}

}  // namespace elhl
