// Persistent FP64 engine for the reference's adaptive-tau Taylor propagator.
//
// Semantics follow Taylor.f:35-239 (Propagation, Convergence, coefficient,
// isConverged) with bra propagated by H'^T and ket by H' (bra_x_op / op_x_ket,
// Matrix_math.f:225-301), for one or two particles (electron, hole) at once.
// In multi-step mode the kernel also runs the step driver of ElHl_Chebyshev
// (ElHl_Chebyshev.f:174-187, :267) for fixed nuclei and records populations
// (pop_Slater, data_output.f:242-262) after every step.
//
// Execution model: one cooperative launch, at most one CTA per SM.  Each CTA
// owns a contiguous block of rows; one "round" = one expansion order for every
// active particle:
//   products   the CTA's rows of H'^T.bra and H'.ket;
//   epilogue   one warp per eight rows forms the scaled term, the partial sum
//              and, where the round decides something, the CTA's record
//              (max |delta|^2 of bra and ket, <bra|ket>);
//   exchange   the vector that follows (as a rule) and the records go from CTA to
//              CTA as words tagged with the round, polled by their readers
//              (exchange.cuh); a bounded grid barrier instead where the kernel is not
//              resident, without L.words, at a step's first round and where another
//              vector follows (both give up after kBarrierNs and report
//              ELHL_ERR_TIMEOUT instead of hanging);
//   advance    one warp per particle sums the records in a fixed order and
//              advances an identical copy of the particle's state machine in
//              every CTA, with no host round trip, while the other warps
//              already form the next round's products on the vector that
//              follows unless this round ended an expansion (then they are
//              formed again).
// Vectors live in kSlots slots per particle; "Psi = new" and the term/partial-
// sum rotation are slot renames, never copies.
//
// What bounds a round is GB300's FP64 unit: a warp instruction takes its SM
// sub-partition 64 cycles whatever the active lanes, and a dependent one waits
// as long, so a round costs what its FP64 warp instructions and their longest
// chain cost.  Hence
//   - kResident (N up to about 1250): H' rows and columns of the CTA stay in
//     shared memory for the whole launch, and a lane owns one of the four sums
//     (re, im of ket and bra) of every row over every 64th column, so that a
//     row's sums meet over eight lanes (one add per row) instead of 32 lanes
//     and 31 adds per four rows;
//   - no hypot in the round (|delta|^2 against tol^2, as integers for the
//     maximum), |<bra|ket>| only where the decision needs it, the expansion's
//     coefficient ratios kept with the coefficients (computed by the lanes of
//     one warp in parallel), and no record exchange in rounds that decide
//     nothing;
//   - at least kMinRows rows per CTA: with fewer rows the barrier's arrivals
//     cost more than the products saved;
//   - grid_arrive / grid_poll (grid_sync.cuh) instead of grid_barrier.
// Measured, one particle at N = 465 (the 150-atom drop-in call, 3254 rounds): 23 us
// per round before (one thread per column, 32 accumulators each), 6.4 us with a barrier
// per round (products 5,900 cycles, 5,400 of them the FP64 unit's time for the 72 warp
// instructions of each sub-partition, barrier 2,750, epilogue 1,950, vectors 850), 4.8 us
// with the words.
#include <cooperative_groups.h>

#include <algorithm>

#include "elhl_internal.cuh"
#include "exchange.cuh"
#include "grid_sync.cuh"

namespace elhl {
namespace {

constexpr int RC = 4;            // rows per register chunk
constexpr int PMAX = 2;          // particles per launch
constexpr int PW = 16;           // record width (doubles)
constexpr int kWarps = kTaylorBlock / 32;
constexpr int kMinRows = 2;      // rows per CTA below which CTAs are left out of the launch
constexpr size_t kResidentSmem = 220 * 1024;

enum Phase { PH_NORM = 0, PH_CONV = 1, PH_MAIN = 2, PH_DONE = 3 };
enum { NEED_COEF = 1, NEED_KMAX = 2 };  // what a state change asks of the particle's warp

struct Ctrl {
    int phase, first, k, kmax;
    int psi, src, old, out_term, out_acc;
    int conv_calls, conv_step, substeps, status;
    long long orders;
    double tau, t, norm_ref, save_tau;
    double g[kOrder];  // |c_k / c_{k-1}|, 0-based k: c_k / c_{k-1} = -i g[k]
};

__device__ void pick_out_slots(Ctrl &c) {
    int found = 0;
    for (int s = 0; s < kSlots && found < 2; ++s) {
        if (s == c.psi || s == c.src || s == c.old) continue;
        if (found == 0) c.out_term = s; else c.out_acc = s;
        ++found;
    }
}

// coefficient(tau): c_1 = 1, c_k = -i c_{k-1} tau/(k-1) (Taylor.f:224-239): |c_k| by
// that recursion and the ratios g, lane k holding order k (0-based); with kmax,
// the first k >= 2 (1-based) with |c_k| < 1e-16, at most kOrder (Taylor.f:165-171).
__device__ void set_coefficients(Ctrl &c, int need, int lane) {
    const double tau = c.tau;
    const double f = lane >= 1 && lane < kOrder ? tau / (double)lane : 0.0;
    double m = 1.0, mine = 1.0, before = 1.0;
    for (int k = 1; k < kOrder; ++k) {
        const double prev = m;
        m = m * __shfl_sync(0xffffffffu, f, k);
        if (k == lane) {
            mine = m;
            before = prev;
        }
    }
    if (lane >= 1 && lane < kOrder) c.g[lane] = (mine * before) / (before * before);
    if (need & NEED_KMAX) {
        const unsigned small = __ballot_sync(0xffffffffu, lane >= 1 && lane < kOrder && fabs(mine) < 1.0e-16);
        if (lane == 0) c.kmax = small ? __ffs(small) : kOrder;
    }
    __syncwarp();
}

__device__ int start_conv(Ctrl &c, int max_calls) {
    if (c.conv_step >= max_calls) {
        c.status = ELHL_ERR_NO_CONVERGENCE;
        c.phase = PH_DONE;
        return 0;
    }
    c.conv_calls++;
    c.conv_step++;
    c.src = c.psi;
    c.old = c.psi;
    c.k = 2;
    c.phase = PH_CONV;
    pick_out_slots(c);
    return NEED_COEF | NEED_KMAX;
}

__device__ void start_main(Ctrl &c) {
    c.src = c.psi;
    c.old = c.psi;
    c.k = 2;
    c.phase = PH_MAIN;
    pick_out_slots(c);
}

// After an accepted convergence sub-step (Taylor.f:71-78 first time, :116-121 later).
__device__ int after_accept(Ctrl &c, double t_init, double t_max) {
    int need = 0;
    c.substeps++;
    if (c.first) {
        c.save_tau = c.tau;
        c.t = t_init + c.tau * kHbar;
        c.first = 0;
    } else {
        c.t = c.t + (c.tau * kHbar);
    }
    if (t_max - c.t < c.tau * kHbar) {
        c.tau = (t_max - c.t) / kHbar;
        need = NEED_COEF;
    }
    if (c.t < t_max) start_main(c); else c.phase = PH_DONE;
    return need;
}

// the next order of the running expansion
__device__ void next_order(Ctrl &c) {
    c.old = c.out_acc;
    c.src = c.out_term;
    c.k++;
    pick_out_slots(c);
}

// does this round end in a decision (the records are read)?
__device__ __forceinline__ bool decides(const Ctrl &c) {
    return c.phase == PH_NORM || c.phase == PH_CONV || (c.phase == PH_MAIN && c.k >= c.kmax);
}

// State change after a round, lane 0 of the particle's warp; tot = max |delta|^2 of
// bra and ket, <bra|ket>.  Returns NEED_* flags for the warp.
__device__ int advance(Ctrl &c, const double *tot, double tol2, double norm_tol, int max_calls, double t_init,
                       double t_max) {
    if (c.phase == PH_NORM) {
        c.norm_ref = hypot(tot[2], tot[3]);  // Taylor.f:62
        c.first = 1;
        c.conv_step = 0;
        return start_conv(c, max_calls);
    }
    if (c.phase == PH_CONV) {
        c.orders++;
        if (!(tot[0] > tol2) && !(tot[1] > tol2) && fabs(hypot(tot[2], tot[3]) - c.norm_ref) < norm_tol) {
            c.psi = c.out_acc;
            return after_accept(c, t_init, t_max);
        }
        if (c.k + 1 > c.kmax) {
            c.tau = c.tau * (c.first ? 0.9 : 0.975);  // Taylor.f:69, :110
            return start_conv(c, max_calls);
        }
        next_order(c);
        return 0;
    }
    if (c.phase == PH_MAIN) {
        c.orders++;
        if (c.k < c.kmax) {
            next_order(c);
            return 0;
        }
        if (fabs(hypot(tot[2], tot[3]) - c.norm_ref) < norm_tol) {  // Taylor.f:103-106
            int need = 0;
            c.psi = c.out_acc;
            c.substeps++;
            c.t = c.t + (c.tau * kHbar);
            if (t_max - c.t < c.tau * kHbar) {
                c.tau = (t_max - c.t) / kHbar;
                need = NEED_COEF;
            }
            if (c.t < t_max) start_main(c); else c.phase = PH_DONE;
            return need;
        }
        c.tau = c.tau * 0.975;  // Taylor.f:107-114
        return start_conv(c, max_calls);
    }
    return 0;
}

// maximum of two non-negative doubles (NaN counts as the largest), on their bits
__device__ __forceinline__ double max_bits(double a, double b) {
    const unsigned long long x = (unsigned long long)__double_as_longlong(a),
                             y = (unsigned long long)__double_as_longlong(b);
    return x > y ? a : b;
}

// columns padded to whole eight-column lane groups
__host__ __device__ constexpr int pad8(int n) { return (n + 7) & ~7; }

// dynamic shared memory: resident [P][pad8 N][4] vectors, [rows][pad8 N][2] matrix
// elements (row i, column i) and the warps' sums [kWarps][P][rows][4]; otherwise
// the row sums [P][rows][4]
size_t taylor_smem(int N, int rows, int P, bool resident) {
    const size_t y = (size_t)P * rows * 4 * sizeof(double);
    if (!resident) return y;
    return (size_t)pad8(N) * (4 * P + 2 * rows) * sizeof(double) + kWarps * y;
}

template <int P, bool kResident>
__global__ void __launch_bounds__(kTaylorBlock, 1) taylor_kernel(TaylorLaunch L) {
    extern __shared__ __align__(16) double dyn[];
    __shared__ Ctrl ctrl[P];
    __shared__ double red[kWarps][16 * P];       // non-resident: a chunk's warp sums
    __shared__ double unit_rec[kWarps][4];       // records of the epilogue's units
    __shared__ int s_step, s_it, s_ok, s_abort;
    __shared__ double s_tinit, s_tmax;

    const int G = gridDim.x;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int N = L.N, ld = L.ld, ldv = L.ldv;
    const int rows = (N + G - 1) / G;            // rows of a CTA (the last ones may have fewer)
    const int r0 = min(N, blockIdx.x * rows), r1 = min(N, r0 + rows), nrow = r1 - r0;
    const int np = pad8(N);
    const int nf = L.nfrag < kMaxFrag ? L.nfrag : kMaxFrag;
    double *sv = dyn;                                    // resident: [P][np][4] ket re, im, bra re, im
    double *sh = dyn + (size_t)P * np * 4;               // resident: [rows][np][2] H'(i, j), H'(j, i)
    double *sy = kResident ? sh + (size_t)rows * np * 2 : dyn;  // [kWarps][P][rows][4] or [P][rows][4]

    auto vec = [&](int p, int slot, int which) -> double2 * {
        return L.slots + ((size_t)(p * kSlots + slot) * 2 + which) * ldv;
    };

    if (tid == 0) {
        s_abort = (int)blockIdx.x + 1 == L.exit_cta1;  // test hook: it leaves after the first round, the others' waits run out
        s_step = 0;
        s_it = L.it0;
        s_tinit = L.t_init;
        s_tmax = L.t_max;
        for (int p = 0; p < P; ++p) {
            Ctrl &c = ctrl[p];
            c.phase = PH_NORM;
            c.first = 1;
            c.psi = 0; c.src = 0; c.old = 0; c.out_term = 1; c.out_acc = 2;
            c.k = 2; c.kmax = kOrder;
            c.conv_calls = 0; c.conv_step = 0; c.substeps = 0; c.status = ELHL_OK; c.orders = 0;
            c.tau = L.part[p].tau_in;
            c.t = L.t_init;
            c.save_tau = 0.0;
        }
    }
    if constexpr (kResident) {
        for (int q = tid; q < rows * np; q += kTaylorBlock) {
            const int r = q / np, j = q % np;
            const bool in = r < nrow && j < N;
            sh[(size_t)q * 2 + 1] = in ? L.H[(size_t)(r0 + r) * ld + j] : 0.0;
        }
        for (int q = tid; q < rows * np; q += kTaylorBlock) {  // lanes along the rows of one column
            const int r = q % rows, j = q / rows;
            const bool in = r < nrow && j < N;
            sh[((size_t)r * np + j) * 2] = in ? L.H[(size_t)j * ld + r0 + r] : 0.0;
        }
        for (int q = tid; q < P * np * 4; q += kTaylorBlock) sv[q] = 0.0;  // padding columns stay zero
    }
    __syncthreads();

    // resident: the vectors of slot `slot` of particle p into shared memory.  Written by
    // other CTAs: L2 loads (L1 is not coherent across SMs).
    auto stage = [&](int p, int slot) {
        const double2 *k = vec(p, slot, 1), *b = vec(p, slot, 0);
        double2 *dst = reinterpret_cast<double2 *>(sv + (size_t)p * np * 4);
#pragma unroll 8
        for (int q = tid; q < 2 * N; q += kTaylorBlock) {
            const int j = q >> 1;
            dst[q] = __ldcg(((q & 1) ? b : k) + j);
        }
    };
    // resident: the warp's t-th group of eight columns.  The warps that advance the
    // particles' states (0 .. P - 1) take half the others' share: their other FP64
    // instructions fall into the products' time.
    auto group_of = [&](int t) {
        constexpr int kOther = kWarps - P, kCycle = 2 * kOther + P;
        return warp < P ? t * kCycle + 2 * kOther + warp : (t >> 1) * kCycle + (t & 1) * kOther + warp - P;
    };
    // the row sums of the active particles' source vectors
    auto products = [&](const int (&src)[P], const bool (&act)[P]) {
        if constexpr (kResident) {
            const int comp = lane & 3, slice = lane >> 2;
#pragma unroll
            for (int p = 0; p < P; ++p) {
                if (!act[p]) continue;
                const double *x = sv + (size_t)p * np * 4 + lane;
                for (int c0 = 0; c0 < nrow; c0 += RC) {
                    const int nr = min(RC, nrow - c0);
                    const double *h = sh + ((size_t)c0 * np + slice) * 2 + (comp >> 1);
                    double v[RC];
#pragma unroll
                    for (int r = 0; r < RC; ++r) v[r] = 0.0;
                    if (nr == RC) {
#pragma unroll 2
                        for (int t = 0, jb; (jb = group_of(t)) < np / 8; ++t) {
                            const double xv = x[jb * 32];
#pragma unroll
                            for (int r = 0; r < RC; ++r)
                                v[r] = fma(h[((size_t)r * np + jb * 8) * 2], xv, v[r]);
                        }
                    } else {
#pragma unroll 2
                        for (int t = 0, jb; (jb = group_of(t)) < np / 8; ++t) {
                            const double xv = x[jb * 32];
#pragma unroll
                            for (int r = 0; r < RC; ++r)
                                if (r < nr) v[r] = fma(h[((size_t)r * np + jb * 8) * 2], xv, v[r]);
                        }
                    }
                    // over the eight lanes of a component: rows split over lane bits 4 and 3, then bit 2
#pragma unroll
                    for (int o = 16, half = RC / 2; half > 0; o >>= 1, half >>= 1) {
                        const bool upper = (lane & o) != 0;
#pragma unroll
                        for (int i = 0; i < half; ++i) {
                            const double send = upper ? v[i] : v[i + half];
                            const double keep = upper ? v[i + half] : v[i];
                            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                        }
                    }
                    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 4);
                    const int row = c0 + ((lane & 16) ? 2 : 0) + ((lane & 8) ? 1 : 0);
                    if (!(lane & 4) && row < nrow) sy[((size_t)(warp * P + p) * rows + row) * 4 + comp] = v[0];
                }
            }
        } else {
            for (int c0 = r0; c0 < r1; c0 += RC) {
                const int nr = min(RC, r1 - c0);
                double v[16 * P];
#pragma unroll
                for (int q = 0; q < 16 * P; ++q) v[q] = 0.0;
                for (int j = tid; j < N; j += kTaylorBlock) {
                    double hk[RC], hb[RC];
#pragma unroll
                    for (int r = 0; r < RC; ++r) {
                        const int i = c0 + (r < nr ? r : 0);
                        hk[r] = L.H[(size_t)j * ld + i];   // H'(i, j): row block (ket)
                        hb[r] = L.H[(size_t)i * ld + j];   // H'(j, i): column block (bra, H'^T)
                    }
#pragma unroll
                    for (int p = 0; p < P; ++p) {
                        if (!act[p]) continue;
                        const double2 vk = __ldcg(vec(p, src[p], 1) + j), vb = __ldcg(vec(p, src[p], 0) + j);
#pragma unroll
                        for (int r = 0; r < RC; ++r) {
                            double *a = v + (p * RC + r) * 4;
                            a[0] = fma(hk[r], vk.x, a[0]);
                            a[1] = fma(hk[r], vk.y, a[1]);
                            a[2] = fma(hb[r], vb.x, a[2]);
                            a[3] = fma(hb[r], vb.y, a[3]);
                        }
                    }
                }
                // warp sums: P = 1 first folds the lane halves, then a transposed butterfly,
                // after which lane l holds the sum of accumulator l % (16 P)
                if constexpr (P == 1) {
#pragma unroll
                    for (int i = 0; i < 16; ++i) v[i] += __shfl_xor_sync(0xffffffffu, v[i], 16);
                }
#pragma unroll
                for (int o = 8 * P; o > 0; o >>= 1) {
                    const bool upper = (lane & o) != 0;
#pragma unroll
                    for (int i = 0; i < o; ++i) {
                        const double send = upper ? v[i] : v[i + o];
                        const double keep = upper ? v[i + o] : v[i];
                        v[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
                    }
                }
                if (lane < 16 * P) red[warp][lane] = v[0];
                __syncthreads();
                if (tid < 16 * P) {
                    const int p = tid / 16, r = (tid / 4) % 4;
                    double s = 0.0;
                    for (int w = 0; w < kWarps; ++w) s += red[w][tid];
                    if (act[p] && r < nr) sy[((size_t)p * rows + c0 - r0 + r) * 4 + (tid & 3)] = s;
                }
                __syncthreads();
            }
        }
    };

    // (All waits take kBarrierNs: a limit that is no constant costs a round 0.3 to 0.5 %.)
    // Exchange without the barrier (resident, L.words): the round's next source and its
    // records go out as words tagged with the round, which the readers poll.  Two buffers
    // suffice: a CTA publishes round r + 2 once it has every CTA's words of round r + 1,
    // and those follow their CTA's use of round r.
    const bool words = kResident && L.words != nullptr;
    unsigned long long round = 0;
    auto word = [&](int p) { return L.words + ((size_t)(round & 1) * PMAX + p) * 4 * N; };
    auto rec_word = [&](int p) {
        return L.words + (size_t)2 * PMAX * 4 * N + ((size_t)(round & 1) * PMAX + p) * 4 * G;
    };
    // particle p's published vectors into shared memory as they arrive
    auto stage_words = [&](int p) {
        constexpr int U = 8;
        const ulonglong2 *src = word(p);
        double *dst = sv + (size_t)p * np * 4;
        for (int base = 0; base < 4 * N; base += U * kTaylorBlock) {
            ulonglong2 w[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int e = base + u * kTaylorBlock + tid;
                w[u] = e < 4 * N ? fetch(src + e) : make_ulonglong2(0ull, round);
            }
            if (!await_words(w, round, src + base + tid, kTaylorBlock, L.error, kBarrierNs)) s_abort = 1;
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int e = base + u * kTaylorBlock + tid;
                if (e < 4 * N) dst[e] = __longlong_as_double((long long)w[u].x);
            }
        }
    };

    int parity = 0;
    unsigned long long arrivals = 0;  // of the whole grid, at the next barrier's end
    double keep[P];                   // this lane's element of the last partial sum (first unit) ...
    int keep_slot[P];                 // ... and the slot it went to
#pragma unroll
    for (int p = 0; p < P; ++p) {
        keep[p] = 0.0;
        keep_slot[p] = -1;
    }
    // this CTA's record field q of particle p
    auto record = [&](int p, int q) -> double * {
        return L.partials + (((size_t)parity * PMAX + p) * G + blockIdx.x) * PW + q;
    };
    // this CTA's record field q of particle p in a decision of an expansion
    auto put_record = [&](int p, int q, double x) {
        if (words) publish(rec_word(p) + 4 * blockIdx.x + q, (unsigned long long)__double_as_longlong(x), round);
        else *record(p, q) = x;
    };
    // wait for the round's arrivals; false: the launch ends with an error
    auto wait_round = [&]() -> bool {
        arrivals += G;
        if (tid == 0) s_ok = grid_poll(L.bar_count, arrivals, L.error);
        __syncthreads();
        return s_ok;
    };
    bool ready = false;  // the next round's products are formed
    for (;;) {
        ++round;
        int src[P];
        bool act[P];
        bool norm = false;  // of every particle that is not done, or of none
#pragma unroll
        for (int p = 0; p < P; ++p) {
            src[p] = ctrl[p].src;
            act[p] = ctrl[p].phase == PH_CONV || ctrl[p].phase == PH_MAIN;
            norm |= ctrl[p].phase == PH_NORM;
        }
        if (!ready) {
            if constexpr (kResident) {
#pragma unroll
                for (int p = 0; p < P; ++p)
                    if (act[p]) stage(p, src[p]);
                __syncthreads();
            }
            products(src, act);
        }
        if (norm && warp < P && ctrl[warp].phase == PH_NORM) {  // <bra|ket> of the own rows
            const double2 *b = vec(warp, ctrl[warp].psi, 0), *k = vec(warp, ctrl[warp].psi, 1);
            double dre = 0.0, dim = 0.0;
            for (int i = r0 + lane; i < r1; i += 32) {
                const double2 bi = __ldcg(b + i), ki = __ldcg(k + i);
                dre += bi.x * ki.x + bi.y * ki.y;  // conj(bra) ket
                dim += bi.x * ki.y - bi.y * ki.x;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                dre += __shfl_xor_sync(0xffffffffu, dre, o);
                dim += __shfl_xor_sync(0xffffffffu, dim, o);
            }
            if (lane == 0) {
                *record(warp, 0) = *record(warp, 1) = 0.0;
                *record(warp, 2) = dre;
                *record(warp, 3) = dim;
            }
        }
        __syncthreads();

        // ------------------------------------------------ epilogue
        // unit u = (particle, eight rows), one warp each: lane = (row, component)
        const int groups = (nrow + 7) / 8;
        for (int p = 0; p < P; ++p) {
            if (!act[p]) continue;
            const Ctrl &c = ctrl[p];
            const bool rec = decides(c);
            const double gk = c.g[c.k - 1];
            const bool give_sum = c.phase == PH_MAIN && c.k >= c.kmax;  // the next source, as guessed below
            double best = 0.0, dot = 0.0;  // lanes of component 0 / 1: Re / Im of <bra|ket>
            // units dealt so that both particles' first units go to different warps
            for (int u = (warp + kWarps - p) % kWarps; u < groups; u += kWarps) {
                const int row = u * 8 + (lane >> 2), comp = lane & 3, i = r0 + row;
                const bool in = row < nrow;
                double y = 0.0;
                if (in) {
                    if constexpr (kResident) {
                        double w[kWarps];
#pragma unroll
                        for (int q = 0; q < kWarps; ++q) w[q] = sy[((size_t)(q * P + p) * rows + row) * 4 + comp];
#pragma unroll
                        for (int o = kWarps / 2; o > 0; o >>= 1)
#pragma unroll
                            for (int q = 0; q < o; ++q) w[q] += w[q + o];
                        y = w[0];
                    } else {
                        y = sy[((size_t)p * rows + row) * 4 + comp];
                    }
                }
                const double yo = __shfl_xor_sync(0xffffffffu, y, 1);  // the other part (re <-> im)
                double o = keep[p];
                const size_t e = (size_t)i * 2 + (comp & 1);
                if (in && (u > 0 || c.old != keep_slot[p])) o = __ldcg(reinterpret_cast<const double *>(vec(p, c.old, comp < 2)) + e);
                const double t = (comp & 1) ? -gk * yo : gk * yo;  // -i g y
                const double n = o + t;
                if (in) {
                    reinterpret_cast<double *>(vec(p, c.out_term, comp < 2))[e] = t;
                    reinterpret_cast<double *>(vec(p, c.out_acc, comp < 2))[e] = n;
                    if (words)
                        publish(word(p) + (size_t)i * 4 + comp,
                                (unsigned long long)__double_as_longlong(give_sum ? n : t), round);
                }
                if (u == 0) keep[p] = n;
                if (rec) {
                    const double d = n - o, d2 = d * d;
                    const double s = d2 + __shfl_xor_sync(0xffffffffu, d2, 1);  // |delta|^2: lanes 0, 1 ket, 2, 3 bra
                    best = max_bits(best, in ? s : 0.0);
                    // conj(bra) ket: re = br kr + bi ki, im = br ki - bi kr
                    const double nb = __shfl_xor_sync(0xffffffffu, n, 2), nbx = __shfl_xor_sync(0xffffffffu, nb, 1);
                    const double a = comp == 0 ? n * nb : comp == 1 ? n * nbx : 0.0;  // kr br | ki br
                    const double n1 = __shfl_xor_sync(0xffffffffu, n, 1);
                    const double b = comp == 0 ? n1 * nbx : comp == 1 ? -n1 * nb : 0.0;  // ki bi | -kr bi
                    if (in) dot += a + b;
                }
            }
            if (rec) {
                // over the unit's rows (lane bits 2-4), then over the warps' units
#pragma unroll
                for (int o = 16; o >= 4; o >>= 1) {
                    best = max_bits(best, __shfl_xor_sync(0xffffffffu, best, o));
                    dot += __shfl_xor_sync(0xffffffffu, dot, o);
                }
                if (groups <= 1) {
                    if (warp == p) {
                        if (lane == 0) {
                            put_record(p, 1, best);
                            put_record(p, 2, dot);
                        } else if (lane == 1) {
                            put_record(p, 3, dot);
                        } else if (lane == 2) {
                            put_record(p, 0, best);
                        }
                    }
                } else {
                    if (lane == 0) {
                        unit_rec[warp][1] = best;
                        unit_rec[warp][2] = dot;
                    } else if (lane == 1) {
                        unit_rec[warp][3] = dot;
                    } else if (lane == 2) {
                        unit_rec[warp][0] = best;
                    }
                    __syncthreads();  // every warp passes here for this particle
                    if (tid < 4) {
                        double s = unit_rec[0][tid];
                        for (int w = 1; w < kWarps; ++w)
                            s = tid < 2 ? max_bits(s, unit_rec[w][tid]) : s + unit_rec[w][tid];
                        put_record(p, tid, s);
                    }
                    __syncthreads();
                }
            }
            keep_slot[p] = c.out_acc;
        }
        const bool barrier = !words || norm;
        if (barrier) {
            if (P == 1 && groups <= 1) {  // warp 0 alone wrote global memory in this round
                __syncwarp();
            } else {
                __syncthreads();
            }
            if (tid == 0) grid_arrive(L.bar_count);
            if (!wait_round()) break;
        }

        // ------------------------------------------------ advance
        // The next round's source unless the advance decides otherwise: this round's
        // term, or the partial sum where a main expansion ends (it is accepted as a rule).
        int guess[P];
#pragma unroll
        for (int p = 0; p < P; ++p) {
            const Ctrl &c = ctrl[p];
            guess[p] = !act[p] ? -1 : c.phase == PH_MAIN && c.k >= c.kmax ? c.out_acc : c.out_term;
        }
        if constexpr (kResident) {
#pragma unroll
            for (int p = 0; p < P; ++p)
                if (act[p]) {
                    if (words) stage_words(p);
                    else stage(p, guess[p]);
                }
        }
        __syncthreads();  // ctrl has been read by every thread; the staged vectors are complete
        if (s_abort) break;
        if (warp < P) {
            // warp p: particle p's records summed in a fixed order (identical in every CTA)
            Ctrl &c = ctrl[warp];
            double v[4] = {0.0, 0.0, 0.0, 0.0};
            if (decides(c)) {
                // lanes 0-15 sum fields 0 and 2 (bra maximum, Re <bra|ket>), lanes 16-31 fields 1 and 3
                const double *rec = L.partials + ((size_t)parity * PMAX + warp) * G * PW + (lane >> 4);
                double m = 0.0, d = 0.0;
                if (barrier) {
#pragma unroll 5
                    for (int g = lane & 15; g < G; g += 16) {
                        m = max_bits(m, __ldcg(rec + (size_t)g * PW));
                        d += __ldcg(rec + (size_t)g * PW + 2);
                    }
                } else {
                    constexpr int U = 5;
                    const ulonglong2 *rw = rec_word(warp) + (lane >> 4);
                    for (int g0 = 0; g0 < G; g0 += 16 * U) {
                        ulonglong2 a[U], b[U];
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            const int g = g0 + 16 * u + (lane & 15);
                            a[u] = b[u] = make_ulonglong2(0ull, round);
                            if (g < G) {
                                a[u] = fetch(rw + 4 * g);
                                b[u] = fetch(rw + 4 * g + 2);
                            }
                        }
                        const ulonglong2 *at = rw + 4 * (g0 + (lane & 15));
                        if (!await_words(a, round, at, 64, L.error, kBarrierNs) ||
                            !await_words(b, round, at + 2, 64, L.error, kBarrierNs))
                            s_abort = 1;
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            m = max_bits(m, __longlong_as_double((long long)a[u].x));
                            d += __longlong_as_double((long long)b[u].x);
                        }
                    }
                }
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) {
                    m = max_bits(m, __shfl_xor_sync(0xffffffffu, m, o));
                    d += __shfl_xor_sync(0xffffffffu, d, o);
                }
                v[0] = m;
                v[2] = d;
                v[1] = __shfl_sync(0xffffffffu, m, 16);
                v[3] = __shfl_sync(0xffffffffu, d, 16);
            }
            int need = 0;
            if (lane == 0) need = advance(c, v, L.tol2, L.norm_tol, L.max_conv_calls, s_tinit, s_tmax);
            need = __shfl_sync(0xffffffffu, need, 0);
            if (need) set_coefficients(c, need, lane);
        }
        products(guess, act);
        __syncthreads();
        if (s_abort) break;
        parity ^= 1;

        bool all_done = true;
        ready = true;
#pragma unroll
        for (int p = 0; p < P; ++p) {
            const Ctrl &c = ctrl[p];
            all_done &= c.phase == PH_DONE;
            if (c.phase == PH_CONV || c.phase == PH_MAIN) ready &= c.src == guess[p];
        }
        if (!all_done) {
            if (!ready && !barrier) {  // another source than guessed: its slots, written before this barrier
                if (tid == 0) grid_arrive(L.bar_count);
                if (!wait_round()) break;
            }
            continue;
        }
        ready = false;

        // ---- step finished for every particle: population round + step driver
        if (L.pops && warp < P) {
            const int p = warp;
            const double2 *b = vec(p, ctrl[p].psi, 0), *k = vec(p, ctrl[p].psi, 1);
            for (int f = 0; f <= nf; ++f) {  // fragments, then the total
                double s = 0.0;
                for (int i = r0 + lane; i < r1; i += 32) {
                    if (f < nf && !(L.ao_frag && L.ao_frag[i] == f)) continue;
                    const double2 bi = __ldcg(b + i), ki = __ldcg(k + i);
                    s += ki.x * bi.x + ki.y * bi.y;  // Re conj(ket) bra
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                if (lane == 0) *record(p, 4 + f) = s;
            }
        }
        if (L.pops) {
            __syncthreads();
            if (tid == 0) grid_arrive(L.bar_count);
            if (!wait_round()) break;
        }
        if (blockIdx.x == 0 && warp < P && L.pops && s_step < L.nsteps) {
            const int p = warp;
            double *dst = L.pops + ((size_t)s_step * P + p) * (L.nfrag + 1);
            for (int f = 0; f <= nf; ++f) {
                double s = 0.0;
                for (int g = lane; g < G; g += 32)
                    s += __ldcg(L.partials + (((size_t)parity * PMAX + p) * G + g) * PW + 4 + f);
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
                if (lane == 0) dst[f == nf ? L.nfrag : f] = s;
            }
        }
        parity ^= 1;
        bool failed = false;
        for (int p = 0; p < P; ++p) failed |= (ctrl[p].status != ELHL_OK);
        const bool last = s_step + 1 >= L.nsteps;
        __syncthreads();
        if (last || failed) break;
        if (tid == 0) {
            // next nuclear step (ElHl_Chebyshev.f:174-187, :267): t_init = t, t_max = dt*fs*(it-1)
            s_step++;
            s_it++;
            s_tinit = s_tinit + L.dt_frame;
            s_tmax = L.dt_frame * (double)(s_it - 1);
            // first_call_ is already false after the launch's first step
            for (int p = 0; p < P; ++p) {
                Ctrl &c = ctrl[p];
                const double tau = c.save_tau * 1.15;
                c.tau = tau > L.tau_max ? L.tau_max : tau;
                c.t = s_tinit;
                c.phase = PH_NORM;
            }
        }
        __syncthreads();
    }

    // ------------------------------------------------ write-out: final Psi into slot 0
    // (own rows only; no other CTA touches them after the last barrier)
    __syncthreads();
    for (int p = 0; p < P; ++p) {
        const Ctrl &c = ctrl[p];
        if (c.psi == 0) continue;
        const double2 *b = vec(p, c.psi, 0), *k = vec(p, c.psi, 1);
        double2 *b0 = vec(p, 0, 0), *k0 = vec(p, 0, 1);
        for (int i = r0 + tid; i < r1; i += kTaylorBlock) {
            b0[i] = __ldcg(b + i);
            k0[i] = __ldcg(k + i);
        }
    }
    if (blockIdx.x == 0 && tid < P) {
        const Ctrl &c = ctrl[tid];
        TaylorParticle &o = L.part[tid];
        o.save_tau = c.save_tau;
        o.tau_out = c.tau;
        o.orders = c.orders;
        o.conv_calls = c.conv_calls;
        o.substeps = c.substeps;
        o.status = c.status;
        o.psi_slot = c.psi;
        if (tid == 0 && L.t_final) {
            // time after the last completed step (the driver's t)
            *L.t_final = s_tinit + L.dt_frame;
        }
    }
}

template <int P, bool kResident>
cudaError_t launch_taylor_t(const TaylorLaunch &L, int grid, int block, size_t smem, cudaStream_t st) {
    auto kern = taylor_kernel<P, kResident>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    TaylorLaunch copy = L;
    if (copy.exit_cta1 > grid) copy.exit_cta1 = grid;
    copy.tol2 = L.tol < 0.0 ? -1.0 : L.tol * L.tol;  // |delta| > tol < 0 always holds
    if (kResident && L.words) {  // no word carries a round's tag before the launch
        e = cudaMemsetAsync(L.words, 0, taylor_words(L.N, grid) * sizeof(ulonglong2), st);
        if (e != cudaSuccess) return e;
    }
    void *args[] = {&copy};
    e = cudaLaunchCooperativeKernel((const void *)kern, dim3(grid), dim3(block), args, smem, st);
    count_launch();
    return e;
}

}  // namespace

size_t taylor_words(int N, int grid) { return (size_t)2 * PMAX * 4 * ((size_t)N + grid); }

int taylor_grid_size(int block, int *grid_out) {
    int dev = 0, sms = 0, per_sm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return -1;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return -1;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, taylor_kernel<PMAX, false>, block, 0) != cudaSuccess)
        return -1;
    if (per_sm < 1) return -1;
    *grid_out = sms;  // one CTA per SM
    return 0;
}

// grid: the CTAs that may run (and that the partials' buffer has room for); the
// launch takes as many as the rows need at kMinRows or more per CTA.
cudaError_t launch_taylor(const TaylorLaunch &L, int grid, int block, cudaStream_t st) {
    if (L.N < 1 || grid < 1 || block != kTaylorBlock || L.nparticles < 1 || L.nparticles > PMAX)
        return cudaErrorInvalidValue;
    const int rows = std::max((L.N + grid - 1) / grid, kMinRows);
    const int ctas = (L.N + rows - 1) / rows;
    const int own = (L.N + ctas - 1) / ctas;  // as the kernel computes it
    const bool resident = taylor_smem(L.N, own, L.nparticles, true) <= kResidentSmem;
    const size_t smem = taylor_smem(L.N, own, L.nparticles, resident);
    if (L.nparticles == 1)
        return resident ? launch_taylor_t<1, true>(L, ctas, block, smem, st)
                        : launch_taylor_t<1, false>(L, ctas, block, smem, st);
    return resident ? launch_taylor_t<2, true>(L, ctas, block, smem, st)
                    : launch_taylor_t<2, false>(L, ctas, block, smem, st);
}

}  // namespace elhl
